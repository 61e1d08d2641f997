"""Timed cases of the framework: what a user has it compute, at the sizes of
the benchmark configurations, between them, and at ragged ones.

    listed()            the named cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) the inputs on the GPU and the plan a program keeps
    run(state)          one pass through the public entry points
    work(case)          bytes and flops of one pass
    exact(case, seed)   the same outputs in 64 bits by plain torch

Every case is an observation of a satellite formation on a lunar orbit (the
law of the repository's synthetic observations): n_sat satellites, n_snap
snapshots, all baselines a < b, a HEALPix sky, optionally the Moon and the
Earth as occulters.  `kind` says which calls a pass makes:

    observe            forward, DCF and weights, imaging adjoint
    day                the same after staging the day's samples (the day loop)
    forward, adjoint   one call
    channels           forward and adjoint of several frequencies in one plan
    formation_forward, formation_adjoint   the calls on satellite vectors
    gridded            the gridded imaging adjoint
    gradient           loss and gradients (sky, satellite offsets) at two points
"""
from __future__ import annotations

import math

import torch

from viss_optimize_3d_b200 import api
from viss_optimize_3d_b200.autograd import VisibilityModel

LIGHT = 299792458.0
R_MOON = 1737.4e3
ORBIT = R_MOON + 300e3
EARTH_CAP = math.radians(0.95)
EXACT_TERMS = 1e12          # sample x pixel terms of exact() at most (under 20 s)


def _case(name, kind, nside, n_sat, n_snap, mhz, moon=False, earth=False, **more):
    c = {"kind": kind, "nside": nside, "n_sat": n_sat, "n_snap": n_snap, "mhz": mhz, "moon": moon,
         "earth": earth, "imaging_mask": True, "fp64": False, "channels": 1}
    c.update(more)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest observation of the configurations (1 MHz, no occultation):
        # launches and latency
        _case("observe_c1", "observe", 32, 8, 360, 1.0),
        # one day of the streaming loop at the 10 MHz Moon configuration: the
        # samples and occulter rows are new every day
        _case("day_c2", "day", 64, 8, 720, 10.0, True),
        # the FP64 option, and sizes that are no multiple of any tile
        _case("observe_fp64_ragged", "observe", 51, 7, 509, 10.0, True, True, fp64=True),
        # the headline configuration, each direction
        _case("forward_c3_10mhz", "forward", 256, 10, 8640, 10.0, True, True),
        _case("adjoint_c3_10mhz", "adjoint", 256, 10, 8640, 10.0, True, True),
        # the noblockage programs at 1 MHz: forward with occultation, imaging without
        _case("observe_c3_1mhz", "observe", 256, 10, 8640, 1.0, True, True, imaging_mask=False),
        # the headline configuration given as satellite vectors
        _case("formation_forward_c3", "formation_forward", 256, 10, 8640, 10.0, True, True),
        _case("formation_adjoint_c3", "formation_adjoint", 256, 10, 8640, 10.0, True, True),
        # the batched configuration with a quarter of its channels (1 to 10 MHz)
        _case("channels_c4", "channels", 128, 10, 2880, 10.0, True, True, channels=16),
        # sky and position gradients of the reconstruction, as a line search asks for them
        _case("gradient_c5", "gradient", 128, 10, 4320, 10.0, True),
        # production imaging at 1 MHz (Nside 512, one day of samples), unmasked
        _case("gridded_prod_1mhz", "gridded", 512, 10, 44448, 1.0, imaging_mask=False),
        # occulted gridded imaging
        _case("gridded_c3_1mhz", "gridded", 256, 10, 8640, 1.0, True, True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["observe", "observe", "day", "forward", "forward", "adjoint", "adjoint", "channels",
                       "formation_forward", "formation_adjoint", "gradient", "gridded"])
    nside = rng.choice([32, 64, 128, 256, _log(rng, 24, 256)])
    n_sat = rng.randint(3, 10)
    n_snap = _log(rng, 150, 8640)
    mhz = rng.choice([1.0, 10.0, round(rng.uniform(1.0, 10.0), 2)])
    moon = rng.random() < 0.7
    earth = moon and rng.random() < 0.6
    more = {"imaging_mask": rng.random() < 0.7}
    if kind == "channels":
        more["channels"] = rng.randint(2, 8)
        nside, n_snap = min(nside, 128), 2 * (min(n_snap, 2880) // 2)     # an even count of samples a channel
    elif kind == "gradient":
        nside, n_snap = min(nside, 128), min(n_snap, 4320)
    elif kind == "gridded":
        nside, mhz = max(nside, 64), min(mhz, 2.0)
    elif kind in ("observe", "forward", "adjoint") and nside <= 64 and rng.random() < 0.25:
        more["fp64"] = True
        n_snap = min(n_snap, 720)
    return _case("", kind, nside, n_sat, n_snap, mhz, moon, earth, **more)


# ------------------------------------------------------------------ inputs
def _shape(case):
    T, S = case["n_snap"], case["n_sat"]
    B = S * (S - 1) // 2
    return T, S, B, T * B, 12 * case["nside"] ** 2


def _lambdas(case):
    """Wavelengths of the channels: 1 MHz up to the case's frequency."""
    C, top = case["channels"], case["mhz"] * 1e6
    if C == 1:
        return [LIGHT / top]
    return [LIGHT / (1e6 + (top - 1e6) * c / (C - 1)) for c in range(C)]


def _inputs(case, seed):
    """Raw inputs of an observation, on the GPU (plain torch)."""
    T, S, B, K, J = _shape(case)
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(1_000_003 * (int(seed) + 1) + 17)

    def uniform(n, lo, hi):
        return lo + (hi - lo) * torch.rand(n, generator=g, device=dev, dtype=torch.float64)

    def normal(*n, dtype=torch.float64):
        return torch.randn(*n, generator=g, device=dev, dtype=dtype)

    along = torch.cat([torch.zeros(1, device=dev, dtype=torch.float64), uniform(S - 1, 1e3, 30e3).cumsum(0)])
    radial, cross = 500.0 * normal(S), 500.0 * normal(S)
    inc = math.radians(30.0)
    e1 = torch.tensor([1.0, 0.0, 0.0], device=dev, dtype=torch.float64)
    e2 = torch.tensor([0.0, math.cos(inc), math.sin(inc)], device=dev, dtype=torch.float64)
    e3 = torch.tensor([0.0, -math.sin(inc), math.cos(inc)], device=dev, dtype=torch.float64)
    t = torch.arange(T, device=dev, dtype=torch.float64) / T
    ang = 2 * math.pi * t[:, None] + along[None, :] / ORBIT
    P = (ORBIT + radial)[None, :, None] * (ang.cos()[..., None] * e1 + ang.sin()[..., None] * e2) \
        + cross[None, :, None] * e3
    a, b = torch.triu_indices(S, S, 1, device=dev)
    metres = (P[:, a] - P[:, b]).reshape(K, 3)
    C = case["channels"]
    sky = torch.exp(normal(C, J, dtype=torch.float32))
    at = torch.randint(J, (20,), generator=g, device=dev)
    sky[:, at] += uniform(20, 10.0, 100.0).float()
    sky = (sky * (4 * math.pi / J)).contiguous()
    d = {"P": P, "a": a, "b": b, "metres": metres, "sky": sky if C > 1 else sky[0],
         "uvw": torch.cat([metres / lam for lam in _lambdas(case)]).contiguous()}
    refs = earth = None
    if case["moon"] or case["earth"]:
        refs = torch.full((T, B, 3), -1, device=dev, dtype=torch.int32)
        snap = torch.arange(T, device=dev)[:, None]
        if case["moon"]:
            refs[:, :, 0], refs[:, :, 1] = snap * S + a, snap * S + b
        if case["earth"]:
            turn = torch.rand(1, generator=g, device=dev, dtype=torch.float64) * 2 * math.pi
            e = turn + math.radians(13.2) * (2.6 / 24) * t
            earth = torch.stack([-e.cos(), -e.sin(), torch.zeros_like(e), torch.full_like(e, -math.cos(EARTH_CAP))], 1)
            refs[:, :, 2] = T * S + snap
        refs = refs.reshape(K, 3).repeat(C, 1).contiguous()
    d["refs"], d["earth"] = refs, earth
    if case["kind"] in ("adjoint", "channels", "formation_adjoint", "gridded"):
        d["coef"] = torch.complex(normal(C * K, dtype=torch.float32), normal(C * K, dtype=torch.float32))
    if case["kind"] in ("observe", "day"):
        d["w"] = d["uvw"][:, 2].float().contiguous()
        d["bll"] = d["uvw"].norm(dim=1).float()
        d["nr"] = int(math.ceil(2.0 * float(d["bll"].max()) + 1.0))
    if case["kind"] == "gradient":
        d["delta"] = 5.0 * normal(2, S, 3)
        d["x"] = torch.exp(0.5 * normal(2, J, dtype=torch.float32))
        d["V_obs"] = torch.complex(normal(K, dtype=torch.float32), normal(K, dtype=torch.float32)) * (4 * math.pi / math.sqrt(J))
        d["wt"] = uniform(K, 0.5, 1.5).float()
    return d


def _occ(d):
    """The occulter table as a program builds it."""
    if d["refs"] is None:
        return None
    occ = api.occulters(d["P"].reshape(-1, 3), R=R_MOON, mode=0)
    return occ if d["earth"] is None else torch.cat([occ, d["earth"]])


def prepare(case, seed):
    d = _inputs(case, seed)
    kind = case["kind"]
    lmn = api.pix2lmn(case["nside"], "ring")
    occ = _occ(d)
    d["case"] = case
    if kind == "gradient":
        d["model"] = VisibilityModel(lmn, d["refs"], occ)
        return d
    if kind == "day":
        d["plan"] = api.Plan(lmn)
        return d
    if kind.startswith("formation"):
        T, S, _B, _K, _J = _shape(case)
        d["plan"] = api.Plan(lmn)
        U = (d["P"] - d["P"].mean(dim=1, keepdim=True)) / _lambdas(case)[0]
        moon = occ[:T * S].reshape(T, S, 4) if case["moon"] else None
        d["plan"].set_formation(U, None, moon, d["earth"])
        return d
    d["plan"] = api.Plan(lmn, d["uvw"], None, d["refs"], occ, channels=case["channels"])
    return d


# --------------------------------------------------------------------- runs
def _observe(d, case):
    V = d["plan"].forward(d["sky"], fp64=case["fp64"])
    gs, _counts, table = api.dcf(d["bll"], d["nr"], multiplicity=2)
    _dg, wt = api.weights(d["w"], d["bll"], gs, table, d["nr"])
    img = d["plan"].adjoint(api.scale_coef(wt, V), scale=2.0, fp64=case["fp64"], mask=case["imaging_mask"])
    return {"V": V, "weights": wt, "image": img}


def _offsets_uvw(d, delta, lam):
    P = d["P"] + delta
    return ((P[:, d["a"]] - P[:, d["b"]]) / lam).reshape(-1, 3)


def _gradient(d, case):
    """Loss and gradients at two points (new satellite offsets each)."""
    lam, omega, out = _lambdas(case)[0], 4 * math.pi / d["x"].shape[1], []
    for x0, delta0 in zip(d["x"], d["delta"]):
        x, delta = x0.clone().requires_grad_(True), delta0.clone().requires_grad_(True)
        V = d["model"](x * omega, _offsets_uvw(d, delta, lam))
        r = (V - d["V_obs"]).to(torch.complex128) * d["wt"].double()
        L = r.real.square().sum() + r.imag.square().sum()
        L.backward()
        out.append({"loss": L.detach().float(), "sky": x.grad, "offsets": delta.grad.float()})
    return out


def run(d):
    case = d["case"]
    kind = case["kind"]
    if kind == "observe":
        return _observe(d, case)
    if kind == "day":
        d["plan"].set_samples(d["uvw"], None, d["refs"], _occ(d))
        return _observe(d, case)
    if kind == "forward":
        return d["plan"].forward(d["sky"], fp64=case["fp64"])
    if kind == "adjoint":
        return d["plan"].adjoint(d["coef"], fp64=case["fp64"], mask=case["imaging_mask"])
    if kind == "channels":
        return {"V": d["plan"].forward(d["sky"]), "image": d["plan"].adjoint(d["coef"], mask=case["imaging_mask"])}
    if kind == "formation_forward":
        return d["plan"].forward_formation(d["sky"])
    if kind == "formation_adjoint":
        return d["plan"].adjoint_formation(d["coef"], mask=case["imaging_mask"])
    if kind == "gridded":
        return d["plan"].adjoint_gridded(d["coef"], mask=case["imaging_mask"])
    return _gradient(d, case)


# --------------------------------------------------------------------- work
_PRODUCTS = {"observe": 2, "day": 2, "channels": 2, "gradient": 10}   # gradient: 2 points x (V, image, 3 phase derivatives)


def work(case):
    _T, _S, _B, K, J = _shape(case)
    n, C = _PRODUCTS.get(case["kind"], 1), case["channels"]
    # a term of the direct sum: phase (3 multiply-adds), sine and cosine, one complex multiply-add
    return {"bytes": n * C * (K * (24 + 8 + (12 if case["moon"] else 0)) + J * 4) + 24 * J,
            "flops": 12.0 * n * C * K * J}


# -------------------------------------------------------------------- exact
def _ring_lmn(nside):
    """(l, m, n) = (x, -y, z) of HEALPix RING pixel centres, FP64."""
    n, npix = nside, 12 * nside * nside
    p = torch.arange(npix, device="cuda", dtype=torch.int64)
    q = torch.minimum(p, npix - 1 - p)                       # the southern cap mirrors the northern one
    cap = 2 * n * (n - 1)
    i = ((1 + torch.sqrt((1 + 2 * q).double())) / 2).long().clamp(min=1)
    i = torch.where(2 * i * (i - 1) > q, i - 1, i)
    i = torch.where(2 * i * (i + 1) <= q, i + 1, i)
    ic = i.double()
    j = (q + 1 - 2 * i * (i - 1)).double()
    zc, phic = 1 - ic * ic / (3.0 * n * n), (j - 0.5) * math.pi / (2 * ic)
    south = p >= npix - cap
    zc, phic = torch.where(south, -zc, zc), torch.where(south, 2 * math.pi - phic, phic)
    e = (p - cap).clamp(min=0)
    ring, k = e // (4 * n) + n, e % (4 * n) + 1
    odd = 0.5 * (1 + ((ring + n) % 2).double())
    ze, phie = (2 * n - ring).double() * 2 / (3 * n), (k.double() - odd) * math.pi / (2 * n)
    inside = (p >= cap) & (p < npix - cap)
    z, phi = torch.where(inside, ze, zc), torch.where(inside, phie, phic)
    r = torch.sqrt((1 - z) * (1 + z))
    return torch.stack([r * phi.cos(), -r * phi.sin(), z], 1)


def _visible(d, case, lmn, t0, t1):
    """(t1 - t0, B, J) visibility of the pixels from the pairs' satellites."""
    vis = None
    if case["moon"]:
        P = d["P"][t0:t1]
        r = P.norm(dim=2)
        cos = (P / r[..., None]).reshape(-1, 3) @ lmn.T
        sat = (cos >= -torch.sqrt(1 - (R_MOON / r) ** 2).reshape(-1, 1)).reshape(t1 - t0, case["n_sat"], -1)
        vis = sat[:, d["a"]] & sat[:, d["b"]]
    if d["earth"] is not None:
        e = d["earth"][t0:t1]
        seen = (e[:, :3] @ lmn.T >= e[:, 3:])[:, None, :]
        vis = seen if vis is None else vis & seen
    return vis


def _terms(d, case, uvw, lmn, masked):
    """Chunks (t0, t1, cos, sin) of e^{2 pi i u.s} with hidden pairs zero, (samples, J) each."""
    T, _S, B, _K, J = _shape(case)
    step = max(1, int(2.5e8 // (B * J)))
    for t0 in range(0, T, step):
        t1 = min(T, t0 + step)
        ph = uvw[t0 * B:t1 * B] @ lmn.T
        ph -= ph.round()
        ph *= 2 * math.pi
        c, s = ph.cos(), ph.sin_()
        if masked and d["refs"] is not None:
            vis = _visible(d, case, lmn, t0, t1).expand(t1 - t0, B, J).reshape(-1, J)
            c *= vis
            s *= vis
        yield t0 * B, t1 * B, c, s


def _forward64(d, case, uvw, lmn, skies, masked=True):
    """(K, n) complex128 of n skies (J, n)."""
    out = torch.empty(uvw.shape[0], skies.shape[1], dtype=torch.complex128, device="cuda")
    for k0, k1, c, s in _terms(d, case, uvw, lmn, masked):
        out[k0:k1] = torch.complex(c @ skies, -(s @ skies))
    return out


def _adjoint64(d, case, uvw, lmn, coef, masked):
    img = torch.zeros(lmn.shape[0], dtype=torch.float64, device="cuda")
    for k0, k1, c, s in _terms(d, case, uvw, lmn, masked):
        img += coef.real[k0:k1] @ c - coef.imag[k0:k1] @ s
    return img


def _weights64(d):
    """min(dcf dg, 1/8): the shell volume over its (doubled) count, and the w factor."""
    nr = d["nr"]
    shell = torch.ceil((d["bll"] - 0.25) * 2.0).long()          # a choice, made in the inputs' 32 bits
    counts = 2.0 * torch.bincount(shell[(shell >= 1) & (shell <= nr)] - 1, minlength=nr).double()
    k = torch.arange(1, nr + 1, device="cuda", dtype=torch.float64)
    R = 0.5 * k + 0.25
    table = torch.cat([torch.tensor([1 / (4 * math.pi)], device="cuda", dtype=torch.float64),
                       (2 * math.pi / 3) * (R ** 3 - (R - 0.5) ** 3) / counts])
    x = d["w"].double() / d["bll"].double()
    dg = torch.where(x.abs() < 1, 1.5 * (1 - 4 * x * x).abs().sqrt() / (1 - x * x).sqrt(),
                     torch.full_like(x, math.inf))
    return (table[shell.clamp(0, nr)] * dg).clamp(max=0.125)


def exact(case, seed):
    _T, S, B, K, J = _shape(case)
    kind, C = case["kind"], case["channels"]
    if float(K) * J * C * _PRODUCTS.get(kind, 1) > EXACT_TERMS:
        return None
    d = _inputs(case, seed)
    lmn = _ring_lmn(case["nside"])
    sky = d["sky"].double().reshape(C, J)
    if kind in ("observe", "day"):
        V = _forward64(d, case, d["uvw"], lmn, sky.T)[:, 0]
        wt = _weights64(d)
        return {"V": V, "weights": wt, "image": 2.0 * _adjoint64(d, case, d["uvw"], lmn, V * wt, case["imaging_mask"])}
    if kind in ("forward", "formation_forward"):
        return _forward64(d, case, d["uvw"], lmn, sky.T)[:, 0]
    if kind in ("adjoint", "formation_adjoint", "gridded"):
        return _adjoint64(d, case, d["uvw"], lmn, d["coef"].to(torch.complex128), case["imaging_mask"])
    if kind == "channels":
        V, img = [], []
        for c in range(C):
            u, coef = d["uvw"][c * K:(c + 1) * K], d["coef"][c * K:(c + 1) * K].to(torch.complex128)
            V.append(_forward64(d, case, u, lmn, sky[c][:, None])[:, 0])
            img.append(_adjoint64(d, case, u, lmn, coef, case["imaging_mask"]))
        return {"V": torch.cat(V), "image": torch.stack(img)}
    lam, omega, out = _lambdas(case)[0], 4 * math.pi / J, []
    for x, delta in zip(d["x"], d["delta"]):
        u = _offsets_uvw(d, delta, lam)
        s = x.double() * omega
        VD = _forward64(d, case, u, lmn, torch.cat([s[:, None], s[:, None] * lmn], 1))
        w2 = d["wt"].double() ** 2
        r = VD[:, 0] - d["V_obs"].to(torch.complex128)
        g = 2.0 * w2 * r                                        # dL/dRe V + i dL/dIm V
        du = (-2 * math.pi / lam) * (g[:, None] * VD[:, 1:].conj()).imag.reshape(-1, B, 3).sum(0)
        grad = torch.zeros(S, 3, device="cuda", dtype=torch.float64)
        grad.index_add_(0, d["a"], du)
        grad.index_add_(0, d["b"], -du)
        out.append({"loss": (w2 * (r.real ** 2 + r.imag ** 2)).sum(),
                    "sky": omega * _adjoint64(d, case, u, lmn, g, True), "offsets": grad})
    return out
