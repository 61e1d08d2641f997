"""Track blocks (csrc/tracks.cu) against the FP64 kernels of the same plan.

The split path's own error is ~5e-7 (SFU, fixed-point phase, FP32 sums) and the
interpolation keeps its errors, node errors included, below that of an
evaluated term, so 1e-6 bounds both; a (sample, tile) pair counted twice or not
at all would move one value by ~1e-2 of its size, so single values are held to
1e-4 of the rms too.
"""
import numpy as np
import pytest
import torch

from viss_optimize_3d_b200 import api, synth

pytestmark = pytest.mark.gpu
REL, SINGLE = 1e-6, 1e-4


def observation(nside, n_sat, n_snap, f_hz, moon, earth):
    cfg = synth.ObsConfig("t", nside=nside, n_sat=n_sat, n_snap=n_snap, freqs_hz=(f_hz,), moon=moon, earth=earth)
    return synth.make_observation(cfg)


def close(got, want):
    got, want = got.to(torch.complex128), want.to(torch.complex128)
    rms = float(want.abs().square().mean().sqrt())
    err = (got - want).abs()
    assert float(err.square().mean().sqrt()) <= REL * rms, float(err.square().mean().sqrt()) / rms
    assert float(err.max()) <= SINGLE * rms, float(err.max()) / rms


def tables(obs, dev):
    from viss_optimize_3d_b200.pipeline import build_occulters
    refs = None if obs.refs is None else torch.as_tensor(obs.refs, device=dev)
    return refs, build_occulters(obs, dev)


@pytest.mark.parametrize("nside,n_sat,n_snap,f_hz,moon,earth,channels", [
    (64, 8, 7777, 2e6, True, True, 1),      # last blocks shorter than 128, several group sizes
    (101, 7, 4099, 1e6, True, False, 1),    # tiles cut by face boundaries, a part of a last tile
    (64, 6, 5000, 1e6, False, False, 3),    # channels of one plan, nothing occulted
    (60, 10, 2300, 1.5e6, True, True, 3),   # channels and occultation, samples too sparse for blocks
    (60, 10, 2300, 4e5, True, True, 3),     # channels and occultation
])
def test_against_fp64(cuda_device, nside, n_sat, n_snap, f_hz, moon, earth, channels):
    obs = observation(nside, n_sat, n_snap, f_hz, moon, earth)
    lmn = api.pix2lmn(nside, "ring", device=cuda_device)
    refs, occ = tables(obs, cuda_device)
    u = torch.as_tensor(obs.uvw(f_hz), device=cuda_device)
    g = torch.Generator(device=cuda_device).manual_seed(3)
    uvw = torch.cat([u * (1 + 0.1 * c) for c in range(channels)])
    off = torch.rand(len(uvw), generator=g, device=cuda_device, dtype=torch.float64) * 50 - 25
    plan = api.Plan(lmn, uvw, off, None if refs is None else refs.repeat(channels, 1), occ, channels=channels)
    assert plan.K * plan.J >= 1e10
    sky = torch.rand(channels * plan.J, generator=g, device=cuda_device) + 0.1
    coef = torch.randn(plan.K, generator=g, device=cuda_device, dtype=torch.complex64)
    for kw in (dict(), dict(mask=False), dict(use_offset=False)):
        close(plan.forward(sky, **kw), plan.forward(sky, fp64=True, **kw))
        close(plan.adjoint(coef, scale=1.5, **kw), plan.adjoint(coef, scale=1.5, fp64=True, **kw))


def test_nodes_take_most_terms(cuda_device):
    """Dense tracks: far fewer exponentials than terms; a captured call of the
    same plan evaluates every term."""
    obs = observation(64, 8, 7777, 1e6, False, False)
    lmn = api.pix2lmn(64, "ring", device=cuda_device)
    plan = api.Plan(lmn, torch.as_tensor(obs.uvw(1e6), device=cuda_device))
    sky = torch.ones(plan.J, device=cuda_device)
    out = plan.forward(sky)
    evaluated, _, total = plan.last_stats()
    assert total == plan.K * plan.J and evaluated < total // 3
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        plan.forward(sky, out=out)
    graph.replay()
    assert plan.last_stats()[0] == total


@pytest.mark.parametrize("order", ["tracks one after the other", "shuffled", "half rough"])
def test_orders_of_the_samples(cuda_device, order):
    """Tracks one after the other (lag 1) go through the nodes; samples in no
    order stay with the direct kernels; tracks with a rough half mix both."""
    nside, n_sat, n_snap, f_hz = 64, 9, 6000, 1e6
    obs = observation(nside, n_sat, n_snap, f_hz, True, True)
    lmn = api.pix2lmn(nside, "ring", device=cuda_device)
    refs, occ = tables(obs, cuda_device)
    uvw = torch.as_tensor(obs.uvw(f_hz), device=cuda_device)
    g = torch.Generator(device=cuda_device).manual_seed(4)
    if order == "tracks one after the other":
        B = obs.pairs.shape[0]
        idx = torch.arange(len(uvw), device=cuda_device).view(-1, B).T.reshape(-1)
        uvw, refs = uvw[idx].contiguous(), refs[idx].contiguous()
    elif order == "shuffled":
        idx = torch.randperm(len(uvw), generator=g, device=cuda_device)
        uvw, refs = uvw[idx].contiguous(), refs[idx].contiguous()
    else:
        rough = torch.arange(len(uvw), device=cuda_device) % obs.pairs.shape[0] % 2 == 1
        uvw = uvw + rough[:, None] * 20 * torch.randn(uvw.shape, generator=g, device=cuda_device, dtype=torch.float64)
    plan = api.Plan(lmn, uvw, None, refs, occ)
    sky = torch.rand(plan.J, generator=g, device=cuda_device) + 0.1
    coef = torch.randn(plan.K, generator=g, device=cuda_device, dtype=torch.complex64)
    close(plan.forward(sky), plan.forward(sky, fp64=True))
    close(plan.adjoint(coef), plan.adjoint(coef, fp64=True))


def test_restaged_samples_and_captured_calls(cuda_device):
    """New samples in the same plan get new blocks; a captured call, replayed
    after the samples were staged again, computes with the new ones."""
    nside, f_hz = 64, 1e6
    obs = observation(nside, 8, 7600, f_hz, True, False)
    lmn = api.pix2lmn(nside, "ring", device=cuda_device)
    refs, occ = tables(obs, cuda_device)
    uvw = torch.as_tensor(obs.uvw(f_hz), device=cuda_device)
    plan = api.Plan(lmn, uvw, None, refs, occ)
    sky = torch.rand(plan.J, device=cuda_device) + 0.1
    out = torch.empty(plan.K, dtype=torch.complex64, device=cuda_device)
    plan.forward(sky, out=out)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        plan.forward(sky, out=out)
    plan.set_samples(uvw * 1.3, None, refs, occ)
    want = plan.forward(sky, fp64=True)
    close(plan.forward(sky), want)
    graph.replay()
    torch.cuda.synchronize()
    close(out, want)


@pytest.mark.parametrize("n_sat,n_snap,channels,rows", [
    (10, 4801, 1, ("moon", "earth")),
    (3, 24000, 3, ("earth",)),              # one occulter kind only, channels
    (4, 35011, 1, ()),                      # few satellites, nothing occulted
])
def test_formation_pairs(cuda_device, n_sat, n_snap, channels, rows):
    """Formation calls whose pairs lie on dense tracks, against the FP64 direct
    kernels on the pairs' baselines and rows."""
    nside, f_hz = 64, 1e6
    obs = observation(nside, n_sat, n_snap, f_hz, True, True)
    lmn = api.pix2lmn(nside, "ring", device=cuda_device)
    T, S, B = n_snap, n_sat, n_sat * (n_sat - 1) // 2
    P = torch.as_tensor(obs.positions, device=cuda_device)
    U = (P - P.mean(dim=1, keepdim=True)) / (synth.C_LIGHT / f_hz)
    U = torch.stack([U * (1 + 0.2 * c) for c in range(channels)])
    _, occ = tables(obs, cuda_device)
    refs = torch.as_tensor(obs.refs, device=cuda_device).clone()
    if "moon" not in rows:
        refs[:, :2] = -1
    if "earth" not in rows:
        refs[:, 2] = -1
    g = torch.Generator(device=cuda_device).manual_seed(6)
    off = torch.rand(channels * T * B, generator=g, device=cuda_device, dtype=torch.float64)
    a, b = (torch.as_tensor(obs.pairs[:, i].astype(np.int64), device=cuda_device) for i in (0, 1))
    uvw = (U[:, :, a] - U[:, :, b]).reshape(-1, 3)
    plan = api.Plan(lmn, uvw, off, refs.repeat(channels, 1), occ, channels=channels)
    plan.set_formation(U if channels > 1 else U[0], off.view(channels, T, B) if channels > 1 else off.view(T, B),
                       occ[:T * S].view(T, S, 4) if "moon" in rows else None,
                       occ[T * S:] if "earth" in rows else None)
    sky = torch.rand(channels * plan.J, generator=g, device=cuda_device) + 0.1
    coef = torch.randn(plan.K, generator=g, device=cuda_device, dtype=torch.complex64)
    assert plan.K * plan.J >= 1e10
    for kw in (dict(), dict(mask=False), dict(use_offset=False)):
        close(plan.forward_formation(sky, **kw), plan.forward(sky, fp64=True, **kw))
        close(plan.adjoint_formation(coef, **kw), plan.adjoint(coef, fp64=True, **kw))
    acc = plan.forward_formation(sky)
    plan.forward_formation(sky, out=acc, accumulate=True)
    close(acc, 2 * plan.forward(sky, fp64=True))


def test_gridded_call_through_the_blocks(cuda_device):
    """The gridded entry point with its own choice of facets: blocks where they
    are modelled faster, reporting that choice; an explicit facet size grids; a
    NaN coefficient is refused either way."""
    from viss_optimize_3d_b200 import _capi
    obs = observation(64, 8, 7600, 1e6, True, True)
    lmn = api.pix2lmn(64, "ring", device=cuda_device)
    refs, occ = tables(obs, cuda_device)
    plan = api.Plan(lmn, torch.as_tensor(obs.uvw(1e6), device=cuda_device), None, refs, occ)
    g = torch.Generator(device=cuda_device).manual_seed(8)
    coef = torch.randn(plan.K, generator=g, device=cuda_device, dtype=torch.complex64)
    for kw in (dict(), dict(mask=False)):
        want = plan.adjoint(coef, fp64=True, **kw)
        close(plan.adjoint_gridded(coef, **kw), want)
        info = plan.gridded_info()
        assert info["facet_pixels"] >= 64 and min(info["grid"]) >= 16
        got = plan.adjoint_gridded(coef, facet_pixels=256, **kw)
        assert float((got - want).double().norm() / want.double().norm()) < 1e-5
        base = torch.ones(plan.J, device=cuda_device)
        close(plan.adjoint_gridded(coef, out=base, accumulate=True, **kw) - 1, want)
    bad = coef.clone()
    bad[7] = complex(float("nan"), 0.0)
    with pytest.raises(_capi.VissError, match="non-finite"):
        plan.adjoint_gridded(bad, mask=False)
    close(plan.adjoint_gridded(coef, mask=False), plan.adjoint(coef, fp64=True, mask=False))
