"""Launch shapes and chunk sums at the sizes where their rules change, against
the defining sums in 64 bits (plain torch).

A split-precision term is within 4e-7 of its value, and at most 128 terms are
added in plain FP32 (2^-24 of the running sum each, at most 128 of them) before
a Kahan or FP64 sum takes over, so a value is within (4e-7 + 128 * 2^-24) of the
sum of its terms' sizes.  A chunk left out or added twice moves a value by
~1e-3 of it or more at these sizes.
"""
import math

import pytest
import torch

from viss_optimize_3d_b200 import api

pytestmark = pytest.mark.gpu
BOUND = 4e-7 + 128 * 2.0 ** -24


def oracle(lmn, uvw, refs, occ, sky, coef):
    V = torch.zeros(len(uvw), dtype=torch.complex128, device=lmn.device)
    img = torch.zeros(len(lmn), dtype=torch.float64, device=lmn.device)
    for k0 in range(0, len(uvw), 1024):
        u = uvw[k0:k0 + 1024]
        ph = u @ lmn.T
        e = torch.polar(torch.ones_like(ph), -2 * math.pi * (ph - ph.round()))
        if refs is not None:
            for r in refs[k0:k0 + 1024].long().T:
                rows = occ[r.clamp(min=0)]
                e = torch.where((r < 0)[:, None] | (rows[:, :3] @ lmn.T >= rows[:, 3:]), e, 0)
        V[k0:k0 + 1024] = e @ sky.to(torch.complex128)
        img += (coef[k0:k0 + 1024].to(torch.complex128)[:, None] * e.conj()).real.sum(0)
    return V, img


@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("nside,K", [
    (2, 1),         # one tile, one chunk
    (4, 31),        # two tiles; less than a row of the chunk sums
    (8, 33),        # a second block of the sums with one sample
    (24, 450),      # fewer blocks than SMs: the occulted forward keeps its wide blocks
    (37, 3330),     # a last pixel block that is mostly padding
    (12, 9001),     # 71 sample chunks of 14 pixel tiles
    (64, 1000),     # wide blocks padded by a quarter
])
def test_sums(cuda_device, nside, K, masked):
    lmn = api.pix2lmn(nside, "ring", device=cuda_device)
    g = torch.Generator(device=cuda_device).manual_seed(K)
    uvw = 60 * torch.randn(K, 3, generator=g, device=cuda_device, dtype=torch.float64)
    refs = occ = None
    if masked:
        n = torch.nn.functional.normalize(torch.randn(20, 3, generator=g, device=cuda_device, dtype=torch.float64), dim=1)
        occ = torch.cat([n, torch.empty(20, 1, device=cuda_device, dtype=torch.float64).uniform_(-0.9, 0.3, generator=g)], 1)
        refs = torch.randint(-1, 20, (K, 3), generator=g, device=cuda_device, dtype=torch.int32)
    sky = torch.rand(len(lmn), generator=g, device=cuda_device) + 0.1
    coef = torch.randn(K, generator=g, device=cuda_device, dtype=torch.complex64)
    V, img = oracle(lmn, uvw, refs, occ, sky, coef)
    plan = api.Plan(lmn, uvw, None, refs, occ)
    assert float((plan.forward(sky) - V).abs().max()) <= BOUND * float(sky.double().sum())
    assert float((plan.adjoint(coef) - img).abs().max()) <= BOUND * math.sqrt(2) * float(coef.abs().double().sum())


@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("nside,K,n", [
    (2, 2, 3),       # one tile, one block
    (13, 254, 3),    # a block that is not full, a part of a last tile
    (24, 4098, 3),   # 17 blocks of samples, several chunks
    (24, 450, 2),    # not three: one sky after the other
    (16, 33, 1),     # one sky, odd count
])
def test_skies(cuda_device, nside, K, n, masked):
    lmn = api.pix2lmn(nside, "ring", device=cuda_device)
    g = torch.Generator(device=cuda_device).manual_seed(K)
    uvw = 60 * torch.randn(K, 3, generator=g, device=cuda_device, dtype=torch.float64)
    refs = occ = None
    if masked:
        v = torch.nn.functional.normalize(torch.randn(20, 3, generator=g, device=cuda_device, dtype=torch.float64), dim=1)
        occ = torch.cat([v, torch.empty(20, 1, device=cuda_device, dtype=torch.float64).uniform_(-0.9, 0.3, generator=g)], 1)
        refs = torch.randint(-1, 20, (K, 3), generator=g, device=cuda_device, dtype=torch.int32)
    sky = torch.randn(n, len(lmn), generator=g, device=cuda_device)
    plan = api.Plan(lmn, uvw, None, refs, occ)
    for fp64 in (False, True):
        V = plan._forward_skies(sky, fp64=fp64)
        assert V.shape == (n, K) and plan.last_stats()[2] == n * K * len(lmn)
        for c in range(n):
            want, _ = oracle(lmn, uvw, refs, occ, sky[c], torch.zeros(K, dtype=torch.complex64, device=cuda_device))
            assert float((V[c] - want).abs().max()) <= BOUND * float(sky[c].abs().double().sum())


def test_skies_refuse_odd_counts(cuda_device):
    """As three channels of repeated samples do."""
    lmn = api.pix2lmn(4, "ring", device=cuda_device)
    plan = api.Plan(lmn, torch.ones(3, 3, dtype=torch.float64, device=cuda_device))
    with pytest.raises(RuntimeError, match="must be even"):
        plan._forward_skies(torch.ones(3, len(lmn), device=cuda_device))


@pytest.mark.parametrize("masked,accumulate", [(False, False), (True, False), (False, True)])
def test_gridded_goes_direct_where_that_is_faster(cuda_device, masked, accumulate):
    """Few samples: the library's choice is the direct sum (the same bits), its
    facets are reported, a facet size that is asked for is gridded, and gridding's
    refusal of non-finite coefficients stays."""
    nside, K = 32, 3001
    lmn = api.pix2lmn(nside, "ring", device=cuda_device)
    g = torch.Generator(device=cuda_device).manual_seed(1)
    uvw = 20 * torch.randn(K, 3, generator=g, device=cuda_device, dtype=torch.float64)
    refs = occ = None
    if masked:
        occ = torch.tensor([[0.0, 0.0, 1.0, -0.5]], device=cuda_device, dtype=torch.float64)
        refs = torch.tensor([[0, -1, -1]], device=cuda_device, dtype=torch.int32).repeat(K, 1)
    coef = torch.randn(K, generator=g, device=cuda_device, dtype=torch.complex64)
    plan = api.Plan(lmn, uvw, None, refs, occ)
    direct = plan.adjoint(coef, scale=0.5)
    if accumulate:
        got = plan.adjoint_gridded(coef, scale=0.5, out=direct.clone(), accumulate=True)
        assert bool(((got - 2 * direct).abs() <= 2.0 ** -22 * direct.abs()).all())   # the two roundings
    else:
        assert torch.equal(plan.adjoint_gridded(coef, scale=0.5), direct)
    facet = plan.gridded_info()["facet_pixels"]
    assert facet >= 64
    gridded = plan.adjoint_gridded(coef, scale=0.5, facet_pixels=facet)
    assert plan.gridded_info()["facet_pixels"] == facet
    assert not torch.equal(gridded, direct) and float((gridded - direct).norm()) <= 5e-6 * float(direct.norm())
    coef[7] = float("nan")
    with pytest.raises(RuntimeError):
        plan.adjoint_gridded(coef)


@pytest.mark.parametrize("nside,K", [(64, 20001), (48, 30000)])
def test_captured_calls_outlive_other_calls(cuda_device, nside, K):
    """A captured unocculted call keeps its workspace when occulted calls, which
    take other launch shapes, follow on the same samples."""
    lmn = api.pix2lmn(nside, "ring", device=cuda_device)
    g = torch.Generator(device=cuda_device).manual_seed(7)
    uvw = 40 * torch.randn(K, 3, generator=g, device=cuda_device, dtype=torch.float64)
    occ = torch.tensor([[0.0, 0.6, 0.8, -0.3]], device=cuda_device, dtype=torch.float64)
    refs = torch.tensor([[0, -1, -1]], device=cuda_device, dtype=torch.int32).repeat(K, 1)
    sky = torch.rand(len(lmn), generator=g, device=cuda_device) + 0.1
    coef = torch.randn(K, generator=g, device=cuda_device, dtype=torch.complex64)
    plan = api.Plan(lmn, uvw, None, refs, occ)
    V, img = torch.empty(K, dtype=torch.complex64, device=cuda_device), torch.empty(len(lmn), device=cuda_device)
    for call, out in ((lambda **kw: plan.forward(sky, **kw), V), (lambda **kw: plan.adjoint(coef, **kw), img)):
        want = call(mask=False)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            call(mask=False, out=out)
        masked = call()
        others = [torch.full((1 << 18,), 7.0, device=cuda_device) for _ in range(8)]   # over what was freed
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want) and not torch.equal(masked, want)
        assert all(bool((o == 7.0).all()) for o in others)
