"""Track blocks (csrc/tracks*.cu) on the inputs at the edge of their rules.
Tolerances as in test_gpu_tracks.py; every case says which path evaluated it.
"""
import pytest
import torch

from viss_optimize_3d_b200 import _capi, api, synth

from test_gpu_tracks import REL, close, observation, tables

pytestmark = pytest.mark.gpu


def inputs(plan, dev, seed=3):
    g = torch.Generator(device=dev).manual_seed(seed)
    return (torch.rand(plan.J, generator=g, device=dev) + 0.1,
            torch.randn(plan.K, generator=g, device=dev, dtype=torch.complex64))


def by_blocks(plan):
    """The last call evaluated far fewer exponentials than terms."""
    evaluated, _, total = plan.last_stats()
    return evaluated < total // 2


def two_patches(n, dev):
    """n directions in two caps of 8 degrees, far apart."""
    g = torch.Generator(device=dev).manual_seed(11)
    c = torch.tensor([[0.36, 0.48, 0.8], [-0.8, 0.6, 0.0]], device=dev, dtype=torch.float64)
    d = c[torch.arange(n, device=dev) % 2] + 0.08 * (2 * torch.rand(n, 3, generator=g, device=dev, dtype=torch.float64) - 1)
    return torch.nn.functional.normalize(d, dim=1)


@pytest.mark.parametrize("pixels,n_sat,n_snap,f_hz,moon", [
    (57, 10, 6000, 2e4, False),     # a tile across two base faces, wider than every group of 1,024
    (57, 10, 6000, 2e4, True),      # the same of a plan with occulters, unmasked
    (55, 10, 6200, 2e4, False),
    ("patches", 10, 6000, 2e4, False),
])
def test_tiles_wider_than_their_group(cuda_device, pixels, n_sat, n_snap, f_hz, moon):
    """Unocculted calls of slow tracks: no tile is left out."""
    obs = observation(64 if pixels == "patches" else pixels, n_sat, n_snap, f_hz, moon, False)
    lmn = two_patches(40000, cuda_device) if pixels == "patches" else api.pix2lmn(pixels, "ring", device=cuda_device)
    refs, occ = tables(obs, cuda_device)
    plan = api.Plan(lmn, torch.as_tensor(obs.uvw(f_hz), device=cuda_device), None, refs, occ)
    assert plan.K * plan.J >= 1e10
    sky, coef = inputs(plan, cuda_device)
    V, img = plan.forward(sky, fp64=True, mask=False), plan.adjoint(coef, fp64=True, mask=False)
    close(plan.forward(sky, mask=False), V)
    assert by_blocks(plan)
    close(plan.adjoint(coef, mask=False), img)
    assert by_blocks(plan)
    P = torch.as_tensor(obs.positions, device=cuda_device)
    plan.set_formation((P - P.mean(dim=1, keepdim=True)) / (synth.C_LIGHT / f_hz))
    close(plan.forward_formation(sky), V)
    assert by_blocks(plan)
    close(plan.adjoint_formation(coef), img)


def test_pixel_that_is_no_direction(cuda_device):
    """A NaN pixel stays in its own terms: every other image pixel is what it
    was, through blocks and without them."""
    obs = observation(57, 10, 6000, 2e4, False, False)
    lmn = api.pix2lmn(57, "ring", device=cuda_device).clone()
    bad = 12345
    lmn[bad] = float("nan")
    plan = api.Plan(lmn, torch.as_tensor(obs.uvw(2e4), device=cuda_device))
    _, coef = inputs(plan, cuda_device)
    keep = torch.arange(plan.J, device=cuda_device) != bad
    want = plan.adjoint(coef, fp64=True)
    got = plan.adjoint(coef)
    assert by_blocks(plan)
    assert bool(torch.isfinite(want[keep]).all())
    close(got[keep], want[keep])


def test_pixels_beyond_the_unit_sphere(cuda_device):
    """Vectors that are no directions (a few of length 4) and baselines near the
    blocks' bound: their phases do not fit the blocks' fixed point."""
    n = 44000
    g = torch.Generator(device=cuda_device).manual_seed(2)
    lmn = torch.nn.functional.normalize(torch.randn(n, 3, generator=g, device=cuda_device, dtype=torch.float64), dim=1)
    lmn[::1000] *= 4.0
    # one baseline that stays where it is: a single node serves a block, whatever the group's width
    uvw = torch.tensor([[1.5e5, -5e4, 4e4]], device=cuda_device, dtype=torch.float64).repeat(240000, 1)
    plan = api.Plan(lmn, uvw)
    sky, coef = inputs(plan, cuda_device)
    # 44 terms of a wrong phase move a value by a few percent, and their pixels by all of it
    for got, want in ((plan.forward(sky), plan.forward(sky, fp64=True)), (plan.adjoint(coef), plan.adjoint(coef, fp64=True))):
        assert float((got - want).abs().max()) <= 1e-4 * float(want.abs().square().mean().sqrt())


def test_skies_through_the_blocks(cuda_device):
    """Three skies a block at a time, and the same call captured afterwards
    (which evaluates every term, in buffers that are there already)."""
    obs = observation(57, 10, 6000, 2e4, False, False)
    plan = api.Plan(api.pix2lmn(57, "ring", device=cuda_device), torch.as_tensor(obs.uvw(2e4), device=cuda_device))
    g = torch.Generator(device=cuda_device).manual_seed(5)
    sky = torch.randn(3, plan.J, generator=g, device=cuda_device) + 0.5
    want = plan._forward_skies(sky, fp64=True)
    got = plan._forward_skies(sky)
    evaluated, _, total = plan.last_stats()
    assert total == 3 * plan.K * plan.J and evaluated < total // 2
    for c in range(3):
        close(got[c], want[c])
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = plan._forward_skies(sky)
    graph.replay()
    assert plan.last_stats()[0] >= total            # and the padding of the last tiles
    for c in range(3):
        close(out[c], want[c])


@pytest.mark.parametrize("tile", [1, 10 ** 6, 1 << 30])
@pytest.mark.parametrize("call", ["forward", "adjoint"])
@pytest.mark.parametrize("f_hz", [2e4, 2e6])      # groups of 1,024 pixels; of 64 among others
def test_wait_that_gives_up(cuda_device, call, tile, f_hz):
    """A staging copy that never comes (a tile past the last one stands for the
    last) or a product whose end is never signalled (2^30): the call ends, the
    next status read reports it, the plan goes on."""
    obs = observation(57, 10, 6000, f_hz, False, False)
    plan = api.Plan(api.pix2lmn(57, "ring", device=cuda_device), torch.as_tensor(obs.uvw(f_hz), device=cuda_device))
    sky, coef = inputs(plan, cuda_device)
    run = (lambda **kw: plan.forward(sky, **kw)) if call == "forward" else (lambda **kw: plan.adjoint(coef, **kw))
    run()
    assert by_blocks(plan)
    _capi.check(_capi.lib.viss_plan_debug_drop_copy(plan._h, tile), "viss_plan_debug_drop_copy")
    run()
    with pytest.raises(_capi.VissError, match="gave up"):
        plan.last_stats()
    close(run(), run(fp64=True))


@pytest.mark.parametrize("seed", [1, 5, 12])
@pytest.mark.parametrize("f_hz,n_sat", [(1e6, 8), (3e6, 10)])
def test_no_further_off_than_evaluated_terms(cuda_device, seed, f_hz, n_sat):
    """A term that the direct kernels evaluate is off by up to 3.7e-7 (a phase of
    23 bits); V, an image of random coefficients and one of V itself (whose terms
    share their errors) stay below that through blocks."""
    obs = observation(128, n_sat, 8640, f_hz, False, False)
    plan = api.Plan(api.pix2lmn(128, "ring", device=cuda_device), torch.as_tensor(obs.uvw(f_hz), device=cuda_device))
    g = torch.Generator(device=cuda_device).manual_seed(seed)
    sky = torch.exp(torch.randn(plan.J, generator=g, device=cuda_device))
    coef = torch.randn(plan.K, generator=g, device=cuda_device, dtype=torch.complex64)
    rel = lambda a, b: float((a.to(torch.complex128) - b.to(torch.complex128)).norm() / b.to(torch.complex128).norm())
    V = plan.forward(sky, fp64=True)
    assert rel(plan.forward(sky), V) <= 3.7e-7
    assert by_blocks(plan)
    for c in (coef, V):
        img = plan.adjoint(c)
        assert by_blocks(plan)
        assert rel(img, plan.adjoint(c, fp64=True)) <= 3.7e-7


@pytest.mark.parametrize("f_hz,n_sat", [(1e6, 8), (3e6, 10)])
def test_scale_of_the_image(cuda_device, f_hz, n_sat):
    """What the SFU and the tensor cores' truncating accumulators leave out is put
    back by rank and direction: 2e-8 is twice the scatter of the measured shortfalls
    about that rule.  The image of random coefficients has no other coherent part."""
    obs = observation(128, n_sat, 8640, f_hz, False, False)
    plan = api.Plan(api.pix2lmn(128, "ring", device=cuda_device), torch.as_tensor(obs.uvw(f_hz), device=cuda_device))
    _, coef = inputs(plan, cuda_device)
    got = plan.adjoint(coef)
    assert by_blocks(plan)
    want = plan.adjoint(coef, fp64=True).double()
    assert abs(float(((got - want) * want).sum() / want.square().sum())) <= 2e-8


@pytest.mark.parametrize("nside,n_sat,n_snap,f_hz,blocks", [
    (256, 10, 600, 3e6, False),      # few snapshots: a limb crosses many tiles within a block
    (256, 10, 600, 1e6, False),
    (128, 10, 4600, 3e6, True),
])
def test_occulted_calls_take_the_faster_way(cuda_device, nside, n_sat, n_snap, f_hz, blocks):
    """Sparse snapshots make the remainder of the blocks dear (measured: the first
    two forwards 16.5 and 10.6 ms through blocks, 10.1 term by term; the third 9.9
    against 19.5)."""
    obs = observation(nside, n_sat, n_snap, f_hz, True, True)
    refs, occ = tables(obs, cuda_device)
    plan = api.Plan(api.pix2lmn(nside, "ring", device=cuda_device), torch.as_tensor(obs.uvw(f_hz), device=cuda_device),
                    None, refs, occ)
    sky, _ = inputs(plan, cuda_device)
    got = plan.forward(sky)
    assert by_blocks(plan) == blocks
    close(got, plan.forward(sky, fp64=True))


@pytest.mark.parametrize("nside,n_sat,n_snap,f_hz,moon,earth,channels", [
    (64, 8, 7777, 2e6, True, True, 1),
    (101, 7, 4099, 1e6, True, False, 1),
    (64, 6, 5000, 1e6, False, False, 3),
    (60, 10, 2300, 4e5, True, True, 3),
])
def test_compared_calls_do_go_through_blocks(cuda_device, nside, n_sat, n_snap, f_hz, moon, earth, channels):
    """The observations that test_gpu_tracks.py compares with FP64, and their
    satellite vectors."""
    obs = observation(nside, n_sat, n_snap, f_hz, moon, earth)
    refs, occ = tables(obs, cuda_device)
    u = torch.as_tensor(obs.uvw(f_hz), device=cuda_device)
    plan = api.Plan(api.pix2lmn(nside, "ring", device=cuda_device),
                    torch.cat([u * (1 + 0.1 * c) for c in range(channels)]), None,
                    None if refs is None else refs.repeat(channels, 1), occ, channels=channels)
    sky = torch.ones(channels * plan.J, device=cuda_device)
    coef = torch.ones(plan.K, dtype=torch.complex64, device=cuda_device)
    for kw in (dict(), dict(mask=False)):
        plan.forward(sky, **kw)
        assert by_blocks(plan)
        plan.adjoint(coef, **kw)
        assert by_blocks(plan)
        plan.forward(sky, all_terms=True, **kw)
        assert not by_blocks(plan)


@pytest.mark.parametrize("bright", [1, 30])
def test_sky_of_a_few_bright_pixels(cuda_device, bright):
    """Weights fitted to directions spread over a group hold for single ones."""
    obs = observation(64, 8, 7777, 1e6, False, False)
    plan = api.Plan(api.pix2lmn(64, "ring", device=cuda_device), torch.as_tensor(obs.uvw(1e6), device=cuda_device))
    g = torch.Generator(device=cuda_device).manual_seed(bright)
    for _ in range(4):
        sky = torch.zeros(plan.J, device=cuda_device)
        sky[torch.randint(plan.J, (bright,), generator=g, device=cuda_device)] = 2.0
        got = plan.forward(sky)
        assert by_blocks(plan)
        close(got, plan.forward(sky, fp64=True))


def test_values_that_are_not_finite(cuda_device):
    """An infinite sky value or coefficient reaches what sees it and nothing else,
    as term by term."""
    obs = observation(64, 8, 7777, 1e6, True, False)
    refs, occ = tables(obs, cuda_device)
    plan = api.Plan(api.pix2lmn(64, "ring", device=cuda_device), torch.as_tensor(obs.uvw(1e6), device=cuda_device),
                    None, refs, occ)
    for bad in (float("inf"), float("nan")):
        sky, coef = inputs(plan, cuda_device)
        sky[31000], coef[4000] = bad, bad
        V, img = plan.forward(sky), plan.adjoint(coef)
        assert by_blocks(plan)
        for got, want in ((V, plan.forward(sky, all_terms=True)), (img, plan.adjoint(coef, all_terms=True))):
            ok = torch.isfinite(want.abs())
            assert 0 < int(ok.sum()) < len(ok) and torch.equal(torch.isfinite(got.abs()), ok)
            close(got[ok], want[ok])


def test_pixels_that_are_no_grid(cuda_device):
    """Directions drawn at random, and the call's pixel groups with them."""
    g = torch.Generator(device=cuda_device).manual_seed(9)
    lmn = torch.nn.functional.normalize(torch.randn(50001, 3, generator=g, device=cuda_device, dtype=torch.float64), dim=1)
    obs = observation(64, 8, 7777, 3e5, True, True)
    refs, occ = tables(obs, cuda_device)
    plan = api.Plan(lmn, torch.as_tensor(obs.uvw(3e5), device=cuda_device), None, refs, occ)
    sky, coef = inputs(plan, cuda_device)
    for kw in (dict(), dict(mask=False)):
        got = plan.forward(sky, **kw)
        assert by_blocks(plan)
        close(got, plan.forward(sky, fp64=True, **kw))
        got = plan.adjoint(coef, **kw)
        assert by_blocks(plan)
        close(got, plan.adjoint(coef, fp64=True, **kw))


@pytest.mark.parametrize("size", [1e-40, 1e-37, 1e35])
def test_sizes_near_the_ends_of_fp32(cuda_device, size):
    """The smallest and largest skies and coefficients are as accurate as term by
    term (1e-40 has 17 bits itself: the same inputs on both sides)."""
    obs = observation(64, 8, 7777, 1e6, True, False)
    refs, occ = tables(obs, cuda_device)
    plan = api.Plan(api.pix2lmn(64, "ring", device=cuda_device), torch.as_tensor(obs.uvw(1e6), device=cuda_device),
                    None, refs, occ)
    sky, coef = inputs(plan, cuda_device)
    rel = lambda a, b: float((a.to(torch.complex128) - b.to(torch.complex128)).norm() / b.to(torch.complex128).norm())
    for call, x in ((plan.forward, sky * size), (plan.adjoint, coef * size)):
        want = call(x, fp64=True)
        err = rel(call(x), want)
        assert by_blocks(plan)
        assert err <= max(1.1 * rel(call(x, all_terms=True), want), REL)


@pytest.mark.parametrize("nside,n_snap,f_hz", [
    (41, 11200, 1e5), (73, 3600, 1e5), (87, 2500, 1e5), (97, 2020, 3e4), (121, 1300, 3e4),
])
def test_no_tile_is_left_out_of_uneven_grids(cuda_device, nside, n_snap, f_hz):
    """Grids whose widest tile, across two base faces, is wider than the widest group
    of 256 or 1,024 pixels, nothing occulted and every radius taken whole."""
    obs = observation(nside, 10, n_snap, f_hz, False, False)
    plan = api.Plan(api.pix2lmn(nside, "ring", device=cuda_device), torch.as_tensor(obs.uvw(f_hz), device=cuda_device))
    assert plan.K * plan.J >= 1e10
    sky, coef = inputs(plan, cuda_device)
    got = plan.forward(sky)
    assert by_blocks(plan)
    close(got, plan.forward(sky, fp64=True))
    got = plan.adjoint(coef)
    assert by_blocks(plan)
    close(got, plan.adjoint(coef, fp64=True))
