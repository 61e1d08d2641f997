"""VISS_ALL_TERMS: calls of 1e10 terms and more evaluated term by term, as
captured calls run them, at full size.  The split path's error is ~5e-7 (see
test_gpu_tracks.py)."""
import pytest
import torch

from viss_optimize_3d_b200 import api, pipeline, synth

from test_gpu_tracks import close

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def c3(cuda_device):
    """Nside 256, 45 baselines x 8,640 snapshots, 10 MHz, Moon + Earth."""
    obs = synth.make_observation(synth.CONFIGS["c3_10mhz"])
    return obs, pipeline.upload(obs, 1e7, device=cuda_device)


def test_visible_counts_are_exact(c3, cuda_device):
    """Zero baselines, unit sky and coefficients: V counts a sample's visible
    pixels and the image a pixel's samples, exactly, in both ways (the blocks'
    counts are pinned to the plain predicate in test_gpu_fullsize.py)."""
    _, g = c3
    plan = api.Plan(g.lmn, torch.zeros_like(g.uvw), None, g.refs, g.occ)
    sky = torch.ones(plan.J, device=cuda_device)
    coef = torch.ones(plan.K, dtype=torch.complex64, device=cuda_device)
    V = plan.forward(sky, all_terms=True)
    evaluated, _, total = plan.last_stats()
    assert evaluated > total // 2
    assert torch.equal(V.real.round(), plan.forward(sky).real.round())
    assert plan.last_stats()[0] < total // 8
    img = plan.adjoint(coef, all_terms=True)
    assert plan.last_stats()[0] > total // 2
    assert torch.equal(img.round(), plan.adjoint(coef).round())


def test_values_and_bits_of_captured_calls(c3, cuda_device):
    obs, g = c3
    plan = api.Plan(g.lmn, g.uvw, None, g.refs, g.occ)
    gen = torch.Generator(device=cuda_device).manual_seed(3)
    sky = torch.rand(plan.J, generator=gen, device=cuda_device) + 0.1
    coef = torch.randn(plan.K, generator=gen, device=cuda_device, dtype=torch.complex64)
    P = torch.as_tensor(obs.positions, device=cuda_device)
    U = (P - P.mean(dim=1, keepdim=True)) / (synth.C_LIGHT / 1e7)
    T, S = U.shape[:2]
    plan.set_formation(U, None, g.occ[:T * S].view(T, S, 4), g.occ[T * S:])
    V64, img64 = plan.forward(sky, fp64=True), plan.adjoint(coef, fp64=True)
    for call, want in ((lambda **kw: plan.forward(sky, **kw), V64), (lambda **kw: plan.adjoint(coef, **kw), img64),
                       (lambda **kw: plan.forward_formation(sky, **kw), V64),
                       (lambda **kw: plan.adjoint_formation(coef, **kw), img64)):
        got = call(all_terms=True)
        close(got, want)
        torch.cuda.synchronize()
        out = torch.empty_like(got)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            call(out=out)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, got)
