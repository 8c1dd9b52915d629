"""Tangents captured in a CUDA graph: replays write the values of a direct call, whatever the context assembled since the
capture."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case(kind, n):
    """(setup, state, history): every branch of the damage law"""
    from nuto_gb300 import configs

    s = {"quad4": configs.quad4_elastic, "hex8": configs.hex8_gradient_damage, "hex20": configs.hex20_local_damage,
         "plate": lambda m: configs.notched_plate(m, 0.4)}[kind](n)
    rng = np.random.default_rng(7)
    u = rng.uniform(-2e-4, 2e-4, s.n_dofs)
    if len(s.layers) == 2:
        nd = s.mesh.layers[s.layers[0]].num_dofs
        u[nd:] = rng.uniform(0.0, 4e-4, s.n_dofs - nd)
    kappa = None if kind == "quad4" else rng.uniform(0.0, 4e-4, (s.mesh.num_cells, s.gauss ** s.mesh.dim))
    return s, u, kappa


def _group(s, kappa, stream):
    import torch

    with torch.cuda.stream(stream):
        g = s.build_gpu()
    if kappa is not None:
        g.history = kappa
    g.synchronize()
    return g


def _capture(g, stream, u, precision, out):
    import torch

    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        g.build_matrix(u, precision, out=out)
    return graph


def _cuda():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    return torch


@pytest.mark.parametrize("kind,n", [("quad4", 9), ("plate", 12), ("hex8", 7), ("hex20", 3)])
@pytest.mark.parametrize("precision", [32, 64])
def test_replay_after_the_first_tangent_of_the_other_arithmetic(kind, n, precision):
    """The element matrices of both arithmetics have their own memory: a captured tangent, replayed after the context's first
    tangent of the other one, gives the direct call's values bit for bit and writes nothing that others hold by then."""
    torch = _cuda()
    s, u0, kappa = _case(kind, n)
    stream = torch.cuda.Stream()
    g = _group(s, kappa, stream)
    u = torch.as_tensor(u0, device="cuda")
    out = g.build_matrix(u, precision)
    graph = _capture(g, stream, u, precision, out)
    other = g.build_matrix(u, 96 - precision)
    # what the allocator hands out now must not be the captured call's scratch
    held = [torch.full((1 << 20,), float("nan"), device="cuda") for _ in range(64)]
    u.mul_(-0.75)
    torch.cuda.synchronize()
    graph.replay()
    torch.cuda.synchronize()
    assert all(bool(torch.isnan(h).all()) for h in held)
    direct = g.build_matrix(u, precision)
    torch.cuda.synchronize()
    if precision == 32:
        assert torch.equal(out, direct)
    else:
        assert (out - direct).abs().max() <= 1e-12 * direct.abs().max()
    assert torch.isfinite(other).all()


@pytest.mark.parametrize("kind,n", [("quad4", 9), ("plate", 12), ("hex8", 7), ("hex20", 3)])
def test_captured_fp64_tangent_is_the_direct_call(kind, n):
    """After one FP64 tangent everything a capture needs is there: the captured call runs the direct call's kernels and its
    replays give the same bits."""
    torch = _cuda()
    s, u0, kappa = _case(kind, n)
    stream = torch.cuda.Stream()
    g = _group(s, kappa, stream)
    u = torch.as_tensor(u0, device="cuda")
    out = g.build_matrix(u, 64)
    graph = _capture(g, stream, u, 64, out)
    u.mul_(-0.75)
    for _ in range(2):
        out.zero_()
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        direct = g.build_matrix(u, 64)
        torch.cuda.synchronize()
        assert torch.equal(out, direct)


@pytest.mark.parametrize("kind,n", [("quad4", 9), ("plate", 12), ("hex8", 7), ("hex20", 3)])
@pytest.mark.parametrize("before", ["residual", "fp32"])
def test_first_fp64_tangent_inside_a_capture(kind, n, before):
    """Without an FP64 tangent before it the captured call allocates nothing and gives the tangent to rounding."""
    torch = _cuda()
    s, u0, kappa = _case(kind, n)
    stream = torch.cuda.Stream()
    g = _group(s, kappa, stream)
    u = torch.as_tensor(u0, device="cuda")
    g.build_vector(u) if before == "residual" else g.build_matrix(u, 32)
    out = torch.empty(g.nnz, dtype=torch.float64, device="cuda")
    graph = _capture(g, stream, u, 64, out)
    graph.replay()
    torch.cuda.synchronize()
    direct = g.build_matrix(u, 64)
    torch.cuda.synchronize()
    assert (out - direct).abs().max() <= 1e-12 * direct.abs().max()


@pytest.mark.parametrize("kind,n", [("quad4", 9), ("hex20", 3)])
def test_first_fp32_element_kernel_inside_a_capture(kind, n, monkeypatch):
    """The FP32 element kernel needs the geometry of the residual and no memory of its own: what it is first called in may be a
    capture. Each value sums at most 8 cells' blocks by atomics, in any order: 2e-6 of the largest."""
    torch = _cuda()
    monkeypatch.setenv("NUTO_GPU_TANGENT", "atomic")
    s, u0, kappa = _case(kind, n)
    stream = torch.cuda.Stream()
    g = _group(s, kappa, stream)
    u = torch.as_tensor(u0, device="cuda")
    g.build_vector(u)
    out = torch.empty(g.nnz, dtype=torch.float32, device="cuda")
    graph = _capture(g, stream, u, 32, out)
    graph.replay()
    torch.cuda.synchronize()
    direct = g.build_matrix(u, 32)
    torch.cuda.synchronize()
    assert (out - direct).abs().max() <= 2e-6 * direct.abs().max()
