"""Tangents and solves where device memory is short: the element matrices are scratch that the other forms do without."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture
def leave_free():
    """leave_free(bytes) holds all device memory but that much, leave_free(None) gives it back"""
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    held = []

    def hold(keep):
        torch.cuda.synchronize()
        held.clear()
        torch.cuda.empty_cache()
        if keep is not None:
            held.append(torch.empty(torch.cuda.mem_get_info()[0] - keep, dtype=torch.uint8, device="cuda"))
            assert torch.cuda.mem_get_info()[0] <= keep

    yield hold
    hold(None)


def _group():
    """A 40^3 gradient-damage beam with its geometry laid out: 524 MB of FP64 element matrices, 262 MB in FP32"""
    import torch
    from nuto_gb300 import configs

    s = configs.hex8_gradient_damage(40)
    rng = np.random.default_rng(3)
    x = rng.uniform(-1e-6, 1e-6, s.n_dofs)
    nd = s.mesh.layers[s.layers[0]].num_dofs
    x[nd:] = rng.uniform(0.0, 4e-4, s.n_dofs - nd)
    g = s.build_gpu()
    g.history = rng.uniform(0.0, 4e-4, (s.mesh.num_cells, 8))
    u = torch.as_tensor(x, device="cuda")
    g.build_vector(u)
    return g, u, torch.as_tensor(rng.uniform(-1.0, 1.0, s.n_dofs), device="cuda")


def test_fp64_tangent_leaves_the_solve_its_memory(leave_free):
    """In 1000 MB the element matrices and what the solve takes (590 MB of basis vectors and padded values alone) do not fit
    together: the tangent comes from the element kernel, which needs no scratch, and the solve runs."""
    import torch

    g, u, b = _group()
    values = torch.empty(g.nnz, dtype=torch.float64, device="cuda")
    leave_free(1000 << 20)
    g.build_matrix(u, 64, out=values)
    x, it, rel, ok = g.solve(values, b, precision=64, rtol=1e-6, max_iterations=1000)
    assert ok, (it, rel)
    leave_free(None)
    ref = values.clone()
    assert (g.build_matrix(u, 64, out=values) - ref).abs().max() <= 1e-12 * ref.abs().max()
    g.build_pattern()  # asks again
    assert (g.build_matrix(u, 64, out=values) - ref).abs().max() <= 1e-12 * ref.abs().max()


def test_exact_phase_tangent_beside_the_fp32_solver(leave_free):
    """The tangent of the exact final phase (precision 65) is multiplied with, not solved: in the same 1000 MB the element
    matrices and the padded values fit, and the values are those of a context with all the memory bit for bit."""
    import torch

    full, u, _ = _group()
    ref = full.build_matrix(u, 65).cpu()
    del full
    g, _, _ = _group()
    values = torch.empty(g.nnz, dtype=torch.float64, device="cuda")
    x = torch.ones(g.n_dofs, dtype=torch.float64, device="cuda")
    leave_free(1000 << 20)
    g.build_matrix(u, 65, out=values)
    g.spmv(values, x)
    torch.cuda.synchronize()
    leave_free(None)
    assert torch.equal(values.cpu(), ref)


def test_fp32_tangent_without_room_for_element_matrices(leave_free):
    """In 200 MB the FP32 tangent comes from the point records (1e-6 of the largest entry from the element matrices, the bound
    of the no-alloc call, which has the same kernels); a new pattern asks for the memory again."""
    import torch

    full, u, _ = _group()
    ref = full.build_matrix(u, 32)
    g, _, _ = _group()
    values = torch.empty(g.nnz, dtype=torch.float32, device="cuda")
    leave_free(200 << 20)
    g.build_matrix(u, 32, out=values)
    leave_free(None)
    assert (values - ref).abs().max() <= 1e-6 * ref.abs().max()
    g.build_pattern()
    assert torch.equal(g.build_matrix(u, 32, out=values), ref)
