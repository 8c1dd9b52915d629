"""Multigrid-preconditioned solves on damaged tangents (loading and unloading points, stiffness that varies by orders of
magnitude, distorted cells), and both Krylov methods in turn on one matrix."""

import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu

STRAIN = 2.5e-4


def _bend(mesh):
    extent = mesh.coords.max(axis=0)

    def f(x):
        bump = np.prod(np.sin(np.pi * x / extent), axis=1)
        return x + bump[:, None] * np.array([0.08, -0.06, 0.05])[: x.shape[1]] * extent

    mesh.transform(f)


def _field(s, n, rng):
    """a stretched body with perturbations of a fifth of a cell's stretch (n cells per unit length), eeq U(0, 4e-4)"""
    x = np.zeros(s.n_dofs)
    L = s.mesh.layers[s.layers[0]]
    xyz = L.node_coords[:, : s.mesh.dim]
    f = -0.2 * STRAIN * (xyz - 0.5)
    f[:, -1] = STRAIN * xyz[:, -1]
    f += rng.uniform(-0.2, 0.2, f.shape) * STRAIN / n
    x[L.dof_numbers.reshape(-1)] = f.reshape(-1)
    x[L.num_dofs:] = rng.uniform(0.0, 4e-4, s.n_dofs - L.num_dofs)
    return x


def _fixed(s):
    return np.concatenate([np.asarray(d, dtype=np.int64) + (s.mesh.layers[s.layers[0]].num_dofs if k else 0)
                           for k, (d, _, _) in enumerate(s.constraints)])


def _cuda():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    return torch


@pytest.mark.parametrize("kind,n", [("hex8", 9), ("hex8", 14), ("plates", 3)])
@pytest.mark.parametrize("precision", [64, 32])
def test_damaged_tangent(kind, n, precision):
    """The right-hand side is K x for a smooth x, so the rounding of its residual is far below 1e-12 of its norm: the solve's
    stopping test at 1e-12 holds for the residual formed here, twice over for its own rounding. Iterations hardly depend on the
    size; the interpolation this cycle has takes below 100 at 20^3 and 24^3, one with piecewise constant transfer took 300."""
    _cuda()
    from nuto_gb300 import batch, configs

    rng = np.random.default_rng(31)
    if kind == "plates":
        s, n = batch.notched_plate_batch(n, seed=5)[0], 100  # 20 to 120 cells a side
    else:
        s = configs.hex8_gradient_damage(n)
        _bend(s.mesh)
    g = s.build_gpu()
    g.history = rng.uniform(0.0, 4e-4, (s.mesh.num_cells, s.gauss ** s.mesh.dim))
    vals = g.build_matrix(_field(s, n, rng), precision)
    rp, ci = g.pattern()
    K = sp.csr_matrix((vals.double().cpu().numpy(), ci, rp), shape=(s.n_dofs, s.n_dofs))
    y = _field(s, n, rng)
    dep = _fixed(s)
    y[dep] = 0.0
    b = K @ y
    b[dep] = 0.0
    x, it, rel, ok = g.solve(vals, b, precision=precision, rtol=1e-12, max_iterations=2000)
    assert ok, (it, rel)
    x = x.cpu().numpy()
    assert not x[dep].any()
    r = b - K @ x
    r[dep] = 0.0
    assert np.linalg.norm(r) <= 2e-12 * np.linalg.norm(b)
    assert it <= 150, it


@pytest.mark.parametrize("precision", [64, 32])
def test_methods_in_turn_on_one_matrix(precision):
    """PCG runs the symmetric cycle, GMRES the cheaper one; each solve after a change of method rebuilds what differs and gives
    the same solution in the iterations it took before (coarse operators are summed by atomics: 2 more or less)."""
    import scipy.sparse.linalg as spla

    torch = _cuda()
    from nuto_gb300 import configs

    s = configs.quad4_elastic(48)
    _bend(s.mesh)
    g = s.build_gpu()
    vals = g.build_matrix(torch.zeros(s.n_dofs, dtype=torch.float64, device="cuda"), precision)
    rp, ci = g.pattern()
    K = sp.csr_matrix((vals.double().cpu().numpy(), ci, rp), shape=(s.n_dofs, s.n_dofs))
    free = np.setdiff1d(np.arange(s.n_dofs), _fixed(s))
    b = np.zeros(s.n_dofs)
    b[free] = np.random.default_rng(37).uniform(-1, 1, len(free))
    y = spla.spsolve(K[free][:, free].tocsc(), b[free])
    its = {}
    for method in (1, 3, 1, 3, 3, 1):  # PCG, GMRES
        x, it, rel, ok = g.solve(vals, b, precision=precision, method=method, rtol=1e-11, max_iterations=500)
        assert ok, (method, it, rel)
        assert np.abs(x.cpu().numpy()[free] - y).max() <= 1e-6 * np.abs(y).max()
        assert abs(it - its.setdefault(method, it)) <= 2, (method, it, its)
