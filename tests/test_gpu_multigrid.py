"""Multigrid-preconditioned solves on meshes whose levels have ragged edges: odd sizes, distorted cells, notches, several bodies
and quadratic cells (corner level first), against a direct solve of the same matrix."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


def _bend(mesh):
    extent = mesh.coords.max(axis=0)

    def f(x):
        bump = np.prod(np.sin(np.pi * x / extent), axis=1)
        return x + bump[:, None] * np.array([0.08, -0.06, 0.05])[: x.shape[1]] * extent

    mesh.transform(f)


# enough nodes for one level only, for two and for several; nodes per side odd and even
@pytest.mark.parametrize("kind,n,bent", [("hex8", 4, False), ("hex8", 9, True), ("hex8", 12, True), ("quad4", 11, True),
                                         ("quad4", 64, False), ("plate", 30, False), ("plates", 2, False),
                                         ("hex20", 3, True), ("hex20", 6, False)])
@pytest.mark.parametrize("precision", [64, 32])
def test_multigrid_solve(kind, n, bent, precision):
    """The matrices are well enough conditioned (below 1e6) that a relative residual of 1e-12 leaves 1e-6 of the largest
    value. The cycle's iteration count hardly depends on the size: at most 120."""
    import scipy.sparse.linalg as spla
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    from nuto_gb300 import batch, configs

    rng = np.random.default_rng(17)
    if kind == "plates":
        s = batch.notched_plate_batch(n, seed=3)[0]
    else:
        s = {"hex8": configs.hex8_gradient_damage, "quad4": configs.quad4_elastic, "hex20": configs.hex20_local_damage,
             "plate": lambda m: configs.notched_plate(m, 0.4)}[kind](n)
    if bent:
        _bend(s.mesh)
    g = s.build_gpu()
    dep = np.concatenate([np.asarray(d, dtype=np.int64) + (s.mesh.layers[s.layers[0]].num_dofs if k else 0)
                          for k, (d, _, _) in enumerate(s.constraints)])
    free = np.setdiff1d(np.arange(s.n_dofs), dep)
    u = torch.zeros(s.n_dofs, dtype=torch.float64, device="cuda")
    vals = g.build_matrix(u, precision)
    rp, ci = g.pattern()
    K = sp.csr_matrix((vals.double().cpu().numpy(), ci, rp), shape=(s.n_dofs, s.n_dofs))
    b = np.zeros(s.n_dofs)
    b[free] = rng.uniform(-1, 1, len(free))
    g.set_preconditioner(2)
    x, it, rel, ok = g.solve(vals, b, precision=precision, method=0, rtol=1e-12, max_iterations=2000)
    assert ok, (it, rel)
    y = spla.spsolve(K[free][:, free].tocsc(), b[free])
    assert np.abs(x.cpu().numpy()[free] - y).max() <= 1e-6 * np.abs(y).max()
    assert it <= 120, it
