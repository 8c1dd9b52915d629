"""FP64 tangent of Hex20 cells (k_cell_matrices64_h20 + k_rows_from_wide_slabs) against the oracle at 1e-12 of the largest
entry: one cell and a few, distorted, elastic and local damage with all, some and no points loading; bitwise reproducible."""

import numpy as np
import pytest

from oracle import core as ocore

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells", [(1, 1, 1), (2, 1, 3)])
@pytest.mark.parametrize("state", ["elastic", "loading", "mixed", "unloading"])
def test_fp64_hex20_tangent(cells, state):
    import nuto_gb300
    from nuto_gb300 import mesh as M
    from nuto_gb300.assembly import GpuCellGroup

    kind = 0 if state == "elastic" else 1
    m = M.create_bricks(*cells)
    m.transform(lambda x: x + np.sin(2.1 * x[:, ::-1] + 0.3) * np.array([0.07, -0.05, 0.04]))
    om = ocore.Mesh.from_arrays(3, ocore.HEX8, m.coords, m.conn)
    params = dict(E=30000.0, nu=0.2, kappa0=1e-4, beta=100.0, alpha=0.99, k=10.0)
    layer, olayer = M.add_dof_interpolation(m, 3, M.HEX20), om.add_dof(3, ocore.HEX20)
    P = ocore.Problem(om, 3, [olayer], ocore.Integrand.make(kind, 3, damage_application=ocore.FULL, **params))
    g = GpuCellGroup(m, [layer], 3)
    g.build_pattern()
    g.set_integrand(kind=kind, dim=3, disp_slot=0, **params)
    rng = np.random.default_rng(5)
    u = rng.uniform(-3e-4, 3e-4, P.n_dofs)
    top = {"elastic": 0.0, "loading": 0.0, "mixed": 3e-3, "unloading": 1.0}[state]
    kappa = rng.uniform(0.5 * top if state == "unloading" else 0.0, top, (P.n_el, P.n_ip))
    if kind:
        P.kappa = kappa
        g.history = kappa
    K = P.build_matrix_scipy(u).tocsr()
    K.sort_indices()
    v = g.build_matrix(u, nuto_gb300.FP64).cpu().numpy()
    assert np.abs(v - K.data).max() <= 1e-12 * np.abs(K.data).max()
    assert np.array_equal(v, g.build_matrix(u, nuto_gb300.FP64).cpu().numpy())
