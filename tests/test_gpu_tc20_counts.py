"""k_tangent_tc20 with one to 22 cells per block: its two accumulators and their barriers are handed between two groups of
warps, so what can go wrong depends on how many cells a block walks (152 blocks on a GB300)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells", [(1, 1, 1), (8, 19, 1), (9, 17, 1), (16, 19, 1), (5, 61, 1), (457, 1, 1), (13, 19, 13)])
@pytest.mark.parametrize("kind", [0, 1])
def test_cells_per_block(cells, kind):
    """FP32 against the FP64 tangent at 2e-6 of the largest entry, twice with the same bits."""
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    import nuto_gb300
    from nuto_gb300 import mesh as M
    from nuto_gb300.assembly import GpuCellGroup

    m = M.create_bricks(*cells)
    m.transform(lambda x: x * np.array(cells))
    g = GpuCellGroup(m, [M.add_dof_interpolation(m, 3, M.HEX20)], 3)
    g.build_pattern()
    g.set_integrand(kind=kind, dim=3, disp_slot=0, E=30000.0, nu=0.2, kappa0=1e-4, beta=100.0, alpha=0.99, k=10.0)
    rng = np.random.default_rng(7)
    u = rng.uniform(-3e-4, 3e-4, g.n_dofs)
    if kind:
        g.history = rng.uniform(0.0, 3e-4, (m.num_cells, 27))
    a = g.build_matrix(u, nuto_gb300.FP32)
    d = g.build_matrix(u, nuto_gb300.FP64)
    assert float((a.double() - d).abs().max()) <= 2e-6 * float(d.abs().max())
    assert torch.equal(a, g.build_matrix(u, nuto_gb300.FP32))
