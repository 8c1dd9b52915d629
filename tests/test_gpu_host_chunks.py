"""build_system_host in its chunked form (values of 16 MB and more): cells and rows of a node chunk, then its copy, on meshes
whose cells follow the node order and on a mesh whose cells come in random order (a chunk's rows may need the last cell)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,shuffled", [(19, False), (21, False), (21, True), (30, True)])
def test_chunked_host_system(n, shuffled):
    """Values and residual equal the device call's: the same kernels on the same data (the residual adds in another order)."""
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    import nuto_gb300
    from nuto_gb300 import mesh as M
    from nuto_gb300.assembly import GpuCellGroup

    m = M.create_bricks(n, n, n + 1)
    rng = np.random.default_rng(n)
    if shuffled:
        m.conn[:] = m.conn[rng.permutation(len(m.conn))]
    layers = [M.add_dof_interpolation(m, 3), M.add_dof_interpolation(m, 1)]
    g = GpuCellGroup(m, layers, 2)
    g.build_pattern()
    g.set_integrand(kind=2, dim=3, disp_slot=0, eeq_slot=1, E=30000.0, nu=0.2, plane_state=1, damage_application=0,
                    kappa0=1e-4, beta=100.0, alpha=0.99, k=10.0, c=0.01)
    nd = m.layers[layers[0]].num_dofs
    u = rng.uniform(-2e-4, 2e-4, g.n_dofs)
    u[nd:] = rng.uniform(0.0, 4e-4, g.n_dofs - nd)
    g.history = rng.uniform(0.0, 4e-4, (m.num_cells, 8))
    ut = torch.from_numpy(u)
    vh = torch.empty(g.nnz, dtype=torch.float32).pin_memory()
    fh = torch.empty(g.n_dofs, dtype=torch.float64).pin_memory()
    v, f = g.build_system(ut.cuda(), nuto_gb300.FP32)
    for _ in range(3):  # the first call is not chunked
        vh.fill_(float("nan"))
        fh.fill_(float("nan"))
        g.build_system_host(ut.pin_memory(), vh, fh, nuto_gb300.FP32)
        assert torch.equal(vh, v.cpu())
        fr = f.cpu()
        assert (fh - fr).abs().max() <= 1e-12 * fr.abs().max()
