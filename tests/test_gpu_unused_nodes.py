"""DOF nodes that no cell uses: their rows are empty, everything else is as without them."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _with_unused_nodes(layer, at):
    """the layer with nodes of no cell inserted at the positions `at` (of the extended numbering)"""
    from nuto_gb300.mesh import DofLayer

    n = layer.num_nodes + len(at)
    kept = np.setdiff1d(np.arange(n), at)
    coords = np.zeros((n, 3))
    coords[kept] = layer.node_coords
    coords[at] = 17.0
    return DofLayer(layer.ncomp, layer.interp, kept[layer.conn], coords), kept


def _group(dim, gd, extra):
    """(group, DOF numbers of the cells' nodes in the combined vector); extra: positions of unused nodes per layer"""
    from nuto_gb300 import mesh as M
    from nuto_gb300.assembly import GpuCellGroup

    m = M.create_quads(5, 4) if dim == 2 else M.create_bricks(3, 4, 2)
    layers = [M.add_dof_interpolation(m, dim)] + ([M.add_dof_interpolation(m, 1)] if gd else [])
    dofs, offset = [], 0
    for k in layers:
        layer, kept = _with_unused_nodes(m.layers[k], np.asarray(extra[k], dtype=np.int64))
        m.layers[k] = layer
        dofs.append(offset + layer.dof_numbers[kept].reshape(-1))
        offset += layer.num_dofs
    g = GpuCellGroup(m, layers, 2)
    g.build_pattern()
    g.set_integrand(kind=2 if gd else 0, dim=dim, disp_slot=0, eeq_slot=1 if gd else -1, E=30000.0, nu=0.2, kappa0=1e-4,
                    beta=100.0, alpha=0.99, k=10.0, c=0.01)
    return g, np.concatenate(dofs)


@pytest.mark.parametrize("dim,gd", [(2, True), (3, True), (2, False), (3, False)])
# positions of the unused nodes (displacements, eeq) on a mesh of n nodes
@pytest.mark.parametrize("extra", [lambda n: ([3], [3]), lambda n: ([0, n + 1], [4, n + 1]), lambda n: ([], [])],
                         ids=["inside", "ends", "none"])
def test_nodes_of_no_cell(dim, gd, extra):
    """Empty rows hold no values, so the tangents' values are those of the mesh without the extra nodes bit for bit, in every
    form; the residual is zero in those rows."""
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    plain, dofs0 = _group(dim, gd, ([], []))
    g, dofs = _group(dim, gd, extra(plain.mesh.coords.shape[0]))
    rng = np.random.default_rng(23)
    u0 = rng.uniform(-2e-4, 2e-4, plain.n_dofs)
    if gd:
        u0[len(dofs0) * dim // (dim + 1):] = rng.uniform(0.0, 4e-4, len(dofs0) // (dim + 1))
        kappa = rng.uniform(0.0, 4e-4, (plain.mesh.num_cells, plain.n_ip))
        plain.history = kappa
        g.history = kappa
    u = np.zeros(g.n_dofs)
    u[dofs] = u0
    assert g.nnz == plain.nnz
    for precision in (64, 32):
        assert torch.equal(g.build_matrix(u, precision), plain.build_matrix(u0, precision))
    assert torch.equal(g.build_matrix_noalloc(u), plain.build_matrix_noalloc(u0))
    f = g.build_vector(u).cpu().numpy()
    assert np.array_equal(f[dofs], plain.build_vector(u0).cpu().numpy())
    assert not np.delete(f, dofs).any()
