"""Quad4 / Hex8 cells with the two-point rule against the oracle on distorted, non-cubic meshes: every integrand kind and
law option, cell counts below one warp's or block's, with remainders, and on both sides of the switch of the residual's cells
per warp. Residual: k_residual_sf (sum-factorised gradients, a warp per 8 or 4 Hex8 cells and per 16 or 8 Quad4 cells); FP64
tangent: k_cell_matrices64 + k_rows_from_slabs (elastic and gradient damage with FULL damage), else the element kernel."""

import numpy as np
import pytest

from oracle import core as ocore

pytestmark = pytest.mark.gpu

FP64_REL = 1e-12

LAWS = {
    "elastic": dict(kind=0),
    "elastic_plane_stress": dict(kind=0, plane_state=0),
    "local": dict(kind=1),
    "local_unilateral": dict(kind=1, damage_application=1),
    "gradient": dict(kind=2),
    "gradient_plane_stress": dict(kind=2, plane_state=0),
    "gradient_unilateral_decreasing": dict(kind=2, damage_application=1, interaction=1, R=0.05, eta=3.0),
}


def _case(dim, cells, law, seed):
    """(group, oracle problem, state, kappa) on a lattice of `cells` cells bent so that no two cells are alike"""
    from nuto_gb300 import mesh as M
    from nuto_gb300.assembly import GpuCellGroup

    m = M.create_quads(*cells) if dim == 2 else M.create_bricks(*cells)
    bend = np.array([0.07, -0.05, 0.04])[:dim]
    m.transform(lambda x: x + np.sin(2.1 * x[:, ::-1] + 0.3) * bend)
    om = ocore.Mesh.from_arrays(dim, ocore.QUAD4 if dim == 2 else ocore.HEX8, m.coords, m.conn)
    params = dict(E=30000.0, nu=0.2, plane_state=1, damage_application=0, kappa0=1e-4, beta=100.0, alpha=0.99, k=10.0,
                  c=0.01)
    params.update({k: v for k, v in law.items() if k != "kind"})
    layers = [M.add_dof_interpolation(m, dim)] + ([M.add_dof_interpolation(m, 1)] if law["kind"] == 2 else [])
    olayers = [om.add_dof(dim)] + ([om.add_dof(1)] if law["kind"] == 2 else [])
    P = ocore.Problem(om, 2, olayers, ocore.Integrand.make(law["kind"], dim, **params))
    g = GpuCellGroup(m, layers, 2)
    g.build_pattern()
    g.set_integrand(kind=law["kind"], dim=dim, disp_slot=0, eeq_slot=1 if law["kind"] == 2 else -1, **params)
    rng = np.random.default_rng(seed)
    u = rng.uniform(-2e-4, 2e-4, P.n_dofs)
    if law["kind"] == 2:
        nd = m.layers[layers[0]].num_dofs
        u[nd:] = rng.uniform(0.0, 4e-4, P.n_dofs - nd)
    kappa = rng.uniform(0.0, 4e-4, (P.n_el, P.n_ip))
    if law["kind"] != 0:
        P.kappa = kappa
        g.history = kappa
    return g, P, u


CASES = [(2, (1, 1), "elastic"), (2, (3, 5), "elastic_plane_stress"), (2, (7, 9), "gradient"),
         (2, (5, 3), "gradient_plane_stress"), (2, (6, 7), "local"), (2, (4, 5), "gradient_unilateral_decreasing"),
         (2, (97, 53), "gradient"),  # above 16 cells per warp, remainder 5
         (3, (1, 1, 1), "gradient"), (3, (1, 2, 3), "local"), (3, (3, 3, 2), "local_unilateral"),
         (3, (3, 2, 5), "elastic"), (3, (5, 3, 1), "gradient_unilateral_decreasing"),
         (3, (13, 14, 15), "gradient")]  # above 8 cells per warp, remainder 2


@pytest.mark.parametrize("dim,cells,law", CASES)
def test_residual_on_distorted_cells(dim, cells, law):
    g, P, u = _case(dim, cells, LAWS[law], 7)
    f_ref = P.build_vector(u)
    f = g.build_vector(u).cpu().numpy()
    assert np.abs(f - f_ref).max() <= FP64_REL * np.abs(f_ref).max()


@pytest.mark.parametrize("dim,cells,law", CASES)
def test_fp64_tangent_on_distorted_cells(dim, cells, law):
    import nuto_gb300

    g, P, u = _case(dim, cells, LAWS[law], 8)
    K = P.build_matrix_scipy(u).tocsr()
    K.sort_indices()
    for precision in (nuto_gb300.FP64, nuto_gb300.FP64X):
        v = g.build_matrix(u, precision).cpu().numpy()
        assert np.abs(v - K.data).max() <= FP64_REL * np.abs(K.data).max()
    if law in ("elastic", "elastic_plane_stress", "gradient", "gradient_plane_stress"):  # no atomics
        assert np.array_equal(v, g.build_matrix(u, nuto_gb300.FP64).cpu().numpy())


@pytest.mark.parametrize("form", ["cells", "pipelined"])
@pytest.mark.parametrize("dim,cells,law", [c for c in CASES if "unilateral" not in c[2] and c[2] != "local"])
def test_fp32_tangent_on_distorted_cells(dim, cells, law, form, monkeypatch):
    """The FP32 element-matrix form, one pass per warp and on resident blocks: the FP32 tangent's tolerance against the
    oracle, 2e-6 of the largest entry."""
    import nuto_gb300

    monkeypatch.setenv("NUTO_GPU_TANGENT", form)
    g, P, u = _case(dim, cells, LAWS[law], 9)
    K = P.build_matrix_scipy(u).tocsr()
    K.sort_indices()
    v = g.build_matrix(u, nuto_gb300.FP32).double().cpu().numpy()
    assert np.abs(v - K.data).max() <= 2e-6 * np.abs(K.data).max()


@pytest.mark.parametrize("dim,cells,law", CASES)
def test_point_values_on_distorted_cells(dim, cells, law):
    """Strain and stress (k_eval_sf) and the scalar quantities at every integration point."""
    g, P, u = _case(dim, cells, LAWS[law], 10)
    for quantity in range(5):
        ref = P.eval_ip(u, quantity)
        v = g.eval_ip(u, quantity).cpu().numpy().reshape(ref.shape)
        assert np.abs(v - ref).max() <= FP64_REL * np.abs(ref).max() + 1e-300, quantity
