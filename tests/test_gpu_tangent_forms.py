"""Forms of the tangent that share no kernel agree: element matrices, point records with the row gather, element atomics."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _values(s, u, kappa, precision, form, monkeypatch):
    monkeypatch.setenv("NUTO_GPU_TANGENT", form)
    g = s.build_gpu()
    if kappa is not None:
        g.history = kappa
    return g.build_matrix(u, precision).double().cpu().numpy()


@pytest.mark.parametrize("kind,n", [("quad4", 11), ("plate", 14), ("hex8", 6), ("hex20", 3)])
def test_forms_agree(kind, n, monkeypatch):
    """FP32: element matrices (Hex20: tensor cores) and records to 2e-6 of the largest entry, the sum of the bounds that each is
    held to against the oracle (1e-6); FP64: element matrices and element atomics to 1e-12. The forms are different kernels: not
    one of the pairs is equal bit for bit."""
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    from nuto_gb300 import configs

    s = {"quad4": configs.quad4_elastic, "hex8": configs.hex8_gradient_damage, "hex20": configs.hex20_local_damage,
         "plate": lambda m: configs.notched_plate(m, 0.4)}[kind](n)
    rng = np.random.default_rng(29)
    u = rng.uniform(-2e-4, 2e-4, s.n_dofs)
    if len(s.layers) == 2:
        nd = s.mesh.layers[s.layers[0]].num_dofs
        u[nd:] = rng.uniform(0.0, 4e-4, s.n_dofs - nd)
    kappa = None if kind == "quad4" else rng.uniform(0.0, 4e-4, (s.mesh.num_cells, s.gauss ** s.mesh.dim))
    for precision, forms, bound in ((32, ("", "records"), 2e-6), (64, ("", "atomic"), 1e-12)):
        a, b = [_values(s, u, kappa, precision, f, monkeypatch) for f in forms]
        assert np.abs(a - b).max() <= bound * np.abs(a).max(), precision
        assert not np.array_equal(a, b), precision
