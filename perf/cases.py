"""The work that a user of this package has it do, as cases that can be timed and compared.

A case is one call (or one pair of calls that belong together) of `nuto_gb300.GpuCellGroup`, at a seeded state of one of
the set-ups in `nuto_gb300.configs` / `nuto_gb300.batch`:

  vector   BuildVector: the FP64 residual, what every line-search trial of a Newton step evaluates
  matrix   BuildMatrix: the tangent's CSR values in FP32, FP64 or FP64X
  system   both at one state, what a Newton iteration asks for
  host     the same with page-locked host buffers (a host code that keeps its state and its matrix in host memory)
  solve    the linear solve of a Newton step or of the adjoint's reverse sweep on an assembled tangent
  post     the end of a load step: history update, then stress and kappa at every integration point for output

`prepare` builds the group (what a program keeps: mesh, pattern, workspaces), sets history and state from the seed and
allocates the output buffers that a Newton loop reuses. `exact` integrates the same cells in 64 bits with plain torch,
from the arrays of the set-up (coordinates, connectivity, DOF numbers) alone.
"""

import functools
import math

import numpy as np
import torch

from nuto_gb300 import FP32, FP64, _lib, batch, configs
from nuto_gb300.mesh import HEX20_EDGES

FP64X = _lib.FP64X
PRECISION = {"f32": FP32, "f64": FP64, "f64x": FP64X}
STRAIN = 2.5e-4  # mean strain of the states: some points below the damage threshold 1e-4 / 1e-4 .. 4e-4, most above


# ---- cases ----------------------------------------------------------------------------------------------------------
def listed():
    return [
        # the smallest call: one residual of a 20 x 20 plate, as in a parameter study of small meshes; latency and
        # launches count, not throughput
        {"name": "vector_quad4_20", "op": "vector", "mesh": "quad4", "n": 20, "precision": "f64", "curved": False},
        # the 2D elastic verification problem at its full size on the FP64 path: matrix and vector of 80,802 DOFs
        {"name": "system_quad4_200_f64", "op": "system", "mesh": "quad4", "n": 200, "precision": "f64",
         "curved": True},
        # a batch of notched plates of uneven size assembled as one system (10 plates, 20 to 120 cells a side)
        {"name": "system_plates_10_f32", "op": "system", "mesh": "plates", "n": 10, "precision": "f32",
         "curved": False},
        # a small 3D gradient-damage beam, odd size: an ordinary Newton iteration of a study on a coarse mesh
        {"name": "system_hex8_17_f32", "op": "system", "mesh": "hex8", "n": 17, "precision": "f32", "curved": True},
        # the headline assembly pass: the 64^3 beam, 1.1 M DOFs, 115 M nonzeros
        {"name": "system_hex8_64_f32", "op": "system", "mesh": "hex8", "n": 64, "precision": "f32", "curved": False},
        # the same pass for a host code: state in, CSR values and residual back through host memory
        {"name": "host_hex8_40_f32", "op": "host", "mesh": "hex8", "n": 40, "precision": "f32", "curved": False},
        # FP64 tangent of the FP64 path and of the adjoint's reverse sweep, distorted cells
        {"name": "matrix_hex8_40_f64", "op": "matrix", "mesh": "hex8", "n": 40, "precision": "f64", "curved": True},
        # quadratic cells with local damage: the FP32 tangent of the mixed path
        {"name": "matrix_hex20_24_f32", "op": "matrix", "mesh": "hex20", "n": 24, "precision": "f32",
         "curved": False},
        # quadratic cells with local damage: the FP64 tangent of the FP64 path, odd size, distorted cells
        {"name": "matrix_hex20_13_f64", "op": "matrix", "mesh": "hex20", "n": 13, "precision": "f64",
         "curved": True},
        # the linear solve of a mixed-precision Newton step: FP32 tangent and Krylov vectors, refined in FP64 (to the
        # tolerance of the adjoint's solves, which leaves an x that two runs agree on)
        {"name": "solve_hex8_24_f32", "op": "solve", "mesh": "hex8", "n": 24, "precision": "f32", "curved": True},
        # the linear solve of the FP64 path and of the adjoint's reverse sweep
        {"name": "solve_hex8_20_f64", "op": "solve", "mesh": "hex8", "n": 20, "precision": "f64", "curved": True},
        # what ends a load step: history update, stress and kappa at every integration point
        {"name": "post_hex8_48", "op": "post", "mesh": "hex8", "n": 48, "precision": "f64", "curved": False},
    ]


# (op, mesh, precisions, smallest and largest n)
RANGES = [
    ("vector", "quad4", ("f64",), 12, 200),
    ("vector", "hex8", ("f64",), 9, 60),
    ("system", "quad4", ("f32", "f64"), 24, 200),
    ("system", "plates", ("f32",), 3, 10),
    ("system", "hex8", ("f32",), 9, 60),
    ("host", "hex8", ("f32",), 9, 40),
    ("matrix", "hex8", ("f32", "f64", "f64x"), 9, 40),
    ("matrix", "hex20", ("f32",), 4, 24),
    ("matrix", "hex20", ("f64",), 4, 13),
    ("solve", "hex8", ("f32",), 8, 24),
    ("solve", "hex8", ("f64",), 8, 20),
    ("post", "hex8", ("f64",), 9, 48),
]


def draw(rng):
    op, mesh, precisions, lo, hi = rng.choice(RANGES)
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return {"op": op, "mesh": mesh, "n": n, "precision": rng.choice(precisions),
            "curved": mesh != "plates" and rng.random() < 0.5}


# ---- set-ups and seeded states --------------------------------------------------------------------------------------
@functools.lru_cache(maxsize=6)
def _setup(mesh, n, curved):
    """The set-up (mesh, numbering, constraints) of a case: host arrays that do not depend on the seed."""
    if mesh == "quad4":
        s = configs.quad4_elastic(n)
    elif mesh == "plates":
        s = batch.notched_plate_batch(n, seed=n)[0]
    elif mesh == "hex8":
        s = configs.hex8_gradient_damage(n)
    else:
        s = configs.hex20_local_damage(n)
    if curved:  # a smooth interior distortion: no two cells alike, the boundary stays where it is
        extent = s.mesh.coords.max(axis=0)

        def bend(x):
            bump = np.prod(np.sin(np.pi * x / extent), axis=1)
            return x + bump[:, None] * np.array([0.08, -0.06, 0.05])[: x.shape[1]] * extent

        s.mesh.transform(bend)
    return s


def _state(s, case, seed):
    """(state vector, kappa): a stretched body with cell-sized perturbations, nodal eeq and history U(0, 4e-4), so that
    loading and unloading, damaged and undamaged points are mixed (an elastic case has no eeq and no history)."""
    rng = np.random.default_rng([seed, case["n"]])
    x = np.zeros(s.n_dofs)
    L = s.mesh.layers[s.layers[0]]
    xyz = L.node_coords[:, : s.mesh.dim]
    axis = s.mesh.dim - 1
    h = 1.0 / (case["n"] if case["mesh"] != "plates" else 100)
    field = -0.2 * STRAIN * (xyz - 0.5)
    field[:, axis] = STRAIN * xyz[:, axis]
    field += rng.uniform(-0.2, 0.2, field.shape) * STRAIN * h
    x[L.dof_numbers.reshape(-1)] = field.reshape(-1)
    n_ip = s.gauss ** s.mesh.dim
    kappa = None
    if case["mesh"] != "quad4":
        kappa = rng.uniform(0.0, 4e-4, (s.mesh.num_cells, n_ip))
    if len(s.layers) == 2:
        x[L.num_dofs:] = rng.uniform(0.0, 4e-4, s.n_dofs - L.num_dofs)
    return x, kappa


def _correction(s, case, seed):
    """A displacement-like vector (smooth field, noise, eeq part), zero at the constrained DOFs: the solution of the
    solve cases."""
    x, _ = _state(s, case, seed + 1)
    for k, (dofs, _, _) in enumerate(s.constraints):
        x[np.asarray(dofs, dtype=np.int64) + (s.mesh.layers[s.layers[0]].num_dofs if k else 0)] = 0.0
    return x


def prepare(case, seed):
    s = _setup(case["mesh"], case["n"], case["curved"])
    x, kappa = _state(s, case, seed)
    g = s.build_gpu()
    if kappa is not None:
        g.history = kappa
    prec = PRECISION[case["precision"]]
    st = {"g": g, "op": case["op"], "precision": prec}
    value_type = torch.float32 if prec == FP32 else torch.float64
    st["u"] = torch.from_numpy(x).cuda()
    if case["op"] in ("matrix", "system"):
        st["values"] = torch.empty(g.nnz, dtype=value_type, device="cuda")
    if case["op"] in ("vector", "system"):
        st["f"] = torch.empty(g.n_dofs, dtype=torch.float64, device="cuda")
    if case["op"] == "host":
        st["u"] = torch.from_numpy(x).pin_memory()
        st["values"] = torch.empty(g.nnz, dtype=value_type).pin_memory()
        st["f"] = torch.empty(g.n_dofs, dtype=torch.float64).pin_memory()
    if case["op"] == "solve":
        st["values"] = g.build_matrix(st["u"], prec)
        rp, ci = g.pattern()
        K = torch.sparse_csr_tensor(torch.from_numpy(rp).cuda(), torch.from_numpy(ci.astype(np.int64)).cuda(),
                                    st["values"].double(), size=(g.n_dofs, g.n_dofs))
        st["b"] = K @ torch.from_numpy(_correction(s, case, seed)).cuda()
    return st


def run(st):
    g, op, prec = st["g"], st["op"], st["precision"]
    if op == "vector":
        return {"f": g.build_vector(st["u"], out=st["f"])}
    if op == "matrix":
        return {"values": g.build_matrix(st["u"], prec, out=st["values"])}
    if op == "system":
        v, f = g.build_system(st["u"], prec, out=st["values"], f_out=st["f"])
        return {"values": v, "f": f}
    if op == "host":
        v, f = g.build_system_host(st["u"], st["values"], st["f"], prec)
        return {"values": v, "f": f}
    if op == "solve":
        x, _, _, ok = g.solve(st["values"], st["b"], precision=prec, rtol=1e-13, max_iterations=4000)
        if not ok:
            raise RuntimeError("the solve did not converge")
        return {"x": x}
    g.update_history(st["u"])
    return {"stress": g.eval_ip(st["u"], _lib.IP_STRESS), "kappa": g.eval_ip(st["u"], _lib.IP_KAPPA)}


# ---- the work that a pass cannot do without ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=16)
def _node_pairs(mesh, n):
    """Ordered pairs of nodes that share a cell (themselves included)."""
    if mesh in ("quad4", "hex8"):  # a lattice: three neighbours per direction, two at its ends
        return (3 * n + 1) ** (2 if mesh == "quad4" else 3)
    conn = _setup(mesh, n, False).mesh.layers[0].conn.astype(np.int64)
    m = int(conn.max()) + 1
    keys = np.concatenate([conn[:, i] * m + conn[:, j] for i in range(conn.shape[1]) for j in range(conn.shape[1])])
    return int(np.unique(keys).size)


def work(case):
    s = _setup(case["mesh"], case["n"], case["curved"])
    comps = sum(s.mesh.layers[l].ncomp for l in s.layers)
    cells, nen, dim = s.mesh.num_cells, s.mesh.layers[s.layers[0]].conn.shape[1], s.mesh.dim
    ips = cells * s.gauss ** dim
    conn = sum(4 * s.mesh.layers[l].conn.size for l in s.layers) + 4 * s.mesh.conn.size
    inputs = conn + 8 * s.mesh.coords.size + 8 * s.n_dofs + (8 * ips if case["mesh"] != "quad4" else 0)
    vd = 3 if dim == 2 else 6
    # residual: H and the B^T sigma sums (and the eeq part) at every point; tangent: one symmetric displacement block per
    # unordered node pair and the coupling blocks
    vec_flops = ips * nen * 2.0 * (2 * dim * dim + (2 * dim + 2 if comps > dim else 0))
    mat_flops = ips * (nen * (nen + 1) * 2.0 * dim * dim + nen * nen * 2.0 * (2 * dim + 2 if comps > dim else 0))
    if case["op"] == "vector":
        return {"bytes": inputs + 8 * s.n_dofs, "flops": vec_flops}
    if case["op"] == "post":
        return {"bytes": inputs + 8 * ips * (1 + vd + 1), "flops": ips * nen * 2.0 * (dim * dim + 1)}
    values = _node_pairs(case["mesh"], case["n"]) * comps ** 2 * (4 if case["precision"] == "f32" else 8)
    if case["op"] == "solve":  # one product with the matrix, whatever the method
        return {"bytes": values + 16 * s.n_dofs, "flops": 2.0 * values / (4 if case["precision"] == "f32" else 8)}
    if case["op"] == "matrix":
        return {"bytes": inputs + values, "flops": mat_flops}
    return {"bytes": inputs + values + 8 * s.n_dofs, "flops": mat_flops + vec_flops}


# ---- the same integrals in 64 bits, plain torch ---------------------------------------------------------------------
_CORNER2 = np.array([[-1, -1], [1, -1], [1, 1], [-1, 1]])
_CORNER3 = np.array([[-1, -1, -1], [1, -1, -1], [1, 1, -1], [-1, 1, -1], [-1, -1, 1], [1, -1, 1], [1, 1, 1],
                     [-1, 1, 1]])


def _shape(nen, p):
    """Shape values [q, n] and natural derivatives [q, n, d] at the points p [q, d]."""
    c = _CORNER2 if p.shape[1] == 2 else _CORNER3
    dim = p.shape[1]
    if nen != 20:
        t = 1.0 + c[None] * p[:, None, :]
        N = np.prod(t, axis=2) / 2 ** dim
        dN = np.stack([c[None, :, d] * np.prod(np.delete(t, d, axis=2), axis=2) / 2 ** dim for d in range(dim)], axis=2)
        return N, dN
    c = np.concatenate([c, (c[HEX20_EDGES[:, 0]] + c[HEX20_EDGES[:, 1]]) // 2])
    N, dN = np.zeros((len(p), 20)), np.zeros((len(p), 20, 3))
    for i in range(20):
        f, df = [], []  # one factor per direction and its derivative
        for d in range(3):
            x = p[:, d]
            f.append(1 - x * x if c[i, d] == 0 else 1 + c[i, d] * x)
            df.append(-2 * x if c[i, d] == 0 else np.full_like(x, c[i, d]))
        scale = 0.125 if i < 8 else 0.25
        prod = f[0] * f[1] * f[2]
        lin = p @ c[i] - 2.0 if i < 8 else np.ones(len(p))
        N[:, i] = scale * prod * lin
        for d in range(3):
            other = f[(d + 1) % 3] * f[(d + 2) % 3]
            dN[:, i, d] = scale * (df[d] * other * lin + (prod * c[i, d] if i < 8 else 0.0))
    return N, dN


def _law(eps, integ, kh, eeq):
    """Stress, isotropic tangent factor, the vectors of the rank-1 parts, the local equivalent strain and kappa at every
    point, Voigt order xx, yy(, zz, yz, zx), xy, plane strain in 2D."""
    E, nu = integ["E"], integ["nu"]
    dim = 2 if eps.shape[-1] == 3 else 3
    normal = torch.zeros(eps.shape[-1], dtype=eps.dtype, device=eps.device)
    normal[:dim] = 1.0
    third = torch.full_like(normal, 0.5)
    third[:dim] = 1.0
    K3, G2 = E / (1 - 2 * nu), E / (1 + nu)
    ev = eps[..., :dim].sum(-1, keepdim=True) / 3
    sig0 = K3 * ev * normal + G2 * (third * eps - ev * normal)
    eye = torch.diag(third)
    C = K3 / 3 * torch.outer(normal, normal) + G2 * (eye - torch.outer(normal, normal) / 3)
    if "kappa0" not in integ:
        one = torch.ones_like(eps[..., 0])
        return sig0, C, one, None, None, None, None
    k, k0, beta, alpha = integ["k"], integ["kappa0"], integ["beta"], integ["alpha"]
    K1, K2 = (k - 1) / (2 * k * (1 - 2 * nu)), 3 / (k * (1 + nu) ** 2)
    e3 = torch.zeros(eps.shape[:-1] + (3,), dtype=eps.dtype, device=eps.device)
    e3[..., :dim] = eps[..., :dim]
    I1 = e3.sum(-1)
    J2 = ((e3[..., 0] - e3[..., 1]) ** 2 + (e3[..., 1] - e3[..., 2]) ** 2 + (e3[..., 2] - e3[..., 0]) ** 2) / 6 \
        + 0.25 * (eps[..., dim:] ** 2).sum(-1)
    A = torch.sqrt(K1 * K1 * I1 * I1 + K2 * J2)
    mises = K1 * I1 + A
    dJ2 = torch.cat([e3[..., :dim] - I1[..., None] / 3, 0.5 * eps[..., dim:]], dim=-1)
    dm = K1 * normal + (K1 * K1 * I1[..., None] * normal + 0.5 * K2 * dJ2) / A[..., None]
    drive = mises if eeq is None else eeq
    kap = torch.maximum(kh, drive)
    damaged = kap >= k0
    ex = torch.exp(beta * (k0 - kap))
    omega = torch.where(damaged, 1 - k0 / kap * (1 - alpha + alpha * ex), 0.0)
    dom = torch.where(damaged, k0 / kap * ((1 / kap + beta) * alpha * ex + (1 - alpha) / kap), 0.0)
    s1 = -sig0 * (dom * (drive >= kh))[..., None]
    return sig0 * (1 - omega)[..., None], C, 1 - omega, s1, dm, mises, kap


class _Cells:
    """The integration-point data of a range of cells."""

    def __init__(self, s, x, kappa, dev, lo, hi):
        def dev64(a):
            return torch.as_tensor(a, device=dev).double()

        def ids(a):
            return torch.as_tensor(a.astype(np.int64), device=dev)

        mesh, dim = s.mesh, s.mesh.dim
        layers = [mesh.layers[l] for l in s.layers]
        g1, w1 = np.polynomial.legendre.leggauss(s.gauss)
        grid = np.meshgrid(*[np.arange(s.gauss)] * dim, indexing="ij")
        idx = np.stack([q.ravel() for q in grid[::-1]], axis=1)  # first coordinate fastest
        pts, w = g1[idx], np.prod(w1[idx], axis=1)
        _, dNg = _shape(mesh.conn.shape[1], pts)
        N, dN = _shape(layers[0].conn.shape[1], pts)
        self.N = dev64(N)
        J = torch.einsum("eni,qnj->eqij", dev64(mesh.coords)[ids(mesh.conn[lo:hi])], dev64(dNg))
        self.w = torch.linalg.det(J) * dev64(w)
        self.dN = torch.einsum("qnj,eqjk->eqnk", dev64(dN), torch.linalg.inv(J))
        conn = ids(layers[0].conn[lo:hi])
        numbers = ids(layers[0].dof_numbers)
        self.rows = numbers[conn].reshape(hi - lo, -1)  # node-major, components consecutive
        u = x[numbers[conn]]
        H = torch.einsum("enc,eqnd->eqcd", u, self.dN)
        e, q, n = self.dN.shape[:3]
        vd = 3 if dim == 2 else 6
        voigt = [(i, i) for i in range(dim)] + ([(0, 1)] if dim == 2 else [(1, 2), (0, 2), (0, 1)])
        B = torch.zeros((e, q, vd, n, dim), dtype=torch.float64, device=dev)
        eps = []
        for v, (i, j) in enumerate(voigt):
            B[:, :, v, :, i] += self.dN[..., j]
            if i != j:
                B[:, :, v, :, j] += self.dN[..., i]
            eps.append(H[..., i, i] if i == j else H[..., i, j] + H[..., j, i])
        self.B = B.reshape(e, q, vd, n * dim)
        kh = None if kappa is None else kappa[lo:hi]
        self.eeq = self.geeq = None
        if len(layers) == 2:
            ne = ids(layers[1].dof_numbers)[ids(layers[1].conn[lo:hi])][..., 0] + layers[0].num_dofs
            self.rows = torch.cat([self.rows, ne], dim=1)
            self.eeq = torch.einsum("qn,en->eq", self.N, x[ne])
            self.geeq = torch.einsum("en,eqnd->eqd", x[ne], self.dN)
        self.c = s.integrand.get("c", 0.0)
        self.law = _law(torch.stack(eps, -1), s.integrand, kh, self.eeq)

    def vectors(self):
        sig, _, _, _, _, mises, _ = self.law
        f = torch.einsum("eqva,eqv,eq->ea", self.B, sig, self.w)
        if self.eeq is None:
            return f
        fe = torch.einsum("qn,eq->en", self.N, (self.eeq - mises) * self.w) \
            + self.c * torch.einsum("eqnd,eqd,eq->en", self.dN, self.geeq, self.w)
        return torch.cat([f, fe], dim=1)

    def matrices(self):
        _, C, factor, s1, dm, _, _ = self.law
        CB = torch.einsum("uv,eqva->equa", C, self.B) * (factor * self.w)[..., None, None]
        if s1 is not None and self.eeq is None:  # local damage: the rank-1 part is in the displacement block
            CB += torch.einsum("equ,eqv,eqva,eq->equa", s1, dm, self.B, self.w)
        e = len(CB)
        K = self.B.reshape(e, -1, self.B.shape[-1]).transpose(1, 2) @ CB.reshape(e, -1, CB.shape[-1])
        if self.eeq is None:
            return K
        P = torch.einsum("eqva,eqv,eq->eqa", self.B, s1, self.w)
        Q = torch.einsum("eqva,eqv,eq->eqa", self.B, dm, self.w)
        ue = torch.einsum("eqa,qn->ean", P, self.N)
        eu = -torch.einsum("qn,eqa->ena", self.N, Q)
        ee = torch.einsum("qn,qm,eq->enm", self.N, self.N, self.w) \
            + self.c * torch.einsum("eqnd,eqmd,eq->enm", self.dN, self.dN, self.w)
        return torch.cat([torch.cat([K, ue], dim=2), torch.cat([eu, ee], dim=2)], dim=1)


def exact(case, seed):
    s = _setup(case["mesh"], case["n"], case["curved"])
    if case["op"] == "solve":  # the right-hand side was made from the solution
        return {"x": _correction(s, case, seed)}
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    x, kappa = _state(s, case, seed)
    x = torch.as_tensor(x, device=dev)
    kappa = None if kappa is None else torch.as_tensor(kappa, device=dev)
    step = 16384 if case["mesh"] != "hex20" else 2048
    ranges = [(lo, min(lo + step, s.mesh.num_cells)) for lo in range(0, s.mesh.num_cells, step)]
    n = s.n_dofs
    if case["op"] == "post":
        parts = [_Cells(s, x, kappa, dev, lo, hi).law for lo, hi in ranges]
        return {"stress": torch.cat([p[0] for p in parts]), "kappa": torch.cat([p[6] for p in parts])[..., None]}
    f = torch.zeros(n, dtype=torch.float64, device=dev)
    keys, mats = [], []
    for lo, hi in ranges:
        cells = _Cells(s, x, kappa, dev, lo, hi)
        if case["op"] != "matrix":
            f.index_add_(0, cells.rows.reshape(-1), cells.vectors().reshape(-1))
        if case["op"] != "vector":
            keys.append((cells.rows[:, :, None] * n + cells.rows[:, None, :]).reshape(-1))
            mats.append(cells.matrices().reshape(-1))
    out = {} if case["op"] == "matrix" else {"f": f}
    if case["op"] != "vector":
        keys, mats = torch.cat(keys), torch.cat(mats)
        pattern = torch.unique(keys)
        values = torch.zeros(len(pattern), dtype=torch.float64, device=dev)
        values.index_add_(0, torch.searchsorted(pattern, keys), mats)
        out["values"] = values
    return out
