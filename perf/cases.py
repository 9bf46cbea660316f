"""The workloads this library's speed is measured on.

Each case is one call (or one short sequence of calls) of the public Python
mirror, as an application makes it: whole drivers on small meshes, PCG solves
on a kept matrix, the re-assembly of a kept matrix, one time step, one batched
solve, one forward/backward pair. Meshes are the generated boxes and squares
that the tests and the benchmark use; loads and coefficients come from a seed.

`exact` gives the same results from plain torch in 64 bits: element matrices
summed into a CSR matrix, and conjugate gradients run to round-off with two
refinement passes.
"""
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fenics-rs_b200"))
import fenics_cuda as fcu  # noqa: E402

MAX_ITER = 200000
NU = 0.3


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------

def listed():
    return [
        # The smallest whole call: the reference's own 2D Poisson case (64 x 64, 4,225 unknowns) through its driver.
        {"name": "poisson_2d_64", "kind": "poisson_2d", "nx": 64, "ny": 64, "tol": 1e-10},
        # An ordinary whole call in 3D, where building the pattern counts beside the solve (odd, ragged sizes).
        {"name": "poisson_3d_41", "kind": "poisson_3d", "nx": 41, "ny": 37, "nz": 33, "tol": 1e-10},
        # A mid-size elasticity solve in FP64: the inner solve of the vibration modes (56,355 unknowns).
        {"name": "elast_pcg_64_f64", "kind": "elast_pcg", "nx": 64, "ny": 16, "nz": 16, "mixed": False, "tol": 1e-9},
        # The benchmark's elasticity solve (421,443 unknowns) in both precisions.
        {"name": "elast_pcg_128_f64", "kind": "elast_pcg", "nx": 128, "ny": 32, "nz": 32, "mixed": False, "tol": 1e-8},
        {"name": "elast_pcg_128_mixed", "kind": "elast_pcg", "nx": 128, "ny": 32, "nz": 32, "mixed": True, "tol": 1e-8},
        # The largest solve (1,568,403 unknowns): the operator exceeds L2 several times over.
        {"name": "elast_pcg_200_f64", "kind": "elast_pcg", "nx": 200, "ny": 50, "nz": 50, "mixed": False, "tol": 1e-8},
        # Re-assembly on a kept space, as each step of an optimisation or a nonlinear loop does: stiffness with a
        # modulus per cell, load, Dirichlet elimination, and one product with the current displacement.
        {"name": "elast_assemble_128", "kind": "elast_assemble", "nx": 128, "ny": 32, "nz": 32},
        # The same for P2 Poisson with a coefficient per cell (2,146,689 unknowns).
        {"name": "p2_assemble_64", "kind": "p2_assemble", "nx": 64, "ny": 64, "nz": 64},
        # The P2 solve with the random coefficient, FP32 operator with FP64 refinement.
        {"name": "p2_pcg_64_mixed", "kind": "p2_pcg", "nx": 64, "ny": 64, "nz": 64, "mixed": True, "tol": 1e-10},
        # One Crank-Nicolson step of the 2D heat equation on 1,050,625 unknowns, from the previous state.
        {"name": "heat_step_1024_f64", "kind": "heat_step", "nx": 1024, "ny": 1024, "dt": 1e-4, "mixed": False,
         "tol": 1e-10},
        # 256 independent Poisson problems of uneven sizes, each solved to its own tolerance in one call.
        {"name": "batch_256_mixed", "kind": "batch", "count": 256, "nmin": 32, "nmax": 256, "sizes": 2024,
         "mixed": True, "tol": 1e-11},
        # Forward and backward of the adjoint pair: u(theta), J and dJ/dtheta for a tip-displacement objective.
        {"name": "adjoint_96", "kind": "adjoint", "nx": 96, "ny": 32, "nz": 32, "compliance": False, "tol": 1e-12},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["poisson_2d", "poisson_3d", "elast_pcg", "elast_pcg", "elast_assemble", "p2_assemble",
                       "p2_pcg", "heat_step", "batch", "adjoint"])
    mixed = rng.random() < 0.5
    if kind == "poisson_2d":
        return {"kind": kind, "nx": _log(rng, 16, 200), "ny": _log(rng, 16, 200), "tol": 1e-10}
    if kind == "poisson_3d":
        return {"kind": kind, "nx": _log(rng, 8, 56), "ny": _log(rng, 8, 56), "nz": _log(rng, 8, 56), "tol": 1e-10}
    if kind == "elast_pcg":
        # (mixed solves end on the true FP64 residual, which rounding keeps above about 2e-9 on the largest meshes)
        if mixed:
            return {"kind": kind, "nx": _log(rng, 24, 144), "ny": _log(rng, 8, 36), "nz": _log(rng, 8, 36),
                    "mixed": True, "tol": 1e-8}
        return {"kind": kind, "nx": _log(rng, 24, 200), "ny": _log(rng, 8, 48), "nz": _log(rng, 8, 48),
                "mixed": False, "tol": 1e-9}
    if kind == "elast_assemble":
        return {"kind": kind, "nx": _log(rng, 24, 200), "ny": _log(rng, 8, 50), "nz": _log(rng, 8, 50)}
    if kind == "p2_assemble":
        return {"kind": kind, "nx": _log(rng, 8, 64), "ny": _log(rng, 8, 64), "nz": _log(rng, 8, 64)}
    if kind == "p2_pcg":
        return {"kind": kind, "nx": _log(rng, 8, 64), "ny": _log(rng, 8, 64), "nz": _log(rng, 8, 64),
                "mixed": mixed, "tol": 1e-10}
    if kind == "heat_step":
        return {"kind": kind, "nx": _log(rng, 96, 1024), "ny": _log(rng, 96, 1024), "dt": 1e-4, "mixed": mixed,
                "tol": 1e-10}
    if kind == "batch":
        return {"kind": kind, "count": _log(rng, 16, 256), "nmin": rng.randint(16, 48), "nmax": rng.randint(64, 256),
                "sizes": rng.randrange(1 << 20), "mixed": mixed, "tol": 1e-11}
    return {"kind": kind, "nx": _log(rng, 24, 96), "ny": _log(rng, 8, 32), "nz": _log(rng, 8, 32),
            "compliance": rng.random() < 0.5, "tol": 1e-12}


# ---------------------------------------------------------------------------
# host geometry (kept between preparations: it does not depend on the seed)
# ---------------------------------------------------------------------------

@functools.lru_cache(maxsize=4)
def _box(length, nx, ny, nz):
    m = fcu.box_beam(length, 1.0, 1.0, nx, ny, nz)
    return m.coords, m.cells


@functools.lru_cache(maxsize=2)
def _square(nx, ny):
    m = fcu.unit_square(nx, ny)
    return m.coords, m.cells


def _batch_sizes(case):
    return np.random.default_rng(case["sizes"]).integers(case["nmin"], case["nmax"] + 1, size=case["count"])


@functools.lru_cache(maxsize=2)
def _squares(ns):
    mesh, offs = fcu.concat_meshes([fcu.unit_square(n, n) for n in ns])
    return mesh.coords, mesh.cells, offs


def _geometry(case):
    kind = case["kind"]
    if kind in ("poisson_2d", "heat_step"):
        return _square(case["nx"], case["ny"])
    if kind == "batch":
        return _squares(tuple(int(n) for n in _batch_sizes(case)))[:2]
    # the cantilever of the elasticity configurations, the adjoint's shorter beam, the unit cube
    length = 4.0 if kind in ("elast_pcg", "elast_assemble") else 3.0 if kind == "adjoint" else 1.0
    return _box(length, case["nx"], case["ny"], case["nz"])


def _clamped(coords):
    """The dofs of the vertices at x = 0, three per vertex."""
    cv = np.nonzero(coords[:, 0] < 1e-6)[0]
    return (3 * cv[:, None] + np.arange(3)).ravel().astype(np.int64)


def _dev(a, dtype=None):
    return torch.as_tensor(np.ascontiguousarray(a), device="cuda", dtype=dtype)


# ---------------------------------------------------------------------------
# inputs from the seed
# ---------------------------------------------------------------------------

def _inputs(case, seed):
    """Loads and coefficients as host values."""
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    coords, cells = _geometry(case)
    if kind == "poisson_2d":
        return {"amp": float(rng.uniform(5.0, 40.0)), "freq": [int(k) for k in rng.integers(1, 4, size=2)]}
    if kind == "poisson_3d":
        return {"amp": float(rng.uniform(5.0, 40.0)), "freq": []}  # a uniform source
    if kind == "elast_pcg":
        return {"E": float(rng.uniform(70e9, 210e9)), "force": rng.uniform(-1.0, 1.0, 3) * 2e4 + [0.0, 0.0, -7.8e4]}
    if kind == "elast_assemble":
        return {"cell_E": rng.uniform(70e9, 210e9, len(cells)), "force": rng.uniform(-1.0, 1.0, 3) * 7.8e4,
                "u": rng.standard_normal(3 * len(coords)) * 1e-3}
    if kind in ("p2_assemble", "p2_pcg"):
        return {"kappa": np.exp(rng.standard_normal(len(cells))), "f": float(rng.uniform(0.5, 2.0)),
                "u_seed": int(rng.integers(1 << 30))}
    if kind == "heat_step":
        x, y = coords[:, 0], coords[:, 1]
        u = np.zeros(len(coords))
        for _ in range(4):
            kx, ky = rng.integers(1, 9, size=2)
            u += rng.standard_normal() * np.sin(kx * math.pi * x) * np.sin(ky * math.pi * y)
        return {"u": u, "f0": rng.uniform(0.0, 1.0, len(coords)) / len(coords),
                "f1": rng.uniform(0.0, 1.0, len(coords)) / len(coords)}
    if kind == "batch":
        return {"kappa": np.exp(rng.standard_normal(len(cells))), "f": rng.uniform(-1.0, 1.0, len(coords))}
    return {"theta": rng.uniform(0.01, 1.0, len(cells)), "traction": rng.uniform(-0.3, 0.3, 3) + [0.0, 0.0, -1.0]}


def _tip(coords, cells):
    """Weights of the mean u_z over the vertices at the free end x = 3."""
    tip = np.nonzero(coords[:, 0] > 3.0 - 1e-9)[0]
    c = np.zeros(3 * len(coords))
    c[3 * tip + 2] = 1.0 / len(tip)
    return c


def _source(inp):
    def f(*x):
        v = inp["amp"]
        for k, xi in zip(inp["freq"], x):
            v = v * np.sin(k * math.pi * xi)
        return v
    return f


def prepare(case, seed):
    kind = case["kind"]
    ctx = fcu.default_context()
    inp = _inputs(case, seed)
    coords, cells = _geometry(case)
    mesh = fcu.Mesh(coords, cells)
    prec = fcu.FCU_MIXED if case.get("mixed") else fcu.FCU_FP64
    s = {"kind": kind, "mesh": mesh, "tol": case.get("tol"), "prec": prec}
    if kind in ("poisson_2d", "poisson_3d"):
        s["source"] = _source(inp)
        return s
    if kind in ("elast_pcg", "elast_assemble"):
        V = s["V"] = fcu.FunctionSpace(ctx, mesh, fcu.FCU_SPACE_P1_VEC3)
        M = s["M"] = fcu.Matrix(ctx, V)
        d = _clamped(coords)
        s["dofs"], s["vals"] = _dev(d), torch.zeros(len(d), dtype=torch.float64, device="cuda")
        s["b"] = torch.empty(V.ndofs, dtype=torch.float64, device="cuda")
        s["x"] = torch.empty_like(s["b"])
        s["force"] = inp["force"]
        if kind == "elast_assemble":
            s["cell_E"], s["u"] = _dev(inp["cell_E"]), _dev(inp["u"])
            return s
        torch.cuda.synchronize()
        M.assemble_elasticity(inp["E"], NU)
        V.body_force(s["force"], out=s["b"])
        M.apply_dirichlet(s["b"], s["dofs"], s["vals"])
        return s
    if kind in ("p2_assemble", "p2_pcg"):
        V = s["V"] = fcu.FunctionSpace(ctx, mesh, fcu.FCU_SPACE_P2)
        M = s["M"] = fcu.Matrix(ctx, V)
        d = V.boundary_dofs()
        s["dofs"], s["vals"] = _dev(d), torch.zeros(len(d), dtype=torch.float64, device="cuda")
        s["b"] = torch.empty(V.ndofs, dtype=torch.float64, device="cuda")
        s["x"] = torch.empty_like(s["b"])
        s["kappa"], s["f"] = _dev(inp["kappa"]), inp["f"]
        torch.cuda.synchronize()
        if kind == "p2_assemble":
            s["u"] = _normal(inp["u_seed"], V.ndofs)
            return s
        M.assemble_stiffness(s["kappa"])
        V.rhs_source(fcu.FCU_SRC_CONSTANT, params=(s["f"],), out=s["b"])
        M.apply_dirichlet(s["b"], s["dofs"], s["vals"])
        return s
    if kind == "heat_step":
        V = s["V"] = fcu.FunctionSpace(ctx, mesh, fcu.FCU_SPACE_P1)
        s["mass"] = fcu.Matrix(ctx, V).assemble_mass(1.0)
        s["stiff"] = fcu.Matrix(ctx, V).assemble_stiffness(None)
        s["solver"] = fcu.TransientHeatSolver(fcu.TimeSteppingScheme.CrankNicolson, case["dt"], ctx, tol=case["tol"],
                                              max_iter=MAX_ITER, precision=prec)
        s["u"], s["f0"], s["f1"] = (_dev(inp[k]) for k in ("u", "f0", "f1"))
        return s
    if kind == "batch":
        s["offs"] = _squares(tuple(int(n) for n in _batch_sizes(case)))[2]
        V = s["V"] = fcu.FunctionSpace(ctx, mesh, fcu.FCU_SPACE_P1)
        kappa, f = _dev(inp["kappa"]), _dev(inp["f"])
        s["b"] = torch.empty(V.ndofs, dtype=torch.float64, device="cuda")
        s["x"] = torch.empty_like(s["b"])
        d = V.boundary_dofs()
        torch.cuda.synchronize()
        M = s["M"] = fcu.Matrix(ctx, V).assemble_stiffness(kappa)
        V.rhs_source(fcu.FCU_SRC_NODAL, nodal=f, out=s["b"])
        M.apply_dirichlet(s["b"], d, np.zeros(len(d)))
        ctx.synchronize()
        return s
    facets = fcu.facets_on_plane(mesh, 0, 3.0, ctx)
    V = fcu.FunctionSpace(ctx, mesh, fcu.FCU_SPACE_P1_VEC3)
    load = fcu.traction_load(V, facets, inp["traction"])
    V.close()
    objective = "compliance" if case["compliance"] else _tip(coords, cells)
    s["pair"] = fcu.ElasticityAdjoint(mesh, NU, load, _clamped(coords), objective=objective, ctx=ctx, tol=case["tol"],
                                      max_iter=MAX_ITER)
    s["theta"] = inp["theta"]
    return s


def run(s):
    kind = s["kind"]
    if kind == "poisson_2d":
        return fcu.solve_poisson_2d(s["mesh"], s["source"], lambda x, y: 0.0, s["tol"], MAX_ITER).u
    if kind == "poisson_3d":
        return fcu.solve_poisson_3d(s["mesh"], s["source"], lambda x, y, z: 0.0, s["tol"], MAX_ITER).u
    if kind in ("elast_pcg", "p2_pcg"):
        return s["M"].pcg(s["b"], x=s["x"], tol=s["tol"], max_iter=MAX_ITER, precision=s["prec"])[0]
    if kind == "elast_assemble":
        s["M"].assemble_elasticity(1.0, NU, s["cell_E"])
        s["V"].body_force(s["force"], out=s["b"])
        s["M"].apply_dirichlet(s["b"], s["dofs"], s["vals"])
        return {"load": s["b"], "product": s["M"].spmv(s["u"], s["x"])}
    if kind == "p2_assemble":
        s["M"].assemble_stiffness(s["kappa"])
        s["V"].rhs_source(fcu.FCU_SRC_CONSTANT, params=(s["f"],), out=s["b"])
        s["M"].apply_dirichlet(s["b"], s["dofs"], s["vals"])
        return {"load": s["b"], "product": s["M"].spmv(s["u"], s["x"])}
    if kind == "heat_step":
        return s["solver"].step(s["mass"], s["stiff"], s["u"], s["f0"], s["f1"])
    if kind == "batch":
        return s["M"].batch_pcg(s["offs"], s["b"], x=s["x"], tol=s["tol"], max_iter=MAX_ITER, precision=s["prec"])[0]
    J = s["pair"].forward(s["theta"])
    grad = s["pair"].backward()
    return {"J": J, "u": s["pair"].u, "grad": grad}


# ---------------------------------------------------------------------------
# bytes and operations
# ---------------------------------------------------------------------------

def work(case):
    """Every input read once and every output written once; operations of one
    product with the matrix (solves repeat it as often as they need)."""
    kind = case["kind"]
    if kind in ("poisson_2d", "heat_step"):
        nx, ny = case["nx"], case["ny"]
        nv, nc, d = (nx + 1) * (ny + 1), 2 * nx * ny, 2
        edges = nx * (ny + 1) + ny * (nx + 1) + nx * ny
    elif kind == "batch":
        ns = _batch_sizes(case).astype(np.float64)
        nv, nc, d = float(np.sum((ns + 1) ** 2)), float(np.sum(2 * ns * ns)), 2
        edges = float(np.sum(2 * ns * (ns + 1) + ns * ns))
    else:
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        nv, nc, d = (nx + 1) * (ny + 1) * (nz + 1), 6 * nx * ny * nz, 3
        edges = (nx * (ny + 1) * (nz + 1) + (nx + 1) * ny * (nz + 1) + (nx + 1) * (ny + 1) * nz
                 + nx * ny * (nz + 1) + nx * (ny + 1) * nz + (nx + 1) * ny * nz + nx * ny * nz)
    entries = nv + 2 * edges  # of the P1 node pattern
    mesh_bytes = 8.0 * d * nv + 8.0 * (d + 1) * nc
    val = 4.0 if case.get("mixed") else 8.0
    if kind in ("poisson_2d", "poisson_3d"):
        return {"bytes": mesh_bytes + 8.0 * nv, "flops": 2.0 * entries}
    if kind == "elast_pcg":
        return {"bytes": entries * (9 * val + 4) + 2 * 24.0 * nv, "flops": 18.0 * entries}
    if kind == "elast_assemble":
        # connectivity and modulus in, values out, the displacement in and the load and product out
        return {"bytes": 24.0 * nv + (16.0 + 8.0) * nc + 12.0 * 9 * entries + 3 * 24.0 * nv, "flops": 18.0 * entries}
    if kind in ("p2_assemble", "p2_pcg"):
        ndofs = (2 * nx + 1) * (2 * ny + 1) * (2 * nz + 1)
        nnz = 28.4 * ndofs
        if kind == "p2_pcg":
            return {"bytes": nnz * (val + 4) + 16.0 * ndofs, "flops": 2.0 * nnz}
        return {"bytes": 24.0 * nv + (40.0 + 8.0) * nc + 12.0 * nnz + 24.0 * ndofs, "flops": 2.0 * nnz}
    if kind == "heat_step":
        return {"bytes": 2 * entries * 12.0 + 32.0 * nv, "flops": 4.0 * entries}
    if kind == "batch":
        return {"bytes": entries * (val + 4) + 16.0 * nv, "flops": 2.0 * entries}
    # two solves with the matrix of this theta, then the gradient
    return {"bytes": mesh_bytes + 16.0 * nc + entries * 76.0 + 48.0 * nv, "flops": 36.0 * entries}


# ---------------------------------------------------------------------------
# the same results in plain torch, 64 bits
# ---------------------------------------------------------------------------

def _normal(seed, n):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return torch.randn(n, dtype=torch.float64, device="cuda", generator=g)


def _barycentric(coords, cells):
    """Gradients of the barycentric coordinates [nc, d+1, d] and cell measures."""
    X = coords[cells]
    d = coords.shape[1]
    J = (X[:, 1:] - X[:, :1]).transpose(1, 2)
    G = torch.linalg.inv(J)
    g = torch.cat([-G.sum(1, keepdim=True), G], 1)
    return g, torch.linalg.det(J).abs() / math.factorial(d)


def _csr(nodes, n, K, comp=1):
    """CSR of the summed element matrices K [nc, k, k, comp, comp] on nodes [nc, k]."""
    k = nodes.shape[1]
    key = (nodes[:, :, None] * n + nodes[:, None, :]).reshape(-1)
    uniq, inv = torch.unique(key, return_inverse=True)
    del key
    vals = torch.zeros(len(uniq), comp * comp, dtype=torch.float64, device="cuda")
    vals.index_add_(0, inv, K.reshape(-1, comp * comp))
    del inv
    row, col = uniq // n, uniq % n
    cnt = torch.bincount(row, minlength=n)
    start = torch.cumsum(cnt, 0) - cnt
    if comp == 1:
        crow = torch.cat([start, start.new_tensor([len(uniq)])])
        return crow.int(), col.int(), vals.reshape(-1), row
    c = torch.arange(comp, device="cuda")
    at = (9 * start[row] + comp * (torch.arange(len(uniq), device="cuda") - start[row]))[:, None, None] \
        + (comp * cnt[row])[:, None, None] * c[None, :, None] + c[None, None, :]
    nnz = 9 * len(uniq)
    cols = torch.empty(nnz, dtype=torch.int32, device="cuda")
    v = torch.empty(nnz, dtype=torch.float64, device="cuda")
    cols[at.reshape(-1)] = (comp * col[:, None, None] + c[None, None, :]).expand(-1, comp, -1).reshape(-1).int()
    v[at.reshape(-1)] = vals.reshape(-1)
    per = (comp * cnt)[:, None].expand(-1, comp).reshape(-1)
    crow = torch.cat([per.new_zeros(1), torch.cumsum(per, 0)])
    return crow.int(), cols, v, torch.repeat_interleave(torch.arange(comp * n, device="cuda"), per)


class _System:
    def __init__(self, parts, fixed=None):
        crow, col, val, row = parts
        n = len(crow) - 1
        if fixed is not None:
            m = torch.zeros(n, dtype=torch.bool, device="cuda")
            m[fixed] = True
            val = torch.where(m[row] | m[col.long()], torch.where(row == col, 1.0, 0.0).double(), val)
        on = row == col
        self.diag = torch.zeros(n, dtype=torch.float64, device="cuda").index_add_(0, row[on], val[on])
        self.A = torch.sparse_csr_tensor(crow, col, val, size=(n, n))

    def mul(self, x):
        return self.A @ x

    def _cg(self, b, tol):
        x = torch.zeros_like(b)
        r, d = b.clone(), 1.0 / self.diag
        z = r * d
        p = z.clone()
        rz = torch.dot(r, z)
        stop = float(torch.linalg.vector_norm(b)) * tol
        if stop == 0.0:
            return x
        for it in range(1, 40001):
            q = self.A @ p
            alpha = rz / torch.dot(p, q)
            x.addcmul_(p, alpha)
            r.addcmul_(q, -alpha)
            z = r * d
            new = torch.dot(r, z)
            p = torch.addcmul(z, p, new / rz)
            rz = new
            if it % 64 == 0 and float(torch.linalg.vector_norm(r)) < stop:
                break
        return x

    def solve(self, b):
        x = self._cg(b, 1e-13)
        for _ in range(2):
            x = x + self._cg(b - self.A @ x, 1e-4)
        return x


def _scalar_element(g, m, coef=None):
    K = torch.einsum("cad,cbd->cab", g, g) * (m if coef is None else m * coef)[:, None, None]
    return K


def _elastic_element(g, m, lam, mu):
    """K[c, a, b, i, j] = m (lam g_ai g_bj + mu g_aj g_bi + mu delta_ij g_a.g_b)."""
    gg = torch.einsum("cai,cbj->cabij", g, g)
    K = lam * gg + mu * gg.transpose(-1, -2)
    K += mu * torch.einsum("cad,cbd->cab", g, g)[..., None, None] * torch.eye(3, dtype=torch.float64, device="cuda")
    return K * m[:, None, None, None, None]


def _lame(E):
    return E * NU / ((1 + NU) * (1 - 2 * NU)), E / (2 * (1 + NU))


def _p2_tensor():
    """T[a, b, m, n]: cell mean of (d phi_a / d lambda_m)(d phi_b / d lambda_n) for the ten P2 functions."""
    edges = [(0, 1), (1, 2), (0, 2), (0, 3), (1, 3), (2, 3)]
    c = np.zeros((10, 4, 5))  # d phi_a / d lambda_m = c[..., 0] + sum_k c[..., 1 + k] lambda_k
    for i in range(4):
        c[i, i, 0], c[i, i, 1 + i] = -1.0, 4.0
    for e, (i, j) in enumerate(edges):
        c[4 + e, i, 1 + j] = 4.0
        c[4 + e, j, 1 + i] = 4.0
    mean = np.full((5, 5), 0.05)
    mean[0, :] = mean[:, 0] = 0.25
    mean[0, 0] = 1.0
    for k in range(4):
        mean[1 + k, 1 + k] = 0.1
    return np.einsum("amk,bnl,kl->abmn", c, c, mean), edges


def _p2_system(coords, cells, kappa):
    nv = len(coords)
    T, edges = _p2_tensor()
    pairs = torch.stack([torch.stack([torch.minimum(cells[:, i], cells[:, j]), torch.maximum(cells[:, i], cells[:, j])], 1)
                         for i, j in edges], 1)
    key = pairs[..., 0] * nv + pairs[..., 1]
    uniq, inv = torch.unique(key.reshape(-1), return_inverse=True)
    nodes = torch.cat([cells, nv + inv.reshape(-1, 6)], 1)
    n = nv + len(uniq)
    g, m = _barycentric(coords, cells)
    G = torch.einsum("cad,cbd->cab", g, g) * (m * kappa)[:, None, None]
    K = G.reshape(-1, 16) @ _dev(T.reshape(100, 16).T.copy())
    load = torch.zeros(n, dtype=torch.float64, device="cuda")
    w = torch.tensor([-0.05] * 4 + [0.2] * 6, dtype=torch.float64, device="cuda")
    load.index_add_(0, nodes.reshape(-1), (m[:, None] * w).reshape(-1))
    X = torch.cat([coords, 0.5 * (coords[uniq // nv] + coords[uniq % nv])])
    fixed = ((X < 1e-12) | (X > 1 - 1e-12)).any(1)
    return _csr(nodes, n, K), load, torch.nonzero(fixed).reshape(-1)


def _vertex_sum(nv, cells, w):
    k = cells.shape[1]
    return torch.zeros(nv, dtype=torch.float64, device="cuda").index_add_(0, cells.reshape(-1), w.repeat_interleave(k))


def _simplex_load(coords, cells, m, f):
    """The drivers' load: f at the rule's points (the edge midpoints of a triangle, the four interior points of a
    tetrahedron), each weighted equally."""
    d = coords.shape[1]
    X = coords[cells]
    if d == 2:
        L = np.array([[0.5, 0.5, 0.0], [0.0, 0.5, 0.5], [0.5, 0.0, 0.5]])
    else:
        a, b = 0.5854101966249685, 0.1381966011250105
        L = np.full((4, 4), b) + (a - b) * np.eye(4)
    L = _dev(L)
    Q = torch.einsum("qa,cad->cqd", L, X).cpu().numpy()
    fq = _dev(np.broadcast_to(f(*[Q[..., k] for k in range(d)]), Q.shape[:2]))
    w = torch.einsum("cq,qa->ca", fq, L) * (m / len(L))[:, None]
    return torch.zeros(len(coords), dtype=torch.float64, device="cuda").index_add_(0, cells.reshape(-1), w.reshape(-1))


def _on_boundary(coords):
    return torch.nonzero(((coords < 1e-12) | (coords > 1 - 1e-12)).any(1)).reshape(-1)


def exact(case, seed):
    kind = case["kind"]
    inp = _inputs(case, seed)
    hc, hcells = _geometry(case)
    coords, cells = _dev(hc), _dev(hcells)
    nv = len(coords)
    if kind in ("p2_assemble", "p2_pcg"):
        parts, load, fixed = _p2_system(coords, cells, _dev(inp["kappa"]))
        load = load * inp["f"]
        load[fixed] = 0.0
        A = _System(parts, fixed)
        if kind == "p2_pcg":
            return A.solve(load)
        return {"load": load, "product": A.mul(_normal(inp["u_seed"], len(load)))}
    g, m = _barycentric(coords, cells)
    if kind in ("poisson_2d", "poisson_3d"):
        b = _simplex_load(coords, cells, m, _source(inp))
        fixed = _on_boundary(coords)
        b[fixed] = 0.0
        return _System(_csr(cells, nv, _scalar_element(g, m)), fixed).solve(b).cpu().numpy()
    if kind == "heat_step":
        K = _scalar_element(g, m)
        mass = (torch.ones(3, 3, dtype=torch.float64, device="cuda") + torch.eye(3, dtype=torch.float64, device="cuda")) / 12
        Mm = m[:, None, None] * mass
        h = 0.5 * case["dt"]
        u = _dev(inp["u"])
        rhs = _System(_csr(cells, nv, Mm - h * K)).mul(u) + h * (_dev(inp["f0"]) + _dev(inp["f1"]))
        return _System(_csr(cells, nv, Mm + h * K)).solve(rhs)
    if kind == "batch":
        mass = (torch.ones(3, 3, dtype=torch.float64, device="cuda") + torch.eye(3, dtype=torch.float64, device="cuda")) / 12
        w = (_dev(inp["f"])[cells] @ mass) * m[:, None]
        b = torch.zeros(nv, dtype=torch.float64, device="cuda").index_add_(0, cells.reshape(-1), w.reshape(-1))
        fixed = _on_boundary(coords)
        b[fixed] = 0.0
        return _System(_csr(cells, nv, _scalar_element(g, m, _dev(inp["kappa"]))), fixed).solve(b)
    fixed = _dev(_clamped(hc))
    if kind in ("elast_pcg", "elast_assemble"):
        E = torch.full_like(m, inp["E"]) if kind == "elast_pcg" else _dev(inp["cell_E"])
        lam, mu = _lame(1.0)
        A = _System(_csr(cells, nv, _elastic_element(g, m * E, lam, mu), 3), fixed)
        b = (_vertex_sum(nv, cells, m / 4)[:, None] * _dev(inp["force"])).reshape(-1)
        b[fixed] = 0.0
        if kind == "elast_pcg":
            return A.solve(b)
        return {"load": b, "product": A.mul(_dev(inp["u"]))}
    theta = _dev(inp["theta"])
    lam, mu = _lame(1.0)
    K1 = _elastic_element(g, m, lam, mu)
    A = _System(_csr(cells, nv, K1 * (theta ** 3)[:, None, None, None, None], 3), fixed)
    # constant traction on x = 3: each boundary triangle gives a third of its area to its vertices
    F = torch.cat([cells[:, [a, b, c]] for a, b, c in ((1, 2, 3), (0, 2, 3), (0, 1, 3), (0, 1, 2))])
    F = F[(coords[F][..., 0] > 3.0 - 1e-9).all(1)]
    X = coords[F]
    area = 0.5 * torch.linalg.vector_norm(torch.linalg.cross(X[:, 1] - X[:, 0], X[:, 2] - X[:, 0]), dim=1)
    f = (_vertex_sum(nv, F, area / 3)[:, None] * _dev(inp["traction"])).reshape(-1)
    c = f if case["compliance"] else _dev(_tip(hc, hcells))
    bf, bc = f.clone(), c.clone()
    bf[fixed], bc[fixed] = 0.0, 0.0
    u = A.solve(bf)
    ad = u if case["compliance"] else A.solve(bc)
    ue, le = u.reshape(-1, 3)[cells], ad.reshape(-1, 3)[cells]
    grad = -3.0 * theta ** 2 * torch.einsum("cai,cabij,cbj->c", le, K1, ue)
    return {"J": float(torch.dot(c, u)), "u": u.cpu().numpy(), "grad": grad.cpu().numpy()}
