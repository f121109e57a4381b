"""What a user of the library has it do, as cases to be timed: fluid_mc assemblies, their
residuals and adjoints, the linear solve and a whole time step, each through the package's
public objects (FluidAssembly, LinearSolver, newton.time_step_device).

A case names its mesh (element type and cells per direction), its number of components and
the call; the meshes are the synthetic ones of the package and a lattice of tetrahedra, the
materials, states and boundary policy are those of the package's synthetic module.  The seed
draws the state, the previous level, the melt's viscosity and the adjoint's lambda; a mesh is
the program's mesh file and does not depend on it.

exact() restates the element integral (interior, boundary, Dirichlet rows, scatter) in plain
torch in 64 bits, with dense matrices; the adjoint is its reverse-mode derivative.
"""
import functools
import importlib
import math

import numpy as np
import torch

gm = importlib.import_module("gales-multi-fluid_gb300")
syn = importlib.import_module("gales-multi-fluid_gb300.synthetic")
newton = importlib.import_module("gales-multi-fluid_gb300.newton")
magma = importlib.import_module("gales-multi-fluid_gb300.magma")

DT = 1e-3
DEVICE = torch.device("cuda" if torch.cuda.is_available() else "cpu")
WALL, OPEN = syn.WALL, syn.OPEN


# ---------------------------------------------------------------------------
# Meshes

def _lattice_tets(nx, ny, nz, jitter=0.1, seed=7):
    """Six tetrahedra per cell of an nx x ny x nz lattice of the unit box, inner nodes
    moved by up to `jitter` cells; walls everywhere but the open top z = 1."""
    g = [np.linspace(0.0, 1.0, n + 1) for n in (nx, ny, nz)]
    pts = np.stack([x.ravel() for x in np.meshgrid(*g, indexing="ij")], axis=1)
    h = np.array([1.0 / nx, 1.0 / ny, 1.0 / nz])
    d = np.random.default_rng(seed).uniform(-1.0, 1.0, size=pts.shape) * jitter * h
    d[(pts < 1e-12) | (pts > 1 - 1e-12)] = 0.0
    pts = pts + d
    idx = np.arange(len(pts)).reshape(nx + 1, ny + 1, nz + 1)

    def c(i, j, k):
        return idx[i:i + nx, j:j + ny, k:k + nz].ravel()
    axes = np.eye(3, dtype=int)
    tets = []
    for perm in ((0, 1, 2), (0, 2, 1), (1, 0, 2), (1, 2, 0), (2, 0, 1), (2, 1, 0)):
        at, corner = np.zeros(3, dtype=int), [np.zeros(3, dtype=int)]
        for ax in perm:
            at = at + axes[ax]
            corner.append(at)
        tets.append(np.stack([c(*v) for v in corner], axis=1))
    conn = np.stack(tets, axis=1).reshape(-1, 4)
    x = pts[conn]
    vol = np.einsum("ij,ij->i", np.cross(x[:, 1] - x[:, 0], x[:, 2] - x[:, 0]), x[:, 3] - x[:, 0])
    flip = vol < 0
    conn[flip, 1], conn[flip, 2] = conn[flip, 2].copy(), conn[flip, 1].copy()
    conn = conn.astype(np.int32)
    # sides of one element only, by a sorted 64-bit key of their nodes
    table = np.asarray(syn.SIDES[(3, 4)])
    f = np.sort(conn[:, table].reshape(-1, 3), axis=1).astype(np.int64)
    key = (f[:, 0] * len(pts) + f[:, 1]) * len(pts) + f[:, 2]
    order = np.argsort(key, kind="stable")
    k = key[order]
    same = k[1:] == k[:-1]
    twice = np.zeros(len(k), dtype=bool)
    twice[1:] |= same
    twice[:-1] |= same
    single = np.sort(order[~twice])
    el, loc = (single // 4).astype(np.int32), (single % 4).astype(np.int32)
    top = np.all(np.abs(pts[conn[el[:, None], table[loc]]][:, :, 2] - 1.0) < 1e-9, axis=1)
    bd = np.stack([el, loc, np.where(top, OPEN, WALL).astype(np.int32)], axis=1)
    el_bd = np.zeros(len(conn), dtype=np.uint8)
    el_bd[el] = 1
    on = (np.abs(pts) < 1e-9) | (np.abs(pts - 1.0) < 1e-9)
    flag = np.where(on.any(axis=1), WALL, 0).astype(np.int32)
    flag[(np.abs(pts[:, 2] - 1.0) < 1e-9) & ~on[:, :2].any(axis=1)] = OPEN
    return gm.Mesh(pts, conn, flag, el_bd, bd, name=f"lattice_tets_{nx}x{ny}x{nz}")


@functools.lru_cache(maxsize=16)
def _mesh(el, nx, ny, nz):
    if el == "tri":
        return syn.channel_tri(nx, ny)
    if el == "quad":
        return syn.channel_quad(nx, ny, jitter=0.2, seed=nx)
    if el == "tet":
        return _lattice_tets(nx, ny, nz)
    return syn.box_hex(nx, ny, nz, jitter=0.1, seed=4)


def _mesh_of(case):
    return _mesh(case["element"], case["nx"], case["ny"], case.get("nz", 0))


def _elements(case):
    per = {"tri": 2, "quad": 1, "tet": 6, "hex": 1}[case["element"]]
    return per * case["nx"] * case["ny"] * (case["nz"] if case["element"] in ("tet", "hex") else 1)


# ---------------------------------------------------------------------------
# The cases

def listed():
    return [
        # the smallest: the 2D two-component channel in the reference's arithmetic, where
        # launches and host work count
        dict(name="channel_tri_fp64", call="assemble", form="fp64", element="tri", nx=64, ny=32, comps=2),
        # an odd-sized 2D mesh of quadrilaterals in the mixed form
        dict(name="channel_quad_mixed", call="assemble", form="mixed", element="quad", nx=193, ny=97, comps=3),
        # the shipped case's material: a mixture of two magmas with solubility tables, T
        # prescribed at every node
        dict(name="channel_tri_magma", call="assemble", form="fp64", element="tri", nx=160, ny=80, comps=2, magma=True),
        # 3D tetrahedra at the benchmark's size: the FP64 form, the mixed form, and the mixed
        # form through pinned host buffers (the reference's interface)
        dict(name="tet_1m_fp64", call="assemble", form="fp64", element="tet", nx=55, ny=55, nz=55, comps=3),
        dict(name="tet_1m_mixed", call="assemble", form="mixed", element="tet", nx=55, ny=55, nz=55, comps=3),
        dict(name="tet_1m_mixed_host", call="assemble_host", form="mixed", element="tet", nx=55, ny=55, nz=55, comps=3),
        # hexahedra with four components: the mixed form at size and the FP64 form
        dict(name="hex_500k_mixed", call="assemble", form="mixed", element="hex", nx=80, ny=80, nz=78, comps=4),
        dict(name="hex_64k_fp64", call="assemble", form="fp64", element="hex", nx=41, ny=40, nz=39, comps=4),
        # the residual alone: the FP64 residual of an inexact Newton step, line searches
        dict(name="tet_residual_fp64", call="residual", form="fp64", element="tet", nx=33, ny=33, nz=33, comps=3),
        # the adjoint: gradients of a scalar with respect to the state and the parameters
        dict(name="tet_vjp_exact", call="vjp", mode="exact", element="tet", nx=33, ny=33, nz=33, comps=3),
        # the linear solve after an assembly with the shipped settings (flexible GMRES, ILU(1))
        dict(name="tet_solve", call="solve", precond="ilu", element="tet", nx=29, ny=29, nz=29, comps=3),
        # one whole time step of the driver on a 2D mesh: assembly, residual check, solve and
        # corrector for three Newton iterations, then the next time step's size
        dict(name="channel_time_step", call="time_step", form="fp64", element="quad", nx=64, ny=32, comps=2),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same calls, element types, component counts and sizes."""
    call = rng.choice(["assemble", "assemble", "assemble", "assemble_host", "residual", "vjp", "solve", "time_step"])
    case = dict(call=call)
    if call == "time_step":
        case.update(element="quad", comps=2, form=rng.choice(["fp64", "mixed"]), nx=rng.randint(20, 64))
        case["ny"] = max(8, case["nx"] // 2 + rng.randint(-3, 3))
        case["ny"] = min(case["ny"], 32)
        return case
    el = rng.choice(["tri", "quad", "tet", "tet", "hex"]) if call != "solve" else rng.choice(["quad", "tet"])
    case.update(element=el, comps=rng.randint(1, 4))
    if call == "vjp":
        case["mode"] = rng.choice(["exact", "frozen"])
    elif call == "solve":
        case["precond"] = rng.choice(["ilu", "ilu_fp32"])
        case["comps"] = min(case["comps"], 3)
    else:
        case["form"] = rng.choice(["fp64", "mixed"])
    # cells: a direction each, log-uniform in the number of cells of the whole mesh; the most
    # that a listed case of that call has, by the work of an element
    heavy = call == "vjp" or (call in ("assemble", "assemble_host", "residual") and case["form"] == "fp64")
    most = {"tri": 200000, "quad": 120000, "tet": 150000, "hex": 400000}[el]
    if heavy:
        most = {"tri": 100000, "quad": 60000, "tet": 35000, "hex": 40000}[el]
    if call == "solve":
        most = {"quad": 8000, "tet": 12000}[el]
    cells = _log(rng, 1500, most)
    if el in ("tri", "quad"):
        a = rng.uniform(0.8, 2.5)
        case["ny"] = max(9, int(math.sqrt(cells / a)))
        case["nx"] = max(9, cells // case["ny"])
    else:
        s = cells ** (1.0 / 3.0)
        case["nx"] = max(7, int(s * rng.uniform(0.8, 1.2)))
        case["ny"] = max(7, int(s * rng.uniform(0.8, 1.2)))
        case["nz"] = max(7, cells // (case["nx"] * case["ny"]))
    return case


def _dof_count(case):
    return gm.nb_dofs(2 if case["element"] in ("tri", "quad") else 3, case["comps"])


def _form(case):
    return gm.FORM_FP64 if case["form"] == "fp64" else gm.FORM_MIXED


def _inputs(case, seed):
    """(mesh, material, setup, I, P) on the host; T is prescribed everywhere with magmas."""
    mesh = _mesh_of(case)
    nc = case["comps"]
    mat = syn.material_for(nc, seed)
    setup = syn.setup_for(mesh.dim, nc, dirichlet_T_everywhere=bool(case.get("magma")))
    if case["call"] == "vjp":  # walls that move: the residual is not differentiable at rest
        I, P = syn.state_for(mesh, nc, seed, no_slip_flag=-1)
    elif case["call"] == "time_step":  # a state that Newton's iterations settle from
        I, P = syn.state_near_rest(mesh, nc, seed)
    else:
        I, P = syn.state_for(mesh, nc, seed)
    if case.get("magma"):  # pressures inside the solubility tables
        for S in (I.reshape(-1, mesh.dim + 1 + nc), P.reshape(-1, mesh.dim + 1 + nc)):
            S[:, 0] = 0.7e8 + 1.2 * S[:, 0]
    return mesh, mat, setup, I, P


def _lambda(case, seed, n):
    lam = np.random.default_rng(seed + 11).normal(size=n)
    return lam / np.linalg.norm(lam)


def prepare(case, seed):
    mesh, mat, setup, I, P = _inputs(case, seed)
    dev = DEVICE
    st = dict(case=case, fa=gm.FluidAssembly(mesh, mat, setup))
    fa = st["fa"]
    if case.get("magma"):
        st["magma"] = magma.MagmaMaterial(syn.magma_pair())
        fa.set_magma(st["magma"])
    call = case["call"]
    if call == "assemble_host":
        st["I"], st["P"] = torch.from_numpy(I).pin_memory(), torch.from_numpy(P).pin_memory()
        vals = torch.zeros(fa.nnz_from_graph(), dtype=torch.float64, pin_memory=True)
        rhs = torch.zeros(fa.n_rows, dtype=torch.float64, pin_memory=True)
        st["lp"] = gm.LinearSystem(None, None, vals, rhs)
        return st
    st["I"], st["P"] = torch.from_numpy(I).to(dev), torch.from_numpy(P).to(dev)
    if call == "assemble":
        st["lp"] = fa.device_system(dev)
    elif call == "residual":
        st["rhs"] = torch.zeros(fa.n_rows, dtype=torch.float64, device=dev)
    elif call == "vjp":
        st["lam"] = torch.from_numpy(_lambda(case, seed, fa.n_rows)).to(dev)
        st["g"] = torch.zeros(fa.n_rows, dtype=torch.float64, device=dev)
        st["gp"] = torch.zeros(3 * case["comps"], dtype=torch.float64, device=dev) if case["mode"] == "exact" else None
    elif call == "solve":
        st["lp"] = fa.device_system(dev)
        fa.set_scatter(gm.SCATTER_COLOURED)
        fa.execute(st["I"], st["P"], DT, st["lp"], form=gm.FORM_MIXED)
        kind = {"ilu": gm.PRECOND_ILU, "ilu_fp32": gm.PRECOND_ILU_FP32}[case["precond"]]
        st["solver"] = fa.linear_solver(gm.SolverParams(precond=kind))
        st["x"] = torch.zeros(fa.n_rows, dtype=torch.float64, device=dev)
    elif call == "time_step":
        st["lp"] = fa.device_system(dev)
        st["solver"] = fa.linear_solver()
    return st


def run(state):
    case, fa = state["case"], state["fa"]
    call = case["call"]
    if call in ("assemble", "assemble_host"):
        lp = state["lp"]
        fa.execute(state["I"], state["P"], DT, lp, form=_form(case))
        return {"vals": lp.vals, "rhs": lp.rhs}
    if call == "residual":
        fa.residual(state["I"], state["P"], DT, state["rhs"], form=_form(case))
        return {"rhs": state["rhs"]}
    if call == "vjp":
        mode = gm.VJP_EXACT if case["mode"] == "exact" else gm.VJP_FROZEN
        fa.vjp(state["I"], state["P"], DT, state["lam"], mode, state["g"], state["gp"])
        out = {"g_state": state["g"]}
        if state["gp"] is not None:
            out["g_params"] = state["gp"]
        return out
    if call == "solve":
        s = state["solver"]
        s.solve(state["lp"].vals, state["lp"].rhs, state["x"])
        return {"x": state["x"], "converged": s.converged}
    r = newton.time_step_device(fa, state["solver"], state["I"], DT, _form(case), max_it=3, lp=state["lp"])
    dt = fa.adaptive_dt(r["state"], DT, 1.0, 1e-6, 1.0)
    return {"state": r["state"], "history": list(r["history"]), "dt": dt}


def work(case):
    """The arrays of the call once each, and the operations of its element integrals: per
    point the mixture, tau and the fluxes (700) and per entry of the block and point four
    multiply-adds (one per shape value and gradient); a solve: the matrix once per
    factorisation and per iteration (30) with its factor of twice its entries."""
    n_el, nd = _elements(case), _dof_count(case)
    nen = {"tri": 3, "quad": 4, "tet": 4, "hex": 8}[case["element"]]
    dim = 2 if case["element"] in ("tri", "quad") else 3
    nodes = (case["nx"] + 1) * (case["ny"] + 1) * ((case["nz"] + 1) if dim == 3 else 1)
    deg = {"tri": 7, "quad": 9, "tet": 15, "hex": 27}[case["element"]]
    call = case["call"]
    rows, nnz = nodes * nd, nodes * deg * nd * nd
    mesh_bytes = 4 * nen * n_el + 8 * dim * nodes
    state = 2 * 8 * rows
    point = 700.0 * n_el * nen
    block = 8.0 * nen * n_el * (nen * nd) ** 2
    if call in ("assemble", "assemble_host"):
        return {"bytes": mesh_bytes + state + 8 * nnz + 8 * rows, "flops": point + block}
    if call == "residual":
        return {"bytes": mesh_bytes + state + 8 * rows, "flops": point + 8.0 * nen * n_el * nen * nd}
    if call == "vjp":
        extra = 3 * point if case["mode"] == "exact" else point + block
        return {"bytes": mesh_bytes + state + 16 * rows, "flops": extra}
    if call == "solve":
        return {"bytes": 8 * nnz + 16 * rows, "flops": 30 * (2.0 * nnz + 4.0 * nnz) + 40.0 * nd * nnz}
    it = 3
    return {"bytes": it * (mesh_bytes + state + 16 * nnz + 24 * rows),
            "flops": it * (point + block + 15 * 6.0 * nnz + 40.0 * nd * nnz)}


# ---------------------------------------------------------------------------
# The same results in plain torch

def _tables(el):
    """Interior points, weight; shape functions and local derivatives at a point; side
    points, side weight and the area vector of a side from the mapping derivatives."""
    s = 1.0 / math.sqrt(3.0)
    if el == "quad":
        return [(-s, -s), (s, -s), (s, s), (-s, s)], 1.0
    if el == "tri":
        return [(1 / 6, 1 / 6), (4 / 6, 1 / 6), (1 / 6, 4 / 6)], 1.0 / 6.0
    if el == "tet":
        a, b = 0.1381966011250105, 0.5854101966249685
        return [(a, a, a), (b, a, a), (a, b, a), (a, a, b)], 1.0 / 24.0
    return [(-s, -s, -s), (s, -s, -s), (s, s, -s), (-s, s, -s), (-s, -s, s), (s, -s, s), (s, s, s), (-s, s, s)], 1.0


def _side_points(el, side):
    s = 1.0 / math.sqrt(3.0)
    m, p = -s, s
    if el == "quad":
        return [[(m, -1.0), (p, -1.0)], [(1.0, m), (1.0, p)], [(p, 1.0), (m, 1.0)], [(-1.0, p), (-1.0, m)]][side], 1.0
    if el == "tri":
        gm_, gp = 0.5 * (1.0 - s), 0.5 * (1.0 + s)
        return [[(gp, 1.0 - gp), (gm_, 1.0 - gm_)], [(0.0, gp), (0.0, gm_)], [(gm_, 0.0), (gp, 0.0)]][side], 0.5
    if el == "tet":
        o, f = 1.0 / 6.0, 4.0 / 6.0
        return [[(f, o, o), (o, f, o), (o, o, f)], [(0.0, o, o), (0.0, o, f), (0.0, f, o)],
                [(o, 0.0, o), (f, 0.0, o), (o, 0.0, f)], [(o, o, 0.0), (o, f, 0.0), (f, o, 0.0)]][side], 1.0 / 6.0
    return [[(m, m, 1.0), (p, m, 1.0), (p, p, 1.0), (m, p, 1.0)],
            [(m, m, -1.0), (m, p, -1.0), (p, p, -1.0), (p, m, -1.0)],
            [(-1.0, m, m), (-1.0, m, p), (-1.0, p, p), (-1.0, p, m)],
            [(1.0, m, m), (1.0, p, m), (1.0, p, p), (1.0, m, p)],
            [(p, 1.0, m), (m, 1.0, m), (m, 1.0, p), (p, 1.0, p)],
            [(p, -1.0, m), (p, -1.0, p), (m, -1.0, p), (m, -1.0, m)]][side], 1.0


def _shape(el, pt):
    if el == "tri":
        x, y = pt
        return [1.0 - x - y, x, y], [[-1.0, 1.0, 0.0], [-1.0, 0.0, 1.0]]
    if el == "tet":
        x, y, z = pt
        return [1.0 - x - y - z, x, y, z], [[-1.0, 1.0, 0.0, 0.0], [-1.0, 0.0, 1.0, 0.0], [-1.0, 0.0, 0.0, 1.0]]
    if el == "quad":
        x, y = pt
        sg = [(-1, -1), (1, -1), (1, 1), (-1, 1)]
        sh = [0.25 * (1.0 + a * x) * (1.0 + b * y) for a, b in sg]
        return sh, [[0.25 * a * (1.0 + b * y) for a, b in sg], [0.25 * b * (1.0 + a * x) for a, b in sg]]
    x, y, z = pt
    sg = [(-1, -1, -1), (1, -1, -1), (1, 1, -1), (-1, 1, -1), (-1, -1, 1), (1, -1, 1), (1, 1, 1), (-1, 1, 1)]
    f = [(1.0 + a * x, 1.0 + b * y, 1.0 + c * z) for a, b, c in sg]
    sh = [0.125 * u * v * w for u, v, w in f]
    return sh, [[0.125 * s[0] * v * w for s, (u, v, w) in zip(sg, f)],
                [0.125 * s[1] * u * w for s, (u, v, w) in zip(sg, f)],
                [0.125 * s[2] * u * v for s, (u, v, w) in zip(sg, f)]]


def _area(el, pt, a):
    """Area vector of the side a side point lies on; a[i][j] = d x_i / d xi_j."""
    dim = len(pt)
    if dim == 2:
        (xx, xe), (yx, ye) = a[0], a[1]
        x, y = pt
        if el == "quad":
            if y == 1.0:
                return [-yx, xx]
            if y == -1.0:
                return [yx, -xx]
            return [ye, -xe] if x == 1.0 else [-ye, xe]
        if x == 0.0:
            return [-ye, xe]
        return [yx, -xx] if y == 0.0 else [ye - yx, xx - xe]

    def col(j):
        return [a[i][j] for i in range(3)]

    def cross(u, v):
        return [u[1] * v[2] - u[2] * v[1], u[2] * v[0] - u[0] * v[2], u[0] * v[1] - u[1] * v[0]]
    x, y, z = pt
    cx, cy, cz = col(0), col(1), col(2)
    if el == "hex":
        if abs(z) == 1.0:
            n, s = cross(cx, cy), z
        elif abs(y) == 1.0:
            n, s = cross(cz, cx), y
        else:
            n, s = cross(cy, cz), x
        return [s * v for v in n]
    if x == 0.0:
        return cross(cz, cy)
    if y == 0.0:
        return cross(cx, cz)
    if z == 0.0:
        return cross(cy, cx)
    return cross([p - q for p, q in zip(cy, cx)], [p - q for p, q in zip(cz, cx)])


def _geometry(el, X, pt):
    """sh, ds[d][i], J, inverse mapping b[j][d] = d xi_j / d x_d, and a; X: (e, nen, dim)."""
    sh, dl = _shape(el, pt)
    dim, nen = len(dl), len(sh)
    a = [[sum(dl[j][n] * X[:, n, i] for n in range(nen)) for j in range(dim)] for i in range(dim)]
    if dim == 2:
        J = a[0][0] * a[1][1] - a[1][0] * a[0][1]
        r = 1.0 / J
        b = [[r * a[1][1], r * -a[0][1]], [r * -a[1][0], r * a[0][0]]]
    else:
        (p, q, u), (v, w, x), (y, z, s) = a
        J = p * (w * s - z * x) - v * (q * s - z * u) + y * (q * x - w * u)
        r = 1.0 / J
        b = [[r * (w * s - z * x), r * (-q * s + z * u), r * (q * x - w * u)],
             [r * (-v * s + y * x), r * (p * s - y * u), r * (-p * x + v * u)],
             [r * (v * z - y * w), r * (-p * z + y * q), r * (p * w - v * q)]]
    ds = []
    for d in range(dim):
        row = []
        for i in range(nen):
            t = dl[0][i] * b[0][d]
            for j in range(1, dim):
                t = t + dl[j][i] * b[j][d]
            row.append(t)
        ds.append(row)
    return sh, ds, J, b, a


class _Plain:
    """The element integral of one case in 64 bits, with dense matrices."""

    def __init__(self, mesh, mat, setup, dev, theta=None):
        self.el = {(2, 3): "tri", (2, 4): "quad", (3, 4): "tet", (3, 8): "hex"}[(mesh.dim, mesh.nen)]
        self.dim, self.nen, self.nc = mesh.dim, mesh.nen, mat.nb_comp
        self.nd = self.dim + 1 + self.nc
        self.iT, self.iY = self.dim + 1, self.dim + 2
        self.g = [setup.desc.gravity[d] for d in range(self.dim)]
        self.scale = setup.desc.dc_scale_fact
        self.ch = []
        for c in range(self.nc):
            q = mat.desc.comp[c]
            gas = q.kind != 0
            if theta is None:
                self.ch.append(dict(gas=gas, rho=q.rho, mu=q.mu, cp=q.cp, cv=q.cv, kappa=q.kappa, alpha=q.alpha,
                                    beta=q.beta, R=q.R, gamma=q.gamma, D=q.chemical_diffusivity))
            else:
                d0, mu, cp = theta[3 * c], theta[3 * c + 1], theta[3 * c + 2]
                if gas:
                    R = 8.314462 / d0
                    self.ch.append(dict(gas=True, mu=mu, cp=cp, cv=cp - R, kappa=q.kappa, R=R, gamma=cp / (cp - R),
                                        D=q.chemical_diffusivity))
                else:
                    self.ch.append(dict(gas=False, rho=d0, mu=mu, cp=cp, kappa=q.kappa, alpha=q.alpha, beta=q.beta,
                                        D=q.chemical_diffusivity))
        one = torch.ones(1, dtype=torch.float64, device=dev)
        ref = self.mixture(setup.desc.p_ref * one, setup.desc.T_ref * one, [0.5 * one] * self.nc)
        u = self.conserved(ref, [setup.desc.v_ref[d] * one for d in range(self.dim)], setup.desc.T_ref * one,
                           [0.5 * one] * self.nc)
        self.uref = []
        for x in u:
            zero = x < 2.220446049250313e-16
            self.uref.append(torch.where(zero, torch.zeros_like(x), 1.0 / torch.where(zero, torch.ones_like(x), x)))

    def split(self, w):
        v = [w[1 + d] for d in range(self.dim)]
        Y = list(w[self.iY:])
        s = torch.zeros_like(w[0])
        for y in Y:
            s = s + y
        return w[0], v, w[self.iT], Y + [1.0 - s]

    def mixture(self, p, T, Y):
        z = torch.zeros_like(p)
        o = dict(mu=z, cp=z, cv=z, kappa=z)
        ir, c2, rc, ec, al, be = z, z, [], [], [], []
        for q, y in zip(self.ch, Y):
            if q["gas"]:
                r, b, a, s2, cv = p / (q["R"] * T), 1.0 / p, 1.0 / T, q["gamma"] * q["R"] * T, q["cv"] + z
            else:
                r, b, a = q["rho"] + z, q["beta"] + z, q["alpha"] + z
                s2 = 1.0 / (r * b)
                cv = q["cp"] - T * a * a / (r * b)
            ir = ir + y / r
            c2 = c2 + y / (r * r * s2)
            for k, x in (("mu", q["mu"]), ("cp", q["cp"]), ("cv", cv), ("kappa", q["kappa"])):
                o[k] = o[k] + y * x
            rc.append(r)
            ec.append(cv * T)
            al.append(a)
            be.append(b)
        rho = 1.0 / ir
        o.update(rho=rho, c=torch.sqrt(1.0 / c2) / rho, rc=rc, ec=ec)
        o["alpha"] = sum(y * a * rho / r for y, a, r in zip(Y, al, rc))
        o["beta"] = sum(y * b * rho / r for y, b, r in zip(Y, be, rc))
        return o

    def conserved(self, pr, v, T, Y):
        E = pr["cv"] * T + 0.5 * sum(x * x for x in v)
        rho = pr["rho"]
        return [rho] + [rho * x for x in v] + [rho * E] + [rho * y for y in Y[:-1]]

    def matrices(self, pr, p, v, T, Y):
        """DUDY, A_k, K_kl, S0 as (e, nd, nd) and the fluxes' scalars."""
        dim, nd, iT, iY, nc = self.dim, self.nd, self.iT, self.iY, self.nc
        n, rho = len(p), pr["rho"]
        E = pr["cv"] * T + 0.5 * sum(x * x for x in v)
        rp, rT = rho * pr["beta"], -rho * pr["alpha"]
        ep = (pr["beta"] * p - pr["alpha"] * T) / rho
        eT = pr["cp"] - p * pr["alpha"] / rho
        rY = [-rho * rho * (1.0 / pr["rc"][i] - 1.0 / pr["rc"][nc - 1]) for i in range(nc - 1)]
        eY = [pr["ec"][i] - pr["ec"][nc - 1] for i in range(nc - 1)]
        z = torch.zeros_like(p)
        r0 = [rp] + [z] * dim + [rT] + rY
        mE = [ep] + list(v) + [eT] + eY
        w = [torch.ones_like(p)] + list(v) + [E] + list(Y[:-1])
        D = [[w[r] * r0[c] for c in range(nd)] for r in range(nd)]
        for r in range(nd):
            if r == iT:
                D[r] = [x + rho * m for x, m in zip(D[r], mE)]
            elif r > 0:
                D[r][r] = D[r][r] + rho
        A = []
        for k in range(dim):
            M = [[v[k] * x for x in row] for row in D]
            for r in range(nd):
                M[r][1 + k] = M[r][1 + k] + rho * w[r] + (p if r == iT else 0.0)
            M[1 + k][0] = M[1 + k][0] + 1.0
            M[iT][0] = M[iT][0] + v[k]
            A.append(M)
        mu, lam = pr["mu"], -2.0 * pr["mu"] / 3.0
        K = {}
        for k in range(dim):
            for l in range(dim):
                M = [[z] * nd for _ in range(nd)]
                for j in range(dim):
                    for m in range(dim):
                        x = (mu if k == l and j == m else 0.0) + (mu if l == j and k == m else 0.0)
                        x = x + (lam if k == j and l == m else 0.0)
                        if torch.is_tensor(x):
                            M[1 + j][1 + m] = x
                            M[iT][1 + m] = M[iT][1 + m] + v[j] * x
                if k == l:
                    M[iT][iT] = pr["kappa"] + z
                    for i in range(nc - 1):
                        H = pr["ec"][i] + p / pr["rc"][i]
                        M[iY + i][iY + i] = rho * self.ch[i]["D"]
                        M[iT][iY + i] = rho * self.ch[i]["D"] * H
                K[k, l] = M
        S0 = [[z] * nd for _ in range(nd)]
        for d in range(dim):
            S0[iT][1 + d] = rho * self.g[d]

        def dense(M):
            return torch.stack([torch.stack([x if x.dim() else x.expand(n) for x in row], -1) for row in M], -2)
        return dense(D), [dense(M) for M in A], {kl: dense(M) for kl, M in K.items()}, dense(S0), E

    def length(self, G, v, dv):
        """Element size along the flow; its branches hang on rounding, so every step is one
        unfused operation in a fixed order."""
        dim = self.dim

        def norm(s):
            t = torch.zeros_like(s[0])
            for x in s:
                t = t + x * x
            return torch.sqrt(t)

        def form(s):
            r = torch.zeros_like(s[0])
            for i in range(dim):
                t = torch.zeros_like(r)
                for j in range(dim):
                    t = t + G[i][j] * s[j]
                r = r + s[i] * t
            return r

        def unit(s):
            n = norm(s)
            big = n > 2.220446049250313e-16
            n = torch.where(big, n, torch.ones_like(n))
            return [torch.where(big, x / n, x) for x in s]
        nv = norm(v)
        s0 = [x / nv for x in v]
        acc = []
        for i in range(dim):
            t = torch.zeros_like(nv)
            for j in range(dim):
                t = t + dv[i][j] * v[j]
            acc.append(t)
        ip = torch.zeros_like(nv)
        for i in range(dim):
            ip = ip + acc[i] * s0[i]
        s1 = unit([acc[i] - ip * s0[i] for i in range(dim)])
        al = [form(s0), form(s1)]
        if dim == 3:
            al.append(form(unit([s0[1] * s1[2] - s0[2] * s1[1], s1[0] * s0[2] - s1[2] * s0[0],
                                 s0[0] * s1[1] - s0[1] * s1[0]])))
        h = torch.zeros_like(nv)
        for a in al:
            h = h + torch.where(a != 0.0, 1.0 / torch.where(a != 0.0, a, torch.ones_like(a)), torch.zeros_like(a))
        return 2.0 * torch.sqrt(torch.abs(h))

    def tau(self, pr, D, v, h, trG, dt):
        nv = torch.sqrt(sum(x * x for x in v))
        c, rho = pr["c"], pr["rho"]
        use = torch.clamp(h / (2.0 * (nv + c)) + h / (2.0 * nv), max=dt * 0.5)
        tm = torch.minimum(use, h * h * rho / (12.0 * pr["mu"]))
        td = [use] + [tm] * self.dim + [torch.minimum(use, h * h * rho * pr["cv"] / (12.0 * pr["kappa"]))]
        td += [torch.minimum(use, h * h / (12.0 * self.ch[i]["D"])) for i in range(self.nc - 1)]
        # rows and columns brought to a like size for the inverse, exactly (powers of two)
        with torch.no_grad():
            col = torch.exp2(-torch.round(torch.log2(D.abs().amax(-2, keepdim=True))))
            row = torch.exp2(-torch.round(torch.log2((D * col).abs().amax(-1, keepdim=True))))
        inv = torch.linalg.inv(D * col * row) * col.transpose(-1, -2) * row.transpose(-1, -2)
        t = inv * torch.stack(td, -1).unsqueeze(-2)
        slow = nv / c < 0.1
        t00 = torch.where(slow, 1.0 / (1.0 / t[:, 0, 0] + 1.0 / (rho * t[:, 1, 1] * trG)), t[:, 0, 0])
        first = torch.cat([t00.unsqueeze(-1), torch.where(slow.unsqueeze(-1), torch.zeros_like(t[:, 0, 1:]), t[:, 0, 1:])], -1)
        t = torch.cat([first.unsqueeze(-2), t[:, 1:]], -2)
        return torch.where((nv < 2.220446049250313e-16).reshape(-1, 1, 1), torch.zeros_like(t), t)

    def sharp(self, dU, AdI, S, U, ds):
        """Discontinuity capturing viscosity, sharpness 2."""
        s = torch.sqrt(sum(u[:, 0] * u[:, 0] for u in dU))
        safe = torch.where(s < 2.220446049250313e-16, torch.ones_like(s), s)
        Jv = [u[:, 0] / safe for u in dU]
        h = sum(torch.abs(sum(Jv[d] * ds[d][i] for d in range(self.dim))) for i in range(self.nen))
        on = (s >= 2.220446049250313e-16) & (h > 2.220446049250313e-16)
        h = 1.0 / torch.where(on, h, torch.ones_like(h))
        ur = torch.stack([x.expand(len(s)) for x in self.uref], -1)
        Z = torch.sqrt(((ur * (AdI - S)) ** 2).sum(-1))
        Un = torch.sqrt(((ur * U) ** 2).sum(-1))
        return torch.where(on, self.scale * (Z * h * h / Un), torch.zeros_like(s))

    def interior(self, X, Ie, Pe, dt, want_m):
        """r (= the rhs' share) and m of (e, nen, nd) states."""
        dim, nen, nd = self.dim, self.nen, self.nd
        pts, W = _tables(self.el)
        r = torch.zeros(len(X), nen, nd, dtype=X.dtype, device=X.device)
        m = torch.zeros(len(X), nen, nd, nen, nd, dtype=X.dtype, device=X.device) if want_m else None
        for pt in pts:
            sh, ds, J, b, _ = _geometry(self.el, X, pt)
            jx = J * W

            def at(S, wts):
                out = []
                for j in range(nd):
                    t = torch.zeros_like(J)
                    for i in range(nen):
                        t = t + wts[i] * S[:, i, j]
                    out.append(t)
                return out
            pP, vP, TP, YP = self.split(at(Pe, sh))
            UP = torch.stack(self.conserved(self.mixture(pP, TP, YP), vP, TP, YP), -1)
            Pq, Iq = torch.stack(at(Pe, sh), -1), torch.stack(at(Ie, sh), -1)
            p, v, T, Y = self.split(at(Ie, sh))
            dI = [torch.stack(at(Ie, ds[d]), -1) for d in range(dim)]
            pr = self.mixture(p, T, Y)
            D, A, K, S0, E = self.matrices(pr, p, v, T, Y)
            U = torch.stack(self.conserved(pr, v, T, Y), -1)
            rho = pr["rho"]
            S = torch.zeros_like(U)
            Sl = [torch.zeros_like(p)] + [rho * g for g in self.g] + [rho * sum(g * x for g, x in zip(self.g, v))]
            S = torch.stack(Sl + [torch.zeros_like(p)] * (self.nc - 1), -1)
            G = [[sum(b[k][i] * b[k][j] for k in range(dim)) for j in range(dim)] for i in range(dim)]
            h = self.length(G, v, [[dI[d][:, 1 + a] for d in range(dim)] for a in range(dim)])
            t = self.tau(pr, D, v, h, sum(G[d][d] for d in range(dim)), dt)

            def mv(M, x):
                return (M @ x.unsqueeze(-1)).squeeze(-1)
            AdI = sum(mv(A[d], dI[d]) for d in range(dim))
            Res = mv(D, (Iq - Pq) / dt) + AdI - S
            dU = [mv(D, dI[d]) for d in range(dim)]
            nu = self.sharp(dU, AdI, S, U, ds)
            tR = mv(t, Res)
            w0 = (U - UP) / dt - S - mv(S0, tR)
            phi = []
            for k in range(dim):
                Fa = v[k].unsqueeze(-1) * U
                Fa = Fa + torch.stack([torch.zeros_like(p)] + [p if j == k else torch.zeros_like(p) for j in range(dim)] +
                                      [p * v[k]] + [torch.zeros_like(p)] * (self.nc - 1), -1)
                phi.append(sum(mv(K[k, l], dI[l]) for l in range(dim)) - Fa + nu.unsqueeze(-1) * dU[k] + mv(A[k], tR))
            for i in range(nen):
                x = sh[i] * w0
                for k in range(dim):
                    x = x + ds[k][i].unsqueeze(-1) * phi[k]
                r[:, i] = r[:, i] - jx.unsqueeze(-1) * x
            if not want_m:
                continue
            WA = [sum(ds[k][i].reshape(-1, 1, 1) * A[k] for k in range(dim)) for i in range(nen)]
            RM = [sh[i] * D / dt + WA[i] - sh[i] * S0 for i in range(nen)]
            for ib in range(nen):
                L = (WA[ib] - sh[ib] * S0) @ t
                Xb = sh[ib] * D / dt - WA[ib] - sh[ib] * S0
                gK = [sum(ds[k][ib].reshape(-1, 1, 1) * K[k, l] for k in range(dim)) +
                      (ds[l][ib] * nu).reshape(-1, 1, 1) * D for l in range(dim)]
                for ia in range(nen):
                    B = L @ RM[ia] + sh[ia] * Xb
                    for l in range(dim):
                        B = B + ds[l][ia].reshape(-1, 1, 1) * gK[l]
                    m[:, ib, :, ia, :] += jx.reshape(-1, 1, 1) * B
        return r, m

    def boundary(self, X, Ie, side, wall, want_m):
        """The boundary integral over one side of each element; on the wall (`wall`) the heat
        flux and the first species' flux are prescribed as zero (p0_policy)."""
        dim, nen, nd, iT, iY = self.dim, self.nen, self.nd, self.iT, self.iY
        pts, W = _side_points(self.el, side)
        r = torch.zeros(len(X), nen, nd, dtype=X.dtype, device=X.device)
        m = torch.zeros(len(X), nen, nd, nen, nd, dtype=X.dtype, device=X.device) if want_m else None
        keep = (~wall).to(X.dtype)
        for pt in pts:
            sh, ds, J, b, a = _geometry(self.el, X, pt)
            n = [W * x for x in _area(self.el, pt, a)]

            def at(wts, S=Ie):
                return torch.stack([sum(wts[i] * S[:, i, j] for i in range(nen)) for j in range(nd)], -1)
            Iq = at(sh)
            p, v, T, Y = self.split(list(Iq.unbind(-1)))
            pr = self.mixture(p, T, Y)
            D, A, K, S0, E = self.matrices(pr, p, v, T, Y)
            U = torch.stack(self.conserved(pr, v, T, Y), -1)
            dI = [at(ds[d]) for d in range(dim)]
            mu, lam, z = pr["mu"], -2.0 * pr["mu"] / 3.0, torch.zeros_like(p)
            div = sum(dI[d][:, 1 + d] for d in range(dim))
            flux = torch.zeros_like(U)
            for k in range(dim):
                Fa = v[k].unsqueeze(-1) * U + torch.stack(
                    [z] + [p if j == k else z for j in range(dim)] + [p * v[k]] + [z] * (self.nc - 1), -1)
                ts = [mu * (dI[k][:, 1 + j] + dI[j][:, 1 + k]) + (lam * div if j == k else 0.0) for j in range(dim)]
                Jf, HJ = [], z
                for i in range(self.nc - 1):
                    x = pr["rho"] * self.ch[i]["D"] * dI[k][:, iY + i]
                    if i == 0:
                        x = x * keep
                    Jf.append(x)
                    HJ = HJ + (pr["ec"][i] + p / pr["rc"][i]) * x
                q = -pr["kappa"] * dI[k][:, iT] * keep
                Fd = torch.stack([z] + ts + [sum(t * x for t, x in zip(ts, v)) - q - HJ] + Jf, -1)
                flux = flux + n[k].unsqueeze(-1) * (Fa - Fd)
            for i in range(nen):
                r[:, i] = r[:, i] - sh[i] * flux
            if not want_m:
                continue
            BA = sum(n[k].reshape(-1, 1, 1) * A[k] for k in range(dim))
            BK = []
            for l in range(dim):
                x = sum(n[k].reshape(-1, 1, 1) * K[k, l] for k in range(dim))
                mask = torch.ones_like(x)
                mask[:, iT, iT] = keep
                if self.nc > 1:
                    mask[:, iY, iY] = keep
                    mask[:, iT, iY] = keep
                BK.append(x * mask)
            for ia in range(nen):
                B = sh[ia] * BA - sum(ds[l][ia].reshape(-1, 1, 1) * BK[l] for l in range(dim))
                for ib in range(nen):
                    m[:, ib, :, ia, :] += sh[ib] * B
        return r, m


def _blocked(mesh, setup, nd):
    mask = torch.zeros(len(mesh.node_flag), nd, dtype=torch.bool)
    flag = torch.from_numpy(mesh.node_flag.astype(np.int64))
    for f in range(32):
        for k in range(nd):
            if setup.desc.dirichlet_mask[f] >> k & 1:
                mask[:, k] |= flag == f
    return mask


def _passes(plain, mesh, dev, chunk):
    """(node ids, call) of each batch of element integrals: the interior, then each
    boundary element's flagged sides."""
    conn = torch.from_numpy(mesh.conn.astype(np.int64)).to(dev)
    X = torch.from_numpy(mesh.coords).to(dev)
    for lo in range(0, len(conn), chunk):
        c = conn[lo:lo + chunk]
        yield c, lambda Ie, Pe, dt, wm, c=c: plain.interior(X[c], Ie, Pe, dt, wm)
    bd = mesh.bd_sides
    for e in np.array_split(np.unique(bd[:, 0]), max(1, len(np.unique(bd[:, 0])) // chunk)):
        c = conn[torch.from_numpy(e.astype(np.int64)).to(dev)]

        def sides(Ie, Pe, dt, wm, c=c, e=e):
            r = torch.zeros(len(c), plain.nen, plain.nd, dtype=torch.float64, device=dev)
            m = torch.zeros(len(c), plain.nen, plain.nd, plain.nen, plain.nd, dtype=torch.float64, device=dev) if wm else None
            sel = bd[np.isin(bd[:, 0], e)]
            for s in range(len(syn.SIDES[(mesh.dim, mesh.nen)])):
                q = sel[sel[:, 1] == s]
                if not len(q):
                    continue
                at = torch.from_numpy(np.searchsorted(e, q[:, 0])).to(dev)
                wall = torch.from_numpy(q[:, 2] == WALL).to(dev)
                rs, ms = plain.boundary(X[c[at]], Ie[at], s, wall, wm)
                r = r.index_add(0, at, rs)
                if wm:
                    m.index_add_(0, at, ms)
            return r, m
        yield c, sides


def _graph(mesh, dev):
    conn = torch.from_numpy(mesh.conn.astype(np.int64)).to(dev)
    n = len(mesh.coords)
    keys = torch.unique((conn.unsqueeze(2) * n + conn.unsqueeze(1)).reshape(-1))
    rp = torch.zeros(n + 1, dtype=torch.int64, device=dev)
    rp[1:] = torch.cumsum(torch.bincount(keys // n, minlength=n), 0)
    return keys, rp


def _exact_assembly(case, seed, want_m):
    mesh, mat, setup, I, P = _inputs(case, seed)
    dev = DEVICE
    plain = _Plain(mesh, mat, setup, dev)
    nd, nen, n = plain.nd, plain.nen, len(mesh.coords)
    I, P = (torch.from_numpy(x).to(dev).reshape(n, nd) for x in (I, P))
    blocked = _blocked(mesh, setup, nd).to(dev)
    rhs = torch.zeros(n * nd, dtype=torch.float64, device=dev)
    dofs = torch.arange(nd, device=dev)
    if want_m:
        keys, rp = _graph(mesh, dev)
        vals = torch.zeros(len(keys) * nd * nd, dtype=torch.float64, device=dev)
    for c, call in _passes(plain, mesh, dev, max(2000, 60000000 // (nen * nd) ** 2)):
        r, m = call(I[c], P[c], DT, want_m)
        off = blocked[c]
        r = torch.where(off, torch.zeros_like(r), r)
        rhs.index_add_(0, (c.unsqueeze(-1) * nd + dofs).reshape(-1), r.reshape(-1))
        if not want_m:
            continue
        N = nen * nd
        flat = m.reshape(-1, N, N)
        avg = (1.0 + torch.diagonal(flat, dim1=1, dim2=2).sum(-1)) / N
        o = off.reshape(-1, N, 1)
        flat = torch.where(o, avg.reshape(-1, 1, 1) * torch.eye(N, dtype=torch.float64, device=dev), flat)
        slot = torch.searchsorted(keys, (c.unsqueeze(2) * n + c.unsqueeze(1)).reshape(-1)).reshape(len(c), nen, nen)
        slot = slot - rp[c].unsqueeze(2)
        deg = (rp[c + 1] - rp[c]) * nd
        at = rp[c].reshape(-1, nen, 1, 1, 1) * nd * nd + dofs.reshape(1, 1, nd, 1, 1) * deg.reshape(-1, nen, 1, 1, 1) + \
            slot.reshape(-1, nen, 1, nen, 1) * nd + dofs
        vals.index_add_(0, at.reshape(-1), flat.reshape(-1))
    return (vals, rhs) if want_m else (None, rhs)


def _exact_vjp(case, seed):
    mesh, mat, setup, I, P = _inputs(case, seed)
    dev = DEVICE
    nd, n, nc = _dof_count(case), len(mesh.coords), case["comps"]
    I, P = (torch.from_numpy(x).to(dev).reshape(n, nd) for x in (I, P))
    lam = torch.from_numpy(_lambda(case, seed, n * nd)).to(dev).reshape(n, nd)
    lam = torch.where(_blocked(mesh, setup, nd).to(dev), torch.zeros_like(lam), lam)
    theta = []
    for c in range(nc):
        q = mat.desc.comp[c]
        theta += [8.314462 / q.R if q.kind != 0 else q.rho, q.mu, q.cp]
    theta = torch.tensor(theta, dtype=torch.float64, device=dev, requires_grad=True)
    g = torch.zeros(n, nd, dtype=torch.float64, device=dev)
    gp = torch.zeros(3 * nc, dtype=torch.float64, device=dev)
    chunk = 20000
    plain = _Plain(mesh, mat, setup, dev, theta=theta.unbind(0))
    for c, call in _passes(plain, mesh, dev, chunk):
        Ie = I[c].detach().requires_grad_(True)
        r, _ = call(Ie, P[c], DT, False)
        gi, gt = torch.autograd.grad((r * lam[c]).sum(), (Ie, theta), retain_graph=True)
        g.index_add_(0, c.reshape(-1), gi.reshape(-1, nd))
        gp += gt
    return {"g_state": g.reshape(-1), "g_params": gp}


def exact(case, seed):
    """None for the magma mixtures (table look-ups and a viscosity model), the linear solve
    and the time step (iterations to a tolerance: a direct solve takes too long)."""
    call = case["call"]
    if case.get("magma") or call in ("solve", "time_step"):
        return None
    if call in ("assemble", "assemble_host"):
        vals, rhs = _exact_assembly(case, seed, True)
        return {"vals": vals, "rhs": rhs}
    if call == "residual":
        return {"rhs": _exact_assembly(case, seed, False)[1]}
    if case["mode"] == "exact":
        return _exact_vjp(case, seed)
    vals, _ = _exact_assembly(dict(case, call="vjp"), seed, True)
    mesh = _mesh_of(case)
    dev = vals.device
    keys, rp = _graph(mesh, dev)
    nd, n = _dof_count(case), len(mesh.coords)
    lam = torch.from_numpy(_lambda(case, seed, n * nd)).to(dev)
    row, col = keys // n, keys % n
    deg = (rp[1:] - rp[:-1])[row] * nd
    slot = torch.arange(len(keys), device=dev) - rp[row]
    g = torch.zeros(n * nd, dtype=torch.float64, device=dev)
    for r in range(nd):
        for c in range(nd):
            a = vals[rp[row] * nd * nd + r * deg + slot * nd + c]
            g.index_add_(0, col * nd + c, a * lam[row * nd + r])
    return {"g_state": g}
