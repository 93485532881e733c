"""The work that users of goma_gb300 have it do, as cases that can be timed.

Four kinds, each through the package's public Python entry points:

fill    one residual (+ Jacobian) assembly on device arrays
        (GomaNewton.matrix_fill_full_device), the call of every Newton step;
solve   one Krylov solve of a Newton step on device arrays
        (GomaNewton.linear_solve_device): ILU(0) of the scaled matrix, then
        GMRES to the given tolerance;
newton  a whole solve_nonlinear_problem on host arrays, the drop-in call;
mlp     the continuation predictor's network: a short online training and one
        prediction over all rows (GpuMLP.train, GpuMLP.forward).

Problems are the repository's own configurations (lid-driven cavity, Carreau
step channel, Boussinesq cube, reacting channel, batches of independent
cavities), on affine or perturbed meshes, at smooth states drawn from the
seed.  `exact` restates the element equations in plain torch (the Jacobian by
forward-mode differentiation), the sparsity and the Dirichlet rows.
"""
import math

import numpy as np
import torch

from goma_gb300 import problem as pb
from goma_gb300.mlp import GpuMLP
from goma_gb300.newton import GomaNewton

# ------------------------------------------------------------------ the cases


def listed():
    return [
        # one Newton assembly of the 32 x 32 lid-driven cavity: a few
        # microseconds of work, so launches and latency count
        dict(name="fill_cavity_32", kind="fill", problem="cavity", nx=32, ny=32, nz=0, amp=0.0,
             jac=True, transient=False),
        # an assembly of the 96 x 32 Carreau-Yasuda step channel, as in every
        # step of the Reynolds-number continuation
        dict(name="fill_carreau_96x32", kind="fill", problem="carreau", nx=96, ny=32, nz=0,
             amp=0.0, jac=True, transient=False),
        # a sweep of independent cavities held as one disjoint union with
        # per-element densities: a large 2-D assembly
        dict(name="fill_batch_64", kind="fill", problem="batch", nx=16, ny=64, nz=64, amp=0.0,
             jac=True, transient=False, meshes=0),
        # the Boussinesq cube, the headline assembly
        dict(name="fill_cube_24", kind="fill", problem="boussinesq", nx=24, ny=24, nz=24,
             amp=0.0, jac=True, transient=False),
        # a time step's assembly on a perturbed, ragged box
        dict(name="fill_box_17x11x9_transient", kind="fill", problem="boussinesq", nx=17, ny=11,
             nz=9, amp=0.1, jac=True, transient=True),
        # the reacting channel: flow, energy and two species
        dict(name="fill_reacting_16x16x8", kind="fill", problem="reacting", nx=16, ny=16, nz=8,
             amp=0.0, jac=True, transient=False),
        # the linear solve of one Newton step of the Boussinesq cube in FP64
        dict(name="solve_cube_16", kind="solve", problem="boussinesq", nx=16, ny=16, nz=16,
             amp=0.0, krylov=150, tol=1e-8),
        # the linear solve of one Newton step of the Carreau channel
        dict(name="solve_carreau_96x32", kind="solve", problem="carreau", nx=96, ny=32, nz=0,
             amp=0.0, krylov=150, tol=1e-8),
        # the linear solve of a batch: one GMRES per member, run together
        dict(name="solve_batch_32", kind="solve", problem="batch", nx=16, ny=32, nz=32, amp=0.0,
             krylov=30, tol=1e-8, meshes=0),
        # the whole Newton solve of the 32 x 32 cavity from rest, FP64
        dict(name="newton_cavity_32", kind="newton", problem="cavity", nx=32, ny=32, nz=0,
             amp=0.0, fp32_prec=False, krylov=60, tol=1e-10),
        # a whole Newton solve of a Boussinesq box from rest with the ILU(0)
        # factorised and swept in FP32
        dict(name="newton_cube_11_fp32prec", kind="newton", problem="boussinesq", nx=11, ny=11,
             nz=11, amp=0.0, fp32_prec=True, krylov=150, tol=1e-10),
        # the predictor's network in an online step of the 96 x 32 channel:
        # the rows of all its unknowns, width 256
        dict(name="mlp_34K_256x3", kind="mlp", rows=34306, width=256, hidden=3, batch=4096,
             steps=10),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fill", "fill", "fill", "solve", "solve", "newton", "mlp"])
    if kind == "mlp":
        return dict(kind=kind, rows=_logint(rng, 1000, 34306), width=rng.choice([64, 128, 200, 256]),
                    hidden=rng.randint(2, 3), batch=_logint(rng, 500, 4096),
                    steps=rng.randint(4, 10))
    if kind == "fill":
        p = rng.choice(["cavity", "carreau", "batch", "boussinesq", "boussinesq", "reacting"])
        c = dict(kind=kind, problem=p, nx=0, ny=0, nz=0, amp=rng.choice([0.0, 0.05, 0.1]),
                 jac=rng.random() < 0.8, transient=rng.random() < 0.3)
        if p in ("cavity", "carreau"):
            c.update(nx=_logint(rng, 5, 128), ny=_logint(rng, 5, 64))
        elif p == "batch":
            lo = rng.randint(5, 20)
            c.update(nx=lo, ny=rng.randint(lo + 1, 48), nz=_logint(rng, 3, 64),
                     meshes=rng.randint(1, 999))
        elif p == "boussinesq":
            c.update(nx=_logint(rng, 3, 24), ny=_logint(rng, 3, 24), nz=_logint(rng, 3, 24))
        else:
            c.update(nx=_logint(rng, 3, 16), ny=_logint(rng, 3, 16), nz=_logint(rng, 3, 8))
        return c
    if kind == "solve":
        p = rng.choice(["cavity", "carreau", "batch", "boussinesq"])
        c = dict(kind=kind, problem=p, nx=0, ny=0, nz=0, amp=rng.choice([0.0, 0.05]),
                 krylov=rng.choice([100, 150, 200]), tol=1e-8)
        if p in ("cavity", "carreau"):
            c.update(nx=_logint(rng, 8, 80), ny=_logint(rng, 8, 32))
        elif p == "batch":
            lo = rng.randint(8, 16)
            c.update(nx=lo, ny=rng.randint(lo + 1, 28), nz=rng.randint(3, 32), krylov=30,
                     meshes=rng.randint(1, 999))
        else:
            c.update(nx=_logint(rng, 4, 15), ny=_logint(rng, 4, 15), nz=_logint(rng, 4, 15))
        return c
    p = rng.choice(["cavity", "boussinesq"])
    c = dict(kind=kind, problem=p, nx=0, ny=0, nz=0, amp=rng.choice([0.0, 0.05]),
             fp32_prec=rng.random() < 0.5, krylov=rng.choice([60, 150]), tol=1e-10)
    if p == "cavity":
        c.update(nx=_logint(rng, 8, 36), ny=_logint(rng, 8, 36))
    else:
        c.update(nx=_logint(rng, 3, 10), ny=_logint(rng, 3, 10), nz=_logint(rng, 3, 10))
    return c


# ------------------------------------------------- a problem, in plain numpy

# grid offsets of the local nodes in the Exodus order
_QUAD9 = np.array([[0, 0], [2, 0], [2, 2], [0, 2], [1, 0], [2, 1], [1, 2], [0, 1], [1, 1]])
_HEX27 = np.array(
    [[0, 0, 0], [2, 0, 0], [2, 2, 0], [0, 2, 0], [0, 0, 2], [2, 0, 2], [2, 2, 2], [0, 2, 2],
     [1, 0, 0], [2, 1, 0], [1, 2, 0], [0, 1, 0], [0, 0, 1], [2, 0, 1], [2, 2, 1], [0, 2, 1],
     [1, 0, 2], [2, 1, 2], [1, 2, 2], [0, 1, 2], [1, 1, 1], [1, 1, 0], [1, 1, 2], [0, 1, 1],
     [2, 1, 1], [1, 0, 1], [1, 2, 1]])
_T, _P, _Y = 3, 9, 100  # variable ids of the Dirichlet cards beside the velocities 0, 1, 2


def _box(n, ext, amp, rng):
    """Coordinates, connectivity and grid indices of a structured box of n[d]
    elements a side; with amp > 0 interior nodes are moved."""
    dim = len(n)
    pts = [2 * k + 1 for k in n]
    idx = np.stack(np.meshgrid(*[np.arange(p) for p in reversed(pts)], indexing="ij"), -1)
    idx = idx.reshape(-1, dim)[:, ::-1]
    h = np.array([e / (p - 1) for e, p in zip(ext, pts)])
    X = idx * h
    inner = np.all((idx > 0) & (idx < np.array(pts) - 1), axis=1)
    X = X + amp * h * rng.uniform(-1, 1, X.shape) * inner[:, None]
    el = np.stack(np.meshgrid(*[np.arange(k) for k in reversed(n)], indexing="ij"), -1)
    el = el.reshape(-1, dim)[:, ::-1]
    strides = np.cumprod([1] + pts[:-1])
    local = _QUAD9 if dim == 2 else _HEX27
    conn = ((2 * el[:, None, :] + local[None]) * strides).sum(-1)
    return X, conn.astype(np.int32), idx, pts


def _wall_cards(p, idx, pts, X):
    """Dirichlet cards (variable, node list, value) in deck order: later win."""
    lo = [idx[:, d] == 0 for d in range(len(pts))]
    hi = [idx[:, d] == pts[d] - 1 for d in range(len(pts))]
    nz = lambda m: np.nonzero(m)[0].astype(np.int32)  # noqa: E731
    if p in ("cavity", "batch"):
        cards = [(v, s, 0.0) for s in (lo[1], hi[0], lo[0]) for v in (0, 1)]
        cards += [(0, hi[1], 1.0), (1, hi[1], 0.0)]
    elif p == "carreau":
        low, up = lo[0] & (2 * idx[:, 1] <= pts[1] - 1), lo[0] & (2 * idx[:, 1] >= pts[1] - 1)
        cards = [(v, s, 0.0) for s in (lo[1], hi[1], low) for v in (0, 1)]
        cards += [(0, up, 1.0), (1, up, 0.0)]
    elif p == "boussinesq":
        cards = [(v, s, 0.0) for d in range(3) for s in (lo[d], hi[d]) for v in (0, 1, 2)]
        cards += [(_T, lo[0], 1.0), (_T, hi[0], 0.0)]
    else:
        cards = [(0, lo[0], 1.0), (1, lo[0], 0.0), (2, lo[0], 0.0)]
        cards += [(v, s, 0.0) for s in (lo[1], hi[1], lo[2], hi[2]) for v in (0, 1, 2)]
        cards += [(_T, lo[0], 2.0), (_T, lo[1], 1.0), (_T, hi[1], 1.0), (_Y, lo[0], 1.0),
                  (_Y + 1, lo[0], 0.0)]
    return [(v, nz(m), val) for v, m, val in cards]


def _describe(c, seed):
    """One problem and state: mesh, material, cards, per-element densities,
    the unknowns' numbering and the vectors x and xdot."""
    rng = np.random.default_rng([seed, 7])
    p, m = c["problem"], {}
    f = float(rng.uniform(0.9, 1.1))
    energy, nspec, datum = False, 0, -1
    if p == "batch":
        # nz members; the meshes are the case's, the Reynolds numbers the seed's
        ns = np.random.default_rng(c["meshes"]).integers(c["nx"], c["ny"] + 1, c["nz"])
        re = np.exp(rng.uniform(math.log(10.0), math.log(400.0), c["nz"]))
    else:
        ns, re = [None], [1.0]
    n = (c["nx"], c["ny"], c["nz"]) if c["nz"] and p != "batch" else (c["nx"], c["ny"])
    ext = {"carreau": (3.0, 1.0), "reacting": (2.0, 2.0, 1.0)}.get(p, (1.0,) * len(n))
    Xs, conns, cards, rho, nodes, shifts = [], [], [], [], 0, []
    for k, r in zip(ns, re):
        X, conn, idx, pts = _box(n if k is None else (int(k), int(k)), ext, c["amp"], rng)
        one = _wall_cards(p, idx, pts, X)
        if p == "batch":
            one.append((_P, conn[0, 8:9], 0.0))
        cards += [(v, s + nodes, val) for v, s, val in one]
        Xs.append(X)
        shifts.append(np.full(len(X), 1.5 * len(shifts)))
        conns.append(conn + nodes)
        rho.append(np.full(len(conn), r))
        nodes += len(X)
    X, conn = np.concatenate(Xs), np.ascontiguousarray(np.concatenate(conns), np.int32)
    if p == "cavity":
        m, datum = dict(density=100.0 * f, viscosity=1.0), 0
    elif p == "batch":
        m = dict(density=1.0, viscosity=1.0)
    elif p == "carreau":
        m = dict(density=100.0 * f, mu0=1.0, mu_inf=0.01, lam=1.0, aexp=2.0, nexp=0.5)
    elif p == "boussinesq":
        energy, datum = True, 0
        m = dict(density=1.0, viscosity=0.71, heat_capacity=1.0, conductivity=1.0,
                 source=(0.0, 0.0, -0.71e4 * f), beta=1.0, tref=0.5)
    else:
        energy, nspec = True, 2
        m = dict(density=1.0, viscosity=0.01, heat_capacity=1.0, conductivity=0.01,
                 diffusivity=1e-3, k0=5.0 * f, activation=2.0)
    dim = X.shape[1]
    nv, npres = dim + energy + nspec, dim + 1
    cent = conn[:, 8 if dim == 2 else 20]
    per = np.full(len(X), nv)
    per[cent] += npres
    fu = np.concatenate([[0], np.cumsum(per)])
    N = int(fu[-1])
    # a smooth state: a few waves per field, O(1) velocities
    x, xdot = np.zeros(N), np.zeros(N)
    for out, size in ((x, 1.0), (xdot, 0.5)):
        for v in range(nv):
            s = np.zeros(len(X))
            for _ in range(3):
                k = rng.integers(1, 4, dim)
                s += rng.uniform(-1, 1) * np.prod(np.sin(math.pi * k * X + rng.uniform(0, 6)), 1)
            if v == dim and energy:
                s = (1.5 if nspec else 0.5) + 0.3 * s
            if v > dim:
                s = 0.5 + 0.2 * s
            out[fu[:-1] + v] = size * 0.5 * s if v < dim else s * (size if out is x else 0.5)
        for q in range(npres):
            out[fu[cent] + nv + q] = size * rng.uniform(-0.1, 0.1, len(cent))
    dirichlet = {}
    for v, s, val in cards:
        off = {_T: dim, _P: nv}.get(v, v if v < 3 else dim + energy + v - _Y)
        for i in fu[s] + off:
            dirichlet[int(i)] = val
    if datum >= 0:
        dirichlet[int(fu[cent[datum]] + nv)] = 0.0
    di = np.array(sorted(dirichlet), np.int64)
    x[di] = [dirichlet[int(i)] for i in di]
    return dict(dim=dim, X=X + np.concatenate(shifts)[:, None] * (np.arange(dim) == 0), conn=conn,
                cards=cards, m=m, energy=energy, nspec=nspec, datum=datum, fu=fu, N=N, nv=nv,
                npres=npres, cent=cent, rho=np.concatenate(rho) if p == "batch" else None, x=x,
                xdot=xdot, di=di, p=p, dt=0.05, theta=0.0)


def _newton_of(d):
    """The context that a user's program keeps for the problem d."""
    m, sets, bcs = d["m"], [], []
    for v, s, val in d["cards"]:
        sets.append(s)
        bcs.append((v, len(sets), val))
    mat = pb.Material(density=m["density"], viscosity=m.get("viscosity", 1.0),
                      heat_capacity=m.get("heat_capacity", 1.0),
                      conductivity=m.get("conductivity", 1.0))
    if d["p"] == "carreau":
        mat.viscosity_model = pb.VISC_CARREAU
        mat.mu0, mat.mu_inf, mat.lam = m["mu0"], m["mu_inf"], m["lam"]
        mat.aexp, mat.nexp = m["aexp"], m["nexp"]
    if "source" in m:
        mat.momentum_source_model = pb.SOURCE_BOUSSINESQ
        mat.momentum_source, mat.volume_expansion = m["source"], m["beta"]
        mat.reference_temperature = m["tref"]
    if d["nspec"]:
        mat.diffusivity = (m["diffusivity"],) * 2
        mat.species_source = tuple((pb.SPECIES_SOURCE_ARRHENIUS,
                                    (m["k0"], m["activation"], nu, 0.0)) for nu in (-1.0, 1.0))
    mesh = pb.Mesh(d["dim"], d["X"], d["conn"], sets)
    gn = GomaNewton(pb.Problem(mesh, mat, d["energy"], bcs, (d["datum"], 0.0), d["nspec"]))
    if d["rho"] is not None:
        gn.set_element_density(d["rho"])
    return gn


# ----------------------------------------------------------- prepare and run


def _mlp_data(c, seed):
    """Rows of the predictor's training set: rates, their changes, a field
    type and a position in, the next rate change out."""
    rng = np.random.default_rng([seed, 11])
    n = c["rows"]
    x = np.concatenate([rng.standard_normal((n, 2)), np.eye(3)[rng.integers(0, 3, n)],
                        rng.uniform(0, 1, (n, 2)), rng.uniform(-1, 1, (n, 1))], 1)
    t = (0.5 * x[:, :1] * np.sin(3 * x[:, 5:6]) + 0.3 * x[:, 1:2] + 0.1 * rng.standard_normal((n, 1)))
    mask = (rng.uniform(0, 1, (n, 1)) < 0.9).astype(np.float32)
    widths = [x.shape[1]] + [c["width"]] * c["hidden"] + [1]
    params = []
    for a, b in zip(widths[:-1], widths[1:]):
        params += [rng.uniform(-1, 1, a * b) * math.sqrt(6.0 / (a + b)), rng.uniform(-.1, .1, b)]
    return x.astype(np.float32), t.astype(np.float32), mask, widths, \
        np.concatenate(params).astype(np.float32)


def prepare(case, seed):
    c = case
    if c["kind"] == "mlp":
        x, t, mask, widths, params = _mlp_data(c, seed)
        net = GpuMLP(widths[0], c["width"], c["hidden"], 1, seed=seed)
        dev = [torch.from_numpy(a).cuda() for a in (x, t, mask)]
        torch.cuda.synchronize()
        return dict(c=c, net=net, data=dev, params=params, seed=seed)
    d = _describe(c, seed)
    gn = _newton_of(d)
    s = dict(c=c, gn=gn, d=d)
    if c["kind"] == "newton":
        s["x0"] = gn.dirichlet_init(0.01 * d["x"])
        return s
    vec = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    s["x"], s["xdot"] = vec(d["x"]), vec(d["xdot"])
    s["R"] = torch.zeros(gn.N, dtype=torch.float64, device="cuda")
    with_vals = c["kind"] == "solve" or c["jac"]
    s["vals"] = torch.zeros(gn.nnz if with_vals else 0, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    if c["kind"] == "solve":
        s["dx"] = torch.zeros_like(s["R"])
        gn.matrix_fill_full_device(s["x"].data_ptr(), s["R"].data_ptr(), s["vals"].data_ptr())
        gn.scale_device(s["vals"].data_ptr(), s["R"].data_ptr())
        gn.status()
    return s


def run(state):
    s, c = state, state["c"]
    if c["kind"] == "fill":
        gn, d = s["gn"], s["d"]
        vals = s["vals"].data_ptr() if c["jac"] else None
        if c["transient"]:
            from goma_gb300 import _lib
            _lib.check(_lib.load().gb_matrix_fill_full_transient_device(
                gn.h, s["x"].data_ptr(), s["xdot"].data_ptr(), d["dt"], d["theta"],
                s["R"].data_ptr(), vals, None))
        else:
            gn.matrix_fill_full_device(s["x"].data_ptr(), s["R"].data_ptr(), vals)
        return {"R": s["R"], "vals": s["vals"]} if c["jac"] else {"R": s["R"]}
    if c["kind"] == "solve":
        s["gn"].linear_solve_device(s["vals"].data_ptr(), s["R"].data_ptr(), s["dx"].data_ptr(),
                                    krylov_dim=c["krylov"], linear_tol=c["tol"],
                                    max_linear_its=3000)
        return {"dx": s["dx"]}
    if c["kind"] == "newton":
        x, _, _ = s["gn"].solve_nonlinear_problem(
            s["x0"], residual_tol=c["tol"], linear_tol=1e-9, krylov_dim=c["krylov"],
            max_linear_its=3000, max_newton=25, fp32_preconditioner=c["fp32_prec"])
        return {"x": x}
    net = s["net"]
    net.set_params(s["params"])
    x, t, mask = s["data"]
    net.train(x, t, mask, c["steps"], batch=c["batch"], lr=2e-3, seed=s["seed"])
    return {"params": net.params(), "y": net.forward(x)}


# ----------------------------------------------------------------- the floor


def _counts(c):
    """Elements, nodes, unknowns and matrix entries."""
    if c["problem"] == "batch":
        ns = np.random.default_rng(c["meshes"]).integers(c["nx"], c["ny"] + 1, c["nz"])
        grids, dim = [(int(k), int(k)) for k in ns], 2
    else:
        g = (c["nx"], c["ny"], c["nz"]) if c["nz"] else (c["nx"], c["ny"])
        grids, dim = [g], len(g)
    energy = c["problem"] in ("boussinesq", "reacting")
    nv, npr = dim + energy + (2 if c["problem"] == "reacting" else 0), dim + 1
    nn = 3 ** dim
    e = sum(math.prod(g) for g in grids)
    nodes = sum(math.prod(2 * k + 1 for k in g) for g in grids)
    pairs = sum(math.prod(8 * k + 1 for k in g) for g in grids)
    faces = sum(math.prod(g) // k * (k - 1) for g in grids for k in g)
    nnz = nv * nv * pairs + e * (npr * nn * (2 * nv - (1 if energy else 0)) + npr * npr)
    nnz += 2 * faces * ((nv + npr) ** 2 - (npr if energy else 0))
    return e, nodes, nv * nodes + npr * e, nnz, dim, nn, nv, npr


def work(case):
    c = case
    if c["kind"] == "mlp":
        w = [8] + [c["width"]] * c["hidden"] + [1]
        macs = sum(a * b for a, b in zip(w[:-1], w[1:]))
        b = min(c["batch"], c["rows"])
        return {"bytes": 4.0 * (c["rows"] * 11 + 8 * macs),
                "flops": 2.0 * macs * (3 * b * c["steps"] + c["rows"])}
    e, nodes, N, nnz, dim, nn, nv, npr = _counts(c)
    mesh = nodes * (8 * dim + 4) + e * nn * 4
    fill_flops = {2: 9 * 9 * 9 * 2 * 11, 3: 363825 if nv == 4 else 363825 + 2 * 27 ** 3 * 14}[dim]
    if c["kind"] == "fill":
        return {"bytes": float(mesh + 16 * N + (8 * nnz if c["jac"] else 0)),
                "flops": float(e * (fill_flops if c["jac"] else 30 * nn * nn * nv))}
    if c["kind"] == "solve":  # the matrix once; the incomplete factors' products
        return {"bytes": float(12 * nnz + 16 * N), "flops": float(nnz * nnz / N / 2)}
    return {"bytes": float(mesh + 16 * N + 12 * nnz), "flops": float(e * fill_flops)}


# --------------------------------------------------------------- in 64 bits


def _tables(dim):
    g = np.sqrt(0.6)
    pt, wt = np.array([g, 0.0, -g]), np.array([5.0, 8.0, 5.0]) / 9.0
    lag = [lambda s: 0.5 * s * (s - 1), lambda s: 1 - s * s, lambda s: 0.5 * s * (s + 1)]
    dlag = [lambda s: s - 0.5, lambda s: -2 * s, lambda s: s + 0.5]
    q = np.stack(np.meshgrid(*[np.arange(3)] * dim, indexing="ij"), -1).reshape(-1, dim)[:, ::-1]
    local = _QUAD9 if dim == 2 else _HEX27
    phi, w = np.ones((len(q), len(local))), np.prod(wt[q], 1)
    dphi = np.ones((len(q), len(local), dim))
    for k, node in enumerate(local):
        for d in range(dim):
            phi[:, k] *= lag[node[d]](pt[q[:, d]])
            for r in range(dim):
                dphi[:, k, r] *= (dlag if r == d else lag)[node[d]](pt[q[:, d]])
    psi = np.concatenate([np.ones((len(q), 1)), pt[q]], 1)
    return phi, dphi, psi, w


def _element(d, dev):
    """(u, ud, X, rho) -> the residual of one element, unknowns ordered as
    nv fields per local node and then the pressures."""
    dim, nv, m, energy = d["dim"], d["nv"], d["m"], d["energy"]
    phi, dphi, psi, w = (torch.from_numpy(a).to(dev) for a in _tables(dim))
    nn = phi.shape[1]
    eye = torch.eye(dim, dtype=torch.float64, device=dev)
    src = torch.tensor(m.get("source", (0.0,) * 3)[:dim], dtype=torch.float64, device=dev)

    def residual(u, ud, X, rho):
        U, Pn = u[:nn * nv].reshape(nn, nv), u[nn * nv:]
        Ud = ud[:nn * nv].reshape(nn, nv)
        Jm = torch.einsum("qki,kj->qij", dphi, X)
        G = torch.einsum("qpi,qki->qkp", torch.linalg.inv(Jm), dphi)
        dA = w * torch.linalg.det(Jm)
        F, Fd, gF = phi @ U, phi @ Ud, torch.einsum("qkp,kf->qpf", G, U)
        v, gv = F[:, :dim], gF[:, :, :dim]
        gam = gv + gv.transpose(1, 2)
        mu = m.get("viscosity", 1.0) * torch.ones_like(dA)
        if "mu0" in m:
            gd = torch.sqrt(0.5 * (gam * gam).sum((1, 2)))
            mu = m["mu_inf"] + (m["mu0"] - m["mu_inf"]) * (
                1 + (m["lam"] * gd) ** m["aexp"]) ** ((m["nexp"] - 1) / m["aexp"])
        P = psi @ Pn
        tau = mu[:, None, None] * gam - P[:, None, None] * eye
        f = torch.zeros_like(v)
        if "source" in m:
            f = -rho * m["beta"] * (F[:, dim] - m["tref"])[:, None] * src
        adv = torch.einsum("qp,qpf->qf", v, gF) + Fd
        rows = [torch.einsum("q,qi,qa->ia", dA, phi, f - rho * adv[:, :dim])
                - torch.einsum("q,qip,qpa->ia", dA, G, tau)]
        if energy:
            rc = rho * m["heat_capacity"]
            rows.append((-rc * phi.T @ (dA * adv[:, dim]) - m["conductivity"] * torch.einsum(
                "q,qip,qp->i", dA, G, gF[:, :, dim]))[:, None])
        for s in range(d["nspec"]):
            k = dim + 1 + s
            rate = (-1.0, 1.0)[s] * m["k0"] * torch.exp(-m["activation"] / F[:, dim]) * F[:, dim + 1]
            rows.append((phi.T @ (dA * (rate - adv[:, k])) - m["diffusivity"] * torch.einsum(
                "q,qip,qp->i", dA, G, gF[:, :, k]))[:, None])
        cont = psi.T @ (dA * torch.diagonal(gv, dim1=1, dim2=2).sum(1))
        return torch.cat([torch.cat(rows, 1).reshape(-1), cont])

    return residual


def _assemble(d, x, xdot, mass, jac, dev):
    """R and (row, column, value) of the assembled system on the device."""
    dim, nv, npr, conn = d["dim"], d["nv"], d["npres"], torch.from_numpy(d["conn"]).to(dev).long()
    fu = torch.from_numpy(d["fu"]).to(dev)
    E, nn = conn.shape
    dofs = (fu[conn][:, :, None] + torch.arange(nv, device=dev)).reshape(E, -1)
    cent = torch.from_numpy(d["cent"]).to(dev).long()
    dofs = torch.cat([dofs, fu[cent][:, None] + nv + torch.arange(npr, device=dev)], 1)
    X = torch.from_numpy(d["X"]).to(dev)[conn]
    rho = torch.from_numpy(d["rho"]).to(dev) if d["rho"] is not None else \
        torch.full((E,), float(d["m"]["density"]), dtype=torch.float64, device=dev)
    res = _element(d, dev)
    # a time step's rates follow its unknowns: d xdot / d x = mass
    moved = lambda u, u0, ud, X, r: res(u, ud + mass * (u - u0), X, r)  # noqa: E731
    R = torch.zeros(d["N"], dtype=torch.float64, device=dev)
    parts = []
    for a in range(0, E, 2048 if dim == 2 else 128):
        b = min(E, a + (2048 if dim == 2 else 128))
        u, ud = x[dofs[a:b]], xdot[dofs[a:b]]
        R.index_add_(0, dofs[a:b].reshape(-1),
                     torch.vmap(res)(u, ud, X[a:b], rho[a:b]).reshape(-1))
        if jac:
            parts.append(torch.vmap(torch.func.jacfwd(moved))(u, u, ud, X[a:b], rho[a:b]))
    dirichlet = torch.zeros(d["N"], dtype=torch.bool, device=dev)
    dirichlet[torch.from_numpy(d["di"]).to(dev)] = True
    R[dirichlet] = 0.0
    if not jac:
        return R, None, dofs, dirichlet
    J = torch.cat(parts)
    mask = dirichlet[dofs]
    J[mask] = 0.0  # the rows of hard-set unknowns: 1 per element on the diagonal
    J.diagonal(dim1=1, dim2=2)[mask] = 1.0
    return R, J, dofs, dirichlet


def _csr_values(d, J, dofs, dev):
    """Values in the matrix's order: every unknown couples with those of the
    nodes of its elements, a centroid node also with the centroid nodes of
    the elements beyond its faces; energy rows hold no pressure columns."""
    N, dim, nv, npr = d["N"], d["dim"], d["nv"], d["npres"]
    nn = 3 ** dim
    keep = torch.ones(J.shape[1:], dtype=torch.bool, device=dev)
    if d["energy"]:
        keep[dim:nn * nv:nv, nn * nv:] = False
    ke = (dofs[:, :, None] * N + dofs[:, None, :])[:, keep].reshape(-1)
    # face neighbours: elements that share the node in the middle of a face
    face = d["conn"][:, 4:8] if dim == 2 else d["conn"][:, 21:27]
    own = np.repeat(np.arange(len(face)), face.shape[1])
    order = np.argsort(face.reshape(-1), kind="stable")
    fs, es = face.reshape(-1)[order], own[order]
    two = np.nonzero(fs[1:] == fs[:-1])[0]
    pair = np.concatenate([np.stack([es[two], es[two + 1]], 1), np.stack([es[two + 1], es[two]], 1)])
    loc = torch.cat([torch.arange(nv, device=dev), nv + torch.arange(npr, device=dev)])
    base = torch.from_numpy(d["fu"][d["cent"]]).to(dev)
    kc = torch.ones((nv + npr, nv + npr), dtype=torch.bool, device=dev)
    if d["energy"]:
        kc[dim, nv:] = False
    r, q = base[torch.from_numpy(pair[:, 0]).to(dev)], base[torch.from_numpy(pair[:, 1]).to(dev)]
    kf = ((r[:, None, None] + loc[:, None]) * N + q[:, None, None] + loc[None])[:, kc].reshape(-1)
    keys = torch.unique(torch.cat([ke, kf]))
    vals = torch.zeros(len(keys), dtype=torch.float64, device=dev)
    vals.index_add_(0, torch.searchsorted(keys, ke), J[:, keep].reshape(-1))
    return keys, vals


def _dense(d, J, dofs, dev):
    A = torch.zeros((d["N"], d["N"]), dtype=torch.float64, device=dev)
    n = dofs.shape[1]
    A.index_put_((dofs[:, :, None].expand(-1, n, n).reshape(-1),
                  dofs[:, None, :].expand(-1, n, n).reshape(-1)), J.reshape(-1), accumulate=True)
    return A


def _mlp_exact(c, seed):
    """The training in 64 bits: the library's documented minibatch hash,
    mask-weighted squared error, Adam."""
    x, t, mask, widths, params = _mlp_data(c, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    x, t, mask = (torch.from_numpy(a).double().to(dev) for a in (x, t, mask))
    p = torch.from_numpy(params).double().to(dev).requires_grad_(True)

    def net(h):
        o = 0
        for l, (a, b) in enumerate(zip(widths[:-1], widths[1:])):
            h = h @ p[o:o + a * b].reshape(b, a).T + p[o + a * b:o + a * b + b]
            o += a * b + b
            h = torch.tanh(h) if l + 2 < len(widths) else h
        return h

    n, B = c["rows"], min(c["batch"], c["rows"])
    M = (1 << 64) - 1
    z = (seed * 0xD1B54A32D192ED03 + 7) & M
    mo, ve = torch.zeros_like(p), torch.zeros_like(p)
    for step in range(1, c["steps"] + 1):
        idx = np.arange(B)
        with np.errstate(over="ignore"):
            r = np.uint64(z) + np.arange(1, B + 1, dtype=np.uint64) * np.uint64(0x9E3779B97F4A7C15)
            z = (z + B * 0x9E3779B97F4A7C15) & M
            r = (r ^ (r >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
            r = (r ^ (r >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
            r = r ^ (r >> np.uint64(31))
        if B < n:
            idx = (r % np.uint64(n)).astype(np.int64)
        i = torch.from_numpy(idx).to(dev)
        loss = (((net(x[i]) - t[i]) * mask[i]) ** 2).sum() / mask[i].sum()
        g, = torch.autograd.grad(loss, p)
        mo, ve = 0.9 * mo + 0.1 * g, 0.999 * ve + 0.001 * g * g
        with torch.no_grad():
            p -= 2e-3 * (mo / (1 - 0.9 ** step)) / (torch.sqrt(ve / (1 - 0.999 ** step)) + 1e-8)
    with torch.no_grad():
        return {"params": p.detach().cpu().numpy(), "y": net(x)}


def exact(case, seed):
    c = case
    if c["kind"] == "mlp":
        return _mlp_exact(c, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    d = _describe(c, seed)
    e, _, N, nnz, dim, nn, nv, npr = _counts(c)
    x = torch.from_numpy(d["x"]).to(dev)
    zero = torch.zeros_like(x)
    if c["kind"] == "fill":
        if nnz > 1.5e8:
            return None
        tr = c["transient"]
        R, J, dofs, _ = _assemble(d, x, torch.from_numpy(d["xdot"]).to(dev) if tr else zero,
                                  (1 + 2 * d["theta"]) / d["dt"] if tr else 0.0, c["jac"], dev)
        if not c["jac"]:
            return {"R": R}
        return {"R": R, "vals": _csr_values(d, J, dofs, dev)[1]}
    if N > 12500:
        return None  # a dense direct solve would take too long
    if c["kind"] == "solve":
        R, J, dofs, _ = _assemble(d, x, zero, 0.0, True, dev)
        return {"dx": torch.linalg.solve(_dense(d, J, dofs, dev), R)}
    x = 0.01 * x
    xs = torch.from_numpy(d["x"]).to(dev)
    di = torch.from_numpy(d["di"]).to(dev)
    x[di] = xs[di]
    for it in range(25):
        R, J, dofs, _ = _assemble(d, x, zero, 0.0, True, dev)
        dx = torch.linalg.solve(_dense(d, J, dofs, dev), R)
        x = x - dx
        if float(dx.norm()) <= 1e-12 * float(x.norm()):
            break
    return {"x": x}
