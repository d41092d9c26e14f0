"""Performance cases: the work a user of this package has it do, through its
public entry points, from the smallest calls to the largest.

Kinds of case (the field ``kind``):

  driver3d   fc3d_driver on host buffers, W's values changed before every call
             (a simulation that reassembles W each step), options kept;
  solve3d    a device-resident 3D problem solved from zero and read back;
  step3d     one time step: velocities and their random walk on the device, the
             learned warm start, the solve from it, r and u read back;
  batch3d    many independent scenes in one launch;
  solver2d   fc2d_driver on host buffers;
  rolling    a device-resident rolling-friction problem;
  global     a device-resident global problem (M v = q + H r);
  train      minibatch training of the warm-start network;
  error3d    fc3d_compute_error on arrays the caller holds on the GPU.

Solves run to a tolerance or to a sweep budget, as in a time-stepping code.
Launch shapes are pinned where the calls allow it (``lanes`` 1: no measuring of
variants in the first solve), so that a pass repeats.  The sweeps of the 2D, 3D
and rolling solvers visit the contacts in an order that the solver itself
chooses, so their results have no value that is independent of it; the error
evaluation, the global problem's iteration and the training step do.
"""
from __future__ import annotations

import ctypes as C
import math
from pathlib import Path

import numpy as np
import torch

import siconos_gb300.learned as learned
import siconos_gb300.numerics as sn
from siconos_gb300.device import DeviceSolver
from siconos_gb300.scene import batch_specs, lattice, lattice_global

GOLDEN = Path(__file__).resolve().parents[1] / "tests" / "golden"
# the 2D granular flows and the rolling rockfall that the tests solve
GRANULAR = {"small": "fc2d_FrictionContactProblem00071", "medium": "fc2d_FrictionContactProblem00727",
            "large": "fc2d_fc2d_granularflowonwall_07002_00801"}
ROCKFALL = "rfc3d_rockfall_21_54029"


def listed():
    return [
        # a hand-sized scene solved to the reference's accuracy: latency and launches
        dict(name="driver3d_tiny", kind="driver3d", nx=3, ny=3, nz=2, precision=0, tol=1e-8, sweeps=300),
        # an ordinary simulation step through the C-ABI
        dict(name="driver3d_mid", kind="driver3d", nx=20, ny=20, nz=10, precision=0, tol=1e-3, sweeps=1000),
        # the reference's own arithmetic (FP64 sweeps only) on an ordinary scene
        dict(name="solve3d_fp64", kind="solve3d", nx=30, ny=31, nz=15, precision=1, tol=1e-8, sweeps=60),
        # the benchmark scene to the tolerance the reference reaches
        dict(name="solve3d_large", kind="solve3d", nx=60, ny=60, nz=30, precision=0, tol=1e-3, sweeps=1000),
        # a step of a long simulation, everything on the device
        dict(name="step3d", kind="step3d", nx=40, ny=41, nz=20, tol=1e-3, sweeps=150),
        # parameter studies: many small scenes of unequal sizes
        dict(name="batch3d", kind="batch3d", scenes=48, hx=20, hy=20, hz=10, precision=0, tol=1e-4, sweeps=100),
        # a small 2D problem in the reference's arithmetic
        dict(name="solver2d_small", kind="solver2d", problem="medium", copies=1, precision=1, tol=1e-5, sweeps=1000),
        # a large granular flow, mixed precision (the driver's default)
        dict(name="solver2d_large", kind="solver2d", problem="large", copies=4, precision=0, tol=1e-5, sweeps=300),
        # rocks with rolling resistance
        dict(name="rolling", kind="rolling", copies=100, precision=1, tol=1e-8, sweeps=100),
        # the global formulation of a middling scene
        dict(name="global", kind="global", nx=40, ny=40, nz=20, tol=1e-12, sweeps=200),
        # an epoch's share of the warm-start network's training
        dict(name="train", kind="train", samples=50000, batch=4096, steps=8),
        # the error of a given reaction, inputs in the caller's GPU memory
        dict(name="error3d", kind="error3d", nx=40, ny=40, nz=20),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _dims(rng, bodies):
    """Lattice sides with at most `bodies` spheres, spread over its logarithm."""
    n = math.exp(rng.uniform(math.log(12), math.log(bodies)))
    nx = max(2, round(n ** (1 / 3) * math.exp(rng.uniform(-0.4, 0.4))))
    ny = max(2, round(n ** (1 / 3) * math.exp(rng.uniform(-0.4, 0.4))))
    return dict(nx=nx, ny=ny, nz=max(2, int(n / (nx * ny))))


def draw(rng):
    kind = rng.choice(["driver3d", "solve3d", "solve3d", "step3d", "batch3d", "solver2d", "rolling", "global", "train",
                       "error3d"])
    if kind == "driver3d":
        return dict(kind=kind, **_dims(rng, 12000), precision=rng.choice([0, 0, 1]), tol=rng.choice([1e-3, 1e-4]),
                    sweeps=rng.randint(50, 200))
    if kind == "solve3d":
        p = rng.choice([0, 1])
        return dict(kind=kind, **_dims(rng, 20000 if p else 108000), precision=p, tol=rng.choice([1e-3, 1e-4, 1e-8]),
                    sweeps=rng.randint(20, 60) if p else rng.randint(50, 400))
    if kind == "step3d":
        return dict(kind=kind, **_dims(rng, 33000), tol=1e-3, sweeps=rng.randint(50, 150))
    if kind == "batch3d":
        return dict(kind=kind, scenes=rng.randint(2, 40), hx=rng.randint(5, 20), hy=rng.randint(5, 20),
                    hz=rng.randint(3, 10), precision=rng.choice([0, 0, 1]), tol=rng.choice([1e-3, 1e-4]),
                    sweeps=rng.randint(20, 60))
    if kind == "solver2d":
        prob = rng.choice(list(GRANULAR))
        return dict(kind=kind, problem=prob, copies=_log(rng, 1, 10 if prob == "large" else 100),
                    precision=rng.choice([0, 1]), tol=1e-5, sweeps=rng.randint(50, 200))
    if kind == "rolling":
        return dict(kind=kind, copies=_log(rng, 1, 1000), precision=rng.choice([0, 1]), tol=1e-8,
                    sweeps=rng.randint(20, 60))
    if kind == "global":
        return dict(kind=kind, **_dims(rng, 32000), tol=1e-12, sweeps=rng.randint(50, 200))
    if kind == "train":
        n = _log(rng, 1000, 50000)
        return dict(kind=kind, samples=n, batch=_log(rng, 128, min(n, 16384)), steps=rng.randint(1, 8))
    return dict(kind=kind, **_dims(rng, 108000))


# ---- inputs ---------------------------------------------------------------
def _lattice(case, seed):
    return lattice(case["nx"], case["ny"], case["nz"], seed=seed)


def _specs(case):
    """Sides, seed and friction of a batch's scenes."""
    return batch_specs(case["scenes"], 7, hi=(case["hx"], case["hy"], case["hz"]))


def _tiled(z, width, copies, seed):
    """`copies` independent copies of a stored problem along W's diagonal, each
    contact's q scaled by its own factor."""
    g = np.random.default_rng(seed)
    nc, nb = int(z["nc"]), int(z["rowptr"][-1])
    rp = np.concatenate([[0]] + [z["rowptr"][1:] + c * nb for c in range(copies)]).astype(np.int64)
    ci = np.concatenate([z["colidx"] + c * nc for c in range(copies)]).astype(np.int64)
    bl = np.tile(np.asarray(z["blocks"]).reshape(nb, width * width), (copies, 1))
    q = np.tile(z["q"], copies) * np.repeat(g.uniform(0.9, 1.1, copies * nc), width)
    return copies * nc, rp, ci, bl, q, np.tile(z["mu"], copies)


def _train_set(case, seed):
    """Features and targets like the warm start's (a smooth map and noise-free
    products of a few features), initial parameters, statistics, minibatches."""
    g = np.random.default_rng(seed)
    X = g.standard_normal((case["samples"], learned.NF)).astype(np.float32) * 2 + 1
    T = np.stack([np.tanh(X[:, 0] + X[:, 3]), X[:, 5] * X[:, 6], np.abs(X[:, 9])], 1).astype(np.float32)
    idx = [g.permutation(case["samples"])[:case["batch"]].astype(np.int32) for _ in range(case["steps"])]
    return X, T, learned.init_params(seed % 100003), learned.make_stats(X, T), idx


def _reaction(nc, seed):
    g = np.random.default_rng(seed)
    r = np.empty((nc, 3))
    r[:, 0] = np.abs(g.standard_normal(nc))
    r[:, 1:] = 0.3 * g.standard_normal((nc, 2))
    return r.reshape(-1)


def prepare(case, seed):
    k = case["kind"]
    st = {"case": case}
    if k == "driver3d":
        sc = _lattice(case, seed)
        o = sn.SolverOptions(sn.SICONOS_FRICTION_3D_NSGS_GPU)
        o.iparam[sn.SICONOS_IPARAM_MAX_ITER] = case["sweeps"]
        o.dparam[sn.SICONOS_DPARAM_TOL] = case["tol"]
        o.iparam[sn.FC3DGPU_IPARAM_PRECISION] = case["precision"]
        o.iparam[sn.FC3DGPU_IPARAM_LANES] = 1
        st.update(P=sc.problem(), o=o, r=np.zeros(3 * sc.nc), u=np.zeros(3 * sc.nc))
    elif k == "solve3d":
        d = DeviceSolver(0)
        d.load(_lattice(case, seed))
        st["d"] = d
    elif k == "step3d":
        sc = _lattice(case, seed)
        geo = sc.contacts()
        d = DeviceSolver(0)
        d.set_contacts(geo)
        d.set_mu(sc.mu)
        mlp = learned.WarmStartMLP(0)
        mlp.load()
        st.update(d=d, mlp=mlp, vel=geo["vel"], gap=sc.gap, seed=seed)
    elif k == "batch3d":
        d = DeviceSolver(0)
        d.load_batch([lattice(*dims, seed=s + seed, mu=mu) for dims, s, mu in _specs(case)])
        st["d"] = d
    elif k == "solver2d":
        nc, rp, ci, bl, q, mu = _tiled(np.load(GOLDEN / (GRANULAR[case["problem"]] + ".npz")), 2, case["copies"], seed)
        o = sn.SolverOptions(sn.SICONOS_FRICTION_2D_NSGS_GPU)
        o.iparam[sn.SICONOS_IPARAM_MAX_ITER] = case["sweeps"]
        o.dparam[sn.SICONOS_DPARAM_TOL] = case["tol"]
        o.iparam[sn.FC3DGPU_IPARAM_PRECISION] = case["precision"]
        st.update(P=sn.FrictionContactProblem(2, nc, sn.SparseBlockMatrix(nc, rp, ci, bl, block_size=2), q, mu), o=o,
                  r=np.zeros(2 * nc), u=np.zeros(2 * nc))
    elif k == "rolling":
        z = np.load(GOLDEN / (ROCKFALL + ".npz"))
        nc, rp, ci, bl, q, mu = _tiled(z, 5, case["copies"], seed)
        ctx = sn.RollingContext(nc, rp, ci, bl, q, mu, np.tile(z["mur"], case["copies"]))
        ctx.set_precision(case["precision"])
        st.update(ctx=ctx, r0=np.zeros(5 * nc))
    elif k == "global":
        G = lattice_global(case["nx"], case["ny"], case["nz"], seed=seed)
        st["ctx"] = sn.Gfc3dContext.from_problem(G)
        st.update(r0=np.zeros(3 * G.nc), v0=np.zeros(G.n))
    elif k == "train":
        X, T, p, stats, idx = _train_set(case, seed)
        m = learned.WarmStartMLP(0)
        m.set_params(p, stats)
        m.set_data(X, T)
        st.update(mlp=m, params=p, stats=stats, idx=idx)
    else:
        sc = _lattice(case, seed)
        dev = {n: torch.from_numpy(np.ascontiguousarray(a)).cuda() for n, a in
               dict(rowptr=sc.rowptr, colidx=sc.colidx, blocks=sc.blocks.reshape(-1), q=sc.q, mu=sc.mu,
                    r=_reaction(sc.nc, seed)).items()}
        st.update(nc=sc.nc, nnzb=sc.nnzb, norm_q=float(np.linalg.norm(sc.q)), dev=dev,
                  u=torch.zeros(3 * sc.nc, dtype=torch.float64, device="cuda"),
                  err=torch.zeros(1, dtype=torch.float64, device="cuda"))
    return st


def run(st):
    case = st["case"]
    k = case["kind"]
    if k == "driver3d":
        st["r"][:] = 0.0
        st["P"].M().bump_version()
        info = sn.fc3d_driver(st["P"], st["r"], st["u"], st["o"])
        return {"r": st["r"], "u": st["u"], "info": info}
    if k == "solve3d":
        st["d"].zero_r()
        s = st["d"].solve(tol=case["tol"], max_iter=case["sweeps"], precision=case["precision"], lanes=1)
        r, u = st["d"].get()
        return {"r": r, "u": u, "info": s["info"]}
    if k == "step3d":
        d = st["d"]
        d.zero_r()
        d.set_velocities(st["vel"])
        d.random_walk(st["seed"] + 1, 0.01)
        ws = learned.warm_start(d, st["mlp"], st["gap"])
        s = d.solve(tol=case["tol"], max_iter=case["sweeps"], lanes=1)
        r, u = d.get()
        return {"r": r, "u": u, "info": s["info"], "error0": ws["error_fallback"]}
    if k == "batch3d":
        st["d"].zero_r()
        s = st["d"].solve_batch(tol=case["tol"], max_iter=case["sweeps"], precision=case["precision"])
        r, u = st["d"].get()
        return {"r": r, "u": u, "info": s["info"], "error": s["error"]}
    if k == "solver2d":
        st["r"][:] = 0.0
        info = sn.fc2d_driver(st["P"], st["r"], st["u"], st["o"])
        return {"r": st["r"], "u": st["u"], "info": info}
    if k == "rolling":
        st["ctx"].set_r(st["r0"])
        s = st["ctx"].solve(case["tol"], case["sweeps"])
        r, u = st["ctx"].get_r_u()
        return {"r": r, "u": u, "info": s["info"], "error": s["error"]}
    if k == "global":
        st["ctx"].set_start(st["r0"], st["v0"])
        s = st["ctx"].solve(case["tol"], case["sweeps"])
        r, u, v = st["ctx"].get()
        return {"r": r, "u": u, "v": v, "error": s["error"]}
    if k == "train":
        st["mlp"].set_params(st["params"], st["stats"])
        g, loss = st["mlp"].grad(st["idx"][0])
        for i in st["idx"]:
            st["mlp"].step(i, 1e-3, 1e-4, want_loss=False)
        return {"grad": g, "loss": loss, "params": st["mlp"].get_params()[0]}
    d = st["dev"]
    rc = sn.lib().fc3dgpu_compute_error_device(st["nc"], st["nnzb"], d["rowptr"].data_ptr(), d["colidx"].data_ptr(),
                                               d["blocks"].data_ptr(), d["q"].data_ptr(), d["mu"].data_ptr(),
                                               d["r"].data_ptr(), st["norm_q"], st["u"].data_ptr(),
                                               st["err"].data_ptr(), torch.cuda.current_stream().cuda_stream)
    if rc != 0:
        raise RuntimeError(sn.last_error())
    return {"u": st["u"], "error": st["err"]}


# ---- the work of one pass -------------------------------------------------
def _lattice_sizes(dims):
    """(contacts, blocks of W, spheres) of a lattice."""
    L = sn.lib()
    h = L.fc3dgpu_lattice_create(*dims, 1, 1e-3, 0.1)
    nb, nc, nnzb = C.c_int(), C.c_int(), C.c_int64()
    L.fc3dgpu_lattice_sizes(h, C.byref(nb), C.byref(nc), C.byref(nnzb))
    L.fc3dgpu_lattice_free(h)
    return nc.value, nnzb.value, nb.value


def _sweeps_work(nc, nnzb, d, sweeps, real):
    """Sweeps of a d-component problem: W with its column indices, q, mu and r
    read, r written, in each; the products with W's blocks and about 40 d
    operations for a contact's local problem."""
    return {"bytes": sweeps * (nnzb * (d * d * real + 4) + nc * (3 * d + 2) * real),
            "flops": sweeps * (2 * d * d * nnzb + 40 * d * nc)}


def work(case):
    k = case["kind"]
    if k in ("driver3d", "solve3d", "step3d"):
        nc, nnzb, _ = _lattice_sizes((case["nx"], case["ny"], case["nz"]))
        # solves to a tolerance end before their budget: about 100 sweeps (a
        # small scene) to 550 (the largest)
        sweeps = min(case["sweeps"], int(100 + 450 * min(1.0, nc / 320400)))
        return _sweeps_work(nc, nnzb, 3, sweeps, 8 if case.get("precision") == 1 else 4)
    if k == "batch3d":
        sizes = [_lattice_sizes(s[0]) for s in _specs(case)]
        return _sweeps_work(sum(s[0] for s in sizes), sum(s[1] for s in sizes), 3, case["sweeps"],
                            8 if case["precision"] == 1 else 4)
    if k in ("solver2d", "rolling"):
        z = np.load(GOLDEN / ((GRANULAR[case["problem"]] if k == "solver2d" else ROCKFALL) + ".npz"))
        return _sweeps_work(int(z["nc"]) * case["copies"], int(z["rowptr"][-1]) * case["copies"],
                            2 if k == "solver2d" else 5, min(case["sweeps"], 300), 8 if case["precision"] == 1 else 4)
    if k == "global":
        # an iteration reads H by rows and by columns, M, q, b, and reads and
        # writes r, u and v
        nc, _, nb = _lattice_sizes((case["nx"], case["ny"], case["nz"]))
        n, nnz = 6 * nb, 36 * nc
        return {"bytes": case["sweeps"] * (2 * nnz * 12 + n * 52 + nc * 104),
                "flops": case["sweeps"] * (4 * nnz + 60 * nc)}
    if k == "train":
        per = 2 * (32 * 128 + 2 * 128 * 128 + 128 * 16) * 3
        n = case["batch"] * (case["steps"] + 1)
        return {"bytes": n * 4 * (learned.NF + learned.NO + 1) + case["steps"] * 39312 * 4 * 7, "flops": n * per}
    nc, nnzb, _ = _lattice_sizes((case["nx"], case["ny"], case["nz"]))
    return {"bytes": nnzb * 80 + nc * (8 + 3 * 24 + 8), "flops": 18 * nnzb + 60 * nc}


# ---- the same results in 64 bits by other means ----------------------------
def _project(w, mu):
    """Projection of the columns of w (3 x n) on the friction cones."""
    n, t = w[0], torch.sqrt(w[1] ** 2 + w[2] ** 2)
    a = (mu * t + n) / (mu * mu + 1.0)
    s = torch.where(t > 0, mu * a / torch.where(t > 0, t, torch.ones_like(t)), torch.zeros_like(t))
    out = torch.stack([a, s * w[1], s * w[2]])
    out = torch.where(t <= mu * n, w, out)
    return torch.where(mu * t <= -n, torch.zeros_like(w), out)


def _natural_map(r, u, mu):
    """Sum over the contacts of the squared natural-map residual."""
    r, u = r.reshape(-1, 3).T, u.reshape(-1, 3).T
    w = r - u
    w = torch.stack([w[0] - mu * torch.sqrt(u[1] ** 2 + u[2] ** 2), w[1], w[2]])
    return ((r - _project(w, mu)) ** 2).sum()


def _exact_error(case, seed):
    sc = _lattice(case, seed)
    r = torch.from_numpy(_reaction(sc.nc, seed))
    rows = torch.from_numpy(np.repeat(np.arange(sc.nc), np.diff(sc.rowptr)))
    B = torch.from_numpy(sc.blocks.reshape(-1, 3, 3))  # [column][row] of each column-major block
    x = r.reshape(-1, 3)[torch.from_numpy(np.ascontiguousarray(sc.colidx))]
    u = torch.from_numpy(sc.q.copy()).reshape(-1, 3).index_add(0, rows, torch.einsum("kji,kj->ki", B, x)).reshape(-1)
    scale = max(float(np.linalg.norm(sc.q)), float(r.norm()), float(u.norm()))
    e = torch.sqrt(_natural_map(r, u, torch.from_numpy(sc.mu))) / scale
    return {"u": u, "error": e.reshape(1)}


def _exact_global(case, seed):
    """The projected unit-step iteration and its error: v = M^-1 (q + H r),
    u = b + H^T v, r <- P_K(r - (u_N + mu |u_T|, u_T))."""
    G = lattice_global(case["nx"], case["ny"], case["nz"], seed=seed)
    if not (np.array_equal(G.Mi, np.arange(G.n)) and np.array_equal(G.Mp, np.arange(G.n + 1))):
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)
    H = torch.sparse_csr_tensor(t(G.Hp), t(G.Hi), t(G.Hx), size=(G.n, 3 * G.nc), dtype=torch.float64)
    rows = torch.repeat_interleave(torch.arange(G.n, device=dev), t(np.diff(G.Hp)))
    HT = torch.sparse_coo_tensor(torch.stack([t(G.Hi), rows]), t(G.Hx), (3 * G.nc, G.n)).coalesce().to_sparse_csr()
    M, q, b, mu = t(G.Mx), t(G.q), t(G.b), t(G.mu)
    r = torch.zeros(3 * G.nc, dtype=torch.float64, device=dev)
    for _ in range(case["sweeps"]):
        v = (q + H @ r) / M
        u = b + HT @ v
        w, uu = r.reshape(-1, 3).T, u.reshape(-1, 3).T
        w = w - torch.stack([uu[0] + mu * torch.sqrt(uu[1] ** 2 + uu[2] ** 2), uu[1], uu[2]])
        r = _project(w, mu).T.reshape(-1)
    Hr, Mv = H @ r, M * v
    e = torch.linalg.norm(q + Hr - Mv) / max(_norm(q), _norm(Hr), _norm(Mv))
    e = e + torch.sqrt(_natural_map(r, u, mu)) / max(_norm(u), _norm(r))
    return {"r": r, "u": u, "v": v, "error": float(e)}


def _norm(x):
    return float(torch.linalg.norm(x))


def _exact_train(case, seed):
    X, T, p, stats, idx = _train_set(case, seed)
    NF, NO = learned.NF, learned.NO
    s = torch.from_numpy(stats.astype(np.float64))
    X = (torch.from_numpy(X).double() - s[:NF]) / s[NF:2 * NF]
    T = (torch.from_numpy(T).double() - s[2 * NF:2 * NF + NO]) / s[2 * NF + NO:]
    p = torch.from_numpy(p.astype(np.float64))
    shapes = [(32, 128), (128, 128), (128, 128), (128, 16)]
    decay = torch.cat([torch.cat([torch.ones(k * n), torch.zeros(n)]) for k, n in shapes]).double()

    def loss_grad(p, i):
        p = p.clone().requires_grad_(True)
        a = torch.nn.functional.pad(X[i], (0, 32 - NF))
        o = 0
        for l, (k, n) in enumerate(shapes):
            a = a @ p[o:o + k * n].reshape(k, n) + p[o + k * n:o + k * n + n]
            a = torch.relu(a) if l < 3 else a[:, :NO]
            o += k * n + n
        loss = ((a - T[i]) ** 2).mean()
        return float(loss.detach()), torch.autograd.grad(loss, p)[0]

    loss, grad = loss_grad(p, torch.from_numpy(idx[0]).long())
    m, v = torch.zeros_like(p), torch.zeros_like(p)
    for t, i in enumerate(idx, 1):
        _, g = loss_grad(p, torch.from_numpy(i).long())
        m = 0.9 * m + 0.1 * g
        v = 0.999 * v + 0.001 * g * g
        p = p - 1e-3 * ((m / (1 - 0.9 ** t)) / (torch.sqrt(v / (1 - 0.999 ** t)) + 1e-8) + 1e-4 * decay * p)
    return {"grad": grad, "loss": loss, "params": p}


def exact(case, seed):
    if case["kind"] == "error3d":
        return _exact_error(case, seed)
    if case["kind"] == "global":
        return _exact_global(case, seed)
    if case["kind"] == "train":
        return _exact_train(case, seed)
    return None
