"""Performance cases of ressim_gb300: the calls a simulator or an ensemble driver makes, over the range of system sizes,
block sizes, preconditioners and precisions the library is used with.

A Newton step of a caller is: new matrix values in (the pattern and its plan stay), preconditioner set-up, solve. That
is what ``run`` of the ``solve``, ``ensemble``, ``generic`` and ``serve`` cases does, from host arrays to a host solution,
on a handle whose plan ``prepare`` has made with the pattern's first system. The ``apply``, ``spmv`` and ``assemble`` cases
are the single layers on device vectors.

Inputs: the geology of a case (grid, permeability, wells: ``ressim_gb300.synth``) is the case's own and is generated once
per process; the seed draws the step -- the length of the time step and the pore volumes (A = accumulation +
dt / PV x flux and well terms), the solution the right-hand side is made from, the reservoir state of an assembly.
"""
import functools
import math

import numpy as np
import torch

from ressim_gb300 import BSR, synth
from ressim_gb300.assembly import BlackOilAssembler
from ressim_gb300.bsr import ScalarCSR
from ressim_gb300.solver import DeviceSolver, Server

TOL = 1e-6          # the engine's linear tolerance
MAXIT = 200


def listed():
    one = dict(kind="solve", inactive=0.0, wells="corners", form="block", acc=False, krylov="bicgstab", restart=40)
    return [
        # the engine's default for small models: one 20x20x4 waterflood system, ILU(0) and BiCGSTAB in FP64
        dict(one, name="newton_20x20x4_bilu0_fp64", nx=20, ny=20, nz=4, sigma=1.0, dt=10.0, precond="bilu0", precision="fp64"),
        # an ordinary model: the Jacobian with its well rows, reduced on the device, CPR with true-IMPES weights, FP64
        dict(one, name="newton_40x40x10_cpr_fp64", nx=40, ny=40, nz=10, sigma=1.5, dt=10.0, inactive=0.3, form="jacobian", acc=True,
             precond="cpr", precision="fp64"),
        # the same size in the precision form, already reduced on the host
        dict(one, name="newton_40x40x10_cpr_f32", nx=40, ny=40, nz=10, sigma=1.5, dt=10.0, inactive=0.3, precond="cpr",
             precision="mixed_f32"),
        # a model larger than one SM holds, FP64 in the reference's order (grid-wide sweeps)
        dict(one, name="newton_100x60x30_cpr_fp64", nx=100, ny=60, nz=30, sigma=1.5, dt=5.0, wells="random4", precond="cpr",
             precision="fp64"),
        # a quarter of the 60x220x85 channelled model: CPR with true-IMPES weights and GMRES(30), precision form
        dict(one, name="newton_60x110x42_gmres_f32", nx=60, ny=110, nz=42, sigma=2.5, dt=1.0, wells="channels", acc=True,
             precond="cpr", krylov="gmres", restart=30, precision="mixed_f32"),
        # the ensemble driver: 64 realisations at a common step, precision form
        dict(name="ensemble64_cpr_f32", kind="ensemble", members=64, nx=40, ny=40, nz=10, precision="mixed_f32"),
        # a small ensemble in plain FP64
        dict(name="ensemble16_cpr_fp64", kind="ensemble", members=16, nx=40, ny=40, nz=10, precision="fp64"),
        # a caller with its own Krylov loop: one CPR application to the ensemble's residual vectors
        dict(name="apply_ensemble64_cpr_f32", kind="apply", members=64, nx=40, ny=40, nz=10, precision="mixed_f32"),
        # and the matrix-vector product of that loop
        dict(name="spmv_ensemble64", kind="spmv", members=64, nx=40, ny=40, nz=10),
        # the Jacobian and residual of 742k cells from the reservoir state
        dict(name="assemble_64x40x40x10", kind="assemble", members=64, nx=40, ny=40, nz=10),
        # a compositional system (8 unknowns per cell): CPR and GMRES(60)
        dict(name="generic_16x12x5_nb8", kind="generic", nx=16, ny=12, nz=5, nb=8, restart=60),
        # a server (one worker) taking a burst of requests of uneven sizes
        dict(name="serve_16_requests", kind="serve", requests=16, lo=1200, hi=30000, precision="mixed_f32"),
    ]


def _box(rng, lo, hi, nz_hi):
    """A box of about exp(U[ln lo, ln hi]) cells, odd sizes included."""
    cells = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    nz = rng.randint(1, max(1, min(nz_hi, int(cells ** 0.5) // 2)))
    nx = max(6, round(math.sqrt(cells / nz) * math.exp(rng.uniform(-0.5, 0.5))))
    return nx, max(6, round(cells / nz / nx)), nz


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "ensemble", "ensemble", "apply", "spmv", "assemble", "generic", "serve"])
    if kind == "solve":
        precision = rng.choice(["fp64", "mixed_f32", "mixed_f32", "mixed"])
        nx, ny, nz = _box(rng, 1000, 200000 if precision == "mixed_f32" else 60000, 40)
        small = nx * ny * nz < 4000
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, sigma=round(rng.uniform(0.5, 2.0), 2), dt=round(math.exp(rng.uniform(0.0, 2.5)), 2),
                    inactive=rng.choice([0.0, round(rng.uniform(0.1, 0.5), 2)]), wells=rng.choice(["corners", "random4"]),
                    form=rng.choice(["block", "jacobian"]), acc=rng.random() < 0.5, precond="bilu0" if small and rng.random() < 0.5 else "cpr",
                    krylov=rng.choice(["bicgstab", "bicgstab", "gmres"]), restart=rng.choice([30, 40]), precision=precision)
    if kind in ("ensemble", "apply", "spmv"):
        nx, ny, nz = rng.randint(10, 40), rng.randint(10, 40), rng.randint(1, 10)
        c = dict(kind=kind, members=max(1, round(math.exp(rng.uniform(math.log(2), math.log(40))))), nx=nx, ny=ny, nz=nz)
        return c if kind == "spmv" else dict(c, precision=rng.choice(["fp64", "mixed_f32", "mixed_f32", "mixed"]))
    if kind == "assemble":
        nx, ny, nz = _box(rng, 100, 20000, 20)
        return dict(kind=kind, members=rng.randint(1, 24), nx=nx, ny=ny, nz=nz)
    if kind == "generic":
        return dict(kind=kind, nx=rng.randint(5, 16), ny=rng.randint(5, 14), nz=rng.randint(1, 6), nb=rng.choice([2, 4, 5, 6, 8]),
                    restart=rng.choice([40, 60, 80]))
    return dict(kind=kind, requests=rng.randint(2, 20), lo=1000, hi=rng.randint(5000, 30000), precision=rng.choice(["mixed_f32", "mixed_f32", "fp64"]))


# ---------------------------------------------------------------------------------------------------- inputs
def _frozen(case):
    """What the geology of a case depends on (the solver's options are not part of it)."""
    c = {k: v for k, v in case.items() if k not in ("name", "precond", "precision", "krylov", "restart", "acc")}
    if c["kind"] in ("apply", "spmv"):
        c["kind"] = "ensemble"
    return tuple(sorted(c.items()))


@functools.lru_cache(maxsize=3)
def _geology(key):
    """The systems of a case at the generator's own step."""
    c = dict(key)
    if c["kind"] == "solve":
        kw = dict(sigma=c["sigma"], seed=3, dt=c["dt"], actnum_fraction=c["inactive"], with_full=c["form"] == "jacobian")
        if c["wells"] == "channels":
            return [synth.make_system(c["nx"], c["ny"], c["nz"], corr=(5, 5, 1), dx=20.0, dy=10.0, dz=2.0, channels=(c["nz"] // 2, c["nz"] - 1, 4, 100.0),
                                      front_radius=0.05, gravity_head=True, p_noise=0.5, **kw)]
        if c["wells"] == "random4":
            return [synth.make_system(c["nx"], c["ny"], c["nz"], wells="random", n_wells=4, **kw)]
        return [synth.make_system(c["nx"], c["ny"], c["nz"], **kw)]
    if c["kind"] == "generic":
        return [synth.make_block_system(c["nx"], c["ny"], c["nz"], c["nb"], seed=c["nb"])]
    if c["kind"] == "serve":
        rng = np.random.default_rng(4242)
        out = []
        for r in range(c["requests"]):
            cells = math.exp(rng.uniform(math.log(c["lo"]), math.log(c["hi"])))
            nz = int(rng.integers(1, 21))
            nx = int(math.sqrt(cells / nz) * math.exp(rng.uniform(-0.5, 0.5))) + 2
            out.append(synth.make_system(nx, max(4, int(cells / nz / nx)), nz, sigma=float(rng.uniform(0.5, 1.5)), seed=r, dt=float(rng.uniform(0.5, 10.0)),
                                         wells="random", n_wells=int(rng.integers(2, 5))))
        return out
    if c["kind"] == "assemble":
        return [synth.assembly_grid(c["nx"], c["ny"], c["nz"], seed=r, actnum_fraction=0.1 + 0.4 * ((r * 7) % 13) / 13) for r in range(c["members"])]
    return synth.ensemble(c["members"], c["nx"], c["ny"], c["nz"])


def _matvec(rowPtr, col, blocks, x):
    y = np.einsum("kij,kj->ki", blocks, x.reshape(-1, blocks.shape[2])[col])
    return np.add.reduceat(y, rowPtr[:-1], axis=0).reshape(-1)


def _solution(n, nb, rng):
    xt = rng.standard_normal((n, nb))
    xt[:, 0] = 20.0 * np.sin(0.01 * np.arange(n) + rng.uniform(0, 6)) + xt[:, 0]
    if nb == 3:
        xt[:, 1:] *= (0.01, 0.005)
    return xt.reshape(-1)


def _step(s, rng):
    """One system at a drawn step: A = acc + f (A0 - acc), f the ratio of dt / PV to the generator's per cell; its
    solution and right-hand side."""
    A = s.A
    f = math.exp(rng.uniform(-0.7, 0.7)) * (1.0 + 0.1 * rng.random(A.n))
    rows = np.repeat(np.arange(A.n), np.diff(A.rowPtr))
    v = A.blocks() * f[rows][:, None, None]
    v[A.diag()] += (1.0 - f)[:, None, None] * s.acc.reshape(-1, A.nb, A.nb)
    xt = _solution(A.n, A.nb, rng)
    return BSR(A.n, A.nb, A.rowPtr, A.col, v.reshape(-1)), _matvec(A.rowPtr, A.col, v, xt), xt, f


def _jacobian_step(s, f, rng):
    """The same step as a scalar Jacobian with its well rows."""
    J, n = s.full, s.na * 3
    rows = np.repeat(np.arange(J.n), np.diff(J.rowPtr))
    v = np.where(rows < n, J.val * f[np.minimum(rows // 3, s.na - 1)], J.val)
    own = np.nonzero((rows < n) & (J.col < n) & (rows // 3 == J.col // 3))[0]
    v[own] += (1.0 - f[rows[own] // 3]) * s.acc.reshape(-1, 3, 3)[rows[own] // 3, rows[own] % 3, J.col[own] % 3]
    xt = np.concatenate([_solution(s.na, 3, rng), 50.0 * rng.standard_normal(s.nw)])
    return ScalarCSR(J.rowPtr, J.col, v), np.add.reduceat(v * xt[J.col], J.rowPtr[:-1]), xt


def _systems(case, seed):
    """(matrix, right-hand side, solution, row factor) of every system of the case for this seed."""
    rng = np.random.default_rng([seed, 17])
    return [_step(s, rng) for s in _geology(_frozen(case))], rng


def _grid_state(case, seed):
    """The assembler's model of the case's grids and a reservoir state drawn by the seed."""
    model, st = _assembly_model(_frozen(case))
    rng = np.random.default_rng([seed, 29])
    na = st["p"].size
    st = dict(st, p=st["p"] + 100.0 * rng.uniform(-1, 1) + 5.0 * rng.standard_normal(na), sw=np.clip(st["sw"] + 0.05 * rng.standard_normal(na), 0.2, 0.79),
              x=st["x"] * rng.uniform(0.8, 1.2, na), acc_old=st["acc_old"] * rng.uniform(0.97, 1.0))
    return model, st, float(rng.uniform(1.0, 30.0))


@functools.lru_cache(maxsize=2)
def _assembly_model(key):
    return synth.assembly_model(_geology(key))


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


# ---------------------------------------------------------------------------------------------------- prepare, run
def prepare(case, seed):
    kind = case["kind"]
    if kind == "assemble":
        model, st, dt = _grid_state(case, seed)
        asm = BlackOilAssembler(model)
        s = {k: _dev(v) for k, v in st.items()}
        return dict(case=case, asm=asm, dt=dt, J=torch.empty(asm.nnz, dtype=torch.float64, device="cuda"),
                    R=torch.empty(asm.nrows, dtype=torch.float64, device="cuda"), **s)
    first = _geology(_frozen(case))
    systems, rng = _systems(case, seed)
    s = dict(case=case, mats=[t[0] for t in systems], b=np.concatenate([t[1] for t in systems]))
    if kind == "serve":
        s["server"] = Server(slots=1, precision=case["precision"])
        for m, (_, b, _, _) in zip(first, systems):          # the server has seen these patterns before
            s["server"].hold(True)
            s.setdefault("ids", []).append(s["server"].submit(m.A, b, tol=TOL, maxit=MAXIT))
        s["server"].hold(False)
        for i in s.pop("ids"):
            s["server"].poll(i)
        s["bs"] = [t[1] for t in systems]
        return s
    opt = dict(precond=case.get("precond", "cpr"), precision=case.get("precision", "fp64"), krylov=case.get("krylov", "bicgstab"),
               restart=case.get("restart", 40))
    if kind == "generic":
        opt["krylov"] = "gmres"
    dev = s["dev"] = DeviceSolver(**opt)
    s["acc"] = first[0].acc if case.get("acc") else None
    if case.get("form") == "jacobian":
        f = first[0]
        s["jac"], s["b"], _ = _jacobian_step(f, systems[0][3], rng)
        s["size"] = (f.na, 3, f.nw)
        dev.set_jacobian(f.full, *s["size"])
        dev.setup(s["acc"])
        dev.solve_jacobian(s["b"], TOL, 2)
        return s
    if kind in ("apply", "spmv"):
        dev.set_batch(s["mats"])
        s["r"] = _dev(s["b"] / np.abs(s["b"]).max() if kind == "apply" else np.concatenate([t[2] for t in systems]))
        s["z"] = torch.empty_like(s["r"])
        s["stream"] = torch.cuda.ExternalStream(dev.stream)
        if kind == "apply":
            dev.setup()
        return s
    if kind == "ensemble":
        dev.set_batch([m.A for m in first])
    else:
        dev.set_matrix(first[0].A)
    dev.setup(s["acc"])
    dev.solve(s["b"], TOL, 2)                               # the Krylov vectors and graphs of a program that is under way
    return s


def run(s):
    case, kind = s["case"], s["case"]["kind"]
    if kind == "assemble":
        s["asm"].assemble_device(s["p"].data_ptr(), s["sw"].data_ptr(), s["x"].data_ptr(), s["state"].data_ptr(), s["acc_old"].data_ptr(), s["dt"],
                                 s["J"].data_ptr(), s["R"].data_ptr(), stream=torch.cuda.current_stream().cuda_stream)
        return dict(J=s["J"], R=s["R"])
    if kind == "serve":
        srv = s["server"]
        srv.hold(True)
        ids = [srv.submit(A, b, tol=TOL, maxit=MAXIT, copy=False) for A, b in zip(s["mats"], s["bs"])]
        srv.hold(False)
        return [srv.poll(i)[0] for i in ids]
    dev = s["dev"]
    if kind in ("apply", "spmv"):
        mine, its = torch.cuda.current_stream(), s["stream"]   # the caller's vectors are made and used on its own stream
        its.wait_stream(mine)
        (dev.precond_apply_device if kind == "apply" else dev.spmv_device)(s["r"].data_ptr(), s["z"].data_ptr())
        mine.wait_stream(its)
        return s["z"]
    if "jac" in s:
        dev.set_jacobian(s["jac"], *s["size"])
        dev.setup(s["acc"])
        return dev.solve_jacobian(s["b"], TOL, MAXIT)[0]
    if kind == "ensemble":
        dev.set_batch(s["mats"])
    else:
        dev.set_matrix(s["mats"][0])
    dev.setup(s["acc"])
    return dev.solve(s["b"], TOL, MAXIT)[0]


def work(case):
    """Matrix (or state and grid) in, vectors in and out, once each; the operations of one pass over the matrix, or of one
    evaluation of every cell and connection."""
    g = _geology(_frozen(case))
    if case["kind"] == "assemble":
        model, st = _assembly_model(_frozen(case))
        na, nconn, nnz = st["p"].size, model["conn_trans"].size, int(model["J_rowPtr"][-1])
        return dict(bytes=na * (3 * 8 + 1 + 3 * 8 + 8 + 4 * 3) + nconn * (4 * 4 + 8 + 8) + 8.0 * nnz + 24.0 * na, flops=400.0 * na + 120.0 * nconn)
    nb, n, nnzb = g[0].A.nb, sum(s.A.n for s in g), sum(s.A.nnzb for s in g)
    return dict(bytes=nnzb * (8.0 * nb * nb + 4) + n * (16.0 * nb + 4), flops=2.0 * nnzb * nb * nb)


# ---------------------------------------------------------------------------------------------------- exact
def exact(case, seed):
    if case["kind"] == "apply":
        return None                       # the AMG hierarchy and the incomplete factors are the library's own
    if case["kind"] == "assemble":
        return _assemble(*_grid_state(case, seed))
    systems, rng = _systems(case, seed)
    if case["kind"] == "spmv":
        return np.concatenate([t[1] for t in systems])
    if case.get("form") == "jacobian":
        return _jacobian_step(_geology(_frozen(case))[0], systems[0][3], rng)[2]
    if case["kind"] == "serve":
        return [t[2] for t in systems]
    return np.concatenate([t[2] for t in systems])


class _Dual:
    """A value per cell with its derivatives in the cell's three unknowns (p, Sw, x)."""

    def __init__(self, v, d=None):
        self.v, self.d = v, np.zeros((3,) + np.shape(v)) if d is None else d

    def __add__(self, o):
        return _Dual(self.v + o.v, self.d + o.d) if isinstance(o, _Dual) else _Dual(self.v + o, self.d)

    def __neg__(self):
        return _Dual(-self.v, -self.d)

    def __sub__(self, o):
        return self + (-o)

    def __mul__(self, o):
        return _Dual(self.v * o.v, self.d * o.v + self.v * o.d) if isinstance(o, _Dual) else _Dual(self.v * o, self.d * o)

    def __truediv__(self, o):
        return _Dual(self.v / o.v, (self.d - self.v / o.v * o.d) / o.v)

    def __getitem__(self, i):
        return _Dual(self.v[i], self.d[:, i])


def _pick(m, a, b):
    return _Dual(np.where(m, a.v, b.v), np.where(m, a.d, b.d))


def _table(x, y, clamp, v):
    i = np.clip(np.searchsorted(x, v, side="right") - 1, 0, x.size - 2)
    s = ((y[1:] - y[:-1]) / (x[1:] - x[:-1]))[i]
    f = y[i] + s * (v - x[i])
    if clamp:
        f = np.where(v <= x[0], y[0], np.where(v >= x[-1], y[-1], f))
        s = np.where((v <= x[0]) | (v >= x[-1]), 0.0, s)
    return f, s


def _assemble(z, st, dt):
    """The fully implicit black-oil Jacobian and residual (TPFA, live oil, upwinded mobilities) in plain numpy."""
    def tab(name, u):
        f, s = _table(z[name + "_x"], z[name + "_y"], int(z[name + "_clamp"][0]), u.v)
        return _Dual(f, s * u.d)

    def live(name, node, p, rs):
        R, xs, ys, off = z["liveRs"], z[name + "_x"], z[name + "_y"], z[name + "_off"]
        k = np.clip(np.searchsorted(R, rs, side="right") - 1, 0, R.size - 2)
        dp = p - _table(z["pbOfRs_x"], z["pbOfRs_y"], 0, rs)[0]
        at = np.stack([node[i] * _table(xs[off[i]:off[i + 1]], ys[off[i]:off[i + 1]], 0, dp)[0] for i in range(R.size)])
        c = np.arange(k.size)
        return at[k, c] + (rs - R[k]) / (R[k + 1] - R[k]) * (at[k + 1, c] - at[k, c])

    def live_ad(name, node, p, rs):
        hp, hr = 1e-4 * np.maximum(1.0, np.abs(p.v)), 1e-5 * np.maximum(1e-2, np.abs(rs.v))
        fp = (live(name, node, p.v + hp, rs.v) - live(name, node, p.v - hp, rs.v)) / (2 * hp)
        fr = (live(name, node, p.v, rs.v + hr) - live(name, node, p.v, rs.v - hr)) / (2 * hr)
        return _Dual(live(name, node, p.v, rs.v), fp * p.d + fr * rs.d)

    na = st["p"].size
    unit = np.eye(3)[:, :, None] * np.ones(na)
    P, Sw, X = _Dual(st["p"], unit[0]), _Dual(st["sw"], unit[1]), _Dual(st["x"], unit[2])
    zero, gas = _Dual(np.zeros(na)), st["state"] == 1
    Sg, rs = _pick(gas, X, zero), _pick(gas, tab("rsOfP", P), X)
    So = -Sw - Sg + 1.0
    series = lambda u: u + u * u * 0.5 + 1.0  # noqa: E731
    pv0, gfac = z["poreVolRef"], z["rhoSC"][2] * z["gasFactor"][0]
    pv = series((P + -z["rock"][0]) * z["rock"][1]) * pv0
    pref, bwr, cw, muw, cv = z["pvtw"]
    Pw, Pg = P - tab("pcow", Sw), P + tab("pcog", Sg)
    bw = series((Pw + -pref) * cw) * (1.0 / bwr)
    bo, bomu = live_ad("uB", z["bSat"], P, rs), live_ad("uBMu", z["bmuSat"], P, rs)
    dw = Sw + -z["swco"][0]
    dw = _pick(dw.v < 0, zero, dw)
    den, eff = Sg + dw, Sw + Sg
    flat = den.v < 1e-9
    kro = _pick(flat, tab("krow", eff), (Sg * tab("krog", eff + -z["swco"][0]) + dw * tab("krow", eff)) / _pick(flat, zero + 1.0, den))
    bg = tab("gasB", Pg)
    mob = [series((Pw + -pref) * (cw - cv)) * (1.0 / (bwr * muw)) * tab("krw", Sw), bomu * kro, tab("gasBMu", Pg) * tab("krg", Sg)]
    rho = [bw * z["rhoSC"][1], bo * (rs * gfac + z["rhoSC"][0]), bg * gfac]
    acc = [pv * bw * Sw, pv * bo * So, pv * (bg * Sg + rs * bo * So)]

    a, b = z["conn_a"], z["conn_b"]
    cells = np.concatenate([np.arange(na), a, b])                 # blocks: own, then both sides of every connection
    cols = np.concatenate([np.arange(na), b, a])
    blocks = np.zeros((cells.size, 3, 3))
    R = np.stack([(acc[e].v - st["acc_old"].reshape(-1, 3)[:, e]) / dt for e in range(3)], axis=1)
    for e in range(3):
        blocks[:na, e] = (acc[e].d / dt).T
    nc = a.size
    for p, (pres, terms) in enumerate(((Pw, [(0, mob[0])]), (P, [(1, mob[1]), (2, mob[1] * rs)]), (Pg, [(2, mob[2])]))):
        gd = z["gravity"][0] * z["conn_dDepth"]
        phi = pres.v[a] - pres.v[b] + 0.5 * (rho[p].v[a] + rho[p].v[b]) * gd
        da, db = pres.d[:, a] + 0.5 * rho[p].d[:, a] * gd, -pres.d[:, b] + 0.5 * rho[p].d[:, b] * gd
        up_a = phi >= 0
        for e, m in terms:
            T = z["conn_trans"]
            mu = m[np.where(up_a, a, b)]
            F = mu.v * phi * T
            Fa, Fb = (np.where(up_a, mu.d * phi, 0.0) + mu.v * da) * T, (np.where(up_a, 0.0, mu.d * phi) + mu.v * db) * T
            np.add.at(R[:, e], a, F)
            np.add.at(R[:, e], b, -F)
            blocks[na:na + nc, e] += Fb.T
            blocks[na + nc:, e] -= Fa.T
            for k in range(3):
                blocks[:na, e, k] += np.bincount(a, Fa[k], na) - np.bincount(b, Fb[k], na)
    order = np.lexsort((cols, cells))                             # the engine's layout: a cell's blocks in column order
    scale = dt / pv0
    blocks = (blocks * scale[cells][:, None, None])[order]
    count = np.bincount(cells, minlength=na)
    start = np.concatenate([[0], np.cumsum(count)])
    J = np.empty(int(z["J_rowPtr"][-1]))
    slot = np.arange(cells.size) - start[cells[order]]
    base = z["J_rowPtr"][:-1].reshape(na, 3)
    for e in range(3):
        for k in range(3):
            J[base[cells[order], e] + 3 * slot + k] = blocks[:, e, k]
    return dict(J=J, R=(R * scale[:, None]).reshape(-1))
