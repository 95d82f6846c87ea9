"""The work that users of this library have it do, as cases that can be timed.

Each case is one call (or the few calls a program makes together) of the public
interface on inputs that are already on the GPU:

    apply    Elastic.Fapply, FP64: a matrix-free operator application
    smooth   agb_op_fsmooth_f32: one Fsmooth (two damped-Jacobi sweeps) in FP32
    post     stress, strain, energy and the traction integral of a solution
    solve    Linear.solve from a zero guess: one elastic equilibrium
    newton   SetModel + Newton.solve: one time step whose moduli have changed
    rve      Batch.solve + mean stress + displacements of periodic RVEs
    conv     agb_conv3_tc: one layer of the learned correction, forward
    train    the backward pass and the Adam update of one such layer

listed() names the cases, draw() takes more of the same ranges, prepare()
makes what a program has in hand before the call, run() makes the call,
work() says what the call cannot do without, and exact() gives the result in
64 bits from plain torch.
"""
import ctypes
import math
import random

import torch

F64, F32, BF16 = torch.float64, torch.float32, torch.bfloat16
DEV = "cuda" if torch.cuda.is_available() else "cpu"
# box edges of solves: their multigrid hierarchies end at 2, 3 or 5 cells
EDGES = (16, 24, 32, 40, 48, 64, 80, 96, 128)
RVE_EDGES = (32, 48, 64, 80, 96)
GRIDS = (17, 33, 49, 65, 97, 129)
LAYERS = ((16, 16), (16, 32), (32, 32), (32, 64), (64, 64), (96, 32), (48, 16))


def listed():
    return [
        # one operator application inside a user's own Krylov loop on a small
        # box: latency and launches
        {"name": "apply_iso_16", "kind": "apply", "sym": "iso", "n0": 16, "n1": 16, "n2": 16, "cube": True},
        # the same on an ordinary box with odd, ragged edges, general
        # anisotropic moduli and cells that are not cubes
        {"name": "apply_cubic_ragged", "kind": "apply", "sym": "mm", "n0": 150, "n1": 83, "n2": 61, "cube": False},
        # a smoother call of a user's own multigrid, FP32, a box that fills the GPU
        {"name": "smooth_cubic_192", "kind": "smooth", "sym": "mm", "n0": 192, "n1": 160, "n2": 144, "cube": True},
        # output fields after a solve, written at every plot interval
        {"name": "post_cubic_128", "kind": "post", "sym": "mm", "n0": 128, "n1": 128, "n2": 128, "cube": True},
        # a small inclusion problem with the default solver (FP64 multigrid)
        {"name": "newton_sphere_32", "kind": "newton", "sym": "iso", "n0": 32, "n1": 32, "n2": 32, "cube": True,
         "mixed": False, "krylov": 0, "tol": 1e-10},
        # the 65^3-node inclusion with eigenstrain, FP64 multigrid
        {"name": "newton_sphere_64", "kind": "newton", "sym": "iso", "n0": 64, "n1": 64, "n2": 64, "cube": True,
         "mixed": False, "krylov": 0, "tol": 1e-10},
        # a polycrystal solved entirely in FP64
        {"name": "solve_poly_64_f64", "kind": "solve", "sym": "mm", "n0": 64, "n1": 64, "n2": 64, "cube": True,
         "mixed": False, "krylov": 0, "tol": 1e-9},
        # a time step of a polycrystal in a bar-shaped box, FP32 cycles under GCR
        {"name": "newton_poly_bar", "kind": "newton", "sym": "mm", "n0": 96, "n1": 96, "n2": 48, "cube": True,
         "mixed": True, "krylov": 8, "tol": 1e-9},
        # the 257^3-node polycrystal, FP32 cycles under GCR in FP64 refinement
        {"name": "solve_poly_256", "kind": "solve", "sym": "mm", "n0": 256, "n1": 256, "n2": 256, "cube": True,
         "mixed": True, "krylov": 8, "tol": 1e-8},
        # homogenization: periodic RVEs of several sizes solved together
        {"name": "rve_48", "kind": "rve", "count": 48, "mixed": True, "krylov": 8, "tol": 1e-10},
        # a wide layer of the learned correction on the finest nodal grid
        {"name": "conv_48x16_129", "kind": "conv", "g0": 129, "g1": 129, "g2": 129, "cin": 48, "cout": 16},
        # training one layer of the middle level
        {"name": "train_32x32_65", "kind": "train", "g0": 65, "g1": 65, "g2": 65, "cin": 32, "cout": 32},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(("apply", "smooth", "post", "solve", "newton", "rve", "conv", "train"))
    if kind in ("apply", "smooth", "post"):
        hi = 150 if kind == "apply" else 190 if kind == "smooth" else 128
        return {"kind": kind, "sym": rng.choice(("iso", "mm")), "n0": _log_int(rng, 12, hi),
                "n1": _log_int(rng, 12, hi), "n2": _log_int(rng, 12, hi), "cube": rng.random() < 0.6}
    if kind in ("solve", "newton"):
        mixed = rng.random() < 0.5
        sym = rng.choice(("iso", "mm"))
        pick = [e for e in EDGES if e <= (128 if mixed else 64) and (sym == "iso" or e % 5)]
        n = [rng.choice(pick)] * 3
        if (mixed or sym == "iso") and rng.random() < 0.5:   # a bar
            n = [rng.choice((48, 64, 96) if mixed else (32, 40, 48, 64)) for _ in range(3)]
        return {"kind": kind, "sym": sym, "n0": n[0], "n1": n[1], "n2": n[2], "cube": True, "mixed": mixed,
                "krylov": 8 if mixed else 0, "tol": 1e-9 if sym == "mm" else 1e-10}
    if kind == "rve":
        mixed = rng.random() < 0.7
        return {"kind": kind, "count": rng.randint(4, 48 if mixed else 8), "mixed": mixed,
                "krylov": 8 if mixed else 0, "tol": 1e-10}
    cin, cout = rng.choice(LAYERS)
    pick = GRIDS if kind == "conv" else GRIDS[:5]
    return {"kind": kind, "g0": rng.choice(pick), "g1": rng.choice(pick), "g2": rng.choice(pick), "cin": cin,
            "cout": cout}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _cells(case):
    return [case["n0"], case["n1"], case["n2"]]


def _dx(case):
    """Cubic cells of a box whose longest edge is 1, or a unit cube of ragged cells."""
    n = _cells(case)
    return [1.0 / max(n)] * 3 if case["cube"] else [1.0 / v for v in n]


def _coords(case):
    n, dx = _cells(case), _dx(case)
    ax = [torch.arange(n[d] + 1, dtype=F64, device=DEV) * dx[d] for d in range(3)]
    return ax[0][None, None, :], ax[1][None, :, None], ax[2][:, None, None]


def _polycrystal(case, seed, grains=64):
    """Cubic Voronoi polycrystal, uniformly random orientations: 21 doubles per node."""
    from alamo_gb300 import microstructure as M
    _, table = M.voronoi_seeds(grains, seed=int(seed))
    rng = random.Random(int(seed))
    n, dx = _cells(case), _dx(case)
    X, Y, Z = _coords(case)
    best, ids = None, None
    for g in range(grains):
        c = [rng.random() * n[d] * dx[d] for d in range(3)]
        d2 = (X - c[0]) ** 2 + (Y - c[1]) ** 2 + (Z - c[2]) ** 2
        if best is None:
            best, ids = d2, torch.zeros_like(d2, dtype=torch.int64)
        else:
            near = d2 < best
            best = torch.where(near, d2, best)
            ids = torch.where(near, torch.full_like(ids, g), ids)
    return torch.from_numpy(table).to(DEV)[ids.reshape(-1)].reshape(-1).contiguous()


def _inclusion(case, seed):
    """A stiff sphere with a diffuse boundary in an isotropic matrix: lambda, mu per node, and its weight."""
    rng = random.Random(int(seed))
    n, dx = _cells(case), _dx(case)
    X, Y, Z = _coords(case)
    c = [n[d] * dx[d] * rng.uniform(0.45, 0.55) for d in range(3)]
    r = torch.sqrt((X - c[0]) ** 2 + (Y - c[1]) ** 2 + (Z - c[2]) ** 2)
    radius = min(n[d] * dx[d] for d in range(3)) * rng.uniform(0.2, 0.3)
    eta = (0.5 * (1 - torch.tanh((r - radius) / (2 * max(dx))))).reshape(-1)
    stiff = rng.uniform(8, 12)
    one = 1 + (stiff - 1) * eta
    return torch.stack((one, one), 1).reshape(-1).contiguous(), eta


def _moduli(case, seed):
    return _polycrystal(case, seed) if case["sym"] == "mm" else _inclusion(case, seed)[0]


def _displacement(case, seed):
    """A stretched box with smooth and rough parts, as an iterate of a solve has them."""
    n, dx = _cells(case), _dx(case)
    X, Y, Z = _coords(case)
    rng = random.Random(int(seed) + 1)
    u = []
    for c in range(3):
        f = 0.01 * (X if c == 0 else -0.3 * (Y if c == 1 else Z)) + 0 * X + 0 * Y + 0 * Z
        for _ in range(3):
            w = [rng.uniform(1, 9) for _ in range(3)]
            f = f + 1e-3 * torch.sin(w[0] * X + w[1] * Y + w[2] * Z + rng.uniform(0, 6))
        u.append(f)
    u = torch.stack(u).reshape(-1)
    return (u + 1e-6 * torch.randn(u.numel(), dtype=F64, device=DEV, generator=_gen(seed))).contiguous()


def _bc():
    from alamo_gb300 import TensionTest
    return TensionTest("uniaxial_stress", disp=0.01)


def _operator(case, ddw):
    from alamo_gb300 import Constant, Elastic
    op = Elastic(_cells(case), _dx(case), "majorminor" if case["sym"] == "mm" else "isotropic")
    clamped = case["sym"] == "iso" and case["kind"] in ("newton", "solve")
    op.SetBC(Constant() if clamped else _bc())
    op.SetModel(ddw)
    return op


def _eigenstrain(case, seed):
    _, eta = _inclusion(case, seed)
    F0 = torch.zeros((eta.numel(), 9), dtype=F64, device=DEV)
    F0[:, 0] = F0[:, 4] = F0[:, 8] = 1e-3 * eta
    return F0.reshape(-1).contiguous()


def _rve_draws(case, seed):
    """Edges, inclusion tables and macroscopic eigenstrains of a batch."""
    from alamo_gb300 import microstructure as M
    return [M.rve_params(q, seed=4242 + int(seed), edges=(RVE_EDGES[q % len(RVE_EDGES)],)) for q in range(case["count"])]


def _ellipsoids(n, table, width=2.0):
    """lambda = mu of an RVE: log-stiffness with a tanh profile across each ellipsoid's surface."""
    x = torch.arange(n + 1, dtype=F64, device=DEV) / n
    Z, Y, X = torch.meshgrid(x, x, x, indexing="ij")
    P = torch.stack((X, Y, Z), -1).reshape(-1, 3)
    logc = torch.zeros(P.shape[0], dtype=F64, device=DEV)
    for row in torch.from_numpy(table).to(DEV):
        d = P - row[0:3]
        d = d - torch.round(d)
        y = d @ row[6:15].reshape(3, 3)
        s = (torch.sqrt(torch.sum((y / row[3:6]) ** 2, 1)) - 1) * row[3:6].mean()
        w = width * max(1.0, float(row[15]) / math.log(10.0))
        logc = torch.maximum(logc, 0.5 * (1 - torch.tanh(s * n / w)) * row[15])
    one = torch.exp(logc)
    return torch.stack((one, one), 1).reshape(-1).contiguous()


def _grid(case):
    return [case["g0"], case["g1"], case["g2"]]


def _layer(case, seed):
    """Input activations (after a ReLU), weights as a network is initialised, biases."""
    g = _gen(seed)
    V, ci, co = math.prod(_grid(case)), case["cin"], case["cout"]
    x = torch.relu(torch.randn(V, ci, device=DEV, generator=g)).to(BF16)
    w = torch.randn(27, co, ci, device=DEV, generator=g) * math.sqrt(2.0 / (27 * ci))
    b = 0.1 * torch.randn(co, device=DEV, generator=g)
    return x, w, b


def _training(case, seed):
    """A layer in the middle of its training: gradient at its output, saved
    activations, Adam's moments."""
    x, w, b = _layer(case, seed)
    g = _gen(seed + 1)
    V, co = x.shape[0], case["cout"]
    dy = (torch.randn(V, co, device=DEV, generator=g) / math.sqrt(V)).to(BF16)
    act = torch.relu(torch.randn(V, co, device=DEV, generator=g)).to(BF16)
    m = 0.1 * torch.randn(w.shape, device=DEV, generator=g)
    v = 0.5 + torch.rand(w.shape, device=DEV, generator=g)
    return {"x": x, "w": w, "b": b, "dy": dy, "act": act, "m": m, "v": v}


# ---------------------------------------------------------------------------
# prepare and run
# ---------------------------------------------------------------------------
def _p(t):
    return ctypes.c_void_p(t.data_ptr())


def _i3(v):
    return (ctypes.c_int * 3)(*v)


def _stream():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


def prepare(case, seed):
    from alamo_gb300._lib import check, lib
    L = lib()
    kind = case["kind"]
    s = {"kind": kind, "L": L, "check": check, "case": case}
    if kind in ("apply", "smooth", "post"):
        s["ddw"] = _moduli(case, seed)
        s["op"] = op = _operator(case, s["ddw"])
        s["u"] = _displacement(case, seed)
        N = s["u"].numel() // 3
        if kind != "post":
            op.prepareForSolve()
        if kind == "apply":
            s["f"] = torch.empty_like(s["u"])
        elif kind == "smooth":
            s["b"] = op.BCInit(torch.zeros_like(s["u"])).to(F32)
            s["u"] = s["u"].to(F32)
        else:
            s["sigma"] = torch.empty(9 * N, dtype=F64, device=DEV)
            s["eps"] = torch.empty(9 * N, dtype=F64, device=DEV)
            s["energy"] = torch.empty(N, dtype=F64, device=DEV)
    elif kind in ("solve", "newton"):
        from alamo_gb300 import Linear, Newton
        s["ddw"] = _moduli(case, seed)
        s["op"] = op = _operator(case, s["ddw"])
        N = math.prod(v + 1 for v in _cells(case))
        s["u"] = torch.zeros(3 * N, dtype=F64, device=DEV)
        s["b"] = op.BCInit(torch.zeros_like(s["u"]))
        s["F0"] = _eigenstrain(case, seed) if case["sym"] == "iso" else None
        if kind == "solve":
            rhs = torch.empty_like(s["u"])
            check(L.agb_newton_rhs(op.h, _p(s["F0"]) if s["F0"] is not None else None, _p(s["u"]), _p(s["b"]),
                                   _p(rhs), 1))
            s["b"] = rhs
        s["solver"] = (Linear if kind == "solve" else Newton)(op, precision=1 if case["mixed"] else 0,
                                                              krylov=case["krylov"])
    elif kind == "rve":
        import numpy as np
        from alamo_gb300.batch import Batch
        draws = _rve_draws(case, seed)
        s["batch"] = bt = Batch([(n,) * 3 for n, _, _ in draws], precision=1 if case["mixed"] else 0,
                                krylov=case["krylov"])
        for q, (n, table, _) in enumerate(draws):
            bt.SetModel(q, _ellipsoids(n, table))
        bt.SetEigenstrain(np.stack([F0 for _, _, F0 in draws]))
        s["u"] = torch.empty(sum(3 * bt.nodes(q) for q in range(bt.np)), dtype=F64, device=DEV)
    else:
        s["g"] = _i3(_grid(case))
        ci, co = case["cin"], case["cout"]
        V = math.prod(_grid(case))
        if kind == "conv":
            s["x"], w, s["b"] = _layer(case, seed)
            s["wp"] = torch.empty(27 * co * ci, dtype=BF16, device=DEV)
            check(L.agb_conv3_tc_pack(ci, co, _p(w.to(BF16).contiguous()), co, 0, _p(s["wp"]), _stream()))
            s["y"] = torch.empty((V, co), dtype=BF16, device=DEV)
        else:
            s.update(_training(case, seed))
            s["wb"] = s["w"].to(BF16)
            s["wt"] = torch.empty(27 * co * ci, dtype=BF16, device=DEV)
            s["wp"] = torch.empty(27 * co * ci, dtype=BF16, device=DEV)
            s["dx"] = torch.empty((V, ci), dtype=BF16, device=DEV)
            s["dw"] = torch.empty((27, co, ci), device=DEV)
            s["db"] = torch.empty(co, device=DEV)
            s["step"] = 100
    return s


def run(s):
    L, check, kind = s["L"], s["check"], s["kind"]
    if kind == "apply":
        s["op"].Fapply(0, s["u"], out=s["f"])
        return s["f"]
    if kind == "smooth":
        check(L.agb_op_fsmooth_f32(s["op"].h, 0, _p(s["u"]), _p(s["b"]), 1))
        return s["u"]
    if kind == "post":
        check(L.agb_stress(s["op"].h, None, _p(s["u"]), _p(s["sigma"]), 1))
        check(L.agb_strain_energy(s["op"].h, _p(s["u"]), _p(s["eps"]), _p(s["energy"]), 1))
        return {"sigma": s["sigma"], "eps": s["eps"], "energy": s["energy"], "traction": s["op"].TractionXhi(s["u"])}
    if kind == "solve":
        s["u"].zero_()
        s["solver"].solve(s["u"], s["b"], s["case"]["tol"], 0.0)
        return s["u"]
    if kind == "newton":
        s["op"].SetModel(s["ddw"])
        s["u"].zero_()
        s["solver"].solve(s["u"], s["b"], s["F0"], s["case"]["tol"], 0.0)
        return s["u"]
    if kind == "rve":
        bt = s["batch"]
        bt.solve(s["case"]["tol"], 0.0)
        at = s["u"].data_ptr()
        for q in range(bt.np):
            check(L.agb_batch_get_solution(bt.h, q, ctypes.c_void_p(at), 1))
            at += 24 * bt.nodes(q)
        return {"u": s["u"], "stress": bt.mean_stress()}
    ci, co, st = s["case"]["cin"], s["case"]["cout"], _stream()
    if kind == "conv":
        check(L.agb_conv3_tc(s["g"], ci, co, _p(s["x"]), ci, 0, _p(s["wp"]), _p(s["b"]), _p(s["y"]), co, 0, 0, 1, st))
        return s["y"]
    V = s["x"].shape[0]
    s["dw"].zero_()
    s["db"].zero_()
    check(L.agb_axpby_mask(V, co, _p(s["dy"]), co, 0, _p(s["dy"]), co, 0, None, 0, 0, 0.0, _p(s["act"]), co, 0, st))
    check(L.agb_conv3_wgrad0(s["g"], ci, co, _p(s["x"]), ci, 0, _p(s["dy"]), co, 0, _p(s["dw"]), _p(s["db"]), st))
    check(L.agb_conv3_flip(ci, co, _p(s["wb"]), _p(s["wt"]), st))
    c0 = 0
    while c0 < ci:
        w = min(64, ci - c0)
        check(L.agb_conv3_tc_pack(co, w, _p(s["wt"]), ci, c0, _p(s["wp"]), st))
        check(L.agb_conv3_tc(s["g"], co, w, _p(s["dy"]), co, 0, _p(s["wp"]), None, _p(s["dx"]), ci, c0, 0, 0, st))
        c0 += w
    check(L.agb_adam_step(s["w"].numel(), _p(s["w"]), _p(s["dw"]), _p(s["m"]), _p(s["v"]), _p(s["wb"]), 1e-5, 0.9,
                          0.999, 1e-8, s["step"], st))
    return {k: s[k] for k in ("dw", "db", "dx", "w", "m", "v", "wb")}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind in ("conv", "train"):
        V, ci, co = math.prod(_grid(case)), case["cin"], case["cout"]
        mac = 2.0 * 27 * ci * co * V
        if kind == "conv":
            return {"bytes": 2.0 * V * (ci + co) + 54.0 * ci * co, "flops": mac}
        # x, dy (read, written masked), saved activations, dx; weights, moments, gradients
        return {"bytes": 2.0 * V * (2 * ci + 3 * co) + 27.0 * ci * co * (4 * 7 + 2 * 2), "flops": 2 * mac}
    if kind == "rve":
        # one residual of each mean RVE (x, b, moduli read, r written), as many
        # as the least a solve takes: one FP32 cycle of two sweeps a decade
        N = case["count"] * sum((n + 1) ** 3 for n in RVE_EDGES) / len(RVE_EDGES)
        sweeps = 2.0 * -math.log10(case["tol"])
        size = 4 if case["mixed"] else 8
        return {"bytes": N * (sweeps * size * (2 + 12) + 24), "flops": N * sweeps * 150}
    nc = 21 if case["sym"] == "mm" else 2
    N = math.prod(v + 1 for v in _cells(case))
    per = 230 if nc == 21 else 130   # operations of one row
    if kind == "apply":
        return {"bytes": 8.0 * N * (nc + 6), "flops": float(N * per)}
    if kind == "smooth":
        return {"bytes": 4.0 * N * (nc + 12), "flops": 2.0 * N * per}
    if kind == "post":
        return {"bytes": 8.0 * N * (nc + 3 + 9 + 9 + 1), "flops": float(N * 100)}
    # a solve: the moduli once, the rhs and the solution, and two sweeps of the
    # finest level a decade in the precision of the cycles
    sweeps = 2.0 * -math.log10(case["tol"])
    size = 4 if case["mixed"] else 8
    return {"bytes": N * (8.0 * (nc + 6) + sweeps * size * (nc + 12)), "flops": N * sweeps * per}


# ---------------------------------------------------------------------------
# results in 64 bits, from plain torch
# ---------------------------------------------------------------------------
SLOT = ((0, 1, 2, 3, 4, 5), (1, 6, 7, 8, 9, 10), (2, 7, 11, 12, 13, 14), (3, 8, 12, 15, 16, 17),
        (4, 9, 13, 16, 18, 19), (5, 10, 14, 17, 19, 20))   # pairs 00, 01, 02, 11, 12, 22
PAIR = ((0, 1, 2), (1, 3, 4), (2, 4, 5))
DISP = 0


class _Box:
    """The nodal elastic operator of one box with no periodic direction."""

    def __init__(self, case, ddw, bc):
        n = _cells(case)
        self.shape = [n[2] + 1, n[1] + 1, n[0] + 1]
        self.dx, self.bc = _dx(case), bc
        iso = ddw.numel() == 2 * math.prod(self.shape)
        a = ddw.reshape(self.shape + [-1]).movedim(-1, 0)
        if iso:
            z = torch.zeros_like(a[0])
            lam, mu = a[0], a[1]
            d = lam + 2 * mu
            self.c = [[d, z, z, lam, z, lam], [z, mu, z, z, z, z], [z, z, mu, z, z, z], [lam, z, z, d, z, lam],
                      [z, z, z, z, mu, z], [lam, z, z, lam, z, d]]
        else:
            self.c = [[a[SLOT[p][q]] for q in range(6)] for p in range(6)]

    @staticmethod
    def shift(f, d, s):
        """f at the neighbour s steps along direction d (the edge value repeated)."""
        ax = 2 - d
        m = f.shape[ax]
        at = torch.clamp(torch.arange(m, device=f.device) + s, 0, m - 1)
        return f.index_select(ax, at)

    def grad(self, f, d):
        """Central difference, one-sided on the two faces."""
        ax = 2 - d
        g = (self.shift(f, d, 1) - self.shift(f, d, -1)) / (2 * self.dx[d])
        for at in (0, f.shape[ax] - 1):
            g.select(ax, at).mul_(2)
        return g

    def stress(self, u, F0=None):
        """C : (grad u - F0), and grad u."""
        G = [[self.grad(u[p], d) for d in range(3)] for p in range(3)]
        E = G if F0 is None else [[G[p][d] - F0[3 * p + d] for d in range(3)] for p in range(3)]
        e = [E[0][0], E[0][1] + E[1][0], E[0][2] + E[2][0], E[1][1], E[1][2] + E[2][1], E[2][2]]
        v = [sum(self.c[p][q] * e[q] for q in range(6)) for p in range(6)]
        return [[v[PAIR[p][d]] for d in range(3)] for p in range(3)], G

    def regions(self):
        """Every face, edge and corner: its index in the BC tables, its nodes, its normal."""
        from alamo_gb300 import FACE
        names = ("xlo", "xhi", "ylo", "yhi", "zlo", "zhi")
        for face, at in FACE.items():
            parts = [names.index(face[i:i + 3]) for i in range(0, len(face), 3)]
            scale = {1: 1.0, 2: 0.70710678118, 3: 0.57735026919}[len(parts)]
            nrm, ix = [0.0, 0.0, 0.0], [slice(1, -1)] * 3
            for p in parts:
                nrm[p // 2] = scale if p % 2 else -scale
                ix[2 - p // 2] = -1 if p % 2 else 0
            yield at, tuple(ix), nrm

    def boundary(self, f, u, S, G):
        """The rows of the boundary nodes: the displacement or the traction."""
        for at, ix, nrm in self.regions():
            for c in range(3):
                f[c][ix] = u[c][ix] if int(self.bc.type[at, c]) == DISP else sum(S[c][d][ix] * nrm[d] for d in range(3))
        return f

    def boundary_values(self):
        """The right-hand side that holds the boundary conditions' values, zero inside."""
        b = torch.zeros([3] + self.shape, dtype=F64, device=DEV)
        for at, ix, _ in self.regions():
            for c in range(3):
                b[c][ix] = float(self.bc.val[at, c])
        return b.reshape(-1)

    def apply(self, flat):
        """A u: C : grad grad u + (div C) : grad u inside, the boundary rows outside."""
        u = flat.reshape([3] + self.shape)
        H = {}
        for p in range(3):
            for a in range(3):
                H[p, a, a] = (self.shift(u[p], a, 1) - 2 * u[p] + self.shift(u[p], a, -1)) / self.dx[a] ** 2
                for b in range(a):
                    H[p, a, b] = H[p, b, a] = (
                        self.shift(self.shift(u[p], a, 1), b, 1) + self.shift(self.shift(u[p], a, -1), b, -1)
                        - self.shift(self.shift(u[p], a, 1), b, -1) - self.shift(self.shift(u[p], a, -1), b, 1)
                    ) / (4 * self.dx[a] * self.dx[b])
        S, G = self.stress(u)
        e = [G[0][0], G[0][1] + G[1][0], G[0][2] + G[2][0], G[1][1], G[1][2] + G[2][1], G[2][2]]
        f = [torch.zeros_like(u[0]) for _ in range(3)]
        for i in range(3):
            for j in range(3):
                row = self.c[PAIR[i][j]]
                he = [H[0, 0, j], H[0, 1, j] + H[1, 0, j], H[0, 2, j] + H[2, 0, j], H[1, 1, j],
                      H[1, 2, j] + H[2, 1, j], H[2, 2, j]]
                for q in range(6):
                    dc = (self.shift(row[q], j, 1) - self.shift(row[q], j, -1)) / (2 * self.dx[j])
                    f[i] = f[i] + row[q] * he[q] + dc * e[q]
        return torch.stack(self.boundary(f, u, S, G)).reshape(-1)

    def diagonal(self):
        """The diagonal: one probe for each component and each colour of nodes three apart."""
        D = torch.zeros([3] + self.shape, dtype=F64, device=DEV)
        for c in range(3):
            for q in range(27):
                at = (slice(q // 9, None, 3), slice(q // 3 % 3, None, 3), slice(q % 3, None, 3))
                e = torch.zeros_like(D)
                e[c][at] = 1
                D[c][at] = self.apply(e.reshape(-1)).reshape(D.shape)[c][at]
        return D.reshape(-1)

    def newton_rhs(self, b, F0):
        """b - div(C : (0 - F0)) inside, b - the boundary rows of that stress outside, at u = 0."""
        u = torch.zeros([3] + self.shape, dtype=F64, device=DEV)
        S, G = self.stress(u, F0.reshape(self.shape + [9]).movedim(-1, 0))
        f = [sum((self.shift(S[r][d], d, 1) - self.shift(S[r][d], d, -1)) / (2 * self.dx[d]) for d in range(3))
             for r in range(3)]
        return b - torch.stack(self.boundary(f, u, S, G)).reshape(-1)

    def solve(self, rhs, tol=1e-13, most=6000):
        """A u = rhs by BiCGStab on the system scaled by the diagonal."""
        D = self.diagonal()
        x, r = torch.zeros_like(rhs), rhs / D
        x_best, best = x, float("inf")
        for _ in range(4):   # restarted from the true residual
            r = (rhs - self.apply(x)) / D
            now = float(r.norm() / (rhs / D).norm())
            if now < best:
                x_best, best = x, now
            if best < tol:
                break
            # a random shadow residual: that of a boundary load alone breaks the recurrence down
            r0 = torch.randn(r.numel(), dtype=F64, device=DEV, generator=_gen(7))
            p, rho = r.clone(), r0 @ r
            x = x_best.clone()
            for it in range(most):
                v = self.apply(p) / D
                alpha = rho / (r0 @ v)
                s = r - alpha * v
                t = self.apply(s) / D
                om = (t @ s) / (t @ t)
                x = x + alpha * p + om * s
                r = s - om * t
                new = r0 @ r
                p = r + (new / rho) * (alpha / om) * (p - om * v)
                rho = new
                if it % 10 == 9 and float(r.norm() / (rhs / D).norm()) < 0.3 * tol:
                    break
        return x_best


def _conv64(case, x, w):
    """sum over the 27 taps of x shifted by the tap times w, zeros outside the grid; [z][y][x][cout]."""
    g = _grid(case)
    xp = torch.nn.functional.pad(x.to(F64).reshape(g[2], g[1], g[0], -1), (0, 0, 1, 1, 1, 1, 1, 1))
    w = w.to(F64)
    out = 0
    for t in range(27):
        dz, dy, dx = t // 9, t // 3 % 3, t % 3
        out = out + xp[dz:dz + g[2], dy:dy + g[1], dx:dx + g[0]] @ w[t].T
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "rve":
        return None   # thousands of Krylov iterations for each of many boxes
    if kind in ("conv", "train"):
        V, ci, co = math.prod(_grid(case)), case["cin"], case["cout"]
        if kind == "conv":
            x, w, b = _layer(case, seed)
            return torch.relu(_conv64(case, x, w.to(BF16)) + b.to(F64)).reshape(V, co)
        t = _training(case, seed)
        g = _grid(case)
        dy = torch.where(t["act"] > 0, t["dy"], torch.zeros_like(t["dy"])).to(F64)
        xp = torch.nn.functional.pad(t["x"].to(F64).reshape(g[2], g[1], g[0], ci), (0, 0, 1, 1, 1, 1, 1, 1))
        dw = torch.stack([dy.T @ xp[q // 9:q // 9 + g[2], q // 3 % 3:q // 3 % 3 + g[1], q % 3:q % 3 + g[0]].reshape(V, ci)
                          for q in range(27)])
        db = dy.sum(0)
        dx = _conv64(case, dy, t["w"].to(BF16).flip(0).transpose(1, 2)).reshape(V, ci)
        m = 0.9 * t["m"].to(F64) + 0.1 * dw
        v = 0.999 * t["v"].to(F64) + 0.001 * dw * dw
        w = t["w"].to(F64) - 1e-5 * (m / (1 - 0.9 ** 100)) / (torch.sqrt(v / (1 - 0.999 ** 100)) + 1e-8)
        return {"dw": dw, "db": db, "dx": dx, "w": w, "m": m, "v": v, "wb": w}
    clamped = case["sym"] == "iso" and kind in ("newton", "solve")
    if kind in ("solve", "newton") and math.prod(_cells(case)) > 40 ** 3:
        return None   # Krylov iterations without multigrid take minutes
    from alamo_gb300 import Constant
    box = _Box(case, _moduli(case, seed), Constant() if clamped else _bc())
    if kind == "apply":
        return box.apply(_displacement(case, seed))
    if kind == "smooth":
        x = _displacement(case, seed).to(F32).to(F64)
        b = box.boundary_values().to(F32).to(F64)
        D = box.diagonal()
        for _ in range(2):
            x = x + (2.0 / 3.0) * (b - box.apply(x)) / D
        return x
    if kind == "post":
        u = _displacement(case, seed).reshape([3] + box.shape)
        S, G = box.stress(u)
        E = [[0.5 * (G[p][d] + G[d][p]) for d in range(3)] for p in range(3)]
        flat = lambda T: torch.stack([T[p][d] for p in range(3) for d in range(3)], -1).reshape(-1)  # noqa: E731
        face = torch.stack([S[r][0][:, :, -1] for r in range(3)])
        quad = 0.25 * (face[:, 1:, 1:] + face[:, 1:, :-1] + face[:, :-1, 1:] + face[:, :-1, :-1])
        return {"sigma": flat(S), "eps": flat(E),
                "energy": sum(0.5 * S[p][d] * E[p][d] for p in range(3) for d in range(3)).reshape(-1),
                "traction": quad.sum((1, 2)) * box.dx[1] * box.dx[2]}
    b = box.boundary_values()
    return box.solve(b if case["sym"] == "mm" else box.newton_rhs(b, _eigenstrain(case, seed)))
