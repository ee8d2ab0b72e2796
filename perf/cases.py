"""The work that users of the framework have it do, as cases that can be timed
and whose outputs can be compared.

A case is one time step of a model (or of an ensemble, or a remesh and the step
after it, or one evaluation of the guess network with its gradient) through the
package's public classes.  Models are stepped as a host program steps them:
`Model.step_host` takes the temperature of the step from host memory and gives
T, V and P back, so that pass after pass the flow evolves as it does in a run
(warm starts included) and nothing of a pass can be reused for the next.

The solvers stop on a residual; two correct solvers stop at different points
within that tolerance.  The converged solvers therefore run here to a Stokes
residual of 1e-12 (on the largest meshes to what FP64 allows), the tolerance this
repository solves to where fields are compared to nine digits or more, instead of
the 1e-8 of a production run: the same kernels, some passes of refinement more.
The pressure of a closed box is determined up to a constant and is given with
its mean removed, as this repository's comparisons take it.
"""
import math

import numpy as np
import torch

from mantle_convection_lab_gb300 import api, ensemble
from mantle_convection_lab_gb300.amr import CFG2_INPUT, uniform_leaves
from mantle_convection_lab_gb300.api import Cnn, Config, Ensemble, Model

CFG1_INPUT = ensemble.BASE_INPUT.replace("cfg3_mg_1024", "cfg1_plain_64")
CFG3_INPUT = ensemble.BASE_INPUT


def _rtol(side):
    """The rounding of the FP64 residual grows with the square of the elements per side."""
    return max(1e-12, 6e-18 * side * side)


def listed():
    return [
        # the smallest call: the reference's own iteration in FP64 on a coarse grid, as
        # a first look at a parameter set or a unit test runs it; launches and latency
        {"name": "replica_16", "kind": "step", "solver": "replica", "side": 16, "rayleigh": 1e4, "contrast": 1.0},
        # configuration 1, the plain FP64 run of the reference's iteration
        {"name": "replica_64", "kind": "step", "solver": "replica", "side": 64, "rayleigh": 1e5, "contrast": 1.0},
        # a small convection model with temperature-dependent viscosity, solved to
        # a true residual with the mixed-precision MINRES solver
        {"name": "mixed_64", "kind": "step", "solver": "mixed", "side": 64, "rayleigh": 1e6, "contrast": 1e3},
        # configuration 3 at the size it is developed on
        {"name": "mixed_256", "kind": "step", "solver": "mixed", "side": 256, "rayleigh": 1e8, "contrast": 1e5},
        # configuration 3, the benchmark's default workload and the largest uniform mesh
        {"name": "mixed_1024", "kind": "step", "solver": "mixed", "side": 1024, "rayleigh": 1e8, "contrast": 1e5},
        # the converged solver without FP32 (precision=fp64mg): what results are checked against
        {"name": "fp64mg_128", "kind": "step", "solver": "fp64mg", "side": 128, "rayleigh": 1e6, "contrast": 1e3},
        # the other correction solve, and the one a .input takes if it names none:
        # Uzawa with an inner multigrid-preconditioned CG, in mixed precision
        {"name": "uzawa_128", "kind": "step", "solver": "uzawa", "side": 128, "rayleigh": 1e5, "contrast": 1e2},
        # configuration 2: a step on a quadtree mesh with hanging nodes
        {"name": "amr_128", "kind": "amr", "base": 128, "extra": 3, "rayleigh": 1e7, "contrast": 1e4},
        # ... and its remesh with the first step on the new mesh
        {"name": "remesh_64", "kind": "remesh", "base": 64, "extra": 2, "rayleigh": 1e6, "contrast": 1e2},
        # configuration 4: a parameter sweep, one batched launch over models of mixed sizes
        {"name": "ensemble_24", "kind": "ensemble", "members": 24, "draw_seed": 4, "largest": 128, "refine": 0},
        # ... with |grad T| refinement of some of the members
        {"name": "ensemble_amr_8", "kind": "ensemble", "members": 8, "draw_seed": 11, "largest": 64, "refine": 1},
        # the learned guess's network on a training batch: forward, and loss with gradient
        {"name": "guess_net", "kind": "net", "batch": 8, "height": 129, "width": 129, "channels": 32, "depth": 6},
    ]


def _logu(rng, lo, hi):
    return 10.0 ** rng.uniform(math.log10(lo), math.log10(hi))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "step", "amr", "remesh", "ensemble", "net"])
    if kind == "step":
        solver = rng.choice(["replica", "mixed", "mixed", "mixed", "fp64mg", "uzawa"])
        sides = {"replica": [16, 32, 64], "mixed": [32, 64, 128, 256, 512, 1024], "fp64mg": [32, 64, 128],
                 "uzawa": [32, 64, 128]}[solver]
        top = {"replica": (1e5, 1.0), "mixed": (1e8, 1e5), "fp64mg": (1e7, 1e4), "uzawa": (1e6, 1e2)}[solver]
        return {"kind": kind, "solver": solver, "side": rng.choice(sides), "rayleigh": _logu(rng, 1e4, top[0]),
                "contrast": _logu(rng, 1.0, top[1]) if top[1] > 1.0 else 1.0}
    if kind in ("amr", "remesh"):
        base = rng.choice([32, 64, 128])
        return {"kind": kind, "base": base, "extra": rng.choice([1, 2, 3]) if base < 128 else rng.choice([1, 2]),
                "rayleigh": _logu(rng, 1e5, 1e7), "contrast": _logu(rng, 1.0, 1e4 if kind == "amr" else 1e2)}
    if kind == "ensemble":
        refine = rng.choice([0, 0, 1])
        return {"kind": kind, "members": rng.randint(3, 24) if not refine else rng.randint(3, 8),
                "draw_seed": rng.randint(1, 10 ** 6), "largest": rng.choice([32, 64, 128]) if not refine else 64,
                "refine": refine}
    return {"kind": kind, "batch": rng.randint(1, 8), "height": rng.randint(17, 160), "width": rng.randint(17, 160),
            "channels": rng.choice([16, 32]), "depth": rng.randint(3, 6)}


# ---- inputs ---------------------------------------------------------------------
def _temperature(x, z, seed, layers):
    """Initial temperature at node (x, z) of the unit box (z = 0: T = 1): the
    conductive profile with a cosine mode, or tanh boundary layers, with seeded
    modes."""
    r = np.random.default_rng(seed)
    if layers:
        d = 0.02
        T = 0.5 + 0.5 * (1.0 - np.tanh(z / d)) - 0.5 * (1.0 - np.tanh((1.0 - z) / d))
        amp = 0.005
    else:
        T = (1.0 - z) + 0.02 * np.sin(np.pi * (1.0 - z)) * np.cos(np.pi * x)
        amp = 0.005
    for _ in range(8):
        p, q, ph = r.integers(1, 5), r.integers(1, 5), r.uniform(0, 2 * np.pi)
        T = T + amp * np.cos(p * np.pi * x + ph) * np.sin(q * np.pi * z)
    T = np.where(z <= 0.0, 1.0, np.where(z >= 1.0, 0.0, T))
    return np.ascontiguousarray(T)


def _step_config(case):
    """configuration 1's input for the replica, configuration 3's for the others,
    at the case's size, Rayleigh number and viscosity contrast."""
    replica = case["solver"] == "replica"
    c = Config.from_input(CFG1_INPUT if replica else CFG3_INPUT)
    c.level = int(round(math.log2(case["side"]))) + 1
    c.Rayleigh = case["rayleigh"]
    c.A = math.log(case["contrast"])
    c.mg_min_level = c.level - 1 if replica else 1
    if replica:
        c.citcom_solver_accu = 1e-10
        return c
    c.vis_min, c.vis_max = 1.0 / case["contrast"], 1.0
    c.stokes_rtol, c.max_refine = _rtol(case["side"]), 40
    if case["solver"] == "fp64mg":
        c.precision = 2
    if case["solver"] == "uzawa":
        c.stokes_method, c.warm_start, c.stokes_rtol = 0, 1, 1e-11
        c.outer_rtol, c.inner_rtol, c.mg_smooth = 1e-3, 1e-4, 2
    return c


def _amr_config(case):
    """configuration 2's input with the solver settings its benchmark runs it with."""
    c = Config.from_input(CFG2_INPUT)
    c.level = int(round(math.log2(case["base"]))) + case["extra"] + 1
    c.mg_min_level = 4
    c.Rayleigh, c.A = case["rayleigh"], math.log(case["contrast"])
    c.precision, c.warm_start, c.stokes_method, c.stokes_rtol = 1, 3, 1, _rtol(1 << (c.level - 1))
    c.outer_rtol, c.max_outer, c.max_refine = 1e-2, 2000, 40
    c.mg_smooth, c.mg_eta_avg = 1, 1
    return c


def _host_state(m, T):
    return {"model": m, "T": T, "V": np.zeros(2 * m.nno), "P": np.zeros(m.nel)}


def _layers(case):
    ch = [api.GUESS_CIN] + [case["channels"]] * (case["depth"] - 1) + [api.GUESS_COUT]
    return list(zip(ch, ch[1:]))


def prepare(case, seed):
    if case["kind"] == "step":
        m = Model(_step_config(case))
        m.initial_temperature()
        return _host_state(m, _temperature(m.get("X0"), m.get("X1"), seed, case["solver"] != "replica")) | {"kind": "step"}
    if case["kind"] in ("amr", "remesh"):
        c = _amr_config(case)
        F = c.level - 1
        base = F - case["extra"]
        m = Model(c, leaves=uniform_leaves(F, base))
        m.initial_temperature()
        m.set("T", _temperature(m.get("X0"), m.get("X1"), seed, True))
        if case["kind"] == "amr":
            m.remesh(0.2, base, F)
        return _host_state(m, m.get("T")) | {"kind": case["kind"], "base": base, "target": F}
    if case["kind"] == "ensemble":
        sizes = [s for s in ensemble.SIZES if s <= case["largest"]]
        n = case["members"]
        make = ensemble.amr_configs if case["refine"] else ensemble.configs
        cfgs = make(n, case["draw_seed"], sizes)
        for i, c in enumerate(cfgs):
            c.ic_seed = 1000 * (seed % 1000003) + i   # a refined member's mesh follows its initial temperature
            c.stokes_rtol, c.max_refine = 1e-12, 40
        e = Ensemble(cfgs, ensemble.amr_levels(n, case["draw_seed"]) if case["refine"] else None)
        e.initial_temperature()
        for _ in range(7):   # a sweep runs for many steps; the first six choose the launch shape by timing it
            e.step()
        return {"kind": "ensemble", "ensemble": e}
    r = np.random.default_rng(seed)
    b, h, w = case["batch"], case["height"], case["width"]
    net = Cnn(api.GUESS_CIN, case["channels"], case["depth"], api.GUESS_COUT, seed=seed % (1 << 31))
    # a fresh network's last layer is zero; in training every layer has moved
    net.set_params(np.concatenate([np.concatenate([r.standard_normal(9 * i * o) * math.sqrt(2.0 / (9 * i)),
                                                   0.1 * r.standard_normal(o)]) for i, o in _layers(case)]))
    return {"kind": "net", "net": net, "x": r.standard_normal((b, api.GUESS_CIN, h, w)).astype(np.float32),
            "t": r.standard_normal((b, api.GUESS_COUT, h, w)).astype(np.float32)}


# ---- one pass -------------------------------------------------------------------
def _fields(state):
    return {"T": state["T"], "V": state["V"], "P": state["P"] - state["P"].mean()}


def run(state):
    kind = state["kind"]
    if kind == "remesh":
        m = state["model"]
        m.remesh(0.2, state["base"], state["target"])
        state |= _host_state(m, m.get("T"))
        mesh = {k: m.mesh(k) for k in ("Mcode", "node", "hang")}
        m.step_host(state["T"], state["T"], state["V"], state["P"])
        return _fields(state) | mesh
    if kind in ("step", "amr"):
        state["model"].step_host(state["T"], state["T"], state["V"], state["P"])
        return _fields(state)
    if kind == "ensemble":
        e = state["ensemble"]
        e.step()
        out = {f: [m.get(f) for m in e.members] for f in ("T", "V0", "V1", "P")}
        out["P"] = [p - p.mean() for p in out["P"]]
        return {f: np.concatenate(v) for f, v in out.items()}
    y = state["net"].forward(state["x"])
    loss, grad = state["net"].gradient(state["x"], state["t"])
    return {"y": y, "loss": loss, "grad": grad}


# ---- what a pass cannot do without ------------------------------------------------
def _step_work(nodes, elements):
    # T in; T, V, P out; per node the Stokes operator and its residual, the heat system
    # and one product with it, once each (an iterative solve cannot do with less)
    return 8 * (nodes + nodes + 2 * nodes + elements), 2 * (36 + 16 + 2 * 9 + 9) * nodes


def work(case):
    if case["kind"] == "step":
        b, f = _step_work((case["side"] + 1) ** 2, case["side"] ** 2)
    elif case["kind"] in ("amr", "remesh"):
        # the boundary layers' share of the box goes to the finest level
        n = int(0.08 * case["base"] ** 2 * 4 ** case["extra"] + 0.9 * case["base"] ** 2)
        b, f = _step_work(n, n)
        b += 12 * n if case["kind"] == "remesh" else 0
    elif case["kind"] == "ensemble":
        sizes = [s for s in ensemble.SIZES if s <= case["largest"]]
        b = f = 0
        grow = ensemble.amr_levels(case["members"], case["draw_seed"]) if case["refine"] else [0] * case["members"]
        for (side, *_), lv in zip(ensemble.draw(case["members"], case["draw_seed"], sizes), grow):
            n = side * side if lv == 0 else int(0.08 * side ** 2 * 4 ** int(lv) + 0.9 * side ** 2)
            mb, mf = _step_work(n, n)
            b, f = b + mb, f + mf
    else:
        px = case["batch"] * case["height"] * case["width"]
        weights = sum(9 * i * o for i, o in _layers(case))
        # forward twice (the call and the gradient's own), both backward products
        # but the first layer's input gradient
        f = 2 * px * (4 * weights - 9 * api.GUESS_CIN * case["channels"])
        b = 4 * (px * (2 * api.GUESS_CIN + 2 * api.GUESS_COUT) + 3 * weights)
    return {"bytes": float(b), "flops": float(f)}


# ---- 64-bit values ------------------------------------------------------------------
_G = 1.0 / math.sqrt(3.0)
_XI, _ETA = np.array([-1.0, -1.0, 1.0, 1.0]), np.array([-1.0, 1.0, 1.0, -1.0])   # corners: z runs first


def _morton(ex, ez):
    m = np.zeros_like(ex)
    for b in range(12):
        m |= ((ez >> b) & 1) << (2 * b) | ((ex >> b) & 1) << (2 * b + 1)
    return m


def _exact_step(case, seed):
    """The first step of a uniform model in 64 bits: the discrete Stokes system
    solved directly, then the SUPG temperature update."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    N = case["side"]
    n, h = N + 1, 1.0 / N
    c = _step_config(case)
    ax = np.arange(n) / N
    X, Z = (a.reshape(-1) for a in np.meshgrid(ax, ax, indexing="ij"))   # node = iz + ix n
    T = _temperature(X, Z, seed, case["solver"] != "replica")
    ex, ez = (a.reshape(-1) for a in np.meshgrid(np.arange(N), np.arange(N), indexing="ij"))
    cn = np.stack([ez + ex * n, ez + 1 + ex * n, ez + 1 + (ex + 1) * n, ez + (ex + 1) * n], 1)
    buoy = (c.Rayleigh * T).reshape(n, n)
    buoy = (buoy - buoy.mean(0, keepdims=True)).reshape(-1)
    vis = np.exp(c.A * (c.refT - T))
    if c.vis_max > 0:
        vis = np.clip(vis, c.vis_min, c.vis_max)
    gx, gz = _XI * _G, _ETA * _G
    sh = 0.25 * (1 + _XI[:, None] * gx) * (1 + _ETA[:, None] * gz)           # [corner, gauss]
    dx = 0.25 * _XI[:, None] * (1 + _ETA[:, None] * gz) * (2 / h)
    dz = 0.25 * _ETA[:, None] * (1 + _XI[:, None] * gx) * (2 / h)
    jac = h * h / 4
    eg = vis[cn] @ sh                                                      # [element, gauss]
    xx, zz, zx = (np.einsum("ag,bg->abg", p, q) for p, q in ((dx, dx), (dz, dz), (dz, dx)))
    ke = np.zeros((N * N, 4, 2, 4, 2))
    ke[:, :, 0, :, 0] = np.einsum("eg,abg->eab", eg, 2 * xx + zz) * jac
    ke[:, :, 1, :, 1] = np.einsum("eg,abg->eab", eg, 2 * zz + xx) * jac
    ke[:, :, 0, :, 1] = np.einsum("eg,abg->eab", eg, zx) * jac
    ke[:, :, 1, :, 0] = np.einsum("eg,abg->eab", eg, zx.transpose(1, 0, 2)) * jac
    dof = (2 * cn[:, :, None] + np.arange(2)).reshape(N * N, 8)
    ge = np.stack([-dx.sum(1) * jac, -dz.sum(1) * jac], 1).reshape(8)
    # free slip: u fixed on the side walls, w on top and bottom
    fixed = np.zeros((n * n, 2), bool)
    fixed[(X <= 0) | (X >= 1), 0] = True
    fixed[(Z <= 0) | (Z >= 1), 1] = True
    free = ~fixed.reshape(-1)
    eq = np.cumsum(free) - 1
    F = np.zeros(2 * n * n)
    np.add.at(F, 2 * cn + 1, (buoy[cn] @ sh) @ sh.T * jac)
    nv, ne = int(free.sum()), N * N
    rows, cols = np.repeat(dof, 8, 1).reshape(-1), np.tile(dof, (1, 8)).reshape(-1)
    ok = free[rows] & free[cols]
    A = torch.zeros(nv + ne, nv + ne, dtype=torch.float64, device=dev)
    put = lambda r, q, v: A.index_put_((torch.tensor(r, device=dev), torch.tensor(q, device=dev)),  # noqa: E731
                                        torch.tensor(v, device=dev), accumulate=True)
    put(eq[rows[ok]], eq[cols[ok]], ke.reshape(-1)[ok])
    me = _morton(ex, ez)
    gr, gc, gv = dof.reshape(-1), np.repeat(me, 8), np.tile(ge, ne)
    ok = free[gr]
    put(eq[gr[ok]], nv + gc[ok], gv[ok])
    put(nv + gc[ok], eq[gr[ok]], gv[ok])
    # the constant is the null vector of G: p of the last element set to 0, its mean removed after
    b = torch.tensor(np.concatenate([F[free], np.zeros(ne - 1)]), device=dev)
    K = A[:-1, :-1].contiguous()
    lu, piv = torch.linalg.lu_factor(K)
    x = torch.linalg.lu_solve(lu, piv, b[:, None])
    x = x + torch.linalg.lu_solve(lu, piv, b[:, None] - K @ x)
    x = x[:, 0].cpu().numpy()
    V = np.zeros(2 * n * n)
    V[free] = x[:nv]
    P = np.append(x[nv:], 0.0)
    P -= P.mean()
    # temperature: SUPG with the element's mean velocity, generalized trapezoid, Jacobi-CG
    u = V.reshape(-1, 2)[cn].mean(1)
    al = 0.5 * u * h
    with np.errstate(all="ignore"):
        xi = np.where(np.abs(al) < c.accuracy, 0.0, np.where(np.abs(al) > 20, np.sign(al), 1 / np.tanh(al)) - 1 / al)
    tau = ((xi * u).sum(1) * h * 0.5)[:, None] * u / (u * u).sum(1)[:, None]
    hat = tau[:, 0, None, None] * dx + tau[:, 1, None, None] * dz          # [element, corner, gauss]
    ub = u[:, 0, None, None] * dx + u[:, 1, None, None] * dz
    kh = (np.einsum("eag,ebg->eab", hat + sh, ub) + np.einsum("abg->ab", xx + zz)) * jac
    # (the reference weights the capacity matrix with its unscaled derivatives)
    ch = np.einsum("eag,bg->eab", hat * jac + sh, sh) * jac
    dt = 0.75 * min(h * h, (0.5 / (np.abs(u).sum(1) / h)).min())
    tfix = (Z <= 0) | (Z >= 1)
    K, C = np.zeros((2, n * n, 9)), None
    slot = lambda a, q: 3 * (q // n - a // n + 1) + q % n - a % n + 1      # noqa: E731
    r9, c9 = np.repeat(cn, 4, 1).reshape(-1), np.tile(cn, (1, 4)).reshape(-1)
    np.add.at(K[0], (r9, slot(r9, c9)), kh.reshape(-1))
    np.add.at(K[1], (r9, slot(r9, c9)), ch.reshape(-1))
    K, C = K

    def mul(M, v):
        p = np.zeros((n + 2, n + 2))
        p[1:-1, 1:-1] = v.reshape(n, n)
        return sum(M[:, 3 * i + j].reshape(n, n) * p[i:i + n, j:j + n] for i in range(3) for j in range(3)).reshape(-1)

    Tb, tf = np.where(tfix, np.where(Z <= 0, 1.0, 0.0), 0.0), ~tfix
    tdt = c.theta * dt
    M = C / tdt + K
    rhs = (-mul(K, Tb) + mul(C, np.where(tf, T, 0.0)) / tdt) * tf
    t = np.where(tf, T, 0.0)
    r = (rhs - mul(M, t)) * tf
    idg = tf / M[:, 4]
    d = r * idg
    dn = d0 = r @ d
    it = 0
    while it < 1000 and dn > 1e-3 * d0:
        q = mul(M, d) * tf
        a = dn / (d @ q)
        t = t + a * d
        r = (rhs - mul(M, t)) * tf if it % 50 == 0 else r - a * q
        s = r * idg
        do, dn = dn, r @ s
        d = s + dn / do * d
        it += 1
        if np.abs(a * r).max() < 1e-3:
            break
    return {"T": np.where(tf, t, Tb), "V": V, "P": P}


def exact(case, seed):
    """64-bit values of the uniform models up to 64 x 64 (a dense factorisation of
    the Stokes system; larger and refined ones would take minutes) and of the network."""
    if case["kind"] == "step" and case["side"] <= 64:
        return _exact_step(case, seed)
    if case["kind"] != "net":
        return None
    s = prepare(case, seed)
    p = torch.tensor(s["net"].params(), dtype=torch.float64).requires_grad_()
    y, at = torch.tensor(s["x"], dtype=torch.float64), 0
    for k, (i, o) in enumerate(_layers(case)):
        w, b = p[at:at + 9 * i * o].view(o, i, 3, 3), p[at + 9 * i * o:at + 9 * i * o + o]
        at += 9 * i * o + o
        y = torch.nn.functional.conv2d(y, w, b, padding=1)
        if k + 1 < case["depth"]:
            y = torch.relu(y)
    loss = (y - torch.tensor(s["t"], dtype=torch.float64)).square().mean()
    loss.backward()
    return {"y": y.detach().numpy(), "loss": float(loss), "grad": p.grad.numpy()}
