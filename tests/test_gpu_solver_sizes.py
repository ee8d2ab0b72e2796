"""The solver and element kernels over the sizes, shapes and options at which
their launches change, each against an independent statement of the system.

- Converged solves: the returned d and p are put into F - K d - G p and G^T d
  with the operators of an FP64 replica model of the same mesh (assembled K in
  the reference's operation order, itself compared with the reference's and the
  CPU oracle's in test_gpu_parity.py).  The solver stops at 1e-10 of |F|; its
  own FP64 residual and the replica's differ by rounding, at most about
  side^2 * 1e-16 of |F| (6.6e-12 at 256), so the bar is 1.2e-10.
- Refined meshes: the same residual under the hanging-node constraints, with the
  constraint matrix of test_gpu_qt.py.
- The replica on meshes that one cluster solves: against the CPU oracle, to the
  parity bar (fields 1e-8, iteration counts within one).
- Assembly and temperature kernels of the converged solvers: FP64 in another
  operation order than the replica's, so 1e-12 for one product or assembled
  vector and 1e-10 for a temperature update (some tens of CG iterations on them).
- The network's gradient: the bar of test_gpu_learned.py (four times the spread
  that BF16 rounding flips give the oracle itself, plus 1e-6).
"""
import math

import numpy as np
import pytest
from conftest import rel
from oracle_port import Oracle
from test_gpu_learned import random_net
from test_gpu_qt import constraint_matrix

import cnn_oracle as co
from mantle_convection_lab_gb300 import Config, Mesh, Model, amr, ensemble

pytestmark = pytest.mark.gpu

CFG1_INPUT = ensemble.BASE_INPUT.replace("cfg3_mg_1024", "cfg1_plain_64")


def lid(c):
    """A moving lid: a tangential velocity on top and none at the bottom."""
    c.top_v_bc, c.bot_v_bc = b"VV", b"VV"
    c.top_v_bc_val[0] = 300.0


def config(side, precision=1, method=1, **opts):
    c = Config.from_input(CFG1_INPUT)
    c.level = int(math.log2(side)) + 1
    c.mg_min_level = max(c.level - 1, 1)
    c.A, c.Q = math.log(100.0), 5.0
    if opts.pop("lid", False):
        lid(c)
    c.precision, c.stokes_method, c.warm_start = precision, method, 3 if method else 1
    c.stokes_rtol, c.max_refine, c.max_outer = 1e-10, 40, 2000
    c.outer_rtol, c.inner_rtol = (1e-2, 1e-2) if method else (1e-3, 1e-4)
    c.mg_coarse = min(4, side // 2)
    for k, v in opts.items():
        setattr(c, k, v)
    return c


def replica_of(c):
    r = Config.from_input(CFG1_INPUT)
    for name, _ in Config._fields_:
        setattr(r, name, getattr(c, name))
    r.precision, r.mg_min_level = 0, c.level - 1
    return r


def temperature(m, seed):
    x, z = m.get("X0"), m.get("X1")
    x = x / x.max()
    rng = np.random.default_rng(seed)
    T = (1.0 - z) + 0.05 * np.sin(np.pi * z) * np.cos(np.pi * x)
    T = T + 0.01 * np.sin(np.pi * z) * rng.standard_normal(z.size)
    return np.where(z <= 0.0, 1.0, np.where(z >= 1.0, 0.0, T))


def load(m, T):
    m.initial_temperature()
    m.set("T", T)
    m.buoyancy_force()
    m.viscosity()
    m.velocity_pressure_KGF_matrix()


def stokes_residual(m, rep, C=None):
    d, p = m.get("d"), m.get("P")
    F = rep.get("F")
    Rm = F - rep.stokes_matvec(d) - rep.stokes_G(p)
    if C is not None:
        Rm, F = C.T @ Rm, C.T @ F
    Rc = rep.stokes_GT(d)
    return math.hypot(np.linalg.norm(Rm), np.linalg.norm(Rc)) / np.linalg.norm(F)


# precision, method, side, options: one block's, one cluster's and the grid's sizes;
# levels of one block from none to all, the dense coarsest solve in shared and in
# global memory, every smoother; elements that are not square; a moving lid
UNIFORM = [(1, 1, s, {}) for s in (4, 8, 16, 32, 64, 128, 256)]
UNIFORM += [(2, 1, s, {}) for s in (4, 16, 32, 64, 128)]
UNIFORM += [(1, 0, s, {}) for s in (8, 128, 256)] + [(2, 0, 32, {}), (2, 0, 64, {})]
UNIFORM += [(p, 1, 32, o) for p in (1, 2) for o in (
    {"mg_coarse": 2}, {"mg_coarse": 8}, {"mg_block_n": 0}, {"mg_block_n": 1}, {"mg_block_n": 64},
    {"mg_smooth": 3, "mg_smooth_coarse": 1}, {"mg_smooth": 1, "mg_smooth_coarse": 1, "mg_eta_avg": 2},
    {"mg_smoother": 1, "mg_smooth": 2, "mg_smooth_coarse": 2, "mg_cheb_lmax": 2.2, "mg_cheb_ratio": 4.0},
    {"model_length": 2.0}, {"lid": True})]
UNIFORM += [(1, 1, 256, {"mg_block_n": 0, "mg_coarse": 8}), (1, 1, 256, {"model_length": 2.0, "lid": True}),
            (1, 1, 256, {"mg_block_n": 256}), (1, 0, 32, {"mg_block_n": 64}), (1, 0, 64, {"lid": True}),
            (1, 1, 64, {"warm_start": 4})]


@pytest.mark.parametrize("precision,method,side,opts", UNIFORM)
def test_uniform_solve_satisfies_the_system(precision, method, side, opts):
    c = config(side, precision, method, **opts)
    host = Mesh(c)
    wall, wall_v = host.get("v_bc").reshape(2, -1) == ord("V"), host.get("v_bc_val").reshape(2, -1)
    with Model(c) as m, Model(replica_of(c)) as rep:
        for seed in (side, side + 1):       # the second solve starts from the first
            load(m, temperature(m, seed))
            load(rep, temperature(m, seed))
            assert rel(m.get("F"), rep.get("F")) < 1e-12
            st = m.solve_velocity_pressure()
            assert st.status == 0, (st.status, st.res_momentum, st.res_continuity)
            e = stokes_residual(m, rep)
            assert e < 1.2e-10, (e, st.res_momentum, st.res_continuity)
            for k, f in enumerate(("V0", "V1")):       # the wall velocities
                np.testing.assert_array_equal(m.get(f)[wall[k]], wall_v[k][wall[k]])


# base side, levels of refinement: one block's levels, one cluster, spread blocks, the grid
@pytest.mark.parametrize("base,extra,precision", [(8, 1, 1), (16, 2, 1), (32, 1, 1), (32, 2, 2), (64, 1, 1),
                                                  (64, 2, 1), (64, 2, 2), (128, 1, 1)])
def test_refined_solve_satisfies_the_system(base, extra, precision):
    c = Config.from_input(amr.CFG2_INPUT)
    lb = int(math.log2(base))
    F = lb + extra
    c.level, c.mg_min_level = F + 1, min(4, lb)
    c.Rayleigh, c.A = 1e6, math.log(100.0)
    c.precision, c.warm_start, c.stokes_method, c.stokes_rtol = precision, 3, 1, 1e-10
    c.outer_rtol, c.max_outer, c.max_refine = 1e-2, 2000, 40
    with Model(c, leaves=amr.uniform_leaves(F, lb)) as m0:
        m0.initial_temperature()
        flags, _ = m0.amr_flags(0.2)
        leaves = m0.amr_leaves(flags, lb, F)
    with Model(c, leaves=leaves) as m, Model(replica_of(c), leaves=leaves) as rep:
        print(base, extra, m.nno, "nodes", m.nh, "hanging")
        assert m.nh > 0
        C, _ = constraint_matrix(m, m.neq)
        T = temperature(m, base)
        load(m, T)
        load(rep, T)
        assert rel(m.get("F"), rep.get("F")) < 1e-12
        x = np.random.default_rng(base).standard_normal(m.neq)
        assert rel(m.stokes_matvec(x), rep.stokes_matvec(x)) < 1e-12
        st = m.solve_velocity_pressure()
        assert st.status == 0
        d = m.get("d")
        assert np.abs(C @ d - d).max() <= 1e-14 * np.abs(d).max()
        e = stokes_residual(m, rep, C)
        assert e < 1.2e-10, (e, st.res_momentum, st.res_continuity)
        # the temperature update from the same T and V
        rep.set("V0", m.get("V0"))
        rep.set("V1", m.get("V1"))
        m.update_temperature()
        rep.update_temperature()
        assert rel(m.get("T"), rep.get("T")) < 1e-10


@pytest.mark.parametrize("side,opts", [(4, {}), (32, {"lid": True}), (64, {"model_length": 2.0}), (128, {"theta": 1.0})])
def test_temperature_update_matches_replica(side, opts):
    """Heat rows, time step and update from the same T and V (internal heating on)."""
    c = config(side, **opts)
    with Model(c) as m, Model(replica_of(c)) as rep:
        T = temperature(m, 3 * side)
        load(m, T)
        load(rep, T)
        x, z = m.get("X0"), m.get("X1")
        V0 = 40.0 * np.sin(np.pi * x / x.max()) * np.cos(np.pi * z)
        V1 = -35.0 * np.cos(np.pi * x / x.max()) * np.sin(np.pi * z)
        for a in (m, rep):
            a.set("V0", V0)
            a.set("V1", V1)
        sm, sr = m.update_temperature(), rep.update_temperature()
        assert sm.heat_cg_cycles == sr.heat_cg_cycles
        assert rel(sm.dt, sr.dt) < 1e-12
        assert rel(m.get("T"), rep.get("T")) < 1e-10
        x = np.random.default_rng(side).standard_normal(m.heat_neq)
        for k in ("K", "C"):
            assert rel(m.heat_matvec(k, x), rep.heat_matvec(k, x)) < 1e-12


@pytest.mark.parametrize("side,opts", [(4, {}), (8, {"lid": True}), (16, {"model_length": 2.0}), (32, {"zero_P": 1}),
                                       (64, {"lid": True}), (16, {"max_cg_cycle": 7}), (32, {"max_citcom_cycle": 5})])
def test_replica_on_one_cluster_matches_oracle(side, opts):
    """Meshes of up to 64 x 64 without hanging nodes, to the reference's stop and at its caps."""
    c = replica_of(config(side, **opts))
    c.A = 0.0
    o = Oracle(c)
    with Model(c) as m:
        T = temperature(m, side)
        m.initial_temperature()
        m.set("T", T)
        o.set_T(T)
        for _ in range(2):
            so, st = o.step(), m.step()
            assert st.status in (0, 1)
            assert abs(st.uzawa_cycles - so["uzawa_cycles"]) <= 1
            for f in ("V0", "V1", "P", "T"):
                assert rel(m.get(f), o.get(f)) < 1e-8, f
    o.close()


# channels around the kernels' 4, 8, 16 and 32 wide forms; images smaller than a
# tile, ragged in both directions and over several tiles and blocks
@pytest.mark.parametrize("shape,cin,width,cout", [((1, 1, 1), 8, 32, 3), ((1, 3, 5), 1, 4, 1), ((2, 17, 31), 8, 5, 2),
                                                  ((1, 64, 33), 3, 16, 4), ((3, 5, 130), 8, 17, 9),
                                                  ((2, 33, 65), 32, 32, 32), ((1, 40, 96), 31, 24, 3)])
def test_network_gradient_matches_oracle(shape, cin, width, cout):
    b, h, w = shape
    net, p, shapes = random_net(13, cin=cin, width=width, depth=3, cout=cout)
    rng = np.random.default_rng(h * w)
    x = rng.standard_normal((b, cin, h, w)).astype(np.float32)
    t = rng.standard_normal((b, cout, h, w)).astype(np.float32)
    loss, g = net.gradient(x, t)
    rloss, rg = co.loss_and_grad(p, shapes, x, t)
    jit = [co.loss_and_grad(p, shapes, x, t, jitter=np.random.default_rng(s)) for s in (11, 12, 13, 14, 15)]
    assert abs(loss - rloss) / rloss < 4 * max(abs(jl - rloss) / rloss for jl, _ in jit) + 1e-6
    off = 0
    for o, i in shapes:
        n = o * i * 9 + o
        env = max(rel(jg[off:off + n], rg[off:off + n]) for _, jg in jit)
        e = rel(g[off:off + n], rg[off:off + n])
        assert e < 4 * env + 1e-6, (off, e, env)
        off += n
