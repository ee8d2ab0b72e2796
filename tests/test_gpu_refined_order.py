"""The refined-mesh solver keeps the order of its operations.

On a mesh of several refinement levels the pressure's least determined modes
follow the rounding of the iterates: half an ulp on the temperature moves P by
up to 1e-8 where the solve stops at the residual that FP64 allows.  Whichever
team of blocks runs a solve (one cluster up to 6144 nodes, a grid with one or
several nodes a thread), its values and sums are formed in one fixed order, and
the fields are those that were recorded with the kernels of one grid pass per
operation (refined_order.npz: two steps, every `STRIDE`-th value of P, V and T).

The bar is nine digits of each field: other orders of operations, equally right,
moved P of the largest mesh here by 2e-9.  The iteration counts are the recorded
ones.  The temperature is formed with +, -, * and / alone, so that it is the same
to the bit on every machine.

    python tests/test_gpu_refined_order.py FILE     records the fields
"""
import os
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)

from mantle_convection_lab_gb300 import Config, Model  # noqa: E402
from mantle_convection_lab_gb300.amr import CFG2_INPUT, uniform_leaves  # noqa: E402

pytestmark = pytest.mark.gpu

STRIDE = 61
# base side, refinement levels above it, ln(viscosity contrast), other options
CASES = {
    "cluster_mixed": (32, 2, 2.3025850929940456, {}),
    "cluster_fp64": (32, 2, 2.3025850929940456, {"precision": 2}),
    "cluster_two_sweeps": (32, 2, 2.3025850929940456, {"mg_smooth": 2}),
    "cluster_long_box": (32, 2, 2.3025850929940456, {"model_length": 1.7}),
    "grid_mixed": (64, 2, 6.907755278982137, {}),
    "grid_three_sweeps": (64, 2, 6.907755278982137, {"mg_smooth": 3}),
    "grid_two_trips_mixed": (128, 3, 9.210340371976184, {}),
}


def temperature(x, z):
    def layer(s):
        s = s / 0.03
        return 1.0 / (1.0 + s * s)

    T = 0.5 + 0.5 * layer(z) - 0.5 * layer(1.0 - z)
    w = z * (1.0 - z)
    T = T + 0.4 * w * x * (1.0 - x) * (x - 0.375) + 0.2 * w * (z - 0.5625) * (x - 0.75) * (x - 0.125)
    return np.where(z <= 0.0, 1.0, np.where(z >= 1.0, 0.0, T))


def fields(base, extra, A, opts):
    c = Config.from_input(CFG2_INPUT)
    F = base.bit_length() - 1 + extra
    c.level, c.mg_min_level = F + 1, 4
    c.Rayleigh, c.A = 1e7, A
    c.precision, c.warm_start, c.stokes_method = 1, 3, 1
    c.stokes_rtol = max(1e-12, 6e-18 * 4.0 ** F)
    c.outer_rtol, c.max_outer, c.max_refine = 1e-2, 2000, 40
    c.mg_smooth, c.mg_eta_avg = 1, 1
    for k, v in opts.items():
        setattr(c, k, v)
    out, its = {}, []
    with Model(c, leaves=uniform_leaves(F, F - extra)) as m:
        m.initial_temperature()
        m.set("T", temperature(m.get("X0"), m.get("X1")))
        m.remesh(0.2, F - extra, F)
        out["nodes"] = np.array(m.nno)
        for step in range(2):
            st = m.step()
            assert st.status == 0
            its.append([st.refine_passes, st.uzawa_cycles])
            P = m.get("P")
            for k, v in (("P", P - P.mean()), ("V0", m.get("V0")), ("V1", m.get("V1")), ("T", m.get("T"))):
                out[f"{k}_{step}"] = v[::STRIDE].copy()
    out["its"] = np.array(its)
    return out


@pytest.mark.parametrize("case", CASES)
def test_fields_are_the_recorded_ones(case):
    want = np.load(os.path.join(ROOT, "tests", "golden", "refined_order.npz"))
    got = fields(*CASES[case])
    for k, v in got.items():
        w = want[f"{case}_{k}"]
        if v.dtype.kind != "f":
            np.testing.assert_array_equal(v, w, err_msg=k)
        else:
            assert np.linalg.norm(v - w) <= 1e-9 * np.linalg.norm(w), k


if __name__ == "__main__":
    np.savez_compressed(sys.argv[1], **{f"{n}_{k}": v for n, c in CASES.items() for k, v in fields(*c).items()})
