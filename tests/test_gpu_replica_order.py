"""The replica on one cluster gives the bits of the cooperative grid kernel.

k_uzawa_cluster (meshes up to 64^2 without hanging nodes) forms its sums in the
order of k_uzawa; at a large viscosity contrast another order moves the Uzawa
count.  replica_order.npz holds what k_uzawa gave for these models on a GB300 (the
iteration counts, and every `STRIDE`-th value of P and V after two steps of at
most 150 Uzawa cycles), and the fields here are those to the bit.  The temperature
is formed with +, -, * and / alone.

    python tests/test_gpu_replica_order.py FILE     records the fields
"""
import os
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)

from mantle_convection_lab_gb300 import Config, Model, ensemble  # noqa: E402

pytestmark = pytest.mark.gpu

STRIDE = 7
CFG1_INPUT = ensemble.BASE_INPUT.replace("cfg3_mg_1024", "cfg1_plain_64")
# level (side 2^(level - 1)), ln(viscosity contrast)
CASES = {"16_flat": (5, 0.0), "32_1e2": (6, 4.605170185988092), "64_flat": (7, 0.0), "64_1e5": (7, 11.512925464970229)}


def fields(level, A):
    c = Config.from_input(CFG1_INPUT)
    c.level, c.mg_min_level, c.Rayleigh, c.A = level, level - 1, 1e5, A
    c.citcom_solver_accu, c.max_citcom_cycle = 1e-10, 150
    out, its = {}, []
    with Model(c) as m:
        m.initial_temperature()
        x, z = m.get("X0"), m.get("X1")
        T = (1.0 - z) + z * (1.0 - z) * (0.5 * (x - 0.5) + 0.3 * (x - 0.25) * (z - 0.625))
        m.set("T", T)
        for step in range(2):
            st = m.step()
            its.append([st.uzawa_cycles, st.cg_cycles])
            for k in ("P", "V0", "V1"):
                out[f"{k}_{step}"] = m.get(k)[::STRIDE].copy()
    out["its"] = np.array(its)
    return out


@pytest.mark.parametrize("case", CASES)
def test_bits_of_the_grid_kernel(case):
    want = np.load(os.path.join(ROOT, "tests", "golden", "replica_order.npz"))
    for k, v in fields(*CASES[case]).items():
        np.testing.assert_array_equal(v, want[f"{case}_{k}"], err_msg=k)


if __name__ == "__main__":
    np.savez_compressed(sys.argv[1], **{f"{n}_{k}": v for n, c in CASES.items() for k, v in fields(*c).items()})
