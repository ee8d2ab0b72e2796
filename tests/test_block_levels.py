"""mg_block_n, the size up to which a grid of the uniform V-cycle runs in one
block: its default stands for the measured choice of the precision, every other
value is the caller's and is taken as given in either precision."""
import ctypes as C

import pytest

from mantle_convection_lab_gb300 import Config, api


def block_n(**opts):
    c = Config.defaults()
    for k, v in opts.items():
        setattr(c, k, v)
    return api.lib().mclg_block_n(C.byref(c))


@pytest.mark.parametrize("precision, limit", [(0, 8), (1, 8), (2, 4)])
def test_default_is_the_measured_choice(precision, limit):
    assert Config.defaults().mg_block_n == 8
    assert block_n(precision=precision) == limit


@pytest.mark.parametrize("precision", [1, 2])
@pytest.mark.parametrize("n", [0, 1, 2, 4, 16, 64, 256])
def test_other_values_are_taken_as_given(precision, n):
    assert block_n(precision=precision, mg_block_n=n) == n
