"""Virgo sumcheck rounds at the sizes where the launch changes form: a few threads,
one CTA, clusters of two to eight CTAs, partial sums of many CTAs; whole and ragged
last CTAs; against the oracle, every folded entry and the round polynomial."""
import numpy as np
import pytest

from orionlib import P61, OrionOracle, elements, virgo_inputs
from test_gpu_virgo import run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("half", [1, 2, 31, 33, 255, 256, 257, 511, 513, 1024, 1793, 2047, 2048, 2049, 4097, 70001])
def test_update_at_launch_edges(half):
    from truepix_b200 import native
    lib = native.gkr()
    orc = OrionOracle()
    vma, addv, ams, r = virgo_inputs(2 * half, half)
    vma[-4:] = P61 - 1
    ams[-4:] = P61 - 1
    for bit in (0, 1):
        want, wret = orc.virgo_update(vma, addv, ams, r, bit)
        got, gret = run(lib, vma, addv, ams, r, bit)
        for g, w in zip(got, want):
            np.testing.assert_array_equal(g, w)
        np.testing.assert_array_equal(gret, wret)
