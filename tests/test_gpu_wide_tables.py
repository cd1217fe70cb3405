"""Sessions over tables of so many wires that the layer's linear form is uploaded by
itself, with and without product terms, against the oracle."""
import pytest

import test_gpu_linear_rounds as rounds
from test_gpu_linear_rounds import lib, oracle  # noqa: F401  (fixtures)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,C,groups", [(1024, 8, 3), (1025, 8, 3), (1025, 2, 0), (5000, 4, 20), (20000, 4, 0)])
def test_wide_tables(lib, oracle, W, C, groups):  # noqa: F811
    rounds.test_table_source(lib, oracle, W, C, groups)
