"""Column lengths around those from which the encoder runs its levels in shared memory:
the whole column (codewords of up to 7,000 rows), one level less just above, and the
shortest columns with any level at all. The largest elements as well as random ones,
since the weighted sums are only reduced every few edges."""
import numpy as np
import pytest

from orionlib import OrionOracle, elements

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("largest", [False, True])
@pytest.mark.parametrize("col_len", [20, 21, 40, 128, 513, 4000, 4060, 4064, 4066, 4068, 4069, 4070, 4071, 4072, 4080, 4100])
def test_commit_root(col_len, largest):
    import torch
    from truepix_b200 import native
    lib, orc = native.gkr(), OrionOracle()
    n = 128 * col_len
    src = elements(col_len, n, "max" if largest else "random")
    tree = np.zeros((2 * lib.tp_orion_tree_leaves(n), 32), np.uint8)
    root = orc.commit(src)
    native.check(lib, lib.tp_orion_commit(src.ctypes.data, n, tree.ctypes.data, None), "commit")
    assert tree[1].tobytes() == root
