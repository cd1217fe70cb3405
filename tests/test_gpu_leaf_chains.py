"""Leaf chains at the row counts where a launch changes form: one warp for the rounds
and one for the schedule of 32 rows (up to two such CTAs an SM), one thread a row
beyond; whole and ragged last CTAs, and chains split over several launches."""
import numpy as np
import pytest

from orionlib import P61, OrionOracle, elements

pytestmark = pytest.mark.gpu


def edge_rows():
    return [1, 13, 31, 33, 64, 500, 2752, 4096, 5495, 5505, 5520, 8192]   # columns of so many elements


@pytest.mark.parametrize("col_len", edge_rows())
def test_commit_root_at_edges(col_len):
    import torch
    from truepix_b200 import native
    lib, orc = native.gkr(), OrionOracle()
    n = 128 * col_len
    src = elements(col_len, n)
    src[:4] = P61 - 1
    tree = np.zeros((2 * lib.tp_orion_tree_leaves(n), 32), np.uint8)
    root = orc.commit(src)
    for chunks in (1, 4):
        assert lib.tp_orion_set_leaf_chunks(chunks) == 0
        try:
            native.check(lib, lib.tp_orion_commit(src.ctypes.data, n, tree.ctypes.data, None), "commit")
        finally:
            assert lib.tp_orion_set_leaf_chunks(1) == 0
        assert tree[1].tobytes() == root, (col_len, chunks)


def fri_leaf(row):
    """h <- SHA256(x || y || h) over the 64 pairs of a row of the interleaved witness"""
    import hashlib
    h = bytes(32)
    for j in range(64):
        h = hashlib.sha256(row[4 * j:4 * j + 4].tobytes() + h).digest()
    return h


@pytest.mark.parametrize("log_m", [2, 3, 7, 8, 13, 14, 15, 16])
def test_fri_step_leaves(log_m):
    """every leaf of small steps, a sample of the leaves of larger ones"""
    import torch
    from truepix_b200 import native
    lib = native.gkr()
    g = torch.Generator(device="cuda")
    g.manual_seed(log_m)
    w = torch.randint(0, P61, (2 * 64 << log_m,), dtype=torch.int64, device="cuda", generator=g)
    nxt = torch.empty(64 << log_m, dtype=torch.int64, device="cuda")
    tree = torch.zeros(32 << (log_m - 1), dtype=torch.uint8, device="cuda")
    s = torch.cuda.current_stream().cuda_stream
    native.check(lib, lib.tp_fri_commit_step_dev(w.data_ptr(), log_m, 5, 7, nxt.data_ptr(), tree.data_ptr(), s), "step")
    leaves = 1 << (log_m - 2)
    rows = nxt.cpu().numpy().view(np.uint64).reshape(leaves, 256)
    t = tree.cpu().numpy().reshape(-1, 32)
    rng = np.random.default_rng(log_m)
    pick = range(leaves) if leaves <= 64 else sorted({0, 31, 32, leaves - 1, *rng.integers(0, leaves, 60).tolist()})
    for i in pick:
        assert t[leaves + i].tobytes() == fri_leaf(rows[i]), i
