"""The opening's combined codeword and answer against Python integers, at row counts
around a warp's four rows and a launch's rows, and at entry counts around a CTA's 1,024
entries and around 256 partial sums."""
import numpy as np
import pytest

from orionlib import P61, elements

pytestmark = pytest.mark.gpu


def dot(a, b):
    """sum of products of Fp2 elements {img, real}, int rows of shape (n, 2)"""
    re = im = 0
    for (ai, ar), (bi, br) in zip(a.tolist(), b.tolist()):
        re += ar * br - ai * bi
        im += ar * bi + ai * br
    return im % P61, re % P61


def dev(a):
    import torch
    return torch.from_numpy(a.view(np.int64)).cuda()


@pytest.mark.parametrize("kind", ["random", "max"])
@pytest.mark.parametrize("col_len", [1, 2, 3, 4, 5, 8, 9, 10, 11, 20, 8256, 8257, 8258, 8259, 16600])
def test_combined_codeword(col_len, kind):
    import torch
    from truepix_b200 import native
    lib = native.gkr()
    n = 128 * col_len
    cw = lib.tp_orion_codeword_len(col_len)
    rows, r0 = elements(col_len, 128 * cw, kind), elements(7, 128, kind)
    d_rows, d_r0 = dev(rows), dev(r0)
    out = torch.full((2 * (cw + 8),), -1, dtype=torch.int64, device="cuda")
    native.check(lib, lib.tp_orion_combine_dev(d_rows.data_ptr(), n, d_r0.data_ptr(), out.data_ptr(), None,
                                               torch.cuda.current_stream().cuda_stream), "combine")
    got = out.cpu().numpy().view(np.uint64).reshape(-1, 2)
    assert (got[cw:] == np.uint64(2**64 - 1)).all()
    rng = np.random.default_rng(col_len)
    pick = range(cw) if cw < 64 else sorted({*range(9), *range(cw - 9, cw), *range(14200, min(cw, 14217)),
                                             *rng.integers(0, cw, 40).tolist()})
    rows, r0 = rows.reshape(cw, 128, 2), r0.reshape(128, 2)
    for t in pick:
        assert tuple(got[t].tolist()) == dot(r0, rows[t]), t


@pytest.mark.parametrize("n", [1, 31, 255, 257, 1023, 1024, 1025, 8191, 262143, 262144, 262145])
def test_answer(n):
    import torch
    from truepix_b200 import native
    lib = native.gkr()
    x, r1 = elements(n, n), elements(n + 1, n)
    x[:2] = r1[:2] = P61 - 1
    d_x, d_r1 = dev(x), dev(r1)
    out = torch.zeros(2, dtype=torch.int64, device="cuda")
    for _ in range(2):
        native.check(lib, lib.tp_orion_answer_dev(d_x.data_ptr(), n, d_r1.data_ptr(), out.data_ptr(),
                                                  torch.cuda.current_stream().cuda_stream), "answer")
    assert tuple(out.cpu().numpy().view(np.uint64).tolist()) == dot(x.reshape(-1, 2), r1.reshape(-1, 2))


@pytest.mark.parametrize("col_len", [1, 2, 3, 130, 300, 16000, 40000])   # 1 to 256 CTAs in the tree's first launch
def test_combined_tree(col_len):
    import hashlib
    import torch
    from truepix_b200 import native
    lib = native.gkr()
    n = 128 * col_len
    cw = lib.tp_orion_codeword_len(col_len)
    leaves = lib.tp_orion_tree_leaves(n)
    d_rows, d_r0 = dev(elements(col_len, 128 * cw)), dev(elements(7, 128))
    comb = torch.zeros(2 * cw, dtype=torch.int64, device="cuda")
    tree = torch.full((64 * leaves,), 7, dtype=torch.uint8, device="cuda")
    native.check(lib, lib.tp_orion_combine_dev(d_rows.data_ptr(), n, d_r0.data_ptr(), comb.data_ptr(), tree.data_ptr(),
                                               torch.cuda.current_stream().cuda_stream), "combine")
    x = comb.cpu().numpy().tobytes() + bytes(16 * max(0, leaves - cw))
    want = [None] * leaves + [hashlib.sha256(x[16 * i:16 * i + 16] + bytes(48)).digest() for i in range(leaves)]
    for k in range(leaves - 1, 0, -1):
        want[k] = hashlib.sha256(want[2 * k] + want[2 * k + 1]).digest()
    t = tree.cpu().numpy().tobytes()
    assert t[32:] == b"".join(want[1:])
