"""A frame that could not be loaded (the vectors of its rounds do not fit the device)
takes no claim, no second fold and no finish, and its batch can be set anew."""
import ctypes

import numpy as np
import pytest

from fp2lib import P61, rand_fp

pytestmark = pytest.mark.gpu
U64P = ctypes.POINTER(ctypes.c_uint64)


def test_a_frame_that_did_not_fit():
    import torch
    from truepix_b200 import native
    lib = native.gkr()
    rng = np.random.default_rng(3)
    W, groups = 256, 16                      # 33 vectors, kept as such (4 * 33 <= W)
    gt = np.zeros(groups, np.int32)          # products
    i0 = np.arange(groups, dtype=np.int32) + 100
    i1 = np.arange(groups, dtype=np.int32)   # 16 wires b, one product each
    z = np.array([rand_fp(rng, groups), rand_fp(rng, groups)], np.uint64)
    s = torch.cuda.current_stream().cuda_stream
    copies = 8
    pixels = torch.from_numpy(rng.integers(0, 256, W * copies, dtype=np.uint8)).cuda()
    beta = torch.from_numpy(rng.integers(0, P61, 2 * copies).astype(np.int64)).cuda()
    claims = torch.zeros(8, dtype=torch.int64, device="cuda")
    out = torch.zeros(2 * W + 2, dtype=torch.int64, device="cuda")
    ch = np.array([3, 5], np.uint64)

    def load(b, n):
        return lib.tp_batch_set_pixels(b, 0, groups, gt.ctypes.data, i0.ctypes.data, i1.ctypes.data, z[0].ctypes.data,
                                       z[1].ctypes.data, pixels.data_ptr(), copies, n, W, W, -1, 0, beta.data_ptr())

    def first_claim(b):
        assert lib.tp_batch_claim(b, claims.data_ptr()) == 0, lib.tp_last_error()
        return claims.cpu().numpy().copy()

    b = lib.tp_batch_create(1, s)
    n = 1 << 28                              # 2 x 4.3 GB of beta; the vectors would take 212 GB
    assert torch.cuda.mem_get_info()[1] < 33 * 24 * n
    assert load(b, n) != 0                   # refused before anything is read
    refused = b"has no table"
    assert lib.tp_batch_claim(b, claims.data_ptr()) != 0 and refused in lib.tp_last_error()
    assert lib.tp_batch_fold(b, ch.ctypes.data_as(U64P)) == 0          # recorded only
    assert lib.tp_batch_fold(b, ch.ctypes.data_as(U64P)) != 0 and refused in lib.tp_last_error()
    assert lib.tp_batch_finish(b, out.data_ptr(), out[2 * W:].data_ptr()) != 0 and refused in lib.tp_last_error()
    lib.tp_batch_reset(b)
    assert load(b, copies) == 0, lib.tp_last_error()
    got = first_claim(b)
    lib.tp_batch_destroy(b)
    b = lib.tp_batch_create(1, s)
    assert load(b, copies) == 0
    np.testing.assert_array_equal(got, first_claim(b))
    lib.tp_batch_destroy(b)
