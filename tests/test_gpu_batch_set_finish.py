"""Wires and final beta of frames set in one call against frames set one by one, with
rounds left and with none, for batches whose frames differ in their number of 512-copy
pieces and whose forms take several uploads; one layer with product groups, one without."""
import ctypes

import numpy as np
import pytest

from fp2lib import P61, rand_fp

pytestmark = pytest.mark.gpu
V = ctypes.c_void_p


@pytest.mark.parametrize("products", [False, True])
@pytest.mark.parametrize("padded", [[4], [8, 2048, 512], [1024, 4096, 2, 512, 8192] + [4, 8, 16] * 22])
def test_finish(padded, products):
    import torch
    from truepix_b200 import native
    lib = native.gkr()
    n, W, cs, const, G = len(padded), 512, 384, 500, 700
    rng = np.random.default_rng(n)
    gt = rng.choice([0, 5, 6, 1] if products else [1, 2, 3, 7], size=G).astype(np.int32)
    i0 = rng.integers(0, cs, size=G).astype(np.int32)
    i1 = rng.choice([3, 9, 200], size=G).astype(np.int32) if products else rng.integers(0, cs, size=G).astype(np.int32)
    padded = np.array(padded, np.int32)
    copies = np.array([max(1, p - 3 * (f % 2)) for f, p in enumerate(padded)], np.int32)
    z1 = np.array([[rand_fp(rng, G), rand_fp(rng, G)] for _ in range(n)], np.uint64)
    pix = [torch.from_numpy(rng.integers(0, 256, int(c) * cs, dtype=np.uint8)).cuda() for c in copies]
    beta = [torch.from_numpy(rng.integers(0, P61, 2 * int(p)).astype(np.int64)).cuda() for p in padded]
    ptrs = lambda ts: (V * n)(*[t.data_ptr() for t in ts])
    rounds = int(padded.max()).bit_length() - 1
    ch = rng.integers(0, P61, (rounds, n, 2)).astype(np.uint64)

    def run(whole):
        b = lib.tp_batch_create(n, torch.cuda.current_stream().cuda_stream)
        if whole:
            assert lib.tp_batch_set_pixels_all(b, G, gt.ctypes.data, i0.ctypes.data, i1.ctypes.data, z1.ctypes.data,
                                               ptrs(pix), copies.ctypes.data, padded.ctypes.data, cs, W, const, 77,
                                               ptrs(beta)) == 0, lib.tp_last_error()
        for f in range(0 if whole else n):
            assert lib.tp_batch_set_pixels(b, f, G, gt.ctypes.data, i0.ctypes.data, i1.ctypes.data,
                                           z1[f, 0].ctypes.data, z1[f, 1].ctypes.data, pix[f].data_ptr(),
                                           int(copies[f]), int(padded[f]), cs, W, const, 77, beta[f].data_ptr()) == 0
        out = []
        for k in range(rounds + 1):
            if k in (0, 1, rounds):
                wires = torch.zeros(2 * W * n, dtype=torch.int64, device="cuda")
                fb = torch.zeros(2 * n, dtype=torch.int64, device="cuda")
                assert lib.tp_batch_finish(b, wires.data_ptr(), fb.data_ptr()) == 0, lib.tp_last_error()
                out += [wires.cpu().numpy(), fb.cpu().numpy()]
            if k < rounds:
                claims = torch.zeros(8 * n, dtype=torch.int64, device="cuda")
                assert lib.tp_batch_claim(b, claims.data_ptr()) == 0, lib.tp_last_error()
                out.append(claims.cpu().numpy())
                assert lib.tp_batch_fold(b, ch[k].ctypes.data_as(ctypes.POINTER(ctypes.c_uint64))) == 0
        lib.tp_batch_destroy(b)
        return out

    for x, y in zip(run(False), run(True)):
        np.testing.assert_array_equal(x, y)
