"""tp_batch_set_pixels_all against tp_batch_set_pixels for each frame: the same claims
and wires for frames of different lengths and layers with and without product terms,
with the caller's weights and betas overwritten right behind the call; a refused
frame leaves none of the batch set."""
import ctypes

import numpy as np
import pytest

from fp2lib import P61, rand_fp

pytestmark = pytest.mark.gpu
V = ctypes.c_void_p


def ptrs(a):
    return (V * len(a))(*a)


@pytest.mark.parametrize("n,products", [(1, False), (3, True), (70, False)])   # 70 frames: several uploads
def test_all_frames_at_once(n, products):
    import torch
    from truepix_b200 import native
    lib = native.gkr()
    rng = np.random.default_rng(n)
    W, cs, const, G = 512, 384, 500, 700
    gt = rng.choice([0, 5, 6, 1] if products else [1, 2, 3, 7], size=G).astype(np.int32)
    i0, i1 = (rng.integers(0, cs, size=G).astype(np.int32) for _ in range(2))
    padded = np.array([4 << (f % 3) for f in range(n)], np.int32)
    copies = np.array([p - f % 2 for f, p in enumerate(padded)], np.int32)
    z1 = np.array([[rand_fp(rng, G), rand_fp(rng, G)] for _ in range(n)], np.uint64)
    pix = [torch.from_numpy(rng.integers(0, 256, int(c) * cs, dtype=np.uint8)).cuda() for c in copies]
    beta = [torch.from_numpy(rng.integers(0, P61, 2 * int(p)).astype(np.int64)).cuda() for p in padded]
    s = torch.cuda.current_stream().cuda_stream

    def run(whole):
        b = lib.tp_batch_create(n, s)
        betas = [x.clone() for x in beta]
        z = z1.copy()
        if whole:
            if n > 1:   # the last frame refused: none is set
                bad = z1.copy()
                bad[-1, 0, 5] = P61
                assert set_all(b, bad, betas) != 0
            assert set_all(b, z, betas) == 0
        else:
            for f in range(n):
                assert lib.tp_batch_set_pixels(b, f, G, gt.ctypes.data, i0.ctypes.data, i1.ctypes.data,
                                               z[f, 0].ctypes.data, z[f, 1].ctypes.data, pix[f].data_ptr(),
                                               int(copies[f]), int(padded[f]), cs, W, const, 77, betas[f].data_ptr()) == 0
        z[...] = 0
        for x in betas:
            x.zero_()
        out = []
        for k in range(2):     # rounds that every frame has
            claims = torch.zeros(8 * n, dtype=torch.int64, device="cuda")
            assert lib.tp_batch_claim(b, claims.data_ptr()) == 0, lib.tp_last_error()
            out.append(claims.cpu().numpy())
            ch = np.full((n, 2), 12345 + k, np.uint64)
            assert lib.tp_batch_fold(b, ch.ctypes.data_as(ctypes.POINTER(ctypes.c_uint64))) == 0
        wires = torch.zeros(2 * W * n, dtype=torch.int64, device="cuda")
        fb = torch.zeros(2 * n, dtype=torch.int64, device="cuda")
        if n == 1:             # four copies: done
            assert lib.tp_batch_finish(b, wires.data_ptr(), fb.data_ptr()) == 0, lib.tp_last_error()
            out += [wires.cpu().numpy(), fb.cpu().numpy()]
        lib.tp_batch_destroy(b)
        return out

    def set_all(b, z, betas):
        return lib.tp_batch_set_pixels_all(b, G, gt.ctypes.data, i0.ctypes.data, i1.ctypes.data, z.ctypes.data,
                                           ptrs([x.data_ptr() for x in pix]), copies.ctypes.data, padded.ctypes.data,
                                           cs, W, const, 77, ptrs([x.data_ptr() for x in betas]))

    a, c = run(False), run(True)
    assert len(a) == len(c)
    for x, y in zip(a, c):
        np.testing.assert_array_equal(x, y)
