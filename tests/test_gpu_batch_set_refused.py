"""What tp_batch_set_pixels_all refuses and takes, against tp_batch_set_pixels for each
frame in turn: betas that are missing or at any address, and a batch in its rounds,
which a refused call leaves as it is."""
import ctypes

import numpy as np
import pytest

from fp2lib import P61, rand_fp

pytestmark = pytest.mark.gpu
V = ctypes.c_void_p
U64P = ctypes.POINTER(ctypes.c_uint64)
W, CS, CONST, G = 512, 384, 500, 64


def ptrs(a):
    return (V * len(a))(*a)


class Frames:
    """n frames of 8, 16 or 32 copies under a layer with one product group"""

    def __init__(self, n):
        import torch
        from truepix_b200 import native
        self.lib, self.n = native.gkr(), n
        rng = np.random.default_rng(n)
        self.gt = rng.choice([0, 1, 2, 3], size=G).astype(np.int32)
        self.i0, self.i1 = (rng.integers(0, CS, size=G).astype(np.int32) for _ in range(2))
        self.i1[self.gt == 0] = 7
        self.padded = np.array([8 << (f % 3) for f in range(n)], np.int32)
        self.copies = np.array([p - f % 2 for f, p in enumerate(self.padded)], np.int32)
        self.z = np.array([[rand_fp(rng, G), rand_fp(rng, G)] for _ in range(n)], np.uint64)
        self.pix = [torch.from_numpy(rng.integers(0, 256, int(c) * CS, dtype=np.uint8)).cuda() for c in self.copies]
        self.beta = [torch.from_numpy(rng.integers(0, P61, 2 * int(p)).astype(np.int64)).cuda() for p in self.padded]
        self.ch = np.array([[11 + f, 13] for f in range(n)], np.uint64)

    def batch(self):
        import torch
        return self.lib.tp_batch_create(self.n, torch.cuda.current_stream().cuda_stream)

    def set_each(self, b):
        for f in range(self.n):
            assert self.lib.tp_batch_set_pixels(
                b, f, G, self.gt.ctypes.data, self.i0.ctypes.data, self.i1.ctypes.data, self.z[f, 0].ctypes.data,
                self.z[f, 1].ctypes.data, self.pix[f].data_ptr(), int(self.copies[f]), int(self.padded[f]), CS, W,
                CONST, 77, self.beta[f].data_ptr()) == 0, self.lib.tp_last_error()

    def set_all(self, b, betas=None):
        return self.lib.tp_batch_set_pixels_all(
            b, G, self.gt.ctypes.data, self.i0.ctypes.data, self.i1.ctypes.data, self.z.ctypes.data,
            ptrs([x.data_ptr() for x in self.pix]), self.copies.ctypes.data, self.padded.ctypes.data, CS, W, CONST, 77,
            ptrs(betas if betas is not None else [x.data_ptr() for x in self.beta]))

    def round(self, b):
        """a claim of every frame, then a fold"""
        import torch
        claims = torch.zeros(8 * self.n, dtype=torch.int64, device="cuda")
        assert self.lib.tp_batch_claim(b, claims.data_ptr()) == 0, self.lib.tp_last_error()
        assert self.lib.tp_batch_fold(b, self.ch.ctypes.data_as(U64P)) == 0
        return claims.cpu().numpy()


@pytest.mark.parametrize("missing", [0, 2])
def test_missing_beta(missing):
    fr = Frames(3)
    b = fr.batch()
    betas = [x.data_ptr() for x in fr.beta]
    betas[missing] = None
    assert fr.set_all(b, betas) != 0 and b"no beta" in fr.lib.tp_last_error()
    assert fr.lib.tp_batch_n_copies(b, 0) == 0      # none is set
    fr.lib.tp_batch_destroy(b)


def test_beta_at_odd_addresses():
    import torch
    fr = Frames(4)
    b = fr.batch()
    fr.set_each(b)
    want = [fr.round(b) for _ in range(3)]
    fr.lib.tp_batch_destroy(b)
    keep = []
    for f, skip in ((1, 8), (3, 4)):
        raw = torch.zeros(16 * int(fr.padded[f]) + 16, dtype=torch.uint8, device="cuda")
        raw[skip:skip + 16 * int(fr.padded[f])] = fr.beta[f].view(torch.uint8)
        keep.append((f, raw[skip:]))
    betas = [x.data_ptr() for x in fr.beta]
    for f, raw in keep:
        betas[f] = raw.data_ptr()
    b = fr.batch()
    assert fr.set_all(b, betas) == 0, fr.lib.tp_last_error()
    for w in want:
        np.testing.assert_array_equal(fr.round(b), w)
    fr.lib.tp_batch_destroy(b)


def test_refused_in_the_middle_of_the_rounds():
    fr = Frames(3)
    b = fr.batch()
    fr.set_each(b)
    want = [fr.round(b) for _ in range(3)]
    fr.lib.tp_batch_destroy(b)
    b = fr.batch()
    assert fr.set_all(b) == 0, fr.lib.tp_last_error()
    for k, w in enumerate(want):
        np.testing.assert_array_equal(fr.round(b), w)
        assert fr.set_all(b) != 0 and b"already configured" in fr.lib.tp_last_error()
        assert [fr.lib.tp_batch_n_copies(b, f) for f in range(3)] == [int(p) >> (k + 1) for p in fr.padded]
    fr.lib.tp_batch_reset(b)
    assert fr.set_all(b) == 0, fr.lib.tp_last_error()
    np.testing.assert_array_equal(fr.round(b), want[0])
    fr.lib.tp_batch_destroy(b)


@pytest.mark.parametrize("one_set", [0, 2])
def test_refused_beside_a_single_frame(one_set):
    fr = Frames(3)
    b = fr.batch()
    f = one_set
    assert fr.lib.tp_batch_set_pixels(
        b, f, G, fr.gt.ctypes.data, fr.i0.ctypes.data, fr.i1.ctypes.data, fr.z[f, 0].ctypes.data,
        fr.z[f, 1].ctypes.data, fr.pix[f].data_ptr(), int(fr.copies[f]), int(fr.padded[f]), CS, W, CONST, 77,
        fr.beta[f].data_ptr()) == 0, fr.lib.tp_last_error()
    assert fr.set_all(b) != 0
    assert [fr.lib.tp_batch_n_copies(b, k) for k in range(3)] == [int(fr.padded[k]) if k == f else 0 for k in range(3)]
    fr.lib.tp_batch_destroy(b)
