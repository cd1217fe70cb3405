"""Byte frames on both sides of the lines between rounds on vectors and on the table of
all wires, and between a launch a round and all rounds in one (copies, product groups,
copies per group), against the oracle's session; frames of both kinds in one batch."""
import ctypes

import numpy as np
import pytest

import test_gpu_linear_rounds as rounds
from fp2lib import P61, rand_fp
from test_gpu_linear_rounds import lib, oracle  # noqa: F401  (fixtures)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,cs,real,C,groups", [
    (64, 48, 2, 2, 0), (64, 48, 4, 4, 0), (64, 48, 4, 4, 4), (64, 48, 900, 1024, 4), (64, 48, 900, 1024, 5),
    (64, 48, 8100, 8192, 2), (64, 48, 4096, 4096, 4), (64, 48, 8100, 8192, 5), (64, 48, 16000, 16384, 5), (128, 72, 8192, 8192, 8), (128, 72, 16384, 16384, 8),
    (256, 140, 32000, 32768, 16), (64, 35, 100, 128, 4), (64, 36, 100, 128, 4)])
def test_byte_frames(lib, oracle, W, cs, real, C, groups):  # noqa: F811
    rounds.test_bytes_source(lib, oracle, W, cs, real, C, -1, groups, 0)


def test_both_kinds_in_a_batch(lib):  # noqa: F811
    """2, 4, 8,192 and 16,384 copies under a layer of five groups, together and alone"""
    import torch
    rng = np.random.default_rng(8)
    W, cs = 64, 48
    gt, i0, i1 = rounds.layer(rng, W, 5, cs)
    C = np.array([2, 4, 8192, 16384], np.int32)
    n = C.size
    z = np.array([[rand_fp(rng, 300), rand_fp(rng, 300)] for _ in C], np.uint64)
    pix = [torch.from_numpy(rng.integers(0, 256, int(c) * cs, dtype=np.uint8)).cuda() for c in C]
    beta = [torch.from_numpy(rng.integers(0, P61, 2 * int(c)).astype(np.int64)).cuda() for c in C]
    ch = rng.integers(0, P61, (14, n, 2)).astype(np.uint64)
    s = torch.cuda.current_stream().cuda_stream

    def run(frames):
        b = lib.tp_batch_create(len(frames), s)
        for k, f in enumerate(frames):
            assert lib.tp_batch_set_pixels(b, k, 300, gt.ctypes.data, i0.ctypes.data, i1.ctypes.data,
                                           z[f, 0].ctypes.data, z[f, 1].ctypes.data, pix[f].data_ptr(), int(C[f]),
                                           int(C[f]), cs, W, -1, 0, beta[f].data_ptr()) == 0, lib.tp_last_error()
        claims = torch.zeros(14, len(frames), 8, dtype=torch.int64, device="cuda")
        fin = torch.zeros(len(frames), W, 2, dtype=torch.int64, device="cuda")
        fb = torch.zeros(len(frames), 2, dtype=torch.int64, device="cuda")
        for k in range(int(C[frames].max()).bit_length() - 1):
            assert lib.tp_batch_claim(b, claims[k].data_ptr()) == 0, lib.tp_last_error()
            r = np.ascontiguousarray(ch[k][frames])
            assert lib.tp_batch_fold(b, r.ctypes.data_as(ctypes.POINTER(ctypes.c_uint64))) == 0
        assert lib.tp_batch_finish(b, fin.data_ptr(), fb.data_ptr()) == 0, lib.tp_last_error()
        lib.tp_batch_destroy(b)
        return claims.cpu(), fin.cpu(), fb.cpu()

    together = run(list(range(n)))
    for f in range(n):
        for a, b in zip(run([f]), together):
            got = b[:, f:f + 1] if b.dim() == 3 and b.shape[0] == 14 else b[f:f + 1]
            assert torch.equal(a, got), f
