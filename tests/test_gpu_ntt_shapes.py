"""Transforms of every size up to 2^17 points, alone and batched with gaps between
the transforms, against the oracle: one to two passes, two to sixteen columns per
CTA, stage groups of one, two and three stages, zero padding and subsampling."""
import numpy as np
import pytest

from orionlib import P61, OrionOracle, elements

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lg", range(18))
def test_every_size(lg):
    import torch
    from truepix_b200 import native
    lib, orc = native.gkr(), OrionOracle()
    n = 1 << lg
    s = torch.cuda.current_stream().cuda_stream
    for batch, pad in ((1, 0), (3, min(lg, 2))):
        m, gap = n >> pad, 5
        coef = [elements(1000 * lg + b, m) for b in range(batch)]
        coef[0][:2] = P61 - 1
        evals = [elements(2000 * lg + b, n) for b in range(batch)]
        place = lambda parts, size: np.concatenate([np.concatenate([p, np.zeros(2 * gap, np.uint64)]) for p in parts])
        dev = lambda a: torch.from_numpy(a.view(np.int64)).cuda()
        d_coef, d_evals = dev(place(coef, m)), dev(place(evals, n))
        fwd = torch.full((2 * batch * (n + gap),), -1, dtype=torch.int64, device="cuda")
        inv = torch.full((2 * batch * (m + gap),), -1, dtype=torch.int64, device="cuda")
        assert lib.tp_fft_dev(d_coef.data_ptr(), m, n, fwd.data_ptr(), batch, m + gap, n + gap, s) == 0
        assert lib.tp_ifft_dev(d_evals.data_ptr(), m, n, inv.data_ptr(), batch, n + gap, m + gap, s) == 0
        f = fwd.cpu().numpy().view(np.uint64).reshape(batch, -1)
        i = inv.cpu().numpy().view(np.uint64).reshape(batch, -1)
        for b in range(batch):
            np.testing.assert_array_equal(f[b, :2 * n], orc.fft(coef[b], n))
            np.testing.assert_array_equal(i[b, :2 * m], orc.ifft(evals[b], m))
            assert (f[b, 2 * n:] == np.uint64(2**64 - 1)).all() and (i[b, 2 * m:] == np.uint64(2**64 - 1)).all()
