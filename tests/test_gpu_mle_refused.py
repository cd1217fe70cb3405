"""A workspace for the batched input MLE that 16-byte stores cannot take is refused on
the host, before anything is queued."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu


def test_unaligned_workspace():
    import torch
    from truepix_b200 import native
    lib = native.gkr()
    x = torch.zeros(4 * 16, dtype=torch.uint8, device="cuda")
    z = torch.zeros(6, 2, dtype=torch.int64, device="cuda")
    out = torch.full((2,), -1, dtype=torch.int64, device="cuda")
    ws = torch.empty(128, dtype=torch.uint8, device="cuda")
    s = torch.cuda.current_stream().cuda_stream

    def call(skip):
        return lib.tp_mle_eval_pixels_batch_at(1, (ctypes.c_void_p * 1)(x.data_ptr()), (ctypes.c_int * 1)(4), 4, 16, 16,
                                               -1, 0, z.data_ptr(), None, out.data_ptr(), ws.data_ptr() + skip, 36, s)

    for skip in (1, 4, 8, 12):
        assert call(skip) != 0 and b"aligned" in lib.tp_last_error()
    assert out.tolist() == [-1, -1]
    assert call(16) == 0 and out.tolist() == [0, 0]
