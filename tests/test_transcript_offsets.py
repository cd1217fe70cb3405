"""The transcript's word-wise absorb and its digests at every number of pending
bytes: the host entry points against hashlib, and the device ones (a warp per
state, the two limbs of a draw closed side by side) against the host ones, the
whole 120-byte state included."""
import ctypes
import hashlib
import struct

import numpy as np
import pytest

from fslib import P61


def fresh(lib, history: bytes):
    st = ctypes.create_string_buffer(lib.tp_fs_state_bytes())
    assert lib.tp_fs_init(st, b"t") == 0
    if history:
        assert lib.tp_fs_absorb(st, history, len(history)) == 0
    return st


def text(s: bytes) -> bytes:
    return b"\x04" + struct.pack("<I", len(s)) + s


def draw(absorbed: bytearray, counter: int, label: bytes):
    """rand_ext on the absorbed bytes; returns the limbs and the next counter"""
    limbs = []
    for part in (b"real", b"imag"):
        absorbed += text(b"ext") + text(label) + text(part)
        while True:
            absorbed += b"\x01" + struct.pack("<IQ", 1, counter)
            counter += 1
            v = int.from_bytes(hashlib.sha256(bytes(absorbed)).digest(), "big") & P61
            if v < P61:
                break
        limbs.append(v)
    return limbs, counter


@pytest.mark.parametrize("label", [b"q", b"eq", b"sc-0-13", b"12345678", b"x" * 17, b"y" * 32])
def test_host_draws_at_every_offset(label):
    from truepix_b200 import native
    lib = native.gkr(require_device=False)
    re, im = ctypes.c_uint64(), ctypes.c_uint64()
    for n in range(64):
        history = bytes(range(n))
        st = fresh(lib, history)
        absorbed, counter = bytearray(b"TruePix,t,binhash1," + history), 0
        for _ in range(3):
            assert lib.tp_fs_rand_ext(st, label, ctypes.byref(re), ctypes.byref(im)) == 0
            want, counter = draw(absorbed, counter, label)
            assert [re.value, im.value] == want, n
            v = np.array([[n, P61 - 1], [re.value, im.value]], np.uint64)
            assert lib.tp_fs_put_fp2s(st, v[0].ctypes.data, v[1].ctypes.data, 2) == 0
            for k in range(2):
                absorbed += b"\x03" + struct.pack("<QQ", int(v[0, k]), int(v[1, k]))
        out = (ctypes.c_ubyte * 32)()
        assert lib.tp_fs_digest(st, out) == 0
        assert bytes(out) == hashlib.sha256(bytes(absorbed)).digest(), n


@pytest.mark.gpu
@pytest.mark.parametrize("label", [b"q", b"sc-0-13", b"12345678", b"y" * 32])
def test_device_states_equal_host_states_at_every_offset(label):
    import torch
    from truepix_b200 import native
    lib = native.gkr()
    n, nb = 64, lib.tp_fs_state_bytes()
    host = [fresh(lib, bytes(range(k))) for k in range(n)]
    dev = torch.from_numpy(np.frombuffer(b"".join(s.raw for s in host), np.uint8).copy()).cuda()
    out = torch.empty(2 * n, dtype=torch.int64, device="cuda")
    s = torch.cuda.current_stream().cuda_stream
    rng = np.random.default_rng(len(label))
    re, im = ctypes.c_uint64(), ctypes.c_uint64()
    for k in (1, 3, 4):
        vals = rng.integers(0, P61, size=(n, k, 2), dtype=np.uint64)
        d_vals = torch.from_numpy(vals.view(np.int64).reshape(-1)).cuda()
        assert lib.tp_fs_put_fp2s_dev(dev.data_ptr(), n, d_vals.data_ptr(), k, s) == 0, lib.tp_last_error()
        assert lib.tp_fs_rand_ext_dev(dev.data_ptr(), n, label, out.data_ptr(), s) == 0, lib.tp_last_error()
        got = out.cpu().numpy().view(np.uint64).reshape(n, 2)
        raw = dev.cpu().numpy().tobytes()
        for f in range(n):
            a, b = np.ascontiguousarray(vals[f, :, 0]), np.ascontiguousarray(vals[f, :, 1])
            assert lib.tp_fs_put_fp2s(host[f], a.ctypes.data, b.ctypes.data, k) == 0
            assert lib.tp_fs_rand_ext(host[f], label, ctypes.byref(re), ctypes.byref(im)) == 0
            assert (re.value, im.value) == (int(got[f, 0]), int(got[f, 1])), (k, f)
        # pending bytes, chaining words, counters (the bytes behind the pending ones
        # are what each side last held there)
        for f in range(n):
            d, h = raw[nb * f:nb * (f + 1)], host[f].raw
            pending = struct.unpack_from("<I", h, 112)[0]
            assert d[:32] == h[:32] and d[32:32 + pending] == h[32:32 + pending] and d[96:116] == h[96:116], (k, f)
