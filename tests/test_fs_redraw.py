"""Draws that have to be drawn again: with a bound that most 61-bit draws miss, the host
transcript against hashlib and the device's against the host's, limbs and whole states,
from every offset within a block."""
import ctypes
import hashlib
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
P61 = (1 << 61) - 1
P = lambda a: ctypes.c_void_p(a.ctypes.data)
STATES, DRAWS = 64, 6
LABELS = [b"", b"sc-0-12", b"a label of thirty-two bytes, all"]


@pytest.fixture(scope="module", params=[1 << 60, 1 << 57])     # 2 draws a limb on average, and 16
def built(request, tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    out = str(tmp_path_factory.mktemp("redraw") / "fs_redraw.so")
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O2", "-std=c++17", "-Xcompiler", "-fPIC",
                    "-shared", "-DTP_FS_DRAW_BOUND=%dull" % request.param, "-o", out,
                    os.path.join(ROOT, "tests", "fs_redraw.cu")], check=True)
    return ctypes.CDLL(out), request.param


class Transcript:
    def __init__(self, data, bound):
        self.data, self.rnum, self.bound, self.redrawn = bytearray(data), 0, bound, 0

    def text(self, t):
        self.data += b"\x04" + len(t).to_bytes(4, "little") + t

    def scalar(self):
        while True:
            self.data += b"\x01" + (1).to_bytes(4, "little") + self.rnum.to_bytes(8, "little")
            self.rnum += 1
            v = int.from_bytes(hashlib.sha256(self.data).digest(), "big") & P61
            if v < self.bound:
                return v
            self.redrawn += 1

    def element(self, label):
        out = []
        for part in (b"real", b"imag"):
            for t in (b"ext", label, part):
                self.text(t)
            out.append(self.scalar())
        return out


def start(lib):
    st = np.zeros((STATES, lib.redraw_state_bytes()), np.uint8)
    lib.redraw_start(P(st), STATES, 1)
    return st


def host(lib, label):
    st, out = start(lib), np.zeros((STATES, DRAWS, 2), np.uint64)
    lib.redraw_host(P(st), STATES, DRAWS, label, P(out))
    return st, out


@pytest.mark.parametrize("label", LABELS)
def test_host_against_hashlib(built, label):
    lib, bound = built
    _, got = host(lib, label)
    again = 0
    for i in range(STATES):
        t = Transcript(bytes((7 * j + 3) & 255 for j in range(64 + i)), bound)
        for k in range(DRAWS):
            for j in range(k):
                t.data += b"\x03" + (1000 + k).to_bytes(8, "little") + j.to_bytes(8, "little")
            assert got[i, k].tolist() == t.element(label)
        again += t.redrawn
    assert again > STATES * DRAWS       # most limbs more than once


@pytest.mark.gpu
@pytest.mark.parametrize("label", LABELS)
def test_device_against_host(built, label):
    lib, _ = built
    want_st, want = host(lib, label)
    st, out = start(lib), np.zeros((STATES, DRAWS, 2), np.uint64)
    assert lib.redraw_device(P(st), STATES, DRAWS, label, P(out)) == 0
    np.testing.assert_array_equal(out, want)
    np.testing.assert_array_equal(st, want_st)
