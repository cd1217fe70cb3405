"""Early rounds on per-copy vectors (gkr_linear.cu) against the oracle's session:
layers with few product groups over every source (bytes at any alignment, copy
sizes around the 32-byte steps of the matrix product, tables), the operations in
orders a session allows (folds without claims, a finish before the last round),
the caller's bytes overwritten once the first claim or fold has run, and the
neighbouring layers whose rounds stay on the table of all wires."""
import ctypes

import numpy as np
import pytest

from fp2lib import P61, Fp2Lib, ORACLE_LIB, rand_fp

pytestmark = pytest.mark.gpu
V = ctypes.c_void_p


@pytest.fixture(scope="module")
def lib():
    from truepix_b200 import native
    return native.gkr()


@pytest.fixture(scope="module")
def oracle():
    return Fp2Lib(ORACLE_LIB, "oracle_fp2_")


def layer(rng, W, groups, top, n_gates=300):
    """gates over the wires below top: linear kinds, and products with `groups` wires"""
    gt = rng.choice([1, 2, 3, 4, 7, 12], size=n_gates).astype(np.int32)
    i0 = rng.integers(0, top, size=n_gates).astype(np.int32)
    i1 = rng.integers(0, top, size=n_gates).astype(np.int32)
    if groups:
        shared = rng.choice(top, size=groups, replace=False)
        n = max(groups, n_gates // 2)
        gt[:n] = rng.choice([0, 5, 6, 8, 11], size=n)
        i1[:n] = np.concatenate([shared, rng.choice(shared, size=n - groups)])
        # wires of a group other than the shared ones, so that every group is kept
        rest = np.setdiff1d(np.arange(top), shared)
        i0[:n] = rng.choice(rest, size=n) if rest.size else i0[:n]
    return gt, i0, i1


def play(oracle, lib, handle, gates, z, C, W, table, beta, ops, chal):
    """the operations on both sides; claims, then wires and beta"""
    import torch
    oh = oracle.early_create(*gates, z[0], z[1], C, W, table, np.zeros_like(table), beta[0], beta[1])
    claims = torch.zeros(8, dtype=torch.int64, device="cuda")
    fin = torch.zeros(2 * (W + 1), dtype=torch.int64, device="cuda")
    k = 0
    for op in ops:
        if op == "c":
            assert lib.tp_early_claim_dev(handle, claims.data_ptr()) == 0, lib.tp_last_error()
            rc, want = oracle.early_claim(oh)
            assert rc == 0
            np.testing.assert_array_equal(claims.cpu().numpy().view(np.uint64), want, err_msg="claim at fold %d" % k)
        elif op == "f":
            r = (int(chal[k][0]), int(chal[k][1]))
            assert lib.native_fp2_early_fold(handle, *r) == 0, lib.tp_last_error()
            assert oracle.early_fold(oh, r) == 0
            k += 1
        elif isinstance(op, int):     # op rounds in one call
            out = torch.zeros(8 * op, dtype=torch.int64, device="cuda")
            ch = np.ascontiguousarray(chal[k:k + op]).reshape(-1)
            assert lib.tp_early_rounds_dev(handle, op, ch.ctypes.data_as(ctypes.POINTER(ctypes.c_uint64)),
                                           out.data_ptr()) == 0, lib.tp_last_error()
            got = out.cpu().numpy().view(np.uint64).reshape(op, 8)
            for q in range(op):
                rc, want = oracle.early_claim(oh)
                assert rc == 0
                np.testing.assert_array_equal(got[q], want, err_msg="round %d" % (k + q))
                assert oracle.early_fold(oh, (int(chal[k + q][0]), int(chal[k + q][1]))) == 0
            k += op
        else:
            assert lib.tp_early_finish_dev(handle, fin.data_ptr(), fin.data_ptr() + 16 * W) == 0, lib.tp_last_error()
            rc, re, im, b = oracle.early_finish(oh, W)
            assert rc == 0
            f = fin.cpu().numpy().view(np.uint64).reshape(W + 1, 2)
            np.testing.assert_array_equal(f[:W, 0], re)
            np.testing.assert_array_equal(f[:W, 1], im)
            assert (int(f[W, 0]), int(f[W, 1])) == b
    oracle.early_destroy(oh)
    lib.native_fp2_early_destroy(handle)


def orders(nb):
    """operation orders over nb rounds"""
    whole = ["c", "f"] * nb + ["x"]
    out = [whole, [nb, "x"], ["f"] + ["c", "f"] * (nb - 1) + ["x"], ["f"] * nb + ["x"], ["x"]]
    if nb >= 3:
        out += [["c", "f", "f"] + ["c", "f"] * (nb - 2) + ["x"], ["c", "f", "x", nb - 1, "x"], ["f", nb - 1, "x"],
                [2, "c", "f", "x"] + ([nb - 3, "x"] if nb > 3 else [])]
    return out


CASES = [  # wires, copy size, real copies, padded copies, constant wire, product groups, byte offset
    (512, 384, 1000, 1024, 384, 0, 0), (512, 384, 1000, 1024, 384, 1, 3), (512, 385, 700, 1024, 385, 1, 0),
    (512, 384, 37, 64, -1, 3, 16), (512, 512, 511, 512, -1, 16, 0), (512, 512, 513, 1024, -1, 17, 0),
    (64, 31, 65, 128, 40, 1, 1), (64, 32, 64, 64, 32, 2, 0), (64, 33, 63, 64, -1, 0, 15), (64, 1, 5, 8, 63, 0, 0),
    (64, 48, 2, 2, -1, 1, 0), (128, 96, 0, 4, 100, 1, 0), (512, 384, 9000, 16384, 384, 1, 0),
]


@pytest.mark.parametrize("W,cs,real,C,const,groups,off", CASES)
def test_bytes_source(lib, oracle, W, cs, real, C, const, groups, off):
    import torch
    rng = np.random.default_rng(W * 31 + cs * 7 + real + groups)
    top = max(cs, const + 1)
    gates = layer(rng, W, groups, top)
    z, beta = [rand_fp(rng, 300), rand_fp(rng, 300)], [rand_fp(rng, C), rand_fp(rng, C)]
    nb = C.bit_length() - 1
    chal = np.stack([rand_fp(rng, nb), rand_fp(rng, nb)], axis=1)
    chal[0] = (P61 - 1, 0)
    pix = rng.integers(0, 256, size=real * cs, dtype=np.uint8)
    pix[:cs] = 255
    vals = np.zeros((C, W), np.uint64)
    vals[:real, :cs] = pix.reshape(real, cs)
    if const >= 0:
        vals[:real, const] = P61 - 2
    table = np.ascontiguousarray(vals.T).reshape(-1)
    d_beta = torch.from_numpy(np.stack(beta, axis=1).reshape(-1).view(np.int64)).cuda()
    s = torch.cuda.current_stream().cuda_stream
    for ops in orders(nb) if C <= 1024 else orders(nb)[:2]:
        room = torch.zeros(off + real * cs + 1, dtype=torch.uint8, device="cuda")
        d_pix = room[off:off + real * cs]
        d_pix.copy_(torch.from_numpy(pix))
        h = lib.tp_early_create_pixels(300, *[V(a.ctypes.data) for a in gates], V(z[0].ctypes.data),
                                       V(z[1].ctypes.data), room.data_ptr() + off, real, C, cs, W, const,
                                       P61 - 2 if const >= 0 else 0, d_beta.data_ptr(), s)
        assert h, lib.tp_last_error()
        play(oracle, Overwriting(lib, d_pix), h, gates, z, C, W, table, beta, ops, chal)


class Overwriting:
    """the library, with the caller's bytes overwritten once the first fold has run
    (behind the second claim): the session holds what it needs from there on"""

    def __init__(self, lib, d_pix):
        self.lib, self.d_pix, self.claims = lib, d_pix, 0

    def __getattr__(self, name):
        return getattr(self.lib, name)

    def tp_early_claim_dev(self, handle, out):
        rc = self.lib.tp_early_claim_dev(handle, out)
        self.claims += 1
        if self.claims == 2:
            self.d_pix.fill_(7)
        return rc


@pytest.mark.parametrize("W,C,groups", [(512, 64, 0), (512, 1024, 1), (100, 32, 3), (512, 8, 16), (40, 2, 1), (64, 512, 17)])
def test_table_source(lib, oracle, W, C, groups):
    import torch
    rng = np.random.default_rng(W + C + groups)
    gates = layer(rng, W, groups, W)
    z, beta = [rand_fp(rng, 300), rand_fp(rng, 300)], [rand_fp(rng, C), rand_fp(rng, C)]
    nb = C.bit_length() - 1
    chal = np.stack([rand_fp(rng, nb), rand_fp(rng, nb)], axis=1)
    re, im = rand_fp(rng, W * C), rand_fp(rng, W * C)
    re[:5] = P61 - 1
    s = torch.cuda.current_stream().cuda_stream
    for borrow in (0, 1):
        for ops in orders(nb):
            d_v = torch.from_numpy(np.stack([re, im], axis=1).reshape(-1).view(np.int64)).cuda()
            d_b = torch.from_numpy(np.stack(beta, axis=1).reshape(-1).view(np.int64)).cuda()
            h = lib.tp_early_create_dev(300, *[V(a.ctypes.data) for a in gates], V(z[0].ctypes.data),
                                        V(z[1].ctypes.data), C, W, d_v.data_ptr(), d_b.data_ptr(), borrow, s)
            assert h, lib.tp_last_error()
            if not borrow:
                d_v.zero_()         # the session holds a copy
                d_b.zero_()
            oracle_create = oracle.early_create

            class Both:
                """the oracle with the table's imaginary limbs"""
                def __getattr__(self, name):
                    return getattr(oracle, name)

                def early_create(self, *a):
                    return oracle_create(*a[:7], re, im, *a[9:])
            play(Both(), lib, h, gates, z, C, W, re, beta, ops, chal)
