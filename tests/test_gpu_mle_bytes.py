"""The batched input MLE over bytes against integer arithmetic: copies around a CTA's
512 and a step's 32, copy sizes around a warp's 32 wires, rows that are whole aligned
words and rows that are not, frames of different lengths (none at all included), all
bytes 255 and the largest challenges."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
P61 = 2**61 - 1


def mul(a, b):
    return (a[0] * b[0] - a[1] * b[1]) % P61, (a[0] * b[1] + a[1] * b[0]) % P61


def eq_table(z):
    t = [(1, 0)]
    for x in z:
        y = ((1 - x[0]) % P61, -x[1] % P61)
        t = [mul(v, y) for v in t] + [mul(v, x) for v in t]
    return t


def weighted(weights, x):
    """sum_c weights[c] x[c][w] for every w, exactly, by 31-bit limbs"""
    out = []
    for part in (0, 1):
        w = np.array([v[part] for v in weights], dtype=object)
        lo = (w & 0x7FFFFFFF).astype(np.int64) @ x
        hi = (w >> 31).astype(np.int64) @ x
        out.append([(int(a) + (int(b) << 31)) % P61 for a, b in zip(lo, hi)])
    return list(zip(*out))


@pytest.mark.parametrize("extreme", [False, True])
@pytest.mark.parametrize("cs,const,W,n_pad,counts,offset", [
    (1, 1, 2, 2, [1, 2], 0), (3, -1, 4, 4, [3], 1), (31, 31, 32, 64, [31, 32, 33], 0), (32, -1, 32, 64, [64, 1], 4),
    (33, 40, 64, 512, [511, 512], 0), (36, 63, 64, 1024, [513, 0, 1024], 8), (96, 100, 128, 2048, [1025, 544], 2),
    (384, 384, 512, 2048, [2048, 1535, 1537], 0), (384, 500, 512, 1024, [700], 3), (511, 511, 512, 512, [77], 0),
    (512, -1, 512, 1024, [545], 0),
    # pieces enough that a CTA takes several, the last one's short or missing
    (16, -1, 16, 32768, [17000, 32768, 1, 512, 8193, 30000, 29999, 24577] * 3, 0),
    (12, 13, 16, 65536, [65536, 40001, 50000, 61440] * 2, 4)])
def test_mle(cs, const, W, n_pad, counts, offset, extreme):
    import torch
    from truepix_b200 import native
    lib = native.gkr()
    rng = np.random.default_rng(cs * 1000 + n_pad)
    nz = W.bit_length() - 1 + n_pad.bit_length() - 1
    const_val = P61 - 1 if extreme else int(rng.integers(P61)) if const >= 0 else 0
    const_val = const_val if const >= 0 else 0
    bufs, ptrs, rows, points = [], [], [], []
    for n in counts:
        x = np.full((n, cs), 255, np.uint8) if extreme else rng.integers(0, 256, (n, cs), dtype=np.uint8)
        b = torch.full((max(1, n * cs) + offset,), 99, dtype=torch.uint8, device="cuda")
        b[offset:offset + n * cs] = torch.from_numpy(x.reshape(-1)).cuda()
        bufs.append(b)
        ptrs.append(b.data_ptr() + offset)
        rows.append(x)
        points.append([(P61 - 1, P61 - 2)] * nz if extreme else [tuple(map(int, rng.integers(0, P61, 2))) for _ in range(nz)])
    z = torch.from_numpy(np.array(points, np.uint64).view(np.int64)).cuda()
    out = torch.zeros(2 * len(counts), dtype=torch.int64, device="cuda")
    rc = lib.tp_mle_eval_pixels_batch(len(counts), (ctypes.c_void_p * len(counts))(*ptrs),
                                      (ctypes.c_int * len(counts))(*counts), n_pad, cs, W, const, const_val,
                                      z.data_ptr(), out.data_ptr(), torch.cuda.current_stream().cuda_stream)
    native.check(lib, rc, "mle")
    got = out.cpu().numpy().view(np.uint64).reshape(-1, 2).tolist()
    h = W.bit_length() - 1
    for f, n in enumerate(counts):
        lo, hi = eq_table(points[f][:h]), eq_table(points[f][h:])[:n]
        y = weighted(hi, rows[f].astype(np.int64)) if n else [(0, 0)] * cs
        terms = [mul(l, v) for l, v in zip(lo, y)]
        if const >= 0:
            s = sum(v[0] for v in hi) % P61, sum(v[1] for v in hi) % P61
            terms.append(mul(lo[const], mul(s, (const_val, 0))))
        assert got[f] == [sum(t[0] for t in terms) % P61, sum(t[1] for t in terms) % P61], f


def test_slots():
    """the values placed at given indices, in the caller's workspace; a negative index and
    a workspace too small are refused"""
    import torch
    from truepix_b200 import native
    lib = native.gkr()
    rng = np.random.default_rng(5)
    x = torch.from_numpy(rng.integers(0, 256, (3, 4 * 16), dtype=np.uint8)).cuda()
    z = torch.from_numpy(rng.integers(0, P61, (3, 6, 2)).astype(np.int64)).cuda()
    s = torch.cuda.current_stream().cuda_stream
    args = (3, (ctypes.c_void_p * 3)(*[x[i].data_ptr() for i in range(3)]), (ctypes.c_int * 3)(4, 3, 4), 4, 16, 16, -1, 0,
            z.data_ptr())
    a = torch.zeros(3, 2, dtype=torch.int64, device="cuda")
    ws = torch.empty(3 * 36, dtype=torch.uint8, device="cuda")
    b = torch.full((7, 2), -1, dtype=torch.int64, device="cuda")
    native.check(lib, lib.tp_mle_eval_pixels_batch(*args, a.data_ptr(), s), "mle")
    native.check(lib, lib.tp_mle_eval_pixels_batch_at(*args, (ctypes.c_int * 3)(6, 0, 3), b.data_ptr(), ws.data_ptr(),
                                                      ws.numel(), s), "mle at")
    assert torch.equal(b[[6, 0, 3]], a) and bool((b[[1, 2, 4, 5]] == -1).all())
    assert lib.tp_mle_eval_pixels_batch_at(*args, (ctypes.c_int * 3)(0, -1, 2), b.data_ptr(), None, 0, s) != 0
    assert lib.tp_mle_eval_pixels_batch_at(*args, None, b.data_ptr(), ws.data_ptr(), 3 * 36 - 1, s) != 0


def test_beside_the_rounds(monkeypatch):
    """MLEs on a stream of their own (large batches) and behind the rounds: the same
    values in two passes over different bytes, for one padded size and for two"""
    import torch
    from truepix_b200.frame import BatchFrameProver, FrameLayout
    rng = np.random.default_rng(9)
    G = 300
    gt, i0, i1 = rng.choice([1, 2, 3], size=G), rng.integers(0, 384, G), rng.integers(0, 384, G)
    for counts in ([100, 128, 90], [100, 60, 128, 33]):
        layouts = [FrameLayout(copies=c, copy_size=384, const_idx=400, const_val=7) for c in counts]
        got = {}
        for aside in (False, True):
            monkeypatch.setattr(BatchFrameProver, "MLE_ASIDE", 1 if aside else 1 << 62)
            p = BatchFrameProver(layouts, gt, i0, i1)
            rng = np.random.default_rng(11)
            field = lambda *shape: rng.integers(0, P61, shape).astype(np.int64)
            for _ in range(2):
                pix = [torch.from_numpy(rng.integers(0, 256, c * 384, dtype=np.uint8)).cuda() for c in counts]
                z1 = [field(2, G).astype(np.uint64) for _ in counts]
                z2, pt = {}, {}
                for C, fs in p.groups.items():
                    nb = C.bit_length() - 1
                    z2[C] = torch.from_numpy(field(len(fs), nb, 2)).cuda()
                    pt[C] = torch.from_numpy(field(len(fs), layouts[0].n_in_bits + nb, 2)).cuda()
                p.prove(pix, z1, z2, pt, field(p.max_rounds, len(counts), 2).astype(np.uint64))
                got.setdefault(aside, []).append((p.mle.cpu(), p.claims.cpu(), p.wires.cpu()))
        for a, b in zip(got[False], got[True]):
            assert all(torch.equal(x, y) for x, y in zip(a, b))
