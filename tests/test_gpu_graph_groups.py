"""Uneven batches under layers with product groups in one CUDA graph of VOLE-committed
rounds, against each frame alone launch by launch: frames that leave early, on rows and on
vectors, rounds a launch each and the last ones in one CTA a frame; a replay on other
bytes."""
import ctypes

import numpy as np
import pytest

import test_gpu_linear_rounds as rounds
from fp2lib import P61

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("groups,copies", [
    (1, [300, 70, 1000, 9, 300, 2]), (3, [2, 4, 9000, 700]), (4, [4000, 8192, 30]), (5, [20000, 3, 500]),
    (17, [40, 300])])
def test_uneven_batch(groups, copies):
    import torch
    from truepix_b200 import native
    from truepix_b200.frame import BatchFrameProver, FrameLayout
    from truepix_b200.pipeline import correlations_needed
    lib = native.gkr()
    rng = np.random.default_rng(groups)
    gates = rounds.layer(rng, 512, groups, 385)
    G = gates[0].size
    layouts = [FrameLayout(copies=c) for c in copies]
    B = len(layouts)
    field = lambda *shape: rng.integers(0, P61, size=shape, dtype=np.uint64)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a).reshape(-1).view(np.int64)).cuda()
    z2 = [field(L.n_copy_bits, 2) for L in layouts]
    count = max(correlations_needed(L) for L in layouts)
    u, v = field(B, count, 2), field(B, count, 2)
    states = []
    for f in range(B):
        st = ctypes.create_string_buffer(lib.tp_fs_state_bytes())
        assert lib.tp_fs_init(st, b"uneven") == 0
        pre = np.arange(f + 1, dtype=np.uint64)
        assert lib.tp_fs_put_u64s(st, pre.ctypes.data, pre.size) == 0
        states.append(st.raw)
    vs0 = ctypes.create_string_buffer(lib.tp_vole_state_bytes())
    assert lib.tp_vole_state_init(vs0, 0, None) == 0

    def prover(idx):
        return BatchFrameProver([layouts[f] for f in idx], *gates, stream=torch.cuda.Stream())

    def run(bp, idx, frames, zg, graph):
        z2d, ptd = {}, {}
        for C in sorted({layouts[f].padded_copies for f in idx}):
            fs = [f for f in idx if layouts[f].padded_copies == C]
            z2d[C] = dev(np.concatenate([z2[f] for f in fs]))
            ptd[C] = torch.zeros(2 * len(fs) * (8 + C.bit_length()), dtype=torch.int64, device="cuda")
        d_st = torch.from_numpy(np.frombuffer(b"".join(states[f] for f in idx), np.uint8).copy()).cuda()
        vole = dict(states=torch.from_numpy(np.frombuffer(vs0.raw * len(idx), np.uint8).copy()).cuda(), u=dev(u[idx]),
                    v=dev(v[idx]), count=count)
        torch.cuda.synchronize()
        bp.prove([frames[f] for f in idx], [zg[f] for f in idx], z2d, ptd, None, transcripts=d_st, vole=vole,
                 graph=graph)
        bp.stream.synchronize()
        R, n = bp.max_rounds, len(idx)
        of = lambda t, *shape: t.cpu().numpy().reshape(*shape)
        return dict(claims=of(bp.claims, R, n, 8), chal=of(bp.device_challenges, R, n, 2),
                    proof=of(bp.device_proof, R, n, 10), wires=of(bp.wires, n, -1), beta=of(bp.fin_beta, n, 2),
                    st=of(d_st, n, -1), vs=of(vole["states"], n, -1))

    whole = prover(list(range(B)))
    for replay in range(2):
        frames = [torch.from_numpy(rng.integers(0, 256, size=c * 384, dtype=np.uint8)).cuda() for c in copies]
        zg = [field(2, G) for _ in range(B)]
        got = run(whole, list(range(B)), frames, zg, True)
        assert lib.tp_batch_graph_replays(whole.handle) == replay + 1
        for f in range(B):
            want = run(prover([f]), [f], frames, zg, False)
            r = layouts[f].n_copy_bits
            for k in ("claims", "chal", "proof"):
                np.testing.assert_array_equal(got[k][:r, f], want[k][:r, 0], err_msg="%s %d" % (k, f))
            for k in ("wires", "beta", "st", "vs"):
                np.testing.assert_array_equal(got[k][f], want[k][0], err_msg="%s %d" % (k, f))
