"""Device transcripts of so many states that each has a thread, against the same states
in calls of few, which have a warp each: puts, draws and VOLE-committed rounds at every
offset within a block, the last states short of correlations."""
import ctypes
import struct

import numpy as np
import pytest

from fp2lib import P61

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("extra", [1, 300])
def test_threads_against_warps(extra):
    import torch
    from truepix_b200 import native
    lib = native.gkr()
    n = 8 * torch.cuda.get_device_properties(0).multi_processor_count + extra
    few, nb, vb = 500, lib.tp_fs_state_bytes(), lib.tp_vole_state_bytes()
    base = []
    for k in range(64):
        st = ctypes.create_string_buffer(nb)
        assert lib.tp_fs_init(st, b"many") == 0 and lib.tp_fs_absorb(st, bytes(range(k + 1)), k + 1) == 0
        base.append(st.raw)
    vs = ctypes.create_string_buffer(vb)
    assert lib.tp_vole_state_init(vs, 0, None) == 0
    rng = np.random.default_rng(extra)
    dev = lambda a: torch.from_numpy(np.array(a)).cuda()
    field = lambda *shape: dev(rng.integers(0, P61, size=shape + (2,)).astype(np.int64))
    states = dev(np.frombuffer(b"".join(base[f % 64] for f in range(n)), np.uint8))
    count = 9                                # two rounds of four; a third runs out
    vals, claims, u, v = field(n, 3), field(3, n, 4), field(n, count), field(n, count)
    s = torch.cuda.current_stream().cuda_stream

    def run(step):
        st, vo = states.clone(), dev(np.frombuffer(vs.raw * n, np.uint8))
        draws, chal = torch.zeros(n, 2, dtype=torch.int64, device="cuda"), []
        proof = torch.zeros(3, n, 5, 2, dtype=torch.int64, device="cuda")
        for a in range(0, n, step):
            m = min(step, n - a)
            fs, w = st.data_ptr() + a * nb, vo.data_ptr() + a * vb
            assert lib.tp_fs_put_fp2s_dev(fs, m, vals[a:].data_ptr(), 3, s) == 0
            assert lib.tp_fs_rand_ext_dev(fs, m, b"a label", draws[a:].data_ptr(), s) == 0
        for k in range(3):
            c = torch.zeros(n, 2, dtype=torch.int64, device="cuda")
            for a in range(0, n, step):
                m = min(step, n - a)
                assert lib.tp_vole_round_dev(st.data_ptr() + a * nb, vo.data_ptr() + a * vb, m, claims[k, a:].data_ptr(),
                                             u[a:].data_ptr(), v[a:].data_ptr(), count, b"sc-0-%d" % k,
                                             c[a:].data_ptr(), proof[k, a:].data_ptr(), s) == 0, lib.tp_last_error()
            chal.append(c.cpu())
        return st.cpu().numpy().reshape(n, nb), vo.cpu(), draws.cpu(), torch.stack(chal), proof.cpu()

    got, want = run(n), run(few)
    for a, b in zip(got[1:], want[1:]):
        assert torch.equal(a, b)
    for f in range(n):                       # the bytes behind the pending ones are stale
        a, b = got[0][f].tobytes(), want[0][f].tobytes()
        pending = struct.unpack_from("<I", b, 112)[0]
        assert a[:32 + pending] == b[:32 + pending] and a[96:116] == b[96:116], f
