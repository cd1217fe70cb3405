"""Performance cases: the work a user of truepix_b200 has the library do.

Every case is a dict of plain values; `prepare` makes what the user's program
holds before the call (inputs on the GPU, made from the seed, and the prover,
committer or layer handle it keeps), `run` makes one pass through the public
entry points and returns all outputs.

Kinds, and what each stands for:

  gkr_frame   the GKR input layer of one frame proved by itself
              (GkrInputLayerProver): the latency of an interactive prover, small
              frames; circuits with and without product gates
  gkr_batch   the GKR input layer of a batch of frames on device transcripts
              with VOLE-committed rounds, as the pipelined prover runs it: early
              rounds as one graph, late rounds and closing proofs
              (BatchFrameProver.prove and prove_late)
  gkr_mixed   the early rounds of frames of several sizes in one batch, with
              the challenges of host transcripts (crops of one clip)
  commit      Orion commitments of frames from their bytes (FrameCommitter),
              plain, or the zero-knowledge pair of masked frame and mask; alone
              or on the committer's side streams
  opening     the device passes of an Orion opening over a codeword held in HBM:
              combined codeword with its tree, answer, queried columns, Merkle
              nodes
  ntt         a forward transform with zero padding and an inverse transform,
              some of them batched
  rs          the rate-2^-5 Reed-Solomon commit of a witness and the chain of
              FRI commit steps over its codeword down to four points a slice
  virgo       both phases of a layer of the Virgo sumcheck: table inits and all
              rounds
  session     the reference-facing C ABI with host buffers: beta table, early
              session round by round, input MLE (the drop-in library under
              TruePix's own Python prover)
  prove       whole proofs of small frames in the default zero-knowledge mode,
              one step after another: commit, proof container, both openings

Frame sizes are the video sizes of the benchmark and the tests (240p to 2160p)
and odd crops; transforms and layers span the sizes the tests and the benchmark
use.
"""
import ctypes
import math
import os

import numpy as np
import torch

from truepix_b200 import native
from truepix_b200.frame import BatchFrameProver, FrameLayout, GkrInputLayerProver, pack_fp2
from truepix_b200.opening import opening_proof, query_count
from truepix_b200.orion import FrameCommitter
from truepix_b200.pipeline import correlations_needed
from truepix_b200.prover import manifests_of, prove_frames

P61 = (1 << 61) - 1
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(native.__file__)))
COPY = 384                       # bytes of a frame in one copy of the circuit


def listed():
    return [
        # one small frame, interactive latency; crop has product gates
        dict(name="gkr_frame_240p", kind="gkr_frame", height=240, width=426, circuit="Crop"),
        # the serving pipeline's batch of full-HD frames
        dict(name="gkr_batch_1080p", kind="gkr_batch", height=1080, width=1920, frames=64, circuit="gray", zk=False),
        # crops of one clip, sizes from 240p to 1080p in one batch
        dict(name="gkr_mixed_12", kind="gkr_mixed", height=1080, width=1920, frames=12, circuit="gray"),
        # one frame's commitment, latency
        dict(name="commit_360p", kind="commit", height=360, width=640, frames=1, zk=False, streams=0),
        # commitments under load: the pipeline's side streams
        dict(name="commit_1080p_x4", kind="commit", height=1080, width=1920, frames=4, zk=False, streams=8),
        # TruePix's default, the zero-knowledge pair
        dict(name="commit_zk_720p", kind="commit", height=720, width=1280, frames=1, zk=True, streams=0),
        dict(name="opening_1080p", kind="opening", height=1080, width=1920),
        dict(name="ntt_2e20", kind="ntt", log_n=20, pad=2, batch=1),
        dict(name="rs_fri_2e16", kind="rs", log_len=16),
        dict(name="virgo_2e18", kind="virgo", length_g=18, length_u=18),
        dict(name="session_480p", kind="session", height=480, width=854, circuit="gray"),
        dict(name="prove_zk_360p", kind="prove", height=360, width=640, frames=1, circuit="gray"),
    ]


def _size(rng, low, high):
    """a frame height in [low, high], spread over its logarithm, and a width near 16:9"""
    h = int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))
    return h, max(16, int(h * rng.uniform(1.3, 1.8)))


def draw(rng):
    kind = rng.choice(["gkr_frame", "gkr_batch", "gkr_mixed", "commit", "commit", "opening", "ntt", "rs", "virgo",
                       "session", "prove"])
    circuit = rng.choice(["gray", "inv", "mask", "Crop"])
    if kind == "gkr_frame":
        h, w = _size(rng, 60, 1080)
        return dict(kind=kind, height=h, width=w, circuit=circuit)
    if kind == "gkr_batch":
        h, w = _size(rng, 120, 1080)
        return dict(kind=kind, height=h, width=w, frames=int(round(math.exp(rng.uniform(0, math.log(64))))),
                    circuit=circuit, zk=rng.random() < 0.5)
    if kind == "gkr_mixed":
        h, w = _size(rng, 360, 1080)
        return dict(kind=kind, height=h, width=w, frames=rng.randint(2, 16), circuit=circuit)
    if kind == "commit":
        h, w = _size(rng, 60, 1440)
        room = max(1, 4 * 16200 * COPY // (h * w * 3))
        zk = rng.random() < 0.5
        return dict(kind=kind, height=h, width=w, frames=rng.randint(1, min(8, max(1, room // (2 if zk else 1)))),
                    zk=zk, streams=rng.choice([0, 0, 8]))
    if kind == "opening":
        h, w = _size(rng, 120, 1440)
        return dict(kind=kind, height=h, width=w)
    if kind == "ntt":
        log_n = rng.randint(6, 20)
        return dict(kind=kind, log_n=log_n, pad=rng.randint(0, min(5, log_n)),
                    batch=1 << rng.randint(0, max(0, min(6, 21 - log_n))))
    if kind == "rs":
        return dict(kind=kind, log_len=rng.randint(8, 17))
    if kind == "virgo":
        return dict(kind=kind, length_g=rng.randint(6, 19), length_u=rng.randint(6, 19))
    if kind == "session":
        h, w = _size(rng, 60, 720)
        return dict(kind=kind, height=h, width=w, circuit=circuit)
    h, w = _size(rng, 120, 360)
    return dict(kind=kind, height=h, width=w, frames=rng.randint(1, 2), circuit=circuit)


# ---- inputs ---------------------------------------------------------------------

_circuits = {}


def _circuit(name):
    """gate tables of one of TruePix's circuits and the layout constants they use"""
    if not _circuits:
        c = np.load(os.path.join(ROOT, "tests", "golden", "circuits.npz"))
        for k in ("gray", "inv", "mask", "Crop"):
            consts = c[k + "_consts"]
            idx, val = (int(consts[0][0]), int(consts[0][1])) if len(consts) else (-1, 0)
            _circuits[k] = (*(np.ascontiguousarray(c[k + s], np.int32) for s in ("_type", "_in0", "_in1")),
                            int(c[k + "_ninputs"][0]), idx, val)
    return _circuits[name]


def _layout(case, height=None, width=None):
    """the frame's layout under the case's circuit (no circuit: gray's)"""
    _, _, _, ninputs, idx, val = _circuit(case.get("circuit") or "gray")
    n = (height or case["height"]) * (width or case["width"]) * 3
    return FrameLayout(copies=-(-n // ninputs), copy_size=ninputs, const_idx=idx, const_val=val)


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _bytes(g, n):
    return torch.randint(0, 256, (n,), dtype=torch.uint8, device="cuda", generator=g)


def _field(g, n):
    """n canonical field elements as packed pairs of limbs, on the device"""
    return torch.randint(0, P61, (2 * n,), dtype=torch.int64, device="cuda", generator=g)


def _host_field(rng, *shape):
    return rng.integers(0, P61, size=shape, dtype=np.uint64)


def _frame(g, L):
    return _bytes(g, L.copies * L.copy_size)


def _transcripts(lib, rng, frames):
    """fresh Fiat-Shamir and VOLE states of a batch, as the IO prefix leaves them"""
    fs, vs = b"", b""
    for _ in range(frames):
        s = ctypes.create_string_buffer(lib.tp_fs_state_bytes())
        native.check(lib, lib.tp_fs_init(s, b"truepix"), "tp_fs_init")
        put = _host_field(rng, 5)
        native.check(lib, lib.tp_fs_put_u64s(s, put.ctypes.data, put.size), "tp_fs_put_u64s")
        fs += s.raw
        v = ctypes.create_string_buffer(lib.tp_vole_state_bytes())
        native.check(lib, lib.tp_vole_state_init(v, 0, None), "tp_vole_state_init")
        vs += v.raw
    as_dev = lambda b: torch.from_numpy(np.frombuffer(b, np.uint8).copy()).cuda()
    return as_dev(fs), as_dev(vs)


def prepare(case, seed):
    lib = native.gkr()
    g, rng = _gen(seed), np.random.default_rng(seed)
    kind = case["kind"]
    s = {"case": case, "lib": lib}
    if kind == "gkr_frame":
        gt, i0, i1 = _circuit(case["circuit"])[:3]
        L = _layout(case)
        s.update(pix=_frame(g, L), z1=_host_field(rng, 2, gt.size), z2=_field(g, L.n_copy_bits),
                 pt=_field(g, L.n_in_bits + L.n_copy_bits), ch=_host_field(rng, L.n_copy_bits, 2),
                 prover=GkrInputLayerProver(L, gt, i0, i1))
    elif kind == "gkr_batch":
        gt, i0, i1 = _circuit(case["circuit"])[:3]
        L, B = _layout(case), case["frames"]
        nb, count = L.n_copy_bits, correlations_needed(L, case["zk"])
        fs, vs = _transcripts(lib, rng, B)
        stream = torch.cuda.Stream()
        s.update(pix=[_frame(g, L) for _ in range(B)], z1=[_host_field(rng, 2, gt.size) for _ in range(B)],
                 z2=_field(g, B * nb), pt=_field(g, B * (L.n_in_bits + nb)), fs0=fs, vs0=vs, fs=fs.clone(),
                 vole=dict(states=vs.clone(), u=_field(g, B * count), v=_field(g, B * count), count=count),
                 stream=stream, prover=BatchFrameProver([L] * B, gt, i0, i1, stream=stream))
    elif kind == "gkr_mixed":
        gt, i0, i1 = _circuit(case["circuit"])[:3]
        B = case["frames"]
        # frame f is a crop of the source: heights and widths from a quarter to the whole
        sides = [(max(16, int(case["height"] * a)), max(16, int(case["width"] * b)))
                 for a, b in np.random.default_rng(B).uniform(0.22, 1.0, size=(B, 2))]
        Ls = [_layout(case, h, w) for h, w in sides]
        z2, pt = {}, {}
        for C in sorted({L.padded_copies for L in Ls}):
            n, nb = sum(L.padded_copies == C for L in Ls), int(math.log2(C))
            z2[C], pt[C] = _field(g, n * nb), _field(g, n * (Ls[0].n_in_bits + nb))
        prover = BatchFrameProver(Ls, gt, i0, i1)
        s.update(pix=[_frame(g, L) for L in Ls], z1=[_host_field(rng, 2, gt.size) for _ in Ls], z2=z2, pt=pt,
                 ch=_host_field(rng, prover.max_rounds, B, 2), prover=prover)
    elif kind == "commit":
        L, B = _layout(case), case["frames"]
        s.update(pix=[_frame(g, L) for _ in range(B)],
                 seeds=[int(x) for x in rng.integers(0, 1 << 63, size=B)] if case["zk"] else None,
                 committer=FrameCommitter([L] * B, side_streams=case["streams"], zk=case["zk"]))
    elif kind == "opening":
        L = _layout(case)
        N = L.padded_copies * L.n_wires
        cw, leaves = lib.tp_orion_codeword_len(N // 128), lib.tp_orion_tree_leaves(N)
        q = rng.integers(0, cw, size=query_count(), dtype=np.int64)
        nodes = np.zeros(q.size * leaves.bit_length(), np.int32)    # at most: a whole path per query
        n_nodes = lib.tp_orion_path_nodes(leaves, q.ctypes.data, q.size, nodes.ctypes.data, nodes.size)
        native.check(lib, 0 if n_nodes >= 0 else -1, "tp_orion_path_nodes")
        empty = lambda n, t=torch.int64: torch.empty(n, dtype=t, device="cuda")
        s.update(N=N, cw=cw, leaves=leaves, n_nodes=n_nodes, rows=_field(g, 128 * cw), tree=_bytes(g, 64 * leaves),
                 r0=_field(g, 128), r1=_field(g, N // 128), q=torch.from_numpy(q).cuda(),
                 idx=torch.from_numpy(nodes[:n_nodes]).cuda(), comb=empty(2 * cw),
                 ctree=torch.zeros(64 * leaves, dtype=torch.uint8, device="cuda"), ans=empty(2),
                 cols=empty(256 * q.size), com=torch.zeros(32 * nodes.size, dtype=torch.uint8, device="cuda"),
                 cmb=torch.zeros(32 * nodes.size, dtype=torch.uint8, device="cuda"))
    elif kind == "ntt":
        n, b = 1 << case["log_n"], case["batch"]
        m = n >> case["pad"]
        out = lambda k: torch.empty(2 * b * k, dtype=torch.int64, device="cuda")
        s.update(n=n, m=m, batch=b, coef=_field(g, b * m), evals=_field(g, b * n), fwd=out(n), inv=out(n))
    elif kind == "rs":
        lg = case["log_len"]
        # the first witness has 2^(log_len - 1) points a slice; steps down to four points
        log_m = lg - 1
        s.update(log_m=log_m, src=_field(g, 1 << lg),
                 l_eval=torch.empty(2 << (lg + 5), dtype=torch.int64, device="cuda"),
                 tree=torch.zeros(32 << (lg - 1), dtype=torch.uint8, device="cuda"),
                 steps=[(m, torch.empty(2 * 64 << (m - 1), dtype=torch.int64, device="cuda"),
                         torch.zeros(32 << (m - 1), dtype=torch.uint8, device="cuda"), _host_field(rng, 2))
                        for m in range(log_m, 1, -1)])
    elif kind == "virgo":
        lg, lu = case["length_g"], case["length_u"]
        n_g, n_u = 1 << lg, 1 << lu
        ty = np.ascontiguousarray(rng.choice([0, 1, 6, 7, 8, 10], size=n_g).astype(np.int32))
        u = rng.integers(0, n_u, size=n_g, dtype=np.int64)
        v = rng.integers(0, n_u, size=n_g, dtype=np.int64)
        p = lambda a: ctypes.c_void_p(a.ctypes.data)
        h = lib.tp_virgo_layer_create(lg, lu, p(ty), p(u), p(v), None, None, None)
        if not h:
            native.check(lib, -1, "tp_virgo_layer_create")
        tables = lambda: [torch.empty(4 * n_u, dtype=torch.int64, device="cuda") for _ in range(3)]
        s.update(layer=_Layer(lib, h), values=_field(g, n_u), r0=_host_field(rng, lg, 2), r1=_host_field(rng, lg, 2),
                 ab=_host_field(rng, 2, 2), r=_host_field(rng, 2 * lu + 1, 2), even=tables(), odd=tables(),
                 polys=torch.empty(2 * lu * 6, dtype=torch.int64, device="cuda"),
                 left=torch.empty(2 * 3 * 4, dtype=torch.int64, device="cuda"))
    elif kind == "session":
        gt, i0, i1, _, idx, val = _circuit(case["circuit"])
        L = _layout(case)
        C, W = L.padded_copies, L.n_wires
        x = np.zeros((C, W), np.uint64)
        x[:L.copies, :L.copy_size] = rng.integers(0, 256, size=(L.copies, L.copy_size), dtype=np.uint64)
        if idx >= 0:
            x[:L.copies, idx] = val
        s.update(gates=(gt, i0, i1), C=C, W=W, nb=L.n_copy_bits, z1=_host_field(rng, 2, gt.size),
                 re=np.ascontiguousarray(x.T).reshape(-1), im=np.zeros(C * W, np.uint64), inputs=x.reshape(-1),
                 z2=_host_field(rng, 2, L.n_copy_bits), pt=_host_field(rng, 2, L.n_in_bits + L.n_copy_bits),
                 ch=_host_field(rng, L.n_copy_bits, 2))
    else:
        gt, i0, i1 = _circuit(case["circuit"])[:3]
        L, B = _layout(case), case["frames"]
        count = correlations_needed(L, True)
        s.update(layout=L, gates=(gt, i0, i1), pix=[_frame(g, L) for _ in range(B)],
                 seeds=[int(x) for x in rng.integers(0, 1 << 63, size=B)], pids=[1000 + f for f in range(B)],
                 cor=[(_host_field(rng, count, 2), _host_field(rng, count, 2)) for _ in range(B)],
                 committer=FrameCommitter([L] * B, zk=True))
    return s


class _Layer:
    """a Virgo layer handle that its program gives back"""

    def __init__(self, lib, handle):
        self.lib, self.handle = lib, handle

    def __del__(self):
        self.lib.tp_virgo_layer_destroy(self.handle)


# ---- one pass -------------------------------------------------------------------

def _run_gkr_frame(s):
    p = s["prover"]
    p.prove(s["pix"], s["z1"], s["z2"], s["pt"], s["ch"])
    return p.claims, p.wires, p.mle


def _run_gkr_batch(s):
    p, stream = s["prover"], s["stream"]
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):     # every pass starts from the transcripts the IO prefix left
        s["fs"].copy_(s["fs0"])
        s["vole"]["states"].copy_(s["vs0"])
        p.prove(s["pix"], s["z1"], s["z2"], s["pt"], None, transcripts=s["fs"], vole=s["vole"], graph=True)
        p.prove_late(s["z1"], transcripts=s["fs"], vole=s["vole"], zk=s["case"]["zk"])
    torch.cuda.current_stream().wait_stream(stream)
    return (p.claims, p.device_challenges, p.device_proof, p.wires, p.fin_beta, p.mle, p.late_coefs, p.line,
            p.late_challenges, p.late_proof, p.closing, p.input_point, p.input_tag, s["fs"], s["vole"]["states"])


def _run_gkr_mixed(s):
    p = s["prover"]
    p.prove(s["pix"], s["z1"], s["z2"], s["pt"], s["ch"])
    return p.claims, p.wires, p.fin_beta, p.mle


def _run_commit(s):
    c = s["committer"]
    c.commit(s["pix"], mask_seeds=s["seeds"])
    return c.rows, c.trees, c.mask_rows, c.mask_trees


def _run_opening(s):
    lib, st = s["lib"], torch.cuda.current_stream().cuda_stream
    p = lambda k: s[k].data_ptr()
    native.check(lib, lib.tp_orion_combine_dev(p("rows"), s["N"], p("r0"), p("comb"), p("ctree"), st), "combine")
    native.check(lib, lib.tp_orion_answer_dev(p("comb"), s["N"] // 128, p("r1"), p("ans"), st), "answer")
    native.check(lib, lib.tp_orion_query_columns_async_dev(p("rows"), s["N"], p("q"), s["q"].numel(), p("cols"), None,
                                                           st), "query columns")
    for tree, out in (("tree", "com"), ("ctree", "cmb")):
        native.check(lib, lib.tp_orion_gather_nodes_dev(p(tree), 2 * s["leaves"], p("idx"), s["n_nodes"], p(out), st),
                     "gather nodes")
    return s["comb"], s["ctree"], s["ans"], s["cols"], s["com"], s["cmb"]


def _run_ntt(s):
    lib, st, n, m, b = s["lib"], torch.cuda.current_stream().cuda_stream, s["n"], s["m"], s["batch"]
    native.check(lib, lib.tp_fft_dev(s["coef"].data_ptr(), m, n, s["fwd"].data_ptr(), b, m, n, st), "fft")
    native.check(lib, lib.tp_ifft_dev(s["evals"].data_ptr(), n, n, s["inv"].data_ptr(), b, n, n, st), "ifft")
    return s["fwd"], s["inv"]


def _run_rs(s):
    lib, st = s["lib"], torch.cuda.current_stream().cuda_stream
    native.check(lib, lib.tp_rs_commit_dev(s["src"].data_ptr(), s["case"]["log_len"], s["l_eval"].data_ptr(),
                                           s["tree"].data_ptr(), st), "rs commit")
    # slice-major codeword -> the witness layout of the FRI steps
    half = 1 << (s["log_m"] - 1)
    w = s["l_eval"].view(64, 2, half, 2).permute(2, 0, 1, 3).contiguous()
    out = [s["l_eval"], s["tree"]]
    for m, nxt, tree, r in s["steps"]:
        native.check(lib, lib.tp_fri_commit_step_dev(w.data_ptr(), m, int(r[0]), int(r[1]), nxt.data_ptr(),
                                                     tree.data_ptr(), st), "fri step")
        out += [nxt, tree]
        w = nxt
    return out


def _run_virgo(s):
    lib, st, lu = s["lib"], torch.cuda.current_stream().cuda_stream, s["case"]["length_u"]
    p = lambda a: ctypes.c_void_p(a.ctypes.data)
    polys, left = s["polys"].view(2, lu, 6), s["left"].view(2, 3, 4)
    ab, r = s["ab"], s["r"]
    alpha, beta = ab[0].copy(), ab[1].copy()
    for phase in range(2):
        src, dst = s["even"], s["odd"]
        if phase == 0:
            rc = lib.tp_virgo_phase1_init_dev(s["layer"].handle, s["values"].data_ptr(), p(s["r0"]), p(s["r1"]),
                                              p(alpha), p(beta), *[t.data_ptr() for t in src], st)
        else:
            prev, r_u = r[lu].copy(), np.ascontiguousarray(r[:lu])
            rc = lib.tp_virgo_phase2_init_dev(s["layer"].handle, s["values"].data_ptr(), p(s["r0"]), p(s["r1"]),
                                              p(alpha), p(beta), left[0, 0].data_ptr(), p(prev), p(r_u),
                                              *[t.data_ptr() for t in src], st)
        native.check(lib, rc, "virgo init")
        for k in range(lu):
            n, c = 1 << (lu - k), r[lu * phase + k]
            native.check(lib, lib.tp_virgo_sumcheck_update_dev(
                src[0].data_ptr(), src[1].data_ptr(), src[2].data_ptr(), n, int(c[0]), int(c[1]), int(k > 0),
                dst[0].data_ptr(), dst[1].data_ptr(), dst[2].data_ptr(), polys[phase, k].data_ptr(), st), "round")
            src, dst = dst, src
        for t in range(3):
            left[phase, t].copy_(src[t][:4])
    return s["polys"], s["left"]


def _run_session(s):
    lib, (gt, i0, i1), C, W, nb = s["lib"], s["gates"], s["C"], s["W"], s["nb"]
    U, I = ctypes.POINTER(ctypes.c_uint64), ctypes.POINTER(ctypes.c_int)
    u = lambda a: a.ctypes.data_as(U)
    i = lambda a: a.ctypes.data_as(I)
    br, bi = np.empty(C, np.uint64), np.empty(C, np.uint64)
    z2, z1, pt = s["z2"], s["z1"], s["pt"]
    lib.native_fp2_compute_beta(u(z2[0]), u(z2[1]), nb, 1, 0, u(br), u(bi))
    h = lib.native_fp2_early_create(gt.size, i(gt), i(i0), i(i1), u(z1[0]), u(z1[1]), C, W, u(s["re"]), u(s["im"]),
                                    u(br), u(bi))
    if not h:
        native.check(lib, -1, "early_create")
    claims = np.empty((nb, 8), np.uint64)
    wr, wi, b = np.empty(W, np.uint64), np.empty(W, np.uint64), np.empty(2, np.uint64)
    try:
        for k in range(nb):
            native.check(lib, lib.native_fp2_early_claim(h, u(claims[k])), "claim")
            native.check(lib, lib.native_fp2_early_fold(h, int(s["ch"][k, 0]), int(s["ch"][k, 1])), "fold")
        native.check(lib, lib.native_fp2_early_finish(h, u(wr), u(wi), u(b), u(b[1:])), "finish")
    finally:
        lib.native_fp2_early_destroy(h)
    m = np.empty(2, np.uint64)
    lib.native_fp2_mle_eval_base(u(s["inputs"]), u(pt[0]), u(pt[1]), pt.shape[1], u(m), u(m[1:]))
    native.check(lib, None, "session")
    as_i64 = lambda a: a.view(np.int64)
    return as_i64(br), as_i64(bi), as_i64(claims), as_i64(wr), as_i64(wi), as_i64(b), as_i64(m)


def _opening_room(lib, L):
    """bytes of an opening file with a whole Merkle path per queried column"""
    N, q = L.padded_copies * L.n_wires, query_count()
    nodes = q * lib.tp_orion_tree_leaves(N).bit_length()
    return lib.tp_orion_opening_file_size(N // 128, lib.tp_orion_codeword_len(N // 128), q, nodes, nodes)


def _run_prove(s):
    c, L, (gt, i0, i1) = s["committer"], s["layout"], s["gates"]
    c.commit(s["pix"], mask_seeds=s["seeds"])
    proofs = prove_frames(s["pix"], L, gt, i0, i1, s["pids"], s["cor"], manifests_of(c), zk=True)
    out = []
    for f, t in enumerate(proofs):
        pt = [(int(x.real), int(x.imag)) for x in t.final_input_point]
        out.append(np.frombuffer(t.fs.state(), np.uint8))
        out.append(np.array(pt, np.uint64).view(np.int64))
        for which in ("masked", "mask"):     # a file's length depends on the drawn columns: zeros behind it
            file = opening_proof(c, f, pt, which)
            whole = np.zeros(_opening_room(s["lib"], L), np.uint8)
            whole[:len(file)] = np.frombuffer(file, np.uint8)
            out.append(whole)
    return out


_RUN = dict(gkr_frame=_run_gkr_frame, gkr_batch=_run_gkr_batch, gkr_mixed=_run_gkr_mixed, commit=_run_commit,
            opening=_run_opening, ntt=_run_ntt, rs=_run_rs, virgo=_run_virgo, session=_run_session, prove=_run_prove)


def run(state):
    return _RUN[state["case"]["kind"]](state)


# ---- the work a pass cannot do without ---------------------------------------------

def _codeword(col_len):
    """codeword length of one column (levels of 0.238, rate 1.72)"""
    if col_len <= 13:
        return col_len
    inner = _codeword(int(0.238 * col_len))
    return col_len + inner + int(col_len * (1.72 - 1) - inner)


def _commit_bytes(L):
    """a frame's bytes in, codeword and tree out"""
    N = L.padded_copies * L.n_wires
    leaves = 1 << max(0, (2 * N // 128 - 1).bit_length())
    return L.copies * L.copy_size + 128 * _codeword(N // 128) * 16 + 64 * leaves


def _codeword_multiplies(L):
    """base-field multiplications of the expander graphs (ten or twenty edges a
    source, three each) over 128 columns"""
    n, total = L.padded_copies * L.n_wires // 128, 0
    while n > 13:
        total += 10 * n + 20 * _codeword(int(0.238 * n))
        n = int(0.238 * n)
    return 2 * 3 * 128 * total


def work(case):
    """bytes: inputs once, outputs once; flops: two per base-field multiply-add of
    the sums, hashes not counted"""
    kind = case["kind"]
    if kind in ("gkr_frame", "session"):
        L = _layout(case)
        C, W = L.padded_copies, L.n_wires
        src = 24 * C * W if kind == "session" else L.copies * L.copy_size
        return {"bytes": src + 16 * (C + W) + 64 * L.n_copy_bits, "flops": 2 * 3 * 2 * C * L.copy_size}
    if kind == "gkr_batch":
        L, B = _layout(case), case["frames"]
        return {"bytes": B * (L.copies * L.copy_size + 16 * L.n_wires),
                "flops": B * 2 * 3 * 2 * L.padded_copies * L.copy_size}
    if kind == "gkr_mixed":
        B = case["frames"]
        px = [max(16, int(case["height"] * a)) * max(16, int(case["width"] * b)) * 3
              for a, b in np.random.default_rng(B).uniform(0.22, 1.0, size=(B, 2))]
        return {"bytes": sum(px) + B * 16 * 512, "flops": 2 * 3 * 2 * sum(px)}
    if kind == "commit":
        L, k = _layout(case), case["frames"] * (2 if case["zk"] else 1)
        return {"bytes": k * _commit_bytes(L), "flops": k * _codeword_multiplies(L)}
    if kind == "opening":
        L = _layout(case)
        N = L.padded_copies * L.n_wires
        cw = _codeword(N // 128)
        leaves = 1 << max(0, (2 * N // 128 - 1).bit_length())
        return {"bytes": 128 * cw * 16 + 16 * cw + 64 * leaves + 16 * N // 128 + 2 * 1222 * 2048,
                "flops": 2 * 3 * 128 * cw}
    if kind == "ntt":
        n, b, lg = 1 << case["log_n"], case["batch"], case["log_n"]
        return {"bytes": b * 16 * ((n >> case["pad"]) + 3 * n), "flops": 2 * b * 2 * 3 * (n // 2) * lg}
    if kind == "rs":
        lg = case["log_len"]
        n = 1 << (lg + 5)
        return {"bytes": 16 * ((1 << lg) + n + n) + 32 * (2 << (lg - 1)), "flops": 2 * 3 * (n // 2) * (lg - 1)}
    if kind == "virgo":
        n_g, n_u = 1 << case["length_g"], 1 << case["length_u"]
        return {"bytes": 20 * n_g + 16 * n_u, "flops": 2 * 2 * 3 * 9 * n_u}
    L, B = _layout(case), case["frames"]
    return {"bytes": B * 2 * _commit_bytes(L), "flops": B * 2 * _codeword_multiplies(L)}


def exact(case, seed):
    """every output is a whole number (field elements, digests, file bytes)"""
    return None
