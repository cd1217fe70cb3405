// Late rounds of the GKR input layer's sumcheck and the line projection that
// ends it, one frame per CTA (TruePix-main/libTruePix/layerprover.py:231-290,
// gateprover.py:105-185, layercompute.py:16-247).
//
// After the early rounds every wire w holds one value V[w] (the input table at
// the copy point) and beta one value; gate g carries a weight A_g (its z1 eq
// value). Rounds 0..n-1 bind the bits of in0 (LSB first), rounds n..2n-1 the
// bits of in1. In round j of a phase, with T the table V folded by that phase's
// earlier challenges and b the gate's input bit j:
//   x / y      the gate's input values: in phase 1 x = T[in0 >> j] and
//              y = V[in1]; in phase 2 x = V(w1) (phase 1's last value) and
//              y = T[in1 >> j]
//   at 0 or 1  A_g * gate(x, y) added to the value at b
//   at -1      gate(x', y') * (b ? -A_g : 2 A_g), the bound input taken at -1
//              along bit j: 2 T[2k] - T[2k + 1], k = in >> (j + 1)
// summed over gates, times beta, interpolated at 0, 1, -1 (util.py:91-113);
// then the challenge r folds T (T'[k] = T[2k] + r (T[2k+1] - T[2k])) and
// A_g *= (b ? r : 1 - r). Phase 2 starts again from V. The line projection: the
// input values on the line w1 + t (w2 - w1), t = 0..n (t = 0, 1 are the two
// phases' last values, the others multilinear evaluations of V), and the
// coefficients of the degree-n polynomial through them.
//
// The CTA's work is written as steps between barriers, each step a function of
// (workspace, thread index) in which a thread reads only what earlier steps
// wrote and writes only its own slots: the device runs them with __syncthreads()
// between, a host loop over the thread indices runs the same code.
#pragma once
#include <stdint.h>

#include "fp2.cuh"
#include "transcript.cuh"
#include "vole.cuh"

namespace tp {
namespace late {

constexpr int kThreads = 256;
constexpr int kMaxInBits = 9;
constexpr int kMaxWires = 1 << kMaxInBits;
constexpr int kMaxGates = 768;

// packed gate table: type << 28 | in0 << 14 | in1
struct Gates {
    uint32_t g[kMaxGates];
};

// native_fp2_core.hpp:32-51 on canonical Fp2 values
TP_HD fp2 gatefn(unsigned t, fp2 x, fp2 y)
{
    const fp2 one = mk(1, 0);
    switch (t) {
    case 0: return f2mul(x, y);
    case 1: return f2add(x, y);
    case 2: return f2sub(x, y);
    case 3: return x;
    case 4: return y;
    case 5: return f2sub(f2add(x, y), f2mul(x, y));
    case 6: return f2sub(f2add(x, y), f2dbl(f2mul(x, y)));
    case 7: return f2sub(one, x);
    case 8: return f2sub(one, f2mul(x, y));
    case 9: return f2sub(f2add(one, f2mul(x, y)), f2add(x, y));
    case 10: return f2sub(f2add(one, f2dbl(f2mul(x, y))), f2add(x, y));
    case 11: return f2mul(f2sub(one, x), y);
    default: return x;
    }
}

// gateprover_vole.py p_com_gatefn_ (GateFunctionsPC, :706-720): a gate's value on
// committed x, y and x*y, by the native type index
TP_HD fp2 pc_gatefn(unsigned t, fp2 x, fp2 y, fp2 xy)
{
    const fp2 one = mk(1, 0);
    switch (t) {
    case 0: return xy;
    case 1: return f2add(x, y);
    case 2: return f2sub(x, y);
    case 3: return x;
    case 4: return y;
    case 5: return f2sub(f2add(x, y), xy);
    case 6: return f2sub(f2add(x, y), f2dbl(xy));
    case 7: return f2sub(one, x);
    case 8: return f2sub(one, xy);
    case 9: return f2sub(f2add(one, xy), f2add(x, y));
    case 10: return f2sub(f2add(one, f2dbl(xy)), f2add(x, y));
    case 11: return f2sub(y, xy);
    default: return x;
    }
}

// one frame's inputs and outputs (pointers already at the frame)
struct Frame {
    const fp2* wires;      // 2^n
    const fp2* beta;       // 1
    const fp2* zg;         // n_gates
    const fp2* chal;       // 2n given challenges, or null: drawn by the VOLE rounds
    fs::State* st;         // VOLE mode: the frame's transcript,
    vole::State* vs;       // its VOLE state,
    const fp2* u;          // and correlations (count each)
    const fp2* v;
    fp2* coefs;            // 2n x 3
    fp2* h;                // n + 1
    fp2* chal_out;         // 2n
    fp2* proof;            // VOLE mode, optional: 2n x 4 (three d, the equality value)
    // the layer's closing proofs (VOLE mode, optional)
    const fp2* z2;         // nb: the copy part of the layer's point
    const fp2* w3;         // the early challenges: w3[k * w3_stride], k < nb
    long long w3_stride;
    fp2* closing;          // n + 10 (zero-knowledge prover: n + 15) values in the order they are put
    fp2* point;            // n + nb: the input point
    fp2* tag;              // 1: its tag
};

struct Shape {
    int n;           // input bits
    int n_gates;
    long long count; // correlations per frame
    int layer;       // labels "sc-<layer>-<round0 + round>"
    int round0;      // the early rounds before (their count: nb)
    int zk;          // closing proofs of the zero-knowledge prover (circuitnizkvec_vole_ZK.py)
};

// the CTA's workspace (shared memory on the device)
struct Work {
    fp2 V[kMaxWires];
    fp2 T[kMaxWires];
    fp2 Tn[kMaxWires / 2];
    fp2 A[kMaxGates];
    union {                    // the sums' slots; a step that hashes has read them before
        fp2 red[3][kThreads];
        fs::TxMem tx;
    };
    fp2 w[2 * kMaxInBits];     // the challenges
    fp2 h[kMaxInBits + 1];     // the line's values
    fp2 hc[kMaxInBits + 1];    // its coefficients
    fp2 vv[kMaxInBits + 1];    // closing: the coefficients' tags
    fp2 pr[3];                 // closing: tags of x, of the line's sum, of the product
    fp2 beta, v1, r;
    fs::State st;
    vole::State vs;
    int bad;
};

static_assert(sizeof(Work) <= 48 * 1024, "the workspace fits the static shared memory of a CTA");

// ---- steps -------------------------------------------------------------------

TP_HD void step_load(Work& w, const Frame& f, const Shape& sh, int tid)
{
    const int W = 1 << sh.n;
    for (int k = tid; k < W; k += kThreads) w.V[k] = w.T[k] = f.wires[k];
    for (int g = tid; g < sh.n_gates; g += kThreads) w.A[g] = f.zg[g];
    if (tid == 0) {
        w.beta = *f.beta;
        w.bad = 0;
        if (!f.chal) {
            w.st = *f.st;
            w.vs = *f.vs;
        }
    }
}

// per-thread partial values at 0, 1, -1 of round rd
TP_HD void step_sums(Work& w, const uint32_t* gates, const Shape& sh, int rd, int tid)
{
    const bool ph1 = rd < sh.n;
    const int j = ph1 ? rd : rd - sh.n;
    fp2 s0 = f2zero(), s1 = f2zero(), s2 = f2zero();
    for (int g = tid; g < sh.n_gates; g += kThreads) {
        const uint32_t t = gates[g];
        const unsigned type = t >> 28;
        const int in0 = (int)((t >> 14) & 0x3FFFu), in1 = (int)(t & 0x3FFFu);
        const int idx = ph1 ? in0 : in1;
        const int bit = (idx >> j) & 1, k = idx >> (j + 1);
        const fp2 t0 = w.T[2 * k], t1 = w.T[2 * k + 1];
        const fp2 cur = bit ? t1 : t0, m1 = f2at_m1(t0, t1);
        fp2 v01, two;
        if (ph1) {
            const fp2 y = w.V[in1];
            v01 = gatefn(type, cur, y);
            two = gatefn(type, m1, y);
        } else {
            v01 = gatefn(type, w.v1, cur);
            two = gatefn(type, w.v1, m1);
        }
        const fp2 a = w.A[g];
        v01 = f2mul(a, v01);
        s2 = f2add(s2, f2mul(two, bit ? f2sub(f2zero(), a) : f2dbl(a)));
        if (bit)
            s1 = f2add(s1, v01);
        else
            s0 = f2add(s0, v01);
    }
    w.red[0][tid] = s0;
    w.red[1][tid] = s1;
    w.red[2][tid] = s2;
}

// one level of the sum over the threads' slots: threads below `left` add the three
// slots left, 2 left and 3 left above theirs (256 slots in four steps)
TP_HD void step_reduce(Work& w, int left, int tid)
{
    if (tid < left)
        for (int q = 0; q < 3; ++q) {
            fp2* r = w.red[q] + tid;
            r[0] = f2add(f2add(r[0], r[left]), f2add(r[2 * left], r[3 * left]));
        }
}

// The steps run by `par.one`: one warp on the device (one call on the host). Its
// lanes do the same work, with the transcript in a Writer (transcript.cuh) and each
// on a copy of its own of the VOLE state, and lane 0 writes. Reads of the workspace
// that the writes below them would change come before the synchronisation in front
// of these.
TP_HD void warp_sync()
{
#ifdef __CUDA_ARCH__
    __syncwarp();
#endif
}

// the round's coefficients and its challenge
#pragma nv_exec_check_disable
TP_HD void step_head(Work& w, const Frame& f, const Shape& sh, int rd)
{
    fp2 c[3];
    vole::interpolate_quadratic(f2mul(w.red[0][0], w.beta), f2mul(w.red[1][0], w.beta),
                                f2mul(w.red[2][0], w.beta), c);
    fp2 r;
    if (f.chal) {
        r = f.chal[rd];
    } else {
        vole::State vs = w.vs;
        fs::Writer st(w.st, &w.tx);
        const fs::Label label = vole::sc_label(sh.layer, sh.round0 + rd);
        const bool ok = vole::round(st, vs, c, 3, f.u, f.v, sh.count, label, f.proof ? f.proof + 4 * rd : nullptr, &r);
        warp_sync();
        st.store(w.st);
        if (fs::lead()) {
            w.vs = vs;
            if (!ok) w.bad = 1;
        }
    }
    if (fs::lead()) {
        for (int q = 0; q < 3; ++q) f.coefs[3 * rd + q] = c[q];
        w.r = r;
        w.w[rd] = r;
        f.chal_out[rd] = r;
    }
}

// fold T by the challenge into Tn, update the gates' weights
TP_HD void step_fold(Work& w, const uint32_t* gates, const Shape& sh, int rd, int tid)
{
    const bool ph1 = rd < sh.n;
    const int j = ph1 ? rd : rd - sh.n;
    const int half = (1 << sh.n) >> (j + 1);
    const fp2 r = w.r, one_m_r = f2sub(mk(1, 0), r);
    for (int k = tid; k < half; k += kThreads) w.Tn[k] = f2fold(w.T[2 * k], w.T[2 * k + 1], r);
    for (int g = tid; g < sh.n_gates; g += kThreads) {
        const uint32_t t = gates[g];
        const int idx = ph1 ? (int)((t >> 14) & 0x3FFFu) : (int)(t & 0x3FFFu);
        w.A[g] = f2mul(w.A[g], ((idx >> j) & 1) ? r : one_m_r);
    }
}

TP_HD void step_copy(Work& w, int n_entries, int tid)
{
    for (int k = tid; k < n_entries; k += kThreads) w.T[k] = w.Tn[k];
}

TP_HD void step_restart(Work& w, const Shape& sh, int tid)
{
    for (int k = tid; k < (1 << sh.n); k += kThreads) w.T[k] = w.V[k];
}

// ---- the line projection: V at the points w1 + t (w2 - w1), t = 2..n, as sums over
// the wires of eq(point, k) V[k], all points at once (one warp's worth of threads
// each); eq from two half tables. T and Tn are free by then.

TP_HD int line_low_bits(const Shape& sh) { return sh.n >> 1; }
TP_HD int line_table(const Shape& sh) { return (1 << line_low_bits(sh)) + (1 << (sh.n - line_low_bits(sh))); }

// the points' coordinates, Tn[(t - 2) n + j]
TP_HD void step_line_points(Work& w, const Shape& sh, int tid)
{
    const int n = sh.n;
    if (tid >= (n - 1) * n) return;
    const int t = 2 + tid / n, j = tid % n;
    w.Tn[tid] = f2add(w.w[j], f2scale(f2sub(w.w[n + j], w.w[j]), (u64)t));
}

// the half tables of eq, T[(t - 2) table + entry]: the low half first
TP_HD void step_line_eq(Work& w, const Shape& sh, int tid)
{
    const int n = sh.n, n1 = line_low_bits(sh), lo = 1 << n1, table = line_table(sh);
    const fp2 one = mk(1, 0);
    for (int e = tid; e < (n - 1) * table; e += kThreads) {
        const int q = e / table, i = e % table;
        const int first = i < lo ? 0 : n1, last = i < lo ? n1 : n, k = i < lo ? i : i - lo;
        fp2 v = one;
        for (int j = first; j < last; ++j) {
            const fp2 p = w.Tn[q * n + j];
            v = f2mul(v, ((k >> (j - first)) & 1) ? p : f2sub(one, p));
        }
        w.T[e] = v;
    }
}

// partial sums of point t = 2 + tid / 32
TP_HD void step_line_sums(Work& w, const Shape& sh, int tid)
{
    const int q = tid >> 5, n1 = line_low_bits(sh);
    fp2 s = f2zero();
    if (q < sh.n - 1) {
        const fp2* lo = w.T + q * line_table(sh);
        const fp2* hi = lo + (1 << n1);
        for (int k = tid & 31; k < (1 << sh.n); k += 32)
            s = f2add(s, f2mul(f2mul(lo[k & ((1 << n1) - 1)], hi[k >> n1]), w.V[k]));
    }
    w.red[0][tid] = s;
}

// one level of the sums within each 32 slots (32 -> 8 -> 2 -> 1)
TP_HD void step_line_reduce(Work& w, int left, int tid)
{
    if ((tid & 31) >= left) return;
    fp2* r = w.red[0] + tid;
    r[0] = left > 1 ? f2add(f2add(r[0], r[left]), f2add(r[2 * left], r[3 * left])) : f2add(r[0], r[1]);
}

TP_HD void step_line_values(Work& w, const Shape& sh, int tid)
{
    if (tid < sh.n - 1) w.h[2 + tid] = w.red[0][32 * tid];
}

// The coefficients of the polynomial of degree n through (t, h[t]), t = 0..n, are a
// fixed matrix times the values: row k, column t is the coefficient of x^k in the
// t-th Lagrange polynomial on the nodes 0..n. The matrices for n <= kMaxInBits are
// made at compile time.
constexpr u64 mul_c(u64 a, u64 b)   // canonical a, b -> a b mod p (compile time)
{
    const u64 a0 = a & 0xFFFFFFFFull, a1 = a >> 32, b0 = b & 0xFFFFFFFFull, b1 = b >> 32;
    const u64 lo = a0 * b0, mid = a0 * b1 + a1 * b0, hi = a1 * b1;
    u64 s = (lo & P61) + (lo >> 61) + (hi << 3) + (mid >> 29) + ((mid & 0x1FFFFFFFull) << 32);
    s = (s & P61) + (s >> 61);
    return s >= P61 ? s - P61 : s;
}
constexpr u64 neg_c(u64 a) { return a ? P61 - a : 0; }
// 1 / k mod p for 1 <= k <= 9: (m p + 1) / k for the m that makes it whole
constexpr u64 inv_c(u64 k)
{
    for (u64 m = 0; m < k; ++m)
        if ((m * P61 + 1) % k == 0) return (m * P61 + 1) / k;
    return 0;
}
struct LineMatrix {
    u64 m[kMaxInBits + 1][kMaxInBits + 1][kMaxInBits + 1];   // [n][k][t]
};
constexpr LineMatrix make_line_matrix()
{
    LineMatrix L{};
    for (int n = 1; n <= kMaxInBits; ++n)
        for (int t = 0; t <= n; ++t) {
            u64 c[kMaxInBits + 2] = {1};   // the product of (x - i) / (t - i) over i != t
            int deg = 0;
            for (int i = 0; i <= n; ++i) {
                if (i == t) continue;
                const u64 inv = t > i ? inv_c((u64)(t - i)) : neg_c(inv_c((u64)(i - t)));
                for (int k = deg + 1; k >= 0; --k) {
                    const u64 up = k > 0 ? c[k - 1] : 0, here = k <= deg ? neg_c(mul_c(c[k], (u64)i)) : 0;
                    const u64 sum = up + here >= P61 ? up + here - P61 : up + here;
                    c[k] = mul_c(sum, inv);
                }
                ++deg;
            }
            for (int k = 0; k <= n; ++k) L.m[n][k][t] = c[k];
        }
    return L;
}
#ifdef __CUDACC__
static __constant__ LineMatrix kLineMatrixDev = make_line_matrix();
#endif
inline u64 line_entry_host(int n, int k, int t)
{
    static constexpr LineMatrix L = make_line_matrix();
    return L.m[n][k][t];
}

// thread k: coefficient k (constant first) of the polynomial through (t, h[t])
#pragma nv_exec_check_disable
TP_HD void step_interpolate(Work& w, const Frame& f, const Shape& sh, int tid)
{
    if (tid > sh.n) return;
    fp2 c = f2zero();
    for (int t = 0; t <= sh.n; ++t) {
#ifdef __CUDA_ARCH__
        const u64 m = kLineMatrixDev.m[sh.n][tid][t];
#else
        const u64 m = line_entry_host(sh.n, tid, t);
#endif
        c = f2add(c, f2scale(w.h[t], m));
    }
    f.h[tid] = w.hc[tid] = c;
}

// ---- the layer's closing proofs (circuitnizkvec_vole.py:433-500, one layer) ----

// index of the equality value among the closing values (before it: two
// commitments, n commitments, two proof-of-knowledge values, with zk three mask
// commitments, the product proof's two values and with zk the masks' two)
TP_HD int close_eq_index(const Shape& sh) { return sh.n + 6 + 5 * (sh.zk != 0); }

// create_final_prod_pok (:175-218; the zero-knowledge prover's,
// circuitnizkvec_vole_ZK.py:188-247, adds three mask commitments of 1 and their
// product proof) on the line's coefficients
#pragma nv_exec_check_disable
TP_HD void step_close_commit(Work& w, const Frame& f, const Shape& sh)
{
    const int n = sh.n;
    const int zk = sh.zk != 0;
    vole::State vs = w.vs;
    if (vs.bad || vs.idx + (unsigned long long)(n + 2 + 3 * zk) > (unsigned long long)sh.count) {
        warp_sync();
        if (fs::lead()) {
            w.vs.bad = 1;
            w.bad = 1;
        }
        return;
    }
    fs::Writer st(w.st, &w.tx);
    fp2* out = f.closing;
    auto put = [&](fp2 v) {   // the next closing value: written out and put
        st.put_fp2(v.re, v.im);
        if (fs::lead()) *out = v;
        ++out;
    };
    fp2 sval = f2zero();
    for (int k = 0; k <= n; ++k) sval = f2add(sval, w.hc[k]);
    const fp2 prod = f2mul(w.hc[0], sval);
    fp2 v1, v3, vv[kMaxInBits + 1], mtag[3];
    const fp2 d0 = vole::commit(vs, w.hc[0], f.u, f.v, &v1);
    const fp2 d1 = vole::commit(vs, prod, f.u, f.v, &v3);
    put(d0);
    put(d1);
    fp2 rest_sum = f2zero(), rest_v = f2zero();
    vv[0] = v1;
    for (int k = 1; k <= n; ++k) {
        put(vole::commit(vs, w.hc[k], f.u, f.v, &vv[k]));
        rest_sum = f2add(rest_sum, w.hc[k]);
        rest_v = f2add(rest_v, vv[k]);
    }
    const fp2 c = st.rand_fp2(fs::label_lit("pok-vec"));
    put(f2mul(rest_sum, c));
    put(f2mul(rest_v, c));
    if (zk)
        for (int q = 0; q < 3; ++q) put(vole::commit(vs, mk(1, 0), f.u, f.v, &mtag[q]));
    const fp2 vsum = f2add(v1, rest_v);
    // prod_finish on (x, sum, x * sum) with tags (v1, sum of tags, v3)
    put(f2mul(v1, vsum));
    put(f2sub(f2add(f2mul(w.hc[0], vsum), f2mul(sval, v1)), v3));
    if (zk) {   // prod_finish on (1, 1, 1) with the masks' tags
        put(f2mul(mtag[0], mtag[1]));
        put(f2sub(f2add(mtag[1], mtag[0]), mtag[2]));
    }
    warp_sync();
    st.store(w.st);
    if (!fs::lead()) return;
    for (int k = 0; k <= n; ++k) w.vv[k] = vv[k];
    w.pr[0] = v1;
    w.pr[1] = vsum;
    w.pr[2] = v3;
    w.vs = vs;
}

// per-thread partial sums of the wiring predicates' multilinear extensions times
// the committed gate values (CircuitVerifier.eval_mlext, circuitverifier.py:224-290,
// with GateFunctionsPC): sum over gates of z1eq_g * eq(w1, in0_g) * eq(w2, in1_g)
// * pc_gate(v1, sum, v3)
TP_HD void step_close_sums(Work& w, const Frame& f, const uint32_t* gates, const Shape& sh, int tid)
{
    const int n = sh.n;
    fp2 s = f2zero();
    const fp2 one = mk(1, 0);
    for (int g = tid; g < sh.n_gates; g += kThreads) {
        const uint32_t t = gates[g];
        const int in0 = (int)((t >> 14) & 0x3FFFu), in1 = (int)(t & 0x3FFFu);
        fp2 e = f.zg[g];
        for (int j = 0; j < n; ++j) {
            e = f2mul(e, ((in0 >> j) & 1) ? w.w[j] : f2sub(one, w.w[j]));
            e = f2mul(e, ((in1 >> j) & 1) ? w.w[n + j] : f2sub(one, w.w[n + j]));
        }
        s = f2add(s, f2mul(e, pc_gatefn(t >> 28, w.pr[0], w.pr[1], w.pr[2])));
    }
    w.red[0][tid] = s;
    w.red[1][tid] = f2zero();
    w.red[2][tid] = f2zero();
}

// per early challenge w its value (Tn) and beta's factor 2 w z + 1 - (w + z) (T); both
// tables are free by then
TP_HD void step_close_load(Work& w, const Frame& f, const Shape& sh, int tid)
{
    if (tid >= sh.round0) return;
    const fp2 wk = f.w3[tid * f.w3_stride], zk = f.z2[tid];
    w.Tn[tid] = wk;
    w.T[tid] = f2sub(f2add(f2dbl(f2mul(wk, zk)), mk(1, 0)), f2add(wk, zk));
}

// the equality proof against the last round's value, tau, the proof of knowledge
// of all round coefficients, the input point and its value proof
#pragma nv_exec_check_disable
TP_HD void step_close_tail(Work& w, const Frame& f, const Shape& sh)
{
    const int n = sh.n, nb = sh.round0;
    fp2 mz = mk(1, 0);
    for (int k = 0; k < nb; ++k) mz = f2mul(mz, w.T[k]);
    const fp2 tv = f2mul(w.red[0][0], mz);
    warp_sync();
    fs::Writer st(w.st, &w.tx);
    fp2* out = f.closing + close_eq_index(sh);
    auto put = [&](fp2 v) {
        st.put_fp2(v.re, v.im);
        if (fs::lead()) *out = v;
        ++out;
    };
    const fp2 e = st.rand_fp2(fs::label_lit("eq"));
    put(f2mul(f2sub(w.vs.prev, tv), e));
    const fp2 tau = st.rand_fp2(vole::tau_label(sh.layer));
    fp2 tag = w.vv[n];
    for (int k = n - 1; k >= 0; --k) tag = f2add(f2mul(tag, tau), w.vv[k]);
    // create_pok_final
    fp2 osum = f2zero(), vsum = f2zero();
    for (int k = 0; k < 4; ++k) {
        osum = f2add(osum, w.vs.out_elem[k]);
        vsum = f2add(vsum, w.vs.v_elem[k]);
    }
    const fp2 c = st.rand_fp2(fs::label_lit("pok-final"));
    put(f2mul(osum, c));
    put(f2mul(vsum, c));
    // put(["gkr_input_point", [[re, im], ...]]): a string, then every coordinate's two ints
    st.put_label(fs::label_lit("gkr_input_point"));
    for (int k = 0; k < n + nb; ++k) {
        const fp2 x = k < n ? f2add(w.w[k], f2mul(f2sub(w.w[n + k], w.w[k]), tau)) : w.Tn[k - n];
        if (fs::lead()) f.point[k] = x;
        st.absorb_le(0x02 | (x.re << 8), 8);
        st.absorb_le((x.re >> 56) | (0x02 << 8) | (x.im << 16), 8);
        st.absorb_le(x.im >> 48, 2);
    }
    // create_input_value_proof
    const fp2 civ = st.rand_fp2(fs::label_lit("input-val"));
    put(f2mul(tag, civ));
    warp_sync();
    st.store(w.st);
    if (!fs::lead()) return;
    w.vs.prev = tag;
    *f.tag = tag;
}

// the VOLE state and transcript back to the frame
TP_HD void step_store(Work& w, const Frame& f)
{
    if (!f.chal && fs::lead()) {
        *f.st = w.st;
        *f.vs = w.vs;
    }
}

// The whole late phase of one frame. par.all(fn) runs fn(thread index) on every
// thread of the CTA and then waits at a barrier; par.one(fn) runs fn once (on the
// device: on every lane of the first warp, see above) and waits. Every branch below depends only on values all threads read alike
// after a barrier.
#pragma nv_exec_check_disable
template <class Par>
TP_HD void run_frame(Work& w, const Frame& f, const Shape& sh, const uint32_t* gates, const Par& par)
{
    const int n = sh.n, W = 1 << n;
    par.all([&](int tid) { step_load(w, f, sh, tid); });
    for (int rd = 0; rd < 2 * n; ++rd) {
        par.all([&](int tid) { step_sums(w, gates, sh, rd, tid); });
        for (int left = kThreads / 4; left > 0; left >>= 2) par.all([&](int tid) { step_reduce(w, left, tid); });
        par.one([&] { step_head(w, f, sh, rd); });
        if (w.bad) break;
        par.all([&](int tid) { step_fold(w, gates, sh, rd, tid); });
        const int j = rd < n ? rd : rd - n;
        par.all([&](int tid) { step_copy(w, W >> (j + 1), tid); });
        if (rd == n - 1) {
            par.all([&](int tid) { if (tid == 0) w.v1 = w.h[0] = w.T[0]; });
            par.all([&](int tid) { step_restart(w, sh, tid); });
        }
        if (rd == 2 * n - 1) par.all([&](int tid) { if (tid == 0) w.h[1] = w.T[0]; });
    }
    if (!w.bad) {
        par.all([&](int tid) { step_line_points(w, sh, tid); });
        par.all([&](int tid) { step_line_eq(w, sh, tid); });
        par.all([&](int tid) { step_line_sums(w, sh, tid); });
        for (int left = 8; left > 0; left = left > 2 ? 2 : left - 1) par.all([&](int tid) { step_line_reduce(w, left, tid); });
        par.all([&](int tid) { step_line_values(w, sh, tid); });
        par.all([&](int tid) { step_interpolate(w, f, sh, tid); });
        if (f.closing) {
            par.one([&] { step_close_commit(w, f, sh); });
            if (!w.bad) {
                par.all([&](int tid) {
                    step_close_load(w, f, sh, tid);
                    step_close_sums(w, f, gates, sh, tid);
                });
                for (int left = kThreads / 4; left > 0; left >>= 2)
                    par.all([&](int tid) { step_reduce(w, left, tid); });
                par.one([&] { step_close_tail(w, f, sh); });
            }
        }
    }
    par.one([&] { step_store(w, f); });
}

}  // namespace late
}  // namespace tp
