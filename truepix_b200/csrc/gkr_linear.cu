// Early rounds of byte frames whose per-copy sums stay in vectors.
//
// A round's claim at copy c needs, besides beta, only
//   s(c) = sum_w L[w] V[w][c]                     (the layer's linear part)
//   M_g(c) = sum_{terms of group g} coef V[a][c]  and  V[b_g][c]
// per group g of product terms that share their wire b. Folding the copies by a
// challenge is linear, so these 1 + 2 G vectors fold by themselves, and the table
// of all wires is not needed until the end, where the wire values are sums over
// the copies weighted with eq(challenges, c). For the layers of TruePix's circuits
// (G = 0 for gray, inv and mask, 1 for crop) a round then moves 32 B per copy and
// vector instead of 32 B per copy and wire: over 64 1080p frames the rounds after the
// first took 2.95 ms (12.9 GB of folded tables written and read) and now 0.1 ms.
// The sums are exact field sums, so every value is the same.
//
//   forms     the vectors from the bytes: an integer matrix product
//             (copies x wires bytes) x (wires x 16 byte-planes of a form's
//             coefficients, eight for each limb) on the tensor cores, u8 x u8
//             accumulated in 32 bits (512 * 255 * 255 < 2^31), recombined mod p;
//             bound by reading the bytes. The bytes are also copied aside (rows of
//             a multiple of 32 bytes), so that the caller's buffer is free after
//             the first claim or fold as before.
//   rounds    one thread a pair of copies, one launch a round (vec_round_kernel), or
//             all rounds of a frame in one CTA once few pairs are left
//             (vec_rounds_kernel), with the challenges given or drawn by the
//             VOLE-committed round on the frame's transcript.
//   finish    the wires from the bytes: (16 byte-planes of eq) x (copies x wires) the
//             same way.
#include "gkr.h"
#include "gkr_internal.cuh"
#include "runtime.h"
#include "vole.cuh"

#include <algorithm>
#include <atomic>

namespace tp {

namespace {

constexpr int kTileRows = 64;        // copies staged at a time by the byte forms
constexpr int kFormThreads = 128;    // a warp per 16 of them
constexpr int kVecThreads = 256;
constexpr int kRoundsThreads = 512;
constexpr int kFinCopies = 512;      // copies per CTA of the finish from bytes

__device__ __forceinline__ void read_job(const Job* jobs, Job& sj)
{
    const int* src = reinterpret_cast<const int*>(jobs + blockIdx.y);
    int* dst = reinterpret_cast<int*>(&sj);
    for (int i = threadIdx.x; i < (int)(sizeof(Job) / 4); i += blockDim.x) dst[i] = __ldg(src + i);
    __syncthreads();
}

// D += A B for a 16 x 32 tile of A and a 32 x 8 tile of B, bytes: lane (g = lane / 4,
// j = lane % 4) holds A[g][4j..], A[g + 8][4j..], A[g][16 + 4j..], A[g + 8][16 + 4j..],
// B[4j..][g], B[16 + 4j..][g] and D[g][2j], D[g][2j + 1], D[g + 8][2j], D[g + 8][2j + 1]
__device__ __forceinline__ void mma_u8(int (&d)[4], u32 a0, u32 a1, u32 a2, u32 a3, u32 b0, u32 b1)
{
    asm volatile(
        "mma.sync.aligned.m16n8k32.row.col.s32.u8.u8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
        "{%0, %1, %2, %3};"
        : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ u32 smem_at(const void* p) { return (u32)__cvta_generic_to_shared(p); }

// four blocks of eight 16-byte rows, lane l's address the row l % 8 of block l / 8: lane
// (g, j) gets bytes 4j.. of row g of each
__device__ __forceinline__ void load_quarters(u32 (&v)[4], u32 at)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3])
                 : "r"(at)
                 : "memory");
}

// 4 x 4 bytes transposed: byte i of out[m] = byte m of in[i]
__device__ __forceinline__ void transpose4(const u32 (&in)[4], u32 (&out)[4])
{
    const u32 a = __byte_perm(in[0], in[1], 0x5140), b = __byte_perm(in[2], in[3], 0x5140);   // bytes 0, 1
    const u32 c = __byte_perm(in[0], in[1], 0x7362), d = __byte_perm(in[2], in[3], 0x7362);   // bytes 2, 3
    out[0] = __byte_perm(a, b, 0x5410);
    out[1] = __byte_perm(a, b, 0x7632);
    out[2] = __byte_perm(c, d, 0x5410);
    out[3] = __byte_perm(c, d, 0x7632);
}

// v 2^sh mod p (nearly) for 0 <= v < 2^36, 0 <= sh < 61
__device__ __forceinline__ u64 shift_mod(u64 v, int sh)
{
    return ((v << sh) & P61) + (sh ? v >> (61 - sh) : 0);
}

__device__ __forceinline__ void async16(void* dst, const void* src, bool in)
{
    const u32 d = (u32)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(in ? 16 : 0) : "memory");
}

// ---- forms from bytes ---------------------------------------------------------
// Dynamic shared memory: two tiles of 64 rows, then the 16 planes of one form, all
// with rows of kp + 16 bytes (kp = J.stride, the copy size rounded up to 32), so that
// the fragments' words of eight rows fall in distinct banks.

// tile t's rows into buf (asynchronously where whole 16-byte vectors can be read)
__device__ void stage_tile(const Job& J, int t, unsigned char* buf, int pitch)
{
    const int c0 = t * kTileRows;
    if (J.vec) {
        const int per = J.cs >> 4;
        for (int i = threadIdx.x; i < kTileRows * per; i += kFormThreads) {
            const int r = i / per, q = i - r * per;
            const bool in = c0 + r < J.n_real;
            async16(buf + r * pitch + 16 * q, J.pix + (size_t)(in ? c0 + r : 0) * J.cs + 16 * q, in);
        }
    } else {
        const int words = J.stride >> 2;
        for (int i = threadIdx.x; i < kTileRows * words; i += kFormThreads) {
            const int r = i / words, q = 4 * (i - r * words);
            u32 v = 0;
            if (c0 + r < J.n_real) {
                const unsigned char* p = J.pix + (size_t)(c0 + r) * J.cs;
#pragma unroll
                for (int b = 0; b < 4; ++b)
                    if (q + b < J.cs) v |= (u32)__ldg(p + q + b) << (8 * b);
            }
            *reinterpret_cast<u32*>(buf + r * pitch + q) = v;
        }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
}

__global__ void __launch_bounds__(kFormThreads) forms_bytes_kernel(const Job* __restrict__ jobs)
{
    __shared__ __align__(16) Job J;
    __shared__ fp2 s_const;    // the form's term of the constant wire
    extern __shared__ __align__(16) unsigned char dsm[];
    read_job(jobs, J);
    const int tiles = (J.n_in + kTileRows - 1) / kTileRows;
    const int t0 = blockIdx.x * J.wpg, t1 = min(tiles, t0 + J.wpg);
    if (t0 >= t1) return;
    const int kp = J.stride, pitch = kp + 16, cs = J.cs;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, j = lane & 3;
    unsigned char* tile[2] = {dsm, dsm + kTileRows * pitch};
    unsigned char* planes = dsm + 2 * kTileRows * pitch;
    if (J.vec) {   // the columns behind the copied vectors stay zero
        const int pad = (kp - cs) >> 2;
        for (int i = tid; i < 2 * kTileRows * pad; i += kFormThreads)
            *reinterpret_cast<u32*>(dsm + (i / pad) * pitch + cs + 4 * (i % pad)) = 0u;
    }
    for (int form = 0; form <= J.G; ++form) {
        stage_tile(J, t0, tile[0], pitch);
        // the form's planes: byte l of a coefficient's limbs in plane l (re), 8 + l (im)
        if (tid == 0) s_const = form == 0 && J.const_idx >= 0 ? J.Lc : f2zero();
        if (form == 0) {
            for (int q = tid; 4 * q < kp; q += kFormThreads) {
                u32 re[2][4], im[2][4], o[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const fp2 l = 4 * q + k < cs ? ld2(J.L + 4 * q + k) : f2zero();
                    re[0][k] = (u32)l.re;
                    re[1][k] = (u32)(l.re >> 32);
                    im[0][k] = (u32)l.im;
                    im[1][k] = (u32)(l.im >> 32);
                }
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    transpose4(re[h], o);
#pragma unroll
                    for (int k = 0; k < 4; ++k) *reinterpret_cast<u32*>(planes + (4 * h + k) * pitch + 4 * q) = o[k];
                    transpose4(im[h], o);
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        *reinterpret_cast<u32*>(planes + (8 + 4 * h + k) * pitch + 4 * q) = o[k];
                }
            }
        } else {
            for (int i = tid; i < 16 * (kp >> 2); i += kFormThreads)
                *reinterpret_cast<u32*>(planes + (i / (kp >> 2)) * pitch + 4 * (i % (kp >> 2))) = 0u;
            __syncthreads();
            // the group's terms: one per wire a
            for (int e = J.gptr[form - 1] + tid; e < J.gptr[form]; e += kFormThreads) {
                const int a = J.ab[e].x;
                const fp2 c = ld2(J.cf + e);
                if (a < cs) {
#pragma unroll
                    for (int l = 0; l < 8; ++l) {
                        planes[l * pitch + a] = (unsigned char)(c.re >> (8 * l));
                        planes[(8 + l) * pitch + a] = (unsigned char)(c.im >> (8 * l));
                    }
                } else if (a == J.const_idx) {
                    s_const = l2canon(mk(lmul(c.re, J.const_val), lmul(c.im, J.const_val)));
                }
            }
        }
        fp2* out = const_cast<fp2*>(J.A) + (size_t)(form == 0 ? 0 : 2 * form - 1) * J.n_in;
        for (int t = t0; t < t1; ++t) {
            const unsigned char* buf = tile[(t - t0) & 1];
            if (t + 1 < t1) {
                stage_tile(J, t + 1, tile[(t + 1 - t0) & 1], pitch);
                asm volatile("cp.async.wait_group 1;" ::: "memory");
            } else {
                asm volatile("cp.async.wait_group 0;" ::: "memory");
            }
            __syncthreads();
            if (form == 0) {   // the copy of the bytes that the finish reads
                const int per = kp >> 4, live = kTileRows * per;
                const int rows = min(kTileRows, J.n_real - t * kTileRows);
                uint4* to = reinterpret_cast<uint4*>(J.bytes + (size_t)(t * kTileRows) * kp);
#pragma unroll 4
                for (int i = tid; i < live; i += kFormThreads) {
                    const int r = i / per, q = i - r * per;
                    if (r < rows) to[i] = *reinterpret_cast<const uint4*>(buf + r * pitch + 16 * q);
                }
            } else if (tid < kTileRows) {   // the group's wire b
                const int c = t * kTileRows + tid, b = J.gb[form - 1];
                if (c < J.n_in) {
                    const u64 v = c >= J.n_real ? 0 : b < cs ? buf[tid * pitch + b] : b == J.const_idx ? J.const_val : 0;
                    st2(out + J.n_in + c, mk(v, 0));
                }
            }
            int d[2][4] = {{0, 0, 0, 0}, {0, 0, 0, 0}};   // limbs of re, of im
            // Both operands by one matrix load a step where eight words were loaded, and the
            // copy aside four vectors at a time: 64 1080p frames 216 -> 180 us (a warp per
            // row in place of the divisions: 271, a quarter of its lanes have no vector).
            // Lane l of a load gives row l % 8 of quarter l / 8: the copies' rows 0..7 and
            // 8..15 at bytes k and k + 16; the planes 0..7 at both, then 8..15
            const int q8 = lane >> 3, r8 = lane & 7;
            const u32 ar = smem_at(buf + (16 * warp + r8 + 8 * (q8 & 1)) * pitch + 16 * (q8 >> 1));
            const u32 br = smem_at(planes + (r8 + 8 * (q8 >> 1)) * pitch + 16 * (q8 & 1));
#pragma unroll 4
            for (int k = 0; k < kp; k += 32) {
                u32 a[4], b[4];
                load_quarters(a, ar + k);
                load_quarters(b, br + k);
                mma_u8(d[0], a[0], a[1], a[2], a[3], b[0], b[1]);
                mma_u8(d[1], a[0], a[1], a[2], a[3], b[2], b[3]);
            }
            // limbs 2j, 2j + 1 of rows g (d[.][0, 1]) and g + 8 (d[.][2, 3])
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                u64 re = shift_mod((u64)(u32)d[0][2 * h] + ((u64)(u32)d[0][2 * h + 1] << 8), 16 * j);
                u64 im = shift_mod((u64)(u32)d[1][2 * h] + ((u64)(u32)d[1][2 * h + 1] << 8), 16 * j);
#pragma unroll
                for (int o = 1; o < 4; o <<= 1) {
                    re += __shfl_xor_sync(0xffffffffu, re, o);
                    im += __shfl_xor_sync(0xffffffffu, im, o);
                }
                const int c = t * kTileRows + 16 * warp + g + 8 * h;
                if (j == h && c < J.n_in) {
                    fp2 v = mk(fold61(re), fold61(im));
                    if (c < J.n_real) v = l2add(v, s_const);
                    st2(out + c, v);
                }
            }
            __syncthreads();
        }
    }
}

// ---- rounds ---------------------------------------------------------------------

// loads of vectors: read-only in a launch of one round, written by the same CTA
// between its rounds in the launch of all
template <bool kSame>
__device__ __forceinline__ fp2 ldv(const fp2* p)
{
    if (!kSame) return ld2(p);
    const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p);
    return mk(v.x, v.y);
}

__device__ __forceinline__ void four_points(fp2 v0, fp2 v1, fp2 (&o)[4])
{
    o[0] = v0;
    o[1] = v1;
    o[2] = l2at_m1(v0, v1);
    o[3] = l2at_2(v0, v1);
}

// entries 2p, 2p + 1 of a vector of n_in entries (fold: of its fold by r, stored)
template <bool kSame>
__device__ __forceinline__ void pair_of(const fp2* in, fp2* out, int p, bool fold, fp2 r, fp2& x0, fp2& x1)
{
    if (!fold) {
        x0 = ldv<kSame>(in + 2 * (size_t)p);
        x1 = ldv<kSame>(in + 2 * (size_t)p + 1);
        return;
    }
    const fp2* q = in + 4 * (size_t)p;
    const fp2 a0 = ldv<kSame>(q), a1 = ldv<kSame>(q + 1), a2 = ldv<kSame>(q + 2), a3 = ldv<kSame>(q + 3);
    x0 = l2fold(a0, a1, r);
    x1 = l2fold(a2, a3, r);
    st2(out + 2 * (size_t)p, x0);
    st2(out + 2 * (size_t)p + 1, x1);
}

// the claim's four points at pair p of the (folded) vectors, nearly canonical
template <bool kSame>
__device__ __forceinline__ void pair_claim(const Job& J, const fp2* in, fp2* out, const fp2* beta, fp2* beta_out,
                                           int n_in, int p, bool fold, fp2 r, fp2 (&acc)[4])
{
    const size_t n = (size_t)n_in, no = n >> 1;
    fp2 x0, x1, V[4], b4[4];
    pair_of<kSame>(in, out, p, fold, r, x0, x1);
    four_points(x0, x1, V);
#pragma unroll
    for (int t = 0; t < 4; ++t) V[t] = l2add(V[t], J.K0);
    for (int g = 0; g < J.G; ++g) {
        fp2 m[4], y[4];
        pair_of<kSame>(in + (2 * g + 1) * n, out + (2 * g + 1) * no, p, fold, r, x0, x1);
        four_points(x0, x1, m);
        pair_of<kSame>(in + (2 * g + 2) * n, out + (2 * g + 2) * no, p, fold, r, x0, x1);
        four_points(x0, x1, y);
#pragma unroll
        for (int t = 0; t < 4; ++t) V[t] = l2add(V[t], l2mul(m[t], y[t]));
    }
    pair_of<kSame>(beta, beta_out, p, fold, r, x0, x1);
    four_points(x0, x1, b4);
#pragma unroll
    for (int t = 0; t < 4; ++t) acc[t] = l2add(acc[t], l2mul(b4[t], V[t]));
}

// The CTA's sum of acc (canonical), valid on the threads of warp 0. Serial between two
// rounds, so: four sums are taken across a warp by halving, in 6 exchanges instead of
// 20, and across the warps by eight lanes each. The nine rounds of a 240p frame in one
// CTA, challenges given: 54 -> 37 us; a launch of a 1080p batch's first round 39 -> 28.
template <int kWarps>
__device__ __forceinline__ void cta_sum(fp2 (&acc)[4], fp2 (*ws)[4])
{
    static_assert(kWarps == 8 || kWarps == 16, "eight lanes a sum, one or two warps each");
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    auto plus = [](fp2 keep, fp2 send, int o) {
        return l2add(keep, mk(__shfl_xor_sync(0xffffffffu, send.re, o), __shfl_xor_sync(0xffffffffu, send.im, o)));
    };
    const bool up = lane & 16, odd = lane & 8;
    const fp2 v0 = plus(up ? acc[2] : acc[0], up ? acc[0] : acc[2], 16);
    const fp2 v1 = plus(up ? acc[3] : acc[1], up ? acc[1] : acc[3], 16);
    fp2 v = plus(odd ? v1 : v0, odd ? v0 : v1, 8);
#pragma unroll
    for (int o = 4; o; o >>= 1) v = plus(v, v, o);
    if ((lane & 7) == 0) ws[warp][lane >> 3] = v;
    __syncthreads();
    if (warp) return;
    v = ws[lane >> 2][lane & 3];
    if (kWarps == 16) v = l2add(v, ws[8 + (lane >> 2)][lane & 3]);
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) v = plus(v, v, o);
    v = l2canon(v);
#pragma unroll
    for (int t = 0; t < 4; ++t) acc[t] = mk(__shfl_sync(0xffffffffu, v.re, t), __shfl_sync(0xffffffffu, v.im, t));
}

// one round of every job: a thread per pair; the job's last CTA (ticket) adds the
// CTAs' sums. A fold's challenge is recorded for the finish.
template <bool kFold>
__global__ void __launch_bounds__(kVecThreads) vec_round_kernel(const Job* __restrict__ jobs)
{
    __shared__ __align__(16) Job J;
    __shared__ fp2 ws[kVecThreads / 32][4];
    __shared__ bool s_last;
    read_job(jobs, J);
    if ((int)blockIdx.x >= J.tiles) return;
    const int p = blockIdx.x * kVecThreads + threadIdx.x;
    fp2 acc[4] = {f2zero(), f2zero(), f2zero(), f2zero()};
    if (p < J.n_pairs) pair_claim<false>(J, J.A, J.Aout, J.beta, J.beta_out, J.n_in, p, kFold, J.r, acc);
    cta_sum<kVecThreads / 32>(acc, ws);
    const int tid = threadIdx.x;
    if (kFold && blockIdx.x == 0 && tid == 0) st2(J.rs + J.nf, J.r);
    if (J.tiles > 1) {
        if (tid == 0) {
#pragma unroll
            for (int t = 0; t < 4; ++t) stcg2(J.partials + (size_t)blockIdx.x * 4 + t, acc[t]);
            __threadfence();
            s_last = atomicAdd(J.ticket, 1u) == (unsigned)(J.tiles - 1);
        }
        __syncthreads();
        if (!s_last) return;
        __threadfence();
#pragma unroll
        for (int t = 0; t < 4; ++t) acc[t] = f2zero();
        for (int i = tid; i < J.tiles; i += kVecThreads)
#pragma unroll
            for (int t = 0; t < 4; ++t) acc[t] = f2add(acc[t], ldcg2(J.partials + (size_t)i * 4 + t));
        cta_sum<kVecThreads / 32>(acc, ws);
        if (tid == 0) *J.ticket = 0u;
    }
    if (tid == 0)
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            J.out8[2 * t] = acc[t].re;
            J.out8[2 * t + 1] = acc[t].im;
        }
}

// All rounds of a frame that are left, one CTA per frame: job J with n_in copies
// (pending fold by J.r when J.has_r), J.n_rounds claims from round k0 on. The last
// challenge's fold is left to the finish. The challenges: J.given[q], or drawn by
// the VOLE-committed round (a.st set). Claims at J.out8 + q a.claim_stride.
struct RoundsArgs {
    fs::State* st;
    vole::State* vs;
    const fp2* u;
    const fp2* v;
    fp2* chal;       // [round][frame]
    fp2* proof;      // [round][frame][5], optional
    long long count;
    long long claim_stride;   // u64s between a frame's claims of successive rounds
    int n_frames, layer, k0;
};

template <bool kVole>
__global__ void __launch_bounds__(kRoundsThreads, 1) vec_rounds_kernel(const Job* __restrict__ jobs, const RoundsArgs a)
{
    __shared__ __align__(16) Job J;
    __shared__ fp2 ws[kRoundsThreads / 32][4];
    __shared__ fp2 s_r;
    __shared__ fs::TxMem tx;
    __shared__ fs::State s_st;      // the transcript between the rounds
    __shared__ vole::State s_vs;
    read_job(jobs, J);
    const int tid = threadIdx.x;
    if (kVole && tid == 0) {
        s_st = a.st[J.frame];
        s_vs = a.vs[J.frame];
    }
    __syncthreads();
    const fp2* in = J.A;
    const fp2* beta = J.beta;
    fp2 *out = J.Aout, *beta_out = J.beta_out;
    int n = J.n_in, nf = J.nf;
    bool fold = J.has_r != 0;
    fp2 r = J.r;
    for (int q = 0; q < J.n_rounds; ++q) {
        fp2 acc[4] = {f2zero(), f2zero(), f2zero(), f2zero()};
        const int pairs = fold ? n >> 2 : n >> 1;
        if (kVole && tid < 8) {   // the round's correlations on their way from memory
            const unsigned long long at = s_vs.idx + (tid & 3);
            if (at < (unsigned long long)a.count)
                asm volatile("prefetch.global.L1 [%0];" ::"l"((tid < 4 ? a.u : a.v) + J.frame * a.count + at));
        }
        for (int p = tid; p < pairs; p += kRoundsThreads)
            pair_claim<true>(J, in, out, beta, beta_out, n, p, fold, r, acc);
        if (fold) {
            if (tid == 0) st2(J.rs + nf, r);
            ++nf;
            n >>= 1;
            const fp2 *ti = in, *tb = beta;
            in = out;
            beta = beta_out;
            out = const_cast<fp2*>(ti);
            beta_out = const_cast<fp2*>(tb);
        }
        cta_sum<kRoundsThreads / 32>(acc, ws);
        if (tid < 32) {
            u64* o = J.out8 + q * a.claim_stride;
            if (tid == 0)
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                    o[2 * t] = acc[t].re;
                    o[2 * t + 1] = acc[t].im;
                }
            fp2 c;
            if (kVole) {
                const int i = J.frame, k = a.k0 + q;
                const size_t at = (size_t)a.n_frames * k + i;
                fp2 coef[4];
                vole::State w = s_vs;
                fs::Writer s(s_st, &tx);
                vole::interpolate_cubic(acc[0], acc[1], acc[2], acc[3], coef);
                vole::round(s, w, coef, 4, a.u + i * a.count, a.v + i * a.count, a.count, vole::sc_label(a.layer, k),
                            a.proof ? a.proof + 5 * at : nullptr, &c);
                s.store(s_st);
                if (tid == 0) {
                    s_vs = w;
                    a.chal[at] = c;
                }
            } else {
                c = ld2(J.given + q);
            }
            if (tid == 0) s_r = c;
        }
        __syncthreads();
        r = s_r;
        fold = true;
    }
    if (kVole && tid == 0) {
        a.st[J.frame] = s_st;
        a.vs[J.frame] = s_vs;
    }
}

// ---- finish ---------------------------------------------------------------------

// eq(point, c) for the copies c of up to 16 chunks of 512 in a row: the products over
// bits 0..3 and 4..8 of c and over each chunk's higher bits, in shared memory (64
// threads or more)
constexpr int kMaxPieces = 16;
struct EqParts {
    fp2 r[64];
    fp2 lo[16], mid[32], hi[kMaxPieces];
};
// from the first n entries of e.r
__device__ void eq_parts(EqParts& e, int n, int chunk, int pieces)
{
    const int tid = threadIdx.x;
    const fp2 one = mk(1, 0);
    auto prod = [&](int idx, int first, int last) {
        fp2 v = one;
        for (int b = first; b < last && b < n; ++b)
            v = l2mul(v, ((idx >> (b - first)) & 1) ? e.r[b] : l2sub(one, e.r[b]));
        return v;
    };
    if (tid < 16) e.lo[tid] = prod(tid, 0, 4);
    else if (tid < 48) e.mid[tid - 16] = prod(tid - 16, 4, 9);
    else if (tid < 48 + pieces) e.hi[tid - 48] = prod(chunk + tid - 48, 9, n);
}
// at a job's challenges
__device__ void eq_parts(const Job& J, int chunk, int pieces, EqParts& e)
{
    const int kf = J.nf + (J.has_r != 0);
    for (int k = threadIdx.x; k < kf; k += blockDim.x) e.r[k] = k < J.nf ? ldcg2(J.rs + k) : J.r;
    __syncthreads();
    eq_parts(e, kf, chunk, pieces);
    __syncthreads();
}
// c: within the piece
__device__ __forceinline__ fp2 eq_of(const EqParts& e, int c, int piece = 0)
{
    return l2mul(l2mul(e.lo[c & 15], e.mid[c >> 4]), e.hi[piece]);
}

// ---- bytes weighted over the copies --------------------------------------------
// sum over copies of eq(c) byte(c, w), a warp per 32 wires: the 16 byte-planes of
// eq are the mma's rows, the wires its columns (words of four copies' four wires,
// transposed in registers), 512 copies' planes at a time.
//
// Read bandwidth is the bound on paper (64 1080p frames: 398 MB, 57 us); what is spent
// besides are the products that make the weights and a CTA's serial start and end, 10
// of 26 us of a CTA of 512 copies, so a CTA takes several such pieces in a row where
// there are CTAs enough (row_pieces): the finish of 64 frames took 173 us with one piece
// a CTA, 93 with eight (282 with each step's loads waited for, one CTA an SM).
constexpr int kPlanePitch = kFinCopies + 16;

// the planes of the piece's first lim copies' weights, zero behind; their sum added to
// the thread's sum
__device__ __forceinline__ void weight_planes(const EqParts& e, int piece, int lim, unsigned char* E, fp2& sum)
{
    for (int c = threadIdx.x; c < kFinCopies; c += blockDim.x) {
        fp2 v = f2zero();
        if (c < lim) {
            v = l2canon(eq_of(e, c, piece));
            sum = l2add(sum, v);
        }
#pragma unroll
        for (int l = 0; l < 8; ++l) {
            E[l * kPlanePitch + c] = (unsigned char)(v.re >> (8 * l));
            E[(8 + l) * kPlanePitch + c] = (unsigned char)(v.im >> (8 * l));
        }
    }
}

// the wire of the warp's 32 whose sum a lane gets
__device__ __forceinline__ int weighed_wire(int lane)
{
    const int g = lane >> 2, j = lane & 3;
    return 4 * (2 * j + (g & 1)) + (g >> 1);
}

struct Weighed {
    int d[4][4];

    // v: the words of the wires 4g .. 4g + 3 of the copies k + 4j + i and k + 16 + 4j + i
    __device__ __forceinline__ void step(const unsigned char* E, int k, const u32 (&v)[8])
    {
        const int lane = threadIdx.x & 31, g = lane >> 2, j = lane & 3;
        const unsigned char* er = E + g * kPlanePitch + k + 4 * j;
        auto word = [](const unsigned char* p) { return *reinterpret_cast<const u32*>(p); };
        const u32 a0 = word(er), a1 = word(er + 8 * kPlanePitch), a2 = word(er + 16),
                  a3 = word(er + 8 * kPlanePitch + 16);
        const u32 lo[4] = {v[0], v[1], v[2], v[3]}, hi[4] = {v[4], v[5], v[6], v[7]};
        u32 b0[4], b1[4];
        transpose4(lo, b0);
        transpose4(hi, b1);
#pragma unroll
        for (int m = 0; m < 4; ++m) mma_u8(d[m], a0, a1, a2, a3, b0[m], b1[m]);
    }
    __device__ __forceinline__ fp2 total() const;
};

// A warp's 32 columns of whole 16-byte vectors, by asynchronous copies: kRowStages - 1
// steps of 32 copies are on their way from before the weights are made. Four copies'
// 32 bytes lie together, and four times four in different banks. The ring starts on a
// 128-byte boundary: with every row 16 bytes off its 32 the finish of 64 1080p frames took
// 133 us in place of 94.
constexpr int kRowStages = 5, kRowStep = 8 * 160;

struct RowCopies {
    const unsigned char* src;   // column 0 of the warp's wires in the chunk's first copy
    int pitch, copies, width;   // width: columns there are, 16 or 32 at least of them
    unsigned char* ring;

    __device__ __forceinline__ void fetch(int step) const
    {
        const int lane = threadIdx.x & 31, q = lane & 1;
        if (32 * step < copies) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int r = 16 * h + (lane >> 1), c = min(32 * step + r, copies - 1);
                const bool in = 16 * q < width;
                async16(ring + (step % kRowStages) * kRowStep + (r >> 2) * 160 + (r & 3) * 32 + 16 * q,
                        src + (size_t)c * pitch + (in ? 16 * q : 0), in);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    __device__ __forceinline__ void start() const
    {
#pragma unroll
        for (int k = 0; k < kRowStages - 1; ++k) fetch(k);
    }
    // the piece's copies, E: its planes
    __device__ __forceinline__ void sum(int piece, const unsigned char* E, Weighed& t) const
    {
        constexpr int kSteps = kFinCopies / 32;
        const int lane = threadIdx.x & 31, g = lane >> 2, j = lane & 3;
        for (int k = kSteps * piece; k < kSteps * (piece + 1) && 32 * k < copies; ++k) {
            asm volatile("cp.async.wait_group %0;" ::"n"(kRowStages - 2) : "memory");
            __syncwarp();   // the step is here, and the one before it read by all lanes
            fetch(k + kRowStages - 1);
            const unsigned char* p = ring + (k % kRowStages) * kRowStep + j * 160 + 4 * g;
            u32 v[8];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                v[i] = *reinterpret_cast<const u32*>(p + 32 * i);
                v[4 + i] = *reinterpret_cast<const u32*>(p + 4 * 160 + 32 * i);
            }
            t.step(E, 32 * (k % kSteps), v);
        }
    }
};

// any other rows' piece, with plain loads; load(c): the word of the wires 4g .. 4g + 3
// of the piece's copy c
template <class Load>
__device__ __forceinline__ void weigh_words(const unsigned char* E, int copies, Weighed& t, Load load)
{
    const int j = threadIdx.x & 3;
    for (int k = 0; k < copies; k += 32) {
        u32 v[8];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            v[i] = load(k + 4 * j + i);
            v[4 + i] = load(k + 16 + 4 * j + i);
        }
        t.step(E, k, v);
    }
}

__device__ __forceinline__ fp2 Weighed::total() const
{
    const int g = (threadIdx.x & 31) >> 2;
    // lane (g, j): limb g of re (d[m][0, 1]) and im (d[m][2, 3]) of the wires
    // 4 (2j) + m and 4 (2j + 1) + m; summed over g by halving
    fp2 v[4][2];
#pragma unroll
    for (int m = 0; m < 4; ++m)
#pragma unroll
        for (int h = 0; h < 2; ++h)
            v[m][h] = mk(shift_mod((u64)(u32)d[m][h], 8 * g), shift_mod((u64)(u32)d[m][2 + h], 8 * g));
    auto halve = [](bool up, fp2 a, fp2 b, int o) {   // a of lanes without the bit, b of those with it
        const fp2 keep = up ? b : a, send = up ? a : b;
        return mk(keep.re + __shfl_xor_sync(0xffffffffu, send.re, o), keep.im + __shfl_xor_sync(0xffffffffu, send.im, o));
    };
    fp2 u[2][2], t[2];
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int h = 0; h < 2; ++h) u[m][h] = halve(g & 4, v[m][h], v[m + 2][h], 16);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        t[h] = halve(g & 2, u[0][h], u[1][h], 8);
        t[h] = mk(fold61(t[h].re), fold61(t[h].im));
    }
    const fp2 s = halve(g & 1, t[0], t[1], 4);
    return mk(fold61(s.re), fold61(s.im));
}

// beta's value: entry 0 after the pending fold
__device__ __forceinline__ void finish_beta(const Job& J)
{
    const fp2 b = J.has_r ? l2fold(ld2(J.beta), ld2(J.beta + 1), J.r) : ld2(J.beta);
    st2(J.fin_beta, l2canon(b));
}

// wires from the copied bytes. CTA = J.wpg pieces of 512 copies; partial sums per CTA,
// the job's last one adds them up.
__global__ void __maxnreg__(80) finish_bytes_kernel(const Job* __restrict__ jobs)
{
    extern __shared__ __align__(128) unsigned char rings[];
    __shared__ __align__(16) Job J;
    __shared__ EqParts e;
    __shared__ __align__(16) unsigned char E[2][16 * kPlanePitch];
    __shared__ fp2 ws[16];
    __shared__ bool s_last;
    read_job(jobs, J);
    const int chunk = blockIdx.x;
    if (chunk >= J.chunks) return;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int kf = J.nf + (J.has_r != 0);
    const int c0 = chunk * J.wpg * kFinCopies;
    const int lim = min(min(J.n_real, 1 << kf) - c0, J.wpg * kFinCopies);   // copies that count
    const int kp = J.stride, warps = blockDim.x >> 5, w0 = 32 * warp;
    const RowCopies rc = {J.bytes + (size_t)c0 * kp + w0, kp, w0 < kp ? lim : 0, 32,
                          rings + warp * (kRowStages * kRowStep)};
    rc.start();
    eq_parts(J, chunk * J.wpg, J.wpg, e);
    fp2 sum = f2zero();
    Weighed t = {};
    for (int p = 0; p < J.wpg; ++p) {
        weight_planes(e, p, lim - p * kFinCopies, E[p & 1], sum);
        __syncthreads();
        rc.sum(p, E[p & 1], t);
    }
    sum = warp_sum(l2canon(sum));
    if (lane == 0) ws[warp] = sum;
    __syncthreads();
    const int Wp = J.W_rows;
    fp2* part = J.fpart + (size_t)chunk * Wp;
    if (w0 < kp) {
        const fp2 v = t.total();
        const int w = w0 + weighed_wire(lane);
        if (w < J.cs) stcg2(part + w, l2canon(v));
    }
    if (tid == 0) {
        fp2 s = f2zero();
        for (int k = 0; k < warps; ++k) s = f2add(s, ws[k]);
        if (J.const_idx >= J.cs) stcg2(part + J.const_idx, f2scale(s, J.const_val));
    }
    __syncthreads();
    if (tid == 0) {
        __threadfence();
        s_last = atomicAdd(J.ticket, 1u) == (unsigned)(J.chunks - 1);
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    for (int w = tid; w < J.W; w += blockDim.x) {
        fp2 v = f2zero();
        if (w < J.cs || (w == J.const_idx && w < Wp)) {
#pragma unroll 8
            for (int k = 0; k < J.chunks; ++k) v = f2add(v, ldcg2(J.fpart + (size_t)k * Wp + w));
        }
        st2(J.fin + w, v);
    }
    if (tid == 0) {
        finish_beta(J);
        *J.ticket = 0u;
    }
}

// ---- MLE of a frame's input vector from its bytes -------------------------------
//   sum_c hi[c] (sum_{w < cs} lo[w] byte(c, w) + const_val lo[const_idx]),
// lo and hi the eq weights of the point's first h and further hb entries. The copies
// are summed first, 512 to a CTA, on the tensor cores; what is left is a dot product
// over the wires. Both weights are made by the CTA that uses them. Bound by reading
// the bytes and by the weights (64 1080p frames, 398 MB: 96 us; a thread per copy with
// four 32 x 32 multiplications a byte took 244, its eq tables 110).
struct MleArgs {
    const MleFrame* frames;
    const fp2* points;
    fp2* partials;
    unsigned* tickets;
    fp2* out;
    u64 const_val;
    int cs, h, hb, const_idx, pieces;   // pieces: a CTA's, of 512 copies
};

// kRows: what every frame's rows are: whole aligned 16-byte vectors, words, or bytes
enum : int { kRowVectors, kRowWords, kRowBytes };
template <int kRows>
__global__ void __maxnreg__(80) mle_bytes_kernel(const MleArgs a)
{
    extern __shared__ __align__(128) unsigned char rings[];
    __shared__ EqParts e, el;
    __shared__ __align__(16) unsigned char E[2][16 * kPlanePitch];
    __shared__ fp2 ws[16], wt[16];
    __shared__ bool s_last;
    const int f = blockIdx.y, chunk = blockIdx.x, per = a.pieces * kFinCopies;
    const MleFrame fr = a.frames[f];
    const int chunks = max(1, (fr.n_real + per - 1) / per);
    if (chunk >= chunks) return;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, warps = blockDim.x >> 5;
    const int cs = a.cs, w0 = 32 * warp;
    const int c0 = chunk * per, lim = min(per, fr.n_real - c0);
    const unsigned char* src = fr.pix + (size_t)c0 * cs + w0;
    const RowCopies rc = {src, cs, w0 < cs ? lim : 0, cs - w0, rings + warp * (kRowStages * kRowStep)};
    if (kRows == kRowVectors) rc.start();
    const fp2* z = a.points + (size_t)f * (a.h + a.hb);
    for (int k = tid; k < a.h + a.hb; k += blockDim.x) {
        const fp2 v = ld2(z + k);
        (k < a.h ? el.r[k] : e.r[k - a.h]) = mk(fold61(v.re), fold61(v.im));
    }
    __syncthreads();
    eq_parts(e, a.hb, chunk * a.pieces, a.pieces);
    eq_parts(el, a.h, 0, 1);
    __syncthreads();
    fp2 sum = f2zero(), acc = f2zero();
    Weighed bytes = {};
    for (int p = 0; p < a.pieces; ++p) {
        const int at = p * kFinCopies;
        weight_planes(e, p, lim - at, E[p & 1], sum);
        __syncthreads();
        if (kRows == kRowVectors)
            rc.sum(p, E[p & 1], bytes);
        else if (w0 < cs)
            weigh_words(E[p & 1], min(kFinCopies, lim - at), bytes, [&](int c) -> u32 {   // rows past the last weigh nothing
                const int col = 4 * (lane >> 2);
                const unsigned char* q = src + (size_t)min(at + c, lim - 1) * cs + col;
                if (kRows == kRowWords) return w0 + col < cs ? __ldg(reinterpret_cast<const u32*>(q)) : 0u;
                u32 x = 0;
#pragma unroll
                for (int b = 0; b < 4; ++b)
                    if (w0 + col + b < cs) x |= (u32)__ldg(q + b) << (8 * b);
                return x;
            });
    }
    sum = warp_sum(l2canon(sum));
    if (lane == 0) ws[warp] = sum;
    if (w0 < cs) {
        const fp2 v = bytes.total();
        const int w = w0 + weighed_wire(lane);
        if (w < cs) acc = l2mul(eq_of(el, w), v);
    }
    acc = warp_sum(l2canon(acc));
    if (lane == 0) wt[warp] = acc;
    __syncthreads();
    if (tid == 0) {
        fp2 s = f2zero(), t = f2zero();
        for (int k = 0; k < warps; ++k) {
            s = f2add(s, ws[k]);
            t = f2add(t, wt[k]);
        }
        if (a.const_idx >= 0) t = l2add(t, l2mul(eq_of(el, a.const_idx), l2canon(f2scale(s, a.const_val))));
        t = l2canon(t);
        stcg2(a.partials + (size_t)f * gridDim.x + chunk, t);
        __threadfence();
        s_last = atomicAdd(a.tickets + f, 1u) == (unsigned)(chunks - 1);
    }
    __syncthreads();
    if (!s_last || warp != 0) return;
    __threadfence();
    fp2 t = f2zero();
    for (int k = lane; k < chunks; k += 32) t = f2add(t, ldcg2(a.partials + (size_t)f * gridDim.x + k));
    t = warp_sum(t);
    if (lane == 0) {
        st2(a.out + fr.slot, t);
        a.tickets[f] = 0u;
    }
}

size_t row_smem(unsigned threads) { return (size_t)(threads / 32) * kRowStages * kRowStep; }

size_t form_smem(int kp) { return (size_t)(2 * kTileRows + 16) * (kp + 16); }

}  // namespace

int lin_stride(int cs) { return (cs + 31) & ~31; }
size_t lin_bytes(int cs, int n_real)
{
    const size_t rows = ((size_t)std::max(1, n_real) + kFinCopies - 1) / kFinCopies * kFinCopies;
    return rows * lin_stride(cs);
}
int lin_chunks(int n_real, int folds)
{
    const long long lim = std::min<long long>(n_real, 1LL << folds);
    return (int)std::max<long long>(1, (lim + kFinCopies - 1) / kFinCopies);
}

// Pieces of 512 copies per CTA of the weighted byte sums, chunks: the frames' pieces.
// What a CTA spends besides its pieces is about one piece's time, and two CTAs fit an
// SM: the number of pieces with the fewest (pieces + 1) x waves. 64 1080p frames, 2,048
// pieces: 8 (256 CTAs); one frame or a few small ones: 1.
int row_pieces(const std::vector<int>& chunks)
{
    Ctx* c = ctx();
    const long long fit = 2LL * (c ? c->n_sm : 148);
    int best = 1;
    long long best_cost = 0;
    for (int p = 1; p <= kMaxPieces; ++p) {
        long long ctas = 0;
        for (int k : chunks) ctas += (k + p - 1) / p;
        const long long cost = (ctas + fit - 1) / fit * (p + 1);
        if (p == 1 || cost < best_cost) best = p, best_cost = cost;
    }
    return best;
}

void plan_linear_finish(std::vector<Job>& jobs)
{
    std::vector<int> chunks;
    for (const Job& j : jobs) chunks.push_back(j.chunks);
    const int p = chunks.empty() ? 1 : row_pieces(chunks);
    for (Job& j : jobs) {
        j.wpg = p;
        j.chunks = (j.chunks + p - 1) / p;
    }
}

bool prepare_linear_kernels()
{
    static std::atomic<bool> done{false};   // sessions of several threads come here
    if (done.load()) return true;
    TP_CUDA_OK(cudaFuncSetAttribute(forms_bytes_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)form_smem(512)),
               "forms smem attr");
    TP_CUDA_OK(cudaFuncSetAttribute(finish_bytes_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)row_smem(512)),
               "finish smem attr");
    TP_CUDA_OK(cudaFuncSetAttribute(mle_bytes_kernel<kRowVectors>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)row_smem(512)),
               "mle smem attr");
    done.store(true);
    return true;
}

// target: CTAs for the byte forms, which take up to 16 tiles each
void plan_linear_job(Job& j, int kind, int target)
{
    if (kind == kFormsBytes) {
        const int tiles = (j.n_in + kTileRows - 1) / kTileRows;
        j.wpg = std::max(1, std::min(16, tiles / target));
        j.tiles = (tiles + j.wpg - 1) / j.wpg;
    } else {
        j.tiles = std::max(1, (j.n_pairs + kVecThreads - 1) / kVecThreads);
    }
    j.groups = 1;
}

bool launch_linear(const Job* d_jobs, const std::vector<Job>& jobs, int kind, cudaStream_t s, int* launches)
{
    if (jobs.empty()) return true;
    if (!prepare_linear_kernels()) return false;
    unsigned ctas = 1;
    int kp = 0;
    for (const Job& j : jobs) {
        ctas = std::max(ctas, (unsigned)j.tiles);
        kp = std::max(kp, j.stride);
    }
    const dim3 grid(ctas, (unsigned)jobs.size());
    if (kind == kFormsBytes) forms_bytes_kernel<<<grid, kFormThreads, form_smem(kp), s>>>(d_jobs);
    else if (kind == kVecClaim) vec_round_kernel<false><<<grid, kVecThreads, 0, s>>>(d_jobs);
    else vec_round_kernel<true><<<grid, kVecThreads, 0, s>>>(d_jobs);
    ++*launches;
    return !cuda_failed(cudaGetLastError(), "linear round launch");
}

bool launch_linear_rounds(const Job* d_jobs, int n_jobs, const VoleRounds* v, int k0, long long claim_stride,
                          cudaStream_t s, int* launches)
{
    RoundsArgs a = {};
    a.k0 = k0;
    a.claim_stride = claim_stride;
    const dim3 grid(1, (unsigned)n_jobs);
    if (v) {
        a.st = static_cast<fs::State*>(v->states);
        a.vs = static_cast<vole::State*>(v->vole_states);
        a.u = v->u;
        a.v = v->v;
        a.chal = v->chal;
        a.proof = v->proof;
        a.count = v->count;
        a.n_frames = v->n_frames;
        a.layer = v->layer;
        vec_rounds_kernel<true><<<grid, kRoundsThreads, 0, s>>>(d_jobs, a);
    } else {
        vec_rounds_kernel<false><<<grid, kRoundsThreads, 0, s>>>(d_jobs, a);
    }
    ++*launches;
    return !cuda_failed(cudaGetLastError(), "linear rounds launch");
}

bool launch_mle_pixels_batch(const MleFrame* h_frames, int n, int n_pad, int cs, int W,
                             int const_idx, u64 const_val, const fp2* d_points, fp2* d_out,
                             cudaStream_t s, int* launches, void* d_ws, size_t ws_bytes)
{
    if (n <= 0) return true;
    if (!prepare_linear_kernels()) return false;
    if ((W & (W - 1)) || (n_pad & (n_pad - 1)) || W > 512 || cs <= 0 || cs > W ||
        const_idx >= W || (const_idx >= 0 && const_idx < cs) || const_val >= P61) {
        set_error(TP_ERR_ARG, "mle over bytes: bad layout (wires %d, copies %d, copy_size %d)", W,
                  n_pad, cs);
        return false;
    }
    MleArgs a = {};
    size_t bits = (size_t)cs;   // what the rows' addresses have in common
    std::vector<int> chunks;
    for (int i = 0; i < n; ++i) {
        if (!h_frames[i].pix || h_frames[i].n_real < 0 || h_frames[i].n_real > n_pad) {
            set_error(TP_ERR_ARG, "mle over bytes: frame %d has %d of %d copies", i,
                      h_frames[i].n_real, n_pad);
            return false;
        }
        chunks.push_back(lin_chunks(h_frames[i].n_real, 30));
        bits |= reinterpret_cast<size_t>(h_frames[i].pix);
    }
    while ((1 << a.h) < W) ++a.h;
    while ((1 << a.hb) < n_pad) ++a.hb;
    a.cs = cs;
    a.const_idx = const_idx;
    a.const_val = const_val;
    a.points = d_points;
    a.out = d_out;
    const int most = *std::max_element(chunks.begin(), chunks.end());
    a.pieces = row_pieces(chunks);
    const int ctas = (most + a.pieces - 1) / a.pieces;
    const size_t np = (size_t)ctas * n;
    const size_t bytes = sizeof(fp2) * np + (sizeof(MleFrame) + sizeof(unsigned)) * n;
    if (d_ws && ws_bytes < bytes) {
        set_error(TP_ERR_ARG, "mle over bytes: a workspace of %zu bytes, %zu needed", ws_bytes, bytes);
        return false;
    }
    if (reinterpret_cast<size_t>(d_ws) & 15) {
        set_error(TP_ERR_ARG, "mle over bytes: a workspace that is not 16-byte aligned");
        return false;
    }
    unsigned char* ws = (unsigned char*)(d_ws ? d_ws : dev_alloc(bytes, s));
    if (!ws) return false;
    a.partials = reinterpret_cast<fp2*>(ws);
    MleFrame* d_frames = reinterpret_cast<MleFrame*>(a.partials + np);
    a.tickets = reinterpret_cast<unsigned*>(d_frames + n);
    a.frames = d_frames;
    bool ok = !cuda_failed(cudaMemsetAsync(a.tickets, 0, sizeof(unsigned) * n, s), "mle tickets") &&
              upload_async(d_frames, h_frames, sizeof(MleFrame) * n, s);
    if (ok) {
        // A warp per 32 wires, and four at least: all threads make the weights (16 frames
        // of 512 copies, 12 bytes each: 34.5 us with two, 30.9; 64 bytes: 34.5 and 28.9).
        const unsigned threads = (unsigned)std::max(128, 32 * ((cs + 31) / 32));
        const dim3 grid((unsigned)ctas, (unsigned)n);
        if ((bits & 15) == 0) mle_bytes_kernel<kRowVectors><<<grid, threads, row_smem(threads), s>>>(a);
        else if ((bits & 3) == 0) mle_bytes_kernel<kRowWords><<<grid, threads, 0, s>>>(a);
        else mle_bytes_kernel<kRowBytes><<<grid, threads, 0, s>>>(a);
        ++*launches;
        ok = !cuda_failed(cudaGetLastError(), "mle batch launch");
    }
    if (!d_ws) dev_free(ws, s);
    return ok;
}

bool launch_linear_finish(const Job* d_jobs, const std::vector<Job>& jobs, cudaStream_t s, int* launches)
{
    if (jobs.empty()) return true;
    int chunks = 1, kp = 32;
    for (const Job& j : jobs) {
        chunks = std::max(chunks, j.chunks);
        kp = std::max(kp, j.stride);
    }
    const unsigned threads = (unsigned)std::max(64, kp);   // a warp per 32 wires, 512 at most
    finish_bytes_kernel<<<dim3((unsigned)chunks, (unsigned)jobs.size()), threads, row_smem(threads), s>>>(d_jobs);
    ++*launches;
    return !cuda_failed(cudaGetLastError(), "linear finish launch");
}

}  // namespace tp
