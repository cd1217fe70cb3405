// Prover-side passes of the Orion tensor-product opening over the row-major
// codeword that commit() leaves in HBM
// (TruePix-main/Orion/Orion_nonzk/src/VPD/linearPC.cpp:480-531, 569-571):
//   combined[t] = sum_j r0[j] * codeword[t][j]        (t < cw_len; the first N/128
//                 entries are combined_message)
//   leaves      = SHA256(combined[i] || 0^48), i < 2 N/128, zero element past
//                 cw_len (merkle_tree.cpp:5-13); tree as in the commit
//   queried     = queried_cols[i][j] = codeword[q_i][j]
//   answer      = sum_{i < N/128} r1[i] * combined[i]
#include <algorithm>

#include "fp2.cuh"
#include "orion.h"
#include "runtime.h"
#include "sha256.cuh"

namespace tp {
namespace orion {

namespace {

constexpr int kTagCombine = 9110, kTagCombineLeaves = 9111;

__device__ __forceinline__ fp2 ld_fe(const ulonglong2* p) { const ulonglong2 v = __ldg(p); return mk(v.y, v.x); }

__device__ __forceinline__ fp2 warp_sum2(fp2 a)
{
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        fp2 b;
        b.re = __shfl_xor_sync(0xffffffffu, a.re, o);
        b.im = __shfl_xor_sync(0xffffffffu, a.im, o);
        a = l2add(a, b);
    }
    return a;
}

// products accumulated over 128 bits before one reduction
struct Acc128 {
    unsigned __int128 ac, bd, s;
};

// v mod p, below 2^61 + 8, for v < 2^127
__device__ __forceinline__ u64 fold128(unsigned __int128 v)
{
    const u64 lo = (u64)v & P61, mid = (u64)(v >> 61) & P61, hi = (u64)(v >> 122);
    return fold61(lo + mid + hi);
}

// Four codeword rows per warp and step: lane l holds r0[l + 32k], k < 4, and multiplies
// the rows' four 512-byte column slices by them. Bound by HBM (2 KB a row) and, nearly
// as much, by the integer pipes, so: the rows come by asynchronous copies, four ahead in
// a ring that only the lane itself reads; a row's four products are added up over 128
// bits (three products each, at most 4 x 2^62 x 2^62.1 for the operands that l2mul
// takes) and reduced once; and the four rows are added across the warp by halving, in 6
// exchanges instead of 20. 1080p, 231 MB: 81 -> 48 us (cold clocks and L2).
constexpr int kCombineWarps = 4, kCombineRows = 4;

__global__ void __launch_bounds__(32 * kCombineWarps, 6)
    combine_kernel(const ulonglong2* __restrict__ rows, long long cw_len, const ulonglong2* __restrict__ r0,
                   ulonglong2* __restrict__ combined)
{
    __shared__ ulonglong2 ring[kCombineWarps][kCombineRows][4][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long step = (long long)gridDim.x * kCombineWarps * kCombineRows;
    const long long first = ((long long)blockIdx.x * kCombineWarps + warp) * kCombineRows;
    auto fetch = [&](long long t, int j) {   // row t into slot j; nothing past the last row
        if (t < cw_len) {
            const ulonglong2* row = rows + t * kColumns + lane;
#pragma unroll
            for (int k = 0; k < 4; ++k)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                                 (unsigned)__cvta_generic_to_shared(&ring[warp][j][k][lane])),
                             "l"(row + 32 * k)
                             : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int j = 0; j < kCombineRows; ++j) fetch(first + j, j);
    fp2 r[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const fp2 v = ld_fe(r0 + lane + 32 * k);
        r[k] = mk(fold61(v.re), fold61(v.im));
    }
    for (long long t = first; t < cw_len; t += step) {
        fp2 v[kCombineRows];
#pragma unroll
        for (int j = 0; j < kCombineRows; ++j) {
            asm volatile("cp.async.wait_group %0;" ::"n"(kCombineRows - 1) : "memory");
            Acc128 a = {0, 0, 0};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const ulonglong2 x = ring[warp][j][k][lane];
                a.ac += (unsigned __int128)r[k].re * x.y;
                a.bd += (unsigned __int128)r[k].im * x.x;
                a.s += (unsigned __int128)(r[k].re + r[k].im) * (x.y + x.x);
            }
            const u64 ac = fold128(a.ac), bd = fold128(a.bd), s = fold128(a.s);
            v[j] = mk(fold61(ac + (2 * P61 - bd)), fold61(s + (4 * P61 - ac - bd)));
            fetch(t + step + j, j);
        }
        // lanes with bit 4 set go on with rows 2 and 3, with bit 3 with the odd one
        auto halve = [&](fp2 keep, fp2 send, int o) {
            fp2 other;
            other.re = __shfl_xor_sync(0xffffffffu, send.re, o);
            other.im = __shfl_xor_sync(0xffffffffu, send.im, o);
            return l2add(keep, other);
        };
        const bool up = lane & 16, odd = lane & 8;
        const fp2 v0 = halve(up ? v[2] : v[0], up ? v[0] : v[2], 16);
        const fp2 v1 = halve(up ? v[3] : v[1], up ? v[1] : v[3], 16);
        fp2 acc = halve(odd ? v1 : v0, odd ? v0 : v1, 8);
#pragma unroll
        for (int o = 4; o; o >>= 1) acc = halve(acc, acc, o);
        const long long row = t + (lane >> 3);
        if ((lane & 7) == 0 && row < cw_len) combined[row] = make_ulonglong2(canon61(acc.im), canon61(acc.re));
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// leaves [0, size): SHA256(element || 0^48) of combined[i] for i < cw_len, of the
// zero element (= SHA256(0^64)) beyond
__global__ void __launch_bounds__(256) single_leaf_kernel(const ulonglong2* __restrict__ combined,
                                                          long long cw_len, long long size,
                                                          unsigned char* __restrict__ tree, uint32_t one)
{
    const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
    if (i >= size) return;
    uint32_t w[16], st[8];
    const ulonglong2 x = i < cw_len ? __ldg(combined + i) : make_ulonglong2(0, 0);
    sha::fe_words(x.x, x.y, w);
#pragma unroll
    for (int k = 4; k < 16; ++k) w[k] = 0;
    sha::hash64(w, st, sha::AddMad{one});
    uint4 a, b;
    a.x = sha::bswap32(st[0]); a.y = sha::bswap32(st[1]); a.z = sha::bswap32(st[2]); a.w = sha::bswap32(st[3]);
    b.x = sha::bswap32(st[4]); b.y = sha::bswap32(st[5]); b.z = sha::bswap32(st[6]); b.w = sha::bswap32(st[7]);
    uint4* p = reinterpret_cast<uint4*>(tree + (size + i) * 32);
    p[0] = a;
    p[1] = b;
}

// out[i] = rows[q[i]] (2 KB each); one CTA of 128 threads per query
__global__ void __launch_bounds__(128) query_kernel(const ulonglong2* __restrict__ rows, long long cw_len,
                                                    const long long* __restrict__ q, int count,
                                                    ulonglong2* __restrict__ out, int* __restrict__ bad)
{
    const int i = blockIdx.x;
    if (i >= count) return;
    const long long r = q[i];
    if (r < 0 || r >= cw_len) {
        if (threadIdx.x == 0) atomicExch(bad, 1);
        return;
    }
    out[(long long)i * kColumns + threadIdx.x] = __ldg(rows + r * kColumns + threadIdx.x);
}

// the same without a host round trip: a row index outside [0, cw_len) gives a
// zero row and raises *bad (when given), which the caller reads later
__global__ void __launch_bounds__(128) query_async_kernel(const ulonglong2* __restrict__ rows, long long cw_len,
                                                          const long long* __restrict__ q, int count,
                                                          ulonglong2* __restrict__ out, int* __restrict__ bad)
{
    const int i = blockIdx.x;
    if (i >= count) return;
    const long long r = q[i];
    const bool in = r >= 0 && r < cw_len;
    if (!in && bad && threadIdx.x == 0) atomicExch(bad, 1);
    out[(long long)i * kColumns + threadIdx.x] = in ? __ldg(rows + r * kColumns + threadIdx.x) : make_ulonglong2(0, 0);
}

// answer = sum_i r1[i] * combined[i], i < n: a CTA takes 1,024 entries, four loads in
// flight per thread, partial sums to `part`; the last CTA (ticket) adds them up with all
// its threads. Bound by that chain's latency. 61,000 entries: 16 us with 4,096 entries a
// CTA and one thread for the partial sums, now 7.5.
constexpr int kAnswerPer = 4;

__device__ __forceinline__ fp2 cta_sum(fp2 acc, fp2 (&sw)[8])
{
    acc = warp_sum2(acc);
    if ((threadIdx.x & 31) == 0) sw[threadIdx.x >> 5] = acc;
    __syncthreads();
    acc = f2zero();
    if (threadIdx.x < 32) {
        if (threadIdx.x < 8) acc = sw[threadIdx.x];
        acc = warp_sum2(acc);
    }
    return acc;   // in warp 0
}

__global__ void __launch_bounds__(256) answer_kernel(const ulonglong2* __restrict__ combined,
                                                     const ulonglong2* __restrict__ r1, long long n,
                                                     fp2* __restrict__ part, unsigned* __restrict__ ticket,
                                                     ulonglong2* __restrict__ answer)
{
    __shared__ fp2 sw[8];
    __shared__ bool last;
    const long long base = (long long)blockIdx.x * (256 * kAnswerPer) + threadIdx.x;
    fp2 x[kAnswerPer], y[kAnswerPer];
#pragma unroll
    for (int k = 0; k < kAnswerPer; ++k) {
        const long long i = base + 256 * k;
        x[k] = i < n ? ld_fe(r1 + i) : f2zero();
        y[k] = i < n ? ld_fe(combined + i) : f2zero();
    }
    fp2 acc = f2zero();
#pragma unroll
    for (int k = 0; k < kAnswerPer; ++k) acc = l2add(acc, l2mul(x[k], y[k]));
    acc = cta_sum(acc, sw);
    if (threadIdx.x == 0) {
        part[blockIdx.x] = acc;
        __threadfence();
        last = atomicAdd(ticket, 1u) == gridDim.x - 1;
        __threadfence();
    }
    __syncthreads();
    if (!last) return;
    acc = f2zero();
    const u64* pv = reinterpret_cast<const u64*>(part);
    for (unsigned b = threadIdx.x; b < gridDim.x; b += 256)
        acc = l2add(acc, mk(__ldcg(pv + 2 * b), __ldcg(pv + 2 * b + 1)));
    acc = cta_sum(acc, sw);
    if (threadIdx.x == 0) {
        *answer = make_ulonglong2(canon61(acc.im), canon61(acc.re));
        *ticket = 0;
    }
}

bool ok(const char* what) { return !cuda_failed(cudaGetLastError(), what); }

}  // namespace

bool combine(const ulonglong2* rows, long long col_len, long long cw_len, const ulonglong2* r0,
             ulonglong2* combined, unsigned char* tree, cudaStream_t s)
{
    const long long size = tree_leaves(col_len);
    Ctx* c = ctx();
    if (!c) return false;
    constexpr int kPerCta = kCombineWarps * kCombineRows;
    const unsigned blocks = (unsigned)std::min<long long>((cw_len + kPerCta - 1) / kPerCta, (long long)c->n_sm * 6);
    timer_begin(s, kTagCombine);
    combine_kernel<<<blocks, 32 * kCombineWarps, 0, s>>>(rows, cw_len, r0, combined);
    timer_end(s);
    if (!ok("orion combine")) return false;
    if (!tree) return true;
    if (cuda_failed(cudaMemsetAsync(tree, 0, 32, s), "orion combined tree clear")) return false;
    timer_begin(s, kTagCombineLeaves);
    single_leaf_kernel<<<(unsigned)((size + 255) / 256), 256, 0, s>>>(combined, cw_len, size, tree, 1u);
    timer_end(s);
    if (!ok("orion combined leaves")) return false;
    return build_tree(tree, size, s);
}

bool query_rows(const ulonglong2* rows, long long cw_len, const long long* q, int count, ulonglong2* out,
                cudaStream_t s)
{
    int* bad = static_cast<int*>(dev_alloc(sizeof(int), s));
    if (!bad) return false;
    int h_bad = 0;
    bool good = !cuda_failed(cudaMemsetAsync(bad, 0, sizeof(int), s), "orion query flag");
    if (good) {
        query_kernel<<<count, 128, 0, s>>>(rows, cw_len, q, count, out, bad);
        good = ok("orion query") &&
               !cuda_failed(cudaMemcpyAsync(&h_bad, bad, sizeof(int), cudaMemcpyDeviceToHost, s), "D2H") &&
               !cuda_failed(cudaStreamSynchronize(s), "synchronize");
    }
    dev_free(bad, s);
    if (good && h_bad) {
        set_error(TP_ERR_ARG, "orion query: a row index is outside [0, %lld)", cw_len);
        return false;
    }
    return good;
}

bool query_rows_async(const ulonglong2* rows, long long cw_len, const long long* q, int count, ulonglong2* out,
                      int* bad, cudaStream_t s)
{
    query_async_kernel<<<count, 128, 0, s>>>(rows, cw_len, q, count, out, bad);
    return ok("orion query");
}

bool answer(const ulonglong2* combined, const ulonglong2* r1, long long n, ulonglong2* out, cudaStream_t s)
{
    const long long blocks = (n + 256 * kAnswerPer - 1) / (256 * kAnswerPer);
    fp2* part = static_cast<fp2*>(dev_alloc(sizeof(fp2) * (size_t)blocks + 256, s));
    if (!part) return false;
    unsigned* ticket = reinterpret_cast<unsigned*>(part + blocks);
    bool good = !cuda_failed(cudaMemsetAsync(ticket, 0, sizeof(unsigned), s), "orion answer ticket");
    if (good) {
        answer_kernel<<<(unsigned)blocks, 256, 0, s>>>(combined, r1, n, part, ticket, out);
        good = ok("orion answer");
    }
    dev_free(part, s);
    return good;
}

}  // namespace orion
}  // namespace tp
