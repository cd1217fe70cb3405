// Reed-Solomon commit: batched slice transforms, FRI leaf chains, Merkle tree.
#include "fp2.cuh"
#include "ntt.h"
#include "orion.h"
#include "runtime.h"
#include "sha256.cuh"

namespace tp {
namespace rs {

namespace {

constexpr int kSlices = 64;   // 2^log_slice_number (include/infrastructure/constants.h)

constexpr int kLeafThreads = 128;

__device__ __forceinline__ void store_leaf(unsigned char* tree, long long node, const uint32_t st[8])
{
    uint4 a, b;
    a.x = sha::bswap32(st[0]); a.y = sha::bswap32(st[1]); a.z = sha::bswap32(st[2]); a.w = sha::bswap32(st[3]);
    b.x = sha::bswap32(st[4]); b.y = sha::bswap32(st[5]); b.z = sha::bswap32(st[6]); b.w = sha::bswap32(st[7]);
    uint4* d = reinterpret_cast<uint4*>(tree + node * 32);
    d[0] = a;
    d[1] = b;
}

// The leaf chains of both commit kinds, h <- SHA256(x || y || h) over the 64 slices
// (fri.cpp:96-110, 396-410: the pair first, the running digest second -- the
// opposite order of the Orion row leaves): leaf t's x and y of slice i stand at
// src + t leaf_step + i slice_step and y_off behind it. One thread per leaf; the
// next pair is loaded behind the hash of the present one. Bound by the chain of
// 128 compressions while the leaves give a scheduler at most one warp (up to
// 18,944 of them: CTAs of 128 threads, so that small steps spread over the SMs),
// by the ALU pipe beyond.
__global__ void __launch_bounds__(kLeafThreads) pair_leaf_kernel(const ulonglong2* __restrict__ src,
                                                                 long long n_leaves, long long leaf_step,
                                                                 long long slice_step, long long y_off,
                                                                 unsigned char* __restrict__ tree, uint32_t one)
{
    const long long t = (long long)blockIdx.x * kLeafThreads + threadIdx.x;
    if (t >= n_leaves) return;
    uint32_t st[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) st[i] = 0;
    const ulonglong2* p = src + t * leaf_step;
    ulonglong2 x = __ldg(p), y = __ldg(p + y_off);
#pragma unroll 1
    for (int i = 0; i < kSlices; ++i) {
        uint32_t w[16];
        sha::fe_words(x.x, x.y, w);
        sha::fe_words(y.x, y.y, w + 4);
        if (i + 1 < kSlices) {
            p += slice_step;
            x = __ldg(p);
            y = __ldg(p + y_off);
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) w[8 + k] = st[k];
        sha::hash64(w, st, sha::AddMad{one});
    }
    store_leaf(tree, n_leaves + t, st);
}

// The same chains with a warp for the rounds and a warp for the schedule of 32
// (sha256.cuh, ChainMem).
__global__ void __launch_bounds__(sha::kFewThreads) pair_leaf_few_kernel(const ulonglong2* __restrict__ src,
                                                                         long long n_leaves, long long leaf_step,
                                                                         long long slice_step, long long y_off,
                                                                         unsigned char* __restrict__ tree)
{
    __shared__ sha::ChainMem mem;
    const long long t = (long long)blockIdx.x * sha::kFewRows + (threadIdx.x & 31);
    const ulonglong2* p = src + (t < n_leaves ? t : n_leaves - 1) * leaf_step;
    uint32_t st[8];
    const bool mine = sha::chain_pair<true>(mem, kSlices, st, sha::AddAlu{}, [&](int n, uint32_t w[8]) {
        const ulonglong2 x = __ldg(p + n * slice_step), y = __ldg(p + n * slice_step + y_off);
        sha::fe_words(x.x, x.y, w);
        sha::fe_words(y.x, y.y, w + 4);
    });
    if (mine && t < n_leaves) store_leaf(tree, n_leaves + t, st);
}

bool launch_pair_leaves(const ulonglong2* src, long long n_leaves, long long leaf_step, long long slice_step,
                        long long y_off, unsigned char* tree, const char* what, cudaStream_t s)
{
    Ctx* c = ctx();
    if (!c) return false;
    const long long few = (n_leaves + sha::kFewRows - 1) / sha::kFewRows;
    if (few <= (long long)sha::kFewPerSm * c->n_sm)
        pair_leaf_few_kernel<<<(unsigned)few, sha::kFewThreads, 0, s>>>(src, n_leaves, leaf_step, slice_step, y_off,
                                                                        tree);
    else
        pair_leaf_kernel<<<(unsigned)((n_leaves + kLeafThreads - 1) / kLeafThreads), kLeafThreads, 0, s>>>(
            src, n_leaves, leaf_step, slice_step, y_off, tree, 1u);
    return !cuda_failed(cudaGetLastError(), what);
}

__device__ __forceinline__ fp2 ld_fe(const ulonglong2* p) { const ulonglong2 v = __ldg(p); return mk(v.y, v.x); }

// v[i][j] = 2^-1 ((x + y) + w_M^-i r (x - y)) into the next interleaved witness;
// one thread per (i, j), j fastest: the 64 pairs of a row are 2 KB contiguous.
__global__ void __launch_bounds__(256) fri_fold_kernel(const ulonglong2* __restrict__ w, long long nxt, fp2 r,
                                                       const fp2* __restrict__ lo, const fp2* __restrict__ hi,
                                                       int h, ulonglong2* __restrict__ next)
{
    const long long t = (long long)blockIdx.x * 256 + threadIdx.x;
    if (t >= nxt * kSlices) return;
    const long long i = t >> 6;
    const int j = (int)(t & 63);
    const fp2 x = ld_fe(w + ((i << 7) | (j << 1))), y = ld_fe(w + ((i << 7) | (j << 1) | 1));
    fp2 inv_mu = lo[i & ((1ll << h) - 1)];
    if (i >> h) inv_mu = l2mul(inv_mu, hi[i >> h]);
    const fp2 d = l2sub(x, y);
    const fp2 v = l2mul(mk(1ull << 60, 0), l2add(l2add(x, y), l2mul(l2mul(inv_mu, r), d)));
    const fp2 c = l2canon(v);
    const long long half = nxt >> 1;
    const long long pos = i < half ? ((i << 7) | (j << 1)) : (((i - half) << 7) | (j << 1) | 1);
    next[pos] = make_ulonglong2(c.im, c.re);
}

}  // namespace

bool fri_step(const ulonglong2* w, int log_m, fp2 r, ulonglong2* next, unsigned char* tree, cudaStream_t s)
{
    if (log_m < 2 || log_m > 26) {
        set_error(TP_ERR_ARG, "fri step: log2 of the per-slice witness size %d outside [2, 26]", log_m);
        return false;
    }
    if (r.re >= P61 || r.im >= P61) {
        set_error(TP_ERR_ARG, "fri step: the random is not canonical");
        return false;
    }
    const fp2 *lo, *hi;
    int h;
    if (!ntt::power_tables(log_m, true, &lo, &hi, &h)) return false;
    const long long nxt = 1LL << (log_m - 1), n_leaves = nxt / 2;
    timer_begin(s, 9210);
    fri_fold_kernel<<<(unsigned)((nxt * kSlices + 255) / 256), 256, 0, s>>>(w, nxt, r, lo, hi, h, next);
    timer_end(s);
    if (cuda_failed(cudaGetLastError(), "fri fold")) return false;
    if (cuda_failed(cudaMemsetAsync(tree, 0, 32, s), "fri tree clear")) return false;
    timer_begin(s, 9211);
    // leaf i: the 64 pairs of row i of the interleaved witness
    const bool leaves = launch_pair_leaves(next, n_leaves, 2 * kSlices, 2, 1, tree, "fri leaves", s);
    timer_end(s);
    return leaves && orion::build_tree(tree, n_leaves, s);
}

bool commit(const ulonglong2* src, int log_len, ulonglong2* l_eval, unsigned char* tree, cudaStream_t s)
{
    if (log_len < kMinLog || log_len > kMaxLog) {
        set_error(TP_ERR_ARG, "rs commit: log_len %d outside [%d, %d]", log_len, kMinLog, kMaxLog);
        return false;
    }
    const long long real_cnt = 1LL << (log_len - 6), slice = 1LL << (log_len - 1);
    // the 64 slices' coefficients (2^log_len elements)
    ulonglong2* coef = static_cast<ulonglong2*>(dev_alloc(sizeof(ulonglong2) * (size_t)(real_cnt * kSlices), s));
    if (!coef) return false;
    bool ok = ntt::inverse(src, real_cnt, real_cnt, coef, kSlices, real_cnt, real_cnt, nullptr, s) &&
              ntt::forward(coef, real_cnt, slice, l_eval, kSlices, real_cnt, slice, nullptr, s);
    dev_free(coef, s);
    if (!ok) return false;
    if (cuda_failed(cudaMemsetAsync(tree, 0, 32, s), "rs tree clear")) return false;
    const long long half = slice >> 1;
    return launch_pair_leaves(l_eval, half, 1, slice, half, tree, "rs leaves", s) && orion::build_tree(tree, half, s);
}

}  // namespace rs
}  // namespace tp
