// Fp2 NTT passes (see ntt.h for the decomposition).
#include <map>
#include <mutex>
#include <tuple>
#include <vector>

#include "ntt.h"
#include "runtime.h"

namespace tp {
namespace ntt {

namespace {

thread_local int g_launches = 0;

constexpr int kThreads = 256;
constexpr int kMaxLogR = 10;
constexpr int kTileElems = 4096;   // R * G elements staged per CTA (64 KB)

// w^t (t < 2^h) and w^(t 2^h) (t < n / 2^h) of one transform size and direction
struct Tables {
    fp2* lo = nullptr;
    fp2* hi = nullptr;
    int h = 0;
};

std::mutex g_mu;
std::map<std::tuple<int, int, int>, Tables> g_tables;   // (device, log n, inverse)
bool g_attr_set[64] = {};

struct Pass {
    int log_r, log_g, logn, log_s;
    int first, last;
    long long in_len, in_step;        // first pass: elements present, read stride
    long long src_batch, dst_batch;   // element strides between transforms
    u64 scale;                        // last pass: multiply by this base-field scalar (0: none)
    int n_dig;                        // last pass: the earlier digits
    int dig_bits[3];
    int dig_shift[3];
};

__device__ __forceinline__ fp2 ld_fe(const ulonglong2* p) { const ulonglong2 v = *p; return mk(v.y, v.x); }
__device__ __forceinline__ void st_fe(ulonglong2* p, fp2 a) { *p = make_ulonglong2(a.im, a.re); }

__device__ __forceinline__ fp2 tw_pow(const fp2* __restrict__ lo, const fp2* __restrict__ hi, int h, u32 e)
{
    const u32 l = e & ((1u << h) - 1), q = e >> h;
    if (l == 0) return hi[q];
    return q ? l2mul(lo[l], hi[q]) : lo[l];
}

__device__ __forceinline__ int bitrev(int j, int bits) { return bits ? (int)(__brev((unsigned)j) >> (32 - bits)) : 0; }

// Shared-memory slot of row r, column c: rows of G columns, one element of
// padding every 8 rows so that the 8-row groups of the first stage group land in
// distinct banks.
__device__ __forceinline__ int at(int r, int c, int log_g) { return (r << log_g) + c + (r >> 3); }

// ---- a stage group in registers ---------------------------------------------------
// K consecutive radix-2 stages lh0 .. lh0 + K - 1: a work item is one column and the
// 2^K rows base + m 2^lh0 (m < 2^K) that these stages combine. Their twiddles are
// w_(2^(lh0+j+1))^lo for the stage times a power of the 2^(j+1)-th root; the first
// factor is taken out of the butterflies: row m is multiplied by T^rev(m), T =
// w_(2^(lh0+K))^lo, up front (7 multiplications for 8 rows, none in the first group,
// where lo = 0), and what is left is a plain 2^K-point DFT. Up to 8 points that needs
// no multiplication in this field: the 4th root is -i (forward; +i inverse) and the
// 8th 2^30 (1 -+ i), since 2^61 = 1 makes 2^30 = 2^(-31) a square root of 1/2, so
// they are swaps, negations and rotations by 30 bits. (With 12 multiplications per 8
// rows and group, two in the first, 2^20 points forward and inverse took 196 us, now 165.)
//
// Bounds: rows come in below 2^61 + 8. The first two levels are left unreduced
// (differences add 2p, then 4p, and stay below 2^64), folded, and the third level's
// sums folded again.

// a + w b and a - w b, w = the 4th root; b below 4 p
template <bool INV>
__device__ __forceinline__ void quarter_pair(fp2 a, fp2 b, fp2& sum, fp2& diff)
{
    const fp2 u = mk(a.re + b.im, a.im + (4 * P61 - b.re));   // a - i b
    const fp2 v = mk(a.re + (4 * P61 - b.im), a.im + b.re);   // a + i b
    sum = INV ? v : u;
    diff = INV ? u : v;
}
__device__ __forceinline__ fp2 fold2(fp2 a) { return mk(fold61(a.re), fold61(a.im)); }
__device__ __forceinline__ u64 rot30(u64 x) { return ((x << 30) & P61) + (x >> 31); }   // x < 2^63 -> < 2^61 + 2^32
// y w8 and y w8^3 for y below 2^61 + 8
template <bool INV>
__device__ __forceinline__ fp2 times_w8(fp2 y)
{
    const u64 s = y.re + y.im, d = y.re + (2 * P61 - y.im), e = y.im + (2 * P61 - y.re);
    return INV ? mk(rot30(d), rot30(s)) : mk(rot30(s), rot30(e));
}
template <bool INV>
__device__ __forceinline__ fp2 times_w8_3(fp2 y)
{
    const u64 s = y.re + y.im, n = 4 * P61 - s, d = y.re + (2 * P61 - y.im), e = y.im + (2 * P61 - y.re);
    return INV ? mk(rot30(n), rot30(d)) : mk(rot30(e), rot30(n));
}

// the 2^K-point DFT of x (rows in bit-reversed order, results in natural order);
// rows below 2^61 + 8 in and out
template <int K, bool INV>
__device__ __forceinline__ void dft_rows(fp2 (&x)[1 << K])
{
    constexpr int N = 1 << K;
#pragma unroll
    for (int m = 0; m < N; m += 2) {
        const fp2 a = x[m], b = x[m + 1];
        x[m] = mk(a.re + b.re, a.im + b.im);                                   // < 2^62 + 16
        x[m + 1] = mk(a.re + (2 * P61 - b.re), a.im + (2 * P61 - b.im));       // < 3 2^61 + 8
    }
    if (K >= 2) {
#pragma unroll
        for (int m = 0; m < N; m += 4) {
            const fp2 a = x[m], b = x[m + 2], c = x[m + 1], d = x[m + 3];
            x[m] = mk(a.re + b.re, a.im + b.im);
            x[m + 2] = mk(a.re + (4 * P61 - b.re), a.im + (4 * P61 - b.im));   // < 2^64
            quarter_pair<INV>(c, d, x[m + 1], x[m + 3]);
        }
    }
#pragma unroll
    for (int m = 0; m < N; ++m) x[m] = fold2(x[m]);
    if (K >= 3) {
        const fp2 y1 = times_w8<INV>(x[(5) & (N - 1)]), y3 = times_w8_3<INV>(x[(7) & (N - 1)]);
        const fp2 y0 = x[4 & (N - 1)], y2 = x[6 & (N - 1)], a0 = x[0], a1 = x[1], a2 = x[2 & (N - 1)],
                  a3 = x[3 & (N - 1)];
        auto sum = [](fp2 a, fp2 b) { return fold2(mk(a.re + b.re, a.im + b.im)); };
        auto dif = [](fp2 a, fp2 b) { return fold2(mk(a.re + (4 * P61 - b.re), a.im + (4 * P61 - b.im))); };
        x[0] = sum(a0, y0);
        x[4 & (N - 1)] = dif(a0, y0);
        x[1] = sum(a1, y1);
        x[5 & (N - 1)] = dif(a1, y1);
        fp2 s, d;
        quarter_pair<INV>(a2, y2, s, d);
        x[2 & (N - 1)] = fold2(s);
        x[6 & (N - 1)] = fold2(d);
        x[3 & (N - 1)] = sum(a3, y3);
        x[7 & (N - 1)] = dif(a3, y3);
    }
}

template <int K, bool FIRST, bool INV>
__device__ __forceinline__ void stage_group(fp2* sm, const fp2* tws, int log_r, int log_g, int lh0)
{
    const int G = 1 << log_g, half = 1 << (log_r - 1);
    const int items = ((1 << log_r) >> K) << log_g;
    for (int it = threadIdx.x; it < items; it += kThreads) {
        const int c = it & (G - 1);
        const int q = it >> log_g;
        const int lo = FIRST ? 0 : (q & ((1 << lh0) - 1));
        const int sh = FIRST ? 0 : lh0;
        const int base = ((q >> sh) << (sh + K)) + lo;
        fp2 x[1 << K];
#pragma unroll
        for (int m = 0; m < (1 << K); ++m) {
            x[m] = sm[at(base + (m << sh), c, log_g)];
            if (!FIRST && m) {
                const int e = K == 1 ? 1 : K == 2 ? ((m & 1) << 1) | (m >> 1) : ((m & 1) << 2) | (m & 2) | (m >> 2);
                const int idx = (lo * e) << (log_r - lh0 - K);
                fp2 w = tws[idx & (half - 1)];
                if (e > (1 << K) / 2 && idx >= half) w = mk(P61 - w.re, P61 - w.im);   // w^(R/2) = -1
                x[m] = l2mul(w, x[m]);
            }
        }
        dft_rows<K, INV>(x);
#pragma unroll
        for (int m = 0; m < (1 << K); ++m) sm[at(base + (m << sh), c, log_g)] = x[m];
    }
}

// One pass: a CTA transforms G = 2^log_g columns of R = 2^log_r elements.
// src and dst may be the same buffer (in-place middle pass): every CTA reads its
// own columns completely before it writes them, and no other CTA touches them.
template <bool INV>
__global__ void __launch_bounds__(kThreads, 4) pass_kernel(const ulonglong2* src, ulonglong2* dst, Pass p,
                                                        const fp2* __restrict__ lo,
                                                        const fp2* __restrict__ hi, int h)
{
    extern __shared__ fp2 sm[];
    const int R = 1 << p.log_r, G = 1 << p.log_g;
    fp2* tws = sm + (R << p.log_g) + (R >> 3) + 1;
    const int tid = threadIdx.x;
    src += (long long)blockIdx.y * p.src_batch;
    dst += (long long)blockIdx.y * p.dst_batch;
    // every element index of a transform (2^28 points at most) fits 32 bits
    __shared__ u32 s_base[16];

    // twiddles of the R-point DFT: w_R^t = w_n^(t n / R), t < R / 2
    for (int t = tid; t < R / 2; t += kThreads) tws[t] = tw_pow(lo, hi, h, (u32)t << (p.logn - p.log_r));

    // columns of this CTA
    u32 col_base = 0, s0 = 0;
    const u32 c0 = blockIdx.x << p.log_g;
    if (!p.last) {
        const int lg = p.log_s - p.log_g;   // column groups per outer index
        s0 = (blockIdx.x & ((1u << lg) - 1)) << p.log_g;
        col_base = ((blockIdx.x >> lg) << (p.log_r + p.log_s)) + s0;
    } else {
        if (tid < G) {   // where the column's row starts: its index, digits reversed
            const u32 cc = c0 + tid;
            u32 base = 0;
            int sh = 0;
            for (int t = 0; t < p.n_dig; ++t) {
                base += ((cc >> sh) & ((1u << p.dig_bits[t]) - 1)) << p.dig_shift[t];
                sh += p.dig_bits[t];
            }
            s_base[tid] = base;
        }
        __syncthreads();
    }

    // load (bit-reversed into shared memory), four elements' loads before their stores
    const int tile = R << p.log_g;
    const u32 in_len = (u32)p.in_len, in_step = (u32)p.in_step;
    for (int i0 = tid; i0 < tile; i0 += 4 * kThreads) {
        fp2 v[4];
        int slot[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int idx = i0 + q * kThreads;
            slot[q] = -1;
            if (idx >= tile) continue;
            int c, j;
            u32 pos;
            if (!p.last) {
                // fewer than eight columns: the lanes of a quarter warp that share a column
                // take elements whose bit-reversed rows are neighbours, not R / 2 apart
                c = idx & (G - 1);
                j = idx >> p.log_g;
                if (p.log_g < 3 && p.log_r >= 3) {
                    const int b = 3 - p.log_g;
                    j = ((j & ((1 << b) - 1)) << (p.log_r - b)) | (j >> b);
                }
                pos = col_base + c + ((u32)j << p.log_s);
            } else {
                // the element of the column: for R >= 2^6, the three lowest lane bits
                // become bits log_r - 6 .. log_r - 4 of j, so that the eight threads of
                // a quarter warp write rows bitrev(j) whose bits 3..5 differ (eight
                // distinct bank groups of the padded tile) while every 64 bytes of
                // the row are still read by four neighbouring lanes
                const int u = idx & (R - 1);
                const int at_bit = p.log_r - 6;
                const int hi = u >> 3;
                j = at_bit < 0 ? u
                               : (hi & ((1 << at_bit) - 1)) | ((u & 7) << at_bit) | ((hi >> at_bit) << (at_bit + 3));
                c = idx >> p.log_r;
                pos = s_base[c] + j;
            }
            if (p.first)
                v[q] = pos < in_len ? ld_fe(src + pos * in_step) : f2zero();
            else
                v[q] = ld_fe(src + pos);
            slot[q] = at(bitrev(j, p.log_r), c, p.log_g);
        }
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if (slot[q] >= 0) sm[slot[q]] = v[q];
    }
    __syncthreads();

    // radix-2 stages in register groups of three (natural-order output)
    for (int lh0 = 0; lh0 < p.log_r; lh0 += 3) {
        const int k = min(3, p.log_r - lh0);
        if (lh0 == 0) {
            if (k == 3) stage_group<3, true, INV>(sm, tws, p.log_r, p.log_g, 0);
            else if (k == 2) stage_group<2, true, INV>(sm, tws, p.log_r, p.log_g, 0);
            else stage_group<1, true, INV>(sm, tws, p.log_r, p.log_g, 0);
        } else {
            if (k == 3) stage_group<3, false, INV>(sm, tws, p.log_r, p.log_g, lh0);
            else if (k == 2) stage_group<2, false, INV>(sm, tws, p.log_r, p.log_g, lh0);
            else stage_group<1, false, INV>(sm, tws, p.log_r, p.log_g, lh0);
        }
        __syncthreads();
    }

    // store
    for (int idx = tid; idx < tile; idx += kThreads) {
        const int c = idx & (G - 1);
        const int k = idx >> p.log_g;
        fp2 val = sm[at(k, c, p.log_g)];
        if (!p.last) {
            // w_{R S}^(k s) = w_n^((k s mod R S) n / (R S))
            const u32 e = (((u32)k * (s0 + c)) & ((1u << (p.log_r + p.log_s)) - 1)) << (p.logn - p.log_r - p.log_s);
            if (e) val = l2mul(val, tw_pow(lo, hi, h, e));
            st_fe(dst + (col_base + c + ((u32)k << p.log_s)), val);
        } else {
            if (p.scale) val = mk(lmul(val.re, p.scale), lmul(val.im, p.scale));
            st_fe(dst + (c0 + c + ((u32)k << (p.logn - p.log_r))), l2canon(val));
        }
    }
}

fp2 f2pow(fp2 a, unsigned long long e)
{
    fp2 r = mk(1, 0);
    while (e) {
        if (e & 1) r = f2mul(r, a);
        a = f2mul(a, a);
        e >>= 1;
    }
    return r;
}

int ilog2(long long n)
{
    int k = 0;
    while ((1LL << k) < n) ++k;
    return k;
}

bool is_pow2(long long n) { return n > 0 && (n & (n - 1)) == 0; }

const Tables* tables(int logn, bool inv)
{
    Ctx* c = ctx();
    if (!c) return nullptr;
    std::lock_guard<std::mutex> lk(g_mu);
    auto key = std::make_tuple(c->device, logn, inv ? 1 : 0);
    auto it = g_tables.find(key);
    if (it != g_tables.end()) return &it->second;
    fp2 w = root_of_unity(logn);
    if (inv) w = f2pow(w, (1ull << logn) - 1);
    Tables t;
    t.h = (logn + 1) / 2;
    const size_t nlo = (size_t)1 << t.h, nhi = (size_t)1 << (logn - t.h);
    std::vector<fp2> lo(nlo), hi(nhi);
    lo[0] = mk(1, 0);
    for (size_t i = 1; i < nlo; ++i) lo[i] = f2mul(lo[i - 1], w);
    const fp2 step = nlo < ((size_t)1 << logn) ? f2mul(lo[nlo - 1], w) : mk(1, 0);   // w^(2^h)
    hi[0] = mk(1, 0);
    for (size_t i = 1; i < nhi; ++i) hi[i] = f2mul(hi[i - 1], step);
    if (cuda_failed(cudaMalloc(&t.lo, sizeof(fp2) * nlo), "ntt twiddle alloc") ||
        cuda_failed(cudaMalloc(&t.hi, sizeof(fp2) * nhi), "ntt twiddle alloc") ||
        cuda_failed(cudaMemcpy(t.lo, lo.data(), sizeof(fp2) * nlo, cudaMemcpyHostToDevice), "ntt twiddle upload") ||
        cuda_failed(cudaMemcpy(t.hi, hi.data(), sizeof(fp2) * nhi, cudaMemcpyHostToDevice), "ntt twiddle upload")) {
        cudaFree(t.lo);
        cudaFree(t.hi);
        return nullptr;
    }
    return &(g_tables[key] = t);
}

// digit split of a 2^logn transform: at most 10 bits per pass
// digit split of a 2^logn transform: at most 10 bits per pass, as even as
// possible -- unless the autotuner stored a measured choice for this device
std::map<std::pair<int, int>, std::vector<int>> g_plans;   // (device, log n) -> digits

std::vector<int> default_split(int logn)
{
    const int P = logn <= kMaxLogR ? 1 : (logn + kMaxLogR - 1) / kMaxLogR;
    std::vector<int> d(P, logn / P);
    for (int i = 0; i < logn % P; ++i) d[i]++;
    return d;
}

std::vector<int> split(int logn)
{
    Ctx* c = ctx();
    if (c) {
        std::lock_guard<std::mutex> lk(g_mu);
        auto it = g_plans.find(std::make_pair(c->device, logn));
        if (it != g_plans.end()) return it->second;
    }
    return default_split(logn);
}

// every split of logn into `parts` digits of 3..10 bits
void splits_of(int logn, int parts, std::vector<int>& cur, std::vector<std::vector<int>>& out)
{
    if (parts == 0) {
        if (logn == 0) out.push_back(cur);
        return;
    }
    for (int b = 3; b <= kMaxLogR && b <= logn; ++b) {
        cur.push_back(b);
        splits_of(logn - b, parts - 1, cur, out);
        cur.pop_back();
    }
}

// n-point DFT (direction by tables) of the first-pass input `in`
bool run(const ulonglong2* in, long long in_len, long long in_step, int logn, bool inv, ulonglong2* out,
         int batch, long long in_batch, long long out_batch, ulonglong2* scratch, u64 scale, cudaStream_t s)
{
    const Tables* tb = tables(logn, inv);
    if (!tb) return false;
    Ctx* c = ctx();
    if (c->device >= 0 && c->device < 64 && !g_attr_set[c->device]) {
        const int most = (kTileElems + kTileElems / 8 + 1 + (1 << kMaxLogR) / 2) * (int)sizeof(fp2);
        for (auto k : {pass_kernel<false>, pass_kernel<true>})
            if (cuda_failed(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, most),
                            "ntt smem attribute"))
                return false;
        g_attr_set[c->device] = true;
    }
    const std::vector<int> d = split(logn);
    const int P = (int)d.size();
    const long long n = 1LL << logn;
    ulonglong2* tmp = scratch;
    bool own = false;
    if (P > 1 && !tmp) {
        tmp = static_cast<ulonglong2*>(dev_alloc(sizeof(ulonglong2) * (size_t)n * batch, s));
        if (!tmp) return false;
        own = true;
    }
    bool ok = true;
    int rest = logn;
    for (int t = 0; t < P && ok; ++t) {
        Pass p = {};
        p.log_r = d[t];
        p.logn = logn;
        rest -= d[t];
        p.log_s = rest;
        p.first = t == 0;
        p.last = t == P - 1;
        p.in_len = in_len;
        p.in_step = in_step;
        p.scale = p.last ? scale : 0;
        const ulonglong2* src = t == 0 ? in : tmp;
        ulonglong2* dst = p.last ? out : tmp;
        p.src_batch = t == 0 ? in_batch : n;
        p.dst_batch = p.last ? out_batch : n;
        int log_g = ilog2(kTileElems) - p.log_r;
        if (log_g > 4) log_g = 4;
        if (!p.last && log_g > p.log_s) log_g = p.log_s;
        if (p.last && log_g > logn - p.log_r) log_g = logn - p.log_r;
        // Columns per CTA: sixteen (a tile of 4,096 elements at most), halved down to two
        // (32-byte runs in memory) while there are fewer CTAs than SMs, or fewer than
        // four an SM and the tile stays at 2,048 elements (a row group per thread).
        // 2^16 points 53 -> 18 us (16 -> 128 CTAs a pass), 2^18 59 -> 27, 2^20 85 -> 77;
        // 64 transforms of 2^12 points, 256 CTAs of 1,024 elements, stay (24.7 us
        // against 30.9 with four columns).
        auto ctas_of = [&](int g) { return (n >> (p.log_r + g)) * batch; };
        while (log_g > 1 && (ctas_of(log_g) < c->n_sm ||
                             (ctas_of(log_g) < 4LL * c->n_sm && p.log_r + log_g - 1 >= 11)))
            --log_g;
        p.log_g = log_g;
        if (p.last) {
            p.n_dig = P - 1;
            int shift = logn;
            for (int u = 0; u < P - 1; ++u) {
                shift -= d[u];
                p.dig_bits[u] = d[u];
                p.dig_shift[u] = shift;
            }
        }
        const long long ctas = n >> (p.log_r + p.log_g);
        const size_t smem = sizeof(fp2) * (((size_t)1 << (p.log_r + p.log_g)) + ((size_t)1 << p.log_r) / 8 + 1 +
                                           ((size_t)1 << p.log_r) / 2);
        auto kernel = inv ? pass_kernel<true> : pass_kernel<false>;
        kernel<<<dim3((unsigned)ctas, (unsigned)batch), kThreads, smem, s>>>(src, dst, p, tb->lo, tb->hi, tb->h);
        ++g_launches;
        ok = !cuda_failed(cudaGetLastError(), "ntt pass");
    }
    if (own) dev_free(tmp, s);
    return ok;
}

bool check_sizes(long long m, long long n, int batch, const char* who)
{
    if (!is_pow2(m) || !is_pow2(n) || m > n || n > (1LL << kMaxLog) || batch < 1 || batch > 65535) {
        set_error(TP_ERR_ARG, "%s: need powers of two coef_len %lld <= order %lld <= 2^%d, batch %d", who, m, n,
                  kMaxLog, batch);
        return false;
    }
    return true;
}

}  // namespace

fp2 root_of_unity(int lg)
{
    fp2 g = mk(2147483648ull, 1033321771269002680ull);
    for (int i = 0; i < 62 - lg; ++i) g = f2mul(g, g);
    return g;
}

int passes(long long n) { return (int)split(ilog2(n)).size(); }

bool power_tables(int logn, bool inverse, const fp2** lo, const fp2** hi, int* h)
{
    const Tables* t = tables(logn, inverse);
    if (!t) return false;
    *lo = t->lo;
    *hi = t->hi;
    *h = t->h;
    return true;
}

bool autotune(int logn, int batch, std::vector<int>& best, float* best_ms)
{
    Ctx* c = ctx();
    if (!c) return false;
    if (logn < 1 || logn > kMaxLog || batch < 1 || batch > 65535) {
        set_error(TP_ERR_ARG, "ntt autotune: log n %d or batch %d out of range", logn, batch);
        return false;
    }
    std::vector<std::vector<int>> cands;
    std::vector<int> cur;
    const int p0 = (int)default_split(logn).size();
    for (int parts = p0; parts <= std::min(p0 + 1, 3); ++parts) splits_of(logn, parts, cur, cands);
    if (cands.empty()) cands.push_back(default_split(logn));
    const size_t n = (size_t)1 << logn;
    cudaStream_t s = c->stream;
    ulonglong2* buf = static_cast<ulonglong2*>(dev_alloc(sizeof(ulonglong2) * n * batch * 3, s));
    if (!buf) return false;
    ulonglong2 *in = buf, *out = buf + n * batch, *tmp = buf + 2 * n * batch;
    bool ok = !cuda_failed(cudaMemsetAsync(in, 0, sizeof(ulonglong2) * n * batch, s), "ntt autotune input");
    cudaEvent_t e0, e1;
    ok = ok && !cuda_failed(cudaEventCreate(&e0), "event") && !cuda_failed(cudaEventCreate(&e1), "event");
    float bt = 1e30f;
    const auto key = std::make_pair(c->device, logn);
    for (const auto& d : cands) {
        if (!ok) break;
        {
            std::lock_guard<std::mutex> lk(g_mu);
            g_plans[key] = d;
        }
        for (int r = 0; r < 2 && ok; ++r)
            ok = run(in, n, 1, logn, false, out, batch, n, n, tmp, 0, s);
        ok = ok && !cuda_failed(cudaEventRecord(e0, s), "event");
        for (int r = 0; r < 5 && ok; ++r) ok = run(in, n, 1, logn, false, out, batch, n, n, tmp, 0, s);
        ok = ok && !cuda_failed(cudaEventRecord(e1, s), "event") && !cuda_failed(cudaEventSynchronize(e1), "event");
        float ms = 0.f;
        ok = ok && !cuda_failed(cudaEventElapsedTime(&ms, e0, e1), "event");
        if (ok && ms / 5 < bt) {
            bt = ms / 5;
            best = d;
        }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    dev_free(buf, s);
    std::lock_guard<std::mutex> lk(g_mu);
    if (ok && !best.empty()) g_plans[key] = best;
    else g_plans.erase(key);
    if (best_ms) *best_ms = bt;
    return ok;
}

int last_launches() { return g_launches; }

bool forward(const ulonglong2* in, long long m, long long n, ulonglong2* out, int batch, long long in_batch,
             long long out_batch, ulonglong2* scratch, cudaStream_t s)
{
    g_launches = 0;
    if (!check_sizes(m, n, batch, "fft")) return false;
    return run(in, m, 1, ilog2(n), false, out, batch, in_batch, out_batch, scratch, 0, s);
}

bool inverse(const ulonglong2* in, long long m, long long n, ulonglong2* out, int batch, long long in_batch,
             long long out_batch, ulonglong2* scratch, cudaStream_t s)
{
    g_launches = 0;
    if (!check_sizes(m, n, batch, "ifft")) return false;
    const int lm = ilog2(m);
    const u64 inv_m = lm ? (1ull << (61 - lm)) : 1ull;   // 2^-lm = 2^(61 - lm) mod 2^61 - 1
    return run(in, m, n / m, lm, true, out, batch, in_batch, out_batch, scratch, inv_m, s);
}

}  // namespace ntt
}  // namespace tp
