// SHA-256 (FIPS 180-4) of one 64-byte message, the only hash the Orion commit
// path uses (TruePix-main/Orion/Orion_nonzk/include/infrastructure/my_hhash.h:46-54:
// a full SHA-256 of 64 bytes, i.e. the message block plus the fixed padding block).
//
// Digests are kept as eight 32-bit state words (big-endian words of the digest
// bytes). A message block is sixteen big-endian words; the padding block of a
// 64-byte message is a constant, so its expanded schedule is a constant too and
// is folded into the round constants at compile time (no schedule work for the
// second compression). Host and device share the code so that constant leaves
// (the all-zero row chain, SHA-256 of 64 zero bytes) are computed on the host.
#pragma once
#include <cstdint>

namespace tp {
namespace sha {

struct Tables {
    uint32_t k[64];
    uint32_t pad_kw[64];  // k[t] + w[t] of the padding block of a 64-byte message
};

__host__ __device__ constexpr uint32_t rotr_c(uint32_t x, int n) { return (x >> n) | (x << (32 - n)); }

__host__ __device__ constexpr Tables make_tables()
{
    Tables t{};
    const uint32_t k[64] = {
        0x428a2f98u, 0x71374491u, 0xb5c0fbcfu, 0xe9b5dba5u, 0x3956c25bu, 0x59f111f1u, 0x923f82a4u, 0xab1c5ed5u,
        0xd807aa98u, 0x12835b01u, 0x243185beu, 0x550c7dc3u, 0x72be5d74u, 0x80deb1feu, 0x9bdc06a7u, 0xc19bf174u,
        0xe49b69c1u, 0xefbe4786u, 0x0fc19dc6u, 0x240ca1ccu, 0x2de92c6fu, 0x4a7484aau, 0x5cb0a9dcu, 0x76f988dau,
        0x983e5152u, 0xa831c66du, 0xb00327c8u, 0xbf597fc7u, 0xc6e00bf3u, 0xd5a79147u, 0x06ca6351u, 0x14292967u,
        0x27b70a85u, 0x2e1b2138u, 0x4d2c6dfcu, 0x53380d13u, 0x650a7354u, 0x766a0abbu, 0x81c2c92eu, 0x92722c85u,
        0xa2bfe8a1u, 0xa81a664bu, 0xc24b8b70u, 0xc76c51a3u, 0xd192e819u, 0xd6990624u, 0xf40e3585u, 0x106aa070u,
        0x19a4c116u, 0x1e376c08u, 0x2748774cu, 0x34b0bcb5u, 0x391c0cb3u, 0x4ed8aa4au, 0x5b9cca4fu, 0x682e6ff3u,
        0x748f82eeu, 0x78a5636fu, 0x84c87814u, 0x8cc70208u, 0x90befffau, 0xa4506cebu, 0xbef9a3f7u, 0xc67178f2u};
    uint32_t w[64] = {};
    w[0] = 0x80000000u;  // 0x80 terminator right after the 64 message bytes
    w[15] = 512u;        // message length in bits
    for (int i = 16; i < 64; ++i) {
        const uint32_t s0 = rotr_c(w[i - 15], 7) ^ rotr_c(w[i - 15], 18) ^ (w[i - 15] >> 3);
        const uint32_t s1 = rotr_c(w[i - 2], 17) ^ rotr_c(w[i - 2], 19) ^ (w[i - 2] >> 10);
        w[i] = w[i - 16] + s0 + w[i - 7] + s1;
    }
    for (int i = 0; i < 64; ++i) {
        t.k[i] = k[i];
        t.pad_kw[i] = k[i] + w[i];
    }
    return t;
}

__host__ __device__ __forceinline__ uint32_t rotr(uint32_t x, int n)
{
#ifdef __CUDA_ARCH__
    return __funnelshift_r(x, x, n);
#else
    return (x >> n) | (x << (32 - n));
#endif
}

__host__ __device__ __forceinline__ uint32_t bswap32(uint32_t x)
{
#ifdef __CUDA_ARCH__
    return __byte_perm(x, 0, 0x0123);
#else
    return __builtin_bswap32(x);
#endif
}

__host__ __device__ __forceinline__ void init(uint32_t st[8])
{
    st[0] = 0x6a09e667u; st[1] = 0xbb67ae85u; st[2] = 0x3c6ef372u; st[3] = 0xa54ff53au;
    st[4] = 0x510e527fu; st[5] = 0x9b05688cu; st[6] = 0x1f83d9abu; st[7] = 0x5be0cd19u;
}

// Additions. On the device the SHA-256 rounds are bound by the integer ALU pipe
// (funnel shifts and LOP3 for the sigma/choice/majority functions); routing the
// additions through the multiply-add pipe as x * one + y, with `one` == 1 known
// only at run time, takes them off that pipe. The host adds directly.
struct AddAlu {
    __host__ __device__ __forceinline__ uint32_t operator()(uint32_t a, uint32_t b) const { return a + b; }
};
struct AddMad {
    uint32_t one;   // 1, passed in at run time
    __host__ __device__ __forceinline__ uint32_t operator()(uint32_t a, uint32_t b) const { return a * one + b; }
};

#define TP_SHA_ROUND(a, b, c, d, e, f, g, h, kw)                                          \
    do {                                                                                  \
        const uint32_t s1 = rotr(e, 6) ^ rotr(e, 11) ^ rotr(e, 25);                       \
        const uint32_t ch = (e & f) ^ (~e & g);                                           \
        const uint32_t t1 = add(add(add(h, s1), ch), (kw));                               \
        const uint32_t s0 = rotr(a, 2) ^ rotr(a, 13) ^ rotr(a, 22);                       \
        const uint32_t mj = (a & b) ^ (a & c) ^ (b & c);                                  \
        d = add(d, t1);                                                                   \
        h = add(t1, add(s0, mj));                                                         \
    } while (0)

// one compression of the message block w[16] into st[8] (w is consumed as the
// rolling schedule)
template <class Add>
__host__ __device__ __forceinline__ void compress(uint32_t st[8], uint32_t w[16], Add add)
{
    constexpr Tables T = make_tables();
    uint32_t a = st[0], b = st[1], c = st[2], d = st[3], e = st[4], f = st[5], g = st[6], h = st[7];
#pragma unroll
    for (int i = 0; i < 64; i += 8) {
        if (i >= 16) {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int t = i + j;
                const uint32_t x = w[(t - 15) & 15], y = w[(t - 2) & 15];
                w[t & 15] = add(add(w[t & 15], rotr(x, 7) ^ rotr(x, 18) ^ (x >> 3)),
                                add(w[(t - 7) & 15], rotr(y, 17) ^ rotr(y, 19) ^ (y >> 10)));
            }
        }
        TP_SHA_ROUND(a, b, c, d, e, f, g, h, add(w[(i + 0) & 15], T.k[i + 0]));
        TP_SHA_ROUND(h, a, b, c, d, e, f, g, add(w[(i + 1) & 15], T.k[i + 1]));
        TP_SHA_ROUND(g, h, a, b, c, d, e, f, add(w[(i + 2) & 15], T.k[i + 2]));
        TP_SHA_ROUND(f, g, h, a, b, c, d, e, add(w[(i + 3) & 15], T.k[i + 3]));
        TP_SHA_ROUND(e, f, g, h, a, b, c, d, add(w[(i + 4) & 15], T.k[i + 4]));
        TP_SHA_ROUND(d, e, f, g, h, a, b, c, add(w[(i + 5) & 15], T.k[i + 5]));
        TP_SHA_ROUND(c, d, e, f, g, h, a, b, add(w[(i + 6) & 15], T.k[i + 6]));
        TP_SHA_ROUND(b, c, d, e, f, g, h, a, add(w[(i + 7) & 15], T.k[i + 7]));
    }
    st[0] = add(st[0], a); st[1] = add(st[1], b); st[2] = add(st[2], c); st[3] = add(st[3], d);
    st[4] = add(st[4], e); st[5] = add(st[5], f); st[6] = add(st[6], g); st[7] = add(st[7], h);
}

// the second compression of a 64-byte message: constant block, constant schedule
template <class Add>
__host__ __device__ __forceinline__ void compress_pad64(uint32_t st[8], Add add)
{
    constexpr Tables T = make_tables();
    uint32_t a = st[0], b = st[1], c = st[2], d = st[3], e = st[4], f = st[5], g = st[6], h = st[7];
#pragma unroll
    for (int i = 0; i < 64; i += 8) {
        TP_SHA_ROUND(a, b, c, d, e, f, g, h, T.pad_kw[i + 0]);
        TP_SHA_ROUND(h, a, b, c, d, e, f, g, T.pad_kw[i + 1]);
        TP_SHA_ROUND(g, h, a, b, c, d, e, f, T.pad_kw[i + 2]);
        TP_SHA_ROUND(f, g, h, a, b, c, d, e, T.pad_kw[i + 3]);
        TP_SHA_ROUND(e, f, g, h, a, b, c, d, T.pad_kw[i + 4]);
        TP_SHA_ROUND(d, e, f, g, h, a, b, c, T.pad_kw[i + 5]);
        TP_SHA_ROUND(c, d, e, f, g, h, a, b, T.pad_kw[i + 6]);
        TP_SHA_ROUND(b, c, d, e, f, g, h, a, T.pad_kw[i + 7]);
    }
    st[0] = add(st[0], a); st[1] = add(st[1], b); st[2] = add(st[2], c); st[3] = add(st[3], d);
    st[4] = add(st[4], e); st[5] = add(st[5], f); st[6] = add(st[6], g); st[7] = add(st[7], h);
}

#ifdef __CUDACC__
// round constants (and the padding block's k + w) for the device's compact form
static __constant__ Tables kShaTables = make_tables();

// One round. The additions are grouped so that behind e only Sigma1 and two of them
// stand before the next e, and behind a Sigma0 and one before the next a; no group
// has more than seven. Cycles a round (average over a message and a padding block)
// at one / two / six warps a scheduler: 38.8 / 67.8 / 194.3; in the order of the
// standard's text 43.3 / 68.8 / 193.1; that order with eight schedule words made in
// front of the eight rounds that use them 50.5 / 69.8 / 192.6. The ALU pipe's own
// bound is 26 a warp (13 instructions a round on 16 lanes).
template <class Add>
__device__ __forceinline__ void round_step(uint32_t a, uint32_t b, uint32_t c, uint32_t& d, uint32_t e, uint32_t f,
                                           uint32_t g, uint32_t& h, uint32_t kw, Add add)
{
    const uint32_t s1 = rotr(e, 6) ^ rotr(e, 11) ^ rotr(e, 25);
    const uint32_t ch = (e & f) ^ (~e & g);
    const uint32_t s0 = rotr(a, 2) ^ rotr(a, 13) ^ rotr(a, 22);
    const uint32_t mj = (a & b) ^ (a & c) ^ (b & c);
    const uint32_t t1 = add(s1, add(ch, add(h, kw)));
    d = add(d, t1);
    h = add(s0, add(mj, t1));
}

// The same on plain additions, three operands to one: behind e only Sigma1 and one of
// them; its 15 instructions a round keep the ALU pipe busy for 30 cycles, and one warp
// alone takes 30.6 (32.1 with the form above, which is ahead from three warps a
// scheduler on: 103 against 105 at four, 145 against 157 at six).
__device__ __forceinline__ void round_step(uint32_t a, uint32_t b, uint32_t c, uint32_t& d, uint32_t e, uint32_t f,
                                           uint32_t g, uint32_t& h, uint32_t kw, AddAlu)
{
    const uint32_t s1 = rotr(e, 6) ^ rotr(e, 11) ^ rotr(e, 25);
    const uint32_t ch = (e & f) ^ (~e & g);
    const uint32_t s0 = rotr(a, 2) ^ rotr(a, 13) ^ rotr(a, 22);
    const uint32_t mj = (a & b) ^ (a & c) ^ (b & c);
    const uint32_t hk = h + kw, dk = d + hk, u = s0 + mj + hk;
    d = s1 + ch + dk;
    h = s1 + ch + u;
}

// Sixteen rounds from round i0 (a multiple of 16); kUpdate: each schedule word is
// replaced by the one sixteen rounds on right behind the round that used it, off
// the chain of the rounds.
template <bool kSched, bool kUpdate, class Add>
__device__ __forceinline__ void sixteen_rounds(uint32_t s[8], uint32_t w[16], const uint32_t* K, Add add)
{
#pragma unroll
    for (int t = 0; t < 16; ++t) {
        const uint32_t kw = kSched ? add(w[t], K[t]) : K[t];
        round_step(s[(0 - t) & 7], s[(1 - t) & 7], s[(2 - t) & 7], s[(3 - t) & 7], s[(4 - t) & 7], s[(5 - t) & 7],
                   s[(6 - t) & 7], s[(7 - t) & 7], kw, add);
        if (kSched && kUpdate) {
            const uint32_t x = w[(t + 1) & 15], y = w[(t + 14) & 15];
            w[t] = add(rotr(y, 17) ^ rotr(y, 19) ^ (y >> 10),
                       add(rotr(x, 7) ^ rotr(x, 18) ^ (x >> 3), add(w[t], w[(t + 9) & 15])));
        }
    }
}

// One compression in compact form: a 16-round body looped (the schedule's rolling
// index and the round variables' rotation repeat every 16 rounds, so the body
// indexes registers statically) with the round constants read from constant
// memory, and for a message block the last 16 rounds, which make no schedule
// words, behind it. Less than half of the fully unrolled code: the leaf and tree
// kernels, which keep one hash in flight per thread, run from the instruction
// cache instead of streaming ~40 KB of straight-line code per hash (65 cycles a
// round at one warp a scheduler, 254 at six in that form).
// kSched: message block w (consumed as the rolling schedule); otherwise the
// constant padding block, K holding its k + w.
template <bool kSched, class Add>
__device__ __forceinline__ void compress_compact(uint32_t st[8], uint32_t w[16], const uint32_t* K, Add add)
{
    uint32_t s[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) s[i] = st[i];
    if (kSched) {
#pragma unroll 1
        for (int i = 0; i < 48; i += 16) sixteen_rounds<true, true>(s, w, K + i, add);
        sixteen_rounds<true, false>(s, w, K + 48, add);
    } else {
#pragma unroll 1
        for (int i = 0; i < 64; i += 16) sixteen_rounds<false, false>(s, w, K + i, add);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) st[i] = add(st[i], s[i]);
}
#endif

// SHA-256 of the 64-byte message given as 16 big-endian words; out = state words
template <class Add = AddAlu>
__host__ __device__ __forceinline__ void hash64(uint32_t w[16], uint32_t out[8], Add add = Add())
{
    init(out);
#ifdef __CUDA_ARCH__
    compress_compact<true>(out, w, kShaTables.k, add);
    compress_compact<false>(out, w, kShaTables.pad_kw, add);
#else
    compress(out, w, add);
    compress_pad64(out, add);
#endif
}

// The message words of a field element (16 bytes: u64 img then u64 real, both
// little-endian, the reference's memory order) -- 4 big-endian words.
__host__ __device__ __forceinline__ void fe_words(uint64_t img, uint64_t real, uint32_t* w)
{
    w[0] = bswap32((uint32_t)img);
    w[1] = bswap32((uint32_t)(img >> 32));
    w[2] = bswap32((uint32_t)real);
    w[3] = bswap32((uint32_t)(real >> 32));
}

#ifdef __CUDACC__
// ---- chains of few rows: a warp for the rounds, a warp for the schedule -------------
// A chain h <- SHA256(...) of 64-byte messages made of the digest h and a pair of
// field elements is serial, and while a scheduler has one warp of rows or less the
// chain's latency is all there is. The schedule shares neither operands nor results
// with the rounds until a word is used, so a second warp makes it: one warp runs
// nothing but rounds, on k + w from shared memory, the other expands the message
// words and loads the next pair. 38.8 cycles a round (averaged over the message and
// the padding block) become 31.
struct ChainMem {
    uint4 h[2][32];          // the running digest, for the schedule
    uint4 pair[2][2][32];    // k + w of the pair's eight words, for the present and the next hash
    uint4 state[2][2][32];   // pair first: the state behind the pair's eight rounds
    uint4 kw[12][32];        // k + w of words 16..63
};

// The pair's named barriers (0 is the CTA's own): the digest is there; words 16..23
// are; 24..39; 40..63; a hash's pair is. At each, one warp only arrives and the
// other waits. None may be shared and the rounds' warp takes kBarPair before it hands
// over the digest: the schedule's warp runs on up to the next digest without waiting,
// so only a digest not yet handed over keeps its next arrival (or its wait for that
// digest, on a shared one) from meeting its last at the same barrier.
enum : int { kBarH = 1, kBarA = 2, kBarB = 3, kBarC = 4, kBarPair = 5 };
__device__ __forceinline__ void bar_arrive(int id)
{
    __threadfence_block();
    asm volatile("bar.arrive %0, 64;" ::"r"(id) : "memory");
}
__device__ __forceinline__ void bar_wait(int id) { asm volatile("bar.sync %0, 64;" ::"r"(id) : "memory"); }

// rounds t0 .. t0 + 7 (t0 a multiple of 8) with k + w in a and b
template <class Add>
__device__ __forceinline__ void eight_rounds(uint32_t s[8], uint4 a, uint4 b, Add add)
{
    const uint32_t kw[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
    for (int t = 0; t < 8; ++t)
        round_step(s[(0 - t) & 7], s[(1 - t) & 7], s[(2 - t) & 7], s[(3 - t) & 7], s[(4 - t) & 7], s[(5 - t) & 7],
                   s[(6 - t) & 7], s[(7 - t) & 7], kw[t], add);
}

// The warp of the rounds: `hashes` hashes from h = 0; st: the digest of the last.
// kPairFirst: messages x || y || h, whose first eight rounds the other warp runs
// ahead; else h || x || y.
template <bool kPairFirst, class Add>
__device__ __forceinline__ void chain_rounds(ChainMem& m, int hashes, uint32_t st[8], Add add)
{
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int i = 0; i < 8; ++i) st[i] = 0;
#pragma unroll 1
    for (int n = 0; n < hashes; ++n) {
        bar_wait(kBarPair);    // this hash's pair, made behind the last padding block's rounds
        m.h[0][lane] = make_uint4(st[0], st[1], st[2], st[3]);
        m.h[1][lane] = make_uint4(st[4], st[5], st[6], st[7]);
        bar_arrive(kBarH);
        const uint32_t* k = kShaTables.k + (kPairFirst ? 8 : 0);
        const uint4 ka = make_uint4(add(st[0], k[0]), add(st[1], k[1]), add(st[2], k[2]), add(st[3], k[3]));
        const uint4 kb = make_uint4(add(st[4], k[4]), add(st[5], k[5]), add(st[6], k[6]), add(st[7], k[7]));
        uint32_t iv[8], s[8];
        init(iv);
        if (kPairFirst) {
            const uint4 a = m.state[n & 1][0][lane], b = m.state[n & 1][1][lane];
            s[0] = a.x; s[1] = a.y; s[2] = a.z; s[3] = a.w;
            s[4] = b.x; s[5] = b.y; s[6] = b.z; s[7] = b.w;
            eight_rounds(s, ka, kb, add);
        } else {
#pragma unroll
            for (int i = 0; i < 8; ++i) s[i] = iv[i];
            eight_rounds(s, ka, kb, add);
            eight_rounds(s, m.pair[n & 1][0][lane], m.pair[n & 1][1][lane], add);
        }
        bar_wait(kBarA);    // words 16..23
        eight_rounds(s, m.kw[0][lane], m.kw[1][lane], add);
        bar_wait(kBarB);    // .. 39
        eight_rounds(s, m.kw[2][lane], m.kw[3][lane], add);
        eight_rounds(s, m.kw[4][lane], m.kw[5][lane], add);
        bar_wait(kBarC);    // .. 63
#pragma unroll 1
        for (int q = 6; q < 12; q += 2) eight_rounds(s, m.kw[q][lane], m.kw[q + 1][lane], add);
#pragma unroll
        for (int i = 0; i < 8; ++i) st[i] = add(iv[i], s[i]);
        compress_compact<false>(st, nullptr, kShaTables.pad_kw, add);
    }
}

// The warp of the schedule. pair(n, x): the eight message words of hash n's pair.
template <bool kPairFirst, class Add, class Pair>
__device__ __forceinline__ void chain_schedule(ChainMem& m, int hashes, Add add, Pair pair)
{
    const int lane = threadIdx.x & 31;
    uint32_t next[8];
    // the next hash's pair: its k + w, or the state behind its eight rounds
    auto place = [&](int n) {
        const uint32_t* k = kShaTables.k + (kPairFirst ? 0 : 8);
        uint32_t kw[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) kw[i] = add(next[i], k[i]);
        const uint4 a = make_uint4(kw[0], kw[1], kw[2], kw[3]), b = make_uint4(kw[4], kw[5], kw[6], kw[7]);
        if (kPairFirst) {
            uint32_t s[8];
            init(s);
            eight_rounds(s, a, b, add);
            m.state[n & 1][0][lane] = make_uint4(s[0], s[1], s[2], s[3]);
            m.state[n & 1][1][lane] = make_uint4(s[4], s[5], s[6], s[7]);
        } else {
            m.pair[n & 1][0][lane] = a;
            m.pair[n & 1][1][lane] = b;
        }
    };
    pair(0, next);
    place(0);
    bar_arrive(kBarPair);
#pragma unroll 1
    for (int n = 0; n < hashes; ++n) {
        uint32_t w[16];
#pragma unroll
        for (int i = 0; i < 8; ++i) w[(kPairFirst ? 0 : 8) + i] = next[i];
        if (n + 1 < hashes) pair(n + 1, next);    // loaded behind this hash's words
        bar_wait(kBarH);
        const uint4 a = m.h[0][lane], b = m.h[1][lane];
        uint32_t* h = w + (kPairFirst ? 8 : 0);
        h[0] = a.x; h[1] = a.y; h[2] = a.z; h[3] = a.w;
        h[4] = b.x; h[5] = b.y; h[6] = b.z; h[7] = b.w;
        // four words from word 16 + 4 q on (registers indexed statically for q mod 4)
        auto four = [&](int q) {
            uint32_t o[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int t = (4 * q + j) & 15;
                const uint32_t x = w[(t + 1) & 15], y = w[(t + 14) & 15];
                w[t] = add(rotr(y, 17) ^ rotr(y, 19) ^ (y >> 10),
                           add(rotr(x, 7) ^ rotr(x, 18) ^ (x >> 3), add(w[t], w[(t + 9) & 15])));
                o[j] = add(w[t], kShaTables.k[16 + 4 * q + j]);
            }
            m.kw[q][lane] = make_uint4(o[0], o[1], o[2], o[3]);
        };
        four(0);
        four(1);
        bar_arrive(kBarA);
        four(2);
        four(3);
        four(4);
        four(5);
        bar_arrive(kBarB);
#pragma unroll
        for (int q = 6; q < 12; ++q) four(q);
        bar_arrive(kBarC);
        if (n + 1 < hashes) {
            place(n + 1);
            bar_arrive(kBarPair);
        }
    }
}

// A CTA of 64 threads: the first warp runs the rounds of 32 chains (their digests on
// its lanes, true is returned there), the second makes their schedules. For launches
// of up to two such CTAs an SM, whose four warps have a scheduler each: 136 us for 64
// hashes against 172 in one warp (146 at 1.7 CTAs an SM). With four pairs an SM, each
// scheduler holding a warp of either kind, the schedule's bursts delay the rounds and
// nothing is gained (168 us), and the two kinds of four CTAs of 64 threads share two
// schedulers (215 us).
constexpr int kFewThreads = 64, kFewRows = 32, kFewPerSm = 2;
template <bool kPairFirst, class Add, class Pair>
__device__ __forceinline__ bool chain_pair(ChainMem& m, int hashes, uint32_t st[8], Add add, Pair pair)
{
    if (threadIdx.x < 32) {
        chain_rounds<kPairFirst>(m, hashes, st, add);
        return true;
    }
    chain_schedule<kPairFirst>(m, hashes, add, pair);
    return false;
}
#endif

}  // namespace sha
}  // namespace tp
