// Fiat-Shamir transcript in the binary format of the reference prover
// (TruePix-main/libTruePix/fiatshamir.py): one running SHA-256 over everything
// absorbed, challenges drawn from digests of the running state.
//
//   init:        "TruePix," || protocol || "," || "binhash1,"          (:70-74)
//   put(list of u64 ints):  0x01 || LE32(count) || LE64 each          (:112-120)
//   put(Fp2):               0x03 || LE64(real) || LE64(imag)          (:129-131)
//   put(str):               0x04 || LE32(byte length) || UTF-8 bytes  (:132-136)
//   put(int inside a mixed list): 0x02 || LE64;  put(None): 0x05    (:126-138)
//   rand_scalar: absorb [rnum] (a one-int list), rnum += 1, take the low 61
//                bits of the digest read as a big-endian integer, again while
//                the value is >= p (:141-148)
//   rand_ext(label): "ext", label, "real" -> rand_scalar; "ext", label,
//                "imag" -> rand_scalar (:150-162)
//
// The state is a plain struct (the SHA-256 chaining words, the pending partial
// block, the byte count and the challenge counter), so it can move between host
// and device memory by a copy; host and device share the code.
#pragma once
#include <stdint.h>

#include "fp2.cuh"
#include "sha256.cuh"

namespace tp {
namespace fs {

struct State {
    uint32_t h[8];
    uint64_t unit[8];   // the pending partial block in memory order: byte b in bits 8 (b mod 8) of unit b / 8
    uint64_t total;     // bytes absorbed
    uint64_t rnum;      // rand_scalar's counter
    uint32_t nbuf;      // bytes pending in unit (those behind them are stale)
    uint32_t pad;
};
static_assert(sizeof(State) == 120, "transcript state layout");

// the low k bytes of a unit
TP_HD uint64_t low_bytes(int k) { return ((uint64_t)1 << (8 * k)) - 1; }   // 0 <= k < 8

// Device code runs a transcript on a whole warp: every lane holds the same state
// and does the same work on it, except where a draw lets two lanes close two
// digests side by side (rand_fp2). Lane 0 writes what leaves the warp.
TP_HD bool lead()
{
#ifdef __CUDA_ARCH__
    return (threadIdx.x & 31) == 0;
#else
    return true;
#endif
}

#ifdef __CUDA_ARCH__
// One compression of the 64 bytes in `unit`. Not inlined: a proof's closing steps
// hash in dozens of places, and one copy of the rounds stays in the instruction
// cache.
static __device__ __noinline__ void compress_units(uint32_t* h, const uint64_t* unit)
{
    uint32_t st[8], w[16];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        st[i] = h[i];
        w[2 * i] = sha::bswap32((uint32_t)unit[i]);
        w[2 * i + 1] = sha::bswap32((uint32_t)(unit[i] >> 32));
    }
    sha::compress_compact<true>(st, w, sha::kShaTables.k, sha::AddMad{sha::kShaOne});
#pragma unroll
    for (int i = 0; i < 8; ++i) h[i] = st[i];
}
#else
inline void compress_units(uint32_t* h, const uint64_t* unit)
{
    uint32_t w[16];
    for (int i = 0; i < 8; ++i) {
        w[2 * i] = sha::bswap32((uint32_t)unit[i]);
        w[2 * i + 1] = sha::bswap32((uint32_t)(unit[i] >> 32));
    }
    sha::compress(h, w, sha::AddAlu{});
}
#endif

// The low `bytes` bytes of v (1 <= bytes <= 8), least significant first: one or
// two 8-byte units are updated, not byte by byte (the byte-wise form, its buffer
// indexed dynamically, took ten times as long as the compressions: a committed
// round of a batch 146 us against 13 us here). Bytes behind the pending ones keep
// what they held.
TP_HD void absorb_le(State& s, uint64_t v, int bytes)
{
    const uint64_t all = bytes < 8 ? low_bytes(bytes) : ~(uint64_t)0;
    const int q = (int)(s.nbuf >> 3), r = (int)(s.nbuf & 7);
    const int over = r + bytes - 8;    // bytes for the next unit
    v &= all;
    s.unit[q] = (s.unit[q] & ~(all << (8 * r))) | (v << (8 * r));
    s.total += (uint64_t)bytes;
    s.nbuf += (uint32_t)bytes;
    if (s.nbuf >= 64) {
        compress_units(s.h, s.unit);
        s.nbuf -= 64;
    }
    if (over > 0) {
        uint64_t& next = s.unit[(q + 1) & 7];
        next = (next & ~low_bytes(over)) | (v >> (8 * (8 - r)));
    }
}

// one byte into the running hash
TP_HD void absorb_byte(State& s, uint8_t b) { absorb_le(s, b, 1); }

// bytes from memory (the host entry points' caller-owned data)
TP_HD void absorb(State& s, const uint8_t* p, uint64_t n)
{
    for (uint64_t i = 0; i < n; ++i) absorb_byte(s, p[i]);
}

// A label of at most 32 bytes held by value in four 64-bit words (byte i in
// bits 8 (i mod 8) of word i / 8). Device code builds, passes and absorbs labels
// only in this form: no pointer to a local byte array is handed to the inlined
// hash code (on sm_100a such a pointer, passed down through the fully inlined
// draw, was observed to read the wrong bytes).
struct Label {
    uint64_t w0, w1, w2, w3;
    uint32_t len;
};

TP_HD Label label_empty()
{
    Label L;
    L.w0 = L.w1 = L.w2 = L.w3 = 0;
    L.len = 0;
    return L;
}

// append one byte (ignored past 32)
TP_HD void label_push(Label& L, uint8_t b)
{
    const uint64_t v = (uint64_t)b << (8 * (L.len & 7));
    const uint32_t q = L.len >> 3;
    L.w0 |= q == 0 ? v : 0;
    L.w1 |= q == 1 ? v : 0;
    L.w2 |= q == 2 ? v : 0;
    L.w3 |= q == 3 ? v : 0;
    L.len += q < 4 ? 1 : 0;
}

// a label from a string literal of at most 32 characters
template <int N>
TP_HD Label label_lit(const char (&str)[N])
{
    static_assert(N - 1 <= 32, "labels hold at most 32 bytes");
    Label L = label_empty();
#pragma unroll
    for (int i = 0; i < N - 1; ++i) label_push(L, (uint8_t)str[i]);
    return L;
}

// the decimal digits of v (|v| < 2^31) appended, as Python's str(int) writes them
TP_HD void label_decimal(Label& L, long long v)
{
    if (v < 0) {
        label_push(L, '-');
        v = -v;
    }
    long long p = 1;
    while (p <= v / 10) p *= 10;
    for (; p > 0; p /= 10) {
        label_push(L, (uint8_t)('0' + (v / p) % 10));
    }
}

TP_HD void init(State& s)
{
    sha::init(s.h);
    s.nbuf = 0;
    s.total = 0;
    s.rnum = 0;
    s.pad = 0;
}

// put(list of ints), every value below 2^64 (the reference's array('Q') path)
TP_HD void put_u64s(State& s, const uint64_t* v, uint64_t n)
{
    absorb_byte(s, 0x01);
    absorb_le(s, n, 4);
    for (uint64_t i = 0; i < n; ++i) absorb_le(s, v[i], 8);
}

TP_HD void put_fp2(State& s, uint64_t re, uint64_t im)
{
    absorb_le(s, 0x03 | (re << 8), 8);
    absorb_le(s, (re >> 56) | (im << 8), 8);
    absorb_le(s, im >> 56, 1);
}

TP_HD void put_str(State& s, const uint8_t* p, uint32_t len)
{
    absorb_byte(s, 0x04);
    absorb_le(s, len, 4);
    absorb(s, p, len);
}

// put(str) of a label held by value
TP_HD void put_label(State& s, const Label& L)
{
    absorb_le(s, 0x04 | ((uint64_t)L.len << 8), 5);
    const uint64_t w[4] = {L.w0, L.w1, L.w2, L.w3};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int left = (int)L.len - 8 * i;
        if (left > 0) absorb_le(s, w[i], left < 8 ? left : 8);
    }
}

// The chaining words after the SHA-256 padding: the digest of everything
// absorbed so far. The running state is unchanged.
TP_HD void digest_words(const State& s, uint32_t h[8])
{
    uint64_t u[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        h[i] = s.h[i];
        const int k = (int)s.nbuf - 8 * i;   // pending bytes in this unit and behind it
        u[i] = k >= 8 ? s.unit[i] : k > 0 ? (s.unit[i] & low_bytes(k)) | ((uint64_t)0x80 << (8 * k)) : k == 0 ? 0x80 : 0;
    }
    if (s.nbuf >= 56) {   // no room for the length
        compress_units(h, u);
#pragma unroll
        for (int i = 0; i < 8; ++i) u[i] = 0;
    }
    const uint64_t bits = s.total * 8;   // big-endian in the last eight bytes
    u[7] = ((uint64_t)sha::bswap32((uint32_t)bits) << 32) | sha::bswap32((uint32_t)(bits >> 32));
    compress_units(h, u);
}

// the digest bytes (big-endian words)
TP_HD void digest(const State& s, uint8_t out[32])
{
    uint32_t h[8];
    digest_words(s, h);
    for (int i = 0; i < 8; ++i) {
        out[4 * i] = (uint8_t)(h[i] >> 24);
        out[4 * i + 1] = (uint8_t)(h[i] >> 16);
        out[4 * i + 2] = (uint8_t)(h[i] >> 8);
        out[4 * i + 3] = (uint8_t)h[i];
    }
}

// put([rnum]): a one-int list of the counter, which then moves on
TP_HD void put_counter(State& s)
{
    absorb_le(s, 0x01 | (1ull << 8) | (s.rnum << 40), 8);
    absorb_le(s, s.rnum >> 24, 5);
    s.rnum += 1;
}

// the low 61 bits of the big-endian digest (its last two words)
TP_HD uint64_t draw_bits(const State& s)
{
    uint32_t h[8];
    digest_words(s, h);
    return (((uint64_t)h[6] << 32) | h[7]) & P61;
}

// A draw is redrawn only when its 61 bits are all ones (probability 2^-61); the
// loop is bounded all the same, and past the bound returns the value reduced.
TP_HD uint64_t rand_scalar(State& s)
{
    uint64_t v = 0;
    for (int it = 0; it < 1000; ++it) {
        put_counter(s);
        v = draw_bits(s);
        if (v < P61) return v;
    }
    return v % P61;
}

// rand_ext(label) as an Fp2: "ext", label, "real" -> the real limb; "ext",
// label, "imag" -> the imaginary limb
TP_HD fp2 rand_fp2_serial(State& s, const Label& L)
{
    const Label ext = label_lit("ext"), real = label_lit("real"), imag = label_lit("imag");
    put_label(s, ext);
    put_label(s, L);
    put_label(s, real);
    const uint64_t re = rand_scalar(s);
    put_label(s, ext);
    put_label(s, L);
    put_label(s, imag);
    const uint64_t im = rand_scalar(s);
    return mk(re, im);
}

#ifdef __CUDA_ARCH__
// The same draw on a warp whose lanes hold the same state. The real limb's value
// does not enter the transcript, so the state runs on to the imaginary limb's
// draw at once and the two digests are closed by an even and an odd lane in the
// same instructions. All-ones values (probability 2^-60) redraw one after the other.
static __device__ __noinline__ fp2 rand_fp2(State& s, const Label& L)
{
    State both[2];   // at the real limb's draw, at the imaginary limb's
    const State s0 = s;
    const Label ext = label_lit("ext");
    for (int q = 0; q < 2; ++q) {
        put_label(s, ext);
        put_label(s, L);
        put_label(s, q ? label_lit("imag") : label_lit("real"));
        put_counter(s);
        both[q] = s;
    }
    const uint64_t v = draw_bits(both[threadIdx.x & 1]);
    const uint64_t re = __shfl_sync(0xffffffffu, v, 0), im = __shfl_sync(0xffffffffu, v, 1);
    if (re < P61 && im < P61) return mk(re, im);
    s = s0;
    return rand_fp2_serial(s, L);
}
#else
inline fp2 rand_fp2(State& s, const Label& L) { return rand_fp2_serial(s, L); }
#endif

// the same draw with a label in memory (host entry points: labels of any length)
TP_HD void rand_ext(State& s, const uint8_t* label, uint32_t len, uint64_t* re, uint64_t* im)
{
    const Label ext = label_lit("ext"), real = label_lit("real"), imag = label_lit("imag");
    put_label(s, ext);
    put_str(s, label, len);
    put_label(s, real);
    *re = rand_scalar(s);
    put_label(s, ext);
    put_str(s, label, len);
    put_label(s, imag);
    *im = rand_scalar(s);
}

}  // namespace fs
}  // namespace tp
