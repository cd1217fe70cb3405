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
// and device memory by a copy. The host, and a device thread that has a transcript to
// itself, append to the state; a warp of the device appends to a stretch in shared
// memory (Writer): two pieces of code with the same bytes, draws and states.
#pragma once
#include <stdint.h>

#include <type_traits>

#include "fp2.cuh"
#include "sha256.cuh"

// A draw below this is taken, one from here on is drawn again (2^-61 of them); tests
// compile with a smaller one.
#ifndef TP_FS_DRAW_BOUND
#define TP_FS_DRAW_BOUND P61
#endif

namespace tp {
namespace fs {

constexpr uint64_t kDrawBound = TP_FS_DRAW_BOUND;

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

// Lane 0 writes what leaves a warp that runs a transcript (Writer below).
TP_HD bool lead()
{
#ifdef __CUDA_ARCH__
    return (threadIdx.x & 31) == 0;
#else
    return true;
#endif
}

// ---- the state's operations (host, or one thread of the device) ------------------

TP_HD void unit_words(uint32_t w[16], const uint64_t* unit)
{
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        w[2 * i] = sha::bswap32((uint32_t)unit[i]);
        w[2 * i + 1] = sha::bswap32((uint32_t)(unit[i] >> 32));
    }
}

#ifdef __CUDACC__
// one copy for all the places that put bytes
static __device__ __noinline__ void compress_units_dev(uint32_t* h, const uint64_t* unit)
{
    uint32_t w[16], st[8];
    unit_words(w, unit);
#pragma unroll
    for (int i = 0; i < 8; ++i) st[i] = h[i];
    sha::compress_compact<true>(st, w, sha::kShaTables.k, sha::AddAlu{});
#pragma unroll
    for (int i = 0; i < 8; ++i) h[i] = st[i];
}
#endif

TP_HD void compress_units(uint32_t* h, const uint64_t* unit)
{
#ifdef __CUDA_ARCH__
    compress_units_dev(h, unit);
#else
    uint32_t w[16];
    unit_words(w, unit);
    sha::compress(h, w, sha::AddAlu{});
#endif
}

// The low `bytes` bytes of v (1 <= bytes <= 8), least significant first. Bytes
// behind the pending ones keep what they held.
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
inline void absorb_byte(State& s, uint8_t b) { absorb_le(s, b, 1); }

// bytes from memory (the host entry points' caller-owned data)
inline void absorb(State& s, const uint8_t* p, uint64_t n)
{
    for (uint64_t i = 0; i < n; ++i) absorb_byte(s, p[i]);
}

// A label of at most 32 bytes held by value in four 64-bit words (byte i in
// bits 8 (i mod 8) of word i / 8): device code builds, passes and absorbs labels
// only in this form.
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
    const uint32_t u = (uint32_t)v;   // 32-bit divisions: a 64-bit one costs the device ten times as much
    uint32_t p = 1;
    while (p <= u / 10) p *= 10;
    for (; p > 0; p /= 10) label_push(L, (uint8_t)('0' + u / p % 10));
}

inline void init(State& s)
{
    sha::init(s.h);
    s.nbuf = 0;
    s.total = 0;
    s.rnum = 0;
    s.pad = 0;
}

// put(list of ints), every value below 2^64 (the reference's array('Q') path)
inline void put_u64s(State& s, const uint64_t* v, uint64_t n)
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

inline void put_str(State& s, const uint8_t* p, uint32_t len)
{
    absorb_byte(s, 0x04);
    absorb_le(s, len, 4);
    absorb(s, p, len);
}

// put(str) of a label held by value
TP_HD void put_label(State& s, const Label& L)
{
    absorb_le(s, 0x04 | ((uint64_t)L.len << 8), 5);
    for (int i = 0; 8 * i < (int)L.len; ++i) {
        const int left = (int)L.len - 8 * i;
        absorb_le(s, i == 0 ? L.w0 : i == 1 ? L.w1 : i == 2 ? L.w2 : L.w3, left < 8 ? left : 8);
    }
}

// The chaining words after the SHA-256 padding: the digest of everything
// absorbed so far. The running state is unchanged.
TP_HD void digest_words(const State& s, uint32_t h[8])
{
    uint64_t u[8];
    for (int i = 0; i < 8; ++i) {
        h[i] = s.h[i];
        const int k = (int)s.nbuf - 8 * i;   // pending bytes in this unit and behind it
        u[i] = k >= 8 ? s.unit[i] : k > 0 ? (s.unit[i] & low_bytes(k)) | ((uint64_t)0x80 << (8 * k)) : k == 0 ? 0x80 : 0;
    }
    if (s.nbuf >= 56) {   // no room for the length
        compress_units(h, u);
        for (int i = 0; i < 8; ++i) u[i] = 0;
    }
    const uint64_t bits = s.total * 8;   // big-endian in the last eight bytes
    u[7] = ((uint64_t)sha::bswap32((uint32_t)bits) << 32) | sha::bswap32((uint32_t)(bits >> 32));
    compress_units(h, u);
}

// the digest bytes (big-endian words)
inline void digest(const State& s, uint8_t out[32])
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
        if (v < kDrawBound) return v;
    }
    return v % P61;
}

// rand_ext(label) as an Fp2: "ext", label, "real" -> the real limb; "ext",
// label, "imag" -> the imaginary limb
TP_HD fp2 rand_fp2(State& s, const Label& L)
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

// the same draw with a label in memory (host entry points: labels of any length)
inline void rand_ext(State& s, const uint8_t* label, uint32_t len, uint64_t* re, uint64_t* im)
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

// ---- a transcript at work ---------------------------------------------------------
// Alone and Writer run a state: opened from it, put to and drawn from, stored back to it.
// Alone is the state itself, on the host or in one thread of the device, and the host's
// form of Writer.
//
// On the device a warp runs Writer: every lane makes the same calls. What is put gathers
// in shared memory (TxMem) without being hashed, a lane writing one byte of it, and a
// draw's own 70 to 134 bytes are written by all lanes at once (a lane that appended
// unit by unit spent a third of a round on that chain, and on fetching its code anew
// each time); a draw hashes the whole stretch at once. The message words of all its
// blocks are known by then, so their schedules are made side by side, one lane per
// block, and the rounds run on k + w from shared memory: about 37 cycles a round (33 in a
// kernel of nothing else) against 49 with the schedule in line. The real limb of a draw does not enter the transcript, so
// the stretch runs on to the imaginary limb's draw and an even and an odd lane close the
// two digests in the same instructions, each with its own padding. Per committed round
// (243 bytes, two draws): ~6 compressions' rounds one after the other and two schedules,
// 10 to 13 thousand cycles a draw by the bytes before it; a launch of one round
// takes 16 us (22 with unit-wise appends; 146 with a thread that appended byte by byte
// and hashed block by block).

constexpr int kTxUnits = 72;     // 8-byte units a stretch may hold (9 blocks)
constexpr int kTxBlocks = 8;     // blocks hashed at once, padding included

struct TxMem {
    uint64_t buf[kTxUnits];      // the stretch, from the pending block's first byte
    uint64_t label[4];           // the draw's label
    uint64_t prev[8];            // the block before it (what a state holds behind its pending bytes)
    uint32_t h[8], h_next[8];    // chaining words in front of the stretch; behind its last whole block
    uint64_t out[2];             // the two digests' low 61 bits
    uint64_t total, rnum;        // a redrawn draw's end
    uint32_t n;
    __align__(16) uint32_t kw[2 * kTxBlocks][68];   // k + w of block b as digest v closes it: row 2 b + v
};

// a state by itself
class Alone {
public:
    TP_HD explicit Alone(const State& state) : s(state) {}
    TP_HD void put_fp2(uint64_t re, uint64_t im) { fs::put_fp2(s, re, im); }
    TP_HD fp2 rand_fp2(const Label& L) { return fs::rand_fp2(s, L); }
    TP_HD void store(State& out) const { out = s; }

protected:
    State s;
};

// whether this thread writes what leaves the one, or the warp, that runs a transcript
template <class Tx>
TP_HD bool writes()
{
    return std::is_same<Tx, Alone>::value || lead();
}

#ifdef __CUDACC__
#ifdef __CUDA_ARCH__
// Hash the stretch's bytes: digest v (the lanes of parity v) closes after its first
// n_v bytes, total_v bytes into the transcript; with close unset only its whole
// blocks are taken. m->h_next: the chaining words behind the whole blocks of n_1.
static __device__ __noinline__ void tx_hash(TxMem* m, uint32_t n0, uint32_t n1, uint64_t total1, bool close)
{
    const uint32_t lane = threadIdx.x & 31, v = lane & 1;
    const int n = (int)(v ? n1 : n0), whole = n >> 6;
    const int blocks = close ? whole + ((n & 63) >= 56 ? 2 : 1) : whole;
    const sha::AddAlu add;
    __syncwarp();
    {
        const int b = (int)(lane >> 1);
        if (b < blocks) {
            uint32_t w[16];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int k = n - 64 * b - 8 * i;   // bytes of this unit and behind it
                uint64_t u = m->buf[8 * min(b, kTxUnits / 8 - 1) + i];
                if (k < 8) u = k > 0 ? (u & low_bytes(k)) | ((uint64_t)0x80 << (8 * k)) : k == 0 ? 0x80 : 0;
                w[2 * i] = sha::bswap32((uint32_t)u);
                w[2 * i + 1] = sha::bswap32((uint32_t)(u >> 32));
            }
            if (close && b == blocks - 1) {
                const uint64_t bits = 8 * (total1 - (n1 - (uint32_t)n));
                w[14] = (uint32_t)(bits >> 32);
                w[15] = (uint32_t)bits;
            }
            uint4* kw = reinterpret_cast<uint4*>(m->kw[lane]);
#pragma unroll 1
            for (int i = 0; i < 64; i += 16) {
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    uint32_t o[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const int t = 4 * q + j;
                        o[j] = add(w[t], sha::kShaTables.k[i + t]);
                        const uint32_t x = w[(t + 1) & 15], y = w[(t + 14) & 15];
                        w[t] = add(sha::rotr(y, 17) ^ sha::rotr(y, 19) ^ (y >> 10),
                                   add(sha::rotr(x, 7) ^ sha::rotr(x, 18) ^ (x >> 3), add(w[t], w[(t + 9) & 15])));
                    }
                    kw[i / 4 + q] = make_uint4(o[0], o[1], o[2], o[3]);
                }
            }
        }
    }
    __syncwarp();
    uint32_t st[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) st[i] = m->h[i];
#pragma unroll 1
    for (int b = 0; b < blocks; ++b) {
        if (b == whole && lane == 1)
#pragma unroll
            for (int i = 0; i < 8; ++i) m->h_next[i] = st[i];
        const uint4* kw = reinterpret_cast<const uint4*>(m->kw[2 * b + v]);
        uint32_t s[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) s[i] = st[i];
        uint4 ka = kw[0], kb = kw[1];
        // eight rounds a pass: 16 are as fast in a small kernel, but this one's other code
        // lies between two calls, and their 7 KB are fetched anew each time
#pragma unroll 1
        for (int i = 2; i <= 16; i += 2) {
            const uint4 x = ka, y = kb;
            ka = kw[i & 15];
            kb = kw[(i & 15) + 1];
            sha::eight_rounds(s, x, y, add);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) st[i] = add(st[i], s[i]);
    }
    if (!close && lane == 1)
#pragma unroll
        for (int i = 0; i < 8; ++i) m->h_next[i] = st[i];
    if (lane < 2) m->out[lane] = (((uint64_t)st[6] << 32) | st[7]) & P61;
    __syncwarp();
}

// the whole blocks of the stretch's n bytes are hashed (m->h_next): the rest to its front
static __device__ __noinline__ void tx_advance(TxMem* m, uint32_t n)
{
    const uint32_t lane = threadIdx.x & 31, whole = n >> 6;
    uint64_t p = 0, u = 0;
    if (whole && lane < 8) {
        p = m->buf[8 * (whole - 1) + lane];
        u = m->buf[8 * whole + lane];
    }
    const uint32_t h = m->h_next[lane & 7];
    __syncwarp();
    if (whole && lane < 8) {
        m->prev[lane] = p;
        m->buf[lane] = u;
        m->h[lane] = h;
    }
    __syncwarp();
}

// One limb of a draw put behind the stretch's n bytes: "ext", the label (in m->label),
// "real" or "imag", [rnum]; 35 + len bytes. No branches: a lane writes one byte of each
// of three pieces.
static __device__ __forceinline__ void tx_draw_bytes(TxMem* m, uint32_t n, uint32_t len, uint64_t rnum, int limb)
{
    const int i = (int)(threadIdx.x & 31);
    uint8_t* to = reinterpret_cast<uint8_t*>(m->buf) + n + i;
    const uint64_t head = i < 8 ? 0x7478650000000304ull : 0x04 | ((uint64_t)len << 8);   // 04, 3, "ext"; 04, len
    if (i < 13) to[0] = (uint8_t)(head >> (8 * (i & 7)));
    to += 13;
    if (i < (int)len) to[0] = reinterpret_cast<const uint8_t*>(m->label)[i];
    to += len;
    const uint64_t name = limb ? 0x616d690000000404ull : 0x6165720000000404ull;          // 04, 4, "ima" / "rea"
    const uint64_t last = (limb ? 'g' : 'l') | 0x010100ull;                               // "g" / "l", 01, 1
    const uint64_t tail = i < 8 ? name : i < 14 ? last : rnum;
    if (i < 22) to[0] = (uint8_t)(tail >> (8 * (i < 8 ? i : i < 14 ? i - 8 : i - 14)));
}

// A draw on the stretch's n bytes: m->out, and the stretch moved on. False when a limb
// has to be drawn again (nothing moved).
static __device__ __noinline__ bool tx_draw(TxMem* m, uint32_t n, uint64_t total, uint64_t rnum, uint32_t len)
{
    const uint32_t per = 35 + len;
    __syncwarp();
    tx_draw_bytes(m, n, len, rnum, 0);
    tx_draw_bytes(m, n + per, len, rnum + 1, 1);
    tx_hash(m, n + per, n + 2 * per, total + 2 * per, true);
    const bool ok = m->out[0] < kDrawBound && m->out[1] < kDrawBound;
    if (ok) tx_advance(m, n + 2 * per);
    return ok;
}

// The same limb by limb, each again while it is all ones (probability 2^-61; the loop
// is bounded all the same, and past the bound the value is reduced).
static __device__ __noinline__ void tx_redraw(TxMem* m, uint32_t n, uint64_t total, uint64_t rnum, uint32_t len)
{
    uint64_t limb[2];
#pragma unroll 1
    for (int k = 0; k < 2; ++k) {
        uint64_t v = 0;
#pragma unroll 1
        for (int it = 0; it < 1000; ++it) {
            __syncwarp();
            if (it == 0) {
                tx_draw_bytes(m, n, len, rnum, k);
                n += 35 + len;
                total += 35 + len;
            } else {   // the counter again
                const int q = threadIdx.x & 31;
                if (q < 13)
                    reinterpret_cast<uint8_t*>(m->buf)[n + q] =
                        (uint8_t)(q < 5 ? 0x0101ull >> (8 * q) : rnum >> (8 * (q - 5)));
                n += 13;
                total += 13;
            }
            ++rnum;
            tx_hash(m, n, n, total, true);
            v = m->out[1];
            tx_advance(m, n);
            n &= 63;
            if (v < kDrawBound) break;
        }
        limb[k] = v % P61;
    }
    __syncwarp();
    if (lead()) {
        m->out[0] = limb[0];
        m->out[1] = limb[1];
        m->total = total;
        m->rnum = rnum;
        m->n = n;
    }
    __syncwarp();
}

class Writer {
public:
    __device__ Writer(const State& s, TxMem* mem) : m(mem), total(s.total), rnum(s.rnum), n(s.nbuf)
    {
        const uint32_t lane = threadIdx.x & 31;
        __syncwarp();
        if (lane < 8) {
            m->buf[lane] = m->prev[lane] = s.unit[lane];
            m->h[lane] = s.h[lane];
        }
        __syncwarp();
    }
    // the low `bytes` bytes of v (1 <= bytes <= 8)
    __device__ void absorb_le(uint64_t v, int bytes)
    {
        const int i = (int)(threadIdx.x & 31);
        room((uint32_t)bytes);
        if (i < bytes) byte(i) = (uint8_t)(v >> (8 * i));
        moved((uint32_t)bytes);
    }
    __device__ void put_fp2(uint64_t re, uint64_t im)
    {
        const int i = (int)(threadIdx.x & 31);
        room(17);
        const uint64_t v = i < 9 ? re : im;
        if (i < 17) byte(i) = i == 0 ? 0x03 : (uint8_t)(v >> (8 * ((i - 1) & 7)));
        moved(17);
    }
    __device__ void put_label(const Label& L)
    {
        const int i = (int)(threadIdx.x & 31), q = i & 7;
        absorb_le(0x04 | ((uint64_t)L.len << 8), 5);
        room(32);
        const uint64_t v = i < 8 ? L.w0 : i < 16 ? L.w1 : i < 24 ? L.w2 : L.w3;
        if (i < (int)L.len) byte(i) = (uint8_t)(v >> (8 * q));
        moved(L.len);
    }
    // rand_ext(label)
    __device__ fp2 rand_fp2(const Label& L)
    {
        if (n > 256) take_whole();   // a draw puts at most 134 bytes, its padding at most 72
        if (lead()) {
            m->label[0] = L.w0;
            m->label[1] = L.w1;
            m->label[2] = L.w2;
            m->label[3] = L.w3;
        }
        if (tx_draw(m, n, total, rnum, L.len)) {
            const uint32_t size = 2 * (35 + L.len);
            total += size;
            rnum += 2;
            n = (n + size) & 63;
        } else {
            tx_redraw(m, n, total, rnum, L.len);
            total = m->total;
            rnum = m->rnum;
            n = m->n;
        }
        return mk(m->out[0], m->out[1]);
    }
    // the state at this point back to s (lanes 0..7 write)
    __device__ void store(State& s)
    {
        if (n >= 64) take_whole();
        const uint32_t lane = threadIdx.x & 31;
        __syncwarp();
        if (lane < 8) {
            const int k = (int)n - 8 * (int)lane;
            const uint64_t mask = k >= 8 ? ~(uint64_t)0 : k > 0 ? low_bytes(k) : 0;
            s.unit[lane] = (m->buf[lane] & mask) | (m->prev[lane] & ~mask);
            s.h[lane] = m->h[lane];
        }
        if (lead()) {
            s.total = total;
            s.rnum = rnum;
            s.nbuf = n;
        }
        __syncwarp();
    }

private:
    __device__ uint8_t& byte(int i) { return reinterpret_cast<uint8_t*>(m->buf)[n + i]; }
    __device__ void room(uint32_t bytes)   // whole blocks leave a stretch before it holds kTxBlocks
    {
        if (n + bytes >= 64 * (kTxBlocks - 1)) take_whole();
    }
    __device__ void moved(uint32_t bytes)
    {
        n += bytes;
        total += bytes;
    }
    __device__ void take_whole()
    {
        tx_hash(m, n, n, total, false);
        tx_advance(m, n);
        n &= 63;
    }
    TxMem* m;
    uint64_t total, rnum;
    uint32_t n;                  // bytes of the stretch
};
#else
class Writer : public Alone {
public:
    Writer(const State& state, TxMem*) : Alone(state) {}
    void absorb_le(uint64_t v, int bytes) { fs::absorb_le(s, v, bytes); }
    void put_label(const Label& L) { fs::put_label(s, L); }
};
#endif
#endif

}  // namespace fs
}  // namespace tp
