// MT19937 output streams for one thread (Matsumoto & Nishimura 1998), seeded with
// init_genrand(seed): mt[0] = seed, mt[i] = 1812433253*(mt[i-1] ^ mt[i-1]>>30) + i, the
// seeding recurrence the reference's twisters use (oplib/opcuda/smc.cu:127-131).
//
// Keyed seeding (key1 != 0): the same recurrence with key1 added to mt[1] before the
// recurrence continues from it (mt[1] = 1812433253*(seed ^ seed>>30) + 1 + key1).  Two
// (seed, key1) pairs give equal initial states only if both members are equal, so one
// seed yields 2^32 distinct generators; key1 = 0 is init_genrand(seed).
//
// Two forms, bit-identical on the outputs they share:
//
// mt19937_first (n <= 623): the whole generator in registers.  The first 623 outputs of
// a freshly seeded MT19937 only need one regeneration of the state, and every regenerated
// word is an XOR of tw() terms of initial words mt[j], each of which is a forward
// recurrence from the seed.  The function walks that recurrence with a few cursors (and
// one saved word, mt[397]) instead of storing 624 words, so it uses no local or shared
// memory:
//   i <  227 : mt'[i] = mt[i+397] ^ tw(mt[i], mt[i+1])
//   i <  454 : mt'[i] = mt[i+170] ^ tw(mt[i-227], mt[i-226]) ^ tw(mt[i], mt[i+1])
//   i <  623 : mt'[i] = mt[i-57] ^ tw(mt[i-454], mt[i-453]) ^ tw(mt[i-227], mt[i-226])
//                       ^ tw(mt[i], mt[i+1])
// and tw is linear over XOR, so that the cursors' words are XORed first and one tw() is left:
// tw(a, b) ^ tw(c, d) = tw(a ^ c, b ^ d); the first operand's XOR is the previous word's second.
// Output 623 would need mt'[0] as the second operand of its tw(), i.e. a word of the
// regenerated state, which is where the cursor form stops.
//
// mt19937_any (any n): the first 623 outputs come from the same cursors, and each
// regenerated word that a later output reads is also stored in a per-thread 624-word array
// (local memory on the device, 2496 bytes a thread), so no separate initialisation pass is
// needed.  Output 623
// closes the first regeneration (mt'[623] = mt'[396] ^ tw(mt[623], mt'[0]), with the
// initial word mt[623] taken from the cursor), and every later output regenerates one word
// of the array:
//   mt[i] = mt[(i+397) mod 624] ^ tw(mt[i], mt[(i+1) mod 624]);  output temper(mt[i])
// Word i of a generation reads mt[i+397] before it is regenerated (i < 227) and after
// (i >= 227), and word 623 reads the regenerated mt[0], exactly as genrand_int32's block
// refill does, so the stream is MT19937's for every n.
//
// The header compiles as plain C++ too, so the host can check both forms against an
// independent MT19937.
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define OPB_MT_FN __host__ __device__ __forceinline__
#else
#define OPB_MT_FN inline
#endif

namespace opb {

// Longest stream mt19937_first serves.
constexpr int kMtCursorMax = 623;

// Outputs per trip of the output loops: four keep enough independent work in flight that a
// caller's dependent loads per output do not idle a warp, and no words are moved between
// registers at the end of one (Monte Carlo at 2^20 paths x 504 steps: 2.30 ms at one output a
// trip, 2.19 at four).
constexpr int kMtUnroll = 4;
OPB_MT_FN uint32_t mt_init_next(uint32_t v, uint32_t i) {
    return 1812433253u * (v ^ (v >> 30)) + i;
}
OPB_MT_FN uint32_t mt_tw(uint32_t a, uint32_t b) {
    uint32_t y = (a & 0x80000000u) | (b & 0x7fffffffu);
    return (y >> 1) ^ ((b & 1u) ? 0x9908b0dfu : 0u);
}
// x ^ tw(a, b)
OPB_MT_FN uint32_t mt_tw_xor(uint32_t a, uint32_t b, uint32_t x) {
    const uint32_t y = (a & 0x80000000u) | (b & 0x7fffffffu);
    return x ^ (y >> 1) ^ (b & 1u) * 0x9908b0dfu;
}
OPB_MT_FN uint32_t mt_temper(uint32_t y) {
    y ^= (y >> 11);
    y ^= (y << 7) & 0x9d2c5680u;
    y ^= (y << 15) & 0xefc60000u;
    y ^= (y >> 18);
    return y;
}

// Calls f(k, w_k) with the regenerated (untempered) state word w_k = mt'[k] for the first
// n (<= 623) words of MT19937 seeded with (seed, key1); returns the initial word mt[n].
template <class F>
OPB_MT_FN uint32_t mt19937_cursor_words(uint32_t seed, uint32_t key1, int n, F &&f) {
    const uint32_t m1 = mt_init_next(seed, 1u) + key1;
    // cursor A: a1 = mt[i+1]; x0 = mt[i], from phase 2 on with the other cursors' words in it
    uint32_t x0 = seed, a1 = m1, a0 = seed;
    // cursor B at i + 397 (its index comes from i: counted in a register of its own, the Monte Carlo
    // with states spilled)
    uint32_t b = m1;
#pragma unroll 4
    for (uint32_t j = 2; j <= 397; j++) b = mt_init_next(b, j);
    const uint32_t m397 = b;
    int i = 0;
    const int n1 = n < 227 ? n : 227;
#pragma unroll kMtUnroll
    for (; i < n1; i++) {
        f(i, mt_tw_xor(x0, a1, b));
        x0 = a0 = a1;
        a1 = mt_init_next(a1, (uint32_t)i + 2u);
        b = mt_init_next(b, (uint32_t)i + 398u);
    }
    if (i >= n) return a0;
    // phase 2: cursor C (c1 = mt[i-226]) from the seed, cursor B restarted at 397
    uint32_t c1 = m1;
    x0 ^= seed;
    b = m397;
    const int n2 = n < 454 ? n : 454;
#pragma unroll kMtUnroll
    for (; i < n2; i++) {
        const uint32_t x1 = a1 ^ c1;
        f(i, mt_tw_xor(x0, x1, b));
        x0 = x1; a0 = a1;
        a1 = mt_init_next(a1, (uint32_t)i + 2u);
        c1 = mt_init_next(c1, (uint32_t)(i - 227) + 2u);
        b = mt_init_next(b, (uint32_t)(i - 227) + 398u);
    }
    if (i >= n) return a0;
    // phase 3: cursor D (d1 = mt[i-453]) from the seed, B restarted at 397 (= i-57 at i = 454)
    uint32_t d1 = m1;
    x0 ^= seed;
    b = m397;
#pragma unroll kMtUnroll
    for (; i < n; i++) {
        const uint32_t x1 = a1 ^ c1 ^ d1;
        f(i, mt_tw_xor(x0, x1, b));
        x0 = x1; a0 = a1;
        a1 = mt_init_next(a1, (uint32_t)i + 2u);
        c1 = mt_init_next(c1, (uint32_t)(i - 227) + 2u);
        d1 = mt_init_next(d1, (uint32_t)(i - 454) + 2u);
        b = mt_init_next(b, (uint32_t)(i - 454) + 398u);
    }
    return a0;
}

// Calls f(k, x_k) for the first n (<= 623) outputs of MT19937 seeded with (seed, key1).
template <class F>
OPB_MT_FN void mt19937_first(uint32_t seed, uint32_t key1, int n, F &&f) {
    mt19937_cursor_words(seed, key1, n, [&](int i, uint32_t w) { f(i, mt_temper(w)); });
}

// Calls f(k, x_k) for the first n outputs of MT19937 seeded with (seed, key1), any n >= 0.
template <class F>
OPB_MT_FN void mt19937_any(uint32_t seed, uint32_t key1, int n, F &&f) {
    uint32_t mt[624];
    const int n1 = n < kMtCursorMax ? n : kMtCursorMax;
    // output 623 + j reads words j - 1, j and (j + 396) mod 624
    const uint32_t more = n > kMtCursorMax ? (uint32_t)(n - kMtCursorMax) : 0u;
    const uint32_t init623 = mt19937_cursor_words(seed, key1, n1, [&](int k, uint32_t w) {
        if ((uint32_t)k < more || (uint32_t)(k - 396) < more) mt[k] = w;
        f(k, mt_temper(w));
    });
    if (n <= kMtCursorMax) return;
    mt[623] = mt[396] ^ mt_tw(init623, mt[0]);
    f(623, mt_temper(mt[623]));
    int i = 0, im = 397;  // im = (i + 397) mod 624
    uint32_t cur = mt[0]; // mt[i], carried from the previous output's mt[i+1] load
#pragma unroll 1
    for (int k = 624; k < n; k++) {
        const int i1 = i == 623 ? 0 : i + 1;
        const uint32_t nxt = mt[i1];
        const uint32_t y = mt[im] ^ mt_tw(cur, nxt);
        mt[i] = y;
        f(k, mt_temper(y));
        i = i1;
        im = im == 623 ? 0 : im + 1;
        cur = nxt;
    }
}

// mt19937_first when ANY_LENGTH is false (n <= 623), mt19937_any otherwise.
template <bool ANY_LENGTH, class F>
OPB_MT_FN void mt19937_stream(uint32_t seed, uint32_t key1, int n, F &&f) {
    if constexpr (ANY_LENGTH) mt19937_any(seed, key1, n, static_cast<F &&>(f));
    else mt19937_first(seed, key1, n, static_cast<F &&>(f));
}

}  // namespace opb
