// plq_packed.cuh -- device helpers of the bit-packed row bodies (one bit per
// q = 2 variable, a row of them per 32- or 64-bit word): neighbour rows by
// rotation, the bit-sliced neighbour counter, and the decision of a row's
// variables of one parity from nibble keys (plq_ensemble.cu's packed members,
// plq_packed3d.cu's single lattices).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "plq_rng.cuh"

namespace plq {

template <class W>
__device__ __forceinline__ W row_xp(W w, uint32_t L0, W full) {  // bit x <- bit x+1
    return ((w >> 1) | (w << (L0 - 1))) & full;
}
template <class W>
__device__ __forceinline__ W row_xm(W w, uint32_t L0, W full) {  // bit x <- bit x-1
    return ((w << 1) | (w >> (L0 - 1))) & full;
}
// bit-sliced counter (c2 c1 c0) += v, per bit position (counts stay below 8)
template <class W>
__device__ __forceinline__ void count_add(W &c0, W &c1, W &c2, W v) {
    const W k0 = c0 & v;
    c0 ^= v;
    c2 |= c1 & k0;
    c1 ^= k0;
}
__device__ __forceinline__ int popc_w(uint32_t v) { return __popc(v); }
__device__ __forceinline__ int popc_w(uint64_t v) { return __popcll(v); }

// Decide the n = L0 / 2 variables of one row that a pass updates.  Cs, c0s,
// c1s, c2s: the row's state bits and the bits of each variable's count
// (c2 c1 c0 in binary: neighbours in state 1, or satisfied staples), all
// shifted so variable j of the pass sits at bit 2j.  Its table key is
// cur + 2 * count, a nibble: eight variables' keys are gathered into one word
// (pairs (cur, c0) and (c1, c2) interleaved at two-bit granularity, Hacker's
// Delight's outer perfect shuffle without its last stage), and the key times
// eight is the byte offset of its entry in the shared-memory table tab.  The
// draw of variable j is the keyed stream's at index v0 + j * DV, composed as
// keyed24 does (mix = keyed_mix(sweep)).  Returns the bits to flip, at 2j:
// Metropolis accepts when the draw k is below the cut point e; heat bath sets
// the new state to (e <= k).
//
// The passes are bound by the integer pipe, so a decision takes as few
// operations as it can.  With v the draw before its closing xorshift
// (lowbias32_open), the draw is k = (v ^ (v >> 16)) >> 8 and, T = e * 2^8 - 1,
//   k < e  <=>  v ^ (v >> 16) <= T  <=>  v ^ (T >> 16) <= T:
// the xorshift leaves v's high half as it is, so the high halves decide unless
// they are equal, and then v >> 16 is T >> 16.  A table entry holds T and
// T >> 16, and three operations (a shift, a xor and the shift by 8) become one
// xor.  512^3 keyed Ising Metropolis, ms per sweep: see packed_pass_kernel.
// e = 2^24 ("always", no 24-bit draw reaches it) has T = 2^32 - 1.  e = 0
// ("never", a probability that underflowed) has no T: a table holding one is
// marked (kTableEntries) and decided from the closed draw instead.
constexpr int kTableEntries = 16;  // tab[kTableEntries].x: a cut point of the table is 0

// The table entry of cut point e >= 1 (the "always" sentinel clamped to 2^24).
__device__ __forceinline__ uint2 table_entry(uint32_t e) {
    const uint32_t t = ((e < (1u << 24) ? e : (1u << 24)) << 8) - 1u;
    return make_uint2(t, t >> 16);
}
// ... and back: the cut point behind an entry of a marked table (T = 2^32 - 1, X = 0: e = 0).
__device__ __forceinline__ uint2 table_entry_marked(uint32_t e) {
    return e ? table_entry(e) : make_uint2(0xFFFFFFFFu, 0u);
}

// Eight keys (nibbles of x) as byte offsets into the table: those of variables
// 0, 2, 4, 6 in the bytes of lo, the others in the bytes of hi, so each takes
// one byte extraction.
struct KeyOffsets {
    uint32_t lo, hi;
    __device__ __forceinline__ explicit KeyOffsets(uint32_t x)
        : lo((x << 3) & 0x78787878u), hi((x >> 1) & 0x78787878u) {}
    __device__ __forceinline__ uint32_t at(int i) const {
        const uint32_t w = (i & 1) ? hi : lo;
        return i >= 6 ? w >> 24 : __byte_perm(w, 0, 0x4440 + (i >> 1));
    }
};

template <bool HB>
__device__ __forceinline__ bool decide_bit(uint32_t v, uint2 t) {
    return HB ? (v ^ t.y) > t.x : (v ^ t.y) <= t.x;
}

// Eight (or, TAIL, the first m < 8) variables of a row from their key word x
// (nibble i: variable i's key): the flip or new-state bits at 2i.
template <int DV, bool HB, bool TAIL>
__device__ __forceinline__ uint32_t decide8(uint32_t x, int m, uint32_t vc, uint32_t seed32, uint32_t mix,
                                            const char *tb) {
    const KeyOffsets key(x);
    uint32_t o = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        if (!TAIL || i < m) {
            const uint2 t = *reinterpret_cast<const uint2 *>(tb + key.at(i));
            const uint32_t v = lowbias32_open(lowbias32_head(seed32 ^ (vc + (uint32_t)(i * DV))) ^ mix);
            if (decide_bit<HB>(v, t)) o |= 1u << (2 * i);
        }
    }
    return o;
}

// decide8 over eight variables whose first rounds lowbias32_head(seed ^ index)
// are given (h1[i] for variable i): half a keyed draw's hashing per variable.
template <bool HB>
__device__ __forceinline__ uint32_t decide8_h1(uint32_t x, const uint32_t (&h1)[8], uint32_t mix,
                                               const char *tb) {
    const KeyOffsets key(x);
    uint32_t o = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const uint2 t = *reinterpret_cast<const uint2 *>(tb + key.at(i));
        const uint32_t v = lowbias32_open(h1[i] ^ mix);
        if (decide_bit<HB>(v, t)) o |= 1u << (2 * i);
    }
    return o;
}

// decide8 (the first m <= 8 variables) for a marked table, one variable at a
// time from the whole draw: only chains so cold that a probability underflows
// come here.
template <int DV, bool HB>
__device__ __forceinline__ uint32_t decide8_marked(uint32_t x, int m, uint32_t vc, uint32_t seed32, uint32_t mix,
                                                   const char *tb) {
    uint32_t o = 0;
#pragma unroll 1
    for (int i = 0; i < m; ++i) {
        const uint2 t = *reinterpret_cast<const uint2 *>(tb + ((x >> (4 * i)) & 15u) * 8u);
        const bool never = t.x == 0xFFFFFFFFu && t.y == 0u;
        const uint32_t v = lowbias32_open(lowbias32_head(seed32 ^ (vc + (uint32_t)(i * DV))) ^ mix);
        if (HB ? never || decide_bit<true>(v, t) : !never && decide_bit<false>(v, t)) o |= 1u << (2 * i);
    }
    return o;
}

// The key word of variables 8c .. 8c + 7: pairs (cur, c0) of P and (c1, c2)
// of Q interleaved at two-bit granularity.
template <class W>
__device__ __forceinline__ uint32_t key_word(W P, W Q, int c) {
    uint32_t x = __byte_perm((uint32_t)(P >> (16 * c)), (uint32_t)(Q >> (16 * c)), 0x5410);
    x = __byte_perm(x, 0, 0x3120);
    uint32_t t = (x ^ (x >> 4)) & 0x00F000F0u;
    x ^= t ^ (t << 4);
    t = (x ^ (x >> 2)) & 0x0C0C0C0Cu;
    x ^= t ^ (t << 2);
    return x;
}

// Group c of a row alone: its variables 8c .. 8c + 7 (those below n), the flips
// at 2i of 16 bits.  Rows as decide_row's.  HEADS: the variables' first rounds
// are given (h1, any value past n).
template <class W, int DV, bool HB, bool HEADS>
__device__ __forceinline__ uint32_t decide_group(W Cs, W c0s, W c1s, W c2s, int c, int n, uint32_t v0, uint32_t seed32,
                                                 uint32_t mix, const uint2 *tab, const uint32_t (&h1)[8]) {
    const W M = (W)0x5555555555555555ull;
    const W P = (Cs & M) | ((c0s << 1) & ~M);
    const W Q = (c1s & M) | ((c2s << 1) & ~M);
    const char *tb = reinterpret_cast<const char *>(tab);
    const uint32_t x = key_word(P, Q, c), vc = v0 + (uint32_t)(8 * c * DV);
    const int m = n - 8 * c < 8 ? n - 8 * c : 8;
    const uint32_t valid = 0x5555u & ((1u << (2 * m)) - 1u);
    uint32_t out;
    if (tab[kTableEntries].x) out = decide8_marked<DV, HB>(x, m, vc, seed32, mix, tb);
    else if (HEADS) out = decide8_h1<HB>(x, h1, mix, tb);
    else out = decide8<DV, HB, false>(x, 8, vc, seed32, mix, tb);
    if (HB) out ^= (uint32_t)(P >> (16 * c));  // new states -> flips
    return out & valid;
}

template <class W, int DV, bool HB>
__device__ __forceinline__ W decide_row(W Cs, W c0s, W c1s, W c2s, int n, uint32_t v0, uint32_t seed32,
                                        uint32_t mix, const uint2 *tab) {
    const W M = (W)0x5555555555555555ull;
    const W P = (Cs & M) | ((c0s << 1) & ~M);
    const W Q = (c1s & M) | ((c2s << 1) & ~M);
    const char *tb = reinterpret_cast<const char *>(tab);
    W out = 0;
    if (tab[kTableEntries].x) {
#pragma unroll 1
        for (int c = 0; 8 * c < n; ++c)
            out |= (W)decide8_marked<DV, HB>(key_word(P, Q, c), n - 8 * c < 8 ? n - 8 * c : 8,
                                             v0 + (uint32_t)(8 * c * DV), seed32, mix, tb)
                   << (16 * c);
    } else {
        const int full = n >> 3;
#pragma unroll 1
        for (int c = 0; c < full; ++c)
            out |= (W)decide8<DV, HB, false>(key_word(P, Q, c), 8, v0 + (uint32_t)(8 * c * DV), seed32, mix, tb)
                   << (16 * c);
        if (n & 7)
            out |= (W)decide8<DV, HB, true>(key_word(P, Q, full), n & 7, v0 + (uint32_t)(8 * full * DV), seed32,
                                            mix, tb)
                   << (16 * full);
    }
    if (HB) {  // new states -> flips, over the n variables
        const W valid = 2 * n >= (int)(8 * sizeof(W)) ? ~(W)0 : (((W)1 << (2 * n)) - 1);
        out ^= P & M & valid;
    }
    return out;
}

}  // namespace plq
