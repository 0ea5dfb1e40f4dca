// plq_resident.cu -- all the sweeps of an advance or of a batch of samples of
// one lattice in one launch.
//
// A small lattice's colour pass is a few microseconds of latency, not work, and
// a launch per pass, with its pack, unpack, snapshot, measurement and fix-up
// launches, is what such a chain spends its time on.  Here the CTAs stay for the
// whole call and a barrier stands where a launch stood: one CTA's, a cluster's in
// hardware (up to 16 CTAs), or a cooperative grid's.  After each sample's sweeps
// the same CTAs write its configuration in the host's order and add up its
// primaries.
//
// us a sweep, a launch per pass / resident, keyed: Ising 64^2 8.3 / 1.1, 48 x 40 x
// 36 heat bath 8.2 / 3.4, 512^2 9.5 / 3.8, 100^3 12.3 / 6.7, 250^3 124 / 31; gauge 24^4
// 49 / 16.7, 48^3 37 / 12.6; Potts q = 3 64^3 heat bath 8.6 / 5.4, PCG stream 12.4 /
// 10.1.  What is left of a small pass is one thread's chain of instructions (about
// 0.55 us) and the barrier: a cluster's with the words' way through L2 0.7 us more, a
// grid's 1.2 us.  (Words copied to every CTA of a cluster through distributed shared
// memory instead were slower: 16 remote stores per group, 4.5 us for 48 x 40 x 36.)
//
// The states of the passes:
//  * q = 2 sites (2D, 3D) and Z2 links (2D to 4D, rows of at most 64) on the
//    keyed stream: one bit a variable, in words of 64 sites of a row (the last
//    word of a row holds what is left) or of a row of links, packed at the
//    launch's start and unpacked at its end (plq_packed.cuh's decisions).  Where one
//    CTA is enough, it keeps the words in shared memory;
//  * every other chain whose draws sit at positions known beforehand: the byte
//    states and the pass bodies of plq_local_impl.cuh and plq_words.cuh.
// Results are the per-pass kernels', bit for bit.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "../../include/plaquette.h"
#include "plq_device.cuh"
#include "plq_items.cuh"
#include "plq_obs.cuh"
#include "plq_packed.cuh"
#include "plq_resident.h"

namespace plq {

namespace {

namespace cg = cooperative_groups;

constexpr int kResidentThreads = 512;  // at most, in a cluster's CTAs
constexpr int kGridThreads = 256;      // in a cooperative grid's
constexpr int kResidentRanks = 2;      // colour ranks per thread of the generic body
constexpr unsigned kClusterCtas = 16;
constexpr int kResidentSpin = 1 << 24;

// Barrier of all CTAs, the launch's `arrived / gridDim.x`-th: a cluster's, or a
// cooperative grid's, which counts arrivals over all of a chain's launches in a
// word of its control block: one release by each CTA and a read until all have
// arrived, half the round-trips to L2 of a barrier that is reset and signalled.
// Bounded: a wait that runs out sets a status bit and goes on.
__device__ void resident_barrier(const ResidentArgs &a, unsigned long long &arrived) {
    if (a.cluster) {
        if (gridDim.x == 1) __syncthreads();
        else cg::this_cluster().sync();
        return;
    }
    arrived += gridDim.x;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long *count = &a.p.ctrl->scratch[2], now;
        asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(count), "l"(1ull) : "memory");
        for (int spins = 0;;) {
            asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(now) : "l"(count) : "memory");
            if (now >= arrived) break;
            if (++spins > kResidentSpin) {
                atomicOr(&a.p.ctrl->status, kStatusLookbackTimeout);
                break;
            }
        }
    }
    __syncthreads();
}

// ------------------------------------------------------------ packed sites
// Word u of the lattice: row u / wpr, 64-site word u % wpr of it.
struct SiteWord {
    uint32_t r, w, len, last;  // row, word, its sites, the sites of a row's last word
};
__device__ __forceinline__ SiteWord site_word(const ResidentArgs &a, uint32_t u) {
    SiteWord s;
    const uint32_t wpr = a.words_per_row;
    s.r = fdiv(u, a.wpr_m, a.wpr_l);
    s.w = u - s.r * wpr;
    s.last = (uint32_t)a.p.g.L[0] - 64u * (wpr - 1u);
    s.len = s.w + 1u < wpr ? 64u : s.last;
    return s;
}
__device__ __forceinline__ uint64_t low_bits(uint32_t len) { return len == 64 ? ~0ull : (1ull << len) - 1ull; }
// The word's sites displaced by +1 / -1 along the row (periodic).
__device__ __forceinline__ uint64_t word_right(const ResidentArgs &a, const uint64_t *pk, const SiteWord &s, uint64_t C) {
    const uint32_t wpr = a.words_per_row;
    const uint64_t next = wpr == 1 ? C : pk[s.r * wpr + (s.w + 1u < wpr ? s.w + 1u : 0u)];
    return (C >> 1) | (next & 1ull) << (s.len - 1u);
}
__device__ __forceinline__ uint64_t word_left(const ResidentArgs &a, const uint64_t *pk, const SiteWord &s, uint64_t C) {
    const uint32_t wpr = a.words_per_row;
    const uint64_t prev = wpr == 1 ? C : pk[s.r * wpr + (s.w > 0 ? s.w - 1u : wpr - 1u)];
    return (C << 1 | ((prev >> ((s.w > 0 ? 64u : s.last) - 1u)) & 1ull)) & low_bits(s.len);
}

template <int D>
__device__ __forceinline__ void site_pass(const ResidentArgs &a, const LocalArgs &p, uint64_t *pk, const uint2 *tab) {
    const uint32_t wpr = a.words_per_row;
    const uint32_t mix = keyed_mix(p.sweep32);
    const bool hb = p.kernel == PLQ_HEATBATH;
    for (uint32_t u = blockIdx.x * blockDim.x + threadIdx.x; u < a.units; u += gridDim.x * blockDim.x) {
        const SiteWord s = site_word(a, u);
        const int n = (int)(s.len / 2);
        int32_t op[4] = {0, 0, 0, 0}, om[4] = {0, 0, 0, 0};
        const int par = row_geometry<D>(p.g, s.r, op, om);
        const uint64_t C = pk[u];
        uint64_t c0 = 0, c1 = 0, c2 = 0;
        count_add(c0, c1, c2, word_right(a, pk, s, C));
        count_add(c0, c1, c2, word_left(a, pk, s, C));
#pragma unroll
        for (int k = 1; k < D; ++k) {
            count_add(c0, c1, c2, pk[u + (uint32_t)op[k] * wpr]);
            count_add(c0, c1, c2, pk[u + (uint32_t)om[k] * wpr]);
        }
        const uint32_t x0 = (uint32_t)((p.color ^ par) & 1);  // (a word's first site has an even x)
        const uint32_t v0 = s.r * (uint32_t)p.g.L[0] + 64u * s.w + x0;
        const uint64_t flip =
            hb ? decide_row<uint64_t, 2, true>(C >> x0, c0 >> x0, c1 >> x0, c2 >> x0, n, v0, p.seed32, mix, tab)
               : decide_row<uint64_t, 2, false>(C >> x0, c0 >> x0, c1 >> x0, c2 >> x0, n, v0, p.seed32, mix, tab);
        pk[u] = C ^ (flip << x0);
    }
}

// The group of eight variables a thread keeps for the whole launch, with what
// does not change from pass to pass: where its word and the neighbours' words
// lie, and the first rounds of both colours' draws.
struct SiteGroup {
    bool any;
    uint32_t u, at[6];  // the word, and the words of its +x, -x, +y, -y, +z, -z neighbours
    int c, n, par;
    uint32_t len, left_bit, v;  // sites of the word; the place of its left neighbour's last site; its first site
    uint32_t head[2][8];
};

template <int D>
__device__ __forceinline__ SiteGroup site_group(const ResidentArgs &a) {
    SiteGroup t;
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x, wpr = a.words_per_row;
    t.u = fdiv(i, a.groups_m, a.groups_l);
    t.c = (int)(i - t.u * a.groups);
    const uint32_t u = t.u < a.units ? t.u : 0u;
    const SiteWord s = site_word(a, u);
    t.n = (int)(s.len / 2);
    t.any = t.u < a.units && 8 * t.c < t.n;
    t.u = u;
    int32_t op[4] = {0, 0, 0, 0}, om[4] = {0, 0, 0, 0};
    t.par = row_geometry<D>(a.p.g, s.r, op, om) & 1;
    t.len = s.len;
    t.left_bit = (s.w > 0 ? 64u : s.last) - 1u;
    t.v = s.r * (uint32_t)a.p.g.L[0] + 64u * s.w;
    t.at[0] = s.r * wpr + (s.w + 1u < wpr ? s.w + 1u : 0u);
    t.at[1] = s.r * wpr + (s.w > 0 ? s.w - 1u : wpr - 1u);
#pragma unroll
    for (int k = 1; k < 3; ++k) {
        t.at[2 * k] = k < D ? u + (uint32_t)op[k] * wpr : 0u;
        t.at[2 * k + 1] = k < D ? u + (uint32_t)om[k] * wpr : 0u;
    }
#pragma unroll
    for (int color = 0; color < 2; ++color)
#pragma unroll
        for (int k = 0; k < 8; ++k)
            t.head[color][k] = lowbias32_head(a.p.seed32 ^ (t.v + (uint32_t)((color ^ t.par) + 2 * (8 * t.c + k))));
    return t;
}

template <int D, int COLOR>
__device__ __forceinline__ void site_group_pass(const LocalArgs &p, const SiteGroup &t, uint64_t *pk, const uint2 *tab) {
    if (!t.any) return;
    const uint32_t mix = keyed_mix(p.sweep32);
    const uint64_t C = pk[t.u], right = pk[t.at[0]], left = pk[t.at[1]];
    uint64_t c0 = 0, c1 = 0, c2 = 0;
    count_add<uint64_t>(c0, c1, c2, (C >> 1) | (right & 1ull) << (t.len - 1u));
    count_add<uint64_t>(c0, c1, c2, (C << 1 | ((left >> t.left_bit) & 1ull)) & low_bits(t.len));
#pragma unroll
    for (int k = 2; k < 2 * D; ++k) count_add(c0, c1, c2, pk[t.at[k]]);
    const uint32_t x0 = (uint32_t)(COLOR ^ t.par);
    const uint32_t flip =
        p.kernel == PLQ_HEATBATH
            ? decide_group<uint64_t, 2, true, true>(C >> x0, c0 >> x0, c1 >> x0, c2 >> x0, t.c, t.n, t.v + x0, p.seed32, mix,
                                                    tab, t.head[COLOR])
            : decide_group<uint64_t, 2, false, true>(C >> x0, c0 >> x0, c1 >> x0, c2 >> x0, t.c, t.n, t.v + x0, p.seed32, mix,
                                                     tab, t.head[COLOR]);
    // (flips are at even bits, so a shift by x0 <= 1 stays in the group's 16)
    reinterpret_cast<uint16_t *>(pk + t.u)[t.c] = (uint16_t)((uint32_t)(C >> (16 * t.c)) ^ (flip << x0));
}

// Bond or agreement sum of the word's +mu bonds, and its count of state 1.
template <int D>
__device__ __forceinline__ void site_word_primaries(const ResidentArgs &a, const uint64_t *pk, uint32_t u, long long &acc,
                                                    long long &ones) {
    const SiteWord s = site_word(a, u);
    int32_t op[4] = {0, 0, 0, 0}, om[4] = {0, 0, 0, 0};
    row_geometry<D>(a.p.g, s.r, op, om);
    const uint64_t C = pk[u];
    int differ = __popcll(C ^ word_right(a, pk, s, C));
#pragma unroll
    for (int k = 1; k < D; ++k) differ += __popcll(C ^ pk[u + (uint32_t)op[k] * a.words_per_row]);
    const long long pairs = (long long)D * s.len;
    acc += a.p.model == PLQ_ISING ? pairs - 2ll * differ : pairs - differ;
    ones += __popcll(C);
}

// `len` bytes (0/1) from or to a word; four at a time where they are aligned.
__device__ __forceinline__ uint64_t pack_bytes(const uint8_t *b, uint32_t len, bool quads) {
    uint64_t w = 0;
    if (quads) {
        for (uint32_t k = 0; k < len / 4; ++k)  // (b_i * 2^(24 - 7 i) lands at bit 24 + i)
            w |= (uint64_t)(((reinterpret_cast<const uint32_t *>(b)[k] * 0x01020408u) >> 24) & 0xFu) << (4 * k);
    } else {
        for (uint32_t k = 0; k < len; ++k) w |= (uint64_t)(b[k] & 1u) << k;
    }
    return w;
}
__device__ __forceinline__ void unpack_bytes(uint64_t w, uint8_t *b, uint32_t len, bool quads) {
    if (quads) {
        for (uint32_t k = 0; k < len / 4; ++k)
            reinterpret_cast<uint32_t *>(b)[k] = ((uint32_t)(w >> (4 * k)) & 0xFu) * 0x00204081u & 0x01010101u;
    } else {
        for (uint32_t k = 0; k < len; ++k) b[k] = (uint8_t)((w >> k) & 1u);
    }
}

// ------------------------------------------------------------ packed links
template <class W>
__device__ __forceinline__ void link_pass(const ResidentArgs &a, const LocalArgs &p, W *pk, const uint2 *tab) {
    for (uint32_t chunk = blockIdx.x; chunk * blockDim.x < a.units; chunk += gridDim.x) {
        switch (p.g.d * 4 + p.dir) {
            case 8: packed_link_item<2, 0, W>(p, pk, chunk, 1, tab); break;
            case 9: packed_link_item<2, 1, W>(p, pk, chunk, 1, tab); break;
            case 12: packed_link_item<3, 0, W>(p, pk, chunk, 1, tab); break;
            case 13: packed_link_item<3, 1, W>(p, pk, chunk, 1, tab); break;
            case 14: packed_link_item<3, 2, W>(p, pk, chunk, 1, tab); break;
            case 16: packed_link_item<4, 0, W>(p, pk, chunk, 1, tab); break;
            case 17: packed_link_item<4, 1, W>(p, pk, chunk, 1, tab); break;
            case 18: packed_link_item<4, 2, W>(p, pk, chunk, 1, tab); break;
            default: packed_link_item<4, 3, W>(p, pk, chunk, 1, tab); break;
        }
    }
}

// As SiteGroup: eight links of each direction's row r.
struct LinkGroup {
    bool any;
    uint32_t r;
    int c, par;
    int32_t op[4], om[4];
};

template <int D>
__device__ __forceinline__ LinkGroup link_group(const ResidentArgs &a) {
    LinkGroup t;
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    t.r = fdiv(i, a.groups_m, a.groups_l);
    t.c = (int)(i - t.r * a.groups);
    t.any = t.r < a.units && 8 * t.c < a.p.g.L[0] / 2;
    if (t.r >= a.units) t.r = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) t.op[k] = t.om[k] = 0;
    t.par = row_geometry<D>(a.p.g, t.r, t.op, t.om) & 1;
    return t;
}

template <int D, int MU, class W>
__device__ __forceinline__ void link_group_pass(const ResidentArgs &a, const LocalArgs &p, const LinkGroup &t, W *pk,
                                                const uint2 *tab) {
    if (!t.any) return;
    const uint32_t L0 = (uint32_t)p.g.L[0], rows = a.units;
    const uint32_t mix = keyed_mix(p.sweep32);
    W U, c0, c1, c2;
    link_row<D, MU, W>(L0, rows, pk, t.r, t.op, t.om, U, c0, c1, c2);
    const uint32_t x0 = (uint32_t)(p.color ^ t.par);
    const uint32_t v0 = (t.r * L0 + x0) * (uint32_t)D + (uint32_t)MU;
    const int n = (int)(L0 / 2);
    const uint32_t none[8] = {};
    const uint32_t flip =
        p.kernel == PLQ_HEATBATH
            ? decide_group<W, 2 * D, true, false>(U >> x0, c0 >> x0, c1 >> x0, c2 >> x0, t.c, n, v0, p.seed32, mix, tab, none)
            : decide_group<W, 2 * D, false, false>(U >> x0, c0 >> x0, c1 >> x0, c2 >> x0, t.c, n, v0, p.seed32, mix, tab, none);
    reinterpret_cast<uint16_t *>(pk + (uint32_t)MU * rows + t.r)[t.c] =
        (uint16_t)((uint32_t)(U >> (16 * t.c)) ^ (flip << x0));
}

template <class W>
__device__ __forceinline__ void link_groups(const ResidentArgs &a, const LocalArgs &p, const LinkGroup &t, W *pk,
                                            const uint2 *tab) {
    switch (p.g.d * 4 + p.dir) {
        case 8: link_group_pass<2, 0, W>(a, p, t, pk, tab); break;
        case 9: link_group_pass<2, 1, W>(a, p, t, pk, tab); break;
        case 12: link_group_pass<3, 0, W>(a, p, t, pk, tab); break;
        case 13: link_group_pass<3, 1, W>(a, p, t, pk, tab); break;
        case 14: link_group_pass<3, 2, W>(a, p, t, pk, tab); break;
        case 16: link_group_pass<4, 0, W>(a, p, t, pk, tab); break;
        case 17: link_group_pass<4, 1, W>(a, p, t, pk, tab); break;
        case 18: link_group_pass<4, 2, W>(a, p, t, pk, tab); break;
        default: link_group_pass<4, 3, W>(a, p, t, pk, tab); break;
    }
}

// Row r of every direction in the host's order: site * d + direction.
template <class W>
__device__ __forceinline__ void unpack_link_row(const ResidentArgs &a, const W *pk, uint32_t r, uint8_t *out) {
    const uint32_t rows = a.units, L0 = (uint32_t)a.p.g.L[0];
    const int d = a.p.g.d;
    if (d == 4) {
        const W w0 = pk[r], w1 = pk[rows + r], w2 = pk[2 * rows + r], w3 = pk[3 * rows + r];
        uint32_t *o = reinterpret_cast<uint32_t *>(out) + (size_t)r * L0;
        for (uint32_t x = 0; x < L0; ++x)
            o[x] = (uint32_t)((w0 >> x) & 1u) | (uint32_t)((w1 >> x) & 1u) << 8 | (uint32_t)((w2 >> x) & 1u) << 16 |
                   (uint32_t)((w3 >> x) & 1u) << 24;
        return;
    }
    for (int dir = 0; dir < d; ++dir) {
        const W w = pk[(uint32_t)dir * rows + r];
        uint8_t *o = out + (size_t)r * L0 * d + dir;
        for (uint32_t x = 0; x < L0; ++x) o[(size_t)x * d] = (uint8_t)((w >> x) & 1u);
    }
}

// --------------------------------------------------- keyed sites in bytes
// One colour site per thread: any q, any even extents (the lattices whose rows
// the four-site words do not fit, and every Potts Metropolis chain).  The same
// keys, draws and tables as plq_local_impl.cuh; that body's eight ranks a
// thread, 64-bit keys and unused packing weights left the pass at two CTAs per SM:
// q = 5 Metropolis on 1002 x 750, 20.6 us a sweep, 10.1 so.
template <int D>
__device__ __forceinline__ void rank_pass(const ResidentArgs &a, const LocalArgs &p) {
    const uint32_t q = (uint32_t)p.q;
    const uint32_t mix = keyed_mix(p.sweep32);
    const bool metropolis = p.kernel == PLQ_METROPOLIS;
    for (uint32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < a.units; r += gridDim.x * blockDim.x) {
        int32_t x[D], op[D], om[D];
        const uint32_t s = site_of_rank<D>(p.g, r, p.color, x);
        wrap_offsets<D>(p.g, x, op, om);
        const uint32_t cur = p.state[s];
        uint32_t nb[2 * D];
#pragma unroll
        for (int mu = 0; mu < D; ++mu) {
            nb[2 * mu] = p.state[s + (uint32_t)op[mu]];
            nb[2 * mu + 1] = p.state[s + (uint32_t)om[mu]];
        }
        const uint32_t k = lowbias32_tail(lowbias32_head(p.seed32 ^ s) ^ mix) >> 8;
        uint32_t out = cur;
        if (metropolis && q > 2) {
            // keyed proposal (metropolis.wgsl:45-55)
            const uint32_t k24 = lowbias32_tail(lowbias32_head(p.seed32 ^ kProposalKey ^ s) ^ mix) >> 8;
            const float scaled = __fmul_rn(__fmul_rn((float)k24, 5.9604644775390625e-8f), (float)(q - 1));
            uint32_t prop = __float2uint_rz(scaled);
            if (prop >= q - 1) prop = q - 2;
            if (prop >= cur) prop += 1;
            uint32_t cp = 0, cc = 0;
#pragma unroll
            for (int i = 0; i < 2 * D; ++i) {
                cp += nb[i] == prop;
                cc += nb[i] == cur;
            }
            constexpr uint32_t B = 2 * D + 1;
            const uint32_t e = p.metro24[((cur * q + prop) * B + cp) * B + cc];
            if (e == 0xFFFFFFFFu || k < e) out = prop;
        } else {
            uint32_t key = 0;
#pragma unroll
            for (int i = 0; i < 2 * D; ++i) key += (uint32_t)p.pw[nb[i]];
            key = cur + q * key;
            if (metropolis) {
                const uint32_t e = p.metro24[key];
                if (e == 0xFFFFFFFFu || k < e) out = 1u - cur;
            } else {
                const uint32_t *cut = p.hb24 + (size_t)key * (q - 1);
                out = 0;
                for (uint32_t j = 0; j + 1 < q; ++j) out += cut[j] <= k ? 1u : 0u;
            }
        }
        p.state[s] = (uint8_t)out;
    }
}

// ------------------------------------------------------------------ kernel
// The packed words from the byte planes, or back.
template <ResidentKind K>
__device__ void repack(const ResidentArgs &a, void *pk, bool to_words) {
    const uint32_t L0 = (uint32_t)a.p.g.L[0];
    const bool quads = (L0 & 3u) == 0;
    const uint32_t total = K == ResidentKind::kSites ? a.units : a.units * (uint32_t)a.p.g.d;
    for (uint32_t u = blockIdx.x * blockDim.x + threadIdx.x; u < total; u += gridDim.x * blockDim.x) {
        uint8_t *bytes;
        uint32_t len = L0;
        if (K == ResidentKind::kSites) {
            const SiteWord s = site_word(a, u);
            bytes = a.p.state + (size_t)s.r * L0 + 64u * s.w;
            len = s.len;
        } else {
            bytes = a.p.state + (size_t)u * L0;  // (planes of rows)
        }
        const bool narrow = K == ResidentKind::kLinks32;
        if (to_words) {
            const uint64_t w = pack_bytes(bytes, len, quads);
            if (narrow) static_cast<uint32_t *>(pk)[u] = (uint32_t)w;
            else static_cast<uint64_t *>(pk)[u] = w;
        } else {
            unpack_bytes(narrow ? static_cast<const uint32_t *>(pk)[u] : static_cast<const uint64_t *>(pk)[u],
                         bytes, len, quads);
        }
    }
}

__device__ __forceinline__ void add_primary(long long *out, long long v) {
    v = warp_sum(v);
    if ((threadIdx.x & 31u) == 0 && v) atomicAdd((unsigned long long *)out, (unsigned long long)v);
}

// One sample of the current configuration: its bytes in the host's order and its
// primaries (out, zero before the launch).
template <ResidentKind K>
__device__ void take_sample(const ResidentArgs &a, const void *words, uint64_t sample, int *s_counts) {
    const uint32_t t0 = blockIdx.x * blockDim.x + threadIdx.x, step = gridDim.x * blockDim.x;
    const Geom &g = a.p.g;
    const uint32_t L0 = (uint32_t)g.L[0];
    uint8_t *snap = a.snapshots ? a.snapshots + (size_t)sample * a.n_vars : nullptr;
    long long *out = a.primaries ? a.primaries + sample * (uint64_t)a.n_primaries : nullptr;
    if (K == ResidentKind::kSites) {
        const uint64_t *pk = static_cast<const uint64_t *>(words);
        long long acc = 0, ones = 0, sites = 0;
        const bool quads = (L0 & 3u) == 0 && (a.n_vars & 3) == 0;
        for (uint32_t u = t0; u < a.units; u += step) {
            const SiteWord s = site_word(a, u);
            if (snap)
                unpack_bytes(pk[u], snap + (size_t)s.r * L0 + 64u * s.w, s.len, quads);
            if (out) {
                if (g.d == 2) site_word_primaries<2>(a, pk, u, acc, ones);
                else site_word_primaries<3>(a, pk, u, acc, ones);
                sites += s.len;
            }
        }
        if (out) {
            add_primary(&out[0], acc);
            if (a.p.model == PLQ_ISING) {
                add_primary(&out[1], sites - 2 * ones);
            } else {
                add_primary(&out[1], sites - ones);
                add_primary(&out[2], ones);
            }
        }
    } else if (K == ResidentKind::kLinks32 || K == ResidentKind::kLinks64) {
        using W = typename std::conditional<K == ResidentKind::kLinks32, uint32_t, uint64_t>::type;
        const W *pk = static_cast<const W *>(words);
        if (snap)
            for (uint32_t r = t0; r < a.units; r += step) unpack_link_row<W>(a, pk, r, snap);
        if (out) {
            long long acc = 0;
            for (uint32_t c = blockIdx.x; c * blockDim.x < a.units; c += gridDim.x) {
                switch (g.d) {
                    case 2: acc += packed_energy_rows<2, W>(a.p, pk, 1, c); break;
                    case 3: acc += packed_energy_rows<3, W>(a.p, pk, 1, c); break;
                    default: acc += packed_energy_rows<4, W>(a.p, pk, 1, c); break;
                }
            }
            add_primary(&out[0], acc);
        }
    } else {
        const uint32_t n = (uint32_t)g.n_sites;
        if (snap) {
            if (a.p.model == PLQ_GAUGE) {
                for (uint32_t s = t0; s < n; s += step)
                    for (int dir = 0; dir < g.d; ++dir) snap[(size_t)s * g.d + dir] = a.p.state[(size_t)dir * n + s];
            } else if ((n & 15u) == 0) {
                for (uint32_t i = t0; i < n / 16; i += step)
                    reinterpret_cast<uint4 *>(snap)[i] = reinterpret_cast<const uint4 *>(a.p.state)[i];
            } else {
                for (uint32_t s = t0; s < n; s += step) snap[s] = a.p.state[s];
            }
        }
        if (out) {
            if (a.p.model == PLQ_POTTS) {
                for (int i = threadIdx.x; i < a.p.q; i += blockDim.x) s_counts[i] = 0;
                __syncthreads();
            }
            long long acc0 = 0, acc1 = 0;
            for (uint32_t s = t0; s < n; s += step) {
                switch (g.d) {
                    case 1: site_primaries<1>(a.p.state, g, a.p.model, s, acc0, acc1, s_counts); break;
                    case 2: site_primaries<2>(a.p.state, g, a.p.model, s, acc0, acc1, s_counts); break;
                    case 3: site_primaries<3>(a.p.state, g, a.p.model, s, acc0, acc1, s_counts); break;
                    default: site_primaries<4>(a.p.state, g, a.p.model, s, acc0, acc1, s_counts); break;
                }
            }
            flush_primaries(acc0, acc1, a.p.model, a.p.q, s_counts, out);
        }
    }
}

// How a packed kind's words are shared out: kStream, a thread takes units in
// turn (whole words or rows); kGroups, a thread keeps one group of eight variables
// for the launch; kLocal, the same with the words in the shared memory of the
// one CTA.  (The other kinds are kStream.)
enum Share { kStream, kGroups, kLocal };

template <ResidentKind K, Share S>
__global__ void __launch_bounds__(kResidentThreads, K == ResidentKind::kGeneric || S != kStream ? 1 : 2)
resident_kernel(const __grid_constant__ ResidentArgs a) {
    constexpr bool kPacked = K == ResidentKind::kSites || K == ResidentKind::kLinks32 || K == ResidentKind::kLinks64;
    extern __shared__ __align__(16) unsigned char s_words[];
    __shared__ LocalArgs s_args;
    __shared__ uint2 s_tab[kTableEntries + 1];
    __shared__ int s_counts[64];
    void *pk = S == kLocal ? s_words : a.packed;
    if (threadIdx.x == 0) s_args = a.p;
    unsigned long long arrived = a.arrived;
    SiteGroup sg;
    LinkGroup lg;
    if (kPacked) {
        uint32_t cut = 1;
        if (threadIdx.x < (unsigned)a.n_keys) cut = (a.p.kernel == PLQ_HEATBATH ? a.p.hb24 : a.p.metro24)[threadIdx.x];
        if (threadIdx.x < kTableEntries) s_tab[threadIdx.x] = table_entry_marked(cut);
        const bool marked = __syncthreads_or(cut == 0);
        if (threadIdx.x == 0) s_tab[kTableEntries].x = marked ? 1u : 0u;
        if (S != kStream && K == ResidentKind::kSites) sg = a.p.g.d == 2 ? site_group<2>(a) : site_group<3>(a);
        if (S != kStream && K != ResidentKind::kSites)
            lg = a.p.g.d == 2 ? link_group<2>(a) : a.p.g.d == 3 ? link_group<3>(a) : link_group<4>(a);
        repack<K>(a, pk, true);
        resident_barrier(a, arrived);
    }
    __syncthreads();
    const int passes = a.p.model == PLQ_GAUGE ? 2 * a.p.g.d : 2;
    const bool sampling = a.snapshots || a.primaries;
    uint64_t sweep = 0;
    for (uint64_t sample = 0; sample < a.samples; ++sample) {
        for (uint64_t t = 0; t < a.sweeps; ++t, ++sweep) {
            for (int pass = 0; pass < passes; ++pass) {
                if (threadIdx.x == 0) {
                    s_args.dir = a.p.model == PLQ_GAUGE ? pass >> 1 : 0;
                    s_args.color = pass & 1;
                    s_args.sweep32 = a.p.sweep32 + (uint32_t)sweep;
                    s_args.pass_offset = a.p.pass_offset + sweep * (uint64_t)a.n_vars +
                                         (uint64_t)pass * (uint64_t)(a.p.g.n_sites / 2);
                }
                __syncthreads();
                if (K == ResidentKind::kSites) {
                    uint64_t *w = static_cast<uint64_t *>(pk);
                    if (S == kStream) {
                        if (a.p.g.d == 2) site_pass<2>(a, s_args, w, s_tab);
                        else site_pass<3>(a, s_args, w, s_tab);
                    } else if (a.p.g.d == 2) {
                        if (pass == 0) site_group_pass<2, 0>(s_args, sg, w, s_tab);
                        else site_group_pass<2, 1>(s_args, sg, w, s_tab);
                    } else {
                        if (pass == 0) site_group_pass<3, 0>(s_args, sg, w, s_tab);
                        else site_group_pass<3, 1>(s_args, sg, w, s_tab);
                    }
                } else if (K == ResidentKind::kLinks32) {
                    if (S == kStream) link_pass<uint32_t>(a, s_args, static_cast<uint32_t *>(pk), s_tab);
                    else link_groups<uint32_t>(a, s_args, lg, static_cast<uint32_t *>(pk), s_tab);
                } else if (K == ResidentKind::kLinks64) {
                    if (S == kStream) link_pass<uint64_t>(a, s_args, static_cast<uint64_t *>(pk), s_tab);
                    else link_groups<uint64_t>(a, s_args, lg, static_cast<uint64_t *>(pk), s_tab);
                } else if (K == ResidentKind::kRanks) {
                    switch (a.p.g.d) {
                        case 1: rank_pass<1>(a, s_args); break;
                        case 2: rank_pass<2>(a, s_args); break;
                        case 3: rank_pass<3>(a, s_args); break;
                        default: rank_pass<4>(a, s_args); break;
                    }
                } else {
                    for (uint32_t c = blockIdx.x; c < a.chunks; c += gridDim.x)
                        run_item<kResidentRanks, K == ResidentKind::kWords>(s_args, a.p.g.d, a.p.model == PLQ_GAUGE, c,
                                                                            a.words_per_thread);
                }
                resident_barrier(a, arrived);
            }
        }
        if (sampling) {
            take_sample<K>(a, pk, sample, s_counts);
            if (sample + 1 < a.samples) resident_barrier(a, arrived);
        }
    }
    // (the last barrier was past every write of the words; the bytes are read by no one here)
    if (kPacked) repack<K>(a, pk, false);
}

// A cluster of the grid's CTAs, or a cooperative grid.
void resident_config(const ResidentPlan &p, cudaLaunchConfig_t &cfg, cudaLaunchAttribute &attr, cudaStream_t stream) {
    cfg.gridDim = dim3(p.grid);
    cfg.blockDim = dim3((unsigned)p.block);
    cfg.dynamicSmemBytes = p.shared_bytes;
    cfg.stream = stream;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    if (p.cluster) {
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = p.grid;
        attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    } else {
        attr.id = cudaLaunchAttributeCooperative;
        attr.val.cooperative = 1;
    }
}

constexpr bool packed_kind(ResidentKind k) {
    return k == ResidentKind::kSites || k == ResidentKind::kLinks32 || k == ResidentKind::kLinks64;
}
// Attributes of the kernel a plan names, and whether the device takes its cluster.
template <ResidentKind K, Share S>
bool cluster_fits(const ResidentPlan &p) {
    auto kern = resident_kernel<K, S>;
    cudaError_t e = cudaSuccess;
    if (p.shared_bytes > 40 * 1024)
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)p.shared_bytes);
    int clusters = 1;
    if (e == cudaSuccess && p.grid > 8) {  // beyond the portable size
        cudaLaunchConfig_t cfg{};
        cudaLaunchAttribute attr{};
        resident_config(p, cfg, attr, nullptr);
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg);
    }
    if (e != cudaSuccess) (void)cudaGetLastError();
    return e == cudaSuccess && clusters > 0;
}

unsigned power_of_two_at_least(unsigned n) {
    unsigned p = 1;
    while (p < n) p *= 2;
    return p;
}

// The launch shape of a pass of p.units units.
template <ResidentKind K>
cudaError_t plan_kind(ResidentPlan &p, int sm_count) {
    if constexpr (packed_kind(K)) {
        // Too small a pass to fill the chip is split into groups of eight variables a thread: its
        // time is a thread's chain of decisions.  Two CTAs of kGridThreads fit an SM.
        const uint32_t items = p.units * p.most_groups;
        if (items <= (uint32_t)sm_count * 2 * kGridThreads) {
            p.groups = p.most_groups;
            const uint32_t warps = (items + 31) / 32;
            p.cluster = true;
            if (items <= kResidentThreads) {
                p.share = kLocal;
                p.grid = 1;
                p.block = (int)warps * 32;
                p.shared_bytes = p.packed_bytes;
                if (cluster_fits<K, kLocal>(p)) return cudaSuccess;
                p.shared_bytes = 0;
            }
            p.share = kGroups;
            if (items <= kClusterCtas * kResidentThreads) {
                p.grid = power_of_two_at_least((warps + 3) / 4);  // at least four warps a CTA
                if (p.grid > kClusterCtas) p.grid = kClusterCtas;
                p.block = (int)((warps + p.grid - 1) / p.grid) * 32;
                if (cluster_fits<K, kGroups>(p)) return cudaSuccess;
            }
            p.cluster = false;
            p.block = kGridThreads;
            p.grid = (items + kGridThreads - 1) / kGridThreads;
            return cudaSuccess;
        }
    }
    auto kern = resident_kernel<K, kStream>;
    p.share = kStream;
    p.groups = 1;
    const uint32_t threads = (p.units + (uint32_t)p.per_thread - 1) / (uint32_t)p.per_thread;
    if (threads <= 8 * 128) {  // few CTAs: the cluster's barrier is the cheaper one
        p.block = 128;
        p.chunks = std::max(1u, (threads + 127) / 128);
        p.grid = power_of_two_at_least(p.chunks);  // (a CTA without a chunk only joins the barriers)
        p.cluster = true;
        return cudaSuccess;
    }
    p.block = kGridThreads;
    p.chunks = (threads + kGridThreads - 1) / kGridThreads;
    int per_sm = 0;
    const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, p.block, 0);
    p.cluster = false;
    p.grid = std::min(p.chunks, (unsigned)(per_sm * sm_count));
    return e != cudaSuccess || p.grid > 0 ? e : cudaErrorLaunchOutOfResources;
}

template <ResidentKind K>
cudaError_t launch_kind(const ResidentPlan &p, const ResidentArgs &a, cudaStream_t stream) {
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr{};
    resident_config(p, cfg, attr, stream);
    if constexpr (packed_kind(K)) {
        if (p.share == kLocal) return cudaLaunchKernelEx(&cfg, resident_kernel<K, kLocal>, a);
        if (p.share == kGroups) return cudaLaunchKernelEx(&cfg, resident_kernel<K, kGroups>, a);
    }
    return cudaLaunchKernelEx(&cfg, resident_kernel<K, kStream>, a);
}

}  // namespace

ResidentKind resident_kind(int model, int q, int d, const int32_t *L, int updater, int rng, bool words) {
    if (rng == PLQ_RNG_KEYED && (updater == PLQ_METROPOLIS || updater == PLQ_HEATBATH)) {
        if (model == PLQ_GAUGE && d >= 2 && d <= 4 && L[0] <= 64)
            return L[0] <= 32 ? ResidentKind::kLinks32 : ResidentKind::kLinks64;
        if (model != PLQ_GAUGE && q == 2 && (d == 2 || d == 3)) return ResidentKind::kSites;
    }
    if (d > 4) return ResidentKind::kNone;
    if (rng == PLQ_RNG_KEYED && model != PLQ_GAUGE && !words) return ResidentKind::kRanks;
    return words ? ResidentKind::kWords : ResidentKind::kGeneric;
}

cudaError_t resident_plan(ResidentKind kind, const Geom &g, bool stream_draws, int sm_count, ResidentPlan &p) {
    p = ResidentPlan{};
    p.kind = kind;
    p.per_thread = 1;
    p.most_groups = 1;
    const uint32_t rows = (uint32_t)(g.n_sites / g.L[0]);
    p.words_per_row = (uint32_t)(g.L[0] + 63) / 64;
    switch (kind) {
        case ResidentKind::kSites:
            p.units = rows * p.words_per_row;
            p.packed_bytes = p.units * sizeof(uint64_t);
            p.most_groups = (uint32_t)(std::min(g.L[0], 64) + 15) / 16;
            return plan_kind<ResidentKind::kSites>(p, sm_count);
        case ResidentKind::kLinks32:
            p.units = rows;
            p.packed_bytes = (size_t)rows * (size_t)g.d * sizeof(uint32_t);
            p.most_groups = (uint32_t)(g.L[0] + 15) / 16;
            return plan_kind<ResidentKind::kLinks32>(p, sm_count);
        case ResidentKind::kLinks64:
            p.units = rows;
            p.packed_bytes = (size_t)rows * (size_t)g.d * sizeof(uint64_t);
            p.most_groups = (uint32_t)(g.L[0] + 15) / 16;
            return plan_kind<ResidentKind::kLinks64>(p, sm_count);
        case ResidentKind::kWords:
            p.units = (uint32_t)(g.n_sites / 4);
            p.per_thread = stream_draws ? kWordsPerThread : 1;  // (on the stream a thread jumps once for its words)
            return plan_kind<ResidentKind::kWords>(p, sm_count);
        case ResidentKind::kRanks:
            p.units = (uint32_t)(g.n_sites / 2);
            return plan_kind<ResidentKind::kRanks>(p, sm_count);
        case ResidentKind::kGeneric:
            p.units = (uint32_t)(g.n_sites / 2);
            p.per_thread = kResidentRanks;
            return plan_kind<ResidentKind::kGeneric>(p, sm_count);
        default: return cudaErrorInvalidValue;
    }
}

uint64_t resident_barriers(const ResidentPlan &p, int passes, uint64_t samples, uint64_t sweeps, bool sampling) {
    const bool packed = p.packed_bytes != 0;
    return (packed ? 1 : 0) + samples * sweeps * (uint64_t)passes + (sampling && samples ? samples - 1 : 0);
}

cudaError_t launch_resident(const ResidentPlan &p, ResidentArgs a, cudaStream_t stream) {
    const Geom &g = a.p.g;
    a.units = p.units;
    a.chunks = p.chunks;
    a.cluster = p.cluster ? 1 : 0;
    a.words_per_thread = p.per_thread;
    a.words_per_row = p.words_per_row;
    a.groups = p.groups;
    Geom w;  // the division constants of words_per_row and groups
    const int64_t shape[2] = {(int64_t)p.words_per_row, (int64_t)p.groups};
    geom_init(w, 2, shape);
    a.wpr_m = w.dm[0];
    a.wpr_l = w.dl[0];
    a.groups_m = w.dm[1];
    a.groups_l = w.dl[1];
    // keys cur + 2 * count of a q = 2 table
    a.n_keys = 2 + 4 * (a.p.model == PLQ_GAUGE ? g.d - 1 : g.d);
    switch (p.kind) {
        case ResidentKind::kSites: return launch_kind<ResidentKind::kSites>(p, a, stream);
        case ResidentKind::kLinks32: return launch_kind<ResidentKind::kLinks32>(p, a, stream);
        case ResidentKind::kLinks64: return launch_kind<ResidentKind::kLinks64>(p, a, stream);
        case ResidentKind::kWords: return launch_kind<ResidentKind::kWords>(p, a, stream);
        case ResidentKind::kRanks: return launch_kind<ResidentKind::kRanks>(p, a, stream);
        case ResidentKind::kGeneric: return launch_kind<ResidentKind::kGeneric>(p, a, stream);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace plq
