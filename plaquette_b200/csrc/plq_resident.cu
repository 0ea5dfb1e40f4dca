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
// 36 heat bath 8.2 / 3.4, 512^2 9.5 / 3.8, 100^3 12.3 / 6.7, 250^3 124 / 28.5; gauge 24^4
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

// How a packed kind's words are shared out: kStream, a thread takes units in
// turn (whole words or rows); kGroups, a thread keeps one group of eight variables
// for the launch; kLocal, the same with the words in the shared memory of the
// one CTA.  (The other kinds are kStream.)
enum Share { kStream, kGroups, kLocal };

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

template <int D, bool HEADS>
__device__ __forceinline__ SiteGroup site_group(const ResidentArgs &a, uint32_t i) {
    SiteGroup t;
    const uint32_t wpr = a.words_per_row;
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
    if (!HEADS) return t;
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

// Keyed sites in bytes, one colour site a thread.
template <int D>
__device__ __forceinline__ void rank_pass(const ResidentArgs &a, const LocalArgs &p) {
    const uint32_t mix = keyed_mix(p.sweep32);
    for (uint32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < a.units; r += gridDim.x * blockDim.x) rank_site<D>(p, r, mix);
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
        if (S != kStream && K == ResidentKind::kSites) {
            const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
            sg = a.p.g.d == 2 ? site_group<2, true>(a, i) : site_group<3, true>(a, i);
        }
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

// ------------------------------------------------- q = 2 on the PCG stream
// Metropolis and heat bath of the packed kinds on the bit-exact stream.  A heat
// bath draws for every variable; Metropolis only uphill (src/updater.rs:90), so a
// variable's draw sits at the number of uphill variables before it in the pass.
// On packed words that count is cheap -- "draws" is a function of the state bit
// and the three bits of the neighbour count, evaluated for 64 sites at once -- so
// a pass first counts: each CTA takes a contiguous run of items (words or rows,
// or groups of eight variables of them) and leaves its total; after a barrier
// every warp knows its first position and decides its run of items from there,
// the offsets inside it by shuffles, each thread one short jump of the stream and
// then a step a draw.  Nothing waits on a predecessor's look-back, which is what bounded the
// pass before (one CTA, kLocal, needs no totals either).
//
// us a sweep, per-pass launches / this: Ising Metropolis 64^2 12.3 / 4.2, 1024^2
// 16.8 / 15.0, 256^3 82 / 68, 250^3 (rows that suit no vector) 229 / 75, 512^3 562 /
// 396; Ising heat bath 250^3 169 / 49; gauge 24^4 heat bath 66 / 34, Metropolis 131 /
// 53.  Large passes are bound by issue, some 75 instructions a site of which the
// LCG step is 18 and its output function 10 a draw (a kernel of nothing else makes
// 900 draws/ns); small ones by a thread's chain of eight draws and its jumps.
constexpr int kStreamMaxGrid = 1024;

struct StreamShared {
    unsigned long long cut[16];  // cut points << 11: compared with all 64 bits of a draw
    u128 pass_base, next_base;   // stream states of this pass's and the next's first draw
    unsigned long long prefix, total;
    uint32_t warp_sum[kResidentThreads / 32];
    uint32_t draws;              // bit key: a variable of that key draws
};

// Bits where the key cur + 2 * count (bit-sliced) has its bit set in `keys`.
__device__ __forceinline__ uint64_t keys_in(uint32_t keys, uint64_t cur, uint64_t c0, uint64_t c1, uint64_t c2) {
    uint64_t leaf[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const uint64_t t0 = 0ull - ((keys >> (2 * k)) & 1u), t1 = 0ull - ((keys >> (2 * k + 1)) & 1u);
        leaf[k] = (t0 & ~cur) | (t1 & cur);
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) leaf[k] = (leaf[2 * k] & ~c0) | (leaf[2 * k + 1] & c0);
#pragma unroll
    for (int k = 0; k < 2; ++k) leaf[k] = (leaf[2 * k] & ~c1) | (leaf[2 * k + 1] & c1);
    return (leaf[0] & ~c2) | (leaf[1] & c2);
}

// One unit (a word of sites, a row of links) in a pass: its bits, and the state
// and counter planes of its pass variables at even bits 2j.
struct UnitPlanes {
    uint64_t C, cur, c0, c1, c2, valid;
    int x0, n;
};

template <int D, int MU, class W>
__device__ __forceinline__ int link_unit(const ResidentArgs &a, const LocalArgs &p, const W *pk, uint32_t r, UnitPlanes &t) {
    int32_t op[4] = {0, 0, 0, 0}, om[4] = {0, 0, 0, 0};
    const int par = row_geometry<D>(p.g, r, op, om);
    W U, c0, c1, c2;
    link_row<D, MU, W>((uint32_t)p.g.L[0], a.units, pk, r, op, om, U, c0, c1, c2);
    t.C = U;
    t.c0 = c0;
    t.c1 = c1;
    t.c2 = c2;
    return par;
}

template <ResidentKind K>
__device__ __forceinline__ UnitPlanes unit_planes(const ResidentArgs &a, const LocalArgs &p, const void *words, uint32_t u) {
    UnitPlanes t;
    int par;
    if (K == ResidentKind::kSites) {
        const uint64_t *pk = static_cast<const uint64_t *>(words);
        const SiteWord s = site_word(a, u);
        int32_t op[4] = {0, 0, 0, 0}, om[4] = {0, 0, 0, 0};
        par = p.g.d == 2 ? row_geometry<2>(p.g, s.r, op, om) : row_geometry<3>(p.g, s.r, op, om);
        t.n = (int)(s.len / 2);
        t.C = pk[u];
        t.c0 = t.c1 = t.c2 = 0;
        count_add(t.c0, t.c1, t.c2, word_right(a, pk, s, t.C));
        count_add(t.c0, t.c1, t.c2, word_left(a, pk, s, t.C));
        const uint32_t wpr = a.words_per_row;
        count_add(t.c0, t.c1, t.c2, pk[u + (uint32_t)op[1] * wpr]);
        count_add(t.c0, t.c1, t.c2, pk[u + (uint32_t)om[1] * wpr]);
        if (p.g.d == 3) {
            count_add(t.c0, t.c1, t.c2, pk[u + (uint32_t)op[2] * wpr]);
            count_add(t.c0, t.c1, t.c2, pk[u + (uint32_t)om[2] * wpr]);
        }
    } else {
        using W = typename std::conditional<K == ResidentKind::kLinks32, uint32_t, uint64_t>::type;
        const W *pk = static_cast<const W *>(words);
        t.n = p.g.L[0] / 2;
        switch (p.g.d * 4 + p.dir) {
            case 8: par = link_unit<2, 0, W>(a, p, pk, u, t); break;
            case 9: par = link_unit<2, 1, W>(a, p, pk, u, t); break;
            case 12: par = link_unit<3, 0, W>(a, p, pk, u, t); break;
            case 13: par = link_unit<3, 1, W>(a, p, pk, u, t); break;
            case 14: par = link_unit<3, 2, W>(a, p, pk, u, t); break;
            case 16: par = link_unit<4, 0, W>(a, p, pk, u, t); break;
            case 17: par = link_unit<4, 1, W>(a, p, pk, u, t); break;
            case 18: par = link_unit<4, 2, W>(a, p, pk, u, t); break;
            default: par = link_unit<4, 3, W>(a, p, pk, u, t); break;
        }
    }
    t.x0 = (p.color ^ par) & 1;
    t.cur = t.C >> t.x0;
    t.c0 >>= t.x0;
    t.c1 >>= t.x0;
    t.c2 >>= t.x0;
    t.valid = 0x5555555555555555ull & low_bits((uint32_t)(2 * t.n));
    return t;
}

// Item i: unit i / groups, all of its variables or (groups > 1) the eight of group i % groups.
struct StreamItem {
    uint32_t u;
    int first;      // first group
    uint64_t mine;  // bits of the item's variables
};
__device__ __forceinline__ StreamItem stream_item(const ResidentArgs &a, uint32_t i) {
    StreamItem t;
    t.u = fdiv(i, a.groups_m, a.groups_l);
    t.first = (int)(i - t.u * a.groups);
    t.mine = a.groups == 1 ? ~0ull : 0xFFFFull << (16 * t.first);
    return t;
}

// unit_planes of a word whose geometry is kept (SiteGroup, without the heads).
__device__ __forceinline__ UnitPlanes site_planes(const LocalArgs &p, const SiteGroup &g, const uint64_t *pk) {
    UnitPlanes t;
    t.n = g.n;
    t.C = pk[g.u];
    const uint64_t right = pk[g.at[0]], left = pk[g.at[1]];
    t.c0 = t.c1 = t.c2 = 0;
    count_add<uint64_t>(t.c0, t.c1, t.c2, (t.C >> 1) | (right & 1ull) << (g.len - 1u));
    count_add<uint64_t>(t.c0, t.c1, t.c2, (t.C << 1 | ((left >> g.left_bit) & 1ull)) & low_bits(g.len));
    count_add(t.c0, t.c1, t.c2, pk[g.at[2]]);
    count_add(t.c0, t.c1, t.c2, pk[g.at[3]]);
    if (p.g.d == 3) {
        count_add(t.c0, t.c1, t.c2, pk[g.at[4]]);
        count_add(t.c0, t.c1, t.c2, pk[g.at[5]]);
    }
    t.x0 = p.color ^ g.par;
    t.cur = t.C >> t.x0;
    t.c0 >>= t.x0;
    t.c1 >>= t.x0;
    t.c2 >>= t.x0;
    t.valid = 0x5555555555555555ull & low_bits((uint32_t)(2 * t.n));
    return t;
}

// Variables of the pass before the item's first (heat bath: its draw's position in the pass).
template <ResidentKind K>
__device__ __forceinline__ unsigned long long item_rank(const ResidentArgs &a, const StreamItem &it) {
    const unsigned long long half = (unsigned long long)(a.p.g.L[0] / 2);
    if (K == ResidentKind::kSites) {
        const SiteWord s = site_word(a, it.u);
        return s.r * half + 32u * s.w + min(8u * (unsigned)it.first, s.len / 2u);  // (a short word's last groups are empty)
    }
    return it.u * half + 8u * (unsigned)it.first;
}

// XSL-RR's high word: the rotation of (x1, x0) right by hi >> 58.
__device__ __forceinline__ uint32_t xsl_rr_high(u128 s) {
    const uint32_t x0 = (uint32_t)s.lo ^ (uint32_t)s.hi, x1 = (uint32_t)(s.lo >> 32) ^ (uint32_t)(s.hi >> 32);
    const uint32_t top = (uint32_t)(s.hi >> 32);
    const bool swap = (int32_t)top < 0;
    return __funnelshift_r(swap ? x0 : x1, swap ? x1 : x0, top >> 26);
}

// The draws of one group of eight (bits 2i of need) from stream state st, which
// moves on by their number: bits 2i where a draw is below its key's cut point.
// The high words decide unless they are equal (once in 2^32 draws), which sends
// the group to the second, whole comparison.  No branches: a warp's lanes differ
// in almost every bit of need, and eight draws' loads and rotations overlap.
template <bool ALL>
__device__ __forceinline__ uint32_t draws_below(uint32_t x, uint32_t need, u128 &st, const u128 &inc,
                                                const unsigned long long *cut) {
    const u128 st0 = st;
    uint32_t o = 0;
    bool equal = false;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const uint32_t e = (uint32_t)(cut[(x >> (4 * i)) & 15u] >> 32);
        const uint32_t k = xsl_rr_high(st);
        if (k < e) o |= 1u << (2 * i);
        equal |= k == e;
        const u128 next = pcg_step(st, inc);
        if (ALL) {
            st = next;
        } else {
            const bool take = (need >> (2 * i)) & 1u;
            st.lo = take ? next.lo : st.lo;
            st.hi = take ? next.hi : st.hi;
        }
    }
    if (equal) {
        u128 t = st0;
        o = 0;
#pragma unroll 1
        for (int i = 0; i < 8; ++i) {
            if (xsl_rr(t) < cut[(x >> (4 * i)) & 15u]) o |= 1u << (2 * i);
            if (ALL || ((need >> (2 * i)) & 1u)) t = pcg_step(t, inc);
        }
    }
    return o;
}

// The item's draws from stream state st: its flips.
template <bool HB>
__device__ __forceinline__ uint64_t stream_decide(const ResidentArgs &a, const UnitPlanes &t, const StreamItem &it,
                                                  uint64_t draws, u128 st, const u128 &inc, const unsigned long long *cut) {
    const uint64_t M = 0x5555555555555555ull;
    const uint64_t P = (t.cur & M) | ((t.c0 << 1) & ~M), Q = (t.c1 & M) | ((t.c2 << 1) & ~M);
    uint64_t out = 0;
    const int end = a.groups == 1 ? (t.n + 7) / 8 : it.first + 1;
#pragma unroll 1
    for (int c = it.first; c < end; ++c)
        out |= (uint64_t)draws_below<HB>(key_word(P, Q, c), (uint32_t)(draws >> (16 * c)), st, inc, cut) << (16 * c);
    // heat bath: the new state is 1 where the draw is not below; Metropolis: downhill moves are taken
    // without a draw, the others where it is below
    const uint64_t flip = HB ? ~out ^ t.cur : out | ~draws;
    return flip & t.valid & it.mine;
}

// S: kStream, a warp takes its run of items in turn; kGroups, one item a thread at
// most, whose place and geometry are kept over the launch and whose planes over a
// pass; kLocal, the same in one CTA with the words in its shared memory.
template <ResidentKind K, bool HB, Share S>
__global__ void __launch_bounds__(S == kLocal ? kResidentThreads : kGridThreads, S == kLocal ? 1 : S == kGroups ? 2 : 4)
stream_kernel(const __grid_constant__ ResidentArgs a) {
    extern __shared__ __align__(16) unsigned char s_words[];
    __shared__ LocalArgs s_args;
    __shared__ StreamShared sh;
    __shared__ int s_counts[64];
    void *pk = S == kLocal ? s_words : a.packed;
    unsigned long long arrived = a.arrived;
    if (threadIdx.x == 0) {
        s_args = a.p;
        uint32_t draws = 0;
        for (int k = 0; k < 16; ++k) {
            const unsigned long long e = k < a.n_keys ? (HB ? a.p.hb53[k] : a.p.metro53[k]) : 0ull;
            sh.cut[k] = e << 11;
            if (HB || e != ~0ull) draws |= 1u << k;
        }
        sh.draws = draws;
        sh.pass_base = jump(a.p.jump, a.p.base, HB ? a.p.pass_offset : a.p.ctrl->pos[a.p.pos_in]);
    }
    unsigned long long position = HB ? 0ull : a.p.ctrl->pos[a.p.pos_in];
    repack<K>(a, pk, true);
    resident_barrier(a, arrived);
    const uint32_t draws_of = sh.draws;
    const int passes = a.p.model == PLQ_GAUGE ? 2 * a.p.g.d : 2;
    const bool sampling = a.snapshots || a.primaries;
    // a warp's items are a contiguous run, so that offsets inside it take no barrier of the block
    const uint32_t items = a.units * a.groups;
    const uint32_t warps = blockDim.x >> 5, lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
    const uint32_t share = (items + gridDim.x * warps - 1) / (gridDim.x * warps);
    const uint32_t i0 = min(items, (blockIdx.x * warps + wid) * share), i1 = min(items, i0 + share);
    constexpr bool once = S != kStream;
    StreamItem own{0, 0, 0};
    SiteGroup geometry;
    if (once && i0 + lane < i1) {
        own = stream_item(a, i0 + lane);
        if (K == ResidentKind::kSites)
            geometry = a.p.g.d == 2 ? site_group<2, false>(a, i0 + lane) : site_group<3, false>(a, i0 + lane);
    }
    uint32_t parity = 0;
    for (uint64_t sample = 0; sample < a.samples; ++sample) {
        for (uint64_t t = 0; t < a.sweeps; ++t) {
            for (int pass = 0; pass < passes; ++pass) {
                if (threadIdx.x == 0) {
                    s_args.dir = a.p.model == PLQ_GAUGE ? pass >> 1 : 0;
                    s_args.color = pass & 1;
                }
                __syncthreads();
                UnitPlanes u{};
                uint64_t draws = 0;
                if (once && i0 + lane < i1) {
                    if (K == ResidentKind::kSites) u = site_planes(s_args, geometry, static_cast<const uint64_t *>(pk));
                    else u = unit_planes<K>(a, s_args, pk, own.u);
                    draws = (HB ? ~0ull : keys_in(draws_of, u.cur, u.c0, u.c1, u.c2)) & u.valid & own.mine;
                }
                // ---- where the CTA's and the warp's draws start
                unsigned long long first;  // of the warp, in the pass
                if (!HB) {
                    uint32_t sum = once ? (uint32_t)__popcll(draws) : 0u;
                    for (uint32_t i = once ? i1 : i0 + lane; i < i1; i += 32) {
                        const StreamItem it = stream_item(a, i);
                        const UnitPlanes u = unit_planes<K>(a, s_args, pk, it.u);
                        sum += __popcll(keys_in(draws_of, u.cur, u.c0, u.c1, u.c2) & u.valid & it.mine);
                    }
                    sum = __reduce_add_sync(0xffffffffu, sum);
                    if (lane == 0) sh.warp_sum[wid] = sum;
                    __syncthreads();
                    uint32_t before = 0, total = 0;
                    for (uint32_t k = 0; k < warps; ++k) {
                        const uint32_t v = sh.warp_sum[k];
                        before += k < wid ? v : 0u;
                        total += v;
                    }
                    if (gridDim.x > 1) {
                        if (threadIdx.x == 0) a.totals[parity * kStreamMaxGrid + blockIdx.x] = total;
                        resident_barrier(a, arrived);
                        if (wid == 0) {
                            unsigned long long lower = 0, all = 0;
                            for (unsigned k = lane; k < gridDim.x; k += 32) {
                                const unsigned long long v = __ldcg(&a.totals[parity * kStreamMaxGrid + k]);
                                all += v;
                                lower += k < blockIdx.x ? v : 0ull;
                            }
#pragma unroll
                            for (int off = 16; off > 0; off >>= 1) {
                                lower += __shfl_xor_sync(0xffffffffu, lower, off);
                                all += __shfl_xor_sync(0xffffffffu, all, off);
                            }
                            if (lane == 0) {
                                sh.prefix = lower;
                                sh.total = all;
                            }
                        }
                        __syncthreads();
                        parity ^= 1u;
                        first = sh.prefix + before;
                        position += sh.total;
                    } else {
                        if (threadIdx.x == 0) sh.total = total;
                        first = before;
                        position += total;
                    }
                } else {
                    first = item_rank<K>(a, stream_item(a, min(i0, items - 1u)));
                    if (threadIdx.x == 0) sh.total = (unsigned long long)(a.p.g.n_sites / 2);
                }
                __syncthreads();  // (the total; the warps' sums are read)
                // one jump per warp (lane 0: to its first draw; lane 31, alike: to the next pass), then
                // the items, each thread a short jump from the warp's state
                u128 base{0, 0};
                if (lane == 0 || lane == 31) base = jump(a.p.jump, sh.pass_base, lane == 0 ? first : sh.total);
                if (threadIdx.x == blockDim.x - 1) sh.next_base = base;
                base.lo = __shfl_sync(0xffffffffu, base.lo, 0);
                base.hi = __shfl_sync(0xffffffffu, base.hi, 0);
                uint32_t run = 0;
                for (uint32_t i = i0 + lane; i - lane < i1; i += 32) {
                    StreamItem it = own;
                    if (!once && i < i1) {
                        it = stream_item(a, i);
                        u = unit_planes<K>(a, s_args, pk, it.u);
                        draws = (HB ? ~0ull : keys_in(draws_of, u.cur, u.c0, u.c1, u.c2)) & u.valid & it.mine;
                    } else if (!once) {
                        draws = 0;
                    }
                    uint32_t at;
                    if (HB) {
                        at = i < i1 ? (uint32_t)(item_rank<K>(a, it) - first) : 0u;
                    } else {
                        const uint32_t mine = (uint32_t)__popcll(draws);
                        uint32_t incl = mine;
#pragma unroll
                        for (int off = 1; off < 32; off <<= 1) {
                            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, off);
                            if (lane >= (uint32_t)off) incl += y;
                        }
                        at = run + incl - mine;
                        run += __shfl_sync(0xffffffffu, incl, 31);
                    }
                    if (i < i1) {
                        const u128 st = jump(a.p.jump, base, at);
                        const uint64_t flip = stream_decide<HB>(a, u, it, draws, st, a.p.inc, sh.cut);
                        const uint64_t now = u.C ^ (flip << u.x0);
                        if (a.groups > 1) {
                            constexpr uint32_t kHalves = K == ResidentKind::kLinks32 ? 2 : 4;
                            uint16_t *h = static_cast<uint16_t *>(pk) +
                                          ((size_t)(K == ResidentKind::kSites ? 0u : (uint32_t)s_args.dir * a.units) + it.u) * kHalves;
                            if (8 * it.first < u.n) h[it.first] = (uint16_t)(now >> (16 * it.first));
                        } else if (K == ResidentKind::kSites) {
                            static_cast<uint64_t *>(pk)[it.u] = now;
                        } else if (K == ResidentKind::kLinks32) {
                            static_cast<uint32_t *>(pk)[(uint32_t)s_args.dir * a.units + it.u] = (uint32_t)now;
                        } else {
                            static_cast<uint64_t *>(pk)[(uint32_t)s_args.dir * a.units + it.u] = now;
                        }
                    }
                }
                resident_barrier(a, arrived);
                if (threadIdx.x == 0) sh.pass_base = sh.next_base;
            }
        }
        if (sampling) {
            take_sample<K>(a, pk, sample, s_counts);
            if (sample + 1 < a.samples) resident_barrier(a, arrived);
        }
    }
    if (!HB && blockIdx.x == 0 && threadIdx.x == 0) a.p.ctrl->pos[a.p.pos_in] = position;
    repack<K>(a, pk, false);
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
// Whether the device takes the plan's cluster of kGroups CTAs.
template <ResidentKind K>
bool cluster_fits(const ResidentPlan &p) {
    if (p.grid <= 8) return true;  // the portable size
    auto kern = resident_kernel<K, kGroups>;
    int clusters = 0;
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr{};
    resident_config(p, cfg, attr, nullptr);
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg);
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
                p.shared_bytes = p.packed_bytes;  // (at most 8 KB: 512 rows of four directions)
                return cudaSuccess;
            }
            p.share = kGroups;
            if (items <= kClusterCtas * kResidentThreads) {
                p.grid = power_of_two_at_least((warps + 3) / 4);  // at least four warps a CTA
                if (p.grid > kClusterCtas) p.grid = kClusterCtas;
                p.block = (int)((warps + p.grid - 1) / p.grid) * 32;
                if (cluster_fits<K>(p)) return cudaSuccess;
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

// The launch shape on the PCG stream: groups, one a thread, while they fill no more than the
// chip (in one CTA, a cluster, a grid); else whole units.
template <ResidentKind K, bool HB>
cudaError_t plan_stream(ResidentPlan &p, int sm_count) {
    const uint32_t items = p.units * p.most_groups;
    p.cluster = true;
    if (items <= kResidentThreads) {
        p.share = kLocal;
        p.groups = p.most_groups;
        p.grid = 1;
        p.block = (int)((items + 31) / 32 * 32);
        p.shared_bytes = p.packed_bytes;  // (at most 8 KB, as above)
        return cudaSuccess;
    }
    p.block = kGridThreads;
    if (items <= (uint32_t)sm_count * 2 * kGridThreads) {
        p.share = kGroups;
        p.groups = p.most_groups;
        p.grid = (items + kGridThreads - 1) / kGridThreads;
        if (p.grid <= 8) p.grid = power_of_two_at_least(p.grid);
        else p.cluster = false;
        return cudaSuccess;
    }
    p.share = kStream;
    p.groups = 1;
    p.cluster = false;
    int per_sm = 0;
    const cudaError_t e =
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, stream_kernel<K, HB, kStream>, kGridThreads, 0);
    p.grid = std::min((p.units + kGridThreads - 1) / kGridThreads,
                      std::min((unsigned)(per_sm * sm_count), (unsigned)kStreamMaxGrid));
    return e != cudaSuccess || p.grid > 0 ? e : cudaErrorLaunchOutOfResources;
}

template <ResidentKind K>
cudaError_t launch_stream_kind(const ResidentPlan &p, const ResidentArgs &a, cudaStream_t stream) {
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr{};
    resident_config(p, cfg, attr, stream);
    const bool hb = a.p.kernel == PLQ_HEATBATH;
    switch (p.share) {
        case kLocal:
            return hb ? cudaLaunchKernelEx(&cfg, stream_kernel<K, true, kLocal>, a)
                      : cudaLaunchKernelEx(&cfg, stream_kernel<K, false, kLocal>, a);
        case kGroups:
            return hb ? cudaLaunchKernelEx(&cfg, stream_kernel<K, true, kGroups>, a)
                      : cudaLaunchKernelEx(&cfg, stream_kernel<K, false, kGroups>, a);
        default:
            return hb ? cudaLaunchKernelEx(&cfg, stream_kernel<K, true, kStream>, a)
                      : cudaLaunchKernelEx(&cfg, stream_kernel<K, false, kStream>, a);
    }
}

template <ResidentKind K>
cudaError_t plan_packed(ResidentPlan &p, bool stream_draws, bool heat_bath, int sm_count) {
    if (!stream_draws) return plan_kind<K>(p, sm_count);
    p.stream_draws = true;
    p.barriers_per_pass = heat_bath ? 1 : 2;  // (a grid's; its totals' barrier)
    return heat_bath ? plan_stream<K, true>(p, sm_count) : plan_stream<K, false>(p, sm_count);
}

}  // namespace

ResidentKind resident_kind(int model, int q, int d, const int32_t *L, int updater, int rng, bool words) {
    if (updater == PLQ_METROPOLIS || updater == PLQ_HEATBATH) {
        if (model == PLQ_GAUGE && d >= 2 && d <= 4 && L[0] <= 64)
            return L[0] <= 32 ? ResidentKind::kLinks32 : ResidentKind::kLinks64;
        if (model != PLQ_GAUGE && q == 2 && (d == 2 || d == 3)) return ResidentKind::kSites;
    }
    // (Metropolis on the stream elsewhere: its draws' positions depend on the pass's decisions)
    if (d > 4 || (rng == PLQ_RNG_STREAM && updater == PLQ_METROPOLIS)) return ResidentKind::kNone;
    if (rng == PLQ_RNG_KEYED && model != PLQ_GAUGE && !words) return ResidentKind::kRanks;
    return words ? ResidentKind::kWords : ResidentKind::kGeneric;
}

cudaError_t resident_plan(ResidentKind kind, const Geom &g, bool stream_draws, bool heat_bath, int sm_count,
                          ResidentPlan &p) {
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
            return plan_packed<ResidentKind::kSites>(p, stream_draws, heat_bath, sm_count);
        case ResidentKind::kLinks32:
            p.units = rows;
            p.packed_bytes = (size_t)rows * (size_t)g.d * sizeof(uint32_t);
            p.most_groups = (uint32_t)(g.L[0] + 15) / 16;
            return plan_packed<ResidentKind::kLinks32>(p, stream_draws, heat_bath, sm_count);
        case ResidentKind::kLinks64:
            p.units = rows;
            p.packed_bytes = (size_t)rows * (size_t)g.d * sizeof(uint64_t);
            p.most_groups = (uint32_t)(g.L[0] + 15) / 16;
            return plan_packed<ResidentKind::kLinks64>(p, stream_draws, heat_bath, sm_count);
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
    return (packed ? 1 : 0) + samples * sweeps * (uint64_t)(passes * p.barriers_per_pass) + (sampling && samples ? samples - 1 : 0);
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
        case ResidentKind::kSites:
            return p.stream_draws ? launch_stream_kind<ResidentKind::kSites>(p, a, stream)
                                  : launch_kind<ResidentKind::kSites>(p, a, stream);
        case ResidentKind::kLinks32:
            return p.stream_draws ? launch_stream_kind<ResidentKind::kLinks32>(p, a, stream)
                                  : launch_kind<ResidentKind::kLinks32>(p, a, stream);
        case ResidentKind::kLinks64:
            return p.stream_draws ? launch_stream_kind<ResidentKind::kLinks64>(p, a, stream)
                                  : launch_kind<ResidentKind::kLinks64>(p, a, stream);
        case ResidentKind::kWords: return launch_kind<ResidentKind::kWords>(p, a, stream);
        case ResidentKind::kRanks: return launch_kind<ResidentKind::kRanks>(p, a, stream);
        case ResidentKind::kGeneric: return launch_kind<ResidentKind::kGeneric>(p, a, stream);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace plq
