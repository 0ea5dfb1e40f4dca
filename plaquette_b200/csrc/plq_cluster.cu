// plq_cluster.cu -- Swendsen-Wang and Wolff chains on the device.
//
// One cluster sweep of ClusterUpdate::sweep (src/updater.rs:541-613) /
// GpuClusterChain::run_sweep (src/gpu_cluster.rs:492-526):
//
//  1. bonds  -- a forward bond (site, axis) opens iff the two sites agree and
//               the draw is below p = 1 - exp(-beta * gap) (the host computes
//               p as ClusterUpdate::bond_probability does).  Keyed stream: the
//               draw is keyed by the bond index (cluster_prelude.wgsl:61-80).
//               PCG stream: one draw per *agreeing* bond in site-major,
//               axis-minor order (cluster.rs:44-62), placed by a device-wide
//               exclusive scan (decoupled look-back) over agreeing bonds.
//  2. labels -- lock-free union-find: every open bond unites its ends by
//               hooking the larger root under the smaller (an atomic minimum), first
//               inside a tile in shared memory (tile_hook_kernel), then
//               for the bonds that leave a tile (boundary_hook_kernel); the
//               relabel pass walks each tile-local root to its cluster's root
//               and hands that to the sites of the tile.  Roots only
//               ever hook under smaller roots, so each component ends rooted
//               at its minimum site: the canonical min-site label of the
//               reference GPU (the fixed point of cluster_prelude.wgsl:113-147),
//               and, ranked, the reference CPU's first-encounter compaction
//               (cluster.rs:199-226).
//  3. relabel -- keyed: per-root keyed draw (cluster_relabel.wgsl:39-90).
//               PCG stream: clusters in root order draw next_below(q) (or the
//               forced-change proposal) at consecutive positions, inside the
//               rank scan; rand's range sampler occasionally takes a second
//               draw, which shifts every later cluster -- the scan lists the
//               outputs that do, and the pass that hands the labels to the sites
//               draws the shifted ones again (SecondDraws).
//
// Wolff on the keyed stream: the reference relabels the cluster of a keyed
// seed site in the full decomposition (cluster_relabel.wgsl:55-66).  Here one
// persistent launch runs all requested updates: a CTA grows the cluster from
// the seed site for a few generations while the others label the tiles
// (wolff_kernel); its minimum site is the root the forced change is keyed on.
// Wolff on the PCG stream (draws in grow_cluster's FIFO order) is sequential by definition and is not run on the device.
//
// Every loop that waits or retries has an iteration cap; hitting one sets a
// status bit the host turns into PLQ_ECAP / PLQ_EDEVICE.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>
#include <vector>

#include "../../include/plaquette.h"
#include "plq_cluster.h"
#include "plq_device.cuh"
#include "plq_geom.cuh"
#include "plq_local.h"
#include "plq_readback.h"
#include "plq_second_draws.h"
#include "plq_tables.h"
#include "plq_wolff_sync.h"

using namespace plq;

namespace {

constexpr int kThreads = 256;
constexpr int kSitesPerThread = 8;
constexpr int kChunk = kThreads * kSitesPerThread;
constexpr int kSpinLimit = 1 << 22;
constexpr int kMaxEvents = 64;
constexpr unsigned long long kDescAgg = 1ull, kDescPrefix = 2ull;

struct ClusterArgs {
    uint8_t *state;
    uint8_t *bonds;
    int32_t *parent;      // union-find over the tile-local roots (flat over all sites after flatten_kernel)
    uint16_t *local_root; // every site's tile-local root: by tile, then the place in the tile
    uint8_t *fresh;
    int32_t *rank;
    struct ChunkBase {     // stream relabel: per root_rank chunk, the state at the label draw of
        u128 st;           // the chunk's first root (no second draws before it) and that root's rank
        int64_t rank0, pad;
    } *chunk_base;
    Geom g;
    int q;
    int extent, relabel;
    uint32_t seed32, sweep32;
    uint32_t kp24;   // keyed: bond open iff k24 < kp24
    uint64_t kp53;   // stream: bond open iff k53 < kp53
    const Affine *jump;
    u128 inc;
    u128 *at;        // stream states: of the draw at ctrl->pos[0] (the sweep's first), and at pos[1] (its first label)
    Control *ctrl;
    unsigned long long *desc;
    int64_t n_chunks;
    uint64_t ticket_base;
    uint32_t epoch;
    int cap;          // iteration cap of finds and unions
    int32_t *events;   // stream relabel: label outputs that ask for a second draw (places from the first label)
    int *event_count;  // ... their number; the list holds the first kMaxEvents
    uint64_t updates; // Wolff: updates in this launch
};

// The launches of a Swendsen-Wang sweep follow each other without a gap: each may take its
// place on the SMs once the one before has started everywhere (programmatic dependent
// launch), and waits here for its end.
__device__ __forceinline__ void after_previous() {
    cudaGridDependencySynchronize();
    cudaTriggerProgrammaticLaunchCompletion();
}
template <class... P, class... A>
void launch_next(void (*kernel)(P...), unsigned grid, cudaStream_t stream, A... args) {
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(kThreads);
    cfg.stream = stream;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    (void)cudaLaunchKernelEx(&cfg, kernel, args...);  // (the sweep asks for the last error)
}

__device__ __forceinline__ unsigned long long ld_relaxed(const unsigned long long *p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ int32_t ld_relaxed32(const int32_t *p) {
    int32_t v;
    asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ unsigned long long make_desc(uint32_t epoch, unsigned long long st, uint32_t value) {
    return ((unsigned long long)(epoch & 0x3FFFFFFFu) << 34) | (st << 32) | value;
}

// Block-wide exclusive scan of `v` with decoupled look-back across chunks
// (taken in ticket order).  Returns the thread's global exclusive prefix and,
// through block_total / ok, the chunk total and whether the wait completed.
__device__ uint64_t chunk_scan(const ClusterArgs &a, int64_t chunk, int v, int &block_total, bool &ok) {
    __shared__ int warp_tot[kThreads / 32];
    __shared__ unsigned long long s_excl;
    __shared__ int s_fail;
    int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int incl = v;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        int y = __shfl_up_sync(0xffffffffu, incl, off);
        if (lane >= off) incl += y;
    }
    if (lane == 31) warp_tot[wid] = incl;
    if (threadIdx.x == 0) s_fail = 0;
    __syncthreads();
    int warp_excl = 0, total = 0;
#pragma unroll
    for (int w = 0; w < kThreads / 32; ++w) {
        int t = warp_tot[w];
        if (w < wid) warp_excl += t;
        total += t;
    }
    // Warp 0 looks back over 32 predecessors per round: the nearest one with an inclusive
    // prefix ends the walk, and the aggregates up to it are summed with one warp reduction.
    if (wid == 0) {
        unsigned long long excl = 0;
        bool fail = false;
        if (chunk == 0) {
            if (lane == 0) atomicExch(&a.desc[0], make_desc(a.epoch, kDescPrefix, (uint32_t)total));
        } else {
            if (lane == 0) atomicExch(&a.desc[chunk], make_desc(a.epoch, kDescAgg, (uint32_t)total));
            const uint32_t ep = a.epoch & 0x3FFFFFFFu;
            int64_t top = chunk - 1;
            int spins = 0;
            while (true) {
                const int64_t idx = top - lane;
                // before chunk 0: an inclusive prefix of 0
                const unsigned long long d = idx >= 0 ? ld_relaxed(&a.desc[idx]) : make_desc(a.epoch, kDescPrefix, 0u);
                const unsigned long long st = (uint32_t)(d >> 34) == ep ? (d >> 32) & 3ull : 0ull;
                const unsigned incl_lanes = __ballot_sync(0xffffffffu, st == kDescPrefix);
                const unsigned ready = __ballot_sync(0xffffffffu, st != 0ull);
                // lanes up to the nearest inclusive prefix (all 32 when none is in this window)
                const unsigned span = incl_lanes ? (((incl_lanes & (0u - incl_lanes)) << 1) - 1u) : 0xffffffffu;
                if ((ready & span) != span) {
                    if (++spins > kSpinLimit) {
                        fail = true;
                        break;
                    }
                    __nanosleep(32);
                    continue;
                }
                unsigned long long v = ((span >> lane) & 1u) ? (unsigned long long)(uint32_t)d : 0ull;
#pragma unroll
                for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
                excl += v;
                if (incl_lanes) break;
                top -= 32;
            }
            if (lane == 0 && !fail) atomicExch(&a.desc[chunk], make_desc(a.epoch, kDescPrefix, (uint32_t)(excl + total)));
        }
        if (lane == 0) {
            if (fail) {
                s_fail = 1;
                atomicOr(&a.ctrl->status, kStatusLookbackTimeout);
            }
            s_excl = excl;
        }
    }
    __syncthreads();
    ok = s_fail == 0;
    block_total = total;
    return s_excl + (uint64_t)(warp_excl + incl - v);
}

__device__ __forceinline__ int64_t take_chunk(const ClusterArgs &a, bool lookback) {
    if (!lookback) return blockIdx.x;
    __shared__ unsigned long long s_ticket;
    if (threadIdx.x == 0) s_ticket = atomicAdd(&a.ctrl->ticket, 1ull) - a.ticket_base;
    __syncthreads();
    return (int64_t)s_ticket;
}

// ------------------------------------------------------------- 1. bonds
static_assert(kSitesPerThread == 8, "the bonds pass loads and stores a thread's sites as one 8-byte word");

// High bit of each byte of the result set iff that byte of a equals that of b.
__device__ __forceinline__ uint64_t bytes_equal(uint64_t a, uint64_t b) {
    const uint64_t e = a ^ b, lo7 = 0x7F7F7F7F7F7F7F7Full;
    return ~(((e & lo7) + lo7) | e) & ~lo7;
}

template <int D, bool STREAM>
__global__ void __launch_bounds__(kThreads) bonds_kernel(ClusterArgs a) {
    after_previous();
    const int64_t n = a.g.n_sites;
    const int64_t chunk = take_chunk(a, STREAM);
    if (chunk >= a.n_chunks) {
        if (threadIdx.x == 0) atomicOr(&a.ctrl->status, kStatusBounds);
        return;
    }
    const int64_t s0 = chunk * kChunk + (int64_t)threadIdx.x * kSitesPerThread;
    // With L0 % 8 == 0 a thread's 8 sites (s0 is a multiple of 8) lie in one row, and every
    // +mu neighbour row is 8-byte aligned: one vector load per direction, one vector store.
    const bool row8 = (a.g.L[0] & 7) == 0;
    uint8_t agree[kSitesPerThread];
    int count = 0;
    if (row8) {
#pragma unroll
        for (int i = 0; i < kSitesPerThread; ++i) agree[i] = 0;
        if (s0 < n) {
            int32_t x[D];
            site_coords<D>(a.g, s0, x);
            const uint64_t cv = *reinterpret_cast<const uint64_t *>(a.state + s0);
            // +x: bytes s0+1 .. s0+8, the last one wrapping to the row start
            const int64_t past = x[0] + kSitesPerThread < a.g.L[0] ? s0 + kSitesPerThread
                                                                   : s0 + kSitesPerThread - a.g.L[0];
            uint64_t eq[D];
            eq[0] = bytes_equal(cv, (cv >> 8) | ((uint64_t)a.state[past] << 56));
#pragma unroll
            for (int mu = 1; mu < D; ++mu)
                eq[mu] = bytes_equal(cv, *reinterpret_cast<const uint64_t *>(a.state + nbr_plus(a.g, s0, x, mu)));
#pragma unroll
            for (int i = 0; i < kSitesPerThread; ++i) {
                uint32_t m = 0;
#pragma unroll
                for (int mu = 0; mu < D; ++mu) m |= (uint32_t)((eq[mu] >> (8 * i + 7)) & 1u) << mu;
                agree[i] = (uint8_t)m;
                count += __popc(m);
            }
        }
    } else {
#pragma unroll
        for (int i = 0; i < kSitesPerThread; ++i) {
            int64_t s = s0 + i;
            agree[i] = 0;
            if (s >= n) continue;
            int32_t x[D];
            site_coords<D>(a.g, s, x);
            uint8_t cur = a.state[s];
            uint8_t m = 0;
#pragma unroll
            for (int mu = 0; mu < D; ++mu)
                if (a.state[nbr_plus(a.g, s, x, mu)] == cur) m |= (uint8_t)(1u << mu);
            agree[i] = m;
            count += __popc(m);
        }
    }
    u128 st{0, 0}, chunk_state{0, 0};
    uint64_t chunk_draws = 0;
    if (STREAM) {
        int total;
        bool ok;
        uint64_t excl = chunk_scan(a, chunk, count, total, ok);
        if (!ok) return;
        chunk_draws = (uint64_t)total;
        // One full jump per chunk, to its first draw (thread 0's prefix is the chunk's); each
        // thread then applies the low digits of its offset inside the chunk (< kChunk * D draws).
        // Jump maps are iterates of one affine map, so they compose in any order.
        __shared__ unsigned long long s_base, s_excl0;
        __shared__ u128 s_state;
        if (threadIdx.x == 0) {
            if (chunk == 0) *a.event_count = 0;
            s_base = a.ctrl->pos[0];
            if (chunk == a.n_chunks - 1) a.ctrl->pos[1] = s_base + excl + (unsigned long long)total;
            s_excl0 = excl;
            s_state = jump(a.jump, a.at[0], excl);
        }
        __syncthreads();
        chunk_state = s_state;
        if (count) st = jump(a.jump, s_state, excl - s_excl0);
    }
    uint64_t opened = 0;
#pragma unroll
    for (int i = 0; i < kSitesPerThread; ++i) {
        int64_t s = s0 + i;
        if (s >= n) continue;
        uint8_t open = 0;
#pragma unroll
        for (int mu = 0; mu < D; ++mu) {
            if (!((agree[i] >> mu) & 1u)) continue;
            bool drawn;
            if (STREAM) {
                uint64_t k = draw53(st);
                st = pcg_step(st, a.inc);
                drawn = k < a.kp53;
            } else {
                drawn = keyed24(a.seed32 ^ kBondKey, (uint32_t)(s * D + mu), a.sweep32) < a.kp24;
            }
            if (drawn) open |= (uint8_t)(1u << mu);
        }
        if (row8) opened |= (uint64_t)open << (8 * i);
        else a.bonds[s] = open;
    }
    if (row8 && s0 < n) *reinterpret_cast<uint64_t *>(a.bonds + s0) = opened;
    if (STREAM && chunk == a.n_chunks - 1 && threadIdx.x == 0) a.at[1] = jump(a.jump, chunk_state, chunk_draws);
}

// ------------------------------------------------------------ 2. labels
__device__ __forceinline__ int32_t find_root(int32_t *parent, int32_t x, int cap, Control *ctrl) {
    int32_t p = ld_relaxed32(&parent[x]);
    int it = 0;
    while (p != x) {
        int32_t gp = ld_relaxed32(&parent[p]);
        if (gp != p) parent[x] = gp;  // path halving: gp is an ancestor, never a wrong set
        x = p;
        p = gp;
        if (++it > cap) {
            atomicOr(&ctrl->status, kStatusPassCap);
            break;
        }
    }
    return x;
}

// Unite the sets of a and b: the larger root is hooked under the smaller by an
// atomic minimum on its parent.  Where that root was hooked in the meantime, its
// parent becomes the smaller of the two all the same, and the link that gave way
// (the old parent's) is united in turn, the reduction of Y. Komura, "GPU-based
// cluster-labeling algorithm without the use of conventional iteration" (Comput.
// Phys. Commun. 194, 2015): no attempt is repeated, so many lanes
// hooking to one root do not wait for each other as they do on a CAS
// (tile_hook_kernel on 2D Ising 4096^2 with 32-row blocks: 145 us with the CAS,
// 131 with this).
__device__ __forceinline__ void unite(int32_t *parent, int32_t a, int32_t b, int cap, Control *ctrl) {
    for (int it = 0;; ++it) {
        a = find_root(parent, a, cap, ctrl);
        b = find_root(parent, b, cap, ctrl);
        if (a == b) return;
        if (a < b) {
            int32_t t = a;
            a = b;
            b = t;
        }
        const int32_t old = atomicMin(&parent[a], b);
        if (old == a) return;  // a was still a root
        a = old;
        if (it > cap) {
            atomicOr(&ctrl->status, kStatusPassCap);
            return;
        }
    }
}

// ---- tile-local labelling.  A CTA labels a tile of TX x TY (x TZ, where the
// lattice has a third direction) sites; its eight warps own blocks of 32
// columns and walk their rows in order.  Within a row the runs of open +x bonds
// come out of one ballot.  A run takes its label from the first open bond into
// it from the row before (its y neighbour, else its z neighbour), so the walk
// itself builds a forest one level deep without an atomic: at the 2D critical
// point two runs in three find such a bond.  The bonds that remain -- a run's
// further bonds to earlier rows, less those that repeat the lane before's pair,
// and the bonds between blocks -- are united on the shared-memory parent array
// (larger root under smaller, so each root is its component's minimum site:
// local and global index orders agree).  What leaves the CTA is every site's
// tile-local root, 16 bits at its place in the tile, and the global parent of
// the roots themselves (the label init of cluster_prelude.wgsl:83-93): the
// global union-find lives on the local roots alone, about one site in eight in
// 2D at beta_c.  Bonds that leave the tile, the periodic ones among them, go
// through it in boundary_hook_kernel; a relabel pass takes a tile per CTA, walks
// once per local root and hands the labels to the sites in shared memory.
//
// Bound by issue: on the keyed stream about half of the instructions are the
// two bond draws of a site.  2D Ising 4096^2 at beta_c in equilibrium, tile
// kernel / relabel us a launch: 248 / 129 with a CAS union per +y bond (64 x 64
// tiles) and a walk per site from a 32-bit parent; 120 / 37 so (the sweep
// 0.41 -> 0.196 ms).  The block's 16 rows: 32 had fewer edges but its lists and
// parents left 4 CTAs per SM (0.215 ms), 8 more boundary unions (0.217 ms).
//
// kSmall: fewer rows per block, for lattices that give the large tiles' CTAs to
// less than two per SM (large_tiles): a block's rows are a serial chain.  kNarrow
// and kWide stack the blocks along y or x, for lattices short along the other one.
// kFlat: a run of consecutive sites, for lattices that fill no block (tile_shape).
enum TileShape { kLarge, kSmall, kNarrow, kWide, kFlat };

template <int D, int SHAPE>
struct Tile {  // block (per warp): 32 x BY x BZ; tile: WX x WY x WZ blocks
    static constexpr bool kTall = SHAPE == kLarge || SHAPE == kNarrow;
    static constexpr int BY = D == 1 ? 1 : D == 2 ? (kTall ? 16 : 8) : (kTall ? 4 : 2), BZ = D >= 3 ? BY : 1;
    static constexpr int WX = D == 1 || SHAPE == kWide ? 8 : D == 2 ? (SHAPE == kNarrow ? 1 : 4) : (SHAPE == kLarge ? 2 : 1),
                         WZ = D >= 3 && SHAPE != kWide ? 2 : 1, WY = 8 / (WX * WZ);
    static constexpr int TX = 32 * WX, TY = BY * WY, TZ = BZ * WZ;
    static constexpr int kSites = TX * TY * TZ;
    static constexpr int kDims = D;
    static constexpr int G = D == 2 ? 8 : BY;  // rows whose bonds are made together
    static_assert(WX * WY * WZ * 32 == kThreads, "a warp per block");
    static_assert(kSites <= 65536 && (BY * BZ) % G == 0 && BY * BZ <= 32, "16-bit local roots, 32 rows a block");

    int32_t L[3];
    uint32_t plane, slab_sites;  // sites of an xy plane, of a slab (the tile's directions)
    uint32_t t0, t1, t2;         // tiles along them
    __host__ __device__ explicit Tile(const Geom &g) {
        L[0] = g.L[0];
        L[1] = D >= 2 ? g.L[1] : 1;
        L[2] = D >= 3 ? g.L[2] : 1;
        plane = (uint32_t)L[0] * (uint32_t)L[1];
        slab_sites = plane * (uint32_t)L[2];
        t0 = (uint32_t)(L[0] + TX - 1) / TX;
        t1 = (uint32_t)(L[1] + TY - 1) / TY;
        t2 = (uint32_t)(L[2] + TZ - 1) / TZ;
    }
    __host__ __device__ int64_t tiles(int64_t n_sites) const { return n_sites / slab_sites * t0 * t1 * t2; }
    // First site of tile b, and its coordinates.
    __device__ uint32_t origin(uint32_t b, int *x) const {
        const uint32_t b1 = b / t0, b2 = b1 / t1, slab = D >= 3 ? b2 / t2 : b2;
        x[0] = (int)(b - b1 * t0) * TX;
        x[1] = (int)(b1 - b2 * t1) * TY;
        x[2] = D >= 3 ? (int)(b2 - slab * t2) * TZ : 0;
        return slab * slab_sites + (uint32_t)x[2] * plane + (uint32_t)x[1] * (uint32_t)L[0] + (uint32_t)x[0];
    }
    // The site at place li of the tile whose first site is s0.
    __device__ uint32_t site(uint32_t s0, uint32_t li) const {
        uint32_t s = s0 + li % TX;
        if (D >= 2) s += li / TX % TY * (uint32_t)L[0];
        if (D >= 3) s += li / (TX * TY) * plane;
        return s;
    }
    // Whether place li of the tile at x is in the lattice (tiles overhang).
    __device__ bool inside(const int *x, uint32_t li) const {
        return x[0] + (int)(li % TX) < L[0] && (D < 2 || x[1] + (int)(li / TX % TY) < L[1]) &&
               (D < 3 || x[2] + (int)(li / (TX * TY)) < L[2]);
    }
    // The tile-local root of the site at coordinates x (x[2] and up: its slab), as a site.
    __device__ uint32_t local_root(const uint16_t *roots, uint32_t s, const int32_t *x) const {
        const uint32_t xx = (uint32_t)x[0], y = D >= 2 ? (uint32_t)x[1] : 0u, z = D >= 3 ? (uint32_t)x[2] : 0u;
        const uint32_t slab = D > 3 ? s / slab_sites : 0u;
        const uint32_t tile = ((slab * t2 + z / TZ) * t1 + y / TY) * t0 + xx / TX;
        const uint32_t li = ((z % TZ) * TY + y % TY) * TX + xx % TX;
        const uint32_t r = roots[(size_t)tile * kSites + li];
        return s - (xx % TX) - (y % TY) * (uint32_t)L[0] - (z % TZ) * plane + site(0, r);
    }
};

// Consecutive sites, whatever directions they run along: the places are the sites in
// order, every bond between two of them is a bond of the tile, periodic ones too.
template <int D>
struct Tile<D, kFlat> {
    static constexpr int TX = 2048, kSites = 2048;

    int32_t L[1];
    uint32_t n;
    __host__ __device__ explicit Tile(const Geom &g) : n((uint32_t)g.n_sites) { L[0] = (int32_t)n; }
    __host__ __device__ int64_t tiles(int64_t n_sites) const { return (n_sites + kSites - 1) / kSites; }
    __device__ uint32_t origin(uint32_t b, int *x) const {
        x[0] = (int)(b * kSites);
        return b * kSites;
    }
    __device__ uint32_t site(uint32_t s0, uint32_t li) const { return s0 + li; }
    __device__ bool inside(const int *x, uint32_t li) const { return (uint32_t)x[0] + li < n; }
    __device__ uint32_t local_root(const uint16_t *roots, uint32_t s, const int32_t *) const {
        return s / kSites * kSites + roots[s];
    }
};

// Whether the large tiles give every SM two CTAs.
template <int D>
bool large_tiles(const Geom &g, int sm_count) {
    return D >= 2 && Tile<D, kLarge>(g).tiles(g.n_sites) >= 2 * (int64_t)sm_count;
}

// The tiles of a lattice (us a keyed sweep on each):
//  * flat where the lattice is one of them, so that all bonds lie inside and the boundary launch
//    falls away (8^2 7 against 13 with kSmall, 32^2 13 / 15; 40^2 17 / 16), and where rows of a few
//    sites would leave most lanes of a block idle (2 x 2^20 61 / 247 kNarrow, 4 x 65536 27 / 37, 8 x
//    65536 32 / 38, 12 x 65536 39 / 40; 2 x 2 x 65536 30 / 156 kSmall, 4 x 256 x 256 35 / 46; 8 x 256 x 256
//    46 / 49 keyed, 76 / 72 on the PCG stream);
//  * kNarrow for rows up to 96, which overhang the other 2D tiles' 128 columns (32 x 2^19 161 against 515
//    with kLarge, 96 x 65536 73 / 88), from the sizes on that fill the chip (28 x 8192 25 both; 34 x
//    4096 26 against 23 with kSmall);
//  * kWide and kSmall for lattices of few rows, which leave a block's other rows idle (2^21 x 8 204 / 290 /
//    285 with kWide / kSmall / kLarge, 2^20 x 16 212 / 193 / 220; 65536 x 2 x 2 26 / 36 / 35, 512 x 512 x 2
//    32 / 30 / 36);
//  * kSmall for 3D rows up to 32, half of kLarge's (30 x 200 x 200 49 / 64).
template <int D>
TileShape fastest_tiles(const Geom &g, int sm_count, bool keyed) {
    const int64_t n = g.n_sites;
    if (D == 1) return kSmall;
    if (n <= 1024) return kFlat;
    if (D == 2) {
        if (g.L[0] <= 8 && n >= 32768) return kFlat;
        if (g.L[0] <= 96 && Tile<D, kSmall>(g).tiles(n) >= 4 * (int64_t)sm_count) return kNarrow;
        if (g.L[1] <= 8 && n >= (int64_t(1) << 20)) return kWide;
        if (g.L[1] <= 16) return kSmall;
    } else {
        if (g.L[0] <= 4 || (g.L[0] <= 8 && keyed && n >= (int64_t(1) << 18))) return kFlat;
        if (g.L[1] <= 2 && g.L[2] <= 4) return kWide;
        if (g.L[0] <= 32 || g.L[2] <= 4) return kSmall;
    }
    return large_tiles<D>(g, sm_count) ? kLarge : kSmall;
}

// ... but flat ones for a lattice of 2^20 sites and more that would have over eight places (2 B each)
// a site: tubes such as 5 x 1 x 1 x N.
template <int D>
TileShape tile_shape(const Geom &g, int sm_count, bool keyed) {
    const TileShape shape = fastest_tiles<D>(g, sm_count, keyed);
    const int64_t n = g.n_sites;
    auto overhangs = [&](auto t) { return t.tiles(n) * t.kSites > 8 * n; };
    const bool far = shape == kLarge    ? overhangs(Tile<D, kLarge>(g))
                     : shape == kNarrow ? overhangs(Tile<D, kNarrow>(g))
                     : shape == kWide   ? overhangs(Tile<D, kWide>(g))
                                        : overhangs(Tile<D, kSmall>(g));
    return D >= 2 && n >= (int64_t(1) << 20) && shape != kFlat && far ? kFlat : shape;
}

// The keyed bond draw of one sweep as an open-draw comparison (plq_packed.cuh):
// k < kp24 with k the 24-bit draw <=> (v ^ X) <= T, v the draw before its
// closing xorshift.
// (kp24 = 0, no bond opens, has no T: some() says so, once for a group of draws.)
struct BondCut {
    uint32_t seed, mix, T, X;
    __device__ __forceinline__ BondCut(const ClusterArgs &a, uint32_t sweep)
        : seed(a.seed32 ^ kBondKey), mix(keyed_mix(sweep)), T((a.kp24 << 8) - 1u),
          X(((a.kp24 << 8) - 1u) >> 16) {}
    __device__ __forceinline__ bool open(uint32_t bond) const {
        return (lowbias32_open(lowbias32_head(seed ^ bond) ^ mix) ^ X) <= T;
    }
    static __device__ __forceinline__ bool some(const ClusterArgs &a) { return a.kp24 != 0; }
};

__device__ __forceinline__ int lfind(int32_t *p, int32_t x, int cap, Control *ctrl) {
    int32_t px = p[x];
    int it = 0;
    while (px != x) {
        // no path halving: the trees inside a tile are shallow (about 2.3 deep at beta_c),
        // and the halving stores cost more than the hops they save
        const int32_t gp = p[px];
        x = px;
        px = gp;
        if (++it > cap) {
            atomicOr(&ctrl->status, kStatusPassCap);
            break;
        }
    }
    return x;
}

__device__ __forceinline__ void lunite(int32_t *p, int32_t a, int32_t b, int cap, Control *ctrl) {
    for (int it = 0;; ++it) {
        a = lfind(p, a, cap, ctrl);
        b = lfind(p, b, cap, ctrl);
        if (a == b) return;
        if (a < b) {
            const int32_t t = a;
            a = b;
            b = t;
        }
        const int32_t old = atomicMin(&p[a], b);  // as unite
        if (old == a) return;
        a = old;
        if (it > cap) {
            atomicOr(&ctrl->status, kStatusPassCap);
            return;
        }
    }
}

// Unite the ends of an edge between blocks, one per lane (open: this lane has
// one); a lane whose ends read as the lane before's pair leaves it to that lane.
__device__ __forceinline__ void edge_unite(int32_t *p, bool open, int32_t u, int32_t v, int cap, Control *ctrl) {
    const int32_t pu = open ? p[u] : -1, pv = open ? p[v] : -1;
    const int32_t qu = __shfl_up_sync(0xffffffffu, pu, 1), qv = __shfl_up_sync(0xffffffffu, pv, 1);
    const bool repeat = (threadIdx.x & 31u) > 0 && qu == pu && qv == pv;
    if (open && !repeat && pu != pv) lunite(p, pu, pv, cap, ctrl);
}

template <class T>
struct LabelShared {
    static constexpr int kBlock = 32 * T::BY * T::BZ;
    static constexpr int kFurther = T::kDims >= 3 ? 2 * kBlock : T::kDims == 2 ? kBlock : 1;
    int32_t p[T::kSites];
    uint16_t further[kThreads / 32][kFurther];
};
template <int D>
struct LabelShared<Tile<D, kFlat>> {
    int32_t p[Tile<D, kFlat>::kSites];
};

// label_tile for consecutive sites, a thread's a CTA's width apart.  A site first takes as its
// parent the lowest site of the tile that an open bond leads to it from (an atomic
// minimum, no find), which makes a forest of long chains along the lattice's long
// direction; pointer jumping flattens it (united bond by bond instead, every find
// would walk those chains); the bonds that made no parent are then united.
template <int D, bool KEYED>
__device__ __forceinline__ void label_flat(const ClusterArgs &a, uint32_t sweep, uint32_t tile, int32_t *p) {
    using T = Tile<D, kFlat>;
    constexpr int S = T::kSites / kThreads;
    static_assert(S * D <= 64, "a bit per bond of a thread's sites");
    const uint32_t s0 = tile * T::kSites, here = min((uint32_t)T::kSites, (uint32_t)a.g.n_sites - s0);
    const int cap = a.cap < T::kSites + 64 ? a.cap : T::kSites + 64;
    const BondCut cut(a, sweep);
    const bool bonds = !KEYED || BondCut::some(a);
    for (uint32_t li = threadIdx.x; li < here; li += kThreads) p[li] = (int32_t)li;
    __syncthreads();
    auto neighbours = [&](uint32_t li, uint32_t (&lb)[D]) {
        int32_t x[D];
        site_coords<D>(a.g, s0 + li, x);
#pragma unroll
        for (int mu = 0; mu < D; ++mu) lb[mu] = (uint32_t)nbr_plus(a.g, s0 + li, x, mu) - s0;
    };
    uint64_t open = 0;  // bit i * D + mu: the +mu bond of site i, within the tile
#pragma unroll 2
    for (int i = 0; i < S; ++i) {
        const uint32_t li = threadIdx.x + (uint32_t)(i * kThreads);
        if (li >= here || !bonds) break;
        uint32_t lb[D];
        neighbours(li, lb);
        const uint32_t own = KEYED ? a.state[s0 + li] : a.bonds[s0 + li];
#pragma unroll
        for (int mu = 0; mu < D; ++mu) {
            if (lb[mu] >= here) continue;
            const bool o = KEYED ? (a.state[s0 + lb[mu]] == own) & cut.open((s0 + li) * (uint32_t)D + (uint32_t)mu)
                                 : (own >> mu) & 1u;
            if (!o) continue;
            open |= 1ull << (i * D + mu);
            if (lb[mu] > li) atomicMin(&p[lb[mu]], (int32_t)li);
        }
    }
    __syncthreads();
    // the bonds that made no parent
#pragma unroll 1
    for (int i = 0; i < S; ++i) {
        const uint32_t li = threadIdx.x + (uint32_t)(i * kThreads), mine = (uint32_t)(open >> (i * D)) & ((1u << D) - 1u);
        if (!mine) continue;
        uint32_t lb[D];
        neighbours(li, lb);
#pragma unroll
        for (int mu = 0; mu < D; ++mu)
            if (((mine >> mu) & 1u) && lb[mu] > li && p[lb[mu]] == (int32_t)li) open &= ~(1ull << (i * D + mu));
    }
    __syncthreads();
    bool moved = true;
    for (int round = 0; moved && round < 16; ++round) {  // (a chain's length halves, at least, with each)
        moved = false;
        for (uint32_t li = threadIdx.x; li < here; li += kThreads) {
            const int32_t up = p[li], r = p[up];
            if (r != up) {
                p[li] = r;
                moved = true;
            }
        }
        moved = __syncthreads_or(moved);
    }
    while (open) {
        const int k = __ffsll((long long)open) - 1, i = k / D, mu = k - i * D;
        open &= open - 1ull;
        const uint32_t li = threadIdx.x + (uint32_t)(i * kThreads);
        uint32_t lb[D], to = 0;
        neighbours(li, lb);
#pragma unroll
        for (int m = 0; m < D; ++m)
            if (m == mu) to = lb[m];
        lunite(p, (int32_t)li, (int32_t)to, cap, a.ctrl);
    }
    __syncthreads();
    for (uint32_t li = threadIdx.x; li < here; li += kThreads) {
        const int32_t r = lfind(p, (int32_t)li, cap, a.ctrl);
        const uint32_t s = s0 + li;
        a.local_root[s] = (uint16_t)r;
        if (r == (int32_t)li) a.parent[s] = (int32_t)s;
        if (!KEYED) a.fresh[s] = r == (int32_t)li ? 1 : 0;  // root_rank_kernel's candidates
    }
}

// Labels tile `tile`; the CTA may reuse `sm` at once.
template <int D, int SHAPE, bool KEYED>
__device__ __forceinline__ void label_tile(const ClusterArgs &a, uint32_t sweep, uint32_t tile,
                                           LabelShared<Tile<D, SHAPE>> &sm) {
    using T = Tile<D, SHAPE>;
    constexpr int BY = T::BY, BZ = T::BZ, TX = T::TX, TY = T::TY, TZ = T::TZ, G = T::G;
    int32_t *p = sm.p;
    const T t(a.g);
    const int L0 = t.L[0], L1 = t.L[1], L2 = t.L[2];
    int xt[3];
    const uint32_t s_tile = t.origin(tile, xt);
    const int cap = a.cap < T::kSites + 64 ? a.cap : T::kSites + 64;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int wx = wid % T::WX, wy = (wid / T::WX) % T::WY, wz = wid / (T::WX * T::WY);
    const int lx = 32 * wx + lane, x = xt[0] + lx;
    const int ly0 = wy * BY, y0 = xt[1] + ly0, lz0 = wz * BZ, z0 = xt[2] + lz0;
    const bool in_x = x < L0;
    const uint32_t plane = t.plane;
    const uint32_t s00 = s_tile + (uint32_t)lz0 * plane + (uint32_t)(ly0 * L0 + lx);
    const int li00 = (lz0 * TY + ly0) * TX + lx;
    const uint32_t le = 0xffffffffu >> (31 - lane);
    const BondCut cut(a, sweep);
    const bool x_in_tile = x + 1 < L0 && lx + 1 < TX;  // the +x neighbour is in the tile

    // ---- the block's rows in order: labels from the row before and the plane before
    // further bonds to the row before (the site's place) or the plane before (| kToPlane), listed per
    // block: about one site in ten has one, and a list keeps whole warps busy uniting them
    constexpr uint32_t kToPlane = 0x8000u;
    static_assert(D < 3 || T::kSites <= 0x8000, "a bit beside the place");
    uint16_t *further = sm.further[wid];
    int n_further = 0;
    uint32_t mine = 0;  // rows whose label is this lane's own site
    auto list = [&](bool mine, uint32_t entry) {
        const unsigned m = __ballot_sync(0xffffffffu, mine);
        if (mine) further[n_further + __popc(m & (le >> 1))] = (uint16_t)entry;
        n_further += __popc(m);
    };
    uint32_t edge_x = 0;              // lane 31: rows with an open bond to the next block
    uint32_t edge_y = 0, edge_z = 0;  // planes / rows with an open bond to the next block
    int32_t lab_plane[D >= 3 ? BY : 1] = {};
    uint32_t open_plane = 0;  // bit y: the plane before's +z bond
    int32_t lab_up = 0;
    bool open_up = false;
#pragma unroll 1
    for (int g = 0; g < BY * BZ / G; ++g) {
        const int jz = D >= 3 ? g : 0, yg = D >= 3 ? 0 : g * G;
        if ((D >= 3 && z0 + jz >= L2) || y0 + yg >= L1) break;
        const uint32_t sg = s00 + (uint32_t)jz * plane + (uint32_t)(yg * L0);
        const bool z_in_tile = D >= 3 && z0 + jz + 1 < L2 && lz0 + jz + 1 < TZ;
        // the bonds of G rows, their loads in flight together
        uint32_t bx = 0, by = 0, bz = 0;
        if (KEYED) {
            uint32_t c[G + 1], cr[G], cz[G];
#pragma unroll
            for (int k = 0; k <= G; ++k) c[k] = in_x && y0 + yg + k < L1 ? a.state[sg + (uint32_t)(k * L0)] : 0u;
#pragma unroll
            for (int k = 0; k < G; ++k) {
                cr[k] = lane == 31 && x_in_tile && y0 + yg + k < L1 ? a.state[sg + (uint32_t)(k * L0) + 1u] : 0u;
                cz[k] = D >= 3 && z_in_tile && in_x && y0 + yg + k < L1 ? a.state[sg + (uint32_t)(k * L0) + plane] : 0u;
            }
            // every lane draws every bond (a branch around a draw that one lane in seven skips
            // costs more than it saves); what is not a bond of the tile is masked at the end
            uint32_t ax = 0, ay = 0, az = 0;
#pragma unroll
            for (int k = 0; k < G; ++k) {
                const uint32_t bond = (sg + (uint32_t)(k * L0)) * (uint32_t)D;
                const uint32_t down = __shfl_down_sync(0xffffffffu, c[k], 1);
                const uint32_t right = lane == 31 ? cr[k] : down;
                if ((c[k] == right) & cut.open(bond)) bx |= 1u << k;
                if (D >= 2 && ((c[k] == c[k + 1]) & cut.open(bond + 1u))) by |= 1u << k;
                if (D >= 3 && ((c[k] == cz[k]) & cut.open(bond + 2u))) bz |= 1u << k;
            }
            if (BondCut::some(a)) {
                const int rows = min(G, L1 - (y0 + yg));  // rows of the group in the lattice
                const uint32_t in_rows = (1u << rows) - 1u;
                if (x_in_tile) ax = in_rows;
                if (in_x && z_in_tile) az = in_rows;
                // a row's +y neighbour: the row after it in the lattice and the tile
                const int rows_y = min(min(G, L1 - 1 - (y0 + yg)), TY - 1 - (ly0 + yg));
                if (in_x && D >= 2) ay = (1u << rows_y) - 1u;
            }
            bx &= ax;
            by &= ay;
            bz &= az;
        } else {
            uint32_t own[G];
#pragma unroll
            for (int k = 0; k < G; ++k) own[k] = in_x && y0 + yg + k < L1 ? a.bonds[sg + (uint32_t)(k * L0)] : 0u;
#pragma unroll
            for (int k = 0; k < G; ++k) {
                if (x_in_tile) bx |= (own[k] & 1u) << k;
                if (y0 + yg + k + 1 < L1 && ly0 + yg + k + 1 < TY) by |= ((own[k] >> 1) & 1u) << k;
                if (z_in_tile) bz |= ((own[k] >> 2) & 1u) << k;
            }
        }
        if (D >= 3) {
            open_up = false;
            if (jz == BZ - 1) edge_z = bz;
        }
        if (lane == 31) edge_x |= bx << (g * G);
        // the labels of the G rows, one after the other
#pragma unroll
        for (int k = 0; k < G; ++k) {
            if (y0 + yg + k >= L1) break;
            // the run of this lane: lanes [st, next start)
            const uint32_t starts = ~(__ballot_sync(0xffffffffu, (bx >> k) & 1u) << 1);
            const int st = 31 - __clz(starts & le);
            const uint32_t later = starts & ~le;
            const uint32_t run = ((later & (0u - later)) - 1u) & (0xffffffffu << st);
            const int li = li00 + (jz * TY + yg + k) * TX;
            int32_t label = li - lane + st;
            const uint32_t up = __ballot_sync(0xffffffffu, open_up) & run;
            const int32_t from_up = __shfl_sync(0xffffffffu, lab_up, (__ffs(up) - 1) & 31);
            if (up) label = from_up;
            if (D >= 3) {
                const bool oz = (open_plane >> k) & 1u;
                const int32_t lab_z = lab_plane[k];
                const uint32_t uz = __ballot_sync(0xffffffffu, oz) & run;
                const int32_t from_z = __shfl_sync(0xffffffffu, lab_z, (__ffs(uz) - 1) & 31);
                if (!up && uz) label = from_z;
                const int32_t before = __shfl_up_sync(0xffffffffu, lab_z, 1);
                const bool repeat = before == lab_z && ((uz << 1) >> lane) & 1u;
                list(oz && !repeat && lab_z != label, (uint32_t)li | kToPlane);
                lab_plane[k] = label;
            }
            {
                const int32_t before = __shfl_up_sync(0xffffffffu, lab_up, 1);
                const bool repeat = before == lab_up && ((up << 1) >> lane) & 1u;
                if (D >= 2) list(open_up && !repeat && lab_up != label, (uint32_t)li);
            }
            p[li] = label;
            if (label == li) mine |= 1u << (g * G + k);
            lab_up = label;
            open_up = (by >> k) & 1u;
        }
        if (yg + G == BY && y0 + BY < L1 && (by >> (G - 1)) & 1u) edge_y |= 1u << jz;
        open_plane = bz;
    }
    __syncthreads();

    // ---- the remaining bonds of the tile
    for (int i = lane; i < n_further; i += 32) {
        const uint32_t e = further[i];
        const int li = D >= 3 ? (int)(e & ~kToPlane) : (int)e;
        lunite(p, li, li - (D >= 3 && (e & kToPlane) ? TX * TY : TX), cap, a.ctrl);
    }
    __syncwarp();
    if (T::WX > 1) {  // bonds between blocks: lane l takes row l of the block's last column, its own column's last rows
        const uint32_t rows = __shfl_sync(0xffffffffu, edge_x, 31);
        const int li = li00 - lane + 31 + (lane / BY * TY + lane % BY) * TX;
        const bool open = lane < BY * BZ && ((rows >> lane) & 1u);
        edge_unite(p, open, li, li + 1, cap, a.ctrl);
    }
    if (D >= 2) {
#pragma unroll
        for (int jz = 0; jz < BZ; ++jz) {
            const int li = li00 + (jz * TY + BY - 1) * TX;
            edge_unite(p, (edge_y >> jz) & 1u, li, li + TX, cap, a.ctrl);
        }
    }
    if (D >= 3) {
#pragma unroll
        for (int jy = 0; jy < BY; ++jy) {
            const int li = li00 + ((BZ - 1) * TY + jy) * TX;
            edge_unite(p, (edge_z >> jy) & 1u, li, li + TX * TY, cap, a.ctrl);
        }
    }
    __syncthreads();

    // ---- the forest is final.  The labels the rows were given (the sites whose label was their
    // own: mine) are pointed at their roots, which leaves every site two steps from its root.
    for (uint32_t m = mine; m; m &= m - 1u) {
        const int j = __ffs(m) - 1;
        const int li = li00 + (j / BY * TY + j % BY) * TX;
        const int32_t r = lfind(p, li, cap, a.ctrl);
        if (r != li) p[li] = r;
    }
    __syncthreads();
    uint16_t *roots = a.local_root + (size_t)tile * T::kSites;
#pragma unroll 1
    for (int jz = 0; jz < BZ; ++jz) {
        if (D >= 3 && z0 + jz >= L2) break;
#pragma unroll 8
        for (int jy = 0; jy < BY; ++jy) {
            if (y0 + jy >= L1) break;
            const int li = li00 + (jz * TY + jy) * TX;
            const int32_t r = p[p[li]];
            const uint32_t s = s00 + (uint32_t)jz * plane + (uint32_t)(jy * L0);
            if (in_x) {
                roots[li] = (uint16_t)r;
                if (r == li) a.parent[s] = (int32_t)s;
                if (!KEYED) a.fresh[s] = r == li ? 1 : 0;  // root_rank_kernel's candidates, in site order
            }
        }
    }
}

template <int D, int SHAPE, bool KEYED>
__global__ void __launch_bounds__(kThreads, D == 2 && (SHAPE == kLarge || SHAPE == kNarrow) ? 5 : 1) tile_hook_kernel(ClusterArgs a) {
    __shared__ LabelShared<Tile<D, SHAPE>> sm;
    after_previous();
    if constexpr (SHAPE == kFlat) label_flat<D, KEYED>(a, a.sweep32, blockIdx.x, sm.p);
    else label_tile<D, SHAPE, KEYED>(a, a.sweep32, blockIdx.x, sm);
}

// unite_edges for tiles of consecutive sites: the bonds whose ends lie in two of them.
template <int D, bool KEYED>
__device__ __forceinline__ void unite_flat_edges(const ClusterArgs &a, uint32_t sweep) {
    using T = Tile<D, kFlat>;
    const T t(a.g);
    const BondCut cut(a, sweep);
    if (KEYED && !BondCut::some(a)) return;
    const int64_t n = a.g.n_sites, stride = (int64_t)gridDim.x * blockDim.x;
    const int lane = threadIdx.x & 31;
    for (int64_t c0 = (int64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31u); c0 < n; c0 += stride) {
        const int64_t s = c0 + lane;
        int32_t x[D];
        site_coords<D>(a.g, s < n ? s : 0, x);
#pragma unroll
        for (int mu = 0; mu < D; ++mu) {
            const int64_t nb = nbr_plus(a.g, s, x, mu);
            int32_t pa = -1, pb = -1;
            if (s < n && nb / T::kSites != s / T::kSites) {
                const bool open = KEYED ? (a.state[s] == a.state[nb]) & cut.open((uint32_t)s * (uint32_t)D + (uint32_t)mu)
                                        : (a.bonds[s] >> mu) & 1u;
                if (open) {
                    pa = (int32_t)t.local_root(a.local_root, (uint32_t)s, x);
                    pb = (int32_t)t.local_root(a.local_root, (uint32_t)nb, x);
                }
            }
            const int32_t qa = __shfl_up_sync(0xffffffffu, pa, 1), qb = __shfl_up_sync(0xffffffffu, pb, 1);
            const bool repeat = lane > 0 && qa == pa && qb == pb;
            if (pa >= 0 && !repeat) unite(a.parent, pa, pb, a.cap, a.ctrl);
        }
    }
}

// Global unions for the open bonds that leave their tile: of the tiles' last
// columns, last rows and last planes (three families of candidate sites in one
// index space), and every bond along the directions past the tile's.  A lane
// whose ends' local roots are the lane before's leaves the union to that lane:
// along a tile edge a large cluster meets another at many sites.
template <int D, int SHAPE, bool KEYED>
__device__ __forceinline__ void unite_edges(const ClusterArgs &a, uint32_t sweep) {
    using T = Tile<D, SHAPE>;
    const T t(a.g);
    const BondCut cut(a, sweep);
    const int64_t n = a.g.n_sites;
    const uint32_t L0 = (uint32_t)t.L[0], L1 = (uint32_t)t.L[1], L2 = (uint32_t)t.L[2];
    const uint32_t rows = (uint32_t)(n / L0), planes = rows / L1;  // planes: over every direction past 1
    const int64_t nx = (int64_t)t.t0 * rows;
    const int64_t ny = D >= 2 ? (int64_t)t.t1 * L0 * planes : 0;
    const int64_t nz = D >= 3 ? (int64_t)t.t2 * t.plane * (planes / L2) : 0;
    const int64_t candidates = nx + ny + nz, all = candidates + (D > 3 ? (int64_t)(D - 3) * n : 0);
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    const int lane = threadIdx.x & 31;
    // whole warps per trip: the comparison with the lane before is warp-wide
    for (int64_t c0 = (int64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31u); c0 < all; c0 += stride) {
        const int64_t c = c0 + lane;
        int64_t s = 0;
        int mu = 0;
        if (c < nx) {
            const uint32_t row = (uint32_t)c / t.t0, k = (uint32_t)c - row * t.t0;
            s = (int64_t)row * L0 + min((k + 1u) * (uint32_t)T::TX, L0) - 1u;
        } else if (c < nx + ny) {
            const uint32_t cy = (uint32_t)(c - nx), r = cy / L0, xx = cy - r * L0, pl = r / t.t1, k = r - pl * t.t1;
            s = ((int64_t)pl * L1 + min((k + 1u) * (uint32_t)T::TY, L1) - 1u) * L0 + xx;
            mu = 1;
        } else if (c < candidates) {
            const uint32_t cz = (uint32_t)(c - nx - ny), r = cz / t.plane, xy = cz - r * t.plane, b = r / t.t2,
                           k = r - b * t.t2;
            s = ((int64_t)b * L2 + min((k + 1u) * (uint32_t)T::TZ, L2) - 1u) * t.plane + xy;
            mu = 2;
        } else if (c < all) {
            const int64_t e = c - candidates;
            mu = 3 + (int)(e / n);
            s = e - (int64_t)(mu - 3) * n;
        }
        bool open = c < all;
        if (!KEYED && open) open = (a.bonds[s] >> mu) & 1u;
        int32_t pa = -1, pb = -1;
        if (open) {
            int32_t x[D];
            site_coords<D>(a.g, s, x);
            int64_t nb = 0;  // compile-time directions keep the coordinates in registers
#pragma unroll
            for (int m = 0; m < D; ++m)
                if (m == mu) nb = nbr_plus(a.g, s, x, m);
            // keyed: open iff the two sites agree and the bond's draw is below p
            // (cluster_prelude.wgsl:61-80)
            if (KEYED)
                open = a.state[s] == a.state[nb] && BondCut::some(a) && cut.open((uint32_t)(s * D + mu));
            if (open) {
                pa = (int32_t)t.local_root(a.local_root, (uint32_t)s, x);
#pragma unroll
                for (int m = 0; m < D; ++m)
                    if (m == mu) x[m] = x[m] + 1 < a.g.L[m] ? x[m] + 1 : 0;
                pb = (int32_t)t.local_root(a.local_root, (uint32_t)nb, x);
            }
        }
        const int32_t qa = __shfl_up_sync(0xffffffffu, pa, 1), qb = __shfl_up_sync(0xffffffffu, pb, 1);
        const bool repeat = lane > 0 && qa == pa && qb == pb;
        if (open && !repeat && pa != pb) unite(a.parent, pa, pb, a.cap, a.ctrl);
    }
}

template <int D, int SHAPE, bool KEYED>
__global__ void __launch_bounds__(kThreads) boundary_hook_kernel(ClusterArgs a) {
    after_previous();
    if constexpr (SHAPE == kFlat) unite_flat_edges<D, KEYED>(a, a.sweep32);
    else unite_edges<D, SHAPE, KEYED>(a, a.sweep32);
}

// Read-only find for the passes after the unions: a compressing find could
// overwrite a root another thread has just stored with a non-root ancestor.
__device__ __forceinline__ int32_t find_root_ro(const int32_t *parent, int32_t x, int cap, Control *ctrl) {
    int32_t p = ld_relaxed32(&parent[x]);
    int it = 0;
    while (p != x) {
        x = p;
        p = ld_relaxed32(&parent[x]);
        if (++it > cap) {
            atomicOr(&ctrl->status, kStatusPassCap);
            break;
        }
    }
    return x;
}

// A relabel pass over one tile.  The tile's local roots are gathered into a list
// in shared memory; each walks to its cluster's root once (and stores it, so
// walks through it end there), and of_root(root, the local root) gives the value of its sites;
// then out takes the sites of each row four at a time.  Bound by the latency of the
// walks, hence the list: full warps of walks instead of one lane in eight.
template <class T>
struct RelabelShared {
    alignas(16) uint16_t root[T::kSites];
    uint16_t list[T::kSites];
    uint8_t value[T::kSites];
    int n;
};

template <class T, class F, class O>
__device__ __forceinline__ void tile_relabel(const ClusterArgs &a, uint32_t tile, RelabelShared<T> &sm, F of_root, O out) {
    uint16_t *s_root = sm.root, *s_list = sm.list;
    uint8_t *s_value = sm.value;
    int &s_n = sm.n;
    const T t(a.g);
    int xt[3];
    const uint32_t s_tile = t.origin(tile, xt);
    if (threadIdx.x == 0) s_n = 0;
    __syncthreads();
    const uint4 *src = reinterpret_cast<const uint4 *>(a.local_root + (size_t)tile * T::kSites);
#pragma unroll(T::kSites / 8 / kThreads > 4 ? 4 : 1)
    for (uint32_t i = threadIdx.x; i < T::kSites / 8; i += kThreads) {
        const uint4 v = src[i];
        reinterpret_cast<uint4 *>(s_root)[i] = v;
        const uint32_t own = 8u * i | (8u * i + 1u) << 16;  // places 8i, 8i + 1; the next pairs step by 2
        const uint32_t d[4] = {v.x ^ own, v.y ^ (own + 0x00020002u), v.z ^ (own + 0x00040004u),
                               v.w ^ (own + 0x00060006u)};
        uint32_t mine = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if ((d[k] & 0xFFFFu) == 0) mine |= 1u << (2 * k);
            if ((d[k] >> 16) == 0) mine |= 2u << (2 * k);
        }
        if (mine) {
            int at = atomicAdd(&s_n, __popc(mine));
            for (; mine; mine &= mine - 1u) s_list[at++] = (uint16_t)(8u * i + (uint32_t)__ffs(mine) - 1u);
        }
    }
    __syncthreads();
    const int n = s_n;
    for (int i0 = threadIdx.x; i0 < n; i0 += 4 * kThreads) {
        uint32_t li[4];
        int32_t s[4], up[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {  // the first steps of four walks in flight together
            const int i = i0 + k * kThreads;
            li[k] = i < n ? s_list[i] : 0u;
            s[k] = i < n && t.inside(xt, li[k]) ? (int32_t)t.site(s_tile, li[k]) : -1;  // (an overhanging place holds anything)
            up[k] = s[k] >= 0 ? ld_relaxed32(&a.parent[s[k]]) : -1;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (s[k] < 0) continue;
            int32_t root = s[k];
            if (up[k] != s[k]) {
                root = find_root_ro(a.parent, up[k], a.cap, a.ctrl);
                if (root != up[k]) a.parent[s[k]] = root;
            }
            s_value[li[k]] = of_root(root, s[k]);
        }
    }
    __syncthreads();
    // four sites of a row per thread
    for (uint32_t li = 4u * threadIdx.x; li < T::kSites; li += 4u * kThreads) {
        if (!t.inside(xt, li)) continue;
        const uint2 r2 = *reinterpret_cast<const uint2 *>(s_root + li);
        constexpr uint32_t kIn = T::kSites - 1;  // (places past the row's end hold anything)
        static_assert((T::kSites & (T::kSites - 1)) == 0, "a power of two");
        const uint32_t r[4] = {r2.x & kIn, (r2.x >> 16) & kIn, r2.y & kIn, (r2.y >> 16) & kIn};
        const int last = t.L[0] - xt[0] - (int)(li % T::TX);  // sites left in the row
        out(t.site(s_tile, li), last < 4 ? last : 4, r, s_value, t, s_tile);
    }
}

// The values of up to four sites of a row into a byte array.
__device__ __forceinline__ void store_row(uint8_t *state, uint32_t s, int count, const uint8_t *v) {
    if (count == 4 && (s & 3u) == 0) {
        *reinterpret_cast<uchar4 *>(state + s) = make_uchar4(v[0], v[1], v[2], v[3]);
    } else {
        for (int k = 0; k < count; ++k) state[s + (uint32_t)k] = v[k];
    }
}

// Every site's parent becomes its root (for the readers of labels and sizes).
template <int D, int SHAPE>
__global__ void __launch_bounds__(kThreads) flatten_kernel(ClusterArgs a) {
    // (the pass has stored each local root's root at the local root)
    using T = Tile<D, SHAPE>;
    __shared__ RelabelShared<T> sm;
    tile_relabel<T>(
        a, blockIdx.x, sm, [](int32_t, int32_t) { return (uint8_t)0; },
        [&](uint32_t s, int count, const uint32_t (&r)[4], const uint8_t *, const T &t, uint32_t s_tile) {
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (k < count) a.parent[s + (uint32_t)k] = a.parent[t.site(s_tile, r[k])];
        });
}

// keyed (cluster_relabel.wgsl:72-89), every cluster
template <int D, int SHAPE>
__global__ void __launch_bounds__(kThreads) relabel_keyed_kernel(ClusterArgs a) {
    after_previous();
    const uint32_t q = (uint32_t)a.q;
    const bool forced = a.relabel == PLQ_RELABEL_FORCED;
    using T = Tile<D, SHAPE>;
    __shared__ RelabelShared<T> sm;
    tile_relabel<T>(
        a, blockIdx.x, sm,
        [&](int32_t root, int32_t) {
            // the forced change's step, or the label itself
            const float u = __fmul_rn((float)keyed24(a.seed32 ^ kRootSalt, (uint32_t)root, a.sweep32),
                                      5.9604644775390625e-8f);
            const uint32_t range = forced ? q - 1u : q;
            const uint32_t draw = __float2uint_rz(__fmul_rn(u, (float)range));
            return (uint8_t)(draw >= range ? range - 1u : draw);
        },
        [&](uint32_t s, int count, const uint32_t (&r)[4], const uint8_t *value, const T &, uint32_t) {
            uint8_t v[4] = {value[r[0]], value[r[1]], value[r[2]], value[r[3]]};
            if (forced)
                for (int k = 0; k < count; ++k) v[k] = (uint8_t)((a.state[s + (uint32_t)k] + 1u + v[k]) % q);
            store_row(a.state, s, count, v);
        });
}

// rand 0.10 random_range(0..range) for range < 2^32 whose first draw is the
// output of state st: returns the value and whether a second draw was taken.
__device__ __forceinline__ uint32_t next_below_from(const ClusterArgs &a, u128 st, uint32_t range, bool &second) {
    uint32_t x = (uint32_t)xsl_rr(st);
    uint64_t m = (uint64_t)x * range;
    uint32_t result = (uint32_t)(m >> 32), lo = (uint32_t)m;
    second = lo > (uint32_t)(0u - range);
    if (second) {
        st = pcg_step(st, a.inc);
        uint32_t x2 = (uint32_t)xsl_rr(st);
        uint32_t hi2 = (uint32_t)(((uint64_t)x2 * range) >> 32);
        if ((uint64_t)lo + hi2 > 0xFFFFFFFFull) result += 1;
    }
    return result;
}

// The fresh label of a cluster (ClusterUpdate::fresh_label, updater.rs:507-521)
// whose first draw is the output of st: next_below(q), or with forced change the
// proposal of updater.rs:659-668 (q >= 3 there).
__device__ __forceinline__ uint32_t label_range(const ClusterArgs &a) {
    return (uint32_t)(a.relabel == PLQ_RELABEL_REDRAW ? a.q : a.q - 1);
}
__device__ __forceinline__ uint32_t fresh_label(const ClusterArgs &a, u128 st, uint32_t cur, bool &second) {
    const uint32_t d = next_below_from(a, st, label_range(a), second);
    return a.relabel == PLQ_RELABEL_REDRAW ? d : d + (d >= cur ? 1u : 0u);
}

// stream: rank of each root among roots (first-encounter order), and each
// root's fresh label as if no label before it took a second draw: rank r draws at
// bond_end + r, so a thread steps the stream from one root to the next.  Whether an
// output asks for a second draw is a property of the output alone, so this pass
// also lists every such place of the stream (SecondDraws resolves them).
template <int D>
__global__ void __launch_bounds__(kThreads) root_rank_kernel(ClusterArgs a) {
    after_previous();
    const int64_t n = a.g.n_sites;
    const int64_t chunk = take_chunk(a, true);
    if (chunk >= a.n_chunks) {
        if (threadIdx.x == 0) atomicOr(&a.ctrl->status, kStatusBounds);
        return;
    }
    const int64_t s0 = chunk * kChunk + (int64_t)threadIdx.x * kSitesPerThread;
    // the tiles' local roots are marked in fresh (tile_hook_kernel); those still their own parent are roots
    int count = 0;
    uint32_t mask = 0;
    if (s0 + kSitesPerThread <= n) {  // s0 is a multiple of 8
        const uint64_t f = *reinterpret_cast<const uint64_t *>(a.fresh + s0);
#pragma unroll
        for (int i = 0; i < kSitesPerThread; ++i) mask |= (uint32_t)((f >> (8 * i)) & 1u) << i;
    } else {
#pragma unroll
        for (int i = 0; i < kSitesPerThread; ++i)
            if (s0 + i < n) mask |= (uint32_t)(a.fresh[s0 + i] & 1u) << i;
    }
#pragma unroll
    for (int i = 0; i < kSitesPerThread; ++i)
        if (((mask >> i) & 1u) && a.parent[s0 + i] != (int32_t)(s0 + i)) mask &= ~(1u << i);
    count = __popc(mask);
    int total;
    bool ok;
    uint64_t excl = chunk_scan(a, chunk, count, total, ok);
    if (!ok) return;
    __shared__ u128 s_state;
    __shared__ unsigned long long s_excl0;
    if (threadIdx.x == 0) {
        if (chunk == a.n_chunks - 1) {  // (apply_fresh_kernel adds the second draws)
            a.ctrl->scratch[0] = excl + (unsigned long long)total;
            a.ctrl->pos[0] = a.ctrl->pos[1] + excl + (unsigned long long)total;
        }
        // labels are drawn from the end of the bond draws, in root rank order
        const u128 st0 = jump(a.jump, a.at[1], excl);
        a.chunk_base[chunk].st = st0;
        a.chunk_base[chunk].rank0 = (int64_t)excl;
        s_state = st0;
        s_excl0 = excl;
    }
    __syncthreads();
    // the state after the labels, beside the draws
    if (chunk == a.n_chunks - 1 && threadIdx.x == kThreads - 1) a.at[0] = jump(a.jump, s_state, (uint64_t)total);
    if (!count) return;
    u128 st = jump(a.jump, s_state, excl - s_excl0);
    int r = (int)excl;
#pragma unroll
    for (int i = 0; i < kSitesPerThread; ++i) {
        if (!((mask >> i) & 1u)) continue;
        const int64_t s = s0 + i;
        a.rank[s] = r;
        bool second;
        a.fresh[s] = (uint8_t)fresh_label(a, st, a.state[s], second);
        if (second) {
            const int k = atomicAdd(a.event_count, 1);
            if (k < kMaxEvents) a.events[k] = r;
        }
        st = pcg_step(st, a.inc);
        ++r;
    }
}

// The labels of a sweep that take a second draw (plq_second_draws.h).
struct SecondDraws {
    int n;
    int32_t place[kMaxEvents], rank[kMaxEvents];
};

// (one thread)  False: more of them than the list holds.
__device__ __noinline__ bool second_draws(const ClusterArgs &a, int listed, SecondDraws &sd) {
    for (int i = 0; i < listed && i < kMaxEvents; ++i) sd.place[i] = a.events[i];
    const int64_t labels = (int64_t)a.ctrl->scratch[0];
    u128 st = jump(a.jump, a.at[1], (uint64_t)labels);
    return resolve_second_draws(sd.place, listed, labels, kMaxEvents, sd.rank, sd.n, [&](int64_t) {
        bool second;
        next_below_from(a, st, label_range(a), second);
        st = pcg_step(st, a.inc);
        return second;
    });
}

// The label of a cluster whose draw `before` second draws have moved, `cur` its present state.
__device__ __noinline__ uint8_t moved_label(const ClusterArgs &a, int32_t root, int32_t rank, int before, uint32_t cur) {
    const ClusterArgs::ChunkBase &cb = a.chunk_base[root / kChunk];
    bool second;
    return (uint8_t)fresh_label(a, jump(a.jump, cb.st, (uint64_t)((int64_t)rank - cb.rank0) + (uint64_t)before), cur, second);
}

// stream: the labels to the sites, those behind a second draw drawn again (by every tile that
// meets the cluster), and the position behind the second draws.  A sweep without one, nearly
// every sweep, pays a load per CTA for it.
template <int D, int SHAPE>
__global__ void __launch_bounds__(kThreads, 8) apply_fresh_kernel(const __grid_constant__ ClusterArgs a) {
    using T = Tile<D, SHAPE>;
    __shared__ RelabelShared<T> sm;
    __shared__ SecondDraws sd;
    after_previous();
    const int listed = *a.event_count;
    if (listed) {
        if (threadIdx.x == 0) {
            if (!second_draws(a, listed, sd)) atomicOr(&a.ctrl->status, kStatusQueueOverflow);
            if (blockIdx.x == 0) {
                const unsigned long long draws = a.ctrl->scratch[0] + (unsigned long long)sd.n;
                a.ctrl->pos[0] = a.ctrl->pos[1] + draws;
                a.at[0] = jump(a.jump, a.at[1], draws);
            }
        }
        __syncthreads();
    }
    tile_relabel<T>(
        a, blockIdx.x, sm,
        [&](int32_t root, int32_t s) {
            if (listed) {
                const int32_t rank = a.rank[root];
                int before = 0;
                for (int k = 0; k < sd.n; ++k) before += sd.rank[k] < rank;
                // (a cluster's sites agree, and this CTA alone writes its own)
                if (before) return moved_label(a, root, rank, before, a.state[s]);
            }
            return a.fresh[root];
        },
        [&](uint32_t s, int count, const uint32_t (&r)[4], const uint8_t *value, const T &, uint32_t) {
            const uint8_t v[4] = {value[r[0]], value[r[1]], value[r[2]], value[r[3]]};
            store_row(a.state, s, count, v);
        });
}

// ------------------------------------------------------- Wolff (keyed)
// An update by growth from the seed site is a chain of generations, some 70 for
// a critical 3D cluster of 10^4 sites and over 1000 for a 2D one of 10^5: at
// about a microsecond each, growth takes many times what labelling the whole
// lattice does on all SMs (2D Ising 1024^2: 3.9 ms an update against 0.034).
// But far from criticality, and for many seeds at it, the cluster is a few
// sites, which a few generations find.  So one CTA of a persistent launch grows
// each update's cluster and goes on to the next as long as they are small; half-way
// to its limit it calls the others, which label the tiles as in a Swendsen-Wang
// sweep while it grows on (they stop when the growth has ended first).  A cluster
// that outgrew the limits is the one the seed site has in the decomposition.  Grid barriers: none for an update of
// fewer generations, one where the growth ended after the call, three for a
// large cluster.
//
// us per update, growth on one CTA / this, in equilibrium at beta_c: 3D Ising
// 128^3 536 / 45, 48 x 50 x 54 226 / 21, 2D Ising 1024^2 3750 / 35, 194 x 172
// 592 / 26, 32 x 26 87 / 23, 3D Potts q = 3 80^3 60 / 19; 3D Ising 128^3 at
// beta = 0.1 4.1 / 3.0.  Calling at generation 4 was 2 us faster on the smallest
// lattices and 1.5 us slower on the hot one.
//
// The limits grow with the labelling they save: 12 generations, and one more for
// each 32 tiles up to 28; the call comes half-way (3D Potts q = 4 128^3 in its
// disordered phase, clusters of some 10^3 sites: 18 us an update by growth alone,
// 25 with 12 generations everywhere, 11 so).
__host__ __device__ inline int grow_generations(uint32_t n_tiles) { return 12 + (int)(n_tiles < 512u ? n_tiles / 32u : 16u); }
constexpr uint32_t kGrowMembers = 2048;
constexpr uint32_t kGrowTable = 8192;  // members' hash table: never more than half full
static_assert(kGrowMembers + kThreads <= kGrowTable / 2, "room for a pass past the limit");

struct GrowShared {
    int32_t table[kGrowTable];
    int32_t queue[kGrowMembers];
    uint32_t tail, min_site;
};

// Device-side state of a Wolff chain's launches.
struct WolffSync {
    unsigned int count, gen;      // the grid barrier's arrivals and generation
    unsigned long long call;      // the update the CTAs are called to label (increasing over all launches)
    unsigned long long small[2];  // by update parity: the last called update whose cluster the growth found whole
};

// Grid barrier (all CTAs are co-resident: a cooperative launch); bounded.
__device__ void wolff_barrier(WolffSync *w, Control *ctrl) {
    __syncthreads();
    if (threadIdx.x == 0 && gridDim.x > 1) {
        volatile unsigned int *gen = &w->gen;
        const unsigned int g = *gen;
        __threadfence();
        if (atomicAdd(&w->count, 1u) == gridDim.x - 1) {
            atomicExch(&w->count, 0u);
            __threadfence();
            atomicAdd(&w->gen, 1u);
        } else {
            for (int spins = 0; *gen == g;) {
                if (++spins > (1 << 24)) {
                    atomicOr(&ctrl->status, kStatusLookbackTimeout);
                    break;
                }
                __nanosleep(20);
            }
        }
        __threadfence();
    }
    __syncthreads();
}

// The new state of the cluster rooted at `root` (cluster_relabel.wgsl:72-89).
__device__ __forceinline__ uint8_t wolff_next(const ClusterArgs &a, uint32_t sweep, uint32_t root, uint32_t cur) {
    const uint32_t q = (uint32_t)a.q;
    const float u = __fmul_rn((float)keyed24(a.seed32 ^ kRootSalt, root, sweep), 5.9604644775390625e-8f);
    if (a.relabel == PLQ_RELABEL_FORCED) {
        uint32_t step = __float2uint_rz(__fmul_rn(u, (float)(q - 1u)));
        if (step >= q - 1u) step = q - 2u;
        return (uint8_t)((cur + 1u + step) % q);
    }
    uint32_t draw = __float2uint_rz(__fmul_rn(u, (float)q));
    if (draw >= q) draw = q - 1u;
    return (uint8_t)draw;
}

// Calls the waiting CTAs to update `id`: everything this CTA has written is visible to them.
__device__ __forceinline__ void wolff_call(WolffSync *w, unsigned long long id) {
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        *(volatile unsigned long long *)&w->call = id;
    }
}

// Growth from `seed` within the limits, one thread per (member, direction): true
// if the whole cluster was found, its members then in sm.queue.  `called`: the
// other CTAs were called to this update.
template <int D>
__device__ bool wolff_grow(const ClusterArgs &a, uint32_t sweep, uint32_t seed, uint8_t cur, GrowShared &sm, WolffSync *w,
                           unsigned long long id, int generations, bool &called) {
    const BondCut cut(a, sweep);
    const bool bonds = BondCut::some(a);
    auto slot_of = [](uint32_t v) { return (v * 0x9e3779b1u) >> 19; };  // kGrowTable = 2^13
    for (uint32_t i = threadIdx.x; i < kGrowTable; i += kThreads) sm.table[i] = -1;
    __syncthreads();
    if (threadIdx.x == 0) {
        sm.table[slot_of(seed)] = (int32_t)seed;
        sm.queue[0] = (int32_t)seed;
        sm.tail = 1;
        sm.min_site = seed;
    }
    __syncthreads();
    uint32_t begin = 0, end = 1;
    called = false;
    for (int gen = 0; begin < end && gen < generations && end <= kGrowMembers; ++gen) {
        if (gen == generations / 2) {
            wolff_call(w, id);
            called = true;
        }
        const uint32_t work = (end - begin) * (2u * D);
        for (uint32_t i = threadIdx.x; i < work; i += kThreads) {
            const uint32_t k = i % (2u * D), u = (uint32_t)sm.queue[begin + i / (2u * D)];
            int32_t x[D];
            site_coords<D>(a.g, u, x);
            const bool plus = (k & 1u) == 0;
            uint32_t v = 0;
#pragma unroll
            for (int mu = 0; mu < D; ++mu)
                if ((k >> 1) == (uint32_t)mu) v = (uint32_t)(plus ? nbr_plus(a.g, u, x, mu) : nbr_minus(a.g, u, x, mu));
            const uint8_t sv = a.state[v];
            if ((sv == cur) & bonds & cut.open((plus ? u : v) * (uint32_t)D + (k >> 1))) {
                // (past the limit the growth has failed: the tail only has to stay above it)
                if (*(volatile uint32_t *)&sm.tail > kGrowMembers) break;
                uint32_t slot = slot_of(v);
                int32_t held;
                while ((held = atomicCAS(&sm.table[slot], -1, (int32_t)v)) != -1 && held != (int32_t)v)
                    slot = (slot + 1u) % kGrowTable;
                if (held == -1) {
                    const uint32_t p = atomicAdd(&sm.tail, 1u);
                    if (p < kGrowMembers) sm.queue[p] = (int32_t)v;
                    if (v < sm.min_site) atomicMin(&sm.min_site, v);
                }
            }
        }
        __syncthreads();
        begin = end;
        end = sm.tail;
        __syncthreads();
    }
    if (begin < end && !called) {
        wolff_call(w, id);
        called = true;
    }
    return begin == end;
}

template <int D, int SHAPE>
__global__ void __launch_bounds__(kThreads, 4)
wolff_kernel(ClusterArgs a, WolffSync *w, uint32_t n_tiles, unsigned long long launch) {
    using T = Tile<D, SHAPE>;
    constexpr size_t kBytes = sizeof(LabelShared<T>) > sizeof(RelabelShared<T>)
                                  ? (sizeof(LabelShared<T>) > sizeof(GrowShared) ? sizeof(LabelShared<T>) : sizeof(GrowShared))
                                  : (sizeof(RelabelShared<T>) > sizeof(GrowShared) ? sizeof(RelabelShared<T>) : sizeof(GrowShared));
    __shared__ __align__(16) unsigned char s_buf[kBytes];
    __shared__ int s_stop;
    __shared__ unsigned long long s_call;
    __shared__ uint32_t s_root, s_flipped;
    const uint32_t n = (uint32_t)a.g.n_sites;
    const bool grower = blockIdx.x == 0;  // (there are others: a grid has a CTA per tile and one more, or fills the chip)
    const unsigned long long base = launch << 32, last = base | 0xFFFFFFFFull;  // (a launch has less than 2^32 - 1 updates)
    unsigned long long id = base;  // update up is base + up + 1
    // a CTA that waits for a call reads the word until the growing CTA has been through every
    // update before it, at a few microseconds each; the limit is some 100 times that
    const unsigned long long spin_limit = (1ull << 24) + (a.updates << 14);
    for (;;) {
        if (grower) {
            if (id == base + a.updates) break;
            ++id;
        } else {
            if (threadIdx.x == 0) {
                volatile unsigned long long *call = &w->call;
                unsigned long long next, spins = 0;
                while ((next = *call) <= id) {
                    if (++spins > spin_limit) {
                        atomicOr(&a.ctrl->status, kStatusLookbackTimeout);
                        next = last;
                        break;
                    }
                    __nanosleep(50);
                }
                __threadfence();
                s_call = next;
            }
            __syncthreads();
            id = s_call;
            __syncthreads();
            if (id == last) break;
        }
        const uint32_t sweep = a.sweep32 + (uint32_t)(id - base - 1ull);
        volatile unsigned long long *small = &w->small[id & 1ull];
        // seed site (cluster_relabel.wgsl:55-61)
        const float us = __fmul_rn((float)keyed24(a.seed32 ^ kSeedSalt, 0u, sweep), 5.9604644775390625e-8f);
        uint32_t seed = __float2uint_rz(__fmul_rn(us, (float)n));
        if (seed >= n) seed = n - 1u;
        // (another CTA may read a state the growth has changed already, but then has no use for it)
        const uint8_t cur = a.state[seed];
        __syncthreads();
        if (grower) {
            GrowShared &sm = *reinterpret_cast<GrowShared *>(s_buf);
            if (threadIdx.x == 0) a.ctrl->scratch[1] = 0;
            bool called;
            const bool whole = wolff_grow<D>(a, sweep, seed, cur, sm, w, id, grow_generations(n_tiles), called);
            if (whole) {
                // (the others may be reading states for tiles that no one will use)
                const uint8_t next = wolff_next(a, sweep, sm.min_site, cur);
                for (uint32_t i = threadIdx.x; i < sm.tail; i += kThreads) a.state[sm.queue[i]] = next;
                if (threadIdx.x == 0) {
                    a.ctrl->scratch[1] = sm.tail;
                    if (called) *small = id;
                }
                __syncthreads();
                if (!called) continue;
            }
        } else {
            LabelShared<T> &sm = *reinterpret_cast<LabelShared<T> *>(s_buf);
            for (uint32_t tile = blockIdx.x - 1u; tile < n_tiles; tile += gridDim.x - 1u) {
                if (threadIdx.x == 0) s_stop = wolff_ended_by_growth(*small, id);
                __syncthreads();
                if (s_stop) break;
                if constexpr (SHAPE == kFlat) label_flat<D, true>(a, sweep, tile, sm.p);
                else label_tile<D, SHAPE, true>(a, sweep, tile, sm);
                __syncthreads();
            }
        }
        wolff_barrier(w, a.ctrl);
        if (threadIdx.x == 0) s_stop = wolff_ended_by_growth(*small, id);
        __syncthreads();
        if (s_stop) continue;
        if constexpr (SHAPE == kFlat) unite_flat_edges<D, true>(a, sweep);
        else unite_edges<D, SHAPE, true>(a, sweep);
        wolff_barrier(w, a.ctrl);
        // the seed's cluster takes its new state
        if (threadIdx.x == 0) {
            int32_t x[D];
            site_coords<D>(a.g, seed, x);
            const T t(a.g);
            s_root = (uint32_t)find_root_ro(a.parent, (int32_t)t.local_root(a.local_root, seed, x), a.cap, a.ctrl);
            s_flipped = 0;
        }
        __syncthreads();
        const int32_t root = (int32_t)s_root;
        const uint8_t next = wolff_next(a, sweep, s_root, cur);
        uint32_t flipped = 0;
        RelabelShared<T> &sm = *reinterpret_cast<RelabelShared<T> *>(s_buf);
        for (uint32_t tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
            tile_relabel<T>(
                a, tile, sm, [&](int32_t r, int32_t) { return (uint8_t)(r == root ? 1 : 0); },
                [&](uint32_t s, int count, const uint32_t (&r)[4], const uint8_t *value, const T &, uint32_t) {
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        if (k < count && value[r[k]]) {
                            a.state[s + (uint32_t)k] = next;
                            ++flipped;
                        }
                });
            __syncthreads();
        }
        flipped = __reduce_add_sync(0xffffffffu, flipped);
        if ((threadIdx.x & 31u) == 0 && flipped) atomicAdd(&s_flipped, flipped);
        __syncthreads();
        if (threadIdx.x == 0 && s_flipped) atomicAdd(&a.ctrl->scratch[1], (unsigned long long)s_flipped);
        wolff_barrier(w, a.ctrl);
    }
    if (grower) wolff_call(w, last);
}

// ------------------------------------------------------------ sizes
// Cluster sizes.  A warp adds up the sites of each distinct root among its 32,
// into its CTA's table of recent roots where that root has (or finds free) its
// slot, else in memory; the table is added to memory at the end.  A cluster
// that holds a good part of the lattice so takes one global atomic per CTA: with
// one per warp on the same address this kernel took 534 of the 617 us of a
// histogram of 4096^2 at beta_c (now 240, the flattening of the labels included).
constexpr int kSizeSlots = 512;
__global__ void __launch_bounds__(kThreads) sizes_kernel(const int32_t *parent, int32_t *size, int64_t n) {
    __shared__ int32_t s_root[kSizeSlots], s_count[kSizeSlots];
    for (int i = threadIdx.x; i < kSizeSlots; i += blockDim.x) {
        s_root[i] = -1;
        s_count[i] = 0;
    }
    __syncthreads();
    const int64_t n_pad = (n + 31) & ~(int64_t)31;  // whole warps per iteration: the match below is warp-wide
    for (int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; s < n_pad; s += (int64_t)gridDim.x * blockDim.x) {
        const int32_t r = s < n ? parent[s] : -1;
        const unsigned peers = __match_any_sync(0xffffffffu, r);
        if (r >= 0 && (int)(threadIdx.x & 31u) == __ffs(peers) - 1) {
            const int slot = (int)(((uint32_t)r * 0x9e3779b1u) >> 23);  // kSizeSlots = 2^9
            const int32_t held = atomicCAS(&s_root[slot], -1, r);
            if (held == -1 || held == r) atomicAdd(&s_count[slot], __popc(peers));
            else atomicAdd(&size[r], __popc(peers));
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kSizeSlots; i += blockDim.x)
        if (s_count[i]) atomicAdd(&size[s_root[i]], s_count[i]);
}
// Clusters per size bin [2^k, 2^(k+1)): counted per CTA in shared memory (bins
// 0..31 cover every int32 size), one global atomic per bin per CTA.
__global__ void size_hist_kernel(const int32_t *parent, const int32_t *size, int64_t n, long long *hist, int nbins) {
    __shared__ unsigned int bins[32];
    if (threadIdx.x < 32) bins[threadIdx.x] = 0;
    __syncthreads();
    for (int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; s < n; s += (int64_t)gridDim.x * blockDim.x) {
        if (parent[s] != (int32_t)s) continue;
        atomicAdd(&bins[31 - __clz(size[s])], 1u);
    }
    __syncthreads();
    if (threadIdx.x < 32 && bins[threadIdx.x]) {
        int bin = (int)threadIdx.x;
        if (bin >= nbins) bin = nbins - 1;
        atomicAdd((unsigned long long *)&hist[bin], (unsigned long long)bins[threadIdx.x]);
    }
}

// ------------------------------------------------------------ host side
struct ClusterDev {
    uint8_t *bonds = nullptr;
    int32_t *parent = nullptr;
    uint16_t *local_root = nullptr;
    uint8_t *fresh = nullptr;
    int32_t *rank = nullptr;
    ClusterArgs::ChunkBase *chunk_base = nullptr;
    WolffSync *wolff = nullptr;
    unsigned wolff_grid = 0;
    uint64_t wolff_launches = 0;
    unsigned long long *desc = nullptr;
    int64_t n_chunks = 0;
    int64_t n_tiles = 0;  // CTAs of the kernels that take a tile each
    TileShape shape = kSmall;
    int32_t *events = nullptr;
    int *event_count = nullptr;
    int32_t *sizes = nullptr;
    uint32_t kp24 = 0;
    uint64_t kp53 = 0;
    uint64_t lookback_launches = 0;
    u128 *at = nullptr;
    bool decomposed = false;
    bool flat = false;  // every site's parent is its root (flatten_kernel has run since the last sweep)
};

unsigned grid_stride_blocks(int64_t n) {
    int64_t b = (n + kThreads - 1) / kThreads;
    if (b > 148 * 16) b = 148 * 16;
    return (unsigned)(b < 1 ? 1 : b);
}

ClusterArgs cluster_args(plq_chain *c) {
    ClusterDev *cd = static_cast<ClusterDev *>(c->cl);
    ClusterArgs a;
    std::memset(&a, 0, sizeof a);
    a.state = c->d_state;
    a.bonds = cd->bonds;
    a.parent = cd->parent;
    a.local_root = cd->local_root;
    a.fresh = cd->fresh;
    a.rank = cd->rank;
    a.chunk_base = cd->chunk_base;
    a.g = c->g;
    a.q = c->q;
    a.extent = c->desc.extent;
    a.relabel = c->desc.relabel;
    a.seed32 = c->seed32;
    a.sweep32 = (uint32_t)c->sweeps_done;
    a.kp24 = cd->kp24;
    a.kp53 = cd->kp53;
    a.jump = c->d_jump;
    a.at = cd->at;
    a.inc = c->inc;
    a.ctrl = c->d_ctrl;
    a.desc = cd->desc;
    a.n_chunks = cd->n_chunks;
    a.cap = (c->desc.flags & PLQ_FLAG_TINY_PASS_CAP) ? 1 : (int)std::min<int64_t>(c->n_sites + 64, 1 << 30);
    a.events = cd->events;
    a.event_count = cd->event_count;
    return a;
}

// The kernels of one tile size (a CTA per tile, and the boundary unions).
template <int D, int SHAPE>
struct TileKernels {
    using T = Tile<D, SHAPE>;
    // The launches it makes.
    static unsigned label(const ClusterArgs &a, bool keyed, unsigned tiles, unsigned blocks, cudaStream_t st) {
        const bool edges = SHAPE != kFlat || tiles > 1;
        if (keyed) {
            launch_next(tile_hook_kernel<D, SHAPE, true>, tiles, st, a);
            if (edges) launch_next(boundary_hook_kernel<D, SHAPE, true>, blocks, st, a);
        } else {
            launch_next(tile_hook_kernel<D, SHAPE, false>, tiles, st, a);
            if (edges) launch_next(boundary_hook_kernel<D, SHAPE, false>, blocks, st, a);
        }
        return edges ? 2 : 1;
    }
    static void relabel_keyed(const ClusterArgs &a, unsigned tiles, cudaStream_t st) {
        launch_next(relabel_keyed_kernel<D, SHAPE>, tiles, st, a);
    }
    static void apply_fresh(const ClusterArgs &a, unsigned tiles, cudaStream_t st) {
        launch_next(apply_fresh_kernel<D, SHAPE>, tiles, st, a);
    }
    static cudaError_t wolff(ClusterArgs a, WolffSync *w, uint32_t tiles, unsigned long long launch, unsigned grid,
                             cudaStream_t st) {
        void *params[] = {&a, &w, &tiles, &launch};
        return cudaLaunchCooperativeKernel((const void *)wolff_kernel<D, SHAPE>, dim3(grid), dim3(kThreads), params, 0, st);
    }
    // A CTA per tile and the growing one, as many as are resident together.
    static cudaError_t wolff_grid(int64_t tiles, int sm_count, unsigned &grid) {
        int per_sm = 0;
        const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, wolff_kernel<D, SHAPE>, kThreads, 0);
        grid = (unsigned)std::min<int64_t>(tiles + 1, (int64_t)per_sm * sm_count);
        return e != cudaSuccess || grid >= 2 ? e : cudaErrorLaunchOutOfResources;
    }
    static void flatten(const ClusterArgs &a, unsigned tiles, cudaStream_t st) {
        flatten_kernel<D, SHAPE><<<tiles, kThreads, 0, st>>>(a);
    }
};

template <int D, class K>
int sweep_t(plq_chain *c, uint64_t sweeps) {
    ClusterDev *cd = static_cast<ClusterDev *>(c->cl);
    const bool stream = c->desc.rng == PLQ_RNG_STREAM;
    const int64_t n = c->n_sites;
    const unsigned gs = grid_stride_blocks(n);
    if (c->desc.extent == PLQ_EXTENT_SEEDED) {
        for (uint64_t left = sweeps; left;) {
            ClusterArgs a = cluster_args(c);
            // (launches of some 20 ms, between which other streams' work takes its turn)
            a.updates = std::min<uint64_t>(left, 1024);
            const cudaError_t e = K::wolff(a, cd->wolff, (uint32_t)cd->n_tiles, ++cd->wolff_launches, cd->wolff_grid,
                                           c->stream);
            c->launches++;
            if (e != cudaSuccess) return plq_fail(PLQ_ECUDA, std::string("wolff launch: ") + cudaGetErrorString(e));
            c->sweeps_done += a.updates;
            left -= a.updates;
        }
        cd->decomposed = false;
        return PLQ_OK;
    }
    for (uint64_t t = 0; t < sweeps; ++t) {
        ClusterArgs a = cluster_args(c);
        auto lookback = [&](ClusterArgs &x) {
            x.epoch = (uint32_t)(cd->lookback_launches + 1);
            x.ticket_base = cd->lookback_launches * (uint64_t)cd->n_chunks;
            cd->lookback_launches++;
        };
        if (stream) {
            // PCG stream: the bond draws sit at scanned positions, so they are made in one pass
            lookback(a);
            launch_next(bonds_kernel<D, true>, (unsigned)cd->n_chunks, c->stream, a);
            c->launches += 1 + K::label(a, false, (unsigned)cd->n_tiles, gs, c->stream);
        } else {
            // keyed: each bond is a closed form of its index, evaluated where it is used
            c->launches += K::label(a, true, (unsigned)cd->n_tiles, gs, c->stream);
        }
        if (!stream) {
            K::relabel_keyed(a, (unsigned)cd->n_tiles, c->stream);
            c->launches++;
        } else {
            lookback(a);
            // ranks, and the labels with no second draws known; the labels to the sites
            launch_next(root_rank_kernel<D>, (unsigned)cd->n_chunks, c->stream, a);
            K::apply_fresh(a, (unsigned)cd->n_tiles, c->stream);
            c->launches += 2;
        }
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return plq_fail(PLQ_ECUDA, std::string("cluster sweep: ") + cudaGetErrorString(e));
        c->sweeps_done++;
        cd->decomposed = true;
        cd->flat = false;
    }
    return PLQ_OK;
}

// f on the kernels of the chain's tiles.
template <int D, class F>
auto with_tiles(const plq_chain *c, F f) {
    const TileShape shape = static_cast<ClusterDev *>(c->cl)->shape;
    if constexpr (D >= 2) {
        if (shape == kFlat) return f(TileKernels<D, kFlat>());
        if (shape == kWide) return f(TileKernels<D, kWide>());
        if (shape == kLarge) return f(TileKernels<D, kLarge>());
    }
    if constexpr (D == 2) {
        if (shape == kNarrow) return f(TileKernels<D, kNarrow>());
    }
    return f(TileKernels<D, kSmall>());
}

template <int D>
int sweep_d(plq_chain *c, uint64_t sweeps) {
    return with_tiles<D>(c, [&](auto k) { return sweep_t<D, decltype(k)>(c, sweeps); });
}

}  // namespace

int cluster_validate(const plq_chain_desc *d) {
    if (d->extent == PLQ_EXTENT_SEEDED && d->rng == PLQ_RNG_STREAM)
        return plq_fail(PLQ_EUNSUPPORTED,
                        "Wolff on the PCG stream draws in grow_cluster's sequential FIFO order; this device path "
                        "runs the seeded extent on the keyed stream only");
    return PLQ_OK;
}

template <int D>
static cudaError_t wolff_grid_d(plq_chain *c, unsigned &grid) {
    ClusterDev *cd = static_cast<ClusterDev *>(c->cl);
    return with_tiles<D>(c, [&](auto k) { return decltype(k)::wolff_grid(cd->n_tiles, c->ctx->sm_count, grid); });
}

static cudaError_t wolff_grid(plq_chain *c, unsigned &grid) {
    switch (c->d) {
        case 1: return wolff_grid_d<1>(c, grid);
        case 2: return wolff_grid_d<2>(c, grid);
        case 3: return wolff_grid_d<3>(c, grid);
        case 4: return wolff_grid_d<4>(c, grid);
        case 5: return wolff_grid_d<5>(c, grid);
        case 6: return wolff_grid_d<6>(c, grid);
        case 7: return wolff_grid_d<7>(c, grid);
        default: return wolff_grid_d<8>(c, grid);
    }
}

// The CTAs of a Wolff launch, of `most` that are resident together.  The launch is cooperative, and
// launches of chains on other streams run beside it only while all of their CTAs fit: where
// large clusters are rare, CTAs that wait to label them would keep other chains waiting
// (eight hot chains, 3D Ising 128^3 at beta = 0.1 on eight streams: 21 us an update of each with
// 513 CTAs, 2.8 with 33, 2.6 alone).  A bond whose ends are not connected otherwise is open with
// probability t = p / (p + q (1 - p)), so on a tree generation k of a growth holds 2 d t ((2 d - 1) t)^(k - 1)
// sites; that bounds how often a cluster outgrows the limit, and a label pass takes
// about 8 us for each time the tiles exceed the CTAs: the CTAs keep that to 0.2 us an update, and
// a pass to 16 tiles a CTA (a cold start's first clusters are large at any coupling).
static unsigned wolff_ctas(unsigned most, int64_t n_tiles, int d, int q, double p) {
    const double t = p / (p + q * (1 - p)), c = (2 * d - 1) * t;
    if (!(c < 1)) return most;
    const double outgrown = 2 * d * t * std::pow(c, grow_generations((uint32_t)n_tiles) - 1);
    const double wanted = 1 + std::max(40 * outgrown, 1.0 / 16) * (double)n_tiles;
    return wanted < most ? std::max(2u, (unsigned)wanted) : most;
}

int cluster_create(plq_chain *c) {
    ClusterDev *cd = new ClusterDev();
    c->cl = cd;
    const int64_t n = c->n_sites;
    double p = plq_bond_probability(c->desc.model, c->desc.j, c->desc.beta);
    // bond open iff u < p: keyed in f32 (cluster_prelude.wgsl:77), stream in f64 (updater.rs:570-572)
    float p32 = (float)p;
    uint32_t lo = 0, hi = 1u << 24;
    while (lo < hi) {
        uint32_t mid = lo + (hi - lo) / 2;
        if ((float)mid * (1.0f / 16777216.0f) < p32) lo = mid + 1;
        else hi = mid;
    }
    cd->kp24 = lo;
    uint64_t lo53 = 0, hi53 = 1ull << 53;
    while (lo53 < hi53) {
        uint64_t mid = lo53 + (hi53 - lo53) / 2;
        if ((double)mid * (1.0 / 9007199254740992.0) < p) lo53 = mid + 1;
        else hi53 = mid;
    }
    cd->kp53 = lo53;
    c->pass_cap = (c->desc.flags & PLQ_FLAG_TINY_PASS_CAP) ? 1 : std::min<int64_t>(n + 64, 1 << 30);
    cd->n_chunks = (n + kChunk - 1) / kChunk;
    size_t tile_sites = 0;
    auto tiles = [&](auto dims) {
        constexpr int D = decltype(dims)::value;
        cd->shape = tile_shape<D>(c->g, c->ctx->sm_count, c->desc.rng == PLQ_RNG_KEYED);
        with_tiles<D>(c, [&](auto k) {
            using T = typename decltype(k)::T;
            cd->n_tiles = T(c->g).tiles(n);
            tile_sites = (size_t)cd->n_tiles * T::kSites;
        });
    };
    switch (c->d) {  // (d > 3 has the tiles of d = 3)
        case 1: tiles(std::integral_constant<int, 1>()); break;
        case 2: tiles(std::integral_constant<int, 2>()); break;
        default: tiles(std::integral_constant<int, 3>()); break;
    }
    cudaError_t e = cudaSuccess;
    auto alloc = [&](void **p, size_t bytes) {
        if (e == cudaSuccess) e = cudaMalloc(p, bytes);
    };
    if (c->desc.extent == PLQ_EXTENT_SEEDED) {
        alloc((void **)&cd->wolff, sizeof(WolffSync));
        if (e == cudaSuccess) e = cudaMemsetAsync(cd->wolff, 0, sizeof(WolffSync), c->stream);
        if (e == cudaSuccess) e = wolff_grid(c, cd->wolff_grid);
        if (e == cudaSuccess) cd->wolff_grid = wolff_ctas(cd->wolff_grid, cd->n_tiles, c->d, c->q, p);
        alloc((void **)&cd->parent, sizeof(int32_t) * (size_t)n);
        alloc((void **)&cd->local_root, sizeof(uint16_t) * tile_sites);
    } else {
        alloc((void **)&cd->bonds, (size_t)n);
        alloc((void **)&cd->parent, sizeof(int32_t) * (size_t)n);
        alloc((void **)&cd->local_root, sizeof(uint16_t) * tile_sites);
        alloc((void **)&cd->desc, sizeof(unsigned long long) * (size_t)cd->n_chunks);
        if (e == cudaSuccess)
            e = cudaMemsetAsync(cd->desc, 0, sizeof(unsigned long long) * (size_t)cd->n_chunks, c->stream);
        if (c->desc.rng == PLQ_RNG_STREAM) {
            alloc((void **)&cd->fresh, (size_t)n);
            alloc((void **)&cd->rank, sizeof(int32_t) * (size_t)n);
            alloc((void **)&cd->chunk_base, sizeof(ClusterArgs::ChunkBase) * (size_t)cd->n_chunks);
            alloc((void **)&cd->events, sizeof(int32_t) * kMaxEvents);
            alloc((void **)&cd->event_count, sizeof(int));
            alloc((void **)&cd->at, 2 * sizeof(u128));
            if (e == cudaSuccess) e = cudaMemcpyAsync(cd->at, &c->base, sizeof(u128), cudaMemcpyHostToDevice, c->stream);
        }
    }
    if (e != cudaSuccess)
        return plq_fail(e == cudaErrorMemoryAllocation ? PLQ_ENOMEM : PLQ_ECUDA,
                        std::string("cluster buffers: ") + cudaGetErrorString(e));
    return PLQ_OK;
}

int cluster_sweep_n(plq_chain *c, uint64_t sweeps) {
    switch (c->d) {
        case 1: return sweep_d<1>(c, sweeps);
        case 2: return sweep_d<2>(c, sweeps);
        case 3: return sweep_d<3>(c, sweeps);
        case 4: return sweep_d<4>(c, sweeps);
        case 5: return sweep_d<5>(c, sweeps);
        case 6: return sweep_d<6>(c, sweeps);
        case 7: return sweep_d<7>(c, sweeps);
        case 8: return sweep_d<8>(c, sweeps);
        default: return plq_fail(PLQ_EINVAL, "dimension out of range");
    }
}

int cluster_sweep(plq_chain *c) { return cluster_sweep_n(c, 1); }

void cluster_free(plq_chain *c) {
    ClusterDev *cd = static_cast<ClusterDev *>(c->cl);
    if (!cd) return;
    void *ptrs[] = {cd->bonds, cd->parent, cd->local_root, cd->fresh, cd->rank, cd->chunk_base, cd->wolff, cd->at,
                    cd->desc, cd->events, cd->event_count, cd->sizes};
    for (void *p : ptrs)
        if (p) cudaFree(p);
    delete cd;
    c->cl = nullptr;
}

template <int D>
static void flatten_d(plq_chain *c) {
    ClusterDev *cd = static_cast<ClusterDev *>(c->cl);
    with_tiles<D>(c, [&](auto k) { decltype(k)::flatten(cluster_args(c), (unsigned)cd->n_tiles, c->stream); });
}

static void flatten(plq_chain *c) {
    ClusterDev *cd = static_cast<ClusterDev *>(c->cl);
    if (cd->flat) return;
    switch (c->d) {
        case 1: flatten_d<1>(c); break;
        case 2: flatten_d<2>(c); break;
        case 3: flatten_d<3>(c); break;
        case 4: flatten_d<4>(c); break;
        case 5: flatten_d<5>(c); break;
        case 6: flatten_d<6>(c); break;
        case 7: flatten_d<7>(c); break;
        default: flatten_d<8>(c); break;
    }
    c->launches++;
    cd->flat = true;
}

int cluster_labels(plq_chain *c, int32_t *out) {
    ClusterDev *cd = static_cast<ClusterDev *>(c->cl);
    if (!cd || !cd->decomposed) return plq_fail(PLQ_EINVAL, "no decomposition yet (run a Swendsen-Wang sweep first)");
    flatten(c);
    cudaError_t e = plq_readback(out, cd->parent, sizeof(int32_t) * (size_t)c->n_sites, c->ctx->device, c->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
    if (e != cudaSuccess) return plq_fail(PLQ_ECUDA, std::string("labels read: ") + cudaGetErrorString(e));
    return PLQ_OK;
}

int cluster_size_histogram(plq_chain *c, int64_t *hist, int32_t nbins) {
    ClusterDev *cd = static_cast<ClusterDev *>(c->cl);
    if (!cd || nbins <= 0) return plq_fail(PLQ_EINVAL, "bad arguments");
    std::vector<long long> h((size_t)nbins, 0);
    if (c->desc.extent == PLQ_EXTENT_SEEDED) {
        unsigned long long members = 0;
        cudaMemcpyAsync(&members, &c->d_ctrl->scratch[1], sizeof members, cudaMemcpyDeviceToHost, c->stream);
        cudaError_t e = cudaStreamSynchronize(c->stream);
        if (e != cudaSuccess) return plq_fail(PLQ_ECUDA, cudaGetErrorString(e));
        if (members) {
            int bin = 63 - __builtin_clzll(members);
            h[(size_t)std::min(bin, nbins - 1)] = 1;
        }
    } else {
        if (!cd->decomposed) return plq_fail(PLQ_EINVAL, "no decomposition yet (run a Swendsen-Wang sweep first)");
        const int64_t n = c->n_sites;
        cudaError_t e = cudaSuccess;
        if (!cd->sizes) e = cudaMalloc((void **)&cd->sizes, sizeof(int32_t) * (size_t)n);
        long long *dh = nullptr;
        if (e == cudaSuccess) e = cudaMalloc((void **)&dh, sizeof(long long) * (size_t)nbins);
        if (e != cudaSuccess) return plq_fail(PLQ_ENOMEM, cudaGetErrorString(e));
        cudaMemsetAsync(cd->sizes, 0, sizeof(int32_t) * (size_t)n, c->stream);
        cudaMemsetAsync(dh, 0, sizeof(long long) * (size_t)nbins, c->stream);
        flatten(c);
        sizes_kernel<<<grid_stride_blocks(n), kThreads, 0, c->stream>>>(cd->parent, cd->sizes, n);
        size_hist_kernel<<<grid_stride_blocks(n), kThreads, 0, c->stream>>>(cd->parent, cd->sizes, n, dh, nbins);
        c->launches += 2;
        cudaMemcpyAsync(h.data(), dh, sizeof(long long) * (size_t)nbins, cudaMemcpyDeviceToHost, c->stream);
        e = cudaStreamSynchronize(c->stream);
        cudaFree(dh);
        if (e != cudaSuccess) return plq_fail(PLQ_ECUDA, cudaGetErrorString(e));
    }
    for (int i = 0; i < nbins; ++i) hist[i] = h[(size_t)i];
    return PLQ_OK;
}
