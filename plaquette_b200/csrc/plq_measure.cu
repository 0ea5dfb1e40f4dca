// plq_measure.cu -- per-configuration measurements beyond the primaries, on
// the device-resident configuration, as exact integers:
//
//  * axis_pair_sums (src/models/mod.rs:44-61): for every axis mu and
//    displacement r = 0..L_mu/2, the sum over sites of pair(s_i, s_{i+r mu}),
//    Ising's product of signs (ising/mod.rs:84-95) or Potts's equality
//    (potts/mod.rs:218-234).  Both follow from the count of *differing* pairs
//    D: Ising n - 2D, Potts n - D.  D is counted four sites per 32-bit word
//    (SWAR nonzero-byte test on the XOR) when extent 0 is a multiple of 4.
//  * Z2Gauge::polyakov_loop (gauge/mod.rs:179-212): the sum over lines along
//    `dir` of the product of the line's links (XOR of the 0/1 states).
//  * Z2Gauge::wilson_rectangles (gauge/mod.rs:226-274): for every r, t <= max,
//    the sum over ordered planes (mu, nu) and base sites of the rectangle
//    product.  A rectangle walked +mu r, +nu t, -mu r, -nu t from x multiplies
//    line_mu(x, r) line_nu(x + r mu, t) line_mu(x + t nu, r) line_nu(x, t),
//    line_mu(x, k) the product of the k links from x along mu; one pass stores
//    those line parities as bit masks (bit k-1 for length k), a second
//    combines them, counting the -1 rectangles per (r, t) with warp ballots
//    into shared-memory counters.
// The host applies the reference's final divisions.
#include <cuda_runtime.h>

#include <algorithm>

#include "../../include/plaquette.h"
#include "plq_device.cuh"
#include "plq_measure.h"

namespace plq {

constexpr int kMeasThreads = 256;

__device__ __forceinline__ uint32_t nonzero_bytes(uint32_t t) {
    return ((((t & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | t) & 0x80808080u);
}

__device__ __forceinline__ uint32_t coord_of(const Geom &g, uint32_t s, int mu) {
    // (s / stride_mu) % L_mu with the invariant-divisor divisions of Geom
    uint32_t t = s;
    for (int k = 0; k < mu; ++k) t = fdiv(t, g.dm[k], g.dl[k]);
    return t - fdiv(t, g.dm[mu], g.dl[mu]) * (uint32_t)g.L[mu];
}

// Differing pairs (s, s + r e_mu) for the pair index blockIdx.y -> (mu, r).
__global__ void __launch_bounds__(kMeasThreads)
pair_differ_kernel(const uint8_t *cfg, Geom g, const int32_t *pair_mu, const int32_t *pair_r, long long *out) {
    const int mu = pair_mu[blockIdx.y];
    const uint32_t r = (uint32_t)pair_r[blockIdx.y];
    const uint32_t n = (uint32_t)g.n_sites;
    const uint32_t L = (uint32_t)g.L[mu];
    const uint32_t st = (uint32_t)g.stride[mu];
    const uint32_t L0 = (uint32_t)g.L[0];
    const uint32_t stride = gridDim.x * blockDim.x;
    uint32_t count = 0;
    if (L0 % 4 == 0) {
        for (uint32_t w = blockIdx.x * blockDim.x + threadIdx.x; w < n / 4; w += stride) {
            const uint32_t s = 4u * w;
            const uint32_t a = *reinterpret_cast<const uint32_t *>(cfg + s);
            uint32_t b;
            if (mu == 0) {
                const uint32_t row = fdiv(s, g.dm[0], g.dl[0]);
                const uint32_t rs = row * L0, x0 = s - rs;
                uint32_t xs = x0 + r;
                if (xs >= L0) xs -= L0;
                const uint32_t lo = xs & ~3u, hi = lo + 4u == L0 ? 0u : lo + 4u;
                const uint32_t w1 = *reinterpret_cast<const uint32_t *>(cfg + rs + lo);
                const uint32_t w2 = *reinterpret_cast<const uint32_t *>(cfg + rs + hi);
                b = __funnelshift_r(w1, w2, 8u * (xs & 3u));
            } else {
                const uint32_t c = coord_of(g, s, mu);
                const uint32_t t = c + r < L ? s + r * st : s - (L - r) * st;
                b = *reinterpret_cast<const uint32_t *>(cfg + t);
            }
            count += __popc(nonzero_bytes(a ^ b));
        }
    } else {
        for (uint32_t s = blockIdx.x * blockDim.x + threadIdx.x; s < n; s += stride) {
            const uint32_t c = coord_of(g, s, mu);
            const uint32_t t = c + r < L ? s + r * st : s - (L - r) * st;
            count += cfg[s] != cfg[t] ? 1u : 0u;
        }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) count += __shfl_down_sync(0xffffffffu, count, off);
    if ((threadIdx.x & 31) == 0 && count) atomicAdd((unsigned long long *)&out[blockIdx.y], (unsigned long long)count);
}

// ---- the same counts from bit planes.  The site-by-site scan reads the lattice
// twice per displacement, 0.8 TB of L1 and L2 traffic for the 384 of 256^3.  Here
// a state's bits (ceil(log2 q) planes) are packed once, 64 sites of a row a word,
// and a CTA holds whole lines along the axis in shared memory -- each followed
// by its own beginning, so that a displaced line is a plain offset -- and counts
// every displacement of them: one xor and population count per 64 pairs, which
// is what bounds it.  us per call (about 40 of them
// the call's copies and synchronisation): 256^3 Ising 3683 -> 155, 1024^2 605 -> 100,
// 100^3 130 -> 62.  Smaller lattices, and long thin ones, stay with the scan (pair_planes_pay).

// Word w of row r, plane p at words[p * rows * wpr + r * wpr + w]; bits past the row are 0.
template <int P>
__global__ void __launch_bounds__(kMeasThreads) pack_planes_kernel(const uint8_t *cfg, uint32_t rows, uint32_t wpr,
                                                                   uint32_t L0, uint64_t *words) {
    const uint32_t total = rows * wpr;
    const bool quads = (L0 & 3u) == 0;
    for (uint32_t u = blockIdx.x * blockDim.x + threadIdx.x; u < total; u += gridDim.x * blockDim.x) {
        const uint32_t r = u / wpr, w = u - r * wpr;
        const uint32_t len = min(64u, L0 - 64u * w);
        const uint8_t *b = cfg + (size_t)r * L0 + 64u * w;
        uint64_t out[P];
#pragma unroll
        for (int p = 0; p < P; ++p) out[p] = 0;
        if (quads) {
            for (uint32_t k = 0; k < len / 4; ++k) {
                const uint32_t v = reinterpret_cast<const uint32_t *>(b)[k];
#pragma unroll
                for (int p = 0; p < P; ++p)  // (b_i * 2^(24 - 7 i) lands at bit 24 + i)
                    out[p] |= (uint64_t)(((((v >> p) & 0x01010101u) * 0x01020408u) >> 24) & 0xFu) << (4 * k);
            }
        } else {
            for (uint32_t k = 0; k < len; ++k)
#pragma unroll
                for (int p = 0; p < P; ++p) out[p] |= (uint64_t)((b[k] >> p) & 1u) << k;
        }
#pragma unroll
        for (int p = 0; p < P; ++p) words[(size_t)p * total + u] = out[p];
    }
}

struct PairLines {
    const uint64_t *words;
    uint32_t plane;            // words of a plane
    uint32_t L, R;             // extent along the axis, displacements 1 .. R
    uint32_t outer, inner, T;  // axes > 0: words [outer][L][inner], T words of inner at once
    uint32_t wpr, slots;       // axis 0: words of a row, rows at once
    long long *out;            // R counts
};

// An axis beyond the first: thread (r, t) of a tile counts displacement r + 1 of the lines at word t.
template <int P>
__global__ void __launch_bounds__(kMeasThreads) pair_axis_kernel(PairLines a) {
    extern __shared__ uint64_t s_lines[];  // [P][L + R][T], then R counters
    const uint32_t rows = a.L + a.R;
    uint32_t *cnt = reinterpret_cast<uint32_t *>(s_lines + (size_t)P * rows * a.T);
    for (uint32_t i = threadIdx.x; i < a.R; i += blockDim.x) cnt[i] = 0;
    const uint32_t across = (a.inner + a.T - 1) / a.T, tiles = a.outer * across;
    const uint32_t total = a.R * a.T;
    // this CTA's share of the (displacement, word) pairs
    const uint32_t per = (total + gridDim.y - 1) / gridDim.y, lo = min(total, blockIdx.y * per), hi = min(total, lo + per);
    for (uint32_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const uint32_t o = tile / across, i0 = (tile - o * across) * a.T;
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < rows * a.T; i += blockDim.x) {
            const uint32_t y = i / a.T, t = i - y * a.T, yw = y < a.L ? y : y - a.L;
#pragma unroll
            for (int p = 0; p < P; ++p)
                s_lines[(size_t)p * rows * a.T + i] =
                    i0 + t < a.inner ? a.words[(size_t)p * a.plane + (size_t)(o * a.L + yw) * a.inner + i0 + t] : 0ull;
        }
        __syncthreads();
        for (uint32_t i = lo + threadIdx.x; i < hi; i += blockDim.x) {
            const uint32_t r = i / a.T, t = i - r * a.T;
            const uint64_t *x = s_lines + t, *y = x + (size_t)(r + 1) * a.T;
            uint32_t n = 0;
#pragma unroll 4
            for (uint32_t k = 0; k < a.L; ++k) {
                uint64_t differ = 0;
#pragma unroll
                for (int p = 0; p < P; ++p)
                    differ |= x[((size_t)p * rows + k) * a.T] ^ y[((size_t)p * rows + k) * a.T];
                n += (uint32_t)__popcll(differ);
            }
            atomicAdd(&cnt[r], n);
        }
        // (a counter holds at most n_sites < 2^31 pairs)
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < a.R; i += blockDim.x)
        if (cnt[i]) atomicAdd((unsigned long long *)&a.out[i], (unsigned long long)cnt[i]);
}

// 64 bits from bit s of the periodic row of L bits at `row` (bits past L are 0 in it).
__device__ __forceinline__ uint64_t ring_bits(const uint64_t *row, uint32_t L, uint32_t s) {
    uint64_t out = 0;
    for (uint32_t have = 0; have < 64;) {
        const uint32_t w = s >> 6, b = s & 63u;
        const uint32_t take = min(min(64u - b, L - s), 64u - have);
        const uint64_t piece = (row[w] >> b) & (take == 64 ? ~0ull : (1ull << take) - 1ull);
        out |= piece << have;
        have += take;
        s = s + take < L ? s + take : 0u;
    }
    return out;
}

// The first axis: thread (slot, r) counts displacement r + 1 of the row in that slot.
template <int P>
__global__ void __launch_bounds__(kMeasThreads) pair_row_kernel(PairLines a) {
    extern __shared__ uint64_t s_lines[];  // [slots][P][ext], then R counters
    const uint32_t ext = (a.L + a.R + 63) / 64 + 1;  // words of a row and its beginning again
    uint32_t *cnt = reinterpret_cast<uint32_t *>(s_lines + (size_t)a.slots * P * ext);
    for (uint32_t i = threadIdx.x; i < a.R; i += blockDim.x) cnt[i] = 0;
    const uint64_t last = (a.L & 63u) ? (1ull << (a.L & 63u)) - 1ull : ~0ull;
    for (uint32_t r0 = blockIdx.x * a.slots; r0 < a.outer; r0 += gridDim.x * a.slots) {
        const uint32_t here = min(a.slots, a.outer - r0);
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < here * P * ext; i += blockDim.x) {
            const uint32_t slot = i / (P * ext), p = (i - slot * P * ext) / ext, j = i % ext;
            s_lines[i] = ring_bits(a.words + (size_t)p * a.plane + (size_t)(r0 + slot) * a.wpr, a.L, (64u * j) % a.L);
        }
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < here * a.R; i += blockDim.x) {
            const uint32_t slot = i / a.R, r = i - slot * a.R, sw = (r + 1) >> 6, sb = (r + 1) & 63u;
            const uint64_t *x = s_lines + (size_t)slot * P * ext;
            uint32_t n = 0;
            for (uint32_t j = 0; j < a.wpr; ++j) {
                uint64_t differ = 0;
#pragma unroll
                for (int p = 0; p < P; ++p) {
                    const uint64_t *e = x + p * ext + j;
                    const uint64_t moved = sb ? (e[sw] >> sb) | (e[sw + 1] << (64u - sb)) : e[sw];
                    differ |= e[0] ^ moved;
                }
                if (j + 1 == a.wpr) differ &= last;
                n += (uint32_t)__popcll(differ);
            }
            atomicAdd(&cnt[r], n);
        }
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < a.R; i += blockDim.x)
        if (cnt[i]) atomicAdd((unsigned long long *)&a.out[i], (unsigned long long)cnt[i]);
}

// Product of the L_dir links of each line along dir, summed as +1 / -1.
__global__ void __launch_bounds__(kMeasThreads) polyakov_kernel(const uint8_t *links, Geom g, int dir, long long *out) {
    const uint32_t n = (uint32_t)g.n_sites;
    const uint32_t L = (uint32_t)g.L[dir], st = (uint32_t)g.stride[dir];
    const uint8_t *U = links + (size_t)dir * n;
    long long acc = 0;
    for (uint32_t l = blockIdx.x * blockDim.x + threadIdx.x; l < n / L; l += gridDim.x * blockDim.x) {
        const uint32_t base = (l % st) + (l / st) * st * L;  // the line's site with coordinate 0 along dir
        uint32_t par = 0;
        for (uint32_t k = 0; k < L; ++k) par ^= U[base + k * st];
        acc += 1 - 2 * (long long)(par & 1u);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, off);
    if ((threadIdx.x & 31) == 0 && acc) atomicAdd((unsigned long long *)out, (unsigned long long)acc);
}

// Line parities: bits[mu * n + x] bit k-1 = parity of the k links from x along mu.
__global__ void __launch_bounds__(kMeasThreads) line_bits_kernel(const uint8_t *links, Geom g, int max_len,
                                                                 uint32_t *bits) {
    const uint32_t n = (uint32_t)g.n_sites;
    const uint32_t total = n * (uint32_t)g.d;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
        const int mu = (int)(i / n);
        const uint32_t x = i - (uint32_t)mu * n;
        const uint32_t L = (uint32_t)g.L[mu], st = (uint32_t)g.stride[mu];
        const uint8_t *U = links + (size_t)mu * n;
        uint32_t c = coord_of(g, x, mu), y = x, acc = 0, out = 0;
        for (int k = 0; k < max_len; ++k) {
            acc ^= U[y];
            out |= (acc & 1u) << k;
            if (++c == L) {
                c = 0;
                y -= (L - 1) * st;
            } else {
                y += st;
            }
        }
        bits[i] = out;
    }
}

constexpr int kWilsonMax = 32;

// Counts of -1 rectangles per (r, t) into out[r * (max + 1) + t].
__global__ void __launch_bounds__(kMeasThreads) wilson_kernel(const uint32_t *bits, Geom g, int max_side,
                                                              unsigned long long *out) {
    __shared__ unsigned int cnt[(kWilsonMax + 1) * (kWilsonMax + 1)];
    const int M = max_side + 1;
    for (int i = threadIdx.x; i < M * M; i += blockDim.x) cnt[i] = 0;
    __syncthreads();
    const uint32_t n = (uint32_t)g.n_sites;
    const int d = g.d;
    const int lane = threadIdx.x & 31;
    // every thread of a warp runs the same loop trips (ballots need the whole warp)
    const uint32_t rounds = (n + gridDim.x * blockDim.x - 1) / (gridDim.x * blockDim.x);
    for (uint32_t k = 0; k < rounds; ++k) {
        const uint32_t x = (k * gridDim.x + blockIdx.x) * blockDim.x + threadIdx.x;
        const bool valid = x < n;
        const uint32_t xv = valid ? x : 0;
        for (int mu = 0; mu < d; ++mu)
            for (int nu = 0; nu < d; ++nu) {
                if (mu == nu) continue;
                const uint32_t pm = bits[(size_t)mu * n + xv], pn = bits[(size_t)nu * n + xv];
                const uint32_t cm = coord_of(g, xv, mu), cn = coord_of(g, xv, nu);
                const uint32_t Lm = (uint32_t)g.L[mu], Ln = (uint32_t)g.L[nu];
                const uint32_t sm = (uint32_t)g.stride[mu], sn = (uint32_t)g.stride[nu];
                for (int r = 1; r <= max_side; ++r) {
                    const uint32_t xr = cm + r < Lm ? xv + r * sm : xv - (Lm - r) * sm;  // x + r mu
                    const uint32_t a = bits[(size_t)nu * n + xr];                       // line_nu(x + r mu, .)
                    for (int t = 1; t <= max_side; ++t) {
                        const uint32_t xt = cn + t < Ln ? xv + t * sn : xv - (Ln - t) * sn;  // x + t nu
                        const uint32_t c = bits[(size_t)mu * n + xt];                       // line_mu(x + t nu, .)
                        const uint32_t w = ((pm >> (r - 1)) ^ (a >> (t - 1)) ^ (c >> (r - 1)) ^ (pn >> (t - 1))) & 1u;
                        const unsigned neg = __ballot_sync(0xffffffffu, valid && w);
                        if (lane == 0 && neg) atomicAdd(&cnt[r * M + t], (unsigned)__popc(neg));
                    }
                }
            }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < M * M; i += blockDim.x)
        if (cnt[i]) atomicAdd(&out[i], (unsigned long long)cnt[i]);
}

static unsigned blocks_for(int64_t work) {
    int64_t b = (work + kMeasThreads - 1) / kMeasThreads;
    if (b > 148 * 8) b = 148 * 8;
    return (unsigned)(b < 1 ? 1 : b);
}

int64_t pair_sum_entries(const Geom &g) {
    int64_t e = 0;
    for (int mu = 0; mu < g.d; ++mu) e += g.L[mu] / 2 + 1;
    return e;
}

cudaError_t launch_pair_differ(const uint8_t *cfg, const Geom &g, const int32_t *pair_mu, const int32_t *pair_r,
                               int n_pairs, long long *out, cudaStream_t stream) {
    if (n_pairs == 0) return cudaSuccess;
    cudaError_t e = cudaMemsetAsync(out, 0, sizeof(long long) * (size_t)n_pairs, stream);
    if (e != cudaSuccess) return e;
    const int64_t units = g.L[0] % 4 == 0 ? g.n_sites / 4 : g.n_sites;
    int64_t bx = (units + kMeasThreads - 1) / kMeasThreads;
    const int64_t want = (148 * 16 + n_pairs - 1) / n_pairs;  // about 16 CTAs per SM in all
    if (bx > want) bx = want;
    if (bx < 1) bx = 1;
    pair_differ_kernel<<<dim3((unsigned)bx, (unsigned)n_pairs), kMeasThreads, 0, stream>>>(cfg, g, pair_mu, pair_r,
                                                                                          out);
    return cudaGetLastError();
}

int pair_planes(int q) {
    int p = 1;
    while ((1 << p) < q) ++p;
    return p;
}

constexpr size_t kPairShared = 160 * 1024;

// Shared memory of an axis's kernel; the words (axis > 0) or rows (axis 0) it takes at once: enough
// (displacement, word) pairs for the CTA's threads.
static size_t pair_shared(const Geom &g, int mu, int planes, uint32_t inner, uint32_t &at_once) {
    const uint32_t L = (uint32_t)g.L[mu], R = L / 2;
    at_once = 1;
    if (mu == 0) {
        while (at_once < 64 && at_once * R < 4 * kMeasThreads) at_once *= 2;
        return ((size_t)at_once * planes * ((L + R + 63) / 64 + 1)) * sizeof(uint64_t) + (size_t)R * sizeof(uint32_t);
    }
    while (at_once < 4 || (at_once < inner && at_once * R < kMeasThreads)) at_once *= 2;
    auto bytes = [&]() {
        return (size_t)planes * (L + R) * at_once * sizeof(uint64_t) + (size_t)R * sizeof(uint32_t);
    };
    while (at_once > 1 && bytes() > kPairShared) at_once /= 2;
    return bytes();
}

// Whether the planes are the faster count.  Both sides from 57 shapes at q = 2, 3, 5 (us a call
// beyond the 40 of either): the scan makes 1.5 M pairs a us; the planes take 15 for their
// launches, a chain of steps along each axis past the first (0.014 + 0.0165 a plane a step: a
// thread walks a line) and 1 M words a us with one plane, 0.5 M with three.  Scan / planes:
// 8^4 39 / 52, 64^2 40 / 47, 128^2 44 / 48, 300 x 200 49 / 54, 4 x 4096 86 / 169, 2 x 2048 64 / 115
// (q = 5: 185), 64 x 2048 128 / 123 (184); 80^3 77 / 59, 384^2 76 / 61 (q = 5: 80).
static bool pair_planes_pay(const Geom &g, int planes) {
    const double n = (double)g.n_sites, words = n / g.L[0] * ((g.L[0] + 63) / 64);
    double displacements = 0, steps = 0;
    for (int mu = 0; mu < g.d; ++mu) {
        displacements += g.L[mu] / 2;
        if (mu) steps += g.L[mu];
    }
    return n * displacements / 1.5e6 >
           15 + steps * (0.014 + 0.0165 * planes) + words * displacements * (planes + 1) / 2 / 1e6;
}

size_t pair_words_bytes(const Geom &g, int q) {
    if (q > 8 || g.d < 1 || !pair_planes_pay(g, pair_planes(q))) return 0;
    const int planes = pair_planes(q);
    uint32_t inner = (uint32_t)(g.L[0] + 63) / 64;
    const size_t words = (size_t)(g.n_sites / g.L[0]) * inner;
    for (int mu = 0; mu < g.d; ++mu) {
        uint32_t at_once;
        if (pair_shared(g, mu, planes, inner, at_once) > kPairShared) return 0;  // (an axis too long for shared memory)
        if (mu) inner *= (uint32_t)g.L[mu];
    }
    return words * (size_t)planes * sizeof(uint64_t);
}

template <int P>
static cudaError_t launch_pair_planes(const uint8_t *cfg, const Geom &g, uint64_t *words, long long *out, int sm_count,
                                      cudaStream_t stream) {
    const uint32_t rows = (uint32_t)(g.n_sites / g.L[0]), wpr = (uint32_t)(g.L[0] + 63) / 64;
    pack_planes_kernel<P><<<blocks_for((int64_t)rows * wpr), kMeasThreads, 0, stream>>>(cfg, rows, wpr, (uint32_t)g.L[0], words);
    uint32_t inner = wpr;
    cudaError_t e = cudaGetLastError();
    for (int mu = 0; mu < g.d && e == cudaSuccess; ++mu) {
        PairLines a{};
        a.words = words;
        a.plane = rows * wpr;
        a.L = (uint32_t)g.L[mu];
        a.R = a.L / 2;
        a.out = out;
        out += a.R;
        uint32_t at_once;
        const size_t shared = pair_shared(g, mu, P, inner, at_once);
        const void *kern = mu ? (const void *)pair_axis_kernel<P> : (const void *)pair_row_kernel<P>;
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPairShared);
        if (e != cudaSuccess) break;
        const uint32_t ctas = 8u * (uint32_t)sm_count;
        if (a.R == 0) {
            // (an extent of 1: no displacement)
        } else if (mu == 0) {
            a.wpr = wpr;
            a.slots = at_once;
            a.outer = rows;
            pair_row_kernel<P><<<std::min((rows + at_once - 1) / at_once, ctas), kMeasThreads, shared, stream>>>(a);
        } else {
            a.T = at_once;
            a.inner = inner;
            a.outer = rows * wpr / (inner * a.L);
            const uint32_t tiles = a.outer * ((inner + at_once - 1) / at_once);
            const uint32_t shares = std::max(1u, (a.R * at_once + kMeasThreads - 1) / kMeasThreads);
            // tiles first; the pairs of a tile split over several CTAs where tiles alone are too few
            const uint32_t y = std::min(shares, std::max(1u, (ctas + tiles - 1) / tiles));
            pair_axis_kernel<P><<<dim3(std::min(tiles, ctas), y), kMeasThreads, shared, stream>>>(a);
        }
        if (mu) inner *= a.L;
        e = cudaGetLastError();
    }
    return e;
}

cudaError_t launch_pair_bits(const uint8_t *cfg, const Geom &g, int q, uint64_t *words, int n_pairs, long long *out,
                             int sm_count, cudaStream_t stream) {
    if (n_pairs == 0) return cudaSuccess;
    const cudaError_t e = cudaMemsetAsync(out, 0, sizeof(long long) * (size_t)n_pairs, stream);
    if (e != cudaSuccess) return e;
    switch (pair_planes(q)) {
        case 1: return launch_pair_planes<1>(cfg, g, words, out, sm_count, stream);
        case 2: return launch_pair_planes<2>(cfg, g, words, out, sm_count, stream);
        default: return launch_pair_planes<3>(cfg, g, words, out, sm_count, stream);
    }
}

cudaError_t launch_polyakov(const uint8_t *links, const Geom &g, int dir, long long *out, cudaStream_t stream) {
    cudaError_t e = cudaMemsetAsync(out, 0, sizeof(long long), stream);
    if (e != cudaSuccess) return e;
    polyakov_kernel<<<blocks_for(g.n_sites / g.L[dir]), kMeasThreads, 0, stream>>>(links, g, dir, out);
    return cudaGetLastError();
}

int wilson_max_supported() { return kWilsonMax; }

cudaError_t launch_wilson(const uint8_t *links, const Geom &g, int max_side, uint32_t *bits, unsigned long long *out,
                          cudaStream_t stream) {
    cudaError_t e = cudaMemsetAsync(out, 0, sizeof(unsigned long long) * (size_t)(max_side + 1) * (max_side + 1),
                                    stream);
    if (e != cudaSuccess) return e;
    line_bits_kernel<<<blocks_for(g.n_sites * g.d), kMeasThreads, 0, stream>>>(links, g, max_side, bits);
    wilson_kernel<<<blocks_for(g.n_sites), kMeasThreads, 0, stream>>>(bits, g, max_side, out);
    return cudaGetLastError();
}

}  // namespace plq
