// plq_items.cuh -- the bodies of one work item (a chunk of one colour pass of
// one lattice) of the persistent kernels: the batched ensembles
// (plq_ensemble.cu) and the resident single lattices (plq_resident.cu).
#pragma once
#include <cuda_runtime.h>

#include "../../include/plaquette.h"
#include "plq_device.cuh"
#include "plq_local_impl.cuh"
#include "plq_packed.cuh"
#include "plq_words.cuh"

namespace plq {

template <int D>
__device__ void run_words(const LocalArgs &a, int link, int64_t chunk, int R) {
    const bool st = a.jump != nullptr;
    if (link) {
        if (D >= 2) {
            if (st) link_words_chunk<D, true>(a, chunk, R);
            else link_words_chunk<D, false>(a, chunk, R);
        }
    } else if (a.q == 3) {
        if (st) site_words_chunk<D, 3, true>(a, chunk, R);
        else site_words_chunk<D, 3, false>(a, chunk, R);
    } else if (a.q == 4) {
        if (st) site_words_chunk<D, 4, true>(a, chunk, R);
        else site_words_chunk<D, 4, false>(a, chunk, R);
    } else {
        if (st) site_words_chunk<D, 2, true>(a, chunk, R);
        else site_words_chunk<D, 2, false>(a, chunk, R);
    }
}

// Keyed sites in bytes, one colour site at a time: any q, any even extents (the
// lattices whose rows the four-site words do not fit, and every Potts Metropolis
// chain).  The same keys, draws and tables as plq_local_impl.cuh; that body's
// eight ranks a thread, 64-bit keys and unused packing weights left the pass at two
// CTAs per SM: q = 5 Metropolis on 1002 x 750, 20.6 us a sweep, 10.1 so.
template <int D>
__device__ __forceinline__ void rank_site(const LocalArgs &p, uint32_t r, uint32_t mix) {
    const uint32_t q = (uint32_t)p.q;
    const bool metropolis = p.kernel == PLQ_METROPOLIS;
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

// One chunk of a colour pass: blockDim.x * R ranks, a thread's blockDim.x apart.
template <int D, int R>
__device__ __forceinline__ void rank_chunk(const LocalArgs &a, int64_t chunk) {
    const uint32_t half = (uint32_t)(a.g.n_sites / 2), mix = keyed_mix(a.sweep32);
    const uint32_t r0 = (uint32_t)(chunk * (int64_t)blockDim.x * R) + threadIdx.x;
#pragma unroll 1
    for (int i = 0; i < R; ++i) {
        const uint32_t r = r0 + (uint32_t)i * blockDim.x;
        if (r < half) rank_site<D>(a, r, mix);
    }
}

// WORDS_ONLY: every member runs four sites at a time, packed, or as keyed sites one
// at a time, so the generic body is compiled out (far fewer registers, more CTAs
// per SM).
template <int R, bool WORDS_ONLY>
__device__ void run_item(const LocalArgs &a, int d, int link, int64_t chunk, int wpt) {
    if (a.words) {
        switch (d) {
            case 1: run_words<1>(a, link, chunk, wpt); break;
            case 2: run_words<2>(a, link, chunk, wpt); break;
            case 3: run_words<3>(a, link, chunk, wpt); break;
            case 4: run_words<4>(a, link, chunk, wpt); break;
            default: break;
        }
        return;
    }
    if (!link && !a.jump) {
        switch (d) {
            case 1: rank_chunk<1, R>(a, chunk); break;
            case 2: rank_chunk<2, R>(a, chunk); break;
            case 3: rank_chunk<3, R>(a, chunk); break;
            case 4: rank_chunk<4, R>(a, chunk); break;
            default: break;
        }
        return;
    }
    if (WORDS_ONLY) return;
    if (link) {
        switch (d) {
            case 2: local_chunk<2, true, false, R>(a, chunk); break;
            case 3: local_chunk<3, true, false, R>(a, chunk); break;
            case 4: local_chunk<4, true, false, R>(a, chunk); break;
            default: break;
        }
    } else {
        switch (d) {
            case 1: local_chunk<1, false, false, R>(a, chunk); break;
            case 2: local_chunk<2, false, false, R>(a, chunk); break;
            case 3: local_chunk<3, false, false, R>(a, chunk); break;
            case 4: local_chunk<4, false, false, R>(a, chunk); break;
            default: break;
        }
    }
}

// ---- Z2 gauge members with L0 <= 32 on the keyed stream: links bit-packed by rows.
// Inside a persistent launch such a member's links live in pk: word dir * rows + r
// holds bit x = U_dir(x, r) for row r (the site index over directions >= 1).  A
// work item takes rows of one (direction mu, parity) pass: the six staples of
// every link of a row come out of XORs of whole row words (a shift along
// direction 0 is a rotation of the row, along the others another row), their
// count of unsatisfied staples out of a bit-sliced counter, and each link of
// the pass's parity then decides exactly as the byte body does -- the same key
// cur + 4(d-1) - 2 * unsatisfied, the same keyed draw of variable site * d + mu,
// the same table -- so results are bit-identical.  The launch packs the bytes
// first and unpacks them at its end (pack_links_kernel).

// Rows of a lattice (sites over directions >= 1): L1 * L2 * ... (extents past
// d are 1), by multiplication.
__host__ __device__ __forceinline__ uint32_t row_count(const Geom &g) {
    uint32_t n = 1;
#pragma unroll
    for (int k = 1; k < kMaxD; ++k) n *= (uint32_t)g.L[k];
    return n;
}

// Row r's coordinates along directions 1..D-1: their parity and the row
// offsets to the +k / -k neighbour rows (periodic).  The row stride of
// direction k is L1 * ... * L(k-1).
template <int D>
__device__ __forceinline__ int row_geometry(const Geom &g, uint32_t r, int32_t *op, int32_t *om) {
    uint32_t rr = r;
    int par = 0;
    int32_t rs = 1;
#pragma unroll
    for (int k = 1; k < D; ++k) {
        const uint32_t q = fdiv(rr, g.dm[k], g.dl[k]);
        const int32_t c = (int32_t)(rr - q * (uint32_t)g.L[k]);
        rr = q;
        par += c;
        op[k] = c + 1 < g.L[k] ? rs : -(g.L[k] - 1) * rs;
        om[k] = c > 0 ? -rs : (g.L[k] - 1) * rs;
        rs *= g.L[k];
    }
    return par;
}

// q = 2 sites (Ising, or Potts at q = 2) packed by rows: the per-site count of
// neighbours in state 1 comes out of the bit-sliced counter over the 2d
// neighbour rows (d <= 3: at most 6), key cur + 2 * count as the byte body's.
template <int D, class W>
__device__ void packed_site_item(const LocalArgs &a, W *pk, int64_t chunk, int R, const uint2 *tab) {
    const uint32_t L0 = (uint32_t)a.g.L[0];
    const uint32_t rows = row_count(a.g);
    const W full = L0 == 8 * sizeof(W) ? ~(W)0 : (((W)1 << L0) - 1);
    const uint32_t r0 = (uint32_t)(chunk * (int64_t)blockDim.x * R) + threadIdx.x * (uint32_t)R;
    const bool hb = a.kernel == PLQ_HEATBATH;
    const uint32_t sweep_mix = keyed_mix(a.sweep32);
#pragma unroll 1
    for (int i = 0; i < R; ++i) {
        const uint32_t r = r0 + (uint32_t)i;
        if (r >= rows) break;
        int32_t op[4] = {0, 0, 0, 0}, om[4] = {0, 0, 0, 0};
        const int par = row_geometry<D>(a.g, r, op, om);
        const W C = pk[r];
        W c0 = 0, c1 = 0, c2 = 0;
        count_add(c0, c1, c2, row_xp(C, L0, full));
        count_add(c0, c1, c2, row_xm(C, L0, full));
#pragma unroll
        for (int k = 1; k < D; ++k) {
            count_add(c0, c1, c2, pk[r + (uint32_t)op[k]]);
            count_add(c0, c1, c2, pk[r + (uint32_t)om[k]]);
        }
        const uint32_t x0 = (uint32_t)((a.color ^ par) & 1);
        const int n = (int)(L0 / 2);
        const uint32_t v0 = r * L0 + x0;  // the keyed stream's index of the row's first variable
        const W flip = hb ? decide_row<W, 2, true>(C >> x0, c0 >> x0, c1 >> x0, c2 >> x0, n, v0, a.seed32, sweep_mix, tab)
                          : decide_row<W, 2, false>(C >> x0, c0 >> x0, c1 >> x0, c2 >> x0, n, v0, a.seed32, sweep_mix, tab);
        pk[r] = C ^ (flip << x0);
    }
}

// Energy integer of packed rows [c * blockDim, (c + 1) * blockDim), one row per
// thread: sites -- the bond sum (Ising) or agreement count (Potts) over the
// +mu bonds; links -- the plaquette sum over mu < nu (as energy_chunk).
template <int D, class W>
__device__ long long packed_energy_rows(const LocalArgs &a, const W *pk, int link, int64_t c) {
    const uint32_t L0 = (uint32_t)a.g.L[0];
    const uint32_t rows = row_count(a.g);
    const W full = L0 == 8 * sizeof(W) ? ~(W)0 : (((W)1 << L0) - 1);
    const uint32_t r = (uint32_t)(c * (int64_t)blockDim.x) + threadIdx.x;
    if (r >= rows) return 0;
    int32_t op[4] = {0, 0, 0, 0}, om[4] = {0, 0, 0, 0};
    row_geometry<D>(a.g, r, op, om);
    long long acc = 0;
    if (!link) {
        const W C = pk[r];
        int diff = popc_w((C ^ row_xp(C, L0, full)) & full);
        long long pairs = L0;
#pragma unroll
        for (int k = 1; k < D; ++k) {
            diff += popc_w(C ^ pk[r + (uint32_t)op[k]]);
            pairs += L0;
        }
        acc = a.model == PLQ_ISING ? pairs - 2ll * diff : pairs - diff;
    } else {
#pragma unroll
        for (int mu = 0; mu < D; ++mu) {
#pragma unroll
            for (int nu = mu + 1; nu < D; ++nu) {
                const W *Pmu = pk + (uint32_t)mu * rows, *Pnu = pk + (uint32_t)nu * rows;
                const W umu = Pmu[r], unu = Pnu[r];
                // U_nu(s + mu): mu = 0 a rotation of the row, else the +mu row
                const W nu_smu = mu == 0 ? row_xp(unu, L0, full) : Pnu[r + (uint32_t)op[mu]];
                const W mu_snu = Pmu[r + (uint32_t)op[nu]];  // nu >= 1
                acc += (long long)L0 - 2ll * popc_w(umu ^ nu_smu ^ mu_snu ^ unu);
            }
        }
    }
    return acc;
}

// Row r of direction MU's links (op, om: row_geometry's offsets): its bits and,
// bit-sliced, the satisfied staples of every link.  MU is a compile-time
// constant, so the staple terms that are row rotations and those that are other
// rows are fixed per variant.  Rows are at most one word long.
template <int D, int MU, class W>
__device__ __forceinline__ void link_row(uint32_t L0, uint32_t rows, const W *pk, uint32_t r, const int32_t *op,
                                         const int32_t *om, W &Umu, W &c0, W &c1, W &c2) {
    constexpr int mu = MU;
    const W full = L0 == 8 * sizeof(W) ? ~(W)0 : (((W)1 << L0) - 1);
    const int32_t op_mu = mu > 0 ? op[mu] : 0;
    Umu = pk[(uint32_t)mu * rows + r];
    c0 = c1 = c2 = 0;
#pragma unroll
    for (int nu = 0; nu < D; ++nu) {
        if (nu == mu) continue;
        const W *Pnu = pk + (uint32_t)nu * rows;
        const W *Pmu = pk + (uint32_t)mu * rows;
        // forward: U_nu(s+mu) U_mu(s+nu) U_nu(s)
        const W nu_s = Pnu[r];
        const W nu_smu = mu == 0 ? row_xp(nu_s, L0, full) : Pnu[r + (uint32_t)op_mu];
        const W mu_snu = nu == 0 ? row_xp(Umu, L0, full) : Pmu[r + (uint32_t)op[nu]];
        count_add(c0, c1, c2, (W) ~(nu_smu ^ mu_snu ^ nu_s));
        // backward: U_nu(s+mu-nu) U_mu(s-nu) U_nu(s-nu)
        W nu_smn, mu_smn, nu_smumn;
        if (nu == 0) {
            nu_smn = row_xm(nu_s, L0, full);
            mu_smn = row_xm(Umu, L0, full);
            nu_smumn = row_xm(nu_smu, L0, full);
        } else {
            nu_smn = Pnu[r + (uint32_t)om[nu]];
            mu_smn = Pmu[r + (uint32_t)om[nu]];
            nu_smumn = mu == 0 ? row_xp(nu_smn, L0, full) : Pnu[r + (uint32_t)op_mu + (uint32_t)om[nu]];
        }
        count_add(c0, c1, c2, (W) ~(nu_smumn ^ mu_smn ^ nu_smn));
    }
}

template <int D, int MU, class W = uint32_t>
__device__ void packed_link_item(const LocalArgs &a, W *pk, int64_t chunk, int R, const uint2 *tab) {
    const uint32_t L0 = (uint32_t)a.g.L[0];
    const uint32_t rows = row_count(a.g);
    const uint32_t r0 = (uint32_t)(chunk * (int64_t)blockDim.x * R) + threadIdx.x * (uint32_t)R;
    const bool hb = a.kernel == PLQ_HEATBATH;
    const uint32_t sweep_mix = keyed_mix(a.sweep32);
#pragma unroll 1
    for (int i = 0; i < R; ++i) {
        const uint32_t r = r0 + (uint32_t)i;
        if (r >= rows) break;
        int32_t op[4] = {0, 0, 0, 0}, om[4] = {0, 0, 0, 0};
        const int par = row_geometry<D>(a.g, r, op, om);
        W Umu, c0, c1, c2;
        link_row<D, MU, W>(L0, rows, pk, r, op, om, Umu, c0, c1, c2);
        // the links of the pass's parity: x with (x + par) % 2 == colour; the byte body's key
        // cur + 4(d-1) - 2 * unsatisfied is cur + 2 * satisfied
        const uint32_t x0 = (uint32_t)((a.color ^ par) & 1);
        const int n = (int)(L0 / 2);
        const uint32_t v0 = (r * L0 + x0) * (uint32_t)D + (uint32_t)MU;  // keyed index of link (x0, r, mu)
        const W flip = hb ? decide_row<W, 2 * D, true>(Umu >> x0, c0 >> x0, c1 >> x0, c2 >> x0, n, v0, a.seed32,
                                                       sweep_mix, tab)
                          : decide_row<W, 2 * D, false>(Umu >> x0, c0 >> x0, c1 >> x0, c2 >> x0, n, v0, a.seed32,
                                                        sweep_mix, tab);
        pk[(uint32_t)MU * rows + r] = Umu ^ (flip << x0);
    }
}

}  // namespace plq
