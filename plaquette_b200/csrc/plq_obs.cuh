// plq_obs.cuh -- a configuration's integer primaries site by site (plq_obs.cu,
// plq_resident.cu).
#pragma once
#include <cuda_runtime.h>

#include "../../include/plaquette.h"
#include "plq_device.cuh"

namespace plq {

__device__ __forceinline__ long long warp_sum(long long v) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
    return v;
}

// One site's (or, gauge, one site's plaquettes') contribution to the
// primaries: acc0 the bond / agreement / plaquette sum, acc1 the Ising spin
// sum; Potts labels counted in the block's shared counters.
template <int D>
__device__ __forceinline__ void site_primaries(const uint8_t *state, const Geom &g, int model, int64_t s,
                                               long long &acc0, long long &acc1, int *s_counts) {
    const int64_t n = g.n_sites;
    int32_t x[D];
    uint32_t t = (uint32_t)s;
#pragma unroll
    for (int mu = 0; mu < D; ++mu) {
        uint32_t qq = fdiv(t, g.dm[mu], g.dl[mu]);
        x[mu] = (int32_t)(t - qq * (uint32_t)g.L[mu]);
        t = qq;
    }
    if (model == PLQ_GAUGE) {
        // plaquettes (s, mu, nu), mu < nu: U_mu(s) U_nu(s+mu) U_mu(s+nu) U_nu(s)
#pragma unroll
        for (int mu = 0; mu < D; ++mu) {
            int64_t s_mu = x[mu] + 1 < g.L[mu] ? s + g.stride[mu] : s - (int64_t)(g.L[mu] - 1) * g.stride[mu];
#pragma unroll
            for (int nu = mu + 1; nu < D; ++nu) {
                int64_t s_nu = x[nu] + 1 < g.L[nu] ? s + g.stride[nu] : s - (int64_t)(g.L[nu] - 1) * g.stride[nu];
                int b = state[mu * n + s] ^ state[nu * n + s_mu] ^ state[mu * n + s_nu] ^ state[nu * n + s];
                acc0 += 1 - 2 * b;
            }
        }
    } else {
        int si = state[s];
        if (model == PLQ_ISING) acc1 += 1 - 2 * si;
        else atomicAdd(&s_counts[si], 1);
#pragma unroll
        for (int mu = 0; mu < D; ++mu) {
            int64_t s_mu = x[mu] + 1 < g.L[mu] ? s + g.stride[mu] : s - (int64_t)(g.L[mu] - 1) * g.stride[mu];
            int sj = state[s_mu];
            if (model == PLQ_ISING) acc0 += (1 - 2 * si) * (1 - 2 * sj);
            else acc0 += si == sj;
        }
    }
}

// The block's partial sums into out (one 64-bit atomic per warp; the Potts
// label counters after a barrier).
__device__ __forceinline__ void flush_primaries(long long acc0, long long acc1, int model, int q, int *s_counts,
                                                long long *out) {
    acc0 = warp_sum(acc0);
    acc1 = warp_sum(acc1);
    if ((threadIdx.x & 31) == 0) {
        if (acc0) atomicAdd((unsigned long long *)&out[0], (unsigned long long)acc0);
        if (model == PLQ_ISING && acc1) atomicAdd((unsigned long long *)&out[1], (unsigned long long)acc1);
    }
    if (model == PLQ_POTTS) {
        __syncthreads();
        for (int i = threadIdx.x; i < q; i += blockDim.x)
            if (s_counts[i]) atomicAdd((unsigned long long *)&out[1 + i], (unsigned long long)s_counts[i]);
    }
}

}  // namespace plq
