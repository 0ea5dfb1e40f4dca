// plq_second_draws.h -- which labels of a Swendsen-Wang sweep on the PCG stream
// take a second draw (plq_cluster.cu), apart so that it can be checked on the host.
//
// rand's range sampler looks at the output of a draw and takes another for about
// one output in 2^32 / (range - 1), none where the range is a power of two.  The
// rank pass draws label r from place r of the stream behind the bonds and lists the
// places whose outputs ask for a second draw.  In order, a listed place is the first
// draw of the label that the second draws before it have moved there, unless the
// label before took it as its second; and n second draws move the last n labels to
// places the rank pass did not reach, which are looked at here.
#pragma once
#include <cstdint>

#if defined(__CUDACC__)
#define PLQ_SECOND_HD __host__ __device__
#else
#define PLQ_SECOND_HD
#endif

namespace plq {

// place[0 .. listed): the listed places, in any order (sorted here).  second(p) is asked for
// p = labels, labels + 1, ... in turn.  rank[0 .. n): the ranks of the labels with two draws, in
// order; false if there are more than cap.
template <class Second>
PLQ_SECOND_HD inline bool resolve_second_draws(int32_t *place, int listed, int64_t labels, int cap, int32_t *rank, int &n,
                                               Second second) {
    n = 0;
    if (listed > cap) return false;
    for (int i = 1; i < listed; ++i) {
        const int32_t p = place[i];
        int k = i;
        for (; k > 0 && place[k - 1] > p; --k) place[k] = place[k - 1];
        place[k] = p;
    }
    int64_t taken = -1;  // the place of the last label's second draw
    for (int i = 0; i < listed; ++i) {
        if (place[i] == taken) continue;
        rank[n] = place[i] - n;
        ++n;
        taken = (int64_t)place[i] + 1;
    }
    for (int64_t p = labels; p - n < labels; ++p) {
        if (!second(p) || p == taken) continue;
        if (n == cap) return false;
        rank[n] = (int32_t)(p - n);
        ++n;
        taken = p + 1;
    }
    return true;
}

}  // namespace plq
