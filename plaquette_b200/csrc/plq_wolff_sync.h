// plq_wolff_sync.h -- the decision every CTA of a Wolff launch takes about a
// called update (plq_cluster.cu's wolff_kernel), apart so that the protocol can
// be explored on the host.
#pragma once

#if defined(__CUDACC__)
#define PLQ_WOLFF_HD __host__ __device__
#else
#define PLQ_WOLFF_HD
#endif

namespace plq {

// Whether update `id` ended with its growth, from the word its parity shares:
// the last called update of that parity whose cluster the growth found whole.
// Nothing holds the growing CTA until every other one has read the word: behind
// the barrier it may end update id + 1 uncalled and mark id + 2 in the same word
// first.  A later update there means that `id` ended with its growth too, for one
// that needs the decomposition has two more barriers, which every CTA joins
// only after this read.
PLQ_WOLFF_HD inline bool wolff_ended_by_growth(unsigned long long word, unsigned long long id) { return word >= id; }

}  // namespace plq
