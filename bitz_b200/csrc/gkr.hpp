// Host interface of the grand-product GKR kernels.
#pragma once
#include <cuda_runtime.h>

#include "device.cuh"
#include "status.hpp"
#include "transcript.hpp"

namespace bz {

struct GkrScratch {
  size_t capacity = 0;         // leaves the layers are sized for: 2^(7+s)
  f128 *layer[8] = {nullptr};  // layer j >= 2 holds 2^(7+s-j) nodes; layer 7 is the output
  f128 *bound = nullptr;       // 2^(s+1): layers 0 and 1 once their rows are bound
  unsigned long long *gram = nullptr;  // gkr_gram_words() words
  f128 *mid = nullptr;                 // 2304 entries
  f128 *eq_low = nullptr;              // 2^14 entries
  unsigned long long *acc = nullptr;  // a pass's sums: 56 words
  RoundChannel *channel = nullptr;    // carries the passes' sums and the last tables
  // Columns at or beyond live_cols hold no set bit (the padding of h), so
  // every node of theirs is one in every layer; the kernels skip their
  // products and add their known contribution. 0: every column is live.
  size_t live_cols = 0;
};

size_t gkr_gram_words();

// Builds layers 2 to 7 from the packed columns (2^s F128, bit b of column c is
// row b) and the 128 row images. Layer 7 holds the column products.
void gkr_build(const f128 *cols, int s, const f128 *images, GkrScratch &sc, cudaStream_t st);

// The seven layer sumchecks from the output point zeta (s coordinates) to the
// leaves: writes 7 + s coordinates and returns the claim on the leaves. The
// layer tables are consumed (bound in place); columns and images as in
// gkr_build.
f128 gkr_prove(const f128 *cols, int s, const f128 *images, const f128 *zeta, uint32_t grind_bits,
               Transcript &ts, GkrScratch &sc, cudaStream_t st, f128 *point_out);

}  // namespace bz
