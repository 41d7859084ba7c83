// Host interface of the post-GKR sumcheck kernels.
#pragma once
#include <cuda_runtime.h>

#include <string>

#include "device.cuh"
#include "passes.cuh"
#include "status.hpp"
#include "transcript.hpp"

namespace bz {

struct PostGkrArgs {
  const f128 *rows;  // device, 2^log_rows weights
  int log_rows;      // t >= 7
  const f128 *cols;  // device, 2^log_cols weights
  int log_cols;      // s
  const f128 *packed;  // device, 2^(t+s-7) committed words
  f128 target;
  uint32_t grind_bits;
};

// Device scratch, reusable across proofs: four tables of `capacity` entries,
// the passes' sums, and where they are posted: the lane's channel, or (without
// one) tagged slots in device memory that the host copies and waits for.
struct PostGkrScratch {
  size_t capacity = 0;
  f128 *w0 = nullptr, *v0 = nullptr, *w1 = nullptr, *v1 = nullptr;
  unsigned long long *acc = nullptr;  // 130 words
  f128 claim_seen{0, 0};              // the weighted sum found when a claim fails
  RoundChannel *channel = nullptr;
  unsigned int *counter = nullptr;         // without a channel
  unsigned long long *handover = nullptr;  // 2 kHandoverWords slots
  // the last publication in those slots, kept between calls: a tag is not used
  // again while the words of an earlier call may still be there
  unsigned long long *seq = nullptr;
};

// The quadratic sumcheck of <W, V> (shared with the Ligerito folds), low
// coordinate first. quad_pass binds both tables at b's challenges (into w2 and
// v2, when there are any), n entries each after that, and posts the 3^k point
// sums of the next k rounds (it returns how many blocks post sums of their own,
// to be added up); quad_bind only binds (v may be null).
int quad_pass(int k, const f128 *w, const f128 *v, f128 *w2, f128 *v2, size_t n,
               const PassBind &b, const PassPost &post, cudaStream_t s);
void quad_bind(const f128 *w, const f128 *v, f128 *w2, f128 *v2, size_t n, const PassBind &b,
               cudaStream_t s);

// Runs the whole reduction: writes t+s challenges to point_out and the
// closing evaluation to value_out, appending every message to `ts`.
int post_gkr_prove(const PostGkrArgs &a, Transcript &ts, PostGkrScratch &sc, cudaStream_t s,
                   f128 *point_out, f128 *value_out);

// The same reduction on fixed file-scope device scratch: allocates nothing.
// Claims up to 2^20 bits; see post_gkr_noalloc.cu for the sharing rules.
int post_gkr_prove_noalloc(const PostGkrArgs &a, Transcript &ts, cudaStream_t s, f128 *point_out,
                           f128 *value_out, std::string &err);
// The tag of that call's last publication on the device (for tests).
unsigned long long noalloc_last_publication(int device);

}  // namespace bz
