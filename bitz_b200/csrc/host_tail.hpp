// The host's rounds on a sumcheck's last GF(2^128) tables: binds and sums four
// elements at a time with VPCLMULQDQ on 512-bit registers (about 1 ns per
// product, against 6 with the 128-bit instruction), one at a time on hosts
// without it or with BITZ_HOST_SIMD=0.
#pragma once
#include <stddef.h>

#include "field.cuh"

namespace bz {

// t[x] += r (t[x] + t[x + h]) for x < h.
void host_bind_high(f128 *t, size_t h, f128 r);
// t[o] = t[2o] + r (t[2o] + t[2o + 1]) for o < n, in place.
void host_bind_low(f128 *t, size_t n, f128 r);
// out[k] = r t[k] for k < n.
void host_scale(const f128 *t, f128 r, size_t n, f128 *out);
// A GKR round over tables of 2h entries, weights e[0, h): out[0] the sum of
// e L R over the lower halves (the upper ones with `one`), out[1] that of
// e (L0 + L1) (R0 + R1).
void host_cubic_sums(const f128 *e, const f128 *L, const f128 *R, size_t h, bool one, f128 out[2]);
// A quadratic round over pairs (2j, 2j + 1), j < n: out[0] the sum of
// W[2j] V[2j], out[1] that of (W[2j] + W[2j + 1]) (V[2j] + V[2j + 1]).
void host_quad_sums(const f128 *W, const f128 *V, size_t n, f128 out[2]);

}  // namespace bz
