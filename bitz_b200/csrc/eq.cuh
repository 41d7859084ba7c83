// Equality tables eq(r, x) = prod_i (x_i ? r_i : 1 + r_i) over GF(2^128)
// (crates/poly/src/eq.rs:63-98, variable i = index bit i), written in one
// launch: the host forms the factor tables of seven coordinates each and passes
// them as a launch argument.
#pragma once
#include <cuda_runtime.h>

#include "device.cuh"

namespace bz {

constexpr int kMaxPoint = 48;

// out[x] = eq(point, x) for x < 2^n, n <= 35.
void eq_table_device(const f128 *point, int n, f128 *out, cudaStream_t s);
// The same, and the sum of eq(point, x) with[x] into acc (two words, zero
// before), posted as publication pub (then zero again) when it has a counter.
void eq_table_dot(const f128 *point, int n, f128 *out, const f128 *with, unsigned long long *acc,
                  Publish pub, cudaStream_t s);

}  // namespace bz
