#include "eq.cuh"

#include "context.hpp"
#include "passes.cuh"

namespace bz {

// Entry x is the product of factor 0 at the low seven bits and the others at
// theirs; those are the same for 128 entries in a row, so a block forms them
// once per run (two threads of each 256 entries) and makes one product per
// entry: 5 us for 2^13 entries, where the factors by doubling and their product
// took two launches and 11 us. With a second table, the sum of the products
// with it as well.
constexpr int kEqRunsMax = 2 * 8;

template <int NF, bool kDot>
__global__ void __launch_bounds__(kThreads) k_eq(const __grid_constant__ EqFactors<NF> eq, int n,
                                                 int per, f128 *__restrict__ out,
                                                 const f128 *__restrict__ with,
                                                 unsigned long long *acc, Publish pub) {
  __shared__ f128 H[kEqRunsMax];
  const int t = threadIdx.x;
  const size_t total = (size_t)1 << n, step = (size_t)per * kThreads;
  constexpr int kMask = (1 << kFacLog) - 1;
  wide sum = wzero();
  for (size_t base = blockIdx.x * step; base < total; base += gridDim.x * step) {
    if (t < 2 * per) {
      const size_t run = (base >> kFacLog) + t;
      f128 h = NF > 1 ? eq.f[NF > 1 ? 1 : 0][run & kMask] : mk(1, 0);
#pragma unroll 1
      for (int g = 2; g < NF && g * kFacLog < n; g++)
        h = gmul(h, eq.f[g][(run >> ((g - 1) * kFacLog)) & kMask]);
      H[t] = h;
    }
    __syncthreads();
    for (int k = 0; k < per; k++) {
      const size_t x = base + (size_t)k * kThreads + t;
      if (x >= total) break;
      const f128 e = gmul(eq.f[0][x & kMask], H[(k * kThreads + t) >> kFacLog]);
      st(out + x, e);
      if (kDot) wacc(sum, gmul_wide(e, ld(with + x)));
    }
    __syncthreads();  // the runs before the next ones
  }
  if (kDot) {
    const f128 r = greduce(sum);
    uint64_t v[2] = {r.lo, r.hi};
    block_xor_publish<2>(v, acc, pub);
  }
}

template <int NF, bool kDot>
static void launch_eq(const f128 *point, int n, f128 *out, const f128 *with,
                      unsigned long long *acc, Publish pub, cudaStream_t s) {
  EqFactors<NF> eq;
  EqHeap heap;
  for (int g = 0; g < NF; g++) {
    const int have = std::min(kFacLog, std::max(0, n - g * kFacLog));
    heap.build(point + g * kFacLog, have);
    memcpy(eq.f[g], heap.prefix(have), sizeof(f128) << have);
  }
  const size_t total = (size_t)1 << n;
  int per = 1;  // entries per thread: more once every SM has two blocks
  while (per < kEqRunsMax / 2 && total / ((size_t)per * kThreads) >= 4 * kSMs) per *= 2;
  k_eq<NF, kDot><<<grid_for(total, per * kThreads), kThreads, 0, s>>>(eq, n, per, out, with, acc,
                                                                      pub);
  BZ_LAUNCH_CHECK();
}

void eq_table_device(const f128 *point, int n, f128 *out, cudaStream_t s) {
  if (n > 5 * kFacLog) throw CudaError("eq_table_device: point too long");
  (n <= 2 * kFacLog ? launch_eq<2, false> : launch_eq<5, false>)(
      point, n, out, nullptr, nullptr, Publish{nullptr, nullptr, 0}, s);
}

void eq_table_dot(const f128 *point, int n, f128 *out, const f128 *with, unsigned long long *acc,
                  Publish pub, cudaStream_t s) {
  if (n > 5 * kFacLog) throw CudaError("eq_table_dot: point too long");
  (n <= 2 * kFacLog ? launch_eq<2, true> : launch_eq<5, true>)(point, n, out, with, acc, pub, s);
}

// Every kernel of this file, loaded when the process's first lane on a device
// is made (lane_bootstrap, context.cpp).
void preload_eq_kernels() {
  load_kernels({(const void *)k_eq<2, false>,
                (const void *)k_eq<2, true>,
                (const void *)k_eq<5, false>,
                (const void *)k_eq<5, true>});
}

}  // namespace bz
