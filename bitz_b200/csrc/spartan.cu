// Spartan's outer and inner sumchecks and the matrix bind over the
// transcript-drawn prime (crates/spartan/src/piop.rs:67-113,
// sumcheck.rs:252-553, matrix.rs:336-467).
//
// Tables hold Montgomery residues. Both sumchecks bind their lowest coordinate
// first and go through the device in passes of up to three rounds (passes.cuh):
// a pass posts the summed polynomial's values at the points {0, 1, infinity}^K
// (infinity: the coefficient of X^2, from the differences of the halves) and
// the host runs K rounds from them. The outer polynomial is
// eq(tau) (A B - C); eq is a product over the coordinates, so the passes sum
// only A B - C, weighted by eq over the coordinates above, and the host
// multiplies the round's own linear factor in. The inner one is D W with W the
// packed bits of h: its first three rounds need 64 sums of D by position and
// bit position within groups of eight, and W after their binds is a 256-entry
// table of the group's byte.
#include "device.cuh"
#include "context.hpp"
#include "passes.cuh"
#include "spartan.hpp"

#include <chrono>
#include <cstdio>

namespace bz {

// eq over n coordinates (Montgomery) in one launch, as eq.cu's: the factors of
// seven coordinates come from the host, a run of 128 entries shares the product
// of the upper ones.
struct FpEqFactors {
  fp f[5][1 << kFacLog];
};

__global__ void __launch_bounds__(kThreads) k_fp_eq(const __grid_constant__ FpEqFactors eq, int n,
                                                    int per, FpCtx c, fp *__restrict__ out) {
  __shared__ fp H[16];
  const int t = threadIdx.x;
  const size_t total = (size_t)1 << n, step = (size_t)per * kThreads;
  constexpr int kMask = (1 << kFacLog) - 1;
  for (size_t base = blockIdx.x * step; base < total; base += gridDim.x * step) {
    if (t < 2 * per) {
      const size_t run = (base >> kFacLog) + t;
      fp h = eq.f[1][run & kMask];
#pragma unroll 1
      for (int g = 2; g * kFacLog < n; g++)
        h = fp_mul(h, eq.f[g][(run >> ((g - 1) * kFacLog)) & kMask], c);
      H[t] = h;
    }
    __syncthreads();
    for (int k = 0; k < per; k++) {
      const size_t x = base + (size_t)k * kThreads + t;
      if (x >= total) break;
      out[x] = fp_mul(eq.f[0][x & kMask], H[(k * kThreads + t) >> kFacLog], c);
    }
    __syncthreads();  // the runs before the next ones
  }
}

// eq over a run of coordinates, coordinate 0 in the lowest bit.
static std::vector<fp> sp_eq(const fp *z, int n, const FpCtx &c, fp scale) {
  std::vector<fp> e{scale};
  e.reserve((size_t)1 << n);
  for (int i = 0; i < n; i++) {
    const size_t h = e.size();
    e.resize(2 * h);
    for (size_t k = 0; k < h; k++) {
      const fp one = fp_mul(e[k], z[i], c);
      e[k + h] = one;
      e[k] = fp_sub(e[k], one, c);
    }
  }
  return e;
}

void fp_eq_table(const fp *point, int n, const FpCtx &c, fp *out, cudaStream_t s) {
  if (n > 5 * kFacLog) throw CudaError("fp_eq_table: point too long");
  FpEqFactors f{};
  for (int g = 0; g < 5; g++) {
    const std::vector<fp> e = sp_eq(point + g * kFacLog, std::min(kFacLog, std::max(0, n - g * kFacLog)),
                                    c, c.one);
    std::copy(e.begin(), e.end(), f.f[g]);
  }
  const size_t total = (size_t)1 << n;
  int per = 1;
  while (per < 8 && total / ((size_t)per * kThreads) >= 4 * kSMs) per *= 2;
  k_fp_eq<<<grid_for(total, per * kThreads), kThreads, 0, s>>>(f, n, per, c, out);
  BZ_LAUNCH_CHECK();
}

__device__ __forceinline__ fp fp_from_i64(int64_t v, const FpCtx &c) {
  fp x;
  if (v >= 0) {
    x = fp{(uint64_t)v, 0};
  } else {
    uint64_t m = (uint64_t)(-(v + 1)) + 1;  // |v|, which is below q
    x.lo = c.q0 - m;
    x.hi = c.q1 - (c.q0 < m);
  }
  return fp_mul(x, c.r2, c);
}

// build_product_mles (matrix.rs:336-370): A h, B h, C h mod q, zero padded.
__global__ void k_products_to_fp(const int64_t *__restrict__ prod, size_t rows, size_t padded,
                                 FpCtx c, fp *__restrict__ A, fp *__restrict__ B,
                                 fp *__restrict__ C) {
  for (size_t r = blockIdx.x * (size_t)blockDim.x + threadIdx.x; r < padded;
       r += (size_t)gridDim.x * blockDim.x) {
    if (r < rows) {
      A[r] = fp_from_i64(prod[r], c);
      B[r] = fp_from_i64(prod[rows + r], c);
      C[r] = fp_from_i64(prod[2 * rows + r], c);
    } else {
      A[r] = B[r] = C[r] = fp_zero();
    }
  }
}

BZ_HD fp interp(fp a, fp b, fp r, const FpCtx &c) {
  return fp_add(a, fp_mul(r, fp_sub(b, a, c), c), c);
}

// One block adds the per-block partials into out.
__global__ void k_fp_finalize(const fp *partial, int nblocks, FpCtx c, fp *out) {
  fp acc[1] = {fp_zero()};
  for (int b = threadIdx.x; b < nblocks; b += blockDim.x) acc[0] = fp_add(acc[0], partial[b], c);
  block_fp_sum<1>(acc, c, out);
}

// The coefficient table of the bind: scale_k * coefficient for every distinct
// (matrix, coefficient) pair.
__global__ void k_bind_table(const int64_t *__restrict__ vals, const uint8_t *__restrict__ which,
                             int n, fp rho, fp rho2, FpCtx c, fp *tab) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  fp v = fp_from_i64(vals[i], c);
  fp s = which[i] == 0 ? c.one : which[i] == 1 ? rho : rho2;
  tab[i] = fp_mul(v, s, c);
}

// bind_and_batch (matrix.rs:429-467) as a gather over the column-major copy of
// A, B and C: D(y) = sum over column y's entries of eq(r_x, row) * table[idx].
// Column 0 (the constant) has an entry per round constant and bit constraint,
// so the launch's last `col0_blocks` blocks share it out, and with it the
// statement-dependent part of C there: the bit constraints whose expected value
// is one put rho^2 eq(r_x, row) there (each thread scales its share of those
// rows, which sums to the same total mod q). The last of them to finish adds
// the blocks' sums up.
__global__ void __launch_bounds__(kThreads) k_bind(
    const uint32_t *__restrict__ off, const uint32_t *__restrict__ row,
    const uint16_t *__restrict__ idx, const fp *__restrict__ tab, const fp *__restrict__ eq,
    size_t cols, size_t padded, const uint32_t *__restrict__ bit_rows, int n_bits, fp rho2,
    int col0_blocks, FpCtx c, fp *partial, unsigned int *counter, fp *D) {
  const int blocks = gridDim.x - col0_blocks;
  if ((int)blockIdx.x < blocks) {
    for (size_t y = blockIdx.x * (size_t)blockDim.x + threadIdx.x; y < padded;
         y += (size_t)blocks * blockDim.x) {
      if (y == 0) continue;
      fp acc = fp_zero();
      if (y < cols)
        for (uint32_t e = off[y]; e < off[y + 1]; e++)
          acc = fp_add(acc, fp_mul(eq[row[e]], tab[idx[e]], c), c);
      D[y] = acc;
    }
    return;
  }
  __shared__ bool last;
  __shared__ fp total[1];
  const int b = blockIdx.x - blocks, stride = col0_blocks * kThreads;
  const uint32_t n = off[1];
  fp acc[1] = {fp_zero()};
  for (uint32_t e = b * kThreads + threadIdx.x; e < n; e += stride)
    acc[0] = fp_add(acc[0], fp_mul(eq[row[e]], tab[idx[e]], c), c);
  fp bits = fp_zero();
  for (int i = b * kThreads + threadIdx.x; i < n_bits; i += stride)
    bits = fp_add(bits, eq[bit_rows[i]], c);
  acc[0] = fp_add(acc[0], fp_mul(bits, rho2, c), c);
  block_fp_sum<1>(acc, c, partial + b - blockIdx.x);
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(counter, 1u) == (unsigned)col0_blocks - 1;
    __threadfence();
  }
  __syncthreads();
  if (!last) return;
  acc[0] = fp_zero();
  for (int k = threadIdx.x; k < col0_blocks; k += kThreads) {
    const ulonglong2 w = __ldcg(reinterpret_cast<const ulonglong2 *>(partial + k));
    acc[0] = fp_add(acc[0], fp{w.x, w.y}, c);
  }
  block_fp_sum<1>(acc, c, total - blockIdx.x);
  if (threadIdx.x == 0) {
    D[0] = total[0];
    *counter = 0;
  }
}

// ------------------------------------------------------------------ passes

// 256-bit sums of products of residues, reduced once. With q < 2^126, eight
// products fit.
struct FpWide {
  uint64_t w[4];
};

__device__ __forceinline__ void fp_mac(FpWide &t, fp a, fp b) {
  typedef unsigned __int128 u128;
  u128 s = (u128)a.lo * b.lo + t.w[0];
  t.w[0] = (uint64_t)s;
  s = (u128)a.lo * b.hi + t.w[1] + (uint64_t)(s >> 64);
  t.w[1] = (uint64_t)s;
  const uint64_t top = (uint64_t)(s >> 64);
  s = (u128)a.hi * b.lo + t.w[1];
  t.w[1] = (uint64_t)s;
  s = (u128)a.hi * b.hi + t.w[2] + (uint64_t)(s >> 64);
  u128 r = (u128)(uint64_t)s + top;
  t.w[2] = (uint64_t)r;
  t.w[3] += (uint64_t)(s >> 64) + (uint64_t)(r >> 64);
}

// t 2^-128 mod q for t < 8 q^2: two reduction steps leave less than 3q.
__device__ __forceinline__ fp fp_reduce(const FpWide &t, const FpCtx &c) {
  typedef unsigned __int128 u128;
  uint64_t m = t.w[0] * c.qinv;
  u128 s = (u128)m * c.q0 + t.w[0];
  s = (u128)m * c.q1 + t.w[1] + (uint64_t)(s >> 64);
  const uint64_t w1 = (uint64_t)s;
  s = (u128)t.w[2] + (uint64_t)(s >> 64);
  const uint64_t w2 = (uint64_t)s;
  const uint64_t w3 = t.w[3] + (uint64_t)(s >> 64);
  m = w1 * c.qinv;
  s = (u128)m * c.q0 + w1;
  s = (u128)m * c.q1 + w2 + (uint64_t)(s >> 64);
  fp r{(uint64_t)s, w3 + (uint64_t)(s >> 64)};
  if (fp_ge(r, c.q0, c.q1)) r = fp_sub_raw(r, c.q0, c.q1);
  if (fp_ge(r, c.q0, c.q1)) r = fp_sub_raw(r, c.q0, c.q1);
  return r;
}

static __device__ __noinline__ fp pass_fp_mul(fp a, fp b, const FpCtx &c) {
  return fp_mul(a, b, c);
}

// The eq weights (Montgomery) of the 2^k entries that a bind joins.
struct FpBind {
  fp e[8];
  int k;
};

// eq over the coordinates above a pass as a product of factor tables: factor 0
// over the lowest `low` of them, each further one over seven.
struct FpFactors {
  fp f[4][1 << kFacLog];
  int low, n;
};

// Entry o of a table after the binds, from the 2^k entries it joins; entries at
// or beyond `live` are zero.
__device__ __forceinline__ fp fp_bound(const fp *in, size_t o, size_t live, const FpBind &b,
                                       const FpCtx &c) {
  const fp *p = in + (o << b.k);
  const size_t left = live > (o << b.k) ? live - (o << b.k) : 0;
  auto at = [&](int j) {
    if ((size_t)j >= left) return fp_zero();
    const ulonglong2 v = *reinterpret_cast<const ulonglong2 *>(p + j);
    return fp{v.x, v.y};
  };
  if (b.k == 0) return at(0);
  FpWide t{{0, 0, 0, 0}};
#pragma unroll 2
  for (int j = 0; j < 1 << b.k; j++) fp_mac(t, b.e[j], at(j));
  return fp_reduce(t, c);
}

// A table's value at a point: the difference of the halves at infinity.
__device__ __forceinline__ fp fp_point(const fp *t, int stride, int one, int inf, const FpCtx &c) {
  fp v = t[(one | inf) * stride];
  for (int sub = inf; sub;) {
    sub = (sub - 1) & inf;
    const fp x = t[(one | sub) * stride];
    v = __popc(inf ^ sub) & 1 ? fp_sub(v, x, c) : fp_add(v, x, c);
    if (!sub) break;
  }
  return v;
}

// A pass's sums over the X lanes of each point, posted by each block (few
// blocks) or left in partial[block][point] for the last block, which adds them
// up (lanes over the blocks) and posts them.
template <int kPoints, int kTurns>
__device__ __forceinline__ void fp_pass_end(fp (&sum)[kTurns], int lx, const FpCtx &c, fp *partial,
                                            const PassPost &post) {
  __shared__ bool last;
  const int X = 1 << lx, t = threadIdx.x;
  const bool direct = pass_direct(gridDim.x, 2 * kPoints);
  auto exchange = [](fp v, int off) {
    return fp{__shfl_xor_sync(0xffffffffu, v.lo, off), __shfl_xor_sync(0xffffffffu, v.hi, off)};
  };
  auto put = [&](int at, fp v) {
    handover_post(post.handover, post.seq, 2 * at, v.lo);
    handover_post(post.handover, post.seq, 2 * at + 1, v.hi);
  };
#pragma unroll
  for (int q = 0; q < kTurns; q++) {
    const int u = t + q * kPassThreads, p = u >> lx;
    if ((u & ~31) >= kPoints << lx) break;  // the whole warp
    fp v = sum[q];
    for (int off = X >> 1; off > 0; off >>= 1) v = fp_add(v, exchange(v, off), c);
    if (p < kPoints && (u & (X - 1)) == 0) {
      if (direct)
        put(blockIdx.x * kPoints + p, v);
      else
        partial[(size_t)blockIdx.x * kPoints + p] = v;
    }
  }
  if (direct) return;
  __threadfence();
  __syncthreads();
  if (t == 0) {
    last = atomicAdd(post.counter, 1u) == gridDim.x - 1;
    __threadfence();
  }
  __syncthreads();
  if (!last) return;
  for (int p = t >> 5; p < kPoints; p += kPassThreads / 32) {
    fp v = fp_zero();
    for (unsigned b = t & 31; b < gridDim.x; b += 32) {
      const ulonglong2 w = __ldcg(reinterpret_cast<const ulonglong2 *>(partial + (size_t)b * kPoints + p));
      v = fp_add(v, fp{w.x, w.y}, c);
    }
    for (int off = 16; off > 0; off >>= 1) v = fp_add(v, exchange(v, off), c);
    if ((t & 31) == 0) put(p, v);
  }
  if (t == 0) *post.counter = 0;
}

// One pass of the outer sumcheck over A, B, C: binds (to `out` when b.k > 0),
// then the 3^K sums of eq (A B - C) over the positions above the low K
// coordinates (C is linear, so it only counts at the points without infinity).
// `live` entries of each input table are not known to be zero. Tiles and
// threads as in the GKR's passes (gkr.cu): bound entries, weighted A and C,
// then the points.
struct SpTabs {
  fp *t[3];
};

template <int K>
__global__ void __launch_bounds__(kPassThreads, 2) sp_outer_pass(
    SpTabs in, SpTabs out, size_t live, uint32_t count, const __grid_constant__ FpBind b,
    const __grid_constant__ FpFactors eq, FpCtx c, int lx, fp *partial, PassPost post) {
  constexpr int kPoints = pow3(K), kBlocks = 1 << K;
  constexpr int kTurns = (kPoints * kPassMaxX + kPassThreads - 1) / kPassThreads;
  constexpr int kRow = kPassMaxX + 1;
  __shared__ fp S[3][kBlocks * kRow], E[kPassMaxX];
  const int t = threadIdx.x, X = 1 << lx;
  fp sum[kTurns];
#pragma unroll
  for (int q = 0; q < kTurns; q++) sum[q] = fp_zero();
  for (uint32_t i0 = blockIdx.x << lx; i0 < count; i0 += gridDim.x << lx) {
    if (t >= kPassThreads - 32 && (t & 31) < X) {  // the last warp: the weights
      const uint32_t x = i0 + (t & 31);
      fp e = fp_zero();
      if (x < count) {
        e = eq.f[0][x & ((1u << eq.low) - 1)];
#pragma unroll 1
        for (int g = 1; g < eq.n; g++)
          e = pass_fp_mul(e, eq.f[g][(x >> (eq.low + kFacLog * (g - 1))) & ((1 << kFacLog) - 1)], c);
      }
      E[t & 31] = e;
    }
    const int size = kBlocks << lx;
    for (int u = t; u < 3 * size; u += kPassThreads) {
      const int tab = u / size, slot = u - tab * size, x = slot >> K, a = slot & (kBlocks - 1);
      fp v = fp_zero();
      if (i0 + x < count) {
        const size_t o = ((size_t)i0 << K) + slot;
        v = fp_bound(in.t[tab], o, live, b, c);
        if (b.k) out.t[tab][o] = v;
      }
      S[tab][a * kRow + x] = v;
    }
    __syncthreads();
    for (int u = t; u < 2 * size; u += kPassThreads) {
      const int tab = u >= size ? 2 : 0, slot = u & (size - 1), x = slot & (X - 1);
      fp *p = &S[tab][(slot >> lx) * kRow + x];
      *p = pass_fp_mul(E[x], *p, c);
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kTurns; q++) {
      const int u = t + q * kPassThreads;
      if (u < kPoints << lx) {
        int one, inf;
        point_bits<K, true>(u >> lx, one, inf);
        const int x = u & (X - 1);
        fp v = pass_fp_mul(fp_point(S[0] + x, kRow, one, inf, c),
                           fp_point(S[1] + x, kRow, one, inf, c), c);
        if (!inf) v = fp_sub(v, S[2][one * kRow + x], c);
        sum[q] = fp_add(sum[q], v, c);
      }
    }
    __syncthreads();  // the tile's tables before the next tile's
  }
  fp_pass_end<kPoints, kTurns>(sum, lx, c, partial, post);
}

// One pass of the inner sumcheck over D and W; with kBits, W comes from h's
// bytes (b.k = 3).
template <int K, bool kBits>
__global__ void __launch_bounds__(kPassThreads, 2) sp_inner_pass(
    const fp *D, const fp *W, fp *D2, fp *W2, size_t live, uint32_t count,
    const __grid_constant__ FpBind b, FpCtx c, int lx, fp *partial, PassPost post) {
  constexpr int kPoints = pow3(K), kBlocks = 1 << K;
  constexpr int kTurns = (kPoints * kPassMaxX + kPassThreads - 1) / kPassThreads;
  constexpr int kRow = kPassMaxX + 1;
  __shared__ fp S[2][kBlocks * kRow], W8[kBits ? 256 : 1];
  const int t = threadIdx.x, X = 1 << lx;
  if (kBits) {
    if (t < 256) {
      fp v = fp_zero();
#pragma unroll 1
      for (int j = 0; j < 8; j++)
        if ((t >> j) & 1) v = fp_add(v, b.e[j], c);
      W8[t] = v;
    }
    __syncthreads();
  }
  fp sum[kTurns];
#pragma unroll
  for (int q = 0; q < kTurns; q++) sum[q] = fp_zero();
  for (uint32_t i0 = blockIdx.x << lx; i0 < count; i0 += gridDim.x << lx) {
    const int size = kBlocks << lx;
    for (int u = t; u < 2 * size; u += kPassThreads) {
      const int tab = u >= size, slot = u & (size - 1), x = slot >> K, a = slot & (kBlocks - 1);
      fp v = fp_zero();
      if (i0 + x < count) {
        const size_t o = ((size_t)i0 << K) + slot;
        if (kBits && tab)
          v = W8[reinterpret_cast<const uint8_t *>(W)[o]];
        else
          v = fp_bound(tab ? W : D, o, live, b, c);
        if (b.k) (tab ? W2 : D2)[o] = v;
      }
      S[tab][a * kRow + x] = v;
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kTurns; q++) {
      const int u = t + q * kPassThreads;
      if (u < kPoints << lx) {
        int one, inf;
        point_bits<K, true>(u >> lx, one, inf);
        const int x = u & (X - 1);
        sum[q] = fp_add(sum[q], pass_fp_mul(fp_point(S[0] + x, kRow, one, inf, c),
                                            fp_point(S[1] + x, kRow, one, inf, c), c), c);
      }
    }
    __syncthreads();  // the tile's tables before the next tile's
  }
  fp_pass_end<kPoints, kTurns>(sum, lx, c, partial, post);
}

// A residue sum of up to 2^32 terms.
struct FpSum160 {
  uint64_t lo, hi;
  uint32_t top;
  __device__ __forceinline__ void add(fp v) {
    asm("add.cc.u64 %0, %0, %3;\n\taddc.cc.u64 %1, %1, %4;\n\taddc.u32 %2, %2, 0;"
        : "+l"(lo), "+l"(hi), "+r"(top)
        : "l"(v.lo), "l"(v.hi));
  }
  // mod q: the low 128 bits times one and the rest times 2^128
  __device__ __forceinline__ fp reduce(const FpCtx &c) const {
    return fp_add(fp_mul(fp{lo, hi}, c.one, c), fp_mul(fp{top, 0}, c.r2, c), c);
  }
};

// The inner sumcheck's first three rounds: H[a][b], the sum over the groups of
// eight columns of D's entry a where h's bit b is set. One lane per column, so
// D is read once, coalesced; 32 columns without a set bit are skipped. The sums
// stay unreduced (160 bits) until the end. 2^25 columns: 0.5 GB.
constexpr int kSpBitsBlocks = 4 * kSMs;
__global__ void __launch_bounds__(kThreads) sp_bits(const fp *__restrict__ D,
                                                    const uint32_t *__restrict__ bits, size_t words,
                                                    FpCtx c, fp *partial, PassPost post) {
  __shared__ fp sums[kThreads / 32][64];
  __shared__ bool last;
  const int t = threadIdx.x, lane = t & 31;
  const size_t warps = (size_t)gridDim.x * (kThreads / 32);
  FpSum160 h[8];
#pragma unroll
  for (int b = 0; b < 8; b++) h[b] = FpSum160{0, 0, 0};
#pragma unroll 2
  for (size_t k = blockIdx.x * (size_t)(kThreads / 32) + (t >> 5); k < words; k += warps) {
    const uint32_t word = __ldg(bits + k);
    if (!word) continue;
    const ulonglong2 w = *reinterpret_cast<const ulonglong2 *>(D + 32 * k + lane);
    const uint32_t byte = word >> (lane & 24);
#pragma unroll
    for (int b = 0; b < 8; b++)
      if ((byte >> b) & 1) h[b].add(fp{w.x, w.y});
  }
#pragma unroll
  for (int b = 0; b < 8; b++) {
    fp v = h[b].reduce(c);
    for (int off = 8; off < 32; off <<= 1)
      v = fp_add(v, fp{__shfl_xor_sync(0xffffffffu, v.lo, off), __shfl_xor_sync(0xffffffffu, v.hi, off)}, c);
    if (lane < 8) sums[t >> 5][8 * lane + b] = v;
  }
  __syncthreads();
  if (t < 64) {
    fp v = sums[0][t];
    for (int w = 1; w < kThreads / 32; w++) v = fp_add(v, sums[w][t], c);
    partial[(size_t)blockIdx.x * 64 + t] = v;
  }
  __threadfence();
  __syncthreads();
  if (t == 0) {
    last = atomicAdd(post.counter, 1u) == gridDim.x - 1;
    __threadfence();
  }
  __syncthreads();
  if (!last) return;
  {  // four threads per sum over the blocks
    fp v = fp_zero();
    for (unsigned b = t & 3; b < gridDim.x; b += 4) {
      const ulonglong2 w = __ldcg(reinterpret_cast<const ulonglong2 *>(partial + (size_t)b * 64 + (t >> 2)));
      v = fp_add(v, fp{w.x, w.y}, c);
    }
    for (int off = 1; off < 4; off <<= 1)
      v = fp_add(v, fp{__shfl_xor_sync(0xffffffffu, v.lo, off), __shfl_xor_sync(0xffffffffu, v.hi, off)}, c);
    if ((t & 3) == 0) {
      handover_post(post.handover, post.seq, 2 * (t >> 2), v.lo);
      handover_post(post.handover, post.seq, 2 * (t >> 2) + 1, v.hi);
    }
  }
  if (t == 0) *post.counter = 0;
}

// The last tables to the host, `tables` of n entries each after the binds.
__global__ void __launch_bounds__(64) sp_handover(SpTabs in, int tables, int n, size_t live,
                                                  const __grid_constant__ FpBind b, FpCtx c,
                                                  unsigned long long *handover,
                                                  unsigned long long seq) {
  const int k = blockIdx.x * 64 + threadIdx.x, tab = k / n, o = k % n;
  if (tab >= tables) return;
  const fp v = fp_bound(in.t[tab], o, live, b, c);
  handover_post(handover, seq, 2 * k, v.lo);
  handover_post(handover, seq, 2 * k + 1, v.hi);
}

// ------------------------------------------------------------------- host

// Tables of this many entries or fewer go to the host.
constexpr int kSpHostLog = 7;
static_assert(6 << kSpHostLog <= kHandoverWords, "the last tables fit one handover");

static std::vector<fp> sp_words(const std::vector<uint64_t> &w, size_t n) {
  std::vector<fp> v(n);
  for (size_t k = 0; k < n; k++) v[k] = fp{w[2 * k], w[2 * k + 1]};
  return v;
}

// Adds the blocks' points up into the first `points`.
static std::vector<fp> sp_combine(const std::vector<uint64_t> &w, int points, int blocks,
                                  const FpCtx &c) {
  std::vector<fp> v = sp_words(w, (size_t)points * blocks);
  for (int b = 1; b < blocks; b++)
    for (int p = 0; p < points; p++) v[p] = fp_add(v[p], v[b * points + p], c);
  v.resize(points);
  return v;
}

// Each table folded at r in place (entry o from 2o and 2o + 1, read before it
// is overwritten).
static void host_sp_fold(std::vector<fp> *tab, int T, fp r, const FpCtx &c) {
  for (int t = 0; t < T; t++) {
    const size_t n = tab[t].size() / 2;
    for (size_t o = 0; o < n; o++) tab[t][o] = interp(tab[t][2 * o], tab[t][2 * o + 1], r, c);
    tab[t].resize(n);
  }
}

// A sumcheck's point sums at the first coordinate's three values, summed over
// the others at zeros and ones with weights e.
static void sp_round_sums(const std::vector<fp> &F, int rest, const std::vector<fp> &e,
                          const FpCtx &c, fp (&s)[3]) {
  const size_t block = F.size() / 3;
  for (int d = 0; d < 3; d++) {
    s[d] = fp_zero();
    for (int x = 0; x < 1 << rest; x++) {
      size_t at = 0;  // the next coordinate is the next digit from the top
      for (int q = 0; q < rest; q++) at = 3 * at + ((x >> q) & 1);
      const fp v = F[d * block + at];
      s[d] = fp_add(s[d], e.empty() ? v : fp_mul(e[x], v, c), c);
    }
  }
}

static void sp_fold_points(std::vector<fp> &F, fp r, const FpCtx &c) {
  const size_t block = F.size() / 3;
  for (size_t x = 0; x < block; x++) {  // h0 + r (h1 - h0 - hinf) + r^2 hinf
    const fp h0 = F[x], h1 = F[block + x], hi = F[2 * block + x];
    const fp mid = fp_sub(fp_sub(h1, h0, c), hi, c);
    F[x] = fp_add(h0, fp_mul(r, fp_add(mid, fp_mul(r, hi, c), c), c), c);
  }
  F.resize(block);
}

static FpBind sp_bind_weights(const fp *r, int k, const FpCtx &c) {
  FpBind b{};
  const std::vector<fp> e = sp_eq(r, k, c, c.one);
  for (size_t j = 0; j < e.size(); j++) b.e[j] = e[j];
  b.k = k;
  return b;
}

static void put_canonical(uint8_t *b, fp mont, const FpCtx &c) {
  fp v = fp_mul(mont, fp{1, 0}, c);
  memcpy(b, &v.lo, 8);
  memcpy(b + 8, &v.hi, 8);
}

// recover_full_round_polynomial_and_sample_next_challenge (sumcheck.rs:787-811)
static fp round_message(Transcript &ts, const FpCtx &c, fp &claim, const fp *wl, int ncoef,
                        u128 q, fp *coefs_out) {
  fp co[4];
  co[0] = wl[0];
  co[1] = fp_zero();
  for (int i = 2; i < ncoef; i++) co[i] = wl[i - 1];
  fp at_one = fp_zero();
  for (int i = 0; i < ncoef; i++) at_one = fp_add(at_one, co[i], c);
  co[1] = fp_sub(fp_sub(claim, co[0], c), at_one, c);
  uint8_t msg[64];
  for (int i = 0; i < ncoef; i++) put_canonical(msg + 16 * i, co[i], c);
  ts.public_message(msg, 16 * (size_t)ncoef);
  u128 rc = ts.challenge_fp(q);
  fp r = fp_mul(fp{(uint64_t)rc, (uint64_t)(rc >> 64)}, c.r2, c);
  fp v = fp_zero();
  for (int i = ncoef - 1; i >= 0; i--) v = fp_add(fp_mul(v, r, c), co[i], c);
  claim = v;
  for (int i = 0; i < ncoef; i++) coefs_out[i] = co[i];
  return r;
}

static void launch_bind(const SpartanArgs &a, const fp *tab, const fp *eq, fp rho2, size_t padded,
                        const FpCtx &c, fp *partial, unsigned int *counter, fp *D,
                        cudaStream_t s) {
  const int col0 = grid_for(std::max<size_t>(a.col0_nnz, (size_t)a.n_bit_rows), 4 * kThreads, kSMs);
  k_bind<<<grid_for(padded) + col0, kThreads, 0, s>>>(
      a.csc_off, a.csc_row, a.csc_idx, tab, eq, a.cols, padded, a.bit_rows, a.n_bit_rows, rho2, col0,
      c, partial, counter, D);
  BZ_LAUNCH_CHECK();
}

void spartan_prove(const SpartanArgs &a, Transcript &ts, SpartanScratch &sc, cudaStream_t s,
                   SpartanOut &out) {
  const FpCtx &c = a.ctx;
  const int nr = a.num_row_vars, nc = a.num_col_vars;
  const size_t R = (size_t)1 << nr, Cn = (size_t)1 << nc;
  ts.public_message(a.digest, 32);
  fp tau[kMaxFpPoint];
  for (int i = 0; i < nr; i++) {
    u128 t = ts.challenge_fp(a.q);
    tau[i] = fp_mul(fp{(uint64_t)t, (uint64_t)(t >> 64)}, c.r2, c);
  }
  SpTabs in{{sc.t[1], sc.t[2], sc.t[3]}};
  k_products_to_fp<<<grid_for(R), kThreads, 0, s>>>(a.prod, a.rows, R, c, in.t[0], in.t[1],
                                                    in.t[2]);
  BZ_LAUNCH_CHECK();
  fp claim = fp_zero();
  out.outer.resize(4 * (size_t)nr);
  out.rx.resize(nr);
  RoundChannel *ch = sc.channel;
  KernelProbe &probe = KernelProbe::get();
  std::vector<uint64_t> words(kHandoverWords);
  std::vector<fp> F;
  auto arm = [&] { return PassPost{nullptr, ch->counter, ch->handover_dev, ch->arm().seq}; };
  // BITZ_ROUND_TRACE=1 prints the host time of every device turn
  static const bool trace = getenv("BITZ_ROUND_TRACE") != nullptr;
  auto t_prev = std::chrono::steady_clock::now();
  auto mark = [&](const char *what, int left) {
    if (!trace) return;
    const auto now = std::chrono::steady_clock::now();
    fprintf(stderr, "[spartan] %s, %d coordinates: %7.2f us\n", what, left,
            std::chrono::duration<double, std::micro>(now - t_prev).count());
    t_prev = now;
  };
  fp fin[3];
  {
    // eq(tau) over the coordinates above a pass: groups of seven from the top,
    // group[g][n] over the lowest n... of the group's highest coordinates
    std::vector<std::vector<fp>> group[4];
    for (int g = 0, hi = nr; hi > 0; g++, hi -= kFacLog) {
      if (g == 4) throw CudaError("spartan: too many row variables");
      const int lo = std::max(0, hi - kFacLog);
      for (int at = hi; at >= lo; at--) group[g].push_back(sp_eq(tau + at, hi - at, c, c.one));
    }
    auto factors = [&](int n) {  // over the top n > 0 coordinates
      FpFactors f{};
      const int groups = (n + kFacLog - 1) / kFacLog;
      f.n = groups;
      f.low = n - kFacLog * (groups - 1);
      for (int g = 0; g < groups; g++) {
        const std::vector<fp> &v = group[groups - 1 - g][g == 0 ? f.low : kFacLog];
        std::copy(v.begin(), v.end(), f.f[g]);
      }
      return f;
    };
    // the outer message from t(0), t(1) and t's X^2 coefficient, times the
    // round's eq factor and the bound coordinates' scale
    fp scale = c.one;
    int round = 0;
    auto message = [&](const fp (&t)[3]) {
      const fp l0 = fp_sub(c.one, tau[round], c), l1 = fp_sub(tau[round], l0, c);
      const fp mid = fp_sub(fp_sub(t[1], t[0], c), t[2], c);
      const fp wl[3] = {fp_mul(scale, fp_mul(l0, t[0], c), c),
                        fp_mul(scale, fp_add(fp_mul(l0, t[2], c), fp_mul(l1, mid, c), c), c),
                        fp_mul(scale, fp_mul(l1, t[2], c), c)};
      fp co[4];
      const fp r = round_message(ts, c, claim, wl, 4, a.q, co);
      for (int i = 0; i < 4; i++) out.outer[4 * round + i] = co[i];
      out.rx[round++] = r;
      scale = fp_mul(scale, fp_add(l0, fp_mul(l1, r, c), c), c);
      return r;
    };
    size_t live = a.rows;
    SpTabs spare[2] = {{{sc.t[4], sc.t[5], sc.t[6]}}, {{sc.t[1], sc.t[2], sc.t[3]}}};
    int to = 0;
    FpBind b{};
    int rem = nr;
    while (rem > kSpHostLog) {
      const int k = kPassMaxK, points = pow3(k);
      const size_t live_out = (live + (((size_t)1 << b.k) - 1)) >> b.k;
      // positions past the live entries add nothing
      const uint32_t count = (uint32_t)((live_out + ((size_t)1 << k) - 1) >> k);
      const int lx = pass_tile_log(count, ch->pass_blocks);
      const unsigned int grid = pass_grid(count, lx);
      const bool probed = probe.on("sp_outer_pass");
      if (probed) probe.before(s);
      const PassPost post = arm();
      sp_outer_pass<3><<<grid, kPassThreads, 0, s>>>(in, spare[to], live, count, b,
                                                     factors(rem - k), c, lx, sc.partial, post);
      BZ_LAUNCH_CHECK();
      // three tables of 16-byte residues read, and written bound
      if (probed)
        probe.after(s, "sp_outer_pass",
                    48.0 * ((double)live + (b.k ? (double)live_out : 0.0)));
      if (b.k) {
        in = spare[to];
        to ^= 1;
        live = (size_t)count << k;
      }
      const int blocks = pass_direct(grid, 2 * points) ? (int)grid : 1;
      ch->wait_handover(s, post.seq, words.data(), 2 * points * blocks);
      mark("outer pass", rem);
      F = sp_combine(words, points, blocks, c);
      fp r[kPassMaxK];
      for (int t = 0; t < k; t++) {
        fp sums[3];
        sp_round_sums(F, k - 1 - t, sp_eq(tau + round + 1, k - 1 - t, c, c.one), c, sums);
        r[t] = message(sums);
        sp_fold_points(F, r[t], c);
      }
      b = sp_bind_weights(r, k, c);
      rem -= k;
    }
    const int n = 1 << rem;
    const PassPost post = arm();
    sp_handover<<<(3 * n + 63) / 64, 64, 0, s>>>(in, 3, n, live, b, c, post.handover, post.seq);
    BZ_LAUNCH_CHECK();
    ch->wait_handover(s, post.seq, words.data(), 6 * n);
    mark("outer tables", rem);
    const std::vector<fp> all = sp_words(words, 3 * (size_t)n);
    std::vector<fp> tab[3];
    for (int t = 0; t < 3; t++) tab[t].assign(all.begin() + t * n, all.begin() + (t + 1) * n);
    while (round < nr) {
      const std::vector<fp> e = sp_eq(tau + round + 1, nr - round - 1, c, c.one);
      fp sums[3] = {fp_zero(), fp_zero(), fp_zero()};
      for (size_t j = 0; j < e.size(); j++) {
        const fp a0 = tab[0][2 * j], a1 = tab[0][2 * j + 1], b0 = tab[1][2 * j],
                 b1 = tab[1][2 * j + 1];
        sums[0] = fp_add(sums[0], fp_mul(e[j], fp_sub(fp_mul(a0, b0, c), tab[2][2 * j], c), c), c);
        sums[1] =
            fp_add(sums[1], fp_mul(e[j], fp_sub(fp_mul(a1, b1, c), tab[2][2 * j + 1], c), c), c);
        sums[2] = fp_add(sums[2], fp_mul(e[j], fp_mul(fp_sub(a1, a0, c), fp_sub(b1, b0, c), c), c), c);
      }
      host_sp_fold(tab, 3, message(sums), c);
    }
    for (int k = 0; k < 3; k++) fin[k] = tab[k][0];
    mark("outer host rounds", 0);
  }
  uint8_t msg[48];
  for (int k = 0; k < 3; k++) {
    out.abc[k] = fin[k];
    put_canonical(msg + 16 * k, fin[k], c);
  }
  ts.public_message(msg, 48);
  u128 rhoc = ts.challenge_fp(a.q);
  fp rho = fp_mul(fp{(uint64_t)rhoc, (uint64_t)(rhoc >> 64)}, c.r2, c);
  fp rho2 = fp_mul(rho, rho, c);
  claim = fp_add(fp_add(fin[0], fp_mul(rho, fin[1], c), c), fp_mul(rho2, fin[2], c), c);
  // bind: eq(r_x) over the rows, then the column gather
  fp *eq = sc.t[0];
  fp_eq_table(out.rx.data(), nr, c, eq, s);
  k_bind_table<<<(a.ntab + 127) / 128, 128, 0, s>>>(a.tab_vals, a.tab_which, a.ntab, rho, rho2, c,
                                                     sc.tab);
  BZ_LAUNCH_CHECK();
  fp *D = sc.d[0];
  launch_bind(a, sc.tab, eq, rho2, Cn, c, sc.partial, sc.counter, D, s);
  // inner sumcheck
  out.inner.resize(3 * (size_t)nc);
  out.ry.resize(nc);
  fp dw[2];
  {
    int round = 0;
    auto message = [&](fp at_zero, fp at_inf) {
      const fp wl[2] = {at_zero, at_inf};
      fp co[3];
      const fp r = round_message(ts, c, claim, wl, 3, a.q, co);
      for (int i = 0; i < 3; i++) out.inner[3 * round + i] = co[i];
      out.ry[round++] = r;
      return r;
    };
    auto from_points = [&](int k) {
      fp r[kPassMaxK];
      for (int t = 0; t < k; t++) {
        fp sums[3];
        sp_round_sums(F, k - 1 - t, {}, c, sums);
        r[t] = message(sums[0], sums[2]);
        sp_fold_points(F, r[t], c);
      }
      return sp_bind_weights(r, k, c);
    };
    FpBind b{};
    int rem = nc;
    size_t live = a.cols;
    bool bits = true;
    const fp *d = D, *w = nullptr;
    // every circuit has a compression's 20,456 columns, so the bits' rounds are
    // followed by a pass
    if (rem <= kSpHostLog + kPassMaxK) throw CudaError("spartan: too few columns");
    {
      const PassPost post = arm();
      const size_t n = (a.cols + 31) / 32;
      const bool probed = probe.on("sp_bits");
      if (probed) probe.before(s);
      sp_bits<<<grid_for(n, kThreads / 32, kSpBitsBlocks), kThreads, 0, s>>>(D, a.hbits, n, c,
                                                                             sc.partial, post);
      BZ_LAUNCH_CHECK();
      if (probed) probe.after(s, "sp_bits", (16.0 + 1.0 / 8) * (double)a.cols);
      ch->wait_handover(s, post.seq, words.data(), 128);
      mark("inner bits", rem);
      const std::vector<fp> H = sp_words(words, 64);
      F.assign(27, fp_zero());
      for (int p = 0; p < 27; p++) {
        int one = 0, inf = 0;
        for (int i = 0, q = p; i < 3; i++, q /= 3) {
          one |= (q % 3 == 1) << (2 - i);
          inf |= (q % 3 == 2) << (2 - i);
        }
        for (int x = 0; x < 8; x++)  // signs: a difference of halves at infinity
          for (int y = 0; y < 8; y++)
            if ((x & ~inf) == one && (y & ~inf) == one)
              F[p] = __builtin_popcount((x ^ y) & inf) & 1 ? fp_sub(F[p], H[8 * x + y], c)
                                                           : fp_add(F[p], H[8 * x + y], c);
      }
      b = from_points(3);
      rem -= 3;
    }
    fp *set[2][2] = {{sc.d[2], sc.d[3]}, {sc.d[0], sc.d[1]}};
    int to = 0;
    while (rem > kSpHostLog) {
      const int k = kPassMaxK, points = pow3(k);
      const size_t live_out = (live + (((size_t)1 << b.k) - 1)) >> b.k;
      const uint32_t count = (uint32_t)((live_out + ((size_t)1 << k) - 1) >> k);
      const int lx = pass_tile_log(count, ch->pass_blocks);
      const unsigned int grid = pass_grid(count, lx);
      const bool probed = probe.on("sp_inner_pass");
      if (probed) probe.before(s);
      const PassPost post = arm();
      if (bits)
        sp_inner_pass<3, true><<<grid, kPassThreads, 0, s>>>(
            d, reinterpret_cast<const fp *>(a.hbits), set[to][0], set[to][1], live, count, b, c, lx,
            sc.partial, post);
      else
        sp_inner_pass<3, false><<<grid, kPassThreads, 0, s>>>(d, w, set[to][0], set[to][1], live,
                                                              count, b, c, lx, sc.partial, post);
      BZ_LAUNCH_CHECK();
      if (probed)
        probe.after(s, "sp_inner_pass",
                    (bits ? 16.125 : 32.0) * (double)live + 32.0 * (double)live_out);
      bits = false;
      d = set[to][0];
      w = set[to][1];
      to ^= 1;
      live = (size_t)count << k;
      const int blocks = pass_direct(grid, 2 * points) ? (int)grid : 1;
      ch->wait_handover(s, post.seq, words.data(), 2 * points * blocks);
      mark("inner pass", rem);
      F = sp_combine(words, points, blocks, c);
      b = from_points(k);
      rem -= k;
    }
    const int n = 1 << rem;
    const PassPost post = arm();
    const SpTabs last{{const_cast<fp *>(d), const_cast<fp *>(w), nullptr}};
    sp_handover<<<(2 * n + 63) / 64, 64, 0, s>>>(last, 2, n, live, b, c, post.handover, post.seq);
    BZ_LAUNCH_CHECK();
    ch->wait_handover(s, post.seq, words.data(), 4 * n);
    mark("inner tables", rem);
    const std::vector<fp> all = sp_words(words, 2 * (size_t)n);
    std::vector<fp> tab[2];
    for (int t = 0; t < 2; t++) tab[t].assign(all.begin() + t * n, all.begin() + (t + 1) * n);
    while (round < nc) {
      fp s0 = fp_zero(), si = fp_zero();
      for (size_t j = 0; j < tab[0].size() / 2; j++) {
        const fp d0 = tab[0][2 * j], d1 = tab[0][2 * j + 1], w0 = tab[1][2 * j],
                 w1 = tab[1][2 * j + 1];
        s0 = fp_add(s0, fp_mul(d0, w0, c), c);
        si = fp_add(si, fp_mul(fp_sub(d1, d0, c), fp_sub(w1, w0, c), c), c);
      }
      host_sp_fold(tab, 2, message(s0, si), c);
    }
    dw[0] = tab[0][0];
    dw[1] = tab[1][0];
    mark("inner host rounds", 0);
  }
  out.d_at_ry = dw[0];
  out.final_claim = claim;
  out.ok = fp_mul(dw[0], dw[1], c).lo == claim.lo && fp_mul(dw[0], dw[1], c).hi == claim.hi;
}

// Per-block partial sums of D[y] * E[y] over n entries (mod q).
__global__ void k_fp_dot(const fp *__restrict__ D, const fp *__restrict__ E, size_t n, FpCtx c,
                         fp *partial) {
  fp acc[1] = {fp_zero()};
  for (size_t y = blockIdx.x * (size_t)blockDim.x + threadIdx.x; y < n;
       y += (size_t)gridDim.x * blockDim.x)
    acc[0] = fp_add(acc[0], fp_mul(D[y], E[y], c), c);
  block_fp_sum<1>(acc, c, partial);
}

fp spartan_matrix_eval(const SpartanArgs &a, const fp *rx, fp rho, const fp *ry,
                       SpartanScratch &sc, cudaStream_t s) {
  const FpCtx &c = a.ctx;
  const int nr = a.num_row_vars, nc = a.num_col_vars;
  const size_t Cn = (size_t)1 << nc;
  const fp rho2 = fp_mul(rho, rho, c);
  // the prover's bind at (r_x, rho): D(y) for every column y
  fp *eq = sc.t[0];
  fp_eq_table(rx, nr, c, eq, s);
  k_bind_table<<<(a.ntab + 127) / 128, 128, 0, s>>>(a.tab_vals, a.tab_which, a.ntab, rho, rho2, c,
                                                     sc.tab);
  BZ_LAUNCH_CHECK();
  fp *D = sc.d[0], *EY = sc.d[1];
  launch_bind(a, sc.tab, eq, rho2, Cn, c, sc.partial, sc.counter, D, s);
  // then sum_y D(y) eq(r_y, y)
  fp_eq_table(ry, nc, c, EY, s);
  const int g = grid_for(Cn);
  k_fp_dot<<<g, kThreads, 0, s>>>(D, EY, Cn, c, sc.partial);
  BZ_LAUNCH_CHECK();
  k_fp_finalize<<<1, kThreads, 0, s>>>(sc.partial, g, c, sc.sums);
  BZ_LAUNCH_CHECK();
  BZ_CUDA(cudaMemcpyAsync(sc.host, sc.sums, sizeof(fp), cudaMemcpyDeviceToHost, s));
  BZ_CUDA(stream_wait(s));
  return sc.host[0];
}

// Per-block partial sums of cols[j] (fold_j mod q), fold_j any 128-bit value: a
// residue times 2^256 over 2^128 needs only one factor below q. One thread per
// fold; on the host the 128-bit remainders alone took 1.2 ms for 2^14 folds.
__global__ void k_fold_claim(const fp *__restrict__ folds, const fp *__restrict__ cols, size_t n,
                             FpCtx c, fp *partial) {
  fp acc[1] = {fp_zero()};
  for (size_t j = blockIdx.x * (size_t)blockDim.x + threadIdx.x; j < n;
       j += (size_t)gridDim.x * blockDim.x)
    acc[0] = fp_add(acc[0], fp_mul(fp_mul(folds[j], c.r2, c), cols[j], c), c);
  block_fp_sum<1>(acc, c, partial);
}

void fold_claim(const u128 *folds, const fp *cols, size_t n, const FpCtx &c, SpartanScratch &sc,
                cudaStream_t s) {
  const int g = grid_for(n);
  k_fold_claim<<<g, kThreads, 0, s>>>(reinterpret_cast<const fp *>(folds), cols, n, c, sc.partial);
  BZ_LAUNCH_CHECK();
  k_fp_finalize<<<1, kThreads, 0, s>>>(sc.partial, g, c, sc.sums);
  BZ_LAUNCH_CHECK();
  BZ_CUDA(cudaMemcpyAsync(sc.host, sc.sums, sizeof(fp), cudaMemcpyDeviceToHost, s));
}

FpCtx make_fp_ctx(u128 q) {
  FpCtx c;
  c.q0 = (uint64_t)q;
  c.q1 = (uint64_t)(q >> 64);
  // -q^{-1} mod 2^64 by Newton iteration on the odd low word
  uint64_t inv = 1;
  for (int i = 0; i < 7; i++) inv *= 2 - c.q0 * inv;
  c.qinv = (uint64_t)0 - inv;
  u128 one = ((~(u128)0) % q + 1) % q;  // 2^128 mod q
  c.one = fp{(uint64_t)one, (uint64_t)(one >> 64)};
  u128 x = one;
  for (int i = 0; i < 128; i++) {
    x <<= 1;  // x < q < 2^126: no overflow
    if (x >= q) x -= q;
  }
  c.r2 = fp{(uint64_t)x, (uint64_t)(x >> 64)};
  return c;
}

u128 fp_canonical(fp mont, const FpCtx &c) {
  fp v = fp_mul(mont, fp{1, 0}, c);
  return (u128)v.lo | ((u128)v.hi << 64);
}

// Montgomery residues to canonical values (the 16-byte little-endian codec of
// crates/field/src/codec.rs:69-73), one thread per element.
__global__ void k_fp_canonical(const fp *__restrict__ in, size_t n, FpCtx c, fp *__restrict__ out) {
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n;
       k += (size_t)gridDim.x * blockDim.x)
    out[k] = fp_mul(in[k], fp{1, 0}, c);
}

void fp_canonical_device(const fp *in, size_t n, const FpCtx &c, fp *out, cudaStream_t s) {
  k_fp_canonical<<<grid_for(n), kThreads, 0, s>>>(in, n, c, out);
  BZ_LAUNCH_CHECK();
}

fp fp_to_mont(u128 v, const FpCtx &c) { return fp_mul(fp{(uint64_t)v, (uint64_t)(v >> 64)}, c.r2, c); }

// Every kernel of this file, loaded when the process's first lane on a device
// is made (lane_bootstrap, context.cpp).
void preload_spartan_kernels() {
  load_kernels({(const void *)k_fp_eq,
                (const void *)k_products_to_fp,
                (const void *)k_fp_finalize,
                (const void *)sp_outer_pass<3>,
                (const void *)sp_inner_pass<3, true>,
                (const void *)sp_inner_pass<3, false>,
                (const void *)sp_bits,
                (const void *)sp_handover,
                (const void *)k_bind_table,
                (const void *)k_bind,
                (const void *)k_fp_dot,
                (const void *)k_fold_claim,
                (const void *)k_fp_canonical});
}

}  // namespace bz
