// The grand-product GKR (crates/gkr/src/lib.rs:24-81,88-240,785-897).
//
// Leaf (b << s) | c of the product tree is the row image b where column c has
// bit b set, one elsewhere (crates/prover/src/reduce.rs:1-5); node k of each
// layer multiplies nodes k and k + half of the layer below. A node of layers 0
// to 3 takes 2, 4, 16 or 256 values, by the column's bits in its rows (the
// reference keeps layers 0-2 in 16-entry lookup tables for the same reason,
// lib.rs:274-303). Layers 2 and 3 are looked up and stored, the layers above
// are products of them; layers 0 and 1 are never stored, their sumchecks start
// from the bits. Round messages are exact field values, so any order of sums
// gives the reference's bytes.
//
// A layer sumcheck binds its point's top coordinate first: with L = C[0, 2^n)
// and R = C[2^n, 2^(n+1)) it sums eq(x) L(x) R(x). Several rounds go through
// the device as one pass. A pass over the top K coordinates X sums, for every
// point p of {0, 1, infinity}^K (infinity: the coefficient of X^1, i.e. the
// sum of the halves),
//
//   F(p) = sum over the lower coordinates x of eq(x) L(p, x) R(p, x),
//
// which determines the product polynomial (degree two in each coordinate), so
// the host reads the 3^K values and runs K rounds by itself; the next pass
// binds the K coordinates at once. What bounds a small round is its
// host-device turn, and a pass of three rounds makes 8 + 27 products where
// three rounds make 4 (4 + 2 + 1) = 28, so a turn per three rounds is the
// better split at every size. Tables of 2^kHostLog entries or fewer go to the
// host, which runs the remaining rounds. Measured for the seven layers, a
// round a turn before and passes now: s = 18 8.57 -> 3.3 ms, s = 14 in a
// proof of 64 blocks 1.52 -> 0.75 ms (77 turns -> 25).
#include <algorithm>
#include <chrono>
#include <cstdio>
#include <vector>

#include "context.hpp"
#include "eq.cuh"
#include "gkr.hpp"
#include "host_tail.hpp"
#include "passes.cuh"

namespace bz {

// Layers 2 and 3 from the bits. Block row y holds nodes y and y + 16 of layer 2
// and node y of layer 3, their product, so a column is 4 + 4 bits, three
// lookups and three coalesced stores: the kernel is bound by its writes
// (48 of the 63 entries a column has in the stored layers).
__device__ __forceinline__ f128 row_value(const f128 *images, int row, int bit) {
  return bit ? ld(images + row) : mk(1, 0);
}

__global__ void __launch_bounds__(kThreads) gkr_low_layers(const f128 *__restrict__ cols, int s,
                                                           const f128 *__restrict__ images,
                                                           f128 *__restrict__ layer2,
                                                           f128 *__restrict__ layer3) {
  __shared__ f128 two[2][16], three[256];
  const int y = blockIdx.y, t = threadIdx.x;
  if (t < 32) {
    const int node = y + (t & 16), v = t & 15;
    f128 p[2];
#pragma unroll
    for (int i = 0; i < 2; i++)
      p[i] = gmul(row_value(images, node + 64 * i, (v >> (2 * i)) & 1),
                  row_value(images, node + 64 * i + 32, (v >> (2 * i + 1)) & 1));
    two[t >> 4][v] = gmul(p[0], p[1]);
  }
  __syncthreads();
  three[t] = gmul(two[0][t & 15], two[1][t >> 4]);
  __syncthreads();
  const size_t n = (size_t)1 << s;
  for (size_t c = blockIdx.x * (size_t)blockDim.x + t; c < n; c += (size_t)gridDim.x * blockDim.x) {
    const uint4 w = __ldg(reinterpret_cast<const uint4 *>(cols + c));
    auto four = [&](int r) {  // bits r, r + 32, r + 64, r + 96
      return (int)(((w.x >> r) & 1) | ((w.y >> r) & 1) << 1 | ((w.z >> r) & 1) << 2 |
                   ((w.w >> r) & 1) << 3);
    };
    const int i = four(y), j = four(y + 16);
    st(layer2 + ((size_t)y << s) + c, two[0][i]);
    st(layer2 + ((size_t)(y + 16) << s) + c, two[1][j]);
    st(layer3 + ((size_t)y << s) + c, three[16 * j + i]);
  }
}

// Layers 4 to 7: a thread takes a column's 16 nodes of layer 3 through the four
// levels, 15 products. Padded columns have only ones.
__global__ void __launch_bounds__(128) gkr_high_layers(const f128 *__restrict__ layer3, int s,
                                                       f128 *__restrict__ l4, f128 *__restrict__ l5,
                                                       f128 *__restrict__ l6, f128 *__restrict__ l7,
                                                       size_t live) {
  const size_t n = (size_t)1 << s;
  for (size_t c = blockIdx.x * (size_t)blockDim.x + threadIdx.x; c < n;
       c += (size_t)gridDim.x * blockDim.x) {
    const bool one = c >= live;
    f128 v[8];
#pragma unroll
    for (int k = 0; k < 8; k++) {
      const size_t at = ((size_t)k << s) + c;
      v[k] = one ? mk(1, 0) : gmul(ld(layer3 + at), ld(layer3 + at + ((size_t)8 << s)));
      st(l4 + at, v[k]);
    }
#pragma unroll
    for (int k = 0; k < 4; k++) {
      if (!one) v[k] = gmul(v[k], v[k + 4]);
      st(l5 + ((size_t)k << s) + c, v[k]);
    }
#pragma unroll
    for (int k = 0; k < 2; k++) {
      if (!one) v[k] = gmul(v[k], v[k + 2]);
      st(l6 + ((size_t)k << s) + c, v[k]);
    }
    st(l7 + c, one ? v[0] : gmul(v[0], v[1]));
  }
}

// ------------------------------------------------------------------ passes

// Padding: the low s bits of every layer index are the column, and a column at
// or beyond `live` has only one-valued nodes, before and after any bind
// (1 + r (1 + 1) = 1). Whenever position x of a block is such a column, so is
// the same position of the higher blocks (same column, or a higher one below
// 2^s), so a pass leaves those positions out: they add eq(x) to F at the points
// without infinity and nothing at the others.
// eq over the lowest 14 coordinates, the product of the first two factors, for
// passes over more: one product per position instead of one per factor.
constexpr int kEqLowLog = 2 * kFacLog;
__global__ void __launch_bounds__(kThreads) gkr_eq_low(const __grid_constant__ EqFactors<2> eq,
                                                       f128 *__restrict__ out) {
  const int x = blockIdx.x * kThreads + threadIdx.x;
  st(out + x, gmul(eq.f[0][x & ((1 << kFacLog) - 1)], eq.f[1][x >> kFacLog]));
}

// One pass. Binds the coordinates of `b` (in place: the entry at pos comes from
// pos + j N), then sums the 3^K points over the live positions of the 2^log_m
// below the top K coordinates, and the eq weights of those positions. The last
// block posts the 3^K + 1 sums as handover publication seq.
//
// A block works tiles of X = 2^lx positions: the 2 2^K X bound entries, one per
// thread into shared memory, the 2^K X products of the weights with L, then the
// 3^K X wide products, whose sums stay in registers (thread t of turn q always
// has the same point). A tenth warp forms the next tile's weights meanwhile: in
// line, their two or three dependent products left nine warps waiting for half
// of a tile's time (layer of 2^22 entries, first pass: 618 us). X shrinks with
// the number of positions, so that a small pass still spreads over the SMs; the
// first pass of a large layer (K = 2, nothing to bind) takes tiles of 64, which
// fill its turns. kLow: the weights' lowest 14 coordinates come from eq_low.
template <int K, bool kLow>
struct PassShape {
  static constexpr int kMaxLx = K == 2 ? 6 : 5, kMaxX = 1 << kMaxLx;
  static constexpr int kFactors = kLow ? 3 : 2, kBlocksPerSm = K == 2 ? 3 : 2;
  static constexpr int kThreadsAll = kPassThreads + 32;
};

__device__ __forceinline__ void main_warps_sync() {
  asm volatile("bar.sync 1, %0;" ::"n"(kPassThreads) : "memory");
}

template <int K, bool kLow>
__global__ void __launch_bounds__(PassShape<K, kLow>::kThreadsAll, PassShape<K, kLow>::kBlocksPerSm)
    gkr_pass(f128 *__restrict__ c, size_t n_half, int log_m, PassBind b,
             const __grid_constant__ EqFactors<PassShape<K, kLow>::kFactors> eq,
             const f128 *__restrict__ eq_low, size_t colmask, uint32_t live, uint32_t count, int lx,
             PassPost post) {
  using S = PassShape<K, kLow>;
  constexpr int kPoints = pow3(K), kBlocks = 1 << K, kWords = 2 * (kPoints + 1);
  constexpr int kTurns = (kPoints * S::kMaxX + kPassThreads - 1) / kPassThreads;
  __shared__ MulTable T[K == 2 ? 1 : kPassMaxK];
  __shared__ f128 G[kBlocks * S::kMaxX], R[kBlocks * S::kMaxX], E[2][S::kMaxX];
  __shared__ uint32_t P[2][S::kMaxX];  // a tile's positions; kNone past the last
  constexpr uint32_t kNone = 0xffffffffu;
  const int t = threadIdx.x;
  const size_t m = (size_t)1 << log_m, n = m << K;
  const int X = 1 << lx;
  const bool eq_warp = t >= kPassThreads;
  if (K > 2) pass_tables(T, b.r, b.k);
  // position of live index i: rows of `live` columns when a block spans whole
  // rows of the column space, else i itself
  const bool by_row = m > colmask;
  auto position = [&](uint32_t i) -> uint32_t {
    if (!by_row) return i;
    const uint32_t row = i / live;
    return row * (uint32_t)(colmask + 1) + (i - row * live);
  };
  auto positions = [&](uint32_t i0, uint32_t *out) {
    for (int k = t & 31; k < X; k += 32) out[k] = i0 + k < count ? position(i0 + k) : kNone;
  };
  f128 sum_e = mk(0, 0);
  auto weights = [&](const uint32_t *at, f128 *out) {  // a tile's weights
    for (int k = t & 31; k < X; k += 32) {
      f128 e = mk(0, 0);
      const uint32_t x = at[k];
      if (x != kNone) {
        constexpr int kMask = (1 << kFacLog) - 1;
        if (kLow) {
          e = pass_mul(ld(eq_low + (x & ((1 << kEqLowLog) - 1))),
                       eq.f[0][(x >> kEqLowLog) & kMask]);
#pragma unroll 1
          for (int g = 1; g < S::kFactors && kEqLowLog + g * kFacLog < log_m; g++)
            e = pass_mul(e, eq.f[g][(x >> (kEqLowLog + g * kFacLog)) & kMask]);
        } else {
          e = eq.f[0][x & kMask];
          if (log_m > kFacLog) e = pass_mul(e, eq.f[1][(x >> kFacLog) & kMask]);
        }
      }
      out[k] = e;
      sum_e = gadd(sum_e, e);
    }
  };
  wide sum[kTurns];
#pragma unroll
  for (int q = 0; q < kTurns; q++) sum[q] = wzero();
  const uint32_t step = gridDim.x << lx;
  if (eq_warp) positions(blockIdx.x << lx, P[0]);
  __syncthreads();
  if (eq_warp) {  // weights of the tile and positions of the next one
    int buf = 0;
    weights(P[0], E[0]);
    for (uint32_t i0 = blockIdx.x << lx; i0 < count; i0 += step, buf ^= 1) {
      if (i0 + step < count) positions(i0 + step, P[buf ^ 1]);
      __syncthreads();  // the tile's entries and weights
      if (i0 + step < count) weights(P[buf ^ 1], E[buf ^ 1]);
    }
  } else {
    int buf = 0;
    int at_one[kTurns], at_inf[kTurns];  // a turn's point
#pragma unroll
    for (int q = 0; q < kTurns; q++)
      point_bits<K, false>((t + q * kPassThreads) >> lx, at_one[q], at_inf[q]);
    for (uint32_t i0 = blockIdx.x << lx; i0 < count; i0 += step, buf ^= 1) {
      // entry `slot` (block slot >> lx, position slot mod X) of the tile of L,
      // then of R
      const int half = kBlocks << lx;
      auto entry = [&](int slot) -> f128 * {
        const uint32_t x = P[buf][slot & (X - 1)];
        if (x == kNone) return nullptr;
        return (slot >= half ? c + n_half : c) + x + (size_t)((slot & (half - 1)) >> lx) * m;
      };
      if (K > 2 && b.k && lx <= kLaneTileLog) {
        const int gl = b.k - 1;
        for (int u = t; u < 2 * half << gl; u += kPassThreads) {
          const int slot = u >> gl;
          f128 *at = entry(slot);
          f128 v = pass_bind_lanes<false>(
              [&](int j) { return at ? ld(at + j * n) : mk(0, 0); }, T, b.k, u & ((1 << gl) - 1));
          if (u & ((1 << gl) - 1)) continue;
          if (at) st(at, v);
          (slot >= half ? R : G)[slot & (half - 1)] = v;
        }
      } else {
        for (int slot = t; slot < 2 * half; slot += kPassThreads) {
          f128 *at = entry(slot);
          f128 v = mk(0, 0);
          if (at && K == 2) {
            v = ld(at);
          } else if (at) {
            v = pass_bind<false>([&](int j) { return ld(at + j * n); }, T, b.k);
            if (b.k) st(at, v);
          }
          (slot >= half ? R : G)[slot & (half - 1)] = v;
        }
      }
      __syncthreads();
      for (int u = t; u < half; u += kPassThreads) G[u] = pass_mul(E[buf][u & (X - 1)], G[u]);
      main_warps_sync();
#pragma unroll
      for (int q = 0; q < kTurns; q++) {
        const int u = t + q * kPassThreads;
        if (u < kPoints << lx) {
          const int x = u & (X - 1);
          wacc(sum[q], pass_wide(point_value(G + x, X, at_one[q], at_inf[q]),
                                 point_value(R + x, X, at_one[q], at_inf[q])));
        }
      }
      main_warps_sync();  // the tile's tables before the next tile's
    }
  }
  const bool direct = pass_direct(gridDim.x, kWords);
  if (!eq_warp) {
    pass_reduce<kPoints, kTurns>(sum, lx, kWords, direct, post);
  } else {
    for (int off = 16; off > 0; off >>= 1) {
      sum_e.lo ^= __shfl_xor_sync(0xffffffffu, sum_e.lo, off);
      sum_e.hi ^= __shfl_xor_sync(0xffffffffu, sum_e.hi, off);
    }
    if ((t & 31) == 0) {
      const int at = 2 * kPoints;
      if (direct) {
        handover_post(post.handover, post.seq, blockIdx.x * kWords + at, sum_e.lo);
        handover_post(post.handover, post.seq, blockIdx.x * kWords + at + 1, sum_e.hi);
      } else {
        atomicXor(post.acc + at, (unsigned long long)sum_e.lo);
        atomicXor(post.acc + at + 1, (unsigned long long)sum_e.hi);
      }
    }
  }
  if (!direct) pass_publish(post.acc, kWords, post.counter, post.handover, post.seq);
}

// The layer's last tables to the host: L, then R, of n entries each after the
// binds of `b`, as handover publication seq (two words per entry).
constexpr int kHandThreads = 256, kHandEntries = 64;  // up to four lanes per entry
__global__ void __launch_bounds__(kHandThreads) gkr_handover(const f128 *__restrict__ c,
                                                             size_t n_half, int n, PassBind b,
                                                             unsigned long long *handover,
                                                             unsigned long long seq) {
  __shared__ MulTable T[kPassMaxK];
  pass_tables(T, b.r, b.k);
  const int gl = b.k > 1 ? b.k - 1 : 0, q = threadIdx.x & ((1 << gl) - 1);
  if (threadIdx.x >> 5 >= (kHandEntries << gl) >> 5) return;  // whole warps
  const int k = blockIdx.x * kHandEntries + (threadIdx.x >> gl);
  const f128 *at = k < n ? c + k : c + n_half + (k - n);
  auto in = [&](int j) { return k < 2 * n ? ld(at + (size_t)j * n) : mk(0, 0); };
  const f128 v = b.k ? pass_bind_lanes<false>(in, T, b.k, q) : in(0);
  if (q || k >= 2 * n) return;
  handover_post(handover, seq, 2 * k, v.lo);
  handover_post(handover, seq, 2 * k + 1, v.hi);
}

// ------------------------------------------ the two lowest layers' row rounds
//
// A node of layer 0 or 1 is a sum over features of the column's bits: layer 0
// has 1 + bit d (d: the row's image plus one), layer 1, with rows a and a + 64,
// 1 + p d + q d' + p q d d'. So the sums of all rounds over row coordinates
// (6 of layer 0, 5 of layer 1) come from the weighted counts
//
//   X[i][j] = sum over the columns with features i and j of eq(column),
//
// i over the features of the rows below the top coordinate and j over those
// above it: 64 x 64 and 96 x 96. Over 128 columns such a sum is one product
// through a window table whose single-bit entries are the columns' weights,
// with the two features' common bits as the other factor. That is 13,600
// lookup products per 128 columns for both layers, where the dense rounds make
// 127 - 31 = 96 x 9 general ones per column.

template <int NFEAT>
struct GramShape {
  static constexpr int kGroups = NFEAT == 64 ? 4 : 3;  // thread groups over j
  static constexpr int kThreadsPer = NFEAT * kGroups;
  static constexpr int kRow = NFEAT + 1;  // X's row; index NFEAT is the constant feature
};

template <int NFEAT>
__device__ __forceinline__ uint4 feature(const uint4 *rows, int i, bool upper) {
  if (NFEAT == 64) return rows[i + (upper ? 64 : 0)];
  const int at = (i & 31) + (upper ? 32 : 0);
  const uint4 p = rows[at], q = rows[at + 64];
  if (i < 32) return p;
  if (i < 64) return q;
  return make_uint4(p.x & q.x, p.y & q.y, p.z & q.z, p.w & q.w);
}

static __device__ __forceinline__ f128 and_bits(uint4 a, uint4 b) {
  return mk((uint64_t)(a.x & b.x) | (uint64_t)(a.y & b.y) << 32,
            (uint64_t)(a.z & b.z) | (uint64_t)(a.w & b.w) << 32);
}

// Thread (i, group) sums J features j of its group over the block's chunks of
// 128 columns; blockIdx.y takes the other j. J = 16 uses a chunk's table 16
// times per thread; J = 4 spreads few chunks over the chip.
template <int NFEAT, int J>
__global__ void __launch_bounds__(GramShape<NFEAT>::kThreadsPer) gkr_gram(
    const f128 *__restrict__ cols, uint32_t live, int log_cols,
    const __grid_constant__ EqFactors<5> eq, unsigned long long *X) {
  using S = GramShape<NFEAT>;
  __shared__ MulTable T;
  __shared__ uint4 rows[128];  // row r's bits of the chunk's 128 columns
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int i = t % NFEAT, group = t / NFEAT;
  const int j0 = (blockIdx.y * S::kGroups + group) * J;
  f128 sum[J], one = mk(0, 0);
#pragma unroll
  for (int q = 0; q < J; q++) sum[q] = mk(0, 0);
  const uint32_t chunks = (live + 127) / 128;
  for (uint32_t ch = blockIdx.x; ch < chunks; ch += gridDim.x) {
    if (t < 128) {
      f128 e = eq.f[0][t];
#pragma unroll 1
      for (int g = 1; g < 5 && g * kFacLog < log_cols; g++)
        e = pass_mul(e, eq.f[g][(ch >> ((g - 1) * kFacLog)) & ((1 << kFacLog) - 1)]);
      T.lo[t >> 2][1 << (t & 3)] = e.lo;
      T.hi[t >> 2][1 << (t & 3)] = e.hi;
    }
    if (warp < 8) {  // 32 columns by 64 rows per warp, transposed by ballots
      const uint32_t c = ch * 128 + (warp & 3) * 32 + lane;
      const ulonglong2 w =
          c < live ? __ldg(reinterpret_cast<const ulonglong2 *>(cols + c)) : make_ulonglong2(0, 0);
      const uint64_t half = warp < 4 ? w.x : w.y;
      uint32_t r0 = 0, r1 = 0;
#pragma unroll 8
      for (int r = 0; r < 32; r++) {
        const uint32_t a = __ballot_sync(0xffffffffu, (half >> r) & 1);
        const uint32_t b = __ballot_sync(0xffffffffu, (half >> (r + 32)) & 1);
        if (lane == r) r0 = a, r1 = b;
      }
      uint32_t *out = reinterpret_cast<uint32_t *>(rows + (warp < 4 ? 0 : 64));
      out[4 * lane + (warp & 3)] = r0;
      out[4 * (lane + 32) + (warp & 3)] = r1;
    }
    __syncthreads();
    fill_windows(T.lo, T.hi, 32);
    __syncthreads();
    const uint4 fa = feature<NFEAT>(rows, i, false);
#pragma unroll
    for (int q = 0; q < J; q++)
      sum[q] = gadd(sum[q], pass_table(&T, and_bits(fa, feature<NFEAT>(rows, j0 + q, true))));
    if (blockIdx.y == 0 && group < 2) {  // the features by themselves
      const uint4 f = group ? feature<NFEAT>(rows, i, true) : fa;
      one = gadd(one, pass_table(&T, and_bits(f, f)));
    }
    __syncthreads();  // the chunk's table before the next chunk's
  }
  auto add = [&](int a, int b, f128 v) {
    unsigned long long *x = X + 2 * (a * S::kRow + b);
    if (v.lo) atomicXor(x, (unsigned long long)v.lo);
    if (v.hi) atomicXor(x + 1, (unsigned long long)v.hi);
  };
#pragma unroll
  for (int q = 0; q < J; q++) add(i, j0 + q, sum[q]);
  if (blockIdx.y == 0 && group < 2) group ? add(NFEAT, i, one) : add(i, NFEAT, one);
}

// From the counts to the point sums of all row rounds: first
// H[a][b] = sum over the columns of eq L(a) R(b) for every pair of rows, then,
// a coordinate at a time, {0, 1, infinity} from the pairs of its bit: the
// entries (0,0), (1,1) and the sum of all four. 16 blocks of 256 threads form H
// and the top coordinates (two, or one) by lane exchanges; the last block to
// finish does the other four in shared memory and posts the 729 or 243 sums.
template <int LAYER>
__global__ void __launch_bounds__(256) gkr_moments(const unsigned long long *__restrict__ X,
                                                   const f128 *__restrict__ images,
                                                   f128 *__restrict__ mid, unsigned int *counter,
                                                   unsigned long long *handover,
                                                   unsigned long long seq) {
  constexpr int kDone = LAYER == 0 ? 9 : 3;  // digit values formed by the lanes
  constexpr int kFeat = LAYER == 0 ? 64 : 96, kRow = GramShape<kFeat>::kRow;
  __shared__ f128 A[27 * 64], B[81 * 16];
  __shared__ bool last;
  const int t = threadIdx.x, u = blockIdx.x * 256 + t;
  const int w = (u >> 4) & 255, a_low = w & 15, b_low = w >> 4;
  auto delta = [&](int row) {
    f128 d = ld(images + row);
    d.lo ^= 1;
    return d;
  };
  auto x_at = [&](int a, int b) {
    if (a == kFeat && b == kFeat) return mk(1, 0);
    const ulonglong2 v = __ldcg(reinterpret_cast<const ulonglong2 *>(X) + (a * kRow + b));
    return mk(v.x, v.y);
  };
  auto lanes_xor = [](f128 v, int m) {
    v.lo ^= __shfl_xor_sync(0xffffffffu, v.lo, m);
    v.hi ^= __shfl_xor_sync(0xffffffffu, v.hi, m);
    return v;
  };
  auto digit = [](int role) { return role == 0 ? 0 : role == 3 ? 1 : 2; };
  const int role2 = (u >> 2) & 3;
  f128 v;
  if (LAYER == 0) {
    const int a = a_low | (role2 & 1) << 4 | (u & 1) << 5;
    const int b = b_low | (role2 >> 1) << 4 | ((u >> 1) & 1) << 5;
    const f128 da = delta(a), db = delta(64 + b);
    v = gadd(gadd(mk(1, 0), pass_mul(da, x_at(a, kFeat))),
             pass_mul(db, gadd(x_at(kFeat, b), pass_mul(da, x_at(a, b)))));
  } else {
    // lane f of four: the terms with feature f of R (none, r, s, r s)
    const int f = u & 3;
    const int a = a_low | (role2 & 1) << 4, b = b_low | (role2 >> 1) << 4;
    const f128 da = delta(a), da2 = delta(a + 64), db = delta(b + 32), db2 = delta(b + 96);
    const int jb = f == 0 ? kFeat : 32 * (f - 1) + b;
    v = gadd(gadd(x_at(kFeat, jb), pass_mul(da, x_at(a, jb))),
             pass_mul(da2, gadd(x_at(32 + a, jb), pass_mul(da, x_at(64 + a, jb)))));
    if (f & 1) v = pass_mul(v, db);
    if (f & 2) v = pass_mul(v, db2);
  }
  // features are ordered r, s, r s: lane 1 has r, lane 2 s, lane 3 both
  const f128 s1 = lanes_xor(lanes_xor(v, 1), 2);
  const int role1 = u & 3;
  if (LAYER == 1 || role1 == 1) v = s1;
  const f128 s2 = lanes_xor(lanes_xor(v, 4), 8);
  if (role2 == 1) v = s2;
  if (role2 != 2) {
    if (LAYER == 0) {
      if (role1 != 2) st(mid + (3 * digit(role1) + digit(role2)) * 256 + w, v);
    } else if (role1 == 0) {
      st(mid + digit(role2) * 256 + w, v);
    }
  }
  __threadfence();
  __syncthreads();
  if (t == 0) {
    last = atomicAdd(counter, 1u) == gridDim.x - 1;
    __threadfence();
  }
  __syncthreads();
  if (!last) return;
  auto ld_mid = [&](int k) {
    const ulonglong2 q = __ldcg(reinterpret_cast<const ulonglong2 *>(mid) + k);
    return mk(q.x, q.y);
  };
  // [done][2^r][2^r] (b, then a) -> [3 done][2^(r-1)][2^(r-1)]
  auto step = [&](auto in, f128 *out, int done, int r) {
    const int q = r - 1, per = 1 << (2 * q);
    for (int k = t; k < 3 * done * per; k += 256) {
      const int d = (k >> (2 * q)) % 3, base = ((k >> (2 * q)) / 3) << (2 * r);
      const int a = k & ((1 << q) - 1), b = (k >> q) & ((1 << q) - 1);
      const int e00 = base + (b << r) + a, e01 = e00 + (1 << q), e10 = e00 + (1 << (q + r)),
                e11 = e10 + (1 << q);
      out[k] = d == 0 ? in(e00) : d == 1 ? in(e11)
                                         : gadd(gadd(in(e00), in(e01)), gadd(in(e10), in(e11)));
    }
    __syncthreads();
  };
  step(ld_mid, A, kDone, 4);
  step([&](int k) { return A[k]; }, B, 3 * kDone, 3);
  step([&](int k) { return B[k]; }, A, 9 * kDone, 2);
  step([&](int k) { return A[k]; }, B, 27 * kDone, 1);
  for (int k = t; k < 2 * 81 * kDone; k += 256)
    handover_post(handover, seq, k, k & 1 ? B[k >> 1].hi : B[k >> 1].lo);
  if (t == 0) *counter = 0;
}

// The layer's tables once its row coordinates are bound: L(c) and R(c) are one
// plus sums over the features of column c of their coefficients (the bound
// row's eq weight times the feature's), through 4-bit windows of the column's
// bits.
struct RowWeights {
  f128 e[64];
};

template <int LAYER>
__global__ void __launch_bounds__(kThreads) gkr_bound_rows(const f128 *__restrict__ cols, int s,
                                                           const f128 *__restrict__ images,
                                                           const __grid_constant__ RowWeights eps,
                                                           f128 *__restrict__ L,
                                                           f128 *__restrict__ R) {
  constexpr int kFeat = LAYER == 0 ? 64 : 96, kWin = kFeat / 4;
  __shared__ uint64_t lo[2 * kWin][16], hi[2 * kWin][16];
  const int t = threadIdx.x;
  for (int u = t; u < 2 * kFeat; u += kThreads) {
    const int side = u / kFeat, i = u % kFeat;
    f128 k;
    if (LAYER == 0) {
      f128 d = ld(images + 64 * side + i);
      d.lo ^= 1;
      k = pass_mul(eps.e[i], d);
    } else {
      const int a = i & 31, row = a + 32 * side;
      f128 d = ld(images + row), d2 = ld(images + row + 64);
      d.lo ^= 1;
      d2.lo ^= 1;
      k = pass_mul(eps.e[a], i < 32 ? d : d2);
      if (i >= 64) k = pass_mul(k, d);
    }
    lo[u >> 2][1 << (u & 3)] = k.lo;
    hi[u >> 2][1 << (u & 3)] = k.hi;
  }
  __syncthreads();
  fill_windows(lo, hi, 2 * kWin);
  __syncthreads();
  const size_t n = (size_t)1 << s;
  for (size_t c = blockIdx.x * (size_t)blockDim.x + t; c < n; c += (size_t)gridDim.x * blockDim.x) {
    const uint4 w = __ldg(reinterpret_cast<const uint4 *>(cols + c));
#pragma unroll
    for (int side = 0; side < 2; side++) {
      uint32_t bits[kFeat / 32];
      if (LAYER == 0) {
        bits[0] = side ? w.z : w.x;
        bits[1] = side ? w.w : w.y;
      } else {
        bits[0] = side ? w.y : w.x;
        bits[1] = side ? w.w : w.z;
        bits[kFeat / 32 - 1] = bits[0] & bits[1];
      }
      uint64_t a = 1, b = 0;
#pragma unroll
      for (int k = 0; k < kWin; k++) {
        const uint32_t v = (bits[k / 8] >> (4 * (k % 8))) & 15u;
        a ^= lo[side * kWin + k][v];
        b ^= hi[side * kWin + k][v];
      }
      st((side ? R : L) + c, mk(a, b));
    }
  }
}

// Tables of this many entries or fewer (per half) go to the host: all rounds on
// 2^10 entries cost it about 8 us and their way there 8 more than one of 2^7,
// a device turn of three rounds about 20.
constexpr int kHostLog = 10;
static_assert(4 << kHostLog <= kHandoverWords, "the last tables fit one handover");
// A layer's first pass binds nothing, so three rounds of it make 4.4 products
// per entry where two make 3.25 (and leave a table 4 times the size for the
// next pass): two rounds from this size on, where products are the cost.
constexpr int kFirstLog = 17;

// Returns how many blocks post sums of their own.
template <int K, bool kLow>
static int launch_pass_as(f128 *c, size_t n_half, int log_m, const PassBind &b, const EqHeap *heap,
                          const f128 *eq_low, size_t colmask, uint32_t live, uint32_t count,
                          int spread, const PassPost &post, cudaStream_t st) {
  using S = PassShape<K, kLow>;
  EqFactors<S::kFactors> eq;
  const int skip = kLow ? 2 : 0;  // factors that eq_low holds
  for (int g = 0; g < S::kFactors; g++) {
    const int have = std::min(kFacLog, std::max(0, log_m - (g + skip) * kFacLog));
    memcpy(eq.f[g], heap[g + skip].prefix(have), sizeof(f128) << have);
  }
  int lx = pass_tile_log(count, spread);
  if (lx == 5 && (count >> S::kMaxLx) >= 2u * kSMs) lx = S::kMaxLx;
  const uint32_t tiles = (count + (1u << lx) - 1) >> lx;
  const unsigned int grid =
      std::max(1u, std::min(tiles, (unsigned int)(S::kBlocksPerSm * kSMs)));
  gkr_pass<K, kLow><<<grid, S::kThreadsAll, 0, st>>>(c, n_half, log_m, b, eq, eq_low, colmask, live,
                                                     count, lx, post);
  BZ_LAUNCH_CHECK();
  return pass_direct(grid, 2 * (pow3(K) + 1)) ? (int)grid : 1;
}

template <int K>
static int launch_pass(f128 *c, size_t n_half, int log_m, const PassBind &b, const EqHeap *heap,
                       const f128 *eq_low, size_t colmask, uint32_t live, uint32_t count,
                       int spread, const PassPost &post, cudaStream_t st) {
  return (log_m <= kEqLowLog ? launch_pass_as<K, false> : launch_pass_as<K, true>)(
      c, n_half, log_m, b, heap, eq_low, colmask, live, count, spread, post, st);
}

void gkr_build(const f128 *cols, int s, const f128 *images, GkrScratch &sc, cudaStream_t st_) {
  if (sc.capacity < (size_t)128 << s) throw CudaError("gkr_build: scratch too small");
  const size_t n = (size_t)1 << s, live = sc.live_cols ? sc.live_cols : n;
  const dim3 grid(grid_for(n, kThreads, kSMs / 2), 16);
  gkr_low_layers<<<grid, kThreads, 0, st_>>>(cols, s, images, sc.layer[2], sc.layer[3]);
  BZ_LAUNCH_CHECK();
  gkr_high_layers<<<grid_for(n, 128, kSMs * 16), 128, 0, st_>>>(
      sc.layer[3], s, sc.layer[4], sc.layer[5], sc.layer[6], sc.layer[7], live);
  BZ_LAUNCH_CHECK();
}

// X of layer 0 or 1 (zeroed before) over the live columns.
template <int NFEAT>
static void launch_gram(const f128 *cols, uint32_t live, int s, const EqHeap *heap,
                        unsigned long long *X, cudaStream_t st) {
  using S = GramShape<NFEAT>;
  EqFactors<5> eq;
  for (int g = 0; g < 5; g++) {
    const int have = std::min(kFacLog, std::max(0, s - g * kFacLog));
    memcpy(eq.f[g], heap[g].prefix(have), sizeof(f128) << have);
  }
  if (s < kFacLog)  // weights of columns that do not exist
    memset(eq.f[0] + ((size_t)1 << s), 0, sizeof(f128) * ((1 << kFacLog) - ((size_t)1 << s)));
  const uint32_t chunks = (live + 127) / 128;
  // with J = 16 a block takes 64 x 64 (or 48 x 96) sums of a chunk; below two
  // chunks per SM that leaves SMs idle, so four times the blocks take a quarter
  if (chunks >= 2 * kSMs)
    gkr_gram<NFEAT, 16><<<dim3(std::min(chunks, (uint32_t)(4 * kSMs)), NFEAT / (16 * S::kGroups)),
                          S::kThreadsPer, 0, st>>>(cols, live, s, eq, X);
  else
    gkr_gram<NFEAT, 4><<<dim3(chunks, NFEAT / (4 * S::kGroups)), S::kThreadsPer, 0, st>>>(
        cols, live, s, eq, X);
  BZ_LAUNCH_CHECK();
}

static f128 eq_factor(f128 r, f128 z) { return gadd(gadd(mk(1, 0), r), z); }

// One layer's rounds: the transcript's side of round i from its two sums (at
// zero, or at one when the point's coordinate is zero, and at infinity).
struct LayerRounds {
  const f128 *point;
  f128 *next;
  uint32_t grind_bits;
  Transcript &ts;
  f128 eq_bound = mk(1, 0);

  f128 round(int i, f128 at_zero, f128 at_one, f128 at_inf) {
    const f128 z = point[i];
    f128 msg[2] = {gmul(eq_bound, gis_zero(z) ? at_one : at_zero), gmul(eq_bound, at_inf)};
    ts.prover_message(msg, 32);
    ts.grind("gkr/cubic/v1", grind_bits);
    const f128 r = ts.challenge_f128();
    next[i] = r;
    eq_bound = gmul(eq_bound, eq_factor(r, z));
    return r;
  }

  // k rounds from the 3^k point sums F (digit k - 1 of the index is coordinate
  // `top`); the challenges go to r.
  void from_points(std::vector<f128> &F, int top, int k, f128 *r) {
    f128 e[32];   // eq over the coordinates below the current one, at zeros and ones
    int at[32];   // and the index of that point
    size_t block = F.size() / 3;
    for (int t = 0; t < k; t++, block /= 3) {
      const int rest = k - 1 - t;
      e[0] = mk(1, 0);
      at[0] = 0;
      for (int q = 0, p = 1; q < rest; q++, p *= 3)
        for (int x = 0; x < 1 << q; x++) {
          const f128 one = gmul(e[x], point[top - k + 1 + q]);
          e[x | 1 << q] = one;
          e[x] = gadd(e[x], one);
          at[x | 1 << q] = at[x] + p;
        }
      f128 s[3];
      for (int d = 0; d < 3; d++) {
        wide a = wzero();
        for (int x = 0; x < 1 << rest; x++) wacc(a, gmul_wide(e[x], F[d * block + at[x]]));
        s[d] = greduce(a);
      }
      r[t] = round(top - t, s[0], s[1], s[2]);
      for (size_t x = 0; x < block; x++) {  // h0 + r (h1 + h0 + hinf) + r^2 hinf
        const f128 h0 = F[x], h1 = F[block + x], hi = F[2 * block + x];
        F[x] = gadd(h0, gmul(r[t], gadd(gadd(h0, h1), gadd(hi, gmul(r[t], hi)))));
      }
    }
  }

  // The remaining n rounds on tables of 2^n entries; leaves the bound pair.
  void from_tables(f128 *L, f128 *R, int n, const f128 *eq_prefix, f128 out[2]) {
    for (int i = n - 1; i >= 0; i--) {
      const size_t h = (size_t)1 << i;
      f128 sums[2];
      // eq_prefix + h: eq over the i coordinates below
      host_cubic_sums(eq_prefix + h, L, R, h, gis_zero(point[i]), sums);
      const f128 r = round(i, sums[0], sums[0], sums[1]);
      host_bind_high(L, h, r);
      host_bind_high(R, h, r);
    }
    out[0] = L[0];
    out[1] = R[0];
  }
};

constexpr size_t kGram0Words = 2 * 65 * 65, kGram1Words = 2 * 97 * 97;
size_t gkr_gram_words() { return kGram0Words + kGram1Words; }

f128 gkr_prove(const f128 *cols, int s, const f128 *images, const f128 *zeta, uint32_t grind_bits,
               Transcript &ts, GkrScratch &sc, cudaStream_t st_, f128 *point_out) {
  f128 point[kMaxPoint], next[kMaxPoint];
  for (int i = 0; i < s; i++) point[i] = zeta[i];
  int n = s;
  const size_t colmask = ((size_t)1 << s) - 1;
  const size_t live = sc.live_cols ? sc.live_cols : colmask + 1;
  f128 claim = mk(0, 0);
  KernelProbe &probe = KernelProbe::get();
  RoundChannel *ch = sc.channel;
  // BITZ_ROUND_TRACE=1 prints the host time of every device turn
  static const bool trace = getenv("BITZ_ROUND_TRACE") != nullptr;
  BZ_CUDA(cudaMemsetAsync(sc.acc, 0, 2 * (pow3(kPassMaxK) + 1) * sizeof(unsigned long long), st_));
  std::vector<EqHeap> heap(5);
  std::vector<uint64_t> words(kHandoverWords);
  std::vector<f128> F, L, R;
  BZ_CUDA(cudaMemsetAsync(sc.gram, 0, gkr_gram_words() * sizeof(unsigned long long), st_));
  for (int j = 6; j >= 0; j--) {
    // layers 0 and 1 have tables only over the columns, once their rows are bound
    f128 *c = j >= 2 ? sc.layer[j] : sc.bound;
    const size_t n_half = (size_t)1 << (j >= 2 ? n : s);
    for (int g = 0; g * kFacLog < n - 1 || g == 0; g++)
      heap[g].build(point + g * kFacLog, std::min(kFacLog, std::max(0, n - 1 - g * kFacLog)));
    for (int g = (n - 2) / kFacLog + 1; g < 5; g++) heap[g].v[1] = mk(1, 0);
    if ((j >= 2 ? n : s) - 2 > kEqLowLog) {  // a pass of this layer has more coordinates below it
      EqFactors<2> low;
      for (int g = 0; g < 2; g++) memcpy(low.f[g], heap[g].prefix(kFacLog), sizeof(f128) << kFacLog);
      gkr_eq_low<<<(1 << kEqLowLog) / kThreads, kThreads, 0, st_>>>(low, sc.eq_low);
      BZ_LAUNCH_CHECK();
    }
    LayerRounds rounds{point, next, grind_bits, ts};
    PassBind b{};
    int rem = n;  // coordinates not bound yet (b's are bound by the next pass)
    auto t_prev = std::chrono::steady_clock::now();
    auto mark = [&](const char *what) {
      if (!trace) return;
      const auto now = std::chrono::steady_clock::now();
      fprintf(stderr, "[gkr] layer %d %s, %d coordinates: %7.2f us\n", j, what, rem,
              std::chrono::duration<double, std::micro>(now - t_prev).count());
      t_prev = now;
    };
    if (j < 2) {  // the rounds over the row coordinates, from the bits
      const int k = 6 - j, points = pow3(k);
      unsigned long long *X = sc.gram + (j == 0 ? 0 : kGram0Words);
      if (j == 0)
        launch_gram<64>(cols, (uint32_t)live, s, heap.data(), X, st_);
      else
        launch_gram<96>(cols, (uint32_t)live, s, heap.data(), X, st_);
      const unsigned long long seq = ch->arm().seq;
      (j == 0 ? gkr_moments<0> : gkr_moments<1>)<<<16, 256, 0, st_>>>(
          X, images, sc.mid, ch->counter, ch->handover_dev, seq);
      BZ_LAUNCH_CHECK();
      ch->wait_handover(st_, seq, words.data(), 2 * points);
      mark("rows");
      F.resize(points);
      for (int p = 0; p < points; p++) F[p] = mk(words[2 * p], words[2 * p + 1]);
      f128 r[6];
      rounds.from_points(F, rem - 1, k, r);
      rem -= k;
      RowWeights eps{};  // r[t] bound row bit k - 1 - t
      eps.e[0] = mk(1, 0);
      for (int q = 0; q < k; q++)
        for (int x = 0; x < 1 << q; x++) {
          const f128 one = gmul(eps.e[x], r[k - 1 - q]);
          eps.e[x | 1 << q] = one;
          eps.e[x] = gadd(eps.e[x], one);
        }
      (j == 0 ? gkr_bound_rows<0> : gkr_bound_rows<1>)<<<grid_for(colmask + 1), kThreads, 0, st_>>>(
          cols, s, images, eps, c, c + n_half);
      BZ_LAUNCH_CHECK();
    }
    while (rem > kHostLog) {
      const int k = b.k == 0 && rem >= kFirstLog ? 2 : 3;
      const int log_m = rem - k;
      const size_t m = (size_t)1 << log_m;
      const uint32_t count = (uint32_t)(m > colmask ? (m >> s) * live : std::min(m, live));
      const int points = pow3(k);
      const bool probed = probe.on("gkr_pass");
      if (probed) probe.before(st_);
      const PassPost post{sc.acc, ch->counter, ch->handover_dev, ch->arm().seq};
      const int blocks = (k == 2 ? launch_pass<2> : launch_pass<3>)(
          c, n_half, log_m, b, heap.data(), sc.eq_low, colmask, (uint32_t)live, count, ch->pass_blocks,
          post, st_);
      if (probed) {
        // per live position: 2^(k+1) entries of the bound tables, each from
        // 2^kb read and one written (none written without a bind), 2^kb - 1
        // products through window tables each; the weight, 2^k products by it
        // and 3^k wide ones
        const double e = (double)count * (2 << k), in = (double)(1 << b.k);
        probe.after(st_, "gkr_pass", 16.0 * e * (in + (b.k ? 1.0 : 0.0)),
                    (double)count * ((1 << k) + 1), (double)count * points,
                    e * (in - 1));
      }
      ch->wait_handover(st_, post.seq, words.data(), 2 * (points + 1) * blocks);
      pass_combine(words.data(), 2 * (points + 1), blocks);
      mark("pass");
      F.resize(points);
      for (int p = 0; p < points; p++) F[p] = mk(words[2 * p], words[2 * p + 1]);
      // the padded positions' weights (all of them sum to one) at the points
      // of zeros and ones
      const f128 pad = mk(words[2 * points] ^ 1, words[2 * points + 1]);
      if (!gis_zero(pad))
        for (int x = 0; x < 1 << k; x++) {
          int p = 0;
          for (int q = k - 1; q >= 0; q--) p = 3 * p + ((x >> q) & 1);
          F[p] = gadd(F[p], pad);
        }
      rounds.from_points(F, rem - 1, k, b.r);
      b.k = k;
      rem -= k;
    }
    const int len = 1 << rem;
    const unsigned long long seq = ch->arm().seq;
    gkr_handover<<<(2 * len + kHandEntries - 1) / kHandEntries, kHandThreads, 0, st_>>>(
        c, n_half, len, b, ch->handover_dev, seq);
    BZ_LAUNCH_CHECK();
    if ((int)L.size() < len) L.resize(len), R.resize(len);
    ch->wait_handover(st_, seq, words.data(), 4 * len);
    mark("tables");
    for (int k = 0; k < len; k++) {
      L[k] = mk(words[2 * k], words[2 * k + 1]);
      R[k] = mk(words[2 * (len + k)], words[2 * (len + k) + 1]);
    }
    f128 lr[2];
    std::vector<f128> prefix((size_t)1 << std::max(1, rem));
    prefix[1] = mk(1, 0);
    for (int i = 0; i + 1 < rem; i++) eq_double(prefix.data() + ((size_t)1 << i), (size_t)1 << i, point[i]);
    rounds.from_tables(L.data(), R.data(), rem, prefix.data(), lr);
    ts.prover_message(lr, 32);
    const f128 t = ts.challenge_f128();
    next[n] = t;
    claim = gadd(lr[0], gmul(t, gadd(lr[1], lr[0])));
    n++;
    for (int i = 0; i < n; i++) point[i] = next[i];
    mark("host rounds");
  }
  for (int i = 0; i < n; i++) point_out[i] = point[i];
  return claim;
}

// Every kernel of this file, loaded when the process's first lane on a device
// is made (lane_bootstrap, context.cpp).
void preload_gkr_kernels() {
  load_kernels({(const void *)gkr_low_layers,
                (const void *)gkr_high_layers,
                (const void *)gkr_gram<64, 4>,
                (const void *)gkr_gram<64, 16>,
                (const void *)gkr_gram<96, 4>,
                (const void *)gkr_gram<96, 16>,
                (const void *)gkr_moments<0>,
                (const void *)gkr_moments<1>,
                (const void *)gkr_bound_rows<0>,
                (const void *)gkr_bound_rows<1>,
                (const void *)gkr_eq_low,
                (const void *)gkr_pass<2, false>,
                (const void *)gkr_pass<2, true>,
                (const void *)gkr_pass<3, false>,
                (const void *)gkr_pass<3, true>,
                (const void *)gkr_handover});
}

}  // namespace bz
