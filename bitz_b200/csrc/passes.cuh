// What the multi-round sumcheck passes share (GKR, post-GKR, Ligerito): several
// rounds go through the device at once, as the product polynomial's values at
// the points {0, 1, infinity}^K of the K coordinates to be bound next.
#pragma once
#include <vector>

#include "device.cuh"
#include "host_tail.hpp"

namespace bz {

constexpr int kPassThreads = 288;  // nine warps: the 27 points of a tile in three turns
constexpr int kPassMaxK = 3;
constexpr int kPassMaxX = 32;  // positions per tile

constexpr int pow3(int k) { return k == 0 ? 1 : 3 * pow3(k - 1); }

// The challenges that the next pass binds, the first one drawn in r[0].
struct PassBind {
  f128 r[kPassMaxK];
  int k;
};

// eq(x) over many coordinates as a product of NF factor tables, factor g over
// coordinates 7g .. 7g + 6. The host forms a layer's tables once (about 130
// products each) and they travel as a launch argument: no copy, no setup
// launch before the first pass.
constexpr int kFacLog = 7;
template <int NF>
struct EqFactors {
  f128 f[NF][1 << kFacLog];
};

// From eq over some coordinates at p[0, n) to eq over one more, z, at p[n, 3n).
inline void eq_double(f128 *p, size_t n, f128 z) {
  f128 *q = p + n;
  host_scale(p, z, n, q + n);
  for (size_t k = 0; k < n; k++) q[k] = gadd(p[k], q[k + n]);
}

// Prefix tables of eq over up to kFacLog coordinates: entries [2^i, 2^(i+1))
// hold eq over the first i of them.
struct EqHeap {
  f128 v[2 << kFacLog];
  void build(const f128 *z, int n) {
    v[1] = mk(1, 0);
    for (int i = 0; i < n; i++) eq_double(v + ((size_t)1 << i), (size_t)1 << i, z[i]);
  }
  const f128 *prefix(int n) const { return v + ((size_t)1 << n); }
};

// Where a pass sums and posts.
struct PassPost {
  unsigned long long *acc;       // zero before, zero after
  unsigned int *counter;         // finished blocks, likewise
  unsigned long long *handover;  // tagged slots
  unsigned long long seq;        // their publication
  int blocks = kSMs;             // the launch's tiles (pass_tile_log)
};

// k rounds of a quadratic sumcheck from its point sums F (the first round's
// coordinate is the top digit): `round` takes a message's (a0, a2) and returns
// the challenge.
template <class Round>
inline void quad_rounds(std::vector<f128> &F, int k, f128 *r, Round round) {
  size_t block = F.size() / 3;
  for (int t = 0; t < k; t++, block /= 3) {
    const int rest = k - 1 - t;
    f128 a0 = mk(0, 0), a2 = mk(0, 0);
    for (int x = 0; x < 1 << rest; x++) {
      size_t at = 0;
      for (int q = rest - 1; q >= 0; q--) at = 3 * at + ((x >> q) & 1);
      a0 = gadd(a0, F[at]);
      a2 = gadd(a2, F[2 * block + at]);
    }
    r[t] = round(a0, a2);
    for (size_t x = 0; x < block; x++) {  // h0 + r (h1 + h0 + hinf) + r^2 hinf
      const f128 h0 = F[x], h1 = F[block + x], hi = F[2 * block + x];
      F[x] = gadd(h0, gmul(r[t], gadd(gadd(h0, h1), gadd(hi, gmul(r[t], hi)))));
    }
  }
}

// A pass's tile for `count` positions, 2^lx of them: the largest that still
// makes `blocks` tiles. Wide tiles fill the turns (27 points of 32 positions
// are three per thread), narrow ones the chip. A lane proving alone wants a tile
// for every SM; lanes that share the GPU want few SMs each: 48 proofs on 24
// lanes take 18.3 ms with 148 tiles, 17.6 with 74, 17.2 with 32, 18.0 with 16.
// The line is drawn by the kind of lane, not by how many prove: a pooled lane at
// work alone takes 32 tiles too, which costs it 1 to 2 % (64 blocks 2.91 ms
// against 2.85 on the default lane, 201 6.53 against 6.46, 1024 22.5 against
// 22.4, the batch call's own thread included).
inline int pass_tile_log(uint32_t count, int blocks) {
  int lx = 5;
  while (lx > 2 && (count >> lx) < (uint32_t)blocks) lx--;
  return lx;
}
// Few blocks post their sums by themselves (the host adds them up) instead of
// through atomics and a last block: three trips to the L2 less, 1.4 us.
__host__ __device__ inline bool pass_direct(unsigned int grid, int words) {
  return grid * (unsigned int)words <= 1536u;
}
// Adds the blocks' words up into the first `words`.
inline void pass_combine(uint64_t *w, int words, int blocks) {
  for (int b = 1; b < blocks; b++)
    for (int k = 0; k < words; k++) w[k] ^= w[b * words + k];
}
inline unsigned int pass_grid(uint32_t count, int lx) {
  const uint32_t tiles = (count + (1u << lx) - 1) >> lx;
  return tiles < 1 ? 1 : tiles < 2u * kSMs ? tiles : 2u * kSMs;
}

#if defined(__CUDACC__)
// Products as calls: a pass is short for most sizes and starts with a cold
// instruction cache (a product inlined 40 times costs more to fetch than to
// run), and the larger ones are bound by the products themselves.
static __device__ __noinline__ wide pass_wide(f128 a, f128 b) { return gmul_wide(a, b); }
// (The lookups by the factor's words: a quarter of the code of the full unroll.)
static __device__ __noinline__ f128 pass_table(const MulTable *T, f128 b) {
  uint32_t w = (uint32_t)b.lo, w1 = (uint32_t)(b.lo >> 32), w2 = (uint32_t)b.hi,
           w3 = (uint32_t)(b.hi >> 32);
  uint64_t lo = 0, hi = 0;
#pragma unroll 1
  for (int i = 0; i < 4; i++) {
#pragma unroll
    for (int n = 0; n < 8; n++) {
      const uint32_t v = (w >> (4 * n)) & 15u;
      lo ^= T->lo[8 * i + n][v];
      hi ^= T->hi[8 * i + n][v];
    }
    w = w1;
    w1 = w2;
    w2 = w3;
  }
  return mk(lo, hi);
}
static __device__ __forceinline__ f128 pass_mul(f128 a, f128 b) { return greduce(pass_wide(a, b)); }

// The other entries of `n` windows whose single-bit entries are in place: every
// thread of the block takes part; the caller synchronises around it.
static __device__ __forceinline__ void fill_windows(uint64_t (*lo)[16], uint64_t (*hi)[16],
                                                    int n) {
  for (int u = threadIdx.x; u < n * 16; u += blockDim.x) {
    const int j = u >> 4, v = u & 15;
    if (v != 0 && (v & (v - 1)) == 0) continue;
    uint64_t a = 0, b = 0;
#pragma unroll
    for (int q = 0; q < 4; q++)
      if ((v >> q) & 1) {
        a ^= lo[j][1 << q];
        b ^= hi[j][1 << q];
      }
    lo[j][v] = a;
    hi[j][v] = b;
  }
}

// v X, reduced.
static __device__ __forceinline__ f128 times_x(f128 v) {
  return mk((v.lo << 1) ^ ((0 - (v.hi >> 63)) & 0x87), (v.hi << 1) | (v.lo >> 63));
}

// The window tables of r[0 .. k), every thread of the block taking part: a
// thread forms a window's four single-bit entries in registers and writes four
// entries of the window, so the build is one step without a barrier inside.
static __device__ __forceinline__ void pass_tables(MulTable *T, const f128 *r, int k) {
  for (int u = threadIdx.x; u < k * 128; u += blockDim.x) {
    const int t = u >> 7, j = (u >> 2) & 31, top = u & 3;
    const f128 v = r[t];
    const int s = (4 * j) & 63;
    const uint64_t w0 = v.lo << s, w1 = (v.hi << s) | ((v.lo >> 1) >> (63 - s)),
                   w2 = (v.hi >> 1) >> (63 - s);
    f128 b[4];
    b[0] = greduce(j >= 16 ? wide{0, w0, w1, w2} : wide{w0, w1, w2, 0});  // r X^(4j)
#pragma unroll
    for (int q = 1; q < 4; q++) b[q] = times_x(b[q - 1]);
    f128 e = mk(0, 0);
    if (top & 1) e = b[2];
    if (top & 2) e = gadd(e, b[3]);
    uint64_t *lo = T[t].lo[j] + 4 * top, *hi = T[t].hi[j] + 4 * top;
    const f128 e1 = gadd(e, b[0]), e2 = gadd(e, b[1]), e3 = gadd(e1, b[1]);
    lo[0] = e.lo, lo[1] = e1.lo, lo[2] = e2.lo, lo[3] = e3.lo;
    hi[0] = e.hi, hi[1] = e1.hi, hi[2] = e2.hi, hi[3] = e3.hi;
  }
  __syncthreads();
}

static __device__ __forceinline__ f128 bind2(const MulTable *T, f128 a, f128 b) {
  return gadd(a, pass_table(T, gadd(a, b)));
}

// 2^k entries in(0), in(1), ... bound at k challenges, the first one bound by
// index bit `first` (0: the lowest bit first; k - 1: the highest first).
template <bool kLowFirst, class In>
static __device__ __forceinline__ f128 pass_bind(In in, const MulTable *T, int k) {
  if (k == 0) return in(0);
  if (k == 1) return bind2(T, in(0), in(1));
  if (k == 2) {
    const f128 x[4] = {in(0), in(kLowFirst ? 1 : 2), in(kLowFirst ? 2 : 1), in(3)};
    const f128 a = bind2(T, x[0], x[1]), b = bind2(T, x[2], x[3]);
    return bind2(T + 1, a, b);
  }
  // pairs of the first challenge, in the order the second one joins them; all
  // loads before the first product
  f128 x[8];
#pragma unroll
  for (int i = 0; i < 8; i++) {
    constexpr int kLow[8] = {0, 1, 2, 3, 4, 5, 6, 7}, kHigh[8] = {0, 4, 2, 6, 1, 5, 3, 7};
    x[i] = in(kLowFirst ? kLow[i] : kHigh[i]);
  }
  const f128 a = bind2(T, x[0], x[1]), b = bind2(T, x[2], x[3]), ab = bind2(T + 1, a, b);
  const f128 c = bind2(T, x[4], x[5]), d = bind2(T, x[6], x[7]);
  return bind2(T + 2, ab, bind2(T + 1, c, d));
}

// The same by 2^(k-1) neighbouring lanes, lane q of them: one pair per lane,
// then joined by exchanges. Three products deep instead of seven, which took
// 11,900 cycles of a 64-block pass; it makes 12 lane products for 7, so only
// where a block has few entries. One call per level for both halves: the seven
// layers over 2^10 columns 393 -> 371 us. k >= 1, every lane of the warp.
template <bool kLowFirst, class In>
static __device__ __forceinline__ f128 pass_bind_lanes(In in, const MulTable *T, int k, int q) {
  const int g = 1 << (k - 1);
  f128 v = kLowFirst ? bind2(T, in(2 * q), in(2 * q + 1)) : bind2(T, in(q), in(q + g));
  for (int l = 1; l < k; l++) {
    const int m = kLowFirst ? 1 << (l - 1) : g >> l;
    const f128 o = mk(__shfl_xor_sync(0xffffffffu, v.lo, m), __shfl_xor_sync(0xffffffffu, v.hi, m));
    const bool upper = q & m;  // one call for both halves of the lanes
    v = bind2(T + l, upper ? o : v, upper ? v : o);
  }
  return v;
}
// Tiles up to this size (log) bind by lanes.
constexpr int kLaneTileLog = 3;

// Which block bits point p has at one and at infinity (the sum over the bit):
// digit i of p (base 3) is bit i of the block, or bit K - 1 - i when the lowest
// bit is bound first (the first round's coordinate is always the top digit).
template <int K, bool kLowFirst>
static __device__ __forceinline__ void point_bits(int p, int &one, int &inf) {
  one = inf = 0;
#pragma unroll
  for (int i = 0; i < K; i++) {
    const int d = p % 3, bit = kLowFirst ? K - 1 - i : i;
    p /= 3;
    one |= (d == 1) << bit;
    inf |= (d == 2) << bit;
  }
}

// A table's value at a point: blocks `stride` entries apart.
static __device__ __forceinline__ f128 point_value(const f128 *t, int stride, int one, int inf) {
  f128 v = t[one * stride];
  for (int sub = inf; sub; sub = (sub - 1) & inf) v = gadd(v, t[(one | sub) * stride]);
  return v;
}

// A pass's sums over the X lanes of each point: turn q of thread t has point
// (t + q kPassThreads) / X. Into acc, or, where every block posts by itself,
// to words 2 p and 2 p + 1 of the block's `words` handover words.
template <int kPoints, int kTurns>
static __device__ __forceinline__ void pass_reduce(const wide (&sum)[kTurns], int lx, int words,
                                                   bool direct, const PassPost &post) {
  const int X = 1 << lx;
#pragma unroll
  for (int q = 0; q < kTurns; q++) {
    const int u = threadIdx.x + q * kPassThreads, p = u >> lx;
    if ((u & ~31) >= kPoints << lx) break;  // the whole warp
    f128 v = greduce(sum[q]);
    for (int off = (X < 32 ? X : 32) >> 1; off > 0; off >>= 1) {
      v.lo ^= __shfl_xor_sync(0xffffffffu, v.lo, off);
      v.hi ^= __shfl_xor_sync(0xffffffffu, v.hi, off);
    }
    if (p < kPoints && (u & (X < 32 ? X - 1 : 31)) == 0) {
      if (direct) {
        handover_post(post.handover, post.seq, blockIdx.x * words + 2 * p, v.lo);
        handover_post(post.handover, post.seq, blockIdx.x * words + 2 * p + 1, v.hi);
      } else {
        atomicXor(post.acc + 2 * p, (unsigned long long)v.lo);
        atomicXor(post.acc + 2 * p + 1, (unsigned long long)v.hi);
      }
    }
  }
}

// Every thread calls it after its atomics: the last block to finish posts the
// first `words` words of acc (and clears them) as handover publication seq.
static __device__ __forceinline__ void pass_publish(unsigned long long *acc, int words,
                                                    unsigned int *counter,
                                                    unsigned long long *handover,
                                                    unsigned long long seq) {
  __shared__ bool last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    last = atomicAdd(counter, 1u) == gridDim.x - 1;
    __threadfence();
  }
  __syncthreads();
  if (!last) return;
  for (int k = threadIdx.x; k < words; k += blockDim.x)
    handover_post(handover, seq, k, atomicExch(acc + k, 0ull));
  if (threadIdx.x == 0) *counter = 0;
}
#endif

}  // namespace bz
