// The post-GKR sumcheck (crates/post_gkr/src/lib.rs:121-148, sumcheck.rs:98-215):
// from the inner-product claim <rows (x) cols, f> = target over the committed
// bits f to an evaluation claim MLE[f](rho) = v.
//
// Rounds bind the lowest coordinate first: first the row coordinates, then the
// columns'. Every message is a sum of products that is linear in f, so the
// tables are as small as the claim's structure allows, not 2^m entries:
//
// - With more than one column, the rows' rounds run on rows[k] and
//   Y[k] = sum over c of cols[c] f[c, k] (2^log_rows entries each). Once the
//   rows are bound, the columns' rounds run on cols[c] and
//   V[c] = sum over k of eq(r, k) f[c, k], scaled by the bound row weight.
// - With one column, f stays bits through the first three rounds: their sums
//   need only the 64 sums of row weights by position and bit position within
//   groups of eight, and V after the three binds is a 256-entry table of the
//   group's byte.
//
// Rounds go through the device in passes of up to three (passes.cuh), and the
// last 2^kHostLog entries to the host.
#include <cstring>
#include <vector>

#include "context.hpp"
#include "host_tail.hpp"
#include "post_gkr.hpp"

namespace bz {

// Tables of this many entries or fewer go to the host.
constexpr int kHostLog = 10;
static_assert(4 << kHostLog <= kHandoverWords, "the last tables fit one handover");

// Y for few columns: a thread per row, its bit of every column.
__global__ void __launch_bounds__(kThreads) pg_row_sums(const uint32_t *__restrict__ bits,
                                                        int log_rows, int log_cols,
                                                        const f128 *__restrict__ cols,
                                                        f128 *__restrict__ Y) {
  const size_t n = (size_t)1 << log_rows;
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n;
       k += (size_t)gridDim.x * blockDim.x) {
    f128 y = mk(0, 0);
    for (int c = 0; c < 1 << log_cols; c++) {
      const uint64_t m = 0 - (uint64_t)((bits[((size_t)c << (log_rows - 5)) + (k >> 5)] >> (k & 31)) & 1);
      const f128 w = ld(cols + c);
      y.lo ^= w.lo & m;
      y.hi ^= w.hi & m;
    }
    st(Y + k, y);
  }
}

// Y for 128 columns or more: over 128 columns a row's sum is one product
// through a window table whose single-bit entries are the columns' weights,
// with the row's bits of those columns (transposed by ballots) as the other
// factor: 128 lookup products per 128 words of f, instead of 2^14 masked adds.
// Y is zeroed before; blockIdx.y strides over the words of a column.
__global__ void __launch_bounds__(kThreads) pg_row_sums_wide(const f128 *__restrict__ packed,
                                                             int log_words, int log_cols,
                                                             const f128 *__restrict__ cols,
                                                             f128 *__restrict__ Y) {
  __shared__ MulTable T;
  __shared__ uint4 rows[128];
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const size_t words = (size_t)1 << log_words, chunks = (size_t)1 << (log_cols - 7);
  f128 sum = mk(0, 0);
  auto add = [&](size_t row, f128 v) {
    unsigned long long *y = reinterpret_cast<unsigned long long *>(Y + row);
    if (v.lo) atomicXor(y, (unsigned long long)v.lo);
    if (v.hi) atomicXor(y + 1, (unsigned long long)v.hi);
  };
  for (size_t ch = blockIdx.x; ch < chunks; ch += gridDim.x) {
    if (t < 128) {
      const f128 w = ld(cols + ch * 128 + t);
      T.lo[t >> 2][1 << (t & 3)] = w.lo;
      T.hi[t >> 2][1 << (t & 3)] = w.hi;
    }
    __syncthreads();
    fill_windows(T.lo, T.hi, 32);
    for (size_t b = blockIdx.y; b < words; b += gridDim.y) {
      const f128 w = ld(packed + ((ch * 128 + (warp & 3) * 32 + lane) << log_words) + b);
      const uint64_t half = warp < 4 ? w.lo : w.hi;
      uint32_t r0 = 0, r1 = 0;
#pragma unroll 8
      for (int r = 0; r < 32; r++) {
        const uint32_t a = __ballot_sync(0xffffffffu, (half >> r) & 1);
        const uint32_t c = __ballot_sync(0xffffffffu, (half >> (r + 32)) & 1);
        if (lane == r) r0 = a, r1 = c;
      }
      uint32_t *out = reinterpret_cast<uint32_t *>(rows + (warp < 4 ? 0 : 64));
      out[4 * lane + (warp & 3)] = r0;
      out[4 * (lane + 32) + (warp & 3)] = r1;
      __syncthreads();
      if (t < 128) {
        const uint4 m = rows[t];
        const f128 v = pass_table(&T, mk((uint64_t)m.x | (uint64_t)m.y << 32,
                                         (uint64_t)m.z | (uint64_t)m.w << 32));
        if (words == 1)
          sum = gadd(sum, v);
        else
          add(b * 128 + t, v);
      }
      __syncthreads();  // the rows and the table before the next ones
    }
  }
  if (words == 1 && t < 128) add(t, sum);
}

// The first three rounds of a one-column claim: H[a][b], the sum over the groups
// of eight rows of weight a where bit b is set (64 sums; every point of the
// three rounds is a sum of them), and the column's weight behind them. One lane
// per row: the kernel reads each weight once, coalesced, and makes eight masked
// adds; stretches of 32 zero bits are skipped (the padding of small
// statements). 2^23 rows: 134 MB, 31 us; the first message, first fold and two
// rounds that it stands for took 600 us.
__global__ void __launch_bounds__(kThreads) pg_bits(const f128 *__restrict__ rows, int log_rows,
                                                    const f128 *__restrict__ cols,
                                                    const uint32_t *__restrict__ bits,
                                                    unsigned long long *acc, unsigned int *counter,
                                                    unsigned long long *handover,
                                                    unsigned long long seq) {
  __shared__ unsigned long long sums[128];
  const int t = threadIdx.x, lane = t & 31;
  if (t < 128) sums[t] = 0;
  __syncthreads();
  const size_t n = (size_t)1 << (log_rows - 5);  // words of 32 rows
  const size_t warps = (size_t)gridDim.x * (kThreads / 32);
  f128 h[8];
#pragma unroll
  for (int b = 0; b < 8; b++) h[b] = mk(0, 0);
#pragma unroll 4
  for (size_t k = blockIdx.x * (size_t)(kThreads / 32) + (t >> 5); k < n; k += warps) {
    const uint32_t word = __ldg(bits + k);
    if (!word) continue;
    const f128 w = ld(rows + 32 * k + lane);
    const uint32_t byte = word >> (lane & 24);
#pragma unroll
    for (int b = 0; b < 8; b++) {
      const uint64_t m = 0 - (uint64_t)((byte >> b) & 1);
      h[b].lo ^= w.lo & m;
      h[b].hi ^= w.hi & m;
    }
  }
#pragma unroll
  for (int b = 0; b < 8; b++) {
    for (int off = 8; off < 32; off <<= 1) {
      h[b].lo ^= __shfl_xor_sync(0xffffffffu, h[b].lo, off);
      h[b].hi ^= __shfl_xor_sync(0xffffffffu, h[b].hi, off);
    }
    if (lane < 8) {
      atomicXor(&sums[2 * (8 * lane + b)], (unsigned long long)h[b].lo);
      atomicXor(&sums[2 * (8 * lane + b) + 1], (unsigned long long)h[b].hi);
    }
  }
  __syncthreads();
  if (t < 128 && sums[t]) atomicXor(acc + t, sums[t]);
  if (blockIdx.x == 0 && t == 0) {
    const f128 c = ld(cols);
    atomicXor(acc + 128, (unsigned long long)c.lo);
    atomicXor(acc + 129, (unsigned long long)c.hi);
  }
  pass_publish(acc, 130, counter, handover, seq);
}

// The eq weights of a group of eight bits at the three bound challenges.
struct BitWeights {
  f128 e[8];
};

// V's values by byte, every thread of the block taking part.
static __device__ __forceinline__ void bit_values(f128 *V8, const BitWeights &e) {
  for (int v = threadIdx.x; v < 256; v += blockDim.x) {
    f128 s = mk(0, 0);
#pragma unroll
    for (int b = 0; b < 8; b++)
      if ((v >> b) & 1) s = gadd(s, e.e[b]);
    V8[v] = s;
  }
}

static __device__ __forceinline__ f128 bind_low(const f128 *tab, size_t o, const MulTable *T,
                                                int k) {
  const f128 *p = tab + (o << k);
  return pass_bind<true>([&](int j) { return ld(p + j); }, T, k);
}

// One pass over the low K coordinates of W and V (n entries each after the binds
// of b, written to w_out and v_out when there are any): the sums of W V at the
// 3^K points, posted as handover publication seq. A block works tiles of
// X = 2^lx groups of 2^K entries: the 2 2^K X bound entries one per thread into
// shared memory (rows of X + 1, so that neither the writes along a group nor
// the reads along a row conflict), then the 3^K X wide products. With kBits, V
// comes from f's bytes (b.k = 3). Binding is 2^k - 1 products through window
// tables per entry and table (bound by shared memory, 72 G/s over the GPU), the
// points 3.4 wide products per entry (45 G/s).
template <int K, bool kBits>
__global__ void __launch_bounds__(kPassThreads, 2) pg_pass(
    const f128 *__restrict__ w_in, const f128 *__restrict__ v_in, f128 *__restrict__ w_out,
    f128 *__restrict__ v_out, uint32_t count, PassBind b, const __grid_constant__ BitWeights e8,
    int lx, PassPost post) {
  constexpr int kPoints = pow3(K), kBlocks = 1 << K;
  constexpr int kTurns = (kPoints * kPassMaxX + kPassThreads - 1) / kPassThreads;
  __shared__ MulTable T[kPassMaxK];
  __shared__ f128 G[kBlocks * (kPassMaxX + 1)], R[kBlocks * (kPassMaxX + 1)];
  __shared__ f128 V8[kBits ? 256 : 1];
  const int t = threadIdx.x, X = 1 << lx;
  if (kBits) bit_values(V8, e8);
  pass_tables(T, b.r, b.k);
  wide sum[kTurns];
#pragma unroll
  for (int q = 0; q < kTurns; q++) sum[q] = wzero();
  for (uint32_t i0 = blockIdx.x << lx; i0 < count; i0 += gridDim.x << lx) {
    const int half = kBlocks << lx;
    const bool lanes = b.k && lx <= kLaneTileLog;
    if (lanes) {
      const int gl = b.k - 1, total = (kBits ? half : 2 * half) << gl;
      for (int u = t; u < total; u += kPassThreads) {
        const int at = u >> gl, q = u & ((1 << gl) - 1);
        const bool right = at >= half;
        const int slot = at & (half - 1), x = slot >> K;
        const bool in = i0 + x < count;
        const size_t o = ((size_t)i0 << K) + slot;
        const f128 *p = (right ? v_in : w_in) + (o << b.k);
        const f128 v = pass_bind_lanes<true>([&](int j) { return in ? ld(p + j) : mk(0, 0); }, T,
                                             b.k, q);
        if (q) continue;
        if (in) st((right ? v_out : w_out) + o, v);
        (right ? R : G)[(slot & (kBlocks - 1)) * (X + 1) + x] = v;
      }
    }
    // one thread per entry (with lanes, only V's bytes are left)
    for (int u = lanes ? t + half : t; u < 2 * half && (!lanes || kBits); u += kPassThreads) {
      const bool right = u >= half;
      const int slot = right ? u - half : u, x = slot >> K, a = slot & (kBlocks - 1);
      f128 v = mk(0, 0);
      if (i0 + x < count) {
        const size_t o = ((size_t)i0 << K) + slot;
        if (kBits && right)
          v = V8[reinterpret_cast<const uint8_t *>(v_in)[o]];
        else
          v = bind_low(right ? v_in : w_in, o, T, b.k);
        if (b.k) st((right ? v_out : w_out) + o, v);
      }
      (right ? R : G)[a * (X + 1) + x] = v;
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kTurns; q++) {
      const int u = t + q * kPassThreads;
      if (u < kPoints << lx) {
        int one, inf;
        point_bits<K, true>(u >> lx, one, inf);
        const int x = u & (X - 1);
        wacc(sum[q], pass_wide(point_value(G + x, X + 1, one, inf),
                               point_value(R + x, X + 1, one, inf)));
      }
    }
    __syncthreads();  // the tile's tables before the next tile's
  }
  const bool direct = pass_direct(gridDim.x, 2 * kPoints);
  pass_reduce<kPoints, kTurns>(sum, lx, 2 * kPoints, direct, post);
  if (!direct) pass_publish(post.acc, 2 * kPoints, post.counter, post.handover, post.seq);
}

// The binds of b alone: n entries of each table.
__global__ void __launch_bounds__(kThreads) pg_bind(const f128 *__restrict__ w_in,
                                                    const f128 *__restrict__ v_in,
                                                    f128 *__restrict__ w_out,
                                                    f128 *__restrict__ v_out, size_t n,
                                                    PassBind b) {
  __shared__ MulTable T[kPassMaxK];
  pass_tables(T, b.r, b.k);
  const size_t total = v_in ? 2 * n : n;
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < total;
       k += (size_t)gridDim.x * blockDim.x) {
    const bool right = k >= n;
    const size_t o = right ? k - n : k;
    st((right ? v_out : w_out) + o, bind_low(right ? v_in : w_in, o, T, b.k));
  }
}

// The last tables to the host: W, then V, of n entries each after the binds of b.
constexpr int kHandThreads = 256, kHandEntries = 64;  // up to four lanes per entry
template <bool kBits>
__global__ void __launch_bounds__(kHandThreads) pg_handover(const f128 *__restrict__ w_in,
                                                            const f128 *__restrict__ v_in, int n,
                                                            PassBind b, BitWeights e8,
                                                            unsigned long long *handover,
                                                            unsigned long long seq) {
  __shared__ MulTable T[kPassMaxK];
  __shared__ f128 V8[kBits ? 256 : 1];
  if (kBits) bit_values(V8, e8);
  pass_tables(T, b.r, b.k);
  const int gl = b.k > 1 ? b.k - 1 : 0, q = threadIdx.x & ((1 << gl) - 1);
  if (threadIdx.x >> 5 >= (kHandEntries << gl) >> 5) return;  // whole warps
  const int k = blockIdx.x * kHandEntries + (threadIdx.x >> gl);
  const f128 *at = k < n ? w_in + ((size_t)k << b.k) : v_in + ((size_t)(k - n) << b.k);
  const bool byte = kBits && k >= n;
  auto in = [&](int j) { return k < 2 * n && !byte ? ld(at + j) : mk(0, 0); };
  f128 v = b.k ? pass_bind_lanes<true>(in, T, b.k, q) : in(0);
  if (q || k >= 2 * n) return;
  if (byte) v = V8[reinterpret_cast<const uint8_t *>(v_in)[k - n]];
  handover_post(handover, seq, 2 * k, v.lo);
  handover_post(handover, seq, 2 * k + 1, v.hi);
}

// V over the columns once the rows are bound: word b of column c is one product
// through the window table of the eq weights of 128 rows, times the weight of
// the word; a column's words are neighbouring lanes. V is zeroed before when a
// column has more than 32 words.
__global__ void __launch_bounds__(kThreads) pg_bound_cols(const f128 *__restrict__ packed,
                                                          int log_words, size_t total,
                                                          const __grid_constant__ EqFactors<5> eq,
                                                          f128 *__restrict__ V) {
  __shared__ MulTable T;
  const int t = threadIdx.x;
  if (t < 128) {
    T.lo[t >> 2][1 << (t & 3)] = eq.f[0][t].lo;
    T.hi[t >> 2][1 << (t & 3)] = eq.f[0][t].hi;
  }
  __syncthreads();
  fill_windows(T.lo, T.hi, 32);
  __syncthreads();
  const size_t words = (size_t)1 << log_words;
  const int seg = words < 32 ? (int)words : 32;
  for (size_t base = blockIdx.x * (size_t)kThreads; base < total;
       base += (size_t)gridDim.x * kThreads) {
    const size_t e = base + t;
    f128 v = mk(0, 0);
    if (e < total) {
      v = pass_table(&T, ld(packed + e));
      const size_t b = e & (words - 1);
#pragma unroll 1
      for (int g = 1; g < 5 && (g - 1) * kFacLog < log_words; g++)
        v = pass_mul(v, eq.f[g][(b >> ((g - 1) * kFacLog)) & ((1 << kFacLog) - 1)]);
    }
    for (int off = seg >> 1; off > 0; off >>= 1) {
      v.lo ^= __shfl_xor_sync(0xffffffffu, v.lo, off);
      v.hi ^= __shfl_xor_sync(0xffffffffu, v.hi, off);
    }
    if (e >= total || (t & (seg - 1))) continue;
    f128 *out = V + (e >> log_words);
    if (words <= 32) {
      st(out, v);
    } else {
      atomicXor(reinterpret_cast<unsigned long long *>(out), (unsigned long long)v.lo);
      atomicXor(reinterpret_cast<unsigned long long *>(out) + 1, (unsigned long long)v.hi);
    }
  }
}

// Returns how many blocks post sums of their own.
template <int K, bool kBits>
static int launch_quad(const f128 *w, const f128 *v, f128 *w2, f128 *v2, size_t n,
                        const PassBind &b, const BitWeights &e8, const PassPost &post,
                        cudaStream_t s) {
  const uint32_t count = (uint32_t)(n >> K);
  const int lx = pass_tile_log(count, post.blocks);
  const unsigned int grid = pass_grid(count, lx);
  pg_pass<K, kBits><<<grid, kPassThreads, 0, s>>>(w, v, w2, v2, count, b, e8, lx, post);
  BZ_LAUNCH_CHECK();
  return pass_direct(grid, 2 * pow3(K)) ? (int)grid : 1;
}

static int quad_pass_from(bool bits, int k, const f128 *w, const f128 *v, f128 *w2, f128 *v2,
                           size_t n, const PassBind &b, const BitWeights &e8,
                           const PassPost &post, cudaStream_t s) {
  KernelProbe &probe = KernelProbe::get();
  const bool probed = probe.on("pg_pass");
  if (probed) probe.before(s);
  const auto launch = bits     ? launch_quad<3, true>
                      : k == 3 ? launch_quad<3, false>
                      : k == 2 ? launch_quad<2, false>
                               : launch_quad<1, false>;
  const int blocks = launch(w, v, w2, v2, n, b, e8, post, s);
  if (probed) {
    // an entry of each table comes from 2^kb (a byte of f for V with bits)
    // and is written when there is a bind; 2^kb - 1 products through window
    // tables each, 3^k wide products per 2^k entries
    const double in = (double)(1 << b.k), tabs = bits ? 1 : 2;
    probe.after(s, "pg_pass",
                (double)n * (16.0 * (tabs * in + (b.k ? 2.0 : 0.0)) + (bits ? 1.0 : 0.0)), 0.0,
                (double)(n >> k) * pow3(k), tabs * (double)n * (in - 1));
  }
  return blocks;
}

int quad_pass(int k, const f128 *w, const f128 *v, f128 *w2, f128 *v2, size_t n,
               const PassBind &b, const PassPost &post, cudaStream_t s) {
  return quad_pass_from(false, k, w, v, w2, v2, n, b, BitWeights{}, post, s);
}

void quad_bind(const f128 *w, const f128 *v, f128 *w2, f128 *v2, size_t n, const PassBind &b,
               cudaStream_t s) {
  pg_bind<<<grid_for(v ? 2 * n : n), kThreads, 0, s>>>(w, v, w2, v2, n, b);
  BZ_LAUNCH_CHECK();
}

// h' = p(rho) with a1 = h + a2 (lib.rs:320-323).
static f128 advance(f128 claim, f128 a0, f128 a2, f128 r) {
  return gadd(a0, gmul(r, gadd(gadd(claim, a2), gmul(r, a2))));
}

// The sumcheck's transcript side and the tables' way through the passes.
struct PostGkrRun {
  const PostGkrArgs &a;
  Transcript &ts;
  PostGkrScratch &sc;
  cudaStream_t s;
  f128 *point;
  f128 claim;
  f128 scale = mk(1, 0);  // of the tables' products
  int done = 0;           // rounds
  std::vector<uint64_t> words = std::vector<uint64_t>(kHandoverWords);
  std::vector<f128> F, W, V;

  // Where the next pass posts, and its words once they are there.
  PassPost arm() {
    if (sc.channel)
      return PassPost{sc.acc, sc.channel->counter, sc.channel->handover_dev,
                      sc.channel->arm().seq, sc.channel->pass_blocks};
    return PassPost{sc.acc, sc.counter, sc.handover, ++*sc.seq, kSMs};
  }
  void wait(const PassPost &post, int n) {
    if (sc.channel) {
      sc.channel->wait_handover(s, post.seq, words.data(), n);
      return;
    }
    std::vector<unsigned long long> slots(2 * (size_t)n);
    BZ_CUDA(cudaMemcpyAsync(slots.data(), sc.handover, 16 * (size_t)n, cudaMemcpyDeviceToHost, s));
    BZ_CUDA(stream_wait(s));
    for (int k = 0; k < 2 * n; k++)
      if (slots[k] >> 32 != (post.seq & 0xffffffffull))
        throw CudaError("a sumcheck pass ended without its sums");
    for (int k = 0; k < n; k++) words[k] = (slots[2 * k] & 0xffffffffull) | (slots[2 * k + 1] << 32);
  }

  f128 round(f128 a0, f128 a2) {
    a0 = gmul(scale, a0);
    a2 = gmul(scale, a2);
    uint64_t msg[4] = {a0.lo, a0.hi, a2.lo, a2.hi};
    ts.prover_message(msg, 32);
    ts.grind("bitz/pcs/sumcheck/v1", a.grind_bits);
    const f128 r = ts.challenge_f128();
    claim = advance(claim, a0, a2, r);
    point[done++] = r;
    return r;
  }

  // Before the first round: the weighted sum must be the target.
  bool claim_holds(f128 total) {
    total = gmul(scale, total);
    if (done > 0 || geq(total, a.target)) return true;
    sc.claim_seen = total;
    return false;
  }

  // k rounds from the point sums in F.
  bool from_points(int k, f128 *r) {
    f128 total = mk(0, 0);
    for (int x = 0; x < 1 << k; x++) {
      int p = 0;
      for (int q = k - 1; q >= 0; q--) p = 3 * p + ((x >> q) & 1);
      total = gadd(total, F[p]);
    }
    if (!claim_holds(total)) return false;
    quad_rounds(F, k, r, [&](f128 a0, f128 a2) { return round(a0, a2); });
    return true;
  }

  // All rounds of tables (w, v) of 2^rem entries, or of their bound form when b
  // has challenges; leaves the bound pair. `set` is the buffer pair the first
  // bound tables go to.
  int tables(const f128 *w, const f128 *v, bool bits, int rem, PassBind b, BitWeights e8, int set,
             f128 out[2]) {
    f128 *bufs[2][2] = {{sc.w0, sc.v0}, {sc.w1, sc.v1}};
    while (rem > kHostLog) {
      // a first pass binds nothing: two rounds of it make 2.25 products per
      // entry, three 3.4, and above 2^17 entries the products are the cost
      const int k = b.k == 0 && rem >= 17 ? 2 : 3;
      const PassPost post = arm();
      const int blocks = quad_pass_from(bits, k, w, v, bufs[set][0], bufs[set][1], (size_t)1 << rem,
                                        b, e8, post, s);
      if (b.k) {
        w = bufs[set][0];
        v = bufs[set][1];
        set ^= 1;
        bits = false;
      }
      wait(post, 2 * pow3(k) * blocks);
      pass_combine(words.data(), 2 * pow3(k), blocks);
      F.resize(pow3(k));
      for (int p = 0; p < pow3(k); p++) F[p] = mk(words[2 * p], words[2 * p + 1]);
      if (!from_points(k, b.r)) return BZ_ERR_CLAIM;
      b.k = k;
      rem -= k;
    }
    const int n = 1 << rem;
    const PassPost post = arm();
    (bits ? pg_handover<true> : pg_handover<false>)<<<(2 * n + kHandEntries - 1) / kHandEntries,
                                                     kHandThreads, 0, s>>>(
        w, v, n, b, e8, post.handover, post.seq);
    BZ_LAUNCH_CHECK();
    wait(post, 4 * n);
    W.resize(n);
    V.resize(n);
    wide total = wzero();
    for (int k = 0; k < n; k++) {
      W[k] = mk(words[2 * k], words[2 * k + 1]);
      V[k] = mk(words[2 * (n + k)], words[2 * (n + k) + 1]);
      if (done == 0) wacc(total, gmul_wide(W[k], V[k]));
    }
    if (!claim_holds(greduce(total))) return BZ_ERR_CLAIM;
    for (int len = n / 2; len > 0; len /= 2) {
      f128 sums[2];
      host_quad_sums(W.data(), V.data(), len, sums);
      const f128 r = round(sums[0], sums[1]);
      host_bind_low(W.data(), len, r);
      host_bind_low(V.data(), len, r);
    }
    out[0] = W[0];
    out[1] = V[0];
    return BZ_OK;
  }

  // One column: the first three rounds from f's bits.
  int one_column(f128 out[2]) {
    const PassPost post = arm();
    const uint32_t *bits = reinterpret_cast<const uint32_t *>(a.packed);
    pg_bits<<<grid_for((size_t)1 << a.log_rows, 4 * kThreads), kThreads, 0, s>>>(
        a.rows, a.log_rows, a.cols, bits, post.acc, post.counter, post.handover, post.seq);
    BZ_LAUNCH_CHECK();
    wait(post, 130);
    scale = mk(words[128], words[129]);
    F.assign(27, mk(0, 0));
    for (int p = 0; p < 27; p++) {  // H over the positions each point takes in
      int one = 0, inf = 0;
      for (int i = 0, q = p; i < 3; i++, q /= 3) {
        one |= (q % 3 == 1) << (2 - i);
        inf |= (q % 3 == 2) << (2 - i);
      }
      for (int x = 0; x < 8; x++)
        for (int y = 0; y < 8; y++)
          if ((x & ~inf) == one && (y & ~inf) == one)
            F[p] = gadd(F[p], mk(words[2 * (8 * x + y)], words[2 * (8 * x + y) + 1]));
    }
    PassBind b;
    if (!from_points(3, b.r)) return BZ_ERR_CLAIM;
    b.k = 3;
    BitWeights e8;
    e8.e[0] = mk(1, 0);
    for (int q = 0; q < 3; q++)
      for (int x = 0; x < 1 << q; x++) {
        const f128 one = gmul(e8.e[x], b.r[q]);
        e8.e[x | 1 << q] = one;
        e8.e[x] = gadd(e8.e[x], one);
      }
    return tables(a.rows, a.packed, true, a.log_rows - 3, b, e8, 1, out);
  }

  int columns(f128 out[2]) {
    const int log_words = a.log_rows - 7;
    f128 *Y = sc.v0;
    if (a.log_cols < 7) {
      pg_row_sums<<<grid_for((size_t)1 << a.log_rows), kThreads, 0, s>>>(
          reinterpret_cast<const uint32_t *>(a.packed), a.log_rows, a.log_cols, a.cols, Y);
    } else {
      BZ_CUDA(cudaMemsetAsync(Y, 0, sizeof(f128) << a.log_rows, s));
      const size_t chunks = (size_t)1 << (a.log_cols - 7), words = (size_t)1 << log_words;
      const unsigned int x = (unsigned int)std::min(chunks, (size_t)kSMs * 4);
      const unsigned int y = (unsigned int)std::min(words, std::max((size_t)1, (size_t)kSMs * 4 / x));
      pg_row_sums_wide<<<dim3(x, y), kThreads, 0, s>>>(a.packed, log_words, a.log_cols, a.cols, Y);
    }
    BZ_LAUNCH_CHECK();
    f128 pair[2];
    if (int rc = tables(a.rows, Y, false, a.log_rows, PassBind{}, BitWeights{}, 1, pair)) return rc;
    scale = pair[0];
    EqFactors<5> eq{};
    {
      EqHeap heap;
      for (int g = 0; g < 5; g++) {
        const int n = std::min(kFacLog, std::max(0, a.log_rows - g * kFacLog));
        heap.build(point + g * kFacLog, n);
        memcpy(eq.f[g], heap.prefix(n), sizeof(f128) << n);
      }
    }
    f128 *V = sc.v0;
    const size_t total = (size_t)1 << (log_words + a.log_cols);
    if (log_words > 5) BZ_CUDA(cudaMemsetAsync(V, 0, sizeof(f128) << a.log_cols, s));
    pg_bound_cols<<<grid_for(total), kThreads, 0, s>>>(a.packed, log_words, total, eq, V);
    BZ_LAUNCH_CHECK();
    return tables(a.cols, V, false, a.log_cols, PassBind{}, BitWeights{}, 1, out);
  }
};

int post_gkr_prove(const PostGkrArgs &a, Transcript &ts, PostGkrScratch &sc, cudaStream_t s,
                   f128 *point_out, f128 *value_out) {
  const int m = a.log_rows + a.log_cols;
  if (sc.capacity < (size_t)1 << (m - 1)) return BZ_ERR_SCRATCH;
  if (a.log_rows > 5 * kFacLog) return BZ_ERR_SCRATCH;
  BZ_CUDA(cudaMemsetAsync(sc.acc, 0, 130 * sizeof(unsigned long long), s));
  if (!sc.channel) BZ_CUDA(cudaMemsetAsync(sc.counter, 0, sizeof(unsigned int), s));
  PostGkrRun run{a, ts, sc, s, point_out, a.target};
  f128 fin[2];
  const int rc = a.log_cols == 0 ? run.one_column(fin) : run.columns(fin);
  if (rc) return rc;
  *value_out = fin[1];
  ts.prover_f128(fin[1]);
  return geq(gmul(run.scale, gmul(fin[0], fin[1])), run.claim) ? BZ_OK : BZ_ERR_INTERNAL;
}

// Every kernel of this file, loaded when the process's first lane on a device
// is made (lane_bootstrap, context.cpp).
void preload_post_gkr_kernels() {
  load_kernels({(const void *)pg_row_sums,
                (const void *)pg_row_sums_wide,
                (const void *)pg_bits,
                (const void *)pg_pass<1, false>,
                (const void *)pg_pass<2, false>,
                (const void *)pg_pass<3, false>,
                (const void *)pg_pass<3, true>,
                (const void *)pg_bind,
                (const void *)pg_handover<false>,
                (const void *)pg_handover<true>,
                (const void *)pg_bound_cols});
}

}  // namespace bz
