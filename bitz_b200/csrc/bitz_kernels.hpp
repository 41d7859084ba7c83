// Host interface of the BitZ opening and PCS kernels.
#pragma once
#include <cuda_runtime.h>

#include "device.cuh"
#include "passes.cuh"
#include "transcript.hpp"

namespace bz {

constexpr int kMaxRsDim = 40;  // largest additive-FFT dimension (row bits of a codeword)

// Small tables travel as launch arguments: no copy to wait for.
struct RowExponents {
  u128 e[128];
};
struct RowWeights128 {
  f128 v[128];
};

// The columns' folds; with a comb table, the exponents' powers into images too.
void fold_columns(const f128 *cols, size_t ncols, const RowExponents &exps, u128 *folds,
                  const f128 *table, f128 *images, cudaStream_t s);
void comb_pow(const f128 *table, const u128 *exps, int n, f128 *out, cudaStream_t s);
// weights[c - 1] = sum over the rows r of column c of u1[r & 127] u2[r >> 7]
// (rows below `rows` <= 2^(7 + log_u2)); column 0 into w0. The row table is
// formed once in `dense` (2^(7 + log_u2) entries) and the columns gather it.
void mt_transpose(const uint32_t *off, const uint32_t *row, size_t ncols, const RowWeights128 &u1,
                  const f128 *u2, f128 *weights, size_t padded, f128 *w0, cudaStream_t s,
                  f128 *dense, int log_u2, size_t rows);
// The non-root chaining value of nchunks (a power of two) whole 1 KiB chunks,
// and the 16 bytes at `extra` (device, may be null) into extra_out. ch: the
// lane's channel (null: a copy and a stream synchronisation).
void blake3_tree_cv(const uint8_t *data, size_t nchunks, const uint32_t key[8], uint32_t flags,
                    uint32_t *scratch, uint32_t cv_out[8], cudaStream_t s, RoundChannel *ch,
                    const f128 *extra, f128 *extra_out);
// The 128 claims, posted as 256 words.
void ring_claims(const f128 *f, const f128 *suffix, size_t n, const PassPost &post,
                 cudaStream_t s);
void packed_basis(const f128 *suffix, size_t n, const RowWeights128 &bw, const f128 *eq_ood,
                  f128 coef, f128 *basis, cudaStream_t s);
// y += a * x
void axpy(f128 *y, f128 a, const f128 *x, size_t n, cudaStream_t s);
// Interleaved Reed-Solomon encode of msg (2^log_n entries, 2^k columns) at
// rate 2^-rate into cw, staged through shared memory by TMA copies; err (a
// word the host reads; null: no report) is set when a copy did not land
// within its time limit.
void rs_encode(const f128 *msg, int log_n, int k, int rate, const f128 *wh, f128 *cw,
               unsigned int *err, cudaStream_t s);
void merkle_build(const f128 *cw, size_t rows, int k, uint32_t *nodes, cudaStream_t s);
// A small tree (at most kMerkleBlockMaxRows rows) in one launch that posts
// the root (node 1, 32 bytes) as four mailbox words of publication pub; false
// (nothing launched) when the tree is larger or there is no mailbox.
constexpr size_t kMerkleBlockMaxRows = 4096;
bool merkle_build_posted(const f128 *cw, size_t rows, int k, uint32_t *nodes, Publish pub,
                         cudaStream_t s);
constexpr int kMaxQueries = 512, kMaxQueryWidth = 64;
struct QueryTerms {
  uint64_t idx[kMaxQueries];
  f128 scale[kMaxQueries];
};
struct QueryRows {
  uint64_t idx[kMaxQueries];
  f128 eqr[kMaxQueryWidth];
};
// basis += sum_q scale[q] * tensor(Wh_t(x_q), t < l), x_q = idx[q]; wh is the
// kMaxRsDim x kMaxRsDim subspace table (Wh_t(X^s) at t * kMaxRsDim + s).
void query_basis(const QueryTerms &terms, const f128 *wh, int nq, int l, f128 *basis,
                 cudaStream_t s);
// Per query (idx[q] < rows): the codeword row and its Merkle siblings, packed
// as width + 2 * depth 16-byte units; behind them all, each row's combination
// with eqr.
void gather_openings(const f128 *cw, const uint32_t *nodes, size_t rows, int width, int depth,
                     const QueryRows &queries, int nq, f128 *out, cudaStream_t s);
// A level's openings in a proof: `at` counts 32-bit words from `proof`, each of
// the nq openings is the row (width 16-byte entries) and `depth` siblings.
// vals[q] = sum over the row of entry c times queries.eqr[c]; *bad is set (it
// starts zero) when a path from leaf queries.idx[q] does not reach the root.
struct B3Root {
  uint32_t w[8];
};
void check_openings(const uint32_t *proof, size_t at, int width, int depth,
                    const QueryRows &queries, int nq, const B3Root &root, f128 *vals,
                    unsigned int *bad, cudaStream_t s);

// Host helpers (GF(2^128) on the CPU for the few scalar steps).
f128 gf_inv_host(f128 a);
// wh[t * kMaxRsDim + s] = Wh_t(X^s): the normalised subspace polynomial of
// span(X^0..X^(t-1)) at X^s, for t, s < d.
void subspace_table(int d, f128 *wh);
// The comb table of `base` with 8-bit windows: 16 x 256 entries.
void comb_table(f128 base, f128 *out);
f128 smallest_generator_host();
void eq_table_host(const f128 *r, int n, f128 *out);

}  // namespace bz
