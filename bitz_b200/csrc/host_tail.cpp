#include "host_tail.hpp"

#include <immintrin.h>

#include "transcript.hpp"

namespace bz {

namespace {

bool vector_products() {
  static const bool on = host_simd_enabled() && __builtin_cpu_supports("avx512f") &&
                         __builtin_cpu_supports("avx512bw") &&
                         __builtin_cpu_supports("vpclmulqdq");
  return on;
}

#define BZ_VEC __attribute__((target("avx512f,avx512bw,vpclmulqdq")))
#define BZ_VEC_INLINE __attribute__((always_inline, target("avx512f,avx512bw,vpclmulqdq"))) inline

// Four 256-bit products: low and high halves.
struct Wide4 {
  __m512i lo, hi;
};

BZ_VEC_INLINE __m512i load4(const f128 *p) { return _mm512_loadu_si512((const void *)p); }
BZ_VEC_INLINE void store4(f128 *p, __m512i v) { _mm512_storeu_si512((void *)p, v); }

BZ_VEC_INLINE Wide4 product4(__m512i a, __m512i b) {
  const __m512i l = _mm512_clmulepi64_epi128(a, b, 0x00), h = _mm512_clmulepi64_epi128(a, b, 0x11);
  const __m512i m = _mm512_xor_si512(_mm512_clmulepi64_epi128(a, b, 0x10),
                                     _mm512_clmulepi64_epi128(a, b, 0x01));
  Wide4 w;
  w.lo = _mm512_xor_si512(l, _mm512_bslli_epi128(m, 8));
  w.hi = _mm512_xor_si512(h, _mm512_bsrli_epi128(m, 8));
  return w;
}

// X^128 = X^7 + X^2 + X + 1 = 0x87: the high half's two words times 0x87, and
// the seven bits that spill over once more.
BZ_VEC_INLINE __m512i reduce4(const Wide4 &w) {
  const __m512i p = _mm512_set_epi64(0, 0x87, 0, 0x87, 0, 0x87, 0, 0x87);
  const __m512i t0 = _mm512_clmulepi64_epi128(w.hi, p, 0x00);
  const __m512i t1 = _mm512_clmulepi64_epi128(w.hi, p, 0x01);
  const __m512i t2 = _mm512_clmulepi64_epi128(t1, p, 0x01);
  return _mm512_xor_si512(_mm512_xor_si512(w.lo, t0),
                          _mm512_xor_si512(_mm512_bslli_epi128(t1, 8), t2));
}

BZ_VEC_INLINE __m512i mul4(__m512i a, __m512i b) { return reduce4(product4(a, b)); }

BZ_VEC_INLINE __m512i broadcast4(f128 r) {
  return _mm512_broadcast_i32x4(_mm_set_epi64x((long long)r.hi, (long long)r.lo));
}

BZ_VEC_INLINE void add4(Wide4 &s, const Wide4 &w) {
  s.lo = _mm512_xor_si512(s.lo, w.lo);
  s.hi = _mm512_xor_si512(s.hi, w.hi);
}

// The four lanes' products added up and reduced.
BZ_VEC_INLINE f128 total4(const Wide4 &s) {
  f128 v[4];
  store4(v, reduce4(s));
  return gadd(gadd(v[0], v[1]), gadd(v[2], v[3]));
}

// Entries 0, 2, 4, 6 and 1, 3, 5, 7 of eight in a row.
BZ_VEC_INLINE void pairs4(const f128 *p, __m512i &even, __m512i &odd) {
  const __m512i a = load4(p), b = load4(p + 4);
  even = _mm512_shuffle_i64x2(a, b, 0x88);
  odd = _mm512_shuffle_i64x2(a, b, 0xdd);
}

BZ_VEC void bind_high4(f128 *t, size_t h, f128 r) {
  const __m512i rr = broadcast4(r);
  for (size_t x = 0; x < h; x += 4) {
    const __m512i a = load4(t + x), b = load4(t + x + h);
    store4(t + x, _mm512_xor_si512(a, mul4(rr, _mm512_xor_si512(a, b))));
  }
}

BZ_VEC void bind_low4(f128 *t, size_t n, f128 r) {
  const __m512i rr = broadcast4(r);
  for (size_t o = 0; o < n; o += 4) {
    __m512i a, b;
    pairs4(t + 2 * o, a, b);
    store4(t + o, _mm512_xor_si512(a, mul4(rr, _mm512_xor_si512(a, b))));
  }
}

BZ_VEC void scale4(const f128 *t, f128 r, size_t n, f128 *out) {
  const __m512i rr = broadcast4(r);
  for (size_t k = 0; k < n; k += 4) store4(out + k, mul4(rr, load4(t + k)));
}

BZ_VEC void cubic_sums4(const f128 *e, const f128 *L, const f128 *R, size_t h, bool one,
                        f128 out[2]) {
  Wide4 s0{_mm512_setzero_si512(), _mm512_setzero_si512()}, s1 = s0;
  for (size_t x = 0; x < h; x += 4) {
    const __m512i w = load4(e + x), l0 = load4(L + x), l1 = load4(L + x + h), r0 = load4(R + x),
                  r1 = load4(R + x + h);
    add4(s0, product4(mul4(w, one ? l1 : l0), one ? r1 : r0));
    add4(s1, product4(mul4(w, _mm512_xor_si512(l0, l1)), _mm512_xor_si512(r0, r1)));
  }
  out[0] = total4(s0);
  out[1] = total4(s1);
}

BZ_VEC void quad_sums4(const f128 *W, const f128 *V, size_t n, f128 out[2]) {
  Wide4 s0{_mm512_setzero_si512(), _mm512_setzero_si512()}, s1 = s0;
  for (size_t j = 0; j < n; j += 4) {
    __m512i w0, w1, v0, v1;
    pairs4(W + 2 * j, w0, w1);
    pairs4(V + 2 * j, v0, v1);
    add4(s0, product4(w0, v0));
    add4(s1, product4(_mm512_xor_si512(w0, w1), _mm512_xor_si512(v0, v1)));
  }
  out[0] = total4(s0);
  out[1] = total4(s1);
}

}  // namespace

void host_bind_high(f128 *t, size_t h, f128 r) {
  if (h % 4 == 0 && vector_products()) return bind_high4(t, h, r);
  for (size_t x = 0; x < h; x++) t[x] = gadd(t[x], gmul(r, gadd(t[x], t[x + h])));
}

void host_bind_low(f128 *t, size_t n, f128 r) {
  if (n % 4 == 0 && vector_products()) return bind_low4(t, n, r);
  for (size_t o = 0; o < n; o++) t[o] = gadd(t[2 * o], gmul(r, gadd(t[2 * o], t[2 * o + 1])));
}

void host_scale(const f128 *t, f128 r, size_t n, f128 *out) {
  if (n % 4 == 0 && vector_products()) return scale4(t, r, n, out);
  for (size_t k = 0; k < n; k++) out[k] = gmul(r, t[k]);
}

void host_cubic_sums(const f128 *e, const f128 *L, const f128 *R, size_t h, bool one,
                     f128 out[2]) {
  if (h % 4 == 0 && vector_products()) return cubic_sums4(e, L, R, h, one, out);
  wide s0 = wzero(), s1 = wzero();
  for (size_t x = 0; x < h; x++) {
    wacc(s0, gmul_wide(gmul(e[x], one ? L[x + h] : L[x]), one ? R[x + h] : R[x]));
    wacc(s1, gmul_wide(gmul(e[x], gadd(L[x], L[x + h])), gadd(R[x], R[x + h])));
  }
  out[0] = greduce(s0);
  out[1] = greduce(s1);
}

void host_quad_sums(const f128 *W, const f128 *V, size_t n, f128 out[2]) {
  if (n % 4 == 0 && vector_products()) return quad_sums4(W, V, n, out);
  wide s0 = wzero(), s1 = wzero();
  for (size_t j = 0; j < n; j++) {
    wacc(s0, gmul_wide(W[2 * j], V[2 * j]));
    wacc(s1, gmul_wide(gadd(W[2 * j], W[2 * j + 1]), gadd(V[2 * j], V[2 * j + 1])));
  }
  out[0] = greduce(s0);
  out[1] = greduce(s1);
}

}  // namespace bz
