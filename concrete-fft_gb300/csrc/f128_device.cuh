// f128_device.cuh -- double-double arithmetic of the reference's fft128 module.
//
// Error-free transformations (TwoSum, TwoDiff, QuickTwoSum, FMA TwoProd) and
// the "estimate" add/sub used by the FFT butterflies, each restated from
// src/fft128/f128_ops.rs with explicit IEEE intrinsics; the library is built
// with --fmad=false so nvcc cannot fuse or reorder any step.
#pragma once
#include <cstdint>

#include "cfft_device.cuh"
#include "int_f128.cuh"

namespace cfft {

struct f128 {
  double hi, lo;
};

// src/fft128/f128_ops.rs:3-40
__device__ __forceinline__ void quick_two_sum(double a, double b, double& s, double& e) {
  s = __dadd_rn(a, b);
  e = __dsub_rn(b, __dsub_rn(s, a));
}
__device__ __forceinline__ void two_sum(double a, double b, double& s, double& e) {
  s = __dadd_rn(a, b);
  const double bb = __dsub_rn(s, a);
  e = __dadd_rn(__dsub_rn(a, __dsub_rn(s, bb)), __dsub_rn(b, bb));
}
__device__ __forceinline__ void two_diff(double a, double b, double& s, double& e) {
  s = __dsub_rn(a, b);
  const double bb = __dsub_rn(s, a);
  e = __dsub_rn(__dsub_rn(a, __dsub_rn(s, bb)), __dadd_rn(b, bb));
}

// N of these at once on the integer pipes (int_f128.cuh, the same bits), with
// the ones outside its range redone on the FP64 pipe one by one, in a loop
// (as sum_diff in int_fp64.cuh, and for its reason).
template <int N, class Redo>
__device__ __forceinline__ void redo_each(uint32_t bits, Redo redo) {
  asm volatile("" : "+r"(bits));
  while (bits) {
    const int i = 31 - __clz((int)bits);
    bits &= ~(1u << i);
    redo(i);
  }
}
template <int N>
__device__ __forceinline__ double pick(const double* v, int i) {
  double x = v[0];
#pragma unroll
  for (int j = 1; j < N; ++j)
    if (i == j) x = v[j];
  return x;
}
template <int N>
__device__ __forceinline__ void put(double* v, int i, double x) {
#pragma unroll
  for (int j = 0; j < N; ++j)
    if (i == j) v[j] = x;
}

template <int N>
__device__ __forceinline__ void quick_two_sums(const double* s, const double* e, double* hi, double* lo) {
  uint32_t bits = 0;
#pragma unroll
  for (int j = 0; j < N; ++j)
    if (!quick_two_sum_int(s[j], e[j], hi[j], lo[j])) bits += 1u << j;
  redo_each<N>(bits, [&](int i) {
    double h, l;
    quick_two_sum(pick<N>(s, i), pick<N>(e, i), h, l);
    put<N>(hi, i, h);
    put<N>(lo, i, l);
  });
}
template <int N>
__device__ __forceinline__ void two_sums(const double* a, const double* b, double* s, double* e) {
  uint32_t bits = 0;
#pragma unroll
  for (int j = 0; j < N; ++j)
    if (!two_sum_int(a[j], b[j], s[j], e[j])) bits += 1u << j;
  redo_each<N>(bits, [&](int i) {
    double h, l;
    two_sum(pick<N>(a, i), pick<N>(b, i), h, l);
    put<N>(s, i, h);
    put<N>(e, i, l);
  });
}
// s + es = a + b, d + ed = a - b
template <int N>
__device__ __forceinline__ void two_sum_diffs(const double* a, const double* b, double* s, double* es, double* d,
                                              double* ed) {
  uint32_t bits = 0;
#pragma unroll
  for (int j = 0; j < N; ++j)
    if (!two_sum_diff_int(a[j], b[j], s[j], es[j], d[j], ed[j])) bits += 1u << j;
  redo_each<N>(bits, [&](int i) {
    const double x = pick<N>(a, i), y = pick<N>(b, i);
    double h, l;
    two_sum(x, y, h, l);
    put<N>(s, i, h);
    put<N>(es, i, l);
    two_diff(x, y, h, l);
    put<N>(d, i, h);
    put<N>(ed, i, l);
  });
}

// p[j] = w[j] * b[j], rounded to nearest
template <int N>
__device__ __forceinline__ void products(const double* w, const double* b, double* p) {
  uint32_t bits = 0;
#pragma unroll
  for (int j = 0; j < N; ++j)
    if (!mul_int(w[j], b[j], p[j])) bits += 1u << j;
  redo_each<N>(bits, [&](int i) { put<N>(p, i, __dmul_rn(pick<N>(w, i), pick<N>(b, i))); });
}

// r[j] = a[j] * b[j]: src/fft128/f128_ops.rs:395-400 (TwoProd by FMA, src/fft128/f128_ops.rs:37-40)
template <int N>
__device__ __forceinline__ void muls(const f128* a, const f128* b, f128* r) {
  double p[N], e[N], hi[N], lo[N], w[2 * N], v[2 * N], x[2 * N];
#pragma unroll
  for (int j = 0; j < N; ++j) {
    w[j] = b[j].lo, v[j] = a[j].hi;
    w[N + j] = b[j].hi, v[N + j] = a[j].lo;
    p[j] = __dmul_rn(a[j].hi, b[j].hi);
    e[j] = __fma_rn(a[j].hi, b[j].hi, -p[j]);
  }
  products<2 * N>(w, v, x);
#pragma unroll
  for (int j = 0; j < N; ++j) e[j] = __dadd_rn(e[j], __dadd_rn(x[j], x[N + j]));
  quick_two_sums<N>(p, e, hi, lo);
#pragma unroll
  for (int j = 0; j < N; ++j) r[j] = f128{hi[j], lo[j]};
}

// r[j] = a[j] + b[j] (add[j]) or a[j] - b[j] by the estimate variants,
// src/fft128/f128_ops.rs:314-320 and :360-367.  two_diff(a, b) is two_sum(a, -b).
template <int N>
__device__ __forceinline__ void ests(const f128* a, const f128* b, const bool* add, f128* r) {
  double x[N], y[N], s[N], e[N], hi[N], lo[N];
#pragma unroll
  for (int j = 0; j < N; ++j) x[j] = a[j].hi, y[j] = add[j] ? b[j].hi : -b[j].hi;
  two_sums<N>(x, y, s, e);
#pragma unroll
  for (int j = 0; j < N; ++j) {
    // e + (a.lo + b.lo) or (e + a.lo) - b.lo, by selected operands: a runtime add[j] must not
    // make both (an FP64 instruction that is predicated off takes its time all the same)
    const double t = __dadd_rn(add[j] ? b[j].lo : e[j], a[j].lo);
    e[j] = __dadd_rn(t, add[j] ? e[j] : -b[j].lo);
  }
  quick_two_sums<N>(s, e, hi, lo);
#pragma unroll
  for (int j = 0; j < N; ++j) r[j] = f128{hi[j], lo[j]};
}
// u[j] = a[j] + b[j] and v[j] = a[j] - b[j] by the estimate variants
template <int N>
__device__ __forceinline__ void est_pairs(const f128* a, const f128* b, f128* u, f128* v) {
  double x[N], y[N], s[2 * N], e[2 * N], hi[2 * N], lo[2 * N];
#pragma unroll
  for (int j = 0; j < N; ++j) x[j] = a[j].hi, y[j] = b[j].hi;
  two_sum_diffs<N>(x, y, s, e, s + N, e + N);
#pragma unroll
  for (int j = 0; j < N; ++j) {
    e[j] = __dadd_rn(e[j], __dadd_rn(a[j].lo, b[j].lo));
    e[N + j] = __dsub_rn(__dadd_rn(e[N + j], a[j].lo), b[j].lo);
  }
  quick_two_sums<2 * N>(s, e, hi, lo);
#pragma unroll
  for (int j = 0; j < N; ++j) u[j] = f128{hi[j], lo[j]}, v[j] = f128{hi[N + j], lo[N + j]};
}

// src/fft128/mod.rs:310-346 (Scalar backend: add/sub are the estimate variants);
// CONJ: times the conjugate of (br, bi)
template <bool CONJ>
__device__ __forceinline__ void cplx_mul(f128 ar, f128 ai, f128 br, f128 bi, f128& orr, f128& oi) {
  const f128 a[4] = {ar, ai, ai, ar}, b[4] = {br, br, bi, bi};
  f128 m[4];  // rr, ir, ii, ri
  muls<4>(a, b, m);
  const bool add[2] = {CONJ, !CONJ};
  f128 o[2];
  ests<2>(m, m + 2, add, o);
  orr = o[0];
  oi = o[1];
}

// Split-array views: four f64 arrays (re0, re1, im0, im1).
struct F128Arrays {
  double* re0;
  double* re1;
  double* im0;
  double* im1;
};
struct F128Tw {
  const double* __restrict__ re0;
  const double* __restrict__ re1;
  const double* __restrict__ im0;
  const double* __restrict__ im1;
};

// Forward radix-2 butterfly of src/fft128/mod.rs:378-397 on element pair (j, j + t).
__device__ __forceinline__ void f128_fwd_bfly(F128Arrays d, long j, long t, const F128Tw& tw, long widx) {
  const f128 wr{__ldg(tw.re0 + widx), __ldg(tw.re1 + widx)};
  const f128 wi{__ldg(tw.im0 + widx), __ldg(tw.im1 + widx)};
  const f128 z0r{d.re0[j], d.re1[j]}, z0i{d.im0[j], d.im1[j]};
  const f128 z1r{d.re0[j + t], d.re1[j + t]}, z1i{d.im0[j + t], d.im1[j + t]};
  const f128 z0[2] = {z0r, z0i};
  f128 z[2], u[2], v[2];
  cplx_mul<false>(z1r, z1i, wr, wi, z[0], z[1]);
  est_pairs<2>(z0, z, u, v);
  d.re0[j] = u[0].hi;
  d.re1[j] = u[0].lo;
  d.im0[j] = u[1].hi;
  d.im1[j] = u[1].lo;
  d.re0[j + t] = v[0].hi;
  d.re1[j + t] = v[0].lo;
  d.im0[j + t] = v[1].hi;
  d.im1[j + t] = v[1].lo;
}

// Inverse radix-2 butterfly of src/fft128/mod.rs:1131-1150.
__device__ __forceinline__ void f128_inv_bfly(F128Arrays d, long j, long t, const F128Tw& tw, long widx) {
  const f128 wr{__ldg(tw.re0 + widx), __ldg(tw.re1 + widx)};
  const f128 wi{__ldg(tw.im0 + widx), __ldg(tw.im1 + widx)};
  const f128 z0r{d.re0[j], d.re1[j]}, z0i{d.im0[j], d.im1[j]};
  const f128 z1r{d.re0[j + t], d.re1[j + t]}, z1i{d.im0[j + t], d.im1[j + t]};
  const f128 z0[2] = {z0r, z0i}, z1[2] = {z1r, z1i};
  f128 u[2], dd[2], mr, mi;
  est_pairs<2>(z0, z1, u, dd);
  cplx_mul<true>(dd[0], dd[1], wr, wi, mr, mi);
  d.re0[j] = u[0].hi;
  d.re1[j] = u[0].lo;
  d.im0[j] = u[1].hi;
  d.im1[j] = u[1].lo;
  d.re0[j + t] = mr.hi;
  d.re1[j + t] = mr.lo;
  d.im0[j + t] = mi.hi;
  d.im1[j + t] = mi.lo;
}

// One radix-2 stage of double-double butterflies with two warps per 32
// butterflies: warp 2k computes the real parts of both outputs of butterflies
// 32k .. 32k+31, warp 2k+1 their imaginary parts.  The real and imaginary
// parts of a butterfly share no operation (cplx_mul, cplx_mul_conj), so each
// half does exactly the operations of its outputs and the results are the
// one-thread butterfly's bits; the inverse's conjugate product needs the other
// half's difference, which passes through xs (4 doubles per butterfly of an
// iteration).  A barrier separates every read of an iteration's elements from
// the stores.  Warp-uniform halves keep each warp on one instruction stream.
// map(b, qa, qb, widx) gives butterfly b's elements and twiddle index; nb
// butterflies; every thread of the CTA calls it.
template <bool FWD, class Map>
__device__ __forceinline__ void f128_half_stage(F128Arrays s, double* xs, int nb, Map map, const F128Tw& tw,
                                                int tid, int nth) {
  const int h = (tid >> 5) & 1;
  const int bi = ((tid >> 6) << 5) + (tid & 31);
  const int step = nth >> 1;
  double* d0 = h ? s.im0 : s.re0;
  double* d1 = h ? s.im1 : s.re1;
  for (int b0 = 0; b0 < nb; b0 += step) {
    const int b = b0 + bi;
    const bool act = b < nb;
    int qa = 0, qb = 0;
    f128 u{0, 0}, v{0, 0}, dd{0, 0}, wr{0, 0}, wi{0, 0};
    if (act) {
      long widx;
      map(b, qa, qb, widx);
      wr = f128{__ldg(tw.re0 + widx), __ldg(tw.re1 + widx)};
      wi = f128{__ldg(tw.im0 + widx), __ldg(tw.im1 + widx)};
      const f128 z0{d0[qa], d1[qa]};
      if (FWD) {
        const f128 z1r{s.re0[qb], s.re1[qb]}, z1i{s.im0[qb], s.im1[qb]};
        // real: mul(z1r, wr) - mul(z1i, wi); imaginary: mul(z1i, wr) + mul(z1r, wi)
        const f128 a[2] = {h ? z1i : z1r, h ? z1r : z1i}, b[2] = {wr, wi};
        f128 m[2], z;
        muls<2>(a, b, m);
        const bool add = h != 0;
        ests<1>(m, m + 1, &add, &z);
        est_pairs<1>(&z0, &z, &u, &v);
      } else {
        const f128 z1{d0[qb], d1[qb]};
        est_pairs<1>(&z0, &z1, &u, &dd);  // dd: dr (h = 0) or di (h = 1)
        double* x = xs + (((b - b0) << 1) + h) * 2;
        x[0] = dd.hi;
        x[1] = dd.lo;
      }
    }
    __syncthreads();  // every read of this iteration's elements is done
    if (act) {
      if (!FWD) {
        const double* x = xs + (((b - b0) << 1) + (h ^ 1)) * 2;
        const f128 od{x[0], x[1]};
        // real: mul(dr, wr) + mul(di, wi); imaginary: mul(di, wr) - mul(dr, wi)
        const f128 a[2] = {dd, od}, b[2] = {wr, wi};
        f128 m[2];
        muls<2>(a, b, m);
        const bool add = h == 0;
        ests<1>(m, m + 1, &add, &v);
      }
      d0[qa] = u.hi;
      d1[qa] = u.lo;
      d0[qb] = v.hi;
      d1[qb] = v.lo;
    }
    __syncthreads();  // the stores are done before the next reads
  }
}

// Stages of a transform of 2^log2n points restricted to one sub-block of
// 2^log2c points (sub-block index sb), all in shared memory.  Forward runs
// t = 2^(log2c-1) .. 1 (src/fft128/mod.rs:363-401), inverse t = 1 .. 2^(log2c-1)
// (src/fft128/mod.rs:1117-1154); twiddle index m + i uses the global block i.
template <bool FWD>
__device__ __forceinline__ void f128_stages_smem(F128Arrays s, int log2n, int log2c, long sb, const F128Tw& tw,
                                                 int tid, int nth) {
  const int half = 1 << (log2c - 1);  // butterflies per sub-block per stage
  for (int st = 0; st < log2c; ++st) {
    const int log2t = FWD ? (log2c - 1 - st) : st;
    const long t = 1L << log2t;
    const long m = 1L << (log2n - 1 - log2t);  // blocks of 2t in the whole transform
    for (int b = tid; b < half; b += nth) {
      const long i_local = b >> log2t;
      const long jj = b & (t - 1);
      const long j = (i_local << (log2t + 1)) + jj;
      const long i_global = (sb << (log2c - 1 - log2t)) + i_local;
      if (FWD) f128_fwd_bfly(s, j, t, tw, m + i_global);
      else f128_inv_bfly(s, j, t, tw, m + i_global);
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------- integers
// One u128 coefficient (lo, hi, read as i128) -> f128: xh = the nearest double, xl =
// the nearest double to the remainder (src/fft128/mod.rs:2006-2016 pattern), without
// going back from xh to an integer: the remainder is the bits that xh's rounding
// drops, less 2^75 of its unit where it rounds up.
__device__ __forceinline__ void u128_to_f128(uint64_t lo, uint64_t hi, double& xh, double& xl) {
  const uint64_t neg = hi >> 63;
  if (neg) {
    lo = 0 - lo;
    hi = ~hi + (lo == 0 ? 1 : 0);
  }
  if ((hi | lo) == 0) {
    xh = xl = 0.0;
    return;
  }
  const int lz = hi != 0 ? __clzll((long long)hi) : 64 + __clzll((long long)lo);
  if (lz >= 64) {
    hi = lo;
    lo = 0;
  }
  const int sh = lz & 63;
  if (sh != 0) {
    hi = (hi << sh) | (lo >> (64 - sh));
    lo <<= sh;
  }
  // leading one at bit 127: 53 bits kept, 75 dropped
  const uint64_t top = hi >> 11;
  const uint64_t dh = hi & 0x7ff;
  const uint64_t half = 0x400;
  const bool up = dh > half || (dh == half && (lo != 0 || (top & 1) != 0));
  xh = __longlong_as_double((long long)((neg << 63) | (((uint64_t)(1023 + 126 - lz) << 52) + top + (up ? 1 : 0))));
  // the remainder's magnitude: 76 bits (rh:rl)
  uint64_t rh = dh, rl = lo;
  if (up) {
    rl = 0 - lo;
    rh = 0x800 - dh - (lo != 0 ? 1 : 0);
  }
  if ((rh | rl) == 0) {
    xl = 0.0;
    return;
  }
  uint64_t th = (rh << 52) | (rl >> 12), tl = rl << 52;  // left-aligned in 128 bits
  const int l2 = th != 0 ? __clzll((long long)th) : 64 + __clzll((long long)tl);
  if (l2 >= 64) {
    th = tl;
    tl = 0;
  }
  const int s2 = l2 & 63;
  if (s2 != 0) {
    th = (th << s2) | (tl >> (64 - s2));
    tl <<= s2;
  }
  const uint64_t m = th >> 11;
  const uint64_t r = th & 0x7ff;
  const bool up2 = r > half || (r == half && (tl != 0 || (m & 1) != 0));
  const uint64_t sign = (neg ^ (up ? 1 : 0)) << 63;
  xl = __longlong_as_double((long long)(sign | (((uint64_t)(1023 + 74 - l2 - lz) << 52) + m + (up2 ? 1 : 0))));
}

// x[j] *= 2^-k, 0 <= k < 64: on the exponent field, or by an FP64 product outside
// the normal range.
template <int N>
__device__ __forceinline__ void scale_down(double* x, int k) {
  uint32_t bits = 0;
  double y[N];
#pragma unroll
  for (int j = 0; j < N; ++j) {
    const uint32_t h = (uint32_t)__double2hiint(x[j]);
    if ((h & 0x7ff00000u) - (64u << 20) >= (0x7bfu << 20)) bits += 1u << j;
    y[j] = __hiloint2double((int)(h - ((uint32_t)k << 20)), __double2loint(x[j]));
  }
  redo_each<N>(bits, [&](int i) {
    put<N>(y, i, __dmul_rn(pick<N>(x, i), __hiloint2double((int)((1023u - (uint32_t)k) << 20), 0)));
  });
#pragma unroll
  for (int j = 0; j < N; ++j) x[j] = y[j];
}

// trunc(x) as an integer mod 2^128 (lo, hi words), and x - trunc(x).
__device__ __forceinline__ void trunc_mod128(double x, uint64_t& lo, uint64_t& hi, double& frac) {
  const double t = trunc(x);
  frac = __dsub_rn(x, t);
  const uint64_t bits = (uint64_t)__double_as_longlong(t);
  const bool neg = (bits >> 63) != 0;
  const int bexp = (int)((bits >> 52) & 0x7ff);
  lo = hi = 0;
  if (bexp == 0x7ff || bexp == 0) return;
  const uint64_t m = (bits & 0xfffffffffffffull) | (1ull << 52);
  const int e = bexp - 1075;
  if (e >= 128) return;
  if (e >= 64) {
    hi = m << (e - 64);
  } else if (e > 11) {
    lo = m << e;
    hi = m >> (64 - e);
  } else if (e >= 0) {
    lo = m << e;
  } else {
    lo = (-e) >= 64 ? 0 : (m >> (-e));
  }
  if (neg) {
    lo = ~lo;
    hi = ~hi;
    lo += 1;
    if (lo == 0) hi += 1;
  }
}

// m * 2^e mod 2^128, 0 <= e
__device__ __forceinline__ void shift_left_mod128(uint64_t m, int e, uint64_t& lo, uint64_t& hi) {
  lo = e < 64 ? m << (e & 63) : 0;
  hi = e >= 128 ? 0 : e >= 64 ? m << (e & 63) : e == 0 ? 0 : m >> (64 - e);
}

// floor(hi + lo + 1/2) mod 2^128 for a double-double, exact.
__device__ __forceinline__ void round_half_up_mod128(double xhi, double xlo, uint64_t& rlo, uint64_t& rhi) {
  const uint64_t hb = (uint64_t)__double_as_longlong(xhi), lb = (uint64_t)__double_as_longlong(xlo);
  const int he = (int)((hb >> 52) & 0x7ff) - 1075, le = (int)((lb >> 52) & 0x7ff) - 1075;
  if (he >= 0 && he < 0x7ff - 1075 && le < 0x7ff - 1075) {
    // the high word is an integer: itself plus floor(lo + 1/2), in integers
    uint64_t al, ah, bl, bh;
    shift_left_mod128((hb & 0xfffffffffffffull) | (1ull << 52), he, al, ah);
    const uint64_t m = (lb & 0xfffffffffffffull) | (1ull << 52);
    const uint64_t lneg = lb >> 63;
    if (le >= 0) {
      shift_left_mod128(m, le, bl, bh);
    } else {
      // |lo| < 2^53: floor(m 2^-k + 1/2), or of -m 2^-k minus floor((m + half - 1) 2^-k); 0 below 1/4
      const int k = -le;
      bl = k > 54 ? 0 : (m + (1ull << ((k - 1) & 63)) - lneg) >> (k & 63);
      bh = 0;
    }
    // two's complement: xor with the sign, the carries below
    const uint64_t hs = 0 - (hb >> 63), ls = 0 - lneg;
    al = (al ^ hs) - hs;
    ah = (ah ^ hs) + (hs & (al == 0 ? 1 : 0));
    bl = (bl ^ ls) - ls;
    bh = (bh ^ ls) + (ls & (bl == 0 ? 1 : 0));
    rlo = al + bl;
    rhi = ah + bh + (rlo < al ? 1 : 0);
    return;
  }
  uint64_t hl, hh, ll, lh;
  double fh, fl;
  trunc_mod128(xhi, hl, hh, fh);
  trunc_mod128(xlo, ll, lh, fl);
  double s, e;
  two_sum(fh, fl, s, e);
  const int f = -2 + (int)(s > -1.5 || (s == -1.5 && e >= 0.0)) + (int)(s > -0.5 || (s == -0.5 && e >= 0.0)) +
                (int)(s > 0.5 || (s == 0.5 && e >= 0.0)) + (int)(s > 1.5 || (s == 1.5 && e >= 0.0));
  uint64_t lo = hl + ll;
  uint64_t hi = hh + lh + (lo < hl ? 1 : 0);
  const uint64_t flo = (uint64_t)(int64_t)f;
  const uint64_t fhi = f < 0 ? ~0ull : 0ull;
  const uint64_t lo2 = lo + flo;
  hi = hi + fhi + (lo2 < lo ? 1 : 0);
  rlo = lo2;
  rhi = hi;
}

}  // namespace cfft
