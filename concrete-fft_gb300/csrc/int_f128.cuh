// int_f128.cuh -- error-free sums of doubles on the integer pipes.
//
// The double-double butterflies are chains of FP64 additions: a TwoSum is 6 of
// them (one warp instruction per ~76 cycles of an SM sub-partition each), a
// QuickTwoSum 3.  Each computes a rounded sum and its exact rounding error.  In
// integers the error is at hand: it is the bits that the rounding drops.  The
// routines below return the same doubles, bit for bit, as the FP64 sequences,
// and false where their range ends; the callers then run the FP64 sequence.
#pragma once
#include "int_fp64.cuh"

namespace cfft {

// r * 2^(x - 1075) for |r| <= 2^12 as the high word of a double (the low word
// is 0): x is the biased exponent in place (bits 20..30) of a double whose last
// place is the unit, sign is 0 or 2^31.  r = 0 gives +0.
__device__ __forceinline__ uint32_t small_times_ulp(int r, uint32_t x, uint32_t sign) {
  const uint32_t f = (uint32_t)__float_as_int(__int2float_rn(r));  // exact
  // float to double: the fraction moves down by 3, the exponent from bias 127 to 1023
  // and by x - 1075
  const uint32_t m = (f & 0x7fffffffu) >> 3;
  const uint32_t v = (m + x - (127u << 20) + ((1023u - 1075u) << 20)) | ((f ^ sign) & 0x80000000u);
  return r == 0 ? 0u : v;
}

// The common part of the sums below: both significands at bits 62..10 of 64-bit
// words, the smaller operand's shifted right by the exponent difference.
struct Aligned {
  uint64_t A, B;
  uint32_t e;  // the larger exponent, in place
  bool ok;
};
__device__ __forceinline__ Aligned align_int(uint32_t ah, uint32_t al, uint32_t bh, uint32_t bl) {
  Aligned r;
  const uint32_t xa = ah & 0x7ff00000u, xb = bh & 0x7ff00000u;
  r.e = max(xa, xb);
  const int dif = (int)(xa - xb) >> 20;
  r.ok = (uint32_t)(dif + 10) <= 20u;
  // down to 2^-894: the errors stay normal numbers
  r.ok = r.ok && (r.e - (128u << 20)) < (0x77eu << 20);
  const uint32_t na = (uint32_t)min(dif + 10, 10), nb = (uint32_t)min(10 - dif, 10);
  const uint32_t ma = (ah & 0xfffffu) | 0x100000u, mb = (bh & 0xfffffu) | 0x100000u;
  r.A = ((uint64_t)__funnelshift_l(al, ma, na) << 32) | (al << (na & 31));
  r.B = ((uint64_t)__funnelshift_l(bl, mb, nb) << 32) | (bl << (nb & 31));
  return r;
}

// N = V << f with the leading one at bit 63, V's unit 2^(e - 1085) in the sense
// above: rounds to nearest even at bit 11 into (h:l) with sign bit `sign`, and
// returns the rounding error's high word.
__device__ __forceinline__ uint32_t round_with_error(uint64_t V, uint32_t e, uint32_t sign, uint32_t& h, uint32_t& l,
                                                     bool& ok) {
  const uint32_t Vh = (uint32_t)(V >> 32), Vl = (uint32_t)V;
  ok = ok && Vh != 0;
  const uint32_t f = leading_zeros_nz(Vh);
  const uint32_t Nh = __funnelshift_l(Vl, Vh, f), Nl = Vl << (f & 31);
  l = __funnelshift_r(Nl, Nh, 11);
  h = Nh >> 11;
  // kept value + up: up is 1 iff the 11 dropped bits are above half, or half and the kept last bit is 1
  const uint32_t rem = Nl & 0x7ffu;
  const uint32_t up = (rem + 0x3ffu + (l & 1u)) >> 11;
  const uint32_t x = e - (f << 20);  // exponent of the result less one, in place
  asm("add.cc.u32 %0, %0, %3;\n\taddc.u32 %1, %1, %2;" : "+r"(l), "+r"(h) : "r"(x + sign), "r"(up));
  // unit of bit 0 of N: 2^-11 of the last place of a result of exponent x + 1
  return small_times_ulp((int)rem - (int)(up << 11), x + (1u << 20) - (11u << 20), sign);
}

// s + es = a + b and d + ed = a - b exactly, s and d rounded to nearest even:
// two_sum(a, b) and two_diff(a, b).
__device__ __forceinline__ bool two_sum_diff_int(double a, double b, double& s, double& es, double& d, double& ed) {
  const uint32_t ah = (uint32_t)__double2hiint(a), al = (uint32_t)__double2loint(a);
  const uint32_t bh = (uint32_t)__double2hiint(b), bl = (uint32_t)__double2loint(b);
  const Aligned g = align_int(ah, al, bh, bl);
  bool ok = g.ok;
  const uint64_t S = g.A + g.B;
  uint64_t D = g.A - g.B;
  const bool swap = (int64_t)D < 0;
  if (swap) D = 0 - D;
  const uint32_t sgn = ah & 0x80000000u;
  const uint32_t sgn_d = swap ? sgn ^ 0x80000000u : sgn;
  uint32_t sh, sl, dh, dl;
  const uint32_t rs = round_with_error(S, g.e, sgn, sh, sl, ok);
  const uint32_t rd = round_with_error(D, g.e, sgn_d, dh, dl, ok);
  const bool same = (int32_t)(ah ^ bh) >= 0;
  s = __hiloint2double((int)(same ? sh : dh), (int)(same ? sl : dl));
  d = __hiloint2double((int)(same ? dh : sh), (int)(same ? dl : sl));
  es = __hiloint2double((int)(same ? rs : rd), 0);
  ed = __hiloint2double((int)(same ? rd : rs), 0);
  return ok;
}

// s + e = a + b exactly, s rounded to nearest even: two_sum(a, b).
__device__ __forceinline__ bool two_sum_int(double a, double b, double& s, double& e) {
  const uint32_t ah = (uint32_t)__double2hiint(a), al = (uint32_t)__double2loint(a);
  const uint32_t bh = (uint32_t)__double2hiint(b), bl = (uint32_t)__double2loint(b);
  const Aligned g = align_int(ah, al, bh, bl);
  bool ok = g.ok;
  const bool same = (int32_t)(ah ^ bh) >= 0;
  uint64_t R = same ? g.A + g.B : g.A - g.B;
  const bool swap = !same && (int64_t)R < 0;
  if (swap) R = 0 - R;
  uint32_t sgn = ah & 0x80000000u;
  if (swap) sgn ^= 0x80000000u;
  uint32_t sh, sl;
  const uint32_t r = round_with_error(R, g.e, sgn, sh, sl, ok);
  s = __hiloint2double((int)sh, (int)sl);
  e = __hiloint2double((int)r, 0);
  return ok;
}

// hi + lo = s + e exactly, hi rounded to nearest even, for |e| at most 2^10
// units in the last place of s: quick_two_sum(s, e).  hi is s plus k units,
// k = round(e / unit), and lo = e - k units.
__device__ __forceinline__ bool quick_two_sum_int(double s, double e, double& hi, double& lo) {
  const uint32_t sh = (uint32_t)__double2hiint(s), sl = (uint32_t)__double2loint(s);
  const uint32_t eh = (uint32_t)__double2hiint(e), el = (uint32_t)__double2loint(e);
  const uint32_t xs = sh & 0x7ff00000u, xe = eh & 0x7ff00000u;
  const int n = (int)(xs - xe) >> 20;  // e's significand times 2^-n is e in units of s
  bool ok = (xs - (128u << 20)) < (0x77eu << 20) && n >= 43;
  const uint32_t me = (eh & 0xfffffu) | 0x100000u;
  // the significand left-aligned in 64 bits, less its integer part: (ip, fraction word, rest)
  const uint32_t Th = __funnelshift_l(el, me, 11), Tl = el << 11;
  const uint32_t t = (uint32_t)min(n - 21, 32);
  uint32_t ip;
  asm("shr.b32 %0, %1, %2;" : "=r"(ip) : "r"(Th), "r"(t));  // 0 from a shift of 32
  const uint32_t fw = Th << ((32 - t) & 31);
  const uint32_t u = fw | min(Tl, 1u) | ((sl ^ ip) & 1u);
  uint32_t k = ip + (u > 0x80000000u ? 1u : 0u);
  if (n >= 54) k = 0;  // below half a unit
  const bool same = (int32_t)(sh ^ eh) >= 0;
  const int kk = same ? (int)k : -(int)k;
  const uint64_t H = (((uint64_t)sh << 32) | sl) + (uint64_t)(int64_t)kk;
  const uint32_t Hh = (uint32_t)(H >> 32), Hl = (uint32_t)H;
  // a result in another binade, or at the low end of its own with a nonzero remainder, has
  // another unit below it
  ok = ok && ((Hh ^ sh) & 0xfff00000u) == 0 && (((Hh & 0xfffffu) | Hl) != 0 || n >= 55);
  // lo = (m - k 2^n) 2^-n units
  int Lh = (int)(me - (k << ((n - 32) & 31)));
  uint32_t Ll = el;
  const bool neg = Lh < 0;
  if (neg) {
    const uint64_t Z = 0 - (((uint64_t)(uint32_t)Lh << 32) | Ll);
    Lh = (int)(Z >> 32);
    Ll = (uint32_t)Z;
  }
  ok = ok && Lh != 0;
  const uint32_t f = leading_zeros_nz((uint32_t)Lh) - 11;
  const uint32_t sg = (eh & 0x80000000u) ^ (neg ? 0x80000000u : 0u);
  const uint32_t Oh = __funnelshift_l(Ll, (uint32_t)Lh, f) + (xe - (f << 20) - 0x100000u + sg);
  hi = __hiloint2double((int)Hh, (int)Hl);
  lo = __hiloint2double((int)Oh, (int)(Ll << (f & 31)));
  return ok;
}

}  // namespace cfft
