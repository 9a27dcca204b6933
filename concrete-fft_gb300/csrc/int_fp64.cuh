// int_fp64.cuh -- IEEE binary64 sums and differences on the integer pipes.
//
// GB300 issues FP64 instructions at 1/64 of its FP32/INT32 rate: one warp
// instruction per ~76 cycles of an SM sub-partition, and every FFT kernel of
// this library was bound by it.  A butterfly adds and subtracts the same two
// values, so sum_diff_int computes both with 32-bit integer instructions: the
// operands are unpacked and aligned once, and only the two roundings are
// separate.  About 73 instructions (52 on the ALU pipe, 2 cycles each) replace
// two FP64 instructions (152 cycles), and the FP64 pipe is left to the
// products.  The results are the IEEE-754 values (round to nearest even), bit
// for bit.
//
// Method: both 53-bit significands go to bits 62..10 of a 64-bit word, the
// smaller operand's shifted right by the exponent difference; up to a
// difference of 10 no bit is lost, so sum and difference are exact integers.
// The sum's leading one is at bit 62 or 63, the difference's is found with one
// count of leading zeros; each is shifted to 53 bits and rounded to nearest
// even, and the rounding carry runs into the exponent field by one addition.
//
// The caller computes the pair on the FP64 pipe when the operands leave that
// range: exponents more than 10 apart (1 pair in 1000 for Gaussian data),
// zeros, subnormals, infinities, NaNs, values near overflow, or a difference
// that loses 31 or more leading bits (exact cancellation among them).
#pragma once
#include <cstdint>

namespace cfft {

// Index of the leading one counted from bit 31 (x != 0; 0xffffffff for 0).
__device__ __forceinline__ uint32_t leading_zeros_nz(uint32_t x) {
  uint32_t r;
  asm("bfind.shiftamt.u32 %0, %1;" : "=r"(r) : "r"(x));
  return r;
}

// (h:l) += (base:0) + round, where u holds the discarded bits left-aligned
// with the kept last bit OR-ed into bit 0: the round is 1 iff u > 2^31, i.e.
// above half, or exactly half with an odd last bit.
__device__ __forceinline__ void round_and_pack(uint32_t& h, uint32_t& l, uint32_t base, uint32_t u) {
  uint32_t t;
  asm("add.cc.u32 %2, %4, 0x7fffffff;\n\taddc.cc.u32 %0, %0, 0;\n\taddc.u32 %1, %1, %3;"
      : "+r"(l), "+r"(h), "=r"(t)
      : "r"(base), "r"(u));
  (void)t;
}

// s = a + b and d = a - b.  False (s and d are then meaningless) when the
// operands are outside the range described above.
__device__ __forceinline__ bool sum_diff_int(double a, double b, double& s, double& d) {
  const uint32_t ah = (uint32_t)__double2hiint(a), al = (uint32_t)__double2loint(a);
  const uint32_t bh = (uint32_t)__double2hiint(b), bl = (uint32_t)__double2loint(b);
  // exponents in place (bits 20..30); dif = ea - eb
  const uint32_t xa = ah & 0x7ff00000u, xb = bh & 0x7ff00000u;
  const uint32_t e = max(xa, xb);
  const int dif = (int)(xa - xb) >> 20;
  bool ok = (uint32_t)(dif + 10) <= 20u;
  ok = ok && (e - (64u << 20)) < (0x7beu << 20);
  const uint32_t na = (uint32_t)min(dif + 10, 10), nb = (uint32_t)min(10 - dif, 10);
  const uint32_t ma = (ah & 0xfffffu) | 0x100000u, mb = (bh & 0xfffffu) | 0x100000u;
  const uint64_t A = ((uint64_t)__funnelshift_l(al, ma, na) << 32) | (al << (na & 31));
  const uint64_t B = ((uint64_t)__funnelshift_l(bl, mb, nb) << 32) | (bl << (nb & 31));
  const uint64_t S = A + B;  // magnitude of the like-signed result
  uint64_t D = A - B;        // magnitude of the unlike-signed one
  const bool swap = (int64_t)D < 0;
  if (swap) D = 0 - D;
  // exponent and sign words, less the hidden bit that the significand brings
  const uint32_t base = e + (ah & 0x80000000u) - 0x100000u;
  const uint32_t base_d = swap ? base + 0x80000000u : base;
  const uint32_t Sh = (uint32_t)(S >> 32), Sl = (uint32_t)S;
  const uint32_t c = Sh >> 31;  // carry: one more bit to drop, exponent + 1
  uint32_t sh = Sh >> (10 + c), sl = __funnelshift_r(Sl, Sh, 10 + c);
  round_and_pack(sh, sl, base + (c << 20), (Sl << (22 - c)) | (sl & 1));
  const uint32_t Dh = (uint32_t)(D >> 32), Dl = (uint32_t)D;
  ok = ok && Dh != 0;
  const uint32_t f = leading_zeros_nz(Dh);
  const uint32_t Nh = __funnelshift_l(Dl, Dh, f), Nl = Dl << (f & 31);
  uint32_t dh = Nh >> 11, dl = __funnelshift_r(Nl, Nh, 11);
  round_and_pack(dh, dl, base_d - (f << 20) + 0x100000u, (Nl << 21) | (dl & 1));
  const bool same = (int32_t)(ah ^ bh) >= 0;
  s = __hiloint2double((int)(same ? sh : dh), (int)(same ? sl : dl));
  d = __hiloint2double((int)(same ? dh : sh), (int)(same ? dl : sl));
  return ok;
}

// w * b, rounded to nearest even, where w and b are normal and so is the
// product (false otherwise).  The significands' 106-bit product comes from four
// 32 x 32 multiplications on the FMA pipe, w's shifted so that the product's
// leading one is at bit 52 or 51 of the upper 64 bits (one w serves several b).
__device__ __forceinline__ bool mul_int(double w, double b, double& p) {
  const uint32_t wh = (uint32_t)__double2hiint(w), wl = (uint32_t)__double2loint(w);
  const uint32_t bh = (uint32_t)__double2hiint(b), bl = (uint32_t)__double2loint(b);
  const uint32_t xw = wh & 0x7ff00000u, xb = bh & 0x7ff00000u;
  const uint32_t mw = (wh & 0xfffffu) | 0x100000u, mb = (bh & 0xfffffu) | 0x100000u;
  const uint32_t Wh = __funnelshift_l(wl, mw, 11), Wl = wl << 11;
  const uint64_t p00 = (uint64_t)Wl * bl;
  const uint64_t p01 = (uint64_t)Wl * mb + (p00 >> 32);
  const uint64_t p10 = (uint64_t)Wh * bl + (uint32_t)p01;
  const uint64_t P = (uint64_t)Wh * mb + (p01 >> 32) + (p10 >> 32);
  const uint32_t Ph = (uint32_t)(P >> 32), Pl = (uint32_t)P, R1 = (uint32_t)p10, R0 = (uint32_t)p00;
  // bring the leading one from bit 51 to bit 52 where it is there
  const uint32_t c = Ph >> 20, f = c ^ 1u;
  uint32_t ph = __funnelshift_l(Pl, Ph, f), pl = __funnelshift_l(R1, Pl, f);
  const uint32_t u = __funnelshift_l(R0, R1, f) | min(R0, 1u) | (pl & 1u);
  // biased exponent of the result less one (the hidden bit adds it back), in place
  const uint32_t x = xw + xb + (c << 20) - (1023u << 20);
  const bool ok = min(xw, xb) >= (1u << 20) && max(xw, xb) < (0x7ffu << 20) && x - (64u << 20) < (0x77eu << 20);
  round_and_pack(ph, pl, x - (1u << 20) + ((wh ^ bh) & 0x80000000u), u);
  p = __hiloint2double((int)ph, (int)pl);
  return ok;
}

// N sums and differences s[j] = a[j] + b[j], d[j] = a[j] - b[j]; the pairs in
// MASK run on the integer pipes, the others on the FP64 pipe.  Pairs outside
// sum_diff_int's range are redone on the FP64 pipe one by one in a loop: a
// loop, because the compiler turns a short conditional into predicated
// instructions, and an FP64 instruction whose lanes are all predicated off
// still takes its ~76 cycles of the pipe (measured: with a predicated
// fallback the integer path gains nothing).
template <int N, int MASK>
__device__ __forceinline__ void sum_diff(const double* a, const double* b, double* s, double* d) {
  uint32_t redo = 0;
#pragma unroll
  for (int j = 0; j < N; ++j) {
    if ((MASK >> j) & 1) {
      if (!sum_diff_int(a[j], b[j], s[j], d[j])) redo += 1u << j;
    } else {
      s[j] = __dadd_rn(a[j], b[j]);
      d[j] = __dsub_rn(a[j], b[j]);
    }
  }
  if constexpr (MASK != 0) {
    asm volatile("" : "+r"(redo));  // keeps the loop a loop where only one bit can be set
    while (redo) {
      const int i = 31 - __clz((int)redo);
      redo &= ~(1u << i);
      double x = a[0], y = b[0];
#pragma unroll
      for (int j = 1; j < N; ++j)
        if (i == j) x = a[j], y = b[j];
      const double ss = __dadd_rn(x, y), dd = __dsub_rn(x, y);
#pragma unroll
      for (int j = 0; j < N; ++j)
        if (i == j) s[j] = ss, d[j] = dd;
    }
  }
}

}  // namespace cfft
