/* Linear combinations c1 k1 + c2 k2 + ... of doubles on the integer pipe.
 *
 * The result is that of the chain of IEEE operations
 *   s = c1 * k1;  s = fma(c2, k2, s);  s = fma(c3, k3, s);  ...
 * bit for bit, every step rounded to nearest even, without a floating-point
 * instruction.  On this GPU a warp's double operation holds the FP64 pipe of
 * its SM sub-partition for 64 cycles, while the integer pipes stand idle (the
 * adaptive Lorenz kernel: FP64 pipe 85% busy, an instruction issued in 15% of
 * cycles).  A step of the chain takes about 38 integer instructions, half of
 * them on the half-rate ALU, so it costs less than the multiply-add it
 * replaces and runs beside the others.
 *
 * The sum is a 96-bit two's complement fixed-point number whose scale is set
 * by the row's largest coefficient and the component's largest stage, so that
 * products need only a right shift.  The products' lowest bits are cut off
 * (towards minus infinity), which leaves the exact sum within one unit above
 * the computed one; a step is rounded by adding half an ulp and clearing the
 * bits below, and where that unit could change the result, or the sum lies
 * at a tie, or has lost more leading bits than the number holds, the step is
 * "undecided" and the caller repeats the row with multiply-adds (2 in 10^4
 * components of a Lorenz solve's final rows, fewer of the others).
 *
 * Compiled by nvcc / NVRTC for the kernels and by a host C++ compiler for the
 * CPU test that checks the chain against fma(). */
#pragma once

#if defined(__CUDACC__) || defined(__CUDACC_RTC__)
#define IC_FN __device__ __forceinline__
#define IC_CX __host__ __device__ constexpr
#else
#define IC_FN static inline
#define IC_CX constexpr
#endif

namespace gbode {

typedef unsigned int ic_u32;
typedef unsigned long long ic_u64;

/* A coefficient c of a row as the chain uses it: |c| as a 53-bit integer moved
 * up by 7 bits less the distance of its exponent from the row's largest
 * (emax, biased), so that the row's products share one scale; what is left of
 * a distance beyond 7 bits is a right shift of the product.  neg_k is c's sign
 * bit and, below it, the stage that c multiplies. */
struct IcTerm {
  ic_u32 a1, a0;
  ic_u32 shift;
  ic_u32 neg_k;
};
IC_CX ic_u64 ic_bits(double x) { return __builtin_bit_cast(ic_u64, x); }
IC_CX int ic_exp(double x) { return (int)(ic_bits(x) >> 52) & 0x7ff; }
IC_CX IcTerm ic_make_term(double c, int k, int emax) {
  const int dist = emax - ic_exp(c), up = dist < 7 ? 7 - dist : 0;
  const ic_u64 m = ((ic_bits(c) & 0xfffffffffffffULL) | 0x10000000000000ULL) << up;
  return {(ic_u32)(m >> 32), (ic_u32)m, (ic_u32)(dist < 7 ? 0 : dist - 7), ((ic_bits(c) >> 63) ? 0x80000000u : 0u) | (ic_u32)k};
}

#if defined(__CUDACC__) || defined(__CUDACC_RTC__)
IC_FN ic_u32 ic_shl(ic_u32 lo, ic_u32 hi, ic_u32 s) { return __funnelshift_l(lo, hi, s); }
IC_FN ic_u32 ic_shr(ic_u32 lo, ic_u32 hi, ic_u32 s) { return __funnelshift_r(lo, hi, s); }
IC_FN ic_u32 ic_shr0(ic_u32 x, ic_u32 s) { ic_u32 r; asm("shr.u32 %0, %1, %2;" : "=r"(r) : "r"(x), "r"(s)); return r; }
IC_FN ic_u32 ic_lzs(ic_u32 x) { ic_u32 r; asm("bfind.shiftamt.s32 %0, %1;" : "=r"(r) : "r"(x)); return r; }
IC_FN void ic_add3(ic_u32& s2, ic_u32& s1, ic_u32& s0, ic_u32 b2, ic_u32 b1, ic_u32 b0) {
  asm("add.cc.u32 %0, %0, %3;\n\taddc.cc.u32 %1, %1, %4;\n\taddc.u32 %2, %2, %5;"
      : "+r"(s0), "+r"(s1), "+r"(s2) : "r"(b0), "r"(b1), "r"(b2));
}
IC_FN ic_u32 ic_mulhi(ic_u32 a, ic_u32 b) { return __umulhi(a, b); }
IC_FN ic_u32 ic_hi(double x) { return (ic_u32)__double2hiint(x); }
IC_FN ic_u32 ic_lo(double x) { return (ic_u32)__double2loint(x); }
IC_FN double ic_double(ic_u32 hi, ic_u32 lo) { return __hiloint2double((int)hi, (int)lo); }
#else
IC_FN ic_u32 ic_shl(ic_u32 lo, ic_u32 hi, ic_u32 s) { return (ic_u32)(((((ic_u64)hi << 32) | lo) << (s & 31)) >> 32); }
IC_FN ic_u32 ic_shr(ic_u32 lo, ic_u32 hi, ic_u32 s) { return (ic_u32)((((ic_u64)hi << 32) | lo) >> (s & 31)); }
IC_FN ic_u32 ic_shr0(ic_u32 x, ic_u32 s) { return s > 31 ? 0 : x >> s; }
IC_FN ic_u32 ic_lzs(ic_u32 x) {
  if ((int)x < 0) x = ~x;
  if (x == 0) return 0xffffffffu;
  return (ic_u32)__builtin_clz(x);
}
IC_FN void ic_add3(ic_u32& s2, ic_u32& s1, ic_u32& s0, ic_u32 b2, ic_u32 b1, ic_u32 b0) {
  const ic_u64 l = (((ic_u64)s1 << 32) | s0), m = l + (((ic_u64)b1 << 32) | b0);
  s2 += b2 + (m < l ? 1u : 0u);
  s1 = (ic_u32)(m >> 32);
  s0 = (ic_u32)m;
}
IC_FN ic_u32 ic_mulhi(ic_u32 a, ic_u32 b) { return (ic_u32)(((ic_u64)a * b) >> 32); }
IC_FN ic_u32 ic_hi(double x) { return (ic_u32)(ic_bits(x) >> 32); }
IC_FN ic_u32 ic_lo(double x) { return (ic_u32)ic_bits(x); }
IC_FN double ic_double(ic_u32 hi, ic_u32 lo) { return __builtin_bit_cast(double, ((ic_u64)hi << 32) | lo); }
#endif

/* A chain's sum as a 96-bit two's complement integer of at most 53
 * significant bits, and whether a step could not be decided. */
struct IcSum {
  ic_u32 s2, s1, s0;
  bool bad;
};

/* The largest and smallest exponents of a component's stages: top = the
 * largest biased exponent << 21 | 0x1fffff, so that (top - 2 * high word)
 * >> 21 is a stage's distance from it whatever its sign; low = the smallest. */
struct IcSpan {
  ic_u32 top, low;
};
IC_FN ic_u32 ic_expo(ic_u32 hi) { return (hi >> 20) & 0x7ffu; }
IC_FN IcSpan ic_span(double k) {
  const ic_u32 e = ic_expo(ic_hi(k));
  return {e << 21 | 0x1fffffu, e};
}
IC_FN void ic_widen(IcSpan& E, double k) {
  const ic_u32 e = ic_expo(ic_hi(k)), top = e << 21 | 0x1fffffu;
  E.top = top > E.top ? top : E.top;
  E.low = e < E.low ? e : E.low;
}
/* whether the row's products all lie in the sum's window: no stage zero,
 * subnormal, infinite or NaN, and none more than 31 bits below the largest */
IC_FN bool ic_in_window(const IcSpan& E, int max_shift) {
  const ic_u32 e = E.top >> 21;
  return e - E.low + (ic_u32)max_shift <= 31u && e - 200u <= 1600u;
}

/* c k at the row's scale as a 96-bit two's complement integer, rounded
 * towards minus infinity, for a stage in the window of E */
struct IcProduct {
  ic_u32 q2, q1, q0;
};
IC_FN IcProduct ic_product(const IcTerm& c, double k, const IcSpan& E) {
  const ic_u32 kh = ic_hi(k), b0 = ic_lo(k), b1 = (kh & 0xfffffu) | 0x100000u;
  const ic_u32 m = (ic_u32)((int)(kh ^ c.neg_k) >> 31), sg = m | 1u;
  const ic_u32 d = ((E.top - 2u * kh) >> 21) + c.shift;
  const ic_u64 t = (ic_u64)c.a1 * b0 + ((ic_u64)c.a0 * b1 + ic_mulhi(c.a0, b0));
  const ic_u64 w = (ic_u64)c.a1 * b1 + (t >> 32);
  const ic_u32 p2 = (ic_u32)(w >> 32), p1 = (ic_u32)w, p0 = (ic_u32)t;
  /* x * sg + m is x or ~x: a multiply-add, which issues beside the shifts */
  return {ic_shr(p2, 0u, d) * sg + m, ic_shr(p1, p2, d) * sg + m, ic_shr(p0, p1, d) * sg + m};
}
/* S <- round53(S + q) */
IC_FN void ic_add_product(IcSum& S, const IcProduct& q) {
  ic_add3(S.s2, S.s1, S.s0, q.q2, q.q1, q.q0);
  /* the bits below the ulp: 32 - y of s0 for a leading bit 11 + y places from
   * the top of s2; none (undecided) when s2 holds no leading bit or an overflow */
  const ic_u32 y = ic_lzs(S.s2) - 11u;
  const ic_u32 mask = ic_shr0(0xffffffffu, y), half = ic_shr0(0x7fffffffu, y);
  ic_add3(S.s2, S.s1, S.s0, 0u, 0u, half);
  /* all but the last of them set: the exact sum may lie at or across the tie */
  S.bad = S.bad || (~S.s0 & mask & 0xfffffffeu) == 0u;
  S.s0 &= ~mask;
}

/* the sum as a double; emax: the row's largest coefficient exponent */
IC_FN double ic_result(const IcSum& S, const IcSpan& E, int emax) {
  const ic_u32 m = (ic_u32)((int)S.s2 >> 31);
  ic_u32 t2 = S.s2 ^ m, t1 = S.s1 ^ m, t0 = S.s0 ^ m;
  ic_add3(t2, t1, t0, 0u, 0u, m & 1u);
  const ic_u32 lz = ic_lzs(t2);
  const ic_u32 hi = ic_shl(t1, t2, lz - 11u), lo = ic_shl(t0, t1, lz - 11u);
  return ic_double((hi + (((E.top >> 21) + (ic_u32)(emax - 1008) - lz) << 20)) | (m & 0x80000000u), lo);
}

}  // namespace gbode
