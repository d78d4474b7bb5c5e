/* The sine and cosine polynomials of a reduced argument on the integer pipe.
 *
 * The results are those of the Horner steps
 *   p = fma(p, z, c)
 * in IEEE double, bit for bit, without a floating-point instruction (a double
 * operation holds this GPU's FP64 pipe for 64 cycles a warp; a step here is
 * about 14 integer instructions).  Both series alternate in sign and their
 * terms fall by 2^5 and more for z = r^2 < 0.62, so every partial value has
 * the binary exponent of the coefficient just added, known at compile time: a
 * step is |c| - |p| z in fixed point at that coefficient's scale, 53 bits and
 * 32 below them, and rounding to nearest is adding half a unit (in the
 * constant) and dropping the lower word.  The product's bits below the window
 * are cut off, so the exact value lies less than a unit of the window under
 * the computed one; only a lower word of 0 leaves the rounding undecided.
 *
 * Compiled by nvcc / NVRTC for the kernels and by a host C++ compiler for the
 * CPU test that checks it against fma(). */
#pragma once
#include "intchain.h"

namespace gbode {

/* (s2, s1, s0) = (c2, c1, c0) - (b2, b1, b0) */
IC_FN void ip_sub3(ic_u32& s2, ic_u32& s1, ic_u32& s0, ic_u32 c2, ic_u32 c1, ic_u32 c0, ic_u32 b2, ic_u32 b1,
                   ic_u32 b0) {
#if defined(__CUDACC__) || defined(__CUDACC_RTC__)
  asm("sub.cc.u32 %0, %3, %6;\n\tsubc.cc.u32 %1, %4, %7;\n\tsubc.u32 %2, %5, %8;"
      : "=&r"(s0), "=&r"(s1), "=r"(s2) : "r"(c0), "r"(c1), "r"(c2), "r"(b0), "r"(b1), "r"(b2));
#else
  const ic_u64 c = ((ic_u64)c1 << 32) | c0, b = ((ic_u64)b1 << 32) | b0;
  s2 = c2 - b2 - (c < b ? 1u : 0u);
  s1 = (ic_u32)((c - b) >> 32);
  s0 = (ic_u32)(c - b);
#endif
}

/* z's significand moved up by 10 bits, and minus its exponent */
struct IpArg {
  ic_u32 a1, a0, e;
};

/* m <- round53(|c| - m z): m, the significand of a value of exponent EP, and
 * c as the significand C of exponent EC; undecided sets bad */
template <int EP, int EC>
IC_FN void ip_step(ic_u32& m1, ic_u32& m0, const IpArg& z, ic_u64 C, bool& bad) {
  const ic_u64 t = (ic_u64)z.a1 * m0 + ((ic_u64)z.a0 * m1 + ic_mulhi(z.a0, m0));
  const ic_u64 w = (ic_u64)z.a1 * m1 + (t >> 32);
  const ic_u32 p2 = (ic_u32)(w >> 32), p1 = (ic_u32)w, p0 = (ic_u32)t;
  const ic_u32 s = z.e + (ic_u32)(EC - EP - 2);
  ic_u32 s0;
  ip_sub3(m1, m0, s0, (ic_u32)(C >> 32), (ic_u32)C, 0x80000000u, ic_shr(p2, 0u, s), ic_shr(p1, p2, s),
          ic_shr(p0, p1, s));
  bad = bad || s0 == 0u;
}

/* significand of a double, hidden bit included */
IC_CX ic_u64 ip_sig(double c) { return (ic_bits(c) & 0xfffffffffffffULL) | 0x10000000000000ULL; }
IC_CX int ip_exp(double c) { return ic_exp(c) - 1023; }

/* sincos_cw's polynomials (near-minimax, gen_sincos.py), highest degree first */
#define GBODE_SIN_C0 0x1.5d8fd0a40698ep-33
#define GBODE_SIN_C1 -0x1.ae5e5a8d61ce7p-26
#define GBODE_SIN_C2 0x1.71de3567ccfe8p-19
#define GBODE_SIN_C3 -0x1.a01a019bfde60p-13
#define GBODE_SIN_C4 0x1.111111110f7d0p-7
#define GBODE_SIN_C5 -0x1.5555555555548p-3
#define GBODE_COS_C0 0x1.1b8b9800ee7dap-29
#define GBODE_COS_C1 -0x1.27df4604d6713p-22
#define GBODE_COS_C2 0x1.a019f81ca810ap-16
#define GBODE_COS_C3 -0x1.6c16c1640a98bp-10
#define GBODE_COS_C4 0x1.555555554f0a9p-5
#define GBODE_COS_C5 -0x1.fffffffffff96p-2

#define GBODE_IP_STEP(m, P, C) ip_step<ip_exp(P), ip_exp(C)>(m##1, m##0, a, ip_sig(C), bad)
/* ps = the sine polynomial at z, cr = 1 + z (the cosine polynomial at z), for
 * 2^-26 <= z < 1; false if a step was undecided (or z lies outside) */
IC_FN bool ip_sincos(double z, double* ps, double* cr) {
  const ic_u32 zh = ic_hi(z), zl = ic_lo(z);
  const IpArg a = {ic_shl(zl, (zh & 0xfffffu) | 0x100000u, 10), zl << 10, 1023u - (zh >> 20)};
  bool bad = a.e - 1u > 25u;
  ic_u32 s1 = (ic_u32)(ip_sig(GBODE_SIN_C0) >> 32), s0 = (ic_u32)ip_sig(GBODE_SIN_C0);
  ic_u32 c1 = (ic_u32)(ip_sig(GBODE_COS_C0) >> 32), c0 = (ic_u32)ip_sig(GBODE_COS_C0);
  GBODE_IP_STEP(s, GBODE_SIN_C0, GBODE_SIN_C1);
  GBODE_IP_STEP(c, GBODE_COS_C0, GBODE_COS_C1);
  GBODE_IP_STEP(s, GBODE_SIN_C1, GBODE_SIN_C2);
  GBODE_IP_STEP(c, GBODE_COS_C1, GBODE_COS_C2);
  GBODE_IP_STEP(s, GBODE_SIN_C2, GBODE_SIN_C3);
  GBODE_IP_STEP(c, GBODE_COS_C2, GBODE_COS_C3);
  GBODE_IP_STEP(s, GBODE_SIN_C3, GBODE_SIN_C4);
  GBODE_IP_STEP(c, GBODE_COS_C3, GBODE_COS_C4);
  GBODE_IP_STEP(s, GBODE_SIN_C4, GBODE_SIN_C5);
  GBODE_IP_STEP(c, GBODE_COS_C4, GBODE_COS_C5);
  /* 1 - z |p| lies below 1: the significand of 1 at the exponent of 1/2 */
  ip_step<ip_exp(GBODE_COS_C5), -1>(c1, c0, a, 0x20000000000000ULL, bad);
  /* the hidden bit adds one to the exponent fields */
  *ps = ic_double(s1 + (0x80000000u | (ic_u32)(1022 + ip_exp(GBODE_SIN_C5)) << 20), s0);
  *cr = ic_double(c1 + (1021u << 20), c0);
  return !bad;
}
#undef GBODE_IP_STEP

}  // namespace gbode
