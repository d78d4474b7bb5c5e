/* The rows of Tsitouras 5(4) as the integer-pipe kernels walk them: each row is
 * a linear combination of earlier stages (intchain.h) and the stage it gives.
 * Rows follow the order of MTsit5::attempt (ode_solver.cuh), terms the order
 * they accumulate in. */
#pragma once
#include "intchain.h"
#include "tableaus.h"

namespace gbode {

/* n coefficients (positions in the table), of stages 0 .. n - 1; the right-hand
 * side fills the next stage at t + c dt */
struct IcSpec {
  int n;
  double c;
  int coef[6];
};
constexpr IcSpec kSpecT5[] = {
    {1, gbtab::tsit5::c1, {tsit5_a21}},
    {2, gbtab::tsit5::c2, {tsit5_a31, tsit5_a32}},
    {3, gbtab::tsit5::c3, {tsit5_a41, tsit5_a42, tsit5_a43}},
    {4, gbtab::tsit5::c4, {tsit5_a51, tsit5_a52, tsit5_a53, tsit5_a54}},
    {5, 1.0, {tsit5_a61, tsit5_a62, tsit5_a63, tsit5_a64, tsit5_a65}},
    {6, 1.0, {tsit5_a71, tsit5_a72, tsit5_a73, tsit5_a74, tsit5_a75, tsit5_a76}}};

struct IcRow {
  int first, n;      /* terms [first, first + n) */
  int emax, shift;   /* the largest biased exponent of the coefficients, the largest shift of a term */
  double c;
};
template <int NR, int NT>
struct IcTable {
  IcRow row[NR];
  IcTerm term[NT];
  double coef[NT]; /* the same coefficients, for the floating-point chain */
};
template <int NR>
IC_CX int ic_count(const IcSpec (&s)[NR]) {
  int n = 0;
  for (int r = 0; r < NR; ++r) n += s[r].n;
  return n;
}
template <int NT, int NR, int NV>
IC_CX IcTable<NR, NT> ic_make_table(const IcSpec (&s)[NR], const double (&v)[NV]) {
  IcTable<NR, NT> t{};
  int at = 0;
  for (int r = 0; r < NR; ++r) {
    int emax = 0;
    for (int j = 0; j < s[r].n; ++j) emax = ic_exp(v[s[r].coef[j]]) > emax ? ic_exp(v[s[r].coef[j]]) : emax;
    t.row[r].first = at;
    t.row[r].n = s[r].n;
    t.row[r].emax = emax;
    t.row[r].shift = 0;
    t.row[r].c = s[r].c;
    for (int j = 0; j < s[r].n; ++j, ++at) {
      t.term[at] = ic_make_term(v[s[r].coef[j]], emax);
      t.coef[at] = v[s[r].coef[j]];
      const int sh = (int)t.term[at].shift;
      t.row[r].shift = sh > t.row[r].shift ? sh : t.row[r].shift;
    }
  }
  return t;
}

constexpr double kValT5[] = GBTAB_TSIT5_INIT;

#if defined(__CUDACC__) || defined(__CUDACC_RTC__)
constexpr int kRowsT5 = sizeof(kSpecT5) / sizeof(kSpecT5[0]), kTermsT5 = ic_count(kSpecT5);
__constant__ IcTable<kRowsT5, kTermsT5> c_ic_t5 = ic_make_table<kTermsT5>(kSpecT5, kValT5);
#endif

}  // namespace gbode
