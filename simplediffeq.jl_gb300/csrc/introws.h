/* The rows of the Runge-Kutta tableaus as the integer-pipe kernels walk them:
 * each row is a linear combination of earlier stages (intchain.h) and the
 * stage it gives.  Rows follow the order of the methods' attempt and
 * dense_stages functions (ode_solver.cuh), terms the order they accumulate in. */
#pragma once
#include "intchain.h"
#include "tableaus.h"

namespace gbode {

/* n terms; the stage the right-hand side fills at t + c dt (-1: the new state,
 * no evaluation); coefficients (positions in the table) and their stages */
struct IcSpec {
  int n, out;
  double c;
  int coef[10], k[10];
};
constexpr IcSpec kSpecT5[] = {
    {1, 1, gbtab::tsit5::c1, {tsit5_a21}, {0}},
    {2, 2, gbtab::tsit5::c2, {tsit5_a31, tsit5_a32}, {0, 1}},
    {3, 3, gbtab::tsit5::c3, {tsit5_a41, tsit5_a42, tsit5_a43}, {0, 1, 2}},
    {4, 4, gbtab::tsit5::c4, {tsit5_a51, tsit5_a52, tsit5_a53, tsit5_a54}, {0, 1, 2, 3}},
    {5, 5, 1.0, {tsit5_a61, tsit5_a62, tsit5_a63, tsit5_a64, tsit5_a65}, {0, 1, 2, 3, 4}},
    {6, 6, 1.0, {tsit5_a71, tsit5_a72, tsit5_a73, tsit5_a74, tsit5_a75, tsit5_a76}, {0, 1, 2, 3, 4, 5}}};
constexpr IcSpec kSpecV7[] = {
    {1, 1, gbtab::vern7::c2, {vern7_a021}, {0}},
    {2, 2, gbtab::vern7::c3, {vern7_a031, vern7_a032}, {0, 1}},
    {2, 3, gbtab::vern7::c4, {vern7_a041, vern7_a043}, {0, 2}},
    {3, 4, gbtab::vern7::c5, {vern7_a051, vern7_a053, vern7_a054}, {0, 2, 3}},
    {4, 5, gbtab::vern7::c6, {vern7_a061, vern7_a063, vern7_a064, vern7_a065}, {0, 2, 3, 4}},
    {5, 6, gbtab::vern7::c7, {vern7_a071, vern7_a073, vern7_a074, vern7_a075, vern7_a076}, {0, 2, 3, 4, 5}},
    {6, 7, gbtab::vern7::c8, {vern7_a081, vern7_a083, vern7_a084, vern7_a085, vern7_a086, vern7_a087}, {0, 2, 3, 4,
     5, 6}},
    {7, 8, 1.0, {vern7_a091, vern7_a093, vern7_a094, vern7_a095, vern7_a096, vern7_a097, vern7_a098}, {0, 2, 3, 4, 5,
     6, 7}},
    {6, 9, 1.0, {vern7_a101, vern7_a103, vern7_a104, vern7_a105, vern7_a106, vern7_a107}, {0, 2, 3, 4, 5, 6}},
    {7, -1, 1.0, {vern7_b1, vern7_b4, vern7_b5, vern7_b6, vern7_b7, vern7_b8, vern7_b9}, {0, 3, 4, 5, 6, 7, 8}}};
/* the extra dense-output stages; stages as the staging rings number them: the
 * first, those from 1 + DSKIP on, then the extra ones (ode_solver.cuh) */
constexpr IcSpec kSpecV7X[] = {
    {7, 7, gbtab::vern7x::c11, {vern7x_a1101, vern7x_a1104, vern7x_a1105, vern7x_a1106, vern7x_a1107, vern7x_a1108,
     vern7x_a1109}, {0, 1, 2, 3, 4, 5, 6}},
    {8, 8, gbtab::vern7x::c12, {vern7x_a1201, vern7x_a1204, vern7x_a1205, vern7x_a1206, vern7x_a1207, vern7x_a1208,
     vern7x_a1209, vern7x_a1211}, {0, 1, 2, 3, 4, 5, 6, 7}},
    {9, 9, gbtab::vern7x::c13, {vern7x_a1301, vern7x_a1304, vern7x_a1305, vern7x_a1306, vern7x_a1307, vern7x_a1308,
     vern7x_a1309, vern7x_a1311, vern7x_a1312}, {0, 1, 2, 3, 4, 5, 6, 7, 8}},
    {10, 10, gbtab::vern7x::c14, {vern7x_a1401, vern7x_a1404, vern7x_a1405, vern7x_a1406, vern7x_a1407, vern7x_a1408,
     vern7x_a1409, vern7x_a1411, vern7x_a1412, vern7x_a1413}, {0, 1, 2, 3, 4, 5, 6, 7, 8, 9}},
    {10, 11, gbtab::vern7x::c15, {vern7x_a1501, vern7x_a1504, vern7x_a1505, vern7x_a1506, vern7x_a1507, vern7x_a1508,
     vern7x_a1509, vern7x_a1511, vern7x_a1512, vern7x_a1513}, {0, 1, 2, 3, 4, 5, 6, 7, 8, 9}},
    {10, 12, gbtab::vern7x::c16, {vern7x_a1601, vern7x_a1604, vern7x_a1605, vern7x_a1606, vern7x_a1607, vern7x_a1608,
     vern7x_a1609, vern7x_a1611, vern7x_a1612, vern7x_a1613}, {0, 1, 2, 3, 4, 5, 6, 7, 8, 9}}};

struct IcRow {
  int first, n, out; /* terms [first, first + n), the stage filled */
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
IC_CX bool ic_consecutive(const IcSpec (&s)[NR]) {
  for (int r = 0; r < NR; ++r)
    for (int j = 0; j < s[r].n; ++j)
      if (s[r].k[j] != j) return false;
  return true;
}
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
    t.row[r].out = s[r].out;
    t.row[r].emax = emax;
    t.row[r].shift = 0;
    t.row[r].c = s[r].c;
    for (int j = 0; j < s[r].n; ++j, ++at) {
      t.term[at] = ic_make_term(v[s[r].coef[j]], s[r].k[j], emax);
      t.coef[at] = v[s[r].coef[j]];
      const int sh = (int)t.term[at].shift;
      t.row[r].shift = sh > t.row[r].shift ? sh : t.row[r].shift;
    }
  }
  return t;
}

constexpr double kValT5[] = GBTAB_TSIT5_INIT;
constexpr double kValV7[] = GBTAB_VERN7_INIT;
constexpr double kValV7X[] = GBTAB_VERN7X_INIT;

#if defined(__CUDACC__) || defined(__CUDACC_RTC__)
/* a table in constant memory, its rows and terms by position, and whether term j of a row multiplies stage j */
#define GBODE_IC_TABLE(NAME, SPEC, VAL)                                                                     \
  __constant__ IcTable<sizeof(SPEC) / sizeof(SPEC[0]), ic_count(SPEC)> c_##NAME =                           \
      ic_make_table<ic_count(SPEC)>(SPEC, VAL);                                                             \
  struct NAME {                                                                                             \
    enum { NR = sizeof(SPEC) / sizeof(SPEC[0]), CONSECUTIVE = ic_consecutive(SPEC) };                       \
    __device__ static __forceinline__ const IcRow& row(int r) { return c_##NAME.row[r]; }                   \
    __device__ static __forceinline__ const IcTerm& term(int i) { return c_##NAME.term[i]; }                \
    __device__ static __forceinline__ double coef(int i) { return c_##NAME.coef[i]; }                       \
  };
GBODE_IC_TABLE(IcT5, kSpecT5, kValT5)
GBODE_IC_TABLE(IcV7, kSpecV7, kValV7)
GBODE_IC_TABLE(IcV7X, kSpecV7X, kValV7X)
#undef GBODE_IC_TABLE
#endif

}  // namespace gbode
