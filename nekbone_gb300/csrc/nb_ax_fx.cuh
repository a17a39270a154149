// nb_ax_fx.cuh -- the FP64 element operator (ax_e, cg.f:142-168, with
// local_grad3 / local_grad3_t, cg.f:170-212) evaluated in 64-bit fixed
// point on the integer pipes instead of GB300's FP64 pipe.
//
// GB300 executes about 0.5e12 FP64 fused multiply-adds per second, but
// about 14e12 32x32->64-bit integer multiply-adds (mad.wide.s32) and 19e12
// simple integer operations (measured).  A product of two 60-bit
// fixed-point numbers built from three integer multiply-adds therefore
// costs a tenth of one DFMA.  So this operator keeps its values as block-floating-point
// integers and leaves only the CG vector arithmetic (p update, +0.1 p, pap)
// on the FP64 pipe:
//
//  * each element's input p is scaled by one power of two chosen from the
//    element's largest exponent and rounded to an integer P, |P| < 2^59
//    (to_fixed); the derivative tables are fixed-point integers with FC
//    fractional bits (|C| <= 2^59, rounded once on the host from D's exact
//    value); the metric g is converted once per solve, one exponent per
//    element (|G| < 2^60);
//  * a product a*b of two such integers is formed from balanced 32-bit
//    halves, a = ah 2^32 + al with al in [-2^31, 2^31):
//        a*b ~= ah*bh 2^64 + (ah*bl + al*bh) 2^32,
//    al*bl (|al*bl| <= 2^62, unbiased: al is symmetric) dropped.  In the
//    metric step the terms of one output are accumulated in int64 registers
//    (Acc) and combined once, rounded to units of 2^64 (hh + x / 2^32: the
//    high word of x, no shift; x starts at half a unit), so one output's
//    error is about one unit, ~2^-55 of its largest product -- the FP64
//    evaluation's own rounding of a 6-term sum.  In the six contraction
//    stages each cross term is a 32-bit mad.hi (its high word, units of
//    2^64) and the floors' mean loss is added back once (AccH): a few
//    units per output, for a fifth fewer instructions;
//  * the even-odd split of the GLL derivative (as k_ax_eo) halves the
//    products: per point and direction 6 multiply-adds at lx1 = 12;
//  * after the gradient and after the metric step the element's values are
//    renormalised by one shift (the element-wide OR of the magnitudes gives
//    the top bit), so every stage starts from ~58 significant bits of the
//    element's largest value;
//  * the result goes back to FP64 rounded to nearest even by the
//    integer-to-FP64 conversion (one FP64-pipe operation a point) and an
//    exact move of the exponent field; the input goes in by an exact FP64
//    scaling and the FP64-to-integer conversion (two more), where the FP64
//    pipe has room beside the integer work.
// Odd lx1 up to 11 takes a form with more bits (FxCoef): 50 CG iterations on
// 12 x 10 x 9 elements at lx1 = 9 in 2.96 ms, 9.05 with the reference-order
// operator on the FP64 pipe (4.28 when the operator alone had changed).
// This is block floating point: the error of a value is bounded relative to
// the largest value of its element (~2^-56), where FP64 bounds it relative
// to the value itself.  Results agree with the reference's FP64 evaluation
// to rounding (~1e-15 of the element's scale), not bit for bit.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "nb_kernels.cuh"

// CTAs per SM of the fixed-point operator at lx1 <= 12: its three
// shared-memory arrays (42 KB at lx1 = 12) allow five, and the bound keeps
// the registers within five (1.90 ms at 32^3, against 2.01 ms with four
// arrays and four CTAs, 2.25 ms with rows padded to lx1 + 1 and three).
// The output rows of a line are unrolled two at a time (fully unrolled,
// the kernel spills and measures slower).
#ifndef NB_FX_MINB
#define NB_FX_MINB 5
#endif
#ifndef NB_FX_AUNROLL
#define NB_FX_AUNROLL 2
#endif
#define NB_FX_PRAGMA(x) _Pragma(#x)
#define NB_FX_UNROLL(n) NB_FX_PRAGMA(unroll n)

namespace nb {
namespace fx {

typedef long long i64;
typedef unsigned long long u64;

// ------------------------------------------------------------ integers --
// balanced halves: x = hi * 2^32 + lo, lo in [-2^31, 2^31)
struct Sp {
  int lo, hi;
};
__device__ __forceinline__ Sp split(i64 x) {
  Sp s;
  const unsigned low = unsigned(u64(x));
  s.lo = int(low);
  s.hi = int(u64(x) >> 32) + int(low >> 31);
  return s;
}

// A sum of products a*b in units of 2^(64-K): hh counts ah*bh, x and x2 count
// ah*bl and al*bh in units of 2^32 (two accumulators: two dependency chains
// of half the length), x started at half a unit so that the high word of
// x + x2 rounds to nearest (al*bl dropped).  Each product is one 32x32 ->
// 64-bit multiply-add (mad.wide.s32), written in C++ so that a coefficient
// can stay a constant-bank operand.  For the three terms of the metric step.
// The FULL form (FxCoef) takes K = 3, three more bits of its outputs, and the
// high word of al*bl (|x + x2| <= 6 * 2^60 for |c|, |v| <= 2^61).
template <int K, bool FULL = false>
struct Acc {
  i64 hh, x, x2;
  __device__ __forceinline__ Acc() : hh(0), x(1ll << (31 - K)), x2(0) {}
  __device__ __forceinline__ void mac(const Sp &c, const Sp &v) {
    hh += i64(c.hi) * i64(v.hi);
    x += i64(c.hi) * i64(v.lo);
    x2 += i64(c.lo) * i64(v.hi);
    if (FULL) x += __mulhi(c.lo, v.lo);
  }
  __device__ __forceinline__ i64 result() const { return (hh << K) + ((x + x2) >> (32 - K)); }
};

// The same (K = 0) for the up to six terms of the FULL form's lines, |c| <=
// 2^61 and |v| <= 2^62: the al*bh of even and odd terms go to two
// accumulators, so that each sum stays within 64 bits (three terms of at most
// 2^61, six of at most 2^60), each rounded to units of 2^64.
struct AccF {
  i64 hh, x, x2[2];
  __device__ __forceinline__ AccF() : hh(0), x(1ll << 31), x2{1ll << 31, 1ll << 31} {}
  __device__ __forceinline__ void mac(int chi, int clo, const Sp &v, int m) {
    hh += i64(chi) * i64(v.hi);
    x += i64(chi) * i64(v.lo);
    x2[m & 1] += i64(clo) * i64(v.hi);
  }
  __device__ __forceinline__ i64 result(int) const {
    return hh + ((x >> 32) + ((x2[0] >> 32) + (x2[1] >> 32)));
  }
};

// The same sum with the two cross terms taken as high words only: each
// ah*bl and al*bh is one 32-bit mad.hi (floor of the product / 2^32, in
// units of 2^64) instead of a 64-bit mad.wide, and the floors' average loss
// of half a unit each is added back once (not for an all-zero sum, so that
// A 0 = 0 stays exact).  An output's error grows from about one unit to a
// few; in the contraction stages, where this form is used, the operator's
// difference from the FP64 reference evaluation stays within 10 % of the
// exact-cross-term form's (3.1e-15 instead of 2.8e-15 of max|w| at lx1 = 12,
// deformed), and the operator takes 1.63 instead of 1.88 ms at 32^3.  The
// metric step keeps Acc: its cross terms carry the error into every later
// stage (8e-15 with mad.hi there).
struct AccH {
  i64 hh;
  int x, x2;  // high words below 2^27 (|ah| < 2^28, |al| <= 2^31); the
              // lx1/2 <= 8 of them and x + x2 stay below 2^31
  __device__ __forceinline__ AccH() : hh(0), x(0), x2(0) {}
  __device__ __forceinline__ void mac(int chi, int clo, const Sp &v, int) {
    hh += i64(chi) * i64(v.hi);
    x = __mulhi(chi, v.lo) + x;
    x2 = __mulhi(clo, v.hi) + x2;
  }
  // nmac multiply-adds were made
  __device__ __forceinline__ i64 result(int nmac) const {
    return hh + i64(x + x2 + ((x | x2) != 0 ? nmac : 0));
  }
};

// v * 2^sh for 0 <= sh < 64.  After the gradient every output is below 2^59
// (lx1 products of |C| <= 2^59 and an even-odd sum below 2^60, in units of
// 2^64, lx1 <= 16; two bits more everywhere in the FULL form), so its
// renormalisation's shift is >= 0; after the metric step every output is below
// 2^56.6 (three products of |G| < 2^60 and a value below 2^59), so its shift
// is >= 2.  The FULL form's metric step leaves at most 3 * 2^61 (three products
// of |G| and a value of at most 2^61, in units of 2^61): its shift is >= -2
// (shift_to).  The operator checks both and reports a violation through the
// device error word.
__device__ __forceinline__ i64 shift_up(i64 v, int sh) { return i64(u64(v) << sh); }
// the same for -2 <= sh, rounded to nearest
__device__ __forceinline__ i64 shift_to(i64 v, int sh) {
  return sh >= 0 ? shift_up(v, sh) : (v + (1ll << (-sh - 1))) >> -sh;
}

// ----------------------------------------------------- FP64 <-> fixed --
__device__ __forceinline__ int bexp(double x) {
  return int((u64(__double_as_longlong(x)) >> 52) & 0x7FFu);
}

// x * 2^(1075 - emax + up) rounded to nearest (ties away from zero), for x
// whose biased exponent is <= emax: |result| < 2^(53 + up).  This and
// to_double are the conversions' fallbacks for exponents out of the fast
// forms' range; out of line, they leave the operator's code smaller (100 CG
// iterations at 32^3: 247.0 instead of 248.3 ms).
static __device__ __noinline__ i64 to_fixed(double x, int emax, int up) {
  const u64 b = u64(__double_as_longlong(x));
  const int e = int((b >> 52) & 0x7FFu);
  const u64 m = (b & 0xFFFFFFFFFFFFFull) | (e ? (1ull << 52) : 0ull);
  const int sh = (e ? e : 1) - emax + up;
  u64 mag;
  if (sh >= 0) mag = m << sh;
  else if (sh > -54) mag = ((m >> (-sh - 1)) + 1ull) >> 1;
  else mag = 0ull;
  return (b >> 63) ? -i64(mag) : i64(mag);
}

// W * 2^s rounded to the nearest FP64 value (ties to even)
static __device__ __noinline__ double to_double(i64 W, int s) {
  if (W == 0) return 0.0;
  const u64 sign = u64(W) & (1ull << 63);
  u64 mag = W < 0 ? u64(-W) : u64(W);
  const int lz = __clzll(i64(mag));
  mag <<= lz;                       // top bit at 63
  int ex = 63 - lz + s;             // unbiased exponent of the value
  u64 mant = mag >> 11;             // 53 bits
  const u64 rem = mag & 0x7FFull;
  if (rem > 0x400ull || (rem == 0x400ull && (mant & 1ull))) ++mant;
  if (mant >> 53) {
    mant >>= 1;
    ++ex;
  }
  int be = ex + 1023;
  if (be >= 2047) return __longlong_as_double(i64(sign | (0x7FFull << 52)));
  if (be <= 0) {  // subnormal: mant * 2^(ex - 52) with 2^-1074 as the unit
    const int rs = 1 - be;
    if (rs > 53) return __longlong_as_double(i64(sign));
    const u64 half = 1ull << (rs - 1), low = mant & ((1ull << rs) - 1ull);
    u64 q = mant >> rs;
    if (low > half || (low == half && (q & 1ull))) ++q;
    return __longlong_as_double(i64(sign | q));
  }
  return __longlong_as_double(i64(sign | (u64(be) << 52) | (mant & 0xFFFFFFFFFFFFFull)));
}


// W * 2^s, bitwise as to_double: the integer-to-FP64 conversion rounds |W|
// to 53 bits to nearest even, as to_double does, and the exponent field is
// then moved by s exactly; results that would be subnormal or overflow take
// to_double.  One FP64-pipe conversion instead of ~25 integer instructions
// (1.93 -> 1.88 ms for the operator at 32^3; the same conversion for
// to_fixed, at two FP64-pipe operations a value, changes the rounding of
// ties and was not kept).
__device__ __forceinline__ double to_double_cvt(i64 W, int s) {
  const double d = __ll2double_rn(W);
  const i64 b = __double_as_longlong(d);
  const int e = int((b >> 52) & 0x7FF);
  const int e2 = e + s;
  // (zero is looked for in W: a comparison of d is one more FP64 operation)
  if (W != 0 && e2 >= 1 && e2 <= 2046) return __longlong_as_double(b + (i64(s) << 52));
  return W == 0 ? 0.0 : to_double(W, s);
}
// x * 2^(1075 - emax + up) rounded to the nearest integer, ties to even
// (to_fixed rounds them away from zero), by an exact FP64 scaling and the
// FP64-to-integer conversion: two FP64-pipe operations instead of ~15
// integer instructions (1.63 -> 1.61 ms for the operator at 32^3)
__device__ __forceinline__ i64 to_fixed_cvt(double x, int emax, int up) {
  const int k = 1075 - emax + up;
  if (k > 1023 || k < -1022) return to_fixed(x, emax, up);  // 2^k not a normal double
  const double sc = __longlong_as_double(i64(k + 1023) << 52);
  return __double2ll_rn(x * sc);
}
// x * 2^(1022 + B - emax) rounded to nearest (halves away from zero), |result|
// <= 2^B, for x whose biased exponent is <= emax, on the integer pipes
template <int B>
__device__ __forceinline__ i64 to_fixed_bits(double x, int emax) {
  if (emax < 128) return to_fixed(x, emax, B - 53);  // (near the subnormals; uniform)
  const u64 b = u64(__double_as_longlong(x));
  const int e = int((b >> 52) & 0x7FFu);
  const int r = min(emax - e, 63);  // a zero (e = 0) shifts out
  const u64 m = ((b & 0xFFFFFFFFFFFFFull) | (1ull << 52)) << (B - 52);
  const i64 v = i64(((m >> r) + 1ull) >> 1), s = i64(b) >> 63;
  return (v ^ s) - s;
}
// ----------------------------------------------------- block reductions --
// lanes of warp w of an nt-thread block
__device__ __forceinline__ unsigned warp_mask(int nt, int w) {
  const int n = nt - 32 * w;
  return n >= 32 ? 0xFFFFFFFFu : ((1u << n) - 1u);
}

// ------------------------------------------------------------ operator --
// Derivative tables in fixed point, as balanced halves.  With h = lx1/2 and
// h1 = lx1 - h, the anti-centrosymmetric part of a matrix (D, then D^T) is E,
// h rows of h1 values, and O, h1 rows of h (row a):
//   y(a) = E ve + O vo,  y(n-1-a) = O vo - E ve;
// for odd lx1 the middle value of a line, its own mirror image, joins the
// sums (last column of E) and the middle output, which the antisymmetry
// leaves to the differences alone, the differences (last row of O).
//
// Even lx1 (FxCoef::FULL false): |coefficient| <= 2^59, |line value| < 2^59,
// cross terms as high words (AccH); the matrix's other part, the rounding
// (~1e-15) by which D misses the symmetry, is dropped.
// Odd lx1 up to 11 (FULL): these orders' other form is the reference's own
// FP64 sums, and this one is no less exact: |coefficient| <= 2^61 and
// |line value| < 2^61, cross terms in full (AccF), the metric to 61 bits and
// its products' low halves too (Acc), and the centrosymmetric remainder of D
// kept as one 32-bit coefficient more a product, in the unit of lo (dE, h1 rows
// of h1 values, and dO, h rows of h):
//   y(a) += dE ve + dO vo,  y(n-1-a) += dE ve - dO vo,
// rounded to nearest: a floor takes half a unit off every point, and CG makes
// much of a constant (x after 40 iterations at lx1 = 9, against quadruple
// precision: 8.4e-16 with floors, 3.1e-16 so, 3.2e-16 with FP64 sums; with the
// metric to 60 bits and its products' high halves alone 3.5e-16).
// A kernel parameter, read as multiply-add operands.
template <int LX>
struct FxCoef {
  static constexpr int H = LX / 2, H1 = LX - H;
  static constexpr bool FULL = LX % 2 != 0;
  static constexpr int Q = 4 * H * H1;                       // main values, D and D^T
  static constexpr int QD = FULL ? 2 * (H1 * H1 + H * H) : 1;  // remainders
  int hi[Q];
  int lo[Q];
  int d[QD];
  int fc;  // fractional bits: coefficient = (hi 2^32 + lo) 2^-fc
};
// bits of a line's values: |v| < 2^kLine (and of a block after renormalising)
template <int LX>
constexpr int fx_bits() { return FxCoef<LX>::FULL ? 61 : 59; }
// Bits of the metric's values: |G| <= 2^fx_gbits, of the element's largest.
constexpr int fx_gbits(int lx) { return lx % 2 != 0 ? 61 : 60; }

// ------------------------------------------------------ separable metric --
// A box of equal cubes (setup_g, prox_setup.f:27-52) has the same block in
// every element, G1 = G4 = G6 = v(i,j,k) and G2 = G3 = G5 = 0, with v a
// product of one-dimensional weights, v = s b_i b_j b_k.  There
//   D^T diag(v) D  along i  =  v K along i,   K(i,m) = sum_q D(q,i) b_q/b_i D(q,m),
// so w_L = v (K u along i + along j + along k): three contractions instead of
// six, no metric step and no metric read but one shared block.  k_sep_check
// establishes the form on the device, once per solve, from g itself (every
// element bitwise, the product to the rounding of its factors), and makes K in
// double-double from D and b as they are.  ok = 0: the general form.
// K is centrosymmetric but for the rounding (~1e-14) by which D and b miss
// their symmetry.  The centrosymmetric part is E and O, h x h each (row a),
// |coefficient| <= 2^61; the rest, dE and dO, is added in FP32, which has 24
// bits of it to spare and whose pipe is idle:
//   y(a) = E ve + O vo + dE ve + dO vo,  y(n-1-a) = E ve - O vo - dE ve + dO vo.
// Without the rest and with b made symmetric an apply was off by 2.7e-15 at
// lx1 = 12 and 5.5e-15 at 16 (random field, 2-norm against quadruple
// precision), with it 1.2e-16 and 1.4e-16, as the FP64 sums; x after 40
// iterations at lx1 = 12 by 2.7e-15 and 3.7e-16.
struct SepTables {
  int ok, fc;        // fc: fractional bits of the tables
  int pad[2];
  int4 tab[64];      // (hi, lo) of E, (hi, lo) of O
  float2 rest[64];   // dE, dO in units of 2^(32 - fc)
  double v[4096];
};

template <int LX>
struct FxShared {
  static constexpr int N = (LX * LX + 1) * LX;
  static constexpr int NT = FxCoef<LX>::FULL ? 1 : (LX / 2) * (LX / 2);
  alignas(16) int4 tab[NT];  // SepTables' tables
  float2 rest[NT];
  i64 A[N];
  i64 C[N];
  i64 D[N];
  int emax[24], gmax[24];
  // one pair for each of the two renormalisations (fx_or_post): a warp may
  // post the second while another still reads the first
  unsigned orl[2][24], orh[2][24];
  double red[32];
};

// Element arrays in shared memory: rows of lx1 8-byte words, planes lx1^2 + 1
// words apart.  The plane pitch is 1 modulo 16, so the r-lines that 16
// consecutive threads start (thread t: j = t / lx1, k = t mod lx1) fall on
// distinct banks; so do the own columns (i + lx1 j).
template <int LX>
__device__ __forceinline__ int fx_at(int i, int j, int k) {
  return i + LX * j + (LX * LX + 1) * k;
}

// y(0..n-1) = C v of one line v (fixed point, |v| < 2^fx_bits), matrix tr of
// cf (0 D, 1 D^T); y in units of 2^64 of the products, handed to put(m,
// y(m)) as soon as each pair y(a), y(n-1-a) is formed (no output array stays
// live).  |y| < 2^59 (2^60 in the FULL form: the rows of D and of D^T sum to
// at most three times the largest coefficient).
template <int LX, typename Put>
__device__ __forceinline__ void fx_line(const i64 *v, const FxCoef<LX> &cf, int tr, Put put) {
  constexpr int H = LX / 2, H1 = LX - H;
  constexpr bool FULL = FxCoef<LX>::FULL;
  typedef typename std::conditional<FULL, AccF, AccH>::type A;
  const int qe0 = tr * 2 * H * H1, qo0 = qe0 + H * H1;
  const int de0 = tr * (H1 * H1 + H * H), do0 = de0 + H1 * H1;
  Sp ve[H1], vo[H];
#pragma unroll
  for (int m = 0; m < H; ++m) {
    ve[m] = split(v[m] + v[LX - 1 - m]);
    vo[m] = split(v[m] - v[LX - 1 - m]);
  }
  if constexpr (H1 > H) ve[H1 - 1] = split(v[H]);
  NB_FX_UNROLL(NB_FX_AUNROLL)
  for (int a = 0; a < H; ++a) {
    A e, o;
#pragma unroll
    for (int m = 0; m < H1; ++m) e.mac(cf.hi[qe0 + a * H1 + m], cf.lo[qe0 + a * H1 + m], ve[m], m);
#pragma unroll
    for (int m = 0; m < H; ++m) o.mac(cf.hi[qo0 + a * H + m], cf.lo[qo0 + a * H + m], vo[m], m);
    const i64 ye = e.result(H1), yo = o.result(H);
    if constexpr (FULL) {
      i64 ze = 1ll << 31, zo = 0;
#pragma unroll
      for (int m = 0; m < H1; ++m) ze += i64(cf.d[de0 + a * H1 + m]) * i64(ve[m].hi);
#pragma unroll
      for (int m = 0; m < H; ++m) zo += i64(cf.d[do0 + a * H + m]) * i64(vo[m].hi);
      put(a, ye + yo + ((ze + zo) >> 32));
      put(LX - 1 - a, yo - ye + ((ze - zo) >> 32));
    } else {
      put(a, ye + yo);
      put(LX - 1 - a, yo - ye);
    }
  }
  if constexpr (FULL) {  // the middle output
    A o;
    i64 ze = 1ll << 31;
#pragma unroll
    for (int m = 0; m < H; ++m)
      o.mac(cf.hi[qo0 + H * H + m], cf.lo[qo0 + H * H + m], vo[m], m);
#pragma unroll
    for (int m = 0; m < H1; ++m) ze += i64(cf.d[de0 + H * H1 + m]) * i64(ve[m].hi);
    put(H, o.result(H) + (ze >> 32));
  }
}

// y = K v of one line, |v| < 2^60 (SepTables)
template <int LX, typename Put>
__device__ __forceinline__ void fx_line_sep(const i64 *v, const int4 *tab, const float2 *rest,
                                            Put put) {
  constexpr int H = LX / 2;
  Sp ve[H], vo[H];
  float fe[H], fo[H];
#pragma unroll
  for (int m = 0; m < H; ++m) {
    ve[m] = split(v[m] + v[LX - 1 - m]);
    vo[m] = split(v[m] - v[LX - 1 - m]);
    fe[m] = float(ve[m].hi);
    fo[m] = float(vo[m].hi);
  }
#pragma unroll 1
  for (int a = 0; a < H; ++a) {
    Acc<0> e, o;
    float ze = 0.f, zo = 0.f;
#pragma unroll
    for (int m = 0; m < H; ++m) {
      const int4 c = tab[a * H + m];
      const float2 d = rest[a * H + m];
      e.mac(Sp{c.y, c.x}, ve[m]);
      o.mac(Sp{c.w, c.z}, vo[m]);
      ze = fma_rn(d.x, fe[m], ze);
      zo = fma_rn(d.y, fo[m], zo);
    }
    const i64 ye = e.result(), yo = o.result();
    put(a, ye + yo + i64(__float2int_rn(zo + ze)));
    put(LX - 1 - a, ye - yo + i64(__float2int_rn(zo - ze)));
  }
}

// OR of the magnitudes of a thread's values, combined over the block after
// the next __syncthreads (fx_or_read): its top bit is the largest's
__device__ __forceinline__ void fx_or_post(u64 v, unsigned *orl, unsigned *orh, int t, int nt) {
  const int w = t >> 5;
  const unsigned msk = warp_mask(nt, w);
  const unsigned l = __reduce_or_sync(msk, unsigned(v)), h = __reduce_or_sync(msk, unsigned(v >> 32));
  if ((t & 31) == 0) {
    orl[w] = l;
    orh[w] = h;
  }
}
// the shift that brings the block's largest magnitude below 2^bits
__device__ __forceinline__ int fx_or_shift(const unsigned *orl, const unsigned *orh, int nt,
                                           int bits) {
  u64 v = 0;
  for (int w = 0; w < (nt + 31) / 32; ++w) v |= (u64(orh[w]) << 32) | orl[w];
  if (v == 0) return 0;
  return bits - 1 - (63 - __clzll(i64(v)));
}
// the second renormalisation of a value (shift_up)
template <int LX>
__device__ __forceinline__ i64 fx_shift2(i64 v, int sh) {
  return FxCoef<LX>::FULL ? shift_to(v, sh) : shift_up(v, sh);
}
// one's complement magnitude: the same top bit as |v| (one lower for an
// exact negative power of two, which the bounds leave room for)
__device__ __forceinline__ u64 mag(i64 v) { return u64(v ^ (v >> 63)); }

// The end of element e at the thread's column (i, j): w_L of its point k is
// wloc(k) (bad: the element has a value that is not finite, which has no
// fixed-point form); the CG epilogue as k_ax_eo's.  Points k0 .. k0 + NK - 1,
// the thread's part of the reduction returned. 
template <int LX, int MODE, int NK, bool WHOLE, typename W>
__device__ __forceinline__ double ax_fx_finish(const AxArgs<double> &a, int e, int t, int k0,
                                               bool bad, unsigned nbr, W wloc) {
  constexpr int L2 = LX * LX, L3 = LX * LX * LX;
  const int i = t % LX, j = t / LX;
  const size_t base = size_t(e) * L3;
  // p (written above by this thread, so in cache), c and f are read again
  // here rather than held in registers through the contractions
  const bool col_interior = (i > 0) && (i < LX - 1) && (j > 0) && (j < LX - 1);
  double part = 0.0;
  double pk[NK], ck[NK], fk[NK];
  if (WHOLE || ((MODE == 1 || MODE == 2 || a.tenth) && col_interior)) {
#pragma unroll
    for (int q = 0; q < NK; ++q) {  // all loads before the first store
      const int k = k0 + q;
      if (k >= LX) break;
      const size_t id = base + size_t(k) * L2 + t;
      const bool interior = k > 0 && k < LX - 1;
      if (WHOLE || interior) pk[q] = MODE == 1 || MODE == 2 ? a.p[id] : a.u[id];
      if (!WHOLE && interior && (MODE == 1 || MODE == 2)) ck[q] = __ldg(a.c + id);
      if (MODE == 2 && interior) fk[q] = __ldg(a.f + id);
    }
  }
#pragma unroll
  for (int q = 0; q < NK; ++q) {
    const int k = k0 + q;
    if (k >= LX) break;
    double wl = wloc(k);
    if (bad) wl = __longlong_as_double(0x7FF8000000000000ll);
    const size_t id = base + size_t(k) * L2 + t;
    const bool interior = col_interior && (k > 0) && (k < LX - 1);
    if (WHOLE) {
      wl = fma_rn(box_tenth<double>(box_ext<LX>(i, j, k) & nbr), pk[q], wl);
      part = fma_rn(wl, pk[q], part);
      a.w[id] = wl;
    } else if (MODE == 1) {
      if (interior) {
        wl = fma_rn(0.1, pk[q], wl);
        part = fma_rn(mul_rn(wl, ck[q]), pk[q], part);
      }
      a.w[id] = wl;
    } else if (MODE == 2) {
      if (interior) {
        const double rv = fk[q] - fma_rn(0.1, pk[q], wl);
        a.r[id] = rv;
        part = fma_rn(mul_rn(rv, ck[q]), rv, part);
      } else {
        a.w[id] = wl;
      }
    } else {
      if (a.tenth && interior) wl = fma_rn(0.1, pk[q], wl);
      a.w[id] = wl;
    }
  }
  return part;
}

// ----------------------------------------------- separable-metric operator --
// The operator where SepTables' form holds (MODE 1 and 2 as ax_fx_body).  Two
// of the shared arrays: the element in fixed point (A), and the sum of the
// three directions' results (C), each direction's lines added by the threads
// that own them.  1.00 ms at 32^3, lx1 = 12, against 1.53 for the general
// form, 0.10 of it for K's part that is not centrosymmetric (SepTables).
// Measured without that part, 0.86 ms then, and left out: the result's
// conversion and product on the integer pipes (40 instructions for two FP64
// operations, 0.88 to 0.95 ms); two elements a CTA (0.88); a kernel of its own
// with six CTAs per SM (0.81 to 0.86, but 3 to 6 us a launch on small meshes,
// since the device decides which of the two runs).
template <int LX, int MODE>
__device__ __forceinline__ void ax_sep_body(const AxArgs<double> &a, FxShared<LX> &sm, bool whole,
                                            unsigned nbr, int fc) {
  constexpr int L2 = LX * LX, L3 = LX * LX * LX, NT = FxShared<LX>::NT;
  const int t = threadIdx.x + LX * threadIdx.y;
  const int i = threadIdx.x, j = threadIdx.y;  // own column (i,j)
  const int e = blockIdx.x;
  const size_t base = size_t(e) * L3;
  if (t < NT) {
    sm.tab[t] = a.sep->tab[t];
    sm.rest[t] = a.sep->rest[t];
  }

  int em = 0;
  {
    double uk[LX];
    const double beta = (MODE == 1 && !a.first) ? a.sc->beta : 0.0;
    constexpr int HB = LX / 2;
#pragma unroll
    for (int k0 = 0; k0 < LX; k0 += HB) {  // two halves: fewer values held at once
      double pold[HB];
#pragma unroll
      for (int q = 0; q < HB; ++q) {  // all loads before the first store
        const size_t id = base + size_t(k0 + q) * L2 + t;
        if (MODE == 1) {
          uk[k0 + q] = a.u[id];
          pold[q] = a.first ? 0.0 : a.pold[id];
        } else {
          uk[k0 + q] = a.p[id];
          pold[q] = a.e ? double(a.e[id]) : 0.0;
        }
      }
#pragma unroll
      for (int q = 0; q < HB; ++q) {
        const int k = k0 + q;
        const size_t id = base + size_t(k) * L2 + t;
        if (MODE == 1) {
          if (!a.first) uk[k] = fma_rn(beta, pold[q], uk[k]);  // add2s1, math.f:534
          a.p[id] = uk[k];
        } else if (a.e) {
          uk[k] = fma_rn(a.scale, pold[q], uk[k]);
          a.p[id] = uk[k];
        }
      }
    }
#pragma unroll
    for (int k = 0; k < LX; ++k) em = max(em, bexp(uk[k]));
    const int w = t >> 5;
    const int r = __reduce_max_sync(warp_mask(L2, w), unsigned(em));
    if ((t & 31) == 0) sm.emax[w] = r;
    __syncthreads();
    em = 0;
    for (int q = 0; q < (L2 + 31) / 32; ++q) em = max(em, sm.emax[q]);
    // (on the integer pipes: this form is held by the FP64 one)
#pragma unroll
    for (int k = 0; k < LX; ++k) sm.A[fx_at<LX>(i, j, k)] = to_fixed_bits<60>(uk[k], em);
  }
  __syncthreads();

  // K along j, then i, then k (the own column); run-time strides keep one copy
  // of the line code
#pragma unroll 1
  for (int d = 0; d < 3; ++d) {
    if (d) __syncthreads();
    const int b0 = d == 0 ? fx_at<LX>(i, 0, j) : d == 1 ? fx_at<LX>(0, j, i) : fx_at<LX>(i, j, 0);
    const int st = d == 0 ? LX : d == 1 ? 1 : (LX * LX + 1);
    i64 v[LX];
#pragma unroll
    for (int m = 0; m < LX; ++m) v[m] = sm.A[b0 + m * st];
    fx_line_sep<LX>(v, sm.tab, sm.rest, [&](int m, i64 y) {
      i64 *o = sm.C + b0 + m * st;
      *o = d ? *o + y : y;
    });
  }

  const int sY = em - 1075 - (60 - 53) + 64 - fc;
  const bool bad = em == 0x7FF;
  constexpr int NK = LX / 2;
  double part = 0.0;
#pragma unroll
  for (int k0 = 0; k0 < LX; k0 += NK) {
    double vk[NK];
#pragma unroll
    for (int q = 0; q < NK; ++q) vk[q] = __ldg(a.sep->v + (k0 + q) * L2 + t);
    auto wloc = [&](int k) {
      return mul_rn(to_double_cvt(sm.C[fx_at<LX>(i, j, k)], sY), vk[k - k0]);
    };
    if (MODE == 1 && whole)
      part += ax_fx_finish<LX, MODE, NK, MODE == 1>(a, e, t, k0, bad, nbr, wloc);
    else
      part += ax_fx_finish<LX, MODE, NK, false>(a, e, t, k0, bad, nbr, wloc);
  }
  const double s = block_sum<double>(part, sm.red);
  if (t == 0) a.partial[e] = s;
}

// MODE 0 / 1 / 2 as k_ax_eo (AxArgs), 3 as 0 from the metric a.g itself: the
// element's largest exponent first (its block read once, from L2 the second
// time), each value converted where it is used.  For a single apply: the
// conversion pass and its traffic (96 B a point written and read back) cost
// more than these 100 instructions a point (16^3, lx1 = 12: 247 us against 160
// for the conversion and 189 for mode 0).  a.gfx / a.gexp hold the metric in
// fixed point (metric_fx_prepare).
template <int LX, int MODE>
__device__ __forceinline__ void ax_fx_body(const AxArgs<double> &a, const FxCoef<LX> &cf) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  FxShared<LX> &sm = *reinterpret_cast<FxShared<LX> *>(smem_raw);
  constexpr int L2 = LX * LX, L3 = LX * LX * LX, BITS = fx_bits<LX>(), MK = FxCoef<LX>::FULL ? 3 : 0;
  const int t = threadIdx.x + LX * threadIdx.y;
  const int i = threadIdx.x, j = threadIdx.y;  // own column (i,j)
  const int e = blockIdx.x;
  const size_t base = size_t(e) * L3;
  const int fc = cf.fc;
  if (a.act && !a.act[size_t(a.el_prob[e]) * a.act_stride]) return;  // the whole CTA
  const bool whole = MODE == 1 && box_flag(a.box_ok);  // pap formed here (BoxMesh)
  const unsigned nbr = whole ? box_neighbours(a.box, e) : 0u;
  if constexpr ((MODE == 1 || MODE == 2) && !FxCoef<LX>::FULL) {
    const int2 sep = a.sep ? *reinterpret_cast<const int2 *>(a.sep) : make_int2(0, 0);
    if (sep.x) {
      ax_sep_body<LX, MODE>(a, sm, whole, nbr, sep.y);
      return;
    }
  }

  // direction update (MODE 1) / correction (MODE 2), in FP64, then the
  // element's exponent and its fixed-point block
  int em = 0;
  {
    double uk[LX];
    double pold[LX];
    const double beta = (MODE == 1 && !a.first) ? a.sc->beta : 0.0;
#pragma unroll
    for (int k = 0; k < LX; ++k) {  // all loads before the first store
      const size_t id = base + size_t(k) * L2 + t;
      if (MODE == 1) {
        uk[k] = a.u[id];
        pold[k] = a.first ? 0.0 : a.pold[id];
      } else if (MODE == 2) {
        uk[k] = a.p[id];
        pold[k] = a.e ? double(a.e[id]) : 0.0;
      } else {
        uk[k] = a.u[id];
      }
    }
#pragma unroll
    for (int k = 0; k < LX; ++k) {
      const size_t id = base + size_t(k) * L2 + t;
      if (MODE == 1) {
        if (!a.first) uk[k] = fma_rn(beta, pold[k], uk[k]);  // add2s1, math.f:534
        a.p[id] = uk[k];
      } else if (MODE == 2 && a.e) {
        uk[k] = fma_rn(a.scale, pold[k], uk[k]);
        a.p[id] = uk[k];
      }
    }
#pragma unroll
    for (int k = 0; k < LX; ++k) em = max(em, bexp(uk[k]));
    const int w = t >> 5;
    const int r = __reduce_max_sync(warp_mask(L2, w), unsigned(em));
    if ((t & 31) == 0) sm.emax[w] = r;
    if constexpr (MODE == 3) {
      // (values in any order: the block's 3 lx1 pairs a thread, coalesced)
      const int4 *gp = reinterpret_cast<const int4 *>(a.g + 6 * base);
      int ge = 0;
#pragma unroll 6
      for (int q = 0; q < 3 * LX; ++q) {
        const int4 v = __ldg(gp + q * L2 + t);
        ge = max(ge, max(v.y & 0x7FF00000, v.w & 0x7FF00000));
      }
      const int rg = __reduce_max_sync(warp_mask(L2, w), unsigned(ge));
      if ((t & 31) == 0) sm.gmax[w] = rg;
    }
    __syncthreads();
    em = 0;
    for (int q = 0; q < (L2 + 31) / 32; ++q) em = max(em, sm.emax[q]);
#pragma unroll
    for (int k = 0; k < LX; ++k) sm.A[fx_at<LX>(i, j, k)] = to_fixed_cvt(uk[k], em, BITS - 53);
  }
  const int sP = em - 1075 - (BITS - 53);  // p = P 2^sP
  __syncthreads();

  // Thread (i,j) takes, in each contraction stage, the r-line (j, k=i),
  // the s-line (i, k=j) and its own column, the t-line (i,j): one loop over
  // the three directions with run-time strides keeps one copy of the line
  // code per stage; every output goes to shared memory.
  const int lb0 = fx_at<LX>(0, j, i), lb1 = fx_at<LX>(i, 0, j), lb2 = fx_at<LX>(i, j, 0);

  // gradient (local_grad3): A -> C (us), D (ut); then, once every s- and
  // t-line of A was read, A -> A (ur) line by line in place
  u64 orv = 0;
#pragma unroll 1
  for (int dd = 0; dd < 3; ++dd) {
    const int d = dd == 2 ? 0 : dd + 1;
    if (dd == 2) __syncthreads();
    const int b0 = d == 0 ? lb0 : d == 1 ? lb1 : lb2;
    const int st = d == 0 ? 1 : d == 1 ? LX : (LX * LX + 1);
    i64 *out = d == 0 ? sm.A : d == 1 ? sm.C : sm.D;
    i64 v[LX];
#pragma unroll
    for (int m = 0; m < LX; ++m) v[m] = sm.A[b0 + m * st];
    fx_line<LX>(v, cf, 0, [&](int m, i64 y) {
      out[b0 + m * st] = y;
      orv |= mag(y);
    });
  }
  fx_or_post(orv, sm.orl[0], sm.orh[0], t, L2);
  __syncthreads();
  int s1 = fx_or_shift(sm.orl[0], sm.orh[0], L2, BITS);
  if (s1 < 0) {  // outside the bounds shift_up relies on: results invalid
    if (t == 0 && a.err) atomicOr(a.err, 2u);
    s1 = 0;
  }
  const int sU = sP - fc + 64 - s1;  // ur = UR 2^sU after the shift

  // metric (cg.f:156-163) at the thread's own points, in place
  int eg = 0;
  if constexpr (MODE == 3) {
    for (int q = 0; q < (L2 + 31) / 32; ++q) eg = max(eg, sm.gmax[q]);
    eg >>= 20;
  } else {
    eg = a.gexp[e];
  }
  const int sW = 64 - MK + (eg - 1022 - fx_gbits(LX)) + sU;  // wr = WR 2^sW before renormalising
  orv = 0;
#pragma unroll 4
  for (int k = 0; k < LX; ++k) {
    const int q = fx_at<LX>(i, j, k);
    const Sp ur = split(shift_up(sm.A[q], s1)), us = split(shift_up(sm.C[q], s1)),
             ut = split(shift_up(sm.D[q], s1));
    Sp G1, G2, G3, G4, G5, G6;
    if constexpr (MODE == 3) {
      const double2 *gp = reinterpret_cast<const double2 *>(a.g + 6 * (base + size_t(k) * L2 + t));
      const double2 g01 = __ldg(gp), g23 = __ldg(gp + 1), g45 = __ldg(gp + 2);
      G1 = split(to_fixed_bits<fx_gbits(LX)>(g01.x, eg));
      G2 = split(to_fixed_bits<fx_gbits(LX)>(g01.y, eg));
      G3 = split(to_fixed_bits<fx_gbits(LX)>(g23.x, eg));
      G4 = split(to_fixed_bits<fx_gbits(LX)>(g23.y, eg));
      G5 = split(to_fixed_bits<fx_gbits(LX)>(g45.x, eg));
      G6 = split(to_fixed_bits<fx_gbits(LX)>(g45.y, eg));
    } else {
      const int4 *gp = reinterpret_cast<const int4 *>(a.gfx + 6 * (base + size_t(k) * L2 + t));
      const int4 g01 = __ldg(gp), g23 = __ldg(gp + 1), g45 = __ldg(gp + 2);
      G1 = Sp{g01.x, g01.y}, G2 = Sp{g01.z, g01.w}, G3 = Sp{g23.x, g23.y};
      G4 = Sp{g23.z, g23.w}, G5 = Sp{g45.x, g45.y}, G6 = Sp{g45.z, g45.w};
    }
    Acc<MK, FxCoef<LX>::FULL> wr, ws, wt;
    wr.mac(G1, ur); wr.mac(G2, us); wr.mac(G3, ut);
    ws.mac(G2, ur); ws.mac(G4, us); ws.mac(G5, ut);
    wt.mac(G3, ur); wt.mac(G5, us); wt.mac(G6, ut);
    const i64 r_ = wr.result(), s_ = ws.result(), t_ = wt.result();
    sm.A[q] = r_;
    sm.C[q] = s_;
    sm.D[q] = t_;
    orv |= mag(r_) | mag(s_) | mag(t_);
  }
  fx_or_post(orv, sm.orl[1], sm.orh[1], t, L2);
  __syncthreads();
  int s2 = fx_or_shift(sm.orl[1], sm.orh[1], L2, BITS);
  if (s2 < (FxCoef<LX>::FULL ? -2 : 0)) {  // as s1
    if (t == 0 && a.err) atomicOr(a.err, 2u);
    s2 = 0;
  }
  const int sT = 64 - fc + sW - s2;  // transposed-gradient outputs: value 2^sT

  // transposed gradient (local_grad3_t) with D^T, each line in place: A
  // (tr), C (ts), D (tt); a thread reads and writes only its own lines
#pragma unroll 1
  for (int d = 0; d < 3; ++d) {
    const int b0 = d == 0 ? lb0 : d == 1 ? lb1 : lb2;
    const int st = d == 0 ? 1 : d == 1 ? LX : (LX * LX + 1);
    i64 *out = d == 0 ? sm.A : d == 1 ? sm.C : sm.D;
    const i64 *src = out;
    i64 v[LX];
#pragma unroll
    for (int m = 0; m < LX; ++m) v[m] = fx_shift2<LX>(src[b0 + m * st], s2);
    fx_line<LX>(v, cf, 1, [&](int m, i64 y) { out[b0 + m * st] = y; });
  }
  __syncthreads();

  // w_L = tr + ts + tt in FP64
  auto wloc = [&](int k) {
    const int q = fx_at<LX>(i, j, k);
    return to_double_cvt(sm.A[q] + sm.C[q] + sm.D[q], sT);
  };
  const bool bad = em == 0x7FF || eg == 0x7FF;
  double part;
  if (MODE == 1 && whole)
    part = ax_fx_finish<LX, MODE, LX, MODE == 1>(a, e, t, 0, bad, nbr, wloc);
  else
    part = ax_fx_finish<LX, MODE, LX, false>(a, e, t, 0, bad, nbr, wloc);
  if (MODE == 1 || MODE == 2) {
    const double s = block_sum<double>(part, sm.red);
    if (t == 0) a.partial[e] = s;
  }
}

// The CG pass (MODE 1) with three threads a column instead of one, for meshes
// too small to fill the SMs: thread (grp, i, j) takes the lines of direction
// grp in the contraction stages and a third of the column's points elsewhere,
// so an element takes a third of the time (and fewer elements fit an SM).  The
// same values as ax_fx_body and ax_sep_body at every point; pap's partial sums
// in another order.  ax_fx_is_wide says where, with both forms measured.
template <int LX>
__device__ __forceinline__ void ax_fx_wide(const AxArgs<double> &a, const FxCoef<LX> &cf) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  FxShared<LX> &sm = *reinterpret_cast<FxShared<LX> *>(smem_raw);
  constexpr int L2 = LX * LX, L3 = LX * LX * LX, NTH = 3 * L2, NW = (NTH + 31) / 32;
  constexpr int BITS = fx_bits<LX>(), MK = FxCoef<LX>::FULL ? 3 : 0, NK = (LX + 2) / 3;
  constexpr bool SEP = !FxCoef<LX>::FULL;
  const int tid = threadIdx.x, grp = tid / L2, t = tid - grp * L2, i = t % LX, j = t / LX;
  const int e = blockIdx.x, w = tid >> 5, k0 = grp * NK;
  const size_t base = size_t(e) * L3;
  const bool whole = box_flag(a.box_ok);
  const unsigned nbr = whole ? box_neighbours(a.box, e) : 0u;
  const int2 sep = SEP && a.sep ? *reinterpret_cast<const int2 *>(a.sep) : make_int2(0, 0);
  if (SEP && sep.x && tid < FxShared<LX>::NT) {
    sm.tab[tid] = a.sep->tab[tid];
    sm.rest[tid] = a.sep->rest[tid];
  }
  const unsigned lanes = warp_mask(NTH, w);
  int em = 0;
  {
    double uk[NK], pold[NK];
    const double beta = !a.first ? a.sc->beta : 0.0;
#pragma unroll
    for (int q = 0; q < NK; ++q) {  // all loads before the first store
      uk[q] = pold[q] = 0.0;
      if (k0 + q >= LX) break;
      const size_t id = base + size_t(k0 + q) * L2 + t;
      uk[q] = a.u[id];
      if (!a.first) pold[q] = a.pold[id];
    }
#pragma unroll
    for (int q = 0; q < NK; ++q) {
      if (k0 + q >= LX) break;
      if (!a.first) uk[q] = fma_rn(beta, pold[q], uk[q]);  // add2s1, math.f:534
      a.p[base + size_t(k0 + q) * L2 + t] = uk[q];
      em = max(em, bexp(uk[q]));
    }
    const int r = __reduce_max_sync(lanes, unsigned(em));
    if ((tid & 31) == 0) sm.emax[w] = r;
    __syncthreads();
    em = 0;
    for (int q = 0; q < NW; ++q) em = max(em, sm.emax[q]);
#pragma unroll
    for (int q = 0; q < NK; ++q) {
      if (k0 + q >= LX) break;
      sm.A[fx_at<LX>(i, j, k0 + q)] =
          SEP && sep.x ? to_fixed_bits<60>(uk[q], em) : to_fixed_cvt(uk[q], em, BITS - 53);
    }
  }
  __syncthreads();

  // the group's lines: along i (j, k), along j (i, k), along k (i, j)
  const int b0 = grp == 0 ? fx_at<LX>(0, j, i) : grp == 1 ? fx_at<LX>(i, 0, j) : fx_at<LX>(i, j, 0);
  const int st = grp == 0 ? 1 : grp == 1 ? LX : (LX * LX + 1);
  i64 *out = grp == 0 ? sm.A : grp == 1 ? sm.C : sm.D;
  i64 v[LX];
#pragma unroll
  for (int m = 0; m < LX; ++m) v[m] = sm.A[b0 + m * st];
  __syncthreads();  // every line of A is read
  double part = 0.0;
  bool done = false;
  if constexpr (SEP) {
    if (sep.x) {
      fx_line_sep<LX>(v, sm.tab, sm.rest, [&](int m, i64 y) { out[b0 + m * st] = y; });
      __syncthreads();
      const int sY = em - 1075 - (60 - 53) + 64 - sep.y;
      const bool bad = em == 0x7FF;
      auto wloc = [&](int k) {
        const int q = fx_at<LX>(i, j, k);
        return mul_rn(to_double_cvt(sm.A[q] + sm.C[q] + sm.D[q], sY),
                      __ldg(a.sep->v + k * L2 + t));
      };
      part = whole ? ax_fx_finish<LX, 1, NK, true>(a, e, t, k0, bad, nbr, wloc)
                   : ax_fx_finish<LX, 1, NK, false>(a, e, t, k0, bad, nbr, wloc);
      done = true;
    }
  }
  if (!done) {
    u64 orv = 0;
    fx_line<LX>(v, cf, 0, [&](int m, i64 y) {
      out[b0 + m * st] = y;
      orv |= mag(y);
    });
    fx_or_post(orv, sm.orl[0], sm.orh[0], tid, NTH);
    __syncthreads();
    int s1 = fx_or_shift(sm.orl[0], sm.orh[0], NTH, BITS);
    if (s1 < 0) {  // outside the bounds shift_up relies on: results invalid
      if (tid == 0 && a.err) atomicOr(a.err, 2u);
      s1 = 0;
    }
    const int eg = a.gexp[e];
    const int sW = 64 - MK + (eg - 1022 - fx_gbits(LX)) + (em - 1075 - (BITS - 53)) - cf.fc + 64 - s1;
    orv = 0;
#pragma unroll
    for (int k_ = 0; k_ < NK; ++k_) {
      const int k = k0 + k_;
      if (k >= LX) break;
      const int q = fx_at<LX>(i, j, k);
      const Sp ur = split(shift_up(sm.A[q], s1)), us = split(shift_up(sm.C[q], s1)),
               ut = split(shift_up(sm.D[q], s1));
      const int4 *gp = reinterpret_cast<const int4 *>(a.gfx + 6 * (base + size_t(k) * L2 + t));
      const int4 g01 = __ldg(gp), g23 = __ldg(gp + 1), g45 = __ldg(gp + 2);
      const Sp G1 = {g01.x, g01.y}, G2 = {g01.z, g01.w}, G3 = {g23.x, g23.y},
               G4 = {g23.z, g23.w}, G5 = {g45.x, g45.y}, G6 = {g45.z, g45.w};
      Acc<MK, FxCoef<LX>::FULL> wr, ws, wt;
      wr.mac(G1, ur); wr.mac(G2, us); wr.mac(G3, ut);
      ws.mac(G2, ur); ws.mac(G4, us); ws.mac(G5, ut);
      wt.mac(G3, ur); wt.mac(G5, us); wt.mac(G6, ut);
      const i64 r_ = wr.result(), s_ = ws.result(), t_ = wt.result();
      sm.A[q] = r_;
      sm.C[q] = s_;
      sm.D[q] = t_;
      orv |= mag(r_) | mag(s_) | mag(t_);
    }
    fx_or_post(orv, sm.orl[1], sm.orh[1], tid, NTH);
    __syncthreads();
    int s2 = fx_or_shift(sm.orl[1], sm.orh[1], NTH, BITS);
    if (s2 < (FxCoef<LX>::FULL ? -2 : 0)) {  // as s1
      if (tid == 0 && a.err) atomicOr(a.err, 2u);
      s2 = 0;
    }
    const int sT = 64 - cf.fc + sW - s2;
#pragma unroll
    for (int m = 0; m < LX; ++m) v[m] = fx_shift2<LX>(out[b0 + m * st], s2);
    fx_line<LX>(v, cf, 1, [&](int m, i64 y) { out[b0 + m * st] = y; });
    __syncthreads();
    const bool bad = em == 0x7FF || eg == 0x7FF;
    auto wloc = [&](int k) {
      const int q = fx_at<LX>(i, j, k);
      return to_double_cvt(sm.A[q] + sm.C[q] + sm.D[q], sT);
    };
    part = whole ? ax_fx_finish<LX, 1, NK, true>(a, e, t, k0, bad, nbr, wloc)
                 : ax_fx_finish<LX, 1, NK, false>(a, e, t, k0, bad, nbr, wloc);
  }
  const double s = block_sum<double>(part, sm.red);
  if (tid == 0) a.partial[e] = s;
}

// (resident CTAs asked for at 10 and 12: the separable form's line would take 88
// and 114 registers there, and 20 CG iterations at lx1 = 12, box / deformed, on
// 6^3 elements 767 / 916 us instead of 676 / 810; elsewhere the bound has no or
// the opposite effect)
template <int LX>
__global__ void __launch_bounds__((3 * LX * LX + 31) / 32 * 32, LX == 10 ? 3 : LX == 12 ? 2 : 0)
    k_ax_fx_wide(AxArgs<double> a, const __grid_constant__ FxCoef<LX> cf) {
  dependent_begin();
  ax_fx_wide<LX>(a, cf);
}

// (the thread bound is the whole warps the block occupies, so that the
// register budget per thread is what NB_FX_MINB resident blocks leave)
template <int LX, int MODE>
__global__ void __launch_bounds__((LX * LX + 31) / 32 * 32, (LX <= 12 ? NB_FX_MINB : 1))
    k_ax_fx(AxArgs<double> a, const __grid_constant__ FxCoef<LX> cf) {
  dependent_begin();
  ax_fx_body<LX, MODE>(a, cf);
}


template <int LX>
constexpr size_t ax_fx_smem_bytes() {
  return sizeof(FxShared<LX>);
}

}  // namespace fx
}  // namespace nb
