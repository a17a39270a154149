// nb_ax_fx.cu -- set-up of the fixed-point FP64 element operator
// (nb_ax_fx.cuh): its derivative tables, computed exactly on the host, and
// the per-solve conversion of the metric g into fixed point.
#include <cmath>
#include <cstdint>
#include <vector>

#include "nb_ax_fx.cuh"
#include "nb_solver.h"

namespace nb {

namespace {

typedef __int128 i128;

// x = m 2^e exactly, |m| < 2^53
void decompose(double x, int64_t *m, int *e) {
  if (x == 0.0) {
    *m = 0;
    *e = 0;
    return;
  }
  int ex = 0;
  const double fr = std::frexp(x, &ex);
  *m = int64_t(std::ldexp(fr, 53));
  *e = ex - 53;
}

// round((x[0] + ... + x[nx-1]) 2^sh) to the nearest integer (ties to even),
// from the exact values (a term below 2^-70 of another is dropped)
int64_t scaled_sum(const double *x, int nx, int sh) {
  int64_t m[4];
  int e[4], top = -100000, e0 = 100000;
  for (int q = 0; q < nx; ++q) {
    decompose(x[q], &m[q], &e[q]);
    if (m[q] != 0) top = std::max(top, e[q]);
  }
  for (int q = 0; q < nx; ++q)
    if (m[q] != 0 && top - e[q] <= 70) e0 = std::min(e0, e[q]);
    else m[q] = 0;
  i128 T = 0;
  for (int q = 0; q < nx; ++q)
    if (m[q] != 0) T += i128(m[q]) << (e[q] - e0);
  if (T == 0) return 0;
  const int s = e0 + sh;
  if (s >= 0) return int64_t(T << s);
  if (-s > 120) return 0;
  const i128 neg = T < 0 ? -T : T;
  i128 q = neg >> (-s);
  const i128 rem = neg - (q << (-s)), half = i128(1) << (-s - 1);
  if (rem > half || (rem == half && (q & 1))) ++q;
  return int64_t(T < 0 ? -q : q);
}

// one block per element: the element's largest exponent over its 6 lx1^3
// metric values, then each value as balanced halves of g 2^(1022 + bits - emax)
// (nothing where the separable form holds)
__global__ void __launch_bounds__(256)
    k_metric_fx(const double *__restrict__ g, int2 *__restrict__ gfx, int *__restrict__ gexp,
                int blk, int bits, const fx::SepTables *sep) {
  __shared__ int wmax[8];
  if (sep && sep->ok) return;
  const int t = threadIdx.x;
  const size_t base = size_t(blockIdx.x) * blk;
  int em = 0;
  for (int q = t; q < blk; q += 256) em = max(em, fx::bexp(g[base + q]));
  const int r = __reduce_max_sync(0xFFFFFFFFu, unsigned(em));
  if ((t & 31) == 0) wmax[t >> 5] = r;
  __syncthreads();
  em = 0;
  for (int w = 0; w < 8; ++w) em = max(em, wmax[w]);
  for (int q = t; q < blk; q += 256) {
    const fx::Sp s = fx::split(fx::to_fixed(g[base + q], em, bits - 53));
    gfx[base + q] = make_int2(s.lo, s.hi);
  }
  if (t == 0) gexp[blockIdx.x] = em;
}

// ------------------------------------------------------ double-double --
struct DD {
  double h, l;
};
__device__ __forceinline__ DD dd_sum(double a, double b) {  // exact (Knuth's two-sum)
  const double s = __dadd_rn(a, b), bb = __dadd_rn(s, -a);
  return {s, __dadd_rn(__dadd_rn(a, -__dadd_rn(s, -bb)), __dadd_rn(b, -bb))};
}
__device__ __forceinline__ DD dd_add(DD a, DD b) {
  const DD s = dd_sum(a.h, b.h);
  return dd_sum(s.h, __dadd_rn(s.l, __dadd_rn(a.l, b.l)));
}

__device__ __forceinline__ DD dd_sub(DD a, DD b) { return dd_add(a, DD{-b.h, -b.l}); }

// K and its tables from D and element 0's v, by one block: K(i,m) in
// double-double, then E and O, each the nearest integer of the value times
// 2^fc, and the rest.  False where a sum of the operator's accumulators (Acc,
// and the three directions) could leave 64 bits, or the rest's 24.
__device__ bool sep_tables(const double *__restrict__ D, int lx, fx::SepTables *sep) {
  __shared__ DD K[256];
  __shared__ double bs[16];
  __shared__ int emax[8];
  const int t = threadIdx.x, h = lx / 2, n1 = lx - 1, nk = lx * lx;
  if (t < lx) bs[t] = sep->v[t + lx * h + lx * lx * h];
  __syncthreads();
  int em = 0;
  if (t < nk) {
    const int i = t / lx, m = t % lx;
    DD k = {0.0, 0.0};
    for (int q = 0; q < lx; ++q) {
      const double a = D[q + i * lx], b = D[q + m * lx], w = bs[q];
      const double p = __dmul_rn(a, b), pe = __fma_rn(a, b, -p);  // a b = p + pe
      const double r = __dmul_rn(p, w), re = __fma_rn(pe, w, __fma_rn(p, w, -r));
      const DD x = dd_sum(k.h, r);
      k = {x.h, __dadd_rn(k.l, __dadd_rn(x.l, re))};
    }
    const double w = bs[i], q = __ddiv_rn(k.h, w), r = __fma_rn(-q, w, k.h);  // r exact
    k = dd_sum(q, __ddiv_rn(__dadd_rn(r, k.l), w));
    K[t] = k;
  }
  __syncthreads();
  // value t of the tables, and the largest exponent among them
  DD p = {0.0, 0.0}, rest = {0.0, 0.0};
  const int at = t % (h * h), which = t / (h * h);  // which: 0 E, 1 O
  if (which < 2) {
    const int a = at / h, c = at % h;
    const DD k00 = K[a * lx + c], k01 = K[a * lx + n1 - c];
    const DD k10 = K[(n1 - a) * lx + c], k11 = K[(n1 - a) * lx + n1 - c];
    const DD x = dd_add(k00, k11), y = dd_add(k01, k10);
    const DD u = dd_sub(k00, k11), w = dd_sub(k01, k10);
    p = which ? dd_sub(x, y) : dd_add(x, y);
    rest = which ? dd_sub(u, w) : dd_add(u, w);
    p = {0.25 * p.h, 0.25 * p.l};
    em = fx::bexp(p.h);
  }
  em = int(__reduce_max_sync(0xFFFFFFFFu, unsigned(em)));
  if ((t & 31) == 0) emax[t >> 5] = em;
  __syncthreads();
  for (int q = 0; q < 8; ++q) em = max(em, emax[q]);
  const int fc = 61 - (em - 1022);  // every value below 2^(em - 1022)
  bool good = em > 1 && em < 2046;
  if (good && which < 2) {
    // the high part times 2^fc has a fraction of at most 52 bits: both exact
    const double hs = scalbn(p.h, fc), hi = rint(hs);
    const long long C = (long long)hi + __double2ll_rn((hs - hi) + scalbn(p.l, fc));
    const fx::Sp sp = fx::split(C);
    reinterpret_cast<int2 *>(sep->tab)[2 * at + which] = make_int2(sp.hi, sp.lo);
    reinterpret_cast<float *>(sep->rest)[2 * at + which] =
        float(scalbn(0.25 * (rest.h + rest.l), fc - 32));
    good = C <= (1ll << 61) && C >= -(1ll << 61);
  }
  __syncthreads();
  if (good && t < h) {  // the rows' sums
    double xe = 0.0, xo = 0.0, hm = 0.0, rm = 0.0;
    for (int c = 0; c < h; ++c) {
      const int4 eo = sep->tab[t * h + c];
      const float2 d = sep->rest[t * h + c];
      const double ae = fabs(double(eo.x)) + 1.0, ao = fabs(double(eo.z)) + 1.0;
      // x + x2 of a sum, in units of 2^31: |hi| 2^31 + |lo| 2^29 a term
      xe += ae + 0.25 * fabs(double(eo.y));
      xo += ao + 0.25 * fabs(double(eo.w));
      hm += fmax(ae, ao);
      rm += fabs(double(d.x)) + fabs(double(d.y));
    }
    // the output: three directions of at most sum max(|E|, |O|) times 2^61, in
    // units of 2^64; the rest: values' high halves of at most 2^29
    good = xe < 4.29e9 && xo < 4.29e9 && 3.0 * hm < 1.7e10 && rm * 0x1p29 < 0x1p24;
  }
  if (t == 0) sep->fc = fc;
  return good;
}

// Whether g has the separable form (SepTables): sep->ok, set before, is
// cleared where it has not, and a block returns at once when it finds it
// cleared.  Block 0 looks at element 0's product form and makes the tables
// meanwhile; every block compares its elements with element 0, bitwise.
// HBM-bound: g read once (48 B a point, 0.39 ms at 32^3, lx1 = 12) where the
// form holds, next to nothing where it does not.
__global__ void __launch_bounds__(256)
    k_sep_check(const double *__restrict__ g, const double *__restrict__ D, int lx, int nelt,
                fx::SepTables *sep) {
  const int l3 = lx * lx * lx, t = threadIdx.x;
  const unsigned long long *g0 = reinterpret_cast<const unsigned long long *>(g);
  __shared__ int on;
  for (int e = blockIdx.x; e < nelt; e += gridDim.x) {
    if (t == 0) on = *reinterpret_cast<volatile int *>(&sep->ok);
    __syncthreads();
    if (!on) return;
    bool ok = true;
    const unsigned long long *ge = g0 + size_t(e) * 6 * l3;
    for (int l = t; l < l3; l += blockDim.x) {
      const unsigned long long v = g0[6 * l];
      const unsigned long long *q = ge + 6 * l;
      ok &= q[0] == v && q[3] == v && q[5] == v && ((q[1] | q[2] | q[4]) << 1) == 0;
    }
    if (e == 0 && __syncthreads_and(ok)) {
      const int m = lx / 2, L2 = lx * lx;
      auto line = [&](int i) { return g[6 * (i + lx * m + L2 * m)]; };
      const double gm = line(m);
      for (int l = t; l < l3; l += blockDim.x) {
        const double v = g[6 * l];
        const double a = line(l % lx), b = line((l / lx) % lx), c = line(l / L2);
        const double l1 = v * gm * gm, l2 = a * b * c;
        // (2e-15: up to eight roundings on each side); b symmetric to 2e-14, so
        // that the rest is small: zwgll's own weights differ by 6e-15 at lx1 =
        // 12 and 1.2e-14 at 16
        ok &= v > 1e-60 && v < 1e60 && fabs(l1 - l2) <= 2e-15 * l2;
        ok &= fabs(a - line(lx - 1 - l % lx)) <= 2e-14 * a;
        sep->v[l] = v;
      }
      if (__syncthreads_and(ok)) ok = sep_tables(D, lx, sep);
    }
    if (!__syncthreads_and(ok)) {
      if (t == 0) atomicExch(&sep->ok, 0);
      return;
    }
  }
}

}  // namespace

// The tables of D and of D^T in FxCoef's order and form, with fc fractional
// bits.
bool fx_tables(const std::vector<double> &D, int lx, std::vector<int> &hi,
               std::vector<int> &lo, std::vector<int> &d, int *fc) {
  // lx1 = 13 and 15 keep the reference's FP64 sums: on random fields one apply
  // of this form has 1.1 to 1.5 times their error there (up to 11 less than it)
  if (lx < 2 || (lx % 2 != 0 && lx > 11)) return false;
  const int h = lx / 2, h1 = lx - h;
  const bool full = h1 > h;
  const int bits = full ? 61 : 59;
  // value (a, m) of E (even) or O of D or, with tr, of D^T as a sum of terms
  // over nx: the matrix's entries at (a, m) and (a, n-1-m) and, in the full
  // form, their mirror images -- subtracted for the main tables (sg = -1),
  // added for the remainder's (sg = 1)
  auto terms = [&](bool tr, bool even, int a, int m, int sg, double *x) {
    auto M = [&](int r, int c) { return tr ? D[c + r * lx] : D[r + c * lx]; };
    const int s2 = even ? 1 : -1, n1 = lx - 1;
    const bool mid = full && m == h;  // the middle column: counted once
    if (!full) {
      x[0] = M(a, m);
      x[1] = s2 * M(a, n1 - m);
      return 2;
    }
    x[0] = M(a, m);
    x[1] = sg * M(n1 - a, n1 - m);
    if (mid) return 2;
    x[2] = s2 * M(a, n1 - m);
    x[3] = s2 * sg * M(n1 - a, m);
    return 4;
  };
  double mx = 0.0;
  for (int tr = 0; tr < 2; ++tr)
    for (int a = 0; a < h1; ++a)
      for (int m = 0; m < h1; ++m)
        for (int even = 0; even < 2; ++even) {
          if (even ? a >= h : m >= h) continue;
          double x[4], s = 0.0;
          const int nx = terms(tr, even, a, m, -1, x);
          for (int q = 0; q < nx; ++q) s += x[q];
          mx = std::max(mx, std::fabs(s) / nx);
        }
  if (!(mx > 0.0)) return false;
  int k = 0;
  std::frexp(mx * (1.0 + 1e-15), &k);  // mx < 2^k
  *fc = bits - k;
  hi.clear();
  lo.clear();
  d.clear();
  bool ok = true;
  for (int tr = 0; tr < 2; ++tr)
    for (int even = 1; even >= 0; --even)
      for (int a = 0; a < (even ? h : h1); ++a)
        for (int m = 0; m < (even ? h1 : h); ++m) {
          double x[4];
          const int nx = terms(tr, even, a, m, -1, x);
          const int64_t C = scaled_sum(x, nx, *fc - (nx == 4 ? 2 : 1));
          const int32_t l = int32_t(uint32_t(uint64_t(C)));
          lo.push_back(l);
          hi.push_back(int32_t((C - int64_t(l)) >> 32));
        }
  if (!full) return true;
  for (int tr = 0; tr < 2; ++tr)
    for (int even = 1; even >= 0; --even) {
      const int nr = even ? h1 : h;
      for (int a = 0; a < nr; ++a)
        for (int m = 0; m < nr; ++m) {
          double x[4];
          const int nx = terms(tr, even, a, m, 1, x);
          const int64_t C = scaled_sum(x, nx, *fc - (nx == 4 ? 2 : 1));
          if (C > (1 << 28) || C < -(1 << 28)) ok = false;
          d.push_back(int(C));
        }
    }
  return ok;
}

void metric_fx_invalidate(const Operator &op) {
  op.gfx_src = nullptr;
  op.metric_single = false;
}
void metric_fx_single(const Operator &op) {
  metric_fx_invalidate(op);
  op.metric_single = true;
}

int metric_fx_prepare(const Operator &op, const double *g, const double *D, bool fused,
                      cudaStream_t s) {
  // (plain applies after fused ones have no separable form to go by)
  if (op.gfx_src == g && op.gfx && (fused || !op.sep_on)) return NB_OK;
  const long nv = 6 * op.n;
  if (op.gfx_cap < nv) {
    if (op.gfx) cudaFree(op.gfx);
    if (op.sep) cudaFree(op.sep);
    op.sep = nullptr;
    op.gfx = nullptr;
    op.gexp = nullptr;
    op.gfx_cap = 0;
    NB_CUDA(cudaMalloc(&op.gfx, size_t(nv) * sizeof(int2)));
    // the separable form's tables and the exponents: one allocation
    NB_CUDA(cudaMalloc(&op.sep, sizeof(fx::SepTables) + size_t(op.nelt) * sizeof(int)));
    op.gexp = reinterpret_cast<int *>(op.sep + 1);
    op.gfx_cap = nv;
  }
  const int blk = 6 * op.lx * op.lx * op.lx;
  // the separable form's check pays from the second apply on
  const bool sep = fused && op.lx % 2 == 0;
  op.sep_on = sep;
  if (sep) {
    NB_CUDA(cudaMemsetAsync(&op.sep->ok, 1, sizeof(int), s));
    k_sep_check<<<std::min(op.nelt, sm_count() * 8), 256, 0, s>>>(g, D, op.lx, op.nelt, op.sep);
  }
  k_metric_fx<<<op.nelt, 256, 0, s>>>(g, op.gfx, op.gexp, blk, fx::fx_gbits(op.lx),
                                       sep ? op.sep : nullptr);
  NB_CUDA(cudaGetLastError());
  op.gfx_src = g;
  return NB_OK;
}

}  // namespace nb
