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
// metric values, then each value as balanced halves of g 2^(1082 - emax)
__global__ void __launch_bounds__(256)
    k_metric_fx(const double *__restrict__ g, int2 *__restrict__ gfx, int *__restrict__ gexp,
                int blk) {
  __shared__ int wmax[8];
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
    const fx::Sp s = fx::split(fx::to_fixed(g[base + q], em, 7));
    gfx[base + q] = make_int2(s.lo, s.hi);
  }
  if (t == 0) gexp[blockIdx.x] = em;
}

}  // namespace

// The tables of D and of D^T in FxCoef's order and form, with fc fractional
// bits.
bool fx_tables(const std::vector<double> &D, int lx, std::vector<int> &hi,
               std::vector<int> &lo, std::vector<int> &d, int *fc) {
  // lx1 = 13 and 15 keep the reference's FP64 sums: on random fields this
  // form's error there is 1.1 to 1.5 times theirs (up to 11 it is smaller)
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

void metric_fx_invalidate(const Operator &op) { op.gfx_src = nullptr; }

int metric_fx_prepare(const Operator &op, const double *g, cudaStream_t s) {
  if (op.gfx_src == g && op.gfx) return NB_OK;
  const long nv = 6 * op.n;
  if (op.gfx_cap < nv) {
    if (op.gfx) cudaFree(op.gfx);
    if (op.gexp) cudaFree(op.gexp);
    op.gfx = nullptr;
    op.gexp = nullptr;
    op.gfx_cap = 0;
    NB_CUDA(cudaMalloc(&op.gfx, size_t(nv) * sizeof(int2)));
    NB_CUDA(cudaMalloc(&op.gexp, size_t(op.nelt) * sizeof(int)));
    op.gfx_cap = nv;
  }
  const int blk = 6 * op.lx * op.lx * op.lx;
  k_metric_fx<<<op.nelt, 256, 0, s>>>(g, op.gfx, op.gexp, blk);
  NB_CUDA(cudaGetLastError());
  op.gfx_src = g;
  return NB_OK;
}

}  // namespace nb
