// nb_ax_fx_launch.cuh -- dispatch of the fixed-point FP64 element operator
// over lx1 (one translation unit per mode includes this).
#pragma once

#include "nb_ax_fx.cuh"
#include "nb_solver.h"

namespace nb {

// Where the CG pass takes three threads a column (k_ax_fx_wide).  20 CG
// iterations in us, box / deformed (odd lx1: one figure, the form is the same),
// one thread -> three.  Small elements fill their warps at any size:
//   lx1  4: 64 elements 329 / 339 -> 307 / 312; 20^3 906 / 1003 -> 795 / 889
//        5: 27 376 -> 330; 8^3 456 -> 432; 20^3 1440 -> 1455
//        6: 6^3 377 / 402 -> 343 / 352; 24^3 2686 / 3487 -> 2368 / 2926
//        7: 27 438 -> 369; 8^3 636 -> 604; 18^3 2436 -> 2361
//        9: 27 490 -> 403; 9^3 1044 -> 928; 24^3 9968 -> 9650
// Others gain while the mesh does not fill the SMs:
//        8: 600 589 / 645 -> 577 / 630; 704 619 / 705 -> 655 / 706; 16^3 1496 /
//           1924 -> 1658 / 2239
//       10: 64 461 / 504 -> 428 / 457; 10^3 1101 / 1388 -> 1099 / 1394; 20^3 4913
//           / 6674 -> 5197 / 7490
//       11: 27 550 -> 489; 304 850 -> 837; 8^3 1194 -> 1248; 14^3 3946 -> 4738
//       12: 64 577 / 626 -> 491 / 547; 304 822 / 963 -> 741 / 874; 8^3 1075 / 1383
//           -> 1083 / 1366
//       14: 27 622 / 721 -> 581 / 672; 150 772 / 870 -> 733 / 826; 6^3 988 / 1223
//           -> 1066 / 1285
//       16: nothing (27 725 / 847 -> 725 / 851; 150 893 / 1033 -> 897 / 1035)
inline bool ax_fx_is_wide(int lx, int nelt) {
  if (lx < 4 || lx > 14) return false;
  if (lx <= 7 || lx == 9) return true;
  return nelt <= sm_count() * (lx == 8 ? 4 : lx == 10 ? 6 : lx <= 12 ? 2 : 1);
}

template <int LX, int MODE>
int launch_ax_fx_shape(const Operator &op, AxArgs<double> a, cudaStream_t s) {
  const size_t sm = fx::ax_fx_smem_bytes<LX>();
  static bool attr_set = false;
  if (!attr_set) {
    NB_CUDA(cudaFuncSetAttribute(fx::k_ax_fx<LX, MODE>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, int(sm)));
    attr_set = true;
  }
  typedef fx::FxCoef<LX> Coef;
  if (int(op.FXhi.size()) != Coef::Q || int(op.FXlo.size()) != Coef::Q ||
      (Coef::FULL && int(op.FXd.size()) != Coef::QD))
    return fail(NB_ERR_STATE, "fixed-point ax: tables for lx1=%d missing", LX);
  Coef cf;
  for (int q = 0; q < Coef::Q; ++q) {
    cf.hi[q] = op.FXhi[q];
    cf.lo[q] = op.FXlo[q];
  }
  for (int q = 0; q < Coef::QD; ++q) cf.d[q] = Coef::FULL ? op.FXd[q] : 0;
  cf.fc = op.fx_fc;
  if constexpr (MODE == 1 && LX >= 4 && LX <= 14) {
    if (ax_fx_is_wide(LX, a.nelt)) {
      static bool wide_set = false;
      if (!wide_set) {
        NB_CUDA(cudaFuncSetAttribute(fx::k_ax_fx_wide<LX>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, int(sm)));
        wide_set = true;
      }
      NB_CUDA(launch_dependent(fx::k_ax_fx_wide<LX>, dim3(a.nelt), dim3(3 * LX * LX), sm, s, a,
                               cf));
      return NB_OK;
    }
  }
  if constexpr (MODE == 1 || MODE == 3) {  // in a CG iteration, an apply
    NB_CUDA(launch_dependent(fx::k_ax_fx<LX, MODE>, dim3(a.nelt), dim3(LX, LX), sm, s, a, cf));
  } else {
    fx::k_ax_fx<LX, MODE><<<a.nelt, dim3(LX, LX), sm, s>>>(a, cf);
    NB_CUDA(cudaGetLastError());
  }
  return NB_OK;
}

template <int MODE>
int launch_ax_fx_mode(const Operator &op, AxArgs<double> a, cudaStream_t s) {
  switch (op.lx) {
#define NB_CASE(L) case L: return launch_ax_fx_shape<L, MODE>(op, a, s);
    NB_CASE(2) NB_CASE(3) NB_CASE(4) NB_CASE(5) NB_CASE(6) NB_CASE(7) NB_CASE(8) NB_CASE(9)
    NB_CASE(10) NB_CASE(11) NB_CASE(12) NB_CASE(14) NB_CASE(16)
#undef NB_CASE
    default:
      return fail(NB_ERR_UNSUPPORTED, "fixed-point ax: lx1=%d", op.lx);
  }
}

}  // namespace nb
