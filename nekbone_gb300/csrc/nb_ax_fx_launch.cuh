// nb_ax_fx_launch.cuh -- dispatch of the fixed-point FP64 element operator
// over lx1 (one translation unit per mode includes this).
#pragma once

#include "nb_ax_fx.cuh"
#include "nb_solver.h"

namespace nb {

// Where the CG pass takes three threads a column (k_ax_fx_wide).  20 CG
// iterations, box / deformed, one thread -> three: small elements fill their
// warps at any size (lx1 = 4 on 20^3: 900 / 1008 -> 795 / 901 us; 6 on 24^3:
// 2707 / 3509 -> 2344 / 2916; 9 on 16^3: 3325 -> 3136), others while the mesh
// does not fill the SMs (8 on 8^3: 573 / 635 -> 557 / 622, on 16^3: 1491 / 1927
// -> 1553 / 2114; 10 on 810 elements: 970 / 1226 -> 946 / 1197, on 20^3: 4832 /
// 6694 -> 4973 / 7465; 12 on 6^3: 736 / 926 -> 673 / 818, on 8^3: 1050 / 1399 ->
// 1062 / 1354; 14 on 125: 734 / 860 -> 700 / 815, on 216: 947 / 1225 -> 1031 /
// 1285).
inline bool ax_fx_is_wide(int lx, int nelt) {
  if (lx < 4) return false;
  if (lx <= 7 || lx == 9) return true;
  return nelt <= (lx == 8 ? 600 : lx == 10 ? 1000 : lx <= 12 ? 304 : 152);
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
  if constexpr (MODE == 1) {
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
