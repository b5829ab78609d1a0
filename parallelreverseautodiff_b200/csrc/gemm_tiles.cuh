// Pieces shared by the register-tiled GEMM kernels (FMA and DMMA): 128-bit vector lengths and the epilogue parameter block.
#pragma once

#include "act_math.cuh"
#include "common.cuh"

namespace prad {

template <typename T> struct VecOf;
template <> struct VecOf<float> { using type = float4; static constexpr int N = 4; };
template <> struct VecOf<double> { using type = double2; static constexpr int N = 2; };

template <typename T> struct EpiParams {
  const T* bias;
  T* z_out;
  int act;
  int dact;
  const T* saved;
  T act_alpha;
};

}  // namespace prad
