// scheme_dispatch.h -- a scheme's compiled variant as a constant.
#pragma once
#include <type_traits>

#include "tile_launch.h"

namespace rb {

// Scheme variants of the godunov kernels: llf (the default of &HYDRO_PARAMS),
// hll and hllc with minmod or moncen slopes, and hllc with the PLMDE
// predictor, are compiled with the solver, the limiter and the predictor
// fixed; any other scheme runs the variant that reads them at run time, which
// carries every solver's registers and branches (llf, minmod: a 64^3 FP64 step
// 100.7 us in it). The kernels take ST = slope type + 10 for PLMDE.
template <typename F>
static cudaError_t with_scheme(const rb_hydro_params& hp, F&& f) {
  switch (scheme_variant(hp)) {
    case 11: return f(std::integral_constant<int, 11>());
    case 12: return f(std::integral_constant<int, 12>());
    case 21: return f(std::integral_constant<int, 21>());
    case 22: return f(std::integral_constant<int, 22>());
    case 31: return f(std::integral_constant<int, 31>());
    case 32: return f(std::integral_constant<int, 32>());
    case 131: return f(std::integral_constant<int, 131>());
    case 132: return f(std::integral_constant<int, 132>());
  }
  return f(std::integral_constant<int, 0>());
}
template <int V> struct SchemeOf {
  static constexpr int RS = V ? (V % 100) / 10 : 0, ST = V ? V % 10 + 10 * (V / 100) : -1;
};

}  // namespace rb
