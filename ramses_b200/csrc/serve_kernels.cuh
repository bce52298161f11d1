// serve_kernels.cuh -- FP64 bookkeeping kernels of the serving engine: the
// initial CFL time step of a dense problem (each batched step advances the
// clocks itself, stream_clock). Compiled without multiply-add contraction so
// the clocks are bitwise those of the single-problem path
// (reduce_partials_kernel).
#pragma once
#include <cstdint>

#include "rb_aux.cuh"
#include "stream_kernel.cuh"

namespace rb {

// Largest CFL wave speed (cmpdt, godunov_utils.f90:5-120) over a dense
// problem; combined across blocks by an integer max on the bit patterns of
// non-negative doubles, which is exact and order-independent.
static __global__ void __launch_bounds__(256) dense_cfl_kernel(const double* __restrict__ u, int64_t n,
                                                        rb_hydro_params hp, unsigned long long* __restrict__ smax_bits) {
  double smax = 0.0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    double q[5];
    for (int v = 0; v < 5; v++) q[v] = u[v * n + i];
    smax = fmx(smax, cfl_speed(q, hp));
  }
  for (int o = 16; o > 0; o >>= 1) smax = fmx(smax, __shfl_xor_sync(0xffffffffu, smax, o));
  if ((threadIdx.x & 31) == 0) atomicMax(smax_bits, (unsigned long long)__double_as_longlong(smax));
}

// clock = (dt, t0, 0, 0, 0, steps=0, done, -) from the largest wave speed,
// as courant_fine + newdt_fine give the first dt (dtnew = min(boxlen/smallc,
// courant_factor*dx/smallc, min cell dt)).
static __global__ void dense_clock_init_kernel(double* __restrict__ clock, unsigned long long* __restrict__ smax_bits,
                                        double t0, double t_end, double max_steps, double dt_max, double dt0,
                                        double dx, double courant_factor) {
  const double smax = __longlong_as_double((long long)*smax_bits);
  *smax_bits = 0ull;  // the steps' running maximum from here on
  const double dt_cell = smax > 0.0 ? cfl_dt_from_speed(smax, dx, courant_factor) : 1.0e300;
  clock[0] = fmn(dt_max, fmn(dt0, dt_cell));
  clock[1] = t0;
  clock[2] = clock[3] = clock[4] = 0.0;
  clock[5] = 0.0;
  clock[6] = (!(t0 < t_end) || !(0.0 < max_steps)) ? 1.0 : 0.0;
  clock[7] = 0.0;
}

}  // namespace rb
