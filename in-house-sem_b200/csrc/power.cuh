// Kernels of the stable time step's power iteration (solver.cpp:583-667).
//
// An iteration is two launches per domain: the element forces of the scaled
// field (element_kernels.cuh), and power_kernel, which assembles them point by
// point, forms the next field and the iteration's FP64 sums, and whose last
// CTA turns these into the Rayleigh quotient and the next scale.  The scale is
// applied where the field is read, so nothing passes over it in between.
// Bound by latency (two chained launches of 3-4 us each): with the assembly,
// the sums, their serial additions and the scaling in eight launches of their
// own an iteration took 45 us at 6,000 order-5 elements.
#pragma once

#include "element_kernels.cuh"

namespace insem_b200 {

// Power-iteration scalars, kept on the device.
enum PowerSlot : int {
  kPwLambda = 0,   // running max of the Rayleigh quotients (uncoupled domains)
  kPwDone = 1,     // the loop has stopped (the reference's break)
  kPwScale = 2,    // factor of the field
  kPwCoupled = 3,  // running max of sqrt(ny / nx) (coupled operator)
  kPwCount = 4
};
constexpr int kPowerThreads = 256;
constexpr int kPowerBlocks = 592;  // at most, 4 per SM

// Which operator: a domain alone, or the solid / fluid half of the coupled one.
enum PowerMode : int { kPowerAlone = 0, kPowerSolid = 1, kPowerFluid = 2 };

struct PowerEntry {  // one interface entry of a point
  int32_t partner;
  float cx, cz;
};
struct PowerDev {
  int32_t ng = 0;
  const int32_t* t_offsets = nullptr;
  const int32_t* t_slots = nullptr;
  const float* t_weights = nullptr;
  const float* f_local = nullptr;
  float* x = nullptr;                // [ncomp][ng]; the field is x times the scale
  const float* mass = nullptr;
  const float* inv_mass = nullptr;
  const uint8_t* zero = nullptr;     // [ng] components held at zero
  const int32_t* cpl_off = nullptr;  // [ng + 1] interface entries of each point (coupled operator)
  const PowerEntry* cpl = nullptr;
  const float* other = nullptr;      // the other domain's x
  int32_t other_ng = 0;
  bool pm = false;                   // three-component solid
  double* partial = nullptr;         // [blocks][3] of this launch
  const double* partial_s = nullptr; // fluid half: the solid half's, of blocks_s CTAs
  int32_t blocks_s = 0;
  uint32_t* counter = nullptr;       // CTAs done (0 between launches)
  double* pw = nullptr;
  bool late = false;                 // coupled: iteration 60 or later
};

struct PowerLaunch {
  PowerDev d;
  int ncomp = 1;
  int mode = kPowerAlone;
  cudaStream_t stream = nullptr;
};
inline int power_blocks(int ng) { return std::min(kPowerBlocks, ceil_div(std::max(ng, 1), kPowerThreads)); }

// Sum over the CTA of N values, the same in every run; valid in thread 0.
template <int N>
__device__ __forceinline__ void power_reduce(double (&v)[N], double (*sh)[kPowerThreads / 32]) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1)
#pragma unroll
    for (int k = 0; k < N; ++k) v[k] = dadd(v[k], __shfl_down_sync(0xffffffffu, v[k], off));
  if ((threadIdx.x & 31) == 0)
#pragma unroll
    for (int k = 0; k < N; ++k) sh[k][threadIdx.x >> 5] = v[k];
  __syncthreads();
  if (threadIdx.x == 0)
#pragma unroll
    for (int k = 0; k < N; ++k) {
      double s = sh[k][0];
      for (int q = 1; q < kPowerThreads / 32; ++q) s = dadd(s, sh[k][q]);
      v[k] = s;
    }
  __syncthreads();
}

template <int NG, int NC, bool WEIGHTED, int MODE>
static __global__ void __launch_bounds__(kPowerThreads) power_kernel(PowerDev d) {
  __shared__ double sh[3][kPowerThreads / 32];
  __shared__ bool last;
  dep_begin(kDepAll);
  dep_wait(kDepAll);
  const double scale = d.pw[kPwScale];
  double acc[3] = {0.0, 0.0, 0.0};
  for (int32_t g = blockIdx.x * kPowerThreads + threadIdx.x; g < d.ng; g += gridDim.x * kPowerThreads) {
    float f[NC];
    assemble_point<NG, NC, WEIGHTED>(d.t_slots, d.t_weights, d.f_local, d.t_offsets[g], d.t_offsets[g + 1], f);
    const double m = d.mass[g];
    const float im = d.inv_mass[g];
    const uint32_t zero = d.zero[g];
    float x[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) x[c] = scaled(d.x[static_cast<size_t>(c) * d.ng + g], scale);
    if constexpr (MODE == kPowerAlone) {
      // x.Kx, x.Mx and |y|^2, y = M^-1 K x (solver.cpp:597-609)
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const double xi = x[c];
        acc[0] = dadd(acc[0], dmul(xi, static_cast<double>(f[c])));
        acc[1] = dadd(acc[1], dmul(dmul(m, xi), xi));
        const double y = dmul(-static_cast<double>(f[c]), static_cast<double>(im));
        acc[2] = dadd(acc[2], dmul(y, y));
        d.x[static_cast<size_t>(c) * d.ng + g] = zero & (1u << c) ? 0.0f : static_cast<float>(y);
      }
    } else {
      // mass norms of the field and of its acceleration under the coupled
      // operator (solver.cpp:628-656); the fluid's x is still the field when
      // the solid half reads it, the solid's already its new acceleration
      // when the fluid half does
      const float h = static_cast<float>(0.70710678118654752440);
      for (int32_t q = d.cpl_off[g]; q < d.cpl_off[g + 1]; ++q) {
        const PowerEntry ce = d.cpl[q];
        if constexpr (MODE == kPowerSolid) {
          const float p = scaled(d.other[ce.partner], scale);
          if (d.pm) {
            const float t = fmul(fmul(h, ce.cx), p);
            f[0] = fadd(f[0], t);
            if constexpr (NC > 1) f[1] = fadd(f[1], t);
          } else {
            f[0] = fadd(f[0], fmul(ce.cx, p));
          }
          f[NC - 1] = fadd(f[NC - 1], fmul(ce.cz, p));
        } else {
          const float* a = d.other + ce.partner;
          const size_t on = d.other_ng;
          const float ar = d.pm ? fmul(h, fadd(a[0], a[on])) : a[0];
          f[0] = fsub(f[0], fadd(fmul(ce.cx, ar), fmul(ce.cz, a[d.pm ? 2 * on : on])));
        }
      }
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const double u = x[c];
        acc[0] = dadd(acc[0], dmul(dmul(m, u), u));
        const float af = zero & (1u << c) ? 0.0f : fmul(f[c], im);
        const double a = af;
        acc[1] = dadd(acc[1], dmul(dmul(m, a), a));
        d.x[static_cast<size_t>(c) * d.ng + g] = af;
      }
    }
  }
  power_reduce<3>(acc, sh);
  if (threadIdx.x == 0) {
#pragma unroll
    for (int k = 0; k < 3; ++k) d.partial[3 * blockIdx.x + k] = acc[k];
    if constexpr (MODE != kPowerSolid) {
      __threadfence();
      last = atomicAdd(d.counter, 1u) == gridDim.x - 1;
    }
  }
  if constexpr (MODE == kPowerSolid) return;
  __syncthreads();
  if (!last) return;
  __threadfence();
  auto sum = [&](const double* part, int32_t n, double (&v)[3]) {
    v[0] = v[1] = v[2] = 0.0;
    for (int32_t q = threadIdx.x; q < n; q += kPowerThreads)
#pragma unroll
      for (int k = 0; k < 3; ++k) v[k] = dadd(v[k], __ldcg(part + 3 * q + k));
    power_reduce<3>(v, sh);
  };
  double v[3], w[3] = {0.0, 0.0, 0.0};
  if constexpr (MODE == kPowerFluid) sum(d.partial_s, d.blocks_s, w);
  sum(d.partial, gridDim.x, v);
  if (threadIdx.x != 0) return;
  *d.counter = 0;
  if (d.pw[kPwDone] != 0.0) return;
  if constexpr (MODE == kPowerAlone) {
    // lambda from x.Kx = -(x . f) over x.Mx, then stop on a zero norm or set
    // the scale 1 / sqrt(norm) (solver.cpp:597-612)
    if (v[1] > 0.0) {
      const double q = -v[0] / v[1];
      if (d.pw[kPwLambda] < q) d.pw[kPwLambda] = q;
    }
    if (v[2] == 0.0) d.pw[kPwDone] = 1.0;
    else d.pw[kPwScale] = 1.0 / sqrt(v[2]);
  } else {
    // stop on a zero norm, sqrt(ny / nx) from iteration 60 on, scale
    // -1 / sqrt(ny) (solver.cpp:641-662)
    const double nx = dadd(w[0], v[0]), ny = dadd(w[1], v[1]);
    if (nx <= 0.0 || ny <= 0.0) {
      d.pw[kPwDone] = 1.0;
      return;
    }
    if (d.late) {
      const double q = sqrt(ny / nx);
      if (d.pw[kPwCoupled] < q) d.pw[kPwCoupled] = q;
    }
    d.pw[kPwScale] = -1.0 / sqrt(ny);
  }
}

template <int NG>
void launch_power_cfg(const PowerLaunch& a) {
  auto go = [&](auto plain, auto weighted) {
    CUDA_CHECK(launch_chained(a.d.t_weights ? weighted : plain, power_blocks(a.d.ng), kPowerThreads, 0, a.stream, true, a.d));
    CUDA_LAUNCH_CHECK();
  };
  if (a.mode == kPowerAlone) {
    if (a.ncomp == 1) go(power_kernel<NG, 1, false, kPowerAlone>, power_kernel<NG, 1, true, kPowerAlone>);
    else if (a.ncomp == 2) go(power_kernel<NG, 2, false, kPowerAlone>, power_kernel<NG, 2, true, kPowerAlone>);
    else go(power_kernel<NG, 3, false, kPowerAlone>, power_kernel<NG, 3, true, kPowerAlone>);
  } else if (a.mode == kPowerSolid) {
    if (a.ncomp == 2) go(power_kernel<NG, 2, false, kPowerSolid>, power_kernel<NG, 2, true, kPowerSolid>);
    else go(power_kernel<NG, 3, false, kPowerSolid>, power_kernel<NG, 3, true, kPowerSolid>);
  } else {
    go(power_kernel<NG, 1, false, kPowerFluid>, power_kernel<NG, 1, true, kPowerFluid>);
  }
}

}  // namespace insem_b200
