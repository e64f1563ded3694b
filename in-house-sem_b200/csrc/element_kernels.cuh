// Element-forces kernel templates and their per-ngll launchers.
//
// One CTA stages EPB elements (EPB * npe threads, one per element point):
//   1. the element field into shared memory -- from an element-local array
//      (the per-block seam) or gathered from the global field through the
//      local-to-global map and the constraint rows (fused DofMap::gather);
//   2. fluxes and hoop/axis terms per point (element_fluxes);
//   3. the weak divergence per point (element_divergence), written to the
//      element-local force array.
// The launchers are compiled once per ngll (element_ng.cu with
// INSEM_NG = 2..9) so that the instantiations build in parallel.
#pragma once

#include "element_ops.cuh"

namespace insem_b200 {

// Value of slot k of element e, component c, of a global field
// (DofMap::gather, dof_map.hpp:95-120): direct, or the constraint row's
// weighted sum in row order starting from zero.
template <class Value>
__device__ __forceinline__ float gather_slot(int32_t m, const RowsDev& rows, Value&& value) {
  if (m >= 0) return value(m);
  const int32_t r = -1 - m;
  float s = 0.0f;
  for (int32_t q = rows.offsets[r]; q < rows.offsets[r + 1]; ++q) s = fadd(s, fmul(rows.weights[q], value(rows.dofs[q])));
  return s;
}
__device__ __forceinline__ float gather_slot(const float* g, int32_t m, const RowsDev& rows) {
  return gather_slot(m, rows, [g](int32_t p) { return g[p]; });
}
// A float field times a double factor, rounded to float (the power
// iteration's fields, whose factor is applied where they are read).
__device__ __forceinline__ float scaled(float x, double scale) {
  return static_cast<float>(dmul(static_cast<double>(x), scale));
}

// DofMap::assemble of one global point (dof_map.hpp:123-141): its contributions
// in ascending slot order from zero, every component at once.  The slots of
// four contributions load together, then their values: two dependent loads
// for most points, where a loop over components and contributions took two
// per contribution (and divided by a run-time ngll^2).  Gather, element forces
// and assembly of 16,384 coupled order-5 elements take 27 us with their
// launches chained, 45-52 before; internal forces of the cased borehole's two
// domains 18, 31 before.
template <int NG, int NC, bool WEIGHTED>
__device__ __forceinline__ void assemble_point(const int32_t* __restrict__ t_slots, const float* __restrict__ t_weights,
                                               const float* local, int32_t b, int32_t e, float (&f)[NC]) {
  constexpr int NPE = NG * NG;
#pragma unroll
  for (int c = 0; c < NC; ++c) f[c] = 0.0f;
  for (int32_t q0 = b; q0 < e; q0 += 4) {
    int32_t slot[4];
    float w[4], v[4][NC];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      slot[k] = q0 + k < e ? t_slots[q0 + k] : -1;
      if constexpr (WEIGHTED) w[k] = q0 + k < e ? t_weights[q0 + k] : 0.0f;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int32_t el = slot[k] / NPE;
      const float* p = local + static_cast<size_t>(el) * NC * NPE + (slot[k] - el * NPE);
#pragma unroll
      for (int c = 0; c < NC; ++c) v[k][c] = slot[k] >= 0 ? p[c * NPE] : 0.0f;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
      for (int c = 0; c < NC; ++c)
        if (slot[k] >= 0) f[c] = fadd(f[c], WEIGHTED ? fmul(w[k], v[k][c]) : v[k][c]);
  }
}

template <int NG, int NC, bool WEIGHTED>
static __global__ void __launch_bounds__(256) assemble_kernel(const int32_t* __restrict__ t_offsets,
                                                              const int32_t* __restrict__ t_slots,
                                                              const float* __restrict__ t_weights, int32_t n_global,
                                                              const float* local, float* __restrict__ global) {
  dep_begin(kDepAll);
  const int32_t g = blockIdx.x * 256 + threadIdx.x;
  const bool in = g < n_global;
  const int32_t b = in ? t_offsets[g] : 0, e = in ? t_offsets[g + 1] : 0;
  dep_wait(kDepAll);
  if (!in) return;
  float f[NC];
  assemble_point<NG, NC, WEIGHTED>(t_slots, t_weights, local, b, e, f);
#pragma unroll
  for (int c = 0; c < NC; ++c) global[static_cast<size_t>(c) * n_global + g] = f[c];
}

// DofMap::gather (dof_map.hpp:95-120): one thread per element slot.
template <int NG, int NC>
static __global__ void __launch_bounds__(256) gather_kernel(const int32_t* __restrict__ l2g, RowsDev rows, int32_t n_slots,
                                                            int32_t n_global, const float* global,
                                                            float* __restrict__ local) {
  constexpr int NPE = NG * NG;
  dep_begin(kDepAll);
  const int32_t s = blockIdx.x * 256 + threadIdx.x;
  const bool in = s < n_slots;
  const int32_t m = in ? l2g[s] : 0;
  dep_wait(kDepAll);
  if (!in) return;
  const int32_t e = s / NPE;
  float* out = local + static_cast<size_t>(e) * NC * NPE + (s - e * NPE);
  float v[NC];
#pragma unroll
  for (int c = 0; c < NC; ++c) v[c] = gather_slot(global + static_cast<size_t>(c) * n_global, m, rows);
#pragma unroll
  for (int c = 0; c < NC; ++c) out[c * NPE] = v[c];
}

// Arguments of a gather or assembly launch.
struct DofMapLaunch {
  int32_t n = 0;  // slots (gather) or global points (assembly)
  int32_t n_global = 0;
  int ncomp = 1;
  const int32_t* l2g = nullptr;
  RowsDev rows;
  const int32_t* t_offsets = nullptr;
  const int32_t* t_slots = nullptr;
  const float* t_weights = nullptr;  // null: all weights 1
  const float* in = nullptr;
  float* out = nullptr;
  bool gather = false;
  bool preload = false;  // load the kernel without launching it
  cudaStream_t stream = nullptr;
};

template <int NG, int NC>
void launch_dofmap_cfg(const DofMapLaunch& a) {
  auto go = [&](auto kernel, auto... args) {
    if (a.preload) {
      cudaFuncAttributes fa;
      CUDA_CHECK(cudaFuncGetAttributes(&fa, kernel));
      return;
    }
    CUDA_CHECK(launch_chained(kernel, ceil_div(a.n, 256), 256, 0, a.stream, true, args...));
    CUDA_LAUNCH_CHECK();
  };
  if (a.gather) go(gather_kernel<NG, NC>, a.l2g, a.rows, a.n, a.n_global, a.in, a.out);
  else if (a.t_weights) go(assemble_kernel<NG, NC, true>, a.t_offsets, a.t_slots, a.t_weights, a.n, a.in, a.out);
  else go(assemble_kernel<NG, NC, false>, a.t_offsets, a.t_slots, a.t_weights, a.n, a.in, a.out);
}

// Where an element kernel takes its field from.  The late sources are those of
// launches without a wait of their own (kDepLate).  Chosen at run time, the loads
// took the estimate of 9,216 order-4 elements from 4.32 to 4.38 ms; with kernels
// of their own it stays at 4.21 (both sides of a later call).
enum FieldSource : int { kFieldLocal = 0, kFieldGlobal = 1, kFieldScaled = 2, kFieldGlobalLate = 3, kFieldScaledLate = 4 };

template <int NG, int KIND, bool ELASTIC, int M, int SOURCE>
__global__ void __launch_bounds__(ElemCfg<NG, KIND, ELASTIC, M>::THREADS)
    element_forces_kernel(BasisDev basis, BlockDev blk, const float* u_in, const int32_t* __restrict__ l2g, RowsDev rows,
                          int32_t n_global, const double* scale, int32_t dep, float* __restrict__ f_local) {
  using C = ElemCfg<NG, KIND, ELASTIC, M>;
  __shared__ ElemSmem<C> sm;
  dep_begin(dep);
  const int tid = threadIdx.x;
  for (int t = tid; t < C::NPE; t += C::THREADS) {
    sm.D[t] = basis.D[t];
    sm.w2[t] = basis.w2[t];
    if constexpr (C::AXI) sm.Dj[t] = basis.Dj ? basis.Dj[t] : 0.0f;
  }
  const int el = tid / C::NPE;
  const int kpt = tid - el * C::NPE;
  const int bb = blockIdx.x * C::EPB + el;
  const bool active = bb < blk.n;
  int e = 0;
  bool axial = false;
  int32_t slot = 0;
  if (active) {
    e = blk.elements[bb];
    if constexpr (C::AXI) axial = blk.axial[bb] != 0;
    if constexpr (SOURCE != kFieldLocal) slot = l2g[static_cast<size_t>(e) * C::NPE + kpt];
  }
  dep_wait(dep);
  if (active) {
    if constexpr (SOURCE != kFieldLocal) {
      constexpr bool LATE = SOURCE >= kFieldGlobalLate, SCALED = SOURCE == kFieldScaled || SOURCE == kFieldScaledLate;
      double f = 1.0;
      if constexpr (SCALED) f = load_step<LATE>(scale);
#pragma unroll
      for (int c = 0; c < C::NC; ++c) {
        const float* g = u_in + static_cast<size_t>(c) * n_global;
        if constexpr (SCALED)
          sm.u[el][c][kpt] = gather_slot(slot, rows, [g, f](int32_t p) { return scaled(load_step<LATE>(g + p), f); });
        else
          sm.u[el][c][kpt] = gather_slot(slot, rows, [g](int32_t p) { return load_step<LATE>(g + p); });
      }
    } else {
#pragma unroll
      for (int c = 0; c < C::NC; ++c) sm.u[el][c][kpt] = u_in[(static_cast<size_t>(e) * C::NC + c) * C::NPE + kpt];
    }
  }
  __syncthreads();
  float direct[2] = {0.0f, 0.0f};
  const float* Dx = (C::AXI && axial) ? sm.Dj : sm.D;
  if (active) {
    element_fluxes<NG, KIND, ELASTIC, M>(blk, bb, kpt, axial, Dx, sm.D, sm.w2, sm.u[el], sm.f1[el], sm.f2[el],
                                         sm.gx[el][0], sm.gy[el][0], sm.gx[el][C::NAX - 1],
                                         sm.gy[el][C::NAX - 1], direct);
  }
  __syncthreads();
  if (active) {
    float out[C::NC];
    element_divergence<NG, KIND, ELASTIC, M>(kpt, axial, Dx, sm.D, sm.f1[el], sm.f2[el], sm.gx[el][0],
                                             sm.gy[el][0], sm.gx[el][C::NAX - 1], sm.gy[el][C::NAX - 1],
                                             direct, out);
#pragma unroll
    for (int c = 0; c < C::NC; ++c) f_local[(static_cast<size_t>(e) * C::NC + c) * C::NPE + kpt] = out[c];
  }
  dep_end(dep);
}

// Arguments of one element-forces launch.
struct ElementLaunch {
  BasisDev basis;
  BlockDev blk;
  const float* u_in = nullptr;     // element-local field, or global field when gathering
  const int32_t* l2g = nullptr;    // gathering only
  RowsDev rows;                    // gathering only
  int32_t n_global = 0;            // gathering only
  float* f_local = nullptr;
  bool gather = false;
  const double* scale = nullptr;   // gathering only: factor of the field
  bool elastic = false;
  int32_t dep = kDepAll;           // how the launch follows the one ahead of it
  bool overlap = false;
  // load the kernel this launch would run (its module, under lazy loading)
  // without launching it
  bool preload = false;
  cudaStream_t stream = nullptr;
};

template <int NG, int KIND, bool ELASTIC, int M>
void launch_element_cfg(const ElementLaunch& a) {
  using C = ElemCfg<NG, KIND, ELASTIC, M>;
  if (a.blk.n <= 0) return;
  auto go = [&](auto kernel) {
    if (a.preload) {
      cudaFuncAttributes fa;
      CUDA_CHECK(cudaFuncGetAttributes(&fa, kernel));
      return;
    }
    CUDA_CHECK(launch_chained(kernel, ceil_div(a.blk.n, C::EPB), C::THREADS, 0, a.stream, a.overlap, a.basis, a.blk, a.u_in,
                              a.l2g, a.rows, a.n_global, a.scale, a.dep, a.f_local));
    CUDA_LAUNCH_CHECK();
  };
  if (!a.gather) go(element_forces_kernel<NG, KIND, ELASTIC, M, kFieldLocal>);
  else if (a.dep == kDepLate && !a.scale) go(element_forces_kernel<NG, KIND, ELASTIC, M, kFieldGlobalLate>);
  else if (a.dep == kDepLate) go(element_forces_kernel<NG, KIND, ELASTIC, M, kFieldScaledLate>);
  else if (!a.scale) go(element_forces_kernel<NG, KIND, ELASTIC, M, kFieldGlobal>);
  else go(element_forces_kernel<NG, KIND, ELASTIC, M, kFieldScaled>);
}

template <int NG>
void launch_element_ng(const ElementLaunch& a) {
  const int kind = a.blk.kind, m = a.blk.m;
  if (kind == INSEM_AXISYM) {
    if (m == 1) {
      a.elastic ? launch_element_cfg<NG, INSEM_AXISYM, true, 1>(a) : launch_element_cfg<NG, INSEM_AXISYM, false, 1>(a);
    } else {
      a.elastic ? launch_element_cfg<NG, INSEM_AXISYM, true, 0>(a) : launch_element_cfg<NG, INSEM_AXISYM, false, 0>(a);
    }
    return;
  }
  switch (kind) {
    case INSEM_RECT:
      a.elastic ? launch_element_cfg<NG, INSEM_RECT, true, 0>(a) : launch_element_cfg<NG, INSEM_RECT, false, 0>(a);
      break;
    case INSEM_AFFINE:
      a.elastic ? launch_element_cfg<NG, INSEM_AFFINE, true, 0>(a) : launch_element_cfg<NG, INSEM_AFFINE, false, 0>(a);
      break;
    case INSEM_CURVED:
      a.elastic ? launch_element_cfg<NG, INSEM_CURVED, true, 0>(a) : launch_element_cfg<NG, INSEM_CURVED, false, 0>(a);
      break;
    default:
      throw Error(INSEM_CUDA_ERR_UNSUPPORTED, "unknown geometry kind " + std::to_string(kind));
  }
}

// Per-ngll launchers (defined in element_ng.cu, one object per ngll).
void launch_element_ng2(const ElementLaunch&);
void launch_element_ng3(const ElementLaunch&);
void launch_element_ng4(const ElementLaunch&);
void launch_element_ng5(const ElementLaunch&);
void launch_element_ng6(const ElementLaunch&);
void launch_element_ng7(const ElementLaunch&);
void launch_element_ng8(const ElementLaunch&);
void launch_element_ng9(const ElementLaunch&);

struct PowerLaunch;
#define INSEM_POWER(N)                         \
  void launch_power_ng##N(const PowerLaunch&); \
  void launch_dofmap_ng##N(const DofMapLaunch&);
INSEM_POWER(2)
INSEM_POWER(3)
INSEM_POWER(4)
INSEM_POWER(5)
INSEM_POWER(6)
INSEM_POWER(7)
INSEM_POWER(8)
INSEM_POWER(9)
#undef INSEM_POWER
void launch_power(int ngll, const PowerLaunch& a);
void launch_dofmap(int ngll, const DofMapLaunch& a);

// Dispatch on the number of GLL points; unsupported values fail like
// physics::select (kernels.cpp:451-468).
void launch_element_forces(int ngll, const ElementLaunch& a);

}  // namespace insem_b200
