// Tiled fused time step.
//
// Elements of each block are grouped into compact tiles (one CTA each).  A
// tile kernel stages the field of the tile's points in shared memory,
// computes every element's force vector, assembles the points whose
// contributions all come from the tile ("complete" points) in shared memory,
// and finishes them in the same pass: a = f / M, corrector, and the next
// step's predictor, writing u^{n+1} to the other field buffer.  Contributions
// to points shared with other tiles, constrained (hanging) slots and every
// point carrying a boundary, coupling, source or receiver term go to a halo
// buffer; a halo kernel finishes those points with the full reference logic.
//
// Bitwise parity with the reference: each point's contributions are summed
// in ascending slot order (DofMap::assemble, dof_map.hpp:123-141).  A complete
// point inside an element has one contribution, which its own thread adds to
// 0; a complete point on element edges has a list of places, in that order,
// of its contributions in shared memory; halo points sum their halo buffer
// entries in the reference's slot order from a CSR list.
//
// Element math: a lane holds an element and a warp a column: warp i of a CTA
// computes column i (points i, NG + i, ...) of the tile's up to 32 elements.
// All data of a tile lie element-minor, [...][32], so every access of a warp
// to shared memory is free of bank conflicts and every access to global
// memory is 32 adjacent values, and the warps of inner columns finish their
// inner points (56 - 69 % of a tile's points at NG 5 - 7) in registers: field
// and velocity come straight from global memory, nothing is staged or listed.
// (A row of the first component is one 128-byte line; components follow at a
// stride of a multiple of 4 points, so a row of the others starts on any
// 16-byte boundary and may touch two lines.)
// The elements' data arrive in one bulk copy; D entries indexed by the
// unrolled loop counters come from the constant bank.  Every sum keeps the
// reference's operand order.
#pragma once

#include <cstddef>


#include "element_ops.cuh"
#include "step_kernels.cuh"

namespace insem_b200 {

// GLL derivative matrix, GLJ derivative matrix and w_i w_j per ngll (2..9).
static __constant__ float c_basis[8][3][81];

// Two-lane FP32 arithmetic on a component pair (sm_100 add/fma .f32x2).  Each
// lane rounds exactly like the scalar instruction.  The assembler fuses a
// two-lane multiply that feeds a two-lane add into one fused multiply-add,
// which rounds once where the reference rounds the product and the sum
// separately; so a product is formed as fma(a, b, z) with z = -0 read from
// constant memory at run time, which is exactly the rounded product (for
// every a, b, including signed zeros) and is not fused further.
static __constant__ float c_neg_zero;  // -0.0f, written with the basis
using f2x = unsigned long long;        // two packed floats (lane 0 low)
__device__ __forceinline__ f2x pk2(float x, float y) {
  f2x r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ float2 upk2(f2x r) {
  float2 v;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(v.x), "=f"(v.y) : "l"(r));
  return v;
}
__device__ __forceinline__ f2x add2(f2x a, f2x b) {
  f2x d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
// a * b rounded once per lane (nz = pk2(-0, -0) from c_neg_zero)
__device__ __forceinline__ f2x mul2(f2x a, f2x b, f2x nz) {
  f2x d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(nz));
  return d;
}
// a * d rounded once per lane, for a d that the compiler takes from the
// constant bank: two scalar products, no packing of (d, d)
__device__ __forceinline__ f2x mulc2(f2x a, float d) {
  const float2 v = upk2(a);
  return pk2(fmul(v.x, d), fmul(v.y, d));
}

// Floats per element of the field / xi-flux rows: [component][point].
__host__ __device__ constexpr int rows_elem_stride(int ng, int nc) { return nc * ng * ng; }

constexpr int kTileLanes = 32;  // elements of a tile (at most)

// Slot descriptors (uint16 per element slot, [tile][point][lane]): the tile
// point that holds the slot's value.  Inner slots of direct elements have none.
constexpr uint32_t kSlotConstrained = 0xffffu;  // the field row is filled from the constrained-slot list

// Tile points: the tile's complete points on element edges first, then the
// halo points it reads.  A direct element is one whose inner points are all
// complete points of the tile; its lanes finish them in registers.
struct TileHdr {
  int32_t tb;      // tile index in its block (element data, coefficients, axial flags)
  int32_t ne;      // elements
  int32_t nd;      // direct elements: lanes [0, nd)
  int32_t cbeg;    // first inner point (device numbering); (i, j) of the lane's element: ((i - 1) (NG - 2) + j - 1) 32 + lane
  int32_t ebeg;    // first edge complete point
  int32_t nc;      // edge complete points
  int32_t ntp;     // tile points: nc + halo points the tile reads
  int32_t hl_off;  // offset of the halo tile points in halo_tp
  int32_t nhs;     // halo slots (entries written to the halo buffer)
  int32_t hs_off;  // offset into hs_slot / hs_dst
  int32_t ncs;     // constrained slots of the tile
  int32_t cs_off;  // offset into cs_slot / cs_row
  int32_t pl_off;  // offset of the edge points' place lists (points; roundup(nc, 4) of them)
  int32_t pad;
};

// One domain of the tiled path, in device numbering.
struct TiledDev {
  int32_t ng = 0;          // points
  int32_t n_complete = 0;  // complete points are [0, n_complete)
  int32_t n_hbuf = 0;      // halo contributions (per component): the halo points' lists, point by point
  int32_t rs = 4;          // places per list of an edge complete point
  const float* inv_mass = nullptr;
  const float* mass = nullptr;
  const float* u_cur = nullptr;
  float* u_nxt = nullptr;
  float* v = nullptr;
  float* a = nullptr;
  float* vn = nullptr;     // v^n at halo points (receivers)
  const uint16_t* sdesc = nullptr;  // [tile][npe][32] slot descriptors
  const uint16_t* plist = nullptr;  // [edge point][rs] staging places in rank order, kLastPlace on the last
  const TileHdr* tiles = nullptr;
  const int32_t* halo_tp = nullptr; // device point of each halo tile point
  const int32_t* hs_slot = nullptr; // staging place (point * 32 + lane) of each halo entry
  const int32_t* hs_dst = nullptr;  // its place in hbuf, or -1 - m: the places mdst[mdst_off[m] ..)
  const int32_t* mdst_off = nullptr;  // entries with several places (constrained slots feeding several points)
  const int32_t* mdst = nullptr;
  const int32_t* cs_slot = nullptr; // staging place of each constrained slot
  const int2* cs_row = nullptr;     // its constraint row: entries [x, y) of row_dofs / row_w
  const int32_t* row_dofs = nullptr;
  const float* row_w = nullptr;
  float* hbuf = nullptr;            // [ncomp][n_hbuf], each halo point's contributions in its slot order
};

struct StepScalars {
  float rdt, half_dt, half_dt2;
  int32_t energy_every;
};

constexpr uint32_t kLastPlace = 0x8000u;

// A CTA has one warp per element column and one lane per element; tiles of
// fewer elements than lanes leave lanes idle.
template <int NG>
struct TileCfg {
  static constexpr int NPE = NG * NG;
  static constexpr int TE = kTileLanes;            // elements per tile (max)
  static constexpr int THREADS = kTileLanes * NG;  // threads per CTA
};

// Kinds of the tile kernels: insem_cuda_kind, and axisymmetric blocks whose
// elements are rectangles as far as their data tell (every borehole's): xi_r,
// eta_r and eta_z carry one value per element and r one per column, bit for
// bit (xi_z does not: it holds rounding noise).  These are kept once, which
// leaves three values per point of seven: less to fetch, and room for one or
// two more CTAs per SM.  A step of the 30k-element dipole borehole went from
// 45.6 to 39.5 us, of 12 boreholes from 316 to 284, of 10 mixed requests from
// 110.5 to 103.3 (with 7, 9 and 8 warps per scheduler: one more or less of the
// NG 6 and 7 classes 282 - 297 and 104 - 109).
constexpr int kAxisymSeparable = 4;
// The same, elastic, with no axial element and no point on the axis (the solid
// of a borehole): no axis terms, one derivative matrix, no test of r.  The step
// of 12 boreholes went from 277 to 259 us, of the 30k-element dipole borehole
// from 39.8 to 38.8, of the 16k-element monopole one from 13.1 to 12.8.
constexpr int kAxisymOffAxis = 5;
__host__ __device__ constexpr bool is_separable(int kind) { return kind == kAxisymSeparable || kind == kAxisymOffAxis; }
__host__ __device__ constexpr bool is_axisym(int kind) { return kind == INSEM_AXISYM || is_separable(kind); }
__host__ __device__ constexpr int element_kind(int kind) { return is_separable(kind) ? INSEM_AXISYM : kind; }

// Element data of a tile.  Kinds whose metric varies in an element (staged in
// shared memory): pairs [point][32][2] of (xi_x, xi_z), (eta_x, eta_z) and,
// axisymmetric, (wr, hoop), then one plane [point][32] of the Jacobian (Curved)
// or r (axisymmetric: the fluxes use the Jacobian only through wr); separable:
// the pairs (wr, hoop) and the plane xi_z.  Read by the lanes themselves: Rect
// and Affine [array][32] of xi_x, eta_z, jac or xi_x, xi_z, eta_x, eta_z, jac;
// separable, behind the staged part, xi_r, eta_r, eta_z and r of the ng columns.
__host__ __device__ constexpr int tile_arrays(int kind) {
  return kind == INSEM_RECT || is_separable(kind) ? 3 : kind == INSEM_AXISYM ? 7 : 5;
}
__host__ __device__ constexpr bool tile_data_staged(int kind) { return kind == INSEM_CURVED || is_axisym(kind); }
__host__ __device__ constexpr int tile_staged_floats(int kind, int ng) {
  return tile_data_staged(kind) ? tile_arrays(kind) * ng * ng * kTileLanes : 0;
}
__host__ __device__ constexpr int tile_lane_floats(int kind, int ng) {
  return kTileLanes * (is_separable(kind) ? 3 + ng : tile_data_staged(kind) ? 0 : tile_arrays(kind));
}
__host__ __device__ constexpr int tile_data_floats(int kind, int ng) {
  return tile_staged_floats(kind, ng) + tile_lane_floats(kind, ng);
}
// Offset (floats) of array a at point place p = point * 32 + lane (staged kinds).
__host__ __device__ constexpr int tile_data_at(int kind, int npe, int a, int p) {
  return a == tile_arrays(kind) - 1 ? a * npe * kTileLanes + p : (a / 2) * 2 * npe * kTileLanes + 2 * p + a % 2;
}

__device__ __forceinline__ float cbasis(int ng, int which, int idx) { return c_basis[ng - 2][which][idx]; }


// ------------------------------------------------------- bulk-copy helpers
// Two mbarriers per CTA track the tile's bulk copies (cp.async.bulk, the
// non-tensor TMA path), one for the copies at the start of a tile and one
// for the late copies: thread 0 announces the byte count and issues the
// copies; every thread waits on the barrier's phase 0 (one tile per CTA).
__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_addr(dst)),
      "l"(src), "r"(bytes), "r"(smem_addr(bar))
      : "memory");
}
// Orders this thread's earlier generic-proxy accesses to shared memory (made
// visible to it by a block barrier) before bulk copies that overwrite them.
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_addr(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait: gives up after `limit` polls (each poll may suspend the
// thread for a hardware-defined interval) and returns false.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity, uint32_t limit) {
  for (uint32_t it = 0; it < limit; ++it)
    if (mbar_try_wait(bar, parity)) return true;
  return false;
}
constexpr uint32_t kBulkWaitLimit = 1u << 22;

// Whether a class with staged element data keeps its f_xi rows outside it: no
// class does (the host check of the layout asks).  A point's element data are
// read by one thread only, which writes its f_xi over them: pairs of components
// over the first pairs, the only or third component over the last plane.
__host__ __device__ constexpr bool early_flux_rows(int, int) { return false; }

// Shared-memory layout of one tile CTA, byte offsets (16-byte aligned).
// `u` holds the tile points' field [component][tp_cap]; `su` the field rows
// and later the slots' contributions, `sfx` the f_xi rows: component pairs
// [point][32][2], then a single component [point][32].  `v`, `im` and `pl` (the
// place lists) of the edge complete points arrive with the first copies, or
// with a second set once the fluxes are formed (`late`): into the element data
// between the pairs and the last plane, which hold the f_xi rows then.
struct TileLayout {
  uint32_t bar, metric, wr, hoop, r, u, v, im, pl, su, sfx, ax, total;
  int32_t tp_cap, nc_cap, rs;
  int32_t late;

  __host__ __device__ static uint32_t up16(uint32_t x) { return (x + 15u) & ~15u; }
  // rs: the most contributions one edge complete point of the class's tiles has
  __host__ __device__ static TileLayout make(int ng, int nc, int kind, bool elastic, int /*te*/, int tp_cap, int nc_cap,
                                            int rs) {
    TileLayout L{};
    L.rs = (rs + 3) & ~3;  // a point's list is read four entries (8 bytes) at a time
    const uint32_t npe = static_cast<uint32_t>(ng * ng), plane = npe * kTileLanes * 4u;
    L.tp_cap = tp_cap;
    L.nc_cap = nc_cap;
    const bool axi = is_axisym(kind), staged = tile_data_staged(kind);
    uint32_t o = 0;
    L.bar = o;  // two mbarriers: the first copies, the late ones
    o = up16(o + 16);
    L.metric = o;
    L.wr = L.hoop = L.r = o;
    if (kind == INSEM_AXISYM) {
      L.wr = L.hoop = o + 4 * plane;
      L.r = o + 6 * plane;
    }
    o += 4u * tile_staged_floats(kind, ng);
    const uint32_t elem = o - L.metric;
    L.u = o;
    o = up16(o + 4u * nc * tp_cap);
    L.su = o;
    const uint32_t rows = plane * nc;
    o += rows;
    L.sfx = staged ? L.metric : o;
    if (!staged) o += rows;
    const uint32_t v_b = up16(4u * nc * nc_cap), im_b = up16(4u * nc_cap), pl_b = up16(2u * L.rs * nc_cap);
    L.late = staged && rows + v_b + im_b + pl_b + plane <= elem ? 1 : 0;
    L.v = L.late ? L.metric + rows : o;
    L.im = L.v + v_b;
    L.pl = L.im + im_b;
    if (!L.late) o += v_b + im_b + pl_b;
    // axis terms (gx, gy of up to two components) [4][ng][32], ng rounded up to
    // 4; last, for launches without axial elements leave them out
    L.ax = o;
    if (axi) o += 4u * 4u * ((ng + 3) & ~3) * kTileLanes;
    L.total = o;
    (void)elastic;
    return L;
  }
};

// A pointer into global memory, which the compiler cannot see where it was
// read from a structure in shared memory: without this the batched kernels
// access everything by generic loads and stores, which also stay in order with
// those to shared memory.
template <class T>
__device__ __forceinline__ T* glob(T* p) {
  __builtin_assume(__isGlobal(p));
  return p;
}

// Mode-dependent completion of a point (solver.cpp:924-944 fused):
//   normal: v = v_half + dt/2 a; u' = u + dt v + dt^2/2 a; v' = v + dt/2 a
//   final:  v = v_half + dt/2 a; u' = u                      (state complete)
//   init:   v unchanged;         u' = u                      (step 0)
__device__ __forceinline__ void complete_point(int mode, const StepScalars& sc, float u, float vh, float a, float& u_out,
                                               float& v_state, float& v_n) {
  if (mode == kModeInit) {
    v_n = vh;
    v_state = vh;
    u_out = u;
    return;
  }
  const float vn = fadd(vh, fmul(sc.half_dt, a));
  v_n = vn;
  if (mode == kModeFinal) {
    v_state = vn;
    u_out = u;
  } else {
    u_out = fadd(u, fadd(fmul(sc.rdt, vn), fmul(sc.half_dt2, a)));
    v_state = fadd(vn, fmul(sc.half_dt, a));
  }
}

// Start of a span of steps: the predictor on the whole of up to two fields in
// place (the state is complete after a final or initial step), the step that
// runs in final mode and, for batched solves, the buffer parity.
struct SpanField {
  float* u;
  float* v;
  const float* a;
  int64_t n;
};
static __global__ void begin_span_kernel(SpanField f0, SpanField f1, float rdt, float half_dt, float half_dt2,
                                         StepState* st, int32_t last_step, int32_t parity) {
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    st->last_step = last_step;
    st->parity = parity;
  }
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < f0.n + f1.n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const SpanField& f = i < f0.n ? f0 : f1;
    const int64_t q = i < f0.n ? i : i - f0.n;
    const float vi = f.v[q], ai = f.a[q];
    f.u[q] = fadd(f.u[q], fadd(fmul(rdt, vi), fmul(half_dt2, ai)));
    f.v[q] = fadd(vi, fmul(half_dt, ai));
  }
}

// Field rows in shared memory: components 0 and 1 as pairs, the only or third
// component in a plane of its own behind them.
// (AT: its offset, for rows kept in the element data).
template <int NC, int NPE, int AT = -1>
struct Rows {
  static constexpr bool PAIR = NC >= 2, ONE = NC != 2;
  static constexpr int ONE_AT = AT >= 0 ? AT : PAIR ? 2 * NPE * kTileLanes : 0;
  static constexpr int ONE_C = NC == 3 ? 2 : 0;  // the component of the single plane
  // place = point * 32 + lane
  __device__ __forceinline__ static void store(float* rows, int place, const float* x) {
    if constexpr (PAIR) *reinterpret_cast<float2*>(rows + 2 * place) = make_float2(x[0], x[1]);
    if constexpr (ONE) rows[ONE_AT + place] = x[ONE_C];
  }
  __device__ __forceinline__ static f2x pair(const float* rows, int place) {
    return *reinterpret_cast<const f2x*>(rows + 2 * place);
  }
  __device__ __forceinline__ static float one(const float* rows, int place) { return rows[ONE_AT + place]; }
  __device__ __forceinline__ static void load(const float* rows, int place, float* x) {
    if constexpr (PAIR) {
      const float2 v = *reinterpret_cast<const float2*>(rows + 2 * place);
      x[0] = v.x;
      x[1] = v.y;
    }
    if constexpr (ONE) x[ONE_C] = rows[ONE_AT + place];
  }
};

// Energy terms of one component of a point (solver.cpp:673-678, 900-915).
__device__ __forceinline__ void add_energy(double& kin, double& pot, float u, float f, float v_n, float a, double m,
                                           double kin_c) {
  pot = dadd(pot, dmul(static_cast<double>(u), static_cast<double>(f)));
  const double vv = v_n, aa = a;
  kin = dadd(kin, dmul(m, dsub(dmul(dmul(0.5, vv), vv), dmul(dmul(kin_c, aa), aa))));
}

// One tile of the fused step (the whole CTA).  `thp` is the tile's header
// (entry `tile` of the domain's tile table, or a copy of it).  `g_first`, if
// not negative, is this thread's first halo tile point (halo_tp entry
// blockDim.x - 1 - threadIdx.x), already loaded.  `bar` is an
// initialised mbarrier whose next phase to complete has parity `phase`.
// The tile's constant data (element data, descriptors, coefficients) is
// requested before dep_wait, ahead of the step before.
// Returns false (after recording the error) if the tile's bulk copies did
// not arrive within the wait limit.
template <int NG, int KIND, bool EL, int M>
__device__ __forceinline__ bool tile_step_body(const BlockDev& blk, const TiledDev& td, const StepScalars& sc,
                                               StepState* __restrict__ st, const StepNow& now, int32_t dep,
                                               double* __restrict__ epartial, int32_t tile, const TileHdr* thp,
                                               const TileLayout& L, unsigned char* smem_raw, uint64_t* bar,
                                               uint32_t phase, int32_t g_first = -1) {
  constexpr int EK = element_kind(KIND);
  constexpr bool SEP = is_separable(KIND), OFF = KIND == kAxisymOffAxis;
  using CE = ElemCfg<NG, EK, EL, M>;
  constexpr int NC = CE::NC;
  constexpr int NPE = NG * NG;
  constexpr int NI = NG - 2;  // inner points per direction
  constexpr bool AXI = is_axisym(KIND), STAGED = tile_data_staged(KIND);
  constexpr int W = kTileLanes, NT = W * NG;
  using R = Rows<NC, NPE>;
  using F = Rows<NC, NPE, STAGED ? (tile_arrays(KIND) - 1) * NPE * W : -1>;  // the f_xi rows
  const float* elem = reinterpret_cast<const float*>(smem_raw + L.metric);
  float* tu = reinterpret_cast<float*>(smem_raw + L.u);          // [NC][tp_cap]
  float* s_v = reinterpret_cast<float*>(smem_raw + L.v);         // [NC][nc_cap]
  float* s_im = reinterpret_cast<float*>(smem_raw + L.im);       // [nc_cap]
  uint16_t* pl = reinterpret_cast<uint16_t*>(smem_raw + L.pl);   // [nc_cap][rs] places, rank order
  float* su = reinterpret_cast<float*>(smem_raw + L.su);         // field rows, later contributions
  float* sfx = reinterpret_cast<float*>(smem_raw + L.sfx);       // f_xi rows
  float* ax = reinterpret_cast<float*>(smem_raw + L.ax) + (threadIdx.x & (W - 1));  // axis terms [4][NG][W]
  const int tp_cap = L.tp_cap, nc_cap = L.nc_cap;

  const TileHdr th = *thp;
  const int tid = threadIdx.x;
  const int lane = tid & (W - 1), i = tid / W;  // element, column
  // thread 0 issues the bulk copies; the halo tile points are gathered from
  // the last thread down, so thread 0 has the fewest of them
  const int tg = NT - 1 - tid;
  const int mode = now.mode;
  const bool energy = energy_step(now, sc.energy_every);
  const int nc4 = (th.nc + 3) & ~3;
  const uint32_t edge_b = 4u * nc4, list_b = 2u * td.rs * nc4;

  // 1. bulk copies of the element data, and of the edge complete points' u (v,
  //    1/M and place lists too unless they come late)
  if (tid == 0) {
    constexpr uint32_t eb = 4u * tile_staged_floats(KIND, NG);
    fence_proxy_async_smem();
    mbar_expect_tx(bar, eb + edge_b * NC + (L.late ? 0u : edge_b * (NC + 1) + list_b));
    if constexpr (STAGED)
      bulk_load(smem_raw + L.metric, glob(blk.metric) + static_cast<size_t>(th.tb) * tile_data_floats(KIND, NG), eb, bar);
    if (!L.late && nc4 > 0) {
      bulk_load(s_im, glob(td.inv_mass) + th.ebeg, edge_b, bar);
      bulk_load(pl, glob(td.plist) + static_cast<size_t>(th.pl_off) * td.rs, list_b, bar);
    }
  }
  // this lane's element and this column's descriptors, while the copies are in flight
  const bool active = lane < th.ne, direct = lane < th.nd;
  const bool inner_col = i > 0 && i < NG - 1;
  const bool all_direct = th.nd == th.ne;
  PointData pd{};
  bool axial = false;  // axisymmetric element on the axis (GLJ basis in xi)
  uint32_t dsc[NG];
  {
    const size_t e = static_cast<size_t>(th.tb) * W + lane;
    pd.c0 = glob(blk.coef0)[e];
    if constexpr (EL) pd.c1 = glob(blk.coef1)[e];
    if constexpr (AXI && !OFF) axial = glob(blk.axial)[e] != 0;
    if constexpr (SEP) {
      const float* m = glob(blk.metric) + static_cast<size_t>(th.tb) * tile_data_floats(KIND, NG) +
                       tile_staged_floats(KIND, NG) + lane;
      pd.xi_x = m[0];
      pd.eta_x = m[W];
      pd.eta_z = m[2 * W];
      pd.r = m[(3 + i) * W];
    } else if constexpr (!STAGED) {
      const float* m = glob(blk.metric) + static_cast<size_t>(th.tb) * tile_data_floats(KIND, NG) + lane;
      if constexpr (KIND == INSEM_RECT) {
        pd.xi_x = m[0];
        pd.eta_z = m[W];
        pd.jac = m[2 * W];
      } else {
        pd.xi_x = m[0];
        pd.xi_z = m[W];
        pd.eta_x = m[2 * W];
        pd.eta_z = m[3 * W];
        pd.jac = m[4 * W];
      }
    }
    const uint16_t* gd = glob(td.sdesc) + (static_cast<size_t>(tile) * NPE + i) * W + lane;
#pragma unroll
    for (int j = 0; j < NG; ++j) {
      dsc[j] = kSlotConstrained;
      if (j == 0 || j == NG - 1 || !inner_col || !all_direct) dsc[j] = gd[j * NG * W];
    }
  }
  if (tg < th.ntp - th.nc && g_first < 0) g_first = glob(td.halo_tp)[th.hl_off + tg];
  dep_wait(dep);
  if (tid == 0 && nc4 > 0) {
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      bulk_load(tu + c * tp_cap, glob(td.u_cur) + static_cast<size_t>(c) * td.ng + th.ebeg, edge_b, bar);
      if (!L.late) bulk_load(s_v + c * nc_cap, glob(td.v) + static_cast<size_t>(c) * td.ng + th.ebeg, edge_b, bar);
    }
  }
  // inner points of direct elements straight into their field rows
  const size_t g0 = static_cast<size_t>(th.cbeg + (i - 1) * NI * W + lane);  // j = 1; the rows are W points apart
  if (inner_col) {
    float x[NI > 0 ? NI : 1][NC];
#pragma unroll
    for (int j = 0; j < NI; ++j)
#pragma unroll
      for (int c = 0; c < NC; ++c) x[j][c] = __ldcg(glob(td.u_cur) + static_cast<size_t>(c) * td.ng + g0 + j * W);
#pragma unroll
    for (int j = 0; j < NI; ++j)
      if (direct) R::store(su, ((j + 1) * NG + i) * W + lane, x[j]);
  }
  // halo tile points
  for (int t = tg; t < th.ntp - th.nc; t += NT) {
    const int32_t g = t == tg ? g_first : glob(td.halo_tp)[th.hl_off + t];
#pragma unroll
    for (int c = 0; c < NC; ++c) tu[c * tp_cap + nc4 + t] = __ldcg(glob(td.u_cur) + static_cast<size_t>(c) * td.ng + g);
  }
  // constrained (hanging) slots straight into their field rows: the row's
  // weighted sum in row order (DofMap::gather, dof_map.hpp:110-115)
  for (int q = tg; q < th.ncs; q += NT) {
    const int32_t place = glob(td.cs_slot)[th.cs_off + q];
    const int2 row = glob(td.cs_row)[th.cs_off + q];
    float s[NC] = {};
    for (int32_t m0 = row.x; m0 < row.y; m0 += 4) {
      float w[4], x[4][NC];
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        const bool in = m0 + m < row.y;
        const int32_t g = in ? glob(td.row_dofs)[m0 + m] : 0;
        w[m] = in ? glob(td.row_w)[m0 + m] : 0.0f;
#pragma unroll
        for (int c = 0; c < NC; ++c) x[m][c] = in ? __ldcg(glob(td.u_cur) + static_cast<size_t>(c) * td.ng + g) : 0.0f;
      }
#pragma unroll
      for (int m = 0; m < 4; ++m)
#pragma unroll
        for (int c = 0; c < NC; ++c)
          if (m0 + m < row.y) s[c] = fadd(s[c], fmul(w[m], x[m][c]));
    }
    R::store(su, place, s);
  }
  const bool arrived = mbar_wait_bounded(bar, phase, kBulkWaitLimit);
  if (__syncthreads_or(!arrived)) {
    if (tid == 0) atomicExch(&st->error, 1);
    // give copies still in flight a second bounded wait before the shared memory is left
    mbar_wait_bounded(bar, phase, kBulkWaitLimit);
    return false;
  }

  // 2. the other slots' field rows from their tile points
#pragma unroll
  for (int j = 0; j < NG; ++j) {
    if (j == 0 || j == NG - 1 || !inner_col || !all_direct) {
      const bool have = active && dsc[j] != kSlotConstrained && !(j > 0 && j < NG - 1 && inner_col && direct);
      if (have) {
        float x[NC];
#pragma unroll
        for (int c = 0; c < NC; ++c) x[c] = tu[c * tp_cap + dsc[j]];
        R::store(su, (j * NG + i) * W + lane, x);
      }
    }
  }
  __syncthreads();

  // 3. derivatives and fluxes, one column per thread.  Rows come from shared
  // memory, the column's own field from registers; pairs of components are
  // summed in two-lane instructions.
  float dxr[NG], dxc[NG], w2c[NG];  // Dx row i, Dx column i, w_i w_j
#pragma unroll
  for (int l = 0; l < NG; ++l) {
    dxr[l] = cbasis(NG, axial ? 1 : 0, i * NG + l);
    dxc[l] = cbasis(NG, axial ? 1 : 0, l * NG + i);
    w2c[l] = cbasis(NG, 2, l * NG + i);
  }
  const float nzs = c_neg_zero;
  const f2x nz = pk2(nzs, nzs);
  float fe[NG][NC], dir[NG][2];  // f_eta column, hoop terms
  {
    f2x uc2[NG];
    float uc1[NG];
#pragma unroll
    for (int l = 0; l < NG; ++l) {
      if constexpr (R::PAIR) uc2[l] = R::pair(su, (l * NG + i) * W + lane);
      if constexpr (R::ONE) uc1[l] = R::one(su, (l * NG + i) * W + lane);
    }
#pragma unroll
    for (int j = 0; j < NG; ++j) {
      float uxi[NC], ueta[NC], upt[NC];
      if constexpr (R::PAIR) {
        f2x a = 0ull, b = 0ull;  // (+0, +0)
#pragma unroll
        for (int l = 0; l < NG; ++l) {
          a = add2(a, mul2(pk2(dxr[l], dxr[l]), R::pair(su, (j * NG + l) * W + lane), nz));
          b = add2(b, mulc2(uc2[l], cbasis(NG, 0, j * NG + l)));
        }
        const float2 av = upk2(a), bv = upk2(b), uv = upk2(uc2[j]);
        uxi[0] = av.x;
        uxi[1] = av.y;
        ueta[0] = bv.x;
        ueta[1] = bv.y;
        upt[0] = uv.x;
        upt[1] = uv.y;
      }
      if constexpr (R::ONE) {
        float a = 0.0f, b = 0.0f;
#pragma unroll
        for (int l = 0; l < NG; ++l) {
          a = fadd(a, fmul(dxr[l], R::one(su, (j * NG + l) * W + lane)));
          b = fadd(b, fmul(cbasis(NG, 0, j * NG + l), uc1[l]));
        }
        uxi[R::ONE_C] = a;
        ueta[R::ONE_C] = b;
        upt[R::ONE_C] = uc1[j];
      }
      if constexpr (SEP) {
        const int p = (j * NG + i) * W + lane;
        const float2 w = *reinterpret_cast<const float2*>(elem + tile_data_at(KIND, NPE, 0, p));
        pd.wr = w.x;
        pd.hoop = w.y;
        pd.xi_z = elem[tile_data_at(KIND, NPE, 2, p)];
      } else if constexpr (STAGED) {
        const int p = (j * NG + i) * W + lane;
        const float2 xi = *reinterpret_cast<const float2*>(elem + tile_data_at(KIND, NPE, 0, p));
        const float2 eta = *reinterpret_cast<const float2*>(elem + tile_data_at(KIND, NPE, 2, p));
        pd.xi_x = xi.x;
        pd.xi_z = xi.y;
        pd.eta_x = eta.x;
        pd.eta_z = eta.y;
        if constexpr (AXI) {
          const float2 w = *reinterpret_cast<const float2*>(elem + tile_data_at(KIND, NPE, 4, p));
          pd.wr = w.x;
          pd.hoop = w.y;
          pd.r = elem[tile_data_at(KIND, NPE, 6, p)];
        } else {
          pd.jac = elem[tile_data_at(KIND, NPE, 4, p)];
        }
      }
      dir[j][0] = dir[j][1] = 0.0f;
      float fx[NC];
      point_flux<NG, EK, EL, M, W, OFF>(pd, i, j, axial, uxi, ueta, upt, fx, fe[j], dir[j], ax, ax + NG * W,
                                          ax + 2 * NG * W, ax + 3 * NG * W, w2c[j]);
      F::store(sfx, (j * NG + i) * W + lane, fx);
    }
  }
  // velocity and 1/M of the inner points, in flight over the barrier
  const bool mine = inner_col && direct && mode == kModeNormal && !energy;
  float vi[NI > 0 ? NI : 1][NC], mi[NI > 0 ? NI : 1];
  if (mine) {
#pragma unroll
    for (int j = 0; j < NI; ++j) {
      mi[j] = glob(td.inv_mass)[g0 + j * W];
#pragma unroll
      for (int c = 0; c < NC; ++c) vi[j][c] = __ldcg(glob(td.v) + static_cast<size_t>(c) * td.ng + g0 + j * W);
    }
  }
  __syncthreads();
  // the element data is dead but for the f_xi rows: the late copies arrive
  // there while the divergence runs
  if (L.late && tid == 0) {
    fence_proxy_async_smem();
    mbar_expect_tx(bar + 1, edge_b * (NC + 1) + list_b);
    if (nc4 > 0) {
#pragma unroll
      for (int c = 0; c < NC; ++c)
        bulk_load(s_v + c * nc_cap, glob(td.v) + static_cast<size_t>(c) * td.ng + th.ebeg, edge_b, bar + 1);
      bulk_load(s_im, glob(td.inv_mass) + th.ebeg, edge_b, bar + 1);
      bulk_load(pl, glob(td.plist) + static_cast<size_t>(th.pl_off) * td.rs, list_b, bar + 1);
    }
  }

  // 4. weak divergence (interleaved xi / eta terms), hoop and axis terms.  Inner
  // points of direct elements are finished here: their force is 0 + this one
  // contribution.  The others' contributions replace their field rows (which
  // nobody reads any more: the inner points read back only their own).
#pragma unroll
  for (int j = 0; j < NG; ++j) {
    float s[NC];
    if constexpr (R::PAIR) {
      f2x acc = 0ull;  // (+0, +0)
#pragma unroll
      for (int l = 0; l < NG; ++l) {
        acc = add2(acc, mul2(pk2(dxc[l], dxc[l]), F::pair(sfx, (j * NG + l) * W + lane), nz));
        acc = add2(acc, mulc2(pk2(fe[l][0], fe[l][1]), cbasis(NG, 0, l * NG + j)));
      }
      const float2 sv = upk2(acc);
      s[0] = sv.x;
      s[1] = sv.y;
    }
    if constexpr (R::ONE) {
      float acc = 0.0f;
#pragma unroll
      for (int l = 0; l < NG; ++l) {
        acc = fadd(acc, fmul(dxc[l], F::one(sfx, (j * NG + l) * W + lane)));
        acc = fadd(acc, fmul(cbasis(NG, 0, l * NG + j), fe[l][R::ONE_C]));
      }
      s[R::ONE_C] = acc;
    }
    float out[NC];
    point_divergence<NG, EK, EL, M, W>(i, j, axial, s, dir[j], dxc[0], [](int q) { return cbasis(NG, 0, q); }, ax,
                                         ax + NG * W, ax + 2 * NG * W, ax + 3 * NG * W, out);
    const int place = (j * NG + i) * W + lane;
    if (j > 0 && j < NG - 1 && mine) {
      float u[NC];
      R::load(su, place, u);
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const size_t gi = static_cast<size_t>(c) * td.ng + g0 + (j - 1) * W;
        const float a = fmul(fadd(0.0f, out[c]), mi[j - 1]);
        float u_out, v_state, v_n;
        complete_point(kModeNormal, sc, u[c], vi[j - 1][c], a, u_out, v_state, v_n);
        glob(td.u_nxt)[gi] = u_out;
        glob(td.v)[gi] = v_state;
      }
    } else {
      R::store(su, place, out);
    }
  }

  // 5. the late copies and every contribution have arrived.  This thread's
  //    first halo entry is fetched ahead of the barrier.
  int32_t hs_first = 0, hd_first = 0;
  if (tid < th.nhs) {
    hs_first = glob(td.hs_slot)[th.hs_off + tid];
    hd_first = glob(td.hs_dst)[th.hs_off + tid];
  }
  const bool late_arrived = !L.late || mbar_wait_bounded(bar + 1, phase, kBulkWaitLimit);
  if (__syncthreads_or(!late_arrived)) {
    if (tid == 0) atomicExch(&st->error, 1);
    mbar_wait_bounded(bar + 1, phase, kBulkWaitLimit);
    return false;
  }

  // 6. halo contributions out, each to its place in its halo point's list
  for (int q = tid; q < th.nhs; q += NT) {
    const int32_t place = q == tid ? hs_first : glob(td.hs_slot)[th.hs_off + q];
    const int32_t dst = q == tid ? hd_first : glob(td.hs_dst)[th.hs_off + q];
    float val[NC];
    R::load(su, place, val);
    if (dst >= 0) {
#pragma unroll
      for (int c = 0; c < NC; ++c) glob(td.hbuf)[static_cast<size_t>(c) * td.n_hbuf + dst] = val[c];
    } else {
      const int32_t mi2 = -1 - dst;
      for (int32_t d = glob(td.mdst_off)[mi2]; d < glob(td.mdst_off)[mi2 + 1]; ++d) {
        const int32_t p = glob(td.mdst)[d];
#pragma unroll
        for (int c = 0; c < NC; ++c) glob(td.hbuf)[static_cast<size_t>(c) * td.n_hbuf + p] = val[c];
      }
    }
  }

  // 7. edge complete points: a = f / M, corrector, predictor; energy partials
  double kin = 0.0, pot = 0.0;
  const int rs = td.rs;
  for (int t = tid; t < th.nc; t += NT) {
    const size_t g = static_cast<size_t>(th.ebeg) + t;
    const float im = s_im[t];
    // the point's force: its contributions added in rank order, 0 + f_0
    // first.  Four list entries come in one load; the values of the valid
    // ones (up to the entry flagged last) load together, then add in order.
    float fsum[NC] = {};
    bool more = true;
    for (int r0 = 0; more && r0 < rs; r0 += 4) {
      const uint2 w = *reinterpret_cast<const uint2*>(pl + t * rs + r0);
      const uint32_t e[4] = {w.x & 0xffffu, w.x >> 16, w.y & 0xffffu, w.y >> 16};
      bool valid[4];
      valid[0] = true;
#pragma unroll
      for (int k = 1; k < 4; ++k) valid[k] = valid[k - 1] && !(e[k - 1] & kLastPlace);
      float x[4][NC] = {};
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (valid[k]) R::load(su, e[k] & (kLastPlace - 1u), x[k]);
#pragma unroll
      for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int c = 0; c < NC; ++c)
          if (valid[k]) fsum[c] = fadd(fsum[c], x[k][c]);
      more = valid[3] && !(e[3] & kLastPlace);
    }
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const size_t gi = static_cast<size_t>(c) * td.ng + g;
      const float a = fmul(fsum[c], im);
      const float u = tu[c * tp_cap + t];
      float u_out, v_state, v_n;
      complete_point(mode, sc, u, s_v[c * nc_cap + t], a, u_out, v_state, v_n);
      glob(td.u_nxt)[gi] = u_out;
      glob(td.v)[gi] = v_state;
      if (mode != kModeNormal) glob(td.a)[gi] = a;
      if (energy) add_energy(kin, pot, u, fsum[c], v_n, a, glob(td.mass)[g], st->kin_c);
    }
  }
  // the inner points of direct elements in the other modes and on energy steps
  if (NI > 0 && (mode != kModeNormal || energy)) {
    for (int t = tid; t < NI * NI * W; t += NT) {
      const int q = t / W;
      if (t - q * W >= th.nd) continue;
      const int ci = q / (NI > 0 ? NI : 1) + 1, cj = q - (ci - 1) * NI + 1;
      const size_t g = static_cast<size_t>(th.cbeg) + t;
      const float im = glob(td.inv_mass)[g];
      float f[NC];
      R::load(su, (cj * NG + ci) * W + lane, f);
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const size_t gi = static_cast<size_t>(c) * td.ng + g;
        const float fc = fadd(0.0f, f[c]);
        const float a = fmul(fc, im);
        const float u = __ldcg(glob(td.u_cur) + gi);
        float u_out, v_state, v_n;
        complete_point(mode, sc, u, __ldcg(glob(td.v) + gi), a, u_out, v_state, v_n);
        glob(td.u_nxt)[gi] = u_out;
        glob(td.v)[gi] = v_state;
        if (mode != kModeNormal) glob(td.a)[gi] = a;
        if (energy) add_energy(kin, pot, u, fc, v_n, a, glob(td.mass)[g], st->kin_c);
      }
    }
  }
  if (energy) {
    // deterministic CTA reduction: warp shuffles in a fixed tree, then warps in order
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      kin = dadd(kin, __shfl_down_sync(0xffffffffu, kin, off));
      pot = dadd(pot, __shfl_down_sync(0xffffffffu, pot, off));
    }
    __shared__ double wk[NG], wp[NG];
    if (lane == 0) {
      wk[i] = kin;
      wp[i] = pot;
    }
    __syncthreads();
    if (tid == 0) {
      double k2 = 0.0, p2 = 0.0;
      for (int q = 0; q < NG; ++q) {
        k2 = dadd(k2, wk[q]);
        p2 = dadd(p2, wp[q]);
      }
      epartial[2 * tile] = k2;
      epartial[2 * tile + 1] = p2;
    }
  }
  return true;
}

// Resident CTAs per SM the compiler makes room for in the register file, from
// the warps each of an SM's four schedulers (16,384 registers) is to hold: 10
// (48 registers) for one component, 8 (64) for the Cartesian elastic classes,
// 9 to 6 (56 to 80) for the axisymmetric ones, where shared memory holds
// about as many CTAs, and 4 or 5 (128 or 96) at NG 8 and 9.  A step of 12
// boreholes of NG 6 and 7 took 444 us with the compiler's own choice (up to 164
// registers, 1 - 2 CTAs of the three-component classes) and 336 with this.
// Compared with one warp more or fewer are the separable elastic classes of NG
// 6 and 7 (kAxisymSeparable above) and, with 9 and 10 for 8, the curved elastic
// ones of NG 6 (147k elements 70.4 us a step for 65.4); the other entries follow
// the same rule without a comparison of their own.
template <int NG, int KIND, bool EL, int M>
constexpr int tile_min_ctas() {
  const int sep = NG >= 8 ? 5 : M == 1 ? 7 : NG == 7 ? 9 : 8;
  const int warps = !EL ? (NG >= 8 || (is_axisym(KIND) && M == 1) ? 8 : 10)
                    : is_separable(KIND) ? sep
                    : KIND != INSEM_AXISYM ? (NG >= 8 ? 5 : 8)
                    : NG >= 8 ? 4
                    : NG >= 6 ? 6
                    : M == 1 && NG == 5 ? 7
                                        : 8;
  return 4 * warps / NG > 1 ? 4 * warps / NG : 1;
}
// ONE_WAVE: the compiler's own choice of registers, for launches whose tiles
// are all resident at once anyway: there a tile's latency counts, and more
// registers keep more loads and sums in flight (3,600 order-4 axisymmetric
// elements 17.5 -> 17.0 us a step, 4,087 order-8 elements 14.4 -> 11.6; but
// 25,600 of these 33 -> 42).
template <int NG, int KIND, bool EL, int M, bool ONE_WAVE>
static __global__ void __launch_bounds__(TileCfg<NG>::THREADS, ONE_WAVE ? 1 : tile_min_ctas<NG, KIND, EL, M>())
    tile_step_kernel(BlockDev blk, TiledDev td, StepScalars sc, StepState* __restrict__ st,
                     double* __restrict__ epartial, int32_t tile0, StepIdx ix, TileLayout L) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  dep_begin(ix.dep);
  uint64_t* bar = reinterpret_cast<uint64_t*>(smem_raw + L.bar);
  if (threadIdx.x == 0) {
    mbar_init(bar, 1);
    mbar_init(bar + 1, 1);
  }
  __syncthreads();
  const int32_t tile = tile0 + blockIdx.x;
  tile_step_body<NG, KIND, EL, M>(blk, td, sc, st, step_now(st, ix), ix.dep, epartial, tile, td.tiles + tile, L,
                                  smem_raw, bar, 0u);
  dep_end(ix.dep);
}

// Tiles of many solves in one launch.  A segment is one block of one
// domain of one solve; its field buffers are chosen by that solve's parity.
struct TileSeg {
  BlockDev blk;
  TiledDev td;          // parity-0 view (u_cur = u0, u_nxt = u1)
  StepScalars sc;
  StepState* st;
  double* epartial;     // the domain's tile partials
};

// One work item of a batched tile launch: a tile of one segment, with a copy
// of its header, its solve's step state and its halo point list, so that a
// CTA needs one load of its item before it can read the segment, the state
// and its first halo tile points (in parallel) and issue the tile's bulk
// copies.
struct __align__(16) TileItem {
  TileHdr th;               // the tile's header (entry `tile` of the domain's table)
  const StepState* st;      // the segment's solve
  int32_t seg;              // segment index
  int32_t tile;             // tile index in the domain's table
  const int32_t* halo_tp;   // the tile's halo tile points (domain halo_tp + th.hl_off)
};
static_assert(sizeof(TileItem) == 80, "TileItem is loaded as 20 words");

// One CTA per work item (CTA b takes item b).  Items of solves past their
// last step (idle) are skipped: the CTA exits.  (CTAs that loop over items
// measured slower: the loop keeps about 40 more registers per thread live,
// which costs resident CTAs per SM.)  One shared memory layout serves the
// class (sized for its largest tile).
template <int NG, int KIND, bool EL, int M>
__device__ __forceinline__ void tile_batch_run(const TileSeg* __restrict__ segs, const TileItem* __restrict__ items,
                                               const StepIdx& ix, const TileLayout& L) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  dep_begin(ix.dep);
  __shared__ __align__(8) uint64_t bar[2];
  __shared__ __align__(16) TileSeg s_seg;   // the item's segment, read by the body from shared memory
  __shared__ __align__(16) TileItem s_it;
  __shared__ StepNow s_now;
  static_assert(sizeof(TileSeg) % 4 == 0, "TileSeg is copied as 32-bit words");
  if (threadIdx.x < 20)
    reinterpret_cast<uint32_t*>(&s_it)[threadIdx.x] = reinterpret_cast<const uint32_t*>(items + blockIdx.x)[threadIdx.x];
  if (threadIdx.x == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
  }
  __syncthreads();
  // this thread's first halo tile point, loaded beside the segment and the state
  const int tg = static_cast<int>(blockDim.x - 1 - threadIdx.x);
  const int32_t g_first = tg < s_it.th.ntp - s_it.th.nc ? s_it.halo_tp[tg] : -1;
  {
    // the segment's words; on steps of odd parity the words of u_cur and
    // u_nxt are exchanged (both candidates and the parity load together)
    constexpr int kUc = static_cast<int>((offsetof(TileSeg, td) + offsetof(TiledDev, u_cur)) / 4);
    constexpr int kUn = static_cast<int>((offsetof(TileSeg, td) + offsetof(TiledDev, u_nxt)) / 4);
    static_assert(kUn == kUc + 2, "u_cur and u_nxt are adjacent pointers");
    const uint32_t* src = reinterpret_cast<const uint32_t*>(segs + s_it.seg);
    uint32_t* dst = reinterpret_cast<uint32_t*>(&s_seg);
    for (int q = threadIdx.x; q < static_cast<int>(sizeof(TileSeg) / 4); q += blockDim.x) {
      if (q >= kUc && q < kUc + 4) {
        const uint32_t own = src[q], other = src[q < kUn ? q + 2 : q - 2];
        dst[q] = (s_it.st->parity ^ ix.k) & 1 ? other : own;
      } else {
        dst[q] = src[q];
      }
    }
  }
  if (threadIdx.x == blockDim.x - 1) s_now = step_now(s_it.st, ix);
  __syncthreads();
  const StepNow now = s_now;
  if (now.mode == kModeIdle) {
    dep_wait(ix.dep);
  } else {
    tile_step_body<NG, KIND, EL, M>(s_seg.blk, s_seg.td, s_seg.sc, s_seg.st, now, ix.dep, s_seg.epartial, s_it.tile,
                                    &s_it.th, L, smem_raw, bar, 0u, g_first);
  }
  dep_end(ix.dep);
}
template <int NG, int KIND, bool EL, int M>
static __global__ void __launch_bounds__(TileCfg<NG>::THREADS, tile_min_ctas<NG, KIND, EL, M>())
    tile_batch_kernel(const TileSeg* __restrict__ segs, const TileItem* __restrict__ items, StepIdx ix, TileLayout L) {
  tile_batch_run<NG, KIND, EL, M>(segs, items, ix, L);
}
// ------------------------------------------------------------ halo kernel
// Special terms of a halo point: ranges of its source contributions and
// coupling entries, Stacey index (or -1), components set to zero.
struct HaloRec {
  int32_t src0, src1, cpl0, cpl1, abs, zero;
};
// One fluid-solid interface entry of a point: the partner point in the other
// domain's device numbering and the interface coefficients.
struct __align__(16) CouplingEntry {
  int32_t partner;
  float cx, cz;
  int32_t pad;
};
// A domain's halo points: device points [n_complete, n_complete + n), the
// coupled ones last, in the order of the coupled chunks.
struct HaloDev {
  int32_t n = 0;
  const int32_t* off = nullptr;      // [n+1] each point's contributions in hbuf, ascending slot order
  const float* w = nullptr;          // its weight (constrained maps), nullptr when all are 1
  const int32_t* spec = nullptr;     // [n] special record or -1
  const HaloRec* rec = nullptr;
  const int32_t* src_which = nullptr;// source index of each contribution (row of the amplitude table)
  const float* src_coef = nullptr;   // [contributions][ncomp]
  const CouplingEntry* cpl = nullptr;
  const float* abs_coef = nullptr;   // [n_abs][ncomp*ncomp]
};

// What of a halo point is constant, requested ahead of the step's waits.
struct HaloPoint {
  float im = 0.0f;
  int32_t b = 0, e = 0;  // contributions
  HaloRec r{0, 0, 0, 0, -1, 0};
  CouplingEntry c{0, 0.0f, 0.0f, 0};  // the first coupling entry
};
__device__ __forceinline__ HaloPoint halo_point(const TiledDev& td, const HaloDev& hd, int32_t h, bool in) {
  HaloPoint p;
  if (in) {
    p.im = glob(td.inv_mass)[td.n_complete + h];
    p.b = glob(hd.off)[h];
    p.e = glob(hd.off)[h + 1];
    const int32_t sp = glob(hd.spec)[h];
    if (sp >= 0) {
      p.r = glob(hd.rec)[sp];
      if (p.r.cpl0 < p.r.cpl1) p.c = glob(hd.cpl)[p.r.cpl0];
    }
  }
  return p;
}

// Finishes halo point h of one domain (every thread of the CTA calls; `in`: it
// has a point): the assembled force from the halo buffer, then
// (solver.cpp:669-762) sources, coupling, a = f / M or the implicit Stacey
// solve, Dirichlet / axis zeros, and the mode's update.  `other` is the
// fluid's current pressure (solid domain) or the solid's new acceleration
// (fluid domain), in that domain's device numbering.  CTAs of 256 threads,
// `part` = the CTA's energy partial.
template <int NC, bool ELASTIC, bool LATE>
__device__ __forceinline__ void halo_finish(const TiledDev& td, const float* u_cur, float* u_nxt, const HaloDev& hd,
                                            const HaloPoint& hp, const float* other, int32_t other_ng, bool pm,
                                            const float* __restrict__ amp, int32_t n_amp, const StepScalars& sc,
                                            double h_damp, const StepState* __restrict__ st, const StepNow& now,
                                            double* __restrict__ epartial, int32_t part, int32_t h, bool in) {
  const int mode = now.mode;
  const int32_t step = now.step;
  const bool energy = energy_step(now, sc.energy_every);
  double kin = 0.0, pot = 0.0;
  if (in) {
    const int32_t g = td.n_complete + h;
    const int32_t b = hp.b, e = hp.e;
    // the point's own values and its partner's first, all loads in flight
    // together (the stores below may alias them for the compiler)
    float uc[NC], vc[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      uc[c] = load_step<LATE>(u_cur + static_cast<size_t>(c) * td.ng + g);
      vc[c] = load_step<LATE>(glob(td.v) + static_cast<size_t>(c) * td.ng + g);
    }
    const bool coupled = hp.r.cpl0 < hp.r.cpl1;
    float o[3] = {0.0f, 0.0f, 0.0f};
    auto partner = [&](int32_t gp) {
      if constexpr (ELASTIC) {
        o[0] = load_step<LATE>(other + gp);
      } else {  // written by this CTA, or by a launch this one has waited for
        o[0] = other[gp];
        o[1] = other[static_cast<size_t>(other_ng) + gp];
        if (pm) o[2] = other[static_cast<size_t>(2) * other_ng + gp];
      }
    };
    if (coupled) partner(hp.c.partner);
    float f[NC], a[NC];
    constexpr int K = 4;  // contributions gathered at once (conforming 2D points have at most 4)
    if (e - b <= K) {
      float vq[NC][K];
#pragma unroll
      for (int q = 0; q < K; ++q)
#pragma unroll
        for (int c = 0; c < NC; ++c) vq[c][q] = b + q < e ? load_step<LATE>(glob(td.hbuf) + static_cast<size_t>(c) * td.n_hbuf + b + q) : 0.0f;
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        float s = 0.0f;
#pragma unroll
        for (int q = 0; q < K; ++q)
          if (b + q < e) s = fadd(s, hd.w ? fmul(glob(hd.w)[b + q], vq[c][q]) : vq[c][q]);
        f[c] = s;
      }
    } else {
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        float s = 0.0f;
        for (int32_t q = b; q < e; ++q) {
          const float v = load_step<LATE>(glob(td.hbuf) + static_cast<size_t>(c) * td.n_hbuf + q);
          s = fadd(s, hd.w ? fmul(glob(hd.w)[q], v) : v);
        }
        f[c] = s;
      }
    }
    if (energy) {
#pragma unroll
      for (int c = 0; c < NC; ++c) pot = dadd(pot, dmul(static_cast<double>(uc[c]), static_cast<double>(f[c])));
    }
    for (int32_t q = hp.r.src0; q < hp.r.src1; ++q) {
      const float am = amp[static_cast<size_t>(glob(hd.src_which)[q]) * n_amp + step];
#pragma unroll
      for (int c = 0; c < NC; ++c) f[c] = fadd(f[c], fmul(glob(hd.src_coef)[static_cast<size_t>(q) * NC + c], am));
    }
    if (coupled) {
      const float hs = static_cast<float>(kSqrtHalf);
      CouplingEntry ce = hp.c;
      for (int32_t q = hp.r.cpl0;;) {
        if constexpr (ELASTIC) {
          const float p = o[0];
          if (pm) {
            const float t = fmul(fmul(hs, ce.cx), p);
            f[0] = fadd(f[0], t);
            f[1] = fadd(f[1], t);
          } else {
            f[0] = fadd(f[0], fmul(ce.cx, p));
          }
          f[NC - 1] = fadd(f[NC - 1], fmul(ce.cz, p));
        } else {
          const float ar = pm ? fmul(hs, fadd(o[0], o[1])) : o[0];
          const float az = pm ? o[2] : o[1];
          f[0] = fsub(f[0], fadd(fmul(ce.cx, ar), fmul(ce.cz, az)));
        }
        if (++q >= hp.r.cpl1) break;
        ce = glob(hd.cpl)[q];
        partner(ce.partner);
      }
    }
#pragma unroll
    for (int c = 0; c < NC; ++c) a[c] = fmul(f[c], hp.im);
    if (hp.r.abs >= 0) {
      const float* cc = glob(hd.abs_coef) + static_cast<size_t>(hp.r.abs) * NC * NC;
      double A[NC * NC], rhs[NC];
      const double mass = glob(td.mass)[g];
#pragma unroll
      for (int r = 0; r < NC; ++r) {
        rhs[r] = static_cast<double>(f[r]);
#pragma unroll
        for (int s2 = 0; s2 < NC; ++s2) {
          rhs[r] = dsub(rhs[r], dmul(static_cast<double>(cc[r * NC + s2]), static_cast<double>(vc[s2])));
          A[r * NC + s2] = dadd(dmul(h_damp, static_cast<double>(cc[r * NC + s2])), r == s2 ? mass : 0.0);
        }
      }
      solve_spd_dev(NC, A, rhs);
#pragma unroll
      for (int r = 0; r < NC; ++r) a[r] = static_cast<float>(rhs[r]);
    }
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      if (hp.r.zero & (1 << c)) a[c] = 0.0f;
      const size_t gi = static_cast<size_t>(c) * td.ng + g;
      float u_out, v_state, v_n;
      complete_point(mode, sc, uc[c], vc[c], a[c], u_out, v_state, v_n);
      u_nxt[gi] = u_out;
      glob(td.v)[gi] = v_state;
      glob(td.a)[gi] = a[c];
      glob(td.vn)[gi] = v_n;
      if (energy) {
        const double vv = v_n, aa = a[c];
        kin = dadd(kin, dmul(static_cast<double>(glob(td.mass)[g]), dsub(dmul(dmul(0.5, vv), vv), dmul(dmul(st->kin_c, aa), aa))));
      }
    }
  }
  if (energy) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      kin = dadd(kin, __shfl_down_sync(0xffffffffu, kin, off));
      pot = dadd(pot, __shfl_down_sync(0xffffffffu, pot, off));
    }
    __shared__ double wk[8], wp[8];
    if ((threadIdx.x & 31) == 0) {
      wk[threadIdx.x >> 5] = kin;
      wp[threadIdx.x >> 5] = pot;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      double k2 = 0.0, p2 = 0.0;
      for (int q = 0; q < 8; ++q) {
        k2 = dadd(k2, wk[q]);
        p2 = dadd(p2, wp[q]);
      }
      epartial[2 * part] = k2;
      epartial[2 * part + 1] = p2;
    }
  }
}

// The halo points of one solve: CTAs [0, n_chunk) finish a coupled chunk each,
// the next nb_s the solid's points that are not coupled, the last nb_f the
// fluid's.  The fluid's coupling term reads its partners' new acceleration, so
// a chunk holds whole groups of coupled points, and its CTA finishes the
// solid's before the fluid's (and starts first: it takes twice as long).  One
// launch and one wait where two dependent launches took two, with the point's
// constant data requested ahead of it: a step of the cased borehole went from
// 17.0 to 12.8 us, one of 40,000 coupled order-5 elements from 25.6 to 22.4.  (A
// group larger than a CTA keeps two launches: n_chunk is 0 then, and the
// fluid's CTAs come after the solid's.)
constexpr int kHaloChunk = 256;
struct HaloArgs {
  TiledDev s_td, f_td;
  HaloDev s_hd, f_hd;
  int32_t nb_s, nb_f, n_chunk;
  int32_t n_amp;
  const int4* chunks;  // halo points [x, y) of the solid, [z, w) of the fluid
  const float* amp;
  StepScalars sc;
  int32_t ep_s, ep_f;  // first energy partials
  double h_damp;
  const StepState* st;
  double* epartial;
};
// NC: the solid's components (0: no solid); odd: the views' field buffers are
// exchanged (steps of odd parity).
template <int NC, bool LATE>
__device__ __forceinline__ void halo_block(const HaloArgs& A, bool odd, const StepNow& now, int32_t dep, int32_t block) {
  constexpr bool PM = NC == 3;
  constexpr int SC = NC == 0 ? 1 : NC;
  const float* s_cur = glob(odd ? A.s_td.u_nxt : A.s_td.u_cur);
  const float* f_cur = glob(odd ? A.f_td.u_nxt : A.f_td.u_cur);
  float* s_nxt = glob(odd ? const_cast<float*>(A.s_td.u_cur) : A.s_td.u_nxt);
  float* f_nxt = glob(odd ? const_cast<float*>(A.f_td.u_cur) : A.f_td.u_nxt);
  auto solid = [&](const HaloPoint& p, int32_t part, int32_t h, bool in) {
    halo_finish<SC, true, LATE>(A.s_td, s_cur, s_nxt, A.s_hd, p, f_cur, A.f_td.ng, PM, glob(A.amp), A.n_amp, A.sc, A.h_damp, A.st, now,
                          A.epartial, A.ep_s + part, h, in);
  };
  auto fluid = [&](const HaloPoint& p, int32_t part, int32_t h, bool in) {
    halo_finish<1, false, LATE>(A.f_td, f_cur, f_nxt, A.f_hd, p, glob(A.s_td.a), A.s_td.ng, PM, glob(A.amp), A.n_amp, A.sc, A.h_damp, A.st,
                          now, A.epartial, A.ep_f + part, h, in);
  };
  const int32_t t = threadIdx.x;
  if (NC > 0 && block < A.n_chunk) {
    const int4 ch = glob(A.chunks)[block];
    const int32_t hs = ch.x + t, hf = ch.z + t;
    const HaloPoint ps = halo_point(A.s_td, A.s_hd, hs, hs < ch.y);
    const HaloPoint pf = halo_point(A.f_td, A.f_hd, hf, hf < ch.w);
    dep_wait(dep);
    solid(ps, block, hs, hs < ch.y);
    __syncthreads();
    fluid(pf, block, hf, hf < ch.w);
    return;
  }
  const int32_t b = block - A.n_chunk;
  if (NC > 0 && b < A.nb_s) {
    const int32_t h = b * kHaloChunk + t;
    const HaloPoint p = halo_point(A.s_td, A.s_hd, h, h < A.s_hd.n);
    dep_wait(dep);
    solid(p, block, h, h < A.s_hd.n);
  } else {
    const int32_t h = (b - A.nb_s) * kHaloChunk + t;
    const HaloPoint p = halo_point(A.f_td, A.f_hd, h, h < A.f_hd.n);
    dep_wait(dep);
    fluid(p, block - A.nb_s, h, h < A.f_hd.n);
  }
}

// Register budgets of the halo kernels (256 threads per CTA): 3 to 5 CTAs per
// SM.  With 16 more or fewer per thread the dipole borehole (30k elements) took
// 49 and 47 us a step for 46, the ocean bottom (147k) 67 and 64 for 66.
template <int NC>
constexpr int kHaloRegs = NC == 3 ? 80 : NC == 2 ? 64 : 48;
template <int NC>
static __global__ void __maxnreg__(kHaloRegs<NC>) halo_step_kernel(const __grid_constant__ HaloArgs A, StepIdx ix) {
  dep_begin(ix.dep);
  halo_block<NC, false>(A, false, step_now(A.st, ix), ix.dep, blockIdx.x);
  dep_end(ix.dep);
}

// energy[sample] = (time, kinetic, potential) from the per-CTA partials of
// the tiled step: kinetic sums all sets, potential = -0.5 x each domain's
// u . f_int, elastic first (solver.cpp:673-678).  Partials of set d are
// [start_d, start_d + count_d).
__device__ __forceinline__ void tiled_energy_body(const double* __restrict__ epartial, int n_dom, int4 sets0, int4 sets1,
                                                  const StepNow& now, int32_t energy_every, double dt,
                                                  double* __restrict__ energy, int32_t max_samples) {
  __shared__ double sh[kReduceThreads];
  const int32_t step = now.step;
  if (!energy_step(now, energy_every)) return;
  const int starts[4] = {sets0.x, sets0.z, sets1.x, sets1.z};
  const int counts[4] = {sets0.y, sets0.w, sets1.y, sets1.w};
  double kin = 0.0, pot = 0.0;
  for (int d = 0; d < n_dom; ++d) {
    double pk = 0.0, pp = 0.0;
    // two partial sets per domain: tiles (set 2d) and halo (set 2d + 1)
    for (int part = 0; part < 2; ++part) {
      const int q = 2 * d + part;
      double sk = 0.0, spp = 0.0;
      for (int i = threadIdx.x; i < counts[q]; i += blockDim.x) {
        sk = dadd(sk, epartial[2 * (starts[q] + i)]);
        spp = dadd(spp, epartial[2 * (starts[q] + i) + 1]);
      }
      const double bk = block_reduce(sk, sh);
      __syncthreads();
      const double bp = block_reduce(spp, sh);
      __syncthreads();
      pk = dadd(pk, bk);
      pp = dadd(pp, bp);
    }
    kin = dadd(kin, pk);
    pot = dsub(pot, dmul(0.5, pp));
  }
  if (threadIdx.x == 0) {
    const int32_t sample = energy_every > 0 ? step / energy_every : 0;
    if (sample < max_samples) {
      energy[sample * 3 + 0] = dmul(static_cast<double>(step), dt);
      energy[sample * 3 + 1] = kin;
      energy[sample * 3 + 2] = pot;
    }
  }
}

static __global__ void tiled_energy_kernel(const double* __restrict__ epartial, int n_dom, int4 sets0, int4 sets1,
                                           const StepState* __restrict__ st, int32_t energy_every, double dt,
                                           double* __restrict__ energy, int32_t max_samples, StepIdx ix) {
  dep_begin(ix.dep);
  dep_wait(ix.dep);
  tiled_energy_body(epartial, n_dom, sets0, sets1, step_now(st, ix), energy_every, dt, energy, max_samples);
  dep_end(ix.dep);
}

// ------------------------------------------------------- batched step kernels
// The point-wise kernels of many solves in one launch each: one CTA per work
// item (segment, chunk); the segment carries one solve's pointers and
// scalars, the solve's StepState its step, mode and buffer parity.

// A segment is one solve (its views at parity 0).  LATE: launched as kDepLate.
template <int NC, bool LATE>
static __global__ void __maxnreg__(kHaloRegs<NC>) halo_batch_kernel(const HaloArgs* __restrict__ segs,
                                                                    const int2* __restrict__ items, StepIdx ix) {
  dep_begin(ix.dep);
  __shared__ __align__(16) uint32_t s_words[sizeof(HaloArgs) / 4];  // the segment
  static_assert(sizeof(HaloArgs) % 4 == 0, "HaloArgs is copied as 32-bit words");
  const int2 it = items[blockIdx.x];
  const uint32_t* src = reinterpret_cast<const uint32_t*>(segs + it.x);
  for (int q = threadIdx.x; q < static_cast<int>(sizeof(HaloArgs) / 4); q += kHaloChunk) s_words[q] = src[q];
  __syncthreads();
  const HaloArgs& A = *reinterpret_cast<const HaloArgs*>(s_words);
  const StepNow now = step_now(A.st, ix);
  if (now.mode == kModeIdle) {
    dep_wait(ix.dep);
  } else {
    halo_block<NC, LATE>(A, (A.st->parity ^ ix.k) & 1, now, ix.dep, it.y);
  }
  dep_end(ix.dep);
}

struct RecSeg {
  ReceiversDev rv;
  AllFields f0, f1;     // fields at parity 0 / 1
  const int32_t* acoustic_recv;
  int32_t n_acoustic;
  double dt;
  const RecordColumn* cols;
  int32_t n_cols;
  const StepState* st;
  int32_t record_every;
  double* traces;
  int32_t max_samples;
};

static __global__ void __launch_bounds__(kRecThreads) particle_velocity_batch_kernel(const RecSeg* __restrict__ segs,
                                                                                     const int2* __restrict__ items,
                                                                                     StepIdx ix) {
  dep_begin(ix.dep);
  dep_wait(ix.dep);
  const int2 it = items[blockIdx.x];
  const RecSeg& sg = segs[it.x];
  if (step_now(sg.st, ix).mode != kModeIdle)
    particle_velocity_body(sg.rv, (sg.st->parity ^ ix.k) & 1 ? sg.f1 : sg.f0, sg.acoustic_recv, sg.n_acoustic, sg.dt, 0,
                           it.y * kRecChunk + static_cast<int32_t>(threadIdx.x >> 5));
  dep_end(ix.dep);
}

static __global__ void __launch_bounds__(kRecThreads) record_batch_kernel(const RecSeg* __restrict__ segs,
                                                                          const int2* __restrict__ items, StepIdx ix) {
  dep_begin(ix.dep);
  dep_wait(ix.dep);
  const int2 it = items[blockIdx.x];
  const RecSeg& sg = segs[it.x];
  const StepNow now = step_now(sg.st, ix);
  if (now.mode != kModeIdle)
    record_body(sg.rv, (sg.st->parity ^ ix.k) & 1 ? sg.f1 : sg.f0, sg.cols, sg.n_cols, now.step, sg.record_every,
                sg.traces, sg.max_samples, it.y * kRecChunk + static_cast<int32_t>(threadIdx.x >> 5));
  dep_end(ix.dep);
}

struct EnergySeg {
  const double* epartial;
  int32_t n_dom;
  int4 s0, s1;
  const StepState* st;
  int32_t energy_every;
  double dt;
  double* energy;
  int32_t max_samples;
};

static __global__ void __launch_bounds__(kReduceThreads) energy_batch_kernel(const EnergySeg* __restrict__ segs,
                                                                             StepIdx ix) {
  dep_begin(ix.dep);
  dep_wait(ix.dep);
  const EnergySeg& sg = segs[blockIdx.x];
  const StepNow now = step_now(sg.st, ix);
  if (now.mode != kModeIdle)
    tiled_energy_body(sg.epartial, sg.n_dom, sg.s0, sg.s1, now, sg.energy_every, sg.dt, sg.energy, sg.max_samples);
  dep_end(ix.dep);
}

// Last kernel of a sequence of n batched steps: every solve's step count and
// buffer parity (a solve past its last step stays where it is).
static __global__ void batch_end_kernel(StepState* const* __restrict__ sts, int32_t n, int32_t steps) {
  pdl_wait();
  const int32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) {
    StepState* s = sts[i];
    const int32_t d = max(0, min(steps, s->last_step - s->step));
    s->step += d;
    s->parity ^= d & 1;
  }
}

}  // namespace insem_b200
