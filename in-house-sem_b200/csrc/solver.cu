// Device-resident twin of solver::Solver (cpp/include/insem/solver/solver.hpp:91-228)
// and its C ABI.  Fields, boundary data, sources and receivers live in HBM;
// the host only launches the steps (CUDA graphs of several) and copies traces,
// energy and state back on request.
//
// Step order per solver.cpp:917-963:
//   predictor (all domains) -> step += 1 ->
//   for elastic, acoustic:  element forces (gather fused) -> assemble (CSR, ascending slots)
//                           -> potential energy dot -> sources -> coupling
//                           -> a = f / M, Stacey solve, Dirichlet/axis
//   -> corrector -> acoustic particle velocity -> record -> energy.
#include <algorithm>
#include <map>
#include <memory>
#include <set>

#include "device_data.cuh"
#include "power.cuh"
#include "solver.cuh"
#include "stf.hpp"

namespace insem_b200 {

void DeviceDomainData::upload(const insem_cuda_domain& d, const insem_cuda_basis& basis) {
  medium = d.medium;
  INSEM_REQUIRE(medium == INSEM_ACOUSTIC || medium == INSEM_ELASTIC, INSEM_CUDA_ERR_INVALID, "unknown medium");
  m = d.azimuthal_order;
  ncomp = d.ncomp;
  INSEM_REQUIRE(ncomp == ncomp_of(medium, m), INSEM_CUDA_ERR_INVALID, "ncomp does not match medium and order");
  INSEM_REQUIRE(d.dofs.ngll == basis.ngll, INSEM_CUDA_ERR_INVALID, "DofMap and basis differ in ngll");
  dofs.upload(d.dofs);
  ng = dofs.n_global;
  npe = dofs.npe;
  n_elements = dofs.n_elements;
  INSEM_REQUIRE(static_cast<int64_t>(ng) * ncomp < (int64_t{1} << 31), INSEM_CUDA_ERR_INVALID, "domain too large");
  blocks.clear();
  blocks.resize(d.n_blocks);
  for (int b = 0; b < d.n_blocks; ++b) {
    blocks[b].upload(d.blocks[b], basis.ngll, medium);
    for (int32_t e : blocks[b].host_elements)
      INSEM_REQUIRE(e >= 0 && e < n_elements, INSEM_CUDA_ERR_INVALID, "block element out of range");
    any_axial |= blocks[b].any_axial;
  }
  std::vector<char> covered(n_elements, 0);
  for (const DeviceBlock& b : blocks)
    for (int32_t e : b.host_elements) covered[e] = 1;
  blocks_cover = std::count(covered.begin(), covered.end(), 1) == n_elements;
  host_mass = host_vec(d.mass, ng);
  mass.upload(host_mass);
  inv_mass.upload(host_vec(d.inv_mass, ng));
  n_abs = d.n_absorbing;
  const auto ap = host_vec(d.absorbing_points, n_abs);
  for (int32_t g : ap) INSEM_REQUIRE(g >= 0 && g < ng, INSEM_CUDA_ERR_INVALID, "absorbing point out of range");
  absorbing_points.upload(ap);
  absorbing_coef.upload(host_vec(d.absorbing_coef, static_cast<std::size_t>(n_abs) * ncomp * ncomp));
  std::vector<int64_t> z;
  const auto dp = host_vec(d.dirichlet_points, d.n_dirichlet);
  for (int c = 0; c < ncomp; ++c)
    for (int32_t g : dp) {
      INSEM_REQUIRE(g >= 0 && g < ng, INSEM_CUDA_ERR_INVALID, "Dirichlet point out of range");
      z.push_back(static_cast<int64_t>(c) * ng + g);
    }
  const auto axp = host_vec(d.axis_points, d.n_axis);
  const auto axc = host_vec(d.axis_components, d.n_axis_components);
  for (int32_t c : axc) {
    INSEM_REQUIRE(c >= 0 && c < ncomp, INSEM_CUDA_ERR_INVALID, "axis component out of range");
    for (int32_t g : axp) {
      INSEM_REQUIRE(g >= 0 && g < ng, INSEM_CUDA_ERR_INVALID, "axis point out of range");
      z.push_back(static_cast<int64_t>(c) * ng + g);
    }
  }
  host_zero = z;
  zero_idx.upload(z);
}

void DeviceDomainData::alloc_fields(cudaStream_t s) {
  if (fields_ready) return;
  const std::size_t nf = static_cast<std::size_t>(ncomp) * ng;
  u.resize(nf);
  v.resize(nf);
  a.resize(nf);
  f.resize(nf);
  f_local.resize(static_cast<std::size_t>(ncomp) * n_elements * npe);
  // zeroed in the order of the stream that uses them next (a memset on the
  // default stream is not ordered with the solver's non-blocking streams)
  u.zero(s);
  v.zero(s);
  a.zero(s);
  f.zero(s);
  f_local.zero(s);
  fields_ready = true;
}

Solver::Solver(const insem_cuda_problem& p, const insem_cuda_options* opt, bool setup_only,
               const insem_cuda_time* time) {
  if (opt) opts = *opt;
  else {
    opts = insem_cuda_options{};
    opts.use_graphs = 1;
    opts.check_finite = 1;
  }
  device = opts.device;
  DeviceGuard dg(device);
  CUDA_CHECK(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking));
  CUDA_CHECK(cudaEventCreate(&ev0));
  CUDA_CHECK(cudaEventCreate(&ev1));
  check_ngll(p.basis.ngll);
  ngll = p.basis.ngll;
  INSEM_REQUIRE(p.n_domains >= 1 && p.n_domains <= 2, INSEM_CUDA_ERR_INVALID, "a problem has 1 or 2 domains");
  INSEM_REQUIRE(p.record_every >= 1, INSEM_CUDA_ERR_INVALID, "record_every must be >= 1");
  INSEM_REQUIRE(p.energy_every >= 0, INSEM_CUDA_ERR_INVALID, "energy_every must be >= 0");
  INSEM_REQUIRE((setup_only || time || p.dt > 0.0) && (time || p.n_steps >= 0), INSEM_CUDA_ERR_INVALID,
                "dt must be positive and n_steps >= 0");
  dt = p.dt;
  n_steps = p.n_steps;
  record_every = p.record_every;
  energy_every = p.energy_every;
  domains.resize(p.n_domains);
  bool need_dj = false;
  for (int i = 0; i < p.n_domains; ++i) {
    domains[i].upload(p.domains[i], p.basis);
    need_dj |= domains[i].any_axial;
  }
  basis.upload(p.basis, need_dj);
  for (int i = 0; i < p.n_domains; ++i) {
    if (domains[i].medium == INSEM_ELASTIC) solid = i;
    else fluid = i;
  }
  INSEM_REQUIRE(p.n_domains == 1 || (solid >= 0 && fluid >= 0), INSEM_CUDA_ERR_INVALID,
                "two domains must be one acoustic and one elastic");
  build_coupling(p.coupling);
  st = static_cast<StepState*>(device_alloc(sizeof(StepState)));
  CUDA_CHECK(cudaMemset(st, 0, sizeof(StepState)));
  partial.resize(static_cast<std::size_t>(kReduceBlocks) * 4);
  if (time) {
    // Solver::Solver (solver.cpp:131-144)
    stable_dt_estimate = stable_dt();
    if (time->dt > 0.0) {
      INSEM_REQUIRE(time->dt <= stable_dt_estimate, INSEM_CUDA_ERR_INVALID,
                    "time step " + std::to_string(time->dt) + " s exceeds the estimated stability limit " +
                        std::to_string(stable_dt_estimate) + " s");
      dt = time->dt;
    } else {
      INSEM_REQUIRE(time->safety > 0.0 && time->safety <= 1.0, INSEM_CUDA_ERR_INVALID,
                    "time step safety factor must be in (0, 1]");
      dt = time->safety * stable_dt_estimate;
    }
    if (time->n_steps > 0) n_steps = time->n_steps;
    else if (time->duration > 0.0) n_steps = static_cast<int32_t>(std::ceil(time->duration / dt - 1e-9));
    else n_steps = 0;
  }
  build_sources(p);
  build_receivers(p);
  const int32_t n_energy = energy_every > 0 ? n_steps / energy_every + 1 : 0;
  energy.resize(static_cast<std::size_t>(std::max(n_energy, 1)) * 3);
  energy.zero();
  {
    StepState hs{};
    hs.kin_c = dt * dt / 8.0;
    CUDA_CHECK(cudaMemcpy(st, &hs, sizeof(hs), cudaMemcpyHostToDevice));
  }
  // the two-pass path's global fields and element-local forces; the tiled
  // path keeps its own fields and allocates these only for internal_forces()
  if (setup_only || opts.path == 1)
    for (auto& d : domains) d.alloc_fields();
  if (!setup_only && opts.path != 1) build_tiled(p);
  if (!setup_only) prepare_noalloc();
  // uploads and zeroing ran on the legacy stream and this solver's stream;
  // other streams (other solvers, batches) are not waited for
  CUDA_CHECK(cudaStreamSynchronize(nullptr));
  CUDA_CHECK(cudaStreamSynchronize(stream));
}

Solver::~Solver() {
  DeviceGuard dg(device);
  // buffers go back to the pool below: the stream must be done with them
  if (stream) cudaStreamSynchronize(stream);
  if (graph_exec) cudaGraphExecDestroy(graph_exec);
  for (auto& kv : tgraph) cudaGraphExecDestroy(kv.second);
  device_free(st);
  if (ev0) cudaEventDestroy(ev0);
  if (ev1) cudaEventDestroy(ev1);
  if (stream) cudaStreamDestroy(stream);
}

void Solver::build_coupling(const insem_cuda_coupling& c) {
  n_cpl = c.n;
  if (n_cpl == 0) return;
  INSEM_REQUIRE(solid >= 0 && fluid >= 0, INSEM_CUDA_ERR_INVALID, "coupling needs both media");
  const auto fp = host_vec(c.fluid_points, n_cpl), sp = host_vec(c.solid_points, n_cpl);
  std::set<int32_t> fs, ss;
  for (int i = 0; i < n_cpl; ++i) {
    INSEM_REQUIRE(fp[i] >= 0 && fp[i] < domains[fluid].ng && sp[i] >= 0 && sp[i] < domains[solid].ng,
                  INSEM_CUDA_ERR_INVALID, "coupling point out of range");
    fs.insert(fp[i]);
    ss.insert(sp[i]);
  }
  // Repeated points make the per-point updates order-dependent: keep the
  // reference's sequential order then.
  cpl_serial_fluid = static_cast<int>(fs.size()) != n_cpl;
  cpl_serial_solid = static_cast<int>(ss.size()) != n_cpl;
  cpl_fluid.upload(fp);
  cpl_solid.upload(sp);
  cpl_cx.upload(host_vec(c.cx, n_cpl));
  cpl_cz.upload(host_vec(c.cz, n_cpl));
}

void Solver::build_sources(const insem_cuda_problem& p) {
  n_sources = p.n_sources;
  n_amp = n_steps + 1;
  std::vector<float> amp(static_cast<std::size_t>(std::max(n_sources, 1)) * n_amp, 0.0f);
  // Per domain: point -> ordered (source, coef) contributions.
  std::vector<std::map<int32_t, std::vector<std::pair<int32_t, std::vector<float>>>>> per(domains.size());
  for (int s = 0; s < n_sources; ++s) {
    const insem_cuda_source& so = p.sources[s];
    INSEM_REQUIRE(so.domain >= 0 && so.domain < static_cast<int>(domains.size()), INSEM_CUDA_ERR_INVALID,
                  "source domain out of range");
    const auto& d = domains[so.domain];
    const auto pts = host_vec(so.points, so.n_points);
    const auto coef = host_vec(so.coef, static_cast<std::size_t>(so.n_points) * d.ncomp);
    for (int i = 0; i < so.n_points; ++i) {
      INSEM_REQUIRE(pts[i] >= 0 && pts[i] < d.ng, INSEM_CUDA_ERR_INVALID, "source point out of range");
      std::vector<float> cs(d.ncomp);
      for (int c = 0; c < d.ncomp; ++c) cs[c] = coef[static_cast<std::size_t>(c) * so.n_points + i];
      per[so.domain][pts[i]].push_back({s, cs});
    }
    for (int k = 0; k < n_amp; ++k)
      amp[static_cast<std::size_t>(s) * n_amp + k] = static_cast<float>(stf_value(so.stf, k * dt));
  }
  src_amp.upload(amp);
  src_per_point = per;
  src.resize(domains.size());
  for (std::size_t di = 0; di < domains.size(); ++di) {
    std::vector<int32_t> points, offsets{0}, which;
    std::vector<float> coefs;
    for (const auto& [g, list] : per[di]) {
      points.push_back(g);
      for (const auto& [s, cs] : list) {
        which.push_back(s);
        coefs.insert(coefs.end(), cs.begin(), cs.end());
      }
      offsets.push_back(static_cast<int32_t>(which.size()));
    }
    auto& sd = src[di];
    sd.n_points = static_cast<int32_t>(points.size());
    sd.points.upload(points);
    sd.offsets.upload(offsets);
    sd.source.upload(which);
    sd.coef.upload(coefs);
  }
}

void Solver::build_receivers(const insem_cuda_problem& p) {
  n_receivers = p.n_receivers;
  std::vector<int32_t> offsets{0}, points, dom, acoustic;
  std::vector<float> value, ddx, ddz;
  std::vector<double> rho;
  std::vector<RecordColumn> cols;
  for (int r = 0; r < n_receivers; ++r) {
    const insem_cuda_receiver& rc = p.receivers[r];
    INSEM_REQUIRE(rc.domain >= 0 && rc.domain < static_cast<int>(domains.size()), INSEM_CUDA_ERR_INVALID,
                  "receiver domain out of range");
    const auto& d = domains[rc.domain];
    const auto pts = host_vec(rc.points, rc.n_points);
    for (int32_t g : pts) INSEM_REQUIRE(g >= 0 && g < d.ng, INSEM_CUDA_ERR_INVALID, "receiver point out of range");
    points.insert(points.end(), pts.begin(), pts.end());
    const auto vv = host_vec(rc.value, rc.n_points), dx = host_vec(rc.d_dx, rc.n_points),
               dz = host_vec(rc.d_dz, rc.n_points);
    value.insert(value.end(), vv.begin(), vv.end());
    ddx.insert(ddx.end(), dx.begin(), dx.end());
    ddz.insert(ddz.end(), dz.begin(), dz.end());
    offsets.push_back(static_cast<int32_t>(points.size()));
    dom.push_back(rc.domain);
    rho.push_back(rc.rho);
    const auto qs = host_vec(rc.quantities, rc.n_quantities);
    // only receivers that record it integrate the particle velocity
    if (d.medium == INSEM_ACOUSTIC && std::count(qs.begin(), qs.end(), INSEM_Q_PARTICLE_VELOCITY) > 0)
      acoustic.push_back(r);
    for (int32_t q : qs) {
      TraceInfo ti;
      ti.first_col = static_cast<int32_t>(cols.size());
      if (q == INSEM_Q_PARTICLE_VELOCITY) {
        INSEM_REQUIRE(d.medium == INSEM_ACOUSTIC, INSEM_CUDA_ERR_INVALID, "particle_velocity needs an acoustic receiver");
        cols.push_back({r, 3, 3, 0});
        cols.push_back({r, 3, 4, 0});
      } else {
        const bool elastic_q = q == INSEM_Q_DISPLACEMENT || q == INSEM_Q_VELOCITY || q == INSEM_Q_ACCELERATION;
        INSEM_REQUIRE(elastic_q == (d.medium == INSEM_ELASTIC) && (elastic_q || q == INSEM_Q_PRESSURE),
                      INSEM_CUDA_ERR_INVALID, "quantity does not exist in the receiver's medium");
        const int32_t field = q == INSEM_Q_VELOCITY ? 1 : q == INSEM_Q_ACCELERATION ? 2 : 0;
        if (d.medium == INSEM_ELASTIC && d.m == 1) {
          cols.push_back({r, field, 1, 0});
          cols.push_back({r, field, 2, 0});
          cols.push_back({r, field, 0, 2});
        } else {
          for (int c = 0; c < d.ncomp; ++c) cols.push_back({r, field, 0, c});
        }
      }
      ti.ncomp = static_cast<int32_t>(cols.size()) - ti.first_col;
      traces.push_back(ti);
    }
  }
  n_cols = static_cast<int32_t>(cols.size());
  rec_offsets.upload(offsets);
  rec_points.upload(points);
  rec_value.upload(value);
  rec_ddx.upload(ddx);
  rec_ddz.upload(ddz);
  rec_rho.upload(rho);
  rec_domain.upload(dom);
  rec_acoustic.upload(acoustic);
  n_acoustic_rec = static_cast<int32_t>(acoustic.size());
  rec_pv.resize(static_cast<std::size_t>(std::max(n_receivers, 1)) * 4);
  rec_pv.zero();
  rec_cols.upload(cols);
  max_samples = n_steps / record_every + 1;
  trace_buf.resize(static_cast<std::size_t>(std::max(n_cols, 1)) * max_samples);
  trace_buf.zero();
}

ReceiversDev Solver::receivers_view() {
  ReceiversDev r;
  r.n = n_receivers;
  r.offsets = rec_offsets.get();
  r.points = rec_points.get();
  r.value = rec_value.get();
  r.d_dx = rec_ddx.get();
  r.d_dz = rec_ddz.get();
  r.rho = rec_rho.get();
  r.domain = rec_domain.get();
  r.pv = rec_pv.get();
  return r;
}

AllFields Solver::fields_view() {
  AllFields f{};
  for (std::size_t i = 0; i < domains.size() && i < 2; ++i)
    f.d[i] = {domains[i].u.get(), domains[i].v.get(), domains[i].a.get(), domains[i].ng};
  return f;
}

void Solver::internal_forces(DeviceDomainData& d, const float* u_global, float* f_global) {
  d.alloc_fields(stream);
  for (const DeviceBlock& b : d.blocks) {
    ElementLaunch a;
    a.basis = basis.view();
    a.blk = b.view();
    a.u_in = u_global;
    a.l2g = d.dofs.l2g.get();
    a.rows = d.dofs.rows();
    a.n_global = d.ng;
    a.f_local = d.f_local.get();
    a.gather = true;
    a.elastic = d.medium == INSEM_ELASTIC;
    a.stream = stream;
    launch_element_forces(ngll, a);
  }
  launch_assemble(d.dofs, d.ncomp, d.f_local.get(), f_global, stream);
}

// compute_acceleration (solver.cpp:669-691) for one domain.
void Solver::domain_acceleration(int di, int pot_set, int force_energy, double h, int step_override) {
  DeviceDomainData& d = domains[di];
  internal_forces(d, d.u.get(), d.f.get());
  dot_partial_kernel<<<kReduceBlocks, kReduceThreads, 0, stream>>>(
      d.u.get(), d.f.get(), static_cast<int64_t>(d.ncomp) * d.ng, st, energy_every, force_energy,
      partial.get() + static_cast<std::size_t>(pot_set) * kReduceBlocks);
  CUDA_LAUNCH_CHECK();
  const auto& sd = src[di];
  if (sd.n_points > 0) {
    SourcesDev s;
    s.n_points = sd.n_points;
    s.points = sd.points.get();
    s.offsets = sd.offsets.get();
    s.source = sd.source.get();
    s.coef = sd.coef.get();
    s.amp = src_amp.get();
    s.n_amp = n_amp;
    sources_kernel<<<ceil_div(sd.n_points, 128), 128, 0, stream>>>(s, st, step_override, d.f.get(), d.ng, d.ncomp);
    CUDA_LAUNCH_CHECK();
  }
  coupling_forces(di);
  inv_mass_kernel<<<grid_for(static_cast<int64_t>(d.ng) * d.ncomp), 256, 0, stream>>>(
      d.f.get(), d.inv_mass.get(), d.a.get(), d.ng, d.ncomp);
  CUDA_LAUNCH_CHECK();
  if (d.n_abs > 0) {
    stacey_kernel<<<ceil_div(d.n_abs, 128), 128, 0, stream>>>(d.n_abs, d.absorbing_points.get(),
                                                               d.absorbing_coef.get(), d.mass.get(), d.f.get(),
                                                               d.v.get(), d.a.get(), d.ng, d.ncomp, h);
    CUDA_LAUNCH_CHECK();
  }
  zero_constrained(d, d.a.get());
}

void Solver::zero_constrained(DeviceDomainData& d, float* x) {
  if (d.host_zero.empty()) return;
  zero_kernel<<<ceil_div(static_cast<int64_t>(d.host_zero.size()), 256), 256, 0, stream>>>(
      static_cast<int32_t>(d.host_zero.size()), d.zero_idx.get(), x);
  CUDA_LAUNCH_CHECK();
}

// add_coupling_forces (solver.cpp:693-727) into domains[di].f.
void Solver::coupling_forces(int di) {
  if (n_cpl == 0) return;
  DeviceDomainData& d = domains[di];
  const bool pm = d.m == 1;
  if (d.medium == INSEM_ELASTIC) {
    coupling_solid_kernel<<<cpl_serial_solid ? 1 : ceil_div(n_cpl, 128), 128, 0, stream>>>(
        n_cpl, cpl_fluid.get(), cpl_solid.get(), cpl_cx.get(), cpl_cz.get(), domains[fluid].u.get(), d.f.get(),
        d.ng, pm, cpl_serial_solid);
  } else {
    const auto& s = domains[solid];
    coupling_fluid_kernel<<<cpl_serial_fluid ? 1 : ceil_div(n_cpl, 128), 128, 0, stream>>>(
        n_cpl, cpl_fluid.get(), cpl_solid.get(), cpl_cx.get(), cpl_cz.get(), s.a.get(), s.ng, d.f.get(),
        s.m == 1, cpl_serial_fluid);
  }
  CUDA_LAUNCH_CHECK();
}

// Runs `body` (launches on `stream` only) n times: captured once as a CUDA
// graph, which the stream replays.  The graph is kept until the caller has
// waited for the stream.
void Solver::replay(int n, const std::function<void()>& body, std::vector<cudaGraphExec_t>& graphs) {
  if (n <= 0) return;
  cudaGraph_t g = nullptr;
  CUDA_CHECK(cudaStreamBeginCapture(stream, cudaStreamCaptureModeThreadLocal));
  try {
    body();
  } catch (...) {
    // leave capture mode before the error propagates
    if (cudaStreamEndCapture(stream, &g) == cudaSuccess && g) cudaGraphDestroy(g);
    cudaGetLastError();
    throw;
  }
  CUDA_CHECK(cudaStreamEndCapture(stream, &g));
  cudaGraphExec_t ge = nullptr;
  const cudaError_t e = cudaGraphInstantiate(&ge, g, 0);
  cudaGraphDestroy(g);
  CUDA_CHECK(e);
  graphs.push_back(ge);
  for (int i = 0; i < n; ++i) CUDA_CHECK(cudaGraphLaunch(ge, stream));
}

namespace {
// The start vectors' numbers: std::uniform_real_distribution<double>(-1, 1)
// over std::mt19937(12345), rounded to float.  The Mersenne twister (Matsumoto
// and Nishimura 1998) refilled a state at a time, in loops the compiler
// vectorises; two outputs a, b make (a + b 2^32) / 2^64, as the standard's
// generate_canonical takes 53 bits from a 32-bit engine.
class StartVector {
 public:
  StartVector() {
    mt_[0] = 12345u;
    for (uint32_t k = 1; k < kN; ++k) mt_[k] = 1812433253u * (mt_[k - 1] ^ (mt_[k - 1] >> 30)) + k;
  }
  void fill(float* out, std::size_t n) {
    for (std::size_t i = 0; i < n; ++i) {
      if (at_ >= kN) refill();
      const double r = (static_cast<double>(out_[at_]) + static_cast<double>(out_[at_ + 1]) * 4294967296.0) / 18446744073709551616.0;
      out[i] = static_cast<float>((r < 1.0 ? r : std::nextafter(1.0, 0.0)) * 2.0 + -1.0);
      at_ += 2;  // 624 is even: a pair never straddles two states
    }
  }

 private:
  static constexpr uint32_t kN = 624, kM = 397;
  static uint32_t mix(uint32_t hi, uint32_t lo) {
    const uint32_t y = (hi & 0x80000000u) | (lo & 0x7fffffffu);
    return (y >> 1) ^ ((0u - (lo & 1u)) & 0x9908b0dfu);
  }
  void refill() {
    for (uint32_t k = 0; k < kN - kM; ++k) mt_[k] = mt_[k + kM] ^ mix(mt_[k], mt_[k + 1]);
    for (uint32_t k = kN - kM; k < kN - 1; ++k) mt_[k] = mt_[k + kM - kN] ^ mix(mt_[k], mt_[k + 1]);
    mt_[kN - 1] = mt_[kM - 1] ^ mix(mt_[kN - 1], mt_[0]);
    for (uint32_t k = 0; k < kN; ++k) {
      uint32_t y = mt_[k];
      y ^= y >> 11;
      y ^= (y << 7) & 0x9d2c5680u;
      y ^= (y << 15) & 0xefc60000u;
      out_[k] = y ^ (y >> 18);
    }
    at_ = 0;
  }
  uint32_t mt_[kN], out_[kN];
  uint32_t at_ = kN;
};
}  // namespace

// estimate_stable_dt (solver.cpp:583-619): 100 power iterations per domain
// with x ~ U(-1, 1), Rayleigh quotients in double; then coupled_lambda_max
// (solver.cpp:621-667): growth of the mass norm under the coupled operator, 120
// iterations, sqrt(ny / nx) from iteration 60 on.
double Solver::stable_dt() {
  DeviceGuard dg(device);
  struct Work {
    DeviceBuffer<float> x, f_local;
    DeviceBuffer<uint8_t> zero;
    DeviceBuffer<int32_t> cpl_off;
    DeviceBuffer<PowerEntry> cpl;
    DeviceBuffer<double> partial;
    std::vector<float> start;
  };
  std::vector<Work> work(domains.size());
  std::vector<float> start2[2];
  std::vector<cudaGraphExec_t> graphs;
  DeviceBuffer<double> pw(kPwCount);
  DeviceBuffer<uint32_t> counter(1);
  const double one = 1.0;
  struct Release {  // the work buffers and host vectors outlive the stream's use of them
    cudaStream_t s;
    std::vector<cudaGraphExec_t>& g;
    ~Release() {
      cudaStreamSynchronize(s);
      for (cudaGraphExec_t e : g) cudaGraphExecDestroy(e);
    }
  } release{stream, graphs};
  StartVector rng;
  pw.zero(stream);
  counter.zero(stream);
  // element forces of a domain's scaled field: the first block that launches
  // waits for what is ahead, unless a launch of this iteration did (`first`,
  // returned for the launches that follow)
  auto forces = [&](int di, bool first) {
    DeviceDomainData& d = domains[di];
    Work& w = work[di];
    for (const DeviceBlock& b : d.blocks) {
      if (b.n == 0) continue;
      ElementLaunch a;
      a.basis = basis.view();
      a.blk = b.view();
      a.u_in = w.x.get();
      a.l2g = d.dofs.l2g.get();
      a.rows = d.dofs.rows();
      a.n_global = d.ng;
      a.f_local = w.f_local.get();
      a.gather = true;
      a.scale = pw.get() + kPwScale;
      a.elastic = d.medium == INSEM_ELASTIC;
      a.dep = first ? kDepFirst : kDepLate;
      a.overlap = true;
      a.stream = stream;
      launch_element_forces(ngll, a);
      first = false;
    }
    return first;
  };
  auto point = [&](int di, int mode, bool late) {
    DeviceDomainData& d = domains[di];
    Work& w = work[di];
    PowerLaunch a;
    a.mode = mode;
    a.ncomp = d.ncomp;
    a.stream = stream;
    a.d.ng = d.ng;
    a.d.t_offsets = d.dofs.t_offsets.get();
    a.d.t_slots = d.dofs.t_slots.get();
    a.d.t_weights = d.dofs.weighted ? d.dofs.t_weights.get() : nullptr;
    a.d.f_local = w.f_local.get();
    a.d.x = w.x.get();
    a.d.mass = d.mass.get();
    a.d.inv_mass = d.inv_mass.get();
    a.d.zero = w.zero.get();
    a.d.cpl_off = w.cpl_off.get();
    a.d.cpl = w.cpl.get();
    a.d.partial = w.partial.get();
    a.d.counter = counter.get();
    a.d.pw = pw.get();
    a.d.late = late;
    if (mode != kPowerAlone) {
      const int oi = di == solid ? fluid : solid;
      a.d.other = work[oi].x.get();
      a.d.other_ng = domains[oi].ng;
      a.d.pm = domains[solid].m == 1;
      a.d.partial_s = work[solid].partial.get();
      a.d.blocks_s = power_blocks(domains[solid].ng);
    }
    launch_power(ngll, a);
  };
  auto begin = [&](int di, const std::vector<float>& x) {
    CUDA_CHECK(cudaMemcpyAsync(work[di].x.get(), x.data(), x.size() * sizeof(float), cudaMemcpyHostToDevice, stream));
    zero_constrained(domains[di], work[di].x.get());
  };
  auto reset = [&] {
    CUDA_CHECK(cudaMemsetAsync(pw.get() + kPwDone, 0, sizeof(double), stream));
    CUDA_CHECK(cudaMemcpyAsync(pw.get() + kPwScale, &one, sizeof(double), cudaMemcpyHostToDevice, stream));
  };
  constexpr int kPerGraph = 10;
  for (std::size_t di = 0; di < domains.size(); ++di) {
    DeviceDomainData& d = domains[di];
    Work& w = work[di];
    const std::size_t n = static_cast<std::size_t>(d.ncomp) * d.ng;
    w.x.resize(n);
    w.f_local.resize(static_cast<std::size_t>(d.ncomp) * d.n_elements * d.npe);
    w.f_local.zero(stream);  // elements of no block contribute nothing
    w.partial.resize(3 * static_cast<std::size_t>(power_blocks(d.ng)));
    std::vector<uint8_t> zero(std::max(d.ng, 1), 0);
    for (int64_t z : d.host_zero) zero[z % d.ng] |= static_cast<uint8_t>(1u << (z / d.ng));
    w.zero.upload(zero);
    w.start.resize(n);
    rng.fill(w.start.data(), n);
    begin(static_cast<int>(di), w.start);
    reset();
    replay(100 / kPerGraph, [&] {
      for (int k = 0; k < kPerGraph; ++k) {
        forces(static_cast<int>(di), true);
        point(static_cast<int>(di), kPowerAlone, false);
      }
    }, graphs);
  }
  if (n_cpl > 0) {
    int q = 0;
    for (int di : {solid, fluid}) {
      DeviceDomainData& d = domains[di];
      Work& w = work[di];
      // interface entries by point, in the interface's order
      const auto own = (di == solid ? cpl_solid : cpl_fluid).download(), other = (di == solid ? cpl_fluid : cpl_solid).download();
      const auto cx = cpl_cx.download(), cz = cpl_cz.download();
      std::vector<int32_t> off(static_cast<std::size_t>(d.ng) + 1, 0);
      for (int32_t g : own) ++off[g + 1];
      for (int g = 0; g < d.ng; ++g) off[g + 1] += off[g];
      std::vector<PowerEntry> e(n_cpl);
      std::vector<int32_t> fill(off.begin(), off.end() - 1);
      for (int i = 0; i < n_cpl; ++i) e[fill[own[i]]++] = PowerEntry{other[i], cx[i], cz[i]};
      w.cpl_off.upload(off);
      w.cpl.upload(e);
      auto& x = start2[q++];
      x.resize(static_cast<std::size_t>(d.ncomp) * d.ng);
      rng.fill(x.data(), x.size());
      begin(di, x);
    }
    reset();
    for (bool late : {false, true})
      replay(60 / kPerGraph, [&] {
        for (int k = 0; k < kPerGraph; ++k) {
          forces(fluid, forces(solid, true));
          point(solid, kPowerSolid, late);
          point(fluid, kPowerFluid, late);
        }
      }, graphs);
  }
  double h[kPwCount];
  CUDA_CHECK(cudaMemcpyAsync(h, pw.get(), sizeof(h), cudaMemcpyDeviceToHost, stream));
  CUDA_CHECK(cudaStreamSynchronize(stream));
  double lambda = h[kPwLambda];
  if (n_cpl > 0) lambda = std::max(lambda, h[kPwCoupled]);
  INSEM_REQUIRE(lambda > 0.0, INSEM_CUDA_ERR_INVALID, "could not estimate the stable time step (empty or rigid model?)");
  return 2.0 / std::sqrt(lambda);
}

// Kernels of the whole acceleration solve, elastic first (solver.cpp:674).
void Solver::compute_acceleration(int force_energy, double h, int step_override) {
  int set = 0;
  n_pot_sets = 0;
  if (solid >= 0) domain_acceleration(solid, 2 + set++, force_energy, h, step_override);
  if (fluid >= 0) domain_acceleration(fluid, 2 + set++, force_energy, h, step_override);
  n_pot_sets = set;
}

void Solver::observers(int force_energy, int init) {
  if (n_acoustic_rec > 0) {
    particle_velocity_kernel<<<ceil_div(n_acoustic_rec, kRecChunk), kRecThreads, 0, stream>>>(
        receivers_view(), fields_view(), rec_acoustic.get(), n_acoustic_rec, dt, init, StepIdx{-1});
    CUDA_LAUNCH_CHECK();
  }
  if (n_cols > 0) {
    record_kernel<<<ceil_div(n_cols, kRecChunk), kRecThreads, 0, stream>>>(receivers_view(), fields_view(), rec_cols.get(), n_cols,
                                                            st, record_every, trace_buf.get(), max_samples,
                                                            StepIdx{-1});
    CUDA_LAUNCH_CHECK();
  }
  if (energy_every > 0 || force_energy) {
    const double c = dt * dt / 8.0;
    int set = 0;
    for (auto& d : domains) {
      kinetic_partial_kernel<<<kReduceBlocks, kReduceThreads, 0, stream>>>(
          d.v.get(), d.a.get(), d.mass.get(), d.ng, d.ncomp, c, st, energy_every, force_energy,
          partial.get() + static_cast<std::size_t>(set++) * kReduceBlocks);
      CUDA_LAUNCH_CHECK();
    }
    energy_finalize_kernel<<<1, kReduceThreads, 0, stream>>>(partial.get(), set, n_pot_sets, st, energy_every,
                                                              force_energy, dt, energy.get(),
                                                              static_cast<int32_t>(energy.size() / 3));
    CUDA_LAUNCH_CHECK();
  }
}

void Solver::enqueue_step() {
  const float rdt = static_cast<float>(dt);
  const float half_dt = static_cast<float>(0.5 * dt);
  const float half_dt2 = static_cast<float>(0.5 * dt * dt);
  for (auto& d : domains) {
    const int64_t n = static_cast<int64_t>(d.ncomp) * d.ng;
    predictor_kernel<<<grid_for(n), 256, 0, stream>>>(d.u.get(), d.v.get(), d.a.get(), n, rdt, half_dt, half_dt2);
    CUDA_LAUNCH_CHECK();
  }
  advance_step_kernel<<<1, 1, 0, stream>>>(st, 1);
  CUDA_LAUNCH_CHECK();
  compute_acceleration(0, 0.5 * dt, -1);
  for (auto& d : domains) {
    const int64_t n = static_cast<int64_t>(d.ncomp) * d.ng;
    corrector_kernel<<<grid_for(n), 256, 0, stream>>>(d.v.get(), d.a.get(), n, half_dt);
    CUDA_LAUNCH_CHECK();
  }
  observers(0, 0);
}

void Solver::initialize() {
  // compute_acceleration(0, energy, explicit damping) then observers at t = 0
  // (Solver::initialize, solver.cpp:878-898).
  const int force = energy_every > 0 ? 1 : 0;
  compute_acceleration(force, 0.0, 0);
  observers(force, 1);
  initialized = true;
}

void Solver::set_state(int32_t medium, const double* u_in, const double* v_in) {
  INSEM_REQUIRE(!initialized, INSEM_CUDA_ERR_STATE, "initial conditions must be set before the first time step");
  int di = -1;
  for (std::size_t i = 0; i < domains.size(); ++i)
    if (domains[i].medium == medium) di = static_cast<int>(i);
  INSEM_REQUIRE(di >= 0, INSEM_CUDA_ERR_INVALID, "the model has no such medium");
  auto& d = domains[di];
  INSEM_REQUIRE(u_in && v_in, INSEM_CUDA_ERR_INVALID, "null state array");
  // rounded to float at the points' places on the device, zero where held
  const int32_t* perm = tiled ? tdom[di].perm.data() : nullptr;
  const int32_t stride = tiled ? tdom[di].ng : d.ng;
  const std::size_t nd = static_cast<std::size_t>(d.ncomp) * stride;
  auto copy = [&](const double* in, float* out) {
    std::vector<float> h(nd, 0.0f);
    for (int c = 0; c < d.ncomp; ++c) {
      const double* x = in + static_cast<std::size_t>(c) * d.ng;
      float* o = h.data() + static_cast<std::size_t>(c) * stride;
      for (int32_t g = 0; g < d.ng; ++g) o[perm ? perm[g] : g] = static_cast<float>(x[g]);
    }
    for (int64_t z : d.host_zero) {
      const int32_t g = static_cast<int32_t>(z % d.ng);
      h[static_cast<std::size_t>(z / d.ng) * stride + (perm ? perm[g] : g)] = 0.0f;
    }
    CUDA_CHECK(cudaMemcpy(out, h.data(), nd * sizeof(float), cudaMemcpyHostToDevice));
  };
  copy(u_in, tiled ? tdom[di].u_cur(parity) : d.u.get());
  copy(v_in, tiled ? tdom[di].v.get() : d.v.get());
  // a copy from pageable memory may return before its DMA has landed; the
  // readers run on the solver's non-blocking stream
  CUDA_CHECK(cudaStreamSynchronize(nullptr));
}

void Solver::advance(int32_t n) {
  DeviceGuard dg(device);
  INSEM_REQUIRE(n >= 0, INSEM_CUDA_ERR_INVALID, "negative step count");
  INSEM_REQUIRE(!in_batch, INSEM_CUDA_ERR_STATE, "this solve is stepped by a batch");
  if (snap_every <= 0) {
    advance_span(n);
    return;
  }
  // spans that end on snapshot steps, where the state is complete
  double ms = 0.0;
  if (!initialized) {
    advance_span(0);
    ms += last_ms;
    record_snapshot();
  }
  int32_t left = std::min<int32_t>(n, n_steps - step);
  while (left > 0) {
    const int32_t k = std::min<int32_t>(left, snap_every - step % snap_every);
    advance_span(k);
    ms += last_ms;
    left -= k;
    if (step % snap_every == 0) record_snapshot();
  }
  last_ms = ms;
}

void Solver::advance_span(int32_t n) {
  if (tiled) {
    int32_t dummy = 0;
    advance_tiled(n, nullptr, nullptr, &dummy);
    return;
  }
  CUDA_CHECK(cudaEventRecord(ev0, stream));
  if (!initialized) initialize();
  const int32_t todo = std::min<int32_t>(n, n_steps - step);
  if (todo > 0) {
    if (opts.use_graphs) {
      ensure_graph();
      for (int32_t s = 0; s < todo; ++s) CUDA_CHECK(cudaGraphLaunch(graph_exec, stream));
    } else {
      for (int32_t s = 0; s < todo; ++s) enqueue_step();
    }
    step += todo;
  }
  CUDA_CHECK(cudaEventRecord(ev1, stream));
  if (opts.check_finite) {
    for (auto& d : domains) {
      const int64_t nn = static_cast<int64_t>(d.ncomp) * d.ng;
      finite_check_kernel<<<grid_for(nn), 256, 0, stream>>>(d.u.get(), nn, nullptr, 0, st);
      CUDA_LAUNCH_CHECK();
    }
  }
  CUDA_CHECK(cudaStreamSynchronize(stream));
  float ms = 0.0f;
  CUDA_CHECK(cudaEventElapsedTime(&ms, ev0, ev1));
  last_ms = ms;
  if (opts.check_finite) {
    StepState hs;
    CUDA_CHECK(cudaMemcpy(&hs, st, sizeof(hs), cudaMemcpyDeviceToHost));
    if (hs.nonfinite) nonfinite_seen = true;
    INSEM_REQUIRE(!hs.nonfinite, INSEM_CUDA_ERR_NONFINITE, "the solution contains NaN or Inf (unstable time step?)");
  }
}

// Captures one step into a CUDA graph (once) and counts its kernel nodes.
void Solver::ensure_graph() {
  if (graph_exec) return;
  cudaGraph_t g = nullptr;
  CUDA_CHECK(cudaStreamBeginCapture(stream, cudaStreamCaptureModeThreadLocal));
  try {
    enqueue_step();
  } catch (...) {
    cudaStreamEndCapture(stream, &g);
    if (g) cudaGraphDestroy(g);
    throw;
  }
  CUDA_CHECK(cudaStreamEndCapture(stream, &g));
  std::size_t n_nodes = 0;
  CUDA_CHECK(cudaGraphGetNodes(g, nullptr, &n_nodes));
  std::vector<cudaGraphNode_t> nodes(n_nodes);
  if (n_nodes) CUDA_CHECK(cudaGraphGetNodes(g, nodes.data(), &n_nodes));
  kernels_per_step = 0;
  for (auto nd : nodes) {
    cudaGraphNodeType t;
    CUDA_CHECK(cudaGraphNodeGetType(nd, &t));
    if (t == cudaGraphNodeTypeKernel) ++kernels_per_step;
  }
  CUDA_CHECK(cudaGraphInstantiate(&graph_exec, g, 0));
  CUDA_CHECK(cudaGraphDestroy(g));
}

// Amplitudes of the next todo steps ([step][source], as the caller has them)
// into the sources' tables, one copy per source; `staged` keeps the transposed
// rows until the stream has been waited for.
void Solver::upload_amplitudes(int32_t todo, const float* amp_in, std::vector<float>& staged) {
  if (n_sources == 0 || todo <= 0) return;
  const float* rows = amp_in;
  if (n_sources > 1) {
    staged.resize(static_cast<std::size_t>(n_sources) * todo);
    for (int32_t k = 0; k < todo; ++k)
      for (int32_t q = 0; q < n_sources; ++q)
        staged[static_cast<std::size_t>(q) * todo + k] = amp_in[static_cast<std::size_t>(k) * n_sources + q];
    rows = staged.data();
  }
  for (int32_t q = 0; q < n_sources; ++q)
    CUDA_CHECK(cudaMemcpyAsync(src_amp.get() + static_cast<std::size_t>(q) * n_amp + step + 1,
                               rows + static_cast<std::size_t>(q) * todo, todo * sizeof(float), cudaMemcpyHostToDevice,
                               stream));
}

// The samples recorded in the todo steps after `step`: consecutive rows of the
// trace buffer, one copy.
int32_t Solver::download_rows(int32_t todo, double* rows_out) {
  const int32_t first = step / record_every + 1, rows = (step + std::max(todo, 0)) / record_every + 1 - first;
  if (rows <= 0 || n_cols == 0) return 0;
  CUDA_CHECK(cudaMemcpyAsync(rows_out, trace_buf.get() + static_cast<std::size_t>(first) * n_cols,
                             static_cast<std::size_t>(rows) * n_cols * sizeof(double), cudaMemcpyDeviceToHost, stream));
  return rows;
}

// n steps with the caller's source amplitudes in and the recorded rows out.
// Copies go once per call: a copy per step of 4 bytes in and a row out (which
// waits for the stream when the caller's memory is pageable) cost 22 us a step
// of 81 at 30k order-6 elements.
void Solver::advance_streamed(int32_t n, const float* amp_in, double* rows_out, int32_t* n_rows) {
  INSEM_REQUIRE(!in_batch, INSEM_CUDA_ERR_STATE, "this solve is stepped by a batch");
  INSEM_REQUIRE(snap_every <= 0, INSEM_CUDA_ERR_STATE, "snapshots are recorded by advance(), not the streamed form");
  DeviceGuard dg(device);
  INSEM_REQUIRE(n >= 0 && n_rows, INSEM_CUDA_ERR_INVALID, "invalid streamed advance");
  INSEM_REQUIRE(n_sources == 0 || amp_in, INSEM_CUDA_ERR_INVALID, "missing source amplitudes");
  if (tiled) {
    advance_tiled(n, amp_in, rows_out, n_rows);
    return;
  }
  if (!initialized) initialize();
  ensure_graph();
  const int32_t todo = std::min<int32_t>(n, n_steps - step);
  CUDA_CHECK(cudaEventRecord(ev0, stream));
  std::vector<float> amp;
  upload_amplitudes(todo, amp_in, amp);
  for (int32_t k = 0; k < todo; ++k) CUDA_CHECK(cudaGraphLaunch(graph_exec, stream));
  const int32_t rows = rows_out ? download_rows(todo, rows_out) : 0;
  CUDA_CHECK(cudaEventRecord(ev1, stream));
  CUDA_CHECK(cudaStreamSynchronize(stream));
  step += todo;
  float ms = 0.0f;
  CUDA_CHECK(cudaEventElapsedTime(&ms, ev0, ev1));
  last_ms = ms;
  *n_rows = rows;
}

int32_t Solver::n_samples() const { return initialized ? step / record_every + 1 : 0; }

void Solver::copy_trace(int32_t t, double* out) {
  INSEM_REQUIRE(t >= 0 && t < static_cast<int32_t>(traces.size()), INSEM_CUDA_ERR_INVALID, "trace index out of range");
  const int32_t ns = n_samples();
  if (ns == 0) return;
  std::vector<double> buf(static_cast<std::size_t>(ns) * n_cols);
  CUDA_CHECK(cudaMemcpy(buf.data(), trace_buf.get(), buf.size() * sizeof(double), cudaMemcpyDeviceToHost));
  const TraceInfo& ti = traces[t];
  for (int32_t s = 0; s < ns; ++s)
    for (int32_t c = 0; c < ti.ncomp; ++c)
      out[static_cast<std::size_t>(s) * ti.ncomp + c] = buf[static_cast<std::size_t>(s) * n_cols + ti.first_col + c];
}

int32_t Solver::n_energy() const {
  if (!initialized || energy_every <= 0) return 0;
  return step / energy_every + 1;
}

namespace {
// Fields of a domain as the caller has them: [field][component][point] in the
// reference numbering, as doubles.  `perm` is null where the device keeps that
// numbering.  Block y: field and component.
struct StateFields {
  const float* f[3];
};
// Up to here one copy to the host, from where the three arrays are filled:
// a pageable copy costs some 7 us however small (65 KB: 62 -> 48 us; 400 KB: 93 -> 152).
constexpr std::size_t kStateOneCopy = std::size_t{1} << 17;
// Values renumbered at a time, and points whose numbering stays on the device
// between calls: 8 and 4 MB (a device without that much to spare is read by
// plain copies).
constexpr std::size_t kStateValues = std::size_t{1} << 20;
constexpr int32_t kStatePoints = 1 << 20;
__global__ void state_out_kernel(StateFields in, const int32_t* __restrict__ perm, int32_t ng, int32_t stride,
                                 int32_t ncomp, double* __restrict__ out) {
  const int32_t field = blockIdx.y / ncomp, c = blockIdx.y - field * ncomp;
  const float* x = in.f[field] + static_cast<size_t>(c) * stride;
  double* o = out + static_cast<size_t>(blockIdx.y) * ng;
  for (int32_t g = blockIdx.x * blockDim.x + threadIdx.x; g < ng; g += gridDim.x * blockDim.x)
    o[g] = static_cast<double>(x[perm ? perm[g] : g]);
}
}  // namespace

// The point numbering of a domain of at most kStatePoints points on the device,
// uploaded by the first state(); null without the memory for it.
const int32_t* Solver::state_numbering(int32_t di) {
  std::lock_guard<std::mutex> lk(perm_mutex);  // several threads may read one solve
  TiledDomain& t = tdom[di];
  if (t.device_perm.size() == 0) {
    try {
      t.device_perm.upload(t.perm);
    } catch (const Error& e) {
      if (e.code != INSEM_CUDA_ERR_NOMEM) throw;
    }
  }
  return t.device_perm.get();
}

void Solver::copy_state(int32_t di, double* u_out, double* v_out, double* a_out) {
  INSEM_REQUIRE(di >= 0 && di < static_cast<int32_t>(domains.size()), INSEM_CUDA_ERR_INVALID, "domain out of range");
  DeviceDomainData& d = domains[di];
  StateFields in{{d.u.get(), d.v.get(), d.a.get()}};
  const int32_t* host_perm = nullptr;
  int32_t stride = d.ng;
  if (tiled) {  // before the first step: the set state, a = 0
    TiledDomain& t = tdom[di];
    host_perm = t.perm.data();
    stride = t.ng;
    in = StateFields{{t.u_cur(parity), t.v.get(), t.a.get()}};
  }
  const std::size_t n = static_cast<std::size_t>(d.ncomp) * d.ng;
  if (n == 0) return;
  double* out[3] = {u_out, v_out, a_out};
  // renumbered and widened on the device (the host took 1.6 ns per value and
  // two more copies); the buffers are given back in the stream's order
  const std::size_t cap = std::min(3 * n, kStateValues);
  const bool send_perm = host_perm && d.ng > kStatePoints;
  double* buf = nullptr;
  int32_t* part = nullptr;
  cudaError_t err = cudaMallocAsync(reinterpret_cast<void**>(&buf), cap * sizeof(double), stream);
  if (err == cudaSuccess && send_perm)
    err = cudaMallocAsync(reinterpret_cast<void**>(&part), kStatePoints * sizeof(int32_t), stream);
  const int32_t* perm = err == cudaSuccess && host_perm && !send_perm ? state_numbering(di) : nullptr;
  if (err != cudaSuccess || (host_perm && !send_perm && !perm)) {
    // no device memory to spare: the fields as they are, renumbered on the host
    cudaGetLastError();
    if (buf) cudaFreeAsync(buf, stream);
    std::vector<float> h(static_cast<std::size_t>(d.ncomp) * stride);
    for (int k = 0; k < 3; ++k) {
      if (!out[k]) continue;
      CUDA_CHECK(cudaMemcpyAsync(h.data(), in.f[k], h.size() * sizeof(float), cudaMemcpyDeviceToHost, stream));
      CUDA_CHECK(cudaStreamSynchronize(stream));
      for (int c = 0; c < d.ncomp; ++c)
        for (int32_t g = 0; g < d.ng; ++g)
          out[k][static_cast<std::size_t>(c) * d.ng + g] = h[static_cast<std::size_t>(c) * stride + (host_perm ? host_perm[g] : g)];
    }
    return;
  }
  auto ok = [&](cudaError_t e) {
    if (err == cudaSuccess) err = e;
    return err == cudaSuccess;
  };
  std::vector<double> small(3 * n * sizeof(double) <= kStateOneCopy ? 3 * n : 0);
  auto renumber = [&](const StateFields& f, const int32_t* pm, int32_t points, int32_t rows, int32_t ncomp) {
    if (err != cudaSuccess) return;
    state_out_kernel<<<dim3(grid_for(points), rows), 256, 0, stream>>>(f, pm, points, stride, ncomp, buf);
    ok(cudaGetLastError());
  };
  auto fetch = [&](double* to, std::size_t from, std::size_t count) {
    if (err == cudaSuccess && to)
      ok(cudaMemcpyAsync(to, buf + from, count * sizeof(double), cudaMemcpyDeviceToHost, stream));
  };
  if (3 * n <= kStateValues) {  // all at once
    renumber(in, perm, d.ng, 3 * d.ncomp, d.ncomp);
    if (!small.empty()) fetch(small.data(), 0, 3 * n);
    else
      for (int k = 0; k < 3; ++k) fetch(out[k], k * n, n);
  } else if (n <= kStateValues && !send_perm) {  // field by field
    for (int k = 0; k < 3; ++k) {
      if (!out[k]) continue;
      renumber(StateFields{{in.f[k]}}, perm, d.ng, d.ncomp, d.ncomp);
      fetch(out[k], 0, n);
    }
  } else {  // by ranges of points
    const int32_t most = std::min<int32_t>(kStatePoints, static_cast<int32_t>(kStateValues));
    for (int32_t g = 0; g < d.ng && err == cudaSuccess; g += most) {
      const int32_t m = std::min(most, d.ng - g);
      if (send_perm) ok(cudaMemcpyAsync(part, host_perm + g, m * sizeof(int32_t), cudaMemcpyHostToDevice, stream));
      for (int k = 0; k < 3; ++k)
        for (int32_t c = 0; c < d.ncomp && out[k]; ++c) {
          const float* x = in.f[k] + static_cast<std::size_t>(c) * stride;
          renumber(StateFields{{host_perm ? x : x + g}}, send_perm ? part : perm ? perm + g : nullptr, m, 1, 1);
          fetch(out[k] + static_cast<std::size_t>(c) * d.ng + g, 0, m);
        }
    }
  }
  if (part) cudaFreeAsync(part, stream);
  cudaFreeAsync(buf, stream);
  const cudaError_t sync = cudaStreamSynchronize(stream);
  CUDA_CHECK(err);
  CUDA_CHECK(sync);
  if (!small.empty())
    for (int k = 0; k < 3; ++k)
      if (out[k]) std::copy_n(small.data() + k * n, n, out[k]);
}

// ------------------------------------------------------------ tiled path
constexpr int32_t kPaddedPoints = 1 << 22;  // most points of a domain in tiles of fewer than 32 elements

void Solver::build_tiled(const insem_cuda_problem& p) {
  const std::size_t npe = static_cast<std::size_t>(ngll) * ngll;
  set_constant_basis(ngll, host_vec(p.basis.D, npe), p.basis.Dj ? host_vec(p.basis.Dj, npe) : std::vector<float>{},
                     host_vec(p.basis.w2, npe));
  const auto fp = host_vec(p.coupling.fluid_points, n_cpl), sp = host_vec(p.coupling.solid_points, n_cpl);
  tdom.resize(domains.size());
  std::vector<int32_t> order[2];  // coupled points of the solid, of the fluid, in chunk order
  std::vector<int4> chunks = coupled_chunks(fp, sp, order[0], order[1]);
  for (std::size_t di = 0; di < domains.size(); ++di) {
    const insem_cuda_domain& d = p.domains[di];
    SpecialTerms terms;
    terms.sources = src_per_point[di];
    for (int32_t i = 0; i < n_cpl; ++i) {
      if (static_cast<int>(di) == fluid) terms.coupling[fp[i]].push_back(i);
      if (static_cast<int>(di) == solid) terms.coupling[sp[i]].push_back(i);
    }
    if (n_cpl > 0) terms.coupled = order[static_cast<int>(di) == solid ? 0 : 1];
    const auto ap = host_vec(d.absorbing_points, d.n_absorbing);
    for (int32_t i = 0; i < d.n_absorbing; ++i) terms.absorbing[ap[i]] = i;
    const uint8_t all = static_cast<uint8_t>((1u << d.ncomp) - 1u);
    for (int32_t g : host_vec(d.dirichlet_points, d.n_dirichlet)) terms.zero[g] |= all;
    const auto axc = host_vec(d.axis_components, d.n_axis_components);
    uint8_t axm = 0;
    for (int32_t c : axc) axm |= static_cast<uint8_t>(1u << c);
    if (axm)
      for (int32_t g : host_vec(d.axis_points, d.n_axis)) terms.zero[g] |= axm;
    for (int r = 0; r < p.n_receivers; ++r)
      if (p.receivers[r].domain == static_cast<int>(di))
        for (int32_t g : host_vec(p.receivers[r].points, p.receivers[r].n_points)) terms.receivers.push_back(g);
    // tile size by the domain's dominant element kind
    std::map<int, int64_t> per_kind;
    for (int b = 0; b < d.n_blocks; ++b) per_kind[d.blocks[b].kind] += d.blocks[b].n_elements;
    int kind = INSEM_RECT;
    int64_t most = -1;
    for (const auto& kv : per_kind)
      if (kv.second > most) {
        most = kv.second;
        kind = kv.first;
      }
    // A tile's data is laid out for 32 elements whatever it holds, so smaller
    // tiles, which only pay where elements are few, are not taken where their
    // padding would cost gigabytes.
    const int te = domains[di].ng > kPaddedPoints
                       ? kTileLanes
                       : choose_tile_elements(ngll, kind, d.medium == INSEM_ELASTIC,
                                              kind == INSEM_AXISYM ? d.azimuthal_order : 0, opts.tile_elements);
    tdom[di].build(d, ngll, te, terms,
                   host_vec(d.absorbing_coef, static_cast<std::size_t>(d.n_absorbing) * d.ncomp * d.ncomp));
  }
  if (n_cpl > 0) {
    std::vector<int32_t> f(n_cpl), s(n_cpl);
    for (int32_t i = 0; i < n_cpl; ++i) {
      f[i] = tdom[fluid].perm[fp[i]];
      s[i] = tdom[solid].perm[sp[i]];
    }
    const auto cx = host_vec(p.coupling.cx, n_cpl), cz = host_vec(p.coupling.cz, n_cpl);
    tdom[solid].set_partners(f, cx, cz);
    tdom[fluid].set_partners(s, cx, cz);
  }
  // the chunks' ranges count from the first coupled halo point
  n_chunks = static_cast<int32_t>(chunks.size());
  for (int k = 0; k < 2; ++k) {
    const int di = k == 0 ? solid : fluid;
    n_free_halo[k] = di < 0 ? 0 : tdom[di].n_halo - static_cast<int32_t>(order[k].size());
  }
  for (int4& c : chunks) {
    c.x += n_free_halo[0];
    c.y += n_free_halo[0];
    c.z += n_free_halo[1];
    c.w += n_free_halo[1];
  }
  tchunks.upload(chunks);
  std::vector<int32_t> rp;
  for (int r = 0; r < p.n_receivers; ++r)
    for (int32_t g : host_vec(p.receivers[r].points, p.receivers[r].n_points))
      rp.push_back(tdom[p.receivers[r].domain].perm[g]);
  trec_points.upload(rp.empty() ? std::vector<int32_t>{0} : rp);
  int base = 0;
  for (std::size_t di = 0; di < tdom.size(); ++di) {
    ep_tile[di] = base;
    ep_ntile[di] = tdom[di].n_tiles;
    base += tdom[di].n_tiles;
    ep_halo[di] = base;
    ep_nhalo[di] = ceil_div(n_free_halo[static_cast<int>(di) == solid ? 0 : 1], kHaloChunk) + n_chunks;
    base += ep_nhalo[di];
  }
  epart.resize(2 * static_cast<std::size_t>(std::max(base, 1)));
  epart.zero();
  tiled = true;
}

// The coupled points in chunks of at most kHaloChunk per side.  A chunk holds
// whole groups (points joined by interface entries), so that the fluid's
// partners are finished by the same CTA.  Returns ranges into the orders;
// nothing if a group is larger than a chunk.
std::vector<int4> Solver::coupled_chunks(const std::vector<int32_t>& fp, const std::vector<int32_t>& sp,
                                         std::vector<int32_t>& solid_order, std::vector<int32_t>& fluid_order) const {
  std::vector<int4> chunks;
  if (n_cpl == 0) return chunks;
  std::map<int32_t, std::vector<int32_t>> of_solid, of_fluid;  // point -> entries
  for (int32_t i = 0; i < n_cpl; ++i) {
    of_solid[sp[i]].push_back(i);
    of_fluid[fp[i]].push_back(i);
  }
  std::vector<char> seen(n_cpl, 0);
  std::set<int32_t> s_done, f_done;
  int4 c{0, 0, 0, 0};
  for (int32_t i0 = 0; i0 < n_cpl; ++i0) {
    if (seen[i0]) continue;
    // the group of entry i0, breadth first
    std::vector<int32_t> entries{i0}, gs, gf;
    seen[i0] = 1;
    for (std::size_t q = 0; q < entries.size(); ++q) {
      const int32_t i = entries[q];
      if (s_done.insert(sp[i]).second) gs.push_back(sp[i]);
      if (f_done.insert(fp[i]).second) gf.push_back(fp[i]);
      for (const auto* next : {&of_solid[sp[i]], &of_fluid[fp[i]]})
        for (int32_t j : *next)
          if (!seen[j]) {
            seen[j] = 1;
            entries.push_back(j);
          }
    }
    const int32_t ns = static_cast<int32_t>(gs.size()), nf = static_cast<int32_t>(gf.size());
    if (ns > kHaloChunk || nf > kHaloChunk) {
      solid_order.clear();
      fluid_order.clear();
      return {};
    }
    if (c.y - c.x + ns > kHaloChunk || c.w - c.z + nf > kHaloChunk) {
      chunks.push_back(c);
      c = int4{c.y, c.y, c.w, c.w};
    }
    solid_order.insert(solid_order.end(), gs.begin(), gs.end());
    fluid_order.insert(fluid_order.end(), gf.begin(), gf.end());
    c.y += ns;
    c.w += nf;
  }
  chunks.push_back(c);
  return chunks;
}

// Arguments of the solve's halo kernel on the field buffers of `par`.
HaloArgs Solver::halo_args(int par, bool init) {
  HaloArgs A{};
  if (solid >= 0) {
    A.s_td = tdom[solid].view(par);
    A.s_hd = tdom[solid].halo_view();
    A.nb_s = ceil_div(n_free_halo[0], kHaloChunk);
    A.ep_s = ep_halo[solid];
    A.s_hd.n = n_free_halo[0];
  }
  if (fluid >= 0) {
    A.f_td = tdom[fluid].view(par);
    A.f_hd = tdom[fluid].halo_view();
    A.nb_f = ceil_div(n_free_halo[1], kHaloChunk);
    A.ep_f = ep_halo[fluid];
    A.f_hd.n = n_free_halo[1];
  }
  A.n_chunk = n_chunks;
  A.chunks = tchunks.get();
  A.amp = src_amp.get();
  A.n_amp = n_amp;
  A.sc = StepScalars{static_cast<float>(dt), static_cast<float>(0.5 * dt), static_cast<float>(0.5 * dt * dt),
                     energy_every};
  A.h_damp = init ? 0.0 : 0.5 * dt;
  A.st = st;
  A.epartial = epart.get();
  return A;
}

AllFields Solver::tiled_fields(int par) {
  AllFields f{};
  for (std::size_t i = 0; i < tdom.size() && i < 2; ++i)
    f.d[i] = {tdom[i].u_cur(par), tdom[i].vn.get(), tdom[i].a.get(), tdom[i].ng};
  return f;
}

// n steps of the tiled path from the field buffers of `par` on (init: step 0,
// explicit damping, no step count), as one chain of launches on the stream
// (see DepMode).  A step's critical path is tiles -> halo points.  The fluid's
// tiles run beside the solid's, and a step's receivers beside the next step's
// tiles: they read halo points only, which the next step's halo kernels
// overwrite, not its tiles.  The first kernel of a sequence keeps a full
// boundary to what is ahead of it.
void Solver::enqueue_tiled(int par0, bool init, int n) {
  const StepScalars sc{static_cast<float>(dt), static_cast<float>(0.5 * dt), static_cast<float>(0.5 * dt * dt),
                       energy_every};
  ReceiversDev rv = receivers_view();
  rv.points = trec_points.get();
  auto observe = [&](int k, bool beside) {
    // particle velocity, then the recorded columns (which read it)
    StepIdx ix{k, init ? 1 : 0, beside ? kDepLate : kDepAll};
    const AllFields f = tiled_fields(par0 ^ (k & 1));
    if (n_acoustic_rec > 0) {
      CUDA_CHECK(launch_chained(particle_velocity_kernel, ceil_div(n_acoustic_rec, kRecChunk), kRecThreads, 0, stream,
                                true, rv, f, rec_acoustic.get(), n_acoustic_rec, dt, init ? 1 : 0, ix));
      ix.dep = kDepAll;
    }
    if (n_cols > 0)
      CUDA_CHECK(launch_chained(record_kernel, ceil_div(n_cols, kRecChunk), kRecThreads, 0, stream, true, rv, f,
                                rec_cols.get(), n_cols, st, record_every, trace_buf.get(), max_samples, ix));
  };
  for (int k = 0; k < n; ++k) {
    const int par = par0 ^ (k & 1);
    bool first = true;
    for (int di : {solid, fluid}) {
      if (di < 0) continue;
      TiledDomain& t = tdom[di];
      for (std::size_t b = 0; b < t.blocks.size(); ++b) {
        if (t.blocks[b].ntiles == 0) continue;
        TileLaunch a;
        a.dom = &t;
        a.block = static_cast<int>(b);
        a.parity = par;
        a.sc = sc;
        a.st = st;
        a.epartial = epart.get() + 2 * static_cast<std::size_t>(ep_tile[di]);
        a.elastic = t.medium == INSEM_ELASTIC;
        a.ix = StepIdx{k, init ? 1 : 0, first ? kDepFirst : kDepLate};
        a.overlap = !first || k > 0;
        a.stream = stream;
        launch_tiles(ngll, a);
        first = false;
      }
    }
    if (k > 0) observe(k - 1, true);
    const HaloArgs A = halo_args(par, init);
    const StepIdx ix{k, init ? 1 : 0, kDepAll};
    auto halo = [&](const HaloArgs& h) {
      const int grid = h.nb_s + h.nb_f + h.n_chunk;
      if (grid == 0) return;
      auto kernel = solid < 0 ? halo_step_kernel<0> : tdom[solid].ncomp == 2 ? halo_step_kernel<2> : halo_step_kernel<3>;
      CUDA_CHECK(launch_chained(kernel, grid, kHaloChunk, 0, stream, true, h, ix));
    };
    if (n_cpl > 0 && n_chunks == 0) {  // a coupled group larger than a CTA: the solid's points, then the fluid's
      HaloArgs one = A;
      one.nb_f = 0;
      halo(one);
      one = A;
      one.nb_s = 0;
      halo(one);
    } else {
      halo(A);
    }
    if (energy_every > 0) {
      // potential order: elastic first
      const int d0 = solid >= 0 ? solid : fluid;
      const int d1 = solid >= 0 ? fluid : -1;
      const int n_dom = d1 >= 0 ? 2 : 1;
      int4 s0{ep_tile[d0], ep_ntile[d0], ep_halo[d0], ep_nhalo[d0]};
      int4 s1{0, 0, 0, 0};
      if (d1 >= 0) s1 = int4{ep_tile[d1], ep_ntile[d1], ep_halo[d1], ep_nhalo[d1]};
      CUDA_CHECK(launch_chained(tiled_energy_kernel, 1, kReduceThreads, 0, stream, true, epart.get(), n_dom, s0, s1, st,
                                energy_every, dt, energy.get(), static_cast<int32_t>(energy.size() / 3),
                                StepIdx{k, init ? 1 : 0, kDepAll}));
    }
  }
  observe(n - 1, false);
  if (!init) CUDA_CHECK(launch_chained(advance_step_kernel, 1, 1, 0, stream, true, st, n));
}

// The state becomes that of a span of steps up to last_step.
void Solver::tiled_begin_steps(int32_t last_step) {
  SpanField f[2] = {};
  int64_t total = 0;
  for (std::size_t i = 0; complete && i < tdom.size() && i < 2; ++i) {
    TiledDomain& t = tdom[i];
    f[i] = SpanField{t.u_cur(parity), t.v.get(), t.a.get(), static_cast<int64_t>(t.ncomp) * t.ng};
    total += f[i].n;
  }
  begin_span_kernel<<<grid_for(total), 256, 0, stream>>>(f[0], f[1], static_cast<float>(dt), static_cast<float>(0.5 * dt),
                                                         static_cast<float>(0.5 * dt * dt), st, last_step, parity);
  CUDA_LAUNCH_CHECK();
  complete = false;
}

// The graph of n steps from the buffers of `par` on, captured at first use.
cudaGraphExec_t Solver::tiled_graph(int par, int n) {
  const auto it = tgraph.find({par, n});
  if (it != tgraph.end()) return it->second;
  cudaGraph_t g = nullptr;
  CUDA_CHECK(cudaStreamBeginCapture(stream, cudaStreamCaptureModeThreadLocal));
  try {
    enqueue_tiled(par, false, n);
  } catch (...) {
    cudaStreamEndCapture(stream, &g);
    if (g) cudaGraphDestroy(g);
    throw;
  }
  CUDA_CHECK(cudaStreamEndCapture(stream, &g));
  if (kernels_per_step == 0) {
    std::size_t nn = 0;
    CUDA_CHECK(cudaGraphGetNodes(g, nullptr, &nn));
    kernels_per_step = static_cast<int32_t>(nn - 1) / n;  // kernel nodes only; the last closes the sequence
  }
  cudaGraphExec_t ge = nullptr;
  const cudaError_t e = cudaGraphInstantiate(&ge, g, 0);
  cudaGraphDestroy(g);
  CUDA_CHECK(e);
  tgraph[{par, n}] = ge;
  return ge;
}

// The initial step (accelerations and observers at t = 0).
void Solver::tiled_initialize() {
  if (initialized) return;
  enqueue_tiled(parity, true, 1);
  parity ^= 1;
  complete = true;
  initialized = true;
}

// advance(n) on the tiled path; with amp_in or rows_out, the streamed variant:
// the steps' amplitudes copied in ahead of the first, their recorded rows out
// after the last.
void Solver::advance_tiled(int32_t n, const float* amp_in, double* rows_out, int32_t* n_rows) {
  const bool streamed = rows_out != nullptr || amp_in != nullptr;
  CUDA_CHECK(cudaEventRecord(ev0, stream));
  tiled_initialize();
  const int32_t todo = std::min<int32_t>(n, n_steps - step);
  int32_t rows = 0;
  if (todo > 0) tiled_begin_steps(step + todo);
  std::vector<float> amp;  // read by the copies until the stream is waited for below
  if (amp_in) upload_amplitudes(todo, amp_in, amp);
  for (int32_t k = 0; k < todo;) {
    // Sequences of 16 steps for long spans, of 4, then single steps: every
    // boundary between graphs costs the overlap of one step with the next and
    // a launch, and every further sequence length a capture on its first use
    // (so the longest only where it is replayed several times).
    const int32_t left = todo - k;
    const int32_t c = (left >= 16 && todo >= 64) ? 16 : left >= 4 ? 4 : 1;
    if (opts.use_graphs) CUDA_CHECK(cudaGraphLaunch(tiled_graph(parity, c), stream));
    else enqueue_tiled(parity, false, c);
    if (c & 1) parity ^= 1;
    k += c;
  }
  if (rows_out) rows = download_rows(todo, rows_out);
  if (todo > 0) complete = true;
  step += todo;
  CUDA_CHECK(cudaEventRecord(ev1, stream));
  if (opts.check_finite && !streamed) enqueue_finite_check();
  StepState hs;
  CUDA_CHECK(cudaMemcpyAsync(&hs, st, sizeof(hs), cudaMemcpyDeviceToHost, stream));
  CUDA_CHECK(cudaStreamSynchronize(stream));
  float ms = 0.0f;
  CUDA_CHECK(cudaEventElapsedTime(&ms, ev0, ev1));
  last_ms = ms;
  *n_rows = rows;
  INSEM_REQUIRE(!hs.error, INSEM_CUDA_ERR_TIMEOUT, "a tile's bulk copies did not arrive within the wait limit");
  if (hs.nonfinite) nonfinite_seen = true;
  if (opts.check_finite && !streamed)
    INSEM_REQUIRE(!hs.nonfinite, INSEM_CUDA_ERR_NONFINITE, "the solution contains NaN or Inf (unstable time step?)");
}

void Solver::enqueue_finite_check() {
  const float* x[2] = {};
  int64_t n[2] = {};
  for (std::size_t i = 0; i < tdom.size() && i < 2; ++i) {
    x[i] = tdom[i].u_cur(parity);
    n[i] = static_cast<int64_t>(tdom[i].ncomp) * tdom[i].ng;
  }
  finite_check_kernel<<<grid_for(n[0] + n[1]), 256, 0, stream>>>(x[0], n[0], x[1], n[1], st);
  CUDA_LAUNCH_CHECK();
}

}  // namespace insem_b200

using namespace insem_b200;

extern "C" {

int insem_cuda_solver_create(const insem_cuda_problem* problem, const insem_cuda_options* options,
                             insem_cuda_solver** out) {
  return guarded([&] {
    INSEM_REQUIRE(problem && out, INSEM_CUDA_ERR_INVALID, "null argument");
    auto h = std::make_unique<insem_cuda_solver>();
    h->s = std::make_unique<Solver>(*problem, options);
    *out = h.release();
  });
}

int insem_cuda_solver_create_timed(const insem_cuda_problem* problem, const insem_cuda_time* time,
                                   const insem_cuda_options* options, insem_cuda_solver** out) {
  return guarded([&] {
    INSEM_REQUIRE(problem && time && out, INSEM_CUDA_ERR_INVALID, "null argument");
    auto h = std::make_unique<insem_cuda_solver>();
    h->s = std::make_unique<Solver>(*problem, options, false, time);
    *out = h.release();
  });
}

double insem_cuda_solver_stable_dt(const insem_cuda_solver* h) { return h ? h->s->stable_dt_estimate : 0.0; }

void insem_cuda_solver_destroy(insem_cuda_solver* h) { delete h; }

int insem_cuda_solver_set_state(insem_cuda_solver* h, int32_t medium, const double* u, const double* v) {
  return guarded([&] {
    INSEM_REQUIRE(h, INSEM_CUDA_ERR_INVALID, "null handle");
    DeviceGuard dg(h->s->device);
    h->s->set_state(medium, u, v);
  });
}

int insem_cuda_solver_advance(insem_cuda_solver* h, int32_t n) {
  return guarded([&] {
    INSEM_REQUIRE(h, INSEM_CUDA_ERR_INVALID, "null handle");
    h->s->advance(n);
  });
}

int insem_cuda_solver_run(insem_cuda_solver* h) {
  return guarded([&] {
    INSEM_REQUIRE(h, INSEM_CUDA_ERR_INVALID, "null handle");
    h->s->advance(h->s->n_steps - h->s->step);
  });
}

int32_t insem_cuda_solver_step(const insem_cuda_solver* h) { return h ? h->s->step : -1; }
int32_t insem_cuda_solver_status(const insem_cuda_solver* h) {
  if (!h) return INSEM_CUDA_ERR_INVALID;
  return h->s->nonfinite_seen ? INSEM_CUDA_ERR_NONFINITE : INSEM_CUDA_OK;
}
int32_t insem_cuda_solver_n_steps(const insem_cuda_solver* h) { return h ? h->s->n_steps : -1; }
double insem_cuda_solver_dt(const insem_cuda_solver* h) { return h ? h->s->dt : 0.0; }
int32_t insem_cuda_solver_n_samples(const insem_cuda_solver* h) { return h ? h->s->n_samples() : -1; }
int32_t insem_cuda_solver_n_traces(const insem_cuda_solver* h) {
  return h ? static_cast<int32_t>(h->s->traces.size()) : -1;
}
int32_t insem_cuda_solver_trace_ncomp(const insem_cuda_solver* h, int32_t t) {
  if (!h || t < 0 || t >= static_cast<int32_t>(h->s->traces.size())) return -1;
  return h->s->traces[t].ncomp;
}

int insem_cuda_solver_trace(insem_cuda_solver* h, int32_t trace, double* out) {
  return guarded([&] {
    INSEM_REQUIRE(h && out, INSEM_CUDA_ERR_INVALID, "null argument");
    DeviceGuard dg(h->s->device);
    h->s->copy_trace(trace, out);
  });
}

int insem_cuda_solver_times(insem_cuda_solver* h, double* out) {
  return guarded([&] {
    INSEM_REQUIRE(h && out, INSEM_CUDA_ERR_INVALID, "null argument");
    const int32_t ns = h->s->n_samples();
    for (int32_t s = 0; s < ns; ++s) out[s] = static_cast<double>(s * h->s->record_every) * h->s->dt;
  });
}

int insem_cuda_solver_energy(insem_cuda_solver* h, double* out, int32_t capacity, int32_t* n_out) {
  return guarded([&] {
    INSEM_REQUIRE(h && n_out, INSEM_CUDA_ERR_INVALID, "null argument");
    DeviceGuard dg(h->s->device);
    const int32_t n = h->s->n_energy();
    *n_out = n;
    if (!out || n == 0) return;
    INSEM_REQUIRE(capacity >= n, INSEM_CUDA_ERR_INVALID, "energy buffer too small");
    CUDA_CHECK(cudaMemcpy(out, h->s->energy.get(), static_cast<std::size_t>(n) * 3 * sizeof(double),
                          cudaMemcpyDeviceToHost));
  });
}

int insem_cuda_solver_state(insem_cuda_solver* h, int32_t domain, double* u, double* v, double* a) {
  return guarded([&] {
    INSEM_REQUIRE(h, INSEM_CUDA_ERR_INVALID, "null handle");
    DeviceGuard dg(h->s->device);
    h->s->copy_state(domain, u, v, a);
  });
}

double insem_cuda_solver_last_advance_ms(const insem_cuda_solver* h) { return h ? h->s->last_ms : 0.0; }

int insem_cuda_solver_internal_forces(insem_cuda_solver* h, int32_t domain, const float* u, float* f) {
  return guarded([&] {
    INSEM_REQUIRE(h && u && f, INSEM_CUDA_ERR_INVALID, "null argument");
    Solver& s = *h->s;
    DeviceGuard dg(s.device);
    INSEM_REQUIRE(domain >= 0 && domain < static_cast<int32_t>(s.domains.size()), INSEM_CUDA_ERR_INVALID,
                  "domain out of range");
    auto& d = s.domains[domain];
    const std::size_t n = static_cast<std::size_t>(d.ncomp) * d.ng;
    DeviceBuffer<float> du, df(n);
    du.upload(u, n);
    s.internal_forces(d, du.get(), df.get());
    CUDA_CHECK(cudaStreamSynchronize(s.stream));
    CUDA_CHECK(cudaMemcpy(f, df.get(), n * sizeof(float), cudaMemcpyDeviceToHost));
  });
}

int insem_cuda_set_tile_elements(int32_t ngll, int32_t kind, int32_t medium, int32_t azimuthal_order,
                                 int32_t tile_elements) {
  return guarded([&] {
    INSEM_REQUIRE(kind >= INSEM_RECT && kind <= INSEM_AXISYM, INSEM_CUDA_ERR_INVALID, "unknown geometry kind");
    INSEM_REQUIRE(azimuthal_order == 0 || (azimuthal_order == 1 && kind == INSEM_AXISYM), INSEM_CUDA_ERR_INVALID,
                  "azimuthal order 1 needs the axisymmetric kind");
    set_tile_elements(ngll, kind, medium == INSEM_ELASTIC, azimuthal_order, tile_elements);
  });
}

int32_t insem_cuda_tile_elements(int32_t ngll, int32_t kind, int32_t medium, int32_t azimuthal_order, int32_t) {
  int32_t out = 0;
  guarded([&] {
    out = choose_tile_elements(ngll, kind, medium == INSEM_ELASTIC, kind == INSEM_AXISYM ? azimuthal_order : 0, 0);
  });
  return out;
}

int32_t insem_cuda_solver_tile_elements(const insem_cuda_solver* h, int32_t domain) {
  if (!h || !h->s->tiled || domain < 0 || domain >= static_cast<int32_t>(h->s->domains.size())) return 0;
  return h->s->tiled_tile_elements(domain);
}

int insem_cuda_solver_point_classes(const insem_cuda_solver* h, int32_t domain, int32_t* n_tile_points,
                                    int32_t* n_halo_points) {
  return guarded([&] {
    INSEM_REQUIRE(h, INSEM_CUDA_ERR_INVALID, "null handle");
    const Solver& s = *h->s;
    INSEM_REQUIRE(domain >= 0 && domain < static_cast<int32_t>(s.domains.size()), INSEM_CUDA_ERR_INVALID,
                  "domain out of range");
    int32_t nt = 0, nh = 0;
    if (s.tiled) {
      nh = s.tiled_halo_points(domain);
      nt = s.domains[domain].ng - nh;
    } else {
      nh = s.domains[domain].ng;
    }
    if (n_tile_points) *n_tile_points = nt;
    if (n_halo_points) *n_halo_points = nh;
  });
}

int insem_cuda_solver_advance_streamed(insem_cuda_solver* h, int32_t n, const float* amp_in, double* rows_out,
                                       int32_t* n_rows) {
  return guarded([&] {
    INSEM_REQUIRE(h, INSEM_CUDA_ERR_INVALID, "null handle");
    h->s->advance_streamed(n, amp_in, rows_out, n_rows);
  });
}

int32_t insem_cuda_solver_n_columns(const insem_cuda_solver* h) { return h ? h->s->n_columns() : -1; }

int32_t insem_cuda_solver_kernels_per_step(insem_cuda_solver* h) {
  if (!h) return -1;
  if (h->s->tiled) return h->s->kernels_per_step;  // counted when the step graphs are captured
  const int rc = guarded([&] {
    DeviceGuard dg(h->s->device);
    h->s->ensure_graph();
  });
  return rc == INSEM_CUDA_OK ? h->s->kernels_per_step : -1;
}

int insem_cuda_stable_dt(const insem_cuda_problem* problem, int32_t device, double* stable_dt) {
  return guarded([&] {
    INSEM_REQUIRE(problem && stable_dt, INSEM_CUDA_ERR_INVALID, "null argument");
    insem_cuda_options o{};
    o.device = device;
    o.use_graphs = 0;
    Solver s(*problem, &o, true);
    *stable_dt = s.stable_dt();
  });
}

}  // extern "C"
