// Batched solves: many independent solves (models, shots) of any ngll,
// geometry kind, medium and azimuthal order advance together, one step of
// every unfinished solve per batched step.
//
// A batched step is a fixed number of launches whatever the number of solves,
// replayed from CUDA graphs of kSequence steps or of one:
//   one tile launch per tile class (ngll, kind, medium, order): one CTA
//     per (segment, tile) item
//   halo points of every solve, by the solid's component count
//   receivers (particle velocity, then recording) and energy of every solve
//   step counters and buffer parities (once per sequence)
// The launches form one chain in which a launch may start before the one
// ahead of it has ended (DepMode in common.cuh): the tile classes fill
// the chip one behind the other without waiting for each other's last tiles.
// Each solve keeps its own device data, time step, parity and step count,
// so its results are the ones it gets alone, bit for bit.  Solves that
// reach their last step run it in final mode and idle (every batched kernel
// skips them) until the tables are rebuilt without them: membership changes
// re-capture the graphs at the next advance.
#pragma once

#include <map>
#include <memory>
#include <vector>

#include "solver.cuh"

namespace insem_b200 {

// Streamed batched steps: where each solve's amplitudes and sample columns sit
// in a step's host row.
struct StreamSeg {
  float* src_amp;        // [n_sources][n_amp] amplitude table of the solve
  int32_t n_amp, n_sources, amp_off;
  const double* traces;  // [max_samples][n_cols]
  int32_t n_cols, col_off, record_every, max_samples;
  const StepState* st;
};

struct TileClass {
  int ngll = 0, kind = 0, m = 0, ncomp = 0;
  bool elastic = false, any_axial = false;
  int tp_cap = 0, nc_cap = 0, rank_cap = 1;  // largest tile of the class
  std::vector<TileSeg> segs;
  std::vector<TileItem> items;
};

constexpr int kHaloClasses = 5;

// Host-side segment tables of one batch composition.
struct BatchTables {
  std::map<int, TileClass> tiles;  // key: ((ngll * 8 + kind) * 2 + elastic) * 2 + m
  // solves without a solid, with a solid of 2 and of 3 components; the fluids
  // of solves whose halo points take two launches
  std::vector<HaloArgs> halo_segs[kHaloClasses];
  std::vector<int2> halo_items[kHaloClasses];
  std::vector<RecSeg> rec_segs;
  std::vector<int2> pv_items, rec_items;
  std::vector<EnergySeg> energy_segs;
  std::vector<StepState*> states;
  std::vector<StreamSeg> stream_segs;
  int32_t amp_cols = 0, row_cols = 0;
};

class Batch {
 public:
  explicit Batch(const insem_cuda_options* opt);
  ~Batch();
  Batch(const Batch&) = delete;
  Batch& operator=(const Batch&) = delete;

  // Builds a solve on the batch's device; returns its index.
  int32_t add(const insem_cuda_problem& p);
  // Takes ownership of an existing solve that no batch has stepped.
  int32_t adopt(insem_cuda_solver* h);
  // n batched steps; a solve with fewer steps left idles after its last one.
  void advance(int32_t n);
  // Steps until every solve is complete.
  void run();
  // n steps (fewer if every solve ends sooner) with amplitudes in and sample
  // rows out, one copy each way per sequence of steps (kSequence, else 1):
  // amp_in[step][amp_cols] are the active solves' source amplitudes (in index
  // order, each solve's sources in order), rows_out[step][row_cols] their
  // latest sample rows.  Returns the steps done.
  int32_t advance_streamed(int32_t n, const float* amp_in, double* rows_out);
  // Column counts of the streamed rows for the current composition.
  void stream_layout(int32_t* amp_cols, int32_t* row_cols);
  // n steps with plain launches and CUDA events around the tile launches of
  // every step: device ms of the tile launches and of the whole steps.
  void profile(int32_t n, double* tile_ms, double* step_ms);
  // Frees a solve (its index stays unused).
  void remove(int32_t index);
  insem_cuda_solver* member(int32_t index);
  int32_t size() const { return static_cast<int32_t>(members.size()); }
  int32_t active() const;
  int32_t steps_to_next_completion() const;
  int32_t max_remaining() const;  // steps until every member is complete

  insem_cuda_options opts{};
  double last_ms = 0.0;           // device time of the last advance()
  int32_t kernels_per_step = 0;   // launches of a step
  int64_t point_updates = 0;      // sum of points x steps of the last advance()

 private:
  void rebuild();
  void finish_steps();       // error flags of the steps just enqueued; waits for them
  void credit(int32_t k);    // host bookkeeping after k batched steps
  void enqueue(int32_t n, cudaEvent_t tiles_begin = nullptr, cudaEvent_t tiles_end = nullptr);
  template <class Fn>
  void enqueue_step(int32_t k, cudaEvent_t tiles_begin, cudaEvent_t tiles_end, Fn&& after_tiles);
  void launch_steps(int32_t n);
  void drop_graphs();
  // Steps per captured sequence, besides single steps: inside a sequence the
  // receivers leave the critical path and streamed copies are shared.
  static constexpr int32_t kSequence = 8;
  static int32_t sequence(int32_t left);

  struct DevClass {
    int ngll = 0, kind = 0, m = 0, ncomp = 1;
    bool elastic = false;
    DeviceBuffer<TileSeg> segs;
    DeviceBuffer<TileItem> items;
    int32_t n_items = 0;
    double work = 0.0;  // elements x points per element x components
    TileLayout L{};
    uint32_t smem = 0;
    int grid = 0;
  };

  cudaStream_t stream = nullptr;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  std::vector<std::unique_ptr<insem_cuda_solver>> members;  // null after remove()
  std::vector<char> prepared;
  bool dirty = true;
  cudaGraphExec_t graph[2] = {nullptr, nullptr};  // one step, kSequence steps
  // device tables of the current composition
  std::vector<DevClass> dclasses;
  DeviceBuffer<HaloArgs> dhalo_segs[kHaloClasses];
  DeviceBuffer<int2> dhalo_items[kHaloClasses];
  int32_t n_halo_items[kHaloClasses] = {};
  DeviceBuffer<RecSeg> drec_segs;
  DeviceBuffer<int2> dpv_items, drec_items;
  int32_t n_pv_items = 0, n_rec_items = 0;
  DeviceBuffer<EnergySeg> denergy;
  int32_t n_energy = 0;
  DeviceBuffer<StepState*> dstates;
  int32_t n_states = 0;
  DeviceBuffer<StreamSeg> dstream;
  int32_t n_stream = 0, amp_cols = 0, row_cols = 0;
  DeviceBuffer<float> amp_stage;
  DeviceBuffer<double> row_stage;
  DeviceBuffer<int32_t> stream_from;  // step counts at the start of the streamed steps in flight
  DeviceBuffer<int32_t> derr;
  int32_t* herr = nullptr;  // pinned
  std::vector<int64_t> member_points;
};

}  // namespace insem_b200
