// ls_solver.h -- device solver behind the C ABI: owns the device copy of the
// patch layout, the step state, the stream and the FIM-iteration graphs.
#pragma once
#include <cuda_runtime.h>

#include <string>
#include <vector>

#include "ls_device.cuh"
#include "ls_layout.h"
#include "ls_mlp.h"

namespace lsgb {

struct Launch {
  int sms;
  int fim_grid, fim_block, fim_smem;
  int fim_ctas;    // resident CTAs of the sweep kernel per SM
  int pair_block;  // threads of the two-copies-per-thread sweep kernel (0: not used)
  int persist_grid;  // CTAs of the persistent FIM kernel (all resident; 0: no persistent form here)
  int upd_grid, upd_block, upd_smem;
  int seed_grid, seed_smem;
  int warp_grid;
  int flat_grid;
};

enum { LEARN_NB_VERTICES = 0, LEARN_WARM, LEARN_SEED_WARM, LEARN_SUPPORT, LEARN_MOVED, LEARN_TARGETS };

// One build of the step kernels (fast or bit-exact).
struct KernelSet {
  cudaError_t (*configure)(const DevMesh& m, const StepParams& sp, Launch& L);
  // step control words; restart: again within a step (the previous narrowband's size is kept)
  cudaError_t (*begin)(const DevState& s, int restart, cudaStream_t st);
  cudaError_t (*seed)(const DevMesh& m, const DevState& s, const StepParams& sp, const Launch& L, cudaStream_t st);
  // one FIM iteration, the off-th of a loop body
  cudaError_t (*fim)(const DevMesh& m, const DevState& s, const StepParams& sp, int off, const Launch& L,
                     cudaStream_t st);
  // every FIM iteration of a step in one cooperative launch (L.persist_grid > 0)
  cudaError_t (*fim_persistent)(const DevMesh& m, const DevState& s, const StepParams& sp, const Launch& L,
                                cudaStream_t st);
  cudaError_t (*narrowband)(const DevMesh& m, const DevState& s, const StepParams& sp, const Launch& L,
                            cudaStream_t st);
  cudaError_t (*update)(const DevMesh& m, const DevState& s, const StepParams& sp, int first, const Launch& L,
                        cudaStream_t st);
  // FIM distances in the layout's vertex order
  cudaError_t (*distances)(const DevMesh& m, const DevState& s, const StepParams& sp, float* out, const Launch& L,
                           cudaStream_t st);
  // n vertices from `first` on in the caller's order (ctl: only if the step was done)
  cudaError_t (*unpermute)(const DevMesh& m, const float* phi, int first, int n, float* out, const int* ctl,
                           const Launch& L, cudaStream_t st);
  cudaError_t (*permute)(const DevMesh& m, const float* in, float* out, const Launch& L, cudaStream_t st);
  // learned warm start / collection kernels (op: LEARN_*)
  cudaError_t (*learn)(int op, const DevMesh& m, const DevState& s, const StepParams& sp, const DevLearn& lr, int arg,
                       float fa, const Launch& L, cudaStream_t st);
  // per-copy geometry records of the two-copies-per-thread sweep (written
  // when L.pair_block > 0; gm: 3 float4 per copy, gh: 1)
  cudaError_t (*geometry)(const DevMesh& m, float4* gm, float4* gh, const Launch& L, cudaStream_t st);
};
const KernelSet& kernels_fast();
const KernelSet& kernels_exact();

struct SolverConfig {
  int update_kind = 0;
  int ref_compat = 0;
  int fp64_flagged = 0;
  int bit_exact = 0;
  int profile = 0;
  int use_graph = 1;
  int niter = 0;
  int inside_niter = 1;
  int max_fim_iters = 100000;
  int graph_chunk = 4;
  int fim_ctas = 0;  // FIM setting (ls_params::fim_ctas_per_sm); 0: chosen by the mesh
  double dt = 1.0;
  double bandwidth = 16.0;
  double curv_coeff = 1.0;
  double smallnum = 1e-5;
  double largenum = 1e9;
  double length_scale = 0.0;
  double fp64_tau = 3.814697265625e-06;  // 2^-18
  int host_staging = 0;  // 1: host arrays go through pinned staging even where the GPU can read pageable memory
  int persistent = 0;    // 1: a step's FIM loop runs as one cooperative launch where the kernel has that form
  int spin_limit = 1 << 22;  // polls of one grid-barrier wait of the persistent kernel (< 0: every FIM
                             // kernel wait gives up at its first check)
  // batches (Layout::patch_mesh set): per-mesh dt, bandwidth, curvature
  // coefficient and FIM length scale (<= 0: the mesh's mean edge)
  std::vector<double> mesh_dt, mesh_bandwidth, mesh_curv, mesh_length_scale;
};

struct SolverStats {
  long long steps_run = 0;
  long long fim_iters = 0, patch_visits = 0, check_visits = 0;
  long long nb_vertex_updates = 0, nb_patch_vertices = 0, nb_patches = 0, flagged_copies = 0;
  double ms_total = 0;
  double ms_sweep = 0, ms_check = 0, ms_schedule = 0, ms_seed = 0, ms_narrowband = 0, ms_update = 0;
  long long n_sweep = 0, n_check = 0, n_schedule = 0, n_seed = 0, n_narrowband = 0, n_update = 0;
  long long sweep_slab_bytes = 0;
  long long kernel_launches = 0;
  // learned warm start
  long long warm_vertices = 0, unsupported_resets = 0, support_rounds = 0, moved_vertices = 0;
  long long learned_fallbacks = 0, pairs_collected = 0;
  long long early_visits = 0;
};

// One profiled FIM launch: 0 sweep (or the persistent FIM loop), 1 check;
// device time; algorithmic slab bytes (-1 when not recorded).
struct LaunchRec {
  int kind;
  double ms;
  long long bytes;
};

class Solver {
 public:
  Solver() = default;
  ~Solver();
  // Upload the layout and the per-copy data; phi0 / vel in the caller's order.
  std::string init(const Layout& L, const SolverConfig& cfg, const float* vel);
  std::string set_phi(const float* phi_orig) { return settled(load_phi(phi_orig)); }  // host, caller order
  std::string get_phi(float* phi_orig) { return get_phi(phi_orig, 0, m_.nv); }        // host, caller order
  std::string get_phi(float* phi_orig, int first, int n) {  // n vertices from `first` on
    return settled(store_phi(phi_orig, first, n));
  }
  // Run nsteps; history (optional) gets phi after each step (host, caller order).
  std::string run(int nsteps, float* history, int* steps_done) { return settled(run_steps(nsteps, history, steps_done)); }
  std::string step_host(const float* phi_in, float* phi_out) { return settled(step_buffers(phi_in, phi_out)); }
  // Distance from arbitrary seed vertices (caller order), whole mesh, no
  // narrowband limit; out: nv floats in the caller's order.
  std::string eikonal(const int* seeds, const float* values, int nseeds, float* out) {
    return settled(solve_eikonal(seeds, values, nseeds, out));
  }
  std::string narrowband(unsigned char* flags);
  std::string active_patches(std::vector<int>& out);
  std::string dt_values(float* dt_new_order);
  void stats(SolverStats& s);  // reads the device counters if a step ran since the last read
  void reset_stats();
  // FIM launches of the profiled steps since the last reset_stats (oldest
  // first, at most kLaunchLogCap kept)
  const std::vector<LaunchRec>& launch_log() {
    if (stats_stale_) pull_stats();
    return launch_log_;
  }
  static constexpr size_t kLaunchLogCap = 1u << 20;
  int status_code() const { return status_; }
  void set_profile(bool on) { cfg_.profile = on ? 1 : 0; }
  // Learned warm start: each step's FIM starts from |network prediction| +
  // margin (FIM frame) on the previous narrowband, followed by support checks
  // (tolerance tol) until no warm value is left unsupported; net = null turns
  // it off.  Collection: steps record (features, post-redistance phi / h)
  // pairs of the previous narrowband's vertices into net's pair buffer.
  std::string set_learned(mlp::Net* net, float margin, float tol, bool whole_patch);
  std::string set_collect(mlp::Net* net);

 private:
  std::string check(cudaError_t e, const char* what);
  std::string one_step(bool* empty_nb);
  std::string learned_step(bool* empty_nb);
  std::string learn_buffers();
  std::string fim_loop(const StepParams& sp);
  std::string build_graph();
  // loop bodies' worth of iterations before the loop: at least 12 (tetrahedra) or 8 iterations
  int first_bodies() const { return ((m_.dim == 3 ? 12 : 8) + cfg_.graph_chunk - 1) / cfg_.graph_chunk; }
  bool build_persistent_graph(std::string* err);
  std::string emit_phi(float* row);
  // the calls above, with work on the caller's arrays still in flight on an error
  std::string settled(std::string r);
  std::string run_steps(int nsteps, float* history, int* steps_done);
  std::string step_buffers(const float* phi_in, float* phi_out);
  std::string solve_eikonal(const int* seeds, const float* values, int nseeds, float* out);
  std::string load_phi(const float* phi_orig);
  std::string store_phi(float* phi_orig, int first, int n);
  std::string run_chained(int nsteps, float* history, int* done);
  std::string enqueue_chain(int nsteps, float* history, int* done);
  cudaError_t end_chain();
  bool chained_ = false;  // CTL_CHAIN is set on the device
  std::string step_done(bool* empty_nb);
  cudaError_t step_head();
  cudaError_t step_tail();
  cudaError_t step_persistent_launches();
  cudaError_t restart_stamps(int from);
  cudaError_t read_ctl();
  std::string fim_status();
  int iter_cap() const;
  bool persistent_ = false;        // the step's FIM loop is one cooperative launch
  std::vector<double> mesh_scale_;  // FIM length unit of each mesh (one entry for a single mesh)
  void pull_stats();
  bool stats_stale_ = false;  // device counters changed since the last pull_stats
  // event pairs around the launches of profiled steps (cfg_.profile); kind 0
  // sweep, 1 check, 2 schedule, 3 seed, 4 narrowband, 5 update.  Each
  // profiled step folds its pairs into the stats when it ends and returns
  // the events to a pool, so the number of events stays that of one step.
  struct ProfEvent {
    cudaEvent_t a, b;
    int kind;
    int snap = -1;  // FIM launches: slot of the slab-byte counter snapshots around the launch
  };
  std::vector<ProfEvent> prof_;
  std::vector<LaunchRec> launch_log_;
  std::vector<cudaEvent_t> ev_pool_;
  cudaError_t prof_begin(ProfEvent& pe, int kind);
  // profiled FIM launches: the device's slab-byte counter (stats[7]) copied
  // before and after each launch into d_snap_ (slots of 2, at most kSnapCap
  // launches between two folds), read back when the times are folded
  static constexpr int kSnapCap = 4096;
  long long* d_snap_ = nullptr;
  long long* h_snap_ = nullptr;
  int nsnap_ = 0;
  cudaError_t prof_fim_begin(ProfEvent& pe, int kind);
  cudaError_t prof_fim_end(ProfEvent& pe);
  void fold_prof(bool keep_times);

  const Layout* lay_ = nullptr;
  const KernelSet* K_ = nullptr;
  SolverConfig cfg_;
  DevMesh m_{};
  DevState s_{};
  StepParams sp_{};
  Launch L_{};
  cudaStream_t stream_ = nullptr;
  cudaGraphExec_t graph_exec_ = nullptr;
  cudaGraph_t graph_ = nullptr;
  std::vector<void*> allocs_;
  int* h_ctl_ = nullptr;              // pinned mirror of the step control words (read_ctl)
  int* h_chunk_ = nullptr;            // two more, of the last chunks of fim_loop
  cudaEvent_t ev_chunk_[2] = {};
  int* d_seeds_ = nullptr;            // eikonal seeds and values, room for seed_cap_ of each
  int seed_cap_ = 0;
  unsigned long long* h_stats_ = nullptr;
  float* h_stage_ = nullptr;          // pinned nv floats
  float* d_tmp_ = nullptr;            // nv floats (caller-order staging)
  bool have_nb_ = false;              // previous narrowband valid (seed search restricted)
  int pageable_ = 0;                  // the GPU can access pageable host memory directly
  int status_ = 0;
  SolverStats st_;
  cudaEvent_t ev0_ = nullptr, ev1_ = nullptr;
  // learned warm start
  mlp::Net* net_ = nullptr;      // warm start on when set
  mlp::Net* collect_ = nullptr;  // pair collection on when set
  float margin_ = 0.f, support_tol_ = 5e-4f;
  bool support_patch_ = true;       // reset whole patches on an unsupported vertex
  DevLearn lr_{};
  int* adj_off_ = nullptr;       // vertex 1-ring CSR (product numbering)
  int* adj_ = nullptr;
  __nv_bfloat16* X_ = nullptr;   // features of the warm set
};

}  // namespace lsgb
