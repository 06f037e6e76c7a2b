// ls_solver.cu -- host orchestration of the device time step.
//
// The reference drives its FIM loop from the host with two synchronous
// device->host copies and a host list update per iteration
// (src/core3d/cuda/redistance3d.cu:85-224).  Here the lists, labels and
// convergence flags stay on the device; the host only launches a fixed
// chunk of FIM iterations (captured once as a CUDA graph) and reads one
// counter per chunk to learn whether the list has drained.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <vector>

#include "ls_solver.h"

namespace lsgb {

namespace {
template <typename T>
cudaError_t dalloc(std::vector<void*>& list, T** p, size_t n) {
  *p = nullptr;
  if (n == 0) n = 1;
  cudaError_t e = cudaMalloc((void**)p, sizeof(T) * n);
  if (e == cudaSuccess) list.push_back(*p);
  return e;
}
template <typename T>
cudaError_t upload(std::vector<void*>& list, const T** p, const std::vector<T>& v, cudaStream_t st) {
  T* d = nullptr;
  cudaError_t e = dalloc(list, &d, v.size());
  if (e != cudaSuccess) return e;
  if (!v.empty()) e = cudaMemcpyAsync(d, v.data(), sizeof(T) * v.size(), cudaMemcpyHostToDevice, st);
  *p = d;
  return e;
}

}  // namespace

Solver::~Solver() {
  if (graph_exec_) cudaGraphExecDestroy(graph_exec_);
  if (graph_) cudaGraphDestroy(graph_);
  for (void* p : allocs_) cudaFree(p);
  if (h_ctl_) cudaFreeHost(h_ctl_);
  if (d_seeds_) cudaFree(d_seeds_);
  if (h_stats_) cudaFreeHost(h_stats_);
  if (h_stage_) cudaFreeHost(h_stage_);
  if (h_snap_) cudaFreeHost(h_snap_);
  if (ev0_) cudaEventDestroy(ev0_);
  if (ev1_) cudaEventDestroy(ev1_);
  for (auto& pe : prof_) {
    cudaEventDestroy(pe.a);
    cudaEventDestroy(pe.b);
  }
  for (cudaEvent_t e : ev_pool_) cudaEventDestroy(e);
  for (cudaEvent_t e : ev_chunk_)
    if (e) cudaEventDestroy(e);
  if (stream_) cudaStreamDestroy(stream_);
}

// Two events for one profiled launch, from the pool where it has some.
cudaError_t Solver::prof_begin(ProfEvent& pe, int kind) {
  pe.kind = kind;
  cudaEvent_t ev[2];
  for (int i = 0; i < 2; ++i) {
    if (!ev_pool_.empty()) {
      ev[i] = ev_pool_.back();
      ev_pool_.pop_back();
    } else {
      cudaError_t e = cudaEventCreate(&ev[i]);
      if (e != cudaSuccess) {
        if (i == 1) ev_pool_.push_back(ev[0]);
        return e;
      }
    }
  }
  pe.a = ev[0];
  pe.b = ev[1];
  return cudaSuccess;
}

// A profiled FIM launch: events around it as for the other kernels, and the
// slab-byte counter copied (on the stream, device to device) just before
// and just after it, outside the event pair.
cudaError_t Solver::prof_fim_begin(ProfEvent& pe, int kind) {
  cudaError_t e = prof_begin(pe, kind);
  if (e != cudaSuccess) return e;
  pe.snap = -1;
  if (!d_snap_) {
    long long* d = nullptr;
    e = dalloc(allocs_, &d, (size_t)2 * kSnapCap);
    if (e == cudaSuccess) e = cudaMallocHost((void**)&h_snap_, sizeof(long long) * 2 * kSnapCap);
    if (e != cudaSuccess) return e;
    d_snap_ = d;
  }
  if (nsnap_ < kSnapCap) {
    pe.snap = nsnap_++;
    e = cudaMemcpyAsync(d_snap_ + 2 * pe.snap, s_.stats + 7, sizeof(long long), cudaMemcpyDeviceToDevice, stream_);
    if (e != cudaSuccess) return e;
  }
  return cudaEventRecord(pe.a, stream_);
}

cudaError_t Solver::prof_fim_end(ProfEvent& pe) {
  cudaError_t e = cudaEventRecord(pe.b, stream_);
  if (e == cudaSuccess && pe.snap >= 0)
    e = cudaMemcpyAsync(d_snap_ + 2 * pe.snap + 1, s_.stats + 7, sizeof(long long), cudaMemcpyDeviceToDevice,
                        stream_);
  prof_.push_back(pe);
  return e;
}

// Adds the pending launch times to the stats (keep_times) or drops them, and
// returns their events to the pool; FIM launches also go to the launch log
// with their slab bytes.
void Solver::fold_prof(bool keep_times) {
  bool snaps = false;
  if (keep_times && nsnap_ > 0)
    snaps = cudaMemcpyAsync(h_snap_, d_snap_, sizeof(long long) * 2 * nsnap_, cudaMemcpyDeviceToHost, stream_) ==
                cudaSuccess &&
            cudaStreamSynchronize(stream_) == cudaSuccess;
  nsnap_ = 0;
  for (auto& pe : prof_) {
    float ms = 0;
    if (keep_times && cudaEventSynchronize(pe.b) == cudaSuccess &&
        cudaEventElapsedTime(&ms, pe.a, pe.b) == cudaSuccess) {
      if (pe.kind <= 1 && launch_log_.size() < kLaunchLogCap)
        launch_log_.push_back(
            {pe.kind, (double)ms, (snaps && pe.snap >= 0) ? h_snap_[2 * pe.snap + 1] - h_snap_[2 * pe.snap] : -1});
      switch (pe.kind) {
        case 0: st_.ms_sweep += ms; st_.n_sweep++; break;
        case 1: st_.ms_check += ms; st_.n_check++; break;
        case 2: st_.ms_schedule += ms; st_.n_schedule++; break;
        case 3: st_.ms_seed += ms; st_.n_seed++; break;
        case 4: st_.ms_narrowband += ms; st_.n_narrowband++; break;
        case 5: st_.ms_update += ms; st_.n_update++; break;
      }
    }
    ev_pool_.push_back(pe.a);
    ev_pool_.push_back(pe.b);
  }
  prof_.clear();
}

std::string Solver::check(cudaError_t e, const char* what) {
  if (e == cudaSuccess) return "";
  status_ = 4;
  return std::string(what) + ": " + cudaGetErrorString(e);
}

#define LS_TRY(expr, what)                         \
  do {                                             \
    std::string _m = check((expr), (what));        \
    if (!_m.empty()) return _m;                    \
  } while (0)

std::string Solver::init(const Layout& L, const SolverConfig& cfg, const float* vel) {
  lay_ = &L;
  cfg_ = cfg;
  K_ = cfg.bit_exact ? &kernels_exact() : &kernels_fast();
  if (L.lep > 1024) { status_ = 2; return "a patch has more than 1024 element copies"; }
  // the limit the patch lists always had (30-bit patch ids)
  if (L.nparts >= (1 << 30)) return "too many patches";
  LS_TRY(cudaStreamCreateWithFlags(&stream_, cudaStreamNonBlocking), "stream");
  {
    int dev = 0;
    LS_TRY(cudaGetDevice(&dev), "device");
    if (cudaDeviceGetAttribute(&pageable_, cudaDevAttrPageableMemoryAccess, dev) != cudaSuccess) pageable_ = 0;
    if (cfg.host_staging) pageable_ = 0;
  }
  LS_TRY(cudaEventCreate(&ev0_), "event");
  LS_TRY(cudaEventCreate(&ev1_), "event");
  const int nv = L.nv, np = L.nparts;
  const long long full = L.full;
  const int d1 = L.dim + 1;

  // per-copy arrays
  std::vector<ushort4> conn(full);
  for (long long c = 0; c < full; ++c)
    conn[c] = make_ushort4(L.conn_local[c * 4], L.conn_local[c * 4 + 1], L.conn_local[c * 4 + 2],
                           L.conn_local[c * 4 + 3]);
  const int nc = L.dim == 3 ? 6 : 3;
  std::vector<float> lc((size_t)nc * full), sig((size_t)3 * full, 0.f);
  // FIM frame: without the reference's semantics, lengths are divided by
  // the mesh scale (mean edge length unless given) so that the local
  // solver's polynomial terms are O(1) in FP32 whatever the caller's units.
  const bool ref = cfg.ref_compat != 0;
  const double scale = ref ? 1.0 : (cfg.length_scale > 0 ? cfg.length_scale : L.mean_edge);
  // batches: each mesh has its own FIM frame
  const bool batch = !L.patch_mesh.empty();
  const int nmesh = batch ? (int)L.mesh_edge.size() : 1;
  std::vector<double> mscale(nmesh, scale);
  std::vector<double> copy_scale;
  if (batch) {
    if ((int)cfg.mesh_dt.size() != nmesh || (int)cfg.mesh_bandwidth.size() != nmesh ||
        (int)cfg.mesh_curv.size() != nmesh || (int)cfg.mesh_length_scale.size() != nmesh) {
      status_ = 1;
      return "per-mesh parameters missing";
    }
    for (int k = 0; k < nmesh; ++k)
      mscale[k] = ref ? 1.0 : (cfg.mesh_length_scale[k] > 0 ? cfg.mesh_length_scale[k] : L.mesh_edge[k]);
    copy_scale.resize(full);
    for (int p = 0; p < np; ++p)
      for (int c = L.ele_offsets[p]; c < L.ele_offsets[p + 1]; ++c) copy_scale[c] = mscale[L.patch_mesh[p]];
  }
  mesh_scale_ = mscale;
  for (long long c = 0; c < full; ++c) {
    const double cs = batch ? copy_scale[c] : scale;
    const int e = L.ele_permute[c];
    if (L.dim == 3) {
      float P[4][3], Lc[6];
      for (int k = 0; k < 4; ++k)
        for (int j = 0; j < 3; ++j) P[k][j] = L.xyz_p[(size_t)j * nv + L.conn[c * 4 + k]];
      tet_local_coords(P, Lc);
      for (int i = 0; i < 6; ++i) lc[i * full + c] = ref ? Lc[i] : (float)((double)Lc[i] / cs);
      if (vel)
        for (int j = 0; j < 3; ++j) sig[j * full + c] = vel[(size_t)e * 3 + j];
    } else {
      double P[3][3], Lc[3], sg[2], vv[3] = {0, 0, 0};
      for (int k = 0; k < 3; ++k)
        for (int j = 0; j < 3; ++j) P[k][j] = L.xyz_p[(size_t)j * nv + L.conn[c * 3 + k]];
      if (vel)
        for (int j = 0; j < 3; ++j) vv[j] = vel[(size_t)e * 3 + j];
      tri_local_coords(P, vv, Lc, sg);
      for (int i = 0; i < 3; ++i) lc[i * full + c] = (float)(ref ? Lc[i] : Lc[i] / cs);
      sig[c] = (float)sg[0];
      sig[full + c] = (float)sg[1];
    }
  }
  // per-patch algorithmic bytes of one FIM visit: owned DT read + DT_out
  // write + seed flags, ghost ids + ghost DT, connectivity (8 B) and local
  // coordinates (4 B each) per copy, 3 patch offsets pairs
  std::vector<int> pbytes(np);
  for (int p = 0; p < np; ++p) {
    const long long nvp = L.vert_offsets[p + 1] - L.vert_offsets[p];
    const long long ngp = L.ghost_offsets[p + 1] - L.ghost_offsets[p];
    const long long nep = L.ele_offsets[p + 1] - L.ele_offsets[p];
    pbytes[p] = (int)(nvp * (4 + 4 + 1) + ngp * (4 + 4) + nep * (8 + 4 * nc) + 24);
  }
  std::vector<int> ipermute(L.vert_ipermute);

  m_.dim = L.dim; m_.nv = nv; m_.nparts = np; m_.full = full;
  std::vector<void*>& A = allocs_;
  LS_TRY(upload(A, &m_.vert_off, L.vert_offsets, stream_), "upload");
  LS_TRY(upload(A, &m_.ele_off, L.ele_offsets, stream_), "upload");
  LS_TRY(upload(A, &m_.ghost_off, L.ghost_offsets, stream_), "upload");
  LS_TRY(upload(A, &m_.ghost_ids, L.ghost_ids, stream_), "upload");
  LS_TRY(upload(A, &m_.conn, conn, stream_), "upload");
  LS_TRY(upload(A, &m_.lc, lc, stream_), "upload");
  LS_TRY(upload(A, &m_.sig, sig, stream_), "upload");
  LS_TRY(upload(A, &m_.vslot_off, L.vslot_off, stream_), "upload");
  LS_TRY(upload(A, &m_.vslot, L.vslot, stream_), "upload");
  LS_TRY(upload(A, &m_.padj_off, L.padj_off, stream_), "upload");
  LS_TRY(upload(A, &m_.padj, L.padj, stream_), "upload");
  LS_TRY(upload(A, &m_.xyz, L.xyz_p, stream_), "upload");
  LS_TRY(upload(A, &m_.ipermute, ipermute, stream_), "upload");
  m_.capped = nullptr;
  m_.slot_cap = ref_slot_cap(L.dim);
  if (ref && L.any_capped) LS_TRY(upload(A, &m_.capped, L.slot_capped, stream_), "upload");
  m_.patch_mesh = nullptr;
  m_.mesh_par = nullptr;
  m_.geo_m = nullptr;
  m_.geo_h = nullptr;
  if (batch) {
    std::vector<float4> mp(nmesh);
    for (int k = 0; k < nmesh; ++k)
      mp[k] = make_float4((float)(cfg.mesh_bandwidth[k] / mscale[k]), (float)mscale[k], (float)cfg.mesh_dt[k],
                          (float)cfg.mesh_curv[k]);
    LS_TRY(upload(A, &m_.patch_mesh, L.patch_mesh, stream_), "upload");
    LS_TRY(upload(A, &m_.mesh_par, mp, stream_), "upload");
  }
  // step state
  LS_TRY(dalloc(A, &s_.phi, nv), "alloc");
  LS_TRY(dalloc(A, &s_.phi_rd, nv), "alloc");
  LS_TRY(dalloc(A, &s_.cell, nv), "alloc");
  LS_TRY(dalloc(A, &s_.slot, np), "alloc");
  LS_TRY(dalloc(A, &s_.pend, np), "alloc");
  LS_TRY(dalloc(A, &s_.reach, np), "alloc");
  LS_TRY(dalloc(A, &s_.lists, (size_t)3 * np), "alloc");
  LS_TRY(dalloc(A, &s_.nblist, np), "alloc");
  LS_TRY(dalloc(A, &s_.ctl, CTL_WORDS), "alloc");
  LS_TRY(dalloc(A, &s_.stats, 9), "alloc");
  LS_TRY(dalloc(A, &s_.sched, 4), "alloc");
  LS_TRY(dalloc(A, &s_.gbar, kGridBarrierWords), "alloc");
  LS_TRY(cudaMemsetAsync(s_.gbar, 0, sizeof(unsigned) * kGridBarrierWords, stream_), "memset");
  LS_TRY(dalloc(A, &d_tmp_, nv), "alloc");
  LS_TRY(cudaMemsetAsync(s_.slot, 0, sizeof(int) * np, stream_), "memset");
  LS_TRY(cudaMemsetAsync(s_.ctl, 0, sizeof(int) * CTL_WORDS, stream_), "memset");
  LS_TRY(cudaMemsetAsync(s_.stats, 0, sizeof(unsigned long long) * 9, stream_), "memset");
  LS_TRY(cudaMemsetAsync(s_.sched, 0, sizeof(int) * 4, stream_), "memset");
  LS_TRY(cudaMemsetAsync(s_.phi, 0, sizeof(float) * nv, stream_), "memset");
  LS_TRY(cudaMallocHost((void**)&h_ctl_, sizeof(int) * 3 * CTL_WORDS), "pinned");
  std::memset(h_ctl_, 0, sizeof(int) * 3 * CTL_WORDS);
  h_chunk_ = h_ctl_ + CTL_WORDS;
  for (cudaEvent_t& e : ev_chunk_) LS_TRY(cudaEventCreateWithFlags(&e, cudaEventDisableTiming), "event");
  // a few steps below the limit, so that every handle's stamps restart early in its life
  LS_TRY(restart_stamps(kStampLimit - 32), "stamps");
  LS_TRY(cudaMallocHost((void**)&h_stats_, sizeof(unsigned long long) * 9), "pinned");
  LS_TRY(cudaMallocHost((void**)&h_stage_, sizeof(float) * nv), "pinned");

  // parameters (FIM quantities in the FIM frame)
  sp_.largenum = (float)cfg.largenum;
  sp_.bandwidth = (float)(cfg.bandwidth / scale);
  sp_.scale = (float)scale;
  sp_.tau = (cfg.fp64_flagged && L.dim == 3) ? (float)cfg.fp64_tau : 0.f;
  sp_.xdiv = (cfg.bit_exact && ref) ? 1 : 0;
  // the planar-wave solver's denormal-keeping form where an edge is so short
  // that products of four lengths, or differences of such products, can be
  // denormal (lengths in the FIM frame: 1e-28 and their last bits)
  sp_.wide = 0;
  for (int k = 0; k < nmesh; ++k) {
    const double e = (batch ? L.mesh_min_edge[k] : L.min_edge) / mscale[k];
    if (e > 0 && e < 1e-7) sp_.wide = 1;
  }
  sp_.ctas = (cfg.fim_ctas >= 2 && cfg.fim_ctas <= 7) ? cfg.fim_ctas : 5;
  sp_.tol = (float)cfg.smallnum;
  sp_.eps_h64 = cfg.smallnum;
  sp_.eps_h = (float)sp_.eps_h64;
  sp_.dt = (float)cfg.dt;
  sp_.curv_coeff = (float)cfg.curv_coeff;
  sp_.niter = cfg.niter > 0 ? cfg.niter : (L.dim == 3 ? 5 : 10);
  sp_.ref_compat = ref ? 1 : 0;
  sp_.update_kind = cfg.update_kind;
  sp_.lvp = L.lvp;
  sp_.lgp = L.lgp;
  sp_.lep = L.lep;
  sp_.max_fim_iters = cfg.max_fim_iters;
  sp_.spin_limit = cfg.spin_limit != 0 ? cfg.spin_limit : (1 << 22);
  (void)d1;
  LS_TRY(K_->configure(m_, sp_, L_), "configure");
  if (cfg.fim_ctas == 0 && !cfg.bit_exact && !cfg.persistent && !(sp_.tau > 0.f) && !sp_.wide && L_.pair_block > 0 &&
      np >= 100 * L_.sms) {
    // The default's tet sweep on large meshes: setting 6's registers (56
    // instead of 64), where they let one more CTA reside -- blocks of 192
    // threads whose shared memory fits six times, of 160 threads where it fits
    // seven times -- and the lists are long.  Step times, 64 / 56 registers,
    // with the further CTA: 27-vertex blocks (324 copies) 32^3 (9 patches per
    // SM) 240 / 248 us, 40^3 (18) 280 / 283, 64^3 (70) 463 / 460, 80^3 (129)
    // 613 / 607, 128^3 (523) 1248 / 1206; 16-vertex graph patches (271) 64^3
    // (113) 794 / 779, 96^3 (375) 1494 / 1439; without it: the same at 80^3
    // (284 copies, 118 ghosts, 219) 1126 / 1166, 12-vertex graph patches 64^3
    // (151) 759 / 778, 8-vertex blocks 128^3 (1807) 1436 / 1471.  The bit-exact
    // build's solver spills more: 48^3 726 / 783 us.  Same results.
    StepParams six = sp_;
    Launch l6{};
    six.ctas = 6;
    LS_TRY(K_->configure(m_, six, l6), "configure");
    if (l6.fim_ctas > L_.fim_ctas) {
      sp_ = six;
      L_ = l6;
    }
  }
  if (L_.pair_block > 0) {
    // the two-copies-per-thread sweep stages precomputed per-copy geometry
    // (metric terms and heights, 64 bytes a copy) instead of the 24 bytes of
    // local coordinates it would otherwise turn into them on every visit
    float4* geo = nullptr;
    LS_TRY(dalloc(A, &geo, (size_t)4 * (size_t)full), "alloc");
    m_.geo_m = geo;
    m_.geo_h = geo + 3 * full;
    LS_TRY(K_->geometry(m_, geo, geo + 3 * full, L_, stream_), "geometry");
    for (int p = 0; p < np; ++p) {
      const long long nep = L.ele_offsets[p + 1] - L.ele_offsets[p];
      pbytes[p] += (int)(nep * (64 - 4 * nc));
    }
  }
  LS_TRY(upload(A, &m_.patch_bytes, pbytes, stream_), "upload");
  // the persistent FIM loop where the chosen sweep kernel has that form
  persistent_ = cfg_.persistent && L_.persist_grid > 0;
  if (cfg_.graph_chunk < 2) cfg_.graph_chunk = 2;
  if (cfg_.graph_chunk & 1) cfg_.graph_chunk++;
  if (cfg_.use_graph) {
    std::string r = build_graph();
    if (!r.empty()) return r;
  }
  LS_TRY(cudaStreamSynchronize(stream_), "init sync");
  return "";
}

// Step control kernel (host orchestration, same for both kernel builds): end
// of one FIM loop body of `chunk` iterations.  Continue while the next list
// is not empty.  The cap: iterations beyond the first `cap` that visited a
// patch (a list can hold candidates only, all found converged, so whether
// the cap is exceeded shows one body later); it sets CTL_CAP, so that the
// host reports a timeout.
namespace {
__device__ __forceinline__ bool body_end(int* ctl, unsigned long long* stats, int chunk, int cap) {
  if (ctl[CTL_STOP]) return false;
  ctl[CTL_BODIES] += 1;
  const int t = ctl[CTL_ITER] + chunk;
  count_iteration(ctl, stats, t - 1);
  ctl[CTL_ITER] = t;
  const bool more = ctl[CTL_VISITS + t % 3] + ctl[CTL_CANDS + t % 3] > 0;
  const bool over = ctl[CTL_ITERS] > cap;
  if (over) ctl[CTL_CAP] = 1;
  return more && !over && ctl[CTL_ERR] == 0;  // a FIM kernel wait that ran out ends the loop
}
__global__ void k_body_end(int* ctl, unsigned long long* stats, int chunk, int cap) {
  if (threadIdx.x == 0) body_end(ctl, stats, chunk, cap);
}
__global__ void k_loop_cond(int* ctl, unsigned long long* stats, cudaGraphConditionalHandle h, int chunk, int cap) {
  if (threadIdx.x == 0) cudaGraphSetConditional(h, body_end(ctl, stats, chunk, cap) ? 1u : 0u);
}
}  // namespace

// Clears every stamped array and starts the stamps again from `from`.
cudaError_t Solver::restart_stamps(int from) {
  cudaError_t e = cudaMemsetAsync(s_.cell, 0xff, sizeof(DtCell) * (size_t)m_.nv, stream_);
  if (e == cudaSuccess) e = cudaMemsetAsync(s_.pend, 0xff, sizeof(int) * m_.nparts, stream_);
  if (e == cudaSuccess) e = cudaMemsetAsync(s_.reach, 0xff, sizeof(int) * m_.nparts, stream_);
  h_ctl_[CTL_ITER] = from;
  if (e != cudaSuccess) return e;
  if (from == 0) return cudaMemsetAsync(s_.ctl + CTL_ITER, 0, sizeof(int), stream_);
  e = cudaMemcpyAsync(s_.ctl + CTL_ITER, h_ctl_ + CTL_ITER, sizeof(int), cudaMemcpyHostToDevice, stream_);
  return e == cudaSuccess ? cudaStreamSynchronize(stream_) : e;  // h_ctl_ is read until then
}

// The step control words on the host, and the stream idle.
cudaError_t Solver::read_ctl() {
  cudaError_t e = cudaMemcpyAsync(h_ctl_, s_.ctl, sizeof(int) * CTL_WORDS, cudaMemcpyDeviceToHost, stream_);
  return e == cudaSuccess ? cudaStreamSynchronize(stream_) : e;
}

// Whether the step's FIM loop ended as it should.
std::string Solver::fim_status() {
  if (h_ctl_[CTL_ERR]) {
    status_ = 3;
    return h_ctl_[CTL_ERR] == 1 ? "a grid barrier wait of the persistent FIM kernel timed out"
                                : "a geometry slab copy wait of the FIM kernel timed out";
  }
  if (h_ctl_[CTL_CAP]) {
    status_ = 3;
    return "FIM did not converge within max_fim_iters iterations";
  }
  return "";
}

// Iterations after which the loop gives up: the cap rounded up to whole bodies.
int Solver::iter_cap() const {
  const long long c = cfg_.graph_chunk, cap = ((long long)cfg_.max_fim_iters + c - 1) / c * c;
  return (int)std::min<long long>(cap, 0x7fffffff);
}

// One time step as one graph: seed part, the first iterations (first_bodies()
// x graph_chunk), a while node running loop bodies of graph_chunk iterations
// until the list drains (or the iteration cap), then narrowband and update.
// The host launches it and reads the control words once per step.
// The first iterations stand in a row because a body's boundary (its end
// kernel and the while node's turn) costs about 8 us, an iteration that finds
// its list empty about 3.  Steps of triangle meshes take 7 to 11 iterations,
// of tet meshes 10 to 13: eight and twelve in a row (whole bodies' worth).  Measured with 8 / 12 /
// 16: 2D 64^2, 20 steps 2042 / 2088 / 2217 us; 3D 32^3, 10 steps 2345 / 2291 /
// 2348 us, 16^3 step 181 / 175 / 181 us (in the loop from the start 2345,
// 2500, 214 us).
// The persistent form: the whole step is one captured sequence (seed part,
// the cooperative FIM launch, narrowband and update), no conditional node.
// Returns false when the runtime will not capture the cooperative launch (the
// step then launches kernel by kernel).
bool Solver::build_persistent_graph(std::string* err) {
  cudaGraph_t g = nullptr;
  if (cudaStreamBeginCapture(stream_, cudaStreamCaptureModeThreadLocal) != cudaSuccess) return false;
  cudaError_t e = step_persistent_launches();
  cudaError_t e2 = cudaStreamEndCapture(stream_, &g);
  if (e != cudaSuccess || e2 != cudaSuccess || !g) {
    if (g) cudaGraphDestroy(g);
    cudaGetLastError();  // clear the capture failure
    return false;
  }
  cudaError_t e3 = cudaGraphInstantiate(&graph_exec_, g, 0);
  graph_ = g;
  if (e3 != cudaSuccess) {
    *err = std::string("graph instantiate: ") + cudaGetErrorString(e3);
    graph_exec_ = nullptr;
    return false;
  }
  return true;
}

// The parts of a step before and after its FIM loop.
cudaError_t Solver::step_head() {
  cudaError_t e = K_->begin(s_, 0, stream_);
  return e == cudaSuccess ? K_->seed(m_, s_, sp_, L_, stream_) : e;
}
cudaError_t Solver::step_tail() {
  cudaError_t e = K_->narrowband(m_, s_, sp_, L_, stream_);
  if (cfg_.update_kind != 2)
    for (int it = 0; it < cfg_.inside_niter && e == cudaSuccess; ++it) e = K_->update(m_, s_, sp_, it == 0, L_, stream_);
  return e;
}

// One step of the persistent form, launch by launch.
cudaError_t Solver::step_persistent_launches() {
  cudaError_t err = step_head();
  if (err == cudaSuccess) err = K_->fim_persistent(m_, s_, sp_, L_, stream_);
  return err == cudaSuccess ? step_tail() : err;
}

std::string Solver::build_graph() {
  if (persistent_) {
    std::string err;
    if (build_persistent_graph(&err)) return "";
    if (!err.empty()) return err;
    return "";  // no graph: the persistent step launches kernel by kernel
  }
  const int chunk = cfg_.graph_chunk, first = first_bodies() * chunk;
  cudaGraph_t post = nullptr;
  cudaError_t err = cudaSuccess;
  LS_TRY(cudaStreamBeginCapture(stream_, cudaStreamCaptureModeThreadLocal), "capture begin");
  err = step_tail();
  cudaError_t e2 = cudaStreamEndCapture(stream_, &post);
  LS_TRY(err, "capture update part");
  LS_TRY(e2, "capture end");

  LS_TRY(cudaGraphCreate(&graph_, 0), "graph create");
  cudaGraphNode_t npre, nloop, npost;
  cudaGraphConditionalHandle hc;
  LS_TRY(cudaGraphConditionalHandleCreate(&hc, graph_, 0, cudaGraphCondAssignDefault), "conditional handle");
  // seed part and the first iterations
  LS_TRY(cudaStreamBeginCaptureToGraph(stream_, graph_, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal),
         "capture begin");
  err = step_head();
  for (int i = 0; i < first && err == cudaSuccess; ++i) err = K_->fim(m_, s_, sp_, i, L_, stream_);
  if (err == cudaSuccess) {
    k_loop_cond<<<1, 32, 0, stream_>>>(s_.ctl, s_.stats, hc, first, iter_cap());
    err = cudaGetLastError();
  }
  const cudaGraphNode_t* deps = nullptr;
  size_t ndeps = 0;
  if (err == cudaSuccess) {
    cudaStreamCaptureStatus status;
    err = cudaStreamGetCaptureInfo(stream_, &status, nullptr, nullptr, &deps, nullptr, &ndeps);
    if (err == cudaSuccess && ndeps != 1) err = cudaErrorUnknown;
  }
  if (err == cudaSuccess) npre = deps[0];
  cudaGraph_t same = nullptr;
  e2 = cudaStreamEndCapture(stream_, &same);
  LS_TRY(err, "capture first part");
  LS_TRY(e2, "capture end");
  cudaGraphNodeParams cp = {};
  cp.type = cudaGraphNodeTypeConditional;
  cp.conditional.handle = hc;
  cp.conditional.type = cudaGraphCondTypeWhile;
  cp.conditional.size = 1;
  LS_TRY(cudaGraphAddNode(&nloop, graph_, &npre, nullptr, 1, &cp), "graph while node");
  cudaGraph_t body = cp.conditional.phGraph_out[0];
  LS_TRY(cudaStreamBeginCaptureToGraph(stream_, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal),
         "capture body");
  err = cudaSuccess;
  for (int i = 0; i < chunk && err == cudaSuccess; ++i) err = K_->fim(m_, s_, sp_, i, L_, stream_);
  if (err == cudaSuccess) {
    k_loop_cond<<<1, 32, 0, stream_>>>(s_.ctl, s_.stats, hc, chunk, iter_cap());
    err = cudaGetLastError();
  }
  e2 = cudaStreamEndCapture(stream_, &body);
  LS_TRY(err, "capture body launch");
  LS_TRY(e2, "capture body end");
  LS_TRY(cudaGraphAddChildGraphNode(&npost, graph_, &nloop, 1, post), "graph child");
  cudaGraphDestroy(post);
  LS_TRY(cudaGraphInstantiate(&graph_exec_, graph_, 0), "graph instantiate");
  return "";
}

// Iterations launched one by one, in chunks of graph_chunk.  The next chunk
// is enqueued before the host waits for the last one's control words, so the
// GPU does not idle for the round trip (about 15 us a chunk); the chunk
// behind the one that drains the list finds it empty.  Profiled steps wait
// for each chunk (their launches are counted).
std::string Solver::fim_loop(const StepParams& sp) {
  auto prof = [&](auto&& fn) -> cudaError_t {
    if (!cfg_.profile) return fn();
    ProfEvent pe;
    cudaError_t e = prof_fim_begin(pe, 0);
    if (e != cudaSuccess) return e;
    e = fn();
    cudaError_t e2 = prof_fim_end(pe);
    return e != cudaSuccess ? e : e2;
  };
  const int ahead = cfg_.profile ? 0 : 1;
  for (int k = 0;; ++k) {
    for (int i = 0; i < cfg_.graph_chunk; ++i)
      LS_TRY(prof([&] { return K_->fim(m_, s_, sp, i, L_, stream_); }), "FIM iteration");
    k_body_end<<<1, 32, 0, stream_>>>(s_.ctl, s_.stats, cfg_.graph_chunk, iter_cap());
    LS_TRY(cudaGetLastError(), "body end");
    st_.kernel_launches += cfg_.graph_chunk + 1;
    int* const mine = h_chunk_ + (k & 1) * CTL_WORDS;
    LS_TRY(cudaMemcpyAsync(mine, s_.ctl, sizeof(int) * CTL_WORDS, cudaMemcpyDeviceToHost, stream_), "d2h");
    LS_TRY(cudaEventRecord(ev_chunk_[k & 1], stream_), "event");
    if (k < ahead) continue;
    const int done = (k - ahead) & 1;
    LS_TRY(cudaEventSynchronize(ev_chunk_[done]), "fim sync");
    const int* c = h_chunk_ + done * CTL_WORDS;
    const int cur = c[CTL_ITER] % 3;
    if (c[CTL_ERR] || c[CTL_CAP] || c[CTL_VISITS + cur] + c[CTL_CANDS + cur] == 0) break;
  }
  LS_TRY(read_ctl(), "fim end");
  return fim_status();
}

// A step run in one go has ended with the control words in h_ctl_.
std::string Solver::step_done(bool* empty_nb) {
  // begin, seed, the FIM loop, narrowband, the updates and the copies between them
  const long long upd = cfg_.update_kind != 2 ? 2LL * cfg_.inside_niter - 1 : 0;
  st_.kernel_launches += 3 + upd + (persistent_ ? 1LL
                                                : (cfg_.graph_chunk + 1LL) * h_ctl_[CTL_BODIES] +
                                                      (first_bodies() - 1LL) * cfg_.graph_chunk);
  std::string r = fim_status();
  if (!r.empty()) return r;
  have_nb_ = h_ctl_[CTL_NB] != 0;
  *empty_nb = !have_nb_;
  return "";
}

// Nothing may be in flight that reads or writes a caller's array when a call
// returns an error: the caller may free it then.
std::string Solver::settled(std::string r) {
  if (!r.empty()) cudaStreamSynchronize(stream_);
  return r;
}

// Ends a chain of steps (run_chained), also one whose end failed before.
cudaError_t Solver::end_chain() {
  if (!chained_) return cudaSuccess;
  const cudaError_t e = cudaMemsetAsync(s_.ctl + CTL_CHAIN, 0, sizeof(int), stream_);
  if (e == cudaSuccess) chained_ = false;
  return e;
}

std::string Solver::one_step(bool* empty_nb) {
  *empty_nb = false;
  LS_TRY(end_chain(), "memset");
  auto prof = [&](int kind, auto&& fn) -> cudaError_t {
    if (!cfg_.profile) return fn();
    ProfEvent pe;
    cudaError_t e = prof_begin(pe, kind);
    if (e != cudaSuccess) return e;
    cudaEventRecord(pe.a, stream_);
    e = fn();
    cudaEventRecord(pe.b, stream_);
    prof_.push_back(pe);
    return e;
  };
  if (h_ctl_[CTL_ITER] > kStampLimit) LS_TRY(restart_stamps(0), "stamps");
  if (net_ || collect_) return learned_step(empty_nb);
  if (persistent_ || (graph_exec_ && !cfg_.profile)) {
    // the whole step in one go: its graph, or the persistent form launch by
    // launch (profiled: the FIM loop kernel's time is recorded as the sweep time)
    if (graph_exec_ && !cfg_.profile) {
      LS_TRY(cudaGraphLaunch(graph_exec_, stream_), "graph launch");
    } else {
      ProfEvent pe{};
      if (cfg_.profile) LS_TRY(prof_fim_begin(pe, 0), "event");
      LS_TRY(step_persistent_launches(), "persistent step");
      if (cfg_.profile) LS_TRY(prof_fim_end(pe), "event");
    }
    LS_TRY(read_ctl(), "step sync");
    return step_done(empty_nb);
  }
  LS_TRY(K_->begin(s_, 0, stream_), "begin");
  LS_TRY(prof(3, [&] { return K_->seed(m_, s_, sp_, L_, stream_); }), "seed");
  st_.kernel_launches += 3;  // begin, seed, narrowband
  std::string r = fim_loop(sp_);
  if (!r.empty()) return r;
  LS_TRY(prof(4, [&] { return K_->narrowband(m_, s_, sp_, L_, stream_); }), "narrowband");
  LS_TRY(read_ctl(), "nb sync");
  have_nb_ = h_ctl_[CTL_NB] != 0;
  if (!have_nb_) {
    *empty_nb = true;
    return "";
  }
  if (cfg_.update_kind != 2) {
    for (int it = 0; it < cfg_.inside_niter; ++it)
      LS_TRY(prof(5, [&] { return K_->update(m_, s_, sp_, it == 0, L_, stream_); }), "update");
    st_.kernel_launches += 2LL * cfg_.inside_niter - 1;
  }
  return "";
}

// ---------------------------------------------------------------------------
// Learned warm start.

std::string Solver::learn_buffers() {
  if (X_) return "";
  const Layout& L = *lay_;
  const int nv = m_.nv, d1 = m_.dim + 1;
  // 1-ring from the element copies (each element once), sorted and unique
  std::vector<std::vector<int>> ring(nv);
  std::vector<char> seen(L.ne, 0);
  for (long long c = 0; c < L.full; ++c) {
    const int e = L.ele_permute[c];
    if (seen[e]) continue;
    seen[e] = 1;
    for (int a = 0; a < d1; ++a)
      for (int b = 0; b < d1; ++b)
        if (a != b) ring[L.conn[c * d1 + a]].push_back(L.conn[c * d1 + b]);
  }
  std::vector<int> off(nv + 1, 0), adj;
  for (int v = 0; v < nv; ++v) {
    auto& r = ring[v];
    std::sort(r.begin(), r.end());
    r.erase(std::unique(r.begin(), r.end()), r.end());
    off[v + 1] = off[v] + (int)r.size();
  }
  adj.reserve(off[nv]);
  for (int v = 0; v < nv; ++v) adj.insert(adj.end(), ring[v].begin(), ring[v].end());
  std::vector<void*>& A = allocs_;
  const int* d_off = nullptr;
  const int* d_adj = nullptr;
  LS_TRY(upload(A, &d_off, off, stream_), "upload");
  LS_TRY(upload(A, &d_adj, adj, stream_), "upload");
  adj_off_ = const_cast<int*>(d_off);
  adj_ = const_cast<int*>(d_adj);
  LS_TRY(dalloc(A, &lr_.vlist, nv), "alloc");
  LS_TRY(dalloc(A, &lr_.cnt, 4), "alloc");
  LS_TRY(dalloc(A, &lr_.pred, nv), "alloc");
  LS_TRY(dalloc(A, &lr_.warm, nv), "alloc");
  LS_TRY(dalloc(A, &lr_.target, nv), "alloc");
  LS_TRY(dalloc(A, &X_, (size_t)nv * 128), "alloc");
  lr_.vinv_h = nullptr;
  if (m_.patch_mesh) {
    // a batch: features and targets in units of each vertex's own mesh
    std::vector<float> vinv(nv, 1.f);
    for (int p = 0; p < m_.nparts; ++p)
      for (int v = L.vert_offsets[p]; v < L.vert_offsets[p + 1]; ++v)
        vinv[v] = (float)(1.0 / mesh_scale_[L.patch_mesh[p]]);
    const float* d = nullptr;
    LS_TRY(upload(A, &d, vinv, stream_), "upload");
    lr_.vinv_h = d;
  }
  LS_TRY(cudaStreamSynchronize(stream_), "sync");
  return "";
}

std::string Solver::set_learned(mlp::Net* net, float margin, float tol, bool whole_patch) {
  support_patch_ = whole_patch;
  if (net) {
    std::string r = learn_buffers();
    if (!r.empty()) return r;
  }
  net_ = net;
  margin_ = margin;
  if (tol > 0.f) support_tol_ = tol;
  return "";
}

std::string Solver::set_collect(mlp::Net* net) {
  if (net) {
    std::string r = learn_buffers();
    if (!r.empty()) return r;
  }
  collect_ = net;
  return "";
}

// One time step with the warm start and / or pair collection, launch by
// launch (the support rounds are decided on the host).
std::string Solver::learned_step(bool* empty_nb) {
  *empty_nb = false;
  const bool prev = have_nb_;
  const bool warm = net_ && prev;
  LS_TRY(K_->begin(s_, 0, stream_), "begin");
  if (prev) {
    LS_TRY(read_ctl(), "sync");
    const int nb_prev = h_ctl_[CTL_NB_PREV];
    LS_TRY(cudaMemsetAsync(lr_.cnt, 0, sizeof(int) * 4, stream_), "memset");
    LS_TRY(K_->learn(LEARN_NB_VERTICES, m_, s_, sp_, lr_, nb_prev, 0.f, L_, stream_), "warm set");
    mlp::k_features<<<L_.flat_grid, 256, 0, stream_>>>(0, lr_.vlist, lr_.cnt, adj_off_, adj_, m_.xyz, m_.nv, s_.phi,
                                                        1.f / sp_.scale, lr_.vinv_h, X_);
    LS_TRY(cudaGetLastError(), "features");
    st_.kernel_launches += 2;
    if (warm) {
      std::string r = net_->forward_dev(X_, 0, lr_.cnt, m_.nv, lr_.pred, stream_);
      if (!r.empty()) return r;
      LS_TRY(K_->learn(LEARN_WARM, m_, s_, sp_, lr_, 0, margin_, L_, stream_), "warm apply");
      st_.kernel_launches += 2;
    }
  }
  if (warm) LS_TRY(K_->learn(LEARN_SEED_WARM, m_, s_, sp_, lr_, 0, 0.f, L_, stream_), "seed");
  else LS_TRY(K_->seed(m_, s_, sp_, L_, stream_), "seed");
  st_.kernel_launches += 2;
  std::string r = fim_loop(sp_);
  if (!r.empty()) return r;
  if (warm) {
    // support rounds: reset unsupported warm values, FIM again, until none
    const int max_rounds = 16;
    bool clean = false;
    for (int round = 0; round < max_rounds; ++round) {
      LS_TRY(K_->learn(LEARN_SUPPORT, m_, s_, sp_, lr_, support_patch_ ? 1 : 0, support_tol_, L_, stream_),
             "support");
      LS_TRY(read_ctl(), "sync");
      st_.kernel_launches += 1;
      st_.support_rounds++;
      if (h_ctl_[CTL_VISITS + h_ctl_[CTL_ITER] % 3] == 0) {
        clean = true;
        break;
      }
      r = fim_loop(sp_);
      if (!r.empty()) return r;
    }
    if (!clean) {
      // plain FIM from the seeds: the fallback
      st_.learned_fallbacks++;
      LS_TRY(K_->begin(s_, 1, stream_), "begin");
      LS_TRY(K_->seed(m_, s_, sp_, L_, stream_), "seed");
      r = fim_loop(sp_);
      if (!r.empty()) return r;
    }
    LS_TRY(K_->learn(LEARN_MOVED, m_, s_, sp_, lr_, 0, 1e-3f, L_, stream_), "moved");
    st_.kernel_launches += 1;
  }
  LS_TRY(K_->narrowband(m_, s_, sp_, L_, stream_), "narrowband");
  st_.kernel_launches += 1;
  if (collect_ && prev) {
    LS_TRY(K_->learn(LEARN_TARGETS, m_, s_, sp_, lr_, 0, 1.f / sp_.scale, L_, stream_), "targets");
    st_.kernel_launches += 1;
    long long added = 0;
    r = collect_->append_pairs(X_, lr_.target, lr_.cnt, m_.nv, stream_, &added);
    if (!r.empty()) return r;
    st_.pairs_collected += added;
  }
  int cnt[4] = {};
  LS_TRY(cudaMemcpyAsync(cnt, lr_.cnt, sizeof(cnt), cudaMemcpyDeviceToHost, stream_), "d2h");
  LS_TRY(read_ctl(), "sync");
  if (warm) {
    st_.warm_vertices += cnt[0];
    st_.unsupported_resets += cnt[1];
    st_.moved_vertices += cnt[2];
  }
  have_nb_ = h_ctl_[CTL_NB] != 0;
  if (!have_nb_) {
    *empty_nb = true;
    return "";
  }
  if (cfg_.update_kind != 2) {
    for (int it = 0; it < cfg_.inside_niter; ++it) {
      LS_TRY(K_->update(m_, s_, sp_, it == 0, L_, stream_), "update");
      st_.kernel_launches += it == 0 ? 1 : 2;
    }
  }
  return "";
}

// The work counters and the profiled launch times are read from the device
// when a caller asks for them (stats), not after every step: a step through
// host buffers then ends with its own result copy and no second round trip.
void Solver::pull_stats() {
  if (cudaMemcpyAsync(h_stats_, s_.stats, sizeof(unsigned long long) * 9, cudaMemcpyDeviceToHost, stream_) !=
          cudaSuccess ||
      cudaStreamSynchronize(stream_) != cudaSuccess)
    return;
  stats_stale_ = false;
  st_.patch_visits = (long long)h_stats_[0];
  st_.check_visits = (long long)h_stats_[1];
  st_.nb_vertex_updates = (long long)h_stats_[2];
  st_.nb_patch_vertices = (long long)h_stats_[3];
  st_.nb_patches = (long long)h_stats_[4];
  st_.fim_iters = (long long)h_stats_[5];
  st_.sweep_slab_bytes = (long long)h_stats_[7];
  st_.flagged_copies = (long long)h_stats_[6];
  st_.early_visits = (long long)h_stats_[8];
  fold_prof(true);
}

// One row of a run's history: where the GPU can write the caller's array, the
// row is on its way when this returns and complete when the stream is (run
// ends with a wait); the next step is enqueued behind it.
std::string Solver::emit_phi(float* row) {
  if (!pageable_) return store_phi(row, 0, m_.nv);
  LS_TRY(K_->unpermute(m_, s_.phi, 0, m_.nv, row, nullptr, L_, stream_), "unpermute");
  return "";
}

// Steps of a run as graphs, each enqueued before the host knows how the
// previous one ended (the round trip, about 15 us, is behind the next step).
// A step behind one that ran out of narrowband or failed does nothing
// (CTL_STOP), and neither does its history row.
std::string Solver::run_chained(int nsteps, float* history, int* done) {
  LS_TRY(end_chain(), "memset");
  std::string r = enqueue_chain(nsteps, history, done);
  const cudaError_t e = end_chain();
  if (r.empty()) r = check(e, "memset");
  if (r.empty()) r = check(cudaStreamSynchronize(stream_), "run sync");
  return r;
}

std::string Solver::enqueue_chain(int nsteps, float* history, int* done) {
  std::string r;
  bool empty = false;
  auto settle = [&](int s) -> std::string {
    const int* c = h_chunk_ + (s & 1) * CTL_WORDS;
    LS_TRY(cudaEventSynchronize(ev_chunk_[s & 1]), "step sync");
    std::memcpy(h_ctl_, c, sizeof(int) * CTL_WORDS);
    std::string e = step_done(&empty);
    if (e.empty() && !empty) ++*done;
    return e;
  };
  int s = 0;
  bool pending = false;  // step s - 1 has not been settled
  for (; s < nsteps && r.empty() && !empty; ++s) {
    if (h_ctl_[CTL_ITER] > kStampLimit) {
      // behind a step whose end is known: the distances of a run's last step
      // stay readable
      if (pending) r = settle(s - 1);
      pending = false;
      if (!r.empty() || empty) break;
      LS_TRY(restart_stamps(0), "stamps");
    }
    LS_TRY(cudaGraphLaunch(graph_exec_, stream_), "graph launch");
    if (history)
      LS_TRY(K_->unpermute(m_, s_.phi, 0, m_.nv, history + (size_t)(s + 1) * m_.nv, s_.ctl, L_, stream_), "unpermute");
    LS_TRY(cudaMemcpyAsync(h_chunk_ + (s & 1) * CTL_WORDS, s_.ctl, sizeof(int) * CTL_WORDS, cudaMemcpyDeviceToHost,
                           stream_), "d2h");
    LS_TRY(cudaEventRecord(ev_chunk_[s & 1], stream_), "event");
    if (s == 0) {
      chained_ = true;
      LS_TRY(cudaMemsetAsync(s_.ctl + CTL_CHAIN, 1, sizeof(int), stream_), "memset");
    }
    if (pending) r = settle(s - 1);
    pending = true;
  }
  // the last enqueued step, unless the one before it ended the run
  if (r.empty() && !empty && pending) r = settle(s - 1);
  return r;
}

std::string Solver::run_steps(int nsteps, float* history, int* steps_done) {
  int done = 0;
  std::string h;
  if (history && !(h = emit_phi(history)).empty()) return h;
  LS_TRY(cudaEventRecord(ev0_, stream_), "event");
  const bool chained = nsteps > 1 && graph_exec_ && !cfg_.profile && !net_ && !collect_ && (!history || pageable_);
  if (chained) {
    h = run_chained(nsteps, history, &done);
    if (!h.empty()) return h;
  }
  for (int s = 0; s < nsteps && !chained; ++s) {
    bool empty = false;
    std::string r = one_step(&empty);
    if (!r.empty()) return r;
    if (cfg_.profile) fold_prof(true);
    if (empty) break;
    done++;
    if (history && !(h = emit_phi(history + (size_t)(s + 1) * m_.nv)).empty()) return h;
  }
  LS_TRY(cudaEventRecord(ev1_, stream_), "event");
  LS_TRY(cudaEventSynchronize(ev1_), "event sync");
  float ms = 0;
  cudaEventElapsedTime(&ms, ev0_, ev1_);
  st_.ms_total += ms;
  st_.steps_run += done;
  if (steps_done) *steps_done = done;
  stats_stale_ = true;
  return "";
}

std::string Solver::step_buffers(const float* phi_in, float* phi_out) {
  const int nv = m_.nv;
  if (pageable_) {
    // the GPU reads and writes the caller's pageable host arrays directly
    // (coherent access over the CPU-GPU link): the permutation kernels read
    // and write the caller's side in its order (coalesced) and scatter or
    // gather on the device side, with no staging copy on either side
    LS_TRY(K_->permute(m_, phi_in, s_.phi, L_, stream_), "permute in");
  } else {
    std::memcpy(h_stage_, phi_in, sizeof(float) * nv);
    LS_TRY(cudaMemcpyAsync(d_tmp_, h_stage_, sizeof(float) * nv, cudaMemcpyHostToDevice, stream_), "h2d");
    LS_TRY(K_->permute(m_, d_tmp_, s_.phi, L_, stream_), "permute");
  }
  st_.kernel_launches += 2;  // permute, unpermute
  bool empty = false;
  std::string r = one_step(&empty);
  if (!r.empty()) return r;
  if (cfg_.profile) fold_prof(true);
  if (pageable_) {
    LS_TRY(K_->unpermute(m_, s_.phi, 0, nv, phi_out, nullptr, L_, stream_), "unpermute out");
    LS_TRY(cudaStreamSynchronize(stream_), "sync");
  } else {
    r = store_phi(phi_out, 0, nv);
    if (!r.empty()) return r;
  }
  if (!empty) st_.steps_run++;
  stats_stale_ = true;
  return "";
}

// Standalone eikonal solve: the seeds, the first list and the result on the
// device (host loops over the copies, the cells and the permutation took 7 of
// 10.5 ms at 64^3).
namespace {
// The last of several values given for one vertex counts.
__global__ void k_eik_order(DevMesh m, const int* seeds, int n, int* order) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) atomicMax(order + __ldg(m.ipermute + seeds[i]), i);
}
__global__ void k_eik_seed(DevMesh m, DevState s, const int* seeds, const float* values, int n, const int* order,
                           float scale, float LN) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int v = __ldg(m.ipermute + seeds[i]);
  if (order[v] != i) return;
  const float a = values[i] >= LN ? LN : values[i] / scale;
  if (a > LN) s.ctl[CTL_ABOVE] = 1;
  *reinterpret_cast<int2*>(s.cell + v) = make_int2(__float_as_int(a), s.ctl[CTL_BASE]);
}
// The patches one of whose element copies holds a seed (the list the seed
// kernel makes at the start of a time step): a patch's copies' vertices are
// its own and its ghosts.  One warp per patch.
__global__ void k_eik_list(DevMesh m, DevState s) {
  const int lane = threadIdx.x & 31, nwarps = (gridDim.x * blockDim.x) >> 5;
  const int base = s.ctl[CTL_BASE], t0 = s.ctl[CTL_ITER];
  for (int p = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; p < m.nparts; p += nwarps) {
    const int vs = m.vert_off[p], nvp = m.vert_off[p + 1] - vs;
    const int gs = m.ghost_off[p], ngp = m.ghost_off[p + 1] - gs;
    bool hit = false;
    for (int i = lane; i < nvp + ngp; i += 32)
      hit |= dt_is_seed(s.cell[i < nvp ? vs + i : __ldg(m.ghost_ids + gs + i - nvp)], base);
    if (__any_sync(0xffffffffu, hit) && lane == 0) {
      s.lists[(size_t)(t0 % 3) * m.nparts + atomicAdd(s.ctl + CTL_VISITS + t0 % 3, 1)] = p;
      s.pend[p] = 2 * t0;
    }
  }
}
// out[old]: the distance in the caller's units
__global__ void k_eik_out(DevMesh m, DevState s, float scale, float LN, float* out) {
  const int base = s.ctl[CTL_BASE];
  for (int o = blockIdx.x * blockDim.x + threadIdx.x; o < m.nv; o += gridDim.x * blockDim.x) {
    const float d = dt_before(s.cell[__ldg(m.ipermute + o)], kStampMax, base, LN);
    out[o] = d >= LN ? LN : d * scale;
  }
}
}  // namespace

std::string Solver::solve_eikonal(const int* seeds, const float* values, int nseeds, float* out) {
  if (m_.patch_mesh) {
    status_ = 1;
    return "the standalone eikonal solve takes one mesh, not a batch";
  }
  const int nv = m_.nv, n = nseeds;
  const float LN = sp_.largenum;
  if (h_ctl_[CTL_ITER] > kStampLimit) LS_TRY(restart_stamps(0), "stamps");
  LS_TRY(end_chain(), "memset");
  LS_TRY(K_->begin(s_, 0, stream_), "begin");
  if (n > 0) {
    if (n > seed_cap_) {
      // seeds and values of the largest call so far
      if (d_seeds_) LS_TRY(cudaFree(d_seeds_), "free");
      d_seeds_ = nullptr;
      seed_cap_ = 0;
      LS_TRY(cudaMalloc((void**)&d_seeds_, (sizeof(int) + sizeof(float)) * (size_t)n), "alloc");
      seed_cap_ = n;
    }
    float* d_values = reinterpret_cast<float*>(d_seeds_ + seed_cap_);
    int* order = reinterpret_cast<int*>(d_tmp_);
    LS_TRY(cudaMemcpyAsync(d_seeds_, seeds, sizeof(int) * (size_t)n, cudaMemcpyHostToDevice, stream_), "h2d");
    LS_TRY(cudaMemcpyAsync(d_values, values, sizeof(float) * (size_t)n, cudaMemcpyHostToDevice, stream_), "h2d");
    LS_TRY(cudaMemsetAsync(order, 0xff, sizeof(int) * (size_t)nv, stream_), "memset");
    const int grid = (n + 255) / 256;
    k_eik_order<<<grid, 256, 0, stream_>>>(m_, d_seeds_, n, order);
    k_eik_seed<<<grid, 256, 0, stream_>>>(m_, s_, d_seeds_, d_values, n, order, sp_.scale, LN);
    k_eik_list<<<L_.warp_grid, 256, 0, stream_>>>(m_, s_);
    LS_TRY(cudaGetLastError(), "eikonal seeds");
  }
  LS_TRY(cudaMemsetAsync(s_.ctl + CTL_NB_VALID, 0, sizeof(int), stream_), "memset");
  StepParams sp = sp_;
  // no narrowband limit: every converged patch that the front has reached
  // (minimum below LARGENUM) activates its neighbours
  sp.bandwidth = LN;
  std::string r = fim_loop(sp);
  if (!r.empty()) return r;
  if (cfg_.profile) fold_prof(true);
  // to the caller's pageable array where the GPU can write it (step_host)
  float* const dst = pageable_ ? out : d_tmp_;
  k_eik_out<<<L_.flat_grid, 256, 0, stream_>>>(m_, s_, sp_.scale, LN, dst);
  LS_TRY(cudaGetLastError(), "eikonal result");
  if (!pageable_)
    LS_TRY(cudaMemcpyAsync(h_stage_, d_tmp_, sizeof(float) * nv, cudaMemcpyDeviceToHost, stream_), "d2h");
  LS_TRY(cudaStreamSynchronize(stream_), "sync");
  if (!pageable_) std::memcpy(out, h_stage_, sizeof(float) * nv);
  have_nb_ = false;  // the step state was overwritten
  stats_stale_ = true;
  return "";
}

std::string Solver::load_phi(const float* phi_orig) {
  const float* src = phi_orig;
  if (!pageable_) {
    std::memcpy(h_stage_, phi_orig, sizeof(float) * m_.nv);
    LS_TRY(cudaMemcpyAsync(d_tmp_, h_stage_, sizeof(float) * m_.nv, cudaMemcpyHostToDevice, stream_), "h2d");
    src = d_tmp_;
  }
  LS_TRY(K_->permute(m_, src, s_.phi, L_, stream_), "permute");
  LS_TRY(cudaMemsetAsync(s_.ctl + CTL_NB_VALID, 0, sizeof(int), stream_), "memset");
  LS_TRY(cudaStreamSynchronize(stream_), "sync");
  have_nb_ = false;
  return "";
}

std::string Solver::store_phi(float* phi_orig, int first, int n) {
  float* const dst = pageable_ ? phi_orig : d_tmp_;
  LS_TRY(K_->unpermute(m_, s_.phi, first, n, dst, nullptr, L_, stream_), "unpermute");
  if (!pageable_)
    LS_TRY(cudaMemcpyAsync(h_stage_, d_tmp_, sizeof(float) * n, cudaMemcpyDeviceToHost, stream_), "d2h");
  LS_TRY(cudaStreamSynchronize(stream_), "sync");
  if (!pageable_) std::memcpy(phi_orig, h_stage_, sizeof(float) * n);
  return "";
}

std::string Solver::narrowband(unsigned char* flags) {
  LS_TRY(read_ctl(), "d2h");
  const int n = h_ctl_[CTL_NB];
  std::vector<int> nb(n > 0 ? n : 1);
  if (n > 0) LS_TRY(cudaMemcpy(nb.data(), s_.nblist, sizeof(int) * n, cudaMemcpyDeviceToHost), "d2h");
  std::memset(flags, 0, m_.nparts);
  for (int i = 0; i < n; ++i) flags[nb[i]] = 1;
  return "";
}

std::string Solver::active_patches(std::vector<int>& out) {
  LS_TRY(read_ctl(), "d2h");
  const int cur = h_ctl_[CTL_ITER] % 3, n = h_ctl_[CTL_VISITS + cur];
  out.assign(n, 0);
  if (n > 0)
    LS_TRY(cudaMemcpy(out.data(), s_.lists + (size_t)cur * m_.nparts, sizeof(int) * n, cudaMemcpyDeviceToHost), "d2h");
  return "";
}

std::string Solver::dt_values(float* dt) {
  LS_TRY(K_->distances(m_, s_, sp_, d_tmp_, L_, stream_), "distances");
  LS_TRY(cudaMemcpyAsync(dt, d_tmp_, sizeof(float) * m_.nv, cudaMemcpyDeviceToHost, stream_), "d2h");
  LS_TRY(cudaStreamSynchronize(stream_), "sync");
  return "";
}

void Solver::stats(SolverStats& s) {
  if (stats_stale_) pull_stats();
  s = st_;
}

void Solver::reset_stats() {
  cudaMemsetAsync(s_.stats, 0, sizeof(unsigned long long) * 9, stream_);
  cudaStreamSynchronize(stream_);
  // launch times recorded before the reset are dropped with the counters
  fold_prof(false);
  launch_log_.clear();
  st_ = SolverStats();
  stats_stale_ = false;
}

}  // namespace lsgb
