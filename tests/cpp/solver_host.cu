// solver_host.cu -- the orchestration of ls_solver.cu on the CPU, over the
// runtime of fake_cuda.h and a set of kernels that only keep the step control
// words as the real ones do.  Each argument names a check; the program prints
// what does not hold and returns the number of failures.
#include <cstdio>
#include <memory>
#include <sstream>

#include "fake_cuda.h"

#define private public
#include "ls_solver.h"
#undef private

namespace lsgb {
namespace {
int failures = 0;
#define CHECK(cond, ...)            \
  do {                              \
    if (!(cond)) {                  \
      ++failures;                   \
      std::printf("FAILED: ");      \
      std::printf(__VA_ARGS__);     \
      std::printf(" [%s]\n", #cond); \
    }                               \
  } while (0)

// Steps with a narrowband that the fake kernels still have to give.
int nb_steps = 1 << 30;
int sms = 152;
int fim_launches = 0;  // captured or enqueued
int ctas[8] = {};  // resident CTAs of each FIM setting; 0: no two-copies kernel

void begin_words(int* c) {
  c[CTL_STOP] = c[CTL_CHAIN] && (c[CTL_NB] == 0 || c[CTL_CAP] || c[CTL_ERR]) ? 1 : 0;
  if (c[CTL_STOP]) return;
  c[CTL_NB] = c[CTL_BODIES] = c[CTL_CAP] = c[CTL_ERR] = 0;
  c[CTL_BASE] = c[CTL_ITER];
  c[CTL_ITER] += 2;
}
void step_words(const DevState& s, int nv) {
  int* c = s.ctl;
  begin_words(c);
  if (c[CTL_STOP]) return;
  c[CTL_ITER] += 12;
  c[CTL_BODIES] = 1;
  s.cell[0] = make_int4(0, c[CTL_BASE], 0, -1);
  c[CTL_NB] = nb_steps-- > 0 ? 1 : 0;
  if (c[CTL_NB])
    for (int v = 0; v < nv; ++v) s.phi[v] += 1.f;
}

cudaError_t put(cudaStream_t st, fake::Work w) {
  FAKE_CALL("kernel");
  fake::enqueue(fake::of(st), std::move(w));
  return cudaSuccess;
}

KernelSet make_kernels() {
  KernelSet k{};
  k.configure = [](const DevMesh&, const StepParams& sp, Launch& L) {
    L = Launch{};
    L.sms = sms;
    L.fim_ctas = ctas[sp.ctas];
    L.pair_block = L.fim_ctas ? 192 : 0;
    L.warp_grid = L.flat_grid = 1;
    return cudaSuccess;
  };
  k.begin = [](const DevState& s, int, cudaStream_t st) { return put(st, [=] { begin_words(s.ctl); }); };
  k.seed = [](const DevMesh&, const DevState&, const StepParams&, const Launch&, cudaStream_t st) { return put(st, [] {}); };
  k.fim = [](const DevMesh&, const DevState& s, const StepParams&, int off, const Launch&, cudaStream_t st) {
    ++fim_launches;
    return put(st, [=] { if (off == 0 && !s.ctl[CTL_STOP]) s.ctl[CTL_ITER] += 4; });
  };
  k.narrowband = [](const DevMesh& m, const DevState& s, const StepParams&, const Launch&, cudaStream_t st) {
    return put(st, [=] {
      s.ctl[CTL_NB] = nb_steps-- > 0 ? 1 : 0;
      if (s.ctl[CTL_NB]) for (int v = 0; v < m.nv; ++v) s.phi[v] += 1.f;
    });
  };
  k.update = [](const DevMesh&, const DevState&, const StepParams&, int, const Launch&, cudaStream_t st) { return put(st, [] {}); };
  k.unpermute = [](const DevMesh& m, const float* phi, int first, int n, float* out, const int* ctl, const Launch&, cudaStream_t st) {
    return put(st, [=] {
      if (ctl && (ctl[CTL_STOP] || ctl[CTL_NB] == 0)) return;
      for (int o = 0; o < n; ++o) out[o] = phi[m.ipermute[first + o]];
    });
  };
  k.permute = [](const DevMesh& m, const float* in, float* out, const Launch&, cudaStream_t st) {
    return put(st, [=] { for (int o = 0; o < m.nv; ++o) out[m.ipermute[o]] = in[o]; });
  };
  k.geometry = [](const DevMesh&, float4*, float4*, const Launch&, cudaStream_t st) { return put(st, [] {}); };
  return k;
}

// Pairs of triangles (dim 2) or tetrahedra, one patch each.
Layout make_layout(int dim, int n) {
  Layout L;
  std::vector<float> xyz;
  std::vector<int> elems, npart;
  for (int k = 0; k < n; ++k) {
    const float x = 2.f * k;
    const float p[12] = {x, 0, 0, x + 1, 0, 0, x, 1, 0, dim == 2 ? x + 1 : x, dim == 2 ? 1.f : 0.f, dim == 2 ? 0.f : 1.f};
    xyz.insert(xyz.end(), p, p + 12);
    for (int v : dim == 2 ? std::vector<int>{0, 1, 2, 1, 3, 2} : std::vector<int>{0, 1, 2, 3}) elems.push_back(4 * k + v);
    npart.insert(npart.end(), 4, k);
  }
  const std::string r = build_layout(dim, 4 * n, xyz.data(), dim == 2 ? 2 * n : n, elems.data(), npart.data(), n, L);
  CHECK(r.empty(), "layout: %s", r.c_str());
  return L;
}

struct Rig {
  Layout L;
  std::unique_ptr<Solver> s{new Solver()};
  std::vector<float> phi;
  explicit Rig(const SolverConfig& cfg, int dim = 3, int n = 1) : L(make_layout(dim, n)), phi(4 * n, 1.f) {
    fake::st.fail_at = -1;
    const std::string r = s->init(L, cfg, nullptr);
    CHECK(r.empty(), "init: %s", r.c_str());
    Solver* p = s.get();
    fake::st.step = [p] { step_words(p->s_, p->m_.nv); };
    CHECK(s->set_phi(phi.data()).empty(), "set_phi");
  }
};

// Whichever runtime call of an entry point fails: nothing that it enqueued is
// left in flight when it returns, and the handle's next step is a step.
void errors() {
  struct Entry { const char* name; int graph, pageable; std::function<std::string(Solver&, float*)> f; };
  const int n = 4;
  const int seed[1] = {1};
  const float value[1] = {0.f};
  std::vector<Entry> entries;
  for (int graph : {1, 0})
    for (int pageable : {1, 0}) {
      entries.push_back({"run with history", graph, pageable, [=](Solver& s, float* b) { int d; return s.run(5, b, &d); }});
      entries.push_back({"run", graph, pageable, [=](Solver& s, float*) { int d; return s.run(5, nullptr, &d); }});
      entries.push_back({"step_host", graph, pageable, [=](Solver& s, float* b) { return s.step_host(b, b + n); }});
      entries.push_back({"set_phi", graph, pageable, [=](Solver& s, float* b) { return s.set_phi(b); }});
      entries.push_back({"get_phi", graph, pageable, [=](Solver& s, float* b) { return s.get_phi(b); }});
      entries.push_back({"eikonal", graph, pageable, [=](Solver& s, float* b) { return s.eikonal(seed, value, 1, b); }});
    }
  for (const Entry& e : entries) {
    int failed = 0;
    for (int k = 0;; ++k) {
      SolverConfig cfg;
      cfg.use_graph = e.graph;
      fake::st.pageable = e.pageable;
      nb_steps = 1 << 30;
      Rig rig(cfg);
      std::vector<float> buf(64, 0.f);
      nb_steps = 3;  // a run of five steps ends after three
      fake::st.calls = 0;
      fake::st.fail_at = k;
      fake::st.failed.clear();
      const std::string r = e.f(*rig.s, buf.data());
      fake::st.fail_at = -1;
      if (fake::st.failed.empty()) break;  // every call of it has failed once
      ++failed;
      // a failed wait leaves what it waited for; elapsed times are not results
      if (fake::st.failed != "cudaStreamSynchronize" && !r.empty())
        CHECK(fake::st.stream->queue.empty(), "%s (graph %d, pageable %d): work in flight after %s failed at call %d", e.name,
              e.graph, e.pageable, fake::st.failed.c_str(), k);
      fake::drain(fake::st.stream);
      // the narrowband was empty at the end: a step that still takes itself
      // for a part of the run would do nothing
      nb_steps = 1 << 30;
      rig.s->s_.ctl[CTL_NB] = 0;
      bool empty = true;
      const std::string q = rig.s->one_step(&empty);
      CHECK(q.empty() && !empty, "%s (graph %d, pageable %d): next step after %s failed at call %d: %s", e.name, e.graph,
            e.pageable, fake::st.failed.c_str(), k, q.c_str());
    }
    CHECK(failed > 1, "%s: only %d calls", e.name, failed);
  }
}
// Counted iterations, whatever the order of CTA 0 (which counts the previous
// iteration when it starts) and of the other CTAs' ends in a launch: every
// pattern of eight iterations that visit a patch or not, with CTA 0 first or
// last in each launch, and the count at body ends of four.
void iterations() {
  for (int visits = 0; visits < 256; ++visits)
    for (int late = 0; late < 256; ++late)
      for (int persistent = 0; persistent < 2; ++persistent) {
        int ctl[CTL_WORDS] = {}, want = 0;
        const int t0 = 2;
        for (int i = 0; i < 8; ++i) {
          const int t = t0 + i;
          const bool v = (visits >> i) & 1, last = (late >> i) & 1, first = !persistent && i % 4 == 0;
          want += v;
          if (last && v) *visited_word(ctl, t) = 1;
          if (!first) take_iteration(ctl, t - 1);
          if (!last && v) *visited_word(ctl, t) = 1;
          if (persistent ? i == 7 : i % 4 == 3) take_iteration(ctl, t);
        }
        CHECK(ctl[CTL_ITERS] == want, "visits %02x, late %02x, persistent %d: %d iterations instead of %d", visits, late,
              persistent, ctl[CTL_ITERS], want);
        if (failures > 5) return;
      }
}
// The distances of a run's last step stay readable, wherever the stamps
// restart within the run (a new handle's do after a few steps).
void restarts() {
  for (int n = 1; n < 9; ++n)
    for (int extra = 0; extra < 4; ++extra) {
      fake::st.pageable = 1;
      nb_steps = 1 << 30;
      Rig rig(SolverConfig{});
      nb_steps = n;
      int done = -1;
      const std::string r = rig.s->run(n + extra, nullptr, &done);
      CHECK(r.empty() && done == n, "run of %d of %d steps: %d done, %s", n, n + extra, done, r.c_str());
      const DevState& d = rig.s->s_;
      CHECK(d.cell[0].y == d.ctl[CTL_BASE], "run of %d of %d steps: distances cleared", n, n + extra);
    }
}
// The FIM setting: a caller's own stays; the default is 5, or 6 where that lets
// one more CTA reside on a mesh of at least 100 patches per SM.
void settings() {
  struct Case { int setting, dim, patches, five, six, exact, persistent, prec, want; } cases[] = {
      {0, 3, 100, 5, 6, 0, 0, 0, 6}, {0, 3, 100, 6, 7, 0, 0, 0, 6}, {0, 3, 100, 5, 5, 0, 0, 0, 5},
      {0, 3, 100, 6, 6, 0, 0, 0, 5}, {0, 3, 99, 5, 6, 0, 0, 0, 5},  {0, 3, 100, 5, 6, 1, 0, 0, 5},
      {0, 3, 100, 5, 6, 0, 1, 0, 5}, {0, 3, 100, 5, 6, 0, 0, 1, 5}, {0, 3, 100, 0, 0, 0, 0, 0, 5},
      {5, 3, 100, 5, 6, 0, 0, 0, 5}, {6, 3, 100, 5, 5, 0, 0, 0, 6}, {7, 3, 100, 5, 6, 0, 0, 0, 7},
      {2, 3, 100, 5, 6, 0, 0, 0, 2}, {9, 3, 100, 5, 6, 0, 0, 0, 5}, {0, 2, 100, 0, 0, 0, 0, 0, 5},
  };
  sms = 1;
  for (const Case& c : cases) {
    std::fill(ctas, ctas + 8, 0);
    ctas[5] = c.five;
    ctas[6] = c.six;
    SolverConfig cfg;
    cfg.fim_ctas = c.setting;
    cfg.bit_exact = c.exact;
    cfg.persistent = c.persistent;
    cfg.fp64_flagged = c.prec;
    Rig rig(cfg, c.dim, c.patches);
    CHECK(rig.s->sp_.ctas == c.want && rig.s->L_.fim_ctas == ctas[c.want],
          "setting %d, dim %d, %d patches, %d and %d CTAs, exact %d, persistent %d, precision %d: %d instead of %d", c.setting,
          c.dim, c.patches, c.five, c.six, c.exact, c.persistent, c.prec, rig.s->sp_.ctas, c.want);
  }
  std::fill(ctas, ctas + 8, 0);
  sms = 152;
}
// The step graph's iterations before its loop: the body's length decides their
// number only up to the next whole body.
void first_iterations() {
  for (int dim : {2, 3})
    for (int chunk : {0, 1, 2, 3, 4, 6, 8, 10, 16, 32, 100}) {
      SolverConfig cfg;
      cfg.graph_chunk = chunk;
      fim_launches = 0;
      Rig rig(cfg, dim);
      const int body = std::max(chunk + (chunk & 1), 2), least = dim == 3 ? 12 : 8;
      const int want = (least + body - 1) / body * body;
      CHECK(fim_launches == want + body, "dim %d, graph_chunk %d: %d launches before the loop instead of %d", dim, chunk,
            fim_launches - body, want);
    }
}
}  // namespace

const KernelSet& kernels_fast() { static const KernelSet k = make_kernels(); return k; }
const KernelSet& kernels_exact() { return kernels_fast(); }
namespace mlp {
__global__ void k_features(int, const int*, const int*, const int*, const int*, const float*, int, const float*, float, const float*,
                           __nv_bfloat16*) {}
std::string Net::forward_dev(const __nv_bfloat16*, int, const int*, int, float*, cudaStream_t) { return ""; }
std::string Net::append_pairs(const __nv_bfloat16*, const float*, const int*, int, cudaStream_t, long long*) { return ""; }
}  // namespace mlp
}  // namespace lsgb

int main(int argc, char** argv) {
  for (int i = 1; i < argc; ++i) {
    const std::string a = argv[i];
    if (a == "errors") lsgb::errors();
    else if (a == "iterations") lsgb::iterations();
    else if (a == "restarts") lsgb::restarts();
    else if (a == "settings") lsgb::settings();
    else if (a == "first_iterations") lsgb::first_iterations();
    else { std::printf("unknown check %s\n", a.c_str()); return 99; }
  }
  std::printf("%d failures\n", lsgb::failures);
  return lsgb::failures ? 1 : 0;
}
