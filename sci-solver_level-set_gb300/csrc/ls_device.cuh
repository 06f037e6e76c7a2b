// ls_device.cuh -- device-side local eikonal solvers and shared types.
//
// The tet and triangle local solvers evaluate the same closed-form updates
// as GPUTUM Level-Set's localSolverTet1Levelset
// (src/core3d/include/redistance_kernels3d.h:124-285) and localSolverTri
// (src/core2d/include/redistance_kernels.h:287-334): three face (edge-pair)
// quadratics plus the interior quadratic for a tet, the two-root law-of-
// cosines update for a triangle, each candidate accepted only when its
// barycentric coordinates lie in [0,1].  tet_solve keeps the formulas term
// for term, so that the bit-exact build reproduces the reference's FP32
// arithmetic (the reference's `/ (2.0 * p)` divisions, evaluated there in
// double and rounded to float, give the same correctly rounded float
// quotient as an IEEE float division).  The fast build's tet sweeps use
// tet_solve_wave instead: the same candidates and validity rules, with the
// stationary points found without the reference's cancelling discriminants,
// so that FP32 stays at the reference's FP64 result.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace lsgb {

// Device view of the patch layout.
struct DevMesh {
  int dim, nv, nparts;
  long long full;
  const int* vert_off;       // nparts+1
  const int* ele_off;        // nparts+1
  const int* ghost_off;      // nparts+1
  const int* ghost_ids;      // ghosts (new vertex ids)
  const ushort4* conn;       // full: slab-local vertex indices
  const float* lc;           // SoA [6|3][full] local coordinates
  const float* sig;          // SoA [3][full] per-copy velocity (2D: projected, 2 rows)
  const int* vslot_off;      // nv+1
  const uint16_t* vslot;     // owned-vertex slots (copy_local*4 + k)
  // per copy: corners beyond the reference's per-vertex slot limit, set only
  // with the reference's semantics on meshes that have such corners (null
  // otherwise): they stay private to their copy in the FIM sweep and are
  // left out of the update's sums (Layout::slot_capped)
  const uint8_t* capped;
  int slot_cap;              // the limit: 32 (tetrahedra) or 16 (triangles)
  const int* padj_off;       // nparts+1
  const int* padj;           // patch adjacency
  const float* xyz;          // SoA [3][nv]
  const int* ipermute;       // old -> new vertex id
  const int* patch_bytes;    // per patch: algorithmic bytes of one FIM visit
  // batches of independent meshes: mesh of each patch and per-mesh
  // parameters {bandwidth in the FIM frame, FIM frame scale, dt, curvature
  // coefficient}; null for a single mesh (StepParams hold them)
  const int* patch_mesh;
  const float4* mesh_par;
  // per copy, precomputed once per mesh for the two-copies-per-thread tet
  // sweep (null otherwise): the 11 metric terms of copy_metric as three
  // float4 (geo_m[3c .. 3c+2], last lane a second copy of CDCD) and the
  // heights of A, B, C, D over their opposite faces (geo_h[c]); a patch's
  // copies are contiguous, so its records are two contiguous slabs, staged
  // by bulk asynchronous copies
  const float4* geo_m;
  const float4* geo_h;
};

// Bandwidth (FIM frame), FIM frame scale, dt and curvature coefficient of
// patch p.
struct PatchPar {
  float bw, scale, dt, cc;
};

// FIM distance of a vertex: two stamped values {v0, t0, v1, t1} (float bits
// and iteration stamp).  A visit in iteration t writes its results with stamp
// t over the older of the two, while every other patch of that iteration
// reads the newest value with a stamp below t: the values of the previous
// iteration stay readable until the next one, so that no copy-back pass
// separates the iterations.  Stamps grow from step to step; a step's first
// stamp (its base) marks its seeds, which are written to {v0, t0} and never
// visited, and a vertex with no stamp of this step holds LARGENUM (no reset
// pass either).
typedef int4 DtCell;

__device__ __forceinline__ float dt_before(const DtCell& c, int t, int base, float LN) {
  const int a = c.y < t ? c.y : -1, b = c.w < t ? c.w : -1;
  const bool second = b > a;
  return (second ? b : a) >= base ? __int_as_float(second ? c.z : c.x) : LN;
}
__device__ __forceinline__ bool dt_is_seed(const DtCell& c, int base) { return c.y == base; }
constexpr int kStampMax = 0x7fffffff;

// Step control words (DevState::ctl, one int each).
enum {
  CTL_VISITS = 0,   // [3] patches to visit in list i (iteration t uses list t % 3)
  CTL_NB = 3,       // narrowband patches
  CTL_CANDS = 4,    // [3] candidates to check in list i
  CTL_NB_PREV = 7,  // previous step's narrowband patches (0: the seed search takes every patch)
  CTL_BODIES = 8,   // FIM loop bodies run this step
  CTL_CAP = 9,      // the iteration cap was hit
  CTL_NB_VALID = 10,  // the narrowband list belongs to the current phi
  CTL_ERR = 11,     // a wait of a FIM kernel timed out and the launch was abandoned (1: grid
                    // barrier of the persistent kernel, 2: geometry slab copy)
  CTL_ITER = 12,    // stamp of the first iteration of the next loop body
  CTL_BASE = 13,    // base stamp of the step
  CTL_ITERS = 14,   // iterations of this step that visited a patch
  // a run enqueues a step before it knows how the previous one ended (host-set
  // CTL_CHAIN, 0 outside a run's later steps): if that one ran out of
  // narrowband or failed, the step finds CTL_STOP set and does nothing
  CTL_CHAIN = 15,
  CTL_STOP = 16,
  CTL_VISITED = 17,  // [3] an iteration visited a patch (visited_word)
  CTL_ABOVE = 20,    // a seed of this step lies above LARGENUM
  CTL_WORDS = 32
};
// Stamps restart (every stamped array cleared) between steps once they pass
// this limit; a new handle starts a few steps below it.
constexpr int kStampLimit = 1 << 29;

// Device step state.
struct DevState {
  float* phi;
  float* phi_rd;    // phi after the redistance, before the update
  DtCell* cell;     // per vertex: FIM distance
  int* slot;        // per patch: the half of its vertices' cells that its last visit wrote
  // per patch, stamps: 2t = in the list of iteration t and not done with it,
  // 2t + 1 = done with iteration t and not in the next list
  int* pend;
  int* reach;       // per patch: last iteration that left it converged with its minimum inside the band
  int* lists;       // [3][nparts]: visits from the front, candidates from the back
  int* nblist;      // narrowband patches
  int* ctl;         // step control words (CTL_*)
  unsigned long long* stats;  // [0] visits [1] checks [2] nb verts [3] nb patch verts [4] nb patches [5] fim iters [6] flagged copies solved [7] FIM slab bytes [8] visits run by checks
  int* sched;       // dynamic patch assignment of the FIM kernels: next list entry; zero between
                    // launches (the launch's last draw resets it)
  unsigned* gbar;   // persistent FIM kernel (kGridBarrierWords, zeroed per step): [0] grid-barrier
                    // arrivals since the launch started, [2 + smid] CTAs on SM smid
};
constexpr int kGridBarrierWords = 2 + 1024;

// An iteration counts if it visited a patch: its CTAs mark the iteration's own
// word, which one thread takes when the next iteration starts or at the end of
// a loop body.  The next iteration's CTAs, some done before that thread has
// looked, mark another word.  (The word goes with the list that the iteration
// makes, whose counters the sweep kernels have at hand: kept for t % 3, the
// stamp cost the 56-register kernels two spills.)
__host__ __device__ __forceinline__ int* visited_word(int* ctl, int t) { return ctl + CTL_VISITED + (t + 1) % 3; }
__host__ __device__ __forceinline__ bool take_iteration(int* ctl, int t) {
  volatile int* w = visited_word(ctl, t);
  if (!*w) return false;
  *w = 0;
  ctl[CTL_ITERS] += 1;
  return true;
}
__device__ __forceinline__ void count_iteration(int* ctl, unsigned long long* stats, int t) {
  if (take_iteration(ctl, t)) atomicAdd(&stats[5], 1ull);
}

// Learned warm start / training-pair collection buffers (null when off).
struct DevLearn {
  int* vlist;     // warm-set vertices (owned vertices of the previous narrowband patches)
  int* cnt;       // [0] warm-set size, [1] unsupported vertices reset, [2] vertices moved beyond
                  // the tolerance, [3] patches re-activated by the support check
  float* pred;    // network output per warm-set vertex (signed distance / h)
  float* warm;    // per vertex: warm-start value in the FIM frame
  float* target;  // collection: signed distance / h after the redistance, per warm-set vertex
  const float* vinv_h;  // batches: per vertex, 1 / its mesh's FIM length unit (null for one mesh)
};

struct StepParams {
  float largenum;
  float bandwidth;   // in the FIM frame (divided by scale)
  float scale;       // FIM frame length unit (1 with the reference's semantics)
  float tau;         // precision form: discriminant cancellation threshold
  int xdiv;          // interior division in double (bit-exact build, reference semantics)
  int ctas;          // FIM CTAs per SM for patches of up to 384 copies (2, 3, 4; 5, 6: two copies per thread, 7: the same kernel with one)
  float tol;       // convergence threshold on oldT - newT
  float eps_h;     // denominator offset of the interior tet update
  double eps_h64;
  float dt;
  float curv_coeff;
  int niter;       // sweeps per visit
  int ref_compat;
  int update_kind; // 0 advect, 1 curvature
  int lvp, lgp, lep;
  int max_fim_iters;  // persistent FIM kernel: iteration cap of one step
  int spin_limit;     // polls of one grid-barrier wait of the persistent FIM kernel before it gives up;
                      // < 0: every wait of the FIM kernels (grid barrier, geometry slab copy) gives up
                      // at its first check (the setting that tests the timeout paths)
  int wide;           // fast build, tetrahedra: the mesh has edges below 1e-7 FIM lengths (tet_solve_wave's WIDE)
};

__device__ __forceinline__ PatchPar patch_par(const DevMesh& m, const StepParams& sp, int p) {
  if (m.patch_mesh) {
    const float4 q = __ldg(&m.mesh_par[__ldg(&m.patch_mesh[p])]);
    return PatchPar{q.x, q.y, q.z, q.w};
  }
  return PatchPar{sp.bandwidth, sp.scale, sp.dt, sp.curv_coeff};
}


template <typename R>
__device__ __forceinline__ R rmin(R a, R b) { return fmin(a, b); }
template <typename R>
__device__ __forceinline__ R rmax(R a, R b) { return fmax(a, b); }
template <>
__device__ __forceinline__ float rmin<float>(float a, float b) { return fminf(a, b); }

// Unit-speed tet update of vertex D from face ABC given the metric terms of
// the edge vectors AC, BC, CD (R = float or double).  Every expression keeps
// the reference's operand order and association, so that a build without
// FMA contraction reproduces the reference arithmetic bit for bit.
//
// XDIV: the reference evaluates the interior barycentric coordinate
// `(s * l1 + t) / (h + SMALLNUM)` with a double SMALLNUM, i.e. in double;
// XDIV = true reproduces that (used only by the bit-exact build with the
// reference's semantics), XDIV = false divides in R.
//
// `tau` > 0 turns on the conditioning check of the precision form: `ill` is
// set when a discriminant q^2 - 4pr cancels, |q^2 - 4pr| <= tau (q^2 + |4pr|),
// i.e. when FP32 has lost about log2(1/tau) bits of it.
// Roots of p x^2 + q x + r given sq = sqrt(q^2 - 4pr).  The reference's
// form (-q +- sq) / 2p, or, for the precision form, the cancellation-free
// pair s / p, r / s with s = -(q + sign(q) sq) / 2 (the same two roots; also
// right when p = 0).
template <typename R, bool STABLE>
__device__ __forceinline__ void roots(R p, R q, R r, R sq, R& ra, R& rb) {
  if (STABLE) {
    const R sh = -(q + (q >= R(0) ? sq : -sq)) * R(0.5);
    ra = sh / p;
    rb = r / sh;
  } else {
    ra = (-q + sq) / (R(2) * p);
    rb = (-q - sq) / (R(2) * p);
  }
}

template <typename R, bool XDIV, bool CHK = true, bool LB = false>
__device__ __forceinline__ R tet_solve(R TA, R TB, R TC, R ACAC, R ACBC, R ACCD, R BCBC, R BCCD,
                                       R CDCD, R eps_h, double eps_h64, R LN, R tau, bool& ill,
                                       R cutoff = R(0)) {
  if (TA >= LN && TB >= LN && TC >= LN) return LN;
  // precision form (CHK): a quadratic is flagged only when all its arrival
  // times are below LARGENUM -- with one at LARGENUM its candidates lie at or
  // above the edge candidates computed separately (equal values, e.g. two
  // LARGENUMs, make the discriminant vanish identically)
  if (CHK || LB) {
    // precision form: a solve whose candidates cannot fall below `cutoff`
    // (the target's current value) is skipped -- every candidate is at
    // least min(TA, TB, TC) plus D's height over the plane ABC (Gram
    // determinants of AC, BC, CD; taken x 0.999)
    const R det2 = ACAC * BCBC - ACBC * ACBC;
    const R det3 = ACAC * (BCBC * CDCD - BCCD * BCCD) - ACBC * (ACBC * CDCD - BCCD * ACCD) +
                   ACCD * (ACBC * BCCD - BCBC * ACCD);
    const R lb = rmin(rmin(TA, TB), TC) + R(0.999) * sqrt(fmax(det3 / det2, R(0)));
    if (lb >= cutoff) return LN;
  }
  const R two = R(2), four = R(4), one = R(1), zero = R(0);
  R p, q, r, lambda1, lambda2, lambda3, delta, TE;
  R FaceTAC = LN, FaceTAB = LN, FaceTBC = LN, TD = LN;
  const R TAC = TC - TA, TBC = TC - TB, TAB = TB - TA;

  // face BC (lambda1 = 0)
  p = BCBC * TBC * TBC - BCBC * BCBC;
  q = (BCCD + BCCD) * TBC * TBC - two * BCBC * BCCD;
  r = TBC * TBC * CDCD - BCCD * BCCD;
  delta = q * q - four * p * r;
  if (CHK && rmax(TB, TC) < LN) ill |= (fabs(delta) <= tau * (q * q + fabs(four * p * r)));
  if (delta >= zero) {
    const R sq = sqrt(delta);
    R ra, rb;
    roots<R, CHK>(p, q, r, sq, ra, rb);
    lambda1 = zero;
    lambda2 = ra;
    lambda3 = one - lambda1 - lambda2;
    if (lambda2 >= zero && lambda2 <= one) {
      TE = TB * lambda2 + TC * lambda3;
      FaceTBC = rmin(FaceTBC, TE + sqrt((lambda2 * BCBC + BCCD) * lambda2 + (lambda2 * BCCD + CDCD)));
    }
    lambda2 = rb;
    lambda3 = one - lambda1 - lambda2;
    if (lambda2 >= zero && lambda2 <= one) {
      TE = TB * lambda2 + TC * lambda3;
      FaceTBC = rmin(FaceTBC, TE + sqrt((lambda2 * BCBC + BCCD) * lambda2 + (lambda2 * BCCD + CDCD)));
    }
  }
  FaceTBC = rmin(FaceTBC, rmin(TB + sqrt((BCBC + BCCD) + (BCCD + CDCD)), TC + sqrt(CDCD)));

  // face AB (lambda3 = 0)
  const R gammax = ACAC - ACBC, gammay = ACBC - BCBC, gammaz = ACCD - BCCD;
  p = (TAB * TAB * ACAC - gammax * gammax) + (BCBC * TAB * TAB - gammay * gammay) -
      ((ACBC + ACBC) * TAB * TAB - two * gammax * gammay);
  q = -(BCBC * TAB * TAB - gammay * gammay) * two + ((ACBC + ACBC) * TAB * TAB - two * gammax * gammay) +
      ((ACCD + ACCD) * TAB * TAB - two * gammax * gammaz) - ((BCCD + BCCD) * TAB * TAB - two * gammay * gammaz);
  r = (TAB * TAB * BCBC - gammay * gammay) + ((BCCD + BCCD) * TAB * TAB - two * gammay * gammaz) +
      (TAB * TAB * CDCD - gammaz * gammaz);
  delta = q * q - four * p * r;
  if (CHK && rmax(TA, TB) < LN) ill |= (fabs(delta) <= tau * (q * q + fabs(four * p * r)));
  if (delta >= zero) {
    const R sq = sqrt(delta);
    R ra, rb;
    roots<R, CHK>(p, q, r, sq, ra, rb);
#pragma unroll
    for (int sgn = 0; sgn < 2; ++sgn) {
      lambda1 = sgn ? rb : ra;
      lambda2 = one - lambda1;
      if (lambda1 >= zero && lambda1 <= one) {
        TE = TA * lambda1 + TB * lambda2;
        FaceTAB = rmin(FaceTAB, TE + sqrt((lambda1 * ACAC + lambda2 * ACBC + ACCD) * lambda1 +
                                          (lambda1 * ACBC + lambda2 * BCBC + BCCD) * lambda2 +
                                          (lambda1 * ACCD + lambda2 * BCCD + CDCD)));
      }
    }
  }
  FaceTAB = rmin(FaceTAB, rmin(TB + sqrt((BCBC + BCCD) + (BCCD + CDCD)), TA + sqrt((ACAC + ACCD) + (ACCD + CDCD))));

  // face AC (lambda2 = 0)
  p = ACAC * TAC * TAC - ACAC * ACAC;
  q = (ACCD + ACCD) * TAC * TAC - two * ACAC * ACCD;
  r = TAC * TAC * CDCD - ACCD * ACCD;
  delta = q * q - four * p * r;
  if (CHK && rmax(TA, TC) < LN) ill |= (fabs(delta) <= tau * (q * q + fabs(four * p * r)));
  if (delta >= zero) {
    const R sq = sqrt(delta);
    R ra, rb;
    roots<R, CHK>(p, q, r, sq, ra, rb);
#pragma unroll
    for (int sgn = 0; sgn < 2; ++sgn) {
      lambda1 = sgn ? rb : ra;
      lambda3 = one - lambda1 - zero;
      if (lambda1 >= zero && lambda1 <= one) {
        TE = TA * lambda1 + TC * lambda3;
        FaceTAC = rmin(FaceTAC, TE + sqrt((lambda1 * ACAC + ACCD) * lambda1 + (lambda1 * ACCD + CDCD)));
      }
    }
  }
  FaceTAC = rmin(FaceTAC, rmin(TA + sqrt((ACAC + ACCD) + (ACCD + CDCD)), TC + sqrt(CDCD)));

  // interior of face ABC
  const R s = TAC * ACBC - TBC * ACAC;
  const R t = TAC * BCCD - TBC * ACCD;
  const R h = -(TAC * BCBC - TBC * ACBC);
  p = (TAC * TAC * ACAC - ACAC * ACAC) * h * h + (BCBC * TAC * TAC - ACBC * ACBC) * s * s +
      ((ACBC + ACBC) * TAC * TAC - two * ACAC * ACBC) * s * h;
  q = (BCBC * TAC * TAC - ACBC * ACBC) * two * s * t + ((ACBC + ACBC) * TAC * TAC - two * ACAC * ACBC) * t * h +
      ((ACCD + ACCD) * TAC * TAC - two * ACAC * ACCD) * h * h + ((BCCD + BCCD) * TAC * TAC - two * ACBC * ACCD) * s * h;
  r = (TAC * TAC * BCBC - ACBC * ACBC) * t * t + ((BCCD + BCCD) * TAC * TAC - two * ACBC * ACCD) * t * h +
      (TAC * TAC * CDCD - ACCD * ACCD) * h * h;
  delta = q * q - four * p * r;
  if (CHK && rmax(rmax(TA, TB), TC) < LN) ill |= (fabs(delta) <= tau * (q * q + fabs(four * p * r)));
  if (delta >= zero) {
    const R sq = sqrt(delta);
    R ra, rb;
    roots<R, CHK>(p, q, r, sq, ra, rb);
#pragma unroll
    for (int sgn = 0; sgn < 2; ++sgn) {
      lambda1 = sgn ? rb : ra;
      if (XDIV)
        lambda2 = (R)((double)(s * lambda1 + t) / ((double)h + eps_h64));
      else
        lambda2 = (s * lambda1 + t) / (h + eps_h);
      lambda3 = one - lambda1 - lambda2;
      if (lambda1 >= zero && lambda1 <= one && lambda2 >= zero && lambda2 <= one && lambda3 >= zero &&
          lambda3 <= one) {
        TE = TA * lambda1 + TB * lambda2 + TC * lambda3;
        TD = rmin(TD, TE + sqrt((lambda1 * ACAC + lambda2 * ACBC + ACCD) * lambda1 +
                                (lambda1 * ACBC + lambda2 * BCBC + BCCD) * lambda2 +
                                (lambda1 * ACCD + lambda2 * BCCD + CDCD)));
      }
    }
  }
  TD = rmin(TD, rmin(FaceTBC, rmin(FaceTAB, FaceTAC)));
  return TD;
}

// The same tet update with predicated candidates instead of branches (fast
// build): every quadratic's roots and candidate distances are evaluated and
// the invalid ones masked, so the lanes of a warp stay converged through the
// solve.  A negative discriminant gives NaN roots, which fail every range
// test, and a candidate whose distance is not a number is dropped by fminf,
// so neither needs a guard.  Valid candidates use the same expressions as
// tet_solve; CHK adds
// the precision form's flags and cancellation-free roots (as tet_solve with
// CHK, without its lower-bound skip, which the caller has applied).
template <bool CHK = false>
__device__ __forceinline__ float tet_solve_pred(float TA, float TB, float TC, float ACAC, float ACBC, float ACCD,
                                                float BCBC, float BCCD, float CDCD, float eps_h, float LN,
                                                float tau = 0.f, bool* ill = nullptr) {
  if (TA >= LN && TB >= LN && TC >= LN) return LN;
  float FaceTAC = LN, FaceTAB = LN, FaceTBC = LN, TD = LN;
  const float TAC = TC - TA, TBC = TC - TB, TAB = TB - TA;
  float p, q, r, delta;
  // face BC (lambda1 = 0)
  p = BCBC * TBC * TBC - BCBC * BCBC;
  q = (BCCD + BCCD) * TBC * TBC - 2.f * BCBC * BCCD;
  r = TBC * TBC * CDCD - BCCD * BCCD;
  delta = q * q - 4.f * p * r;
  if (CHK && fmaxf(TB, TC) < LN && fabsf(delta) <= tau * (q * q + fabsf(4.f * p * r))) *ill = true;
  {
    const float sq = sqrtf(delta);  // NaN when delta < 0: every root test fails
    float ra, rb;
    roots<float, CHK>(p, q, r, sq, ra, rb);
#pragma unroll
    for (int sgn = 0; sgn < 2; ++sgn) {
      const float l2 = sgn ? rb : ra;
      const float l3 = 1.f - l2;
      const float c = TB * l2 + TC * l3 + sqrtf((l2 * BCBC + BCCD) * l2 + (l2 * BCCD + CDCD));
      if (l2 >= 0.f && l2 <= 1.f) FaceTBC = fminf(FaceTBC, c);
    }
  }
  FaceTBC = fminf(FaceTBC, fminf(TB + sqrtf((BCBC + BCCD) + (BCCD + CDCD)), TC + sqrtf(CDCD)));
  // face AB (lambda3 = 0)
  const float gammax = ACAC - ACBC, gammay = ACBC - BCBC, gammaz = ACCD - BCCD;
  p = (TAB * TAB * ACAC - gammax * gammax) + (BCBC * TAB * TAB - gammay * gammay) -
      ((ACBC + ACBC) * TAB * TAB - 2.f * gammax * gammay);
  q = -(BCBC * TAB * TAB - gammay * gammay) * 2.f + ((ACBC + ACBC) * TAB * TAB - 2.f * gammax * gammay) +
      ((ACCD + ACCD) * TAB * TAB - 2.f * gammax * gammaz) - ((BCCD + BCCD) * TAB * TAB - 2.f * gammay * gammaz);
  r = (TAB * TAB * BCBC - gammay * gammay) + ((BCCD + BCCD) * TAB * TAB - 2.f * gammay * gammaz) +
      (TAB * TAB * CDCD - gammaz * gammaz);
  delta = q * q - 4.f * p * r;
  if (CHK && fmaxf(TA, TB) < LN && fabsf(delta) <= tau * (q * q + fabsf(4.f * p * r))) *ill = true;
  {
    const float sq = sqrtf(delta);  // NaN when delta < 0: every root test fails
    float ra, rb;
    roots<float, CHK>(p, q, r, sq, ra, rb);
#pragma unroll
    for (int sgn = 0; sgn < 2; ++sgn) {
      const float l1 = sgn ? rb : ra;
      const float l2 = 1.f - l1;
      const float c = TA * l1 + TB * l2 +
                      sqrtf((l1 * ACAC + l2 * ACBC + ACCD) * l1 + (l1 * ACBC + l2 * BCBC + BCCD) * l2 +
                            (l1 * ACCD + l2 * BCCD + CDCD));
      if (l1 >= 0.f && l1 <= 1.f) FaceTAB = fminf(FaceTAB, c);
    }
  }
  FaceTAB = fminf(FaceTAB, fminf(TB + sqrtf((BCBC + BCCD) + (BCCD + CDCD)), TA + sqrtf((ACAC + ACCD) + (ACCD + CDCD))));
  // face AC (lambda2 = 0)
  p = ACAC * TAC * TAC - ACAC * ACAC;
  q = (ACCD + ACCD) * TAC * TAC - 2.f * ACAC * ACCD;
  r = TAC * TAC * CDCD - ACCD * ACCD;
  delta = q * q - 4.f * p * r;
  if (CHK && fmaxf(TA, TC) < LN && fabsf(delta) <= tau * (q * q + fabsf(4.f * p * r))) *ill = true;
  {
    const float sq = sqrtf(delta);  // NaN when delta < 0: every root test fails
    float ra, rb;
    roots<float, CHK>(p, q, r, sq, ra, rb);
#pragma unroll
    for (int sgn = 0; sgn < 2; ++sgn) {
      const float l1 = sgn ? rb : ra;
      const float l3 = 1.f - l1;
      const float c = TA * l1 + TC * l3 + sqrtf((l1 * ACAC + ACCD) * l1 + (l1 * ACCD + CDCD));
      if (l1 >= 0.f && l1 <= 1.f) FaceTAC = fminf(FaceTAC, c);
    }
  }
  FaceTAC = fminf(FaceTAC, fminf(TA + sqrtf((ACAC + ACCD) + (ACCD + CDCD)), TC + sqrtf(CDCD)));
  // interior of face ABC
  const float s = TAC * ACBC - TBC * ACAC;
  const float t = TAC * BCCD - TBC * ACCD;
  const float h = -(TAC * BCBC - TBC * ACBC);
  p = (TAC * TAC * ACAC - ACAC * ACAC) * h * h + (BCBC * TAC * TAC - ACBC * ACBC) * s * s +
      ((ACBC + ACBC) * TAC * TAC - 2.f * ACAC * ACBC) * s * h;
  q = (BCBC * TAC * TAC - ACBC * ACBC) * 2.f * s * t + ((ACBC + ACBC) * TAC * TAC - 2.f * ACAC * ACBC) * t * h +
      ((ACCD + ACCD) * TAC * TAC - 2.f * ACAC * ACCD) * h * h + ((BCCD + BCCD) * TAC * TAC - 2.f * ACBC * ACCD) * s * h;
  r = (TAC * TAC * BCBC - ACBC * ACBC) * t * t + ((BCCD + BCCD) * TAC * TAC - 2.f * ACBC * ACCD) * t * h +
      (TAC * TAC * CDCD - ACCD * ACCD) * h * h;
  delta = q * q - 4.f * p * r;
  if (CHK && fmaxf(fmaxf(TA, TB), TC) < LN && fabsf(delta) <= tau * (q * q + fabsf(4.f * p * r))) *ill = true;
  {
    const float sq = sqrtf(delta);  // NaN when delta < 0: every root test fails
    float ra, rb;
    roots<float, CHK>(p, q, r, sq, ra, rb);
#pragma unroll
    for (int sgn = 0; sgn < 2; ++sgn) {
      const float l1 = sgn ? rb : ra;
      const float l2 = (s * l1 + t) / (h + eps_h);
      const float l3 = 1.f - l1 - l2;
      const float c = TA * l1 + TB * l2 + TC * l3 +
                      sqrtf((l1 * ACAC + l2 * ACBC + ACCD) * l1 + (l1 * ACBC + l2 * BCBC + BCCD) * l2 +
                            (l1 * ACCD + l2 * BCCD + CDCD));
      if (l1 >= 0.f && l1 <= 1.f && l2 >= 0.f && l2 <= 1.f && l3 >= 0.f && l3 <= 1.f) TD = fminf(TD, c);
    }
  }
  return fminf(TD, fminf(FaceTBC, fminf(FaceTAB, FaceTAC)));
}

// l in [+0, 1] as one unsigned compare of the bits (negative values, -0.0
// and NaN fail).  A candidate rejected for l = -0.0 sits at the side's end
// point, where the edge candidate gives the same value.
__device__ __forceinline__ bool in_unit(float l) { return __float_as_uint(l) <= 0x3f800000u; }

// The same test of three numbers.
__device__ __forceinline__ bool in_unit(float a, float b, float c) {
  return __vimax3_u32(__float_as_uint(a), __float_as_uint(b), __float_as_uint(c)) <= 0x3f800000u;
}

// Tet update of D from the face ABC in FP32 without the quadratics (fast
// build).  It returns the same quantity as tet_solve -- the least T_lin(x) +
// |x - D| over the face, T_lin interpolating TA, TB, TC, with the reference's
// candidates (three edges, three sides, the face interior) and its validity
// rules -- but finds each stationary point from the planar wave that passes
// through the known values instead of from a squared equation.  For a side
// PQ with f = Q - P, w = D - P and u = TQ - TP, the point P + l f with
//   l = (f.w - |f x w| u / sqrt(|f|^2 - u^2)) / |f|^2
// is where the characteristic through D meets the side (none when |u| >=
// |f|), and its distance to D is |f x w| / sqrt(|f|^2 - u^2) (the same
// quantity the reference evaluates at that point, without a square root of
// its own).  For the interior, the in-plane gradient g solves the 2x2 Gram
// system of AC, BC; the characteristic leaves the plane at sqrt(1 - |g|^2),
// so the weight of A is the foot point's first barycentric minus (hD /
// sqrt(1 - |g|^2)) times g's first coefficient (hD: D's height over ABC),
// and the weight of B comes from the reference's own relation l2 = (s l1 +
// t) / (h + eps_h), so that its SMALLNUM offset acts as in the reference; the
// candidate is evaluated at that point as the reference does.  The
// reference's quadratic also has the mirror root (the foot point plus the
// same offset), taken too: where h is small the offset moves the first
// root's point by far more than rounding, and the mirror's point can then be
// the better one.  The reference's discriminants q^2 -
// 4pr vanish analytically whenever two arrival times along a side are equal,
// so in FP32 they come out as rounding noise of either sign (a negative one
// drops the candidate: errors up to ~0.3 h); none of the quantities here
// cancel, and the result stays within ~5e-5 h of the reference's solver run
// in FP64.  Invalid points come out as NaN or out of range and fail the
// range tests.
// Evaluation: sm_100 issues one FP32x2 instruction (add, multiply, fused
// multiply-add, each lane rounded as the scalar operation) for two lanes, so
// some independent halves run as pairs -- edges PX and QX, sides RQ and RP
// (both from R), the two interior roots -- with the square roots, side QP
// and the interior's set-up per lane.  Every multiply-add is written out:
// left to the compiler's contraction, the kernels that inline this solver
// would round differently.  Of a difference of products the first is fused;
// s has its products in the other order than g2's numerator, and the weights
// of T_lin are those of all three vertices: a value's last bit decides range
// tests and the front's last patches, so cheaper forms of these (shared
// numerators, differences to TR: 1 % of the FIM time) were not worth another
// set of bits.
// Arguments: the face's vertices are P, Q, R and the target X; the dot
// products of p = P - R, q = Q - R and x = X - R (PP = p.p, PQ = p.q, ...),
// and hX, X's height over the face.  (tet_solve's ACCD and BCCD are -PX and
// -QX: with all three vectors from R the four solves of a tet only permute
// the products, without signs.)  Not all of TP, TQ, TR are LARGENUM (the
// listings leave those solves out).
__device__ __forceinline__ float2 f2(float a, float b) { return make_float2(a, b); }
// The approximate square root, its reciprocal and the reciprocal.  WIDE keeps
// denormals; without it they are the bare hardware operations: with denormals
// kept, each of the solver's 17 carries a test and a rescaling of its argument
// (same bits for normal arguments and results).  The arguments are squared
// lengths, products of two of them (squared face areas, whose square roots
// are distances: flushed to zero they put vertices on the front that they are
// a length away from) and differences of such products, so the bare form is
// for meshes whose shortest edge is at least 1e-7 in the FIM frame
// (StepParams::wide).
template <bool WIDE>
__device__ __forceinline__ float fast_sqrt(float x) {
  float r;
  if constexpr (WIDE) asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
  else asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
template <bool WIDE>
__device__ __forceinline__ float fast_rsqrt(float x) {
  float r;
  if constexpr (WIDE) asm("rsqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
  else asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
template <bool WIDE>
__device__ __forceinline__ float fast_rcp(float x) {
  float r;
  if constexpr (WIDE) asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
  else asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

template <bool WIDE>
__device__ __forceinline__ float tet_solve_wave(float TP, float TQ, float TR, float PP, float PQ, float PX, float QQ,
                                                float QX, float XX, float hX, float eps_h) {
  // edges PX, QX (lanes x, y) and RX
  const float2 d2 = f2((PP - PX) + (XX - PX), (QQ - QX) + (XX - QX));
  const float2 ed = __fadd2_rn(f2(TP, TQ), f2(fast_sqrt<WIDE>(d2.x), fast_sqrt<WIDE>(d2.y)));
  float best = fminf(fminf(ed.x, ed.y), TR + fast_sqrt<WIDE>(XX));
  const float up = TP - TR, uq = TQ - TR;
  // sides: y = lam F + (1 - lam) B with |F - B|^2 = ff, (F - B).(X - B) = fw,
  // |X - B|^2 = ww and u = T_F - T_B.  At the stationary point of
  // T_B + lam u + |y - X| the distance is r = sqrt(ff ww - fw^2) /
  // sqrt(ff - u^2) (no root when ff <= u^2: the rsqrt is then NaN or inf and
  // the candidate is rejected) and lam = (fw - u r) / ff.
  {  // sides RQ (lane x) and RP (lane y), both from R
    const float2 G = f2(fmaf(QQ, XX, -__fmul_rn(QX, QX)), fmaf(PP, XX, -__fmul_rn(PX, PX)));  // ff ww - fw^2
    const float2 q = f2(fmaf(-uq, uq, QQ), fmaf(-up, up, PP));                                // ff - u^2
    const float2 r = __fmul2_rn(f2(fast_sqrt<WIDE>(G.x), fast_sqrt<WIDE>(G.y)), f2(fast_rsqrt<WIDE>(q.x), fast_rsqrt<WIDE>(q.y)));
    const float lx = __fmul_rn(fmaf(-uq, r.x, QX), fast_rcp<WIDE>(QQ)), ly = __fmul_rn(fmaf(-up, r.y, PX), fast_rcp<WIDE>(PP));
    const float2 c = __fadd2_rn(__ffma2_rn(f2(lx, ly), f2(uq, up), f2(TR, TR)), r);
    if (in_unit(lx)) best = fminf(best, c.x);
    if (in_unit(ly)) best = fminf(best, c.y);
  }
  {  // side QP, from Q
    const float u = TP - TQ;
    const float ff = (QQ - PQ) + (PP - PQ), fw = (QQ - QX) - (PQ - PX);
    const float r = __fmul_rn(fast_sqrt<WIDE>(fmaf(ff, d2.y, -__fmul_rn(fw, fw))), fast_rsqrt<WIDE>(fmaf(-u, u, ff)));
    const float lam = __fmul_rn(fmaf(-u, r, fw), fast_rcp<WIDE>(ff));
    if (in_unit(lam)) best = fminf(best, __fadd_rn(fmaf(lam, u, TQ), r));
  }
  {  // interior: y = l1 P + l2 Q + l3 R
    const float idet = fast_rcp<WIDE>(fmaf(PP, QQ, -__fmul_rn(PQ, PQ)));
    // the reference's h (also the numerator of g1), s and t
    const float h = fmaf(QQ, up, -__fmul_rn(PQ, uq));
    const float s = fmaf(-up, PQ, __fmul_rn(uq, PP)), t = fmaf(up, QX, -__fmul_rn(uq, PX));
    const float g1 = __fmul_rn(h, idet);                                   // in-plane gradient, coefficient of P - R
    const float g2 = __fmul_rn(fmaf(PP, uq, -__fmul_rn(PQ, up)), idet);  // and of Q - R
    const float foot1 = __fmul_rn(fmaf(PQ, -QX, __fmul_rn(QQ, PX)), idet);  // X's foot point, weight of P
    // the point downhill of the foot point (lane x) and its mirror uphill
    // (lane y): the reference's SMALLNUM offset in l2 = (s l1 + t) / (h +
    // eps_h) can move the first point out of the face where h is small, and
    // the mirror's point is then the better one, as in the reference
    const float dl = __fmul_rn(__fmul_rn(hX, fast_rsqrt<WIDE>(__fsub_rn(1.f, fmaf(g1, up, __fmul_rn(g2, uq))))), g1);
    const float ih = fast_rcp<WIDE>(h + eps_h);
    const float2 l1 = f2(foot1 - dl, foot1 + dl);
    const float2 l2 = __fmul2_rn(__ffma2_rn(f2(s, s), l1, f2(t, t)), f2(ih, ih));
    const float2 l3 = f2((1.f - l1.x) - l2.x, (1.f - l1.y) - l2.y);
    // |y - X|^2 as the quadratic form of (l1, l2), and T_lin(y)
    const float2 a1 = __ffma2_rn(l1, f2(PP, PP), __ffma2_rn(l2, f2(PQ, PQ), f2(-PX, -PX)));
    const float2 a2 = __ffma2_rn(l1, f2(PQ, PQ), __ffma2_rn(l2, f2(QQ, QQ), f2(-QX, -QX)));
    const float2 a3 = __ffma2_rn(l1, f2(-PX, -PX), __ffma2_rn(l2, f2(-QX, -QX), f2(XX, XX)));
    const float2 Q = __ffma2_rn(a1, l1, __ffma2_rn(a2, l2, a3));
    const float2 lin = __ffma2_rn(f2(TP, TP), l1, __ffma2_rn(f2(TQ, TQ), l2, __fmul2_rn(f2(TR, TR), l3)));
    const float2 c = __fadd2_rn(lin, f2(fast_sqrt<WIDE>(Q.x), fast_sqrt<WIDE>(Q.y)));
    if (in_unit(l1.x, l2.x, l3.x)) best = fminf(best, c.x);
    if (in_unit(l1.y, l2.y, l3.y)) best = fminf(best, c.y);
  }
  return best;
}

// Triangle update of C from edge AB (speed 1); the square roots are taken in
// single precision as in the reference, which passes doubles to sqrtf.
template <typename R>
__device__ __forceinline__ R tri_solve(R TA, R TB, R LenAB, R LenBC, R LenAC, R LN) {
  if (TA >= LN && TB >= LN) return LN;
  const R speedI = R(1);
  const R TAB = TB - TA;
  const R a = (speedI * speedI * LenAB * LenAB - TAB * TAB) * LenAB * LenAB;
  const R EdgeTA = TA + LenAC * speedI, EdgeTB = TB + LenBC * speedI;
  R TC1 = LN, TC2 = LN;
  if (a > R(0)) {
    const R cosA = (LenAC * LenAC + LenAB * LenAB - LenBC * LenBC) / (R(2) * LenAC * LenAB);
    const R b = R(2) * LenAB * LenAC * cosA * (TAB * TAB - speedI * speedI * LenAB * LenAB);
    const R delta = R(4) * LenAC * LenAC * a * TAB * TAB * (R(1) - cosA * cosA);
    const R sq = (R)sqrtf((float)delta);
    const R l1 = (-b + sq) / (R(2) * a);
    const R l2 = (-b - sq) / (R(2) * a);
    if (l1 >= R(0) && l1 <= R(1)) {
      const R LenAD = l1 * LenAB;
      const R LenCD = (R)sqrtf((float)(LenAC * LenAC + LenAD * LenAD - R(2) * LenAC * LenAD * cosA));
      TC1 = l1 * TAB + TA + LenCD * speedI;
    }
    if (l2 >= R(0) && l2 <= R(1)) {
      const R LenAD = l2 * LenAB;
      const R LenCD = (R)sqrtf((float)(LenAC * LenAC + LenAD * LenAD - R(2) * LenAC * LenAD * cosA));
      TC2 = l2 * TAB + TA + LenCD * speedI;
    }
    return rmin(TC2, rmin(TC1, rmin(EdgeTA, EdgeTB)));
  }
  return rmin(EdgeTA, EdgeTB);
}

// The fast build's triangle sweep: tri_solve's quantity (the least of the two
// edges and the stationary point of T_lin(y) + |y - X| over the side PQ) in
// the planar-wave form of tet_solve_wave's sides.  What depends on the
// triangle alone is computed once per visit: of its sides (0: BC, 1: CA, 2:
// AB, each opposite the target of its number) the length, its square and
// that square's reciprocal, and (Q - P).(X - P); and twice the area.
struct TriGeo {
  float len[3], ff[3], inv[3], fw[3], area2;
};
// lc: B = (c0, 0), C = (c1, c2) with A at the origin
__device__ __forceinline__ TriGeo tri_geo(float c0, float c1, float c2) {
  TriGeo g;
  const float e = c1 - c0;
  g.ff[0] = fmaf(e, e, __fmul_rn(c2, c2));
  g.ff[1] = fmaf(c1, c1, __fmul_rn(c2, c2));
  g.ff[2] = __fmul_rn(c0, c0);
  g.fw[0] = -__fmul_rn(e, c0);             // (C - B).(A - B)
  g.fw[1] = fmaf(c1, e, __fmul_rn(c2, c2));  // (A - C).(B - C)
  g.fw[2] = __fmul_rn(c0, c1);             // (B - A).(C - A)
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    g.len[k] = sqrtf(g.ff[k]);
    g.inv[k] = 1.f / g.ff[k];
  }
  g.area2 = fabsf(__fmul_rn(c0, c2));
  return g;
}
// Target K from the side opposite it (P = vertex K + 1, Q = vertex K + 2, mod 3).
template <int K>
__device__ __forceinline__ float tri_solve_wave(const TriGeo& g, const float* T) {
  constexpr int P = (K + 1) % 3, Q = (K + 2) % 3;
  const float u = T[Q] - T[P];
  // none when ff <= u^2: the rsqrt is NaN or inf and the range test fails
  // (denormals only where an edge is below 1e-19: its square is one).
  // Rounded down, a mode chosen by fit: of 196 eikonal runs (40^2 to 300^2)
  // the mean error against 64 bits is 1.47e-7 this way, 1.57e-7 rounded to
  // nearest, 1.53e-7 in the quadratic form.  (A front stops up to the
  // tolerance too high; that is the stopping rule's, not this product's.)
  const float r = __fmul_rd(g.area2, fast_rsqrt<false>(fmaf(-u, u, g.ff[K])));
  const float lam = __fmul_rn(fmaf(-u, r, g.fw[K]), g.inv[K]);
  // |X - P| is the side opposite Q, |X - Q| the one opposite P
  const float best = fminf(T[P] + g.len[Q], T[Q] + g.len[P]);
  return in_unit(lam) ? fminf(best, __fadd_rn(fmaf(lam, u, T[P]), r)) : best;
}

}  // namespace lsgb
