// Device engine of one system: its HBM state, kernel argument builders and the step
// pieces queued on its stream.  Shared by the single-system C ABI (engine.cu) and the
// batched ensemble / serving loop (batch.cu).
#pragma once
#include <atomic>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>
#include <vector>

#include "host/host.h"
#include "kernels/kernels.h"

namespace fz {

#define FZ_CUDA(call)                                                                                  \
  do {                                                                                                 \
    cudaError_t e_ = (call);                                                                           \
    if (e_ != cudaSuccess) return fail(FZ_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
  } while (0)

struct Engine {
  int dev = 0;
  cudaStream_t st = nullptr;
  bool own_stream = false;
  fzk::SysParams p{};
  int n = 0, nunits = 0, ncol = 0, nslots = 0, mask_cap = 0, all_images = 0;
  int ocap = 0;            // per-block pair-list capacity (multiple of 32)
  float rp2 = 0.f, prune_half2 = 0.f;
  int nb_grid = 0, nb_per_sm = 3, n_sm = 148;
  int dcx = 1, dcy = 1;
  int* blk_col = nullptr;
  std::vector<void*> allocs;
  // atoms
  float4 *pos4 = nullptr, *vel4 = nullptr, *pos_build = nullptr;
  long long *facc = nullptr, *energy = nullptr, *psum = nullptr;
  int* type = nullptr;
  // sorted slots / neighbour tiles
  float4 *xyzq_s = nullptr, *bb_lo = nullptr, *bb_hi = nullptr;
  int *typ_s = nullptr, *perm = nullptr, *inv_perm = nullptr, *col_of = nullptr, *col_count = nullptr,
      *col_cursor = nullptr, *col_start = nullptr, *col_tmp = nullptr;
  uint32_t *outer = nullptr, *inner = nullptr, *masks = nullptr, *dmask = nullptr;
  int *outer_n = nullptr, *inner_nt = nullptr, *inner_m = nullptr, *flag_prune = nullptr;
  float4* pos_prune = nullptr;
  int2* items = nullptr;
  int chunk = 16;
  int tiles = 0;  // pair tiles of the first pruned list (sizes the work items)
  int *excl_off = nullptr, *excl_idx = nullptr;
  int *xn = nullptr, *xs = nullptr, xmax = 1;  // per-slot excluded-partner slots
  int2* xrange = nullptr;                          // per slot: partner block range
  int *flag = nullptr, *counters = nullptr, *status = nullptr;
  float2 *ljtab = nullptr, *lj14 = nullptr;
  // bonded
  int nbond = 0, nangle = 0, nub = 0, ndihe = 0, nimpr = 0, nexcl = 0, n14 = 0;
  int2 *bond = nullptr, *ub = nullptr, *excl = nullptr, *p14 = nullptr;
  int4 *angle = nullptr, *dihe = nullptr, *impr = nullptr;
  float2 *bond_prm = nullptr, *angle_prm = nullptr, *ub_prm = nullptr, *impr_prm = nullptr;
  float4* dihe_prm = nullptr;
  int nfixed = 0;  // atoms of fixed (consfix) segments
  // consharm restraint: segment of every atom (0, 1, -1), masses, fixed-point mass
  // centre sums (x0 y0 z0 x1 y1 z1), inverse segment masses, target offset, constant
  bool restraint = false;
  // of each kind of bonded term, the first *_step are those the bonded kernel evaluates in
  // a step (the rest belong to rigid waters: the integrator's pass has them, see
  // UnitTerms); a force evaluation outside a step takes all
  int nbond_step = 0, nangle_step = 0, nexcl_step = 0;
  fzk::UnitTerms* unit_terms = nullptr;
  int* unit_term_of = nullptr;
  int unit_term_begin = 0;
  int few_waters = 0;  // see IntegrateArgs
  float4* pos_drift = nullptr;  // drifted positions of this step, never wrapped by a rebuild
  int* rs_seg = nullptr;
  float* rs_mass = nullptr;
  long long* rs_acc = nullptr;
  double rs_inv_m[2] = {0, 0}, rs_dist[3] = {0, 0, 0}, rs_fc = 0;
  // minimiser state (allocated on first use): previous force, search direction,
  // positions before the last move
  float4 *min_prev_f = nullptr, *min_dir = nullptr, *min_pos = nullptr;
  // integration units, grouped in classes of equal (atoms, constraints)
  int ncls = 0, cls_na[8] = {}, cls_nc[8] = {}, cls_begin[9] = {};
  int4* unit_atoms = nullptr;
  int* unit_meta = nullptr;
  float4* unit_d = nullptr;
  // PME
  int K[3] = {0, 0, 0}, B[3] = {0, 0, 0}, nbk[3] = {0, 0, 0};
  int gather_mode = 0;  // PME gather kernel (PmeArgs::gather)
  bool tuned = false;   // launch shapes picked by the autotuner
  int *brick_of = nullptr, *brick_count = nullptr, *brick_cursor = nullptr, *brick_start = nullptr,
      *brick_atoms = nullptr;
  float* grid = nullptr;
  float2* cgrid = nullptr;
  float2* tw[3] = {nullptr, nullptr, nullptr};
  float *gfac[3] = {nullptr, nullptr, nullptr}, *f2[3] = {nullptr, nullptr, nullptr};
  float gscale = 0.f;
  // which kernel arguments this engine hands out: another number in every engine and after
  // every change of the box or of the list tests, so that a batch knows when its own are old
  unsigned long long args_stamp = next_stamp();
  static unsigned long long next_stamp() {
    static std::atomic<unsigned long long> last{0};
    return ++last;
  }
  // run state
  bool forces_valid = false;
  long long step = 0;
  double self_energy = 0, inv_mtot = 0, dtu = 0, shake_tol = 1e-10;
  int settle = 0;  // (3,3) units solved by SETTLE (all are symmetric triangles)
  double box_d[3] = {0, 0, 0};
  int ncons = 0;
  int temp_reset_every = 0;
  double temperature = 300.0;
  unsigned long long seed = 0;
  long long launches = 0;
  // per-stage timing
  bool timing = false;
  cudaEvent_t ev[12] = {};
  double stage_ms[5] = {0, 0, 0, 0, 0};
  long long timed_steps = 0;
  // CUDA graph of one MD step (kick/drift/SHAKE, neighbour maintenance, forces,
  // kick/RATTLE); captured on first use, replayed with one launch per step
  cudaGraph_t step_graph = nullptr;
  cudaGraphExec_t step_exec = nullptr;
  // graph of `chunk_steps` consecutive steps (one launch per chunk): replayed for the
  // runs of steps with no velocity reassignment inside; 0 or 1 disables (FZ_GRAPH_CHUNK)
  cudaGraph_t chunk_graph = nullptr;
  cudaGraphExec_t chunk_exec = nullptr;
  int chunk_steps = 100;
  // chunk graphs fuse each step's closing kick + RATTLE into the next step's opening
  // kick + drift pass (FZ_FUSE_CLOSE=0 keeps the two passes apart)
  bool fuse_close = true;
  // prune with one CTA per i-block (systems with few blocks; identical lists)
  int prune_split = 0;
  int outer_split = 0;
  bool use_graph = true;
  cudaError_t capture_error = cudaSuccess;
  // PME runs on a second stream concurrently with the pair and bonded kernels
  cudaStream_t st2 = nullptr;
  cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
  // bonded terms outside rigid waters on a third
  cudaStream_t st3 = nullptr;
  cudaEvent_t ev_top = nullptr, ev_join3 = nullptr;
  // device side of host transfers: 6n floats (positions | velocities) or 3n doubles
  double* xfer = nullptr;
  // pinned staging
  void* pinned = nullptr;
  size_t pinned_bytes = 0;
  // Andersen barostat (isotropic; the box keeps its aspect ratios).  L is the x edge;
  // the piston obeys L'' = (P - Pref) / (3 M L^2) - 2 L'^2 / L, P = (2 KE + W) / (3 V)
  // (src/cell_based_kernels.cu:569-579).
  bool npt = false;
  double pmass = 1e-5, pref_atm = 1.0;
  double ratio[3] = {1.0, 1.0, 1.0};
  double Ldot = 0.0, Lacc = 0.0;
  double L_build = 0.0, L_prune = 0.0;  // box x edge at the last list build / prune
  long long seen_rebuilds = 0, seen_prunes = 0;
  double last_pressure = 0.0;
  double plist = 0.0, cutoff = 0.0, col_a = 0.0;
  float skin_half2_nve = 0.f, prune_half2_nve = 0.f;
  double prune_delta = 0.0;
  double* bm2[3] = {nullptr, nullptr, nullptr};  // per dimension: |b(m)|^2 of the splines
  int ncx = 1, ncy = 1;

  template <class T>
  fz_status alloc(T** ptr, size_t count) {
    *ptr = nullptr;
    if (count == 0) count = 1;
    void* p = nullptr;
    cudaError_t e = cudaMalloc(&p, count * sizeof(T));
    if (e != cudaSuccess) return fail(FZ_ERR_NOMEM, std::string("cudaMalloc: ") + cudaGetErrorString(e));
    allocs.push_back(p);
    e = cudaMemsetAsync(p, 0, count * sizeof(T), st);
    if (e != cudaSuccess) return fail(FZ_ERR_CUDA, std::string("cudaMemset: ") + cudaGetErrorString(e));
    *ptr = static_cast<T*>(p);
    return FZ_OK;
  }
  template <class T>
  fz_status upload(T** ptr, const std::vector<T>& v) {
    fz_status s = alloc(ptr, v.size());
    if (s) return s;
    if (!v.empty()) FZ_CUDA(cudaMemcpyAsync(*ptr, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice, st));
    return FZ_OK;
  }
  void release(void* ptr) {
    for (auto& a : allocs)
      if (a == ptr) {
        cudaFree(a);
        a = allocs.back();
        allocs.pop_back();
        return;
      }
  }
  fz_status staging(size_t bytes) {
    if (pinned_bytes >= bytes) return FZ_OK;
    if (pinned) cudaFreeHost(pinned);
    pinned = nullptr;
    FZ_CUDA(cudaMallocHost(&pinned, bytes));
    pinned_bytes = bytes;
    return FZ_OK;
  }
  ~Engine() {
    if (st) cudaStreamSynchronize(st);
    if (step_exec) cudaGraphExecDestroy(step_exec);
    if (step_graph) cudaGraphDestroy(step_graph);
    if (chunk_exec) cudaGraphExecDestroy(chunk_exec);
    if (chunk_graph) cudaGraphDestroy(chunk_graph);
    if (ev_fork) cudaEventDestroy(ev_fork);
    if (ev_join) cudaEventDestroy(ev_join);
    if (ev_top) cudaEventDestroy(ev_top);
    if (ev_join3) cudaEventDestroy(ev_join3);
    if (st3) cudaStreamDestroy(st3);
    if (st2) cudaStreamDestroy(st2);
    for (auto& x : ev)
      if (x) cudaEventDestroy(x);
    for (void* p : allocs) cudaFree(p);
    if (pinned) cudaFreeHost(pinned);
    if (own_stream && st) cudaStreamDestroy(st);
  }

  fzk::RebuildArgs rebuild_args() const {
    fzk::RebuildArgs a{};
    a.p = p;
    a.flag = flag;
    a.counters = counters;
    a.status = status;
    a.pos4 = pos4;
    a.pos_build = pos_build;
    a.type = type;
    a.col_of = col_of;
    a.col_count = col_count;
    a.col_cursor = col_cursor;
    a.col_start = col_start;
    a.col_tmp = col_tmp;
    a.perm = perm;
    a.inv_perm = inv_perm;
    a.xyzq_s = xyzq_s;
    a.typ_s = typ_s;
    a.bb_lo = bb_lo;
    a.bb_hi = bb_hi;
    a.excl_off = excl_off;
    a.excl_idx = excl_idx;
    a.xn = xn;
    a.xs = xs;
    a.xrange = xrange;
    a.xmax = xmax;
    a.masks = masks;
    a.mask_cap = mask_cap;
    a.all_images = all_images;
    a.outer = outer;
    a.outer_n = outer_n;
    a.inner = inner;
    a.inner_nt = inner_nt;
    a.inner_m = inner_m;
    a.dmask = dmask;
    a.ocap = ocap;
    a.flag_prune = flag_prune;
    a.rp2 = rp2;
    a.pos_prune = pos_prune;
    a.items = items;
    a.chunk = chunk;
    a.prune_split = prune_split;
    a.outer_split = outer_split;
    a.blk_col = blk_col;
    a.dcx = dcx;
    a.dcy = dcy;
    return a;
  }
  fzk::NonbondedArgs nb_args() const {
    fzk::NonbondedArgs a{};
    a.p = p;
    a.xyzq_s = xyzq_s;
    a.typ_s = typ_s;
    a.perm = perm;
    a.inner = inner;
    a.inner_nt = inner_nt;
    a.inner_m = inner_m;
    a.dmask = dmask;
    a.masks = masks;
    a.counters = counters;
    a.ljtab = ljtab;
    a.facc = facc;
    a.energy = energy;
    a.ocap = ocap;
    a.items = items;
    a.chunk = chunk;
    a.grid = nb_grid;
    // FZ_NB_GRID_PER_SM: fewer CTAs than the build's occupancy, leaving room on every SM
    // for the PME kernels of the second stream (a measurement knob)
    if (const char* v = std::getenv("FZ_NB_GRID_PER_SM")) a.grid = n_sm * std::max(1, std::min(8, std::atoi(v)));
    a.minb = nb_per_sm;
    a.flag = flag;
    a.flag_prune = flag_prune;
    a.close_lists = 1;
    return a;
  }
  // step: the forces of a step, after its drift (pos_drift)
  fzk::PmeArgs pme_args(bool step = false) const {
    fzk::PmeArgs a{};
    a.p = p;
    a.pos4 = step ? pos_drift : pos4;
    a.n = n;
    for (int d = 0; d < 3; ++d) {
      a.K[d] = K[d];
      a.set_scale(d, box_d[d]);
      a.B[d] = B[d];
      a.nb[d] = nbk[d];
      a.tw[d] = tw[d];
      a.gfac[d] = gfac[d];
      a.f2[d] = f2[d];
    }
    a.brick_of = brick_of;
    a.brick_count = brick_count;
    a.brick_cursor = brick_cursor;
    a.brick_start = brick_start;
    a.brick_atoms = brick_atoms;
    a.grid = grid;
    a.cgrid = cgrid;
    a.gscale = gscale;
    a.facc = facc;
    a.energy = energy;
    a.status = status;
    a.gather = gather_mode;
    return a;
  }
  fzk::BondedArgs bonded_args(bool step = false) const {
    fzk::BondedArgs a{};
    a.p = p;
    a.pos4 = step ? pos_drift : pos4;
    a.nbond = step ? nbond_step : nbond;
    a.nangle = step ? nangle_step : nangle;
    a.nub = nub;
    a.ndihe = ndihe;
    a.nimpr = nimpr;
    a.nexcl = step ? nexcl_step : nexcl;
    a.n14 = n14;
    a.bond = bond;
    a.bond_prm = bond_prm;
    a.angle = angle;
    a.angle_prm = angle_prm;
    a.ub = ub;
    a.ub_prm = ub_prm;
    a.dihe = dihe;
    a.dihe_prm = dihe_prm;
    a.impr = impr;
    a.impr_prm = impr_prm;
    a.excl = excl;
    a.p14 = p14;
    a.type = type;
    a.lj14 = lj14;
    a.facc = facc;
    a.energy = energy;
    return a;
  }
  fzk::IntegrateArgs int_args() const {
    fzk::IntegrateArgs a{};
    a.p = p;
    a.nunits = nunits;
    a.unit_atoms = unit_atoms;
    a.unit_meta = unit_meta;
    a.unit_d = unit_d;
    a.pos4 = pos4;
    a.pos_drift = pos_drift;
    a.unit_terms = unit_terms;
    a.unit_term_of = unit_term_of;
    a.unit_term_begin = unit_term_begin;
    a.fuse_terms = unit_terms ? 1 : 0;
    a.few_waters = few_waters;
    a.vel4 = vel4;
    a.facc = facc;
    a.xyzq_s = xyzq_s;
    a.inv_perm = inv_perm;
    a.pos_build = pos_build;
    a.pos_prune = pos_prune;
    a.flag = flag;
    a.flag_prune = flag_prune;
    a.prune_half2 = prune_half2;
    a.status = status;
    a.energy = energy;
    a.dtu = dtu;
    for (int d = 0; d < 3; ++d) {
      a.box_d[d] = box_d[d];
      a.inv_box_d[d] = 1.0 / box_d[d];
    }
    a.shake_tol = shake_tol;
    a.shake_maxit = 500;
    a.settle = settle;
    a.lam = 1.0;
    a.vfric = 1.0;
    a.u_begin = 0;
    a.u_end = nunits;
    a.ncls = ncls;
    for (int c = 0; c < 8; ++c) {
      a.cls_na[c] = cls_na[c];
      a.cls_nc[c] = cls_nc[c];
    }
    for (int c = 0; c < 9; ++c) a.cls_begin[c] = cls_begin[c];
    return a;
  }

  // ---------------------------------------------------------------- step pieces
  void mark(int k) {
    if (timing) cudaEventRecord(ev[k], st);
  }
  // step: after a drift whose pass has evaluated the rigid waters' own terms
  void forces(bool energies, int terms = FZ_TERM_ALL, bool step = false) {
    mark(1);
    const bool close = !(terms & FZ_TERM_NONBONDED);
    fzk::launch_rebuild(rebuild_args(), st, close);
    launches += rebuild_launches() + (close ? 1 : 0);
    mark(2);
    // PME beside the pair and bonded kernels (in line when the stages are timed)
    const bool beside = (terms & FZ_TERM_PME) && st2 && !timing;
    if (beside) {
      cudaEventRecord(ev_fork, st);
      cudaStreamWaitEvent(st2, ev_fork, 0);
      fzk::launch_pme(pme_args(step), energies, st2);
      cudaEventRecord(ev_join, st2);
    }
    if (terms & FZ_TERM_NONBONDED) {
      fzk::launch_nonbonded(nb_args(), energies, st);
      launches += 1;
    }
    mark(3);
    if (terms & (FZ_TERM_BONDED | FZ_TERM_BONDED_PARTS)) {
      fzk::BondedArgs a = bonded_args(step);
      if (!(terms & FZ_TERM_BONDED)) {
        // selected parts only: the kernel's flattened term range skips empty classes
        if (!(terms & FZ_TERM_BONDS)) a.nbond = 0;
        if (!(terms & FZ_TERM_ANGLES)) a.nangle = 0;
        if (!(terms & FZ_TERM_UREYB)) a.nub = 0;
        if (!(terms & FZ_TERM_DIHEDRALS)) a.ndihe = 0;
        if (!(terms & FZ_TERM_IMPROPERS)) a.nimpr = 0;
        if (!(terms & FZ_TERM_PAIRS14)) a.n14 = 0;
        if (!(terms & FZ_TERM_EXCLUSIONS)) a.nexcl = 0;
      }
      fzk::launch_bonded(a, energies, st);
      launches += step ? bonded_step_launches() : bonded_launches();
    }
    if ((terms & FZ_TERM_BONDED) && restraint) {
      restraint_forces(st);
      launches += 2;
    }
    mark(4);
    if (terms & FZ_TERM_PME) {
      if (beside) cudaStreamWaitEvent(st, ev_join, 0);
      else fzk::launch_pme(pme_args(step), energies, st);
      launches += fzk::pme_launches(pme_args());
    }
    mark(5);
  }
  // the forces a step opens with: those the last step or evaluation left, or new ones where
  // the positions have changed since
  fz_status own_forces() {
    if (forces_valid) return FZ_OK;
    FZ_CUDA(cudaMemsetAsync(facc, 0, 3 * sizeof(long long) * n, st));
    forces(false);
    forces_valid = true;
    return FZ_OK;
  }
  // accumulates the events of one timed step: 0 start, 1..5 forces, 6 end
  void collect_step() {
    cudaEventSynchronize(ev[6]);
    float ms = 0.f;
    auto el = [&](int a, int b) {
      cudaEventElapsedTime(&ms, ev[a], ev[b]);
      return (double)ms;
    };
    stage_ms[0] += el(1, 2);
    stage_ms[1] += el(2, 3);
    stage_ms[2] += el(3, 4);
    stage_ms[3] += el(4, 5);
    stage_ms[4] += el(0, 1) + el(5, 6);
    timed_steps++;
  }
  // consharm: mass centres of the two segments, then the pull on segment 1's atoms
  void restraint_forces(cudaStream_t s) {
    cudaMemsetAsync(rs_acc, 0, 8 * sizeof(long long), s);
    fzk::launch_restraint(p, pos4, rs_seg, rs_mass, rs_acc, rs_inv_m[0], rs_inv_m[1], rs_dist, rs_fc, facc, s);
  }
  // kernels one captured step launches
  long long graph_step_launches() const {
    return fzk::drift_launches(int_args()) + ncls + rebuild_launches() + 1 + bonded_step_launches() +
           fzk::pme_launches(pme_args()) + (restraint ? 2 : 0);
  }
  int rebuild_launches() const {
    return fzk::kRebuildLaunches + (fzk::columns_scan_in_block(rebuild_args()) ? 0 : 1);
  }
  int bonded_step_launches() const {
    return (nbond_step + nangle_step + nub + ndihe + nimpr + nexcl_step + n14 > 0) ? 1 : 0;
  }
  int bonded_launches() const { return (nbond + nangle + nub + ndihe + nimpr + nexcl + n14 > 0) ? 1 : 0; }
  // One pass of the integrator over all unit classes, which touch disjoint atoms: where
  // they take more than one launch, the first half of them runs on st3 beside the rest.
  template <class L>
  void integrate(const fzk::IntegrateArgs& ia, int passes, L launch) {
    if (passes < 2) return launch(ia, st);
    const int h = ia.ncls / 2;
    fzk::IntegrateArgs first = ia, rest = ia;
    first.ncls = h;
    rest.ncls = ia.ncls - h;
    for (int c = 0; c < rest.ncls; ++c) {
      rest.cls_na[c] = ia.cls_na[c + h];
      rest.cls_nc[c] = ia.cls_nc[c + h];
      rest.cls_begin[c] = ia.cls_begin[c + h];
    }
    rest.cls_begin[rest.ncls] = ia.cls_begin[ia.ncls];
    cudaEventRecord(ev_top, st);
    cudaStreamWaitEvent(st3, ev_top, 0);
    launch(first, st3);
    cudaEventRecord(ev_join3, st3);
    launch(rest, st);
    cudaStreamWaitEvent(st, ev_join3, 0);
  }
  // One MD step.  open: the step starts with its own kick + drift pass (else the
  // previous step left its closing kick + RATTLE to this step's first pass); close: the
  // step ends with the kick + RATTLE pass (else the next step's first pass does it).
  //
  // PME runs on st2 beside the pair kernel, the bonded terms outside rigid waters on
  // st3.  Both read pos_drift, which a rebuild does not wrap, so they need only the
  // drift and start beside the neighbour launches: the step's length is the longer of
  // the two chains.
  void step_body(bool open = true, bool close = true) {
    const fzk::IntegrateArgs ia = int_args();
    if (!st2) {
      if (open) fzk::launch_kick_drift(ia, st);
      else fzk::launch_close_kick_drift(ia, st);
      forces(false, FZ_TERM_ALL, true);
      if (close) fzk::launch_kick_rattle(ia, false, true, st);
      return;
    }
    const fzk::PmeArgs pa = pme_args(true);
    cudaEventRecord(ev_top, st);
    cudaStreamWaitEvent(st2, ev_top, 0);
    fzk::launch_pme_clear(pa, st2);
    integrate(ia, fzk::drift_launches(ia), [&](const fzk::IntegrateArgs& a, cudaStream_t s) {
      if (open) fzk::launch_kick_drift(a, s);
      else fzk::launch_close_kick_drift(a, s);
    });
    cudaEventRecord(ev_fork, st);
    cudaStreamWaitEvent(st2, ev_fork, 0);
    fzk::launch_pme(pa, false, st2, true);
    const bool bonded = bonded_step_launches() > 0;
    if (bonded) {
      cudaStreamWaitEvent(st3, ev_fork, 0);
      fzk::launch_bonded(bonded_args(true), false, st3);
      cudaEventRecord(ev_join3, st3);
    }
    fzk::launch_rebuild(rebuild_args(), st, false);
    fzk::launch_nonbonded(nb_args(), false, st);
    if (restraint) restraint_forces(st);
    if (bonded) cudaStreamWaitEvent(st, ev_join3, 0);
    cudaEventRecord(ev_join, st2);
    cudaStreamWaitEvent(st, ev_join, 0);
    if (close)
      integrate(ia, ia.ncls, [](const fzk::IntegrateArgs& a, cudaStream_t s) {
        fzk::launch_kick_rattle(a, false, true, s);
      });
  }
  fz_status graph_step() {
    if (!step_exec) {
      capture_error = cudaSuccess;
      FZ_CUDA(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
      const long long l0 = launches;
      step_body();
      launches = l0;
      cudaGraph_t g = nullptr;
      FZ_CUDA(cudaStreamEndCapture(st, &g));
      step_graph = g;
      if (capture_error != cudaSuccess)
        return fail(FZ_ERR_CUDA, std::string("step capture: ") + cudaGetErrorString(capture_error));
      FZ_CUDA(cudaGraphInstantiate(&step_exec, step_graph, 0));
    }
    FZ_CUDA(cudaGraphLaunch(step_exec, st));
    launches += graph_step_launches();
    return FZ_OK;
  }
  // chunk_steps steps in one graph launch (captured on first use)
  fz_status graph_chunk() {
    if (!chunk_exec) {
      capture_error = cudaSuccess;
      FZ_CUDA(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
      const long long l0 = launches;
      // inside the chunk each step's closing pass joins the next step's opening one
      for (int k = 0; k < chunk_steps; ++k) step_body(k == 0 || !fuse_close, k == chunk_steps - 1 || !fuse_close);
      launches = l0;
      cudaGraph_t g = nullptr;
      FZ_CUDA(cudaStreamEndCapture(st, &g));
      chunk_graph = g;
      if (capture_error != cudaSuccess)
        return fail(FZ_ERR_CUDA, std::string("chunk capture: ") + cudaGetErrorString(capture_error));
      FZ_CUDA(cudaGraphInstantiate(&chunk_exec, chunk_graph, 0));
    }
    FZ_CUDA(cudaGraphLaunch(chunk_exec, st));
    launches += (long long)chunk_steps * graph_step_launches() - (fuse_close ? (long long)(chunk_steps - 1) * ncls : 0);
    return FZ_OK;
  }
  void drop_graph() {
    if (step_exec) cudaGraphExecDestroy(step_exec);
    if (step_graph) cudaGraphDestroy(step_graph);
    if (chunk_exec) cudaGraphExecDestroy(chunk_exec);
    if (chunk_graph) cudaGraphDestroy(chunk_graph);
    step_exec = nullptr;
    step_graph = nullptr;
    chunk_exec = nullptr;
    chunk_graph = nullptr;
  }
  // what the host reads back after a call: energy slots, list counters and the status
  // word lie together on the device, one copy (and one wait) brings them
  struct Readback {
    long long energy[fzk::EN_COUNT];
    int counters[fzk::CNT_COUNT];
    int status, pad;
  };
  fz_status read_back(Readback* b) {
    FZ_CUDA(cudaMemcpyAsync(b, energy, sizeof(Readback), cudaMemcpyDeviceToHost, st));
    FZ_CUDA(cudaStreamSynchronize(st));
    FZ_CUDA(cudaGetLastError());
    return status_of(b->status);
  }
  fz_status check() {
    Readback b;
    return read_back(&b);
  }
  static fz_status status_of(int h) {
    if (h) {
      std::string m = "device status:";
      if (h & fzk::ST_TILE_OVERFLOW) m += " pair-tile capacity exceeded;";
      if (h & fzk::ST_MASK_OVERFLOW) m += " exclusion-mask capacity exceeded;";
      if (h & fzk::ST_SLOT_OVERFLOW) m += " sorted-slot capacity exceeded;";
      if (h & fzk::ST_COLUMN_OVERFLOW) m += " column occupancy exceeded;";
      if (h & fzk::ST_SHAKE_NOCONV) m += " SHAKE did not converge within its iteration cap;";
      if (h & fzk::ST_BAD_COORD) m += " non-finite or runaway coordinates;";
      const int code = (h & fzk::ST_SHAKE_NOCONV) ? FZ_ERR_SHAKE : FZ_ERR_CAPACITY;
      return fail(code, m);
    }
    return FZ_OK;
  }
};

// moves an engine to the box with x edge L (aspect ratios kept): kernel parameters,
// column reach and PME influence tables (engine.cu)
fz_status set_box(Engine* e, double L);
// upper estimate of an uploaded system's device memory (engine.cu)
size_t device_bytes(const fz_system* sys);

}  // namespace fz
