// Real-space nonbonded pair kernel: CHARMM LJ with the switch from ron to rc plus
// erfc real-space Ewald, the functional form of nonbondforce (src/nonbonded_forces.cu:114-245).
//
// B200 design: one warp per tile (16 i-atoms of half a sorted block x 32 j-atoms of the
// pair list), each pair evaluated once (Newton's third law).  i data live in
// registers, two atoms a lane; the tile's j data (x, y, z, q, LJ type, periodic image
// applied) are staged once into a doubled shared-memory ring, so at step k a lane reads
// its j with a constant-offset load and no wrap arithmetic; only the j force
// accumulator rotates through the lanes (3 shuffles per two pairs).  Tiles without
// excluded pairs (the large majority) run a mask-free loop.  The kernel is FP32-issue
// bound, so every pair-step instruction counts (230,400 atoms: 246 M warp instructions
// and 280 us a launch with one i atom a lane, 232 M and 262 us with two):
//   erfc(x) = t P(t) exp(-x^2), t = 1/(1 + p x)  (Abramowitz & Stegun, Handbook of
//     Mathematical Functions (1964) eq. 7.1.26, |error| <= 1.5e-7), with exp2 and the
//     constants pre-scaled so exp(-x^2) is one multiply and one MUFU.EX2;
//   the CHARMM switch (rc^2-r^2)^2 (rc^2+2r^2-3ron^2)/(rc^2-ron^2)^3 written as
//     1 - t^2 (3 - 2t) with t = sat((r^2-ron^2)/(rc^2-ron^2)) (identical polynomial),
//     its derivative exact (the reference's force at src/nonbonded_forces.cu:210-214
//     carries an extra Swcoeff2*invDist term);
// Forces go to int64 fixed point at the end of each tile (RED atomics, order
// independent): bit-reproducible run to run.
#include "common.cuh"
#include "kernels.h"

namespace fzk {

constexpr float kAS_p = 0.3275911f;
constexpr float kAS_a1 = 0.254829592f;
constexpr float kAS_a2 = -0.284496736f;
constexpr float kAS_a3 = 1.421413741f;
constexpr float kAS_a4 = -1.453152027f;
constexpr float kAS_a5 = 1.061405429f;
constexpr float kTwoOverSqrtPi = 1.1283791670955126f;
constexpr float kLog2e = 1.4426950408889634f;
constexpr int kWarps = 8;

// single-instruction MUFU approximations (PTX ISA: rsqrt/ex2/rcp .approx.ftz.f32)
__device__ __forceinline__ float rsqrt_a(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float ex2_a(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float rcp_a(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

struct PairConst {
  float rc2, beta, eb2;   // eb2 = -beta^2 log2(e)
  float p_b;              // p * beta
  float c2b;              // 2 beta / sqrt(pi)
  float sw_a, sw_b;       // t = sat(r2 * sw_a + sw_b)
  float dsw_k;            // 12 / (rc^2 - ron^2) / 6 (the LJ table in shared memory holds 6 eps4)
};

__host__ __device__ inline PairConst pair_const(const SysParams& p) {
  PairConst c;
  c.rc2 = p.rc2;
  c.beta = p.beta;
  c.eb2 = -p.beta * p.beta * kLog2e;
  c.p_b = kAS_p * p.beta;
  c.c2b = kTwoOverSqrtPi * p.beta;
  const float d = p.rc2 - p.ron2;
  c.sw_a = d > 0.f ? 1.f / d : 0.f;
  c.sw_b = d > 0.f ? -p.ron2 / d : 0.f;
  c.dsw_k = d > 0.f ? 2.f / d : 0.f;
  return c;
}

// force/r for one pair (FP32); returns 0 outside the cutoff or when masked.  ls.x is
// 6 eps4 (the shared-memory table is scaled by 6 when loaded), so with a6 = 6 eps4 s^6 and
// b6 = a6 s^6 the unswitched LJ force/r is (2 b6 - a6) / r^2 and the LJ energy
// (b6 - a6) / 6; both force parts share the 1 / r^2:
//   F/r = [(2 b6 - a6) sw + qq e^{-b^2 r^2} (erfc(br)/(r e^{-b^2 r^2}) + 2b/sqrt(pi))] / r^2
//         + (b6 - a6)/6 dsw
template <bool ENERGY>
__device__ __forceinline__ float pair_force(const PairConst& c, float r2, float qq, float2 ls, bool ok, float& ev,
                                            float& ee) {
  const float rinv = rsqrt_a(r2);
  const float r2inv = rinv * rinv;
  const float ex = ex2_a(r2 * c.eb2);                    // exp(-beta^2 r^2)
  const float tt = rcp_a(fmaf(c.p_b, r2 * rinv, 1.f));   // 1 / (1 + p beta r)
  const float poly = tt * fmaf(tt, fmaf(tt, fmaf(tt, fmaf(tt, kAS_a5, kAS_a4), kAS_a3), kAS_a2), kAS_a1);
  // erfc(beta r) = poly exp(-beta^2 r^2): F_C r / r^2 = qq exp(-beta^2 r^2) (poly / r + 2 beta/sqrt(pi)) / r^2
  const float qex = qq * ex;
  const float s2 = ls.y * r2inv;
  const float s6 = s2 * s2 * s2;
  const float a6 = ls.x * s6;
  const float e6 = fmaf(a6, s6, -a6);  // b6 - a6
  const float t = __saturatef(fmaf(r2, c.sw_a, c.sw_b));
  const float t2 = t * t;
  const float sw = fmaf(-t2, fmaf(-2.f, t, 3.f), 1.f);
  const float h = fmaf(fmaf(2.f, e6, a6), sw, qex * fmaf(poly, rinv, c.c2b));
  const float fr = fmaf(h, r2inv, e6 * ((t - t2) * c.dsw_k));
  if (ENERGY) {
    ev += ok ? e6 * sw * (1.f / 6.f) : 0.f;
    ee += ok ? qex * poly * rinv : 0.f;
  }
  return ok ? fr : 0.f;
}

// One tile of kIG i atoms x 32 j entries (xj, tyj: this lane's entry, loaded by the
// caller one tile ahead).  Lane = seg * kIL + il holds i atoms il and il + kIL of the
// group and works on segment seg of the j entries (kIL of them); the tile's j data
// (image shift applied) are staged in this warp's shared ring, doubled within each
// segment, so at step k lane il reads entry seg * kIL + (il + k) % kIL at a constant
// offset for both of its i atoms; the i forces stay in registers, each j force
// accumulator takes both pairs of the step, then rotates through its segment (3
// width-kIL shuffles per two pairs) and is back on the lane that loaded the entry
// after kIL steps.  Two i atoms a lane against one: per pair half the ring loads and
// half the shuffles, and two independent chains of arithmetic.
// ex0, ex1: bit e set when entry e is excluded for i atom il / il + kIL.
constexpr int kIL = kIG / 2;        // lanes across the i atoms
constexpr int kSeg = 32 / kIL;      // j segments of a tile
constexpr int kTyStride = 3 * kIL;  // ring of j types: segments on different banks

template <bool ENERGY>
__device__ __forceinline__ float pair_step(const PairConst& c, const float4& xi, float qi, const char* ljrow,
                                           const float4& b, int tyb, bool allowed, float& dx, float& dy, float& dz,
                                           float& fx, float& fy, float& fz, float& ev, float& ee, float* vir) {
  dx = xi.x - b.x;
  dy = xi.y - b.y;
  dz = xi.z - b.z;
  const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
  const float2 ls = *reinterpret_cast<const float2*>(ljrow + tyb);
  const float fr = pair_force<ENERGY>(c, r2, qi * b.w, ls, r2 < c.rc2 && allowed, ev, ee);
  if (ENERGY) {
    vir[0] = fmaf(fr * dx, dx, vir[0]);
    vir[1] = fmaf(fr * dy, dy, vir[1]);
    vir[2] = fmaf(fr * dz, dz, vir[2]);
  }
  fx = fmaf(fr, dx, fx);
  fy = fmaf(fr, dy, fy);
  fz = fmaf(fr, dz, fz);
  return fr;
}

template <bool ENERGY, bool MASKED>
__device__ __forceinline__ void tile_steps(const PairConst& c, const float4& x0, const float4& x1, float q0, float q1,
                                           const char* lj0, const char* lj1, uint32_t m0, uint32_t m1,
                                           const float4* jxl, const int* jtl, int src, float* f0, float* f1, float& ev,
                                           float& ee, float* vir, float& fjx, float& fjy, float& fjz) {
  // the common loop whole, the rare one rolled: the two must stay in the instruction cache
  // together (both whole: 47 % of the stalls were instruction fetches, 1.4 times the time)
  constexpr int kUnroll = MASKED ? 1 : kIL;
#pragma unroll kUnroll
  for (int k = 0; k < kIL; ++k) {
    const float4 b = jxl[k];
    const int ty = jtl[k];
    float dx, dy, dz, ex, ey, ez;
    const float fa = pair_step<ENERGY>(c, x0, q0, lj0, b, ty, !MASKED || !((m0 >> k) & 1u), dx, dy, dz, f0[0], f0[1],
                                       f0[2], ev, ee, vir);
    const float fb = pair_step<ENERGY>(c, x1, q1, lj1, b, ty, !MASKED || !((m1 >> k) & 1u), ex, ey, ez, f1[0], f1[1],
                                       f1[2], ev, ee, vir);
    fjx = __shfl_sync(0xffffffffu, fmaf(-fb, ex, fmaf(-fa, dx, fjx)), src, kIL);
    fjy = __shfl_sync(0xffffffffu, fmaf(-fb, ey, fmaf(-fa, dy, fjy)), src, kIL);
    fjz = __shfl_sync(0xffffffffu, fmaf(-fb, ez, fmaf(-fa, dz, fjz)), src, kIL);
  }
}

// bits of segment seg of an exclusion word, rotated so that bit k belongs to step k
__device__ __forceinline__ uint32_t seg_mask(uint32_t excl, int seg, int il) {
  constexpr uint32_t m = (1u << kIL) - 1u;
  const uint32_t w = (excl >> (seg * kIL)) & m;
  return ((w >> il) | (w << (kIL - il))) & m;
}

template <bool ENERGY>
__device__ __forceinline__ void run_tile(const PairConst& c, const SysParams& p, const float4& x0, const float4& x1,
                                         float q0, float q1, const char* lj0, const char* lj1, uint32_t je,
                                         uint32_t ex0, uint32_t ex1, float4 xj, int tyj, float4* jx, int* jt,
                                         const int* __restrict__ perm, long long* __restrict__ facc, int lane, int src,
                                         float* f0, float* f1, float& ev, float& ee, float* vir) {
  const int jslot = (int)(je & kSlotMask);
  const int code = (int)(je >> kSlotBits);
  const int aj = perm[jslot];  // needed at the tile's end: asked for now
  if (code != kNoShift) {
    const float3 s = shift_of(code, p);
    xj.x += s.x;
    xj.y += s.y;
    xj.z += s.z;
  }
  const int il = lane & (kIL - 1), seg = lane / kIL;
  float4* jxs = jx + seg * 2 * kIL + il;
  int* jts = jt + seg * kTyStride + il;
  __syncwarp();
  jxs[0] = xj;
  jxs[kIL] = xj;
  jts[0] = tyj * (int)sizeof(float2);
  jts[kIL] = tyj * (int)sizeof(float2);
  __syncwarp();
  const uint32_t m0 = seg_mask(ex0, seg, il), m1 = seg_mask(ex1, seg, il);
  float fjx = 0.f, fjy = 0.f, fjz = 0.f;
  if (__any_sync(0xffffffffu, (m0 | m1) != 0u))
    tile_steps<ENERGY, true>(c, x0, x1, q0, q1, lj0, lj1, m0, m1, jxs, jts, src, f0, f1, ev, ee, vir, fjx, fjy, fjz);
  else
    tile_steps<ENERGY, false>(c, x0, x1, q0, q1, lj0, lj1, 0u, 0u, jxs, jts, src, f0, f1, ev, ee, vir, fjx, fjy, fjz);
  if (aj >= 0) {
    const int n = p.n;
    red_add(facc + aj, to_fix(fjx));
    red_add(facc + n + aj, to_fix(fjy));
    red_add(facc + 2 * n + aj, to_fix(fjz));
  }
}

// A warp per work item, `chunk` tiles of one i-group (the first item by the warp's own number,
// further ones from a counter): the diagonal tile, then the group's inner tiles; the i forces
// stay in registers across the item's tiles and are flushed once.
template <bool ENERGY>
__device__ __forceinline__ void nonbonded_body(const SysParams& p, const PairConst& c, const float4* __restrict__ xyzq, const int* __restrict__ typ,
    const int* __restrict__ perm, const uint32_t* __restrict__ inner, const int* __restrict__ inner_nt,
    const int* __restrict__ inner_m, const uint32_t* __restrict__ dmask, const uint32_t* __restrict__ masks,
    int* __restrict__ counters, const int2* __restrict__ items, int chunk, const float2* __restrict__ ljtab,
    long long* __restrict__ facc, long long* __restrict__ energy, int ocap, int* closing, int* closing_prune, int bid, int nbid) {
  griddep_wait();
  if (closing && threadIdx.x == 0) lists_close(closing, closing_prune, counters);
  extern __shared__ float2 lj[];
  __shared__ float4 jx_all[kWarps][64];
  __shared__ int jt_all[kWarps][kSeg * kTyStride];
  const int nt1 = p.ntypes + 1;
  for (int k = threadIdx.x; k < nt1 * nt1; k += blockDim.x) lj[k] = make_float2(6.f * ljtab[k].x, ljtab[k].y);
  __syncthreads();
  const int nitems = counters[CNT_ITEMS];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float4* jx = jx_all[warp];
  int* jt = jt_all[warp];
  const int n = p.n;
  const int il = lane & (kIL - 1);
  const int src = (il + 1) & (kIL - 1);  // segment-relative source lane of the j-force rotation
  // energy and virial sums per lane in fixed point, item by item: integer sums do not
  // depend on which items a warp happens to fetch, so energies are bit-reproducible
  long long e_vdw = 0, e_el = 0, w_acc[3] = {0, 0, 0};
  // Work items: a warp starts with the item of its own number and takes further ones
  // from the counter, each asked for while the last tile of the one before is worked on
  // (asked for earlier, a warp holds an item that another could start on).  All warps
  // starting at the counter queue at one L2 address: 3,500 warps for the few hundred
  // items of a 648-atom system.
  const int nwarps = nbid * kWarps;
  int it = bid * kWarps + warp;
  int2 item = it < nitems ? items[it] : make_int2(0, 0);
  while (it < nitems) {
    int it_next = nitems;
    const int g = item.x, t_first = item.y;  // i-group: block I, atoms s * kIG .. s * kIG + kIG - 1
    const int I = g / kNG, s = g % kNG;
    const int ib = s * kIG + il;  // this lane's first i atom, index within the block; the second is ib + kIL
    const int islot = I * 32 + ib;
    const float4 x0 = xyzq[islot], x1 = xyzq[islot + kIL];
    const char* lj0 = reinterpret_cast<const char*>(lj + typ[islot] * nt1);
    const char* lj1 = reinterpret_cast<const char*>(lj + typ[islot + kIL] * nt1);
    const int ai = lane < kIG ? perm[I * 32 + s * kIG + lane] : -1;
    const float q0 = x0.w * p.cc, q1 = x1.w * p.cc;
    float f0[3] = {0.f, 0.f, 0.f}, f1[3] = {0.f, 0.f, 0.f};
    float ev = 0.f, ee = 0.f, vir[3] = {0.f, 0.f, 0.f};
    // tile 0 of a group is the group against its own block (upper triangle j > i);
    // each tile's entry, exclusion word and j data are loaded one tile ahead
    int t = t_first;
    const int tend = min(inner_nt[g] + 1, t + chunk);
    const uint32_t* jl = inner + (size_t)g * ocap - 32;  // inner tile t-1
    const int* ml = inner_m + (size_t)g * (ocap >> 5) - 1;
    // (and the entry of the tile after that, so that no load waits for its own address)
    auto entry = [&](int tt) {
      return tt == 0 ? (uint32_t)(I * 32 + lane) | ((uint32_t)kNoShift << kSlotBits) : jl[tt * 32 + lane];
    };
    auto fetch = [&](int tt, uint32_t je, uint32_t& ex0, uint32_t& ex1, float4& xj, int& tyj) {
      if (tt == 0) {
        ex0 = dmask[islot] | ((2u << ib) - 1u);
        ex1 = dmask[islot + kIL] | ((ib + kIL == 31) ? 0xffffffffu : ((2u << (ib + kIL)) - 1u));
      } else {
        const int m = ml[tt];
        ex0 = m >= 0 ? masks[(size_t)m * kIG + il] : 0u;
        ex1 = m >= 0 ? masks[(size_t)m * kIG + il + kIL] : 0u;
      }
      xj = xyzq[je & kSlotMask];
      tyj = typ[je & kSlotMask];
    };
    uint32_t je_n = entry(t), je_n2 = t + 1 < tend ? entry(t + 1) : 0u, e0_n, e1_n;
    float4 xj_n;
    int ty_n;
    fetch(t, je_n, e0_n, e1_n, xj_n, ty_n);
    for (; t < tend; ++t) {
      const uint32_t je = je_n, e0 = e0_n, e1 = e1_n;
      const float4 xj = xj_n;
      const int ty = ty_n;
      if (t + 1 < tend) {
        je_n = je_n2;
        fetch(t + 1, je_n, e0_n, e1_n, xj_n, ty_n);
        if (t + 2 < tend) je_n2 = entry(t + 2);
      } else if (nitems > nwarps && lane == 0) {
        it_next = nwarps + atomicAdd(&counters[CNT_WORK], 1);
      }
      run_tile<ENERGY>(c, p, x0, x1, q0, q1, lj0, lj1, je, e0, e1, xj, ty, jx, jt, perm, facc, lane, src, f0, f1, ev,
                       ee, vir);
    }
    it = __shfl_sync(0xffffffffu, it_next, 0);
    if (it < nitems) item = items[it];
    // the i forces are split over the segments; then lane l < kIG flushes i atom l
#pragma unroll
    for (int d = 0; d < 3; ++d) {
#pragma unroll
      for (int off = kIL; off < 32; off <<= 1) {
        f0[d] += __shfl_xor_sync(0xffffffffu, f0[d], off);
        f1[d] += __shfl_xor_sync(0xffffffffu, f1[d], off);
      }
    }
    const bool second = lane >= kIL;
    if (ai >= 0) {
      red_add(facc + ai, to_fix(second ? f1[0] : f0[0]));
      red_add(facc + n + ai, to_fix(second ? f1[1] : f0[1]));
      red_add(facc + 2 * n + ai, to_fix(second ? f1[2] : f0[2]));
    }
    if (ENERGY) {
      e_vdw += __double2ll_rn((double)ev * kFixE);
      e_el += __double2ll_rn((double)ee * kFixE);
      for (int d = 0; d < 3; ++d) w_acc[d] += __double2ll_rn((double)vir[d] * kFixE);
    }
  }
  if (ENERGY) {
    energy_add_fix(energy + EN_VDW, e_vdw);
    energy_add_fix(energy + EN_ELEC, e_el);
    energy_add_fix(energy + EN_VIR_X, w_acc[0]);
    energy_add_fix(energy + EN_VIR_Y, w_acc[1]);
    energy_add_fix(energy + EN_VIR_Z, w_acc[2]);
  }
}

template <bool ENERGY, int MINB>
__global__ void __launch_bounds__(256, MINB)
    k_nonbonded(SysParams p, PairConst c, const float4* __restrict__ xyzq, const int* __restrict__ typ,
                const int* __restrict__ perm, const uint32_t* __restrict__ inner, const int* __restrict__ inner_nt,
                const int* __restrict__ inner_m, const uint32_t* __restrict__ dmask,
                const uint32_t* __restrict__ masks, int* __restrict__ counters, const int2* __restrict__ items,
                int chunk, const float2* __restrict__ ljtab, long long* __restrict__ facc,
                long long* __restrict__ energy, int ocap, int* flag, int* flag_prune) { griddep_wait();
  nonbonded_body<ENERGY>(p, c, xyzq, typ, perm, inner, inner_nt, inner_m, dmask, masks, counters, items, chunk, ljtab,
                         facc, energy, ocap, blockIdx.x == 0 ? flag : nullptr, flag_prune, blockIdx.x, gridDim.x);
}

// batched: every CTA serves one system's work queue (force variant only)
__global__ void __launch_bounds__(256, kNbBatchCtasPerSm) k_nonbonded_b(const NonbondedArgs* __restrict__ args,
                                                        const int4* __restrict__ tab) { griddep_wait();
  const int4 t = tab[blockIdx.x];
  const NonbondedArgs a = args[t.x];
  const PairConst c = pair_const(a.p);
  nonbonded_body<false>(a.p, c, a.xyzq_s, a.typ_s, a.perm, a.inner, a.inner_nt, a.inner_m, a.dmask, a.masks,
                        a.counters, a.items, a.chunk, a.ljtab, a.facc, a.energy, a.ocap,
                        t.y == 0 ? a.flag : nullptr, a.flag_prune, t.y, t.z);
}

void launch_nonbonded(const NonbondedArgs& a, bool energy, cudaStream_t st, bool zero_work) {
  const int nt1 = a.p.ntypes + 1;
  const size_t smem = (size_t)nt1 * nt1 * sizeof(float2);
  const PairConst c = pair_const(a.p);
  if (zero_work) cudaMemsetAsync(a.counters + CNT_WORK, 0, sizeof(int), st);
  // 3 CTAs per SM fit 80 registers a thread; the 4-CTA build is held to 64
  auto k = energy ? (a.minb >= 4 ? k_nonbonded<true, 4> : k_nonbonded<true, 3>)
                  : (a.minb >= 4 ? k_nonbonded<false, 4> : k_nonbonded<false, 3>);
  launch_pdl(k, dim3(a.grid), dim3(kWarps * 32), smem, st, a.p, c, a.xyzq_s, a.typ_s, a.perm, a.inner, a.inner_nt, a.inner_m, a.dmask,
                                       a.masks, a.counters, a.items, a.chunk, a.ljtab, a.facc, a.energy, a.ocap,
                                       a.close_lists ? a.flag : nullptr, a.flag_prune);
}

void launch_nonbonded_b(const NonbondedArgs* args, const BatchTables& t, int max_ntypes, cudaStream_t st) {
  const size_t smem = (size_t)(max_ntypes + 1) * (max_ntypes + 1) * sizeof(float2);
  launch_pdl(k_nonbonded_b, dim3(t.n[BT_NB]), dim3(kWarps * 32), smem, st, args, t.tab[BT_NB]);
}

}  // namespace fzk
