// post.cuh -- post_process (DG_solver.f90:128-661) as sm_100a kernels.
//
//   pp_avg_ldf_kernel   loop 1 (DG_solver.f90:161-277): cell averages of every interior and
//                       non-corner ghost element, admissibility of the average, the LDF projection
//                       of (Bx,By) as one dense nodal operator.  In the time-step pipeline a stage
//                       without OEDG also runs loop 3 here (fused), and the stages after the first
//                       mostly run loops 1 and 3 in the previous residual (stage_post, residual.cuh).
//   pp_reduce_kernel    the global average sum in a fixed order (DG_solver.f90:227-229,282-286).
//   pp_sigsum_kernel    the OEDG face jump indicators OEDG_sigsum_x/y (DG_solver.f90:295-422), and
//                       the max and min of the post-LDF interior node values (read from the tile
//                       it stages anyway).
//   pp_limit_kernel     loop 3 (DG_solver.f90:428-656): OEDG damping, with u_vari_global
//                       (DG_solver.f90:287-294) = max|u - g| = max(umax - g, g - umin) (rounding
//                       is monotone), Zhang-Shu positivity
//                       scaling with its bounded re-limit loop, entropy-offset limiting, cell
//                       entropy (segment partials, fixed order); in the time-step pipeline the
//                       final stage's result goes to u_con only (the accepted state).
//   pp_entsum_kernel    total entropy from the partials (fixed order).
//   stage_end_bc_kernel the end of a stage of the time-step pipeline in one launch: the entropy sum
//                       (final stage), the stage-end decision, the next stage's pseudo-time and
//                       the ghost fill of the stage state.
//
// Loops 1 and 3 work element-locally, so they map one element to a group of lanes of a warp (GS
// in loop 1, GSL in the limiter kernel; PPCfg), one lane per GLL node, each lane holding its node's
// 8 variables in registers.  Loads and stores of a variable are then 8*NN-byte runs per group
// (coalesced), per-element sums, minima and maxima are reductions inside the group (butterflies for
// power-of-two groups, a fold plus a butterfly for the 9-lane groups; every lane ends with the same
// value), and no CTA-wide barrier sits between the steps of one element.  A CTA of NT threads handles
// a chunk of TE = (NT/32) * (32/GS) consecutive elements.  The single-instance loop-1 kernel is a
// persistent grid over the chunks in which each warp copies its elements of the next
// chunk into shared memory (cp.async) while it works on the current one.  In the first stage of
// a time step loop 1 also forms the stage state from u_con and k1 (Stage1Src).  The indicator
// kernel stages each tile of elements in shared memory with cp.async, row by row.
#pragma once
#include "common.cuh"
#include "misc.cuh"

namespace mhd {

constexpr unsigned FULL_MASK = 0xffffffffu;

// Per degree: threads per CTA and CTAs per SM (the register budget) of the loop-1 and loop-3
// kernels (MHD_PP_CFG<p> = NT, MINB), and the element tile and CTAs per SM of the OEDG indicator
// kernel (MHD_SIG_CFG<p> = TX, TY, MINB).  autotune.py times candidates on the GPU at hand and
// writes post_tuned.h, which takes precedence when present.
#if __has_include("post_tuned.h")
#include "post_tuned.h"
#endif
#ifndef MHD_PP_CFG1
#define MHD_PP_CFG1 256, 4
#endif
#ifndef MHD_PP_CFG2
#define MHD_PP_CFG2 256, 4
#endif
#ifndef MHD_PP_CFG3
#define MHD_PP_CFG3 256, 4
#endif
#ifndef MHD_SIG_CFG1
#define MHD_SIG_CFG1 16, 4, 4
#endif
#ifndef MHD_SIG_CFG2
#define MHD_SIG_CFG2 8, 4, 5
#endif
#ifndef MHD_SIG_CFG3
#define MHD_SIG_CFG3 4, 4, 4
#endif
struct PPParams {
  int NT, MINB;
};
struct SigParams {
  int TX, TY, MINB;
};
template <int P>
struct PPTune;
template <>
struct PPTune<1> {
  static constexpr PPParams pp{MHD_PP_CFG1};
  static constexpr SigParams sig{MHD_SIG_CFG1};
};
template <>
struct PPTune<2> {
  static constexpr PPParams pp{MHD_PP_CFG2};
  static constexpr SigParams sig{MHD_SIG_CFG2};
};
template <>
struct PPTune<3> {
  static constexpr PPParams pp{MHD_PP_CFG3};
  static constexpr SigParams sig{MHD_SIG_CFG3};
};

// Lanes per element: loop 1 takes a power-of-two group of GS lanes (16 for the 9 nodes of p = 2);
// the final stage's limiter kernel takes GSL lanes, 9 at p = 2 (three elements per warp, lanes
// 27-31 idle), where its per-node work outweighs the dearer reductions of a 9-lane group (measured
// on the 400x400 p = 2 blast: limiter 0.115 -> 0.088 ms; loop 1 with 9-lane groups and its cell
// sums through shared memory was 3 % slower and stays at 16 lanes).
template <int P>
struct PPCfg {
  static constexpr int N = P + 1, NN = N * N, EB = 8 * NN, N2 = 2 * NN;
  static constexpr int NT = PPTune<P>::pp.NT, MINB = PPTune<P>::pp.MINB;
  static constexpr int GS = NN <= 4 ? 4 : (NN <= 8 ? 8 : (NN <= 16 ? 16 : 32));  // loop 1: lanes per element
  static constexpr int G = 32 / GS;                                               // elements per warp
  static constexpr int TE = (NT / 32) * G;                                        // elements per CTA chunk
  static constexpr int GSL = NN == 9 ? 9 : GS;                                    // limiter kernel: lanes per element
  static constexpr int GL = 32 / GSL;
  static constexpr int TEL = (NT / 32) * GL;                                      // elements per limiter CTA
  static_assert(NT % 32 == 0 && NT <= 1024, "whole warps");
};

// This lane's group and node for groups of GS lanes.  Where GS does not divide 32 the lanes past
// the last group are idle: they take group 0's lanes as partners in the group reductions (their
// results are unused) and a node number beyond every element (node >= NN).
template <int GS>
struct GrpLane {
  int grp, node;
  bool idle;
};
template <int GS>
__device__ __forceinline__ GrpLane<GS> grp_lane() {
  const int lane = threadIdx.x & 31, g = lane / GS;
  const bool idle = g >= 32 / GS;
  return GrpLane<GS>{idle ? 0 : g, idle ? lane : lane - g * GS, idle};
}
// the smallest chunk of any degree: per-chunk partial buffers are sized by it
constexpr int pp_min_chunk() {
  return PPCfg<1>::TE < PPCfg<2>::TE ? (PPCfg<1>::TE < PPCfg<3>::TE ? PPCfg<1>::TE : PPCfg<3>::TE)
                                     : (PPCfg<2>::TE < PPCfg<3>::TE ? PPCfg<2>::TE : PPCfg<3>::TE);
}

// global -> shared copies that do not pass through registers (cp.async, sm_80 and later): 8 bytes,
// or 16 bytes with both addresses 16-byte aligned
__device__ __forceinline__ void cp_async8(double* dst_shared, const double* src_global) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(dst_shared);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(sa), "l"(src_global) : "memory");
}
__device__ __forceinline__ void cp_async16(double* dst_shared, const double* src_global) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(dst_shared);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(src_global) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

// Reduction over a group of GS lanes, the result in every lane of the group.  A power-of-two group
// uses the xor butterfly.  Otherwise (GS = 9) the lanes past the largest power of two P2 are
// folded onto the group's first lanes, the P2 lanes reduce by a butterfly with partners inside the
// group (explicit lane indices), and every lane takes the group's first lane's result: a fixed
// order, and one value for the whole group.
template <int GS, class Op>
__device__ __forceinline__ double grp_reduce(double v, Op op) {
  if constexpr ((GS & (GS - 1)) == 0) {
#pragma unroll
    for (int o = GS / 2; o > 0; o >>= 1) v = op(v, __shfl_xor_sync(FULL_MASK, v, o));
    return v;
  } else {
    constexpr int P2 = GS >= 16 ? 16 : (GS >= 8 ? 8 : (GS >= 4 ? 4 : 2));
    static_assert(GS - P2 <= P2, "one fold");
    const GrpLane<GS> gl = grp_lane<GS>();
    const int gb = gl.grp * GS, node = gl.node;
    const double hi = __shfl_sync(FULL_MASK, v, gb + (node + P2 < GS ? node + P2 : 0));
    if (node + P2 < GS) v = op(v, hi);
#pragma unroll
    for (int o = P2 / 2; o > 0; o >>= 1) v = op(v, __shfl_sync(FULL_MASK, v, gb + ((node ^ o) & (P2 - 1))));
    return __shfl_sync(FULL_MASK, v, gb);
  }
}
struct OpAdd {
  __device__ __forceinline__ double operator()(double a, double b) const { return a + b; }
};
struct OpMin {
  __device__ __forceinline__ double operator()(double a, double b) const { return fmin(a, b); }
};
struct OpMax {
  __device__ __forceinline__ double operator()(double a, double b) const { return fmax(a, b); }
};
template <int GS>
__device__ __forceinline__ double grp_sum(double v) { return grp_reduce<GS>(v, OpAdd{}); }
template <int GS>
__device__ __forceinline__ double grp_min(double v) { return grp_reduce<GS>(v, OpMin{}); }
template <int GS>
__device__ __forceinline__ double grp_max(double v) { return grp_reduce<GS>(v, OpMax{}); }

// Maximum over a group of values that are not negative (NaN counts as zero).  Such doubles order as
// their bit patterns do, so groups of more than four lanes take the maximum of the upper words and then
// of the lower words among the lanes that hold it, by the warp's integer reduction (two instead of
// four exchanges of a double with a comparison each).
template <int GS>
__device__ __forceinline__ double grp_max_nonneg(double v) {
  v = at_least(v, 0.0);
  if constexpr (GS <= 4) {
    return grp_max<GS>(v);
  } else {
    const GrpLane<GS> gl = grp_lane<GS>();
    const unsigned all = (0xffffffffu >> (32 - GS)) << (gl.grp * GS);
    const unsigned mask = gl.idle ? 0xffffffffu << (32 / GS * GS & 31) : all;  // idle lanes among themselves
    const unsigned hi = (unsigned)__double2hiint(v), lo = (unsigned)__double2loint(v);
    const unsigned mh = __reduce_max_sync(mask, hi);
    const unsigned ml = __reduce_max_sync(mask, hi == mh ? lo : 0u);
    return __hiloint2double((int)mh, (int)ml);
  }
}

// All eight sums of a[0..7] over each group of GS lanes, in every lane of the group, by a
// reduce-scatter (each exchange halves the values a lane carries, one lane bit per level: 8
// exchanges at GS = 16 instead of 8 butterflies of 4) and an all-gather through the group's
// shared row `row` (8 doubles, 16-byte aligned; they stay there: the caller's __syncwarp comes before
// the row is rewritten).  Deterministic, and every lane of a group ends with the same sums
// (each final sum is formed in one lane pair as x + y and y + x, which IEEE addition makes equal,
// and read from the one copy in `row`).
template <int GS>
__device__ __forceinline__ void grp_sum8(double* a, double* row) {
  static_assert((GS & (GS - 1)) == 0, "power-of-two groups");
  constexpr int LV = GS >= 8 ? 3 : (GS == 4 ? 2 : 1);  // halving levels
  const int lane = threadIdx.x & 31;
  constexpr int CNT = 8 >> LV;                          // values a lane keeps after them
#pragma unroll
  for (int j = 0; j < LV; ++j) {
    const int o = GS >> (j + 1);
    const int half = 4 >> j;
    const bool hi = (lane & o) != 0;
#pragma unroll
    for (int i = 0; i < half; ++i) {
      const double send = hi ? a[i] : a[i + half];
      const double recv = __shfl_xor_sync(FULL_MASK, send, o);
      a[i] = (hi ? a[i + half] : a[i]) + recv;
    }
  }
#pragma unroll
  for (int o = GS >> (LV + 1); o > 0; o >>= 1)
#pragma unroll
    for (int i = 0; i < CNT; ++i) a[i] = a[i] + __shfl_xor_sync(FULL_MASK, a[i], o);
  // all-gather through the group's shared row: the lane that holds variables vb..vb+CNT-1 (and
  // whose low bits are zero) writes them, every lane reads all 8
  int vb = 0;
#pragma unroll
  for (int j = 0; j < LV; ++j)
    if (lane & (GS >> (j + 1))) vb += 4 >> j;
  if ((lane & ((GS >> LV) - 1)) == 0)
#pragma unroll
    for (int i = 0; i < CNT; ++i) row[vb + i] = a[i];
  __syncwarp();
#pragma unroll
  for (int v = 0; v < 8; v += 2) {
    const double2 t = *reinterpret_cast<const double2*>(row + v);
    a[v] = t.x;
    a[v + 1] = t.y;
  }
}

__device__ __forceinline__ double node_prs(const double* x, double gamma) {
  return prs_of(x[0], x[1], x[2], x[3], x[4], x[5], x[6], x[7], gamma);
}

// ---------------------------------------------------------------------------------------------
// Loop 3 for the element of this lane's group (DG_solver.f90:526-649): Zhang-Shu positivity with
// its bounded re-limit loop, entropy-offset limiting, and the cell entropy.  x = this lane's node,
// avg = the element average (all lanes of the group), node = lane's node (active = node < NN and
// the group's element is limited).  Every lane of the warp calls this (the group reductions need
// the whole warp); returns the cell entropy (0 where not computed) and sets *negcell.  GS: lanes
// per element of the caller's layout.
// ---------------------------------------------------------------------------------------------
template <int P, int GS = PPCfg<P>::GS>
__device__ __forceinline__ double limit_group(double* x, const double* avg, bool active, bool lead, int node,
                                              long long ce, const Geo& g, Ctrl* ctrl, int ent_offset,
                                              int comput_ent, const double* __restrict__ cell_ent_DG,
                                              const double* __restrict__ cell_ent_FV,
                                              const unsigned char* __restrict__ cell_ent_nan, bool* negcell,
                                              bool* scaled = nullptr) {
  using C = PPCfg<P>;
  constexpr int N = C::N;
  constexpr double BIG = 1.7976931348623157e308;
  const double gamma = g.gamma;
  const DegConst& dc = c_deg[P];
  // density: theta from the minimum nodal density (DG_solver.f90:538-553).  The minimum only
  // matters below PP_EPS, so the reduction runs only when some lane of the warp is below it.
  double thd = -1.0;
  if (__any_sync(FULL_MASK, active && x[0] < PP_EPS)) {
    const double den_min = grp_min<GS>(active ? x[0] : BIG);
    if (den_min < PP_EPS) thd = fmax(fmin((avg[0] - PP_EPS) / (avg[0] - den_min), 1.0), 0.0);
  }
  if (active && thd >= 0.0) x[0] = fmax(avg[0] + thd * (x[0] - avg[0]), PP_EPS);
  // pressure: theta from the minimum nodal pressure (DG_solver.f90:556-571), likewise
  const double pq = active ? node_prs(x, gamma) : BIG;
  double pmin = BIG;
  if (__any_sync(FULL_MASK, pq < PP_EPS)) pmin = grp_min<GS>(pq);
  double thp = -1.0;
  if (pmin < PP_EPS) {
    const double pa = prs_of(avg[0], avg[1], avg[2], avg[3], avg[4], avg[5], avg[6], avg[7], gamma);
    thp = fmax(fmin((pa - PP_EPS) / (pa - pmin), 1.0), 0.0);
  }
  *negcell = lead && active && (thd >= 0.0 || thp >= 0.0);  // neg_node (DG_solver.f90:602)
  if (scaled) *scaled = active && (thd >= 0.0 || thp >= 0.0);  // this lane's node values changed
  if (active && thp >= 0.0)
#pragma unroll
    for (int v = 0; v < 8; ++v) x[v] = avg[v] + thp * (x[v] - avg[v]);
  // re-check after the FP-inexact theta (DG_solver.f90:573-599): at most two extra shrinks; the
  // loop runs while any group of the warp still checks, so that the reductions see the whole warp
  bool pending = active && thp >= 0.0;
  double theta = thp;
  for (int it_count = 0; __any_sync(FULL_MASK, pending); ++it_count) {
    const double pm = grp_min<GS>(pending ? node_prs(x, gamma) : BIG);
    if (pending) {
      if (!(pm < 0.99 * PP_EPS)) {
        pending = false;
      } else if (it_count > 1) {
        if (lead) atomicOr(&ctrl->pp_relimit, 1);
        pending = false;
      } else {
        theta = 0.6 * theta;
#pragma unroll
        for (int v = 0; v < 8; ++v) x[v] = avg[v] + theta * (x[v] - avg[v]);
      }
    }
  }
  const int k = node % N, l = node / N;
  const double wq = (node < C::NN) ? 0.25 * g.hx * g.hy * dc.qw[k] * dc.qw[l] : 0.0;
  // entropy-offset limiter (DG_solver.f90:606-633)
  if (ent_offset) {
    const bool use = active && !cell_ent_nan[ce];
    const double nw = grp_sum<GS>(use ? wq * ent_of(x[0], at_least(node_prs(x, gamma), PP_EPS), gamma, g.igm1) : 0.0);
    if (use) {
      const double old = cell_ent_DG[ce], eavg = cell_ent_FV[ce];
      if (nw > old) {
        const double th = fmax(fmin((old - eavg) / (nw - eavg), 1.0), 0.0);
#pragma unroll
        for (int v = 0; v < 8; ++v) x[v] = avg[v] + th * (x[v] - avg[v]);
        if (scaled) *scaled = true;
      }
    }
  }
  // cell entropy (DG_solver.f90:635-649)
  if (comput_ent) return grp_sum<GS>(active ? wq * ent_of(x[0], at_least(node_prs(x, gamma), PP_EPS), gamma, g.igm1) : 0.0);
  return 0.0;
}

// ---------------------------------------------------------------------------------------------
// LDF projection of one element's (Bx - avg, By - avg), in place: (bx, by) = this lane's node.  It works
// on the sums and differences of mirror nodes (tables.h, ldf_table): butterflies along x and y, this
// lane's output place from at most 2 M^2 input places through the group's row, butterflies back.  gb = the
// group's first lane, nd = this lane holds one of its nodes (the other lanes take part with their own
// value as partner), row = the group's 2 NN doubles, A = the table (shared or global memory).
//
// In loop 1 the shared-memory pipe is the bound, and the dense operator (2n^2 products an output) read
// its rows from there: 400^2 without / with the OEDG sums, p = 3: 92 -> 75 / 90 -> 61 us, p = 2: 77 -> 70 /
// 70 -> 61 us; p = 1, 500^2: 38.5 -> 37.7 us.
// ---------------------------------------------------------------------------------------------
template <int P>
__device__ __forceinline__ void ldf_project(double& bx, double& by, int gb, int node, bool nd, double* row,
                                            const double2* __restrict__ A) {
  constexpr int N = P + 1, NN = N * N, M = (N + 1) / 2;
  const int lane = threadIdx.x & 31, k = node % N, l = node / N;
  const int mx = nd ? gb + (N - 1 - k) + N * l : lane, my = nd ? gb + k + N * (N - 1 - l) : lane;
  const double sx = 2 * k < N - 1 ? 1.0 : (2 * k == N - 1 ? 0.0 : -1.0);
  const double sy = 2 * l < N - 1 ? 1.0 : (2 * l == N - 1 ? 0.0 : -1.0);
  bx = __fma_rn(sx, __shfl_sync(FULL_MASK, bx, mx), bx);
  by = __fma_rn(sx, __shfl_sync(FULL_MASK, by, mx), by);
  bx = __fma_rn(sy, __shfl_sync(FULL_MASK, bx, my), bx);
  by = __fma_rn(sy, __shfl_sync(FULL_MASK, by, my), by);
  double2* in = reinterpret_cast<double2*>(row);
  if (nd) in[node] = make_double2(bx, by);
  __syncwarp();
  double ox = 0.0, oy = 0.0;
  if (nd) {
    const double2* w = A + node;
    const bool px = 2 * k > N - 1, py = 2 * l > N - 1;  // the parity of this lane's place
#pragma unroll
    for (int jy = 0; jy < M; ++jy)
#pragma unroll
      for (int jx = 0; jx < M; ++jx) {
        const int s = jx + M * jy;
        const double2 c = w[s * NN], f = in[(px ? N - 1 - jx : jx) + N * (py ? N - 1 - jy : jy)];
        ox = __fma_rn(c.x, f.x, ox);
        oy = __fma_rn(c.y, f.y, oy);
        const double2 d = w[(s + M * M) * NN], h = in[(px ? jx : N - 1 - jx) + N * (py ? jy : N - 1 - jy)];
        ox = __fma_rn(d.x, h.y, ox);
        oy = __fma_rn(d.y, h.x, oy);
      }
  }
  __syncwarp();  // the row may be rewritten
  ox = __fma_rn(-sy, __shfl_sync(FULL_MASK, ox, my), ox);
  oy = __fma_rn(-sy, __shfl_sync(FULL_MASK, oy, my), oy);
  bx = __fma_rn(-sx, __shfl_sync(FULL_MASK, ox, mx), ox);
  by = __fma_rn(-sx, __shfl_sync(FULL_MASK, oy, mx), oy);
}

// ---------------------------------------------------------------------------------------------
// loop 1 for one chunk of TE consecutive element blocks of the ghosted grid (one contiguous run of
// memory).  s_A = the LDF table in shared memory (load_ldf).
//
// LIMIT fuses loop 3 for a stage without OEDG and without the entropy sum: the interior
// elements are limited in registers before the one write-back.  The reference skips loop 3
// altogether when any element has an inadmissible average (neg_avg); here other CTAs may already
// have limited their elements by then.  That is only allowed where the stage result is discarded
// on neg_avg (the time-step pipeline re-tries the step from u_con), so the stand-alone
// post_process never fuses.
// ---------------------------------------------------------------------------------------------
// Stage-1 source of loop 1 (time-step pipeline only).  With u0 set, the stage state is formed
// here instead of being read from u: u0 + (coef*dt)*k1 on interior elements, rounded as
// combine_value rounds stage 1, and the ghost ring from those values by bc_source, as the boundary
// fill would leave it.  Every element is then written back, the inadmissible ones unchanged.
struct Stage1Src {
  const double* u0;  // state at the start of the step (ghosted layout)
  const double* k1;  // stage-1 residual (interior layout)
  const double* dt;
  double coef;       // 1 for SSP-RK(1,1), (2,2), (3,3); the first stage weight of SSP-RK(5,4)
};

template <int P>
__device__ __forceinline__ double stage1_node(const Stage1Src& s1, const Geo& g, int i, int j, bool inner, int v,
                                              int q, double dts) {
  constexpr int NN = (P + 1) * (P + 1), EB = 8 * NN;
  int si = i, sj = j, sq = q;
  bool neg = false;
  if (!inner) {
    const BcSrc b = bc_source<P>(g, i, j, v, q);
    if (b.fixed) return g.bc_state[v];
    si = b.si;
    sj = b.sj;
    sq = b.sq;
    neg = b.neg;
  }
  const long long gi = ((long long)sj * (g.nx + 2) + si) * EB + v * NN + sq;
  const long long ki = ((long long)(sj - 1) * g.nx + (si - 1)) * EB + v * NN + sq;
  const double x = __dadd_rn(s1.u0[gi], __dmul_rn(dts, s1.k1[ki]));
  return neg ? -x : x;
}

// Row and column of element e of the ghosted grid (rows of nxg elements) by one 32-bit division
// (the element count of any mesh that fits on the device is below 2^32; a 64-bit division by a
// run-time divisor is a long software sequence), and a position advanced along the rows.
struct GridRC {
  int j, i;
};
__device__ __forceinline__ GridRC grid_rc(long long e, int nxg) {
  const unsigned q = (unsigned)e / (unsigned)nxg;
  return GridRC{(int)q, (int)((unsigned)e - q * (unsigned)nxg)};
}
__device__ __forceinline__ GridRC grid_adv(GridRC p, int d, int nxg) {  // d >= 0 elements further
  p.i += d;
  while (p.i >= nxg) {
    p.i -= nxg;
    ++p.j;
  }
  return p;
}

// Queues this warp's elements of `chunk` into its shared buffers as one cp.async group (16-byte
// pieces; element blocks are multiples of 16 bytes): the blocks of u, or, with a stage-1 source,
// the blocks of u_con (bu) and k1 (bk) of the interior elements (ghost elements are formed from
// direct loads).  bu, bk: G * EB doubles each, 16-byte aligned.
template <int P>
__device__ __forceinline__ void pp_prefetch(const double* __restrict__ u, const Geo& g, long long chunk,
                                            GridRC cpos, const Stage1Src& s1, double* bu, double* bk) {
  using C = PPCfg<P>;
  constexpr int EB = C::EB, G = C::G, TE = C::TE, H2 = EB / 2;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nx = g.nx, NXG = nx + 2;
  const long long total = (long long)NXG * (g.ny + 2);
  const long long ef = chunk * TE + warp * G;  // the warp's first element (cpos: the chunk's first)
  const GridRC fp = grid_adv(cpos, warp * G, NXG);
  const int jf = fp.j, if_ = fp.i;
#pragma unroll
  for (int it = lane; it < G * H2; it += 32) {
    const int k = it / H2, o = 2 * (it - k * H2);
    const long long e = ef + k;
    if (e >= total) continue;
    if (!s1.u0) {
      cp_async16(bu + k * EB + o, u + e * EB + o);
    } else {
      int i = if_ + k, j = jf;
      while (i >= NXG) {
        i -= NXG;
        ++j;
      }
      if (i >= 1 && i <= nx && j >= 1 && j <= g.ny) {
        cp_async16(bu + k * EB + o, s1.u0 + e * EB + o);
        cp_async16(bk + k * EB + o, s1.k1 + ((long long)(j - 1) * nx + (i - 1)) * EB + o);
      }
    }
  }
  cp_async_commit();
}

template <int P, bool LIMIT, bool PF>
__device__ __forceinline__ void pp_avg_ldf_chunk(double* __restrict__ u, double* __restrict__ u_avg, const Geo& g,
                                                 Ctrl* ctrl, long long chunk, GridRC cpos, int apply_ldf, int ent_offset,
                                                 double* __restrict__ cell_ent_DG, double* __restrict__ cell_ent_FV,
                                                 unsigned char* __restrict__ cell_ent_nan,
                                                 const double* s_A, double* s_ldf, int* s_cnt,
                                                 const Stage1Src& s1,
                                                 double* bu, double* bk, long long next_chunk, GridRC npos) {
  using C = PPCfg<P>;
  constexpr int N = C::N, NN = C::NN, EB = C::EB, N2 = C::N2, GS = C::GS, G = C::G, TE = C::TE;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const GrpLane<GS> gl = grp_lane<GS>();
  const int grp = gl.grp, node = gl.node;
  const int nx = g.nx, ny = g.ny, NXG = nx + 2;
  const long long total = (long long)NXG * (ny + 2);
  const long long e0 = chunk * TE;
  const int ne = (int)min((long long)TE, total - e0);
  const int el = warp * G + grp;  // element of this group within the chunk
  const long long e = e0 + el;
  const DegConst& dc = c_deg[P];
  const double gamma = g.gamma;
  bool valid = false, inner = false;
  int i = 0, j = 0;
  if (el < ne && !gl.idle) {
    const GridRC me = grid_adv(cpos, el, NXG);  // cpos: the chunk's first element
    j = me.j;
    i = me.i;
    const bool ii = (i >= 1 && i <= nx), jj = (j >= 1 && j <= ny);
    valid = ii || jj;  // DG_solver.f90:165 (corners are skipped)
    inner = ii && jj;
  }
  const bool nd = node < NN;
  const bool act = valid && nd;
  double x[8];
  if (PF) {  // this chunk's blocks are in the warp's buffers (pp_prefetch)
    const double* pu = bu + grp * EB + node;
    const double* pk = bk + grp * EB + node;
    if (s1.u0) {
      const double dts = __dmul_rn(s1.coef, *s1.dt);
      if (inner && nd) {  // the common case, one branch for all eight variables
#pragma unroll
        for (int v = 0; v < 8; ++v) x[v] = __dadd_rn(pu[v * NN], __dmul_rn(dts, pk[v * NN]));
      } else if (act) {  // a ghost element
#pragma unroll
        for (int v = 0; v < 8; ++v) x[v] = stage1_node<P>(s1, g, i, j, false, v, node, dts);
      } else {
#pragma unroll
        for (int v = 0; v < 8; ++v) x[v] = 0.0;
      }
    } else {
#pragma unroll
      for (int v = 0; v < 8; ++v) x[v] = act ? pu[v * NN] : 0.0;
    }
    __syncwarp();  // every lane has read the buffers: queue the next chunk into them
    if (next_chunk >= 0) pp_prefetch<P>(u, g, next_chunk, npos, s1, bu, bk);
  } else if (s1.u0) {
    const double dts = __dmul_rn(s1.coef, *s1.dt);
    if (inner && nd) {  // an interior node: u_con and k1 at this node (stage1_node's interior case)
      const double* pu = s1.u0 + e * EB + node;
      const double* pk = s1.k1 + ((long long)(j - 1) * nx + (i - 1)) * EB + node;
#pragma unroll
      for (int v = 0; v < 8; ++v) x[v] = __dadd_rn(pu[v * NN], __dmul_rn(dts, pk[v * NN]));
    } else if (act) {  // a ghost element
#pragma unroll
      for (int v = 0; v < 8; ++v) x[v] = stage1_node<P>(s1, g, i, j, false, v, node, dts);
    } else {
#pragma unroll
      for (int v = 0; v < 8; ++v) x[v] = 0.0;
    }
  } else {
#pragma unroll
    for (int v = 0; v < 8; ++v) x[v] = act ? u[e * EB + v * NN + node] : 0.0;
  }
  // cell averages (DG_solver.f90:177-184)
  const int k = node % N, l = node / N;
  const double w = nd ? 0.25 * dc.qw[k] * dc.qw[l] : 0.0;
  double avg[8];
#pragma unroll
  for (int v = 0; v < 8; ++v) avg[v] = w * x[v];
  double* row = s_ldf + (warp * G + grp) * (N2 + 2);
  grp_sum8<GS>(avg, row);
  // the averages this lane stores below: variables node, node + GS, ...
  double mine[GS >= 8 ? 1 : 8 / GS];
#pragma unroll
  for (int v0 = 0; v0 < 8; v0 += GS) mine[v0 / GS] = row[(node + v0) & 7];
  __syncwarp();  // the row is rewritten next
  // admissibility of the average (DG_solver.f90:186-193): an inadmissible element is left unwritten
  if (valid) {
    const double prs = prs_of(avg[0], avg[1], avg[2], avg[3], avg[4], avg[5], avg[6], avg[7], gamma);
    if (avg[0] < PP_EPS || prs < PP_EPS) {
      if (node == 0) atomicOr(&ctrl->neg_avg, 1);
      valid = inner = false;
    }
  }
  if (valid)
#pragma unroll
    for (int v0 = 0; v0 < 8; v0 += GS)
      if (node + v0 < 8) u_avg[e * 8 + node + v0] = mine[v0 / GS];
  // cell entropies for the entropy-offset limiter (DG_solver.f90:195-224)
  if (ent_offset) {
    const double pq = act ? node_prs(x, gamma) : 0.0;
    const bool okq = !act || (x[0] >= PP_EPS && pq >= PP_EPS);
    const double okall = grp_min<GS>(okq ? 1.0 : 0.0);
    const double ce = grp_sum<GS>((act && okall > 0.5) ? 0.25 * g.hx * g.hy * dc.qw[k] * dc.qw[l] * ent_of(x[0], pq, gamma, g.igm1) : 0.0);
    if (valid && node == 0) {
      const double prs = prs_of(avg[0], avg[1], avg[2], avg[3], avg[4], avg[5], avg[6], avg[7], gamma);
      cell_ent_FV[e] = ent_of(avg[0], prs, gamma, g.igm1);
      cell_ent_DG[e] = okall > 0.5 ? ce : 0.0;
      cell_ent_nan[e] = okall > 0.5 ? 0 : 1;
    }
  }
  if (apply_ldf) {
    double fx = x[4] - avg[4], fy = x[5] - avg[5];
    ldf_project<P>(fx, fy, lane - node, node, nd, row, reinterpret_cast<const double2*>(s_A));
    if (valid) {
      x[4] = fx + avg[4];
      x[5] = fy + avg[5];
    }
  }
  bool neg = false, scaled = false;
  if constexpr (LIMIT) {
    __syncwarp();  // the group's lane 0 wrote the cell entropies limit_group reads
    limit_group<P>(x, avg, inner && nd, inner && node == 0, node, e, g, ctrl, ent_offset, 0, cell_ent_DG, cell_ent_FV,
                   cell_ent_nan, &neg, &scaled);
    const unsigned cnt = __popc(__ballot_sync(FULL_MASK, neg));
    if (lane == 0 && cnt) atomicAdd(s_cnt, (int)cnt);
  }
  // write back the state of every element formed here, and of an admissible element what changed
  // in place: (Bx, By) after the LDF, all eight variables where the limiter scaled the element
  // (the positivity and entropy-offset scalings are conditional, so most elements keep six of
  // their eight variables bit for bit and need not store them)
  if (act) {
    if (s1.u0 || scaled) {
#pragma unroll
      for (int v = 0; v < 8; ++v) u[e * EB + v * NN + node] = x[v];
    } else if (valid && apply_ldf) {
      u[e * EB + 4 * NN + node] = x[4];
      u[e * EB + 5 * NN + node] = x[5];
    }
  }
}


template <int P>
__device__ __forceinline__ void load_ldf(const double* __restrict__ A, double* s_A) {
  for (int it = threadIdx.x; it < ldf_table_doubles(P); it += PPCfg<P>::NT) s_A[it] = __ldg(A + it);
}

// one CTA walks chunks blockIdx.x, blockIdx.x + gridDim.x, ... (the LDF operator is loaded once).
template <int P, bool LIMIT>
__global__ void __launch_bounds__(PPCfg<P>::NT, PPCfg<P>::MINB)
    pp_avg_ldf_kernel(double* __restrict__ u, double* __restrict__ u_avg, Geo g, Ctrl* ctrl,
                      int gate, int apply_ldf, int ent_offset,
                      double* __restrict__ cell_ent_DG, double* __restrict__ cell_ent_FV,
                      unsigned char* __restrict__ cell_ent_nan, int nchunks, Stage1Src s1) {
  using C = PPCfg<P>;
  __shared__ __align__(16) double s_A[ldf_table_doubles(P)];
  __shared__ __align__(16) double s_ldf[C::TE * (C::N2 + 2)];
  __shared__ __align__(16) double s_pf[(C::NT / 32) * 2 * C::G * C::EB];  // per warp: u (or u_con), k1
  __shared__ int s_cnt;
  if (threadIdx.x == 0) s_cnt = 0;
  if (apply_ldf) load_ldf<P>(g.ldfA, s_A);  // (written when the instance was created)
  grid_begin();
  if (!gate_open(ctrl, gate)) return;
  __syncthreads();
  // the copies of a warp's next chunk are in flight while it works on this one
  double* bu = s_pf + (threadIdx.x >> 5) * 2 * C::G * C::EB;
  double* bk = bu + C::G * C::EB;
  // grid positions of the chunks' first elements, advanced by the CTA's stride (no division in
  // the loop)
  const int NXG = g.nx + 2;
  const GridRC stride = grid_rc((long long)gridDim.x * C::TE, NXG);
  GridRC pos = grid_rc((long long)blockIdx.x * C::TE, NXG);
  if (blockIdx.x < nchunks) pp_prefetch<P>(u, g, blockIdx.x, pos, s1, bu, bk);
  for (int c = blockIdx.x; c < nchunks; c += gridDim.x) {
    cp_async_wait_all();
    __syncwarp();
    const long long nxt = c + gridDim.x < nchunks ? (long long)c + gridDim.x : -1;
    GridRC npos{pos.j + stride.j, pos.i + stride.i};
    if (npos.i >= NXG) {
      npos.i -= NXG;
      ++npos.j;
    }
    pp_avg_ldf_chunk<P, LIMIT, true>(u, u_avg, g, ctrl, c, pos, apply_ldf, ent_offset, cell_ent_DG, cell_ent_FV,
                                     cell_ent_nan, s_A, s_ldf, &s_cnt, s1, bu, bk, nxt, npos);
    pos = npos;
  }
  __syncthreads();
  if (threadIdx.x == 0 && s_cnt) atomicAdd(&ctrl->num_negcell, s_cnt);
}

// many instances, stage 1: items = every member's chunks; LIMIT: loop 3 fused (unless the stage is the
// final one)
template <int P, bool LIMIT>
__global__ void __launch_bounds__(PPCfg<P>::NT, PPCfg<P>::MINB > 3 ? 3 : PPCfg<P>::MINB)
    pp_avg_ldf_batched(const InstDesc* __restrict__ insts, const int* __restrict__ pref,
                       const int* __restrict__ nwork, const int* __restrict__ ninst, int gate) {
  using C = PPCfg<P>;
  __shared__ __align__(16) double s_A[ldf_table_doubles(P)];
  __shared__ __align__(16) double s_ldf[C::TE * (C::N2 + 2)];
  __shared__ int s_cnt;
  __shared__ SharedWalk s_walk;  // the walker's state, out of the registers the chunk needs
  if (threadIdx.x == 0) s_walk.start(pref, *ninst, *nwork);
  __syncthreads();
  int loaded = -1;  // member whose LDF operator s_A holds
  while (s_walk.w < s_walk.last) {
    const int m = s_walk.m, chunk = s_walk.w - s_walk.mstart;
    const InstDesc& d = insts[m];
    const bool open = gate_open(d.ctrl, gate);
    if (open) {
      if (d.use_ldf && loaded != m) {  // (the previous item ended with a barrier)
        load_ldf<P>(d.g.ldfA, s_A);
        loaded = m;
      }
      if (threadIdx.x == 0) s_cnt = 0;
    }
    __syncthreads();  // every thread has read the walker; s_A and s_cnt are in place
    if (threadIdx.x == 0) s_walk.advance(pref);
    if (open) {
      const Stage1Src s1{d.u[0], d.ut[1], &d.ctrl->dt, stage1_coef(d.R)};
      pp_avg_ldf_chunk<P, LIMIT, false>(d.u[1], d.u_avg, d.g, d.ctrl, chunk,
                                        grid_rc((long long)chunk * C::TE, d.g.nx + 2), d.use_ldf, d.ent_offset,
                                        d.cell_ent_DG, d.cell_ent_FV, d.cell_ent_nan, s_A, s_ldf, &s_cnt, s1,
                                        nullptr, nullptr, -1, GridRC{0, 0});
    }
    __syncthreads();  // the item is done; the walker has advanced
    if (open && threadIdx.x == 0 && s_cnt) atomicAdd(&d.ctrl->num_negcell, s_cnt);
  }
}

// ---------------------------------------------------------------------------------------------
// Global average (DG_solver.f90:227-229,282-286): the sum of (hx*hy)*avg over the interior elements, in a
// fixed order.  An item is SUM_CHUNK consecutive elements of u_avg; the CTA that finishes the last item
// of an instance adds up the items' partial sums.  Thread 8r + v takes variable v of every 32nd element.
// Bound by latency (512^2: 258 CTAs, 17 MB out of L2); alone it runs beside the face indicators.
// ---------------------------------------------------------------------------------------------
constexpr int SUM_CHUNK = 1024;
__host__ __device__ inline int pp_sum_chunks(int nx, int ny) {
  return (int)(((long long)(nx + 2) * (ny + 2) + SUM_CHUNK - 1) / SUM_CHUNK);
}

// sum over the CTA's 32 rows of threads; threads 0..7 return the eight totals
__device__ __forceinline__ double pp_sum_rows(double acc, double* s) {
  const int tid = threadIdx.x;
  s[tid] = acc;
  __syncthreads();
#pragma unroll
  for (int w = 128; w >= 8; w >>= 1) {
    if (tid < w) s[tid] = s[tid] + s[tid + w];
    __syncthreads();
  }
  return s[tid & 7];
}

__device__ __forceinline__ void pp_sum_chunk(const double* __restrict__ u_avg, const Geo& g, int chunk, double* partial,
                                             Ctrl* ctrl) {
  __shared__ double s[256];
  __shared__ bool s_last;
  const int tid = threadIdx.x, v = tid & 7, nx = g.nx, ny = g.ny, nchunk = pp_sum_chunks(nx, ny);
  const long long total = (long long)(nx + 2) * (ny + 2);
  const long long e0 = (long long)chunk * SUM_CHUNK + (tid >> 3);
  GridRC at = grid_rc(e0, nx + 2);
  const double h2 = g.hx * g.hy;
  double acc = 0.0;
#pragma unroll 8
  for (int q = 0; q < SUM_CHUNK / 32; ++q) {
    const long long e = e0 + 32 * q;
    if (e < total && at.i >= 1 && at.i <= nx && at.j >= 1 && at.j <= ny) acc = __dadd_rn(acc, __dmul_rn(h2, u_avg[e * 8 + v]));
    at = grid_adv(at, 32, nx + 2);
  }
  acc = pp_sum_rows(acc, s);
  if (tid < 8) partial[chunk * 8 + tid] = acc;
  __threadfence();
  __syncthreads();
  if (tid == 0) s_last = atomicAdd(&ctrl->sum_ticket, 1u) == (unsigned)nchunk - 1u;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  acc = 0.0;
  for (int b = tid >> 3; b < nchunk; b += 32) acc = __dadd_rn(acc, __ldcg(partial + b * 8 + v));
  acc = pp_sum_rows(acc, s);
  if (tid < 8) ctrl->u_avg_global[tid] = acc;
  if (tid == 0) ctrl->sum_ticket = 0u;
}

__global__ void __launch_bounds__(256) pp_reduce_kernel(const double* __restrict__ u_avg, Geo g, double* partial,
                                                        Ctrl* ctrl, int gate) {
  if (!gate_open(ctrl, gate)) return;
  pp_sum_chunk(u_avg, g, blockIdx.x, partial, ctrl);
}

// many instances: items = the chunks of every member (the final stage of those that use OEDG)
__global__ void __launch_bounds__(256) pp_reduce_batched(const InstDesc* __restrict__ insts, const int* __restrict__ pref,
                                                         const int* __restrict__ nwork, const int* __restrict__ ninst,
                                                         int gate) {
  const int nw = *nwork, n = *ninst;
  for (BatchWalk it(pref, n, nw); it.more(); it.next()) {
    const InstDesc& d = insts[it.m];
    if (!gate_open(d.ctrl, gate) || !d.use_oedg) continue;
    pp_sum_chunk(d.u_avg, d.g, it.local(), d.partial, d.ctrl);
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------------------------
// OEDG face jump indicators (DG_solver.f90:295-422), one value per (face, variable):
//   sigsum = sum_{kk,ll} (2m+1) h^m / (2 max(2p-1,1) kk! ll!) * <0.5 w, |d^kk_x d^ll_y jump|>
// A CTA owns a TX x TY tile of interior elements and computes the left x face and the bottom y
// face of each (plus the right/top boundary faces on the last tile of a row/column).  The tile
// and its left/bottom neighbours (and the ghost column/row on the last tiles) are staged in
// shared memory with coalesced loads; each (face, variable) item then reads two variable blocks.
// Shared records take an odd number of doubles per variable (padded where (p+1)^2 is even), so that the
// eight variables of two neighbouring elements fall in 16 different bank pairs.
// ---------------------------------------------------------------------------------------------
// Derivatives along the face of a polynomial given by its values f at the N GLL nodes, in units of the
// reference coordinate, by the closed form of the interpolant (N = 4: its even part alpha + beta x^2 and
// odd part gamma x + delta x^3 at +-1, +-1/sqrt 5; 27 operations for the three derivatives against
// 48 for three products with D).  d1, d2: nodal values of the first and second derivative; d3: the
// third, a constant (as are d2 at N = 3 and d1 at N = 2, which then stand at index 0 alone).
template <int N>
__device__ __forceinline__ void face_derivs(const double* f, double* d1, double* d2, double& d3) {
  if constexpr (N == 4) {
    constexpr double R5 = 2.2360679774997896964, I5 = 1.0 / R5;  // sqrt 5 and 1/sqrt 5
    const double b2 = 1.25 * ((f[0] + f[3]) - (f[1] + f[2]));    // 2 beta
    const double o = f[3] - f[0], dl = o - R5 * (f[2] - f[1]);   // delta = 0.625 dl
    const double e1 = I5 * b2;
    const double q3 = 0.5 * o + 1.25 * dl, q2 = 0.5 * o - 0.25 * dl;  // gamma + 3 delta x^2
    d1[0] = q3 - b2;
    d1[1] = q2 - e1;
    d1[2] = q2 + e1;
    d1[3] = q3 + b2;
    d2[0] = b2 - 3.75 * dl;
    d2[1] = b2 - (3.75 * I5) * dl;
    d2[2] = b2 + (3.75 * I5) * dl;
    d2[3] = b2 + 3.75 * dl;
    d3 = 3.75 * dl;
  } else if constexpr (N == 3) {
    d2[0] = (f[0] + f[2]) - 2.0 * f[1];
    d1[1] = 0.5 * (f[2] - f[0]);
    d1[0] = d1[1] - d2[0];
    d1[2] = d1[1] + d2[0];
  } else {
    d1[0] = 0.5 * (f[1] - f[0]);
  }
}
// <w/2, |f|> at the N GLL nodes
template <int N>
__device__ __forceinline__ double face_l1(const double* f) {
  if constexpr (N == 4) return (1.0 / 12.0) * (fabs(f[0]) + fabs(f[3])) + (5.0 / 12.0) * (fabs(f[1]) + fabs(f[2]));
  else if constexpr (N == 3) return (1.0 / 6.0) * (fabs(f[0]) + fabs(f[2])) + (2.0 / 3.0) * fabs(f[1]);
  else return 0.5 * (fabs(f[0]) + fabs(f[1]));
}

// One face, either direction.  Rp, Lm = the variable's nodes of the element after and before the
// face; node (a along the normal, b along the face) sits at a*sn + b*st (x face: sn = 1, st = N; y
// face: sn = N, st = 1).  coef[n][t] = (2(n+t)+1) h^(n+t) / (2 max(2p-1,1) n! t!) with h the element
// size along the normal, times (2/h)^n (2/h_t)^t, the scales of the derivatives.  The x face of the
// reference (DG_solver.f90:296-343) is this with (R, L, hx, hy); its y face (:360-407) with (T, B,
// hy, hx): the two loops are the same arithmetic with the roles of the directions exchanged.
//
// The n-th normal derivative is R0[n] . R at the first node of R and RN[n] . L at the last of L, with
// RN[n][a] = (-1)^n R0[n][N-1-a] (the nodes are symmetric): the jump of an odd (even) order is R0[n]
// times the sums (differences) R[a] +- L[N-1-a].  Scales applied to the sums of magnitudes, the
// derivatives along the face in closed form: about 185 operations a face and variable at p = 3
// (295 as products with the scaled D), in 64 registers, so that one thread takes a whole face where
// two warps shared it.  With the faces ordered along rows (16 different bank pairs per half-warp):
// 400 x 400, p = 3 135 -> 75 us, p = 2 63 -> 40, 500 x 500 p = 1 48 -> 34.  Bound by the
// shared-memory pipe (each node value is read by four faces) and its staging.
template <int P>
__device__ __forceinline__ double sigsum_face(const double* Rp, const double* Lm, int sn, int st, const double* coef) {
  constexpr int N = P + 1;
  const DegConst& dc = c_deg[P];
  double J[N][N];  // J[n][b] = the jump of the n-th normal derivative at face node b
#pragma unroll
  for (int b = 0; b < N; ++b) {
    double sum[N], dif[N];
#pragma unroll
    for (int a = 0; a < N; ++a) {
      const double r = Rp[a * sn + b * st], l = Lm[(N - 1 - a) * sn + b * st];
      sum[a] = r + l;
      dif[a] = r - l;
    }
    J[0][b] = dif[0];
#pragma unroll
    for (int n = 1; n <= P; ++n) {
      const double* x = (n & 1) ? sum : dif;
      double t = dc.R0[n][0] * x[0];
#pragma unroll
      for (int a = 1; a < N; ++a) t += dc.R0[n][a] * x[a];
      J[n][b] = t;
    }
  }
  double total = 0.0, d1[N], d2[N], d3 = 0.0;
#pragma unroll
  for (int n = 0; n <= P; ++n) {
    total += coef[n * N] * face_l1<N>(J[n]);
    if (n < P) {  // orders along the face up to P - n; the last of a degree-P polynomial is a constant
      face_derivs<N>(J[n], d1, d2, d3);
      total += coef[n * N + 1] * (N == 2 ? fabs(d1[0]) : face_l1<N>(d1));
      if (P >= 2 && n + 2 <= P) total += coef[n * N + 2] * (N == 3 ? fabs(d2[0]) : face_l1<N>(d2));
      if (P == 3 && n == 0) total += coef[3] * fabs(d3);
    }
  }
  return total;
}

// coef[n][t] of sigsum_face for element size h along the normal (the reference's running products
// h^(n+t), n! t!) and the derivative scales sn = 2/h, st = 2/h_t
template <int P>
__device__ __forceinline__ double sigsum_coef(int n, int t, double h, double sn, double st) {
  const int denom_base = 2 * max(2 * P - 1, 1);
  double hp = 1.0;
  int fn = 1, ft = 1;
  for (int i = 0; i < n; ++i) {
    hp *= h * sn;
    fn *= (i + 1);
  }
  for (int i = 0; i < t; ++i) {
    hp *= h * st;
    ft *= (i + 1);
  }
  return ((2 * (n + t) + 1) * hp) / (double)(denom_base * fn * ft);
}

template <int P>
struct SigCfg {
  static constexpr int TX = PPTune<P>::sig.TX, TY = PPTune<P>::sig.TY, MINB = PPTune<P>::sig.MINB;
};

template <int P>
struct SigLayout {
  static constexpr int N = P + 1, NN = N * N, EB = 8 * NN;
  static constexpr int TX = SigCfg<P>::TX, TY = SigCfg<P>::TY;
  static constexpr int VS = NN | 1, ES = 8 * VS;   // variable / element record: an odd variable stride
  static constexpr int RW = TX + 2, RH = TY + 2;   // staged rectangle (max)
  static constexpr int DOUBLES = RW * RH * ES;
};


// The tile's own elements also give the max and min of every variable over their nodes, merged
// into ctrl->umax_bits / umin_bits (order-preserving encodings; max and min are exact, so neither
// the order of the merge nor the tiling changes the result).  The atomic is skipped when the value
// already there is not exceeded, so that most tiles issue none.
// Where the indicator tile's results go.  Taken by reference, so that the batched kernel can keep
// it in shared memory instead of in registers for the whole tile.
struct SigOut {
  double* sig_x;
  double* sig_y;
  Ctrl* ctrl;
};

template <int P>
__device__ __forceinline__ void pp_sigsum_tile(const double* __restrict__ u, const Geo& g, const SigOut& so,
                                               int tile_x, int tile_y) {
  using L = SigLayout<P>;
  constexpr int NN = L::NN, EB = L::EB, VS = L::VS, ES = L::ES, TX = L::TX, TY = L::TY, RW = L::RW;
  constexpr int NT = 256;
  __shared__ double s_e[L::DOUBLES];  // face math reads its two variable blocks from here
  __shared__ double s_coef[2 * (P + 1) * (P + 1)];  // x faces (h = hx), then y faces (h = hy)
  __shared__ double s_mm[2][NT / 32][8];              // per warp: max, min of each variable
  const int tid = threadIdx.x;
  const int nx = g.nx, ny = g.ny;
  const int i0 = 1 + tile_x * TX, j0 = 1 + tile_y * TY;
  const int W = min(TX, nx - i0 + 1), H = min(TY, ny - j0 + 1);
  const int right = (i0 + W - 1 == nx), top = (j0 + H - 1 == ny);
  const int cw = W + 1 + right, rh = H + 1 + top;  // staged columns i0-1 .., rows j0-1 ..
  // stage: rect row rr = grid row j0-1+rr (a contiguous run of cw elements in u), rect column
  // cc = grid column i0-1+cc.  The copies go straight to shared memory; the divisions are by
  // compile-time constants.
  {
    const int run = cw * EB;
    const long long row = (long long)(nx + 2) * EB;
    const double* src = u + ((long long)(j0 - 1) * (nx + 2) + (i0 - 1)) * EB;
    for (int rr = 0; rr < rh; ++rr, src += row) {
      double* dst = s_e + rr * RW * ES;
      for (int rem = tid; rem < run; rem += NT) {
        const int cc = rem / EB, w = rem - cc * EB, v = w / NN, q = w - v * NN;
        cp_async8(dst + cc * ES + v * VS + q, src + rem);
      }
    }
    cp_async_commit();
  }
  if (tid < 2 * (P + 1) * (P + 1)) {
    const int d = tid / ((P + 1) * (P + 1)), r = tid - d * (P + 1) * (P + 1), n = r / (P + 1), t = r - n * (P + 1);
    s_coef[tid] = (n + t <= P) ? sigsum_coef<P>(n, t, d == 0 ? g.hx : g.hy, d == 0 ? g.sxh : g.syh, d == 0 ? g.syh : g.sxh) : 0.0;
  }
  cp_async_wait_all();
  __syncthreads();
  {  // extrema of the own elements: thread tid takes variable tid & 7 of elements tid/8, tid/8 + NT/8, ...
    const int v = tid & 7;
    double mx = -1.0e308, mn = 1.0e308;
    for (int e = tid >> 3; e < W * H; e += NT / 8) {
      const int r = e / W, c = e - r * W;
      const double* src = s_e + ((r + 1) * RW + c + 1) * ES + v * VS;
#pragma unroll
      for (int q = 0; q < NN; ++q) {
        mx = at_least(src[q], mx);
        mn = at_most(src[q], mn);
      }
    }
#pragma unroll
    for (int o = 8; o < 32; o <<= 1) {
      mx = fmax(mx, __shfl_xor_sync(FULL_MASK, mx, o));
      mn = fmin(mn, __shfl_xor_sync(FULL_MASK, mn, o));
    }
    if ((tid & 31) < 8) {
      s_mm[0][tid >> 5][v] = mx;
      s_mm[1][tid >> 5][v] = mn;
    }
  }
  const int wr = W + right, ht = H + top;  // TX and TY on interior tiles
  const int nfx = H * wr, nfy = W * ht;
  // face-variable items: 8 variables of a face in consecutive threads, faces along a row, so that
  // 16 threads (2 faces x 8 variables) read 16 different bank pairs
  for (int q = tid; q < 8 * (nfx + nfy); q += NT) {
    const int v = q & 7, f = q >> 3;
    const bool xf = f < nfx;
    const int f2 = xf ? f : f - nfx, n = xf ? wr : W;
    const int r = (n == TX) ? f2 / TX : f2 / n, c = f2 - r * n;
    // the block of the element before the face: left of x face (r, c), below y face (r, c)
    const double* lo = s_e + ((xf ? (r + 1) * RW + c : r * RW + c + 1)) * ES + v * VS;
    double* dst = xf ? so.sig_x + (((long long)(j0 + r - 1) * (nx + 1)) + (i0 + c - 1)) * 8 + v
                     : so.sig_y + (((long long)(j0 + r - 1) * nx) + (i0 + c - 1)) * 8 + v;
    // one call site for both directions (the strides select the direction)
    *dst = sigsum_face<P>(lo + (xf ? ES : RW * ES), lo, xf ? 1 : P + 1, xf ? P + 1 : 1,
                          s_coef + (xf ? 0 : (P + 1) * (P + 1)));
  }
  __syncthreads();
  if (tid < 16) {  // threads 0-7: max of variable tid; 8-15: min of variable tid - 8
    const int v = tid & 7, lo = tid >> 3;
    double m = s_mm[lo][0][v];
    for (int w = 1; w < NT / 32; ++w) m = lo ? fmin(m, s_mm[1][w][v]) : fmax(m, s_mm[0][w][v]);
    unsigned long long* dst = lo ? &so.ctrl->umin_bits[v] : &so.ctrl->umax_bits[v];
    const unsigned long long enc = ord_enc(m), cur = *reinterpret_cast<volatile unsigned long long*>(dst);
    if (lo ? (m < 1.0e308 && enc < cur) : (m > -1.0e308 && enc > cur)) {
      if (lo) atomicMin(dst, enc);
      else atomicMax(dst, enc);
    }
  }
}

template <int P>
__global__ void __launch_bounds__(256, SigCfg<P>::MINB)
    pp_sigsum_kernel(const double* u, Geo g, Ctrl* ctrl, int gate,
                     double* __restrict__ sig_x, double* __restrict__ sig_y) {
  grid_begin();
  if (!gate_open(ctrl, gate)) return;
  pp_sigsum_tile<P>(u, g, SigOut{sig_x, sig_y, ctrl}, blockIdx.x, blockIdx.y);
}

// many instances: items = every member's tiles (row-major)
template <int P>
__global__ void __launch_bounds__(256, SigCfg<P>::MINB)
    pp_sigsum_batched(const InstDesc* __restrict__ insts, const int* __restrict__ pref,
                      const int* __restrict__ nwork, const int* __restrict__ ninst, int slot, int final, int gate) {
  __shared__ Geo s_g;  // the member's geometry and outputs, per tile (see SigOut)
  __shared__ SigOut s_so;
  __shared__ SharedWalk s_walk;
  if (threadIdx.x == 0) s_walk.start(pref, *ninst, *nwork);
  __syncthreads();
  while (s_walk.w < s_walk.last) {
    const int m = s_walk.m, local = s_walk.w - s_walk.mstart;
    const InstDesc& d = insts[m];
    const bool open = gate_open(d.ctrl, gate) && d.use_oedg && final;
    if (open && threadIdx.x == 0) {
      s_g = d.g;
      s_so = SigOut{d.sig_x, d.sig_y, d.ctrl};
    }
    __syncthreads();  // every thread has read the walker; the item's arguments are in place
    if (threadIdx.x == 0) s_walk.advance(pref);
    if (open) {
      const int ntx = (d.g.nx + SigCfg<P>::TX - 1) / SigCfg<P>::TX;
      pp_sigsum_tile<P>(d.u[slot], s_g, s_so, local % ntx, local / ntx);
    }
    __syncthreads();  // the item is done (the next one reuses shared memory); the walker has advanced
  }
}

// ---------------------------------------------------------------------------------------------
// loop 3: OEDG damping, positivity, entropy offset, entropy.  A CTA owns TE consecutive
// interior elements of one row j (a contiguous run of memory).
// ---------------------------------------------------------------------------------------------
// The arrays and switches of one limiter segment.  Taken by reference, so that the batched kernel
// can keep them in shared memory (read where used) instead of in registers for the whole segment.
struct LimitIO {
  double* u;                  // the stage state (interior updated in place unless accept_only)
  const double* u_avg;        // cell averages (loop 1)
  Ctrl* ctrl;
  const double* sig_x;        // OEDG face indicators (x faces, y faces)
  const double* sig_y;
  const double* cell_ent_DG;  // entropy-offset inputs of loop 1
  const double* cell_ent_FV;
  const unsigned char* cell_ent_nan;
  double* ent_out;            // the segment's entropy partial (comput_ent)
  double* accept_dst;         // the accepted state (u_con) or nullptr
  double oedg_dt;
  int apply_oedg, ent_offset, comput_ent, accept_only;
};

template <int P>
__device__ __forceinline__ void pp_limit_segment(const LimitIO& io, const Geo& g, int seg, int jrow, double* s_ent,
                                                 int* s_cnt) {
  using C = PPCfg<P>;
  constexpr int NN = C::NN, EB = C::EB, GS = C::GSL, G = C::GL, TE = C::TEL;  // the limiter's groups
  if (io.ctrl->neg_avg) return;  // the reference skips loop 3 once neg_avg is set (DG_solver.f90:431)
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const GrpLane<GS> gl = grp_lane<GS>();
  const int grp = gl.grp, node = gl.node;
  const int nx = g.nx, NXG = nx + 2;
  const int j = 1 + jrow;
  const int i0 = 1 + seg * TE;
  const int ne = min(TE, nx - i0 + 1);
  const int el = warp * G + grp;
  const bool inside = el < ne && !gl.idle, nd = node < NN;
  const bool act = inside && nd;
  const long long e = (long long)j * NXG + i0 + el;
  const double gamma = g.gamma;
  double x[8], avg[8];
#pragma unroll
  for (int v = 0; v < 8; ++v) x[v] = act ? io.u[e * EB + v * NN + node] : 0.0;
#pragma unroll
  for (int v = 0; v < 8; v += 2) {
    const double2 t = inside ? *reinterpret_cast<const double2*>(io.u_avg + e * 8 + v) : make_double2(1.0, 1.0);
    avg[v] = t.x;
    avg[v + 1] = t.y;
  }
  // Instructions bound this kernel (most of them 64-bit), so quotients are products with rcp_nr, roots are
  // sqrt_nr, and a maximum of values that are not negative goes through the integer reduction: 98 -> 88 us
  // at p = 3, 76 -> 67 us at p = 2 (400^2), 48 -> 41 us at p = 1 (500^2).
  if (io.apply_oedg) {  // DG_solver.f90:448-524
    double sx = 0.0, sy = 0.0;
    if (act) {
      const double rho = at_least(x[0], PP_EPS);
      const double ir = rcp_any(rho);
      const double vx = ir * x[1], vy = ir * x[2];
      const double ek = 0.5 * ir * (x[1] * x[1] + x[2] * x[2] + x[3] * x[3]);
      const double bx = x[4], by = x[5], bz = x[6];
      const double bsq = bx * bx + by * by + bz * bz;
      const double pf = at_least((gamma - 1.0) * (x[7] - (ek + 0.5 * bsq)), PP_EPS);
      const double cs = gamma * pf * ir, ss = cs + bsq * ir, sqsq = ss * ss, coef = 4.0 * cs * ir;
      const double dx = at_least(sqsq - coef * (bx * bx), TINY), dy = at_least(sqsq - coef * (by * by), TINY);
      sx = fabs(vx) + sqrt_nr(0.5 * at_least(ss + sqrt_nr(dx), TINY));
      sy = fabs(vy) + sqrt_nr(0.5 * at_least(ss + sqrt_nr(dy), TINY));
      if (!(dx + dy < 1.0e270)) {  // beyond sqrt_nr: an infinite speed damps to the average
        sx = fabs(vx) + sqrt_any(0.5 * at_least(ss + sqrt_any(dx), TINY));
        sy = fabs(vy) + sqrt_any(0.5 * at_least(ss + sqrt_any(dy), TINY));
      }
    }
    const double mx = grp_max_nonneg<GS>(sx), my = grp_max_nonneg<GS>(sy);
    // lane `node` of the group forms delta_v for v = node, node + GS, ... from the element's four faces
    double d = 0.0;
    if (inside) {
      const int i = i0 + el;
      const long long fxl = ((long long)(j - 1) * (nx + 1) + (i - 1)) * 8;
      const long long fyb = ((long long)(j - 1) * nx + (i - 1)) * 8;
      const long long fyt = ((long long)j * nx + (i - 1)) * 8;
      const Ctrl* ctrl = io.ctrl;
      const double* sig_x = io.sig_x;
      const double* sig_y = io.sig_y;
      const double wx = 0.5 * g.sxh * mx, wy = 0.5 * g.syh * my;
      for (int v = node; v < 8; v += GS) {
        const double gs = ctrl->u_avg_global[v];
        const double uv = at_least(fmax(ord_dec(ctrl->umax_bits[v]) - gs, gs - ord_dec(ctrl->umin_bits[v])), 0.0);
        if (uv > OEDG_EPS)
          d = at_least((wx * (sig_x[fxl + v] + sig_x[fxl + 8 + v]) + wy * (sig_y[fyb + v] + sig_y[fyt + v])) * rcp_any(uv), d);
      }
    }
    const double dmax = grp_max_nonneg<GS>(d);
    const double theta = exp(-io.oedg_dt * dmax);
    if (act)
#pragma unroll
      for (int v = 0; v < 8; ++v) x[v] = avg[v] + theta * (x[v] - avg[v]);
  }
  bool neg = false;
  const double ce = limit_group<P, GS>(x, avg, act, inside && node == 0, node, e, g, io.ctrl, io.ent_offset,
                                       io.comput_ent, io.cell_ent_DG, io.cell_ent_FV, io.cell_ent_nan, &neg);
  const unsigned cnt = __popc(__ballot_sync(FULL_MASK, neg));
  if (lane == 0 && cnt) atomicAdd(s_cnt, (int)cnt);
  if (act)
#pragma unroll
    for (int v = 0; v < 8; ++v) {
      if (!io.accept_only) io.u[e * EB + v * NN + node] = x[v];
      if (io.accept_dst) io.accept_dst[e * EB + v * NN + node] = x[v];
    }
  if (io.comput_ent) {  // chunk partial in a fixed order
    if (inside && node == 0) s_ent[el] = ce;
    __syncthreads();
    if (warp == 0) {
      double tot = 0.0;
      for (int q = lane; q < ne; q += 32) tot = tot + s_ent[q];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) tot = tot + __shfl_xor_sync(FULL_MASK, tot, o);
      if (lane == 0) *io.ent_out = tot;
    }
  }
}

template <int P>
__global__ void __launch_bounds__(PPCfg<P>::NT, PPCfg<P>::MINB)
    pp_limit_kernel(double* __restrict__ u, const double* u_avg, Geo g, Ctrl* ctrl,
                    int gate, int apply_oedg, const double* dt_ptr, double oedg_dt_arg,
                    int ent_offset, int comput_ent, const double* sig_x,
                    const double* sig_y, const double* cell_ent_DG,
                    const double* cell_ent_FV, const unsigned char* cell_ent_nan,
                    double* __restrict__ ent_partial, double* __restrict__ accept_dst, int accept_only) {
  grid_begin();
  __shared__ double s_ent[PPCfg<P>::TEL];
  __shared__ int s_cnt;
  if (!gate_open(ctrl, gate)) return;
  if (threadIdx.x == 0) s_cnt = 0;
  __syncthreads();
  const LimitIO io{u, u_avg, ctrl, sig_x, sig_y, cell_ent_DG, cell_ent_FV, cell_ent_nan,
                   ent_partial + (long long)blockIdx.y * gridDim.x + blockIdx.x, accept_dst,
                   dt_ptr ? *dt_ptr : oedg_dt_arg, apply_oedg, ent_offset, comput_ent, accept_only};
  pp_limit_segment<P>(io, g, blockIdx.x, blockIdx.y, s_ent, &s_cnt);
  __syncthreads();
  if (threadIdx.x == 0 && s_cnt) atomicAdd(&ctrl->num_negcell, s_cnt);
}

// many instances: items = every member's row segments (row-major); the final stage applies OEDG
// (if the instance uses it), computes the entropy and writes the accepted interior into slot 0
// only, as the single-instance pipeline does
template <int P>
__global__ void __launch_bounds__(PPCfg<P>::NT, PPCfg<P>::MINB > 3 ? 3 : PPCfg<P>::MINB)
    pp_limit_batched(const InstDesc* __restrict__ insts, const int* __restrict__ pref,
                     const int* __restrict__ nwork, const int* __restrict__ ninst, int slot, int final, int gate) {
  __shared__ double s_ent[PPCfg<P>::TEL];
  __shared__ int s_cnt;
  __shared__ Geo s_g;      // the member's geometry and arrays, per item (see LimitIO)
  __shared__ LimitIO s_io;
  __shared__ SharedWalk s_walk;
  if (threadIdx.x == 0) s_walk.start(pref, *ninst, *nwork);
  __syncthreads();
  while (s_walk.w < s_walk.last) {
    const int m = s_walk.m, local = s_walk.w - s_walk.mstart;
    const InstDesc& d = insts[m];
    const bool open = gate_open(d.ctrl, gate);
    if (open && threadIdx.x == 0) {
      s_cnt = 0;
      s_g = d.g;
      s_io = LimitIO{d.u[slot], d.u_avg, d.ctrl, d.sig_x, d.sig_y, d.cell_ent_DG, d.cell_ent_FV, d.cell_ent_nan,
                     d.ent_partial + local, final ? d.u[0] : nullptr, d.ctrl->dt, d.use_oedg && final,
                     d.ent_offset, final, final};
    }
    __syncthreads();  // every thread has read the walker; the item's arguments are in place
    if (threadIdx.x == 0) s_walk.advance(pref);
    if (open) {
      const int nseg = (d.g.nx + PPCfg<P>::TEL - 1) / PPCfg<P>::TEL;
      pp_limit_segment<P>(s_io, s_g, local % nseg, local / nseg, s_ent, &s_cnt);
    }
    __syncthreads();  // the item is done; the walker has advanced
    if (open && threadIdx.x == 0 && s_cnt) atomicAdd(&s_io.ctrl->num_negcell, s_cnt);
  }
}

// total entropy = fixed-order sum of the per-CTA partials.  One CTA.
__device__ __forceinline__ void pp_entsum_body(const double* __restrict__ partial, int nblk, Ctrl* ctrl) {
  __shared__ double s[256];
  const int tid = threadIdx.x;
  double acc = 0.0;
  for (int b = tid; b < nblk; b += 256) acc = acc + partial[b];
  s[tid] = acc;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if (tid < w) s[tid] = s[tid] + s[tid + w];
    __syncthreads();
  }
  if (tid == 0) ctrl->tot_ent = s[0];
}

// The end of a stage of the time-step pipeline in one launch over the ghost values of the stage
// state u: block 0 forms the total entropy from the limiter's partials (final stage only:
// ent_partial != NULL) and then, in one thread, the stage-end decision (ctl_stage_end_body) and the
// pseudo-time of the next stage (next_stage > 0); every block fills the ghost ring of u if the
// stage was still running when the launch began.  A block that already sees the stage abandoned
// skips its fill, and a fill of an abandoned stage only writes scratch ghosts, so the result is
// that of the separate launches in sequence.
// The stage's record goes to the driver log (log may be nullptr).
// src: the array whose interior the ghost ring is filled from (u itself, or u_con after the final
// stage, whose limiter writes the accepted interior to u_con only).
template <int P>
__global__ void __launch_bounds__(256) stage_end_bc_kernel(const double* src, double* u, Geo g, Ctrl* ctrl, int R,
                                                          int stage, int next_stage,
                                                          const double* ent_partial, int ent_nblk,
                                                          LogEntry* log, int log_cap) {
  grid_begin();
  __shared__ int s_run, s_ent;
  bool run;
  if (blockIdx.x == 0) {  // one read of the state for the whole block, before thread 0 updates it
    if (threadIdx.x == 0) {
      s_run = ctrl->state == ST_RUN;
      s_ent = s_run && ent_partial && !ctrl->neg_avg;
    }
    __syncthreads();
    run = s_run;
    if (s_ent) pp_entsum_body(ent_partial, ent_nblk, ctrl);  // whole block
    if (threadIdx.x == 0) {
      ctl_stage_end_body(ctrl);
      if (run) ctl_log_stage(ctrl, stage, log, log_cap);
      if (next_stage > 0) ctl_stage_time_body(ctrl, R, next_stage);
    }
  } else {
    run = *reinterpret_cast<volatile const int*>(&ctrl->state) == ST_RUN;
  }
  if (run) bc_value<P>(src, u, g, (long long)blockIdx.x * blockDim.x + threadIdx.x);
}

__global__ void __launch_bounds__(256) pp_entsum_kernel(const double* partial, int nblk,
                                                        Ctrl* ctrl, int gate) {
  grid_begin();
  if (!gate_open(ctrl, gate)) return;
  if (ctrl->neg_avg) return;
  pp_entsum_body(partial, nblk, ctrl);
}

// many instances: stage_end_bc_kernel for every member of a batch -- the ghost fills of all
// members (items = every member's blocks of 256 ghost values) and, one CTA per member, the entropy
// sum (final stage), the stage-end decision and the next stage's pseudo-time.  A fill that runs
// after its member's decision abandoned the stage is skipped, which changes nothing (the stage's
// state is scratch then).
template <int P>
__global__ void __launch_bounds__(256) stage_end_bc_batched(const InstDesc* __restrict__ insts,
                                                           const int* __restrict__ pref, const int* __restrict__ nwork,
                                                           const int* __restrict__ ninst, int slot, int R,
                                                           int next_stage, int final) {
  __shared__ int s_run, s_ent;
  const int nw = *nwork, n = *ninst;
  for (BatchWalk it(pref, n, nw); it.more(); it.next()) {
    const InstDesc& d = insts[it.m];
    if (*reinterpret_cast<volatile const int*>(&d.ctrl->state) != ST_RUN) continue;
    // after the final stage the ring is filled from u_con, which alone holds the accepted interior
    bc_value<P>(final ? d.u[0] : d.u[slot], d.u[slot], d.g, (long long)it.local() * 256 + threadIdx.x);
  }
  for (int i = blockIdx.x; i < n; i += gridDim.x) {
    const InstDesc& d = insts[i];
    __syncthreads();  // s_run and s_ent of the previous member are read
    if (threadIdx.x == 0) {
      s_run = d.ctrl->state == ST_RUN;
      s_ent = s_run && final && !d.ctrl->neg_avg;
    }
    __syncthreads();
    if (s_ent) pp_entsum_body(d.ent_partial, d.nseg_limit, d.ctrl);  // whole block
    if (threadIdx.x == 0) {
      ctl_stage_end_body(d.ctrl);
      if (s_run) ctl_log_stage(d.ctrl, slot, d.log, d.log_cap);
      if (next_stage > 0) ctl_stage_time_body(d.ctrl, R, next_stage);
    }
  }
}

// ---------------------------------------------------------------------------------------------
// Stage diagnostics (optional, for checking the invariants the method promises): over the interior
// nodes of a state, the minimum density, the minimum pressure (_macro_prs_, DG_solver.f90:125) and
// the domain integrals of the eight conserved variables by the GLL rule the cell averages use
// (sum of (hx hy / 4) w_k w_l u, DG_solver.f90:177-184,227-229).  Block b takes a fixed contiguous
// range of elements and reduces in a fixed order; the last block to finish (a ticket counter, no
// waiting) combines the block partials in block order and writes the newest log record.  The
// result is therefore independent of timing.  `part` holds DIAG_MAX_BLOCKS x 10 doubles and the
// ticket; the ticket is left at zero.
// ---------------------------------------------------------------------------------------------
constexpr int DIAG_MAX_BLOCKS = 592;  // 4 x 148 SMs
constexpr int DIAG_VALS = 18;          // per block: min rho, min p, 8 sums and their 8 compensations

// Neumaier's compensated summation (a running sum s and the sum c of its rounding errors): the
// domain integrals are checked against conservation at the 1e-13 level, below the rounding error of
// a plain sum of 10^5-10^7 terms.
__device__ __forceinline__ void neu_add(double& s, double& c, double x) {
  const double t = __dadd_rn(s, x);
  c = __dadd_rn(c, fabs(s) >= fabs(x) ? __dadd_rn(__dadd_rn(s, -t), x) : __dadd_rn(__dadd_rn(x, -t), s));
  s = t;
}

template <int P>
__global__ void __launch_bounds__(256) stage_diag_kernel(const double* u, Geo g, Ctrl* ctrl, int gate,
                                                        double* __restrict__ part, unsigned int* ticket,
                                                        LogEntry* log, int log_cap) {
  grid_begin();
  constexpr int N = P + 1, NN = N * N, EB = 8 * NN;
  __shared__ double s[DIAG_VALS][256];
  __shared__ bool s_last;
  if (!gate_open(ctrl, gate) || !log || log_cap <= 0 || ctrl->log_seq <= 0) return;
  const int tid = threadIdx.x;
  const int nx = g.nx, ny = g.ny;
  const long long E = (long long)nx * ny;
  const long long e0 = E * blockIdx.x / gridDim.x, e1 = E * (blockIdx.x + 1) / gridDim.x;
  const DegConst& dc = c_deg[P];
  const double gamma = g.gamma, q4 = __dmul_rn(__dmul_rn(0.25, g.hx), g.hy);
  double rmin = 1.0e308, pmin = 1.0e308, sum[8], cmp[8];
#pragma unroll
  for (int v = 0; v < 8; ++v) sum[v] = cmp[v] = 0.0;
  for (long long it = e0 * NN + tid; it < e1 * NN; it += 256) {
    const long long e = it / NN;
    const int q = (int)(it - e * NN), k = q % N, l = q / N;
    const int j = 1 + (int)(e / nx), i = 1 + (int)(e - (long long)(j - 1) * nx);
    const double* x = u + ((long long)j * (nx + 2) + i) * EB + q;
    double w[8];
#pragma unroll
    for (int v = 0; v < 8; ++v) w[v] = x[v * NN];
    rmin = fmin(rmin, w[0]);
    pmin = fmin(pmin, prs_of(w[0], w[1], w[2], w[3], w[4], w[5], w[6], w[7], gamma));
    const double wq = __dmul_rn(__dmul_rn(q4, dc.qw[k]), dc.qw[l]);
#pragma unroll
    for (int v = 0; v < 8; ++v) neu_add(sum[v], cmp[v], __dmul_rn(wq, w[v]));
  }
  s[0][tid] = rmin;
  s[1][tid] = pmin;
#pragma unroll
  for (int v = 0; v < 8; ++v) {
    s[2 + v][tid] = sum[v];
    s[10 + v][tid] = cmp[v];
  }
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if (tid < w) {
      s[0][tid] = fmin(s[0][tid], s[0][tid + w]);
      s[1][tid] = fmin(s[1][tid], s[1][tid + w]);
#pragma unroll
      for (int v = 0; v < 8; ++v) {  // (s, c) + (s', c'): the sums by Neumaier, the compensations plainly
        double a = s[2 + v][tid], c = __dadd_rn(s[10 + v][tid], s[10 + v][tid + w]);
        neu_add(a, c, s[2 + v][tid + w]);
        s[2 + v][tid] = a;
        s[10 + v][tid] = c;
      }
    }
    __syncthreads();
  }
  if (tid < DIAG_VALS) part[blockIdx.x * DIAG_VALS + tid] = s[tid][0];
  __threadfence();
  __syncthreads();
  if (tid == 0) s_last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  const volatile double* vp = part;
  LogEntry* e = log + ((ctrl->log_seq - 1) % log_cap);
  if (tid < 2) {
    double r = vp[tid];
    for (unsigned b = 1; b < gridDim.x; ++b) r = fmin(r, vp[b * DIAG_VALS + tid]);
    if (tid == 0) e->rho_min = r;
    else e->p_min = r;
  } else if (tid < 10) {  // the blocks' (sum, compensation) pairs in block order
    double a = vp[tid], c = vp[tid + 8];
    for (unsigned b = 1; b < gridDim.x; ++b) {
      c = __dadd_rn(c, vp[b * DIAG_VALS + tid + 8]);
      neu_add(a, c, vp[b * DIAG_VALS + tid]);
    }
    e->total[tid - 2] = __dadd_rn(a, c);
  }
  if (tid == 0) *ticket = 0u;
}

}  // namespace mhd
