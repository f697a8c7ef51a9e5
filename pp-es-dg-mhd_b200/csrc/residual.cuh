// residual.cuh -- DG_semidiscretize (DG_solver.f90:663-892) as one sm_100a kernel.
//
// ut = L(u): the entropy-conservative two-point flux differencing over the GLL nodes of each
// element, the ESPP-HLL interface flux, the Godunov-Powell source and the surface terms, and
// dt_lim.  One warp owns a few neighbouring elements, one lane one node (see residual_item below).
// Sums are formed in a fixed order, so the kernel is deterministic.
#pragma once
#include "common.cuh"
#include "misc.cuh"
#include "post.cuh"

namespace mhd {

// swap_xy (DG_solver.f90:1556-1568) as a variable permutation: 1 <-> 2, 4 <-> 5
__host__ __device__ constexpr int swap_xy_var(int v) { return v == 1 ? 2 : v == 2 ? 1 : v == 4 ? 5 : v == 5 ? 4 : v; }

// What a residual leaves behind.  RES_UT: L(u), in ut.  RES_COMBINE, SSP-RK(2,2) and (3,3): in place of
// L(u) the next stage's SSP-RK combination (drive.f90:185-241, :148-183), rounded exactly as combine_value
// forms it.  RES_POST: in addition loop 1 of the next stage's post-process (averages, admissibility, LDF projection,
// cell entropies), with loop 3 where the stage is not the final one (see post.cuh, stage_post below).
// RES_POST54, SSP-RK(5,4): the same and L(u), in ut: stage 5 reads that of stage 4, and all are the run's
// ut_con(:,2..5).  (One kernel for both kinds of scheme costs SSP-RK(3,3) 0.5-1.5 %.)
enum ResMode : int { RES_UT = 0, RES_COMBINE = 1, RES_POST = 2, RES_POST54 = 3 };
struct StagePost {
  const double* u0;     // u_con (ghosted layout)
  double* out;          // the next stage's state (ghosted layout)
  double ca, cb;        // stage_value's coefficients
  const double* dt;     // the try's dt (device control block)
  double* u_avg;        // from here on: RES_POST
  double *cell_ent_DG, *cell_ent_FV;
  unsigned char* cell_ent_nan;
  int use_ldf, ent_offset, final;
  int stage;            // the stage formed; from here on: RES_POST54
  double cc;            // SSP-RK(5,4): the coefficient of dt*L(u)
  const double *r2, *r3;  // stage 5: the states of stages 2 and 3 (ghosted layout)
  const double* k4;       // stage 5: L of stage 3 (interior layout)
};

// stage s > 1 of an R-stage scheme from the previous stage's residual (the coefficients of combine_value);
// u, ut: the instance's arrays.
__host__ __device__ inline void stage_scheme(StagePost& sp, int R, int s, double* const* u, double* const* ut) {
  sp.u0 = u[0];
  sp.out = u[s];
  sp.final = s == R;
  sp.stage = s;
  if (R == 2) {
    sp.ca = sp.cb = 0.5;
  } else if (R == 3) {
    sp.ca = s == 2 ? 0.75 : 1.0 / 3.0;
    sp.cb = s == 2 ? 0.25 : 2.0 / 3.0;
  } else {
    sp.ca = s == 2 ? 0.444370493651235 : s == 3 ? 0.620101851488403 : s == 4 ? 0.178079954393132 : 0.386708617503269;
    sp.cb = s == 2 ? 0.555629506348765 : s == 3 ? 0.379898148511597 : s == 4 ? 0.821920045606868 : 0.0;
    sp.cc = s == 2 ? 0.368410593050371 : s == 3 ? 0.251891774271694 : s == 4 ? 0.544974750228521 : 0.226007483236906;
    sp.r2 = u[2];
    sp.r3 = u[3];
    sp.k4 = ut[4];
  }
}

// A node of the next stage, rounded as combine_value rounds it: x = its eight values, NN apart in memory; u = the
// current stage's state there, k = its L; at, ki: the node's place in the ghosted and in the interior layout.
template <int NN, int MODE>
__device__ __forceinline__ void stage_node(double* x, const StagePost& sp, double dt, const double* u, const double* k,
                                           long long at, long long ki) {
  if constexpr (MODE != RES_POST54) {
#pragma unroll
    for (int v = 0; v < 8; ++v) x[v] = add(mul(sp.ca, __ldg(sp.u0 + at + v * NN)), mul(sp.cb, add(u[v * NN], mul(dt, k[v]))));
  } else if (sp.stage < 5) {
    const double cdt = mul(sp.cc, dt);
#pragma unroll
    for (int v = 0; v < 8; ++v)
      x[v] = add(add(mul(sp.ca, __ldg(sp.u0 + at + v * NN)), mul(sp.cb, u[v * NN])), mul(cdt, k[v]));
  } else {
    const double cdt = mul(sp.cc, dt), c4 = mul(0.063692468666290, dt);
#pragma unroll
    for (int v = 0; v < 8; ++v)
      x[v] = add(add(add(add(mul(0.517231671970585, __ldg(sp.r2 + at + v * NN)), mul(0.096059710526147, __ldg(sp.r3 + at + v * NN))),
                         mul(c4, __ldg(sp.k4 + ki + v * NN))), mul(sp.ca, u[v * NN])), mul(cdt, k[v]));
  }
}

// =============================================================================================
// One warp per item, one lane per node.
//
// An item is a block of EX x EY neighbouring elements (p = 3: 2 x 1, p = 2: 3 x 1, p = 1: 4 x 2)
// whose nodes fill a warp.  The warp computes everything its nodes need, the interface fluxes of the
// item's whole boundary included, so no barrier of the CTA separates any two steps of an item and
// the warps of an SM run independently: one warp's loads and FP64 chains are covered by the others.
//   0. the item's element blocks and those next to it arrive in the warp's shared memory by bulk
//      asynchronous copies completed on the warp's mbarrier;
//   1. interface fluxes, one face node per lane, to a record per face in shared memory.  Faces between
//      two items are computed by both;
//   2. the nodes' primitives, to a record per node in shared memory;
//   3. the entropy-conservative flux of every node pair of a line, computed once, by one of the
//      pair's two lanes, from the partner's record; the other lane receives the flux by a shuffle
//      (the shared-memory pipe carries a shuffled value once, a stored and loaded one twice).  Rounds per
//      degree (k along x, l along y; every round gives each lane exactly one flux to compute):
//        p = 1  one round: lanes with k == l take their x pair, the others their y pair
//        p = 2  a ring along x (partner k+1 mod 3, received from k+2 mod 3), then the same along y:
//               the three pairs of a line are the ring's three edges
//        p = 3  rings along x and y (four of the six pairs of a line), then a round for the pairs
//               (k, k^2) / (l, l^2): lanes with (k>>1)^(l>>1) == 0 take the x pair, the others the y
//               pair (each such pair has exactly one endpoint of each kind)
//   4. the interface fluxes from their records, the Godunov-Powell terms, dt_lim, the store.
// What bounds it, by counters at p = 3: issue slots (59 %), the shared-memory pipe (64 %, p = 2 78 %)
// and the FP64 pipe (55 %) are all half taken by 16 warps per SM (126 registers).  A warp waits 1.7 cycles an
// instruction for its own FP64 results, 1.1 for the copies, 0.8 for its turn; leaving out the flux
// arithmetic saves only 10 %, and at 18-20 warps (96 registers) the spills cost more than the warps
// bring.  Before it a CTA owned a tile and shared its interface fluxes between two barriers: 400 x 400,
// p = 3 214 us -> 173 us, p = 2 blast 140 -> 121, 700 x 700 p = 1 201 -> 155; the interface fluxes cost
// a quarter more, and the barriers, the uneven split of the face work and 15 % of the instructions
// are gone.  Reading the traces straight from global memory was as fast at p = 2, 3 (181, 127 us) and
// slower at p = 1 (183 us), where a trace's line holds four useful values of sixteen.
// =============================================================================================
#if __has_include("residual2_tuned.h")
#include "residual2_tuned.h"
#endif
// MHD_RES2_CFG<p> = TX, TY, threads, CTAs per SM: a CTA's warps take the items of a TX x TY block of
// elements, one item per warp (CTAs of one warp measured 0-5 % faster than of four: a finished warp is
// replaced at once)
#ifndef MHD_RES2_CFG1
#define MHD_RES2_CFG1 4, 2, 32, 16
#endif
#ifndef MHD_RES2_CFG2
#define MHD_RES2_CFG2 3, 1, 32, 16
#endif
#ifndef MHD_RES2_CFG3
#define MHD_RES2_CFG3 2, 1, 32, 16
#endif
struct Res2Params {
  int TX, TY, NT, MINB;
};
template <int P>
struct Res2Cfg;
template <>
struct Res2Cfg<1> {
  static constexpr Res2Params c{MHD_RES2_CFG1};
  static constexpr int EX = 4, EY = 2;
};
template <>
struct Res2Cfg<2> {
  static constexpr Res2Params c{MHD_RES2_CFG2};
  static constexpr int EX = 3, EY = 1;
};
template <>
struct Res2Cfg<3> {
  static constexpr Res2Params c{MHD_RES2_CFG3};
  static constexpr int EX = 2, EY = 1;
};

template <int P>
struct Res2Layout {
  static constexpr int N = P + 1, NN = N * N, EB = 8 * NN;
  static constexpr int EX = Res2Cfg<P>::EX, EY = Res2Cfg<P>::EY, G = EX * EY;  // an item's elements
  static constexpr int NT = Res2Cfg<P>::c.NT, NW = NT / 32, MINB = Res2Cfg<P>::c.MINB;
  static constexpr int TX = Res2Cfg<P>::c.TX, TY = Res2Cfg<P>::c.TY;  // a CTA's elements
  static constexpr int IX = TX / EX, IY = TY / EY;                    // a CTA's items
  static_assert(TX % EX == 0 && TY % EY == 0 && IX * IY == NW, "one item per warp");
  static_assert(G == 32 / NN, "an item's nodes fill a warp");
  static constexpr int NFX = (EX + 1) * EY * N, NFY = EX * (EY + 1) * N, NF = NFX + NFY;
  // Shared memory of a warp: the staged element blocks (ES doubles apart: padded so that neighbouring
  // elements' traces fall in different banks) -- per row of the item its elements and the ones to their
  // left and right, then the row below and the row above; the mbarrier; the face records.  The
  // node records take the place of the rows below and above, which only step 1 reads.  Records are
  // moved 16 bytes at a time: 14 doubles per face (12 used) and 10 per node (strides of 112 and 80
  // bytes), so that 8 consecutive records start in 8 different bank groups.
  static constexpr int ES = EB + (P == 1 ? 6 : P == 2 ? 4 : 2), SX = EX + 2, NCOPY = EY * SX + 2 * EX;
  static constexpr int FS = 14, NS = 10;
  static constexpr int O_NB = EY * SX * ES, O_NODE = O_NB;
  static constexpr int NB = 2 * EX * ES > 32 * NS ? 2 * EX * ES : 32 * NS;
  static constexpr int O_BAR = O_NB + NB, O_FACE = O_BAR + 2, WARP = O_FACE + NF * FS;
  static_assert(NF * FS >= G * (2 * NN + 2) + ((NN & (NN - 1)) ? G * 8 * NN : 0), "stage_post's scratch fits the face records");
  static_assert(NCOPY <= 32 && (EB * 8) % 16 == 0 && (ES * 8) % 16 == 0, "one copy per lane, 16-byte blocks");
  static constexpr size_t BYTES = sizeof(double) * NW * WARP;
  static_assert((BYTES + 1024) * MINB <= 228 * 1024, "the CTAs of an SM fit its shared memory");
};

// Where the two traces of face f of an item sit among the staged blocks (offsets in doubles), and, for
// a y face, the distance between variables, by which its exchanged vector components are shifted.
// The interior faces of a ragged item and the ones beyond it need no case of their own: the row
// above an item of H < EY rows is staged as its row H, and a face that no element of the item has
// reads whatever is there, into a record that nothing reads.
struct alignas(16) FaceDesc {
  int lo, hi, d, pad_;
};
template <int P>
struct FaceTable {
  FaceDesc f[Res2Layout<P>::NF];
  constexpr FaceTable() : f{} {
    using L = Res2Layout<P>;
    constexpr int N = L::N, EX = L::EX, EY = L::EY, SX = L::SX, ES = L::ES;
    for (int q = 0; q < L::NFX; ++q) {  // x face (r, c), node l
      const int l = q % N, t = q / N, c = t % (EX + 1), r = t / (EX + 1);
      f[q].lo = (r * SX + c) * ES + (N - 1) + N * l;
      f[q].hi = (r * SX + c + 1) * ES + N * l;
    }
    for (int q = 0; q < L::NFY; ++q) {  // y face (r, c), node k
      const int k = q % N, t = q / N, c = t % EX, r = t / EX;
      f[L::NFX + q].lo = (r == 0 ? EY * SX + c : (r - 1) * SX + c + 1) * ES + k + N * (N - 1);
      f[L::NFX + q].hi = (r == EY ? EY * SX + EX + c : r * SX + c + 1) * ES + k;
      f[L::NFX + q].d = L::NN;
    }
  }
};
template <int P>
__device__ const FaceTable<P> d_faces = FaceTable<P>();

// Once per warp, before its first item: its copy barrier.
template <int P>
__device__ __forceinline__ void res2_prologue(double* wsm) {
  if ((threadIdx.x & 31) == 0) mbar_init(reinterpret_cast<unsigned long long*>(wsm + Res2Layout<P>::O_BAR), 1);
  __syncwarp();
}

// max over the NN lanes of this lane's element group (every lane of the group gets it); gbase =
// the group's first lane
template <int NN>
__device__ __forceinline__ double group_max(double v, int gbase) {
  if constexpr ((NN & (NN - 1)) == 0) {
#pragma unroll
    for (int o = NN / 2; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
  } else {
    double m = __shfl_sync(0xffffffffu, v, gbase);
#pragma unroll
    for (int r = 1; r < NN; ++r) m = fmax(m, __shfl_sync(0xffffffffu, v, gbase + r));
    return m;
  }
}

// Where an item's results go: the L(u) array and the control block (dt_lim).  Taken by reference,
// so that the batched kernel can keep it in shared memory, out of the registers.
struct TileOut {
  double* ut;
  Ctrl* ctrl;
};

__device__ __forceinline__ void st2(double* p, double a, double b) { *reinterpret_cast<double2*>(p) = make_double2(a, b); }
__device__ __forceinline__ double2 ld2(const double* p) { return *reinterpret_cast<const double2*>(p); }

// The next stage's element of this lane's group, from its combined node values x (ie, je: the element,
// act: this lane holds one of its nodes, base: the group's first lane).  Where the element is the source of ghost
// elements, those are formed first, as the boundary fill would from the values before the projection.
// scratch: shared memory of the warp, free of use.  An element whose average is inadmissible keeps its combined
// values, and its average and entropies of the stage before (the try is abandoned then).
//
// In place of a boundary fill and loop 1 as launches of their own for every stage after the first: the
// state is neither written before the projection nor read again.  400^2, p = 3, one stage (us): residual
// with its combination 176 + fill 3 + loop 1 61-75 -> 240-250 and 330 MB less traffic; on small meshes two
// launches less a stage (fold_post, mhd_gpu.cu).  Staging u_con's blocks with the others by bulk copies gains 1.3 % of
// a step where the state exceeds L2 and costs 1-2 % elsewhere and 4 % of a batch; fetching them to L2
// ahead gains nothing.
template <int P>
__device__ __forceinline__ void stage_post(const double* x, const StagePost& sp, const Geo& g, Ctrl* ctrl, int ie,
                                           int je, bool rim, bool act, int grp, int base, int node, double* scratch) {
  using L = Res2Layout<P>;
  constexpr int N = L::N, NN = L::NN, EB = L::EB, G = L::G;
  constexpr unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, k = node % N, l = node / N;
  const bool nd = grp < G;  // (the lanes past the groups mirror the first)
  const DegConst& dc = c_deg[P];
  const double w = 0.25 * dc.qw[k] * dc.qw[l];
  double* row = scratch + (nd ? grp : 0) * (2 * NN + 2);
  // the left, right, bottom and top ghost of the element, where it is their source; then itself
#pragma unroll 1
  for (int side = rim ? 0 : 4; side <= 4; ++side) {
    const int ti = side == 0 ? 0 : side == 1 ? g.nx + 1 : ie, tj = side == 2 ? 0 : side == 3 ? g.ny + 1 : je;
    const bool ghost = side < 4;
    bool mine = act;
    double y[8];
    if (ghost) {
      const BcSrc b = bc_source<P>(g, ti, tj, 0, node);
      const int si = b.fixed ? min(max(ti, 1), g.nx) : b.si, sj = b.fixed ? min(max(tj, 1), g.ny) : b.sj;
      mine = act && si == ie && sj == je;
      if (!__any_sync(FULL, mine)) continue;
#pragma unroll
      for (int v = 0; v < 8; ++v) {
        const double t = __shfl_sync(FULL, x[v], base + b.sq);
        y[v] = b.fixed ? g.bc_state[v] : (bc_source<P>(g, ti, tj, v, node).neg ? -t : t);
      }
    } else {
#pragma unroll
      for (int v = 0; v < 8; ++v) y[v] = x[v];
    }
    // cell averages (DG_solver.f90:177-184)
    double avg[8];
#pragma unroll
    for (int v = 0; v < 8; ++v) avg[v] = w * y[v];
    if constexpr ((NN & (NN - 1)) == 0) {
      grp_sum8<NN>(avg, row);
    } else {  // nine lanes: variable q is summed by lane q of the group
      double* t = scratch + G * (2 * NN + 2) + (nd ? grp : 0) * (8 * NN);
      if (nd)
#pragma unroll
        for (int v = 0; v < 8; ++v) t[v * NN + node] = avg[v];
      __syncwarp();
      if (nd && node < 8) {
        const double* r = t + node * NN;
        row[node] = (((r[0] + r[8]) + r[4]) + (r[2] + r[6])) + ((r[1] + r[5]) + (r[3] + r[7]));  // as grp_sum8 adds
      }
      __syncwarp();
#pragma unroll
      for (int v = 0; v < 8; v += 2) {
        const double2 p = ld2(row + v);
        avg[v] = p.x;
        avg[v + 1] = p.y;
      }
    }
    const long long e = (long long)tj * (g.nx + 2) + ti;
    // admissibility of the average (DG_solver.f90:186-193)
    const double pa = prs_of(avg[0], avg[1], avg[2], avg[3], avg[4], avg[5], avg[6], avg[7], g.gamma);
    const bool ok = mine && !(avg[0] < PP_EPS || pa < PP_EPS);
    if (mine && !ok && node == 0) atomicOr(&ctrl->neg_avg, 1);
    if (ok) {
#pragma unroll
      for (int v0 = 0; v0 < 8; v0 += NN)
        if (node + v0 < 8) sp.u_avg[e * 8 + node + v0] = row[node + v0];
    }
    __syncwarp();  // the row is rewritten next
    if (!ghost && sp.ent_offset) {  // cell entropies (DG_solver.f90:195-224)
      const double pq = act ? node_prs(y, g.gamma) : 0.0;
      const bool okq = !act || (y[0] >= PP_EPS && pq >= PP_EPS);
      const double okall = grp_min<NN>(okq ? 1.0 : 0.0);
      const double ce = grp_sum<NN>((act && okall > 0.5) ? 0.25 * g.hx * g.hy * dc.qw[k] * dc.qw[l] * ent_of(y[0], pq, g.gamma, g.igm1) : 0.0);
      if (ok && node == 0) {
        sp.cell_ent_FV[e] = ent_of(avg[0], pa, g.gamma, g.igm1);
        sp.cell_ent_DG[e] = okall > 0.5 ? ce : 0.0;
        sp.cell_ent_nan[e] = okall > 0.5 ? 0 : 1;
      }
      __syncwarp();  // limit_group reads them
    }
    if (ghost && !sp.final) continue;  // the end of the stage fills its ghosts again
    if (sp.use_ldf) {
      double bx = y[4] - avg[4], by = y[5] - avg[5];
      ldf_project<P>(bx, by, base, node, nd, row, reinterpret_cast<const double2*>(g.ldfA));
      if (ok) {
        y[4] = bx + avg[4];
        y[5] = by + avg[5];
      }
    }
    if (!sp.final) {
      bool neg = false;
      limit_group<P, NN>(y, avg, ok, node == 0, node, e, g, ctrl, sp.ent_offset, 0, sp.cell_ent_DG, sp.cell_ent_FV,
                         sp.cell_ent_nan, &neg);
      const unsigned cnt = __popc(__ballot_sync(FULL, neg));
      if (lane == 0 && cnt) atomicAdd(&ctrl->num_negcell, (int)cnt);
    }
    if (mine) {
      double* o = sp.out + e * EB + node;
#pragma unroll
      for (int v = 0; v < 8; ++v) o[v * NN] = y[v];
    }
  }
}

// One item: elements i0 = ix*EX + 1 .., j0 = iy*EY + 1 .. of the mesh (at least one of them inside).
// wsm = the warp's shared memory (after res2_prologue).  ug = the array whose ghost
// ring the boundary traces come from (u itself, or the last stage array whose ring was filled from
// u's interior after the final stage; the interior always comes from u).  `phase` = the parity of the
// warp's barrier (flipped here).  The whole warp calls it.  Returns false if the wait for the copies
// ran out (FLAG_DEVICE_WAIT is then set): the warp must stop.
template <int P, int MODE>
__device__ __forceinline__ bool residual_item(const double* __restrict__ u, const double* __restrict__ ug,
                                              const TileOut& to, const Geo& g, int ix, int iy, double* wsm,
                                              unsigned& phase, const StagePost& sp) {
  using L = Res2Layout<P>;
  constexpr int N = L::N, NN = L::NN, EB = L::EB, EX = L::EX, EY = L::EY, NFX = L::NFX, NF = L::NF;
  constexpr int ES = L::ES, SX = L::SX;
  constexpr unsigned FULL = 0xffffffffu;
  double* s_node = wsm + L::O_NODE;
  const DegRows& rows = d_rows[P];
  const int lane = threadIdx.x & 31;
  const int nx = g.nx, ny = g.ny;
  const int i0 = 1 + ix * EX, j0 = 1 + iy * EY;
  const int W = min(EX, nx - i0 + 1), H = min(EY, ny - j0 + 1);
  const long long rowstride = (long long)(nx + 2) * EB;
  const double gamma = g.gamma, igm1 = g.igm1;
  // dt_lim so far: a bound that spares most items the exact reduction of step 4
  const unsigned long long dt_bits = *reinterpret_cast<const volatile unsigned long long*>(&to.ctrl->dt_lim_bits);

  // ---- 0. the element blocks, one copy per lane ----
  unsigned long long* bar = reinterpret_cast<unsigned long long*>(wsm + L::O_BAR);
  {
    int c, r, slot = lane;  // column i0 + c, row j0 + r of the lane's block
    bool live;
    if (lane < EY * SX) {
      r = lane / SX;
      c = lane - r * SX - 1;
      live = r < H && c <= W;
    } else {
      const int q = lane - EY * SX;
      r = q < EX ? -1 : H;
      c = q < EX ? q : q - EX;
      live = lane < L::NCOPY && c < W;
      if (EY > 1 && q >= EX && H < EY) slot = H * SX + c + 1;  // a ragged item's row above (FaceDesc)
    }
    fence_proxy_async_smem();  // the previous item's accesses of this memory come before the copies
    const unsigned n = __popc(__ballot_sync(FULL, live));
    if (lane == 0) mbar_arrive_expect_tx(bar, n * (EB * 8));
    __syncwarp();
    if (live) {
      const int i = i0 + c, j = j0 + r;
      const double* src = (i == 0 || i == nx + 1 || j == 0 || j == ny + 1) ? ug : u;
      bulk_copy_g2s(wsm + slot * ES, src + j * rowstride + (long long)i * EB, EB * 8, bar);
    }
  }
  if (!__all_sync(FULL, mbar_wait_bounded(bar, phase & 1u))) {  // flag it, give the copies one more bound, stop
    if (lane == 0) atomicOr(&to.ctrl->flags, FLAG_DEVICE_WAIT);
    mbar_wait_bounded(bar, phase & 1u);
    __syncwarp();
    return false;
  }
  phase ^= 1u;

  // ---- 1. interface fluxes ----
#pragma unroll 1
  for (int f = lane; f < NF; f += 32) {
    const int4 desc = __ldg(reinterpret_cast<const int4*>(&d_faces<P>.f[f]));
    const double *plo = wsm + desc.x, *phi = wsm + desc.y;
    // a y face takes its vectors with the first two components exchanged (swap_xy): 1 <-> 2, 4 <-> 5
    const double *plo_p = plo + desc.z, *plo_m = plo - desc.z, *phi_p = phi + desc.z, *phi_m = phi - desc.z;
    double wl[8], wr[8], o[12];
#pragma unroll
    for (int v = 0; v < 8; ++v) {
      const bool up = v == 1 || v == 4, down = v == 2 || v == 5;
      wl[v] = (up ? plo_p : down ? plo_m : plo)[v * NN];
      wr[v] = (up ? phi_p : down ? phi_m : phi)[v * NN];
    }
    espp_hll(wl, wr, gamma, igm1, o);
    double* rec = wsm + L::O_FACE + f * L::FS;
    st2(rec, o[0], o[1]);
    st2(rec + 2, o[2], o[3]);
    st2(rec + 4, o[4], o[5]);
    st2(rec + 6, o[6], o[7]);
    st2(rec + 8, o[8], o[11]);
    st2(rec + 10, o[9], o[10]);
  }

  __syncwarp();  // the rows below and above are read: the node records take their place

  // ---- 2. the nodes' primitives ----
  const int grp = lane / NN, gq = grp < L::G ? grp : 0;  // lanes beyond the groups mirror the first
  const int node = lane - grp * NN;
  const int gc = gq % EX, gr = gq / EX;
  const bool act = grp < L::G && gc < W && gr < H;
  const int gbase = gq * NN;
  const int k = node % N, l = node / N;
  const double* un = wsm + ((act ? gr : 0) * SX + (act ? gc : 0) + 1) * ES + node;  // the node's staged state
  const double sxh = g.sxh, syh = g.syh;
  const double sxq = 0.5 * sxh, syq = 0.5 * syh;  // 2 (2/h) / 4: the pair fluxes come as four times the flux
  // (all arithmetic of L(u) is exactly rounded as written: dmul/dadd/dsub/dfma of common.cuh, so
  // that each kernel it is inlined into rounds it the same way: a batch member equals its solo run)
  double sgx, sgy, bsq, pp[8];  // bounds of the wave speeds, |B|^2; pp: (rho, vx, vy, vz, Bx, By, Bz, beta), the EC flux's inputs
  {
    double w[8];
#pragma unroll
    for (int v = 0; v < 8; ++v) w[v] = un[v * NN];
    const double ir = rcp_any(w[0]);
    const double vx = dmul(ir, w[1]), vy = dmul(ir, w[2]), vz = dmul(ir, w[3]);
    bsq = dsq3(w[4], w[5], w[6]);
    const double pf = gas_pressure(dsub(gamma, 1.0), ddot3(w[1], vx, w[2], vy, w[3], vz), bsq, w[7]);
    pp[0] = w[0];
    pp[1] = vx;
    pp[2] = vy;
    pp[3] = vz;
    pp[4] = w[4];
    pp[5] = w[5];
    pp[6] = w[6];
    pp[7] = dmul(dmul(0.5, w[0]), rcp_nr(pf));
    double* rec = s_node + lane * L::NS;
    st2(rec, pp[0], pp[7]);
    st2(rec + 2, pp[1], pp[2]);
    st2(rec + 4, pp[3], pp[6]);
    st2(rec + 6, pp[4], pp[5]);
    st2(rec + 8, bsq, pf);
    // an upper bound of the node's fast speeds, c_f^2 <= gamma p/rho + |B|^2/rho (see dt_lim below)
    const double cb = sqrt_nr(dmul(dfma(gamma, pf, bsq), ir));
    sgx = dadd(fabs(vx), cb);
    sgy = dadd(fabs(vy), cb);
  }
  __syncwarp();  // the face and node records are in place

  // ---- 3. node-pair fluxes ----
  const double pref = s_node[gbase * L::NS + 9], pref4 = dmul(4.0, pref);  // the element's reference pressure (ec_flux4)
  // the lane d nodes further along x or y (cyclically) in this lane's element
  auto along_x = [&](int d) {
    if constexpr (P == 1) return lane ^ 1;
    else if constexpr (P == 3) return (lane & ~3) | ((lane + d) & 3);
    else return gbase + N * l + (k + d < N ? k + d : k + d - N);
  };
  auto along_y = [&](int d) {
    if constexpr (P == 1) return lane ^ 2;
    else if constexpr (P == 3) return (lane & ~12) | ((lane + 4 * d) & 12);
    else return gbase + k + N * (l + d < N ? l + d : l + d - N);
  };
  // The node's own flux never appears: the diagonal of the flux differencing, -2 (2/h) D_kk F(u_k)
  // (DG_solver.f90:833), is zero inside the element (D_kk = 0), and at an end node it is cancelled by
  // the own-flux part of that face's surface term (DG_solver.f90:872-882), because 2 D_NN = 1/w_N =
  // -2 D_00 (the summation-by-parts property of the GLL rule).  What remains of the surface term is
  // the interface flux and a multiple of the Godunov-Powell vector, which joins the -div B one.
  //
  // Four times this lane's flux with the node of record `src` (x frame, or y through swap_xy); the
  // result F is in the global frame.
  double F[8];
  auto pair_flux = [&](int src, bool ydir) {
    const double* rec = s_node + src * L::NS;
    const double2 b0 = ld2(rec), b1 = ld2(rec + 2), b2 = ld2(rec + 4), b3 = ld2(rec + 6);
    const double bsq_src = rec[8];
    double A[8], B[8];
    A[0] = pp[0];
    A[1] = ydir ? pp[2] : pp[1];
    A[2] = ydir ? pp[1] : pp[2];
    A[3] = pp[3];
    A[4] = ydir ? pp[5] : pp[4];
    A[5] = ydir ? pp[4] : pp[5];
    A[6] = pp[6];
    A[7] = pp[7];
    B[0] = b0.x;
    B[1] = ydir ? b1.y : b1.x;
    B[2] = ydir ? b1.x : b1.y;
    B[3] = b2.x;
    B[4] = ydir ? b3.y : b3.x;
    B[5] = ydir ? b3.x : b3.y;
    B[6] = b2.y;
    B[7] = b0.y;
    double f[8];
    ec_flux4(A, B, bsq, bsq_src, igm1, pref4, f);
#pragma unroll
    for (int v = 0; v < 8; ++v) F[v] = ydir ? f[swap_xy_var(v)] : f[v];
  };
  // the flux that lane `src` computed, but for component `skip` (every lane of the warp calls it)
  auto received = [&](int src, double* R, int skip) {
#pragma unroll
    for (int v = 0; v < 8; ++v)
      if (v != skip) R[v] = __shfl_sync(FULL, F[v], src);
  };
  // row k (or l) of D starting at its diagonal: Dk(r) = D[k][(k + r) mod N]
  auto Dk = [&](int r) { return __ldg(&rows.row[k][r]); };
  auto Dl = [&](int r) { return __ldg(&rows.row[l][r]); };
  double acc[8], R[8];
  if constexpr (P == 1) {
    const bool xb = (k == l);
    pair_flux(xb ? along_x(1) : along_y(1), !xb);
    received(xb ? along_y(1) : along_x(1), R, -1);
    const double cx = -(sxq * Dk(1)), cy = -(syq * Dl(1));
    const double c1 = xb ? cx : cy, c2 = xb ? cy : cx;
#pragma unroll
    for (int v = 0; v < 8; ++v) acc[v] = dfma(c2, R[v], dmul(c1, F[v]));
  } else {
    // rings along x and y: compute with the next node, receive from the previous one
#pragma unroll
    for (int dir = 0; dir < 2; ++dir) {
      pair_flux(dir == 0 ? along_x(1) : along_y(1), dir == 1);
      received(dir == 0 ? along_x(N - 1) : along_y(N - 1), R, dir == 0 ? 4 : 5);
      const double h2 = dir == 0 ? -sxq : -syq;
      const double c1 = h2 * (dir == 0 ? Dk(1) : Dl(1)), c2 = h2 * (dir == 0 ? Dk(N - 1) : Dl(N - 1));
#pragma unroll
      for (int v = 0; v < 8; ++v) {
        if (v == (dir == 0 ? 4 : 5)) continue;  // that component of the flux is identically zero
        acc[v] = dfma(c2, R[v], (dir == 0 || v == 4) ? dmul(c1, F[v]) : dfma(c1, F[v], acc[v]));
      }
    }
    if constexpr (P == 3) {  // the pairs (k, k^2) along x and (l, l^2) along y
      const bool xb = ((k >> 1) ^ (l >> 1)) == 0;
      pair_flux(xb ? along_x(2) : along_y(2), !xb);
      received(xb ? along_y(2) : along_x(2), R, -1);
      const double cx = -(sxq * Dk(2)), cy = -(syq * Dl(2));
      const double c1 = xb ? cx : cy, c2 = xb ? cy : cx;
#pragma unroll
      for (int v = 0; v < 8; ++v) acc[v] = dfma(c2, R[v], dfma(c1, F[v], acc[v]));
    }
  }

  // ---- 4. interface fluxes, Godunov-Powell terms; dt_lim; store ----
  double fx = 0.0, fy = 0.0;  // the node's interface speeds
  {
    // local div B (DG_solver.f90:813)
    double dbx = 0.0, dby = 0.0;
#pragma unroll
    for (int r = 1; r < N; ++r) {  // the rows of D sum to zero: of differences, so that a constant field has none
      dbx = dfma(Dk(r), dsub(__shfl_sync(FULL, pp[4], along_x(r)), pp[4]), dbx);
      dby = dfma(Dl(r), dsub(__shfl_sync(FULL, pp[5], along_y(r)), pp[5]), dby);
    }
    // (2/h)/w times the interface flux, + at the first node of a line and - at the last; `src`
    // collects the factor of the Godunov-Powell vector (0, B, v, v.B) (DG_solver.f90:794-799)
    double src = -dfma(syh, dby, dmul(sxh, dbx));
    if (k == 0 || k == N - 1) {
      const bool right = (k == N - 1);
      const double* fr = wsm + L::O_FACE + ((gr * (EX + 1) + gc + (right ? 1 : 0)) * N + l) * L::FS;
      const double2 f0 = ld2(fr), f1 = ld2(fr + 2), f2 = ld2(fr + 4), f3 = ld2(fr + 6), f4 = ld2(fr + 8), s = ld2(fr + 10);
      const double c = (right ? -sxh : sxh) * __ldg(&rows.iqw[k]);
      src = dfma(-c, dsub(pp[4], f4.x), src);
      acc[0] = dfma(c, f0.x, acc[0]);
      acc[1] = dfma(c, dadd(f0.y, dsub(f4.y, pref)), acc[1]);
      acc[2] = dfma(c, f1.x, acc[2]);
      acc[3] = dfma(c, f1.y, acc[3]);
      acc[4] = dfma(c, f2.x, acc[4]);
      acc[5] = dfma(c, f2.y, acc[5]);
      acc[6] = dfma(c, f3.x, acc[6]);
      acc[7] = dfma(c, f3.y, acc[7]);
      fx = right ? -s.x : s.y;
    }
    if (l == 0 || l == N - 1) {
      const bool top = (l == N - 1);
      const double* fr = wsm + L::O_FACE + (NFX + ((gr + (top ? 1 : 0)) * EX + gc) * N + k) * L::FS;
      const double2 f0 = ld2(fr), f1 = ld2(fr + 2), f2 = ld2(fr + 4), f3 = ld2(fr + 6), f4 = ld2(fr + 8), s = ld2(fr + 10);
      const double c = (top ? -syh : syh) * __ldg(&rows.iqw[l]);
      src = dfma(-c, dsub(pp[5], f4.x), src);
      acc[0] = dfma(c, f0.x, acc[0]);
      acc[1] = dfma(c, f1.x, acc[1]);  // (the record is in the face's frame: swap_xy)
      acc[2] = dfma(c, dadd(f0.y, dsub(f4.y, pref)), acc[2]);
      acc[3] = dfma(c, f1.y, acc[3]);
      acc[4] = dfma(c, f2.y, acc[4]);
      acc[5] = dfma(c, f2.x, acc[5]);
      acc[6] = dfma(c, f3.x, acc[6]);
      acc[7] = dfma(c, f3.y, acc[7]);
      fy = top ? -s.x : s.y;
    }
    const double gp[8] = {0.0, pp[4], pp[5], pp[6], pp[1], pp[2], pp[3],
                          ddot3(pp[4], pp[1], pp[5], pp[2], pp[6], pp[3])};
    // The terms with a factor of zero that the reference's sum has matter where a value is not finite: the
    // vector's mass part, and the energy's own flux, in which alone an energy that is NaN is not clamped away.
#pragma unroll
    for (int v = 0; v < 8; ++v) acc[v] = dfma(src, gp[v], acc[v]);
    acc[7] = dfma(0.0, un[7 * NN], acc[7]);
  }
  if ((MODE == RES_UT || MODE == RES_POST54) && act) {
    double* o = to.ut + ((long long)(j0 + gr - 1) * nx + (i0 + gc - 1)) * EB + node;
#pragma unroll
    for (int v = 0; v < 8; ++v) o[v * NN] = acc[v];
  }
  // dt_lim of an element: the largest node speed and interface speed per direction.  The exact
  // node speeds and maxima are only formed where the item could lower dt_lim: the largest bounds of
  // the whole warp, rounded up to single precision, bound every element's dt from below (1e-12 covers
  // the rounding of the bound and of the exact value).  A node's bound that is NaN, as where its density is negative
  // or zero, stays NaN here (at_least, not fmax), orders above all others, and like an empty dt_lim takes the
  // exact path, where only what is NaN itself is left out.
  const unsigned ux = __reduce_max_sync(FULL, __float_as_uint(__double2float_ru(act ? at_least(fx, sgx) : 0.0)));
  const unsigned uy = __reduce_max_sync(FULL, __float_as_uint(__double2float_ru(act ? at_least(fy, sgy) : 0.0)));
  const double bound = (P + 0.5) * ((double)__uint_as_float(ux) * sxh + (double)__uint_as_float(uy) * syh);
  const double dt_now = __longlong_as_double((long long)__shfl_sync(FULL, dt_bits, 0));  // one value for the warp
  if (!(bound * dt_now * (1.0 + 1.0e-12) <= 1.0)) {
    const double pf = s_node[lane * L::NS + 9], ir = rcp_any(pp[0]);
    const double cs = dmul(dmul(gamma, pf), ir), ss = dfma(bsq, ir, cs), coef = dmul(dmul(4.0, cs), ir);
    auto speed = [&](double v, double bn) {  // |v| + the fast speed along the direction of bn (DG_solver.f90:784-787)
      const double disc = at_least(dfma(ss, ss, -dmul(coef, dmul(bn, bn))), TINY);
      return dadd(fabs(v), sqrt_any(dmul(0.5, at_least(dadd(ss, sqrt_any(disc)), TINY))));
    };
    const double ax = group_max<NN>(act ? fmax(fx, speed(pp[1], pp[4])) : 0.0, gbase);
    const double ay = group_max<NN>(act ? fmax(fy, speed(pp[2], pp[5])) : 0.0, gbase);
    double my_dt = 1.0e300;
    if (act && node == 0) my_dt = 1.0 / dmul(P + 0.5, dfma(ax, sxh, dmul(ay, syh)));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) my_dt = fmin(my_dt, __shfl_xor_sync(FULL, my_dt, o));
    if (lane == 0) atomicMin(&to.ctrl->dt_lim_bits, (unsigned long long)__double_as_longlong(my_dt));
  }
  if constexpr (MODE != RES_UT) {  // the next stage
    const int ie = i0 + gc, je = j0 + gr;
    const long long at = ((long long)je * (nx + 2) + ie) * EB + node, ki = ((long long)(je - 1) * nx + (ie - 1)) * EB + node;
    double x[8];
#pragma unroll
    for (int v = 0; v < 8; ++v) x[v] = 0.0;
    if (act) {
      const double dt = *sp.dt;
      stage_node<NN, MODE>(x, sp, dt, un, acc, at, ki);
    }
    if constexpr (MODE == RES_COMBINE) {
      if (act)
#pragma unroll
        for (int v = 0; v < 8; ++v) sp.out[at + v * NN] = x[v];
    } else {
      __syncwarp();  // the face records are read: their place is scratch from here on
      const bool rim = i0 == 1 || j0 == 1 || i0 + EX > nx || j0 + EY > ny;  // an element on the boundary
      stage_post<P>(x, sp, g, to.ctrl, ie, je, rim, act, grp, gbase, node, wsm + L::O_FACE);
    }
  }
  return true;
}

// items of a mesh: columns and rows
template <int P>
__host__ __device__ inline int res2_item_cols(int nx) { return (nx + Res2Layout<P>::EX - 1) / Res2Layout<P>::EX; }
template <int P>
__host__ __device__ inline int res2_item_rows(int ny) { return (ny + Res2Layout<P>::EY - 1) / Res2Layout<P>::EY; }

// single instance: one CTA per TX x TY block of elements, rows counted through y and z (residual_grid; ug: the
// ghost-ring source, see residual_item)
template <int P, int MODE>
__global__ void __launch_bounds__(Res2Layout<P>::NT, Res2Layout<P>::MINB)
    residual2_kernel(const double* u, const double* ug, double* __restrict__ ut, Geo g,
                     Ctrl* ctrl, int gate, StagePost sp) {
  using L = Res2Layout<P>;
  extern __shared__ __align__(16) double sm[];
  const int warp = threadIdx.x >> 5;
  const int ix = blockIdx.x * L::IX + warp % L::IX, iy = (blockIdx.z * gridDim.y + blockIdx.y) * L::IY + warp / L::IX;
  double* wsm = sm + warp * L::WARP;
  res2_prologue<P>(wsm);
  grid_begin();
  if (!gate_open(ctrl, gate) || ix * L::EX >= g.nx || iy * L::EY >= g.ny) return;
  unsigned phase = 0;
  residual_item<P, MODE>(u, ug, TileOut{ut, ctrl}, g, ix, iy, wsm, phase, sp);
}

// single instance, persistent: the grid's warps take the items in turn (row-major, ncol per row).
// For a launch that is usually gated off (the re-try residual of every try): a grid of resident
// CTAs that return at once costs far less than one CTA per block.
template <int P>
__global__ void __launch_bounds__(Res2Layout<P>::NT, Res2Layout<P>::MINB)
    residual2_persistent(const double* u, double* __restrict__ ut, Geo g, Ctrl* ctrl, int gate,
                         int ncol, int nitems) {
  grid_begin();
  using L = Res2Layout<P>;
  if (!gate_open(ctrl, gate)) return;
  extern __shared__ __align__(16) double sm[];
  const int warp = threadIdx.x >> 5;
  double* wsm = sm + warp * L::WARP;
  res2_prologue<P>(wsm);
  unsigned phase = 0;
  for (int t = blockIdx.x * L::NW + warp; t < nitems; t += gridDim.x * L::NW)
    if (!residual_item<P, RES_UT>(u, u, TileOut{ut, ctrl}, g, t % ncol, t / ncol, wsm, phase, StagePost{}))
      return;
}

// many instances of degree P: each warp of a persistent grid walks its share of every member's items
// (row-major per member); the state is slot `src`, the result goes to ut[dst], or stage
// dst to slot dst (RES_POST).  L(u) and the combination are fully rounded as written (explicit fused
// multiply-adds, see common.cuh), so a member is bitwise equal to its solo run although this is a different
// kernel.  Loops 1 and 3 of the stage formed (stage_post) are not: there the equality with the solo kernels and
// with the launches of their own rests on the compiler contracting the same inlined code alike, and on
// tests/test_gpu_folded_stages.py and test_gpu_folded_solo.py, which compare the three.
template <int P, int MODE>
__global__ void __launch_bounds__(Res2Layout<P>::NT, Res2Layout<P>::MINB)
    residual2_batched(const InstDesc* __restrict__ insts, const int* __restrict__ pref,
                      const int* __restrict__ nwork, const int* __restrict__ ninst, int src, int dst, int gate) {
  using L = Res2Layout<P>;
  extern __shared__ __align__(16) double sm[];
  // per warp: the walker and the member's geometry, stage combination and outputs, read where they
  // are used instead of held in registers (the single-instance kernel reads them from its parameters)
  struct WarpArgs {
    SharedWalk walk;
    Geo g;
    StagePost sp;
    TileOut to;
  };
  __shared__ WarpArgs s_args[L::NW];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  WarpArgs& a = s_args[warp];
  double* wsm = sm + warp * L::WARP;
  if (lane == 0) a.walk.start(pref, *ninst, *nwork, blockIdx.x * L::NW + warp, gridDim.x * L::NW);
  res2_prologue<P>(wsm);  // (ends with a barrier of the warp)
  unsigned phase = 0;
  while (a.walk.w < a.walk.last) {
    const int m = a.walk.m, local = a.walk.w - a.walk.mstart;
    const InstDesc& d = insts[m];
    const bool open = gate_open(d.ctrl, gate);
    __syncwarp();  // every lane has read the walker, and is done with the previous item's arguments
    if (lane == 0) {
      if (open) {
        a.g = d.g;
        if constexpr (MODE >= RES_POST)
        {
          stage_scheme(a.sp, d.R, dst, d.u, d.ut);
          a.sp.dt = &d.ctrl->dt;
          a.sp.u_avg = d.u_avg;
          a.sp.cell_ent_DG = d.cell_ent_DG;
          a.sp.cell_ent_FV = d.cell_ent_FV;
          a.sp.cell_ent_nan = d.cell_ent_nan;
          a.sp.use_ldf = d.use_ldf;
          a.sp.ent_offset = d.ent_offset;
        }
        a.to = TileOut{d.ut[dst], d.ctrl};
      }
      a.walk.advance(pref);
    }
    __syncwarp();
    if (open) {
      const int ncol = res2_item_cols<P>(a.g.nx);
      // the state after the final stage: u_con's interior with the last stage array's ghost ring
      const int srci = (src == d.R) ? 0 : src;
      if (!residual_item<P, MODE>(d.u[srci], d.u[src], a.to, a.g, local % ncol, local / ncol, wsm, phase, a.sp))
        return;
    }
  }
}

}  // namespace mhd
