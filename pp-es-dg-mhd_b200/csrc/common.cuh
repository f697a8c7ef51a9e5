// common.cuh -- shared device definitions of the sm_100a DG-MHD stage pipeline.
//
// Device data layout (HBM): a state is element-blocked,
//     u[ j ][ i ][ var ][ node ],  j in 0..ny+1, i in 0..nx+1 (one ghost ring),
// node = k + n*l with n = p+1 GLL nodes per direction, var in 0..7 = (rho, mx, my, mz, Bx, By,
// Bz, E).  One element block is 8*n*n doubles (256 B at p=1, 576 B at p=2, 1 KiB at p=3), so a
// row of a tile of elements is one contiguous, 16-byte aligned run and every kernel moves tiles
// with 128-bit loads.  The time derivative ut has the same per-element blocks without the ghost
// ring: ut[ j-1 ][ i-1 ][ var ][ node ].
#pragma once
#include <cstring>
#include <cstdint>
#include <cuda_runtime.h>

namespace mhd {

constexpr double PP_EPS = 1.0e-11;   // DG_solver.f90:17
constexpr double OEDG_EPS = 1.0e-8;  // DG_solver.f90:148
constexpr int MAXP = 3;              // kernels are instantiated for p = 1, 2, 3
constexpr int MAXN = MAXP + 1;

// Per-degree tables in constant memory (gauss.f90 tables computed on the host).
struct DegConst {
  double qx[MAXN];          // GLL nodes
  double qw[MAXN];          // GLL weights
  double iqw[MAXN];         // their reciprocals
  double D[MAXN * MAXN];    // nodal differentiation matrix, column-major D[i + n*j]
  double R0[MAXN][MAXN];    // R0[kk][k] = (D^kk)(0,k)    first row of D^kk
  double RN[MAXN][MAXN];    // RN[kk][k] = (D^kk)(n-1,k)  last row of D^kk
};
// Defined here: the device code of the library is one translation unit (mhd_gpu.cu).
__constant__ DegConst c_deg[MAXP + 1];
// The rows of D for lanes that each want their own (a constant-memory read is replayed once per
// distinct address): row k starting at its diagonal, row[k][r] = D(k, (k + r) mod n), 16-byte aligned,
// and 1/w_k.  In global memory, read through L1.
struct DegRows {
  double row[MAXN][4];
  double iqw[MAXN];
};
__device__ DegRows d_rows[MAXP + 1];

// Status flag bits of the control block (the MHD_FLAG_* values of mhd_gpu.h).  FLAGS_FATAL: the
// bits that end a run (every bit but the per-stage inadmissible average).
constexpr int FLAG_DEVICE_WAIT = 16;
constexpr int FLAGS_FATAL = 2 | 4 | 8 | FLAG_DEVICE_WAIT;

// Gate values: a kernel launched with gate >= 0 runs only if ctrl->state == gate.
enum GateState : int { GATE_ALWAYS = -1, ST_IDLE = 0, ST_RUN = 1, ST_RECOMPUTE = 2, ST_FAILED = 3 };

// Device-resident control block: the scalars of solve_execute (drive.f90:39-48) and the global
// reductions of post_process / DG_semidiscretize.
constexpr long long NO_STEP_LIMIT = 0x7fffffffffffffffLL;

struct Ctrl {
  double t, dt, dt_lim, final_T, cfl_total, tot_ent;
  double t_rk[6];
  double u_avg_global[8];   // DG_solver.f90:146,228
  unsigned long long dt_lim_bits;  // atomicMin target, bit pattern of a positive double
  unsigned long long umax_bits[8]; // max / min of the interior node values (u_vari_global,
                                   // DG_solver.f90:287-294), order-preserving encodings
  unsigned long long umin_bits[8];
  long long steps, retries, num_negcell_total;
  long long step_limit;  // ctl_step_begin idles once steps >= step_limit
  long long steps_from;  // steps when the budget was last set (ctl_step_budget)
  int state;
  int try_num;
  int last_step;     // flag == .false. in drive.f90:115-120
  int done;
  int flags;         // MHD_FLAG_* bits
  int neg_avg;       // post_process out (this stage)
  int num_negcell;   // post_process out (this stage)
  int num_negcell_last;
  int pp_relimit;
  int pending_dtlim; // a residual wrote dt_lim_bits that is not yet decoded
  unsigned sum_ticket;  // CTAs done with the global-average sum (pp_reduce_kernel); zero between launches
  int pad_;
  long long log_seq; // records written to the driver log so far (LogEntry)
};

// One record of the device-resident driver's log: per stage what drive.f90:285-294 prints (the
// PP-limited cell count, an abandoned stage), per accepted step what drive.f90:314 appends (t and
// the total entropy).  The public struct mhd_log_entry (mhd_gpu.h) has the same layout.  The
// diagnostic fields (rho_min, p_min, total) are NaN unless the instance runs the stage diagnostics.
struct LogEntry {
  long long seq;       // running record number
  long long step;      // time step (1-based; 0 = the initial state)
  int kind;            // LOG_STAGE or LOG_STEP
  int stage;           // RK stage (stage records)
  int try_num;         // try of the step (1 = first)
  int num_negcell;     // PP-limited cells of the stage (stage records)
  int neg_avg;         // the stage had an inadmissible average and the try was abandoned
  int flags;           // MHD_FLAG_* bits after the record
  double t;            // stage: its pseudo-time t_RK(s); step: the time reached
  double dt;           // dt of the try
  double dt_lim;       // step records: dt_lim of the last residual
  double tot_ent;      // step records: total entropy of the accepted state
  double rho_min, p_min;  // minimum nodal density and pressure of the stage state
  double total[8];        // sum over interior nodes of (hx hy / 4) w_k w_l u: the domain integrals
};
enum LogKind : int { LOG_STAGE = 1, LOG_STEP = 2 };

// The next record of a log ring of `cap` records (nullptr if the instance keeps no log); its
// diagnostic fields start as NaN.  Single thread.
__device__ __forceinline__ LogEntry* log_next(LogEntry* log, int cap, Ctrl* c) {
  if (!log || cap <= 0) return nullptr;
  const long long s = c->log_seq;
  c->log_seq = s + 1;
  LogEntry* e = log + (s % cap);
  const double nan = __longlong_as_double(0x7ff8000000000000LL);
  e->seq = s;
  e->rho_min = e->p_min = nan;
  for (int v = 0; v < 8; ++v) e->total[v] = nan;
  return e;
}

// Per-instance geometry passed by value.
struct Geo {
  int nx, ny;
  double hx, hy, gamma;
  int bc_kind;
  int pad_;
  double bc_state[8];
  const double* ldfA;  // the LDF operator as loop 1 applies it (tables.h, ldf_table), device memory
  double sxh, syh, igm1;  // 2/hx, 2/hy, 1/(gamma-1) (geo_constants)
};

// doubles of the LDF table of degree p: 2 per node and input slot
__host__ __device__ constexpr int ldf_table_doubles(int p) {
  return 2 * (p + 1) * (p + 1) * 2 * ((p + 2) / 2) * ((p + 2) / 2);
}

// Launch of a kernel of a chain, each of which waits by grid_begin: its CTAs may start while its predecessor in
// the stream still runs, so that the end of one kernel hides the start of the next.  Plain -> early (us a step): p = 1, 48^2
// (a run of 0.25 time units) 9.3 -> 8.5 ms, 512^2 486 -> 475; p = 2, 400^2 blast 691 -> 683; p = 3, 200^2
// 338 -> 332, 512^2 vortex 1506 -> 1494.  Nearest to a loss: p = 3, 250^2 413 -> 414.
template <typename... K, typename... A>
void launch_next(cudaStream_t st, dim3 grid, int block, size_t smem, void (*kernel)(K...), A... args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, static_cast<K>(args)...);
}

// the quotients every thread would form again
inline void geo_constants(Geo& g) {
  g.sxh = 2.0 / g.hx;
  g.syh = 2.0 / g.hy;
  g.igm1 = 1.0 / (g.gamma - 1.0);
}

// One solver instance as the batched kernels see it (a device-resident table entry).
struct InstDesc {
  Geo g;
  double* u[6];   // slot 0 = u_con, s = uRK_con(:,s)
  double* ut[6];  // 1..R
  double* u_avg;
  double* sig_x;
  double* sig_y;
  double* partial;
  double* ent_partial;
  double* cell_ent_DG;
  double* cell_ent_FV;
  unsigned char* cell_ent_nan;
  Ctrl* ctrl;
  LogEntry* log;   // driver log ring (nullptr: none)
  int log_cap;
  int use_oedg, use_ldf, ent_offset, R;
  int nseg_limit;  // pp_limit segments of this instance (entropy partials)
};

// Batched kernels see a group's work of one kind as the concatenation of every member's items;
// pref[m] is the first item of member m (pref[0] = 0, pref[n] = total).  Member of item w:
__device__ __forceinline__ int batch_member(const int* __restrict__ pref, int n, int w) {
  int lo = 0, hi = n;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (__ldg(pref + mid) <= w) lo = mid;
    else hi = mid;
  }
  return lo;
}

// The items a worker of a batched kernel (a CTA, or a warp of the residual) takes: one contiguous
// share [b*nw/G, (b+1)*nw/G) of the group's nw items (worker b of G), visited in order.  The member is found by binary search once and
// then walked forward, so consecutive items of one member reuse its descriptor (and whatever the
// kernel staged for it), and neighbouring tiles of a member are processed close in time.
// pref == nullptr: a single instance owns all nw items.
struct BatchWalk {
  const int* pref;
  int w, last, m, mstart, mend;
  __device__ __forceinline__ BatchWalk(const int* __restrict__ pref_, int n, int nw)
      : BatchWalk(pref_, n, nw, blockIdx.x, gridDim.x) {}
  __device__ __forceinline__ BatchWalk(const int* __restrict__ pref_, int n, int nw, long long b, long long G)
      : pref(pref_) {
    w = (int)(b * nw / G);
    last = (int)((b + 1) * nw / G);
    m = mstart = 0;
    mend = nw;
    if (pref && w < last) {
      m = batch_member(pref, n, w);
      mstart = __ldg(pref + m);
      mend = __ldg(pref + m + 1);
    }
  }
  __device__ __forceinline__ bool more() const { return w < last; }
  __device__ __forceinline__ int local() const { return w - mstart; }
  __device__ __forceinline__ void next() {
    ++w;
    while (w < last && w >= mend) {
      ++m;
      mstart = mend;
      mend = __ldg(pref + m + 1);
    }
  }
};

// BatchWalk's order of items with the walker's state in shared memory, for kernels whose items need
// every register: one thread starts and advances it, between barriers of the worker (CTA or warp).
struct SharedWalk {
  int w, last, m, mstart, mend;
  __device__ __forceinline__ void start(const int* __restrict__ pref, int n, int nw) {
    start(pref, n, nw, blockIdx.x, gridDim.x);
  }
  __device__ __forceinline__ void start(const int* __restrict__ pref, int n, int nw, long long b, long long G) {
    const BatchWalk it(pref, n, nw, b, G);
    w = it.w;
    last = it.last;
    m = it.m;
    mstart = it.mstart;
    mend = it.mend;
  }
  __device__ __forceinline__ void advance(const int* __restrict__ pref) {
    ++w;
    while (w < last && w >= mend) {
      ++m;
      mstart = mend;
      mend = __ldg(pref + m + 1);
    }
  }
};

// ---- order-preserving encodings of doubles for atomicMax / atomicMin --------------------------
__device__ __forceinline__ unsigned long long ord_enc(double x) {
  long long b = __double_as_longlong(x);
  return b < 0 ? ~(unsigned long long)b : ((unsigned long long)b | 0x8000000000000000ULL);
}
__device__ __forceinline__ double ord_dec(unsigned long long e) {
  return (e & 0x8000000000000000ULL) ? __longlong_as_double((long long)(e & 0x7FFFFFFFFFFFFFFFULL))
                                     : __longlong_as_double((long long)~e);
}

// the same decoding on the host (for reduction results copied back)
inline double ord_dec_host(unsigned long long e) {
  const unsigned long long b = (e & 0x8000000000000000ULL) ? (e & 0x7FFFFFFFFFFFFFFFULL) : ~e;
  double d;
  std::memcpy(&d, &b, sizeof(d));
  return d;
}

__device__ __forceinline__ bool gate_open(const Ctrl* c, int gate) {
  return gate < 0 || c->state == gate;
}

// In every kernel that launch_next may launch, before its first read of anything a kernel writes: wait
// until the kernels before it in the stream have completed and their writes are visible, then let the next
// one's CTAs take their places as this kernel's leave theirs.  Every thread of every CTA waits, also
// those with nothing to do, so that a kernel's completion implies that of all before it.
__device__ __forceinline__ void grid_begin() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// ---- asynchronous bulk copies global -> shared (sm_90+ cp.async.bulk, completed on an mbarrier) ---
// Used for element blocks, which are contiguous and 16-byte aligned.  The source is
// always this GPU's own memory; no multicast.
__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(unsigned long long* bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_addr(bar)), "r"(count) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
}
// one arrival that also announces `bytes` of copies completing on the barrier's current phase
__device__ __forceinline__ void mbar_arrive_expect_tx(unsigned long long* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.release.cta.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_addr(bar)), "r"(bytes)
               : "memory");
}
// `bytes` (a multiple of 16; both addresses 16-byte aligned) from global src to shared dst
__device__ __forceinline__ void bulk_copy_g2s(void* dst, const void* src, unsigned bytes, unsigned long long* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
                   smem_addr(dst)),
               "l"(src), "r"(bytes), "r"(smem_addr(bar))
               : "memory");
}
// orders this thread's earlier generic-proxy accesses of shared memory before later async-proxy ones
__device__ __forceinline__ void fence_proxy_async_smem() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }
__device__ __forceinline__ bool mbar_try_wait(unsigned long long* bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_addr(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Wait for the phase of `parity` to complete, at most `limit` polls (each poll may itself suspend
// the thread for a short time).  Returns false if the limit ran out.
__device__ __forceinline__ bool mbar_wait_bounded(unsigned long long* bar, unsigned parity, int limit = 1 << 22) {
  for (int i = 0; i < limit; ++i)
    if (mbar_try_wait(bar, parity)) return true;
  return false;
}

// ---- physics (MHD_PDE.f90 formulas as inlined in DG_solver.f90) -------------------------------

// Exactly rounded arithmetic for the residual's flux functions: every product, sum and fused
// multiply-add is written out, so the compiler has no freedom to contract or re-use products
// differently in different kernels, and every kernel that inlines these functions (single
// instance, re-try, batched, allocation-free) rounds them the same way.
__device__ __forceinline__ double dmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double dadd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double dsub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double dfma(double a, double b, double c) { return __fma_rn(a, b, c); }
// x, or the clamp c where x is smaller (larger) or NaN: the result of fmax (fmin) for a clamp that is
// not NaN, as one comparison and a select
__device__ __forceinline__ double at_least(double x, double c) { return x > c ? x : c; }
__device__ __forceinline__ double at_most(double x, double c) { return x < c ? x : c; }
// a*a + b*b + c*c, left to right with fused multiply-adds
__device__ __forceinline__ double dsq3(double a, double b, double c) { return dfma(c, c, dfma(b, b, dmul(a, a))); }
// a1*b1 + a2*b2 + a3*b3, likewise
__device__ __forceinline__ double ddot3(double a1, double b1, double a2, double b2, double a3, double b3) {
  return dfma(a3, b3, dfma(a2, b2, dmul(a1, b1)));
}

// 1/x for 2^-900 <= |x| <= 2^900: one step r + r(e + e^2), e = 1 - x r, of Householder's iteration of third
// order (the geometric series of 1/(1-e) to e^2), from the hardware's approximation r, |e| below 2^-19.9.
// The terms left out are below 2^-59: the error is at most 1.02 x 2^-53, relative.
// sqrt(x) for 2^-900 <= x <= 2^900: with y the hardware's approximation of 1/sqrt(x), to 2^-20, and h = x y,
// sqrt(x) = h (1 - 2t)^(-1/2), t = (1 - h y)/2, by the binomial series 1 + t + 3t^2/2 + ...  The terms left out are
// below 2^-58, half of h's rounding stays: the error is at most 1.55 x 2^-53.
// Zero, subnormal and infinite arguments give no finite value (mostly NaN), nor does the root of a negative
// number; arguments that may be zero carry TINY, whose root vanishes beside what it is added to.
// (tests/test_gpu_reciprocal_root.py.)  With 1.0 / x and sqrt(x) in their place the residual's error against extended
// precision is the same: geometric mean 3.5e-15 over 55 states, either way.
constexpr double TINY = 1.0e-280;
__device__ __forceinline__ double rcp_nr(double x) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  const double e = dfma(-x, r, 1.0);
  return dfma(r, dfma(e, e, e), r);
}
__device__ __forceinline__ double sqrt_nr(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double h = dmul(x, y), t = dfma(-h, dmul(0.5, y), 0.5);
  return dfma(dmul(h, t), dfma(1.5, t, 1.0), h);
}
// The same where an argument may lie outside: 1/0 and 1/inf as the division gives them (a subnormal number
// counts as zero), sqrt(0) = 0 and sqrt(inf) = inf.
__device__ __forceinline__ double rcp_any(double x) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  const double e = dfma(-x, r, 1.0), q = dfma(r, dfma(e, e, e), r);
  return q == q ? q : r;
}
__device__ __forceinline__ double sqrt_any(double x) {  // x >= 0
  const double s = sqrt_nr(x);
  return s == s ? s : x;
}

// _macro_prs_ (DG_solver.f90:125), its quotient as a product with rcp_nr
__device__ __forceinline__ double prs_of(double rho, double mx, double my, double mz, double bx,
                                         double by, double bz, double e, double gamma) {
  return (gamma - 1.0) * (e - 0.5 * ((mx * mx + my * my + mz * mz) * rcp_nr(rho) + (bx * bx + by * by + bz * bz)));
}
// _macro_ent_ (DG_solver.f90:126); igm1 = 1/(gamma-1)
__device__ __forceinline__ double ent_of(double rho, double prs, double gamma, double igm1) {
  return -(rho * (log(prs) - gamma * log(rho)) * igm1);
}

// Four times the entropy-conservative two-point flux along the first direction (ec_flux_x,
// DG_solver.f90:1570-1609; the y flux :1611-1650 is the same with the two directions exchanged).
// a, b = (rho, vn, vt, vz, bn, bt, bz, beta); a_bsq, b_bsq = |B|^2 of each.
//
// The reference forms rho_hat = rho_bar / ff(rho) and beta_hat = beta_bar / ff(beta) with
// ff = log_avg_divisor (zeta = a/b, f = (zeta-1)/(zeta+1), the series when f^2 < 1.4e-4, else
// 0.5 log(zeta)/f).  Here everything is formed from the sums S = a + b instead of the means, the
// factors 1/2 and 1/4 of the means going into the caller's coefficient (hence four times the flux):
//   f = (a-b)/(a+b)                                  (= (zeta-1)/(zeta+1))
//   series:  rho_hat = rho_bar / (1 + u/3 + u^2/5 + u^3/7),  u = f^2, formed as rho_bar times the
//            inverse series (inv_series_divisor)
//   log:     rho_hat = rho_bar / (0.5 log(zeta)/f) with f = (zeta-1)/(zeta+1) of the rounded zeta: with
//            f from a - b instead, the rounding of zeta would come back 1/|log zeta| times larger
//   igm1 = 1/(gamma-1) from the caller.
// The energy flux is the reference's sum with its exactly cancelling parts taken out: with
// f_m = v_bar f_0 - bn_bar B_bar + n p_tot, v_bar.f_m = f_0 |v_bar|^2 - bn_bar (v_bar.B_bar) +
// vn_bar p_tot, whose second part cancels the last term (v_bar.B_bar) bn_bar, and vn_bar p_tot -
// vn_bar b_sq_bar / 2 = vn_bar rho_bar / (2 beta_bar); |v_bar|^2 - v_sq_bar / 2 = va.vb / 2.  So
//   f_7 = f_0 (ff(beta)/((gamma-1) beta_bar) + va.vb)/2 + vn_bar rho_bar/(2 beta_bar) + B_bar.f_B.
// pref4 = 4 p_ref, a constant pressure left out of the normal momentum flux (f[1] / 4 = f_1 - p_ref):
// it drops out of a line's flux differences, and with it goes their largest rounding error.
// 65 FP64 operations and a reciprocal against 107 for the expressions as the reference writes them
// (the kernel that calls this is bound by its FP64 chains).
__device__ __forceinline__ double series_divisor(double u) {
  return dfma(u, dfma(u, dfma(u, 1.0 / 7.0, 1.0 / 5.0), 1.0 / 3.0), 1.0);
}
// half of 1 / series_divisor(u) by its own series, 1 - u/3 - 4u^2/45 - 44u^3/945 + 1147u^4/14175 (the
// inverse of the power series; the truncation error is below 3e-22 relative for u < 1.4e-4),
// so that the logarithmic mean of the common smooth case takes no division
__device__ __forceinline__ double half_inv_series_divisor(double u) {
  return dfma(u, dfma(u, dfma(u, dfma(u, 1147.0 / 28350.0, -22.0 / 945.0), -2.0 / 45.0), -1.0 / 6.0), 0.5);
}

__device__ __forceinline__ void ec_flux4(const double* a, const double* b, double a_bsq, double b_bsq, double igm1,
                                         double pref4, double* f) {
  const double rho_s = dadd(a[0], b[0]), beta_s = dadd(a[7], b[7]);
  const double rho_d = dsub(a[0], b[0]), beta_d = dsub(a[7], b[7]);
  const double ib = rcp_nr(beta_s);
  const double fr = dmul(rho_d, rcp_nr(rho_s)), ur = dmul(fr, fr);
  const double fb = dmul(beta_d, ib), ub = dmul(fb, fb);
  // logarithmic mean of rho and divisor of that of beta: the series forms, replaced by the
  // logarithmic forms in the uncommon case
  double rho_hat = dmul(rho_s, half_inv_series_divisor(ur));
  double ffb = series_divisor(ub);
  if (ur >= 1.4e-4 || ub >= 1.4e-4) {
    if (ur >= 1.4e-4) {
      const double z = dmul(a[0], rcp_nr(b[0]));
      rho_hat = dmul(dmul(rho_s, dsub(z, 1.0)), rcp_nr(dmul(dadd(z, 1.0), log(z))));
    }
    if (ub >= 1.4e-4) {
      const double z = dmul(a[7], rcp_nr(b[7]));
      ffb = dmul(dmul(0.5, log(z)), dmul(dadd(z, 1.0), rcp_nr(dsub(z, 1.0))));
    }
  }
  const double vn = dadd(a[1], b[1]), vt = dadd(a[2], b[2]), vz = dadd(a[3], b[3]);
  const double bn = dadd(a[4], b[4]), bt = dadd(a[5], b[5]), bz = dadd(a[6], b[6]);
  const double h = dmul(rho_hat, vn);  // 2 f_0
  // rho_bar / beta_bar (twice the pressure of equal states) with one correction step, so that equal
  // states give their pressure to the last bit and pref4 takes it out
  const double q0 = dmul(rho_s, ib), q = dfma(ib, dfma(-q0, beta_s, rho_s), q0);
  const double i2 = dadd(ib, ib);      // 1 / beta_bar
  const double p4 = dadd(dadd(a_bsq, b_bsq), dfma(2.0, q, -pref4));  // 4 (p_tot - p_ref)
  f[0] = dadd(h, h);
  f[1] = dfma(vn, h, dfma(-bn, bn, p4));
  f[2] = dfma(vt, h, -dmul(bn, bt));
  f[3] = dfma(vz, h, -dmul(bn, bz));
  f[4] = 0.0;
  const double gn = dfma(b[7], b[1], dmul(a[7], a[1]));
  const double gt = dfma(b[7], b[2], dmul(a[7], a[2]));
  const double gz = dfma(b[7], b[3], dmul(a[7], a[3]));
  f[5] = dmul(dfma(gn, bt, -dmul(gt, bn)), i2);
  f[6] = dmul(dfma(gn, bz, -dmul(gz, bn)), i2);
  const double x = dfma(dmul(ffb, i2), igm1, ddot3(a[1], b[1], a[2], b[2], a[3], b[3]));
  f[7] = dfma(0.5, dfma(bz, f[6], dmul(bt, f[5])), dfma(vn, q, dmul(h, x)));
}

// The gas pressure, clamped (DG_solver.f90:779,951-954), from m.v, |B|^2 and the total energy: one
// expression for nodes and interface states, so that the reference pressure cancels to the last bit.
__device__ __forceinline__ double gas_pressure(double gm1, double mv, double bsq, double e) {
  return at_least(dmul(gm1, dfma(-0.5, dadd(mv, bsq), e)), PP_EPS);
}

// ESPP_HLL_flux_x (DG_solver.f90:894-1071).  wl, wr: conserved states already rotated into the
// face normal frame (swap_xy for y faces).  out[0..7] = numerical flux, out[8] = nBn,
// out[9] = sl, out[10] = sr, out[11] = the smaller of the two pressures, which is left out of the
// normal momentum flux (the flux is out[1] + out[11]): the elements subtract their reference
// pressure from it before it meets the rest of the flux (see ec_flux4).  igm1 = 1/(gamma-1).
// Quotients are formed as products with reciprocals (rcp_nr); the values agree with the reference's
// expression order to a few ulp.
//
// The entropy s = log p - gamma log rho enters only through its jump ds = s_r - s_l: with the entropy
// flux q = -m s/(gamma-1) (m the normal momentum) and the first entropy variable
// v_0 = (gamma - s)/(gamma-1) - k (k = the kinetic energy over p),
//   q_r - q_l - v_0l (m_r - m_l) = -(m_r ds + gamma (m_r - m_l))/(gamma-1) + k_l (m_r - m_l),
// likewise with v_0r and m_l ds, and v_0r - v_0l = -ds/(gamma-1) - (k_r - k_l).  So two logarithms
// of ratios replace four, with the series log z = 2f (1 + u/3 + u^2/5 + ...), f = (z-1)/(z+1), u = f^2,
// where both ratios are close to one (u < 1.4e-4, as in the two-point flux; truncation 5e-17
// relative).  The sums over the entropy variables are taken as scalar products of the momentum and
// field jumps.  Against four logarithms and component-by-component sums: 253 x 261 p = 3 residual
// 105.2 -> 94.2 us, 301 x 199 p = 1 step 256 -> 242 us.
__device__ __forceinline__ void espp_hll(const double* wl, const double* wr, double gamma, double igm1, double* out) {
  const double gm1 = dsub(gamma, 1.0);
  double ir[2], v[2][3], mv[2], bsq[2], prs[2], ip[2], ith[2], bu[2], cf[2], f[2][8];
#pragma unroll
  for (int h = 0; h < 2; ++h) {  // the two sides
    const double* w = h ? wr : wl;
    ir[h] = rcp_nr(w[0]);
#pragma unroll
    for (int q = 0; q < 3; ++q) v[h][q] = dmul(ir[h], w[1 + q]);
    mv[h] = ddot3(w[1], v[h][0], w[2], v[h][1], w[3], v[h][2]);
    bsq[h] = dsq3(w[4], w[5], w[6]);
    prs[h] = gas_pressure(gm1, mv[h], bsq[h], w[7]);
    ip[h] = rcp_nr(prs[h]);
    ith[h] = dmul(w[0], ip[h]);
    bu[h] = ddot3(w[4], v[h][0], w[5], v[h][1], w[6], v[h][2]);
    const double bn2 = dmul(w[4], w[4]);
    const double cs = dmul(dmul(gamma, prs[h]), ir[h]), ss = dfma(bsq[h], ir[h], cs);
    const double disc = at_least(dfma(ss, ss, -dmul(dmul(dmul(4.0, cs), ir[h]), bn2)), TINY);
    cf[h] = sqrt_nr(dmul(0.5, dadd(ss, sqrt_nr(disc))));
    f[h][0] = w[1];
    f[h][2] = dfma(v[h][0], w[2], -dmul(w[5], w[4]));
    f[h][3] = dfma(v[h][0], w[3], -dmul(w[6], w[4]));
    f[h][4] = 0.0;
    f[h][5] = dfma(w[5], v[h][0], -dmul(w[4], v[h][1]));
    f[h][6] = dfma(w[6], v[h][0], -dmul(w[4], v[h][2]));
    f[h][7] = dfma(v[h][0], dadd(w[7], dfma(0.5, bsq[h], prs[h])), -dmul(w[4], bu[h]));
  }
  const double pb = at_most(prs[0], prs[1]);
#pragma unroll
  for (int h = 0; h < 2; ++h) {  // rounded as ec_flux4 rounds its p_tot - B_n^2, so that the two cancel where the field is constant
    const double* w = h ? wr : wl;
    f[h][1] = dfma(v[h][0], w[1], dfma(-w[4], w[4], dfma(0.5, bsq[h], dsub(prs[h], pb))));
  }
  const double rho_s = dadd(wl[0], wr[0]);
  double ds;
  {
    const double fp = dmul(dsub(prs[1], prs[0]), rcp_nr(dadd(prs[0], prs[1]))), up = dmul(fp, fp);
    const double fd = dmul(dsub(wr[0], wl[0]), rcp_nr(rho_s)), ud = dmul(fd, fd);
    double lp = dmul(dadd(fp, fp), series_divisor(up)), ld = dmul(dadd(fd, fd), series_divisor(ud));
    if (up >= 1.4e-4 || ud >= 1.4e-4) {
      if (up >= 1.4e-4) lp = log(dmul(prs[1], ip[0]));
      if (ud >= 1.4e-4) ld = log(dmul(wr[0], ir[0]));
    }
    ds = dmul(dfma(-gamma, ld, lp), igm1);  // (s_r - s_l)/(gamma-1)
  }
  double j[8], d[8];
#pragma unroll
  for (int s = 0; s < 8; ++s) {
    j[s] = dsub(wr[s], wl[s]);
    if (s != 4) d[s] = dsub(f[1][s], f[0][s]);
  }
  d[4] = 0.0;
  // Roe's weights with one root, s = sqrt(rho_l rho_r): both quotients over (sqrt rho_l + sqrt rho_r)^2.
  // A density that is not positive makes them NaN, with them the speeds and so the whole flux, as the
  // logarithms and roots of each density do in the reference (the product of two negative ones is positive:
  // it takes the left one's sign).
  const double rho_p = dmul(wl[0], wr[0]);
  const int sign_l = __double2hiint(wl[0]) & (int)0x80000000;
  const double s_rho = sqrt_nr(__hiloint2double(__double2hiint(rho_p) | sign_l, __double2loint(rho_p)));
  const double irs = rcp_nr(dfma(2.0, s_rho, rho_s));
  const double vx_roe = dmul(dfma(s_rho, dadd(v[0][0], v[1][0]), dadd(wl[1], wr[1])), irs);
  const double db = sqrt_nr(dfma(dsq3(j[4], j[5], j[6]), irs, TINY));
  const double sl_pp = dsub(dsub(at_most(vx_roe, v[0][0]), cf[0]), db);
  const double sr_pp = dadd(dadd(at_least(vx_roe, v[1][0]), cf[1]), db);
  // a = sum (v_r - v_l)(w_r - w_l); b = q_r - q_l - sum v (f_r - f_l) - phi (B_r - B_l)_n per side
  const double gg = dmul(gamma, igm1);
  double k[2], b[2], mj[2], bj[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const double* w = h ? wr : wl;
    k[h] = dmul(dmul(0.5, mv[h]), ip[h]);
    mj[h] = dmul(ip[h], ddot3(w[1], j[1], w[2], j[2], w[3], j[3]));
    bj[h] = dmul(ith[h], ddot3(w[4], j[4], w[5], j[5], w[6], j[6]));
    const double md = dmul(ip[h], ddot3(w[1], d[1], w[2], d[2], w[3], d[3]));
    const double vd = dfma(ith[h], dfma(w[6], d[6], dfma(w[5], d[5], -d[7])), md);
    b[h] = -dfma(dmul(ith[h], bu[h]), j[4], dfma(dsub(gg, k[h]), d[0], dfma(h ? wl[1] : wr[1], ds, vd)));
  }
  const double da = dadd(dfma(dsub(ith[0], ith[1]), j[7], -dmul(dadd(ds, dsub(k[1], k[0])), j[0])),
                         dadd(dsub(mj[1], mj[0]), dsub(bj[1], bj[0])));
  const double ia = rcp_nr(dadd(at_least(da, 0.0), 1e-8));
  const double al = at_least(dmul(b[0], ia), 0.0);
  const double ar = at_least(dmul(b[1], ia), 0.0);
  const double aa = sqrt_nr(dfma(al, ar, TINY));
  const double sl = at_most(-dadd(ar, aa), sl_pp);  // (never above zero: ar, aa >= 0; NaN where sl_pp is)
  const double sr = at_least(dadd(al, aa), sr_pp);
  const double idsl = rcp_nr(dsub(sr, sl));
  // (sr fl - sl fr)/(sr - sl) from the side with the larger weight, plus the other weight (at most
  // 1/2) times the difference: equal states give exactly their flux, a supersonic face its upwind one
  const bool left = sr >= -sl;
  const double w = dmul(left ? -sl : -sr, idsl), wd = dmul(dmul(sl, sr), idsl);
#pragma unroll
  for (int s = 0; s < 8; ++s) out[s] = dfma(wd, j[s], dfma(w, d[s], left ? f[0][s] : f[1][s]));
  out[8] = dfma(w, j[4], left ? wl[4] : wr[4]);
  out[9] = sl;
  out[10] = sr;
  out[11] = pb;
}

}  // namespace mhd
