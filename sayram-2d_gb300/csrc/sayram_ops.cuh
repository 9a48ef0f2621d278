// sayram_ops.cuh -- the kernels of one backward-Euler step (see sayram_kernels.cuh for layout).
//
//   k_setup      once per instance: coefficients -> per-cell face factors, UKK, loss diagonal
//   k_dtable     on demand: D fields interpolated from a D table -> the face factors again
//   k_begin      per step: resets the per-instance solver state
//   k_assemble   fused vertex interpolation + PPFV face fluxes + diagonal/RHS + Jacobi scaling
//   k_resid      outer residual r = R - A~ y (adds the last Krylov correction first)
//   k_bicg1/2    one BiCGSTAB iteration in T precision (FP64 or FP32) with fused SpMV + dots
//   k_after_*    the decisions after each of these passes, a block per instance
//   k_polish     positivity polish y' = R + (I - A~) y+, f = y'/D, min / clamp / mass checks
//                (these in sayram_solve.cuh)
//   k_team       all of a step but the set-up in one launch, for batches that fit the chip
//                (sayram_team.cuh)
//   k_field_*    alpha-major FP64 <-> padded system order transposes for the host-buffer step
//
// The assembly, residual, polish and state are written once over an arithmetic policy A:
//   F64A  IEEE binary64 (the FP64 drop-in and the FP32 + FP64-residual mode)
//   DWA   double-word pairs of FP32 (dword.cuh): FP64-class accuracy on the FP32 pipes
// Per-cell "wide" arrays (f, 1/D, R, column sums, y, the face factors, the weights and Dirichlet
// values) hold 8 bytes per entry in both: one double, or one (hi, lo) float pair.
#pragma once

#include "dword.cuh"
#include "sayram_kernels.cuh"

namespace sg {

// ------------------------------------------------------------------------------ arguments
struct Geo {  // per-cell face factors (time independent while the coefficients are)
  double *aAx, *aBx, *Sx, *aAy, *aBy, *Sy, *ukk, *sdiag;
  double* G;  // G per cell, FP64 (kept so that new D fields can re-derive the face factors)
  double* decay;  // 1 / (1 + dt/tau): one step of pure loss (extrapolated start); null: 1
};

struct Common {
  const InstDev* inst;
  InstState* st;
  Ctl* ctl;
  const int* chunk_inst;
  int nchunks;
  const int* tile_inst;
  int ntiles;
  int ninst;
  const double* wx;    // per vertex column: (wL, wR) bilinear weights (Solver.cc:333-336)
  const double* wy;    // per vertex row: (wB, wT)
  const double* dirv;  // Dirichlet vertex values
  double* part;        // kPartQ segment sums of 8 bytes per reduction segment, quantity by quantity
  long long pstride;   // segments per quantity
  // when set, [nchunks, ntiles, ninst] are read from device memory (lists that change between
  // steps, as in the server) instead of the by-value counts above
  const int* dyn;
  int pmax;  // largest row pitch of any instance (shared-memory halo of the SpMV kernels)
  // device-side loops of the per-step CUDA graph (use_cond = 0: the host drives the loops; 1: the
  // graph's WHILE nodes)
  unsigned long long h_outer, h_inner;  // cudaGraphConditionalHandle of the two WHILE nodes
  int use_cond;
  int guard_refine, guard_iters;  // hard caps on loop trips, whatever the bookkeeping says
  int hist_cap;  // history depth used for the starting point (kHist; 1 when the buffers alias)
  int precond;   // 1: the inner Krylov solve is preconditioned on the left by the alpha-line blocks
};

__device__ __forceinline__ int n_chunks(const Common& cm) { return cm.dyn ? cm.dyn[0] : cm.nchunks; }
__device__ __forceinline__ int n_tiles(const Common& cm) { return cm.dyn ? cm.dyn[1] : cm.ntiles; }
__device__ __forceinline__ int n_inst(const Common& cm) { return cm.dyn ? cm.dyn[2] : cm.ninst; }

// The last block of a deciding kernel (k_after_resid, k_after_t) sets the graph's WHILE conditions from the number of
// instances still active. The trip counters make both loops terminate after guard_refine
// residual evaluations and guard_iters Krylov iterations even if the counts were inconsistent.
// which = 0: after the residual (decides both loops); which = 1: after a Krylov iteration.
__device__ __forceinline__ void loop_epilogue(const Common& cm, int which) {
  if (!cm.use_cond) return;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    const unsigned prev = atomicAdd(&cm.ctl->kdone[which], 1u);
    if (prev == gridDim.x - 1) {
      __threadfence();
      const int nout = atomicAdd(&cm.ctl->n_outer, 0);
      const int nin = atomicAdd(&cm.ctl->n_inner, 0);
      unsigned go_o = 0u, go_i;
      if (which == 0) {
        const unsigned lo = atomicAdd(&cm.ctl->outer_loops, 1u) + 1u;
        atomicExch(&cm.ctl->inner_loops, 0u);
        go_o = (nout > 0 && lo < (unsigned)cm.guard_refine) ? 1u : 0u;
        go_i = (nin > 0 && lo < (unsigned)cm.guard_refine) ? 1u : 0u;
      } else {
        const unsigned li = atomicAdd(&cm.ctl->inner_loops, 1u) + 1u;
        go_i = (nin > 0 && li < (unsigned)cm.guard_iters) ? 1u : 0u;
      }
      if (which == 0) cudaGraphSetConditional(cm.h_outer, go_o);
      cudaGraphSetConditional(cm.h_inner, go_i);
      atomicExch(&cm.ctl->kdone[which], 0u);
    }
  }
}

template <typename C>
struct Coef {  // row-oriented scaled off-diagonal magnitudes (hi parts when split)
  C *cw, *ce, *cs, *cn;
  float *lw, *le, *ls, *ln;  // low parts for the FP32-split storage (null for FP64)
};

constexpr int kOrder = 4;  // earlier states the extrapolated start of each solve goes back
constexpr int kHist = 3;   // history buffers: with f^n (the state the polish replaces) they hold kOrder

struct Fields {
  double* f;       // state, padded system order
  double* fh[kHist];  // earlier states f^(n-1) .. f^(n-3), rotated per instance (InstState::hslot)
  const double* decay;  // 1 / (1 + dt/tau) per cell (the extrapolated start); null: 1
  double* invD;    // 1 / diag(M)
  double* R;       // right-hand side
  double* colsum;  // 1^T M per column (conservation check)
  double* y64[2];  // scaled solution y = D f (ping-pong)
};

// Krylov vectors. The residual a solve starts from is left in rh (the shadow residual); r and p
// of the first iteration are that same array, so it writes neither.
template <typename T>
struct Kry {
  T *rh, *t, *x;
  T *r[2], *p[2], *v[2];  // iteration i uses [i & 1]
};
constexpr int kPartQ = 5;     // most sums any pass forms at once
constexpr int kPartSets = 2;  // sets of partial sums (k_team alternates; the per-pass kernels use the first)

// ------------------------------------------------------------------------------ arithmetic
struct F64A {
  using V = double;
  static constexpr int kAsmBlocks = 4;  // k_assemble: resident blocks (64 registers)
  template <typename Ix>
  __device__ static V ld(const double* p, Ix i) { return p[i]; }
  template <typename Ix>
  __device__ static void st(double* p, Ix i, V v) { p[i] = v; }
  __device__ static Q4<V> ld4(const double* p) { return sg::ld4(p); }
  __device__ static void st4(double* p, const Q4<V>& q) { sg::st4(p, q); }
  // every operation is fused or rounded explicitly, so that all kernels sharing a formula give the
  // same bits whatever the compiler would contract
  __device__ static V add(V a, V b) { return __dadd_rn(a, b); }
  __device__ static V sub(V a, V b) { return __dadd_rn(a, -b); }
  __device__ static V mul(V a, V b) { return __dmul_rn(a, b); }
  __device__ static V fma(V a, V b, V c) { return __fma_rn(a, b, c); }
  // a*x + b*y and a*x - b*y (the same expression trees as fma(a, x, mul(b, y)) and
  // sub(mul(a, x), mul(b, y)))
  __device__ static V dot2(V a, V x, V b, V y) { return __fma_rn(a, x, __dmul_rn(b, y)); }
  __device__ static V fma0(V a, V b) { return __dmul_rn(a, b); }  // fma(a, b, 0)
  __device__ static V dot2s(V a, V x, V b, V y) { return __fma_rn(a, x, -__dmul_rn(b, y)); }
  // sums whose terms all have the same sign (cheaper in double-word form)
  __device__ static V addp(V a, V b) { return __dadd_rn(a, b); }
  __device__ static V fmap(V a, V b, V c) { return __fma_rn(a, b, c); }
  __device__ static V addf(V a, float b) { return __dadd_rn(a, (double)b); }
  __device__ static V rcp(V a) { return rcp64(a); }
  __device__ static V div(V a, V b) { return div64(a, b); }
  __device__ static V abs(V a) { return fabs(a); }
  __device__ static V neg(V a) { return -a; }
  // g, the polynomial extrapolation in time through f and n earlier states h1..h4 (n = 1..4) of
  // the loss-compensated sequence c_k = h_k r^k (r = 1/(1 + dt/tau), one step of pure loss), times
  // r: g = r (c0 + d1), r (c0 + 2 d1 - d2), r (c0 + 3 (d1 - d2) + d3),
  // r (c0 + 4 (d1 + d3) - 6 d2 - d4) with d_m = c_(m-1) - c_m, c0 = f. Exact for pure loss;
  // r = 1 gives the plain polynomial. The next solve starts from y0 = D g.
  __device__ static V extrap(V f, V h1, V h2, V h3, V h4, int n, V r) {
    // the closed forms 2 c0 - c1, 3 (c0 - c1) + c2, 4 (c0 + c2) - 6 c1 - c3 and
    // 5 (c0 - c3) - 10 (c1 - c2) + c4, by Horner in r: at most 9 FP64 operations
    double a;
    if (n >= 4)
      a = __fma_rn(r, __fma_rn(r, __fma_rn(r, __fma_rn(r, h4, __dmul_rn(-5.0, h3)), __dmul_rn(10.0, h2)),
                               __dmul_rn(-10.0, h1)), __dmul_rn(5.0, f));
    else if (n == 3)
      a = __fma_rn(r, __fma_rn(r, __fma_rn(-r, h3, __dmul_rn(4.0, h2)), __dmul_rn(-6.0, h1)), __dmul_rn(4.0, f));
    else if (n == 2)
      a = __fma_rn(r, __fma_rn(r, h2, __dmul_rn(-3.0, h1)), __dmul_rn(3.0, f));
    else
      a = __fma_rn(-r, h1, __dadd_rn(f, f));
    return __dmul_rn(r, a);
  }
  __device__ static V rsub1(V a) { return 1.0 - a; }
  __device__ static V max0(V a) { return fmax(a, 0.0); }
  __device__ static V k(double c) { return c; }
  __device__ static bool lt0(V a) { return a < 0.0; }
  // sign tests on the bits: a comparison is one more operation on the FP64 pipe
  __device__ static bool gt0(V a) { return __double_as_longlong(a) > 0; }
  __device__ static V pos_part(V a) { return __double_as_longlong(a) > 0 ? a : 0.0; }
  __device__ static float f32(V a) { return (float)a; }
  __device__ static float sq32(V a) { return (float)(a * a); }
  __device__ static double to_d(V a) { return a; }
  __device__ static V from_d(double a) { return a; }
  // the conversions of the layout transforms (none here)
  __device__ static double to_d_io(V a) { return a; }
  __device__ static V from_d_io(double a) { return a; }
  __device__ static void split(V a, float& hi, float& lo) {
    hi = __double2float_rn(a);
    lo = __double2float_rn(a - (double)hi);
  }
  // a pair of split(), joined in integers: as two conversions and an FP64 addition the four coefficients
  // of a cell took 160 of the mixed-mode residual's 490 cycles per SM and warp of cells (192 uneven
  // instances, 4 steps with Jacobi scaling: residuals 2.98 -> 2.38 ms, polish 1.21 -> 0.98 ms)
  __device__ static V hilo(float hi, float lo) { return dw_join_int(dw{hi, lo}); }
  // r * s for a power-of-two s, in the Krylov precision T
  template <typename T>
  __device__ static T scaled(V a, float s) { return (T)__dmul_rn(a, (double)s); }
  // y + x*s for the FP32/FP64 Krylov correction x in scaled units
  template <typename T>
  __device__ static V add_scaled(V y, T x, float s) { return __fma_rn((double)x, (double)s, y); }
  using Acc = double;  // per-thread accumulator of scaled squares
  __device__ static Acc sq_scaled(V a, float s, Acc q) {
    const double t = __dmul_rn(a, (double)s);
    return __fma_rn(t, t, q);
  }
  using R = double;  // what the residual's sums are carried in
};

struct DWA {
  using V = dw;
  // k_assemble: 6 resident blocks (40 registers, no spill); measured on the 4096-instance batch
  // with 64 launched blocks per SM: 4 blocks 5.72 ms, 5 blocks (48 registers) 5.27 ms, 6 blocks
  // 5.16 ms per launch (with 96 launched per SM: 5.09 ms)
  static constexpr int kAsmBlocks = 6;
  template <typename Ix>
  __device__ static V ld(const double* p, Ix i) {
    const float2 q = reinterpret_cast<const float2*>(p)[i];
    return dw{q.x, q.y};
  }
  template <typename Ix>
  __device__ static void st(double* p, Ix i, V v) { reinterpret_cast<float2*>(p)[i] = make_float2(v.hi, v.lo); }
  __device__ static Q4<V> ld4(const double* p) {
    const float4 a = reinterpret_cast<const float4*>(p)[0];
    const float4 b = reinterpret_cast<const float4*>(p)[1];
    return Q4<V>{{dw{a.x, a.y}, dw{a.z, a.w}, dw{b.x, b.y}, dw{b.z, b.w}}};
  }
  __device__ static void st4(double* p, const Q4<V>& q) {
    reinterpret_cast<float4*>(p)[0] = make_float4(q.a[0].hi, q.a[0].lo, q.a[1].hi, q.a[1].lo);
    reinterpret_cast<float4*>(p)[1] = make_float4(q.a[2].hi, q.a[2].lo, q.a[3].hi, q.a[3].lo);
  }
  // Sums and multiply-adds are accurate to a few u^2 of their operands' magnitudes (SloppyDWPlusDW,
  // dw_fma), which is the accuracy every use needs: matrix entries against their forward-error
  // scale, residuals against |R|, increments against |f|.
  __device__ static V add(V a, V b) { return dw_add_same(a, b); }
  __device__ static V sub(V a, V b) { return dw_add_same(a, dw_neg(b)); }
  __device__ static V mul(V a, V b) { return dw_mul(a, b); }
  __device__ static V fma(V a, V b, V c) { return dw_fma(a, b, c); }
  __device__ static V dot2(V a, V x, V b, V y) { return dw_dot2(a, x, b, y); }
  __device__ static V fma0(V a, V b) { return dw_fma0(a, b); }  // fma(a, b, 0)
  __device__ static V dot2s(V a, V x, V b, V y) { return dw_dot2(a, x, dw_neg(b), y); }
  __device__ static V addp(V a, V b) { return dw_add_same(a, b); }
  __device__ static V fmap(V a, V b, V c) { return dw_fma(a, b, c); }
  __device__ static V addf(V a, float b) { return dw_add_f(a, b); }
  __device__ static V rcp(V a) { return dw_rcp(a); }
  __device__ static V div(V a, V b) { return dw_div(a, b); }
  __device__ static V abs(V a) { return dw_abs(a); }
  __device__ static V neg(V a) { return dw_neg(a); }
  // as F64A::extrap, in double-word: with loss rates up to 10 per day an increment is ~10 % of f, so
  // FP32 increments would leave ~1e-8 of f in the start, above what the extrapolation achieves. (The
  // closed forms leave up to 31 u^2 ~ 1e-13 of f, a hundredth of the residual target; the starting
  // point only steers the iteration, the converged answer does not depend on it.)
  __device__ static V extrap(V f, V h1, V h2, V h3, V h4, int n, V r) {
    dw a;
    if (n >= 4)
      a = dw_fma(r, dw_fma(r, dw_fma(r, dw_fma(r, h4, dw_mul_f(h3, -5.0f)), dw_mul_f(h2, 10.0f)),
                           dw_mul_f(h1, -10.0f)), dw_mul_f(f, 5.0f));
    else if (n == 3)
      a = dw_fma(r, dw_fma(r, dw_fma(dw_neg(r), h3, times4(h2)), dw_mul_f(h1, -6.0f)), times4(f));
    else if (n == 2)
      a = dw_fma(r, dw_fma(r, h2, dw_mul_f(h1, -3.0f)), dw_mul_f(f, 3.0f));
    else
      a = dw_fma(dw_neg(r), h1, dw{2.0f * f.hi, 2.0f * f.lo});
    return dw_mul(r, a);
  }
  __device__ static V times4(V a) { return dw{4.0f * a.hi, 4.0f * a.lo}; }
  __device__ static V rsub1(V a) { return dw_add_f(dw_neg(a), 1.0f); }  // 1 - a (DWPlusFP)
  __device__ static V max0(V a) { return dw_max0(a); }
  __device__ static V k(double c) { return dw_from_double(c); }
  __device__ static bool lt0(V a) { return a.hi < 0.0f; }
  __device__ static bool gt0(V a) { return a.hi > 0.0f; }
  __device__ static V pos_part(V a) { return dw_max0(a); }
  __device__ static float f32(V a) { return a.hi; }
  __device__ static float sq32(V a) { return a.hi * a.hi; }
  __device__ static double to_d(V a) { return dw_to_double(a); }
  __device__ static V from_d(double a) { return dw_from_double(a); }
  // the same bits with integer rounding (the layout transforms convert every cell per call)
  __device__ static double to_d_io(V a) { return dw_to_double_int(a); }
  __device__ static V from_d_io(double a) { return dw_from_double_int(a); }
  __device__ static void split(V a, float& hi, float& lo) {
    hi = a.hi;
    lo = a.lo;
  }
  __device__ static V hilo(float hi, float lo) { return dw{hi, lo}; }
  template <typename T>
  __device__ static T scaled(V a, float s) { return (T)__fmul_rn(a.hi, s); }
  template <typename T>
  __device__ static V add_scaled(V y, T x, float s) { return dw_add_f(y, __fmul_rn((float)x, s)); }
  using Acc = float;
  __device__ static Acc sq_scaled(V a, float s, Acc q) {
    const float t = __fmul_rn(a.hi, s);
    return __fmaf_rn(t, t, q);
  }
  using R = dw;
};

// Power-of-two scale of an instance's refinement system: 2^-e with max|R| = m * 2^e, m in
// [0.5, 1). Residuals are handed to the Krylov solver as r * scale, so its vectors and dot
// products stay O(1) or below whatever the magnitude of f (no FP32 underflow).
__device__ __forceinline__ float rhs_scale(unsigned int rmax_bits) {
  const float m = __uint_as_float(rmax_bits);
  if (!(m > 0.0f) || !isfinite(m)) return 1.0f;
  int e;
  frexpf(m, &e);
  return ldexpf(1.0f, -e);
}

// ------------------------------------------------------------------------------ setup
// Face factors of cell (i,j) from the reference's general formula (Solver.cc:68-97) evaluated on
// the XNEG and YNEG edges (Mesh.cc:80-151); the XPOS/YPOS edges of a rectangular cell give the
// same pair. Uses non-contracting intrinsics so the values match the CPU evaluation.
__device__ __forceinline__ void face_pair(double Kx, double Ky, double Ax, double Ay, double Bx,
                                          double By, double n0, double n1, const double L[4],
                                          double* aa, double* ab) {
  const double ex = __dadd_rn(Bx, -Ax), ey = __dadd_rn(By, -Ay);
  const double length = __dsqrt_rn(__dadd_rn(__dmul_rn(ex, ex), __dmul_rn(ey, ey)));
  const double vkb0 = __dadd_rn(Bx, -Kx), vkb1 = __dadd_rn(By, -Ky);
  const double vka0 = __dadd_rn(Ax, -Kx), vka1 = __dadd_rn(Ay, -Ky);
  const double rvkb0 = vkb1, rvkb1 = -vkb0, rvka0 = vka1, rvka1 = -vka0;
  const double t0 = __dadd_rn(__dmul_rn(n0, L[0]), __dmul_rn(n1, L[2]));
  const double t1 = __dadd_rn(__dmul_rn(n0, L[1]), __dmul_rn(n1, L[3]));
  *aa = __ddiv_rn(__dmul_rn(length, __dadd_rn(__dmul_rn(t0, rvkb0), __dmul_rn(t1, rvkb1))),
                  __dadd_rn(__dmul_rn(vka0, rvkb0), __dmul_rn(vka1, rvkb1)));
  *ab = __ddiv_rn(__dmul_rn(length, __dadd_rn(__dmul_rn(t0, rvka0), __dmul_rn(t1, rvka1))),
                  __dadd_rn(__dmul_rn(vkb0, rvka0), __dmul_rn(vkb1, rvka1)));
}

// Face factors of cell K from G and D (Solver::update_Lambda, Solver.cc:57-65, then the general
// a_sigma formula on the XNEG and YNEG edges), stored in the policy's wide format.
template <typename A>
__device__ __forceinline__ void setup_faces(const Geo& geo, long long K, double xl, double xr, double yb,
                                            double yt, double g, double dxx, double dxy, double dyy) {
  const double Kx = __dmul_rn(0.5, __dadd_rn(xl, xr)), Ky = __dmul_rn(0.5, __dadd_rn(yb, yt));
  const double L[4] = {__dmul_rn(dxx, g), __dmul_rn(dxy, g), __dmul_rn(dxy, g), __dmul_rn(dyy, g)};
  double aa, ab;
  face_pair(Kx, Ky, xl, yt, xl, yb, -1.0, 0.0, L, &aa, &ab);  // XNEG: A=(i,j+1) B=(i,j)
  A::st(geo.aAx, K, A::from_d(aa));
  A::st(geo.aBx, K, A::from_d(ab));
  A::st(geo.Sx, K, A::from_d(__dadd_rn(aa, ab)));
  face_pair(Kx, Ky, xl, yb, xr, yb, 0.0, -1.0, L, &aa, &ab);  // YNEG: A=(i,j) B=(i+1,j)
  A::st(geo.aAy, K, A::from_d(aa));
  A::st(geo.aBy, K, A::from_d(ab));
  A::st(geo.Sy, K, A::from_d(__dadd_rn(aa, ab)));
}

// Every time-independent per-cell value of cell K from its edges, dt, G, D and 1/tau: the face
// factors (setup_faces), G (when kept), UKK = G * (dx*dy/dt), the diagonal term UKK*(1 + dt/tau)
// (Solver.cc:190-199, Mesh.h:61-63) and the one-step loss factor 1/(1 + dt/tau) (when kept). The
// one definition k_setup and the allocation-free entry point's set-up both call.
template <typename A>
__device__ __forceinline__ void setup_cell(const Geo& geo, long long K, double xl, double xr, double yb,
                                           double yt, double dt, double g, double dxx, double dxy, double dyy,
                                           double itau) {
  const double dx = __dadd_rn(xr, -xl), dy = __dadd_rn(yt, -yb);
  setup_faces<A>(geo, K, xl, xr, yb, yt, g, dxx, dxy, dyy);
  if (geo.G) geo.G[K] = g;
  const double ukk = __dmul_rn(g, __ddiv_rn(__dmul_rn(dx, dy), dt));
  A::st(geo.ukk, K, A::from_d(ukk));
  const double lossd = __dadd_rn(1.0, __dmul_rn(dt, itau));
  A::st(geo.sdiag, K, A::from_d(__dmul_rn(ukk, lossd)));
  if (geo.decay) A::st(geo.decay, K, A::from_d(__ddiv_rn(1.0, lossd)));
}

// One instance: stage holds alpha-major G, Dxx, Dxy, Dyy, inv_tau, f0 (each nx*ny). mask bits
// 0-4 select the coefficient sections (all five together), bit 5 the initial state. Values are
// computed in FP64 and stored in the policy's wide format.
template <typename A>
__global__ void k_setup(Common cm, Geo geo, double* f, const double* stage, const double* xe,
                        const double* ye, int b, int mask) {
  const InstDev I = cm.inst[b];
  const long long ncell = (long long)I.nx * I.ny;
  const double* G = stage;
  const double* Dxx = stage + ncell;
  const double* Dxy = stage + 2 * ncell;
  const double* Dyy = stage + 3 * ncell;
  const double* itau = stage + 4 * ncell;
  const double* f0 = stage + 5 * ncell;
  for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < ncell;
       c += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(c / I.ny), j = (int)(c % I.ny);
    const long long K = I.base + (long long)j * I.pitch + i;
    if (mask & 31)
      setup_cell<A>(geo, K, xe[I.xe + i], xe[I.xe + i + 1], ye[I.ye + j], ye[I.ye + j + 1], I.dt, G[c], Dxx[c],
                    Dxy[c], Dyy[c], itau[c]);
    if (mask & 32) A::st(f, K, A::from_d(f0[c]));
  }
}

// A diffusion-coefficient table on the device and the host-side values it is read with (see
// k_dtable). Row factors are per E row of each instance, at the instance's y-edge offset.
struct DTab {
  int na, ne;
  double xmin, xmax;      // alpha0 of the first and last node (radians)
  double lymin, lymax;    // log E of the first and last node
  double denorm;          // gME^2 gC^2
  const double *Daa, *Dap, *Dpp;        // (na, ne) row-major
  const double *rp, *rdl, *rdl2;        // per row: p, dlogE/dp, (dlogE/dp)^2
};

// calWeight (utils.h:44-58): weight of the lower node; past the last node, the last node with
// weight 1 (i = n-1, w = 0). Below the first node the reference converts a negative floor() to
// size_t (undefined in C++); its own i < 0 branch (first node, weight 1) is what is done here.
__device__ __forceinline__ void cal_weight(long long* i, double* w, long long n, double pos) {
  if (pos < 0.0) {
    *i = 0;
    *w = 1.0;
  } else if (*i < n) {
    *w = __dadd_rn(1.0, -__dadd_rn(pos, -(double)*i));
  } else {
    *i = n - 1;
    *w = 0.0;
  }
}

// D fields of Albert_Young(_LC)::constructD (Albert_Young.cc:112-134) at the cell centres, then
// the face factors of those cells. locate (Albert_Young.cc:94-110) places a centre in the table
// from its end points (uniform in alpha0 and log E); interp2D (utils.h:24-41) is bilinear. The
// transcendental row factors p = e2p(exp(log E)), dlogE/dp and its square (utils.h:12-20), the
// logs of the table's energy bounds and the unit factor come from the host's libm, so every
// operation here is a separately rounded IEEE add, multiply or divide in the reference's order.
// Tiles [t0, t1) of the tile list.
template <typename A>
__global__ void k_dtable(Common cm, Geo geo, DTab t, const double* xe, const double* ye, int t0, int t1) {
  const double s2d = 86400.0;  // 3600 * 24
  for (int tl = t0 + blockIdx.x; tl < t1; tl += gridDim.x) {
    const int b = cm.tile_inst[tl];
    const InstDev I = cm.inst[b];
    if (!I.enabled) continue;
    const int lt = tl - I.tile0, i0t = (lt % I.ntx) * kTX, j0t = (lt / I.ntx) * kTY;
    for (int q = threadIdx.x; q < kTX * kTY; q += blockDim.x) {
      const int i = i0t + (q % kTX), j = j0t + (q / kTX);
      if (i >= I.nx || j >= I.ny) continue;
      const long long K = I.base + (long long)j * I.pitch + i;
      const double xl = xe[I.xe + i], xr = xe[I.xe + i + 1];
      const double yb = ye[I.ye + j], yt = ye[I.ye + j + 1];
      const double alpha0 = __dmul_rn(0.5, __dadd_rn(xl, xr)), logE = __dmul_rn(0.5, __dadd_rn(yb, yt));
      const double px = __dmul_rn(__ddiv_rn(__dadd_rn(alpha0, -t.xmin), __dadd_rn(t.xmax, -t.xmin)), (double)(t.na - 1));
      const double py = __dmul_rn(__ddiv_rn(__dadd_rn(logE, -t.lymin), __dadd_rn(t.lymax, -t.lymin)), (double)(t.ne - 1));
      long long ia = px >= 0.0 ? (long long)floor(px) : 0, je = py >= 0.0 ? (long long)floor(py) : 0;
      double wi, wj;
      cal_weight(&ia, &wi, t.na - 1, px);
      cal_weight(&je, &wj, t.ne - 1, py);
      const double ui = __dadd_rn(1.0, -wi), uj = __dadd_rn(1.0, -wj);
      const long long r00 = ia * t.ne + je, r10 = r00 + t.ne;
      const double* raw[3] = {t.Daa, t.Dap, t.Dpp};
      double v[3];
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const double* r = raw[k];
        const double s1 = __dmul_rn(__dmul_rn(r[r00], wi), wj);
        const double s2 = __dmul_rn(__dmul_rn(r[r10], ui), wj);
        const double s3 = __dmul_rn(__dmul_rn(r[r10 + 1], ui), uj);
        const double s4 = __dmul_rn(__dmul_rn(r[r00 + 1], wi), uj);
        v[k] = __dadd_rn(__dadd_rn(__dadd_rn(s1, s2), s3), s4);
      }
      const double p = t.rp[I.ye + j], dl = t.rdl[I.ye + j], dl2 = t.rdl2[I.ye + j];
      const double dxx = __ddiv_rn(__dmul_rn(__dmul_rn(v[0], t.denorm), s2d), __dmul_rn(p, p));
      const double dxy = __ddiv_rn(__dmul_rn(__dmul_rn(__dmul_rn(v[1], t.denorm), s2d), dl), p);
      const double dyy = __dmul_rn(__dmul_rn(__dmul_rn(v[2], t.denorm), s2d), dl2);
      setup_faces<A>(geo, K, xl, xr, yb, yt, geo.G[K], dxx, dxy, dyy);
    }
  }
}

// alpha-major FP64 (packed at hoff) -> padded system order in the wide format, for tiles
// [t0, t1) of the tile list (t1 < 0: all), one 32x16 tile at a time: read along j (contiguous on the host side), transposed through shared memory,
// written along i (contiguous on the device side).
// When `restart` is set, a cell given back exactly the double it would be read out as keeps its
// stored value (in the double-word format that value can carry low bits a double does not), and
// an instance with any other cell loses its history of earlier states (the extrapolated start
// restarts from the new state). An instance given back its own state is left exactly as it was.
template <typename A>
__global__ void __launch_bounds__(kFieldThreads) k_field_in(Common cm, double* dst, const double* src, int restart,
                                                             int t0, int t1) {
  using V = typename A::V;
  count_launch(cm.ctl);
  constexpr int kItems = kTX * kTY / kFieldThreads;
  static_assert(kItems * kFieldThreads == kTX * kTY, "a tile splits evenly over the block");
  __shared__ double tile[kTY][kTX + 1];
  if (t1 < 0) t1 = n_tiles(cm);
  for (int t = t0 + blockIdx.x; t < t1; t += gridDim.x) {
    const int b = cm.tile_inst[t];
    const InstDev I = cm.inst[b];
    if (!I.enabled) continue;
    const int lt = t - I.tile0, i0 = (lt % I.ntx) * kTX, j0 = (lt / I.ntx) * kTY;
    // the stored values of this thread's cells of the second pass, loaded ahead of the barrier so
    // that their latency overlaps the host-order loads
    V old[kItems] = {};
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
      const int q = threadIdx.x + k * kFieldThreads;
      const int i = i0 + (q % kTX), j = j0 + (q / kTX);  // i fastest
      if (restart && i < I.nx && j < I.ny) old[k] = A::ld(dst, I.base + (long long)j * I.pitch + i);
    }
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
      const int q = threadIdx.x + k * kFieldThreads;
      const int i = i0 + (q / kTY), j = j0 + (q % kTY);  // j fastest
      if (i < I.nx && j < I.ny) tile[j - j0][i - i0] = src[I.hoff + (long long)i * I.ny + j];
    }
    __syncthreads();
    int changed = 0;
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
      const int q = threadIdx.x + k * kFieldThreads;
      const int i = i0 + (q % kTX), j = j0 + (q / kTX);  // i fastest
      if (i < I.nx && j < I.ny) {
        const double v = tile[j - j0][i - i0];
        if (restart && __double_as_longlong(A::to_d_io(old[k])) == __double_as_longlong(v)) continue;
        changed = 1;
        A::st(dst, I.base + (long long)j * I.pitch + i, A::from_d_io(v));
      }
    }
    if (__syncthreads_or(restart && changed) && threadIdx.x == 0) cm.st[b].nhist = 0;
  }
}

// padded system order in the wide format -> alpha-major FP64, transposed like k_field_in (tiles
// [t0, t1) of the tile list; t1 < 0: all)
template <typename A>
__global__ void k_field_out(Common cm, double* dst, const double* src, int t0, int t1) {
  count_launch(cm.ctl);
  __shared__ double tile[kTY][kTX + 1];
  if (t1 < 0) t1 = n_tiles(cm);
  for (int t = t0 + blockIdx.x; t < t1; t += gridDim.x) {
    const int b = cm.tile_inst[t];
    const InstDev I = cm.inst[b];
    if (!I.enabled) continue;
    const int lt = t - I.tile0, i0 = (lt % I.ntx) * kTX, j0 = (lt / I.ntx) * kTY;
    for (int q = threadIdx.x; q < kTX * kTY; q += blockDim.x) {
      const int i = i0 + (q % kTX), j = j0 + (q / kTX);  // i fastest
      if (i < I.nx && j < I.ny) tile[j - j0][i - i0] = A::to_d_io(A::ld(src, I.base + (long long)j * I.pitch + i));
    }
    __syncthreads();
    for (int q = threadIdx.x; q < kTX * kTY; q += blockDim.x) {
      const int i = i0 + (q / kTY), j = j0 + (q % kTY);  // j fastest
      if (i < I.nx && j < I.ny) dst[I.hoff + (long long)i * I.ny + j] = tile[j - j0][i - i0];
    }
    __syncthreads();
  }
}

// ------------------------------------------------------------------------------ step control
static __global__ void k_begin(Common cm) {
  count_launch(cm.ctl);
  for (int b = blockIdx.x * blockDim.x + threadIdx.x, ni_ = n_inst(cm); b < ni_; b += gridDim.x * blockDim.x) {
    InstState& s = cm.st[b];
    const bool on = cm.inst[b].enabled != 0;
    s.outer_active = on ? 1 : 0;
    s.inner_active = 0;
    s.restart = 0;
    s.has_x = 0;
    s.iters = 0;
    s.iters_total = 0;
    s.refines = 0;
    s.clamped = 0;
    s.rmax_bits = 0u;
    if (on) atomicAdd(&cm.ctl->n_outer, 1);
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    cm.ctl->outer_loops = 0u;
    cm.ctl->inner_loops = 0u;
    cm.ctl->kdone[0] = 0u;
    cm.ctl->kdone[1] = 0u;
  }
}

// ------------------------------------------------------------------------------ assembly
template <typename C, typename A>
struct AsmOut;
template <typename A>
struct AsmOut<double, A> {
  template <typename Ix>
  __device__ static void put(const Coef<double>& c, int which, Ix idx, typename A::V v) {
    double* a = which == 0 ? c.cw : which == 1 ? c.ce : which == 2 ? c.cs : c.cn;
    a[idx] = A::to_d(v);
  }
};
template <typename A>
struct AsmOut<float, A> {
  template <typename Ix>
  __device__ static void put(const Coef<float>& c, int which, Ix idx, typename A::V v) {
    float hi, lo;
    A::split(v, hi, lo);
    float* a = which == 0 ? c.cw : which == 1 ? c.ce : which == 2 ? c.cs : c.cn;
    float* l = which == 0 ? c.lw : which == 1 ? c.le : which == 2 ? c.ls : c.ln;
    a[idx] = hi;
    l[idx] = lo;
  }
};

// Inner face (Solver.cc:99-141, calculate_mu Solver.h:63-67). K and L one-sided data:
// a_sigma = aA*fA + aB*fB, S = aA + aB, inv = 1/(f + eps).
template <typename A>
__device__ __forceinline__ void inner_face(typename A::V aK, typename A::V SK, typename A::V invK,
                                           typename A::V aL, typename A::V SL, typename A::V invL,
                                           typename A::V* AK, typename A::V* AL) {
  using V = typename A::V;
  const V absK = A::abs(aK), absL = A::abs(aL);
  const V denom = A::addf(A::addp(absK, absL), (float)(2 * kEps));  // both constants are powers of two
  const V muK = A::div(A::addf(absL, (float)kEps), denom);
  const V muL = A::rsub1(muK);
  const V B = A::dot2s(muL, aL, muK, aK);
  // B+ = (|B| + B)/2 goes to K's coefficient, B- = (|B| - B)/2 to L's; at most one is nonzero,
  // so only that one is multiplied by its 1/(f + eps) and added (all terms >= 0)
  const V mK = A::mul(muK, SK), mL = A::mul(muL, SL);
  const bool pos = A::gt0(B);
  const V X = A::fmap(pos ? B : A::pos_part(A::neg(B)), pos ? invK : invL, pos ? mK : mL);
  *AK = pos ? X : mK;
  *AL = pos ? mL : X;
}

// Dirichlet face (Solver.cc:143-164): B = -a_sigma; A = S + B+/(f+eps); R += B-.
template <typename A>
__device__ __forceinline__ void dirichlet_face(typename A::V aK, typename A::V SK, typename A::V invK,
                                               typename A::V* Aout, typename A::V* Bm) {
  *Aout = A::fmap(A::max0(A::neg(aK)), invK, SK);
  *Bm = A::max0(aK);
}

// Shared memory of one tile of kTX x (up to) kTY cells: vertices and faces are computed once per
// tile, plus a one-cell halo.
template <typename A>
struct AsmTile {
  using V = typename A::V;
  static constexpr int HX = kTX + 2, HY = kTY + 2, VX = kTX + 1, VY = kTY + 1;
  V fS[HY][HX];
  V iS[HY][HX];
  V vS[VY][VX];
  // x-faces: outflow to the left / right cell; y-faces: to the cell below / above. On a Dirichlet
  // side the slot of the missing outside cell holds the face's RHS part instead.
  V xL[kTY][VX], xR[kTY][VX];
  V yB[VY][kTX], yT[VY][kTX];
  V hS[VY][2];  // the tile's vertex rows: bilinear weights (wB, wT), Solver.cc:333-336
};

// Barrier among the threads that share a tile: the whole block, or (bar > 0) n of them.
__device__ __forceinline__ void tile_sync(int bar, int n) {
  if (bar == 0) __syncthreads();
  else asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(n) : "memory");
}

// Assembles the tile of up to kTX x ty cells at (i0, j0) of instance I by NT threads (tid: 0 .. NT; a
// power of two); returns this warp's max of the right-hand side. yc: the current y buffer; has_g: the idle
// one holds the extrapolated start. The cells, vertices and faces of a tile at the grid's right or upper edge
// are dealt to the threads without gaps: an idle lane takes as long as a busy one (both policies
// are bound by their arithmetic), and on grids of 64 to 256 a side a tenth of the lanes were idle.
// Measured with it (and, in FP64, the shorter reciprocal and the sign tests on bits), per 4-step call:
// double-word, 1024 uneven instances, 4.26 -> 4.05 ms; FP64, 192 instances, 3.46 -> 2.98 ms; mixed
// 4.07 -> 3.54 ms.
template <typename C, typename A>
__device__ __forceinline__ float asm_tile(AsmTile<A>& S, const Common& cm, const Geo& geo, const Fields& fl,
                                          const Coef<C>& co, const InstDev& I, int i0, int j0, const int ty,
                                          bool has_g, int yc, const int tid, const int NT, const int bar) {
  using V = typename A::V;
  constexpr int VX = AsmTile<A>::VX;
  const int nx = I.nx, ny = I.ny, P = I.pitch;
  const int w = min(kTX, nx - i0), h = min(ty, ny - j0), W1 = w + 1;
  // q / w and q / (w + 1) for q < 1900 as a multiplication and a shift
  const int rw = w == kTX ? 65536 / kTX + 1 : 65536 / w + 1, rW1 = w == kTX ? 65536 / (kTX + 1) + 1 : 65536 / W1 + 1;
  // f interpolated along each halo row at each vertex column (steps 1-2 only: shares the x-face
  // arrays' storage, which step 3 fills after a barrier)
  static_assert(AsmTile<A>::HY * VX <= 2 * kTY * VX, "row interpolations must fit in the x-face arrays");
  V(*const rS)[VX] = reinterpret_cast<V(*)[VX]>(&S.xL[0][0]);
  // the y-faces start at another warp than the x-faces, so that what is left over of each after whole
  // rounds of the block falls on different warps
  const int tid2 = (tid + NT / 2) & (NT - 1);
  const V zero = A::k(0.0);
  // 32-bit cell indices: every batch holds fewer than 2^31 cells (checked at allocation), and an
  // int index makes each address one wide multiply-add
  const int K0 = (int)I.base + j0 * P + i0;  // the tile's first cell
  const double* gp = sel2(fl.y64, yc ^ 1);
  // the per-cell data of step 4 is only needed after three barriers: start its trip to L2 now
#pragma unroll 1
  for (int q = tid; q < w * h; q += NT) {
    const int cy = (q * rw) >> 16, K = K0 + cy * P + (q - cy * w);
    asm volatile("prefetch.global.L2 [%0];" ::"l"(geo.sdiag + K));
    asm volatile("prefetch.global.L2 [%0];" ::"l"(geo.ukk + K));
    if (has_g) asm volatile("prefetch.global.L2 [%0];" ::"l"(gp + K));
  }
  // 1) per vertex column Iv and halo row j: f and 1/(f+eps) of the cell left of the column, and r = wL
  //    f_left + wR f_right, f interpolated along the row at the column (Solver.cc:333-336; a boundary
  //    column takes its adjacent cell's f). A thread keeps its column and walks halo rows `rows`
  //    apart; then the right halo column and the vertex rows' weights.
  {
    const int hy0 = (tid * rW1) >> 16, vx = tid - hy0 * W1, rows = (NT * rW1) >> 16, Iv = i0 + vx;
    if (hy0 < rows) {
      const bool xin = Iv > 0 && Iv < nx;
      const V wL = xin ? A::ld(cm.wx, 2 * (I.xe + Iv)) : zero;
      const V wR = xin ? A::ld(cm.wx, 2 * (I.xe + Iv) + 1) : zero;
      for (int hy = hy0; hy < h + 2; hy += rows) {
        const int j = j0 + hy - 1;
        V fa = zero, ia = zero, r = zero;
        if (j >= 0 && j < ny) {
          const int K = K0 + (hy - 1) * P + vx;  // the cell right of the column
          V fb = zero;
          if (Iv > 0) {
            fa = A::ld(fl.f, K - 1);
            ia = A::rcp(A::addf(fa, (float)kEps));
          }
          if (Iv < nx) fb = A::ld(fl.f, K);
          r = xin ? A::dot2(wL, fa, wR, fb) : (Iv == 0 ? fb : fa);
        }
        S.fS[hy][vx] = fa;
        S.iS[hy][vx] = ia;
        rS[hy][vx] = r;
      }
    }
    if (tid2 < h + 2) {
      const int i = i0 + w, j = j0 + tid2 - 1;
      V fv = zero, iv = zero;
      if (i < nx && j >= 0 && j < ny) {
        fv = A::ld(fl.f, K0 + (tid2 - 1) * P + w);
        iv = A::rcp(A::addf(fv, (float)kEps));
      }
      S.fS[tid2][W1] = fv;
      S.iS[tid2][W1] = iv;
    }
    if (NT - 1 - tid < h + 1) {
      const int vy = NT - 1 - tid, Jv = j0 + vy;
      const bool in = Jv > 0 && Jv < ny;
      S.hS[vy][0] = in ? A::ld(cm.wy, 2 * (I.ye + Jv)) : zero;
      S.hS[vy][1] = in ? A::ld(cm.wy, 2 * (I.ye + Jv) + 1) : zero;
    }
  }
  tile_sync(bar, NT);
  // 2) vertex values (Solver.cc:299-422): corners copy, interior bilinear, boundary edges
  //    linear, then Dirichlet overrides with XMIN < XMAX < YMIN < YMAX precedence. The bilinear
  //    value wB (wL f00 + wR f10) + wT (wL f01 + wR f11) is formed from the two row
  //    interpolations of step 1 with the same operations in the same order.
  for (int q = tid; q < W1 * (h + 1); q += NT) {
    const int vy = (q * rW1) >> 16, vx = q - vy * W1;
    const int Iv = i0 + vx, Jv = j0 + vy;
    V val;
    if (Jv == ny && I.bc[YMAX] == DIRICHLET) val = A::ld(cm.dirv, I.dir[YMAX] + Iv);
    else if (Jv == 0 && I.bc[YMIN] == DIRICHLET) val = A::ld(cm.dirv, I.dir[YMIN] + Iv);
    else if (Iv == nx && I.bc[XMAX] == DIRICHLET) val = A::ld(cm.dirv, I.dir[XMAX] + Jv);
    else if (Iv == 0 && I.bc[XMIN] == DIRICHLET) val = A::ld(cm.dirv, I.dir[XMIN] + Jv);
    else {
      // cell rows below / above vertex row Jv (halo rows vy, vy + 1), clamped to the domain at the edges
      const V r0 = rS[Jv > 0 ? vy : vy + 1][vx];
      if (Jv > 0 && Jv < ny) {  // interior and vertical boundary edges: linear in y
        const V r1 = rS[vy + 1][vx];
        val = A::dot2(S.hS[vy][0], r0, S.hS[vy][1], r1);
      } else {
        val = r0;  // horizontal boundary edges (linear in x) and corners
      }
    }
    S.vS[vy][vx] = val;
  }
  tile_sync(bar, NT);
  // 3a) x-faces (vertex column Iv between cells Iv-1 and Iv)
  for (int q = tid; q < W1 * h; q += NT) {
    const int ry = (q * rW1) >> 16, vx = q - ry * W1;
    const int Iv = i0 + vx, K = K0 + ry * P + vx, L = K - 1;
    V aL = zero, aR = zero, bm = zero;
    const V vLo = S.vS[ry][vx], vHi = S.vS[ry + 1][vx];  // vertices (Iv, j), (Iv, j+1)
    if (Iv > 0 && Iv < nx) {
      // K's XNEG edge: A=(Iv, j+1), B=(Iv, j); L's XPOS edge: A=(Iv, j), B=(Iv, j+1)
      const V aK = A::dot2(A::ld(geo.aAx, K), vHi, A::ld(geo.aBx, K), vLo);
      const V aLs = A::dot2(A::ld(geo.aAx, L), vLo, A::ld(geo.aBx, L), vHi);
      inner_face<A>(aK, A::ld(geo.Sx, K), S.iS[ry + 1][vx + 1], aLs, A::ld(geo.Sx, L), S.iS[ry + 1][vx], &aR, &aL);
    } else if (Iv == 0 && I.bc[XMIN] == DIRICHLET) {
      dirichlet_face<A>(A::dot2(A::ld(geo.aAx, K), vHi, A::ld(geo.aBx, K), vLo), A::ld(geo.Sx, K),
                        S.iS[ry + 1][vx + 1], &aR, &bm);
    } else if (Iv == nx && I.bc[XMAX] == DIRICHLET) {  // XPOS edge: A=(nx, j), B=(nx, j+1)
      dirichlet_face<A>(A::dot2(A::ld(geo.aAx, L), vLo, A::ld(geo.aBx, L), vHi), A::ld(geo.Sx, L),
                        S.iS[ry + 1][vx], &aL, &bm);
    }
    S.xL[ry][vx] = Iv == 0 ? bm : aL;
    S.xR[ry][vx] = Iv == nx ? bm : aR;
  }
  // 3b) y-faces (vertex row Jv between cells Jv-1 and Jv)
  for (int q = tid2; q < w * (h + 1); q += NT) {
    const int vy = (q * rw) >> 16, cx = q - vy * w;
    const int Jv = j0 + vy, K = K0 + vy * P + cx, L = K - P;
    V aB = zero, aT = zero, bm = zero;
    const V vLe = S.vS[vy][cx], vRi = S.vS[vy][cx + 1];  // vertices (i, Jv), (i+1, Jv)
    if (Jv > 0 && Jv < ny) {
      // K's YNEG edge: A=(i, Jv), B=(i+1, Jv); L's YPOS edge: A=(i+1, Jv), B=(i, Jv)
      const V aK = A::dot2(A::ld(geo.aAy, K), vLe, A::ld(geo.aBy, K), vRi);
      const V aLs = A::dot2(A::ld(geo.aAy, L), vRi, A::ld(geo.aBy, L), vLe);
      inner_face<A>(aK, A::ld(geo.Sy, K), S.iS[vy + 1][cx + 1], aLs, A::ld(geo.Sy, L), S.iS[vy][cx + 1], &aT, &aB);
    } else if (Jv == 0 && I.bc[YMIN] == DIRICHLET) {
      dirichlet_face<A>(A::dot2(A::ld(geo.aAy, K), vLe, A::ld(geo.aBy, K), vRi), A::ld(geo.Sy, K),
                        S.iS[vy + 1][cx + 1], &aT, &bm);
    } else if (Jv == ny && I.bc[YMAX] == DIRICHLET) {  // YPOS edge: A=(i+1,ny), B=(i,ny)
      dirichlet_face<A>(A::dot2(A::ld(geo.aAy, L), vRi, A::ld(geo.aBy, L), vLe), A::ld(geo.Sy, L),
                        S.iS[vy][cx + 1], &aB, &bm);
    }
    S.yB[vy][cx] = Jv == 0 ? bm : aB;
    S.yT[vy][cx] = Jv == ny ? bm : aT;
  }
  tile_sync(bar, NT);
  // 4) per cell: diagonal in the reference's triplet order, RHS, scaling, scatter
  float rmax = 0.0f;
#pragma unroll 1
  for (int q = tid; q < w * h; q += NT) {
    const int cy = (q * rw) >> 16, cx = q - cy * w;
    const int i = i0 + cx, j = j0 + cy, K = K0 + cy * P + cx;
    const V Aw = S.xR[cy][cx], Ae = S.xL[cy][cx + 1], As = S.yT[cy][cx], An = S.yB[cy + 1][cx];
    const bool wIn = i > 0, eIn = i < nx - 1, sIn = j > 0, nIn = j < ny - 1;
    // every term below is >= 0; a sum that is still zero takes its first term as it is (0 + x
    // = x), which spares an interior cell three double-word additions
    V D = wIn ? Aw : zero, Rv = zero, dir = zero;
    bool has_dir = false;
    if (eIn) D = A::addp(D, Ae);
    if (sIn) D = A::addp(D, As);
    if (nIn) D = A::addp(D, An);
    if (!wIn && I.bc[XMIN] == DIRICHLET) { D = A::addp(D, Aw); dir = A::addp(dir, Aw); Rv = A::addp(Rv, S.xL[cy][cx]); has_dir = true; }
    if (!eIn && I.bc[XMAX] == DIRICHLET) { D = A::addp(D, Ae); dir = A::addp(dir, Ae); Rv = A::addp(Rv, S.xR[cy][cx + 1]); has_dir = true; }
    if (!sIn && I.bc[YMIN] == DIRICHLET) { D = A::addp(D, As); dir = A::addp(dir, As); Rv = A::addp(Rv, S.yB[cy][cx]); has_dir = true; }
    if (!nIn && I.bc[YMAX] == DIRICHLET) { D = A::addp(D, An); dir = A::addp(dir, An); Rv = A::addp(Rv, S.yT[cy + 1][cx]); has_dir = true; }
    const V sd = A::ld(geo.sdiag, K);
    D = A::addp(D, sd);
    const V fK = S.fS[cy + 1][cx + 1];
    const V ukk = A::ld(geo.ukk, K);
    Rv = has_dir ? A::fmap(ukk, fK, Rv) : A::fma0(ukk, fK);
    rmax = fmaxf(rmax, fabsf(A::f32(Rv)));
    const V inv = A::rcp(D);
    A::st(fl.invD, K, inv);
    A::st(fl.R, K, Rv);
    A::st(fl.colsum, K, has_dir ? A::addp(sd, dir) : sd);
    // start the solve from D g, g the loss-compensated polynomial extrapolation in time the
    // last polish formed (only the starting point of the iteration; the converged answer does
    // not depend on it)
    A::st(sel2(fl.y64, yc), K, A::mul(D, has_g ? A::ld(gp, K) : fK));
    if (wIn) AsmOut<C, A>::put(co, 1, K - 1, A::mul(Aw, inv));  // row K-1, east entry
    if (eIn) AsmOut<C, A>::put(co, 0, K + 1, A::mul(Ae, inv));  // row K+1, west entry
    if (sIn) AsmOut<C, A>::put(co, 3, K - P, A::mul(As, inv));  // row K-P, north entry
    if (nIn) AsmOut<C, A>::put(co, 2, K + P, A::mul(An, inv));  // row K+P, south entry
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) rmax = fmaxf(rmax, __shfl_xor_sync(0xffffffffu, rmax, o));
  return rmax;
}

// One tile of kTX x kTY cells per iteration. Tiles [t0, t1) of the tile list (t1 < 0: all of them).
template <typename C, typename A>
__global__ void __launch_bounds__(kAsmThreads, A::kAsmBlocks) k_assemble(Common cm, Geo geo, Fields fl, Coef<C> co,
                                                                       int t0, int t1) {
  count_launch(cm.ctl);
  __shared__ AsmTile<A> S;
  const int nt_ = t1 < 0 ? n_tiles(cm) : t1;
  for (int t = t0 + blockIdx.x; t < nt_; t += gridDim.x) {
    const int b = cm.tile_inst[t];
    const InstDev I = cm.inst[b];
    if (!I.enabled) continue;  // uniform in the block
    const int lt = t - I.tile0;
    // the extrapolated start g the last polish left in the idle y buffer (none before the first
    // step or after the state was replaced: then y0 = D f)
    const float rmax = asm_tile<C, A>(S, cm, geo, fl, co, I, (lt % I.ntx) * kTX, (lt / I.ntx) * kTY, kTY,
                                      cm.st[b].nhist > 0, cm.st[b].ycur, threadIdx.x, kAsmThreads, 0);
    if ((threadIdx.x & 31) == 0 && rmax > 0.0f) atomicMax(&cm.st[b].rmax_bits, __float_as_uint(rmax));
    __syncthreads();
  }
}

}  // namespace sg

#include "sayram_solve.cuh"
