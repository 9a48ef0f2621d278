// sayram_solve.cuh -- the solve of one backward-Euler step: outer residual, BiCGSTAB, polish.
#pragma once

#include "sayram_ops.cuh"

namespace sg {

// ------------------------------------------------------------------------------ streaming helpers
// Resident blocks per SM the Krylov kernels are compiled for: in FP32, 6 (registers capped at
// 40; their shared memory allows 6, and the extra blocks in flight raised their bandwidth by
// 8-14 %); in FP64, 4 (a cap of 40 registers spills).
template <typename T>
constexpr int krylov_blocks() { return sizeof(T) == 4 ? 6 : 4; }

template <int CH>
__device__ __forceinline__ long long chunk_start(int c, const InstDev& I) {
  return I.base + (long long)(c - I.chunk0) * CH;
}
__device__ __forceinline__ long long inst_end(const InstDev& I) { return I.base + (long long)I.ny * I.pitch; }

// Runs body(c) for every chunk c of this block (c = blockIdx.x + k*gridDim.x) whose instance
// passes want(instance). The instance checks run in parallel, one chunk per thread, and the
// passing chunks are compacted in shared memory: a launch in which most instances have finished
// costs one round of checks per block instead of two dependent loads per chunk. Chunks are
// independent, so the order in which a block takes them does not change any result.
// Chunks [c0, c1) of the list only (c1 < 0: to the end).
template <typename W, typename Body>
__device__ __forceinline__ void for_active_chunks(const Common& cm, W&& want, Body&& body, int c0 = 0, int c1 = -1) {
  __shared__ int s_list[kThreads];
  __shared__ int s_cnt;
  const int nc = (c1 < 0 ? n_chunks(cm) : c1) - c0;
  const int per = (int)blockIdx.x < nc ? (nc - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
  for (int r0 = 0; r0 < per; r0 += kThreads) {
    if (threadIdx.x == 0) s_cnt = 0;
    __syncthreads();
    const int k = r0 + (int)threadIdx.x;
    if (k < per) {
      const int c = c0 + (int)blockIdx.x + k * (int)gridDim.x;
      if (want(cm.chunk_inst[c])) s_list[atomicAdd(&s_cnt, 1)] = c;
    }
    __syncthreads();
    const int m = s_cnt;
    for (int q = 0; q < m; ++q) body(s_list[q]);
    __syncthreads();
  }
}

// Fills smem[0 .. n) with a 4-aligned stretch [e0, e0 + n) of a vector computed cell-wise by
// f(k) -> Q4<T> (k a multiple of 4): the chunk plus one row above and below, so that the stencil
// of every cell in the chunk reads shared memory only.
template <typename T, int U = 2, typename F>
__device__ __forceinline__ void stage_rows(T* sm, long long e0, int n, F&& f) {
#pragma unroll U
  for (int q = 4 * threadIdx.x; q < n; q += 4 * kThreads) {
    const Q4<T> v = f(e0 + q);
    *reinterpret_cast<Q4<T>*>(sm + q) = v;
  }
}

// ------------------------------------------------------------------------------ Krylov arithmetic
// Every operation fused or rounded explicitly, so that all kernels that run a formula give the
// same bits.
__device__ __forceinline__ float fmaT(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fmaT(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float mulT(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mulT(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float subT(float a, float b) { return __fadd_rn(a, -b); }
__device__ __forceinline__ double subT(double a, double b) { return __dadd_rn(a, -b); }

// FP64 <-> FP32 of the preconditioner's factors (non-negative, at most a few units) by moving the
// fields: conversions run at the FP64 rate, 1/64 of the integer rate. Truncated; below FP32's
// normal range they become 0.
__device__ __forceinline__ float narrow(float a) { return a; }
__device__ __forceinline__ float narrow(double a) {
  const unsigned hi = (unsigned)__double2hiint(a), lo = (unsigned)__double2loint(a);
  return hi < 0x38100000u ? 0.0f : __uint_as_float(__funnelshift_l(lo, hi - 0x38000000u, 3));
}
template <typename T>
__device__ __forceinline__ T widen(float a);
template <>
__device__ __forceinline__ float widen<float>(float a) { return a; }
template <>
__device__ __forceinline__ double widen<double>(float a) {
  const unsigned b = __float_as_uint(a);
  return b < 0x00800000u ? 0.0 : __hiloint2double((int)((b >> 3) + 0x38000000u), (int)(b << 29));
}

// Alpha-line block preconditioner. Every 4-cell group of the padded layout lies inside one row
// (rows start at multiples of 4), and B is the tridiagonal of the group's own west/east couplings
// -- unit diagonal, -cw below, -ce above -- with the couplings to the neighbouring groups dropped:
// block Jacobi with 4-cell alpha-line blocks, the direction in which the scaled systems are
// stiffest (Dxx/dalpha^2 against Dyy/dlogE^2). line4 returns B^-1 q by Thomas elimination
// without pivoting (B is a column-diagonally-dominant M-matrix: every column of the outflow
// fractions sums to < 1, so each pivot stays in (0, 1]). The pivots are inverted in FP32, to a few ulps,
// whatever the vector precision (any map close to B^-1 preconditions as well; every kernel applies
// the same one); padding cells (q = cw = ce = 0) stay 0.
template <typename T>
struct Line {
  T w1, w2, w3, c0, c1, c2, i1, i2, i3;
};
__device__ __forceinline__ float rcp_fast(float a) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
  return r;
}
template <typename T>
__device__ __forceinline__ Line<T> line_of(const Q4<T>& cw, const Q4<T>& ce) {
  Line<T> L;
  L.w1 = cw.a[1];
  L.w2 = cw.a[2];
  L.w3 = cw.a[3];
  L.c0 = ce.a[0];
  const float i1 = rcp_fast(__fmaf_rn(-narrow(cw.a[1]), narrow(ce.a[0]), 1.0f));
  const float c1 = __fmul_rn(narrow(ce.a[1]), i1);
  const float i2 = rcp_fast(__fmaf_rn(-narrow(cw.a[2]), c1, 1.0f));
  const float c2 = __fmul_rn(narrow(ce.a[2]), i2);
  const float i3 = rcp_fast(__fmaf_rn(-narrow(cw.a[3]), c2, 1.0f));
  L.i1 = widen<T>(i1);
  L.i2 = widen<T>(i2);
  L.i3 = widen<T>(i3);
  L.c1 = widen<T>(c1);
  L.c2 = widen<T>(c2);
  return L;
}
template <typename T>
__device__ __forceinline__ Q4<T> line4(const Q4<T>& q, const Line<T>& L) {
  // forward: d_j = (q_j + w_j d_(j-1)) / pivot_j; backward: z_j = d_j + c_j z_(j+1)
  const T d0 = q.a[0];
  const T d1 = mulT(fmaT(L.w1, d0, q.a[1]), L.i1);
  const T d2 = mulT(fmaT(L.w2, d1, q.a[2]), L.i2);
  const T d3 = mulT(fmaT(L.w3, d2, q.a[3]), L.i3);
  Q4<T> z;
  z.a[3] = d3;
  z.a[2] = fmaT(L.c2, d3, d2);
  z.a[1] = fmaT(L.c1, z.a[2], d1);
  z.a[0] = fmaT(L.c0, z.a[1], d0);
  return z;
}

// A row of the matrix for one 4-cell group.
template <typename T>
struct Row {
  Q4<T> cw, ce, cs, cn;
};
template <typename T>
__device__ __forceinline__ Row<T> row_of(const Coef<T>& co, long long K) {
  return Row<T>{ld4(co.cw + K), ld4(co.ce + K), ld4(co.cs + K), ld4(co.cn + K)};
}
// B^-1 A~ x (or A~ x) over a group from a staged vector (sm + o: its first cell; rows P apart).
// In FP32: A~ = B - (couplings to other groups), so B^-1 A~ x = x - B^-1 q with q the inflow from the rows
// below and above and, at the group's ends, from its neighbours in the row; the couplings inside the
// group drop out. That takes B^-1 to the vectors' own precision (with FP64 vectors and FP32 pivots
// the solve's system would be off by 1e-7 and cost a refinement), so in FP64 it is B^-1 (A~ x).
template <typename T>
__device__ __forceinline__ Q4<T> product(const T* sm, int o, int P, const Row<T>& w, int precond) {
  const Q4<T> c = *reinterpret_cast<const Q4<T>*>(sm + o);
  const Q4<T> d = *reinterpret_cast<const Q4<T>*>(sm + o - P);
  const Q4<T> u = *reinterpret_cast<const Q4<T>*>(sm + o + P);
  const T w0 = sm[o - 1], e3 = sm[o + 4];
  Q4<T> q;
  if (sizeof(T) == 4 && precond) {
#pragma unroll
    for (int k = 0; k < 4; ++k) q.a[k] = fmaT(w.cn.a[k], u.a[k], mulT(w.cs.a[k], d.a[k]));
    q.a[0] = fmaT(w.cw.a[0], w0, q.a[0]);
    q.a[3] = fmaT(w.ce.a[3], e3, q.a[3]);
    q = line4<T>(q, line_of<T>(w.cw, w.ce));
#pragma unroll
    for (int k = 0; k < 4; ++k) q.a[k] = subT(c.a[k], q.a[k]);
    return q;
  }
  const T wv[4] = {w0, c.a[0], c.a[1], c.a[2]};
  const T ev[4] = {c.a[1], c.a[2], c.a[3], e3};
#pragma unroll
  for (int k = 0; k < 4; ++k)
    q.a[k] = fmaT(-w.cn.a[k], u.a[k], fmaT(-w.cs.a[k], d.a[k], fmaT(-w.ce.a[k], ev[k], fmaT(-w.cw.a[k], wv[k], c.a[k]))));
  if (precond) q = line4<T>(q, line_of<T>(w.cw, w.ce));
  return q;
}
template <typename T>
__device__ __forceinline__ T dot4(const Q4<T>& a, const Q4<T>& b, T q) {
#pragma unroll
  for (int m = 0; m < 4; ++m) q = fmaT(a.a[m], b.a[m], q);
  return q;
}

// ------------------------------------------------------------------------------ solver scalars
// The decisions of one instance's solve, shared by every kernel that runs it, on the types of the
// sums they follow from: one thread's FP64 divisions and conversions between two passes would cost
// more than the passes.
// after the residual: tot = ||r sc||^2, ||R sc||^2, ||B^-1 r sc||^2 (R: its sums' type, RK: the Krylov
// scalars'). Returns 0 when the step's solve ends here, 1 when a Krylov solve starts.
template <typename RK, typename R>
__device__ __forceinline__ int after_resid(InstState& st, const R (&tot)[3], double tol, double inner_tol,
                                           int max_refine, int precond) {
  if (st.has_x) {
    st.ycur ^= 1;  // the pass has written y + x to the other buffer
    if (st.iters == 1) st.swapped ^= 1;  // and r to x's place (resid_body)
  }
  st.has_x = 0;
  if (st.refines == 0) st.bb = stored(tot[1]);
  st.refines += 1;
  st.cum_refines += 1;
  st.rr64 = stored(tot[0]);
  const R bb = num<R>(st.bb);
  const R bound = rmul(rfrom<R>(tol * tol), bb);  // ||r|| <= tol ||R||, or R = 0
  if (!rgt(tot[0], bound) || !rgt(bb, rfrom<R>(0.0f))) {
    // A residual that is not a number, or that an infinite bound lets pass, is not below any tolerance (a
    // double-word sum that overflows becomes NaN: 2Sum subtracts infinities), and no solve starts from it
    st.outer_active = 0;
    st.status = isfinite(rhead(tot[0])) && isfinite(rhead(bb)) ? ST_OK : ST_NOT_CONVERGED;
    return 0;
  }
  if (st.refines >= max_refine) {
    st.outer_active = 0;
    st.status = ST_NOT_CONVERGED;
    return 0;
  }
  st.restart = 1;
  st.iters = 0;
  // the Krylov's residual is B^-1 r: its target is the relative reduction asked, or the final
  // tolerance carried into preconditioned units by this pass's norm ratio
  const R rrk = precond ? tot[2] : tot[0];
  st.rr = stored(rto(rrk, RK{}));
  const R a = rmul(rfrom<R>(inner_tol * inner_tol), rrk);
  R bnd = rmul(rfrom<R>(0.0625), bound);
  if (precond && rgt(tot[0], rfrom<R>(0.0f))) bnd = rmul(bnd, rdiv(rrk, tot[0]));
  st.rr_target = stored(rto(rgt(a, bnd) ? a : bnd, RK{}));
  return 1;
}
// after v = B^-1 A~ p: tot = (r^, v), (r, r) (the latter only formed on a restart)
template <typename R>
__device__ __forceinline__ void after_v(InstState& st, const R (&tot)[2]) {
  if (st.restart) {
    st.rho = st.iters == 0 ? st.rr : stored(tot[1]);  // (r^, r) with r^ = r
    st.restart = 0;
  }
  const R rho = num<R>(st.rho), alpha = rdiv(rho, tot[0]);
  if (rhead(tot[0]) != 0 && isfinite(rhead(tot[0])) && isfinite(rhead(alpha)) && rhead(rho) != 0) {
    st.alpha = stored(alpha);
  } else {
    st.alpha = 0.0;  // breakdown: this iteration degenerates to a minimal-residual step
    st.restart = 1;
  }
}
// after t = B^-1 A~ s: tot = (t, s), (t, t), (s, s), (r^, s), (r^, t). The next residual is r = s -
// omega t, so (r, r) and (r^, r) follow from these sums and the pass that would form them is not
// needed. (r^, s) is zero by the choice of alpha, but for rounding, and is summed all the same: without
// it the error of rho stays from one iteration to the next, and long solves stall (four sums were 3 % faster
// on most double-word cases, but a burst of 48 server requests took 378 instead of 39 ms and, from the same
// fields, four FP64 steps of 1024 x 1024 23.6 instead of 12.7). Returns 1 when this Krylov solve ends.
template <typename R>
__device__ __forceinline__ int after_t(InstState& st, const R (&tot)[5], int max_iters) {
  const R ts = tot[0], tt = tot[1];
  R om = rfrom<R>(0.0f);
  if (rhead(tt) > 0 && isfinite(rhead(ts))) om = rdiv(ts, tt);
  if (!isfinite(rhead(om))) om = rfrom<R>(0.0f);
  st.omega = stored(om);
  if (rhead(om) == 0) st.restart = 1;
  const R rr = rfma(om, rfma(om, tt, rneg(radd(ts, ts))), tot[2]);
  const R rhoN = rfma(rneg(om), tot[4], tot[3]);
  st.rr = stored(rr);
  st.iters += 1;
  st.iters_total += 1;
  st.cum_iters += 1;
  if (!rgt(rr, num<R>(st.rr_target)) || st.iters >= max_iters || !isfinite(rhead(rr))) {
    st.has_x = 1;
    return 1;
  }
  const R beta = rmul(rdiv(rhoN, num<R>(st.rho)), rdiv(num<R>(st.alpha), om));
  st.rho = stored(rhoN);
  if (!isfinite(rhead(beta)) || rhead(rhoN) == 0) {
    st.restart = 1;
    st.beta = 0.0;
  } else {
    st.beta = stored(beta);
  }
  // A restart writes r^, which the second iteration's first pass still reads as r and p, also where a
  // neighbouring block writes: the next residual is the restart there.
  if (st.restart && st.iters == 1) {
    st.has_x = 1;
    return 1;
  }
  return 0;
}

// Coefficients of a row in the wide arithmetic: from the FP64 arrays or the (hi, lo) split
template <typename C, typename A>
struct CoefW;
template <typename A>
struct CoefW<double, A> {
  __device__ static typename A::V cell(const Coef<double>& c, int which, long long K) {
    const double* a = which == 0 ? c.cw : which == 1 ? c.ce : which == 2 ? c.cs : c.cn;
    return A::from_d(a[K]);
  }
  __device__ static Q4<typename A::V> row(const Coef<double>& c, int which, long long K) {
    const double* a = which == 0 ? c.cw : which == 1 ? c.ce : which == 2 ? c.cs : c.cn;
    const Q4<double> q = ld4(a + K);
    Q4<typename A::V> o;
#pragma unroll
    for (int k = 0; k < 4; ++k) o.a[k] = A::from_d(q.a[k]);
    return o;
  }
};
template <typename A>
struct CoefW<float, A> {
  __device__ static typename A::V cell(const Coef<float>& c, int which, long long K) {
    const float* a = which == 0 ? c.cw : which == 1 ? c.ce : which == 2 ? c.cs : c.cn;
    const float* l = which == 0 ? c.lw : which == 1 ? c.le : which == 2 ? c.ls : c.ln;
    return A::hilo(a[K], l[K]);
  }
  __device__ static Q4<typename A::V> row(const Coef<float>& c, int which, long long K) {
    const float* a = which == 0 ? c.cw : which == 1 ? c.ce : which == 2 ? c.cs : c.cn;
    const float* l = which == 0 ? c.lw : which == 1 ? c.le : which == 2 ? c.ls : c.ln;
    const Q4<float> h = ld4(a + K), lo = ld4(l + K);
    Q4<typename A::V> o;
#pragma unroll
    for (int k = 0; k < 4; ++k) o.a[k] = A::hilo(h.a[k], lo.a[k]);
    return o;
  }
};

template <typename T>
constexpr bool kStoreS = sizeof(T) == 8;  // s of an iteration is stored (see k_bicg1)
// The shadow residual and the solution of an instance's solve. A solve's first iteration has p = r =
// r^ and no x, so the residual after a solve of one iteration reads r^ in its neighbours' rows too:
// it writes the next solve's into x's array, and the two change places.
template <typename T>
__device__ __forceinline__ T* rh_of(const Kry<T>& kr, const InstState& st) { return st.swapped ? kr.x : kr.rh; }
template <typename T>
__device__ __forceinline__ T* x_of(const Kry<T>& kr, const InstState& st) { return st.swapped ? kr.rh : kr.x; }

// ------------------------------------------------------------------------------ outer residual
// One 4-cell group of r = R - A~ y in the wide arithmetic from the staged y (sm + o): y itself, the
// scaled residual with the preconditioner applied, and the group's terms of ||r||^2, ||R||^2 and
// ||B^-1 r||^2.
template <typename T, typename C, typename A>
__device__ __forceinline__ void resid_group(const typename A::V* sm, int o, int P, const Coef<C>& co, long long K,
                                            const double* Rp, float sc, int precond, bool first, Q4<typename A::V>& yc,
                                            Q4<T>& r, typename A::Acc& q0, typename A::Acc& q1, T& q2) {
  using V = typename A::V;
  const Q4<V> cw = CoefW<C, A>::row(co, 0, K), ce = CoefW<C, A>::row(co, 1, K);
  const Q4<V> cs = CoefW<C, A>::row(co, 2, K), cn = CoefW<C, A>::row(co, 3, K);
  const Q4<V> R = A::ld4(Rp + K);
  yc = *reinterpret_cast<const Q4<V>*>(sm + o);
  const Q4<V> d = *reinterpret_cast<const Q4<V>*>(sm + o - P), u = *reinterpret_cast<const Q4<V>*>(sm + o + P);
  const V w0 = sm[o - 1], e3 = sm[o + 4];
#pragma unroll
  for (int m = 0; m < 4; ++m) {
    // (R - y) + the neighbours' inflow, one multiply-add each
    const V rv = A::fma(cn.a[m], u.a[m], A::fma(cs.a[m], d.a[m],
                        A::fma(ce.a[m], m < 3 ? yc.a[(m + 1) & 3] : e3,
                               A::fma(cw.a[m], m > 0 ? yc.a[(m + 3) & 3] : w0, A::sub(R.a[m], yc.a[m])))));
    r.a[m] = A::template scaled<T>(rv, sc);
    q0 = A::sq_scaled(rv, sc, q0);
    if (first) q1 = A::sq_scaled(R.a[m], sc, q1);  // ||R|| does not change within a step
  }
  if (precond) {  // the Krylov matrix's couplings (the hi parts in the FP32 modes)
    r = line4<T>(r, line_of<T>(ld4(co.cw + K), ld4(co.ce + K)));
    q2 = dot4<T>(r, r, q2);
  }
}

// ---- one cell per lane. A share of few cells keeps few warps busy with four cells per lane, one after
// another; with a cell per lane it keeps four times as many. The lanes of a group chain its sums
// in the order of the 4-cell form, so the bits are the same.
// acc over the group's cells in order: f(a, x) with this lane's x, a from the lane before; all lanes get
// the group's result
template <typename X>
__device__ __forceinline__ X lane_get(X a, int from) { return __shfl_sync(0xffffffffu, a, from); }
__device__ __forceinline__ dw lane_get(dw a, int from) {
  return dw{__shfl_sync(0xffffffffu, a.hi, from), __shfl_sync(0xffffffffu, a.lo, from)};
}
template <typename X, typename F>
__device__ __forceinline__ X group_chain(X zero, F&& f) {
  const int base = threadIdx.x & 28;
  X acc = zero;
#pragma unroll
  for (int j = 0; j < 4; ++j) acc = lane_get(f(acc), base + j);
  return acc;
}
// resid_group for the cell of this lane (on: the cell is in the share; every lane of a warp comes here);
// q0, q1, q2: the group's terms, in each of its lanes
template <typename T, typename C, typename A>
__device__ __forceinline__ void resid_cell(const typename A::V* sm, int o, int P, const Coef<C>& co, long long K, bool on,
                                           const double* Rp, float sc, int precond, bool first, typename A::V& yc, T& r,
                                           typename A::Acc& q0, typename A::Acc& q1, T& q2) {
  using V = typename A::V;
  V rv = A::k(0.0), R = A::k(0.0);
  Q4<T> cwq{}, ceq{};
  r = (T)0;
  if (on) {
    R = A::ld(Rp, K);
    yc = sm[o];
    if (precond) {
      cwq = ld4(co.cw + (K & ~3LL));
      ceq = ld4(co.ce + (K & ~3LL));
    }
    rv = A::fma(CoefW<C, A>::cell(co, 3, K), sm[o + P], A::fma(CoefW<C, A>::cell(co, 2, K), sm[o - P],
                A::fma(CoefW<C, A>::cell(co, 1, K), sm[o + 1], A::fma(CoefW<C, A>::cell(co, 0, K), sm[o - 1],
                A::sub(R, yc)))));
    r = A::template scaled<T>(rv, sc);
  }
  using Acc = typename A::Acc;
  q0 = group_chain<Acc>((Acc)0, [&](Acc a) { return A::sq_scaled(rv, sc, a); });
  q1 = first ? group_chain<Acc>((Acc)0, [&](Acc a) { return A::sq_scaled(R, sc, a); }) : (Acc)0;
  q2 = (T)0;
  if (precond) {
    const int base = threadIdx.x & 28;
    Q4<T> g;
#pragma unroll
    for (int j = 0; j < 4; ++j) g.a[j] = __shfl_sync(0xffffffffu, r, base + j);
    g = line4<T>(g, line_of<T>(cwq, ceq));
    const int c = threadIdx.x & 3;
    r = c == 0 ? g.a[0] : c == 1 ? g.a[1] : c == 2 ? g.a[2] : g.a[3];
    q2 = dot4<T>(g, g, (T)0);
  }
}

// r = R - A~ (y + x) in the wide arithmetic; writes y + x to the other y buffer (where there is an x)
// and the Krylov's right-hand side B^-1 r (T precision, scaled) to rh.
template <typename T, typename C, typename A, int CH>
__device__ __forceinline__ void resid_body(const Common& cm, const Fields& fl, const Coef<C>& co, const Kry<T>& kr) {
  using V = typename A::V;
  using R = typename A::R;
  using Sums = ChunkSums<CH, 3, R>;
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ double s_part[3 * Sums::kParts];
  V* sm = reinterpret_cast<V*>(smraw);
  for_active_chunks(cm, [&](int b_) { return cm.st[b_].outer_active != 0; }, [&](int c) {
    const int b = cm.chunk_inst[c];
    const InstState& st = cm.st[b];
    const InstDev& I = cm.inst[b];  // fields are read where they are needed: registers are short
    const double* yin = sel2(fl.y64, st.ycur);
    double* yout = sel2(fl.y64, st.ycur ^ 1);
    const bool hx = st.has_x != 0;
    T* const rout = hx && st.iters == 1 ? x_of(kr, st) : rh_of(kr, st);
    const float sc = rhs_scale(st.rmax_bits);  // r is handed over as r * sc
    const float isc = 1.0f / sc;                // exact: sc is a power of two
    const int P = I.pitch;
    const long long c0 = chunk_start<CH>(c, I);
    const long long c1 = min(c0 + (long long)CH, inst_end(I));
    const long long e0 = c0 - P;
    Sums sums{reinterpret_cast<R(*)[Sums::kParts]>(s_part)};
    // y, or y + x (the last Krylov correction, in scaled units), over the chunk and one row each side.
    // The last iteration's part of x is formed here from its vectors: a pass of its own over the
    // instances that finish in an iteration would move more bytes and take a launch.
    if (!hx) {
      stage_rows<V>(sm, e0, (int)(c1 - c0) + 2 * P, [&](long long k) { return A::ld4(yin + k); });
    } else {
      using RK = typename RedOf<T>::R;
      const int it = st.iters;
      const T alpha = rhead(num<RK>(st.alpha)), omega = rhead(num<RK>(st.omega));
      const T* rr = kStoreS<T> ? kr.r[1] : it > 1 ? sel2(kr.r, it & 1) : rh_of(kr, st);  // s, or r
      const T* pp = it > 1 ? sel2(kr.p, it & 1) : rh_of(kr, st);
      const T* xx = x_of(kr, st);
      const T* vv = sel2(kr.v, it & 1);
      stage_rows<V>(sm, e0, (int)(c1 - c0) + 2 * P, [&](long long k) {
        Q4<V> y = A::ld4(yin + k);
        Q4<T> s = ld4(rr + k), v;
        if (!kStoreS<T>) v = ld4(vv + k);
        const Q4<T> p = kStoreS<T> || it > 1 ? ld4(pp + k) : s;
        Q4<T> x{{(T)0, (T)0, (T)0, (T)0}};
        if (it > 1) x = ld4(xx + k);
#pragma unroll
        for (int m = 0; m < 4; ++m) {
          const T sv = kStoreS<T> ? s.a[m] : fmaT(-alpha, v.a[m], s.a[m]);
          const T xv = fmaT(alpha, p.a[m], fmaT(omega, sv, x.a[m]));
          y.a[m] = A::template add_scaled<T>(y.a[m], xv, isc);
        }
        return y;
      });
    }
    __syncthreads();
    typename A::Acc q0 = 0, q1 = 0;
    T q2 = (T)0;
    for_parts<CH>(I.seg, [&](int g) {
      const long long K = c0 + 4 * g;
      if (K >= c1) return;
      Q4<V> yc;
      Q4<T> r;
      resid_group<T, C, A>(sm, (int)(K - e0), P, co, K, fl.R, sc, cm.precond, st.refines == 0, yc, r, q0, q1, q2);
      if (hx) A::st4(yout + K, yc);
      st4(rout + K, r);
    }, [&](int p) {
      const typename A::Acc w[3] = {q0, q1, q2};
      sums.put(p, w);
      q0 = q1 = 0;
      q2 = (T)0;
    });
    const int sl = (c - I.chunk0) * (CH / I.seg);
    sums.store(reinterpret_cast<R*>(cm.part), cm.pstride, I.seg0 + sl, I.nseg - sl, I.seg);
  });
}
template <typename T, typename C, typename A, int CH>
__global__ void __launch_bounds__(kThreads, sizeof(typename A::Acc) == 4 ? 4 : 3) k_resid(Common cm, Fields fl, Coef<C> co, Kry<T> kr) {
  count_launch(cm.ctl);
  resid_body<T, C, A, CH>(cm, fl, co, kr);
}

// ------------------------------------------------------------------------------ BiCGSTAB
// Left-preconditioned BiCGSTAB on B^-1 A~ x = B^-1 r (B = I without the preconditioner; the
// residual r the kernels carry is the preconditioned one, and x is the correction itself), in
// two passes per iteration:
// k1: r = s - omega t and x += alpha p + omega s of the previous iteration, p = r + beta (p - omega
//     v) (p = r on a restart, which also sets r^ = r), v = B^-1 A~ p; sums (r^, v). r and p are
//     computed once per cell into shared memory (chunk plus one row above and below) and the
//     stencil reads p there. The first iteration of a solve has p = r = r^ and writes only v.
// k2: s = r - alpha v staged likewise, t = B^-1 A~ s; the five sums of after_t.
// The residual kernel forms x's last part (alpha p + omega s) of a solve that has ended.
// The residual's own dot products come from k2's sums (after_t), so no third pass over the vectors
// separates r from p: 88 B per cell and iteration in FP32 (first iteration 52 B) against 100 B (88
// B) for update, product and update as three passes, and one barrier or launch less. FP64 is bound
// by its pipe (525 GFMA/s): 26 operations per cell and iteration against 39, with the stencil as
// four multiply-adds and no FP64-rate conversions in the preconditioner. Measured, whole calls: 192
// uneven FP64 instances, 4 steps, 19.2 -> 15.8 ms; 1024 in double-word 22.5 -> 20.2 ms; 24 in
// double-word, 6 steps, 2.94 -> 2.47 ms; 192 mixed with Jacobi scaling 14.7 -> 14.0 ms.
// FP64 is bound by its pipe, not by HBM: there k2 stores s (in r[1]; r stays in r[0]), and neither the
// next k1 nor the residual kernel forms it again (192 uneven instances, 4 steps: k1 4.15 -> 3.95, k2
// 3.47 -> 3.52, residuals 1.24 -> 1.21 ms).
template <typename T, int CH>
__device__ __forceinline__ void bicg1_body(const Common& cm, const Coef<T>& co, const Kry<T>& kr) {
  using R = typename RedOf<T>::R;
  using Sums = ChunkSums<CH, 2, R>;
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ double s_part[2 * Sums::kParts];
  T* sm = reinterpret_cast<T*>(smraw);
  for_active_chunks(cm, [&](int b_) { return cm.st[b_].inner_active != 0; }, [&](int c) {
    const int b = cm.chunk_inst[c];
    const InstState& st = cm.st[b];
    const InstDev& I = cm.inst[b];  // fields are read where they are needed: registers are short
    const int it = st.iters;  // iterations finished; this one is it + 1
    const bool rs = st.restart != 0;
    const T alpha = rhead(num<R>(st.alpha)), beta = rhead(num<R>(st.beta)), omega = rhead(num<R>(st.omega));
    T* const rhat = rh_of(kr, st);
    T* const xx = x_of(kr, st);
    const T* ro = kStoreS<T> ? kr.r[1] : it > 1 ? sel2(kr.r, it & 1) : rhat;  // s, or r
    const T* po = it > 1 ? sel2(kr.p, it & 1) : rhat;
    const T* vo = sel2(kr.v, it & 1);
    T* rn = kStoreS<T> ? kr.r[0] : sel2(kr.r, (it + 1) & 1);
    T* pn = sel2(kr.p, (it + 1) & 1);
    T* vn = sel2(kr.v, (it + 1) & 1);
    const int P = I.pitch;
    const long long c0 = chunk_start<CH>(c, I);
    const long long c1 = min(c0 + (long long)CH, inst_end(I));
    const long long e0 = c0 - P;
    Sums sums{reinterpret_cast<R(*)[Sums::kParts]>(s_part)};
    if (it == 0) {
      stage_rows<T>(sm, e0, (int)(c1 - c0) + 2 * P, [&](long long k) { return ld4(rhat + k); });
    } else {
      stage_rows<T, 1>(sm, e0, (int)(c1 - c0) + 2 * P, [&](long long k) {
        const Q4<T> r = ld4(ro + k), v = ld4(vo + k), t = ld4(kr.t + k);
        Q4<T> p = kStoreS<T> || it > 1 ? ld4(po + k) : r;
        const bool mine = k >= c0 && k < c1;
        Q4<T> s, q;
#pragma unroll
        for (int m = 0; m < 4; ++m) {
          s.a[m] = kStoreS<T> ? r.a[m] : fmaT(-alpha, v.a[m], r.a[m]);
          q.a[m] = fmaT(-omega, t.a[m], s.a[m]);
        }
        if (mine) {
          Q4<T> x{{(T)0, (T)0, (T)0, (T)0}};
          if (it > 1) x = ld4(xx + k);
#pragma unroll
          for (int m = 0; m < 4; ++m) x.a[m] = fmaT(alpha, p.a[m], fmaT(omega, s.a[m], x.a[m]));
          st4(xx + k, x);
        }
#pragma unroll
        for (int m = 0; m < 4; ++m) p.a[m] = rs ? q.a[m] : fmaT(beta, fmaT(-omega, v.a[m], p.a[m]), q.a[m]);
        if (mine) {
          st4(rn + k, q);
          st4(pn + k, p);
          if (rs) st4(rhat + k, q);
        }
        return p;
      });
    }
    __syncthreads();
    T q0 = (T)0, q1 = (T)0;
    for_parts<CH>(I.seg, [&](int g) {
      const long long K = c0 + 4 * g;
      if (K < c1) {
        const int o = (int)(K - e0);
        const Q4<T> v = product<T>(sm, o, P, row_of<T>(co, K), cm.precond);  // v = B^-1 A~ p
        st4(vn + K, v);
        // r^ (on a restart it is p itself)
        const Q4<T> rh = rs ? *reinterpret_cast<const Q4<T>*>(sm + o) : ld4(rhat + K);
        q0 = dot4<T>(rh, v, q0);
        if (rs && it > 0) q1 = dot4<T>(rh, rh, q1);
      }
    }, [&](int p) {
      const T w[2] = {q0, q1};
      sums.put(p, w);
      q0 = q1 = (T)0;
    });
    const int sl = (c - I.chunk0) * (CH / I.seg);
    sums.store(reinterpret_cast<R*>(cm.part), cm.pstride, I.seg0 + sl, I.nseg - sl, I.seg);
  });
}
template <typename T, int CH>
__global__ void __launch_bounds__(kThreads, krylov_blocks<T>()) k_bicg1(Common cm, Coef<T> co, Kry<T> kr) {
  count_launch(cm.ctl);
  bicg1_body<T, CH>(cm, co, kr);
}

template <typename T, int CH>
__device__ __forceinline__ void bicg2_body(const Common& cm, const Coef<T>& co, const Kry<T>& kr) {
  using R = typename RedOf<T>::R;
  using Sums = ChunkSums<CH, 5, R>;
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ double s_part[5 * Sums::kParts];
  T* sm = reinterpret_cast<T*>(smraw);
  for_active_chunks(cm, [&](int b_) { return cm.st[b_].inner_active != 0; }, [&](int c) {
    const int b = cm.chunk_inst[c];
    const InstState& st = cm.st[b];
    const InstDev& I = cm.inst[b];  // fields are read where they are needed: registers are short
    const int it = st.iters;
    const T alpha = rhead(num<R>(st.alpha));
    const T* const rhat = rh_of(kr, st);
    const T* r = it == 0 ? rhat : kStoreS<T> ? kr.r[0] : sel2(kr.r, (it + 1) & 1);
    const T* vv = sel2(kr.v, (it + 1) & 1);
    const int P = I.pitch;
    const long long c0 = chunk_start<CH>(c, I);
    const long long c1 = min(c0 + (long long)CH, inst_end(I));
    const long long e0 = c0 - P;
    Sums sums{reinterpret_cast<R(*)[Sums::kParts]>(s_part)};
    stage_rows<T>(sm, e0, (int)(c1 - c0) + 2 * P, [&](long long k) {
      Q4<T> x = ld4(r + k);
      const Q4<T> v = ld4(vv + k);
#pragma unroll
      for (int m = 0; m < 4; ++m) x.a[m] = fmaT(-alpha, v.a[m], x.a[m]);
      if (kStoreS<T> && k >= c0 && k < c1) st4(kr.r[1] + k, x);
      return x;
    });
    __syncthreads();
    T q[5] = {(T)0, (T)0, (T)0, (T)0, (T)0};
    for_parts<CH>(I.seg, [&](int g) {
      const long long K = c0 + 4 * g;
      if (K < c1) {
        const int o = (int)(K - e0);
        const Q4<T> s = *reinterpret_cast<const Q4<T>*>(sm + o);
        const Q4<T> t = product<T>(sm, o, P, row_of<T>(co, K), cm.precond);  // t = B^-1 A~ s
        st4(kr.t + K, t);
        const Q4<T> rh = ld4(rhat + K);
        q[0] = dot4<T>(t, s, q[0]);
        q[1] = dot4<T>(t, t, q[1]);
        q[2] = dot4<T>(s, s, q[2]);
        q[3] = dot4<T>(rh, s, q[3]);
        q[4] = dot4<T>(rh, t, q[4]);
      }
    }, [&](int p) {
      sums.put(p, q);
#pragma unroll
      for (int k = 0; k < 5; ++k) q[k] = (T)0;
    });
    const int sl = (c - I.chunk0) * (CH / I.seg);
    sums.store(reinterpret_cast<R*>(cm.part), cm.pstride, I.seg0 + sl, I.nseg - sl, I.seg);
  });
}
template <typename T, int CH>
__global__ void __launch_bounds__(kThreads, krylov_blocks<T>()) k_bicg2(Common cm, Coef<T> co, Kry<T> kr) {
  count_launch(cm.ctl);
  bicg2_body<T, CH>(cm, co, kr);
}

// The decisions that follow from a pass's sums, in a small kernel of their own after it (one block per
// instance concerned). The passes' blocks leave right after their sums: counting themselves in (a
// fence and an atomic per chunk, so that the last could decide) held each of them up for ~2 us
// of its ~20, and k_bicg2 on 1024 instances took 3.30 ms a call instead of 2.74.
template <int NQ, typename R, typename W, typename D>
__device__ __forceinline__ void decide(const Common& cm, W&& want, D&& body) {
  __shared__ double s_tot[8 * NQ];
  R* sm = reinterpret_cast<R*>(s_tot);
  for (int b = blockIdx.x, ni = n_inst(cm); b < ni; b += gridDim.x) {
    InstState& st = cm.st[b];
    if (!want(st)) continue;  // uniform in the block
    const InstDev& I = cm.inst[b];
    __syncthreads();
    seg_total<NQ, kThreads / 32, R>(reinterpret_cast<const R*>(cm.part), cm.pstride, I.seg0, I.nseg, sm);
    if (threadIdx.x == 0) {
      R tot[NQ];
#pragma unroll
      for (int q = 0; q < NQ; ++q) tot[q] = sm[q];
      body(st, tot);
    }
  }
}
template <typename T, typename A>
__global__ void __launch_bounds__(kThreads) k_after_resid(Common cm, double tol, double inner_tol, int max_refine) {
  using R = typename A::R;
  count_launch(cm.ctl);
  decide<3, R>(cm, [](const InstState& st) { return st.outer_active != 0; }, [&](InstState& st, const R(&tot)[3]) {
    if (after_resid<typename RedOf<T>::R, R>(st, tot, tol, inner_tol, max_refine, cm.precond)) {
      st.inner_active = 1;
      atomicAdd(&cm.ctl->n_inner, 1);
    } else {
      atomicSub(&cm.ctl->n_outer, 1);
    }
  });
  loop_epilogue(cm, 0);
}
template <typename T>
__global__ void __launch_bounds__(kThreads) k_after_v(Common cm) {
  using R = typename RedOf<T>::R;
  count_launch(cm.ctl);
  decide<2, R>(cm, [](const InstState& st) { return st.inner_active != 0; },
               [&](InstState& st, const R(&tot)[2]) { after_v(st, tot); });
}
template <typename T>
__global__ void __launch_bounds__(kThreads) k_after_t(Common cm, int max_iters) {
  using R = typename RedOf<T>::R;
  count_launch(cm.ctl);
  decide<5, R>(cm, [](const InstState& st) { return st.inner_active != 0; }, [&](InstState& st, const R(&tot)[5]) {
    if (after_t(st, tot, max_iters)) {
      st.inner_active = 0;
      atomicSub(&cm.ctl->n_inner, 1);
    }
  });
  loop_epilogue(cm, 1);
}

// ------------------------------------------------------------------------------ polish + checks
// The polish's pointers for one instance: its solution y, the idle y buffer (which takes the next
// start g) and the earlier states the start goes back to (f^n, the current f, and up to kOrder - 1
// from the history).
struct PolishAt {
  const double* y;
  double* gout;
  const double *h2, *h3, *h4;
  double* hw;  // the oldest slot (f^(n-3)) takes f^n
  int nh;
};
__device__ __forceinline__ PolishAt polish_at(const Fields& fl, int ycur, int nhist, int hslot, int hist_cap) {
  PolishAt a;
  a.y = sel2(fl.y64, ycur);
  a.gout = sel2(fl.y64, ycur ^ 1);
  a.nh = min(min(nhist + 1, kOrder), hist_cap);
  a.h2 = sel3(fl.fh, hslot);
  a.h3 = sel3(fl.fh, (hslot + 2) % kHist);
  a.h4 = sel3(fl.fh, (hslot + 1) % kHist);
  a.hw = sel3(fl.fh, (hslot + 1) % kHist);
  return a;
}
// One 4-cell group from the staged max(y, 0) (sm + o); real: cells of the group inside the grid
// EARLY: every load is issued before the first is used (more registers: for few warps in flight).
template <typename C, typename A, bool EARLY>
__device__ __forceinline__ void polish_group(const typename A::V* sm, int o, int P, const Coef<C>& co, long long K,
                                             const Fields& fl, const PolishAt& at, int real, typename A::V& mass,
                                             typename A::V& rsum, float& mn) {
  using V = typename A::V;
  // y' = R + sum over the neighbours of the outflow fraction times max(y, 0): every term is
  // >= 0, accumulated one direction at a time so that one coefficient row is live at once
  const Q4<V> R = A::ld4(fl.R + K);
  Q4<V> yp = R, e_inv, e_cols, e_fn, e_h2, e_h3, e_h4, e_r;
  if (EARLY) {
    e_inv = A::ld4(fl.invD + K);
    e_cols = A::ld4(fl.colsum + K);
    e_fn = A::ld4(fl.f + K);
    e_h2 = at.nh >= 2 ? A::ld4(at.h2 + K) : e_fn;
    e_h3 = at.nh >= 3 ? A::ld4(at.h3 + K) : e_h2;
    e_h4 = at.nh >= 4 ? A::ld4(at.h4 + K) : e_h3;
    if (fl.decay) e_r = A::ld4(fl.decay + K);
  }
#pragma unroll
  for (int dir = 0; dir < 4; ++dir) {
    const Q4<V> c = CoefW<C, A>::row(co, dir, K);
    // the neighbours' values: the group's own shifted by one cell, or the group in the row below or above
    Q4<V> y = *reinterpret_cast<const Q4<V>*>(sm + o + (dir == 2 ? -P : dir == 3 ? P : 0));
    if (dir == 0) {
      y.a[3] = y.a[2];
      y.a[2] = y.a[1];
      y.a[1] = y.a[0];
      y.a[0] = sm[o - 1];
    } else if (dir == 1) {
      y.a[0] = y.a[1];
      y.a[1] = y.a[2];
      y.a[2] = y.a[3];
      y.a[3] = sm[o + 4];
    }
#pragma unroll
    for (int m = 0; m < 4; ++m) yp.a[m] = A::fmap(c.a[m], y.a[m], yp.a[m]);
  }
  const Q4<V> inv = EARLY ? e_inv : A::ld4(fl.invD + K), cols = EARLY ? e_cols : A::ld4(fl.colsum + K);
  Q4<V> fo;
#pragma unroll
  for (int m = 0; m < 4; ++m) {
    const V fv = A::mul(yp.a[m], inv.a[m]);
    fo.a[m] = fv;
    mass = A::fmap(cols.a[m], fv, mass);
    rsum = A::addp(rsum, R.a[m]);
    if (m < real) mn = fminf(mn, A::f32(fv));
  }
  const Q4<V> fn = EARLY ? e_fn : A::ld4(fl.f + K);
  Q4<V> g;
#pragma unroll
  for (int m = 0; m < 4; ++m) {
    // the states read here (the oldest one included) are read before the slot is replaced
    const V h2 = EARLY ? e_h2.a[m] : at.nh >= 2 ? A::ld(at.h2, K + m) : fn.a[m];
    const V h3 = EARLY ? e_h3.a[m] : at.nh >= 3 ? A::ld(at.h3, K + m) : h2;
    const V h4 = EARLY ? e_h4.a[m] : at.nh >= 4 ? A::ld(at.h4, K + m) : h3;
    const V r = !fl.decay ? A::k(1.0) : EARLY ? e_r.a[m] : A::ld(fl.decay, K + m);
    g.a[m] = A::extrap(fo.a[m], fn.a[m], h2, h3, h4, at.nh, r);
  }
  A::st4(at.gout + K, g);
  A::st4(at.hw + K, fn);  // f^n into the oldest slot
  A::st4(fl.f + K, fo);
}
// polish_group for the cell of this lane (see resid_cell); real: the cell is in the grid
template <typename C, typename A>
__device__ __forceinline__ void polish_cell(const typename A::V* sm, int o, int P, const Coef<C>& co, long long K, bool on,
                                            const Fields& fl, const PolishAt& at, bool real, typename A::V& mass,
                                            typename A::V& rsum, float& mn) {
  using V = typename A::V;
  V R = A::k(0.0), fo = A::k(0.0), cols = A::k(0.0);
  if (on) {
    R = A::ld(fl.R, K);
    const V cw = CoefW<C, A>::cell(co, 0, K), ce = CoefW<C, A>::cell(co, 1, K);
    const V cs = CoefW<C, A>::cell(co, 2, K), cn = CoefW<C, A>::cell(co, 3, K);
    const V inv = A::ld(fl.invD, K), fn = A::ld(fl.f, K);
    cols = A::ld(fl.colsum, K);
    const V h2 = at.nh >= 2 ? A::ld(at.h2, K) : fn;
    const V h3 = at.nh >= 3 ? A::ld(at.h3, K) : h2;
    const V h4 = at.nh >= 4 ? A::ld(at.h4, K) : h3;
    const V r = fl.decay ? A::ld(fl.decay, K) : A::k(1.0);
    const V yp = A::fmap(cn, sm[o + P], A::fmap(cs, sm[o - P], A::fmap(ce, sm[o + 1], A::fmap(cw, sm[o - 1], R))));
    fo = A::mul(yp, inv);
    if (real) mn = fminf(mn, A::f32(fo));
    const V g = A::extrap(fo, fn, h2, h3, h4, at.nh, r);
    A::st(at.gout, K, g);
    A::st(at.hw, K, fn);
    A::st(fl.f, K, fo);
  }
  mass = group_chain<V>(A::k(0.0), [&](V a) { return A::fmap(cols, fo, a); });
  rsum = group_chain<V>(A::k(0.0), [&](V a) { return A::addp(a, R); });
}
// an instance's step is complete: sums of colsum f, R and the clamped count, and the minimum of f
__device__ __forceinline__ void after_polish(InstState& st, double mass, double rsum, double clamped, double gmin) {
  st.min_f = gmin;
  st.clamped = (long long)clamped;
  st.mass_drift = rsum != 0.0 ? div64(fabs(mass - rsum), fabs(rsum)) : 0.0;
  st.steps += 1;
  st.hslot = (st.hslot + 1) % kHist;
  st.nhist = min(st.nhist + 1, kOrder);
  if (!(gmin >= 0.0)) st.status = ST_NEGATIVE;
}

// y' = R + (I - A~) max(y, 0) >= 0 (R >= 0, fractions >= 0), f = y' / D; sums of colsum*f, R and the
// clamped count (carried in doubles above the segments); the minimum of f travels as a fourth
// quantity. Chunks [c0, c1) of the list (c1 < 0: all); a range must hold whole instances.
// It also forms the next solve's start g (extrap over the new f, f^n and up to kOrder - 1 earlier
// states from the history) into the idle y buffer, and moves f^n into the oldest history slot.
// 4 resident blocks per SM (64 registers; measured on the 4096-instance batch: 2.55 ms per
// launch against 2.81 ms with 3 blocks and 80 registers)
template <typename C, typename A, int CH>
__global__ void __launch_bounds__(kThreads, 4) k_polish(Common cm, Fields fl, Coef<C> co, int c0, int c1) {
  using V = typename A::V;
  using R = typename A::R;
  using Sums = ChunkSums<CH, 2, R>;
  count_launch(cm.ctl);
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ double s_part[2 * Sums::kParts];
  __shared__ float s_min[kThreads / 32], s_clamp[kThreads / 32];
  V* sm = reinterpret_cast<V*>(smraw);
  for_active_chunks(cm, [&](int b_) { return cm.inst[b_].enabled != 0; }, [&](int c) {
    const int b = cm.chunk_inst[c];
    InstState& st = cm.st[b];
    const InstDev& I = cm.inst[b];  // fields are read where they are needed: registers are short
    const PolishAt at = polish_at(fl, st.ycur, st.nhist, st.hslot, cm.hist_cap);
    const int P = I.pitch;
    const long long c0 = chunk_start<CH>(c, I);
    const long long c1 = min(c0 + (long long)CH, inst_end(I));
    const long long e0 = c0 - P;
    Sums sums{reinterpret_cast<R(*)[Sums::kParts]>(s_part)};
    float clamp = 0.0f;
    stage_rows<V>(sm, e0, (int)(c1 - c0) + 2 * P, [&](long long k) {
      Q4<V> v = A::ld4(at.y + k);
      const bool mine = k >= c0 && k < c1;
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        if (mine && A::lt0(v.a[m])) clamp += 1.0f;  // padding cells are 0
        v.a[m] = A::max0(v.a[m]);
      }
      return v;
    });
    __syncthreads();
    V mass = A::k(0.0), rsum = A::k(0.0);
    float mn = 3.0e38f;
    for_parts<CH>(I.seg, [&](int g) {
      const long long K = c0 + 4 * g;
      if (K < c1)
        polish_group<C, A, false>(sm, (int)(K - e0), P, co, K, fl, at, I.nx - (int)(K - I.base) % P, mass, rsum, mn);
    }, [&](int p) {
      const R w[2] = {mass, rsum};
      sums.put(p, w);
      mass = rsum = A::k(0.0);
    });
    // clamped cells (whole numbers) and the minimum: the chunk's, with the first of its segments
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
      clamp += __shfl_xor_sync(0xffffffffu, clamp, o);
    }
    if ((threadIdx.x & 31) == 0) {
      s_min[threadIdx.x >> 5] = mn;
      s_clamp[threadIdx.x >> 5] = clamp;
    }
    const int sl = (c - I.chunk0) * (CH / I.seg), left = I.nseg - sl;
    sums.template store<double>(cm.part, cm.pstride, I.seg0 + sl, left, I.seg);
    if ((int)threadIdx.x < min(CH / I.seg, left)) {
      float m = s_min[0], cl = s_clamp[0];
      for (int w = 1; w < kThreads / 32; ++w) {
        m = fminf(m, s_min[w]);
        cl += s_clamp[w];
      }
      cm.part[2 * (size_t)cm.pstride + I.seg0 + sl + threadIdx.x] = threadIdx.x == 0 ? (double)cl : 0.0;
      cm.part[3 * (size_t)cm.pstride + I.seg0 + sl + threadIdx.x] = (double)m;
    }
    double tot[3];
    if (chunk_finish<3, double>(st, PH_POLISH, I, cm.part, cm.pstride, tot)) {
      // the last block of the instance: minimum over its segments, by the whole block
      double m = 1.0e300;
      for (int k = threadIdx.x; k < I.nseg; k += blockDim.x)
        m = fmin(m, __ldcg(&cm.part[3 * (size_t)cm.pstride + I.seg0 + k]));
      __shared__ double s_gmin[kThreads / 32];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) m = fmin(m, __shfl_xor_sync(0xffffffffu, m, o));
      if ((threadIdx.x & 31) == 0) s_gmin[threadIdx.x >> 5] = m;
      __syncthreads();
      if (threadIdx.x == 0) {
        double gmin = s_gmin[0];
        for (int w = 1; w < (int)(blockDim.x >> 5); ++w) gmin = fmin(gmin, s_gmin[w]);
        after_polish(st, tot[0], tot[1], tot[2], gmin);
      }
    }
    __syncthreads();
  }, c0, c1);
}

}  // namespace sg
