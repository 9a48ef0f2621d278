// sayram_kernels.cuh -- sm_103a kernels of the Sayram-2D per-step hot path.
//
// Storage (all instances of a batch share one flat, padded, system-ordered layout):
//   instance b, cell (i, j) lives at index base_b + j*pitch_b + i, with pitch_b = nx_b rounded up
//   to a multiple of 4 and one zero row above (j = -1) and below (j = ny) every instance. The
//   reference's system order K = j*nx + i (Mesh.h:66-68) is kept inside each row. Every array
//   is zero in the padding and the pad rows and no kernel ever writes there, so the 5-point
//   stencil needs no bounds tests: out-of-domain neighbours contribute 0 * 0.
//
// Linear system (Jacobi-scaled, column form): with D = diag(M) the solver works on y = D f and
//   A~ = M D^{-1}, which has a unit diagonal.  Row L stores the four off-diagonal magnitudes
//   cw[L] = A_{W->L}/D_W (the west neighbour's outflow fraction through the face it shares with
//   L), ce, cs, cn likewise, so (A~ y)_L = y_L - (cw y_W + ce y_E + cs y_S + cn y_N).  Column K of
//   A~ holds -A_{K,sigma}/D_K, the fractions of K's outflow; they are >= 0 and sum to < 1 (M is a
//   column-diagonally-dominant M-matrix), which keeps FP32 storage well scaled and makes the
//   positivity polish y' = R + (I - A~) max(y, 0) a 1-norm contraction.
//
// Reductions are deterministic and have one order, whichever kernel runs them: the cells of an
// instance are cut into segments (seg_cells: 128 to 4096, by its size and the batch's chunk size),
// every segment's sum is a fixed tree over its cells, and an instance's total is a fixed tree over
// its segments (seg_total). After a pass of the per-pass kernels a small kernel with a block per
// instance forms the totals and updates the instance's scalars (k_after_*; for the polish the last
// block to finish the instance's chunks); no block waits on another. In k_team every block of an
// instance's team forms them, after the team's barrier.
#pragma once

#include <type_traits>

#include <cuda_runtime.h>
#include <float.h>
#include <stdint.h>

#include "dword.cuh"

namespace sg {

constexpr int kThreads = 256;  // threads per block of the streaming kernels
constexpr int kTX = 32;        // assembly tile width (alpha0, contiguous)
constexpr int kTY = 16;        // assembly tile height (log E)
constexpr int kAsmThreads = 256;
constexpr int kAsmGridPerSm = 96;  // k_assemble blocks launched per SM (grid-stride over tiles)
constexpr int kFieldThreads = 256;  // threads per block of the layout transforms
constexpr double kEps = DBL_EPSILON;  // gEPS, source/common.h:38

enum { XMIN = 0, XMAX = 1, YMIN = 2, YMAX = 3 };
enum { DIRICHLET = 0, ZEROFLUX = 1 };
enum { ST_OK = 0, ST_NOT_CONVERGED = 3, ST_NEGATIVE = 4 };
enum { PH_POLISH = 0, PH_COUNT = 2 };

// Per-instance constants.
struct InstDev {
  int nx, ny, pitch, enabled;
  int bc[4];
  long long base;  // index of cell (0,0) in the padded storage
  long long hoff;  // offset of the instance in the packed alpha-major host layout
  int chunk0, nchunks;
  int tile0, ntx, nty;
  int seg0, nseg;  // its reduction segments in the partial-sum arrays
  int seg, pad0;   // cells of one of them
  int xe, ye;     // offsets into the per-vertex-column / per-vertex-row arrays (nx+1 / ny+1)
  int dir[4];     // offsets into the Dirichlet vertex value array (-1 for zero-flux sides)
  double dt;
};

// Per-instance solver state (mutable, device resident).
struct InstState {
  // 8-byte scalars of the solve: IEEE doubles, or double words (bit patterns, see num/set_num) where
  // the sums behind them are double words -- the Krylov scalars in both FP32 modes, bb and rr64
  // in the double-word mode
  double rho, alpha, omega, beta;
  double rr, rr_target, bb, rr64;
  double mass_drift, min_f;
  long long clamped, steps;
  long long cum_iters, cum_refines;  // totals since creation (work accounting)
  int ycur, outer_active, inner_active;
  int restart, has_x;
  int iters;               // Krylov iterations of this solve finished so far
  int swapped;             // rh and x of the per-pass kernels have changed places (rh_of)
  int iters_total, refines, status;
  int nhist;               // earlier states held in the history buffers (extrapolated start)
  int lost;                // a barrier of k_team gave up: launches queued behind it leave the instance alone
  int hslot;               // history buffer holding f^(n-1); f^(n-2), ... are in the ones before it
  unsigned int rmax_bits;  // bits of max |R| over the instance (non-negative float; atomicMax order)
  unsigned int cnt[PH_COUNT];
};

// Batch-wide control words.
struct Ctl {
  int n_outer;   // instances still refining in this step
  int n_inner;   // instances inside an inner Krylov solve
  unsigned long long launches;  // kernel launches (block 0 of every kernel adds one)
  unsigned int kdone[8];        // blocks finished per kernel (graph-conditional updates)
  unsigned int outer_loops;     // residual evaluations run by the device-side loop this step
  unsigned int inner_loops;     // Krylov iterations run by the device-side loop this solve
};

// Four cells of a row. Aligned, so that one in shared memory moves by 16-byte accesses; with 4-byte
// ones, which the lanes' distance turned into 4- and 8-way bank conflicts, k_team's steps took 4502
// instead of 4165 us (eight, 1024 x 1024 in double-word) and 1250 instead of 1155 us (24 uneven
// instances). FP64 quads keep 8-byte accesses, which conflict no more than 16-byte ones (one 1024 x
// 1024 FP64 instance: 10482 against 10555 us).
template <typename T>
struct alignas(alignof(T) == 8 ? 8 : 16) Q4 {
  T a[4];
};

__device__ __forceinline__ Q4<float> ld4(const float* p) {
  const float4 v = *reinterpret_cast<const float4*>(p);
  return Q4<float>{{v.x, v.y, v.z, v.w}};
}
__device__ __forceinline__ Q4<double> ld4(const double* p) {
  const double2 u = reinterpret_cast<const double2*>(p)[0];
  const double2 w = reinterpret_cast<const double2*>(p)[1];
  return Q4<double>{{u.x, u.y, w.x, w.y}};
}
__device__ __forceinline__ void st4(float* p, const Q4<float>& q) {
  *reinterpret_cast<float4*>(p) = make_float4(q.a[0], q.a[1], q.a[2], q.a[3]);
}
__device__ __forceinline__ void st4(double* p, const Q4<double>& q) {
  reinterpret_cast<double2*>(p)[0] = make_double2(q.a[0], q.a[1]);
  reinterpret_cast<double2*>(p)[1] = make_double2(q.a[2], q.a[3]);
}

// Element i of a small pointer array inside a kernel parameter, chosen by selects: indexing the
// array with a run-time value makes every thread of every block copy the whole parameter to
// local memory first (with a grid of ~14,000 assembly blocks, ~300 MB of local stores a launch).
template <typename P>
__device__ __forceinline__ P sel2(P const (&a)[2], int i) {
  return i ? a[1] : a[0];
}
template <typename P>
__device__ __forceinline__ P sel3(P const (&a)[3], int i) {
  return i == 0 ? a[0] : (i == 1 ? a[1] : a[2]);
}

__device__ __forceinline__ void count_launch(Ctl* ctl) {
  if (blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(&ctl->launches, 1ull);
}

// ------------------------------------------------------------------------------ FP64 reciprocals
// 1/b and a/b in FP64 from an FP32 reciprocal r0 (Markstein, "Computation of elementary functions on
// the IBM RISC System/6000 processor", IBM J. Res. Dev. 34(1), 1990): with e = 1 - m r0, at most
// 2^-21, 1/m = r0 (1 + e + e^2 + ...) and what the first three terms leave, e^3, is 2^-10 of an ulp;
// one residual step rounds the quotient. Three (six) operations on the FP64 pipe, which takes 19
// cycles per SM for a warp's operation. Divisors that are zeros, subnormals, infinities, NaNs or of the
// outermost exponents take the plain operators, against which the results are otherwise within one unit in
// the last place.
__device__ __forceinline__ double rcp64(double b) {
  const int hi = __double2hiint(b), lo = __double2loint(b), e = (hi >> 20) & 0x7ff;
  if (e < 3 || e > 2042) return 1.0 / b;
  const double m = __hiloint2double((hi & 0x000fffff) | 0x3ff00000, lo);  // |b| = m 2^(e - 1023)
  // m to FP32 (truncated), its reciprocal and back, by moving the fields
  const float f = __uint_as_float(__funnelshift_l((unsigned)lo, (unsigned)((hi & 0x000fffff) | 0x07f00000), 3));
  const unsigned s = __float_as_uint(__fdividef(1.0f, f));
  const double r0 = __hiloint2double((int)((s >> 3) + 0x38000000u), (int)(s << 29));
  const double d = __fma_rn(-m, r0, 1.0);
  const double r = __fma_rn(r0, __fma_rn(d, d, d), r0);
  return __hiloint2double((__double2hiint(r) + (1023 - e) * 0x100000) | (hi & 0x80000000), __double2loint(r));
}
__device__ __forceinline__ double div64(double a, double b) {
  const int e = (__double2hiint(b) >> 20) & 0x7ff;
  if (e < 3 || e > 2042) return a / b;
  const double r = rcp64(b), q = __dmul_rn(a, r);
  const double t = __fma_rn(__fma_rn(-b, q, a), r, q);
  return (__double2hiint(q) & 0x7ff00000) == 0x7ff00000 ? q : t;
}

// ------------------------------------------------------------------------------ reductions
// Sums are carried in R: IEEE double, or a double word where the terms are FP32 (the FP64 pipe is
// far too slow for the trees: 2 lanes per SM and cycle).
__device__ __forceinline__ double radd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ dw radd(dw a, dw b) { return dw_add_same(a, b); }
__device__ __forceinline__ double rshfl(double a, int o) { return __shfl_xor_sync(0xffffffffu, a, o); }
__device__ __forceinline__ dw rshfl(dw a, int o) {
  return dw{__shfl_xor_sync(0xffffffffu, a.hi, o), __shfl_xor_sync(0xffffffffu, a.lo, o)};
}
__device__ __forceinline__ double rdbl(double a) { return a; }
__device__ __forceinline__ double rdbl(dw a) { return dw_to_double(a); }
template <typename R>
__device__ __forceinline__ R rfrom(double a);
template <>
__device__ __forceinline__ double rfrom<double>(double a) { return a; }
template <>
__device__ __forceinline__ dw rfrom<dw>(double a) { return dw_from_double(a); }
template <typename R>
__device__ __forceinline__ R rfrom(float a);
template <>
__device__ __forceinline__ double rfrom<double>(float a) { return (double)a; }
template <>
__device__ __forceinline__ dw rfrom<dw>(float a) { return dw{a, 0.0f}; }
template <typename S>
__device__ __forceinline__ S rconv(double a) { return (S)a; }
template <typename S>
__device__ __forceinline__ S rconv(dw a);
template <>
__device__ __forceinline__ dw rconv<dw>(dw a) { return a; }
template <>
__device__ __forceinline__ double rconv<double>(dw a) { return dw_to_double(a); }
// scalars of type R in 8-byte storage
template <typename R>
__device__ __forceinline__ R num(double s) {
  return *reinterpret_cast<const R*>(&s);
}
template <>
__device__ __forceinline__ dw num<dw>(double s) {
  return dw{__int_as_float(__double2loint(s)), __int_as_float(__double2hiint(s))};
}
__device__ __forceinline__ double stored(double a) { return a; }
__device__ __forceinline__ double stored(dw a) { return __hiloint2double(__float_as_int(a.lo), __float_as_int(a.hi)); }
__device__ __forceinline__ double rmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ dw rmul(dw a, dw b) { return dw_mul(a, b); }
__device__ __forceinline__ double rfma(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ dw rfma(dw a, dw b, dw c) { return dw_fma(a, b, c); }
__device__ __forceinline__ double rneg(double a) { return -a; }
__device__ __forceinline__ dw rneg(dw a) { return dw_neg(a); }
__device__ __forceinline__ double rdiv(double a, double b) { return div64(a, b); }
__device__ __forceinline__ dw rdiv(dw a, dw b) { return dw_div(a, b); }
__device__ __forceinline__ bool rgt(double a, double b) { return a > b; }
__device__ __forceinline__ bool rgt(dw a, dw b) { return a.hi > b.hi || (a.hi == b.hi && a.lo > b.lo); }
__device__ __forceinline__ double rhead(double a) { return a; }
__device__ __forceinline__ float rhead(dw a) { return a.hi; }
__device__ __forceinline__ double rto(double a, double) { return a; }  // a in the second argument's type
__device__ __forceinline__ dw rto(dw a, dw) { return a; }
__device__ __forceinline__ dw rto(double a, dw) { return dw_from_double(a); }
// the type a pass's sums are carried in: by the precision T of its terms
template <typename T>
struct RedOf;
template <>
struct RedOf<double> { using R = double; };
template <>
struct RedOf<float> { using R = dw; };

template <int NQ>
__host__ __device__ constexpr int red_pow2() { return NQ <= 1 ? 1 : NQ <= 2 ? 2 : NQ <= 4 ? 4 : 8; }

// Sums of NQ quantities over a warp, the transposed way: at each of the first steps a lane hands
// half of its quantities to its partner and keeps the other half, so NQ = 5 takes 9 additions
// instead of 25. Quantity q ends in the lanes with lane / (32 / P) = q (P: NQ rounded up to a power
// of two); the value returned is this lane's.
// In: the type of the terms. FP32 terms of double-word sums become double words in the first addition
// (2Sum is exact; the bits are those of adding them with zero low parts).
__device__ __forceinline__ float rshfl(float a, int o) { return __shfl_xor_sync(0xffffffffu, a, o); }
__device__ __forceinline__ dw radd_up(float a, float b, dw) { return two_sum(a, b); }
__device__ __forceinline__ dw radd_up(dw a, dw b, dw) { return dw_add_same(a, b); }
__device__ __forceinline__ double radd_up(double a, double b, double) { return __dadd_rn(a, b); }
template <int NQ, typename R, typename In>
__device__ __forceinline__ R warp_totals(const In (&in)[NQ]) {
  constexpr int P = red_pow2<NQ>();
  static_assert(P >= 2, "at least two quantities");
  const int lane = threadIdx.x & 31;
  R v[P / 2];
#pragma unroll
  for (int q = 0; q < P / 2; ++q) {
    const In lo = in[q], hi = q + P / 2 < NQ ? in[q + P / 2] : In{};
    const bool up = (lane & 16) != 0;
    v[q] = radd_up(up ? hi : lo, rshfl(up ? lo : hi, 16), R{});
  }
  int off = 8;
#pragma unroll
  for (int n = P / 2; n > 1; n >>= 1) {
    const bool up = (lane & off) != 0;
#pragma unroll
    for (int q = 0; q < n / 2; ++q) {
      const R send = up ? v[q] : v[q + n / 2];
      const R keep = up ? v[q + n / 2] : v[q];
      v[q] = radd(keep, rshfl(send, off));
    }
    off >>= 1;
  }
#pragma unroll
  for (; off > 0; off >>= 1) v[0] = radd(v[0], rshfl(v[0], off));
  return v[0];
}
// the quantity this lane's warp_totals value belongs to, and whether it is the lane that hands it on
template <int NQ>
__device__ __forceinline__ int red_q() { return (threadIdx.x & 31) / (32 / red_pow2<NQ>()); }
template <int NQ>
__device__ __forceinline__ bool red_writes() {
  return (threadIdx.x & (32 / red_pow2<NQ>() - 1)) == 0 && red_q<NQ>() < NQ;
}

// Cells of a reduction segment. 4096 in chunks of 4096, so that a thread sums four groups before the
// warp's tree; else the fewest of 128 (one warp's 4-cell groups), 256, 512 or 1024 that leave at most
// 512 segments: short segments let a small instance be spread over many SMs, and the totals are
// one more chain over the segments in every pass (at 1577 segments of 128 cells, 389 x 517, that
// took 3.1 us a pass, at 394 of 512 1 us).
__host__ __device__ inline int seg_cells(int chunk, long long cells) {
  if (chunk == 4096) return 4096;
  int s = 128;
  while (s < 1024 && cells > 512LL * s) s *= 2;
  return s;
}

// Cells whose terms one warp adds up before its tree: two 4-cell groups per lane in the longest
// segments, which halves the trees where they are most of a pass's instructions.
__host__ __device__ inline int part_cells(int seg) { return seg == 1024 ? 256 : 128; }

// n = 1, 2, 4 or 8 warp sums -> one segment sum, as a fixed tree
template <typename R>
__device__ __forceinline__ R tree(const R* a, int n) {
  if (n == 1) return a[0];
  R x = radd(a[0], a[1]);
  if (n >= 4) x = radd(x, radd(a[2], a[3]));
  if (n == 8) x = radd(x, radd(radd(a[4], a[5]), radd(a[6], a[7])));
  return x;
}

// The totals of NQ quantities over nseg segment sums part[q * stride + seg0 ...]: task (q, h) is one
// warp adding every eighth run of 32 segments, lane by lane, then its tree; a total is the tree over
// its eight tasks. In sm[0 .. NQ) for the first warp after the call (sm holds 8 * NQ entries). NW:
// warps of the block; a warp issues the loads of all its tasks before it adds. Bound by latency: L2's
// and the additions'. Steps of a 33 x 32 FP64 instance 1135 -> 1070 us (twenty), of a 90 x 90 one 863 ->
// 835 us with the short form for up to 256 segments (in double-word it gains nothing there, and its
// code costs larger instances 1 %), of a 1024 x 1024 double-word one 4173 -> 4142 us with trees side by
// side, -> 4080 us with four runs on their way at a time above 512 segments (below, where two hold
// all, four cost 4 % of a 389 x 517 instance's steps: additions of zero).
template <int NQ, int NW, typename R>
__device__ __forceinline__ void seg_total(const R* part, long long stride, int seg0, int nseg, R* sm) {
  constexpr int G = NW / 8, NT = (NQ + G - 1) / G;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const double* src = reinterpret_cast<const double*>(part) + seg0;
  R a[NT];
  constexpr bool DW = sizeof(rhead(R{})) == 4;
  if (!DW && nseg <= 256) {  // one run each, as it is: spares two additions on the FP64 pipe
#pragma unroll
    for (int t = 0; t < NT; ++t) {
      const int q = (warp >> 3) + G * t, s = ((warp - q) & 7) * 32 + lane;
      a[t] = q < NQ && s < nseg ? num<R>(__ldcg(src + (size_t)q * stride + s)) : rfrom<R>(0.0f);
    }
  } else {
#pragma unroll
    for (int t = 0; t < NT; ++t) a[t] = rfrom<R>(0.0f);
    // one round of the segments from r0 on: NL runs of each task
    const auto round = [&](int r0, auto nl) {
      constexpr int NL = decltype(nl)::value;
      double w[NT][NL];
#pragma unroll
      for (int t = 0; t < NT; ++t) {
        const int q = (warp >> 3) + G * t;
        const int h = (warp - q) & 7;  // the first tasks of different quantities fall on different warps
#pragma unroll
        for (int k = 0; k < NL; ++k) {
          const int s = r0 + lane + h * 32 + 256 * k;
          w[t][k] = q < NQ && s < nseg ? __ldcg(src + (size_t)q * stride + s) : 0.0;
        }
      }
#pragma unroll
      for (int t = 0; t < NT; ++t)
#pragma unroll
        for (int k = 0; k < NL; ++k) a[t] = radd(a[t], num<R>(w[t][k]));
    };
    int r0 = 0;
    if (NW > 8) {
      if (__builtin_expect(nseg > 512, 0)) {
#pragma unroll 1
        for (; r0 < nseg; r0 += 1024) round(r0, std::integral_constant<int, 4>{});
      } else {
        round(0, std::integral_constant<int, 2>{});
      }
    } else {
#pragma unroll 1
      for (; r0 < nseg; r0 += 256) round(r0, std::integral_constant<int, 1>{});
    }
  }
  if constexpr (DW) {
    // the trees of a warp's tasks side by side
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int t = 0; t < NT; ++t) a[t] = radd(a[t], rshfl(a[t], o));
#pragma unroll
    for (int t = 0; t < NT; ++t) {
      const int q = (warp >> 3) + G * t, h = (warp - q) & 7;
      if (q < NQ && lane == 0) sm[8 * q + h] = a[t];
    }
  } else {  // one after another where there is something to add: the FP64 pipe is what they wait for
#pragma unroll
    for (int t = 0; t < NT; ++t) {
      const int q = (warp >> 3) + G * t, h = (warp - q) & 7;
      if (q >= NQ) break;
      if (h * 32 < nseg) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) a[t] = radd(a[t], rshfl(a[t], o));
      }
      if (lane == 0) sm[8 * q + h] = a[t];
    }
  }
  __syncthreads();
  if (warp == 0) {
    R t = rfrom<R>(0.0f);
    if (lane < NQ) t = tree(sm + 8 * lane, nseg > 32 ? 8 : 1);
    __syncwarp();
    if (lane < NQ) sm[lane] = t;
    __syncwarp();
  }
}

// Segment-partial bookkeeping of the per-pass kernels: after the block has stored the segment sums
// of one chunk, it learns whether it is the last of the instance's chunks for this phase; if so
// the totals are returned in tot (valid in thread 0) and the phase counter is reset.
template <int NQ, typename R>
__device__ __forceinline__ bool chunk_finish(InstState& st, int phase, const InstDev& I, const R* part,
                                             long long stride, R (&tot)[NQ]) {
  __shared__ int s_last;
  __shared__ double s_tot[8 * NQ];
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    const unsigned prev = atomicAdd(&st.cnt[phase], 1u);
    s_last = (prev == (unsigned)(I.nchunks - 1));
  }
  __syncthreads();
  if (!s_last) return false;
  __threadfence();
  R* sm = reinterpret_cast<R*>(s_tot);
  seg_total<NQ, kThreads / 32, R>(part, stride, I.seg0, I.nseg, sm);
  if (threadIdx.x == 0) {
#pragma unroll
    for (int q = 0; q < NQ; ++q) tot[q] = sm[q];
    st.cnt[phase] = 0;
  }
  return true;
}

// One block's sums of one chunk: put() closes a part (a warp's sum; in chunks of 4096 cells a warp's
// share of the whole chunk), store() writes the chunk's segment sums.
template <int CH, int NQ, typename R>
struct ChunkSums {
  static constexpr bool kWhole = CH == 4096;              // one segment per chunk
  static constexpr int kParts = kWhole ? 8 : CH / 128;    // most parts of a chunk
  R (*sm)[kParts];  // [NQ][kParts] in shared memory
  template <typename In>
  __device__ __forceinline__ void put(int p, const In (&v)[NQ]) {
    const R t = warp_totals<NQ, R>(v);
    if (red_writes<NQ>()) sm[red_q<NQ>()][p] = t;
  }
  // seg: the chunk's first segment in the partials; nseg: how many of them the instance has from there
  // on; cells: of a segment; S: what a segment's sum is stored as (R, or double)
  template <typename S = R>
  __device__ __forceinline__ void store(S* part, long long stride, int seg, int nseg, int cells) {
    __syncthreads();
    if (kWhole) {
      if (threadIdx.x < NQ) part[(size_t)threadIdx.x * stride + seg] = rconv<S>(tree(sm[threadIdx.x], 8));
      return;
    }
    const int pp = cells / part_cells(cells), ns = min(CH / cells, nseg);
    for (int k = threadIdx.x; k < NQ * kParts; k += blockDim.x) {
      const int q = k / kParts, s = k % kParts;
      if (s < ns) part[(size_t)q * stride + seg + s] = rconv<S>(tree(&sm[q][s * pp], pp));
    }
  }
};

// Runs group(g) for the 4-cell groups g of a chunk that this thread owns, part by part, and put(p) after
// the last group of part p.
template <int CH, typename F, typename P>
__device__ __forceinline__ void for_parts(int seg, F&& group, P&& put) {
  if (CH == 4096) {
#pragma unroll 1
    for (int k = 0; k < CH / (4 * kThreads); ++k) group((int)threadIdx.x + k * kThreads);
    put((int)threadIdx.x >> 5);
  } else {
    const int part = part_cells(seg);
#pragma unroll 1
    for (int p = threadIdx.x >> 5; p < CH / part; p += kThreads / 32) {
#pragma unroll 1
      for (int k = 0; k < part / 4; k += 32) group(p * (part / 4) + k + (int)(threadIdx.x & 31));
      put(p);
    }
  }
}

}  // namespace sg
