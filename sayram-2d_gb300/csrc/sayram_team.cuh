// sayram_team.cuh -- k_team: whole steps of a small batch in one cooperative launch.
//
// Every instance is advanced by a team of blocks (one block per SM, in all at most the chip), each
// owning a run of the instance's reduction segments. A team runs assembly, refinement loop and
// polish of one step after another by itself: its blocks meet at a barrier of their own after
// each pass, and instances do not wait for one another. What such batches spend their time on
// in separate kernels is not arithmetic but launches, the reload of every vector in every pass and
// the ramp of each; here a share's Krylov vectors stay in shared memory and its coefficients in
// registers for the whole solve, and a pass only exchanges the boundary rows of its product and
// the sums (through L2).
//
// The arithmetic, the reduction segments and the order of the totals are those of the per-pass
// kernels (sayram_solve.cuh), so both give the same bits.
#pragma once

#include "sayram_team.h"

namespace sg {

// Meets the team's other blocks: counts this block in and waits until nb blocks have arrived that
// often. The wait is bounded (a launch is cooperative, so the others are running: milliseconds at
// most); a block that gives up records it and leaves, and so do the others of its team in their turn; the
// launches queued behind leave the instance alone. The block
// barriers around one thread's release and acquire order every thread's accesses. Measured with 512
// bytes written before and read after it by every block: 1.42 us at 9 to 152 blocks; further
// fences around the two cost 0.27 us, and a flag per block that every block polls 2.98 us at 152.
constexpr int kFineParts = 4;  // most parts of a share that takes a cell per lane
struct TeamBar {
  unsigned* cnt;
  unsigned target;
  int nb;
};
__device__ __forceinline__ bool team_sync(TeamBar& tb, const TeamArgs& ta, InstState* st) {
  __shared__ int s_ok;
  __syncthreads();
  if (tb.nb == 1) return true;
  if (threadIdx.x == 0) {
    tb.target += (unsigned)tb.nb;
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(tb.cnt) : "memory");
    unsigned v;
    int ok = 0;
    for (int k = 0; k < ta.polls; ++k) {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(tb.cnt) : "memory");
      if ((int)(v - tb.target) >= 0) {
        ok = 1;
        break;
      }
    }
    if (!ok) {
      ta.stat[TEAM_GAVE_UP] = 1;
      atomicExch(&st->lost, 1);
    }
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}
// after a block's last barrier: the last one to leave clears the counters for the next launch
__device__ __forceinline__ void team_leave(const TeamBar& tb) {
  if (tb.nb == 1 || threadIdx.x != 0) return;
  if (atomicAdd(tb.cnt + 1, 1u) == (unsigned)tb.nb - 1u) {
    tb.cnt[0] = 0u;
    tb.cnt[1] = 0u;
    __threadfence();
  }
}

__device__ __forceinline__ Q4<float> ld4cg(const float* p) {
  const float4 v = __ldcg(reinterpret_cast<const float4*>(p));
  return Q4<float>{{v.x, v.y, v.z, v.w}};
}
__device__ __forceinline__ Q4<double> ld4cg(const double* p) {
  const double2 u = __ldcg(reinterpret_cast<const double2*>(p));
  const double2 w = __ldcg(reinterpret_cast<const double2*>(p) + 1);
  return Q4<double>{{u.x, u.y, w.x, w.y}};
}

// a plain struct of 4-byte words, copied by the block's first threads
template <typename X>
__device__ __forceinline__ void copy_words(X& to, const X& from) {
  static_assert(sizeof(X) % 4 == 0 && sizeof(X) / 4 <= kTeamThreads, "one word per thread");
  if (threadIdx.x < sizeof(X) / 4)
    reinterpret_cast<unsigned*>(&to)[threadIdx.x] = reinterpret_cast<const unsigned*>(&from)[threadIdx.x];
}

// Warp sums of a share -> segment sums in the global partials. parts[q][p]: the sum over part p.
template <int NQ, typename R, typename S>
__device__ __forceinline__ void team_store(const R* parts, int np, int seg, int nseg, S* part, long long stride,
                                           int at) {
  __syncthreads();
  const int pp = seg / part_cells(seg);
  for (int k = threadIdx.x; k < NQ * nseg; k += kTeamThreads) {
    const int q = k / nseg, s = k - q * nseg;
    part[(size_t)q * stride + at + s] = rconv<S>(tree(&parts[q * np + pp * s], pp));
  }
}

// G: 4-cell groups per thread whose coefficients stay in registers with the Krylov vectors in
// shared memory (the on-chip form); 0: any number of groups, with x, t, v and the shadow residual in
// global memory (an instance too large for the chip: one 1024 x 1024 FP64 instance).
template <typename T, typename C, typename A, int G>
__global__ void __launch_bounds__(kTeamThreads, 1) k_team(Common cm, Geo geo, Fields fl, Coef<C> cf, Coef<T> ck,
                                                           Kry<T> kr, TeamArgs ta) {
  using V = typename A::V;
  using R = typename A::R;             // sums of the residual and polish
  using RK = typename RedOf<T>::R;     // sums of the Krylov passes
  constexpr bool ON = G > 0;
  constexpr int GN = ON ? G : 1;
  count_launch(cm.ctl);
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ InstState S;
  __shared__ InstDev sI;
  __shared__ double s_tot[8 * kPartQ];
  __shared__ float s_w[kTeamThreads / 32];
  __shared__ int s_go;
  __shared__ double s_gs[3 * kFineParts * 32];  // group sums of a share handled cell by cell
  const int tid = threadIdx.x, warp = tid >> 5;
  const int np = ta.own_cap / 128;  // warp sums of the largest share
  const size_t ext_cap = (size_t)ta.own_cap + 2 * (size_t)ta.pmax;
  double* const parts = reinterpret_cast<double*>(smraw);
  unsigned char* const mem = smraw + (((size_t)kPartQ * np * 8 + 15) & ~(size_t)15);

  const int e_end = ta.first ? ta.first[blockIdx.x + 1] : (int)blockIdx.x + 1;
  for (int e = ta.first ? ta.first[blockIdx.x] : (int)blockIdx.x; e < e_end; ++e) {
    const TeamShare sh = ta.share[e];
    __syncthreads();
    copy_words(sI, cm.inst[sh.inst]);
    copy_words(S, cm.st[sh.inst]);
    __syncthreads();
    const InstDev& I = sI;
    const int P = I.pitch, SEG = I.seg;
    const long long c0 = I.base + (long long)sh.s0 * SEG;
    const long long c1 = min(I.base + (long long)sh.s1 * SEG, inst_end(I));
    const int own = sh.s1 > sh.s0 ? (int)(c1 - c0) : 0, ext = own > 0 ? own + 2 * P : 0;
    const int nseg = sh.s1 - sh.s0, seg0 = I.seg0 + sh.s0;
    // warps take parts in turn; a part is part/128 groups of every lane
    const int part_c = part_cells(SEG), pend = nseg * (SEG / part_c), lane = tid & 31;
    const bool two = part_c == 256;
    // a cell per lane instead of four (resid_cell, polish_cell) where that leaves no SM sub-partition more
    // warps than it can hide: FP64 work is bound by the pipe, which a warp's operation holds for 64
    // cycles, so it only gains while some sub-partitions would have had nothing
    const bool fine = ON && !two && pend <= (sizeof(typename A::Acc) == 8 ? 2 : kFineParts);
    const long long e0 = c0 - P;
    TeamBar bar{ta.bar + (size_t)sh.inst * kTeamBarStride, 0u, sh.nb};
    float* const tmax = ta.tmax + (blockIdx.x - sh.rank);
    // shared memory: r and p with halos, then (on chip) v and x with halos, t and the shadow residual; the
    // staged 8-byte solution lies over p (and v). In the other form the halos of v and x only; in FP32
    // v has the room that the staged solution needs beyond p.
    T* const sr = reinterpret_cast<T*>(mem);
    T* const sp = sr + ext_cap;
    V* const sv = reinterpret_cast<V*>(sp);
    constexpr bool VON = ON || sizeof(T) == 4;
    T* const sv_ = VON ? sp + ext_cap : reinterpret_cast<T*>(sv + ext_cap);  // v: own + halo, else halo
    T* const sx = VON ? sv_ + ext_cap : sv_ + 2 * ta.pmax;
    T* const st_ = sx + ext_cap;               // t of the share (on chip)
    T* const srh = st_ + ta.own_cap;           // shadow residual of the share (on chip)
    // a cell of the share that a neighbouring share reads
    const auto edge = [&](int l) { return l < P || l >= own - P; };
    // x, v of extended index l (0 .. ext): in shared memory, or own cells in global memory
    const auto at_x = [&](int l) -> T* {
      if (ON) return sx + l;
      return l < P ? sx + l : l < P + own ? kr.x + e0 + l : sx + (l - own);
    };
    const auto at_v = [&](int l) -> T* {
      if (VON) return sv_ + l;
      return l < P ? sv_ + l : l < P + own ? kr.v[0] + e0 + l : sv_ + (l - own);
    };

    // the sums of a pass, in turn in one of two sets: a block may write the next pass's while another
    // still reads this one's
    int flip = 0;
    const auto part = [&]() { return cm.part + (size_t)flip * kPartQ * cm.pstride; };
    bool ok = S.lost == 0;
    for (int step = 0; ok && step < ta.nsteps; ++step) {
      // ---------------------------------------------------------------- assembly
      if (ta.phases & TEAM_ASSEMBLE) {
        // a tile's steps are short between its barriers: four tiles at a time, by a quarter of the block each.
        // A block with one or two of them gives all its threads to those, as far as a tile has faces for
        // them (33 cells across need 99 to 1089 threads). Microseconds a step before and after: 33 x 32
        // FP64 22.2 / 21.4, 90 x 90 FP64 37.6 / 36.8, 256 x 256 double-word 42.4 / 34.5 (FP64 78.4 / 70.3),
        // 24 instances of up to 64 x 64 39 / 32; with more tiles the number of threads as a variable
        // costs a little, 400 x 400 57.2 / 58.0.
        const int nty = (I.ny + sh.ty - 1) / sh.ty, nt = I.ntx * nty;
        const int tiles = (nt + sh.nb - 1) / sh.nb, faces = (min(kTX, I.nx) + 1) * (2 * sh.ty + 1);
        int QT = kTeamThreads / (tiles > 2 ? kTeamParts : tiles);
        while (QT > kTeamThreads / kTeamParts && QT >= 2 * faces) QT /= 2;
        const int parts_ = kTeamThreads / QT, part_ = tid / QT;
        AsmTile<A>& tile = reinterpret_cast<AsmTile<A>*>(mem)[part_];
        const bool has_g = S.nhist > 0;
        float rmax = 0.0f;
        for (int t = sh.rank + part_ * sh.nb; t < nt; t += sh.nb * parts_) {
          rmax = fmaxf(rmax, asm_tile<C, A>(tile, cm, geo, fl, cf, I, (t % I.ntx) * kTX, (t / I.ntx) * sh.ty, sh.ty,
                                            has_g, S.ycur, tid % QT, QT, 1 + part_));
          tile_sync(1 + part_, QT);
        }
        if ((tid & 31) == 0) s_w[warp] = rmax;
        __syncthreads();
        if (tid == 0) {
#pragma unroll
          for (int w = 1; w < kTeamThreads / 32; ++w) rmax = fmaxf(rmax, s_w[w]);
          tmax[sh.rank] = rmax;
        }
        if (!(ok = team_sync(bar, ta, cm.st + sh.inst))) break;
        float m = 0.0f;
        for (int k = tid; k < sh.nb; k += kTeamThreads) m = fmaxf(m, __ldcg(tmax + k));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        if ((tid & 31) == 0) s_w[warp] = m;
        __syncthreads();
        if (tid == 0) {
#pragma unroll
          for (int w = 1; w < kTeamThreads / 32; ++w) m = fmaxf(m, s_w[w]);
          S.rmax_bits = m > 0.0f ? __float_as_uint(m) : 0u;
        }
        __syncthreads();
      }
      // ---------------------------------------------------------------- refinement loop
      if (ta.phases & TEAM_SOLVE) {
        const float sc = rhs_scale(S.rmax_bits), isc = 1.0f / sc;
        __syncthreads();
        if (tid == 0) {
          S.restart = 0;
          S.has_x = 0;
          S.iters = 0;
          S.iters_total = 0;
          S.refines = 0;
          S.clamped = 0;
          S.rmax_bits = 0u;  // where a kernel of its own assembles, it collects the next step's maximum here
        }
        __syncthreads();
        for (;;) {
          const double* yin = sel2(fl.y64, S.ycur);
          double* yout = sel2(fl.y64, S.ycur ^ 1);
          const bool hx = S.has_x != 0;
          for (int l = 4 * tid; l < ext; l += 4 * kTeamThreads) {
            Q4<V> y = A::ld4(yin + e0 + l);
            if (hx) {
              const Q4<T> x = ld4(at_x(l));
#pragma unroll
              for (int m = 0; m < 4; ++m) y.a[m] = A::template add_scaled<T>(y.a[m], x.a[m], isc);
            }
            *reinterpret_cast<Q4<V>*>(sv + l) = y;
          }
          __syncthreads();
          if (fine) {
            const int p = warp >> 2, l = 4 * 8 * warp + lane;  // part and cell
            if (p < pend) {
              V yc;
              T r;
              typename A::Acc q0, q1;
              T q2;
              resid_cell<T, C, A>(sv, P + l, P, cf, c0 + l, l < own, fl.R, sc, cm.precond, S.refines == 0, yc, r, q0,
                                  q1, q2);
              if (l < own) {
                if (hx) A::st(yout, c0 + l, yc);
                sr[P + l] = r;
                if (ON) srh[l] = r;
                if (!ON || edge(l)) kr.rh[c0 + l] = r;
              }
              if ((lane & 3) == 0) {
                typename A::Acc* gs = reinterpret_cast<typename A::Acc*>(s_gs) + 3 * (l >> 2);
                gs[0] = q0;
                gs[1] = q1;
                gs[2] = q2;
              }
            }
            __syncthreads();
            if (warp < pend) {
              const typename A::Acc* gs = reinterpret_cast<const typename A::Acc*>(s_gs) + 3 * (32 * warp + lane);
              const typename A::Acc w[3] = {gs[0], gs[1], gs[2]};
              const R t = warp_totals<3, R>(w);
              if (red_writes<3>()) reinterpret_cast<R*>(parts)[red_q<3>() * np + warp] = t;
            }
          } else {
            for (int p = warp; p < pend; p += kTeamThreads / 32) {
              typename A::Acc q0 = 0, q1 = 0;
              T q2 = (T)0;
              for (int k = 0; k < part_c; k += 128) {
                const int l = p * part_c + k + 4 * lane;
                if (l >= own) continue;
                Q4<V> yc;
                Q4<T> r;
                resid_group<T, C, A>(sv, P + l, P, cf, c0 + l, fl.R, sc, cm.precond, S.refines == 0, yc, r, q0, q1, q2);
                if (hx) A::st4(yout + c0 + l, yc);
                st4(sr + P + l, r);
                if (ON) st4(srh + l, r);
                if (!ON || edge(l)) st4(kr.rh + c0 + l, r);
              }
              const typename A::Acc w[3] = {q0, q1, q2};
              const R t = warp_totals<3, R>(w);
              if (red_writes<3>()) reinterpret_cast<R*>(parts)[red_q<3>() * np + p] = t;
            }
          }
          team_store<3, R, R>(reinterpret_cast<const R*>(parts), np, SEG, nseg, reinterpret_cast<R*>(part()),
                              cm.pstride, seg0);
          if (!(ok = team_sync(bar, ta, cm.st + sh.inst))) break;
          seg_total<3, kTeamThreads / 32, R>(reinterpret_cast<const R*>(part()), cm.pstride, I.seg0, I.nseg,
                          reinterpret_cast<R*>(s_tot));
          flip ^= 1;
          if (tid == 0) {
            const R* tt = reinterpret_cast<const R*>(s_tot);
            const R tot[3] = {tt[0], tt[1], tt[2]};
            s_go = after_resid<RK, R>(S, tot, ta.tol, ta.inner_tol, ta.max_refine, cm.precond);
          }
          __syncthreads();
          if (!s_go) break;
          // -------------------------------------------------------------- Krylov solve
          // this thread's k-th group: its first cell in the share
          const auto cell_of = [&](int k) {
            return two ? (warp + kTeamThreads / 32 * (k >> 1)) * 256 + (k & 1) * 128 + 4 * lane
                       : (warp + kTeamThreads / 32 * k) * 128 + 4 * lane;
          };
          Row<T> row[GN];
          if (ON) {
#pragma unroll
            for (int k = 0; k < GN; ++k) {
              const int l = cell_of(k);
              if (l < own) row[k] = row_of<T>(ck, c0 + l);
            }
          }
          // p = r = r^; the neighbours' rows of r
          for (int l = 4 * tid; l < ext; l += 4 * kTeamThreads) {
            Q4<T> r;
            if (l < P || l >= P + own) {
              r = ld4cg(kr.rh + e0 + l);
              st4(sr + l, r);
            } else {
              r = ld4(sr + l);
            }
            st4(sp + l, r);
          }
          for (;;) {
            const int it = S.iters;
            const bool rs = S.restart != 0;
            if (it > 0) {  // update by the previous iteration's products; sr holds s
              const T alpha = rhead(num<RK>(S.alpha)), beta = rhead(num<RK>(S.beta)),
                      omega = rhead(num<RK>(S.omega));
              for (int l = 4 * tid; l < ext; l += 4 * kTeamThreads) {
                const bool halo = l < P || l >= P + own;
                const Q4<T> t = halo ? ld4cg(kr.t + e0 + l) : ON ? ld4(st_ + (l - P)) : ld4(kr.t + e0 + l);
                const Q4<T> s = ld4(sr + l), v = ld4(at_v(l));
                Q4<T> p = ld4(sp + l), q, x{{(T)0, (T)0, (T)0, (T)0}};
                if (it > 1) x = ld4(at_x(l));
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                  q.a[m] = fmaT(-omega, t.a[m], s.a[m]);
                  x.a[m] = fmaT(alpha, p.a[m], fmaT(omega, s.a[m], x.a[m]));
                  p.a[m] = rs ? q.a[m] : fmaT(beta, fmaT(-omega, v.a[m], p.a[m]), q.a[m]);
                }
                st4(sr + l, q);
                st4(sp + l, p);
                st4(at_x(l), x);
                if (rs && !halo) st4(ON ? srh + (l - P) : kr.rh + e0 + l, q);
              }
            }
            __syncthreads();
            // v = B^-1 A~ p
            const auto product_v = [&](int l, const Row<T>& w, T& q0, T& q1) {
              const Q4<T> v = product<T>(sp, P + l, P, w, cm.precond);
              st4(at_v(P + l), v);
              if (VON && edge(l)) st4(kr.v[0] + c0 + l, v);
              const Q4<T> rh = rs ? ld4(sp + P + l) : ON ? ld4(srh + l) : ld4(kr.rh + c0 + l);
              q0 = dot4<T>(rh, v, q0);
              if (rs && it > 0) q1 = dot4<T>(rh, rh, q1);
            };
            const auto put2 = [&](int p, T q0, T q1) {
              const T w[2] = {q0, q1};
              const RK t = warp_totals<2, RK>(w);
              if (red_writes<2>()) reinterpret_cast<RK*>(parts)[red_q<2>() * np + p] = t;
            };
            if (ON) {
              T q0 = (T)0, q1 = (T)0;
#pragma unroll
              for (int k = 0; k < GN; ++k) {
                const int l = cell_of(k), p = warp + kTeamThreads / 32 * (two ? k >> 1 : k);
                if (p >= pend) break;
                if (l < own) product_v(l, row[k], q0, q1);
                if (two && !(k & 1)) continue;
                put2(p, q0, q1);
                q0 = q1 = (T)0;
              }
            } else {
              for (int p = warp; p < pend; p += kTeamThreads / 32) {
                T q0 = (T)0, q1 = (T)0;
                for (int k = 0; k < part_c; k += 128) {
                  const int l = p * part_c + k + 4 * lane;
                  if (l >= own) continue;
                  product_v(l, row_of<T>(ck, c0 + l), q0, q1);
                }
                put2(p, q0, q1);
              }
            }
            team_store<2, RK, RK>(reinterpret_cast<const RK*>(parts), np, SEG, nseg, reinterpret_cast<RK*>(part()),
                                  cm.pstride, seg0);
            if (!(ok = team_sync(bar, ta, cm.st + sh.inst))) break;
            seg_total<2, kTeamThreads / 32, RK>(reinterpret_cast<const RK*>(part()), cm.pstride, I.seg0, I.nseg,
                             reinterpret_cast<RK*>(s_tot));
            flip ^= 1;
            if (tid == 0) {
              const RK* tt = reinterpret_cast<const RK*>(s_tot);
              const RK tot[2] = {tt[0], tt[1]};
              after_v(S, tot);
            }
            __syncthreads();
            // s = r - alpha v over the share and its halo
            {
              const T alpha = rhead(num<RK>(S.alpha));
              for (int l = 4 * tid; l < ext; l += 4 * kTeamThreads) {
                Q4<T> v, s = ld4(sr + l);
                if (l < P || l >= P + own) {
                  v = ld4cg(kr.v[0] + e0 + l);
                  st4(at_v(l), v);
                } else {
                  v = ld4(at_v(l));
                }
#pragma unroll
                for (int m = 0; m < 4; ++m) s.a[m] = fmaT(-alpha, v.a[m], s.a[m]);
                st4(sr + l, s);
              }
            }
            __syncthreads();
            // t = B^-1 A~ s
            const auto product_t = [&](int l, const Row<T>& w, T (&q)[5]) {
              const Q4<T> t = product<T>(sr, P + l, P, w, cm.precond);
              if (ON) st4(st_ + l, t);
              if (!ON || edge(l)) st4(kr.t + c0 + l, t);
              const Q4<T> s = ld4(sr + P + l), rh = ON ? ld4(srh + l) : ld4(kr.rh + c0 + l);
              q[0] = dot4<T>(t, s, q[0]);
              q[1] = dot4<T>(t, t, q[1]);
              q[2] = dot4<T>(s, s, q[2]);
              q[3] = dot4<T>(rh, s, q[3]);
              q[4] = dot4<T>(rh, t, q[4]);
            };
            const auto put5 = [&](int p, const T (&q)[5]) {
              const RK t = warp_totals<5, RK>(q);
              if (red_writes<5>()) reinterpret_cast<RK*>(parts)[red_q<5>() * np + p] = t;
            };
            if (ON) {
              T q[5] = {(T)0, (T)0, (T)0, (T)0, (T)0};
#pragma unroll
              for (int k = 0; k < GN; ++k) {
                const int l = cell_of(k), p = warp + kTeamThreads / 32 * (two ? k >> 1 : k);
                if (p >= pend) break;
                if (l < own) product_t(l, row[k], q);
                if (two && !(k & 1)) continue;
                put5(p, q);
#pragma unroll
                for (int m = 0; m < 5; ++m) q[m] = (T)0;
              }
            } else {
              for (int p = warp; p < pend; p += kTeamThreads / 32) {
                T q[5] = {(T)0, (T)0, (T)0, (T)0, (T)0};
                for (int k = 0; k < part_c; k += 128) {
                  const int l = p * part_c + k + 4 * lane;
                  if (l >= own) continue;
                  product_t(l, row_of<T>(ck, c0 + l), q);
                }
                put5(p, q);
              }
            }
            team_store<5, RK, RK>(reinterpret_cast<const RK*>(parts), np, SEG, nseg, reinterpret_cast<RK*>(part()),
                                  cm.pstride, seg0);
            if (!(ok = team_sync(bar, ta, cm.st + sh.inst))) break;
            seg_total<5, kTeamThreads / 32, RK>(reinterpret_cast<const RK*>(part()), cm.pstride, I.seg0, I.nseg,
                             reinterpret_cast<RK*>(s_tot));
            flip ^= 1;
            if (tid == 0) {
              const RK* tt = reinterpret_cast<const RK*>(s_tot);
              RK tot[5];
#pragma unroll
              for (int k = 0; k < 5; ++k) tot[k] = tt[k];
              s_go = !after_t(S, tot, ta.max_iters);
            }
            __syncthreads();
            if (!s_go) break;
          }
          if (!ok) break;
          // the solve's correction over the share and its halo
          {
            const bool one = S.iters == 1;
            const T alpha = rhead(num<RK>(S.alpha)), omega = rhead(num<RK>(S.omega));
            for (int l = 4 * tid; l < ext; l += 4 * kTeamThreads) {
              const Q4<T> s = ld4(sr + l), p = ld4(sp + l);
              Q4<T> x{{(T)0, (T)0, (T)0, (T)0}};
              if (!one) x = ld4(at_x(l));
#pragma unroll
              for (int m = 0; m < 4; ++m) x.a[m] = fmaT(alpha, p.a[m], fmaT(omega, s.a[m], x.a[m]));
              st4(at_x(l), x);
            }
            __syncthreads();
          }
        }
        if (!ok) break;
      }
      // ---------------------------------------------------------------- polish
      if (ta.phases & TEAM_POLISH) {
        const PolishAt at = polish_at(fl, S.ycur, S.nhist, S.hslot, cm.hist_cap);
        const bool staged = (ta.phases & TEAM_SOLVE) != 0;  // the last residual's y is still there
        const bool last = step == ta.nsteps - 1;
        // max(y, 0), and the cells it changes, counted per thread and then as part of its first group
        float clamp = 0.0f;
        for (int l = 4 * tid; l < ext; l += 4 * kTeamThreads) {
          Q4<V> y = staged ? *reinterpret_cast<const Q4<V>*>(sv + l) : A::ld4(at.y + e0 + l);
          const bool mine = l >= P && l < P + own;
#pragma unroll
          for (int m = 0; m < 4; ++m) {
            if (mine && A::lt0(y.a[m])) clamp += 1.0f;  // padding cells are 0
            y.a[m] = A::max0(y.a[m]);
          }
          *reinterpret_cast<Q4<V>*>(sv + l) = y;
        }
        __syncthreads();
        float mn = 3.0e38f;
        if (fine) {
          const int p = warp >> 2, l = 4 * 8 * warp + lane;
          if (p < pend) {
            const long long K = c0 + l;
            V mass, rsum;
            polish_cell<C, A>(sv, P + l, P, cf, K, l < own, fl, at, (int)(K - I.base) % P < I.nx, mass, rsum, mn);
            if ((lane & 3) == 0) {
              V* gs = reinterpret_cast<V*>(s_gs) + 2 * (l >> 2);
              gs[0] = mass;
              gs[1] = rsum;
            }
          }
          __syncthreads();
          if (warp < pend) {
            const V* gs = reinterpret_cast<const V*>(s_gs) + 2 * (32 * warp + lane);
            const R w[2] = {gs[0], gs[1]};
            const R t = warp_totals<2, R>(w);
            if (red_writes<2>()) reinterpret_cast<R*>(parts)[red_q<2>() * np + warp] = t;
          }
        } else {
          for (int p = warp; p < pend; p += kTeamThreads / 32) {
            V mass = A::k(0.0), rsum = A::k(0.0);
            for (int k = 0; k < part_c; k += 128) {
              const int l = p * part_c + k + 4 * lane;
              if (l >= own) continue;
              const long long K = c0 + l;
              polish_group<C, A, true>(sv, P + l, P, cf, K, fl, at, I.nx - (int)(K - I.base) % P, mass, rsum, mn);
            }
            const R w[2] = {mass, rsum};
            const R t = warp_totals<2, R>(w);
            if (red_writes<2>()) reinterpret_cast<R*>(parts)[red_q<2>() * np + p] = t;
          }
        }
        team_store<2, R, double>(reinterpret_cast<const R*>(parts), np, SEG, nseg, part(), cm.pstride, seg0);
        // clamped cells (whole numbers) and the minimum: one entry per share, the rest of its segments 0
        // and no minimum
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          clamp += __shfl_xor_sync(0xffffffffu, clamp, o);
          mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
        }
        __shared__ float s_c[kTeamThreads / 32];
        if ((tid & 31) == 0) {
          s_w[warp] = mn;
          s_c[warp] = clamp;
        }
        __syncthreads();
        if (tid < nseg || tid == 0) {
          float m = s_w[0], c = s_c[0];
          for (int w = 1; w < kTeamThreads / 32; ++w) {
            m = fminf(m, s_w[w]);
            c += s_c[w];
          }
          for (int k = tid; k < nseg; k += kTeamThreads) {
            part()[2 * (size_t)cm.pstride + seg0 + k] = k == 0 ? (double)c : 0.0;
            part()[3 * (size_t)cm.pstride + seg0 + k] = (double)m;
          }
        }
        if (!(ok = team_sync(bar, ta, cm.st + sh.inst))) break;
        double tot[3] = {0.0, 0.0, 0.0}, gmin = 0.0;
        if (last && sh.rank == 0) {
          float m = 3.0e38f;  // the minima are FP32 values
          for (int k = tid; k < I.nseg; k += kTeamThreads)
            m = fminf(m, (float)__ldcg(part() + 3 * (size_t)cm.pstride + I.seg0 + k));
          seg_total<3, kTeamThreads / 32, double>(part(), cm.pstride, I.seg0, I.nseg, s_tot);
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) m = fminf(m, __shfl_xor_sync(0xffffffffu, m, o));
          if ((tid & 31) == 0) s_w[warp] = m;
          __syncthreads();
          if (tid == 0) {
#pragma unroll
            for (int w = 1; w < kTeamThreads / 32; ++w) m = fminf(m, s_w[w]);
            gmin = (double)m;
#pragma unroll
            for (int k = 0; k < 3; ++k) tot[k] = s_tot[k];
          }
        }
        flip ^= 1;
        if (tid == 0) after_polish(S, tot[0], tot[1], tot[2], gmin);
        __syncthreads();
      }
    }
    // the instance's state goes back once, by the team's first block (the others only read it
    // before their first barrier)
    if (ok && sh.rank == 0) {
      if (tid == 0) S.outer_active = S.inner_active = 0;
      __syncthreads();
      copy_words(cm.st[sh.inst], S);
    }
    if (ok && sh.rank == 0 && tid == 0) {
      if (ta.report && S.status == ST_NEGATIVE) ta.stat[TEAM_NEGATIVE] = 1;
      if (ta.report && S.status == ST_NOT_CONVERGED) ta.stat[TEAM_NOT_CONVERGED] = 1;
    }
    team_leave(bar);
  }
}

template <typename T, typename C, typename A, int G>
size_t team_limit() {
  cudaFuncAttributes fa;
  int dev = 0, optin = 0;
  if (cudaFuncGetAttributes(&fa, k_team<T, C, A, G>) != cudaSuccess || cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  const size_t left = (size_t)optin > fa.sharedSizeBytes ? (size_t)optin - fa.sharedSizeBytes : 0;
  if (cudaFuncSetAttribute(k_team<T, C, A, G>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)left) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return left;
}

template <typename T, typename C, typename A, int G>
cudaError_t team_launch(const TeamLaunch& l, const Common& cm, const Geo& geo, const Fields& fl, const Coef<C>& cf,
                        const Coef<T>& ck, const Kry<T>& kr, const TeamArgs& ta) {
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)l.grid);
  cfg.blockDim = dim3(kTeamThreads);
  cfg.dynamicSmemBytes = l.smem;
  cfg.stream = l.stream;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k_team<T, C, A, G>, cm, geo, fl, cf, ck, kr, ta);
}

}  // namespace sg
