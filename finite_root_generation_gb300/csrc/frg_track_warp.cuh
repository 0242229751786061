// Warp-per-path tracker of the plug-in systems: the state machine, decisions, counters and
// random draws of track_kernel (frg_track.cu, which includes this file), with one path's
// linear step spread over a warp's lanes. The results are those of track_kernel bit for bit.
//
// What bounds it: one thread's step is a serial chain, for burmester5 about 2,200 FP64
// instructions of some 75 cycles each (80 us), whatever the other lanes do, and the longest
// of a launch's paths takes thousands of steps. Here the rows come from the generated
// schedule (16 independent complex operations a step, one lane per real component: 29
// FP64 instructions where the straight-line code has 834), the parameters q(t) take one
// lane each, the elimination a lane per row and column class, the back substitution a
// lane per real component. GB300, thread / warp: 64 burmester5 paths FP64 135 / 14.5 ms, 64
// conic2 paths 16.2 / 2.9 ms, mixed 4.8 / 0.97 ms. A step: FP64 31k cycles (conic2 19k), of
// which the elimination is a third and each FP64 instruction some 75; FP32 8.0k (5.1k).
//
// Sums of products in the stage combinations and the error's squares are rounded as
// track_kernel's compiled form rounds them (product, then sum; re * re fused onto im * im),
// spelled out so that no compiler choice can separate the two kernels.
#pragma once

#include "frg_device.cuh"
#include "frg_kernels.h"
#include "frg_warp.cuh"

namespace frg {

constexpr int WARP_PATHS = 4;  // warps (paths) per block

// Shared state of one path. `reg` is the schedule's register file: the point's homogeneous
// unknowns, q(t), dq/dt, constants, results. Row r of the linear system: M[r * LD ...],
// right-hand side in column NY.
template <typename T, class S>
struct WarpPath {
  static constexpr int NV = S::NV, NZ = NV + 1, NY = NV + 2, NP = S::NP, LD = NY + 2;
  cx<T> Yc[NY], Vc[NY], Yn[NY], Vn[NY], YN[NY], u[NY], x[NY];
  cx<T> k[8][NY];
  cx<T> sp[NP], fp[NP];
  cx<T> reg[S::TAPE_REGS];
  cx<T> M[NY * LD];
  T t;
  T cn[NY];
};

// Shared memory of a block.
template <typename T, class S>
struct WarpShared {
  WarpPath<T, S> paths[WARP_PATHS];
  uint32_t tape[S::TAPE_STEPS * 16];
  uint16_t outs[S::NV * (S::NV + 2) + S::NV];
};

// Whether system S has a schedule and a block of it fits an SM (FP64, the larger): the
// shipped systems take 12 and 24 KB; one that does not fit runs on track_kernel alone.
template <class S>
constexpr bool warp_fits() {
  if constexpr (S::TAPE_STEPS == 0) return false;
  else return sizeof(WarpShared<double, S>) <= 227 * 1024;
}

template <typename T>
struct WarpStep {
  T ratio;  // pivot ratio (FP32 stage)
  T xnorm;  // |x| (corrector)
  T hnorm;  // |H| (corrector, when asked for)
};

// One component (im: the imaginary one) of a b and of s + a b, the operations of the complex
// product and cfma; the operands are selected, so that both kinds of lane share them
template <typename T>
__device__ __forceinline__ T mul_component(cx<T> a, cx<T> b, bool im) {
  return fma(a.re, im ? b.im : b.re, mul_rn(neg_if(a.im, !im), im ? b.re : b.im));
}
template <typename T>
__device__ __forceinline__ T fma_component(cx<T> a, cx<T> b, T s, bool im) {
  return fma(neg_if(a.im, !im), im ? b.re : b.im, fma(a.re, im ? b.im : b.re, s));
}

// sum_{i < n} |v_i|^2 in index order from the magnitudes in cn
template <typename T>
__device__ __forceinline__ T sum_in_order(const T* cn, int n) {
  T s = T(0);
#pragma unroll 8
  for (int i = 0; i < n; ++i) s += cn[i];
  return s;
}

// One linear step at the point in W.reg[0..NZ), W.t, as track_kernel's: rows, patch rows,
// row scaling, elimination with partial pivoting (first maximum by the rows' current
// order, kept as a position per row instead of moving rows), back substitution; a
// tangent is normalised. The solution goes to W.x.
template <bool LO, typename T, class S>
__device__ __forceinline__ WarpStep<T> warp_step(WarpPath<T, S>& W, const uint32_t* tape, const uint16_t* outs,
                                                 cx<T> gamma, const cx<T>* patch, bool newton, bool tstep, T tgoal,
                                                 bool want_hnorm, int lane) {
  typedef WarpPath<T, S> P;
  constexpr int NV = P::NV, NZ = P::NZ, NY = P::NY, NP = P::NP, LD = P::LD;
  static_assert(NY <= 32, "a lane per row");
  constexpr int RP = NY <= 4 ? 4 : (NY <= 8 ? 8 : (NY <= 16 ? 16 : 32));  // lanes for the rows
  constexpr int CL = 32 / RP;                                             // column classes
  const bool im = lane & 1;
  WarpStep<T> out;
  out.ratio = out.xnorm = out.hnorm = T(0);

  // ---- q(t), dq/dt (htpysupport.cu:37-62)
  {
    const T t = W.t;
    const cx<T> g1t = gamma * (T(1) - t);
    const cx<T> iden = cinv(g1t + cx<T>(t));
    const cx<T> gid2 = gamma * (iden * iden);
#pragma unroll 1
    for (int i = lane; i < NP; i += 32) {
      const cx<T> s = W.sp[i], f = W.fp[i];
      W.reg[NZ + i] = (g1t * s + t * f) * iden;
      W.reg[NZ + NP + i] = (f - s) * gid2;
    }
  }
  __syncwarp();
  // ---- the rows: lane 2 o + c computes component c of the step's operation o
  uint32_t wn = tape[lane >> 1];  // the next step's, loaded ahead
#pragma unroll 1
  for (int st = 0; st < S::TAPE_STEPS; ++st) {
    const uint32_t w = wn;
    wn = tape[(st + 1 < S::TAPE_STEPS ? st + 1 : 0) * 16 + (lane >> 1)];
    const cx<T> a = W.reg[(w >> 10) & 1023], b = W.reg[(w >> 20) & 1023];
    T r;
    if (w >> 31) {
      r = mul_component(a, b, im);
    } else {
      const T x = im ? a.im : a.re, y = im ? b.im : b.re;
      r = x + neg_if(y, (w >> 30) & 1);
    }
    reinterpret_cast<T*>(&W.reg[w & 1023])[im] = r;
    __syncwarp();
  }
  // ---- the system: rows, projective patch (htpysupport.cu:139-142), velocity patch
#pragma unroll 1
  for (int o = lane; o < NV * NY; o += 32) {
    const unsigned w = outs[o];
    const cx<T> v = W.reg[w & 1023];
    W.M[(o / NY) * LD + o % NY] = cx<T>(neg_if(v.re, w >> 10), neg_if(v.im, w >> 10));
  }
  if (lane < NY) {
    W.M[NV * LD + lane] = W.u[lane];
    W.M[(NV + 1) * LD + lane] = patch[lane];
    if (!newton) W.M[lane * LD + NY] = cx<T>(T(lane == NY - 1 ? 1 : 0));
  }
  if (newton) {
    if (lane < NV) {
      const unsigned w = outs[NV * NY + lane];
      const cx<T> v = W.reg[w & 1023];
      W.M[lane * LD + NY] = cx<T>(neg_if(v.re, w >> 10), neg_if(v.im, w >> 10));
    }
    // u . Y - 1, one lane per component
    T d = T(0);
#pragma unroll 8
    for (int e = 0; e < NY; ++e) {
      const cx<T> b = W.u[e], y = e < NZ ? W.reg[e] : cx<T>(W.t);
      d = fma_component(b, y, d, im);
    }
    d -= im ? T(0) : T(1);
    if (lane < 2) reinterpret_cast<T*>(&W.M[NV * LD + NY])[im] = d;
    __syncwarp();
    if (want_hnorm) {
      if (lane < NZ) W.cn[lane] = cnorm2(W.M[lane * LD + NY]);
      __syncwarp();
      out.hnorm = sqrt(sum_in_order(W.cn, NZ));
    }
  }
  __syncwarp();
  // ---- row scaling by 1/max(|re|,|im|) (htpysupport.cu:259-277, :446-471); b = -F. From
  //      here the elimination keeps row r's columns cl, cl + CL, ... in registers; in shared
  //      memory, with a load and a store per pivot on the chain, a burmester5 step was 11.4k
  //      cycles in FP32 and 32.0k in FP64, with it 8.3k and 30.7k (64 paths mixed: 2.5 -> 1.75
  //      and 3.3 -> 3.1 ms)
  const int r = lane % RP, cl = lane / RP;
  constexpr int KC = (NY + CL) / CL;  // a lane's columns of NY + 1
  cx<T> m[KC];
  {
    MaxAbs<T> mx;
#pragma unroll
    for (int k = 0; k < KC; ++k) {
      const int c = cl + k * CL;
      m[k] = c <= NY ? W.M[(r < NY ? r : 0) * LD + c] : cx<T>(T(0));
      if (c < NY) mx.take(m[k]);
    }
#pragma unroll
    for (int off = RP; off < 32; off <<= 1) mx.across(off);
    const T s = T(1) / mx.value();
#pragma unroll
    for (int k = 0; k < KC; ++k) {
      const int c = cl + k * CL;
      if (r < NZ && (c < NY || newton)) {
        const cx<T> v = s * m[k];
        m[k] = cx<T>(neg_if(v.re, c == NY), neg_if(v.im, c == NY));
      }
    }
  }
  // ---- elimination (htpysupport.cu:146-232; the corrector leaves the last row out,
  //      :302-400)
  const int nelim = newton ? NZ : NY;
  int pos = r;  // current position of row r
  T pmax = T(0), pmin = T(-1);
  cx<T> ips[NY];
#pragma unroll
  for (int i = 0; i < NY; ++i) {
    if (i >= nelim) continue;  // the last row of a corrector step
    const cx<T> e = warp_shfl(m[i / CL], r + RP * (i % CL));
    const bool live = r < NY && pos >= i && pos < nelim;
    const T v = cnorm2(e);
    cx<T> ip;
    if constexpr (sizeof(T) == 4) ip = cinv_norm(e, v);  // every candidate's, while the search runs
    int pr = -1;
    {
      // rows with a magnitude above zero, not NaN, compared as integers
      unsigned cand;
      if constexpr (sizeof(T) == 8) {
        const long long bits = __double_as_longlong(v);
        const bool ok = live && bits > 0 && bits <= 0x7ff0000000000000ll;
        const int hi = ok ? (int)(bits >> 32) : -1;
        const int mh = __reduce_max_sync(FULL, hi);
        const unsigned lo = ok && hi == mh ? (unsigned)bits : 0u;
        cand = __ballot_sync(FULL, ok && hi == mh);
        if (__popc(cand) > CL) {
          const unsigned ml = __reduce_max_sync(FULL, lo);
          cand = __ballot_sync(FULL, ok && hi == mh && (unsigned)bits == ml);
        }
      } else {
        const int bits = __float_as_int(v);
        const bool ok = live && bits > 0 && bits <= 0x7f800000;
        const int mh = __reduce_max_sync(FULL, ok ? bits : -1);
        cand = __ballot_sync(FULL, ok && bits == mh);
      }
      if (cand) {
        if (__popc(cand) > CL) {  // equal magnitudes: the first by position
          const int mp = __reduce_min_sync(FULL, (cand >> lane) & 1 ? pos : 99);
          cand = __ballot_sync(FULL, pos == mp && r < NY);
        }
      } else {
        cand = __ballot_sync(FULL, pos == i && r < NY);
      }
      pr = (__ffs(cand) - 1) % RP;
    }
    const int ppos = __shfl_sync(FULL, pos, pr);
    if (r == pr) pos = i;
    else if (pos == i) pos = ppos;
    const T pa = __shfl_sync(FULL, v, pr);
    if constexpr (sizeof(T) == 4) ip = warp_shfl(ip, pr);
    else ip = cinv_norm(warp_shfl(e, pr), pa);
    ips[i] = ip;
    if (LO) {
      const T a = sqrt(pa);
      pmax = fmax(pmax, a);
      pmin = (pmin < T(0)) ? a : fmin(pmin, a);
    }
    cx<T> l;
    if constexpr (sizeof(T) == 8 && CL > 1) {
      // the two components on neighbouring column classes
      const T own = mul_component(e, ip, cl & 1), other = __shfl_xor_sync(FULL, own, RP);
      l = cl & 1 ? cx<T>(other, own) : cx<T>(own, other);
    } else {
      l = e * ip;
    }
    const bool below = r < NY && pos > i && pos < nelim;
#pragma unroll
    for (int k = (i + 1) / CL; k < KC; ++k) {
      const cx<T> pv = warp_shfl(m[k], pr + RP * cl);
      if (below && cl + k * CL > i) m[k] = cfms(m[k], pv, l);
    }
  }
  if (LO) out.ratio = pmin > T(0) ? pmax / pmin : T(1e30);
  // the factor's rows by position, right-hand side in column NY
  __syncwarp();
  if (r < NY) {
#pragma unroll
    for (int k = 0; k < KC; ++k)
      if (cl + k * CL <= NY) W.M[pos * LD + cl + k * CL] = m[k];
  }
  __syncwarp();
  // ---- back substitution, row by row, one lane per component, the solution in registers
  cx<T> x[NY];
#pragma unroll
  for (int i = NY - 1; i >= 0; --i) {
    if (i == NY - 1 && newton) {
      x[i] = cx<T>(tgoal - W.t);
      if (lane == 0) W.x[i] = x[i];
      continue;
    }
    const cx<T>* mi = W.M + i * LD;
    T sum = T(0);
#pragma unroll
    for (int c = i + 1; c < NY; ++c) sum = fma_component(mi[c], x[c], sum, im);
    const T d = (im ? mi[NY].im : mi[NY].re) - sum, o = __shfl_xor_sync(FULL, d, 1);
    const cx<T> v = im ? cx<T>(o, d) : cx<T>(d, o);
    const T xi = mul_component(ips[i], v, im), xo = __shfl_xor_sync(FULL, xi, 1);
    x[i] = im ? cx<T>(xo, xi) : cx<T>(xi, xo);
    if (lane == 0) W.x[i] = x[i];
  }
  __syncwarp();
  // ---- |x|, and the tangent's normalisation (htpysupport.cu:285-296)
  const cx<T> xe = W.x[lane < NY ? lane : 0];
  if (lane < NY) W.cn[lane] = cnorm2(xe);
  __syncwarp();
  const T n2 = sum_in_order(W.cn, NY);
  if (newton) {
    out.xnorm = sqrt(n2);
  } else {
    const cx<T> xt = W.x[NY - 1];
    cx<T> sc;
    if (!tstep) {
      const T nr = sqrt((lane & 1) ? n2 : cnorm2(xt));
      sc = cx<T>(xt.re, neg_if(xt.im, true)) * (T(1) / (__shfl_sync(FULL, nr, 0) * __shfl_sync(FULL, nr, 1)));
    } else {
      sc = cinv(xt);
    }
    __syncwarp();
    if (lane < NY) {
      cx<T> v = sc * xe;
      if (lane == NY - 1) v.im = T(0);
      W.x[lane] = v;
    }
  }
  __syncwarp();
  return out;
}

// A new random patch (entry e from draws base + 2 e, base + 2 e + 1)
template <typename T>
__device__ __forceinline__ cx<T> patch_entry(uint64_t seed, uint64_t stream, uint64_t base, double range, int e) {
  return cx<T>(T(2.0 * range * frg_uniform01(seed, stream, base + 2 * e) - range),
               T(2.0 * range * frg_uniform01(seed, stream, base + 2 * e + 1) - range));
}

// Modes as track_kernel's. With a.from_tail the launch continues the paths that a
// track_kernel launch of the same mode left in a.tail.
template <int MODE, typename T, class S>
__global__ void __launch_bounds__(32 * WARP_PATHS) warp_kernel(TrackArgs a) {
  typedef WarpPath<T, S> P;
  constexpr int NV_ = P::NV, NZ_ = P::NZ, NY_ = P::NY, NP_ = P::NP;
  constexpr bool LO = (MODE == MODE_LO);
  extern __shared__ __align__(16) unsigned char warp_smem[];
  WarpShared<T, S>& sh = *reinterpret_cast<WarpShared<T, S>*>(warp_smem);
  uint32_t* const tape = sh.tape;
  uint16_t* const outs = sh.outs;
  const frg_config& c = a.cfg;
  const int lane = threadIdx.x & 31;
  const bool el = lane < NY_;
  P& W = sh.paths[threadIdx.x >> 5];
  for (int i = threadIdx.x; i < S::TAPE_STEPS * 16; i += blockDim.x) tape[i] = S::tape()[i];
  for (int i = threadIdx.x; i < NV_ * NY_ + NV_; i += blockDim.x) outs[i] = S::tape_out()[i];
  for (int i = lane; i < S::TAPE_REGS; i += 32) W.reg[i] = cx<T>(T(0));
  __syncthreads();
  for (int i = lane; i < S::TAPE_CONSTS; i += 32) W.reg[NZ_ + 2 * NP_ + i] = cx<T>(T(S::tape_const()[i]));
  const T newt_tol = LO ? T(c.newt_tol_lo) : T(c.newt_tol);
  const int64_t ntail = a.from_tail ? (int64_t)*a.tail_count : 0;
  const int64_t nqueue = a.from_tail ? (ntail < a.tail_cap ? ntail : a.tail_cap)
                         : (MODE == MODE_RESUME) ? (int64_t)*a.handoff_count : a.npaths;
  unsigned long long fp64_solves = 0;

  for (;;) {
    // ------------------------------------------------------------------ fetch
    unsigned long long qi = 0;
    if (lane == 0) qi = atomicAdd(a.queue, 1ull);
    qi = __shfl_sync(FULL, qi, 0);
    if ((int64_t)qi >= nqueue) break;
    const int64_t id = a.from_tail ? a.tail[qi].id : (MODE == MODE_RESUME) ? a.handoff_list[qi] : (int64_t)qi;
    const bool resumed = MODE == MODE_RESUME || a.from_tail;
    int task = 0, hi = a.ntasks - 1;  // task of this path
    while (task < hi) {
      const int mid = (task + hi + 1) >> 1;
      if (a.task_start[mid] <= id) task = mid; else hi = mid - 1;
    }
    const uint64_t stream = (uint64_t)(id + c.path_offset);
    const cx<T> gamma = task_gamma<T>(a, task);
    {
      const cd* st = a.starts + (size_t)id * (NV_ + NP_);
      for (int i = lane; i < NP_; i += 32) W.sp[i] = cx<T>(st[NV_ + i]);
      if (!resumed && el) W.Yc[lane] = lane < NV_ ? cx<T>(st[lane]) : cx<T>(T(lane == NV_ ? 1 : 0));
    }
    const cx<T>* fpmT = TaskFpm<T, NP_>::get(a, task);
    for (int i = lane; i < NP_; i += 32) W.fp[i] = fpmT[i];
    T s = T(0), err = T(0), scale = T(0), residual = T(100);
    int tstepQ = 0, streak = 0, step = 0, ministep = 0, stage = 0, attempt = 0, it = 0, code = 0;
    int n_ivp = 0, n_newton = 0, phase = PH_TANGENT0;
    uint64_t rng_index = 4 * NY_;
    if (resumed) {
      const Handoff& h = a.from_tail ? a.tail[qi] : a.handoff[id];
      if (el) { W.Yc[lane] = cx<T>(h.Yc[lane]); W.Vc[lane] = cx<T>(h.Vc[lane]); W.u[lane] = cx<T>(h.u[lane]); }
      s = T(h.s); rng_index = h.rng_index; streak = h.streak; step = h.step; ministep = h.ministep;
      tstepQ = h.tstepQ; n_ivp = h.n_ivp; n_newton = h.n_newton;
      phase = PH_RK;
    } else {
      if (el) {
        W.u[lane] = patch_entry<T>(a.seed, stream, 0, c.patch_range, lane);
        W.Vc[lane] = patch_entry<T>(a.seed, stream, 2 * NY_, c.patch_range, lane);
      }
      __syncwarp();
      if (lane == 0) switch_patch<T, NY_>(W.u, W.Yc, W.Yc);
      s = T(c.s_init); streak = c.caution_steps - 1;
    }
    __syncwarp();

    for (;;) {  // the path's steps
      // ------------------------------------------------ set up the linear step
      const bool newton = (phase == PH_NEWTON || phase == PH_SHARP);
      const bool tstep = phase == PH_RK && tstepQ != 0;
      const cx<T>* patch = W.Vc;
      cx<T> y;
      if (phase == PH_TANGENT0 || (phase == PH_RK && stage == 0)) {
        y = W.Yc[el ? lane : 0];
      } else if (phase == PH_RK) {
        patch = W.k[stage - 1];
        const T ws = lane < stage ? Dp<T>::a(stage)[lane] * s : T(0);
        cx<T> acc(T(0));
#pragma unroll
        for (int l = 6; l >= 0; --l) {
          const T wl = __shfl_sync(FULL, ws, l);
          if (l < stage) {
            const cx<T> term = mul_rn(wl, W.k[l][el ? lane : 0]);
            acc = l == stage - 1 ? term : term + acc;
          }
        }
        y = W.Yc[el ? lane : 0] + acc;
      } else {
        y = W.YN[el ? lane : 0];
      }
      if (lane < NZ_) W.reg[lane] = y;
      if (lane == NY_ - 1) W.t = y.re;
      const T tgoal = (phase == PH_SHARP) ? T(1) : W.Yn[NY_ - 1].re;
      __syncwarp();

      // ------------------------------------------------------ the linear step
      const bool sharp = phase == PH_SHARP;
      const int restype = sharp ? c.sharp_residual : c.newt_residual;
      if (MODE != MODE_LO) fp64_solves++;
      const WarpStep<T> r = warp_step<LO, T, S>(W, tape, outs, gamma, patch, newton, tstep, tgoal,
                                                newton && restype == 0, lane);
      if (newton) n_newton++; else n_ivp++;

      // ------------------------------------------------------------- transitions
      bool finished = false;
      int handoff = 0;
      const cx<T>* final_src = W.Yc;  // the reference's Yc aliases Yfinal (htpytrack.cu:46)
      if (LO && !(r.ratio <= T(c.cond_switch))) {
        handoff = 2;  // ill-conditioned (or non-finite) step: continue in FP64 from Yc
      } else if (phase == PH_TANGENT0) {
        if (el) W.Vc[lane] = W.x[lane];
        if (c.max_steps == 0) { code = 1; finished = true; }
        stage = 0;
        phase = PH_RK;
      } else if (phase == PH_RK) {
        if (el) W.k[stage][lane] = W.x[lane];
        __syncwarp();
        if (++stage == 8) {
          stage = 0;
          // error estimate and step factor (rungekutta.cu:99-112), prediction (:115-122)
          const T we = Dp<T>::e()[lane & 7] * s, wb = Dp<T>::b()[lane & 7] * s;
          const cx<T> k7 = W.k[7][el ? lane : 0];
          cx<T> le = mul_rn(__shfl_sync(FULL, we, 7), k7);
          cx<T> yb = mul_rn(__shfl_sync(FULL, wb, 7), k7);
#pragma unroll
          for (int l = 6; l >= 0; --l) {
            if (l == 1) continue;  // weight zero in both
            const cx<T> kl = W.k[l][el ? lane : 0];
            le = mul_rn(__shfl_sync(FULL, we, l), kl) + le;
            yb = mul_rn(__shfl_sync(FULL, wb, l), kl) + yb;
          }
          if (el) {
            W.cn[lane] = fma(le.re, le.re, mul_rn(le.im, le.im));
            W.Yn[lane] = W.Yc[lane] + yb;
            W.Vn[lane] = k7;
          }
          __syncwarp();
          err = sqrt(sum_in_order(W.cn, NY_));
          scale = (err > T(10e-17)) ? T(0.8) * pow(T(c.rk_tol) / err, T(1) / T(6)) : T(5);
          if (scale > T(5)) scale = T(5);
          if (ministep++ == c.max_ministeps) { code = 2; finished = true; }
          else if (err <= T(c.rk_tol)) {
            const T tn = W.Yn[NY_ - 1].re;
            if (LO && tn > T(1.0 - c.nudge_trigger)) handoff = 5;  // the endgame runs in FP64
            else if (tn <= T(1.0 - c.nudge_trigger)) { attempt = 0; phase = PH_NEWTON; }
            else if (fabs(T(1) - tn) < T(c.sharp_trigger)) { attempt = 0; phase = PH_SHARP; }
            else { tstepQ = 1; s = T(1) - W.Yc[NY_ - 1].re; }  // land on t = 1 (htpytrack.cu:120-123)
            if (phase != PH_RK) {
              if (el) W.YN[lane] = W.Yn[lane];
              residual = T(100);
              it = 0;
            }
          } else if (s <= T(c.s_min)) {
            if (LO) handoff = 4; else { code = 3; finished = true; }
          } else {
            s *= scale;
            if (s < T(c.s_min)) s = T(c.s_min * 0.9);
            streak = 0;
          }
        }
      } else {
        // one corrector or sharpening iteration (htpysupport.cu:427-492)
        const int max_its = sharp ? c.sharp_its : c.newt_its;
        const T tol = sharp ? T(c.sharp_tol) : newt_tol;
        bool done = false;
        if (restype == 0 && it > 0) {
          // |H| at the current point is the residual of the previous update
          residual = r.hnorm;
          if (!(it < max_its && residual > tol)) done = true;
        }
        if (!done) {
          if (el) W.YN[lane] += W.x[lane];
          it++;
          if (restype != 0) {
            residual = r.xnorm;
            if (!(it < max_its && residual > tol)) done = true;
          }
        }
        __syncwarp();
        if (done) {
          if (sharp) final_src = W.YN;
          const bool ok = residual < (sharp ? T(c.sharp_tol) : newt_tol);
          if (ministep++ == c.max_ministeps) { code = 2; finished = true; }
          else if (ok && sharp) { code = 0; finished = true; }
          else if (ok) {
            if (fabs(T(1) - W.Yn[NY_ - 1].re) < T(c.sharp_trigger)) {
              attempt = 0; phase = PH_SHARP; residual = T(100); it = 0;
              if (el) W.YN[lane] = W.Yn[lane];
            } else {
              // accept the step (htpytrack.cu:176-183)
              if (el) { W.Yc[lane] = W.YN[lane]; W.Vc[lane] = W.Vn[lane]; }
              streak++;
              if (streak < c.caution_steps && scale > T(1)) scale = T(1);
              s *= scale;
              if (s > T(c.s_max)) s = T(c.s_max);
              else if (s < T(c.s_min)) s = T(c.s_min * 0.9);
              step++;
              if (step == c.max_steps) { code = 1; finished = true; }
              else if (LO && W.YN[NY_ - 1].re >= T(c.t_switch)) handoff = 1;
              else { stage = 0; phase = PH_RK; }
            }
          } else {
            // new random patch and retry (htpytrack.cu:145-153, :204-213)
            if (el) W.u[lane] = patch_entry<T>(a.seed, stream, rng_index, c.patch_range, lane);
            rng_index += 2 * NY_;
            __syncwarp();
            if (lane == 0) switch_patch<T, NY_>(W.u, W.Yn, W.Yn);
            __syncwarp();
            if (++attempt < (sharp ? c.sharp_attempts : c.newt_attempts)) {
              residual = T(100); it = 0;
              if (el) W.YN[lane] = W.Yn[lane];
            } else if (sharp) {
              code = 5; finished = true;
            } else if (s <= T(c.s_min)) {
              if (LO) handoff = 3; else { code = 4; finished = true; }
            } else {
              s *= T(0.5);
              if (s < T(c.s_min)) s = T(c.s_min * 0.9);
              streak = 0;
              stage = 0;
              phase = PH_RK;
            }
          }
        }
      }
      __syncwarp();
      if (LO && handoff) {
        Handoff& h = a.handoff[id];
        if (el) { h.Yc[lane] = cd(W.Yc[lane]); h.Vc[lane] = cd(W.Vc[lane]); h.u[lane] = cd(W.u[lane]); }
        if (lane == 0) {
          h.s = double(s); h.rng_index = rng_index; h.streak = streak; h.step = step; h.ministep = ministep;
          h.tstepQ = tstepQ; h.n_ivp = n_ivp; h.n_newton = n_newton; h.reason = handoff; h.code = 0;
          if (a.counters) { atomicAdd(&a.counters[12], 1ull); atomicAdd(&a.counters[15 + handoff], 1ull); }
          const unsigned long long slot = atomicAdd(a.handoff_count, 1ull);
          a.handoff_list[slot] = id;
        }
        __syncwarp();
        break;
      }
      if (finished) {
        if (el) a.finals[(size_t)id * NY_ + lane] = cd(final_src[lane]);  // finish_kernel does the rest
        if (lane == 0) {
          a.codes[id] = code;
          if (a.work) {
            a.work[(size_t)id * 3 + 0] = n_ivp;
            a.work[(size_t)id * 3 + 1] = n_newton;
            a.work[(size_t)id * 3 + 2] = step;
          }
          if (a.counters) {
            atomicAdd(&a.counters[8], (unsigned long long)n_ivp);
            atomicAdd(&a.counters[9], (unsigned long long)n_newton);
            atomicAdd(&a.counters[10], (unsigned long long)step);
          }
        }
        __syncwarp();
        break;
      }
    }
  }
  if (a.counters && fp64_solves && lane == 0) atomicAdd(&a.counters[11], fp64_solves);
}

}  // namespace frg
