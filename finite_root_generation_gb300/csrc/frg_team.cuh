// Building blocks of the warp-cooperative tracker: one path per warp, four paths per
// block, every linear step in two parts.
//
// Evaluation, by the block. The seven equation groups of a path (group j = rows j-1,
// j+6, j+13 of the reference's JH, htpysupport.cu:89-144) run on seven lanes, so a warp
// holds the groups of the block's four paths; the straight-line code of a group is cut
// into four parts of equal cost, one per warp (frg_eval_slice, generated), and what the
// parts share (q(t), reciprocals, the quantities of FrgEvalIn) is computed once by the
// path's own warp (eval_prep).
//
// Solve, by the path's own warp (solve_step). The reference's 23x23 row-scaled dense LU
// (LinearSolve / LinearSolveNewton, htpysupport.cu:146-400) is solved with the system's
// structure: U_j appears only in group j's three equations and in the two patch rows, so
// each group pivots U_j out of its own rows (partial pivoting among its three rows; lane
// 8 q + g holds the columns c = q mod 4 of group g + 1) and the eliminations are folded
// into the patch rows with one butterfly reduction. What remains is a dense 16 x 16
// system in the links A..Hc, the homogenizer Z0 and t: lane 16 h + r holds the columns
// c = h mod 2 of row r, partial pivoting across the lanes, then column-oriented back
// substitution; U_j follows from the group's pivot row. The solution is the same as the
// dense solve up to rounding (checked against the dense LU in the tests). The Newton
// variant replaces the velocity patch by the t-selector row with right-hand side
// t_goal - t, which fixes dt exactly like LinearSolveNewton's x[22] = tdiff
// (htpysupport.cu:374).
//
// What bounds it: on this part a warp-wide FP64 instruction holds its sub-partition's
// FP64 pipe for 64 cycles and answers after about 73, whatever the number of active
// lanes, so an FP64 step takes (FP64 warp instructions on its longest warp) x 64..91
// cycles and everything else hides behind them; the FP32 step is bound by instruction
// issue and fetch. With one path per 8 lanes (four paths in a warp, the layout before
// this one) an FP64 step was 5,800 FP64 instructions in one warp, 421k cycles; cut over
// the four sub-partitions, with 32 lanes on the elimination and equal operations of
// different quantities in the same instructions, it is about 1,400 on the longest warp,
// 123k cycles, and 1,150, 105k cycles, while a block has one or two paths (PairCx). The
// FP32 step went from 105k to 15k. With every SM full the FP64 work per path falls as
// well (fewer repeated sums and idle lanes): FP64 rounds of 32,768 paths, three in flight,
// 6,815 to 3,696 ms a round. Comparisons, maxima and stored negations of FP64 values run
// on their bit patterns in the integer pipes for the same reason.
#pragma once

#include <cstddef>

#include "frg_device.cuh"
#include "frg_df.cuh"
#include "frg_warp.cuh"

namespace frg {

__device__ __forceinline__ df neg_if(df x, bool neg) { return neg ? -x : x; }
__device__ __forceinline__ cx<df> warp_shfl(cx<df> v, int src) {
  return cx<df>(df(__shfl_sync(FULL, v.re.hi, src), __shfl_sync(FULL, v.re.lo, src)),
                df(__shfl_sync(FULL, v.im.hi, src), __shfl_sync(FULL, v.im.lo, src)));
}

namespace team {

// Type of the path's points (Yc, Yn, YN) and of the FP32 stage's refinement residual:
// FP64 by default; the FP32 stage can instead keep them in double-float (P = df), which
// runs on the FP32 pipes but is ~10x more code than the FP64 form.
template <typename T> struct PointOf { typedef double type; };

constexpr int TEAM = 8;    // lanes of one path in the evaluation (7 groups)
constexpr int PATHS = 4;   // paths (warps) per block
constexpr int VS = 24;     // shared-memory vector stride (23 used)
constexpr int LDU = 21;    // leading dimension of the dense system and its factor (odd: no bank conflicts)

// reduced-system column -> state index
__device__ __forceinline__ constexpr int gstate(int c) { return c < 14 ? c : (c == 14 ? 21 : 22); }

template <typename T>
__device__ __forceinline__ T shfl_xor(unsigned mask, T v, int off) { return __shfl_xor_sync(mask, v, off, TEAM); }
__device__ __forceinline__ df shfl_xor(unsigned mask, df v, int off) {
  return df(__shfl_xor_sync(mask, v.hi, off, TEAM), __shfl_xor_sync(mask, v.lo, off, TEAM));
}
// sums and maxima over each group of 8 lanes (in every lane of the group)
template <typename T>
__device__ __forceinline__ T team_sum(unsigned mask, T v) {
  v += shfl_xor(mask, v, 4);
  v += shfl_xor(mask, v, 2);
  v += shfl_xor(mask, v, 1);
  return v;
}
template <typename T>
__device__ __forceinline__ T team_max(unsigned mask, T v) {
  v = fmax(v, shfl_xor(mask, v, 4));
  v = fmax(v, shfl_xor(mask, v, 2));
  v = fmax(v, shfl_xor(mask, v, 1));
  return v;
}

// Task and start parameters in the working precision, when it is not the point type's.
template <typename T, typename P> struct LowTask { cx<T> sp[32], fp[32]; };
template <typename T> struct LowTask<T, T> {};
template <typename T, typename P> struct HighEval { FrgEvalIn<P> in; };
template <typename T> struct HighEval<T, T> {};

// Shared state of one path. The points Yc (accepted), Yn (predicted) and YN (corrector
// iterate) are in the point type (FP64, or double-float in the FP32 stage, whose
// corrector refines on double-float residuals with an FP32 solve); directions, patches
// and stage vectors are in the working precision T. `M` holds the group rows
// (frg_eval_slice's layout; its structural zeros are written once). The evaluation's
// inputs and what the solve writes (the dense system with its factor, the groups' pivot
// rows) share memory: the block's barriers keep them apart.
template <typename T, typename P = typename PointOf<T>::type>
struct Smem {
  struct Inputs {
    FrgEvalIn<T> in;
    cx<T> dq[32];
    alignas(16) HighEval<T, P> hi;
  };
  static constexpr size_t kSolve = sizeof(cx<T>) * (16 * LDU + 17 * 8);
  static constexpr size_t kWork = sizeof(Inputs) > kSolve ? sizeof(Inputs) : kSolve;
  cx<P> Yc[VS], Yn[VS], YN[VS];
  cx<P> sp[32], fp[32];
  cx<P> gamma;
  LowTask<T, P> lo;
  cx<T> Vc[VS], Vn[VS], u[VS], Ye[VS];
  alignas(16) cx<T> X[16];  // solution; X .. k are free during a corrector step's evaluation (Residual)
  cx<T> XU[8], dx[VS], k[8][VS];
  cx<T> M[3 * 18 * 8];
  cx<T> R[3][8], Rd;  // refined residuals and patch residual
  T cn[16];
  alignas(16) unsigned char work[kWork];
  int active, refine;
  double ck_t[2];  // checkpoint history of the early-retirement features: t at the last two
  float ck_s[2];   // checkpoints, step sizes there, largest condition estimate since
  float ck_rmax;
  unsigned long long cyc[8];  // cycle accounting (lane 0)
  __device__ __forceinline__ Inputs& inputs() { return *reinterpret_cast<Inputs*>(work); }
  __device__ __forceinline__ cx<T>* U() { return reinterpret_cast<cx<T>*>(work); }
  // pivot rows of the groups: [column][group], right-hand side at column 16
  __device__ __forceinline__ cx<T>* piv() { return U() + 16 * LDU; }
};

__device__ __forceinline__ int param_index(int slot, int j) {
  switch (slot) {
    case 0: return 0;
    case 1: return 8;
    case 2: return j;
    case 3: return 8 + j;
    case 4: return 15 + j;
    default: return 22 + j;
  }
}

template <typename T>
struct StepOut {
  T ratio;   // condition estimate (pivot ratios of the elimination), +inf if not finite
  T xnorm2;  // |x|^2 of the solution (Newton)
  T hnorm;   // |H| at the evaluation point (Newton, when asked for)
};

// What the evaluation of one path at Y needs: the reciprocals, one per lane (1 / U_j on
// lanes 0..6, e on 8..11, q's denominator on 12); q(t) (and dq/dt, htpysupport.cu:37-62),
// one parameter per lane, with z^2 and z^3 on lane 31 in the same products; then the
// hoisted quantities, lanes 8 s + g those of side s and group g, lanes 16 + s those that
// are the same for every group, again in the same instructions. 81 FP64 instructions; with
// each quantity in instructions of its own it was 143. RESID (the refinement residual): the
// reciprocals and q(t) alone, as its schedules hold the rest.
template <bool RESID, typename V>
__device__ __forceinline__ void eval_prep(const cx<V>* Y, const cx<V>* sp, const cx<V>* fp, cx<V> gamma,
                                          FrgEvalIn<V>& in, cx<V>* dq, int lane) {
  const V t = Y[22].re;
  const cx<V> z = Y[21];
  const cx<V> g1t = gamma * (V(1) - t);
  cx<V> ib;
  {
    const int ea = lane == 8 ? 4 : lane == 9 ? 6 : lane == 10 ? 11 : 13;  // F, H, Fc, Hc
    const int eb = lane == 8 ? 1 : lane == 9 ? 2 : lane == 10 ? 8 : 9;    // B, C, Bc, Cc
    // a - b with b = -t on lane 12 (a + t and a - (-t) round alike)
    const cx<V> x = lane == 12 ? g1t : Y[ea], y = lane == 12 ? cx<V>(neg_if(t, true)) : Y[eb];
    const cx<V> d = x - y;
    ib = cinv(lane < 7 ? Y[14 + lane] : d);
  }
  if (lane < 7) in.iU[lane] = ib;
  if (lane >= 8 && lane < 12) in.e[lane - 8] = ib;
  const cx<V> iden = warp_shfl(ib, 12);
  {
    const int i = lane < NP ? lane : 0;
    const cx<V> s = sp[i], f = fp[i];
    const cx<V> q = (g1t * s + t * f) * iden;
    if (lane < NP) in.q[lane] = q;
    if constexpr (!RESID) {
      const bool l31 = lane == 31;
      const cx<V> a = l31 ? z : iden;
      const cx<V> sq = a * a;
      const cx<V> cu = (l31 ? sq : gamma) * (l31 ? z : sq);
      if (l31) { in.z2 = sq; in.z3 = cu; }
      const cx<V> v = (f - s) * cu;
      if (lane < NP) dq[lane] = v;
    }
  }
  __syncwarp();
  if constexpr (!RESID) {
    const bool all = lane >= 16;  // lanes 16, 17: the same for every group
    const int s = all ? lane & 1 : lane >> 3, g = (lane & 7) < 7 ? lane & 7 : 6;
    const cx<V>* L = Y + 7 * s;  // A, B, C, D, F, G, H of this side
    const cx<V> e2 = in.e[2 * s + 1];
    const cx<V> m0 = in.q[all ? 8 * s : 8 * s + 1 + g] * z;                  // pjz | pz
    const cx<V> d0 = L[all ? 4 : 0] - m0, d1 = L[all ? 6 : 1] - m0;          // ap, bp | fp, hp
    const cx<V> d2 = L[all ? 1 : 0] - L[all ? 3 : 2];                        // ac | bd
    const cx<V> m1 = (all ? in.e[2 * s] : in.q[15 + 7 * s + 1 + g]) * d2;    // qa | ebd
    const cx<V> d3 = (all ? L[2] : d0) - (all ? L[5] : m1);                  // aq | cg
    const cx<V> m2 = e2 * d3;                                                // eaq | ecg
    const cx<V> ebd = warp_shfl(m1, 16 + s);
    const cx<V> w0 = L[1] - L[0] + m1;
    const cx<V> t0 = (all ? d0 : d1) * ebd;                                  // bp ebd | fp ebd
    const cx<V> w1 = w0 + t0;
    const cx<V> cg = warp_shfl(d3, 16 + s);
    const cx<V> t1 = (all ? d1 : cg) * m2;                                   // cg eaq | hp ecg
    const cx<V> w = (all ? t0 : w1) - t1;                                    // w | v
    if (lane < 16) {
      cx<V>(*o)[8] = in.sb[s];
      const int c = lane & 7;
      o[FRG_IN_PJZ][c] = m0; o[FRG_IN_AP][c] = d0; o[FRG_IN_BP][c] = d1;
      o[FRG_IN_QA][c] = m1;  o[FRG_IN_AQ][c] = d3; o[FRG_IN_W][c] = w;   o[FRG_IN_EAQ][c] = m2;
      if (c == 0) in.sa[s][FRG_IN_AC] = d2;
    } else if (lane < 18) {
      cx<V>* o = in.sa[s];
      o[FRG_IN_PZ] = m0;  o[FRG_IN_FP] = d0; o[FRG_IN_HP] = d1;  o[FRG_IN_BD] = d2;
      o[FRG_IN_EBD] = m1; o[FRG_IN_CG] = d3; o[FRG_IN_ECG] = m2; o[FRG_IN_V] = w;
    }
  }
}

// u . Y over the first n entries in the point type: lane g of each group of 8 adds its
// entries g, g + 8, g + 16 in turn, then the group sums (htpysupport.cu:9-34, :446).
template <typename T, typename P>
__device__ __forceinline__ cx<P> patch_dot(const cx<T>* u, const cx<P>* Y, int n, int g, unsigned mask) {
  cx<P> d(P(0));
  for (int e = g; e < n; e += TEAM) d = cfma(cx<P>(u[e]), Y[e], d);
  return cx<P>(team_sum(mask, d.re), team_sum(mask, d.im));
}

// The corrector's refinement residual of one path (F_j at the point YN, htpysupport.cu:64-86)
// in the point type, by the four warps of its part: warp `part` runs its generated schedule,
// lane 2 o + c computing component c of a step's operation o, from what eval_prep<true> left
// in the path's inputs. The temporaries take the vectors that a corrector step does not need
// (X .. k), then the place of the inputs that the schedules compute themselves.
// What bounds it: the chain of operations, 200 to 250 cycles each. As straight-line code, a
// group's three equations on a lane of three warps after the hoisted quantities on one, it was
// 52 operations long in 13 % of a path's steps, and of 16 paths in step nearly always one is
// in such a step; the schedule has 17 steps (3.8k cycles). GB300, FP32 stage of 140 paths
// 113 -> 104 ms, of 2,400 236 -> 213, of 9,600 333 -> 282, and with the hoisted quantities in
// the schedules 203 -> 191 and 293 -> 256; 65,536-path rounds, four in flight, 1,448 -> 1,365
// and 1,349 -> 1,311 ms a round.
template <typename P>
struct Residual {
  typedef Smem<float, P> S;
  static constexpr unsigned kY = offsetof(S, YN) / 16, kT = offsetof(S, X) / 16,
                            kIn = (offsetof(S, work) + offsetof(typename S::Inputs, hi)) / 16;
  static_assert(sizeof(cx<P>) == 16 && offsetof(S, YN) % 16 == 0 && offsetof(S, X) % 16 == 0 &&
                offsetof(S, work) % 16 == 0 && offsetof(typename S::Inputs, hi) % 16 == 0, "16-byte units");
  static constexpr unsigned kFirst = (offsetof(S, k) + sizeof(S::k)) / 16 - kT,  // temporaries in X .. k
                            kFree = kIn + offsetof(FrgEvalIn<P>, sa) / 16;
  static_assert(FRG_RESIDUAL_TEMPS - kFirst <= sizeof(FrgEvalIn<P>) / 16 - offsetof(FrgEvalIn<P>, sa) / 16, "temporaries");
  static constexpr unsigned y(unsigned i) { return kY + i; }
  static constexpr unsigned in(unsigned i) { return kIn + i; }
  static constexpr unsigned t(unsigned i) { return i < kFirst ? kT + i : kFree + (i - kFirst); }
  static_assert(kIn + sizeof(FrgEvalIn<P>) / 16 <= 1024, "10-bit units");
};
static_assert(Residual<df>::kY == Residual<double>::kY && Residual<df>::kT == Residual<double>::kT &&
              Residual<df>::kIn == Residual<double>::kIn, "one table for both point types");
#define FRG_OP(r, a, b, sub, mul) (unsigned)(r) | (unsigned)(a) << 10 | (unsigned)(b) << 20 | sub##u << 30 | mul##u << 31
#define FRG_OUT(r, eq, g, minus) (r) | (g) << 10 | (eq) << 13 | (minus) << 15
static __device__ const unsigned residual_code[] = {FRG_RESIDUAL_CODE(FRG_OP, Residual<df>::y, Residual<df>::in, Residual<df>::t)};
static __device__ const unsigned short residual_outs[] = {FRG_RESIDUAL_OUTS(FRG_OUT, Residual<df>::t)};
#undef FRG_OP
#undef FRG_OUT

// component im of a b
__device__ __forceinline__ df mul_comp(cx<df> a, cx<df> b, bool im) {
  return df_dot2(a.re, im ? b.im : b.re, neg_if(a.im, !im), im ? b.re : b.im, 1.f);
}
__device__ __forceinline__ double mul_comp(cx<double> a, cx<double> b, bool im) {
  return fma(a.re, im ? b.im : b.re, mul_rn(neg_if(a.im, !im), im ? b.re : b.im));
}
__device__ __forceinline__ cx<df> load_point(const cx<df>* p) {
  const float4 v = *reinterpret_cast<const float4*>(p);
  return cx<df>(df(v.x, v.y), df(v.z, v.w));
}
__device__ __forceinline__ cx<double> load_point(const cx<double>* p) {
  const double2 v = *reinterpret_cast<const double2*>(p);
  return cx<double>(v.x, v.y);
}

__device__ __forceinline__ void put_comp(cx<df>* p, bool im, df r) {
  reinterpret_cast<float2*>(p)[im] = make_float2(r.hi, r.lo);
}
__device__ __forceinline__ void put_comp(cx<double>* p, bool im, double r) { reinterpret_cast<double*>(p)[im] = r; }

template <typename P>
__device__ __forceinline__ void residual_part(Smem<float, P>& E, int part, int lane) {
  constexpr int start[5] = FRG_RESIDUAL_START;
  cx<P>* const base = reinterpret_cast<cx<P>*>(&E);
  const int from = part == 0 ? start[0] : (part == 1 ? start[1] : (part == 2 ? start[2] : start[3]));
  const int to = part == 0 ? start[1] : (part == 1 ? start[2] : (part == 2 ? start[3] : start[4]));
  const bool im = lane & 1;
  const unsigned* code = residual_code + from * 16 + (lane >> 1);
  unsigned w = __ldg(code), wn = __ldg(code + 16);  // two steps ahead; two steps of padding end the list
#pragma unroll 1
  for (int i = from; i < to; ++i) {
    code += 16;
    const unsigned wm = __ldg(code + 16);
    const cx<P> a = load_point(base + ((w >> 10) & 1023)), b = load_point(base + ((w >> 20) & 1023));
    P r;
    if (w >> 31) {
      r = mul_comp(a, b, im);
    } else {
      r = (im ? a.im : a.re) + neg_if(im ? b.im : b.re, (w >> 30) & 1);
    }
    put_comp(base + (w & 1023), im, r);
    __syncwarp();
    w = wn;
    wn = wm;
  }
  const unsigned o = lane < 7 ? residual_outs[part * 7 + lane] : 0xffffu;
  if (o != 0xffffu) {
    const cx<P> v = load_point(base + (o & 1023));
    E.R[(o >> 13) & 3][(o >> 10) & 7] = cx<float>(cx<P>(neg_if(v.re, o >> 15), neg_if(v.im, o >> 15)));
  }
}

// 1 / max(|re|, |im|) of the projective patch, its row's scale in every step
template <typename T>
__device__ __forceinline__ T patch_scale(const cx<T>* u, int lane) {
  MaxAbs<T> m;
  if (lane < NY) m.take(u[lane]);
  for (int off = 16; off >= 1; off >>= 1) m.across(off);
  return T(1) / m.value();
}

// Pivot search: the row with the largest v (ties: the lowest), as its lane's bit. Row r's
// value is on lane base + r, v >= 0 or NaN, or -1 for used rows; the other lanes hold -1. The
// values' bits as integers have their order; a NaN comes out above infinity or, with a
// negative sign, below zero, but never below the -1 of a used row: such a row must not win, or a
// later part of the elimination finds more unused rows than it has room for. (Which of the
// others wins then is all the same, the step has no finite solution.) A branch to a search of
// its own for infinities and NaN cost 50 cycles a pivot: the FP32 stage of 140 paths 104 -> 100
// ms, of 2,048 200 -> 191, of 9,600 267 -> 257.
__device__ __forceinline__ unsigned pivot_lane(float v) {
  const int key = __float_as_int(v);
  const unsigned c = __ballot_sync(FULL, key == __reduce_max_sync(FULL, key));
  return c & (0u - c);
}
__device__ __forceinline__ unsigned pivot_lane(double v) {
  const int hi = __double2hiint(v);
  const unsigned lo = (unsigned)__double2loint(v);
  const int m = __reduce_max_sync(FULL, hi);
  unsigned c = __ballot_sync(FULL, hi == m);
  if (c & (c - 1)) {
    const unsigned ml = __reduce_max_sync(FULL, hi == m ? lo : 0u);
    c = __ballot_sync(FULL, hi == m && lo == ml);
  }
  return c & (0u - c);
}

// a * b where lanes that differ in `bit` hold the same operands: in FP64 each computes one
// component (the same operations as the complex product's) and they exchange
__device__ __forceinline__ cx<float> mul_split(cx<float> a, cx<float> b, int, int) { return a * b; }
__device__ __forceinline__ cx<double> mul_split(cx<double> a, cx<double> b, int lane, int bit) {
  const bool im = lane & bit;
  const double own = fma(a.re, im ? b.im : b.re, __dmul_rn(neg_if(a.im, !im), im ? b.re : b.im));
  const double ot = __shfl_xor_sync(FULL, own, bit);
  return im ? cx<double>(ot, own) : cx<double>(own, ot);
}

// Four steps k0..k0 + 3 of the dense elimination of RP rows, W columns per lane. Lane
// RP h + r holds row r's remaining columns c = h mod 32 / RP (the right-hand side is column
// 16) from index 0; a step drops the pivot column, so the lanes that held it move their
// window up one. The pivot row goes to U and every lane reads it back from there; U[k][k]
// keeps the pivot's reciprocal; pn and pv (16 entries) pass the pivot and its norm on. In
// FP32 the steps are chains of latencies (search, reciprocal, memory), in FP64 of the
// FP64 instructions: 9 for the reciprocal and factor, 4 per column.
template <int W, int RP, typename T>
__device__ __forceinline__ void lu_stage(cx<T>* U, T* pn, cx<T>* pv, int k0, int lane, cx<T>* R, bool& used,
                                         T& pmax, T& pmin) {
  constexpr int CL = 32 / RP;
  const int h = lane / RP, r = lane % RP;
#pragma unroll 1
  for (int k = k0; k < k0 + 4; ++k) {
    const int base = (k & (CL - 1)) * RP;  // the lanes that hold column k
    const bool own = h == (k & (CL - 1)), cand = own && !used;
    const T v = cand ? cnorm2(R[0]) : T(-1);
    const cx<T> e = warp_shfl(R[0], base + r);  // this row's entry in column k
    // FP32: every candidate's reciprocal is taken while the pivot is searched for
    cx<T> ip = R[0];
    if constexpr (sizeof(T) == 4) ip = cinv(cand ? R[0] : cx<T>(T(1)));
    const unsigned pl = pivot_lane(v);
    cx<T>* Uk = U + k * LDU + k + 1 + ((h - (k + 1)) & (CL - 1));
    cx<T> X[W], pivot[W];
#pragma unroll
    for (int i = 0; i < W; ++i) X[i] = own ? R[i + 1] : R[i];
    if ((pl >> (base + r)) & 1) {
      used = true;
#pragma unroll
      for (int i = 0; i < W; ++i) Uk[CL * i] = X[i];
      if (own) {
        (sizeof(T) == 4 ? U[k * LDU + k] : pv[k]) = ip;
        pn[k] = v;
      }
    }
    __syncwarp();
    ip = sizeof(T) == 4 ? U[k * LDU + k] : pv[k];
    const T pa = pn[k];
#pragma unroll
    for (int i = 0; i < W; ++i) pivot[i] = Uk[CL * i];
    if constexpr (sizeof(T) == 8) {
      ip = cinv_norm(ip, pa);
      if (lane == 0) U[k * LDU + k] = ip;
    }
    pmax = max_mag(pmax, pa);
    pmin = min_mag(pmin, pa);
    const cx<T> el = mul_split(e, ip, lane, RP), l = used ? cx<T>(T(0)) : el;
#pragma unroll
    for (int i = 0; i < W; ++i) R[i] = cfms(X[i], l, pivot[i]);
  }
}

// Dense 16 x 16 LU with partial pivoting across the lanes. Eight steps with two lanes a
// row, then the eight remaining rows, in their order, with four lanes a row: 68 complex
// updates per lane (80 with two lanes a row throughout; the triangle needs 64).
template <typename T>
__device__ __forceinline__ void dense_lu(cx<T>* U, T* pn, cx<T>* pv, int lane, T& pmax, T& pmin) {
  cx<T> R[9];
  bool used = false;
  {
    const int h = lane >> 4, r = lane & 15;
#pragma unroll
    for (int i = 0; i < 8; ++i) R[i] = U[r * LDU + h + 2 * i];
    R[8] = h == 0 ? U[r * LDU + 16] : cx<T>(T(0));
    __syncwarp();
    lu_stage<8, 16>(U, pn, pv, 0, lane, R, used, pmax, pmin);
    lu_stage<6, 16>(U, pn, pv, 4, lane, R, used, pmax, pmin);
    // columns 8 + h, 10 + h, ... of the unused rows to rows 8..15 of U
    const unsigned left = ~__ballot_sync(FULL, used) & 0xffffu;
    if (!used) {
      cx<T>* d = U + (8 + __popc(left & ((1u << r) - 1))) * LDU + 8 + h;
#pragma unroll
      for (int i = 0; i < 4; ++i) d[2 * i] = R[i];
      if (h == 0) d[8] = R[4];
    }
    __syncwarp();
  }
  const int h = lane >> 3, r = lane & 7;
  R[0] = U[(8 + r) * LDU + 8 + h];
  R[1] = U[(8 + r) * LDU + 12 + h];
  R[2] = h == 0 ? U[(8 + r) * LDU + 16] : cx<T>(T(0));
  __syncwarp();
  used = false;
  lu_stage<2, 8>(U, pn, pv, 8, lane, R, used, pmax, pmin);
  lu_stage<1, 8>(U, pn, pv, 12, lane, R, used, pmax, pmin);
}

// Sums over each group of 8 lanes (g = lane & 7) of N values a lane, those of team_sum, to
// out[0..N) in memory: the lanes halve the values among themselves three times, N - 1 or so
// additions a lane where a butterfly per value takes 3 N.
template <int N, typename T>
__device__ __forceinline__ void halve(T* v, bool up, int off) {
  constexpr int H = (N + 1) / 2;
#pragma unroll
  for (int i = 0; i < H; ++i) {
    const T hi = H + i < N ? v[H + i] : T(0);
    const T keep = up ? hi : v[i], send = up ? v[i] : hi;
    v[i] = keep + __shfl_xor_sync(FULL, send, off);
  }
}
template <int N, typename T>
__device__ __forceinline__ void team_sums(T* v, T* out, int g) {
  constexpr int H = (N + 1) / 2, H2 = (H + 1) / 2, H3 = (H2 + 1) / 2;
  halve<N>(v, g & 4, 4);
  halve<H>(v, g & 2, 2);
  halve<H2>(v, g & 1, 1);
  const int end = (g & 4) ? N : H;  // this lane's values: first .. first + H3, within its halves
  const int mid = (g & 4 ? H : 0) + (g & 2 ? H2 : 0), last = (g & 2) ? end : mid + H2;
  const int first = mid + (g & 1 ? H3 : 0), stop = (g & 1) ? last : mid + H3;
#pragma unroll
  for (int i = 0; i < H3; ++i)
    if (first + i < (stop < end ? stop : end)) out[first + i] = v[i];
}

// Back substitution, column by column; lane r holds the right-hand side of pivot row r.
// FP32: both halves of the warp do the same.
__device__ __forceinline__ void back_substitute(const cx<float>* U, cx<float>* X, int lane) {
  const int r = lane & 15;
  cx<float> rb = U[r * LDU + 16];
  const cx<float> ip = U[r * LDU + r];
#pragma unroll 4
  for (int k = 15; k >= 0; --k) {
    const cx<float> xk = warp_shfl(rb * ip, k), next = cfms(rb, U[r * LDU + k], xk);
    if (r < k) rb = next;
  }
  if (lane < 16) X[lane] = rb * ip;
}
// FP64: lanes 0..15 hold the real parts, lanes 16..31 the imaginary parts, which halves
// the FP64 instructions of the chain (4 per column; the operations and their order are
// those of the complex product and cfms).
__device__ __forceinline__ void back_substitute(const cx<double>* U, cx<double>* X, int lane) {
  const int r = lane & 15;
  const bool im = lane >= 16;
  double rb = im ? U[r * LDU + 16].im : U[r * LDU + 16].re;
  const cx<double> ip = U[r * LDU + r];
  const double pa = im ? ip.im : ip.re, pb = im ? ip.re : neg_if(ip.im, true);
  double x = 0.0;
#pragma unroll 1
  for (int k = 15; k >= 0; --k) {
    const cx<double> u = U[r * LDU + k];
    const double ot = __shfl_xor_sync(FULL, rb, 16);
    const double are = im ? ot : rb, aim = im ? rb : ot;
    const double m = fma(are, pa, __dmul_rn(aim, pb));
    const double xr = __shfl_sync(FULL, m, k), xi = __shfl_sync(FULL, m, 16 + k);
    if (k == r) x = m;  // row k's right-hand side is final
    if (r < k) rb = fma(neg_if(u.im, im), im ? xr : xi, fma(-u.re, im ? xi : xr, rb));
  }
  reinterpret_cast<double*>(&X[r])[im] = x;
}

// U_j from the group's pivot row, lane g of each group of 8 (every such lane returns it)
__device__ __forceinline__ cx<float> solve_u(const cx<float>* piv, const cx<float>* X, cx<float> ipu, int lane) {
  const int g = lane & 7;
  cx<float> xu = piv[16 * 8 + g];
#pragma unroll 4
  for (int c = 0; c < 16; ++c) xu = cfms(xu, piv[c * 8 + g], X[c]);
  return xu * ipu;
}
__device__ __forceinline__ cx<double> solve_u(const cx<double>* piv, const cx<double>* X, cx<double> ipu, int lane) {
  const int g = lane & 7;
  const bool im = lane & 8;
  double xu = im ? piv[16 * 8 + g].im : piv[16 * 8 + g].re;
#pragma unroll 4
  for (int c = 0; c < 16; ++c) {
    const cx<double> p = piv[c * 8 + g], x = X[c];
    xu = fma(neg_if(p.im, im), im ? x.re : x.im, fma(-p.re, im ? x.im : x.re, xu));
  }
  const double ot = __shfl_xor_sync(FULL, xu, 8);
  return (im ? cx<double>(ot, xu) : cx<double>(xu, ot)) * ipu;
}

// One linear-system solve of the warp's path from the group rows in S.M, evaluated at
// S.Ye:
//   tangent (newton = false): [JH; W] x = e_23 with W = the velocity patch Wsrc,
//     then normalised to unit length with real dt/ds (or dt = 1 when tstep),
//     Im(dt) = 0 (htpysupport.cu:237-299);
//   Newton (newton = true): [JH; e_t] x = [-H; tgoal - t] (htpysupport.cu:427-477),
//     H from S.M, or from the refined residuals S.R, S.Rd at S.YN when `hires`.
// su = patch_scale(S.u). The solution is written to dst[0..22]. `newton`, `tstep`,
// `hires` and the results are the same in every lane.
template <typename T, typename P>
__device__ __forceinline__ StepOut<T> solve_step(Smem<T, P>& S, const cx<T>* Wsrc, cx<T>* dst, bool newton,
                                                 bool tstep, T tgoal, T su, bool hires, bool want_ratio,
                                                 bool want_hnorm, int lane) {
  const int g = lane & 7, q = lane >> 3;
  const bool grp = g < 7;
  const int jj = grp ? g : 6;
  const cx<T> zero(T(0));
  StepOut<T> out;

  // ---- the group's three rows, columns q, q + 4, q + 8, q + 12, then U_j and the rhs
  cx<T> r0[6], r1[6], r2[6];
#pragma unroll
  for (int i = 0; i < 5; ++i) {
    const int c = i < 4 ? q + 4 * i : 16;
    r0[i] = S.M[c * 8 + jj];
    r1[i] = S.M[(18 + c) * 8 + jj];
    r2[i] = S.M[(36 + c) * 8 + jj];
  }
  r0[5] = r1[5] = r2[5] = zero;
  cx<T> hU = zero;
  out.hnorm = T(0);
  if (newton) {
    cx<T> f0, f1, f2;
    if (hires) {
      f0 = S.R[0][jj]; f1 = S.R[1][jj]; f2 = S.R[2][jj];
      hU = S.Rd;
    } else {
      f0 = S.M[17 * 8 + jj]; f1 = S.M[(18 + 17) * 8 + jj]; f2 = S.M[(36 + 17) * 8 + jj];
      hU = patch_dot<T, T>(S.u, S.Ye, NY, g, FULL) - cx<T>(T(1));
    }
    r0[5] = neg(f0); r1[5] = neg(f1); r2[5] = neg(f2);
    if (want_hnorm) {
      const T hsq = grp ? cnorm2(f0) + cnorm2(f1) + cnorm2(f2) : cnorm2(hU);
      out.hnorm = sqrt(team_sum(FULL, hsq));
    }
  }
  // ---- row scaling by 1/max(|re|,|im|) (htpysupport.cu:259-277, :446-471); the three
  //      reciprocals in one division, row q on lane 8 q + g
  {
    MaxAbs<T> m0, m1, m2;
#pragma unroll
    for (int i = 0; i < 5; ++i) { m0.take(r0[i]); m1.take(r1[i]); m2.take(r2[i]); }
    m0.across(8); m1.across(8); m2.across(8);
    m0.across(16); m1.across(16); m2.across(16);
    const T s = T(1) / (q == 0 ? m0.value() : (q == 1 ? m1.value() : m2.value()));
    const T s0 = __shfl_sync(FULL, s, g), s1 = __shfl_sync(FULL, s, 8 + g), s2 = __shfl_sync(FULL, s, 16 + g);
#pragma unroll
    for (int i = 0; i < 5; ++i) { r0[i] = s0 * r0[i]; r1[i] = s1 * r1[i]; r2[i] = s2 * r2[i]; }
    if (newton) { r0[5] = s0 * r0[5]; r1[5] = s1 * r1[5]; r2[5] = s2 * r2[5]; }
  }
  // ---- eliminate U_j inside the group: partial pivoting among its three rows (a tangent's
  //      group rows have the right-hand side zero throughout)
  const T a0 = cnorm2(r0[4]), a1 = cnorm2(r1[4]), a2 = cnorm2(r2[4]);
  const int p = (a0 >= a1 && a0 >= a2) ? 0 : (a1 >= a2 ? 1 : 2);
  const T ap = p == 0 ? a0 : (p == 1 ? a1 : a2);
  cx<T> piv[6], R0[5], R1[5];  // [4] of R0, R1: the right-hand side
#pragma unroll
  for (int i = 0; i < 6; ++i) piv[i] = p == 0 ? r0[i] : (p == 1 ? r1[i] : r2[i]);
  cx<T> ipu = cinv_norm(piv[4], ap);
  {
    const cx<T> la = (p == 0 ? r1[4] : r0[4]) * ipu;
    const cx<T> lb = (p == 2 ? r1[4] : r2[4]) * ipu;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      R0[i] = cfms(p == 0 ? r1[i] : r0[i], la, piv[i]);
      R1[i] = cfms(p == 2 ? r1[i] : r2[i], lb, piv[i]);
    }
    R0[4] = R1[4] = zero;
    if (newton) {
      R0[4] = cfms(p == 0 ? r1[5] : r0[5], la, piv[5]);
      R1[4] = cfms(p == 2 ? r1[5] : r2[5], lb, piv[5]);
    }
  }
  cx<T>* pivs = S.piv();
  if (grp) {
#pragma unroll
    for (int i = 0; i < 4; ++i) pivs[(q + 4 * i) * 8 + g] = piv[i];
    if (q == 0) pivs[16 * 8 + g] = piv[5];
  }
  // ---- the folding of every group's pivot row into the patch rows (lanes g = 7 repeat
  //      group 7's rows with weight zero and then hold the patch rows). A Newton step's
  //      t-selector row has no entry to fold, a tangent's right-hand sides none either.
  cx<T>* U = S.U();
  if (!grp) ipu = zero;
  {
    T* sums = reinterpret_cast<T*>(U) + q * 16;  // the dense system's place, free until it is written
    const cx<T> mu = (su * S.u[14 + jj]) * ipu;
    T v[16];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const cx<T> m = mu * piv[i];
      v[2 * i] = m.re;
      v[2 * i + 1] = m.im;
    }
    if (newton) {
      const cx<T> m = mu * piv[5];
      v[8] = m.re;
      v[9] = m.im;
      team_sums<10>(v, sums, g);
    } else {
      const cx<T> mw = Wsrc[14 + jj] * ipu;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const cx<T> m = mw * piv[i];
        v[8 + 2 * i] = m.re;
        v[9 + 2 * i] = m.im;
      }
      team_sums<16>(v, sums, g);
    }
    __syncwarp();
    if (!grp) {
      const cx<T>* Su = reinterpret_cast<const cx<T>*>(sums);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int c = q + 4 * i, st = gstate(c);
        R0[i] = su * S.u[st] - Su[i];
        R1[i] = newton ? (c == 15 ? cx<T>(T(1)) : zero) : Wsrc[st] - Su[4 + i];
      }
      R0[4] = newton ? -mul_rn(su, hU) - Su[4] : zero;
      R1[4] = newton ? cx<T>(tgoal - S.Ye[22].re) : cx<T>(T(1));
    }
    __syncwarp();
  }
  // ---- re-scale the 16 dense rows (max(|re|,|im|) = 1): eliminating U_j can shrink a
  //      group row by cancellation, and unequal rows would mislead both the pivot
  //      choice and the pivot-ratio condition estimate (with the re-scaling the ratio
  //      tracks the reference's 23 x 23 row-scaled elimination). Rows 2 g and 2 g + 1 to
  //      the dense system.
  {
    MaxAbs<T> m0, m1;
#pragma unroll
    for (int i = 0; i < 4; ++i) { m0.take(R0[i]); m1.take(R1[i]); }
    m0.across(8); m1.across(8);
    m0.across(16); m1.across(16);
    const T s = T(1) / ((q & 1) ? m1.value() : m0.value());
    const T s0 = __shfl_sync(FULL, s, g), s1 = __shfl_sync(FULL, s, 8 + g);
#pragma unroll
    for (int i = 0; i < 5; ++i) {
      R0[i] = s0 * R0[i];
      R1[i] = s1 * R1[i];
      if (i < 4 || q == 0) {
        const int c = i < 4 ? q + 4 * i : 16;
        U[(2 * g) * LDU + c] = R0[i];
        U[(2 * g + 1) * LDU + c] = R1[i];
      }
    }
  }
  __syncwarp();
  // ---- dense 16 x 16 LU with partial pivoting across the lanes
  T pmax = T(0), pmin = T(3.0e38);
  dense_lu(U, S.cn, S.X, lane, pmax, pmin);
  __syncwarp();
  back_substitute(U, S.X, lane);
  __syncwarp();
  const cx<T> xu = solve_u(pivs, S.X, ipu, lane);
  if (lane < 16) S.cn[lane] = cnorm2(S.X[lane]);
  if (lane < 8) S.XU[lane] = xu;
  __syncwarp();
  T n2 = T(0);
#pragma unroll
  for (int c = 0; c < 16; ++c) n2 += S.cn[c];
  n2 += team_sum(FULL, grp ? cnorm2(xu) : T(0));
  // ---- condition estimate: the larger of the dense phase's pivot ratio and the
  //      worst group amplification 1/|u_jj| (a group's pivot row is row-scaled, so its
  //      largest entry is about 1, and U_j's error grows like eps / |u_jj|). A
  //      non-finite solution (zero or non-finite pivot) makes it infinite.
  out.ratio = T(0);
  if (want_ratio) {
    const T ig = grp ? T(1) / ap : T(0);
    const T ratio = sqrt(fmax(pmax / pmin, team_max(FULL, ig)));
    out.ratio = (n2 - n2 == T(0)) ? ratio : T(INFINITY);  // n2 - n2 is NaN iff n2 is not finite
  }
  out.xnorm2 = n2;
  // ---- normalisation and output, one entry per lane
  cx<T> sc(T(1));
  if (!newton) {
    const cx<T> xt = S.X[15];
    if (!tstep) {
      const T nr = sqrt((lane & 1) ? n2 : cnorm2(xt));
      sc = cx<T>(xt.re, neg_if(xt.im, true)) * (T(1) / (__shfl_sync(FULL, nr, 0) * __shfl_sync(FULL, nr, 1)));
    } else {
      sc = cinv(xt);
    }
  }
  if (lane < NY) {
    cx<T> x = lane < 14 ? S.X[lane] : (lane < 21 ? S.XU[lane - 14] : S.X[lane - 7]);
    if (!newton) {
      x = sc * x;
      if (lane == 22) x.im = T(0);
    }
    dst[lane] = x;
  }
  __syncwarp();
  return out;
}

}  // namespace team
}  // namespace frg
