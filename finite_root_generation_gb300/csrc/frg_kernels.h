// Internal interface between the C ABI (frg_capi.cu) and the tracking kernels.
#pragma once

#include <cuda_runtime.h>
#include <limits.h>
#include <stdint.h>

#include "../../include/frg_gb300.h"
#include "frg_complex.cuh"
#include "frg_df.cuh"
#include "frg_mlp.cuh"

#ifndef FRG_TRACK_THREADS
#define FRG_TRACK_THREADS 64
#endif
#define FRG_START_THREADS 64

namespace frg {

// Saved state of a path handed from the FP32 stage to the FP64 stage: what the
// reference's tracker carries across loop iterations (htpytrack.cu:36-77).
struct Handoff {
  cx<double> Yc[23], Vc[23], u[23];
  double s;
  uint64_t rng_index;
  int streak, step, ministep, tstepQ, n_ivp, n_newton, reason, code;  // reason 6: finished with code
  int bounces, pad;  // times the path returned from FP64 to FP32
  int64_t id;        // the path (tail records)
};

// Device-side arguments of one tracking launch. All arrays are device memory.
constexpr int FRG_START_STRIDE = 51;
// counters: codes[8], ivp, newton, steps, fp64 solves, handoffs, hand-backs, -, -, handoff
// reasons 1..6 at [16..21], refinement solves and warp steps at [22..23], kernel cycles at
// [24..35], retired paths at [36], FP32-stage refinement-residual cycles at [37],
// FP64-segment histogram at [40..45], longest FP64 segment at [46]
#define FRG_NCOUNTERS 48

struct TrackArgs {
  frg_config cfg;
  const cx<double>* fpm;        // ntasks x 30 target parameters
  const cx<double>* gamma;      // ntasks
  const cx<float>* fpm_lo;      // FP32 copies for the FP32 stage
  const cx<float>* gamma_lo;
  const cx<df>* fpm_df;         // double-float copies for the FP32 stage's refinement residuals
  const cx<df>* gamma_df;
  const int64_t* task_start;    // ntasks + 1 prefix sums of paths per task
  int ntasks;
  int64_t npaths;               // paths of one round
  uint64_t seed;
  // Paths are addressed by a global index gid = round * npaths + (index within the round):
  // records, lists and outputs use gid; the random stream, start values and task use the
  // index within the round; task parameters and gammas are indexed by round * ntasks + task.
  // A single call is round 0 (gid = index within the round).
  int64_t round_base;           // gid of this launch's first fresh path (round * npaths)
  const uint64_t* seeds;        // per-round seeds (null: every path uses `seed`)
  int carry;                    // FP32 stage: lo_list holds paths carried over from an earlier
                                // round's FP64 launch, taken before this round's fresh paths
  unsigned long long* queue;    // work-queue head, zeroed before launch
  cx<double>* roots;            // npaths x 21
  int32_t* codes;               // npaths
  cx<double>* yfinal;           // npaths x 23, optional
  double* resid;                // npaths, optional
  int32_t* work;                // npaths x 3 (ivp solves, newton iterations, steps), optional
  unsigned long long* counters; // FRG_NCOUNTERS counters (layout above)
  const cx<double>* starts;     // npaths x FRG_START_STRIDE start values (null: generated inline); plug-ins:
                                // npaths x (unknowns + parameters)
  cx<double>* finals;           // plug-ins: the paths' endpoints, npaths x (unknowns + 2)
  Handoff* handoff;             // npaths slots (mixed precision)
  int64_t* handoff_list;        // ids of paths handed to the FP64 kernel
  unsigned long long* handoff_count;
  const int64_t* lo_list;       // FP32 kernel: paths to resume from their saved state (null: fresh paths)
  const unsigned long long* lo_count;
  int64_t* back_list;           // FP64 kernel: paths handed back to FP32 (null: none, e.g. the last round)
  unsigned long long* back_count;
  int sms;                      // the device's SMs
  Handoff* tail;                // thread kernel: where a launch leaves its last paths (tail_cap records, 0 = none);
  unsigned long long* tail_count;  // warp kernel with from_tail: the paths it continues
  int64_t tail_cap;
  int from_tail;
  int lo_keep_ill;              // FP32 kernel: 1 = no hand-off for ill-conditioned steps (last round)
  float* feat;                  // optional: FRG_MLP_IN features per checkpoint, feat_max checkpoints per path
  int32_t* nfeat;               // checkpoints written per path (zeroed before launch)
  int feat_max;
  int feat_every;               // checkpoint every this many accepted steps (features and retirement)
  MlpDevice mlp;                // early-retirement network (mlp.w null: off)
};

}  // namespace frg

// Grid of a thread-per-path launch over n paths with at most bps blocks per SM: one warp
// per SM sub-partition while the paths fit there (the kernel then spreads them over the
// warps, one path per lane at most), beyond that one path per thread.
inline int frg_thread_grid(int sms, int bps, int64_t n) {
  const int64_t wpb = FRG_TRACK_THREADS / 32, spread = (int64_t)sms * 4;
  const int64_t want = n <= spread * 32 ? ((n < spread ? n : spread) + wpb - 1) / wpb
                                        : (n + FRG_TRACK_THREADS - 1) / FRG_TRACK_THREADS;
  const int64_t cap = (int64_t)sms * bps;
  const int64_t grid = want < cap ? want : cap;
  return (int)(grid < 1 ? 1 : grid);
}

// Grid of a team launch (a warp per path) over at most n paths, with at most bps blocks of
// four warps per SM: one block per SM until its warps are taken, then as many as fit. In
// the FP32 stage (lo) a block grows with the paths per SM, from 4 warps to 16.
struct TeamGrid { int blocks, warps; };
inline TeamGrid frg_team_grid(int sms, int64_t bps, int64_t n, bool lo) {
  const int64_t most = lo ? (bps < 4 ? 4 * bps : 16) : 4, per_sm = (n + sms - 1) / sms;
  int64_t warps = (per_sm + 3) / 4 * 4;
  warps = warps < 4 ? 4 : (warps < most ? warps : most);
  const int64_t want = n <= sms * warps ? (n < sms ? n : sms) : (n + warps - 1) / warps;
  const int64_t per = 4 * bps / warps, cap = sms * (per < 1 ? 1 : per);
  const int64_t blocks = want < cap ? want : cap;
  return {(int)(blocks < 1 ? 1 : (blocks < INT_MAX ? blocks : INT_MAX)), (int)warps};
}

// Grid of a warp-per-path launch of a plug-in over at most n paths, four to a block.
inline int frg_warp_grid(int sms, int64_t bps, int64_t n) {
  const int64_t want = (n + 3) / 4, cap = sms * bps, blocks = want < cap ? want : cap;
  return (int)(blocks < INT_MAX ? blocks : INT_MAX);
}

// A plug-in's call is tracked in pieces of at most this many paths, so that its start values
// and endpoints (288 B a path for conic2, 512 B for burmester5; in mixed precision 1.2 KB of
// records more) never take more than 8.6 GB (29 GB), whatever the call. The last paths of each
// piece leave the GPU partly idle: 16.8 M conic2 paths in FP64 take 4,454 ms in one piece and 4,510
// in two, in mixed precision 1,410 and 1,408.
constexpr int64_t FRG_PLUGIN_PIECE = (int64_t)1 << 24;

// A plug-in launch of at most this many paths per SM sub-partition tracks a path per warp,
// a larger one a path per thread and its last paths per warp. GB300 (152 SMs), warp / thread,
// medians of three seeds, FP64: conic2 2,432 paths 14.8 / 18.4 ms, 4,864 25.1 / 25.7, 9,728
// 28.8 / 27.3, 14,592 33.4 / 28.4; burmester5 4,864 89 / 112, 9,728 402 / 422, 14,592 426 / 429,
// 19,456 450 / 434. Mixed: conic2 4,864 2.6 / 3.1, 9,728 3.9 / 3.6, 14,592 5.5 / 4.1; burmester5
// 9,728 379 / 409, 19,456 393 / 414. One line for all: at 9,728 paths conic2 loses a twentieth by
// it and burmester5 gains as much.
constexpr int FRG_WARP_PATHS = 16;

// A warp of a thread-per-path launch gives its paths up to a warp-per-path launch when the
// queue is empty and at most this many of its lanes still track one: a warp's step costs
// the same with few lanes as with 32, four to seven times a warp_kernel step in FP64.
// FP64, 4 / 8 / 12 lanes: 19,456 conic2 paths 46.2 / 43.7 ms, 262,144 116.0 / 115.5 / 115.9,
// 131,072 burmester5 paths 652 / 639 / 642. FP32 stage of 120,000 conic2 paths, never / 2 / 3
// lanes: 8.2 / 7.7 / 7.2 ms.
__host__ __device__ constexpr int frg_tail_lanes(bool fp32) { return fp32 ? 4 : 8; }

#define FRG_NQUEUE 16  // queue heads and counts of a slot

// A plug-in call's start values (before its tracking launches) and its paths' roots, codes
// and residuals from `finals` and the codes tracking ended with (after them).
cudaError_t frg_launch_plugin_starts(const frg::TrackArgs& args, cx<double>* starts, cudaStream_t stream);
cudaError_t frg_launch_plugin_finish(const frg::TrackArgs& args, cudaStream_t stream);

// Warp-per-path kernel of the plug-in systems (mode and arguments as frg_launch_track's),
// four paths per block.
cudaError_t frg_launch_warp(int mode, const frg::TrackArgs& args, int grid, cudaStream_t stream);
cudaError_t frg_warp_occupancy(int system, int mode, int* blocks_per_sm);

// mode: 0 plain FP64, 1 FP32 stage with handoff, 2 FP64 resume of handed-off paths
cudaError_t frg_launch_track(int mode, const frg::TrackArgs& args, int grid, cudaStream_t stream);
cudaError_t frg_track_occupancy(int mode, int* blocks_per_sm);
cudaError_t frg_launch_team(int mode, const frg::TrackArgs& args, TeamGrid grid, cudaStream_t stream);
// GenerateStart for every path into args.starts (FRG_START_STRIDE complex per path:
// the 21 start unknowns, then the 30 start parameters)
cudaError_t frg_launch_starts(const frg::TrackArgs& args, cx<double>* starts, cudaStream_t stream);
cudaError_t frg_team_occupancy(int mode, int* blocks_per_sm);
cudaError_t frg_launch_to_float(const cx<double>* in, cx<float>* out, int n, cudaStream_t stream);
cudaError_t frg_launch_to_df(const cx<double>* in, cx<df>* out, int n, cudaStream_t stream);
// Occupancy of the thread kernel of `system` (0 = Stephenson II, k = plug-in k) in `mode`
// (0 plain FP64, 1 FP32 stage, 2 FP64 resume).
cudaError_t frg_track_occupancy_system(int system, int mode, int* blocks_per_sm);
// Name, unknowns and parameters of `system`; 0 for an unknown id. Host only.
int frg_system_dims(int system, const char** name, int* nv, int* np);
// Number of systems: Stephenson II and the generated plug-ins.
int frg_system_count();
// Validates a run configuration (every field frg_create and frg_set_config accept);
// ctx may be null, otherwise it receives the error text.
frg_status frg_check_config(frg_ctx* ctx, const frg_config* c);
