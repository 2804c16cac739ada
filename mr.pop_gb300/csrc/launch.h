// launch.h -- host-side launch interface between the C ABI and the kernel
// instantiations (one translation unit per arm count, compiled in parallel).
#pragma once
#include <cuda_runtime.h>

#include "edge_kernel.cuh"

namespace mrpop {

// Which kernel to launch.
// kFusedPair: the fused kernel with two warps per edge (granularity above 32);
// timed as kFused.
// kArmwise: the fused kernel with one warp per arm; timed as kFused.
// kRows: the rows kernel that follows kNarrow for more than one arm; timed as
// kNarrow.
// kNarrowAll: kNarrow and kRows in one kernel; timed as kNarrow.
enum KernelKind { kFused = 0, kBroad = 1, kNarrow = 2, kFusedPair = 3, kArmwise = 4, kRows = 5, kNarrowAll = 6 };

// Launch a validator kernel for `arms` arms (1..5).  smem_bytes: dynamic
// shared memory (staged scene + per-warp scratch).  Returns the launch error.
cudaError_t launch_validate(int arms, KernelKind kind, const EdgeParams &p, size_t smem_bytes, cudaStream_t stream);

template <int A>
cudaError_t launch_validate_arms(KernelKind kind, const EdgeParams &p, size_t smem_bytes, cudaStream_t stream);

// Batch kernels (BatchParams: the instances of one arm count, samples per
// lane and segmentation kind; mode = kBatchBroad / kBatchNarrow / kBatchRows / kBatchFused,
// seg = segmented instances): resident CTAs per SM at a shared-memory size
// and CTA size (warps of 32 threads, 1..kWarpsPerBlock), and a launch on
// `grid` CTAs of `warps` warps.  The dispatchers switch on the arm count
// (api.cu).
cudaError_t batch_occupancy(int arms, int mode, bool seg, int spl, size_t smem_bytes, int warps, int *blocks_per_sm);
cudaError_t launch_batch(int arms, int mode, bool seg, int spl, const BatchParams &b, size_t smem_bytes, int grid,
                         int warps, cudaStream_t stream);
template <int A>
cudaError_t batch_occupancy_arms(int mode, bool seg, int spl, size_t smem_bytes, int warps, int *blocks_per_sm);
template <int A>
cudaError_t launch_batch_arms(int mode, bool seg, int spl, const BatchParams &b, size_t smem_bytes, int grid,
                              int warps, cudaStream_t stream);

}  // namespace mrpop

#include "../../include/mrpop.h"

namespace mrpop {

// Argument checks, parameter block and launch(es) behind every validate entry
// point (api.cu).  ext_scratch: device scratch for the single-segment
// pipeline, or nullptr to use the library's stream-ordered pool.
mrpop_status run_validator(const mrpop_scene *scene, const mrpop_robotset *robots, const float *q0,
                           const float *q1, int64_t n_edges, int g, int rule, float range, uint32_t flags,
                           int arm, uint8_t *valid, int32_t *first_hit, int32_t *n_seg_out, double *flops,
                           cudaStream_t stream, void *ext_scratch);

// Argument checks and the parameter block of one validate call (run_validator
// and the batch path).  A = arm count of the check, smem = dynamic shared
// memory of its kernels.  n_edges == 0 passes.
mrpop_status make_params(const mrpop_scene *scene, const mrpop_robotset *robots, const float *q0, const float *q1,
                         int64_t n_edges, int g, int rule, float range, uint32_t flags, int arm, uint8_t *valid,
                         int32_t *first_hit, int32_t *n_seg_out, double *flops, EdgeParams &p, int &A,
                         size_t &smem);

// Shared-memory scratch of one warp (the per-CTA dynamic size is the staged
// scene plus this times the warps per CTA).
size_t warp_scratch_bytes();

// Scratch of the single-segment pipeline (staged flags, candidate masks and
// arm-pair joints): its size, and its slices in p.  Three work counters
// in a 128-byte head (every edge's flag words start on an L2 line), then per
// edge: 32 * spl samples x {env, self} flag words, {env, self} candidate
// masks, kPairSlots arm-pair words and the segment state.
constexpr size_t kSplitScratchHead = 128;
constexpr int kPairSlots = 2 * num_pairs(kMaxArms);
constexpr size_t split_scratch_bytes(int64_t n_edges, int g) {
    return kSplitScratchHead +
           (size_t)n_edges * (32 * (g > 32 ? 2 : 1) * 2 * sizeof(uint64_t) + 2 * sizeof(uint64_t) +
                              kPairSlots * sizeof(uint16_t) + 2 * sizeof(int32_t));
}
void set_split_scratch(EdgeParams &p, void *scratch, int64_t n_edges, int g);

// Largest calls whose narrow phase is one kernel (kNarrowAll) instead of
// kNarrow and kRows.  Up to some edges per resident warp each kernel of a round
// takes as long as its slowest edge, so a third kernel adds a third tail; above
// that the larger kernel's instruction fetches cost more (its hot code grows with
// the arm pairs and passes the SM's instruction cache).  Whole calls, one kernel
// against two, us: 4 arms x 32 samples, 4134 edges 164 / 202, 9000 219 / 246, 22000
// 404 / 363; 5 arms x 64, 3000 237 / 305, 6000 391 / 442, 22000 879 / 849; 5 arms x
// 32, 4134 206 / 236, 6000 282 / 280; 2 arms x 64, 24990 325 / 328, x 16 221 / 236.
// Segment rounds get emptier one by one, so their call may be twice as large:
// shortcut, 4 arms x 32, 12000 778 / 882, 26000 1257 / 1221; 5 arms x 64, 8000
// 1304 / 1441, 18000 2161 / 2070.
// Service waves, whose kernels read the endpoints from host memory (the rows kernel
// once more), device time of a wave: 2 arms x 64 connect, 4500 edges 529 / 697,
// 20000 975 / 1059; 4 arms x 64, connect 4500 738 / 941, shortcut 7200 in 12
// steps 527 / 613; above the limit, plain x 64, 20000 edges, 4 arms 715 / 662, 5
// arms 783 / 701.
constexpr int64_t one_narrow_edges(int A, bool rounds) { return 100000 / (A * A) * (rounds ? 2 : 1); }

// The dRRT / AO-x planner (drrt.cu) with any validator (validate_many, if
// not null, takes the groups of checks of the roadmap rounds in one call);
// device_nn: tree searches as a kernel on the current device, else on the host.
using check_many_fn = int (*)(void *ctx, const mrpop_check_call *calls, int n_calls);
mrpop_status drrt_run(int arms, mrpop_check_fn validate, check_many_fn validate_many, void *ctx, bool device_nn,
                      const float *start, const float *goals, int num_goals, const mrpop_drrt_settings *settings,
                      float *path_out, int64_t max_waypoints, mrpop_drrt_solution_fn on_solution, void *solution_ctx,
                      mrpop_drrt_result *out);

// Arm count of a robot set (0 for null).
int robotset_arms(const mrpop_robotset *robots);

// Records msg as the calling thread's last error and returns st.
mrpop_status fail_status(mrpop_status st, const char *msg);
// The fused-edge limit of run_validator (mrpop_set_fused_edges); returns the previous one.
int64_t set_fused_edges(int64_t max_edges);

}  // namespace mrpop
