// edge_kernel.cuh -- the batched edge validator (sm_103a).
//
// One warp owns one edge at a time; warps take edges from a per-launch work
// counter (persistent grid).  Lane L evaluates samples k = L+1 (+32) of the
// edge.  Single-segment edges run as a broad and a narrow kernel and, in large
// composite calls, a rows kernel (each a programmatic dependent of the one
// before); segmented rules run those per segment round and a fused kernel for
// the tail; small calls run one fused kernel.
//   broad phase  per lane: FK of every arm (FP32 FMA, __sinf/__cosf as the
//                reference), the 11 broad-phase spheres per arm against the
//                scene staged in shared memory (one bulk-async copy per CTA,
//                bounded mbarrier wait), the intra-arm pairs and the arm-vs-arm
//                pairs, each screened one pair per lane against swept bounds of
//                the warp's samples first; the result is a per-(arm, joint)
//                flag word and per-sample sphere counts, staged in HBM with the
//                arm pairs those bounds connect for the narrow kernel.
//   decision     per warp: shuffle reductions give the edge totals; the
//                reference's proportional 4g-thread split (utils.cuh:476-517)
//                is evaluated exactly to pick the samples that get a detailed
//                check (or every flagged sample in EXACT mode); ballots form
//                the candidate masks.
//   narrow phase lane per candidate sample: all lanes walk the arms' joint
//                chains in step (lanes without a candidate keep the others
//                company), test the detailed spheres of flagged joints against
//                obstacles that survive a warp-wide screen per sphere group,
//                the flagged intra-arm rows (the forearm-hand rows skipped
//                where a (q6, q7) table certifies them apart) and the
//                arm-vs-arm groups of the joints the broad phase left
//                connected; the first hit is the lowest set bit of a warp ballot.
// Culling: every obstacle carries a bounding sphere (1 mm margin) and every
// arm / joint group a bounding sphere computed from its own sphere set; an
// exact test is skipped only where the bounds prove it cannot fire, so the
// set of tests that can fire -- and therefore every verdict -- is unchanged.
#pragma once
#include <cstddef>
#include <type_traits>

#include "panda_model.cuh"

namespace mrpop {

#ifndef MRPOP_MIN_BLOCKS
#define MRPOP_MIN_BLOCKS 3
#endif
// CTAs per SM of the broad kernels, whose warps need half the scratch: 24 warps
// per SM at 80 registers in place of 18.
constexpr int kBroadMinBlocks = 4;
// Optional per-phase warp timers (development builds with
// -DMRPOP_PHASE_TIMERS; compiled out otherwise): clock64() deltas of lane 0
// accumulated into P.phase[i].
#ifdef MRPOP_PHASE_TIMERS
#define MRPOP_PHASE_START() long long _phase_t = clock64();
#define MRPOP_PHASE(P, i)                                                                          \
    do {                                                                                           \
        __syncwarp();                                                                              \
        const long long _n = clock64();                                                            \
        if ((P).phase && (threadIdx.x & 31) == 0)                                                  \
            atomicAdd((P).phase + (i), (unsigned long long)(_n - _phase_t));                       \
        _phase_t = _n;                                                                             \
    } while (0)
#define MRPOP_COUNT(P, i, v)                                                                       \
    do {                                                                                           \
        if ((P).phase && (threadIdx.x & 31) == 0) atomicAdd((P).phase + (i), (unsigned long long)(v)); \
    } while (0)
// counter update from code without the parameter block (warp-uniform v)
// (per translation unit; set from the parameter block by the kernel prologue)
static __device__ unsigned long long *g_dev_phase;
#define MRPOP_PHASE_BIND(P) do { if (threadIdx.x == 0) g_dev_phase = (P).phase; __syncthreads(); } while (0)
// count of lanes with pred set; the vote runs on every lane of the warp,
// only the add is lane 0's
#define MRPOP_COUNT_LANES(i, pred)                                                                 \
    do {                                                                                           \
        const uint32_t _votes = __ballot_sync(kFull, (pred));                                      \
        MRPOP_COUNT_W(i, __popc(_votes));                                                          \
    } while (0)
#define MRPOP_COUNT_W(i, v)                                                                        \
    do {                                                                                           \
        if (g_dev_phase && (threadIdx.x & 31) == 0) atomicAdd(g_dev_phase + (i), (unsigned long long)(v)); \
    } while (0)
#else
#define MRPOP_COUNT_W(i, v) do { } while (0)
#define MRPOP_PHASE_BIND(P) do { } while (0)
#define MRPOP_COUNT_LANES(i, pred) do { } while (0)
#define MRPOP_PHASE_START()
#define MRPOP_PHASE(P, i) do { } while (0)
#define MRPOP_COUNT(P, i, v) do { } while (0)
#endif

constexpr int kWarpsPerBlock = 6;
constexpr int kMaxArms = 5;
constexpr int kMaxDof = 7 * kMaxArms;
// Per-lane arm-vs-arm candidate spheres: a full stash costs another walk of both
// arms, a larger one scratch.  The arm-per-warp kernels run few CTAs and take as
// long as their slowest edge; the others fill the SMs.
constexpr int kCrossStash = 7, kArmCrossStash = 10;
constexpr float kCullMargin = 1e-3f;   // metres added to every bounding radius

struct SceneCounts {
    int n_sph, n_cap, n_zcap, n_cub, n_zcub;
};

// Float4 offsets inside the packed scene buffer: obstacle records by class,
// then one bounding sphere {cx, cy, cz, radius + margin} per obstacle in the
// order cuboids, z-cuboids, capsules, z-capsules, spheres.
struct SceneLayout {
    int sph, cap, zcap, cub, zcub;
    int b_cub, b_zcub, b_cap, b_zcap, b_sph;
    int total;
};

__host__ __device__ inline SceneLayout scene_layout(const SceneCounts &c) {
    SceneLayout l;
    l.sph = 0;
    l.cap = l.sph + c.n_sph;
    l.zcap = l.cap + 2 * c.n_cap;
    l.cub = l.zcap + 2 * c.n_zcap;
    l.zcub = l.cub + 4 * c.n_cub;
    l.b_cub = l.zcub + 4 * c.n_zcub;
    l.b_zcub = l.b_cub + c.n_cub;
    l.b_cap = l.b_zcub + c.n_zcub;
    l.b_zcap = l.b_cap + c.n_cap;
    l.b_sph = l.b_zcap + c.n_zcap;
    l.total = l.b_sph + c.n_sph;
    return l;
}

// Segmented rules: segments checked by rounds of the split kernels before the
// fused kernel takes the remaining ones.
constexpr int kSegRounds = 4;

struct EdgeParams {
    const float *q0;
    const float *q1;
    long long n_edges;
    int g;           // samples per segment
    int flags;       // MRPOP_CHECK_* | MRPOP_MODE_EXACT
    int single;      // 1: single-arm (fkcc_single_buffer_mr) semantics
    int rigid;       // bit a: arm a's base is a rigid transform near the origin (see kRegularRad)
    float cull;      // margin of the broad phase's swept bounds: kCullMargin + slack
    float slack;     // metres added to bounds of detailed spheres (0 if every base is rigid; see base_slack)
    int rule;        // MRPOP_RULE_*
    int seg0;        // segmented rules: the segment this launch checks (split kernels) or starts at (fused)
    float range;
    uint8_t *valid;
    int32_t *first_hit;
    int32_t *n_seg_out;
    double *flops;   // optional per-edge algorithmic flop tally
    double fbp;      // broad-phase flops per sample (for the tally)
    double env_test_flops;
    const float4 *scene;
    SceneCounts sc;
    unsigned int *status;
    unsigned long long *phase;  // phase timers (MRPOP_PHASE_TIMERS builds only)
    uint64_t *sflags;           // split pipeline: per-sample {env, self} flag words (32-bit for <= 4 arms)
    uint64_t *smasks;           // split pipeline: per-edge {env, self} candidate masks
    uint16_t *spairs;           // split pipeline: per-edge arm-pair joints [SPL][num_pairs(A)] (kPairSlots reserved)
    int32_t *snseg;             // segmented rules: per-edge segment count (-1: too many), from segment 0
    int32_t *sdone;             // segmented rules: per-edge verdict written
    unsigned long long *work;   // split kernels: next-edge counters {broad, narrow, rows}, zero before each launch
    const uint32_t *row5;       // forearm-hand rows table (kRow5N6 x kRow5N7 bits), or nullptr (a base is not rigid)
    float base[kMaxArms][12];   // row-major 3x4 per arm of this check
};

// Per-warp shared scratch: the edge's segment start and steps, and the broad
// phase's or the narrow phase's storage (never live at the same time).
struct EdgeScratch {
    float base[kMaxDof];   // segment start (accumulated for CONNECT)
    float stepg[kMaxDof];  // per-sample step (delta/g or vec/g)
    float delta[kMaxDof];  // per-segment step (B-spline / shortcut accumulation)
};

struct BroadPart {
    float4 swept[kMaxArms][kNumApprox]; // per-arm swept bound of each approx sphere
    float cur[kNumApprox][3][32];       // per-lane approx spheres of the current arm
};

// Scratch of the split pipeline's broad kernel, half of WarpScratch.
struct BroadScratch : EdgeScratch {
    BroadPart broad;
};

template <int STASH>
struct WarpScratchT : EdgeScratch {
    static constexpr int kStash = STASH;
    union {
        BroadPart broad;
        struct {                                // arm-per-warp kernel: the warp's own arm, both slots
            float4 swept[2][kNumApprox];
            float sp[2][kNumApprox][3][32];
        } arm;
        float stash[kDetRows][3][32];           // first sphere of each detailed self row
        struct {                                // arm-vs-arm test of one arm pair
            float gc[13][3][32];                // the upper arm's sub-group and hand part centres
            float xs[STASH][4][32];             // the lower arm's candidate spheres {x, y, z, r} ...
            uint32_t xm[STASH][32];             // ... and the upper arm's sub-groups each can reach
        } cross;
    };
};
using WarpScratch = WarpScratchT<kCrossStash>;
// store_swept reads the sphere columns 16 bytes at a time, and the scratch of the
// warps follows the scene (16-byte records)
static_assert(offsetof(BroadPart, cur) % 16 == 0 && alignof(BroadPart) >= 16 && sizeof(BroadScratch) % 16 == 0 &&
                  sizeof(WarpScratch) % 16 == 0,
              "sphere columns on 16 bytes");
using ArmScratch = WarpScratchT<kArmCrossStash>;  // arm-per-warp kernels

// Flag words of one sample: 8 bits (joints) per arm.
template <int A>
using Flags = std::conditional_t<(A > 4), uint64_t, uint32_t>;

constexpr unsigned kFull = 0xffffffffu;
constexpr int kEnvBit = 1, kSelfBit = 2, kExactBit = 16;
constexpr int kRulePlain = 0, kRuleConnect = 1, kRuleBspline = 2, kRuleShortcut = 3;
constexpr int kMaxSegments = 1 << 16;

// ---------------------------------------------------------------------------
// shared-memory staging of the scene: one bulk asynchronous copy (TMA engine)
// completed on an mbarrier, with a bounded wait.
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// The global nanosecond timer.
__device__ __forceinline__ uint64_t global_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Every wait on an mbarrier is bounded in time: a copy that has not completed
// after kWaitLimitNs is reported (scene status bit) instead of waited for.
constexpr uint64_t kWaitLimitNs = 1000000000ull;

// Wait for phase `parity` of mbarrier `bar`: true once it has completed,
// false after limit_ns of global time without it.
__device__ __forceinline__ bool bar_wait(uint64_t *bar, uint32_t parity, uint64_t limit_ns) {
    const uint64_t t0 = global_ns();
    for (;;) {
        uint32_t done;
        asm volatile(
            "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
            : "=r"(done)
            : "r"(smem_u32(bar)), "r"(parity)
            : "memory");
        if (done) return true;
        if (global_ns() - t0 > limit_ns) return false;
    }
}

// The wait of a bulk copy into shared memory.  If it runs out, the status bit
// is set and the copy, which may still be writing this CTA's shared memory,
// gets a second bounded wait before the caller reports its edges and leaves.
__device__ __forceinline__ bool copy_wait(uint64_t *bar, uint32_t parity, unsigned int *status, uint64_t limit_ns) {
    if (bar_wait(bar, parity, limit_ns)) return true;
    atomicOr(status, 1u);
    bar_wait(bar, parity, limit_ns);
    return false;
}

__device__ __forceinline__ bool stage_scene(float4 *dst, const float4 *src, uint32_t bytes, uint64_t *bar,
                                            unsigned int *status) {
    if (bytes == 0) return true;
    if (threadIdx.x == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(bar)));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                     : "memory");
        asm volatile(
            "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                smem_u32(dst)),
            "l"(src), "r"(bytes), "r"(smem_u32(bar))
            : "memory");
    }
    return __syncthreads_and(copy_wait(bar, 0, status, kWaitLimitNs));
}

__device__ __forceinline__ bool near3(float x, float y, float z, float4 b, float r) {
    const float dx = x - b.x, dy = y - b.y, dz = z - b.z;
    const float rr = r + b.w;
    return dx * dx + dy * dy + dz * dz < rr * rr;
}

// ---------------------------------------------------------------------------
// FK of one arm for one sample: approx sphere centres
// ---------------------------------------------------------------------------
struct ArmSpheres {
    float x[kNumApprox], y[kNumApprox], z[kNumApprox];
};

template <int I>
__device__ __forceinline__ void place_approx(const Xf &T, ArmSpheres &s) {
    s.x[I] = place_coord<I, false>(T, 0);
    s.y[I] = place_coord<I, false>(T, 1);
    s.z[I] = place_coord<I, false>(T, 2);
}

__device__ __forceinline__ void fk_approx_arm(const float *base12, const float (&q)[7], ArmSpheres &s) {
    Xf T;
    load_base(T, base12);
    place_approx<0>(T, s);
    joint_step<1>(T, q[0]);
    place_approx<1>(T, s);
    joint_step<2>(T, q[1]);
    place_approx<2>(T, s);
    joint_step<3>(T, q[2]);
    place_approx<3>(T, s);
    joint_step<4>(T, q[3]);
    place_approx<4>(T, s);
    joint_step<5>(T, q[4]);
    place_approx<5>(T, s);
    joint_step<6>(T, q[5]);
    place_approx<6>(T, s);
    joint_step<7>(T, q[6]);
    place_approx<7>(T, s);
    place_approx<8>(T, s);
    place_approx<9>(T, s);
    place_approx<10>(T, s);
}

// Joint values of arm `a` for sample k of segment `seg` (call-site formulas,
// see the rule constants).
__device__ __forceinline__ void sample_q(const EdgeScratch &W, int rule, int seg, int a, int k, float (&q)[7]) {
    const float fk = (float)k;
#pragma unroll
    for (int d = 0; d < 7; d++) {
        const int i = 7 * a + d;
        float v = __fmaf_rn(fk, W.stepg[i], W.base[i]);
        if (rule == kRuleBspline || rule == kRuleShortcut)
            for (int s = 0; s < seg; s++) v = __fadd_rn(v, W.delta[i]);
        q[d] = v;
    }
}

// One joint value (dof index i) of sample k of segment `seg`.
__device__ __forceinline__ float sample_q1(const EdgeScratch &W, int rule, int seg, int i, int k) {
    float v = __fmaf_rn((float)k, W.stepg[i], W.base[i]);
    if (rule == kRuleBspline || rule == kRuleShortcut)
        for (int s = 0; s < seg; s++) v = __fadd_rn(v, W.delta[i]);
    return v;
}

// Warp-wide float min / max (redux.sync on f32, sm_100a family).  NaN inputs
// are ignored; a lane with a NaN position can never pass an exact test, so the
// bounds built from these stay conservative.
__device__ __forceinline__ float warp_min(float v) {
    float r;
    asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ float warp_max(float v) {
    float r;
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}

// Three-input float min / max (sm_100 family); NaN inputs are ignored, as
// fminf / fmaxf do.
__device__ __forceinline__ float min3(float a, float b, float c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// Facts that hold for every pose of the arm (link lengths, distances between
// spheres that depend on a joint or two) are used only where the joint frames
// are accurate: joint values that add up to at most this many radians, where
// __sinf / __cosf err by about 1e-5 at most (beyond, or with a NaN, the
// computed frames need not be rotations), on a base that is a rigid transform
// (EdgeParams::rigid).  FP32 positions then err by far less than a millimetre.
constexpr float kRegularRad = 64.0f;

// The approx spheres s of one arm for this lane's sample go to column `lane` of
// dst, and a bound of every sphere over the warp's 32 samples to swept: the
// centre of the box around its 32 centres, radius = half the box diagonal
// (+0.4 %) + sphere radius + cull (EdgeParams::cull).  If the sphere touches
// something at any of the samples, its swept bound touches it too (the margin
// covers FP rounding).
__device__ __forceinline__ void store_swept(const ArmSpheres &s, float (*dst)[3][32], int lane, float4 *swept,
                                            float cull) {
#pragma unroll
    for (int i = 0; i < kNumApprox; i++) {
        dst[i][0][lane] = s.x[i];
        dst[i][1][lane] = s.y[i];
        dst[i][2][lane] = s.z[i];
    }
    __syncwarp();
    // spheres 1..10: lane t < 30 takes coordinate t % 3 of sphere 1 + t / 3
    // over the 32 columns, four at a time (start skewed by lane: each
    // quarter warp reads eight different 16-byte bank groups) and three
    // values per min / max: 8 loads and 32 min / max in place of 31 loads
    // and 62 (with the pairs of sphere 5 left out below, the broad kernel
    // on 65536 4-arm edges: 531 -> 470 us); sphere 0 sits on the base and
    // does not move
    float lo = 0.0f, hi = 0.0f;
    if (lane < 30) {
        const float4 *col = reinterpret_cast<const float4 *>(&dst[1][0][0] + 32 * lane);
        const float4 f = col[lane & 7];
        lo = fminf(min3(f.x, f.y, f.z), f.w);
        hi = fmaxf(max3(f.x, f.y, f.z), f.w);
#pragma unroll
        for (int l = 1; l < 8; l++) {
            const float4 v = col[(l + lane) & 7];
            lo = min3(min3(lo, v.x, v.y), v.z, v.w);
            hi = max3(max3(hi, v.x, v.y), v.z, v.w);
        }
    }
    const float ly = __shfl_down_sync(kFull, lo, 1), hy = __shfl_down_sync(kFull, hi, 1);
    const float lz = __shfl_down_sync(kFull, lo, 2), hz = __shfl_down_sync(kFull, hi, 2);
    const bool own = lane < 30 && lane % 3 == 0;
    const int i = own ? 1 + lane / 3 : 0;
    if (own || lane == 30) {
        const float ax = own ? lo : s.x[0], bx = own ? hi : s.x[0];
        const float ay = own ? ly : s.y[0], by = own ? hy : s.y[0];
        const float az = own ? lz : s.z[0], bz = own ? hz : s.z[0];
        const float dx = bx - ax, dy = by - ay, dz = bz - az;
        swept[i] = make_float4(0.5f * (ax + bx), 0.5f * (ay + by), 0.5f * (az + bz),
                               0.5f * sqrtf(dx * dx + dy * dy + dz * dz) * 1.004f + c_approx[i].w + cull);
    }
    __syncwarp();
}

// Joint values of one arm within kRegularRad.
__device__ __forceinline__ bool regular_pose(const float (&q)[7]) {
    float sum = 0.0f;  // NaN if any is
#pragma unroll
    for (int d = 0; d < 7; d++) sum += fabsf(q[d]);
    return sum <= kRegularRad;
}

// ---------------------------------------------------------------------------
// broad phase: approx spheres 1..10 of one arm (lane column `lane` of sp)
// against the scene.  Returns this lane's joints with a sphere that touches an
// obstacle.  The obstacles of all classes, in one order, are screened one per
// lane against the 10 spheres' swept bounds (sw, shared by the warp): the
// obstacle's bounding sphere, then for cuboids with orthonormal axes the exact
// sphere-cuboid test (both conservative).  Exact per-sample tests then run, for
// the whole warp, only for the (sphere, obstacle) pairs that survive, and only
// while some lane's joint is not flagged yet.
// TWO: two spheres per step against an obstacle (the last one twice), so that
// their chains of operations overlap.  One-arm calls, which take as long as
// their slowest edges, gain (30011 edges 84 -> 76 us); composite ones, which
// fill the SMs, pay for the tests done twice (262144 5-arm edges 3.80 -> 3.93
// ms).
// ---------------------------------------------------------------------------
template <bool TWO>
__device__ __forceinline__ uint32_t env_joints(const float4 *S, const SceneLayout &L, const SceneCounts &C,
                                               const float (*sp)[3][32], int lane, const float4 *sw) {
    const int n_obst = C.n_cub + C.n_zcub + C.n_cap + C.n_zcap + C.n_sph;
    uint32_t jm = 0;
    uint32_t open = 0x7feu;  // spheres whose joint some lane has not flagged (the same in every lane)
#pragma unroll 1
    for (int o0 = 0; o0 < n_obst && open; o0 += 32) {
        // one obstacle per lane: which swept sphere bounds reach it
        const int o = o0 + lane;
        uint32_t cand = 0;
        if (o < n_obst) {
            const float4 bs = S[L.b_cub + o];
#pragma unroll
            for (int i = 1; i < kNumApprox; i++) {
                const float4 u = sw[i];
                if (near3(u.x, u.y, u.z, bs, u.w)) cand |= 1u << i;
            }
            cand &= open;
            if (o < C.n_cub + C.n_zcub && bs.w <= 1e17f) {
#pragma unroll 1
                for (uint32_t c = cand; c; c &= c - 1) {
                    const int i = __ffs(c) - 1;
                    const float4 u = sw[i];
                    bool in;
                    if (o < C.n_cub) {
                        const float4 *r = S + L.cub + 4 * o;
                        in = hit_cuboid(r[0], r[1], r[2], r[3], u.x, u.y, u.z, u.w * u.w);
                    } else {
                        const float4 *r = S + L.zcub + 4 * (o - C.n_cub);
                        in = hit_zcuboid(r[0], r[1], r[2], u.x, u.y, u.z, u.w * u.w);
                    }
                    if (!in) cand &= ~(1u << i);
                }
            }
        }
        // exact per-sample tests of the surviving (sphere, obstacle) pairs
        uint32_t obal = __ballot_sync(kFull, cand != 0);
#pragma unroll 1
        while (obal) {
            const int src = __ffs(obal) - 1;
            obal &= obal - 1;
            uint32_t cm = __shfl_sync(kFull, cand, src) & open;
            // the spheres cm against one obstacle, whose record stays in registers
            auto spheres = [&](auto hit) {
#pragma unroll 1
                while (cm) {
                    const int i = __ffs(cm) - 1;
                    cm &= cm - 1;
                    const uint32_t ji = 1u << approx_joint(i);
                    if constexpr (TWO) {
                        const int k = cm ? __ffs(cm) - 1 : i;
                        cm &= cm - 1;
                        const uint32_t jk = 1u << approx_joint(k);
                        const bool hi = hit(sp[i][0][lane], sp[i][1][lane], sp[i][2][lane], c_approx[i].w);
                        const bool hk = hit(sp[k][0][lane], sp[k][1][lane], sp[k][2][lane], c_approx[k].w);
                        jm |= (hi ? ji : 0u) | (hk ? jk : 0u);
                        if (__all_sync(kFull, jm & jk)) open &= ~(k < 7 ? 1u << k : 0x780u);
                    } else {
                        if (hit(sp[i][0][lane], sp[i][1][lane], sp[i][2][lane], c_approx[i].w)) jm |= ji;
                    }
                    if (__all_sync(kFull, jm & ji)) open &= ~(i < 7 ? 1u << i : 0x780u);
                    cm &= open;
                }
            };
            int t = o0 + src;
            if (t < C.n_cub) {
                const float4 *c = S + L.cub + 4 * t;
                const float4 c0 = c[0], c1 = c[1], c2 = c[2], c3 = c[3];
                spheres([&](float x, float y, float z, float r) {
                    return hit_cuboid(c0, c1, c2, c3, x, y, z, __fmul_rn(r, r));
                });
            } else if ((t -= C.n_cub) < C.n_zcub) {
                const float4 *c = S + L.zcub + 4 * t;
                const float4 c0 = c[0], c1 = c[1], c2 = c[2];
                spheres([&](float x, float y, float z, float r) {
                    return hit_zcuboid(c0, c1, c2, x, y, z, __fmul_rn(r, r));
                });
            } else if ((t -= C.n_zcub) < C.n_cap) {
                const float4 *c = S + L.cap + 2 * t;
                const float4 c0 = c[0], c1 = c[1];
                spheres([&](float x, float y, float z, float r) { return hit_capsule(c0, c1, x, y, z, r); });
            } else if ((t -= C.n_cap) < C.n_zcap) {
                const float4 *c = S + L.zcap + 2 * t;
                const float4 c0 = c[0], c1 = c[1];
                spheres([&](float x, float y, float z, float r) { return hit_zcapsule(c0, c1, x, y, z, r); });
            } else {
                const float4 c0 = S[L.sph + t - C.n_zcap];
                spheres([&](float x, float y, float z, float r) {
                    return hit_sphere_sphere(c0.x, c0.y, c0.z, c0.w, x, y, z, r);
                });
            }
        }
    }
    return jm;
}

// Arm pairs (a < b) in order: pair index of (a, b), and the count.
__host__ __device__ __forceinline__ constexpr int pair_index(int a, int b, int A) {
    return a * (2 * A - a - 1) / 2 + (b - a - 1);
}
__host__ __device__ __forceinline__ constexpr int num_pairs(int A) { return A * (A - 1) / 2; }

// Arm pair p (pair_index order): its lower and upper arm.
template <int A>
__host__ __device__ __forceinline__ constexpr void pair_arms(int p, int &a, int &b) {
    a = 0;
    while (p >= A - 1 - a) {
        p -= A - 1 - a;
        a++;
    }
    b = a + 1 + p;
}

// pair_arms inverts pair_index for every pair of up to 5 arms
template <int A>
constexpr bool pair_order_round_trips() {
    for (int p = 0; p < num_pairs(A); p++) {
        int a = 0, b = 0;
        pair_arms<A>(p, a, b);
        if (!(0 <= a && a < b && b < A) || pair_index(a, b, A) != p) return false;
    }
    return true;
}
static_assert(pair_order_round_trips<2>() && pair_order_round_trips<3>() && pair_order_round_trips<4>() &&
                  pair_order_round_trips<5>(),
              "arm pair order");

// Every detailed sphere lies inside an approx sphere of its joint grown by
// 0.9 mm (0.6 mm in fact), so two arms' joints whose approx spheres' swept
// bounds (which carry kCullMargin each) do not meet cannot collide.
constexpr bool approx_cover_detailed() {
    for (int i = 0; i < kNumDet; i++) {
        bool in = false;
        for (int a = 0; a < kNumApprox; a++) {
            if (approx_joint(a) != det_joint(i)) continue;
            const double x = (double)kDet[i].x - kApprox[a].x, y = (double)kDet[i].y - kApprox[a].y,
                         z = (double)kDet[i].z - kApprox[a].z, r = (double)kApprox[a].r + 9e-4 - kDet[i].r;
            in = in || (r > 0.0 && x * x + y * y + z * z <= r * r);
        }
        if (!in) return false;
    }
    return true;
}
static_assert(kCullMargin >= 1e-3f && approx_cover_detailed(), "approx spheres cover the detailed ones");

// Largest distance between two sphere centres of one joint, approx or detailed.
constexpr double kJointSpan = 0.25;
constexpr bool joint_span_holds() {
    auto at = [](int i) { return i < kNumDet ? kDet[i] : kApprox[i - kNumDet]; };
    auto joint = [](int i) { return i < kNumDet ? det_joint(i) : approx_joint(i - kNumDet); };
    for (int i = 0; i < kNumDet + kNumApprox; i++)
        for (int k = 0; k < i; k++) {
            const double x = (double)at(i).x - at(k).x, y = (double)at(i).y - at(k).y, z = (double)at(i).z - at(k).z;
            if (joint(i) == joint(k) && x * x + y * y + z * z > kJointSpan * kJointSpan) return false;
        }
    return true;
}
static_assert(joint_span_holds(), "span of a joint's spheres");

// Broad-phase intra-arm rows (panda_multi_geometry.cuh:133-139) as 21 pairs.
static __constant__ uint8_t c_intra_pairs[21][2] = {
    {0, 5}, {0, 6}, {0, 7}, {0, 8}, {0, 9}, {0, 10}, {1, 5}, {1, 6}, {1, 7}, {1, 8}, {1, 9},
    {1, 10}, {2, 5}, {2, 7}, {2, 8}, {2, 9}, {2, 10}, {5, 7}, {5, 8}, {5, 9}, {5, 10}};

constexpr double const_sqrt(double v) {
    double x = v > 1.0 ? v : 1.0;
    for (int i = 0; i < 64; i++) x = 0.5 * (x + v / x);
    return x;
}
constexpr double const_hypot(double x, double y) { return const_sqrt(x * x + y * y); }

// Approx spheres 5 and 8 overlap in every pose.  Joint 6's axis is the y axis of
// joint 5's frame, through its origin; sphere 8 is at F_7 Rz(q7) x from joint 6.
constexpr bool spheres_5_8_overlap() {
    const SphereDef &a = kApprox[5], &b = kApprox[8];
    const double out = const_hypot(kJointK.v[5][1] + const_hypot(b.x, b.y), b.z);  // from joint 6's axis, at most
    const double along = (a.y > 0 ? a.y : -a.y) + const_hypot(b.x, b.y);           // along it
    const double far = const_hypot(out + const_hypot(a.x, a.z), along);
    return kJointK.v[4][1] == 0.f && kJointK.v[4][2] == 0.f && far < (double)a.r + b.r - 2e-3;
}
static_assert(spheres_5_8_overlap(), "pair (5, 8) overlaps in every pose");

// Intra-arm pairs of one arm (panda_four.cuh:140-176): the 21 approx sphere
// pairs, one per lane, screened by the swept bounds sw of the warp's samples;
// exact per-sample tests for the survivors.  Returns the lane's flag bits (by
// joint of the pair's first sphere).
// regular (warp-uniform): the pairs of sphere 5 are not tested, its joint is
// flagged.  Pair (5, 8) overlaps in every pose: sphere 8 lies on joint 7's axis
// at (0.088, -0.129) from joint 6's, 0.156 m, and sphere 5 0.111 m from joint
// 6's axis and 0.037 m along it, so their centres are at most
// sqrt(0.267^2 + 0.037^2) = 0.270 m apart with radii adding up to 0.280 m.
__device__ __forceinline__ uint32_t intra_flags(const float (*sp)[3][32], const float4 *sw, int lane, bool regular) {
    // pair `lane` of c_intra_pairs, computed rather than read per lane
    const int p1 = lane < 6 ? 0 : lane < 12 ? 1 : lane < 17 ? 2 : 5;
    const int p2 = lane < 12 ? 5 + lane % 6 : lane == 12 ? 5 : lane < 17 ? lane - 6 : lane - 10;
    const float4 u1 = sw[p1];
    const bool c = lane < (regular ? 17 : 21) && near3(u1.x, u1.y, u1.z, sw[p2], u1.w);
    uint32_t bal = __ballot_sync(kFull, c);
    uint32_t jm = regular ? 1u << approx_joint(5) : 0u;
    while (bal) {
        const int t = __ffs(bal) - 1;
        bal &= bal - 1;
        const int s1 = c_intra_pairs[t][0], s2 = c_intra_pairs[t][1];
        if (hit_sphere_sphere(sp[s1][0][lane], sp[s1][1][lane], sp[s1][2][lane], c_approx[s1].w, sp[s2][0][lane],
                              sp[s2][1][lane], sp[s2][2][lane], c_approx[s2].w))
            jm |= 1u << approx_joint(s1);
    }
    return jm;
}

// Broad phase of one sample (every lane of the warp calls it; lanes past the
// segment's last sample evaluate sample g and discard the result).  One loop
// places arms: arm b, with its env and intra-arm tests and the screen of its
// sphere pairs with every lower arm by swept bounds (lane (a, i): sphere i of
// arm a against arm b's 11), then each lower arm that a pair survived with,
// whose spheres stay in registers for the exact tests against arm b's columns.
// Flags of an arm pair go to its lower arm (panda_four.cuh:178-214); lane p of
// pm receives pair p's connected joints, the lower arm's in bits 0..7 and the
// upper arm's in bits 8..15.
// Bound by instruction issue.  With one placement loop and one obstacle order
// (code shared, a lower arm's spheres in registers: half the scratch) the broad
// kernels run 24 warps per SM: 65536 4-arm edges 467 -> 414 us, 262144 5-arm
// edges x 64 samples 5.28 -> 3.82 ms, 65536 shortcut edges 2.47 -> 1.92 ms;
// 30011 one-arm edges, one class of obstacle, 81 -> 83 us.
template <int A>
__device__ __forceinline__ void broad_sample(const EdgeParams &P, const EdgeScratch &W, BroadPart &B, const float4 *S,
                                             const SceneLayout &L, int seg, int k, Flags<A> &envw, Flags<A> &selfw,
                                             uint32_t &pm) {
    const int lane = threadIdx.x & 31;
    envw = 0;
    selfw = 0;
    pm = 0;
    const bool do_env = P.flags & kEnvBit, do_self = P.flags & kSelfBit;
    auto &cur = B.cur;
#pragma unroll 1
    for (int b = 0; b < A; b++) {
        float4 *sw = B.swept[b];
        uint32_t xm[2] = {0u, 0u};  // lane 11 * (a & 1) + i of word a >> 1: arm b's spheres that sphere i of arm a meets
        uint32_t pend = 0;          // lower arms left to test
#pragma unroll 1
        for (int x = b;;) {
            MRPOP_PHASE_START();
            float q[7];
            sample_q(W, P.rule, seg, P.single ? 0 : x, k, q);
            ArmSpheres s;
            fk_approx_arm(P.base[x], q, s);
            if (A == 1 || x == b) {
                store_swept(s, cur, lane, sw, P.cull);
                MRPOP_PHASE(P, 0);
                if (do_env) envw |= (Flags<A>)env_joints<A == 1>(S, L, P.sc, cur, lane, sw) << (8 * b);
                MRPOP_PHASE(P, 1);
                if (!do_self) break;
                const bool reg = regular_pose(q);
                const bool regular = __all_sync(kFull, reg) && (P.rigid >> b & 1);
                selfw |= (Flags<A>)intra_flags(cur, sw, lane, regular) << (8 * b);
                MRPOP_PHASE(P, 2);
                if (A == 1) break;
                const int la = lane >= kNumApprox ? 1 : 0, i = min(lane - kNumApprox * la, kNumApprox - 1);
#pragma unroll
                for (int w = 0; w < (A > 3 ? 2 : 1); w++) {
                    if (2 * w >= b) break;
                    const int a = 2 * w + la;
                    const float4 u = B.swept[a < b ? a : 0][i];
                    uint32_t m = 0;
#pragma unroll
                    for (int j = 0; j < kNumApprox; j++)
                        if (near3(u.x, u.y, u.z, sw[j], u.w)) m |= 1u << j;
                    xm[w] = a < b && lane < 2 * kNumApprox ? m : 0u;
                    const uint32_t nz = __ballot_sync(kFull, xm[w] != 0);
                    pend |= ((nz & 0x7ffu ? 1u : 0u) | (nz >> kNumApprox ? 2u : 0u)) << (2 * w);
                }
            } else {
                const int a = x;
                const uint32_t word = A > 3 && a > 1 ? xm[1] : xm[0];
                uint32_t am = 0, ja = 0, sb = 0;
#pragma unroll
                for (int i = 0; i < kNumApprox; i++) {
                    uint32_t m = __shfl_sync(kFull, word, kNumApprox * (a & 1) + i);
                    if (!m) continue;
                    ja |= 1u << approx_joint(i);
                    sb |= m;
                    bool h = false;
#pragma unroll 1
                    for (; m; m &= m - 1) {
                        const int j = __ffs(m) - 1;
                        h |= hit_sphere_sphere(s.x[i], s.y[i], s.z[i], c_approx[i].w, cur[j][0][lane], cur[j][1][lane],
                                               cur[j][2][lane], c_approx[j].w);
                    }
                    if (h) am |= 1u << approx_joint(i);
                }
                selfw |= (Flags<A>)am << (8 * a);
                const uint32_t jb = (sb & 0x7fu) | (sb >> 7 ? 0x80u : 0u);
                if (lane == pair_index(a, b, A)) pm = ja | jb << 8;
                MRPOP_PHASE(P, 3);
            }
            if (!pend) break;
            x = __ffs(pend) - 1;
            pend &= pend - 1;
        }
        __syncwarp();  // arm b's columns are read before the next arm's overwrite them
    }
}

// Detailed spheres on the joints flagged in w (8 bits per arm).  Joints with equal counts share a population count.
template <int A>
__device__ __forceinline__ int flag_count(Flags<A> w) {
    static_assert(det_count(0) == 1 && det_count(1) == 4 && det_count(2) == 4 && det_count(3) == 4 &&
                      det_count(4) == 4 && det_count(5) == 12 && det_count(6) == 3 && det_count(7) == 27,
                  "counts per joint");
    auto bits = [&](uint32_t joints) {
        int n = __popc((uint32_t)w & 0x01010101u * joints);
        if constexpr (A > 4) n += __popc((uint32_t)(w >> 32) & joints);
        return n;
    };
    return bits(0x01u) + 4 * bits(0x1eu) + 12 * bits(0x20u) + 3 * bits(0x40u) + 27 * bits(0x80u);
}

// reference thread split (utils.cuh:478-497): share of 4g threads, truncated
__device__ __forceinline__ int ref_share(int cnt, int total, int g) {
    if (total == 0) return 0; // 0/0 is NaN on the device; its int conversion is 0
    return __float2int_rz(__fmul_rn(__fdiv_rn((float)cnt, (float)total), (float)(4 * g)));
}

// dense narrow-phase tally for one sample (per the flop convention)
static __device__ __noinline__ double narrow_flops(const EdgeParams &P, int A, uint64_t envw, uint64_t selfw, bool de,
                                               bool ds) {
    double f = 0.0;
    const bool quirk = !P.single && !(P.flags & kExactBit);
    for (int a = 0; a < A; a++) {
        const uint32_t em = de ? (uint32_t)(envw >> (8 * a)) & 0xffu : 0u;
        const uint32_t sm = ds ? (uint32_t)(selfw >> (8 * a)) & 0xffu : 0u;
        for (int j = 0; j < 8; j++) {
            if ((em | sm) >> j & 1u) f += 18.0 * det_count(j);
            if (em >> j & 1u) f += P.env_test_flops * (j == 0 ? 0 : det_count(j));
        }
        if (sm) {
            for (int r = 0; r < kDetRows; r++) {
                const int idx = quirk ? r : det_row_first(r);
                if (sm >> det_joint(idx) & 1u) f += 11.0 * (det_row_hi(r) - det_row_lo(r) + 1);
            }
            for (int j = 0; j < 8; j++)
                if (sm >> j & 1u) f += 11.0 * kNumDet * (A - 1 - a) * det_count(j);
        }
    }
    return f;
}

// ---------------------------------------------------------------------------
// narrow phase
// ---------------------------------------------------------------------------
// Rows whose first-read sphere is on joint j (quirk: sphere r, else first(r)).
__host__ __device__ constexpr uint32_t joint_rows(int j, bool quirk) {
    uint32_t m = 0;
    for (int r = 0; r < kDetRows; r++)
        if (det_joint(quirk ? r : det_row_first(r)) == j) m |= 1u << r;
    return m;
}

// bit r set: detailed self row r is checked for an arm with self flags sm
__device__ __forceinline__ uint32_t row_mask(uint32_t sm, bool quirk) {
    uint32_t m = 0;
#pragma unroll
    for (int j = 0; j < kNumJoints; j++)
        if (sm >> j & 1u) m |= quirk ? joint_rows(j, true) : joint_rows(j, false);
    return m;
}

// Rows whose targets are the forearm's spheres alone.
constexpr uint32_t forearm_rows() {
    uint32_t m = 0;
    for (int r = 0; r < kDetRows; r++)
        if (det_joint(det_row_hi(r)) == 5) m |= 1u << r;
    return m;
}
constexpr uint32_t kForearmRows = forearm_rows();

// Row bookkeeping of the detailed self check:
//   cover[i]     rows whose target range lo..hi contains sphere i
//   jfirst[q][j] rows whose first-read sphere is on joint j (q = 1: the composite
//                robots' reading, sphere r; q = 0: sphere first(r))
struct RowTab {
    uint32_t cover[kNumDet];
    uint32_t jfirst[2][kNumJoints];
};

__host__ __device__ constexpr RowTab make_row_tab() {
    RowTab t{};
    for (int r = 0; r < kDetRows; r++)
        for (int i = det_row_lo(r); i <= det_row_hi(r); i++) t.cover[i] |= 1u << r;
    for (int q = 0; q < 2; q++)
        for (int j = 0; j < kNumJoints; j++) t.jfirst[q][j] = joint_rows(j, q != 0);
    return t;
}

static __constant__ RowTab c_rows = make_row_tab();

// Detailed sphere centre, transform in registers (the reference's full
// expression, panda_four.cuh:363-366).
__device__ __forceinline__ float3 place_reg(const Xf &T, float4 s) {
    float3 p;
    p.x = __fadd_rn(__fmaf_rn(T.m[2], s.z, pair_fma(T.m[0], s.x, T.m[1], s.y)), T.m[3]);
    p.y = __fadd_rn(__fmaf_rn(T.m[6], s.z, pair_fma(T.m[4], s.x, T.m[5], s.y)), T.m[7]);
    p.z = __fadd_rn(__fmaf_rn(T.m[10], s.z, pair_fma(T.m[8], s.x, T.m[9], s.y)), T.m[11]);
    return p;
}

// Sub-groups of the detailed spheres (contiguous index ranges within one
// joint): [0] [1-4] [5-8] [9-12] [13-16] [17-18] [19-20] [21-28] [29-31]
// [32-36] [37-58].  SetBounds::grp holds each group's bounding sphere in its
// joint frame; a group's world bound is that centre through the joint frame.
constexpr int kNumGroups = 11;
__host__ __device__ __forceinline__ constexpr int grp_first(int g) {
    return g == 0 ? 0 : g == 1 ? 1 : g == 2 ? 5 : g == 3 ? 9 : g == 4 ? 13 : g == 5 ? 17 : g == 6 ? 19 : g == 7 ? 21
         : g == 8 ? 29 : g == 9 ? 32 : g == 10 ? 37 : 59;
}
// groups of joint j: [jgrp_first(j), jgrp_first(j + 1))
__host__ __device__ __forceinline__ constexpr int jgrp_first(int j) {
    return j < 5 ? j : j == 5 ? 5 : j == 6 ? 8 : j == 7 ? 9 : 11;
}
// The hand group (spheres 37..58: a 6 x 3 grid along the gripper's diagonal
// plus four finger-tip spheres) is screened in three parts along the diagonal:
// the two columns and finger tips on each side, and the two middle columns.
// Bits are sphere index - kHandFirst; SetBounds::hsub holds each part's bound.
constexpr int kHandGroup = 10;
constexpr int kHandFirst = 37;
constexpr int kHandParts = 3;
__host__ __device__ __forceinline__ constexpr uint32_t hand_part(int s) {
    return s == 0 ? 0x3030C3u : s == 1 ? 0x00C30Cu : 0x0F0C30u;
}

// Bounding spheres of the sub-groups and of the hand's parts in their joint
// frames (+margin): the centre of the box around the spheres' centres.  In
// constant memory, not in the kernels' parameters: the batch kernels, which keep
// those in shared memory, read them as operands too.
struct SetBounds {
    float4 grp[kNumGroups];
    float4 hsub[kHandParts];
};
// the spheres first + (bits of m)
constexpr float4 set_ball(int first, uint32_t m) {
    double lo[3] = {1e9, 1e9, 1e9}, hi[3] = {-1e9, -1e9, -1e9}, r = 0.0;
    for (int i = 0; i < 32; i++) {
        if (!(m >> i & 1u)) continue;
        const double v[3] = {kDet[first + i].x, kDet[first + i].y, kDet[first + i].z};
        for (int c = 0; c < 3; c++) {
            lo[c] = v[c] < lo[c] ? v[c] : lo[c];
            hi[c] = v[c] > hi[c] ? v[c] : hi[c];
        }
    }
    const double x = 0.5 * (lo[0] + hi[0]), y = 0.5 * (lo[1] + hi[1]), z = 0.5 * (lo[2] + hi[2]);
    for (int i = 0; i < 32; i++) {
        if (!(m >> i & 1u)) continue;
        const SphereDef &d = kDet[first + i];
        const double e = const_sqrt((d.x - x) * (d.x - x) + (d.y - y) * (d.y - y) + (d.z - z) * (d.z - z)) + d.r;
        r = e > r ? e : r;
    }
    return float4{(float)x, (float)y, (float)z, (float)(r * 1.001 + kCullMargin)};
}
constexpr SetBounds make_set_bounds() {
    SetBounds b{};
    for (int g = 0; g < kNumGroups; g++)
        b.grp[g] = set_ball(grp_first(g), (1u << (grp_first(g + 1) - grp_first(g))) - 1u);
    for (int s = 0; s < kHandParts; s++) b.hsub[s] = set_ball(kHandFirst, hand_part(s));
    return b;
}
static __constant__ SetBounds c_bounds = make_set_bounds();

// Conservative screen of obstacle o (index over all classes, in the order of
// load_obstacle) against ball U: the obstacle's bounding sphere, then for cuboids
// with orthonormal axes the exact sphere-cuboid test with U's radius.
__device__ __forceinline__ bool screen_obstacle(const float4 *S, const SceneLayout &L, const SceneCounts &C, int o,
                                                float4 U) {
    const float4 bs = S[L.b_cub + o];
    if (!near3(U.x, U.y, U.z, bs, U.w)) return false;
    if (bs.w > 1e17f) return true;
    if (o < C.n_cub) {
        const float4 *c = S + L.cub + 4 * o;
        return hit_cuboid(c[0], c[1], c[2], c[3], U.x, U.y, U.z, U.w * U.w);
    }
    o -= C.n_cub;
    if (o < C.n_zcub) {
        const float4 *c = S + L.zcub + 4 * o;
        return hit_zcuboid(c[0], c[1], c[2], U.x, U.y, U.z, U.w * U.w);
    }
    return true;
}

// Lanes 0..lane: a hit on any of them settles the lane's sample.
__device__ __forceinline__ uint32_t lanes_upto(int lane) { return (2u << lane) - 1u; }

// One obstacle, its record in registers (the same in every lane).  kind: 0
// cuboid, 1 z-cuboid, 2 capsule, 3 z-capsule, 4 sphere.
struct Obstacle {
    float4 c0, c1, c2, c3;
    float4 bound;  // bounding sphere (+margin); radius 1e18 for a cuboid with skewed axes
    int kind;
    // the reference's test of a sphere
    __device__ __forceinline__ bool hit(float3 p, float r) const {
        if (kind == 0) return hit_cuboid(c0, c1, c2, c3, p.x, p.y, p.z, __fmul_rn(r, r));
        if (kind == 1) return hit_zcuboid(c0, c1, c2, p.x, p.y, p.z, __fmul_rn(r, r));
        if (kind == 2) return hit_capsule(c0, c1, p.x, p.y, p.z, r);
        if (kind == 3) return hit_zcapsule(c0, c1, p.x, p.y, p.z, r);
        return hit_sphere_sphere(c0.x, c0.y, c0.z, c0.w, p.x, p.y, p.z, r);
    }
    // the test itself bounds what a ball holds (distance to a box)
    __device__ __forceinline__ bool metric() const { return kind < 2 && bound.w <= 1e17f; }
};

// Obstacle o over all classes, in the order of the bounds.
__device__ __forceinline__ Obstacle load_obstacle(const float4 *S, const SceneLayout &L, const SceneCounts &C, int o) {
    Obstacle b;
    b.bound = S[L.b_cub + o];
    const float4 *r;
    if (o < C.n_cub) {
        b.kind = 0;
        r = S + L.cub + 4 * o;
        b.c3 = r[3];
    } else if ((o -= C.n_cub) < C.n_zcub) {
        b.kind = 1;
        r = S + L.zcub + 4 * o;
    } else if ((o -= C.n_zcub) < C.n_cap) {
        b.kind = 2;
        r = S + L.cap + 2 * o;
    } else if ((o -= C.n_cap) < C.n_zcap) {
        b.kind = 3;
        r = S + L.zcap + 2 * o;
    } else {
        b.kind = 4;
        r = S + L.sph + o - C.n_zcap;
    }
    b.c0 = r[0];
    if (b.kind < 4) b.c1 = r[1];
    if (b.kind < 2) b.c2 = r[2];
    return b;
}

// Env test of the detailed spheres first + (bits of spheres), one sub-group or
// hand part with bound gl in frame T, for the lanes with act set; every lane of
// the warp calls it.  The active lanes' bounds are merged into one ball U (box
// of their centres, half diagonal + bound); obstacles are screened against U one
// per lane, 32 at a time.  Each survivor then meets the lanes' own bounds (the
// exact test for boxes with orthonormal axes, the bounding sphere otherwise) and,
// if some lane's reaches it, its spheres.  A hit settles the lane and those
// above it.  Returns true for a lane that hit.
// The slowest edges set the time of calls of up to some ten thousand edges; in
// those, most survivors of U are near no lane's bound, and every lane tested
// every sphere of the whole hand against them: the slowest of 30011 one-arm
// edges takes 94 k cycles in place of 246 k, the kernel 139 -> 81 us; 65536
// 4-arm edges 457 -> 433 us.
__device__ __forceinline__ bool env_group_warp(const float4 *S, const SceneLayout &L, const SceneCounts &C,
                                                   const Xf &T, int first, uint32_t spheres, float4 gl, bool act) {
    const int lane = threadIdx.x & 31;
    const float3 gc = place_reg(T, gl);
    constexpr float kBig = 3.0e38f;
    const float lx = warp_min(act ? gc.x : kBig), hx = warp_max(act ? gc.x : -kBig);
    const float ly = warp_min(act ? gc.y : kBig), hy = warp_max(act ? gc.y : -kBig);
    const float lz = warp_min(act ? gc.z : kBig), hz = warp_max(act ? gc.z : -kBig);
    const float dx = hx - lx, dy = hy - ly, dz = hz - lz;
    const float4 U = make_float4(0.5f * (lx + hx), 0.5f * (ly + hy), 0.5f * (lz + hz),
                                 0.5f * sqrtf(dx * dx + dy * dy + dz * dz) * 1.004f + gl.w);
    const int n_obst = C.n_cub + C.n_zcub + C.n_cap + C.n_zcap + C.n_sph;
    bool hit = false;
#pragma unroll 1
    for (int base = 0; base < n_obst; base += 32) {
        const int o = base + lane;
        uint32_t m = __ballot_sync(kFull, o < n_obst && screen_obstacle(S, L, C, o, U));
        MRPOP_COUNT_W(11, 1);
        MRPOP_COUNT_W(12, __popc(m));
        MRPOP_COUNT_LANES(13, act);
#pragma unroll 1
        for (; m; m &= m - 1) {
            const Obstacle b = load_obstacle(S, L, C, base + __ffs(m) - 1);
            // the bound first, then the spheres: one copy of the tests
            float4 sd = gl;
            float3 p = gc;
            uint32_t rest = spheres;
            bool reached = false, h = false;
            for (bool bound = true;; bound = false) {
                const bool t = bound && !b.metric() ? near3(p.x, p.y, p.z, b.bound, sd.w) : b.hit(p, sd.w);
                if (bound) {
                    reached = act && t;
                    if (!__any_sync(kFull, reached)) break;
                } else {
                    h |= t;
                }
                if (!rest) break;
                sd = c_det[first + __ffs(rest) - 1];
                rest &= rest - 1;
                p = place_reg(T, sd);
            }
            const uint32_t hb = __ballot_sync(kFull, reached && h);
            if (hb) {
                hit |= reached && h;
                act = act && !(hb & lanes_upto(lane));
                if (!__any_sync(kFull, act)) return hit;
            }
        }
    }
    return hit;
}

// True when the forearm-hand rows cannot fire at joint values (q6, q7): the
// cell's bit of the table is set.  NaN or out-of-range values give false.
__device__ __forceinline__ bool row5_apart(const uint32_t *tab, float q6, float q7) {
    const float f6 = (q6 - kRow5Lo6) * ((float)kRow5N6 / (kRow5Hi6 - kRow5Lo6));
    const float f7 = (q7 - kRow5Lo7) * ((float)kRow5N7 / (kRow5Hi7 - kRow5Lo7));
    if (!(f6 >= 0.0f && f6 < (float)kRow5N6 && f7 >= 0.0f && f7 < (float)kRow5N7)) return false;
    const int cell = (int)f6 * kRow5N7 + (int)f7;
    return (__ldg(tab + (cell >> 5)) >> (cell & 31)) & 1u;
}

// Per-lane state of the lane-parallel detailed check of one arm.  A lane with
// em = rm = 0 takes no further part: it has no tests here, its sample has hit,
// or a lower lane's sample has (only the first colliding sample is reported).
struct LaneCtx {
    uint32_t em;  // env-flagged joints
    uint32_t rm;  // flagged detailed self rows
    int quirk;
    bool hit;
    __device__ __forceinline__ void set_hit() {
        hit = true;
        em = rm = 0;
    }
};

// Sphere sets of the arm-pair and env tests: the sub-groups, the hand whole as
// set 10 or (PARTS) in its three parts as sets 10..12.  Sets of joint j:
// [jgrp_first(j), set_end(j)); the bound of set t; its spheres, first + (bits of
// set_spheres); the sets of the joints in jm.
template <bool PARTS>
__device__ __forceinline__ int set_end(int j) {
    return jgrp_first(j + 1) + (PARTS && j == 7 ? kHandParts - 1 : 0);
}
template <bool PARTS>
__device__ __forceinline__ float4 set_bound(int t) {
    return !PARTS || t < kHandGroup ? c_bounds.grp[t] : c_bounds.hsub[t - kHandGroup];
}
__device__ __forceinline__ int set_first(int t) { return t < kHandGroup ? grp_first(t) : kHandFirst; }
template <bool PARTS>
__device__ __forceinline__ uint32_t set_spheres(int t) {
    return !PARTS || t < kHandGroup ? (1u << (grp_first(t + 1) - grp_first(t))) - 1u : hand_part(t - kHandGroup);
}
template <bool PARTS>
__device__ __forceinline__ uint32_t joint_sets(uint32_t jm) {
    return (jm & 0x1fu) | (jm >> 5 & 1u) * 0xe0u | (jm >> 6 & 1u) << 8 | (jm >> 7 & 1u) * (PARTS ? 0x1e00u : 0x600u);
}

// Joint j of one arm, frame T: env tests of an env-flagged joint (lane_env);
// stash of the first spheres of flagged rows, and the row tests whose targets
// are here, screened by the target group's bound (lane_rows).
__device__ __forceinline__ void lane_env(int j, const EdgeParams &P, const Xf &T, LaneCtx &c, const float4 *S,
                                         const SceneLayout &L) {
    // every lane takes part in the env screening (warp-wide votes inside)
    if (__any_sync(kFull, c.em >> j & 1u)) {
        // the hand's spheres in its three parts
#pragma unroll 1
        for (int g = jgrp_first(j); g < set_end<true>(j); g++) {
            float4 gl = set_bound<true>(g);
            gl.w += P.slack;
            if (env_group_warp(S, L, P.sc, T, set_first(g), set_spheres<true>(g), gl, c.em >> j & 1u)) c.set_hit();
            const uint32_t hb = __ballot_sync(kFull, c.hit);
            if (hb & lanes_upto(threadIdx.x & 31)) c.em = c.rm = 0;
            if (!__any_sync(kFull, c.em >> j & 1u)) break;
        }
    }
}

template <int A, typename WS>
__device__ __forceinline__ void lane_rows(int j, const EdgeParams &P, const Xf &T, LaneCtx &c, WS &W,
                                          const float4 *det_tab, int lane) {
    if (!c.rm) return;
    uint32_t m1 = c.rm & c_rows.jfirst[c.quirk][j];
    while (m1) {
        const int r = __ffs(m1) - 1;
        m1 &= m1 - 1;
        const float3 p = place_reg(T, det_tab[c.quirk ? r : det_row_first(r)]);
        W.stash[r][0][lane] = p.x;
        W.stash[r][1][lane] = p.y;
        W.stash[r][2][lane] = p.z;
    }
#pragma unroll 1
    for (int g = jgrp_first(j); g < jgrp_first(j + 1); g++) {
        uint32_t rows = c.rm & c_rows.cover[grp_first(g)];
        if (!rows) continue;
        float4 gl = c_bounds.grp[g];
        gl.w += P.slack;
        const float3 gc = place_reg(T, gl);
        uint32_t nr = 0;
        while (rows) {
            const int r = __ffs(rows) - 1;
            rows &= rows - 1;
            if (near3(W.stash[r][0][lane], W.stash[r][1][lane], W.stash[r][2][lane],
                      make_float4(gc.x, gc.y, gc.z, gl.w), det_tab[det_row_first(r)].w))
                nr |= 1u << r;
        }
        if (!nr) continue;
        bool h = false;
        if (A == 1 && g == kHandGroup) {
            // single-arm form: the hand's parts screened per row first, then
            // their spheres (in the composite forms the extra screens cost
            // more than they save)
#pragma unroll 1
            for (int s = 0; s < kHandParts; s++) {
                float4 sl = c_bounds.hsub[s];
                sl.w += P.slack;
                const float3 sc = place_reg(T, sl);
                uint32_t ns = 0;
                for (uint32_t m = nr; m; m &= m - 1) {
                    const int r = __ffs(m) - 1;
                    if (near3(W.stash[r][0][lane], W.stash[r][1][lane], W.stash[r][2][lane],
                              make_float4(sc.x, sc.y, sc.z, sl.w), det_tab[det_row_first(r)].w))
                        ns |= 1u << r;
                }
                if (!ns) continue;
                for (uint32_t pm = hand_part(s); pm; pm &= pm - 1) {
                    const float4 sd = c_det[kHandFirst + __ffs(pm) - 1];
                    const float3 p = place_reg(T, sd);
                    for (uint32_t m = ns; m; m &= m - 1) {
                        const int r = __ffs(m) - 1;
                        h |= hit_sphere_sphere(W.stash[r][0][lane], W.stash[r][1][lane],
                                               W.stash[r][2][lane], det_tab[det_row_first(r)].w, p.x, p.y,
                                               p.z, sd.w);
                    }
                }
            }
        } else {
            for (int i = grp_first(g); i < grp_first(g + 1); i++) {
                const float4 sd = c_det[i];
                const float3 p = place_reg(T, sd);
                uint32_t m = nr;
                while (m) {
                    const int r = __ffs(m) - 1;
                    m &= m - 1;
                    h |= hit_sphere_sphere(W.stash[r][0][lane], W.stash[r][1][lane],
                                           W.stash[r][2][lane], det_tab[det_row_first(r)].w, p.x, p.y, p.z,
                                           sd.w);
                }
            }
        }
        if (h) {
            c.set_hit();
            return;
        }
    }
}

// ---------------------------------------------------------------------------
// Screen of the detailed intra-arm rows whose first sphere is on joints 0..4
// (the "low" rows: 0..16 in the composite reading, 0..12 by sphere index).
// They are flagged whenever the arm's big approx spheres overlap, in most
// edges, and hardly ever fire; finding that out by walking the chain costs a
// row x sub-group test per lane and joint.  Here one pass covers every arm
// with low rows flagged: the warp's lanes are (arm, sub-interval of the slot's
// samples), each evaluates the arm at its sub-interval's middle and tests each
// low row's first sphere against the target sub-groups' bounds, grown by how
// far the joints between can move the target within the sub-interval.  The
// target centres are carried inward frame by frame (F_j Rz(q_j) from joint 7
// to joint 2), so that the first spheres are compile-time constants of their
// own frames and the base and joint 1 do not enter.  Of the arms with low rows
// flagged, five in six (5 arms) to half (one arm) need no walk after it.
// Measured with the rows in a kernel of their own, detailed phase: 262144
// 5-arm edges x 64 samples 4.47 -> 3.35 ms, 65536 shortcut edges 3.82 -> 2.55
// ms, 65536 4-arm edges 505 -> 457 us, 30011 one-arm edges 147 -> 139 us.
// ---------------------------------------------------------------------------
struct RowScreen {
    uint32_t rows;  // this lane's (arm, sub-interval): rows that may fire
    uint32_t arms;  // arms screened, in lane order
    int sub;        // sub-intervals per arm
};

// Largest distance of the centre of target sub-group 5 + t from joint j's
// axis (2..7) over all poses, in metres, rounded up; 0 where joint j does not
// move it against joints 0..4.  In frame 4 a target of joint 5 at (rho, c_z)
// from axis 5 is within hypot(0.0825, 0.384 + c_z) + rho of the origin, one
// further out within 0.393 m plus its distance from joint 6's origin; every
// frame inward adds its translation (0.0825, 0.316).
__host__ __device__ __forceinline__ constexpr float row_reach(int t, int j) {
    constexpr float kReach[6][6] = {
        //  j = 2   3       4       5       6       7
        {0.860f, 0.544f, 0.461f, 0.067f, 0.000f, 0.000f},  // 5
        {0.630f, 0.313f, 0.230f, 0.027f, 0.000f, 0.000f},  // 6
        {0.790f, 0.473f, 0.391f, 0.089f, 0.000f, 0.000f},  // 7
        {0.837f, 0.520f, 0.437f, 0.044f, 0.044f, 0.000f},  // 8
        {0.955f, 0.638f, 0.556f, 0.162f, 0.162f, 0.044f},  // 9
        {0.981f, 0.664f, 0.581f, 0.188f, 0.188f, 0.002f}}; // 10
    return kReach[t][j - 2];
}
// The table against the model's numbers, by the argument above.
constexpr bool row_reach_holds() {
    constexpr int kJoint[6] = {5, 5, 5, 6, 7, 7};
    const double fold = const_hypot(kJointK.v[3][1], kJointK.v[3][2]);  // joint 6's origin in frame 4
    for (int t = 0; t < 6; t++) {
        const float4 c = set_ball(grp_first(5 + t), (1u << (grp_first(6 + t) - grp_first(5 + t))) - 1u);
        const double rho = const_hypot(c.x, c.y), z = c.z > 0 ? c.z : -c.z;
        // from joint 6's origin, at most
        const double wrist = kJoint[t] == 7 ? const_hypot(kJointK.v[5][1] + rho, z) : const_hypot(rho, z);
        double need[6] = {};  // joints 2..7
        if (kJoint[t] == 7) need[5] = rho;
        if (kJoint[t] >= 6) need[4] = kJoint[t] == 6 ? rho : wrist;
        need[3] = kJoint[t] == 5 ? rho : wrist;
        need[2] = kJoint[t] == 5 ? const_hypot(kJointK.v[3][1], kJointK.v[3][2] + c.z) + rho : fold + wrist;
        need[1] = need[2] + kJointK.v[2][1];
        need[0] = need[1] - kJointK.v[1][2];
        for (int j = 2; j <= 7; j++)
            if (row_reach(t, j) < need[j - 2] || (j <= kJoint[t] && row_reach(t, j) == 0.0f)) return false;
    }
    return kJointK.v[0][1] == 0.f && kJointK.v[0][2] == 0.f && kJointK.v[1][1] == 0.f && kJointK.v[2][2] == 0.f &&
           kJointK.v[4][1] == 0.f && kJointK.v[4][2] == 0.f && kJointK.v[5][2] == 0.f;
}
static_assert(row_reach_holds(), "reach of the rows' targets");

// The rows as screen_rows reads them: radii of their first spheres, and targets
// that are the sub-groups 5..10, 5..7 or 9..10.
constexpr bool low_rows_as_screened() {
    if (kDet[0].r > 0.08f || kDet[0].x != 0.f || kDet[0].y != 0.f) return false;
    for (int r = 1; r <= 16; r++)
        if (kDet[det_row_first(r)].r > 0.06f) return false;
    for (int r = 0; r <= 16; r++) {
        const int lo = r <= 4 ? 5 : r <= 12 && r % 2 == 1 ? 5 : 9, hi = lo == 5 && r > 4 ? 7 : 10;
        if (det_row_lo(r) < grp_first(lo) || det_row_hi(r) >= grp_first(hi + 1)) return false;
    }
    for (int r = 5; r <= 12; r++)
        if (det_row_first(r) != 5 + (r - 5) / 2) return false;
    return det_joint(4) == 1 && det_joint(8) == 2 && det_joint(12) == 3 && det_joint(16) == 4;
}
static_assert(low_rows_as_screened(), "rows of the screen");

// Target centre p through joint J: F_J Rz(q) p (see joint_step for F_J).
template <int J>
__device__ __forceinline__ void carry_inward(float3 &p, float c, float s) {
    const float x = c * p.x - s * p.y, y = s * p.x + c * p.y;
    if constexpr (J == 2) p = make_float3(x, p.z, -y);
    else if constexpr (J == 5) p = make_float3(x - 0.0825f, p.z + 0.384f, -y);
    else if constexpr (J == 3) p = make_float3(x, -p.z - 0.316f, y);
    else if constexpr (J == 4) p = make_float3(x + 0.0825f, -p.z, y);
    else if constexpr (J == 6) p = make_float3(x, -p.z, y);
    else p = make_float3(x + 0.088f, -p.z, y);  // J == 7
}

// The targets' centres and squared reaches (bound + the row's sphere radius +
// motion) in the current frame.
struct RowTargets {
    float3 c[6];   // sub-groups 5..10
    float mv[6];   // motion within the sub-interval against the current frame
    float rr[6];   // (bound + first sphere's radius + motion)^2 for the current joint
    template <int J>
    __device__ __forceinline__ void step(float cq, float sq, float dq) {
#pragma unroll
        for (int t = 0; t < 6; t++) {
            if (row_reach(t, J) == 0.0f) continue;
            carry_inward<J>(c[t], cq, sq);
            mv[t] = fmaf(dq, row_reach(t, J), mv[t]);
        }
    }
    __device__ __forceinline__ void reach(const EdgeParams &P, float r) {
#pragma unroll
        for (int t = 0; t < 6; t++) {
            const float v = c_bounds.grp[5 + t].w + r + mv[t];
            rr[t] = v * v;
        }
    }
    // some sub-group of t0..t1 within reach of a sphere at (x, y, z)
    template <int T0, int T1>
    __device__ __forceinline__ bool near(float x, float y, float z) const {
        bool n = false;
#pragma unroll
        for (int t = T0 - 5; t <= T1 - 5; t++) {
            const float dx = c[t].x - x, dy = c[t].y - y, dz = c[t].z - z;
            n |= dx * dx + dy * dy + dz * dz < rr[t];
        }
        return n;
    }
};

// Every lane of the warp calls it.  sw: the lane's self flag words (0 for a
// lane without a self candidate); arms_in: arms to screen.
template <int A>
__device__ __forceinline__ RowScreen screen_rows(const EdgeParams &P, const EdgeScratch &W, int seg, int k0, Flags<A> sw,
                                                 int quirk, uint32_t arms_in) {
    const int lane = threadIdx.x & 31;
    RowScreen out;
    out.rows = kFull;
    out.arms = 0;
    out.sub = 32;
    const uint32_t lo = __reduce_or_sync(kFull, (uint32_t)sw & 0x1f1f1f1fu);
    uint32_t hi = 0;
    if constexpr (A > 4) hi = __reduce_or_sync(kFull, (uint32_t)(sw >> 32) & 0x1fu);
    uint32_t joints = 0;
#pragma unroll
    for (int a = 0; a < A; a++) {
        const uint32_t u = a < 4 ? lo >> (8 * a) & 0x1fu : hi;
        if (u && (P.rigid & arms_in) >> a & 1) {
            out.arms |= 1u << a;
            joints |= u;
        }
    }
    if (!out.arms) return out;
    int arm = 0, sub = lane;
    if (A > 1) {
        const int n = __popc(out.arms);
        out.sub = n == 1 ? 32 : n == 2 ? 16 : n == 3 ? 10 : n == 4 ? 8 : 6;
        int ai = min(lane / out.sub, n - 1);
        sub = min(lane - ai * out.sub, out.sub - 1);
        uint32_t m = out.arms;
        for (; ai > 0; ai--) m &= m - 1;
        arm = __ffs(m) - 1;
    }
    // lanes ilo..ihi of the slot (lane i belongs to sub-interval i * sub / 32)
    const int ilo = (32 * sub + out.sub - 1) / out.sub, ihi = (32 * (sub + 1) + out.sub - 1) / out.sub - 1;
    const int klo = min(k0 + 1 + ilo, P.g), khi = min(k0 + 1 + ihi, P.g);
    const float mid = 0.5f * (float)(klo + khi), half = 0.5f * (float)(khi - klo);
    float q[7], dq[7], sum = 0.0f;  // joint 1 enters only the range check
#pragma unroll
    for (int j = 0; j < 7; j++) {
        const int i = 7 * (P.single ? 0 : arm) + j;
        q[j] = fmaf(mid, W.stepg[i], W.base[i]);
        dq[j] = fmaf(half, fabsf(W.stepg[i]), 1e-5f);
        if (P.rule == kRuleBspline || P.rule == kRuleShortcut) {
            // the samples add delta seg times (sample_q): each addition errs by
            // up to 2^-24 of a value no larger than `big` and the error so far,
            // always the same way within a power of two (4000 segments at 20 rad:
            // 3.7e-3 rad).  6.05e-8 is 2^-24 and the 1/256 that the errors of
            // 65536 additions can add to `big`, with room for the rounding here
            static_assert(kMaxSegments <= 1 << 16, "room for the additions' own errors");
            const float n = (float)seg, move = n * fabsf(W.delta[i]);
            const float big = fmaf(half, fabsf(W.stepg[i]), fabsf(q[j]) + move);
            q[j] = fmaf(n, W.delta[i], q[j]);
            dq[j] = fmaf(n * 6.05e-8f, big, dq[j]);
        }
        sum += fabsf(q[j]) + dq[j];
    }
    RowTargets t;
#pragma unroll
    for (int i = 0; i < 6; i++) {
        t.c[i] = make_float3(c_bounds.grp[5 + i].x, c_bounds.grp[5 + i].y, c_bounds.grp[5 + i].z);
        t.mv[i] = 0.0f;
    }
    uint32_t rows = quirk ? ~0x1ffffu : ~0x1fffu;
    t.step<7>(__cosf(q[6]), __sinf(q[6]), dq[6]);
    t.step<6>(__cosf(q[5]), __sinf(q[5]), dq[5]);
    t.step<5>(__cosf(q[4]), __sinf(q[4]), dq[4]);
#define MRPOP_NEAR(i, T0, T1) t.near<T0, T1>(kDet[i].x, kDet[i].y, kDet[i].z)
    // composite reading: row r reads sphere r (first radii 0.06 at most)
    if (quirk && joints >> 4) {
        t.reach(P, 0.06f);
        if (MRPOP_NEAR(13, 9, 10)) rows |= 1u << 13;
        if (MRPOP_NEAR(14, 9, 10)) rows |= 1u << 14;
        if (MRPOP_NEAR(15, 9, 10)) rows |= 1u << 15;
        if (MRPOP_NEAR(16, 9, 10)) rows |= 1u << 16;
    }
    t.step<4>(__cosf(q[3]), __sinf(q[3]), dq[3]);
    if (quirk && (joints >> 3 & 1)) {
        t.reach(P, 0.06f);
        if (MRPOP_NEAR(9, 5, 7)) rows |= 1u << 9;
        if (MRPOP_NEAR(10, 9, 10)) rows |= 1u << 10;
        if (MRPOP_NEAR(11, 5, 7)) rows |= 1u << 11;
        if (MRPOP_NEAR(12, 9, 10)) rows |= 1u << 12;
    }
    t.step<3>(__cosf(q[2]), __sinf(q[2]), dq[2]);
    if (joints >> 2 & 1) {
        t.reach(P, 0.06f);
        if (quirk) {
            if (MRPOP_NEAR(5, 5, 7)) rows |= 1u << 5;
            if (MRPOP_NEAR(6, 9, 10)) rows |= 1u << 6;
            if (MRPOP_NEAR(7, 5, 7)) rows |= 1u << 7;
            if (MRPOP_NEAR(8, 9, 10)) rows |= 1u << 8;
        } else {  // spheres 5..8, a forearm and a hand row each
            if (MRPOP_NEAR(5, 5, 7)) rows |= 1u << 5;
            if (MRPOP_NEAR(5, 9, 10)) rows |= 1u << 6;
            if (MRPOP_NEAR(6, 5, 7)) rows |= 1u << 7;
            if (MRPOP_NEAR(6, 9, 10)) rows |= 1u << 8;
            if (MRPOP_NEAR(7, 5, 7)) rows |= 1u << 9;
            if (MRPOP_NEAR(7, 9, 10)) rows |= 1u << 10;
            if (MRPOP_NEAR(8, 5, 7)) rows |= 1u << 11;
            if (MRPOP_NEAR(8, 9, 10)) rows |= 1u << 12;
        }
    }
    t.step<2>(__cosf(q[1]), __sinf(q[1]), dq[1]);
    if (joints >> 1 & 1) {
        t.reach(P, 0.06f);
        if (MRPOP_NEAR(1, 5, 10)) rows |= 1u << 1;
        if (MRPOP_NEAR(2, 5, 10)) rows |= 1u << 2;
        if (MRPOP_NEAR(3, 5, 10)) rows |= 1u << 3;
        if (MRPOP_NEAR(4, 5, 10)) rows |= 1u << 4;
    }
    if (joints & 1u) {
        t.reach(P, 0.08f);
        // sphere 0 of the base lies on joint 1's axis, 0.283 m below its frame
        if (t.near<5, 10>(0.0f, 0.0f, kDet[0].z - 0.333f)) rows |= 1u;
    }
#undef MRPOP_NEAR
    if (sum <= kRegularRad) out.rows = rows;  // (false for NaN)
    return out;
}

// Lower arm, joint j (flagged for this lane): its spheres from index `from` on
// that can reach one of the upper arm's sets gb (bounds, centres in W.cross.gc)
// go to the lane's stash with the sets they reach; `next` receives the first
// sphere left out when the stash is full.
template <bool PARTS, typename WS>
__device__ __forceinline__ void stash_joint(int j, const EdgeParams &P, const Xf &T, uint32_t gb, int from, int &n,
                                            int &next, WS &W, int lane) {
    auto &X = W.cross;
#pragma unroll 1
    for (int g = jgrp_first(j); g < jgrp_first(j + 1); g++) {
        if (grp_first(g + 1) <= from) continue;
        const float4 gl = c_bounds.grp[g];
        const float3 gc = place_reg(T, gl);
        const float gr = gl.w + P.slack;  // (covers both sets)
        uint32_t near = 0;
        for (uint32_t m = gb; m; m &= m - 1) {
            const int t = __ffs(m) - 1;
            if (near3(gc.x, gc.y, gc.z,
                      make_float4(X.gc[t][0][lane], X.gc[t][1][lane], X.gc[t][2][lane], set_bound<PARTS>(t).w), gr))
                near |= 1u << t;
        }
        if (!near) continue;
#pragma unroll 1
        for (int at = max(grp_first(g), from); at < grp_first(g + 1); at++) {
            const float4 sd = c_det[at];
            const float3 p = place_reg(T, sd);
            const float sr = sd.w + P.slack;
            uint32_t nm = 0;
            for (uint32_t m = near; m; m &= m - 1) {
                const int t = __ffs(m) - 1;
                if (near3(p.x, p.y, p.z,
                          make_float4(X.gc[t][0][lane], X.gc[t][1][lane], X.gc[t][2][lane], set_bound<PARTS>(t).w), sr))
                    nm |= 1u << t;
            }
            if (!nm) continue;
            if (n == WS::kStash) {
                next = at;
                return;
            }
            X.xs[n][0][lane] = p.x;
            X.xs[n][1][lane] = p.y;
            X.xs[n][2][lane] = p.z;
            X.xs[n][3][lane] = sd.w;
            X.xm[n][lane] = nm;
            n++;
        }
    }
}

// Upper arm, joint j: its spheres against the stashed spheres that reach their
// set.
template <bool PARTS, typename WS>
__device__ __forceinline__ void probe_joint(int j, const Xf &T, int n, bool &hit, WS &W, int lane) {
    auto &X = W.cross;
#pragma unroll 1
    for (int g = jgrp_first(j); g < set_end<PARTS>(j); g++) {
        uint32_t em = 0;
        for (int e = 0; e < n; e++) em |= (X.xm[e][lane] >> g & 1u) << e;
        if (!em) continue;
        bool h = false;
        for (uint32_t rest = set_spheres<PARTS>(g); rest; rest &= rest - 1) {
            const float4 sd = c_det[set_first(g) + __ffs(rest) - 1];
            const float3 p = place_reg(T, sd);
            for (uint32_t m = em; m; m &= m - 1) {
                const int e = __ffs(m) - 1;
                // sphere_1 = the lower arm's sphere (panda_four.cuh:441-443)
                h |= hit_sphere_sphere(X.xs[e][0][lane], X.xs[e][1][lane], X.xs[e][2][lane], X.xs[e][3][lane], p.x,
                                       p.y, p.z, sd.w);
            }
        }
        if (h) {
            hit = true;
            return;
        }
    }
}

// Shared words of a CTA whose warps take one arm each (armwise_kernel).
struct ArmShare {
    unsigned long long env[2][32], self[2][32];  // [slot][lane] flag words of the segment
    unsigned int hits[2];                        // [slot] lanes whose sample collided
    unsigned int pm[2][num_pairs(kMaxArms)];     // [slot][pair] joints connected by swept bounds
    unsigned int next[3];                        // arm pairs handed out: broad, narrow slot 0, slot 1
};

// The next arm pair for this warp from counter *c (lane 0 takes it).
__device__ __forceinline__ int take_pair(unsigned int *c, int lane) {
    unsigned int p = 0;
    if (lane == 0) p = atomicAdd(c, 1u);
    return (int)__shfl_sync(kFull, p, 0);
}

// Detailed check of one slot: this lane's sample is k0 + lane + 1 (lanes past
// the segment's last sample keep the others company on it, so that the warp's
// merged bounds stay on real samples); dE, dS: it is an env / self candidate.
// Every lane of the warp calls it.  Returns the lanes whose test fired, of
// which the lowest counts: once a lane's test has fired the lanes above it
// stop.
//
// Every test is a walk along one arm's joint chain with all lanes in step, and
// one loop runs them all (a job each), so that the kernel holds the chain step
// once and its code stays within the instruction cache.
//   arm      obstacles against the env-flagged joints (warp-wide screens), and
//            the intra-arm rows left by screen_rows and the forearm-hand table
//   centres, stash, probe
//            one arm pair a < b (panda_four.cuh:415-453), cut to the joints
//            that some approx sphere pair's swept bounds connect in the slot
//            (pms: lane p holds pair p's; a joint's detailed spheres lie inside
//            its approx spheres but for 0.6 mm, and those bounds carry 1 mm
//            each).  Arm b's sub-group centres are placed first (the hand in
//            its three parts); arm a's spheres are tested against them by
//            sub-group and one by one, so
//            that only spheres that can reach arm b are stashed; arm b is
//            walked again only if some lane stashed any.
// Bound by instruction issue.  Against the first form of the arm-pair test
// (all 121 sub-group pairs of every arm pair screened, every flagged sphere
// stashed, lanes above a hit going on): 262144 5-arm edges x 64 samples 11.90
// -> 10.26 ms, 65536 shortcut edges 7.36 -> 6.37 ms.
//
// STAGE: which tests this kernel runs.  The split pipeline's composite kernels
// run the rows, which seldom fire, in a kernel of their own after the others
// (rows_kernel): with all of them the narrow kernel's code, 51 KB, missed the
// SM's instruction cache (15 times the misses of a 45 KB build; 65536 4-arm
// edges 505 -> 603 us), and random edges that collide mostly do so with an
// obstacle or another arm at their first samples.
// ONE (armwise_kernel): only arm one_arm's env and row tests, then the slot's
// arm pairs one at a time to whichever warp of the CTA is free (X->next); hits
// are shared through X->hits (a stale read only costs tests).
constexpr int kStageAll = 0, kStageEnvPairs = 1, kStageRows = 2;

template <int A, bool ONE = false, int STAGE = kStageAll, typename WS>
__device__ __forceinline__ uint32_t narrow_slot(const EdgeParams &P, WS &W, const float4 *S,
                                                const SceneLayout &L, const float4 *det_tab, int seg, int k0,
                                                Flags<A> ew, Flags<A> sw, bool dE, bool dS, uint32_t pms,
                                                int one_arm = 0, ArmShare *X = nullptr, int slot = 0) {
    const int lane = threadIdx.x & 31;
    const int k = min(k0 + lane + 1, P.g);
    static_assert(!ONE || STAGE == kStageAll, "the arm-per-warp kernel runs every test");
    constexpr bool with_env = STAGE != kStageRows, with_rows = STAGE == kStageAll || STAGE == kStageRows;
    constexpr bool with_pairs = A > 1 && STAGE != kStageRows;
    constexpr int kArm = 0, kCentres = 1, kStash = 2, kProbe = 3;  // jobs
    // The upper arm's hand in its three parts: fewer spheres reach it, at more
    // tests each.  The slowest edges gain (300 5-arm extend checks 92.7 -> 80
    // us, with a stash of 10 in place of 8), and 65536 4-arm edges (433 -> 411
    // us); 262144 5-arm edges, most of which collide at their first sample,
    // took 3.43 in place of 3.27 ms.
    constexpr bool kParts = ONE || A <= 4;
    const int arm0 = ONE ? one_arm : 0, arm1 = ONE ? one_arm + 1 : A;
    LaneCtx c;
    c.quirk = (!P.single && !(P.flags & kExactBit)) ? 1 : 0;
    c.hit = false;
    bool act = dE || dS;  // this lane's sample is not settled
    bool pair_phase = false;
    int arm_next = arm0;
    RowScreen rs = {kFull, 0u, 32};
    if (with_rows) rs = screen_rows<A>(P, W, seg, k0, dS ? sw : 0, c.quirk, ONE ? 1u << one_arm : kFull);
    // the arm pair in hand: its state (0: none, 1: centres placed, 2: stashed,
    // 3: probed), arms, joints, and the lane's stash
    int xs = 0, pa = 0, pb = 0, from = 0, n = 0, next = 0;
    uint32_t pairs = with_pairs && !ONE ? __ballot_sync(kFull, pms != 0) : 0u, jb = 0, uj = 0, sma = 0;
#pragma unroll 1
    for (;;) {
        // the next job: its kind, arm and last joint (the same in every lane)
        int job, arm, top;
        if (with_pairs && pair_phase) {
            if (xs == 2 && __any_sync(kFull, act && n > 0)) {
                job = kProbe;
                xs = 3;
            } else {
                if (xs >= 2) {  // this stash is done: the spheres left out, if any
                    from = act ? next : kNumDet;
                    xs = __any_sync(kFull, from < kNumDet) ? 1 : 0;
                }
                if (xs == 1) {
                    job = kStash;
                    xs = 2;
                    n = 0;
                    next = kNumDet;
                } else {
                    uint32_t m = 0, rest = pairs;
                    if (ONE) {
                        const int t = take_pair(&X->next[1 + slot], lane);
                        for (int i = 0; i < t && rest; i++) rest &= rest - 1;
                    }
                    if (!rest) break;
                    const int p = __ffs(rest) - 1;
                    if (!ONE) pairs &= pairs - 1;
                    m = ONE ? X->pm[slot][p] : __shfl_sync(kFull, pms, p);
                    pair_arms<A>(p, pa, pb);
                    jb = m >> 8;
                    sma = act && dS ? (uint32_t)(sw >> (8 * pa)) & m & 0xffu : 0u;
                    uj = __reduce_or_sync(kFull, sma);
                    if (!uj) continue;
                    from = sma ? 0 : kNumDet;
                    job = kCentres;
                    xs = 1;
                }
            }
            arm = job == kStash ? pa : pb;
            top = 31 - __clz(job == kStash ? uj : jb);
        } else {
            if (arm_next == arm1) {
                if (!with_pairs) break;
                pair_phase = true;
                if (ONE) pairs = __ballot_sync(kFull, lane < num_pairs(A) && X->pm[slot][lane] != 0);
                continue;
            }
            arm = arm_next++;
            c.em = c.rm = 0;
            top = -1;
            if (with_env) {
                if (act && dE) c.em = (uint32_t)(ew >> (8 * arm)) & 0xffu;
                const uint32_t u = __reduce_or_sync(kFull, c.em);
                if (u) top = 31 - __clz(u);
            }
            if (with_rows) {
                const uint32_t sm = act && dS ? (uint32_t)(sw >> (8 * arm)) & 0xffu : 0u;
                if (sm) c.rm = row_mask(sm, c.quirk != 0);
                const int q6 = 7 * (P.single ? 0 : arm) + 5;
                if (P.row5 && (c.rm & row5_rows(c.quirk)) &&
                    row5_apart(P.row5, sample_q1(W, P.rule, seg, q6, k), sample_q1(W, P.rule, seg, q6 + 1, k)))
                    c.rm &= ~row5_rows(c.quirk);
                if (rs.arms >> arm & 1u)
                    c.rm &= __shfl_sync(kFull, rs.rows,
                                        __popc(rs.arms & ((1u << arm) - 1u)) * rs.sub + (lane * rs.sub >> 5));
                const uint32_t u = __reduce_or_sync(kFull, c.rm);
                if (u) top = max(top, u & ~kForearmRows ? 7 : 5);
            }
            if (top < 0) continue;
            job = kArm;
        }
        // walk the arm's chain
        const uint32_t before = __ballot_sync(kFull, c.hit);
        const uint32_t gb = joint_sets<kParts>(jb);
        Xf T;
        load_base(T, P.base[arm]);
#pragma unroll 1
        for (int j = 0;; j++) {
            if (with_pairs && job != kArm) {
                if (job == kStash) {
                    if ((sma >> j & 1u) && next == kNumDet && from < det_first(j + 1))
                        stash_joint<kParts>(j, P, T, gb, from, n, next, W, lane);
                } else if (jb >> j & 1u) {
                    if (job == kCentres) {
#pragma unroll 1
                        for (int g = jgrp_first(j); g < set_end<kParts>(j); g++) {
                            const float3 ctr = place_reg(T, set_bound<kParts>(g));
                            W.cross.gc[g][0][lane] = ctr.x;
                            W.cross.gc[g][1][lane] = ctr.y;
                            W.cross.gc[g][2][lane] = ctr.z;
                        }
                    } else if (act && !c.hit && n > 0) {
                        probe_joint<kParts>(j, T, n, c.hit, W, lane);
                    }
                }
            } else {
                if (with_env) lane_env(j, P, T, c, S, L);
                if (with_rows) lane_rows<A>(j, P, T, c, W, det_tab, lane);
                const uint32_t hb = __ballot_sync(kFull, c.hit);
                if (hb != before) {
                    if (hb & lanes_upto(lane)) c.em = c.rm = 0;
                    if (!__any_sync(kFull, c.em | c.rm)) break;
                }
            }
            if (j == top) break;
            joint_step_rt(T, sample_q1(W, P.rule, seg, 7 * (P.single ? 0 : arm) + j, k), j + 1);
        }
        uint32_t hb = __ballot_sync(kFull, c.hit);
        if (ONE) {
            if (lane == 0 && hb != before) atomicOr(&X->hits[slot], hb);
            hb |= *(const volatile unsigned int *)&X->hits[slot];
            if (slot > 0 && *(const volatile unsigned int *)&X->hits[0]) hb = kFull;  // settles the edge
        }
        act = act && !(hb & lanes_upto(lane));
        if (!__any_sync(kFull, act)) break;
    }
    return __ballot_sync(kFull, c.hit);
}

// ---------------------------------------------------------------------------
// per-edge building blocks shared by the kernels
// ---------------------------------------------------------------------------
// Edge set-up: segment start and per-sample / per-segment steps of every dof
// into warp scratch (call-site formulas, see the rule constants).  Returns
// the segment count; too_many marks counts beyond kMaxSegments.
__device__ __forceinline__ int edge_setup(const EdgeParams &P, EdgeScratch &W, long long e, int dof, int g, int lane,
                                          bool &too_many) {
    const float *qa = P.q0 + e * dof, *qb = P.q1 + e * dof;
    float diff0 = 0.f, diff1 = 0.f;
    if (lane < dof) diff0 = __fsub_rn(qb[lane], qa[lane]);
    if (lane + 32 < dof) diff1 = __fsub_rn(qb[lane + 32], qa[lane + 32]);
    int nseg = 1;
    too_many = false;
    if (P.rule != kRulePlain) {
        // |q1 - q0| with the reference's sequential FMA chain (utils.cuh:123-133)
        float acc = 0.0f;
        for (int d = 0; d < dof; d++) {
            const float v = __shfl_sync(kFull, d < 32 ? diff0 : diff1, d & 31);
            acc = __fmaf_rn(v, v, acc);
        }
        const float dist = __fsqrt_rn(acc);
        float n;
        if (P.rule == kRuleConnect) n = truncf(__fdiv_rn(dist, P.range)) + 1.0f;
        else if (P.rule == kRuleBspline) n = ceilf(__fdiv_rn(dist, P.range));
        else n = ceilf(__fdiv_rn(__fsub_rn(dist, 0.001f), P.range));
        if (n > (float)kMaxSegments) too_many = true;
        else nseg = (int)n; // may be <= 0: no segment is checked (the reference's loop runs 0 times)
    }
    for (int d = lane; d < dof; d += 32) {
        const float df = d < 32 ? diff0 : diff1;
        W.base[d] = qa[d];
        if (P.rule == kRulePlain) {
            W.stepg[d] = __fdiv_rn(df, (float)g);
            W.delta[d] = 0.0f;
        } else {
            const float step = __fdiv_rn(df, (float)nseg);
            W.delta[d] = step;
            W.stepg[d] = __fdiv_rn(step, (float)g);
        }
    }
    __syncwarp();
    return nseg;
}

// CONNECT: the segment start of segment `seg` (the caller's loop adds the
// per-segment step once per finished segment, pop_planner.cu:697).
__device__ __forceinline__ void connect_advance(EdgeScratch &W, int dof, int seg, int lane) {
    for (int d = lane; d < dof; d += 32) {
        float b = W.base[d];
        for (int s = 0; s < seg; s++) b = __fadd_rn(b, W.delta[d]);
        W.base[d] = b;
    }
    __syncwarp();
}

// The candidate masks of a segment from its samples' flag counts (totals over
// the segment given): every flagged sample in EXACT mode, else the samples the
// reference's proportional 4g-thread split gives at least one thread
// (utils.cuh:476-517), the remainder going to the last sample.
template <int SPL>
__device__ __forceinline__ void thread_split(bool exact, int g, int lane, const int (&envc)[SPL],
                                             const int (&selfc)[SPL], int tot_env, int tot_self, uint64_t &cand_env,
                                             uint64_t &cand_self) {
    if (exact) {
#pragma unroll
        for (int s = 0; s < SPL; s++) {
            const uint64_t be = __ballot_sync(kFull, envc[s] > 0);
            const uint64_t bs = __ballot_sync(kFull, selfc[s] > 0);
            cand_env |= be << (32 * s);
            cand_self |= bs << (32 * s);
        }
        return;
    }
    int de[SPL], ds[SPL], sum_e = 0, sum_s = 0;
#pragma unroll
    for (int s = 0; s < SPL; s++) {
        const int k = lane + 1 + 32 * s;
        de[s] = k <= g ? ref_share(envc[s], tot_env, g) : 0;
        ds[s] = k <= g ? ref_share(selfc[s], tot_self, g) : 0;
        sum_e += de[s];
        sum_s += ds[s];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        sum_e += __shfl_xor_sync(kFull, sum_e, o);
        sum_s += __shfl_xor_sync(kFull, sum_s, o);
    }
#pragma unroll
    for (int s = 0; s < SPL; s++) {
        const int k = lane + 1 + 32 * s;
        if (k == g) { // the remainder goes to the last sample
            de[s] += 4 * g - sum_e;
            ds[s] += 4 * g - sum_s;
        }
        const uint64_t be = __ballot_sync(kFull, tot_env > 0 && de[s] > 0);
        const uint64_t bs = __ballot_sync(kFull, tot_self > 0 && ds[s] > 0);
        cand_env |= be << (32 * s);
        cand_self |= bs << (32 * s);
    }
}

// Broad phase of one segment for this lane's samples plus the decision: which
// samples get the detailed check (the reference's thread split, or every
// flagged sample in EXACT mode).  Returns false when no sample is flagged.
template <int A, int SPL>
__device__ __forceinline__ bool broad_decide(const EdgeParams &P, const EdgeScratch &W, BroadPart &B, const float4 *S,
                                             const SceneLayout &L, int seg, int g, int lane, Flags<A> (&envw)[SPL],
                                             Flags<A> (&selfw)[SPL], uint32_t (&pm)[SPL], uint64_t &cand_env,
                                             uint64_t &cand_self, long long e, bool first) {
    MRPOP_PHASE_START();
    int envc[SPL], selfc[SPL];
    int tot_env = 0, tot_self = 0;
    // one copy of the per-sample code for both slots (not unrolled); slot
    // arrays are written by constant index so they stay in registers
#pragma unroll 1
    for (int s = 0; s < SPL; s++) {
        const int k = lane + 1 + 32 * s;
        Flags<A> ew, sw;
        uint32_t pw;
        broad_sample<A>(P, W, B, S, L, seg, k <= g ? k : g, ew, sw, pw);
        if (k > g) ew = sw = 0;
        const int ec = flag_count<A>(ew), sc = flag_count<A>(sw);
        if (s == 0) {
            envw[0] = ew;
            selfw[0] = sw;
            pm[0] = pw;
            envc[0] = ec;
            selfc[0] = sc;
        } else {
            envw[SPL - 1] = ew;
            selfw[SPL - 1] = sw;
            pm[SPL - 1] = pw;
            envc[SPL - 1] = ec;
            selfc[SPL - 1] = sc;
        }
        tot_env += ec;
        tot_self += sc;
    }
    __syncwarp();
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        tot_env += __shfl_xor_sync(kFull, tot_env, o);
        tot_self += __shfl_xor_sync(kFull, tot_self, o);
    }
    if (P.flops && lane == 0) P.flops[e] = (first ? 0.0 : P.flops[e]) + P.fbp * g;
    cand_env = cand_self = 0;
    if (tot_env == 0 && tot_self == 0) return false;
    MRPOP_PHASE(P, 7);
    thread_split<SPL>((P.flags & kExactBit) != 0, g, lane, envc, selfc, tot_env, tot_self, cand_env, cand_self);
    if (P.flops) {
        double f = 0.0;
#pragma unroll
        for (int s = 0; s < SPL; s++) {
            const int bit = lane + 32 * s;
            const bool dE = cand_env >> bit & 1ull, dS = cand_self >> bit & 1ull;
            if (dE || dS) f += narrow_flops(P, P.single ? 1 : A, envw[s], selfw[s], dE, dS);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) f += __shfl_xor_sync(kFull, f, o);
        if (lane == 0) P.flops[e] += f;
    }
    MRPOP_PHASE(P, 4);
    return true;
}

// Detailed phase of one segment: every candidate sample in parallel, one lane
// each (samples k0 + 1 ..; k0 = 32 for the second warp of a pair).  Returns
// the 0-based index (from k0) of the first colliding sample, or 64.
template <int A, int SPL, int STAGE = kStageAll>
__device__ __forceinline__ int narrow_segment(const EdgeParams &P, WarpScratch &W, const float4 *S,
                                              const SceneLayout &L, const float4 *det_tab, int seg, int lane,
                                              const Flags<A> (&envw)[SPL], const Flags<A> (&selfw)[SPL],
                                              const uint32_t (&pm)[SPL], uint64_t cand_env, uint64_t cand_self,
                                              int k0 = 0) {
    MRPOP_PHASE_START();
    uint64_t hits = 0;
    // one copy of the per-sample code for both slots (not unrolled)
#pragma unroll 1
    for (int s = 0; s < SPL; s++) {
        const int bit = lane + 32 * s;
        const bool dE = cand_env >> bit & 1ull, dS = cand_self >> bit & 1ull;
        const Flags<A> ew = s == 0 ? envw[0] : envw[SPL - 1], sw = s == 0 ? selfw[0] : selfw[SPL - 1];
        const uint32_t hb = narrow_slot<A, false, STAGE>(P, W, S, L, det_tab, seg, k0 + 32 * s, ew, sw, dE, dS,
                                                         s == 0 ? pm[0] : pm[SPL - 1]);
        hits |= (uint64_t)hb << (32 * s);
        if (hits) break; // later slots hold only later samples
    }
    return hits ? __ffsll((long long)hits) - 1 : 64;
}

// Common kernel prologue: scene staged in shared memory, warp scratch.
#define MRPOP_KERNEL_PROLOGUE(Scratch)                                                                 \
    extern __shared__ __align__(128) unsigned char smem_raw[];                                         \
    __shared__ __align__(8) uint64_t bar;                                                              \
    __shared__ float4 det_tab[kNumDet];                                                                \
    const SceneLayout L = scene_layout(P.sc);                                                          \
    float4 *S = reinterpret_cast<float4 *>(smem_raw);                                                  \
    Scratch *Wall = reinterpret_cast<Scratch *>(smem_raw + (size_t)L.total * sizeof(float4));          \
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;                                        \
    Scratch &W = Wall[warp];                                                                           \
    for (int i = threadIdx.x; i < kNumDet; i += blockDim.x) det_tab[i] = c_det[i];                     \
    const bool staged = stage_scene(S, P.scene, (uint32_t)(L.total * sizeof(float4)), &bar, P.status); \
    MRPOP_PHASE_BIND(P);                                                                               \
    const int g = P.g;                                                                                 \
    const int dof = 7 * (P.single ? 1 : A);                                                            \
    const long long nwarps = (long long)gridDim.x * kWarpsPerBlock;                                    \
    (void)det_tab;

// ---------------------------------------------------------------------------
// fused kernel: every rule, segments in order with early exit
// ---------------------------------------------------------------------------
// One edge through the fused kernel: segments from P.seg0 in order, both
// phases per segment, early exit at the first colliding one.  Edges decided by
// earlier split rounds (P.seg0 > 0) are skipped.
template <int A, int SPL>
__device__ __forceinline__ void fused_edge(const EdgeParams &P, WarpScratch &W, const float4 *S, const SceneLayout &L,
                                           const float4 *det_tab, long long e, int dof, int g, int lane,
                                           bool staged) {
    if (!staged) {
        if (lane == 0) {
            P.valid[e] = 0;
            P.first_hit[e] = -2;
        }
        return;
    }
    if (P.seg0 > 0 && (P.sdone[e] || P.snseg[e] <= P.seg0)) return; // decided by the split rounds
    bool too_many;
    const int nseg = edge_setup(P, W, e, dof, g, lane, too_many);
    int first = 0;
    if (P.flops && P.seg0 == 0 && lane == 0) P.flops[e] = 0.0;
    const int nseg_run = too_many ? 0 : nseg;
    if (P.rule == kRuleConnect && P.seg0 > 0) connect_advance(W, dof, P.seg0, lane);
    for (int seg = P.seg0; seg < nseg_run && first == 0; seg++) {
        Flags<A> envw[SPL], selfw[SPL];
        uint64_t cand_env, cand_self;
        uint32_t pm[SPL];
        if (broad_decide<A, SPL>(P, W, W.broad, S, L, seg, g, lane, envw, selfw, pm, cand_env, cand_self, e,
                                 false)) {
            const int fb =
                narrow_segment<A, SPL>(P, W, S, L, det_tab, seg, lane, envw, selfw, pm, cand_env, cand_self);
            if (fb < 64) first = seg * g + fb + 1;
        }
        if (P.rule == kRuleConnect) {
            __syncwarp();
            for (int d = lane; d < dof; d += 32) W.base[d] = __fadd_rn(W.base[d], W.delta[d]);
            __syncwarp();
        }
    }
    if (lane == 0) {
        P.valid[e] = (first == 0 && !too_many) ? 1 : 0;
        P.first_hit[e] = too_many ? -2 : (first ? first : -1);
        if (P.n_seg_out) P.n_seg_out[e] = nseg;
    }
    __syncwarp();
}

template <int A, int SPL>
__global__ void __launch_bounds__(32 * kWarpsPerBlock, MRPOP_MIN_BLOCKS)
    validate_kernel(const __grid_constant__ EdgeParams P) {
    MRPOP_KERNEL_PROLOGUE(WarpScratch)
    for (long long e = (long long)blockIdx.x * kWarpsPerBlock + warp; e < P.n_edges; e += nwarps)
        fused_edge<A, SPL>(P, W, S, L, det_tab, e, dof, g, lane, staged);
}

// ---------------------------------------------------------------------------
// fused kernel, two warps per edge (granularity above 32, small calls): warp
// `half` of a pair takes samples 32 * half + 1 .. 32 * half + 32 of every
// segment, so an edge takes the time of one 32-sample slot instead of two.
// The thread split's totals and shares are summed over the pair (integers,
// so in any order), and both warps leave a segment together at its first hit:
// the verdicts are those of the one-warp kernels.
// ---------------------------------------------------------------------------
struct PairShare {
    int tot[2][2];  // [half] env, self flag totals of the slot
    int sum[2][2];  // [half] env, self thread shares of the slot
    int fb[2];      // [half] first colliding sample of the slot (from its k0), or 64
};

__device__ __forceinline__ void pair_sync(int id) { asm volatile("bar.sync %0, 64;" ::"r"(id) : "memory"); }

template <int A>
__device__ __forceinline__ void fused_edge_pair(const EdgeParams &P, WarpScratch &W, const float4 *S,
                                                const SceneLayout &L, const float4 *det_tab, long long e, int dof, int g,
                                                int lane, int half, PairShare &X, int bar_id, bool staged) {
    if (!staged) {
        if (half == 0 && lane == 0) {
            P.valid[e] = 0;
            P.first_hit[e] = -2;
        }
        return;
    }
    bool too_many;
    const int nseg = edge_setup(P, W, e, dof, g, lane, too_many);
    const int nseg_run = too_many ? 0 : nseg;
    const int k = lane + 1 + 32 * half;
    int first = 0;
    for (int seg = 0; seg < nseg_run && first == 0; seg++) {
        Flags<A> ew, sw;
        uint32_t pw;
        broad_sample<A>(P, W, W.broad, S, L, seg, k <= g ? k : g, ew, sw, pw);
        if (k > g) ew = sw = 0;
        const int ec = flag_count<A>(ew), sc = flag_count<A>(sw);
        int te = ec, ts = sc;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            te += __shfl_xor_sync(kFull, te, o);
            ts += __shfl_xor_sync(kFull, ts, o);
        }
        if (lane == 0) {
            X.tot[half][0] = te;
            X.tot[half][1] = ts;
        }
        pair_sync(bar_id);  // A: both slots' totals written
        const int tot_env = X.tot[0][0] + X.tot[1][0], tot_self = X.tot[0][1] + X.tot[1][1];
        if (tot_env > 0 || tot_self > 0) {
            bool cE, cS;
            if (P.flags & kExactBit) {
                cE = ec > 0;
                cS = sc > 0;
            } else {
                int de = k <= g ? ref_share(ec, tot_env, g) : 0, ds = k <= g ? ref_share(sc, tot_self, g) : 0;
                int se = de, ss = ds;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    se += __shfl_xor_sync(kFull, se, o);
                    ss += __shfl_xor_sync(kFull, ss, o);
                }
                if (lane == 0) {
                    X.sum[half][0] = se;
                    X.sum[half][1] = ss;
                }
                pair_sync(bar_id);  // B: shares written
                if (k == g) {  // the remainder goes to the last sample
                    de += 4 * g - (X.sum[0][0] + X.sum[1][0]);
                    ds += 4 * g - (X.sum[0][1] + X.sum[1][1]);
                }
                cE = tot_env > 0 && de > 0;
                cS = tot_self > 0 && ds > 0;
            }
            const uint64_t cand_env = __ballot_sync(kFull, cE), cand_self = __ballot_sync(kFull, cS);
            __syncwarp();
            const Flags<A> envw[1] = {ew}, selfw[1] = {sw};
            const uint32_t pm[1] = {pw};
            const int fb = (cand_env | cand_self)
                               ? narrow_segment<A, 1>(P, W, S, L, det_tab, seg, lane, envw, selfw, pm, cand_env,
                                                      cand_self, 32 * half)
                               : 64;
            if (lane == 0) X.fb[half] = fb;
            pair_sync(bar_id);  // C: both slots' first hits written
            const int f0 = X.fb[0], f1 = X.fb[1];
            if (f0 < 64) first = seg * g + f0 + 1;
            else if (f1 < 64) first = seg * g + 32 + f1 + 1;
        }
        if (P.rule == kRuleConnect) {
            __syncwarp();
            for (int d = lane; d < dof; d += 32) W.base[d] = __fadd_rn(W.base[d], W.delta[d]);
            __syncwarp();
        }
        pair_sync(bar_id);  // D: the pair's shared words are read before the next segment writes them
    }
    if (half == 0 && lane == 0) {
        P.valid[e] = (first == 0 && !too_many) ? 1 : 0;
        P.first_hit[e] = too_many ? -2 : (first ? first : -1);
        if (P.n_seg_out) P.n_seg_out[e] = nseg;
    }
    __syncwarp();
}

template <int A>
__global__ void __launch_bounds__(32 * kWarpsPerBlock, MRPOP_MIN_BLOCKS)
    pair_kernel(const __grid_constant__ EdgeParams P) {
    MRPOP_KERNEL_PROLOGUE(WarpScratch)
    static_assert(kWarpsPerBlock % 2 == 0, "warps come in pairs");
    __shared__ PairShare X[kWarpsPerBlock / 2];
    const int pair = warp >> 1, half = warp & 1;
    (void)nwarps;
    for (long long e = (long long)blockIdx.x * (kWarpsPerBlock / 2) + pair; e < P.n_edges;
         e += (long long)gridDim.x * (kWarpsPerBlock / 2))
        fused_edge_pair<A>(P, W, S, L, det_tab, e, dof, g, lane, half, X[pair], 1 + pair, staged);
}

// ---------------------------------------------------------------------------
// fused kernel, one warp per arm (small calls of 3 to 5 arms): a CTA of A
// warps takes one edge at a time and warp a does arm a's share of it -- its
// forward kinematics, env and intra-arm screens and exact tests, its detailed
// chain walk -- over every slot of the segment; the arm pairs of the arm-vs-arm
// screens and tests go to whichever warp is free.  Flag words are ORed together in
// shared memory, the thread split is evaluated from them by every warp (the
// same integers), and a sample collides when any warp's tests fire: the
// verdicts are those of the one-warp kernels.  The lower arm's spheres of a
// pair are read from the warp that placed them instead of being placed again.
// ---------------------------------------------------------------------------
// G = 2 (64 samples per segment, calls so small that the SMs have room): two
// warps per arm, each one 32-sample slot of it; a slot's arm pairs are shared by
// the slot's warps.
template <int A, int SPL, int G>
__device__ __forceinline__ void armwise_edge(const EdgeParams &P, unsigned char *wbase, const float4 *S,
                                             const SceneLayout &L, const float4 *det_tab, long long e, int dof,
                                             int g, int lane, int warp, ArmShare &X, bool staged) {
    ArmScratch &W = reinterpret_cast<ArmScratch *>(wbase)[warp];
    const int arm = G > 1 && warp >= A ? warp - A : warp, grp = G > 1 && warp >= A ? 1 : 0;
    static_assert(G == 1 || SPL == 2, "a warp per slot");
    constexpr bool by_slot = G > 1;
    const int s0 = by_slot ? grp : 0, s1 = by_slot ? grp + 1 : SPL;  // this warp's slots
    if (!staged) {
        if (warp == 0 && lane == 0) {
            P.valid[e] = 0;
            P.first_hit[e] = -2;
        }
        return;
    }
    bool too_many;
    const int nseg = edge_setup(P, W, e, dof, g, lane, too_many);
    const int nseg_run = too_many ? 0 : nseg;
    const bool do_env = P.flags & kEnvBit, do_self = P.flags & kSelfBit;
    int first = 0;
    for (int seg = 0; seg < nseg_run && first == 0; seg++) {
        if (warp == 0) {
#pragma unroll
            for (int t = 0; t < 2; t++) X.env[t][lane] = X.self[t][lane] = 0;
            if (lane < 2) X.hits[lane] = 0;
            if (lane < 3) X.next[lane] = 0;
        }
        __syncthreads();
        // this arm: placement, swept bounds, env and intra-arm screens (the
        // slots' spheres stay in arm.sp for the pair tests)
#pragma unroll 1
        for (int s = s0; s < s1; s++) {
            const int k = lane + 1 + 32 * s;
            auto &sp = W.arm.sp[s];
            float4 *sw = W.arm.swept[s];
            float q[7];
            sample_q(W, P.rule, seg, P.single ? 0 : arm, k <= g ? k : g, q);
            ArmSpheres as;
            fk_approx_arm(P.base[arm], q, as);
            store_swept(as, sp, lane, sw, P.cull);
            const bool reg = regular_pose(q);
            const bool regular = __all_sync(kFull, reg) && (P.rigid >> arm & 1);
            uint32_t em = 0, im = 0;
            if (do_env) em = env_joints<false>(S, L, P.sc, sp, lane, sw);
            if (do_self) im = intra_flags(sp, sw, lane, regular);
            if (k <= g) {
                if (em) atomicOr(&X.env[s][lane], (unsigned long long)em << (8 * arm));
                if (im) atomicOr(&X.self[s][lane], (unsigned long long)im << (8 * arm));
            }
        }
        __syncthreads();
        // arm pairs (a, b), a < b, handed out one at a time to the warps as
        // they finish (their costs differ): flags go to arm a
        // (panda_four.cuh:178-214); screened by the slot's swept bounds
        if (A > 1 && do_self) {
            const ArmScratch *Wa = reinterpret_cast<const ArmScratch *>(wbase);
#pragma unroll 1
            for (int t = take_pair(&X.next[0], lane); t < num_pairs(A) * (by_slot ? 2 : 1);
                 t = take_pair(&X.next[0], lane)) {
                const int p = by_slot && t >= num_pairs(A) ? t - num_pairs(A) : t;
                const int p0 = by_slot && t >= num_pairs(A) ? 1 : 0, p1 = by_slot ? p0 + 1 : SPL;  // slots
                int a, b;
                pair_arms<A>(p, a, b);
#pragma unroll 1
                for (int s = p0; s < p1; s++) {
                    const int k = lane + 1 + 32 * s;
                    const ArmScratch &Wl = Wa[(by_slot ? A * s : 0) + a], &Wu = Wa[(by_slot ? A * s : 0) + b];
                    const float4 *swa = Wl.arm.swept[s], *swb = Wu.arm.swept[s];
                    uint32_t bal[4];
#pragma unroll
                    for (int r = 0; r < 4; r++) {
                        const int t = 32 * r + lane;
                        const int i = t / kNumApprox, j = t - kNumApprox * i;
                        bal[r] = __ballot_sync(kFull, t < kNumApprox * kNumApprox &&
                                                          near3(swa[i].x, swa[i].y, swa[i].z, swb[j], swa[i].w));
                    }
                    if (!(bal[0] | bal[1] | bal[2] | bal[3])) {
                        if (lane == 0) X.pm[s][p] = 0;
                        continue;
                    }
                    const auto &low = Wl.arm.sp[s];
                    const auto &cur = Wu.arm.sp[s];
                    uint32_t am = 0, ja = 0, jb = 0;
#pragma unroll
                    for (int r = 0; r < 4; r++) {
                        uint32_t q = bal[r];
                        while (q) {
                            const int t = 32 * r + __ffs(q) - 1;
                            q &= q - 1;
                            const int i = t / kNumApprox, j = t - kNumApprox * i;
                            ja |= 1u << approx_joint(i);
                            jb |= 1u << approx_joint(j);
                            if (hit_sphere_sphere(low[i][0][lane], low[i][1][lane], low[i][2][lane],
                                                  c_approx[i].w, cur[j][0][lane], cur[j][1][lane],
                                                  cur[j][2][lane], c_approx[j].w))
                                am |= 1u << approx_joint(i);
                        }
                    }
                    if (am && k <= g) atomicOr(&X.self[s][lane], (unsigned long long)am << (8 * a));
                    if (lane == 0) X.pm[s][p] = ja | jb << 8;
                }
            }
        }
        __syncthreads();
        // the thread split, from the ORed words (every warp alike)
        Flags<A> envw[SPL], selfw[SPL];
        int envc[SPL], selfc[SPL], tot_env = 0, tot_self = 0;
#pragma unroll
        for (int s = 0; s < SPL; s++) {
            envw[s] = (Flags<A>)X.env[s][lane];
            selfw[s] = (Flags<A>)X.self[s][lane];
            envc[s] = flag_count<A>(envw[s]);
            selfc[s] = flag_count<A>(selfw[s]);
            tot_env += envc[s];
            tot_self += selfc[s];
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            tot_env += __shfl_xor_sync(kFull, tot_env, o);
            tot_self += __shfl_xor_sync(kFull, tot_self, o);
        }
        if (tot_env > 0 || tot_self > 0) {
            uint64_t cand_env = 0, cand_self = 0;
            thread_split<SPL>((P.flags & kExactBit) != 0, g, lane, envc, selfc, tot_env, tot_self, cand_env,
                              cand_self);
#pragma unroll 1
            for (int s = s0; s < s1; s++) {
                // a hit that some warp found in an earlier slot settles the
                // edge.  Other warps write the word meanwhile, so the branch
                // takes lane 0's reading for the whole warp
                if (s > 0 && __shfl_sync(kFull, *(const volatile unsigned int *)&X.hits[0], 0)) break;
                const int bit = lane + 32 * s;
                const bool dE = cand_env >> bit & 1ull, dS = cand_self >> bit & 1ull;
                const Flags<A> ew = s == 0 ? envw[0] : envw[SPL - 1], sw = s == 0 ? selfw[0] : selfw[SPL - 1];
                narrow_slot<A, true>(P, W, S, L, det_tab, seg, 32 * s, ew, sw, dE, dS, 0u, arm, &X, s);
            }
            __syncthreads();
            const uint64_t hits = (uint64_t)X.hits[0] | (SPL > 1 ? (uint64_t)X.hits[1] << 32 : 0ull);
            if (hits) first = seg * g + __ffsll((long long)hits);
        }
        if (P.rule == kRuleConnect) {
            __syncwarp();
            for (int d = lane; d < dof; d += 32) W.base[d] = __fadd_rn(W.base[d], W.delta[d]);
            __syncwarp();
        }
        __syncthreads();  // the shared words are read before the next segment clears them
    }
    if (warp == 0 && lane == 0) {
        P.valid[e] = (first == 0 && !too_many) ? 1 : 0;
        P.first_hit[e] = too_many ? -2 : (first ? first : -1);
        if (P.n_seg_out) P.n_seg_out[e] = nseg;
    }
}

// CTAs of the arm-per-warp kernels that fit an SM (228 KB) by their warps' scratch,
// 3 KB of static shared memory and the 1 KB that the system takes of each, beside
// a scene of some boxes.  Given as a launch bound because ptxas, left to choose,
// cuts 5 arms at 64 samples to 72 registers and spills.
__host__ __device__ constexpr int armwise_min_blocks(int A, int G = 1) {
    return (int)(228 * 1024 / (A * G * sizeof(ArmScratch) + 4096));
}
static_assert(armwise_min_blocks(3) == 5 && armwise_min_blocks(4) == 4 && armwise_min_blocks(5) == 3 &&
                  armwise_min_blocks(3, 2) == 3 && armwise_min_blocks(4, 2) == 2 && armwise_min_blocks(5, 2) == 1,
              "CTAs per SM");

template <int A, int SPL, int G>
__global__ void __launch_bounds__(32 * A * G, armwise_min_blocks(A, G))
    armwise_kernel(const __grid_constant__ EdgeParams P) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t bar;
    __shared__ float4 det_tab[kNumDet];
    __shared__ ArmShare X;
    const SceneLayout L = scene_layout(P.sc);
    const float4 *S = reinterpret_cast<const float4 *>(smem_raw);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int i = threadIdx.x; i < kNumDet; i += blockDim.x) det_tab[i] = c_det[i];
    const bool staged = stage_scene(reinterpret_cast<float4 *>(smem_raw), P.scene,
                                    (uint32_t)(L.total * sizeof(float4)), &bar, P.status);
    unsigned char *wbase = smem_raw + (size_t)L.total * sizeof(float4);
    const int dof = 7 * (P.single ? 1 : A);
    for (long long e = blockIdx.x; e < P.n_edges; e += gridDim.x)
        armwise_edge<A, SPL, G>(P, wbase, S, L, det_tab, e, dof, P.g, lane, warp, X, staged);
}

// ---------------------------------------------------------------------------
// split pipeline for single-segment edges: the broad kernel writes every
// sample's flag words, each edge's candidate masks and the joints that swept
// bounds connect per arm pair to HBM (P.sflags, P.smasks, P.spairs); the narrow
// kernel runs the detailed phase of edges with candidates.  Each kernel's code fits the
// instruction cache on its own.  broad_edge / narrow_edge are one warp's work
// on edge e, shared by the plain kernels and the batch kernels.
// ---------------------------------------------------------------------------
// Staged flag words of sample slot o (= edge * 32 * SPL + sample - 1): 8 flag
// bits per arm, so 32-bit words hold up to 4 arms.
template <int A>
__device__ __forceinline__ void store_flags(const EdgeParams &P, long long o, Flags<A> env, Flags<A> self) {
    if (A <= 4) reinterpret_cast<uint2 *>(P.sflags)[o] = make_uint2((uint32_t)env, (uint32_t)self);
    else reinterpret_cast<ulonglong2 *>(P.sflags)[o] = make_ulonglong2(env, self);
}
template <int A>
__device__ __forceinline__ void load_flags(const EdgeParams &P, long long o, Flags<A> &env, Flags<A> &self) {
    if (A <= 4) {
        const uint2 v = reinterpret_cast<const uint2 *>(P.sflags)[o];
        env = v.x;
        self = v.y;
    } else {
        const ulonglong2 v = reinterpret_cast<const ulonglong2 *>(P.sflags)[o];
        env = v.x;
        self = v.y;
    }
}

template <int A, int SPL, bool SEG>
__device__ __forceinline__ void broad_edge(const EdgeParams &P, BroadScratch &W, const float4 *S, const SceneLayout &L,
                                           long long e, int dof, int g, int lane, bool staged) {
    if (!staged) {
        if (lane == 0) {
            P.valid[e] = 0;
            P.first_hit[e] = -2;
            P.smasks[2 * e] = P.smasks[2 * e + 1] = 0;
        }
        return;
    }
    // SEG: a segment round of a segmented rule (r = P.seg0); otherwise a
    // single-segment edge (r = 0, compiled as a constant)
    const int r = SEG ? P.seg0 : 0;
    constexpr bool segmented = SEG;
    if (segmented && r > 0 && (P.sdone[e] || P.snseg[e] <= r)) {
        if (lane == 0) P.smasks[2 * e] = P.smasks[2 * e + 1] = 0;
        return;
    }
    bool too_many;
    const int nseg = edge_setup(P, W, e, dof, g, lane, too_many);
    if (segmented) {
        if (r == 0) {
            const bool none = too_many || nseg <= 0; // decided without a check
            if (lane == 0) {
                P.snseg[e] = too_many ? -1 : nseg;
                if (P.n_seg_out) P.n_seg_out[e] = nseg;
                P.sdone[e] = none ? 1 : 0;
                if (none) {
                    P.valid[e] = too_many ? 0 : 1;
                    P.first_hit[e] = too_many ? -2 : -1;
                    P.smasks[2 * e] = P.smasks[2 * e + 1] = 0;
                    if (P.flops) P.flops[e] = 0.0;
                }
            }
            if (none) {
                __syncwarp();
                return;
            }
        } else if (P.rule == kRuleConnect) {
            connect_advance(W, dof, r, lane);
        }
    } else {
        (void)nseg;
    }
    Flags<A> envw[SPL], selfw[SPL];
    uint64_t cand_env, cand_self;
    uint32_t pm[SPL];
    const bool any = broad_decide<A, SPL>(P, W, W.broad, S, L, r, g, lane, envw, selfw, pm, cand_env, cand_self, e,
                                          !segmented || r == 0);
    if (any) {
#pragma unroll
        for (int s = 0; s < SPL; s++) {
            store_flags<A>(P, e * (32 * SPL) + lane + 32 * s, envw[s], selfw[s]);
            if (lane < num_pairs(A)) P.spairs[(e * SPL + s) * num_pairs(A) + lane] = (uint16_t)pm[s];
        }
    }
    if (lane == 0) {
        P.smasks[2 * e] = cand_env;
        P.smasks[2 * e + 1] = cand_self;
        if (!any && (!segmented || r == nseg - 1)) { // the last segment passed the broad phase
            P.valid[e] = 1;
            P.first_hit[e] = -1;
            if (segmented) P.sdone[e] = 1;
        }
        if (!segmented && P.n_seg_out) P.n_seg_out[e] = 1;
    }
    __syncwarp();
}

// The detailed phase of edge e.  One arm, and composite calls of a middle size:
// all of it (kStageAll), in one kernel.  Larger composite calls: the obstacles and
// arm pairs (STAGE kStageEnvPairs, narrow_kernel), then the intra-arm rows (kStageRows, rows_kernel) of the samples below the
// first hit; between the two P.smasks[2 * e] says whether a sample has hit and
// P.smasks[2 * e + 1] which samples are left.
template <int A, int SPL, bool SEG, int STAGE>
__device__ __forceinline__ void narrow_edge(const EdgeParams &P, WarpScratch &W, const float4 *S, const SceneLayout &L,
                                            const float4 *det_tab, long long e, int dof, int g, int lane,
                                            bool staged) {
    constexpr bool first_stage = STAGE == kStageEnvPairs, rows = STAGE == kStageRows;
    const uint64_t m0 = P.smasks[2 * e], cand_self = P.smasks[2 * e + 1];
    const uint64_t cand_env = rows ? 0ull : m0;
    if (!(cand_env | cand_self)) return; // verdict written by an earlier kernel
    if (!staged) {
        if (lane == 0) {
            P.valid[e] = 0;
            P.first_hit[e] = -2;
            if (first_stage) P.smasks[2 * e] = P.smasks[2 * e + 1] = 0;
        }
        return;
    }
    Flags<A> envw[SPL], selfw[SPL];
    uint32_t pm[SPL];
    uint32_t any_pair = 0;
#pragma unroll
    for (int s = 0; s < SPL; s++) {
        pm[s] = !rows && lane < num_pairs(A) ? P.spairs[(e * SPL + s) * num_pairs(A) + lane] : 0u;
        any_pair |= pm[s];
    }
    if (first_stage && !cand_env && !__any_sync(kFull, any_pair)) return; // rows alone
    // (loaded before the set-up waits for the endpoints, so that both are under way)
#pragma unroll
    for (int s = 0; s < SPL; s++) load_flags<A>(P, e * (32 * SPL) + lane + 32 * s, envw[s], selfw[s]);
    const int r = SEG ? P.seg0 : 0;
    constexpr bool segmented = SEG;
    bool too_many;
    const int nseg = edge_setup(P, W, e, dof, g, lane, too_many);
    if (SEG && P.rule == kRuleConnect && r > 0) connect_advance(W, dof, r, lane);
    const int fb =
        narrow_segment<A, SPL, STAGE>(P, W, S, L, det_tab, r, lane, envw, selfw, pm, cand_env, cand_self);
    if (lane == 0) {
        const uint64_t left = first_stage ? (fb < 64 ? cand_self & ((1ull << fb) - 1ull) : cand_self) : 0ull;
        if (first_stage) {
            P.smasks[2 * e] = fb < 64 ? 1ull : 0ull;
            P.smasks[2 * e + 1] = left;
        }
        if (fb < 64) {
            P.valid[e] = 0;
            P.first_hit[e] = r * g + fb + 1;
            if (segmented) P.sdone[e] = 1;
        } else if (left == 0 && !(rows && m0) && (!segmented || r == nseg - 1)) {
            P.valid[e] = 1;
            P.first_hit[e] = -1;
            if (segmented) P.sdone[e] = 1;
        }
    }
    __syncwarp();
}

// Next edge for this warp: a shared counter handed out one edge at a time, so
// that warps whose edges finish early take more (edge costs vary by orders of
// magnitude: an edge without candidates skips the narrow phase entirely).
__device__ __forceinline__ long long next_edge(unsigned long long *counter, int lane) {
    unsigned long long e = 0;
    if (lane == 0) e = atomicAdd(counter, 1ull);
    return (long long)__shfl_sync(kFull, e, 0);
}

template <int A, int SPL, bool SEG>
__global__ void __launch_bounds__(32 * kWarpsPerBlock, kBroadMinBlocks)
    broad_kernel(const __grid_constant__ EdgeParams P) {
    MRPOP_KERNEL_PROLOGUE(BroadScratch)
    (void)nwarps;
    for (long long e = next_edge(P.work, lane); e < P.n_edges; e = next_edge(P.work, lane))
        broad_edge<A, SPL, SEG>(P, W, S, L, e, dof, g, lane, staged);
    // no edges left for this warp: the narrow kernel (launched as a
    // programmatic dependent) may start its CTAs once every CTA got here
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <int A, int SPL, bool SEG, int STAGE>
__global__ void __launch_bounds__(32 * kWarpsPerBlock, MRPOP_MIN_BLOCKS)
    narrow_kernel(const __grid_constant__ EdgeParams P) {
    MRPOP_KERNEL_PROLOGUE(WarpScratch)
    (void)nwarps;
    // the scene is staged; wait for the broad kernel (complete, its writes
    // visible) before reading its output
    asm volatile("griddepcontrol.wait;" ::: "memory");
    for (long long e = next_edge(P.work + 1, lane); e < P.n_edges; e = next_edge(P.work + 1, lane))
        narrow_edge<A, SPL, SEG, STAGE>(P, W, S, L, det_tab, e, dof, g, lane, staged);
    if (STAGE == kStageEnvPairs) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");  // the rows kernel
}

// Composite checks: the intra-arm rows, after the narrow kernel.
template <int A, int SPL, bool SEG>
__global__ void __launch_bounds__(32 * kWarpsPerBlock, MRPOP_MIN_BLOCKS)
    rows_kernel(const __grid_constant__ EdgeParams P) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ float4 det_tab[kNumDet];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    WarpScratch &W = reinterpret_cast<WarpScratch *>(smem_raw)[warp];  // no scene
    for (int i = threadIdx.x; i < kNumDet; i += blockDim.x) det_tab[i] = c_det[i];
    __syncthreads();
    const SceneLayout L{};
    asm volatile("griddepcontrol.wait;" ::: "memory");
    for (long long e = next_edge(P.work + 2, lane); e < P.n_edges; e = next_edge(P.work + 2, lane))
        narrow_edge<A, SPL, SEG, kStageRows>(P, W, nullptr, L, det_tab, e, 7 * A, P.g, lane, true);
}

// ---------------------------------------------------------------------------
// batch kernels: many independent instances (each with its own scene, arm
// layout, edges, granularity and outputs; one EdgeParams each, all of arm
// count A and samples-per-lane SPL) in one persistent launch.  An instance's
// edges form chunks; CTAs take chunks from a counter, in instance order, and
// copy the instance's parameters to shared memory and restage its scene with
// the bulk-copy engine when the instance changes; the CTA's warps then take
// the chunk's edges one at a time.  MODE picks the broad, narrow or fused
// per-edge body; SEG marks groups of segmented instances (connect, B-spline,
// shortcut), which run the split kernels in rounds (BatchParams::seg0) and
// the fused kernel for the edges left after them.
// ---------------------------------------------------------------------------
struct BatchParams {
    const EdgeParams *items;      // device array, one per instance
    const int4 *chunks;           // {instance, first edge, edge count, -}, instances in order
    int n_chunks;
    int seg0;                     // segmented groups: the round (split kernels) or first segment (fused)
    unsigned long long *work;     // next-chunk counter, zero before each launch
};

// Batch kernel modes: the split pipeline's two kernels, and the fused kernel
// that finishes segmented edges after the split rounds.
constexpr int kBatchBroad = 0, kBatchNarrow = 1, kBatchFused = 2;
// Batch mode of the arm-per-warp kernel (whole edges from segment 0, a CTA of
// A warps per edge): batch_armwise_kernel.
constexpr int kBatchArmwise = 3;
// The rows kernel of composite groups, after kBatchNarrow.
constexpr int kBatchRows = 4;
// kBatchNarrow and kBatchRows in one kernel (service waves).
constexpr int kBatchNarrowAll = 5;

// CTAs per SM of the batch kernels.  The fused composite ones, whose groups are
// small (a wave's, or the edges that segment rounds leave), are built for 2: at 3,
// their 96 registers spill 112 bytes at 64 samples.  Whole wave of fused steps, 3
// against 2: 2 arms x 64 connect, 300 edges 192 -> 169 us on the device, 3000 351
// -> 309; 3 arms x 64 connect, 3000 edges 471 -> 401; one arm, which does not
// spill, 4000 x 64 79 -> 101.
constexpr int batch_min_blocks(int arms, int mode) {
    return mode == kBatchBroad ? kBroadMinBlocks : mode == kBatchFused && arms > 1 ? 2 : MRPOP_MIN_BLOCKS;
}

// One bulk copy of `bytes` from global to shared memory, completed on `bar`
// in phase `parity`; bounded wait.  Every thread of the CTA calls it after a
// barrier that follows its last read of `dst`; the proxy fence orders those
// reads before the copy's writes.  Returns false (for the whole CTA) if the
// copy did not complete in time.
__device__ __forceinline__ bool stage_bulk(float4 *dst, const float4 *src, uint32_t bytes, uint64_t *bar,
                                           uint32_t parity, unsigned int *status) {
    if (threadIdx.x == 0) {
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                     : "memory");
        asm volatile(
            "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                smem_u32(dst)),
            "l"(src), "r"(bytes), "r"(smem_u32(bar))
            : "memory");
    }
    return __syncthreads_and(copy_wait(bar, parity, status, kWaitLimitNs));
}

template <int A, int SPL, int MODE, bool SEG>
__global__ void __launch_bounds__(32 * kWarpsPerBlock, batch_min_blocks(A, MODE))
    batch_kernel(const __grid_constant__ BatchParams B) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t bar;
    __shared__ float4 det_tab[kNumDet];
    __shared__ __align__(16) EdgeParams Ps;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int i = threadIdx.x; i < kNumDet; i += blockDim.x) det_tab[i] = c_det[i];
    if (threadIdx.x == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&bar)));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    __shared__ int s_chunk;
    __shared__ unsigned int s_next;
    int item = -1;
    uint32_t parity = 0;
    bool staged = false;
    for (;;) {
        // the CTA takes the next chunk of one instance's edges ...
        if (threadIdx.x == 0) {
            s_chunk = (int)atomicAdd(B.work, 1ull);
            s_next = 0;
        }
        __syncthreads();
        const int c = s_chunk;
        if (c >= B.n_chunks) break;
        const int4 ch = B.chunks[c];
        if (ch.x != item) {
            const uint32_t *src = reinterpret_cast<const uint32_t *>(B.items + ch.x);
            uint32_t *dst = reinterpret_cast<uint32_t *>(&Ps);
            for (int i = threadIdx.x; i < (int)(sizeof(EdgeParams) / 4); i += blockDim.x) dst[i] = src[i];
            __syncthreads();
            if (SEG) { // the round of this launch
                if (threadIdx.x == 0) Ps.seg0 = B.seg0;
                __syncthreads();
            }
            const uint32_t bytes = (uint32_t)(scene_layout(Ps.sc).total * sizeof(float4));
            staged = true;
            if (bytes && MODE != kBatchRows) {
                staged = stage_bulk(reinterpret_cast<float4 *>(smem_raw), Ps.scene, bytes, &bar, parity, Ps.status);
                parity ^= 1u;
            }
            item = ch.x;
        }
        const EdgeParams &P = Ps;
        const SceneLayout L = scene_layout(P.sc);
        const float4 *S = reinterpret_cast<const float4 *>(smem_raw);
        using Scratch = std::conditional_t<MODE == kBatchBroad, BroadScratch, WarpScratch>;
        Scratch &W = reinterpret_cast<Scratch *>(smem_raw + (size_t)L.total * sizeof(float4))[warp];
        const int dof = 7 * (P.single ? 1 : A);
        // ... and its warps take the chunk's edges one at a time
        for (;;) {
            unsigned int k = 0;
            if (lane == 0) k = atomicAdd(&s_next, 1u);
            k = __shfl_sync(kFull, k, 0);
            if ((int)k >= ch.z) break;
            const long long e = (long long)ch.y + k;
            if constexpr (MODE == kBatchBroad) broad_edge<A, SPL, SEG>(P, W, S, L, e, dof, P.g, lane, staged);
            else if constexpr (MODE == kBatchNarrow || MODE == kBatchNarrowAll)
                narrow_edge<A, SPL, SEG, A == 1 || MODE == kBatchNarrowAll ? kStageAll : kStageEnvPairs>(
                    P, W, S, L, det_tab, e, dof, P.g, lane, staged);
            else if constexpr (MODE == kBatchRows)
                narrow_edge<A, SPL, SEG, kStageRows>(P, W, S, L, det_tab, e, dof, P.g, lane, staged);
            else fused_edge<A, SPL>(P, W, S, L, det_tab, e, dof, P.g, lane, staged);
        }
        __syncthreads(); // every warp is done with this chunk (and instance)
    }
}

// Batch form of armwise_kernel: the CTA takes chunks (of single edges) from the
// launch's counter, stages each instance's parameters and scene as
// batch_kernel does, and runs the arm-per-warp body on every edge of the chunk.
template <int A, int SPL>
__global__ void __launch_bounds__(32 * A, armwise_min_blocks(A))
    batch_armwise_kernel(const __grid_constant__ BatchParams B) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t bar;
    __shared__ float4 det_tab[kNumDet];
    __shared__ __align__(16) EdgeParams Ps;
    __shared__ ArmShare X;
    __shared__ int s_chunk;
    const int arm = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int i = threadIdx.x; i < kNumDet; i += blockDim.x) det_tab[i] = c_det[i];
    if (threadIdx.x == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&bar)));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    int item = -1;
    uint32_t parity = 0;
    bool staged = false;
    for (;;) {
        if (threadIdx.x == 0) s_chunk = (int)atomicAdd(B.work, 1ull);
        __syncthreads();
        const int c = s_chunk;
        if (c >= B.n_chunks) break;
        const int4 ch = B.chunks[c];
        if (ch.x != item) {
            const uint32_t *src = reinterpret_cast<const uint32_t *>(B.items + ch.x);
            uint32_t *dst = reinterpret_cast<uint32_t *>(&Ps);
            for (int i = threadIdx.x; i < (int)(sizeof(EdgeParams) / 4); i += blockDim.x) dst[i] = src[i];
            __syncthreads();
            const uint32_t bytes = (uint32_t)(scene_layout(Ps.sc).total * sizeof(float4));
            staged = true;
            if (bytes) {
                staged = stage_bulk(reinterpret_cast<float4 *>(smem_raw), Ps.scene, bytes, &bar, parity, Ps.status);
                parity ^= 1u;
            }
            item = ch.x;
        }
        const SceneLayout L = scene_layout(Ps.sc);
        const float4 *S = reinterpret_cast<const float4 *>(smem_raw);
        unsigned char *wbase = smem_raw + (size_t)L.total * sizeof(float4);
        const int dof = 7 * (Ps.single ? 1 : A);
        for (int k = 0; k < ch.z; k++)
            armwise_edge<A, SPL, 1>(Ps, wbase, S, L, det_tab, (long long)ch.y + k, dof, Ps.g, lane, arm, X, staged);
        __syncthreads();  // every warp is done with this chunk (and instance)
    }
}

}  // namespace mrpop
