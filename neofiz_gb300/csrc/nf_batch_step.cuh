// nf_batch_step.cuh -- one step of one batched instance by a block or a cluster of them, shared by the
// batched kernel (k_batch.cu) and the adjoint kernels (k_adjoint.cu).
#pragma once

#include "nf_bodies.cuh"

#include <cooperative_groups.h>

namespace nf {

// The blocks that step one instance together: one block, or (TEAM) a thread-block cluster, for
// batches with fewer instances than SMs. Warps are dealt round-robin over the blocks, so an
// instance with few warps of elements spreads over every block's quarter SMs; a cluster barrier
// orders global memory and the blocks' shared memory as a block barrier does within a block.
template <bool TEAM>
struct Team {
    int rank, size;
    __device__ __forceinline__ Team() {
        if (TEAM) {
            const auto c = cooperative_groups::this_cluster();
            rank = (int)c.block_rank();
            size = (int)c.num_blocks();
        } else {
            rank = 0;
            size = 1;
        }
    }
    // this thread's place among the team's threads, of which each block has T
    __device__ __forceinline__ int tid() const {
        return TEAM ? (((int)threadIdx.x >> 5) * size + rank) * 32 + ((int)threadIdx.x & 31)
                    : (int)threadIdx.x;
    }
    __device__ __forceinline__ bool first() const { return threadIdx.x == 0 && rank == 0; }
    __device__ __forceinline__ void sync() const {
        if (TEAM) cooperative_groups::this_cluster().sync();
        else __syncthreads();
    }
    // block r's copy of a shared variable
    template <typename V>
    __device__ __forceinline__ V *at(V *p, int r) const {
        return TEAM ? cooperative_groups::this_cluster().map_shared_rank(p, r) : p;
    }
};
constexpr int TEAM_MAX = 8;                  // blocks of a team (the portable cluster size)

__device__ __forceinline__ unsigned long long bbits(double x) {
    return (unsigned long long)__double_as_longlong(x);
}
__device__ __forceinline__ double bdouble(unsigned long long u) {
    return __longlong_as_double((long long)u);
}

// Exact block minimum of the per-thread shortest squared edges, returned to every thread. The
// warps combine with jmin and the warps' results by the integer order of their bits, as the
// single-scene kernels do with shuffles and atomicMin.
template <int T>
__device__ double block_min_edge(double v, double *sh) {
    for (int o = 16; o > 0; o >>= 1) v = jmin(v, __shfl_down_sync(0xffffffffu, v, o));
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) sh[warp] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long m = bbits(sh[0]);
        for (int w = 1; w < T / 32; w++) m = min(m, bbits(sh[w]));
        sh[T / 32] = bdouble(m);
    }
    __syncthreads();
    return sh[T / 32];
}

template <int T>
__device__ double block_min_edge_f(float v, double *sh) {
    for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_down_sync(0xffffffffu, v, o));
    return block_min_edge<T>((double)v, sh);
}

// Sums over an instance's items (nodes, elements, pressure edges) that do not depend on how many
// blocks step it, and so not on its neighbours in the batch. The items are dealt to 8 T lanes,
// T of them a block of the widest team: item j adds to lane j mod 8 T, item after item. A team
// of fewer blocks gives each thread several lanes, one per slot: those of its first, second ...
// item. Lanes add up by warps and the warps by one tree. Blocks of another width T deal the same
// way while there are no more than 8 T items.
template <bool TEAM>
constexpr int SUM_SLOTS = TEAM ? TEAM_MAX / 2 : TEAM_MAX;
template <bool TEAM>
__device__ __forceinline__ int next_slot(const Team<TEAM> &team, int slot) {
    return (slot + 1) & (TEAM_MAX / team.size - 1);
}
__device__ __forceinline__ double warp_sum(double v) {
    // lanes of +0 alone add up to +0: the common case of sums that few items add to
    if (!__any_sync(0xffffffffu, __double_as_longlong(v) != 0)) return v;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}
// The tree over the warps' sums: `used` rows of the table, the others zero; valid in the calling
// warp's first lane.
template <int COUNT>
__device__ __forceinline__ void table_sums(const double (*table)[COUNT], int used,
                                           double (&out)[COUNT]) {
    const int lane = threadIdx.x & 31;
    for (int i = 0; i < COUNT; i++) {
        const double low = lane < used ? table[lane][i] : 0.0;
        const double high = lane + 32 < used ? table[lane + 32][i] : 0.0;
        out[i] = warp_sum(low + high);
    }
}
// COUNT sums of `items` items at most from the threads' slots, in out[] of every block's thread 0.
// `table` has a row per warp of the widest team, block-shared; a team barrier separates one use
// of it from the next.
template <bool TEAM, int T, int COUNT>
__device__ __forceinline__ void team_sums(const Team<TEAM> &team, int items,
                                          const double (*part)[COUNT], double (*table)[COUNT],
                                          double (&out)[COUNT]) {
    const int warps = T / 32 * team.size, lane = threadIdx.x & 31, warp = team.tid() >> 5;
    int slots = (items + 32 * warps - 1) / (32 * warps);
    if (slots > TEAM_MAX / team.size) slots = TEAM_MAX / team.size;
    for (int s = 0; s < slots; s++)
        for (int i = 0; i < COUNT; i++) {
            const double v = warp_sum(part[s][i]);
            if (lane == 0)
                for (int r = 0; r < team.size; r++) team.at(table, r)[s * warps + warp][i] = v;
        }
    team.sync();
    if (threadIdx.x < 32) table_sums<COUNT>(table, slots * warps, out);
}

// The wall's impulse, energy loss and friction work go to the same lanes. One-warp blocks keep a
// single sum a lane, in registers: they run instances of a few dozen nodes, none of whose lanes
// have two at the wall, and they wait for instructions (2.8 of the 7 cycles between two), so that
// eight slots cost them 3 % (512 burst slices: 87.3 ms, 89.9 with the slots).
template <bool TEAM, int T>
constexpr int WALL_SLOTS = T == 32 ? 1 : SUM_SLOTS<TEAM>;
// Their totals over a chunk of steps, the warps added in turn, in out[] of the first block's first
// thread. Out of line, once a chunk; the team by value, so that the caller's stays in registers.
// sh: a row of T / 32; table: a row per warp of the widest team, used by teams alone, so that
// the staged kernels' shared memory stays the nodes'.
template <bool TEAM, int T>
static __device__ __noinline__ void wall_totals(const Team<TEAM> team, int nodes,
                                                const double (*part)[3], double *sh,
                                                double (*table)[3], double (&out)[3]) {
    const int warps = T / 32 * team.size, lane = threadIdx.x & 31, warp = team.tid() >> 5;
    int slots = (nodes + 32 * warps - 1) / (32 * warps);
    if (slots > TEAM_MAX / team.size) slots = TEAM_MAX / team.size;
    out[0] = out[1] = out[2] = 0.0;
#pragma unroll 1
    for (int s = 0; s < slots; s++)
#pragma unroll 1
        for (int i = 0; i < 3; i++) {
            const double v = warp_sum(part[s][i]);
            if (TEAM) {
                if (lane == 0) team.at(table, 0)[s * warps + warp][i] = v;
            } else {
                __syncthreads();
                if (lane == 0) sh[warp] = v;
                __syncthreads();
                if (threadIdx.x == 0)
                    for (int w = 0; w < warps; w++) out[i] += sh[w];
            }
        }
    if (TEAM) {
        team.sync();
        if (team.rank == 0 && threadIdx.x < 32) {
            double sum = 0.0;
#pragma unroll 1
            for (int row = 0; lane < 3 && row < slots * warps; row++) sum += table[row][lane];
            __syncwarp();
            for (int i = 0; i < 3; i++) out[i] = __shfl_sync(0xffffffffu, sum, i);
        }
    }
}

// The coming step's size and nodal coefficients (:947-956, :985-990), computed once per block
// by thread 0 and read by every thread: the same formulas as each thread would evaluate, so
// the same bits, without every thread spending FP64 divisions and a square root on them.
struct BlockStep {
    double dt, decay, gain, dtAvg;
    float fdt, fdecay, fgain, fdtAvg;               // the same in FP32 (the FP32 forms)
    float plane, friction, gravR, gravZ, hourglass; // the instance's constants in FP32
};

__device__ __forceinline__ void block_step_coef(BlockStep &bs, const BatchInst &in, double dt,
                                                double dtPrev) {
    const double dtAvg = 0.5 * (dtPrev + dt);
    const double half = 0.5 * in.damping * dtAvg;
    bs.dt = dt;
    const nf_divisor by = nf_divisor_of(1.0 + half);
    bs.decay = nf_div_by(1.0 - half, 1.0 + half, by);
    bs.gain = nf_div_by(dtAvg, 1.0 + half, by);
    bs.dtAvg = dtAvg;
    bs.fdt = (float)bs.dt;
    bs.fdecay = (float)bs.decay;
    bs.fgain = (float)bs.gain;
    bs.fdtAvg = (float)bs.dtAvg;
}

// At the start of a chunk (thread 0): the coefficients and the FP32 constants.
__device__ __forceinline__ void block_step_init(BlockStep &bs, const Dev &d, const BatchInst &in,
                                                double dt, double dtPrev) {
    block_step_coef(bs, in, dt, dtPrev);
    bs.plane = (float)in.wallPlane;
    bs.friction = (float)in.wallFriction;
    bs.gravR = (float)d.gravR;
    bs.gravZ = (float)d.gravZ;
    bs.hourglass = (float)in.hourglass;
}

// Thread 0's part of a step's end: the minimum of `count` minima (exact, by the order of the
// bits), the CFL step (:985-990) and the next step's coefficients. Out of line: one thread runs
// it once a step, and its division and square root stay out of the registers of the element and
// node loops.
__device__ __forceinline__ double min_of(const double *v, int count) {
    unsigned long long m = bbits(v[0]);
    for (int w = 1; w < count; w++) m = min(m, bbits(v[w]));
    return bdouble(m);
}
static __device__ __noinline__ double block_step_advance(const double *v, int count, BlockStep *bs,
                                                         const BatchInst &in, double dt,
                                                         double dtPrev, int finite) {
    const double me = min_of(v, count);
    if (finite) block_step_coef(*bs, in, nf_div(in.cfl * nf_sqrt(me * in.massScale), in.wave), dt);
    else block_step_coef(*bs, in, dt, dtPrev);
    return me;
}

// The team's exact minimum of the warps' minima (each warp's in sh[warp]), returned to every
// thread, with each block's thread 0 preparing the next step in its bs between the barriers.
template <bool TEAM, int T>
__device__ __forceinline__ double team_min_tail(const Team<TEAM> &team, double *sh, BlockStep *bs,
                                                const BatchInst &in, double dt, double dtPrev,
                                                int finite) {
    __shared__ double ranks[TEAM_MAX];
    __syncthreads();
    if (TEAM) {
        if (threadIdx.x == 0) {
            const double mine = min_of(sh, T / 32);
            for (int r = 0; r < team.size; r++) team.at(ranks, r)[team.rank] = mine;
        }
        team.sync();
        if (threadIdx.x == 0)
            sh[T / 32] = block_step_advance(ranks, team.size, bs, in, dt, dtPrev, finite);
    } else if (threadIdx.x == 0) {
        sh[T / 32] = block_step_advance(sh, T / 32, bs, in, dt, dtPrev, finite);
    }
    __syncthreads();
    return sh[T / 32];
}

template <bool TEAM, int T>
__device__ double team_min_edge_next(const Team<TEAM> &team, double v, double *sh, BlockStep *bs,
                                     const BatchInst &in, double dt, double dtPrev, int finite) {
    for (int o = 16; o > 0; o >>= 1) v = jmin(v, __shfl_down_sync(0xffffffffu, v, o));
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    return team_min_tail<TEAM, T>(team, sh, bs, in, dt, dtPrev, finite);
}

// The same for FP32 edges: the warps reduce in FP32 (exact), lane 0 widens its minimum.
template <bool TEAM, int T>
__device__ double team_min_edge_next_f(const Team<TEAM> &team, float v, double *sh, BlockStep *bs,
                                       const BatchInst &in, double dt, double dtPrev, int finite) {
    for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_down_sync(0xffffffffu, v, o));
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = (double)v;
    return team_min_tail<TEAM, T>(team, sh, bs, in, dt, dtPrev, finite);
}

// One step of instance `in` by its team of blocks, ExplicitSolver.step :940-991: the nodal update
// (with the mixed form's float geometry when geo.pMid is set), the assembly with the exact
// shortest squared edge, the per-node gather, the next CFL step. dt, dtPrev, time and steps
// advance in place; returns the shortest squared edge. wall: the threads' slots (team_sums) of the
// wall's impulse, energy loss and friction work. COMP (with MIXED): the compensated form's
// FP32 nodal update and gather (nf_bodies.cuh). INT: batch_int_products. The step's coefficients and
// the next step size come from bs, which each block's thread 0 keeps prepared.
template <bool MIXED, int T, bool COMP, bool INT, bool TEAM>
__device__ __forceinline__ double batch_step(const Team<TEAM> &team, const Dev &d,
                                             const BatchInst &in, double &dt, double &dtPrev,
                                             double &time, long long &steps, const MixedGeo &geo,
                                             const float4 *pMid, const float2 *vdt, int base,
                                             uint32_t *status, int *wallContact, int *wallStuck,
                                             double (*wall)[3], double *shMin, BlockStep *bs) {
    static_assert(!COMP || MIXED, "the compensated form assembles in FP32");
    const NodalCoef co{bs->decay, bs->gain, bs->dtAvg, dt};
    const WallRef w{in.hasWall, in.wallPlane, in.wallFriction, wallContact, wallStuck};
    const int tid = team.tid(), stride = TEAM ? team.size * T : T;
    for (int i = in.n0 + tid, slot = 0; i < in.n1; i += stride, slot = next_slot(team, slot)) {
        double *const sum = wall[WALL_SLOTS<TEAM, T> == 1 ? 0 : slot];
        if (COMP)
            nodal_node_comp(d, i, bs->fdecay, bs->fgain, bs->fdtAvg, bs->fdt, bs->plane,
                            bs->friction, w, geo, status, sum[0], sum[1], sum[2]);
        else
            nodal_node<INT>(d, i, co, w, geo, status, sum[0], sum[1], sum[2]);
    }
    team.sync();
    time += dt;                                                       // :973-974
    steps += 1;
    double me;
    if (MIXED) {
        float m = 3.4028235e38f;
        for (int e = in.e0 + tid; e < in.e1; e += stride)
            element_reduced_f32(d, e, bs->fdt, bs->hourglass, pMid, vdt, base, m);
        for (int k = in.k0 + tid; k < in.k1; k += stride) {   // applyPressure, :1203-1207
            if (COMP) pressure_edge_comp(d, k, time, in.pressure, in.ramp);
            else pressure_edge_f32(d, k, time, in.pressure, in.ramp);
        }
        me = team_min_edge_next_f<TEAM, T>(team, m, shMin, bs, in, dt, dtPrev, d.finite);
    } else {
        double m = DMAX;
        for (int e = in.e0 + tid; e < in.e1; e += stride)
            element_reduced<INT>(d, e, dt, in.hourglass, m);
        for (int k = in.k0 + tid; k < in.k1; k += stride)
            pressure_edge(d, k, time, in.pressure, in.ramp);
        me = team_min_edge_next<TEAM, T>(team, m, shMin, bs, in, dt, dtPrev, d.finite);
    }
    // the gather keeps the nodal loop's node-to-thread map, so the next nodal update reads
    // only forces its own thread wrote
    for (int i = in.n0 + tid; i < in.n1; i += stride) {
        if (COMP) d.fC[i] = gather_node_comp(d, i, bs->gravR, bs->gravZ);
        else d.F[i] = MIXED ? gather_node_f32<INT>(d, i) : gather_node<INT>(d, i);
    }
    if (d.finite) {                                                   // :985-990
        dtPrev = dt;
        dt = bs->dt;
    }
    return me;
}

}  // namespace nf
