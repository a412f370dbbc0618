// k_batch.cu -- many independent scenes (a parameter sweep: the reference runs one solver per
// thread through Sweep.over, src/main/java/org/neofiz/app/Sweep.java:82-105) stepped by one
// persistent kernel.
//
// One block, or for a batch with fewer instances than fill the device a cluster of up to eight
// (choose_team), owns one instance at a time and runs its whole step with block or cluster
// barriers between the phases: nodal update, element assembly with the block's exact minimum edge, the
// per-node gather, the next CFL step. They take instances from a queue (most expensive
// first), each for a chunk of steps, so uneven meshes and uneven step counts balance. Every
// phase calls the same per-node and per-element bodies as the single-scene kernels
// (nf_bodies.cuh), in the same order per node and per element, so an instance's trajectory is
// bit-identical to the same scene run alone in the same precision. The audit totals (wall
// impulse, energy loss, friction work) are summed by lanes over the steps of a chunk and the lanes
// in a fixed order (nf_batch_step.cuh): the same bits whatever the neighbours and so the blocks per
// instance, and for every block width while an instance has no more nodes than eight blocks of it
// have threads (one-warp blocks: while no two of its nodes at the wall are a multiple of 32
// apart); but not in the single-scene kernels' association.
//
// Launch shape: block size (32, 128, 256), whether the mixed form stages each instance's float
// node geometry in shared memory, blocks per SM and the chunk length are chosen by the
// autotuner (api_batch.cu). None of them changes an FP64 or mixed trajectory; the compensated
// one-warp kernels, which the tuner may choose, round differently from that form's wider ones.
#include "nf_batch_kernels.cuh"

#include <algorithm>
#include <functional>

namespace nf {

constexpr int MEASURE_BLOCK = 256;

// The first assembly of every instance (zero strain increment), in the batch's precision, as
// the single-scene path runs it before its first step; records the shortest edge.
template <bool MIXED>
__global__ void __launch_bounds__(256) k_batch_initial(Dev d, BatchDev b) {
    __shared__ double shMin[256 / 32 + 1];
    const BatchInst in = b.inst[blockIdx.x];
    double me;
    if (MIXED) {
        for (int i = in.n0 + threadIdx.x; i < in.n1; i += 256)
            prepare_node(d, i, 0.0, MixedGeo{d.pMid, nullptr, d.vdt, 0});
        __syncthreads();
        float m = 3.4028235e38f;
        for (int e = in.e0 + threadIdx.x; e < in.e1; e += 256)
            element_reduced_f32(d, e, 0.0f, (float)in.hourglass, d.pMid, d.vdt, 0, m);
        me = block_min_edge_f<256>(m, shMin);
    } else {
        double m = DMAX;
        for (int e = in.e0 + threadIdx.x; e < in.e1; e += 256)
            element_reduced<false>(d, e, 0.0, in.hourglass, m);
        me = block_min_edge<256>(m, shMin);
    }
    const double t0 = b.sc[blockIdx.x].time;
    for (int k = in.k0 + threadIdx.x; k < in.k1; k += 256) {
        if (MIXED) pressure_edge_f32(d, k, t0, in.pressure, in.ramp);
        else pressure_edge(d, k, t0, in.pressure, in.ramp);
    }
    __syncthreads();
    for (int i = in.n0 + threadIdx.x; i < in.n1; i += 256)
        d.F[i] = MIXED ? gather_node_f32<false>(d, i) : gather_node<false>(d, i);
    if (threadIdx.x == 0) b.sc[blockIdx.x].minEdgeSquared = me;
}

// Arms a run: every instance may take maxSteps more steps; counts the instances left to run.
__global__ void k_batch_arm(BatchDev b, long long maxSteps) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k == 0) *b.queue = 0;
    if (k >= b.count) return;
    BatchScalars &s = b.sc[k];
    s.stepLimit = s.steps + maxSteps;
    const int every = b.burst.every;
    const bool ended = every > 0 ? (s.steps % every == 0 && !(s.time < b.inst[k].tEnd)) ||
                                       b.burst.state[k].traversed
                                 : !(s.time < b.inst[k].tEnd);
    const bool done = ended || maxSteps <= 0;
    s.done = done ? 1 : 0;
    if (!done) atomicAdd(b.remaining, 1);
}

// TaylorImpactCase.java:272-288 per instance: max z, min z, max r of the current
// configuration, as order-preserving integer images (exact in any order).
__device__ __forceinline__ unsigned long long okey_b(double v) {
    const unsigned long long u = bbits(v);
    return (u >> 63) ? ~u : (u | 0x8000000000000000ULL);
}

__global__ void __launch_bounds__(MEASURE_BLOCK) k_batch_measure(Dev d, BatchDev b) {
    __shared__ unsigned long long sh[3][MEASURE_BLOCK / 32];
    const BatchInst in = b.inst[blockIdx.x];
    unsigned long long zmax = 0ULL, zmin = ~0ULL, rmax = 0ULL;
    for (int i = in.n0 + threadIdx.x; i < in.n1; i += MEASURE_BLOCK) {
        const double2 x = d.X0[i], u = d.U[i];
        const unsigned long long kz = okey_b(x.y + u.y), kr = okey_b(x.x + u.x);
        zmax = max(zmax, kz);
        zmin = min(zmin, kz);
        rmax = max(rmax, kr);
    }
    for (int o = 16; o > 0; o >>= 1) {
        zmax = max(zmax, __shfl_down_sync(0xffffffffu, zmax, o));
        zmin = min(zmin, __shfl_down_sync(0xffffffffu, zmin, o));
        rmax = max(rmax, __shfl_down_sync(0xffffffffu, rmax, o));
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) {
        sh[0][warp] = zmax;
        sh[1][warp] = zmin;
        sh[2][warp] = rmax;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < MEASURE_BLOCK / 32; w++) {
            zmax = max(zmax, sh[0][w]);
            zmin = min(zmin, sh[1][w]);
            rmax = max(rmax, sh[2][w]);
        }
        b.measure[3 * blockIdx.x + 0] = zmax;
        b.measure[3 * blockIdx.x + 1] = zmin;
        b.measure[3 * blockIdx.x + 2] = rmax;
    }
}

// ------------------------------------------------------------------------------------ launch

template <bool MIXED, bool STAGE>
static const void *by_threads(int threads, bool ints) {
    if (threads == 32) return (const void *)k_batch_steps<MIXED, STAGE, 32, false, false>;
    if (threads == 128) return (const void *)k_batch_steps<MIXED, STAGE, 128, false, false>;
    if (MIXED && ints) return (const void *)k_batch_steps<MIXED, STAGE, TEAM_THREADS, MIXED, false>;
    return (const void *)k_batch_steps<MIXED, STAGE, TEAM_THREADS, false, false>;
}

// The kernel of a shape. ints: the node products on the integer units (batch_int_products).
static const void *select_kernel(int mode, const BatchShape &s, bool ints, bool team) {
    if (mode == NF_PRECISION_COMPENSATED) return comp_steps_kernel(s, team);
    if (mode == NF_PRECISION_MIXED) {
        if (team) return ints ? (const void *)k_batch_steps<true, false, TEAM_THREADS, true, true>
                              : (const void *)k_batch_steps<true, false, TEAM_THREADS, false, true>;
        return s.stage ? by_threads<true, true>(s.threads, ints) : by_threads<true, false>(s.threads, ints);
    }
    return team ? (const void *)k_batch_steps<false, false, TEAM_THREADS, false, true>
                : by_threads<false, false>(s.threads, false);
}
// Whether a shape's products go to the integer units: in the mixed form, whose products are the
// nodes' alone, with blocks of 256 threads of which a quarter SM has more than one warp with
// elements (150 rods of 24 x 120: 6.64 ms per 100 steps and 7.07 without, 256 ragged ones 26.9
// and 27.4; narrower blocks lose, 1,200 rods of 10 x 30 in blocks of 128: 8.4 ms and 6.9). The
// FP64 step has no room for it: its 255 registers leave a quarter SM two warps at most, and
// with a whole element's products in integer code they wait for instructions: 1,200 rods of
// 10 x 30: 99 ms and 55 without, 512 burst slices 6.7 and 4.8, 256 ragged rods 223 and 157, and no
// size of 1 to 1,200 instances the other way round.
static bool batch_int_products(int mode, const BatchShape &s, int maxElems, int team) {
    if (mode != NF_PRECISION_MIXED || s.threads != TEAM_THREADS) return false;
    const int most = s.threads / 32 * team, needed = (maxElems + 31) / 32;
    const int warps = needed < most ? needed : most;
    return int_products((long long)s.blocksPerSm * ((warps + team - 1) / team), 1);
}

size_t batch_shared_bytes(int mode, const BatchShape &s, int maxNodes) {
    return mode != NF_PRECISION_FP64 && s.stage ? (sizeof(float4) + sizeof(float2)) * (size_t)maxNodes
                                                : 0;
}

static cudaLaunchConfig_t team_config(cudaLaunchAttribute &at, int teams, int team, int threads,
                                      cudaStream_t st) {
    cudaLaunchConfig_t cfg = {};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = team;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.gridDim = dim3(teams * team);
    cfg.blockDim = dim3(threads);
    cfg.stream = st;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cfg;
}
// Teams of `team` blocks that kernel k keeps resident (0: none).
int max_teams(const void *k, int team, int threads) {
    cudaLaunchAttribute at;
    const cudaLaunchConfig_t cfg = team_config(at, 1, team, threads, nullptr);
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, k, &cfg) != cudaSuccess) {
        (void)cudaGetLastError();
        return 0;
    }
    return n;
}
// Blocks per instance for the `count` most expensive instances (their element counts in `elems`),
// given the teams of 1, 2, 4 and 8 blocks that can be resident. A step costs an instance a fixed
// part and its elements' rounds over the team's threads, half a round at least (below four warps
// a block its quarter SMs have one warp each already): 0.6 + elements / (256 team). Teams take
// the instances in this order, each the next when it is free; the time until the last is done,
// plus half the longest instance's (which goes on when most have ended), is compared. The constants
// are fitted, to runs of 10 to 1,500 ragged rods in three forms and of 16 equal ones, with 1 to
// 8 blocks each (profiles/batch_teams.md): this picks the fastest, or one within 2 % of it, of 21
// groups of 22 (64 FP64 rods 196, 106, 62 and 85 ms with 1, 2, 4 and 8 blocks, 256 mixed ones 44.6,
// 27.2, 26.9 and 37.9), and in the other, 1,500 compensated rods, 52.5 ms where one block takes 49.8.
int choose_team(const int *elems, int count, const int (&teams)[4]) {
    if (count >= 8 * teams[0]) return 1;     // long queues: nothing to share out
    int best = 1;
    double least = 0.0;
    std::vector<double> busy;                // a heap: the team free first on top
    for (int q = 0; q < 4; q++) {
        const int team = 1 << q, n = teams[q] < count ? teams[q] : count;
        if (n < 1) continue;
        busy.assign(n, 0.0);
        double longest = 0.0, last = 0.0;
        for (int k = 0; k < count; k++) {
            const double rounds = elems[k] / (256.0 * team);
            const double t = 0.6 + (rounds > 0.5 ? rounds : 0.5);
            if (t > longest) longest = t;
            std::pop_heap(busy.begin(), busy.end(), std::greater<double>());
            busy.back() += t;
            if (busy.back() > last) last = busy.back();
            std::push_heap(busy.begin(), busy.end(), std::greater<double>());
        }
        const double cost = last + 0.5 * longest;
        if (q == 0 || cost < 0.98 * least) {
            best = team;
            least = cost;
        }
    }
    return best;
}
cudaError_t launch_team(const void *k, int teams, int team, int threads, void **args,
                        cudaStream_t st) {
    cudaLaunchAttribute at;
    const cudaLaunchConfig_t cfg = team_config(at, teams, team, threads, st);
    return cudaLaunchKernelExC(&cfg, k, args);
}

// Teams of 1, 2, 4 and 8 blocks that a shape keeps resident; only the 256-thread kernels without
// staged nodes come as teams.
void batch_teams(int mode, const BatchShape &s, int sms, int (&teams)[4]) {
    teams[0] = sms * s.blocksPerSm;
    for (int q = 1; q < 4; q++) {
        teams[q] = 0;
        if (s.threads != TEAM_THREADS || s.stage) continue;
        const int n = max_teams(select_kernel(mode, s, true, true), 1 << q, TEAM_THREADS);
        teams[q] = n < teams[0] >> q ? n : teams[0] >> q;
    }
}

// Resident blocks per SM of a shape (0 when it cannot launch, e.g. too much shared memory). The
// kernels with and without integer products are both made ready: which one a launch takes depends
// on the blocks per SM that the answer bounds.
int batch_max_blocks_per_sm(int mode, const BatchShape &s, int maxNodes, int maxElems) {
    const size_t smem = batch_shared_bytes(mode, s, maxNodes);
    for (const bool ints : {false, true}) {
        if (smem > 48 * 1024 &&
            cudaFuncSetAttribute(select_kernel(mode, s, ints, false),
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
            (void)cudaGetLastError();
            return 0;
        }
    }
    const void *k = select_kernel(mode, s, batch_int_products(mode, s, maxElems, 1), false);
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, s.threads, smem) != cudaSuccess) {
        (void)cudaGetLastError();
        return 0;
    }
    return n;
}

// Blocks per SM that a shape may ask for even where fewer are resident: the FP64 kernels once
// took 168 registers a thread, 384 threads an SM (1, 3 and 12 blocks of 256, 128 and 32), and
// shapes chosen then, by hand or by the tuner, stay valid. They launch what is resident: the
// blocks share a queue, and further ones would find it empty.
int batch_blocks_promised(int mode, const BatchShape &s) {
    return mode == NF_PRECISION_FP64 ? 384 / s.threads : 0;
}

// team: blocks per instance (choose_team); teams: how many of them.
cudaError_t launch_batch_steps(const Dev &d, const BatchDev &b, int mode, const BatchShape &s,
                               int team, int teams, cudaStream_t st) {
    Dev dd = d;
    BatchDev bb = b;
    int chunk = s.chunk;
    void *args[] = {&dd, &bb, &chunk};
    const bool ints = batch_int_products(mode, s, b.maxElems, team);
    if (teams > b.count) teams = b.count;
    if (teams < 1) teams = 1;
    if (team > 1)
        return launch_team(select_kernel(mode, s, ints, true), teams, team, TEAM_THREADS, args, st);
    const size_t smem = batch_shared_bytes(mode, s, b.maxNodes);
    return cudaLaunchKernel(select_kernel(mode, s, ints, false), dim3(teams), dim3(s.threads), args,
                            smem, st);
}

void launch_batch_initial(const Dev &d, const BatchDev &b, bool mixed, cudaStream_t st) {
    if (b.count <= 0) return;
    if (mixed) k_batch_initial<true><<<b.count, 256, 0, st>>>(d, b);
    else k_batch_initial<false><<<b.count, 256, 0, st>>>(d, b);
}

void launch_batch_arm(const BatchDev &b, long long maxSteps, cudaStream_t st) {
    cudaMemsetAsync(b.remaining, 0, sizeof(int32_t), st);
    k_batch_arm<<<grid_for(b.count > 0 ? b.count : 1, 256), 256, 0, st>>>(b, maxSteps);
}

void launch_batch_measure(const Dev &d, const BatchDev &b, cudaStream_t st) {
    if (b.count > 0) k_batch_measure<<<b.count, MEASURE_BLOCK, 0, st>>>(d, b);
}

}  // namespace nf
