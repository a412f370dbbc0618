// k_setup.cu -- the arrays a scene or a batch derives from its meshes: node positions, shortest
// edge, the sources of every node, the edge groups of the free surface, lumped masses, the damage model's
// element geometry and the surface's edge ends. Every value is the host expression's (no
// contraction, sums in the same order), so the results are those of the serial loops.
//
// One core took 64 ms over these for 1M quads, half as long as the 400 steps that followed;
// here they are 1 ms of kernels (each a pass or two over the mesh, bound by its gathers) behind
// the upload of the mesh (a batch of 512 rods, 580k quads:
// 46 ms on one core and 15 so, which leaves the allocations, the checks and the upload). A scene of
// up to a thousand nodes takes one block and one launch (k_set_up_small). The orderings are counting sorts: an entry's place in its node's list is the
// number of smaller entries there, which each entry counts for itself, so no list is walked by
// one thread alone whatever the mesh's valences.
#include "nf_bodies.cuh"
#include "nf_internal.h"

namespace nf {

constexpr int SB = 256;

__device__ __forceinline__ int conn_at(const Dev &d, long long q) {
    return reinterpret_cast<const int *>(d.conn)[q];
}
__device__ __forceinline__ int edge_end(const Dev &d, long long q) {
    return conn_at(d, (q & ~3LL) + ((q + 1) & 3));
}

// The passes, each for one item; the kernels below run them over a grid, or (set_up_small) all of
// them in one block.
__device__ __forceinline__ void position(const Dev &d, int n) {
    const double *r = reinterpret_cast<const double *>(d.U);
    d.X0[n] = make_double2(r[n], r[d.N + n]);
}

// QuadMesh.minimumEdgeLength squared, as bits (a NaN is passed over).
__device__ __forceinline__ unsigned long long shortest_edge(const Dev &d, int e) {
    unsigned long long best = 0x7ff0000000000000ULL;
    const int4 c = d.conn[e];
    const int nn[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const double2 a = d.X0[nn[k]], b = d.X0[nn[(k + 1) & 3]];
        const double dr = b.x - a.x, dz = b.y - a.y;
        const unsigned long long q = __double_as_longlong(dr * dr + dz * dz);
        best = q < best ? q : best;
    }
    return best;
}
__global__ void __launch_bounds__(SB) k_positions(Dev d) {
    const int n = blockIdx.x * SB + threadIdx.x;
    if (n < d.N) position(d, n);
}
// The scene's shortest edge, or the element's instance's.
__global__ void __launch_bounds__(SB) k_shortest_edge(Dev d, unsigned long long *instances) {
    const int e = blockIdx.x * SB + threadIdx.x;
    const unsigned long long best = e < d.E ? shortest_edge(d, e) : 0x7ff0000000000000ULL;
    if (!instances) {
        commit_min_bits(best, &d.s->minEdgeBits);
    } else if (e < d.E) {
        unsigned long long *of = instances + d.emat[e];
        if (best < __ldcg(of)) atomicMin(of, best);
    }
}

// A block per instance: its elements' material, its nodes' velocity and fixed bits, and its
// local node numbers moved to the batch's.
__global__ void __launch_bounds__(SB) k_batch_fill(Dev d, const BatchInst *inst,
                                                   const double2 *velocity) {
    const BatchInst &in = inst[blockIdx.x];
    const double2 v = velocity[blockIdx.x];
    for (int n = in.n0 + threadIdx.x; n < in.n1; n += SB) {
        d.V[n] = v;
        d.flags[n] &= 3;
    }
    for (int e = in.e0 + threadIdx.x; e < in.e1; e += SB) {
        const int4 c = d.conn[e];
        d.conn[e] = make_int4(c.x + in.n0, c.y + in.n0, c.z + in.n0, c.w + in.n0);
        d.emat[e] = blockIdx.x;
    }
    for (int k = in.k0 + threadIdx.x; k < in.k1; k += SB) {
        const int2 p = d.pedges[k];
        d.pedges[k] = make_int2(p.x + in.n0, p.y + in.n0);
    }
}

// The sources of every node: element corner q (slot 8 e + corner), pressure-edge end k.
__device__ __forceinline__ int source_node(const Dev &d, long long q) {
    const long long n4 = 4LL * d.E;
    return q < n4 ? conn_at(d, q) : reinterpret_cast<const int *>(d.pedges)[q - n4];
}
__device__ __forceinline__ int source_slot(const Dev &d, long long q) {
    const long long n4 = 4LL * d.E;
    if (q < n4) return (int)((q >> 2) * 8 + (q & 3));
    const long long k = q - n4;
    return (int)((d.E + (k >> 1)) * 8 + (k & 1));
}

__device__ __forceinline__ void count_source(const Dev &d, long long q, int *sources, int *edges) {
    atomicAdd(&sources[source_node(d, q)], 1);
    if (edges && q < 4LL * d.E) atomicAdd(&edges[min(conn_at(d, q), edge_end(d, q))], 1);
}
// Into the nodes' ranges in any order; the counts run down to zero.
__device__ __forceinline__ void file_source(const Dev &d, long long q, int *sources, int *edges,
                                            const int *edgeStart, int *sourceBin, int *edgeBin) {
    const int n = source_node(d, q);
    sourceBin[d.nodeSlotStart[n] + atomicSub(&sources[n], 1) - 1] = source_slot(d, q);
    if (edges && q < 4LL * d.E) {
        const int lo = min(conn_at(d, q), edge_end(d, q));
        edgeBin[edgeStart[lo] + atomicSub(&edges[lo], 1) - 1] = (int)q;
    }
}
// buildNodeSlots (ExplicitSolver.java:347-366): a node's sources ascending; and the edges of one
// lower node by higher node, then by element edge.
__device__ __forceinline__ void rank_source(const Dev &d, long long q, const int *edgeStart,
                                            const int *sourceBin, const int *edgeBin) {
    {
        const int n = source_node(d, q), slot = source_slot(d, q);
        const int begin = d.nodeSlotStart[n], end = d.nodeSlotStart[n + 1];
        int rank = 0;
        for (int j = begin; j < end; j++) rank += sourceBin[j] < slot;
        d.nodeSlot[begin + rank] = slot;
    }
    if (edgeStart && q < 4LL * d.E) {
        const int a = conn_at(d, q), b = edge_end(d, q);
        const int lo = min(a, b), hi = max(a, b);
        const int begin = edgeStart[lo], end = edgeStart[lo + 1];
        int rank = 0;
        for (int j = begin; j < end; j++) {
            const int p = edgeBin[j], h = max(conn_at(d, p), edge_end(d, p));
            rank += h < hi || (h == hi && p < (int)q);
        }
        d.groupMember[begin + rank] = (int)q;
    }
}
// Equal undirected node pairs are neighbours now: a group starts where the pair changes.
__device__ __forceinline__ int group_head(const Dev &d, long long i) {
    int first = 1;
    if (i > 0) {
        const int q = d.groupMember[i], p = d.groupMember[i - 1];
        const int a = conn_at(d, q), b = edge_end(d, q), f = conn_at(d, p), g = edge_end(d, p);
        first = min(a, b) != min(f, g) || max(a, b) != max(f, g);
    }
    return first;
}
__device__ __forceinline__ void file_group(const Dev &d, long long i, const int *head,
                                           const int *before) {
    const int g = before[i] + head[i] - 1;
    d.edgeGroup[d.groupMember[i]] = g;
    if (head[i]) d.groupStart[g] = (int)i;
    if (i == 4LL * d.E - 1) d.groupStart[g + 1] = 4 * d.E;
}

// lumpMass, ExplicitSolver.java:1559-1597: 2x2 Gauss lumping. The four points' volumes by
// element, then each node adds its corners' shares: in element order, for each element point by
// point, and where an element has the node at several corners, those in turn within the point.
__device__ __forceinline__ double4 lump_volumes(const Dev &d, int e) {
    const double G = 0.5773502691896258;
    const double gx[4] = {-G, G, G, -G}, ge[4] = {-G, -G, G, G};
    const int4 c = d.conn[e];
    const double2 p0 = d.X0[c.x], p1 = d.X0[c.y], p2 = d.X0[c.z], p3 = d.X0[c.w];
    double v[4];
#pragma unroll
    for (int g = 0; g < 4; g++) {
        const double xi = gx[g], eta = ge[g];
        const double xm = 1.0 - xi, xp = 1.0 + xi;
        const double em = 1.0 - eta, ep = 1.0 + eta;
        const double N0 = 0.25 * xm * em, N1 = 0.25 * xp * em;
        const double N2 = 0.25 * xp * ep, N3 = 0.25 * xm * ep;
        const double dN0x = -0.25 * em, dN1x = 0.25 * em, dN2x = 0.25 * ep, dN3x = -0.25 * ep;
        const double dN0e = -0.25 * xm, dN1e = -0.25 * xp, dN2e = 0.25 * xp, dN3e = 0.25 * xm;
        const double J00 = dN0x * p0.x + dN1x * p1.x + dN2x * p2.x + dN3x * p3.x;
        const double J01 = dN0x * p0.y + dN1x * p1.y + dN2x * p2.y + dN3x * p3.y;
        const double J10 = dN0e * p0.x + dN1e * p1.x + dN2e * p2.x + dN3e * p3.x;
        const double J11 = dN0e * p0.y + dN1e * p1.y + dN2e * p2.y + dN3e * p3.y;
        const double det = J00 * J11 - J01 * J10;
        const double rg = N0 * p0.x + N1 * p1.x + N2 * p2.x + N3 * p3.x;
        v[g] = d.axi ? 2.0 * NF_PI * rg * det : d.thickness * det;
    }
    return make_double4(v[0], v[1], v[2], v[3]);
}
// Returns how many elements are around the node (its corners, counted once each).
__device__ __forceinline__ int lump_node(const Dev &d, int n, const double4 *volumes) {
    const double G = 0.5773502691896258;
    const double gx[4] = {-G, G, G, -G}, ge[4] = {-G, -G, G, G};
    double m = 0.0;
    const int begin = d.nodeSlotStart[n], end = d.nodeSlotStart[n + 1];
    int k = begin;
    while (k < end) {
        const int e = d.nodeSlot[k] >> 3;
        if (e >= d.E) break;                              // pressure edges come last
        int corners = 0;
        for (; k < end && (d.nodeSlot[k] >> 3) == e; k++) corners |= 1 << (d.nodeSlot[k] & 7);
        const double rho = d.mats[d.emat[e]].density;
        const double4 v4 = volumes[e];
        const double v[4] = {v4.x, v4.y, v4.z, v4.w};
#pragma unroll
        for (int g = 0; g < 4; g++) {
            const double xm = 1.0 - gx[g], xp = 1.0 + gx[g];
            const double em = 1.0 - ge[g], ep = 1.0 + ge[g];
            const double shape[4] = {0.25 * xm * em, 0.25 * xp * em, 0.25 * xp * ep,
                                     0.25 * xm * ep};
#pragma unroll
            for (int c = 0; c < 4; c++)
                if (corners >> c & 1) m += rho * shape[c] * v[g];
        }
    }
    d.mass[n] = m;
    d.invMass[n] = 1.0 / m;                               // nodalUpdate's 1/m, once
    return k - begin;
}

__global__ void __launch_bounds__(SB) k_count(Dev d, int *sources, int *edges) {
    const long long q = (long long)blockIdx.x * SB + threadIdx.x;
    if (q < 4LL * d.E + 2LL * d.K) count_source(d, q, sources, edges);
}
__global__ void __launch_bounds__(SB) k_file(Dev d, int *sources, int *edges, const int *edgeStart,
                                             int *sourceBin, int *edgeBin) {
    const long long q = (long long)blockIdx.x * SB + threadIdx.x;
    if (q < 4LL * d.E + 2LL * d.K) file_source(d, q, sources, edges, edgeStart, sourceBin, edgeBin);
}
__global__ void __launch_bounds__(SB) k_rank(Dev d, const int *edgeStart, const int *sourceBin,
                                             const int *edgeBin) {
    const long long q = (long long)blockIdx.x * SB + threadIdx.x;
    if (q < 4LL * d.E + 2LL * d.K) rank_source(d, q, edgeStart, sourceBin, edgeBin);
}
__global__ void __launch_bounds__(SB) k_heads(Dev d, int *head) {
    const long long i = (long long)blockIdx.x * SB + threadIdx.x;
    if (i < 4LL * d.E) head[i] = group_head(d, i);
}
__global__ void __launch_bounds__(SB) k_groups(Dev d, const int *head, const int *before) {
    const long long i = (long long)blockIdx.x * SB + threadIdx.x;
    if (i < 4LL * d.E) file_group(d, i, head, before);
}
__global__ void __launch_bounds__(SB) k_lump_volumes(Dev d, double4 *volumes) {
    const int e = blockIdx.x * SB + threadIdx.x;
    if (e < d.E) volumes[e] = lump_volumes(d, e);
}
__global__ void __launch_bounds__(SB) k_lump(Dev d, const double4 *volumes, int *most) {
    const int n = blockIdx.x * SB + threadIdx.x;
    const int corners = n < d.N ? lump_node(d, n, volumes) : 0;
    if (!most) return;
    const int m = __reduce_max_sync(0xffffffffu, corners);
    if ((threadIdx.x & 31) == 0 && m > __ldcg(most)) atomicMax(most, m);
}

// All of a small scene's passes in one block, a barrier between two of them: their dozen and a
// half launches took 75 us, a third of creating a scene of 32 quads.
constexpr int SMALL_BLOCK = 1024;
constexpr int SMALL_NODES = 1024;                          // and as many elements and pressure edges
__device__ void small_scan(const int *in, int *out, int n) {     // exclusive
    __shared__ int warps[SMALL_BLOCK / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int per = (n + SMALL_BLOCK - 1) / SMALL_BLOCK;
    const int begin = min((int)threadIdx.x * per, n), end = min(begin + per, n);
    int own = 0;
    for (int i = begin; i < end; i++) own += in[i];
    int sum = own;                                         // inclusive in the warp
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, sum, o);
        if (lane >= o) sum += t;
    }
    if (lane == 31) warps[warp] = sum;
    __syncthreads();
    if (warp == 0) {
        int w = warps[lane];
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += t;
        }
        warps[lane] = w;
    }
    __syncthreads();
    int at = sum - own + (warp ? warps[warp - 1] : 0);
    for (int i = begin; i < end; i++) {
        const int v = in[i];
        out[i] = at;
        at += v;
    }
    __syncthreads();
}
__global__ void __launch_bounds__(SMALL_BLOCK) k_set_up_small(Dev d, int *sources, int *edges,
                                                              int *edgeStart, int *most,
                                                              int *sourceBin, int *edgeBin,
                                                              int *head, int *before) {
    const int N = d.N, E = d.E, entries = 4 * E + 2 * d.K, t = threadIdx.x;
    double4 *volumes = reinterpret_cast<double4 *>(d.contribution);
    for (int n = t; n < N; n += SMALL_BLOCK) position(d, n);
    for (int q = t; q < entries; q += SMALL_BLOCK) count_source(d, q, sources, edges);
    __syncthreads();
    for (int n = t; n < N; n += SMALL_BLOCK) d.U[n] = make_double2(0.0, 0.0);
    for (int e = t; e < E; e += SMALL_BLOCK) atomicMin(&d.s->minEdgeBits, shortest_edge(d, e));
    small_scan(sources, d.nodeSlotStart, N + 1);
    small_scan(edges, edgeStart, N + 1);
    for (int q = t; q < entries; q += SMALL_BLOCK)
        file_source(d, q, sources, edges, edgeStart, sourceBin, edgeBin);
    __syncthreads();
    for (int q = t; q < entries; q += SMALL_BLOCK) rank_source(d, q, edgeStart, sourceBin, edgeBin);
    __syncthreads();
    for (int i = t; i < 4 * E; i += SMALL_BLOCK) head[i] = group_head(d, i);
    __syncthreads();
    small_scan(head, before, 4 * E);
    for (int i = t; i < 4 * E; i += SMALL_BLOCK) file_group(d, i, head, before);
    __syncthreads();                                       // the lists in `contribution` are done
    for (int e = t; e < E; e += SMALL_BLOCK) volumes[e] = lump_volumes(d, e);
    __syncthreads();
    for (int n = t; n < N; n += SMALL_BLOCK) atomicMax(most, lump_node(d, n, volumes));
    __syncthreads();
    for (int i = t; i < 8 * (E + d.K); i += SMALL_BLOCK) d.contribution[i] = 0.0;
}

// The damage model's element geometry, ExplicitSolver.java:767-789.
__global__ void __launch_bounds__(SB) k_damage_geometry(Dev d) {
    const int e = blockIdx.x * SB + threadIdx.x;
    if (e >= d.E) return;
    const int4 c = d.conn[e];
    const double2 p[4] = {d.X0[c.x], d.X0[c.y], d.X0[c.z], d.X0[c.w]};
    double a = 0.0;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const double2 i = p[k], j = p[(k + 1) & 3];
        a += i.x * j.y - j.x * i.y;
    }
    double o[5];
    o[0] = fabs(0.5 * a);
    o[1] = 0.5 * (p[1].x - p[0].x + p[2].x - p[3].x);
    o[2] = 0.5 * (p[1].y - p[0].y + p[2].y - p[3].y);
    o[3] = 0.5 * (p[3].x - p[0].x + p[2].x - p[1].x);
    o[4] = 0.5 * (p[3].y - p[0].y + p[2].y - p[1].y);
#pragma unroll
    for (int k = 0; k < 5; k++) {
        d.dGeom[5 * (size_t)e + k] = o[k];
        if (d.dGeomF) d.dGeomF[5 * (size_t)e + k] = (float)o[k];
    }
    if (d.dGeomF) {
        d.dFailF[e] = (float)d.dFail[e];
        d.dGfF[e] = (float)d.dGf[e];
    }
}

// The end nodes of every element edge (QuadMesh.surface's edge k of element e runs from corner
// k to corner k + 1).
__global__ void __launch_bounds__(SB) k_segments(Dev d) {
    const long long q = (long long)blockIdx.x * SB + threadIdx.x;
    if (q >= 4LL * d.E) return;
    d.segA[q] = conn_at(d, q);
    d.segB[q] = edge_end(d, q);
}

__global__ void __launch_bounds__(SB) k_component(const double2 *src, double *dst, int n, int y) {
    const int i = blockIdx.x * SB + threadIdx.x;
    if (i < n) dst[i] = y ? src[i].y : src[i].x;
}

__global__ void __launch_bounds__(SB) k_widen(const float *src, double *dst, int n, int stride) {
    const int i = blockIdx.x * SB + threadIdx.x;
    if (i < n) dst[i] = src[(size_t)i * stride];
}

// Doubles of a handle's staging buffer for fields on their way to the host, of `most` at a time:
// the set-up works in it first (a count and, for a scene's surface, two ints more per node, and
// the scan's space).
size_t stage_doubles(size_t most, int N, int E, bool surface) {
    const size_t ints = scan_tmp_ints(std::max(4 * E, N + 1)) + (surface ? 3 : 1) * ((size_t)N + 1);
    return std::max(most, (ints + 1) / 2);
}

// conn, emat, mats and pedges are in place, and r and z in U. The lists in between use
// `contribution`, which like U is zeroed again, and the staging buffer, zeroed.
static void node_arrays(Dev &d, cudaStream_t st, int *scratch, bool surface, int *most,
                        unsigned long long *instances) {
    const int N = d.N, E = d.E;
    const long long entries = 4LL * E + 2LL * d.K;
    int *sources = scratch, *edges = surface ? sources + N + 1 : nullptr;
    int *edgeStart = surface ? edges + N + 1 : nullptr;
    int *tmp = scratch + (surface ? 3 : 1) * ((size_t)N + 1);
    int *sourceBin = reinterpret_cast<int *>(d.contribution), *edgeBin = sourceBin + entries;
    int *head = edgeBin + 4LL * E, *before = head + 4LL * E;   // 16 E + 2 K of 16 (E + K)
    if (surface && E > 0 && N <= SMALL_NODES && E <= SMALL_NODES && d.K <= SMALL_NODES) {
        k_set_up_small<<<1, SMALL_BLOCK, 0, st>>>(d, sources, edges, edgeStart, most, sourceBin,
                                                  edgeBin, head, before);
        return;
    }
    if (N > 0) k_positions<<<grid_for(N, SB), SB, 0, st>>>(d);
    cudaMemsetAsync(d.U, 0, sizeof(double2) * (size_t)N, st);
    if (entries > 0) {
        const int grid = grid_for(entries, SB);
        if (E > 0) k_shortest_edge<<<grid_for(E, SB), SB, 0, st>>>(d, instances);
        k_count<<<grid, SB, 0, st>>>(d, sources, edges);
        scan_exclusive(sources, d.nodeSlotStart, N + 1, nullptr, tmp, st, nullptr, nullptr);
        if (surface) scan_exclusive(edges, edgeStart, N + 1, nullptr, tmp, st, nullptr, nullptr);
        k_file<<<grid, SB, 0, st>>>(d, sources, edges, edgeStart, sourceBin, edgeBin);
        k_rank<<<grid, SB, 0, st>>>(d, edgeStart, sourceBin, edgeBin);
    }
    if (E > 0 && surface) {
        const int grid = grid_for(4LL * E, SB);
        k_heads<<<grid, SB, 0, st>>>(d, head);
        scan_exclusive(head, before, 4 * E, nullptr, tmp, st, nullptr, nullptr);
        k_groups<<<grid, SB, 0, st>>>(d, head, before);
    }
    double4 *volumes = reinterpret_cast<double4 *>(d.contribution);
    if (E > 0) k_lump_volumes<<<grid_for(E, SB), SB, 0, st>>>(d, volumes);
    if (N > 0) k_lump<<<grid_for(N, SB), SB, 0, st>>>(d, volumes, most);
    cudaMemsetAsync(d.contribution, 0, sizeof(double) * 8 * ((size_t)E + d.K), st);
}

// A scene's arrays; its shortest edge goes to s, and the most elements around a node to surfNodes
// there, one read of both.
void launch_setup(Solver &S) {
    node_arrays(S.d, S.stream, reinterpret_cast<int *>(S.stage), true, &S.d.s->surfNodes, nullptr);
}
// A batch's: conn and pedges arrive with the instances' local numbers, flags as the caller's
// bytes, `edges` (per instance) at infinity.
void launch_batch_setup(Dev &d, const BatchInst *inst, int count, const double2 *velocity,
                        unsigned long long *edges, double *stage, cudaStream_t st) {
    k_batch_fill<<<count, SB, 0, st>>>(d, inst, velocity);
    node_arrays(d, st, reinterpret_cast<int *>(stage), false, nullptr, edges);
}
void setup_damage_geometry(Dev &d, cudaStream_t st) {
    if (d.E > 0) k_damage_geometry<<<grid_for(d.E, SB), SB, 0, st>>>(d);
}
void launch_segments(Solver &S) {
    if (S.d.E > 0) k_segments<<<grid_for(4LL * S.d.E, SB), SB, 0, S.stream>>>(S.d);
}
// The destination's pages first: a copy of 32 MB into pages not mapped yet took 13.6 ms (the
// device faults them in one by one), with them touched it takes 1.3 ms.
cudaError_t copy_to_host(void *dst, const void *src, size_t bytes, cudaStream_t st) {
    for (size_t i = 0; i < bytes; i += 4096) ((volatile char *)dst)[i] = 0;
    const cudaError_t e = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, st);
    return e == cudaSuccess ? cudaStreamSynchronize(st) : e;
}

// One component of a field of pairs, or a float field widened, in doubles: split on the device
// through `stage`, or on the host where the field is small and a launch costs more than its copy
// (45 nodes: 13 us a read by the copy, 20 by the kernel).
constexpr size_t SMALL_READ = 4096;
cudaError_t read_component(const double2 *src, double *dst, size_t count, int y, double *stage,
                           cudaStream_t st) {
    if (count <= SMALL_READ) {
        std::vector<double2> pairs(count);
        const cudaError_t e = copy_to_host(pairs.data(), src, sizeof(double2) * count, st);
        for (size_t i = 0; i < count; i++) dst[i] = y ? pairs[i].y : pairs[i].x;
        return e;
    }
    k_component<<<grid_for((long long)count, SB), SB, 0, st>>>(src, stage, (int)count, y);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? copy_to_host(dst, stage, sizeof(double) * count, st) : e;
}
cudaError_t read_widened(const float *src, double *dst, size_t count, int stride, double *stage,
                         cudaStream_t st) {
    if (count <= SMALL_READ) {
        std::vector<float> values((count - 1) * stride + 1);
        const cudaError_t e = copy_to_host(values.data(), src, sizeof(float) * values.size(), st);
        for (size_t i = 0; i < count; i++) dst[i] = values[i * stride];
        return e;
    }
    k_widen<<<grid_for((long long)count, SB), SB, 0, st>>>(src, stage, (int)count, stride);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? copy_to_host(dst, stage, sizeof(double) * count, st) : e;
}

}  // namespace nf
