// The whole sweep of a small system in one launch: the cell-list rebuild and every checkerboard
// phase inside one thread-block cluster, phases separated by the cluster's hardware barrier.
//
// A small system's sweep is bound by launches, not by work: with at most 256 active cells a phase,
// a rebuild of six launches and 8 to 27 phases of two launches each (the sweep and the rerun of
// overfull neighbourhoods) took 180 us a sweep for 1000 hard spheres; one launch takes 69.  Up to 16 blocks (one per SM of a GPC) give every active cell a warp of its own; the
// blocks of a cluster are scheduled together, so the barrier needs no cooperative launch and
// several handles' sweeps may run side by side.  Cells, moves and their order within a cell are
// the phase-by-phase sweep's, so the results are the same.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include "rp_sweep.cuh"

namespace rp {

constexpr int CL_MAX_WARPS = 16;             // warps per block (the sweep's 128 registers a thread)
constexpr size_t CL_SMEM = 208 * 1024;       // a block's shared memory: also one overfull cell's staging

// What the host adds to the sweep's arguments.
struct ClusterSweep {
    int nphases, cap_big;
    int8_t phase[MAX_PHASES + 1];
};

namespace {

// The rebuild of launch_rebuild (assign, scan, scatter, finish), without the cells' occupancy
// order, by all threads of the cluster; the scan by the first block.  Also zeroes the phases' counts of
// overfull neighbourhoods.
__device__ void cluster_rebuild(const DevState &s, const GridDev &g, int32_t *overfull, int nphases,
                                const cooperative_groups::cluster_group &cl) {
    __shared__ int32_t warp_tot[CL_MAX_WARPS], warp_max[CL_MAX_WARPS];
    const int rank = cl.block_rank(), T = blockDim.x;
    const int tid = rank * T + threadIdx.x, nth = cl.num_blocks() * T;
    for (int c = tid; c < g.ncell; c += nth) g.count[c] = 0;
    if (tid < nphases) overfull[tid] = 0;
    cl.sync();
    for (int64_t i = tid; i < s.n; i += nth) assign_one(s, g, i);
    cl.sync();
    if (rank == 0) {
        const int per = (g.ncell + T - 1) / T, b = threadIdx.x * per, e = min(g.ncell, b + per);
        const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
        int sum = 0, mx = 0;
        for (int c = b; c < e; c++) {
            sum += g.count[c];
            mx = max(mx, g.count[c]);
        }
        int incl = sum;
        for (int d = 1; d < 32; d <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= d) incl += y;
        }
        mx = __reduce_max_sync(0xffffffffu, mx);
        if (lane == 31) {
            warp_tot[w] = incl;
            warp_max[w] = mx;
        }
        __syncthreads();
        int run = incl - sum;
        for (int k = 0; k < w; k++) run += warp_tot[k];
        if (threadIdx.x == 0) {
            int total = 0, most = 0;
            for (int k = 0; k < T / 32; k++) {
                total += warp_tot[k];
                most = max(most, warp_max[k]);
            }
            g.start[g.ncell] = total;
            *g.max_occ = most;
        }
        for (int c = b; c < e; c++) {
            g.start[c] = run;
            run += g.count[c];
        }
    }
    cl.sync();
    for (int64_t i = tid; i < s.n; i += nth) scatter_one(g, i);
    cl.sync();
    for (int c = tid; c < g.ncell; c += nth) finish_one(s, g, c);
    cl.sync();
}

template <int KIND, int MODE, bool SEG>
__global__ void __launch_bounds__(CL_MAX_WARPS * 32, 1)
    k_cluster_sweep(const __grid_constant__ SweepArgs A, const __grid_constant__ ClusterSweep P) {
    extern __shared__ float4 smem[];
    const cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, W = blockDim.x >> 5;
    const int rank = cl.block_rank(), nb = cl.num_blocks();
    const GridDev &G = A.g;
    cluster_rebuild(A.s, G, A.overflow_count, P.nphases, cl);
    __shared__ WarpStats stats[CL_MAX_WARPS];
    WarpStats &ws = stats[w];
    if (lane == 0) ws = WarpStats{};
    __syncwarp();
    for (int p = 0; p < P.nphases; p++) {
        const int ph = P.phase[p];
        int act[3];
        for (int d = 0; d < 3; d++) act[d] = ring_count(G.dims[d], phase_digit(ph, d));
        // pass 0: the phase's cells, one warp each; pass 1: those whose neighbourhood exceeds a
        // warp's share of the shared memory, one block each.  Their count is the phase's own: a warp
        // that reads it late, after others went on to the next phase, must not meet that phase's
        int32_t *const overfull = A.overflow_count + p;
        int items = act[0] * act[1] * act[2];
        for (int pass = 0; pass < 2; pass++) {
            const int cap = pass == 0 ? A.cap : P.cap_big;
            const int extra = KIND == 1 ? cap : (KIND == 2 ? cap / 4 : 0);
            const int per_warp = cap + extra + cap / 4 + cap / 16 + sweep_scratch(KIND);
            float4 *cpos = smem + (pass == 0 ? (size_t)w * per_warp : 0);
            float4 *cax = cpos + cap;
            uint32_t *cslot = reinterpret_cast<uint32_t *>(cpos + cap);
            uint16_t *qseg = reinterpret_cast<uint16_t *>(cpos + cap + extra);
            uint16_t *qun = qseg + cap;
            uint8_t *nacc = reinterpret_cast<uint8_t *>(qun + cap);
            float4 *wx = reinterpret_cast<float4 *>(nacc + cap);
            // cells spread over the blocks first
            const int first = pass == 0 ? w * nb + rank : (w == 0 ? rank : items);
            const int stride = pass == 0 ? nb * W : nb;
            for (int item = first; item < items; item += stride) {
                int cell;
                if (pass == 0) {
                    const int a0 = item % act[0], q = item / act[0], a1 = q % act[1], a2 = q / act[1];
                    cell = ring_cell(G.dims[0], phase_digit(ph, 0), a0) +
                           G.dims[0] * (ring_cell(G.dims[1], phase_digit(ph, 1), a1) +
                                        G.dims[1] * ring_cell(G.dims[2], phase_digit(ph, 2), a2));
                } else {
                    cell = __ldcg(A.overflow + item);
                }
                sweep_cell<KIND, false, MODE, 32, SEG>(A, item, cell, cap, pass == 0 ? A.overflow : nullptr,
                                                       overfull, cpos, cax, qseg, qun, nacc, nullptr, cslot, wx, ws);
                __syncwarp();
            }
            cl.sync();
            if (pass == 0) {
                items = __ldcg(overfull);
                if (items == 0) break;
            }
        }
    }
    if (lane == 0 && ws.moves) {
        unsigned long long *C = A.s.counters;
        atomicAdd(C + 0, (unsigned long long)ws.moves);
        atomicAdd(C + 1, (unsigned long long)ws.accepted);
        atomicAdd(C + 2, (unsigned long long)ws.rej_overlap);
        atomicAdd(C + 3, (unsigned long long)ws.rej_domain);
        atomicAdd(C + 4, (unsigned long long)ws.pairs);
        atomicAdd(C + 5, (unsigned long long)ws.fp64);
        atomicAdd(C + 6, (unsigned long long)ws.trans);
        atomicAdd(C + 7, (unsigned long long)ws.rots);
        atomicAdd(C + 8, (unsigned long long)ws.acc_trans);
    }
}

template <int KIND, int MODE, bool SEG = KIND == 2>
cudaError_t launch_t(const SweepArgs &a, const ClusterSweep &p, int blocks, int warps, cudaStream_t st, bool probe, int *fits) {
    auto kernel = k_cluster_sweep<KIND, MODE, SEG>;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CL_SMEM);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return e;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = (unsigned)blocks;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)blocks);
    cfg.blockDim = dim3((unsigned)warps * 32);
    cfg.dynamicSmemBytes = CL_SMEM;
    cfg.stream = st;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    if (probe) return cudaOccupancyMaxActiveClusters(fits, kernel, &cfg);
    e = cudaLaunchKernelEx(&cfg, kernel, a, p);
    const cudaError_t last = cudaGetLastError();   // (taken: the next launch must not report this one's)
    return e != cudaSuccess ? e : last;
}

cudaError_t dispatch(const SweepArgs &a, const ClusterSweep &p, int blocks, int warps, cudaStream_t st, bool probe, int *fits) {
    const bool count = a.s.counting != 0, rt = a.types == SWEEP_ROTOTRANSLATION && !count;
    if (a.s.kind == 0) {
        if (count) return launch_t<0, 2>(a, p, blocks, warps, st, probe, fits);
        if (a.soft32) return launch_t<0, 4>(a, p, blocks, warps, st, probe, fits);
        return rt ? launch_t<0, 3>(a, p, blocks, warps, st, probe, fits) : launch_t<0, 0>(a, p, blocks, warps, st, probe, fits);
    }
    if (a.s.kind == 1) {
        if (count) return launch_t<1, 2>(a, p, blocks, warps, st, probe, fits);
        return rt ? launch_t<1, 3>(a, p, blocks, warps, st, probe, fits) : launch_t<1, 0>(a, p, blocks, warps, st, probe, fits);
    }
    if (count) return launch_t<2, 2>(a, p, blocks, warps, st, probe, fits);
    if (rt) return launch_t<2, 3>(a, p, blocks, warps, st, probe, fits);
    return a.s.segs ? launch_t<2, 0>(a, p, blocks, warps, st, probe, fits)
                    : launch_t<2, 0, false>(a, p, blocks, warps, st, probe, fits);
}

}  // namespace

size_t sweep_smem_per_warp(int kind, int cap, bool learn, int ncen);

// Blocks of the largest cluster (16 or 8) that fits the device with a block's 208 KB; 0: none.
int cluster_blocks() {
    SweepArgs a{};
    ClusterSweep p{};
    for (int blocks = 16; blocks >= 8; blocks /= 2) {
        int fits = 0;
        if (dispatch(a, p, blocks, CL_MAX_WARPS, nullptr, true, &fits) == cudaSuccess && fits > 0) return blocks;
        cudaGetLastError();
    }
    return 0;
}

// Warps per block of a cluster sweep over at most `active` cells a phase (0: the phases have more
// cells than the cluster can hold warps for).
int cluster_warps(const SweepArgs &a, int blocks, int active) {
    const size_t per = sweep_smem_per_warp(a.s.kind, a.cap, false, a.s.ncen);
    const int room = (int)(CL_SMEM / per < (size_t)CL_MAX_WARPS ? CL_SMEM / per : CL_MAX_WARPS);
    const int need = (active + blocks - 1) / blocks;
    if (blocks == 0 || need > room) return 0;
    return need < 4 ? (room < 4 ? room : 4) : need;
}

cudaError_t launch_cluster_sweep(const SweepArgs &a, const int *phases, int nphases, int blocks, int warps, cudaStream_t st) {
    ClusterSweep p{};
    p.nphases = nphases;
    for (int k = 0; k < nphases; k++) p.phase[k] = (int8_t)phases[k];
    // candidates one warp stages in a whole block's shared memory (16-bit queue entries)
    const size_t fixed = sweep_smem_per_warp(a.s.kind, 0, false, a.s.ncen);
    const size_t cap = (CL_SMEM - fixed) * 32 / (sweep_smem_per_warp(a.s.kind, 32, false, a.s.ncen) - fixed);
    p.cap_big = (int)((cap < 65504 ? cap : 65504) / 32 * 32);
    return dispatch(a, p, blocks, warps, st, false, nullptr);
}

}  // namespace rp
