// sbx_obs.cu — per-network observables of dense networks (single or packed): the filament
// RMS extent (FullSystemDemoHarness.filRms, FullSystemDemoHarness.java:1047-1055), the
// largest-cluster fraction, and the mean in-plane network stress.
//
// Reductions are deterministic: per network, 256 chains of additions in FP64 (chain t takes
// items t, t+256, ... of its network in index order), then a fixed shared-memory tree over
// the chains (strides 128 .. 1). The oracle restates this order, so results are
// bit-identical to it (and equal the reference's serial sums to ~1e-13 relative).
// The order leaves 256 serial chains, each cheap: what a reduction costs is the latency of
// the loads behind its terms (a link's two rods, a head's rod). So a cluster of OBS_CTAS
// blocks takes a network, 32 chains a block; the block's 16 warps make a window of terms
// (row w of the window: the next item of each of the 32 chains) in shared memory and its
// first warp adds the window before it, one chain a lane. On 12 packed networks (0.17e6
// rods, 0.18e6 heads) that takes 25 us (stress) and 24 us (extent); one block of 256 threads
// per network took 159 us and 103 us.
//
// Clusters: nodes are the segments and the backbones; edges are chain links, ACTIVE
// crosslinks and bound heads (segment -- the head's backbone). Each edge joins its components
// completely: the larger root is hooked onto the smaller one with a compare-and-swap and the
// edge tries again from the roots it finds when another edge was first. A root only ever gets
// a smaller parent, so the final root of a component is its smallest node id and the
// labelling does not depend on the order in which edges are processed. The chain links go
// first, then paths are flattened, then the other edges join and every node is labelled.
// Rounds of hooking and compressing, launched up to the caller's limit whether or not anything
// was left to do, took 128 launches and 425 us on the 12 networks; the six launches take 44.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include "../../include/softbox_b200.h"
#include "sbx_internal.cuh"

namespace cg = cooperative_groups;

namespace {

constexpr int OBS_THREADS = 256;
constexpr int OBS_CTAS = 8;               // blocks of a network's cluster (256 / OBS_CTAS = 32 chains each)
constexpr int OBS_WARPS = 16;             // warps making terms
constexpr int OBS_ROWS = 4;               // rows a warp has in flight: a window is OBS_WARPS * OBS_ROWS rows
constexpr int EXT_ROWS = 1;               // the extent's first pass: four sums a chain, so shorter windows
constexpr int OBS_MAX_FIND = 1 << 20;

__device__ __forceinline__ void tree_sum(double* sh, int w) {
    for (int s = OBS_THREADS / 2; s > 0; s >>= 1) {
        __syncthreads();
        if (threadIdx.x < s)
            for (int k = 0; k < w; k++) sh[k * OBS_THREADS + threadIdx.x] += sh[k * OBS_THREADS + threadIdx.x + s];
    }
    __syncthreads();
}

__device__ __forceinline__ double seg_c(const float* c, const double* c64, int n, int i, int k) {
    return c64 ? c64[(int64_t)k * n + i] : (double)c[(int64_t)k * n + i];
}

// Adds the terms of items [k0, k1) to the block's 32 chains in chain order: lane l of warp 0
// ends with the W sums of chain 32 * rank + l in acc. make(i, v) writes item i's W terms; an
// item that does not count writes zeros, which leave a sum that starts at +0.0 as it is.
template <int W, int ROWS, class Make>
__device__ void chain_sums(int k0, int k1, int rank, double (*win)[OBS_WARPS * ROWS][W][32], const Make& make,
                           double acc[W]) {
    constexpr int WIN = OBS_WARPS * ROWS;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int rows = (k1 - k0 + OBS_THREADS - 1) / OBS_THREADS;
    const int windows = (rows + WIN - 1) / WIN;
    for (int w = 0; w <= windows; w++) {
        if (w < windows) {
#pragma unroll
            for (int q = 0; q < ROWS; q++) {
                const int r = q * OBS_WARPS + warp;
                const int i = k0 + (w * WIN + r) * OBS_THREADS + 32 * rank + lane;
                double v[W];
#pragma unroll
                for (int c = 0; c < W; c++) v[c] = 0.0;
                if (i < k1) make(i, v);
#pragma unroll
                for (int c = 0; c < W; c++) win[w & 1][r][c][lane] = v[c];
            }
        }
        if (w > 0 && warp == 0) {
            const int left = rows - (w - 1) * WIN, n = left < WIN ? left : WIN;
            for (int r = 0; r < n; r++)
#pragma unroll
                for (int c = 0; c < W; c++) acc[c] += win[(w - 1) & 1][r][c][lane];
        }
        __syncthreads();
    }
}

// out[2*net] = RMS extent (um), out[2*net+1] = active segment count
__global__ void __cluster_dims__(OBS_CTAS, 1, 1) __launch_bounds__(32 * OBS_WARPS)
    k_extent(int n, const int* segBase, const float* coord, const double* coord64, const int* filState, double* out) {
    __shared__ union {
        double first[2][OBS_WARPS * EXT_ROWS][4][32], second[2][OBS_WARPS * OBS_ROWS][1][32];
    } win;
    __shared__ double sh[4 * OBS_THREADS];
    __shared__ double mean[4];
    cg::cluster_group cl = cg::this_cluster();
    const int net = blockIdx.x / OBS_CTAS, rank = (int)cl.block_rank(), t = threadIdx.x;
    const int b0 = segBase[net], b1 = segBase[net + 1];
    double* sh0 = cl.map_shared_rank(sh, 0);
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    cl.sync();                             // every block of the cluster runs before its memory is used
    chain_sums<4, EXT_ROWS>(b0, b1, rank, win.first, [&](int i, double v[4]) {
        const bool on = !filState || filState[i] >= 0;
        double c[3];
        for (int k = 0; k < 3; k++) c[k] = seg_c(coord, coord64, n, i, k);
        if (on) { v[0] = 1.0; v[1] = c[0]; v[2] = c[1]; v[3] = c[2]; }
    }, acc);
    if (t < 32)
        for (int c = 0; c < 4; c++) sh0[c * OBS_THREADS + 32 * rank + t] = acc[c];
    cl.sync();
    if (rank == 0) {
        tree_sum(sh, 4);
        if (t == 0) {
            double c = sh[0];
            mean[0] = c;
            for (int k = 1; k < 4; k++) mean[k] = c > 0 ? sh[k * OBS_THREADS] / c : 0.0;
        }
    }
    cl.sync();
    const double* m0 = cl.map_shared_rank(mean, 0);
    const double cnt = m0[0], mx = m0[1], my = m0[2], mz = m0[3];
    double s2[1] = {0.0};
    chain_sums<1, OBS_ROWS>(b0, b1, rank, win.second, [&](int i, double v[1]) {
        const bool on = !filState || filState[i] >= 0;
        double dx = seg_c(coord, coord64, n, i, 0) - mx;
        double dy = seg_c(coord, coord64, n, i, 1) - my;
        double dz = seg_c(coord, coord64, n, i, 2) - mz;
        if (on) v[0] = dx * dx + dy * dy + dz * dz;
    }, s2);
    // (the first block read its own chains' sums before the cluster barrier above)
    if (t < 32) sh0[32 * rank + t] = s2[0];
    cl.sync();
    if (rank == 0) {
        tree_sum(sh, 1);
        if (t == 0) {
            out[2 * net] = cnt > 0 ? sqrt(sh[0] / cnt) : 0.0;
            out[2 * net + 1] = cnt;
        }
    }
}

// virial of the link and bond payloads: out[net] = -(sum r_x F_x + r_y F_y) / (2 V), Pa
__global__ void __cluster_dims__(OBS_CTAS, 1, 1) __launch_bounds__(32 * OBS_WARPS) k_stress(
    int nSeg, const float* fC, const float* fU, const float* fE1, const float* fLen, const int* linkBase,
    const int* linkA, const int* linkB, const int* linkState, const float* loc1, const float* loc2, const float* xd,
    int nB, const int* motBase, const float* mC, const float* mU, const int* boundSeg, const float* bindArc,
    const float* bd, double headLen, const float* volume, double* out) {
    __shared__ double win[2][OBS_WARPS * OBS_ROWS][1][32];
    __shared__ double sh[OBS_THREADS];
    cg::cluster_group cl = cg::this_cluster();
    const int net = blockIdx.x / OBS_CTAS, rank = (int)cl.block_rank(), t = threadIdx.x;
    double w[1] = {0.0};
    cl.sync();                             // every block of the cluster runs before its memory is used
    if (linkBase)
        chain_sums<1, OBS_ROWS>(linkBase[net], linkBase[net + 1], rank, win, [&](int k, double v[1]) {
            int a = linkA[k], b = linkB[k];
            if (linkState[k] < 0 || a < 0 || b < 0) return;
            double l1 = loc1[k], l2 = loc2[k];
            double rx = (fE1[a] + l1 * fU[a]) - (fE1[b] + l2 * fU[b]);
            double ry = (fE1[nSeg + a] + l1 * fU[nSeg + a]) - (fE1[nSeg + b] + l2 * fU[nSeg + b]);
            v[0] = 1.0e-6 * rx * xd[12 * (int64_t)k] + 1.0e-6 * ry * xd[12 * (int64_t)k + 1];
        }, w);
    if (motBase)
        chain_sums<1, OBS_ROWS>(motBase[net], motBase[net + 1], rank, win, [&](int m, double v[1]) {
            int s = boundSeg[m];
            if (s < 0) return;
            int h = 3 * m + 2;
            double hx = mC[h] + 0.5 * headLen * mU[h], hy = mC[nB + h] + 0.5 * headLen * mU[nB + h];
            double off = (double)bindArc[m] - 0.5 * fLen[s];
            double ax = fC[s] + off * fU[s], ay = fC[nSeg + s] + off * fU[nSeg + s];
            v[0] = 1.0e-6 * (hx - ax) * bd[13 * (int64_t)m] + 1.0e-6 * (hy - ay) * bd[13 * (int64_t)m + 1];
        }, w);
    if (t < 32) cl.map_shared_rank(sh, 0)[32 * rank + t] = w[0];
    cl.sync();
    if (rank == 0) {
        tree_sum(sh, 1);
        if (t == 0) out[net] = -sh[0] / (2.0 * volume[net] * 1.0e-18);
    }
}

// ---------------------------------------------------------------- clusters
// The root of x's component, or -1 past OBS_MAX_FIND steps. The path is halved on the way, from
// step FROM on: a node's parent may be replaced by any of its ancestors, every walk through it
// still ends at the same root, and the walks of all nodes of a long chain shorten one another
// (one chain of 2^21 rods without that took 240 ms, now 2.2). Other blocks move parents meanwhile,
// so parents are read past L1. FINAL: where roots are written as labels beside the walks; a
// late, larger ancestor must not replace one.
constexpr int SHORT_PATH = 4;            // a filament's path: cheaper walked than halved
template <int FROM, bool FINAL>
__device__ __forceinline__ int find_root(int* label, int x) {
    int p = __ldcg(label + x);
    for (int it = 0; it < OBS_MAX_FIND; it++) {
        if (p == x) return p;
        const int g = __ldcg(label + p);
        if (g == p) return p;
        if (it >= FROM) {
            if (FINAL) atomicMin(label + x, g);
            else __stcg(label + x, g);
        }
        x = g;
        p = __ldcg(label + x);
    }
    return -1;
}

__global__ void k_cl_init(int nSeg, int nNode, const int* filState, int* label, int* size, int* flags, int rounds,
                          int nNet, int* out) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < nNode) {
        label[i] = (i < nSeg && filState && filState[i] < 0) ? -1 : i;
        size[i] = 0;
    }
    if (i <= rounds) flags[i] = 0;
    if (i < 2 * nNet) out[i] = 0;
}

// Joins the components of every edge, one thread an edge. The larger root takes the smaller
// one as its parent if it still is a root; otherwise another edge got there first and this
// one goes on from the two nodes' roots as they are now. A failed exchange means that a root
// has gone, so the tries of all edges together are bounded by the nodes; a thread that runs
// out of its own limit marks the labelling as not converged. The chain links go first (edges
// [0, nSeg)), then every path is flattened, then the other edges ([nSeg, ..)): a walk from a
// crosslink or a head then starts one step from its filament's root, not at the end of a chain.
__global__ void k_cl_join(int first, int nSeg, const int* e2, int nLinks, const int* linkA, const int* linkB,
                          const int* linkState, int nM, const int* boundSeg, const int* motorBackbone, int* label,
                          int* notDone) {
    int i = first + blockIdx.x * blockDim.x + threadIdx.x;
    int u = -1, v = -1;
    if (i < nSeg) {
        u = i;
        v = e2[i];
    } else if (i < nSeg + nLinks) {
        int k = i - nSeg;
        if (linkState[k] >= 0) { u = linkA[k]; v = linkB[k]; }
    } else if (i < nSeg + nLinks + nM) {
        int m = i - nSeg - nLinks;
        int s = boundSeg[m];
        if (s >= 0 && motorBackbone[m] >= 0) { u = s; v = nSeg + motorBackbone[m]; }
    }
    if (u < 0 || v < 0 || u == v || __ldcg(label + u) < 0 || __ldcg(label + v) < 0) return;
    // a chain link's larger end, still a root, can take the smaller one itself: no walk along the chain
    if (i < nSeg && atomicCAS(&label[max(u, v)], max(u, v), min(u, v)) == max(u, v)) return;
    for (int it = 0; it < OBS_MAX_FIND; it++) {
        u = find_root<0, false>(label, u);
        v = find_root<0, false>(label, v);
        if (u < 0 || v < 0) break;
        if (u == v) return;
        const int hi = u > v ? u : v, lo = u > v ? v : u;
        if (atomicCAS(&label[hi], hi, lo) == hi) return;
    }
    *notDone = 1;
}

__global__ void k_cl_flatten(int nNode, int* label) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nNode || __ldcg(label + i) < 0) return;
    const int root = find_root<SHORT_PATH, false>(label, i);
    if (root >= 0) __stcg(label + i, root);
}

// every node's label: its component's root; the component sizes in segments
__global__ void k_cl_label(int nSeg, int nNode, int* label, int* size, int* notDone) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    int root = -1;
    if (i < nNode && __ldcg(label + i) >= 0) {
        root = find_root<SHORT_PATH, true>(label, i);
        if (root >= 0) __stcg(label + i, root);
        else *notDone = 1;
    }
    if (i >= nSeg) root = -1;
    // one addition per component of a warp: most rods of a network share one component
    const unsigned same = __match_any_sync(0xffffffffu, root);
    if (root >= 0 && (int)(threadIdx.x & 31) == __ffs(same) - 1) atomicAdd(&size[root], __popc(same));
}

// out[2*net] = largest component size (segments), out[2*net+1] = active segments: blocks
// (network, part) over the network's segments, joined by integer atomics (no order)
constexpr int CL_PARTS = 16;
__global__ void __launch_bounds__(OBS_THREADS) k_cl_largest(const int* segBase, const int* label, const int* size,
                                                            int* out) {
    __shared__ int shMax[OBS_THREADS], shCnt[OBS_THREADS];
    int net = blockIdx.x / CL_PARTS, t = threadIdx.x;
    int best = 0, cnt = 0;
    for (int i = segBase[net] + (blockIdx.x % CL_PARTS) * OBS_THREADS + t; i < segBase[net + 1];
         i += CL_PARTS * OBS_THREADS) {
        int l = label[i];
        if (l < 0) continue;
        cnt++;
        int s = size[l];
        best = s > best ? s : best;
    }
    shMax[t] = best; shCnt[t] = cnt;
    for (int s = OBS_THREADS / 2; s > 0; s >>= 1) {
        __syncthreads();
        if (t < s) {
            shMax[t] = max(shMax[t], shMax[t + s]);
            shCnt[t] += shCnt[t + s];
        }
    }
    if (t == 0 && shCnt[0] > 0) {
        atomicMax(&out[2 * net], shMax[0]);
        atomicAdd(&out[2 * net + 1], shCnt[0]);
    }
}

}  // namespace

extern "C" sbx_status sbx_obs_extent(sbx_ctx* ctx, int32_t nNet, const int32_t* segBase, int32_t nSeg,
                                     const float* coord, const double* coord64, const int32_t* filState,
                                     double* out) {
    SBX_REQUIRE(ctx && nNet >= 0 && nSeg >= 0 && (nNet == 0 || (segBase && (coord || coord64) && out)));
    if (nNet == 0) return SBX_OK;
    SBX_LAUNCH(ctx, k_extent, nNet * OBS_CTAS, 32 * OBS_WARPS, nSeg, segBase, coord, coord64, filState, out);
    return check_launch(ctx, "sbx_obs_extent");
}

extern "C" sbx_status sbx_obs_stress(sbx_ctx* ctx, int32_t nNet, int32_t nSeg, const float* coord, const float* uVec,
                                     const float* end1, const float* segLength, const int32_t* linkBase,
                                     const int32_t* linkFilA, const int32_t* linkFilB, const int32_t* linkState,
                                     const float* loc1, const float* loc2, const float* xlinkData, int32_t nMotors,
                                     const int32_t* motBase, const float* motCoord, const float* motUVec,
                                     const int32_t* boundSeg, const float* bindArc, const float* bondData,
                                     double headLen, const float* volume, double* out) {
    SBX_REQUIRE(ctx && nNet >= 0 && nSeg >= 0 && nMotors >= 0);
    if (nNet == 0) return SBX_OK;
    SBX_REQUIRE(coord && uVec && end1 && segLength && volume && out &&
                (!linkBase || (linkFilA && linkFilB && linkState && loc1 && loc2 && xlinkData)) &&
                (!motBase || (motCoord && motUVec && boundSeg && bindArc && bondData)));
    SBX_LAUNCH(ctx, k_stress, nNet * OBS_CTAS, 32 * OBS_WARPS, nSeg, coord, uVec, end1, segLength, linkBase, linkFilA, linkFilB,
               linkState, loc1, loc2, xlinkData, 3 * nMotors, motBase, motCoord, motUVec, boundSeg, bindArc, bondData,
               headLen, volume, out);
    return check_launch(ctx, "sbx_obs_stress");
}

extern "C" sbx_status sbx_obs_clusters(sbx_ctx* ctx, int32_t nNet, const int32_t* segBase, int32_t nSeg,
                                       const int32_t* filState, const int32_t* end2NbrSlot, int32_t nLinks,
                                       const int32_t* linkFilA, const int32_t* linkFilB, const int32_t* linkState,
                                       int32_t nMotors, const int32_t* boundSeg, const int32_t* motorBackbone,
                                       int32_t nBackbones, int32_t rounds, int32_t* label, int32_t* size,
                                       int32_t* flags, int32_t* out) {
    SBX_REQUIRE(ctx && nNet >= 0 && nSeg >= 0 && nLinks >= 0 && nMotors >= 0 && nBackbones >= 0 && rounds >= 1);
    if (nNet == 0) return SBX_OK;
    SBX_REQUIRE(segBase && end2NbrSlot && label && size && flags && out && (nLinks == 0 || (linkFilA && linkFilB &&
                linkState)) && (nMotors == 0 || (boundSeg && motorBackbone)));
    int nNode = nSeg + nBackbones;
    int nInit = nNode > rounds + 1 ? nNode : rounds + 1;
    if (nInit < 2 * nNet) nInit = 2 * nNet;
    SBX_LAUNCH(ctx, k_cl_init, blocks(nInit), 256, nSeg, nNode, filState, label, size, flags, rounds, nNet, out);
    SBX_LAUNCH(ctx, k_cl_join, blocks(nSeg), 256, 0, nSeg, end2NbrSlot, 0, linkFilA, linkFilB, linkState, 0, boundSeg,
               motorBackbone, label, flags + (rounds - 1));
    if (nLinks + nMotors > 0) {
        SBX_LAUNCH(ctx, k_cl_flatten, blocks(nNode), 256, nNode, label);
        SBX_LAUNCH(ctx, k_cl_join, blocks((int64_t)nLinks + nMotors), 256, nSeg, nSeg, end2NbrSlot, nLinks, linkFilA,
                   linkFilB, linkState, nMotors, boundSeg, motorBackbone, label, flags + (rounds - 1));
    }
    SBX_LAUNCH(ctx, k_cl_label, blocks(nNode), 256, nSeg, nNode, label, size,
               flags + (rounds - 1));
    SBX_LAUNCH(ctx, k_cl_largest, nNet * CL_PARTS, OBS_THREADS, segBase, label, size, out);
    return check_launch(ctx, "sbx_obs_clusters");
}
