// sbx_wide.cu — the dense contractile step (DenseContractileHarness.cpuStep,
// DenseContractileHarness.java:350-429) as fourteen wide kernels, single or packed networks.
//
//   main stream                                      ahead          link               csr
//   publish: body view, release, cells, row slots    draws          rows, unbinding
//   scan: cell offsets                               myosin terms   scan
//   place: contents, endpoints in cell order         joints         forces, lists
//   bind: reach, nearest, cycle
//   mini: one block a minifilament <- all ahead, links                                 scan
//   rods: gathers, walls, integration                                                  lists
//
// At the small sizes a step is a chain of latencies, so a kernel with one predecessor starts
// before that one is done (programmatic dependent launch): it reads and computes what it does not
// take from it, then waits (after_previous). A kernel lets the next start after its own wait
// (let_next_start), so that whatever comes before the predecessor is complete by then. mini has
// several predecessors and waits for all of them at its launch; rods then has one, and does the
// chain and the links while the minifilaments are computed.
// The per-system sequence (sbx_dense.cu: dense_sequence) takes 53 launches: five counting sorts
// of five kernels and many kernels of 3-5 us each, in a row. Here the inverse maps are made as
// the fused kernel makes them (fixed slots per row filled by atomics, placed by rank), what
// needs only the step's start view runs beside the grid, a minifilament is one block's work, and
// what a later kernel reads again is written once.
// Every slot is computed by the same device functions as the per-system kernels, in the
// reference's accumulation order: the same bits.
// A step takes 26 us at 1,000 rods, 35 at 20,000, 75 at 100,000 and 325 at 500,000 (46, 57, 97 and
// 370 with full waits, serial gathers and fewer warps; 200 and 434 at the last two as the
// per-system sequence), a packed step of 12 networks (0.17e6 rods, 0.18e6 heads) 219 us (269; 366).
#include <cuda_runtime.h>

#include <algorithm>

#include "../../include/softbox_b200.h"
#include "sbx_scan.cuh"
#include "sbx_step.cuh"
#include "sbx_trace.h"
#include "sbx_wide.cuh"

namespace {

// network and local index of an item in packed networks (a single network: 0 and the index)
template <bool B>
__device__ __forceinline__ int2 key_of(const int* key, int i) {
    return B ? make_int2(key[2 * i], key[2 * i + 1]) : make_int2(0, i);
}

template <bool B>
__device__ __forceinline__ GridView grid_view(const WideArgs& w, int net) {
    const sbx_grid_state& g = w.a.sc.grid;
    if (B) {
        const int* gd = w.bt.gridDims + 4 * net;
        return GridView{w.bt.gridParams + 6 * net, gd[0], gd[1], gd[2], w.a.segCellOff + gd[3]};
    }
    return GridView{g.gridParams, g.gridDims[0], g.gridDims[1], g.gridDims[2], w.a.segCellOff};
}

// the cell of a centre in its network's grid
template <bool B>
__device__ __forceinline__ int body_cell(const WideArgs& w, int net, const float c[3]) {
    const GridView v = grid_view<B>(w, net);
    return (int)(v.off - w.a.segCellOff) + cell_coord(c[0], v.gp[0], v.gp[4], v.nX) +
           cell_coord(c[1], v.gp[1], v.gp[4], v.nY) * v.nX + cell_coord(c[2], v.gp[2], v.gp[4], v.nZ) * (v.nX * v.nY);
}

// the kernel before this one in its stream is complete, and what it wrote can be read
__device__ __forceinline__ void after_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// the next kernel of the stream may start its blocks once every block is here or done
__device__ __forceinline__ void let_next_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

__device__ __forceinline__ void prefetch_l1(const void* p) { asm volatile("prefetch.global.L1 [%0];" ::"l"(p)); }

struct AfterPrevious {
    __device__ __forceinline__ void operator()() const { after_previous(); }
};

// a link end names a rod; one at or past the rod count is left out and reported
__device__ __forceinline__ bool end_ok(const WideArgs& w, int s) {
    if (s < 0) return false;
    if (SBX_IDX_OK(s, w.a.nSeg, CK_LINK_END) && s < w.a.nSeg) return true;
    if (w.errDev) *(volatile int*)w.errDev = 1;
    return false;
}

// one addition per distinct tile of a warp: tile sums[tile] += the warp's items of that tile
__device__ __forceinline__ void tile_add(int* sums, int tile) {
    const unsigned same = __match_any_sync(0xffffffffu, tile);
    if (tile >= 0 && (int)(threadIdx.x & 31) == __ffs(same) - 1)
        atomicAdd(&sums[tile * WIDE_SUM_STRIDE], __popc(same));
}

// ---------------------------------------------------------------- ahead: draws and joints
// What depends only on the step's start poses and the step index. The Brownian forces of every
// body (BrownianForceSystem.java:44-106), one body a thread: its three Box-Muller pairs are
// independent chains of FP64 operations.
template <bool B>
__global__ void __launch_bounds__(256) k_wide_draws(const __grid_constant__ WideArgs w) {
    let_next_start();
    const FusedArgs& a = w.a;
    const sbx_dense_scene& sc = a.sc;
    const int nB = a.nB, nBb = a.nBb;
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= nB + nBb + a.nSeg) return;
    const int t = *a.d_step;
    if (j == 0 && sc.mot.publishParams[0] != a.nSeg && w.errDev) *(volatile int*)w.errDev = ERR_DEV_VIEW;
    const WideNoise nz = *w.noise;
    if (j == 0 && nz.fil && nz.err && (t < nz.t0 || t >= nz.t0 + nz.n)) atomicOr(nz.err, 1);
    const sbx_rigid_body* b;
    const float* noise;
    int i, key, seed;
    float mag;
    if (j < nB) {
        b = &sc.mot.body;
        i = j;
        const int m = j / 3;
        const int2 k = key_of<B>(w.bt.motKey, m);
        key = 3 * k.y + (j - 3 * m);
        seed = B ? w.bt.seeds[3 * k.x] : sc.seed;
        mag = sc.mot.bodyParams[1];
        noise = nz.mot;
    } else if (j < nB + nBb) {
        b = &sc.mini.backbone;
        i = j - nB;
        const int2 k = key_of<B>(w.bt.bbKey, i);
        key = k.y;
        seed = B ? w.bt.seeds[3 * k.x + 1] : sc.seedBb;
        mag = sc.mini.bbBodyParams[1];
        noise = nz.bb;
    } else {
        b = &sc.fil.body;
        i = j - nB - nBb;
        const int2 k = key_of<B>(w.bt.segKey, i);
        key = k.y;
        seed = B ? w.bt.seeds[3 * k.x + 2] : sc.fil.counts[2];
        mag = sc.fil.params[1];
        noise = nz.fil;
    }
    const int n = b->n;
    float g[6];
    if (noise) {
        const int s = t - nz.t0;
        const bool in = s >= 0 && s < nz.n;
        const float* q = noise + (int64_t)(in ? s : 0) * 6 * n + i;
        for (int k = 0; k < 6; k++) g[k] = in ? q[(int64_t)k * n] : 0.f;
    } else {
        gauss6_wang(key, t, seed, g);
    }
    float gT[3], gR[3], rf[3], rt[3];
    for (int k = 0; k < 3; k++) { gT[k] = b->bTransGam[k * n + i]; gR[k] = b->bRotGam[k * n + i]; }
    brownian_amplitudes(g, b->brownTransScale[i], b->brownRotScale[i], mag, gT, gR, rf, rt);
    for (int k = 0; k < 3; k++) { b->randForce[k * n + i] = rf[k]; b->randTorque[k * n + i] = rt[k]; }
}

// the chain joints, each by its lower-slot rod (as k_chain); the latency of the FP64 chains is
// hidden by warps: 64 registers, eight blocks an SM
__global__ void __launch_bounds__(128, 8) k_wide_joints(const __grid_constant__ WideArgs w) {
    const FusedArgs& a = w.a;
    const sbx_filament_store& fs = a.sc.fil;
    const sbx_rigid_body& fb = fs.body;
    const int n = a.nSeg, i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int s2 = fs.end2NbrSlot[i], s1 = fs.end1NbrSlot[i];
    if (!SBX_IDX_OK_OR_NONE(s2, n, CK_NEIGHBOUR)) s2 = -1;
    if (!SBX_IDX_OK_OR_NONE(s1, n, CK_NEIGHBOUR)) s1 = -1;
    const ChainParams cp = chain_params(fs.chainParams);
    for (int side = 0; side < 2; side++) {
        const int nb = side == 0 ? s2 : s1;
        if (nb <= i) continue;
        joint_store(a, i, side,
                    chain_joint(cp, i, side, nb, side == 0 ? fs.end2NbrSide[i] : fs.end1NbrSide[i],
                                load_rod(n, i, fb.coord, fb.uVec, fb.segLength, fb.bTransGam, fb.bRotGam),
                                load_rod(n, nb, fb.coord, fb.uVec, fb.segLength, fb.bTransGam, fb.bRotGam)));
    }
    after_previous();                    // (done when the kernels before it are)
}

// ---------------------------------------------------------------- publish
// The body view, the release of the heads, the cells with their row slots and tile sums, the
// largest reach of a segment from its centre, the start view's orientations
// (the rods kernel reads a neighbour from the start view: its own block may have stepped it
// already) and the step's counts.
// (MORE: the view has room for bodies of the caller's)
template <bool B, bool MORE>
__global__ void __launch_bounds__(256) k_wide_publish(const __grid_constant__ WideArgs w) {
    let_next_start();
    const FusedArgs& a = w.a;
    const sbx_dense_scene& sc = a.sc;
    const sbx_grid_state& g = sc.grid;
    const int nSeg = a.nSeg, nM = a.nM, nB = a.nB, cap = a.cap;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0) {
        const int t = *a.d_step;
        int* mc = sc.mot.counts; mc[0] = nM; mc[1] = t; mc[2] = sc.seed; mc[3] = nSeg;
        int* bc = sc.mini.bbCounts; bc[0] = a.nBb; bc[1] = t; bc[2] = sc.seedBb; bc[3] = a.nBb;
        sc.fil.counts[1] = t;
        if (a.xlOn) { sc.xl.counts[1] = t; sc.xl.counts[2] = sc.seed; }
    }
    int cell = -1;
    float span = 0.f;
    if (i < nSeg + nM) {
        float c[3];
        int net;
        if (i < nSeg) {
            const sbx_rigid_body& fb = sc.fil.body;
            const int* state = sc.fil.filState;              // FREE (< 0) slots of turnover, or none
            // (all loads before the first store: nothing tells the compiler that they differ)
            float u[3], e1[3], e2[3];
            for (int k = 0; k < 3; k++) {
                c[k] = fb.coord[k * nSeg + i];
                u[k] = fb.uVec[k * nSeg + i];
                e1[k] = fb.end1[k * nSeg + i];
                e2[k] = fb.end2[k * nSeg + i];
            }
            const float r = 0.5f * fb.segLength[i] + g.viewParams[0];
            const int owner = (state && state[i] < 0) ? STORE_NONE : STORE_FILAMENT;
            net = key_of<B>(w.bt.segKey, i).x;
            if (owner == STORE_FILAMENT) span = segment_span(c, e1, e2);
            for (int k = 0; k < 3; k++) a.uSnap[k * nSeg + i] = u[k];
            g.boundingRadius[i] = r;
            g.ownerStore[i] = owner;
            g.ownerSlot[i] = i;
            // the motor rows of the previous step were last read by its rods and motor CSR kernels
            a.headM[i] = -1;
            a.cntM[i] = 0;
        } else {
            const sbx_rigid_body& mb = sc.mot.body;
            const int m = i - nSeg, h = 3 * m + 2, r = 3 * m;
            const float hl = mb.segLength[h], reach = sc.mot.reach[m];
            float u[3], ru[3];
            for (int k = 0; k < 3; k++) {
                u[k] = mb.uVec[k * nB + h];
                ru[k] = mb.uVec[k * nB + r];
                c[k] = mb.coord[k * nB + h] + 0.5f * hl * u[k];
            }
            // the catch-slip release and cooldown (NucleotideCycleSystem.java:77-134): previous step's
            // forces only
            const sbx_motor_store& mot = sc.mot;
            const int2 key = key_of<B>(w.bt.motKey, m);
            int bs = mot.boundSeg[m], cd = mot.cooldown[m], sb = mot.stats[2 * m], sr = mot.stats[2 * m + 1],
                cs = mot.capStats[m];
            const float dot = mot.forceDotFil[m], mag = mot.forceMag[m];
            net = key.x;
            for (int k = 0; k < 3; k++) {
                sc.mot.head[k * nM + m] = c[k];
                sc.mot.uVec[k * nM + m] = u[k];
                sc.mot.rodUVec[k * nM + m] = ru[k];
            }
            g.boundingRadius[i] = reach;
            g.ownerStore[i] = STORE_MOTOR;
            g.ownerSlot[i] = m;
            release_one(key.y, bs, cd, sb, sr, cs, dot, mag, mot.kinParams, *a.d_step, B ? w.bt.seeds[3 * key.x] : sc.seed);
            mot.boundSeg[m] = bs; mot.cooldown[m] = cd; mot.stats[2 * m] = sb; mot.stats[2 * m + 1] = sr;
            mot.capStats[m] = cs;
        }
        for (int k = 0; k < 3; k++) g.center[k * cap + i] = c[k];
        if (i < g.gridCounts[1]) cell = body_cell<B>(w, net, c);
    } else if (MORE && !B && i < cap && i < g.gridCounts[1]) {
        // a body of the caller's beyond the published ones (counted in after the plan was made)
        const float c[3] = {g.center[i], g.center[cap + i], g.center[2 * cap + i]};
        cell = body_cell<B>(w, 0, c);
        if (g.ownerStore[i] == STORE_FILAMENT && w.errDev) *(volatile int*)w.errDev = ERR_DEV_VIEW;
    }
    if (i < cap) g.bodyCell[i] = cell;
    int over = 0;
    if (cell >= 0) {
        if (i < nSeg) atomicAdd(&a.cntSeg[cell], 1);
        over = row_insert(a.cntCell, a.cellSlot, WIDE_CELL_SLOTS, a.cellUse, a.cellHead, a.cellNext, cell, i);
    }
    __syncwarp();
    const int tile = cell >= 0 ? cell / WIDE_TILE : -1;
    tile_add(w.sumCell, tile);
    tile_add(w.sumSeg, i < nSeg ? tile : -1);
    span_max(a.reachMax, span);
    stat_add(a, ST_CELL_LIST, over);
}

// ---------------------------------------------------------------- link rows
// One link a thread: its entries in the rows of its two rods, the Bell unbinding
// (CrosslinkerSystem.java:727-756) and the active counts (:694-708)
template <bool B>
__global__ void __launch_bounds__(128) k_wide_link_rows(const __grid_constant__ WideArgs w) {
    let_next_start();
    const FusedArgs& a = w.a;
    const sbx_dense_scene& sc = a.sc;
    const sbx_crosslinker_store& xl = sc.xl;
    const sbx_rigid_body& fb = sc.fil.body;
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    int la = -1, lb = -1, over = 0;
    bool act = false;
    if (k < a.nL) {
        la = xl.linkFilA[k];
        lb = xl.linkFilB[k];
        const bool on = xl.linkState[k] >= 0;
        if (!end_ok(w, la)) la = -1;
        if (!end_ok(w, lb)) lb = -1;
        // (the two counters and the unbinding's inputs are in flight together)
        int jA = 0, jB = 0;
        if (la >= 0) jA = atomicAdd(&a.cntA[la], 1);
        if (lb >= 0) jB = atomicAdd(&a.cntB[lb], 1);
        act = la >= 0 && lb >= 0 && on;
        if (act && a.xlUnbind) {
            const int2 key = key_of<B>(w.bt.linkKey, k);
            // the draw is keyed by the local index, which also indexes the strain ring: shift the
            // ring pointers so that it addresses this link's own ring
            const int off = k - key.y;
            if (unbind_one(key.y, a.nSeg, fb.uVec, fb.end1, la, lb, xl.loc1[k], xl.loc2[k],
                           xl.strainHist + (int64_t)off * STRAIN_WIN, xl.strainPlace + off, xl.offParams, *a.d_step,
                           B ? w.bt.seeds[3 * key.x] : sc.seed)) {
                xl.linkState[k] = LINK_FREE;
                act = false;
            }
        }
        if (la >= 0) over += row_put(a.slotA, WIDE_ROW_SLOTS, a.rowUse, a.headA, a.nextA, la, k, jA);
        if (lb >= 0) over += row_put(a.slotB, WIDE_ROW_SLOTS, a.rowUse, a.headB, a.nextB, lb, k, jB);
    }
    __syncwarp();
    tile_add(w.sumA, la >= 0 ? la / WIDE_TILE : -1);
    tile_add(w.sumB, lb >= 0 ? lb / WIDE_TILE : -1);
    stat_add(a, ST_LINK_LIST, over);
    if (!act) return;
    atomicAdd(&a.cntAct[la], 1);
    atomicAdd(&a.cntAct[lb], 1);
}

// ---------------------------------------------------------------- scans
// Exclusive scan of one tile of a histogram into out, with the tile sums made by the kernel that
// filled it: a block adds the sums before its tile and scans the tile through shared memory.
// copy (optional) gets the row lengths, chunkOut (optional) the prefix of every SCAN_CHUNK rows;
// the histogram is left at zero for the next step.
__device__ void scan_one_tile(int tile, int tiles, int* cnt, int n, const int* sums, int* out, int* copy, int clampTotal,
                              int* chunkOut, bool keep) {
    __shared__ int sv[WIDE_TILE + WIDE_TILE / 32];
    static_assert(WIDE_TILE == SCAN_TILE_ROWS, "the scan's tile");
    const int base = tile * WIDE_TILE;
    int v[TILE_PER_THREAD], s = 0;
#pragma unroll
    for (int k = 0; k < TILE_PER_THREAD; k++) {
        const int g = base + threadIdx.x + 256 * k;
        v[k] = g < n ? cnt[g] : 0;
    }
    int p = 0;
    for (int k = threadIdx.x; k < tile; k += 256) p += sums[k * WIDE_SUM_STRIDE];
    int prefix;
    block_exclusive_scan<256>(p, &prefix);
#pragma unroll
    for (int k = 0; k < TILE_PER_THREAD; k++) {
        const int r = threadIdx.x + 256 * k, g = base + r;
        sv[tile_slot(r)] = v[k];
        if (g < n) {
            if (copy) copy[g] = v[k];
            if (!keep) cnt[g] = 0;
        }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < TILE_PER_THREAD; k++) {
        v[k] = sv[tile_slot(TILE_PER_THREAD * threadIdx.x + k)];
        s += v[k];
    }
    int tot;
    int run = block_exclusive_scan<256>(s, &tot);
#pragma unroll
    for (int k = 0; k < TILE_PER_THREAD; k++) {
        sv[tile_slot(TILE_PER_THREAD * threadIdx.x + k)] = run;
        run += v[k];
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < TILE_PER_THREAD; k++) {
        const int r = threadIdx.x + 256 * k, g = base + r;
        if (g < n) out[g] = prefix + sv[tile_slot(r)];
    }
    if (chunkOut && threadIdx.x < WIDE_TILE / SCAN_CHUNK) {
        const int c = tile * (WIDE_TILE / SCAN_CHUNK) + threadIdx.x;
        if (c < (n + SCAN_CHUNK - 1) / SCAN_CHUNK) chunkOut[c] = prefix + sv[tile_slot(threadIdx.x * SCAN_CHUNK)];
    }
    if (tile == tiles - 1 && threadIdx.x == 0) {
        const int total = prefix + tot;
        out[n] = total < clampTotal ? total : clampTotal;
        if (chunkOut) chunkOut[(n + SCAN_CHUNK - 1) / SCAN_CHUNK] = total;
    }
}

__global__ void __launch_bounds__(256) k_wide_cell_scan(const __grid_constant__ WideArgs w) {
    after_previous();
    let_next_start();
    const FusedArgs& a = w.a;
    const sbx_grid_state& g = a.sc.grid;
    const int b = blockIdx.x;
    if (b < w.tilesC)
        scan_one_tile(b, w.tilesC, a.cntCell, a.C, w.sumCell, g.gridCellOffsets, g.cellCount, a.cap, g.chunkSum, true);
    else
        scan_one_tile(b - w.tilesC, w.tilesC, a.cntSeg, a.C, w.sumSeg, a.segCellOff, nullptr, a.nSeg, nullptr, false);
}

__global__ void __launch_bounds__(256) k_wide_link_scan(const __grid_constant__ WideArgs w) {
    after_previous();
    let_next_start();
    const FusedArgs& a = w.a;
    const sbx_crosslinker_store& xl = a.sc.xl;
    const int b = blockIdx.x;
    if (b < w.tilesS)
        scan_one_tile(b, w.tilesS, a.cntA, a.nSeg, w.sumA, xl.segOffsetsA, xl.segCountA, a.nL, nullptr, true);
    else
        scan_one_tile(b - w.tilesS, w.tilesS, a.cntB, a.nSeg, w.sumB, xl.segOffsetsB, xl.segCountB, a.nL, nullptr, true);
}

// ---------------------------------------------------------------- place
// Each body at its rank in its cell: the serial scatter's position. The segments' endpoints go
// into cell order for the reach walk (segments precede heads within a cell, so a segment's
// rank in its cell is its rank among the cell's segments). Only the offsets come from the scan:
// the rest is read before it is done.
__global__ void __launch_bounds__(256) k_wide_place(const __grid_constant__ WideArgs w) {
    const FusedArgs& a = w.a;
    const sbx_grid_state& g = a.sc.grid;
    const sbx_rigid_body& fb = a.sc.fil.body;
    const int nSeg = a.nSeg;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    int c = i < a.cap ? g.bodyCell[i] : -1;
    if (!SBX_IDX_OK_OR_NONE(c, a.C, CK_CELL)) c = -1;
    const bool seg = i < nSeg;
    int rank = 0;
    float4 e1 = make_float4(0.f, 0.f, 0.f, __int_as_float(-1)), e2 = make_float4(0.f, 0.f, 0.f, 0.f);
    if (c >= 0) {
        if (seg && g.ownerStore[i] == STORE_FILAMENT) {
            e1 = make_float4(fb.end1[i], fb.end1[nSeg + i], fb.end1[2 * nSeg + i], __int_as_float(i));
            e2 = make_float4(fb.end2[i], fb.end2[nSeg + i], fb.end2[2 * nSeg + i], 0.f);
        }
        rank = row_rank<WIDE_CELL_SLOTS>(a, a.cntCell, a.cellSlot, a.cellUse, a.cellHead, a.cellNext, c, i, a.cap);
    }
    after_previous();
    let_next_start();
    if (c < 0) return;
    const int pos = g.gridCellOffsets[c] + rank, q = seg ? a.segCellOff[c] + rank : 0;
    if (!SBX_IDX_OK(pos, a.cap, CK_CSR_POS)) return;
    g.gridCellContents[pos] = i;
    if (seg && SBX_IDX_OK(q, nSeg, CK_CSR_POS)) {
        a.segE1[q] = e1;
        a.segE2[q] = e2;
    }
}

// ---------------------------------------------------------------- bind
constexpr int BIND_LANES = 8;        // lanes a head
// The reach walk with the nearest choice, the nucleotide cycle and the bound head's entry in its
// rod's motor row: a warp takes 32 / BIND_LANES consecutive heads. (64 registers here and in the
// terms: 222 us a packed step of 12 networks, 228 with 68 and 76.)
constexpr int BIND_HEADS = 32 / BIND_LANES;
template <bool B>
__global__ void __launch_bounds__(128, 8) k_wide_bind(const __grid_constant__ WideArgs w) {
    const FusedArgs& a = w.a;
    const sbx_dense_scene& sc = a.sc;
    const sbx_motor_store& mot = sc.mot;
    const float* kp = mot.kinParams;
    const int lane = threadIdx.x & 31, nM = a.nM;
    const int base = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * BIND_HEADS;
    if (base >= nM) { after_previous(); return; }
    const int m = base + lane / BIND_LANES;
    const bool valid = m < nM, mine = valid && (lane & (BIND_LANES - 1)) == 0;
    const int mm = valid ? m : base;
    const int2 key = key_of<B>(w.bt.motKey, mm);
    const float mx = mot.head[mm], my = mot.head[nM + mm], mz = mot.head[2 * nM + mm];
    const float ux = mot.uVec[mm], uy = mot.uVec[nM + mm], uz = mot.uVec[2 * nM + mm];
    const float rx = mot.rodUVec[mm], ry = mot.rodUVec[nM + mm], rz = mot.rodUVec[2 * nM + mm];
    int bs = mot.boundSeg[mm], state = mot.nucleotideState[mm];
    int best;
    float arc;
    const int rc = group_reach_bind<BIND_LANES>(
        a, grid_view<B>(w, key.x), lane, valid, mx, my, mz, ux, uy, uz, rx, ry, rz,
        sc.grid.reachSeg + (int64_t)mm * MAX_CAND, kp[7], kp[8], &best, &arc, AfterPrevious());
    int row = -1, over = 0;
    if (mine) {
        sc.grid.reachCount[m] = rc;
        if (rc > MAX_CAND) {
            atomicOr(a.err, ERR_REACH_OVERFLOW);
            stat_add(a, ST_REACH_OVER, 1);
        }
        if (bs == FREE_BINDABLE && best >= 0) {
            bs = best;
            mot.boundSeg[m] = bs;
            mot.bindArc[m] = arc;
        }
        mot.nucleotideState[m] = cycle_one(key.y, state, bs >= 0, mot.forceDotHist + 10 * m, mot.nucParams,
                                           mot.counts[1], B ? w.bt.seeds[3 * key.x] : sc.seed);
        if (bs >= 0 && SBX_IDX_OK(bs, a.nSeg, CK_BOUND_SEG) && bs < a.nSeg) {
            row = bs;
            over = row_insert(a.cntM, a.slotM, FUSED_MOTOR_SLOTS, a.mRowUse, a.headM, a.nextM, bs, m);
        } else if (bs >= 0 && w.errDev) {
            *(volatile int*)w.errDev = 1;
        }
    }
    __syncwarp();
    tile_add(w.sumM, row >= 0 ? row / WIDE_TILE : -1);
    stat_add(a, ST_MOTOR_LIST, over);
}

// ---------------------------------------------------------------- terms and mini
// The position-only myosin terms, one a thread, beside the grid kernels: FP64 chains of some
// thousand cycles that would otherwise sit between binding and integration.
__global__ void __launch_bounds__(128, 8) k_wide_terms(const __grid_constant__ WideArgs w) {
    let_next_start();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < 2 * w.a.nM + 4 * w.a.nD && !myosin_term<true>(w.a, k) && w.errDev) *(volatile int*)w.errDev = ERR_DEV_VIEW;
    after_previous();                    // (done when the kernels before it are)
}

// One block a minifilament: a warp for its heads (with their bonds), its rods, its levers, then
// the integration of its sub-bodies in body order. The backbones, one a thread, take the
// blocks after them. A block waits for memory twice (terms, then bodies), so blocks in flight
// count for more than registers: at ten an SM (64 registers, 150 bytes spilled) a step of
// 500,000 rods takes 337 us, at seven (88 registers) 355; a packed step of 12 networks 228 and
// 250. (Twelve an SM gave the same as ten; prefetching the bodies to L1 was slower.)
constexpr int MINI_THREADS = 96;
template <bool B>
__global__ void __launch_bounds__(MINI_THREADS, 10) k_wide_mini(const __grid_constant__ WideArgs w) {
    let_next_start();
    __shared__ MiniSmem sm;
    const FusedArgs& a = w.a;
    const sbx_minifilament_store& mini = a.sc.mini;
    if ((int)blockIdx.x < a.nBb) {
        mini_bodies<true>(a, sm, blockIdx.x);
        return;
    }
    const int u = (blockIdx.x - a.nBb) * MINI_THREADS + threadIdx.x;
    if (u >= a.nBb) return;
    mini_backbone<true>(a, u, mini.bbCounts[1], B ? w.bt.boxParams + 8 * w.bt.bbKey[2 * u] : a.sc.boxParams,
                  B ? mini.bbBodyParams[0] : a.sc.boxParams[7]);
}

// ---------------------------------------------------------------- links
// how many of the slots v, the first of them slot q of n, hold items below k
__device__ __forceinline__ int below(int4 v, int q, int n, int k) {
    return (q < n && v.x < k) + (q + 1 < n && v.y < k) + (q + 2 < n && v.z < k) + (q + 3 < n && v.w < k);
}

// Crosslinker forces and torsion (CrosslinkerSystem.java:61-123, :777-806), one thread a link,
// and the link at its rank in both CSRs: the lists, and its two payload rows in list order
// (zeros for a FREE link). The minifilaments wait for it, and it is a chain of latencies: with
// the loads of each round together, and the rank from a row's slots (a row of nine links was a
// list walked entry by entry), it takes 10 us at 20,000 rods (13 before) and ends 5 us earlier.
__global__ void __launch_bounds__(128) k_wide_links(const __grid_constant__ WideArgs w) {
    const FusedArgs& a = w.a;
    const sbx_crosslinker_store& xl = a.sc.xl;
    const sbx_rigid_body& fb = a.sc.fil.body;
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= a.nL) { after_previous(); return; }
    // two rounds of loads, each in flight together: what the link's index names, then what its
    // ends name (row 0 stands in for an end that is left out)
    int la = xl.linkFilA[k], lb = xl.linkFilB[k];
    const int state = xl.linkState[k], orient = xl.linkOrientSame[k];
    const float loc1 = xl.loc1[k], loc2 = xl.loc2[k];
    const bool torsion = xl.torsionParams[1] >= 0.5f;
    TorsionWindow win;
    if (torsion) win = torsion_window(k, xl.torqueMagHist, xl.torqueMagPlace);
    if (!end_ok(w, la)) la = -1;
    if (!end_ok(w, lb)) lb = -1;
    const int ia = la < 0 ? 0 : la, ib = lb < 0 ? 0 : lb;
    const LinkEnd ea = link_end(ia, a.nSeg, fb.coord, fb.uVec, fb.end1, fb.bTransGam, a.cntAct);
    const LinkEnd eb = link_end(ib, a.nSeg, fb.coord, fb.uVec, fb.end1, fb.bTransGam, a.cntAct);
    const int nA = a.cntA[ia], nB = a.cntB[ib];
    const int4* sA = reinterpret_cast<const int4*>(a.slotA + (size_t)ia * WIDE_ROW_SLOTS);
    const int4* sB = reinterpret_cast<const int4*>(a.slotB + (size_t)ib * WIDE_ROW_SLOTS);
    const int4 vA = sA[0], vB = sB[0];
    int pA = below(vA, 0, min(nA, a.rowUse), k), pB = below(vB, 0, min(nB, a.rowUse), k);
    float out[XL_STRIDE];
#pragma unroll
    for (int j = 0; j < XL_STRIDE; j++) out[j] = 0.f;
    if (la >= 0 && lb >= 0) {
        link_forces(ea, eb, loc1, loc2, xl.xlParams, out);
        if (torsion)
            link_torsion_row(k, a.nSeg, fb.uVec, la, lb, state, orient, win, xl.torqueMagHist, xl.torqueMagPlace, out,
                             xl.torsionParams[0]);
    }
    for (int q = 1; q < WIDE_ROW_SLOTS / 4; q++) {
        if (nA > 4 * q) pA += below(sA[q], 4 * q, min(nA, a.rowUse), k);
        if (nB > 4 * q) pB += below(sB[q], 4 * q, min(nB, a.rowUse), k);
    }
    if (la >= 0 && nA > a.rowUse) pA += list_rank(a, a.headA[la], a.nextA, k, a.nL);
    if (lb >= 0 && nB > a.rowUse) pB += list_rank(a, a.headB[lb], a.nextB, k, a.nL);
    after_previous();                    // the offsets
    pA = la >= 0 ? pA + xl.segOffsetsA[la] : -1;
    pB = lb >= 0 ? pB + xl.segOffsetsB[lb] : -1;
    // (a row is 48 bytes: 16-byte stores where the array is aligned)
    float* row = xl.xlinkData + (int64_t)k * XL_STRIDE;
    if (((uintptr_t)xl.xlinkData & 15u) == 0)
        for (int j = 0; j < 3; j++)
            reinterpret_cast<float4*>(row)[j] = make_float4(out[4 * j], out[4 * j + 1], out[4 * j + 2], out[4 * j + 3]);
    else
        for (int j = 0; j < XL_STRIDE; j++) row[j] = out[j];
    if (pA >= 0) xl.segIdxA[pA] = k;
    if (pB >= 0) xl.segIdxB[pB] = k;
    const bool on = state >= 0;
    float2* oA = reinterpret_cast<float2*>(w.payA + 6 * (int64_t)(pA < 0 ? 0 : pA));
    float2* oB = reinterpret_cast<float2*>(w.payB + 6 * (int64_t)(pB < 0 ? 0 : pB));
    for (int j = 0; j < 3; j++) {
        if (pA >= 0) oA[j] = on ? make_float2(out[2 * j], out[2 * j + 1]) : make_float2(0.f, 0.f);
        if (pB >= 0) oB[j] = on ? make_float2(out[6 + 2 * j], out[7 + 2 * j]) : make_float2(0.f, 0.f);
    }
}

// ---------------------------------------------------------------- motor CSR
// The reference's motor CSR arrays (CrossBridgeSystem.java:190-217), outputs of the step that
// the rods kernel does not wait for (it reads the row slots; the row lengths stay in cntM)
__global__ void __launch_bounds__(256) k_wide_motor_scan(const __grid_constant__ WideArgs w) {
    const FusedArgs& a = w.a;
    scan_one_tile(blockIdx.x, w.tilesS, a.cntM, a.nSeg, w.sumM, a.sc.segMotorOffsets, a.sc.segMotorCount, a.nM, nullptr,
                  true);
}

// the motors at their ranks; the overflow lists' heads of the cells (last read by the place
// kernel) and every scan's tile sums are emptied for the next step, which begins after this
__global__ void __launch_bounds__(256) k_wide_motor_place(const __grid_constant__ WideArgs w) {
    const FusedArgs& a = w.a;
    const sbx_dense_scene& sc = a.sc;
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m < a.C) { a.cntCell[m] = 0; a.cellHead[m] = -1; }
    if (m < w.tilesC) { w.sumCell[m * WIDE_SUM_STRIDE] = 0; w.sumSeg[m * WIDE_SUM_STRIDE] = 0; }
    if (m < w.tilesS) w.sumM[m * WIDE_SUM_STRIDE] = 0;
    if (m >= a.nM) return;
    const int bs = sc.mot.boundSeg[m];
    if (bs < 0 || bs >= a.nSeg) return;
    const int pos = sc.segMotorOffsets[bs] + row_rank<FUSED_MOTOR_SLOTS>(a, a.cntM, a.slotM, a.mRowUse, a.headM,
                                                                         a.nextM, bs, m, a.nM);
    if (pos < a.nM) sc.segMotorMyo[pos] = m;
}

// ---------------------------------------------------------------- rods
// Adds row [k0, k1) of a link payload in list order, FP64, into the float sums (segGatherA/B,
// CrosslinkerSystem.java:129-173)
__device__ __forceinline__ void add_row(const float* pay, int k0, int k1, float F[3], float T[3]) {
    double f[3] = {0.0, 0.0, 0.0}, t[3] = {0.0, 0.0, 0.0};
    for (int k = k0; k < k1; k++) {
        const float2* q = reinterpret_cast<const float2*>(pay + 6 * (int64_t)k);
        const float2 x = q[0], y = q[1], z = q[2];
        f[0] += x.x; f[1] += x.y; f[2] += y.x;
        t[0] += y.y; t[1] += z.x; t[2] += z.y;
    }
    for (int k = 0; k < 3; k++) { F[k] = (float)(F[k] + f[k]); T[k] = (float)(T[k] + t[k]); }
}

constexpr int ROD_MOTORS = 16;        // bound motors of a rod that are held in registers
static_assert(ROD_MOTORS % 4 == 0 && ROD_MOTORS <= FUSED_MOTOR_SLOTS && FUSED_MOTOR_SLOTS % 4 == 0, "16-byte loads");

// sorts the first N of a row's slots, ascending (odd-even transposition)
template <int N>
__device__ __forceinline__ void sort_slots(int (&v)[ROD_MOTORS]) {
#pragma unroll
    for (int r = 0; r < N; r++)
#pragma unroll
        for (int j = r & 1; j + 1 < N; j += 2) {
            const int lo = min(v[j], v[j + 1]), hi = max(v[j], v[j + 1]);
            v[j] = lo;
            v[j + 1] = hi;
        }
}

// a neighbour rod as the step found it
__device__ __forceinline__ RodGeom start_rod(const FusedArgs& a, int j) {
    const sbx_rigid_body& fb = a.sc.fil.body;
    const float* c = a.sc.grid.center;
    const int n = a.nSeg, cap = a.cap;
    RodGeom r;
    r.cx = c[j]; r.cy = c[cap + j]; r.cz = c[2 * cap + j];
    r.ux = a.uSnap[j]; r.uy = a.uSnap[n + j]; r.uz = a.uSnap[2 * n + j];
    r.len = fb.segLength[j];
    r.bTGx = fb.bTransGam[j]; r.bTGy = fb.bTransGam[n + j]; r.bRGy = fb.bRotGam[n + j];
    return r;
}

// Chain forces from the joints made ahead, the crosslinker and motor gathers, the walls and the
// Langevin update of one rod a thread, in the reference's order; the rod's histograms are reset
// for the next step. A joint whose neighbour does not point back is computed from this side.
// MANY: for more rods than are on the chip at once at four blocks an SM (75,776 on 148 SMs), six
// (80 registers): what only the integration takes goes towards L1 first and is read after the
// bonds. 78.5 and 74.5 us a step at 100,000 rods, 329 and 325 at 500,000, 221 and 218.6 a packed
// step of 12 networks; but 25.9 and 26.6 at 1,000, 35.3 and 36.7 at 20,000, where the last read
// is on the step's path.
constexpr int RODS_AN_SM = 4 * 128;
template <bool B, bool MANY>
__global__ void __launch_bounds__(128, MANY ? 6 : 4) k_wide_rods(const __grid_constant__ WideArgs w) {
    const FusedArgs& a = w.a;
    const sbx_dense_scene& sc = a.sc;
    const sbx_filament_store& fs = sc.fil;
    const sbx_rigid_body& fb = fs.body;
    const sbx_crosslinker_store& xl = sc.xl;
    const int n = a.nSeg, i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) { after_previous(); return; }
    // what does not wait for anything first, all in flight together
    const int t = fs.counts[1];
    const int nm = a.cntM[i];
    int slots[2] = {fs.end2NbrSlot[i], fs.end1NbrSlot[i]};
    const int sides[2] = {fs.end2NbrSide[i], fs.end1NbrSide[i]};
    int a0 = 0, a1 = 0, b0 = 0, b1 = 0, act = 0;
    if (a.xlOn) {
        a0 = xl.segOffsetsA[i]; a1 = xl.segOffsetsA[i + 1];
        b0 = xl.segOffsetsB[i]; b1 = xl.segOffsetsB[i + 1];
        act = a.cntAct[i];
    }
    BodyIn in;
    if (MANY) {
        for (int k = 0; k < 3; k++) { in.p.c[k] = fb.coord[k * n + i]; in.p.u[k] = fb.uVec[k * n + i]; }
        in.len = fb.segLength[i]; in.gT[0] = fb.bTransGam[i]; in.gT[1] = fb.bTransGam[n + i]; in.gR[1] = fb.bRotGam[n + i];
        for (int k = 0; k < 3; k++) {
            prefetch_l1(fb.yVec + k * n + i); prefetch_l1(fb.randForce + k * n + i); prefetch_l1(fb.randTorque + k * n + i);
            if (fb.coord64) prefetch_l1(fb.coord64 + k * n + i);
        }
    } else {
        in = body_load(fb, i);
    }
    const ChainParams cp = chain_params(fs.chainParams);
    double fd[3] = {0.0, 0.0, 0.0}, td[3] = {0.0, 0.0, 0.0};
    RodGeom me;
    me.cx = in.p.c[0]; me.cy = in.p.c[1]; me.cz = in.p.c[2];
    me.ux = in.p.u[0]; me.uy = in.p.u[1]; me.uz = in.p.u[2];
    me.len = in.len; me.bTGx = in.gT[0]; me.bTGy = in.gT[1]; me.bRGy = in.gR[1];
    for (int side = 0; side < 2; side++) {
        int slot = slots[side];
        const int nside = sides[side];
        if (!SBX_IDX_OK_OR_NONE(slot, n, CK_NEIGHBOUR)) slot = -1;
        if (slot < 0) continue;
        const RodGeom nb = start_rod(a, slot);
        ChainJoint J;
        bool have = slot > i;
        if (have) {
            J = joint_load(a, i, side);
        } else if (nside == 0 || nside == 1) {
            const int ps = 1 - nside;                    // the partner's side facing rod i
            const int back = ps == 0 ? fs.end2NbrSlot[slot] : fs.end1NbrSlot[slot];
            const int backSide = ps == 0 ? fs.end2NbrSide[slot] : fs.end1NbrSide[slot];
            have = slot < i && back == i && backSide == 1 - side;
            if (have) J = joint_load(a, slot, ps);
        }
        if (!have) J = chain_joint(cp, i, side, slot, nside, me, nb);
        chain_apply(cp, i, side, slot, nside, me, nb, J, fd, td);
    }
    float F[3], T[3];
    for (int k = 0; k < 3; k++) { F[k] = (float)(0.0f + fd[k]); T[k] = (float)(0.0f + td[k]); }
    if (a.xlOn) {
        add_row(w.payA, a0, a1, F, T);
        add_row(w.payB, b0, b1, F, T);
    }
    // the bound motors in ascending slot: a short row is sorted here
    int ids[ROD_MOTORS];
    const bool fits = nm <= a.mRowUse && nm <= ROD_MOTORS;
#pragma unroll
    for (int q = 0; q < ROD_MOTORS; q += 4) {
        const int4 v = fits && nm > q ? *reinterpret_cast<const int4*>(a.slotM + (size_t)i * FUSED_MOTOR_SLOTS + q)
                                      : make_int4(0, 0, 0, 0);
        ids[q] = v.x; ids[q + 1] = v.y; ids[q + 2] = v.z; ids[q + 3] = v.w;
    }
#pragma unroll
    for (int j = 0; j < ROD_MOTORS; j++)
        if (j >= nm) ids[j] = 0x7fffffff;
    if (fits && nm > 4) sort_slots<ROD_MOTORS>(ids);
    else if (fits && nm > 1) sort_slots<4>(ids);
    after_previous();                    // the bonds; nothing is written before them
    if (i == 0) {
        *a.d_step = t + 1;               // (every reader of this step's index has run)
        *a.reachMax = 0;
        *a.odd = 0;
    }
    if (a.xlOn) {
        xl.activeLinkCount[i] = act;
        a.cntAct[i] = 0; a.cntA[i] = 0; a.cntB[i] = 0; a.headA[i] = -1; a.headB[i] = -1;
        if (i < w.tilesS) { w.sumA[i * WIDE_SUM_STRIDE] = 0; w.sumB[i * WIDE_SUM_STRIDE] = 0; }
    }
    // CrossBridgeSystem.segGather (CrossBridgeSystem.java:302-320): the bound motors' reactions
    // in ascending slot, GATHER of them in flight (one after another a rod with 15 motors held
    // its warp, and the step, for 9 us at 20,000 rods; now 3); a longer row by repeated minimum over its slots
    // and list
    double gf[3] = {0.0, 0.0, 0.0}, gt[3] = {0.0, 0.0, 0.0};
    constexpr int GATHER = 4;
#pragma unroll
    for (int q = 0; q < ROD_MOTORS; q += GATHER) {
        if (!fits || q >= nm) break;
        float p[GATHER][6];
#pragma unroll
        for (int j = 0; j < GATHER; j++) {
            const int m = ids[q + j];
            const bool on = m != 0x7fffffff && SBX_IDX_OK(m, a.nM, CK_MOTOR_SLOT);
            const float* r = sc.bondData + (int64_t)(on ? m : 0) * XB_STRIDE + 6;
#pragma unroll
            for (int k = 0; k < 6; k++) p[j][k] = on ? r[k] : 0.f;
            if (!on && q + j < nm) atomicOr(a.err, ERR_LIST);
        }
#pragma unroll
        for (int j = 0; j < GATHER; j++) {
            if (q + j >= nm) break;
            gf[0] += p[j][0]; gf[1] += p[j][1]; gf[2] += p[j][2];
            gt[0] += p[j][3]; gt[1] += p[j][4]; gt[2] += p[j][5];
        }
    }
    for (int q = 0, last = -1; !fits && q < nm; q++) {
        int next = 0x7fffffff;
        for (int j = 0; j < FUSED_MOTOR_SLOTS && j < nm && j < a.mRowUse; j++) {
            const int m = a.slotM[(size_t)i * FUSED_MOTOR_SLOTS + j];
            if (m > last && m < next) next = m;
        }
        if (nm > a.mRowUse) {
            int it = 0;
            for (int m = a.headM[i]; m >= 0 && it <= a.nM; m = a.nextM[m], it++) {
                if (!SBX_IDX_OK(m, a.nM, CK_MOTOR_SLOT)) break;
                if (m > last && m < next) next = m;
            }
        }
        if (next == 0x7fffffff || !SBX_IDX_OK(next, a.nM, CK_MOTOR_SLOT)) {
            atomicOr(a.err, ERR_LIST);
            break;
        }
        const float* p = sc.bondData + (int64_t)next * XB_STRIDE + 6;
        gf[0] += p[0]; gf[1] += p[1]; gf[2] += p[2];
        gt[0] += p[3]; gt[1] += p[4]; gt[2] += p[5];
        last = next;
    }
    for (int k = 0; k < 3; k++) { F[k] = (float)(F[k] + gf[k]); T[k] = (float)(T[k] + gt[k]); }
    if (MANY) in = body_load(fb, i);
    const float* box = B ? w.bt.boxParams + 8 * w.bt.segKey[2 * i] : sc.boxParams;
    const BoxParams bx = box_params(box, t);
    if (bx.active) confine_one(bx, in.p.c, in.p.u, in.len, in.gT[0], F, T);
    body_step(fb, i, in, F, T, B ? fs.params[0] : sc.boxParams[7]);
}

__global__ void k_wide_noise(WideNoise* dst, const WideNoise noise) { *dst = noise; }

}  // namespace

sbx_status wide_set_noise(sbx_ctx* ctx, const WideArgs& w, const WideNoise& noise) {
    SBX_LAUNCH(ctx, k_wide_noise, 1, 1, w.noise, noise);
    return check_launch(ctx, "dense step: noise");
}

bool wide_streams_create(WideStreams& ws) {
    for (cudaStream_t* s : {&ws.ahead, &ws.link, &ws.csr})
        if (cudaStreamCreateWithFlags(s, cudaStreamNonBlocking) != cudaSuccess) return false;
    for (cudaEvent_t* e : {&ws.start, &ws.bound, &ws.joined, &ws.linkDone, &ws.csrDone})
        if (cudaEventCreateWithFlags(e, cudaEventDisableTiming) != cudaSuccess) return false;
    return true;
}

void wide_streams_destroy(WideStreams& ws) {
    for (cudaStream_t s : {ws.ahead, ws.link, ws.csr})
        if (s) cudaStreamDestroy(s);
    for (cudaEvent_t e : {ws.start, ws.bound, ws.joined, ws.linkDone, ws.csrDone})
        if (e) cudaEventDestroy(e);
    ws = WideStreams{};
}

namespace {

template <bool B>
sbx_status wide_step_impl(sbx_ctx* ctx, const WideArgs& w, const WideStreams& ws) {
    const FusedArgs& a = w.a;
    cudaStream_t s = ctx->stream;
    cudaError_t e = cudaSuccess;
    auto ok = [&](cudaError_t r) { if (e == cudaSuccess) e = r; };
    int sms = 0;
    ok(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device));
    auto fork = [&](cudaEvent_t ev, cudaStream_t to) { ok(cudaEventRecord(ev, s)); ok(cudaStreamWaitEvent(to, ev, 0)); };
    auto join = [&](cudaEvent_t ev, cudaStream_t from) { ok(cudaEventRecord(ev, from)); ok(cudaStreamWaitEvent(s, ev, 0)); };
    // early: the kernel waits for its predecessor itself
    auto launch = [&](cudaStream_t to, bool early, auto kernel, int64_t items, int block) {
        cudaLaunchAttribute attr;
        attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr.val.programmaticStreamSerializationAllowed = 1;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(blocks(items, block));
        cfg.blockDim = dim3(block);
        cfg.stream = to;
        cfg.attrs = &attr;
        cfg.numAttrs = early ? 1 : 0;
        ok(cudaLaunchKernelEx(&cfg, kernel, w));
        ctx->launches++;
    };
    fork(ws.start, ws.ahead);
    if (a.xlOn) ok(cudaStreamWaitEvent(ws.link, ws.start, 0));
    // The three kernels ahead need nothing of each other: they start together while their threads
    // fit on the chip at once (2048 an SM), else one after another, as their blocks would go
    // before the main stream's. Together and in turn: 28.8 and 30.0 us a step at 1,000 rods, 85.0
    // and 86.4 at 100,000; 360 and 356 at 500,000 with all three let through.
    const bool side = (int64_t)a.nB + a.nBb + a.nSeg <= (int64_t)sms * 2048;
    launch(ws.ahead, false, k_wide_draws<B>, (int64_t)a.nB + a.nBb + a.nSeg, 256);
    launch(ws.ahead, side, k_wide_terms, 2 * (int64_t)a.nM + 4 * (int64_t)a.nD, 128);
    launch(ws.ahead, side, k_wide_joints, a.nSeg, 128);
    if (a.xlOn) {
        launch(ws.link, false, k_wide_link_rows<B>, a.nL, 128);
        launch(ws.link, true, k_wide_link_scan, (int64_t)2 * w.tilesS * 256, 256);
        launch(ws.link, true, k_wide_links, a.nL, 128);
    }
    if (a.cap > a.nSeg + a.nM) launch(s, false, k_wide_publish<B, true>, a.cap, 256);
    else launch(s, false, k_wide_publish<B, false>, a.cap, 256);
    launch(s, true, k_wide_cell_scan, (int64_t)2 * w.tilesC * 256, 256);
    launch(s, true, k_wide_place, a.cap, 256);
    launch(s, true, k_wide_bind<B>, ((int64_t)a.nM + BIND_HEADS - 1) / BIND_HEADS * 32, 128);
    fork(ws.bound, ws.csr);
    launch(ws.csr, false, k_wide_motor_scan, (int64_t)w.tilesS * 256, 256);
    launch(ws.csr, false, k_wide_motor_place, std::max(std::max(a.nM, a.C), w.tilesS), 256);
    join(ws.joined, ws.ahead);
    if (a.xlOn) join(ws.linkDone, ws.link);
    launch(s, false, k_wide_mini<B>, ((int64_t)a.nBb + (a.nBb + MINI_THREADS - 1) / MINI_THREADS) * MINI_THREADS,
           MINI_THREADS);
    if (a.nSeg > (int64_t)sms * RODS_AN_SM) launch(s, true, k_wide_rods<B, true>, a.nSeg, 128);
    else launch(s, true, k_wide_rods<B, false>, a.nSeg, 128);
    join(ws.csrDone, ws.csr);
    if (e != cudaSuccess) return fail(ctx, SBX_ECUDA, std::string("dense step: streams: ") + cudaGetErrorString(e));
    return check_launch(ctx, "dense step");
}

}  // namespace

sbx_status wide_step(sbx_ctx* ctx, const WideArgs& w, bool batched, const WideStreams& ws) {
    SBX_TRACE("sbx.dense.step");
    return batched ? wide_step_impl<true>(ctx, w, ws) : wide_step_impl<false>(ctx, w, ws);
}

SBX_CHECK_EXPORT(wide)
