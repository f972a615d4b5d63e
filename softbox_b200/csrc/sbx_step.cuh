// sbx_step.cuh — device code of the dense step that its two shapes share: the persistent fused
// kernel (sbx_fused.cu) and the step as a few wide kernels (sbx_wide.cu).
#pragma once
#include "sbx_fused.cuh"
#include "sbx_internal.cuh"
#include "sbx_physics.cuh"

using namespace sbx;

namespace {

__device__ __forceinline__ int vload(const int* p) { return *(const volatile int*)p; }

// error word: a reach list past MAX_CAND, a linked-list walk past its bound
constexpr int ERR_REACH_OVERFLOW = 2, ERR_LIST = 8;

// force and torque sums of one minifilament's sub-bodies; with odd dimer tables each of its
// motors' place in a dimer (2 d, 2 d + 1 as motor B, or -1) and the dimer that tethers its rod
struct MiniSmem {
    float sF[3 * FUSED_MAX_SUB], sT[3 * FUSED_MAX_SUB];
    int dimer[32], tether[32];
};

// BrownianForceSystem.brownianForce (BrownianForceSystem.java:44-106), component j (0..2) of
// one slot: the slot's j-th Box-Muller pair gives its random force and torque components j
// (randF = ((tS * mag) * sqrt(gamma)) * g, :94-104). In supplied-noise mode the Gaussians come
// from noise[t - t0][6][n] (a step outside the supplied range, which the host rejects before
// the launch, draws zeros).
// `key` is the slot the draw is keyed by (in packed networks the slot within its network).
__device__ __forceinline__ void brownian_component(const FusedArgs& a, const sbx_rigid_body& b, int s, int key, int j,
                                                   int t, int seed, float mag, const float* noise) {
    const int n = b.n;
    float gf, gt;
    if (noise) {
        int k = t - a.nzT0;
        bool in = k >= 0 && k < a.nzN;
        const float* q = noise + (int64_t)(in ? k : 0) * 6 * n + s;
        gf = in ? q[(int64_t)j * n] : 0.f;
        gt = in ? q[(int64_t)(3 + j) * n] : 0.f;
    } else {
        gauss_pair_wang(key, t, seed, j, &gf, &gt);
    }
    const float tS = b.brownTransScale[s], rS = b.brownRotScale[s];
    b.randForce[j * n + s] = tS * mag * fsqrt(b.bTransGam[j * n + s]) * gf;
    b.randTorque[j * n + s] = rS * mag * fsqrt(b.bRotGam[j * n + s]) * gt;
}

// ---------------------------------------------------------------- rows: slots + overflow lists
// Rank of `self` in a row = the number of the row's items with a smaller index, counted
// along the row's list: the position the reference's serial scatter gives it (items are
// scattered in ascending index). A walk longer than `bound` marks the list corrupt.
__device__ __forceinline__ int list_rank(const FusedArgs& a, int head, const int* next, int self, int bound) {
    int r = 0, it = 0;
    for (int j = head; j >= 0; j = next[j]) {
        if (!SBX_IDX_OK(j, bound, CK_LIST_ENTRY)) break;
        r += j < self;
        if (++it > bound) {
            atomicOr(a.err, ERR_LIST);
            break;
        }
    }
    return r;
}

// Appends `item` to row r: the histogram's old count is its arrival index j; the first `use`
// (<= S, the slot stride) arrivals take the row's fixed slots, later ones join the row's
// overflow list (returns 1).
__device__ __forceinline__ int row_put(int* slot, int S, int use, int* head, int* next, int r, int item, int j) {
    if (j < use) {
        slot[(size_t)r * S + j] = item;
        return 0;
    }
    next[item] = atomicExch(&head[r], item);
    return 1;
}
__device__ __forceinline__ int row_insert(int* cnt, int* slot, int S, int use, int* head, int* next, int r,
                                          int item) {
    return row_put(slot, S, use, head, next, r, item, atomicAdd(&cnt[r], 1));
}

// adds a thread's count of a capacity fallback to the plan's counters, one addition per warp (of
// the threads that get here together): all counts meet in one word
__device__ __forceinline__ void stat_add(const FusedArgs& a, int which, int v) {
    const unsigned here = __activemask();
    const int sum = __reduce_add_sync(here, v);
    if (sum && (int)(threadIdx.x & 31) == __ffs(here) - 1) atomicAdd(&a.stats[which], (unsigned long long)sum);
}

// rank of `item` in row r of n items: the row's members with a smaller index (slots, then the list)
template <int S>
__device__ __forceinline__ int row_rank(const FusedArgs& a, int n, const int* slot, int use, const int* head,
                                        const int* next, int r, int item, int bound) {
    int rank = 0;
#pragma unroll
    for (int j = 0; j < S; j++)
        if (j < n && j < use) rank += slot[(size_t)r * S + j] < item;
    if (n > use) rank += list_rank(a, head[r], next, item, bound);
    return rank;
}
template <int S>
__device__ __forceinline__ int row_rank(const FusedArgs& a, const int* cnt, const int* slot, int use,
                                        const int* head, const int* next, int r, int item, int bound) {
    return row_rank<S>(a, cnt[r], slot, use, head, next, r, item, bound);
}

// ---------------------------------------------------------------- scans (B, C, G, H)
struct ScanArr {
    const int* cnt;   // histogram
    int n;            // rows
    int tile0;        // first tile index in the shared tile-sum array
};

__device__ __forceinline__ int warp_sum(int v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ void tile_sums(const ScanArr* arrs, int narr, int* tileSum, int warp, int nwarps) {
    int lane = threadIdx.x & 31;
    int total = arrs[narr - 1].tile0 + (arrs[narr - 1].n + SCAN_CHUNK - 1) / SCAN_CHUNK;
    for (int tl = warp; tl < total; tl += nwarps) {
        int ai = 0;
        while (ai + 1 < narr && tl >= arrs[ai + 1].tile0) ai++;
        const ScanArr& s = arrs[ai];
        int base = (tl - s.tile0) * SCAN_CHUNK;
        int v = 0;
        for (int j = lane; j < SCAN_CHUNK; j += 32) v += (base + j < s.n) ? s.cnt[base + j] : 0;
        v = warp_sum(v);
        if (lane == 0) tileSum[tl] = v;
    }
}

// exclusive scan of each array into out[ai][0..n] (terminator = min(total, clamp[ai]));
// copy[ai] (optional) receives the counts — the row lengths the reference's serial
// scatter leaves in its write cursors; chunkOut (optional, array 0) gets the tile-prefix
// layout of SpatialGrid.gridScanChunks.
__device__ void tile_scan(const ScanArr* arrs, int narr, const int* tileSum, int* const* out, int* const* copy,
                          const int* clampTotal, int* chunkOut, int warp, int nwarps) {
    int lane = threadIdx.x & 31;
    int total = arrs[narr - 1].tile0 + (arrs[narr - 1].n + SCAN_CHUNK - 1) / SCAN_CHUNK;
    for (int tl = warp; tl < total; tl += nwarps) {
        int ai = 0;
        while (ai + 1 < narr && tl >= arrs[ai + 1].tile0) ai++;
        const ScanArr& s = arrs[ai];
        int ntiles = (s.n + SCAN_CHUNK - 1) / SCAN_CHUNK;
        int local = tl - s.tile0;
        // the preceding tiles' sums: 16 predicated loads per lane in flight together
        int b = 0;
#pragma unroll
        for (int q = 0; q < 16; q++) {
            int j = lane + 32 * q;
            b += (j < local) ? tileSum[s.tile0 + j] : 0;
        }
        for (int j = lane + 512; j < local; j += 32) b += tileSum[s.tile0 + j];
        b = warp_sum(b);
        int base = local * SCAN_CHUNK;
        constexpr int PER = SCAN_CHUNK / 32;
        // coalesced: row j of the tile is elements base + 32 j + lane
        int vals[PER];
#pragma unroll
        for (int j = 0; j < PER; j++) {
            int r = base + 32 * j + lane;
            vals[j] = r < s.n ? s.cnt[r] : 0;
        }
        int run = b;
#pragma unroll
        for (int j = 0; j < PER; j++) {
            int v = vals[j], x = v;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                int y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += y;
            }
            int r = base + 32 * j + lane;
            if (r < s.n) {
                out[ai][r] = run + x - v;
                if (copy[ai]) copy[ai][r] = v;
            }
            run += __shfl_sync(0xffffffffu, x, 31);
        }
        if (lane == 0 && ai == 0 && chunkOut) chunkOut[local] = b;
        if (local == ntiles - 1) {
            int tot = run;
            if (lane == 0) {
                out[ai][s.n] = tot < clampTotal[ai] ? tot : clampTotal[ai];
                if (ai == 0 && chunkOut) chunkOut[ntiles] = tot;
            }
        }
    }
}

// ---------------------------------------------------------------- binding and minifilaments
// The step's joints and myosin terms as planes: the lanes of a warp write and read consecutive
// items of a plane (as one struct after another a warp's 16-byte accesses touched 20 lines
// each: at 500,000 rods the terms kernel went from 42 to 27 us, the step from 377 to 370, at
// 100,000 from 102 to 96.5).
__device__ __forceinline__ void joint_store(const FusedArgs& a, int i, int side, const ChainJoint& J) {
    const size_t n = a.nSeg;
    double* p = a.joints + 6 * n * side + i;
    p[0] = J.forceMag; p[n] = J.luX; p[2 * n] = J.luY; p[3 * n] = J.luZ; p[4 * n] = J.invMag; p[5 * n] = J.torsionMag;
    reinterpret_cast<int*>(a.joints + 12 * n)[n * side + i] = J.tvOK;
}
__device__ __forceinline__ ChainJoint joint_load(const FusedArgs& a, int i, int side) {
    const size_t n = a.nSeg;
    const double* p = a.joints + 6 * n * side + i;
    ChainJoint J;
    J.forceMag = p[0]; J.luX = p[n]; J.luY = p[2 * n]; J.luZ = p[3 * n]; J.invMag = p[4 * n]; J.torsionMag = p[5 * n];
    J.tvOK = reinterpret_cast<const int*>(a.joints + 12 * n)[n * side + i];
    return J;
}

struct GlobalTerms {
    const FusedArgs& a;
    __device__ __forceinline__ double* motor(int which, int m) const { return a.terms + (size_t)9 * a.nM * which + m; }
    __device__ __forceinline__ double* dimer(int plane, int d) const {
        return a.terms + (size_t)FUSED_MOTOR_PLANES * a.nM + (size_t)plane * a.nD + d;
    }
    __device__ __forceinline__ MotorJoint joint(int m, int which) const {
        const double* p = motor(which, m);
        const size_t n = a.nM;
        MotorJoint J;
        J.forceMag = p[0]; J.lx = p[n]; J.ly = p[2 * n]; J.lz = p[3 * n];
        J.tvx = p[4 * n]; J.tvy = p[5 * n]; J.tvz = p[6 * n]; J.tm[0] = p[7 * n]; J.tm[1] = p[8 * n];
        return J;
    }
    __device__ __forceinline__ void put(int m, int which, const MotorJoint& J) const {
        double* p = motor(which, m);
        const size_t n = a.nM;
        p[0] = J.forceMag; p[n] = J.lx; p[2 * n] = J.ly; p[3 * n] = J.lz;
        p[4 * n] = J.tvx; p[5 * n] = J.tvy; p[6 * n] = J.tvz; p[7 * n] = J.tm[0]; p[8 * n] = J.tm[1];
    }
    __device__ __forceinline__ CoupleTerm couple(int d, int v) const {
        const double* p = dimer(10 * v, d);
        const size_t n = a.nD;
        CoupleTerm C;
        C.FAx = p[0]; C.FAy = p[n]; C.FAz = p[2 * n]; C.TAx = p[3 * n]; C.TAy = p[4 * n]; C.TAz = p[5 * n];
        C.TBx = p[6 * n]; C.TBy = p[7 * n]; C.TBz = p[8 * n];
        C.ok = *reinterpret_cast<const int*>(p + 9 * n);
        return C;
    }
    __device__ __forceinline__ void put(int d, int v, const CoupleTerm& C) const {
        double* p = dimer(10 * v, d);
        const size_t n = a.nD;
        *reinterpret_cast<int*>(p + 9 * n) = C.ok;
        if (!C.ok) return;
        p[0] = C.FAx; p[n] = C.FAy; p[2 * n] = C.FAz; p[3 * n] = C.TAx; p[4 * n] = C.TAy; p[5 * n] = C.TAz;
        p[6 * n] = C.TBx; p[7 * n] = C.TBy; p[8 * n] = C.TBz;
    }
    __device__ __forceinline__ LeverTerm lever(int d) const {
        const double* p = dimer(20, d);
        const size_t n = a.nD;
        LeverTerm L;
        L.px = p[0]; L.py = p[n]; L.pz = p[2 * n];
        L.ok = *reinterpret_cast<const int*>(p + 3 * n);
        return L;
    }
    __device__ __forceinline__ void put(int d, const LeverTerm& L) const {
        double* p = dimer(20, d);
        const size_t n = a.nD;
        *reinterpret_cast<int*>(p + 3 * n) = L.ok;
        if (!L.ok) return;
        p[0] = L.px; p[n] = L.py; p[2 * n] = L.pz;
    }
    // (the rows' floats take three planes of doubles, as six planes of floats)
    __device__ __forceinline__ float* row(int d) const { return reinterpret_cast<float*>(dimer(31, 0)) + d; }
    __device__ __forceinline__ TetherTerm tether(int d, int& odd) const {
        const double* p = dimer(24, d);
        const size_t n = a.nD;
        TetherTerm T;
        T.Fx = p[0]; T.Fy = p[n]; T.Fz = p[2 * n]; T.Tx = p[3 * n]; T.Ty = p[4 * n]; T.Tz = p[5 * n];
        const int ok = *reinterpret_cast<const int*>(p + 6 * n);
        T.fOK = ok & 1;
        T.tOK = (ok >> 1) & 1;
        odd = ok >> 2;
        return T;
    }
    // (odd: the device's tables have another dimer there than the harness layout)
    __device__ __forceinline__ void put(int d, const TetherTerm& T, bool odd) const {
        double* p = dimer(24, d);
        const size_t n = a.nD;
        if (T.fOK) { p[0] = T.Fx; p[n] = T.Fy; p[2 * n] = T.Fz; }
        if (T.tOK) { p[3 * n] = T.Tx; p[4 * n] = T.Ty; p[5 * n] = T.Tz; }
        *reinterpret_cast<int*>(p + 6 * n) = (T.fOK ? 1 : 0) | (T.tOK ? 2 : 0) | (odd ? 4 : 0);
        float* q = row(d);
        for (int j = 0; j < 6; j++) q[j * n] = T.row[j];
    }
};

// The reach of a segment's points from its centre, the largest coordinate difference of its ends
// to it; anything that is not a number counts as out of bounds (the walk then takes all cells).
__device__ __forceinline__ float segment_span(const float c[3], const float e1[3], const float e2[3]) {
    float v = 0.f, sum = 0.f;
    for (int k = 0; k < 3; k++) {
        const float p = fabsf(e1[k] - c[k]), q = fabsf(e2[k] - c[k]);
        v = fmaxf(v, fmaxf(p, q));
        sum += p + q;
    }
    return sum < 1.0e30f ? v : 3.0e38f;
}

// raises *reachMax (float bits of a non-negative value) by a warp's largest span
__device__ __forceinline__ void span_max(int* reachMax, float v) {
    const unsigned m = __reduce_max_sync(0xffffffffu, __float_as_uint(v));
    if ((threadIdx.x & 31) == 0 && (int)m > vload(reachMax)) atomicMax(reachMax, (int)m);
}

// how far from the head the centre of a segment in reach can be, with room for the rounding of
// the test and of the cell coordinates
__device__ __forceinline__ float reach_span(const FusedArgs& a, float tol, float x, float y, float z) {
    const float d = fabsf(tol) + __int_as_float(vload(a.reachMax));
    return d * 1.001f + 1.0e-5f + 2.0e-6f * (fabsf(x) + fabsf(y) + fabsf(z));
}

// BindingDetectionSystem.gridReachable (BindingDetectionSystem.java:161-227) over the
// segment-only cell-ordered endpoints, fused with bindNearest's selection
// (BindingDetectionSystem.java:366-388): the same 27 cells in the same order (nine rows of
// three consecutive x-cells), the same predicate, and the first nearest among the first
// MAX_CAND candidates. A group of W lanes (8 or 16) walks one head (the 32 / W groups of a
// warp walk as many heads side by side; every lane of a group calls it with its group's
// head, `valid` false for a group without one): lane r of the group reads stencil row r's
// range (with 8 lanes, lane 0 also row 8), then the entries are tested W at a time, lane k
// of the group taking entry k0 + k. Passing entries are appended in entry order (ballot,
// and the popcount of the group's lower lanes' passes), so the list is the serial walk's
// list; the nearest of the first MAX_CAND (strict <, the first in list order wins) is the
// serial choice: a chunk's minimum with ties to its lowest lane replaces the running best
// only when strictly smaller. Every group runs the same number of chunks (the longest
// walk's), so every shuffle has the whole warp. Returns the reach count; best and arc are
// the same on every lane of the group.
// Of the 27 cells only those within reach_span of the head are walked. A segment that passes
// has a point within tol of the head, and that point is within *reachMax of its centre in every
// coordinate (segment_span, over all segments of the step), so its centre lies in those cells:
// cell_coord is monotonic. With rods and reach well below a cell (0.05 + 0.03 um against 0.24)
// that leaves about five of them.
struct GridView {
    const float* gp;             // gridParams
    int nX, nY, nZ;
    const int* off;              // segment-only cell offsets of the grid's first cell
};
struct NoWait {
    __device__ void operator()() const {}
};
// (ready() comes before the first read of the endpoints)
template <int W, class Ready = NoWait>
__device__ int group_reach_bind(const FusedArgs& a, const GridView& gv, int lane, bool valid, float mx, float my, float mz, float mux,
                                float muy, float muz, float rux, float ruy, float ruz, int* out, float tol,
                                float align, int* bestSeg, float* bestArc, Ready ready = Ready()) {
    static_assert(W == 8 || W == 16, "a group of 8 or 16 lanes walks one head");
    const float* gp = gv.gp;
    const int* off = gv.off;
    const int hl = lane & (W - 1), grp = lane / W;
    const int nX = gv.nX, nY = gv.nY, nZ = gv.nZ, nXY = nX * nY;
    const int cx = cell_coord(mx, gp[0], gp[4], nX), cy = cell_coord(my, gp[1], gp[4], nY),
              cz = cell_coord(mz, gp[2], gp[4], nZ);
    const float span = reach_span(a, tol, mx, my, mz);
    const int x0 = max(cx - 1, cell_coord(mx - span, gp[0], gp[4], nX)),
              x1 = min(cx + 1, cell_coord(mx + span, gp[0], gp[4], nX));
    const int y0 = max(cy - 1, cell_coord(my - span, gp[1], gp[4], nY)),
              y1 = min(cy + 1, cell_coord(my + span, gp[1], gp[4], nY));
    const int z0 = max(cz - 1, cell_coord(mz - span, gp[2], gp[4], nZ)),
              z1 = min(cz + 1, cell_coord(mz + span, gp[2], gp[4], nZ));
    // lane hl reads stencil row hl; with 8 lanes, lane 0 also reads row 8
    int rs = 0, len = 0, rs8 = 0, len8 = 0;
    auto row = [&](int r, int& s, int& l) {
        int zz = cz - 1 + r / 3, yy = cy - 1 + r % 3;
        if (zz >= z0 && zz <= z1 && yy >= y0 && yy <= y1) {
            int c0 = x0 + yy * nX + zz * nXY;
            s = off[c0];
            l = off[c0 + (x1 - x0) + 1] - s;
        }
    };
    if (valid && hl < 9) row(hl, rs, len);
    if (W == 8 && valid && hl == 0) row(8, rs8, len8);
    int inc = len;
#pragma unroll
    for (int o = 1; o < W; o <<= 1) {
        int y = __shfl_up_sync(0xffffffffu, inc, o, W);
        if (hl >= o) inc += y;
    }
    const int lanesTotal = __shfl_sync(0xffffffffu, inc, W - 1, W);     // rows 0 .. min(8, W - 1)
    const int total = lanesTotal + (W == 8 ? __shfl_sync(0xffffffffu, len8, 0, W) : 0);
    int totalMax = total;
#pragma unroll
    for (int o = W; o < 32; o <<= 1) totalMax = max(totalMax, __shfl_xor_sync(0xffffffffu, totalMax, o));
    // every lane holds its group's nine (start of row in the sequence, start of row in memory) pairs
    int preR[9], rsR[9];
#pragma unroll
    for (int r = 0; r < 9; r++) {
        if (r < W) {
            preR[r] = __shfl_sync(0xffffffffu, inc - len, r, W);
            rsR[r] = __shfl_sync(0xffffffffu, rs, r, W);
        } else {
            preR[r] = lanesTotal;
            rsR[r] = __shfl_sync(0xffffffffu, rs8, 0, W);
        }
    }
    const unsigned lower = (1u << hl) - 1u;
    int cnt = 0, best = -1;
    float bestD = 1.0e30f, arc = 0.f;
    ready();
    for (int k0 = 0; k0 < totalMax; k0 += W) {
        const int k = k0 + hl;
        bool pass = false;
        float d = 0.f;
        float4 e1 = make_float4(0.f, 0.f, 0.f, 0.f), e2 = e1;
        if (k < total) {
            int idx = rsR[0] + k;
#pragma unroll
            for (int r = 1; r < 9; r++)
                if (k >= preR[r]) idx = rsR[r] + (k - preR[r]);
            if (SBX_IDX_OK(idx, a.nSeg, CK_REACH_ENTRY)) {
                e1 = a.segE1[idx];
                e2 = a.segE2[idx];
                d = reach_test_dist_sq(mx, my, mz, mux, muy, muz, rux, ruy, ruz, e1.x, e1.y, e1.z, e2.x, e2.y, e2.z,
                                       tol, align);
                pass = d >= 0.f && __float_as_int(e1.w) >= 0;
            }
        }
        const unsigned mask = (__ballot_sync(0xffffffffu, pass) >> (W * grp)) & ((1u << W) - 1u);
        const int pos = cnt + __popc(mask & lower);
        const int sg = __float_as_int(e1.w);
        const bool elig = pass && pos < MAX_CAND;
        if (elig) out[pos] = sg;
        float v = elig ? d : 3.0e38f;
        int who = hl;
#pragma unroll
        for (int o = W / 2; o > 0; o >>= 1) {
            float ov = __shfl_xor_sync(0xffffffffu, v, o);
            int ow = __shfl_xor_sync(0xffffffffu, who, o);
            if (ov < v || (ov == v && ow < who)) { v = ov; who = ow; }
        }
        float myArc = 0.f;
        if (v < bestD && hl == who) myArc = bind_arc(mx, my, mz, e1.x, e1.y, e1.z, e2.x, e2.y, e2.z);
        const int bw = __shfl_sync(0xffffffffu, sg, who, W);
        const float ba = __shfl_sync(0xffffffffu, myArc, who, W);
        if (v < bestD) {
            bestD = v;
            best = bw;
            arc = ba;
        }
        cnt += __popc(mask);
    }
    *bestSeg = best;
    *bestArc = arc;
    return cnt;
}

// CrossBridgeSystem.bondForces of head m (CrossBridgeSystem.java:58-141), stored
__device__ __forceinline__ void bond_store(const FusedArgs& a, int m, float out[XB_STRIDE]) {
    const sbx_motor_store& mot = a.sc.mot;
    const sbx_rigid_body& mb = mot.body;
    const sbx_rigid_body& fb = a.sc.fil.body;
    int bs = mot.boundSeg[m];
    if (!SBX_IDX_OK_OR_NONE(bs, a.nSeg, CK_BOUND_SEG)) bs = -1;
    bond_one(m, a.nB, mb.coord, mb.uVec, mb.yVec, mb.bRotGam, a.nSeg, fb.coord, fb.uVec, fb.yVec, fb.bRotGam,
             fb.segLength, bs, mot.bindArc[m], mot.nucleotideState[m], a.sc.xbParams, out);
    for (int k = 0; k < XB_STRIDE; k++) a.sc.bondData[m * XB_STRIDE + k] = out[k];
}

// MiniFilamentSystem.backboneGather over backbone u's CSR row (its dimers, ascending;
// MiniFilamentSystem.java:140-147), then walls, integration and derived geometry; the
// reference's CSR arrays (rows = backbones, items = dimers in index order)
template <bool LIVE>
__device__ __forceinline__ void mini_backbone(const FusedArgs& a, int u, int t, const float* boxParams, float dt) {
    const GlobalTerms terms{a};
    const sbx_minifilament_store& mini = a.sc.mini;
    const sbx_rigid_body& bb = mini.backbone;
    const int nBb = a.nBb, nD = a.nD;
    int dpm = a.dpm, d0 = u * dpm;
    double f[3] = {0, 0, 0}, tq[3] = {0, 0, 0};
    auto add = [&](int d) {
        const float* p = terms.row(d);                // the dimer's miniData row
        const size_t n = nD;
        f[0] += p[0]; f[1] += p[n]; f[2] += p[2 * n];
        tq[0] += p[3 * n]; tq[1] += p[4 * n]; tq[2] += p[5 * n];
    };
    if (LIVE && vload(a.odd)) {
        // (any table: the row's place from all dimers, its members where they are)
        dpm = d0 = 0;
        for (int d = 0; d < nD; d++) {
            const int h = mini.headBackboneSlot[d];
            dpm += h == u;
            d0 += h >= 0 && h < u;
        }
        for (int d = 0, q = d0; d < nD; d++)
            if (mini.headBackboneSlot[d] == u) {
                mini.bbDimerList[q++] = d;
                add(d);
            }
    } else {
        for (int d = d0; d < d0 + dpm; d++) add(d);
    }
    mini.bbDimerCount[u] = dpm;
    mini.bbDimerOffsets[u] = d0;
    if (u == nBb - 1) mini.bbDimerOffsets[nBb] = d0 + dpm;
    float F[3], T[3];
    for (int k = 0; k < 3; k++) { F[k] = (float)(0.0f + f[k]); T[k] = (float)(0.0f + tq[k]); }
    BoxParams bx = box_params(boxParams, t);
    float c[3] = {bb.coord[u], bb.coord[nBb + u], bb.coord[2 * nBb + u]};
    float uu[3] = {bb.uVec[u], bb.uVec[nBb + u], bb.uVec[2 * nBb + u]};
    if (bx.active) confine_one(bx, c, uu, bb.segLength[u], bb.bTransGam[u], F, T);
    integrate_derive_store(bb, u, F, T, dt);
}

// the sums of motor ml's rod (role 0) or lever (1) of minifilament u begin with its joints; returns
// the sub-body
__device__ __forceinline__ int joint_sums(const FusedArgs& a, MiniSmem& ms, int u, int role, int ml) {
    const GlobalTerms terms{a};
    const sbx_motor_store& mot = a.sc.mot;
    const sbx_rigid_body& mb = mot.body;
    const int nB = a.nB, spm = 6 * a.dpm;
    const int m = 2 * u * a.dpm + ml, sl = 3 * ml + role, s = u * spm + sl;
    int nuc = mot.nucleotideState[m];
    double f[3] = {0.0, 0.0, 0.0}, tq[3] = {0.0, 0.0, 0.0};
    if (role == 0) {
        motor_joint_apply(terms.joint(m, 0), 0, false, nuc, s, nB, mb.uVec, mb.segLength, mot.jointParams, f, tq);
    } else {
        motor_joint_apply(terms.joint(m, 0), 0, true, nuc, s, nB, mb.uVec, mb.segLength, mot.jointParams, f, tq);
        motor_joint_apply(terms.joint(m, 1), 1, false, nuc, s, nB, mb.uVec, mb.segLength, mot.jointParams, f, tq);
    }
    for (int k = 0; k < 3; k++) {
        ms.sF[k * spm + sl] = (float)(0.0 + f[k]);
        ms.sT[k * spm + sl] = (float)(0.0 + tq[k]);
    }
    return s;
}

// The rods' and levers' sums of minifilament u again, with the dimers as odd tables have them (96
// threads): each motor's dimer by a scan of all, its terms computed here. Such a scene keeps
// its bits, not its speed; the others pay for a vote. (A motor belongs to one dimer, so where
// a minifilament's own dimers are the layout's, so are its motors'.)
__device__ __noinline__ void odd_sums(const FusedArgs& a, MiniSmem& ms, int u) {
    const sbx_dense_scene& sc = a.sc;
    const sbx_rigid_body& mb = sc.mot.body;
    const int mpm = 2 * a.dpm, spm = 6 * a.dpm, m0 = u * mpm, tid = threadIdx.x, ml = tid & 31;
    if (tid < 32) ms.dimer[tid] = ms.tether[tid] = -1;
    asm volatile("bar.sync 1, 96;" ::: "memory");
    for (int d = tid; d < a.nD; d += 96) {
        const int mA = sc.dim.motorA[d] - m0, mB = sc.dim.motorB[d] - m0, rA = sc.mini.motorA[d] - m0;
        if (mA >= 0 && mA < mpm) ms.dimer[mA] = 2 * d;
        if (mB >= 0 && mB < mpm) ms.dimer[mB] = 2 * d + 1;
        if (rA >= 0 && rA < mpm) ms.tether[rA] = d;
    }
    asm volatile("bar.sync 1, 96;" ::: "memory");
    if (tid < 32 || ml >= mpm) return;
    LocalAcc acc{ms.sF, ms.sT, u * spm, spm};
    const int role = (tid - 32) >> 5, s = joint_sums(a, ms, u, role, ml);
    const int at = ms.dimer[ml], d = at >> 1;
    const bool isA = (at & 1) == 0;
    const int mA = at < 0 ? -1 : sc.dim.motorA[d], mB = at < 0 ? -1 : sc.dim.motorB[d];
    const bool paired = mA >= 0 && mA < a.nM && mB >= 0 && mB < a.nM;
    const bool par = paired && sc.dim.parallel[d] != 0;
    if (role == 0) {
        for (int v = 0; v < 2 && paired; v++)
            couple_apply_rod(acc, s, isA, couple_variant(a.nB, mb.coord, mb.uVec, mb.segLength, mb.bTransGam, mb.bRotGam,
                                                         mA, mB, par, sc.dim.dimerParams, v));
        int odd;
        if (ms.tether[ml] >= 0) tether_apply(acc, s, GlobalTerms{a}.tether(ms.tether[ml], odd));
    } else if (par && !(sc.mot.boundSeg[mA] >= 0 && sc.mot.boundSeg[mB] >= 0)) {
        couple_apply_lever(acc, s, isA, couple_lever(a.nB, mb.uVec, mb.bRotGam, mA, mB, sc.dim.dimerParams));
    }
}

// The sub-bodies of minifilament u on the first three warps of a block (its heads' binding and
// the position-only terms ran before). Each sub-body accumulates its terms in the order of the
// reference's System sequence (joints, coupling, tether; the head's bond after its joint): a
// warp for the heads, the rods, the levers; then they integrate in body order. LIVE: the dimers
// as the device's tables have them now, else as the harness layout has them.
template <bool LIVE>
__device__ __forceinline__ void mini_bodies(const FusedArgs& a, MiniSmem& ms, int u) {
    const GlobalTerms terms{a};
    const sbx_dense_scene& sc = a.sc;
    const sbx_motor_store& mot = sc.mot;
    const sbx_rigid_body& mb = mot.body;
    const int nB = a.nB;
    const int dpm = a.dpm, mpm = 2 * dpm, spm = 6 * dpm;
    const int m0 = u * mpm, s0 = u * spm, d0 = u * dpm;
    const int tid = threadIdx.x;
    float* sF = ms.sF;
    float* sT = ms.sT;
    LocalAcc acc{sF, sT, s0, spm};
    int odd = 0;
    if (tid < 32) {
        if (tid < mpm) {
            // CrossBridgeSystem.bondForces, then the head's sums: joint 1, then the bond
            int m = m0 + tid;
            float out[XB_STRIDE];
            bond_store(a, m, out);
            int hl = 3 * tid + 2;
            double f[3] = {0.0, 0.0, 0.0}, tq[3] = {0.0, 0.0, 0.0};
            motor_joint_apply(terms.joint(m, 1), 1, true, mot.nucleotideState[m], s0 + hl, nB, mb.uVec,
                              mb.segLength, mot.jointParams, f, tq);
            for (int k = 0; k < 3; k++) {
                float F = (float)(0.0 + f[k]), T = (float)(0.0 + tq[k]);
                sF[k * spm + hl] = F + out[k];
                sT[k * spm + hl] = T + out[3 + k];
            }
        }
    } else {
        const int role = (tid - 32) >> 5, ml = tid & 31;      // 0 rods, 1 levers
        if (ml < mpm) {
            const int s = joint_sums(a, ms, u, role, ml);
            int dl = ml >> 1, d = d0 + dl;
            bool isA = (ml & 1) == 0;            // motorA = 2d, motorB = 2d + 1
            if (role == 0) {
                couple_apply_rod(acc, s, isA, terms.couple(d, 0));
                couple_apply_rod(acc, s, isA, terms.couple(d, 1));
                if (isA) tether_apply(acc, s, terms.tether(d, odd));
            } else {
                bool bothBound = mot.boundSeg[2 * d] >= 0 && mot.boundSeg[2 * d + 1] >= 0;
                if (sc.dim.parallel[d] != 0 && !bothBound) couple_apply_lever(acc, s, isA, terms.lever(d));
            }
        }
    }
    if (LIVE) {
        if (__syncthreads_or(odd)) {
            odd_sums(a, ms, u);
            __syncthreads();
        }
    } else {
        asm volatile("bar.sync 1, 96;" ::: "memory");         // the three warps, without a fourth
    }
    // integrate + derive the sub-bodies; force-dot registry
    if (tid < spm) {
        int s = s0 + tid;
        float F[3] = {sF[tid], sF[spm + tid], sF[2 * spm + tid]};
        float T[3] = {sT[tid], sT[spm + tid], sT[2 * spm + tid]};
        integrate_derive_store(mb, s, F, T, mot.bodyParams[0]);
    }
    if (tid < mpm) {
        int m = m0 + tid;
        register_force_dot_one(m, sc.bondData, mot.boundSeg[m] >= 0, mot.forceDotFil, mot.forceMag,
                               mot.forceDotHist, mot.forceDotPlace);
    }
}

// dimer d's tether to backbone u by motor mA's rod, with its row
__device__ __forceinline__ void tether_term(const FusedArgs& a, int d, int u, int mA, bool odd) {
    const sbx_minifilament_store& mini = a.sc.mini;
    const sbx_rigid_body &mb = a.sc.mot.body, &bb = mini.backbone;
    TetherTerm T = tether_terms(a.nB, mb.coord, mb.uVec, mb.segLength, mb.bTransGam, mb.bRotGam, a.nBb, bb.coord,
                                bb.uVec, mini.bbInvDragY, u, mA, mini.attachAxial[d], mini.miniParams);
    GlobalTerms{a}.put(d, T, odd);
    float* o = mini.miniData + (int64_t)MINI_STRIDE * d;
    for (int j = 0; j < 6; j++) o[j] = T.row[j];
}
// (out of line: the layout's own term is made while the tables are read)
__device__ __noinline__ void odd_tether_term(const FusedArgs& a, int d, int u, int mA) {
    tether_term(a, d, u, mA, true);
}

// The position-only terms of the myosin mechanics, none of which depends on a step's binding or
// forces (MotorJointSystem.java:72-123 joint geometry, DimerCouplingSystem.java:99-182 end
// variants and lever torsion, MiniFilamentSystem tethers with their backbone reaction rows):
// item k of 2 nM + 4 nD, of the harness layout's dimers. LIVE: a dimer's tether item looks at the
// dimer tables as the device has them now, sets *a.odd where they are not the layout's and
// makes that tether from them (the rest: odd_sums); false where they name no motor or backbone.
template <bool LIVE>
__device__ __forceinline__ bool myosin_term(const FusedArgs& a, int k) {
    const sbx_dense_scene& sc = a.sc;
    const sbx_motor_store& mot = sc.mot;
    const sbx_rigid_body& mb = mot.body;
    const sbx_minifilament_store& mini = sc.mini;
    const int nM = a.nM, nD = a.nD, nB = a.nB;
    const GlobalTerms terms{a};
    if (k < 2 * nM) {
        const int which = k >= nM, m = k - which * nM;
        terms.put(m, which, motor_joint(m, which, nB, mb.coord, mb.uVec, mb.segLength, mb.bTransGam, mb.bRotGam,
                                        mot.jointParams));
    } else if (k < 2 * nM + 2 * nD) {
        const int v = k >= 2 * nM + nD, d = k - 2 * nM - v * nD;
        terms.put(d, v, couple_variant(nB, mb.coord, mb.uVec, mb.segLength, mb.bTransGam, mb.bRotGam, 2 * d, 2 * d + 1,
                                       sc.dim.parallel[d] != 0, sc.dim.dimerParams, v));
    } else if (k < 2 * nM + 3 * nD) {
        const int d = k - 2 * nM - 2 * nD;
        terms.put(d, couple_lever(nB, mb.uVec, mb.bRotGam, 2 * d, 2 * d + 1, sc.dim.dimerParams));
    } else {
        const int d = k - 2 * nM - 3 * nD, u = d / a.dpm;
        int h = u, r = 2 * d, mA = 2 * d, mB = 2 * d + 1;
        if (LIVE) { h = mini.headBackboneSlot[d]; r = mini.motorA[d]; mA = sc.dim.motorA[d]; mB = sc.dim.motorB[d]; }
        tether_term(a, d, u, 2 * d, false);
        // backbone CSR of the reference (rows = backbones, items = dimers in index order)
        mini.bbDimerList[d] = d;
        if (LIVE && (h != u || r != 2 * d || mA != 2 * d || mB != 2 * d + 1)) {
            *(volatile int*)a.odd = 1;
            const bool ok = h >= 0 && h < a.nBb && r >= 0 && r < nM && mA >= 0 && mA < nM && mB >= 0 && mB < nM;
            odd_tether_term(a, d, ok ? h : u, ok ? r : 2 * d);
            return ok;
        }
    }
    return true;
}

}  // namespace
