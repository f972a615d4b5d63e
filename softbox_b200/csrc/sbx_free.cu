// sbx_free.cu — free Brownian rods: the DiffusionHarness.cpuStepFdt step
// (DiffusionHarness.java:161-169: brownianForce -> integrate -> derive) advanced for many
// steps in ONE launch. Free rods do not interact, so each thread keeps its rod's pose in
// registers across steps and touches HBM only to load the rod once and store it once;
// the per-step work is the counter-keyed RNG, Box-Muller and the Langevin update. The
// arrays written at the end (pose, derived geometry, the last step's randForce /
// randTorque) equal running the three systems step by step.
#include <cuda_runtime.h>

#include "../../include/softbox_b200.h"
#include "sbx_internal.cuh"
#include "sbx_physics.cuh"
#include "sbx_trace.h"

using namespace sbx;

namespace {

// One rod's per-step inputs that do not depend on its pose: the six Gaussians of step t0 + s.
template <int MODE>   // 0 wang, 1 philox, 2 supplied
__device__ __forceinline__ void rod_gaussians(int n, int i, int t0, int s, int seed, uint64_t seed64,
                                              const float* noise, float g[6]) {
    if (MODE == 0) gauss6_wang(i, t0 + s, seed, g);
    else if (MODE == 1) gauss6_philox(i, t0 + s, seed64, g);
    else for (int k = 0; k < 6; k++) g[k] = noise[((int64_t)s * 6 + k) * n + i];
}

// A rod in registers: loaded once, stepped, stored once.
struct RodState {
    Pose p;
    float f[3], t[3], gT[3], gR[3], rf[3], rt[3], z[3];
    double c64[3];
    float tS, rS, mag, dt, L;
};

struct FreeArgs {
    int n;
    float* coord; double* coord64; float *uVec, *yVec, *zVec, *end1, *end2;
    const float *segLength, *F, *T;
    float *rF, *rT;
    const float *bTG, *bRG, *tSc, *rSc, *params;
    int* counts;
    int t0, nsteps;
    uint64_t seed64;
    const float* noise;
};

__device__ __forceinline__ void rod_load(const FreeArgs& a, int i, RodState& r) {
    const int n = a.n;
    for (int k = 0; k < 3; k++) {
        r.p.c[k] = a.coord[k * n + i]; r.p.u[k] = a.uVec[k * n + i]; r.p.y[k] = a.yVec[k * n + i];
        r.f[k] = a.F[k * n + i]; r.t[k] = a.T[k * n + i];
        r.gT[k] = a.bTG[k * n + i]; r.gR[k] = a.bRG[k * n + i];
        if (a.coord64) r.c64[k] = a.coord64[k * n + i];
        r.rf[k] = r.rt[k] = r.z[k] = 0.f;
    }
    r.tS = a.tSc[i]; r.rS = a.rSc[i]; r.mag = a.params[1]; r.dt = a.params[0]; r.L = a.segLength[i];
}

// the Langevin update and derived geometry of one step with the step's forces in rf / rt
__device__ __forceinline__ void rod_step(RodState& r, bool fp64) {
    Pose q;
    float dc[3];
    integrate_pose(r.p, r.f, r.t, r.rf, r.rt, r.gT, r.gR, r.dt, q, dc);
    if (fp64)
        for (int k = 0; k < 3; k++) { r.c64[k] = r.c64[k] + (double)dc[k]; q.c[k] = (float)r.c64[k]; }
    float e1[3], e2[3];                   // (the stored ones follow from the last pose: rod_store)
    derive_pose(q.c, q.u, q.y, r.z, e1, e2, r.L);
    r.p = q;
}

// rod_step with the step's body velocities in rf / rt
__device__ __forceinline__ void rod_step_vel(RodState& r, bool fp64) {
    Pose q;
    float dc[3], z[3];
    pose_normal(r.p, z);
    advance_pose(r.p, z, r.rf, r.rt, r.dt, q, dc);
    if (fp64)
        for (int k = 0; k < 3; k++) { r.c64[k] = r.c64[k] + (double)dc[k]; q.c[k] = (float)r.c64[k]; }
    float e1[3], e2[3];
    derive_pose(q.c, q.u, q.y, r.z, e1, e2, r.L);
    r.p = q;
}

__device__ __forceinline__ void rod_store(const FreeArgs& a, int i, const RodState& r) {
    const int n = a.n;
    const float half = r.L * 0.5f;        // derive_pose's ends: c -/+ (L/2) u
    for (int k = 0; k < 3; k++) {
        a.coord[k * n + i] = r.p.c[k]; a.uVec[k * n + i] = r.p.u[k]; a.yVec[k * n + i] = r.p.y[k];
        a.zVec[k * n + i] = r.z[k];
        a.end1[k * n + i] = r.p.c[k] - half * r.p.u[k]; a.end2[k * n + i] = r.p.c[k] + half * r.p.u[k];
        if (a.coord64) a.coord64[k * n + i] = r.c64[k];
    }
    if (i == 0) a.counts[1] = a.t0 + a.nsteps - 1;
}

// one thread a rod: each step's draw, then its update
template <int MODE>
__global__ void __launch_bounds__(128) k_free_rods(const FreeArgs a) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.n) return;
    RodState r;
    rod_load(a, i, r);
    const int seed = a.counts[2];
    for (int s = 0; s < a.nsteps; s++) {
        float g[6];
        rod_gaussians<MODE>(a.n, i, a.t0, s, seed, a.seed64, a.noise, g);
        brownian_amplitudes(g, r.tS, r.rS, r.mag, r.gT, r.gR, r.rf, r.rt);
        rod_step(r, a.coord64 != nullptr);
    }
    rod_store(a, i, r);
    for (int k = 0; k < 3; k++) { a.rF[k * a.n + i] = r.rf[k]; a.rT[k * a.n + i] = r.rt[k]; }
}

// A block of RODS rods: warp 0 steps them, one rod a lane, while the other warps draw the forces
// of the next chunk of steps into shared memory. The draws are keyed by (rod, step) and do not
// depend on the pose, so only the update (three square roots and divisions in a row) is left
// on a rod's serial chain; the draw (three Box-Muller pairs in FP64, most of a step's work)
// spreads over the block. For a rod without external force and torque the drawing threads
// also make its body velocities (six more divisions off the chain): with F = T = 0 the body
// forces are sums of zeros and the draw, so they equal the draw wherever it is not zero.
// 1,024 rods take 0.43 us a step, one thread a rod 1.67 us.
template <int RODS>
struct PipeShape {
    static constexpr int STEPS = 256 / RODS;                 // steps of a chunk: 256 draws
    static constexpr int THREADS = 32 + 256;                 // the stepping warp, one thread a draw
};

__device__ __forceinline__ bool all_zero(const float f[3], const float t[3]) {
    return f[0] == 0.f && f[1] == 0.f && f[2] == 0.f && t[0] == 0.f && t[1] == 0.f && t[2] == 0.f;
}

template <int MODE, int RODS>
__global__ void __launch_bounds__(PipeShape<RODS>::THREADS) k_free_pipe(const FreeArgs a) {
    constexpr int STEPS = PipeShape<RODS>::STEPS;
    __shared__ float buf[2][STEPS][6][RODS];
    __shared__ unsigned char vel[2][STEPS][RODS];            // buf holds body velocities, not forces
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int first = blockIdx.x * RODS;
    const int seed = a.counts[2];
    const int chunks = (a.nsteps + STEPS - 1) / STEPS;
    const bool steps = warp == 0 && lane < RODS && first + lane < a.n;
    RodState r;
    if (steps) rod_load(a, first + lane, r);
    // the drawing threads: rod (threadIdx - 32) % RODS, step (threadIdx - 32) / RODS of a chunk
    const int d = (int)threadIdx.x - 32, dr = d & (RODS - 1), ds = d / RODS;
    const int di = first + dr;
    const bool draws = warp > 0 && di < a.n;
    float gT[3], gR[3], tS = 0.f, rS = 0.f, mag = 0.f;
    bool loose = false;                                      // the rod has no external force or torque
    if (draws) {
        float f[3], t[3];
        for (int k = 0; k < 3; k++) {
            gT[k] = a.bTG[k * a.n + di]; gR[k] = a.bRG[k * a.n + di];
            f[k] = a.F[k * a.n + di]; t[k] = a.T[k * a.n + di];
        }
        tS = a.tSc[di]; rS = a.rSc[di]; mag = a.params[1];
        loose = all_zero(f, t);
    }
    for (int c = 0; c <= chunks; c++) {
        if (draws && c < chunks) {
            const int s = c * STEPS + ds;
            if (s < a.nsteps) {
                float g[6], rf[3], rt[3];
                rod_gaussians<MODE>(a.n, di, a.t0, s, seed, a.seed64, a.noise, g);
                brownian_amplitudes(g, tS, rS, mag, gT, gR, rf, rt);
                if (s == a.nsteps - 1)
                    for (int k = 0; k < 3; k++) { a.rF[k * a.n + di] = rf[k]; a.rT[k * a.n + di] = rt[k]; }
                const bool v = loose && rf[0] != 0.f && rf[1] != 0.f && rf[2] != 0.f && rt[0] != 0.f &&
                               rt[1] != 0.f && rt[2] != 0.f;
                vel[c & 1][ds][dr] = v;
                for (int k = 0; k < 3; k++) {
                    buf[c & 1][ds][k][dr] = v ? 1.0e6f * rf[k] / gT[k] : rf[k];
                    buf[c & 1][ds][3 + k][dr] = v ? rt[k] / gR[k] : rt[k];
                }
            }
        }
        if (steps && c > 0) {
            const int left = a.nsteps - (c - 1) * STEPS, m = left < STEPS ? left : STEPS;
            for (int s = 0; s < m; s++) {
                for (int k = 0; k < 3; k++) { r.rf[k] = buf[(c - 1) & 1][s][k][lane]; r.rt[k] = buf[(c - 1) & 1][s][3 + k][lane]; }
                if (vel[(c - 1) & 1][s][lane]) rod_step_vel(r, a.coord64 != nullptr);
                else rod_step(r, a.coord64 != nullptr);
            }
        }
        __syncthreads();
    }
    if (steps) rod_store(a, first + lane, r);                // (the last step's forces: stored by its draw)
}

// Rods a block of the pipeline, 0 for one thread a rod. As few rods a block as give at most two
// blocks an SM, else 32. Its registers let two blocks on an SM (three with supplied noise), so up
// to there it leads from a few steps on; more blocks follow one another, and then the steps
// must be worth the filling of the pipeline twice, up to where the draws fill the GPU anyway.
// us a call, pipeline / one thread a rod (rods without, and with, external forces; the former
// also leave the velocities to the drawing warps), on 148 SMs:
//   4,736 rods, Philox        8 steps 18 / 25, 20 / 25     32 steps 31 / 66, 38 / 66
//   9,472 (two blocks an SM)  8 steps 18 / 25, 20 / 25     32 steps 32 / 66, 38 / 66
//   14,208 (three)            8 steps 22 / 24, 26 / 24     16 steps 30 / 37, 36.5 / 37
//   18,944 (four)             8 steps 23 / 24, 26 / 24     24 steps 42 / 50, 51.5 / 50.5
//   14,208, supplied noise   16 steps 41 / 44, 41 / 41    100 steps 90 / 116, 112 / 116
//   18,944, supplied noise   16 steps 46 / 41, 54 / 40     64 steps 102 / 88, 131 / 88
constexpr int pipe_rods(int n, int nsteps, int sms, bool supplied) {
    const int64_t wave = (int64_t)32 * sms;            // rods at one block of 32 an SM
    if (n > 4 * wave || (supplied && n > 3 * wave) || nsteps > 0x7fffffff - 64) return 0;
    if (nsteps < (n <= 2 * wave ? 4 : n <= 3 * wave ? 16 : 24)) return 0;
    return n <= 16 * (int64_t)sms ? 8 : n <= 32 * (int64_t)sms ? 16 : 32;
}
static_assert(pipe_rods(2368, 4, 148, false) == 8 && pipe_rods(2369, 4, 148, true) == 16 &&
              pipe_rods(4737, 4, 148, false) == 32 && pipe_rods(2368, 3, 148, false) == 0, "few rods");
static_assert(pipe_rods(9473, 15, 148, false) == 0 && pipe_rods(9473, 16, 148, true) == 32 &&
              pipe_rods(14209, 23, 148, false) == 0 && pipe_rods(14209, 24, 148, false) == 32 &&
              pipe_rods(14209, 1000, 148, true) == 0 && pipe_rods(18945, 1000, 148, false) == 0, "more than two blocks an SM");
static_assert(pipe_rods(1, 0x7fffffff, 148, false) == 0, "a step index past the chunks");

template <int MODE>
void free_launch(sbx_ctx* ctx, const FreeArgs& a) {
    int sms = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device) != cudaSuccess) sms = 0;
    switch (pipe_rods(a.n, a.nsteps, sms, MODE == 2)) {
    case 8: SBX_LAUNCH(ctx, (k_free_pipe<MODE, 8>), blocks(a.n, 8), PipeShape<8>::THREADS, a); break;
    case 16: SBX_LAUNCH(ctx, (k_free_pipe<MODE, 16>), blocks(a.n, 16), PipeShape<16>::THREADS, a); break;
    case 32: SBX_LAUNCH(ctx, (k_free_pipe<MODE, 32>), blocks(a.n, 32), PipeShape<32>::THREADS, a); break;
    default: SBX_LAUNCH(ctx, k_free_rods<MODE>, blocks(a.n, 128), 128, a);
    }
}

}  // namespace

extern "C" sbx_status sbx_free_rods_run(sbx_ctx* ctx, sbx_filament_store* fil, int32_t t0, int32_t nsteps,
                                        int32_t noise_mode, uint64_t philox_seed, const float* noise) {
    SBX_TRACE("sbx.free.run");
    if (!ctx || !fil || nsteps < 0 || noise_mode < 0 || noise_mode > 2) return SBX_EINVAL;
    const sbx_rigid_body& b = fil->body;
    int n = b.n;
    if (n <= 0 || nsteps == 0) return SBX_OK;
    if (!b.coord || !b.uVec || !b.yVec || !b.zVec || !b.end1 || !b.end2 || !b.segLength || !b.forceSum ||
        !b.torqueSum || !b.randForce || !b.randTorque || !b.bTransGam || !b.bRotGam || !b.brownTransScale ||
        !b.brownRotScale || !fil->params || !fil->counts)
        return fail(ctx, SBX_EINVAL, "sbx_free_rods_run: null array");
    if (noise_mode == 2) {
        if (!noise) return fail(ctx, SBX_EINVAL, "sbx_free_rods_run: supplied noise is null");
        bool bad = false;
        sbx_status st = any_nonfinite(ctx, noise, (int64_t)nsteps * 6 * n, &bad);
        if (st) return st;
        if (bad) return fail(ctx, SBX_ENONFINITE, "sbx_free_rods_run: noise holds NaN/Inf");
    }
    FreeArgs a{n, b.coord, b.coord64, b.uVec, b.yVec, b.zVec, b.end1, b.end2, b.segLength, b.forceSum, b.torqueSum,
               b.randForce, b.randTorque, b.bTransGam, b.bRotGam, b.brownTransScale, b.brownRotScale, fil->params,
               fil->counts, t0, nsteps, philox_seed, noise};
    if (noise_mode == 0) free_launch<0>(ctx, a);
    else if (noise_mode == 1) free_launch<1>(ctx, a);
    else free_launch<2>(ctx, a);
    return check_launch(ctx, "sbx_free_rods_run");
}
