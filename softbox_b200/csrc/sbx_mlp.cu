// sbx_mlp.cu — the surrogate ensemble's kernels: BF16 GEMMs on the 5th-generation tensor
// cores (tcgen05.mma, FP32 accumulators in tensor memory) with fused bias / GELU / transpose
// epilogues, and the small elementwise kernels of training (loss gradient, GELU backward,
// bias gradients, Adam).
//
// GEMM: C[M x N] = A[M x K] . B[N x K]^T, A and B row-major BF16 (K contiguous, "K-major"),
// K <= 256. One CTA (16 warps) per SM keeps its B tile (up to 256 columns) in shared memory
// and loops over 128-row tiles of C, staging the next tile's A while the current tile's
// epilogue runs: the A and B tiles are staged in shared memory in the
// canonical no-swizzle K-major layout (8 x 16-byte core matrices; core matrix (row group g,
// k group c) at ((g * Kp/8) + c) * 128 bytes), one thread issues K/16 MMAs (M = 128, N = the
// tile width) into TMEM and commits them to an mbarrier, and the epilogue reads the
// accumulators back with tcgen05.ld: warp w takes TMEM lanes (rows) 32 (w mod 4) .. +31 and
// every fourth 16-column chunk from chunk w / 4, adds the bias, applies GELU and writes each
// row's 16 values with vector stores (the transposed output by lanes along the rows).
// blockIdx.z selects an independent problem (an ensemble member) by strides.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "../../include/softbox_b200.h"
#include "sbx_internal.cuh"

namespace {

constexpr int MT = 128;              // rows of a C tile (the MMA's M)
constexpr int NT = 256;              // max columns of a C tile (the MMA's N)
constexpr int KMAX = 256;            // max contraction length
constexpr int GEMM_THREADS = 512;   // 16 warps: 4 TMEM lane quarters x 4 column groups
constexpr int COL_GROUPS = GEMM_THREADS / 128;
constexpr long long WAIT_NS = 1000000000LL;

__device__ __forceinline__ unsigned smem_u32(const void* p) {
    return (unsigned)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ long long gtimer() {
    long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// canonical K-major no-swizzle shared-memory descriptor (sm_100 version bits = 1)
__device__ __forceinline__ unsigned long long kmajor_desc(unsigned addr, unsigned lbo, unsigned sbo) {
    return (unsigned long long)((addr >> 4) & 0x3FFFu) | ((unsigned long long)((lbo >> 4) & 0x3FFFu) << 16) |
           ((unsigned long long)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

// kind::f16 instruction descriptor: F32 accumulate, BF16 A and B, both K-major, M x N
__host__ __device__ constexpr unsigned idesc_bf16(int M, int N) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(N >> 3) << 17) | ((unsigned)(M >> 4) << 24);
}

__device__ __forceinline__ float gelu(float x) { return 0.5f * x * (1.0f + erff(x * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_grad(float x) {
    return 0.5f * (1.0f + erff(x * 0.70710678118654752f)) + x * 0.39894228040143268f * expf(-0.5f * x * x);
}

struct GemmArgs {
    int M, N, K;
    const __nv_bfloat16* A; int lda; long long sA;
    const __nv_bfloat16* B; int ldb; long long sB;
    const float* bias; long long sBias;
    int act;
    __nv_bfloat16* out; int ldo; long long sOut;
    __nv_bfloat16* outT; int ldt; long long sOutT;
    float* outF; int ldf; long long sOutF;
    int* err;
};

// rows [r0, r0 + rows) x [0, Kp) of a row-major BF16 matrix into the core-matrix layout;
// rows past `rowsValid` and columns past K are zero. Aligned 16-byte pieces go by cp.async
// (every thread keeps all its copies in flight), the rest by plain loads; the caller waits
// with cp_async_wait_all() before the block barrier.
__device__ void stage(char* dst, const __nv_bfloat16* src, int ld, int r0, int rows, int rowsValid, int K, int Kp,
                      bool vec) {
    int kg = Kp >> 3;
    for (int u = threadIdx.x; u < rows * kg; u += GEMM_THREADS) {
        int r = u / kg, c = u - r * kg;
        int gr = r0 + r, k0 = c * 8;
        char* d = dst + ((r >> 3) * kg + c) * 128 + (r & 7) * 16;
        if (gr < rowsValid && vec && k0 + 8 <= K) {
            const __nv_bfloat16* p = src + (long long)gr * ld + k0;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(d)), "l"(p));
            continue;
        }
        uint4 v = make_uint4(0, 0, 0, 0);
        if (gr < rowsValid) {
            const __nv_bfloat16* p = src + (long long)gr * ld + k0;
            unsigned short h[8];
            for (int j = 0; j < 8; j++) h[j] = (k0 + j < K) ? __bfloat16_as_ushort(p[j]) : (unsigned short)0;
            v = make_uint4(h[0] | (unsigned)h[1] << 16, h[2] | (unsigned)h[3] << 16, h[4] | (unsigned)h[5] << 16,
                           h[6] | (unsigned)h[7] << 16);
        }
        *reinterpret_cast<uint4*>(d) = v;
    }
}

__device__ __forceinline__ void cp_async_wait_all() {
    asm volatile("cp.async.commit_group;");
    asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// One CTA keeps its B tile (up to 256 x 256 BF16) in shared memory and loops over M tiles
// blockIdx.x, blockIdx.x + gridDim.x, ...: per tile it stages A, issues the MMA chain into
// TMEM, waits for the tile's commit (mbarrier phase = tile iteration parity) and runs the
// epilogue, then syncs before the next tile's MMAs overwrite the accumulators.
__global__ void __launch_bounds__(GEMM_THREADS, 1) k_gemm(GemmArgs g) {
    extern __shared__ __align__(1024) char smem[];
    const int z = blockIdx.z;
    const int n0 = blockIdx.y * NT;
    const int nCols = min(NT, g.N - n0);
    const int Np = (nCols + 15) & ~15;             // MMA N: a multiple of 16 for M = 128
    const int Kp = (g.K + 15) & ~15;
    const int tilesM = (g.M + MT - 1) / MT;
    char* sA = smem;
    char* sB = smem + MT * Kp * 2;
    unsigned long long* mbar = reinterpret_cast<unsigned long long*>(sB + NT * Kp * 2);
    unsigned* tmemSlot = reinterpret_cast<unsigned*>(mbar + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    unsigned ncolsAlloc = 32;
    while ((int)ncolsAlloc < Np) ncolsAlloc <<= 1;

    if (threadIdx.x == 0)
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(mbar)));
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmemSlot)),
                     "r"(ncolsAlloc));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    const __nv_bfloat16* A = g.A + z * g.sA;
    const __nv_bfloat16* B = g.B + z * g.sB;
    bool vecA = (g.lda % 8 == 0) && (((uintptr_t)A & 15) == 0);
    bool vecB = (g.ldb % 8 == 0) && (((uintptr_t)B & 15) == 0);
    stage(sB, B, g.ldb, n0, Np, g.N, g.K, Kp, vecB);
    const float* bias = g.bias ? g.bias + z * g.sBias : nullptr;
    __nv_bfloat16* out = g.out ? g.out + z * g.sOut : nullptr;
    __nv_bfloat16* outT = g.outT ? g.outT + z * g.sOutT : nullptr;
    float* outF = g.outF ? g.outF + z * g.sOutF : nullptr;
    // 16-byte row stores where every row start is 16-byte aligned
    const bool vecOut = out && (g.ldo % 8 == 0) && (((uintptr_t)out & 15) == 0);
    const bool vecOutF = outF && (g.ldf % 4 == 0) && (((uintptr_t)outF & 15) == 0);
    const int quarter = warp & 3, cgroup = warp >> 2;
    bool ok = true;
    unsigned tmem = 0;

    int iter = 0;
    if ((int)blockIdx.x < tilesM) stage(sA, A, g.lda, (int)blockIdx.x * MT, MT, g.M, g.K, Kp, vecA);
    for (int tile = blockIdx.x; tile < tilesM && ok; tile += gridDim.x, iter++) {
        const int m0 = tile * MT;
        // this tile's A was staged before the previous tile's epilogue (or above)
        cp_async_wait_all();
        asm volatile("fence.proxy.async.shared::cta;");
        asm volatile("tcgen05.fence::before_thread_sync;");
        __syncthreads();
        asm volatile("tcgen05.fence::after_thread_sync;");
        tmem = *tmemSlot;
        if (threadIdx.x == 0) {
            const unsigned idesc = idesc_bf16(MT, Np);
            const unsigned aBase = smem_u32(sA), bBase = smem_u32(sB);
            const unsigned sbo = (unsigned)(Kp >> 3) * 128u;
            for (int kk = 0; kk < Kp / 16; kk++) {
                unsigned long long ad = kmajor_desc(aBase + kk * 256u, 128u, sbo);
                unsigned long long bd = kmajor_desc(bBase + kk * 256u, 128u, sbo);
                unsigned acc = kk > 0 ? 1u : 0u;
                asm volatile(
                    "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                    "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem),
                    "l"(ad), "l"(bd), "r"(idesc), "r"(acc));
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                smem_u32(mbar)));
        }
        // bounded wait for this tile's MMAs: phase `iter` of the barrier
        {
            const unsigned parity = (unsigned)(iter & 1);
            bool done_ok = false;
            long long t0 = gtimer();
            for (;;) {
                unsigned done;
                asm volatile(
                    "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                    "selp.u32 %0, 1, 0, p;\n\t}"
                    : "=r"(done)
                    : "r"(smem_u32(mbar)), "r"(parity));
                if (done) { done_ok = true; break; }
                if (gtimer() - t0 > WAIT_NS) break;
            }
            ok = __syncthreads_and(done_ok ? 1 : 0) != 0;   // one verdict for the whole CTA
        }
        if (!ok && threadIdx.x == 0 && g.err) atomicOr(g.err, 1);
        asm volatile("tcgen05.fence::after_thread_sync;");
        // the MMAs have read A: stage the next tile's A while this tile's epilogue runs
        if (ok && tile + (int)gridDim.x < tilesM)
            stage(sA, A, g.lda, (tile + (int)gridDim.x) * MT, MT, g.M, g.K, Kp, vecA);
        if (ok) {
            const int row = m0 + quarter * 32 + lane;
            for (int c0 = cgroup * 16; c0 < Np; c0 += COL_GROUPS * 16) {
                unsigned r[16];
                unsigned taddr = tmem + ((unsigned)(quarter * 32) << 16) + (unsigned)c0;
                asm volatile(
                    "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, "
                    "[%16];"
                    : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                      "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]),
                      "=r"(r[15])
                    : "r"(taddr));
                asm volatile("tcgen05.wait::ld.sync.aligned;");
                const int nb = n0 + c0;                    // this chunk's first column
                float v[16], a[16];
#pragma unroll
                for (int j = 0; j < 16; j++) {
                    v[j] = __uint_as_float(r[j]);
                    if (bias && nb + j < g.N) v[j] += bias[nb + j];
                    a[j] = g.act ? gelu(v[j]) : v[j];
                }
                if (outT) {
#pragma unroll
                    for (int j = 0; j < 16; j++)
                        if (row < g.M && nb + j < g.N) outT[(long long)(nb + j) * g.ldt + row] = __float2bfloat16_rn(a[j]);
                }
                if (row < g.M) {
                    const bool full = nb + 16 <= g.N;
                    if (out) {
                        __nv_bfloat16* o = out + (long long)row * g.ldo + nb;
                        if (vecOut && full) {
                            unsigned w[8];
#pragma unroll
                            for (int j = 0; j < 8; j++) {
                                __nv_bfloat162 h = __floats2bfloat162_rn(a[2 * j], a[2 * j + 1]);
                                w[j] = *reinterpret_cast<unsigned*>(&h);
                            }
                            reinterpret_cast<uint4*>(o)[0] = make_uint4(w[0], w[1], w[2], w[3]);
                            reinterpret_cast<uint4*>(o)[1] = make_uint4(w[4], w[5], w[6], w[7]);
                        } else {
                            for (int j = 0; j < 16; j++)
                                if (nb + j < g.N) o[j] = __float2bfloat16_rn(a[j]);
                        }
                    }
                    if (outF) {
                        float* o = outF + (long long)row * g.ldf + nb;
                        if (vecOutF && full) {
#pragma unroll
                            for (int j = 0; j < 4; j++)
                                reinterpret_cast<float4*>(o)[j] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2],
                                                                              v[4 * j + 3]);
                        } else {
                            for (int j = 0; j < 16; j++)
                                if (nb + j < g.N) o[j] = v[j];
                        }
                    }
                }
            }
        }
        // every warp is done with sA and the accumulators before the next tile
        asm volatile("tcgen05.fence::before_thread_sync;");
        __syncthreads();
    }
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;");
        tmem = *tmemSlot;
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(ncolsAlloc));
    }
}

// ---------------------------------------------------------------- whole networks
// The ensemble's networks as the whole-network kernels take them: layer l is Np[l] x Kp[l]
// (inputs and outputs padded to 16), arrays hold nz networks one after another.
constexpr int NET_MAX_LAYERS = 8;
struct Net {
    int nz, L, nin, nout;
    int Kp[NET_MAX_LAYERS], Np[NET_MAX_LAYERS];
    const __nv_bfloat16* Wb[NET_MAX_LAYERS];
    const float* b[NET_MAX_LAYERS];
};

// one 128 x N x Kp product from the staged operands into tensor memory, issued by one thread;
// the commit arrives on mbar
__device__ __forceinline__ void issue_mma(unsigned tmem, unsigned aBase, unsigned bBase, int N, int Kp,
                                          unsigned long long* mbar) {
    const unsigned idesc = idesc_bf16(MT, N);
    const unsigned sbo = (unsigned)(Kp >> 3) * 128u;
    for (int kk = 0; kk < Kp / 16; kk++) {
        unsigned long long ad = kmajor_desc(aBase + kk * 256u, 128u, sbo);
        unsigned long long bd = kmajor_desc(bBase + kk * 256u, 128u, sbo);
        unsigned acc = kk > 0 ? 1u : 0u;
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem),
            "l"(ad), "l"(bd), "r"(idesc), "r"(acc));
    }
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
        smem_u32(mbar)));
}

// bounded wait for phase `parity` of mbar; one verdict for the block
__device__ __forceinline__ bool wait_mma(unsigned long long* mbar, unsigned parity) {
    bool done_ok = false;
    long long t0 = gtimer();
    for (;;) {
        unsigned done;
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(smem_u32(mbar)), "r"(parity));
        if (done) { done_ok = true; break; }
        if (gtimer() - t0 > WAIT_NS) break;
    }
    return __syncthreads_and(done_ok ? 1 : 0) != 0;
}

// 16 accumulator columns of this warp's 32 rows (TMEM lanes 32 * quarter ..): the load is
// issued here, its registers are valid after acc_wait
__device__ __forceinline__ void acc_load16(unsigned tmem, int quarter, int c0, unsigned r[16]) {
    unsigned taddr = tmem + ((unsigned)(quarter * 32) << 16) + (unsigned)c0;
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, "
        "[%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
}
// waits for the warp's loads; the registers pass through, so that no use moves before it
__device__ __forceinline__ void acc_wait(unsigned r[16], float v[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                   "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]),
                   "+r"(r[15])::"memory");
#pragma unroll
    for (int j = 0; j < 16; j++) v[j] = __uint_as_float(r[j]);
}
__device__ __forceinline__ float4 load_acc4(unsigned tmem, int quarter, int c0) {
    unsigned r[4];
    unsigned taddr = tmem + ((unsigned)(quarter * 32) << 16) + (unsigned)c0;
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3])::"memory");
    return make_float4(__uint_as_float(r[0]), __uint_as_float(r[1]), __uint_as_float(r[2]), __uint_as_float(r[3]));
}
__device__ __forceinline__ void load_acc16(unsigned tmem, int quarter, int c0, float v[16]) {
    unsigned r[16];
    acc_load16(tmem, quarter, c0, r);
    acc_wait(r, v);
}

__device__ __forceinline__ void pack16(const float a[16], uint4& lo, uint4& hi) {
    unsigned w[8];
#pragma unroll
    for (int j = 0; j < 8; j++) {
        __nv_bfloat162 h = __floats2bfloat162_rn(a[2 * j], a[2 * j + 1]);
        w[j] = *reinterpret_cast<unsigned*>(&h);
    }
    lo = make_uint4(w[0], w[1], w[2], w[3]);
    hi = make_uint4(w[4], w[5], w[6], w[7]);
}

// byte offset of element (r, c) of a staged operand with contraction length Kp
__device__ __forceinline__ int core_at(int r, int c, int Kp) {
    return ((r >> 3) * (Kp >> 3) + (c >> 3)) * 128 + (r & 7) * 16 + (c & 7) * 2;
}

// rows [0, rows) x [0, Kp) of a row-major BF16 matrix (16-byte aligned rows, rows a multiple of
// 8) into the core-matrix layout by 16-byte async copies; rows past rowsValid are zero. Item u
// is row u & 7 of core matrix u >> 3, so the shared addresses run with u and a warp's copies
// meet no bank twice (the copies' latency bounds it: with the columns along the lanes, and all
// copies on one bank, a pass took the same time).
__device__ __forceinline__ void stage_rows(char* dst, const __nv_bfloat16* src, int ld, int rows, int rowsValid,
                                           int Kp) {
    const int kg = Kp >> 3, r8 = threadIdx.x & 7, step = blockDim.x >> 3, cores = (rows >> 3) * kg;
    // a thread keeps its 8 columns where the block holds whole rows of core matrices
    const bool even = step % kg == 0;
    int v = threadIdx.x >> 3, rg = v / kg, c = v - rg * kg;
    const int dr = step / kg;
    for (; v < cores; v += step) {
        if (!even) { rg = v / kg; c = v - rg * kg; }
        const int r = rg * 8 + r8;
        char* d = dst + v * 128 + r8 * 16;
        if (r < rowsValid) {
            const __nv_bfloat16* p = src + (long long)r * ld + c * 8;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(d)), "l"(p));
        } else {
            *reinterpret_cast<uint4*>(d) = make_uint4(0, 0, 0, 0);
        }
        rg += dr;
    }
}

// ---------------------------------------------------------------- prediction
// Every layer of every network for 128 points a tile, in one launch: the activations of the
// tile stay in shared memory between layers (BF16, as the GEMM path stores them), a whole
// layer's weights sit beside them, and the next layer's are fetched while the epilogue runs.
// What bounds it is the epilogue: GELU on 1,024 hidden values a point and network, some 30
// instructions each, an order of magnitude above the MMAs' time. So one block of 16 warps an
// SM does the epilogues back to back; the separate GEMMs moved each layer's activations
// through memory and left normalisation, de-normalisation and the ensemble statistics to the
// host. 100,000 points on 5 networks: 1.13 ms, and 1.63 ms in ten GEMMs before (17 ms a call with
// the host's part, 2.4 ms now).
// The inputs are normalised here ((x - mean) / std in FP64, then FP32, then BF16) and the
// outputs de-normalised in FP64 (y * std + mean), operation for operation as the host does.
struct PredictArgs {
    Net net;
    const double *X, *xMean, *xStd, *yMean, *yStd;
    int P;
    double* out;      // [2 + nz][P][nout]: mean, standard deviation, each network's outputs
    int* err;
};

__global__ void __launch_bounds__(GEMM_THREADS, 1) k_predict(const __grid_constant__ PredictArgs g) {
    extern __shared__ __align__(1024) char smem[];
    char* sA = smem;                               // 128 x 256
    char* sB = smem + MT * KMAX * 2;               // 256 x 256
    __shared__ __align__(8) unsigned long long mbar;
    __shared__ unsigned tmemSlot;
    __shared__ float sBias[2][NT];
    const Net& net = g.net;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, quarter = warp & 3, cgroup = warp >> 2;
    const int tiles = (g.P + MT - 1) / MT, z = blockIdx.y, L = net.L;
    if (threadIdx.x == 0) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&mbar)));
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmemSlot)),
                     "r"(256));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    auto weights = [&](int l, int slot) {
        stage_rows(sB, net.Wb[l] + (long long)z * net.Np[l] * net.Kp[l], net.Kp[l], net.Np[l], net.Np[l], net.Kp[l]);
        if ((int)threadIdx.x < net.Np[l]) sBias[slot][threadIdx.x] = net.b[l][z * net.Np[l] + threadIdx.x];
    };
    bool ok = true;
    unsigned phase = 0;                            // the barrier's phase, and the bias slot in use
    if ((int)blockIdx.x < tiles) weights(0, 0);
    for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
        const int m0 = tile * MT;
        // the tile's inputs: 16 padded columns, thread (row, half)
        if (threadIdx.x < 2 * MT) {
            const int r = threadIdx.x >> 1, c0 = (threadIdx.x & 1) * 8, row = m0 + r;
            unsigned short h[8];
#pragma unroll
            for (int j = 0; j < 8; j++) {
                float x = 0.f;
                if (row < g.P && c0 + j < net.nin)
                    x = (float)((g.X[(long long)row * net.nin + c0 + j] - g.xMean[c0 + j]) / g.xStd[c0 + j]);
                h[j] = __bfloat16_as_ushort(__float2bfloat16_rn(x));
            }
            *reinterpret_cast<uint4*>(sA + core_at(r, c0, 16)) =
                make_uint4(h[0] | (unsigned)h[1] << 16, h[2] | (unsigned)h[3] << 16, h[4] | (unsigned)h[5] << 16,
                           h[6] | (unsigned)h[7] << 16);
        }
        for (int l = 0; l < L && ok; l++) {
            const int Np = net.Np[l], Kp = net.Kp[l];
            const bool last = l == L - 1;
            cp_async_wait_all();                           // this layer's weights
            asm volatile("fence.proxy.async.shared::cta;");
            asm volatile("tcgen05.fence::before_thread_sync;");
            __syncthreads();
            asm volatile("tcgen05.fence::after_thread_sync;");
            const unsigned tmem = tmemSlot;
            if (threadIdx.x == 0) issue_mma(tmem, smem_u32(sA), smem_u32(sB), Np, Kp, &mbar);
            ok = wait_mma(&mbar, phase);
            const float* bias = sBias[phase];
            phase ^= 1u;
            if (!ok && threadIdx.x == 0 && g.err) atomicOr(g.err, 1);
            asm volatile("tcgen05.fence::after_thread_sync;");
            if (!ok) break;
            // the product has read both operands: fetch the next weights, then the epilogue
            if (!last) weights(l + 1, phase);
            else if (tile + (int)gridDim.x < tiles) weights(0, phase);
            const int r = quarter * 32 + lane, row = m0 + r;
            unsigned acc[16];
            if (cgroup * 16 < Np) acc_load16(tmem, quarter, cgroup * 16, acc);
            for (int c0 = cgroup * 16; c0 < Np; c0 += COL_GROUPS * 16) {
                float v[16];
                acc_wait(acc, v);
                // the next columns are on their way while these are worked on
                if (c0 + COL_GROUPS * 16 < Np) acc_load16(tmem, quarter, c0 + COL_GROUPS * 16, acc);
#pragma unroll
                for (int j = 0; j < 16; j++) v[j] += bias[c0 + j];
                if (!last) {
#pragma unroll
                    for (int j = 0; j < 16; j++) v[j] = gelu(v[j]);
                    uint4 lo, hi;
                    pack16(v, lo, hi);
                    *reinterpret_cast<uint4*>(sA + core_at(r, c0, Np)) = lo;
                    *reinterpret_cast<uint4*>(sA + core_at(r, c0 + 8, Np)) = hi;
                } else if (row < g.P) {
                    double* o = g.out + ((long long)(2 + z) * g.P + row) * net.nout;
                    for (int j = 0; j < 16; j++)
                        if (c0 + j < net.nout) o[c0 + j] = (double)v[j] * g.yStd[c0 + j] + g.yMean[c0 + j];
                }
            }
        }
    }
    cp_async_wait_all();
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmemSlot), "r"(256));
    }
}

// the ensemble's mean and (population) standard deviation of every output, networks in order
__global__ void k_predict_stats(int nz, long long n, double* out) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double* y = out + 2 * n;
    double s = y[i];
    for (int z = 1; z < nz; z++) s += y[z * n + i];
    const double mean = s / (double)nz;
    double q = 0.0;
    for (int z = 0; z < nz; z++) {
        const double d = y[z * n + i] - mean;
        q = z == 0 ? d * d : q + d * d;
    }
    out[i] = mean;
    out[n + i] = sqrt(q / (double)nz);
}

// ---------------------------------------------------------------- training
// Whole Adam steps of the ensemble in one cooperative launch. A network's blocks (gridDim.x of
// them, all resident) work on its passes together and meet at a barrier of their own
// after each: L forward products, then for each layer from the last the input gradient
// together with the weight gradient and Adam update of the layer above it (whose weights
// nothing reads any more). Every product is split into 128 x 32 tiles; the epilogues take in
// what the separate kernels passed through memory: bias and GELU, the loss gradient, the GELU
// gradient, Adam with the BF16 copies; the bias gradients are summed from the staged operand
// in row order. The arithmetic, element by element, is that of the separate kernels.
// What bounds it is latency: per pass an operand fetch from L2, a short MMA chain, an
// epilogue and a barrier. As 42 launches a step the host's calls bounded it: 551 us a step of 5 networks at a batch of 256,
// 110 us now.
constexpr int TRAIN_THREADS = 256;
constexpr int TRAIN_N = 32;                        // columns of a tile
constexpr int TRAIN_STEPS = 64;                    // steps a launch takes (the bias corrections are arguments)
struct TrainArgs {
    Net net;
    int B, nsteps;
    const float *X, *Y;                            // [points][nin], [points][nout], normalised
    const long long* idx;                          // [nz][idxStride] points of each network's steps, or null:
    long long idxStride;                           //   network z's row r is point z * B + r
    float *W[NET_MAX_LAYERS], *bias[NET_MAX_LAYERS], *mW[NET_MAX_LAYERS], *vW[NET_MAX_LAYERS], *mb[NET_MAX_LAYERS],
        *vb[NET_MAX_LAYERS], *dW[NET_MAX_LAYERS], *db[NET_MAX_LAYERS];
    __nv_bfloat16 *Wb[NET_MAX_LAYERS], *WbT[NET_MAX_LAYERS];
    // the pass's activations and gradients, [nz][B][Np] (and transposed)
    __nv_bfloat16 *A[NET_MAX_LAYERS], *AT[NET_MAX_LAYERS], *G[NET_MAX_LAYERS], *GT[NET_MAX_LAYERS], *X0T;
    float* Z[NET_MAX_LAYERS];
    float* loss;
    float lr, b1, b2, eps, c1[TRAIN_STEPS], c2[TRAIN_STEPS];
    unsigned long long* bar;                       // [nz] arrival counters (and NET_FAILED), zero at launch
    int* err;                                      // bit 0: an MMA or barrier wait ran out
};

__device__ __forceinline__ unsigned long long ld_acquire_u64(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

// A network's counter also carries the word that its launch is given up: with NET_FAILED set its
// blocks leave their barrier, whatever they have counted; the next launch begins from zero.
constexpr unsigned long long NET_FAILED = 1ULL << 63;

// this launch of the network is given up (a wait ran out), its loss not a number
__device__ __forceinline__ void net_fail(unsigned long long* ctr, float* loss, int* err) {
    asm volatile("red.release.gpu.global.or.b64 [%0], %1;" ::"l"(ctr), "l"(NET_FAILED) : "memory");
    *(volatile float*)loss = __int_as_float(0x7fc00000);
    atomicOr(err, 1);
}

// barrier of a network's blocks; false (for the whole block) once a wait of theirs has run out
__device__ bool net_sync(unsigned long long* ctr, unsigned long long& target, float* loss, int* err) {
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        target += gridDim.x;
        asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(ctr), "l"(1ULL) : "memory");
        unsigned long long at;
        long long t0 = 0;
        unsigned it = 0;
        while ((at = ld_acquire_u64(ctr)) < target) {      // (a failed network's counter is past any target)
            if ((++it & 63u) == 0) {
                long long now = gtimer();
                if (t0 == 0) t0 = now;
                else if (now - t0 > WAIT_NS) { net_fail(ctr, loss, err); at = NET_FAILED; break; }
            }
        }
        s_ok = (at & NET_FAILED) == 0;
    }
    __syncthreads();
    return s_ok != 0;
}

// Adam of one weight with the step's corrections (the arithmetic of k_adam)
__device__ __forceinline__ float adam_one(const TrainArgs& g, int s, float gg, float& m, float& v, float w) {
    m = g.b1 * m + (1.0f - g.b1) * gg;
    v = g.b2 * v + (1.0f - g.b2) * gg * gg;
    return w - g.lr * (m / g.c1[s]) / (sqrtf(v / g.c2[s]) + g.eps);
}

__global__ void __launch_bounds__(TRAIN_THREADS, 2) k_train(const __grid_constant__ TrainArgs g) {
    extern __shared__ __align__(1024) char smem[];
    char* sA = smem;                               // 128 x 256
    char* sB = smem + MT * KMAX * 2;               // 32 x 256
    __shared__ __align__(8) unsigned long long mbar;
    __shared__ unsigned tmemSlot;
    const Net& net = g.net;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, quarter = warp & 3, half = warp >> 2;
    const int z = blockIdx.y, L = net.L, B = g.B;
    const int mTiles = (B + MT - 1) / MT;
    if (threadIdx.x == 0) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&mbar)));
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmemSlot)),
                     "r"(TRAIN_N));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    const unsigned tmem = tmemSlot;
    unsigned phase = 0;
    unsigned long long target = 0;
    bool ok = true;

    // the product of the staged operands (128 x N x Kp): true when it is in tensor memory
    auto product = [&](int N, int Kp) {
        cp_async_wait_all();
        asm volatile("fence.proxy.async.shared::cta;");
        asm volatile("tcgen05.fence::before_thread_sync;");
        __syncthreads();
        asm volatile("tcgen05.fence::after_thread_sync;");
        if (threadIdx.x == 0) issue_mma(tmem, smem_u32(sA), smem_u32(sB), N, Kp, &mbar);
        const bool done = wait_mma(&mbar, phase);
        phase ^= 1u;
        if (!done && threadIdx.x == 0) net_fail(g.bar + z, g.loss + z, g.err);
        asm volatile("tcgen05.fence::after_thread_sync;");
        return done;
    };
    // every warp is done with the operands and the accumulators
    auto release = [&]() {
        asm volatile("tcgen05.fence::before_thread_sync;");
        __syncthreads();
    };
    // row-major [rows][N] BF16 and its transpose [N][rows] from 16 columns of a row
    auto put = [&](__nv_bfloat16* rowMajor, __nv_bfloat16* transposed, int rows, int N, int row, int c0,
                   const float a[16]) {
        if (row >= rows) return;
        uint4 lo, hi;
        pack16(a, lo, hi);
        uint4* o = reinterpret_cast<uint4*>(rowMajor + (long long)row * N + c0);
        o[0] = lo;
        o[1] = hi;
#pragma unroll
        for (int j = 0; j < 16; j++) transposed[(long long)(c0 + j) * rows + row] = __float2bfloat16_rn(a[j]);
    };

    // dW of layer l for rows [128 mt, ..) and columns [32 kt, ..), its Adam update and, with the
    // first columns, the rows' bias gradient and update
    auto weight_tile = [&](int l, int tile, int s) {
        const int N = net.Np[l], K = net.Kp[l], kTiles = (K + TRAIN_N - 1) / TRAIN_N;
        const int mt = tile / kTiles, kt = tile - mt * kTiles, n0 = mt * MT, k0 = kt * TRAIN_N;
        const int kc = min(TRAIN_N, K - k0);
        const long long wz = (long long)z * N * K;
        const __nv_bfloat16* prevT = l == 0 ? g.X0T : g.AT[l - 1];
        stage_rows(sA, g.GT[l] + ((long long)z * N + n0) * B, B, MT, min(MT, N - n0), B);
        stage_rows(sB, prevT + ((long long)z * K + k0) * B, B, kc, kc, B);
        const int n = n0 + quarter * 32 + lane, c0 = 16 * half;
        const bool mine = n < N && c0 < kc;
        const long long o = wz + (long long)n * K + k0 + c0;
        float4 w = {}, m = {}, v = {};
        auto fetch = [&](int j) {
            w = reinterpret_cast<const float4*>(g.W[l] + o)[j];
            m = reinterpret_cast<const float4*>(g.mW[l] + o)[j];
            v = reinterpret_cast<const float4*>(g.vW[l] + o)[j];
        };
        if (mine) fetch(0);
        if (!product(kc, B)) return false;
        if (kt == 0 && threadIdx.x < MT && n0 + (int)threadIdx.x < N) {
            // the bias gradient: the row's B values in row order, from the staged operand
            const int r = threadIdx.x;
            float sum = 0.f;
            for (int c = 0; c < B; c += 8) {
                const uint4 q = *reinterpret_cast<const uint4*>(sA + core_at(r, c, B));
                const unsigned h[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    sum += __bfloat162float(__ushort_as_bfloat16((unsigned short)(h[j] & 0xffffu)));
                    sum += __bfloat162float(__ushort_as_bfloat16((unsigned short)(h[j] >> 16)));
                }
            }
            const int bo = z * N + n0 + r;
            g.db[l][bo] = sum;
            float mm = g.mb[l][bo], vv = g.vb[l][bo];
            g.bias[l][bo] = adam_one(g, s, sum, mm, vv, g.bias[l][bo]);
            g.mb[l][bo] = mm;
            g.vb[l][bo] = vv;
        }
        // four columns at a time, the next four's state on its way
        if (c0 < kc) {
#pragma unroll 1
            for (int j = 0; j < 4; j++) {
                __syncwarp();                          // the load below is the whole warp's
                const float4 d = load_acc4(tmem, quarter, c0 + 4 * j);
                if (mine) {
                    float4 w1 = w, m1 = m, v1 = v;
                    if (j < 3) fetch(j + 1);
                    w1.x = adam_one(g, s, d.x, m1.x, v1.x, w1.x);
                    w1.y = adam_one(g, s, d.y, m1.y, v1.y, w1.y);
                    w1.z = adam_one(g, s, d.z, m1.z, v1.z, w1.z);
                    w1.w = adam_one(g, s, d.w, m1.w, v1.w, w1.w);
                    reinterpret_cast<float4*>(g.dW[l] + o)[j] = d;
                    reinterpret_cast<float4*>(g.W[l] + o)[j] = w1;
                    reinterpret_cast<float4*>(g.mW[l] + o)[j] = m1;
                    reinterpret_cast<float4*>(g.vW[l] + o)[j] = v1;
                    __nv_bfloat162 h[2] = {__floats2bfloat162_rn(w1.x, w1.y), __floats2bfloat162_rn(w1.z, w1.w)};
                    *reinterpret_cast<uint2*>(g.Wb[l] + o + 4 * j) = *reinterpret_cast<uint2*>(h);
                    __nv_bfloat16* t = g.WbT[l] + wz + (long long)(k0 + c0 + 4 * j) * N + n;
                    t[0] = h[0].x;
                    t[N] = h[0].y;
                    t[2 * N] = h[1].x;
                    t[3 * N] = h[1].y;
                }
            }
            __syncwarp();
        }
        release();
        return true;
    };
    auto weight_tiles = [&](int l) { return ((net.Np[l] + MT - 1) / MT) * ((net.Kp[l] + TRAIN_N - 1) / TRAIN_N); };

    for (int s = 0; s < g.nsteps && ok; s++) {
        auto point = [&](int row) {
            return g.idx ? g.idx[z * g.idxStride + (long long)s * B + row] : (long long)z * B + row;
        };
        // ---- forward
        for (int l = 0; l < L && ok; l++) {
            const int N = net.Np[l], K = net.Kp[l], nTiles = (N + TRAIN_N - 1) / TRAIN_N;
            const bool last = l == L - 1;
            if (l == 0 && blockIdx.x == 0 && threadIdx.x == 0) g.loss[z] = 0.f;
            for (int tile = blockIdx.x; tile < mTiles * nTiles && ok; tile += gridDim.x) {
                const int mt = tile / nTiles, nt = tile - mt * nTiles, m0 = mt * MT, n0 = nt * TRAIN_N;
                const int nc = min(TRAIN_N, N - n0);
                if (l == 0) {
                    // the batch's inputs (16 padded columns), with their transpose for dW of layer 0
                    const int r = threadIdx.x >> 1, q0 = (threadIdx.x & 1) * 8, row = m0 + r;
                    unsigned short h[8];
                    const long long pt = row < B ? point(row) : 0;
#pragma unroll
                    for (int j = 0; j < 8; j++) {
                        const float x = (row < B && q0 + j < net.nin) ? g.X[pt * net.nin + q0 + j] : 0.f;
                        h[j] = __bfloat16_as_ushort(__float2bfloat16_rn(x));
                        if (nt == 0 && row < B)
                            g.X0T[((long long)z * K + q0 + j) * B + row] = __ushort_as_bfloat16(h[j]);
                    }
                    *reinterpret_cast<uint4*>(sA + core_at(r, q0, 16)) =
                        make_uint4(h[0] | (unsigned)h[1] << 16, h[2] | (unsigned)h[3] << 16,
                                   h[4] | (unsigned)h[5] << 16, h[6] | (unsigned)h[7] << 16);
                } else {
                    stage_rows(sA, g.A[l - 1] + ((long long)z * B + m0) * K, K, MT, min(MT, B - m0), K);
                }
                stage_rows(sB, g.Wb[l] + ((long long)z * N + n0) * K, K, nc, nc, K);
                const int r = quarter * 32 + lane, row = m0 + r, c0 = 16 * half;
                ok = product(nc, K);
                if (ok && c0 < nc) {
                    float v[16];
                    load_acc16(tmem, quarter, c0, v);
#pragma unroll
                    for (int j = 0; j < 16; j++) v[j] += __ldcg(g.bias[l] + z * N + n0 + c0 + j);
                    if (row < B) {
                        float4* zo = reinterpret_cast<float4*>(g.Z[l] + ((long long)z * B + row) * N + n0 + c0);
#pragma unroll
                        for (int j = 0; j < 4; j++)
                            zo[j] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
                    }
                    if (!last) {
#pragma unroll
                        for (int j = 0; j < 16; j++) v[j] = gelu(v[j]);
                        put(g.A[l] + (long long)z * B * N, g.AT[l] + (long long)z * B * N, B, N, row, n0 + c0, v);
                    } else {
                        // the loss gradient of the outputs (0 on the padding), and the loss
                        float e = 0.f;
                        const long long pt = row < B ? point(row) : 0;
#pragma unroll
                        for (int j = 0; j < 16; j++) {
                            float gr = 0.f;
                            if (row < B && c0 + j < net.nout) {
                                const float d = v[j] - g.Y[pt * net.nout + c0 + j];
                                gr = 2.0f * d / (float)(B * net.nout);
                                e += d * d / (float)(B * net.nout);
                            }
                            v[j] = gr;
                        }
                        put(g.G[l] + (long long)z * B * N, g.GT[l] + (long long)z * B * N, B, N, row, c0, v);
                        for (int q = 16; q > 0; q >>= 1) e += __shfl_xor_sync(0xffffffffu, e, q);
                        if (lane == 0) atomicAdd(&g.loss[z], e);
                    }
                }
                if (ok) release();
            }
            ok = ok && net_sync(g.bar + z, target, g.loss + z, g.err);
        }
        // ---- backward: the gradient of layer l's input, with the update of layer l + 1
        for (int l = L - 1; l >= 1 && ok; l--) {
            const int N = net.Np[l], K = net.Kp[l], kTiles = (K + TRAIN_N - 1) / TRAIN_N;
            const int nGrad = mTiles * kTiles, nAll = nGrad + (l + 1 < L ? weight_tiles(l + 1) : 0);
            for (int tile = blockIdx.x; tile < nAll && ok; tile += gridDim.x) {
                if (tile >= nGrad) {
                    ok = weight_tile(l + 1, tile - nGrad, s);
                    continue;
                }
                const int mt = tile / kTiles, kt = tile - mt * kTiles, m0 = mt * MT, k0 = kt * TRAIN_N;
                const int kc = min(TRAIN_N, K - k0);
                stage_rows(sA, g.G[l] + ((long long)z * B + m0) * N, N, MT, min(MT, B - m0), N);
                stage_rows(sB, g.WbT[l] + ((long long)z * K + k0) * N, N, kc, kc, N);
                const int row = m0 + quarter * 32 + lane, c0 = 16 * half;
                float zv[16];
                if (row < B && c0 < kc) {
                    const float4* zp = reinterpret_cast<const float4*>(g.Z[l - 1] + ((long long)z * B + row) * K + k0 + c0);
#pragma unroll
                    for (int j = 0; j < 4; j++) *reinterpret_cast<float4*>(zv + 4 * j) = __ldcg(zp + j);
                }
                ok = product(kc, N);
                if (ok && c0 < kc) {
                    float v[16];
                    load_acc16(tmem, quarter, c0, v);
                    if (row < B) {
#pragma unroll
                        for (int j = 0; j < 16; j++) v[j] *= gelu_grad(zv[j]);
                        put(g.G[l - 1] + (long long)z * B * K, g.GT[l - 1] + (long long)z * B * K, B, K, row, k0 + c0, v);
                    }
                }
                if (ok) release();
            }
            ok = ok && net_sync(g.bar + z, target, g.loss + z, g.err);
        }
        // ---- the updates that are left: layer 0, and layer 1 of a network with more than one
        const int w1 = L > 1 ? weight_tiles(1) : 0, w0 = weight_tiles(0);
        for (int tile = blockIdx.x; tile < w1 + w0 && ok; tile += gridDim.x)
            ok = weight_tile(tile < w1 ? 1 : 0, tile < w1 ? tile : tile - w1, s);
        ok = ok && net_sync(g.bar + z, target, g.loss + z, g.err);
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TRAIN_N));
    }
}

// dZ = dA * GELU'(Z) (or dA when Z is NULL) -> BF16 row-major and transposed; M x N, per z
__global__ void k_gelu_back(int M, int N, const float* dA, const float* Z, long long sMN, __nv_bfloat16* g,
                            __nv_bfloat16* gT, long long sG, long long sGT) {
    int z = blockIdx.y;
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)M * N) return;
    int row = (int)(i / N), n = (int)(i - (long long)row * N);
    float d = dA[z * sMN + i];
    if (Z) d *= gelu_grad(Z[z * sMN + i]);
    __nv_bfloat16 h = __float2bfloat16_rn(d);
    g[z * sG + i] = h;
    gT[z * sGT + (long long)n * M + row] = h;
}

// column sums over rows (bias gradients), fixed row order: out[n] = sum_r in[r*N + n]
__global__ void k_colsum_bf16(int M, int N, const __nv_bfloat16* in, long long sIn, float* out, long long sOut) {
    int z = blockIdx.y, n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= N) return;
    float s = 0.f;
    for (int r = 0; r < M; r++) s += __bfloat162float(in[z * sIn + (long long)r * N + n]);
    out[z * sOut + n] = s;
}

// MSE gradient on the first `nOut` of Np output columns: g = 2 (y - t) / (M nOut) (0 on padding)
__global__ void k_mse_grad(int M, int Np, int nOut, const float* y, long long sY, const float* t, long long sT,
                           float* g, long long sG, float* loss) {
    int z = blockIdx.y;
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)M * Np) return;
    int row = (int)(i / Np), n = (int)(i - (long long)row * Np);
    float v = 0.f;
    if (n < nOut) {
        float d = y[z * sY + i] - t[z * sT + (long long)row * nOut + n];
        v = 2.0f * d / (float)(M * nOut);
        if (loss) atomicAdd(&loss[z], d * d / (float)(M * nOut));
    }
    g[z * sG + i] = v;
}

// Adam on FP32 master weights W[N x K] (per z); writes the BF16 copies W (N x K) and W^T (K x N)
__global__ void k_adam(int N, int K, float* w, const float* gw, float* m, float* v, long long s, float lr, float b1,
                       float b2, float eps, float c1, float c2, __nv_bfloat16* wb, __nv_bfloat16* wbT, long long sb,
                       long long sbT) {
    int z = blockIdx.y;
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)N * K) return;
    long long o = z * s + i;
    float gg = gw[o];
    float mm = b1 * m[o] + (1.0f - b1) * gg;
    float vv = b2 * v[o] + (1.0f - b2) * gg * gg;
    m[o] = mm;
    v[o] = vv;
    float ww = w[o] - lr * (mm / c1) / (sqrtf(vv / c2) + eps);
    w[o] = ww;
    if (wb) {
        __nv_bfloat16 h = __float2bfloat16_rn(ww);
        wb[z * sb + i] = h;
        if (wbT) {
            int n = (int)(i / K), k = (int)(i - (long long)n * K);
            wbT[z * sbT + (long long)k * N + n] = h;
        }
    }
}

}  // namespace

#define SBX_LAUNCH_SMEM(ctx, kernel, grid, block, smem, ...)                \
    do {                                                                  \
        kernel<<<(grid), (block), (smem), (ctx)->stream>>>(__VA_ARGS__);  \
        (ctx)->launches++;                                                \
    } while (0)

extern "C" sbx_status sbx_mlp_gemm_bf16(sbx_ctx* ctx, int32_t nz, int32_t M, int32_t N, int32_t K,
                                        const void* A, int32_t lda, int64_t strideA, const void* B, int32_t ldb,
                                        int64_t strideB, const float* bias, int64_t strideBias, int32_t act,
                                        void* out, int32_t ldo, int64_t strideOut, void* outT, int32_t ldt,
                                        int64_t strideOutT, float* outF, int32_t ldf, int64_t strideOutF,
                                        int32_t* errFlag) {
    SBX_REQUIRE(ctx && nz >= 1 && M >= 0 && N >= 1 && K >= 1 && K <= KMAX && A && B && lda >= K && ldb >= K &&
                (act == 0 || act == 1) && (out || outT || outF) && (!out || ldo >= N) && (!outT || ldt >= M) &&
                (!outF || ldf >= N) && nz <= 65535);
    if (M == 0) return SBX_OK;
    static bool attr = false;
    const int Kp = (K + 15) & ~15;
    size_t smem = (size_t)(MT + NT) * Kp * 2 + 16;
    if (!attr) {
        cudaFuncSetAttribute(k_gemm, cudaFuncAttributeMaxDynamicSharedMemorySize, (MT + NT) * KMAX * 2 + 16);
        attr = true;
    }
    GemmArgs g{M, N, K, (const __nv_bfloat16*)A, lda, strideA, (const __nv_bfloat16*)B, ldb, strideB, bias,
               strideBias, act, (__nv_bfloat16*)out, ldo, strideOut, (__nv_bfloat16*)outT, ldt, strideOutT, outF, ldf,
               strideOutF, errFlag};
    // one wave of CTAs (1 per SM, shared memory bound), each looping over its M tiles with
    // its B tile resident
    int sms = 148;
    {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    }
    const int tilesM = (M + MT - 1) / MT, tilesN = (N + NT - 1) / NT;
    int gx = sms / (tilesN * nz);                  // a single wave: no SM runs two of them
    gx = gx < 1 ? 1 : (gx > tilesM ? tilesM : gx);
    dim3 grid(gx, tilesN, nz);
    SBX_LAUNCH_SMEM(ctx, k_gemm, grid, GEMM_THREADS, smem, g);
    return check_launch(ctx, "sbx_mlp_gemm_bf16");
}

extern "C" sbx_status sbx_mlp_gelu_backward(sbx_ctx* ctx, int32_t nz, int32_t M, int32_t N, const float* dA,
                                            const float* Z, int64_t strideMN, void* g, void* gT, int64_t strideG,
                                            int64_t strideGT) {
    SBX_REQUIRE(ctx && nz >= 1 && M >= 0 && N >= 1 && dA && g && gT);
    if (M == 0) return SBX_OK;
    long long n = (long long)M * N;
    dim3 grid((unsigned)((n + 255) / 256), nz);
    SBX_LAUNCH_SMEM(ctx, k_gelu_back, grid, 256, 0, M, N, dA, Z, strideMN, (__nv_bfloat16*)g, (__nv_bfloat16*)gT,
               strideG, strideGT);
    return check_launch(ctx, "sbx_mlp_gelu_backward");
}

extern "C" sbx_status sbx_mlp_colsum_bf16(sbx_ctx* ctx, int32_t nz, int32_t M, int32_t N, const void* in,
                                          int64_t strideIn, float* out, int64_t strideOut) {
    SBX_REQUIRE(ctx && nz >= 1 && M >= 0 && N >= 1 && in && out);
    dim3 grid((N + 127) / 128, nz);
    SBX_LAUNCH_SMEM(ctx, k_colsum_bf16, grid, 128, 0, M, N, (const __nv_bfloat16*)in, strideIn, out, strideOut);
    return check_launch(ctx, "sbx_mlp_colsum_bf16");
}

extern "C" sbx_status sbx_mlp_mse_grad(sbx_ctx* ctx, int32_t nz, int32_t M, int32_t Np, int32_t nOut, const float* y,
                                       int64_t strideY, const float* t, int64_t strideT, float* g, int64_t strideG,
                                       float* loss) {
    SBX_REQUIRE(ctx && nz >= 1 && M >= 1 && Np >= nOut && nOut >= 1 && y && t && g);
    long long n = (long long)M * Np;
    dim3 grid((unsigned)((n + 255) / 256), nz);
    SBX_LAUNCH_SMEM(ctx, k_mse_grad, grid, 256, 0, M, Np, nOut, y, strideY, t, strideT, g, strideG, loss);
    return check_launch(ctx, "sbx_mlp_mse_grad");
}

extern "C" sbx_status sbx_mlp_adam(sbx_ctx* ctx, int32_t nz, int32_t N, int32_t K, float* w, const float* gw,
                                   float* m, float* v, int64_t stride, float lr, float beta1, float beta2, float eps,
                                   int32_t stepNumber, void* wBf16, void* wBf16T, int64_t strideB, int64_t strideBT) {
    SBX_REQUIRE(ctx && nz >= 1 && N >= 1 && K >= 1 && w && gw && m && v && stepNumber >= 1);
    float c1 = 1.0f - powf(beta1, (float)stepNumber), c2 = 1.0f - powf(beta2, (float)stepNumber);
    long long n = (long long)N * K;
    dim3 grid((unsigned)((n + 255) / 256), nz);
    SBX_LAUNCH_SMEM(ctx, k_adam, grid, 256, 0, N, K, w, gw, m, v, stride, lr, beta1, beta2, eps, c1, c2,
               (__nv_bfloat16*)wBf16, (__nv_bfloat16*)wBf16T, strideB, strideBT);
    return check_launch(ctx, "sbx_mlp_adam");
}

// ---------------------------------------------------------------- whole networks
// Which ensembles the whole-network kernels take: inputs and outputs within their 16 padded
// columns, hidden widths whole tiles. Others keep the GEMM path.
static bool net_fits(const sbx_mlp_net* n, bool train) {
    if (!n || n->nz < 1 || n->nz > 65535 || n->nLayers < (train ? 2 : 1) || n->nLayers > NET_MAX_LAYERS || n->nin < 1 ||
        n->nin > 16 || n->nout < 1 || n->nout > 16)
        return false;
    for (int l = 0; l < n->nLayers; l++) {
        const int N = n->Np[l], K = n->Kp[l];
        if (K != (l == 0 ? 16 : n->Np[l - 1])) return false;
        if (l == n->nLayers - 1 ? N != 16 : (N < 32 || N > KMAX || N % 32)) return false;
        if (!n->Wb[l] || !n->b[l] || ((uintptr_t)n->Wb[l] & 15)) return false;
    }
    return true;
}

static Net net_of(const sbx_mlp_net* n) {
    Net o{};
    o.nz = n->nz; o.L = n->nLayers; o.nin = n->nin; o.nout = n->nout;
    for (int l = 0; l < o.L; l++) {
        o.Kp[l] = n->Kp[l];
        o.Np[l] = n->Np[l];
        o.Wb[l] = (const __nv_bfloat16*)n->Wb[l];
        o.b[l] = n->b[l];
    }
    return o;
}

static int sm_count(sbx_ctx* ctx) {
    int sms = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device) != cudaSuccess) sms = 0;
    return sms;
}

constexpr size_t TRAIN_SMEM = (size_t)(MT + TRAIN_N) * KMAX * 2;

// blocks of the training kernel that the current device holds at once; 0 if it cannot tell
static int train_blocks() {
    int dev = 0, sms = 0, per = 0;
    if (cudaGetDevice(&dev) == cudaSuccess &&
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess &&
        cudaFuncSetAttribute(k_train, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TRAIN_SMEM) == cudaSuccess &&
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_train, TRAIN_THREADS, TRAIN_SMEM) == cudaSuccess)
        return per * sms;
    cudaGetLastError();
    return 0;
}

// Where the one launch leads the separate kernels. A network's blocks must all be resident: more
// networks than that cannot run whole. With two blocks a network or more it leads at every width
// and batch that was measured (32 to 256 wide, 2 to 8 layers, batches of 16 to 256): 1.06 to 8
// times. With one block it depends on how many tiles of a layer's weights that block walks
// through: up to ONE_BLOCK_TILES it leads or is even (75 to 148 networks: 96 wide 3 tiles, 1.5 to
// 2.4 times; 256-64-256 8 tiles, 1.04 to 1.36; 160 wide 10 tiles, 0.97 to 1.23), beyond them
// mostly not (192 wide 12 tiles, 0.86 to 1.14; 256 wide 16 tiles, 0.67 to 1.03).
constexpr int ONE_BLOCK_TILES = 10;
static bool train_leads(const sbx_mlp_net* n) {
    const int per = train_blocks() / n->nz;
    if (per != 1) return per > 1;
    for (int l = 0; l < n->nLayers; l++)
        if (((n->Np[l] + MT - 1) / MT) * ((n->Kp[l] + TRAIN_N - 1) / TRAIN_N) > ONE_BLOCK_TILES) return false;
    return true;
}

extern "C" int32_t sbx_mlp_net_fits(const sbx_mlp_net* net, int32_t train) {
    return net_fits(net, train != 0) && (!train || train_leads(net)) ? 1 : 0;
}

extern "C" sbx_status sbx_mlp_predict(sbx_ctx* ctx, const sbx_mlp_net* net, const double* X, int32_t P,
                                      const double* xMean, const double* xStd, const double* yMean,
                                      const double* yStd, double* out, int32_t* errFlag) {
    SBX_REQUIRE(ctx && net_fits(net, false) && P >= 0 && (P == 0 || (X && xMean && xStd && yMean && yStd && out)));
    if (P == 0) return SBX_OK;
    const size_t smem = (size_t)(MT + NT) * KMAX * 2;
    if (cudaFuncSetAttribute(k_predict, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
        return fail(ctx, SBX_ECUDA, "sbx_mlp_predict: shared memory attribute");
    PredictArgs g{net_of(net), X, xMean, xStd, yMean, yStd, P, out, errFlag};
    const int sms = sm_count(ctx), tiles = (P + MT - 1) / MT;
    int gx = sms / net->nz;                        // one wave: a block's shared memory fills an SM
    gx = gx < 1 ? 1 : (gx > tiles ? tiles : gx);
    SBX_LAUNCH_SMEM(ctx, k_predict, dim3(gx, net->nz), GEMM_THREADS, smem, g);
    const long long n = (long long)P * net->nout;
    SBX_LAUNCH(ctx, k_predict_stats, blocks(n), 256, net->nz, n, out);
    return check_launch(ctx, "sbx_mlp_predict");
}

extern "C" sbx_status sbx_mlp_train(sbx_ctx* ctx, const sbx_mlp_net* net, const sbx_mlp_train_state* st, int32_t B,
                                    const float* X, const float* Y, const int64_t* idx, int64_t idxStride,
                                    int32_t nsteps, int32_t stepNumber, float lr, float beta1, float beta2, float eps) {
    SBX_REQUIRE(ctx && net_fits(net, true) && st && B >= 16 && B <= KMAX && B % 16 == 0 && X && Y && nsteps >= 0 &&
                stepNumber >= 1 && st->X0T && st->loss && st->bar && st->err);
    auto aligned = [](const void* p) { return p && ((uintptr_t)p & 15) == 0; };
    SBX_REQUIRE(aligned(st->X0T) && ((uintptr_t)st->bar & 7) == 0);
    for (int l = 0; l < net->nLayers; l++)
        SBX_REQUIRE(aligned(st->W[l]) && aligned(st->mW[l]) && aligned(st->vW[l]) && aligned(st->dW[l]) && st->mb[l] &&
                    st->vb[l] && st->db[l] && aligned(st->WbT[l]) && aligned(st->Z[l]) && aligned(st->G[l]) &&
                    aligned(st->GT[l]) && (l == net->nLayers - 1 || (aligned(st->A[l]) && aligned(st->AT[l]))));
    const size_t smem = TRAIN_SMEM;
    // a network's blocks: all resident, no more than a backward pass has tiles (two products of 16)
    int gx = train_blocks() / net->nz;
    if (gx < 1) return fail(ctx, SBX_EINVAL, "sbx_mlp_train: more networks than resident blocks");
    if (gx > 32) gx = 32;
    TrainArgs g{};
    g.net = net_of(net);
    g.B = B;
    g.X = X; g.Y = Y;
    g.idx = (const long long*)idx;
    g.idxStride = idxStride;
    for (int l = 0; l < net->nLayers; l++) {
        g.W[l] = st->W[l]; g.bias[l] = net->b[l]; g.mW[l] = st->mW[l]; g.vW[l] = st->vW[l];
        g.mb[l] = st->mb[l]; g.vb[l] = st->vb[l]; g.dW[l] = st->dW[l]; g.db[l] = st->db[l];
        g.Wb[l] = (__nv_bfloat16*)net->Wb[l]; g.WbT[l] = (__nv_bfloat16*)st->WbT[l];
        g.A[l] = (__nv_bfloat16*)st->A[l]; g.AT[l] = (__nv_bfloat16*)st->AT[l];
        g.G[l] = (__nv_bfloat16*)st->G[l]; g.GT[l] = (__nv_bfloat16*)st->GT[l];
        g.Z[l] = st->Z[l];
    }
    g.X0T = (__nv_bfloat16*)st->X0T;
    g.loss = st->loss;
    g.bar = (unsigned long long*)st->bar;
    g.err = st->err;
    g.lr = lr; g.b1 = beta1; g.b2 = beta2; g.eps = eps;
    for (int s0 = 0; s0 < nsteps; s0 += TRAIN_STEPS) {
        g.nsteps = nsteps - s0 < TRAIN_STEPS ? nsteps - s0 : TRAIN_STEPS;
        g.idx = idx ? (const long long*)idx + (int64_t)s0 * B : nullptr;
        for (int s = 0; s < g.nsteps; s++) {
            g.c1[s] = 1.0f - powf(beta1, (float)(stepNumber + s0 + s));
            g.c2[s] = 1.0f - powf(beta2, (float)(stepNumber + s0 + s));
        }
        if (cudaMemsetAsync(g.bar, 0, sizeof(unsigned long long) * net->nz, ctx->stream) != cudaSuccess)
            return fail(ctx, SBX_ECUDA, "sbx_mlp_train: memset");
        void* args[] = {&g};
        cudaError_t e = cudaLaunchCooperativeKernel((const void*)k_train, dim3(gx, net->nz), dim3(TRAIN_THREADS), args,
                                                    smem, ctx->stream);
        ctx->launches++;
        if (e != cudaSuccess) {
            cudaGetLastError();
            return fail(ctx, SBX_ECUDA, std::string("sbx_mlp_train: ") + cudaGetErrorString(e));
        }
    }
    return check_launch(ctx, "sbx_mlp_train");
}
