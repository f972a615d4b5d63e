// sbx_wide.cuh — the dense step as a few wide kernels (sbx_wide.cu).
#pragma once
#include "sbx_fused.cuh"

constexpr int WIDE_CELL_SLOTS = 8;    // fixed slots per grid cell (one 32-byte sector)
// fixed slots per segment row of link A ends, of link B ends: four are read with the row's
// count, the rest only by longer rows
constexpr int WIDE_ROW_SLOTS = 16;
constexpr int WIDE_TILE = 4096;       // rows of a scan tile
constexpr int WIDE_SUM_STRIDE = 8;    // ints between two tiles' sums: each in a sector of its own

// the supplied noise as the captured steps find it, in device memory: planar [n][6][items] from
// step t0 on, all null without; err is set when a step outside that range runs
struct WideNoise {
    const float *fil, *mot, *bb;
    int t0, n;
    int* err;
};

// `a` holds the scene and this path's own scratch (not the fused kernel's)
struct WideArgs {
    FusedArgs a;
    int tilesC, tilesS;      // scan tiles of the cells and of the rods
    // per tile: bodies and segments of the cells, A ends, B ends, bound motors of the rods
    int *sumCell, *sumSeg, *sumA, *sumB, *sumM;
    sbx_batch bt;            // packed networks' tables (packed plans)
    WideNoise* noise;
    int* errDev;             // the context's input-range error word
    float *payA, *payB;      // the links' A-side and B-side payloads in CSR order, 6 floats each
};

// the streams and events of one step: `ahead` runs what needs only the step's start view, `link`
// the crosslinkers, `csr` the motor CSR
struct WideStreams {
    cudaStream_t ahead = nullptr, link = nullptr, csr = nullptr;
    cudaEvent_t start = nullptr, bound = nullptr, joined = nullptr, linkDone = nullptr,
                csrDone = nullptr;
};

bool wide_streams_create(WideStreams& ws);
void wide_streams_destroy(WideStreams& ws);

// the noise of the steps that follow on the context's stream
sbx_status wide_set_noise(sbx_ctx* ctx, const WideArgs& w, const WideNoise& noise);

// queues one step on the context's stream (for capture); the step index is *d_step, advanced at
// the end
sbx_status wide_step(sbx_ctx* ctx, const WideArgs& w, bool batched, const WideStreams& ws);
