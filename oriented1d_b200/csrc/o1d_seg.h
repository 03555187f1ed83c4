// Host-callable interface of the segment kernels (o1d_seg.cuh), compiled in their own translation unit.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace o1d {

constexpr int kSegGeos = 6, kSegRuns = 20;
// Order of the sums (o1d_seg.cuh): taps ascending, or as in the tiled kernels.
enum : int { SEG_UNSET = 0, SEG_ASCENDING, SEG_TILED, SEG_FIRST, SEG_LAST };

// How the maps of a run of chunks are cut into items: G whole images, or one tile of an image.
struct SegGeo {
    int G, items;                        // images per item; items per chunk
    int nth, ntw, TH, TW;                // output tiles of one image
    int halo_h, halo_w;                  // 1: cut along that axis, tiles overlap by the reach of the lines
    int oh, ow;                          // smem row / pixel of the tile's first output
    int P, RT;                           // smem pixels per row, rows per image
    // positions that a line is clamped to: the zeros around a whole map (-1, H or W), or a cut tile's first and
    // last row / pixel (what lies past those reaches no output of the tile)
    int plo_w, phi_w, plo_h, phi_h;
    int img_bytes, tile_bytes, buf_bytes, nbuf;
};
// Consecutive chunks with the same lines.
struct SegRun {
    int chunk0, nchunks, geo;
    int cost;                            // of one item
    int ctas;                            // CTAs per chunk (per_chunk)
};
struct SegParams {
    int N, H, W, C, K;
    int CC, px;                          // channels and bytes of a chunk
    int nruns, per_chunk;
    int off_tile, off_tab, off_bar;
    int flip, identity;
    long long total_cost;
    SegGeo geo[kSegGeos];
    SegRun run[kSegRuns];
};
struct SegMaps { CUtensorMap m[kSegGeos]; };

struct SegConfig {
    SegParams p;
    int esize, short_reach, line_block, smem_bytes, grid, ngeos;
    bool patchy;                         // lines change often from channel to channel (see make_config)
    int order;                           // order of the sums, for the caller to keep here: SEG_UNSET at first
    int rank;                            // place among the kernel families, likewise: SEG_UNSET, SEG_FIRST, SEG_LAST
};

// Do the segment kernels take this request (NHWC, stride 1, canonical lines)?  `chan`: canonical line of
// every channel (host copy of the plan's table).  The answer for a shape is kept per thread.
bool seg_configure(const int8_t *chan, int N, int H, int W, int C, int K, int esize, int smem_optin, int sms, bool wgrad,
                   SegConfig **cfg);

// y = conv(x) + bias (flip = 1: input gradient).  w, bias fp32, or bf16 when wbf16 is set.
// order: SEG_ASCENDING (bf16 only) or SEG_TILED.
cudaError_t seg_launch_conv(const SegConfig &cfg, const SegMaps &maps, const void *w, const void *bias, int wbf16,
                            const int8_t *chan, void *y, int flip, int identity, int order, int *err_flag, cudaStream_t st);

// Weight gradient (and bias gradient when db is not null): dw, db fp32, or bf16 when out_bf16 is set.
// `partial`: seg_wgrad_bytes() of scratch.
size_t seg_wgrad_bytes(const SegConfig &cfg);
cudaError_t seg_launch_wgrad(const SegConfig &cfg, const SegMaps &maps, const SegMaps &dy_maps, const int8_t *chan, const void *dy,
                             void *dw, void *db, int out_bf16, float *partial, int *err_flag, cudaStream_t st);

}  // namespace o1d
