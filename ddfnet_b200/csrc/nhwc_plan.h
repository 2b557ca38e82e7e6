// The channels_last forward's plan and the host-side arithmetic that needs no CUDA (see nhwc.cu), so that it can be
// checked without a GPU.
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define NHWC_HD __host__ __device__ __forceinline__
#else
#define NHWC_HD inline
#endif

namespace ddf {

constexpr int kNhwcThreads = 256;
constexpr int kNhwcRows = 8;                 // output rows of a tile at most
constexpr uint32_t kNhwcSmem = 112 * 1024;   // shared memory of a CTA at most: two per SM

struct NhwcPlan {
    const void* x;          // (B, H, W, C)
    const void* cf;         // (B, C, K, K)
    const void* sf;         // K*K values per output pixel, addressed by the two strides below
    const float* sf_bias;   // K*K values added to the raw filter, or null
    void* out;              // (B, OH, OW, C)
    const float* oscale;    // per-channel output scale / shift, or null
    const float* oshift;
    int B, C, H, W, OH, OW;
    long long sf_batch_stride, sf_pixel_stride, sf_tap_stride;   // in elements
    int relu;
    float sf_scale;
    int vecs;               // C / 8
    int cols, rows;         // output columns and rows of a tile
    int tiles_x, tiles_y;   // tiles of an image
    int tiles;              // of all images
    int sf_bulk;            // a pixel's K*K values are contiguous, 16-byte aligned, and so are a row's pixels: bulk copies
    uint32_t off_sf, sf_stride, off_affine, off_buf, buf_stride, off_raw, row_bytes;  // off_raw: inside a buffer
    int* fault;
    long long wait_cycles;  // limit of every mbarrier wait, in SM clocks
    int starve;             // self-test: this tile of every CTA (1: the first) is announced 16 bytes too large and never completes
};

// A row of a tile's raw filters, as one bulk copy (sf_bulk): `nx` pixels from column ox0 of row oy of sample b.  Behind
// the last pixel of a sample there may be nothing to read, whatever comes after it in memory (sf_batch_stride may be 0,
// or lead backwards): 8 of its values come by the copy, the ninth apart.
struct NhwcRun {
    long long from;   // in elements
    uint32_t bytes;
};
NHWC_HD bool nhwc_last_pixel(const NhwcPlan& pl, int oy, int ox) { return oy == pl.OH - 1 && ox == pl.OW - 1; }
NHWC_HD NhwcRun nhwc_filter_run(const NhwcPlan& pl, int b, int oy, int ox0, int nx) {
    const uint32_t pixel = (uint32_t)pl.sf_pixel_stride * 2u;
    return {b * pl.sf_batch_stride + ((long long)oy * pl.OW + ox0) * pl.sf_pixel_stride,
            (uint32_t)nx * pixel - (nhwc_last_pixel(pl, oy, ox0 + nx - 1) ? pixel - 16u : 0u)};
}

// Tiles and shared-memory layout of a problem; `pixel`: bytes of a pixel's filter in shared memory.  Returns the bytes of
// shared memory, 0 where there would be too many tiles.
// Equal column counts, as many as the threads cover; rows as two buffers of two CTAs leave room for (the two halo rows are
// then a quarter of the copies at most), fewer where the chip would not be full.  More tiles across where one row of that
// many columns does not fit: C = 8 alone, whose 256 columns with 16-map filters at stride 2 take 115 072 bytes.
inline uint32_t nhwc_tiles(NhwcPlan& pl, int s, uint32_t pixel, int sm_count) {
    const int most = kNhwcThreads / pl.vecs;
    auto layout = [&](int r) {
        pl.row_bytes = (uint32_t)(((pl.cols - 1) * s + 3) * pl.C * 2);
        pl.off_sf = 64;
        pl.sf_stride = (uint32_t)pl.cols * ((uint32_t)r * pixel + 16u);
        pl.off_affine = pl.off_sf + 2u * pl.sf_stride;
        pl.off_buf = (pl.off_affine + 8u * (uint32_t)pl.C + 127u) & ~127u;
        pl.off_raw = (uint32_t)((r - 1) * s + 3) * pl.row_bytes;
        pl.buf_stride = (pl.off_raw + (pl.sf_bulk ? (uint32_t)(r * pl.cols * (int)pl.sf_pixel_stride) * 2u : 0u) + 127u) & ~127u;
        return pl.off_buf + 2u * pl.buf_stride;
    };
    for (int across = (pl.OW + most - 1) / most;; ++across) {
        pl.cols = (pl.OW + across - 1) / across;
        if (pl.cols == 1 || layout(1) <= kNhwcSmem) break;
    }
    pl.tiles_x = (pl.OW + pl.cols - 1) / pl.cols;
    int rows = pl.OH < kNhwcRows ? pl.OH : kNhwcRows;
    while (rows > 1 && layout(rows) > kNhwcSmem) --rows;
    auto tiles = [&](int r) { return (long long)pl.B * pl.tiles_x * ((pl.OH + r - 1) / r); };
    while (rows > 2 && tiles(rows) < 2ll * sm_count) rows = (rows + 1) / 2;
    rows = (pl.OH + (pl.OH + rows - 1) / rows - 1) / ((pl.OH + rows - 1) / rows);   // equal heights
    pl.rows = rows;
    pl.tiles_y = (pl.OH + rows - 1) / rows;
    if (tiles(rows) > (1ll << 30)) return 0;
    pl.tiles = (int)tiles(rows);
    const uint32_t smem = layout(rows);
    return smem <= kNhwcSmem ? smem : 0;
}

}  // namespace ddf
