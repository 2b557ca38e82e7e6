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

}  // namespace ddf
