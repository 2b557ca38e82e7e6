// Channels-innermost (NHWC, torch "channels_last") DDF forward for 2-byte element types, and
// the pooled sums the channel branch needs, so that a channels_last network runs its DDF
// layers without any layout copy.
//
// Mapping.  A thread owns 8 adjacent channels (one 16-byte vector) of one output pixel column.  Its channel-filter
// values -- K*K taps x 8 channels, fixed for a sample -- sit in
// registers as packed 2-byte pairs laid out like the input words (channels 2q, 2q+1 in word
// q), so the mixed-precision FMA forms x * cf for both halves of a word without any
// unpacking:  y = x * cf (exact in float),  acc = fma(y, sf, acc)  with the pixel's
// spatial-filter value in float.  An optional per-channel affine map
// and ReLU (an eval-mode BatchNorm + activation) ride on the store.
//
// Movement.  A CTA's threads cover all channels of a few columns; a tile is these columns of a few output rows.
// The CTAs are persistent and walk neighbouring tiles, the next tile's input rows (one contiguous run each, with the
// halo columns) arriving by bulk copies in the other of two buffers meanwhile.  Three columns' threads read each
// vector, and a row serves three output rows; loaded from global memory by each of them, one row ahead, the kernel had
// some 8 KB of distinct data in flight per SM and ran at a sixth of the memory's rate.  Pixels outside
// the image are not read (zeros take their place).  The spatial filter is the same for all channels of a pixel: bias
// and FilterNorm are applied once per pixel, by one thread, and the result is left in shared memory.
// The sixteen layers of a ResNet-50 at 256 images of 224 x 224, float16: 822 -> 670 us.  Bound now by the 16 warps that an SM
// holds at 128 registers (stride 1 spills up to 36 bytes beyond them; at 64 channels 28 of 32 columns have pixels), which
// meet at a barrier once per tile, and the FMA pipe.
#include <atomic>

#include "common.cuh"
#include "nhwc_plan.h"
#include "ring_fwd.cuh"

namespace ddf {

extern std::atomic<unsigned long long> g_launches;
int device_facts(int* sm_count, int** fault, int* index);

__device__ __forceinline__ uint4 ldg128(const void* p) {
    uint4 v;
    asm volatile("ld.global.nc.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}

template <typename T> __device__ __forceinline__ float elem_to_float(uint32_t h);
template <> __device__ __forceinline__ float elem_to_float<__nv_bfloat16>(uint32_t h) { return __uint_as_float(h << 16); }
template <> __device__ __forceinline__ float elem_to_float<__half>(uint32_t h) {
    return __uint_as_float(Mix<__half>::f32_bits(h));
}
template <typename T> __device__ __forceinline__ uint32_t pack2(float a, float b) { return Word<T>::put(a, b); }

template <typename T> __device__ __forceinline__ uint32_t relu2(uint32_t v);   // of two packed values; NaN becomes 0, as fmaxf makes it
template <> __device__ __forceinline__ uint32_t relu2<__half>(uint32_t v) {
    uint32_t r;
    asm("max.f16x2 %0, %1, %2;" : "=r"(r) : "r"(v), "r"(0u));
    return r;
}
template <> __device__ __forceinline__ uint32_t relu2<__nv_bfloat16>(uint32_t v) {
    uint32_t r;
    asm("max.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(v), "r"(0u));
    return r;
}

// Bytes of a pixel's filter in shared memory: mul (s, s) float pairs, add packed 2-byte values; whole 16s.
template <int MODE> constexpr uint32_t kNhwcPixel = MODE == DDF_B200_MUL ? 80 : 32;

// NORM: `sf` holds the raw output of the spatial branch's convolution; bias and FilterNorm here.
template <typename T, int S, int MODE, bool NORM>
__global__ void __launch_bounds__(kNhwcThreads, 2) nhwc_forward_kernel(const __grid_constant__ NhwcPlan pl) {
    constexpr int K = 3, KK = 9;
    constexpr bool MUL = MODE == DDF_B200_MUL;
    constexpr uint32_t PXB = kNhwcPixel<MODE>;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const uint32_t sbase = smem_u32(smem_raw);
    const int tid = threadIdx.x;
    const int vec = tid % pl.vecs, col = tid / pl.vecs;
    const int C = pl.C, W = pl.W, H = pl.H, OW = pl.OW, OH = pl.OH;
    const uint32_t affine = sbase + pl.off_affine;
#define NH_FULL(i) (sbase + 8u * (uint32_t)(i))
#define NH_BUF(i) (sbase + pl.off_buf + (uint32_t)(i) * pl.buf_stride)

    if (tid == 0) {
        mbar_init(NH_FULL(0), 1);
        mbar_init(NH_FULL(1), 1);
        mbar_fence_init();
    }
    if (tid < KK) sts32(sbase + 16u + 4u * tid, pl.sf_bias != nullptr ? __float_as_uint(__ldg(pl.sf_bias + tid)) : 0u);
    if (pl.oscale != nullptr)
        for (int c = tid; c < C; c += kNhwcThreads) {
            sts32(affine + 4u * c, __float_as_uint(__ldg(pl.oscale + c)));
            sts32(affine + 4u * (C + c), __float_as_uint(__ldg(pl.oshift + c)));
        }
    __syncthreads();

    const int t_lo = (int)(((long long)pl.tiles * blockIdx.x) / gridDim.x);
    const int t_hi = (int)(((long long)pl.tiles * (blockIdx.x + 1)) / gridDim.x);
    // tiles run along a row of tiles, down an image, image by image; found by division once
    struct Tile { int b, ox0, oy0, nx, ny; };
    auto clip = [&](Tile& r) {
        r.nx = OW - r.ox0 < pl.cols ? OW - r.ox0 : pl.cols;
        r.ny = OH - r.oy0 < pl.rows ? OH - r.oy0 : pl.rows;
    };
    auto next_of = [&](Tile r) {
        r.ox0 += pl.cols;
        if (r.ox0 >= OW) {
            r.ox0 = 0;
            r.oy0 += pl.rows;
            if (r.oy0 >= OH) {
                r.oy0 = 0;
                ++r.b;
            }
        }
        clip(r);
        return r;
    };
    Tile r;
    {
        const int per = pl.tiles_x * pl.tiles_y, in = t_lo % per, ty = in / pl.tiles_x;
        r.b = t_lo / per;
        r.ox0 = (in - ty * pl.tiles_x) * pl.cols;
        r.oy0 = ty * pl.rows;
        clip(r);
    }
    // the first warp: the tile's input rows and its raw filters into a buffer, a row per lane.  Window column 0 of the
    // tile lies at a row's start, window row 0 at the buffer's.
    auto request = [&](const Tile& r, int t) {
        const int buf = (t - t_lo) & 1;
        const int ix0 = r.ox0 * S - 1, iy0 = r.oy0 * S - 1;
        const int cx0 = ix0 > 0 ? ix0 : 0, cx1 = (ix0 + (r.nx - 1) * S + K) < W ? (ix0 + (r.nx - 1) * S + K) : W;
        const int cy0 = iy0 > 0 ? iy0 : 0, cy1 = (iy0 + (r.ny - 1) * S + K) < H ? (iy0 + (r.ny - 1) * S + K) : H;
        const int n = cy1 - cy0;
        const uint32_t bytes = (uint32_t)(cx1 - cx0) * (uint32_t)C * 2u;
        // the filters of the tile's rows: as many bytes each, but for the last one of an image
        const uint32_t sfb = pl.sf_bulk ? (uint32_t)(r.nx * (int)pl.sf_pixel_stride) * 2u : 0u;
        const uint32_t sfb_last = pl.sf_bulk ? nhwc_filter_run(pl, r.b, r.oy0 + r.ny - 1, r.ox0, r.nx).bytes : 0u;
        if (tid == 0)
            mbar_arrive_expect_tx(NH_FULL(buf), (uint32_t)n * bytes + (uint32_t)(r.ny - 1) * sfb + sfb_last +
                                                    (t - t_lo + 1 == pl.starve ? 16u : 0u));
        __syncwarp();
        if (tid < n) {
            bulk_g2s(NH_BUF(buf) + (uint32_t)(cy0 - iy0 + tid) * pl.row_bytes + (uint32_t)((cx0 - ix0) * C * 2),
                     reinterpret_cast<const T*>(pl.x) + (((size_t)r.b * H + cy0 + tid) * W + cx0) * C, bytes, NH_FULL(buf));
        } else if (pl.sf_bulk && tid < n + r.ny) {
            const int y = tid - n;
            const NhwcRun run = nhwc_filter_run(pl, r.b, r.oy0 + y, r.ox0, r.nx);
            bulk_g2s(NH_BUF(buf) + pl.off_raw + (uint32_t)(y * pl.cols * (int)pl.sf_pixel_stride) * 2u,
                     reinterpret_cast<const T*>(pl.sf) + run.from, run.bytes, NH_FULL(buf));
        }
    };
    static_assert((kNhwcRows - 1) * S + K + kNhwcRows <= 32, "a lane per row of a tile and of its filters");
    if (tid < 32) {
        if (t_lo < t_hi) request(r, t_lo);
        if (t_lo + 1 < t_hi) request(next_of(r), t_lo + 1);
    }

    // a thread's constants of the row loop, kept (see pin)
    uint32_t row_bytes = pl.row_bytes, pixel_bytes = (uint32_t)C * 2u, aff_s = affine + 32u * (uint32_t)vec;
    unsigned long long out_step = (unsigned long long)OW * C * 2u;
    pin(row_bytes);
    pin(pixel_bytes);
    pin(aff_s);
    pin(out_step);
    uint32_t cfw[KK][4];
    int cf_of = -1;   // the sample whose channel filters are in registers
    for (int t = t_lo; t < t_hi; ++t) {
        const int buf = (t - t_lo) & 1;
        const bool active = col < r.nx;
        if (r.b != cf_of) {
            // channel filter of this thread's 8 channels: 72 contiguous values -> cfw[t][q] = channels (2q, 2q+1) of tap t
            cf_of = r.b;
            const uint4* cp = reinterpret_cast<const uint4*>(reinterpret_cast<const T*>(pl.cf) + ((size_t)r.b * C + vec * 8) * KK);
            uint32_t raw[36];
#pragma unroll
            for (int v = 0; v < 9; ++v) {
                const uint4 u = ldg128(cp + v);
                raw[4 * v] = u.x; raw[4 * v + 1] = u.y; raw[4 * v + 2] = u.z; raw[4 * v + 3] = u.w;
            }
#pragma unroll
            for (int k = 0; k < KK; ++k) {
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int ha = (2 * q) * KK + k, hb = (2 * q + 1) * KK + k;   // element indices
                    const uint32_t lo = (ha & 1) ? (raw[ha / 2] >> 16) : (raw[ha / 2] & 0xffffu);
                    const uint32_t hi = (hb & 1) ? (raw[hb / 2] & 0xffff0000u) : (raw[hb / 2] << 16);
                    cfw[k][q] = lo | hi;
                }
            }
        }
        const bool late = !mbar_wait_for(NH_FULL(buf), (uint32_t)(((t - t_lo) >> 1) & 1), pl.wait_cycles);
        if (late) atomicCAS(pl.fault, 0, (int)kFaultConsumerFull);
        // Window columns and rows outside the image: zeros, where the copies left something else.
        {
            const int ix0 = r.ox0 * S - 1, iy0 = r.oy0 * S - 1, cols = (r.nx - 1) * S + K, rows = (r.ny - 1) * S + K;
            auto zero_column = [&](int c) {
                for (int e = tid; e < rows * pl.vecs; e += kNhwcThreads)
                    sts128(NH_BUF(buf) + (uint32_t)(e / pl.vecs) * pl.row_bytes + (uint32_t)((c * pl.vecs + e % pl.vecs) * 16), 0u, 0u, 0u, 0u);
            };
            auto zero_row = [&](int y) {
                for (int e = tid; e < cols * pl.vecs; e += kNhwcThreads)
                    sts128(NH_BUF(buf) + (uint32_t)y * pl.row_bytes + (uint32_t)(e * 16), 0u, 0u, 0u, 0u);
            };
            if (ix0 < 0) zero_column(0);
            if (ix0 + cols > W) zero_column(cols - 1);
            if (iy0 < 0) zero_row(0);
            if (iy0 + rows > H) zero_row(rows - 1);
            if (ix0 < 0 || iy0 < 0 || ix0 + cols > W || iy0 + rows > H)
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // before the copies that come here next
        }
        // the filters of the tile's pixels, a pixel per thread and turn
        const uint32_t filters = sbase + pl.off_sf + (uint32_t)buf * pl.sf_stride;
        for (int i = tid; i < r.nx * r.ny; i += kNhwcThreads) {
            const int py = i / r.nx, px = i - py * r.nx;
            float sv[KK];
            if (pl.sf_bulk) {
                const uint32_t from = NH_BUF(buf) + pl.off_raw + (uint32_t)((py * pl.cols + px) * (int)pl.sf_pixel_stride) * 2u;
                uint32_t raw[5];
                lds128(from, raw[0], raw[1], raw[2], raw[3]);
                if (nhwc_last_pixel(pl, r.oy0 + py, r.ox0 + px))
                    raw[4] = __ldg(reinterpret_cast<const uint16_t*>(pl.sf) + r.b * pl.sf_batch_stride +
                                   ((long long)OH * OW - 1) * pl.sf_pixel_stride + 8);
                else raw[4] = lds16(from + 16u);
#pragma unroll
                for (int k = 0; k < KK; ++k) sv[k] = elem_to_float<T>((k & 1) ? (raw[k / 2] >> 16) : (raw[k / 2] & 0xffffu));
            } else {
                const T* spp = reinterpret_cast<const T*>(pl.sf) + r.b * pl.sf_batch_stride +
                               ((long long)(r.oy0 + py) * OW + r.ox0 + px) * pl.sf_pixel_stride;
#pragma unroll
                for (int k = 0; k < KK; ++k)
                    sv[k] = elem_to_float<T>(__ldg(reinterpret_cast<const uint16_t*>(spp + k * pl.sf_tap_stride)));
            }
            if constexpr (NORM) {
                float sum = 0.f;
#pragma unroll
                for (int k = 0; k < KK; ++k) {
                    sv[k] += ldsf(sbase + 16u + 4u * k);   // (zeros without one)
                    sum += sv[k];
                }
                const float mean = sum * (1.f / KK);
                float var = 0.f;
#pragma unroll
                for (int k = 0; k < KK; ++k) {
                    sv[k] -= mean;
                    var = fmaf(sv[k], sv[k], var);
                }
                const float inv = norm_gain(var * (1.f / (KK - 1)), pl.sf_scale);
#pragma unroll
                for (int k = 0; k < KK; ++k) sv[k] *= inv;
            }
            // a column's pixels in a row, and 16 bytes, so that neighbouring columns lie in different banks
            const uint32_t at = filters + (uint32_t)px * ((uint32_t)pl.rows * PXB + 16u) + (uint32_t)py * PXB;
            if constexpr (MUL) {
#pragma unroll
                for (int k = 0; k < KK; ++k) sts64(at + 8u * k, __float_as_uint(sv[k]), __float_as_uint(sv[k]));
            } else {
                sts128(at, pack2<T>(sv[0], sv[1]), pack2<T>(sv[2], sv[3]), pack2<T>(sv[4], sv[5]), pack2<T>(sv[6], sv[7]));
                sts32(at + 16u, pack2<T>(sv[8], 0.f));
            }
        }
        if (__syncthreads_or(late)) {
            // All threads leave together and store no more.  The copies under way -- this tile's, and behind the first
            // one the next tile's too -- land before the block's memory goes.
            if (tid == 0) {
                bool landed = mbar_wait_for(NH_FULL(buf), (uint32_t)(((t - t_lo) >> 1) & 1), pl.wait_cycles);
                if (t == t_lo && t + 1 < t_hi) landed &= mbar_wait_for(NH_FULL(buf ^ 1), 0u, pl.wait_cycles);
                if (!landed && pl.starve == 0) atomicExch(pl.fault, (int)kFaultDrain);
            }
            __syncthreads();
            return;
        }
        // every thread is done with the tile before: its buffer takes the next one
        const Tile next = next_of(r);
        if (tid < 32 && t > t_lo && t + 1 < t_hi) request(next, t + 1);

        if (active) {
            const int ox = r.ox0 + col;
            uint32_t row_s = NH_BUF(buf) + (uint32_t)((col * S * C + vec * 8) * 2);   // the next window row to read
            auto load_row = [&](uint32_t (&v)[K][4]) {
#pragma unroll
                for (int j = 0; j < K; ++j) lds128(row_s + (uint32_t)j * pixel_bytes, v[j][0], v[j][1], v[j][2], v[j][3]);
                row_s += row_bytes;
            };
            uint32_t w[3][K][4];   // input rows, round robin
            load_row(w[0]);
            if constexpr (S == 1) load_row(w[1]);
            uint32_t sf_s = filters + (uint32_t)col * ((uint32_t)pl.rows * PXB + 16u);
            char* op = reinterpret_cast<char*>(pl.out) + ((((size_t)r.b * OH + r.oy0) * OW + ox) * C + vec * 8) * 2;
            for (int y = 0; y < r.ny;) {
#pragma unroll
                for (int u = 0; u < 3; ++u) {
                    uint32_t (&r0)[K][4] = w[(S * u) % 3];
                    uint32_t (&r1)[K][4] = w[(S * u + 1) % 3];
                    uint32_t (&r2)[K][4] = w[(S * u + 2) % 3];
                    if constexpr (S == 2) load_row(r1);
                    load_row(r2);
                    unsigned long long acc2[4] = {0ull, 0ull, 0ull, 0ull};
                    float acc[8];
                    unsigned long long sd[MUL ? 10 : 1];
                    uint32_t sw[MUL ? 1 : 5];
                    if constexpr (MUL) {
#pragma unroll
                        for (int k = 0; k < 10; k += 2)
                            asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(sd[k]), "=l"(sd[k + 1]) : "r"(sf_s + 8u * k));
                    } else {
                        lds128(sf_s, sw[0], sw[1], sw[2], sw[3]);
                        sw[4] = lds32(sf_s + 16u);
#pragma unroll
                        for (int c = 0; c < 8; ++c) acc[c] = 0.f;
                    }
#pragma unroll
                    for (int i = 0; i < K; ++i) {
#pragma unroll
                        for (int j = 0; j < K; ++j) {
                            const int k = i * K + j;
#pragma unroll
                            for (int q = 0; q < 4; ++q) {
                                const uint32_t xw = i == 0 ? r0[j][q] : (i == 1 ? r1[j][q] : r2[j][q]);
                                if constexpr (MUL) {
                                    // the two channels of a word: exact products, then one packed f32x2 FMA
                                    // against the tap's spatial-filter value (half the issue slots of two FFMAs)
                                    const float y0 = Mix<T>::fmaw(0, 0, xw, cfw[k][q], 0.f);
                                    const float y1 = Mix<T>::fmaw(1, 1, xw, cfw[k][q], 0.f);
                                    acc2[q] = f2_fma(f2_pack(y0, y1), sd[k], acc2[q]);
                                } else {
#pragma unroll
                                    for (int h = 0; h < 2; ++h) {
                                        float a = acc[2 * q + h];
                                        a = Mix<T>::fmaw(h, h, xw, cfw[k][q], a);
                                        a = Mix<T>::fmaw(h, k & 1, xw, sw[k / 2], a);
                                        acc[2 * q + h] = a;
                                    }
                                }
                            }
                        }
                    }
                    if constexpr (!MUL) {
#pragma unroll
                        for (int q = 0; q < 4; ++q) acc2[q] = f2_pack(acc[2 * q], acc[2 * q + 1]);
                    }
                    if (pl.oscale != nullptr) {
                        unsigned long long sc[4], sh[4];
#pragma unroll
                        for (int q = 0; q < 4; q += 2) {
                            asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(sc[q]), "=l"(sc[q + 1]) : "r"(aff_s + 8u * q));
                            asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(sh[q]), "=l"(sh[q + 1]) : "r"(aff_s + 2u * pixel_bytes + 8u * q));
                        }
#pragma unroll
                        for (int q = 0; q < 4; ++q) acc2[q] = f2_fma(acc2[q], sc[q], sh[q]);
                    }
                    uint32_t o[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        float lo, hi;
                        f2_unpack(acc2[q], lo, hi);
                        o[q] = pack2<T>(lo, hi);
                        if (pl.relu) o[q] = relu2<T>(o[q]);
                    }
                    *reinterpret_cast<uint4*>(op) = make_uint4(o[0], o[1], o[2], o[3]);
                    op += out_step;
                    sf_s += PXB;
                    if (++y >= r.ny) break;
                }
            }
        }
        r = next;
    }
#undef NH_FULL
#undef NH_BUF
}

// Partial sums of x over tiles of up to 196 pixels: partials[b][tile][c] (float), for the channel branch's
// global average pool.  One CTA per (tile, sample).
// A quarter of the image at most, so that small maps have CTAs enough for their loads to be in flight
// (a tile is a CTA).  Float16, 256 images, us: (256,14x14) 10.5 -> 8.1, (512,14x14) 18.4 -> 11.9, (256,28x28) 24.3 -> 19.4,
// (64,56x56) 26.7 -> 24.2.  Bound by the latency of the loads.
constexpr int kPoolTile = 196;
__host__ __device__ __forceinline__ int pool_tile(int HW) { return HW < 4 * kPoolTile ? (HW + 3) / 4 : kPoolTile; }
template <typename T>
__global__ void __launch_bounds__(256) nhwc_pool_kernel(const T* __restrict__ x, float* __restrict__ partials, int C,
                                                        int HW, int n_tiles) {
    extern __shared__ float red[];   // [lanes][C]
    const int vecs = C / 8, tid = threadIdx.x;
    const int vec = tid % vecs, lane = tid / vecs, lanes = blockDim.x / vecs;
    const int b = blockIdx.y, tile = blockIdx.x;
    const int step = pool_tile(HW), p0 = tile * step, p1 = (p0 + step) < HW ? (p0 + step) : HW;
    float s[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    const T* xb = x + (size_t)b * HW * C + vec * 8;
    for (int p = p0 + lane; p < p1; p += lanes) {
        const uint4 u = ldg128(xb + (size_t)p * C);
        const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            s[2 * q] += elem_to_float<T>(w[q] & 0xffffu);
            s[2 * q + 1] += elem_to_float<T>(w[q] >> 16);
        }
    }
#pragma unroll
    for (int c = 0; c < 8; ++c) red[lane * C + vec * 8 + c] = s[c];
    __syncthreads();
    for (int c = tid; c < C; c += blockDim.x) {
        float t = 0.f;
        for (int l = 0; l < lanes; ++l) t += red[l * C + c];   // fixed order
        partials[((size_t)b * n_tiles + tile) * C + c] = t;
    }
}

template <typename T, int S, int MODE>
static int nhwc_launch(const NhwcPlan& pl, int norm, uint32_t smem, int device, dim3 grid, cudaStream_t st) {
    auto kern = norm ? nhwc_forward_kernel<T, S, MODE, true> : nhwc_forward_kernel<T, S, MODE, false>;
    static std::atomic<unsigned long long> opted_in[2];
    const unsigned long long bit = 1ull << (device & 63);
    if (!(opted_in[norm ? 1 : 0].load(std::memory_order_acquire) & bit)) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kNhwcSmem);
        if (e != cudaSuccess) return (int)e;
        opted_in[norm ? 1 : 0].fetch_or(bit, std::memory_order_release);
    }
    kern<<<grid, kNhwcThreads, smem, st>>>(pl);
    return (int)cudaGetLastError();
}

template <typename T>
static int nhwc_dispatch(const NhwcPlan& pl, int s, int combine, int norm, uint32_t smem, int device, dim3 grid, cudaStream_t st) {
    if (combine == DDF_B200_MUL)
        return s == 1 ? nhwc_launch<T, 1, DDF_B200_MUL>(pl, norm, smem, device, grid, st)
                      : nhwc_launch<T, 2, DDF_B200_MUL>(pl, norm, smem, device, grid, st);
    return s == 1 ? nhwc_launch<T, 1, DDF_B200_ADD>(pl, norm, smem, device, grid, st)
                  : nhwc_launch<T, 2, DDF_B200_ADD>(pl, norm, smem, device, grid, st);
}

}  // namespace ddf

using namespace ddf;

extern "C" {

int ddf_b200_pool_nhwc_tiles(int H, int W) {
    if (H < 1 || W < 1) return DDF_B200_E_SHAPE;
    return (H * W + pool_tile(H * W) - 1) / pool_tile(H * W);
}

int ddf_b200_pool_nhwc(const void* x, float* partials, int B, int C, int H, int W, int dtype, void* stream) {
    if (!x || !partials) return DDF_B200_E_NULL;
    if (B < 1 || C < 1 || H < 1 || W < 1) return DDF_B200_E_SHAPE;
    if (dtype != DDF_B200_F16 && dtype != DDF_B200_BF16) return DDF_B200_E_UNSUPPORTED;
    if (C % 8 != 0 || C > 2048 || 256 % (C / 8) != 0 || B > 65535) return DDF_B200_E_UNSUPPORTED;
    if ((reinterpret_cast<uintptr_t>(x) & 15u) != 0) return DDF_B200_E_UNSUPPORTED;
    const int nt = ddf_b200_pool_nhwc_tiles(H, W);
    const int lanes = 256 / (C / 8);
    const size_t smem = (size_t)lanes * C * sizeof(float);   // = 8 KB
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    dim3 grid((unsigned)nt, (unsigned)B);
    if (dtype == DDF_B200_F16)
        nhwc_pool_kernel<__half><<<grid, 256, smem, st>>>((const __half*)x, partials, C, H * W, nt);
    else
        nhwc_pool_kernel<__nv_bfloat16><<<grid, 256, smem, st>>>((const __nv_bfloat16*)x, partials, C, H * W, nt);
    g_launches.fetch_add(1, std::memory_order_relaxed);
    return (int)cudaGetLastError();
}

static int nhwc_forward(const void* x, const void* cf, const void* sf, const float* sf_bias, void* out,
                        const float* out_scale, const float* out_shift, int relu, int B, int C, int H, int W,
                        int k, int d, int s, int combine, int dtype, long long sf_batch_stride,
                        long long sf_pixel_stride, long long sf_tap_stride, int norm, double sf_scale,
                        long long wait_cycles, int starve, void* stream) {
    if (!x || !cf || !sf || !out) return DDF_B200_E_NULL;
    if ((out_scale == nullptr) != (out_shift == nullptr)) return DDF_B200_E_NULL;
    if (B < 1 || C < 1 || H < 1 || W < 1 || s < 1 || H / s < 1 || W / s < 1) return DDF_B200_E_SHAPE;
    if (combine != DDF_B200_MUL && combine != DDF_B200_ADD) return DDF_B200_E_COMBINE;
    if (dtype < DDF_B200_F32 || dtype > DDF_B200_F64) return DDF_B200_E_DTYPE;
    if (k < 1 || (k - 1) % 2 != 0 || d < 1) return DDF_B200_E_KERNEL;
    // built for the DDF-ResNet layers: k = 3, d = 1, stride 1 or 2, 2-byte types, C a multiple of 8
    if (k != 3 || d != 1 || s > 2 || (dtype != DDF_B200_F16 && dtype != DDF_B200_BF16)) return DDF_B200_E_UNSUPPORTED;
    if (C % 8 != 0 || C > 2048 || kNhwcThreads % (C / 8) != 0 || B > 65535) return DDF_B200_E_UNSUPPORTED;
    if (W != (W / s) * s) return DDF_B200_E_UNSUPPORTED;
    auto al16 = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15u) == 0; };
    if (!al16(x) || !al16(cf) || !al16(out)) return DDF_B200_E_UNSUPPORTED;
    int sm_count = 0, index = 0;
    int* fault = nullptr;
    int rc = device_facts(&sm_count, &fault, &index);
    if (rc) return rc;

    NhwcPlan pl;
    pl.x = x; pl.cf = cf; pl.sf = sf; pl.sf_bias = sf_bias; pl.out = out;
    pl.oscale = out_scale; pl.oshift = out_shift;
    pl.B = B; pl.C = C; pl.H = H; pl.W = W; pl.OH = H / s; pl.OW = W / s;
    pl.sf_batch_stride = sf_batch_stride; pl.sf_pixel_stride = sf_pixel_stride; pl.sf_tap_stride = sf_tap_stride;
    pl.relu = relu; pl.sf_scale = (float)sf_scale;
    pl.vecs = C / 8;
    pl.fault = fault; pl.wait_cycles = wait_cycles; pl.starve = starve;
    // bulk copies of the raw filters: taps contiguous, whole 16 bytes a pixel, pixels of a row one after the other
    pl.sf_bulk = (sf_tap_stride == 1 && sf_pixel_stride % 8 == 0 && sf_pixel_stride >= 16 && sf_pixel_stride <= 64 &&
                  sf_batch_stride % 8 == 0 && al16(sf)) ? 1 : 0;
    const uint32_t smem = nhwc_tiles(pl, s, combine == DDF_B200_MUL ? kNhwcPixel<DDF_B200_MUL> : kNhwcPixel<DDF_B200_ADD>, sm_count);
    if (smem == 0) return DDF_B200_E_UNSUPPORTED;
    dim3 grid((unsigned)(pl.tiles < 2 * sm_count ? pl.tiles : 2 * sm_count));
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    rc = dtype == DDF_B200_F16 ? nhwc_dispatch<__half>(pl, s, combine, norm, smem, index, grid, st)
                               : nhwc_dispatch<__nv_bfloat16>(pl, s, combine, norm, smem, index, grid, st);
    if (rc == 0) g_launches.fetch_add(1, std::memory_order_relaxed);
    return rc;
}

int ddf_b200_forward_nhwc(const void* x, const void* cf, const void* sf, const float* sf_bias, void* out,
                          const float* out_scale, const float* out_shift, int relu, int B, int C, int H, int W,
                          int k, int d, int s, int combine, int dtype, long long sf_batch_stride,
                          long long sf_pixel_stride, long long sf_tap_stride, int norm, double sf_scale,
                          void* stream) {
    return nhwc_forward(x, cf, sf, sf_bias, out, out_scale, out_shift, relu, B, C, H, W, k, d, s, combine, dtype,
                        sf_batch_stride, sf_pixel_stride, sf_tap_stride, norm, sf_scale, kWaitCycles, 0, stream);
}

int ddf_b200_nhwc_waitlimit(const void* x, const void* cf, const void* sf, void* out, int B, int C, int H, int W, int k,
                            int d, int s, int combine, int dtype, long long sf_batch_stride, long long sf_pixel_stride,
                            long long sf_tap_stride, long long wait_cycles, int starve, void* stream) {
    if (wait_cycles < 1 || starve < 0) return DDF_B200_E_SHAPE;
    return nhwc_forward(x, cf, sf, nullptr, out, nullptr, nullptr, 0, B, C, H, W, k, d, s, combine, dtype, sf_batch_stride,
                        sf_pixel_stride, sf_tap_stride, 0, 1.0, wait_cycles, starve, stream);
}

}  // extern "C"
