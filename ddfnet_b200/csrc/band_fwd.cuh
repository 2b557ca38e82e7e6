// Band kernel: DDF forward (and grad-x at stride 1) for planes of any height and any width up to 320 output
// columns (352 at k = 5: a band holds whole rows, a CTA a column per thread), k = 3 and 5, dilation 1 and 2
// (stride 1) or stride 2 (k = 3, dilation 1), float and the 2-byte types.  It takes
// what the plane kernels (row, ring, stream) decline: planes too large for one CTA's threads, widths
// that no vector divides, H or W that the stride does not divide, channel counts without a factor.
//
// Work split.  A plane is cut into bands of output rows over the whole width.  The input rows of a band
// are one contiguous run of a plane, so a channel's share is ONE untiled bulk copy whatever the width;
// runs start anywhere, the copy fetches the 16-byte-aligned superset (span_prepare) and the readers add
// the remainder.  Small planes travel several to a copy.  The (sample, band, channel) units form one line
// that a persistent grid cuts into equal shares: no last wave, and a producer lane keeps a ring of slots
// full across the changes of band.  At such a change the compute warps reload their filters.
//
// A thread owns PH output pixels of one column, D rows apart (so neighbouring windows share rows at
// every dilation).  Lanes of a warp own neighbouring columns: every shared load is conflict-free and
// every store coalesced at any width and alignment, which vectors along x would not be.  The k*k*PH
// filter values stay in registers, paired (p, p + PH/2) for the two-wide FMA.  A column of the window is
// loaded once and serves k taps of PH pixels.
//
// What bounds it: instruction issue and the latency of a pass at 20 warps per SM ((2,256,200x300) f32: 57% of
// issue slots busy, DRAM at 31% of its peak, shared loads at 29%), and on small problems the filters' way into
// registers: one pointer per pixel instead of an address per value took (4,128,50x67) f16 from 17.7 to 11.3 us.
// (2,256,200x300) f32: 80 us, 3.1 TB/s; the generic kernel 655.  Eight pixels per thread instead of four (half
// the CTAs fit): 97; scalar instead of two-wide FMAs: 93 (k = 5, (8,96,75x101): 50 against 58 before the
// pointers, 48 after).
//
// Zero padding.  Rows outside the plane are read from a zeroed spot of the slot (their offset is a
// per-thread constant), columns outside are masked.  A zero times an infinite filter value would be
// NaN where the definition skips the tap: while the filters hold anything not below kBandFilterMax
// in magnitude (so that cf * sf is finite too) a CTA takes a plain loop that skips those taps.
//
// Every mbarrier wait is bounded by the plan's wait_cycles.  A thread whose wait ran out records a fault,
// stays for the barriers of the others, and neither stores nor hands slots back: the producer's own wait
// then runs out and it issues no more.  The producer leaves, always, after the last copies have landed.
#pragma once

#include <atomic>

#include "common.cuh"
#include "stream_fwd.cuh"

namespace ddf {

constexpr int kBandSlots = 8;
constexpr int kBandStage = 64;       // channels whose filters are staged together
constexpr float kBandFilterMax = 1e18f;
constexpr uint32_t kBandGuard = 32;  // readable bytes before a slot's data (left halo of its first row)
constexpr uint32_t kBandZero = 80;   // zeroed bytes after it
constexpr uint32_t kBandDead = 2;    // bit of a compute thread's ring phase: one of its waits ran out

struct BandPlan {
    const void* in;
    const void* cf;
    const void* sf;
    void* out;
    int C, H, W, OH, OW;      // input plane, output plane
    int bands, groups;        // bands per plane; column groups (PH pixels each) per band
    int planes;               // planes per unit (> 1 only when a band is the whole plane)
    int passes;               // units per (sample, band) = ceil(C / planes)
    int stage_passes;         // units whose channel filters are staged together
    int units;
    int n_slots, n_warps;
    int bwdx, norm;
    float sf_scale;
    unsigned long long in_total;
    uint32_t off_cf, off_slot0, slot_stride, zero_off;  // zero_off: from a slot's data start
    int* fault;
    long long wait_cycles;    // limit of every mbarrier wait, in SM clocks
    uint32_t tx_skew;         // self-test: bytes announced beyond what is copied, so that no stage completes
};

// Ring hand-over of the band kernels' producer lane: its wait for a free slot, and, before it leaves, the
// waits for the last copies (the block's shared memory must not go while they are in flight).
__device__ __forceinline__ bool band_slot_free(uint32_t bar_empty, int issued, int nst, long long wait_cycles, uint32_t skew) {
    // with the self-test's skew the compute warps, whose limit is shorter, report first
    return issued < nst || mbar_wait_for(bar_empty, (uint32_t)((issued / nst - 1) & 1), skew ? 2 * wait_cycles : wait_cycles);
}
__device__ __forceinline__ void band_leave(uint32_t bar_full0, int issued, int n, int nst, long long wait_cycles, uint32_t skew,
                                           int* fault) {
    if (issued < n) atomicCAS(fault, 0, (int)kFaultService);
    bool landed = true;
    for (int j = issued > nst ? issued - nst : 0; j < issued; ++j)
        landed &= mbar_wait_for(bar_full0 + 8u * (uint32_t)(j % nst), (uint32_t)((j / nst) & 1), wait_cycles);
    if (!landed && skew == 0) atomicExch(fault, (int)kFaultDrain);
}

// Element loads with a per-thread column mask folded into the conversion.
template <typename T> struct Masked;
template <> struct Masked<float> {
    static __device__ __forceinline__ uint32_t mask(bool ok) { return ok ? 0xffffffffu : 0u; }
    static __device__ __forceinline__ float load(uint32_t a, uint32_t m) { return __uint_as_float(lds32(a) & m); }
    static __device__ __forceinline__ float load(uint32_t a) { return ldsf(a); }
};
template <> struct Masked<__nv_bfloat16> {
    static __device__ __forceinline__ uint32_t mask(bool ok) { return ok ? 0x1044u : 0x4444u; }
    static __device__ __forceinline__ float load(uint32_t a, uint32_t m) {
        return __uint_as_float(__byte_perm(lds16(a), 0u, m));
    }
    static __device__ __forceinline__ float load(uint32_t a) { return __uint_as_float(lds16(a) << 16); }
};
template <> struct Masked<__half> {
    static __device__ __forceinline__ uint32_t mask(bool ok) { return ok ? 0xffffffffu : 0u; }
    static __device__ __forceinline__ float load(uint32_t a, uint32_t m) { return Word<__half>::get(lds16(a) & m, 0); }
    static __device__ __forceinline__ float load(uint32_t a) { return Word<__half>::get(lds16(a), 0); }
};

// Bytes of a channel's filter in shared memory: (c, c) pairs column by column, each column padded to
// whole 16 bytes.
template <int K> constexpr int kBandCf = K * ((K + 1) / 2 * 16);

__device__ __forceinline__ void lds128_pairs(uint32_t a, unsigned long long& x, unsigned long long& y) {
    asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(x), "=l"(y) : "r"(a));
}

// Barriers among the `n` compute threads only: the producer runs ahead.
__device__ __forceinline__ void band_sync(int n) { asm volatile("barrier.cta.sync 1, %0;" ::"r"(n) : "memory"); }
__device__ __forceinline__ bool band_sync_or(int n, int v) {
    int r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.s32 p, %1, 0;\n\t"
        "barrier.cta.red.or.pred q, 1, %2, p;\n\t"
        "selp.s32 %0, 1, 0, q;\n\t}"
        : "=r"(r)
        : "r"(v), "r"(n)
        : "memory");
    return r != 0;
}

// k = 3: two CTAs per SM at 80 registers a thread; k = 5: the 100 filter values a thread holds leave one.
template <int K> constexpr int kBandThreads = K == 3 ? 352 : 384;
template <int K> constexpr int kBandCtas = K == 3 ? 2 : 1;
template <int K> constexpr int kBandRegs = K == 3 ? 80 : 168;

// Output row of a thread's first pixel.  Groups count in blocks of D: group g of a band covers rows
// (g / D) * PH * D + g % D, + D, + 2D ...
template <int D, int PH>
__device__ __forceinline__ int band_row(int group) { return D == 1 ? group * PH : (group / D) * (PH * D) + group % D; }

// Output rows from a band's first to its last.  Bands hold whole blocks of D groups, or, where the D groups
// of a wide plane would need more threads than a CTA has, one group.
template <int D, int PH>
__host__ __device__ __forceinline__ int band_rows(int groups) { return groups % D == 0 ? groups * PH : D * (PH - 1) + 1; }

template <typename T, int K, int D, int S, int PH, int MODE>
__global__ void __launch_bounds__(kBandThreads<K>, kBandCtas<K>)
band_kernel(const __grid_constant__ BandPlan pl) {
    constexpr int KK = K * K, R = (K - 1) / 2, ES = (int)sizeof(T);
    constexpr int NR = S * (PH - 1) + K;      // window rows of a thread, D input rows apart
    constexpr int HP = PH / 2;
    constexpr int CFC = (K + 1) / 2 * 16;     // bytes of one tap column's (c, c) pairs, whole 16s
    constexpr int CFB = kBandCf<K>;
    static_assert(D == 1 || S == 1, "dilated windows are built at stride 1");

    extern __shared__ __align__(128) unsigned char smem_raw[];
    const uint32_t sbase = smem_u32(smem_raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int NST = pl.n_slots, NW = pl.n_warps, G = pl.planes;
#define BAND_FULL(s) (sbase + 8u * (uint32_t)(s))
#define BAND_EMPTY(s) (sbase + 8u * (uint32_t)(kBandSlots + (s)))
#define BAND_DATA(s) (sbase + pl.off_slot0 + (uint32_t)(s) * pl.slot_stride + kBandGuard)

    if (tid == 0) {
        for (int s = 0; s < NST; ++s) {
            mbar_init(BAND_FULL(s), 1);
            mbar_init(BAND_EMPTY(s), (uint32_t)NW);
        }
        mbar_fence_init();
    }
    for (int e = tid; e < NST * (int)(kBandZero / 4); e += blockDim.x) {
        const int s = e / (int)(kBandZero / 4);
        sts32(BAND_DATA(s) + pl.zero_off + 4u * (uint32_t)(e - s * (int)(kBandZero / 4)), 0u);
    }
    __syncthreads();
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");

    const int u_lo = (int)(((unsigned long long)pl.units * blockIdx.x) / gridDim.x);
    const int u_hi = (int)(((unsigned long long)pl.units * (blockIdx.x + 1)) / gridDim.x);
    const unsigned long long plane_bytes = (unsigned long long)pl.H * pl.W * ES;
    // a (sample, band)'s rows
    struct Rows { int b, y_lo, iy_lo, iy_hi; };
    auto rows_of = [&](int seg) {
        Rows r;
        r.b = seg / pl.bands;
        const int band = seg - r.b * pl.bands;
        r.y_lo = band_row<D, PH>(band * pl.groups);
        const int y_next = r.y_lo + band_rows<D, PH>(pl.groups);
        const int y_hi = y_next < pl.OH ? y_next : pl.OH;
        r.iy_lo = r.y_lo * S - R * D > 0 ? r.y_lo * S - R * D : 0;
        const int iy_end = (y_hi - 1) * S + R * D + 1;
        r.iy_hi = iy_end < pl.H ? iy_end : pl.H;
        if (D > 1 && r.y_lo >= pl.OH) {  // the plane ends before this group: any row will do
            r.iy_lo = 0;
            r.iy_hi = 1;
        }
        return r;
    };
    auto run_start = [&](const Rows& r, int c) {
        return ((unsigned long long)r.b * pl.C + c) * plane_bytes + (unsigned long long)r.iy_lo * pl.W * ES;
    };

    if (warp == NW) {
        // ------------------------------------------------------------- producer
        if (lane != 0) return;
        int seg = u_lo / pl.passes;
        int pass = u_lo - seg * pl.passes;
        Rows r = rows_of(seg);
        const int n = u_hi - u_lo;
        int issued = 0;
        for (; issued < n; ++issued) {
            const int slot = issued % NST;
            if (!band_slot_free(BAND_EMPTY(slot), issued, NST, pl.wait_cycles, pl.tx_skew)) break;
            const int c = pass * G;
            const int count = pl.C - c < G ? pl.C - c : G;
            const unsigned long long g0 = run_start(r, c);
            const Span sp = span_prepare(BAND_DATA(slot), pl.in, g0,
                                         g0 + (unsigned long long)(count - 1) * plane_bytes +
                                             (unsigned long long)(r.iy_hi - r.iy_lo) * pl.W * ES,
                                         pl.in_total);
            mbar_arrive_expect_tx(BAND_FULL(slot), sp.bytes + pl.tx_skew);
            span_issue(sp, BAND_FULL(slot));
            if (++pass == pl.passes) {
                pass = 0;
                r = rows_of(++seg);
            }
        }
        band_leave(BAND_FULL(0), issued, n, NST, pl.wait_cycles, pl.tx_skew, pl.fault);
        return;
    }

    // ----------------------------------------------------------------- compute warps
    const int npos = pl.groups * pl.OW;
    int pip = tid / npos;
    int pos = tid - pip * npos;
    const bool owner = pip < G;
    if (!owner) { pip = 0; pos = 0; }
    const int grp = pos / pl.OW;
    const int x = pos - grp * pl.OW;
    uint32_t cmask[K];
#pragma unroll
    for (int j = 0; j < K; ++j) {
        const int ix = x * S + D * (j - R);
        cmask[j] = Masked<T>::mask(ix >= 0 && ix < pl.W);
    }
    const long long out_plane = (long long)pl.OH * pl.OW;
    const int row_step = D * pl.OW;
    const uint32_t g_step = (uint32_t)((unsigned long long)G * plane_bytes);

    int slot = -1;
    uint32_t ph = 1;
    int seg = u_lo / pl.passes;
    int pass = u_lo - seg * pl.passes;
    bool fresh = true;  // the next unit starts another (sample, band)
    Rows rw = rows_of(seg);
    int big_sf = 0;     // a spatial-filter value too large for products with padding zeros (or NaN)
    uint32_t rowoff[NR];
    unsigned long long sf2[KK][HP];  // spatial filters of this thread's pixels, [column-major tap][pair]
    int y0 = 0, rows_left = 0;
    for (int u = u_lo; u < u_hi;) {
        int npass = pl.passes - pass;
        if (npass > u_hi - u) npass = u_hi - u;
        if (npass > pl.stage_passes) npass = pl.stage_passes;
        const int c_lo = pass * G;
        const int c_hi = c_lo + npass * G < pl.C ? c_lo + npass * G : pl.C;
        if (fresh) {
            fresh = false;
            y0 = rw.y_lo + band_row<D, PH>(grp);
            const bool active = owner && y0 < pl.OH;
            rows_left = active ? (pl.OH - y0 + D - 1) / D : 0;  // pixels of this thread inside the plane (or more)
#pragma unroll
            for (int r = 0; r < NR; ++r) {
                const int iy = y0 * S + D * (r - R);
                rowoff[r] = (active && iy >= 0 && iy < pl.H)
                                ? (uint32_t)pip * (uint32_t)plane_bytes + (uint32_t)(((iy - rw.iy_lo) * pl.W + x * S) * ES)
                                : pl.zero_off + 16u;
            }
            // Loads from clamped addresses and values dropped after: a load behind a branch would wait for
            // the one before.
            const T* sfb = reinterpret_cast<const T*>(pl.sf) + (long long)rw.b * KK * out_plane;
            float sum_abs = 0.f;
#pragma unroll
            for (int q = 0; q < HP; ++q) {
                float v[2][KK];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int p = q + h * HP;
                    if (!pl.bwdx) {
                        const bool ok = p < rows_left;
                        const T* at = ok ? sfb + (y0 + D * p) * pl.OW + x : sfb;
#pragma unroll
                        for (int t = 0; t < KK; ++t) v[h][t] = Elem<T>::load(at + t * out_plane);
                        if (!ok) {
#pragma unroll
                            for (int t = 0; t < KK; ++t) v[h][t] = 0.f;
                        }
                    } else {
#pragma unroll
                        for (int i = 0; i < K; ++i) {
                            const int yy = y0 + D * (p + i - R);
                            const bool row = p < rows_left && yy >= 0 && yy < pl.OH;
                            const T* at = row ? sfb + (KK - 1 - i * K) * out_plane + yy * pl.OW + x : sfb;
#pragma unroll
                            for (int j = 0; j < K; ++j) {
                                const bool ok = row && x + D * (j - R) >= 0 && x + D * (j - R) < pl.OW;
                                const float w = Elem<T>::load(ok ? at + (D * (j - R) - j * out_plane) : sfb);
                                v[h][i * K + j] = ok ? w : 0.f;
                            }
                        }
                    }
                }
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    if (pl.norm) {
                        float sum = 0.f;
#pragma unroll
                        for (int t = 0; t < KK; ++t) sum += v[h][t];
                        const float mean = sum / (float)KK;
                        float var = 0.f;
#pragma unroll
                        for (int t = 0; t < KK; ++t) {
                            v[h][t] -= mean;
                            var = fmaf(v[h][t], v[h][t], var);
                        }
                        const float inv = pl.sf_scale / (sqrtf(var / (float)(KK - 1)) + 1e-10f);
#pragma unroll
                        for (int t = 0; t < KK; ++t) v[h][t] *= inv;
                    }
#pragma unroll
                    for (int t = 0; t < KK; ++t) sum_abs += fabsf(v[h][t]);
                }
#pragma unroll
                for (int t = 0; t < KK; ++t) sf2[(t % K) * K + t / K][q] = f2_pack(v[0][t], v[1][t]);
            }
            big_sf = !(sum_abs < kBandFilterMax);
        }
        // Channel filters of the next units as (c, c) pairs, one column of taps after the other; grad-x
        // pairs window tap (i, j) with the mirrored filter tap.
        int big = big_sf;
        if (u != u_lo) band_sync(NW * 32);  // every warp is done with the filters staged before
        {
            const T* cfp = reinterpret_cast<const T*>(pl.cf) + ((long long)rw.b * pl.C + c_lo) * KK;
            const int n = (c_hi - c_lo) * KK;
            for (int e = tid; e < n; e += NW * 32) {
                const int c = e / KK, t = e - c * KK;
                const int w = pl.bwdx ? KK - 1 - t : t;
                const float v = Elem<T>::load(cfp + e);
                big |= !(fabsf(v) < kBandFilterMax);
                const uint32_t bits = __float_as_uint(v);
                sts64(sbase + pl.off_cf + (uint32_t)c * CFB + (uint32_t)((w % K) * CFC + 8 * (w / K)), bits, bits);
            }
        }
        const bool plain = band_sync_or(NW * 32, big);

        T* outp = reinterpret_cast<T*>(pl.out) + ((long long)rw.b * pl.C + c_lo + pip) * out_plane +
                  (long long)y0 * pl.OW + x;
        uint32_t g_lo = (uint32_t)run_start(rw, c_lo);
        uint32_t cf_s = sbase + pl.off_cf + (uint32_t)pip * CFB;
        int left = c_hi - c_lo - pip;  // > 0 while this thread's plane of the unit exists
        for (int i = 0; i < npass; ++i) {
            if (++slot == NST) slot = 0;
            if (slot == 0) ph ^= 1u;
            if (ph < kBandDead && !mbar_wait_for(BAND_FULL(slot), ph, pl.wait_cycles)) {
                atomicCAS(pl.fault, 0, (int)kFaultConsumerFull);
                ph |= kBandDead;
            }
            const uint32_t base = BAND_DATA(slot) + (g_lo & 15u);
            unsigned long long acc2[HP];
#pragma unroll
            for (int q = 0; q < HP; ++q) acc2[q] = 0ull;
            if (!plain) {
                uint32_t row[NR];
#pragma unroll
                for (int r = 0; r < NR; ++r) row[r] = base + rowoff[r];
#pragma unroll
                for (int j = 0; j < K; ++j) {
                    unsigned long long cp[(K + 1) / 2 * 2];
#pragma unroll
                    for (int t = 0; t < (K + 1) / 2; ++t)
                        lds128_pairs(cf_s + (uint32_t)(j * CFC + 16 * t), cp[2 * t], cp[2 * t + 1]);
                    float v[NR];
#pragma unroll
                    for (int r = 0; r < NR; ++r)
                        v[r] = j == R ? Masked<T>::load(row[r])
                                      : Masked<T>::load(row[r] + (uint32_t)((D * (j - R)) * ES), cmask[j]);
#pragma unroll
                    for (int k = 0; k < K; ++k) {
#pragma unroll
                        for (int q = 0; q < HP; ++q) {
                            const unsigned long long w2 = MODE == DDF_B200_MUL ? f2_mul(cp[k], sf2[j * K + k][q])
                                                                               : f2_add(cp[k], sf2[j * K + k][q]);
                            acc2[q] = f2_fma(w2, f2_pack(v[S * q + k], v[S * (q + HP) + k]), acc2[q]);
                        }
                    }
                }
            } else {
                // taps outside the plane are skipped, not multiplied by zero
                auto tap = [&](int iy, int ix, float cv, float sv, float a) {
                    if (iy < 0 || iy >= pl.H || ix < 0 || ix >= pl.W) return a;
                    const uint32_t at = base + (uint32_t)pip * (uint32_t)plane_bytes +
                                        (uint32_t)(((iy - rw.iy_lo) * pl.W + ix) * ES);
                    return fmaf(combine_w<MODE, float>(cv, sv), Masked<T>::load(at), a);
                };
#pragma unroll
                for (int q = 0; q < HP; ++q) {
                    float a0 = 0.f, a1 = 0.f;
#pragma unroll
                    for (int t = 0; t < KK; ++t) {  // t = column-major tap
                        float s0, s1;
                        f2_unpack(sf2[t][q], s0, s1);
                        const float cv = ldsf(cf_s + (uint32_t)((t / K) * CFC + 8 * (t % K)));
                        const int ix = x * S + D * (t / K - R), iy = y0 * S + D * (t % K - R);
                        if (q < rows_left) a0 = tap(iy + q * S * D, ix, cv, s0, a0);
                        if (q + HP < rows_left) a1 = tap(iy + (q + HP) * S * D, ix, cv, s1, a1);
                    }
                    acc2[q] = f2_pack(a0, a1);
                }
            }
            // the slot is handed back before the stores: nothing below reads it
            __syncwarp();
            if (lane == 0 && ph < kBandDead) mbar_arrive(BAND_EMPTY(slot));
            if (left > 0 && ph < kBandDead) {
                T* o = outp;
                float res[PH];
#pragma unroll
                for (int q = 0; q < HP; ++q) f2_unpack(acc2[q], res[q], res[q + HP]);
#pragma unroll
                for (int p = 0; p < PH; ++p) {
                    if (p < rows_left) Elem<T>::store(o, res[p]);
                    o += row_step;
                }
            }
            outp += G * out_plane;
            cf_s += (uint32_t)G * CFB;
            g_lo += g_step;
            left -= G;
        }
        u += npass;
        pass += npass;
        if (pass == pl.passes) {
            pass = 0;
            rw = rows_of(++seg);
            fresh = true;
        }
    }
#undef BAND_FULL
#undef BAND_EMPTY
#undef BAND_DATA
}

// ------------------------------------------------------------------------ host side
struct BandArgs {
    const void* in;
    const void* cf;
    const void* sf;
    void* out;
    Problem p;
    bool bwdx;
    int sm_count;
    int* fault;
    int device;
    long long wait_cycles = kWaitCycles;
    uint32_t tx_skew = 0;
};

// Bands of a problem; shared with the filter-gradient form.
struct BandSplit {
    int groups, bands, planes, warps;
};

// `whole_warps`: a plane's positions are padded to whole warps.
inline bool band_split(int B, int C, int OH, int OW, int D, int PH, int max_threads, bool whole_warps, BandSplit& s) {
    const int max_pos = max_threads - 32;  // one warp is the producer
    if (OW < 1 || OW > max_pos) return false;
    const int step = OW > max_pos / D ? 1 : D;
    const int total = (OH + PH * D - 1) / (PH * D) * D;  // column groups of a plane
    // Groups per band: the fewest warps over all bands (a short last band and a half-empty last warp
    // both cost whole warps), the bigger band where equal.
    int best = step;
    long long best_cost = -1;
    for (int n = step; n * OW <= max_pos && n <= total; n += D) {
        if (n * OW > 288 && n > step) break;  // two or three CTAs per SM hide one another's start
        const int bands = (total + n - 1) / n;
        const long long cost = (long long)bands * ((n * OW + 31) / 32);
        if (best_cost < 0 || cost <= best_cost) { best = n; best_cost = cost; }
    }
    s.groups = best;
    s.bands = (total + best - 1) / best;
    s.planes = 1;
    if (s.bands == 1) {
        s.planes = 256 / (whole_warps ? (best * OW + 31) / 32 * 32 : best * OW);
        if (s.planes < 1) s.planes = 1;
        if (s.planes > C) s.planes = C;
    }
    s.warps = whole_warps ? s.planes * ((best * OW + 31) / 32) : (s.planes * best * OW + 31) / 32;
    return (long long)B * s.bands * C <= (1ll << 40);
}

// Slot layout for runs of up to `run` bytes: [guard | data + 16 | zeros], ring depth within `budget`.
inline int band_slots(uint32_t run, uint32_t off_slot0, uint32_t budget, uint32_t& zero_off, uint32_t& stride) {
    zero_off = round_up(run + 16u + 32u, 16);
    stride = round_up(kBandGuard + zero_off + kBandZero, 128);
    for (int n = kBandSlots; n >= 2; --n)
        if (off_slot0 + (uint32_t)n * stride <= budget) return n;
    return 0;
}

template <typename T, int K, int D, int S, int PH, int MODE>
int band_launch(const BandArgs& a, cudaStream_t stream) {
    const Problem& p = a.p;
    constexpr int ES = (int)sizeof(T), R = (K - 1) / 2;
    if ((reinterpret_cast<uintptr_t>(a.in) & 15u) != 0) return kNotHandled;
    if (a.bwdx && p.sf_norm) return kNotHandled;
    BandPlan pl;
    pl.in = a.in; pl.cf = a.cf; pl.sf = a.sf; pl.out = a.out;
    pl.C = p.C;
    pl.OH = p.OH; pl.OW = p.OW;
    pl.H = a.bwdx ? p.OH : p.H;
    pl.W = a.bwdx ? p.OW : p.W;
    BandSplit sp;
    if (!band_split(p.B, p.C, p.OH, p.OW, D, PH, kBandThreads<K>, false, sp)) return kNotHandled;
    pl.bands = sp.bands; pl.groups = sp.groups; pl.planes = sp.planes; pl.n_warps = sp.warps;
    pl.passes = (p.C + sp.planes - 1) / sp.planes;
    const long long units = (long long)p.B * sp.bands * pl.passes;
    if (units > (1ll << 30)) return kNotHandled;
    pl.units = (int)units;
    pl.stage_passes = kBandStage / sp.planes > 1 ? kBandStage / sp.planes : 1;
    if (pl.stage_passes > pl.passes) pl.stage_passes = pl.passes;
    pl.bwdx = a.bwdx; pl.norm = p.sf_norm; pl.sf_scale = (float)p.sf_scale;
    pl.in_total = (unsigned long long)p.B * p.C * pl.H * pl.W * ES;
    pl.fault = a.fault; pl.wait_cycles = a.wait_cycles; pl.tx_skew = a.tx_skew;
    const long long plane_bytes = (long long)pl.H * pl.W * ES;
    const long long rows = (long long)(band_rows<D, PH>(sp.groups) - 1) * S + 2 * R * D + 1;
    const long long run = (sp.planes - 1) * plane_bytes + (rows < pl.H ? rows : pl.H) * (long long)pl.W * ES;
    if (run > (100 << 10)) return kNotHandled;
    pl.off_cf = round_up(16u * kBandSlots, 128);
    pl.off_slot0 = round_up(pl.off_cf + (uint32_t)(pl.stage_passes * sp.planes) * kBandCf<K>, 128);
    // as many CTAs per SM as the registers allow, each with at least three slots
    const int threads = (sp.warps + 1) * 32;
    int ctas = 65536 / (kBandRegs<K> * threads);
    if (ctas > 4) ctas = 4;
    for (;; --ctas) {
        if (ctas < 1) return kNotHandled;
        const uint32_t budget = ctas == 1 ? kSmemBudget : (227u << 10) / (uint32_t)ctas - 1024u;
        pl.n_slots = band_slots((uint32_t)run, pl.off_slot0, budget, pl.zero_off, pl.slot_stride);
        if (pl.n_slots >= 3 || (ctas == 1 && pl.n_slots == 2)) break;
    }
    const long long most = (long long)ctas * a.sm_count;
    const long long grid = units < most ? units : most;
    const uint32_t smem = pl.off_slot0 + (uint32_t)pl.n_slots * pl.slot_stride;
    auto kern = band_kernel<T, K, D, S, PH, MODE>;
    static std::atomic<unsigned long long> opted_in{0};
    const unsigned long long bit = 1ull << (a.device & 63);
    if (!(opted_in.load(std::memory_order_acquire) & bit)) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBudget);
        if (e != cudaSuccess) return (int)e;
        opted_in.fetch_or(bit, std::memory_order_release);
    }
    return (int)launch_overlapped(kern, dim3((unsigned)grid), dim3((unsigned)threads), smem, stream, true, pl);
}

// Defined once per element type in band_inst_<type>.cu.
template <typename T>
int band_dispatch(const BandArgs& a, cudaStream_t stream);

}  // namespace ddf
