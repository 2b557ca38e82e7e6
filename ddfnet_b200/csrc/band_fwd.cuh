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
// A thread owns four output pixels of one column, D rows apart (so neighbouring windows share rows at
// every dilation).  Lanes of a warp own neighbouring columns: every shared load is conflict-free and
// every store coalesced at any width and alignment, which vectors along x would not be.
//
// The filters of a thread's pixels when a band begins, in one of two ways.  Straight into the thread's registers (DIRECT),
// every load in flight at once: the forward but for 2-byte mul at k = 3, and at k = 5 but for the two rules of band_launch.
// Or by one thread per position to shared memory, laid out for its own later loads; k = 3 takes them into registers from
// there, k = 5 a column of taps at a time, for two channels, at 96 registers a thread and not 168.  That way costs up to
// 3 us at the start: us, forward, by way of shared memory alone -> as it is (and before there was that way):
// (2,16,46x70) f32 k = 5 8.6 -> 5.4 (5.7), (3,24,56x56) bf16 add 5.7 -> 4.3 (4.8), (1,300,60x60) f32 9.0 -> 7.2 (8.2),
// (2,64,29x31) f32 5.4 -> 3.7 (4.1), (7,96,48x29) f32 k = 5 add 17.5 -> 11.1 (13.6).
//
// Arithmetic.  2-byte types, mul: x * sf exact by the mixed-precision FMA from the 2-byte operands, then a float FMA
// with cf (two-wide FMAs there wait for the pipe: 42.3 against 39.7 us at (2,128,200x280) bf16).  Float, add, and
// filters normalised here: w = cf * sf (or cf + sf) and x * w, two pixels (p, p + 2) an instruction.
//
// What bounds it: instruction issue (38 instructions per output at k = 3 float32, 52 of which 18 are FMAs at 2-byte mul; at 300
// columns half of the issue slots and two thirds of them are busy), and the latency of the few warps that fit.  Half
// of what it issued before were products and selects that the compiler formed again in each pass (see pin); stores
// under a predicate instead of a branch took another eighth.  Not all that is pinned stays in registers: -Xptxas -v shows
// up to 132 bytes a thread spilled with MIX, 192 in grad-x and the normalised k = 5 without, 128 in the DIRECT forms (0 to 20 at
// k = 3, stride 1).  us, forward / grad-x, before (a CTA of 80 to 168 registers a thread for both) -> now:
// (2,256,200x300) f32 80.7 / 84.4 -> 67.6 / 79.0 and bf16 85.0 / 89.7 -> 69.5 / 69.7, (4,128,50x67) f16 11.4 / 15.0 ->
// 10.5 / 11.9, (8,48,150x130) f16 add 26.1 / 30.7 -> 21.5 / 25.8, k = 5 (8,96,75x101) f16 50.4 / 55.1 -> 35.6 / 38.3, f32
// 48.0 / 52.6 -> 37.8 / 42.6, and (128,64,56x56) bf16 178 / 191 -> 138 / 139; (1,300,60x60) f32 8.2 / 11.3 -> 7.2 / 9.5.
// float32 at more than 288 columns is one CTA of ten compute warps an SM (96 registers), and the faster one all the same.
// Not kept: four channels a unit (the same or slower), the filters of k = 3 out of shared memory in every pass.
//
// Zero padding.  Rows outside the plane are read from a zeroed spot of the slot (their offset is a
// per-thread constant), columns outside are masked.  A zero times an infinite filter value would be
// NaN where the definition skips the tap: while the filters hold anything not below kBandFilterMax
// in magnitude (so that cf * sf is finite too) a CTA takes a plain loop that skips those taps.  A thread takes it too
// where x * sf may have left float's range although x * (cf * sf) does not (bfloat16 alone): where a result is not
// finite, and, while a channel filter holds a value of kLargeCf or more, where one is below kBandSmall (x * sf below
// 2^-126 is rounded, an error of up to 2^-150 |cf| a tap, which for results below 2^-60 may be more than 2^-24 of them).
//
// Every mbarrier wait is bounded by the plan's wait_cycles.  A thread whose wait ran out records a fault,
// stays for the barriers of the others, and neither stores nor hands slots back: the producer's own wait
// then runs out and it issues no more.  The producer leaves, always, after the last copies have landed.
#pragma once

#include <atomic>
#include <type_traits>

#include "common.cuh"
#include "ring_fwd.cuh"
#include "stream_fwd.cuh"

namespace ddf {

constexpr int kBandSlots = 8;
constexpr int kBandStage = 64;       // channels whose filters are staged together
constexpr float kBandFilterMax = 1e18f;
constexpr float kBandSmall = 8.6736173798840355e-19f;   // 2^-60
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
    uint32_t off_cf, off_sf, off_slot0, slot_stride;
    uint32_t part_stride, zero_off;  // a slot's channel parts, and from a part's data to its zeros
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
    template <int OFF> static __device__ __forceinline__ float at(uint32_t a) { return __uint_as_float(lds32i<OFF>(a)); }
    template <int OFF> static __device__ __forceinline__ float at(uint32_t a, uint32_t m) { return __uint_as_float(lds32i<OFF>(a) & m); }
    static __device__ __forceinline__ float load(uint32_t a) { return ldsf(a); }
};
template <> struct Masked<__nv_bfloat16> {
    static __device__ __forceinline__ uint32_t mask(bool ok) { return ok ? 0x1044u : 0x4444u; }
    static __device__ __forceinline__ float load(uint32_t a, uint32_t m) {
        return __uint_as_float(__byte_perm(lds16(a), 0u, m));
    }
    static __device__ __forceinline__ float load(uint32_t a) { return __uint_as_float(lds16(a) << 16); }
    template <int OFF> static __device__ __forceinline__ float at(uint32_t a) { return __uint_as_float(lds16i<OFF>(a) << 16); }
    template <int OFF> static __device__ __forceinline__ float at(uint32_t a, uint32_t m) {
        return __uint_as_float(__byte_perm(lds16i<OFF>(a), 0u, m));
    }
};
template <> struct Masked<__half> {
    static __device__ __forceinline__ uint32_t mask(bool ok) { return ok ? 0xffffffffu : 0u; }
    static __device__ __forceinline__ float load(uint32_t a, uint32_t m) { return Word<__half>::get(lds16(a) & m, 0); }
    static __device__ __forceinline__ float load(uint32_t a) { return Word<__half>::get(lds16(a), 0); }
    template <int OFF> static __device__ __forceinline__ float at(uint32_t a) { return Word<__half>::get(lds16i<OFF>(a), 0); }
    template <int OFF> static __device__ __forceinline__ float at(uint32_t a, uint32_t m) { return Word<__half>::get(lds16i<OFF>(a) & m, 0); }
};

// An element's bits as they are loaded, and as a float's.
template <typename T> struct Raw {
    static __device__ __forceinline__ uint32_t load(const T* p) { return __ldg(reinterpret_cast<const uint16_t*>(p)); }
    static __device__ __forceinline__ uint32_t f32_bits(uint32_t v) { return Mix<T>::f32_bits(v); }
};
template <> struct Raw<float> {
    static __device__ __forceinline__ uint32_t load(const float* p) { return __float_as_uint(__ldg(p)); }
    static __device__ __forceinline__ uint32_t f32_bits(uint32_t v) { return v; }
};

// Bytes of a channel's filter in shared memory: (c, c) pairs column by column, each column padded to
// whole 16 bytes; SINGLE: plain floats.
template <int K, bool SINGLE = false> constexpr int kBandCf = K * (SINGLE ? (K + 3) / 4 * 16 : (K + 1) / 2 * 16);

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

template <int K> constexpr int kBandThreads = K == 3 ? 352 : 384;
constexpr int kBandPixels = 4;  // rows a thread owns in its column
// Registers of a thread: 24 warps of an SM, or 20 where 36 filter values (k = 3, float) or two channels' rows of a
// 5 x 5 window are held, or 12 where 100 filter values are (whole CTAs of them: one of 11 warps at 300 columns).
template <int K, bool MIX, bool DIRECT = false> constexpr int kBandRegs = K == 5 && DIRECT ? 168 : K == 3 && MIX ? 80 : 96;

// Stores v where pixel P is one of the first n; a predicate and no branch.
template <int P>
__device__ __forceinline__ void store_below(float* at, float v, int n) {
    asm volatile("{\n\t.reg .pred q;\n\tsetp.gt.s32 q, %2, %3;\n\t@q st.global.b32 [%0], %1;\n\t}" ::"l"(at), "f"(v), "r"(n), "n"(P) : "memory");
}
template <int P, typename T>
__device__ __forceinline__ void store_below(T* at, float v, int n) {
    const uint32_t h = Word<T>::put(v, 0.f);
    asm volatile("{\n\t.reg .pred q;\n\t.reg .b16 l, u;\n\tmov.b32 {l, u}, %1;\n\tsetp.gt.s32 q, %2, %3;\n\t@q st.global.b16 [%0], l;\n\t}"
                 ::"l"(at), "r"(h), "r"(n), "n"(P) : "memory");
}

// Output row of a thread's first pixel.  Groups count in blocks of D: group g of a band covers rows
// (g / D) * PH * D + g % D, + D, + 2D ...
template <int D, int PH>
__device__ __forceinline__ int band_row(int group) { return D == 1 ? group * PH : (group / D) * (PH * D) + group % D; }

// Output rows from a band's first to its last.  Bands hold whole blocks of D groups, or, where the D groups
// of a wide plane would need more threads than a CTA has, one group.
template <int D, int PH>
__host__ __device__ __forceinline__ int band_rows(int groups) { return groups % D == 0 ? groups * PH : D * (PH - 1) + 1; }

// One column of taps of one channel: its window values, then the taps of the four pixels.  s: the column's filters,
// pixel halves (p0, p1) (p2, p3) or float pairs (p0, p2) (p1, p3).
template <int J, typename T, int K, int D, int S, bool MUL, bool MIX, int NR, typename SF, typename A>
__device__ __forceinline__ void band_column(const uint32_t (&row)[NR], uint32_t cmask, uint32_t ca, const SF (*s)[2], A& acc) {
    constexpr int R = (K - 1) / 2, CFC = kBandCf<K, MIX> / K, DX = D * (J - R) * (int)sizeof(T);
    if constexpr (MIX) {
        uint32_t c[(K + 3) / 4 * 4];
        lds128i<J * CFC>(ca, c[0], c[1], c[2], c[3]);
        if constexpr (K > 4) c[4] = lds32i<J * CFC + 16>(ca);
        uint32_t v[NR];
#pragma unroll
        for (int r = 0; r < NR; ++r) v[r] = J == R ? lds16i<DX>(row[r]) : lds16i<DX>(row[r]) & cmask;
#pragma unroll
        for (int k = 0; k < K; ++k) {
#pragma unroll
            for (int p = 0; p < kBandPixels; ++p)
                acc[p] = fmaf(Mix<T>::fmaw(0, p & 1, v[S * p + k], s[k][p / 2], 0.f), __uint_as_float(c[k]), acc[p]);
        }
    } else {
        unsigned long long cp[(K + 1) / 2 * 2];
        lds128i_pairs<J * CFC>(ca, cp[0], cp[1]);
        lds128i_pairs<J * CFC + 16>(ca, cp[2], cp[3]);
        if constexpr (K > 4) lds128i_pairs<J * CFC + 32>(ca, cp[4], cp[5]);
        float v[NR];
#pragma unroll
        for (int r = 0; r < NR; ++r) v[r] = J == R ? Masked<T>::template at<DX>(row[r]) : Masked<T>::template at<DX>(row[r], cmask);
#pragma unroll
        for (int k = 0; k < K; ++k) {
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const unsigned long long w2 = MUL ? f2_mul(cp[k], s[k][q]) : f2_add(cp[k], s[k][q]);
                acc[q] = f2_fma(w2, f2_pack(v[S * q + k], v[S * (q + 2) + k]), acc[q]);
            }
        }
    }
}
// All columns of one channel, the filters in registers.
template <int J, typename T, int K, int D, int S, bool MUL, bool MIX, int NR, typename SF, typename A>
__device__ __forceinline__ void band_columns(const uint32_t (&row)[NR], const uint32_t (&cmask)[K], uint32_t ca, const SF (*s)[2], A& acc) {
    if constexpr (J < K) {
        band_column<J, T, K, D, S, MUL, MIX>(row, cmask[J], ca, s + J * K, acc);
        band_columns<J + 1, T, K, D, S, MUL, MIX>(row, cmask, ca, s, acc);
    }
}
// All columns of CH channels, the filters of a column at a time out of shared memory.
template <int J, typename T, int K, int D, int S, bool MUL, bool MIX, int CH, int NR, typename A>
__device__ __forceinline__ void band_columns_shared(const uint32_t (&row)[CH][NR], const uint32_t (&cmask)[K], uint32_t ca,
                                                    uint32_t sf_s, uint32_t sf_tap, A (&acc)[CH]) {
    if constexpr (J < K) {
        std::conditional_t<MIX, uint32_t, unsigned long long> s[K][2];
#pragma unroll
        for (int k = 0; k < K; ++k) {
            if constexpr (MIX) lds64(sf_s, s[k][0], s[k][1]);
            else lds128_pairs(sf_s, s[k][0], s[k][1]);
            sf_s += sf_tap;
        }
#pragma unroll
        for (int ch = 0; ch < CH; ++ch)
            band_column<J, T, K, D, S, MUL, MIX>(row[ch], cmask[J], ca + (uint32_t)(ch * kBandCf<K, MIX>), s, acc[ch]);
        band_columns_shared<J + 1, T, K, D, S, MUL, MIX, CH>(row, cmask, ca, sf_s, sf_tap, acc);
    }
}

// MIX: 2-byte filters as they are, x * sf exact by the mixed-precision FMA; else float filters (float tensors, and
// filters normalised here).  CH: channels a thread has of a unit.  DIRECT: the forward's filters of a thread's pixels come into
// its registers straight from global memory, at k = 5 as they are (1) or normalised here (2: code for both in one kernel
// takes (2,64,200x300) k = 5 add from 39 to 44 us).
template <typename T, int K, int D, int S, int MODE, bool MIX, int CH, int DIRECT>
__global__ void __maxnreg__((kBandRegs<K, MIX, DIRECT != 0>))
band_kernel(const __grid_constant__ BandPlan pl) {
    constexpr int KK = K * K, R = (K - 1) / 2, ES = (int)sizeof(T);
    constexpr int PH = kBandPixels, NR = S * (PH - 1) + K;   // window rows of a thread, D input rows apart
    constexpr bool MUL = MODE == DDF_B200_MUL;
    constexpr int CFB = kBandCf<K, MIX>;
    constexpr int CFC = CFB / K;              // bytes of one tap column
    constexpr uint32_t SFB = PH * (MIX ? 2 : 4);   // bytes of a tap of a thread's pixels
    constexpr bool REG = K == 3 || DIRECT;    // the filters of a thread's pixels stay in registers
    constexpr bool NORM = DIRECT && !MIX && (K == 3 || DIRECT == 2);
    static_assert(D == 1 || S == 1, "dilated windows are built at stride 1");
    static_assert(!MIX || (ES == 2 && MUL), "mixed-precision products take 2-byte factors; w = cf + sf is float");

    extern __shared__ __align__(128) unsigned char smem_raw[];
    const uint32_t sbase = smem_u32(smem_raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int NST = pl.n_slots, NW = pl.n_warps, G = pl.planes;
#define BAND_FULL(s) (sbase + 8u * (uint32_t)(s))
#define BAND_EMPTY(s) (sbase + 8u * (uint32_t)(kBandSlots + (s)))
#define BAND_DATA(s) (sbase + pl.off_slot0 + (uint32_t)(s) * pl.slot_stride + kBandGuard)

    if (tid == 0) {
        for (int s = 0; s < NST; ++s) {
            mbar_init(BAND_FULL(s), CH);
            mbar_init(BAND_EMPTY(s), (uint32_t)NW);
        }
        mbar_fence_init();
    }
    for (int e = tid; e < NST * CH * (int)(kBandZero / 4); e += blockDim.x) {
        const int s = e / (int)(kBandZero / 4);
        sts32(BAND_DATA(s / CH) + (uint32_t)(s % CH) * pl.part_stride + pl.zero_off + 4u * (uint32_t)(e - s * (int)(kBandZero / 4)), 0u);
    }
    __syncthreads();
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");

    const int u_lo = (int)(((unsigned long long)pl.units * blockIdx.x) / gridDim.x);
    const int u_hi = (int)(((unsigned long long)pl.units * (blockIdx.x + 1)) / gridDim.x);
    const unsigned long long plane_bytes = (unsigned long long)pl.H * pl.W * ES;
    const int GC = G * CH;   // channels of a unit: part ch holds planes [ch * G, ch * G + G) of it
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
        // ------------------------------------------------------------- producer: a lane per part
        int seg = u_lo / pl.passes;
        int pass = u_lo - seg * pl.passes;
        Rows r = rows_of(seg);
        const int n = u_hi - u_lo;
        int issued = 0;
        for (; issued < n; ++issued) {
            const int slot = issued % NST;
            if (!__all_sync(0xffffffffu, band_slot_free(BAND_EMPTY(slot), issued, NST, pl.wait_cycles, pl.tx_skew))) break;
            if (lane < CH) {
                const int c = pass * GC + lane * G;
                const int count = pl.C - c < G ? pl.C - c : G;
                Span sp{0u, nullptr, 0u};
                if (count > 0) {
                    const unsigned long long g0 = run_start(r, c);
                    sp = span_prepare(BAND_DATA(slot) + (uint32_t)lane * pl.part_stride, pl.in, g0,
                                      g0 + (unsigned long long)(count - 1) * plane_bytes +
                                          (unsigned long long)(r.iy_hi - r.iy_lo) * pl.W * ES,
                                      pl.in_total);
                }
                mbar_arrive_expect_tx(BAND_FULL(slot), sp.bytes + (lane == 0 ? pl.tx_skew : 0u));
                span_issue(sp, BAND_FULL(slot));
            }
            __syncwarp();
            if (++pass == pl.passes) {
                pass = 0;
                r = rows_of(++seg);
            }
        }
        if (lane == 0) band_leave(BAND_FULL(0), issued, n, NST, pl.wait_cycles, pl.tx_skew, pl.fault);
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
        const bool ok = ix >= 0 && ix < pl.W;
        cmask[j] = MIX ? (ok ? 0xffffu : 0u) : Masked<T>::mask(ok);
        pin(cmask[j]);
    }
    const long long out_plane = (long long)pl.OH * pl.OW;
    // steps from a channel part to the next, in bytes: kept, since products of 64 bits in every pass were a sixth of
    // the instructions
    unsigned long long out_step = (unsigned long long)G * out_plane * ES;
    uint32_t in_step = (uint32_t)((unsigned long long)G * plane_bytes);   // (its remainder of 16 is all that matters)
    uint32_t row_step = (uint32_t)(D * pl.OW * ES);
    pin(out_step);
    pin(in_step);
    pin(row_step);
    const uint32_t sf_s = sbase + pl.off_sf + (uint32_t)pos * SFB;   // taps column by column, a tap of all positions after the other
    const uint32_t sf_tap = (uint32_t)npos * SFB;

    int slot = -1;
    uint32_t ph = 1, data = BAND_DATA(0) - pl.slot_stride;
    uint32_t cf_step = (uint32_t)(G * CH) * CFB;
    pin(cf_step);
    int seg = u_lo / pl.passes;
    int pass = u_lo - seg * pl.passes;
    bool fresh = true;  // the next unit starts another (sample, band)
    Rows rw = rows_of(seg);
    int big_sf = 0;     // a spatial-filter value too large for products with padding zeros (or NaN)
    uint32_t rowoff[NR];
    // the filters of this thread's pixels, [column-major tap][pair]: halves (p0, p1) (p2, p3), or floats (p0, p2) (p1, p3)
    std::conditional_t<MIX, uint32_t, unsigned long long> sfr[REG ? KK : 1][2];
    int y0 = 0, rows_left = 0;
    for (int u = u_lo; u < u_hi;) {
        int npass = pl.passes - pass;
        if (npass > u_hi - u) npass = u_hi - u;
        if (npass > pl.stage_passes) npass = pl.stage_passes;
        const int c_lo = pass * GC;
        const int c_hi = c_lo + npass * GC < pl.C ? c_lo + npass * GC : pl.C;
        if (u != u_lo) band_sync(NW * 32);  // every warp is done with the filters staged before
        const bool started = fresh;
        if (fresh) {
            fresh = false;
            y0 = rw.y_lo + band_row<D, PH>(grp);
            const bool active = owner && y0 < pl.OH;
            rows_left = active ? (pl.OH - y0 + D - 1) / D : 0;  // pixels of this thread inside the plane (or more)
#pragma unroll
            for (int r = 0; r < NR; ++r) {
                const int iy = y0 * S + D * (r - R);
                // (a row that no pixel of the thread needs may not have been copied: odd heights at stride 2)
                const bool needed = rows_left >= PH || r < S * (rows_left - 1) + K;
                rowoff[r] = (active && needed && iy >= 0 && iy < pl.H)
                                ? (uint32_t)pip * (uint32_t)plane_bytes + (uint32_t)(((iy - rw.iy_lo) * pl.W + x * S) * ES)
                                : pl.zero_off + 16u;
                pin(rowoff[r]);
            }
            pin(rows_left);
            // Spatial filters of the position's pixels, by one thread each.  Loads from clamped addresses and
            // values dropped after: a load behind a branch would wait for the one before.
            big_sf = 0;
            if constexpr (DIRECT) {
                const T* sfb = reinterpret_cast<const T*>(pl.sf) + (long long)rw.b * KK * out_plane;
                float sum_abs = 0.f;
                const T* at[PH];
#pragma unroll
                for (int p = 0; p < PH; ++p) at[p] = p < rows_left ? sfb + (y0 + D * p) * pl.OW + x : sfb;
#pragma unroll
                for (int t = 0; t < KK; ++t) {
                    uint32_t v[PH];
#pragma unroll
                    for (int p = 0; p < PH; ++p) {
                        v[p] = Raw<T>::load(at[p]);
                        at[p] += out_plane;
                        if (p >= rows_left) v[p] = 0u;
                        sum_abs += fabsf(__uint_as_float(Raw<T>::f32_bits(v[p])));
                    }
                    auto& to = sfr[(t % K) * K + t / K];
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        if constexpr (MIX) to[q] = v[2 * q] | (v[2 * q + 1] << 16);
                        else to[q] = f2_pack(__uint_as_float(Raw<T>::f32_bits(v[q])), __uint_as_float(Raw<T>::f32_bits(v[q + 2])));
                    }
                }
                if constexpr (NORM) {
                    if (K == 5 || pl.norm) {
                        sum_abs = 0.f;
#pragma unroll
                        for (int q = 0; q < 2; ++q) {
                            unsigned long long sum2 = 0ull, var2 = 0ull;
#pragma unroll
                            for (int t = 0; t < KK; ++t) sum2 = f2_add(sum2, sfr[(t % K) * K + t / K][q]);
                            float lo, hi;
                            f2_unpack(sum2, lo, hi);
                            const unsigned long long less2 = f2_pack(-(lo / (float)KK), -(hi / (float)KK));
#pragma unroll
                            for (int t = 0; t < KK; ++t) {
                                auto& v2 = sfr[(t % K) * K + t / K][q];
                                v2 = f2_add(v2, less2);
                                var2 = f2_fma(v2, v2, var2);
                            }
                            f2_unpack(var2, lo, hi);
                            const unsigned long long inv2 = f2_pack(pl.sf_scale / (sqrtf(lo / (float)(KK - 1)) + 1e-10f),
                                                                    pl.sf_scale / (sqrtf(hi / (float)(KK - 1)) + 1e-10f));
#pragma unroll
                            for (int t = 0; t < KK; ++t) {
                                auto& v2 = sfr[(t % K) * K + t / K][q];
                                v2 = f2_mul(v2, inv2);
                                f2_unpack(v2, lo, hi);
                                sum_abs += fabsf(lo) + fabsf(hi);
                            }
                        }
                    }
                }
                big_sf = !(sum_abs < kBandFilterMax);
            } else if (owner && pip == 0) {
                const T* sfb = reinterpret_cast<const T*>(pl.sf) + (long long)rw.b * KK * out_plane;
                float sum_abs = 0.f;
                // (The forward's branch stays where grad-x alone is launched, k = 3 without MIX: without it the compiler keeps
                // others of the thread's constants in registers, and (2,256,200x300) f32 takes 82.5 us, not 78.6.)
                if (!pl.bwdx) {
                    const T* at[PH];
                    bool ok[PH];
#pragma unroll
                    for (int p = 0; p < PH; ++p) {
                        ok[p] = p < rows_left;
                        at[p] = ok[p] ? sfb + (y0 + D * p) * pl.OW + x : sfb;
                    }
                    if constexpr (MIX) {
#pragma unroll
                        for (int t = 0; t < KK; ++t) {
                            uint32_t v[PH];
#pragma unroll
                            for (int p = 0; p < PH; ++p) {
                                v[p] = __ldg(reinterpret_cast<const uint16_t*>(at[p]));
                                at[p] += out_plane;
                                if (!ok[p]) v[p] = 0u;
                            }
                            const uint32_t lo = v[0] | (v[1] << 16), hi = v[2] | (v[3] << 16);
                            sum_abs += fabsf(Word<T>::get(lo, 0)) + fabsf(Word<T>::get(lo, 1)) + fabsf(Word<T>::get(hi, 0)) +
                                       fabsf(Word<T>::get(hi, 1));
                            sts64(sf_s + (uint32_t)((t % K) * K + t / K) * sf_tap, lo, hi);
                        }
                    } else {
#pragma unroll
                        for (int h = 0; h < PH; h += 2) {   // two pixels' taps at a time
                            float v[2][KK];
#pragma unroll
                            for (int e = 0; e < 2; ++e) {
#pragma unroll
                                for (int t = 0; t < KK; ++t) v[e][t] = Elem<T>::load(at[h + e] + t * (long long)out_plane);
                            }
#pragma unroll
                            for (int e = 0; e < 2; ++e) {
                                if (pl.norm) {
                                    float sum = 0.f;
#pragma unroll
                                    for (int t = 0; t < KK; ++t) sum += v[e][t];
                                    const float mean = sum / (float)KK;
                                    float var = 0.f;
#pragma unroll
                                    for (int t = 0; t < KK; ++t) {
                                        v[e][t] -= mean;
                                        var = fmaf(v[e][t], v[e][t], var);
                                    }
                                    const float inv = pl.sf_scale / (sqrtf(var / (float)(KK - 1)) + 1e-10f);
#pragma unroll
                                    for (int t = 0; t < KK; ++t) v[e][t] *= inv;
                                }
#pragma unroll
                                for (int t = 0; t < KK; ++t) {
                                    if (!ok[h + e]) v[e][t] = 0.f;
                                    sum_abs += fabsf(v[e][t]);
                                }
                            }
#pragma unroll
                            for (int t = 0; t < KK; ++t) {
                                const uint32_t to = sf_s + (uint32_t)((t % K) * K + t / K) * sf_tap + 2u * h;  // p0 p2 p1 p3
                                sts32(to, __float_as_uint(v[0][t]));
                                sts32(to + 8u, __float_as_uint(v[1][t]));
                            }
                        }
                    }
                } else {
                    // grad-x pairs a window tap with the mirrored tap's filter at the neighbour it came from
#pragma unroll
                    for (int i = 0; i < K; ++i) {
                        const T* at[PH];
                        bool row[PH];
#pragma unroll
                        for (int p = 0; p < PH; ++p) {
                            const int yy = y0 + D * (p + i - R);
                            row[p] = p < rows_left && yy >= 0 && yy < pl.OH;
                            at[p] = sfb + (KK - 1 - i * K) * (long long)out_plane + (row[p] ? yy * pl.OW + x : x);
                        }
#pragma unroll
                        for (int j = 0; j < K; ++j) {
                            const bool col = x + D * (j - R) >= 0 && x + D * (j - R) < pl.OW;
                            const int step = col ? D * (j - R) : 0;
                            uint32_t v[PH];
#pragma unroll
                            for (int p = 0; p < PH; ++p) {
                                const T* from = at[p] + (step - j * (long long)out_plane);
                                if constexpr (MIX) v[p] = __ldg(reinterpret_cast<const uint16_t*>(from));
                                else v[p] = __float_as_uint(Elem<T>::load(from));
                                if (!(row[p] && col)) v[p] = 0u;
                            }
                            const uint32_t to = sf_s + (uint32_t)(j * K + i) * sf_tap;
                            if constexpr (MIX) {
                                const uint32_t lo = v[0] | (v[1] << 16), hi = v[2] | (v[3] << 16);
                                sum_abs += fabsf(Word<T>::get(lo, 0)) + fabsf(Word<T>::get(lo, 1)) + fabsf(Word<T>::get(hi, 0)) +
                                           fabsf(Word<T>::get(hi, 1));
                                sts64(to, lo, hi);
                            } else {
                                sts128(to, v[0], v[2], v[1], v[3]);
#pragma unroll
                                for (int p = 0; p < PH; ++p) sum_abs += fabsf(__uint_as_float(v[p]));
                            }
                        }
                    }
                }
                big_sf = !(sum_abs < kBandFilterMax);
            }
        }
        // Channel filters of the next units, one column of taps after the other; grad-x pairs window tap (i, j)
        // with the mirrored filter tap.
        int big = big_sf;
        constexpr bool SMALL = MIX && std::is_same<T, __nv_bfloat16>::value;   // x * sf may lose what cf would bring back
        int large = 0;
        {
            const T* cfp = reinterpret_cast<const T*>(pl.cf) + ((long long)rw.b * pl.C + c_lo) * KK;
            const int n = (c_hi - c_lo) * KK;
            for (int e = tid; e < n; e += NW * 32) {
                const int c = e / KK, t = e - c * KK;
                const int unit = c / GC, part = (c - unit * GC) / G, plane = c - unit * GC - part * G;
                const int w = pl.bwdx ? KK - 1 - t : t;
                const float v = Elem<T>::load(cfp + e);
                big |= !(fabsf(v) < kBandFilterMax);
                if constexpr (SMALL) large |= fabsf(v) >= kLargeCf;
                const uint32_t bits = __float_as_uint(v);
                const uint32_t to = sbase + pl.off_cf + (uint32_t)((unit * G + plane) * CH + part) * CFB + (uint32_t)((w % K) * CFC);
                if constexpr (MIX) sts32(to + (uint32_t)(4 * (w / K)), bits);
                else sts64(to + (uint32_t)(8 * (w / K)), bits, bits);
            }
        }
        bool plain = band_sync_or(NW * 32, big | large);
        float usual = __int_as_float(0x7f800000);   // the sum of a thread's magnitudes below which its results stand
        if constexpr (SMALL) {
            if (plain) {   // rarely
                plain = band_sync_or(NW * 32, big);
                if (!plain) usual = 0.f;
            }
        }

        if constexpr (REG && !DIRECT) {
            if (started) {
#pragma unroll
                for (int t = 0; t < KK; ++t) {
                    const uint32_t from = sf_s + (uint32_t)t * sf_tap;
                    if constexpr (MIX) lds64v(from, sfr[t][0], sfr[t][1]);
                    else {
                        uint32_t w[4];
                        lds128v(from, w[0], w[1], w[2], w[3]);
                        sfr[t][0] = f2_pack(__uint_as_float(w[0]), __uint_as_float(w[1]));
                        sfr[t][1] = f2_pack(__uint_as_float(w[2]), __uint_as_float(w[3]));
                    }
                }
            }
        }

        char* outp = reinterpret_cast<char*>(pl.out) +
                     (((long long)rw.b * pl.C + c_lo + pip) * out_plane + (long long)y0 * pl.OW + x) * ES;
        uint32_t g_lo = (uint32_t)run_start(rw, c_lo);
        uint32_t cf_s = sbase + pl.off_cf + (uint32_t)(pip * CH) * CFB;
        int left = c_hi - c_lo - pip;  // channel ch of a unit exists for this thread: left > ch * G
        for (int i = 0; i < npass; ++i) {
            data += pl.slot_stride;
            if (++slot == NST) {
                slot = 0;
                data = BAND_DATA(0);
            }
            if (slot == 0) ph ^= 1u;
            if (ph < kBandDead && !mbar_wait_for(BAND_FULL(slot), ph, pl.wait_cycles)) {
                atomicCAS(pl.fault, 0, (int)kFaultConsumerFull);
                ph |= kBandDead;
            }
            const uint32_t alive = ph < kBandDead;
            auto base_of = [&](int ch) {
                return data + (uint32_t)ch * pl.part_stride + ((g_lo + (uint32_t)ch * in_step) & 15u);
            };
            // the results of one channel, one after the other
            auto finish = [&](int ch, const float (&res)[PH]) {
                const int n = alive && left > ch * G ? rows_left : 0;
                store_below<0>(reinterpret_cast<T*>(outp), res[0], n);
                store_below<1>(reinterpret_cast<T*>(outp + row_step), res[1], n);
                store_below<2>(reinterpret_cast<T*>(outp + 2ull * row_step), res[2], n);
                store_below<3>(reinterpret_cast<T*>(outp + 3ull * row_step), res[3], n);
                outp += out_step;
            };
            using Acc = std::conditional_t<MIX, float[PH], unsigned long long[2]>;
            auto clear = [](Acc& acc) {
#pragma unroll
                for (auto& a : acc) a = 0;
            };
            auto unpack = [](const Acc& acc, float (&res)[PH]) {
                if constexpr (MIX) {
#pragma unroll
                    for (int p = 0; p < PH; ++p) res[p] = acc[p];
                } else {
                    f2_unpack(acc[0], res[0], res[2]);
                    f2_unpack(acc[1], res[1], res[3]);
                }
            };
            // the slot is handed back before the last stores: nothing below reads it
            auto hand_back = [&] {
                __syncwarp();
                if (lane == 0 && alive) mbar_arrive(BAND_EMPTY(slot));
            };
            // one channel, tap by tap: w = cf * sf before it meets x, taps outside the plane skipped, not multiplied by zero
            auto exact = [&](int ch, float (&res)[PH]) {
                const uint32_t base = base_of(ch);
#pragma unroll
                for (int p = 0; p < PH; ++p) {
                    float a = 0.f, mean = 0.f, inv = 1.f;
                    const T* sfp = reinterpret_cast<const T*>(pl.sf) + (long long)rw.b * KK * out_plane + (y0 + p * D) * pl.OW + x;
                    if constexpr (NORM) {
                        if ((K == 5 || pl.norm) && p < rows_left) {
                            float var = 0.f;
#pragma unroll 1
                            for (int t = 0; t < KK; ++t) mean += Elem<T>::load(sfp + t * out_plane);
                            mean /= (float)KK;
#pragma unroll 1
                            for (int t = 0; t < KK; ++t) {
                                const float v = Elem<T>::load(sfp + t * out_plane) - mean;
                                var = fmaf(v, v, var);
                            }
                            inv = pl.sf_scale / (sqrtf(var / (float)(KK - 1)) + 1e-10f);
                        }
                    }
#pragma unroll 1
                    for (int t = 0; t < KK; ++t) {  // t = column-major tap
                        const int col = t / K, k = t - col * K;
                        const int ix = x * S + D * (col - R), iy = (y0 + p * D) * S + D * (k - R);
                        if (p >= rows_left || iy < 0 || iy >= pl.H || ix < 0 || ix >= pl.W) continue;
                        const uint32_t sa = sf_s + (uint32_t)t * sf_tap;
                        float sv;
                        if constexpr (DIRECT)
                            sv = (Elem<T>::load(sfp + (k * K + col) * out_plane) - mean) * inv;
                        else if constexpr (MIX) sv = Word<T>::get(lds16(sa + 2u * p), 0);
                        else sv = ldsf(sa + 4u * (uint32_t)((p & 1) * 2 + (p >> 1)));
                        const float cv = ldsf(cf_s + (uint32_t)(ch * CFB + col * CFC + (MIX ? 4 : 8) * k));
                        const uint32_t at = base + (uint32_t)pip * (uint32_t)plane_bytes +
                                            (uint32_t)(((iy - rw.iy_lo) * pl.W + ix) * ES);
                        a = fmaf(combine_w<MODE, float>(cv, sv), Masked<T>::load(at), a);
                    }
                    res[p] = a;
                }
            };
            // (2-byte values of float16 have products of three inside float's range)
            auto out_of_range = [&](const float (&res)[PH]) {
                if constexpr (!SMALL) return false;
                const float sum = fabsf(res[0]) + fabsf(res[1]) + fabsf(res[2]) + fabsf(res[3]);
                if (sum < usual) return false;
                bool again = !(sum < __int_as_float(0x7f800000));
#pragma unroll
                for (int p = 0; p < PH; ++p) again |= p < rows_left && usual == 0.f && fabsf(res[p]) < kBandSmall;
                return again;
            };
            if (plain) {
#pragma unroll 1
                for (int ch = 0; ch < CH; ++ch) {
                    float res[PH];
                    exact(ch, res);
                    if (ch == CH - 1) hand_back();
                    finish(ch, res);
                }
            } else if constexpr (REG) {
#pragma unroll
                for (int ch = 0; ch < CH; ++ch) {
                    const uint32_t base = base_of(ch);
                    uint32_t row[NR];
#pragma unroll
                    for (int r = 0; r < NR; ++r) row[r] = base + rowoff[r];
                    Acc acc;
                    clear(acc);
                    band_columns<0, T, K, D, S, MUL, MIX>(row, cmask, cf_s + (uint32_t)(ch * CFB), sfr, acc);
                    float res[PH];
                    unpack(acc, res);
                    if (left > ch * G && out_of_range(res)) exact(ch, res);  // (a missing channel holds anything)
                    if (ch == CH - 1) hand_back();
                    finish(ch, res);
                }
            } else {
                uint32_t row[CH][NR];
                Acc acc[CH];
#pragma unroll
                for (int ch = 0; ch < CH; ++ch) {
                    const uint32_t base = base_of(ch);
#pragma unroll
                    for (int r = 0; r < NR; ++r) row[ch][r] = base + rowoff[r];
                    clear(acc[ch]);
                }
                band_columns_shared<0, T, K, D, S, MUL, MIX, CH>(row, cmask, cf_s, sf_s, sf_tap, acc);
                float res[CH][PH];
#pragma unroll
                for (int ch = 0; ch < CH; ++ch) {
                    unpack(acc[ch], res[ch]);
                    if (left > ch * G && out_of_range(res[ch])) exact(ch, res[ch]);
                }
                hand_back();
#pragma unroll
                for (int ch = 0; ch < CH; ++ch) finish(ch, res[ch]);
            }
            cf_s += cf_step;
            g_lo += CH * in_step;
            left -= GC;
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

// The launch of one instantiation; kNotHandled where it does not fit.
template <typename T, int K, int D, int S, int MODE, bool MIX, int CH, int DIRECT>
int band_launch_split(const BandArgs& a, const BandSplit& sp, cudaStream_t stream) {
    const Problem& p = a.p;
    constexpr int ES = (int)sizeof(T), R = (K - 1) / 2, PH = kBandPixels;
    BandPlan pl;
    pl.in = a.in; pl.cf = a.cf; pl.sf = a.sf; pl.out = a.out;
    pl.C = p.C;
    pl.OH = p.OH; pl.OW = p.OW;
    pl.H = a.bwdx ? p.OH : p.H;
    pl.W = a.bwdx ? p.OW : p.W;
    pl.bands = sp.bands; pl.groups = sp.groups; pl.planes = sp.planes; pl.n_warps = sp.warps;
    const int per_unit = sp.planes * CH;
    pl.passes = (p.C + per_unit - 1) / per_unit;
    const long long units = (long long)p.B * sp.bands * pl.passes;
    if (units > (1ll << 30)) return kNotHandled;
    pl.units = (int)units;
    pl.bwdx = a.bwdx; pl.norm = p.sf_norm; pl.sf_scale = (float)p.sf_scale;
    pl.in_total = (unsigned long long)p.B * p.C * pl.H * pl.W * ES;
    pl.fault = a.fault; pl.wait_cycles = a.wait_cycles; pl.tx_skew = a.tx_skew;
    const long long plane_bytes = (long long)pl.H * pl.W * ES;
    const long long rows = (long long)(band_rows<D, PH>(sp.groups) - 1) * S + 2 * R * D + 1;
    const long long run = (sp.planes - 1) * plane_bytes + (rows < pl.H ? rows : pl.H) * (long long)pl.W * ES;
    if (run > (100 << 10)) return kNotHandled;
    pl.off_cf = round_up(16u * kBandSlots, 128);
    pl.zero_off = round_up((uint32_t)run + 16u + 32u, 16);
    pl.part_stride = round_up(kBandGuard + pl.zero_off + kBandZero, 128);
    pl.slot_stride = CH * pl.part_stride;
    // as many CTAs per SM as the registers allow, each with at least two slots; fewer channels' filters staged
    // together where only that makes them fit
    const int threads = (sp.warps + 1) * 32;
    int ctas = 0;
    for (int stage = kBandStage; stage >= 16 && ctas < 1; stage /= 4) {
        pl.stage_passes = stage / per_unit > 1 ? stage / per_unit : 1;
        if (pl.stage_passes > pl.passes) pl.stage_passes = pl.passes;
        pl.off_sf = round_up(pl.off_cf + (uint32_t)(pl.stage_passes * per_unit) * kBandCf<K, MIX>, 128);
        pl.off_slot0 = round_up(pl.off_sf + (DIRECT ? 0u : (uint32_t)(K * K * sp.groups * p.OW * PH * (MIX ? 2 : 4))), 128);
        const int fit = 4 * (65536 / 4 / 32 / kBandRegs<K, MIX, DIRECT != 0>) / (sp.warps + 1);  // whole warps in each quarter of an SM
        for (ctas = fit < 1 ? 1 : fit < 4 ? fit : 4; ctas >= 1; --ctas) {
            const uint32_t budget = ctas == 1 ? kSmemBudget : (227u << 10) / (uint32_t)ctas - 1024u;
            if (pl.off_slot0 >= budget) continue;
            pl.n_slots = (int)((budget - pl.off_slot0) / pl.slot_stride);
            if (pl.n_slots > kBandSlots) pl.n_slots = kBandSlots;
            if (pl.n_slots >= 2) break;
        }
    }
    if (ctas < 1) return kNotHandled;
    const long long most = (long long)ctas * a.sm_count;
    const long long grid = units < most ? units : most;
    const uint32_t smem = pl.off_slot0 + (uint32_t)pl.n_slots * pl.slot_stride;
    auto kern = band_kernel<T, K, D, S, MODE, MIX, CH, DIRECT>;
    static std::atomic<unsigned long long> opted_in{0};
    const unsigned long long bit = 1ull << (a.device & 63);
    if (!(opted_in.load(std::memory_order_acquire) & bit)) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBudget);
        if (e != cudaSuccess) return (int)e;
        opted_in.fetch_or(bit, std::memory_order_release);
    }
    return (int)launch_overlapped(kern, dim3((unsigned)grid), dim3((unsigned)threads), smem, stream, true, pl);
}

template <typename T, int K, int D, int S, int MODE, bool MIX>
int band_launch(const BandArgs& a, cudaStream_t stream) {
    const Problem& p = a.p;
    if ((reinterpret_cast<uintptr_t>(a.in) & 15u) != 0) return kNotHandled;
    if (a.bwdx && p.sf_norm) return kNotHandled;
    BandSplit sp;
    if (!band_split(p.B, p.C, p.OH, p.OW, D, kBandPixels, kBandThreads<K>, false, sp)) return kNotHandled;
    // Two channels a thread and unit share the waits and, at k = 5, the filters' way out of shared memory; one where
    // the units of two would not go evenly into the CTAs ((1,300,60x60) f32: two or three each, 9.3 us against 8.3).
    auto units = [&](int planes, int ch) { return (long long)p.B * sp.bands * ((p.C + planes * ch - 1) / (planes * ch)); };
    // Filters straight into registers, us by way of shared memory against it.  Level at 50 units of one channel per SM for
    // 2-byte mul at k = 5 ((8,96,75x101) f16 35.5 / 35.8; (1,135,135x162) f16 25.0 / 23.3, (128,64,56x56) bf16 138 / 152),
    // whose filters take half the shared memory; at three for normalised ones at k = 5 ((8,61,24x37) f16 11.9 / 12.6,
    // (2,40,40x45) bf16 add 9.3 / 7.3); the faster way at every size without MIX (k = 5 (2,64,200x300) bf16 add 46.7 / 39.0,
    // (2,16,46x70) f32 8.6 / 5.4; k = 3 (2,256,200x300) f32 76.6 / 67.6, normalised 77.5 / 69.4).
    const bool direct = !a.bwdx && (K == 3 ? !MIX : MIX ? units(sp.planes, 1) < 50ll * a.sm_count
                                                         : !p.sf_norm || units(sp.planes, 1) < 3ll * a.sm_count);
    // fewer planes together while there are SMs without a unit
    while ((K == 3 || direct) && sp.planes > 1 && units(sp.planes, 1) < a.sm_count) sp.planes = (sp.planes + 1) / 2;
    sp.warps = (sp.planes * sp.groups * p.OW + 31) / 32;
    if constexpr (K == 5) {
        if (direct) {
            if constexpr (!MIX)
                if (p.sf_norm) return band_launch_split<T, K, D, S, MODE, MIX, 1, 2>(a, sp, stream);
            return band_launch_split<T, K, D, S, MODE, MIX, 1, 1>(a, sp, stream);
        }
        return band_launch_split<T, K, D, S, MODE, MIX, 2, 0>(a, sp, stream);
    } else {
        const bool one = units(sp.planes, 2) < 6ll * a.sm_count;
        if constexpr (!MIX)
            if (direct)
                return one ? band_launch_split<T, K, D, S, MODE, MIX, 1, 1>(a, sp, stream)
                           : band_launch_split<T, K, D, S, MODE, MIX, 2, 1>(a, sp, stream);
        if constexpr (MIX || S == 1)
            return one ? band_launch_split<T, K, D, S, MODE, MIX, 1, 0>(a, sp, stream)
                       : band_launch_split<T, K, D, S, MODE, MIX, 2, 0>(a, sp, stream);
        return kNotHandled;
    }
}

// Defined once per element type in band_inst_<type>.cu.
template <typename T>
int band_dispatch(const BandArgs& a, cudaStream_t stream);

}  // namespace ddf
