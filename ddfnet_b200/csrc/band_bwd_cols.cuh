// Filter gradients of the 2-byte types at stride 1, a thread per tap column (see band_bwd.cuh for the sums, the bands,
// the chunks of channels and the second launch, and band_fwd.cuh for the ring).
//
// A tap's products go * x serve that tap alone, so the taps may be dealt to threads without work done twice: a
// warp has one column j of the k x k taps and 32 positions, a thread k taps of four pixels D rows apart.  It loads
// its own column of x (k + 3 values for 4 k products), holds 4 k filter values and 4 k sums instead of 4 k^2 of
// each, and where its column lies outside the plane it does nothing: there are no column masks.  go * x is exact by
// the mixed-precision FMA, without unpacking.  A band wider than a CTA's warps is shared by several CTAs.
//
// grad-cf of a channel is a sum over lanes.  A warp leaves its lanes' values of four channels in shared memory
// and adds them there, 16 bytes at a time: a third of the instructions of a butterfly of shuffles per channel.
//
// Sums of gsf are plain over up to 64 channels; the pixel form's were at k = 5 over up to 24.  Relative error against 64 bits
// over 76 problems (bands and whole planes, k = 3 and 5): gsf at most 1.0000001 times that form's, gcf the same to six digits;
// at k = 5 290 of a million elements of gsf are not rounded as the exact value is, 244 there.  Not kept: chunks of 24
// ((128,64,56x56) k = 5 384 -> 582 us), a second sum every 24 channels (4 to 12 % for a few of those elements).
//
// Bound by instruction issue: 90 a (channel, pixel) at k = 3, of which 36 are the arithmetic.  us, pixel form (band_bwd.cuh; at
// 14 and 7 columns the plane-streaming form) -> this one: (2,256,200x300) bf16 179 -> 131, (8,48,150x130) f16 add 86.7 -> 43.8,
// (16,64,99x51) d = 2 bf16 52.9 -> 38.2, (4,128,50x67) f16 23.0 -> 19.3, k = 5 (128,64,56x56) bf16 804 -> 384,
// (8,96,75x101) f16 207 -> 130, (64,512,14x14) bf16 167 -> 124, (64,512,7x7) bf16 123 -> 64.  Registers: 64 (k = 3)
// and 96 leave room for 32 and 20 warps; mul spills there, 84 and 64 bytes a thread loaded, k = 5 at 80 far more.  Not kept:
// scalar instead of two-wide sums (154 at (2,256,200x300)).
#pragma once

#include "band_bwd.cuh"

namespace ddf {

constexpr int kColsCh = 4;          // channels of a pass
constexpr int kColsPixels = 4;
constexpr int kColsChunk = 64;      // channels per CTA at most
constexpr uint32_t kColsRow = 36;   // floats of a warp's 32 values, padded: 16-byte reads of eight rows do not collide
template <int K> constexpr int kColsThreads = K == 3 ? 1024 : 640;

struct BandColsSplit : BandBwdSplit {
    int col_warps;  // warps of a plane's tap column
    int x_parts;    // CTAs that share a band's positions (each copies the whole band); `bands` counts them
};

struct BandColsPlan {
    BandBwdPlan p;           // planes: G; n_slots, offsets as there
    int col_warps, x_parts;
    uint32_t off_red, part_stride;
};

template <typename T, int K, int D, int MODE>
__global__ void __launch_bounds__(kColsThreads<K>, 1)
band_cols_kernel(const __grid_constant__ BandColsPlan cp) {
    constexpr int KK = K * K, R = (K - 1) / 2, ES = (int)sizeof(T), PH = kColsPixels, CH = kColsCh;
    constexpr int NR = PH - 1 + K;
    constexpr int CFB = kBandCf<K>, CFC = CFB / K;
    constexpr bool MUL = MODE == DDF_B200_MUL;
    constexpr int SUMS = CH * K;                       // sums over lanes of a pass
    constexpr int LPS = 32 / SUMS >= 2 ? 2 : 1;        // lanes that share one
    static_assert(ES == 2 && SUMS * LPS <= 32, "2-byte types; one lane a sum at least");

    const BandBwdPlan& pl = cp.p;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const uint32_t sbase = smem_u32(smem_raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int NST = pl.n_slots, NW = pl.n_warps, G = pl.planes, GC = G * CH;
#define BAND_FULL(s) (sbase + 8u * (uint32_t)(s))
#define BAND_EMPTY(s) (sbase + 8u * (uint32_t)(kBandSlots + (s)))
#define BAND_DATA(s) (sbase + pl.off_slot0 + (uint32_t)(s) * pl.slot_stride)

    if (tid == 0) {
        for (int s = 0; s < NST; ++s) {
            mbar_init(BAND_FULL(s), CH);
            mbar_init(BAND_EMPTY(s), (uint32_t)NW);
        }
        mbar_fence_init();
    }
    for (int e = tid; e < NST * CH * (int)(kBandZero / 4); e += blockDim.x) {
        const int s = e / (int)(kBandZero / 4);
        sts32(BAND_DATA(s / CH) + (uint32_t)(s % CH) * cp.part_stride + pl.zero_off + 4u * (uint32_t)(e - s * (int)(kBandZero / 4)), 0u);
    }
    __syncthreads();
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");

    // bands are innermost: neighbouring bands of the same planes run together and share halo rows in L2
    int item = blockIdx.x;
    const int band = item % pl.bands;   // of x_parts times the plane's bands
    item /= pl.bands;
    const int chunk_i = item % pl.chunks;
    const int bs = item / pl.chunks;  // sample within the slice
    const int b = pl.b0 + bs;
    const int c_lo = chunk_i * pl.chunk;
    const int c_hi = c_lo + pl.chunk < pl.C ? c_lo + pl.chunk : pl.C;
    const int npass = (c_hi - c_lo + GC - 1) / GC;
    const int y_lo = band_row<D, PH>(band / cp.x_parts * pl.groups);
    const int y_next = y_lo + band_rows<D, PH>(pl.groups);
    int y_hi = y_next < pl.OH ? y_next : pl.OH;
    int iy_lo = y_lo - R * D > 0 ? y_lo - R * D : 0;
    const int iy_end = y_hi + R * D;
    int iy_hi = iy_end < pl.H ? iy_end : pl.H;
    int go_row = y_lo;
    if (D > 1 && y_lo >= pl.OH) {  // the plane ends before this group: any row will do
        iy_lo = go_row = 0;
        iy_hi = y_hi = 1;
    }
    const unsigned long long xplane = (unsigned long long)pl.H * pl.W * ES;
    const unsigned long long gplane = (unsigned long long)pl.OH * pl.OW * ES;
    const unsigned long long first_plane = (unsigned long long)b * pl.C + c_lo;
    const unsigned long long x_first = first_plane * xplane + (unsigned long long)iy_lo * pl.W * ES;
    const unsigned long long go_first = first_plane * gplane + (unsigned long long)go_row * pl.OW * ES;

    if (warp == NW) {
        // ------------------------------------------------------------- producer: a lane per channel part
        int issued = 0;
        for (; issued < npass; ++issued) {
            const int slot = issued % NST;
            if (!__all_sync(0xffffffffu, band_slot_free(BAND_EMPTY(slot), issued, NST, pl.wait_cycles, pl.tx_skew))) break;
            if (lane < CH) {
                const int c = issued * GC + lane * G;
                const int left = c_hi - c_lo - c;
                Span sx{0u, nullptr, 0u}, sg{0u, nullptr, 0u};
                if (left > 0) {
                    const unsigned long long more = (unsigned long long)((left < G ? left : G) - 1);
                    const unsigned long long x0 = x_first + (unsigned long long)c * xplane;
                    const unsigned long long g0 = go_first + (unsigned long long)c * gplane;
                    const uint32_t to = BAND_DATA(slot) + (uint32_t)lane * cp.part_stride;
                    sx = span_prepare(to, pl.x, x0, x0 + more * xplane + (unsigned long long)(iy_hi - iy_lo) * pl.W * ES, pl.x_total);
                    sg = span_prepare(to + pl.go_off, pl.go, g0, g0 + more * gplane + (unsigned long long)(y_hi - go_row) * pl.OW * ES,
                                      pl.go_total);
                }
                mbar_arrive_expect_tx(BAND_FULL(slot), sx.bytes + sg.bytes + (lane == 0 ? pl.tx_skew : 0u));
                span_issue(sx, BAND_FULL(slot));
                span_issue(sg, BAND_FULL(slot));
            }
            __syncwarp();
        }
        if (lane == 0) band_leave(BAND_FULL(0), issued, npass, NST, pl.wait_cycles, pl.tx_skew, pl.fault);
        return;
    }

    // ----------------------------------------------------------------- compute warps
    const int PW = cp.col_warps;
    const int pip = warp / (K * PW);  // a warp has one plane and one tap column
    const int j = warp / PW - pip * K;
    const int pos = (band % cp.x_parts * PW + warp % PW) * 32 + lane;
    const int grp = pos / pl.OW;
    const int x = pos - grp * pl.OW;
    const int y0 = y_lo + band_row<D, PH>(grp);
    int rows_in = pos < pl.groups * pl.OW && y0 < pl.OH ? (pl.OH - y0 + D - 1) / D : 0;  // pixels inside the plane
    if (rows_in > PH) rows_in = PH;
    const int ix = x + D * (j - R);
    const int rows_left = ix >= 0 && ix < pl.W ? rows_in : 0;                            // and with this tap column

    // Rows no pixel of this thread needs, and pixels it does not have, read zeros.
    uint32_t rowoff[NR], gooff[PH];
    uint32_t rowbits = 0;
#pragma unroll
    for (int r = 0; r < NR; ++r) {
        const int iy = y0 + D * (r - R);
        const bool ok = rows_left > 0 && r < rows_left - 1 + K && iy >= 0 && iy < pl.H;
        rowbits |= ok ? 1u << r : 0u;
        rowoff[r] = ok ? (uint32_t)pip * (uint32_t)xplane + (uint32_t)(((iy - iy_lo) * pl.W + ix) * ES) : pl.zero_off + 16u;
        pin(rowoff[r]);
    }
#pragma unroll
    for (int p = 0; p < PH; ++p) {
        gooff[p] = p < rows_left ? pl.go_off + (uint32_t)pip * (uint32_t)gplane + (uint32_t)(((y0 + D * p - y_lo) * pl.OW + x) * ES)
                                 : pl.zero_off + 16u;
        pin(gooff[p]);
    }
    // products with padding zeros, or of pixels outside the plane, in this thread / warp
    const bool edge = rows_left > 0 && (rowbits != (1u << NR) - 1u || rows_left < PH);
    const bool edge_warp = __any_sync(0xffffffffu, edge);
    auto inside = [&](int k, int p) { return p < rows_left && ((rowbits >> (p + k)) & 1u) != 0u; };

    if constexpr (MUL) {
        const T* cfp = reinterpret_cast<const T*>(pl.cf) + (long long)first_plane * KK;
        const int n = (c_hi - c_lo) * KK;
        for (int e = tid; e < n; e += NW * 32) {
            const int c = e / KK, t = e - c * KK;
            const uint32_t u = __float_as_uint(Elem<T>::load(cfp + e));
            sts64(sbase + pl.off_cf + (uint32_t)c * CFB + (uint32_t)((t % K) * CFC + 8 * (t / K)), u, u);
        }
    }
    const long long opl = (long long)pl.OH * pl.OW;
    unsigned long long sf2[MUL ? K : 1][2];  // [tap row][pixel pair]
    if constexpr (MUL) {
        const T* sfb = reinterpret_cast<const T*>(pl.sf) + ((long long)b * KK + j) * opl;
        float v[K][PH];
#pragma unroll
        for (int p = 0; p < PH; ++p) {
            const T* at = p < rows_left ? sfb + (y0 + p * D) * pl.OW + x : sfb;  // a clamped address, the value dropped after
#pragma unroll
            for (int k = 0; k < K; ++k) {
                const float w = Elem<T>::load(at + k * K * opl);
                v[k][p] = p < rows_left ? w : 0.f;
            }
        }
#pragma unroll
        for (int k = 0; k < K; ++k) {
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                sf2[k][q] = f2_pack(v[k][2 * q], v[k][2 * q + 1]);
                pin(sf2[k][q]);
            }
        }
    }
    band_sync(NW * 32);

    unsigned long long gsf2[K][2];
#pragma unroll
    for (int k = 0; k < K; ++k) gsf2[k][0] = gsf2[k][1] = 0ull;

    const uint32_t red = sbase + cp.off_red + (uint32_t)warp * (SUMS * kColsRow * 4u);
    uint32_t x_lo = (uint32_t)x_first, go_lo = (uint32_t)go_first;   // modulo 16 is all that matters
    uint32_t x_step = (uint32_t)G * (uint32_t)xplane, go_step = (uint32_t)G * (uint32_t)gplane, cf_step = (uint32_t)G * CFB;
    uint32_t part_step = 4u * (uint32_t)(CH * NW * K);
    pin(x_step);
    pin(go_step);
    pin(cf_step);
    pin(part_step);
    uint32_t cf_s = sbase + pl.off_cf + (uint32_t)pip * CFB + (uint32_t)j * CFC;
    // the lane's (or two lanes') sum of a pass: where its values lie, and where it goes
    const int sum_i = LPS == 2 ? lane >> 1 : lane, half = LPS == 2 ? lane & 1 : 0;
    uint32_t from = red + 4u * ((uint32_t)sum_i * kColsRow + (uint32_t)half * 16u);
    uint32_t part_s = sbase + pl.off_part + 4u * (uint32_t)(warp * K + sum_i / K * NW * K + sum_i % K);
    pin(from);
    int left = c_hi - c_lo - pip;

    int slot = -1;
    uint32_t ph = 1;
    for (int i = 0; i < npass; ++i) {
        if (++slot == NST) slot = 0;
        if (slot == 0) ph ^= 1u;
        if (ph < kBandDead && !mbar_wait_for(BAND_FULL(slot), ph, pl.wait_cycles)) {
            atomicCAS(pl.fault, 0, (int)kFaultConsumerFull);
            ph |= kBandDead;
        }
        uint32_t data = BAND_DATA(slot);
        const uint32_t mine = red + 4u * (uint32_t)lane;
#pragma unroll
        for (int ch = 0; ch < CH; ++ch) {
            if (left > ch * G) {  // this warp's plane of the part exists
                const uint32_t xbase = data + (x_lo & 15u), gbase = data + (go_lo & 15u);
                uint32_t g[PH], v[NR];
#pragma unroll
                for (int p = 0; p < PH; ++p) g[p] = lds16(gbase + gooff[p]);
#pragma unroll
                for (int r = 0; r < NR; ++r) v[r] = lds16(xbase + rowoff[r]);
                float part[K];
#pragma unroll
                for (int k = 0; k < K; ++k) {
                    unsigned long long c2 = 0ull, prod2[2];
                    if constexpr (MUL) c2 = lds64_pair(cf_s + 8u * k);
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        prod2[q] = f2_pack(Mix<T>::fmaw(0, 0, v[2 * q + k], g[2 * q], 0.f),
                                           Mix<T>::fmaw(0, 0, v[2 * q + 1 + k], g[2 * q + 1], 0.f));
                        if constexpr (MUL) gsf2[k][q] = f2_fma(prod2[q], c2, gsf2[k][q]);
                        else gsf2[k][q] = f2_add(gsf2[k][q], prod2[q]);
                    }
                    const unsigned long long part2 = MUL ? f2_fma(prod2[1], sf2[k][1], f2_mul(prod2[0], sf2[k][0]))
                                                         : f2_add(prod2[0], prod2[1]);
                    float lo, hi;
                    f2_unpack(part2, lo, hi);
                    part[k] = lo + hi;
                    sts32(mine + 4u * (uint32_t)(ch * K + k) * kColsRow, __float_as_uint(part[k]));
                }
                if (edge_warp) {
                    // a product with padding may have met an infinity: formed again without those
                    float sum = 0.f;
#pragma unroll
                    for (int k = 0; k < K; ++k) sum += part[k];
                    if (__any_sync(0xffffffffu, edge && !(fabsf(sum) < __int_as_float(0x7f800000)))) {
#pragma unroll
                        for (int k = 0; k < K; ++k) {
                            float a = 0.f;
#pragma unroll
                            for (int p = 0; p < PH; ++p) {
                                float s = 1.f;
                                if constexpr (MUL) {
                                    float lo, hi;
                                    f2_unpack(sf2[k][p / 2], lo, hi);
                                    s = p & 1 ? hi : lo;
                                }
                                if (inside(k, p)) a = fmaf(Mix<T>::fmaw(0, 0, v[p + k], g[p], 0.f), s, a);
                            }
                            sts32(mine + 4u * (uint32_t)(ch * K + k) * kColsRow, __float_as_uint(a));
                        }
                    }
                }
            }
            data += cp.part_stride;
            cf_s += cf_step;
            x_lo += x_step;
            go_lo += go_step;
        }
        __syncwarp();
        if (lane == 0 && ph < kBandDead) mbar_arrive(BAND_EMPTY(slot));
        // the warp's sums of the pass: four interleaved sums a lane, then they
        {
            float tot = 0.f;
            if (sum_i < SUMS) {
                unsigned long long a2 = 0ull, b2 = 0ull;
#pragma unroll
                for (int v = 0; v < 8 / LPS; ++v) {
                    unsigned long long u, w;
                    lds128_pairs(from + 16u * v, u, w);
                    a2 = f2_add(a2, u);
                    b2 = f2_add(b2, w);
                }
                float lo, hi;
                f2_unpack(f2_add(a2, b2), lo, hi);
                tot = lo + hi;
            }
            if constexpr (LPS == 2) tot += __shfl_xor_sync(0xffffffffu, tot, 1);
            if (half == 0 && sum_i < SUMS)
                sts32(part_s, __float_as_uint(tot));
            __syncwarp();
        }
        part_s += part_step;
        left -= GC;
    }
    if (band_sync_or(NW * 32, ph >= kBandDead ? 1 : 0)) return;  // a fault is recorded, and there are no whole sums

    if (pl.gcf != nullptr) {  // this band's share of gcf: the warps of a plane's tap column added up
        const int n = (c_hi - c_lo) * KK;
        for (int e = tid; e < n; e += NW * 32) {
            const int c = e / KK, t = e - c * KK;
            const int part_i = c / G, plane = c - part_i * G;   // part of all passes' parts in a row
            const uint32_t src = sbase + pl.off_part + 4u * (uint32_t)((part_i * NW + (plane * K + t % K) * PW) * K + t / K);
            CompSum<float> tot;
            for (int w = 0; w < PW; ++w) tot.add(ldsf(src + 4u * (uint32_t)(w * K)));
            if (pl.part_cf != nullptr)
                pl.part_cf[(((long long)bs * pl.bands + band) * pl.C + c_lo) * KK + e] = tot.value();
            else
                Elem<T>::store(reinterpret_cast<T*>(pl.gcf) + (long long)first_plane * KK + e, tot.value());
        }
    }
    if (pl.gsf != nullptr) {
        float* ps = pl.part_sf == nullptr
                        ? nullptr
                        : reinterpret_cast<float*>(pl.part_sf) + ((long long)bs * pl.chunks + chunk_i) * KK * opl;
        T* os = reinterpret_cast<T*>(pl.gsf) + (long long)b * KK * opl;
        auto put = [&](long long o, float v) {
            if (ps != nullptr) ps[o] = v;
            else Elem<T>::store(os + o, v);
        };
        // Several planes per pass: a band is then the whole plane, and the planes' sums meet in the slots
        // (every copy has landed and been read).
        float* meet = reinterpret_cast<float*>(smem_raw + pl.off_slot0);
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const int ft = k * K + j;
            float v[PH];
            f2_unpack(gsf2[k][0], v[0], v[1]);
            f2_unpack(gsf2[k][1], v[2], v[3]);
#pragma unroll
            for (int p = 0; p < PH; ++p) {
                if (p < rows_in) {
                    const long long o = ft * opl + (long long)(y0 + p * D) * pl.OW + x;
                    const float r = inside(k, p) ? v[p] : 0.f;
                    if (G > 1) meet[pip * KK * (int)opl + (int)o] = r;
                    else put(o, r);
                }
            }
        }
        if (G > 1) {
            band_sync(NW * 32);
            const int n = KK * (int)opl;
            for (int e = tid; e < n; e += NW * 32) {
                CompSum<float> tot;
                for (int g = 0; g < G; ++g) tot.add(meet[g * n + e]);
                put(e, tot.value());
            }
        }
    }
#undef BAND_FULL
#undef BAND_EMPTY
#undef BAND_DATA
}

// ------------------------------------------------------------------------ host side
// Shared-memory layout; false: it does not fit.
struct BandColsLayout {
    uint32_t off_cf, off_red, off_part, off_slot0, zero_off, go_off, part_stride, slot_stride, smem;
    int n_slots, ctas;
};

inline bool band_cols_layout(const Problem& p, const BandColsSplit& s, BandColsLayout& l) {
    const int k = p.k, es = 2;
    const int out_rows = s.groups % p.d == 0 ? s.groups * kColsPixels : p.d * (kColsPixels - 1) + 1;
    const long long rows = (long long)(out_rows - 1) + (k - 1) * p.d + 1;
    const long long xrun = ((s.planes - 1) * (long long)p.H + (rows < p.H ? rows : p.H)) * p.W * es;
    const long long grun = ((s.planes - 1) * (long long)p.OH + (out_rows < p.OH ? out_rows : p.OH)) * p.OW * es;
    if (xrun > (32 << 10)) return false;
    const uint32_t per_unit = (uint32_t)(s.planes * kColsCh);
    const uint32_t passes = ((uint32_t)s.chunk + per_unit - 1) / per_unit;
    l.off_cf = round_up(16u * kBandSlots, 128);
    l.off_red = round_up(l.off_cf + (uint32_t)s.chunk * (k == 3 ? kBandCf<3> : kBandCf<5>), 128);
    l.off_part = l.off_red + (uint32_t)(s.warps * kColsCh * k) * kColsRow * 4u;
    l.off_slot0 = round_up(l.off_part + passes * (uint32_t)(kColsCh * s.warps * k * 4), 128);
    l.zero_off = round_up((uint32_t)xrun + 16u + 32u, 16);
    l.go_off = round_up(l.zero_off + kBandZero, 16);
    l.part_stride = round_up(l.go_off + (uint32_t)grun + 32u, 128);
    l.slot_stride = kColsCh * l.part_stride;
    const uint32_t meet = s.planes > 1 ? (uint32_t)(s.planes * k * k * p.OH * p.OW * 4) : 0u;
    const int threads = (s.warps + 1) * 32;
    const int regs = k == 3 ? 64 : 96;  // of a thread
    for (l.ctas = 65536 / (regs * threads) < 4 ? 65536 / (regs * threads) : 4; l.ctas >= 1; --l.ctas) {
        const uint32_t budget = l.ctas == 1 ? kSmemBudget : (227u << 10) / (uint32_t)l.ctas - 1024u;
        if (l.off_slot0 + meet > budget) continue;
        l.n_slots = (int)((budget - l.off_slot0) / l.slot_stride);
        const int most = (int)passes < kBandSlots ? (int)passes : kBandSlots;
        if (l.n_slots > most) l.n_slots = most;
        if (l.n_slots >= 2 || (l.n_slots == 1 && passes == 1)) {
            const uint32_t ring = (uint32_t)l.n_slots * l.slot_stride;
            l.smem = l.off_slot0 + (ring > meet ? ring : meet);
            return true;
        }
    }
    return false;
}

// The split of a problem; false: the pixel form (band_filters_kernel) takes it.
inline bool band_cols_split(const Problem& p, int sm_count, BandColsSplit& s) {
    // (stride 2: a column of x then serves a tap of every other pixel alone, and the pixel form is the faster one:
    // (16,128,100x75) bf16 34.6 us against 40.6)
    const bool built = (p.k == 3 || p.k == 5) && p.d <= 2 && p.s == 1;
    if (!built || (p.dtype != DDF_B200_F16 && p.dtype != DDF_B200_BF16)) return false;
    // warps of a tap column at most, and the number up to which bands are made larger
    const int most = ((p.k == 3 ? kColsThreads<3> : kColsThreads<5>) / 32 - 1) / p.k, wide = 3;
    const int step = p.OW > most * 32 / p.d ? 1 : p.d;
    const int total = (p.OH + kColsPixels * p.d - 1) / (kColsPixels * p.d) * p.d;  // column groups of a plane
    int best = step;
    long long best_cost = -1;
    for (int n = step; n <= total; n += p.d) {
        const int warps = (n * p.OW + 31) / 32;
        if (warps > wide && n > step) break;
        const long long cost = (long long)((total + n - 1) / n) * warps;
        if (best_cost < 0 || cost <= best_cost) { best = n; best_cost = cost; }
    }
    s.groups = best;
    s.col_warps = (best * p.OW + 31) / 32;
    s.x_parts = (s.col_warps + most - 1) / most;
    s.col_warps = (s.col_warps + s.x_parts - 1) / s.x_parts;
    s.bands = (total + best - 1) / best * s.x_parts;
    s.planes = 1;
    if (s.bands == 1) {
        s.planes = wide / s.col_warps;
        if (s.planes < 1) s.planes = 1;
        if (s.planes > p.C) s.planes = p.C;
    }
    s.warps = s.planes * p.k * s.col_warps;
    if ((long long)p.B * s.bands * p.C > (1ll << 40)) return false;
    // Channels per CTA: the count with the least (waves of CTAs) x (channels a warp walks + the start's worth), and a
    // channel's worth for each set of partials ((8,48,150x130) f16: a start's worth of 12 channels 56.6 us, of 32 43.8).
    const int per_unit = s.planes * kColsCh;
    BandColsLayout l;
    // (a launch's host time is part of a small problem's: the layout of the largest chunk stands for all, and 32-bit
    // arithmetic does)
    s.chunk = (p.C < kColsChunk ? p.C + per_unit - 1 : kColsChunk) / per_unit * per_unit;
    if (s.chunk < per_unit) s.chunk = per_unit;
    if (!band_cols_layout(p, s, l)) return false;
    const long long items = (long long)p.B * s.bands;
    if (items * p.C > (1ll << 30)) return false;
    const unsigned slots = (unsigned)(sm_count * l.ctas), C = (unsigned)p.C, unit = (unsigned)per_unit;
    unsigned long long best_cost_chunk = ~0ull;
    for (unsigned chunk = unit;; chunk += unit) {
        const unsigned chunks = (C + chunk - 1) / chunk;
        const bool last = chunk + unit > (unsigned)kColsChunk || chunks == 1;
        if (chunks > (unsigned)kBandBwdParts && !last) continue;
        const unsigned waves = ((unsigned)items * chunks + slots - 1) / slots;
        const unsigned long long cost = (unsigned long long)waves * (chunk / (unsigned)s.planes + 32u) + chunks;
        if (cost < best_cost_chunk) {
            best_cost_chunk = cost;
            s.chunk = (int)chunk;
            s.chunks = (int)chunks;
        }
        if (last) break;
    }
    return (long long)p.B * s.bands * s.chunks <= (1ll << 30);
}

template <typename T, int K, int D, int MODE>
int band_cols_launch(const BandBwdArgs& a, const BandColsSplit& sp, cudaStream_t stream, int* launches) {
    constexpr int ES = (int)sizeof(T);
    const Problem& p = a.p;
    if (((reinterpret_cast<uintptr_t>(a.go) | reinterpret_cast<uintptr_t>(a.x)) & 15u) != 0) return kNotHandled;
    BandColsLayout l;
    if (!band_cols_layout(p, sp, l)) return kNotHandled;
    BandColsPlan cp;
    BandBwdPlan& pl = cp.p;
    pl.go = a.go; pl.x = a.x; pl.cf = a.cf; pl.sf = a.sf; pl.gcf = a.gcf; pl.gsf = a.gsf;
    // samples per slice: what the scratch holds
    const size_t n_sf = band_part_sf(p, sp), n_cf = band_part_cf(p, sp);
    const size_t fit = n_sf + n_cf > 0 ? a.workspace_bytes / (n_sf + n_cf) : (size_t)p.B;
    if (fit < 1) return DDF_B200_E_WORKSPACE;
    const int samples = fit < (size_t)p.B ? (int)fit : p.B;
    char* ws = reinterpret_cast<char*>(a.workspace);
    pl.part_sf = a.gsf && n_sf ? ws : nullptr;
    pl.part_cf = a.gcf && n_cf ? reinterpret_cast<float*>(ws + n_sf * (size_t)samples) : nullptr;
    pl.C = p.C; pl.H = p.H; pl.W = p.W; pl.OH = p.OH; pl.OW = p.OW;
    pl.bands = sp.bands; pl.groups = sp.groups; pl.chunk = sp.chunk; pl.chunks = sp.chunks; pl.planes = sp.planes;
    pl.n_warps = sp.warps;
    pl.plane_warps = K * sp.col_warps;
    cp.col_warps = sp.col_warps;
    cp.x_parts = sp.x_parts;
    pl.x_total = (unsigned long long)p.B * p.C * p.H * p.W * ES;
    pl.go_total = (unsigned long long)p.B * p.C * p.OH * p.OW * ES;
    pl.fault = a.fault; pl.wait_cycles = a.wait_cycles; pl.tx_skew = a.tx_skew;
    pl.off_cf = l.off_cf; pl.off_part = l.off_part; pl.off_slot0 = l.off_slot0; pl.slot_stride = l.slot_stride;
    pl.zero_off = l.zero_off; pl.go_off = l.go_off; pl.n_slots = l.n_slots;
    cp.off_red = l.off_red; cp.part_stride = l.part_stride;
    auto kern = band_cols_kernel<T, K, D, MODE>;
    static std::atomic<unsigned long long> opted_in{0};
    const unsigned long long bit = 1ull << (a.device & 63);
    if (!(opted_in.load(std::memory_order_acquire) & bit)) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBudget);
        if (e != cudaSuccess) return (int)e;
        opted_in.fetch_or(bit, std::memory_order_release);
    }
    for (int b0 = 0; b0 < p.B; b0 += samples) {
        const int nb = p.B - b0 < samples ? p.B - b0 : samples;
        pl.b0 = b0;
        cudaError_t e = launch_overlapped(kern, dim3((unsigned)(nb * sp.bands * sp.chunks)),
                                          dim3((unsigned)(sp.warps + 1) * 32), l.smem, stream, true, cp);
        if (e != cudaSuccess) return (int)e;
        ++*launches;
        const int rc = band_reduce_launch<T>(a, sp, pl, b0, nb, stream, launches);
        if (rc) return rc;
    }
    return 0;
}

}  // namespace ddf
