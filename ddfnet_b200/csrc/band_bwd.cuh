// Band form of the two filter gradients, for planes of any height and any width up to 320 output columns (see
// band_fwd.cuh for the bands, the ring and the thread layout; the 2-byte types take it at stride 2, at stride 1 see
// band_bwd_cols.cuh):
//
//   gcf[b,c,t]   = sum_{y,x} go[b,c,y,x] * x[b,c,y*s+oi,x*s+oj] * (sf[b,t,y,x] | 1)
//   gsf[b,t,y,x] = sum_c     go[b,c,y,x] * x[b,c,y*s+oi,x*s+oj] * (cf[b,c,t]   | 1)
//
// One pass over go and x makes both.  A CTA takes one band and a chunk of a sample's channels.  gsf stays
// in registers while the CTA walks its channels, and leaves as one float partial per channel chunk; gcf is
// folded over a warp by a butterfly per channel and over the CTA's warps at its end, and leaves as one
// partial per band.  A second launch adds the partials in a fixed order (no atomics) and rounds; where
// there is one partial, the CTA rounds it.
//
// The sums over channels are compensated for float tensors, as in the generic kernels this one stands in
// for, and their partials are doubles: relative error of gsf against 64 bits at (4,128,50x67) 4.4e-8, as the
// generic kernel's; Kahan sums and float partials gave 5.4e-8 (and 256 us instead of 300 at (2,256,200x300), now 280;
// the generic kernels 3230).  For the 2-byte types the final rounding is 2^13 (f16) or 2^16 (bf16) times a
// float's, and the sums are plain, over 64 channels at most before a compensated sum takes them: the error of
// gsf against 64 bits is the generic kernel's to six digits (2.1e-4 f16, 1.66e-3 bf16; 77 drawn problems, on this form,
// which they now take at stride 2 alone); Kahan's sum took (2,256,200x300) bf16 from 180 to 265 us.
// gcf: the pixels of a warp are added as a tree, in plain float, the warps and bands compensated.  Error for
// float against 64 bits 0.94 to 1.005 times the generic kernel's (which adds a thread's pixels compensated and
// the threads plainly), for the 2-byte types the same to six digits.
//
// Padding.  Taps outside the plane contribute nothing, whatever the other factors hold: gsf of such a tap
// is zero by definition and stored as such; a gcf partial that is not finite in a warp at the plane's edge
// (a zero may have met an infinity) is formed again with those products left out.
#pragma once

#include <type_traits>

#include "band_fwd.cuh"
#include "bwd_stream_impl.cuh"
#include "generic.cuh"

namespace ddf {

// Threads: a thread holds k*k*PH filter values and k*k*PH sums (float: and their corrections).
constexpr int kBandBwdThreads = 352;
// Channels per CTA at most: the per-warp gcf partials of all of them wait in shared memory.
template <int K> constexpr int kBandBwdChunk = K == 3 ? 64 : 24;
template <int K> constexpr int kBandBwdPixels = K == 3 ? 4 : 2;
constexpr int kBandBwdParts = 32;  // gsf partials per element at most (unless the chunk limit asks for more)
// Scratch asked for at most, unless one sample needs more: the partials can be several times x's bytes (k = 5,
// 24 channels a chunk: twice), so a large batch goes through the scratch in slices of
// samples.  A slice of this size is still some 3000 CTAs, ten waves.
constexpr size_t kBandBwdScratch = 256u << 20;

template <typename T> using BandPart = std::conditional_t<sizeof(T) == 4, double, float>;

struct BandBwdPlan {
    const void* go;
    const void* x;
    const void* cf;
    const void* sf;
    void* gcf;         // may be null
    void* gsf;         // may be null
    void* part_sf;     // [b][chunk][t][pixel], BandPart<T>; null: one chunk, rounded here
    float* part_cf;    // [b][band][c][t]; null likewise
    int C, H, W, OH, OW;
    int b0;            // the slice's first sample
    int bands, groups, chunk, chunks, planes;
    int n_slots, n_warps, plane_warps;
    unsigned long long x_total, go_total;
    uint32_t off_cf, off_part, off_slot0, slot_stride, zero_off, go_off;  // zero_off, go_off: from a slot's data
    int* fault;
    long long wait_cycles;
    uint32_t tx_skew;  // see BandPlan
};

template <typename T, int K, int D, int S, int PH, int MODE>
__global__ void __launch_bounds__(kBandBwdThreads, 1)
band_filters_kernel(const __grid_constant__ BandBwdPlan pl) {
    constexpr int KK = K * K, R = (K - 1) / 2, ES = (int)sizeof(T);
    constexpr int NR = S * (PH - 1) + K;
    constexpr int HP = PH / 2;
    constexpr int CFC = (K + 1) / 2 * 16, CFB = kBandCf<K>;
    constexpr bool MUL = MODE == DDF_B200_MUL;
    constexpr bool COMP = sizeof(T) == 4;
    constexpr int GROUP = K == 3 ? KK : K;   // values per butterfly: all taps, or a column of them
    constexpr int COLS = GROUP / K;          // tap columns per butterfly
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

    // bands are innermost: neighbouring bands of the same planes run together and share halo rows in L2
    int item = blockIdx.x;
    const int band = item % pl.bands;
    item /= pl.bands;
    const int chunk_i = item % pl.chunks;
    const int bs = item / pl.chunks;  // sample within the slice
    const int b = pl.b0 + bs;
    const int c_lo = chunk_i * pl.chunk;
    const int c_hi = c_lo + pl.chunk < pl.C ? c_lo + pl.chunk : pl.C;
    const int npass = (c_hi - c_lo + G - 1) / G;
    const int y_lo = band_row<D, PH>(band * pl.groups);
    const int y_next = y_lo + band_rows<D, PH>(pl.groups);
    int y_hi = y_next < pl.OH ? y_next : pl.OH;
    int iy_lo = y_lo * S - R * D > 0 ? y_lo * S - R * D : 0;
    const int iy_end = (y_hi - 1) * S + R * D + 1;
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
        // ------------------------------------------------------------- producer
        if (lane == 0) {
            int issued = 0;
            for (; issued < npass; ++issued) {
                const int slot = issued % NST;
                if (!band_slot_free(BAND_EMPTY(slot), issued, NST, pl.wait_cycles, pl.tx_skew)) break;
                const int left = c_hi - c_lo - issued * G;
                const unsigned long long more = (unsigned long long)((left < G ? left : G) - 1);
                const unsigned long long x0 = x_first + (unsigned long long)issued * G * xplane;
                const unsigned long long g0 = go_first + (unsigned long long)issued * G * gplane;
                const Span sx = span_prepare(BAND_DATA(slot), pl.x, x0,
                                             x0 + more * xplane + (unsigned long long)(iy_hi - iy_lo) * pl.W * ES, pl.x_total);
                const Span sg = span_prepare(BAND_DATA(slot) + pl.go_off, pl.go, g0,
                                             g0 + more * gplane + (unsigned long long)(y_hi - go_row) * pl.OW * ES, pl.go_total);
                mbar_arrive_expect_tx(BAND_FULL(slot), sx.bytes + sg.bytes + pl.tx_skew);
                span_issue(sx, BAND_FULL(slot));
                span_issue(sg, BAND_FULL(slot));
            }
            band_leave(BAND_FULL(0), issued, npass, NST, pl.wait_cycles, pl.tx_skew, pl.fault);
        }
        return;
    }

    // ----------------------------------------------------------------- compute warps
    const int npos = pl.groups * pl.OW;
    const int pip = warp / pl.plane_warps;  // a warp never holds two planes
    const int wip = warp - pip * pl.plane_warps;
    int pos = wip * 32 + lane;
    bool active = pos < npos;
    if (!active) pos = 0;
    const int grp = pos / pl.OW;
    const int x = pos - grp * pl.OW;
    const int y0 = y_lo + band_row<D, PH>(grp);
    if (y0 >= pl.OH) active = false;
    int rows_left = active ? (pl.OH - y0 + D - 1) / D : 0;
    if (rows_left > PH) rows_left = PH;

    // Rows no pixel of this thread needs, and pixels outside the plane, read zeros.
    uint32_t rowoff[NR], gooff[PH];
    uint32_t rowbits = 0, colbits = 0;
#pragma unroll
    for (int r = 0; r < NR; ++r) {
        const int iy = y0 * S + D * (r - R);
        const bool ok = rows_left > 0 && r <= S * (rows_left - 1) + K - 1 && iy >= 0 && iy < pl.H;
        rowbits |= ok ? 1u << r : 0u;
        rowoff[r] = ok ? (uint32_t)pip * (uint32_t)xplane + (uint32_t)(((iy - iy_lo) * pl.W + x * S) * ES)
                       : pl.zero_off + 16u;
        pin(rowoff[r]);
    }
#pragma unroll
    for (int p = 0; p < PH; ++p) {
        gooff[p] = p < rows_left ? (uint32_t)pip * (uint32_t)gplane + (uint32_t)(((y0 + D * p - y_lo) * pl.OW + x) * ES)
                                 : pl.zero_off + 16u - pl.go_off;
        pin(gooff[p]);
    }
    uint32_t cmask[K];
#pragma unroll
    for (int j = 0; j < K; ++j) {
        const int ix = x * S + D * (j - R);
        const bool ok = ix >= 0 && ix < pl.W;
        colbits |= ok ? 1u << j : 0u;
        cmask[j] = Masked<T>::mask(ok);
        pin(cmask[j]);
    }
    // products with padding zeros, or of pixels outside the plane, in this thread / warp
    const bool edge = colbits != (1u << K) - 1u || rowbits != (1u << NR) - 1u || rows_left < PH;
    const bool edge_warp = __any_sync(0xffffffffu, edge);
    auto inside = [&](int j, int k, int p) {  // tap (row k, column j) of pixel p lies in the plane
        return p < rows_left && ((colbits >> j) & 1u) != 0u && ((rowbits >> (S * p + k)) & 1u) != 0u;
    };

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
    unsigned long long sf2[MUL ? KK : 1][HP];  // [column-major tap][pair]
    if constexpr (MUL) {
        const T* sfb = reinterpret_cast<const T*>(pl.sf) + (long long)b * KK * opl;
        const T* at[PH];  // a clamped address and values dropped after: see band_kernel
#pragma unroll
        for (int p = 0; p < PH; ++p) at[p] = p < rows_left ? sfb + (y0 + p * D) * pl.OW + x : sfb;
#pragma unroll
        for (int t = 0; t < KK; ++t) {
            float v[PH];
#pragma unroll
            for (int p = 0; p < PH; ++p) {
                const float w = Elem<T>::load(at[p] + t * opl);
                v[p] = p < rows_left ? w : 0.f;
            }
#pragma unroll
            for (int q = 0; q < HP; ++q) {
                sf2[(t % K) * K + t / K][q] = f2_pack(v[q], v[q + HP]);
                pin(sf2[(t % K) * K + t / K][q]);
            }
        }
    }
    band_sync(NW * 32);

    unsigned long long gsf2[KK][HP], lost2[COMP ? KK : 1][HP];
#pragma unroll
    for (int t = 0; t < KK; ++t)
#pragma unroll
        for (int q = 0; q < HP; ++q) {
            gsf2[t][q] = 0ull;
            if constexpr (COMP) lost2[t][q] = 0ull;
        }
    const unsigned long long minus1 = f2_pack(-1.f, -1.f);
    const int my_slot = butterfly_slot<GROUP>(lane);

    uint32_t x_lo = (uint32_t)x_first, go_lo = (uint32_t)go_first;
    const uint32_t x_step = (uint32_t)((unsigned long long)G * xplane), go_step = (uint32_t)((unsigned long long)G * gplane);
    uint32_t cf_s = sbase + pl.off_cf + (uint32_t)pip * CFB;
    uint32_t part_s = sbase + pl.off_part + 4u * (uint32_t)((pip * pl.plane_warps + wip) * KK);
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
        if (left > 0) {  // this warp's plane of the pass exists
            const uint32_t xbase = BAND_DATA(slot) + (x_lo & 15u);
            const uint32_t gbase = BAND_DATA(slot) + pl.go_off + (go_lo & 15u);
            float g[PH];
#pragma unroll
            for (int p = 0; p < PH; ++p) g[p] = Masked<T>::load(gbase + gooff[p]);
            unsigned long long g2[HP];
#pragma unroll
            for (int q = 0; q < HP; ++q) g2[q] = f2_pack(g[q], g[q + HP]);
            uint32_t row[NR];
#pragma unroll
            for (int r = 0; r < NR; ++r) row[r] = xbase + rowoff[r];

            auto load_column = [&](int j, float (&v)[NR]) {
#pragma unroll
                for (int r = 0; r < NR; ++r)
                    v[r] = j == R ? Masked<T>::load(row[r])
                                  : Masked<T>::load(row[r] + (uint32_t)((D * (j - R)) * ES), cmask[j]);
            };
#pragma unroll
            for (int j0 = 0; j0 < K; j0 += COLS) {
                float part[GROUP];
#pragma unroll
                for (int jj = 0; jj < COLS; ++jj) {
                    const int j = j0 + jj;
                    unsigned long long cp[MUL ? (K + 1) / 2 * 2 : 1];
                    if constexpr (MUL) {
#pragma unroll
                        for (int t = 0; t < (K + 1) / 2; ++t)
                            lds128_pairs(cf_s + (uint32_t)(j * CFC + 16 * t), cp[2 * t], cp[2 * t + 1]);
                    }
                    float v[NR];
                    load_column(j, v);
#pragma unroll
                    for (int k = 0; k < K; ++k) {
                        const int t = j * K + k;
                        unsigned long long part2 = 0ull;
#pragma unroll
                        for (int q = 0; q < HP; ++q) {
                            const unsigned long long prod2 = f2_mul(g2[q], f2_pack(v[S * q + k], v[S * (q + HP) + k]));
                            if constexpr (COMP) {
                                // the exact error of each addition is summed apart
                                unsigned long long v2 = prod2;
                                if constexpr (MUL) v2 = f2_mul(prod2, cp[k]);
                                const unsigned long long t2 = f2_add(gsf2[t][q], v2);
                                const unsigned long long d2 = f2_fma(gsf2[t][q], minus1, t2);
                                const unsigned long long e2 = f2_fma(f2_fma(d2, minus1, t2), minus1, gsf2[t][q]);
                                lost2[t][q] = f2_add(lost2[t][q], f2_add(e2, f2_fma(d2, minus1, v2)));
                                gsf2[t][q] = t2;
                            } else {
                                if constexpr (MUL) gsf2[t][q] = f2_fma(prod2, cp[k], gsf2[t][q]);
                                else gsf2[t][q] = f2_add(gsf2[t][q], prod2);
                            }
                            if constexpr (HP == 1) part2 = prod2;
                            else if constexpr (MUL) part2 = f2_fma(prod2, sf2[t][q], part2);
                            else part2 = f2_add(part2, prod2);
                        }
                        float lo, hi;
                        f2_unpack(part2, lo, hi);
                        if constexpr (MUL && HP == 1) {
                            // one rounding less for the same two instructions
                            float s_lo, s_hi;
                            f2_unpack(sf2[t][0], s_lo, s_hi);
                            part[jj * K + k] = fmaf(hi, s_hi, lo * s_lo);
                        } else {
                            part[jj * K + k] = lo + hi;
                        }
                    }
                }
                if (edge_warp) {
                    float sum = 0.f;
#pragma unroll
                    for (int t = 0; t < GROUP; ++t) sum += part[t];
                    if (edge && !(fabsf(sum) < __int_as_float(0x7f800000))) {
#pragma unroll
                        for (int jj = 0; jj < COLS; ++jj) {
                            const int j = j0 + jj;
                            float v[NR];
                            load_column(j, v);
#pragma unroll
                            for (int k = 0; k < K; ++k) {
                                float a = 0.f;
#pragma unroll
                                for (int p = 0; p < PH; ++p) {
                                    float s = 1.f;
                                    if constexpr (MUL) {
                                        float lo, hi;
                                        f2_unpack(sf2[j * K + k][p % HP], lo, hi);
                                        s = p < HP ? lo : hi;
                                    }
                                    if (inside(j, k, p)) a = fmaf(g[p] * v[S * p + k], s, a);
                                }
                                part[jj * K + k] = a;
                            }
                        }
                    }
                    __syncwarp();
                }
                butterfly_reduce<GROUP>(part, lane);
                if (my_slot >= 0) sts32(part_s + 4u * (uint32_t)(j0 * K + my_slot), __float_as_uint(part[0]));
            }
        }
        __syncwarp();
        if (lane == 0 && ph < kBandDead) mbar_arrive(BAND_EMPTY(slot));
        x_lo += x_step;
        go_lo += go_step;
        cf_s += (uint32_t)G * CFB;
        part_s += 4u * (uint32_t)(NW * KK);
        left -= G;
    }
    if (band_sync_or(NW * 32, ph >= kBandDead ? 1 : 0)) return;  // a fault is recorded, and there are no whole sums

    if (pl.gcf != nullptr) {  // this band's share of gcf: the plane's warps added up; taps back in row order
        const int n = (c_hi - c_lo) * KK;
        for (int e = tid; e < n; e += NW * 32) {
            const int c = e / KK, t = e - c * KK;
            const int i = c / G;
            const uint32_t src = sbase + pl.off_part +
                                 4u * (uint32_t)((i * NW + (c - i * G) * pl.plane_warps) * KK + (t % K) * K + t / K);
            CompSum<float> tot;
            for (int w = 0; w < pl.plane_warps; ++w) tot.add(ldsf(src + 4u * (uint32_t)(w * KK)));
            if (pl.part_cf != nullptr)
                pl.part_cf[(((long long)bs * pl.bands + band) * pl.C + c_lo) * KK + e] = tot.value();
            else
                Elem<T>::store(reinterpret_cast<T*>(pl.gcf) + (long long)first_plane * KK + e, tot.value());
        }
    }
    if (pl.gsf != nullptr) {
        using P = BandPart<T>;
        P* ps = pl.part_sf == nullptr
                    ? nullptr
                    : reinterpret_cast<P*>(pl.part_sf) + ((long long)bs * pl.chunks + chunk_i) * KK * opl;
        T* os = reinterpret_cast<T*>(pl.gsf) + (long long)b * KK * opl;
        auto put = [&](long long o, P v) {
            if (ps != nullptr) ps[o] = v;
            else Elem<T>::store(os + o, (float)v);
        };
        // Several planes per pass: a band is then the whole plane, and the planes' sums meet in the slots
        // (every copy has landed and been read).
        P* meet = reinterpret_cast<P*>(smem_raw + pl.off_slot0 + kBandGuard);
#pragma unroll
        for (int t = 0; t < KK; ++t) {  // column-major tap
            const int ft = (t % K) * K + t / K;
#pragma unroll
            for (int q = 0; q < HP; ++q) {
                float v0, v1, l0 = 0.f, l1 = 0.f;
                f2_unpack(gsf2[t][q], v0, v1);
                if constexpr (COMP) f2_unpack(lost2[t][q], l0, l1);
                const P v[2] = {(P)v0 + (P)l0, (P)v1 + (P)l1};
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int p = q + h * HP;
                    if (p < rows_left) {
                        const long long o = ft * opl + (long long)(y0 + p * D) * pl.OW + x;
                        const P r = inside(t / K, t % K, p) ? v[h] : (P)0;
                        if (G > 1) meet[pip * KK * (int)opl + (int)o] = r;
                        else put(o, r);
                    }
                }
            }
        }
        if (G > 1) {
            band_sync(NW * 32);
            const int n = KK * (int)opl;
            for (int e = tid; e < n; e += NW * 32) {
                CompSum<P> tot;
                for (int g = 0; g < G; ++g) tot.add(meet[g * n + e]);
                put(e, tot.value());
            }
        }
    }
#undef BAND_FULL
#undef BAND_EMPTY
#undef BAND_DATA
}

// out[s][e] = sum over the partials part[s][0 .. n-1][e], fixed order, compensated, from element `first` on.
template <typename T, typename P>
__device__ __forceinline__ void band_reduce(const P* __restrict__ part, T* __restrict__ out, int n, long long size, int B,
                                            long long first, long long step) {
    for (long long e = first; e < size * B; e += step) {
        const long long s = e / size;
        const P* src = part + s * n * size + (e - s * size);
        CompSum<P> tot;
        for (int j0 = 0; j0 < n; j0 += 8) {  // eight loads in flight
            P v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) v[u] = j0 + u < n ? __ldg(src + (long long)(j0 + u) * size) : (P)0;
#pragma unroll
            for (int u = 0; u < 8; ++u) tot.add(v[u]);
        }
        Elem<T>::store(out + e, (float)tot.value());
    }
}

// The first `sf_blocks` blocks add up gsf, the others gcf.
template <typename T>
__global__ void __launch_bounds__(256)
band_reduce_kernel(const BandPart<T>* part_sf, T* gsf, int n_sf, long long sf_size, const float* part_cf, T* gcf, int n_cf,
                   long long cf_size, int B, int sf_blocks) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int block = (int)blockIdx.x - sf_blocks;
    if (block < 0)
        band_reduce(part_sf, gsf, n_sf, sf_size, B, blockIdx.x * 256ll + threadIdx.x, sf_blocks * 256ll);
    else
        band_reduce(part_cf, gcf, n_cf, cf_size, B, block * 256ll + threadIdx.x, (gridDim.x - sf_blocks) * 256ll);
}

// ------------------------------------------------------------------------ host side
struct BandBwdSplit : BandSplit {
    int chunk, chunks;  // channels per CTA, CTAs per (sample, band)
};

// The split of a problem; false: not built for it.
inline bool band_filters_split(const Problem& p, int sm_count, BandBwdSplit& s) {
    const bool built = (p.k == 3 && ((p.d <= 2 && p.s == 1) || (p.d == 1 && p.s == 2))) ||
                       (p.k == 5 && p.d <= 2 && p.s == 1);
    if (!built || p.dtype == DDF_B200_F64) return false;
    const int PH = p.k == 3 ? kBandBwdPixels<3> : kBandBwdPixels<5>;
    const int max_chunk = p.k == 3 ? kBandBwdChunk<3> : kBandBwdChunk<5>;
    if (!band_split(p.B, p.C, p.OH, p.OW, p.d, PH, kBandBwdThreads, true, s)) return false;
    // Channels per CTA: the count with the least (waves of CTAs) x (passes + about six passes' worth of
    // start and partial sums).
    const long long slots = (long long)sm_count * (s.warps <= 5 ? 2 : 1);
    long long best = -1;
    for (int n = 1; n <= kBandBwdParts || best < 0; ++n) {
        int chunk = (p.C + n - 1) / n;
        chunk = (chunk + s.planes - 1) / s.planes * s.planes;
        if (chunk > max_chunk && chunk > s.planes) continue;
        const int chunks = (p.C + chunk - 1) / chunk;
        const long long waves = ((long long)p.B * s.bands * chunks + slots - 1) / slots;
        const long long cost = waves * (chunk / s.planes + 6);
        if (best < 0 || cost < best) {
            best = cost;
            s.chunk = chunk;
            s.chunks = chunks;
        }
        if (chunk == s.planes) break;
    }
    if ((long long)p.B * s.bands * s.chunks > (1ll << 30)) return false;
    const int es = p.dtype == DDF_B200_F32 ? 4 : 2;
    const int out_rows = s.groups % p.d == 0 ? s.groups * PH : p.d * (PH - 1) + 1;
    const long long rows = (long long)(out_rows - 1) * p.s + (p.k - 1) * p.d + 1;
    const long long run = ((s.planes - 1) * (long long)p.H + (rows < p.H ? rows : p.H)) * p.W * es;
    return run <= (64 << 10);
}

// Bytes that one sample's gsf / gcf partials take (0: none needed).
inline size_t band_part_sf(const Problem& p, const BandBwdSplit& s) {
    return s.chunks > 1 ? (size_t)s.chunks * p.k * p.k * p.OH * p.OW *
                              (p.dtype == DDF_B200_F32 ? sizeof(double) : sizeof(float)) : 0;
}
inline size_t band_part_cf(const Problem& p, const BandBwdSplit& s) {
    return s.bands > 1 ? (size_t)s.bands * p.C * p.k * p.k * sizeof(float) : 0;
}

struct BandBwdArgs {
    const void* go;
    const void* x;
    const void* cf;
    const void* sf;
    void* gcf;
    void* gsf;
    void* workspace;
    size_t workspace_bytes;
    Problem p;
    int sm_count;
    int* fault;
    int device;
    long long wait_cycles = kWaitCycles;
    uint32_t tx_skew = 0;
};

// The second launch of a slice of samples: the partials added up.
template <typename T>
int band_reduce_launch(const BandBwdArgs& a, const BandBwdSplit& sp, const BandBwdPlan& pl, int b0, int nb, cudaStream_t stream,
                       int* launches) {
    if (!pl.part_sf && !pl.part_cf) return 0;
    const long long kk = a.p.k * a.p.k, sf_size = kk * a.p.OH * a.p.OW, cf_size = a.p.C * kk;
    auto blocks = [&](long long n) {
        const long long most = 4ll * a.sm_count;
        return (int)((n + 255) / 256 < most ? (n + 255) / 256 : most);
    };
    const int nb_sf = pl.part_sf ? blocks(sf_size * nb) : 0, nb_cf = pl.part_cf ? blocks(cf_size * nb) : 0;
    T* gsf = pl.part_sf ? reinterpret_cast<T*>(a.gsf) + b0 * sf_size : nullptr;
    T* gcf = pl.part_cf ? reinterpret_cast<T*>(a.gcf) + b0 * cf_size : nullptr;
    const cudaError_t e = launch_overlapped(band_reduce_kernel<T>, dim3((unsigned)(nb_sf + nb_cf)), dim3(256), 0, stream, true,
                                            (const BandPart<T>*)pl.part_sf, gsf, sp.chunks, sf_size, (const float*)pl.part_cf,
                                            gcf, sp.bands, cf_size, nb, nb_sf);
    if (e != cudaSuccess) return (int)e;
    ++*launches;
    return 0;
}

template <typename T, int K, int D, int S, int MODE>
int band_filters_launch(const BandBwdArgs& a, cudaStream_t stream, int* launches) {
    constexpr int PH = kBandBwdPixels<K>, ES = (int)sizeof(T);
    const Problem& p = a.p;
    if (((reinterpret_cast<uintptr_t>(a.go) | reinterpret_cast<uintptr_t>(a.x)) & 15u) != 0) return kNotHandled;
    BandBwdSplit sp;
    if (!band_filters_split(p, a.sm_count, sp)) return kNotHandled;
    BandBwdPlan pl;
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
    pl.plane_warps = sp.warps / sp.planes;
    pl.x_total = (unsigned long long)p.B * p.C * p.H * p.W * ES;
    pl.go_total = (unsigned long long)p.B * p.C * p.OH * p.OW * ES;
    pl.fault = a.fault; pl.wait_cycles = a.wait_cycles; pl.tx_skew = a.tx_skew;
    const long long rows = (long long)(band_rows<D, PH>(sp.groups) - 1) * S + (K - 1) * D + 1;
    const long long grows = band_rows<D, PH>(sp.groups);
    const uint32_t xrun = (uint32_t)(((sp.planes - 1) * (long long)p.H + (rows < p.H ? rows : p.H)) * p.W * ES);
    const uint32_t grun = (uint32_t)(((sp.planes - 1) * (long long)p.OH + (grows < p.OH ? grows : p.OH)) * p.OW * ES);
    pl.off_cf = round_up(16u * kBandSlots, 128);
    pl.off_part = round_up(pl.off_cf + (uint32_t)sp.chunk * kBandCf<K>, 128);
    const uint32_t passes = (uint32_t)((sp.chunk + sp.planes - 1) / sp.planes);
    pl.off_slot0 = round_up(pl.off_part + passes * (uint32_t)(sp.warps * K * K * 4), 128);
    pl.zero_off = round_up(xrun + 16u + 32u, 16);
    pl.go_off = round_up(pl.zero_off + kBandZero, 16);
    pl.slot_stride = round_up(kBandGuard + pl.go_off + grun + 32u, 128);
    pl.n_slots = 0;
    for (uint32_t budget : {100u << 10, kSmemBudget}) {  // two CTAs per SM where three slots fit
        for (int n = kBandSlots; n >= 2 && pl.n_slots == 0; --n)
            if (pl.off_slot0 + (uint32_t)n * pl.slot_stride <= budget && (n >= 3 || budget == kSmemBudget)) pl.n_slots = n;
    }
    if (pl.n_slots < 2) return kNotHandled;
    uint32_t smem = pl.off_slot0 + (uint32_t)pl.n_slots * pl.slot_stride;
    if (sp.planes > 1) {  // room for the planes' sums to meet
        const uint32_t meet = pl.off_slot0 + kBandGuard + (uint32_t)(sp.planes * K * K * p.OH * p.OW) * (uint32_t)sizeof(BandPart<T>);
        if (smem < meet) smem = meet;
        if (smem > kSmemBudget) return kNotHandled;
    }
    auto kern = band_filters_kernel<T, K, D, S, PH, MODE>;
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
                                          dim3((unsigned)(sp.warps + 1) * 32), smem, stream, true, pl);
        if (e != cudaSuccess) return (int)e;
        ++*launches;
        const int rc = band_reduce_launch<T>(a, sp, pl, b0, nb, stream, launches);
        if (rc) return rc;
    }
    return 0;
}

// Defined once per element type in band_bwd_inst_<type>.cu.
template <typename T>
int band_filters_dispatch(const BandBwdArgs& a, cudaStream_t stream, int* launches);

}  // namespace ddf
