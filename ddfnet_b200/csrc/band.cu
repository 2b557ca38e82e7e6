// Band filter gradients: host-side entry (see band.cuh).
#include "band.cuh"

#include "band_bwd_cols.cuh"

namespace ddf {

// The plane-streaming form takes a row in pieces of four pixels where four divide it, else of two or one, and its
// instructions per channel are then spread over as few pixels.  us, plane-streaming -> a thread per tap column:
// (64,512,14x14) f16 59.6 -> 41.8, bf16 k = 5 167 -> 124; (64,512,7x7) f16 35.3 -> 28.8, bf16 k = 5 123 -> 64.  With
// four: (64,256,28x28) bf16 49.7 -> 80.6, k = 5 186 -> 188; (128,64,56x56) bf16 117 -> 120.  Where five eighths of the
// lanes have no pixel it takes many planes to be worth it ((16,256,9x11) bf16 11.1 -> 12.5, (8,512,7x7) 11.0 both), and
// two-pixel pieces with dilation 2 are level ((16,256,22x26) bf16 22.2 -> 22.9).  Where a plane is several bands, at k = 3,
// two-pixel pieces are the faster ones unless there are few planes: over 63 drawn problems 0.8 times below 600 planes, 0.98
// to 1500, 1.09 from there ((99,456,17x22) bf16 add 76 -> 129, (51,88,26x26) f16 23.3 -> 35.5); one-pixel pieces 0.94 of 44.
bool band_cols_preferred(const Problem& p, int sm_count) {
    BandColsSplit s;
    if (p.OW % 4 == 0 || (p.k == 3 && p.d != 1) || !band_cols_split(p, sm_count, s)) return false;
    if (p.k == 3 && p.OW % 2 == 0 && s.bands > 1 && (long long)p.B * p.C >= 1500) return false;
    const long long lanes = (long long)s.bands * s.col_warps * 32 * kColsPixels;
    return 5 * lanes <= 8ll * p.OH * p.OW || (long long)p.B * p.C >= 8192;
}

bool band_filters_workspace(const Problem& p, int sm_count, size_t* bytes, size_t* least) {
    BandColsSplit s;
    const bool cols = p.dtype != DDF_B200_F32 && p.s == 1;
    if (!(cols ? band_cols_split(p, sm_count, s) : band_filters_split(p, sm_count, s))) return false;
    *least = band_part_sf(p, s) + band_part_cf(p, s);
    size_t samples = *least > 0 ? kBandBwdScratch / *least : 1;
    if (samples < 1) samples = 1;
    if (samples > (size_t)p.B) samples = (size_t)p.B;
    *bytes = *least * samples;
    return true;
}

int band_filters(const Problem& p, const void* go, const void* x, const void* cf, const void* sf, void* gcf, void* gsf,
                 void* workspace, size_t workspace_bytes, int sm_count, int* fault, int device, cudaStream_t st, int* launches,
                 long long wait_cycles, uint32_t tx_skew) {
    *launches = 0;
    const BandBwdArgs a{go, x, cf, sf, gcf, gsf, workspace, workspace_bytes, p, sm_count, fault, device, wait_cycles, tx_skew};
    switch (p.dtype) {
        case DDF_B200_F32: return band_filters_dispatch<float>(a, st, launches);
        case DDF_B200_F16: return band_filters_dispatch<__half>(a, st, launches);
        case DDF_B200_BF16: return band_filters_dispatch<__nv_bfloat16>(a, st, launches);
        default: return kNotHandled;
    }
}

}  // namespace ddf
