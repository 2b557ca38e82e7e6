// Band filter gradients: host-side entry (see band.cuh).
#include "band.cuh"

#include "band_bwd.cuh"

namespace ddf {

bool band_filters_workspace(const Problem& p, int sm_count, size_t* bytes, size_t* least) {
    BandBwdSplit s;
    if (!band_filters_split(p, sm_count, s)) return false;
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
