// Host-side entries of the band filter gradients (band_bwd.cuh).
#pragma once

#include "common.cuh"

namespace ddf {

// Scratch bytes of the filter gradients: what they take, and the least that they run with (0 is possible);
// false when the band form is not built for p.
bool band_filters_workspace(const Problem& p, int sm_count, size_t* bytes, size_t* least);

// Whether AUTO takes the form of a thread per tap column (band_bwd_cols.cuh) where the plane-streaming form is built too.
bool band_cols_preferred(const Problem& p, int sm_count);
constexpr size_t kColsScratch = 16u << 20;

// kNotHandled: not built, or a tensor is not aligned for bulk copies.  `workspace` holds at
// least what band_filters_workspace says, aligned to 8 bytes; the results do not depend on how much.
int band_filters(const Problem& p, const void* go, const void* x, const void* cf, const void* sf, void* gcf, void* gsf,
                 void* workspace, size_t workspace_bytes, int sm_count, int* fault, int device, cudaStream_t st, int* launches,
                 long long wait_cycles = kWaitCycles, uint32_t tx_skew = 0);

}  // namespace ddf
