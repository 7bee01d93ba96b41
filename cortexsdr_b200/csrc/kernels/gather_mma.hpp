// Gather of wide token tiles on the tensor cores (gather_mma.cu).
#pragma once

#include <cstdint>

#include "gemm_tcgen05.hpp"
#include "views.cuh"

namespace csdr {

// Row tiles whose dictionary is pairs of 64-atom blocks up to 512 atoms and whose stage scales are such
// that a row's coefficient on an atom is exact in bf16, at a batch where the tensor cores are quicker.
// Builds the segment's coefficient entries on the way; false where they cannot be had.
bool gather_mma_ready(csdr_context* ctx, const csdr_segment* seg, size_t batch);
// y = gather of Dx (* 1/rms) (+ bias) (+ residual), as launch_wide_gather.
void launch_gather_mma(csdr_context* ctx, const csdr_segment* seg, const DxPlanes& dx, uint32_t M, const YView& y,
                       const float* residual, const TokenScale& ts);

}  // namespace csdr
