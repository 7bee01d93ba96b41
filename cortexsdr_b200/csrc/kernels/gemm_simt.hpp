// fp32 projection on the CUDA cores for the shapes the tensor-core path does not take.
#pragma once

#include <cstddef>
#include <cstdint>

#include "views.cuh"

struct csdr_context;

namespace csdr {

// y = W x (+ bias) with W fp32 [rows][cols] row-major in device memory, any rows, cols and batch;
// sums in fp32. y may be any YView over all tokens (the Dx of a dictionary is the feature-major
// view with stride y.Mtotal). Uses scratch slot 1 for the partial sums of its column ranges.
// w_fresh: W was written by earlier work on the stream (else it is resident and may be read ahead).
void launch_gemm_simt(csdr_context* ctx, const float* W, uint32_t rows, uint32_t cols, const XView& x, const YView& y,
                      bool w_fresh);

// The same for several weights of one width, each over its own activations (x.x is not read; the form of
// all is x's): member i's rows start at row row_off of the result, which has `rows` rows in all.
constexpr uint32_t kSimtMembers = 16;
struct SimtMember {
    const float* W;
    const void* x;
    uint32_t rows, row_off;
};
void launch_gemm_simt_many(csdr_context* ctx, const SimtMember* members, uint32_t n_members, uint32_t rows, uint32_t cols, const XView& x,
                           const YView& y, bool w_fresh);

}  // namespace csdr
