// fp32 matrix product on the CUDA cores: y[r][t] = sum_c W[r][c] * x[c][t].
//
// Serves the products whose fp32 operands the tensor-core path does not take - dictionaries whose
// atom count is not a multiple of 128 or whose width is not a multiple of 8, and rebuilt weights
// with ragged edges - in the arithmetic they always had (fp32 multiply-add, no 16-bit splits).
#include <cuda_bf16.h>

#include <algorithm>

#include "../internal.hpp"
#include "gemm_simt.hpp"

namespace csdr {

namespace {

// Tile of 64 rows x TOK tokens x 32 columns, 128 threads. Both operands lie in shared memory with
// the columns contiguous (36 floats a row: 16-byte aligned, and eight rows cover the 32 banks), so
// global rows are copied as they are and the inner product runs over pairs of columns on packed
// fp32 multiply-adds; a thread's 8 x 4 results take 12 128-bit reads per 64 packed instructions.
// The bound is fp32 issue for 64 tokens and the weight's bytes for 16; small products are bound by
// the launches. Measured, whole products: 300 atoms of width 350 at 95 tokens 266 -> 21 us (rebuilt
// weight and a row-a-warp product before), 128 of 2579 at 6 tokens, three members, 441 -> 33 us.
constexpr uint32_t kRows = 64, kCols = 32, kPitch = 36, kThreads = 128;

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}

struct SimtParams {
    const float* W;
    uint32_t rows, cols, n_kb, kb_per_split, n_split;
    uint32_t vec;      // rows of W start on 16-byte boundaries
    uint32_t w_fresh;  // W is the output of earlier work on the stream
    XView x;
    YView y;           // n_split == 1
    float* part;       // [split][rows][tokens] otherwise
};

// Copies one 64 x 32 block of W; what lies outside the matrix becomes zero.
__device__ __forceinline__ void load_w(const SimtParams& p, float* ws, uint32_t row0, uint32_t c0, uint32_t tid) {
    if (p.vec) {
#pragma unroll
        for (uint32_t i = 0; i < kRows * kCols / 4u / kThreads; ++i) {
            const uint32_t e = tid + i * kThreads, r = e >> 3, c = (e & 7u) * 4u;
            const bool in = row0 + r < p.rows && c0 + c < p.cols;   // cols is a multiple of four
            const float* src = in ? p.W + static_cast<size_t>(row0 + r) * p.cols + c0 + c : p.W;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(ws + r * kPitch + c)), "l"(src),
                         "r"(in ? 16u : 0u)
                         : "memory");
        }
    } else {
#pragma unroll
        for (uint32_t i = 0; i < kRows * kCols / kThreads; ++i) {
            const uint32_t e = tid + i * kThreads, r = e >> 5, c = e & 31u;
            const bool in = row0 + r < p.rows && c0 + c < p.cols;
            const float* src = in ? p.W + static_cast<size_t>(row0 + r) * p.cols + c0 + c : p.W;
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_u32(ws + r * kPitch + c)), "l"(src),
                         "r"(in ? 4u : 0u)
                         : "memory");
        }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
}

// A thread's share of a TOK x 32 block of the activations, in registers: lanes run along whichever
// of the two dimensions is contiguous in memory.
template <uint32_t TOK>
struct XBlock {
    static constexpr uint32_t N = TOK * kCols / kThreads;
    float v[N];
    __device__ __forceinline__ static void at(const SimtParams& p, uint32_t e, uint32_t& t, uint32_t& c) {
        if (p.x.layout == CSDR_LAYOUT_FEATURE_MAJOR) {
            t = e % TOK;
            c = e / TOK;
        } else {
            t = e / kCols;
            c = e % kCols;
        }
    }
    __device__ __forceinline__ void load(const SimtParams& p, uint32_t t0, uint32_t c0, uint32_t tid) {
#pragma unroll
        for (uint32_t i = 0; i < N; ++i) {
            uint32_t t, c;
            at(p, tid + i * kThreads, t, c);
            v[i] = t0 + t < p.x.M && c0 + c < p.cols ? load_x(p.x, c0 + c, t0 + t) : 0.0f;
        }
    }
    __device__ __forceinline__ void store(const SimtParams& p, float* xs, uint32_t tid) const {
#pragma unroll
        for (uint32_t i = 0; i < N; ++i) {
            uint32_t t, c;
            at(p, tid + i * kThreads, t, c);
            xs[t * kPitch + c] = v[i];
        }
    }
};

// grid (row tiles, token tiles, column ranges). SWAP: lanes run along the rows of W instead of the
// tokens, so that a token-major result leaves in contiguous pieces.
template <uint32_t TOK, bool SWAP>
__global__ void __launch_bounds__(kThreads)
hsdr_gemm_simt_kernel(const __grid_constant__ SimtParams p) {
    __shared__ __align__(16) float ws[2][kRows * kPitch];
    __shared__ __align__(16) float xs[2][TOK * kPitch];
    constexpr uint32_t A = SWAP ? TOK : kRows, B = SWAP ? kRows : TOK;   // slow and fast dimension of the result
    constexpr uint32_t TB = B >= 64u ? 16u : 8u, TA = kThreads / TB;     // threads along each
    constexpr uint32_t NA = A / TA, NB = B / TB;
    const uint32_t tid = threadIdx.x, tb = tid % TB, ta = tid / TB;
    const uint32_t row0 = blockIdx.x * kRows, t0 = blockIdx.y * TOK;
    const uint32_t kb0 = blockIdx.z * p.kb_per_split, kb1 = min(p.n_kb, kb0 + p.kb_per_split);
    unsigned long long acc[NA][NB];
#pragma unroll
    for (uint32_t i = 0; i < NA; ++i)
#pragma unroll
        for (uint32_t j = 0; j < NB; ++j) acc[i][j] = 0ull;
    XBlock<TOK> xb;
    // a resident weight is no other launch's output; a rebuilt one and the activations may be
    if (p.w_fresh) asm volatile("griddepcontrol.wait;" ::: "memory");
    if (kb0 < kb1) load_w(p, ws[0], row0, kb0 * kCols, tid);
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (kb0 < kb1) {
        xb.load(p, t0, kb0 * kCols, tid);
        xb.store(p, xs[0], tid);
    }
    for (uint32_t kb = kb0; kb < kb1; ++kb) {
        const uint32_t s = (kb - kb0) & 1u;
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        const bool more = kb + 1u < kb1;
        if (more) {
            load_w(p, ws[s ^ 1u], row0, (kb + 1u) * kCols, tid);
            xb.load(p, t0, (kb + 1u) * kCols, tid);
        }
        const float* as = (SWAP ? xs[s] : ws[s]) + ta * kPitch;
        const float* bs = (SWAP ? ws[s] : xs[s]) + tb * kPitch;
#pragma unroll 2
        for (uint32_t c = 0; c < kCols; c += 4u) {
            ulonglong2 a[NA], b[NB];
#pragma unroll
            for (uint32_t i = 0; i < NA; ++i) a[i] = *reinterpret_cast<const ulonglong2*>(as + i * TA * kPitch + c);
#pragma unroll
            for (uint32_t j = 0; j < NB; ++j) b[j] = *reinterpret_cast<const ulonglong2*>(bs + j * TB * kPitch + c);
#pragma unroll
            for (uint32_t i = 0; i < NA; ++i)
#pragma unroll
                for (uint32_t j = 0; j < NB; ++j) acc[i][j] = fma2(a[i].y, b[j].y, fma2(a[i].x, b[j].x, acc[i][j]));
        }
        if (more) xb.store(p, xs[s ^ 1u], tid);   // the other buffer: its readers met the barrier above
    }
    asm volatile("griddepcontrol.launch_dependents;");
#pragma unroll
    for (uint32_t i = 0; i < NA; ++i)
#pragma unroll
        for (uint32_t j = 0; j < NB; ++j) {
            const uint32_t a = ta + i * TA, b = tb + j * TB;
            const uint32_t r = row0 + (SWAP ? b : a), t = t0 + (SWAP ? a : b);
            if (r >= p.rows || t >= p.x.M) continue;
            const float v = __uint_as_float(static_cast<uint32_t>(acc[i][j])) + __uint_as_float(static_cast<uint32_t>(acc[i][j] >> 32));
            if (p.n_split > 1u) {
                const size_t o = SWAP ? static_cast<size_t>(t) * p.rows + r : static_cast<size_t>(r) * p.x.M + t;
                p.part[static_cast<size_t>(blockIdx.z) * p.rows * p.x.M + o] = v;
            } else {
                p.y.y[y_index(p.y, r, t)] = v + (p.y.bias ? p.y.bias[r] : 0.0f);
            }
        }
}

// The column ranges' shares added up in range order; one thread per result, laid out like y.
__global__ void __launch_bounds__(256)
simt_reduce_kernel(const float* __restrict__ part, uint32_t rows, uint32_t M, uint32_t n_split, YView y) {
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const size_t n = static_cast<size_t>(rows) * M;
    const size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x;
    if (i >= n) return;
    float v = 0.0f;
    for (uint32_t s0 = 0; s0 < n_split; s0 += 8u) {
        float a[8];
#pragma unroll
        for (uint32_t j = 0; j < 8u; ++j) a[j] = s0 + j < n_split ? __ldcg(part + (s0 + j) * n + i) : 0.0f;
#pragma unroll
        for (uint32_t j = 0; j < 8u; ++j) v += a[j];
    }
    const bool fm = y.layout == CSDR_LAYOUT_FEATURE_MAJOR;
    const uint32_t w = fm ? M : rows, hi = static_cast<uint32_t>(i / w), lo = static_cast<uint32_t>(i - static_cast<size_t>(hi) * w);
    const uint32_t r = fm ? hi : lo, t = fm ? lo : hi;
    y.y[y_index(y, r, t)] = v + (y.bias ? y.bias[r] : 0.0f);
}

}  // namespace

void launch_gemm_simt(csdr_context* ctx, const float* W, uint32_t rows, uint32_t cols, const XView& x, const YView& y,
                      bool w_fresh) {
    if (rows == 0 || x.M == 0) return;
    const bool narrow = x.M <= 16u;
    const bool swap = y.layout == CSDR_LAYOUT_TOKEN_MAJOR;
    const uint32_t tok = narrow ? 16u : 64u;
    SimtParams p{};
    p.W = W;
    p.rows = rows;
    p.cols = cols;
    p.vec = cols % 4u == 0 && (reinterpret_cast<uintptr_t>(W) & 15u) == 0;
    p.w_fresh = w_fresh ? 1u : 0u;
    p.n_kb = (cols + kCols - 1u) / kCols;
    const uint32_t row_tiles = (rows + kRows - 1u) / kRows, tok_tiles = (x.M + tok - 1u) / tok;
    // column ranges: enough CTAs for four per SM, at least two blocks of columns each, and partial
    // sums that stay in L2
    const uint64_t tiles = static_cast<uint64_t>(row_tiles) * tok_tiles, want = 4ull * static_cast<uint32_t>(ctx->sm_count);
    const uint64_t by_part = std::max<uint64_t>(1u, (64ull << 20) / (4ull * rows * x.M));
    uint32_t split = static_cast<uint32_t>(std::min<uint64_t>({std::max<uint64_t>(1u, want / tiles), (p.n_kb + 1u) / 2u, by_part}));
    split = std::max(1u, split);
    p.kb_per_split = (p.n_kb + split - 1u) / split;
    p.n_split = std::max(1u, (p.n_kb + p.kb_per_split - 1u) / p.kb_per_split);
    p.x = x;
    p.y = y;
    const size_t n = static_cast<size_t>(rows) * x.M;
    p.part = p.n_split > 1u ? static_cast<float*>(ctx->scratch_get(1, n * p.n_split * 4u)) : nullptr;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(row_tiles, tok_tiles, p.n_split);
    cfg.blockDim = dim3(kThreads, 1, 1);
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = ctx->pdl ? 1 : 0;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    {
        auto kern = narrow ? (swap ? hsdr_gemm_simt_kernel<16, true> : hsdr_gemm_simt_kernel<16, false>)
                           : (swap ? hsdr_gemm_simt_kernel<64, true> : hsdr_gemm_simt_kernel<64, false>);
        LaunchScope ls(ctx, KC_DX);
        CSDR_CUDA(cudaLaunchKernelEx(&cfg, kern, p));
        ls.done("hsdr_gemm_simt_kernel");
    }
    if (p.n_split > 1u) {
        cfg.gridDim = dim3(static_cast<unsigned>((n + 255u) / 256u), 1, 1);
        cfg.blockDim = dim3(256, 1, 1);
        LaunchScope ls(ctx, KC_DX);
        CSDR_CUDA(cudaLaunchKernelEx(&cfg, simt_reduce_kernel, static_cast<const float*>(p.part), rows, x.M, p.n_split, y));
        ls.done("simt_reduce_kernel");
    }
}

}  // namespace csdr
