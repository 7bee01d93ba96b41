// fp32 matrix product on the CUDA cores: y[r][t] = sum_c W[r][c] * x[c][t].
//
// Serves the products whose fp32 operands the tensor-core path does not take - dictionaries whose
// atom count is not a multiple of 128 or whose width is not a multiple of 8, and rebuilt weights
// with ragged edges - in the arithmetic they always had (fp32 multiply-add, no 16-bit splits).
#include <cuda_bf16.h>

#include <algorithm>
#include <type_traits>

#include "../internal.hpp"
#include "gemm_simt.hpp"

namespace csdr {

namespace {

// Tile of 64 rows x TOK (16, 32, 64) tokens x 32 columns, 128 threads. Both operands lie in shared memory with
// the columns contiguous (36 floats a row: 16-byte aligned, and eight rows cover the 32 banks), so
// global rows are copied as they are and the inner product runs over pairs of columns on packed
// fp32 multiply-adds; a thread's 8 x 4 results take 12 128-bit reads per 64 packed instructions.
// Two to four stages in flight. The bound is fp32 issue for 64 tokens (37 TFLOP/s at 11001 x 8100 x
// 300, half the units' peak; 24 with the addresses worked out per element) and the weight's bytes for
// 16 (copied four bytes at a time where its width is odd); small products are bound by the launches.
// Measured, whole products: 300 atoms of width 350 at 95 tokens 266 -> 21 us (rebuilt weight and a
// row-a-warp product before), 128 of 2579 at 6 tokens, three members, 441 -> 33 us.
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
    struct {
        const float* W;
        const void* x;
        uint32_t rows, row_off, tile0;   // rows of the member, where they start in the result, its first row tile
    } m[kSimtMembers];
    uint32_t n_members;
    uint32_t rows, cols, n_kb, kb_per_split, n_split;
    uint32_t vec;      // rows of every W start on 16-byte boundaries
    uint32_t w_fresh;  // W is the output of earlier work on the stream
    XView x;           // x.x: see m
    YView y;           // n_split == 1
    float* part;       // [split][rows][tokens] otherwise
};

// A thread's share of the 64 x 32 blocks of W: where its copies come from and go to, fixed but for
// the column. What lies outside the matrix becomes zero.
struct WBlock {
    const float* W;
    const float* src;      // of the first copy at column 0
    uint32_t dst, c, rows_in;
    __device__ __forceinline__ WBlock(const SimtParams& p, const float* w, uint32_t rows, uint32_t row0, uint32_t tid) {
        W = w;
        const uint32_t r = p.vec ? tid >> 3 : tid >> 5;
        c = p.vec ? (tid & 7u) * 4u : tid & 31u;
        src = W + static_cast<size_t>(row0 + r) * p.cols + c;
        dst = (r * kPitch + c) * 4u;
        rows_in = rows > row0 + r ? rows - row0 - r : 0u;         // rows of the matrix from this copy's on
    }
    __device__ __forceinline__ void load(const SimtParams& p, const float* ws, uint32_t c0) const {
        const uint32_t base = smem_u32(ws) + dst;
        const bool col = c0 + c < p.cols;
        if (p.vec) {   // cols is a multiple of four
            constexpr uint32_t step = kThreads / 8u;
#pragma unroll
            for (uint32_t i = 0; i < kRows / step; ++i) {
                const bool in = col && i * step < rows_in;
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(base + i * step * kPitch * 4u),
                             "l"(in ? src + c0 + static_cast<size_t>(i) * step * p.cols : W), "r"(in ? 16u : 0u)
                             : "memory");
            }
        } else {
            constexpr uint32_t step = kThreads / 32u;
#pragma unroll
            for (uint32_t i = 0; i < kRows / step; ++i) {
                const bool in = col && i * step < rows_in;
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(base + i * step * kPitch * 4u),
                             "l"(in ? src + c0 + static_cast<size_t>(i) * step * p.cols : W), "r"(in ? 4u : 0u)
                             : "memory");
            }
        }
    }
};

// A thread's share of the TOK x 32 blocks of the activations: lanes run along whichever of the two
// dimensions is contiguous in memory. fp32 is copied asynchronously like W; bf16 is widened on its
// way through registers.
template <uint32_t TOK, typename X, bool FEATURE_MAJOR>
struct XBlock {
    static constexpr uint32_t N = TOK * kCols / kThreads;
    static constexpr uint32_t step_t = FEATURE_MAJOR ? 0u : kThreads / kCols, step_c = FEATURE_MAJOR ? kThreads / TOK : 0u;
    const X* x;
    const X* src;
    uint32_t t, c, toks_in;
    size_t stride;         // between this thread's elements; col: between neighbouring columns
    size_t col;
    float v[N];
    __device__ __forceinline__ XBlock(const SimtParams& p, const void* from, uint32_t t0, uint32_t tid) {
        x = static_cast<const X*>(from);
        t = FEATURE_MAJOR ? tid % TOK : tid / kCols;
        c = FEATURE_MAJOR ? tid / TOK : tid % kCols;
        const size_t tok = FEATURE_MAJOR ? 1u : p.x.C;
        col = FEATURE_MAJOR ? p.x.Mtotal : 1u;
        src = x + (p.x.b0 + t0 + t) * tok + c * col;
        stride = step_t * tok + step_c * col;
        toks_in = p.x.M > t0 + t ? p.x.M - t0 - t : 0u;
    }
    __device__ __forceinline__ void load(const SimtParams& p, uint32_t c0) {
        const X* at = src + c0 * col;
        const uint32_t cols_in = p.cols > c0 + c ? p.cols - c0 - c : 0u;
#pragma unroll
        for (uint32_t i = 0; i < N; ++i)
            v[i] = i * step_t < toks_in && i * step_c < cols_in ? static_cast<float>(at[i * stride]) : 0.0f;
    }
    __device__ __forceinline__ void load_async(const SimtParams& p, const float* xs, uint32_t c0) const {
        const X* at = src + c0 * col;
        const uint32_t cols_in = p.cols > c0 + c ? p.cols - c0 - c : 0u;
        const uint32_t base = smem_u32(xs) + (t * kPitch + c) * 4u;
#pragma unroll
        for (uint32_t i = 0; i < N; ++i) {
            const bool in = i * step_t < toks_in && i * step_c < cols_in;
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(base + (i * step_t * kPitch + i * step_c) * 4u),
                         "l"(in ? at + i * stride : x), "r"(in ? 4u : 0u)
                         : "memory");
        }
    }
    __device__ __forceinline__ void store(float* xs) const {
#pragma unroll
        for (uint32_t i = 0; i < N; ++i) xs[(t + i * step_t) * kPitch + c + i * step_c] = v[i];
    }
};

template <uint32_t TOK>
constexpr uint32_t stages() { return TOK == 64u ? 2u : TOK == 32u ? 3u : 4u; }   // all that static shared memory holds

// grid (row tiles, token tiles, column ranges). SWAP: lanes run along the rows of W instead of the
// tokens, so that a token-major result leaves in contiguous pieces.
template <uint32_t TOK, bool SWAP, typename X, bool FEATURE_MAJOR>
__global__ void __launch_bounds__(kThreads, 3)
hsdr_gemm_simt_kernel(const __grid_constant__ SimtParams p) {
    constexpr uint32_t NS = stages<TOK>();
    constexpr bool ASYNC_X = sizeof(X) == 4u;
    __shared__ __align__(16) float ws[NS][kRows * kPitch];
    __shared__ __align__(16) float xs[NS][TOK * kPitch];
    constexpr uint32_t A = SWAP ? TOK : kRows, B = SWAP ? kRows : TOK;   // slow and fast dimension of the result
    constexpr uint32_t TB = B >= 32u ? 16u : 8u, TA = kThreads / TB;     // threads along each
    constexpr uint32_t NA = A / TA, NB = B / TB;
    const uint32_t tid = threadIdx.x, tb = tid % TB, ta = tid / TB;
    uint32_t mi = 0;
    for (uint32_t i = 1; i < p.n_members; ++i)
        if (blockIdx.x >= p.m[i].tile0) mi = i;
    const uint32_t rows = p.m[mi].rows, row_off = p.m[mi].row_off;
    const uint32_t row0 = (blockIdx.x - p.m[mi].tile0) * kRows, t0 = blockIdx.y * TOK;
    const uint32_t kb0 = blockIdx.z * p.kb_per_split, kb1 = min(p.n_kb, kb0 + p.kb_per_split);
    unsigned long long acc[NA][NB];
#pragma unroll
    for (uint32_t i = 0; i < NA; ++i)
#pragma unroll
        for (uint32_t j = 0; j < NB; ++j) acc[i][j] = 0ull;
    const WBlock wb(p, p.m[mi].W, rows, row0, tid);
    XBlock<TOK, X, FEATURE_MAJOR> xb(p, p.m[mi].x, t0, tid);
    // a resident weight is no other launch's output; a rebuilt one and the activations may be
    if (p.w_fresh) asm volatile("griddepcontrol.wait;" ::: "memory");
#pragma unroll
    for (uint32_t i = 0; i + 1u < NS; ++i)
        if (kb0 + i < kb1) wb.load(p, ws[i], (kb0 + i) * kCols);
    asm volatile("griddepcontrol.wait;" ::: "memory");
#pragma unroll
    for (uint32_t i = 0; i + 1u < NS; ++i) {   // the first group covers every copy of W so far
        if (ASYNC_X && kb0 + i < kb1) xb.load_async(p, xs[i], (kb0 + i) * kCols);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    if (!ASYNC_X && kb0 < kb1) {
        xb.load(p, kb0 * kCols);
        xb.store(xs[0]);
    }
    uint32_t s = 0;
    for (uint32_t kb = kb0; kb < kb1; ++kb) {
        asm volatile("cp.async.wait_group %0;" ::"n"(static_cast<int>(NS) - 2) : "memory");
        __syncthreads();                       // block kb is here, and block kb - 1 has been read
        const uint32_t next = s + 1u == NS ? 0u : s + 1u, ahead = s == 0u ? NS - 1u : s - 1u;
        if (kb + NS - 1u < kb1) {
            wb.load(p, ws[ahead], (kb + NS - 1u) * kCols);
            if (ASYNC_X) xb.load_async(p, xs[ahead], (kb + NS - 1u) * kCols);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        if (!ASYNC_X && kb + 1u < kb1) xb.load(p, (kb + 1u) * kCols);
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
        if (!ASYNC_X && kb + 1u < kb1) xb.store(xs[next]);
        s = next;
    }
    asm volatile("griddepcontrol.launch_dependents;");
#pragma unroll
    for (uint32_t i = 0; i < NA; ++i)
#pragma unroll
        for (uint32_t j = 0; j < NB; ++j) {
            const uint32_t a = ta + i * TA, b = tb + j * TB;
            const uint32_t in = row0 + (SWAP ? b : a), r = row_off + in, t = t0 + (SWAP ? a : b);
            if (in >= rows || t >= p.x.M) continue;
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

// At most kMostTokens tokens: their tiles are the grid's second dimension.
constexpr uint32_t kMostTokens = 65535u * 64u;

void launch_tokens(csdr_context* ctx, const SimtMember* members, uint32_t n_members, uint32_t rows, uint32_t cols, const XView& x,
                   const YView& y, bool w_fresh) {
    const bool swap = y.layout == CSDR_LAYOUT_TOKEN_MAJOR;
    const uint32_t tok = x.M <= 16u ? 16u : x.M <= 32u ? 32u : 64u;
    SimtParams p{};
    p.rows = rows;
    p.cols = cols;
    p.vec = cols % 4u == 0;
    p.n_members = n_members;
    uint32_t row_tiles = 0;
    for (uint32_t i = 0; i < n_members; ++i) {
        p.m[i] = {members[i].W, members[i].x, members[i].rows, members[i].row_off, row_tiles};
        p.vec = p.vec && (reinterpret_cast<uintptr_t>(members[i].W) & 15u) == 0;
        row_tiles += (members[i].rows + kRows - 1u) / kRows;
    }
    p.w_fresh = w_fresh ? 1u : 0u;
    p.n_kb = (cols + kCols - 1u) / kCols;
    const uint32_t tok_tiles = (x.M + tok - 1u) / tok;
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
        auto pick = [&](auto type, auto fm) {
            using X = decltype(type);
            constexpr bool FM = decltype(fm)::value;
            return tok == 16u ? (swap ? hsdr_gemm_simt_kernel<16, true, X, FM> : hsdr_gemm_simt_kernel<16, false, X, FM>)
                   : tok == 32u ? (swap ? hsdr_gemm_simt_kernel<32, true, X, FM> : hsdr_gemm_simt_kernel<32, false, X, FM>)
                          : (swap ? hsdr_gemm_simt_kernel<64, true, X, FM> : hsdr_gemm_simt_kernel<64, false, X, FM>);
        };
        const bool fm = x.layout == CSDR_LAYOUT_FEATURE_MAJOR;
        auto kern = x.dtype == CSDR_DTYPE_BF16 ? (fm ? pick(__nv_bfloat16{}, std::true_type{}) : pick(__nv_bfloat16{}, std::false_type{}))
                                               : (fm ? pick(float{}, std::true_type{}) : pick(float{}, std::false_type{}));
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

}  // namespace

void launch_gemm_simt(csdr_context* ctx, const float* W, uint32_t rows, uint32_t cols, const XView& x, const YView& y,
                      bool w_fresh) {
    const SimtMember one{W, x.x, rows, 0u};
    launch_gemm_simt_many(ctx, &one, 1, rows, cols, x, y, w_fresh);
}

void launch_gemm_simt_many(csdr_context* ctx, const SimtMember* members, uint32_t n_members, uint32_t rows, uint32_t cols, const XView& x,
                           const YView& y, bool w_fresh) {
    if (rows == 0) return;
    if (n_members == 0 || n_members > kSimtMembers) throw Error(CSDR_ERR_LIMIT, "fp32 product: 1 to 16 members");
    for (uint64_t t = 0; t < x.M; t += kMostTokens) {
        XView xt = x;
        YView yt = y;
        xt.b0 += static_cast<uint32_t>(t);
        yt.b0 += static_cast<uint32_t>(t);
        xt.M = yt.M = static_cast<uint32_t>(std::min<uint64_t>(kMostTokens, x.M - t));
        launch_tokens(ctx, members, n_members, rows, cols, xt, yt, w_fresh);
    }
}

}  // namespace csdr
