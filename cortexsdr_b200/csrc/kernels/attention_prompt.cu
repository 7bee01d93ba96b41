// Causal attention of a prompt: T tokens of ONE sequence at consecutive positions against its cache
// (multi_head_attention, kernels/attention_kernels.cpp:59-113; softmax kernels/simd_kernels.cpp:198-217;
// repeat_kv_heads, api/cortex_sdk.cpp:1453-1478), fp32 scores, weights and sums.
//
// attention_kernel walks the cache once per (token, head), which is right for a decode step; for a
// prompt of T tokens it reads every key T / 2 times through L2 (1024 tokens, 32 heads of 128: 767 us,
// here 263).
// Here a CTA owns 64 query rows of one kv head - rows run over (token, query head of the group), so
// grouped heads share the keys too - and takes 64 keys at a time through shared memory: scores as a
// 64 x 64 tile (4 x 4 a thread, packed fp32 multiply-adds over pairs of columns), an online softmax
// whose rows live in 16 neighbouring lanes, and the weighted sum of the values (4 rows x HD / 16
// columns a thread). Keys and values of a step share one buffer, so two CTAs fit an SM and one loads
// while the other computes. The bound is shared-memory bandwidth
// (77 % of it while the SMs are busy) and fp32 issue.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <cmath>

#include "../internal.hpp"
#include "decoder_ops.hpp"

namespace csdr {

namespace {

constexpr uint32_t kQ = 64, kK = 64, kAttnThreads = 256, kPPitch = kK + 4;
typedef unsigned long long u64;

template <int HD>
constexpr uint32_t pitch() { return HD + 4; }
template <int HD>
constexpr size_t prompt_smem() { return (static_cast<size_t>(kQ + kK) * pitch<HD>() + kQ * kPPitch) * 4u; }

__device__ __forceinline__ u64 fma2(u64 a, u64 b, u64 c) {
    u64 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ u64 mul2(u64 a, u64 b) {
    u64 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ u64 twice(float v) {
    const uint32_t b = __float_as_uint(v);
    return (static_cast<u64>(b) << 32) | b;
}
__device__ __forceinline__ float lo_of(u64 v) { return __uint_as_float(static_cast<uint32_t>(v)); }
__device__ __forceinline__ float hi_of(u64 v) { return __uint_as_float(static_cast<uint32_t>(v >> 32)); }
__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

__device__ __forceinline__ float widen(__nv_bfloat16 v) { return __bfloat162float(v); }
__device__ __forceinline__ float widen(__half v) { return __half2float(v); }

// 64 cache rows into shared memory as fp32; rows from n on become zero. fp32 rows are copied
// asynchronously (the caller waits), 16-bit rows are widened on the way.
template <typename KV, int HD>
__device__ __forceinline__ void load_keys(const KV* src, size_t row, uint32_t n, float* dst, uint32_t tid) {
    constexpr uint32_t V = 16u / sizeof(KV), per = HD / V;
#pragma unroll
    for (uint32_t i = 0; i < kK * per / kAttnThreads; ++i) {
        const uint32_t e = tid + i * kAttnThreads, r = e / per, c = (e % per) * V;
        float* d = dst + r * pitch<HD>() + c;
        if constexpr (sizeof(KV) == 4) {
            const KV* s = r < n ? src + r * row + c : src;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(d))),
                         "l"(s), "r"(r < n ? 16u : 0u)
                         : "memory");
        } else {
            uint4 w = make_uint4(0u, 0u, 0u, 0u);
            if (r < n) w = *reinterpret_cast<const uint4*>(src + r * row + c);
            const KV* h = reinterpret_cast<const KV*>(&w);
#pragma unroll
            for (uint32_t q = 0; q < 8u; q += 4u)
                *reinterpret_cast<float4*>(d + q) = make_float4(widen(h[q]), widen(h[q + 1]), widen(h[q + 2]), widen(h[q + 3]));
        }
    }
}

// grid (kv heads, row blocks): the row blocks with the most keys start first, of every head (with the
// heads on the slow dimension a third of the SMs' time went into the tail: 369 us)
template <typename KV, int HD>
__global__ void __launch_bounds__(kAttnThreads, 2)
attention_prompt_kernel(const float* __restrict__ q, const KV* __restrict__ kc, const KV* __restrict__ vc,
                        const int32_t* __restrict__ seq_of, const int32_t* __restrict__ pos_of, uint32_t T, uint32_t QH, uint32_t KVH,
                        uint32_t max_seq, float qscale, float* __restrict__ out, __nv_bfloat16* __restrict__ hi,
                        __nv_bfloat16* __restrict__ lo) {
    extern __shared__ __align__(16) float psm[];
    constexpr uint32_t P = pitch<HD>(), NH = HD / 64u;     // NH: 64-column halves of a value row
    float* qs = psm;
    float* ks = qs + kQ * P;                               // keys, then the values of the same step
    float* ps = ks + kK * P;
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const uint32_t tid = threadIdx.x, tx = tid & 15u, ty = tid >> 4;
    const uint32_t rep = QH / KVH, rows = T * rep, kvh = blockIdx.x;
    const uint32_t row0 = (gridDim.y - 1u - blockIdx.y) * kQ;
    const int32_t p0 = pos_of[0];
    const size_t krow = static_cast<size_t>(KVH) * HD;
    const size_t base = static_cast<size_t>(seq_of[0]) * max_seq * krow + static_cast<size_t>(kvh) * HD;

    for (uint32_t i = tid; i < kQ * (HD / 4u); i += kAttnThreads) {
        const uint32_t r = i / (HD / 4u), c = (i % (HD / 4u)) * 4u, rr = row0 + r;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (rr < rows) v = *reinterpret_cast<const float4*>(q + (static_cast<size_t>(rr / rep) * QH + kvh * rep + rr % rep) * HD + c);
        *reinterpret_cast<float4*>(qs + r * P + c) = make_float4(v.x * qscale, v.y * qscale, v.z * qscale, v.w * qscale);
    }
    // a row's keys: positions 0 .. limit - 1
    uint32_t limit[4];
#pragma unroll
    for (uint32_t i = 0; i < 4u; ++i) {
        const uint32_t t = min(row0 + ty + 16u * i, rows - 1u) / rep;
        limit[i] = min(static_cast<uint32_t>(p0) + t + 1u, max_seq);
    }
    const uint32_t all = min(static_cast<uint32_t>(p0) + min(row0 + kQ - 1u, rows - 1u) / rep + 1u, max_seq);   // keys of the block's last row
    const uint32_t common = min(static_cast<uint32_t>(p0) + row0 / rep + 1u, max_seq);                          // keys every row sees
    float m[4], l[4];
    u64 acc[4][2 * NH];
#pragma unroll
    for (uint32_t i = 0; i < 4u; ++i) {
        m[i] = -INFINITY;
        l[i] = 0.0f;
#pragma unroll
        for (uint32_t d = 0; d < 2u * NH; ++d) acc[i][d] = 0ull;
    }
    load_keys<KV, HD>(kc + base, krow, min(kK, all), ks, tid);
    for (uint32_t j0 = 0; j0 < all; j0 += kK) {
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        // scores: rows ty + 16 i, keys tx + 16 j
        u64 s2[4][4];
#pragma unroll
        for (uint32_t i = 0; i < 4u; ++i)
#pragma unroll
            for (uint32_t j = 0; j < 4u; ++j) s2[i][j] = 0ull;
#pragma unroll 4
        for (uint32_t c = 0; c < HD; c += 4u) {
            ulonglong2 a[4], b[4];
#pragma unroll
            for (uint32_t i = 0; i < 4u; ++i) a[i] = *reinterpret_cast<const ulonglong2*>(qs + (ty + 16u * i) * P + c);
#pragma unroll
            for (uint32_t j = 0; j < 4u; ++j) b[j] = *reinterpret_cast<const ulonglong2*>(ks + (tx + 16u * j) * P + c);
#pragma unroll
            for (uint32_t i = 0; i < 4u; ++i)
#pragma unroll
                for (uint32_t j = 0; j < 4u; ++j) s2[i][j] = fma2(a[i].y, b[j].y, fma2(a[i].x, b[j].x, s2[i][j]));
        }
        __syncthreads();                                   // the keys have been read: values take their place
        load_keys<KV, HD>(vc + base + static_cast<size_t>(j0) * krow, krow, min(kK, all - j0), ks, tid);
        const bool whole = j0 + kK <= common;              // no row of the block ends inside this step
#pragma unroll
        for (uint32_t i = 0; i < 4u; ++i) {
            float s[4], mx = m[i];
#pragma unroll
            for (uint32_t j = 0; j < 4u; ++j) {
                s[j] = lo_of(s2[i][j]) + hi_of(s2[i][j]);
                if (!whole && j0 + tx + 16u * j >= limit[i]) s[j] = -INFINITY;
                mx = fmaxf(mx, s[j]);
            }
#pragma unroll
            for (int off = 8; off > 0; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, off));
            const float corr = ex2(m[i] - mx);             // 2^-inf = 0 on the first step; key 0 is always valid
            float sum = 0.0f;
#pragma unroll
            for (uint32_t j = 0; j < 4u; ++j) {
                s[j] = ex2(s[j] - mx);
                sum += s[j];
                ps[(ty + 16u * i) * kPPitch + tx + 16u * j] = s[j];
            }
#pragma unroll
            for (int off = 8; off > 0; off >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, off);
            l[i] = fmaf(l[i], corr, sum);
            m[i] = mx;
            const u64 c2 = twice(corr);
#pragma unroll
            for (uint32_t d = 0; d < 2u * NH; ++d) acc[i][d] = mul2(acc[i][d], c2);
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        // values: a thread's columns are 4 tx .. + 3 of every half. Where a row ends inside the step,
        // its masked keys are left out rather than weighted with zero (they may hold anything).
        auto weigh = [&](auto masked, uint32_t k_hi) {
#pragma unroll 2
            for (uint32_t k = 0; k < k_hi; k += 4u) {
                float4 w[4];
#pragma unroll
                for (uint32_t i = 0; i < 4u; ++i) w[i] = *reinterpret_cast<const float4*>(ps + (ty + 16u * i) * kPPitch + k);
#pragma unroll
                for (uint32_t kk = 0; kk < 4u; ++kk) {
                    ulonglong2 v[NH];
#pragma unroll
                    for (uint32_t h = 0; h < NH; ++h)
                        v[h] = *reinterpret_cast<const ulonglong2*>(ks + (k + kk) * P + 64u * h + 4u * tx);
#pragma unroll
                    for (uint32_t i = 0; i < 4u; ++i) {
                        if (decltype(masked)::value && j0 + k + kk >= limit[i]) continue;
                        const u64 w2 = twice(kk == 0u ? w[i].x : kk == 1u ? w[i].y : kk == 2u ? w[i].z : w[i].w);
#pragma unroll
                        for (uint32_t h = 0; h < NH; ++h) {
                            acc[i][2 * h] = fma2(w2, v[h].x, acc[i][2 * h]);
                            acc[i][2 * h + 1] = fma2(w2, v[h].y, acc[i][2 * h + 1]);
                        }
                    }
                }
            }
        };
        if (whole) weigh(std::false_type{}, kK);
        else weigh(std::true_type{}, kK);
        __syncthreads();                                   // the values have been read
        if (j0 + kK < all) load_keys<KV, HD>(kc + base + static_cast<size_t>(j0 + kK) * krow, krow, min(kK, all - j0 - kK), ks, tid);
    }
#pragma unroll
    for (uint32_t i = 0; i < 4u; ++i) {
        const uint32_t rr = row0 + ty + 16u * i;
        if (rr >= rows) continue;
        const float inv = l[i] > 0.0f ? 1.0f / l[i] : 0.0f;
        const size_t o = (static_cast<size_t>(rr / rep) * QH + kvh * rep + rr % rep) * HD + 4u * tx;
#pragma unroll
        for (uint32_t h = 0; h < NH; ++h) {
            const float4 v = make_float4(lo_of(acc[i][2 * h]) * inv, hi_of(acc[i][2 * h]) * inv, lo_of(acc[i][2 * h + 1]) * inv,
                                         hi_of(acc[i][2 * h + 1]) * inv);
            if (hi) {
                const __nv_bfloat162 h0 = __floats2bfloat162_rn(v.x, v.y), h1 = __floats2bfloat162_rn(v.z, v.w);
                const __nv_bfloat162 l0 = __floats2bfloat162_rn(v.x - __low2float(h0), v.y - __high2float(h0));
                const __nv_bfloat162 l1 = __floats2bfloat162_rn(v.z - __low2float(h1), v.w - __high2float(h1));
                *reinterpret_cast<uint2*>(hi + o + 64u * h) = make_uint2(*reinterpret_cast<const uint32_t*>(&h0), *reinterpret_cast<const uint32_t*>(&h1));
                *reinterpret_cast<uint2*>(lo + o + 64u * h) = make_uint2(*reinterpret_cast<const uint32_t*>(&l0), *reinterpret_cast<const uint32_t*>(&l1));
            } else {
                *reinterpret_cast<float4*>(out + o + 64u * h) = v;
            }
        }
    }
}

template <typename KV, int HD>
void launch(csdr_context* ctx, const float* q, const void* kc, const void* vc, const int32_t* seq_of, const int32_t* pos_of, uint32_t T,
            uint32_t QH, uint32_t KVH, uint32_t max_seq, float* out, __nv_bfloat16* hi, __nv_bfloat16* lo) {
    auto kern = attention_prompt_kernel<KV, HD>;
    const size_t smem = prompt_smem<HD>();
    ctx->opt_in_smem(reinterpret_cast<const void*>(kern), smem);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(KVH, (T * (QH / KVH) + kQ - 1u) / kQ, 1);
    cfg.blockDim = dim3(kAttnThreads, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = ctx->pdl ? 1 : 0;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    // scores are kept as log2 of the softmax weights: the query carries scale * log2 e
    const float qscale = 1.0f / sqrtf(static_cast<float>(HD)) * 1.4426950408889634f;
    LaunchScope ls(ctx, KC_ATTENTION);
    CSDR_CUDA(cudaLaunchKernelEx(&cfg, kern, q, static_cast<const KV*>(kc), static_cast<const KV*>(vc), seq_of, pos_of, T, QH, KVH, max_seq,
                                 qscale, out, hi, lo));
    ls.done("attention_prompt_kernel");
}

template <int HD>
void launch_kv(csdr_context* ctx, const float* q, const void* kc, const void* vc, int kv_dtype, const int32_t* seq_of, const int32_t* pos_of,
               uint32_t T, uint32_t QH, uint32_t KVH, uint32_t max_seq, float* out, __nv_bfloat16* hi, __nv_bfloat16* lo) {
    if (kv_dtype == CSDR_DTYPE_BF16) launch<__nv_bfloat16, HD>(ctx, q, kc, vc, seq_of, pos_of, T, QH, KVH, max_seq, out, hi, lo);
    else if (kv_dtype == CSDR_DTYPE_F16) launch<__half, HD>(ctx, q, kc, vc, seq_of, pos_of, T, QH, KVH, max_seq, out, hi, lo);
    else launch<float, HD>(ctx, q, kc, vc, seq_of, pos_of, T, QH, KVH, max_seq, out, hi, lo);
}

}  // namespace

// Short prompts stay with the kernel that has a CTA for every (token, head): at 128 tokens it takes
// 25 us against 29 (32 heads of 128) and 15 against 19 (14 heads of 64), at 256 64 against 48 and 29
// against 29, at 512 214 against 104 and 80 against 50.
// Row blocks are the grid's second dimension: 65535 of 64 (token, query head of a group) rows.
bool attention_prompt_supported(const csdr_context* ctx, uint32_t T, uint32_t QH, uint32_t KVH, uint32_t HD) {
    return (HD == 64u || HD == 128u) && T >= ctx->prompt_attention_min && static_cast<uint64_t>(T) * (QH / KVH) <= 65535ull * kQ;
}

void op_attention_prompt(csdr_context* ctx, const float* q, const void* kc, const void* vc, int kv_dtype, const int32_t* seq_of,
                         const int32_t* pos_of, uint32_t T, uint32_t QH, uint32_t KVH, uint32_t HD, uint32_t max_seq, float* out,
                         __nv_bfloat16* hi, __nv_bfloat16* lo) {
    if (HD == 128u) launch_kv<128>(ctx, q, kc, vc, kv_dtype, seq_of, pos_of, T, QH, KVH, max_seq, out, hi, lo);
    else if (HD == 64u) launch_kv<64>(ctx, q, kc, vc, kv_dtype, seq_of, pos_of, T, QH, KVH, max_seq, out, hi, lo);
    else throw Error(CSDR_ERR_UNSUPPORTED, "prompt attention: head_dim must be 64 or 128");
}

}  // namespace csdr
