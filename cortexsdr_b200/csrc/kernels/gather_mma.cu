// The gather y[r][t] = sum over the row's codes of +-gamma * Dx[atom][t] as a matrix product on the
// tensor cores (tcgen05), for wide token tiles.
//
// A row's coefficients on the atoms are S * k entries of a row of K; the 128 x 64 blocks of that
// coefficient matrix are put together in shared memory from a re-laid code stream (never stored
// densely), and multiplied with Dx, which stays in shared memory for the CTA's 64 tokens:
//   * the coefficients are sums of stage scales; they are integers times a power of two below 2^8
//     (checked on the host), so bf16 holds them exactly;
//   * Dx arrives as three bf16 planes that add up to the fp32 value to 24 bits. The planes lie side by
//     side as the N = 192 columns of ONE product per 16 atoms, so the coefficient block is read once
//     for all three; their sums meet in the epilogue in fp32.
// hsdr_gather_wide_kernel looks every code up in shared memory instead: S * k * 4 bytes per result,
// 15 us of shared-memory bandwidth for 11008 rows at 512 tokens behind 2.5 us of staging, 28 us
// measured; the products here are 10 us of tensor time behind 3.5 us of planes, 19 us measured (what keeps
// them waiting is the hand-over of coefficient blocks, a barrier each way).
//
// Warp 0 fetches the planes by TMA (one barrier per 64 atoms), warp 1 issues the products, warps 2-5 and
// 6-9 write the even and the odd coefficient blocks into their one of two buffers (a block takes four
// warps about 600 cycles from the release of its buffer, the products of a block 384), warps 10-17 take
// finished 128 x 192 accumulators (two, in tensor memory) out: a lane is a row, so token-major results
// leave in 128-byte pieces.
// A projection that is not finite (an atom that is not, or a sum past fp32) belongs only into the rows
// that name its atom, but a zero coefficient times it is NaN in every row: results that come out not
// finite are worked out once more from the row's codes, as the lookups have them.
// Every wait is bounded; one that runs out sets the status word and every role leaves.
#include <cuda.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>

#include "../internal.hpp"
#include "gather_mma.hpp"

namespace csdr {

namespace {

constexpr uint32_t kGmThreads = 576;
constexpr uint32_t kRowsTile = 128, kTok = 64, kAtomBlock = 64;
constexpr uint32_t kABytes = kRowsTile * 128u;        // one coefficient block
constexpr uint32_t kNCols = 3u * kTok;                // hi | mid | lo
constexpr uint32_t kMaxBlocks = 8;                    // 512 atoms
constexpr uint32_t kMaxSlots = 64;
constexpr uint32_t kHeld = 4;                         // entries a thread keeps of a block (128 threads: 512)

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, uint32_t limit, const volatile int* failed) {
    for (uint32_t i = 0; i < limit; ++i) {
        uint32_t done;
        asm volatile(
            "{\n"
            ".reg .pred p;\n"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
            "selp.u32 %0, 1, 0, p;\n"
            "}\n"
            : "=r"(done)
            : "r"(bar), "r"(parity)
            : "memory");
        if (done) return true;
        if (*failed) return false;
    }
    return false;
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

// Shared-memory descriptors, 128-byte swizzle, as their two halves. Coefficients: atoms (the
// reduction) contiguous, groups of eight rows 1024 B apart. Dx: tokens contiguous, groups of eight
// atoms 1024 B apart (stride) and the next 64 columns - the next plane - `leading` bytes on.
__device__ __forceinline__ uint32_t desc_lo(uint32_t addr, uint32_t leading) {
    return ((addr & 0x3FFFFu) >> 4) | (leading >> 4) << 16;
}
constexpr uint32_t kDescHi = (1024u >> 4) | (1u << 14) | (2u << 29);

// kind::f16: D fp32, A and B bf16, A K-major, B MN-major, M = 128, N = 192.
constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | ((kNCols >> 3) << 17) | ((kRowsTile >> 4) << 24);

// Issued by one lane, with the whole warp going along: descriptors stay in uniform registers and no
// branch stands between the products.
__device__ __forceinline__ void mma(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, bool accumulate, uint32_t leader) {
    asm volatile(
        "{\n"
        ".reg .pred p, q;\n"
        ".reg .b64 a, b;\n"
        "setp.ne.b32 p, %5, 0;\n"
        "setp.ne.b32 q, %6, 0;\n"
        "mov.b64 a, {%1, %4};\n"
        "mov.b64 b, {%2, %4};\n"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, p;\n"
        "}\n" ::"r"(d_tmem),
        "r"(a_lo), "r"(b_lo), "r"(kIdesc), "r"(kDescHi), "r"(static_cast<uint32_t>(accumulate)), "r"(leader)
        : "memory");
}

__device__ __forceinline__ void commit(uint32_t bar, uint32_t leader) {
    asm volatile(
        "{\n"
        ".reg .pred q;\n"
        "setp.ne.b32 q, %1, 0;\n"
        "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n"
        "}\n" ::"r"(bar),
        "r"(leader)
        : "memory");
}

// An entry of a coefficient block: where its bf16 goes (half the byte offset inside the swizzled
// block) above the bf16 itself.
__device__ __forceinline__ uint32_t entry(uint32_t row, uint32_t atom, float v) {
    const uint32_t off = row * 128u + (((atom & (kAtomBlock - 1u)) * 2u) ^ ((row & 7u) << 4));
    const __nv_bfloat16 b = __float2bfloat16_rn(v);
    return (off >> 1) << 16 | *reinterpret_cast<const unsigned short*>(&b);
}

// Code stream -> entries sorted by (row tile, atom block), codes that name an atom twice added up (exactly:
// see exact_in_bf16). CTA = row tile, a thread takes every 1024th code; inside a block's list the order is
// whatever the counters gave, as every entry has a place of its own in the block.
// starts[tile * (blocks + 1) + block]: first entry of a block's list (the last one: its end); a tile's
// lists lie in its own rows-x-slots piece of `entries`.
constexpr uint32_t kEntryThreads = 1024, kCodesEach = kRowsTile * kMaxSlots / kEntryThreads;
__global__ void __launch_bounds__(kEntryThreads)
coefficient_entries_kernel(const uint16_t* __restrict__ codes, const float* __restrict__ scales, uint32_t R, uint32_t S, uint32_t k,
                           uint32_t n_blocks, uint32_t* __restrict__ entries, uint32_t* __restrict__ starts) {
    __shared__ uint16_t code_s[kRowsTile * kMaxSlots];
    __shared__ float scale_s[kMaxSlots];
    __shared__ uint32_t count_s[kMaxBlocks], start_s[kMaxBlocks + 1];
    const uint32_t slots = S * k, tid = threadIdx.x, row0 = blockIdx.x * kRowsTile;
    const uint32_t n = min(kRowsTile, R - row0) * slots;
    for (uint32_t i = tid; i < n; i += kEntryThreads) code_s[i] = codes[static_cast<size_t>(row0) * slots + i];
    if (tid < S) scale_s[tid] = scales[tid];
    if (tid < n_blocks) count_s[tid] = 0;
    __syncthreads();
    uint32_t held[kCodesEach], place[kCodesEach];      // an entry; its block and index there (none: all ones)
#pragma unroll
    for (uint32_t j = 0; j < kCodesEach; ++j) {
        place[j] = 0xFFFFFFFFu;
        const uint32_t i = tid + j * kEntryThreads;
        if (i >= n) continue;
        const uint32_t r = i / slots, s = i - r * slots, a = code_s[i] & 0x7FFFu;
        const uint16_t* row = code_s + r * slots;
        bool first = true;
        for (uint32_t q = 0; q < s; ++q) first = first && (row[q] & 0x7FFFu) != a;
        if (!first) continue;                          // the first code that names an atom stands for all
        float coef = 0.0f;
        for (uint32_t q = s; q < slots; ++q)
            if ((row[q] & 0x7FFFu) == a) coef += (row[q] & 0x8000u) ? -scale_s[q / k] : scale_s[q / k];
        held[j] = entry(r, a, coef);
        place[j] = (a / kAtomBlock) << 16 | atomicAdd(&count_s[a / kAtomBlock], 1u);
    }
    __syncthreads();
    if (tid == 0) {
        start_s[0] = row0 * slots;
        for (uint32_t b = 0; b < n_blocks; ++b) start_s[b + 1u] = start_s[b] + count_s[b];
    }
    __syncthreads();
    if (tid <= n_blocks) starts[blockIdx.x * (n_blocks + 1u) + tid] = start_s[tid];
#pragma unroll
    for (uint32_t j = 0; j < kCodesEach; ++j)
        if (place[j] != 0xFFFFFFFFu) entries[start_s[place[j] >> 16] + (place[j] & 0xFFFFu)] = held[j];
}

struct GatherMmaParams {
    const uint32_t* entries;
    const uint32_t* starts;
    const uint16_t* codes;
    const float* scales;
    const __nv_bfloat16* planes;      // hi | mid | lo, each [K][stride]
    uint32_t stride;
    uint32_t R, S, k, n_tiles, n_blocks, M, per_slice;
    YView y;
    const float* residual;
    TokenScale ts;
    int* status;
    uint32_t spin;
};

// What is not finite among a row's results for n tokens, from the row's codes. Out of the way of the loop
// that leads here.
__device__ __noinline__ void look_up(const GatherMmaParams& p, uint32_t row, uint32_t tok, uint32_t n, float* sum) {
    const size_t plane = static_cast<size_t>(p.n_blocks) * kAtomBlock * p.stride;
    const uint16_t* c = p.codes + static_cast<size_t>(row) * p.S * p.k;
    for (uint32_t j = 0; j < n; ++j) {
        if (isfinite(sum[j])) continue;
        float v = 0.0f;
        for (uint32_t s = 0; s < p.S * p.k; ++s) {
            const uint32_t code = c[s];
            const float gamma = p.scales[s / p.k];
            const __nv_bfloat16* at = p.planes + static_cast<size_t>(code & 0x7FFFu) * p.stride + tok + j;
            float dx = __bfloat162float(at[0]);
            if (isfinite(dx)) dx += __bfloat162float(at[plane]) + __bfloat162float(at[2u * plane]);
            v += __fmul_rn((code & 0x8000u) ? -gamma : gamma, dx);
        }
        sum[j] = v;
    }
}

// grid (per_slice CTAs over the row tiles, 64-token slices)
__global__ void __launch_bounds__(kGmThreads, 1)
hsdr_gather_mma_kernel(const __grid_constant__ CUtensorMap map, const __grid_constant__ GatherMmaParams p) {
    extern __shared__ __align__(1024) unsigned char gm_smem_raw[];
    asm volatile("griddepcontrol.launch_dependents;");
    __shared__ __align__(8) unsigned long long b_full[kMaxBlocks], a_full[2], a_empty[2], acc_full[2], acc_empty[2];
    __shared__ uint32_t tmem_base_s;
    __shared__ volatile int failed_s;
    __shared__ float inv_s[kTok];
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
    unsigned char* smem = reinterpret_cast<unsigned char*>(
        (reinterpret_cast<uintptr_t>(gm_smem_raw) + 1023u) & ~static_cast<uintptr_t>(1023));
    const uint32_t nb = p.n_blocks, plane = nb * kAtomBlock * 128u;
    unsigned char* bs = smem;                              // [plane][atom][64 tokens], swizzled
    unsigned char* as = smem + 3u * plane;                 // two coefficient blocks
    const uint32_t t0 = blockIdx.y * kTok;
    const uint32_t lo = static_cast<uint32_t>(static_cast<uint64_t>(p.n_tiles) * blockIdx.x / p.per_slice);
    const uint32_t hi = static_cast<uint32_t>(static_cast<uint64_t>(p.n_tiles) * (blockIdx.x + 1u) / p.per_slice);
    if (tid == 0) {
        for (uint32_t i = 0; i < kMaxBlocks; ++i) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&b_full[i])));
        for (uint32_t i = 0; i < 2u; ++i) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 4;" ::"r"(smem_u32(&a_full[i])));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&a_empty[i])));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&acc_full[i])));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 8;" ::"r"(smem_u32(&acc_empty[i])));
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        failed_s = 0;
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&tmem_base_s)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    for (uint32_t i = tid; i < 2u * kABytes / 16u; i += kGmThreads) reinterpret_cast<uint4*>(as)[i] = make_uint4(0u, 0u, 0u, 0u);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = tmem_base_s;
    const volatile int* failed = &failed_s;

    if (warp == 0) {
        // ---- Dx: 64 atoms of the three planes per barrier ----
        asm volatile("griddepcontrol.wait;" ::: "memory");
        if (lane == 0)
            for (uint32_t b = 0; b < nb; ++b) {
                const uint32_t bar = smem_u32(&b_full[b]);
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(3u * kAtomBlock * 128u) : "memory");
                for (uint32_t q = 0; q < 3u; ++q)
                    asm volatile(
                        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
                            smem_u32(bs + q * plane + b * kAtomBlock * 128u)),
                        "l"(reinterpret_cast<uint64_t>(&map)), "r"(t0), "r"((q * nb + b) * kAtomBlock), "r"(bar)
                        : "memory");
            }
    } else if (warp == 1) {
        // ---- products ----
        // This warp's instructions are on the critical path (a block's products take 384 cycles):
        // descriptors are additions, and the planes' barriers are only looked at in the first tile.
        bool ok = true;
        const uint32_t leader = lane == 0u ? 1u : 0u;
        const uint32_t a_lo[2] = {desc_lo(smem_u32(as), 16u), desc_lo(smem_u32(as + kABytes), 16u)};
        const uint32_t b_lo0 = desc_lo(smem_u32(bs), plane);
        const uint32_t full[2] = {smem_u32(&a_full[0]), smem_u32(&a_full[1])}, empty[2] = {smem_u32(&a_empty[0]), smem_u32(&a_empty[1])};
        uint32_t phase = 0;                                // of both buffers: nb is even
        for (uint32_t ti = 0; ti < hi - lo && ok; ++ti) {
            const uint32_t acc = ti & 1u, d = tmem_base + acc * 256u;
            if (ti >= 2u) ok = __all_sync(0xFFFFFFFFu, mbar_wait(smem_u32(&acc_empty[acc]), (ti / 2u - 1u) & 1u, p.spin, failed));
            uint32_t b_lo = b_lo0;
            for (uint32_t b = 0; b < nb && ok; b += 2u, phase ^= 1u) {
#pragma unroll
                for (uint32_t h = 0; h < 2u; ++h) {
                    if (ti == 0u) ok = ok && mbar_wait(smem_u32(&b_full[b + h]), 0u, p.spin, failed);
                    ok = __all_sync(0xFFFFFFFFu, ok && mbar_wait(full[h], phase, p.spin, failed));
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                    for (uint32_t q = 0; q < kAtomBlock / 16u; ++q)   // 16 atoms: 32 bytes of a coefficient row, 16 rows of Dx
                        mma(d, a_lo[h] + q * (32u >> 4), b_lo + q * (2048u >> 4), (b | h | q) != 0u, leader);
                    commit(empty[h], leader);
                    b_lo += kAtomBlock * 128u >> 4;
                }
            }
            ok = __all_sync(0xFFFFFFFFu, ok);
            if (ok) commit(smem_u32(&acc_full[acc]), leader);
        }
        if (!ok) failed_s = 1;
    } else if (warp < 10) {
        // ---- coefficient blocks buf, buf + 2, ...: what the last one left is taken back, the next written ----
        const uint32_t buf = warp < 6 ? 0u : 1u, bt = (tid - 64u) & 127u;
        const uint32_t n_g = (hi - lo) * nb;
        unsigned char* a = as + buf * kABytes;
        bool live = true;                                  // after a wait that ran out: barriers only
        // The entries of a block are requested a whole block before their use. A lane holds one of the
        // list starts of the tile being fetched and of the one behind it.
        auto load = [&](const uint32_t* at) {              // volatile: not to be moved to where it is used
            uint32_t v;
            asm volatile("ld.global.nc.u32 %0, [%1];" : "=r"(v) : "l"(at));
            return v;
        };
        auto starts_of = [&](uint32_t tile) { return tile < hi && lane <= nb ? load(p.starts + tile * (nb + 1u) + lane) : 0u; };
        uint32_t f_tile = lo, f_block = buf;               // nb is even: a group stays in its column of blocks
        uint32_t st = starts_of(lo), st_next = starts_of(lo + 1u);
        uint32_t held[kHeld], h_first = 0, h_last = 0, next[kHeld], n_first = 0, n_last = 0;
        auto fetch = [&]() {
            n_first = __shfl_sync(0xFFFFFFFFu, st, f_block);
            n_last = __shfl_sync(0xFFFFFFFFu, st, f_block + 1u);
#pragma unroll
            for (uint32_t j = 0; j < kHeld; ++j) {
                const uint32_t i = n_first + bt + j * 128u;
                next[j] = 0xFFFFFFFFu;
                if (i < n_last) next[j] = load(p.entries + i);
            }
            f_block += 2u;
            if (f_block >= nb) {
                f_block = buf;
                ++f_tile;
                st = st_next;
                st_next = starts_of(f_tile + 1u);
            }
        };
        auto put = [&](uint32_t e, unsigned short v) { *reinterpret_cast<unsigned short*>(a + (e >> 16) * 2u) = v; };
        if (n_g) fetch();
        for (uint32_t g = buf; g < n_g; g += 2u) {
            if (g >= 2u) {
                live = live && __all_sync(0xFFFFFFFFu, mbar_wait(smem_u32(&a_empty[buf]), ((g >> 1) - 1u) & 1u, p.spin, failed));
                if (live) {
#pragma unroll
                    for (uint32_t j = 0; j < kHeld; ++j)
                        if (held[j] != 0xFFFFFFFFu) put(held[j], 0);
                    for (uint32_t i = h_first + bt + kHeld * 128u; i < h_last; i += 128u) put(__ldg(p.entries + i), 0);
                }
                // an entry may fall where another thread of the group took one back
                asm volatile("bar.sync %0, 128;" ::"r"(1u + 2u * buf) : "memory");
            }
            if (!live) continue;
#pragma unroll
            for (uint32_t j = 0; j < kHeld; ++j) {
                held[j] = next[j];
                if (held[j] != 0xFFFFFFFFu) put(held[j], static_cast<unsigned short>(held[j]));
            }
            h_first = n_first;
            h_last = n_last;
            for (uint32_t i = h_first + bt + kHeld * 128u; i < h_last; i += 128u) {
                const uint32_t e = __ldg(p.entries + i);
                put(e, static_cast<unsigned short>(e));
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&a_full[buf]));
            if (g + 2u < n_g) fetch();
        }
        if (!live) failed_s = 1;
    } else {
        // ---- results: two warps a row quarter, 32 tokens each ----
        asm volatile("griddepcontrol.wait;" ::: "memory");
        const uint32_t et = tid - 320u;
        if (et < kTok)
            inv_s[et] = p.ts.sumsq && t0 + et < p.M ? rsqrtf(p.ts.sumsq[t0 + et] * p.ts.inv_width + p.ts.eps) : 1.0f;
        asm volatile("bar.sync 2, 256;" ::: "memory");
        const uint32_t quad = warp & 3u, first = warp < 14u ? 0u : 32u;
        const uint32_t tw = min(kTok, p.M - t0) > first ? min(32u, min(kTok, p.M - t0) - first) : 0u;   // this warp's tokens
        const bool feature = p.y.layout == CSDR_LAYOUT_FEATURE_MAJOR;
        const size_t row_step = feature ? p.y.Mtotal : 1u, tok_step = feature ? 1u : p.y.R;
        uint32_t odd = 0;            // of the warp's two runs of sixteen tokens: some projection is not finite
        for (uint32_t ti = 0; ti < hi - lo; ++ti) {
            const uint32_t acc = ti & 1u;
            if (!__all_sync(0xFFFFFFFFu, mbar_wait(smem_u32(&acc_full[acc]), (ti / 2u) & 1u, p.spin, failed))) {
                failed_s = 1;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t row = (lo + ti) * kRowsTile + quad * 32u + lane;
            const bool in = row < p.R;
            const float bias = in && p.y.bias ? p.y.bias[row] : 0.0f;
            const size_t o0 = row * row_step + (static_cast<size_t>(p.y.b0) + t0 + first) * tok_step;
            float* dst = p.y.y + o0;
            const float* res = p.residual ? p.residual + o0 : nullptr;
            const bool vec = feature && (reinterpret_cast<uintptr_t>(dst) & 15u) == 0 && (reinterpret_cast<uintptr_t>(res) & 15u) == 0;
#pragma unroll
            for (uint32_t ch = 0; ch < 2u; ++ch) {
                if (ch * 16u >= tw) break;
                uint32_t r[3][16];
#pragma unroll
                for (uint32_t q = 0; q < 3u; ++q) {
                    const uint32_t taddr = tmem_base + acc * 256u + q * kTok + first + ((quad * 32u) << 16) + ch * 16u;
                    asm volatile(
                        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
                        : "=r"(r[q][0]), "=r"(r[q][1]), "=r"(r[q][2]), "=r"(r[q][3]), "=r"(r[q][4]), "=r"(r[q][5]), "=r"(r[q][6]),
                          "=r"(r[q][7]), "=r"(r[q][8]), "=r"(r[q][9]), "=r"(r[q][10]), "=r"(r[q][11]), "=r"(r[q][12]), "=r"(r[q][13]),
                          "=r"(r[q][14]), "=r"(r[q][15])
                        : "r"(taddr)
                        : "memory");
                }
                alignas(16) float h[16];
                const uint32_t n = in ? min(16u, tw - ch * 16u) : 0u;
                const bool quads = vec && n == 16u;
                if (res) {
                    if (quads) {
#pragma unroll
                        for (uint32_t j = 0; j < 16u; j += 4u) *reinterpret_cast<float4*>(h + j) = *reinterpret_cast<const float4*>(res + j);
                    } else {
                        const float* at = res;
#pragma unroll
                        for (uint32_t j = 0; j < 16u; ++j, at += tok_step) h[j] = j < n ? *at : 0.0f;
                    }
                    res += 16u * tok_step;
                } else {
#pragma unroll
                    for (uint32_t j = 0; j < 16u; ++j) h[j] = 0.0f;
                }
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (ti == 0u) {
                    // a projection that is not finite leaves NaN in its low plane, so in every row: the first
                    // tile tells for all
                    float all[8];
#pragma unroll
                    for (uint32_t j = 0; j < 8u; ++j) all[j] = __uint_as_float(r[2][j]) + __uint_as_float(r[2][j + 8u]);
#pragma unroll
                    for (uint32_t w = 4u; w > 0u; w >>= 1)
#pragma unroll
                        for (uint32_t j = 0; j < w; ++j) all[j] += all[j + w];
                    if (__any_sync(0xFFFFFFFFu, !isfinite(all[0]))) odd |= 1u << ch;
                }
                if (odd >> ch & 1u) {
                    float again[16];
#pragma unroll
                    for (uint32_t j = 0; j < 16u; ++j)
                        again[j] = __uint_as_float(r[0][j]) + (__uint_as_float(r[1][j]) + __uint_as_float(r[2][j]));
                    look_up(p, row, t0 + first + ch * 16u, n, again);
#pragma unroll
                    for (uint32_t j = 0; j < 16u; ++j) {
                        r[0][j] = __float_as_uint(again[j]);
                        r[1][j] = r[2][j] = 0u;
                    }
                }
#pragma unroll
                for (uint32_t j = 0; j < 16u; ++j)
                    h[j] += fmaf(__uint_as_float(r[0][j]) + (__uint_as_float(r[1][j]) + __uint_as_float(r[2][j])), inv_s[first + ch * 16u + j], bias);
                if (quads) {
#pragma unroll
                    for (uint32_t j = 0; j < 16u; j += 4u) *reinterpret_cast<float4*>(dst + j) = make_float4(h[j], h[j + 1], h[j + 2], h[j + 3]);
                } else if (n == 16u) {
                    float* at = dst;
#pragma unroll
                    for (uint32_t j = 0; j < 16u; ++j, at += tok_step) *at = h[j];
                } else {
                    float* at = dst;
#pragma unroll
                    for (uint32_t j = 0; j < 16u; ++j, at += tok_step)
                        if (j < n) *at = h[j];
                }
                dst += 16u * tok_step;
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&acc_empty[acc]));
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (tid == 0 && failed_s) atomicExch(p.status, 1);
    if (warp == 1) {
        __syncwarp();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem_base) : "memory");
    }
}

// Every coefficient a row can have is u * n with a power of two u and |n| <= 256: exact in bf16.
bool exact_in_bf16(const std::vector<float>& scales, uint32_t k) {
    int unit = 1 << 20;                       // exponent of the lowest bit set in any scale
    for (float g : scales) {
        if (!std::isfinite(g)) return false;
        if (g == 0.0f) continue;
        int e = 0;
        float m = std::frexp(std::fabs(g), &e);              // m in [0.5, 1)
        int bits = 0;
        while (m != std::floor(m)) {
            m *= 2.0f;
            ++bits;
        }
        unit = std::min(unit, e - bits);
    }
    if (unit < -100 || unit > 100) return false;              // far from bf16's limits (also: no scale but zero)
    double sum = 0.0;
    for (float g : scales) sum += static_cast<double>(k) * std::ldexp(std::fabs(static_cast<double>(g)), -unit);
    return sum <= 256.0;
}

using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                              const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                              CUtensorMapFloatOOBfill);

EncodeFn encode_fn() {
    static EncodeFn fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q{};
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess)
            p = nullptr;
        return reinterpret_cast<EncodeFn>(p);
    }();
    return fn;
}

// The segment's entries, built on its first wide product and kept with it (4 bytes a code). False where
// they are missing: under capture, or without room.
bool build_entries(csdr_context* ctx, const csdr_segment* seg) {
    if (seg->coefficients) return true;
    if (ctx->capturing()) return false;
    const Geometry& g = seg->g;
    const uint32_t tiles = (g.rows + kRowsTile - 1u) / kRowsTile, nb = g.n_atoms / kAtomBlock;
    const size_t n_entries = static_cast<size_t>(tiles) * kRowsTile * g.slots();
    const DevPtr buf = ctx->try_keep((n_entries + static_cast<size_t>(tiles) * (nb + 1u)) * 4u);
    if (!buf) return false;
    uint32_t* e = static_cast<uint32_t*>(buf->ptr);
    LaunchScope ls(ctx, KC_GATHER);
    coefficient_entries_kernel<<<tiles, kEntryThreads, 0, ctx->stream>>>(seg->codes_ptr(), static_cast<const float*>(seg->scales->ptr), g.rows,
                                                                         g.n_stages, g.k, nb, e, e + n_entries);
    ls.done("coefficient_entries_kernel");
    buf->built.record(ctx->stream);
    seg->coefficients = buf;
    return true;
}

size_t gather_mma_smem(uint32_t n_atoms) { return 3u * static_cast<size_t>(n_atoms) * 128u + 2u * kABytes + 1024u; }

}  // namespace

bool gather_mma_ready(csdr_context* ctx, const csdr_segment* seg, size_t batch) {
    const Geometry& g = seg->g;
    if (!ctx->gather_mma || !ctx->tensor_cores || !ctx->tma || !encode_fn()) return false;
    if (!g.row_tiles() || g.n_atoms % (2u * kAtomBlock) || g.n_atoms > kMaxBlocks * kAtomBlock || g.slots() > kMaxSlots) return false;
    if (batch <= 16u || batch > 65535u * static_cast<size_t>(kTok)) return false;   // slices: the grid's second dimension
    // A CTA first takes in 384 bytes of planes per atom, and its fixed part has to be shared by enough
    // (row tile, slice) pairs. Whole products, lookups against this: 512 atoms of 4096, 11008 rows, 128
    // tokens 20.2 / 20.7 us, 256 30.1 / 26.7, 512 45.7 / 37.1; 1024 rows, 256 tokens (32 pairs) 19.3 /
    // 19.9, 512 (64 pairs) 23.7 / 23.5; 256 atoms, 2000 rows, 64 tokens 11.7 / 11.7, 128 14.3 / 13.8;
    // 128 atoms, 4096 rows, 128 tokens 13.9 / 11.8.
    const uint64_t pairs = static_cast<uint64_t>((g.rows + kRowsTile - 1u) / kRowsTile) * ((batch + kTok - 1u) / kTok);
    if (ctx->gather_mma_min ? batch < ctx->gather_mma_min
                            : g.n_atoms <= 256u ? batch <= kTok : batch <= 2u * kTok || pairs < 64u)
        return false;
    if (static_cast<uint64_t>((g.rows + kRowsTile - 1u) / kRowsTile) * kRowsTile * g.slots() > 0x7FFFFFFFull) return false;
    if (gather_mma_smem(g.n_atoms) + 1024u > ctx->smem_optin || !exact_in_bf16(seg->scales_host, g.k)) return false;
    return build_entries(ctx, seg);
}

void launch_gather_mma(csdr_context* ctx, const csdr_segment* seg, const DxPlanes& dx, uint32_t M, const YView& y, const float* residual,
                       const TokenScale& ts) {
    const Geometry& g = seg->g;
    GatherMmaParams p{};
    p.entries = static_cast<const uint32_t*>(seg->coefficients->ptr);
    p.starts = p.entries + static_cast<size_t>((g.rows + kRowsTile - 1u) / kRowsTile) * kRowsTile * g.slots();
    p.codes = seg->codes_ptr();
    p.scales = static_cast<const float*>(seg->scales->ptr);
    p.planes = dx.p;
    p.stride = dx.stride;
    p.R = g.rows;
    p.S = g.n_stages;
    p.k = g.k;
    p.n_tiles = (g.rows + kRowsTile - 1u) / kRowsTile;
    p.n_blocks = g.n_atoms / kAtomBlock;
    p.M = M;
    p.y = y;
    p.residual = residual;
    p.ts = ts;
    p.status = ctx->status_word;
    p.spin = ctx->spin_limit_barrier;
    const uint32_t slices = (M + kTok - 1u) / kTok;
    p.per_slice = std::min(p.n_tiles, std::max(1u, static_cast<uint32_t>(ctx->sm_count) / slices));
    CUtensorMap map{};
    const cuuint64_t dims[2] = {M, 3ull * g.n_atoms};
    const cuuint64_t strides[1] = {dx.stride * 2ull};
    const cuuint32_t box[2] = {kTok, kAtomBlock}, estr[2] = {1u, 1u};
    const CUresult rc = encode_fn()(&map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, dx.p, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                    CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (rc != CUDA_SUCCESS) throw Error(CSDR_ERR_CUDA, "cuTensorMapEncodeTiled failed (" + std::to_string(rc) + ")");
    const size_t smem = gather_mma_smem(g.n_atoms);
    ctx->opt_in_smem(reinterpret_cast<const void*>(hsdr_gather_mma_kernel), smem);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(p.per_slice, slices, 1);
    cfg.blockDim = dim3(kGmThreads, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = seg->coefficients->built.read_ahead(ctx) && ctx->pdl ? 1 : 0;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    LaunchScope ls(ctx, KC_GATHER);
    CSDR_CUDA(cudaLaunchKernelEx(&cfg, hsdr_gather_mma_kernel, map, p));
    ls.done("hsdr_gather_mma_kernel");
}

}  // namespace csdr
