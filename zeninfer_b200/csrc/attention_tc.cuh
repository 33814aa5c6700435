// Causal grouped-query attention for a block of new tokens on the tensor cores, heads of 128 values (attention.cuh has the form for
// other sizes, and the arithmetic's references).
//
// fp32 throughout, by splitting: a float is the exact sum of three bfloat16 values (its 24 mantissa bits, eight at a time, by
// truncation), so a product of two floats is six products of bfloat16 values (the three left out are below 2^-21 of it together, and of its
// sign), each exact in the fp32 accumulator.  Six bf16 products run at 270 TFLOP/s where fp32 multiply-adds run at 70, and they leave the issue slots
// to the softmax, which with the fp32 form waits behind them.
//
// A CTA takes 128 rows: 128 / group consecutive tokens times the query heads of one KV head, so that keys and values serve the whole
// group.  It walks the keys 64 at a time.  Sixteen warps:
//   8 rows      a thread is half a row (32 keys of a block, 64 columns of the output): scores from TMEM, mask, running maximum (shared
//               with the other half), exponentials, P in three planes back to TMEM, from where the tensor cores read it as their A
//               operand; then out = out * factor + O' of the block before, in fp32 registers
//   4 + 3       read the next keys and values (fp32, from L2, asked for a block ahead) and store their three planes in shared memory in
//               the operands' 128-byte swizzle, the values transposed (both operands are then K-major)
//   1 issues    S = Q K^T into four accumulators, because the tensor core truncates a sum at every 16 columns: the leading products of
//               three parts of the head, and all the corrections; the rows add them up in fp32.  O' = P V, corrections first
// The scores of block j + 1 are formed while block j is exponentiated (a block leaves TMEM before anything else); keys and values
// have one buffer each in shared memory (Q's planes take 96 KB of the 192), refilled while the other one's product runs.
//
// Rows whose output is not finite are formed once more with fp32 multiply-adds at the end, over the positions they attend alone: the
// products multiply every value of a block by every row's weights, zeros among them, so that an infinite or NaN value would reach
// rows of the tile that do not attend it.
//
// What bounds it: a block's chain through the row warps, about 6 us a block of 64 keys, of which the exponentials are a third; the
// tensor pipe (72 products a block) is busy for a third of that, memory hardly at all.  The row warps have 128 registers, of which 64 hold
// the output and 32 the scores: 160 bytes a thread are spilled (244 with windows).  B200, 512 tokens, 32 heads on 8, at position 0 /
// 1488: 54 / 190 us, with fp32 multiply-adds on the CUDA cores 142 / 551; error against 64 bits (2-norm, unit normal inputs) 2.0e-7 /
// 2.9e-7, before 2.1e-7 / 7.5e-7.  Five tokens at position 1500: 95 us, before 301.  The host does not know the position: all sizes of
// these heads come here, and a tile of few keys leaves the tensor cores aside (attention_tc_few).
#pragma once
#include <cuda_bf16.h>

#include <algorithm>

#include "attention.cuh"

namespace zk {

constexpr uint32_t kTcRows = 128, kTcKeys = 64, kTcDim = 128;
constexpr uint32_t kTcFewKeys = 128, kTcFewCtas = 24;
constexpr uint32_t kTcKeyWarp = 8, kTcValueWarp = 12, kTcIssueWarp = 15, kTcThreads = 16 * 32;       // first warps of the roles
constexpr uint32_t kTcQPlane = kTcRows * kTcDim * 2, kTcKPlane = kTcKeys * kTcDim * 2, kTcVPlane = kTcDim * kTcKeys * 2;
constexpr uint32_t kTcSmem = 1024 + 3 * (kTcQPlane + kTcKPlane + kTcVPlane) + 4 * kTcRows * 4 + 2 * kTcRows * 8 + 128;
// TMEM columns: leading scores of three parts of the head, corrections; three planes of P; O'
constexpr uint32_t kTcCorrections = 3 * kTcKeys, kTcP = 256, kTcOut = 384, kTcColumns = 512;

// x = plane 0 + plane 1 + plane 2, exactly, as the upper halves of the returned words; where x is infinite plane 0 says so and the
// others are NaN.
__device__ __forceinline__ void split3(float x, uint32_t& a, uint32_t& b, uint32_t& c) {
    a = __float_as_uint(x);
    const float r = x - __uint_as_float(a & 0xffff0000u);
    b = __float_as_uint(r);
    c = __float_as_uint(r - __uint_as_float(b & 0xffff0000u));
}
__device__ __forceinline__ uint32_t upper_halves(uint32_t lo, uint32_t hi) { return __byte_perm(lo, hi, 0x7632); }
// Eight values as sixteen bytes of each plane.
__device__ __forceinline__ void split3_8(const float (&x)[8], uint4 (&plane)[3]) {
    uint32_t w[3][8];
#pragma unroll
    for (int i = 0; i < 8; ++i) split3(x[i], w[0][i], w[1][i], w[2][i]);
#pragma unroll
    for (int p = 0; p < 3; ++p)
        plane[p] = make_uint4(upper_halves(w[p][0], w[p][1]), upper_halves(w[p][2], w[p][3]), upper_halves(w[p][4], w[p][5]), upper_halves(w[p][6], w[p][7]));
}
// D[tmem] (+)= A[tmem] * B[smem], bf16 x bf16 -> fp32; A: a row per lane, two columns of K per 32-bit word.
__device__ __forceinline__ void tc_mma_f16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{ .reg .pred p; setp.ne.b32 p, %4, 0; tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p; }"
        ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
// 32 lanes x 8 consecutive 32-bit columns to and from 8 registers per thread.
__device__ __forceinline__ void tmem_ld_32x8(uint32_t taddr, uint32_t (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_st_32x8(uint32_t taddr, const uint32_t (&r)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void async_proxy_fence() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ bool warp_waited(uint64_t* bar, uint32_t parity) { return __all_sync(0xffffffffu, mbar_wait(bar, parity)); }

// Blocks this kernel takes: their grid, or 0.
inline size_t attention_tc_ctas(size_t head_dim, size_t tokens, size_t heads, size_t kv_heads) {
    const size_t group = heads / kv_heads;
    if (head_dim != kTcDim || group > kTcRows || kTcRows % group) return 0;
    const size_t tile_tokens = kTcRows / group;
    return (tokens + tile_tokens - 1) / tile_tokens * kv_heads;
}

// Whether a tile of so many rows and keys, in `parts` CTAs, goes without the tensor cores: a warp then takes a row at a time, about 0.7 us
// for eight keys while a CTA has eight rows at most, twice that with sixteen (its loads queue); the tensor cores take 9 us for the
// first block of 64 keys and 4 for the next, whatever the rows.  B200, us, few keys / tensor cores / the fp32 kernel for other heads:
// 5 tokens at position 0, 32 heads on 8: 6.0 / 9.7 / 6.2; 33 tokens at 0 / 80: 6.0 / 13.1 / 9.9 and 16.0 / 17.6 / 26.3; 16 tokens of 32
// heads on 32 (sixteen rows a CTA) at 0 / 40 / 100: 4.4 / 10.0 / 5.1, 9.8 / 10.4 / 12.2 and 17.8 / 14.7 / 23.5.
__host__ __device__ inline bool attention_tc_few(uint32_t rows, uint32_t keys, uint32_t parts) {
    const uint32_t turns = (rows + 8 * parts - 1) / (8 * parts);               // of eight warps
    return turns <= 2 ? keys <= kTcFewKeys / 4 * (5 - turns) : static_cast<uint64_t>(keys) * turns <= kTcFewKeys;
}

// CTAs per tile (the grid's y): more than one where the last tile may have few keys, as many as leave a CTA four rows, on SMs that
// would have no tile.  Where such a call then takes the tensor cores, the CTAs that leave at once cost it 0.3 to 0.6 us (12 to 25 us
// calls); with 32 tiles and four parts, calls back to back took 90 us instead of 70 (16 tokens at 1000), so beyond 24 tiles there are none.
inline unsigned attention_tc_parts(size_t ctas, size_t tokens, size_t heads, size_t kv_heads, int sms) {
    if (tokens > kTcFewKeys || ctas > kTcFewCtas) return 1;
    const uint32_t rows = static_cast<uint32_t>(std::min<size_t>(kTcRows, tokens * (heads / kv_heads)));
    const uint32_t parts = std::min((rows + 3) / 4, static_cast<uint32_t>(sms / ctas));
    return parts > 1 && attention_tc_few(rows, static_cast<uint32_t>(tokens), parts) ? parts : 1;
}

// Arguments as attention_prefill_kernel's.  heads / kv_heads divides 128; grid: token tiles x kv_heads, the last tokens' tiles first,
// times attention_tc_parts.
template <bool kWindowed>
__global__ void __launch_bounds__(kTcThreads, 1) attention_prefill_tc_kernel(const float* __restrict__ q, const float* __restrict__ k_cache,
                                                                              const float* __restrict__ v_cache, const int* __restrict__ pos_ptr,
                                                                              float* __restrict__ out, uint32_t tokens, uint32_t heads, uint32_t kv_heads,
                                                                              float scale, uint32_t window, uint32_t max_positions, int* error_word, AttnWindow win) {
    extern __shared__ uint8_t tc_smem_raw[];
    uint8_t* const smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(tc_smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    uint8_t* const q_smem = smem;                             // [plane][half of the head][128 rows][128 bytes]
    uint8_t* const k_smem = q_smem + 3 * kTcQPlane;           // [plane][half of the head][64 rows][128 bytes]
    uint8_t* const v_smem = k_smem + 3 * kTcKPlane;           // [plane][128 rows: the head's values][64 keys]
    float* const top = reinterpret_cast<float*>(v_smem + 3 * kTcVPlane);        // [block parity][half][128 rows]: the largest score of half a row
    double* const sum = reinterpret_cast<double*>(top + 4 * kTcRows);           // [half][128 rows]: its share of the denominator
    uint64_t* const k_full = reinterpret_cast<uint64_t*>(sum + 2 * kTcRows);
    uint64_t* const v_full = k_full + 1;
    uint64_t* const s_full = v_full + 1;                      // block j's scores are formed, and its keys no longer read
    uint64_t* const s_empty = s_full + 1;
    uint64_t* const p_full = s_empty + 1;
    uint64_t* const o_full = p_full + 1;                      // block j's O' is formed, and its values and P no longer read
    uint64_t* const o_empty = o_full + 1;
    uint32_t* const tmem_slot = reinterpret_cast<uint32_t*>(o_empty + 1);
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        mbar_init(k_full, kTcValueWarp - kTcKeyWarp); mbar_init(v_full, kTcIssueWarp - kTcValueWarp);
        mbar_init(s_full, 1); mbar_init(s_empty, 8); mbar_init(p_full, 8); mbar_init(o_full, 1); mbar_init(o_empty, 8);
        mbar_fence_init();
    }
    if (warp == kTcIssueWarp && blockIdx.y == 0) tmem_alloc(tmem_slot, kTcColumns);
    const uint32_t group = heads / kv_heads, tile_tokens = kTcRows / group, kw = kv_heads * kTcDim, qw = heads * kTcDim;
    const uint32_t n_tiles = gridDim.x / kv_heads, tile = n_tiles - 1 - blockIdx.x / kv_heads, kh = blockIdx.x % kv_heads;
    const uint32_t t0 = tile * tile_tokens, t_end = min(tokens, t0 + tile_tokens);
    const uint32_t live_rows = (t_end - t0) * group, each = (live_rows + gridDim.y * (kTcThreads / 32) - 1) / (gridDim.y * (kTcThreads / 32));
    pdl_launch_dependents();
    pdl_wait();
    const int pos0 = __ldcg(pos_ptr);
    const bool good = pos0 >= 0 && static_cast<uint64_t>(pos0) + tokens <= max_positions;
    if (!good && threadIdx.x == 0 && blockIdx.x == 0 && blockIdx.y == 0) atomicExch(error_word, kErrBadPosition);

    const uint32_t last_pos = static_cast<uint32_t>(pos0) + t_end - 1;
    const uint32_t first_any = (window && static_cast<uint32_t>(pos0) + t0 + 1 > window) ? static_cast<uint32_t>(pos0) + t0 + 1 - window : 0u;
    const uint32_t kept_end = kWindowed ? min(win.keep_first, first_any) : 0u;      // kept tokens the window of the tile's first token has left behind
    const uint32_t start = kWindowed && kept_end ? 0u : first_any;
    const bool few = good && attention_tc_few(live_rows, last_pos + 1 - first_any + kept_end, gridDim.y);
    if (blockIdx.y && !few) return;
    auto next_block = [&](uint32_t p0) { return kWindowed && p0 < kept_end && p0 + kTcKeys >= kept_end ? first_any : p0 + kTcKeys; };
    auto part_last = [&](uint32_t p0) { return kWindowed && p0 < kept_end ? kept_end - 1 : last_pos; };      // last position of the part a block lies in
    auto gave_up = [&](int code) { if (lane == 0) atomicExch(error_word, code); };

    if (good && !few) {                                       // Q in three planes, all threads; rows past the block are zeros
        for (uint32_t i = threadIdx.x; i < kTcRows * (kTcDim / 8); i += kTcThreads) {
            const uint32_t row = i / (kTcDim / 8), chunk = i % (kTcDim / 8), t = t0 + row / group;
            float x[8] = {};
            if (t < t_end) {
                const float4* src = reinterpret_cast<const float4*>(q + static_cast<size_t>(t) * qw + static_cast<size_t>(kh * group + row % group) * kTcDim + chunk * 8);
                const float4 a = __ldcg(src), b = __ldcg(src + 1);        // the launch before may write them
                x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w; x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
            }
            uint4 plane[3];
            split3_8(x, plane);
            const uint32_t at = (chunk / 8) * (kTcQPlane / 2) + row * 128 + (((chunk % 8) ^ (row & 7)) << 4);
#pragma unroll
            for (int p = 0; p < 3; ++p) *reinterpret_cast<uint4*>(q_smem + p * kTcQPlane + at) = plane[p];
        }
        async_proxy_fence();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = *tmem_slot;                         // (parts other than the first have none and use none)

    uint32_t todo = 0, first_row = 0, lanes_of = 2;           // rows left to this warp below: bits from first_row on; half of the head it stores (2: both)
    // A wait that runs out ends its role's loop, and the others' follow.
    if (!good) {
    } else if (few) {                                         // fp32 multiply-adds alone, the warps of all parts
        first_row = (warp * gridDim.y + blockIdx.y) * each;
        if (first_row < live_rows) todo = (1u << min(each, live_rows - first_row)) - 1u;
    } else if (warp < kTcKeyWarp) {                           // rows
        const uint32_t quad = warp & 3, half = warp >> 2, row = quad * 32 + lane, lane_base = (quad * 32) << 16;
        const uint32_t t = t0 + row / group, h = kh * group + row % group;
        const bool live = t < t_end;
        const uint32_t my_last = static_cast<uint32_t>(pos0) + t;
        const uint32_t my_first = (window && my_last + 1 > window) ? my_last + 1 - window : 0u;
        const float slope = kWindowed && win.biased ? attn_slope(h, heads) : 0.0f;
        constexpr int kMine = kTcKeys / 2;                    // keys of a block
        // the two warps of a row meet; true where one of them has given up
        auto meet = [&](bool failed) {
            uint32_t any;
            asm volatile(
                "{ .reg .pred p, q; setp.ne.u32 q, %3, 0; barrier.red.or.pred p, %1, %2, q; selp.u32 %0, 1, 0, p; }"
                : "=r"(any) : "r"(quad + 1), "r"(64u), "r"(static_cast<uint32_t>(failed)) : "memory");
            return any != 0;
        };
        bool again = false;
        float acc[kTcDim / 2], m = -INFINITY, factor = 0.0f;
        double l = 0.0;
#pragma unroll
        for (int i = 0; i < static_cast<int>(kTcDim / 2); ++i) acc[i] = 0.0f;
        auto take_output = [&]() {                            // acc = acc * factor + O'
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                uint32_t v[2][16];
#pragma unroll
                for (int b = 0; b < 2; ++b) tmem_ld_32x16(tmem + kTcOut + half * (kTcDim / 2) + 32 * c + 16 * b + lane_base, v[b]);
                tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < 32; ++i) acc[32 * c + i] = fmaf(acc[32 * c + i], factor, __uint_as_float(v[i / 16][i % 16]));
            }
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(o_empty);
        };
        bool ok = true;
        uint32_t j = 0;
        for (uint32_t p0 = start; p0 <= last_pos; p0 = next_block(p0), ++j) {
            ok = ok && warp_waited(s_full, j & 1);
            float s[kMine], most = m;
            if (ok) {
                tc_fence_after_sync();
                float nonfinite = 0.0f;
                auto fetch = [&](bool lead_alone) {
#pragma unroll
                    for (int c = 0; c < kMine / 8; ++c) {
                        uint32_t part[4][8];
#pragma unroll
                        for (int i = 0; i < 4; ++i) tmem_ld_32x8(tmem + i * kTcKeys + half * kMine + 8 * c + lane_base, part[i]);
                        tmem_ld_wait();
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            const float lead = __uint_as_float(part[0][i]) + __uint_as_float(part[1][i]) + __uint_as_float(part[2][i]);
                            const bool alone = lead_alone && (__float_as_uint(lead) & 0x7f800000u) == 0x7f800000u;
                            s[8 * c + i] = (alone ? lead : lead + __uint_as_float(part[3][i])) * scale;
                            nonfinite = fmaf(s[8 * c + i], 0.0f, nonfinite);
                        }
                    }
                };
                fetch(false);
                if (__any_sync(0xffffffffu, nonfinite != 0.0f)) fetch(true);    // an infinite product is the sum: its corrections are zeros times infinities
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(s_empty);
                const uint32_t first = p0 + half * kMine, to = min(my_last, part_last(p0));
                if (kWindowed && win.biased) {
                    const float back = static_cast<float>(static_cast<int>(my_last) - static_cast<int>(first));
#pragma unroll
                    for (int i = 0; i < kMine; ++i) s[i] -= slope * (back - static_cast<float>(i));
                }
                if (!__all_sync(0xffffffffu, live && first >= my_first && first + kMine - 1 <= to)) {
#pragma unroll
                    for (int i = 0; i < kMine; ++i) {
                        const uint32_t pos = first + i;
                        if (!live || (pos < my_first && !(kWindowed && pos < win.keep_first)) || pos > to) s[i] = -INFINITY;      // no weight
                    }
                }
                float part[4] = {m, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
                for (int i = 0; i < kMine; ++i) part[i & 3] = fmaxf(part[i & 3], s[i]);
                most = fmaxf(fmaxf(part[0], part[1]), fmaxf(part[2], part[3]));
                top[((j & 1) * 2 + half) * kTcRows + row] = most;
            }
            if (meet(!ok)) { ok = false; break; }
            most = fmaxf(most, top[((j & 1) * 2 + (half ^ 1)) * kTcRows + row]);
            const float f = most > m ? expf(m - most) : 1.0f;                   // exp(-inf) = 0 on the first position
            m = most;
            const float from = m == -INFINITY ? 0.0f : m;                       // nothing seen yet: exp(-inf - 0) = 0
            float part[4] = {};
#pragma unroll
            for (int i = 0; i < kMine; ++i) {
                s[i] = expf(s[i] - from);
                part[i & 3] += s[i];
            }
            l = l * f + (static_cast<double>(part[0] + part[1]) + static_cast<double>(part[2] + part[3]));
            if (j > 0) ok = warp_waited(o_full, (j - 1) & 1);                   // the block before: its output is formed, and P's place free
            if (ok) {
                tc_fence_after_sync();
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    uint32_t plane[3][8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        uint32_t a[3], b[3];
                        split3(s[16 * c + 2 * i], a[0], a[1], a[2]);
                        split3(s[16 * c + 2 * i + 1], b[0], b[1], b[2]);
#pragma unroll
                        for (int p = 0; p < 3; ++p) plane[p][i] = upper_halves(a[p], b[p]);
                    }
#pragma unroll
                    for (int p = 0; p < 3; ++p) tmem_st_32x8(tmem + kTcP + 32 * p + 16 * half + 8 * c + lane_base, plane[p]);
                }
                tmem_st_wait();
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(p_full);
                if (j > 0) take_output();
            }
            factor = f;
        }
        if (ok) ok = warp_waited(o_full, (j - 1) & 1);
        if (ok) { tc_fence_after_sync(); take_output(); }
        sum[half * kTcRows + row] = l;
        if (meet(!ok)) {
            gave_up(kErrTmemWaitTimeout);
        } else if (live) {
            l += sum[(half ^ 1) * kTcRows + row];
            if (!(l > 0.0) || !isfinite(l)) {
                atomicExch(error_word, kErrNonFinite);
            } else {
                const float inv = 1.0f / static_cast<float>(l);
                float nonfinite[4] = {};
#pragma unroll
                for (int i = 0; i < static_cast<int>(kTcDim / 2); ++i) { acc[i] *= inv; nonfinite[i & 3] = fmaf(acc[i], 0.0f, nonfinite[i & 3]); }
                again = (nonfinite[0] + nonfinite[1]) + (nonfinite[2] + nonfinite[3]) != 0.0f;
                float4* dst = reinterpret_cast<float4*>(out + static_cast<size_t>(t) * qw + static_cast<size_t>(h) * kTcDim + half * (kTcDim / 2));
#pragma unroll
                for (int i = 0; i < static_cast<int>(kTcDim / 8); ++i)
                    if (!again) dst[i] = make_float4(acc[4 * i], acc[4 * i + 1], acc[4 * i + 2], acc[4 * i + 3]);
            }
        }
        first_row = quad * 32;
        todo = __ballot_sync(0xffffffffu, again);
        lanes_of = half;
    } else if (warp < kTcValueWarp) {                         // keys: a thread takes eight values of a key at a time
        constexpr uint32_t kId = (kTcValueWarp - kTcKeyWarp) * 32, kItems = kTcKeys * kTcDim / 8, kEach = kItems / kId;
        const uint32_t id = threadIdx.x - kTcKeyWarp * 32;
        const float* const kb = k_cache + static_cast<size_t>(kh) * kTcDim;
        float4 x[kEach][2];
        auto fetch = [&](uint32_t p0, uint32_t item, float4 (&v)[2]) {
            const uint32_t pos = p0 + item / 16;
            const bool in = pos <= part_last(p0);
            const float4* src = reinterpret_cast<const float4*>(kb + static_cast<size_t>(in ? pos : p0) * kw + (item % 16) * 8);
#pragma unroll
            for (int i = 0; i < 2; ++i) v[i] = in ? __ldcg(src + i) : make_float4(0.f, 0.f, 0.f, 0.f);
        };
        auto store = [&](uint32_t item, const float4 (&v)[2]) {
            const uint32_t r = item / 16, chunk = item % 16;
            const float y[8] = {v[0].x, v[0].y, v[0].z, v[0].w, v[1].x, v[1].y, v[1].z, v[1].w};
            uint4 plane[3];
            split3_8(y, plane);
            const uint32_t at = (chunk / 8) * (kTcKPlane / 2) + r * 128 + (((chunk % 8) ^ (r & 7)) << 4);
#pragma unroll
            for (int p = 0; p < 3; ++p) *reinterpret_cast<uint4*>(k_smem + p * kTcKPlane + at) = plane[p];
        };
#pragma unroll
        for (uint32_t i = 0; i < kEach; ++i) fetch(start, id + kId * i, x[i]);
        uint32_t j = 0;
        for (uint32_t p0 = start; p0 <= last_pos; p0 = next_block(p0), ++j) {
            if (j > 0 && !warp_waited(s_full, (j - 1) & 1)) { gave_up(kErrEmptyWaitTimeout); break; }      // the last block's keys are no longer read
#pragma unroll
            for (uint32_t i = 0; i < kEach; ++i) store(id + kId * i, x[i]);
            async_proxy_fence();
            __syncwarp();
            if (lane == 0) mbar_arrive(k_full);
            const uint32_t p1 = next_block(p0);
            if (p1 <= last_pos) {
#pragma unroll
                for (uint32_t i = 0; i < kEach; ++i) fetch(p1, id + kId * i, x[i]);
            }
        }
    } else if (warp < kTcIssueWarp) {                         // values: a thread takes one of the head's 128 for eight keys at a time
        constexpr uint32_t kId = (kTcIssueWarp - kTcValueWarp) * 32, kItems = kTcDim * kTcKeys / 8, kEach = (kItems + kId - 1) / kId, kAhead = kEach / 2;
        const uint32_t id = threadIdx.x - kTcValueWarp * 32;
        const float* const vb = v_cache + static_cast<size_t>(kh) * kTcDim;
        float x[kEach - kAhead][8];
        auto fetch = [&](uint32_t p0, uint32_t item, float (&v)[8]) {
            const uint32_t last = part_last(p0), first = p0 + item / kTcDim * 8;
            const float* src = vb + item % kTcDim;
#pragma unroll
            for (uint32_t i = 0; i < 8; ++i) v[i] = item < kItems && first + i <= last ? __ldcg(src + static_cast<size_t>(first + i) * kw) : 0.0f;
        };
        auto store = [&](uint32_t item, const float (&v)[8]) {
            if (item >= kItems) return;
            const uint32_t d = item % kTcDim;
            uint4 plane[3];
            split3_8(v, plane);
#pragma unroll
            for (int p = 0; p < 3; ++p) *reinterpret_cast<uint4*>(v_smem + p * kTcVPlane + d * 128 + (((item / kTcDim) ^ (d & 7)) << 4)) = plane[p];
        };
#pragma unroll
        for (uint32_t i = 0; i < kAhead; ++i) fetch(start, id + kId * i, x[i]);
        uint32_t j = 0;
        for (uint32_t p0 = start; p0 <= last_pos; p0 = next_block(p0), ++j) {
            if (j > 0 && !warp_waited(o_full, (j - 1) & 1)) { gave_up(kErrEmptyWaitTimeout); break; }      // the last block's values are no longer read
#pragma unroll
            for (uint32_t i = 0; i < kAhead; ++i) store(id + kId * i, x[i]);
#pragma unroll
            for (uint32_t i = kAhead; i < kEach; ++i) fetch(p0, id + kId * i, x[i - kAhead]);
#pragma unroll
            for (uint32_t i = kAhead; i < kEach; ++i) store(id + kId * i, x[i - kAhead]);
            async_proxy_fence();
            __syncwarp();
            if (lane == 0) mbar_arrive(v_full);
            const uint32_t p1 = next_block(p0);
            if (p1 <= last_pos) {
#pragma unroll
                for (uint32_t i = 0; i < kAhead; ++i) fetch(p1, id + kId * i, x[i]);
            }
        }
    } else if (lane == 0) {                                   // the tensor cores
        constexpr uint32_t score_desc = umma_idesc_bf16(kTcRows, kTcKeys), out_desc = umma_idesc_bf16(kTcRows, kTcDim);
        constexpr uint32_t kFirst[6] = {2, 0, 1, 1, 0, 0}, kSecond[6] = {0, 2, 1, 0, 1, 0};      // planes of the two operands, the smallest products first
        const uint64_t q_desc = umma_desc_k_sw128(smem_u32(q_smem)), k_desc = umma_desc_k_sw128(smem_u32(k_smem)), v_desc = umma_desc_k_sw128(smem_u32(v_smem));
        // a descriptor's start address counts 16-byte units; 16 columns of K are two of them
        auto scores = [&]() {
#pragma unroll
            for (int c = 0; c < 6; ++c)
#pragma unroll
                for (uint32_t k = 0; k < 8; ++k)
                    tc_mma_f16(tmem + (c == 5 ? k / 3 * kTcKeys : kTcCorrections), q_desc + ((kFirst[c] * kTcQPlane + (k / 4) * (kTcQPlane / 2)) >> 4) + 2 * (k % 4),
                                  k_desc + ((kSecond[c] * kTcKPlane + (k / 4) * (kTcKPlane / 2)) >> 4) + 2 * (k % 4), score_desc, c == 5 ? k % 3 > 0 : (c | k) > 0);
            tc_commit(s_full);
        };
        bool ok = mbar_wait(k_full, 0);
        if (ok) { tc_fence_after_sync(); scores(); }
        uint32_t j = 0;
        for (uint32_t p0 = start; ok && p0 <= last_pos; ++j) {
            const uint32_t p1 = next_block(p0);
            if (p1 <= last_pos) {
                ok = mbar_wait(k_full, (j + 1) & 1) && mbar_wait(s_empty, j & 1);
                if (!ok) break;
                tc_fence_after_sync();
                scores();
            }
            ok = mbar_wait(v_full, j & 1) && mbar_wait(p_full, j & 1) && (j == 0 || mbar_wait(o_empty, (j - 1) & 1));
            if (!ok) break;
            tc_fence_after_sync();
#pragma unroll
            for (int c = 0; c < 6; ++c)
#pragma unroll
                for (uint32_t k = 0; k < 4; ++k)
                    tc_mma_f16_ts(tmem + kTcOut, tmem + kTcP + 32 * kFirst[c] + 8 * k, v_desc + (kSecond[c] * kTcVPlane >> 4) + 2 * k, out_desc, (c | k) > 0);
            tc_commit(o_full);
            p0 = p1;
        }
        if (!ok) atomicExch(error_word, kErrFullWaitTimeout);
    }
    __syncwarp();
    // Rows with fp32 multiply-adds, one after another, eight keys a round, a lane holding four columns.  Few keys: all rows, since a block's
    // chain above costs more than they do.  Otherwise those with an output that is not finite: the products above multiply every value of
    // a block, by zero where a row does not attend it, and a value's lower planes are NaN where it is infinite; here a row meets the
    // values it attends and no others, each as it is.
    for (; todo; todo &= todo - 1u) {
        const uint32_t row = first_row + __ffs(todo) - 1, t = t0 + row / group, h = kh * group + row % group;
        const uint32_t my_last = static_cast<uint32_t>(pos0) + t, my_first = (window && my_last + 1 > window) ? my_last + 1 - window : 0u;
        const size_t at_row = static_cast<size_t>(t) * qw + static_cast<size_t>(h) * kTcDim + lane * 4;
        float4 x, o = make_float4(0.f, 0.f, 0.f, 0.f);
        if (few) {
            x = __ldcg(reinterpret_cast<const float4*>(q + at_row));
        } else {                                              // out may lie over q: from the planes, exactly, the smallest first
            const uint32_t at = (lane / 16) * (kTcQPlane / 2) + row * 128 + (((lane % 16 / 2) ^ (row & 7)) << 4) + (lane & 1) * 8;
            uint2 plane[3];
#pragma unroll
            for (int p = 0; p < 3; ++p) plane[p] = *reinterpret_cast<const uint2*>(q_smem + p * kTcQPlane + at);
            auto sum3 = [&](auto part) { return part(plane[0]) + (part(plane[1]) + part(plane[2])); };
            x = make_float4(sum3([](uint2 w) { return __uint_as_float(w.x << 16); }), sum3([](uint2 w) { return __uint_as_float(w.x & 0xffff0000u); }),
                            sum3([](uint2 w) { return __uint_as_float(w.y << 16); }), sum3([](uint2 w) { return __uint_as_float(w.y & 0xffff0000u); }));
        }
        const float slope = kWindowed && win.biased ? attn_slope(h, heads) : 0.0f;
        const size_t column = static_cast<size_t>(kh) * kTcDim + lane * 4;
        constexpr uint32_t kRound = 8;                        // a lane keeps key lane / 4 of a round
        float m = -INFINITY;
        double l = 0.0;
        for (uint32_t p0 = start; p0 <= my_last; p0 = kWindowed && p0 < kept_end && p0 + kRound >= kept_end ? first_any : p0 + kRound) {
            const uint32_t last = part_last(p0), pos = p0 + lane / 4;
            const bool attended = pos <= min(my_last, last) && (pos >= my_first || (kWindowed && pos < win.keep_first));
            if (!__any_sync(0xffffffffu, attended)) continue;
            float4 key[kRound], value[kRound];
#pragma unroll
            for (uint32_t k = 0; k < kRound; ++k) {
                const size_t off = static_cast<size_t>(min(p0 + k, last)) * kw + column;
                key[k] = __ldca(reinterpret_cast<const float4*>(k_cache + off));
                value[k] = __ldca(reinterpret_cast<const float4*>(v_cache + off));
            }
            float s[kRound];                                  // summed over the lanes, which at each exchange keep half of the sums they carry
#pragma unroll
            for (uint32_t k = 0; k < kRound; ++k) s[k] = fmaf(x.w, key[k].w, fmaf(x.z, key[k].z, fmaf(x.y, key[k].y, x.x * key[k].x)));
#pragma unroll
            for (int n = kRound / 2; n > 0; n >>= 1) {
                const bool up = lane & (4 * n);
#pragma unroll
                for (int i = 0; i < n; ++i) s[i] = (up ? s[i + n] : s[i]) + __shfl_xor_sync(0xffffffffu, up ? s[i] : s[i + n], 4 * n);
            }
            float score = s[0] + __shfl_xor_sync(0xffffffffu, s[0], 2);
            score = (score + __shfl_xor_sync(0xffffffffu, score, 1)) * scale;
            if (kWindowed) score -= slope * static_cast<float>(static_cast<int>(my_last) - static_cast<int>(pos));
            float most = attended ? fmaxf(m, score) : m;
#pragma unroll
            for (int n = 4; n < 32; n *= 2) most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, n));
            if (most > m) {
                const float f = expf(m - most);               // exp(-inf) = 0 on the first position
                l *= f;
                m = most;
                o.x *= f; o.y *= f; o.z *= f; o.w *= f;
            }
            const float e = attended ? expf(score - (m == -INFINITY ? 0.0f : m)) : -1.0f;      // below zero: not attended
            if (attended) l += e;
#pragma unroll
            for (uint32_t k = 0; k < kRound; ++k) {
                const float p = __shfl_sync(0xffffffffu, e, 4 * k);
                if (p < 0.0f) continue;
                o.x = fmaf(p, value[k].x, o.x); o.y = fmaf(p, value[k].y, o.y); o.z = fmaf(p, value[k].z, o.z); o.w = fmaf(p, value[k].w, o.w);
            }
        }
#pragma unroll
        for (int n = 4; n < 32; n *= 2) l += __shfl_xor_sync(0xffffffffu, l, n);
        if (!(l > 0.0) || !isfinite(l)) {
            atomicExch(error_word, kErrNonFinite);
        } else if (lanes_of > 1 || lane / 16 == lanes_of) {
            const float inv = 1.0f / static_cast<float>(l);
            *reinterpret_cast<float4*>(out + at_row) = make_float4(o.x * inv, o.y * inv, o.z * inv, o.w * inv);
        }
    }
    tc_fence_before_sync();
    __syncthreads();
    if (warp == kTcIssueWarp && blockIdx.y == 0) {
        tc_fence_after_sync();
        tmem_dealloc(tmem, kTcColumns);
    }
}

}  // namespace zk
