// Decode-time matrix-vector products for Q4_0, Q4_K, Q5_K and, below 4096 columns, Q6_K (batch 1..8).
//
// The reference evaluates these formats with fp32 activations: Q4_0 through its generic dequantise-then-dot route
// (src/quant.cpp:1135-1162 over gemv_avx2, kernels/avx2.cpp:16-40), Q6_K through gemv_q6k_avx2 / gemm_q6k_kblk_avx2
// (kernels/avx2.cpp:380-422, :1762-1770), Q4_K and Q5_K through gemv_q4k_q5k_avx2 (kernels/avx2.cpp:329-378; its GPU entry is
// zen::d3d12::gemm_kquant, include/zen/d3d12_backend.h:75).
//
// Decoding every weight to fp32 costs several instructions per weight, more than an SM can issue at HBM speed, and so does dp4a on
// activations in two int8 digits (gate|up of a Llama-3-8B layer in Q4_0: 192 clocks per 32 blocks and scheduler where HBM allows
// 99).  Here the multiply-adds run on the warp-level f16 matrix instruction (m16n8k16, 8.2 clocks a scheduler on a B200):
//   * weights: a code of up to ten bits IS an f16 number, the subnormal code * 2^-24, so a pair of weights costs one AND (high
//     nibbles stay in place and count sixteenfold; their activations are divided by sixteen).  16 rows are the A operand;
//   * activations: x * 2^e, one power of two per 256 columns, as the sum of two f16 numbers (22 bits), two columns of the B operand;
//   * the scales differ per row and block, so a column may collect products of one block only.  One token (not of Q6_K): the four lanes that
//     share a row hold four different blocks, and B's eight columns are two digits of those four blocks, zero wherever column and
//     lane belong to different blocks: a lane reads its weights as 16-byte words and ends up with the sums of its own block.  Two
//     and more tokens: the four lanes hold four words of the same block and the columns are two digits of four tokens;
//   * per block and row the sum is then multiplied by the block's scale in fp32.  Zero points and minimums enter there, times the
//     block's sum of activations.
//       Q4_0 : y += d_w * sum (n - 8) x                 per 32 weights
//       Q6_K : y += d * sc_g * sum (q - 32) x           per 16 weights
//       Q4_K / Q5_K : y += d * sc_g * sum q x  -  dmin * m_g * sum x        per 32 weights
// What is dropped of an activation is below 2^-22 of it, or below 2^-39 (high nibbles: 2^-35) of the largest of its 256 columns: next to
// very much larger activations small ones lose bits that a scale per 32 columns would keep, and below that they vanish.  The
// instruction adds its sixteen products with the bits of fp32 below the exponents' largest sum, and a code of a few bits has the exponent
// of 1024: a product loses what lies below 2^-14 of a code times the largest activation of the sixteen, where int8 digits lose
// up to 2^-13.  Results are 4e-7 to 1.2e-6 from 64 bits at 4096 columns, those of the digits 2.2e-5.
//
// The unpacking (a shift and four ANDs for eight weights, on a pipe that takes one every other clock) and the steps' own instructions
// bound one token, the products from five tokens on, and the operands that every CTA forms first bound small launches; times and
// those of the digits: kq_takes_mma.  Tried and slower: the shift on the multiplier pipe, steps of two units by eight warps.
//
// Weights stream as in gemv_bf16.cuh: one CTA per SM owns a contiguous row slice (the cut of ComputePool::parallel_for,
// src/compute_pool.cpp:104-106), its warps split it by 16-row tiles and 256-column units, and each warp's share arrives by
// cp.async in a ring of its own.  Algorithmic traffic is the raw GGUF size (18 B per Q4_0 block, 210 B per Q6_K super-block,
// 144 / 176 B per Q4_K / Q5_K super-block; the device planes of the last two are 4 bytes per super-block larger, because the 12
// packed bytes of 6-bit scales and minimums are kept unpacked as 16, see repack.cuh).
#pragma once
#include <cuda_fp16.h>

#include "gemv_kq.cuh"  // formats, tasks, row slices

namespace zk {

// kWide 0: one token; 1, 2: up to four or eight tokens (and one of Q6_K).  Sixteen warps hide each other's chains of loads, unpacking and products; five
// and more tokens have twice the products per weight and need more registers than that leaves.
template <int kWide> __host__ __device__ constexpr int kqm_threads() { return kWide == 2 ? 256 : 512; }
constexpr uint32_t kKqUnit = 256;      // columns of a unit: a super-block, or eight Q4_0 blocks
constexpr uint32_t kKqTile = 16;       // rows of a step

// Per format: the planes a row is split into (repack.cuh) and a step's bytes in a warp's ring slot, one behind the other:
//   words   nibbles, codes or ql: per set of four 16-byte chunks and half of the rows 512 bytes
//   high    Q5_K: fifth bits [row][32]; packed Q6_K: qh [row][64]
//   scales  [row][16]: eight f16 (Q4_0), sixteen int8 (Q6_K), eight scales and eight minimums (Q4_K / Q5_K)
//   supers  [row][4]: (d, dmin), or the f16 d and its neighbour (Q6_K)
template <int kFormat> struct KqmFormat;
template <> struct KqmFormat<2> {                    // Q4_0: nibbles [K/2], f16 scales [K/32]
    static constexpr int kPlanes = 2, kSlots = 5, kSets = 2, kSums = 8;
    static constexpr uint32_t kHigh = 0, kSupers = 0;
};
template <> struct KqmFormat<12> {                   // Q4_K: nibbles [K/2], scales|minimums [K/16], (d, dmin) f16 pairs [K/256]
    static constexpr int kPlanes = 3, kSlots = 5, kSets = 2, kSums = 8;
    static constexpr uint32_t kHigh = 0, kSupers = 64;
};
template <> struct KqmFormat<13> {                   // Q5_K: nibbles, fifth bits [K/8], scales|minimums, (d, dmin)
    static constexpr int kPlanes = 4, kSlots = 4, kSets = 2, kSums = 8;
    static constexpr uint32_t kHigh = 512, kSupers = 64;
};
template <> struct KqmFormat<14> {                   // Q6_K: ql [K/2], qh [K/4], int8 sc [K/16], f16 d [K/256]
    static constexpr int kPlanes = 4, kSlots = 3, kSets = 2, kSums = 16;
    static constexpr uint32_t kHigh = 1024, kSupers = 64;
};
template <> struct KqmFormat<kFormatQ6KCodes> {      // codes [K] int8, sc, d
    static constexpr int kPlanes = 3, kSlots = 3, kSets = 4, kSums = 16;
    static constexpr uint32_t kHigh = 0, kSupers = 64;
};
template <int kFormat> constexpr bool kq_is_k45 = kFormat == 12 || kFormat == 13;      // alike but for the fifth bits
template <int kFormat> constexpr bool kq_is_q6 = kFormat == 14 || kFormat == kFormatQ6KCodes;

template <int kFormat> __host__ __device__ constexpr uint32_t kqm_words_bytes() { return KqmFormat<kFormat>::kSets * 1024; }
template <int kFormat> __host__ __device__ constexpr uint32_t kqm_scales_at() { return kqm_words_bytes<kFormat>() + KqmFormat<kFormat>::kHigh; }
template <int kFormat> __host__ __device__ constexpr uint32_t kqm_slot_bytes() { return kqm_scales_at<kFormat>() + 256 + KqmFormat<kFormat>::kSupers; }
// A warp's ring: 70 to 140 KB for all of them.
template <int kFormat, int kWide> __host__ __device__ constexpr int kqm_slots() { return kWide == 2 ? KqmFormat<kFormat>::kSlots : (KqmFormat<kFormat>::kSlots + 1) / 2; }
template <int kFormat, int kWide> __host__ __device__ constexpr uint32_t kqm_ring_bytes() { return kqm_slots<kFormat, kWide>() * (kqm_threads<kWide>() / 32) * kqm_slot_bytes<kFormat>(); }
// Shared memory per (unit, token): the activations as operands, their scale, and their sums by block.
template <int kFormat> __host__ __device__ constexpr uint32_t kqm_unit_bytes() { return 1024 + 4 + 4 * KqmFormat<kFormat>::kSums; }

struct KqmParams {
    KqTask task[kMaxTasks];
    uint32_t ntasks, total_rows;
    const float* x;         // [batch][K] fp32; null with a gather: the vector gathered by the previous launch
    uint32_t K;             // columns, a multiple of the format's block size
    uint32_t tokens, token_magic;   // token_magic: 2^32 / tokens, rounded up; 0 for one token
    uint32_t partials;      // sums that a row is added up from (kqm_partials)
    uint32_t k_split;       // warps that share a tile: a power of two, at most `partials`
    uint32_t pass_units;    // units whose activations are in shared memory at a time
    uint32_t block_rows;    // rows of a slice whose sums are in shared memory at a time: all of it, or whole tiles
    uint32_t sums_ld;       // floats between the sums of two tokens
    uint32_t pitch[kKqMaxPlanes];  // global row pitch of each plane, bytes
    int* error_word;
    PeerGather gather;      // world == 0: outputs go to task[].y only
};

__host__ __device__ inline uint32_t kqm_units(uint32_t K) { return (K + kKqUnit - 1) / kKqUnit; }
// A row is added up from so many sums, of every kqm_partials-th unit each.  The number comes from the columns and the kernel's width
// alone, not from how many warps share a tile: a row's bits then depend neither on the tensors and rows of its launch nor on the
// shard it is in.  As many as warps may share a tile; long rows of several tokens, whose activations take the shared memory, do with eight.
template <int kWide> inline uint32_t kqm_partials(uint32_t units) {
    const uint32_t most = kWide == 2 || (kWide == 1 && units >= 48) ? 8 : 16;
    uint32_t n = 1;
    while (2 * n <= most && 2 * n <= units) n *= 2;
    return n;
}

// 16 or 4 bytes global -> shared.
__device__ __forceinline__ void kq_copy16(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void kq_copy4(uint32_t dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
// 16 rows x 16 columns of A (f16) times 16 x 8 of B, fp32 sums.
__device__ __forceinline__ void kq_mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// The same with zero in front.
__device__ __forceinline__ void kq_mma_first(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.0f));
}
__device__ __forceinline__ float kq_half(uint32_t word, int upper) {
    return __half2float(__ushort_as_half(static_cast<unsigned short>(upper ? word >> 16 : word & 0xffffu)));
}
// Byte k of a word as a float, through 2^23 + byte.
__device__ __forceinline__ float kq_byte(uint32_t word, int k) { return __uint_as_float(__byte_perm(word, 0x4B000000u, 0x7440u | k)) - 8388608.0f; }
__device__ __forceinline__ float kq_signed_byte(uint32_t flipped, int k) {    // of a word whose bytes were XORed with 0x80
    return __uint_as_float(__byte_perm(flipped, 0x4B000000u, 0x7440u | k)) - 8388736.0f;
}
__device__ __forceinline__ uint32_t kq_word(const uint4& v, int i) { return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w; }

// The two operand registers of a word's low or high nibbles (bytes 0 and 2; bytes 1 and 3), with Q5_K's fifth bits.  q5: the word
// of the qh plane shifted so that bit 0 of a byte belongs to the low nibble and bit 1 to the high one.
template <int kFormat> __device__ __forceinline__ uint32_t kq_low(uint32_t w, uint32_t q5) {
    const uint32_t v = w & 0x000f000fu;
    return kFormat == 13 ? v | ((q5 << 4) & 0x00100010u) : v;
}
template <int kFormat> __device__ __forceinline__ uint32_t kq_high(uint32_t w, uint32_t q5) {
    const uint32_t v = w & 0x00f000f0u;
    return kFormat == 13 ? v | ((q5 << 7) & 0x01000100u) : v;
}

// Which products come here: decided by format and columns alone, so that a row has the same arithmetic whatever tokens, tensors and rows
// share its launch and whatever shard it is in (gemv_kq.cuh's digits are 2e-5 away).  A B200, us here and of the digits:
//   one token      Q4_0         Q4_K         Q5_K         Q6_K      two tokens Q4_0   Q6_K       four tokens Q4_0   Q6_K
//   256 x 1024      2.9   2.9    2.9   3.1    3.1   3.4    3.3   3.0    3.5   3.9    3.7   3.7     4.4   6.0    4.5   5.5
//   1024 x 1024     3.3   2.8    3.2   3.1    3.3   3.3    3.6   3.0    3.9   3.9    4.0   3.7     4.6   6.0    4.7   5.6
//   2048 x 2048     3.8   4.1    3.8   4.7    4.1   5.9    4.5   4.6    4.5   4.9    4.9   5.2     5.7   7.4    6.1   6.7
//   8192 x 2048     5.8  10.2    5.9  12.5    7.3  16.8    8.3  12.2    6.8  11.1    8.8  12.6     7.9  16.0    9.8  14.0
//   1536 x 4096     4.4   3.5    4.5   3.9    5.2   4.3    5.6   3.7    5.9   6.2    6.6   5.3     7.8  10.7    8.6   8.7
//   6144 x 4096     7.0   6.3    7.2   7.5    9.2   9.0   10.1   7.3    8.4  11.4   11.2   9.6    10.3  20.0   13.1  15.4
//   28672 x 4096   16.5  19.1   16.6  24.6   23.6  31.4   27.2  23.1   18.7  40.3   28.2  31.9    20.6  73.0   32.3  52.4
//   4096 x 14336   14.8  14.7   14.6  17.0   18.9  21.0   20.4  15.3   18.3  24.3   24.0  20.6
// One token of Q6_K, whose codes are bytes here, costs up to half as much again from 4096 columns on, where the digits' rows arrive in whole
// segments; there Q6_K stays with them for all tokens, at the price of the last column.
inline bool kq_takes_mma(bool q6, uint32_t K) { return !q6 || K < static_cast<uint32_t>(kKqSegElems); }

template <int kFormat, int kWide>
__global__ void __launch_bounds__(kqm_threads<kWide>(), 1) gemv_kq_mma_kernel(const __grid_constant__ KqmParams p) {
    using F = KqmFormat<kFormat>;
    static_assert(kWide || !kq_is_q6<kFormat>, "a column per block of a token is for blocks of 32 weights");
    constexpr int kThreads = kqm_threads<kWide>(), kWarps = kThreads / 32, kSlots = kqm_slots<kFormat, kWide>();
    constexpr bool kK45 = kq_is_k45<kFormat>, kQ6 = kq_is_q6<kFormat>, kCodes = kFormat == kFormatQ6KCodes;
    constexpr uint32_t kSlot = kqm_slot_bytes<kFormat>(), kHighAt = kqm_words_bytes<kFormat>(), kScalesAt = kqm_scales_at<kFormat>(), kSupersAt = kScalesAt + 256;
    constexpr uint32_t kUnitBytes = kCodes ? 256 : 128;                  // of a row's words
    extern __shared__ __align__(128) uint8_t smem[];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;      // g: row of the tile, t: chunk or word
    const uint32_t tokens = kWide ? p.tokens : 1;
    uint8_t* const xop = smem + kqm_ring_bytes<kFormat, kWide>();                // [unit of the pass][1024 * tokens]
    float* const xscale = reinterpret_cast<float*>(xop + static_cast<size_t>(p.pass_units) * tokens * 1024);     // [unit][token]
    float* const xsum = xscale + ((p.pass_units * tokens + 3) & ~3u);                                            // [unit][token][kSums]
    const uint32_t span = p.block_rows, ld = p.sums_ld;
    float* const sums = xsum + p.pass_units * tokens * F::kSums;                                  // [partial][token][row of the block]
    float* const stash = sums + static_cast<size_t>(p.partials) * tokens * ld;                  // gather only: [token][row of the slice]
    uint32_t r_first, r_last;
    cta_row_slice(p.total_rows, blockIdx.x, gridDim.x, r_first, r_last);
    const uint32_t n_mine = r_last - r_first, units = kqm_units(p.K), ks = p.k_split;
    const uint32_t team = warp / ks, part = warp % ks, teams = kWarps / ks;
    pdl_launch_dependents();

    // A warp's steps are (block of rows, pass, unit, task, tile), in this order: a unit's activations stay in its registers while it goes
    // over the rows.  (Read anew for every tile they took 32 of the 117 wavefronts of shared memory a step, where HBM allows 90 clocks.)
    // Rows past the block's end ask for its last row once more; their sums are not used.
    struct Walk {                                                // what is asked for next
        const uint8_t *words, *scales, *supers, *high;           // the lane's place in row 0 of the task, at the unit
        uint32_t ti, r, r_end, u, pass, first;                   // r: the tile's first row in its task; u: the unit in its pass; first: the block's first row, the slice's end behind the last step
    };
    const uint32_t stride = teams * kKqTile;
    auto pass_size = [&](uint32_t pass) { return min(p.pass_units, units - pass * p.pass_units); };
    auto rows_of = [&](uint32_t first, uint32_t ti, uint32_t& r, uint32_t& r_end) {      // the team's first tile of a task in a block; false where it has none
        const KqTask& k = p.task[ti];
        const uint32_t a = max(first, k.first_row) + team * kKqTile, b = min(min(first + span, r_last), k.first_row + k.rows);
        r = a - k.first_row;
        r_end = b - k.first_row;
        return a < b;
    };
    auto enter = [&](Walk& w) {      // from task ti of unit u on
        while (w.first < r_last) {
            if (w.u < pass_size(w.pass)) {
                for (; w.ti < p.ntasks; ++w.ti) {
                    if (!rows_of(w.first, w.ti, w.r, w.r_end)) continue;
                    const KqTask& k = p.task[w.ti];
                    const uint32_t unit = w.pass * p.pass_units + w.u;
                    w.words = k.plane[0] + unit * kUnitBytes + t * 16;
                    w.scales = k.plane[kFormat == 2 ? 1 : F::kPlanes - 2] + unit * 16;
                    if (kFormat != 2) w.supers = k.plane[F::kPlanes - 1] + (kQ6 ? unit >> 1 : unit) * 4;
                    if (kFormat == 13) w.high = k.plane[1] + unit * 32 + (lane & 1) * 16;
                    if (kFormat == 14) w.high = k.plane[1] + unit * 64 + t * 16;
                    return;
                }
                w.u += ks;
            } else {
                w.u = part;
                if (++w.pass * p.pass_units >= units) {
                    w.pass = 0;
                    w.first += min(span, r_last - w.first);
                }
            }
            w.ti = 0;
        }
    };
    auto advance = [&](Walk& w) {
        w.r += stride;
        if (w.r < w.r_end) return;
        ++w.ti;
        enter(w);
    };
    // Lane (g, t) asks for chunks t, t + 4, ... of rows g and g + 8.  Its 16-byte places are permuted within a row so that the reads
    // by words (several tokens) meet no bank conflicts either.
    uint8_t* const ring = smem + warp * kSlots * kSlot;
    const uint32_t place16 = (g * 4 + (t ^ ((g >> 1) & 3))) * 16;
    const uint32_t scales_at = kScalesAt + lane * 16, supers_at = kSupersAt + lane * 4;
    const bool ragged = kFormat == 2 && p.K % kKqUnit != 0;
    auto ask = [&](const Walk& w, int slot) {
        const uint32_t dst = smem_u32(ring) + slot * kSlot, unit = w.pass * p.pass_units + w.u, last = w.r_end - 1;
        const uint8_t* a = w.words + static_cast<uint64_t>(min(w.r + g, last)) * p.pitch[0];
        const uint8_t* b = w.words + static_cast<uint64_t>(min(w.r + g + 8, last)) * p.pitch[0];
#pragma unroll
        for (int i = 0; i < F::kSets; ++i) {
            const uint32_t to = dst + i * 1024 + place16;
            if (kFormat == 2 && ragged) {      // behind the row's last block: zeros, and no address to read at
                const bool real = unit * kKqUnit + i * 128 + t * 32 < p.K;
                copy16_or_zero(to, real ? a + i * 64 : p.task[w.ti].plane[0], real);
                copy16_or_zero(to + 512, real ? b + i * 64 : p.task[w.ti].plane[0], real);
            } else {
                kq_copy16(to, a + i * 64);
                kq_copy16(to + 512, b + i * 64);
            }
        }
        if (kFormat == 13) kq_copy16(dst + kHighAt + lane * 16, w.high + static_cast<uint64_t>(min(w.r + (lane >> 1), last)) * p.pitch[1]);
        if (kFormat == 14) {
            kq_copy16(dst + kHighAt + g * 64 + t * 16, w.high + static_cast<uint64_t>(min(w.r + g, last)) * p.pitch[1]);
            kq_copy16(dst + kHighAt + (g + 8) * 64 + t * 16, w.high + static_cast<uint64_t>(min(w.r + g + 8, last)) * p.pitch[1]);
        }
        if (lane < 16) {
            const uint64_t row = min(w.r + lane, last);
            kq_copy16(dst + scales_at, w.scales + row * p.pitch[kFormat == 2 ? 1 : F::kPlanes - 2]);
            if (kFormat != 2) kq_copy4(dst + supers_at, w.supers + row * p.pitch[F::kPlanes - 1]);
        }
    };
    Walk in{};
    in.u = part;
    in.first = r_first;
    enter(in);
#pragma unroll
    for (int s = 0; s < kSlots; ++s) {
        if (in.first < r_last) { ask(in, s); advance(in); }
        asm volatile("cp.async.commit_group;" ::: "memory");
    }

    pdl_wait();
    // Row-sharded launch (peer_gather.cuh): announce the previous launch, then wait for every rank's; a null x means "what it gathered".
    unsigned long long epoch = 0;
    const float* x_src = p.x;
    bool failed = false;
    if (p.gather.world) {
        if (blockIdx.x == 0 && threadIdx.x == kThreads - 1) gather_publish_pending(p.gather);
        __syncwarp();
        epoch = gather_epoch(p.gather);
        if (!x_src) {   // chained: the other ranks' previous outputs are this launch's input, so they are needed now
            failed = !gather_wait(p.gather, lane, epoch);
            if (failed && lane == 0) atomicExch(p.error_word, kErrPeerWaitTimeout);
            x_src = gather_previous(p.gather, epoch);
        }
        failed = __syncthreads_or(failed);
    }

    // A pass's activations as operands: per unit and token 1024 bytes.  A word's four columns make two registers (bytes 0 and 2,
    // bytes 1 and 3) for each of two digits; nibble formats have those of the high nibbles 8 bytes behind the low ones', byte
    // formats those of the next chunk.
    //   one token:  [set][word][chunk of the set][digit] 16 bytes
    //   several:    [chunk (byte formats: pair of chunks)][token][digit][word] 16 bytes
    auto prepare = [&](uint32_t pass) {
        const uint32_t first = pass * p.pass_units, jobs = pass_size(pass) * tokens;
        constexpr int kAtOnce = 4;
        auto unit_of = [&](uint32_t j) { return kWide && p.token_magic ? __umulhi(j, p.token_magic) : j; };
        for (uint32_t j0 = warp; j0 < jobs; j0 += kWarps * kAtOnce) {
            float4 raw[kAtOnce][2];
#pragma unroll
            for (int i = 0; i < kAtOnce; ++i) {
                const uint32_t j = j0 + i * kWarps, unit = unit_of(j), token = kWide ? j - unit * tokens : 0, column = (first + unit) * kKqUnit + lane * 8;
                const bool live = j < jobs && column < p.K;
                const float4* src = reinterpret_cast<const float4*>(x_src + (live ? static_cast<size_t>(token) * p.K + column : 0));
                raw[i][0] = live ? __ldcg(src) : make_float4(0.f, 0.f, 0.f, 0.f);       // L2: coherent with peers' stores
                raw[i][1] = live ? __ldcg(src + 1) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
            for (int i = 0; i < kAtOnce; ++i) {
                const uint32_t j = j0 + i * kWarps, unit = unit_of(j), token = kWide ? j - unit * tokens : 0;
                if (j >= jobs) break;
                float v[8] = {raw[i][0].x, raw[i][0].y, raw[i][0].z, raw[i][0].w, raw[i][1].x, raw[i][1].y, raw[i][1].z, raw[i][1].w};
                float most = 0.0f;
#pragma unroll
                for (int k = 0; k < 8; ++k) most = fmaxf(most, fabsf(v[k]));
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, o));
                // 2^e with most * 2^e in [2^14, 2^15): below f16's largest number, and a factor 2^29 above its smallest
                const int exponent = max(static_cast<int>(__float_as_uint(most) >> 23), 15);
                const float up = __uint_as_float(static_cast<uint32_t>(most > 0.0f ? 127 + 127 + 14 - exponent : 127) << 23);
                const float down = __uint_as_float(static_cast<uint32_t>(most > 0.0f ? exponent - 14 + 12 : 127 + 12) << 23);     // 2^-e * 2^12
                float sum = 0.0f;
#pragma unroll
                for (int k = 0; k < 8; ++k) { v[k] *= up; sum += v[k]; }
                sum += __shfl_xor_sync(0xffffffffu, sum, 1);
                if (F::kSums == 8) sum += __shfl_xor_sync(0xffffffffu, sum, 2);
                constexpr float kZero = kFormat == 2 ? -8.0f : kQ6 ? -32.0f : 1.0f;      // Q4_K / Q5_K: for the minimums
                constexpr uint32_t kPer = 32 / F::kSums;
                const uint32_t at = unit * tokens + token;
                if (lane % kPer == 0) xsum[at * F::kSums + lane / kPer] = sum * (kZero * 5.9604644775390625e-08f);
                if (lane == 0) xscale[at] = down;
                // the lane's eight columns: words w0 and w0 + 1 of chunk c, in its low or high nibbles
                uint32_t c, w0, upper = 0;
                if (kFormat == 2) { c = lane >> 2; upper = (lane >> 1) & 1; w0 = (lane & 1) * 2; }
                else if (kK45) { c = (lane >> 3) * 2 + ((lane >> 1) & 1); upper = (lane >> 2) & 1; w0 = (lane & 1) * 2; }
                else { c = lane >> 1; w0 = (lane & 1) * 2; }
                const float scale = !kQ6 && upper ? 0.0625f : 1.0f;
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    uint2 big, small;
                    auto digits = [&](float a, float b, uint32_t& hi, uint32_t& lo) {
                        a *= scale;
                        b *= scale;
                        const __half2 h = __floats2half2_rn(a, b);
                        const float2 back = __half22float2(h);
                        const __half2 l = __floats2half2_rn(a - back.x, b - back.y);
                        hi = *reinterpret_cast<const uint32_t*>(&h);
                        lo = *reinterpret_cast<const uint32_t*>(&l);
                    };
                    digits(v[4 * k], v[4 * k + 2], big.x, small.x);
                    digits(v[4 * k + 1], v[4 * k + 3], big.y, small.y);
                    const uint32_t w = w0 + k;
                    uint8_t* dst = xop + static_cast<size_t>(unit) * tokens * 1024;
                    uint32_t step;
                    if (kWide == 0) {
                        dst += ((c >> 2) * 4 + w) * 128 + (c & 3) * 32 + upper * 8;
                        step = 16;
                    } else {
                        dst += ((kQ6 ? c >> 1 : c) * tokens + token) * 128 + w * 16 + (kQ6 ? c & 1 : upper) * 8;
                        step = 64;
                    }
                    *reinterpret_cast<uint2*>(dst) = big;
                    *reinterpret_cast<uint2*>(dst + step) = small;
                }
            }
        }
    };

    constexpr int kN = kWide ? kWide : 1;
    // The unit's operands, by groups of four tokens; what they are of, see prepare.  One token: what zero points and minimums subtract,
    // for the lane's blocks.  Several: the same in shared memory.
    uint4 x[kN][8];
    float down[kN], begin[2];
    const float* xs[kN];
    auto take = [&](uint32_t u) {
#pragma unroll
        for (int n = 0; n < kN; ++n) {
            const uint32_t column = kWide ? n * 4 + (g >> 1) : 0, token = kWide ? min(n * 4 + t, tokens - 1) : 0;      // of B, and of the lane's results
            const uint8_t* from = xop + u * tokens * 1024 + (kWide ? column * 128 + (g & 1) * 64 + t * 16 : t * 32 + (g & 1) * 16);
#pragma unroll
            for (int i = 0; i < 8; ++i) {      // one token: the column belongs to the lane's block, in one of the sets for Q4_K / Q5_K
                const bool own = kWide ? column < tokens : kK45 ? (g >> 2) == static_cast<uint32_t>(i >> 2) && ((g >> 1) & 1) == (t >> 1) : (g >> 1) == t;
                x[n][i] = own ? *reinterpret_cast<const uint4*>(from + i * tokens * 128) : make_uint4(0, 0, 0, 0);
            }
            xs[n] = xsum + (u * tokens + token) * F::kSums;
            down[n] = xscale[u * tokens + token];
        }
        if constexpr (kWide == 0) {
            begin[0] = xs[0][kK45 ? 2 * t : t];
            begin[1] = xs[0][kK45 ? 2 * t + 1 : 4 + t];
        }
    };

    // ---- one token: the lane's sums over its own blocks, of rows g and g + 8 ----
    auto consume_one = [&](const uint8_t* st, float (&row)[2]) {
        uint4 words[2][2], high[2];
#pragma unroll
        for (int s = 0; s < 2; ++s)
#pragma unroll
            for (int h = 0; h < 2; ++h) words[s][h] = *reinterpret_cast<const uint4*>(st + (s * 2 + h) * 512 + place16);
        if (kFormat == 13)
#pragma unroll
            for (int h = 0; h < 2; ++h) high[h] = *reinterpret_cast<const uint4*>(st + kHighAt + (g + 8 * h) * 32 + (t & 1) * 16);
        float low[2][4], upp[2][4];      // K45: [0] alone, its columns are both sets' sub-blocks
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            float (&lo)[4] = low[kK45 ? 0 : s];
            float (&up)[4] = upp[kK45 ? 0 : s];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const uint4& b = x[0][s * 4 + k];
                const uint32_t w0 = kq_word(words[s][0], k), w1 = kq_word(words[s][1], k), v0 = w0 >> 8, v1 = w1 >> 8;
                uint32_t q0 = 0, q1 = 0;
                if (kFormat == 13) { q0 = kq_word(high[0], k) >> (4 * s + 2 * (t >> 1)); q1 = kq_word(high[1], k) >> (4 * s + 2 * (t >> 1)); }
                const uint32_t al[4] = {kq_low<kFormat>(w0, q0), kq_low<kFormat>(w1, q1), kq_low<kFormat>(v0, q0 >> 8), kq_low<kFormat>(v1, q1 >> 8)};
                const uint32_t au[4] = {kq_high<kFormat>(w0, q0), kq_high<kFormat>(w1, q1), kq_high<kFormat>(v0, q0 >> 8), kq_high<kFormat>(v1, q1 >> 8)};
                if (k == 0 && (s == 0 || !kK45)) {
                    kq_mma_first(lo, al[0], al[1], al[2], al[3], b.x, b.y);
                    kq_mma_first(up, au[0], au[1], au[2], au[3], b.z, b.w);
                } else {
                    kq_mma(lo, al[0], al[1], al[2], al[3], b.x, b.y);
                    kq_mma(up, au[0], au[1], au[2], au[3], b.z, b.w);
                }
            }
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint8_t* sc = st + kScalesAt + (g + 8 * h) * 16;
            if (kFormat == 2) {      // blocks t and t + 4
                const float d0 = __half2float(*reinterpret_cast<const __half*>(sc + t * 2)), d1 = __half2float(*reinterpret_cast<const __half*>(sc + 8 + t * 2));
                row[h] = d0 * (((low[0][2 * h] + low[0][2 * h + 1]) + (upp[0][2 * h] + upp[0][2 * h + 1])) + begin[0]) +
                         d1 * (((low[1][2 * h] + low[1][2 * h + 1]) + (upp[1][2 * h] + upp[1][2 * h + 1])) + begin[1]);
            } else {                 // sub-blocks 2 t and 2 t + 1
                const uint32_t s2 = *reinterpret_cast<const uint16_t*>(sc + t * 2), m2 = *reinterpret_cast<const uint16_t*>(sc + 8 + t * 2);
                const uint32_t dd = *reinterpret_cast<const uint32_t*>(st + kSupersAt + (g + 8 * h) * 4);
                const float pos = fmaf(kq_byte(s2, 0), low[0][2 * h] + low[0][2 * h + 1], kq_byte(s2, 1) * (upp[0][2 * h] + upp[0][2 * h + 1]));
                const float neg = fmaf(kq_byte(m2, 0), begin[0], kq_byte(m2, 1) * begin[1]);
                row[h] = fmaf(kq_half(dd, 0), pos, -kq_half(dd, 1) * neg);
            }
        }
        // the sums of the four lanes that share the rows
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            row[h] *= down[0];
            row[h] += __shfl_xor_sync(0xffffffffu, row[h], 1);
            row[h] += __shfl_xor_sync(0xffffffffu, row[h], 2);
        }
    };

    // ---- several tokens: the lane's sums are of rows g and g + 8 and tokens t (and t + 4) ----
    auto consume_several = [&](const uint8_t* st, uint32_t unit, float (&acc)[kN][2]) {
        // word t of chunk c of row g + 8 h
        const uint32_t swap = (g >> 1) & 3;
        auto word = [&](int c, int h) { return *reinterpret_cast<const uint32_t*>(st + ((c >> 2) * 2 + h) * 512 + (g * 4 + ((c & 3) ^ swap)) * 16 + t * 4); };
        float row[kN][2];
#pragma unroll
        for (int n = 0; n < kN; ++n) row[n][0] = row[n][1] = 0.0f;
        uint4 sc[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) sc[h] = *reinterpret_cast<const uint4*>(st + kScalesAt + (g + 8 * h) * 16);
        if constexpr (kQ6) {
#pragma unroll
            for (int h = 0; h < 2; ++h) sc[h] = make_uint4(sc[h].x ^ 0x80808080u, sc[h].y ^ 0x80808080u, sc[h].z ^ 0x80808080u, sc[h].w ^ 0x80808080u);
#pragma unroll
            for (int pair = 0; pair < 8; ++pair) {
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    const int grp = 2 * pair + k;
                    uint32_t q[2];
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        if (kCodes) {
                            q[h] = (word(grp, h) & 0x3f3f3f3fu) ^ 0x20202020u;
                        } else {
                            const uint32_t hi = *reinterpret_cast<const uint32_t*>(st + kHighAt + (g + 8 * h) * 64 + ((grp >> 3) * 2 + (grp & 1)) * 16 + t * 4);
                            q[h] = ((word((grp >> 3) * 4 + (grp & 3), h) >> (4 * ((grp >> 2) & 1))) & 0x0f0f0f0fu) | (((hi >> (2 * ((grp >> 1) & 3))) & 0x03030303u) << 4);
                        }
                    }
#pragma unroll
                    for (int n = 0; n < kN; ++n) {
                        const float start = xs[n][grp];
                        float c[4];
                        kq_mma_first(c, q[0] & 0x00ff00ffu, q[1] & 0x00ff00ffu, (q[0] >> 8) & 0x00ff00ffu, (q[1] >> 8) & 0x00ff00ffu, k ? x[n][pair].z : x[n][pair].x, k ? x[n][pair].w : x[n][pair].y);
#pragma unroll
                        for (int h = 0; h < 2; ++h) row[n][h] = fmaf(kq_signed_byte(kq_word(sc[h], grp >> 2), grp & 3), (c[2 * h] + c[2 * h + 1]) + start, row[n][h]);
                    }
                }
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const float d = kq_half(*reinterpret_cast<const uint32_t*>(st + kSupersAt + (g + 8 * h) * 4), unit & 1);
#pragma unroll
                for (int n = 0; n < kN; ++n) acc[n][h] = down[n] * (d * row[n][h]);
            }
        } else if constexpr (kFormat == 2) {
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                const uint32_t w0 = word(c, 0), w1 = word(c, 1), v0 = w0 >> 8, v1 = w1 >> 8;
#pragma unroll
                for (int n = 0; n < kN; ++n) {
                    const uint4& b = x[n][c];
                    const float start = xs[n][c];
                    float s[4];
                    kq_mma_first(s, kq_low<2>(w0, 0), kq_low<2>(w1, 0), kq_low<2>(v0, 0), kq_low<2>(v1, 0), b.x, b.y);
                    kq_mma(s, kq_high<2>(w0, 0), kq_high<2>(w1, 0), kq_high<2>(v0, 0), kq_high<2>(v1, 0), b.z, b.w);
#pragma unroll
                    for (int h = 0; h < 2; ++h) row[n][h] = fmaf(kq_half(kq_word(sc[h], c >> 1), c & 1), (s[2 * h] + s[2 * h + 1]) + start, row[n][h]);
                }
            }
#pragma unroll
            for (int n = 0; n < kN; ++n)
#pragma unroll
                for (int h = 0; h < 2; ++h) acc[n][h] = down[n] * row[n][h];
        } else {
            uint32_t q5[2][2] = {{0, 0}, {0, 0}};      // [half of a sub-block][half of the rows]
            if (kFormat == 13)
#pragma unroll
                for (int l = 0; l < 2; ++l)
#pragma unroll
                    for (int h = 0; h < 2; ++h) q5[l][h] = *reinterpret_cast<const uint32_t*>(st + kHighAt + (g + 8 * h) * 32 + l * 16 + t * 4);
            float neg[kN][2];
#pragma unroll
            for (int n = 0; n < kN; ++n) neg[n][0] = neg[n][1] = 0.0f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {      // sub-blocks 2 j and 2 j + 1
                float low[kN][4], upp[kN][4];
#pragma unroll
                for (int n = 0; n < kN; ++n)
#pragma unroll
                    for (int i = 0; i < 4; ++i) low[n][i] = upp[n][i] = 0.0f;
#pragma unroll
                for (int l = 0; l < 2; ++l) {
                    const uint32_t w0 = word(2 * j + l, 0), w1 = word(2 * j + l, 1), v0 = w0 >> 8, v1 = w1 >> 8, q0 = q5[l][0] >> (2 * j), q1 = q5[l][1] >> (2 * j);
#pragma unroll
                    for (int n = 0; n < kN; ++n) {
                        const uint4& b = x[n][2 * j + l];
                        kq_mma(low[n], kq_low<kFormat>(w0, q0), kq_low<kFormat>(w1, q1), kq_low<kFormat>(v0, q0 >> 8), kq_low<kFormat>(v1, q1 >> 8), b.x, b.y);
                        kq_mma(upp[n], kq_high<kFormat>(w0, q0), kq_high<kFormat>(w1, q1), kq_high<kFormat>(v0, q0 >> 8), kq_high<kFormat>(v1, q1 >> 8), b.z, b.w);
                    }
                }
#pragma unroll
                for (int n = 0; n < kN; ++n) {
                    const float2 x2 = *reinterpret_cast<const float2*>(xs[n] + 2 * j);
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const uint32_t s4 = kq_word(sc[h], j >> 1), m4 = kq_word(sc[h], 2 + (j >> 1));
                        const int k = (j & 1) * 2;
                        row[n][h] = fmaf(kq_byte(s4, k), low[n][2 * h] + low[n][2 * h + 1], row[n][h]);
                        row[n][h] = fmaf(kq_byte(s4, k + 1), upp[n][2 * h] + upp[n][2 * h + 1], row[n][h]);
                        neg[n][h] = fmaf(kq_byte(m4, k), x2.x, neg[n][h]);
                        neg[n][h] = fmaf(kq_byte(m4, k + 1), x2.y, neg[n][h]);
                    }
                }
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint32_t dd = *reinterpret_cast<const uint32_t*>(st + kSupersAt + (g + 8 * h) * 4);
#pragma unroll
                for (int n = 0; n < kN; ++n) acc[n][h] = down[n] * fmaf(kq_half(dd, 0), row[n][h], -kq_half(dd, 1) * neg[n][h]);
            }
        }
    };

    int slot = 0;
    for (uint32_t first = r_first; first < r_last && !failed; first += span) {
        for (uint32_t pass = 0; pass * p.pass_units < units; ++pass) {
            if (pass || first != r_first) __syncthreads();                     // the operands and sums of before have been read
            if (first == r_first || p.pass_units < units) prepare(pass);       // operands of all units stay
            __syncthreads();
            const uint32_t count = pass_size(pass);
            for (uint32_t u = part; u < count; u += ks) {
                take(u);
                const uint32_t unit = pass * p.pass_units + u;
                const bool add = unit >= p.partials;
                for (uint32_t ti = 0; ti < p.ntasks; ++ti) {
                    uint32_t r, r_end;
                    if (!rows_of(first, ti, r, r_end)) continue;
                    const uint32_t token = kWide ? t : 0;
                    float* to = sums + ((unit & (p.partials - 1)) * tokens + token) * ld + (p.task[ti].first_row + r + g - first);
                    for (; r < r_end; r += stride, to += stride) {
                        asm volatile("cp.async.wait_group %0;" ::"n"(kSlots - 1) : "memory");
                        __syncwarp();
                        float v[kN][2];
                        const uint8_t* st = ring + slot * kSlot;
                        if constexpr (kWide == 0) consume_one(st, v[0]);
                        else consume_several(st, unit, v);
                        __syncwarp();                 // every lane has read the slot
                        if (in.first < r_last) { ask(in, slot); advance(in); }
                        asm volatile("cp.async.commit_group;" ::: "memory");
                        if (++slot == kSlots) slot = 0;
                        if (kWide == 0 && t) continue;
                        const uint32_t rows = r_end - r;
#pragma unroll
                        for (int n = 0; n < kN; ++n) {
                            if (kWide && token + 4 * n >= tokens) break;
                            float* sum = to + 4 * n * ld;
                            if (g < rows) *sum = add ? *sum + v[n][0] : v[n][0];
                            if (g + 8 < rows) sum[8] = add ? sum[8] + v[n][1] : v[n][1];
                        }
                    }
                }
            }
        }
        __syncthreads();
        const uint32_t count = min(span, r_last - first);
        for (uint32_t token = 0; token < tokens; ++token) {
            for (uint32_t i = threadIdx.x; i < count; i += kThreads) {
                const uint32_t row = first + i;
                uint32_t ti = 0;
                while (row >= p.task[ti].first_row + p.task[ti].rows) ++ti;
                const KqTask& k = p.task[ti];
                float v = 0.0f;
#pragma unroll 4
                for (uint32_t s = 0; s < p.partials; ++s) v += sums[(s * tokens + token) * ld + i];
                v *= 4096.0f;                     // 2^24 of the weights, 2^12 of which are in the activations' scales
                if (k.y) k.y[static_cast<size_t>(token) * k.rows + (row - k.first_row)] = v;
                if (p.gather.world) stash[token * n_mine + (row - r_first)] = v;
            }
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    if (p.gather.world) {
        __syncthreads();
        // With an input of its own the launch needs the other ranks only now: they must have finished the previous
        // launch (whose reads used the parity about to be overwritten) before anything is stored into their regions.
        bool may_push = !failed;
        if (p.x && !gather_wait(p.gather, lane, epoch)) {
            if (lane == 0) atomicExch(p.error_word, kErrPeerWaitTimeout);
            may_push = false;
        }
        if (may_push) gather_push(p.gather, epoch, stash, n_mine, r_first, p.total_rows, tokens, warp, kWarps, lane);
        __syncthreads();
        if (threadIdx.x == 0) gather_finish(p.gather, epoch);
    }
}

}  // namespace zk
