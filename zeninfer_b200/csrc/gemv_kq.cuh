// Decode-time matrix-vector products for Q6_K from 4096 columns on (batch 1..8).  Which products come here and which to the matrix
// instructions of gemv_kq_mma.cuh, which has the other small formats: kq_takes_mma there.
//
// The reference evaluates the format with fp32 activations, through gemv_q6k_avx2 / gemm_q6k_kblk_avx2
// (kernels/avx2.cpp:380-422, :1762-1770).  Decoding every weight to fp32 costs several ALU operations per weight, more than an
// SM can issue at HBM speed, so the dot products here stay in integers: weights are used as the small integers they
// are, and each activation enters as two int8 digits, x ~= (d/256) * (256*q1 + q2) with an error
// below d/512 (quantize_acts.cuh).  Results agree with the fp32-activation reference to ~1e-5.
//
//   y += d * sc_g * (d_x/256) * sum (q-32)*(256*q1+q2)                        per 16-weight group
//
// Same streaming skeleton as the Q8_0 kernel (gemv_q8_0.cuh): a persistent CTA per SM owns a
// byte-balanced row slice, a producer warp feeds a ring of shared-memory stages with TMA bulk
// copies, sixteen consumer warps in two teams own one row each.  Algorithmic traffic is the raw
// GGUF size (210 B per super-block).
#pragma once
#include <cuda.h>
#include <cuda_fp16.h>

#include "gemv_q8_0.cuh"

namespace zk {

constexpr int kKqSegElems = 4096;   // weights per row per stage segment (16 super-blocks)
constexpr int kKqMaxPlanes = 4;
constexpr int kKqPartialFloats = kTeams * 2 * kTeamWarps * kTeamWarps;   // [team][unit parity][K slice][row]

// Per-format geometry of the planes a row is split into (repack.cuh).
template <int kFormat> struct KqFormat;

template <> struct KqFormat<14> {  // Q6_K: ql [K/2], qh [K/4], int8 sc [K/16], f16 d [K/256]
    static constexpr int kPlanes = 4;
    static constexpr int kStages = 4;   // a multiple of the team count, see kGemvStages
    __host__ __device__ static constexpr uint32_t seg_bytes(int plane) {
        return plane == 0 ? kKqSegElems / 2 : plane == 1 ? kKqSegElems / 4 : plane == 2 ? kKqSegElems / 16 : kKqSegElems / 256 * 2;
    }
    __host__ __device__ static constexpr uint32_t bytes_per_256(int plane) { return plane == 0 ? 128 : plane == 1 ? 64 : plane == 2 ? 16 : 2; }
};
// Q6_K with the codes unpacked on upload (kFormatQ6KCodes): q - 32 as one int8 per weight in element order, the group
// scales and super-block scales as in the packed layout.  The device copy is 1.07 bytes per weight instead of the file's
// 0.82, and the inner loop loses the 24 shift/mask operations per 16 weights that rebuild a code from ql and qh: the
// packed kernel is bound by instruction issue at 0.45 of the HBM rate, this one streams 1.3 x the bytes at 0.9 of it.
// The integer sums, and therefore the results, are the packed kernel's bit for bit.
constexpr int kFormatQ6KCodes = 114;
template <> struct KqFormat<kFormatQ6KCodes> {  // codes [K] int8, sc [K/16] int8, d [K/256] f16
    static constexpr int kPlanes = 3;
    static constexpr int kStages = 4;
    __host__ __device__ static constexpr uint32_t seg_bytes(int plane) { return plane == 0 ? kKqSegElems : plane == 1 ? kKqSegElems / 16 : kKqSegElems / 256 * 2; }
    __host__ __device__ static constexpr uint32_t bytes_per_256(int plane) { return plane == 0 ? 256 : plane == 1 ? 16 : 2; }
};
template <int kFormat> __host__ __device__ constexpr uint32_t kq_row_stage_bytes() {
    uint32_t b = 0;
    for (int i = 0; i < KqFormat<kFormat>::kPlanes; ++i) b += KqFormat<kFormat>::seg_bytes(i);
    return b;
}
template <int kFormat> __host__ __device__ constexpr uint32_t kq_plane_offset(int plane) {  // within a stage
    uint32_t b = 0;
    for (int i = 0; i < plane; ++i) b += KqFormat<kFormat>::seg_bytes(i) * kTeamWarps;
    return b;
}
template <int kFormat> __host__ __device__ constexpr uint32_t kq_stage_bytes() { return kq_row_stage_bytes<kFormat>() * kTeamWarps; }

// Tensor maps of one resident tensor whose rows span several K segments (built on upload, kept in device memory): per
// plane, boxes of 8, 4, 2 and 1 rows x one segment.  A plane whose segment is at most 256 bytes is a 2-D byte view
// [rows][pitch]; a wider one is the 3-D view [rows][pitch / 256][256], because a tile's innermost extent is limited to
// 256 elements.  One copy per plane then fetches a row group's segment where the per-row path issues 16 to 32 small ones.
struct alignas(64) KqTileMaps {
    CUtensorMap map[kKqMaxPlanes][4];
};

struct KqTask {
    const uint8_t* plane[kKqMaxPlanes];
    float* y;               // [batch][rows]
    uint32_t rows;
    uint32_t first_row;
};

struct KqParams {
    KqTask task[kMaxTasks];
    uint32_t ntasks, total_rows;
    const float* x;         // [batch][K] fp32; null with a gather: the vector gathered by the previous launch
    uint32_t K;             // columns, a multiple of the format's block size
    uint32_t nseg;          // ceil(K / kKqSegElems)
    uint32_t pitch[kKqMaxPlanes];  // global row pitch of each plane, bytes
    int* error_word;
    PeerGather gather;      // world == 0: outputs go to task[].y only
    const KqTileMaps* tile_maps[kMaxTasks];   // null: the tensor's rows go one copy per row and plane when K spans several segments
};

template <int kFormat>
__host__ __device__ inline size_t gemv_kq_smem_bytes(uint32_t nseg, int batch) {
    const size_t kpad = static_cast<size_t>(nseg) * kKqSegElems;
    return static_cast<size_t>(KqFormat<kFormat>::kStages) * kq_stage_bytes<kFormat>()
           + static_cast<size_t>(batch) * 2 * kpad                 // two digit planes, natural order
           + static_cast<size_t>(batch) * (kpad / 32) * 8          // per-block scale (d/256); half of it unused (the limit of columns x tokens counts it)
           + 2 * KqFormat<kFormat>::kStages * 8 + 16
           + kKqPartialFloats * sizeof(float);                      // batch 1: per-warp partial row sums
}

// The limit of columns x tokens that entry points and callers know of Q4_0, Q4_K and Q5_K: what their activations take as two digits
// beside a ring of six (Q5_K: four) stages of eight rows.
inline size_t gemv_kq_limit_bytes(int format, uint32_t nseg, int batch) {
    const size_t kpad = static_cast<size_t>(nseg) * kKqSegElems, stages = format == 13 ? 4 : 6;
    const size_t row = kKqSegElems / 2 + (format == 2 ? kKqSegElems / 32 * 2 : kKqSegElems / 16 + kKqSegElems / 256 * 4 + (format == 13 ? kKqSegElems / 8 : 0));
    return stages * kTeamWarps * row + static_cast<size_t>(batch) * (2 * kpad + kpad / 32 * 8) + 2 * stages * 8 + 16 + kKqPartialFloats * sizeof(float);
}

struct KqWalk {  // GroupWalk over KqParams
    uint32_t r, r_end, ti;
    __device__ KqWalk(uint32_t first, uint32_t last) : r(first), r_end(last), ti(0) {}
    __device__ bool done() const { return r >= r_end; }
    __device__ RowGroup next(const KqParams& p) {
        RowGroup g{0, 0, 0};
        if (done()) return g;
        while (r >= p.task[ti].first_row + p.task[ti].rows) ++ti;
        g.task = ti;
        g.row0 = r - p.task[ti].first_row;
        g.nrows = min(min(static_cast<uint32_t>(kTeamWarps), p.task[ti].rows - g.row0), r_end - r);
        r += g.nrows;
        return g;
    }
};

__device__ __forceinline__ int dot16(const uint4& w, const uint4& x) {
    int s = dp4a_ss(w.x, x.x, 0);
    s = dp4a_ss(w.y, x.y, s);
    s = dp4a_ss(w.z, x.z, s);
    return dp4a_ss(w.w, x.w, s);
}

// Bytes 0..63 minus 32, per byte, as signed bytes: setting the top bit first keeps the subtraction
// from borrowing across bytes, flipping it back afterwards leaves the two's-complement difference.
__device__ __forceinline__ uint32_t sub32_bytes(uint32_t q) { return ((q | 0x80808080u) - 0x20202020u) ^ 0x80808080u; }

// Sum of `v` over the lanes of a warp for eight rows at once.  Each exchange step halves the number of rows a lane still
// carries, so they cost 9 shuffles instead of 40.  On return every lane holds the complete sum
// of row `row` (lanes that share the low bits hold the same row); the order of additions is fixed.
__device__ __forceinline__ float kq_reduce_rows(const float (&acc)[8], int lane, uint32_t& row) {
    float a4[4];
    {
        const bool up = lane & 16;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float send = up ? acc[i] : acc[i + 4], keep = up ? acc[i + 4] : acc[i];
            a4[i] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
        }
    }
    float a2[2];
    {
        const bool up = lane & 8;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const float send = up ? a4[i] : a4[i + 2], keep = up ? a4[i + 2] : a4[i];
            a2[i] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
        }
    }
    float a1;
    {
        const bool up = lane & 4;
        const float send = up ? a2[0] : a2[1], keep = up ? a2[1] : a2[0];
        a1 = keep + __shfl_xor_sync(0xffffffffu, send, 4);
    }
#pragma unroll
    for (int o = 2; o > 0; o >>= 1) a1 += __shfl_xor_sync(0xffffffffu, a1, o);
    row = ((lane >> 4) & 1) * 4 + ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1);
    return a1;
}

// Team-wide barrier that also agrees on failure: true when any of the team's threads passed `failed`.
__device__ __forceinline__ bool team_barrier_any(int team, bool failed) {
    uint32_t any;
    asm volatile(
        "{ .reg .pred p, q; setp.ne.u32 q, %3, 0; barrier.red.or.pred p, %1, %2, q; selp.u32 %0, 1, 0, p; }"
        : "=r"(any) : "r"(2 + team), "r"(kTeamWarps * 32), "r"(static_cast<uint32_t>(failed)) : "memory");
    return any != 0;
}

template <int kFormat, int kBatch>
__global__ void __launch_bounds__(kGemvThreads, 1) gemv_kq_kernel(const __grid_constant__ KqParams p) {
    using F = KqFormat<kFormat>;
    constexpr int kStages = F::kStages;
    static_assert(kStages % kTeams == 0, "ring depth must be a multiple of the number of consumer teams");
    constexpr uint32_t kStageBytes = kq_stage_bytes<kFormat>();
    extern __shared__ __align__(128) uint8_t smem[];
    const uint32_t kpad = p.nseg * kKqSegElems;
    uint8_t* ring = smem;
    uint8_t* xd = ring + kStages * kStageBytes;                                  // [batch][2][kpad] int8, natural order
    float* xscale = reinterpret_cast<float*>(xd + static_cast<size_t>(kBatch) * 2 * kpad);   // [batch][kpad/32]  d/256
    uint64_t* full = reinterpret_cast<uint64_t*>(xscale + static_cast<size_t>(kBatch) * 2 * (kpad / 32));
    uint64_t* empty = full + kStages;
    volatile int* abort_word = reinterpret_cast<volatile int*>(empty + kStages);
    float* partial = reinterpret_cast<float*>(empty + kStages + 2);   // batch 1: [team][unit parity][K slice][row]
    float* stash = partial + kKqPartialFloats;                        // gather only: [batch][rows of this CTA's slice]

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint32_t r_first, r_last;
    cta_row_slice(p.total_rows, blockIdx.x, gridDim.x, r_first, r_last);
    const uint32_t n_mine = r_last - r_first;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], kTeamWarps);
        }
        *abort_word = 0;
        mbar_fence_init();
    }
    __syncthreads();
    pdl_launch_dependents();

    if (warp == kGemvWarps) {
        // ---------------- producer warp ----------------
        uint32_t unit = 0;
        bool ok = true;
        bool announce = p.gather.world != 0 && blockIdx.x == 0;   // see gemv_q8_0_kernel
        KqWalk walk(r_first, r_last);
        const int my_row = lane / F::kPlanes, my_plane = lane % F::kPlanes;  // one copy per (row, plane) of a unit
        bool contiguous = p.nseg == 1 && p.K == static_cast<uint32_t>(kKqSegElems);
#pragma unroll
        for (int pl = 0; pl < F::kPlanes; ++pl) contiguous = contiguous && p.pitch[pl] == F::seg_bytes(pl);
        while (!walk.done() && ok) {
            RowGroup pair[kTeams];
#pragma unroll
            for (int m = 0; m < kTeams; ++m) pair[m] = walk.next(p);
            for (uint32_t s = 0; s < p.nseg && ok; ++s) {
#pragma unroll
                for (int m = 0; m < kTeams; ++m, ++unit) {
                    const uint32_t stage = unit % kStages;
                    if (unit >= static_cast<uint32_t>(kStages) && announce) {
                        announce = false;
                        if (lane == 0) { pdl_wait(); gather_publish_pending(p.gather); }
                        __syncwarp();
                    }
                    if (unit >= static_cast<uint32_t>(kStages)) {
                        if (!mbar_wait(&empty[stage], ((unit / kStages) - 1) & 1)) {
                            if (lane == 0) { *abort_word = 1; atomicExch(p.error_word, kErrEmptyWaitTimeout); }
                            ok = false;
                        }
                    }
                    if (*abort_word) ok = false;
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                    const RowGroup g = pair[m];
                    if (g.nrows == 0) {
                        if (lane == 0) mbar_arrive(&full[stage]);
                        continue;
                    }
                    const KqTask& t = p.task[g.task];
                    const uint32_t elems = min(static_cast<uint32_t>(kKqSegElems), p.K - s * kKqSegElems);  // multiple of the block size
                    uint32_t row_bytes = 0;
#pragma unroll
                    for (int pl = 0; pl < F::kPlanes; ++pl) row_bytes += (elems / 256 * F::bytes_per_256(pl) + (elems % 256) * F::bytes_per_256(pl) / 256 + 15) & ~15u;
                    const bool tiled = !contiguous && p.tile_maps[g.task] != nullptr;
                    // A tiled copy always delivers whole segments (columns past the row arrive as zeros).  A tile must land on a
                    // 128-byte boundary, so planes whose segment is narrower than that always arrive as ONE box of eight rows
                    // (the rows past a partial group are a few bytes that nobody reads; past the tensor they are zeros).
                    uint32_t tiled_bytes = 0;
#pragma unroll
                    for (int pl = 0; pl < F::kPlanes; ++pl) tiled_bytes += (F::seg_bytes(pl) < 128 ? static_cast<uint32_t>(kTeamWarps) : g.nrows) * F::seg_bytes(pl);
                    if (lane == 0) mbar_arrive_expect_tx(&full[stage], tiled ? tiled_bytes : g.nrows * row_bytes);
                    __syncwarp();
                    if (contiguous) {
                        // rows of one full segment follow each other in every plane: one copy per plane for the whole group
                        if (lane < F::kPlanes) {
                            bulk_g2s(ring + stage * kStageBytes + kq_plane_offset<kFormat>(lane),
                                     t.plane[lane] + static_cast<size_t>(g.row0) * p.pitch[lane], g.nrows * F::seg_bytes(lane), &full[stage]);
                        }
                    } else if (tiled) {
                        // tiled copies: per plane one for a whole row group, or boxes of 4, 2 and 1 rows for a partial one
                        if (lane == 0) {
                            const KqTileMaps* maps = p.tile_maps[g.task];
#pragma unroll
                            for (int pl = 0; pl < F::kPlanes; ++pl) {
                                uint32_t done_rows = 0;
                                const uint32_t want = F::seg_bytes(pl) < 128 ? static_cast<uint32_t>(kTeamWarps) : g.nrows;
#pragma unroll
                                for (int k = 0; k < 4; ++k) {
                                    const uint32_t box = 8u >> k;
                                    if (want - done_rows >= box) {
                                        uint8_t* dst = ring + stage * kStageBytes + kq_plane_offset<kFormat>(pl) + done_rows * F::seg_bytes(pl);
                                        if (F::seg_bytes(pl) <= 256)
                                            tma_load_2d(dst, &maps->map[pl][k], static_cast<int>(s * F::seg_bytes(pl)), static_cast<int>(g.row0 + done_rows), &full[stage]);
                                        else
                                            tma_load_3d(dst, &maps->map[pl][k], 0, static_cast<int>(s * (F::seg_bytes(pl) / 256)), static_cast<int>(g.row0 + done_rows), &full[stage]);
                                        done_rows += box;
                                    }
                                }
                            }
                        }
                    } else if (my_row < static_cast<int>(g.nrows) && my_row < kTeamWarps) {
                        const uint32_t per256 = F::bytes_per_256(my_plane);
                        const uint32_t bytes = (elems / 256 * per256 + (elems % 256) * per256 / 256 + 15) & ~15u;
                        const uint32_t seg_off = static_cast<uint32_t>(static_cast<uint64_t>(s) * kKqSegElems / 256 * per256);
                        uint8_t* dst = ring + stage * kStageBytes + kq_plane_offset<kFormat>(my_plane) + my_row * F::seg_bytes(my_plane);
                        bulk_g2s(dst, t.plane[my_plane] + static_cast<size_t>(g.row0 + my_row) * p.pitch[my_plane] + seg_off, bytes, &full[stage]);
                    }
                }
            }
        }
        if (announce && lane == 0) { pdl_wait(); gather_publish_pending(p.gather); }
        if (lane == 0) {
            const uint32_t armed = unit < static_cast<uint32_t>(kStages) ? unit : kStages;
            for (uint32_t k = 0; k < armed; ++k) {
                const uint32_t u = unit - 1 - k;
                if (!mbar_wait(&full[u % kStages], (u / kStages) & 1)) atomicExch(p.error_word, kErrDrainTimeout);
            }
        }
        return;
    }

    // ---------------- consumer warps ----------------
    pdl_wait();
    // Row-sharded launch (peer_gather.cuh): wait for every rank's previous launch; a null x means "what it gathered".
    unsigned long long epoch = 0;
    const float* x_src = p.x;
    if (p.gather.world) {
        epoch = gather_epoch(p.gather);
        if (!x_src) {   // chained: the other ranks' previous outputs are this launch's input, so they are needed now
            if (!gather_wait(p.gather, lane, epoch)) {
                if (lane == 0 && !*abort_word) { *abort_word = 1; atomicExch(p.error_word, kErrPeerWaitTimeout); }
            }
            x_src = gather_previous(p.gather, epoch);
        }
    }
    // Prologue: two-digit quantisation of the activations, natural element order.
    {
        const uint32_t quad = static_cast<uint32_t>(lane) >> 2, part = static_cast<uint32_t>(lane) & 3;
        const uint32_t nblk = p.K / 32;
        for (int t = 0; t < kBatch; ++t) {
            for (uint32_t b0 = warp * 8; b0 < nblk; b0 += kGemvWarps * 8) {
                const uint32_t b = b0 + quad;
                const bool live = b < nblk;
                const float4* src = reinterpret_cast<const float4*>(x_src + static_cast<size_t>(t) * p.K + b * 32 + part * 8);
                const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
                const float4 lo = live ? __ldcg(src) : zero, hi = live ? __ldcg(src + 1) : zero;  // L2: coherent with peers' stores
                const float v[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
                uint2 c1, c2;
                const float d = quantise_block_quad(v, c1, c2);
                if (!live) continue;
                uint8_t* base = xd + static_cast<size_t>(t) * 2 * kpad + b * 32 + part * 8;
                *reinterpret_cast<uint2*>(base) = c1;
                *reinterpret_cast<uint2*>(base + kpad) = c2;
                if (part == 0) xscale[static_cast<size_t>(t) * (kpad / 32) + b] = d * (1.0f / 256.0f);
            }
        }
    }
    asm volatile("bar.sync 1, %0;" ::"r"(kGemvWarps * 32) : "memory");

    const int team = warp / kTeamWarps, twarp = warp % kTeamWarps;
    bool ok = *abort_word == 0;
    if constexpr (kBatch == 1) {
        // ---- batch 1: a warp owns a slice of K and walks every row of the unit with its activations in registers ----
        // Shared memory is then read for weights only (reading two activation digits per weight from it costs several
        // times the weight bytes in wavefronts and capped the kernel at a third of the HBM rate).
        // A warp has a K slice of two super-blocks and all eight rows; a lane owns one 16-weight scale group.
        constexpr bool kCodes = kFormat == kFormatQ6KCodes;   // a lane owns the 16 weights of group (lane & 15) of its super-block, in element order
        constexpr int kR = kTeamWarps;             // rows per warp
        constexpr int kSlices = 8;                 // K slices per segment
        const uint32_t kslice = static_cast<uint32_t>(twarp);
        // Q6_K lane geometry (src/quant.cpp:500-517): element e = half*128 + group*32 + l lives in ql byte
        // half*64 + (group%2)*32 + l (low nibble for group < 2), qh byte half*32 + l bits 2*group.., scale half*8 + group*2 + l/16
        const uint32_t sg = lane & 15, qhalf = sg >> 3, group = (sg >> 1) & 3, six = sg & 1;
        const uint32_t shift4 = group >= 2 ? 4u : 0u, shift2 = group * 2;
        const uint32_t sbl = kslice * 2 + (static_cast<uint32_t>(lane) >> 4);   // super-block within the segment

        uint4 xa = make_uint4(0, 0, 0, 0), xc = xa;   // digit 1, digit 2
        float xs = 0.0f;     // activation scale of the lane's block
        int bias = 0;        // minus (zero point x sum of the lane's activation codes), the dp4a chain's starting value
        // A lane whose block lies past the end of the row reads the segment's first block instead (valid bytes, so a
        // finite scale) with zero activations and a zero scale: its terms are exactly zero and need no select.
        uint32_t wofs = 0;   // the lane's super-block
        auto load_x = [&](uint32_t seg) {
            const uint4 zero = make_uint4(0, 0, 0, 0);
            if (kCodes) {
                const uint32_t e0 = seg * kKqSegElems + sbl * 256 + sg * 16;
                const bool live = e0 < p.K;
                xa = live ? *reinterpret_cast<const uint4*>(xd + e0) : zero;
                xc = live ? *reinterpret_cast<const uint4*>(xd + kpad + e0) : zero;
                xs = live ? xscale[e0 / 32] : 0.0f;
                wofs = live ? sbl : 0u;
            } else {
                const uint32_t e0 = seg * kKqSegElems + sbl * 256 + qhalf * 128 + group * 32 + six * 16;
                const bool live = e0 < p.K;
                xa = live ? *reinterpret_cast<const uint4*>(xd + e0) : zero;
                xc = live ? *reinterpret_cast<const uint4*>(xd + kpad + e0) : zero;
                xs = live ? xscale[e0 / 32] : 0.0f;
                const uint4 ones = make_uint4(0x01010101u, 0x01010101u, 0x01010101u, 0x01010101u);
                bias = -32 * (dot16(ones, xa) * 256 + dot16(ones, xc));
                wofs = live ? sbl : 0u;
            }
        };
        if (p.nseg == 1) load_x(0);

        uint32_t pair_index = 0;
        KqWalk walk(r_first, r_last);
        while (!walk.done()) {
            RowGroup pair[kTeams];
#pragma unroll
            for (int m = 0; m < kTeams; ++m) pair[m] = walk.next(p);
            RowGroup g = pair[0];
            if constexpr (kTeams > 1) { if (team == 1) g = pair[kTeams - 1]; }
            const KqTask& t = p.task[g.task];
            float acc[kR];
#pragma unroll
            for (int r = 0; r < kR; ++r) acc[r] = 0.0f;
            bool failed = false;
            for (uint32_t s = 0; s < p.nseg; ++s) {
                const uint32_t unit = (pair_index * p.nseg + s) * kTeams + team;
                const uint32_t stage = unit % kStages;
                if (*abort_word || !mbar_wait(&full[stage], (unit / kStages) & 1)) {
                    if (lane == 0 && !*abort_word) { *abort_word = 1; atomicExch(p.error_word, kErrFullWaitTimeout); }
                    failed = true;
                    break;
                }
                if (p.nseg > 1) load_x(s);
                const uint8_t* st = ring + stage * kStageBytes;
                const uint8_t* w0;   // the lane's weights in row 0 of the stage
                const uint8_t* w1;
                const int8_t* sc = nullptr;
                const __half* dd = nullptr;
                if (kCodes) {
                    w0 = st + kq_plane_offset<kFormat>(0) + wofs * 256 + sg * 16;   // codes
                    w1 = w0;
                    sc = reinterpret_cast<const int8_t*>(st + kq_plane_offset<kFormat>(1)) + wofs * 16 + sg;
                    dd = reinterpret_cast<const __half*>(st + kq_plane_offset<kFormat>(2)) + wofs;
                } else {
                    w0 = st + kq_plane_offset<kFormat>(0) + wofs * 128 + qhalf * 64 + (group & 1) * 32 + six * 16;   // ql
                    w1 = st + kq_plane_offset<kFormat>(1) + wofs * 64 + qhalf * 32 + six * 16;                       // qh
                    sc = reinterpret_cast<const int8_t*>(st + kq_plane_offset<kFormat>(2)) + wofs * 16 + sg;
                    dd = reinterpret_cast<const __half*>(st + kq_plane_offset<kFormat>(3)) + wofs;
                }
                auto row_body = [&](int r) {
                    if (kCodes) {
                        const uint4 q = *reinterpret_cast<const uint4*>(w0 + r * F::seg_bytes(0));
                        const int a = dot16(q, xa), c = dot16(q, xc);
                        const float dsc = __half2float(dd[r * (F::seg_bytes(2) / 2)]) * static_cast<float>(sc[r * F::seg_bytes(1)]);  // (d * scale), the reference's order
                        acc[r] = fmaf(dsc * xs, static_cast<float>(a * 256 + c), acc[r]);
                    } else {
                        const uint4 l4 = *reinterpret_cast<const uint4*>(w0 + r * F::seg_bytes(0));
                        const uint4 h4 = *reinterpret_cast<const uint4*>(w1 + r * F::seg_bytes(1));
                        // codes stay 0..63; the zero point 32 is in `bias`
                        const uint32_t q0 = ((l4.x >> shift4) & 0x0F0F0F0Fu) | (((h4.x >> shift2) & 0x03030303u) << 4);
                        const uint32_t q1 = ((l4.y >> shift4) & 0x0F0F0F0Fu) | (((h4.y >> shift2) & 0x03030303u) << 4);
                        const uint32_t q2 = ((l4.z >> shift4) & 0x0F0F0F0Fu) | (((h4.z >> shift2) & 0x03030303u) << 4);
                        const uint32_t q3 = ((l4.w >> shift4) & 0x0F0F0F0Fu) | (((h4.w >> shift2) & 0x03030303u) << 4);
                        int a = dp4a_us(q0, xa.x, 0), c = dp4a_us(q0, xc.x, bias);
                        a = dp4a_us(q1, xa.y, a); c = dp4a_us(q1, xc.y, c);
                        a = dp4a_us(q2, xa.z, a); c = dp4a_us(q2, xc.z, c);
                        a = dp4a_us(q3, xa.w, a); c = dp4a_us(q3, xc.w, c);
                        const float dsc = __half2float(dd[r * (F::seg_bytes(3) / 2)]) * static_cast<float>(sc[r * F::seg_bytes(2)]);  // (d * scale), the reference's order
                        acc[r] = fmaf(dsc * xs, static_cast<float>(a * 256 + c), acc[r]);
                    }
                };
                if (g.nrows == static_cast<uint32_t>(kTeamWarps)) {   // the common case: no per-row test
#pragma unroll
                    for (int r = 0; r < kR; ++r) row_body(r);
                } else {
#pragma unroll
                    for (int r = 0; r < kR; ++r)
                        if (static_cast<uint32_t>(r) < g.nrows) row_body(r);
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&empty[stage]);
            }
            // rows of the unit: sum over the warp's lanes, then over the K slices through shared memory
            uint32_t prow;
            const float psum = kq_reduce_rows(acc, lane, prow);
            float* part = partial + (team * 2 + (pair_index & 1)) * (kTeamWarps * kTeamWarps);
            if ((lane & 3) == 0) part[kslice * kTeamWarps + prow] = psum;
            if (team_barrier_any(team, failed)) { ok = false; break; }
            if (twarp == 0 && static_cast<uint32_t>(lane) < g.nrows) {
                float v = part[lane];
#pragma unroll
                for (int k = 1; k < kSlices; ++k) v += part[k * kTeamWarps + lane];
                const uint32_t row = g.row0 + lane;
                if (t.y) t.y[row] = v;
                if (p.gather.world) stash[t.first_row + row - r_first] = v;
            }
            ++pair_index;
        }
    } else {
        uint32_t pair_base = 0;
        KqWalk walk(r_first, r_last);
        while (!walk.done() && ok) {
            RowGroup pair[kTeams];
    #pragma unroll
            for (int m = 0; m < kTeams; ++m) pair[m] = walk.next(p);
            RowGroup g = pair[0];
            if constexpr (kTeams > 1) { if (team == 1) g = pair[kTeams - 1]; }
            const KqTask& t = p.task[g.task];
            const uint32_t row = g.row0 + twarp;
            const bool valid = static_cast<uint32_t>(twarp) < g.nrows;
            float acc[kBatch];
    #pragma unroll
            for (int b = 0; b < kBatch; ++b) acc[b] = 0.0f;

            for (uint32_t s = 0; s < p.nseg; ++s) {
                const uint32_t unit = pair_base + s * kTeams + team;
                const uint32_t stage = unit % kStages;
                if (*abort_word || !mbar_wait(&full[stage], (unit / kStages) & 1)) {
                    if (lane == 0 && !*abort_word) { *abort_word = 1; atomicExch(p.error_word, kErrFullWaitTimeout); }
                    ok = false;
                    break;
                }
                if (valid) {
                    const uint8_t* st = ring + stage * kStageBytes;
                    const uint32_t e_base = s * kKqSegElems;
                    const uint32_t elems = min(static_cast<uint32_t>(kKqSegElems), p.K - e_base);
                    if (kFormat == kFormatQ6KCodes) {
                        // ---- Q6_K, unpacked codes: a lane owns one 16-weight group in element order; two super-blocks a pass ----
                        const uint8_t* qc = st + kq_plane_offset<kFormat>(0) + twarp * F::seg_bytes(0);
                        const int8_t* sc = reinterpret_cast<const int8_t*>(st + kq_plane_offset<kFormat>(1) + twarp * F::seg_bytes(1));
                        const __half* dd = reinterpret_cast<const __half*>(st + kq_plane_offset<kFormat>(2) + twarp * F::seg_bytes(2));
                        const uint32_t sg = lane & 15;
    #pragma unroll 4
                        for (int i = 0; i < kKqSegElems / 256 / 2; ++i) {
                            const uint32_t sbl = i * 2 + (lane >> 4);
                            if (sbl * 256 < elems) {
                                const uint4 q = *reinterpret_cast<const uint4*>(qc + sbl * 256 + sg * 16);
                                const float dsc = __half2float(dd[sbl]) * static_cast<float>(sc[sbl * 16 + sg]);
                                const uint32_t e0 = e_base + sbl * 256 + sg * 16;
    #pragma unroll
                                for (int tk = 0; tk < kBatch; ++tk) {
                                    const uint4 x1 = *reinterpret_cast<const uint4*>(xd + static_cast<size_t>(tk) * 2 * kpad + e0);
                                    const uint4 x2 = *reinterpret_cast<const uint4*>(xd + static_cast<size_t>(tk) * 2 * kpad + kpad + e0);
                                    const int isum = dot16(q, x1) * 256 + dot16(q, x2);
                                    acc[tk] = fmaf(dsc * xscale[static_cast<size_t>(tk) * (kpad / 32) + e0 / 32], static_cast<float>(isum), acc[tk]);
                                }
                            }
                        }
                    } else {
                        // ---- Q6_K: a lane owns one 16-weight scale group; a warp covers two super-blocks a pass ----
                        const uint8_t* ql = st + kq_plane_offset<kFormat>(0) + twarp * F::seg_bytes(0);
                        const uint8_t* qh = st + kq_plane_offset<kFormat>(1) + twarp * F::seg_bytes(1);
                        const int8_t* sc = reinterpret_cast<const int8_t*>(st + kq_plane_offset<kFormat>(2) + twarp * F::seg_bytes(2));
                        const __half* dd = reinterpret_cast<const __half*>(st + kq_plane_offset<kFormat>(3) + twarp * F::seg_bytes(3));
                        const uint32_t sg = lane & 15, half = sg >> 3, group = (sg >> 1) & 3, six = sg & 1;
                        const uint32_t shift4 = group >= 2 ? 4u : 0u, shift2 = group * 2;
                        // element e = half*128 + group*32 + l: ql byte half*64 + (group%2)*32 + l, qh byte half*32 + l,
                        // scale half*8 + group*2 + l/16 == sg (src/quant.cpp:500-517)
    #pragma unroll 4
                        for (int i = 0; i < kKqSegElems / 256 / 2; ++i) {
                            const uint32_t sbl = i * 2 + (lane >> 4);
                            if (sbl * 256 < elems) {
                                const uint4 l4 = *reinterpret_cast<const uint4*>(ql + sbl * 128 + half * 64 + (group & 1) * 32 + six * 16);
                                const uint4 h4 = *reinterpret_cast<const uint4*>(qh + sbl * 64 + half * 32 + six * 16);
                                uint4 q;
                                q.x = sub32_bytes(((l4.x >> shift4) & 0x0F0F0F0Fu) | (((h4.x >> shift2) & 0x03030303u) << 4));
                                q.y = sub32_bytes(((l4.y >> shift4) & 0x0F0F0F0Fu) | (((h4.y >> shift2) & 0x03030303u) << 4));
                                q.z = sub32_bytes(((l4.z >> shift4) & 0x0F0F0F0Fu) | (((h4.z >> shift2) & 0x03030303u) << 4));
                                q.w = sub32_bytes(((l4.w >> shift4) & 0x0F0F0F0Fu) | (((h4.w >> shift2) & 0x03030303u) << 4));
                                const float dsc = __half2float(dd[sbl]) * static_cast<float>(sc[sbl * 16 + sg]);  // (d * scale), the reference's order
                                const uint32_t e0 = e_base + sbl * 256 + half * 128 + group * 32 + six * 16;
    #pragma unroll
                                for (int tk = 0; tk < kBatch; ++tk) {
                                    const uint4 x1 = *reinterpret_cast<const uint4*>(xd + static_cast<size_t>(tk) * 2 * kpad + e0);
                                    const uint4 x2 = *reinterpret_cast<const uint4*>(xd + static_cast<size_t>(tk) * 2 * kpad + kpad + e0);
                                    const int isum = dot16(q, x1) * 256 + dot16(q, x2);
                                    acc[tk] = fmaf(dsc * xscale[static_cast<size_t>(tk) * (kpad / 32) + e0 / 32], static_cast<float>(isum), acc[tk]);
                                }
                            }
                        }
                    }
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&empty[stage]);
            }
            if (!ok) break;
            pair_base += kTeams * p.nseg;
            if (valid) {
    #pragma unroll
                for (int tk = 0; tk < kBatch; ++tk) {
                    float v = acc[tk];
    #pragma unroll
                    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                    if (lane == 0 && t.y) t.y[static_cast<size_t>(tk) * t.rows + row] = v;
                    if (lane == 0 && p.gather.world) stash[static_cast<size_t>(tk) * n_mine + (t.first_row + row - r_first)] = v;
                }
            }
        }
    }
    if (p.gather.world) {
        asm volatile("bar.sync 1, %0;" ::"r"(kGemvWarps * 32) : "memory");
        // With an input of its own the launch needs the other ranks only now: they must have finished the previous
        // launch (whose reads used the parity about to be overwritten) before anything is stored into their regions.
        bool may_push = true;
        if (p.x && !gather_wait(p.gather, lane, epoch)) {
            if (lane == 0) atomicExch(p.error_word, kErrPeerWaitTimeout);
            may_push = false;
        }
        if (may_push) gather_push(p.gather, epoch, stash, n_mine, r_first, p.total_rows, kBatch, warp, kGemvWarps, lane);
        asm volatile("bar.sync 1, %0;" ::"r"(kGemvWarps * 32) : "memory");
        if (threadIdx.x == 0) gather_finish(p.gather, epoch);
    }
}

}  // namespace zk
