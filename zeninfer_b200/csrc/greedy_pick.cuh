// Greedy token pick over fp32 logits: per token row, the index of the first maximum among the finite
// entries, -1 when the row has none.
//
// This is the greedy branch of the reference's sampler (sample_logits,
// src/adapters/dense_transformer_runtime.cpp:391-418): candidates are the finite logits in ascending
// index order, a candidate replaces the best only when it is strictly greater, so the lowest index wins
// ties and -0.0 ties with +0.0.
//
// A row of logits may be laid out in up to eight segments (the gathered shards of a row-sharded
// lm_head: [rank][token][shard rows]); a segment carries the index of its first entry.  Every
// candidate is packed into one 64-bit key, (order-preserving bits of the value) << 32 | (2^32-1 - index),
// so that an unsigned maximum is exactly the reference's rule; key 0 means "no candidate".
//
// A cluster of eight CTAs takes a row: 8192 threads, sixteen bytes a load where the row allows it, so that a vocabulary of
// 32000 is one load per thread; the CTAs' maxima meet in CTA 0's shared memory.  One launch and nothing to clear before it:
// what this takes in a decode step is latency.  B200, 32000 entries: 4.9 us a token less than a fill, a scan with atomics and a
// finishing launch (four layers of width 1024: 139 us a token before, 134 now).
#pragma once
#include <cooperative_groups.h>

#include <cstdint>
#include <utility>

#include "zk_ptx.cuh"

namespace zk {

constexpr int kPickMaxSegments = 8;
constexpr uint32_t kPickThreads = 1024, kPickCtas = 8;

struct PickSegment {
    const float* base;       // first entry of token 0
    uint32_t len;            // entries per token
    uint32_t first_index;    // index of the segment's first entry within the row
    uint32_t token_stride;   // floats between consecutive tokens
    uint32_t pad;
};

struct PickParams {
    PickSegment seg[kPickMaxSegments];
    uint32_t nseg;
    long long* pick;           // [tokens]
    // Row 0's pick once more, at note[*position % notes]: host memory the device can write, read by a host that waits for an event
    // behind the launch.  null: none.
    long long* note;
    const int* position;
    uint32_t notes;
};

__device__ __forceinline__ unsigned long long pick_key(float v, uint32_t index) {
    v += 0.0f;  // -0.0 -> +0.0: the reference compares values, and the two zeros are equal
    const uint32_t bits = __float_as_uint(v);
    if ((bits & 0x7f800000u) == 0x7f800000u) return 0ull;  // infinities and NaNs are never candidates
    const uint32_t ordered = (bits & 0x80000000u) ? ~bits : (bits | 0x80000000u);
    return (static_cast<unsigned long long>(ordered) << 32) | (0xffffffffu - index);
}

// grid = (kPickCtas, tokens)
__global__ void __cluster_dims__(kPickCtas, 1, 1) __launch_bounds__(kPickThreads) pick_kernel(const __grid_constant__ PickParams p) {
    __shared__ unsigned long long warp_best[kPickThreads / 32];
    __shared__ unsigned long long cta_best[kPickCtas];          // CTA 0's are the ones filled
    cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    auto started = cluster.barrier_arrive();                   // nobody writes to CTA 0 before it runs
    pdl_launch_dependents();
    pdl_wait();   // the logits come from an earlier launch, and the last pick may still be read by one
    const uint32_t first = blockIdx.x * kPickThreads + threadIdx.x;
    unsigned long long best = 0ull;
    auto take = [&](float v, uint32_t index) {
        const unsigned long long k = pick_key(v, index);
        best = k > best ? k : best;
    };
    for (uint32_t s = 0; s < p.nseg; ++s) {
        const PickSegment& sg = p.seg[s];
        const float* row = sg.base + static_cast<size_t>(blockIdx.y) * sg.token_stride;
        const uint32_t quads = (reinterpret_cast<uintptr_t>(row) & 15) ? 0u : sg.len / 4;
#pragma unroll 4
        for (uint32_t i = first; i < quads; i += kPickCtas * kPickThreads) {
            const float4 v = __ldcg(reinterpret_cast<const float4*>(row) + i);  // L2: the producer may be a peer's store
            const uint32_t at = sg.first_index + 4 * i;
            take(v.x, at); take(v.y, at + 1); take(v.z, at + 2); take(v.w, at + 3);
        }
#pragma unroll 4
        for (uint32_t i = 4 * quads + first; i < sg.len; i += kPickCtas * kPickThreads) take(__ldcg(row + i), sg.first_index + i);
    }
    auto warp_max = [&]() {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long other = __shfl_xor_sync(0xffffffffu, best, o);
            best = other > best ? other : best;
        }
    };
    warp_max();
    if ((threadIdx.x & 31) == 0) warp_best[threadIdx.x >> 5] = best;
    __syncthreads();
    if (threadIdx.x < 32) {
        best = warp_best[threadIdx.x];
        warp_max();
    }
    cluster.barrier_wait(std::move(started));
    if (threadIdx.x == 0) cluster.map_shared_rank(cta_best, 0)[blockIdx.x] = best;
    cluster.sync();
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        for (uint32_t c = 0; c < kPickCtas; ++c) best = cta_best[c] > best ? cta_best[c] : best;
        const long long pick = best ? static_cast<long long>(0xffffffffu - static_cast<uint32_t>(best)) : -1ll;
        p.pick[blockIdx.y] = pick;
        if (p.note && blockIdx.y == 0) p.note[static_cast<uint32_t>(*reinterpret_cast<const volatile int*>(p.position)) % p.notes] = pick;
    }
}

}  // namespace zk
