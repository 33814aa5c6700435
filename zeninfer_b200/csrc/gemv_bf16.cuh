// Decode-time products of bfloat16 matrices with one fp32 vector, memory-bound by design.
//
//   * one CTA per SM owns a contiguous slice of the launch's rows (over all its tensors); its eight warps split K in units of
//     256 columns (and, where K has fewer units than warps, the row groups too), eight rows per step: a lane takes 16 bytes of
//     each of eight rows and eight values of x;
//   * weights arrive by cp.async in a ring of shared memory that belongs to one lane: a lane reads back the words it asked for
//     itself, so a step needs no barrier, and the bytes in flight (three steps, 96 KB per CTA) cost no registers.  The first are
//     asked for before the previous grid has finished (weights are constants; griddepcontrol).  B200, one product behind the
//     other: 45056 x 4096 with a norm in front 65.0 -> 56.1 us, 4096 x 18432 30.6 -> 26.8, 6416 x 2048 with norm and shift
//     9.0 -> 8.1, against sixteen warps that held two steps in registers (128 KB).  More in flight is slower (five steps: 58.6),
//     sixteen warps too (58.9), and so is a CTA small enough to have the next launch's beside it: the SMs that finish first then
//     take two of those each, and the pair above goes from 82.7 to 97.8;
//   * nothing else is read before the previous grid has finished, because it may be what that grid writes (a residual as the bias, a
//     norm weight or shift made per token).  The vectors among it that seldom are, bias, norm weights and shift, are only asked
//     into L2 by then, so that they need not come from HBM later;
//   * the prologue can finish the sublayer before it (row_ops.cuh: grouped norm, residual add, token shift or output norm), so
//     a decode step needs no launches for them: every CTA forms the input vector itself, CTA 0 stores the residual stream;
//   * the epilogue adds a bias and applies the product's activation (squared ReLU, or the logits' soft cap) in fp32; a matrix may
//     begin with pairs of rows (gate, up) that leave the launch as silu(gate) * up.
// Activations are fp32 throughout: the product is exact up to fp32 accumulation.
#pragma once
#include "row_ops.cuh"

namespace zk {

constexpr int kDenseThreads = 256, kDenseWarps = kDenseThreads / 32;
constexpr uint32_t kDenseUnit = 256;          // columns a warp takes at a time: eight per lane
constexpr int kDenseRows = 8;                 // rows per step
constexpr int kDenseMaxTasks = 4;
constexpr uint32_t kDenseStepBytes = kDenseRows * kDenseUnit * 2;                                       // of one warp
__host__ __device__ constexpr uint32_t dense_ring_bytes(int slots) { return slots * kDenseWarps * kDenseStepBytes; }
constexpr int kPreQuads = 4;                  // four-value words of a row a lane keeps in the prologue: rows of up to 4096 values

enum : int { kActNone = 0, kActSquaredRelu = 1, kActSoftcap = 2 };

struct DenseTask {
    const __nv_bfloat16* w;   // [rows][ld], zero beyond the real columns
    const float* x;           // [K]; ignored when the launch carries a prologue
    float* y;                 // [rows - 2 pairs]
    const float* bias;        // [rows - 2 pairs], or null
    float* gated;             // [pairs]
    uint32_t rows, K, ld;
    uint32_t first_row;       // index of its first row in the launch's row space
    uint32_t pairs;           // rows 2 i and 2 i + 1 (i < pairs) give gated[i]; first_row is even then
    int act;
    float cap;
};

struct DenseGemvParams {
    DenseTask task[kDenseMaxTasks];
    uint32_t tasks, total_rows;
    uint32_t k_split;         // warps that share a row group: a power of two, at most kDenseWarps
    uint32_t row_unit;        // a CTA's slice begins at a multiple of this many rows: 2 where a task has pairs
    uint32_t has_prologue;    // 1: one task, whose input is the prologue's view
    uint32_t row_in_registers;  // the prologue by sublayer_in_registers; otherwise by row_ops.cuh's functions
    uint32_t scratch_floats;
    SublayerEnd pre;
};

__host__ __device__ inline uint32_t dense_units(uint32_t ld) { return (ld + kDenseUnit - 1) / kDenseUnit; }

__device__ __forceinline__ float dense_activation(float v, int act, float cap) {
    if (act == kActSquaredRelu) { const float r = fmaxf(v, 0.0f); return r * r; }
    if (act == kActSoftcap) return cap * tanhf(v / cap);
    return v;
}
__device__ __forceinline__ void dense_fma8(const uint4& w, const float (&x)[8], float& acc) {
    const uint32_t u[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        acc = fmaf(__uint_as_float(u[i] << 16), x[2 * i], acc);
        acc = fmaf(__uint_as_float(u[i] & 0xffff0000u), x[2 * i + 1], acc);
    }
}
__device__ __forceinline__ unsigned long long dense_pair(float lo, float hi) {
    unsigned long long v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
    return v;
}
// The same with even and odd columns in the two halves of acc.
__device__ __forceinline__ void dense_fma8_pairs(const uint4& w, const unsigned long long (&x)[4], unsigned long long& acc) {
    const uint32_t u[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int i = 0; i < 4; ++i)
        asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(dense_pair(__uint_as_float(u[i] << 16), __uint_as_float(u[i] & 0xffff0000u))), "l"(x[i]));
}

// The prologue of rows of up to 4096 values (a multiple of 32, in 1, 2, 4 or 8 parts, every array 16-byte aligned), formed as
// sublayer_row and sublayer_view form it: a warp holds an eighth of the row in registers and all arrays are asked for at once.
// row_ops.cuh's functions go over the row in shared memory three to five times with a barrier after each.
struct RowWords { float4 v[kPreQuads]; };
__device__ __forceinline__ void row_words(RowWords& r, const float* src, uint32_t first, uint32_t chunk, uint32_t lane) {
#pragma unroll
    for (int q = 0; q < kPreQuads; ++q) {
        const uint32_t i = 4 * (lane + 32 * q);
        r.v[q] = src && i < chunk ? __ldcg(reinterpret_cast<const float4*>(src + first + i)) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
}
__device__ __forceinline__ float row_square_sum(const RowWords& r) {
    float s = 0.0f;
#pragma unroll
    for (int q = 0; q < kPreQuads; ++q) s += (r.v[q].x * r.v[q].x + r.v[q].y * r.v[q].y) + (r.v[q].z * r.v[q].z + r.v[q].w * r.v[q].w);
    return s;
}
template <typename F> __device__ __forceinline__ void row_each(RowWords& r, F f) {
#pragma unroll
    for (int q = 0; q < kPreQuads; ++q) {
        f(r.v[q].x, q, 0);
        f(r.v[q].y, q, 1);
        f(r.v[q].z, q, 2);
        f(r.v[q].w, q, 3);
    }
}
__device__ __forceinline__ float row_at(const RowWords& r, int q, int c) { return c == 0 ? r.v[q].x : c == 1 ? r.v[q].y : c == 2 ? r.v[q].z : r.v[q].w; }

__device__ __forceinline__ const float* prologue_post(const SublayerEnd& p) { return p.shift ? p.shift : p.out_norm; }
// Asks norm weights and shift into L2: no value is read, so this may go in front of the wait.
__device__ __forceinline__ void prologue_prefetch(const SublayerEnd& p) {
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, chunk = p.n / kDenseWarps;
    const float* const post = prologue_post(p);
#pragma unroll
    for (int q = 0; q < kPreQuads; ++q) {
        const uint32_t i = 4 * (lane + 32 * q);
        if (lane % 2 || i >= chunk) continue;      // a lane per 32 bytes
        if (p.norm_weight) prefetch_l2(p.norm_weight + warp * chunk + i);
        if (post) prefetch_l2(post + warp * chunk + i);
    }
}
// xs [n] and a barrier; scratch: 4 * kDenseWarps floats.
__device__ __forceinline__ void sublayer_in_registers(const SublayerEnd& p, float* xs, float* scratch) {
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, chunk = p.n / kDenseWarps, first = warp * chunk;
    const float part_size = static_cast<float>(p.n / p.groups);
    const uint32_t per = kDenseWarps / p.groups, part = warp / per * per;      // the warps that share this warp's part of the norm
    auto inverse_rms = [&](const float* sums, uint32_t from, uint32_t count, float size) {
        float s = 0.0f;
        for (uint32_t w = 0; w < count; ++w) s += sums[from + w];
        return 1.0f / sqrtf(s / size + p.eps);
    };
    RowWords x, y, z, norm, post;
    row_words(x, p.x_in, first, chunk, lane);
    row_words(y, p.y_a, first, chunk, lane);
    row_words(z, p.y_b ? p.y_b : p.shift ? p.before : nullptr, first, chunk, lane);
    row_words(norm, p.norm_weight, first, chunk, lane);
    row_words(post, prologue_post(p), first, chunk, lane);
    if (p.y_b) {
        RowWords a, b;
        row_words(a, p.weight_a, first, chunk, lane);
        row_words(b, p.weight_b, first, chunk, lane);
        const float sa = warp_sum(row_square_sum(y)), sb = warp_sum(row_square_sum(z));
        row_each(y, [&](float& v, int q, int k) { v *= row_at(a, q, k); });
        row_each(z, [&](float& v, int q, int k) { v *= row_at(b, q, k); });
        if (lane == 0) { scratch[warp] = sa; scratch[kDenseWarps + warp] = sb; }
        __syncthreads();
        const float ra = inverse_rms(scratch, 0, kDenseWarps, static_cast<float>(p.n)), rb = inverse_rms(scratch, kDenseWarps, kDenseWarps, static_cast<float>(p.n));
        row_each(y, [&](float& v, int q, int k) { v = 0.5f * (v * ra + row_at(z, q, k) * rb); });
        if (p.shift) row_words(z, p.before, first, chunk, lane);
    }
    if (p.y_a && p.norm_weight) {
        const float s = warp_sum(row_square_sum(y));
        if (lane == 0) scratch[2 * kDenseWarps + warp] = s;
        __syncthreads();
        const float r = inverse_rms(scratch, 2 * kDenseWarps + part, per, part_size);
        row_each(y, [&](float& v, int q, int k) { v = row_at(x, q, k) + v * r * row_at(norm, q, k); });
    } else {
        row_each(y, [&](float& v, int q, int k) { v += row_at(x, q, k); });      // y_a null: y is zero
    }
    if (blockIdx.x == 0) {
#pragma unroll
        for (int q = 0; q < kPreQuads; ++q) {
            const uint32_t i = 4 * (lane + 32 * q);
            if (i < chunk && p.x_out) *reinterpret_cast<float4*>(p.x_out + first + i) = y.v[q];
            if (i < chunk && p.keep) *reinterpret_cast<float4*>(p.keep + first + i) = x.v[q];
        }
    }
    if (p.shift) {
        row_each(y, [&](float& v, int q, int k) { v += (row_at(z, q, k) - v) * row_at(post, q, k); });
    } else if (p.out_norm) {
        const float s = warp_sum(row_square_sum(y));
        if (lane == 0) scratch[3 * kDenseWarps + warp] = s;
        __syncthreads();
        const float r = inverse_rms(scratch, 3 * kDenseWarps + part, per, part_size);
        row_each(y, [&](float& v, int q, int k) { v = v * r * row_at(post, q, k); });
    }
#pragma unroll
    for (int q = 0; q < kPreQuads; ++q) {
        const uint32_t i = 4 * (lane + 32 * q);
        if (i < chunk) *reinterpret_cast<float4*>(xs + first + i) = y.v[q];
    }
    __syncthreads();
}

// kSlots: steps of a warp on their way at any time, in shared memory; 0: weights straight from memory, for inputs that leave no
// room for a ring.
template <int kSlots>
__global__ void __launch_bounds__(kDenseThreads, 2) gemv_bf16_kernel(const __grid_constant__ DenseGemvParams p) {
    extern __shared__ __align__(16) float dense_smem[];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint64_t row_units = (p.total_rows + p.row_unit - 1) / p.row_unit;
    const uint32_t slice0 = static_cast<uint32_t>(row_units * blockIdx.x / gridDim.x) * p.row_unit;
    const uint32_t slice1 = min(static_cast<uint32_t>(row_units * (blockIdx.x + 1) / gridDim.x) * p.row_unit, p.total_rows);
    const uint32_t team = warp / p.k_split, part = warp % p.k_split, teams = kDenseWarps / p.k_split;
    pdl_launch_dependents();

    // A warp's steps: (task, row group, K unit), walked in that order, once to ask for the weights and once to use them; what a step
    // needs of its task stays in registers.  Where the warps that share a row group do not divide its units evenly (9, 17 or 20 units
    // on eight warps), the ones with a unit more are others in the next group: the same warps every time would keep the rest waiting,
    // half of them for a tenth of the launch where sixteen warps shared 72 units.
    struct Walk {
        const __nv_bfloat16* w;       // the lane's word of row r
        uint32_t ti, r, r_end, u, units, ld, x;
    };
    auto place = [&](Walk& w) { w.w = p.task[w.ti].w + static_cast<size_t>(w.r) * w.ld + w.u * kDenseUnit + lane * 8; };
    auto enter = [&](Walk& w) {      // the next task of the slice with work for this warp
        for (; w.ti < p.tasks; ++w.ti) {
            const DenseTask& t = p.task[w.ti];
            const uint32_t a = max(slice0, t.first_row), b = min(slice1, t.first_row + t.rows);
            w.ld = t.ld;
            w.units = dense_units(t.ld);
            if (a < b && a + team * kDenseRows < b && part < w.units) {
                w.r = a - t.first_row + team * kDenseRows;
                w.r_end = b - t.first_row;
                w.u = part;
                place(w);
                return;
            }
            w.x += w.units * kDenseUnit;
        }
    };
    auto advance = [&](Walk& w) {    // to the step after w
        w.u += p.k_split;
        w.w += p.k_split * kDenseUnit;
        if (w.u >= w.units) {
            w.u = (w.u + (w.units > p.k_split ? w.units : 0u)) & (p.k_split - 1);
            w.r += teams * kDenseRows;
            if (w.r < w.r_end) {
                place(w);
            } else {
                w.x += w.units * kDenseUnit;
                ++w.ti;
                enter(w);
            }
        }
    };
    // the lane's words of a step lie 512 bytes apart, lane behind lane: neither the copies nor the reads meet bank conflicts
    uint8_t* const mine = reinterpret_cast<uint8_t*>(dense_smem) + warp * kSlots * kDenseStepBytes + lane * 16;
    auto ask = [&](const Walk& w, int slot) {      // rows past the slice's end keep what the slot held: their sums are not used
        const uint32_t dst = smem_u32(mine) + slot * kDenseStepBytes;
        const bool real = w.u * kDenseUnit + lane * 8 < w.ld;
        const __nv_bfloat16* src = real ? w.w : w.w - lane * 8;
#pragma unroll
        for (int i = 0; i < kDenseRows; ++i)
            if (w.r + i < w.r_end) copy16_or_zero(dst + i * 512, src + static_cast<size_t>(i) * w.ld, real);
    };
    Walk in{}, at;
    enter(in);
    at = in;
#pragma unroll
    for (int s = 0; s < kSlots; ++s) {
        if (in.ti < p.tasks) { ask(in, s); advance(in); }
        asm volatile("cp.async.commit_group;" ::: "memory");
    }

    // the input vectors in shared memory, each padded with zeros to whole units; then per-row partial sums of the slice
    float* const xs = dense_smem + dense_ring_bytes(kSlots) / sizeof(float);
    uint32_t x_floats = 0;
    const float* bias_at = nullptr;      // the bias of the thread's first row
    {
        const uint32_t row = slice0 + threadIdx.x;
        if (row < slice1) {
            uint32_t ti = 0;
            while (row >= p.task[ti].first_row + p.task[ti].rows) ++ti;
            const DenseTask& t = p.task[ti];
            const uint32_t r = row - t.first_row;
            if (t.bias && r >= 2 * t.pairs) bias_at = t.bias + r - 2 * t.pairs;
        }
        if (bias_at) prefetch_l2(bias_at);
    }
    if (p.has_prologue) {
        x_floats = dense_units(p.task[0].ld) * kDenseUnit;
        float* scratch = xs + x_floats;
        for (uint32_t i = p.pre.n + threadIdx.x; i < x_floats; i += kDenseThreads) xs[i] = 0.0f;
        if (p.row_in_registers) {
            prologue_prefetch(p.pre);
            pdl_wait();
            sublayer_in_registers(p.pre, xs, scratch);
        } else {
            pdl_wait();
            sublayer_row<kDenseThreads>(p.pre, 0, xs, scratch);
            if (blockIdx.x == 0) {
                if (p.pre.x_out)
                    for (uint32_t i = threadIdx.x; i < p.pre.n; i += kDenseThreads) p.pre.x_out[i] = xs[i];
                if (p.pre.keep)
                    for (uint32_t i = threadIdx.x; i < p.pre.n; i += kDenseThreads) p.pre.keep[i] = p.pre.x_in[i];
            }
            sublayer_view<kDenseThreads>(p.pre, xs, p.pre.before, scratch);
        }
    } else {
        pdl_wait();
        for (uint32_t ti = 0; ti < p.tasks; ++ti) {
            const DenseTask& t = p.task[ti];
            const uint32_t padded = dense_units(t.ld) * kDenseUnit, words = reinterpret_cast<uintptr_t>(t.x) % 16 ? 0u : t.K / 4;
            float4* dst = reinterpret_cast<float4*>(xs + x_floats);
#pragma unroll 8
            for (uint32_t i = threadIdx.x; i < words; i += kDenseThreads) dst[i] = __ldcg(reinterpret_cast<const float4*>(t.x) + i);
            for (uint32_t i = 4 * words + threadIdx.x; i < padded; i += kDenseThreads) xs[x_floats + i] = i < t.K ? __ldcg(t.x + i) : 0.0f;
            x_floats += padded;
        }
        __syncthreads();
    }
    float* sums = xs + x_floats + p.scratch_floats;      // [rows of the slice][k_split]
    const float bias = bias_at ? __ldcg(bias_at) : 0.0f;

    unsigned long long acc2[kDenseRows];
#pragma unroll
    for (int i = 0; i < kDenseRows; ++i) acc2[i] = 0ull;
    auto consume = [&](const Walk& at, int slot) {
        const float4* xv = reinterpret_cast<const float4*>(xs + at.x + at.u * kDenseUnit + lane * 8);
        const float4 x0 = xv[0], x1 = xv[1];
        const unsigned long long x[4] = {dense_pair(x0.x, x0.y), dense_pair(x0.z, x0.w), dense_pair(x1.x, x1.y), dense_pair(x1.z, x1.w)};
        if constexpr (kSlots > 0) {
#pragma unroll
            for (int i = 0; i < kDenseRows; ++i) dense_fma8_pairs(*reinterpret_cast<const uint4*>(mine + slot * kDenseStepBytes + i * 512), x, acc2[i]);
        } else if (at.u * kDenseUnit + lane * 8 < at.ld) {
#pragma unroll
            for (int i = 0; i < kDenseRows; ++i)
                if (at.r + i < at.r_end) dense_fma8_pairs(__ldg(reinterpret_cast<const uint4*>(at.w + static_cast<size_t>(i) * at.ld)), x, acc2[i]);
        }
        if (at.u + p.k_split < at.units) return;
        // the row group is done: its sums over 32 lanes; at each of the first exchanges a lane keeps half of the rows it carries
        float acc[kDenseRows];
#pragma unroll
        for (int i = 0; i < kDenseRows; ++i) {
            float lo, hi;
            asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(acc2[i]));
            acc[i] = lo + hi;
            acc2[i] = 0ull;
        }
        uint32_t kept = 0;
#pragma unroll
        for (int n = kDenseRows / 2, o = 16; o > 0; n >>= 1, o >>= 1) {
            if (n > 0) {
                const bool up = lane & o;
#pragma unroll
                for (int i = 0; i < n; ++i) {
                    const float keep = up ? acc[i + n] : acc[i], give = up ? acc[i] : acc[i + n];
                    acc[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
                }
                kept += up ? n : 0;
            } else {
                acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], o);
            }
        }
        if ((lane & (32 / kDenseRows - 1)) == 0 && at.r + kept < at.r_end) sums[static_cast<size_t>(p.task[at.ti].first_row + at.r + kept - slice0) * p.k_split + (at.u & (p.k_split - 1))] = acc[0];
    };
    for (int slot = 0; at.ti < p.tasks; advance(at)) {
        if constexpr (kSlots > 0) asm volatile("cp.async.wait_group %0;" ::"n"(kSlots - 1) : "memory");
        consume(at, slot);
        if constexpr (kSlots > 0) {
            if (in.ti < p.tasks) { ask(in, slot); advance(in); }      // into the slot that was just read by the same lane
            asm volatile("cp.async.commit_group;" ::: "memory");
            if (++slot == kSlots) slot = 0;
        }
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < slice1 - slice0; i += kDenseThreads) {
        const uint32_t row = slice0 + i;
        uint32_t ti = 0;
        while (row >= p.task[ti].first_row + p.task[ti].rows) ++ti;
        const DenseTask& t = p.task[ti];
        const uint32_t parts = min(p.k_split, dense_units(t.ld));
        auto total = [&](uint32_t at) {
            float v = 0.0f;
            for (uint32_t s = 0; s < parts; ++s) v += sums[static_cast<size_t>(at) * p.k_split + s];
            return v;
        };
        const uint32_t r = row - t.first_row, paired = 2 * t.pairs;
        if (r < paired) {
            if (!(r & 1)) t.gated[r / 2] = silu_f(total(i)) * total(i + 1);
        } else {
            t.y[r - paired] = dense_activation(total(i) + (i < kDenseThreads ? bias : t.bias ? __ldcg(t.bias + r - paired) : 0.0f), t.act, t.cap);
        }
    }
}

}  // namespace zk
