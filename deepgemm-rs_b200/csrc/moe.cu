// Row movement around the grouped GEMM for MoE layers: building the 128-row-padded contiguous
// layout (token rows and their packed scale factors) and combining expert outputs back per
// token.  These are the steps the reference leaves to the caller of
// Serving::moe_grouped_layer (deepgemm/src/api_serving.rs:293-377); they are pure HBM streaming.
#include "host.h"
#include "ptx.cuh"

#include <cuda_bf16.h>

namespace dg {

// dst[i, :] = src[idx[i], :], or zeros when idx[i] < 0.  One warp per row, 16-byte vectors.
__global__ void __launch_bounds__(256) gather_rows_kernel(const uint4* __restrict__ src, const int32_t* __restrict__ idx,
                                                         uint4* __restrict__ dst, uint32_t n_rows, uint32_t vec_per_row,
                                                         uint64_t src_pitch_vec, uint64_t dst_pitch_vec) {
    const uint32_t row = blockIdx.x * 8u + (threadIdx.x >> 5), lane = threadIdx.x & 31u;
    if (row >= n_rows) return;
    const int32_t s = __ldg(idx + row);
    uint4* d = dst + (size_t)row * dst_pitch_vec;
    if (s < 0) {
        for (uint32_t v = lane; v < vec_per_row; v += 32u) d[v] = make_uint4(0, 0, 0, 0);
    } else {
        // source rows are read once per top-k copy: keep them cached, stream the copies out
        const uint4* p = src + (size_t)s * src_pitch_vec;
        uint32_t v = lane;
        for (; v + 96u < vec_per_row; v += 128u) {     // four loads in flight per lane before the stores
            const uint4 r0 = __ldg(p + v), r1 = __ldg(p + v + 32u), r2 = __ldg(p + v + 64u), r3 = __ldg(p + v + 96u);
            __stcs(d + v, r0); __stcs(d + v + 32u, r1); __stcs(d + v + 64u, r2); __stcs(d + v + 96u, r3);
        }
        for (; v < vec_per_row; v += 32u) __stcs(d + v, __ldg(p + v));
    }
}

// dst[r * dst_sr + i * dst_si] = src[r * src_sr + idx[i] * src_si] (0 when idx[i] < 0), words.
// With (sr, si) = (cols, 1) on both sides this permutes the MN columns of a packed SF tensor;
// with one side (1, sf_rows) it converts to / from a row-per-token wire format.
__global__ void __launch_bounds__(256) gather_sf_kernel(const uint32_t* __restrict__ src, uint64_t src_sr, uint64_t src_si,
                                                       const int32_t* __restrict__ idx, uint32_t* __restrict__ dst,
                                                       uint64_t dst_sr, uint64_t dst_si, uint32_t sf_rows, uint32_t n) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int32_t s = __ldg(idx + i);
    for (uint32_t r = 0; r < sf_rows; ++r)
        dst[r * dst_sr + (size_t)i * dst_si] = s < 0 ? 0u : __ldg(src + r * src_sr + (size_t)s * src_si);
}

// Rows and scale-factor columns of the contiguous MoE layout in one pass: slot i takes row idx[i] of x and column idx[i]
// of its packed scale factors (zeros for idx[i] < 0).  A block owns 32 slots: every warp copies four rows, one vector of
// each in flight at a time and two vectors deep, then the words of every eighth scale-factor row, one slot per lane.
// Slots of blocks that no expert owns (block_expert < 0) are left as they are: the GEMM visits none of them.
// HBM-bound by the rows written (the rows read are a top-k-th of them and stay in L2).  Against gather_rows and gather_sf,
// which write the unowned blocks too: 163584 slots of 7168 bytes, a tenth of them unowned, 278 us and 294; 24320 of 7168 29
// and 38; 49024 of 4096 32 and 40; 2304 of 2048 11 and 18 (launches).
__global__ void __launch_bounds__(256) gather_tokens_kernel(const uint4* __restrict__ x, uint64_t x_pitch_vec, const uint32_t* __restrict__ sf,
                                                           uint64_t sf_cols, uint32_t sf_rows, const int32_t* __restrict__ idx,
                                                           const int32_t* __restrict__ block_expert, uint32_t block_rows, uint32_t n,
                                                           uint32_t vec_per_row, uint4* __restrict__ dst, uint32_t* __restrict__ dst_sf) {
    griddep_wait();
    griddep_launch_dependents();
    const uint32_t slot0 = blockIdx.x * 32u, warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    if (__ldg(block_expert + slot0 / block_rows) < 0) return;
    const int32_t my_src = slot0 + lane < n ? __ldg(idx + slot0 + lane) : -1;
    const uint4* from[4];
    uint4* to[4];
#pragma unroll
    for (uint32_t i = 0; i < 4; ++i) {
        const uint32_t r = warp * 4u + i;
        const int32_t s = __shfl_sync(0xffffffffu, my_src, r);
        from[i] = s < 0 ? nullptr : x + (size_t)s * x_pitch_vec;
        to[i] = slot0 + r < n ? dst + (size_t)(slot0 + r) * vec_per_row : nullptr;
    }
#pragma unroll 2
    for (uint32_t v = lane; v < vec_per_row; v += 32u) {
        uint4 q[4];
#pragma unroll
        for (uint32_t i = 0; i < 4; ++i) q[i] = from[i] ? __ldg(from[i] + v) : make_uint4(0, 0, 0, 0);
#pragma unroll
        for (uint32_t i = 0; i < 4; ++i)
            if (to[i]) __stcs(to[i] + v, q[i]);
    }
    if (slot0 + lane < n)
        for (uint32_t r = warp; r < sf_rows; r += 8u)
            dst_sf[(size_t)r * n + slot0 + lane] = my_src < 0 ? 0u : __ldg(sf + r * sf_cols + (uint32_t)my_src);
}

// out[t, :] = sum_j w[t, j] * src[pos[t, j], :] over the top-k copies of token t (f32 sum in the
// order j = 0..topk-1, one bf16 rounding at the end); pos < 0 skips a copy; w == NULL means 1.
// HBM-bound: one block per token, 8 columns per thread.  Four copies are requested before the first is added: with
// one load at a time a thread waited out the memory latency once per copy.
__global__ void __launch_bounds__(256) combine_kernel(const __nv_bfloat16* __restrict__ src, const int32_t* __restrict__ pos,
                                                     const float* __restrict__ w, __nv_bfloat16* __restrict__ out,
                                                     uint32_t tokens, uint32_t topk, uint32_t cols, uint64_t src_pitch,
                                                     uint64_t out_pitch) {
    constexpr uint32_t kBatch = 4;
    const uint32_t t = blockIdx.x;
    if (t >= tokens) return;
    const int32_t* tpos = pos + (size_t)t * topk;
    const float* tw = w ? w + (size_t)t * topk : nullptr;
    for (uint32_t c = threadIdx.x * 8u; c < cols; c += blockDim.x * 8u) {
        float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        for (uint32_t j0 = 0; j0 < topk; j0 += kBatch) {
            int32_t p[kBatch];
            float g[kBatch];
            uint4 v[kBatch];
#pragma unroll
            for (uint32_t i = 0; i < kBatch; ++i) {
                p[i] = j0 + i < topk ? __ldg(tpos + j0 + i) : -1;
                g[i] = tw && j0 + i < topk ? __ldg(tw + j0 + i) : 1.f;
            }
#pragma unroll
            for (uint32_t i = 0; i < kBatch; ++i)
                if (p[i] >= 0) v[i] = __ldcs(reinterpret_cast<const uint4*>(src + (size_t)p[i] * src_pitch + c));
#pragma unroll
            for (uint32_t i = 0; i < kBatch; ++i) {
                if (p[i] < 0) continue;
                const uint32_t u[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    acc[2 * q] += g[i] * __uint_as_float(u[q] << 16);
                    acc[2 * q + 1] += g[i] * __uint_as_float(u[q] & 0xffff0000u);
                }
            }
        }
        uint32_t o[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            __nv_bfloat162 h = __floats2bfloat162_rn(acc[2 * q], acc[2 * q + 1]);
            o[q] = *reinterpret_cast<uint32_t*>(&h);
        }
        *reinterpret_cast<uint4*>(out + (size_t)t * out_pitch + c) = make_uint4(o[0], o[1], o[2], o[3]);
    }
}

// ---- grouping plan: rows -> expert-contiguous slots ---------------------------------------------
// plan_count: counts[e] = number of rows routed to expert e (counts zeroed by the caller's stream).
__global__ void __launch_bounds__(256) plan_count_kernel(const int32_t* __restrict__ expert_of_row, uint32_t n_rows,
                                                        uint32_t num_experts, int32_t* __restrict__ counts) {
    const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n_rows) return;
    const int32_t e = __ldg(expert_of_row + r);
    if (e >= 0 && (uint32_t)e < num_experts) atomicAdd(counts + e, 1);
}

// plan_scan (one block): offsets[e] = first slot of expert e with every group padded to `align`
// rows, offsets[E] = total; block_expert[b] = expert owning the b-th `align`-row block or -1;
// cursors reset to 0.
__global__ void __launch_bounds__(1024) plan_scan_kernel(const int32_t* __restrict__ counts, uint32_t num_experts,
                                                        uint32_t align, uint32_t capacity, int32_t* __restrict__ offsets,
                                                        int32_t* __restrict__ cursors, int32_t* __restrict__ block_expert) {
    extern __shared__ int32_t sh_off[];  // [num_experts + 1]
    if (threadIdx.x == 0) {
        int32_t acc = 0;
        for (uint32_t e = 0; e < num_experts; ++e) {
            sh_off[e] = acc;
            acc += (int32_t)(((uint32_t)counts[e] + align - 1) / align * align);
        }
        sh_off[num_experts] = acc;
    }
    __syncthreads();
    for (uint32_t e = threadIdx.x; e <= num_experts; e += blockDim.x) {
        offsets[e] = sh_off[e];
        if (e < num_experts) cursors[e] = 0;
    }
    if (block_expert) {
        const uint32_t total = (uint32_t)sh_off[num_experts];
        for (uint32_t b = threadIdx.x; b < capacity / align; b += blockDim.x) {
            const uint32_t row = b * align;
            int32_t owner = -1;
            if (row < total) {
                uint32_t lo = 0, hi = num_experts;      // last e with sh_off[e] <= row
                while (hi - lo > 1) {
                    const uint32_t mid = (lo + hi) >> 1;
                    if ((uint32_t)sh_off[mid] <= row) lo = mid; else hi = mid;
                }
                owner = (int32_t)lo;
            }
            block_expert[b] = owner;
        }
    }
}

// plan_place: every row takes the next free slot of its expert.  slot_src[slot] = r / div (the
// token of copy r when div = top-k), slot_of_row[r] = slot.  The order of rows inside a group is
// not fixed from run to run; no result depends on it (a GEMM row does not see its neighbours).
__global__ void __launch_bounds__(256) plan_place_kernel(const int32_t* __restrict__ expert_of_row, uint32_t n_rows,
                                                        uint32_t num_experts, uint32_t div, const int32_t* __restrict__ offsets,
                                                        int32_t* __restrict__ cursors, int32_t* __restrict__ slot_src,
                                                        int32_t* __restrict__ slot_of_row) {
    const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n_rows) return;
    const int32_t e = __ldg(expert_of_row + r);
    if (e < 0 || (uint32_t)e >= num_experts) { slot_of_row[r] = -1; return; }
    const int32_t slot = offsets[e] + atomicAdd(cursors + e, 1);
    slot_src[slot] = (int32_t)(r / div);
    slot_of_row[r] = slot;
}

// The whole plan in one launch: a cluster of eight blocks of 1024 threads, every thread holding up to kPlanRows rows.
// Each block counts its rows per expert in shared memory; the value the shared atomic returns is the row's rank among
// its block's rows, so placing needs no second atomic.  The blocks read one another's counts through distributed
// shared memory, each scans all experts for itself, and slot = offset of the expert + rows of the blocks before + rank.
// The padding slots are filled here too.  Bound by launch and latency, not by bytes; two fills and the three kernels
// below took 61 us for 131072 rows and 256 experts and 19 us for 16152 rows and 64 experts, this one 21 and 12 us.  Rows are
// held in registers, which ends it at 131072; beyond, the fills and kernels below cost some 40 us more.
constexpr uint32_t kPlanBlocks = 8, kPlanThreads = 1024, kPlanRows = 16;
constexpr uint32_t kPlanMaxRows = kPlanBlocks * kPlanThreads * kPlanRows;
constexpr uint32_t kPlanMaxExperts = 2048;
__device__ __forceinline__ int32_t ld_cluster_i32(uint32_t addr) {
    int32_t v;
    asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
    return v;
}
__global__ void __cluster_dims__(kPlanBlocks, 1, 1) __launch_bounds__(kPlanThreads)
plan_cluster_kernel(const int32_t* __restrict__ expert_of_row, uint32_t n_rows, uint32_t num_experts, uint32_t align, uint32_t div,
                    uint32_t capacity, int32_t* __restrict__ counts, int32_t* __restrict__ offsets, int32_t* __restrict__ slot_src,
                    int32_t* __restrict__ slot_of_row, int32_t* __restrict__ block_expert) {
    extern __shared__ int32_t sh[];
    int32_t* hist = sh;                          // [E] this block's rows per expert
    int32_t* first = hist + num_experts;         // [E] first slot of this block's rows of an expert
    int32_t* total = first + num_experts;        // [E] rows per expert over all blocks
    int32_t* off = total + num_experts;          // [E + 1] first slot of an expert
    __shared__ int32_t warp_sum[32];
    griddep_wait();
    griddep_launch_dependents();
    const uint32_t tid = threadIdx.x, rank = cluster_ctarank(), lane = tid & 31u, warp = tid >> 5;
    for (uint32_t e = tid; e < num_experts; e += kPlanThreads) hist[e] = 0;
    int32_t ex[kPlanRows];
#pragma unroll
    for (uint32_t i = 0; i < kPlanRows; ++i) {
        const uint32_t r = (i * kPlanBlocks + rank) * kPlanThreads + tid;
        ex[i] = r < n_rows ? __ldg(expert_of_row + r) : -1;
    }
    __syncthreads();
    // expert and rank share a word (11 and 14 bits); negative = the row is dropped
    static_assert(kPlanMaxExperts == 1u << 11 && kPlanThreads * kPlanRows <= 1u << 14, "packing of expert and rank");
#pragma unroll
    for (uint32_t i = 0; i < kPlanRows; ++i)
        ex[i] = (ex[i] >= 0 && (uint32_t)ex[i] < num_experts) ? ex[i] | (atomicAdd(hist + ex[i], 1) << 11) : -1;
    cluster_sync_all();
    for (uint32_t e = tid; e < num_experts; e += kPlanThreads) {
        const uint32_t mine = smem_u32(hist + e);
        int32_t before = 0, sum = 0;
#pragma unroll
        for (uint32_t b = 0; b < kPlanBlocks; ++b) {
            const int32_t h = ld_cluster_i32(mapa(mine, b));
            if (b < rank) before += h;
            sum += h;
        }
        first[e] = before;
        total[e] = sum;
    }
    // the blocks' counts have been read: no block leaves before the others got here
    cluster_sync_all();
    // exclusive scan of the padded counts, 1024 experts at a time
    int32_t carry = 0;
    for (uint32_t e0 = 0; e0 < num_experts; e0 += kPlanThreads) {
        const uint32_t e = e0 + tid;
        const int32_t padded = e < num_experts ? (int32_t)(((uint32_t)total[e] + align - 1u) / align * align) : 0;
        int32_t incl = padded;
#pragma unroll
        for (uint32_t d = 1; d < 32; d <<= 1) {
            const int32_t o = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= d) incl += o;
        }
        if (lane == 31) warp_sum[warp] = incl;
        __syncthreads();
        if (warp == 0) {
            int32_t s = warp_sum[lane];
#pragma unroll
            for (uint32_t d = 1; d < 32; d <<= 1) {
                const int32_t o = __shfl_up_sync(0xffffffffu, s, d);
                if (lane >= d) s += o;
            }
            warp_sum[lane] = s;
        }
        __syncthreads();
        const int32_t excl = carry + (warp ? warp_sum[warp - 1] : 0) + incl - padded;
        if (e < num_experts) { off[e] = excl; first[e] += excl; }
        carry += warp_sum[31];
        __syncthreads();
    }
    if (tid == 0) off[num_experts] = carry;
    __syncthreads();
#pragma unroll
    for (uint32_t i = 0; i < kPlanRows; ++i) {
        const uint32_t r = (i * kPlanBlocks + rank) * kPlanThreads + tid;
        if (r >= n_rows) break;
        int32_t slot = -1;
        if (ex[i] >= 0) {
            slot = first[ex[i] & (int32_t)(kPlanMaxExperts - 1u)] + (ex[i] >> 11);
            slot_src[slot] = (int32_t)(r / div);
        }
        slot_of_row[r] = slot;
    }
    const uint32_t gtid = rank * kPlanThreads + tid, gwarp = gtid >> 5;
    constexpr uint32_t kAll = kPlanBlocks * kPlanThreads;
    if (rank == 0)
        for (uint32_t e = tid; e <= num_experts; e += kPlanThreads) {
            offsets[e] = off[e];
            if (e < num_experts) counts[e] = total[e];
        }
    for (uint32_t e = gwarp; e < num_experts; e += kAll / 32u)
        for (int32_t i = off[e] + total[e] + (int32_t)lane; i < off[e + 1]; i += 32) slot_src[i] = -1;
    for (uint32_t i = (uint32_t)off[num_experts] + gtid; i < capacity; i += kAll) slot_src[i] = -1;
    if (block_expert)
        for (uint32_t b = gtid; b < capacity / align; b += kAll) {
            const uint32_t row = b * align;
            int32_t owner = -1;
            if (row < (uint32_t)off[num_experts]) {
                uint32_t lo = 0, hi = num_experts;      // last e with off[e] <= row
                while (hi - lo > 1) {
                    const uint32_t mid = (lo + hi) >> 1;
                    if ((uint32_t)off[mid] <= row) lo = mid; else hi = mid;
                }
                owner = (int32_t)lo;
            }
            block_expert[b] = owner;
        }
}

}  // namespace dg

extern "C" {

int32_t dg_moe_plan(const int32_t* expert_of_row, uint32_t n_rows, uint32_t num_experts, uint32_t align, uint32_t div,
                    uint32_t capacity, int32_t* counts, int32_t* offsets, int32_t* cursors, int32_t* slot_src,
                    int32_t* slot_of_row, int32_t* block_expert, void* stream) {
    if (!expert_of_row || !counts || !offsets || !cursors || !slot_src || !slot_of_row)
        return dg::fail(DG_ERR_INVALID_ARG, "moe_plan: null buffer");
    if (num_experts == 0 || num_experts > 8192 || align == 0 || div == 0 || capacity % align != 0)
        return dg::fail(DG_ERR_INVALID_ARG, "moe_plan: need 1..8192 experts, align > 0, div > 0 and capacity %% align == 0");
    if ((uint64_t)capacity < (uint64_t)n_rows + (uint64_t)num_experts * (align - 1))
        return dg::fail(DG_ERR_INVALID_ARG, "moe_plan: capacity %u cannot hold %u rows in %u groups padded to %u", capacity,
                        n_rows, num_experts, align);
    const dg::DeviceInfo* dev;
    int32_t st = dg::current_device(&dev);
    if (st != DG_OK) return st;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (n_rows <= dg::kPlanMaxRows && num_experts <= dg::kPlanMaxExperts) {
        DG_CUDA_CHECK(dg::launch_dependent(dg::plan_cluster_kernel, dg::kPlanBlocks, dg::kPlanThreads,
                                     (uint32_t)sizeof(int32_t) * (4u * num_experts + 1u), s, expert_of_row, n_rows, num_experts, align,
                                     div, capacity, counts, offsets, slot_src, slot_of_row, block_expert));
        return DG_OK;
    }
    DG_CUDA_CHECK(cudaMemsetAsync(counts, 0, sizeof(int32_t) * num_experts, s));
    DG_CUDA_CHECK(cudaMemsetAsync(slot_src, 0xff, sizeof(int32_t) * (size_t)capacity, s));
    if (n_rows) {
        dg::plan_count_kernel<<<dg::ceil_div(n_rows, 256), 256, 0, s>>>(expert_of_row, n_rows, num_experts, counts);
        dg::note_launch();
    }
    dg::plan_scan_kernel<<<1, 1024, sizeof(int32_t) * (num_experts + 1), s>>>(counts, num_experts, align, capacity, offsets,
                                                                              cursors, block_expert);
    dg::note_launch();
    if (n_rows) {
        dg::plan_place_kernel<<<dg::ceil_div(n_rows, 256), 256, 0, s>>>(expert_of_row, n_rows, num_experts, div, offsets,
                                                                        cursors, slot_src, slot_of_row);
        dg::note_launch();
    }
    DG_CUDA_CHECK(cudaGetLastError());
    return DG_OK;
}

int32_t dg_gather_rows(const void* src, uint64_t src_pitch_bytes, const int32_t* idx, void* dst, uint64_t dst_pitch_bytes,
                       uint32_t n_rows, uint32_t row_bytes, void* stream) {
    if (!src || !idx || !dst) return dg::fail(DG_ERR_INVALID_ARG, "gather_rows: null buffer");
    if (row_bytes % 16 || src_pitch_bytes % 16 || dst_pitch_bytes % 16 || (reinterpret_cast<uintptr_t>(src) & 15u) ||
        (reinterpret_cast<uintptr_t>(dst) & 15u))
        return dg::fail(DG_ERR_INVALID_ARG, "gather_rows: rows, pitches and bases must be 16-byte multiples");
    if (n_rows == 0) return DG_OK;
    const dg::DeviceInfo* dev;
    int32_t st = dg::current_device(&dev);
    if (st != DG_OK) return st;
    dg::gather_rows_kernel<<<dg::ceil_div(n_rows, 8), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const uint4*>(src), idx, static_cast<uint4*>(dst), n_rows, row_bytes / 16, src_pitch_bytes / 16,
        dst_pitch_bytes / 16);
    dg::note_launch();
    DG_CUDA_CHECK(cudaGetLastError());
    return DG_OK;
}

int32_t dg_gather_sf(const uint32_t* src, uint64_t src_row_stride, uint64_t src_col_stride, const int32_t* idx, uint32_t* dst,
                     uint64_t dst_row_stride, uint64_t dst_col_stride, uint32_t sf_rows, uint32_t n, void* stream) {
    if (!src || !idx || !dst) return dg::fail(DG_ERR_INVALID_ARG, "gather_sf: null buffer");
    if (n == 0 || sf_rows == 0) return DG_OK;
    const dg::DeviceInfo* dev;
    int32_t st = dg::current_device(&dev);
    if (st != DG_OK) return st;
    dg::gather_sf_kernel<<<dg::ceil_div(n, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        src, src_row_stride, src_col_stride, idx, dst, dst_row_stride, dst_col_stride, sf_rows, n);
    dg::note_launch();
    DG_CUDA_CHECK(cudaGetLastError());
    return DG_OK;
}

int32_t dg_moe_gather(const void* x, uint64_t x_pitch_bytes, uint32_t row_bytes, const uint32_t* x_sf, uint32_t sf_rows,
                      uint64_t sf_cols, const int32_t* slot_src, const int32_t* block_expert, uint32_t align, uint32_t capacity,
                      void* rows_out, uint32_t* sf_out, void* stream) {
    if (!x || !x_sf || !slot_src || !block_expert || !rows_out || !sf_out) return dg::fail(DG_ERR_INVALID_ARG, "moe_gather: null buffer");
    if (row_bytes == 0 || row_bytes % 16 || x_pitch_bytes % 16 || (reinterpret_cast<uintptr_t>(x) & 15u) ||
        (reinterpret_cast<uintptr_t>(rows_out) & 15u))
        return dg::fail(DG_ERR_INVALID_ARG, "moe_gather: rows, pitches and bases must be 16-byte multiples");
    if (align == 0 || align % 32 || capacity % align) return dg::fail(DG_ERR_INVALID_ARG, "moe_gather: blocks must be multiples of 32 slots");
    if (capacity == 0) return DG_OK;
    const dg::DeviceInfo* dev;
    int32_t st = dg::current_device(&dev);
    if (st != DG_OK) return st;
    DG_CUDA_CHECK(dg::launch_dependent(dg::gather_tokens_kernel, dg::ceil_div(capacity, 32u), 256u, 0u, static_cast<cudaStream_t>(stream),
                                 static_cast<const uint4*>(x), x_pitch_bytes / 16u, x_sf, sf_cols, sf_rows, slot_src, block_expert, align,
                                 capacity, row_bytes / 16u, static_cast<uint4*>(rows_out), sf_out));
    return DG_OK;
}

int32_t dg_moe_combine(const void* src_bf16, uint64_t src_pitch, const int32_t* pos, const float* weights, void* out_bf16,
                       uint64_t out_pitch, uint32_t tokens, uint32_t topk, uint32_t cols, void* stream) {
    if (!src_bf16 || !pos || !out_bf16) return dg::fail(DG_ERR_INVALID_ARG, "moe_combine: null buffer");
    if (cols % 8 || src_pitch % 8 || out_pitch % 8 || (reinterpret_cast<uintptr_t>(src_bf16) & 15u) ||
        (reinterpret_cast<uintptr_t>(out_bf16) & 15u))
        return dg::fail(DG_ERR_INVALID_ARG, "moe_combine: columns and pitches must be multiples of 8 elements, bases 16-byte aligned");
    if (tokens == 0) return DG_OK;
    const dg::DeviceInfo* dev;
    int32_t st = dg::current_device(&dev);
    if (st != DG_OK) return st;
    // launched plainly: as a dependent launch its blocks sat on the SMs through the whole GEMM before it (MoE layer 1 % slower)
    dg::combine_kernel<<<tokens, 256, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const __nv_bfloat16*>(src_bf16), pos, weights, static_cast<__nv_bfloat16*>(out_bf16), tokens, topk, cols,
        src_pitch, out_pitch);
    dg::note_launch();
    DG_CUDA_CHECK(cudaGetLastError());
    return DG_OK;
}

}  // extern "C"
