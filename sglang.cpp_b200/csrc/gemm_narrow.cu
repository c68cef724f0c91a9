// y = x W^T for a handful of rows (decode steps of a few requests): weights go from memory to registers.
//
// Such a call reads W once and computes next to nothing, and a decode step is a chain of them.  What bounds a small
// one is not bandwidth but what happens between the end of the kernel before it and its own end, so that part is
// kept short, and everything else is moved in front of it:
//   * 16 rows of W per CTA and the whole of K, dealt to its warps: no exchange between CTAs.  A lane loads 16
//     contiguous bytes of a row; which of the k of a 32-wide step these are does not matter, because x is loaded
//     the same way, so the bytes are the operands of two m16n8k16 products as they are (weights as the left one,
//     8 tokens as the right one).  No exchange through shared memory, no barrier before the sums meet.
//   * the weights that fit in registers (or, in a chain of such calls, in shared memory) are requested before griddepcontrol.wait.  CTAs are small (8 warps, a few
//     KB of shared memory), so those of the next kernels of the chain become resident beside the running one.
//   * behind the wait: x (from L2), the products, one exchange through shared memory, the epilogue.
// tcgen05 has no place here: its operands would have to pass through shared memory, and 128 x 64 tiles of W leave
// most SMs without one.
//
// The rows of W of a CTA's tile are two groups of 8, g and g + 8 of the product: neighbours in plain projections, the
// same features' gate and up rows, or the two halves of an attention head, so that what an epilogue has to bring
// together is in one thread.  Head norms need the whole head: 8 CTAs of a cluster exchange sums of squares.
//
// One layer's projections of hidden 1024, one request (us; the split-K clusters of gemm_skinny.cu before): 4096 x 1024 3.5 (6.3),
// 1024 x 2048 3.5 (5.9), 6144 x 1024 with SwiGLU 4.2 (8.8), 1024 x 3072 4.8 (6.9); their weights take 0.6 to 1.9 at the copy
// bandwidth.  151936 x 1024: 47 (57), which is the bandwidth.
//
// "Normalised input": x is an un-normalised residual row.  Each CTA reads whole rows anyway, so it sums their squares
// itself; the products run on bf16(x * weight of the norm), and the result is scaled by the row's 1 / rms.
#include "common.cuh"
#include "kernels.h"
#include "narrow.cuh"

namespace b200 {
namespace {

constexpr int kSteps = 4;        // k-steps of 32 per register buffer
constexpr int kHeadRanks = 8;    // CTAs that share an attention head
enum Kind { kPlain, kResidual, kHeads };

struct NarrowParams : NarrowOut {
    const __nv_bfloat16 *x, *w, *bias, *norm_w;
    int M, n_rows, up_row_offset, steps;
    int64_t ldx, K;
    float norm_eps;
    __nv_bfloat16* residual;
    // attention heads (see HeadEpilogue)
    const __nv_bfloat16 *q_norm_w, *k_norm_w;
    const float *cos_t, *sin_t;
    const int32_t *positions, *out_loc;
    __nv_bfloat16 *k_cache, *v_cache;
    int q_heads, kv_heads, max_pos;
    long long num_slots;
    float qk_eps;
    int* status;
    int early;   // let the next kernel's CTAs in at once
};

// Weights are read once: past L1.
__device__ __forceinline__ uint4 load_weights(const uint4* p) {
    uint4 v;
    asm volatile("ld.global.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void stage_weights(uint4* to, const uint4* from) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(to)), "l"(from) : "memory");
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void store_in_cluster(const float* mine, uint32_t rank, float v) {
    uint32_t remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smem_u32(mine)), "r"(rank));
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(remote), "f"(v) : "memory");
}

// BUFS register buffers of kSteps steps: with one, a warp's whole share of K is requested ahead of the wait.
// STAGED: the share goes to shared memory instead (every lane reads back what it has copied itself).
template <int KIND, bool NORM, int NT, int WARPS, int BUFS, bool STAGED>
__global__ void __launch_bounds__(WARPS * 32)
narrow_gemm_kernel(const NarrowParams p) {
    extern __shared__ uint4 s_weights[];   // STAGED: [warp][step][row group][lane]
    __shared__ float s_part[WARPS][NT * 8 * kTokenPitch];
    __shared__ float s_ssq[WARPS][NT * 8];
    __shared__ float s_head[kHeadRanks][NT * 8];
    if (p.early) pdl_launch_dependents();
    if (KIND == kHeads) cluster_arrive();   // (waited for before the first store to another CTA of the cluster)
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const bool gated = KIND == kPlain && p.up_row_offset > 0;
    const int tile = static_cast<int>(blockIdx.x);
    int row_a, row_b;
    if (KIND == kHeads) {
        row_a = (tile >> 3) * 128 + (tile & 7) * 8 + g;
        row_b = row_a + 64;
    } else if (gated) {
        row_a = tile * 8 + g;
        row_b = row_a + p.up_row_offset;
    } else {
        row_a = tile * 16 + g;
        row_b = min(row_a + 8, p.n_rows - 1);   // (n_out may be an odd multiple of 8)
    }
    const uint4* wa = reinterpret_cast<const uint4*>(p.w + row_a * p.K) + t;
    const uint4* wb = reinterpret_cast<const uint4*>(p.w + row_b * p.K) + t;
    const int first = warp * p.steps / WARPS, last = (warp + 1) * p.steps / WARPS;
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    constexpr int kShare = BUFS * kSteps;   // steps of a warp that are requested ahead of the wait
    uint4* staged = s_weights + warp * kShare * 64 + lane;
    uint4 a[STAGED ? 1 : BUFS][kSteps], b[STAGED ? 1 : BUFS][kSteps];
    auto fetch = [&](int buf, int at) {
#pragma unroll
        for (int u = 0; u < kSteps; ++u) {
            const bool there = at + u < last;
            a[buf][u] = there ? load_weights(wa + (at + u) * 4) : zero;
            b[buf][u] = there ? load_weights(wb + (at + u) * 4) : zero;
        }
    };
    if constexpr (STAGED) {
#pragma unroll
        for (int u = 0; u < kShare; ++u)
            if (first + u < last) {
                stage_weights(staged + u * 64, wa + (first + u) * 4);
                stage_weights(staged + u * 64 + 32, wb + (first + u) * 4);
            }
        asm volatile("cp.async.commit_group;" ::: "memory");
    } else {
#pragma unroll
        for (int i = 0; i < BUFS; ++i) fetch(i, first + i * kSteps);
    }
    // what the epilogue needs and no kernel of the chain writes: one thread per token and pair of features
    const int m = static_cast<int>(threadIdx.x) >> 3, f = static_cast<int>(threadIdx.x) & 7;
    const bool finishes = threadIdx.x < NT * 64;
    const bool live = finishes && m < p.M;
    const int head = tile >> 3, rank = tile & 7;
    const int head_kind = head < p.q_heads ? 0 : head < p.q_heads + p.kv_heads ? 1 : 2;   // q, k, v
    const __nv_bfloat16* head_w = head_kind == 0 ? p.q_norm_w : head_kind == 1 ? p.k_norm_w : nullptr;
    float cs = 1.f, sn = 0.f, w0 = 1.f, w1 = 1.f, bias0 = 0.f, bias1 = 0.f;
    int slot = -1;
    const int n0 = KIND == kHeads ? head * 128 + rank * 8 + f : gated ? tile * 8 + f : tile * 16 + f;
    const int n1 = n0 + (KIND == kHeads ? 64 : 8);
    if (live) {
        if (KIND != kResidual && !gated && p.bias != nullptr) {
            bias0 = __bfloat162float(p.bias[n0]);
            if (n1 < p.n_out) bias1 = __bfloat162float(p.bias[n1]);
        }
        if (KIND == kHeads) {
            if (head_kind < 2) {
                int pos = p.positions[m];
                if (pos < 0 || pos >= p.max_pos) {
                    if (rank == 0 && f == 0) atomicExch(&p.status[kStatusBadIndex], pos + 1);
                    pos = min(max(pos, 0), p.max_pos - 1);
                }
                cs = p.cos_t[static_cast<int64_t>(pos) * 64 + rank * 8 + f];
                sn = p.sin_t[static_cast<int64_t>(pos) * 64 + rank * 8 + f];
                if (head_w != nullptr) {
                    w0 = __bfloat162float(head_w[rank * 8 + f]);
                    w1 = __bfloat162float(head_w[64 + rank * 8 + f]);
                }
            }
            if (head_kind > 0) {
                slot = p.out_loc[m];
                if (slot < 0 || slot >= p.num_slots) {
                    if (rank == 0 && f == 0) atomicExch(&p.status[kStatusBadIndex], slot + 1);
                    slot = -1;
                }
            }
        }
    }
    pdl_wait_prior();

    float acc[NT][4] = {}, ss[NT] = {};
    const uint4* xr[NT];
#pragma unroll
    for (int n = 0; n < NT; ++n) xr[n] = reinterpret_cast<const uint4*>(p.x + (n * 8 + g) * p.ldx) + t;
    // products of one step's weights with the tokens' x, normalised input included
    auto step = [&](const uint4& wa4, const uint4& wb4, const uint4 (&x)[NT], const uint4& nw) {
#pragma unroll
        for (int n = 0; n < NT; ++n) {
            uint32_t v[4] = {x[n].x, x[n].y, x[n].z, x[n].w};
            if (NORM) {
                const uint32_t w4[4] = {nw.x, nw.y, nw.z, nw.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float lo = bf16_lo(v[e]), hi = bf16_hi(v[e]);
                    ss[n] = fmaf(lo, lo, fmaf(hi, hi, ss[n]));
                    v[e] = pack_bf16(lo * bf16_lo(w4[e]), hi * bf16_hi(w4[e]));
                }
            }
            mma_bf16_16816(acc[n], {wa4.x, wb4.x, wa4.y, wb4.y}, v[0], v[1]);
            mma_bf16_16816(acc[n], {wa4.z, wb4.z, wa4.w, wb4.w}, v[2], v[3]);
        }
    };
    auto multiply = [&](int buf, int at) {
        uint4 x[kSteps][NT], nw[kSteps];
#pragma unroll
        for (int u = 0; u < kSteps; ++u) {
#pragma unroll
            for (int n = 0; n < NT; ++n) x[u][n] = at + u < last && n * 8 + g < p.M ? xr[n][(at + u) * 4] : zero;
            if (NORM) nw[u] = at + u < last ? *(reinterpret_cast<const uint4*>(p.norm_w) + (at + u) * 4 + t) : zero;
        }
#pragma unroll
        for (int u = 0; u < kSteps; ++u) step(a[buf][u], b[buf][u], x[u], nw[u]);
    };
    if constexpr (STAGED) {
        uint4 x[kShare][NT], nw[kShare];
#pragma unroll
        for (int u = 0; u < kShare; ++u) {
#pragma unroll
            for (int n = 0; n < NT; ++n) x[u][n] = first + u < last && n * 8 + g < p.M ? xr[n][(first + u) * 4] : zero;
            if (NORM) nw[u] = first + u < last ? *(reinterpret_cast<const uint4*>(p.norm_w) + (first + u) * 4 + t) : zero;
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
        for (int u = 0; u < kShare; ++u)
            if (first + u < last) step(staged[u * 64], staged[u * 64 + 32], x[u], nw[u]);
    } else if (BUFS == 1) {
        multiply(0, first);
    } else {
        for (int at = first; at < last; at += BUFS * kSteps) {
#pragma unroll
            for (int i = 0; i < BUFS; ++i) {
                multiply(i, at + i * kSteps);
                fetch(i, at + (BUFS + i) * kSteps);
            }
        }
    }
#pragma unroll
    for (int n = 0; n < NT; ++n) {
        float* part = &s_part[warp][(n * 8 + 2 * t) * kTokenPitch + g];
        part[0] = acc[n][0];
        part[kTokenPitch] = acc[n][1];
        part[8] = acc[n][2];
        part[kTokenPitch + 8] = acc[n][3];
        if (NORM) {
            ss[n] += __shfl_xor_sync(0xffffffffu, ss[n], 1);
            ss[n] += __shfl_xor_sync(0xffffffffu, ss[n], 2);
            if (t == 0) s_ssq[warp][n * 8 + g] = ss[n];
        }
    }
    __syncthreads();

    float v0 = 0.f, v1 = 0.f;
    if (finishes) {
#pragma unroll
        for (int i = 0; i < WARPS; ++i) {
            v0 += s_part[i][m * kTokenPitch + f];
            v1 += s_part[i][m * kTokenPitch + 8 + f];
        }
        if (NORM) {
            float sum = 0.f;
#pragma unroll
            for (int i = 0; i < WARPS; ++i) sum += s_ssq[i][m];
            const float rstd = rsqrtf(sum / static_cast<float>(p.K) + p.norm_eps);
            v0 *= rstd;
            v1 *= rstd;
        }
        v0 += bias0;
        v1 += bias1;
    }
    if (KIND == kHeads) {
        // the projection's own output, as it would be stored; then head norm, rotation, store
        v0 = round_bf16(v0);
        v1 = round_bf16(v1);
        cluster_wait();
        if (head_w != nullptr) {   // (the same for a whole cluster)
            float sq = v0 * v0 + v1 * v1;
            sq += __shfl_xor_sync(0xffffffffu, sq, 4);
            sq += __shfl_xor_sync(0xffffffffu, sq, 2);
            sq += __shfl_xor_sync(0xffffffffu, sq, 1);
            if (finishes) store_in_cluster(&s_head[rank][m], f, sq);   // thread f tells rank f
            cluster_arrive();
            cluster_wait();
            if (finishes) {
                float sum = 0.f;
#pragma unroll
                for (int i = 0; i < kHeadRanks; ++i) sum += s_head[i][m];
                const float scale = rsqrtf(sum / 128.f + p.qk_eps);
                v0 = round_bf16(v0 * scale * w0);
                v1 = round_bf16(v1 * scale * w1);
            }
        }
        if (!live) return;
        float r0 = v0, r1 = v1;   // (values as they are: 0 times what is not finite would reach the other half)
        if (head_kind < 2) {
            r0 = v0 * cs - v1 * sn;
            r1 = v1 * cs + v0 * sn;
        }
        __nv_bfloat16* dst = nullptr;
        if (head_kind == 0)
            dst = p.y + m * p.y_pitch + head * 128;
        else if (slot >= 0)
            dst = (head_kind == 1 ? p.k_cache : p.v_cache) +
                  (static_cast<int64_t>(slot) * p.kv_heads + head - p.q_heads - (head_kind == 2 ? p.kv_heads : 0)) * 128;
        if (dst != nullptr) {
            dst[rank * 8 + f] = __float2bfloat16_rn(r0);
            dst[64 + rank * 8 + f] = __float2bfloat16_rn(r1);
        }
        return;
    }
    if (!live) return;
    if (KIND == kResidual) {
        __nv_bfloat16* r = p.residual + static_cast<int64_t>(m) * p.n_out;
        r[n0] = __float2bfloat16_rn(round_bf16(v0) + __bfloat162float(r[n0]));
        if (n1 < p.n_out) r[n1] = __float2bfloat16_rn(round_bf16(v1) + __bfloat162float(r[n1]));
        return;
    }
    store_plain(p, gated, m, n0, n1, v0, v1);
}

// Experts: group g multiplies rows [offsets[g], offsets[g] + counts[g]) of x by its own n_rows rows of w.  A handful of rows
// per group: a CTA keeps its 16 rows of W in registers (BUFS buffers hold a warp's whole share of K) and takes the group's
// rows 8 at a time.  The group table comes from the kernel before, so nothing is requested ahead of the wait.  No tiles of 128
// rows of W and 32 of x to fill, and no ring to drain between a CTA's few k-blocks: 64 experts of 3 x 1024 x 2048, 32 tokens
// with 4 experts each, 12 layers: 2.37 ms per decode step against 2.61.
template <int BUFS>
__global__ void __launch_bounds__(256)
narrow_grouped_kernel(const NarrowParams p, const int32_t* __restrict__ counts, const int32_t* __restrict__ offsets) {
    constexpr int WARPS = 8;
    __shared__ float s_part[WARPS][8 * kTokenPitch];
    pdl_launch_dependents();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int tile = static_cast<int>(blockIdx.x), group = static_cast<int>(blockIdx.y);
    const bool gated = p.up_row_offset > 0;
    const int row_a = gated ? tile * 8 + g : tile * 16 + g;
    const int row_b = gated ? row_a + p.up_row_offset : min(row_a + 8, p.n_rows - 1);
    const __nv_bfloat16* w = p.w + static_cast<int64_t>(group) * p.n_rows * p.K;
    const uint4* wa = reinterpret_cast<const uint4*>(w + row_a * p.K) + t;
    const uint4* wb = reinterpret_cast<const uint4*>(w + row_b * p.K) + t;
    const int first = warp * p.steps / WARPS, last = (warp + 1) * p.steps / WARPS;
    pdl_wait_prior();
    const int count = counts[group];
    if (count <= 0) return;
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    uint4 a[BUFS * kSteps], b[BUFS * kSteps];
#pragma unroll
    for (int u = 0; u < BUFS * kSteps; ++u) {
        const bool there = first + u < last;
        a[u] = there ? load_weights(wa + (first + u) * 4) : zero;
        b[u] = there ? load_weights(wb + (first + u) * 4) : zero;
    }
    const int64_t row0 = offsets[group];
    const int m = static_cast<int>(threadIdx.x) >> 3, f = static_cast<int>(threadIdx.x) & 7;
    const int n0 = gated ? tile * 8 + f : tile * 16 + f;
    for (int m0 = 0; m0 < count; m0 += 8) {
        const uint4* x = reinterpret_cast<const uint4*>(p.x + (row0 + m0 + min(g, count - 1 - m0)) * p.ldx) + first * 4 + t;
        float acc[4] = {};
        uint4 v[BUFS * kSteps];
#pragma unroll
        for (int u = 0; u < BUFS * kSteps; ++u) v[u] = first + u < last ? x[u * 4] : zero;   // (columns of rows that are not there: unused)
#pragma unroll
        for (int u = 0; u < BUFS * kSteps; ++u) {
            mma_bf16_16816(acc, {a[u].x, b[u].x, a[u].y, b[u].y}, v[u].x, v[u].y);
            mma_bf16_16816(acc, {a[u].z, b[u].z, a[u].w, b[u].w}, v[u].z, v[u].w);
        }
        float* part = &s_part[warp][2 * t * kTokenPitch + g];
        part[0] = acc[0];
        part[kTokenPitch] = acc[1];
        part[8] = acc[2];
        part[kTokenPitch + 8] = acc[3];
        __syncthreads();
        if (threadIdx.x < 64 && m0 + m < count) {
            float v0 = 0.f, v1 = 0.f;
#pragma unroll
            for (int i = 0; i < WARPS; ++i) {
                v0 += s_part[i][m * kTokenPitch + f];
                v1 += s_part[i][m * kTokenPitch + 8 + f];
            }
            store_plain(p, gated, row0 + m0 + m, n0, n0 + 8, v0, v1);
        }
        if (m0 + 8 < count) __syncthreads();
    }
}

template <int KIND, bool NORM, int NT>
cudaError_t launch(const NarrowParams& p, int tiles, cudaStream_t stream) {
    const dim3 cluster(KIND == kHeads ? kHeadRanks : 1, 1, 1);
    auto go = [&](auto kernel, int warps, size_t smem) {
        if (smem > 0) {
            const cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
            if (err != cudaSuccess) return err;
        }
        return launch_kernel(kernel, dim3(tiles), dim3(warps * 32), smem, stream, cluster, p);
    };
    // In a decode step whose projections are all this kernel's (dense models: norms and residual ride in them) the weights are
    // staged in shared memory.  In registers they keep the next kernels' CTAs out: 64 CTAs of 1024 x 3072 with 16 warps and 128
    // registers each wait for empty SMs until gate and up (384 CTAs) end, and then take 4 us to request their weights.  Steps of
    // Qwen3-0.6B, 1 request of 700 keys / 2 of 300 / 5 of 200 to 3000 / 12 of 500: 598 / 627 / 872 / 976 us against 674 / 696 /
    // 987 / 1050.  Elsewhere L1 is worth more to the kernels around than shared memory to this one (Qwen3-MoE, 1 request: 660 us
    // against 649; Saluzen, 2 requests: 426 against 407).
    constexpr bool kStage = NORM || KIND == kResidual;
    auto share_bytes = [](int warps, int bufs) { return kStage ? static_cast<size_t>(warps) * bufs * kSteps * 1024 : 0; };
    // Few tiles: more warps each.  A share of K that one buffer holds needs fewer registers.
    if (tiles <= sm_count() && p.steps > 8 * kSteps) {
        if (p.steps <= 16 * kSteps) return go(narrow_gemm_kernel<KIND, NORM, NT, 16, 1, kStage>, 16, share_bytes(16, 1));
        if constexpr (KIND != kHeads && !NORM) {
            if (p.steps <= 32 * kSteps) return go(narrow_gemm_kernel<KIND, NORM, NT, 16, 2, kStage>, 16, share_bytes(16, 2));
            return go(narrow_gemm_kernel<KIND, NORM, NT, 16, 2, false>, 16, 0);
        }
    }
    if (p.steps <= 8 * kSteps) return go(narrow_gemm_kernel<KIND, NORM, NT, 8, 1, kStage>, 8, share_bytes(8, 1));
    if (p.steps <= 16 * kSteps) return go(narrow_gemm_kernel<KIND, NORM, NT, 8, 2, kStage>, 8, share_bytes(8, 2));
    return go(narrow_gemm_kernel<KIND, NORM, NT, 8, 2, false>, 8, 0);   // (K beyond what is requested ahead)
}

template <int KIND, bool NORM>
cudaError_t launch(const NarrowParams& p, int tiles, cudaStream_t stream) {
    return p.M <= 8 ? launch<KIND, NORM, 1>(p, tiles, stream) : launch<KIND, NORM, 2>(p, tiles, stream);
}

}  // namespace

// Plain projections, us, this kernel against the weight-streaming one of gemm_skinny.cu:
//   * Up to 8 rows it is the faster one, but CTAs with little to load cost more than they bring: 151936 x 64 26 and 17 (2048 x 64
//     2.0 and 3.8), and with K a little above 1024 half of the second register buffer stays empty: 32768 x 1088 21 and 17,
//     32768 x 1536 23 and 22, 16384 x 1088 11.8 and 12.9; 32768 x 2048 with 4 rows 27 and 27.  In a chain of programmatic launches
//     they load beside the kernels before: as the head of a decode step 32768 x 1536 is 10 us ahead, 32768 x 1280 3 to 7 behind.
//   * A long K is walked a buffer at a time behind the wait, where the TMA ring over there keeps more bytes in flight: 2048 x 6144
//     with 4 rows 8.9 and 14.4, 28672 x 4096 43 and 45; 12288 x 2048 with 16 rows 18.6 and 16.1.
//   * Two tiles of tokens double a warp's operands and products; with more than 1024 columns and more CTAs than SMs it is ahead
//     up to 6144 rows of W only (16 rows: 6144 x 1536 9.6 and 10.4, 8192 x 1536 12.0 and 11.2, with SwiGLU 12.1 and 10.4), with more
//     than 2048 columns only without a gate (4096 x 3072 10.6 and 11.1; 3584 x 3584 with SwiGLU 11.1 and 10.8).
// With the norm (and the chain of a decode step around it: the residual, the heads), every CTA computes it, which grows with K
// and with the CTAs: a step of 12 layers against the split-K kernel with folded norms (us)
//   hidden 768   1 request 254, 371   8: 279, 401   16: 312, 409     hidden 1024, gate and up of 16 MB   1: 330, 412   8: 356, 438   16: 428, 444
//   hidden 1280  1 request 407, 475   8: 479, 491   16: 654, 498     ... of 32 MB   1: 414, 508   4: 502, 524   8: 564, 548
//   hidden 2048  1 request 636, 650   4: 693, 675   8: 709, 695
bool narrow_gemm_takes(const void* x, const void* w, int M, int N, int K, int64_t ldx, int epilogue, bool normed) {
    const int64_t bytes = static_cast<int64_t>(N) * K * 2;
    if (normed && (K > (M <= 2 ? 2048 : 1024) || (M > 4 && bytes > (18ll << 20)))) return false;
    const int n_out = epilogue_is_gated(epilogue) ? N / 2 : N;
    const bool light = bytes <= (26ll << 20);
    bool faster;
    if (N > 8192 && K < 512)
        faster = false;
    else if (M <= 8)
        faster = K <= 1024 || light || (K <= 2048 && (N <= 16384 || (M <= 4 && K > 31 * 64) || (K >= 1536 && pdl_launches_enabled())));
    else
        faster = M <= kNarrowRows && light &&
                 (K <= 1024 || div_ceil(N, 16) <= sm_count() || (K <= 2048 ? N <= 6144 : N <= 4096 && !epilogue_is_gated(epilogue)));
    return M >= 1 && faster && n_out % 8 == 0 && K % 32 == 0 && ldx % 8 == 0 &&
           ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w)) & 15) == 0;
}

// How rows fall to groups is not known here, so the rule is by the worst of it: every row in as few groups as there can be.
// What this kernel gains by starting at once (two launches of a layer together 20 us) goes into CTAs of groups without rows,
// 0.65 ns each, and into turns after a CTA's first 8 rows, 2.2 ns more than the 256 columns that the other kernel takes at once.
// Layers (us, this kernel against the other one; rows spread at random, and all tokens with the same experts):
//   64 experts of 2 x 1024 x 2048, 4 per token   48 tokens 162, 182 and 58, 59;   64: 170, 186 and 65, 61;   128: 185, 190 and 87, 70
//   128 of 2 x 768 x 2048, 8 per token            8 tokens 129, 148 and 68, 67;   32: 225, 238 and 82, 70;   128: 281, 276 and 136, 84
//   32 of 2 x 1024 x 2048, 2 per token           64 tokens 96, 97 and 42, 53;    128: 104, 99 and 58, 61
bool narrow_grouped_takes(const void* x, const void* w, int64_t total_rows, int max_rows, int num_groups, int n_out, int K, int epilogue) {
    const int64_t tiles = epilogue_is_gated(epilogue) ? div_ceil(n_out, 8) : div_ceil(n_out, 16);
    const int64_t turns = max_rows > 8 ? tiles * total_rows * (max_rows - 8) / (8ll * max_rows) : 0;
    return 0.65 * tiles * num_groups + 2.2 * turns <= 11000. && total_rows <= 8ll * num_groups && num_groups <= 65535 && K <= 64 * 32 &&
           K % 32 == 0 && n_out % 8 == 0 && ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w)) & 15) == 0;
}

int launch_narrow_grouped(void* y, const void* x, const void* w, const int32_t* counts, const int32_t* offsets, int num_groups, int N,
                          int K, int epilogue, cudaStream_t stream, float act_limit) {
    const bool gated = epilogue_is_gated(epilogue);
    NarrowParams p = {};
    p.y = static_cast<__nv_bfloat16*>(y);
    p.x = static_cast<const __nv_bfloat16*>(x);
    p.w = static_cast<const __nv_bfloat16*>(w);
    p.n_rows = N;
    p.n_out = gated ? N / 2 : N;
    p.up_row_offset = gated ? N / 2 : 0;
    p.steps = K / 32;
    p.epilogue = epilogue;
    p.ldx = p.K = K;
    p.y_pitch = p.n_out;
    p.act_limit = act_limit;
    const dim3 grid(gated ? div_ceil(p.n_out, 8) : div_ceil(N, 16), num_groups);
    auto kernel = p.steps <= 8 * kSteps ? narrow_grouped_kernel<1> : narrow_grouped_kernel<2>;
    B200_CHECK_CUDA(launch_kernel(kernel, grid, dim3(256), 0, stream, dim3(1, 1, 1), p, counts, offsets));
    return B200_OK;
}

int launch_narrow_gemm(void* y, const void* x, const void* w, const void* bias, int M, int N, int K, int64_t ldx, int epilogue,
                       int* status, cudaStream_t stream, const NarrowFusion* fuse, float act_limit) {
    const bool gated = epilogue_is_gated(epilogue);
    const HeadEpilogue* h = fuse ? fuse->heads : nullptr;
    NarrowParams p = {};
    p.y = static_cast<__nv_bfloat16*>(y);
    p.x = static_cast<const __nv_bfloat16*>(x);
    p.w = static_cast<const __nv_bfloat16*>(w);
    p.bias = static_cast<const __nv_bfloat16*>(bias);
    p.norm_w = fuse ? static_cast<const __nv_bfloat16*>(fuse->norm_w) : nullptr;
    p.norm_eps = fuse ? fuse->eps : 0.f;
    p.residual = fuse ? static_cast<__nv_bfloat16*>(fuse->residual) : nullptr;
    p.M = M;
    p.n_rows = N;
    p.n_out = gated ? N / 2 : N;
    p.up_row_offset = gated ? N / 2 : 0;
    p.steps = K / 32;
    p.epilogue = epilogue;
    p.ldx = ldx;
    p.K = K;
    p.y_pitch = p.n_out;
    p.act_limit = act_limit;
    p.status = status;
    p.early = K < kWalkedK ? 1 : 0;
    if (h != nullptr) {
        B200_CHECK_ARG(!gated && N == (h->q_heads + 2 * h->kv_heads) * 128,
                       "linear: the head epilogue wants a plain projection of (q_heads + 2 kv_heads) x 128 features");
        p.q_norm_w = static_cast<const __nv_bfloat16*>(h->q_norm_w);
        p.k_norm_w = static_cast<const __nv_bfloat16*>(h->k_norm_w);
        p.cos_t = h->cos_t;
        p.sin_t = h->sin_t;
        p.positions = h->positions;
        p.out_loc = h->out_loc;
        p.k_cache = static_cast<__nv_bfloat16*>(h->k_cache);
        p.v_cache = static_cast<__nv_bfloat16*>(h->v_cache);
        p.q_heads = h->q_heads;
        p.kv_heads = h->kv_heads;
        p.max_pos = h->max_pos;
        p.num_slots = h->num_slots;
        p.qk_eps = h->eps;
    }
    const int tiles = gated ? div_ceil(p.n_out, 8) : div_ceil(N, 16);
    cudaError_t err;
    if (h != nullptr)
        err = p.norm_w ? launch<kHeads, true>(p, tiles, stream) : launch<kHeads, false>(p, tiles, stream);
    else if (p.residual != nullptr)
        err = launch<kResidual, false>(p, tiles, stream);
    else
        err = p.norm_w ? launch<kPlain, true>(p, tiles, stream) : launch<kPlain, false>(p, tiles, stream);
    B200_CHECK_CUDA(err);
    return B200_OK;
}

}  // namespace b200
