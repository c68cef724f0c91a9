// y = x W^T for a handful of rows and a W that takes longer to read than a kernel takes to start: one CTA per SM streams its
// share of W through a ring in shared memory.
//
// What bounds it is the memory, and what keeps a kernel from the memory's rate here is that nothing is requested while a CTA
// finishes, while the next one starts, and while the kernel before ends.  So
//   * a CTA walks over tiles of 16 rows of W; one thread does nothing but request them, 16 KB at a time (512 of K: one copy, or two
//     where gate and up rows lie apart) and x of the same columns, as far ahead as the ring goes, from one tile to the next
//     without a break (x by the multiplying warps themselves, two stages ahead: trips to L2 beside a memory in full use take 1500
//     cycles, 97 us more for an expert layer);
//   * the weights do not depend on the kernel before, so the ring fills with them ahead of griddepcontrol.wait;
//   * the ring holds 96 KB of weights (64 KB, so that two CTAs share an SM: 3350 us per step of Llama-3-8B with 4 requests against
//     3077; 128 KB 3134).
// A warp multiplies 64 of a stage's 512 columns: 16 bytes of a row are operands of two mma.sync products as they are (as in
// gemm_narrow.cu), the sums of the eight warps meet once per tile.
//
// Experts (GROUPED): the same over the tiles of all groups that have rows, 8 rows at a time.
#include "common.cuh"
#include "kernels.h"
#include "narrow.cuh"
#include "tensormap.cuh"

namespace b200 {
namespace {

constexpr int kChunk = 512;                        // columns per stage, 64 per warp
constexpr uint32_t kWBytes = 16 * kChunk * 2, kXBytes = 8 * kChunk * 2;   // of a stage, x per block of 8 tokens
constexpr int kStages = 6;
constexpr int kWideStages = 4;                     // GROUPED, where many groups have more than 8 rows
constexpr uint32_t ring_bytes(int blocks) { return kStages * (kWBytes + blocks * kXBytes); }
static_assert(kWideStages * (kWBytes + 2 * kXBytes) <= ring_bytes(1), "");
constexpr int kWarps = 8;                          // that multiply; one more requests
constexpr int kMaxRingGroups = 1024;

struct RingPass {   // of a group's rows over its weights
    int group, x_row, count;
};

struct RingShared {
    alignas(8) uint64_t full[kStages];
    alignas(8) uint64_t empty[kStages];
    float part[2][kWarps][8 * kTokenPitch];
    int passes, wide;
};

struct RingParams : NarrowOut {
    const __nv_bfloat16* bias;
    int M, n_rows, up_row_offset, tiles, chunks, K;
    int x_box;        // rows of x per copy
    int early;        // let the next kernel's CTAs in at once
    int* status;
    const int32_t *counts, *offsets;   // GROUPED
    int groups;
};

// A CTA's share: tiles of every pass.  BLOCKS of 8 tokens (GROUPED: at most that many of a group in one pass over its weights).
template <bool GROUPED, int BLOCKS, int STAGES>
__device__ __forceinline__ void ring_walk(const CUtensorMap& tmap_w, const CUtensorMap& tmap_x, const RingParams& p, uint32_t ring,
                                          const RingPass* s_pass, RingShared& s, int warp, int lane) {
    constexpr uint32_t kStageBytes = kWBytes + BLOCKS * kXBytes;
    const bool gated = p.up_row_offset > 0;
    // this CTA's tiles: neighbours, so that experts change rarely
    const int64_t items = static_cast<int64_t>(GROUPED ? s.passes : 1) * p.tiles;
    const int first = static_cast<int>(items * blockIdx.x / gridDim.x), last = static_cast<int>(items * (blockIdx.x + 1) / gridDim.x);
    bool failed = false;

    // a place in the walk: stepped, not found by division
    struct Place {
        int pass, tile, w_row, x_row, count;
    };
    auto open = [&](Place& at) {
        const RingPass r = GROUPED ? s_pass[at.pass] : RingPass{0, 0, p.M};
        at.w_row = r.group * p.n_rows + at.tile * (gated ? 8 : 16);
        at.x_row = r.x_row;
        at.count = r.count;
    };
    auto start = [&]() {
        Place at = {GROUPED ? first / p.tiles : 0, GROUPED ? first % p.tiles : first, 0, 0, 0};
        if (first < last) open(at);
        return at;
    };
    auto next = [&](Place& at, int item) {   // `item`: the one to come
        ++at.tile;
        at.w_row += gated ? 8 : 16;
        if (GROUPED && at.tile == p.tiles) {
            at.tile = 0;
            ++at.pass;
            if (item < last) open(at);
        }
    };

    if (warp == kWarps) {
        // ================= requests =================
        if (lane == 0) {
            auto request_w = [&](const Place& at, int c, uint32_t slot) {
                const uint32_t bar = smem_u32(&s.full[slot]), dst = ring + slot * kStageBytes;
                mbar_arrive_expect_tx(bar, kWBytes + (GROUPED && BLOCKS > 1 && at.count > 8 ? 2 : 1) * p.x_box * (kChunk * 2));
                tma_load_3d(dst, &tmap_w, 0, at.w_row, c * (kChunk / 64), bar);
                if (gated) tma_load_3d(dst + kWBytes / 2, &tmap_w, 0, at.w_row + p.up_row_offset, c * (kChunk / 64), bar);
            };
            auto request_x = [&](const Place& at, int c, uint32_t slot) {
                const uint32_t dst = ring + slot * kStageBytes + kWBytes;
                tma_load_3d(dst, &tmap_x, 0, at.x_row, c * (kChunk / 64), smem_u32(&s.full[slot]));
                if (GROUPED && BLOCKS > 1 && at.count > 8)
                    tma_load_3d(dst + kXBytes, &tmap_x, 0, at.x_row + 8, c * (kChunk / 64), smem_u32(&s.full[slot]));
            };
            // the first ring-full of weights does not wait for the kernel before this one
            const int early = GROUPED ? 0 : min(STAGES, (last - first) * p.chunks);
            Place ahead = start();
            for (int i = 0, c = 0; i < early; ++i) {
                request_w(ahead, c, i);
                if (++c == p.chunks) {
                    c = 0;
                    next(ahead, first + (i + 1) / p.chunks);
                }
            }
            if (!GROUPED) pdl_wait_prior();
            uint32_t slot = 0, phase = 1;   // (the first waits are for stages that nobody has used)
            int it = 0;
            Place at = start();
            for (int item = first; item < last && !failed; next(at, ++item)) {
                for (int c = 0; c < p.chunks; ++c, ++it) {
                    if (!mbar_wait_mostly_ready(smem_u32(&s.empty[slot]), phase, p.status, 131)) {
                        failed = true;
                        break;
                    }
                    if (it >= early) request_w(at, c, slot);
                    request_x(at, c, slot);
                    if (++slot == STAGES) {
                        slot = 0;
                        phase ^= 1;
                    }
                }
            }
        }
        return;
    }

    // ================= products =================
    if (!GROUPED) pdl_wait_prior();
    const int g = lane >> 2, t = lane & 3;
    // Rows of the operands are rows of W, and tokens, in an order in which neighbouring lanes' 16 bytes lie in different banks.
    const int local = (g >> 1) | ((g & 1) << 2);
    const uint32_t row_a = static_cast<uint32_t>(warp) * (gated ? 1024u : 2048u) + local * 128;
    const uint32_t row_b = row_a + (gated ? kWBytes / 2 : 1024u);
    const uint32_t at[2] = {static_cast<uint32_t>(t ^ local) << 4, static_cast<uint32_t>((t + 4) ^ local) << 4};
    // (x has p.x_box rows per block of 64 columns; what a token that is not there reads is used by nobody)
    const uint32_t x_local = static_cast<uint32_t>(warp) * p.x_box + local;
    const uint32_t row_x = kWBytes + x_local * 128;
    const uint32_t at_x[2] = {(static_cast<uint32_t>(t) ^ (x_local & 7)) << 4, (static_cast<uint32_t>(t + 4) ^ (x_local & 7)) << 4};
    auto lds = [&](uint32_t from) {
        uint4 v;
        asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(from) : "memory");
        return v;
    };
    uint32_t slot = 0, phase = 0;
    int parity = 0;
    Place here = start();
    for (int item = first; item < last; next(here, ++item)) {
        float acc[BLOCKS][4] = {};
        for (int c = 0; c < p.chunks; ++c) {
            if (!failed && !mbar_wait_mostly_ready(smem_u32(&s.full[slot]), phase, p.status, 132)) failed = true;
            const uint32_t base = ring + slot * kStageBytes;
            // (columns behind K are zeros in both operands)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint4 a = lds(base + row_a + at[h]), b = lds(base + row_b + at[h]);
#pragma unroll
                for (int i = 0; i < BLOCKS; ++i) {
                    if (GROUPED && i > 0 && here.count <= i * 8) break;
                    const uint4 v = lds(base + row_x + i * (GROUPED ? kXBytes : 1024u) + at_x[h]);
                    mma_bf16_16816(acc[i], {a.x, b.x, a.y, b.y}, v.x, v.y);
                    mma_bf16_16816(acc[i], {a.z, b.z, a.w, b.w}, v.z, v.w);
                }
            }
            mbar_release_stage(smem_u32(&s.empty[slot]), lane);
            if (++slot == STAGES) {
                slot = 0;
                phase ^= 1;
            }
        }
        const int m = static_cast<int>(threadIdx.x) >> 3, f = static_cast<int>(threadIdx.x) & 7;
        const int n0 = here.tile * (gated ? 8 : 16) + f;
#pragma unroll
        for (int i = 0; i < BLOCKS; ++i) {
            if (GROUPED && i > 0 && here.count <= i * 8) break;
            // a thread's two tokens are t and t + 4
            float* part = &s.part[parity][warp][t * kTokenPitch + local];
            part[0] = acc[i][0];
            part[4 * kTokenPitch] = acc[i][1];
            part[8] = acc[i][2];
            part[4 * kTokenPitch + 8] = acc[i][3];
            // (two buffers: whoever writes one of them again has passed the barrier in between)
            asm volatile("bar.sync 1, %0;" ::"n"(kWarps * 32) : "memory");
            if (threadIdx.x < 64 && i * 8 + m < here.count && n0 < p.n_out) {
                float v0 = 0.f, v1 = 0.f;
#pragma unroll
                for (int w = 0; w < kWarps; ++w) {
                    v0 += s.part[parity][w][m * kTokenPitch + f];
                    v1 += s.part[parity][w][m * kTokenPitch + 8 + f];
                }
                if (!gated && p.bias != nullptr) {
                    v0 += __bfloat162float(p.bias[n0]);
                    if (n0 + 8 < p.n_out) v1 += __bfloat162float(p.bias[n0 + 8]);
                }
                store_plain(p, gated, static_cast<int64_t>(here.x_row) + i * 8 + m, n0, n0 + 8, v0, v1);
            }
            parity ^= 1;
        }
    }
}

template <bool GROUPED, int BLOCKS>
__global__ void __launch_bounds__((kWarps + 1) * 32)
ring_gemm_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x, const RingParams p) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ RingShared s;
    const int warp = static_cast<int>(threadIdx.x) >> 5, lane = static_cast<int>(threadIdx.x) & 31;
    const uint32_t ring = (smem_u32(smem_raw) + 1023u) & ~1023u;
    RingPass* passes = reinterpret_cast<RingPass*>(smem_raw + (ring - smem_u32(smem_raw)) + ring_bytes(BLOCKS));

    if (p.early) pdl_launch_dependents();
    if (threadIdx.x == 0) {
        for (int i = 0; i < kStages; ++i) {
            mbar_init(smem_u32(&s.full[i]), 1);
            mbar_init(smem_u32(&s.empty[i]), kWarps);
        }
        fence_mbar_init();
        tma_prefetch_desc(&tmap_w);
        tma_prefetch_desc(&tmap_x);
    }
    if (GROUPED) {
        pdl_wait_prior();   // (the group table comes from the kernel before this one)
        if (warp == 0) {
            // 16 rows per pass where that saves a third of the passes.  (Where one expert with more than 8 rows was enough for it, all the
            // others paid: 64 experts of 2 x 1024 x 2048, 4 per token, a quarter of 32 tokens with the same experts 144.5 us per layer
            // against 127.6, all of them 44.7 and 45.2; steps of 12 such layers, 24 requests of a batch of 32 2283 us against 2087.)
            int narrow_passes = 0, wide_passes = 0;
            for (int g = lane; g < p.groups; g += 32) {
                const int rows = max(p.counts[g], 0);
                narrow_passes += (rows + 7) / 8;
                wide_passes += (rows + 15) / 16;
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                narrow_passes += __shfl_xor_sync(0xffffffffu, narrow_passes, o);
                wide_passes += __shfl_xor_sync(0xffffffffu, wide_passes, o);
            }
            const bool wide = 2 * narrow_passes >= 3 * wide_passes;
            const int width = wide ? 16 : 8;
            int total = 0;
            for (int base = 0; base < p.groups; base += 32) {
                const int g = base + lane;
                const int rows = g < p.groups ? max(p.counts[g], 0) : 0, n = (rows + width - 1) / width;
                int incl = n;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int up = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl += up;
                }
                const int row0 = n > 0 ? p.offsets[g] : 0;
                for (int i = 0; i < n; ++i) passes[total + incl - n + i] = {g, row0 + i * width, min(rows - i * width, width)};
                total += __shfl_sync(0xffffffffu, incl, 31);
            }
            if (lane == 0) {
                s.passes = total;
                s.wide = wide;
            }
        }
    }
    __syncthreads();
    if (GROUPED && s.wide)
        ring_walk<true, 2, kWideStages>(tmap_w, tmap_x, p, ring, passes, s, warp, lane);
    else
        ring_walk<GROUPED, BLOCKS, kStages>(tmap_w, tmap_x, p, ring, passes, s, warp, lane);
}

// [rows, K] bf16 as 64-column blocks of rows: boxes of `box_rows` rows x 512 columns under the 128-byte swizzle.
int make_ring_tmap(CUtensorMap* out, const void* w, int64_t rows, int K, int64_t ld, int box_rows) {
    struct Entry {
        const void* w = nullptr;
        int64_t rows, ld;
        int K, box_rows;
        CUtensorMap map;
    };
    constexpr int kEntries = 1024;
    thread_local Entry cache[kEntries];   // (encoding a tensor map costs about a microsecond)
    Entry& e = cache[(reinterpret_cast<uintptr_t>(w) * 0x9E3779B97F4A7C15ull >> 20) % kEntries];
    if (e.w != w || e.rows != rows || e.ld != ld || e.K != K || e.box_rows != box_rows) {
        EncodeTiledFn fn = encode_tiled_fn();
        if (!fn) {
            set_last_error("cuTensorMapEncodeTiled is not available from this driver");
            return B200_ERR_CUDA;
        }
        const cuuint64_t dims[3] = {64, static_cast<cuuint64_t>(rows), static_cast<cuuint64_t>(K / 64)};
        const cuuint64_t strides[2] = {static_cast<cuuint64_t>(ld) * 2, 128};
        const cuuint32_t box[3] = {64, static_cast<cuuint32_t>(box_rows), kChunk / 64};
        const cuuint32_t es[3] = {1, 1, 1};
        e.w = nullptr;
        const CUresult r = fn(&e.map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(w), dims, strides, box, es,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) {
            set_last_error("cuTensorMapEncodeTiled (weight blocks) failed with CUresult %d", static_cast<int>(r));
            return B200_ERR_CUDA;
        }
        e.w = w;
        e.rows = rows;
        e.ld = ld;
        e.K = K;
        e.box_rows = box_rows;
    }
    *out = e.map;
    return B200_OK;
}

int launch_ring(RingParams p, const void* x, int64_t x_rows, int64_t ldx, const void* w, int64_t w_rows, bool grouped, cudaStream_t stream) {
    const bool gated = p.up_row_offset > 0;
    const int blocks = grouped || p.M <= 8 ? 1 : 2;
    CUtensorMap tmap_w, tmap_x;
    p.x_box = grouped ? 8 : p.M;   // (rows that a copy has to fill with zeros cost it: 151936 x 1024 with 1 row 66 us, with 4 rows 52)
    int err = make_ring_tmap(&tmap_w, w, w_rows, p.K, p.K, gated ? 8 : 16);
    if (err == B200_OK) err = make_ring_tmap(&tmap_x, x, x_rows, p.K, ldx, p.x_box);
    if (err != B200_OK) return err;
    p.tiles = gated ? div_ceil(p.n_out, 8) : div_ceil(p.n_rows, 16);
    p.chunks = div_ceil(p.K, kChunk);
    auto kernel = grouped ? ring_gemm_kernel<true, 1> : blocks == 1 ? ring_gemm_kernel<false, 1> : ring_gemm_kernel<false, 2>;
    const size_t smem = ring_bytes(blocks) + 1024 +
                        (grouped ? (p.groups + x_rows / 8 + 1) * sizeof(RingPass) : 0);
    const int grid = grouped || p.tiles > sm_count() ? sm_count() : p.tiles;
    B200_CHECK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
    B200_CHECK_CUDA(launch_kernel(kernel, dim3(grid), dim3((kWarps + 1) * 32), smem, stream, dim3(1, 1, 1), tmap_w, tmap_x, p));
    return B200_OK;
}

bool aligned16(const void* a, const void* b) { return ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b)) & 15) == 0; }

RingParams ring_params(void* y, int N, int K, int epilogue, float act_limit, int* status) {
    const bool gated = epilogue_is_gated(epilogue);
    RingParams p = {};
    p.y = static_cast<__nv_bfloat16*>(y);
    p.n_out = gated ? N / 2 : N;
    p.epilogue = epilogue;
    p.y_pitch = p.n_out;
    p.act_limit = act_limit;
    p.early = 1;
    p.n_rows = N;
    p.up_row_offset = gated ? N / 2 : 0;
    p.K = K;
    p.status = status;
    return p;
}

}  // namespace

// Rows of W long and many enough to outlast the start of a walk.  us, this kernel against the ones of gemm_skinny.cu and (the first
// three lines) gemm_narrow.cu, weights not in L2:
//   1 x 4096 x 1024 6.2, 5.7;  1 x 8192 x 1024 8.3, 6.3;  16 x 6144 x 1024 with SwiGLU 8.0, 6.2;  1 x 151936 x 1024 51, 48
//   8 x 4096 x 2048 8.3, 8.2;  1 x 6144 x 2048 8.4, 10.2;  1 x 2048 x 6144 8.3, 10.3;  16 rows of it 10.3, 10.3
//   16 x 4096 x 2048 8.3, 10.0;  16 x 2048 x 2048 6.2, 6.2;  16 x 1024 x 4096 6.9, 7.1;  16 x 6144 x 2048 10.3, 12.3
//   8 x 4096 x 4096 10.3, 14.4;  8 x 6144 x 4096 12.6, 20.2;  8 x 4096 x 14336 22.8, 29.4;  16 x 4096 x 14336 24.7, 30.0
//   8 x 28672 x 4096 with SwiGLU 41.1, 46.4;  9 rows of it 43.2, 46.4;  8 x 128256 x 4096 155, 167
// Steps: Llama-3-8B, 1 request 2906 us against 3542, 4 requests 3025 against 3726, 8 requests 3097 against 3745; Saluzen, 12 requests 470
// against 566, 16 requests 498 against 594.
//
// Where the registers' kernel would take the call it is ahead up to 8 rows while the ring's CTAs have one tile each and some a second one,
// and its warps request their whole share of K at once (K up to 4096): 1 row / 8 rows, programmatic launches, the ring first
//   3328 x 3840 6.9, 5.7 / 6.9, 6.2;  3584 x 3712 6.7, 5.8 / 6.8, 6.3;  3840 x 3328 6.2, 5.7 / 6.3, 6.2;  4096 x 3264 6.4, 5.7 / 6.6, 6.3
//   4736 x 2688 (two tiles each) 6.2, 6.2 / 6.2, 6.4;  4800 x 2688 7.4, 8.8 / 7.5, 9.2;  3072 x 4352 8.1, 8.6 / 8.2, 9.0;  9 rows of 3328 x 3840 7.5, 9.0
// Fewer tiles than SMs are no reason against the ring: 512 x 24576 14.1, 16.0 / 14.1, 16.8; 1024 x 12288 8.5, 10.2 / 8.5, 10.7;
// 512 x 32768 17.5, 27.2 against the weight-streaming kernel.
bool ring_gemm_takes(const void* x, const void* w, int M, int N, int K, int64_t ldx, int epilogue, bool narrow) {
    const int n_out = epilogue_is_gated(epilogue) ? N / 2 : N;
    const int tiles = div_ceil(N, 16);
    const bool uneven = M <= 8 && K <= 4096 && tiles > sm_count() && tiles < 2 * sm_count();
    const bool large = narrow ? static_cast<int64_t>(N) * K >= 12ll << 20 && !uneven : static_cast<int64_t>(N) * K >= 4ll << 20;
    return M >= 1 && M <= 16 && K >= 2048 && large && n_out % 8 == 0 && K % 64 == 0 && ldx % 8 == 0 && aligned16(x, w);
}

int launch_ring_gemm(void* y, const void* x, const void* w, const void* bias, int M, int N, int K, int64_t ldx, int epilogue, int* status,
                     cudaStream_t stream, float act_limit) {
    RingParams p = ring_params(y, N, K, epilogue, act_limit, status);
    p.bias = static_cast<const __nv_bfloat16*>(bias);
    p.M = M;
    // Where the registers' kernel would take the call, the next kernels are let in as that one lets them in: 2048 x 6144 with 16 rows
    // at the end of a layer is no faster with them let in at once, 501 us per step against 498.
    p.early = K < kWalkedK || !narrow_gemm_takes(x, w, M, N, K, ldx, epilogue);
    return launch_ring(p, x, M, ldx, w, N, false, stream);
}

// Of the calls that narrow_grouped_takes: many groups, and few enough rows that a group with all of them does not take more turns than
// there.  A K of three whole stages and more hides what a tile costs beside its weights (the warps' sums meet, a stage fills only in
// part), one of two does where there are many tiles; with a shorter one the kernel is ahead only of what a launch of CTAs for groups without
// rows costs there.  us that this kernel adds to a layer in which narrow_grouped_kernel runs, and the layer with that (one projection
// at a time; rows spread at random, and all tokens with the same experts, 4 per token unless stated):
//   64 experts, 2 x 1024 x 2048   1 token -6.1 of 36;   8 -8.8 of 82, -5.4 of 35;   24 -15.4 of 137, -1.4 of 42;
//       32 -15.3 of 147, -3.1 of 47;   48 -17.4 of 161, +0.1 of 53
//   32 experts of it             1 token -1.1 of 26;   8 -3.3 of 61, -2.9 of 28;   24 -9.7 of 88, +2.2 of 37;   32 -8.9 of 92, -1.1 of 42;
//       48 -8.0 of 98, +4.2 of 49
//   32 experts, 2 x 512 x 1536   1 token -0.3 of 19;   16 -2.0 of 41, -0.1 of 22;   24 -2.3 of 47, +0.1 of 26;   32 -2.2 of 47, +0.0 of 27
//   64 experts, 1024 x 2048      1 token -0.2 of 34;   8 -1.1 of 73, -3.7 of 38;   32 -9.1 of 160, +0.7 of 43;   48 -12.1 of 183, +1.0 of 50
//   64 experts, 2048 x 1024      1 token -3.1 of 36;   8 +3.1 of 82, -3.9 of 35;   16 +1.8 of 109, -5.2 of 42;   32 +1.0 of 147, -1.4 of 47;
//       48 -0.8 of 161, +2.2 of 53
//   32 experts of it             1 token -0.1 of 26;   8 +2.2 of 61, -1.7 of 28;   32 +0.3 of 92, -0.3 of 42;   48 +1.4 of 98, +3.0 of 49
//   64 experts, 2048 x 768       1 token -2.2 of 30;   8 +3.1 of 68, -4.0 of 32;   32 +6.6 of 112, -0.5 of 42
//   32 experts, 2048 x 256       1 token -1.1 of 19;   8 +1.2 of 30, +0.1 of 17;   32 +1.3 of 43, +0.5 of 27
//   128 experts, 2048 x 256      1 token -11.4 of 34;   8 -4.8 of 47, -13.1 of 38
//   128 experts, 1536 x 1024     1 token -6.5 of 45;   8 +2.3 of 84, -9.0 of 47;   16 -0.9 of 114, -7.2 of 50
//   128 experts, 1024 x 512, 8 per token   4 tokens -1.0 of 38, -3.0 of 30;   16 +0.5 of 66, -1.4 of 30;   48 +2.4 of 94, -0.8 of 49
//   128 experts, 512 x 1024      1 token +0.2 of 31;   4 +0.5 of 34, -0.1 of 32;   32 +1.2 of 78, -2.6 of 34
// Steps of 12 layers of 64 experts of 2 x 1024 x 2048, gate and up / down as well: 16 requests 1671, 1648 us; 32 2122, 2092; 8 1218, 1214.
bool ring_grouped_takes(const void* x, const void* w, int64_t total_rows, int max_rows, int num_groups, int n_out, int K, int epilogue) {
    const int tiles = epilogue_is_gated(epilogue) ? div_ceil(n_out, 8) : div_ceil(n_out, 16);
    bool faster;
    if (K >= 3 * kChunk)
        faster = total_rows <= (tiles >= 96 ? 4ll : 3ll) * num_groups;
    else if (K >= 2 * kChunk && tiles >= 128 && num_groups >= 64)
        faster = total_rows <= 3ll * num_groups;
    else
        faster = num_groups >= 64 && tiles >= 64 && total_rows * 4 <= num_groups;
    return faster && num_groups >= 32 && num_groups <= kMaxRingGroups && max_rows <= 48 && n_out % 8 == 0 && K % 64 == 0 && aligned16(x, w);
}

int launch_ring_grouped(void* y, const void* x, const void* w, const int32_t* counts, const int32_t* offsets, int num_groups,
                        int64_t total_rows, int N, int K, int epilogue, int* status, cudaStream_t stream, float act_limit) {
    RingParams p = ring_params(y, N, K, epilogue, act_limit, status);
    p.counts = counts;
    p.offsets = offsets;
    p.groups = num_groups;
    return launch_ring(p, x, total_rows, K, w, static_cast<int64_t>(num_groups) * N, true, stream);
}

}  // namespace b200
