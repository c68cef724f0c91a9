// y = x W^T for many rows (prefill batches, M > 256): a persistent tiled GEMM on the tcgen05
// tensor cores.  Bound by the tensor pipe, so the layout is chosen for MMA issue rate:
//   * output tiles of 128 tokens x 256 features; the 128-token block of x is the MMA "A" operand
//     (tokens run along the TMEM lanes), 256 rows of W are the "B" operand; one k-block of 64
//     elements is four 128x256x16 MMAs fed from a 48 KB shared-memory stage (4-stage TMA ring);
//   * one CTA per SM walks its tiles in a fixed order; two 256-column accumulators in TMEM
//     (all 512 columns) let the epilogue of tile i run under the MMAs of tile i+1;
//   * tiles are ordered in bands of 16 token blocks (2048 tokens): inside a band the feature
//     tile moves slowest, so the CTAs running at one time share a few W tiles and the band's x
//     stays in L2 while W streams past once per band;
//   * gated epilogue (gate_up projection + SwiGLU): the B operand is 128 gate rows followed by
//     the 128 matching up rows, so one thread holds gate[m][n] and up[m][n] in the same
//     accumulator and writes act(gate) * up for 128 features.
// Most batches run on pairs of CTAs instead (pair_gemm_kernel below); pick_tile has the line.
#include <math.h>

#include "common.cuh"
#include "kernels.h"
#include "tcgen05.cuh"
#include "tensormap.cuh"

namespace b200 {
namespace {

constexpr int kTM = 128;      // tokens per tile (UMMA M)
constexpr int kTN = 256;      // W rows per tile (UMMA N)
constexpr int kBK = 64;       // bf16 elements per k-block (one 128-byte swizzle row)
constexpr int kStages = 4;
constexpr int kBand = 16;     // token blocks per band
constexpr int kThreads = 192; // warp 0: TMA, warp 1: MMA + TMEM owner, warps 2-5: epilogue
constexpr uint32_t kABytes = kTM * kBK * 2;   // 16 KB
constexpr uint32_t kBBytes = kTN * kBK * 2;   // 32 KB
constexpr uint32_t kStageBytes = kABytes + kBBytes;

struct TileParams {
    __nv_bfloat16* y;           // [M, n_out]
    const __nv_bfloat16* bias;  // [n_out] or NULL (plain epilogue only)
    int M;
    int n_out;          // output features (N, or N/2 with a gated epilogue)
    int up_row_offset;  // row of W where the "up" half starts (gated only)
    int kb_total;       // K / 64
    int epilogue;       // B200_EPILOGUE_*
    int m_tiles, n_tiles;
    int* status;
    // Grouped mode (expert GEMMs with many rows per expert): group g multiplies rows
    // [offsets[g], offsets[g] + counts[g]) of x by rows [g * w_rows_per_group, ...) of w; counts and
    // offsets live in device memory, so the tile list is built on the device by every CTA.
    const int32_t* group_counts;
    const int32_t* group_offsets;
    int num_groups;
    int w_rows_per_group;
    float act_limit;    // B200_EPILOGUE_CLAMPED_SWIGLU
};

constexpr int kMaxGroups = 256;

// Where a tile lives: first row of x / y, rows of it that belong to the tile, first feature, first
// row of the weights (of the "gate" half when gated).
struct TileAt {
    int row0, valid, n0, w_row0;
};

template <int EPI>
__device__ __forceinline__ float gated_act_tile(float g) {
    if (EPI == B200_EPILOGUE_SWIGLU) return __fdividef(g, 1.0f + __expf(-g));  // 2 ulp in fp32, far below the bf16 step
    if (EPI == B200_EPILOGUE_GEGLU_ERF) return 0.5f * g * (1.0f + erff(g * 0.70710678118654752f));
    return 0.5f * g * (1.0f + tanhf(0.7978845608f * (g + 0.044715f * g * g * g)));
}

// Tile t of the walk: bands of kBand token blocks, feature tile slowest inside a band.
__device__ __forceinline__ void tile_coords(int t, int m_tiles, int n_tiles, int& mt, int& ntile) {
    const int per_band = kBand * n_tiles;
    const int band = t / per_band;
    const int r = t - band * per_band;
    const int bm = min(kBand, m_tiles - band * kBand);
    ntile = r / bm;
    mt = band * kBand + (r - ntile * bm);
}

// One warp's 32 rows of an accumulator (columns from tmem_acc on), finished and stored.
template <int EPI, int TN>
__device__ __forceinline__ void store_tile(const TileParams& p, const TileAt& at, int q, int lane, uint32_t tmem_acc) {
    constexpr bool GATED = epilogue_is_gated(EPI);
    const int m_local = q * 32 + lane;
    const int m = at.row0 + m_local;
    const uint32_t t0 = tmem_acc + (static_cast<uint32_t>(q * 32) << 16);
    constexpr int kOutCols = GATED ? TN / 2 : TN;
    const int n_base = at.n0;
    __nv_bfloat16* yrow = p.y + static_cast<int64_t>(m) * p.n_out;
#pragma unroll 1
    for (int c = 0; c < kOutCols / 32; ++c) {
        uint32_t g[32], u[32];
        tmem_ld_32x32b_x32(t0 + static_cast<uint32_t>(c * 32), g);
        if (GATED) tmem_ld_32x32b_x32(t0 + static_cast<uint32_t>(TN / 2 + c * 32), u);
        tmem_ld_wait();
        const int n = n_base + c * 32;
        if (m_local < at.valid && n < p.n_out) {
            float v[32];
#pragma unroll
            for (int j = 0; j < 32; ++j) {
                if (GATED) {
                    const float gv = round_bf16(__uint_as_float(g[j]));
                    const float uv = round_bf16(__uint_as_float(u[j]));
                    v[j] = EPI == B200_EPILOGUE_CLAMPED_SWIGLU ? clamped_swiglu<false>(gv, uv, p.act_limit)
                                                               : gated_act_tile<EPI>(gv) * uv;
                } else {
                    v[j] = __uint_as_float(g[j]);
                }
            }
            if (!GATED && p.bias) {
#pragma unroll
                for (int j = 0; j < 32; ++j)
                    if (n + j < p.n_out) v[j] += __bfloat162float(p.bias[n + j]);
            }
            if (EPI == B200_EPILOGUE_RELU2) {
#pragma unroll
                for (int j = 0; j < 32; ++j) v[j] = fmaxf(v[j], 0.f) * fmaxf(v[j], 0.f);
            }
            if (EPI == B200_EPILOGUE_GELU_ERF) {
#pragma unroll
                for (int j = 0; j < 32; ++j) v[j] = 0.5f * v[j] * (1.0f + erff(v[j] * 0.70710678118654752f));
            }
            if (EPI == B200_EPILOGUE_F32) {
                float* frow = reinterpret_cast<float*>(p.y) + static_cast<int64_t>(m) * p.n_out;
#pragma unroll
                for (int j = 0; j < 32; j += 4)
                    if (n + j < p.n_out)
                        *reinterpret_cast<float4*>(frow + n + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
                continue;
            }
#pragma unroll
            for (int j = 0; j < 32; j += 8) {
                if (n + j < p.n_out) {  // n_out is a multiple of 8: whole 16-byte groups
                    uint4 o;
                    o.x = pack_bf16(v[j], v[j + 1]);
                    o.y = pack_bf16(v[j + 2], v[j + 3]);
                    o.z = pack_bf16(v[j + 4], v[j + 5]);
                    o.w = pack_bf16(v[j + 6], v[j + 7]);
                    *reinterpret_cast<uint4*>(yrow + n + j) = o;
                }
            }
        }
    }
}

template <int EPI>
__global__ void __launch_bounds__(kThreads, 1)
tile_gemm_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_w,
                 const TileParams p) {
    constexpr bool GATED = epilogue_is_gated(EPI);
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t full_bar[kStages];
    __shared__ __align__(8) uint64_t empty_bar[kStages];
    __shared__ __align__(8) uint64_t acc_full_bar[2];
    __shared__ __align__(8) uint64_t acc_empty_bar[2];
    __shared__ uint32_t tmem_base_slot;

    pdl_launch_dependents();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) {
            mbar_init(smem_u32(&full_bar[s]), 1);
            mbar_init(smem_u32(&empty_bar[s]), 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(smem_u32(&acc_full_bar[a]), 1);
            mbar_init(smem_u32(&acc_empty_bar[a]), 4);  // one arrival per epilogue warp
        }
        fence_mbar_init();
    }
    if (warp == 0 && lane == 0) {
        tma_prefetch_desc(&tmap_x);
        tma_prefetch_desc(&tmap_w);
    }
    if (warp == 1) {
        tmem_alloc(smem_u32(&tmem_base_slot), 512);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = tmem_base_slot;
    pdl_wait_prior();

    __shared__ int s_first_tile[kMaxGroups + 1];   // grouped mode: first tile of every group
    __shared__ int s_cnt[kMaxGroups], s_off[kMaxGroups];
    const bool grouped = p.group_counts != nullptr;
    constexpr int kOutTile = GATED ? kTN / 2 : kTN;
    if (grouped) {
        for (int g = threadIdx.x; g < p.num_groups; g += kThreads) {
            s_cnt[g] = p.group_counts[g];
            s_off[g] = p.group_offsets[g];
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            int run = 0;
            for (int g = 0; g < p.num_groups; ++g) {
                s_first_tile[g] = run;
                run += ((max(s_cnt[g], 0) + kTM - 1) / kTM) * p.n_tiles;
            }
            s_first_tile[p.num_groups] = run;
        }
        __syncthreads();
    }
    const int total_tiles = grouped ? s_first_tile[p.num_groups] : p.m_tiles * p.n_tiles;
    auto locate = [&](int t) -> TileAt {
        TileAt a;
        if (!grouped) {
            int mt, ntile;
            tile_coords(t, p.m_tiles, p.n_tiles, mt, ntile);
            a.row0 = mt * kTM;
            a.valid = min(kTM, p.M - a.row0);
            a.n0 = ntile * kOutTile;
            a.w_row0 = 0;
            return a;
        }
        int lo = 0, hi = p.num_groups;   // largest g with s_first_tile[g] <= t
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (s_first_tile[mid] <= t) lo = mid; else hi = mid;
        }
        const int r = t - s_first_tile[lo];
        const int mtiles = (s_cnt[lo] + kTM - 1) / kTM;
        const int ntile = r / mtiles, mt = r - ntile * mtiles;   // token block fastest: neighbours share W
        a.row0 = s_off[lo] + mt * kTM;
        a.valid = min(kTM, s_cnt[lo] - mt * kTM);
        a.n0 = ntile * kOutTile;
        a.w_row0 = lo * p.w_rows_per_group;
        return a;
    };

    if (warp == 0) {
        if (lane == 0) {
            int it = 0;
            bool failed = false;
            for (int t = blockIdx.x; t < total_tiles && !failed; t += gridDim.x) {
                const TileAt at = locate(t);
                const int m0 = at.row0;
                const int n0 = at.w_row0 + at.n0;
                for (int kb = 0; kb < p.kb_total; ++kb, ++it) {
                    const int s = it % kStages;
                    if (it >= kStages) {
                        const uint32_t par = static_cast<uint32_t>(it / kStages - 1) & 1u;
                        if (!mbar_wait_bounded(smem_u32(&empty_bar[s]), par, p.status, 111)) {
                            failed = true;
                            break;
                        }
                    }
                    const uint32_t bar = smem_u32(&full_bar[s]);
                    const uint32_t dst = smem_base + s * kStageBytes;
                    mbar_arrive_expect_tx(bar, kStageBytes);
                    tma_load_2d(dst, &tmap_x, kb * kBK, m0, bar);
                    if (GATED) {
                        tma_load_2d(dst + kABytes, &tmap_w, kb * kBK, n0, bar);
                        tma_load_2d(dst + kABytes + kBBytes / 2, &tmap_w, kb * kBK, p.up_row_offset + n0, bar);
                    } else {
                        tma_load_2d(dst + kABytes, &tmap_w, kb * kBK, n0, bar);
                    }
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            const uint32_t idesc = idesc_bf16_m128(kTN);
            int it = 0, tcount = 0;
            bool failed = false;
            for (int t = blockIdx.x; t < total_tiles && !failed; t += gridDim.x, ++tcount) {
                const int acc = tcount & 1;
                if (tcount >= 2) {
                    const uint32_t par = static_cast<uint32_t>((tcount >> 1) - 1) & 1u;
                    if (!mbar_wait_bounded(smem_u32(&acc_empty_bar[acc]), par, p.status, 112)) {
                        failed = true;
                        break;
                    }
                    tc_fence_after();
                }
                const uint32_t d = tmem_base + static_cast<uint32_t>(acc * kTN);
                for (int kb = 0; kb < p.kb_total; ++kb, ++it) {
                    const int s = it % kStages;
                    const uint32_t par = static_cast<uint32_t>(it / kStages) & 1u;
                    if (!mbar_wait_bounded(smem_u32(&full_bar[s]), par, p.status, 113)) {
                        failed = true;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t a0 = smem_base + s * kStageBytes;
                    const uint32_t b0 = a0 + kABytes;
#pragma unroll
                    for (int k = 0; k < kBK / 16; ++k)
                        tc_mma_bf16(d, kmajor_sw128_desc(a0 + k * 32), kmajor_sw128_desc(b0 + k * 32), idesc,
                                    (kb > 0 || k > 0) ? 1u : 0u);
                    tc_commit(smem_u32(&empty_bar[s]));
                }
                if (failed) break;
                tc_commit(smem_u32(&acc_full_bar[acc]));
            }
        }
    } else {
        const int q = warp & 3;  // TMEM lane quarter this warp may read
        int tcount = 0;
        bool failed = false;
        for (int t = blockIdx.x; t < total_tiles && !failed; t += gridDim.x, ++tcount) {
            const TileAt at = locate(t);
            const int acc = tcount & 1;
            const uint32_t par = static_cast<uint32_t>(tcount >> 1) & 1u;
            if (!mbar_wait_warp(smem_u32(&acc_full_bar[acc]), par, p.status, 114)) {
                failed = true;
                break;
            }
            tc_fence_after();
            store_tile<EPI, kTN>(p, at, q, lane, tmem_base + static_cast<uint32_t>(acc * kTN));
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&acc_empty_bar[acc]));
        }
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem_base, 512);
}


// ---- the same work by pairs of CTAs -------------------------------------------------------------

constexpr int kPairM = 256;                    // tokens per tile: 128 per CTA
constexpr int kPairBand = 8;                   // token blocks per band
constexpr int kPairRing = 192 * 1024;          // bytes of operand stages per CTA

// Two CTAs of a cluster (TPC neighbours) share a tile of 256 tokens x TN features: each holds its own 128 tokens and half
// of the W rows in shared memory, and tcgen05.mma with cta_group::2 reads both halves, so every CTA fetches 32 KB per
// 128 x 256 x 64 block of products instead of 48.  One thread of the first CTA issues; loads of both signal its "full"
// barrier, its commits signal the "empty" and "accumulator full" barriers of both.
template <int EPI, int TN>
__global__ void __launch_bounds__(kThreads, 1)
pair_gemm_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_w, const TileParams p) {
    constexpr bool GATED = epilogue_is_gated(EPI);
    constexpr int kHalfRows = TN / 2;                                  // W rows per CTA
    constexpr uint32_t kPairStage = kABytes + kHalfRows * kBK * 2;
    constexpr int STAGES = kPairRing / kPairStage;
    constexpr uint32_t kAccCols = TN > 128 ? 256 : TN;                 // TMEM is handed out in powers of two
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t full_bar[STAGES];
    __shared__ __align__(8) uint64_t empty_bar[STAGES];
    __shared__ __align__(8) uint64_t acc_full_bar[2];
    __shared__ __align__(8) uint64_t acc_empty_bar[2];
    __shared__ uint32_t tmem_base_slot;
    __shared__ int s_first_tile[kMaxGroups + 1];   // grouped mode: first tile of every group
    __shared__ int s_cnt[kMaxGroups], s_off[kMaxGroups];

    pdl_launch_dependents();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;   // (the same in both CTAs)
    const int rank = static_cast<int>(blockIdx.x) & 1;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(smem_u32(&full_bar[s]), 1);
            mbar_init(smem_u32(&empty_bar[s]), 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(smem_u32(&acc_full_bar[a]), 1);
            mbar_init(smem_u32(&acc_empty_bar[a]), 8);  // one arrival per epilogue warp of both CTAs
        }
        fence_mbar_init();
        tma_prefetch_desc(&tmap_x);
        tma_prefetch_desc(&tmap_w);
    }
    if (warp == 1) {
        tmem_alloc_pair(smem_u32(&tmem_base_slot), 2 * kAccCols);
        tmem_relinquish_pair();
    }
    tc_fence_before();
    cluster_sync_all();      // the barriers of both CTAs are there
    tc_fence_after();
    const uint32_t tmem_base = tmem_base_slot;

    const bool grouped = p.group_counts != nullptr;
    constexpr int kOutTile = GATED ? TN / 2 : TN;
    if (grouped) {
        pdl_wait_prior();   // (the group table comes from the kernel before this one)
        for (int g = threadIdx.x; g < p.num_groups; g += kThreads) {
            s_cnt[g] = p.group_counts[g];
            s_off[g] = p.group_offsets[g];
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            int run = 0;
            for (int g = 0; g < p.num_groups; ++g) {
                s_first_tile[g] = run;
                run += ((max(s_cnt[g], 0) + kPairM - 1) / kPairM) * p.n_tiles;
            }
            s_first_tile[p.num_groups] = run;
        }
        __syncthreads();
    }
    const int total_tiles = grouped ? s_first_tile[p.num_groups] : p.m_tiles * p.n_tiles;
    const int first = static_cast<int>(blockIdx.x) >> 1, step = static_cast<int>(gridDim.x) >> 1;
    auto locate = [&](int t) -> TileAt {   // (of this CTA's 128 tokens; valid may be 0)
        TileAt a;
        if (!grouped) {
            const int per_band = kPairBand * p.n_tiles, band = t / per_band, r = t - band * per_band;
            const int bm = min(kPairBand, p.m_tiles - band * kPairBand), ntile = r / bm;
            a.row0 = (band * kPairBand + (r - ntile * bm)) * kPairM + rank * kTM;
            a.valid = min(kTM, p.M - a.row0);
            a.n0 = ntile * kOutTile;
            a.w_row0 = 0;
            return a;
        }
        int lo = 0, hi = p.num_groups;   // largest g with s_first_tile[g] <= t
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (s_first_tile[mid] <= t) lo = mid; else hi = mid;
        }
        const int r = t - s_first_tile[lo];
        const int mtiles = (s_cnt[lo] + kPairM - 1) / kPairM;
        const int ntile = r / mtiles, mt = r - ntile * mtiles;   // token block fastest: neighbours share W
        a.row0 = s_off[lo] + mt * kPairM + rank * kTM;
        a.valid = min(kTM, s_cnt[lo] - mt * kPairM - rank * kTM);
        a.n0 = ntile * kOutTile;
        a.w_row0 = lo * p.w_rows_per_group;
        return a;
    };

    if (warp == 0) {
        if (elect_one()) {
            int it = 0;
            bool failed = false;
            auto w_row_of = [&](const TileAt& at) { return at.w_row0 + at.n0 + (rank == 0 ? 0 : GATED ? p.up_row_offset : kHalfRows); };
            // The first ring-full of weights does not depend on the kernel before this one.
            const int early = first < total_tiles ? min(p.kb_total, STAGES) : 0;
            for (int s = 0; s < early; ++s) {
                if (rank == 0) mbar_arrive_expect_tx(smem_u32(&full_bar[s]), 2 * kPairStage);
                tma_load_2d_pair(smem_base + s * kPairStage + kABytes, &tmap_w, s * kBK, w_row_of(locate(first)),
                                 in_first_cta(smem_u32(&full_bar[s])));
            }
            pdl_wait_prior();
            for (int t = first; t < total_tiles && !failed; t += step) {
                const TileAt at = locate(t);
                const int w_row = w_row_of(at);
                for (int kb = 0; kb < p.kb_total; ++kb, ++it) {
                    const int s = it % STAGES;
                    if (it >= STAGES) {
                        const uint32_t par = static_cast<uint32_t>(it / STAGES - 1) & 1u;
                        if (!mbar_wait_bounded(smem_u32(&empty_bar[s]), par, p.status, 121)) {
                            failed = true;
                            break;
                        }
                    }
                    const uint32_t dst = smem_base + s * kPairStage;
                    const uint32_t bar = in_first_cta(smem_u32(&full_bar[s]));
                    if (rank == 0 && it >= early) mbar_arrive_expect_tx(smem_u32(&full_bar[s]), 2 * kPairStage);
                    tma_load_2d_pair(dst, &tmap_x, kb * kBK, at.row0, bar);
                    if (it >= early) tma_load_2d_pair(dst + kABytes, &tmap_w, kb * kBK, w_row, bar);
                }
            }
        }
    } else if (warp == 1) {
        if (rank == 0 && elect_one()) {
            const uint32_t idesc = idesc_bf16(kPairM, TN);
            // Neither CTA may end while something is under way to its memory.  So stages that are not filled again are not
            // handed back: nothing would order those arrivals before the accumulator's, which the epilogue waits for.
            const int fills = first < total_tiles ? ((total_tiles - 1 - first) / step + 1) * p.kb_total : 0;
            int it = 0, tcount = 0;
            bool failed = false;
            for (int t = first; t < total_tiles && !failed; t += step, ++tcount) {
                const int acc = tcount & 1;
                if (tcount >= 2) {
                    const uint32_t par = static_cast<uint32_t>((tcount >> 1) - 1) & 1u;
                    if (!mbar_wait_bounded(smem_u32(&acc_empty_bar[acc]), par, p.status, 122)) {
                        failed = true;
                        break;
                    }
                    tc_fence_after();
                }
                const uint32_t d = tmem_base + acc * kAccCols;
                for (int kb = 0; kb < p.kb_total; ++kb, ++it) {
                    const int s = it % STAGES;
                    const uint32_t par = static_cast<uint32_t>(it / STAGES) & 1u;
                    if (!mbar_wait_bounded(smem_u32(&full_bar[s]), par, p.status, 123)) {
                        failed = true;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t a0 = smem_base + s * kPairStage;
                    const uint32_t b0 = a0 + kABytes;
#pragma unroll
                    for (int k = 0; k < kBK / 16; ++k)
                        tc_mma_bf16_pair(d, kmajor_sw128_desc(a0 + k * 32), kmajor_sw128_desc(b0 + k * 32), idesc,
                                         (kb > 0 || k > 0) ? 1u : 0u);
                    if (it + STAGES < fills) tc_commit_pair(smem_u32(&empty_bar[s]));
                }
                if (failed) break;
                tc_commit_pair(smem_u32(&acc_full_bar[acc]));
            }
            // Where a wait ran out: the copies of both CTAs that may still be on their way.
            for (int i = it; failed && i < fills && i < it + STAGES; ++i)
                if (!mbar_wait_bounded(smem_u32(&full_bar[i % STAGES]), static_cast<uint32_t>(i / STAGES) & 1u, p.status, 125)) break;
        }
    } else {
        pdl_wait_prior();   // (y may still be read)
        const int q = warp & 3;  // TMEM lane quarter this warp may read
        int tcount = 0;
        bool failed = false;
        for (int t = first; t < total_tiles && !failed; t += step, ++tcount) {
            const TileAt at = locate(t);
            const int acc = tcount & 1;
            const uint32_t par = static_cast<uint32_t>(tcount >> 1) & 1u;
            if (!mbar_wait_warp(smem_u32(&acc_full_bar[acc]), par, p.status, 124)) {
                failed = true;
                break;
            }
            tc_fence_after();
            store_tile<EPI, TN>(p, at, q, lane, tmem_base + acc * kAccCols);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(in_first_cta(smem_u32(&acc_empty_bar[acc])));
        }
    }
    __syncwarp();
    tc_fence_before();
    cluster_sync_all();   // neither CTA's memory is in use any more
    if (warp == 1) tmem_dealloc_pair(tmem_base, 2 * kAccCols);
}

using TileKernel = void (*)(CUtensorMap, CUtensorMap, TileParams);
template <int TN>
TileKernel pair_kernel_for(int epilogue) {
    switch (epilogue) {
        case B200_EPILOGUE_SWIGLU: return pair_gemm_kernel<B200_EPILOGUE_SWIGLU, TN>;
        case B200_EPILOGUE_GEGLU: return pair_gemm_kernel<B200_EPILOGUE_GEGLU, TN>;
        case B200_EPILOGUE_GEGLU_ERF: return pair_gemm_kernel<B200_EPILOGUE_GEGLU_ERF, TN>;
        case B200_EPILOGUE_RELU2: return pair_gemm_kernel<B200_EPILOGUE_RELU2, TN>;
        case B200_EPILOGUE_GELU_ERF: return pair_gemm_kernel<B200_EPILOGUE_GELU_ERF, TN>;
        case B200_EPILOGUE_CLAMPED_SWIGLU: return pair_gemm_kernel<B200_EPILOGUE_CLAMPED_SWIGLU, TN>;
        case B200_EPILOGUE_F32: return pair_gemm_kernel<B200_EPILOGUE_F32, TN>;
        default: return pair_gemm_kernel<B200_EPILOGUE_NONE, TN>;
    }
}

// Which tiles a GEMM runs on: 0 for single CTAs (128 x 256), or the features of a pair's tile, and about how many
// microseconds it takes.  Modelled as waves of tiles, each as long as its k-blocks; time per block, and once per launch, as
// measured on B200 (M 64 to 8192, K 1024 to 14336).  Pairs fetch a third less per product, which is what bounds full waves
// (8192 x 4096 x 1024: 57 us against 62; 3000 x 28672 x 4096: 479 against 523); blocks of 128 tokens waste less of a short
// batch (300 x 28672 x 4096: 92 against 96); narrow tiles put more SMs to work where there are few (600 x 1024 x 3072: 18 us
// with 64 features, 19 with 128, 26 with 256), or leave fewer of them idle in the last wave.  With a short K a pair's longer start
// counts (8000 x 4096 x 512: 41.9 us against 39.8), and of 128 features a single CTA multiplies and loads half a tile (300 x 128 x
// 512: 7.5 against 6.8).
struct TilePick {
    int tn;
    float us;
};
TilePick pick_tile(int M, int n_out, bool gated, int kb) {
    const char* forced = getenv("B200_TILE_TN");
    if (forced && *forced)
        for (int tn : {0, 64, 128, 192, 256})
            if (atoi(forced) == tn) return {tn, 0.f};
    const int sms = sm_count(), per = gated ? 2 : 1;
    auto cost = [&](int tm, int tn, int slots, float each, float once) {
        return static_cast<float>(div_ceil(div_ceil(M, tm) * div_ceil(n_out * per, tn), slots)) * kb * each + once;
    };
    const bool one_wave = div_ceil(M, kTM) * div_ceil(n_out * per, kTN) <= sms;
    TilePick best = {0, cost(kTM, kTN, sms, (one_wave ? 0.42f : 0.44f) * (n_out * per <= kTN / 2 ? 0.8f : 1.f), 2.5f)};
    const float margin = kb < 12 ? 1.05f : 1.f;
    const struct { int tn; float each; } pairs[] = {{256, 0.40f}, {192, 0.32f}, {128, 0.25f}, {64, 0.22f}};
    for (const auto& t : pairs) {
        const float c = cost(kPairM, t.tn, sms / 2, t.each, 4.0f);
        if (c * margin < best.us) best = {t.tn, c};
    }
    return best;
}

// Launches `p` on pairs of CTAs with tiles of `tn` features (64, 128, 192 or 256); `rows` of x, `w_rows` of w.
int launch_pairs(TileParams p, int tn, const void* x, const void* w, int64_t rows, int64_t w_rows, int K, int64_t ldx, int tiles,
                 cudaStream_t stream) {
    CUtensorMap tmap_x, tmap_w;
    int err = cached_tmap(&tmap_x, x, static_cast<uint64_t>(K), static_cast<uint64_t>(rows), static_cast<uint64_t>(ldx) * 2, kBK, kTM);
    if (err != B200_OK) return err;
    err = cached_tmap(&tmap_w, w, static_cast<uint64_t>(K), static_cast<uint64_t>(w_rows), static_cast<uint64_t>(K) * 2, kBK, tn / 2);
    if (err != B200_OK) return err;
    TileKernel kernel = tn == 64 ? pair_kernel_for<64>(p.epilogue) : tn == 128 ? pair_kernel_for<128>(p.epilogue)
                              : tn == 192 ? pair_kernel_for<192>(p.epilogue) : pair_kernel_for<256>(p.epilogue);
    const int smem = kPairRing + 1024;
    const int pairs = tiles < sm_count() / 2 ? tiles : sm_count() / 2;
    B200_CHECK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    B200_CHECK_CUDA(launch_kernel(kernel, dim3(2 * pairs), dim3(kThreads), smem, stream, dim3(2, 1, 1), tmap_x, tmap_w, p));
    return B200_OK;
}

}  // namespace

float tile_gemm_us(int M, int N, int K, int epilogue) {
    const bool gated = epilogue_is_gated(epilogue);
    // (memory is the bound where the weights are: 64 x 28672 x 4096 takes 47 us)
    return fmaxf(pick_tile(M, gated ? N / 2 : N, gated, K / kBK).us, static_cast<float>(N) * K * 2e-6f / 5.7f) + 1.f;
}

int tile_gemm_features(int M, int N, int K, int epilogue) {
    const bool gated = epilogue_is_gated(epilogue);
    return pick_tile(M, gated ? N / 2 : N, gated, K / kBK).tn;
}

// Blocks of 256 tokens on a pair of CTAs where a group's rows, give or take a seventh, fill one of them and more than one of the
// 128 of a single CTA (151 to 222 rows on average; 64 groups of 189 rows, 2048 x 2048 and 1024 x 2048: a layer of 430 us against
// 456).  Beyond, it depends on how blocks fall to waves (16 groups of 256, 300, 400, 560 rows: pairs 1.07, 0.93, 1.07 and 0.985 times
// as fast), until the blocks are many (640 rows on, 8, 16 and 32 groups: 0.994 to 1.09; but 0.92 and 0.985 for 8 groups of 1100,
// some of which need a fifth block).
bool grouped_on_pairs(int64_t total_rows, int num_groups) {
    const float rows = static_cast<float>(total_rows) / num_groups;
    if (rows >= 640.f) return rows < 1024.f || rows >= 1152.f;
    return rows * 0.85f > kTM && rows * 1.15f <= kPairM;
}

int launch_tile_gemm(void* y, const void* x, const void* w, const void* bias, int M, int N, int K,
                     int64_t ldx, int epilogue, int* status, cudaStream_t stream, float act_limit) {
    const bool gated = epilogue_is_gated(epilogue);
    const int n_out = gated ? N / 2 : N;
    TileParams p;
    p.y = static_cast<__nv_bfloat16*>(y);
    p.bias = static_cast<const __nv_bfloat16*>(bias);
    p.M = M;
    p.n_out = n_out;
    p.up_row_offset = N / 2;
    p.kb_total = K / kBK;
    p.epilogue = epilogue;
    p.m_tiles = div_ceil(M, kTM);
    p.n_tiles = div_ceil(n_out, gated ? kTN / 2 : kTN);
    p.status = status;
    p.group_counts = nullptr;
    p.group_offsets = nullptr;
    p.num_groups = 0;
    p.w_rows_per_group = 0;
    p.act_limit = act_limit;
    const int tn = pick_tile(M, n_out, gated, p.kb_total).tn;
    if (tn > 0) {
        p.m_tiles = div_ceil(M, kPairM);
        p.n_tiles = div_ceil(n_out, gated ? tn / 2 : tn);
        return launch_pairs(p, tn, x, w, M, N, K, ldx, p.m_tiles * p.n_tiles, stream);
    }

    CUtensorMap tmap_x, tmap_w;
    int err = cached_tmap(&tmap_x, x, static_cast<uint64_t>(K), static_cast<uint64_t>(M),
                          static_cast<uint64_t>(ldx) * 2, kBK, kTM);
    if (err != B200_OK) return err;
    err = cached_tmap(&tmap_w, w, static_cast<uint64_t>(K), static_cast<uint64_t>(N),
                      static_cast<uint64_t>(K) * 2, kBK, gated ? kTN / 2 : kTN);
    if (err != B200_OK) return err;

    const uint32_t smem_bytes = kStages * kStageBytes + 1024;
    const int tiles = p.m_tiles * p.n_tiles;
    const int grid = tiles < sm_count() ? tiles : sm_count();
    void (*kernel)(CUtensorMap, CUtensorMap, TileParams) = tile_gemm_kernel<B200_EPILOGUE_NONE>;
    if (epilogue == B200_EPILOGUE_SWIGLU) kernel = tile_gemm_kernel<B200_EPILOGUE_SWIGLU>;
    if (epilogue == B200_EPILOGUE_GEGLU) kernel = tile_gemm_kernel<B200_EPILOGUE_GEGLU>;
    if (epilogue == B200_EPILOGUE_GEGLU_ERF) kernel = tile_gemm_kernel<B200_EPILOGUE_GEGLU_ERF>;
    if (epilogue == B200_EPILOGUE_RELU2) kernel = tile_gemm_kernel<B200_EPILOGUE_RELU2>;
    if (epilogue == B200_EPILOGUE_GELU_ERF) kernel = tile_gemm_kernel<B200_EPILOGUE_GELU_ERF>;
    if (epilogue == B200_EPILOGUE_CLAMPED_SWIGLU) kernel = tile_gemm_kernel<B200_EPILOGUE_CLAMPED_SWIGLU>;
    if (epilogue == B200_EPILOGUE_F32) kernel = tile_gemm_kernel<B200_EPILOGUE_F32>;
    B200_CHECK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(smem_bytes)));
    B200_CHECK_CUDA(launch_kernel(kernel, dim3(grid), dim3(kThreads), smem_bytes, stream, dim3(1, 1, 1),
                                  tmap_x, tmap_w, p));
    return B200_OK;
}

// Grouped form (expert layers with many rows per expert): group g multiplies rows
// [offsets[g], offsets[g] + counts[g]) of x [total_rows, K] by w[g] ([N, K], groups stacked).
int launch_grouped_tile_gemm(void* y, const void* x, const void* w, const int32_t* counts,
                             const int32_t* offsets, int num_groups, int64_t total_rows, int N, int K,
                             int epilogue, int* status, cudaStream_t stream, float act_limit) {
    if (num_groups > kMaxGroups) {
        set_last_error("grouped GEMM: %d groups exceed %d", num_groups, kMaxGroups);
        return B200_ERR_UNSUPPORTED;
    }
    const bool gated = epilogue_is_gated(epilogue);
    const int n_out = gated ? N / 2 : N;
    TileParams p;
    p.y = static_cast<__nv_bfloat16*>(y);
    p.bias = nullptr;
    p.M = static_cast<int>(total_rows);
    p.n_out = n_out;
    p.up_row_offset = N / 2;
    p.kb_total = K / kBK;
    p.epilogue = epilogue;
    p.m_tiles = 0;
    p.n_tiles = div_ceil(n_out, gated ? kTN / 2 : kTN);
    p.status = status;
    p.group_counts = counts;
    p.group_offsets = offsets;
    p.num_groups = num_groups;
    p.w_rows_per_group = N;
    p.act_limit = act_limit;
    if (grouped_on_pairs(total_rows, num_groups))
        return launch_pairs(p, kTN, x, w, total_rows, static_cast<int64_t>(num_groups) * N, K, K, sm_count() / 2, stream);
    CUtensorMap tmap_x, tmap_w;
    int err = cached_tmap(&tmap_x, x, static_cast<uint64_t>(K), static_cast<uint64_t>(total_rows),
                          static_cast<uint64_t>(K) * 2, kBK, kTM);
    if (err != B200_OK) return err;
    err = cached_tmap(&tmap_w, w, static_cast<uint64_t>(K), static_cast<uint64_t>(num_groups) * N,
                      static_cast<uint64_t>(K) * 2, kBK, gated ? kTN / 2 : kTN);
    if (err != B200_OK) return err;
    const uint32_t smem_bytes = kStages * kStageBytes + 1024;
    void (*kernel)(CUtensorMap, CUtensorMap, TileParams) = tile_gemm_kernel<B200_EPILOGUE_NONE>;
    if (epilogue == B200_EPILOGUE_SWIGLU) kernel = tile_gemm_kernel<B200_EPILOGUE_SWIGLU>;
    if (epilogue == B200_EPILOGUE_GEGLU) kernel = tile_gemm_kernel<B200_EPILOGUE_GEGLU>;
    if (epilogue == B200_EPILOGUE_GEGLU_ERF) kernel = tile_gemm_kernel<B200_EPILOGUE_GEGLU_ERF>;
    if (epilogue == B200_EPILOGUE_RELU2) kernel = tile_gemm_kernel<B200_EPILOGUE_RELU2>;
    if (epilogue == B200_EPILOGUE_GELU_ERF) kernel = tile_gemm_kernel<B200_EPILOGUE_GELU_ERF>;
    if (epilogue == B200_EPILOGUE_CLAMPED_SWIGLU) kernel = tile_gemm_kernel<B200_EPILOGUE_CLAMPED_SWIGLU>;
    if (epilogue == B200_EPILOGUE_F32) kernel = tile_gemm_kernel<B200_EPILOGUE_F32>;
    B200_CHECK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(smem_bytes)));
    // the number of tiles is only known on the device: one persistent CTA per SM
    B200_CHECK_CUDA(launch_kernel(kernel, dim3(sm_count()), dim3(kThreads), smem_bytes, stream, dim3(1, 1, 1),
                                  tmap_x, tmap_w, p));
    return B200_OK;
}

}  // namespace b200
