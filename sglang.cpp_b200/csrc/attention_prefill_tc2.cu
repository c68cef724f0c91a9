// Paged-KV causal prefill (extend) attention on the tcgen05 tensor cores, two query tiles per CTA.
//
// One CTA owns (request, KV head, block of 2 x 128/G query tokens), G = q_heads / kv_heads: two tiles
// of 128 rows, each row a (token, head-in-group) pair that reads the same KV head.  The two tiles share
// every K/V tile the producers load and take turns on the tensor core: while the rows of one tile are
// in their softmax, the MMAs of the other run.  Per tile and K/V tile:
//     S = Q K^T            128 x 128 x 128, accumulator in TMEM (columns 0 .., the same for both tiles)
//     softmax              one thread per row takes its 128 scores into registers (the columns are free again at once: the
//                          other tile's scores go there), keeps a running row maximum and sum in the log2 domain and writes
//                          the probabilities into TMEM as bf16 (columns 128 + i*64 ..)
//     O += P V             P is the A operand straight from TMEM, V MN-major from the layout TMA
//                          delivers, O accumulates in TMEM (columns 256 + i*128 ..) for the whole row
// The row maximum used for the exponentials is only moved when the true maximum has grown by more than
// 2^8 since (the sum and the final division use the same reference, so the result is exact); on those
// rare occasions the row's O is rescaled in TMEM by the threads that own the row.  Nothing else touches
// O until the end, so the softmax threads carry no accumulator and no P tile goes through shared memory.
//
// Roles: warp 0 fetches K tiles, warp 2 V tiles, one thread of warp 1 issues the products S, one of warp 3 the products P V,
// warps 4-7 softmax of tile 0, warps 8-11 softmax of tile 1 (thread = TMEM lane).
// A row's scores fit its thread's registers: S is read once and the row's maximum needs no exchange.
//
// K and V tiles have a ring of slots each.  A slot's barriers are tested by parity, which tells a phase from the one before it
// and from no other: whoever tests one has to know that the phase before is over.  With a ring per kind it does.  The producer of
// a ring waits for the release of the slot's last tile, which it has copied there itself, behind the release of the tile before
// that one; the issuer waits for a tile behind the slot's last one, which it has multiplied.  (Both kinds in turn through one ring of
// five slots: V tile j + 5 waits for the release of K tile j + 3, and nothing that its producer has seen tells it that V tile
// j, in the same slot before, has been multiplied with the second query tile; neither does the issuer of S know that it has arrived.)
//
// What bounds it: 2048 cycles of products and 2048 of exponentials (16 per cycle and SM) per K/V tile; 2900 are taken, the
// rest of a row's softmax (scores, maximum, waits: 900 cycles) being hidden only in part.  Both kinds of products from one
// thread, S and P in the same columns: 4500, because a thread that has issued products cannot even test a barrier before the
// tensor core has accepted them, and each wait and each ring position formed anew then lay between two products.  Polynomials
// on the FMA pipe for a part of the exponentials (1/8 to 3/8): no faster.  The steps from there (us; 16 / 8 heads, pages of 16
// in no order): 4 x 2048 tokens behind 2048 cached / 8000 tokens / six prompts of 512 to 2048 / 181 tokens
//     as it was                                                            321 / 417 / 98.9 / 14.5
//     heaviest blocks of all requests and heads first                      295 / 338 / 77.2 / 14.5
//     whole rows of a page per copy, two producers, positions stepped      251 / 278 / 74.6 / 15.5
//     scores in columns of their own, packed arithmetic                    221 / 241 / 68.7 / 14.8
//     S and P V from two threads                                           214 / 233 / 65.7 / 14.5
//     queries and outputs by half warps per row, first K tile early        203 / 227 / 57.6 / 12.4
//     unmasked tiles without tests, one wait per tile for P V              188 / 215 / 54.1 / 12.3
// A ring of slots each for K and V, any number of heads, waits that lanes agree on; one launch at a time between two events:
// 198 / 223 / 61 / 14.3.
// Queries are the LAST extend_len positions of the request, so tiles left of the diagonal need no mask
// and tiles right of it are never loaded.
//
// WINDOW: everything AttentionWindow has (tiles that no row of the block sees are never loaded; the tiles at a
// window's or a chunk's edges are masked per element).
#include <type_traits>

#include "common.cuh"
#include "kernels.h"
#include "tcgen05.cuh"
#include "tensormap.cuh"

namespace b200 {
namespace {

constexpr int kD = 128;
constexpr int kTile = 128;                  // keys per K/V tile and rows per query tile
constexpr int kThreads = 384;               // a warpgroup of producers and issuers, one of softmax per query tile
// The first warpgroup leaves its registers to the others; 384 x 168 are launched.
constexpr int kIssueRegs = 72, kSoftmaxRegs = 216;
static_assert(128 * (kIssueRegs + 2 * kSoftmaxRegs) <= kThreads * 168, "");
constexpr uint32_t kAtomBytes = 128 * 128;  // 128 rows x 64 bf16: one swizzle atom column
constexpr uint32_t kQOff = 0;               // Q: 2 tiles x 2 atoms (d 0-63, d 64-127)
constexpr uint32_t kKVOff = 4 * kAtomBytes; // K tiles, then V tiles, in groups of 8 keys (KvMaps)
constexpr uint32_t kSlotBytes = 2 * kAtomBytes;
constexpr int kKSlots = 2, kVSlots = 3, kSlots = kKSlots + kVSlots;   // a ring of tiles each
constexpr uint32_t kSmemBytes = kKVOff + kSlots * kSlotBytes;
constexpr uint32_t kColS = 0, kColP = 128, kColO = 256;  // TMEM columns: S (128), P0, P1 (64 each), O0, O1 (128 each)
constexpr float kLazyLog2 = 8.0f;           // the reference maximum moves when the true one is 2^8 ahead

struct PrefillTc2Params {
    __nv_bfloat16* out;
    const __nv_bfloat16* q;
    int64_t q_st, q_sh;
    const int32_t* page_table;
    int64_t pt_stride;
    const int32_t* table_idx;
    const int32_t* seq_lens;
    const int32_t* qo_indptr;
    int q_heads, kv_heads, group, batch;
    int group_inverse;       // 65536 / group, rounded up: r / group = r * group_inverse >> 16 for r <= 128
    int blocks;              // of 2 x 128/G query tokens in the longest extension
    int kpc;  // keys of a page in a tile = min(page_size, 128)
    int whole_pages;       // KvMaps::page is there: pages and a cache of 8 slots and more (the map counts groups of 8)
    int whole_tile_boxes;  // KvMaps::tile is there (kpc < 128 <= num_slots)
    int64_t num_slots;
    float scale_log2;
    int* status;
    AttentionWindow w;          // WINDOW only
};

// How K and V tiles are copied ([0] K, [1] V).  In shared memory a tile is 16 groups of 8 keys, each both halves of the head
// dimension, 8 rows of 128 bytes: one copy can bring whole rows of a page (a copy's issue costs the producer 50 cycles and
// more beside the softmax warps, whatever its size).
struct KvMaps {
    CUtensorMap rows[2];   // half rows of min(page, 8) keys: any slot
    CUtensorMap page[2];   // whole rows of min(page, 128) keys from a slot that 8 divides (PrefillTc2Params::whole_pages)
    CUtensorMap tile[2];   // whole rows of 128 keys: tiles whose pages are consecutive slots
};

// Two fp32 operations per instruction, and the maximum of three.
__device__ __forceinline__ uint64_t as_pair(float2 x) { return *reinterpret_cast<uint64_t*>(&x); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(as_pair(a)), "l"(as_pair(b)), "l"(as_pair(c)));
    return *reinterpret_cast<float2*>(&d);
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
    uint64_t d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(as_pair(a)), "l"(as_pair(b)));
    return *reinterpret_cast<float2*>(&d);
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

template <bool WINDOW>
__global__ void __launch_bounds__(kThreads, 1)
attention_prefill_tc2_kernel(const __grid_constant__ KvMaps maps, const PrefillTc2Params p) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t full[kSlots];    // slots of K tiles, then of V tiles
    __shared__ __align__(8) uint64_t empty[kSlots];
    __shared__ __align__(8) uint64_t s_full[2];    // per query tile: S of the current K/V tile is in TMEM
    __shared__ __align__(8) uint64_t s_free[2];    // ... and has been read from there (4 warp arrivals)
    __shared__ __align__(8) uint64_t p_full[2];    // per query tile: P is in TMEM (4 warp arrivals)
    __shared__ __align__(8) uint64_t pv_done[2];   // per query tile: O += P V has completed
    __shared__ uint32_t tmem_base_slot;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
    const int G = p.group;
    auto token_of = [&](int r) { return r * p.group_inverse >> 16; };   // of a tile's row
    auto head_of = [&](int r) { return r - token_of(r) * G; };
    const int QB = token_of(kTile);       // query tokens per tile; rows behind them (3 or 5 heads ...) are the next tile's first ones again
    // Blocks of all requests and heads, the last (heaviest) ones of every prompt first: CTAs that start late are short.
    const int heads = p.kv_heads * p.batch;
    const int h = static_cast<int>(blockIdx.x) % heads % p.kv_heads;
    const int b = static_cast<int>(blockIdx.x) % heads / p.kv_heads;
    const int qb = p.blocks - 1 - static_cast<int>(blockIdx.x) / heads;

    pdl_launch_dependents();
    if (threadIdx.x == 0) {
        for (int kv = 0; kv < 2; ++kv) {
            if (p.whole_pages) tma_prefetch_desc(&maps.page[kv]);
            if (p.whole_tile_boxes) tma_prefetch_desc(&maps.tile[kv]);
        }
        for (int s = 0; s < kSlots; ++s) {
            mbar_init(smem_u32(&full[s]), 1);
            mbar_init(smem_u32(&empty[s]), 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(smem_u32(&s_full[i]), 1);
            mbar_init(smem_u32(&s_free[i]), 4);   // one arrival per softmax warp of the tile
            mbar_init(smem_u32(&p_full[i]), 4);
            mbar_init(smem_u32(&pv_done[i]), 1);
        }
        fence_mbar_init();
        fence_proxy_async_smem();
    }
    __syncwarp();
    pdl_wait_prior();

    const int q_begin = p.qo_indptr[b];
    const int ext = p.qo_indptr[b + 1] - q_begin;
    const int len = p.seq_lens[b];
    const int table = p.table_idx[b];
    const int nqb = (ext + 2 * QB - 1) / (2 * QB);
    if (qb >= nqb || ext <= 0 || len <= 0) return;          // whole CTA, before any barrier or TMEM use
    const int t0 = qb * 2 * QB;                   // first token of tile 0; tile 1 starts QB further
    const int t_end = min(t0 + 2 * QB, ext);
    const int pos0 = len - ext;                   // position of query token 0
    const int kv_end = min(len, pos0 + t_end);    // keys [0, kv_end) are visible to this block
    // tiles [0, head_tiles) and, `skip` tiles further, those from the oldest key that the first row sees
    const int head_tiles = WINDOW ? (min(p.w.keep_first, kv_end) + kTile - 1) / kTile : 0;
    const int skip = WINDOW ? max(0, p.w.oldest(pos0 + t0) / kTile - head_tiles) : 0;
    const int ntiles = (kv_end + kTile - 1) / kTile - skip;
    auto first_key = [&](int kt) { return (WINDOW && kt >= head_tiles ? kt + skip : kt) * kTile; };

    // ---- K and V tiles (warp 0 and warp 2) ----
    const int32_t* pt_row = p.page_table + static_cast<int64_t>(table) * p.pt_stride;
    auto copies_of = [&](int kt) { return (min(kTile, kv_end - first_key(kt)) + p.kpc - 1) / p.kpc; };
    int next[4];
    // this lane's slots of a tile's copies, fetched a tile ahead: the table's trip to L2 would otherwise stand between
    // a slot's release and its next copy
    auto fetch_slots = [&](int kt) {
        const int n = copies_of(kt), k0 = first_key(kt);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int copy = i * 32 + lane;
            next[i] = copy < n ? pt_row[k0 + copy * p.kpc] : 0;
        }
    };
    // How tile kt is copied: a tile whose pages are consecutive slots with one copy; so is a page, unless it is smaller than a group or
    // starts inside one.  (Before its slot is free.)
    int sl[4], ncopies = 0;
    bool whole = false, groups = false;
    auto plan_tile = [&](int kt) {
        ncopies = copies_of(kt);
        whole = kv_end - first_key(kt) >= kTile && p.whole_tile_boxes;
        groups = p.whole_pages;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            sl[i] = next[i];
            if (sl[i] < 0 || static_cast<int64_t>(sl[i]) + p.kpc > p.num_slots) {
                atomicExch(&p.status[kStatusBadIndex], sl[i] + 1);
                sl[i] = 0;
            }
            if ((sl[i] & 7) != 0) groups = false;
        }
        const int first = __shfl_sync(0xffffffffu, sl[0], 0);
        if ((first & 7) != 0) whole = false;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int copy = i * 32 + lane;
            if (copy < ncopies && sl[i] != first + copy * p.kpc) whole = false;
        }
        whole = __all_sync(0xffffffffu, whole);
        groups = __all_sync(0xffffffffu, groups);
    };
    // That K (kv = 0) or V tile into `slot`.
    auto load_tile = [&](int kv, uint32_t slot) {
        const uint32_t bar = smem_u32(&full[slot]);
        const uint32_t base = smem_base + kKVOff + slot * kSlotBytes;
        if (lane == 0) mbar_arrive_expect_tx(bar, static_cast<uint32_t>(ncopies * p.kpc) * kD * 2u);
        __syncwarp();
        if (whole) {
            if (lane == 0) tma_load_5d(base, &maps.tile[kv], 0, 0, 0, sl[0] >> 3, h, bar);
        } else {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int copy = i * 32 + lane;
                if (copy >= ncopies) continue;
                if (groups) {
                    tma_load_5d(base + copy * p.kpc * (kD * 2), &maps.page[kv], 0, 0, 0, sl[i] >> 3, h, bar);
                    continue;
                }
                for (int key = copy * p.kpc; key < (copy + 1) * p.kpc; key += 8) {
                    const uint32_t dst = base + (key >> 3) * 2048 + (key & 7) * 128;
                    const int from = sl[i] + key - copy * p.kpc;
                    tma_load_3d(dst, &maps.rows[kv], 0, h, from, bar);
                    tma_load_3d(dst + 1024, &maps.rows[kv], 64, h, from, bar);
                }
            }
        }
    };
    if (warp == 0 || warp == 2) fetch_slots(0);
    if (warp == 0) {   // the first K tile is under way while the others fetch the queries (this warp has made the barriers)
        plan_tile(0);
        load_tile(0, 0);
        if (ntiles > 1) fetch_slots(1);
    }

    // Rows of V that no copy ever writes (behind the last key, in a slot that had no tile before) must not hold NaN
    // patterns: their probabilities are 0.
    if (ntiles <= kVSlots) {
        const int written = (kv_end - first_key(ntiles - 1) + p.kpc - 1) / p.kpc * p.kpc;
        uint4* z = reinterpret_cast<uint4*>(smem_gen + kKVOff + (kKSlots + ntiles - 1) * kSlotBytes);
        for (int i = threadIdx.x; i < max(0, kTile - written) * 16; i += kThreads) {
            const int key = written + (i >> 4), at = i & 15;   // 16 bytes of a key's row
            z[(key >> 3) * 128 + (at >> 3) * 64 + (key & 7) * 8 + (at & 7)] = make_uint4(0, 0, 0, 0);
        }
    }
    if (warp == 1) {
        tmem_alloc(smem_u32(&tmem_base_slot), 512);
        tmem_relinquish();
    }
    // Q rows into shared memory in the swizzled K-major layout: tile i, row r = (token t0 + i*QB + r / G,
    // head h * G + r % G); rows past the request's last token are zero.
    if (warp >= 4) {
        const int sw = warp - 4;                  // 0..7
        const int tile = sw >> 2;
        uint4 v[16];
        // (half a warp per row: neighbouring lanes read neighbouring addresses)
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const int r = (sw & 3) * 32 + i * 2 + (lane >> 4);
            const int tok = t0 + tile * QB + token_of(r);
            const int head = h * G + head_of(r);
            v[i] = make_uint4(0, 0, 0, 0);
            if (tok < t_end)
                v[i] = reinterpret_cast<const uint4*>(p.q + static_cast<int64_t>(q_begin + tok) * p.q_st +
                                                      static_cast<int64_t>(head) * p.q_sh)[lane & 15];
        }
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const int r = (sw & 3) * 32 + i * 2 + (lane >> 4);
            const uint32_t a = swz128(smem_base + kQOff + (tile * 2 + (lane >> 3 & 1)) * kAtomBytes + r * 128, lane & 7);
            asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(a), "r"(v[i].x), "r"(v[i].y), "r"(v[i].z), "r"(v[i].w)
                         : "memory");
        }
    }
    fence_proxy_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = tmem_base_slot;

    if (warp < 4) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kIssueRegs));
    if (warp == 0 || warp == 2) {
        // ================= producers: K tiles, V tiles =================
        const int kv = warp >> 1;
        const uint32_t ring = kv == 0 ? 0 : kKSlots, ring_end = kv == 0 ? kKSlots : kSlots;
        uint32_t slot = kv == 0 ? 1 : kKSlots, phase = 1;   // (the first waits are for slots that nobody has used)
        for (int kt = kv == 0 ? 1 : 0; kt < ntiles; ++kt) {
            plan_tile(kt);
            if (kt + 1 < ntiles) fetch_slots(kt + 1);
            if (!__all_sync(0xffffffffu, mbar_wait_mostly_ready(smem_u32(&empty[slot]), phase, p.status, 321))) break;   // (see mbar_wait_warp)
            load_tile(kv, slot);
            if (++slot == ring_end) {
                slot = ring;
                phase ^= 1;
            }
        }
    } else if (warp == 1) {
        // ================= issuer of S_i = Q_i K^T =================
        if (elect_one()) {
            const uint32_t idesc = idesc_bf16_128x128(false);
            const uint64_t q_desc = kmajor_sw128_desc(smem_base + kQOff);
            const uint64_t k_desc = grouped_keys_desc(smem_base + kKVOff, 0);      // head dimension along the row
            uint32_t slot = 0, phase = 0;
            bool failed = false;
            auto wait = [&](uint32_t bar, uint32_t parity, int site) {
                if (!failed && !mbar_wait_mostly_ready(bar, parity, p.status, site)) failed = true;
            };
            for (int kt = 0; kt < ntiles && !failed; ++kt) {
                const uint64_t k = k_desc + slot * (kSlotBytes >> 4);
                const uint32_t parity = static_cast<uint32_t>(kt) & 1u;
                wait(smem_u32(&full[slot]), phase, 322);
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    // both query tiles use the same columns in turn: the other tile's scores have to have been read
                    if (i == 1 || kt > 0) wait(smem_u32(&s_free[i ^ 1]), i == 1 ? parity : parity ^ 1u, 328);
                    if (failed) break;
                    tc_fence_after();
                    const uint64_t a = q_desc + static_cast<uint32_t>(i) * (2 * kAtomBytes >> 4);
#pragma unroll
                    for (int ks = 0; ks < 8; ++ks)
                        tc_mma_bf16(tmem_base + kColS, a + (((ks >> 2) * kAtomBytes + (ks & 3) * 32) >> 4),
                                    k + (((ks >> 2) * 1024 + (ks & 3) * 32) >> 4), idesc, ks > 0 ? 1u : 0u);
                    tc_commit(smem_u32(&s_full[i]));
                }
                if (failed) break;
                // both tiles have read this K tile (a slot that is not filled again is not handed back: nobody would wait for that
                // arrival, and it could still be under way when the block ends)
                if (kt + kKSlots < ntiles) tc_commit(smem_u32(&empty[slot]));
                if (++slot == kKSlots) {
                    slot = 0;
                    phase ^= 1;
                }
            }
        }
    } else if (warp == 3) {
        // ================= issuer of O_i += P_i V =================
        if (elect_one()) {
            const uint32_t idesc = idesc_bf16_128x128(true);
            const uint64_t v_desc = grouped_keys_desc(smem_base + kKVOff, 1024);   // second half of the head dimension 1024 bytes on
            uint32_t slot = kKSlots, phase = 0;
            bool failed = false;
            auto wait = [&](uint32_t bar, uint32_t parity, int site) {
                if (!failed && !mbar_wait_mostly_ready(bar, parity, p.status, site)) failed = true;
            };
            for (int kt = 0; kt < ntiles && !failed; ++kt) {
                const uint64_t v = v_desc + slot * (kSlotBytes >> 4);
                const uint32_t parity = static_cast<uint32_t>(kt) & 1u;
                wait(smem_u32(&full[slot]), phase, 326);
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const uint32_t prob = tmem_base + kColP + static_cast<uint32_t>(i) * 64u;
                    const uint32_t d = tmem_base + kColO + static_cast<uint32_t>(i) * 128u;
                    wait(smem_u32(&p_full[i]), parity, 323);
                    if (failed) break;
                    tc_fence_after();
#pragma unroll
                    for (int ks = 0; ks < 8; ++ks)   // keys ks*16 .. +15: eight packed columns
                        tc_mma_bf16_ts(d, prob + static_cast<uint32_t>(ks * 8), v + (ks * 4096 >> 4), idesc, (kt > 0 || ks > 0) ? 1u : 0u);
                    tc_commit(smem_u32(&pv_done[i]));
                }
                if (failed) break;
                if (kt + kVSlots < ntiles) tc_commit(smem_u32(&empty[slot]));   // both tiles have read this V tile
                if (++slot == kSlots) {
                    slot = kKSlots;
                    phase ^= 1;
                }
            }
        }
    } else if (warp >= 4) {
        // ================= softmax / output rows =================
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kSoftmaxRegs));
        const int tile = (warp >> 2) - 1;         // query tile of this warp
        const int qtr = warp & 3;                 // TMEM lane quarter this warp may read
        const int r = qtr * 32 + lane;            // query row = TMEM lane
        const int tok = t0 + tile * QB + token_of(r);
        const int head = h * G + head_of(r);
        const int limit = min(pos0 + tok, len - 1);   // last visible key of this row
        const int oldest = WINDOW ? p.w.oldest(limit) : 0;   // keys before it are seen below keep_first only
        const uint32_t lane_addr = tmem_base + (static_cast<uint32_t>(qtr * 32) << 16);
        const uint32_t s_addr = lane_addr + kColS;
        const uint32_t p_addr = lane_addr + kColP + static_cast<uint32_t>(tile) * 64u;
        const uint32_t o_addr = lane_addr + kColO + static_cast<uint32_t>(tile) * 128u;
        const float sc = p.scale_log2;
        float m_ref = -INFINITY;   // the maximum the exponentials refer to, in units of the raw scores
        float l_run = 0.f;
        bool failed = false;
        auto low_bits = [](int n) { return n >= 32 ? ~0u : n <= 0 ? 0u : (1u << n) - 1u; };
        auto ex2 = [](float x) {
            float y;
            asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
            return y;
        };

        for (int kt = 0; kt < ntiles; ++kt) {
            if (!failed && !mbar_wait_mostly_ready(smem_u32(&s_full[tile]), static_cast<uint32_t>(kt) & 1u, p.status, 324))
                failed = true;
            tc_fence_after();
            const int k0 = first_key(kt);
            // (masking is decided per warp, so that the common case carries no per-element tests at all)
            const bool need_mask =
                __any_sync(0xffffffffu, k0 + kTile - 1 > limit || (WINDOW && k0 < oldest && k0 + kTile - 1 >= p.w.keep_first));
            uint32_t s[4][32];
#pragma unroll
            for (int c = 0; c < 4; ++c) tmem_ld_32x32b_x32(s_addr + c * 32, s[c]);
            tmem_ld_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&s_free[tile]));
            float m4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
            // a masked tile: which of each 32 keys the row sees, as bits
            uint32_t seen[4] = {~0u, ~0u, ~0u, ~0u};
            if (need_mask) {
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const int at = k0 + c * 32;
                    seen[c] = low_bits(limit + 1 - at);
                    if (WINDOW) seen[c] &= ~low_bits(oldest - at) | low_bits(p.w.keep_first - at);
#pragma unroll
                    for (int i = 0; i < 32; ++i)
                        m4[i & 3] = fmaxf(m4[i & 3], (seen[c] >> i & 1) != 0 ? __uint_as_float(s[c][i]) : -INFINITY);
                }
            } else {
#pragma unroll
                for (int c = 0; c < 4; ++c)
#pragma unroll
                    for (int i = 0; i < 32; i += 2)
                        m4[(i >> 1) & 3] = max3(m4[(i >> 1) & 3], __uint_as_float(s[c][i]), __uint_as_float(s[c][i + 1]));
            }
            const float mx = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3]));
            // the previous tile's product has read P and has added to O
            if (kt > 0 && !failed && !mbar_wait_mostly_ready(smem_u32(&pv_done[tile]), static_cast<uint32_t>(kt - 1) & 1u, p.status, 327))
                failed = true;
            tc_fence_after();
            // Move the reference only when the row's maximum has outgrown it by 2^8; O and the running sum shrink by the
            // same factor.  The TMEM accesses are warp-wide instructions, so a warp rescales all of its rows (by 1 where
            // nothing moved) as soon as one of them has to.
            float alpha = 1.f;
            if (mx != -INFINITY && (m_ref == -INFINITY || (mx - m_ref) * sc > kLazyLog2)) {
                if (m_ref != -INFINITY) alpha = ex2((m_ref - mx) * sc);
                m_ref = mx;
            }
            if (__any_sync(0xffffffffu, alpha != 1.f)) {
                l_run *= alpha;
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    uint32_t ov[16];
                    tmem_ld_32x32b_x16(o_addr + c * 16, ov);
                    tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < 16; ++i) ov[i] = __float_as_uint(__uint_as_float(ov[i]) * alpha);
                    tmem_st_32x32b_x16(o_addr + c * 16, ov);
                }
            }
            // a row that has seen no key yet: every exponent becomes -inf, every probability 0
            const float mb = m_ref == -INFINITY ? INFINITY : m_ref * sc;
            float2 sum = make_float2(0.f, 0.f);
            const float2 sc2 = make_float2(sc, sc), mb2 = make_float2(-mb, -mb);
            // (two copies of the code, so that an unmasked tile's has no tests)
            auto probabilities = [&](auto masked) {
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    uint32_t packed[16];
#pragma unroll
                    for (int i = 0; i < 32; i += 2) {
                        const float2 e = fma2(make_float2(__uint_as_float(s[c][i]), __uint_as_float(s[c][i + 1])), sc2, mb2);
                        float2 pr = make_float2(ex2(e.x), ex2(e.y));
                        if (masked) {
                            if ((seen[c] >> i & 1) == 0) pr.x = 0.f;
                            if ((seen[c] >> (i + 1) & 1) == 0) pr.y = 0.f;
                        }
                        sum = add2(sum, pr);
                        packed[i >> 1] = pack_bf16(pr.x, pr.y);
                    }
                    tmem_st_32x32b_x16(p_addr + c * 16, packed);
                }
            };
            if (need_mask) probabilities(std::true_type{});
            else probabilities(std::false_type{});
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&p_full[tile]));
            l_run += sum.x + sum.y;
        }
        // the last product, then O / sum
        if (!failed && !mbar_wait_mostly_ready(smem_u32(&pv_done[tile]), static_cast<uint32_t>(ntiles - 1) & 1u, p.status, 325))
            failed = true;
        tc_fence_after();
        float l_tot = l_run;
        if (WINDOW && p.w.sinks != nullptr) l_tot += ex2(fmaf(p.w.sinks[head], 1.4426950408889634f, -m_ref * sc));
        {
            // (the TMEM loads are warp-wide: every lane takes part, only the stores are per row)
            const bool store = !failed && tok < t_end;
            float inv = l_tot > 0.f ? 1.f / l_tot : 0.f;
            const int64_t row = q_begin + (store ? tok : 0);
            const __nv_bfloat16* gates = WINDOW ? static_cast<const __nv_bfloat16*>(p.w.gate) : nullptr;
            if (WINDOW) inv *= p.w.out_scale;
            if (WINDOW && gates != nullptr && p.w.gate_per_head) inv *= sigmoid_f(__bfloat162float(gates[row * p.w.gate_st + head]));
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                uint32_t ov[32];
                tmem_ld_32x32b_x32(o_addr + c * 32, ov);
                tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < 32; ++i) ov[i] = __float_as_uint(__uint_as_float(ov[i]) * inv);
                if (WINDOW && gates != nullptr && !p.w.gate_per_head && store) {
                    const uint4* gate = reinterpret_cast<const uint4*>(gates + row * p.w.gate_st + head * kD);
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const uint4 g4 = gate[c * 4 + j];
                        const uint32_t gw[4] = {g4.x, g4.y, g4.z, g4.w};
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            ov[j * 8 + 2 * i] = __float_as_uint(__uint_as_float(ov[j * 8 + 2 * i]) * sigmoid_f(bf16_lo(gw[i])));
                            ov[j * 8 + 2 * i + 1] = __float_as_uint(__uint_as_float(ov[j * 8 + 2 * i + 1]) * sigmoid_f(bf16_hi(gw[i])));
                        }
                    }
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    uint4 w;
                    w.x = pack_bf16(__uint_as_float(ov[j * 8 + 0]), __uint_as_float(ov[j * 8 + 1]));
                    w.y = pack_bf16(__uint_as_float(ov[j * 8 + 2]), __uint_as_float(ov[j * 8 + 3]));
                    w.z = pack_bf16(__uint_as_float(ov[j * 8 + 4]), __uint_as_float(ov[j * 8 + 5]));
                    w.w = pack_bf16(__uint_as_float(ov[j * 8 + 6]), __uint_as_float(ov[j * 8 + 7]));
                    const int at = c * 4 + j;
                    const uint32_t a = swz128(smem_base + kQOff + (tile * 2 + (at >> 3)) * kAtomBytes + r * 128, at & 7);
                    asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(a), "r"(w.x), "r"(w.y), "r"(w.z), "r"(w.w) : "memory");
                }
            }
            // Through the query tile's place in shared memory (its last product is done), so that half a warp writes a row.
            const bool ok = __all_sync(0xffffffffu, !failed);
            __syncwarp();   // (a vote orders no memory)
            const int64_t out_st = WINDOW ? p.w.out_st : static_cast<int64_t>(p.q_heads) * kD;
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const int row2 = qtr * 32 + i * 2 + (lane >> 4);
                const int at2 = token_of(row2), tok2 = t0 + tile * QB + at2;
                const uint32_t a = swz128(smem_base + kQOff + (tile * 2 + (lane >> 3 & 1)) * kAtomBytes + row2 * 128, lane & 7);
                uint4 w;
                asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(w.x), "=r"(w.y), "=r"(w.z), "=r"(w.w) : "r"(a) : "memory");
                if (ok && at2 < QB && tok2 < t_end)
                    reinterpret_cast<uint4*>(p.out + (q_begin + tok2) * out_st + (h * G + row2 - at2 * G) * kD)[lane & 15] = w;
            }
        }
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem_base, 512);
}

}  // namespace

int make_kv_tile_tmap(CUtensorMap* out, const void* cache, int64_t num_slots, int kv_heads, int kpc) {
    EncodeTiledFn fn = encode_tiled_fn();
    if (!fn) {
        set_last_error("cuTensorMapEncodeTiled is not available from this driver");
        return B200_ERR_CUDA;
    }
    const cuuint64_t dims[3] = {kD, static_cast<cuuint64_t>(kv_heads), static_cast<cuuint64_t>(num_slots)};
    const cuuint64_t strides[2] = {kD * 2, static_cast<cuuint64_t>(kv_heads) * kD * 2};
    const cuuint32_t box[3] = {64, 1, static_cast<cuuint32_t>(kpc)};
    const cuuint32_t es[3] = {1, 1, 1};
    CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(cache), dims, strides,
                    box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                    CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_last_error("cuTensorMapEncodeTiled (3-D KV map) failed with CUresult %d", static_cast<int>(r));
        return B200_ERR_CUDA;
    }
    return B200_OK;
}

namespace {

// Whole rows of `keys` (a multiple of 8) neighbouring slots of 8 or more, the first of them a multiple of 8: groups of 8 keys, in each
// both halves of the head dimension (coordinates: element of a half, key of a group, half, group, head).
int make_kv_groups_tmap(CUtensorMap* out, const void* cache, int64_t num_slots, int kv_heads, int keys) {
    EncodeTiledFn fn = encode_tiled_fn();
    if (!fn) {
        set_last_error("cuTensorMapEncodeTiled is not available from this driver");
        return B200_ERR_CUDA;
    }
    const cuuint64_t slot = static_cast<cuuint64_t>(kv_heads) * kD * 2;
    const cuuint64_t dims[5] = {64, 8, 2, static_cast<cuuint64_t>(num_slots / 8), static_cast<cuuint64_t>(kv_heads)};
    const cuuint64_t strides[4] = {slot, 128, slot * 8, kD * 2};
    const cuuint32_t box[5] = {64, 8, 2, static_cast<cuuint32_t>(keys / 8), 1};
    const cuuint32_t es[5] = {1, 1, 1, 1, 1};
    CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<void*>(cache), dims, strides, box, es,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_last_error("cuTensorMapEncodeTiled (KV groups) failed with CUresult %d", static_cast<int>(r));
        return B200_ERR_CUDA;
    }
    return B200_OK;
}

}  // namespace

int launch_attention_prefill_tc2(void* out, const void* q, int64_t q_st, int64_t q_sh, const void* k_cache,
                                 const void* v_cache, int64_t num_slots, const int32_t* page_table,
                                 int64_t pt_stride, const int32_t* table_idx, const int32_t* seq_lens,
                                 const int32_t* qo_indptr, int batch, int max_extend_len, int q_heads,
                                 int kv_heads, int page_size, float sm_scale, int* status,
                                 cudaStream_t stream, const AttentionWindow* window) {
    if (batch == 0 || max_extend_len == 0) return B200_OK;
    PrefillTc2Params p;
    p.out = static_cast<__nv_bfloat16*>(out);
    p.q = static_cast<const __nv_bfloat16*>(q);
    p.q_st = q_st;
    p.q_sh = q_sh;
    p.page_table = page_table;
    p.pt_stride = pt_stride;
    p.table_idx = table_idx;
    p.seq_lens = seq_lens;
    p.qo_indptr = qo_indptr;
    p.q_heads = q_heads;
    p.kv_heads = kv_heads;
    p.group = q_heads / kv_heads;
    p.group_inverse = (65536 + p.group - 1) / p.group;
    p.batch = batch;
    p.kpc = page_size < kTile ? page_size : kTile;
    p.num_slots = num_slots;
    p.scale_log2 = sm_scale * 1.4426950408889634f;
    p.status = status;
    if (window) p.w = *window;
    if (p.w.out_st == 0) p.w.out_st = static_cast<int64_t>(q_heads) * kD;
    KvMaps maps = {};
    p.whole_pages = p.kpc >= 8 && num_slots >= 8 ? 1 : 0;
    p.whole_tile_boxes = p.kpc < kTile && num_slots >= kTile ? 1 : 0;
    for (int kv = 0; kv < 2; ++kv) {
        const void* cache = kv == 0 ? k_cache : v_cache;
        int err = make_kv_tile_tmap(&maps.rows[kv], cache, num_slots, kv_heads, p.kpc < 8 ? p.kpc : 8);
        if (err == B200_OK && p.whole_pages) err = make_kv_groups_tmap(&maps.page[kv], cache, num_slots, kv_heads, p.kpc);
        if (err == B200_OK && p.whole_tile_boxes) err = make_kv_groups_tmap(&maps.tile[kv], cache, num_slots, kv_heads, kTile);
        if (err != B200_OK) return err;
    }
    const int QB = kTile / p.group;
    const int smem = kSmemBytes + 1024;
    auto kernel = window ? attention_prefill_tc2_kernel<true> : attention_prefill_tc2_kernel<false>;
    B200_CHECK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    p.blocks = div_ceil(max_extend_len, 2 * QB);
    B200_CHECK_CUDA(launch_kernel(kernel, dim3(static_cast<unsigned>(p.blocks) * kv_heads * batch), dim3(kThreads), smem, stream,
                                  dim3(1, 1, 1), maps, p));
    return B200_OK;
}

}  // namespace b200
