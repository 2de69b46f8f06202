// GQA forward for sm_100a: O = softmax(scale * Q K^T [+ causal]) V, LSE.
//
// A work item is two 128-row query tiles (one, where every tile gets an SM of its own, and for the longest tiles of some causal
// launches) of one (batch, query head); the KV head's 128-row key/value blocks stream through a TMA ring.  A thread block works through
// several items (see the work-item comment).  Roles:
//   warps 0-3  softmax warpgroup for query tile 0 (thread = query row = TMEM lane)
//   warps 4-7  softmax warpgroup for query tile 1
//   warp  8    TMA producer (Q once per item, K and V rings) and taker of further items
//   warps 9,10 UMMA issuers, one per query tile: S = Q K^T and O += P V (P read from TMEM)
// Every key block is handled as two half-blocks of 64 keys, and the 128 fp32 S columns of a tile are two
// 64-column buffers: while the softmax warpgroup works on half-block j, the issuer has already produced
// S(j+1) in the other buffer, so the warpgroup never waits for the tensor core in steady state (with one
// 128-column S buffer per tile the chain softmax -> P V -> Q K^T -> softmax was serial and set the period).
// P(j) overwrites the first 32 columns of its own S buffer as packed bf16; S(j+2) may overwrite it only after
// P(j) V has completed (pv_done barrier; different accumulators, so issue order alone guarantees nothing).
// The running maximum is only refreshed when it grows by more than 2^8, so O is rescaled rarely (and then
// only after the previous P V has completed); the final division by the row sum uses the same maximum.
//
// Replaces gqa62::gqa_v62 / launch_gqa_v62 (src/attention/GQA_fwd_ref.cu:336-651):
// same inputs/outputs, LSE = natural-log of the scaled-logit sum (:611-614).
#include <algorithm>
#include <type_traits>

#include "gqa_common.cuh"
#include "gqa_kernels.cuh"
#include "packed_list.cuh"
#include "sm100_ptx.cuh"

namespace gqa {
namespace {

using namespace sm100;

// Optional timeline tracing (development builds only): block 0 stamps clock64 at a few points per key block.
#ifdef GQA_FWD_TRACE
__device__ long long g_fwd_trace[6][64][4];
#define GQA_FTRACE(role, it, slot)                                                                 \
    do {                                                                                           \
        if (blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0 && (it) < 64 && (threadIdx.x & 31) == 0) \
            g_fwd_trace[role][it][slot] = clock64();                                               \
    } while (0)
#else
#define GQA_FTRACE(role, it, slot) \
    do {                           \
    } while (0)
#endif

constexpr int kTile = 128;             // query rows per tile and key rows per block
constexpr int kPanel = kTile * 128;    // bytes of one 64-column panel of a 128-row tile
constexpr int kHalf = 64;               // keys per half-block
constexpr int kFwdThreads = 352;
constexpr int kWarpTma = 8, kWarpMma0 = 9;
constexpr int kItemSlots = 2;
constexpr int kMaxPassedOver = 256;  // empty items of a packed batch that are taken over before one is published
constexpr size_t kOrderKvBytes = (size_t)48 << 20;  // K and V of a causal launch whose items come longest first
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;
constexpr float kRescaleThreshold = 8.0f;  // in log2 units

template <int D>
struct FwdCfg {
    static constexpr int kPanels = D / 64;
    static constexpr int kTileBytes = kPanels * kPanel;  // one 128 x D bf16 tile
    static constexpr int kStages = (D == 64) ? 4 : 2;
    static constexpr int kSmemQ = 2 * kTileBytes;
    static constexpr int kSmemKV = 2 * kStages * kTileBytes;
    static constexpr int kBarBytes = 512;
    static constexpr int kSmemTotal = kSmemQ + kSmemKV + kBarBytes;  // the dynamic window must start 1024-byte aligned (checked)
    static constexpr int kOffList = kSmemTotal;  // packed batches: the work list
    static constexpr uint32_t kTmemCols = 512;
    static constexpr uint32_t kColS0 = 0, kColS1 = 128, kColO0 = 256, kColO1 = 256 + D;
    static_assert(256 + 2 * D <= 512, "TMEM budget");
    static_assert(kOffList % alignof(PackedList) == 0 && kSmemTotal + (int)sizeof(PackedList) <= 227 * 1024, "shared memory budget");
    static_assert(kSmemTotal > kHalfSharedMemory, "one CTA per SM is assumed by the 512-column TMEM allocation");
};

struct FwdParams {
    __nv_bfloat16* O;
    float* LSE;
    unsigned int* status;
    int Hq, Hkv, S, causal, bshd;
    int tiles, n_groups;  // query tiles per item (1 or 2), items per (sequence, query head)
    int tile_slow;        // the place in the sequence is the slowest index of the items (x = head, y = sequence, z = place)
    int singles;          // ... and so many of its last tiles are items of their own (see SingleTiles)
    const int* cu;     // packed variable-length batch: sequence starts (z of an item = sequence), else null
    int n_listed;      // packed batch with a work list (x of an item = place in the list): the sequences in it, else 0
    int d_real;        // head dimension of the tensors (<= D of the kernel; the columns beyond it read as zeros)
    float scale_log2;  // scale * log2(e)
};

// What a launch of the kernel has beside the plain case.
enum Form {
    kNative,  // one length for the whole batch, all columns of the kernel (the ones beyond the head dimension are zeros)
    kPadded,  // K steps and columns of nothing but padding are left out (see padded_form)
    kPacked,  // packed variable-length batch
};

// kMore: the launch has more items than SMs, so blocks ask for further ones; without it the kernel is the plain
// one-item-per-block form (every running count below is a constant 0 there): a launch of the kMore form that has nothing to
// hand out is 1.5 us slower at B1 Hq4 S128 D64 (8.2 against 6.7 us) and 3 % at B2 Hq12 S1000 D128.
// kAlone: causal, some of a head's tiles are items of their own and the others pairs (see SingleTiles).  A form of its own because the
// others are 1 to 3 % slower with that in their item arithmetic (B16 Hq16 Hkv2 S2048 D64 364 -> 375 us, B8 Hq12 Hkv4 S4096 D64 causal
// 286 -> 293).
template <int D, Form kForm, bool kMore, bool kAlone>
__global__ void __launch_bounds__(kFwdThreads, 1)
gqa_fwd_sm100_kernel(const __grid_constant__ CUtensorMap mapQ, const __grid_constant__ CUtensorMap mapK,
                     const __grid_constant__ CUtensorMap mapV, const FwdParams p) {
    using Cfg = FwdCfg<D>;
    extern __shared__ __align__(1024) uint8_t smem[];
    if ((smem_u32(smem) & 1023u) != 0) {  // swizzled panels need 1024-byte alignment; report instead of computing garbage
        pdl_wait();
        if (threadIdx.x == 0) atomicCAS(p.status, 0u, 0x80000000u | (99u << 20));
        return;
    }
    uint8_t* sQ = smem;
    uint8_t* sK = sQ + Cfg::kSmemQ;
    uint8_t* sV = sK + Cfg::kStages * Cfg::kTileBytes;
    uint64_t* bars = reinterpret_cast<uint64_t*>(sV + Cfg::kStages * Cfg::kTileBytes);
    uint64_t* q_full = bars;                       // [2]  per tile
    uint64_t* o_full = bars + 2;                   // [2]  per tile
    uint64_t* s_full = bars + 4;                   // [4]  per (tile, S buffer): S(j) written
    uint64_t* p_full = bars + 8;                   // [4]  per (tile, S buffer): P(j) written by the warpgroup
    uint64_t* pv_done = bars + 12;                 // [4]  per (tile, S buffer): P(j) V completed
    uint64_t* k_full = bars + 16;                  // [kStages]
    uint64_t* k_empty = k_full + Cfg::kStages;     // [kStages]
    uint64_t* v_full = k_empty + Cfg::kStages;     // [kStages]
    uint64_t* v_empty = v_full + Cfg::kStages;     // [kStages]
    uint64_t* q_empty = v_empty + Cfg::kStages;    // [2]  per tile: the last S of the item has been computed
    uint64_t* o_empty = q_empty + 2;               // [2]  per tile: the epilogue has read O
    uint64_t* item_full = o_empty + 2;             // [kItemSlots] producer -> everybody: the block's next item
    uint64_t* item_empty = item_full + kItemSlots; // [kItemSlots]
    uint64_t* clc_full = item_empty + kItemSlots;  // answer to a request for another item
    uint8_t* clc_answer = reinterpret_cast<uint8_t*>(clc_full + 2);
    constexpr int kBars = 16 + 4 * Cfg::kStages + 4 + 2 * kItemSlots + 2;
    static_assert(kBars % 2 == 0, "the answer is 16-byte aligned");
    volatile int* item_slot = reinterpret_cast<volatile int*>(clc_answer + 16);  // [kItemSlots][4]: x, y, z of the block (packed: hq, q0, y0, len)
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(clc_answer + 16 + kItemSlots * 16);
    volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(tmem_slot + 1);
    static_assert(kBars * 8 + 16 + kItemSlots * 16 + 8 <= Cfg::kBarBytes, "barrier area");

    const int tid = threadIdx.x;
    const int warp = tid >> 5;
    const int lane = tid & 31;
    AbortCtx ctx{abort_flag, p.status};

    // ---- work items.  An item is what one thread block of the grid stands for: `tiles` query tiles of one query head.
    // A block works through its own item and then takes over blocks of the same launch that have not started yet, one
    // after the other (cluster launch control hands them out in grid order), with every ring and barrier carrying on:
    // the next item's Q, K and V are loaded and its first S is computed while the last products and the epilogue of the
    // one before run, and the set-up of a block is paid once per SM.  One block per item cost about 12 000 cycles of
    // start and finish per item.  B200, back to back: B16 Hq16 S2048 D64 414 -> 380 us (804 -> 703 thousand SM cycles),
    // S1024 136 -> 116 us, causal B8 Hq12 S4096 380 -> 343 us; D = 128, where the power cap sets the clock, 1 to 2 %
    // (B16 Hq16 S4096 1 940 -> 1 904 us); a launch of one item per SM is unchanged.  The same loop without the take-over
    // is as slow as before (412 us), so it is the overlap that pays.
    struct Item {
        int hq, q0, b, y0, len, n_tiles;
        int n_blk0, n_blk1, n_max;  // key blocks of the two tiles and the larger of the two
    };
    // Packed variable-length batch: the sequence is a row range [y0, y0 + len) of the one [T, H*D] matrix; rows past
    // its end belong to the next sequence (or read as zeros past T): as keys they are masked like keys beyond S,
    // as queries they are computed and not stored.  An item beyond its sequence (the grid covers max_seqlen) or beyond the
    // end of the work list has n_tiles = 0 and no key blocks; the producer passes most of them over, and every role does
    // nothing in one.
    [[maybe_unused]] PackedList* list = reinterpret_cast<PackedList*>(smem + Cfg::kOffList);
    auto item_at = [&](int hq, int q0, int b, int y0, int len, bool pair) -> Item {
        Item w;
        w.hq = hq;
        w.q0 = q0;
        w.b = b;
        w.y0 = y0;
        w.len = len;
        w.n_tiles = w.q0 >= w.len ? 0 : (pair && w.q0 + kTile < w.len) ? 2 : 1;
        const int n_blocks_all = (w.len + kTile - 1) / kTile;  // the last block may be partial: keys at and beyond len are masked
        w.n_blk0 = (w.n_tiles == 0) ? 0 : p.causal ? (w.q0 / kTile + 1) : n_blocks_all;
        w.n_blk1 = (w.n_tiles == 2) ? (p.causal ? (w.q0 / kTile + 2) : n_blocks_all) : 0;
        w.n_max = max(w.n_blk0, w.n_blk1);
        return w;
    };
    auto decode = [&](int x, int y, int z) -> Item {
        int n_groups = p.n_groups;
        if constexpr (kForm == kPacked) {
            if (p.n_listed > 0) {  // the longest sequence first, head by head
                const int u = list->run_of(x, p.n_listed);
                const int r = x - list->first[u];
                n_groups = (list->first[u + 1] - list->first[u]) / p.Hq;
                if (r >= n_groups * p.Hq) return Item{};  // beyond the end of the list
                z = list->seq[u];
                y = r / n_groups;
                x = r % n_groups;
            }
        } else if (kAlone || p.tile_slow) {
            const int place = z;
            z = y;
            y = x;
            x = place;
        }
        if constexpr (kAlone) {  // the last p.singles tiles of a head one by one, the others in pairs
            const bool pair = x >= p.singles;
            return item_at(y, (pair ? 2 * (n_groups - 1 - x) : 2 * n_groups - p.singles - 1 - x) * kTile, z, 0, p.S, pair);
        }
        const int q0 = (p.causal ? (n_groups - 1 - x) : x) * p.tiles * kTile;  // heavy causal tiles first
        if constexpr (kForm == kPacked) {
            const int y0 = p.cu[z];
            return item_at(y, q0, 0, y0, p.cu[z + 1] - y0, p.tiles == 2);
        } else {
            return item_at(y, q0, z, 0, p.S, p.tiles == 2);
        }
    };
    // The j-th item of this block, published by the producer; false = no more (or give up).  In the plain form every role
    // knows the only one.  (Knowing the first one here as well, with no wait for it: 389 against 382 us at B16 Hq16 S2048.)
    // Of a packed batch the producer publishes the item itself: with every role looking the place up for itself (a search, two
    // divisions and the sequence's limits from memory) short items are slower: B200, Hq16 Hkv4 D128 causal, 128 sequences of
    // 300 tokens 208 us against 178, 600 of 1 to 200 tokens 290 against 268.
    auto fetch_item = [&](int j, Item& w) -> bool {
        int x = blockIdx.x, y = blockIdx.y, z = blockIdx.z;
        if constexpr (kMore) {
            const int sl = j % kItemSlots;
            if (!mbar_wait(&item_full[sl], (j / kItemSlots) & 1, ctx, 14)) return false;
            x = item_slot[sl * 4 + 0];
            y = item_slot[sl * 4 + 1];
            z = item_slot[sl * 4 + 2];
            [[maybe_unused]] const int len = kForm == kPacked ? item_slot[sl * 4 + 3] : 0;
            mbar_arrive(&item_empty[sl]);
            if (x < 0) return false;
            if constexpr (kForm == kPacked) {
                w = item_at(x, y, 0, z, len, p.tiles == 2);
                return true;
            }
        }
        w = decode(x, y, z);
        return true;
    };

    // ---- setup ------------------------------------------------------------------
    if (tid == 0) {
        for (int i = 0; i < 2; ++i) {
            mbar_init(&q_full[i], 1);
            mbar_init(&q_empty[i], 1);
            mbar_init(&o_full[i], 1);
            mbar_init(&o_empty[i], 128);
        }
        for (int i = 0; i < 4; ++i) {
            mbar_init(&s_full[i], 1);
            mbar_init(&p_full[i], 128);
            mbar_init(&pv_done[i], 1);
        }
        for (int i = 0; i < Cfg::kStages; ++i) {
            mbar_init(&k_full[i], 1);
            mbar_init(&k_empty[i], 2);  // both issuers release every block, also one they do not use
            mbar_init(&v_full[i], 1);
            mbar_init(&v_empty[i], 2);
        }
        for (int i = 0; i < kItemSlots; ++i) {
            mbar_init(&item_full[i], 1);
            mbar_init(&item_empty[i], 320);  // every softmax and issuer thread
        }
        mbar_init(clc_full, 1);
        fence_mbar_init();
    }
    // Everything above overlaps the end of the kernel in front in the stream; global memory is first used from here on.  Tensor
    // memory is taken after the wait as well: held before it, a kernel in front that lets its dependents come up before it has
    // taken its own would wait for this block, and this block for the end of that kernel.
    // It pays for forwards back to back only.  B200: B1 Hq4 S128 D64 5.75 -> 4.8 us, on inputs from memory 6.3 -> 5.1; B2 Hq12 S1000
    // D128 19.8 -> 19.1; behind a cuBLAS product or an element-wise kernel no gain (8.0 -> 8.0 and 23.8 -> 24.1 with that kernel).
    pdl_wait();
    if (warp == kWarpMma0) {
        tmem_alloc(tmem_slot, Cfg::kTmemCols);
        tmem_relinquish();
    }
    // a non-zero status word (a bounded wait gave up earlier and nobody has read the report yet) makes
    // every later thread block skip its work, so a wedged launch drains in one wave
    if (tid == 0) *abort_flag = (*reinterpret_cast<volatile unsigned int*>(p.status) != 0u) ? 98u : 0u;
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = *tmem_slot;
    if (*abort_flag != 0) {  // uniform: every thread reads the flag after the barrier
        if (warp == kWarpMma0) tmem_dealloc(tmem, Cfg::kTmemCols);
        return;
    }

    if constexpr (kForm == kPacked) {
        if (p.n_listed > 0) list->build(p.cu, p.n_listed, p.tiles * kTile, p.n_groups, p.Hq, 1);
    }

    if (warp == kWarpTma) {
        // ======================= TMA producer =======================
        if (elect_one()) {
            tma_prefetch_desc(&mapQ);
            tma_prefetch_desc(&mapK);
            tma_prefetch_desc(&mapV);
            uint32_t n_claims = 0;
            int x = blockIdx.x, y = blockIdx.y, z = blockIdx.z;
            [[maybe_unused]] Item next;  // packed batch: the item there
            // The next item: x = -1 when there is none.  False: a wait gave up.  Empty items of a packed batch are passed
            // over here, at 0.3 to 0.4 us each, while the other roles wait for the next one.  Long runs of them (a batch with many
            // empty sequences beside a long one) would outlast that wait, so every kMaxPassedOver-th is published: the
            // roles find nothing to do in it and wait anew, and the look at the status word comes round.
            auto claim = [&]() -> bool {
                for (int passed_over = 0;; ++passed_over) {
                    mbar_expect_tx(clc_full, 16);
                    clc_try_cancel(clc_answer, clc_full);
                    if (!mbar_wait(clc_full, n_claims & 1, ctx, 15)) return false;
                    ++n_claims;
                    const bool taken = clc_read_answer(clc_answer, x, y, z);
                    fence_proxy_async_smem();  // the answer has been read before the next one is written
                    if (!taken) {
                        x = -1;
                        return true;
                    }
                    if constexpr (kForm != kPacked) return true;
                    next = decode(x, y, z);
                    if (passed_over >= kMaxPassedOver || next.n_tiles > 0) return true;
                }
            };
            bool ok = true;
            if constexpr (kMore && kForm == kPacked) {
                next = decode(x, y, z);
                if (next.n_tiles == 0) ok = claim();
            }
            uint32_t kb = 0;             // key blocks loaded so far, over all items
            int n_q[2] = {0, 0};         // loads of the two Q tiles so far
            for (int j = 0; ok; ++j) {
                if constexpr (kMore) {
                    const int sl = j % kItemSlots;
                    if (j >= kItemSlots && !mbar_wait(&item_empty[sl], (j / kItemSlots - 1) & 1, ctx, 13)) break;
                    // a block of this launch that gave up has left a non-zero status word: stop taking items
                    if (j > 0 && *reinterpret_cast<volatile unsigned int*>(p.status) != 0u) {
                        *abort_flag = 98u;
                        break;
                    }
                    if constexpr (kForm == kPacked) {
                        item_slot[sl * 4 + 0] = x < 0 ? -1 : next.hq;
                        item_slot[sl * 4 + 1] = next.q0;
                        item_slot[sl * 4 + 2] = next.y0;
                        item_slot[sl * 4 + 3] = next.len;
                    } else {
                        item_slot[sl * 4 + 0] = x;
                        item_slot[sl * 4 + 1] = y;
                        item_slot[sl * 4 + 2] = z;
                    }
                    mbar_arrive(&item_full[sl]);
                    if (x < 0) {
                        pdl_launch_dependents();
                        break;
                    }
                }
                const Item w = kMore && kForm == kPacked ? next : decode(x, y, z);
                const int hkv = w.hq / (p.Hq / p.Hkv);
                // Tensor-map coordinates (x = column, y = position in the sequence, z = matrix).  [B,H,S,D] is B*H matrices
                // [S, D]; [B,S,H,D] is B matrices [S, H*D] with the head at x = head * D.  Rows at y >= S read as zeros.
                const int q_x = p.bshd ? w.hq * D : 0, q_z = p.bshd ? w.b : w.b * p.Hq + w.hq;
                const int kv_x = p.bshd ? hkv * D : 0, kv_z = p.bshd ? w.b : w.b * p.Hkv + hkv;
                for (int t = 0; t < w.n_tiles && ok; ++t) {
                    if (n_q[t] > 0 && !mbar_wait(&q_empty[t], (n_q[t] - 1) & 1, ctx, 12)) { ok = false; break; }
                    ++n_q[t];
                    mbar_expect_tx(&q_full[t], Cfg::kTileBytes);
                    for (int pn = 0; pn < Cfg::kPanels; ++pn)
                        tma_load_3d(sQ + t * Cfg::kTileBytes + pn * kPanel, &mapQ, &q_full[t], q_x + pn * 64, w.y0 + w.q0 + t * kTile, q_z);
                }
                for (int n = 0; n < w.n_max && ok; ++n, ++kb) {
                    const uint32_t st = kb % Cfg::kStages;
                    const uint32_t use = kb / Cfg::kStages;
                    if (use > 0 && !mbar_wait(&k_empty[st], (use - 1) & 1, ctx, 10)) { ok = false; break; }
                    mbar_expect_tx(&k_full[st], Cfg::kTileBytes);
                    for (int pn = 0; pn < Cfg::kPanels; ++pn)
                        tma_load_3d(sK + st * Cfg::kTileBytes + pn * kPanel, &mapK, &k_full[st], kv_x + pn * 64, w.y0 + n * kTile, kv_z);
                    if (use > 0 && !mbar_wait(&v_empty[st], (use - 1) & 1, ctx, 11)) { ok = false; break; }
                    mbar_expect_tx(&v_full[st], Cfg::kTileBytes);
                    for (int pn = 0; pn < Cfg::kPanels; ++pn)
                        tma_load_3d(sV + st * Cfg::kTileBytes + pn * kPanel, &mapV, &v_full[st], kv_x + pn * 64, w.y0 + n * kTile, kv_z);
                }
                if constexpr (!kMore) {
                    pdl_launch_dependents();  // the last loads are on their way
                    break;
                }
                if (ok) ok = claim();
            }
        }
    } else if (warp >= kWarpMma0) {
        // ======================= issuer of tile t: S(j) = Q K(j)^T per half-block, O += P(j) V(j) =======================
        // The whole warp runs the loop (uniform control flow); `leader` marks the one lane that issues.
        const int t = warp - kWarpMma0;
        const uint32_t leader = elect_one() ? 1u : 0u;
        const uint32_t idesc_qk = make_idesc_bf16(128, kHalf, false, false);
        const int n_cols = kForm == kPadded ? product_cols(p.d_real) : D;  // columns of Q, K, V that are not all padding
        const uint32_t idesc_pv = make_idesc_bf16(128, n_cols, false, true);
        const uint32_t q_addr = smem_u32(sQ) + t * Cfg::kTileBytes, k_addr = smem_u32(sK), v_addr = smem_u32(sV);
        const uint32_t colS = tmem + (t ? Cfg::kColS1 : Cfg::kColS0), colO = tmem + (t ? Cfg::kColO1 : Cfg::kColO0);
        bool ok = true;
        // running counts over all items of this block (ring stages and barrier parities): key blocks of the rings,
        // key blocks and items of this tile
        uint32_t kb = 0, cb = 0, n_done = 0;
        Item w;
        for (int it = 0; ok && fetch_item(it, w); ++it) {
            const uint32_t n_blk = t ? w.n_blk1 : w.n_blk0, n_max = w.n_max;
            if (n_blk > 0) {
                ok = mbar_wait(&q_full[t], n_done & 1, ctx, 20);
                // S of half h of key block n: rows 64h.. of the block are the B operand (K-major panels, 64 rows = 8192
                // bytes down).  It goes where P of the same half of the block before lives: that product must have completed.
                auto issue_qk = [&](uint32_t n, uint32_t h) -> bool {
                    const uint32_t st = (kb + n) % Cfg::kStages;
                    if (cb + n > 0 && !mbar_wait(&pv_done[t * 2 + h], (cb + n - 1) & 1, ctx, 22)) return false;
                    if (h == 0 && !mbar_wait(&k_full[st], ((kb + n) / Cfg::kStages) & 1, ctx, 21)) return false;
                    tc_fence_after_sync();
                    const uint32_t b0 = k_addr + st * Cfg::kTileBytes + h * (kHalf * 128);
                    auto step = [&](int kk) {
                        const uint32_t off = (kk >> 2) * kPanel + (kk & 3) * 32;
                        umma_ss_pred(leader, colS + h * kHalf, make_sdesc_sw128(q_addr + off, 16, 1024),
                                     make_sdesc_sw128(b0 + off, 16, 1024), idesc_qk, kk > 0);
                    };
                    if constexpr (kForm == kPadded) {
                        for (int kk = 0; kk < n_cols / 16; ++kk) step(kk);
                    } else {
#pragma unroll
                        for (int kk = 0; kk < D / 16; ++kk) step(kk);
                    }
                    umma_commit_pred(leader, &s_full[t * 2 + h]);
                    if (h == 1) umma_commit_pred(leader, &k_empty[st]);
                    if (kMore && h == 1 && n + 1 == n_blk) umma_commit_pred(leader, &q_empty[t]);
                    if (t == 0) GQA_FTRACE(1, 2 * n + h, 0);
                    return true;
                };
                if (ok) ok = issue_qk(0, 0);
#pragma unroll 1
                for (uint32_t n = 0; n < n_blk && ok; ++n) {
                    const uint32_t st = (kb + n) % Cfg::kStages;
#pragma unroll
                    for (uint32_t h = 0; h < 2; ++h) {
                        if (ok && (h == 0 || n + 1 < n_blk)) ok = issue_qk(n + h, h ^ 1);  // the next S
                        if (ok && h == 0) ok = mbar_wait(&v_full[st], ((kb + n) / Cfg::kStages) & 1, ctx, 23);
                        if (ok && h == 0 && n == 0 && n_done > 0) ok = mbar_wait(&o_empty[t], (n_done - 1) & 1, ctx, 25);  // the item before has read O
                        if (ok) ok = mbar_wait(&p_full[t * 2 + h], (cb + n) & 1, ctx, 24);
                        if (!ok) break;
                        tc_fence_after_sync();
                        if (t == 0) GQA_FTRACE(1, 2 * n + h, 1);
                        const uint32_t b0 = v_addr + st * Cfg::kTileBytes + h * (kHalf / 16) * 2048;
#pragma unroll
                        for (int kk = 0; kk < kHalf / 16; ++kk)
                            umma_ts_pred(leader, colO, colS + h * kHalf + kk * 8, make_sdesc_sw128(b0 + kk * 2048, kPanel, 1024),
                                         idesc_pv, (n > 0 || h > 0 || kk > 0));
                        umma_commit_pred(leader, &pv_done[t * 2 + h]);
                        if (h == 1) umma_commit_pred(leader, &v_empty[st]);
                        if (h == 1 && n + 1 == n_blk) umma_commit_pred(leader, &o_full[t]);
                        if (t == 0) GQA_FTRACE(1, 2 * n + h, 2);
                    }
                }
                ++n_done;
            }
            // blocks that only the other tile uses: released as soon as they are there (waited for, so that the arrival
            // falls into the right phase)
            for (uint32_t n = n_blk; n < n_max && ok; ++n) {
                const uint32_t st = (kb + n) % Cfg::kStages;
                const uint32_t par = ((kb + n) / Cfg::kStages) & 1;
                ok = mbar_wait(&k_full[st], par, ctx, 26);
                if (ok && leader) mbar_arrive(&k_empty[st]);
                if (ok) ok = mbar_wait(&v_full[st], par, ctx, 27);
                if (ok && leader) mbar_arrive(&v_empty[st]);
            }
            if constexpr (!kMore) break;
            kb += n_max;
            cb += n_blk;
        }
    } else {
        // ======================= softmax warpgroups =======================
        const int t = warp >> 2;                      // query tile owned by this warpgroup
        const int r = (warp & 3) * 32 + lane;         // row inside the tile == TMEM lane
        uint32_t cb = 0, n_done = 0;                  // key blocks and items of this tile so far (barrier parities)
        bool ok = true;
        Item w;
        for (int it = 0; ok && fetch_item(it, w); ++it) {
            const int n_blk = t ? w.n_blk1 : w.n_blk0;
            if (n_blk == 0) {
                if constexpr (kMore) continue;
                else break;
            }
            const int q0 = w.q0, len = w.len, hq = w.hq, b = w.b, y0 = w.y0;
            const int q_row0 = (b * p.Hq + hq) * p.S + y0 + q0;   // row in [B,Hq,S] order (LSE)
            const uint32_t lane_addr = (uint32_t)((warp & 3) * 32) << 16;
            const uint32_t tS = tmem + lane_addr + (t == 0 ? Cfg::kColS0 : Cfg::kColS1);
            const uint32_t tO = tmem + lane_addr + (t == 0 ? Cfg::kColO0 : Cfg::kColO1);
            const float c = p.scale_log2;
            const uint64_t c2 = pack_f32x2(c, c);
            const int total = 2 * n_blk;
            const int diag_block = (q0 + t * kTile) / kTile;  // only this block needs the causal mask
            float m_run = -INFINITY;  // running maximum of the raw logits that P is measured against
            float l_run = 0.f;
            for (int j = 0; j < total; ++j) {
                const int n = j >> 1, h = j & 1;
                ok = mbar_wait(&s_full[t * 2 + h], (cb + n) & 1, ctx, 30);
                if (!ok) break;
                tc_fence_after_sync();
                if (warp == 0) GQA_FTRACE(0, j, 0);
                if (warp == 4) GQA_FTRACE(2, j, 0);
                if (t == 0) GQA_FTRACE(4, j, warp & 3);
                // last valid column of this row inside the 128-key block: the causal diagonal and / or the end of S
                const bool diag = p.causal && (n == diag_block);
                const int s_left = len - n * kTile;  // keys of this block that exist
                const bool masked = diag || s_left < kTile;
                const int lim = min(diag ? r : kTile - 1, s_left - 1);
                const int col0 = h * kHalf;  // column of v[0] inside the 128-key block
                // the 64-column half row of S into registers (one TMEM round trip), then the row maximum with
                // four independent chains of three-input maxima
                uint32_t v[kHalf];
                tmem_ld32p(tS + col0, v);
                tmem_ld32p(tS + col0 + 32, v + 32);
                tmem_wait_ld();
                float mx;
                {
                    float m4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
                    if (masked) {
#pragma unroll
                        for (int i = 0; i < kHalf; ++i)
                            m4[i & 3] = (col0 + i > lim) ? m4[i & 3] : fmaxf(m4[i & 3], __uint_as_float(v[i]));
                    } else {
#pragma unroll
                        for (int i = 0; i < kHalf; i += 2)
                            m4[(i >> 1) & 3] = max3_f32(m4[(i >> 1) & 3], __uint_as_float(v[i]), __uint_as_float(v[i + 1]));
                    }
                    mx = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3]));
                }
                if (warp == 0) GQA_FTRACE(0, j, 1);
                const float m_new = fmaxf(m_run, mx);
                const bool grow = (m_new - m_run) * c > kRescaleThreshold;  // true on the first half-block (m_run = -inf)
                if (__any_sync(0xffffffffu, grow)) {
                    const float m_next = grow ? m_new : m_run;
                    const float alpha = ex2_approx((m_run - m_next) * c);
                    l_run *= alpha;
                    m_run = m_next;
                    if (j > 0) {
                        // O holds P(0..j-1) V; the last of those products may still be running
                        ok = mbar_wait(&pv_done[t * 2 + (h ^ 1)], (cb + ((j - 1) >> 1)) & 1, ctx, 32);
                        if (!ok) break;
                        tc_fence_after_sync();
#pragma unroll 1
                        for (int ch = 0; ch < D / 32 && (kForm != kPadded || ch * 32 < p.d_real); ++ch) {
                            uint32_t w[32];
                            tmem_ld32(tO + ch * 32, w);
                            tmem_wait_ld();
#pragma unroll
                            for (int i = 0; i < 32; ++i) w[i] = __float_as_uint(__uint_as_float(w[i]) * alpha);
                            tmem_st32(tO + ch * 32, w);
                        }
                    }
                }
                // P = exp2(c*s - c*m) (packed fma), row sum (two packed partial sums), packed bf16 into the first
                // 32 columns of this S buffer
                const float mc = m_run * c;
                float l_add;
                if (!masked) {
                    const uint64_t nmc2 = pack_f32x2(-mc, -mc);
                    uint64_t l2[2] = {0ull, 0ull};
#pragma unroll
                    for (int ch = 0; ch < 2; ++ch) {
                        uint32_t pk[16];
#pragma unroll
                        for (int i = 0; i < 16; ++i) {
                            const uint64_t x = fma_f32x2(
                                pack_f32x2(__uint_as_float(v[ch * 32 + 2 * i]), __uint_as_float(v[ch * 32 + 2 * i + 1])), c2, nmc2);
                            float x0, x1;
                            unpack_f32x2(x, x0, x1);
                            const float e0 = ex2_approx(x0), e1 = ex2_approx(x1);
                            l2[i & 1] = add_f32x2(l2[i & 1], pack_f32x2(e0, e1));
                            pk[i] = pack_bf16x2(e0, e1);
                        }
                        tmem_st16(tS + col0 + ch * 16, pk);
                    }
                    float a0, a1, b0, b1;
                    unpack_f32x2(l2[0], a0, a1);
                    unpack_f32x2(l2[1], b0, b1);
                    l_add = (a0 + a1) + (b0 + b1);
                } else {
                    float l4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                    for (int ch = 0; ch < 2; ++ch) {
                        uint32_t pk[16];
#pragma unroll
                        for (int i = 0; i < 16; ++i) {
                            const int cc = col0 + ch * 32 + 2 * i;
                            float e0 = ex2_approx(fmaf(__uint_as_float(v[ch * 32 + 2 * i]), c, -mc));
                            float e1 = ex2_approx(fmaf(__uint_as_float(v[ch * 32 + 2 * i + 1]), c, -mc));
                            if (cc > lim) e0 = 0.f;
                            if (cc + 1 > lim) e1 = 0.f;
                            l4[i & 3] += e0 + e1;
                            pk[i] = pack_bf16x2(e0, e1);
                        }
                        tmem_st16(tS + col0 + ch * 16, pk);
                    }
                    l_add = (l4[0] + l4[1]) + (l4[2] + l4[3]);
                }
                l_run += l_add;
                tmem_wait_st();
                tc_fence_before_sync();
                mbar_arrive(&p_full[t * 2 + h]);
                if (warp == 0) GQA_FTRACE(0, j, 2);
                if (warp == 4) GQA_FTRACE(2, j, 2);
                GQA_FTRACE(t == 0 ? 3 : 5, j, warp & 3);
            }
            // epilogue: O / l -> bf16, LSE
            if (ok) ok = mbar_wait(&o_full[t], n_done & 1, ctx, 31);
            if (ok) {
                tc_fence_after_sync();
                // rows beyond the end of the sequence are not stored (the TMEM loads below are warp-wide
                // instructions: every lane runs them, only the stores are guarded)
                const bool row_ok = q0 + t * kTile + r < len;
                const float inv_l = 1.0f / l_run;
                const size_t grow_ = (size_t)q_row0 + t * kTile + r;
                __nv_bfloat16* orow = p.bshd ? p.O + ((size_t)(b * p.S + y0 + q0 + t * kTile + r) * p.Hq + hq) * D
                                             : p.O + grow_ * p.d_real;
#pragma unroll 1
                for (int ch = 0; ch < D / 32 && (kForm != kPadded || ch * 32 < p.d_real); ++ch) {
                    uint32_t v[32];
                    tmem_ld32(tO + ch * 32, v);
                    tmem_wait_ld();
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        uint4 o;
                        o.x = pack_bf16x2(__uint_as_float(v[8 * i + 0]) * inv_l, __uint_as_float(v[8 * i + 1]) * inv_l);
                        o.y = pack_bf16x2(__uint_as_float(v[8 * i + 2]) * inv_l, __uint_as_float(v[8 * i + 3]) * inv_l);
                        o.z = pack_bf16x2(__uint_as_float(v[8 * i + 4]) * inv_l, __uint_as_float(v[8 * i + 5]) * inv_l);
                        o.w = pack_bf16x2(__uint_as_float(v[8 * i + 6]) * inv_l, __uint_as_float(v[8 * i + 7]) * inv_l);
                        if (row_ok && ch * 32 + i * 8 < p.d_real) *reinterpret_cast<uint4*>(orow + ch * 32 + i * 8) = o;
                    }
                }
                if (p.LSE && row_ok) p.LSE[grow_] = (m_run * c + log2f(l_run)) * kLn2;
                // every column of O has been read: the next item's first product may overwrite them
                tc_fence_before_sync();
                mbar_arrive(&o_empty[t]);
            }
            if constexpr (!kMore) break;
            cb += n_blk;
            ++n_done;
        }
    }

    // ---- teardown ---------------------------------------------------------------
    tc_fence_before_sync();
    __syncthreads();
    if (warp == kWarpMma0) {
        if (*abort_flag != 0) abort_grace_period();  // in-flight copies and MMAs land before TMEM is released
        tmem_dealloc(tmem, Cfg::kTmemCols);
    }
}

// Causal launches of more query tiles than SMs, longest items first: how many of a head's last tiles are items of their own, the
// rest being pairs.  A pair takes 3 130 cycles per key block and one tile alone 2 450, so where the longest pair bounds the launch
// (bound_by_longest) it ends sooner with that pair's tiles on two SMs.  They then take 1.57 times as much of the SMs' time, which an
// idle chip has and one with several streams has not: so only as many tiles stand alone as shorten the launch.
// Units of 800 cycles: a key block of a pair takes 4 and a pair 3 more, one of a single tile 3 and the tile 2 more; of more items than
// SMs the ones of the second round start when the shortest of the first round end.
// B200, graph replays, us per launch of a stream with one / two / four streams, all pairs; this rule; all single tiles: B2 Hq12 S1000
// D128 (4 of 8 tiles) 20.7 / 21.7 / 38; 16.4 / 24.8 / 48; 17.1 / 28.1 / 55.  B1 Hq16 S2048 D128 (6 of 16) 35 / 39 / 74; 29 / 48 / 93;
// 29 / 54 / 107.  B1 Hq4 S8192 D128 (18 of 64) 110 / 114 / 212; 91 / 136 / 263; 91 / 161 / 318.  B4 Hq8 S700 D128 (2 of 6) 16.6 / 17.9 /
// 32.8; 13.8 / 20.2 / 38.7; 14.3 / 24.3 / 47.4.  B1 Hq32 S1024 D128 (2 of 8) 21.5 / 26.4 / 50; 18.4 / 30.5 / 59; 20.0 / 35.6 / 70.
struct SingleTiles {
    long long n, heads, sms;  // query tiles of a head; heads of the batch
    // The launches in question: as pairs they take as long as the longest one (with so few items the SMs' share of the key blocks
    // never bounds them), and that is longer than all tiles on their own take: as long as the longest of them, or the SMs' share and a
    // sixth for what list scheduling leaves over.  (Launches of more heads would end sooner in one stream as well, B1 Hq10 S4096 D128 in 54 us instead
    // of 67, but take longer in several, 93 instead of 80 and 179 instead of 152, and stay pairs.)
    bool bound_by_longest() const {
        const long long blocks = heads * n * (n + 1) / 2, longest_pair = n % 2 == 0 ? 4 * n : std::max(4 * (n - 1), 3 * n);
        return std::max(6 * n * sms, 7 * blocks) + 8 * sms < 2 * longest_pair * sms;
    }
    long long length(long long singles, long long place) const {
        return place < singles ? 3 * (n - place) + 2 : 4 * (n - singles - 2 * (place - singles)) + 3;
    }
    long long time(long long singles) const {  // an even number of tiles in pairs
        const long long places = singles + (n - singles) / 2, items = heads * places;
        long long t = std::max(length(singles, 0), singles < places ? length(singles, singles) : 0);
        if (items <= sms) return t;
        for (long long place = sms / heads; place < places; ++place) {  // the last of the heads' items there: it has the longest one to wait for
            const long long behind = (place + 1) * heads - 1 - sms;
            if (behind >= 0) t = std::max(t, length(singles, place) + (behind < sms ? length(singles, (sms - 1 - behind) / heads) : t));
        }
        return t;
    }
    int count() const {
        if (!bound_by_longest()) return 0;
        long long singles = (n + 4) / 4;  // from here on the longest pair is no longer than the longest tile
        singles += (n - singles) % 2;
        long long best = singles, best_time = time(singles);
        while ((singles -= 2) > 0 && length(singles, singles) <= best_time) {
            const long long t = time(singles);
            if (t <= best_time) best = singles, best_time = t;
        }
        return (int)best;
    }
};

template <int D>
int launch_fwd_t(const void* Q, const void* K, const void* V, void* O, float* LSE, const Shape& s, unsigned int* status,
                 cudaStream_t stream) {
    using Cfg = FwdCfg<D>;
    CUtensorMap mq, mk, mv;
    // see the coordinates in the kernel
    // (the matrices are s.D columns wide; a box that reaches beyond them reads zeros there)
    const uint64_t S = s.S, qc = s.bshd ? (uint64_t)s.Hq * D : s.D, kc = s.bshd ? (uint64_t)s.Hkv * D : s.D;
    const uint64_t nq = s.bshd ? s.B : (uint64_t)s.B * s.Hq, nkv = s.bshd ? s.B : (uint64_t)s.B * s.Hkv;
    int rc = make_tile3_tmap(&mq, Q, qc, S, nq, S * qc, kTile);
    if (rc) return rc;
    rc = make_tile3_tmap(&mk, K, kc, S, nkv, S * kc, kTile);
    if (rc) return rc;
    rc = make_tile3_tmap(&mv, V, kc, S, nkv, S * kc, kTile);
    if (rc) return rc;
    FwdParams p;
    p.O = static_cast<__nv_bfloat16*>(O);
    p.LSE = LSE;
    p.status = status;
    p.Hq = s.Hq;
    p.Hkv = s.Hkv;
    p.S = s.S;
    p.causal = s.causal;
    p.bshd = s.bshd;
    p.d_real = s.D;
    p.cu = s.cu_seqlens;
    // Two query tiles per item share the K/V blocks and keep the tensor core busy in turns: 3 130 cycles per key block for both,
    // against 2 450 for one tile alone.  One tile per item finishes sooner when every tile gets an SM of its own (B200, D = 128
    // causal: 128 tiles, B1 Hq16 S1024, 22.5 us as single tiles against 25.6 us as pairs; with four streams 36 against 25 per launch
    // of one); the longest ones also where they bound a launch of more tiles (SingleTiles).
    const int n_tiles = ((s.cu_seqlens ? s.max_seqlen : s.S) + kTile - 1) / kTile, n_seqs = s.cu_seqlens ? s.n_seqs : s.B;
    // Items of a packed batch are listed where that pays and the lengths differ (equal ones are in order as they are: with the
    // list 8 sequences of 300 tokens, Hq16 D128, take 18.4 us instead of 17.3).  Every sequence ends with one partial item at
    // the most, which bounds the list.
    const bool listed = s.cu_seqlens && lengths_differ(n_seqs, s.max_seqlen, s.S) &&
                        list_pays(n_seqs, s.max_seqlen, s.S, 2 * kTile, s.Hq, sm_count());
    p.n_listed = listed ? n_seqs : 0;
    auto items = [&](int tiles) -> long long {
        const long long all = (long long)((n_tiles + tiles - 1) / tiles) * n_seqs;
        return s.Hq * (p.n_listed ? std::min(all, (long long)s.S / (tiles * kTile) + n_seqs) : all);
    };
    // Causal items are of very different length: the longest of all heads first keeps the end of the launch short, as long as
    // L2 holds K and V of what runs at a time (head by head they are read from memory once, however long the launch).  B200, us:
    // B1 Hq16 S4096 D128 94.0 -> 65.0, D64 82.2 -> 55.3; B1 Hq32 S2048 D128 71.9 -> 51.5; B16 Hq16 Hkv2 S4096 D64 (34 MB of K and
    // V) 764 -> 737, but B8 Hq32 Hkv8 S8192 D128 (268 MB) 3 968 -> 4 130.
    p.tile_slow = s.causal && !s.cu_seqlens && s.kv_rows() * s.D * 4 <= kOrderKvBytes;
    p.tiles = items(1) <= sm_count() ? 1 : 2;
    p.singles = p.tiles == 2 && p.tile_slow ? SingleTiles{n_tiles, (long long)n_seqs * s.Hq, sm_count()}.count() : 0;
    p.n_groups = p.singles + (n_tiles - p.singles + p.tiles - 1) / p.tiles;
    p.scale_log2 = s.scale * kLog2e;
    const dim3 grid = p.n_listed    ? dim3((unsigned)items(p.tiles))
                      : p.tile_slow ? dim3(s.Hq, n_seqs, p.n_groups)
                                    : dim3(p.n_groups, s.Hq, n_seqs);
    const bool more = (p.n_listed ? items(p.tiles) : (long long)p.n_groups * s.Hq * n_seqs) > sm_count();
    auto pick = [&](auto form) {
        constexpr Form F = decltype(form)::value;
        constexpr bool kCanStandAlone = F != kPacked;
        if (kCanStandAlone && p.singles > 0) return more ? gqa_fwd_sm100_kernel<D, F, true, kCanStandAlone> : gqa_fwd_sm100_kernel<D, F, false, kCanStandAlone>;
        return more ? gqa_fwd_sm100_kernel<D, F, true, false> : gqa_fwd_sm100_kernel<D, F, false, false>;
    };
    auto kernel = s.cu_seqlens ? pick(std::integral_constant<Form, kPacked>{})
                  : padded_form(s) ? pick(std::integral_constant<Form, kPadded>{})
                               : pick(std::integral_constant<Form, kNative>{});
    const int smem = Cfg::kSmemTotal + (s.cu_seqlens ? (int)sizeof(PackedList) : 0);
    GQA_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    GQA_CUDA_TRY(launch_after(kernel, grid, kFwdThreads, smem, stream, mq, mk, mv, p));
    count_launch();
    return GQA_OK;
}

}  // namespace

#ifdef GQA_FWD_TRACE
extern "C" int gqa_debug_copy_fwd_trace(long long* host) {
    return (int)cudaMemcpyFromSymbol(host, g_fwd_trace, sizeof(g_fwd_trace));
}
#endif

int launch_fwd_sm100(const void* Q, const void* K, const void* V, void* O, float* LSE, const Shape& s,
                     unsigned int* status, cudaStream_t stream) {
    if (s.Dp() == 64) return launch_fwd_t<64>(Q, K, V, O, LSE, s, status, stream);
    return launch_fwd_t<128>(Q, K, V, O, LSE, s, status, stream);
}

}  // namespace gqa
