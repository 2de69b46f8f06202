// GQA backward, the alternative dQ path for sm_100a: a separate query-parallel pass.
//
// One CTA owns one 128-row query tile of one (batch, query head) and streams the KV head's 128-row key/value
// blocks through TMA rings, as the forward does.  It recomputes, in the natural orientation (a TMEM lane is a
// query row),
//   S  = Q K^T,  dP = dO V^T        (both operands K-major from TMA panels)
//   P  = exp2(scale*log2e * S - LSE*log2e)  -> rounded to bf16
//   dS = bf16(P * (dP - Delta))             -> packed into the head of the S buffer in TMEM
//   dQ += dS K                              (A from TMEM, B = the key block read MN-major)
// and writes dQ = bf16(scale * sum) once.  dQ needs no accumulator in global memory, no zeroing, no finalise pass,
// and its summation order is fixed: it is bit-reproducible by construction.  The price is that S and dP are
// computed a second time (the KV-parallel main kernel still needs them for dK and dV) -- 3 products here plus 4
// there instead of 5 -- and with them a second set of exponentials.
//
// Roles (18 warps):
//   warps 0-15 four elementwise warpgroups; all cover the 128 query rows (thread = row = TMEM lane), warpgroup w
//              handles key columns [32w, 32w+32) of every block
//   warp  16   TMA producer (Q and dO once, K and V rings)
//   warp  17   UMMA issuer (one thread: the products into the one dQ accumulator stay ordered)
// S has two buffers (2 x 128 TMEM columns; dS(n) overwrites the head of S(n)), dP one, which is handed back as soon as it is in
// registers: while the warpgroups work on block n the issuer produces dP(n+1) and S(n+1).  Per block of D = 128 the products
// take 1 650 cycles (two of 128 x 128 x 128 and the 78 cycles of a K step with A in TMEM) and the exponentials 1 024.
//
// The kernel is launched behind the main kernel and runs beside it on the SMs that it leaves idle.  It is the one dependent launch
// that does not wait for the kernel in front before it touches global memory.  What makes that safe: the main kernel's
// trigger stands behind its wait for the preprocess kernel and behind its release of `prep_seen`; nothing is launched between the
// two; dQ overlaps nothing that the main kernel reads (the host looks); the shared memory of both keeps their blocks off one another's
// SMs.
//
// B200, whole call, us, one after the other with blocks of 64 keys and two warpgroups -> now: B2 Hq16 Hkv4 S1024 causal D64 77.7 -> 53.6, D80 105 -> 71.6,
// D128 109 -> 78.9; B1 Hq32 Hkv8 S2048 D128 279 -> 254; B1 Hq64 Hkv8 S4096 D128 causal 1 123 -> 1 023.  (Accumulated dQ: 60.4,
// 79.1, 90.8, 174, 780.)
//
// The reference's first generations are built this way (a dQ kernel per query tile looping over key tiles beside a
// dK/dV kernel per key tile: src/attention/GQA_bwd.cu:29, :415, :1416); its shipped kernel accumulates dQ with
// TMA reduce-add instead (src/attention/GQA_bwd_baseline.cu:360-365), as this library's default path does.
#include "gqa_common.cuh"
#include "gqa_kernels.cuh"
#include "sm100_ptx.cuh"

namespace gqa {
namespace {

using namespace sm100;

constexpr int kTile = 128;             // query rows per tile and key rows per block
constexpr int kPanel = kTile * 128;    // bytes of one 64-column panel of a 128-row tile
constexpr int kEwGroups = 4;           // elementwise warpgroups, 32 keys of a block each
constexpr int kEwThreads = kEwGroups * 128;
constexpr int kWarpTma = kEwThreads / 32, kWarpMma = kWarpTma + 1;
constexpr int kThreads = (kWarpMma + 1) * 32;
constexpr float kLog2e = 1.4426950408889634f;

template <int D>
struct DqCfg {
    static constexpr int kPanels = D / 64;
    static constexpr int kTileBytes = kPanels * kPanel;  // one 128 x D bf16 tile
    // D = 128 (shared memory is full): a key block is released one block later than a value block
    static constexpr int kKStages = (D == 64) ? 4 : 3, kVStages = (D == 64) ? 4 : 2;
    static constexpr int kOffQ = 0;
    static constexpr int kOffDO = kOffQ + kTileBytes;
    static constexpr int kOffK = kOffDO + kTileBytes;
    static constexpr int kOffV = kOffK + kKStages * kTileBytes;
    static constexpr int kOffBars = kOffV + kVStages * kTileBytes;
    static constexpr int kSmemTotal = kOffBars + 512;  // the dynamic window must start 1024-byte aligned (checked)
    static constexpr uint32_t kTmemCols = 512;
    static constexpr uint32_t kColS = 0, kColDP = 256, kColDQ = 384;  // S: two buffers of 128 columns
    static_assert(kColDQ + D <= 512, "TMEM budget");
    static_assert(kSmemTotal <= 227 * 1024, "shared memory budget");
    // (nor beside a block of the main kernel, which may not have taken its tensor memory yet when this one comes up)
    static_assert(kSmemTotal > kHalfSharedMemory, "one CTA per SM is assumed by the 512-column TMEM allocation");
};

struct DqParams {
    __nv_bfloat16* dQ;
    const float* lse;    // [B*Hq*S] natural log
    const float* delta;  // [B*Hq*S] rowsum(dO * O)
    unsigned int* status;
    unsigned int* prep_seen;  // set by the main kernel, which has seen the preprocess kernel's writes
    int Hq, Hkv, S, causal, n_qtiles, bshd, d_real;
    float scale, scale_log2;
};

template <int D, bool kPadded>
__global__ void __launch_bounds__(kThreads, 1)
gqa_bwd_dq_sm100_kernel(const __grid_constant__ CUtensorMap mapQ, const __grid_constant__ CUtensorMap mapDO,
                        const __grid_constant__ CUtensorMap mapK, const __grid_constant__ CUtensorMap mapV,
                        const DqParams p) {
    using Cfg = DqCfg<D>;
    extern __shared__ __align__(1024) uint8_t smem[];
    // The next kernel of the stream waits for this one: so that it waits for the main kernel too, the last block does, on every
    // way out (the others leave their SMs to blocks that have not started).
    auto wait_for_main = [&]() {
        if (threadIdx.x == 0 && blockIdx.x + 1 == gridDim.x && blockIdx.y + 1 == gridDim.y && blockIdx.z + 1 == gridDim.z) pdl_wait();
    };
    if ((smem_u32(smem) & 1023u) != 0) {  // swizzled panels need 1024-byte alignment; report instead of computing garbage
        if (threadIdx.x == 0) atomicCAS(p.status, 0u, 0x80000000u | (99u << 20));
        wait_for_main();
        return;
    }
    uint8_t* sQ = smem + Cfg::kOffQ;
    uint8_t* sDO = smem + Cfg::kOffDO;
    uint8_t* sK = smem + Cfg::kOffK;
    uint8_t* sV = smem + Cfg::kOffV;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::kOffBars);
    uint64_t* qdo_full = bars;              // TMA: Q and dO tiles
    uint64_t* dq_full = bars + 1;           // issuer: every product complete
    uint64_t* s_full = bars + 2;            // [2] per buffer: S(n) written
    uint64_t* dp_full = bars + 4;           // dP(n) written
    uint64_t* dp_free = bars + 5;           // dP(n) in the warpgroups' registers
    uint64_t* ds_ready = bars + 6;          // [2] per buffer: dS(n) stored by the warpgroups (a fast thread may be a block ahead)
    uint64_t* dq_done = bars + 8;           // dS(n) K completed
    uint64_t* k_full = bars + 9;            // [kKStages]
    uint64_t* k_empty = k_full + Cfg::kKStages;
    uint64_t* v_full = k_empty + Cfg::kKStages;  // [kVStages]
    uint64_t* v_empty = v_full + Cfg::kVStages;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(v_empty + Cfg::kVStages);
    volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(tmem_slot + 1);

    const int tid = threadIdx.x;
    const int warp = tid >> 5;
    const int lane = tid & 31;
    AbortCtx ctx{abort_flag, p.status};

    // ---- work decode ------------------------------------------------------------
    const int qt = p.causal ? (p.n_qtiles - 1 - (int)blockIdx.x) : (int)blockIdx.x;  // heavy causal tiles first
    const int hq = blockIdx.y, b = blockIdx.z;
    const int hkv = hq / (p.Hq / p.Hkv);
    const int q0 = qt * kTile;
    const int n_blocks_all = (p.S + kTile - 1) / kTile;
    const int n_blk = p.causal ? qt + 1 : n_blocks_all;
    // Tensor-map coordinates (x = column, y = position in the sequence, z = matrix), as in the other kernels.
    const int q_x = p.bshd ? hq * D : 0, q_z = p.bshd ? b : b * p.Hq + hq;
    const int kv_x = p.bshd ? hkv * D : 0, kv_z = p.bshd ? b : b * p.Hkv + hkv;

    // ---- setup ------------------------------------------------------------------
    const int n_cols = kPadded ? product_cols(p.d_real) : D;  // columns of the products that are not all padding
    if (tid == 0) {
        // This kernel runs beside the main kernel, which is not waited for before the end (see there).  That one's block 0
        // sets the word before this one can start; the wait is for the order of the memory accesses and ends at once.
        bool seen = false;
        for (int i = 0; i < (1 << 16) && !seen; ++i) seen = ld_acquire_gpu(p.prep_seen) != 0u;
        if (!seen) atomicCAS(p.status, 0u, 0x80000000u | (97u << 20));
        *abort_flag = (*reinterpret_cast<volatile unsigned int*>(p.status) != 0u) ? 98u : 0u;  // see the main kernel
        mbar_init(qdo_full, 1);
        mbar_init(dq_full, 1);
        for (int i = 0; i < 2; ++i) {
            mbar_init(&s_full[i], 1);
            mbar_init(&ds_ready[i], kEwThreads);
        }
        mbar_init(dp_full, 1);
        mbar_init(dp_free, kEwThreads);
        mbar_init(dq_done, 1);
        for (int i = 0; i < Cfg::kKStages; ++i) {
            mbar_init(&k_full[i], 1);
            mbar_init(&k_empty[i], 1);
        }
        for (int i = 0; i < Cfg::kVStages; ++i) {
            mbar_init(&v_full[i], 1);
            mbar_init(&v_empty[i], 1);
        }
        fence_mbar_init();
    }
    if (warp == kWarpMma) {
        tmem_alloc(tmem_slot, Cfg::kTmemCols);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = *tmem_slot;
    if (*abort_flag != 0) {  // uniform: every thread reads the flag after the barrier
        if (warp == kWarpMma) tmem_dealloc(tmem, Cfg::kTmemCols);
        wait_for_main();
        return;
    }

    if (warp == kWarpTma) {
        // ======================= TMA producer =======================
        if (elect_one()) {
            tma_prefetch_desc(&mapQ);
            tma_prefetch_desc(&mapDO);
            tma_prefetch_desc(&mapK);
            tma_prefetch_desc(&mapV);
            mbar_expect_tx(qdo_full, 2 * Cfg::kTileBytes);
            for (int pn = 0; pn < Cfg::kPanels; ++pn) {
                tma_load_3d(sQ + pn * kPanel, &mapQ, qdo_full, q_x + pn * 64, q0, q_z);
                tma_load_3d(sDO + pn * kPanel, &mapDO, qdo_full, q_x + pn * 64, q0, q_z);
            }
            for (int n = 0; n < n_blk; ++n) {
                const int ks = n % Cfg::kKStages, vs = n % Cfg::kVStages;
                const uint32_t k_use = n / Cfg::kKStages, v_use = n / Cfg::kVStages;
                if (k_use > 0 && !mbar_wait(&k_empty[ks], (k_use - 1) & 1, ctx, 10)) break;
                mbar_expect_tx(&k_full[ks], Cfg::kTileBytes);
                for (int pn = 0; pn < Cfg::kPanels; ++pn)
                    tma_load_3d(sK + ks * Cfg::kTileBytes + pn * kPanel, &mapK, &k_full[ks], kv_x + pn * 64, n * kTile, kv_z);
                if (v_use > 0 && !mbar_wait(&v_empty[vs], (v_use - 1) & 1, ctx, 11)) break;
                mbar_expect_tx(&v_full[vs], Cfg::kTileBytes);
                for (int pn = 0; pn < Cfg::kPanels; ++pn)
                    tma_load_3d(sV + vs * Cfg::kTileBytes + pn * kPanel, &mapV, &v_full[vs], kv_x + pn * 64, n * kTile, kv_z);
            }
        }
    } else if (warp == kWarpMma) {
        // ======================= issuer: dP(n+1), S(n+1), dQ += dS(n) K(n) =======================
        // The whole warp runs the loop (uniform control flow); `leader` marks the one lane that issues.
        const uint32_t leader = elect_one() ? 1u : 0u;
        const uint32_t idesc_sdp = make_idesc_bf16(128, kTile, false, false);
        const uint32_t idesc_dq = make_idesc_bf16(128, n_cols, false, true);
        const uint32_t q_addr = smem_u32(sQ), do_addr = smem_u32(sDO), k_addr = smem_u32(sK), v_addr = smem_u32(sV);
        auto issue = [&](uint32_t col, uint32_t a0, uint32_t b0) {
#pragma unroll
            for (int kk = 0; kk < D / 16; ++kk) {
                if (kPadded && kk * 16 >= n_cols) break;
                const uint32_t off = (kk >> 2) * kPanel + (kk & 3) * 32;
                umma_ss_pred(leader, tmem + col, make_sdesc_sw128(a0 + off, 16, 1024), make_sdesc_sw128(b0 + off, 16, 1024),
                             idesc_sdp, kk > 0);
            }
        };
        auto issue_s = [&](int n) -> bool {
            const int st = n % Cfg::kKStages;
            // dS(n-2), in the same buffer, has been read
            if (!mbar_wait(&k_full[st], (n / Cfg::kKStages) & 1, ctx, 21) || (n >= 2 && !mbar_wait(dq_done, n & 1, ctx, 23))) return false;
            tc_fence_after_sync();
            issue(Cfg::kColS + (n & 1) * kTile, q_addr, k_addr + st * Cfg::kTileBytes);
            umma_commit_pred(leader, &s_full[n & 1]);
            return true;
        };
        auto issue_dp = [&](int n) -> bool {
            const int st = n % Cfg::kVStages;
            if (!mbar_wait(&v_full[st], (n / Cfg::kVStages) & 1, ctx, 22) || (n >= 1 && !mbar_wait(dp_free, (n - 1) & 1, ctx, 25))) return false;
            tc_fence_after_sync();
            issue(Cfg::kColDP, do_addr, v_addr + st * Cfg::kTileBytes);
            umma_commit_pred(leader, dp_full);
            umma_commit_pred(leader, &v_empty[st]);  // the value block is only read by dP
            return true;
        };
        bool ok = mbar_wait(qdo_full, 0, ctx, 20) && issue_s(0) && issue_dp(0);
        for (int n = 0; n < n_blk && ok; ++n) {
            const int st = n % Cfg::kKStages;
            if (n + 1 < n_blk) ok = n == 0 ? issue_s(1) && issue_dp(1) : issue_dp(n + 1) && issue_s(n + 1);
            if (ok) ok = mbar_wait(&ds_ready[n & 1], (n >> 1) & 1, ctx, 24);
            if (!ok) break;
            tc_fence_after_sync();
            // dS(n) (packed bf16, 16 columns at the head of each warpgroup's 32 S columns) times the key block read MN-major
            const uint32_t b0 = k_addr + st * Cfg::kTileBytes;
#pragma unroll
            for (int kk = 0; kk < kTile / 16; ++kk)
                umma_ts_pred(leader, tmem + Cfg::kColDQ, tmem + Cfg::kColS + (n & 1) * kTile + (kk >> 1) * 32 + (kk & 1) * 8,
                             make_sdesc_sw128(b0 + kk * 2048, kPanel, 1024), idesc_dq, (n > 0 || kk > 0));
            umma_commit_pred(leader, dq_done);
            umma_commit_pred(leader, &k_empty[st]);
            if (n + 1 == n_blk) umma_commit_pred(leader, dq_full);
        }
    } else {
        // ======================= elementwise warpgroups =======================
        const int w = warp >> 2;                      // which 32 keys of every block
        const int r = (warp & 3) * 32 + lane;         // query row inside the tile == TMEM lane
        const uint32_t lane_addr = (uint32_t)((warp & 3) * 32) << 16;
        const size_t row = (size_t)(b * p.Hq + hq) * p.S + q0 + r;  // in [B,Hq,S] order
        const bool row_ok = q0 + r < p.S;
        const float c = p.scale_log2;
        const float nlse2 = row_ok ? -p.lse[row] * kLog2e : 0.f;   // rows beyond S: finite garbage, never stored
        const float delta = row_ok ? p.delta[row] : 0.f;
        bool ok = true;
        for (int n = 0; n < n_blk; ++n) {
            ok = mbar_wait(&s_full[n & 1], (n >> 1) & 1, ctx, 30);
            if (ok) ok = mbar_wait(dp_full, n & 1, ctx, 32);
            if (!ok) break;
            tc_fence_after_sync();
            // last visible key column of this row inside the 128-key block: the causal diagonal and / or the end of S
            const bool diag = p.causal && (n == qt);
            const int s_left = p.S - n * kTile;
            const bool masked = diag || s_left < kTile;
            const int lim = min(diag ? r : kTile - 1, s_left - 1);
            const int col0 = w * 32;  // column of v[0] inside the block
            const uint32_t s_col = tmem + lane_addr + Cfg::kColS + (n & 1) * kTile + col0;
            uint32_t vs[32], vd[32];
            tmem_ld32(s_col, vs);
            tmem_ld32(tmem + lane_addr + Cfg::kColDP + col0, vd);
            tmem_wait_ld();
            tc_fence_before_sync();
            mbar_arrive(dp_free);
            uint32_t pk[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                float e0 = ex2_approx(fmaf(__uint_as_float(vs[2 * i]), c, nlse2));
                float e1 = ex2_approx(fmaf(__uint_as_float(vs[2 * i + 1]), c, nlse2));
                if (masked) {
                    if (col0 + 2 * i > lim) e0 = 0.f;
                    if (col0 + 2 * i + 1 > lim) e1 = 0.f;
                }
                // P rounded to bf16 first (what the dV product of the main kernel uses), then one fp32 product, one rounding
                const uint32_t pb = pack_bf16x2(e0, e1);
                const float p_lo = __uint_as_float(pb << 16), p_hi = __uint_as_float(pb & 0xffff0000u);
                pk[i] = pack_bf16x2(p_lo * (__uint_as_float(vd[2 * i]) - delta), p_hi * (__uint_as_float(vd[2 * i + 1]) - delta));
            }
            // dS of these 32 keys = 16 packed columns, stored over the head of this warpgroup's OWN S columns (which it
            // has just read), so the warpgroups never touch each other's columns: K step kk of the dQ product
            // (16 keys) finds its A operand at column 32 * (kk / 2) + 8 * (kk % 2) of the buffer
            tmem_st16(s_col, pk);
            tmem_wait_st();
            tc_fence_before_sync();
            mbar_arrive(&ds_ready[n & 1]);
        }
        // ---- epilogue: dQ = bf16(scale * sum), D / 4 columns per warpgroup
        if (ok) ok = mbar_wait(dq_full, 0, ctx, 31);
        if (ok) {
            tc_fence_after_sync();
            constexpr int kColsPerWg = D / kEwGroups;
            __nv_bfloat16* out = p.bshd ? p.dQ + ((size_t)(b * p.S + q0 + r) * p.Hq + hq) * D : p.dQ + row * p.d_real;
            uint32_t v[kColsPerWg];
            if constexpr (kColsPerWg == 32) tmem_ld32(tmem + lane_addr + Cfg::kColDQ + w * kColsPerWg, v);
            else tmem_ld16(tmem + lane_addr + Cfg::kColDQ + w * kColsPerWg, v);
            tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < kColsPerWg / 8; ++i) {
                uint4 o;
                o.x = pack_bf16x2(__uint_as_float(v[8 * i + 0]) * p.scale, __uint_as_float(v[8 * i + 1]) * p.scale);
                o.y = pack_bf16x2(__uint_as_float(v[8 * i + 2]) * p.scale, __uint_as_float(v[8 * i + 3]) * p.scale);
                o.z = pack_bf16x2(__uint_as_float(v[8 * i + 4]) * p.scale, __uint_as_float(v[8 * i + 5]) * p.scale);
                o.w = pack_bf16x2(__uint_as_float(v[8 * i + 6]) * p.scale, __uint_as_float(v[8 * i + 7]) * p.scale);
                const int col = w * kColsPerWg + i * 8;
                if (row_ok && col < p.d_real) *reinterpret_cast<uint4*>(out + col) = o;
            }
        }
    }

    // ---- teardown ---------------------------------------------------------------
    tc_fence_before_sync();
    __syncthreads();
    wait_for_main();
    if (warp == kWarpMma) {
        if (*abort_flag != 0) abort_grace_period();  // in-flight copies and MMAs land before TMEM is released
        tmem_dealloc(tmem, Cfg::kTmemCols);
    }
}

template <int D>
int launch_dq_t(const void* Q, const void* K, const void* V, const void* dO, const float* lse, const float* delta,
                void* dQ, const Shape& s, unsigned int* status, bool beside, cudaStream_t stream) {
    using Cfg = DqCfg<D>;
    CUtensorMap mq, mdo, mk, mv;
    const uint64_t S = s.S, qc = s.bshd ? (uint64_t)s.Hq * D : s.D, kc = s.bshd ? (uint64_t)s.Hkv * D : s.D;
    const uint64_t nq = s.bshd ? s.B : (uint64_t)s.B * s.Hq, nkv = s.bshd ? s.B : (uint64_t)s.B * s.Hkv;
    int rc = make_tile3_tmap(&mq, Q, qc, S, nq, S * qc, kTile);
    if (rc) return rc;
    rc = make_tile3_tmap(&mdo, dO, qc, S, nq, S * qc, kTile);
    if (rc) return rc;
    rc = make_tile3_tmap(&mk, K, kc, S, nkv, S * kc, kTile);
    if (rc) return rc;
    rc = make_tile3_tmap(&mv, V, kc, S, nkv, S * kc, kTile);
    if (rc) return rc;
    auto kernel = padded_form(s) ? gqa_bwd_dq_sm100_kernel<D, true> : gqa_bwd_dq_sm100_kernel<D, false>;
    GQA_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemTotal));
    DqParams p;
    p.dQ = static_cast<__nv_bfloat16*>(dQ);
    p.lse = lse;
    p.delta = delta;
    p.status = status;
    p.prep_seen = status + kPrepSeenWord;
    p.Hq = s.Hq;
    p.Hkv = s.Hkv;
    p.S = s.S;
    p.causal = s.causal;
    p.bshd = s.bshd;
    p.d_real = s.D;
    p.n_qtiles = (s.S + kTile - 1) / kTile;
    p.scale = s.scale;
    p.scale_log2 = s.scale * kLog2e;
    dim3 grid(p.n_qtiles, s.Hq, s.B);
    if (beside) {
        GQA_CUDA_TRY(launch_after(kernel, grid, kThreads, Cfg::kSmemTotal, stream, mq, mdo, mk, mv, p));
    } else {
        kernel<<<grid, kThreads, Cfg::kSmemTotal, stream>>>(mq, mdo, mk, mv, p);
        GQA_CUDA_TRY(cudaGetLastError());
    }
    count_launch();
    return GQA_OK;
}

}  // namespace

int launch_bwd_dq_sm100(const void* Q, const void* K, const void* V, const void* dO, const float* lse,
                        const float* delta, void* dQ, const Shape& s, unsigned int* status, bool beside,
                        cudaStream_t stream) {
    if (s.Dp() == 64) return launch_dq_t<64>(Q, K, V, dO, lse, delta, dQ, s, status, beside, stream);
    return launch_dq_t<128>(Q, K, V, dO, lse, delta, dQ, s, status, beside, stream);
}

}  // namespace gqa
