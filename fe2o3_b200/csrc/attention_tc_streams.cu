// Tensor-core attention for sm_100a, bf16 Q/K/V, f32 output, head_dim 64: causal rows, and calls with few rows.
//
// The recurrence, the precision of P and the products are those of attention_tc.cu, which takes many rows without a causal
// limit.  There a unit is two 128-row tiles that share every key block; causal units of such length come out uneven (B4 H16 S2048
// took as long with the limit as without), and a call of few rows leaves a tile of every SM idle.  Here a unit is one tile
// of 128 rows, and its key blocks go to two streams in turn, each with S, P, O, reference and sum of its own; the streams meet in
// shared memory.  us, tiles / streams: B4 H16 S2048 causal 98 / 67, B2 H12 S1900 causal 48 / 27, B1 H1 S4096 41 / 29.5, B1 H8 S1024 14.2 /
// 12; not causal, where it is not taken, B4 H16 S2048 105.6 / 110.5: a step of two blocks fetches two key blocks for one
// and comes to 3700 cycles for 3300 (attention_tc_plan holds the rule).
//
// Causal units are ordered by length, longest first, and dealt out in alternating direction.  Twelve warps: 0 = TMA
// producer, 1 = Q*K^T of both streams, 2 and 3 = P*V of a stream, 4-7 and 8-11 = softmax of the streams, a thread a row.
// The end of a unit is put off into the first block of the next, between the exponentials and P, when its last P*V is long
// done, and only the stream that is half a step behind picks the other's part up, so that neither waits.
// Bound: the exponential unit (1024 of a block's cycles a stream and SM) and the chains of the softmax warps, two a
// scheduler.  All waits are bounded.
#include "common.cuh"
#include "gemm_tc.h"


namespace {

constexpr int D = 64;            // head dimension handled by this kernel
constexpr int BQ = 128;          // query rows per unit
constexpr int BKV = 128;         // keys per block
constexpr int STREAMS = 2;       // key blocks of a unit go to them in turn
constexpr int Q_STAGES = 2;
constexpr int KV_STAGES = 4;
constexpr int kSoftmaxWarps = 4 * STREAMS;
constexpr int kRegsControl = 48, kRegsSoftmax = 224;   // registers a thread of warps 0-3 and of the softmax warps
static_assert(128 * kRegsControl + 256 * kRegsSoftmax <= 384 * 168, "the warpgroups share what the block is launched with");
constexpr int kThreads = 32 * (4 + kSoftmaxWarps);
constexpr float kRescaleThreshold = 8.0f;  // log2 units
constexpr float kTruncGain = 1.001953125f;           // 1 + 2^-9: half a bf16 ulp, relative
constexpr float kTruncBiasLog2 = 0.0028150157f;      // log2(kTruncGain)

constexpr uint32_t kTileBytes = 128 * D * 2;     // 16 KiB: a 128 x 64 bf16 tile
constexpr uint32_t kOffQ = 0;
constexpr uint32_t kOffK = kOffQ + Q_STAGES * kTileBytes;
constexpr uint32_t kOffV = kOffK + KV_STAGES * kTileBytes;
constexpr uint32_t kOffMerge = kOffV + KV_STAGES * kTileBytes;       // a unit's output: [4 warps][2 x 32 columns][32 rows][128 bytes]
constexpr uint32_t kOffRow = kOffMerge + BQ * D * 4;                   // reference and sum of each row in stream 0
constexpr uint32_t kOffBar = kOffRow + 2 * BQ * 4;
constexpr uint32_t kSmemTotal = kOffBar + 512 + 1024;   // + alignment slack

// TMEM columns: S of stream t at t*128 (128 f32 columns), O at 256 + t*64 (64 f32 columns),
// P at 384 + t*64 (128 bf16 per row = 64 columns).
constexpr uint32_t kTmemCols = 512;
constexpr uint32_t kColO = 256, kColP = 384;

struct AttnParams {
    float *out;
    uint32_t bh, seq;
    float scale_log2;   // scale * log2(e)
    uint32_t causal;
    uint32_t q_blocks;  // 128-row blocks per head
    uint32_t units;     // work units: heads * q_blocks
    uint32_t *status;
};

struct Unit {
    uint32_t head, q0, n;   // n: key blocks
};

// The i-th unit of this CTA; false when the CTA has no i-th unit.  Every role walks the same sequence.  Causal units
// are ordered by length, longest first, and dealt out in alternating direction.
__device__ __forceinline__ bool unit_at(const AttnParams &p, uint32_t i, Unit &u) {
    const uint32_t idx = i * gridDim.x + ((i & 1) ? gridDim.x - 1 - blockIdx.x : blockIdx.x);
    if (idx >= p.units) return false;
    const uint32_t qb = p.causal ? p.q_blocks - 1 - idx / p.bh : idx % p.q_blocks;
    u.head = p.causal ? idx % p.bh : idx / p.q_blocks;
    u.q0 = qb * BQ;
    u.n = ((p.causal ? min(p.seq, u.q0 + BQ) : p.seq) + BKV - 1) / BKV;
    return true;
}

// Waits on another role of the block.  Few instructions: the roles' loops share the instruction caches with the softmax
// warps' long ones.
__device__ __forceinline__ bool wait(uint64_t *bar, uint32_t parity) {
    uint32_t polls = 0;
    while (!__all_sync(0xffffffffu, mbar_try_wait(bar, parity)))
        if (++polls >= FE2O3_SPIN_LIMIT) return false;
    return true;
}

__global__ void __launch_bounds__(kThreads, 1)
attention_streams_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                    const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmO, AttnParams p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + kOffBar);
    uint64_t *q_full = bars;                       // Q_STAGES
    uint64_t *q_empty = q_full + Q_STAGES;
    uint64_t *k_full = q_empty + Q_STAGES;         // KV_STAGES
    uint64_t *k_empty = k_full + KV_STAGES;
    uint64_t *v_full = k_empty + KV_STAGES;
    uint64_t *v_empty = v_full + KV_STAGES;
    uint64_t *s_full = v_empty + KV_STAGES;        // STREAMS
    uint64_t *s_empty = s_full + STREAMS;
    uint64_t *p_ready = s_empty + STREAMS;
    uint64_t *pv_done = p_ready + STREAMS;
    uint64_t *merge_full = pv_done + STREAMS;
    uint64_t *merge_empty = merge_full + 1;
    uint64_t *stagger = merge_empty + 1;           // 1: stream 0 finished its first exponential phase
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(stagger + 1);

    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        for (int i = 0; i < Q_STAGES; ++i) {
            mbar_init(&q_full[i], 1);
            mbar_init(&q_empty[i], 1);
        }
        for (int i = 0; i < KV_STAGES; ++i) {
            mbar_init(&k_full[i], 1);
            mbar_init(&k_empty[i], 1);
            mbar_init(&v_full[i], 1);
            mbar_init(&v_empty[i], 1);
        }
        for (int t = 0; t < STREAMS; ++t) {
            mbar_init(&s_full[t], 1);
            mbar_init(&s_empty[t], 4);
            mbar_init(&p_ready[t], 4);
            mbar_init(&pv_done[t], 1);
        }
        mbar_init(merge_full, 4);
        mbar_init(merge_empty, 4);
        mbar_init(stagger, 4);
        mbar_fence_init();
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, kTmemCols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    begin_after_previous();   // launched early: everything above ran beside the kernel before
    // Each branch below opens with its own register re-balance, so that the code of a role is compiled
    // against that role's register count (a re-balance ahead of the branches would hold every role to
    // the smaller count).
    if (warp < 4) {
    regs_release<kRegsControl>();
    if (warp == 0) {
        // ---------------------------------------------------------- TMA producer
        // The whole warp runs the loop converged; one elected lane issues the copies.
        if (elect_one()) {
            tma_prefetch_desc(&tmQ);
            tma_prefetch_desc(&tmK);
            tma_prefetch_desc(&tmV);
            tma_prefetch_desc(&tmO);
        }
        __syncwarp();
        bool ok = true;
        uint32_t g = 0;          // K/V blocks loaded so far, over all units
        uint32_t n_units = 0;
        Unit u;
        for (uint32_t i = 0; ok && unit_at(p, i, u); ++i) {
            const uint32_t qs = n_units % Q_STAGES, qph = (n_units / Q_STAGES) & 1;
            ++n_units;
            if (!wait(&q_empty[qs], qph ^ 1)) { ok = false; break; }
            if (elect_one()) {
                mbar_arrive_expect_tx(&q_full[qs], kTileBytes);
                tma_load_3d(smem + kOffQ + qs * kTileBytes, &tmQ, &q_full[qs], 0, (int32_t)u.q0, (int32_t)u.head);
            }
            __syncwarp();
            for (uint32_t j = 0; j < u.n; ++j, ++g) {
                const uint32_t st = g % KV_STAGES, ph = (g / KV_STAGES) & 1;
                if (!wait(&k_empty[st], ph ^ 1)) { ok = false; break; }
                if (elect_one()) {
                    mbar_arrive_expect_tx(&k_full[st], kTileBytes);
                    tma_load_3d(smem + kOffK + st * kTileBytes, &tmK, &k_full[st], 0, (int32_t)(j * BKV), (int32_t)u.head);
                }
                __syncwarp();
                if (!wait(&v_empty[st], ph ^ 1)) {
                    ok = false;
                    mbar_wait_warp(&k_full[st], ph);   // the K copy just issued must land before the CTA exits
                    break;
                }
                if (elect_one()) {
                    mbar_arrive_expect_tx(&v_full[st], kTileBytes);
                    tma_load_3d(smem + kOffV + st * kTileBytes, &tmV, &v_full[st], 0, (int32_t)(j * BKV), (int32_t)u.head);
                }
                __syncwarp();
            }
        }
        if (!ok && lane == 0) kstatus_set(p.status, FE2O3_KSTATUS_WAIT_EXPIRED);
        // drain the copies before the CTA can exit: the newest phase of every ring slot in use
        for (uint32_t b = 0; b < KV_STAGES && b < g; ++b) {
            const uint32_t last = g - 1 - b, st = last % KV_STAGES, ph = (last / KV_STAGES) & 1;
            mbar_wait_warp(&k_full[st], ph);
            mbar_wait_warp(&v_full[st], ph);
        }
        for (uint32_t b = 0; b < Q_STAGES && b < n_units; ++b) {
            const uint32_t last = n_units - 1 - b;
            mbar_wait_warp(&q_full[last % Q_STAGES], (last / Q_STAGES) & 1);
        }
    } else if (warp == 1) {
        // ---------------------------------------------------------- Q*K^T of both streams, in the order of the key blocks
        // (S of a stream is free as soon as its softmax has read the block before)
        constexpr uint32_t idesc_qk = umma_idesc(1u, BQ, BKV, 0u, 0u);
        const uint64_t dQ = umma_smem_desc(smem_u32(smem + kOffQ), 16, 1024), dK = umma_smem_desc(smem_u32(smem + kOffK), 16, 1024);
        bool ok = true;
        uint32_t st = 0, ph = 0;   // ring position
        uint32_t given = 0;        // a bit a stream: parity of its blocks so far
        uint32_t n = 0;            // units so far
        Unit u;
        for (uint32_t i = 0; ok && unit_at(p, i, u); ++i, ++n) {
            const uint32_t qs = n % Q_STAGES;
            if (!wait(&q_full[qs], (n / Q_STAGES) & 1)) { ok = false; break; }
            for (uint32_t j = 0; j < u.n; ++j) {
                const uint32_t t = j % STREAMS;
                if (!wait(&k_full[st], ph) || !wait(&s_empty[t], (given >> t & 1) ^ 1)) { ok = false; break; }
                tc_fence_after();
                if (elect_one()) {
                    const uint64_t q = dQ + ((qs * kTileBytes) >> 4), k = dK + ((st * kTileBytes) >> 4);
#pragma unroll 1
                    for (uint32_t kk = 0; kk < D / 16; ++kk) umma_f16(tmem_base + t * BKV, q + kk * 2, k + kk * 2, idesc_qk, kk != 0);
                    umma_commit(&s_full[t]);
                    umma_commit(&k_empty[st]);
                    if (j + 1 == u.n) umma_commit(&q_empty[qs]);
                }
                __syncwarp();
                given ^= 1u << t;
                if (++st == KV_STAGES) { st = 0; ph ^= 1; }
            }
        }
        if (!ok && lane == 0) kstatus_set(p.status, FE2O3_KSTATUS_WAIT_EXPIRED);
    } else if (warp < 4) {
        // ---------------------------------------------------------- P*V, one warp per stream
        constexpr uint32_t idesc_pv = umma_idesc(1u, BQ, D, 0u, 1u);
        const uint32_t t = warp - 2;
        const uint64_t dV = umma_smem_desc(smem_u32(smem + kOffV), 8192, 1024);
        const uint32_t tO = tmem_base + kColO + t * D, tP = tmem_base + kColP + t * (BKV / 2);
        bool ok = true;
        uint32_t g0 = 0;   // key blocks of the units before: ring position of V
        uint32_t gt = 0;   // blocks of this stream: parity of p_ready / pv_done
        Unit u;
        for (uint32_t i = 0; ok && unit_at(p, i, u); ++i) {
            for (uint32_t j = t; j < u.n; j += STREAMS, ++gt) {
                const uint32_t g = g0 + j, st = g % KV_STAGES;
                if (!wait(&v_full[st], (g / KV_STAGES) & 1) || !wait(&p_ready[t], gt & 1)) { ok = false; break; }
                tc_fence_after();
                if (elect_one()) {
                    const uint64_t v = dV + ((st * kTileBytes) >> 4);
#pragma unroll 1
                    for (uint32_t kk = 0; kk < BKV / 16; ++kk) umma_f16_ts(tO, tP + kk * 8, v + kk * 128, idesc_pv, kk != 0 || j >= STREAMS);
                    umma_commit(&pv_done[t]);
                    umma_commit(&v_empty[st]);
                }
                __syncwarp();
            }
            g0 += u.n;
        }
        if (!ok && lane == 0) kstatus_set(p.status, FE2O3_KSTATUS_WAIT_EXPIRED);
    }
    } else {
        regs_take<kRegsSoftmax>();
        // ---------------------------------------------------------- softmax warps
        constexpr int NCH = BKV / 32;                       // 32-column chunks of the score row
        const uint32_t sw = warp - 4;                       // 0 .. kSoftmaxWarps-1
        const uint32_t t = sw / 4;                          // stream of this warp
        const uint32_t quad = warp & 3;                     // TMEM lane quadrant this warp may access
        const uint32_t r = quad * 32 + lane;                // row inside the unit
        const uint32_t lane_addr = (quad * 32u) << 16;
        const uint32_t tS = tmem_base + t * BKV + lane_addr;
        const uint32_t tO = tmem_base + kColO + t * D + lane_addr;
        const uint32_t tP = tmem_base + kColP + t * (BKV / 2) + lane_addr;
        const float c = p.scale_log2;
        bool ok = true;
        uint32_t gt = 0;             // key blocks this stream has processed, over all units
        uint32_t n = 0;              // units so far
        // This warp's 32 rows of the output, a 4 KiB piece of 32 columns after the other, swizzled as the copy engine stores them.
        // Stream 0 leaves its part there, stream 1 adds its own and stores the rows.
        uint8_t *const rows_out = smem + kOffMerge + quad * 8192;
        auto piece = [&](int h, int q) { return reinterpret_cast<float4 *>(rows_out + h * 4096 + lane * 128 + ((q ^ (lane & 7)) * 16)); };
        bool storing = false;        // the copy engine may still be reading rows_out
        auto release_rows = [&]() {
            if (lane == 0) tma_store_wait_read();
            __syncwarp();
            if (lane == 0) mbar_arrive(merge_empty);
            storing = false;
        };
        // The end of a unit.  It takes place in the first block of the next one, between the exponentials and P, when the last
        // P*V is long done.  The stream that is half a step ahead leaves its part, the other one picks it up: neither waits
        // for the other, and they stay half a step apart.  (Each finishing half of the columns brought them into step after
        // every unit, and their exponentials on top of one another: 3700 cycles a step for 2950.)
        Unit before{0u, 0u, 0u};
        float m_before = 0.0f, l_before = 0.0f;
        auto finish_unit = [&]() {
            const bool any = t < before.n;   // (a unit of one block has none for stream 1)
            if (any) {
                if (!wait(&pv_done[t], (gt - 1) & 1)) return false;
                tc_fence_after();
            }
            float *const ref = reinterpret_cast<float *>(smem + kOffRow) + r;
            if (t == 0) {
                if (!wait(merge_empty, (n & 1) ^ 1)) return false;
#pragma unroll 1
                for (int h = 0; h < 2; ++h) {
                    uint32_t o[32];
                    tmem_ld_32x32b_x32(tO + h * 32, o);
                    tmem_ld_wait();
#pragma unroll
                    for (int q = 0; q < 8; ++q) *reinterpret_cast<uint4 *>(piece(h, q)) = make_uint4(o[4 * q], o[4 * q + 1], o[4 * q + 2], o[4 * q + 3]);
                }
                ref[0] = m_before;
                ref[BQ] = l_before;
                // the next unit's first P*V overwrites O: order this thread's reads of O before its p_ready arrival
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(merge_full);
                ++n;
                return true;
            }
            if (storing) {   // (the units are so short that the rows before last are still held)
                release_rows();
            }
            if (!wait(merge_full, n & 1)) return false;
            ++n;
            const float m0 = ref[0], m = fmaxf(m_before, m0), mb = m == -INFINITY ? 0.0f : m;
            const float f0 = ex2_approx((m0 - mb) * c), f1 = ex2_approx((m_before - mb) * c);
            const float l_row = ref[BQ] * f0 + l_before * f1;
            const float inv = kTruncGain / l_row;   // the sums carry the gain of the truncation bias
            const float g0 = f0 * inv, g1 = any ? f1 * inv : 0.0f;
            const uint32_t row0 = before.q0 + quad * 32;   // first query row of this warp
            float check = 0.0f;                            // 0, or NaN once a value was not finite
#pragma unroll 1
            for (int h = 0; h < 2; ++h) {
                uint32_t o[32];
                tmem_ld_32x32b_x32(tO + h * 32, o);
                tmem_ld_wait();
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const float4 v = *piece(h, q);
                    float4 w;
                    w.x = fmaf(any ? __uint_as_float(o[4 * q]) : 0.0f, g1, v.x * g0);
                    w.y = fmaf(any ? __uint_as_float(o[4 * q + 1]) : 0.0f, g1, v.y * g0);
                    w.z = fmaf(any ? __uint_as_float(o[4 * q + 2]) : 0.0f, g1, v.z * g0);
                    w.w = fmaf(any ? __uint_as_float(o[4 * q + 3]) : 0.0f, g1, v.w * g0);
                    check = fmaf(w.x, 0.0f, check);
                    check = fmaf(w.y, 0.0f, check);
                    check = fmaf(w.z, 0.0f, check);
                    check = fmaf(w.w, 0.0f, check);
                    *piece(h, q) = w;
                }
            }
            tc_fence_before();
            // full-line writes by the copy engine that do not hold the warp; rows beyond seq are clipped
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
                if (row0 < p.seq)
                    for (int h = 0; h < 2; ++h) tma_store_3d(&tmO, rows_out + h * 4096, h * 32, (int32_t)row0, (int32_t)before.head);
                tma_store_commit();
            }
            storing = true;
            // finite-input policy: a non-finite result is reported through the status word
            if (!(isfinite(l_row) && l_row > 0.0f && check == 0.0f) && before.q0 + r < p.seq) kstatus_set(p.status, FE2O3_KSTATUS_NONFINITE);
            __syncwarp();
            return true;
        };
        Unit u;
        for (uint32_t ui = 0; ok; ++ui) {
            const bool have = unit_at(p, ui, u);
            if (!have) {
                u.n = 0;
                if (ui == 0) break;
            }
            const uint32_t qrow = u.q0 + r;   // query index inside the head
            float m_ref = -INFINITY;   // exponent offset, in raw score units
            float l = 0.0f;            // this stream's share of the denominator
            bool s_early = false;      // s_full of the coming block was seen complete by the early probe

            for (uint32_t j = t;; j += STREAMS) {
                const bool block = j < u.n;   // (the first time round there may be none)
                if (!block && j != t) break;
                uint32_t pk[NCH][16];
                float sum[4] = {0.0f, 0.0f, 0.0f, 0.0f}, factor = 1.0f;
                bool move = false, pv_early = false;
                if (block) {
                // A probe of a barrier takes about 200 cycles even when the phase is complete, so the two
                // waits of a step are probed ahead of the long phases (S of the next block before the P
                // store of this one, P*V of the previous block before the exponentials) and only fall
                // back to the bounded wait when the early answer was "not yet".
                if (!__all_sync(0xffffffffu, s_early) && !wait(&s_full[t], gt & 1)) { ok = false; break; }
                s_early = false;
                tc_fence_after();
                // this thread's part of the score row into registers, then S is free for the next Q*K^T
                uint32_t s[NCH][32];
#pragma unroll
                for (int ch = 0; ch < NCH; ++ch) tmem_ld_32x32b_x32(tS + ch * 32, s[ch]);
                tmem_ld_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&s_empty[t]);

                const uint32_t key0 = j * BKV;
                const bool need_mask = (j * BKV + BKV > p.seq) || (p.causal && j * BKV + BKV - 1 > u.q0);
                if (need_mask) {
                    const uint32_t end = p.causal ? min(p.seq, qrow + 1) : p.seq, limit = end > key0 ? end - key0 : 0u;
#pragma unroll
                    for (int ch = 0; ch < NCH; ++ch) {
#pragma unroll
                        for (int i = 0; i < 32; ++i)
                            if (ch * 32 + i >= limit) s[ch][i] = 0xff800000u;  // -inf
                    }
                }
                float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
                for (int ch = 0; ch < NCH; ++ch) {
#pragma unroll
                    for (int i = 0; i < 32; i += 8) {
#pragma unroll
                        for (int q = 0; q < 4; ++q)
                            mx[q] = max3(mx[q], __uint_as_float(s[ch][i + 2 * q]), __uint_as_float(s[ch][i + 2 * q + 1]));
                    }
                }
                const float rowmax = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
                // move the reference only when the block maximum outgrows it by more than the threshold
                move = (rowmax - m_ref) * c > kRescaleThreshold;  // true for the first admitted key (m_ref = -inf)
                factor = move ? ex2_approx((m_ref - rowmax) * c) : 1.0f;  // 0 when m_ref = -inf
                if (move) m_ref = rowmax;
                // p = 2^(s*c - m_ref*c); a row with no admitted key so far keeps m_ref = -inf: use offset 0, p = 0
                const float mc = (m_ref == -INFINITY ? 0.0f : m_ref) * c;
                // The two streams share the exponential unit: stream 1 starts its first exponential phase when
                // stream 0 has finished its own, so that afterwards one stream's exponentials overlap the
                // other's loads, maxima and stores.
                if (gt == 0 && t == 1 && !wait(stagger, 0)) { ok = false; break; }
                // Exponentials stay in registers as packed bf16 pairs until the P buffer is free.  The scale
                // and the sums run as packed pairs of f32.  P is cut to bf16 by truncation, which one byte
                // permute does for two values; the exponent carries a bias of log2(1 + 2^-9) so that the
                // truncation error is centred on zero like a rounding error, and the bias (also present in
                // the sums) is divided out with the denominator at the end.
                pv_early = j >= STREAMS && mbar_test(&pv_done[t], (gt - 1) & 1);
                const float mcb = mc - kTruncBiasLog2;
                const uint64_t c2 = pack_f32x2(c, c), nmc2 = pack_f32x2(-mcb, -mcb);
                uint64_t sum2[4] = {0ull, 0ull, 0ull, 0ull};   // four pairs of +0.0f
#pragma unroll
                for (int ch = 0; ch < NCH; ++ch) {
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        float e[8];
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const uint64_t x2 = fma_f32x2(
                                pack_f32x2(__uint_as_float(s[ch][q * 8 + 2 * i]), __uint_as_float(s[ch][q * 8 + 2 * i + 1])), c2, nmc2);
                            float x0, x1;
                            unpack_f32x2(x2, x0, x1);
                            e[2 * i] = ex2_approx(x0);
                            e[2 * i + 1] = ex2_approx(x1);
                        }
#pragma unroll
                        for (int i = 0; i < 4; ++i) sum2[i] = add_f32x2(sum2[i], pack_f32x2(e[2 * i], e[2 * i + 1]));
#pragma unroll
                        for (int i = 0; i < 4; ++i)
                            pk[ch][q * 4 + i] = __byte_perm(__float_as_uint(e[2 * i]), __float_as_uint(e[2 * i + 1]), 0x7632);
                    }
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    float lo, hi;
                    unpack_f32x2(sum2[i], lo, hi);
                    sum[i] = lo + hi;
                }
                if (gt == 0 && t == 0) {
                    __syncwarp();
                    if (lane == 0) mbar_arrive(stagger);
                }
                }
                // P of the previous block must have been consumed and O must be quiescent
                if (j == t) {
                    if (ui != 0 && !finish_unit()) { ok = false; break; }
                    if (!block) break;
                } else {
                    if (!__all_sync(0xffffffffu, pv_early) && !wait(&pv_done[t], (gt - 1) & 1)) { ok = false; break; }
                    tc_fence_after();
                    if (__any_sync(0xffffffffu, move)) {   // each thread rescales its own output columns
#pragma unroll 1
                        for (int g = 0; g < D / 8; ++g) {
                            uint32_t ov[8];
                            tmem_ld_32x32b_x8(tO + g * 8, ov);
                            tmem_ld_wait();
#pragma unroll
                            for (int i = 0; i < 8; ++i) ov[i] = __float_as_uint(__uint_as_float(ov[i]) * factor);
                            tmem_st_32x32b_x8(tO + g * 8, ov);
                        }
                    }
                }
                l = fmaf(l, factor, (sum[0] + sum[1]) + (sum[2] + sum[3]));
                if (j + STREAMS < u.n) s_early = mbar_test(&s_full[t], (gt + 1) & 1);
                // P as packed bf16 pairs into tensor memory: 16 columns per 32 keys
#pragma unroll
                for (int ch = 0; ch < NCH; ++ch) tmem_st_32x32b_x16(tP + ch * 16, pk[ch]);
                tmem_st_wait();
                // publish P and any O rescale (both TMEM stores) to the MMA issuer
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&p_ready[t]);
                if (storing && j != t) release_rows();   // the unit before's: by now they have been read
                ++gt;
            }
            if (!ok || !have) break;
            before = u;
            m_before = m_ref;
            l_before = l;
        }
        if (storing && lane == 0) tma_store_wait_read();   // the rows must stay until the copies have read them
        if (!ok && lane == 0) kstatus_set(p.status, FE2O3_KSTATUS_WAIT_EXPIRED);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, kTmemCols);
    }
}

}  // namespace

// The maps are those of attention_tc_plan.
int32_t attention_streams_init_device() {
    FE2O3_CUDA(cudaFuncSetAttribute(attention_streams_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemTotal));
    return FE2O3_OK;
}

cudaError_t attention_streams_launch(cudaStream_t s, uint32_t grid, const CUtensorMap &tmQ, const CUtensorMap &tmK, const CUtensorMap &tmV,
                                     const CUtensorMap &tmO, float *out, uint32_t bh, uint32_t seq, float scale_log2, uint32_t causal,
                                     uint32_t *status) {
    const uint32_t q_blocks = (seq + BQ - 1) / BQ;
    const AttnParams p{out, bh, seq, scale_log2, causal, q_blocks, bh * q_blocks, status};
    return fe2o3_launch_early(attention_streams_kernel, grid, kThreads, kSmemTotal, s, 1, tmQ, tmK, tmV, tmO, p);
}

uint32_t attention_streams_smem() { return kSmemTotal; }
