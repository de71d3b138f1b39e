// Tensor-core attention for sm_100a with probabilities kept at f32 precision:
// bf16 Q/K/V, f32 output, head sizes up to 128 that are multiples of 8 (size 64
// has a kernel of its own, attention_tc.cu, which carries bf16 probabilities).
//
// The recurrence is the reference's (examples/flash_attention_v1/src/kernel.rs:56-113)
// per block of 64 keys: S = Q*K^T and O += P*V on tcgen05 with S and O in tensor
// memory.  These head sizes used to run on the CUDA-core kernel alone, whose
// probabilities are f32; a bf16 P would lose 16 of their 24 bits.  So P is cut by
// truncation into three bf16 terms, hi + mid + lo, which hold the 24 bits exactly
// (each term takes the top eight significant bits of what is left), and P*V is three
// products accumulated into the same O: every product is exact, only the f32
// accumulation rounds.
//   That accumulation truncates, twelve times a block and always towards zero, which
// over a whole row is up to ten times the error of the CUDA-core kernel (4096 keys of
// head size 128: 1.4e-5 against 1.5e-6 of the result, 2-norm, against f64).  So a sum
// in tensor memory covers a group of one, two or four blocks (starts_group: short rows
// have the least error to hide it behind) and the groups are added in registers, where
// additions round to nearest: 7.5e-7 at 4096 keys, and not above the CUDA cores from 333
// to 4096 keys; at 50, one block, either may be the nearer by a fifth.  The price is a read of O per group between one
// P*V and the next, and the registers of a row of O: beyond 64 columns half of the scores is fetched twice, and the
// probabilities wait as f32 in the scores' registers and are cut after the wait for the previous P*V (before it, 96
// words do not fit beside the row).
//
// Structure: persistent CTAs, one per SM, over units of 128 query rows.  The key blocks of a unit go to two streams in
// turn, each with S, P, O, reference and sum of its own, so that one stream's exponentials overlap the other's products;
// the streams meet in shared memory at the end of the unit, where each finishes half of the columns.  Two 128-row tiles
// that shared their key blocks (until then) made units twice as long for the same work a block: B2 H12 S1900 D128 causal
// came to 30 steps on the longest SM of 23 on average, 20 of 19.5 so, and a call with few rows leaves no stream idle.
//   Warp 0 loads (TMA), warp 1 issues Q*K^T of both streams, warps 2 and 3 P*V of a stream each, warps 4-7 and
// 8-11 are the softmax warps of the streams, one thread per row, with most of the registers.  With one issuer a
// tile, Q*K^T of a block waited behind P*V of the block before and that for its softmax: 3500 of a block's 3800 cycles
// were the issuer's.  Its loops are rolled and its waits short because code is what they cost: eight warps run through
// some 900 instructions a block, and what runs once in between is fetched anew each time (some 6 cycles an instruction).
//   What bounds it: of some 3700 cycles for a block of each stream the softmax warps, two a scheduler, work 2800 (a look for
// the maximum, 64 exponentials, the cut: 18 cycles of the ALU, 16 of the exponential unit and 8 of the f32 pipe a pair of keys
// and warp), the tensor pipe 2300.  Tried: four warps a tile of 16 rows each (20 instructions a score for 14: no faster), the
// cut in a rolled loop that fetches scores as it goes (5400), exponentials of half a block ahead of its maximum (4400).
//   A reference is a whole number of log2 units, so rescaling and the meeting of the streams are exact.
//   64-key blocks and P's lo term in shared memory instead of tensor memory are what fits two streams at head size 128:
//   S 2 x 64, O 2 x 128 and hi, mid 2 x 2 x 32 make the 512 columns.  So S has columns of its own and the next Q*K^T overlaps
//   the exponentials.
//   Causal units are ordered by length, longest first, and dealt out in alternating
//   direction (round 0 forwards, round 1 backwards).
//   Head sizes below 64 or between 64 and 128 are zero-filled by the copy engine on the
//   way in and clipped on the way out; Q*K^T takes only the k steps in use.
//   A row that met a non-finite score or value is settled one by one: the tensor core
//   also multiplies the values of keys that a causal row does not admit, by probabilities
//   of 0, and 0 x Inf is NaN.  The first key of the head with a non-finite K or V is
//   searched once; a row that admits it is left unwritten and reported, the others are
//   computed by the CUDA-core recurrence (attention_row.cuh).
//   The other warps may wait long meanwhile, so waits that run out start over as long as
//   rows are being settled (Waits).
// Two tiles a unit / so, us, the same inputs again and again: B2 H12 S1900 D128 causal 79.8 / 56.0 (with others each time
// 83.7 / 63.2), not causal 156 / 97; B1 H1 S4096 D128 111 / 63; B8 H8 S256 D128 15.7 / 11.3; B4 H16 S2048 D32 262 / 223.  On the CUDA
// cores the first takes 8017.
// The rule in front (attention_split_supported) is what the copy engine can address:
// rows of whole 16 bytes and 16-byte aligned bases; the rest, f32 inputs and head sizes
// above 128 stay on the CUDA cores.  All waits are bounded.
#include "attention_row.cuh"
#include "gemm_tc.h"

#include <new>

namespace {

constexpr int BQ = 128;          // query rows per unit
constexpr int BKV = 64;          // keys per block
constexpr int STREAMS = 2;       // key blocks of a unit go to them in turn
constexpr int KV_STAGES = 3;
constexpr int kThreads = 32 * (4 + 4 * STREAMS);
constexpr int kRegsControl = 40, kRegsSoftmax = 232;
static_assert(128 * kRegsControl + STREAMS * 128 * kRegsSoftmax <= kThreads * 168, "the warpgroups share what the block is launched with");
constexpr float kRescaleThreshold = 8.0f;              // log2 units

// NG: groups of 64 head columns (128 bytes) per row
template <int NG>
struct Layout {
    static constexpr uint32_t kQTile = NG * BQ * 128;      // [group][128 rows][128 bytes]
    static constexpr uint32_t kKvTile = NG * BKV * 128;    // [group][64 keys][128 bytes]
    static constexpr uint32_t kPTile = BQ * 128;           // lo term: [128 rows][64 keys]
    static constexpr uint32_t kOffK = kQTile;
    static constexpr uint32_t kOffV = kOffK + KV_STAGES * kKvTile;
    static constexpr uint32_t kOffP = kOffV + KV_STAGES * kKvTile;
    static constexpr uint32_t kOffMerge = kOffP + STREAMS * kPTile;        // a unit's output: [stream][4 warps][NG x 32 columns][32 rows][128 bytes]
    static constexpr uint32_t kOffRow = kOffMerge + NG * 64 * BQ * 4;      // reference and sum of each row, a stream
    static constexpr uint32_t kOffBar = kOffRow + STREAMS * 2 * BQ * 4;
    static constexpr uint32_t kTotal = kOffBar + 256;
    static_assert(kTotal <= 227 * 1024, "shared memory of a block");
};

// TMEM columns: S of stream t at t*64, O at 128 + t*128, P at 384 + t*64 (hi 32, mid 32)
constexpr uint32_t kTmemCols = 512, kColO = 128, kColP = 384;

struct SplitParams {
    const uint16_t *q, *k, *v;   // for rows that are settled one by one
    float *out;
    uint32_t bh, seq, dim;
    float scale, scale_log2;   // scale_log2 = scale * log2(e)
    uint32_t causal;
    uint32_t q_blocks;  // 128-row blocks per head
    uint32_t units;     // work units: heads * q_blocks
    float whole;        // 1: references are whole numbers; 0: the maxima themselves (rows of one block, never rescaled)
    uint32_t *status;
};

struct Unit {
    uint32_t head, q0, n;   // n: key blocks
};

// The i-th unit of this CTA; false when there is none.  Every role walks the same sequence.
__device__ __forceinline__ bool unit_at(const SplitParams &p, uint32_t i, Unit &u) {
    const uint32_t idx = i * gridDim.x + ((i & 1) ? gridDim.x - 1 - blockIdx.x : blockIdx.x);
    if (idx >= p.units) return false;
    const uint32_t qb = p.causal ? p.q_blocks - 1 - idx / p.bh : idx % p.q_blocks;
    u.head = p.causal ? idx % p.bh : idx / p.q_blocks;
    u.q0 = qb * BQ;
    u.n = ((p.causal ? min(p.seq, u.q0 + BQ) : p.seq) + BKV - 1) / BKV;
    return true;
}

// Key blocks whose P*V starts a new sum in tensor memory; the sum before is added to the row's registers.
__device__ __forceinline__ bool starts_group(uint32_t j) { return (j & (j < 2 ? 0u : j < 8 ? 1u : 3u)) == 0; }

__device__ __forceinline__ uint64_t sub_f32x2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

// Cuts a pair of f32 to bf16 by truncation; `rest` is what that leaves (exact).
__device__ __forceinline__ uint32_t cut_bf16x2(uint64_t v, uint64_t &rest) {
    float lo, hi;
    unpack_f32x2(v, lo, hi);
    const uint32_t l = __float_as_uint(lo), h = __float_as_uint(hi);
    rest = sub_f32x2(v, pack_f32x2(__uint_as_float(l & 0xffff0000u), __uint_as_float(h & 0xffff0000u)));
    return __byte_perm(l, h, 0x7632);
}

// Waits on another role of the block.  `settled` moves on as long as rows are being settled one by one.  Few instructions:
// the roles' loops share the instruction caches with the softmax warps' long ones.
struct Waits {
    const volatile uint32_t *settled;
    __device__ __forceinline__ bool operator()(uint64_t *bar, uint32_t parity) const {
        uint32_t polls = 0, seen = 0;
        while (!__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) {
            if (++polls < FE2O3_SPIN_LIMIT) continue;
            const uint32_t now = __shfl_sync(0xffffffffu, *settled, 0);
            if (now == seen) return false;
            seen = now;
            polls = 0;
        }
        return true;
    }
};

// The first of a head's first `keys` keys whose K or V row holds a non-finite value, or `keys`: no row that admits it has
// a result.  Rows are whole 16-byte pieces.
template <typename Tick>
__device__ __forceinline__ uint32_t first_nonfinite_key(const uint16_t *k, const uint16_t *v, uint32_t keys, uint32_t dim, uint32_t lane, Tick tick) {
    constexpr int kAhead = 4;
    const uint32_t pieces = dim / 8;
    const uint64_t end = (uint64_t)keys * pieces;
    auto holds = [](uint4 w) {
        auto one = [](uint32_t x) { return (x & 0x7f80u) == 0x7f80u || (x & 0x7f800000u) == 0x7f800000u; };
        return one(w.x) || one(w.y) || one(w.z) || one(w.w);
    };
    for (uint64_t i0 = 0; i0 < end; i0 += 32 * kAhead) {
        tick(0u);
        uint4 w[kAhead][2];
#pragma unroll
        for (int a = 0; a < kAhead; ++a) {
            const uint64_t i = i0 + a * 32 + lane;
            w[a][0] = w[a][1] = make_uint4(0u, 0u, 0u, 0u);
            if (i < end) {
                w[a][0] = __ldg(reinterpret_cast<const uint4 *>(k) + i);
                w[a][1] = __ldg(reinterpret_cast<const uint4 *>(v) + i);
            }
        }
        uint32_t first = keys;
#pragma unroll
        for (int a = kAhead - 1; a >= 0; --a)
            if (holds(w[a][0]) || holds(w[a][1])) first = (uint32_t)((i0 + a * 32 + lane) / pieces);
        first = __reduce_min_sync(0xffffffffu, first);
        if (first < keys) return first;
    }
    return keys;
}

template <int NG>
__global__ void __launch_bounds__(kThreads, 1)
attention_split_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                       const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmO, SplitParams p) {
    using L = Layout<NG>;
    extern __shared__ __align__(1024) uint8_t smem[];   // (swizzle atoms are 1 KiB; there is no room to round up)
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + L::kOffBar);
    uint64_t *q_full = bars;
    uint64_t *q_empty = q_full + 1;
    uint64_t *k_full = q_empty + 1;                // KV_STAGES each
    uint64_t *k_empty = k_full + KV_STAGES;
    uint64_t *v_full = k_empty + KV_STAGES;
    uint64_t *v_empty = v_full + KV_STAGES;
    uint64_t *s_full = v_empty + KV_STAGES;        // STREAMS each
    uint64_t *s_empty = s_full + STREAMS;
    uint64_t *p_ready = s_empty + STREAMS;
    uint64_t *pv_done = p_ready + STREAMS;
    uint64_t *merge_full = pv_done + STREAMS;
    uint64_t *merge_empty = merge_full + STREAMS;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(merge_empty + STREAMS);
    uint32_t *settled = tmem_slot + 1;
    const Waits wait{settled};

    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        mbar_init(q_full, 1);
        mbar_init(q_empty, 1);
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
            mbar_init(&merge_full[t], 4);
            mbar_init(&merge_empty[t], 4);
        }
        *settled = 0;
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
    if (warp < 4) {
    regs_release<kRegsControl>();
    if (warp == 0) {
        // ---------------------------------------------------------- TMA producer (warp converged, one lane issues)
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
            if (!wait(q_empty, (n_units & 1) ^ 1)) { ok = false; break; }
            ++n_units;
            if (elect_one()) {
                mbar_arrive_expect_tx(q_full, L::kQTile);
#pragma unroll
                for (int h = 0; h < NG; ++h) tma_load_3d(smem + h * BQ * 128, &tmQ, q_full, h * 64, (int32_t)u.q0, (int32_t)u.head);
            }
            __syncwarp();
            for (uint32_t j = 0; j < u.n; ++j, ++g) {
                const uint32_t st = g % KV_STAGES, ph = (g / KV_STAGES) & 1;
                if (!wait(&k_empty[st], ph ^ 1)) { ok = false; break; }
                if (elect_one()) {
                    mbar_arrive_expect_tx(&k_full[st], L::kKvTile);
#pragma unroll
                    for (int h = 0; h < NG; ++h)
                        tma_load_3d(smem + L::kOffK + st * L::kKvTile + h * BKV * 128, &tmK, &k_full[st], h * 64, (int32_t)(j * BKV),
                                    (int32_t)u.head);
                }
                __syncwarp();
                if (!wait(&v_empty[st], ph ^ 1)) {
                    ok = false;
                    mbar_wait_warp(&k_full[st], ph);   // the K copy just issued must land before the CTA exits
                    break;
                }
                if (elect_one()) {
                    mbar_arrive_expect_tx(&v_full[st], L::kKvTile);
#pragma unroll
                    for (int h = 0; h < NG; ++h)
                        tma_load_3d(smem + L::kOffV + st * L::kKvTile + h * BKV * 128, &tmV, &v_full[st], h * 64, (int32_t)(j * BKV),
                                    (int32_t)u.head);
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
        if (n_units) mbar_wait_warp(q_full, (n_units - 1) & 1);
    } else if (warp == 1) {
        // ---------------------------------------------------------- Q*K^T of both streams, in the order of the key blocks
        constexpr uint32_t idesc_qk = umma_idesc(1u, BQ, BKV, 0u, 0u);
        const uint32_t k_steps = (p.dim + 15) / 16;
        const uint64_t dQ = umma_smem_desc(smem_u32(smem), 16, 1024), dK = umma_smem_desc(smem_u32(smem) + L::kOffK, 16, 1024);
        bool ok = true;
        uint32_t st = 0, ph = 0;          // ring position
        uint32_t given = 0;               // blocks: even bits of a count a stream (parity of s_full / s_empty)
        uint32_t n = 0;                   // units seen so far
        Unit u;
        for (uint32_t i = 0; ok && unit_at(p, i, u); ++i, ++n) {
            if (!wait(q_full, n & 1)) { ok = false; break; }
            for (uint32_t j = 0; j < u.n; ++j) {
                const uint32_t t = j % STREAMS;
                if (!wait(&k_full[st], ph) || !wait(&s_empty[t], (given >> t & 1) ^ 1)) { ok = false; break; }
                tc_fence_after();
                if (elect_one()) {
                    uint64_t q = dQ, k = dK + ((st * L::kKvTile) >> 4);
#pragma unroll 1
                    for (uint32_t kk = 0; kk < k_steps; ++kk) {
                        umma_f16(tmem_base + t * BKV, q, k, idesc_qk, kk != 0);
                        q += kk == 3 ? (BQ * 128 - 96) >> 4 : 2;   // 16 columns on; the second 64 columns are a group of their own
                        k += kk == 3 ? (BKV * 128 - 96) >> 4 : 2;
                    }
                    umma_commit(&s_full[t]);
                    umma_commit(&k_empty[st]);
                    if (j + 1 == u.n) umma_commit(q_empty);
                }
                __syncwarp();
                given ^= 1u << t;
                if (++st == KV_STAGES) { st = 0; ph ^= 1; }
            }
        }
        if (!ok && lane == 0) kstatus_set(p.status, FE2O3_KSTATUS_WAIT_EXPIRED);
    } else if (warp < 4) {
        // ---------------------------------------------------------- P*V, one warp per stream
        constexpr uint32_t idesc_pv = umma_idesc(1u, BQ, NG * 64, 0u, 1u);   // whole column groups: zeros past the head size
        const uint32_t t = warp - 2;
        const uint64_t dV = umma_smem_desc(smem_u32(smem) + L::kOffV, BKV * 128, 1024),
                       dP = umma_smem_desc(smem_u32(smem) + L::kOffP + t * L::kPTile, 16, 1024);
        const uint32_t tO = tmem_base + kColO + t * 128, tP = tmem_base + kColP + t * BKV;
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
                    const uint64_t v = dV + ((st * L::kKvTile) >> 4);
                    const uint32_t first = starts_group(j / STREAMS) ? 0u : 1u;
#pragma unroll 1
                    for (uint32_t kk = 0; kk < BKV / 16; ++kk)   // lo term: P from shared memory
                        umma_f16(tO, dP + kk * 2, v + kk * 128, idesc_pv, kk == 0 ? first : 1u);
#pragma unroll 1
                    for (uint32_t kk = 0; kk < BKV / 8; ++kk)    // mid, then hi: P from tensor memory
                        umma_f16_ts(tO, tP + ((kk ^ 4u) * 8), v + (kk & 3) * 128, idesc_pv, 1u);
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
        // ---------------------------------------------------------- softmax warps, one thread per query row and stream
        const uint32_t t = (warp - 4) / 4;
        const uint32_t quad = warp & 3;
        const uint32_t r = quad * 32 + lane;                // row inside the unit
        const uint32_t lane_addr = (quad * 32u) << 16;
        const uint32_t tS = tmem_base + t * BKV + lane_addr;
        const uint32_t tO = tmem_base + kColO + t * 128 + lane_addr;
        const uint32_t tP = tmem_base + kColP + t * BKV + lane_addr;
        uint8_t *slice = smem + L::kOffP + t * L::kPTile + quad * 4096;   // this warp's 32 rows of the lo term
        const float c = p.scale_log2;
        constexpr int kHalves = NG == 1 ? 2 : 1;   // halves of a block's scores that stay in registers after the first look
        bool ok = true;
        uint32_t gt = 0;
        uint32_t n = 0;        // units so far
        // Each stream finishes half of the columns: this warp's 32 rows of them, a 4 KiB piece of 32 columns after the
        // other, swizzled as the copy engine stores them.  The other stream writes its part there.
        constexpr uint32_t kHalfCols = NG * 32;
        uint8_t *const rows_out = smem + L::kOffMerge + (t * 4 + quad) * (NG * 4096);
        uint8_t *const rows_given = smem + L::kOffMerge + ((t ^ 1) * 4 + quad) * (NG * 4096);
        auto piece = [&](uint8_t *rows, int q) { return reinterpret_cast<float4 *>(rows + (q >> 3) * 4096 + lane * 128 + (((q & 7) ^ (lane & 7)) * 16)); };
        const uint32_t tMine = tO + t * kHalfCols, tGiven = tO + (t ^ 1) * kHalfCols;
        bool storing = false;  // the copy engine may still be reading rows_out
        auto release_rows = [&]() {
            if (lane == 0) tma_store_wait_read();
            __syncwarp();
            if (lane == 0) mbar_arrive(&merge_empty[t]);
            storing = false;
        };
        Unit u;
        for (uint32_t i = 0; ok && unit_at(p, i, u); ++i) {
            const uint32_t qrow = u.q0 + r;
            float m_ref = -INFINITY;   // exponent offset: a whole number of log2 units, so that every rescaling is exact
            float l = 0.0f;
            bool bad = false;          // a non-finite score of an admitted key
            uint64_t o2[NG * 32];      // the row's output so far, two columns a word; the columns that this stream finishes come first
#pragma unroll
            for (int q = 0; q < NG * 32; ++q) o2[q] = 0ull;
            auto add_group = [&]() {   // the group of blocks that tensor memory holds, once it is complete
#pragma unroll
                for (int h = 0; h < NG * 4; ++h) {
                    uint32_t v[16];
                    tmem_ld_32x32b_x16((h < NG * 2 ? tMine : tGiven) + h % (NG * 2) * 16, v);
                    tmem_ld_wait();
#pragma unroll
                    for (int q = 0; q < 8; ++q)
                        o2[h * 8 + q] = add_f32x2(o2[h * 8 + q], pack_f32x2(__uint_as_float(v[2 * q]), __uint_as_float(v[2 * q + 1])));
                }
            };

            for (uint32_t j = t; j < u.n; j += STREAMS, ++gt) {
                if (!wait(&s_full[t], gt & 1)) { ok = false; break; }
                tc_fence_after();
                const uint32_t key0 = j * BKV;
                const bool edge = key0 + BKV > p.seq || (p.causal && key0 + BKV - 1 > u.q0);
                // Keys of this block that the row admits.  A score of -inf would pass unseen as p = 0, so the least score is
                // looked at too; the other non-finite ones reach the sums.  That of a key that is not admitted makes
                // the row suspect as well, no more: suspects are settled one by one.
                const uint32_t end = p.causal ? min(p.seq, qrow + 1) : p.seq, limit = end > key0 ? end - key0 : 0u;
                float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
                float mn[4] = {INFINITY, INFINITY, INFINITY, INFINITY};
                auto look = [&](uint32_t (&x)[32], uint32_t first) {
#pragma unroll
                    for (int q = 0; q < 32; q += 2) {
                        float d;
                        asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(mn[q / 2 % 4]), "f"(__uint_as_float(x[q])), "f"(__uint_as_float(x[q + 1])));
                        mn[q / 2 % 4] = d;
                    }
                    if (edge) {
#pragma unroll
                        for (int q = 0; q < 32; ++q)
                            if (first + q >= limit) x[q] = 0xff800000u;  // -inf
                    }
#pragma unroll
                    for (int q = 0; q < 32; q += 8)
#pragma unroll
                        for (int w = 0; w < 4; ++w)
                            mx[w] = max3(mx[w], __uint_as_float(x[q + 2 * w]), __uint_as_float(x[q + 2 * w + 1]));
                };
                auto release_scores = [&]() {
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&s_empty[t]);
                };
                const uint64_t c2 = pack_f32x2(c, c);
                uint64_t e2[32];   // the probabilities, two keys a word
                uint64_t sum2[2][2] = {{0ull, 0ull}, {0ull, 0ull}};
                auto exponentials = [&](const uint32_t (&x)[32], int half, uint64_t nmc2) {
                    sum2[half][0] = sum2[half][1] = 0ull;
#pragma unroll
                    for (int q = 0; q < 16; ++q) {
                        float x0, x1;
                        unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(x[2 * q]), __uint_as_float(x[2 * q + 1])), c2, nmc2), x0, x1);
                        e2[half * 16 + q] = pack_f32x2(ex2_approx(x0), ex2_approx(x1));
                        sum2[half][q & 1] = add_f32x2(sum2[half][q & 1], e2[half * 16 + q]);
                    }
                };
                // What fits beside the row's output stays in registers after this look: both halves at head sizes up to 64, else
                // the second; the first is fetched again.
                uint32_t x[kHalves][32];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    if (kHalves == 1 || h == 0) {
                        tmem_ld_32x32b_x32(tS + h * 32, x[0]);
                        if (kHalves == 2) tmem_ld_32x32b_x32(tS + 32, x[kHalves - 1]);
                        tmem_ld_wait();
                        if (kHalves == 2) release_scores();
                    }
                    look(x[h % kHalves], h * 32);
                }
                bad = bad || fminf(fminf(mn[0], mn[1]), fminf(mn[2], mn[3])) == -INFINITY;
                const float rowmax = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
                // move the reference only when the block maximum outgrows it by more than the threshold
                const float top = rowmax * c;
                const bool move = top - m_ref > kRescaleThreshold;  // true for the first admitted key (m_ref = -inf)
                const float moved = fmaf(rintf(top) - top, p.whole, top);
                const float factor = move ? ex2_approx(m_ref - moved) : 1.0f;
                if (move) m_ref = moved;
                const float mc = m_ref == -INFINITY ? 0.0f : m_ref;
                const uint64_t nmc2 = pack_f32x2(-mc, -mc);
                exponentials(x[kHalves - 1], 1, nmc2);
                if constexpr (kHalves == 1) {
                    tmem_ld_32x32b_x32(tS, x[0]);
                    tmem_ld_wait();
                    release_scores();
                    if (edge) {
#pragma unroll
                        for (int q = 0; q < 32; ++q)
                            if (q >= limit) x[0][q] = 0xff800000u;  // -inf
                    }
                }
                exponentials(x[0], 0, nmc2);
                // P of the previous block must have been consumed and O must be quiescent
                if (j >= STREAMS) {
                    if (!wait(&pv_done[t], (gt - 1) & 1)) { ok = false; break; }
                    tc_fence_after();
                    const bool first = starts_group(j / STREAMS);
                    if (first) add_group();
                    if (__any_sync(0xffffffffu, move)) {
                        const uint64_t f2 = pack_f32x2(factor, factor);
#pragma unroll
                        for (int q = 0; q < NG * 32; ++q) o2[q] = mul_f32x2(o2[q], f2);
                        if (!first) {
#pragma unroll 1
                            for (uint32_t gcol = 0; gcol < p.dim; gcol += 8) {
                                uint32_t ov[8];
                                tmem_ld_32x32b_x8(tO + gcol, ov);
                                tmem_ld_wait();
#pragma unroll
                                for (int q = 0; q < 8; ++q) ov[q] = __float_as_uint(__uint_as_float(ov[q]) * factor);
                                tmem_st_32x32b_x8(tO + gcol, ov);
                            }
                        }
                    }
                }
                auto store_p = [&](int h, const uint64_t *e) {   // 16 keys
                    uint32_t hi[8], mid[8], lo[8];   // two probabilities a word
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        uint64_t rest;
                        hi[q] = cut_bf16x2(e[q], rest);
                        mid[q] = cut_bf16x2(rest, rest);
                        float r0, r1;
                        unpack_f32x2(rest, r0, r1);   // at most eight bits are left
                        lo[q] = __byte_perm(__float_as_uint(r0), __float_as_uint(r1), 0x7632);
                    }
                    tmem_st_32x32b_x8(tP + h * 8, hi);
                    tmem_st_32x32b_x8(tP + 32 + h * 8, mid);
#pragma unroll
                    for (int k = 0; k < 2; ++k)
                        *reinterpret_cast<uint4 *>(slice + lane * 128 + (((2 * h + k) ^ (lane & 7)) * 16)) =
                            make_uint4(lo[4 * k], lo[4 * k + 1], lo[4 * k + 2], lo[4 * k + 3]);
                };
#pragma unroll
                for (int h = 0; h < 4; ++h) store_p(h, e2 + h * 8);
                float sum[4];
#pragma unroll
                for (int w = 0; w < 4; ++w) {
                    float a, b;
                    unpack_f32x2(sum2[w >> 1][w & 1], a, b);
                    sum[w] = a + b;
                }
                l = fmaf(l, factor, (sum[0] + sum[1]) + (sum[2] + sum[3]));
                tmem_st_wait();
                fence_proxy_async_smem();   // the lo term is read by the tensor core
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&p_ready[t]);
                if (storing) release_rows();   // the unit before's: by now they have been read
            }
            if (!ok) break;
            if (t < u.n) {
                if (!wait(&pv_done[t], (gt - 1) & 1)) { ok = false; break; }
                tc_fence_after();
                add_group();
                // the next unit's first P*V overwrites O: order this thread's reads of O before its p_ready arrival
                tc_fence_before();
            }
            if (storing) release_rows();
            // The streams' parts of the row meet in shared memory.  A part that is not finite makes the sum NaN for both.
            float *const ref = reinterpret_cast<float *>(smem + L::kOffRow) + r;
            uint64_t check2[2] = {0ull, 0ull};        // 0, or NaN once a value was not finite
#pragma unroll
            for (int q = 0; q < NG * 32; ++q) check2[q & 1] = fma_f32x2(o2[q], 0ull, check2[q & 1]);   // (columns past the head size are zeros)
            float4 check;
            unpack_f32x2(check2[0], check.x, check.y);
            unpack_f32x2(check2[1], check.z, check.w);
            if (bad) l = NAN;
            l += (check.x + check.y) + (check.z + check.w);
            if (!wait(&merge_empty[t ^ 1], (n & 1) ^ 1)) { ok = false; break; }
#pragma unroll
            for (int q = 0; q < NG * 8; ++q) {
                float4 v;
                unpack_f32x2(o2[NG * 16 + 2 * q], v.x, v.y);
                unpack_f32x2(o2[NG * 16 + 2 * q + 1], v.z, v.w);
                *piece(rows_given, q) = v;
            }
            ref[t * 2 * BQ] = m_ref;
            ref[t * 2 * BQ + BQ] = l;
            __syncwarp();
            if (lane == 0) mbar_arrive(&merge_full[t ^ 1]);
            if (!wait(&merge_full[t], n & 1)) { ok = false; break; }
            ++n;
            const float m1 = ref[(t ^ 1) * 2 * BQ], l1 = ref[(t ^ 1) * 2 * BQ + BQ];
            const float m = fmaxf(m_ref, m1), mc = m == -INFINITY ? 0.0f : m;
            const float f0 = ex2_approx(m_ref - mc), f1 = ex2_approx(m1 - mc);   // powers of two
            const float sum = l * f0 + l1 * f1;   // one rounding: the streams agree on it
            const float inv = 1.0f / sum;
            const bool good = isfinite(sum) && sum > 0.0f;
            const uint32_t row0 = u.q0 + quad * 32;   // first query row of this warp
            const uint64_t f02 = pack_f32x2(f0, f0), f12 = pack_f32x2(f1, f1), inv2 = pack_f32x2(inv, inv);
#pragma unroll
            for (int q = 0; q < NG * 8; ++q) {
                const float4 v = *piece(rows_out, q);
                float4 w;
                unpack_f32x2(mul_f32x2(fma_f32x2(o2[2 * q], f02, mul_f32x2(pack_f32x2(v.x, v.y), f12)), inv2), w.x, w.y);
                unpack_f32x2(mul_f32x2(fma_f32x2(o2[2 * q + 1], f02, mul_f32x2(pack_f32x2(v.z, v.w), f12)), inv2), w.z, w.w);
                *piece(rows_out, q) = w;
            }
            const uint32_t unsettled = __ballot_sync(0xffffffffu, !good && qrow < p.seq);
            if (unsettled == 0) {   // full-line writes that do not hold the warp
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) {   // rows beyond seq and columns beyond the head size are clipped
#pragma unroll
                    for (uint32_t h = 0; h < NG; ++h)
                        if (t * kHalfCols + h * 32 < p.dim && row0 < p.seq)
                            tma_store_3d(&tmO, rows_out + h * 4096, (int32_t)(t * kHalfCols + h * 32), (int32_t)row0, (int32_t)u.head);
                    tma_store_commit();
                }
                storing = true;
            } else {
                if (good && qrow < p.seq) {
                    float *dst = p.out + ((uint64_t)u.head * p.seq + qrow) * p.dim + t * kHalfCols;
#pragma unroll 1
                    for (uint32_t q = 0; q < NG * 8; ++q)
                        if (t * kHalfCols + 4 * q < p.dim) reinterpret_cast<float4 *>(dst)[q] = *piece(rows_out, q);
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&merge_empty[t]);
            }
            if (unsettled != 0 && t == 0) {
                auto tick = [settled, lane](uint32_t) { if (lane == 0) atomicAdd(settled, 1u); };
                const uint64_t head = (uint64_t)u.head * p.seq * p.dim;
                const uint32_t last = row0 + 31 - __clz(unsettled);
                const uint32_t bad_key = first_nonfinite_key(p.k + head, p.v + head, p.causal ? last + 1 : p.seq, p.dim, lane, tick);
                for (uint32_t rows = unsettled; rows != 0; rows &= rows - 1) {
                    const uint32_t row = row0 + __ffs(rows) - 1, keys = p.causal ? row + 1 : p.seq;
                    if ((bad_key < keys || !attention_row<uint16_t, NG * 2, 4, false>(p.q, p.k, p.v, p.out, head, row, keys, p.dim, p.scale, lane, tick)) &&
                        lane == 0)
                        kstatus_set(p.status, FE2O3_KSTATUS_NONFINITE);
                }
            }
            __syncwarp();
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

struct AttnSplitPlan {
    CUtensorMap tmQ, tmK, tmV, tmO;
    SplitParams p;
    uint32_t grid, groups;
};

bool attention_split_supported(const fe2o3_flash_attention_v1_args *a) {
    return a->input_dtype == FE2O3_DTYPE_BF16 && a->dim <= 128 && a->dim % 8 == 0 && a->seq >= 1 &&
           (uint64_t)a->batch * a->heads >= 1 && (uint64_t)a->batch * a->heads < (1u << 24) &&
           ((a->q.ptr | a->k.ptr | a->v.ptr | a->output.ptr) & 15u) == 0 && a->scale > 0.0f && a->scale < 1e30f;
}

int32_t attention_split_plan(fe2o3_ctx *ctx, const fe2o3_flash_attention_v1_args *a, AttnSplitPlan **out) {
    AttnSplitPlan *plan = new (std::nothrow) AttnSplitPlan();
    if (!plan) return FE2O3_ERR_SIZE_OVERFLOW;
    const uint32_t bh = a->batch * a->heads;
    uint64_t dims[3] = {a->dim, a->seq, bh};
    uint64_t strides[2] = {(uint64_t)a->dim * 2, (uint64_t)a->seq * a->dim * 2};
    uint32_t qbox[3] = {64, BQ, 1}, kvbox[3] = {64, BKV, 1};
    int32_t st = fe2o3_make_tmap_bf16(&plan->tmQ, a->q.ptr, 3, dims, strides, qbox);
    if (st == FE2O3_OK) st = fe2o3_make_tmap_bf16(&plan->tmK, a->k.ptr, 3, dims, strides, kvbox);
    if (st == FE2O3_OK) st = fe2o3_make_tmap_bf16(&plan->tmV, a->v.ptr, 3, dims, strides, kvbox);
    if (st == FE2O3_OK) {
        uint64_t ostrides[2] = {(uint64_t)a->dim * 4, (uint64_t)a->seq * a->dim * 4};
        uint32_t obox[3] = {32, 32, 1};
        st = fe2o3_make_tmap_f32(&plan->tmO, a->output.ptr, 3, dims, ostrides, obox);
    }
    if (st != FE2O3_OK) { delete plan; return st; }
    const uint32_t q_blocks = (uint32_t)(((uint64_t)a->seq + BQ - 1) / BQ);
    const uint64_t units = (uint64_t)bh * q_blocks;
    const uint32_t sms = ctx->sm_count > 0 ? (uint32_t)ctx->sm_count : 1u;
    if (units > 0x7fffffffull) { delete plan; fe2o3_set_error("UnsupportedShape: too many rows"); return FE2O3_ERR_UNSUPPORTED_SHAPE; }
    plan->p = SplitParams{reinterpret_cast<const uint16_t *>(a->q.ptr), reinterpret_cast<const uint16_t *>(a->k.ptr),
                          reinterpret_cast<const uint16_t *>(a->v.ptr), reinterpret_cast<float *>(a->output.ptr), bh, a->seq, a->dim,
                          a->scale, a->scale * 1.4426950408889634f, a->causal,
                          q_blocks, (uint32_t)units, a->seq <= BKV ? 0.0f : 1.0f, ctx->status_word};
    plan->grid = plan->p.units < sms ? plan->p.units : sms;
    plan->groups = a->dim <= 64 ? 1 : 2;
    *out = plan;
    return FE2O3_OK;
}

// Function attributes are per device: called by fe2o3_ctx_create with the context's device current.
int32_t attention_split_init_device() {
    FE2O3_CUDA(cudaFuncSetAttribute(attention_split_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Layout<1>::kTotal));
    FE2O3_CUDA(cudaFuncSetAttribute(attention_split_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Layout<2>::kTotal));
    return FE2O3_OK;
}

int32_t attention_split_launch(const AttnSplitPlan *plan, cudaStream_t s) {
    const cudaError_t e =
        plan->groups == 1 ? fe2o3_launch_early(attention_split_kernel<1>, plan->grid, kThreads, Layout<1>::kTotal, s, 1, plan->tmQ,
                                               plan->tmK, plan->tmV, plan->tmO, plan->p)
                          : fe2o3_launch_early(attention_split_kernel<2>, plan->grid, kThreads, Layout<2>::kTotal, s, 1, plan->tmQ,
                                               plan->tmK, plan->tmV, plan->tmO, plan->p);
    fe2o3_count_launch(1);
    return fe2o3_cuda_status(e, "flash_attention_v1(tcgen05, split)");
}

void attention_split_geometry(const AttnSplitPlan *plan, fe2o3_geometry *geo) {
    *geo = fe2o3_geometry{{plan->grid, 1, 1}, {kThreads, 1, 1}, plan->groups == 1 ? Layout<1>::kTotal : Layout<2>::kTotal, 1};
}

void attention_split_free(AttnSplitPlan *plan) { delete plan; }
