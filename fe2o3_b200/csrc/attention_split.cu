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
// additions round to nearest: 7.7e-7 at 4096 keys, and not above the CUDA cores from 333
// to 4096 keys; at 50, one block, either may be the nearer by a fifth.  The price is a read of O per group between one P*V and the next, and
// the registers of a row of O: beyond 64 columns half of the scores is fetched twice,
// and the probabilities wait as f32 in the scores' registers and are cut after the wait
// for the previous P*V (cut before it, 96 words do not fit beside the row; both looks
// after it: 110 us for the 82.6 below; one half's exponentials after it: 87).
// B2 H12 S1900 D128 causal: 65 us with one sum per row, 82.6 so; not causal 127, 158;
// 64 heads of 1024 x 32, causal: 41, 52.5.
//   Per 128 x 64 block at head size 128 the tensor pipe then
// works 256 (Q*K^T) + 3 x 256 cycles, against 512 of the exponential unit.
//
// Structure, as in attention_tc.cu: persistent CTAs, one per SM, over units of 256
// query rows handled as two 128-row tiles that share every K/V block; warp 0 loads
// (TMA), warps 1 and 2 issue the MMAs of tile 0 and tile 1, warps 4-7 and 8-11 are
// the softmax warps of the tiles, one thread per row, with most of the registers.
//   64-key blocks and P's lo term in shared memory instead of tensor memory are what
//   fits two tiles at head size 128: S 2 x 64, O 2 x 128 and hi, mid 2 x 2 x 32 make
//   the 512 columns.  So S has columns of its own and the next Q*K^T overlaps the
//   exponentials.  The lo buffer doubles as the staging buffer of the output.
//   Causal units are ordered by length, longest first, and dealt out in alternating
//   direction (round 0 forwards, round 1 backwards); a tile stops at its own last block.
//   Head sizes below 64 or between 64 and 128 are zero-filled by the copy engine on the
//   way in and clipped on the way out; Q*K^T takes only the k steps in use.
//   A row that met a non-finite score or value is settled one by one: the tensor core
//   also multiplies the values of keys that a causal row does not admit, by probabilities
//   of 0, and 0 x Inf is NaN.  The first key of the head with a non-finite K or V is
//   searched once; a row that admits it is left unwritten and reported, the others are
//   computed by the CUDA-core recurrence (attention_row.cuh).
//   The other warps may wait long meanwhile, so waits that run out start over as long as
//   rows are being settled (Waits).
// B2 H12 S1900 D128 causal: 8017 us on the CUDA cores, 82.6 us here (longest unit 30 of
// an average 19.5 block pairs).
// The rule in front (attention_split_supported) is what the copy engine can address:
// rows of whole 16 bytes and 16-byte aligned bases; the rest, f32 inputs and head sizes
// above 128 stay on the CUDA cores.  All waits are bounded.
#include "attention_row.cuh"
#include "gemm_tc.h"

#include <new>

namespace {

constexpr int BQ = 128;          // query rows per tile
constexpr int BKV = 64;          // keys per block
constexpr int QT = 2;            // query tiles per unit
constexpr int KV_STAGES = 4;
constexpr int kThreads = 32 * (4 + 4 * QT);
// (56 and 224: 84.8 us for 82.6, in spite of fewer bytes spilled, 168 against 256 at two column groups, 20 against 84 at one)
constexpr int kRegsControl = 40, kRegsSoftmax = 232;
static_assert(128 * kRegsControl + QT * 128 * kRegsSoftmax <= kThreads * 168, "the warpgroups share what the block is launched with");
constexpr float kRescaleThreshold = 8.0f;              // log2 units

// NG: groups of 64 head columns (128 bytes) per row
template <int NG>
struct Layout {
    static constexpr uint32_t kQTile = NG * BQ * 128;      // [group][128 rows][128 bytes]
    static constexpr uint32_t kKvTile = NG * BKV * 128;    // [group][64 keys][128 bytes]
    static constexpr uint32_t kPTile = BQ * 128;           // lo term: [128 rows][64 keys]
    static constexpr uint32_t kOffK = QT * kQTile;
    static constexpr uint32_t kOffV = kOffK + KV_STAGES * kKvTile;
    static constexpr uint32_t kOffP = kOffV + KV_STAGES * kKvTile;
    static constexpr uint32_t kOffBar = kOffP + QT * kPTile;
    static constexpr uint32_t kTotal = kOffBar + 512 + 1024;   // + alignment slack
};

// TMEM columns: S tile t at t*64, O tile t at 128 + t*128, P tile t at 384 + t*64 (hi 32, mid 32)
constexpr uint32_t kTmemCols = 512, kColO = 128, kColP = 384;

struct SplitParams {
    const uint16_t *q, *k, *v;   // for rows that are settled one by one
    float *out;
    uint32_t bh, seq, dim;
    float scale, scale_log2;   // scale_log2 = scale * log2(e)
    uint32_t causal;
    uint32_t q_blocks;  // 256-row blocks per head
    uint32_t units;     // work units; `half`: of one tile each, two per block
    uint32_t half;
    uint32_t *status;
};

struct Unit {
    uint32_t head, q0, nkv;
    uint32_t n[QT];     // key blocks of each tile, 0 = no such tile here; nkv = the larger
};

// The i-th unit of this CTA; false when there is none.  Every role walks the same sequence.
__device__ __forceinline__ bool unit_at(const SplitParams &p, uint32_t i, Unit &u) {
    const uint32_t idx = i * gridDim.x + ((i & 1) ? gridDim.x - 1 - blockIdx.x : blockIdx.x);
    if (idx >= p.units) return false;
    const uint32_t block = p.half ? idx >> 1 : idx;
    const uint32_t qb = p.causal ? p.q_blocks - 1 - block / p.bh : block % p.q_blocks;
    u.head = p.causal ? block % p.bh : block / p.q_blocks;
    u.q0 = qb * (QT * BQ) + (p.half ? (idx & 1) * BQ : 0);
    u.nkv = 0;
#pragma unroll
    for (uint32_t t = 0; t < QT; ++t) {
        const uint32_t first = u.q0 + t * BQ;
        u.n[t] = 0;
        if (first < p.seq && !(p.half && t > 0))
            u.n[t] = ((p.causal ? min(p.seq, first + BQ) : p.seq) + BKV - 1) / BKV;
        u.nkv = max(u.nkv, u.n[t]);
    }
    return true;
}

// Key blocks whose P*V starts a new sum in tensor memory; the sum before is added to the row's registers.
__device__ __forceinline__ bool starts_group(uint32_t j) { return (j & (j < 4 ? 0u : j < 16 ? 1u : 3u)) == 0; }

template <int N>
__device__ __forceinline__ void regs_release() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N>
__device__ __forceinline__ void regs_take() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }

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

// Waits on another role of the block.  `settled` moves on as long as rows are being settled one by one.
struct Waits {
    const volatile uint32_t *settled;
    __device__ __forceinline__ bool operator()(uint64_t *bar, uint32_t parity) const {
        uint32_t seen = 0;
        while (!mbar_wait_warp(bar, parity)) {
            const uint32_t now = __shfl_sync(0xffffffffu, *settled, 0);
            if (now == seen) return false;
            seen = now;
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
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + L::kOffBar);
    uint64_t *q_full = bars;
    uint64_t *q_empty = q_full + 1;
    uint64_t *k_full = q_empty + 1;                // KV_STAGES each
    uint64_t *k_empty = k_full + KV_STAGES;
    uint64_t *v_full = k_empty + KV_STAGES;
    uint64_t *v_empty = v_full + KV_STAGES;
    uint64_t *s_full = v_empty + KV_STAGES;        // QT each
    uint64_t *s_empty = s_full + QT;
    uint64_t *p_ready = s_empty + QT;
    uint64_t *pv_done = p_ready + QT;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(pv_done + QT);
    uint32_t *settled = tmem_slot + 1;
    const Waits wait{settled};

    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        mbar_init(q_full, 1);
        mbar_init(q_empty, QT);
        for (int i = 0; i < KV_STAGES; ++i) {
            mbar_init(&k_full[i], 1);
            mbar_init(&k_empty[i], QT);
            mbar_init(&v_full[i], 1);
            mbar_init(&v_empty[i], QT);
        }
        for (int t = 0; t < QT; ++t) {
            mbar_init(&s_full[t], 1);
            mbar_init(&s_empty[t], 4);
            mbar_init(&p_ready[t], 4);
            mbar_init(&pv_done[t], 1);
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
            if (u.nkv == 0) continue;   // every role skips a unit whose rows all lie beyond seq
            if (!wait(q_empty, (n_units & 1) ^ 1)) { ok = false; break; }
            ++n_units;
            if (elect_one()) {
                mbar_arrive_expect_tx(q_full, ((u.n[0] ? 1u : 0u) + (u.n[1] ? 1u : 0u)) * L::kQTile);
                for (uint32_t t = 0; t < QT; ++t) {
                    if (u.n[t] == 0) continue;
#pragma unroll
                    for (int h = 0; h < NG; ++h)
                        tma_load_3d(smem + t * L::kQTile + h * BQ * 128, &tmQ, q_full, h * 64, (int32_t)(u.q0 + t * BQ), (int32_t)u.head);
                }
            }
            __syncwarp();
            for (uint32_t j = 0; j < u.nkv; ++j, ++g) {
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
    } else if (warp == 1 || warp == 2) {
        // ---------------------------------------------------------- MMA issuers, one warp per query tile
        // Per tile: Q*K^T of block b+1 (its S columns are free once the softmax has read block b), then P*V of
        // block b; block b+1 may already belong to the next unit.
        const uint32_t t = warp - 1;
        const uint32_t k_steps = (p.dim + 15) / 16;
        constexpr uint32_t idesc_qk = umma_idesc(1u, BQ, BKV, 0u, 0u);
        constexpr uint32_t idesc_pv = umma_idesc(1u, BQ, NG * 64, 0u, 1u);   // whole column groups: zeros past the head size
        const uint64_t dQ = umma_smem_desc(smem_u32(smem) + t * L::kQTile, 16, 1024),
                       dK = umma_smem_desc(smem_u32(smem) + L::kOffK, 16, 1024),
                       dV = umma_smem_desc(smem_u32(smem) + L::kOffV, BKV * 128, 1024),
                       dP = umma_smem_desc(smem_u32(smem) + L::kOffP + t * L::kPTile, 16, 1024);
        const uint32_t tS = tmem_base + t * BKV, tO = tmem_base + kColO + t * 128, tP = tmem_base + kColP + t * BKV;
        bool ok = true;
        uint32_t g = 0;    // key blocks over all units: ring position of K/V
        uint32_t gt = 0;   // key blocks this tile has processed: parity of s_* / p_ready / pv_done
        uint32_t n = 0;    // units with keys seen so far
        bool pending = false;
        uint32_t pv_st = 0, pv_ph = 0, pv_gt = 0, pv_acc = 0;
        auto issue_pv = [&]() {
            pending = false;
            if (!wait(&p_ready[t], pv_gt & 1) || !wait(&v_full[pv_st], pv_ph)) { ok = false; return; }
            tc_fence_after();
            if (elect_one()) {
                const uint64_t dVs = dV + ((pv_st * L::kKvTile) >> 4);
#pragma unroll
                for (int kk = 0; kk < BKV / 16; ++kk)   // lo term: P from shared memory
                    umma_f16(tO, dP + ((kk * 32) >> 4), dVs + ((kk * 2048) >> 4), idesc_pv, kk == 0 ? pv_acc : 1u);
#pragma unroll
                for (int term = 1; term >= 0; --term)   // mid, then hi: P from tensor memory
#pragma unroll
                    for (int kk = 0; kk < BKV / 16; ++kk)
                        umma_f16_ts(tO, tP + term * (BKV / 2) + kk * 8, dVs + ((kk * 2048) >> 4), idesc_pv, 1u);
                umma_commit(&pv_done[t]);
                umma_commit(&v_empty[pv_st]);
            }
            __syncwarp();
        };
        Unit u;
        for (uint32_t i = 0; ok && unit_at(p, i, u); ++i) {
            if (u.nkv == 0) continue;
            const uint32_t qph = n & 1, mine = t == 0 ? u.n[0] : u.n[1];
            ++n;
            if (!wait(q_full, qph)) { ok = false; break; }
            if (mine == 0 && lane == 0) mbar_arrive(q_empty);   // no such tile here: nothing of Q is read
            for (uint32_t j = 0; ok && j < u.nkv; ++j, ++g) {
                const uint32_t st = g % KV_STAGES, ph = (g / KV_STAGES) & 1;
                if (j >= mine) {   // past this tile's last block: only hand the other tile's K/V blocks on
                    if (pending) issue_pv();
                    if (!ok || !wait(&k_full[st], ph)) { ok = false; break; }
                    if (lane == 0) mbar_arrive(&k_empty[st]);
                    if (!wait(&v_full[st], ph)) { ok = false; break; }
                    if (lane == 0) mbar_arrive(&v_empty[st]);
                    continue;
                }
                if (!wait(&s_empty[t], (gt & 1) ^ 1) || !wait(&k_full[st], ph)) { ok = false; break; }
                tc_fence_after();
                if (elect_one()) {
                    const uint64_t dKs = dK + ((st * L::kKvTile) >> 4);
#pragma unroll
                    for (uint32_t kk = 0; kk < NG * 4; ++kk)
                        if (kk < k_steps)
                            umma_f16(tS, dQ + (((kk >> 2) * BQ * 128 + (kk & 3) * 32) >> 4),
                                     dKs + (((kk >> 2) * BKV * 128 + (kk & 3) * 32) >> 4), idesc_qk, kk != 0);
                    umma_commit(&s_full[t]);
                    umma_commit(&k_empty[st]);
                    if (j + 1 == mine) umma_commit(q_empty);
                }
                __syncwarp();
                if (pending) issue_pv();
                pv_st = st; pv_ph = ph; pv_gt = gt; pv_acc = starts_group(j) ? 0u : 1u;
                pending = true;
                ++gt;
            }
        }
        if (ok && pending) issue_pv();
        if (!ok && lane == 0) kstatus_set(p.status, FE2O3_KSTATUS_WAIT_EXPIRED);
    }
    // warp 3 idles: it keeps the softmax warps at four per scheduler and their TMEM quadrant equal to warp % 4
    } else {
        regs_take<kRegsSoftmax>();
        // ---------------------------------------------------------- softmax warps, one thread per query row
        const uint32_t t = (warp - 4) / 4;
        const uint32_t quad = warp & 3;
        const uint32_t r = quad * 32 + lane;                // row inside the tile
        const uint32_t lane_addr = (quad * 32u) << 16;
        const uint32_t tS = tmem_base + t * BKV + lane_addr;
        const uint32_t tO = tmem_base + kColO + t * 128 + lane_addr;
        const uint32_t tP = tmem_base + kColP + t * BKV + lane_addr;
        uint8_t *slice = smem + L::kOffP + t * L::kPTile + quad * 4096;   // this warp's 32 rows of the lo term
        const float c = p.scale_log2;
        constexpr int kHalves = NG == 1 ? 2 : 1;   // halves of a block's scores that stay in registers after the first look
        bool ok = true;
        uint32_t gt = 0;
        Unit u;
        for (uint32_t i = 0; ok && unit_at(p, i, u); ++i) {
            const uint32_t mine = t == 0 ? u.n[0] : u.n[1];
            if (mine == 0) continue;
            const uint32_t first_row = u.q0 + t * BQ, qrow = first_row + r;
            float m_ref = -INFINITY;   // exponent offset, in raw score units
            float l = 0.0f;
            bool bad = false;          // a non-finite score of an admitted key
            uint64_t o2[NG * 32];      // the row's output so far, two columns a word
#pragma unroll
            for (int q = 0; q < NG * 32; ++q) o2[q] = 0ull;
            auto add_group = [&]() {   // the group of blocks that tensor memory holds, once it is complete
#pragma unroll
                for (int h = 0; h < NG * 4; ++h) {
                    uint32_t v[16];
                    tmem_ld_32x32b_x16(tO + h * 16, v);
                    tmem_ld_wait();
#pragma unroll
                    for (int q = 0; q < 8; ++q)
                        o2[h * 8 + q] = add_f32x2(o2[h * 8 + q], pack_f32x2(__uint_as_float(v[2 * q]), __uint_as_float(v[2 * q + 1])));
                }
            };

            for (uint32_t j = 0; j < mine; ++j, ++gt) {
                if (!wait(&s_full[t], gt & 1)) { ok = false; break; }
                tc_fence_after();
                const uint32_t key0 = j * BKV;
                const bool edge = key0 + BKV > p.seq || (p.causal && key0 + BKV - 1 > first_row);
                auto admitted = [&](uint32_t key) { return key < p.seq && (!p.causal || key <= qrow); };
                // A first look at the scores, 32 keys at a time, for their maximum.  What fits beside the row's output stays in
                // registers: both halves at head sizes up to 64, else the second.
                uint32_t s[kHalves][32];
                float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
                float mn[4] = {INFINITY, INFINITY, INFINITY, INFINITY};
                auto release_scores = [&]() {
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&s_empty[t]);
                };
                auto mask = [&](uint32_t (&x)[32], uint32_t first_key) {
#pragma unroll
                    for (int q = 0; q < 32; ++q)
                        if (!admitted(first_key + q)) x[q] = 0xff800000u;  // -inf
                };
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    uint32_t (&x)[32] = s[h % kHalves];
                    if (kHalves == 1 || h == 0) {
                        tmem_ld_32x32b_x32(tS + h * 32, x);
                        if (kHalves == 2) tmem_ld_32x32b_x32(tS + 32, s[kHalves - 1]);
                        tmem_ld_wait();
                        if (kHalves == 2) release_scores();
                    }
                    if (edge) {
#pragma unroll
                        for (int q = 0; q < 32; ++q)
                            if (admitted(key0 + h * 32 + q)) bad = bad || !isfinite(__uint_as_float(x[q]));
                        mask(x, key0 + h * 32);
                    } else {
                        // a score of -inf would pass unseen as p = 0; the other non-finite ones reach the sums
#pragma unroll
                        for (int q = 0; q < 32; q += 2) {
                            float d;
                            asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(mn[q / 2 % 4]), "f"(__uint_as_float(x[q])), "f"(__uint_as_float(x[q + 1])));
                            mn[q / 2 % 4] = d;
                        }
                    }
#pragma unroll
                    for (int q = 0; q < 32; q += 8)
#pragma unroll
                        for (int w = 0; w < 4; ++w)
                            mx[w] = max3(mx[w], __uint_as_float(x[q + 2 * w]), __uint_as_float(x[q + 2 * w + 1]));
                }
                bad = bad || fminf(fminf(mn[0], mn[1]), fminf(mn[2], mn[3])) == -INFINITY;
                const float rowmax = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
                // move the reference only when the block maximum outgrows it by more than the threshold
                const bool move = (rowmax - m_ref) * c > kRescaleThreshold;  // true for the first admitted key (m_ref = -inf)
                const float factor = move ? ex2_approx((m_ref - rowmax) * c) : 1.0f;
                if (move) m_ref = rowmax;
                const float mc = (m_ref == -INFINITY ? 0.0f : m_ref) * c;
                const uint64_t c2 = pack_f32x2(c, c), nmc2 = pack_f32x2(-mc, -mc);
                uint64_t sum2[4] = {0ull, 0ull, 0ull, 0ull};
                auto probability = [&](uint32_t s0, uint32_t s1, int q) {
                    const uint64_t x2 = fma_f32x2(pack_f32x2(__uint_as_float(s0), __uint_as_float(s1)), c2, nmc2);
                    float x0, x1;
                    unpack_f32x2(x2, x0, x1);
                    const uint64_t e = pack_f32x2(ex2_approx(x0), ex2_approx(x1));
                    sum2[q & 3] = add_f32x2(sum2[q & 3], e);
                    return e;
                };
                uint64_t e2[32];   // the probabilities, in the registers of their scores
#pragma unroll
                for (int q = 0; q < kHalves * 16; ++q) e2[32 - kHalves * 16 + q] = probability(s[q / 16][2 * (q % 16)], s[q / 16][2 * (q % 16) + 1], q);
                if constexpr (kHalves == 1) {   // the scores of the first half are fetched again
                    tmem_ld_32x32b_x32(tS, s[0]);
                    tmem_ld_wait();
                    release_scores();
                    if (edge) mask(s[0], key0);
#pragma unroll
                    for (int q = 0; q < 16; ++q) e2[q] = probability(s[0][2 * q], s[0][2 * q + 1], q);
                }
                // P of the previous block must have been consumed and O must be quiescent
                if (j > 0) {
                    if (!wait(&pv_done[t], (gt - 1) & 1)) { ok = false; break; }
                    tc_fence_after();
                    const bool first = starts_group(j);
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
                    unpack_f32x2(sum2[w], a, b);
                    sum[w] = a + b;
                }
                l = fmaf(l, factor, (sum[0] + sum[1]) + (sum[2] + sum[3]));
                tmem_st_wait();
                fence_proxy_async_smem();   // the lo term is read by the tensor core
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&p_ready[t]);
            }
            if (!ok) break;
            if (!wait(&pv_done[t], (gt - 1) & 1)) { ok = false; break; }
            tc_fence_after();
            add_group();
            const float inv = 1.0f / l;
            bool good = !bad && isfinite(l) && l > 0.0f;
            const uint32_t row0 = first_row + quad * 32;   // first query row of this warp
            const uint64_t inv2 = pack_f32x2(inv, inv);
#pragma unroll
            for (int q = 0; q < NG * 32; ++q) {
                o2[q] = mul_f32x2(o2[q], inv2);
                float v0, v1;
                unpack_f32x2(o2[q], v0, v1);
                if (2 * q < p.dim) good = good && isfinite(v0) && isfinite(v1);   // (the head size is even)
            }
            const uint32_t unsettled = __ballot_sync(0xffffffffu, !good && qrow < p.seq);
            if (unsettled == 0) {
                // through shared memory and the copy engine: full-line writes that do not hold the warp
#pragma unroll
                for (int h = 0; h < NG * 2; ++h) {
                    if (h * 32 >= p.dim) break;
                    if (h > 0) {
                        if (lane == 0) tma_store_wait_read();   // the slice is still being read by the previous copy
                        __syncwarp();
                    }
#pragma unroll
                    for (int k = 0; k < 8; ++k)
                        *reinterpret_cast<uint4 *>(slice + lane * 128 + ((k ^ (lane & 7)) * 16)) =
                            make_uint4((uint32_t)o2[h * 16 + 2 * k], (uint32_t)(o2[h * 16 + 2 * k] >> 32), (uint32_t)o2[h * 16 + 2 * k + 1],
                                       (uint32_t)(o2[h * 16 + 2 * k + 1] >> 32));
                    fence_proxy_async_smem();
                    __syncwarp();
                    if (lane == 0 && row0 < p.seq) {   // rows beyond seq and columns beyond the head size are clipped
                        tma_store_3d(&tmO, slice, h * 32, (int32_t)row0, (int32_t)u.head);
                        tma_store_commit();
                    }
                }
                if (lane == 0) tma_store_wait_read();   // before the next unit's lo term overwrites the slice
            } else if (good && qrow < p.seq) {
                float *dst = p.out + ((uint64_t)u.head * p.seq + qrow) * p.dim;
#pragma unroll
                for (int q = 0; q < NG * 32; ++q)
                    if (2 * q < p.dim) {
                        float2 v;
                        unpack_f32x2(o2[q], v.x, v.y);
                        reinterpret_cast<float2 *>(dst)[q] = v;
                    }
            }
            if (unsettled != 0) {
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
            // the next unit's first P*V overwrites O: order this thread's reads of O before its p_ready arrival
            tc_fence_before();
            __syncwarp();
        }
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
    // Two-tile units share their K/V loads and overlap one tile's exponentials with the other's MMAs; where they
    // would leave half of the SMs without work, single tiles.
    const uint32_t q_blocks = (uint32_t)(((uint64_t)a->seq + QT * BQ - 1) / (QT * BQ));
    const uint64_t units = (uint64_t)bh * q_blocks;
    const uint32_t sms = ctx->sm_count > 0 ? (uint32_t)ctx->sm_count : 1u;
    if (units > 0x7fffffffull) { delete plan; fe2o3_set_error("UnsupportedShape: too many rows"); return FE2O3_ERR_UNSUPPORTED_SHAPE; }
    const bool half = 2 * units <= sms;
    plan->p = SplitParams{reinterpret_cast<const uint16_t *>(a->q.ptr), reinterpret_cast<const uint16_t *>(a->k.ptr),
                          reinterpret_cast<const uint16_t *>(a->v.ptr), reinterpret_cast<float *>(a->output.ptr), bh, a->seq, a->dim,
                          a->scale, a->scale * 1.4426950408889634f, a->causal,
                          q_blocks, (uint32_t)(half ? 2 * units : units), half ? 1u : 0u, ctx->status_word};
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
