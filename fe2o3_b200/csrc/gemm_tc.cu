// Tensor-core GEMM schedule for sm_100a: bf16 x bf16 -> f32 on tcgen05 with the
// accumulator in TMEM, operands staged by TMA into 128-byte-swizzled shared
// memory through an mbarrier ring.
//
// Replaces the MFMA + LDS schedule of examples/tiled_gemm_v1/src/kernel.rs:63-124
// and examples/tiled_gemm_general_v1/src/kernel.rs:67-120 (one wave per 16x16
// tile, single-buffered LDS, two barriers per K phase) and, in grouped mode,
// the per-expert GEMM launches of examples/moe_expert_v1/src/pipeline.rs:181-187.
//
// Layout.  A is row-major [M][K] (K contiguous, "K-major"); B is row-major
// [K][N] (N contiguous, "MN-major") exactly as the reference stores them, so no
// transpose pass is needed: the instruction descriptor marks B as MN-major.
// A CTA owns a 128 x BN output tile (BN 64, 128, 192 or 256); one K block is 64 bf16 = 128 bytes.
//   A stage: one TMA box {64 k, 128 rows}  -> 128 rows x 128 B, 8-row groups 1 KiB apart
//   B stage: BN/64 TMA boxes {64 n, 64 k}   -> per box 64 k-rows x 128 B (8 KiB)
// What bounds the large products is power (at 1000 W the clock falls to 1.1 GHz, and the tensor pipe is 90 % busy
// at it) and, before that, the 48 KiB of operands that a 128 x 256 tile stages per k block: a pair of CTAs on two
// SMs (CG = 2) owns a 256 x 256 tile, each staging its rows of A and half of B, one issuer driving both tensor
// pipes (cta_group::2).  8192^3: 907 us with single CTAs, 832 so.
// Persistent CTAs (one per SM) walk a static tile list; ten warps:
//   warp 0  TMA producer (one lane)        warp 1  MMA issuer (one lane) + TMEM owner
//   warps 2-9  epilogue: TMEM -> registers -> shared memory -> bulk tensor store,
//              two warps per TMEM lane quadrant, half of the tile's columns each
// Two accumulator buffers in TMEM let the epilogue of tile i overlap the main
// loop of tile i+1.  Every wait is bounded: on expiry the kernel records
// FE2O3_KSTATUS_WAIT_EXPIRED, drains its own copies and returns.
#include "gemm_tc.h"

#include <mutex>

namespace {

constexpr int BM = 128;
constexpr int BK = 64;          // bf16 elements per K block (128 bytes)
constexpr int UMMA_K = 16;
constexpr int kEpilogueWarps = 8;
constexpr int kThreads = 32 * (2 + kEpilogueWarps);
constexpr int kGatherThreads = 128;  // four more warps when A is gathered row by row (copy-engine gathers, so that the bytes
                                     // are counted like every other load's), on the 128-register build
constexpr uint32_t kEarlyWeights = 2;   // GemmParams::after_previous
constexpr int kGroupM = 16;     // m-tiles per rasterisation band (keeps a wave's A and B panels in L2)

// CG = blocks per tile.  CG = 2: a pair of blocks on two neighbouring SMs owns a 256 x BN tile; each block stages its
// own 128 rows of A and its half of B's columns, so a k block costs 32 KiB of staging per SM instead of 48.
template <int BN, int CG>
struct SmemLayout {
    static constexpr int kStages = BN == 64 ? 8 : BN == 128 || CG == 2 ? 6 : 4;   // 192 KiB in flight, 160 at 192 columns
    static constexpr uint32_t kTmemCols = BN == 192 ? 512 : 2 * BN;            // (a power of two)
    static constexpr uint32_t kABytes = BM * BK * 2;
    static constexpr uint32_t kBBytes = BN / CG * BK * 2;
    static constexpr uint32_t kStageBytes = kABytes + kBBytes;
    static constexpr uint32_t kStagingOffset = kStages * kStageBytes;          // 4 KiB output slice per epilogue warp
    static constexpr uint32_t kBarOffset = kStagingOffset + kEpilogueWarps * 4096;
    static constexpr uint32_t kTotal = kBarOffset + 256 + 1024;  // barriers + alignment slack
};

struct TileCoord {
    uint32_t m0, n0, m_end, expert;
    uint32_t mt_index;   // running index of the 128-row tile over all groups (expert-parallel hand-over counters)
    bool valid;
};

// What a build of the kernel is for.  One for all of them was 0.5 us slower a launch, whatever it was launched for: code that
// a launch steps over still has to come past the instruction caches.
enum GemmKind : int { kPlain, kUpdate /* alpha/beta */, kGrouped /* f32 rows, or added to token rows */, kGroupedGelu,
                      kPeer /* expert-parallel: rows scattered to their home ranks */, kPeerGelu };
__host__ __device__ constexpr bool is_grouped(int kind) { return kind >= kGrouped; }
__host__ __device__ constexpr bool is_gelu(int kind) { return kind == kGroupedGelu || kind == kPeerGelu; }
__host__ __device__ constexpr bool is_peer(int kind) { return kind >= kPeer; }

// Static tile order.  Plain: bands of kGroupM m-tiles, m fastest inside a band.
// Grouped: expert-major; inside an expert m fastest.  Grouped with per-source waiting (first GEMM of
// the expert-parallel FFN): by the source rank of the tile's first row, this rank's own rows first
// (they never cross NVLink), then ranks +1, +2, ... which is the order in which the other ranks send
// to this one; inside a source by local expert, then m, n fastest.
// TM: rows of a tile (128, or 256 for a pair of blocks).
template <int TM, int KIND>
__device__ __forceinline__ TileCoord decode_tile(uint32_t id, const GemmParams &p, uint32_t n_tiles,
                                                 const uint32_t *s_off, const uint32_t *s_pair) {
    TileCoord t;
    t.valid = false;
    t.expert = 0;
    t.m0 = t.n0 = t.m_end = t.mt_index = 0;
    if constexpr (!is_grouped(KIND)) {
        constexpr uint32_t kBand = kGroupM * BM / TM;
        const uint32_t m_tiles = (p.M + TM - 1) / TM;
        if (id >= m_tiles * n_tiles) return t;
        const uint32_t band = id / (kBand * n_tiles);
        const uint32_t first_m = band * kBand;
        const uint32_t band_m = min(kBand, m_tiles - first_m);
        const uint32_t local = id - band * kBand * n_tiles;
        t.m0 = (first_m + local % band_m) * TM;
        t.n0 = (local / band_m);
        t.m_end = p.M;
        t.valid = true;
        return t;
    }
    if (is_peer(KIND) && TM == BM && (p.ep.rows_flags || p.ep.progress_mode)) {
        // groups = (run j, local expert le): the tiles whose first row belongs to source (rank + j) mod W; inside
        // an expert's segment the runs lie in exactly that order (the owner's own rows first)
        const uint32_t W = p.ep.world;
        uint32_t base = 0;
        for (uint32_t g = 0; g < W * p.experts; ++g) {
            const uint32_t j = g / p.experts, le = g % p.experts;
            const uint32_t pi = le * W + j;
            const uint32_t seg = s_off[le], lo = s_pair[pi] - seg, hi = s_pair[pi + 1] - seg;
            const uint32_t i0 = (lo + BM - 1) / BM, i1 = (hi + BM - 1) / BM;   // tile starts seg + i * BM in [lo, hi)
            const uint32_t cnt = hi > lo ? (i1 - i0) * n_tiles : 0u;
            if (id < base + cnt) {
                const uint32_t local = id - base;
                const uint32_t mi = i0 + local / n_tiles;
                t.m0 = seg + mi * BM;
                t.n0 = local % n_tiles;
                t.m_end = s_off[le + 1];
                t.expert = le;
                t.mt_index = mi;
                for (uint32_t l2 = 0; l2 < le; ++l2) t.mt_index += (s_off[l2 + 1] - s_off[l2] + BM - 1) / BM;
                t.valid = true;
                break;
            }
            base += cnt;
        }
    } else {
        uint32_t base = 0;
        for (uint32_t e = 0; e < p.experts; ++e) {
            const uint32_t rows = s_off[e + 1] - s_off[e];
            const uint32_t mt = (rows + TM - 1) / TM;
            const uint32_t cnt = mt * n_tiles;
            if (id < base + cnt) {
                const uint32_t local = id - base;
                t.m0 = s_off[e] + (local % mt) * TM;
                t.n0 = local / mt;
                t.m_end = s_off[e + 1];
                t.expert = p.expert_mod ? e % p.expert_mod : e;   // index of the B matrix
                t.valid = true;
                break;
            }
            base += cnt;
        }
    }
    // The offsets come from shared memory, which the compiler must treat as lane-varying.  Every lane
    // of the (converged) calling warp holds the same values; taking them from lane 0 lets the TMA
    // coordinates live in uniform registers instead of being made uniform instruction by instruction
    // (that made the producer, not the tensor pipe, set the pace of the grouped GEMMs).
    t.m0 = __shfl_sync(0xffffffffu, t.m0, 0);
    t.n0 = __shfl_sync(0xffffffffu, t.n0, 0);
    t.m_end = __shfl_sync(0xffffffffu, t.m_end, 0);
    t.expert = __shfl_sync(0xffffffffu, t.expert, 0);
    t.mt_index = __shfl_sync(0xffffffffu, t.mt_index, 0);
    t.valid = __shfl_sync(0xffffffffu, (uint32_t)t.valid, 0) != 0;
    return t;
}

// Reads a table of n + 1 <= 33 row offsets as a running maximum cut off at `limit`; true when that changed an entry.
// One lane per entry: read one after the other they cost nine trips to L2 at the start of every grouped GEMM.
__device__ __forceinline__ bool load_table(uint32_t *dst, const uint32_t *src, uint32_t stride, uint32_t n, uint32_t limit,
                                           uint32_t lane) {
    const uint32_t raw = lane <= n ? __ldcg(src + lane * stride) : 0u;
    const uint32_t last = n == 32 ? __ldcg(src + 32u * stride) : 0u;   // the 33rd entry, in every lane
    uint32_t v = min(raw, limit);
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const uint32_t o = __shfl_up_sync(0xffffffffu, v, off);
        if ((int)lane >= off) v = max(v, o);
    }
    if (lane <= n) dst[lane] = v;
    bool changed = lane <= n && v != raw;
    if (n == 32) {
        const uint32_t top = max(min(last, limit), __shfl_sync(0xffffffffu, v, 31));
        if (lane == 31) dst[32] = top;
        changed = changed || top != last;
    }
    return __any_sync(0xffffffffu, changed) != 0;
}

// Four-row pieces of a 128-row tile at m0 that hold rows of its group.
__device__ __forceinline__ uint32_t gathered_quads(uint32_t m0, uint32_t m_end) {
    return m_end > m0 ? (min(m_end - m0, (uint32_t)BM) + 3) / 4 : 0u;
}

// ... and those that its four gather warps, which take them in turn, fetch: one each at least.
__device__ __forceinline__ uint32_t fetched_quads(uint32_t m0, uint32_t m_end) { return max(gathered_quads(m0, m_end), 4u); }

// Two f32 to packed bf16, round to nearest even (hardware conversion; lo in the lower half).
__device__ __forceinline__ uint32_t cvt_bf16x2(float lo, float hi) {
    uint32_t d;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
    return d;
}

// GELU(x) = x * (1 + erf(x / sqrt 2)) / 2 = max(x, 0) - |x| * Q(|x|), where Q(u) = erfc(u / sqrt 2) / 2 is the upper tail
// of the normal distribution.  log2 Q is smooth: a polynomial of degree 6 (fitted here by linear programming, the
// error of u * Q(u) with these coefficients at most 8.7e-8) and one exp2 give it, so a pair of values costs nine packed f32
// operations and two of the special function unit, which together bound the epilogue (Abramowitz & Stegun 7.1.26, used
// before, costs twelve and four; its error is 2.1e-7).  64 tokens of d 2048: the tail of the first GEMM 8 -> 4.7 us, the
// layer 77.5 -> 73.6.  At |x| = 10 the tail is below 2^-75 either way, and the clamp
// keeps the polynomial where it falls.
//   Four pairs go side by side: one after the other, the chain of dependent operations of each would set the pace.
template <int N>
__device__ __forceinline__ void gelu_pairs(const uint32_t *x, uint32_t *out) {   // 2 N f32 -> N pairs of bf16
    auto both = [](float v) { return pack_f32x2(v, v); };
    uint64_t u2[N], r2[N], q2[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {   // u = -|x|; r = max(x, 0), as (x + |x|) / 2 so that -Inf and NaN stay NaN
        const float lo = __uint_as_float(x[2 * i] | 0x80000000u), hi = __uint_as_float(x[2 * i + 1] | 0x80000000u);
        r2[i] = fma_f32x2(pack_f32x2(lo, hi), both(-0.5f), mul_f32x2(pack_f32x2(__uint_as_float(x[2 * i]), __uint_as_float(x[2 * i + 1])), both(0.5f)));
        u2[i] = pack_f32x2(fmaxf(lo, -10.0f), fmaxf(hi, -10.0f));
    }
    constexpr float c[7] = {-1.0f, 1.15114708f, -0.458915684f, 0.0532381899f, 0.00797746515f, 0.000739875041f, 2.99242899e-05f};
#pragma unroll
    for (int i = 0; i < N; ++i) q2[i] = fma_f32x2(u2[i], both(c[6]), both(c[5]));
#pragma unroll
    for (int k = 4; k >= 0; --k)
#pragma unroll
        for (int i = 0; i < N; ++i) q2[i] = fma_f32x2(q2[i], u2[i], both(c[k]));
#pragma unroll
    for (int i = 0; i < N; ++i) {
        float lo, hi;
        unpack_f32x2(q2[i], lo, hi);
        q2[i] = pack_f32x2(ex2_approx(lo), ex2_approx(hi));
    }
#pragma unroll
    for (int i = 0; i < N; ++i) {
        float lo, hi;
        unpack_f32x2(fma_f32x2(u2[i], q2[i], r2[i]), lo, hi);
        out[i] = cvt_bf16x2(lo, hi);
    }
}

// One 32 x 32 chunk of f32 output out of a warp's swizzled slice into C, VEC elements per access: 32 / VEC lanes
// cover a row's 128 bytes, so an instruction touches VEC whole row segments.  With one lane per row (each lane
// walking its own row) the alpha/beta form cost 32 sectors per 4-byte access: 1000 x 3001 x 1111 took 98.8 us
// for 22.5 (with 128 columns a tile; 16.5 now).
// `old` holds the chunk's old values for alpha/beta, from fetch_chunk with the same lane layout.
template <int VEC>
__device__ __forceinline__ void fetch_chunk(float (&old)[32], const float *chunk, uint32_t ldc, uint32_t rows, uint32_t cols, uint32_t lane) {
    constexpr uint32_t kLanes = 32 / VEC;        // lanes per row
    const uint32_t sub = lane / kLanes, c = (lane % kLanes) * VEC;
#pragma unroll
    for (uint32_t i = 0; i < 32 / VEC; ++i) {
        const uint32_t rr = i * VEC + sub;
        const float *src = chunk + (uint64_t)rr * ldc + c;
        if (rr < rows && c < cols) {
            if constexpr (VEC == 4) {
                const float4 v = *reinterpret_cast<const float4 *>(src);
                old[4 * i] = v.x; old[4 * i + 1] = v.y; old[4 * i + 2] = v.z; old[4 * i + 3] = v.w;
            } else {
                old[i] = *src;
            }
        }
    }
}
template <int VEC, bool UPDATE>
__device__ __forceinline__ void write_chunk(float *chunk, uint32_t ldc, uint32_t rows, uint32_t cols, const uint8_t *slice,
                                            uint32_t lane, const GemmParams &p, const float (&old)[32]) {
    constexpr uint32_t kLanes = 32 / VEC;
    const uint32_t sub = lane / kLanes, c = (lane % kLanes) * VEC;
#pragma unroll
    for (uint32_t i = 0; i < 32 / VEC; ++i) {
        const uint32_t rr = i * VEC + sub;
        if (rr < rows && c < cols) {
            const uint8_t *at = slice + rr * 128 + (((c >> 2) ^ (rr & 7)) * 16) + (c & 3) * 4;
            float v[VEC];
            if constexpr (VEC == 4) {
                const float4 x = *reinterpret_cast<const float4 *>(at);
                v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
            } else {
                v[0] = *reinterpret_cast<const float *>(at);
            }
            if constexpr (UPDATE) {
#pragma unroll
                for (int q = 0; q < VEC; ++q) v[q] = __fadd_rn(__fmul_rn(p.alpha, v[q]), __fmul_rn(p.beta, old[VEC * i + q]));
            }
            float *dst = chunk + (uint64_t)rr * ldc + c;
            if constexpr (VEC == 4) *reinterpret_cast<float4 *>(dst) = make_float4(v[0], v[1], v[2], v[3]);
            else *dst = v[0];
        }
    }
}

// One step of a role along the ring: waits for the stage it is at, issues for it and, AHEAD, for all after it that are
// ready too.  Returns the k blocks issued, 0 when the wait ran out.  FENCE: what is issued reads or writes tensor memory.
// A wait, a vote and an election a stage take 350 to 450 cycles, as long as nothing hides them: the k block of a tile of
// 64 or 128 columns is multiplied in 220 or 260, that of 256 columns in 512.  128 x 64 tiles: 0.236 -> 0.185 us a k block
// (1024^3: 8.20 -> 7.45 us, 512^3: 5.94 -> 5.63); tiles of 256 columns lost 0.03 us a k block to the second look.
template <int STAGES, bool AHEAD, bool FENCE = false, typename F>
__device__ __forceinline__ uint32_t walk_ring(uint64_t *bars, uint32_t &stage, uint32_t &phase, uint32_t flip, uint32_t kb, uint32_t num_kb,
                                              uint32_t lane, const volatile int *abort, F issue) {
    uint32_t n = AHEAD ? ready_stages<STAGES>(bars, stage, phase ^ flip, num_kb - kb, lane) : 0u;
    if (n == 0) {
        if (!mbar_wait_warp(&bars[stage], phase ^ flip, abort)) return 0;
        n = 1;
    }
    if (FENCE) tc_fence_after();
    if (elect_one()) {
        if constexpr (AHEAD) {
            uint32_t st = stage;
#pragma unroll 1
            for (uint32_t i = 0; i < n; ++i) {
                issue(i, kb + i, st);
                if (++st == STAGES) st = 0;
            }
        } else {
            issue(0u, kb, stage);
        }
    }
    __syncwarp();
    stage += n;
    if (stage >= STAGES) { stage -= STAGES; phase ^= 1; }
    return n;
}

// REGS = 168 is what the block's 320 threads can have; REGS = 128 (no spills) is for the GEMM that runs
// beside the expert-parallel dispatch kernel: registers are handed out to four warps at a time, so the ten
// warps count as twelve, and 12 x 32 x 128 leaves room for one block of that kernel on the same SM.  It and the
// build with loader warps (a gathered A) run the first GEMM of an expert FFN only, so REGS = 128 has no f32 output.
template <int BN, int REGS, int CG, int KIND>
__global__ void __maxnreg__(REGS)
gemm_tc_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
               const __grid_constant__ CUtensorMap tmC, GemmParams p) {
    using L = SmemLayout<BN, CG>;
    // what this kind of launch does not have is known here
    const GemmEp ep = is_peer(KIND) ? p.ep : GemmEp{};
    const uint32_t experts = is_grouped(KIND) ? p.experts : 0u;
    const uint32_t epilogue = KIND == kPlain ? EPI_STORE : KIND == kUpdate ? EPI_ALPHA_BETA : is_gelu(KIND) ? EPI_GELU_BF16 : KIND == kPeer ? EPI_SCATTER_PEER : p.epilogue;
    const uint32_t *const gather_perm = KIND == kGroupedGelu ? p.gather_perm : nullptr;
    constexpr int kStages = L::kStages;
    constexpr bool kAhead = BN < 256;   // roles issue for every stage that is ready (walk_ring)
    extern __shared__ uint8_t smem_raw[];
    // 128-byte swizzle atoms are 1 KiB: align the tile region.
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + L::kBarOffset);
    uint64_t *empty = full + kStages;
    uint64_t *tmem_full = empty + kStages;
    uint64_t *tmem_empty = tmem_full + 2;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(tmem_empty + 2);
    __shared__ uint32_t s_off[33];             // row segments of the groups
    __shared__ uint32_t s_pair[33];            // expert-parallel: rows of (local expert, source) pairs
    __shared__ unsigned long long s_peer[32];  // expert-parallel: return buffer of every rank
    __shared__ int s_abort;

    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t n_tiles = (p.N + BN - 1) / BN;
    const uint32_t num_kb = (p.K + BK - 1) / BK;
    // this block's place in its pair, and the tiles it walks (both blocks of a pair walk the same ones)
    const uint32_t crank = CG == 2 ? cluster_rank() : 0u;
    const uint32_t first_tile = blockIdx.x / CG, tile_step = gridDim.x / CG;
    // the second GEMM of the expert FFN may take over each SM as this kernel's CTA leaves it
    if (ep.progress_mode == 1) launch_dependents();

    if (threadIdx.x == 0) {
        // Expert-parallel passes chain kernels through flags on other ranks: once a kernel of the pass has
        // reported a fault (a wait that ran out, a bad table), the later ones must not publish anything.
        // They find the status word set and do nothing but their arrival counting.
        s_abort = (ep.pair_offsets && p.status && __ldcg(p.status) != 0u) ? 1 : 0;
        for (int i = 0; i < kStages; ++i) {
            mbar_init(&full[i], 1);   // the producer's expect-tx arrival; in a pair rank 0's barrier counts both blocks' bytes
            mbar_init(&empty[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&tmem_full[i], 1);
            mbar_init(&tmem_empty[i], kEpilogueWarps * CG);
        }
        mbar_fence_init();
    }
    __shared__ int s_table_bad;
    const uint32_t ep_epoch = ep.epoch_counter ? __ldcg(ep.epoch_counter) + 1u : ep.epoch;
    // hand-over counters: two sets used by alternate passes; this pass's set was cleared during the previous one
    uint32_t *const progress = ep.progress ? ep.progress + (ep_epoch & 1u) * ep.progress_len : nullptr;
    // A launch that starts early (programmatic stream serialization) touches nothing of the kernels before it until
    // they have completed; only then may the next one start early, so that what lies two launches back is complete.
    // The second GEMM of a pair launched together (kEarlyWeights) does read its weights and the segment table ahead:
    // the GEMM just before it writes neither, and everything before that one is complete.
    const bool early = is_grouped(KIND) && p.after_previous == kEarlyWeights;
    if (experts && warp == 2) {
        // The dispatch kernel that writes the table may still be running beside this kernel: wait for its
        // "table written" flag before reading (bounded like every wait).
        if (p.after_previous && !early) grid_dependency_wait();
        const bool here = !ep.table_flag || flag_wait(ep.table_flag, ep_epoch, ep.spin_limit);
        if (!__all_sync(0xffffffffu, here) && lane == 0) kstatus_set(p.status, FE2O3_KSTATUS_WAIT_EXPIRED);
        if (lane == 0) s_table_bad = !here;
#ifdef FE2O3_EP_TRACE
        if (lane == 0 && ep.trace_flags && ep.table_flag && ep.progress_mode != 2 && blockIdx.x == 0) ep_trace(ep.trace_flags, FE2O3_EP_T_FFN1_TABLE_HERE);
#endif
        // The segment table is device data (in the expert-parallel layer it derives from other ranks'
        // counts): it is made monotone and cut off at M here, so that no row index derived from it can
        // leave A or C, and the fault is reported instead.
        if (load_table(s_off, p.expert_offsets, ep.pair_offsets ? ep.world : 1u, experts, p.M, lane) && lane == 0)
            kstatus_set(p.status, FE2O3_KSTATUS_SLOT_RANGE);
        if (ep.pair_offsets) load_table(s_pair, ep.pair_offsets, 1u, experts * ep.world, p.M, lane);   // at most 32 pairs
    }
    if (ep.peer_ret)
        for (uint32_t i = threadIdx.x; i < ep.world; i += blockDim.x) s_peer[i] = ep.peer_ret[i];
#ifdef FE2O3_EP_TRACE
    if (ep.trace_flags && blockIdx.x == 0 && threadIdx.x == 0)
        ep_trace(ep.trace_flags, ep.rows_flags ? FE2O3_EP_T_FFN1_BEGIN : FE2O3_EP_T_FFN2_BEGIN);
#endif
    if (warp == 1) {
        if constexpr (CG == 2) {
            tmem_alloc_pair(tmem_slot, L::kTmemCols);
            tmem_relinquish_pair();
        } else {
            tmem_alloc(tmem_slot, L::kTmemCols);
            tmem_relinquish();
        }
    }
    tc_fence_before();
    __syncthreads();
    if constexpr (CG == 2) cluster_sync();   // the other block's barriers are initialised
    tc_fence_after();
    if (p.after_previous && !(early && warp == 0)) {
        grid_dependency_wait();
        launch_dependents();
    }
    const uint32_t tmem_base = *tmem_slot;
    // A role that gives up ends the other roles' waits too, in both blocks of a pair.
    auto give_up = [&] {
        kstatus_set(p.status, FE2O3_KSTATUS_WAIT_EXPIRED);
        atomicExch(&s_abort, 1);
        if constexpr (CG == 2) st_shared_cluster(cluster_addr(&s_abort, crank ^ 1u), 1u);
    };
    const bool dead = s_abort != 0 || (experts && s_table_bad);   // uniform over the CTA: read after the barrier, before any role can set it

    if (warp == 0) {
        // ------------------------------------------------ TMA producer (warp converged, one elected lane issues)
        if (elect_one()) {
            tma_prefetch_desc(&tmA);
            tma_prefetch_desc(&tmB);
        }
        __syncwarp();
        uint32_t stage = 0, phase = 0, loaded = 0;
        uint32_t primed = 0; // k blocks of the first tile whose weights were fetched ahead of the wait
        uint32_t seen = 0;   // sources whose "rows complete" flag this CTA has already acquired
        bool ok = !dead;
        for (uint32_t id = first_tile; ok; id += tile_step) {
            TileCoord t = decode_tile<BM * CG, KIND>(id, p, n_tiles, s_off, s_pair);
            if (!t.valid) break;
            if constexpr (CG == 2) t.m0 += crank * BM;   // this block's rows of the pair's tile
            if (ep.rows_flags) {
                // Sources with rows in this tile.  Their rows were written by the source ranks' SMs
                // (generic proxy, then a system-scope release of the flag); this warp acquires the flag
                // and orders that observation before its bulk tensor loads (asynchronous proxy) with a
                // proxy fence.
                const uint32_t hi = min(t.m0 + BM, t.m_end);
                uint32_t need = 0;
                if (lane < experts * ep.world && s_pair[lane] < hi && s_pair[lane + 1] > t.m0)
                    need = 1u << (lane % ep.world);
                need = __reduce_or_sync(0xffffffffu, need) & ~seen;
                seen |= need;
                while (need) {   // bit k = run k of a segment = source (rank + k) mod W
                    const uint32_t src = (ep.rank + __ffs(need) - 1) % ep.world;
                    need &= need - 1;
                    if (!__all_sync(0xffffffffu, flag_wait(ep.rows_flags + src, ep_epoch, ep.spin_limit))) { ok = false; break; }
                }
                if (!ok) break;
                fence_proxy_async_global();
#ifdef FE2O3_EP_TRACE
                if (blockIdx.x == 0 && lane == 0 && ep.trace_flags) {
                    if (id == first_tile) ep_trace(ep.trace_flags, FE2O3_EP_T_FFN1_FIRST_WAIT_DONE);
                    if (seen == (1u << ep.world) - 1u) ep_trace(ep.trace_flags, FE2O3_EP_T_FFN1_LAST_WAIT_DONE);
                }
#endif
            }
            if (ep.progress_mode == 2) {
                // The rows of this tile are the first GEMM's output, stored by the copy engine (asynchronous
                // proxy) and announced through a counter: acquire the count, then order it before the bulk
                // tensor loads below.
                if (t.mt_index >= ep.progress_len ||
                    !__all_sync(0xffffffffu, flag_wait(progress + t.mt_index, ep.progress_target, ep.spin_limit))) {
                    ok = false;
                    break;
                }
                fence_proxy_async_global();
            }
            // bytes of a k block that rank 0's (or the only) barrier counts: of A only what holds rows of the group
            uint32_t bytes = CG * L::kStageBytes;
            if (gather_perm) {
                bytes = CG * L::kBBytes + fetched_quads(t.m0, t.m_end) * 512u;
                if (CG == 2) bytes += fetched_quads(t.m0 + BM, t.m_end) * 512u;   // (rank 1's rows; only rank 0 uses this)
            } else if (CG == 1 && p.a_box_rows < (uint32_t)BM) {
                bytes = L::kBBytes + (gathered_quads(t.m0, t.m_end) * 4 + p.a_box_rows - 1) / p.a_box_rows * p.a_box_rows * 128u;
            }
            auto load_a = [&](uint32_t kb, uint32_t st) {   // one lane
                uint8_t *sa = smem + st * L::kStageBytes;
                const int32_t x = (int32_t)(kb * BK);
                if constexpr (CG == 2) {
                    tma_load_2d_pair(sa, &tmA, cluster_addr(&full[st], 0), x, (int32_t)t.m0);
                } else {
                    tma_load_2d(sa, &tmA, &full[st], x, (int32_t)t.m0);
                    for (uint32_t r = p.a_box_rows; r < (uint32_t)BM && t.m0 + r < t.m_end; r += p.a_box_rows)
                        tma_load_2d(sa + r * 128, &tmA, &full[st], x, (int32_t)(t.m0 + r));
                }
            };
            auto load_b = [&](uint32_t kb, uint32_t st) {   // one lane; sets the expectation first
                uint8_t *sb = smem + st * L::kStageBytes + L::kABytes;
                if constexpr (CG == 2) {
                    // both blocks' bytes are counted by rank 0's barrier; rank 1's may arrive before the
                    // expectation is set, which the barrier's pending arrival makes harmless
                    const uint32_t bar = cluster_addr(&full[st], 0);
                    if (crank == 0) mbar_arrive_expect_tx(&full[st], bytes);
#pragma unroll
                    for (int j = 0; j < BN / CG / 64; ++j) {
                        const int32_t col = (int32_t)(t.n0 * BN + crank * (BN / CG) + j * 64);
                        if (experts) tma_load_3d_pair(sb + j * 8192, &tmB, bar, col, (int32_t)(kb * BK), (int32_t)t.expert);
                        else tma_load_2d_pair(sb + j * 8192, &tmB, bar, col, (int32_t)(kb * BK));
                    }
                } else {
                    mbar_arrive_expect_tx(&full[st], bytes);
#pragma unroll
                    for (int j = 0; j < BN / 64; ++j) {
                        const int32_t col = (int32_t)(t.n0 * BN + j * 64);
                        if (experts) tma_load_3d(sb + j * 8192, &tmB, &full[st], col, (int32_t)(kb * BK), (int32_t)t.expert);
                        else tma_load_2d(sb + j * 8192, &tmB, &full[st], col, (int32_t)(kb * BK));
                    }
                }
            };
            if (early && id == first_tile) {   // the whole ring is free: its weights first, then the rows once they are there
                primed = min((uint32_t)kStages, num_kb);
                if (elect_one())
                    for (uint32_t kb = 0; kb < primed; ++kb) load_b(kb, kb);
                __syncwarp();
                grid_dependency_wait();
            }
            auto load = [&](uint32_t i, uint32_t kb, uint32_t st) {
                if (loaded + i >= primed) load_b(kb, st);
                if (!gather_perm) load_a(kb, st);
            };
            for (uint32_t kb = 0; kb < num_kb;) {
                const uint32_t n = walk_ring<kStages, kAhead>(empty, stage, phase, 1, kb, num_kb, lane, &s_abort, load);
                if (n == 0) { ok = false; break; }
                kb += n;
                loaded += n;
            }
        }
        if (!ok && lane == 0) give_up();
        if (early && primed == 0) grid_dependency_wait();
        // Drain: every copy issued must have landed before the CTA exits (the newest phase of each ring slot).
        // Rank 1's copies are counted by rank 0's barriers, and no block of a pair leaves before the other.
        for (uint32_t b = 0; crank == 0 && b < kStages && b < loaded; ++b) {
            const uint32_t last = loaded - 1 - b;
            mbar_wait_warp(&full[last % kStages], (last / kStages) & 1);
        }
    } else if (warp == 1) {
        // ------------------------------------------------ MMA issuer (warp converged, one elected lane issues; rank 0 of a pair)
        constexpr uint32_t idesc = umma_idesc(1u, BM * CG, BN, 0u, 1u);
        uint32_t stage = 0, phase = 0, it = 0;
        bool ok = !dead && crank == 0;
        const uint64_t desc_a0 = umma_smem_desc(smem_u32(smem), 16, 1024);
        const uint64_t desc_b0 = umma_smem_desc(smem_u32(smem) + L::kABytes, 8192, 1024);
        for (uint32_t id = first_tile; ok; id += tile_step, ++it) {
            TileCoord t = decode_tile<BM * CG, KIND>(id, p, n_tiles, s_off, s_pair);
            if (!t.valid) break;
            if constexpr (CG == 2) t.m0 += crank * BM;   // this block's rows of the pair's tile
            const uint32_t buf = it & 1, acc_phase = (it >> 1) & 1;
            if (!mbar_wait_warp(&tmem_empty[buf], acc_phase ^ 1, &s_abort)) { ok = false; break; }
            tc_fence_after();
            const uint32_t d_tmem = tmem_base + buf * BN;
            auto multiply = [&](uint32_t, uint32_t kb, uint32_t st) {
                // only the 16-byte-unit start address field of the descriptors moves
                const uint64_t adesc = desc_a0 + ((st * L::kStageBytes) >> 4);
                const uint64_t bdesc = desc_b0 + ((st * L::kStageBytes) >> 4);
                // A: K-major, advance 16 elements = 32 bytes inside the 128-byte row
                // B: MN-major, advance 16 k-rows = 2 KiB; 64-column groups are 8 KiB apart
                if constexpr (CG == 2) {
#pragma unroll
                    for (int k = 0; k < BK / UMMA_K; ++k)
                        umma_f16_pair(d_tmem, adesc + ((k * UMMA_K * 2) >> 4), bdesc + ((k * UMMA_K * 128) >> 4), idesc,
                                      (uint32_t)(k != 0) | (uint32_t)(kb != 0u));
                    umma_commit_pair(&empty[st]);
                    if (kb + 1 == num_kb) umma_commit_pair(&tmem_full[buf]);
                } else {
                    umma_f16(d_tmem, adesc, bdesc, idesc, kb != 0u);
#pragma unroll
                    for (int k = 1; k < BK / UMMA_K; ++k)
                        umma_f16(d_tmem, adesc + ((k * UMMA_K * 2) >> 4), bdesc + ((k * UMMA_K * 128) >> 4), idesc, 1u);
                    umma_commit(&empty[st]);
                    if (kb + 1 == num_kb) umma_commit(&tmem_full[buf]);
                }
            };
            for (uint32_t kb = 0; kb < num_kb;) {
                const uint32_t n = walk_ring<kStages, kAhead, true>(full, stage, phase, 0, kb, num_kb, lane, &s_abort, multiply);
                if (n == 0) { ok = false; break; }
                kb += n;
            }
        }
        if (!ok && crank == 0 && lane == 0) give_up();
    } else if (warp >= 2 + kEpilogueWarps) {
        // ------------------------------------------------ gather issuers (blocks launched with them only)
        // Four warps fetch the tile's rows in turn, four rows an instruction, by the copy engine: the rows' token
        // numbers sit in registers for the whole tile.  A slot without a route names the row after the last token,
        // which the copy engine fills with zeros; whole quads past the group's end are not fetched (what they leave in
        // the stage only reaches rows of the accumulator that nobody stores).  Every warp fetches one quad of each k block
        // at least: if nothing of a stage waited for it, the ring could run on while it still waits for an earlier
        // phase, whose parity would then have come and gone.
        const uint32_t gw = warp - (2 + kEpilogueWarps);   // quads gw, gw + 4, ...
        uint32_t stage = 0, phase = 0;
        bool ok = !dead;
        for (uint32_t id = first_tile; ok; id += tile_step) {
            TileCoord t = decode_tile<BM * CG, KIND>(id, p, n_tiles, s_off, s_pair);
            if (!t.valid) break;
            if constexpr (CG == 2) t.m0 += crank * BM;
            const uint32_t quads = (fetched_quads(t.m0, t.m_end) + 3 - gw) / 4;   // this warp's: 1 to 8
            const uint32_t row = t.m0 + ((lane >> 2) * 4 + gw) * 4 + (lane & 3);
            const uint32_t route = row < t.m_end ? __ldg(gather_perm + row) : 0xffffffffu;
            const uint32_t mine = route == 0xffffffffu ? p.gather_tokens : min(route >> 1, p.gather_tokens);
            int32_t tok[32];
#pragma unroll
            for (int i = 0; i < 32; ++i) tok[i] = (int32_t)__shfl_sync(0xffffffffu, mine, i);
            auto gather = [&](uint32_t, uint32_t kb, uint32_t st) {
                uint8_t *sa = smem + st * L::kStageBytes + gw * 512;
                const uint32_t bar = CG == 2 ? cluster_addr(&full[st], 0) : smem_u32(&full[st]);
                auto fetch = [&](int i) {
                    tma_gather4<CG == 2>(sa + i * 2048, &tmA, bar, (int32_t)(kb * BK), tok[4 * i], tok[4 * i + 1], tok[4 * i + 2],
                                         tok[4 * i + 3]);
                };
                if (quads >= 8) {
#pragma unroll
                    for (int i = 0; i < 8; ++i) fetch(i);
                } else {
#pragma unroll
                    for (int i = 0; i < 7; ++i)
                        if (i == 0 || i < (int)quads) fetch(i);
                }
            };
            for (uint32_t kb = 0; kb < num_kb;) {
                const uint32_t n = walk_ring<kStages, kAhead>(empty, stage, phase, 1, kb, num_kb, lane, &s_abort, gather);
                if (n == 0) { ok = false; break; }
                kb += n;
            }
        }
        if (!ok && lane == 0) give_up();
    } else {
        // ------------------------------------------------ epilogue warps
        // Eight warps: two per TMEM lane quadrant, each taking half of the tile's columns.  A warp
        // turns 128 bytes of each of its 32 rows at a time (32 f32 or 64 bf16 columns) into a
        // 128-byte-swizzled 4 KiB slice of shared memory and hands it to the copy engine, so the
        // global writes are full lines and do not hold the warp; ragged rows and outputs the copy engine cannot
        // address are written by the threads directly, and so is the alpha/beta form, in a branch of its own.
        const uint32_t ew = warp - 2;
        const uint32_t quad = warp & 3;  // TMEM lane quadrant this warp may read
        const uint32_t col_half = ew >> 2;
        constexpr int kChunks = BN / 32 / 2;   // 32-column chunks per warp
        uint8_t *slice = smem + L::kStagingOffset + ew * 4096;
        uint32_t it = 0;
        bool ok = !dead;
        bool store_pending = false;
        auto release_accumulator = [&](uint32_t buf) {   // the issuer of a pair is rank 0
            if constexpr (CG == 2) mbar_arrive_cluster(cluster_addr(&tmem_empty[buf], 0));
            else mbar_arrive(&tmem_empty[buf]);
        };
        if (KIND == kGroupedGelu && p.zero_ptr && !dead) {
            const uint64_t stride = (uint64_t)gridDim.x * (kEpilogueWarps * 32);
            for (uint64_t i = (uint64_t)blockIdx.x * (kEpilogueWarps * 32) + ew * 32 + lane; i < p.zero_vecs; i += stride)
                p.zero_ptr[i] = make_uint4(0u, 0u, 0u, 0u);
        }
        for (uint32_t id = first_tile; ok; id += tile_step, ++it) {
            TileCoord t = decode_tile<BM * CG, KIND>(id, p, n_tiles, s_off, s_pair);
            if (!t.valid) break;
            if constexpr (CG == 2) t.m0 += crank * BM;   // this block's rows of the pair's tile
            const uint32_t buf = it & 1, acc_phase = (it >> 1) & 1;
            const uint32_t row0 = t.m0 + quad * 32;
            const uint32_t row = row0 + lane;
            const bool row_ok = row < t.m_end;
            const bool bulk = p.bulk_store && row0 + 32 <= t.m_end;   // warp-uniform
            const uint32_t col_base = t.n0 * BN + col_half * (BN / 2);
            // alpha/beta: the old values of C, those of the first 32 columns while the tile is being multiplied; the rest of them
            // come into L2 meanwhile
            const uint32_t rows_here = min(32u, t.m_end > row0 ? t.m_end - row0 : 0u);
            float *const c0 = reinterpret_cast<float *>(p.c) + (uint64_t)row0 * p.ldc;
            const bool vec = p.ldc % 4u == 0 && (reinterpret_cast<uintptr_t>(p.c) & 15u) == 0;
            auto fetch = [&](float (&to)[32], uint32_t col) {
                if (col >= p.N) return;
                if (vec && col + 32 <= p.N) fetch_chunk<4>(to, c0 + col, p.ldc, rows_here, 32, lane);
                else fetch_chunk<1>(to, c0 + col, p.ldc, rows_here, min(32u, p.N - col), lane);
            };
            float old[32];
            if constexpr (KIND == kUpdate) {
                fetch(old, col_base);
#pragma unroll
                for (uint32_t g = 1; g < kChunks; ++g)
                    if (row_ok && col_base + g * 32 < p.N) asm volatile("prefetch.global.L2 [%0];" ::"l"(c0 + (uint64_t)lane * p.ldc + col_base + g * 32));
            }
            if (!mbar_wait_warp(&tmem_full[buf], acc_phase, &s_abort)) { ok = false; break; }
            tc_fence_after();
            const uint32_t taddr = tmem_base + buf * BN + col_half * (BN / 2) + ((quad * 32u) << 16);
            // scatter epilogue: where this lane's row goes (0 = nowhere)
            unsigned long long dst_row = 0;
            if (epilogue == EPI_SCATTER_PEER && row_ok) {
                const uint2 meta = __ldcg(ep.row_meta + row);   // (route id, home rank), written by the source rank
                if (meta.y < ep.world && meta.x < ep.ret_rows)
                    dst_row = s_peer[meta.y] + (unsigned long long)meta.x * p.N * sizeof(float);
                else
                    kstatus_set(p.status, FE2O3_KSTATUS_SLOT_RANGE);
            }
            float row_weight = 0.0f;
            if (epilogue == EPI_COMBINE_ADD && row_ok) {
                // where this lane's row is added and with which weight: route id of the slot, the token's two
                // weights checked like the separate combine does (finite, non-negative, summing to exactly 1)
                const uint32_t route = __ldg(p.combine_perm + row);
                if (route != 0xffffffffu && (route >> 1) < p.combine_tokens) {
                    const float w0 = __ldg(p.combine_weights + (route & ~1u)), w1 = __ldg(p.combine_weights + (route | 1u));
                    if (!isfinite(w0) || !isfinite(w1) || w0 < 0.f || w1 < 0.f || __fadd_rn(w0, w1) != 1.0f) {
                        kstatus_set(p.status, FE2O3_KSTATUS_WEIGHTS);
                    } else {
                        dst_row = reinterpret_cast<unsigned long long>(p.c) + (unsigned long long)(route >> 1) * p.N * sizeof(float);
                        row_weight = (route & 1u) ? w1 : w0;
                    }
                }
            }
            if (is_grouped(KIND) && row0 >= t.m_end) {   // none of this warp's rows belong to the group
                tc_fence_before();
                __syncwarp();
                if (lane == 0) release_accumulator(buf);
            } else if constexpr (is_gelu(KIND)) {
                // ---- GELU, bf16 output: 64 columns to a 128-byte group, 16 at a time.  The loops stay rolled: a block of a
                // small batch runs this code once, and waits for its instructions (unrolled: 2 us more a pass of 64 tokens).
                // The next 16 columns are on their way meanwhile, and are there before the loop goes back: registers that a
                // load has yet to fill may not be copied from.
                uint32_t x[16];
                tmem_ld_32x32b_x16(taddr, x);
                tmem_ld_wait_for(x);
#pragma unroll 1
                for (int q = 0; q < BN / 32; ++q) {
                    const uint32_t at = (q & 3) * 2;   // 16-byte pieces of the group
                    const bool more = q + 1 < BN / 32;
                    uint32_t next[16], w[8];
                    if (more) {
                        tmem_ld_32x32b_x16(taddr + (q + 1) * 16, next);
                    } else {   // the accumulator has been read completely
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) release_accumulator(buf);
                    }
                    gelu_pairs<4>(x, w);
                    gelu_pairs<4>(x + 8, w + 4);
                    if (more) {
                        tmem_ld_wait_for(next);
#pragma unroll
                        for (int i = 0; i < 16; ++i) x[i] = next[i];
                    }
                    if (at == 0) {   // the slice has been read out
                        if (store_pending && lane == 0) tma_store_wait_read();
                        __syncwarp();
                    }
                    *reinterpret_cast<uint4 *>(slice + lane * 128 + ((at ^ (lane & 7)) * 16)) = make_uint4(w[0], w[1], w[2], w[3]);
                    *reinterpret_cast<uint4 *>(slice + lane * 128 + (((at + 1) ^ (lane & 7)) * 16)) = make_uint4(w[4], w[5], w[6], w[7]);
                    const uint32_t col = col_base + (q & ~3) * 16;
                    if (at != 6 || col >= p.N) continue;
                    store_pending = bulk;
                    if (bulk) {
                        fence_proxy_async_smem();
                        __syncwarp();
                        if (lane == 0) {
                            tma_store_2d(&tmC, slice, (int32_t)col, (int32_t)row0);
                            tma_store_commit();
                        }
                    } else {   // whole row segments, eight lanes to a row
                        __syncwarp();
                        const uint32_t piece = lane & 7;
#pragma unroll 1
                        for (uint32_t rr = lane >> 3; rr < min(32u, t.m_end - row0); rr += 4) {
                            const uint4 v = *reinterpret_cast<const uint4 *>(slice + rr * 128 + ((piece ^ (rr & 7)) * 16));
                            uint16_t *dst = reinterpret_cast<uint16_t *>(p.c) + (uint64_t)(row0 + rr) * p.ldc + col + piece * 8;
                            if (col + 64 <= p.N && ((reinterpret_cast<uintptr_t>(dst) & 15u) == 0)) {
                                *reinterpret_cast<uint4 *>(dst) = v;
                            } else {
                                const uint32_t e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                                for (int j = 0; j < 8; ++j)
                                    if (col + piece * 8 + j < p.N) dst[j] = (uint16_t)(e[j >> 1] >> ((j & 1) * 16));
                            }
                        }
                    }
                }
            } else if constexpr (KIND == kUpdate) {
                // ---- alpha/beta.  A chunk's old values are asked for as soon as those before them have been used, into the same
                // registers: a second set, copied at the end of each turn, made every turn wait for its own loads (3000 x 2900 x 130
                // with an odd pitch 28.1 us for 25.1).
#pragma unroll 1
                for (int g = 0; g < kChunks; ++g) {
                    const uint32_t col = col_base + g * 32;
                    uint32_t r[32];
                    tmem_ld_32x32b_x32(taddr + g * 32, r);
                    tmem_ld_wait();
                    if (g == kChunks - 1) {   // the accumulator has been read completely
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) release_accumulator(buf);
                    }
                    if (col >= p.N) continue;
                    __syncwarp();   // the previous chunk has been read out of the slice
#pragma unroll
                    for (int k = 0; k < 8; ++k)
                        *reinterpret_cast<uint4 *>(slice + lane * 128 + ((k ^ (lane & 7)) * 16)) =
                            make_uint4(r[4 * k], r[4 * k + 1], r[4 * k + 2], r[4 * k + 3]);
                    __syncwarp();
                    if (vec && col + 32 <= p.N) write_chunk<4, true>(c0 + col, p.ldc, rows_here, 32, slice, lane, p, old);
                    else write_chunk<1, true>(c0 + col, p.ldc, rows_here, min(32u, p.N - col), slice, lane, p, old);
                    if (g + 1 < kChunks) fetch(old, col + 32);
                }
            } else {
                // ---- f32 output: one chunk (32 columns) per 128-byte group
#pragma unroll 1
                for (int g = 0; g < kChunks; ++g) {
                    uint32_t r[32];
                    tmem_ld_32x32b_x32(taddr + g * 32, r);
                    tmem_ld_wait();
                    if (g == kChunks - 1) {   // the accumulator has been read completely
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) release_accumulator(buf);
                    }
                    const uint32_t col = col_base + g * 32;
                    if (col >= p.N) continue;
                    if (epilogue == EPI_SCATTER_PEER || epilogue == EPI_COMBINE_ADD) {
                        // Every row of the tile has its own destination (the return buffer of its home
                        // rank, at its route id).  The chunk is transposed through the warp's slice of
                        // shared memory so that each store instruction writes four whole 128-byte
                        // segments: eight lanes per row, one 16-byte piece each.
                        __syncwarp();   // the previous chunk has been read out of the slice
#pragma unroll
                        for (int k = 0; k < 8; ++k)
                            *reinterpret_cast<uint4 *>(slice + lane * 128 + ((k ^ (lane & 7)) * 16)) =
                                make_uint4(r[4 * k], r[4 * k + 1], r[4 * k + 2], r[4 * k + 3]);
                        __syncwarp();
                        const uint32_t piece = lane & 7;
#pragma unroll
                        for (int it = 0; it < 8; ++it) {
                            const uint32_t rr = it * 4 + (lane >> 3);
                            const uint4 v = *reinterpret_cast<const uint4 *>(slice + rr * 128 + ((piece ^ (rr & 7)) * 16));
                            const unsigned long long dst = __shfl_sync(0xffffffffu, dst_row, rr);
                            const float wgt = __shfl_sync(0xffffffffu, row_weight, rr);
                            if (dst != 0 && col + piece * 4 < p.N) {
                                const unsigned long long at = dst + (unsigned long long)(col + piece * 4) * sizeof(float);
                                if (epilogue == EPI_COMBINE_ADD)   // weight * row (one rounding), then one addition per element
                                    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(at),
                                                 "f"(__fmul_rn(wgt, __uint_as_float(v.x))), "f"(__fmul_rn(wgt, __uint_as_float(v.y))),
                                                 "f"(__fmul_rn(wgt, __uint_as_float(v.z))), "f"(__fmul_rn(wgt, __uint_as_float(v.w)))
                                                 : "memory");
                                else
                                    *reinterpret_cast<uint4 *>(at) = v;
                            }
                        }
                    } else if (bulk && epilogue == EPI_STORE) {
                        if (store_pending) {
                            if (lane == 0) tma_store_wait_read();
                            __syncwarp();
                        }
#pragma unroll
                        for (int k = 0; k < 8; ++k)
                            *reinterpret_cast<uint4 *>(slice + lane * 128 + ((k ^ (lane & 7)) * 16)) =
                                make_uint4(r[4 * k], r[4 * k + 1], r[4 * k + 2], r[4 * k + 3]);
                        fence_proxy_async_smem();
                        __syncwarp();
                        if (lane == 0) {
                            tma_store_2d(&tmC, slice, (int32_t)col, (int32_t)row0);
                            tma_store_commit();
                        }
                        store_pending = true;
                    } else {
                        // Rows the copy engine cannot take (a ragged group's last rows, C it cannot address): the chunk
                        // goes through the warp's slice of shared memory so that every access to C is a run of whole
                        // row segments.
                        if (store_pending) {
                            if (lane == 0) tma_store_wait_read();
                            store_pending = false;
                        }
                        __syncwarp();   // the previous chunk has been read out of the slice
#pragma unroll
                        for (int k = 0; k < 8; ++k)
                            *reinterpret_cast<uint4 *>(slice + lane * 128 + ((k ^ (lane & 7)) * 16)) =
                                make_uint4(r[4 * k], r[4 * k + 1], r[4 * k + 2], r[4 * k + 3]);
                        __syncwarp();
                        float *chunk = c0 + col;
                        const float none[32] = {};
                        if (vec && col + 32 <= p.N)
                            write_chunk<4, false>(chunk, p.ldc, rows_here, 32, slice, lane, p, none);
                        else
                            write_chunk<1, false>(chunk, p.ldc, rows_here, min(32u, p.N - col), slice, lane, p, none);
                    }
                }
            }
            if (ep.progress_mode == 1) {
                // this warp's part of the hidden rows of the tile is in memory: bulk stores complete (not merely
                // read out of shared memory), direct stores fenced; then one count per warp
                if (store_pending) {
                    if (lane == 0) tma_store_wait_all();
                    store_pending = false;
                }
                __threadfence();
                __syncwarp();
                fence_proxy_async_global();
                if (lane == 0 && t.mt_index < ep.progress_len) atomicAdd(progress + t.mt_index, 1u);
            }
        }
        // the staging slice must stay intact until the last copy has read it
        if (store_pending && lane == 0) tma_store_wait_read();
        // rows stored into other ranks' memory must be visible there before "outputs ready" is raised
        if (epilogue == EPI_SCATTER_PEER) __threadfence_system();
        if (!ok && lane == 0) give_up();
    }
    tc_fence_before();
    __syncthreads();
    // no block of a pair leaves while the other may still signal its barriers or read its shared memory
    if constexpr (CG == 2) cluster_sync();
    if (warp == 1) {
        tc_fence_after();
        if constexpr (CG == 2) tmem_dealloc_pair(tmem_base, L::kTmemCols);
        else tmem_dealloc(tmem_base, L::kTmemCols);
    }
#ifdef FE2O3_EP_TRACE
    if (ep.trace_flags && blockIdx.x == gridDim.x - 1 && threadIdx.x == 0)
        ep_trace(ep.trace_flags, ep.rows_flags ? FE2O3_EP_T_FFN1_END : FE2O3_EP_T_FFN2_END);
#endif
    if (ep.done_counter && threadIdx.x == 0) {
        // The last CTA of the grid to finish raises "outputs ready" on every rank, unless some CTA gave
        // up on a wait (the pass is void then).  A failed CTA still arrives, so the counter is re-armed.
        const bool failed = s_abort != 0;
        const uint32_t old = atomicAdd(ep.done_counter, failed ? 0x10001u : 1u);
        if ((old & 0xffffu) == gridDim.x - 1) {
            atomicExch(ep.done_counter, 0u);
            if (ep.progress_mode == 2)   // the other set of hand-over counters, for the next pass (nobody uses it during this one)
                for (uint32_t i = 0; i < ep.progress_len; ++i) ep.progress[((ep_epoch & 1u) ^ 1u) * ep.progress_len + i] = 0u;
            if (!failed && (old >> 16) == 0) {
                __threadfence_system();
                for (uint32_t w = 0; w < ep.world; ++w)
                    st_release_sys(reinterpret_cast<uint32_t *>(ep.peer_flags[w]) + FE2O3_EP_FLAG_OUTPUTS(ep.world) + ep.rank,
                                   ep_epoch);
            }
        }
    }
}

// ---- host side ------------------------------------------------------------------

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
    });
    return fn;
}

}  // namespace

// Encodes a tensor map with 128-byte swizzle.  dims/strides innermost first;
// strides in bytes for dimensions 1..rank-1.
static int32_t make_tmap(CUtensorMap *out, CUtensorMapDataType dtype, uint64_t base, uint32_t rank, const uint64_t *dims,
                         const uint64_t *strides_bytes, const uint32_t *box) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) {
        fe2o3_set_error("cuTensorMapEncodeTiled is not available from the driver");
        return FE2O3_ERR_NO_DEVICE;
    }
    cuuint64_t d[5];
    cuuint64_t st[4];
    cuuint32_t b[5], es[5];
    for (uint32_t i = 0; i < rank; ++i) { d[i] = dims[i]; b[i] = box[i]; es[i] = 1; }
    for (uint32_t i = 0; i + 1 < rank; ++i) st[i] = strides_bytes[i];
    CUresult r = fn(out, dtype, rank, reinterpret_cast<void *>(base), d, st, b, es,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        fe2o3_set_error("cuTensorMapEncodeTiled failed with CUresult %d", (int)r);
        return FE2O3_ERR_INVALID_ARGUMENT;
    }
    return FE2O3_OK;
}

int32_t fe2o3_make_tmap_bf16(CUtensorMap *out, uint64_t base, uint32_t rank, const uint64_t *dims,
                             const uint64_t *strides_bytes, const uint32_t *box) {
    return make_tmap(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, base, rank, dims, strides_bytes, box);
}
int32_t fe2o3_make_tmap_f32(CUtensorMap *out, uint64_t base, uint32_t rank, const uint64_t *dims,
                            const uint64_t *strides_bytes, const uint32_t *box) {
    return make_tmap(out, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, base, rank, dims, strides_bytes, box);
}

// The tensor-core schedule needs 16-byte aligned bases and leading dimensions
// that are multiples of 8 elements (TMA strides are multiples of 16 bytes).
bool gemm_tc_supported(uint64_t a, uint64_t b, uint32_t lda, uint32_t ldb, uint32_t K) {
    return K > 0 && (a & 15u) == 0 && (b & 15u) == 0 && (lda % 8u) == 0 && (ldb % 8u) == 0;
}

// experts == 0: plain C[M][N] = A[M][K] * B[K][N].  experts > 0: grouped, A rows
// partitioned by expert_offsets (device array), B = [experts][K][N], M = upper
// bound on rows (the capacity of A and C).
int32_t gemm_tc_plan(fe2o3_ctx *ctx, GemmTcPlan *plan, uint64_t a, uint64_t b, uint64_t c, uint32_t M, uint32_t N,
                     uint32_t K, uint32_t lda, uint32_t ldb, uint32_t ldc, float alpha, float beta, uint32_t epilogue,
                     const uint32_t *expert_offsets, uint32_t experts, uint32_t expert_mod, uint32_t b_matrices,
                     const GemmEp *ep) {
    plan->bn = N > 128 ? 256 : 128;
    plan->pair = 0;
    uint32_t a_box = BM;
    const uint64_t sms = ctx->sm_count, k_blocks = (K + BK - 1) / BK;
    if (!ep && !experts) {
        // Tile shape: the cheapest of what a launch costs by itself, its k blocks in every round of tiles, and what of
        // the output of a round the next one does not hide (alpha/beta reads C too).  Fitted to 90 products of up to
        // 8192 x 8192 x 8192, all five shapes each: the choice is within 0.1 % of the best on average, 1.5 % at worst.  A narrow
        // tile has the shortest launch and the dearest multiply-add, a pair of SMs the opposite: it stages a third less.
        // us, the same operands again and again, 64 / 128 / 192 / 256 columns / pair: 512^3 4.8 / 5.8 / 6.8 / 7.6 / 8.4; 1000 x 3001 x
        // 1111 alpha/beta, C's pitch 3004, 22.4 / 22.2 / 16.5 / 20.1 / 18.4 (pitch 3001: 22.6 / 23.5 / 18.8 / 22.8 / 20.8);
        // 3072 x 3072 x 1024 31.0 / 22.9 / 22.9 / 19.0 / 18.5.
        static const struct { uint32_t bn, pair, launch, k_block, output; } shapes[] = {   // ns
            {64, 0, 4380, 195, 1080}, {128, 0, 4800, 258, 1650}, {192, 0, 5440, 320, 2500}, {256, 0, 5200, 380, 3460}, {256, 1, 6900, 277, 3630}};
        uint64_t best = ~0ull;
        for (const auto &shape : shapes) {
            const uint64_t rows = shape.pair ? 2 * BM : BM, slots = shape.pair ? sms / 2 : sms;
            if (slots == 0) continue;
            const uint64_t tiles = ((M + rows - 1) / rows) * ((N + shape.bn - 1) / shape.bn), rounds = (tiles + slots - 1) / slots;
            const uint64_t product = k_blocks * shape.k_block, output = epilogue == EPI_ALPHA_BETA ? shape.output * 9 / 5 : shape.output;
            const uint64_t cost = shape.launch + rounds * product + (output > product && rounds > 1 ? (rounds - 1) * (output - product) : 0);
            if (cost < best) { best = cost; plan->bn = shape.bn; plan->pair = shape.pair; }
        }
        // Few rows: copies of A hold 32 or 64.  What a copy fills in beyond the last row delays the blocks that want the same few
        // rows of A (us, 128 / 32 or 64 rows a copy: 8 x 3707 x 2317 16.2 / 10.1, 16 x 5120 x 2304 17.0 / 9.3, 48 x 3707 x 2317 10.6 / 10.2).
        if (!plan->pair) a_box = M <= 32 ? 32 : M <= 64 ? 64 : BM;
    } else if (!ep) {
        // Groups: rounds of tiles times what a round takes, as 0.55 : 0.68 : 1 for 64, 128 and 256 columns; a group ends in
        // a partly filled tile, half of one on average.  256-row tiles on pairs of SMs shorten a round by about a tenth where
        // the k loop sets its length, but not where coarser tiles make more rounds (512 rows an expert, d 2048: 194
        // against 209 us a layer pass).
        // The expert-parallel GEMMs count finished 256-wide tiles and keep them: half-width ones re-read A twice as
        // often and were slower there on 4096 and 8192 rows (530 against 481 us and 686 against 590 us a pass).
        auto rounds = [&](uint64_t tile_rows, uint64_t tile_cols, uint64_t slots) {
            const uint64_t m_tiles = M <= experts * tile_rows / 2 ? experts : (2 * (uint64_t)M + experts * tile_rows) / (2 * tile_rows);
            return (m_tiles * ((N + tile_cols - 1) / tile_cols) + slots - 1) / slots;
        };
        uint64_t best = 100 * rounds(BM, 256, sms);
        plan->bn = 256;
        auto consider = [&](uint32_t bn, uint32_t pair, uint64_t cost) {
            if (cost < best) { best = cost; plan->bn = bn; plan->pair = pair; }
        };
        if (K > 1024 && N > 128 && sms >= 2) consider(256, 1, 90 * rounds(2 * BM, 256, sms / 2));
        consider(128, 0, 68 * rounds(BM, 128, sms));
        // (bf16 output leaves in pieces of 64 columns a warp, half a tile's columns)
        if (epilogue != EPI_GELU_BF16) consider(64, 0, 55 * rounds(BM, 64, sms));
        // A group's tile takes only the copies of A that hold its rows: of 32 rows up to 24 rows a group on average
        // (16 rows, d 2048: 96.5 -> 93.6 us a layer pass), of 64 up to 48; with more, one copy of the whole tile is
        // cheaper than several (64 rows a group: 98.2 against 96.3 us)
        if (!plan->pair) a_box = M <= 24 * experts ? 32 : M <= 48 * experts ? 64 : BM;
    }
    uint64_t dA[2] = {K, M}, sA[1] = {(uint64_t)lda * 2};
    uint32_t bA[2] = {BK, a_box};
    int32_t st = fe2o3_make_tmap_bf16(&plan->tmA, a, 2, dA, sA, bA);
    if (st != FE2O3_OK) return st;
    if (experts) {
        uint64_t dB[3] = {N, K, b_matrices ? b_matrices : experts}, sB[2] = {(uint64_t)ldb * 2, (uint64_t)ldb * 2 * K};
        uint32_t bB[3] = {64, BK, 1};
        st = fe2o3_make_tmap_bf16(&plan->tmB, b, 3, dB, sB, bB);
    } else {
        uint64_t dB[2] = {N, K}, sB[1] = {(uint64_t)ldb * 2};
        uint32_t bB[2] = {64, BK};
        st = fe2o3_make_tmap_bf16(&plan->tmB, b, 2, dB, sB, bB);
    }
    if (st != FE2O3_OK) return st;
    // Output through the copy engine when it can address C: 16-byte aligned base and row pitch.
    const uint32_t esize = epilogue == EPI_GELU_BF16 ? 2u : 4u;
    uint32_t bulk = 0;
    plan->tmC = plan->tmA;   // a valid map when the bulk path is off (never used then)
    if (epilogue != EPI_ALPHA_BETA && epilogue != EPI_SCATTER_PEER && epilogue != EPI_COMBINE_ADD && (c & 15u) == 0 && ((uint64_t)ldc * esize) % 16u == 0 &&
        M > 0 && N > 0) {
        uint64_t dC[2] = {N, M}, sC[1] = {(uint64_t)ldc * esize};
        uint32_t bC[2] = {128u / esize, 32};
        st = esize == 2 ? fe2o3_make_tmap_bf16(&plan->tmC, c, 2, dC, sC, bC) : fe2o3_make_tmap_f32(&plan->tmC, c, 2, dC, sC, bC);
        if (st != FE2O3_OK) return st;
        bulk = 1;
    }
    plan->p = GemmParams{reinterpret_cast<void *>(c), M, N, K, ldc, alpha, beta, epilogue, expert_offsets, experts,
                         expert_mod, bulk, ctx->status_word, ep ? *ep : GemmEp{}, nullptr, 0u, nullptr, nullptr, 0u, nullptr, 0ull, a_box, 0u};
    plan->p.after_previous = ep ? 0u : 1u;
    const uint32_t n_tiles = (N + plan->bn - 1) / plan->bn;
    const uint64_t tile_rows = plan->pair ? 2 * BM : BM;
    const uint64_t m_tiles = (M + tile_rows - 1) / tile_rows + experts;  // grouped: each expert may add a ragged tile
    const uint32_t group = plan->pair ? 2 : 1;   // blocks per tile
    const uint64_t tiles = m_tiles * n_tiles, slots = ctx->sm_count / group;
    plan->grid = group * (uint32_t)(tiles < slots ? (tiles ? tiles : 1) : slots);
    plan->smem = plan->pair ? SmemLayout<256, 2>::kTotal : plan->bn == 256 ? SmemLayout<256, 1>::kTotal : plan->bn == 192 ? SmemLayout<192, 1>::kTotal : plan->bn == 128 ? SmemLayout<128, 1>::kTotal : SmemLayout<64, 1>::kTotal;
    plan->overlap_previous = 0;
    return FE2O3_OK;
}

// The builds in use: every tile shape of a plain or alpha/beta product (192 columns there only), of the others what
// their plans choose.  REGS = 128: see the kernel.
template <typename F>
static void with_kernel(const GemmTcPlan *plan, F f) {
    const GemmParams &p = plan->p;
    if (p.experts == 0) {
#define FE2O3_SHAPES(KIND)                                                                                       \
        if (plan->pair) f(gemm_tc_kernel<256, 168, 2, KIND>);                                                     \
        else if (plan->bn == 256) f(gemm_tc_kernel<256, 168, 1, KIND>);                                           \
        else if (plan->bn == 192) f(gemm_tc_kernel<192, 168, 1, KIND>);                                           \
        else if (plan->bn == 128) f(gemm_tc_kernel<128, 168, 1, KIND>);                                           \
        else f(gemm_tc_kernel<64, 168, 1, KIND>)
        if (p.epilogue == EPI_ALPHA_BETA) { FE2O3_SHAPES(kUpdate); }
        else { FE2O3_SHAPES(kPlain); }
#undef FE2O3_SHAPES
    } else if (p.ep.pair_offsets) {
        // the first GEMM may share its SM with the small blocks of the dispatch kernel before it
        if (p.epilogue == EPI_GELU_BF16) {
            if (plan->bn == 256) f(gemm_tc_kernel<256, 128, 1, kPeerGelu>);
            else f(gemm_tc_kernel<128, 128, 1, kPeerGelu>);
        } else {
            if (plan->bn == 256) f(gemm_tc_kernel<256, 168, 1, kPeer>);
            else f(gemm_tc_kernel<128, 168, 1, kPeer>);
        }
    } else if (p.epilogue == EPI_GELU_BF16) {   // (with or without the warps that gather A)
        if (plan->pair) f(gemm_tc_kernel<256, 128, 2, kGroupedGelu>);
        else if (plan->bn == 256) f(gemm_tc_kernel<256, 128, 1, kGroupedGelu>);
        else f(gemm_tc_kernel<128, 128, 1, kGroupedGelu>);
    } else {
        if (plan->pair) f(gemm_tc_kernel<256, 168, 2, kGrouped>);
        else if (plan->bn == 256) f(gemm_tc_kernel<256, 168, 1, kGrouped>);
        else if (plan->bn == 128) f(gemm_tc_kernel<128, 168, 1, kGrouped>);
        else f(gemm_tc_kernel<64, 168, 1, kGrouped>);
    }
}

// Function attributes are per device: called by fe2o3_ctx_create with the context's device current.
int32_t gemm_tc_init_device() {
    cudaError_t e = cudaSuccess;
    auto set = [&](auto kernel, uint32_t bytes) {
        if (e == cudaSuccess) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    };
#define FE2O3_SHAPES(KIND)                                                     \
    set(gemm_tc_kernel<256, 168, 2, KIND>, SmemLayout<256, 2>::kTotal);        \
    set(gemm_tc_kernel<256, 168, 1, KIND>, SmemLayout<256, 1>::kTotal);        \
    set(gemm_tc_kernel<128, 168, 1, KIND>, SmemLayout<128, 1>::kTotal);        \
    set(gemm_tc_kernel<64, 168, 1, KIND>, SmemLayout<64, 1>::kTotal)
    FE2O3_SHAPES(kPlain);
    FE2O3_SHAPES(kUpdate);
    FE2O3_SHAPES(kGrouped);
#undef FE2O3_SHAPES
    set(gemm_tc_kernel<192, 168, 1, kPlain>, SmemLayout<192, 1>::kTotal);
    set(gemm_tc_kernel<192, 168, 1, kUpdate>, SmemLayout<192, 1>::kTotal);
    set(gemm_tc_kernel<256, 128, 2, kGroupedGelu>, SmemLayout<256, 2>::kTotal);
    set(gemm_tc_kernel<256, 128, 1, kGroupedGelu>, SmemLayout<256, 1>::kTotal);
    set(gemm_tc_kernel<128, 128, 1, kGroupedGelu>, SmemLayout<128, 1>::kTotal);
    set(gemm_tc_kernel<256, 168, 1, kPeer>, SmemLayout<256, 1>::kTotal);
    set(gemm_tc_kernel<128, 168, 1, kPeer>, SmemLayout<128, 1>::kTotal);
    set(gemm_tc_kernel<256, 128, 1, kPeerGelu>, SmemLayout<256, 1>::kTotal);
    set(gemm_tc_kernel<128, 128, 1, kPeerGelu>, SmemLayout<128, 1>::kTotal);
    return fe2o3_cuda_status(e, "cudaFuncSetAttribute(gemm_tc)");
}

int32_t gemm_tc_launch(const GemmTcPlan *plan, cudaStream_t s) {
    if (plan->p.M == 0 || plan->p.N == 0) return FE2O3_OK;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(plan->grid, 1, 1);
    cfg.blockDim = dim3(kThreads + (plan->p.gather_perm ? kGatherThreads : 0), 1, 1);
    cfg.dynamicSmemBytes = plan->smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    cfg.attrs = attr;
    if (plan->pair) {
        attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
        attr[cfg.numAttrs++].val.clusterDim = {2, 1, 1};
    }
    if (plan->overlap_previous || plan->p.after_previous) {
        // programmatic dependent launch: the kernel may start while the kernel before it in the stream is still
        // running.  The expert-parallel GEMMs and the kernels before them (which say when) synchronise through
        // flags; the others wait inside for that kernel to complete, with their set-up behind them.
        attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
    }
    cudaError_t e = cudaSuccess;
    with_kernel(plan, [&](auto kernel) { e = cudaLaunchKernelEx(&cfg, kernel, plan->tmA, plan->tmB, plan->tmC, plan->p); });
    fe2o3_count_launch(1);
    return fe2o3_cuda_status(e, "gemm_tc");
}

// Makes the plan's A operand a gather: row r of A = row (perm[r] >> 1) of src.  Needs whole 64-column K blocks and at
// least one token: the copy engine's gather form wants a map whose box is one row high, and src without rows has none.
bool gemm_tc_set_gather(GemmTcPlan *plan, const uint32_t *perm, const void *src, uint32_t tokens) {
    if (plan->p.K % BK != 0 || (reinterpret_cast<uintptr_t>(src) & 15u) != 0 || tokens == 0) return false;
    const uint64_t dims[2] = {plan->p.K, tokens}, stride[1] = {(uint64_t)plan->p.K * 2};
    const uint32_t box[2] = {BK, 1};
    if (fe2o3_make_tmap_bf16(&plan->tmA, reinterpret_cast<uint64_t>(src), 2, dims, stride, box) != FE2O3_OK) return false;
    plan->p.gather_perm = perm;
    plan->p.gather_tokens = tokens;
    return true;
}

// Makes the plan's output a weighted accumulation into token rows (see GemmParams); the plan must have been made
// with EPI_COMBINE_ADD and c = the [tokens][N] f32 output.
void gemm_tc_set_combine(GemmTcPlan *plan, const uint32_t *perm, const float *weights, uint32_t tokens) {
    plan->p.combine_perm = perm;
    plan->p.combine_weights = weights;
    plan->p.combine_tokens = tokens;
}

// The launch just before this one on the stream is the GEMM whose output is this one's A, and writes nothing else that
// this one reads: its weights may be fetched while that one still runs.
void gemm_tc_set_early_weights(GemmTcPlan *plan) {
    if (plan->p.after_previous) plan->p.after_previous = kEarlyWeights;
}

void gemm_tc_geometry(const GemmTcPlan *plan, fe2o3_geometry *geo) {
    *geo = fe2o3_geometry{{plan->grid, 1, 1}, {(uint32_t)(kThreads + (plan->p.gather_perm ? kGatherThreads : 0)), 1, 1}, plan->smem, 1};
}

// kernel symbols of the runtime adapter carried by this source (the schedule a large launch resolves to)
static Fe2o3KernelRegistration reg_tiled("tiled_gemm_lds_slice1", reinterpret_cast<const void *>(gemm_tc_kernel<256, 168, 1, kPlain>));
static Fe2o3KernelRegistration reg_general("tiled_gemm_general_v1", reinterpret_cast<const void *>(gemm_tc_kernel<256, 168, 1, kUpdate>));
static Fe2o3KernelRegistration reg_ffn("moe_expert_ffn_v1", reinterpret_cast<const void *>(gemm_tc_kernel<256, 128, 1, kGroupedGelu>));
static Fe2o3KernelRegistration reg_gffn("moe_grouped_ffn_v1", reinterpret_cast<const void *>(gemm_tc_kernel<256, 128, 1, kGroupedGelu>));
static Fe2o3KernelRegistration reg_ffnc("moe_expert_ffn_combine_v1", reinterpret_cast<const void *>(gemm_tc_kernel<256, 128, 1, kGroupedGelu>));
static Fe2o3KernelRegistration reg_epffn("moe_ep_ffn_v1", reinterpret_cast<const void *>(gemm_tc_kernel<256, 128, 1, kPeerGelu>));
