// Device-wide inclusive / exclusive prefix sum of u32 values (wrapping addition) and of f32 values
// (each addition rounded to nearest; one kernel template, values carried as 32-bit patterns).
//
// The reference defines prefix sums at two scopes: a 64-lane wave
// (crates/fe2o3-device/src/collective.rs:413-460, Hillis-Steele over lane
// shuffles; lane 0 of the exclusive form receives zero) and a workgroup through
// LDS scratch (collective.rs:503-571).  This kernel keeps their meaning (element
// i of the inclusive form is values[0] + ... + values[i], the exclusive form
// shifts by one and starts at zero, addition wraps) and extends the scope to a
// whole array in one pass over HBM: 4 bytes read and 4 bytes written per element.
//
// Single pass, staged through shared memory, with the carries between tiles taken
// from published tile sums.  One persistent block per SM; tiles of 8192 elements are
// handed out by an atomic ticket, so a tile only ever waits for tiles that started
// before it.  Four roles:
//   warp 0      producer: takes tickets and fills a six-stage ring of 32 KiB tiles
//               with bulk copies (an mbarrier per stage counts the bytes)
//   warps 1-4   aggregate: as soon as a tile has landed they sum it and publish its
//               aggregate, so the aggregates of all tiles in flight appear at the
//               speed of the memory system, whatever the rest of the block waits for
//   warp 5      prefix: keeps the sum of everything up to the block's previous tile and
//               adds the aggregates of the tiles between that one and the next (about
//               one per SM, fetched in one round trip).  No block waits for another
//               block's prefix, only for aggregates, so there is no chain across blocks
//   warps 6-13  finish: scan the tile from shared memory with that prefix and store it
//               with 16-byte writes; the warp scans of a tile run in lockstep
// The ring keeps 192 KiB per SM in flight, three times what a register-resident tile
// per thread allows.  Two earlier forms were measured and replaced: one pass over
// registers with a decoupled look-back in the same warps (0.53 of the HBM copy rate,
// bound by the wait for the predecessor's prefix), and this staging with a look-back
// warp that walked back to the nearest published inclusive prefix (0.68-0.76: with
// every tile of a wave in flight at once the nearest such prefix is a wave or more
// behind, and the walk became a serial chain of L2 round trips per SM).
// In the f32 form the order of additions must not depend on scheduling, so the prefix warp only
// ever accumulates whole chunks of 192 tiles from tile 0 and adds the part of the current chunk
// separately: whichever block computes a tile's prefix performs the same chain of additions, and
// repeated runs give identical bits.  The lane prefix inside a warp scan comes from a shuffle
// instead of a subtraction.
// A descriptor is one 64-bit word {launch tag, value}; it carries everything its reader
// needs, so relaxed device-scope accesses are enough.  The tag follows the count of launches
// so far, kept on the device, so nothing has to be cleared between launches (a memset in
// front of each cost 2 us): words of earlier launches never match.  scan_state.h has the rules.
// Every wait is bounded and records FE2O3_KSTATUS_WAIT_EXPIRED.
// Arrays of up to kWaveTilesPerSm tiles an SM take device_scan_wave_kernel below instead.
#include "common.cuh"
#include "scan_state.h"

namespace {

constexpr int kStages = 6;
constexpr uint32_t kTileElems = 8192;
constexpr uint32_t kTileBytes = kTileElems * 4;
constexpr int kAggWarps = 4;                                        // aggregate warps: 2048 consecutive elements each
constexpr int kFinishWarps = 8;                                     // scan-and-store warps: 1024 consecutive elements each
constexpr uint32_t kPart = kTileElems / kFinishWarps;               // 1024
constexpr int kPartVecs = kPart / 128;                              // a part is 8 rows of 32 lanes x 16 bytes
constexpr int kLaneVecs = 2;                                        // consecutive 16-byte groups a finish lane owns per pass
constexpr int kPasses = kPartVecs / kLaneVecs;                      // warp scans per finish warp and tile
constexpr int kScanThreads = 32 * (1 + kAggWarps + 1 + kFinishWarps);   // 448
constexpr int kWindow = 6;                                          // descriptors per lane and step of the prefix warp: 192, a little over one tile per SM
constexpr uint32_t kDescSpin = 1u << 22;
// Up to here one tile per block in registers (2^20 + 3 elements: 12.5 -> 7.5 us, 4 M: 16.7 in the ring, 13.9 so; 6 M:
// 19.6 against 21.7); beyond, the ring's bytes in flight win.
constexpr uint32_t kWaveTilesPerSm = 4;
constexpr uint32_t kNoTile = 0xffffffffu;

struct __align__(16) ScanShared {
    uint64_t full[kStages], empty[kStages], agg_ready[kStages], prefix_ready[kStages];
    uint32_t tile[kStages];                // ticket of the tile in each stage (kNoTile: the array is exhausted)
    uint32_t part[kStages][kFinishWarps];  // sums of the eight parts of the tile
    uint32_t prefix[kStages];              // exclusive prefix of the tile (sum of everything before it)
    uint32_t arrivals[kStages];            // aggregate warps done with the stage
};
constexpr uint32_t kSmemBytes = kStages * kTileBytes + sizeof(ScanShared) + 1024;

__device__ __forceinline__ void desc_store(uint64_t *p, uint32_t tag, uint32_t value) {
    const uint64_t v = ((uint64_t)tag << 32) | value;
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ uint64_t desc_load(const uint64_t *p) {
    uint64_t v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

// Values travel as 32-bit patterns; kFloat selects IEEE binary32 addition (round to nearest) instead of
// wrapping integer addition.  Zero is the all-zero pattern in both.
template <bool kFloat>
__device__ __forceinline__ uint32_t add(uint32_t a, uint32_t b) {
    if constexpr (kFloat) return __float_as_uint(__fadd_rn(__uint_as_float(a), __uint_as_float(b)));
    else return a + b;
}
template <bool kFloat>
__device__ __forceinline__ uint32_t sum4(const uint4 &x) {
    return add<kFloat>(add<kFloat>(x.x, x.y), add<kFloat>(x.z, x.w));
}
// sum over the warp in a fixed order (every lane receives it)
template <bool kFloat>
__device__ __forceinline__ uint32_t warp_sum(uint32_t v) {
    if constexpr (kFloat) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v = add<true>(v, __shfl_xor_sync(0xffffffffu, v, o));
        return v;
    } else {
        return __reduce_add_sync(0xffffffffu, v);
    }
}

// What outlives a launch, as scan_state.h wants it.
struct DeviceWords {
    static __device__ __forceinline__ scan_word add(scan_word *p, scan_word v) { return atomicAdd(p, v); }
    static __device__ __forceinline__ void fetch_or(scan_word *p, scan_word v) { atomicOr(p, v); }
    static __device__ __forceinline__ void store(scan_word *p, scan_word v) { *p = v; }
};
constexpr uint32_t kMaxTiles = (uint32_t)(FE2O3_SCAN_MAX_ELEMENTS / kTileElems);
constexpr uint32_t kMaxBlocks = 1024;
static_assert(kMaxTiles + kMaxBlocks < 1u << kScanTicketBits && kMaxBlocks < 1u << kScanBlockBits, "counts of one launch fit their fields");

// Last act of a block (one thread, when nobody in the block still reads descriptors).
__device__ __forceinline__ void block_done(scan_word *state, uint64_t *desc, uint32_t tag, uint32_t tickets, uint32_t *status) {
    if (!scan_finish<DeviceWords>(state, reinterpret_cast<scan_word *>(desc), kMaxTiles, tag, gridDim.x, tickets))
        kstatus_set(status, FE2O3_KSTATUS_SCAN_STATE);
}

// ---- arrays of a few tiles per SM -------------------------------------------------------------
// What bounds these is latency: one round trip for the data, one for the aggregates of the tiles before, one for
// the stores (the ring above adds its own hand-overs: 2^20 elements took 12.4 us with it).  A block keeps one tile
// of 8192 elements in registers, 16 a thread, publishes its sum and adds up the sums of all tiles before, one or
// a few per thread in an order fixed by the tile's number.  The tile is a ticket here too: a block only waits for
// blocks that have started, in whatever order they do, whether or not all are resident at once.
constexpr int kWaveThreads = 512, kWaveWarps = kWaveThreads / 32, kWaveRows = kTileElems / (kWaveThreads * 4);

template <bool kFloat>
__global__ void __launch_bounds__(kWaveThreads, 3)   // three blocks an SM: 40 registers
device_scan_wave_kernel(const uint32_t *in, uint32_t *out, uint64_t n, uint32_t exclusive, scan_word *state, uint64_t *desc,
                        uint32_t *status) {
    __shared__ uint32_t s_warp[kWaveWarps], s_before[kWaveWarps];
    __shared__ uint32_t s_tile, s_tag;
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    begin_after_previous();
    if (tid == 0) {
        scan_word drawn;
        s_tile = kNoTile;
        if (scan_take<DeviceWords>(state, gridDim.x, drawn)) s_tile = scan_tickets(drawn);
        else kstatus_set(status, FE2O3_KSTATUS_SCAN_STATE);
        s_tag = scan_tag(drawn);
    }
    __syncthreads();
    const uint32_t tile = s_tile, tag = s_tag;
    if (tile == kNoTile) return;
    const uint64_t first = (uint64_t)tile * kTileElems, base = first + warp * (kTileElems / kWaveWarps) + lane * 4;
    const bool vec = ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) & 15u) == 0 && first + kTileElems <= n;
    uint4 x[kWaveRows];   // row j: 128 consecutive elements of the warp's part
#pragma unroll
    for (int j = 0; j < kWaveRows; ++j) {
        const uint64_t e = base + j * 128;
        if (vec) {
            x[j] = __ldcs(reinterpret_cast<const uint4 *>(in + e));
        } else {
            x[j].x = e < n ? in[e] : 0u;
            x[j].y = e + 1 < n ? in[e + 1] : 0u;
            x[j].z = e + 2 < n ? in[e + 2] : 0u;
            x[j].w = e + 3 < n ? in[e + 3] : 0u;
        }
    }
    uint32_t own[kWaveRows], t[kWaveRows];   // each lane's total per row; the same scanned over the warp
#pragma unroll
    for (int j = 0; j < kWaveRows; ++j) own[j] = t[j] = sum4<kFloat>(x[j]);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
#pragma unroll
        for (int j = 0; j < kWaveRows; ++j) {
            const uint32_t up = __shfl_up_sync(0xffffffffu, t[j], o);
            if (lane >= (uint32_t)o) t[j] = add<kFloat>(up, t[j]);
        }
    }
    uint32_t total[kWaveRows], sum = 0;
#pragma unroll
    for (int j = 0; j < kWaveRows; ++j) {
        total[j] = __shfl_sync(0xffffffffu, t[j], 31);
        sum = add<kFloat>(sum, total[j]);
    }
    if (lane == 0) s_warp[warp] = sum;
    __syncthreads();
    if (tid == 0) {
        uint32_t aggregate = 0;
#pragma unroll
        for (int q = 0; q < kWaveWarps; ++q) aggregate = add<kFloat>(aggregate, s_warp[q]);
        desc_store(desc + tile, tag, aggregate);
    }
    uint32_t before = 0;
    bool ok = true;
    for (uint32_t i = tid; i < tile; i += kWaveThreads) {
        uint64_t d = desc_load(desc + i);
        for (uint32_t spins = 0; (uint32_t)(d >> 32) != tag; d = desc_load(desc + i)) {
            if (++spins > kDescSpin) { ok = false; break; }
            __nanosleep(20);
        }
        before = add<kFloat>(before, (uint32_t)d);
    }
    if (!ok) kstatus_set(status, FE2O3_KSTATUS_WAIT_EXPIRED);
    before = warp_sum<kFloat>(before);
    if (lane == 0) s_before[warp] = before;
    __syncthreads();
    if (tid == 0) block_done(state, desc, tag, gridDim.x, status);
    uint32_t carry = 0;   // everything before this warp's first element
#pragma unroll
    for (int q = 0; q < kWaveWarps; ++q) carry = add<kFloat>(carry, s_before[q]);
    for (uint32_t q = 0; q < warp; ++q) carry = add<kFloat>(carry, s_warp[q]);
#pragma unroll
    for (int j = 0; j < kWaveRows; ++j) {
        uint32_t run;   // everything before this lane's first element of the row
        if constexpr (kFloat) {
            const uint32_t below = __shfl_up_sync(0xffffffffu, t[j], 1);
            run = lane == 0 ? carry : add<true>(carry, below);
        } else {
            run = carry + t[j] - own[j];
        }
        carry = add<kFloat>(carry, total[j]);
        uint32_t inc[4];
        inc[0] = add<kFloat>(run, x[j].x);
        inc[1] = add<kFloat>(inc[0], x[j].y);
        inc[2] = add<kFloat>(inc[1], x[j].z);
        inc[3] = add<kFloat>(inc[2], x[j].w);
        const uint4 r = exclusive ? make_uint4(run, inc[0], inc[1], inc[2]) : make_uint4(inc[0], inc[1], inc[2], inc[3]);
        const uint64_t e = base + j * 128;
        if (vec) {
            __stcs(reinterpret_cast<uint4 *>(out + e), r);
        } else {
            if (e < n) out[e] = r.x;
            if (e + 1 < n) out[e + 1] = r.y;
            if (e + 2 < n) out[e + 2] = r.z;
            if (e + 3 < n) out[e + 3] = r.w;
        }
    }
}

template <bool kFloat>
__global__ void __launch_bounds__(kScanThreads, 1)
device_scan_kernel(const uint32_t *in, uint32_t *out, uint64_t n, uint32_t exclusive, scan_word *state,
                   uint64_t *desc, uint32_t *status) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint32_t *ring = reinterpret_cast<uint32_t *>(smem);
    ScanShared &sh = *reinterpret_cast<ScanShared *>(smem + kStages * kTileBytes);
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const bool aligned = ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) & 15u) == 0;

    if (tid == 0) {
        for (int i = 0; i < kStages; ++i) {
            mbar_init(&sh.full[i], 1);
            mbar_init(&sh.empty[i], kFinishWarps);
            mbar_init(&sh.agg_ready[i], 1);
            mbar_init(&sh.prefix_ready[i], 1);
            sh.arrivals[i] = 0;
        }
        mbar_fence_init();
    }
    __syncthreads();
    begin_after_previous();
    const uint32_t tag = scan_tag(__ldcg(state));
    const uint32_t tickets = (uint32_t)((n + kTileElems - 1) / kTileElems) + gridDim.x;   // every block draws one past the last tile

    if (warp == 0) {
        // ------------------------------------------------------------ producer
        bool ok = true;
        for (uint32_t k = 0; ok; ++k) {
            const uint32_t st = k % kStages, ph = (k / kStages) & 1;
            if (!mbar_wait_warp(&sh.empty[st], ph ^ 1)) { ok = false; break; }
            uint32_t t = 0;
            if (lane == 0) {
                scan_word drawn;
                t = kNoTile;
                if (scan_take<DeviceWords>(state, tickets, drawn)) t = scan_tickets(drawn);
                else kstatus_set(status, FE2O3_KSTATUS_SCAN_STATE);
            }
            t = __shfl_sync(0xffffffffu, t, 0);
            const uint64_t base = (uint64_t)t * kTileElems;
            if (base >= n) {
                // the array is exhausted: tell the consumers and stop
                if (lane == 0) {
                    sh.tile[st] = kNoTile;
                    mbar_arrive(&sh.full[st]);
                }
                __syncwarp();
                break;
            }
            uint32_t *dst = ring + st * kTileElems;
            if (aligned && base + kTileElems <= n) {
                if (lane == 0) {
                    sh.tile[st] = t;
                    mbar_arrive_expect_tx(&sh.full[st], kTileBytes);
                    bulk_load_1d(dst, in + base, kTileBytes, &sh.full[st]);
                }
            } else if (aligned) {
                // the last tile: whole 16-byte pieces by the copy engine, the rest by the lanes, zero beyond the end (one
                // element after the other it took up to 50 us and set the time of every length that is not whole tiles)
                const uint32_t have = (uint32_t)(n - base), whole = have & ~3u;
                if (lane < 4 && whole < kTileElems) dst[whole + lane] = whole + lane < have ? in[base + whole + lane] : 0u;
                for (uint32_t i = whole / 4 + 1 + lane; i < kTileElems / 4; i += 32) reinterpret_cast<uint4 *>(dst)[i] = make_uint4(0, 0, 0, 0);
                __syncwarp();
                if (lane == 0) {
                    sh.tile[st] = t;
                    if (whole) {
                        mbar_arrive_expect_tx(&sh.full[st], whole * 4);
                        bulk_load_1d(dst, in + base, whole * 4, &sh.full[st]);
                    } else {
                        mbar_arrive(&sh.full[st]);
                    }
                }
            } else {   // input the copy engine cannot address: plain loads, sixteen in flight a lane
                for (uint32_t i0 = lane; i0 < kTileElems; i0 += 32 * 16) {
                    uint32_t v[16];
#pragma unroll
                    for (int q = 0; q < 16; ++q) v[q] = base + i0 + 32 * q < n ? in[base + i0 + 32 * q] : 0u;
#pragma unroll
                    for (int q = 0; q < 16; ++q) dst[i0 + 32 * q] = v[q];
                }
                __syncwarp();
                if (lane == 0) {
                    sh.tile[st] = t;
                    mbar_arrive(&sh.full[st]);
                }
            }
            __syncwarp();
        }
        if (!ok && lane == 0) kstatus_set(status, FE2O3_KSTATUS_WAIT_EXPIRED);
    } else if (warp <= kAggWarps) {
        // ------------------------------------------------------------ aggregate warps
        const uint32_t w = warp - 1;
        for (uint32_t k = 0;; ++k) {
            const uint32_t st = k % kStages, ph = (k / kStages) & 1;
            if (!mbar_wait_warp(&sh.full[st], ph)) {
                if (lane == 0) kstatus_set(status, FE2O3_KSTATUS_WAIT_EXPIRED);
                break;
            }
            const uint32_t tile = sh.tile[st];
            if (tile == kNoTile) break;
            // this warp sums parts 2w and 2w + 1 of the tile
            const uint4 *src = reinterpret_cast<const uint4 *>(ring + st * kTileElems + w * 2 * kPart) + lane;
            uint32_t sum0 = 0, sum1 = 0;
#pragma unroll
            for (int j = 0; j < kPartVecs; ++j) {
                const uint4 x = src[j * 32], y = src[(kPartVecs + j) * 32];
                sum0 = add<kFloat>(sum0, sum4<kFloat>(x));
                sum1 = add<kFloat>(sum1, sum4<kFloat>(y));
            }
            sum0 = warp_sum<kFloat>(sum0);
            sum1 = warp_sum<kFloat>(sum1);
            // the last of the four warps to finish publishes the tile's aggregate
            uint32_t last = 0;
            if (lane == 0) {
                sh.part[st][2 * w] = sum0;
                sh.part[st][2 * w + 1] = sum1;
                __threadfence_block();
                last = atomicAdd(&sh.arrivals[st], 1u) == kAggWarps - 1 ? 1u : 0u;
            }
            last = __shfl_sync(0xffffffffu, last, 0);
            if (last && lane == 0) {
                __threadfence_block();
                uint32_t aggregate = 0;
                for (int q = 0; q < kFinishWarps; ++q) aggregate = add<kFloat>(aggregate, sh.part[st][q]);
                sh.arrivals[st] = 0;
                desc_store(desc + tile, tag, aggregate);
                mbar_arrive(&sh.agg_ready[st]);
            }
        }
    } else if (warp == kAggWarps + 1) {
        // ------------------------------------------------------------ prefix warp: runs ahead of the finish warps
        // The block's tiles arrive in ticket order.  The warp keeps the sum of everything up to and
        // including the block's previous tile, so the prefix of the next one only needs the aggregates
        // of the tiles in between (about one per SM), which other blocks publish as their data lands.
        bool ok = true;
        uint32_t covered = 0;   // tiles [0, covered) are summed in `running`
        uint32_t running = 0;
        for (uint32_t k = 0; ok; ++k) {
            const uint32_t st = k % kStages, ph = (k / kStages) & 1;
            if (!mbar_wait_warp(&sh.full[st], ph)) { ok = false; break; }
            const uint32_t tile = sh.tile[st];
            if (tile == kNoTile) break;
            // sum of the published aggregates of tiles [lo, hi): lanes take them 32 apart, then a warp sum
            auto range_sum = [&](uint32_t lo, uint32_t hi) -> uint32_t {
                uint32_t acc = 0;
                for (uint32_t b = lo; ok && b < hi; b += 32 * kWindow) {
                    uint64_t d[kWindow];
#pragma unroll
                    for (int q = 0; q < kWindow; ++q) {   // all loads of the step in flight together
                        const uint32_t mine = b + 32 * q + lane;
                        d[q] = mine < hi ? desc_load(desc + mine) : ((uint64_t)tag << 32);
                    }
#pragma unroll
                    for (int q = 0; q < kWindow; ++q) {
                        const uint32_t mine = b + 32 * q + lane;
                        uint32_t spins = 0;
                        while ((uint32_t)(d[q] >> 32) != tag) {
                            if (++spins > kDescSpin) { ok = false; break; }
                            __nanosleep(100);
                            d[q] = desc_load(desc + mine);
                        }
                        acc = add<kFloat>(acc, (uint32_t)d[q]);
                    }
                    ok = __all_sync(0xffffffffu, ok);
                }
                return warp_sum<kFloat>(acc);
            };
            uint32_t prefix;
            if constexpr (kFloat) {
                // Rounding makes the order matter.  `running` only ever stops at multiples of kChunk tiles and
                // advances by whole chunks, so the prefix of a tile is the same chain of additions whichever
                // block computes it: results do not depend on how the tickets fell.
                constexpr uint32_t kChunk = 32 * kWindow;
                while (ok && covered + 2 * kChunk <= tile) {
                    running = add<true>(running, range_sum(covered, covered + kChunk));
                    covered += kChunk;
                }
                if (covered + kChunk <= tile) {
                    // the usual case, one whole chunk and a part of the next: both windows' loads go out
                    // together, so the step costs one round trip; the additions are the same as above
                    const uint32_t mid = covered + kChunk;
                    uint64_t d[2][kWindow];
#pragma unroll
                    for (int h = 0; h < 2; ++h)
#pragma unroll
                        for (int q = 0; q < kWindow; ++q) {
                            const uint32_t mine = (h ? mid : covered) + 32 * q + lane;
                            d[h][q] = mine < (h ? tile : mid) ? desc_load(desc + mine) : ((uint64_t)tag << 32);
                        }
                    uint32_t acc[2] = {0, 0};
#pragma unroll
                    for (int h = 0; h < 2; ++h)
#pragma unroll
                        for (int q = 0; q < kWindow; ++q) {
                            const uint32_t mine = (h ? mid : covered) + 32 * q + lane;
                            uint32_t spins = 0;
                            while ((uint32_t)(d[h][q] >> 32) != tag) {
                                if (++spins > kDescSpin) { ok = false; break; }
                                __nanosleep(100);
                                d[h][q] = desc_load(desc + mine);
                            }
                            acc[h] = add<true>(acc[h], (uint32_t)d[h][q]);
                        }
                    ok = __all_sync(0xffffffffu, ok);
                    running = add<true>(running, warp_sum<true>(acc[0]));
                    covered = mid;
                    prefix = add<true>(running, warp_sum<true>(acc[1]));
                } else {
                    prefix = add<true>(running, range_sum(covered, tile));
                }
            } else {
                prefix = running + range_sum(covered, tile);
            }
            if (!ok) break;
            if (!mbar_wait_warp(&sh.agg_ready[st], ph)) { ok = false; break; }
            // The stage's partial sums are read BEFORE the arrival below: that arrival lets the finish
            // warps release the stage, after which the aggregate warps may overwrite sh.part[st].
            uint32_t aggregate = 0;
            if constexpr (!kFloat) {
                for (int q = 0; q < kFinishWarps; ++q) aggregate += sh.part[st][q];
            }
            __syncwarp();
            if (lane == 0) {
                sh.prefix[st] = prefix;
                mbar_arrive(&sh.prefix_ready[st]);
            }
            if constexpr (!kFloat) {
                running = prefix + aggregate;
                covered = tile + 1;
            }
        }
        if (!ok && lane == 0) kstatus_set(status, FE2O3_KSTATUS_WAIT_EXPIRED);   // the finish warps' waits expire in turn
    } else {
        // ------------------------------------------------------------ finish warps
        const uint32_t w = warp - 2 - kAggWarps;
        for (uint32_t k = 0;; ++k) {
            const uint32_t st = k % kStages, ph = (k / kStages) & 1;
            const bool ok = mbar_wait_warp(&sh.full[st], ph);
            const uint32_t tile = ok ? sh.tile[st] : kNoTile;
            if (!ok && lane == 0) kstatus_set(status, FE2O3_KSTATUS_WAIT_EXPIRED);
            if (tile == kNoTile) break;
            if (!mbar_wait_warp(&sh.prefix_ready[st], ph)) {
                if (lane == 0) kstatus_set(status, FE2O3_KSTATUS_WAIT_EXPIRED);
                break;
            }
            uint32_t carry = sh.prefix[st];   // everything before this warp's first element
            for (uint32_t q = 0; q < w; ++q) carry = add<kFloat>(carry, sh.part[st][q]);
            const uint64_t base = (uint64_t)tile * kTileElems + (uint64_t)w * kPart + lane * (4 * kLaneVecs);
            const bool vec = aligned && (uint64_t)tile * kTileElems + kTileElems <= n;
            const uint4 *src = reinterpret_cast<const uint4 *>(ring + st * kTileElems + w * kPart) + lane * kLaneVecs;
            // Each lane owns kLaneVecs consecutive 16-byte groups per pass, so one warp scan covers
            // 32 * 4 * kLaneVecs elements.  The passes' warp scans are independent and run in
            // lockstep: each shuffle step issues one shuffle per pass back to back, and the latency
            // of a chain is paid once per tile, not once per pass.
            uint4 x[kPasses][kLaneVecs];
            uint32_t own[kPasses], t[kPasses];   // each lane's total per pass; the same scanned over the warp
#pragma unroll
            for (int j = 0; j < kPasses; ++j) {
                own[j] = 0;
#pragma unroll
                for (int c = 0; c < kLaneVecs; ++c) {
                    x[j][c] = src[j * 32 * kLaneVecs + c];
                    own[j] = add<kFloat>(own[j], sum4<kFloat>(x[j][c]));
                }
                t[j] = own[j];
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh.empty[st]);   // the part is in registers: the stage may be refilled
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
#pragma unroll
                for (int j = 0; j < kPasses; ++j) {
                    const uint32_t up = __shfl_up_sync(0xffffffffu, t[j], o);
                    if (lane >= (uint32_t)o) t[j] = add<kFloat>(up, t[j]);
                }
            }
#pragma unroll
            for (int j = 0; j < kPasses; ++j) {
                // everything before this lane's first element of the pass
                uint32_t run;
                if constexpr (kFloat) {   // no subtraction in floating point: take the lower lane's inclusive total
                    const uint32_t below = __shfl_up_sync(0xffffffffu, t[j], 1);
                    run = lane == 0 ? carry : add<true>(carry, below);
                } else {
                    run = carry + t[j] - own[j];
                }
                carry = add<kFloat>(carry, __shfl_sync(0xffffffffu, t[j], 31));
#pragma unroll
                for (int c = 0; c < kLaneVecs; ++c) {
                    // inclusive values of the four elements, each the previous one plus the element
                    uint32_t inc[4];
                    inc[0] = add<kFloat>(run, x[j][c].x);
                    inc[1] = add<kFloat>(inc[0], x[j][c].y);
                    inc[2] = add<kFloat>(inc[1], x[j][c].z);
                    inc[3] = add<kFloat>(inc[2], x[j][c].w);
                    uint32_t r[4];
                    if (exclusive) {   // element i of the exclusive form is the inclusive value of element i - 1
                        r[0] = run; r[1] = inc[0]; r[2] = inc[1]; r[3] = inc[2];
                    } else {
                        r[0] = inc[0]; r[1] = inc[1]; r[2] = inc[2]; r[3] = inc[3];
                    }
                    run = inc[3];
                    const uint64_t e = base + (uint64_t)j * (128 * kLaneVecs) + c * 4;
                    if (vec) {
                        __stcs(reinterpret_cast<uint4 *>(out + e), make_uint4(r[0], r[1], r[2], r[3]));
                    } else {
#pragma unroll
                        for (int i = 0; i < 4; ++i)
                            if (e + i < n) out[e + i] = r[i];
                    }
                }
            }
        }
    }
    __syncthreads();
    if (tid == 0) block_done(state, desc, tag, tickets, status);
}

}  // namespace

template <bool kFloat>
int32_t launch_device_scan(fe2o3_ctx *ctx, cudaStream_t s, const void *args, fe2o3_geometry *geo, bool plan_only) {
    const fe2o3_device_scan_u32_args *a = static_cast<const fe2o3_device_scan_u32_args *>(args);
    const uint64_t n = a->values.len;
    const uint32_t tiles = (uint32_t)((n + kTileElems - 1) / kTileElems);
    const uint32_t sms = min(ctx->sm_count > 0 ? (uint32_t)ctx->sm_count : 1u, kMaxBlocks / kWaveTilesPerSm);
    const bool wave = tiles <= kWaveTilesPerSm * sms;
    const uint32_t grid = wave || tiles < sms ? (tiles ? tiles : 1u) : sms;
    if (geo) *geo = wave ? fe2o3_geometry{{grid, 1, 1}, {kWaveThreads, 1, 1}, 0, 1} : fe2o3_geometry{{grid, 1, 1}, {kScanThreads, 1, 1}, kSmemBytes, 1};
    if (plan_only || n == 0) return FE2O3_OK;
    // the state at byte 0, descriptors from byte 64
    scan_word *state = reinterpret_cast<scan_word *>(ctx->scan_scratch);
    uint64_t *desc = reinterpret_cast<uint64_t *>(ctx->scan_scratch + 16);
    const uint32_t *in = reinterpret_cast<const uint32_t *>(a->values.ptr);
    uint32_t *out = reinterpret_cast<uint32_t *>(a->output.ptr);
    const cudaError_t e = wave ? fe2o3_launch_early(device_scan_wave_kernel<kFloat>, grid, kWaveThreads, 0, s, 1, in, out, n,
                                                    a->exclusive, state, desc, ctx->status_word)
                               : fe2o3_launch_early(device_scan_kernel<kFloat>, grid, kScanThreads, kSmemBytes, s, 1, in, out, n,
                                                    a->exclusive, state, desc, ctx->status_word);
    fe2o3_count_launch(1);
    return fe2o3_cuda_status(e, kFloat ? "device_scan_sum_f32" : "device_scan_sum_u32");
}

// Function attributes are per device: called by fe2o3_ctx_create with the context's device current.
int32_t device_scan_init_device() {
    FE2O3_CUDA(cudaFuncSetAttribute(device_scan_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBytes));
    FE2O3_CUDA(cudaFuncSetAttribute(device_scan_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBytes));
    return FE2O3_OK;
}

int32_t launch_device_scan_u32(fe2o3_ctx *ctx, cudaStream_t s, const void *args, fe2o3_geometry *geo, bool plan_only) {
    return launch_device_scan<false>(ctx, s, args, geo, plan_only);
}
int32_t launch_device_scan_f32(fe2o3_ctx *ctx, cudaStream_t s, const void *args, fe2o3_geometry *geo, bool plan_only) {
    return launch_device_scan<true>(ctx, s, args, geo, plan_only);
}

static Fe2o3KernelRegistration reg_scan_u32("device_scan_sum_u32", reinterpret_cast<const void *>(device_scan_kernel<false>));
static Fe2o3KernelRegistration reg_scan_f32("device_scan_sum_f32", reinterpret_cast<const void *>(device_scan_kernel<true>));
