// Exact-order GEMM schedule on CUDA cores.
//
// Every output element is computed with the reference recurrence: accumulator
// starts at +0.0f, k increases from 0, each step is one IEEE f32 product
// followed by one IEEE f32 sum (no fused contraction), then the optional
// epilogue alpha*acc + beta*c as two products and one sum
// (examples/tiled_gemm_v1/src/oracle.rs:284-321,
//  examples/tiled_gemm_v1/src/numerical_contract.rs:310-326,
//  examples/scalar_gemm_v1/src/kernel.rs:8-27).  Results are therefore
// bit-identical to the CPU oracle for every finite or non-finite input, any
// strides and any tails.
//
// Bound: the f32 pipe, two operations per multiply-add that may not be fused (512^3: 7.5 us on 148 SMs).  A block of 128
// threads owns 8 RM x 16 RN outputs, RM x RN a thread.
//   f32: tiles of 32 k go to shared memory by asynchronous copies, a ring of three (two for 64 rows), one barrier a tile; pieces of four
// bytes where rows do not start on 16.  Both operands lie as they do in memory: a thread reads four k of each of its
// rows and four rows of B, 16 bytes each, for RM x RN x 4 products.  Products are scalar, sums packed f32x2 (each half
// rounded like the scalar instruction; a packed product feeding a packed sum came out fused, with one rounding).
// us, with operands passed through registers and A transposed on the way (until then) / so: 512^3 18.2 / 15.8, 1024^3 134 / 91,
// 256^3 9.8 / 5.8, 900 x 40 x 800 31 / 15; at 1024^3 the f32 pipe is three quarters busy.
//   bf16: operands are widened on the way, through registers.  Products of bf16 values are exact in f32 unless they leave its
// range, so a fused multiply-add rounds just as a product and a sum do: where every value of a tile is zero or between
// 2^-62 and 2^63 the fused form is used, which halves the work of the pipe; other tiles take the two-step form.
// us, alpha/beta, always two steps / so: 2999^3 at odd addresses 2299 / 1445, 300 x 1001 x 501 55 / 33, 100^3 13.0 / 5.3.
#include "bf16_piece.h"
#include "common.cuh"

#include <math.h>

namespace {

constexpr int TK = 32, kThreads = 128;

template <int RM, int RN, int STAGES>
struct __align__(16) ExactTiles {
    float a[STAGES][8 * RM][TK + 4];   // rows of 144 bytes: a warp's two rows fall on different banks
    float b[STAGES][TK][16 * RN];
};

template <int BYTES>
__device__ __forceinline__ void copy_async(void *dst, const void *src, uint32_t valid) {
    if constexpr (BYTES == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(valid) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(valid) : "memory");
}

// The operands of a thread for four k, and its RM x RN sums over them.
template <int RM, int RN>
struct Operands {
    float4 a[RM];
    float b[4][RN];
    __device__ __forceinline__ void load(const float (*as)[TK + 4], const float (*bs)[16 * RN], int row, int col, int kk) {
#pragma unroll
        for (int i = 0; i < RM; ++i) a[i] = *reinterpret_cast<const float4 *>(&as[row + i][kk]);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if constexpr (RN == 4) {
                const float4 v = *reinterpret_cast<const float4 *>(&bs[kk + q][col]);
                b[q][0] = v.x; b[q][1] = v.y; b[q][2] = v.z; b[q][3] = v.w;
            } else {
                const float2 v = *reinterpret_cast<const float2 *>(&bs[kk + q][col]);
                b[q][0] = v.x; b[q][1] = v.y;
            }
        }
    }
};

template <int RM, int RN, bool FUSED>
__device__ __forceinline__ void one_step(uint64_t (&acc)[RM][RN / 2], const float (&a)[RM], const float (&b)[RN]) {
#pragma unroll
    for (int i = 0; i < RM; ++i)
#pragma unroll
        for (int j = 0; j < RN / 2; ++j) {
            if constexpr (FUSED) acc[i][j] = fma_f32x2(pack_f32x2(a[i], a[i]), pack_f32x2(b[2 * j], b[2 * j + 1]), acc[i][j]);
            else acc[i][j] = add_f32x2(acc[i][j], pack_f32x2(__fmul_rn(a[i], b[2 * j]), __fmul_rn(a[i], b[2 * j + 1])));
        }
}

template <int RM, int RN, bool FUSED>
__device__ __forceinline__ void four_steps(uint64_t (&acc)[RM][RN / 2], const Operands<RM, RN> &o) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        float a[RM];
#pragma unroll
        for (int i = 0; i < RM; ++i) a[i] = q == 0 ? o.a[i].x : q == 1 ? o.a[i].y : q == 2 ? o.a[i].z : o.a[i].w;
        one_step<RM, RN, FUSED>(acc, a, o.b[q]);
    }
}

// The first `steps` k of a tile.
template <int RM, int RN, bool FUSED>
__device__ __forceinline__ void multiply_tile(uint64_t (&acc)[RM][RN / 2], const float (*as)[TK + 4], const float (*bs)[16 * RN], int row, int col,
                                              uint32_t steps) {
    if (steps == TK && RM == 2 && RN == 2) {
        // few blocks, and a scheduler has one warp at most: operands come four k ahead
        Operands<RM, RN> even, odd;
        even.load(as, bs, row, col, 0);
#pragma unroll 1
        for (int kk = 0; kk < TK; kk += 8) {
            odd.load(as, bs, row, col, kk + 4);
            four_steps<RM, RN, FUSED>(acc, even);
            even.load(as, bs, row, col, (kk + 8) % TK);   // (the last of a tile are not used)
            four_steps<RM, RN, FUSED>(acc, odd);
        }
    } else if (steps == TK) {
#pragma unroll
        for (int kk = 0; kk < TK; kk += 4) {
            Operands<RM, RN> o;
            o.load(as, bs, row, col, kk);
            four_steps<RM, RN, FUSED>(acc, o);
        }
    } else {   // the recurrence stops at K: the padding of the last tile is never multiplied
        uint32_t kk = 0;
        if constexpr (RM > 2) {   // (two rows a thread lose 2 % of their whole tiles to it: other registers)
#pragma unroll 1
            for (; kk + 4 <= steps; kk += 4) {
                Operands<RM, RN> o;
                o.load(as, bs, row, col, kk);
                four_steps<RM, RN, FUSED>(acc, o);
            }
        }
#pragma unroll 1
        for (; kk < steps; ++kk) {
            float a[RM], b[RN];
#pragma unroll
            for (int i = 0; i < RM; ++i) a[i] = as[row + i][kk];
#pragma unroll
            for (int j = 0; j < RN; ++j) b[j] = bs[kk][col + j];
            one_step<RM, RN, FUSED>(acc, a, b);
        }
    }
}

template <int RM, int RN, bool EPILOGUE>
__device__ __forceinline__ void write_sums(const uint64_t (&acc)[RM][RN / 2], float *C, uint32_t row0, uint32_t c0, uint32_t M, uint32_t N,
                                           uint32_t ldc, float alpha, float beta) {
    const bool vec = ldc % RN == 0 && reinterpret_cast<uintptr_t>(C) % (4 * RN) == 0 && c0 + RN <= N;
    // all old values are asked for before the first sum is written, for a load may not overtake a store to C
    float old[RM][RN];
    if constexpr (EPILOGUE) {
#pragma unroll
        for (int i = 0; i < RM; ++i) {
            const float *src = C + (uint64_t)(row0 + i) * ldc + c0;
            if (row0 + i < M && vec) {
                if constexpr (RN == 4) {
                    const float4 x = *reinterpret_cast<const float4 *>(src);
                    old[i][0] = x.x; old[i][1] = x.y; old[i][2] = x.z; old[i][3] = x.w;
                } else {
                    const float2 x = *reinterpret_cast<const float2 *>(src);
                    old[i][0] = x.x; old[i][1] = x.y;
                }
            } else {
#pragma unroll
                for (int j = 0; j < RN; ++j) old[i][j] = row0 + i < M && c0 + j < N ? src[j] : 0.0f;
            }
        }
    }
#pragma unroll
    for (int i = 0; i < RM; ++i) {
        if (row0 + i >= M) continue;
        float v[RN];
#pragma unroll
        for (int j = 0; j < RN / 2; ++j) unpack_f32x2(acc[i][j], v[2 * j], v[2 * j + 1]);
        if constexpr (EPILOGUE) {
#pragma unroll
            for (int j = 0; j < RN; ++j) v[j] = __fadd_rn(__fmul_rn(alpha, v[j]), __fmul_rn(beta, old[i][j]));
        }
        float *dst = C + (uint64_t)(row0 + i) * ldc + c0;
        if (vec) {
            if constexpr (RN == 4) *reinterpret_cast<float4 *>(dst) = make_float4(v[0], v[1], v[2], v[3]);
            else *reinterpret_cast<float2 *>(dst) = make_float2(v[0], v[1]);
        } else {
#pragma unroll
            for (int j = 0; j < RN; ++j)
                if (c0 + j < N) dst[j] = v[j];
        }
    }
}

// ---- f32 operands: asynchronous copies
template <int RM>
constexpr int kF32Stages = RM == 8 ? 2 : 3;   // (a block's 48 KiB)
template <int RM, int RN>
__global__ void __launch_bounds__(kThreads)
gemm_exact_f32_kernel(const float *__restrict__ A, const float *__restrict__ B, float *C, uint32_t M, uint32_t N, uint32_t K, uint32_t lda,
                      uint32_t ldb, uint32_t ldc, float, float) {
    constexpr int TM = 8 * RM, TN = 16 * RN, STAGES = kF32Stages<RM>;
    __shared__ ExactTiles<RM, RN, STAGES> tiles;
    const uint32_t tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const uint32_t row_tiles = (M - 1) / TM + 1;
    const uint32_t row0 = blockIdx.x % row_tiles * TM, col0 = blockIdx.x / row_tiles * TN;
    const bool vec_a = lda % 4 == 0 && reinterpret_cast<uintptr_t>(A) % 16 == 0;
    const bool vec_b = ldb % 4 == 0 && reinterpret_cast<uintptr_t>(B) % 16 == 0;
    // what lies past M, N or K arrives as zeros; nothing past a row's end is read
    auto copy = [&](uint32_t k0, uint32_t st) {
        if (vec_a) {
#pragma unroll
            for (int i = 0; i < TM * TK / 4 / kThreads; ++i) {
                const uint32_t g = i * kThreads + tid, r = g / (TK / 4), k = g % (TK / 4) * 4;
                const bool in = row0 + r < M && k0 + k < K;
                copy_async<16>(&tiles.a[st][r][k], in ? A + (uint64_t)(row0 + r) * lda + k0 + k : A, in ? min(K - k0 - k, 4u) * 4 : 0u);
            }
        } else {
            const uint32_t k = tid % TK, r0 = tid / TK;   // every thread keeps its k
            const float *src = A + min(k0 + k, K - 1);
#pragma unroll 8
            for (int i = 0; i < TM * TK / kThreads; ++i) {
                const uint32_t r = r0 + i * (kThreads / TK);
                copy_async<4>(&tiles.a[st][r][k], src + (uint64_t)min(row0 + r, M - 1) * lda, row0 + r < M && k0 + k < K ? 4u : 0u);
            }
        }
        if (vec_b) {
#pragma unroll
            for (int i = 0; i < TK * TN / 4 / kThreads; ++i) {
                const uint32_t g = i * kThreads + tid, k = g / (TN / 4), c = g % (TN / 4) * 4;
                const bool in = k0 + k < K && col0 + c < N;
                copy_async<16>(&tiles.b[st][k][c], in ? B + (uint64_t)(k0 + k) * ldb + col0 + c : B, in ? min(N - col0 - c, 4u) * 4 : 0u);
            }
        } else {
            const uint32_t c = tid % TN, q0 = tid / TN;   // every thread keeps its column
            const float *src = B + min(col0 + c, N - 1);
#pragma unroll 8
            for (int i = 0; i < TK * TN / kThreads; ++i) {
                const uint32_t k = q0 + i * (kThreads / TN);
                copy_async<4>(&tiles.b[st][k][c], src + (uint64_t)min(k0 + k, K - 1) * ldb, col0 + c < N && k0 + k < K ? 4u : 0u);
            }
        }
    };
    uint64_t acc[RM][RN / 2];
#pragma unroll
    for (int i = 0; i < RM; ++i)
#pragma unroll
        for (int j = 0; j < RN / 2; ++j) acc[i][j] = 0ull;   // pairs of +0.0f
    begin_after_previous();
#pragma unroll 1
    for (uint32_t s = 0; s + 1 < STAGES; ++s) {
        if (s * TK < K) copy(s * TK, s);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    uint32_t st = 0, next = STAGES - 1;
    for (uint32_t k0 = 0; k0 < K; k0 += TK) {
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
        __syncthreads();   // the tile is there, and everybody is done with the one before, whose place the next copy takes
        if (K - k0 > (STAGES - 1) * TK) copy(k0 + (STAGES - 1) * TK, next);
        asm volatile("cp.async.commit_group;" ::: "memory");
        multiply_tile<RM, RN, false>(acc, tiles.a[st], tiles.b[st], ty * RM, tx * RN, min(K - k0, (uint32_t)TK));
        st = st + 1 == STAGES ? 0 : st + 1;
        next = next + 1 == STAGES ? 0 : next + 1;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    write_sums<RM, RN, false>(acc, C, row0 + ty * RM, col0 + tx * RN, M, N, ldc, 1.0f, 0.0f);
}

// ---- bf16 operands: widened on the way through registers
struct GlobalPieces {
    static __device__ __forceinline__ uint32_t half(const uint16_t *p) { return __ldg(p); }
    static __device__ __forceinline__ uint32_t word(const uint16_t *p) { return __ldg(reinterpret_cast<const uint32_t *>(p)); }
    static __device__ __forceinline__ void two_words(const uint16_t *p, uint32_t &a, uint32_t &b) {
        const uint2 v = __ldg(reinterpret_cast<const uint2 *>(p));
        a = v.x; b = v.y;
    }
};

template <int RM, int RN, bool EPILOGUE>
__global__ void __launch_bounds__(kThreads)
gemm_exact_bf16_kernel(const uint16_t *__restrict__ A, const uint16_t *__restrict__ B, float *C, uint32_t M, uint32_t N, uint32_t K, uint32_t lda,
                       uint32_t ldb, uint32_t ldc, float alpha, float beta) {
    constexpr int TM = 8 * RM, TN = 16 * RN, GA = TM * TK / 4 / kThreads, GB = TK * TN / 4 / kThreads;
    __shared__ ExactTiles<RM, RN, 2> tiles;
    const uint32_t tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const uint32_t row_tiles = (M - 1) / TM + 1;
    const uint32_t row0 = blockIdx.x % row_tiles * TM, col0 = blockIdx.x / row_tiles * TN;
    const bool vec_a = lda % 4 == 0 && reinterpret_cast<uintptr_t>(A) % 8 == 0;
    const bool vec_b = ldb % 4 == 0 && reinterpret_cast<uintptr_t>(B) % 8 == 0;
    uint32_t a_next[GA][3], b_next[GB][3], halves = 0;   // halves: a bit for each piece that starts in the middle of a word
    auto fetch = [&](uint32_t k0) {
        halves = 0;
#pragma unroll
        for (int i = 0; i < GA; ++i) {
            const uint32_t g = i * kThreads + tid, r = g / (TK / 4), k = g % (TK / 4) * 4;
            const bool in = row0 + r < M;
            halves |= (uint32_t)load_piece<GlobalPieces>(a_next[i], A + (uint64_t)(in ? row0 + r : 0) * lda, k0 + k, K, in, vec_a) << i;
        }
#pragma unroll
        for (int i = 0; i < GB; ++i) {
            const uint32_t g = i * kThreads + tid, k = k0 + g / (TN / 4), c = g % (TN / 4) * 4;
            halves |= (uint32_t)load_piece<GlobalPieces>(b_next[i], B + (uint64_t)(k < K ? k : 0) * ldb, col0 + c, N, k < K, vec_b) << (GA + i);
        }
    };
    // Returns whether a product with one of the values may not be exact: exponents other than that of zero and those
    // between 65 and 189 (2^-62 to below 2^63).
    auto stage = [&](uint32_t st) {
        uint32_t least = 0xffffffffu, most = 0u;
        auto put = [&](float *dst, const uint32_t (&w)[3], bool half) {
            uint32_t x, y;
            join_piece(w, half, x, y);
            const uint32_t v[4] = {x << 16, x & 0xffff0000u, y << 16, y & 0xffff0000u};
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const uint32_t size = v[q] << 1;   // without its sign
                least = min(least, size - 1u);      // (zero is the largest then)
                most = max(most, size);
            }
            *reinterpret_cast<uint4 *>(dst) = make_uint4(v[0], v[1], v[2], v[3]);
        };
#pragma unroll
        for (int i = 0; i < GA; ++i) {
            const uint32_t g = i * kThreads + tid;
            put(&tiles.a[st][g / (TK / 4)][g % (TK / 4) * 4], a_next[i], halves >> i & 1u);
        }
#pragma unroll
        for (int i = 0; i < GB; ++i) {
            const uint32_t g = i * kThreads + tid;
            put(&tiles.b[st][g / (TN / 4)][g % (TN / 4) * 4], b_next[i], halves >> (GA + i) & 1u);
        }
        return least < (65u << 24) - 1u || most >= (190u << 24);
    };
    uint64_t acc[RM][RN / 2];
#pragma unroll
    for (int i = 0; i < RM; ++i)
#pragma unroll
        for (int j = 0; j < RN / 2; ++j) acc[i][j] = 0ull;   // pairs of +0.0f
    begin_after_previous();
    int wide = 0;
    if (K > 0) {
        fetch(0);
        wide = __syncthreads_or(stage(0));
    }
    uint32_t st = 0;
    for (uint32_t k0 = 0; k0 < K; k0 += TK, st ^= 1) {
        const bool more = K - k0 > (uint32_t)TK;
        if (more) fetch(k0 + TK);
        const uint32_t steps = min(K - k0, (uint32_t)TK);
        if (wide) multiply_tile<RM, RN, false>(acc, tiles.a[st], tiles.b[st], ty * RM, tx * RN, steps);
        else multiply_tile<RM, RN, true>(acc, tiles.a[st], tiles.b[st], ty * RM, tx * RN, steps);
        if (more) wide = __syncthreads_or(stage(st ^ 1));   // nobody reads that buffer: the barrier before ended its last use
    }
    write_sums<RM, RN, EPILOGUE>(acc, C, row0 + ty * RM, col0 + tx * RN, M, N, ldc, alpha, beta);
}

}  // namespace

// Function attributes are per device: called by fe2o3_ctx_create with the context's device current.  What a launch may ask for
// beside its own shared memory (see launch_gemm_exact): the limit without opt-in, 48 KiB, is for both together.
int32_t gemm_exact_init_device() {
    constexpr int kSpreadMax = 64 * 1024;
    FE2O3_CUDA(cudaFuncSetAttribute(gemm_exact_f32_kernel<2, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSpreadMax));
    FE2O3_CUDA(cudaFuncSetAttribute(gemm_exact_f32_kernel<4, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSpreadMax));
    FE2O3_CUDA(cudaFuncSetAttribute(gemm_exact_f32_kernel<8, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSpreadMax));
    return FE2O3_OK;
}

// dtype: FE2O3_DTYPE_F32 (without epilogue only) or FE2O3_DTYPE_BF16 inputs.
int32_t launch_gemm_exact(fe2o3_ctx *ctx, cudaStream_t s, uint32_t dtype, bool epilogue, uint64_t a, uint64_t b, uint64_t c,
                          uint32_t M, uint32_t N, uint32_t K, uint32_t lda, uint32_t ldb, uint32_t ldc, float alpha,
                          float beta, fe2o3_geometry *geo, bool plan_only) {
    // Tiles of f32: 16, 32 or 64 rows by 64 columns, the cheapest by a cost of the launch and, for each k, of the tiles on the SM
    // that has most, fitted in ns to 56 products of up to 4096 x 4096: the choice is within 5 % of the best.  Larger tiles read
    // less shared memory a product, smaller ones share the SMs more evenly; a tile alone on an SM waits for itself, and beyond
    // what the SMs hold at once 16 rows never win.  us, 16 / 32 / 64 rows: 512^3 15.6 / 16.6 / 32, 900 x 900 x 300 25.3 / 23.2 / 30,
    // 1024^3 90 / 94 / 96, 1200 x 1200 x 512 64 / 58 / 70, 2048 x 2048 x 256 88 / 78 / 77.
    // Where 16 x 64 leaves every other SM without a block, 16 x 32 (64 x 64 x 1024: 18.4 for 21.2).
    // bf16, whose staging costs more: 64 x 64 from four blocks an SM on (2999^3 1445 us for 1672), 32 x 64 from two
    // (500 x 2001 x 77 13.4 for 16.2), else 16 x 32 (300 x 1001 x 501 33 for 40).
    const uint64_t sms = ctx->sm_count > 0 ? ctx->sm_count : 1;
    auto count = [&](uint32_t rows, uint32_t cols) { return (uint64_t)ceil_div_u32(M, rows) * ceil_div_u32(N, cols); };
    const bool f32 = dtype == FE2O3_DTYPE_F32;
    uint32_t rows = count(64, 64) >= 4 * sms ? 64 : count(32, 64) >= 2 * sms ? 32 : 16, spread = 0;
    if (f32) {
        static const struct { uint32_t rows; double launch, tile, alone; uint32_t held, bytes; } shapes[] = {   // held: blocks that an SM holds
            {16, 2650, 12.2, 20.1, 7, sizeof(ExactTiles<2, 4, kF32Stages<2>>)},
            {32, 2700, 22.1, 27.5, 5, sizeof(ExactTiles<4, 4, kF32Stages<4>>)},
            {64, 4400, 43.2, 55.3, 4, sizeof(ExactTiles<8, 4, kF32Stages<8>>)}};
        double best = HUGE_VAL;
        for (const auto &shape : shapes) {
            const uint64_t tiles = count(shape.rows, 64), most = (tiles + sms - 1) / sms;
            if (shape.rows == 16 && most > shape.held) continue;
            const double on_sm = most <= shape.held ? (double)most : (double)tiles / (double)sms;
            const double cost = shape.launch + K * (most > 1 ? on_sm * shape.tile : shape.alone);
            if (cost >= best) continue;
            best = cost;
            rows = shape.rows;
            // Launched early, the blocks would pile up on the SMs that the kernel before leaves first, up to as many as these hold,
            // where two launches do not fit side by side (900 x 900 x 300 back to back, 32 rows: 34.7 us for 23.2): they ask
            // for so much shared memory that they spread evenly.
            spread = most <= shape.held && 2 * most > shape.held ? (228u * 1024u / (uint32_t)most - 1024u - shape.bytes) / 128u * 128u : 0u;
        }
    }
    const uint32_t cols = (f32 ? rows == 16 && 2 * count(16, 64) <= sms : rows == 16) ? 32 : 64;
    // one flat index, rows first: the second and third grid dimensions end at 65535 tiles, which either a tall or a
    // wide result can have
    const uint64_t tiles = count(rows, cols);
    if (tiles > 0x7fffffffull) { fe2o3_set_error("UnsupportedShape: too many output tiles"); return FE2O3_ERR_UNSUPPORTED_SHAPE; }
    const uint32_t grid = (uint32_t)tiles;
    if (geo) *geo = fe2o3_geometry{{grid, 1, 1}, {kThreads, 1, 1}, spread, 1};
    if (plan_only || M == 0 || N == 0) return FE2O3_OK;
    float *C = reinterpret_cast<float *>(c);
    cudaError_t e;
    if (f32) {
        const float *A = reinterpret_cast<const float *>(a), *B = reinterpret_cast<const float *>(b);
        auto kernel = cols == 32 ? gemm_exact_f32_kernel<2, 2> : rows == 16 ? gemm_exact_f32_kernel<2, 4> : rows == 32 ? gemm_exact_f32_kernel<4, 4> : gemm_exact_f32_kernel<8, 4>;
        e = fe2o3_launch_early(kernel, grid, kThreads, spread, s, 1, A, B, C, M, N, K, lda, ldb, ldc, alpha, beta);
    } else {
        const uint16_t *A = reinterpret_cast<const uint16_t *>(a), *B = reinterpret_cast<const uint16_t *>(b);
        auto kernel = epilogue ? (rows == 64   ? gemm_exact_bf16_kernel<8, 4, true>
                                  : rows == 32 ? gemm_exact_bf16_kernel<4, 4, true>
                                               : gemm_exact_bf16_kernel<2, 2, true>)
                               : (rows == 64   ? gemm_exact_bf16_kernel<8, 4, false>
                                  : rows == 32 ? gemm_exact_bf16_kernel<4, 4, false>
                                               : gemm_exact_bf16_kernel<2, 2, false>);
        e = fe2o3_launch_early(kernel, grid, kThreads, 0, s, 1, A, B, C, M, N, K, lda, ldb, ldc, alpha, beta);
    }
    fe2o3_count_launch(1);
    return fe2o3_cuda_status(e, "gemm_exact");
}

static Fe2o3KernelRegistration reg_scalar("scalar_gemm_v1", reinterpret_cast<const void *>(gemm_exact_f32_kernel<2, 4>));
