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
// Bound: the f32 pipe, two operations per multiply-add that may not be fused
// (512^3: 7.5 us on 148 SMs).  The sizes that come here are small, so the tile is
// 32x64 outputs per 128-thread block, which makes 128 blocks of a 512x512 result
// (64x64 tiles made 64 blocks for 148 SMs): one warp per scheduler, each thread
// with 4x4 outputs.  The 16 chains advance by 16 products and eight packed f32x2
// sums per k (each half rounded exactly like the scalar instruction; the products
// stay scalar because a packed product feeding a packed sum came out fused, with
// one rounding), enough independent work for one warp to cover the latency of the
// additions; operands
// come as one 16-byte shared-memory read each per k, and the next 32-deep k block
// is on its way from global memory in registers while the current one is
// multiplied (two shared-memory buffers, one barrier per block).  512^3: 51.2 us a
// launch with 64x64 tiles and a single buffer, 19.0 us so.
#include "common.cuh"

namespace {

constexpr int TM = 32, TN = 64, TK = 32, kThreads = 128;

template <typename T>
__device__ __forceinline__ float widen(T v);
template <>
__device__ __forceinline__ float widen<float>(float v) { return v; }
template <>
__device__ __forceinline__ float widen<uint16_t>(uint16_t v) { return bf16_bits_to_f32(v); }

// Four consecutive elements of a row, widened; `vec` when all four exist and their address is aligned to their size.
__device__ __forceinline__ float4 load4(const float *p) { return __ldg(reinterpret_cast<const float4 *>(p)); }
__device__ __forceinline__ float4 load4(const uint16_t *p) {
    const uint2 w = __ldg(reinterpret_cast<const uint2 *>(p));
    return make_float4(__uint_as_float(w.x << 16), __uint_as_float(w.x & 0xffff0000u), __uint_as_float(w.y << 16),
                       __uint_as_float(w.y & 0xffff0000u));
}
template <typename T>
__device__ __forceinline__ float4 load4_guarded(const T *row, uint32_t first, uint32_t end, bool row_ok, bool vec) {
    if (row_ok && vec && first + 4 <= end) return load4(row + first);
    float v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = row_ok && first + i < end ? widen<T>(row[first + i]) : 0.0f;
    return make_float4(v[0], v[1], v[2], v[3]);
}

template <typename T, bool EPILOGUE>
__global__ void __launch_bounds__(kThreads)
gemm_exact_kernel(const T *__restrict__ A, const T *__restrict__ B, float *C, uint32_t M, uint32_t N, uint32_t K,
                  uint32_t lda, uint32_t ldb, uint32_t ldc, float alpha, float beta) {
    __shared__ __align__(16) float As[2][TK][TM + 4];   // k-major, so that a thread's four rows are one 16-byte read
    __shared__ __align__(16) float Bs[2][TK][TN];
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const uint32_t row_tiles = (M - 1) / TM + 1;
    const uint32_t row0 = blockIdx.x % row_tiles * TM, col0 = blockIdx.x / row_tiles * TN;
    const bool vec_a = lda % 4 == 0 && reinterpret_cast<uintptr_t>(A) % (4 * sizeof(T)) == 0;
    const bool vec_b = ldb % 4 == 0 && reinterpret_cast<uintptr_t>(B) % (4 * sizeof(T)) == 0;

    // A: row = thread / 4, eight k values in two groups of four, 16 apart; B: 16 groups of four columns, 8 k rows a pass
    const uint32_t ar = threadIdx.x >> 2, ak = (threadIdx.x & 3) * 4;
    const uint32_t bc = tx * 4, bk = ty;
    const bool a_ok = row0 + ar < M;
    const T *a_row = A + (uint64_t)(a_ok ? row0 + ar : 0) * lda;
    float4 a_next[2], b_next[4];
    auto fetch = [&](uint32_t k0) {
#pragma unroll
        for (int i = 0; i < 2; ++i) a_next[i] = load4_guarded<T>(a_row, k0 + ak + i * 16, K, a_ok, vec_a);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint32_t k = k0 + bk + i * 8;
            b_next[i] = load4_guarded<T>(B + (uint64_t)(k < K ? k : 0) * ldb, col0 + bc, N, k < K, vec_b);
        }
    };
    auto stage = [&](int buf) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            As[buf][ak + i * 16 + 0][ar] = a_next[i].x;
            As[buf][ak + i * 16 + 1][ar] = a_next[i].y;
            As[buf][ak + i * 16 + 2][ar] = a_next[i].z;
            As[buf][ak + i * 16 + 3][ar] = a_next[i].w;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) *reinterpret_cast<float4 *>(&Bs[buf][bk + i * 8][bc]) = b_next[i];
    };

    uint64_t acc[4][2];   // rows ty*4 + i, columns tx*4 + {0,1} and {2,3}
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[i][0] = acc[i][1] = 0ull;   // pairs of +0.0f
    auto step = [&](int buf, int kk) {
        const float4 a = *reinterpret_cast<const float4 *>(&As[buf][kk][ty * 4]);
        const float4 b = *reinterpret_cast<const float4 *>(&Bs[buf][kk][tx * 4]);
        const float av[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            acc[i][0] = add_f32x2(acc[i][0], pack_f32x2(__fmul_rn(av[i], b.x), __fmul_rn(av[i], b.y)));
            acc[i][1] = add_f32x2(acc[i][1], pack_f32x2(__fmul_rn(av[i], b.z), __fmul_rn(av[i], b.w)));
        }
    };

    begin_after_previous();
    if (K > 0) {
        fetch(0);
        stage(0);
        __syncthreads();
    }
    int buf = 0;
    for (uint32_t k0 = 0; k0 < K; k0 += TK, buf ^= 1) {
        const bool more = k0 + TK < K;
        if (more) fetch(k0 + TK);
        if (K - k0 >= (uint32_t)TK) {
#pragma unroll
            for (int kk = 0; kk < TK; ++kk) step(buf, kk);
        } else {
            // the recurrence stops at K: the zero padding of the last block is never multiplied
            const int kmax = (int)(K - k0);
            for (int kk = 0; kk < kmax; ++kk) step(buf, kk);
        }
        if (more) stage(buf ^ 1);   // nobody reads that buffer: the barrier below ended its last use
        __syncthreads();
    }
    const bool vec_c = ldc % 4 == 0 && reinterpret_cast<uintptr_t>(C) % 16 == 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t r = row0 + ty * 4 + i, c0 = col0 + tx * 4;
        if (r >= M) continue;
        float v[4];
        unpack_f32x2(acc[i][0], v[0], v[1]);
        unpack_f32x2(acc[i][1], v[2], v[3]);
        float *dst = C + (uint64_t)r * ldc + c0;
        if (vec_c && c0 + 4 <= N) {
            if (EPILOGUE) {
                const float4 old = *reinterpret_cast<const float4 *>(dst);
                const float o[4] = {old.x, old.y, old.z, old.w};
#pragma unroll
                for (int j = 0; j < 4; ++j) v[j] = __fadd_rn(__fmul_rn(alpha, v[j]), __fmul_rn(beta, o[j]));
            }
            *reinterpret_cast<float4 *>(dst) = make_float4(v[0], v[1], v[2], v[3]);
            continue;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (c0 + j >= N) continue;
            dst[j] = EPILOGUE ? __fadd_rn(__fmul_rn(alpha, v[j]), __fmul_rn(beta, dst[j])) : v[j];
        }
    }
}

}  // namespace

// dtype: FE2O3_DTYPE_F32 or FE2O3_DTYPE_BF16 inputs.
int32_t launch_gemm_exact(cudaStream_t s, uint32_t dtype, bool epilogue, uint64_t a, uint64_t b, uint64_t c,
                          uint32_t M, uint32_t N, uint32_t K, uint32_t lda, uint32_t ldb, uint32_t ldc, float alpha,
                          float beta, fe2o3_geometry *geo, bool plan_only) {
    // one flat index, rows first: the second and third grid dimensions end at 65535 tiles, which either a tall or a
    // wide result can have
    const uint64_t tiles = (uint64_t)ceil_div_u32(M, TM) * ceil_div_u32(N, TN);
    if (tiles > 0x7fffffffull) { fe2o3_set_error("UnsupportedShape: too many output tiles"); return FE2O3_ERR_UNSUPPORTED_SHAPE; }
    const uint32_t grid = (uint32_t)tiles;
    if (geo) *geo = fe2o3_geometry{{grid, 1, 1}, {kThreads, 1, 1}, 0, 1};
    if (plan_only || M == 0 || N == 0) return FE2O3_OK;
    float *C = reinterpret_cast<float *>(c);
    cudaError_t e;
    if (dtype == FE2O3_DTYPE_F32) {
        const float *A = reinterpret_cast<const float *>(a), *B = reinterpret_cast<const float *>(b);
        e = fe2o3_launch_early(epilogue ? gemm_exact_kernel<float, true> : gemm_exact_kernel<float, false>, grid, kThreads, 0, s, 1, A, B, C, M, N, K, lda, ldb, ldc, alpha, beta);
    } else {
        const uint16_t *A = reinterpret_cast<const uint16_t *>(a), *B = reinterpret_cast<const uint16_t *>(b);
        e = fe2o3_launch_early(epilogue ? gemm_exact_kernel<uint16_t, true> : gemm_exact_kernel<uint16_t, false>, grid, kThreads, 0, s, 1, A, B, C, M, N, K, lda, ldb, ldc, alpha, beta);
    }
    fe2o3_count_launch(1);
    return fe2o3_cuda_status(e, "gemm_exact");
}

static Fe2o3KernelRegistration reg_scalar("scalar_gemm_v1", reinterpret_cast<const void *>(gemm_exact_kernel<float, false>));
