// Row softmax: examples/row_softmax_v1/src/kernel.rs:13-42 generalised from one
// 64-element row to rows x cols, with the oracle's optional activity mask
// (src/numerical_contract.rs:130-199): f32 maximum over active elements,
// weights exp(x - max), row sum, quotient; masked outputs are +0.0; a row with
// a non-finite physical input or no active element is left unwritten and a
// status word is recorded instead of trapping.
//
// HBM-bound: each element is read once and written once (8 bytes per element, 9
// with a mask).  A row lives in the registers of LANES threads (8 to 32 lanes of a
// warp, or two or four warps), NV 16-byte vectors each, so every byte of a row is
// requested before the first one is needed and the row is never read again.
//   Rows whose start is not 16-byte aligned (cols not a multiple of 4, or an
//   unaligned base) are still read and written as aligned vectors: the row is
//   covered from the aligned address at or before its start, elements outside it
//   count as inactive, and only the vectors that straddle a row end fall apart
//   into single elements.
//   An inactive element is carried as -inf: its weight is exp(-inf) = +0, no mask
//   bits stay in registers.
//   Rows of up to 64 columns share a warp (8 or 16 lanes a row), otherwise most
//   lanes of the warp would idle.
//   There is a build for every number of vectors a thread: what a row does not need
//   costs instructions (5000 rows of 3001 columns are as much issue time as traffic) and
//   registers, hence blocks an SM.
// 65536 x 1024: 91.6 us -> 79.5 us (6.75 TB/s) against the earlier form that kept
// activity bits per element; 5000 x 3001 masked: 79.9 -> 29.3 us against one block
// per row with scalar accesses, four block barriers and a division per element, and
// -> 24.9 (5.4 TB/s) with six vectors a thread instead of eight (25.5) and the tests for
// the row's ends and for finite inputs only where they are needed; 8000 x 2560 28.3 -> 25.5,
// 20000 x 701 22.6 -> 19.4.  Two warps a row of 3001 with twelve vectors a thread take 26.9,
// one with 24 takes 39.
// Input, output and mask that are not aligned to one another (views at different
// offsets) take one block per row with scalar accesses.
#include "common.cuh"

namespace {

__device__ __forceinline__ bool finite4(float4 v) {
    return isfinite(v.x) && isfinite(v.y) && isfinite(v.z) && isfinite(v.w);
}

constexpr int kThreads = 256, kMaxCols = 4096;

// Combines over the LANES threads of a row; every one receives the result.  Up to 32 lanes: a shuffle
// tree.  More: each warp leaves its value in shared memory (`slots`, one per warp of the row) and the row's
// warps meet at a named barrier of their own.
template <int LANES, typename F>
__device__ __forceinline__ float row_combine(float v, F op, float *slots, uint32_t barrier) {
    constexpr int kTree = LANES < 32 ? LANES : 32;
#pragma unroll
    for (int off = kTree / 2; off >= 1; off >>= 1) v = op(v, __shfl_xor_sync(0xffffffffu, v, off));
    if constexpr (LANES > 32) {
        constexpr int kWarps = LANES / 32;
        const uint32_t w = (threadIdx.x >> 5) % kWarps;
        if ((threadIdx.x & 31) == 0) slots[w] = v;
        asm volatile("bar.sync %0, %1;" ::"r"(barrier), "n"(LANES) : "memory");
        v = slots[0];
#pragma unroll
        for (int i = 1; i < kWarps; ++i) v = op(v, slots[i]);
    }
    return v;
}

// SHIFTED: rows may start anywhere in a 16-byte vector (same phase for input and output, the mask's
// 4-byte phase alike); otherwise every row starts on a vector and cols is a multiple of 4.
#pragma nv_diag_suppress 186   // rows that start on a vector compare with a shift of 0
template <int LANES, int NV, bool MASKED, bool SHIFTED>
__global__ void __launch_bounds__(kThreads)
row_softmax_kernel(const float *__restrict__ in, float *__restrict__ out, const uint8_t *__restrict__ mask, uint32_t rows,
                   uint32_t cols, uint32_t *status) {
    constexpr int kRowsPerBlock = kThreads / LANES;
    __shared__ float s_red[LANES > 32 ? 2 : 1][kThreads / 32];   // one set per exchange: no barrier before the next one
    const uint32_t local = threadIdx.x / LANES, lane = threadIdx.x % LANES;
    begin_after_previous();
    uint32_t row = blockIdx.x * kRowsPerBlock + local;
    // a warp may hold several rows, all of which take part in its shuffles: those past the end redo the last row
    const bool beyond = row >= rows;
    if (beyond) {
        if (LANES >= 32) return;   // whole warps, and with them whole row groups
        row = rows - 1;
    }
    const uint64_t base = (uint64_t)row * cols;
    const uint32_t shift = SHIFTED ? (uint32_t)(((reinterpret_cast<uintptr_t>(in) >> 2) + base) & 3u) : 0u;
    const float *src = in + base - shift;      // aligned; elements [shift, shift + cols) are the row
    float *dst = out + base - shift;
    const uint8_t *msk = MASKED ? mask + base - shift : nullptr;
    const uint32_t end = shift + cols;

    // No thread has vectors to spare (launch_row_softmax), so only the first and the last ones can straddle an end of the row or
    // lie outside it; shifted rows may end one vector earlier.  (Aligned rows under a mask keep the test at every vector:
    // without it the compiler takes other registers, and 16384 x 2000 goes from 45.5 to 47.5 us.  So do four shifted ones under a
    // mask: with one vector of them inside, it makes do with 32 registers, and 5000 x 401 takes 5.77 us for 4.91.)
    auto inside = [](int i) { return SHIFTED ? !(MASKED && NV == 4) && i > 0 && i < NV - 2 : !MASKED && i < NV - 1; };
    // One vector a thread without a mask has the ends of the row in every thread: tests there are cheaper than fillers put right
    // (60000 x 101 13.2 / 13.7 us; under a mask 16.2 / 15.2).
    constexpr bool kZeros = SHIFTED && (MASKED || NV > 1);   // what lies outside the row is filled with zeros, else with -inf
    float4 v[NV];
    float poison = 0.f;   // NaN once an input was not finite
    bool ok = true;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const uint32_t e = (i * LANES + lane) * 4;
        v[i] = kZeros ? make_float4(0.f, 0.f, 0.f, 0.f) : make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
        const bool whole = inside(i) || (SHIFTED ? e >= shift && e + 4 <= end : e < end);
        if (whole) {
            v[i] = __ldcs(reinterpret_cast<const float4 *>(src + e));
        } else if (SHIFTED && e < end) {   // straddles an end of the row (e + 4 > shift always: shift < 4)
            if (e + 0 >= shift && e + 0 < end) v[i].x = src[e];
            if (e + 1 >= shift && e + 1 < end) v[i].y = src[e + 1];
            if (e + 2 >= shift && e + 2 < end) v[i].z = src[e + 2];
            if (e + 3 >= shift && e + 3 < end) v[i].w = src[e + 3];
        }
    }
    uint32_t m4[NV];
    if (MASKED) {
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const uint32_t e = (i * LANES + lane) * 4;
            m4[i] = 0;
            const bool whole = inside(i) || (SHIFTED ? e >= shift && e + 4 <= end : e < end);
            if (whole) {
                m4[i] = *reinterpret_cast<const uint32_t *>(msk + e);
            } else if (SHIFTED && e < end) {
#pragma unroll
                for (uint32_t q = 0; q < 4; ++q)
                    if (e + q >= shift && e + q < end) m4[i] |= (uint32_t)msk[e + q] << (8 * q);
            }
        }
    }
    float mx = -INFINITY;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const uint32_t e = (i * LANES + lane) * 4;
        if (kZeros) {
            poison = fmaf(v[i].x, 0.f, fmaf(v[i].y, 0.f, fmaf(v[i].z, 0.f, fmaf(v[i].w, 0.f, poison))));
            const bool whole = inside(i) || (e >= shift && e + 4 <= end);
            if (!MASKED && !whole) {   // (the mask's words hold zeros there)
                if (e + 0 < shift || e + 0 >= end) v[i].x = -INFINITY;
                if (e + 1 < shift || e + 1 >= end) v[i].y = -INFINITY;
                if (e + 2 < shift || e + 2 >= end) v[i].z = -INFINITY;
                if (e + 3 < shift || e + 3 >= end) v[i].w = -INFINITY;
            }
        } else if (SHIFTED) {   // the filler outside the row is not an input
            ok = ok && (e + 0 < shift || e + 0 >= end || isfinite(v[i].x)) && (e + 1 < shift || e + 1 >= end || isfinite(v[i].y)) &&
                 (e + 2 < shift || e + 2 >= end || isfinite(v[i].z)) && (e + 3 >= end || isfinite(v[i].w));
        } else {
            ok = ok && (inside(i) || e < end ? finite4(v[i]) : true);
        }
        if (MASKED) {
            if ((m4[i] & 0xffu) == 0) v[i].x = -INFINITY;
            if ((m4[i] & 0xff00u) == 0) v[i].y = -INFINITY;
            if ((m4[i] & 0xff0000u) == 0) v[i].z = -INFINITY;
            if ((m4[i] & 0xff000000u) == 0) v[i].w = -INFINITY;
        }
        mx = fmaxf(mx, fmaxf(fmaxf(v[i].x, v[i].y), fmaxf(v[i].z, v[i].w)));
    }
    const uint32_t barrier = 1 + local;
    float *slots = &s_red[0][0] + local * (LANES / 32);
    // a non-finite input anywhere in the row travels with the maximum, as +inf, which no row of finite inputs has
    mx = row_combine<LANES>(ok && poison == 0.f ? mx : INFINITY, [](float a, float b) { return fmaxf(a, b); }, slots, barrier);
    const bool good = mx != INFINITY && mx != -INFINITY;   // -inf: no active element
    float sum = 0.f;
    if (good) {
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            v[i].x = expf(v[i].x - mx);
            v[i].y = expf(v[i].y - mx);
            v[i].z = expf(v[i].z - mx);
            v[i].w = expf(v[i].w - mx);
            sum += (v[i].x + v[i].y) + (v[i].z + v[i].w);
        }
    }
    sum = row_combine<LANES>(sum, [](float a, float b) { return a + b; }, slots + kThreads / 32, barrier);
    if (!good) {
        if (lane == 0) kstatus_set(status, FE2O3_KSTATUS_NONFINITE);
        return;
    }
    if (beyond) return;
    const float inv = 1.0f / sum;  // one IEEE division per row
    // quotient with Markstein's correction step: the residual of w * inv against w, folded back in
    auto quotient = [&](float w) {
        const float q = w * inv;
        return fmaf(fmaf(-q, sum, w), inv, q);
    };
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const uint32_t e = (i * LANES + lane) * 4;
        const bool whole = inside(i) || (SHIFTED ? e >= shift && e + 4 <= end : e < end);
        const float4 r = make_float4(quotient(v[i].x), quotient(v[i].y), quotient(v[i].z), quotient(v[i].w));
        if (whole) {
            __stcs(reinterpret_cast<float4 *>(dst + e), r);
        } else if (SHIFTED && e < end) {
            if (e + 0 >= shift && e + 0 < end) dst[e] = r.x;
            if (e + 1 >= shift && e + 1 < end) dst[e + 1] = r.y;
            if (e + 2 >= shift && e + 2 < end) dst[e + 2] = r.z;
            if (e + 3 >= shift && e + 3 < end) dst[e + 3] = r.w;
        }
    }
}

#pragma nv_diag_default 186

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, off));
    return v;
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    return v;
}

// One 256-thread block per row, scalar accesses: any alignment.
constexpr int kBlockRowItems = kMaxCols / kThreads;

__global__ void __launch_bounds__(kThreads)
row_softmax_block_kernel(const float *__restrict__ in, float *__restrict__ out, const uint8_t *__restrict__ mask,
                         uint32_t rows, uint32_t cols, uint32_t *status) {
    __shared__ float red[kThreads / 32];
    __shared__ int flags[2];
    const uint32_t row = blockIdx.x;
    begin_after_previous();
    if (row >= rows) return;
    const float *src = in + (uint64_t)row * cols;
    const uint8_t *msk = mask ? mask + (uint64_t)row * cols : nullptr;
    float v[kBlockRowItems];
    bool on[kBlockRowItems];
    if (threadIdx.x == 0) { flags[0] = 1; flags[1] = 0; }
    __syncthreads();
    bool ok = true, any = false;
    float mx = -INFINITY;
#pragma unroll
    for (int i = 0; i < kBlockRowItems; ++i) {
        const uint32_t c = i * kThreads + threadIdx.x;
        on[i] = false;
        v[i] = 0.f;
        if (c < cols) {
            v[i] = src[c];
            ok = ok && isfinite(v[i]);
            on[i] = msk ? (msk[c] != 0) : true;
            if (on[i]) { mx = fmaxf(mx, v[i]); any = true; }
        }
    }
    if (!ok) atomicExch(&flags[0], 0);
    if (any) atomicExch(&flags[1], 1);
    mx = warp_max(mx);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = mx;
    __syncthreads();
    if (!flags[0] || !flags[1]) {
        if (threadIdx.x == 0) kstatus_set(status, FE2O3_KSTATUS_NONFINITE);
        return;
    }
    mx = red[0];
#pragma unroll
    for (int w = 1; w < kThreads / 32; ++w) mx = fmaxf(mx, red[w]);
    __syncthreads();
    float sum = 0.f;
#pragma unroll
    for (int i = 0; i < kBlockRowItems; ++i) {
        v[i] = on[i] ? expf(v[i] - mx) : 0.f;
        sum += v[i];
    }
    sum = warp_sum(sum);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = sum;
    __syncthreads();
    sum = 0.f;
#pragma unroll
    for (int w = 0; w < kThreads / 32; ++w) sum += red[w];
    float *dst = out + (uint64_t)row * cols;
#pragma unroll
    for (int i = 0; i < kBlockRowItems; ++i) {
        const uint32_t c = i * kThreads + threadIdx.x;
        if (c < cols) dst[c] = on[i] ? v[i] / sum : 0.0f;
    }
}

template <int LANES, int NV>
cudaError_t launch_row(const fe2o3_row_softmax_v1_args *a, bool shifted, cudaStream_t s, uint32_t grid, uint32_t *status) {
    const float *in = reinterpret_cast<const float *>(a->input.ptr);
    float *out = reinterpret_cast<float *>(a->output.ptr);
    const uint8_t *mask = reinterpret_cast<const uint8_t *>(a->mask.ptr);
    auto kernel = mask ? row_softmax_kernel<LANES, NV, true, true> : row_softmax_kernel<LANES, NV, false, true>;
    if constexpr (LANES * NV <= kMaxCols / 4)   // more vectors than that only rows have that start inside one
        if (!shifted) kernel = mask ? row_softmax_kernel<LANES, NV, true, false> : row_softmax_kernel<LANES, NV, false, false>;
    return fe2o3_launch_early(kernel, grid, kThreads, 0, s, 1, in, out, mask, a->rows, a->cols, status);
}

}  // namespace

int32_t launch_row_softmax(fe2o3_ctx *ctx, cudaStream_t s, const void *args, fe2o3_geometry *geo, bool plan_only) {
    const fe2o3_row_softmax_v1_args *a = static_cast<const fe2o3_row_softmax_v1_args *>(args);
    // vectors need one phase for all three arrays: elements of a 16-byte input vector, of a 16-byte output vector
    // and of a 4-byte mask word must be the same ones
    const bool vec = ((a->input.ptr ^ a->output.ptr) & 15u) == 0 &&
                     (a->mask.ptr == 0 || ((a->input.ptr >> 2) & 3u) == (a->mask.ptr & 3u));
    const bool shifted = (a->cols & 3u) != 0 || (a->input.ptr & 15u) != 0;
    // threads per row: the most vectors any row covers, with the largest phase that can occur
    const uint32_t vectors = ((shifted ? 3u : 0u) + a->cols + 3u) / 4u;
    uint32_t lanes = vectors <= 8 ? 8 : vectors <= 16 ? 16 : vectors <= 256 ? 32 : vectors <= 512 ? 64 : 128;
    const uint32_t grid = vec ? ceil_div_u32(a->rows, kThreads / lanes) : a->rows;
    if (geo) *geo = fe2o3_geometry{{grid, 1, 1}, {kThreads, 1, 1}, 0, 1};
    if (plan_only || a->rows == 0) return FE2O3_OK;
    cudaError_t e;
    if (vec) {
        uint32_t *st = ctx->status_word;
        switch ((vectors + lanes - 1) / lanes) {
            case 1:
                if (lanes == 8) e = launch_row<8, 1>(a, shifted, s, grid, st);
                else if (lanes == 16) e = launch_row<16, 1>(a, shifted, s, grid, st);
                else e = launch_row<32, 1>(a, shifted, s, grid, st);
                break;
            case 2: e = launch_row<32, 2>(a, shifted, s, grid, st); break;
            case 3: e = launch_row<32, 3>(a, shifted, s, grid, st); break;
            case 4: e = launch_row<32, 4>(a, shifted, s, grid, st); break;
            case 5:
                if (lanes == 32) e = launch_row<32, 5>(a, shifted, s, grid, st);
                else if (lanes == 64) e = launch_row<64, 5>(a, shifted, s, grid, st);
                else e = launch_row<128, 5>(a, shifted, s, grid, st);
                break;
            case 6:
                if (lanes == 32) e = launch_row<32, 6>(a, shifted, s, grid, st);
                else if (lanes == 64) e = launch_row<64, 6>(a, shifted, s, grid, st);
                else e = launch_row<128, 6>(a, shifted, s, grid, st);
                break;
            case 7:
                if (lanes == 32) e = launch_row<32, 7>(a, shifted, s, grid, st);
                else if (lanes == 64) e = launch_row<64, 7>(a, shifted, s, grid, st);
                else e = launch_row<128, 7>(a, shifted, s, grid, st);
                break;
            case 9: e = launch_row<128, 9>(a, shifted, s, grid, st); break;   // up to 1025 vectors: 4095 columns at phase 3
            default:
                if (lanes == 32) e = launch_row<32, 8>(a, shifted, s, grid, st);
                else if (lanes == 64) e = launch_row<64, 8>(a, shifted, s, grid, st);
                else e = launch_row<128, 8>(a, shifted, s, grid, st);
        }
    } else {
        e = fe2o3_launch_early(row_softmax_block_kernel, grid, kThreads, 0, s, 1,
            reinterpret_cast<const float *>(a->input.ptr), reinterpret_cast<float *>(a->output.ptr),
            reinterpret_cast<const uint8_t *>(a->mask.ptr), a->rows, a->cols, ctx->status_word);
    }
    fe2o3_count_launch(1);
    return fe2o3_cuda_status(e, "row_softmax_v1");
}

static Fe2o3KernelRegistration reg_softmax("row_softmax_v1", reinterpret_cast<const void *>(row_softmax_kernel<32, 8, false, false>));
