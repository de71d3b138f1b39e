// CUDA-core attention: the recurrence of attention_row.cuh for any [B][H][S][D] shape, f32
// or bf16 inputs, causal or not.  One warp owns one query row; lanes split the
// head dimension.  It serves the fixed f32 B1/H1/N8/D16 profile and every shape
// the tensor-core kernels do not admit.
#include "attention_row.cuh"

namespace {

constexpr int kMaxPerLane = 8;  // head_dim <= 256

template <typename T>
__global__ void __launch_bounds__(128)
attention_simt_kernel(const T *__restrict__ q, const T *__restrict__ k, const T *__restrict__ v,
                      float *__restrict__ out, uint32_t bh, uint32_t seq, uint32_t dim, float scale, uint32_t causal,
                      uint32_t *status) {
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t row = (uint64_t)blockIdx.x * 4 + (threadIdx.x >> 5);
    if (row >= (uint64_t)bh * seq) return;
    const uint32_t head = (uint32_t)(row / seq), qr = (uint32_t)(row % seq);
    // finite-input policy: a row that reads a non-finite value is left unwritten, and a status word recorded
    if (!attention_row<T, kMaxPerLane, 1, true>(q, k, v, out, (uint64_t)head * seq * dim, qr, causal ? qr + 1 : seq, dim, scale, lane,
                                            [](uint32_t) {}) && lane == 0)
        kstatus_set(status, FE2O3_KSTATUS_NONFINITE);
}

}  // namespace

int32_t launch_attention_simt(fe2o3_ctx *ctx, cudaStream_t s, const fe2o3_flash_attention_v1_args *a,
                              fe2o3_geometry *geo, bool plan_only) {
    const uint64_t rows = (uint64_t)a->batch * a->heads * a->seq;
    const uint32_t grid = ceil_div_u32(rows, 4);
    if (geo) *geo = fe2o3_geometry{{grid, 1, 1}, {128, 1, 1}, 0, 1};
    if (plan_only || rows == 0) return FE2O3_OK;
    float *out = reinterpret_cast<float *>(a->output.ptr);
    if (a->input_dtype == FE2O3_DTYPE_F32)
        attention_simt_kernel<float><<<grid, 128, 0, s>>>(
            reinterpret_cast<const float *>(a->q.ptr), reinterpret_cast<const float *>(a->k.ptr),
            reinterpret_cast<const float *>(a->v.ptr), out, a->batch * a->heads, a->seq, a->dim, a->scale, a->causal,
            ctx->status_word);
    else
        attention_simt_kernel<uint16_t><<<grid, 128, 0, s>>>(
            reinterpret_cast<const uint16_t *>(a->q.ptr), reinterpret_cast<const uint16_t *>(a->k.ptr),
            reinterpret_cast<const uint16_t *>(a->v.ptr), out, a->batch * a->heads, a->seq, a->dim, a->scale,
            a->causal, ctx->status_word);
    fe2o3_count_launch(1);
    return fe2o3_cuda_status(cudaGetLastError(), "flash_attention_v1(simt)");
}
