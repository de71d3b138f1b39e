// One query row of attention on the CUDA cores by one warp: the reference kernel's per-key online recurrence
// (examples/flash_attention_v1/src/kernel.rs:56-113: m' = max(m, s),
// p = exp(m - m'), c = exp(s - m'), l = l*p + c, acc = acc*p + v*c, out = acc/l,
// first key initialises m = s, l = 1, acc = v).  Lanes split the head dimension.
#pragma once
#include "common.cuh"

template <typename T>
__device__ __forceinline__ float attention_ld(const T *p, uint64_t i);
template <>
__device__ __forceinline__ float attention_ld<float>(const float *p, uint64_t i) { return p[i]; }
template <>
__device__ __forceinline__ float attention_ld<uint16_t>(const uint16_t *p, uint64_t i) { return bf16_bits_to_f32(p[i]); }

// Row `qr` of the head at element `base` over its first `keys` keys, written to `out` unless a value that the row reads
// or its sum is not finite; false then.  PER_LANE * 32 >= dim.  STOP_EARLY ends at the first such value.
template <typename T, int PER_LANE, bool STOP_EARLY>
__device__ __forceinline__ bool attention_row(const T *__restrict__ q, const T *__restrict__ k, const T *__restrict__ v,
                                              float *__restrict__ out, uint64_t base, uint32_t qr, uint32_t keys,
                                              uint32_t dim, float scale, uint32_t lane) {
    float qv[PER_LANE], acc[PER_LANE];
    bool finite = true;
#pragma unroll
    for (int i = 0; i < PER_LANE; ++i) {
        const uint32_t f = lane + 32 * i;
        qv[i] = f < dim ? attention_ld<T>(q, base + (uint64_t)qr * dim + f) : 0.0f;
        acc[i] = 0.0f;
        finite = finite && isfinite(qv[i]);
    }
    float m = 0.0f, l = 0.0f;
    for (uint32_t kr = 0; kr < keys; ++kr) {
        float part = 0.0f;
        float vv[PER_LANE];
#pragma unroll
        for (int i = 0; i < PER_LANE; ++i) {
            const uint32_t f = lane + 32 * i;
            float kv = 0.0f;
            vv[i] = 0.0f;
            if (f < dim) {
                kv = attention_ld<T>(k, base + (uint64_t)kr * dim + f);
                vv[i] = attention_ld<T>(v, base + (uint64_t)kr * dim + f);
            }
            finite = finite && isfinite(kv) && isfinite(vv[i]);
            part = fmaf(qv[i], kv, part);
        }
        if (STOP_EARLY && !__all_sync(0xffffffffu, finite)) return false;
#pragma unroll
        for (int off = 16; off >= 1; off >>= 1) part += __shfl_xor_sync(0xffffffffu, part, off);
        const float s = part * scale;
        if (kr == 0) {
            m = s;
            l = 1.0f;
#pragma unroll
            for (int i = 0; i < PER_LANE; ++i) acc[i] = vv[i];
            continue;
        }
        const float nm = fmaxf(m, s);
        const float pw = expf(m - nm), cw = expf(s - nm);
        l = l * pw + cw;
#pragma unroll
        for (int i = 0; i < PER_LANE; ++i) acc[i] = acc[i] * pw + vv[i] * cw;
        m = nm;
    }
    if (!__all_sync(0xffffffffu, finite && isfinite(l) && l > 0.0f)) return false;
#pragma unroll
    for (int i = 0; i < PER_LANE; ++i) {
        const uint32_t f = lane + 32 * i;
        if (f < dim) out[base + (uint64_t)qr * dim + f] = acc[i] / l;
    }
    return true;
}
