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
// or its sum is not finite; false then.  PER_LANE * 32 >= dim.  AHEAD keys are fetched together and their scores summed up
// side by side, with the same result for any AHEAD.  CHECK: the keys may hold non-finite values.  A row may take long:
// `tick` is called every AHEAD keys.
template <typename T, int PER_LANE, int AHEAD, bool CHECK, typename Tick>
__device__ __forceinline__ bool attention_row(const T *__restrict__ q, const T *__restrict__ k, const T *__restrict__ v,
                                              float *__restrict__ out, uint64_t base, uint32_t qr, uint32_t keys,
                                              uint32_t dim, float scale, uint32_t lane, Tick tick) {
    float qv[PER_LANE], acc[PER_LANE];
    bool finite = true;
#pragma unroll
    for (int i = 0; i < PER_LANE; ++i) {
        const uint32_t f = lane + 32 * i;
        qv[i] = f < dim ? attention_ld<T>(q, base + (uint64_t)qr * dim + f) : 0.0f;
        acc[i] = 0.0f;
        finite = finite && isfinite(qv[i]);
    }
    if (!__all_sync(0xffffffffu, finite)) return false;
    float m = 0.0f, l = 0.0f;
    for (uint32_t k0 = 0; k0 < keys; k0 += AHEAD) {
        tick(k0);
        float part[AHEAD], vv[AHEAD][PER_LANE];
#pragma unroll
        for (int a = 0; a < AHEAD; ++a) {
            const uint32_t kr = k0 + a;
            part[a] = 0.0f;
#pragma unroll
            for (int i = 0; i < PER_LANE; ++i) {
                const uint32_t f = lane + 32 * i;
                float kv = 0.0f;
                vv[a][i] = 0.0f;
                if (f < dim && (AHEAD == 1 || kr < keys)) {
                    kv = attention_ld<T>(k, base + (uint64_t)kr * dim + f);
                    vv[a][i] = attention_ld<T>(v, base + (uint64_t)kr * dim + f);
                }
                if (CHECK) finite = finite && isfinite(kv) && isfinite(vv[a][i]);
                part[a] = fmaf(qv[i], kv, part[a]);
            }
        }
#pragma unroll
        for (int off = 16; off >= 1; off >>= 1) {
#pragma unroll
            for (int a = 0; a < AHEAD; ++a) part[a] += __shfl_xor_sync(0xffffffffu, part[a], off);
        }
#pragma unroll
        for (int a = 0; a < AHEAD; ++a) {
            const uint32_t kr = k0 + a;
            if (AHEAD > 1 && kr >= keys) break;
            const float s = part[a] * scale;
            if (kr == 0) {
                m = s;
                l = 1.0f;
#pragma unroll
                for (int i = 0; i < PER_LANE; ++i) acc[i] = vv[a][i];
                continue;
            }
            const float nm = fmaxf(m, s);
            const float pw = expf(m - nm), cw = expf(s - nm);
            l = l * pw + cw;
#pragma unroll
            for (int i = 0; i < PER_LANE; ++i) acc[i] = acc[i] * pw + vv[a][i] * cw;
            m = nm;
        }
    }
    if (!__all_sync(0xffffffffu, finite && isfinite(l) && l > 0.0f)) return false;
#pragma unroll
    for (int i = 0; i < PER_LANE; ++i) {
        const uint32_t f = lane + 32 * i;
        if (f < dim) out[base + (uint64_t)qr * dim + f] = acc[i] / l;
    }
    return true;
}
