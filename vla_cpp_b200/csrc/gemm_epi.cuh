// Epilogue arithmetic of the bf16 GEMM kernels (gemm.cu, gemm_rows.cu).
#pragma once
#include <cuda_bf16.h>

#include "gemm.h"
#include "tc5.cuh"

namespace vb {

// Both activations are x * sigmoid(.): SiLU(x) = x / (1 + e^-x) and, since 1 + tanh(u) = 2 / (1 + e^-2u),
// tanh-GELU(x) = 0.5 x (1 + tanh(u)) = x / (1 + e^-2u) with u = k0 x (1 + k1 x^2) (constants of
// src/cuda/vla_cuda_bf16.cu:470-474).  One ex2 and one reciprocal each (relative error ~1e-6) keep the
// epilogue off the critical path; tanhf and an IEEE division cost several times the issue slots.
template <int ACT>
__device__ __forceinline__ float act_t(float x) {
    if (ACT == ACT_SILU) return __fdividef(x, 1.0f + __expf(-x));
    if (ACT == ACT_GELU_TANH) {
        const float k0 = 0.79788456080286535587989211986876f, k1 = 0.044715f;
        const float u = k0 * x * (1.0f + k1 * x * x);
        return __fdividef(x, 1.0f + __expf(-2.0f * u));
    }
    if (ACT == ACT_GELU_ERF) return 0.5f * x * (1.0f + erff(x * 0.70710678118654752440f));
    return x;
}

// The activation is uniform over a launch: the epilogues branch on it ONCE per 32-column chunk and run a loop compiled
// for that activation.  (With the activation as a run-time argument of the element function the compiler evaluated
// every variant for every element and selected: the epilogue of a plain projection paid for SiLU, tanh-GELU and erf.)
template <int ACT>
__device__ __forceinline__ void gated_chunk(const uint32_t (&v)[32], float rms, uint32_t (&w)[8]) {
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        const float g0 = act_t<ACT>(__uint_as_float(v[4 * e]) * rms) * (__uint_as_float(v[4 * e + 1]) * rms);
        const float g1 = act_t<ACT>(__uint_as_float(v[4 * e + 2]) * rms) * (__uint_as_float(v[4 * e + 3]) * rms);
        const __nv_bfloat162 h2 = __floats2bfloat162_rn(g0, g1);
        w[e] = *reinterpret_cast<const uint32_t *>(&h2);
    }
}

template <int ACT>
__device__ __forceinline__ void act_chunk(float (&f)[32]) {
#pragma unroll
    for (int e = 0; e < 32; ++e) f[e] = act_t<ACT>(f[e]);
}

// 32 accumulator columns [n, n + 32) of row m through the BIAS_ACT epilogue; mo: the output row (re-mapped).
__device__ __forceinline__ void bias_act_chunk(const GemmParams &p, const uint32_t (&v)[32], float rms, int m, size_t mo, int n) {
    float f[32];
#pragma unroll
    for (int e = 0; e < 32; ++e)
        f[e] = __uint_as_float(v[e]) * rms + ((p.bias && n + e < p.N) ? __ldg(p.bias + n + e) : 0.0f);
    if (p.act == ACT_SILU) act_chunk<ACT_SILU>(f);
    else if (p.act == ACT_GELU_TANH) act_chunk<ACT_GELU_TANH>(f);
    else if (p.act == ACT_GELU_ERF) act_chunk<ACT_GELU_ERF>(f);
    if (p.out_f32) {
        float *fr = p.out_f32 + mo * p.ld_out + n;  // (whole sectors: 16 bytes at a time cost a prefill of 1,416 rows 3 %)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (n + 8 * q >= p.N) break;
            uint32_t t[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) t[e] = __float_as_uint(f[8 * q + e]);
            if (p.al32) {
                st_global_v8(fr + 8 * q, t);
            } else {
                reinterpret_cast<uint4 *>(fr)[2 * q] = make_uint4(t[0], t[1], t[2], t[3]);
                reinterpret_cast<uint4 *>(fr)[2 * q + 1] = make_uint4(t[4], t[5], t[6], t[7]);
            }
        }
    }
    if (p.out_bf) {
        size_t off = mo * p.ld_out + n;
        if (p.scatter_hd > 0)  // head-major pages: [obs][head][cap][hd]
            off = ((size_t)(m / p.rows_in) * (p.N / p.scatter_hd) + (size_t)(n / p.scatter_hd)) *
                      ((size_t)p.scatter_cap * p.scatter_hd) +
                  (size_t)(m % p.rows_in) * p.scatter_hd + (n % p.scatter_hd);
        uint4 *bp = reinterpret_cast<uint4 *>(p.out_bf + off);
#pragma unroll
        for (int q4 = 0; q4 < 4; ++q4) {
            if (n + 8 * q4 >= p.N) break;
            uint32_t w[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const __nv_bfloat162 h2 = __floats2bfloat162_rn(f[8 * q4 + 2 * e], f[8 * q4 + 2 * e + 1]);
                w[e] = *reinterpret_cast<const uint32_t *>(&h2);
            }
            bp[q4] = make_uint4(w[0], w[1], w[2], w[3]);
        }
    }
}

// The 32 float32 columns [n, n + 32) of row m that a RESIDUAL epilogue adds to (those below N).
__device__ __forceinline__ void load_h32(const GemmParams &p, size_t m, int n, uint32_t (&r)[32]) {
    const float *src = p.h + m * p.ld_out + n;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        if (n + 8 * q >= p.N) break;
        if (p.al32) {
            uint32_t t[8];
            ld_global_v8(src + 8 * q, t);
#pragma unroll
            for (int e = 0; e < 8; ++e) r[8 * q + e] = t[e];
        } else {
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const uint4 t = *reinterpret_cast<const uint4 *>(src + 8 * q + 4 * e);
                r[8 * q + 4 * e] = t.x; r[8 * q + 4 * e + 1] = t.y; r[8 * q + 4 * e + 2] = t.z; r[8 * q + 4 * e + 3] = t.w;
            }
        }
    }
}

// 32 accumulator columns [n, n + 32) of row m through the RESIDUAL epilogue: h += v (* colscale) (+ bias), the bf16 mirror.  h holds the
// old values, requested a chunk ahead by the caller, so that no column waits for a round trip of its own.  With many tiles per CTA the
// epilogue hides behind the next tile's products and the two forms take the same time within the spread (26,112 x 1024 x 2048 back to
// back, five runs each: median 135 us ahead, 138 read where they are added; K = 4096: 179, 180).
__device__ __forceinline__ void residual_chunk(const GemmParams &p, uint32_t (&v)[32], const uint32_t (&h)[32], size_t m, int n) {
    float *hrow = p.h + m * p.ld_out + n;
    __nv_bfloat16 *brow = p.out_bf + m * p.ld_out + n;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        if (n + 8 * q >= p.N) break;
        uint32_t t[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) t[e] = v[8 * q + e];
        if (p.colscale) {  // gated residual: the projection's column n is multiplied by colscale[n] first
#pragma unroll
            for (int e = 0; e < 8; ++e) t[e] = __float_as_uint(__uint_as_float(t[e]) * __ldg(p.colscale + n + 8 * q + e));
        }
        if (p.bias) {
#pragma unroll
            for (int e = 0; e < 8; ++e) t[e] = __float_as_uint(__uint_as_float(t[e]) + __ldg(p.bias + n + 8 * q + e));
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) t[e] = __float_as_uint(__uint_as_float(h[8 * q + e]) + __uint_as_float(t[e]));
        if (p.al32) {
            st_global_v8(hrow + 8 * q, t);
        } else {
            reinterpret_cast<uint4 *>(hrow)[2 * q] = make_uint4(t[0], t[1], t[2], t[3]);
            reinterpret_cast<uint4 *>(hrow)[2 * q + 1] = make_uint4(t[4], t[5], t[6], t[7]);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const __nv_bfloat162 b2 = __floats2bfloat162_rn(__uint_as_float(t[2 * e]), __uint_as_float(t[2 * e + 1]));
            v[4 * q + e] = *reinterpret_cast<const uint32_t *>(&b2);  // (columns 4 q .. 4 q + 3 are used up)
        }
    }
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        if (n + 16 * q >= p.N) break;
        const uint32_t w[8] = {v[8 * q], v[8 * q + 1], v[8 * q + 2], v[8 * q + 3], v[8 * q + 4], v[8 * q + 5], v[8 * q + 6], v[8 * q + 7]};
        const bool two = n + 16 * q + 8 < p.N;
        if (p.al32 && two) {
            st_global_v8(brow + 16 * q, w);
        } else {
            reinterpret_cast<uint4 *>(brow)[2 * q] = make_uint4(w[0], w[1], w[2], w[3]);
            if (two) reinterpret_cast<uint4 *>(brow)[2 * q + 1] = make_uint4(w[4], w[5], w[6], w[7]);
        }
    }
}

// The row of the output that row m of the problem goes to.
__device__ __forceinline__ size_t mapped_row(const GemmParams &p, int m) {
    if (p.rows_in > 0 && p.scatter_hd == 0) return (size_t)(m / p.rows_in) * p.rows_out + p.row_off + (m % p.rows_in);
    return (size_t)m;
}

}  // namespace vb
