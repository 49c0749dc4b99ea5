// BitVLA ternary (2-bit packed) x int8 linear for sm_100a.
//
//   act_quant_kernel        per-token absmax int8 quantisation (HBM-bound)
//   ternary_gemv_kernel     M <= 8: packed weights streamed once, dp4a, HBM-bound
//   ternary_gemm_tc_kernel  M  > 8: 2-bit weights decoded to int8 in shared memory,
//                           int8 activations staged by TMA, tcgen05.mma kind::i8 with
//                           the int32 accumulator in TMEM
//
// The packed operand is the reference's "ladder" layout (scripts/convert_bitvla_to_gguf.py:103-152,
// src/models/bitvla.cpp:453-483): every 16 output rows form a contiguous run of 4*K bytes; inside
// it each 128-k chunk is 512 bytes = 128 four-byte slots; slot r holds 16 consecutive k of row
// 8*((r%32)/16) + r%8 starting at k = 32*(r/32) + 16*((r%16)/8); byte b bits 2j..2j+1 encode
// element 4j+b as value+2.
#include <cuda_bf16.h>

#include "host_common.h"
#include "tc5.cuh"

namespace vb {

// ------------------------------------------------------------------ act-quant --
// Follows src/kernels/bitvla/bitnet_kernels.h:465-521 (scale = 127 / max(amax, 1e-5),
// round-half-even, clamp) with IEEE division/multiplication, i.e. the arithmetic of the
// reference's CPU form (src/models/bitvla.cpp:69-96).
__global__ void __launch_bounds__(256) act_quant_kernel(const __nv_bfloat16 *__restrict__ in,
                                                        int8_t *__restrict__ out, float *__restrict__ scales,
                                                        int K) {
    const int m = blockIdx.x;
    const int tid = threadIdx.x;
    const uint4 *row = reinterpret_cast<const uint4 *>(in + (size_t)m * K);
    const int nvec = K >> 3;  // 8 bf16 per 16-byte vector
    constexpr int kMaxCached = 4;
    uint4 cache[kMaxCached];
    float amax = 0.0f;
#pragma unroll
    for (int i = 0; i < kMaxCached; ++i) {
        const int v = tid + i * 256;
        if (v < nvec) {
            cache[i] = __ldg(row + v);
            const __nv_bfloat162 *h = reinterpret_cast<const __nv_bfloat162 *>(&cache[i]);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float2 f = __bfloat1622float2(h[j]);
                amax = fmaxf(amax, fmaxf(fabsf(f.x), fabsf(f.y)));
            }
        }
    }
    for (int v = tid + kMaxCached * 256; v < nvec; v += 256) {
        const uint4 u = __ldg(row + v);
        const __nv_bfloat162 *h = reinterpret_cast<const __nv_bfloat162 *>(&u);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float2 f = __bfloat1622float2(h[j]);
            amax = fmaxf(amax, fmaxf(fabsf(f.x), fabsf(f.y)));
        }
    }
    for (int k = (nvec << 3) + tid; k < K; k += 256)  // K not a multiple of 8
        amax = fmaxf(amax, fabsf(__bfloat162float(in[(size_t)m * K + k])));
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, off));
    __shared__ float red[8];
    if ((tid & 31) == 0) red[tid >> 5] = amax;
    __syncthreads();
    amax = red[0];
#pragma unroll
    for (int i = 1; i < 8; ++i) amax = fmaxf(amax, red[i]);
    amax = amax < 1e-5f ? 1e-5f : amax;
    const float scale = __fdiv_rn(127.0f, amax);
    if (tid == 0) scales[m] = scale;

    auto quant8 = [&](const uint4 &u) -> uint2 {
        const __nv_bfloat162 *h = reinterpret_cast<const __nv_bfloat162 *>(&u);
        uint32_t w[2] = {0u, 0u};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float2 f = __bfloat1622float2(h[j]);
            float a = rintf(__fmul_rn(f.x, scale)), b = rintf(__fmul_rn(f.y, scale));
            a = fminf(fmaxf(a, -128.0f), 127.0f);
            b = fminf(fmaxf(b, -128.0f), 127.0f);
            const uint32_t qa = (uint32_t)(int)a & 0xffu, qb = (uint32_t)(int)b & 0xffu;
            w[j >> 1] |= (qa | (qb << 8)) << ((j & 1) * 16);
        }
        return make_uint2(w[0], w[1]);
    };
    uint2 *orow = reinterpret_cast<uint2 *>(out + (size_t)m * K);
#pragma unroll
    for (int i = 0; i < kMaxCached; ++i) {
        const int v = tid + i * 256;
        if (v < nvec) orow[v] = quant8(cache[i]);
    }
    for (int v = tid + kMaxCached * 256; v < nvec; v += 256) orow[v] = quant8(__ldg(row + v));
    for (int k = (nvec << 3) + tid; k < K; k += 256) {
        float a = rintf(__fmul_rn(__bfloat162float(in[(size_t)m * K + k]), scale));
        a = fminf(fmaxf(a, -128.0f), 127.0f);
        out[(size_t)m * K + k] = (int8_t)(int)a;
    }
}

// ------------------------------------------------------------ shared decode ----
// One 4-byte ladder slot -> four words of int8x4 (16 consecutive k), value = code - 2.
// Per byte: code c in {0..3} -> c - 2 as int8.  The low two bits of c - 2 are c ^ 2 and the upper
// six bits are ones exactly when c < 2, so with u = (x & 3) ^ 2 and neg = u & 2 (set when c < 2)
// the result is u + neg * 126 (0x02 * 126 = 0xFC, no carry between bytes).
__device__ __forceinline__ uint32_t decode_word(uint32_t x) {
    uint32_t u, neg;
    asm("lop3.b32 %0, %1, 0x03030303, 0x02020202, 0x6a;" : "=r"(u) : "r"(x));    // (x & a) ^ b
    asm("lop3.b32 %0, %1, 0x02020202, 0x02020202, 0x0c;" : "=r"(neg) : "r"(x));  // ~x & b  (c < 2)
    return neg * 126u + u;
}
__device__ __forceinline__ void decode_slot(uint32_t w, uint32_t (&d)[4]) {
#pragma unroll
    for (int j = 0; j < 4; ++j) d[j] = decode_word(w >> (2 * j));
}

__device__ __forceinline__ float ternary_scale_out(int acc, float s, float ws) {
    // out = float(acc) / s * ws   (src/kernels/bitvla/bitnet_kernels.h:245,404-405), IEEE ops
    return __fmul_rn(__fdiv_rn((float)acc, s), ws);
}

// ------------------------------------------------------------------- GEMV -------
// grid = N/16 (one 16-row weight block per CTA), 128 threads; warp w takes the 128-k
// chunks w, w+4, ...  Lane t reads the 16 bytes (4 slots) at offset 16*t of a 512-byte
// chunk: rows 8*((t%8)/4) + 4*(t%2) + {0..3}, k offset 32*(t/8) + 16*((t%4)/2).
// Eight warps split the K range of a 16-row weight block: with one CTA per SM at N = 2560 the loads in flight per
// SM, not the bandwidth, set the time.
constexpr int GEMV_WARPS = 8, GEMV_THREADS = GEMV_WARPS * 32;
template <int MT>
__global__ void __launch_bounds__(GEMV_THREADS) ternary_gemv_kernel(const int8_t *A,
                                                           const uint8_t *__restrict__ Wp,
                                                           __nv_bfloat16 *__restrict__ out,
                                                           int32_t *__restrict__ acc_out,
                                                           const float *s,
                                                           const float *__restrict__ ws, int ws_num, int M, int N,
                                                           int K, int m0) {
    extern __shared__ __align__(16) uint8_t gemv_smem[];
    int8_t *As = reinterpret_cast<int8_t *>(gemv_smem);              // [MT][K]
    int *red = reinterpret_cast<int *>(gemv_smem + (size_t)MT * K);  // [GEMV_WARPS][MT][16 rows]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nb = blockIdx.x;
    const int rows_here = min(MT, M - m0);
    // The packed weights never depend on the kernel that runs before this one: the first batch of weight loads is
    // issued before the wait on that kernel (programmatic dependent launch), so it travels during its tail.
    const int nchunks = K >> 7;
    const uint4 *wbase = reinterpret_cast<const uint4 *>(Wp + (size_t)nb * 4 * K) + lane;
    constexpr int UNROLL = 4;
    const uint4 kZeroWeights = make_uint4(0xAAAAAAAAu, 0xAAAAAAAAu, 0xAAAAAAAAu, 0xAAAAAAAAu);
    uint4 wv[UNROLL];
#pragma unroll
    for (int u = 0; u < UNROLL; ++u) {
        const int c = warp + GEMV_WARPS * u;
        wv[u] = (c < nchunks) ? __ldg(wbase + (size_t)c * 32) : kZeroWeights;
    }
    pdl_launch_dependents();
    pdl_wait();
    for (int i = tid; i < MT * (K >> 4); i += GEMV_THREADS) {
        const int mm = i / (K >> 4), kk = i % (K >> 4);
        uint4 v = make_uint4(0, 0, 0, 0);
        if (mm < rows_here) v = reinterpret_cast<const uint4 *>(A + (size_t)(m0 + mm) * K)[kk];
        reinterpret_cast<uint4 *>(As + (size_t)mm * K)[kk] = v;
    }
    __syncthreads();

    int acc[MT][4];
#pragma unroll
    for (int mm = 0; mm < MT; ++mm)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[mm][i] = 0;

    const int koff = 32 * (lane >> 3) + 16 * ((lane & 3) >> 1);
    for (int c0 = warp; c0 < nchunks; c0 += GEMV_WARPS * UNROLL) {
        if (c0 != warp) {  // the first batch is already in registers
#pragma unroll
            for (int u = 0; u < UNROLL; ++u) {
                const int c = c0 + GEMV_WARPS * u;
                wv[u] = (c < nchunks) ? __ldg(wbase + (size_t)c * 32) : kZeroWeights;
            }
        }
#pragma unroll
        for (int u = 0; u < UNROLL; ++u) {
            const int c = c0 + GEMV_WARPS * u;
            if (c >= nchunks) break;
            const uint32_t words[4] = {wv[u].x, wv[u].y, wv[u].z, wv[u].w};
            uint32_t d[4][4];
#pragma unroll
            for (int i = 0; i < 4; ++i) decode_slot(words[i], d[i]);
#pragma unroll
            for (int mm = 0; mm < MT; ++mm) {
                const uint4 av = *reinterpret_cast<const uint4 *>(As + (size_t)mm * K + c * 128 + koff);
                const uint32_t aw[4] = {av.x, av.y, av.z, av.w};
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) acc[mm][i] = __dp4a((int)aw[j], (int)d[i][j], acc[mm][i]);
            }
        }
    }
    // lanes that share rows differ in bits 1, 3, 4
#pragma unroll
    for (int mm = 0; mm < MT; ++mm)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            int v = acc[mm][i];
            v += __shfl_xor_sync(0xffffffffu, v, 2);
            v += __shfl_xor_sync(0xffffffffu, v, 8);
            v += __shfl_xor_sync(0xffffffffu, v, 16);
            acc[mm][i] = v;
        }
    if ((lane & 0x1A) == 0) {
        const int r0 = 8 * ((lane & 7) >> 2) + 4 * (lane & 1);
#pragma unroll
        for (int mm = 0; mm < MT; ++mm)
#pragma unroll
            for (int i = 0; i < 4; ++i) red[(warp * MT + mm) * 16 + r0 + i] = acc[mm][i];
    }
    __syncthreads();
    for (int i = tid; i < MT * 16; i += GEMV_THREADS) {
        const int mm = i >> 4, r = i & 15;
        if (mm >= rows_here) continue;
        int v = 0;
#pragma unroll
        for (int w8 = 0; w8 < GEMV_WARPS; ++w8) v += red[(w8 * MT + mm) * 16 + r];
        const int n = nb * 16 + r;
        const int m = m0 + mm;
        if (acc_out) acc_out[(size_t)m * N + n] = v;
        out[(size_t)m * N + n] = __float2bfloat16(ternary_scale_out(v, s[m], ws[n / (N / ws_num)]));
    }
}

// ----------------------------------------------------------------- tcgen05 GEMM --
// C[m, n] = sum_k A[m, k] * W[n, k].  MMA M = 128 activation rows (TMA, SWIZZLE_128B),
// MMA N = BN weight rows decoded from the ladder pack into the same swizzled K-major
// layout, K step 128 bytes = 4 MMAs of K = 32.  Persistent CTAs (one per SM) walk the output
// tiles; the s32 accumulator is double-buffered in TMEM so a tile's epilogue overlaps the next
// tile's main loop.
//   warp 0      TMA loader (activations)
//   warp 1      tcgen05.mma issuer
//   warps 2-9   decoders: 2-bit ladder slots -> int8, written into the swizzled B tile
//   warps 10-13 epilogue (one per TMEM lane quarter): acc / s[m] * ws -> bf16
//
// This is the kernel for few rows, where a launch is a chain of latencies.  Two things shorten it:
//   * The packed weights do not depend on the kernel before this one, so (e.w_early) the decoders fill their ring while that kernel
//     is still running; at K = 1152 the ring of the 64-column form holds all of a tile's weights.  What is left behind the
//     dependency wait is the activation tile, the products and the epilogue.
//   * `slices` CTAs of a cluster share a tile's K range.  The sums are whole numbers, so they add up to the same result in any
//     order: every CTA of the cluster finishes BN / slices of the tile's columns and gets the others' sums for them through
//     distributed shared memory.
constexpr int GEMM_BM = 128;
constexpr int GEMM_BK = 128;
constexpr int GEMM_THREADS = 448;

// What the epilogue does behind bf16(acc * ws / s): nothing, [+ bias, rounded] [tanh-GELU, rounded], or with gate_up
// relu(gate)^2 * up of columns n and N / 2 + n (the output then has N / 2 columns).
struct TernEpi {
    const __nv_bfloat16 *bias, *bias_2, *bias_3;  // of columns [0, split), [split, 2 split) and the rest, each indexed by the column
    int split, gelu, gate_up, w_early;
    TernaryRope rope;
};

__device__ __forceinline__ float tern_bias(const TernEpi &e, int n, int N) {
    const __nv_bfloat16 *b = n < e.split ? e.bias : (n < 2 * e.split ? e.bias_2 : e.bias_3);
    return n < N ? __bfloat162float(b[n]) : 0.0f;
}

// tanh.approx: what the reference's tanhf becomes under its --use_fast_math build
__device__ __forceinline__ float gelu_tanh_fast(float v) {
    const float u = 0.7978845608028654f * (v + 0.044715f * v * v * v);
    float th;
    asm("tanh.approx.f32 %0, %1;" : "=f"(th) : "f"(u));
    return 0.5f * v * (1.0f + th);
}

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t *>(&h);
}

// NV accumulators of consecutive columns -> packed bf16 of the linear's output, bias (float, in shared memory) and GELU included.
template <int NV>
__device__ __forceinline__ void tern_finish(const uint32_t (&r)[NV], float cs, const float *bias, int gelu, uint32_t (&w)[NV / 2]) {
#pragma unroll
    for (int e = 0; e < NV / 2; ++e) w[e] = pack_bf16((float)(int)r[2 * e] * cs, (float)(int)r[2 * e + 1] * cs);
    if (!bias) return;
#pragma unroll
    for (int e = 0; e < NV / 2; ++e) {
        const float2 v = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(&w[e]));
        w[e] = pack_bf16(v.x + bias[2 * e], v.y + bias[2 * e + 1]);
    }
    if (!gelu) return;
#pragma unroll
    for (int e = 0; e < NV / 2; ++e) {
        const float2 v = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(&w[e]));
        w[e] = pack_bf16(gelu_tanh_fast(v.x), gelu_tanh_fast(v.y));
    }
}

// relu(bf16(g))^2 * bf16(u) -> packed bf16 (gate_up_fused_sqrelu_mul_bf16_kernel, bitvla_lm_cuda.cu:527-542)
__device__ __forceinline__ void tern_gate_up(const uint32_t (&g)[32], const uint32_t (&u)[32], float csg, float csu, uint32_t (&w)[16]) {
#pragma unroll
    for (int e = 0; e < 16; ++e) {
        const uint32_t gp = pack_bf16((float)(int)g[2 * e] * csg, (float)(int)g[2 * e + 1] * csg);
        const uint32_t up = pack_bf16((float)(int)u[2 * e] * csu, (float)(int)u[2 * e + 1] * csu);
        const float2 gf = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(&gp));
        const float2 uf = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(&up));
        const float g0 = fmaxf(gf.x, 0.f), g1 = fmaxf(gf.y, 0.f);
        w[e] = pack_bf16(g0 * g0 * uf.x, g1 * g1 * uf.y);
    }
}

// A lane's 32 columns (packed bf16) into half `hf` of its 128-byte line of the staging area.
__device__ __forceinline__ void tern_stage(uint8_t *line, int hf, uint32_t sw, const uint32_t (&w)[16]) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
        *reinterpret_cast<uint4 *>(line + (((uint32_t)(4 * hf + i) ^ sw) << 4)) = make_uint4(w[4 * i], w[4 * i + 1], w[4 * i + 2], w[4 * i + 3]);
}

// A warp's 32 rows x up to 64 columns (bf16), staged by rows in swizzled 128-byte lines, out to global memory as whole lines.
__device__ __forceinline__ void tern_store_rows(const uint8_t *stg, __nv_bfloat16 *out, int m_first, int M, size_t ld, int n, int cols, int lane) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int rr = (lane >> 3) + 4 * i, ch = lane & 7;
        const uint4 v = *reinterpret_cast<const uint4 *>(stg + rr * 128 + (((uint32_t)ch ^ (uint32_t)(rr & 7)) << 4));
        if (m_first + rr < M && ch * 8 < cols) *reinterpret_cast<uint4 *>(out + (size_t)(m_first + rr) * ld + n + ch * 8) = v;
    }
}

// One warp's part of a tile's epilogue: 32 rows from m_first (this lane's is m_first + lane, at TMEM address lane_addr), BN accumulator
// columns.  A thread owns one accumulator row; writing its 128 bytes straight to global memory would scatter 16-byte pieces over 32 rows
// per instruction, so 32 rows x 64 columns at a time are staged in shared memory (stg) and written as whole 128-byte lines.
// acc / s * ws is evaluated as acc * (ws / s): at most one float ulp from the two-step form.  A 32-column chunk never straddles a scale
// group (the group size is a multiple of 32).
template <int BN>
__device__ __forceinline__ void tern_epilogue_tile(uint32_t lane_addr, uint8_t *stg, const float *bias, const TernEpi &e, __nv_bfloat16 *out,
                                                   int32_t *acc_out, const float *ws, int group, float sm, int m_first, int M, int N, int n0, int lane) {
    uint8_t *mine = stg + lane * 128;
    const uint32_t sw = (uint32_t)(lane & 7);
    const int m = m_first + lane;
    if constexpr (BN == 128) {
        if (e.rope.cos_t) {
            // Heads of 128: 32 columns of a head's first half and the 32 they are rotated with make a row's 128-byte line of the staging area.
            // The rotation works on the rounded projection and rounds again, as rope_split does.  Not for the pair kernel, whose epilogue of a
            // thousand rows hides behind the next tile's products only as long as it is short: 4,800 x 3840 x 2560 71 us with the rotation
            // in it, 33 without and 12 for rope_split.
            const TernaryRope &rp = e.rope;
            const float *cs_row = rp.cos_t + (size_t)(min(m, M - 1) % rp.seq) * 64, *sn_row = rp.sin_t + (size_t)(min(m, M - 1) % rp.seq) * 64;
            const int head = n0 / 128;
            const bool rot = head < rp.n_q + rp.n_kv;
            const float cs = __fdiv_rn(ws[n0 / group], sm);
#pragma unroll 1
            for (int k0 = 0; k0 < 64; k0 += 32) {
#pragma unroll 1
                for (int k = 0; k < 32; k += 16) {
                    uint32_t lo[16], hi[16], wl[8], wh[8];
                    tmem_ld16(lane_addr + (uint32_t)(k0 + k), lo);
                    tmem_ld16(lane_addr + (uint32_t)(64 + k0 + k), hi);
                    tmem_ld_wait();
                    tern_finish<16>(lo, cs, nullptr, 0, wl);
                    tern_finish<16>(hi, cs, nullptr, 0, wh);
                    if (rot) {
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const float4 co = __ldg(reinterpret_cast<const float4 *>(cs_row + k0 + k) + i), si = __ldg(reinterpret_cast<const float4 *>(sn_row + k0 + k) + i);
                            const float cv[4] = {co.x, co.y, co.z, co.w}, sv[4] = {si.x, si.y, si.z, si.w};
#pragma unroll
                            for (int j = 0; j < 2; ++j) {
                                const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(&wl[2 * i + j]));
                                const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(&wh[2 * i + j]));
                                wl[2 * i + j] = pack_bf16(a.x * cv[2 * j] - b.x * sv[2 * j], a.y * cv[2 * j + 1] - b.y * sv[2 * j + 1]);
                                wh[2 * i + j] = pack_bf16(b.x * cv[2 * j] + a.x * sv[2 * j], b.y * cv[2 * j + 1] + a.y * sv[2 * j + 1]);
                            }
                        }
                    }
                    const uint32_t p0 = (uint32_t)(k >> 3);
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        *reinterpret_cast<uint4 *>(mine + (((p0 + i) ^ sw) << 4)) = make_uint4(wl[4 * i], wl[4 * i + 1], wl[4 * i + 2], wl[4 * i + 3]);
                        *reinterpret_cast<uint4 *>(mine + (((4 + p0 + i) ^ sw) << 4)) = make_uint4(wh[4 * i], wh[4 * i + 1], wh[4 * i + 2], wh[4 * i + 3]);
                    }
                }
                __syncwarp();
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int rr = (lane >> 3) + 4 * i, ch = lane & 7, mr = m_first + rr;
                    const uint4 v = *reinterpret_cast<const uint4 *>(stg + rr * 128 + (((uint32_t)ch ^ (uint32_t)(rr & 7)) << 4));
                    if (mr >= M) continue;
                    const size_t sq = mr / rp.seq, tok = mr % rp.seq;
                    __nv_bfloat16 *dst;
                    if (head < rp.n_q) dst = static_cast<__nv_bfloat16 *>(rp.q) + ((sq * rp.n_q + head) * rp.seq + tok) * 128;
                    else if (rot) dst = static_cast<__nv_bfloat16 *>(rp.k_pages) + ((sq * rp.n_kv + head - rp.n_q) * rp.cap + tok) * 128;
                    else dst = static_cast<__nv_bfloat16 *>(rp.v_pages) + ((sq * rp.n_kv + head - rp.n_q - rp.n_kv) * rp.cap + tok) * 128;
                    *reinterpret_cast<uint4 *>(dst + k0 + (ch & 3) * 8 + (ch >> 2) * 64) = v;
                }
                __syncwarp();
            }
            return;
        }
    }
    if (e.gate_up) {
        const int n_out = N / 2;
        constexpr int STEP = BN / 2 < 64 ? BN / 2 : 64;
#pragma unroll 1
        for (int c = 0; c < BN / 2; c += STEP) {
            const int n = n0 + c;
            if (n >= n_out) break;
#pragma unroll 1
            for (int hf = 0; hf < STEP / 32; ++hf) {
                uint32_t g[32], u[32], w[16];
                tmem_ld32(lane_addr + (uint32_t)(c + 32 * hf), g);
                tmem_ld32(lane_addr + (uint32_t)(BN / 2 + c + 32 * hf), u);
                tmem_ld_wait();
                const int nh = min(n + 32 * hf, n_out - 1);
                tern_gate_up(g, u, __fdiv_rn(ws[nh / group], sm), __fdiv_rn(ws[(n_out + nh) / group], sm), w);
                tern_stage(mine, hf, sw, w);
            }
            __syncwarp();
            tern_store_rows(stg, out, m_first, M, (size_t)n_out, n, min(STEP, n_out - n), lane);
            __syncwarp();
        }
        return;
    }
#pragma unroll 1
    for (int c = 0; c < BN; c += 64) {
        const int n = n0 + c;
        if (n >= N) break;  // uniform; N % 16 == 0, so the chunk may be cut after any multiple of 16 columns
#pragma unroll 1
        for (int hf = 0; hf < 2; ++hf) {
            uint32_t r[32], w[16];
            const int ch = c + 32 * hf, nh = n + 32 * hf;
            tmem_ld32(lane_addr + (uint32_t)ch, r);
            tmem_ld_wait();
            if (acc_out && m < M) {
                int4 *dst = reinterpret_cast<int4 *>(acc_out + (size_t)m * N + nh);
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    if (nh + 4 * i < N) dst[i] = make_int4((int)r[4 * i], (int)r[4 * i + 1], (int)r[4 * i + 2], (int)r[4 * i + 3]);
            }
            tern_finish<32>(r, __fdiv_rn(ws[min(nh, N - 1) / group], sm), bias ? bias + ch : nullptr, e.gelu, w);
            tern_stage(mine, hf, sw, w);
        }
        __syncwarp();
        tern_store_rows(stg, out, m_first, M, (size_t)N, n, min(64, N - n), lane);
        __syncwarp();
    }
}

// Separate rings: SA activation tiles (TMA latency from L2 is several main-loop steps), SW decoded weight tiles.
template <int BN>
struct GemmSmem {
    static constexpr int SA = BN == 64 ? 6 : 5, SW = BN == 64 ? 12 : 5;
    static constexpr int A_BYTES = GEMM_BM * GEMM_BK;
    static constexpr int W_BYTES = BN * GEMM_BK;
    static constexpr int W_OFFSET = SA * A_BYTES;
    static constexpr int EPI_OFFSET = W_OFFSET + SW * W_BYTES;  // 4 warps x 32 rows x 128 bytes, or the other slices' sums
    static constexpr int EPI_BYTES = 3 * GEMM_BM * (BN / 4) * 4;
    static constexpr int BIAS_OFFSET = EPI_OFFSET + EPI_BYTES;  // 4 warps x BN floats
    static constexpr int BAR_OFFSET = BIAS_OFFSET + 4 * BN * 4;
    static constexpr int TOTAL = BAR_OFFSET + 512 + 1024;  // + alignment slack
};

template <int BN>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
ternary_gemm_tc_kernel(const __grid_constant__ CUtensorMap a_map, const uint8_t *__restrict__ Wp,
                       __nv_bfloat16 *__restrict__ out, int32_t *__restrict__ acc_out,
                       const float *s, const float *__restrict__ ws, int ws_num, int M, int N, int K,
                       int tiles_m, int tiles_n, int slices, const TernEpi e, int *status) {
    using L = GemmSmem<BN>;
    extern __shared__ uint8_t gemm_smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(gemm_smem_raw) + 1023) &
                                                ~static_cast<uintptr_t>(1023));
    uint64_t *full_a = reinterpret_cast<uint64_t *>(smem + L::BAR_OFFSET);
    uint64_t *empty_a = full_a + L::SA;
    uint64_t *full_w = empty_a + L::SA;
    uint64_t *empty_w = full_w + L::SW;
    uint64_t *accum_full = empty_w + L::SW;
    uint64_t *accum_empty = accum_full + 2;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(accum_empty + 2);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);

    constexpr int WPS = BN / 64;  // decode warps per step
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = slices > 1 ? (int)cluster_ctarank() : 0;  // this CTA's slice of the K steps
    const int unit = (int)blockIdx.x / slices, n_units = (int)gridDim.x / slices;
    const int kbeg = rank * (K / GEMM_BK) / slices, ksteps = (rank + 1) * (K / GEMM_BK) / slices - kbeg;
    const int n_tiles = tiles_m * tiles_n;
    const WaitCtx wc{abort_flag, status};

    if (threadIdx.x == 0) {
        for (int i = 0; i < L::SA; ++i) {
            mbar_init(&full_a[i], 1);
            mbar_init(&empty_a[i], 1);
        }
        for (int i = 0; i < L::SW; ++i) {
            mbar_init(&full_w[i], WPS);  // one arrival per decode warp of the step
            mbar_init(&empty_w[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&accum_full[i], 1);
            mbar_init(&accum_empty[i], 128);
        }
        *abort_flag = 0;
        fence_barrier_init();
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, 2 * BN);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    if (slices > 1) cluster_sync_all();  // every CTA of the cluster runs before another one writes to its shared memory
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    pdl_launch_dependents();
    // the set-up above overlapped the previous kernel's tail; the decoders go on without waiting for it if they may
    if (warp < 2 || warp >= 10 || !e.w_early) pdl_wait();

    // tiles are ordered m-fastest so that CTAs running at the same time share a weight slab
    if (warp == 0) {
        if (lane == 0) {
            tma_prefetch_desc(&a_map);
            uint32_t st = 0, ph = 0;
            bool ok = true;
            for (int tile = unit; ok && tile < n_tiles; tile += n_units) {
                const int m0 = (tile % tiles_m) * GEMM_BM;
                for (int kt = kbeg; kt < kbeg + ksteps; ++kt) {
                    ok = mbar_wait(&empty_a[st], ph ^ 1u, wc, DEV_TIMEOUT_EMPTY);
                    if (!ok) break;
                    mbar_expect_tx(&full_a[st], L::A_BYTES);
                    tma_load_2d(smem + st * L::A_BYTES, &a_map, &full_a[st], kt * GEMM_BK, m0);
                    if (++st == L::SA) { st = 0; ph ^= 1u; }
                }
            }
        }
    } else if (warp == 1) {
        {  // the whole warp walks the tiles, one elected lane issues (uniform control: see gemm.cu)
            constexpr uint32_t idesc = make_idesc(2, 1, 1, 0, 0, GEMM_BM, BN);
            const uint64_t a_desc0 = smem_desc_sw128(smem_u32(smem), 16, 1024), w_desc0 = smem_desc_sw128(smem_u32(smem + L::W_OFFSET), 16, 1024);
            uint32_t st = 0, ph = 0, sw = 0, pw = 0, j = 0;
            bool ok = true;
            for (int tile = unit; ok && tile < n_tiles; tile += n_units, ++j) {
                const uint32_t buf = j & 1u;
                ok = warp_wait(&accum_empty[buf], ((j >> 1) & 1u) ^ 1u, wc, DEV_TIMEOUT_EMPTY);
                if (!ok) break;
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + buf * BN;
                for (int kt = 0; kt < ksteps; ++kt) {
                    ok = warp_wait(&full_a[st], ph, wc, DEV_TIMEOUT_FULL);
                    if (ok) ok = warp_wait(&full_w[sw], pw, wc, DEV_TIMEOUT_FULL);
                    if (!ok) break;
                    tc_fence_after();
                    const uint64_t a_desc = a_desc0 + (uint64_t)(st * (L::A_BYTES >> 4)), w_desc = w_desc0 + (uint64_t)(sw * (L::W_BYTES >> 4));
                    if (elect_one()) {
#pragma unroll
                        for (int k = 0; k < GEMM_BK / 32; ++k) mma_i8(d_tmem, a_desc + 2 * k, w_desc + 2 * k, idesc, (kt | k) != 0 ? 1u : 0u);
                        tc_commit(&empty_a[st]);
                        tc_commit(&empty_w[sw]);
                    }
                    if (++st == L::SA) { st = 0; ph ^= 1u; }
                    if (++sw == L::SW) { sw = 0; pw ^= 1u; }
                }
                if (!ok) break;
                if (elect_one()) tc_commit(&accum_full[buf]);
            }
        }
    } else if (warp < 10) {
        // ---- decode warps: ladder slots -> swizzled K-major int8 tile ----
        // A step is four weight blocks (64 rows) per warp, BN / 64 warps; the warps take steps round-robin, so a warp has several steps
        // of time for one and the barrier wait, the proxy fence and the arrival are paid once per 64 decoded rows.
        const int dw = warp - 2;  // 0..7
        const int first = dw / WPS, blk0 = (dw % WPS) * 4;  // steps first, first + STEP, ...; blocks blk0 .. blk0 + 3 of the tile
        // lane geometry inside one 512-byte chunk (lane t holds the 4 slots at byte offset 16 t)
        const int row_in_blk = 8 * ((lane & 7) >> 2) + 4 * (lane & 1);  // + slot 0..3
        const int chunk16 = 2 * (lane >> 3) + ((lane & 3) >> 1);        // 16-byte column 0..7
        // 128-bit shared stores are served a quarter-warp at a time.  Lanes t and t ^ 4 of a quarter
        // write rows 8 apart (same banks); the upper one walks its slots in the order 2, 3, 0, 1 so that
        // the two never hit the same 16-byte column in the same instruction.
        const bool swap_slots = (lane & 4) != 0;
        constexpr int NBLK = BN / 16, STEP = 8 / WPS;
        const int my_tiles = unit < n_tiles ? (n_tiles - 1 - unit) / n_units + 1 : 0;
        const int total = my_tiles * ksteps;
        auto fetch = [&](int g, uint4 (&dst)[4]) {  // g: flat step index over this CTA's tiles
            const int tn = (unit + (g / ksteps) * n_units) / tiles_m, kt = kbeg + g % ksteps;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int blk = blk0 + i;
                int nb = tn * NBLK + blk, end = N / 16;
                if (e.gate_up) {  // half of the tile's rows are gate rows, half the up rows of the same columns
                    nb = tn * (NBLK / 2) + (blk & (NBLK / 2 - 1));
                    end = N / 32;
                }
                const bool in = g < total && nb < end;
                if (e.gate_up && blk >= NBLK / 2) nb += N / 32;
                dst[i] = in ? __ldg(reinterpret_cast<const uint4 *>(Wp + (size_t)nb * 4 * K + (size_t)kt * 512) + lane)
                            : make_uint4(0xAAAAAAAAu, 0xAAAAAAAAu, 0xAAAAAAAAu, 0xAAAAAAAAu);
            }
        };
        uint4 nxt[4];
        if (ksteps > 0) fetch(first, nxt);
        uint32_t st = (uint32_t)first, ph = 0;
        bool ok = true;
        for (int g = first; ok && g < total; g += STEP) {
            uint4 cur[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) cur[i] = nxt[i];
            fetch(g + STEP, nxt);
            uint8_t *wt = smem + L::W_OFFSET + st * L::W_BYTES;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint32_t words[4] = {cur[i].x, cur[i].y, cur[i].z, cur[i].w};
                uint32_t d[4][4];
#pragma unroll
                for (int sl = 0; sl < 4; ++sl) decode_slot(swap_slots ? words[sl ^ 2] : words[sl], d[sl]);
                if (i == 0) {  // the first block is decoded before the stage is known to be free
                    ok = mbar_wait(&empty_w[st], ph ^ 1u, wc, DEV_TIMEOUT_EMPTY);
                    if (!ok) break;
                }
#pragma unroll
                for (int sl = 0; sl < 4; ++sl) {
                    const int r = (blk0 + i) * 16 + row_in_blk + (swap_slots ? (sl ^ 2) : sl);  // row inside the BN tile
                    uint8_t *dst = wt + (r >> 3) * 1024 + (r & 7) * 128 + ((chunk16 ^ (r & 7)) << 4);
                    *reinterpret_cast<uint4 *>(dst) = make_uint4(d[sl][0], d[sl][1], d[sl][2], d[sl][3]);
                }
            }
            if (!ok) break;
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(&full_w[st]);
            st += STEP;
            if (st >= L::SW) { st -= L::SW; ph ^= 1u; }
        }
    } else if (slices == 1) {
        // ---- epilogue warps 10..13 ----
        const int q = warp & 3;  // TMEM lane quarter this warp may read
        uint8_t *stg = smem + L::EPI_OFFSET + (warp - 10) * 4096;
        float *bias = e.bias ? reinterpret_cast<float *>(smem + L::BIAS_OFFSET) + (warp - 10) * BN : nullptr;
        const int cols_tile = e.gate_up ? BN / 2 : BN;
        uint32_t j = 0;
        bool ok = true;
        for (int tile = unit; ok && tile < n_tiles; tile += n_units, ++j) {
            const uint32_t buf = j & 1u;
            const int m_first = (tile % tiles_m) * GEMM_BM + q * 32, n0 = (tile / tiles_m) * cols_tile;
            const float sm = (m_first + lane < M) ? s[m_first + lane] : 1.0f;
            if (bias) {
                for (int c = lane; c < BN; c += 32) bias[c] = tern_bias(e, n0 + c, N);
                __syncwarp();
            }
            ok = mbar_wait(&accum_full[buf], (j >> 1) & 1u, wc, DEV_TIMEOUT_ACCUM);
            if (!ok) break;
            tc_fence_after();
            tern_epilogue_tile<BN>(tmem_base + buf * BN + ((uint32_t)(q * 32) << 16), stg, bias, e, out, acc_out, ws, N / ws_num, sm, m_first, M, N,
                                   n0, lane);
            tc_fence_before();
            mbar_arrive(&accum_empty[buf]);
        }
    }
    if (slices > 1) {
        // One tile per cluster.  The sums of the columns that another CTA finishes go into its shared memory, [sender][4 columns][row] so
        // that a warp writes 512 contiguous bytes; then each CTA adds what it received to its own sums and finishes its columns.
        const int q = warp & 3, width = BN / slices;
        const int m0 = (unit % tiles_m) * GEMM_BM, n0 = (unit / tiles_m) * BN + rank * width;
        const int row = q * 32 + lane, m = m0 + row;
        const bool epi = warp >= 10;
        const uint32_t lane_addr = tmem_base + ((uint32_t)(q * 32) << 16);
        uint8_t *recv = smem + L::EPI_OFFSET;
        const int slot_bytes = width * GEMM_BM * 4;
        float *bias = e.bias ? reinterpret_cast<float *>(smem + L::BIAS_OFFSET) + (warp & 3) * BN : nullptr;
        bool ok = epi;
        float sm = 1.0f;
        if (epi) {
            if (m < M) sm = s[m];
            if (bias) {
                for (int c = lane; c < width; c += 32) bias[c] = tern_bias(e, n0 + c, N);
                __syncwarp();
            }
            ok = mbar_wait(&accum_full[0], 0u, wc, DEV_TIMEOUT_ACCUM);
            tc_fence_after();
            if (ok) {
                for (int r = 0; r < slices; ++r) {
                    if (r == rank) continue;
                    const uint32_t dst = cluster_addr(smem_u32(recv) + (uint32_t)((rank < r ? rank : rank - 1) * slot_bytes + row * 16), (uint32_t)r);
                    for (int c = 0; c < width; c += 16) {
                        uint32_t v[16];
                        tmem_ld16(lane_addr + (uint32_t)(r * width + c), v);
                        tmem_ld_wait();
#pragma unroll
                        for (int i = 0; i < 4; ++i)
                            st_cluster_v4(dst + (uint32_t)((c / 4 + i) * GEMM_BM * 16), v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
                    }
                }
            }
        }
        __syncwarp();  // the cluster barrier is for converged warps
        cluster_sync_all();
        if (ok) {
            const int group = N / ws_num;
            for (int c = 0; c < width; c += 16) {
                const int n = n0 + c;
                if (n >= N) break;  // N % 16 == 0: a piece of 16 columns is inside or outside
                uint32_t v[16], w[8];
                tmem_ld16(lane_addr + (uint32_t)(rank * width + c), v);
                tmem_ld_wait();
                for (int t = 0; t < slices - 1; ++t)
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const uint4 o = *reinterpret_cast<const uint4 *>(recv + t * slot_bytes + (c / 4 + i) * GEMM_BM * 16 + row * 16);
                        v[4 * i] += o.x; v[4 * i + 1] += o.y; v[4 * i + 2] += o.z; v[4 * i + 3] += o.w;
                    }
                tern_finish<16>(v, __fdiv_rn(ws[n / group], sm), bias ? bias + c : nullptr, e.gelu, w);
                if (m < M) {
                    if (acc_out) {
                        int4 *dst = reinterpret_cast<int4 *>(acc_out + (size_t)m * N + n);
#pragma unroll
                        for (int i = 0; i < 4; ++i) dst[i] = make_int4((int)v[4 * i], (int)v[4 * i + 1], (int)v[4 * i + 2], (int)v[4 * i + 3]);
                    }
                    uint4 *dst = reinterpret_cast<uint4 *>(out + (size_t)m * N + n);
                    dst[0] = make_uint4(w[0], w[1], w[2], w[3]);
                    dst[1] = make_uint4(w[4], w[5], w[6], w[7]);
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, 2 * BN);
    }
}

// ------------------------------------------------------- tcgen05 GEMM, CTA pairs --
// Same computation on clusters of two CTAs (tcgen05 cta_group::2): one MMA covers 256
// activation rows x 256 weight rows, each CTA holding its own 128 activation rows (TMA) and
// decoding only ITS half of the weight tile, so per SM the decode work, the shared-memory
// writes of decoded weights and the operand bytes the tensor core reads per flop all halve.
// The even CTA issues the MMAs; tcgen05.commit multicasts the "slot free" / "accumulator
// ready" arrivals to both CTAs; the odd CTA's MMA warp forwards "my A tile and my W half are
// in shared memory" to the even CTA's weight barrier, its epilogue warps "accumulator
// drained" to the even CTA's accum_empty barrier.
constexpr int PAIR_STAGES = 6;
struct PairSmem {
    static constexpr int A_BYTES = GEMM_BM * GEMM_BK;  // 128 activation rows
    static constexpr int W_BYTES = 128 * GEMM_BK;      // 128 of the tile's 256 weight rows
    static constexpr int STAGE_BYTES = A_BYTES + W_BYTES;
    static constexpr int BAR_OFFSET = PAIR_STAGES * STAGE_BYTES;
    static constexpr int STAGING_OFFSET = BAR_OFFSET + 256;
    static constexpr int BIAS_OFFSET = STAGING_OFFSET + 4 * 4096;  // 4 warps x 256 floats
    static constexpr int TOTAL = BIAS_OFFSET + 4 * 256 * 4 + 1024;
};

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(GEMM_THREADS, 1)
ternary_gemm_pair_kernel(const __grid_constant__ CUtensorMap a_map, const uint8_t *__restrict__ Wp,
                         __nv_bfloat16 *__restrict__ out, int32_t *__restrict__ acc_out,
                         const float *s, const float *__restrict__ ws, int ws_num, int M, int N, int K,
                         int tiles_mp, int tiles_n, const TernEpi e, int *status) {
    using L = PairSmem;
    constexpr int BN = 256;
    extern __shared__ uint8_t gemm_smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(gemm_smem_raw) + 1023) &
                                                ~static_cast<uintptr_t>(1023));
    // One ring: stage = this CTA's activation tile + its decoded half of the weight tile.
    //   full[s]   loader's expect_tx arrival + TMA bytes + the two decode warps of the step
    //             (+ in the even CTA the odd CTA's "my stage is full" forward)
    //   empty[s]  tcgen05.commit of the MMAs that read stage s, multicast to both CTAs
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + L::BAR_OFFSET);
    uint64_t *empty = full + PAIR_STAGES;
    uint64_t *accum_full = empty + PAIR_STAGES;
    uint64_t *accum_empty = accum_full + 2;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(accum_empty + 2);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();
    const int cid = blockIdx.x >> 1, ncl = gridDim.x >> 1;
    const int ksteps = K / GEMM_BK;
    const int n_tiles = tiles_mp * tiles_n;
    const WaitCtx wc{abort_flag, status};

    if (threadIdx.x == 0) {
        for (int i = 0; i < PAIR_STAGES; ++i) {
            mbar_init(&full[i], rank == 0 ? 4 : 3);
            mbar_init(&empty[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&accum_full[i], 1);
            mbar_init(&accum_empty[i], 8);  // 4 epilogue warps of each CTA (used in the even CTA)
        }
        *abort_flag = 0;
        fence_barrier_init();
    }
    __syncthreads();
    cluster_sync_all();  // both CTAs' barriers exist before anything arrives on them remotely
    if (warp == 1) {
        tmem_alloc_pair(tmem_slot, 2 * BN);
        tmem_relinquish_pair();
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    // Programmatic dependent launch: the activations, scales and the output belong to the kernels around this one,
    // the packed weights do not -- the decode warps fetch their first weight blocks before they wait.
    pdl_launch_dependents();
    if (warp < 2 || warp >= 10) pdl_wait();

    if (warp == 0) {
        if (lane == 0) {
            tma_prefetch_desc(&a_map);
            uint32_t st = 0, ph = 0;
            bool ok = true;
            for (int tile = cid; ok && tile < n_tiles; tile += ncl) {
                const int m0 = (tile % tiles_mp) * 256 + (int)rank * 128;
                for (int kt = 0; kt < ksteps; ++kt) {
                    ok = mbar_wait_backoff(&empty[st], ph ^ 1u, wc, DEV_TIMEOUT_EMPTY, 64);
                    if (!ok) break;
                    mbar_expect_tx(&full[st], L::A_BYTES);
                    tma_load_2d(smem + st * L::STAGE_BYTES, &a_map, &full[st], kt * GEMM_BK, m0);
                    if (++st == PAIR_STAGES) { st = 0; ph ^= 1u; }
                }
            }
        }
    } else if (warp == 1) {
        if (rank == 0) {  // the whole warp walks the tiles, one elected lane issues (uniform control: see gemm.cu)
            constexpr uint32_t idesc = make_idesc(2, 1, 1, 0, 0, 256, BN);
            // descriptors differ between stages and k sub-steps only in the 14-bit start address
            const uint64_t a_desc0 = smem_desc_sw128(smem_u32(smem), 16, 1024);
            const uint64_t w_desc0 = smem_desc_sw128(smem_u32(smem + L::A_BYTES), 16, 1024);
            uint32_t st = 0, ph = 0, j = 0;
            bool ok = true;
            for (int tile = cid; ok && tile < n_tiles; tile += ncl, ++j) {
                const uint32_t buf = j & 1u;
                ok = warp_wait(&accum_empty[buf], ((j >> 1) & 1u) ^ 1u, wc, DEV_TIMEOUT_EMPTY);
                if (!ok) break;
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + buf * BN;
                for (int kt = 0; kt < ksteps; ++kt) {
                    ok = warp_wait(&full[st], ph, wc, DEV_TIMEOUT_FULL);
                    if (!ok) break;
                    tc_fence_after();
                    const uint64_t off = (uint64_t)(st * (L::STAGE_BYTES >> 4));
                    if (elect_one()) {
#pragma unroll
                        for (int k = 0; k < GEMM_BK / 32; ++k)
                            mma_i8_pair(d_tmem, a_desc0 + off + 2 * k, w_desc0 + off + 2 * k, idesc, (kt | k) != 0 ? 1u : 0u);
                        tc_commit_pair(&empty[st], 3);
                    }
                    if (++st == PAIR_STAGES) { st = 0; ph ^= 1u; }
                }
                if (!ok) break;
                if (elect_one()) tc_commit_pair(&accum_full[buf], 3);
            }
        } else if (lane == 0) {
            // odd CTA: tell the even CTA when this CTA's stage is in shared memory
            uint32_t st = 0, ph = 0;
            bool ok = true;
            for (int tile = cid; ok && tile < n_tiles; tile += ncl) {
                for (int kt = 0; kt < ksteps; ++kt) {
                    ok = mbar_wait(&full[st], ph, wc, DEV_TIMEOUT_FULL);
                    if (!ok) break;
                    mbar_arrive_cluster(&full[st], 0);
                    if (++st == PAIR_STAGES) { st = 0; ph ^= 1u; }
                }
            }
        }
    } else if (warp < 10) {
        // ---- decode warps ----
        // Two warps share a step (4 of this CTA's 8 weight blocks each) and the four warp pairs take
        // steps round-robin, so a warp has four steps of time for one unit of work and the barrier
        // wait, proxy fence and arrival are paid once per 64 decoded rows.
        const int dw = warp - 2;
        const int pi = dw >> 1, hb = dw & 1;
        // gate_up: the even CTA decodes 128 gate rows, the odd one the up rows of the same columns
        const int nblk_tile = e.gate_up ? 8 : BN / 16, nblk_total = e.gate_up ? N / 32 : N / 16;
        const int row_in_blk = 8 * ((lane & 7) >> 2) + 4 * (lane & 1);  // + slot 0..3
        const int chunk16 = 2 * (lane >> 3) + ((lane & 3) >> 1);        // 16-byte column 0..7
        const bool swap_slots = (lane & 4) != 0;  // see ternary_gemm_tc_kernel: avoids 2-way bank conflicts
        const int my_tiles = cid < n_tiles ? (n_tiles - 1 - cid) / ncl + 1 : 0;
        const int total = my_tiles * ksteps;
        auto fetch = [&](int g, uint4 (&dst)[4]) {
            const int tile = cid + (g / ksteps) * ncl, kt = g % ksteps;
            const int nb0 = (tile / tiles_mp) * nblk_tile + (e.gate_up ? 0 : (int)rank * 8) + hb * 4, up0 = e.gate_up && rank ? nblk_total : 0;
#pragma unroll
            for (int i = 0; i < 4; ++i)
                dst[i] = (g < total && nb0 + i < nblk_total)
                             ? __ldg(reinterpret_cast<const uint4 *>(Wp + (size_t)(up0 + nb0 + i) * 4 * K + (size_t)kt * 512) + lane)
                             : make_uint4(0xAAAAAAAAu, 0xAAAAAAAAu, 0xAAAAAAAAu, 0xAAAAAAAAu);
        };
        uint4 nxt[4];
        fetch(pi, nxt);
        pdl_wait();
        uint32_t st = (uint32_t)pi, ph = 0;
        bool ok = true;
        for (int g = pi; ok && g < total; g += 4) {
            uint4 cur[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) cur[i] = nxt[i];
            fetch(g + 4, nxt);
            uint8_t *wt = smem + st * L::STAGE_BYTES + L::A_BYTES;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint32_t words[4] = {cur[i].x, cur[i].y, cur[i].z, cur[i].w};
                uint32_t d[4][4];
#pragma unroll
                for (int sl = 0; sl < 4; ++sl) decode_slot(swap_slots ? words[sl ^ 2] : words[sl], d[sl]);
                if (i == 0) {  // the first block is decoded before the stage is known to be free
                    ok = mbar_wait(&empty[st], ph ^ 1u, wc, DEV_TIMEOUT_EMPTY);
                    if (!ok) break;
                }
#pragma unroll
                for (int sl = 0; sl < 4; ++sl) {
                    const int r = (hb * 4 + i) * 16 + row_in_blk + (swap_slots ? (sl ^ 2) : sl);  // row in the half tile
                    uint8_t *dst = wt + (r >> 3) * 1024 + (r & 7) * 128 + ((chunk16 ^ (r & 7)) << 4);
                    *reinterpret_cast<uint4 *>(dst) = make_uint4(d[sl][0], d[sl][1], d[sl][2], d[sl][3]);
                }
            }
            if (!ok) break;
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(&full[st]);
            st += 4;
            if (st >= PAIR_STAGES) { st -= PAIR_STAGES; ph ^= 1u; }
        }
    } else {
        // ---- epilogue warps 10..13: this CTA's 128 rows of the pair tile ----
        const int q = warp & 3;
        uint8_t *stg = smem + L::STAGING_OFFSET + (warp - 10) * 4096;
        float *bias = e.bias ? reinterpret_cast<float *>(smem + L::BIAS_OFFSET) + (warp - 10) * BN : nullptr;
        uint32_t j = 0;
        bool ok = true;
        for (int tile = cid; ok && tile < n_tiles; tile += ncl, ++j) {
            const uint32_t buf = j & 1u;
            const int m0 = (tile % tiles_mp) * 256 + (int)rank * 128, m_first = m0 + q * 32, n0 = (tile / tiles_mp) * (e.gate_up ? BN / 2 : BN);
            const float sm = (m_first + lane < M) ? s[m_first + lane] : 1.0f;
            if (bias) {
                for (int c = lane; c < BN; c += 32) bias[c] = tern_bias(e, n0 + c, N);
                __syncwarp();
            }
            ok = mbar_wait_backoff(&accum_full[buf], (j >> 1) & 1u, wc, DEV_TIMEOUT_ACCUM, 256);
            if (!ok) break;
            tc_fence_after();
            if (m0 < M)  // warp-uniform: the odd CTA's rows may all lie past M
                tern_epilogue_tile<BN>(tmem_base + buf * BN + ((uint32_t)(q * 32) << 16), stg, bias, e, out, acc_out, ws, N / ws_num, sm, m_first, M,
                                       N, n0, lane);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                if (rank == 0) mbar_arrive(&accum_empty[buf]);
                else mbar_arrive_cluster(&accum_empty[buf], 0);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();  // neither CTA may exit while the other can still signal its barriers
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc_pair(tmem_base, 2 * BN);
    }
}

// ------------------------------------------------------------------ host side --
static int check_gemm_args(const void *A, const void *W, const void *out, const void *s, const void *ws, int ws_num,
                           int M, int N, int K) {
    if (!A || !W || !out || !s || !ws) return VLAB200_ERR_ARG;
    if (M < 0 || N <= 0 || K <= 0 || ws_num <= 0) return VLAB200_ERR_ARG;
    if (N % 16 || K % 128 || N % ws_num) return VLAB200_ERR_UNSUPPORTED;
    return VLAB200_OK;
}

template <int MT>
static int launch_gemv(const int8_t *A, const uint8_t *W, __nv_bfloat16 *out, int32_t *acc, const float *s,
                       const float *ws, int ws_num, int M, int N, int K, int m0, cudaStream_t st) {
    const size_t smem = (size_t)MT * K + GEMV_WARPS * MT * 16 * sizeof(int);
    if (smem > 48 * 1024)
        if (int rc = ensure_dyn_smem(ternary_gemv_kernel<MT>, (int)smem)) return rc;
    return launch_pdl(ternary_gemv_kernel<MT>, dim3(N / 16), dim3(GEMV_THREADS), smem, st, A, W, out, acc, s, ws, ws_num, M, N, K, m0);
}

// How many clusters of `cluster` CTAs of the kernel the device holds at once (0: none).
template <int BN>
static int tc_clusters(int cluster) {
    if (ensure_dyn_smem(ternary_gemm_tc_kernel<BN>, GemmSmem<BN>::TOTAL) != VLAB200_OK) return 0;
    return max_active_clusters(reinterpret_cast<const void *>(ternary_gemm_tc_kernel<BN>), GEMM_THREADS, GemmSmem<BN>::TOTAL, cluster);
}

template <int BN>
static int launch_gemm_tc(const int8_t *A, const uint8_t *W, __nv_bfloat16 *out, int32_t *acc, const float *s,
                          const float *ws, int ws_num, int M, int N, int K, const TernEpi &e, int slices, cudaStream_t st) {
    int *status = device_status_ptr();
    if (!status) return cuda_fail(cudaGetLastError(), "device_status_ptr");
    CUtensorMap amap;
    const uint64_t dims[2] = {(uint64_t)K, (uint64_t)M};
    const uint64_t strides[1] = {(uint64_t)K};
    const uint32_t box[2] = {GEMM_BK, GEMM_BM};
    int rc = make_tensor_map(&amap, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, A, dims, strides, box,
                             CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc) return rc;
    using L = GemmSmem<BN>;
    if ((rc = ensure_dyn_smem(ternary_gemm_tc_kernel<BN>, L::TOTAL))) return rc;
    const int n_sm = sm_count();
    if (n_sm <= 0) return cuda_fail(cudaGetLastError(), "sm_count");
    const int bn_out = e.gate_up ? BN / 2 : BN, n_out = e.gate_up ? N / 2 : N;
    const int tiles_m = (M + GEMM_BM - 1) / GEMM_BM, tiles_n = (n_out + bn_out - 1) / bn_out;
    const int nt = tiles_m * tiles_n;
    if (slices > 1)
        return launch_pdl_cluster(ternary_gemm_tc_kernel<BN>, dim3(nt * slices), dim3(GEMM_THREADS), L::TOTAL, slices, st, amap, W, out, acc, s, ws,
                                  ws_num, M, N, K, tiles_m, tiles_n, slices, e, status);
    return launch_pdl(ternary_gemm_tc_kernel<BN>, dim3(nt < n_sm ? nt : n_sm), dim3(GEMM_THREADS), L::TOTAL, st, amap, W, out,
                      acc, s, ws, ws_num, M, N, K, tiles_m, tiles_n, 1, e, status);
}

static int launch_gemm_pair(const int8_t *A, const uint8_t *W, __nv_bfloat16 *out, int32_t *acc, const float *s,
                            const float *ws, int ws_num, int M, int N, int K, const TernEpi &e, cudaStream_t st) {
    int *status = device_status_ptr();
    if (!status) return cuda_fail(cudaGetLastError(), "device_status_ptr");
    CUtensorMap amap;
    const uint64_t dims[2] = {(uint64_t)K, (uint64_t)M};
    const uint64_t strides[1] = {(uint64_t)K};
    const uint32_t box[2] = {GEMM_BK, GEMM_BM};
    int rc = make_tensor_map(&amap, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, A, dims, strides, box,
                             CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc) return rc;
    if ((rc = ensure_dyn_smem(ternary_gemm_pair_kernel, PairSmem::TOTAL))) return rc;
    const int n_sm = sm_count();
    if (n_sm <= 0) return cuda_fail(cudaGetLastError(), "sm_count");
    const int tiles_mp = (M + 255) / 256, tiles_n = e.gate_up ? (N / 2 + 127) / 128 : (N + 255) / 256;
    const int nt = tiles_mp * tiles_n, pairs = n_sm / 2;
    return launch_pdl(ternary_gemm_pair_kernel, dim3(2 * (nt < pairs ? nt : pairs)), dim3(GEMM_THREADS), PairSmem::TOTAL, st, amap,
                      W, out, acc, s, ws, ws_num, M, N, K, tiles_mp, tiles_n, e, status);
}

// The tiling of a call with more than eight rows, by ns of a launch: set-up and epilogue, plus waves times 128-wide K steps.  Pair tiles
// move the fewest bytes per product and win as soon as there are enough of them; with few rows (one image, one prompt) they leave
// most SMs without work and narrow tiles win, and where even those are few, K slices over a cluster.
struct TernTiling {
    int bn, slices;  // bn 256: pair tiles
};
static TernTiling choose_tiling(int M, int N, int K, bool gate_up, int n_sm) {
    const int tm = (M + 127) / 128, tp = (M + 255) / 256, ks = K / 128;
    auto waves = [](int tiles, int units) { return (tiles + units - 1) / units; };
    TernTiling best{64, 1};
    int cost = 0x7fffffff;
    auto consider = [&](int bn, int slices, int c) {
        if (c < cost) {
            cost = c;
            best = {bn, slices};
        }
    };
    const int t64 = tm * ((N + 63) / 64), t128 = tm * ((N + 127) / 128);
    consider(64, 1, 3600 + 370 * ks * waves(t64, n_sm));
    consider(128, 1, 4400 + 460 * ks * waves(t128, n_sm));
    if (N >= 256 && n_sm >= 2) consider(256, 1, 6400 + 360 * ks * waves(tp * ((N + 255) / 256), n_sm / 2));
    if (!gate_up)
        for (int sl = 2; sl <= 4 && ks >= 4 * sl; sl *= 2) {
            if (t64 * sl <= n_sm && t64 <= tc_clusters<64>(sl)) consider(64, sl, 5400 + 370 * waves(ks, sl));
            if (t128 * sl <= n_sm && t128 <= tc_clusters<128>(sl)) consider(128, sl, 6200 + 460 * waves(ks, sl));
        }
    return best;
}

int ternary_linear(const TernaryCall &c, cudaStream_t st) {
    const int8_t *A = c.A;
    const uint8_t *W = c.W;
    __nv_bfloat16 *out = static_cast<__nv_bfloat16 *>(c.out);
    const int ws_num = c.ws_num, M = c.M, N = c.N, K = c.K, path = c.path;
    int rc = check_gemm_args(A, W, out, c.s, c.ws, ws_num, M, N, K);
    if (rc) return rc;
    if (M == 0) return VLAB200_OK;
    const bool gemv = path == 1 || (path == 0 && M <= 8);
    TernEpi e{};
    e.bias = e.bias_2 = e.bias_3 = static_cast<const __nv_bfloat16 *>(c.bias);
    e.split = N; e.gelu = c.gelu; e.gate_up = c.gate_up; e.w_early = c.w_early; e.rope = c.rope;
    if (c.bias_2) {
        e.split = N / 3;
        e.bias_2 = static_cast<const __nv_bfloat16 *>(c.bias_2) - e.split;
        e.bias_3 = static_cast<const __nv_bfloat16 *>(c.bias_3) - 2 * e.split;
    }
    if (gemv) {
        if (e.bias || e.gelu || e.gate_up || e.rope.cos_t) return VLAB200_ERR_UNSUPPORTED;
        if ((size_t)8 * K + 4 * 8 * 16 * sizeof(int) > 200 * 1024) return VLAB200_ERR_UNSUPPORTED;
        for (int m0 = 0; m0 < M; m0 += 8) {
            const int left = M - m0;
            if (left >= 5) rc = launch_gemv<8>(A, W, out, c.acc, c.s, c.ws, ws_num, M, N, K, m0, st);
            else if (left >= 3) rc = launch_gemv<4>(A, W, out, c.acc, c.s, c.ws, ws_num, M, N, K, m0, st);
            else if (left == 2) rc = launch_gemv<2>(A, W, out, c.acc, c.s, c.ws, ws_num, M, N, K, m0, st);
            else rc = launch_gemv<1>(A, W, out, c.acc, c.s, c.ws, ws_num, M, N, K, m0, st);
            if (rc) return rc;
        }
        return VLAB200_OK;
    }
    if ((reinterpret_cast<uintptr_t>(A) & 15) || (reinterpret_cast<uintptr_t>(out) & 15) ||
        (c.acc && (reinterpret_cast<uintptr_t>(c.acc) & 15)))
        return VLAB200_ERR_ARG;
    // a 32-column epilogue chunk must not straddle two weight-scale groups; with one group N % 16 == 0 is enough
    if (ws_num > 1 && (N / ws_num) % 32) return VLAB200_ERR_UNSUPPORTED;
    if (e.gate_up && (N % 64 || c.acc || e.bias)) return VLAB200_ERR_UNSUPPORTED;
    const int n_sm = sm_count();
    if (n_sm <= 0) return cuda_fail(cudaGetLastError(), "sm_count");
    TernTiling t{128, 1};  // path 2
    if (path == 0) t = choose_tiling(M, N, K, e.gate_up != 0, n_sm);
    else if (path == 3) t = {256, 1};
    else if ((path & 0xff) == 64 || (path & 0xff) == 128) t = {path & 0xff, (path >> 8) > 1 ? path >> 8 : 1};
    if (t.slices != 1 && ((t.slices != 2 && t.slices != 4) || K / GEMM_BK < t.slices || e.gate_up)) return VLAB200_ERR_UNSUPPORTED;
    if (e.rope.cos_t && (t.bn != 128 || t.slices != 1 || N % 128 || c.acc || e.bias || e.gate_up || (N / ws_num) % 128)) return VLAB200_ERR_UNSUPPORTED;
    if (t.bn == 256) return launch_gemm_pair(A, W, out, c.acc, c.s, c.ws, ws_num, M, N, K, e, st);
    if (t.bn == 64) return launch_gemm_tc<64>(A, W, out, c.acc, c.s, c.ws, ws_num, M, N, K, e, t.slices, st);
    return launch_gemm_tc<128>(A, W, out, c.acc, c.s, c.ws, ws_num, M, N, K, e, t.slices, st);
}

bool ternary_can_rope(int M, int N, int K) {
    const int n_sm = sm_count();
    if (M <= 8 || n_sm <= 0 || N % 128) return false;
    const TernTiling t = choose_tiling(M, N, K, false, n_sm);
    return t.bn == 128 && t.slices == 1;
}

static int ternary_linear(const int8_t *A, const uint8_t *W, void *out, int32_t *acc, const float *s, const float *ws, int ws_num, int M, int N,
                          int K, cudaStream_t st, int path) {
    TernaryCall c{};
    c.A = A; c.W = W; c.out = out; c.acc = acc; c.s = s; c.ws = ws; c.ws_num = ws_num; c.M = M; c.N = N; c.K = K; c.path = path;
    return ternary_linear(c, st);
}

// ws_num for the fused projections the reference registers (src/kernels/bitvla/bitnet_kernels.cu:31-116)
static int reference_ws_num(int N, int K) {
    if (N == 13824 && K == 2560) return 2;  // gate_up
    if (N == 3840 && K == 2560) return 3;   // head qkv
    if (N == 20480 && K == 3200) return 2;
    if (N == 4800 && K == 3200) return 6;
    return 1;
}


// ---- load-time ternarisation of a float weight matrix + ladder packing, on the device ---------------
// sum_i |W[i]| in double: per-block tree sums, one atomicAdd(double) per block.  The total differs from the
// reference's sequential host sum (src/models/bitvla.cpp:430-451) by rounding of the double only; the float
// mean derived from it is the same value unless the double lands within ~1e-13 of a float rounding boundary.
__global__ void __launch_bounds__(256) absum_kernel(const float *__restrict__ w, size_t n, double *__restrict__ total) {
    __shared__ double part[8];
    double acc = 0.0;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        acc += fabs((double)w[i]);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int i = 0; i < 8; ++i) t += part[i];
        atomicAdd(total, t);
    }
}

// One thread per 4-byte slot of the ladder layout (16 ternaries of one output row, consecutive k): the slot
// index decomposes as in scripts/convert_bitvla_to_gguf.py:103-152 / src/models/bitvla.cpp:453-483; byte b holds
// the values t = b + 4j at bits 2j..2j+1 encoded (w + 2) & 3; w = clamp(rne(W / absmean), -1, 1).
__global__ void __launch_bounds__(256) ternarize_pack_kernel(const float *__restrict__ w, int64_t N, int64_t K,
                                                             const double *__restrict__ total,
                                                             uint32_t *__restrict__ packed, float *__restrict__ scale) {
    const int64_t n_elems = N * K;
    float mean = (float)(*total / (double)n_elems);
    if (mean < 1e-5f) mean = 1e-5f;
    const float inv = __fdiv_rn(1.0f, mean);
    const int64_t n_slots = n_elems / 16;
    for (int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; s < n_slots; s += (int64_t)gridDim.x * blockDim.x) {
        const int64_t n_block = s / K;  // 16 rows x K columns = K slots per row block
        int64_t r = s % K;
        const int64_t k0 = r / 128;
        r %= 128;
        const int64_t major = r / 32;
        r %= 32;
        const int64_t y_half = r / 16;
        r %= 16;
        const int64_t sub_k = r / 8, y = r % 8;
        const int64_t n = 16 * n_block + 8 * y_half + y, k_start = 128 * k0 + 32 * major + 16 * sub_k;
        const float4 *src = reinterpret_cast<const float4 *>(w + n * K + k_start);  // K % 128 == 0: 64-byte aligned
        float v[16];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float4 f = __ldg(src + i);
            v[4 * i] = f.x; v[4 * i + 1] = f.y; v[4 * i + 2] = f.z; v[4 * i + 3] = f.w;
        }
        uint32_t word = 0;
#pragma unroll
        for (int b = 0; b < 4; ++b)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                float q = rintf(__fmul_rn(v[b + 4 * j], inv));
                q = fminf(fmaxf(q, -1.0f), 1.0f);
                word |= (uint32_t)(((int)q + 2) & 3) << (8 * b + 2 * j);
            }
        packed[s] = word;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) *scale = mean;
}

}  // namespace vb

extern "C" {

int32_t vlab200_act_quant(const void *x_bf16, int8_t *q, float *scales, int32_t M, int32_t K, void *stream) {
    if (!x_bf16 || !q || !scales || M < 0 || K <= 0) return VLAB200_ERR_ARG;
    if ((reinterpret_cast<uintptr_t>(x_bf16) & 15) || (reinterpret_cast<uintptr_t>(q) & 7) || (K % 8))
        return VLAB200_ERR_UNSUPPORTED;
    if (M == 0) return VLAB200_OK;
    vb::act_quant_kernel<<<M, 256, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const __nv_bfloat16 *>(x_bf16), q, scales, K);
    VB_CUDA(cudaGetLastError());
    return VLAB200_OK;
}

int32_t vlab200_ternary_linear(const int8_t *A, const uint8_t *W_ladder, void *out_bf16, int32_t *acc_out,
                               const float *s, const float *ws, int32_t ws_num, int32_t M, int32_t N, int32_t K,
                               int32_t path, void *stream) {
    return vb::ternary_linear(A, W_ladder, out_bf16, acc_out, s, ws, ws_num, M, N, K, static_cast<cudaStream_t>(stream), path);
}

// Drop-in names of the reference (src/kernels/bitvla/bitnet_kernels.cu:31,76,118).  The
// reference aborts the process on a shape it has no kernel for; these print and return.
int32_t vlab200_ternarize_pack(const float *W, int64_t N, int64_t K, uint8_t *packed_out, float *scale_out,
                               double *scratch, void *stream) {
    if (!W || !packed_out || !scale_out || !scratch || N <= 0 || K <= 0) return VLAB200_ERR_ARG;
    if (N % 16 || K % 128) return VLAB200_ERR_UNSUPPORTED;
    if ((reinterpret_cast<uintptr_t>(W) & 15) || (reinterpret_cast<uintptr_t>(packed_out) & 3)) return VLAB200_ERR_ARG;
    cudaStream_t cs = static_cast<cudaStream_t>(stream);
    const size_t n = (size_t)N * (size_t)K;
    int n_sm = vb::sm_count();
    if (n_sm <= 0) n_sm = 148;
    VB_CUDA(cudaMemsetAsync(scratch, 0, sizeof(double), cs));
    vb::absum_kernel<<<n_sm * 8, 256, 0, cs>>>(W, n, scratch);
    vb::ternarize_pack_kernel<<<n_sm * 8, 256, 0, cs>>>(W, N, K, scratch, reinterpret_cast<uint32_t *>(packed_out),
                                                        scale_out);
    VB_CUDA(cudaGetLastError());
    return VLAB200_OK;
}

void bitlinear_int8xint2(int8_t *input0, int8_t *input1, void *output0, float *s, float *ws, int M, int N, int K,
                         void *stream) {
    const int rc = vb::ternary_linear(input0, reinterpret_cast<const uint8_t *>(input1),
                                      output0, nullptr, s, ws,
                                      vb::reference_ws_num(N, K), M, N, K, static_cast<cudaStream_t>(stream), 0);
    if (rc) std::fprintf(stderr, "vla_b200: bitlinear_int8xint2(M=%d,N=%d,K=%d) failed: %d %s\n", M, N, K, rc,
                         vlab200_last_error());
}

void bitlinear_int8xint2_m(int8_t *input0, int8_t *input1, void *output0, float *s, float *ws, int M, int N, int K,
                           void *stream) {
    bitlinear_int8xint2(input0, input1, output0, s, ws, M, N, K, stream);
}

void bitvla_act_quant_cuda(const void *in, int8_t *out, float *scales, int M, int K, void *stream) {
    const int rc = vlab200_act_quant(in, out, scales, M, K, stream);
    if (rc) std::fprintf(stderr, "vla_b200: bitvla_act_quant_cuda(M=%d,K=%d) failed: %d %s\n", M, K, rc,
                         vlab200_last_error());
}

}  // extern "C"
