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
__global__ void __launch_bounds__(GEMV_THREADS) ternary_gemv_kernel(const int8_t *__restrict__ A,
                                                           const uint8_t *__restrict__ Wp,
                                                           __nv_bfloat16 *__restrict__ out,
                                                           int32_t *__restrict__ acc_out,
                                                           const float *__restrict__ s,
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
        if (mm < rows_here) v = __ldg(reinterpret_cast<const uint4 *>(A + (size_t)(m0 + mm) * K) + kk);
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
constexpr int GEMM_BM = 128;
constexpr int GEMM_BK = 128;
constexpr int GEMM_THREADS = 448;

// Separate rings: the activation ring is deep (TMA latency from L2 is several main-loop steps),
// the decoded-weight ring shallow (its producers are warps of this CTA).
constexpr int GEMM_SA = 7, GEMM_SW = 3;

template <int BN, int STAGES>
struct GemmSmem {
    static constexpr int A_BYTES = GEMM_BM * GEMM_BK;
    static constexpr int W_BYTES = BN * GEMM_BK;
    static constexpr int W_OFFSET = GEMM_SA * A_BYTES;
    static constexpr int BAR_OFFSET = W_OFFSET + GEMM_SW * W_BYTES;
    static constexpr int STAGING_OFFSET = BAR_OFFSET + 256;  // 4 epilogue warps x 32 rows x 128 bytes
    static constexpr int TOTAL = STAGING_OFFSET + 4 * 4096 + 1024;  // + alignment slack
};

template <int BN, int STAGES>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
ternary_gemm_tc_kernel(const __grid_constant__ CUtensorMap a_map, const uint8_t *__restrict__ Wp,
                       __nv_bfloat16 *__restrict__ out, int32_t *__restrict__ acc_out,
                       const float *__restrict__ s, const float *__restrict__ ws, int ws_num, int M, int N, int K,
                       int tiles_m, int tiles_n, int *status) {
    using L = GemmSmem<BN, STAGES>;
    extern __shared__ uint8_t gemm_smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(gemm_smem_raw) + 1023) &
                                                ~static_cast<uintptr_t>(1023));
    uint64_t *full_a = reinterpret_cast<uint64_t *>(smem + L::BAR_OFFSET);
    uint64_t *empty_a = full_a + GEMM_SA;
    uint64_t *full_w = empty_a + GEMM_SA;
    uint64_t *empty_w = full_w + GEMM_SW;
    uint64_t *accum_full = empty_w + GEMM_SW;
    uint64_t *accum_empty = accum_full + 2;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(accum_empty + 2);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);

    constexpr bool HALF = BN < 128;  // fewer than eight 16-row weight blocks: four warps decode even K steps, four odd ones
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int ksteps = K / GEMM_BK;
    const int n_tiles = tiles_m * tiles_n;
    const WaitCtx wc{abort_flag, status};

    if (threadIdx.x == 0) {
        for (int i = 0; i < GEMM_SA; ++i) {
            mbar_init(&full_a[i], 1);
            mbar_init(&empty_a[i], 1);
        }
        for (int i = 0; i < GEMM_SW; ++i) {
            mbar_init(&full_w[i], HALF ? 4 : 8);  // one arrival per decode warp of the step
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
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    pdl_launch_dependents();
    pdl_wait();  // the set-up above overlapped the previous kernel's tail

    // tiles are ordered m-fastest so that CTAs running at the same time share a weight slab
    if (warp == 0) {
        if (lane == 0) {
            tma_prefetch_desc(&a_map);
            uint32_t st = 0, ph = 0;
            bool ok = true;
            for (int tile = blockIdx.x; ok && tile < n_tiles; tile += gridDim.x) {
                const int m0 = (tile % tiles_m) * GEMM_BM;
                for (int kt = 0; kt < ksteps; ++kt) {
                    ok = mbar_wait(&empty_a[st], ph ^ 1u, wc, DEV_TIMEOUT_EMPTY);
                    if (!ok) break;
                    mbar_expect_tx(&full_a[st], L::A_BYTES);
                    tma_load_2d(smem + st * L::A_BYTES, &a_map, &full_a[st], kt * GEMM_BK, m0);
                    if (++st == GEMM_SA) { st = 0; ph ^= 1u; }
                }
            }
        }
    } else if (warp == 1) {
        {  // the whole warp walks the tiles, one elected lane issues (uniform control: see gemm.cu)
            constexpr uint32_t idesc = make_idesc(2, 1, 1, 0, 0, GEMM_BM, BN);
            uint32_t st = 0, ph = 0, sw = 0, pw = 0, j = 0;
            bool ok = true;
            for (int tile = blockIdx.x; ok && tile < n_tiles; tile += gridDim.x, ++j) {
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
                    if (elect_one()) {
                        const uint32_t a_addr = smem_u32(smem + st * L::A_BYTES);
                        const uint32_t w_addr = smem_u32(smem + L::W_OFFSET + sw * L::W_BYTES);
#pragma unroll
                        for (int k = 0; k < GEMM_BK / 32; ++k)
                            mma_i8(d_tmem, smem_desc_sw128(a_addr + k * 32, 16, 1024),
                                   smem_desc_sw128(w_addr + k * 32, 16, 1024), idesc, (kt | k) != 0 ? 1u : 0u);
                        tc_commit(&empty_a[st]);
                        tc_commit(&empty_w[sw]);
                    }
                    if (++st == GEMM_SA) { st = 0; ph ^= 1u; }
                    if (++sw == GEMM_SW) { sw = 0; pw ^= 1u; }
                }
                if (!ok) break;
                if (elect_one()) tc_commit(&accum_full[buf]);
            }
        }
    } else if (warp < 10) {
        // ---- decode warps: ladder slots -> swizzled K-major int8 tile ----
        const int dw = warp - 2;                  // 0..7
        constexpr int NBLK = BN / 16;             // 16-row weight blocks in the tile
        constexpr int PER_WARP = HALF ? 1 : NBLK / 8;
        const int blk0 = HALF ? dw & 3 : dw;
        const int nblk_total = N / 16;
        // lane geometry inside one 512-byte chunk (lane t holds the 4 slots at byte offset 16 t)
        const int row_in_blk = 8 * ((lane & 7) >> 2) + 4 * (lane & 1);  // + slot 0..3
        const int chunk16 = 2 * (lane >> 3) + ((lane & 3) >> 1);        // 16-byte column 0..7
        // 128-bit shared stores are served a quarter-warp at a time.  Lanes t and t ^ 4 of a quarter
        // write rows 8 apart (same banks); the upper one walks its slots in the order 2, 3, 0, 1 so that
        // the two never hit the same 16-byte column in the same instruction.
        const bool swap_slots = (lane & 4) != 0;
        // Packed weights are prefetched three main-loop steps ahead into registers: one step is
        // shorter than the latency of a load that misses L2.
        constexpr int PF = 3;
        uint4 pf[PF][PER_WARP];
        const int my_tiles = blockIdx.x < n_tiles ? (n_tiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
        const int total = my_tiles * ksteps;
        auto fetch = [&](int g, uint4 (&dst)[PER_WARP]) {  // g: flat step index over this CTA's tiles
            const int tile = blockIdx.x + (g / ksteps) * gridDim.x, kt = g % ksteps;
            const int nb0 = (tile / tiles_m) * NBLK;
#pragma unroll
            for (int i = 0; i < PER_WARP; ++i) {
                const int nb = nb0 + blk0 + 8 * i;
                dst[i] = (g < total && nb < nblk_total)
                             ? __ldg(reinterpret_cast<const uint4 *>(Wp + (size_t)nb * 4 * K + (size_t)kt * 512) + lane)
                             : make_uint4(0xAAAAAAAAu, 0xAAAAAAAAu, 0xAAAAAAAAu, 0xAAAAAAAAu);
            }
        };
        auto decode_store = [&](const uint4 (&cur)[PER_WARP], uint8_t *wt) {
#pragma unroll
            for (int i = 0; i < PER_WARP; ++i) {
                const int blk = blk0 + 8 * i;
                const uint32_t words[4] = {cur[i].x, cur[i].y, cur[i].z, cur[i].w};
#pragma unroll
                for (int sl = 0; sl < 4; ++sl) {
                    uint32_t d[4];
                    decode_slot(swap_slots ? words[sl ^ 2] : words[sl], d);
                    const int r = blk * 16 + row_in_blk + (swap_slots ? (sl ^ 2) : sl);  // row inside the BN tile
                    uint8_t *dst = wt + (r >> 3) * 1024 + (r & 7) * 128 + ((chunk16 ^ (r & 7)) << 4);
                    *reinterpret_cast<uint4 *>(dst) = make_uint4(d[0], d[1], d[2], d[3]);
                }
            }
        };
        constexpr int STEP = HALF ? 2 : 1;  // this warp decodes steps first, first + STEP, ...
        const int first = HALF ? dw >> 2 : 0;
        bool ok = true;
#pragma unroll
        for (int i = 0; i < PF; ++i) fetch(first + i * STEP, pf[i]);
        for (int g0 = first; ok && g0 < total; g0 += PF * STEP) {
#pragma unroll
            for (int u = 0; u < PF; ++u) {
                const int g = g0 + u * STEP;
                if (g >= total) break;
                uint4 cur[PER_WARP];
#pragma unroll
                for (int i = 0; i < PER_WARP; ++i) cur[i] = pf[u][i];
                fetch(g + PF * STEP, pf[u]);
                const uint32_t st = (uint32_t)g % GEMM_SW, ph = ((uint32_t)g / GEMM_SW) & 1u;
                ok = mbar_wait(&empty_w[st], ph ^ 1u, wc, DEV_TIMEOUT_EMPTY);
                if (!ok) break;
                decode_store(cur, smem + L::W_OFFSET + st * L::W_BYTES);
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(&full_w[st]);
            }
        }
    } else {
        // ---- epilogue warps 10..13: TMEM -> registers -> shared-memory transpose -> global ----
        // A thread owns one accumulator row; writing its 128 bytes straight to global memory would
        // scatter 16-byte pieces over 32 rows per instruction.  Each warp instead stages 32 rows x 64
        // columns (bf16) in shared memory and writes them back as whole 128-byte lines.
        const int q = warp & 3;  // TMEM lane quarter this warp may read
        const int group = N / ws_num;
        uint8_t *stg = smem + L::STAGING_OFFSET + (warp - 10) * 4096;
        const uint32_t my_sw = (uint32_t)(lane & 7);
        uint32_t j = 0;
        bool ok = true;
        for (int tile = blockIdx.x; ok && tile < n_tiles; tile += gridDim.x, ++j) {
            const uint32_t buf = j & 1u;
            const int m0 = (tile % tiles_m) * GEMM_BM, n0 = (tile / tiles_m) * BN;
            const int m = m0 + q * 32 + lane;
            ok = mbar_wait(&accum_full[buf], (j >> 1) & 1u, wc, DEV_TIMEOUT_ACCUM);
            if (!ok) break;
            tc_fence_after();
            const float sm = (m < M) ? s[m] : 1.0f;
            const uint32_t lane_addr = tmem_base + buf * BN + ((uint32_t)(q * 32) << 16);
#pragma unroll 1
            for (int c = 0; c < BN; c += 64) {
                uint32_t r0[32], r1[32];
                tmem_ld32(lane_addr + (uint32_t)c, r0);
                tmem_ld32(lane_addr + (uint32_t)(c + 32), r1);
                tmem_ld_wait();
                const int n = n0 + c;
                if (n >= N) break;  // uniform; N % 16 == 0, so the chunk may be cut after any multiple of 16 columns
                if (acc_out && m < M) {
                    int4 *dst = reinterpret_cast<int4 *>(acc_out + (size_t)m * N + n);
#pragma unroll
                    for (int e = 0; e < 8; ++e)
                        if (n + 4 * e < N)
                            dst[e] = make_int4((int)r0[4 * e], (int)r0[4 * e + 1], (int)r0[4 * e + 2], (int)r0[4 * e + 3]);
#pragma unroll
                    for (int e = 0; e < 8; ++e)
                        if (n + 32 + 4 * e < N)
                            dst[8 + e] = make_int4((int)r1[4 * e], (int)r1[4 * e + 1], (int)r1[4 * e + 2], (int)r1[4 * e + 3]);
                }
                // acc / s * ws evaluated as acc * (ws / s): at most one float ulp from the two-step form.
                // A 32-column chunk never straddles a scale group (the group size is a multiple of 32).
                const float cs0 = __fdiv_rn(ws[n / group], sm);
                const float cs1 = __fdiv_rn(ws[min(n + 32, N - 1) / group], sm);
                uint8_t *mine = stg + lane * 128;
#pragma unroll
                for (int e4 = 0; e4 < 4; ++e4) {
                    uint32_t pa[4], pb[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const __nv_bfloat162 ha = __floats2bfloat162_rn((float)(int)r0[8 * e4 + 2 * e] * cs0,
                                                                        (float)(int)r0[8 * e4 + 2 * e + 1] * cs0);
                        const __nv_bfloat162 hb = __floats2bfloat162_rn((float)(int)r1[8 * e4 + 2 * e] * cs1,
                                                                        (float)(int)r1[8 * e4 + 2 * e + 1] * cs1);
                        pa[e] = *reinterpret_cast<const uint32_t *>(&ha);
                        pb[e] = *reinterpret_cast<const uint32_t *>(&hb);
                    }
                    *reinterpret_cast<uint4 *>(mine + (((uint32_t)e4 ^ my_sw) << 4)) = make_uint4(pa[0], pa[1], pa[2], pa[3]);
                    *reinterpret_cast<uint4 *>(mine + (((uint32_t)(4 + e4) ^ my_sw) << 4)) = make_uint4(pb[0], pb[1], pb[2], pb[3]);
                }
                __syncwarp();
                const int cols_valid = min(64, N - n);  // 32 or 64
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int rr = (lane >> 3) + 4 * i;
                    const int ch = lane & 7;
                    const uint4 v = *reinterpret_cast<const uint4 *>(stg + rr * 128 + (((uint32_t)ch ^ (uint32_t)(rr & 7)) << 4));
                    const int mr = m0 + q * 32 + rr;
                    if (mr < M && ch * 8 < cols_valid)
                        *reinterpret_cast<uint4 *>(out + (size_t)mr * N + n + ch * 8) = v;
                }
                __syncwarp();
            }
            tc_fence_before();
            mbar_arrive(&accum_empty[buf]);
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
    static constexpr int TOTAL = STAGING_OFFSET + 4 * 4096 + 1024;
};

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(GEMM_THREADS, 1)
ternary_gemm_pair_kernel(const __grid_constant__ CUtensorMap a_map, const uint8_t *__restrict__ Wp,
                         __nv_bfloat16 *__restrict__ out, int32_t *__restrict__ acc_out,
                         const float *__restrict__ s, const float *__restrict__ ws, int ws_num, int M, int N, int K,
                         int tiles_mp, int tiles_n, int *status) {
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
        const int nblk_total = N / 16;
        const int row_in_blk = 8 * ((lane & 7) >> 2) + 4 * (lane & 1);  // + slot 0..3
        const int chunk16 = 2 * (lane >> 3) + ((lane & 3) >> 1);        // 16-byte column 0..7
        const bool swap_slots = (lane & 4) != 0;  // see ternary_gemm_tc_kernel: avoids 2-way bank conflicts
        const int my_tiles = cid < n_tiles ? (n_tiles - 1 - cid) / ncl + 1 : 0;
        const int total = my_tiles * ksteps;
        auto fetch = [&](int g, uint4 (&dst)[4]) {
            const int tile = cid + (g / ksteps) * ncl, kt = g % ksteps;
            const int nb0 = (tile / tiles_mp) * (BN / 16) + (int)rank * 8 + hb * 4;
#pragma unroll
            for (int i = 0; i < 4; ++i)
                dst[i] = (g < total && nb0 + i < nblk_total)
                             ? __ldg(reinterpret_cast<const uint4 *>(Wp + (size_t)(nb0 + i) * 4 * K + (size_t)kt * 512) + lane)
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
        const int group = N / ws_num;
        uint8_t *stg = smem + L::STAGING_OFFSET + (warp - 10) * 4096;
        const uint32_t my_sw = (uint32_t)(lane & 7);
        uint32_t j = 0;
        bool ok = true;
        for (int tile = cid; ok && tile < n_tiles; tile += ncl, ++j) {
            const uint32_t buf = j & 1u;
            const int m0 = (tile % tiles_mp) * 256 + (int)rank * 128, n0 = (tile / tiles_mp) * BN;
            const int m = m0 + q * 32 + lane;
            ok = mbar_wait_backoff(&accum_full[buf], (j >> 1) & 1u, wc, DEV_TIMEOUT_ACCUM, 256);
            if (!ok) break;
            tc_fence_after();
            const float sm = (m < M) ? s[m] : 1.0f;
            const uint32_t lane_addr = tmem_base + buf * BN + ((uint32_t)(q * 32) << 16);
            if (m0 < M) {  // warp-uniform: the odd CTA's rows may all lie past M
#pragma unroll 1
                for (int c = 0; c < BN; c += 64) {
                    uint32_t r0[32], r1[32];
                    tmem_ld32(lane_addr + (uint32_t)c, r0);
                    tmem_ld32(lane_addr + (uint32_t)(c + 32), r1);
                    tmem_ld_wait();
                    const int n = n0 + c;
                    if (n >= N) break;
                    if (acc_out && m < M) {
                        int4 *dst = reinterpret_cast<int4 *>(acc_out + (size_t)m * N + n);
#pragma unroll
                        for (int e = 0; e < 8; ++e)
                            if (n + 4 * e < N)
                                dst[e] = make_int4((int)r0[4 * e], (int)r0[4 * e + 1], (int)r0[4 * e + 2], (int)r0[4 * e + 3]);
#pragma unroll
                        for (int e = 0; e < 8; ++e)
                            if (n + 32 + 4 * e < N)
                                dst[8 + e] = make_int4((int)r1[4 * e], (int)r1[4 * e + 1], (int)r1[4 * e + 2], (int)r1[4 * e + 3]);
                    }
                    const float cs0 = __fdiv_rn(ws[n / group], sm);
                    const float cs1 = __fdiv_rn(ws[min(n + 32, N - 1) / group], sm);
                    uint8_t *mine = stg + lane * 128;
#pragma unroll
                    for (int e4 = 0; e4 < 4; ++e4) {
                        uint32_t pa[4], pb[4];
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const __nv_bfloat162 ha = __floats2bfloat162_rn((float)(int)r0[8 * e4 + 2 * e] * cs0,
                                                                            (float)(int)r0[8 * e4 + 2 * e + 1] * cs0);
                            const __nv_bfloat162 hb = __floats2bfloat162_rn((float)(int)r1[8 * e4 + 2 * e] * cs1,
                                                                            (float)(int)r1[8 * e4 + 2 * e + 1] * cs1);
                            pa[e] = *reinterpret_cast<const uint32_t *>(&ha);
                            pb[e] = *reinterpret_cast<const uint32_t *>(&hb);
                        }
                        *reinterpret_cast<uint4 *>(mine + (((uint32_t)e4 ^ my_sw) << 4)) = make_uint4(pa[0], pa[1], pa[2], pa[3]);
                        *reinterpret_cast<uint4 *>(mine + (((uint32_t)(4 + e4) ^ my_sw) << 4)) = make_uint4(pb[0], pb[1], pb[2], pb[3]);
                    }
                    __syncwarp();
                    const int cols_valid = min(64, N - n);
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const int rr = (lane >> 3) + 4 * i;
                        const int ch = lane & 7;
                        const uint4 v = *reinterpret_cast<const uint4 *>(stg + rr * 128 + (((uint32_t)ch ^ (uint32_t)(rr & 7)) << 4));
                        const int mr = m0 + q * 32 + rr;
                        if (mr < M && ch * 8 < cols_valid)
                            *reinterpret_cast<uint4 *>(out + (size_t)mr * N + n + ch * 8) = v;
                    }
                    __syncwarp();
                }
            }
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

template <int BN, int STAGES>
static int launch_gemm_tc(const int8_t *A, const uint8_t *W, __nv_bfloat16 *out, int32_t *acc, const float *s,
                          const float *ws, int ws_num, int M, int N, int K, cudaStream_t st) {
    int *status = device_status_ptr();
    if (!status) return cuda_fail(cudaGetLastError(), "device_status_ptr");
    CUtensorMap amap;
    const uint64_t dims[2] = {(uint64_t)K, (uint64_t)M};
    const uint64_t strides[1] = {(uint64_t)K};
    const uint32_t box[2] = {GEMM_BK, GEMM_BM};
    int rc = make_tensor_map(&amap, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, A, dims, strides, box,
                             CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc) return rc;
    using L = GemmSmem<BN, STAGES>;
    if ((rc = ensure_dyn_smem(ternary_gemm_tc_kernel<BN, STAGES>, L::TOTAL))) return rc;
    const int n_sm = sm_count();
    if (n_sm <= 0) return cuda_fail(cudaGetLastError(), "sm_count");
    const int tiles_m = (M + GEMM_BM - 1) / GEMM_BM, tiles_n = (N + BN - 1) / BN;
    const int nt = tiles_m * tiles_n;
    return launch_pdl(ternary_gemm_tc_kernel<BN, STAGES>, dim3(nt < n_sm ? nt : n_sm), dim3(GEMM_THREADS), L::TOTAL, st, amap, W, out,
                      acc, s, ws, ws_num, M, N, K, tiles_m, tiles_n, status);
}

static int launch_gemm_pair(const int8_t *A, const uint8_t *W, __nv_bfloat16 *out, int32_t *acc, const float *s,
                            const float *ws, int ws_num, int M, int N, int K, cudaStream_t st) {
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
    const int tiles_mp = (M + 255) / 256, tiles_n = (N + 255) / 256;
    const int nt = tiles_mp * tiles_n, pairs = n_sm / 2;
    return launch_pdl(ternary_gemm_pair_kernel, dim3(2 * (nt < pairs ? nt : pairs)), dim3(GEMM_THREADS), PairSmem::TOTAL, st, amap,
                      W, out, acc, s, ws, ws_num, M, N, K, tiles_mp, tiles_n, status);
}

static int ternary_linear(const int8_t *A, const uint8_t *W, __nv_bfloat16 *out, int32_t *acc, const float *s,
                          const float *ws, int ws_num, int M, int N, int K, cudaStream_t st, int force_path) {
    int rc = check_gemm_args(A, W, out, s, ws, ws_num, M, N, K);
    if (rc) return rc;
    if (M == 0) return VLAB200_OK;
    const bool gemv = force_path == 1 || (force_path == 0 && M <= 8);
    if (gemv) {
        if ((size_t)8 * K + 4 * 8 * 16 * sizeof(int) > 200 * 1024) return VLAB200_ERR_UNSUPPORTED;
        for (int m0 = 0; m0 < M; m0 += 8) {
            const int left = M - m0;
            if (left >= 5) rc = launch_gemv<8>(A, W, out, acc, s, ws, ws_num, M, N, K, m0, st);
            else if (left >= 3) rc = launch_gemv<4>(A, W, out, acc, s, ws, ws_num, M, N, K, m0, st);
            else if (left == 2) rc = launch_gemv<2>(A, W, out, acc, s, ws, ws_num, M, N, K, m0, st);
            else rc = launch_gemv<1>(A, W, out, acc, s, ws, ws_num, M, N, K, m0, st);
            if (rc) return rc;
        }
        return VLAB200_OK;
    }
    if ((reinterpret_cast<uintptr_t>(A) & 15) || (reinterpret_cast<uintptr_t>(out) & 15) ||
        (acc && (reinterpret_cast<uintptr_t>(acc) & 15)))
        return VLAB200_ERR_ARG;
    // a 32-column epilogue chunk must not straddle two weight-scale groups; with one group N % 16 == 0 is enough
    if (ws_num > 1 && (N / ws_num) % 32) return VLAB200_ERR_UNSUPPORTED;
    if (force_path == 3) return launch_gemm_pair(A, W, out, acc, s, ws, ws_num, M, N, K, st);
    if (force_path == 0) {
        // ns of a launch (measured back to back, 64 <= M <= 2000): set-up and epilogue, plus waves times 128-wide K steps.  Pair tiles
        // move the fewest bytes per product and win as soon as there are enough of them; with few rows (one image, one prompt) they
        // leave most SMs without work and narrow tiles win: 256 x 1152 x 1152 9.7 -> 7.0 us, 300 x 2560 x 2560 13.8 -> 11.3 us,
        // 256 x 1152 (K 4352) 18.5 -> 16.0 us; 300 x 13824 x 2560 takes 22.2 us in pairs and 33.1 / 41.5 us in tiles of 128 / 64.
        const int n_sm = sm_count(), tm = (M + 127) / 128, tp = (M + 255) / 256, ks = K / 128;
        if (n_sm <= 0) return cuda_fail(cudaGetLastError(), "sm_count");
        auto waves = [](int tiles, int units) { return (tiles + units - 1) / units; };
        const int c64 = 3600 + 370 * ks * waves(tm * ((N + 63) / 64), n_sm), c128 = 4400 + 460 * ks * waves(tm * ((N + 127) / 128), n_sm);
        const int cpair = N >= 256 && n_sm >= 2 ? 6400 + 360 * ks * waves(tp * ((N + 255) / 256), n_sm / 2) : c64 + c128;
        if (cpair <= c64 && cpair <= c128) return launch_gemm_pair(A, W, out, acc, s, ws, ws_num, M, N, K, st);
        if (c64 < c128) return launch_gemm_tc<64, 4>(A, W, out, acc, s, ws, ws_num, M, N, K, st);
        return launch_gemm_tc<128, 4>(A, W, out, acc, s, ws, ws_num, M, N, K, st);
    }
    if (N >= 256) return launch_gemm_tc<256, 4>(A, W, out, acc, s, ws, ws_num, M, N, K, st);
    return launch_gemm_tc<128, 4>(A, W, out, acc, s, ws, ws_num, M, N, K, st);
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
    return vb::ternary_linear(A, W_ladder, static_cast<__nv_bfloat16 *>(out_bf16), acc_out, s, ws, ws_num, M, N, K,
                              static_cast<cudaStream_t>(stream), path);
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
                                      static_cast<__nv_bfloat16 *>(output0), nullptr, s, ws,
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
