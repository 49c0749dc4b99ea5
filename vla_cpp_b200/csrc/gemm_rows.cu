// The bf16 GEMM for few rows: what a handful of observations, a prompt or the views of one request make of a projection.
//
// There a launch is a chain of latencies, not a stream of work: dependency wait, first operand tile, K loop, epilogue, drain.  This kernel
// keeps the tiles and the arithmetic of gemm.cu's 128 x 64 and 128 x 128 tilings and shortens the chain around them:
//
//   * One tile per CTA and less than half an SM per CTA (96 KB ring, at most 128 TMEM columns, 96 registers a thread): the next kernel's
//     CTAs become resident while this kernel's still run, so their set-up is over when the dependency resolves, and where a call has
//     more tiles than SMs two tiles share one and cover each other's epilogue.
//   * The weights do not depend on the kernel in front: the whole ring's weight tiles are requested before the dependency wait
//     (p.w_early), only the activation tiles come after it.
//   * Residual epilogue: the float32 rows it adds to are fetched during the K loop.
//   * K slices (long K, narrow N): the `slices` CTAs of a cluster each take a part of K; then every CTA collects the partial sums of
//     BN / slices of the tile's columns from its peers through distributed shared memory and adds them in slice order.
//     No float workspace, no second launch.
//   * ROPE epilogue: q | k | v leave rotated, in the q buffer and the K / V pages.  A tile holds columns [k, k + 32) of a head's first half
//     and the matching columns of its second half (two 32-row weight boxes), so a thread has both elements of every pair.
//
//   warp 0 TMA, warp 1 tcgen05.mma, warps 2-9 epilogue (quarter = warp & 3, column half = (warp - 2) / 4); warps 2-5 sum a^2 per row
//   during the K loop where an RMS factor is wanted.
#include <cuda_bf16.h>

#include "gemm.h"
#include "gemm_epi.cuh"
#include "host_common.h"
#include "tc5.cuh"

namespace vb {

constexpr int R_BM = 128, R_BK = 64, R_THREADS = 320;

// DEEP: a ring of most of an SM's shared memory for calls whose tiles leave no SM with two of them.  A K step of the shallow ring takes
// 0.28 us there, a quarter (third) of a load's latency.
template <int BN, bool DEEP>
struct RowsCfg {
    static constexpr int STAGES = (BN == 64 ? 4 : 3) * (DEEP ? 2 : 1);
    static constexpr int A_BYTES = R_BM * 128, STAGE_BYTES = A_BYTES + BN * 128;
    static constexpr int BAR_OFFSET = STAGES * STAGE_BYTES, STATS_OFFSET = BAR_OFFSET + 256;
    static constexpr int SMEM = STATS_OFFSET + R_BM * 4 + 1024;  // + alignment slack
};

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
}

__device__ __forceinline__ uint32_t rows_pack(float a, float b) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t *>(&h);
}

template <int BN, int EPI, bool DEEP>
__global__ void __launch_bounds__(R_THREADS, DEEP ? 1 : 2)
gemm_rows_kernel(const __grid_constant__ CUtensorMap a_map, const __grid_constant__ CUtensorMap w_map, const __grid_constant__ GemmParams p,
                 const __grid_constant__ RopeParams rp, int tiles_n, int slices) {
    using Cfg = RowsCfg<BN, DEEP>;
    constexpr int STAGES = Cfg::STAGES;
    extern __shared__ uint8_t rows_smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(rows_smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + Cfg::BAR_OFFSET), *empty = full + STAGES, *accum_full = empty + STAGES;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(accum_full + 1);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    float *stats = reinterpret_cast<float *>(smem + Cfg::STATS_OFFSET);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = slices > 1 ? (int)cluster_ctarank() : 0;
    const int tile = (int)blockIdx.x / slices;
    const int m0 = (tile / tiles_n) * R_BM, n0 = (tile % tiles_n) * BN;
    const int ksteps = (p.K + R_BK - 1) / R_BK;
    const int kbeg = rank * ksteps / slices, nk = (rank + 1) * ksteps / slices - kbeg;
    const bool use_rms = EPI != EPI_RESIDUAL && p.use_rms;
    const WaitCtx wc{abort_flag, p.status};

    if (threadIdx.x == 0) {
        for (int i = 0; i < STAGES; ++i) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], use_rms ? 5 : 1);
        }
        mbar_init(accum_full, 1);
        *abort_flag = 0;
        fence_barrier_init();
        tma_prefetch_desc(&a_map);
        tma_prefetch_desc(&w_map);
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, BN);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    if (slices > 1) cluster_sync_all();  // every CTA of the cluster runs before another one writes to its shared memory
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    pdl_launch_dependents();

    const int qtr = warp & 3, grp = (warp - 2) >> 2, row = qtr * 32 + lane, m = m0 + row;
    const bool row_ok = m < p.M;
    const uint32_t lane_addr = tmem_base + ((uint32_t)(qtr * 32) << 16);
    // the columns of the tile that this CTA finishes, and of those the ones of this warp's column half
    const int own_w = BN / slices, own0 = rank * own_w;
    const int my_w = own_w >= 16 ? own_w / 2 : (grp == 0 ? own_w : 0), my0 = own0 + (own_w >= 16 ? grp * my_w : 0);
    bool ok = true;

    if (warp == 0) {
        if (lane == 0) {
            // weight rows of the tile's two halves
            int w_lo = n0, w_hi = n0 + BN / 2;
            if (EPI == EPI_ROPE) {
                const int head = n0 / rp.hd;
                if (head < rp.n_q + rp.n_kv_proj) {
                    w_lo = head * rp.hd + (n0 % rp.hd) / 2;
                    w_hi = w_lo + rp.hd / 2;
                }
            }
            auto load_w = [&](int st, int kt) {
                uint8_t *sw = smem + st * Cfg::STAGE_BYTES + Cfg::A_BYTES;
                mbar_expect_tx(&full[st], Cfg::STAGE_BYTES);
                tma_load_2d(sw, &w_map, &full[st], kt * R_BK, w_lo);
                tma_load_2d(sw + BN * 64, &w_map, &full[st], kt * R_BK, w_hi);
            };
            const int pre = nk < STAGES ? nk : STAGES;
            if (!p.w_early) pdl_wait();
            for (int i = 0; i < pre; ++i) load_w(i, kbeg + i);
            if (p.w_early) pdl_wait();
            for (int i = 0; i < pre; ++i) tma_load_2d(smem + i * Cfg::STAGE_BYTES, &a_map, &full[i], (kbeg + i) * R_BK, m0);
            uint32_t st = 0, ph = 0;
            for (int kt = pre; kt < nk; ++kt) {
                if (!mbar_wait(&empty[st], ph, wc, DEV_TIMEOUT_EMPTY)) break;
                load_w(st, kbeg + kt);
                tma_load_2d(smem + st * Cfg::STAGE_BYTES, &a_map, &full[st], (kbeg + kt) * R_BK, m0);
                if (++st == STAGES) { st = 0; ph ^= 1u; }
            }
        }
    } else if (warp == 1) {
        constexpr uint32_t idesc = make_idesc(1, 1, 1, 0, 0, R_BM, BN);
        const uint64_t a_desc0 = smem_desc_sw128(smem_u32(smem), 16, 1024), b_desc0 = smem_desc_sw128(smem_u32(smem + Cfg::A_BYTES), 16, 1024);
        uint32_t st = 0, ph = 0;
        for (int kt = 0; kt < nk; ++kt) {
            ok = warp_wait(&full[st], ph, wc, DEV_TIMEOUT_FULL);
            if (!ok) break;
            tc_fence_after();
            const uint64_t off = (uint64_t)(st * (Cfg::STAGE_BYTES >> 4));
            if (elect_one()) {
#pragma unroll
                for (int k = 0; k < R_BK / 16; ++k) mma_f16(tmem_base, a_desc0 + off + 2 * k, b_desc0 + off + 2 * k, idesc, (kt | k) != 0 ? 1u : 0u);
                tc_commit(&empty[st]);
            }
            if (++st == STAGES) { st = 0; ph ^= 1u; }
        }
        if (ok && elect_one()) tc_commit(accum_full);
    } else {
        pdl_wait();
        if (use_rms && grp == 0) {
            // sum a^2 per row from the A tiles, in the order of gemm.cu (the same bits)
            const uint32_t row_base = (row >> 3) * 1024 + (row & 7) * 128, sw = row & 7;
            uint32_t st = 0, ph = 0;
            float s0 = 0.0f, s1 = 0.0f;
            for (int kt = 0; kt < nk; ++kt) {
                ok = mbar_wait(&full[st], ph, wc, DEV_TIMEOUT_FULL);
                if (!ok) break;
                const uint8_t *at = smem + st * Cfg::STAGE_BYTES + row_base;
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    const uint4 v = *reinterpret_cast<const uint4 *>(at + ((c ^ sw) << 4));
                    const __nv_bfloat162 *h2 = reinterpret_cast<const __nv_bfloat162 *>(&v);
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const float2 f = __bfloat1622float2(h2[e]);
                        s0 = fmaf(f.x, f.x, s0);
                        s1 = fmaf(f.y, f.y, s1);
                    }
                }
                stage_release(&empty[st], s0 + s1, lane);
                if (++st == STAGES) { st = 0; ph ^= 1u; }
            }
            stats[row] = s0 + s1;
        }
        __syncwarp();
        if (use_rms) asm volatile("bar.sync 1, 256;" ::: "memory");  // the epilogue warps
    }

    // ---- what the epilogue needs besides the accumulator, fetched while the products run ----
    uint32_t pre[EPI == EPI_RESIDUAL || EPI == EPI_ROPE ? 32 : 1];
    int obs = 0, tok = 0, head = 0, k0 = 0;  // ROPE
    if (EPI == EPI_RESIDUAL && warp >= 2 && row_ok) {
        const float *hrow = p.h + (size_t)m * p.ld_out;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int n = n0 + my0 + 8 * i;
            if (8 * i < my_w && n < p.N) {
                if (p.al32) {
                    uint32_t t[8];
                    ld_global_v8(hrow + n, t);
#pragma unroll
                    for (int e = 0; e < 8; ++e) pre[8 * i + e] = t[e];
                } else {
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const uint4 t = *reinterpret_cast<const uint4 *>(hrow + n + 4 * e);
                        pre[8 * i + 4 * e] = t.x; pre[8 * i + 4 * e + 1] = t.y; pre[8 * i + 4 * e + 2] = t.z; pre[8 * i + 4 * e + 3] = t.w;
                    }
                }
            }
        }
    }
    if (EPI == EPI_ROPE && warp >= 2) {
        obs = m / rp.seq;
        tok = m % rp.seq;
        head = n0 / rp.hd;
        k0 = (n0 % rp.hd) / 2 + 16 * grp;
        if (row_ok && head < rp.n_q + rp.n_kv_proj) {
            const uint4 *cp = reinterpret_cast<const uint4 *>(rp.cos_t + (size_t)tok * (rp.hd / 2) + k0);
            const uint4 *sp = reinterpret_cast<const uint4 *>(rp.sin_t + (size_t)tok * (rp.hd / 2) + k0);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint4 c = __ldg(cp + i), s = __ldg(sp + i);
                pre[4 * i] = c.x; pre[4 * i + 1] = c.y; pre[4 * i + 2] = c.z; pre[4 * i + 3] = c.w;
                pre[16 + 4 * i] = s.x; pre[16 + 4 * i + 1] = s.y; pre[16 + 4 * i + 2] = s.z; pre[16 + 4 * i + 3] = s.w;
            }
        }
    }
    if (warp >= 2 && ok) {
        ok = mbar_wait(accum_full, 0u, wc, DEV_TIMEOUT_ACCUM);
        tc_fence_after();
    }

    // ---- K slices: partial sums to the CTA that finishes their columns, [sender][4 columns][row], over the drained ring ----
    const int slot_bytes = own_w * R_BM * 4;
    if (EPI == EPI_RESIDUAL && slices > 1) {
        __syncwarp();
        cluster_sync_all();  // every CTA's products are done: nothing reads a ring any more
        if (warp >= 2 && ok && my_w > 0) {
            for (int r = 0; r < slices; ++r) {
                if (r == rank) continue;
                const uint32_t dst = cluster_addr(smem_u32(smem) + (uint32_t)((rank < r ? rank : rank - 1) * slot_bytes + row * 16), (uint32_t)r);
                for (int c = 0; c < my_w; c += 8) {
                    const int rel = my0 - own0 + c;
                    uint32_t v[8];
                    tmem_ld8(lane_addr + (uint32_t)(r * own_w + rel), v);
                    tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < 2; ++i)
                        st_cluster_v4(dst + (uint32_t)((rel / 4 + i) * R_BM * 16), v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
                }
            }
        }
        __syncwarp();
        cluster_sync_all();
    }

    if (warp >= 2 && ok) {
        const float rms = use_rms ? rsqrtf(stats[row] / (float)p.K + p.eps) : 1.0f;
        if constexpr (EPI == EPI_RESIDUAL) {
#pragma unroll 1
            for (int c32 = 0; c32 < my_w; c32 += 32) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int c = c32 + 8 * i, n = n0 + my0 + c;
                    if (c >= my_w || n >= p.N) break;
                    uint32_t v[8], a[8], w[4];
                    tmem_ld8(lane_addr + (uint32_t)(my0 + c), v);
                    tmem_ld_wait();
                    if (slices > 1) {
                        float acc[8];
                        const uint8_t *src = smem + (my0 - own0 + c) / 4 * R_BM * 16 + row * 16;
                        for (int s = 0; s < slices; ++s) {
                            float f[8];
                            if (s == rank) {
#pragma unroll
                                for (int e = 0; e < 8; ++e) f[e] = __uint_as_float(v[e]);
                            } else {
                                const float4 *o = reinterpret_cast<const float4 *>(src + (s < rank ? s : s - 1) * slot_bytes);
                                const float4 x = o[0], y = o[R_BM];
                                f[0] = x.x; f[1] = x.y; f[2] = x.z; f[3] = x.w; f[4] = y.x; f[5] = y.y; f[6] = y.z; f[7] = y.w;
                            }
#pragma unroll
                            for (int e = 0; e < 8; ++e) acc[e] = s == 0 ? f[e] : acc[e] + f[e];
                        }
#pragma unroll
                        for (int e = 0; e < 8; ++e) v[e] = __float_as_uint(acc[e]);
                    }
                    if (!row_ok) continue;
                    if (p.colscale) {
#pragma unroll
                        for (int e = 0; e < 8; ++e) v[e] = __float_as_uint(__uint_as_float(v[e]) * __ldg(p.colscale + n + e));
                    }
                    if (p.bias) {
#pragma unroll
                        for (int e = 0; e < 8; ++e) v[e] = __float_as_uint(__uint_as_float(v[e]) + __ldg(p.bias + n + e));
                    }
                    float *hrow = p.h + (size_t)m * p.ld_out + n;
                    if (c32 == 0) {
#pragma unroll
                        for (int e = 0; e < 8; ++e) a[e] = pre[8 * i + e];
                    } else {  // 128-column tiles: the second half of the warp's columns
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            const uint4 t = *reinterpret_cast<const uint4 *>(hrow + 4 * e);
                            a[4 * e] = t.x; a[4 * e + 1] = t.y; a[4 * e + 2] = t.z; a[4 * e + 3] = t.w;
                        }
                    }
#pragma unroll
                    for (int e = 0; e < 8; ++e) a[e] = __float_as_uint(__uint_as_float(a[e]) + __uint_as_float(v[e]));
                    if (p.al32) {
                        st_global_v8(hrow, a);
                    } else {
                        reinterpret_cast<uint4 *>(hrow)[0] = make_uint4(a[0], a[1], a[2], a[3]);
                        reinterpret_cast<uint4 *>(hrow)[1] = make_uint4(a[4], a[5], a[6], a[7]);
                    }
#pragma unroll
                    for (int e = 0; e < 4; ++e) w[e] = rows_pack(__uint_as_float(a[2 * e]), __uint_as_float(a[2 * e + 1]));
                    *reinterpret_cast<uint4 *>(p.out_bf + (size_t)m * p.ld_out + n) = make_uint4(w[0], w[1], w[2], w[3]);
                }
            }
        } else if constexpr (EPI == EPI_ROPE) {
            uint32_t lo[16], hi[16], wl[8], wh[8];
            tmem_ld16(lane_addr + (uint32_t)(16 * grp), lo);
            tmem_ld16(lane_addr + (uint32_t)(BN / 2 + 16 * grp), hi);
            tmem_ld_wait();
            if (row_ok) {
                const bool rot = head < rp.n_q + rp.n_kv_proj;
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    float l[2], h[2];
#pragma unroll
                    for (int t = 0; t < 2; ++t) {
                        const float a = __uint_as_float(lo[2 * e + t]) * rms, b = __uint_as_float(hi[2 * e + t]) * rms;
                        const float cs = __uint_as_float(pre[2 * e + t]), sn = __uint_as_float(pre[16 + 2 * e + t]);
                        l[t] = rot ? a * cs - b * sn : a;
                        h[t] = rot ? b * cs + a * sn : b;
                    }
                    wl[e] = rows_pack(l[0], l[1]);
                    wh[e] = rows_pack(h[0], h[1]);
                }
                __nv_bfloat16 *dst;
                if (head < rp.n_q) dst = rp.q_out + (((size_t)obs * rp.n_q + head) * rp.seq + tok) * rp.hd;
                else if (rot) dst = rp.k_pages + (((size_t)obs * rp.n_kv_store + head - rp.n_q) * rp.cap + rp.row0 + tok) * rp.hd;
                else dst = rp.v_pages + (((size_t)obs * rp.n_kv_store + head - rp.n_q - rp.n_kv_proj) * rp.cap + rp.row0 + tok) * rp.hd;
                st_global_v8(dst + (rot ? k0 : n0 % rp.hd + 16 * grp), wl);
                st_global_v8(dst + (rot ? k0 + rp.hd / 2 : n0 % rp.hd + BN / 2 + 16 * grp), wh);
            }
        } else {
            const size_t mo = mapped_row(p, m);
#pragma unroll 1
            for (int c = my0; c < my0 + my_w; c += 32) {
                const int n = n0 + c;
                if (n >= p.N) break;
                uint32_t v[32];
                tmem_ld32(lane_addr + (uint32_t)c, v);
                tmem_ld_wait();
                if (!row_ok) continue;
                if constexpr (EPI == EPI_GATED) {
                    uint32_t w[8];
                    if (p.act == ACT_SILU) gated_chunk<ACT_SILU>(v, rms, w);
                    else gated_chunk<ACT_GELU_TANH>(v, rms, w);
                    __nv_bfloat16 *brow = p.out_bf + mo * p.ld_out + (n >> 1);
                    if (p.al32 && n + 16 < p.N) {
                        st_global_v8(brow, w);
                    } else {
                        reinterpret_cast<uint4 *>(brow)[0] = make_uint4(w[0], w[1], w[2], w[3]);
                        if (n + 16 < p.N) reinterpret_cast<uint4 *>(brow)[1] = make_uint4(w[4], w[5], w[6], w[7]);
                    }
                } else {
                    bias_act_chunk(p, v, rms, m, mo, n);
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, BN);
    }
}

template <int BN>
static int rows_clusters(int slices) {
    // (of the deep form: one CTA an SM, which is also what the cost rule counts on)
    if (ensure_dyn_smem(gemm_rows_kernel<BN, EPI_RESIDUAL, true>, RowsCfg<BN, true>::SMEM) != VLAB200_OK) return 0;
    return max_active_clusters(reinterpret_cast<const void *>(gemm_rows_kernel<BN, EPI_RESIDUAL, true>), R_THREADS, RowsCfg<BN, true>::SMEM, slices);
}
int gemm_rows_clusters(int bn, int slices) { return bn == 64 ? rows_clusters<64>(slices) : rows_clusters<128>(slices); }

template <int BN, int EPI, bool DEEP>
static int launch_rows_as(const CUtensorMap &amap, const CUtensorMap &wmap, const GemmParams &p, const RopeParams &rp, int tiles, int tiles_n, int slices,
                          cudaStream_t st) {
    if (int rc = ensure_dyn_smem(gemm_rows_kernel<BN, EPI, DEEP>, RowsCfg<BN, DEEP>::SMEM)) return rc;
    if (slices > 1)
        return launch_pdl_cluster(gemm_rows_kernel<BN, EPI, DEEP>, dim3(tiles * slices), dim3(R_THREADS), RowsCfg<BN, DEEP>::SMEM, slices, st, amap, wmap, p, rp,
                                  tiles_n, slices);
    return launch_pdl(gemm_rows_kernel<BN, EPI, DEEP>, dim3(tiles), dim3(R_THREADS), RowsCfg<BN, DEEP>::SMEM, st, amap, wmap, p, rp, tiles_n, 1);
}

template <int BN, int EPI>
static int launch_rows(const CUtensorMap &amap, const CUtensorMap &wmap, const GemmParams &p, const RopeParams &rp, int slices, cudaStream_t st) {
    const int tiles_n = (p.N + BN - 1) / BN, tiles = (p.M + R_BM - 1) / R_BM * tiles_n, nk = ((p.K + R_BK - 1) / R_BK + slices - 1) / slices;
    const bool deep = tiles * slices <= sm_count() && nk > RowsCfg<BN, false>::STAGES;
    if (deep) return launch_rows_as<BN, EPI, true>(amap, wmap, p, rp, tiles, tiles_n, slices, st);
    return launch_rows_as<BN, EPI, false>(amap, wmap, p, rp, tiles, tiles_n, slices, st);
}

// Arguments were checked by the callers (dense_gemm and qkv_rope_rows): 16-byte aligned A and W, N % 8, K % 8, lda % 8 == 0.
static int gemm_rows(const void *A, int lda, const void *W, GemmParams p, const RopeParams &rp, int bn, int slices, cudaStream_t stream) {
    p.status = device_status_ptr();
    if (!p.status) return cuda_fail(cudaGetLastError(), "device_status_ptr");
    CUtensorMap amap, wmap;
    const uint64_t adims[2] = {(uint64_t)p.K, (uint64_t)p.M}, wdims[2] = {(uint64_t)p.K, (uint64_t)p.N};
    const uint64_t astrides[1] = {(uint64_t)lda * 2}, wstrides[1] = {(uint64_t)p.K * 2};
    const uint32_t abox[2] = {R_BK, R_BM}, wbox[2] = {R_BK, (uint32_t)bn / 2};
    int rc = make_tensor_map(&amap, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, A, adims, astrides, abox, CU_TENSOR_MAP_SWIZZLE_128B);
    if (!rc) rc = make_tensor_map(&wmap, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, W, wdims, wstrides, wbox, CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc) return rc;
    if (p.epi == EPI_ROPE) return launch_rows<64, EPI_ROPE>(amap, wmap, p, rp, 1, stream);
    if (bn == 64) {
        if (p.epi == EPI_RESIDUAL) return launch_rows<64, EPI_RESIDUAL>(amap, wmap, p, rp, slices, stream);
        if (p.epi == EPI_GATED) return launch_rows<64, EPI_GATED>(amap, wmap, p, rp, 1, stream);
        return launch_rows<64, EPI_BIAS_ACT>(amap, wmap, p, rp, 1, stream);
    }
    if (p.epi == EPI_RESIDUAL) return launch_rows<128, EPI_RESIDUAL>(amap, wmap, p, rp, slices, stream);
    if (p.epi == EPI_GATED) return launch_rows<128, EPI_GATED>(amap, wmap, p, rp, 1, stream);
    return launch_rows<128, EPI_BIAS_ACT>(amap, wmap, p, rp, 1, stream);
}

int dense_gemm_rows(const void *A, int lda, const void *W, const GemmParams &p, int bn, int slices, cudaStream_t stream) {
    return gemm_rows(A, lda, W, p, RopeParams{}, bn, slices, stream);
}

int qkv_rope_rows(const void *A, const void *W, int M, int K, bool use_rms, float eps, const RopeParams &rp, cudaStream_t stream) {
    if (!A || !W || M <= 0 || K <= 0 || K % 8 || rp.hd % 64 || rp.seq <= 0) return VLAB200_ERR_ARG;
    auto al32 = [](const void *q) { return (reinterpret_cast<uintptr_t>(q) & 31) == 0; };
    if (!al32(A) || !al32(W) || !al32(rp.q_out) || !al32(rp.k_pages) || !al32(rp.v_pages) || !al32(rp.cos_t) || !al32(rp.sin_t)) return VLAB200_ERR_UNSUPPORTED;
    GemmParams p{};
    p.M = M; p.N = (rp.n_q + 2 * rp.n_kv_proj) * rp.hd; p.K = K; p.epi = EPI_ROPE; p.use_rms = use_rms ? 1 : 0; p.eps = eps; p.w_early = 1;
    return gemm_rows(A, K, W, p, rp, 64, 1, stream);
}

}  // namespace vb
