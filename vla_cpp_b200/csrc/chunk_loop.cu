// One observation, the whole Euler loop, ONE kernel.
//
// With a single observation the suffix is 50 / 51 rows: every product of the loop streams its weights once and does
// almost no arithmetic, and a launch per operator spends most of its time between kernels (about 1,600 launches per
// chunk for a pi0-shaped expert).  Here one persistent cooperative kernel (clusters of eight CTAs, one CTA of 256 + 64
// threads per SM) walks a table of PHASES -- the operators of one Euler step, src/models/pi0.cpp:570-588,
// src/models/smolvla.cpp:1393-1418 -- and separates them with a grid-wide barrier (one atomic arrival + a bounded acquire
// spin per CTA).  Per layer: q|k|v, attention, Wo + residual, gate/up, Wdown + residual = five phases.
//
// Phase kinds
//   GEMM     C[M <= 64][N] = A[M][K] W[N][K]^T on the tensor cores with the operands SWAPPED: 128 weight rows are tcgen05's M, the
//            tokens its N = 64 columns, so a tile of the accumulator is [weight row = TMEM lane][token].  Groups of kd = 1, 2, 4
//            or 8 CTAs of one cluster share a contiguous range of 8-column groups; each CTA multiplies ITS 1 / kd of K and sends
//            every column's partial sums to the CTA of the group that owns the column (one bulk copy into its shared memory per
//            destination, counted on an mbarrier there), which adds the kd parts in a fixed order and runs the epilogue: residual +=
//            projection with the bf16 mirror and sums of squares (the consumer's RMS factor), act(gate) * up, RMS factor + NeoX
//            rotation + append of q|k|v, bias + activation, the Euler update.  A CTA so reads M x K / kd of the activations
//            instead of all of them: without the split the 148 copies of A alone were 2 us of L2 traffic per phase (4 x that
//            for Wdown), and Wo / Wdown kept 64 of 148 SMs busy.  kd is chosen per product by choose_kd; a product too wide for
//            the shared memory of one phase (an MLP above about 5,700 columns at a width of 1024) is cut into several by plan_gemm.
//            Weights and activations lie as tcgen05 reads them (K-major, SWIZZLE_128B blocks of 64 columns), weights as
//            [CTA group][64-column block][row], so that any range of blocks is one contiguous cp.async.bulk (a bulk copy costs
//            its issuing thread 40-60 ns whatever its size; 51 row copies of 2 KB took 3 us).  They arrive in a ring that one
//            thread feeds from a cursor which runs AHEAD of the computation, across phase boundaries and barriers (weights do
//            not depend on anything the loop computes), so HBM streams while the CTAs wait for each other; another warp
//            issues the products as soon as the A tile and the next ring stage have landed.
//            (mma.sync on the same tiles ran at 410 - 460 multiply-adds per clock and SM, a ninth of tcgen05's rate: 2840
//            clocks for Wo's 64 x 72 x 256, 5755 for Wdown's.)
//   ATT      units of (kv head, 32 stacked query rows), a group of CTAs each, the keys split between its CTAs: S = Q K^T and P V
//            by mma.sync on tiles staged by bulk copies, several key blocks with a running maximum where a CTA's keys do not fit
//            at once; un-normalised O rows, maximum and row sum go to the CTA of the group that merges the row.
//   EMBED    action-in projection (+ pi0's state token) on CUDA cores.
// Everything one CTA writes for another outside its cluster goes through L2 (st / ld .cg, bulk copies), never through L1.  Phase
// descriptors are fetched one phase ahead into shared memory (cp.async), the weight feeder's table sits there too.
// Results do not depend on the run: every sum has a fixed order.  They may differ in rounding between GPUs, where another number of clusters
// fits: the order follows from the number of CTAs.
// What bounds a phase here is a chain of round trips (barrier arrival + poll, A tile, products, exchange, store drain),
// not the tensor pipe and not HBM.
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <new>
#include <vector>

#include "chunk_loop.h"
#include "gemm.h"
#include "host_common.h"
#include "tc5.cuh"

namespace vb {
namespace {

enum { PH_GEMM = 0, PH_ATT = 2, PH_EMBED = 4 };
enum { OUT_RESID = 0, OUT_GATED = 1, OUT_QKV = 2, OUT_BIAS_ACT = 3, OUT_EULER = 4 };

constexpr int CL_THREADS = 256;   // the eight computing warps
constexpr int CL_BLOCK = 320;     // + one warp whose lane 0 feeds the weight ring, one that issues the products
constexpr int CL_CLUSTER = 8;     // CTAs per cluster (the portable maximum)
constexpr int CL_STAGES = 4;
constexpr int CL_STAGE_BYTES = 22528;                             // 22 tiles (8 columns x 64 K) of 1 KB
constexpr int CL_GROUP_N8 = 22;                                   // most 8-column groups of a CTA group in one phase: 176 weight rows, two tiles of 128
constexpr int CL_LAYER_PRODUCTS = 7;                              // most phases of a layer beside attention (make_plan)
constexpr int CL_TMEM_COLS = 128;                                 // an accumulator of 64 columns (tokens) per tile of 128 weight rows
constexpr int CL_DESC_BYTES = 352;                                // one phase descriptor slot (two of them: this phase, the next)
constexpr int CL_DESC_OFF = 1536;
constexpr int CL_WTAB_OFF = 2304;                                 // weight feeder table: one 16-byte entry per GEMM phase of a step
constexpr int CL_WTAB_MAX = 240;
constexpr int CL_HEADER = 6144;                                   // barriers, abort flag, small float arrays, descriptors, feeder table
constexpr int CL_RING_OFF = CL_HEADER;
constexpr int CL_ARENA_OFF = CL_RING_OFF + CL_STAGES * CL_STAGE_BYTES;
constexpr int CL_SMEM = 232448;
constexpr int CL_ARENA = CL_SMEM - CL_ARENA_OFF;
constexpr int CL_EMBED_ROWS = 10;
constexpr int CL_DEV_TIMEOUT = 105;

// A bf16 matrix [rows][cols] as tcgen05 reads it: blocks of 64 columns, each rows8 rows (rows rounded up to 8) of 128 bytes whose
// 16-byte chunks are permuted by the row (SWIZZLE_128B).  Element (row, col) sits at this byte offset.
__host__ __device__ __forceinline__ uint32_t sw_off(int rows8, int row, int col) {
    return (uint32_t)((col >> 6) * rows8 + row) * 128u + (uint32_t)((((col >> 3) & 7) ^ (row & 7)) << 4) + (uint32_t)(col & 7) * 2u;
}

struct alignas(16) LoopPhase {
    int type, out_mode, act, use_rms;
    int M, N8, K, kd;                   // N8: 8-column groups; kd: CTAs that share a product's K / an attention unit's keys
    int n8_0, N;                        // the phase's first 8-column group, columns of the whole product
    int half, ssq_n, row_off, out_rows8;  // half = head_dim / 2 (q|k|v)
    float eps, scale_log2, dt;
    int bias_step_stride;
    const uint8_t *Ap, *Wp;             // images of A ([M][K]) and W ([N][K])
    float *out_f32, *h, *x;
    float *ssq_out;                     // [N8][64]: sum of squares of the bf16 values this phase writes, per 8-column group and row (optional)
    const float *ssq_in;                // use_rms: the producer's partials, ssq_n of them per row
    // pi0.5 (adaptive RMSNorm, gated residuals): per-step vectors, element stride mod_stride between steps
    const float *colscale;              // OUT_RESID: gate on the projection before it is added
    const float *scale_next;            // OUT_RESID / EMBED: the mirror is written as bf16(h * (1 + scale_next[col])) for the norm that reads it
    long long mod_stride;
    uint8_t *outp;                      // image the phase writes
    uint8_t *hbp;                       // EMBED: image of the residual mirror [S][H]
    uint8_t *qp, *kpp, *vpp;            // padded rows of hd * 2 + 16 bytes: q [n_q S][hd], this layer's K / V pages [n_kv cap][hd]
    const float *bias, *rope;
    int n_q, n_kvp, n_kv, g, S, R, n_rt, per, ks, kv_len, P, mask_mode, cap, chunk, A_dim, sd, H;
    int k_off, p_off, stage_off, recv_off, early_k, early_v;  // ATT: K, probabilities, staged and received rows in the arena; may K / V be copied before the barrier
    const __nv_bfloat16 *w_dense, *w2;  // EMBED: W_ain [H][A], W_sp [H][sd] (plain row-major)
    const float *b2;                    // EMBED: b_sp
};

struct LoopParams {
    const LoopPhase *phases;
    const void *wtab;  // WEntry per GEMM phase of a step, in phase order
    int n_phases, steps, n_wtab, att_cta;  // att_cta: CTAs per attention unit
    unsigned *counter;
    int *status;
    const float *state;
    const int32_t *pad;
    unsigned long long *trace;  // developer aid: global-timer stamp of CTA 0 after every barrier (nullptr: off)
    // prefix rows of the engine's pages -> padded pages, once per call
    const __nv_bfloat16 *k_src, *v_src;
    uint8_t *kpp, *vpp;
    size_t src_layer_stride;  // elements
    int L, n_kv, cap, P, hd;
};


// ------------------------------------------------------------------------------------------ device helpers
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldsm4_t(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldsm2_t(uint32_t (&r)[2], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "r"(addr));
}
__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ float ex2f(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
template <int ACT>
__device__ __forceinline__ float act_f(float x) {
    if (ACT == ACT_SILU) return __fdividef(x, 1.0f + __expf(-x));
    if (ACT == ACT_GELU_TANH) {
        const float k0 = 0.79788456080286535587989211986876f, k1 = 0.044715f;
        const float u = k0 * x * (1.0f + k1 * x * x);
        return __fdividef(x, 1.0f + __expf(-2.0f * u));
    }
    return x;
}
__device__ __forceinline__ float act_rt(float x, int act) {
    return act == ACT_SILU ? act_f<ACT_SILU>(x) : act == ACT_GELU_TANH ? act_f<ACT_GELU_TANH>(x) : x;
}
__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t *>(&v);
}

// what other CTAs wrote with ordinary stores (seen through the grid barrier) -> the bulk copies this thread issues next
__device__ __forceinline__ void fence_proxy_async_all() { asm volatile("fence.proxy.async;" ::: "memory"); }

// Distributed shared memory: the address of the same variable in another CTA of the cluster, a bulk copy into it that counts its
// bytes on an mbarrier there, an arrival on an mbarrier there.  (Plain stores of 16 bytes a lane followed by a release arrival,
// or st.async, took 3100 clocks for the 18 KB a CTA sends after q|k|v.)
__device__ __forceinline__ uint32_t map_rank(uint32_t addr, int rank) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void bulk_s2rank(uint32_t dst, uint32_t src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "r"(src), "r"(bytes), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void arrive_rank(uint32_t bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}

struct WEntry {  // what the weight feeder and the product issuer need to know about one GEMM phase
    const uint8_t *Wp;
    uint32_t n8_kb, kd_m;  // 8-column groups | 64-column blocks of K << 16, CTAs that share K | tokens << 16
};
static_assert(sizeof(LoopPhase) <= CL_DESC_BYTES && sizeof(LoopPhase) % 16 == 0, "descriptor slot");
static_assert(sizeof(WEntry) == 16 && CL_WTAB_OFF + CL_WTAB_MAX * 16 <= CL_HEADER, "feeder table");

// barrier of the computing warps (the feeder warp is not part of it)
__device__ __forceinline__ void cons_sync() { asm volatile("bar.sync 1, 256;" ::: "memory"); }

struct Smem {
    uint64_t *full, *empty, *a_full, *acc_full, *k_full, *v_full, *x_full, *xa_full, *rdy, *done;
    const WEntry *wtab;
    int n_wtab;
    volatile int *abort_flag;
    volatile unsigned *issued, *consumed;
    uint32_t *tmem_slot;
    float *row_m, *red, *red_max, *red_sum;
    uint8_t *ring, *arena;
};

// The carve-up of the dynamic shared memory; every phase function rebuilds it from the base (a few constant offsets) instead
// of taking it by reference, which would put it into local memory.
__device__ __forceinline__ Smem get_smem() {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    Smem sm;
    sm.full = reinterpret_cast<uint64_t *>(smem_raw);  // [CL_STAGES]
    sm.empty = sm.full + CL_STAGES;                    // [CL_STAGES]
    sm.a_full = sm.empty + CL_STAGES;                  // a product's A tile has landed
    sm.acc_full = sm.a_full + 1;                       // its accumulator is complete
    sm.k_full = sm.acc_full + 1;                       // attention: Q and K, V
    sm.v_full = sm.k_full + 1;
    sm.x_full = sm.v_full + 1;                         // the group's partial sums have arrived
    sm.xa_full = sm.x_full + 1;                        // attention: its rows have
    sm.rdy = sm.xa_full + 1;
    sm.done = sm.rdy + 1;
    sm.abort_flag = reinterpret_cast<volatile int *>(smem_raw + 224);
    sm.n_wtab = *reinterpret_cast<const int *>(smem_raw + 228);
    sm.issued = reinterpret_cast<volatile unsigned *>(smem_raw + 232);
    sm.consumed = reinterpret_cast<volatile unsigned *>(smem_raw + 236);
    sm.tmem_slot = reinterpret_cast<uint32_t *>(smem_raw + 240);
    sm.row_m = reinterpret_cast<float *>(smem_raw + 256);     // [32]
    sm.red = reinterpret_cast<float *>(smem_raw + 512);       // GEMM: [4][64] partial sums of squares; attention: [32][4] maxima, sums
    sm.red_max = sm.red;
    sm.red_sum = sm.red + 128;
    sm.wtab = reinterpret_cast<const WEntry *>(smem_raw + CL_WTAB_OFF);
    sm.ring = smem_raw + CL_RING_OFF;
    sm.arena = smem_raw + CL_ARENA_OFF;
    return sm;
}

// The computing warps' barrier parities, one bit each, carried from phase to phase.
constexpr unsigned PAR_K = 0, PAR_V = 1, PAR_RDY = 2, PAR_XA = 3, PAR_ACC = 4, PAR_X = 5;
__device__ __forceinline__ uint32_t par_bit(unsigned par, unsigned which) { return (par >> which) & 1u; }

// This CTA's part of a product: its group's 8-column groups [j0, j0 + w8) and the 64-column blocks [kb0, kb1) of K it multiplies.
struct GemmPart {
    int kr, j0, w8, kb0, kb1;
};
__device__ __forceinline__ GemmPart gemm_part(int N8, int kb, int kd) {
    const int sh = 31 - __clz(kd), G = gridDim.x >> sh, grp = blockIdx.x >> sh;
    GemmPart r;
    r.kr = blockIdx.x & (kd - 1);
    r.j0 = (int)((unsigned)(N8 * grp) / (unsigned)G);
    r.w8 = (int)((unsigned)(N8 * (grp + 1)) / (unsigned)G) - r.j0;
    r.kb0 = kb * r.kr >> sh;
    r.kb1 = kb * (r.kr + 1) >> sh;
    return r;
}

// The feeder: one thread walks the GEMM phases of every step in order and copies each weight chunk of this CTA into the next
// ring stage as soon as the products of its last content are done.  It runs ahead of the computation by the depth of the ring,
// across phase boundaries and grid barriers.
__device__ __noinline__ void feeder_loop(const LoopParams &lp) {
    const Smem sm = get_smem();
    const WaitCtx wc{sm.abort_flag, lp.status};
    unsigned issued = 0;
    bool ok = true;
    for (int step = 0; ok && step < lp.steps; ++step)
        for (int gi = 0; ok && gi < sm.n_wtab; ++gi) {
            const WEntry w = sm.wtab[gi];
            const int kb = (int)(w.n8_kb >> 16);
            const GemmPart gp = gemm_part((int)(w.n8_kb & 0xffffu), kb, (int)(w.kd_m & 0xffffu));
            if (gp.w8 <= 0) continue;
            const int kc = CL_STAGE_BYTES / (gp.w8 * 1024);
            const uint8_t *src = w.Wp + (size_t)gp.j0 * kb * 1024;
            for (int k0 = gp.kb0; k0 < gp.kb1; k0 += kc, ++issued) {
                const unsigned stage = issued % CL_STAGES;
                if (issued >= CL_STAGES && !mbar_wait_backoff(&sm.empty[stage], ((issued / CL_STAGES) - 1u) & 1u, wc, CL_DEV_TIMEOUT, 20)) {
                    ok = false;
                    break;
                }
                const uint32_t bytes = (uint32_t)(min(kc, gp.kb1 - k0) * gp.w8) * 1024u;
                mbar_expect_tx(&sm.full[stage], bytes);
                bulk_g2s(sm.ring + (size_t)stage * CL_STAGE_BYTES, src + (size_t)k0 * gp.w8 * 1024, bytes, &sm.full[stage]);
            }
        }
    *sm.issued = issued;
    mbar_arrive(sm.done);
}

// The issuer: one warp walks the same list and issues the products of a chunk as soon as it and the phase's A tile have landed.  The whole
// warp runs the loop and one elected lane issues: control that is the same for the warp lets the descriptors stay in uniform
// registers, which the instruction reads; from one lane of a diverged warp each product paid for moving them (pi0 6924 -> 6712 us).
// (A is copied after the grid barrier before the phase, so the accumulator of the phase before has been read by then).
__device__ __noinline__ void issuer_loop(const LoopParams &lp, uint32_t tmem) {
    const Smem sm = get_smem();
    const WaitCtx wc{sm.abort_flag, lp.status};
    unsigned cons = 0, a_cnt = 0;
    bool ok = true;
    const uint64_t a_desc0 = smem_desc_sw128(smem_u32(sm.ring), 16, 1024), b_desc0 = smem_desc_sw128(smem_u32(sm.arena), 16, 1024);
    for (int step = 0; ok && step < lp.steps; ++step)
        for (int gi = 0; ok && gi < sm.n_wtab; ++gi) {
            const WEntry &w = sm.wtab[gi];
            const uint32_t n8_kb = __shfl_sync(0xffffffffu, w.n8_kb, 0), kd_m = __shfl_sync(0xffffffffu, w.kd_m, 0);
            const GemmPart gp = gemm_part((int)(n8_kb & 0xffffu), (int)(n8_kb >> 16), (int)(kd_m & 0xffffu));
            const int M = (int)(kd_m >> 16);
            if (gp.w8 <= 0) continue;
            const uint32_t idesc = make_idesc(1, 1, 1, 0, 0, 128, (M + 15) & ~15);
            const uint32_t b_blk = (uint32_t)((M + 7) & ~7) * 8u;  // one 64-column block of A, in descriptor units of 16 bytes
            ok = warp_wait(sm.a_full, a_cnt & 1u, wc, CL_DEV_TIMEOUT);
            ++a_cnt;
            if (!ok) break;
            tc_fence_after();
            const int kc = CL_STAGE_BYTES / (gp.w8 * 1024);
            for (int k0 = gp.kb0; k0 < gp.kb1; k0 += kc, ++cons) {
                const unsigned stage = cons % CL_STAGES;
                ok = warp_wait(&sm.full[stage], (cons / CL_STAGES) & 1u, wc, CL_DEV_TIMEOUT);
                if (!ok) break;
                tc_fence_after();
                const int nk = min(kc, gp.kb1 - k0);
#pragma unroll 1  // unrolled, its code does not stay in the instruction cache beside the phases' (pi0 6,715 -> 6,497 us)
                for (int kk = 0; kk < nk; ++kk) {
                    const uint64_t a = a_desc0 + (uint64_t)(stage * (CL_STAGE_BYTES / 16) + (unsigned)(kk * gp.w8) * 64u);
                    const uint64_t b = b_desc0 + (uint64_t)((uint32_t)(k0 + kk - gp.kb0) * b_blk);
                    const uint32_t acc = k0 + kk > gp.kb0 ? 1u : 0u;
                    if (elect_one()) {
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            mma_f16(tmem, a + 2 * k, b + 2 * k, idesc, k ? 1u : acc);
                            if (gp.w8 > 16) mma_f16(tmem + 64u, a + 1024 + 2 * k, b + 2 * k, idesc, k ? 1u : acc);
                        }
                    }
                }
                if (elect_one()) tc_commit(&sm.empty[stage]);
            }
            if (ok && elect_one()) tc_commit(sm.acc_full);
        }
    if (elect_one()) {
        *sm.consumed = cons;
        mbar_arrive(sm.done);
    }
}

// Grid-wide barrier in two halves, so that what a phase can prepare without the phase before is done between them.
__device__ __forceinline__ void grid_arrive(const LoopParams &lp) {
    cons_sync();
    if (threadIdx.x == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(lp.counter) : "memory");
}
// thread 0 only: `target` counts arrivals since the launch
__device__ __forceinline__ bool grid_poll(const LoopParams &lp, unsigned target, const Smem &sm) {
    const long long t0 = clock64();
    for (uint32_t it = 0;; ++it) {
        unsigned v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(lp.counter) : "memory");
        if (v >= target) return true;
        if ((it & 255u) == 255u) {
            int st;
            asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(st) : "l"(lp.status) : "memory");
            if (st != 0 || *sm.abort_flag || clock64() - t0 > kWaitCycles) {
                atomicCAS(lp.status, 0, CL_DEV_TIMEOUT);
                *sm.abort_flag = 1;
                return false;
            }
        }
    }
}
__device__ __forceinline__ void grid_wait(const LoopParams &lp, unsigned target, const Smem &sm) {
    if (threadIdx.x == 0) grid_poll(lp, target, sm);
    cons_sync();
}

// ------------------------------------------------------------------------------------------------ GEMM
// One item of the epilogue: a row and the 8 columns of a group that this CTA owns (q|k|v: 4 columns and their rotation partners).
// What it needs besides the products is fetched before the products are waited for.
struct EpiPre {
    float4 a0, a1, b0, b1, c0, c1;  // residual, gate, next scale; q|k|v: cos, sin (a0, b0), bias (c); others: bias, x
};
__device__ __forceinline__ float4 ldg4(const float *p) { return __ldg(reinterpret_cast<const float4 *>(p)); }
__device__ __forceinline__ float4 ldcg4(const float *p) { return __ldcg(reinterpret_cast<const float4 *>(p)); }
// what does not depend on the phases before
__device__ __forceinline__ void epi_static(const LoopPhase &pg, EpiPre &e, int step, int n8, int row) {
    const int col = n8 * 8;
    if (pg.out_mode == OUT_RESID) {
        if (pg.colscale) {
            const float *s = pg.colscale + (size_t)step * pg.mod_stride + col, *n = pg.scale_next + (size_t)step * pg.mod_stride + col;
            e.b0 = ldg4(s); e.b1 = ldg4(s + 4);
            e.c0 = ldg4(n); e.c1 = ldg4(n + 4);
        }
    } else if (pg.out_mode == OUT_QKV) {
        const int per = pg.half >> 2, head = (int)((unsigned)n8 / (unsigned)per), k = (n8 - head * per) * 4;
        if (head < pg.n_q + pg.n_kvp) {
            e.a0 = ldg4(pg.rope + (size_t)row * pg.half + k);
            e.b0 = ldg4(pg.rope + (size_t)(pg.S + row) * pg.half + k);
        }
        if (pg.bias) {
            const float *bp = pg.bias + (size_t)step * pg.bias_step_stride + head * 2 * pg.half + k;
            e.c0 = ldg4(bp); e.c1 = ldg4(bp + pg.half);
        }
    } else if (pg.bias) {
        const float *bp = pg.bias + (size_t)step * pg.bias_step_stride + col;
        e.a0 = ldg4(bp); e.a1 = ldg4(bp + 4);
    }
}
// what they wrote
__device__ __forceinline__ void epi_dynamic(const LoopPhase &pg, EpiPre &e, int n8, int row) {
    const int col = n8 * 8, N = pg.N;
    if (pg.out_mode == OUT_RESID) {
        const float *h = pg.h + (size_t)row * N + col;
        e.a0 = ldcg4(h); e.a1 = ldcg4(h + 4);
    } else if (pg.out_mode == OUT_EULER && row >= pg.S - pg.chunk) {
        const float *x = pg.x + (size_t)(row - (pg.S - pg.chunk)) * N + col;
        e.b0 = ldcg4(x); e.b1 = ldcg4(x + 4);
    }
}
__device__ __forceinline__ float4 add4(float4 a, float4 b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }
__device__ __forceinline__ float4 mul4(float4 a, float4 b) { return make_float4(a.x * b.x, a.y * b.y, a.z * b.z, a.w * b.w); }
__device__ __forceinline__ float sq4(float4 a) { return fmaf(a.x, a.x, fmaf(a.y, a.y, fmaf(a.z, a.z, a.w * a.w))); }
__device__ __forceinline__ uint4 pack8(float4 a, float4 b) {
    return make_uint4(pack_bf16(a.x, a.y), pack_bf16(a.z, a.w), pack_bf16(b.x, b.y), pack_bf16(b.z, b.w));
}
__device__ __forceinline__ float4 act4(float4 v, int act) {
    return make_float4(act_rt(v.x, act), act_rt(v.y, act), act_rt(v.z, act), act_rt(v.w, act));
}
__device__ __forceinline__ float bf2_sq(uint32_t v) {
    const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(&v));
    return fmaf(f.x, f.x, f.y * f.y);
}
__device__ __forceinline__ float sq8(uint4 v) { return (bf2_sq(v.x) + bf2_sq(v.y)) + (bf2_sq(v.z) + bf2_sq(v.w)); }
// v, w: the products of the group's columns 0 .. 3 and 4 .. 7, RMS factor applied.  Returns the sum of squares of what the next norm reads.
__device__ __forceinline__ float epi_item(const LoopPhase &pg, const EpiPre &e, int n8, int row, float4 v, float4 w) {
    const int N = pg.N, col = n8 * 8;
    switch (pg.out_mode) {
    case OUT_RESID: {  // residual stream += projection; bf16 mirror; sums of squares of the mirror
        if (pg.colscale) {
            v = mul4(v, e.b0);
            w = mul4(w, e.b1);
        }
        const float4 h0 = add4(e.a0, v), h1 = add4(e.a1, w);
        float *hp = pg.h + (size_t)row * N + col;
        __stcg(reinterpret_cast<float4 *>(hp), h0);
        __stcg(reinterpret_cast<float4 *>(hp + 4), h1);
        uint4 *mp = reinterpret_cast<uint4 *>(pg.outp + sw_off(pg.out_rows8, row, col));
        if (pg.colscale) {  // the adaptive norm's (1 + scale) goes into the mirror, its sums of squares come from h itself
            __stcg(mp, pack8(add4(h0, mul4(h0, e.c0)), add4(h1, mul4(h1, e.c1))));
            return sq4(h0) + sq4(h1);
        }
        const uint4 pk = pack8(h0, h1);
        __stcg(mp, pk);
        return sq8(pk);
    }
    case OUT_GATED: {  // interleaved weight rows: even = gate, odd = up
        v = add4(v, e.a0);
        w = add4(w, e.a1);
        const int act = pg.act;
        __stcg(reinterpret_cast<uint2 *>(pg.outp + sw_off(pg.out_rows8, row, col >> 1)),
               make_uint2(pack_bf16(act_rt(v.x, act) * v.y, act_rt(v.z, act) * v.w), pack_bf16(act_rt(w.x, act) * w.y, act_rt(w.z, act) * w.w)));
        return 0.0f;
    }
    case OUT_QKV: {
        const int half = pg.half, per = half >> 2, head = (int)((unsigned)n8 / (unsigned)per), k = (n8 - head * per) * 4;
        v = add4(v, e.c0);
        w = add4(w, e.c1);
        const int n_q = pg.n_q, n_kvp = pg.n_kvp, S = pg.S;
        const uint32_t sq = (uint32_t)half * 4u + 16u;
        uint8_t *dst;
        float4 lo = v, hi = w;
        if (head < n_q + n_kvp) {
            const float4 c = e.a0, sn = e.b0;
            lo = make_float4(v.x * c.x - w.x * sn.x, v.y * c.y - w.y * sn.y, v.z * c.z - w.z * sn.z, v.w * c.w - w.w * sn.w);
            hi = make_float4(w.x * c.x + v.x * sn.x, w.y * c.y + v.y * sn.y, w.z * c.z + v.z * sn.z, w.w * c.w + v.w * sn.w);
            dst = head < n_q ? pg.qp + ((size_t)head * S + row) * sq : pg.kpp + ((size_t)(head - n_q) * pg.cap + pg.P + row) * sq;
        } else {
            dst = pg.vpp + ((size_t)(head - n_q - n_kvp) * pg.cap + pg.P + row) * sq;
        }
        __stcg(reinterpret_cast<uint2 *>(dst + k * 2), make_uint2(pack_bf16(lo.x, lo.y), pack_bf16(lo.z, lo.w)));
        __stcg(reinterpret_cast<uint2 *>(dst + (k + half) * 2), make_uint2(pack_bf16(hi.x, hi.y), pack_bf16(hi.z, hi.w)));
        return 0.0f;
    }
    case OUT_EULER: {
        const int t = row - (pg.S - pg.chunk);
        if (t >= 0) {
            const float dt = pg.dt;
            const float4 d4 = make_float4(dt, dt, dt, dt);
            float *xp = pg.x + (size_t)t * N + col;
            __stcg(reinterpret_cast<float4 *>(xp), add4(e.b0, mul4(d4, add4(v, e.a0))));
            __stcg(reinterpret_cast<float4 *>(xp + 4), add4(e.b1, mul4(d4, add4(w, e.a1))));
        }
        return 0.0f;
    }
    default: {
        v = act4(add4(v, e.a0), pg.act);
        w = act4(add4(w, e.a1), pg.act);
        const int orow = row + pg.row_off;
        const uint4 pk = pack8(v, w);
        __stcg(reinterpret_cast<uint4 *>(pg.outp + sw_off(pg.out_rows8, orow, col)), pk);
        if (pg.out_f32) {
            float *fp = pg.out_f32 + (size_t)orow * N + col;
            __stcg(reinterpret_cast<float4 *>(fp), v);
            __stcg(reinterpret_cast<float4 *>(fp + 4), w);
        }
        return sq8(pk);
    }
    }
}

// Floats per column of exchanged sums: the tokens, rounded up so that columns are an odd number of 16-byte chunks apart.
__host__ __device__ __forceinline__ int token_pitch(int M) { return ((M + 3) >> 2 | 1) * 4; }

// A group of kd CTAs computes a range of 8-column groups; this CTA multiplies its 1 / kd of K and sends every owner its part.
__device__ __noinline__ unsigned gemm_phase(const LoopPhase &pg, const LoopParams &lp, int step, unsigned par, unsigned target, uint32_t tmem) {
    const Smem sm = get_smem();
    const WaitCtx wc{sm.abort_flag, lp.status};
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int M = pg.M, K = pg.K, kd = pg.kd, kb = (K + 63) >> 6;
    const GemmPart gp = gemm_part(pg.N8, kb, kd);
    const int w8 = gp.w8;
    if (w8 <= 0) {
        grid_wait(lp, target, sm);
        return par;
    }
    const int sh = 31 - __clz(kd), kr = gp.kr, base_rank = (int)(blockIdx.x % CL_CLUSTER) - kr;
    const uint32_t blk_bytes = (uint32_t)((M + 7) & ~7) * 128u, a_bytes = (uint32_t)(gp.kb1 - gp.kb0) * blk_bytes;
    // arena: A (the longest of the group) | what the group sends, [source][owned column][token]; this CTA's own sums are staged over A
    // where they fit (A has been multiplied by then), else behind
    const int tp = token_pitch(M), row = tid & 63, cg = tid >> 6;
    const uint32_t recv_bytes = (uint32_t)((((w8 + kd - 1) >> sh) << sh) * 8 * tp) * 4u;  // kd parts of the most columns one CTA owns
    const uint32_t recv_off = (uint32_t)((kb + kd - 1) >> sh) * blk_bytes;
    const uint32_t stage_off = recv_bytes <= recv_off ? 0u : recv_off + recv_bytes;
    const int hw = warp & 3, th = warp >> 2;  // this warp's quarter of the TMEM lanes and half of the tokens
    // ---- before the barrier: everything that does not depend on the phase before
    const int own0 = w8 * kr >> sh, ownN = (w8 * (kr + 1) >> sh) - own0, n8_own = pg.n8_0 + gp.j0 + own0;
    EpiPre pre;
    pre.a0 = pre.a1 = pre.b0 = pre.b1 = pre.c0 = pre.c1 = make_float4(0.f, 0.f, 0.f, 0.f);
    const bool first = row < M && cg < ownN;
    if (first) epi_static(pg, pre, step, n8_own + cg, row);
    if (tid == 0) {
        mbar_expect_tx(sm.x_full, (uint32_t)(kd * ownN * 8 * tp) * 4u);
        if (grid_poll(lp, target, sm)) {
            fence_proxy_async_all();
            mbar_expect_tx(sm.a_full, a_bytes);
            bulk_g2s(sm.arena, pg.Ap + (size_t)gp.kb0 * blk_bytes, a_bytes, sm.a_full);
        }
    }
    cons_sync();
    // ---- after it
    if (first) epi_dynamic(pg, pre, n8_own + cg, row);
    const bool use_rms = pg.use_rms != 0;
    if (use_rms) {  // row sums of squares from the producer's partial sums, fixed order
        const int n = pg.ssq_n;
        const float *src = pg.ssq_in + row;
        float ss = 0.0f;
        for (int p0 = cg; p0 < n; p0 += 128) {
            float part[32];
#pragma unroll
            for (int j = 0; j < 32; ++j) part[j] = (row < M && p0 + 4 * j < n) ? __ldcg(src + (size_t)(p0 + 4 * j) * 64) : 0.0f;
#pragma unroll
            for (int j = 0; j < 32; ++j) ss += part[j];
        }
        sm.red[cg * 64 + row] = ss;
    }
    mbar_wait(sm.acc_full, par_bit(par, PAR_ACC), wc, CL_DEV_TIMEOUT);
    par ^= 1u << PAR_ACC;
    tc_fence_after();
    // ---- this CTA's K part into its staging area, [column][token]: a lane holds one column, 32 tokens
    float *stg = reinterpret_cast<float *>(sm.arena + stage_off);
    for (int n0 = hw * 32; n0 < w8 * 8; n0 += 128) {
        uint32_t v[32];
        tmem_ld32(tmem + (uint32_t)((n0 >> 7) * 64 + th * 32) + ((uint32_t)(hw * 32) << 16), v);
        tmem_ld_wait();
        const int n = n0 + lane;
        if (n < w8 * 8) {
            float4 *dst = reinterpret_cast<float4 *>(stg + (size_t)n * tp + th * 32);
#pragma unroll
            for (int e = 0; e < 8; ++e)
                if (th * 32 + e * 4 < M)
                    dst[e] = make_float4(__uint_as_float(v[4 * e]), __uint_as_float(v[4 * e + 1]), __uint_as_float(v[4 * e + 2]), __uint_as_float(v[4 * e + 3]));
        }
    }
    tc_fence_before();
    fence_proxy_async_smem();
    cons_sync();  // staged; and the partial sums of squares are in place
    if (lane == 0 && warp < kd) {  // warp w sends rank w of the group its columns
        const int b = w8 * warp >> sh, oN = (w8 * (warp + 1) >> sh) - b;
        const uint32_t bytes = (uint32_t)(oN * 8 * tp) * 4u;
        if (oN > 0)
            bulk_s2rank(map_rank(smem_u32(sm.arena + recv_off), base_rank + warp) + (uint32_t)kr * bytes, smem_u32(stg) + (uint32_t)(b * 8 * tp) * 4u,
                        bytes, map_rank(smem_u32(sm.x_full), base_rank + warp));
    }
    const float rms = use_rms ? rsqrtf(((sm.red[row] + sm.red[64 + row]) + (sm.red[128 + row] + sm.red[192 + row])) / (float)K + pg.eps) : 1.0f;
    mbar_wait_cluster(sm.x_full, par_bit(par, PAR_X), wc, CL_DEV_TIMEOUT);
    par ^= 1u << PAR_X;
    if (row < M) {
        const float *recv = reinterpret_cast<const float *>(sm.arena + recv_off) + row;
        const int ld = ownN * 8 * tp;
        for (int jl = cg; jl < ownN; jl += 4) {
            const int n8 = n8_own + jl;
            if (jl != cg) {
                epi_static(pg, pre, step, n8, row);
                epi_dynamic(pg, pre, n8, row);
            }
            const float *src = recv + (size_t)jl * 8 * tp;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f), w = v;
#pragma unroll 2
            for (int s = 0; s < kd; ++s, src += ld) {
                v.x += src[0]; v.y += src[tp]; v.z += src[2 * tp]; v.w += src[3 * tp];
                w.x += src[4 * tp]; w.y += src[5 * tp]; w.z += src[6 * tp]; w.w += src[7 * tp];
            }
            if (use_rms) {
                v.x *= rms; v.y *= rms; v.z *= rms; v.w *= rms;
                w.x *= rms; w.y *= rms; w.z *= rms; w.w *= rms;
            }
            const float ssq = epi_item(pg, pre, n8, row, v, w);
            if (pg.ssq_out) __stcg(pg.ssq_out + (size_t)n8 * 64 + row + pg.row_off, ssq);
        }
    }
    return par;
}

// ----------------------------------------------------------------------------------------------- EMBED
__device__ __noinline__ void embed_phase(const LoopPhase &p, const LoopParams &lp, int step, unsigned target) {
    const Smem sm = get_smem();
    grid_wait(lp, target, sm);
    float *xs = reinterpret_cast<float *>(sm.arena);
    const int A = p.A_dim, H = p.H, chunk = p.chunk, sd = p.sd;
    for (int i = threadIdx.x; i < chunk * A; i += CL_THREADS) xs[i] = __ldcg(p.x + i);
    float *ss = xs + chunk * A;
    for (int i = threadIdx.x; i < sd; i += CL_THREADS) ss[i] = lp.state[i];
    cons_sync();
    const int nrb = (chunk + CL_EMBED_ROWS - 1) / CL_EMBED_ROWS;
    const int gt = blockIdx.x * CL_THREADS + threadIdx.x, gn = gridDim.x * CL_THREADS;
    for (int item = gt; item < nrb * H; item += gn) {
        const int o = item % H, rb = item / H;
        uint4 wv[8];
        const uint4 *wr = reinterpret_cast<const uint4 *>(p.w_dense + (size_t)o * A);
#pragma unroll
        for (int k8 = 0; k8 < 8; ++k8)
            if (k8 * 8 < A) wv[k8] = __ldg(wr + k8);
        const float bias = p.bias ? p.bias[o] : 0.0f;
        const int rend = min(chunk, (rb + 1) * CL_EMBED_ROWS);
        for (int r = rb * CL_EMBED_ROWS; r < rend; ++r) {
            float acc = bias;
#pragma unroll
            for (int k8 = 0; k8 < 8; ++k8) {
                if (k8 * 8 >= A) break;
                const __nv_bfloat162 *h2 = reinterpret_cast<const __nv_bfloat162 *>(&wv[k8]);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float2 f = __bfloat1622float2(h2[e]);
                    acc = fmaf(f.x, xs[r * A + k8 * 8 + 2 * e], acc);
                    acc = fmaf(f.y, xs[r * A + k8 * 8 + 2 * e + 1], acc);
                }
            }
            if (!p.scale_next) {
                *reinterpret_cast<__nv_bfloat16 *>(p.outp + sw_off((chunk + 7) & ~7, r, o)) = __float2bfloat16(acc);
            } else {
                // pi0.5: the embedding IS the residual stream (rows = action tokens); mirror with the first norm's (1 + scale),
                // sums of squares per 32 columns (a warp holds 32 consecutive columns of one row block)
                __stcg(p.h + (size_t)r * H + o, acc);
                const float sn = p.scale_next[(size_t)step * p.mod_stride + o];
                *reinterpret_cast<__nv_bfloat16 *>(p.hbp + sw_off((p.S + 7) & ~7, r, o)) = __float2bfloat16(acc + acc * sn);
                float sq = acc * acc;
#pragma unroll
                for (int off = 16; off > 0; off >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, off);
                if ((threadIdx.x & 31) == 0) __stcg(p.ssq_out + (size_t)(o >> 5) * 64 + r, sq);
            }
        }
    }
    if (sd > 0)  // pi0: the state token is row 0 of the residual stream; a warp holds 32 consecutive columns
        for (int o = gt; o - (int)(threadIdx.x & 31) < H; o += gn) {
            float sq = 0.0f;
            if (o < H) {
                const __nv_bfloat16 *wr = p.w2 + (size_t)o * sd;
                float acc = p.b2 ? p.b2[o] : 0.0f;
                for (int k = 0; k < sd; ++k) acc = fmaf(__bfloat162float(wr[k]), ss[k], acc);
                __stcg(p.h + o, acc);
                const __nv_bfloat16 hb = __float2bfloat16(acc);
                *reinterpret_cast<__nv_bfloat16 *>(p.hbp + sw_off((p.S + 7) & ~7, 0, o)) = hb;
                sq = __bfloat162float(hb) * __bfloat162float(hb);
            }
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, off);
            if ((threadIdx.x & 31) == 0) __stcg(p.ssq_out + (size_t)(o >> 5) * 64, sq);
        }
}

// ------------------------------------------------------------------------------------------- ATTENTION
template <int HD>
__device__ __noinline__ unsigned att_phase(const LoopPhase &pg, const LoopParams &lp, unsigned par, unsigned target) {
    const Smem sm = get_smem();
    const WaitCtx wc{sm.abort_flag, lp.status};
    constexpr int SQ = HD * 2 + 16;   // bytes per staged row
    constexpr int NGV = HD / 64;      // 8-column groups of the output per warp
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int mt = warp & 1, kp = warp >> 1;
    const int mi = lane >> 3, lr = lane & 7, g = lane >> 2, q2 = (lane & 3) * 2;
    const int ks = pg.ks, n_rt = pg.n_rt, kv_len = pg.kv_len, R = pg.R, S = pg.S, P = pg.P, cap = pg.cap, mask_mode = pg.mask_mode;
    const int ad = pg.kd, rpo = 32 / ad;  // key ranges = CTAs per unit; query rows each of them merges
    const int grp = blockIdx.x / ad, ar = blockIdx.x - grp * ad, base_rank = (int)(blockIdx.x % CL_CLUSTER) - ar;
    const int gq = pg.g;
    const float scale_log2 = pg.scale_log2;
    constexpr int OP = HD + 8;        // floats per exchanged row: O, maximum and sum behind it
    uint8_t *Qs = sm.arena, *Ks = Qs + pg.k_off, *Vs = Ks + (size_t)ks * SQ, *Ps = sm.arena + pg.p_off, *recv = sm.arena + pg.recv_off;
    const int SP = (((ks + 15) & ~15) + 8) * 2;
    const int n_units = pg.n_kv * n_rt;
    int pad_lo = 0, pad_hi = 0;
    if (lp.pad) {
        pad_lo = lp.pad[0];
        pad_hi = lp.pad[1];
    }
    const int n_grp = gridDim.x / ad, k_begin = ar * pg.per, k_end = min(kv_len, k_begin + pg.per);
    // Before the barrier: the rows of the first key block that lie in the prefix (they do not change during the loop).
    const int nk0 = max(0, min(ks, k_end - k_begin)), n_prefix = max(0, min(nk0, P - k_begin));
    const int n_early_k = pg.early_k ? n_prefix : 0, n_early = pg.early_v ? n_prefix : 0;
    if (tid == 0) {
        const bool work = grp < n_units && nk0 > 0;
        const int kvh = grp / n_rt, row0 = (grp - kvh * n_rt) * 32;
        const uint32_t q_bytes = (uint32_t)min(32, R - row0) * SQ;
        const uint8_t *kp0 = pg.kpp + ((size_t)kvh * cap + k_begin) * SQ, *vp0 = pg.vpp + ((size_t)kvh * cap + k_begin) * SQ;
        if (work) {
            fence_proxy_async_all();
            mbar_expect_tx(sm.k_full, q_bytes + (uint32_t)nk0 * SQ);
            mbar_expect_tx(sm.v_full, (uint32_t)nk0 * SQ);
            if (n_early_k > 0) bulk_g2s(Ks, kp0, (uint32_t)n_early_k * SQ, sm.k_full);
            if (n_early > 0) bulk_g2s(Vs, vp0, (uint32_t)n_early * SQ, sm.v_full);
        }
        const bool open = grid_poll(lp, target, sm);
        if (grp < n_units) fence_proxy_async_all();  // also for the rows that a CTA without keys sends
        if (open && work) {
            bulk_g2s(Qs, pg.qp + ((size_t)kvh * gq * S + row0) * SQ, q_bytes, sm.k_full);
            if (n_early_k < nk0) bulk_g2s(Ks + (size_t)n_early_k * SQ, kp0 + (size_t)n_early_k * SQ, (uint32_t)(nk0 - n_early_k) * SQ, sm.k_full);
            if (n_early < nk0) bulk_g2s(Vs + (size_t)n_early * SQ, vp0 + (size_t)n_early * SQ, (uint32_t)(nk0 - n_early) * SQ, sm.v_full);
        }
    }
    cons_sync();
    for (int u = grp; u < n_units; u += n_grp) {  // several units per group only when ad == 1
        const int kvh = u / n_rt, rt = u - kvh * n_rt;
        const int row0 = rt * 32, nrows = min(32, R - row0);
        const int vrows = max(0, min(rpo, nrows - ar * rpo));  // rows this CTA merges
        if (u != grp) cons_sync();  // the unit before has been merged: the arena is free
        if (tid == 0) mbar_expect_tx(sm.xa_full, (uint32_t)(ad * rpo * OP) * 4u);
        float oacc[2][NGV][4], ms[2] = {-INFINITY, -INFINITY}, mo[2][2] = {{-INFINITY, -INFINITY}, {-INFINITY, -INFINITY}}, sum[2] = {0.0f, 0.0f};
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < NGV; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) oacc[i][j][e] = 0.0f;
        const int c0 = warp * (HD / 8);
        for (int key0 = k_begin; key0 < k_end; key0 += ks) {
            const int nkeys = min(ks, k_end - key0), ks16 = (nkeys + 15) & ~15;
            if (key0 != k_begin) cons_sync();  // the block before has been consumed
            if (tid == 0 && (u != grp || key0 != k_begin)) {
                fence_proxy_async_all();
                const uint32_t q_bytes = key0 == k_begin ? (uint32_t)nrows * SQ : 0u;
                mbar_expect_tx(sm.k_full, q_bytes + (uint32_t)nkeys * SQ);
                if (q_bytes) bulk_g2s(Qs, pg.qp + ((size_t)kvh * gq * S + row0) * SQ, q_bytes, sm.k_full);
                bulk_g2s(Ks, pg.kpp + ((size_t)kvh * cap + key0) * SQ, (uint32_t)nkeys * SQ, sm.k_full);
                mbar_expect_tx(sm.v_full, (uint32_t)nkeys * SQ);
                bulk_g2s(Vs, pg.vpp + ((size_t)kvh * cap + key0) * SQ, (uint32_t)nkeys * SQ, sm.v_full);
            }
            for (int i = tid; i < (ks16 - nkeys) * (HD / 8); i += CL_THREADS) {
                const int r = nkeys + i / (HD / 8), c = i % (HD / 8);
                *reinterpret_cast<uint4 *>(Vs + (size_t)r * SQ + c * 16) = make_uint4(0, 0, 0, 0);
            }
            mbar_wait(sm.k_full, par_bit(par, PAR_K), wc, CL_DEV_TIMEOUT);
            par ^= 1u << PAR_K;
            // ---- S = Q K^T for this warp's 16 rows and its share of the 8-key groups
            const int ng = ks16 >> 3, g0 = kp * ng / 4, g1 = (kp + 1) * ng / 4, n_g = g1 - g0;  // n_g <= 4
            float sacc[4][4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int e = 0; e < 4; ++e) sacc[i][e] = 0.0f;
            {
                const int qrow = min(mt * 16 + lr + (mi & 1) * 8, nrows - 1);
                const uint32_t q_addr = smem_u32(Qs) + (uint32_t)qrow * SQ + (uint32_t)(mi >> 1) * 16u;
                const uint32_t k_addr = smem_u32(Ks) + (uint32_t)(g0 * 8 + lr) * SQ + (uint32_t)mi * 16u;
#pragma unroll 2
                for (int kk = 0; kk < HD / 32; ++kk) {
                    uint32_t a0[4], a1[4];
                    ldsm4(a0, q_addr + kk * 64);
                    ldsm4(a1, q_addr + kk * 64 + 32);
#pragma unroll
                    for (int gi = 0; gi < 4; ++gi) {
                        if (gi >= n_g) break;
                        uint32_t b[4];
                        ldsm4(b, k_addr + (uint32_t)gi * 8u * SQ + kk * 64);
                        mma_bf16(sacc[gi], a0, b[0], b[1]);
                        mma_bf16(sacc[gi], a1, b[2], b[3]);
                    }
                }
            }
            // ---- mask, row maximum over the unit's keys
            const int rl[2] = {mt * 16 + g, mt * 16 + g + 8};
            int jmax[2];
#pragma unroll
            for (int hr = 0; hr < 2; ++hr) {
                const int tok = (row0 + rl[hr]) % S;
                const int n_suf = kv_len - P;
                int limit = n_suf;
                if (mask_mode == 2) limit = min(tok + 1, n_suf);
                else if (mask_mode == 1) limit = tok == 0 ? min(1, n_suf) : n_suf;
                jmax[hr] = min(P + limit, key0 + nkeys);
            }
            float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
            for (int gi = 0; gi < 4; ++gi) {
                if (gi >= n_g) break;
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int j = key0 + (g0 + gi) * 8 + q2 + (e & 1), hr = e >> 1;
                    const bool vis = j < jmax[hr] && !(j >= pad_lo && j < pad_hi);
                    sacc[gi][e] = vis ? sacc[gi][e] * scale_log2 : -INFINITY;
                    mx[hr] = fmaxf(mx[hr], sacc[gi][e]);
                }
            }
#pragma unroll
            for (int hr = 0; hr < 2; ++hr) {
                mx[hr] = fmaxf(mx[hr], __shfl_xor_sync(0xffffffffu, mx[hr], 1));
                mx[hr] = fmaxf(mx[hr], __shfl_xor_sync(0xffffffffu, mx[hr], 2));
                if ((lane & 3) == 0) sm.red_max[rl[hr] * 4 + kp] = mx[hr];
            }
            // K's last block has been read.  Where the rows of the group's CTAs land over it, they do so by bulk copies, which an arrival
            // alone does not order behind these loads (see stage_release in tc5.cuh)
            if (key0 + ks >= k_end && pg.recv_off == pg.k_off) fence_proxy_async_smem();
            cons_sync();  // the maxima are in place; Q (P may lie over it) and K have been read
            if (key0 + ks >= k_end && tid < ad) arrive_rank(map_rank(smem_u32(sm.rdy), base_rank + tid));
#pragma unroll
            for (int hr = 0; hr < 2; ++hr) {
                const float *rm = sm.red_max + rl[hr] * 4;
                const float m = fmaxf(ms[hr], fmaxf(fmaxf(rm[0], rm[1]), fmaxf(rm[2], rm[3])));
                mx[hr] = m == -INFINITY ? 0.0f : m;
                sum[hr] *= ex2f(ms[hr] - mx[hr]);  // 0 before the first block
                ms[hr] = m;
                if (kp == 0 && (lane & 3) == 0) sm.row_m[rl[hr]] = m;
            }
#pragma unroll
            for (int gi = 0; gi < 4; ++gi) {
                if (gi >= n_g) break;
                float pv[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    pv[e] = ex2f(sacc[gi][e] - mx[e >> 1]);
                    sum[e >> 1] += pv[e];
                }
                const int col = (g0 + gi) * 8 + q2;
                *reinterpret_cast<uint32_t *>(Ps + (size_t)rl[0] * SP + col * 2) = pack_bf16(pv[0], pv[1]);
                *reinterpret_cast<uint32_t *>(Ps + (size_t)rl[1] * SP + col * 2) = pack_bf16(pv[2], pv[3]);
            }
#pragma unroll
            for (int hr = 0; hr < 2; ++hr) {
                float s = sum[hr];
                s += __shfl_xor_sync(0xffffffffu, s, 1);
                s += __shfl_xor_sync(0xffffffffu, s, 2);
                if ((lane & 3) == 0) sm.red_sum[rl[hr] * 4 + kp] = s;
            }
            mbar_wait(sm.v_full, par_bit(par, PAR_V), wc, CL_DEV_TIMEOUT);
            par ^= 1u << PAR_V;
            cons_sync();
            // ---- O = P V: this warp's HD / 8 output columns, all 32 rows
            if (pg.per > ks) {  // several key blocks: earlier sums follow the running maximum
#pragma unroll
                for (int m2 = 0; m2 < 2; ++m2)
#pragma unroll
                    for (int hr = 0; hr < 2; ++hr) {
                        const float m = sm.row_m[m2 * 16 + g + hr * 8], f = ex2f(mo[m2][hr] - (m == -INFINITY ? 0.0f : m));
                        mo[m2][hr] = m;
#pragma unroll
                        for (int j = 0; j < NGV; ++j) {
                            oacc[m2][j][2 * hr] *= f;
                            oacc[m2][j][2 * hr + 1] *= f;
                        }
                    }
            }
            {
                const uint32_t p_addr = smem_u32(Ps) + (uint32_t)(lr + (mi & 1) * 8) * SP + (uint32_t)(mi >> 1) * 16u;
                const uint32_t v_addr = smem_u32(Vs) + (uint32_t)(lr + (mi & 1) * 8) * SQ + (uint32_t)(c0 + (NGV > 1 ? (mi >> 1) * 8 : 0)) * 2u;
                for (int kk = 0; kk < (ks16 >> 4); ++kk) {
                    uint32_t a[2][4];
                    ldsm4(a[0], p_addr + kk * 32);
                    ldsm4(a[1], p_addr + 16 * SP + kk * 32);
                    if (NGV == 1) {
                        uint32_t b[2];
                        ldsm2_t(b, v_addr + (uint32_t)kk * 16u * SQ);
                        mma_bf16(oacc[0][0], a[0], b[0], b[1]);
                        mma_bf16(oacc[1][0], a[1], b[0], b[1]);
                    } else {
#pragma unroll
                        for (int gp = 0; gp < NGV / 2; ++gp) {
                            uint32_t b[4];
                            ldsm4_t(b, v_addr + (uint32_t)kk * 16u * SQ + gp * 32);
                            mma_bf16(oacc[0][2 * gp], a[0], b[0], b[1]);
                            mma_bf16(oacc[1][2 * gp], a[1], b[0], b[1]);
                            mma_bf16(oacc[0][2 * gp + 1], a[0], b[2], b[3]);
                            mma_bf16(oacc[1][2 * gp + 1], a[1], b[2], b[3]);
                        }
                    }
                }
            }
        }
        if (k_begin >= k_end) {  // no keys in this CTA's range: it contributes nothing, but its peers count on its arrival
            if (tid < ad) arrive_rank(map_rank(smem_u32(sm.rdy), base_rank + tid));
            if (tid < 128) sm.red_sum[tid] = 0.0f;
            if (tid < 32) sm.row_m[tid] = -INFINITY;
            cons_sync();
        }
        // ---- un-normalised O rows, maximum and row sum: staged over V (read by everyone), then one copy per CTA that merges rows
        cons_sync();
        float *stg = reinterpret_cast<float *>(sm.arena + pg.stage_off);
#pragma unroll
        for (int m2 = 0; m2 < 2; ++m2)
#pragma unroll
            for (int hr = 0; hr < 2; ++hr) {
                float *rp = stg + (size_t)(m2 * 16 + g + hr * 8) * OP + c0 + q2;
#pragma unroll
                for (int j = 0; j < NGV; ++j) *reinterpret_cast<float2 *>(rp + j * 8) = make_float2(oacc[m2][j][2 * hr], oacc[m2][j][2 * hr + 1]);
            }
        if (tid < 32) {
            const float *rs = sm.red_sum + tid * 4;
            *reinterpret_cast<float2 *>(stg + (size_t)tid * OP + HD) = make_float2(sm.row_m[tid], ((rs[0] + rs[1]) + rs[2]) + rs[3]);
        }
        fence_proxy_async_smem();
        cons_sync();
        const uint32_t xblk = (uint32_t)(rpo * OP) * 4u;
        if (lane == 0 && warp < ad && mbar_wait_cluster(sm.rdy, par_bit(par, PAR_RDY), wc, CL_DEV_TIMEOUT))  // the group has read its K blocks, where the rows may land
            bulk_s2rank(map_rank(smem_u32(recv), base_rank + warp) + (uint32_t)ar * xblk, smem_u32(stg) + (uint32_t)warp * xblk, xblk,
                        map_rank(smem_u32(sm.xa_full), base_rank + warp));
        par ^= 1u << PAR_RDY;
        // ---- merge
        mbar_wait_cluster(sm.xa_full, par_bit(par, PAR_XA), wc, CL_DEV_TIMEOUT);
        par ^= 1u << PAR_XA;
        if (vrows <= 0) continue;
        for (int it = tid; it < vrows * (HD / 4); it += CL_THREADS) {
            const int c4 = it % (HD / 4), lrow = it / (HD / 4);
            const float *rv = reinterpret_cast<const float *>(recv) + (size_t)lrow * OP;
            float mmax = -INFINITY, L = 0.0f;
            for (int s = 0; s < ad; ++s) mmax = fmaxf(mmax, rv[(size_t)s * rpo * OP + HD]);
            float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
            for (int s = 0; s < ad; ++s) {
                const float2 m = *reinterpret_cast<const float2 *>(rv + (size_t)s * rpo * OP + HD);
                if (m.x == -INFINITY) continue;
                const float4 v = *reinterpret_cast<const float4 *>(rv + (size_t)s * rpo * OP + c4 * 4);
                const float w = ex2f(m.x - mmax);
                o.x = fmaf(w, v.x, o.x); o.y = fmaf(w, v.y, o.y); o.z = fmaf(w, v.z, o.z); o.w = fmaf(w, v.w, o.w);
                L = fmaf(w, m.y, L);
            }
            const float inv = L > 0.0f ? 1.0f / L : 0.0f;
            const int r = row0 + ar * rpo + lrow, head_l = r / S, tok = r - head_l * S, col = (kvh * gq + head_l) * HD + c4 * 4;
            __stcg(reinterpret_cast<uint2 *>(pg.outp + sw_off(pg.out_rows8, tok, col)),
                   make_uint2(pack_bf16(o.x * inv, o.y * inv), pack_bf16(o.z * inv, o.w * inv)));
        }
    }
    return par;
}

// prefix rows of the engine's K / V pages (observation 0) -> the padded pages the attention tiles are copied from
__device__ __noinline__ void pages_prologue(const LoopParams &lp) {
    const int c16 = lp.hd / 8;  // 16-byte chunks per row
    const size_t per_layer = (size_t)lp.n_kv * lp.P * c16, total = per_layer * lp.L;
    const uint32_t sq = (uint32_t)lp.hd * 2u + 16u;
    for (size_t i = (size_t)blockIdx.x * CL_THREADS + threadIdx.x; i < total; i += (size_t)gridDim.x * CL_THREADS) {
        const int l = (int)(i / per_layer);
        size_t r = i - (size_t)l * per_layer;
        const int c = (int)(r % c16);
        r /= c16;
        const int tok = (int)(r % lp.P), kvh = (int)(r / lp.P);
        const size_t so = (size_t)l * lp.src_layer_stride + ((size_t)kvh * lp.cap + tok) * lp.hd + (size_t)c * 8;
        const size_t dof = ((size_t)l * lp.n_kv * lp.cap + (size_t)kvh * lp.cap + tok) * sq + (size_t)c * 16;
        __stcg(reinterpret_cast<uint4 *>(lp.kpp + dof), __ldg(reinterpret_cast<const uint4 *>(lp.k_src + so)));
        __stcg(reinterpret_cast<uint4 *>(lp.vpp + dof), __ldg(reinterpret_cast<const uint4 *>(lp.v_src + so)));
    }
}

// ---------------------------------------------------------------------------------------------- kernel
// One instantiation per head_dim: the kernel's code has to stay small (each phase runs its code once every few microseconds
// and what does not fit the SM's instruction cache is fetched from L2 every time).
template <int HD>
__global__ void __launch_bounds__(CL_BLOCK, 1) chunk_loop_kernel(const __grid_constant__ LoopParams lp) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    if (threadIdx.x == 0) *reinterpret_cast<int *>(smem_raw + 228) = lp.n_wtab;
    __syncthreads();
    const Smem sm = get_smem();
    WEntry *wtab = reinterpret_cast<WEntry *>(smem_raw + CL_WTAB_OFF);
    if (threadIdx.x == 0) {
        for (int i = 0; i < CL_STAGES; ++i) {
            mbar_init(&sm.full[i], 1);
            mbar_init(&sm.empty[i], 1);
        }
        mbar_init(sm.a_full, 1);
        mbar_init(sm.acc_full, 1);
        mbar_init(sm.k_full, 1);
        mbar_init(sm.v_full, 1);
        mbar_init(sm.x_full, 1);
        mbar_init(sm.xa_full, 1);
        mbar_init(sm.rdy, lp.att_cta);
        mbar_init(sm.done, 2);
        *sm.abort_flag = smem_u32(smem_raw) & 1023u ? 1 : 0;  // the swizzled tiles count on it; an unaligned base is reported like a time-out
        if (*sm.abort_flag) atomicCAS(lp.status, 0, CL_DEV_TIMEOUT);
        *sm.issued = 0;
        *sm.consumed = 0;
        fence_barrier_init();
    }
    if (threadIdx.x < 32) {
        tmem_alloc(sm.tmem_slot, CL_TMEM_COLS);
        tmem_relinquish();
    }
    for (int i = threadIdx.x; i < lp.n_wtab * 4; i += CL_BLOCK)
        reinterpret_cast<uint32_t *>(wtab)[i] = reinterpret_cast<const uint32_t *>(lp.wtab)[i];
    // descriptor of phase 0 into slot 0; from then on every phase fetches its successor's while it works
    for (int i = threadIdx.x; i < (int)(sizeof(LoopPhase) / 4); i += CL_BLOCK)
        reinterpret_cast<uint32_t *>(smem_raw + CL_DESC_OFF)[i] = reinterpret_cast<const uint32_t *>(lp.phases)[i];
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();  // every CTA's barriers exist before another CTA of the cluster signals them
    tc_fence_after();
    const uint32_t tmem = *sm.tmem_slot;
    if (threadIdx.x >= CL_THREADS) {  // the feeder (lane 0) and the issuer warp; they take no part in any barrier of the computing ones
        if (threadIdx.x == CL_THREADS) feeder_loop(lp);
        if (threadIdx.x >= CL_THREADS + 32) issuer_loop(lp, tmem);
        __syncwarp();
    } else {
        const WaitCtx wc{sm.abort_flag, lp.status};
        unsigned target = gridDim.x, seq = 0, par = 0;
        pages_prologue(lp);
        grid_arrive(lp);
        bool ok = true;
        for (int step = 0; ok && step < lp.steps; ++step) {
            for (int ph = 0; ok && ph < lp.n_phases; ++ph, ++seq) {
                const LoopPhase &p = *reinterpret_cast<const LoopPhase *>(smem_raw + CL_DESC_OFF + (seq & 1u) * CL_DESC_BYTES);
                if (threadIdx.x < (int)(sizeof(LoopPhase) / 16)) {  // the next phase's descriptor: asynchronous 16-byte copies
                    const int nx = ph + 1 == lp.n_phases ? 0 : ph + 1;
                    const uint32_t dst = smem_u32(smem_raw + CL_DESC_OFF + ((seq + 1) & 1u) * CL_DESC_BYTES) + threadIdx.x * 16u;
                    const uint8_t *src = reinterpret_cast<const uint8_t *>(lp.phases + nx) + threadIdx.x * 16u;
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
                    asm volatile("cp.async.commit_group;" ::: "memory");
                }
                switch (p.type) {  // every phase waits for `target` arrivals once it has prepared what it can
                case PH_GEMM: par = gemm_phase(p, lp, step, par, target, tmem); break;
                case PH_EMBED: embed_phase(p, lp, step, target); break;
                default: par = att_phase<HD>(p, lp, par, target); break;
                }
                asm volatile("cp.async.wait_all;" ::: "memory");
                target += gridDim.x;
                grid_arrive(lp);  // (and every warp's part of the next descriptor is in place)
                ok = *sm.abort_flag == 0;
                if (lp.trace && blockIdx.x == 0 && threadIdx.x == 0) {
                    unsigned long long t;
                    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
                    lp.trace[seq] = t;
                }
            }
        }
        grid_wait(lp, target, sm);
        // Weight chunks still on their way must land before the CTA gives its shared memory back (only after a failure are
        // there any: the feeder stops with the computation).
        if (threadIdx.x == 0 && mbar_wait(sm.done, 0u, wc, CL_DEV_TIMEOUT))
            for (unsigned i = *sm.consumed, n = *sm.issued; i < n; ++i) mbar_wait(&sm.full[i % CL_STAGES], (i / CL_STAGES) & 1u, wc, CL_DEV_TIMEOUT);
        if (*sm.abort_flag) __nanosleep(1000000);  // after a failure: products in flight, peers that may still be writing
        tc_fence_before();
        __syncwarp();
    }
    __syncthreads();
    cluster_sync_all();  // no CTA leaves while another of its cluster may still write into its shared memory
    if (threadIdx.x < 32) {
        tc_fence_after();
        tmem_dealloc(tmem, CL_TMEM_COLS);
    }
}

// Columns n8_0 * 8 .. (n8_0 + N8) * 8 and K range [k0, k0 + K) of a dense [N][ld] bf16 matrix -> weight image for G CTA groups: [group]
// [64-column block][8-column group][8 rows x 128 bytes, 16-byte chunks permuted by the row]; zeros beyond K.
// half > 0 (q|k|v): a group's 8 columns are dims 4 j .. 4 j + 3 of a head and their rotation partners, `half` further on.
__global__ void weight_image_kernel(const __nv_bfloat16 *__restrict__ src, uint4 *__restrict__ dst, int n8_0, int N8, int k0, int K, int ld, int G,
                                    int half) {
    const int kb = (K + 63) >> 6;
    const size_t total = (size_t)N8 * kb * 64;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const int c16 = (int)(i & 7), c = (int)(i >> 3) & 7;
        size_t r = i >> 6;
        const int b = (int)(r % kb), n8 = (int)(r / kb);
        const int grp = (int)((((long long)n8 + 1) * G - 1) / N8), j0 = (int)((long long)N8 * grp / G), w8 = (int)((long long)N8 * (grp + 1) / G) - j0;
        int row = (n8_0 + n8) * 8 + c;
        if (half > 0) {
            const int per = half >> 2, head = (n8_0 + n8) / per, jj = n8_0 + n8 - head * per;
            row = head * 2 * half + 4 * jj + (c & 3) + (c >= 4 ? half : 0);
        }
        const int k = b * 64 + c16 * 8;
        const uint4 v = k < K ? *reinterpret_cast<const uint4 *>(src + (size_t)row * ld + k0 + k) : make_uint4(0u, 0u, 0u, 0u);
        dst[((size_t)j0 * kb + (size_t)b * w8 + (n8 - j0)) * 64 + c * 8 + (c16 ^ c)] = v;
    }
}


// pi0.5: the adaptive norm's shift passes through the projection as a per-column constant,
// out[s][n] = (add ? add[n] : 0) + sum_k W[n][k] shift_s[k]   (shift_s = shift + s * stride; one warp per (s, n))
__global__ void shift_bias_kernel(const __nv_bfloat16 *__restrict__ W, const float *__restrict__ shift, size_t stride, const float *__restrict__ add,
                                  float *__restrict__ out, int steps, int N, int K) {
    const size_t warp = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (warp >= (size_t)steps * N) return;
    const int s = (int)(warp / N), n = (int)(warp % N);
    const __nv_bfloat16 *wr = W + (size_t)n * K;
    const float *sh = shift + (size_t)s * stride;
    float acc = 0.0f;
    for (int k = lane; k < K; k += 32) acc = fmaf(__bfloat162float(wr[k]), sh[k], acc);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
    if (lane == 0) out[warp] = acc + (add ? add[n] : 0.0f);
}

}  // namespace

// ------------------------------------------------------------------------------------------------ host
struct ChunkLoop {
    const void *kernel = nullptr;
    DevBuf phases, wtab, counter, trace;
    DevBuf hbp, ap, m1p, attp, gp, qp, kpp, vpp;  // padded activations and pages
    DevBuf ssq0, ssq;                              // [H / 8][64] partial sums of squares of the residual mirror: embedding's, residual updates'
    std::vector<DevBuf> cvec;                      // pi0.5: the shift terms of every norm, [steps][N] each
    std::vector<DevBuf> wp;                        // weight images
    int n_phases = 0, steps = 0, n_cta = 0;
    LoopParams lp{};
};

namespace {

// one CTA per SM in clusters, all co-resident (the kernel's CTAs wait for one another)
void loop_launch_config(cudaLaunchConfig_t *cfg, cudaLaunchAttribute *attr, int n_cta, cudaStream_t stream) {
    cfg->gridDim = dim3(n_cta);
    cfg->blockDim = dim3(CL_BLOCK);
    cfg->dynamicSmemBytes = CL_SMEM;
    cfg->stream = stream;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = CL_CLUSTER;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeCooperative;
    attr[1].val.cooperative = 1;
    cfg->attrs = attr;
    cfg->numAttrs = 2;
}

int round_up(int v, int m) { return (v + m - 1) / m * m; }
size_t image_bytes(int rows, int K) { return (size_t)round_up(rows, 8) * 128 * ((K + 63) / 64); }

// kd parts of the most columns one CTA owns
size_t exchange_bytes(int M, int w8, int kd) { return (size_t)round_up(w8, kd) * 8 * token_pitch(M) * 4; }

// Arena bytes of a product of kb 64-column blocks shared by kd CTAs: A of one CTA + what the group sends it + its own sums (over A
// where they fit there).
size_t gemm_arena(int M, int w8, int kb, int kd) {
    const size_t a = (size_t)((kb + kd - 1) / kd) * round_up(M, 8) * 128, x = exchange_bytes(M, w8, kd);
    return a + x * (x <= a ? 1 : 2);
}

// End of the arena range in which its own sums are staged (gemm_phase).
size_t staged_end(int M, int w8, int kb, int kd) {
    const size_t a = (size_t)((kb + kd - 1) / kd) * round_up(M, 8) * 128, x = exchange_bytes(M, w8, kd);
    return x <= a ? x : a + 2 * x;
}

// How a product runs: kd CTAs share K; `cols` phases each take a part of the columns, `ks` phases each a part of K (only where the
// output is added to).
struct GemmPlan {
    int kd, cols, ks;
};

// CTAs that share a product's K: least (A in at ~50 B/ns and SM, partial sums out at ~20 B/ns, products at ~48 clocks per 128 x 64 x
// 16).  More CTAs per group read less of A and send more partial sums.  0: no number of them fits.  kb_min: blocks of the shortest part.
int choose_kd(int M, int N8, int kb, int kb_min, int n_cta, double *cost_out) {
    int best = 0;
    for (int kd = 1; kd <= CL_CLUSTER && kd <= kb_min; kd *= 2) {
        const int G = n_cta / kd, w8 = (N8 + G - 1) / G, kbc = (kb + kd - 1) / kd;
        // (a shorter part may have to stage its sums behind A where the longest does not)
        if (w8 > CL_GROUP_N8 || std::max(gemm_arena(M, w8, kb, kd), gemm_arena(M, w8, kb_min, kd)) > (size_t)CL_ARENA) continue;
        const double a = (double)M * kbc * 128 / 50.0, x = (double)M * w8 * 32 * (kd - 1) / kd / 20.0;
        const double cost = a + x + kbc * 4 * (w8 > 16 ? 2 : 1) * 48 / 1.9;
        if (!best || cost < *cost_out) {
            best = kd;
            *cost_out = cost;
        }
    }
    return best;
}

// The fewest phases in which the product fits (each costs a round of its own: barrier, A, exchange), then the cheapest way to cut it.
// kd == 0: none.
GemmPlan plan_gemm(int M, int N8, int K, bool adds, int n_cta) {
    const int kb = (K + 63) / 64;
    GemmPlan best{0, 1, 1};
    if (N8 > 65535 || kb > 65535) return best;
    double best_cost = 0;
    for (int parts = 1; parts < CL_LAYER_PRODUCTS && !best.kd; ++parts)
        for (int ks = 1; ks <= parts; ++ks) {
            const int cols = parts / ks;
            if (cols * ks != parts || (ks > 1 && !adds) || ks > kb || cols > N8) continue;
            double cost = 0;
            const int kd = choose_kd(M, (N8 + cols - 1) / cols, (kb + ks - 1) / ks, kb / ks, n_cta, &cost);
            if (kd && (!best.kd || cost < best_cost)) {
                best = {kd, cols, ks};
                best_cost = cost;
            }
        }
    return best;
}

// What the kernel does for an expert of these sizes with n_cta CTAs resident.
struct LoopPlan {
    GemmPlan qkv, gu, o, dn, mlp, head;  // qkv: of self layers, cross layers have fewer columns; mlp: the two products of the suffix embedding
    int att_cta, n_phases, n_wtab;  // CTAs per attention unit; phases and products per Euler step
};

bool make_plan(const ChunkLoopDesc &d, int n_cta, LoopPlan *out) {
    const int hd = d.hd, qf = d.n_q * hd, H = d.H, S = d.S;
    if (n_cta < CL_CLUSTER || n_cta % CL_CLUSTER || d.model < 0 || d.model > 2 || (d.model == 2 && H % 32)) return false;
    if (hd != 64 && hd != 128 && hd != 256) return false;
    if (S > 64 || H % 16 || d.A % 16 || qf % 16 || d.I % 16) return false;
    if ((size_t)(d.chunk * d.A + 64) * 4 > (size_t)CL_ARENA || d.A > 64) return false;
    LoopPlan &p = *out;
    p.qkv = plan_gemm(S, (d.n_q + 2 * d.n_kv) * hd / 8, H, false, n_cta);
    p.gu = plan_gemm(S, 2 * d.I / 8, H, false, n_cta);
    p.o = plan_gemm(S, H / 8, qf, true, n_cta);
    p.dn = plan_gemm(S, H / 8, d.I, true, n_cta);
    p.mlp = plan_gemm(d.chunk, H / 8, H, false, n_cta);
    p.head = plan_gemm(S, d.A / 8, H, false, n_cta);
    for (const GemmPlan *g : {&p.qkv, &p.gu, &p.o, &p.dn, &p.mlp, &p.head})
        if (!g->kd) return false;
    // attention units of 32 query rows: as many CTAs each as there are for one round (they split the keys)
    const int units = d.n_kv * ((d.n_q / d.n_kv * S + 31) / 32);
    p.att_cta = 1;
    while (p.att_cta < CL_CLUSTER && units <= n_cta / (2 * p.att_cta)) p.att_cta *= 2;
    // With nine phases a layer a launch per operator is as fast (pi0's depth and width, ms per chunk here and there: MLP width 4096
    // 6.4 and 10.7, 8192 9.2 and 11.4, 12288 11.2 and 13.7, 14336 in eight phases 11.6 and 12.7, 16384 in nine 13.4 and 13.2).
    const int layer = p.qkv.cols + p.gu.cols + p.o.cols * p.o.ks + p.dn.cols * p.dn.ks;
    p.n_wtab = d.L * layer + p.head.cols + (d.model == 2 ? 0 : 2 * p.mlp.cols);
    p.n_phases = p.n_wtab + d.L + 1;
    return layer <= CL_LAYER_PRODUCTS && p.n_wtab <= CL_WTAB_MAX;
}

}  // namespace

int chunk_loop_plan_phases(const ChunkLoopDesc &d, int n_cta) {
    LoopPlan plan;
    return make_plan(d, n_cta, &plan) ? plan.n_phases : 0;
}

int chunk_loop_create(const ChunkLoopDesc &d, ChunkLoop **out) {
    *out = nullptr;
    const int n_sm = sm_count();
    if (n_sm <= 0) return VLAB200_ERR_CUDA;
    const int hd = d.hd, half = hd / 2, qf = d.n_q * hd, H = d.H, S = d.S;
    if ((hd != 64 && hd != 128 && hd != 256) || (d.model == 2 && !d.mods)) return VLAB200_ERR_UNSUPPORTED;
    const void *kernel = hd == 64    ? reinterpret_cast<const void *>(chunk_loop_kernel<64>)
                         : hd == 128 ? reinterpret_cast<const void *>(chunk_loop_kernel<128>)
                                     : reinterpret_cast<const void *>(chunk_loop_kernel<256>);
    if (ensure_dyn_smem(kernel, CL_SMEM)) return VLAB200_ERR_CUDA;
    int coop = 0, dev = 0, n_clusters = 0;
    VB_CUDA(cudaGetDevice(&dev));
    VB_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
    {
        cudaLaunchConfig_t cfg{};
        cudaLaunchAttribute attr[2];
        loop_launch_config(&cfg, attr, n_sm / CL_CLUSTER * CL_CLUSTER, nullptr);
        VB_CUDA(cudaOccupancyMaxActiveClusters(&n_clusters, kernel, &cfg));
    }
    n_clusters = std::min(n_clusters, n_sm / CL_CLUSTER);
    if (n_clusters < 1 || !coop) return VLAB200_ERR_UNSUPPORTED;
    const int n_cta = n_clusters * CL_CLUSTER;
    LoopPlan plan;
    if (!make_plan(d, n_cta, &plan)) return VLAB200_ERR_UNSUPPORTED;
    const int g = d.n_q / d.n_kv, R = g * S, n_rt = (R + 31) / 32, att_cta = plan.att_cta;

    ChunkLoop *cl = new (std::nothrow) ChunkLoop();
    if (!cl) return VLAB200_ERR_CUDA;
    int rc = VLAB200_OK;
    auto fail = [&](int code) {
        delete cl;
        return code;
    };
    const uint32_t sq = (uint32_t)hd * 2u + 16u;
    const size_t page_layer = (size_t)d.n_kv * d.cap * sq;
    struct {
        DevBuf *b;
        size_t bytes;
    } const zeroed[] = {{&cl->hbp, image_bytes(S, H)},     {&cl->ap, image_bytes(d.chunk, H)}, {&cl->m1p, image_bytes(d.chunk, H)},
                        {&cl->attp, image_bytes(S, qf)},   {&cl->gp, image_bytes(S, d.I)},     {&cl->qp, (size_t)d.n_q * S * sq},
                        {&cl->kpp, page_layer * d.L},            {&cl->vpp, page_layer * d.L},             {&cl->ssq0, (size_t)(H / 8) * 64 * 4},
                        {&cl->ssq, (size_t)(H / 8) * 64 * 4}};
    for (const auto &z : zeroed) {
        if ((rc = z.b->alloc(z.bytes))) return fail(rc);
        if (cudaMemset(z.b->p, 0, z.bytes) != cudaSuccess) return fail(VLAB200_ERR_CUDA);
    }
    cl->wp.reserve((size_t)plan.n_wtab);
    auto no_room = [&] {  // for a second copy of the weights: not an error of the call
        cudaGetLastError();
        return fail(VLAB200_ERR_UNSUPPORTED);
    };
    std::vector<LoopPhase> ph;
    // One product: p says what goes in (Ap, M) and out; its weights as tcgen05 reads them, in the order of the CTA groups.
    auto push_gemm = [&](LoopPhase p, const void *w_dense, int N, int K, const GemmPlan &gp) -> int {
        const int N8 = N / 8, kb = (K + 63) / 64;
        p.type = PH_GEMM; p.N = N; p.kd = gp.kd; p.half = p.out_mode == OUT_QKV ? half : 0; p.eps = d.rms_eps; p.S = S; p.chunk = d.chunk;
        const uint8_t *a_image = p.Ap;
        for (int ci = 0; ci < gp.cols; ++ci)
            for (int ki = 0; ki < gp.ks; ++ki) {
                const int kb0 = kb * ki / gp.ks, kb1 = kb * (ki + 1) / gp.ks;
                p.n8_0 = N8 * ci / gp.cols; p.N8 = N8 * (ci + 1) / gp.cols - p.n8_0;
                p.K = std::min(K, kb1 * 64) - kb0 * 64;
                p.Ap = a_image + (size_t)kb0 * round_up(p.M, 8) * 128;
                cl->wp.emplace_back();
                DevBuf &b = cl->wp.back();
                const int r = b.alloc((size_t)p.N8 * (kb1 - kb0) * 1024);
                if (r) return r;
                weight_image_kernel<<<n_sm * 4, 256>>>(static_cast<const __nv_bfloat16 *>(w_dense), b.as<uint4>(), p.n8_0, p.N8, kb0 * 64, p.K, K,
                                                       n_cta / gp.kd, p.half);
                VB_CUDA(cudaGetLastError());
                p.Wp = b.as<uint8_t>();
                ph.push_back(p);
            }
        return VLAB200_OK;
    };
    auto product = [&](const uint8_t *Ap, int M, int out_mode) {
        LoopPhase p{};
        p.Ap = Ap; p.M = M; p.out_mode = out_mode;
        return p;
    };
    auto to_mirror = [&](LoopPhase &p) {  // the phase writes the residual mirror
        p.outp = cl->hbp.as<uint8_t>(); p.out_rows8 = round_up(S, 8);
    };
    const bool ada = d.model == 2;
    const size_t mod_step = (size_t)3 * H, mod_block = (size_t)d.steps * mod_step;  // one norm's vectors for every step
    auto mod_in = [&](int l) { return d.mods + (size_t)(2 * l) * mod_block; };
    auto mod_post = [&](int l) { return d.mods + (size_t)(2 * l + 1) * mod_block; };
    const float *mod_final = ada ? d.mods + (size_t)(2 * d.L) * mod_block : nullptr;
    // W shift (+ bias) of a norm whose output feeds `w_dense` [N][H]
    auto shift_bias = [&](const void *w_dense, int N, const float *mod, const float *add, const float **out_vec) -> int {
        cl->cvec.emplace_back();
        DevBuf &b = cl->cvec.back();
        int r = b.alloc((size_t)d.steps * N * 4);
        if (r) return r;
        const size_t warps = (size_t)d.steps * N;
        shift_bias_kernel<<<(unsigned)((warps * 32 + 255) / 256), 256>>>(static_cast<const __nv_bfloat16 *>(w_dense), mod + H, mod_step, add,
                                                                          b.as<float>(), d.steps, N, H);
        VB_CUDA(cudaGetLastError());
        *out_vec = b.as<float>();
        return VLAB200_OK;
    };
    cl->cvec.reserve((size_t)d.L * 2 + 2);
    // ---- suffix embedding
    {
        LoopPhase p{};
        p.type = PH_EMBED; p.w_dense = static_cast<const __nv_bfloat16 *>(d.w_ain); p.bias = d.b_ain; p.x = d.x;
        p.outp = cl->ap.as<uint8_t>(); p.chunk = d.chunk; p.A_dim = d.A; p.H = H; p.S = S;
        p.sd = d.model == 0 ? d.sd : 0; p.w2 = static_cast<const __nv_bfloat16 *>(d.w_sp); p.b2 = d.b_sp; p.h = d.h;
        p.hbp = cl->hbp.as<uint8_t>();
        p.ssq_out = cl->ssq0.as<float>();
        if (ada) {  // the embedding is the residual stream; its mirror carries the first norm's (1 + scale)
            p.scale_next = mod_in(0); p.mod_stride = (long long)mod_step;
        }
        ph.push_back(p);
        if (!ada) {
            LoopPhase m1 = product(cl->ap.as<uint8_t>(), d.chunk, OUT_BIAS_ACT);
            m1.act = ACT_SILU; m1.bias = d.tvec; m1.bias_step_stride = H; m1.outp = cl->m1p.as<uint8_t>(); m1.out_rows8 = round_up(d.chunk, 8);
            if (push_gemm(m1, d.w_at1l, H, H, plan.mlp)) return no_room();
            LoopPhase m2 = product(cl->m1p.as<uint8_t>(), d.chunk, OUT_BIAS_ACT);
            m2.act = ACT_NONE; m2.bias = d.b_at2; m2.out_f32 = d.h; m2.row_off = S - d.chunk; m2.ssq_out = cl->ssq0.as<float>();
            to_mirror(m2);
            if (push_gemm(m2, d.w_at2, H, H, plan.mlp)) return no_room();
        }
    }
    for (int l = 0; l < d.L; ++l) {
        const bool self = d.is_self[l];
        uint8_t *kp = cl->kpp.as<uint8_t>() + (size_t)l * page_layer, *vp = cl->vpp.as<uint8_t>() + (size_t)l * page_layer;
        const int n_heads = d.n_q + (self ? 2 * d.n_kv : 0);
        LoopPhase qkv = product(cl->hbp.as<uint8_t>(), S, OUT_QKV);
        qkv.use_rms = 1; qkv.ssq_in = l == 0 ? cl->ssq0.as<float>() : cl->ssq.as<float>(); qkv.ssq_n = (l == 0 && ada) ? H / 32 : H / 8;
        qkv.qp = cl->qp.as<uint8_t>();
        if (ada) {
            if ((rc = shift_bias(d.wqkv[l], n_heads * hd, mod_in(l), nullptr, &qkv.bias))) return fail(rc);
            qkv.bias_step_stride = n_heads * hd;
        }
        qkv.kpp = kp; qkv.vpp = vp; qkv.rope = self ? d.rope_self : d.rope_cross; qkv.n_q = d.n_q; qkv.n_kvp = self ? d.n_kv : 0;
        qkv.cap = d.cap; qkv.P = d.P;
        if (push_gemm(qkv, d.wqkv[l], n_heads * hd, H, plan.qkv)) return no_room();
        LoopPhase at{};
        at.type = PH_ATT; at.qp = cl->qp.as<uint8_t>(); at.kpp = kp; at.vpp = vp; at.n_kv = d.n_kv; at.g = g;
        at.S = S; at.R = R; at.n_rt = n_rt; at.kv_len = self ? d.P + S : d.P; at.P = d.P; at.cap = d.cap; at.n_q = d.n_q;
        at.mask_mode = (self && !ada) ? (d.model == 0 ? 1 : 2) : 0;  // pi0.5: every action token sees the prefix and every action token
        at.scale_log2 = 1.4426950408889634f / std::sqrt((float)hd);
        at.kd = att_cta;
        at.per = (at.kv_len + att_cta - 1) / att_cta;  // keys per CTA
        at.outp = cl->attp.as<uint8_t>(); at.out_rows8 = round_up(S, 8);
        {   // the fewest key blocks whose tiles fit: Q | K | V | probabilities (over Q when there is one block) | exchanged rows
            // (over K when there is no room behind: a CTA sends only after its group has read K)
            // Own rows are staged over V, or behind.  K and V may be copied before the grid barrier where they lie behind q|k|v's
            // staged sums, which may still be on their way to its group.
            const int rows = 32 * (hd + 8) * 4, q_bytes = 32 * (int)sq;
            const int n8q = (n_heads * hd / 8 + plan.qkv.cols - 1) / plan.qkv.cols, gq = n_cta / plan.qkv.kd;
            const int stg_end = (int)staged_end(S, (n8q + gq - 1) / gq, (H + 63) / 64, plan.qkv.kd);
            bool found = false;
            for (int nb = 1; !found && nb <= at.per; ++nb) {
                const int ks = (at.per + nb - 1) / nb, ks16 = round_up(ks, 16), pbytes = 32 * (ks16 + 8) * 2;
                if (ks > 128) continue;
                for (int apart = 1; !found && apart >= 0; --apart) {
                    const int k_off = apart ? std::max(q_bytes, round_up(stg_end, 16)) : q_bytes, v_off = k_off + ks * (int)sq, v_end = v_off + ks16 * (int)sq;
                    const bool p_over_q = nb == 1 && pbytes <= k_off;
                    int end = v_end + (p_over_q ? 0 : pbytes);
                    at.p_off = p_over_q ? 0 : v_end;
                    at.k_off = at.recv_off = k_off;
                    at.stage_off = v_off;
                    if (rows > ks16 * (int)sq) {
                        at.stage_off = end;
                        end += rows;
                    }
                    if (end + rows <= CL_ARENA || rows > ks * (int)sq) {
                        at.recv_off = end;
                        end += rows;
                    }
                    if (end > CL_ARENA) continue;
                    at.ks = ks;
                    at.early_k = k_off >= stg_end;
                    at.early_v = v_off >= stg_end;
                    found = true;
                }
            }
            if (!found) return fail(VLAB200_ERR_UNSUPPORTED);
        }
        ph.push_back(at);
        LoopPhase o = product(cl->attp.as<uint8_t>(), S, OUT_RESID);
        to_mirror(o);
        o.h = d.h; o.ssq_out = cl->ssq.as<float>();
        if (ada) {
            o.colscale = mod_in(l) + 2 * H; o.scale_next = mod_post(l); o.mod_stride = (long long)mod_step;
        }
        if (push_gemm(o, d.wo[l], H, qf, plan.o)) return no_room();
        LoopPhase gu = product(cl->hbp.as<uint8_t>(), S, OUT_GATED);
        gu.use_rms = 1; gu.ssq_in = cl->ssq.as<float>(); gu.ssq_n = H / 8;
        gu.act = d.act; gu.outp = cl->gp.as<uint8_t>(); gu.out_rows8 = round_up(S, 8);
        if (ada) {
            if ((rc = shift_bias(d.wgu[l], 2 * d.I, mod_post(l), nullptr, &gu.bias))) return fail(rc);
            gu.bias_step_stride = 2 * d.I;
        }
        if (push_gemm(gu, d.wgu[l], 2 * d.I, H, plan.gu)) return no_room();
        LoopPhase dn = product(cl->gp.as<uint8_t>(), S, OUT_RESID);
        to_mirror(dn);
        dn.h = d.h; dn.ssq_out = cl->ssq.as<float>();
        if (ada) {
            dn.colscale = mod_post(l) + 2 * H; dn.scale_next = l + 1 < d.L ? mod_in(l + 1) : mod_final; dn.mod_stride = (long long)mod_step;
        }
        if (push_gemm(dn, d.wdown[l], H, d.I, plan.dn)) return no_room();
    }
    {
        LoopPhase hdp = product(cl->hbp.as<uint8_t>(), S, OUT_EULER);
        hdp.use_rms = 1; hdp.ssq_in = cl->ssq.as<float>(); hdp.ssq_n = H / 8; hdp.bias = d.b_aout; hdp.x = d.x; hdp.dt = -1.0f / (float)d.steps;
        if (ada) {
            if ((rc = shift_bias(d.w_aout, d.A, mod_final, d.b_aout, &hdp.bias))) return fail(rc);
            hdp.bias_step_stride = d.A;
        }
        if (push_gemm(hdp, d.w_aout, d.A, H, plan.head)) return no_room();
    }
    if ((rc = cl->phases.alloc(ph.size() * sizeof(LoopPhase))) || (rc = cl->counter.alloc(64))) return fail(rc);
    std::vector<WEntry> wt;
    for (const LoopPhase &p : ph)
        if (p.type == PH_GEMM) {
            WEntry w{};
            w.Wp = p.Wp; w.n8_kb = (uint32_t)p.N8 | (uint32_t)((p.K + 63) / 64) << 16; w.kd_m = (uint32_t)p.kd | (uint32_t)p.M << 16;
            wt.push_back(w);
        }
    if ((rc = cl->wtab.alloc(wt.size() * sizeof(WEntry)))) return fail(rc);
    cudaError_t ce = cudaMemcpy(cl->wtab.p, wt.data(), wt.size() * sizeof(WEntry), cudaMemcpyHostToDevice);
    if (ce == cudaSuccess) ce = cudaMemcpy(cl->phases.p, ph.data(), ph.size() * sizeof(LoopPhase), cudaMemcpyHostToDevice);
    if (ce == cudaSuccess) ce = cudaDeviceSynchronize();  // the weight images are complete
    if (ce != cudaSuccess) {
        delete cl;
        return cuda_fail(ce, "chunk loop: phase table / weight images");
    }
    cl->n_phases = (int)ph.size();
    cl->steps = d.steps;
    cl->n_cta = n_cta;
    cl->kernel = kernel;
    LoopParams &lp = cl->lp;
    lp.phases = cl->phases.as<LoopPhase>();
    lp.n_phases = cl->n_phases;
    lp.wtab = cl->wtab.p;
    lp.n_wtab = (int)wt.size();
    lp.att_cta = att_cta;
    lp.steps = d.steps;
    lp.counter = cl->counter.as<unsigned>();
    lp.status = device_status_ptr();
    lp.k_src = static_cast<const __nv_bfloat16 *>(d.k_pages);
    lp.v_src = static_cast<const __nv_bfloat16 *>(d.v_pages);
    lp.kpp = cl->kpp.as<uint8_t>();
    lp.vpp = cl->vpp.as<uint8_t>();
    lp.src_layer_stride = d.layer_stride;
    lp.L = d.L; lp.n_kv = d.n_kv; lp.cap = d.cap; lp.P = d.P; lp.hd = hd;
    *out = cl;
    return VLAB200_OK;
}

void chunk_loop_free(ChunkLoop *cl) { delete cl; }

int chunk_loop_phases(const ChunkLoop *cl) { return cl ? cl->n_phases : 0; }

int chunk_loop_run(ChunkLoop *cl, const float *state, const int32_t *pad, cudaStream_t stream) {
    if (!cl) return VLAB200_ERR_ARG;
    VB_CUDA(cudaMemsetAsync(cl->counter.p, 0, 4, stream));
    LoopParams lp = cl->lp;
    lp.state = state;
    lp.pad = pad;
    const char *trace_path = std::getenv("VLAB200_CHUNK_LOOP_TRACE");  // developer aid: per-phase durations into a text file
    if (trace_path) {
        if (!cl->trace.p && cl->trace.alloc((size_t)(cl->n_phases * cl->steps + 1) * 8)) return VLAB200_ERR_CUDA;
        lp.trace = cl->trace.as<unsigned long long>();
    }
    void *args[] = {&lp};
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr[2];
    loop_launch_config(&cfg, attr, cl->n_cta, stream);
    const cudaError_t le = cudaLaunchKernelExC(&cfg, cl->kernel, args);
    if (le == cudaErrorCooperativeLaunchTooLarge) {  // fewer SMs than the device reports are ours (a partitioned GPU): not an error of the call
        cudaGetLastError();
        return VLAB200_ERR_UNSUPPORTED;
    }
    if (le != cudaSuccess) return cuda_fail(le, "cudaLaunchKernelExC");
    if (lp.trace) {
        const size_t n = (size_t)cl->n_phases * cl->steps;
        std::vector<unsigned long long> t(n);
        VB_CUDA(cudaStreamSynchronize(stream));
        VB_CUDA(cudaMemcpy(t.data(), lp.trace, n * 8, cudaMemcpyDeviceToHost));
        if (FILE *f = std::fopen(trace_path, "w")) {
            for (size_t i = 1; i < n; ++i) std::fprintf(f, "%d %llu\n", (int)(i % cl->n_phases), t[i] - t[i - 1]);  // phase index, ns
            std::fclose(f);
        }
    }
    return VLAB200_OK;
}

}  // namespace vb
