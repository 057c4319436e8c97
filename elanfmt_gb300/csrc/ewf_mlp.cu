// ewf_mlp.cu -- kernels of the learned Green's-function surrogate (training and inference).
//
// A small MLP maps (source x, y, depth, receiver offset, azimuth) to the 6 x 3 x nt elementary
// Green's-function seismograms; the solver generates its training data and measures its error.
// Everything here works on caller-owned device buffers (plain pointers):
//   ewf_mlp_gemm        C[M,N] = A[M,K] . B[N,K]^T (+ bias), bf16 operands on the tcgen05 tensor
//                       cores (TMA-fed, fp32 accumulator in tensor memory), epilogue: fp32 out,
//                       bf16 out, pre-activation out, GELU
//   ewf_mlp_transpose   bf16 [R,C] -> [C,R] (so every product is an A.B^T GEMM)
//   ewf_mlp_gelu_grad   dX = dY * GELU'(pre)  (bf16 out)
//   ewf_mlp_bias_grad   db[n] = sum_m dY[m,n]
//   ewf_mlp_mse_grad    dY = 2 (Y - T) / count (bf16), and the loss sum
//   ewf_mlp_adam        Adam step on fp32 master weights, refreshing the bf16 copy
//   ewf_mlp_combine     out[m,o,t] = sum_f R[m,o,f] G[m,f,t]: per-sample mixing of the predicted
//                       fundamental traces into the 18 moment-tensor x component traces
// The GEMM requires M, N multiples of 128 and K a multiple of 32 (checked on the host).
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cstring>
#include <mutex>
#include <set>
#include <utility>

#include "ewf_umma.h"
#include "ewfd.h"
#include "ewfd_internal.h"

namespace {

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ float gelu(float x) { return 0.5f * x * (1.0f + erff(x * 0.70710678118654752f)); }

__device__ __forceinline__ float gelu_grad(float x)
{
    const float cdf = 0.5f * (1.0f + erff(x * 0.70710678118654752f));
    const float pdf = 0.39894228040143268f * expf(-0.5f * x * x);
    return cdf + x * pdf;
}

// ---------------------------------------------------------------------------------------------
// tcgen05 GEMM: C[M,N] = A[M,K] . B[N,K]^T on the 5th-generation tensor cores; A and B are stored either
// K-major as written or transposed ([K, M], [K, N]: TA, TB), so gradients need no transposed copies.
// Persistent: one CTA per SM walks tiles of one product (a launch may hold two independent ones, each with
// CTAs of its own).  Two fp32 accumulators of 128 lanes x bn columns in tensor memory, so the
// epilogue of one tile overlaps the MMAs of the next.  Warp roles, 352 threads:
//   warps 0 and 10: TMA producers -- per k-stage the boxes of A and of B (128-byte swizzle, ewf_umma.h)
//     into the next free slot of a ring of stages, completing on that slot's "full" mbarrier; the ring
//     runs on across items; rows and K beyond a matrix's end read as zeros;
//   warp 1: MMA issuer -- waits for a free accumulator ("acc_empty"), then per stage for
//     "full", issues 4 tcgen05.mma (K = 16 each) and commits them to the slot's "empty" mbarrier
//     (freeing it for the producer); after the item's last stage commits "acc_full";
//   warps 2-9: epilogue -- wait for "acc_full", read the accumulator with tcgen05.ld (a pair of
//     warps per quarter of the TMEM lanes, each half of the columns), add the bias, GELU or its
//     gradient, release the accumulator ("acc_empty", one arrival per warp).  Every output goes
//     through 32 rows x 32 columns of shared memory, swizzled so that neither the writes nor the TMA
//     store that sends them off meet bank conflicts; the store clips rows beyond M.
// What bounds it at the network's K = 512, where a tile has 8 k-stages: few rows, latency (launch, first
// loads, epilogue); hidden layers of many rows, the GELU's erff; the output layer, the operands' way
// from L2 and the output bytes.  With four epilogue warps storing a row per lane, and now: 128 x 512 x
// 512 24.9 and 6.8 us, 8192 x 512 x 512 25.1 and 12.8, 8192 x 10240 x 512 140 and 82.
// 8192^3 921 and 712 (its 256-column MMAs take 0.27 of a stage's 0.29 us).
// Narrow tiles with a long K are bound by the MMA issuer's chain per k-stage, measured alone with 64 columns:
// four MMAs take 192 cycles, with their commit 218, a wait on a barrier that is ready +130, a commit of the
// accumulator under a condition in the loop +50: 399 in all, as they were.  With the warp's index made uniform by
// a shuffle (addresses and descriptors then stay in uniform registers) those are 192, 195, +80 and +57;
// asking for the next slot while this one's MMAs go out and committing the accumulator after the loop takes the
// last two off the chain.  Gradients of 256 x 512 from 10240 outputs 52 -> 40.5 us, of 1024 x 512 from
// 18432 93 -> 79 (there a 128 x 64 tile's operands come at 54 bytes a cycle, what an SM gets from L2).
// Every mbarrier wait is bounded (g_umma_wait_limit polls): on timeout the wait raises g_umma_err and
// gives up (the outputs of that launch are then invalid, ewf_mlp_status reports it), and no later wait
// of the launch waits at all.  Before the CTA frees its tensor memory and returns, the producer waits
// (again bounded, with a fixed limit) for the last TMA loads it issued and the MMA issuer for every MMA
// it issued, whether or not a wait gave up.  Test hook (ewf_mlp_test_hold): the MMA issuers of the
// CTAs whose first tiles lie in the first 128 x 256 of C withhold the accumulator-ready signal of one
// of their tiles, so the epilogue's wait on it runs out.
// ---------------------------------------------------------------------------------------------
__device__ int g_umma_err = 0;
constexpr int kWaitPolls = 1 << 22;
__device__ int g_umma_wait_limit = kWaitPolls;
__device__ int g_umma_hold = -1;  // tile (CTA-local index) whose acc_full is withheld; -1: none

__device__ __forceinline__ void mbar_init(uint64_t *b, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(b)), "r"(count) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t *b, uint32_t parity)
{
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok)
                 : "r"(smem_u32(b)), "r"(parity)
                 : "memory");
    return ok != 0;
}
// Whether the barrier's phase is over already, without waiting.
__device__ __forceinline__ bool mbar_test(uint64_t *b, uint32_t parity)
{
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok)
                 : "r"(smem_u32(b)), "r"(parity)
                 : "memory");
    return ok != 0;
}
// One lane of a converged warp.  The producer's and the MMA issuer's warps run their loops whole and elect a
// lane for the instructions themselves: as a loop of one lane under a branch, every wait cost 250 cycles
// on a barrier that was ready and every MMA 70, a third of a microsecond per k-stage.
__device__ __forceinline__ bool elect_one()
{
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
    return p != 0;
}
__device__ __forceinline__ bool umma_failed() { return *(volatile int *)&g_umma_err != 0; }
__device__ __forceinline__ bool warp_all(bool x) { return __all_sync(0xffffffffu, x) != 0; }
// Bounded wait of a whole warp, one answer for all its lanes (warp_wait; `limit` polls: g_umma_wait_limit, which each
// warp reads once -- read here, it put a global load's latency, 0.4 us, on every k-stage); gives up at once when another
// wait of the launch has.
__device__ __noinline__ bool mbar_wait_on(uint64_t *b, uint32_t parity, int limit)
{
    if (ewf_umma::warp_wait(limit, [&] { return mbar_try_wait(b, parity); }, umma_failed, warp_all)) return true;
    atomicExch(&g_umma_err, 1);
    return false;
}
__device__ __forceinline__ bool mbar_wait(uint64_t *b, uint32_t parity, int limit)
{
    return warp_all(mbar_try_wait(b, parity)) || mbar_wait_on(b, parity, limit);
}
__device__ __forceinline__ void mbar_drain(uint64_t *b, uint32_t parity)
{
    ewf_umma::bounded_drain([&] { return mbar_test(b, parity); });
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *b, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(b)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void tma_load_2d(void *dst, const CUtensorMap *map, int x, int y, uint64_t *bar)
{
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
                     smem_u32(dst)),
                 "l"((uint64_t)map), "r"(x), "r"(y), "r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accum)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem_d),
                 "l"(da), "l"(db), "r"(idesc), "r"(accum)
                 : "memory");
}
__device__ __forceinline__ void umma_commit(uint64_t *b)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(b))
                 : "memory");
}
// 16 consecutive fp32 accumulator columns of this thread's lane (load and wait in one block so
// no use of the values can be scheduled before the wait)
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[16])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n\t"
                 "tcgen05.wait::ld.sync.aligned;"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                   "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
                 : "r"(taddr)
                 : "memory");
}

// tcgen05.fence::before pairs with the mbarrier arrive that releases an accumulator
constexpr int GEMM_THREADS = ewf_umma::THREADS + ewf_umma::MORE_EPILOGUE + 32;
constexpr int EPI_WARPS = (GEMM_THREADS - 96) / 32;
constexpr int EPI_BOX = 32;                                    // rows and columns of an output box
constexpr int EPI_BUF = EPI_BOX * EPI_BOX * 4;

// Shared memory of a kernel: the operand ring and the epilogue's buffers, one or two per warp.  256 columns:
// one buffer and four stages (three stages and two buffers: 8192 x 10240 x 512 98 us instead of 93 --
// what bounds it is the operand traffic from L2, 393 KB a tile, not the epilogue's wait for a box).
// The ring is cut into stages of the tile's own size, rows + bn rows of 128 bytes: a small tile has
// more of them in flight.  An MMA always reads 128 rows from a stage's start; what lies beyond the tile's
// rows belongs to lanes that are never stored.
constexpr int MAX_STAGES = 16;
template <int BN>
struct Shape {
    static constexpr int BUFS = BN == 128 ? 2 : 1;
    static constexpr int RING = BN == 128 ? 160 * 1024 : 192 * 1024;
    static constexpr int SMEM = RING + EPI_WARPS * BUFS * EPI_BUF + 1024;  // + alignment slack
    static_assert(SMEM <= 227 * 1024, "shared memory of one CTA");
    static_assert(EPI_WARPS * BUFS * EPI_BUF >= ewf_umma::a_bytes(), "an MMA on the last stage reads inside the allocation");
};

enum {
    OUT_F32 = 1, OUT_BF16 = 2, OUT_PRE = 4,  // outputs: fp32, bf16, the fp32 value before the activation
    ACT_GELU = 8,
    ACT_GRAD = 16,                           // bf16(value) * GELU'(gpre): the gradient through the activation
    BF16_DIRECT = 32,                        // the bf16 output is not 16-byte aligned: plain stores
    TRANS_A = 64, TRANS_B = 128              // the operand is stored [K, rows]
};

// One product.  Maps of unused outputs are never read.
struct GemmJob {
    CUtensorMap a, b, f32, bf16, pre;
    const float *bias, *gpre;
    __nv_bfloat16 *cb;
    int M, N, rows, bn;     // tile: rows (32 to 128 of the accumulator's 128 lanes) x bn columns (at most BN)
    int tiles_n, items, nk;
    int cta0, ctas;         // its CTAs
    int flags;
};
constexpr int MAX_JOBS = 2;
struct GemmArgs {
    GemmJob job[MAX_JOBS];
    int njobs;
};

__device__ __forceinline__ float gelu_grad_bf16(float x, float pre)
{
    return __bfloat162float(__float2bfloat16_rn(x)) * gelu_grad(pre);
}

// Sends the warp's 32 x 32 staged values off (one lane), after the writes of every lane.
__device__ __forceinline__ void epi_store(const CUtensorMap *map, const void *buf, int n, int m, int lane)
{
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncwarp();
    if (lane == 0) {
        asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];" ::"l"((uint64_t)map),
                     "r"(n), "r"(m), "r"(smem_u32(buf))
                     : "memory");
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    }
}
template <int BN>
__global__ void __launch_bounds__(GEMM_THREADS, 1) k_gemm(const __grid_constant__ GemmArgs g)
{
    namespace U = ewf_umma;
    constexpr int BUFS = Shape<BN>::BUFS;
    constexpr int COLS = 2 * BN;  // tensor-memory columns: two accumulators
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint64_t full[MAX_STAGES], empty[MAX_STAGES], acc_full[2], acc_empty[2], mma_drain;
    __shared__ uint32_t s_tmem;
    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);  // uniform to the compiler too: the roles' loops run on uniform registers
    uint8_t *smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);

    if (tid == 0) {
        for (int s = 0; s < MAX_STAGES; ++s) {
            mbar_init(&full[s], 2);
            mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], EPI_WARPS);  // one arrival per epilogue warp
        }
        mbar_init(&mma_drain, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        __syncwarp();
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)), "r"(COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem;
    const int limit = __shfl_sync(0xffffffffu, *(volatile int *)&g_umma_wait_limit, 0);
    bool ok = true;  // the same in every lane of a warp, as all that the roles' loops go by
    // a dependent launch may start setting up; nothing of an earlier launch is read or written before it has completed
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");

    const GemmJob &J = g.job[g.njobs > 1 && (int)blockIdx.x >= g.job[1].cta0 ? 1 : 0];
    // (copied to registers: every asm volatile below would have them read again)
    const int t0 = (int)blockIdx.x - J.cta0, bn = J.bn, rows = J.rows, items = J.items, ctas = J.ctas, tiles_n = J.tiles_n, nk = J.nk,
              flags = J.flags, M = J.M, N = J.N;
    const CUtensorMap *const map_a = &J.a, *const map_b = &J.b;
    const int a_part = rows * U::ROW_BYTES, stage = a_part + bn * U::ROW_BYTES;
    const int ns = min(MAX_STAGES, Shape<BN>::RING / stage);
    const bool ta = flags & TRANS_A, tb = flags & TRANS_B;

    if (warp == 0 || warp == 10) {  // TMA producers of the one and the other operand: every k-stage of every tile of this CTA, one ring
        const bool is_b = warp != 0;
        const bool tr = is_b ? tb : ta;
        const int ext = is_b ? bn : rows, boxes = tr ? (ext + U::MN_ATOM - 1) / U::MN_ATOM : 1;
        const CUtensorMap *const map = is_b ? map_b : map_a;
        const uint32_t bytes = (uint32_t)(ext * U::ROW_BYTES);
        uint8_t *const base = smem + (is_b ? a_part : 0);
        int q = 0, s = 0;          // k-stages issued; slot of the next, and
        uint32_t free_parity = 1;  // the parity its "empty" wait passes with (1: a fresh barrier)
        bool ready = true;         // that wait has passed already
        for (int t = t0; t < items && ok; t += ctas) {
            const int r0 = is_b ? (t % tiles_n) * bn : (t / tiles_n) * rows;
            for (int kt = 0; kt < nk; ++kt, ++q) {
                if (!ready && !mbar_wait(&empty[s], free_parity, limit)) { ok = false; break; }
                int s1;
                uint32_t p1;
                U::ring_next(s, free_parity, ns, &s1, &p1);
                const bool next = mbar_test(&empty[s1], p1);
                if (elect_one()) {
                    uint8_t *dst = base + s * stage;
                    mbar_expect_tx(&full[s], bytes);
                    if (tr) {
                        for (int r = 0; r < boxes; ++r) tma_load_2d(dst + r * U::MN_BLOCK_BYTES, map, r0 + r * U::MN_ATOM, kt * U::BK, &full[s]);
                    } else {
                        tma_load_2d(dst, map, kt * U::BK, r0, &full[s]);
                    }
                }
                ready = warp_all(next);
                s = s1;
                free_parity = p1;
            }
        }
        // the loads issued last into each slot land before the CTA's shared memory goes
        for (int p = (q > ns ? q - ns : 0); p < q; ++p)
            mbar_drain(&full[U::ring_slot(p, ns)], U::ring_full_parity(p, ns));
    } else if (warp == 1) {  // MMA issuer
        const uint32_t idesc = U::instr_desc_bf16_f32(U::BM, bn, ta, tb);
        const bool first = (t0 / tiles_n) * rows < U::BM && (t0 % tiles_n) * bn < 256;
        const int hold = __shfl_sync(0xffffffffu, first ? *(volatile int *)&g_umma_hold : -1, 0);
        // the K = 16 slices of a stage: start addresses (16-byte units) and descriptors without them
        const uint64_t da0 = ta ? U::smem_desc_sw128_mn(0) : U::smem_desc_sw128(0), db0 = tb ? U::smem_desc_sw128_mn(0) : U::smem_desc_sw128(0);
        const int sa = (ta ? U::MN_K_STEP : 32) >> 4, sb = (tb ? U::MN_K_STEP : 32) >> 4;
        int s = 0, i = 0;
        uint32_t full_parity = 0;
        bool ready = false;  // the wait for slot s has passed already
        for (int t = t0; t < items && ok; t += ctas, ++i) {
            const int b = U::acc_buf(i);
            if (U::acc_needs_free(i) && !mbar_wait(&acc_empty[b], U::acc_free_parity(i), limit)) { ok = false; break; }
            tc_fence_after();
            const uint32_t d = tmem + (uint32_t)(b * BN);  // accumulators BN columns apart
            for (int kt = 0; kt < nk; ++kt) {
                if (!ready && !mbar_wait(&full[s], full_parity, limit)) { ok = false; break; }
                tc_fence_after();
                int s1;
                uint32_t p1;
                U::ring_next(s, full_parity, ns, &s1, &p1);
                const bool next = mbar_test(&full[s1], p1);
                if (elect_one()) {
                    const uint32_t a0 = smem_u32(smem + s * stage) >> 4, b0 = a0 + (uint32_t)(a_part >> 4);
#pragma unroll
                    for (int j = 0; j < U::BK / U::MMA_K; ++j)
                        umma_bf16(d, da0 + a0 + (uint32_t)(sa * j), db0 + b0 + (uint32_t)(sb * j), idesc, (kt > 0 || j > 0) ? 1u : 0u);
                    umma_commit(&empty[s]);
                }
                ready = warp_all(next);
                s = s1;
                full_parity = p1;
            }
            if (ok && i != hold && elect_one()) umma_commit(&acc_full[b]);
            __syncwarp();
        }
        // every MMA issued completes before the tensor memory is freed
        if (elect_one()) umma_commit(&mma_drain);
        __syncwarp();
        mbar_drain(&mma_drain, 0);
    } else {  // epilogue warps 2..9: TMEM lane quarter warp % 4, half of the columns each
        const int quarter = warp & 3, half = (warp - 2) >> 2;
        uint8_t *const bufs = smem + Shape<BN>::RING + (warp - 2) * (BUFS * EPI_BUF);
        int i = 0, nb = 0;
        // the next staging buffer, free once the store before last (BUFS = 2) or the last one has read it
        auto next_buf = [&]() {
            if (lane == 0) {
                if (BUFS == 2) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
                else asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
            }
            __syncwarp();
            return bufs + (BUFS == 2 ? (nb++ & 1) * EPI_BUF : 0);
        };
        for (int t = t0; t < items; t += ctas, ++i) {
            const int m0 = (t / tiles_n) * rows, n0 = (t % tiles_n) * bn;
            const int b = U::acc_buf(i);
            const bool got = warp_all(!umma_failed()) && mbar_wait(&acc_full[b], U::acc_full_parity(i), limit);
            tc_fence_after();
            const int mrow = m0 + 32 * quarter, row = mrow + lane;
#pragma unroll 1
            for (int c0 = half * (bn / 2); c0 < (half + 1) * (bn / 2); c0 += EPI_BOX) {
                const int n = n0 + c0;
                float x[EPI_BOX];
#pragma unroll
                for (int h = 0; h < EPI_BOX; h += 16) {
                    uint32_t v[16];
                    tmem_ld16(tmem + ((uint32_t)(32 * quarter) << 16) + (uint32_t)(b * BN + c0 + h), v);
#pragma unroll
                    for (int e = 0; e < 16; ++e) x[h + e] = got ? __uint_as_float(v[e]) : __int_as_float(0x7fc00000);
                }
                if (c0 + EPI_BOX == (half + 1) * (bn / 2)) {  // this warp's part of the accumulator is in registers
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&acc_empty[b])) : "memory");
                }
                if (32 * quarter >= rows) continue;  // lanes past the tile's rows: what they hold is not part of C
                if (n >= N) continue;                // columns past the last (N not a multiple of bn)
                if (J.bias) {
#pragma unroll
                    for (int e = 0; e < EPI_BOX; ++e) x[e] += J.bias[n + e];
                }
                // staged rows: 16-byte chunk q of row r at chunk q ^ (r % 8) (fp32) or q ^ (r / 2 % 4) (bf16)
                if ((flags & OUT_PRE)) {
                    uint8_t *buf = next_buf();
#pragma unroll
                    for (int q = 0; q < 8; ++q)
                        *reinterpret_cast<float4 *>(buf + lane * 128 + ((q ^ (lane & 7)) << 4)) =
                            make_float4(x[4 * q], x[4 * q + 1], x[4 * q + 2], x[4 * q + 3]);
                    epi_store(&J.pre, buf, n, mrow, lane);
                }
                if ((flags & ACT_GELU)) {
#pragma unroll
                    for (int e = 0; e < EPI_BOX; ++e) x[e] = gelu(x[e]);
                }
                if ((flags & ACT_GRAD)) {
                    const float4 *p = reinterpret_cast<const float4 *>(J.gpre + (size_t)min(row, M - 1) * N + n);
#pragma unroll
                    for (int e = 0; e < EPI_BOX; e += 4) {
                        const float4 pv = p[e / 4];
                        x[e] = gelu_grad_bf16(x[e], pv.x);
                        x[e + 1] = gelu_grad_bf16(x[e + 1], pv.y);
                        x[e + 2] = gelu_grad_bf16(x[e + 2], pv.z);
                        x[e + 3] = gelu_grad_bf16(x[e + 3], pv.w);
                    }
                }
                if (flags & OUT_F32) {
                    uint8_t *buf = next_buf();
#pragma unroll
                    for (int q = 0; q < 8; ++q)
                        *reinterpret_cast<float4 *>(buf + lane * 128 + ((q ^ (lane & 7)) << 4)) =
                            make_float4(x[4 * q], x[4 * q + 1], x[4 * q + 2], x[4 * q + 3]);
                    epi_store(&J.f32, buf, n, mrow, lane);
                }
                if ((flags & OUT_BF16)) {
                    __nv_bfloat162 y[EPI_BOX / 2];
#pragma unroll
                    for (int e = 0; e < EPI_BOX; e += 2) y[e / 2] = __floats2bfloat162_rn(x[e], x[e + 1]);
                    if (flags & BF16_DIRECT) {
                        if (row < M) {
                            __nv_bfloat162 *o = reinterpret_cast<__nv_bfloat162 *>(J.cb + (size_t)row * N + n);
#pragma unroll
                            for (int e = 0; e < EPI_BOX / 2; ++e) o[e] = y[e];
                        }
                    } else {
                        uint8_t *buf = next_buf();
#pragma unroll
                        for (int q = 0; q < 4; ++q)
                            *reinterpret_cast<uint4 *>(buf + lane * 64 + ((q ^ ((lane >> 1) & 3)) << 4)) = *reinterpret_cast<uint4 *>(&y[4 * q]);
                        epi_store(&J.bf16, buf, n, mrow, lane);
                    }
                }
            }
        }
        if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        __syncwarp();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(COLS) : "memory");
    }
}
int check(cudaError_t e, const char *what);

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn tensor_map_encoder()
{
    static const EncodeTiledFn enc = [] {
        cudaDriverEntryPointQueryResult q;
        void *fn = nullptr;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q) == cudaSuccess && fn &&
            q == cudaDriverEntryPointSuccess)
            return (EncodeTiledFn)fn;
        return (EncodeTiledFn) nullptr;
    }();
    return enc;
}

// 2-D map of a bf16 operand of `rows` rows: K-major [rows, K] in boxes of BK x box_rows, or (mn)
// transposed, [K, rows], in boxes of 64 rows x BK
int operand_map(CUtensorMap *m, const void *ptr, int rows, int K, int box_rows, bool mn)
{
    const EncodeTiledFn enc = tensor_map_encoder();
    if (!enc) return ewf_fail(EWF_ERR_CUDA, "gemm: cuTensorMapEncodeTiled unavailable");
    const cuuint64_t inner = mn ? (cuuint64_t)rows : (cuuint64_t)K;
    const cuuint64_t dims[2] = {inner, mn ? (cuuint64_t)K : (cuuint64_t)rows};
    const cuuint64_t strides[1] = {inner * 2};
    const cuuint32_t box[2] = {(cuuint32_t)(mn ? ewf_umma::MN_ATOM : ewf_umma::BK), (cuuint32_t)(mn ? ewf_umma::BK : box_rows)};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult r = enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(ptr), dims, strides, box, estr,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? EWF_OK : ewf_fail(EWF_ERR_ARG, "gemm: tensor map rejected (CUresult %d)", (int)r);
}

// map of an output [M, N], fp32 or bf16, in boxes of 32 x 32
int output_map(CUtensorMap *m, void *C, int M, int N, bool f32)
{
    const EncodeTiledFn enc = tensor_map_encoder();
    if (!enc) return ewf_fail(EWF_ERR_CUDA, "gemm: cuTensorMapEncodeTiled unavailable");
    const cuuint64_t dims[2] = {(cuuint64_t)N, (cuuint64_t)M};
    const cuuint64_t strides[1] = {(cuuint64_t)N * (f32 ? 4 : 2)};
    const cuuint32_t box[2] = {EPI_BOX, EPI_BOX};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult r = enc(m, f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, C, dims, strides, box, estr,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, f32 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
                           CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? EWF_OK : ewf_fail(EWF_ERR_ARG, "gemm: output tensor map rejected (CUresult %d)", (int)r);
}

// A kernel's shared-memory attribute is a per-device setting: set once per device ordinal.
template <typename K>
int gemm_smem_attribute(K kernel, int dev, int bytes)
{
    static std::mutex mu;
    static std::set<std::pair<const void *, int>> done;
    std::lock_guard<std::mutex> lock(mu);
    const auto key = std::make_pair((const void *)kernel, dev);
    if (done.count(key)) return EWF_OK;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) return check(e, "gemm smem attribute");
    done.insert(key);
    return EWF_OK;
}

struct Device {
    int id = 0, sms = 1;
};
int this_device(Device *d)
{
    int st = check(cudaGetDevice(&d->id), "device");
    if (st) return st;
    return check(cudaDeviceGetAttribute(&d->sms, cudaDevAttrMultiProcessorCount, d->id), "device");
}

// A launch that may start while the stream's previous kernel still runs (its kernel waits for it with
// griddepcontrol.wait before it reads or writes anything).
template <typename... P, typename... A>
int launch_pdl(const char *what, void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A &&...args)
{
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return check(cudaLaunchKernelEx(&cfg, kern, std::forward<A>(args)...), what);
}

int gemm_tiles(int M, int N, int rows, int bn) { return ((M + rows - 1) / rows) * ((N + bn - 1) / bn); }

// What a product is, apart from its tiles
struct Product {
    const void *A = nullptr, *B = nullptr;
    bool ta = false, tb = false;   // stored [K, M], [K, N]
    int M = 0, N = 0, K = 0;
    float *f32 = nullptr;
    void *bf16 = nullptr;
    float *pre = nullptr;
    const float *bias = nullptr, *gpre = nullptr;
    int act = 0;                   // ACT_GELU, ACT_GRAD or 0
};

int make_job(GemmJob *J, const Product &p, int rows, int bn)
{
    int st = operand_map(&J->a, p.A, p.M, p.K, rows, p.ta);
    if (!st) st = operand_map(&J->b, p.B, p.N, p.K, bn, p.tb);
    if (!st && p.f32) st = output_map(&J->f32, p.f32, p.M, p.N, true);
    const bool direct = p.bf16 && ((uintptr_t)p.bf16 & 15);
    if (!st && p.bf16 && !direct) st = output_map(&J->bf16, p.bf16, p.M, p.N, false);
    if (!st && p.pre) st = output_map(&J->pre, p.pre, p.M, p.N, true);
    if (st) return st;
    J->bias = p.bias;
    J->gpre = p.gpre;
    J->cb = (__nv_bfloat16 *)p.bf16;
    J->M = p.M;
    J->N = p.N;
    J->rows = rows;
    J->bn = bn;
    J->tiles_n = (p.N + bn - 1) / bn;
    J->items = gemm_tiles(p.M, p.N, rows, bn);
    J->nk = (p.K + ewf_umma::BK - 1) / ewf_umma::BK;
    J->flags = (p.f32 ? OUT_F32 : 0) | (p.bf16 ? OUT_BF16 : 0) | (p.pre ? OUT_PRE : 0) | p.act | (direct ? BF16_DIRECT : 0) |
               (p.ta ? TRANS_A : 0) | (p.tb ? TRANS_B : 0);
    return EWF_OK;
}

template <int BN>
int gemm_go(const GemmArgs &g, int ctas, const Device &dev, cudaStream_t stream)
{
    const int st = gemm_smem_attribute(k_gemm<BN>, dev.id, Shape<BN>::SMEM);
    if (st) return st;
    return launch_pdl("gemm launch", k_gemm<BN>, dim3(ctas), dim3(GEMM_THREADS), Shape<BN>::SMEM, stream, g);
}

// One product.  The tile width: 256 columns once there is a tile per SM, as each stage then feeds the most
// MMA work; below that narrower tiles and, as long as every tile still has an SM, fewer rows, which spread
// operands and epilogue over more of them (128 x 512 x 512 runs on 32 CTAs instead of 2).
int gemm_one(const Product &p, cudaStream_t stream)
{
    Device dev;
    int st = this_device(&dev);
    if (st) return st;
    int bn = 64, rows = ewf_umma::BM;
    if (p.N % 256 == 0 && gemm_tiles(p.M, p.N, ewf_umma::BM, 256) >= dev.sms) bn = 256;
    else if (gemm_tiles(p.M, p.N, ewf_umma::BM, 128) >= dev.sms) bn = 128;
    else if (!p.ta)
        while (rows > 32 && gemm_tiles(p.M, p.N, rows / 2, 64) <= dev.sms) rows /= 2;
    alignas(64) GemmArgs g;
    memset(&g, 0, sizeof(g));
    GemmJob &J = g.job[0];
    if ((st = make_job(&J, p, rows, bn))) return st;
    J.ctas = J.items < dev.sms ? J.items : dev.sms;
    g.njobs = 1;
    if (bn == 256) return gemm_go<256>(g, J.ctas, dev, stream);
    if (bn == 128) return gemm_go<128>(g, J.ctas, dev, stream);
    return gemm_go<64>(g, J.ctas, dev, stream);
}

// The two products of a layer's backward pass in one launch: dH = dY . W (its K, the layer's outputs, may be
// far larger than its tiles are many) and gW = dY^T . H.  dH gets a CTA per tile and gW the SMs that are
// left, so the second hides behind the first.  A dH tile multiplies stage after stage, 0.16 us each up to 64 rows
// and 0.24 with 128 -- its K is not split, so that its sums keep their order -- so small tiles spread the
// work: 32 or 64 of the accumulator's 128 lanes while CTAs for them and as many again for gW are there.
// 256 x 512 from K = 10240: 110 us on 4 CTAs of 128 x 256 at 0.7 us a stage, now 28 with the weight gradient
// behind it.
// How the SMs are shared: the tile height that has the slower of the two done first, by the measured time of a
// k-stage.  1024 x 512 from K = 18432 beside 18432 x 512: 64 tiles of 128 rows take 69 us and the other 88
// SMs 33, 88 of 96 rows about 60 (a backward pass of these layers 79.6 -> 71.7).
float stage_us(int rows, int bn) { return std::max(0.16f, (float)(rows + bn) * ewf_umma::ROW_BYTES / 104e3f); }
int gemm_pair(const Product &dh, const Product &gw, cudaStream_t stream)
{
    Device dev;
    int st = this_device(&dev);
    if (st) return st;
    const int bn = gemm_tiles(gw.M, gw.N, ewf_umma::BM, 128) >= dev.sms / 2 ? 128 : 64, gw_items = gemm_tiles(gw.M, gw.N, ewf_umma::BM, bn);
    const int nk_dh = (dh.K + ewf_umma::BK - 1) / ewf_umma::BK, nk_gw = (gw.K + ewf_umma::BK - 1) / ewf_umma::BK;
    int rows = ewf_umma::BM;
    float best = 1e30f;
    for (int r = 32; r <= ewf_umma::BM; r += 32) {
        const int tiles = gemm_tiles(dh.M, dh.N, r, 64), left = dev.sms - tiles;
        if (left < dev.sms / 4 && r < ewf_umma::BM) continue;
        const float t_dh = (float)((tiles + dev.sms - 1) / dev.sms) * nk_dh * stage_us(r, 64),
                    t_gw = (float)((gw_items + std::max(left, 1) - 1) / std::max(left, 1)) * (nk_gw * stage_us(ewf_umma::BM, bn) + 1.f);
        const float t = std::max(t_dh, t_gw);
        if (t < best) {
            best = t;
            rows = r;
        }
    }
    alignas(64) GemmArgs g;
    memset(&g, 0, sizeof(g));
    GemmJob &a = g.job[0], &b = g.job[1];
    if ((st = make_job(&a, dh, rows, 64))) return st;
    if ((st = make_job(&b, gw, ewf_umma::BM, bn))) return st;
    const int left = dev.sms - a.items;
    a.ctas = left >= dev.sms / 4 ? a.items : a.items < dev.sms ? a.items : dev.sms;
    g.njobs = 2;
    b.cta0 = a.ctas;
    b.ctas = left >= dev.sms / 4 ? left : dev.sms;  // dH fills the GPU by itself: gW's CTAs follow
    if (b.ctas > b.items) b.ctas = b.items;
    return gemm_go<128>(g, a.ctas + b.ctas, dev, stream);
}

__global__ void k_transpose(const __nv_bfloat16 *__restrict__ in, __nv_bfloat16 *__restrict__ out, int R, int Cc)
{
    __shared__ __nv_bfloat16 t[32][33];
    const int c0 = blockIdx.x * 32, r0 = blockIdx.y * 32;
    for (int y = threadIdx.y; y < 32; y += blockDim.y) {
        const int r = r0 + y, c = c0 + threadIdx.x;
        if (r < R && c < Cc) t[y][threadIdx.x] = in[(size_t)r * Cc + c];
    }
    __syncthreads();
    for (int y = threadIdx.y; y < 32; y += blockDim.y) {
        const int c = c0 + y, r = r0 + threadIdx.x;
        if (r < R && c < Cc) out[(size_t)c * R + r] = t[threadIdx.x][y];
    }
}

__global__ void k_gelu_grad(const __nv_bfloat16 *__restrict__ dy, const float *__restrict__ pre, __nv_bfloat16 *__restrict__ dx,
                            size_t n)
{
    for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x)
        dx[e] = __float2bfloat16_rn(__bfloat162float(dy[e]) * gelu_grad(pre[e]));
}

__global__ void k_bias_grad(const __nv_bfloat16 *__restrict__ dy, float *__restrict__ db, int M, int N)
{
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= N) return;
    float s = 0.f;
    for (int m = 0; m < M; ++m) s += __bfloat162float(dy[(size_t)m * N + n]);
    db[n] = s;
}

// dY = 2 (Y - T) / count; loss partial sums (one per block) into part[blockIdx.x]
__global__ void k_mse_grad(const float *__restrict__ y, const float *__restrict__ t, __nv_bfloat16 *__restrict__ dy, size_t n,
                           float scale, float *__restrict__ part)
{
    __shared__ float red[256];
    float s = 0.f;
    for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x) {
        const float d = y[e] - t[e];
        s += d * d;
        dy[e] = __float2bfloat16_rn(2.f * d * scale);
    }
    red[threadIdx.x] = s;
    __syncthreads();
    for (int w = 128; w > 0; w >>= 1) {
        if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) part[blockIdx.x] = red[0];
}

__global__ void k_adam(float *__restrict__ w, float *__restrict__ m, float *__restrict__ v, const float *__restrict__ g,
                       __nv_bfloat16 *__restrict__ wb, size_t n, float lr, float b1, float b2, float eps, float c1, float c2,
                       float wd)
{
    for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x) {
        const float ge = g[e] + wd * w[e];
        const float me = b1 * m[e] + (1.f - b1) * ge;
        const float ve = b2 * v[e] + (1.f - b2) * ge * ge;
        m[e] = me;
        v[e] = ve;
        const float we = w[e] - lr * (me / c1) / (sqrtf(ve / c2) + eps);
        w[e] = we;
        if (wb) wb[e] = __float2bfloat16_rn(we);
    }
}

// ---------------------------------------------------------------------------------------------
// The training step's own forms of the kernels above: every layer's work of one kind in one launch,
// 16-byte accesses, started while the launch before ends.
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ void pdl_wait()
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Bias gradients of every layer: a CTA sums 64 columns, a pair of columns per lane and every 32nd row per
// warp, then the 32 warps' sums in order.  (A thread per column over all rows: 256 x 10240 20 us.)
constexpr int BIAS_GROUP = 8;
struct BiasJobs {
    const __nv_bfloat16 *dy[BIAS_GROUP];
    float *db[BIAS_GROUP];
    int N[BIAS_GROUP], block0[BIAS_GROUP];
    int n, M;
};
__global__ void __launch_bounds__(1024) k_bias_grads(const BiasJobs J)
{
    __shared__ float2 part[32][33];
    pdl_wait();
    int q = 0;
    while (q + 1 < J.n && (int)blockIdx.x >= J.block0[q + 1]) ++q;
    const int N = J.N[q], lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int col = ((int)blockIdx.x - J.block0[q]) * 64 + 2 * lane;
    float2 s = make_float2(0.f, 0.f);
    if (col < N) {
        const __nv_bfloat162 *p = reinterpret_cast<const __nv_bfloat162 *>(J.dy[q] + col);
#pragma unroll 8
        for (int m = warp; m < J.M; m += 32) {
            const float2 v = __bfloat1622float2(p[(size_t)m * (N / 2)]);
            s.x += v.x;
            s.y += v.y;
        }
    }
    part[warp][lane] = s;
    __syncthreads();
    if (warp == 0 && col < N) {
        float2 t = part[0][lane];
        for (int w = 1; w < 32; ++w) {
            t.x += part[w][lane].x;
            t.y += part[w][lane].y;
        }
        J.db[q][col] = t.x;
        J.db[q][col + 1] = t.y;
    }
}

// k_mse_grad four values at a time (n % 4 == 0, aligned), with the loss from the partial sums by the last
// CTA to finish: done counts the CTAs and is left at zero.
__global__ void __launch_bounds__(256) k_mse_loss(const float4 *y, const float4 *t, uint2 *dy,
                                                  size_t n4, float scale, float *__restrict__ part, unsigned *__restrict__ done,
                                                  float *__restrict__ loss)
{
    __shared__ float red[256];
    __shared__ bool last;
    pdl_wait();
    float s = 0.f;
    for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < n4; e += (size_t)gridDim.x * blockDim.x) {
        const float4 a = y[e], b = __ldcs(t + e);
        const float d[4] = {a.x - b.x, a.y - b.y, a.z - b.z, a.w - b.w};
#pragma unroll
        for (int q = 0; q < 4; ++q) s += d[q] * d[q];
        __nv_bfloat162 o[2] = {__floats2bfloat162_rn(2.f * d[0] * scale, 2.f * d[1] * scale),
                               __floats2bfloat162_rn(2.f * d[2] * scale, 2.f * d[3] * scale)};
        dy[e] = *reinterpret_cast<uint2 *>(o);
    }
    auto block_sum = [&](float v) {
        red[threadIdx.x] = v;
        __syncthreads();
        for (int w = 128; w > 0; w >>= 1) {
            if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
            __syncthreads();
        }
    };
    block_sum(s);
    if (threadIdx.x == 0) {
        part[blockIdx.x] = red[0];
        __threadfence();
        last = atomicAdd(done, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    float v = 0.f;
    for (unsigned b = threadIdx.x; b < gridDim.x; b += 256) v += *(volatile float *)&part[b];
    block_sum(v);
    if (threadIdx.x == 0) {
        *loss = red[0] * scale;
        *done = 0u;
    }
}

// k_adam over several tensors, four elements per thread (16-byte aligned; a tensor's tail by its last
// threads).  Bound by memory, 28 bytes an element and 2 for the bf16 copy.
constexpr int ADAM_GROUP = 16, ADAM_BLOCK = 256 * 4;  // elements per CTA
struct AdamJobs {
    float *w[ADAM_GROUP], *m[ADAM_GROUP], *v[ADAM_GROUP];
    const float *g[ADAM_GROUP];
    __nv_bfloat16 *wb[ADAM_GROUP];
    unsigned n[ADAM_GROUP], block0[ADAM_GROUP];
    float wd[ADAM_GROUP];
    int njobs;
    float lr, b1, b2, eps, c1, c2;
};
__device__ __forceinline__ void adam_one(const AdamJobs &J, float wd, float &w, float &m, float &v, float g)
{
    const float ge = g + wd * w;
    const float me = J.b1 * m + (1.f - J.b1) * ge;
    const float ve = J.b2 * v + (1.f - J.b2) * ge * ge;
    m = me;
    v = ve;
    w = w - J.lr * (me / J.c1) / (sqrtf(ve / J.c2) + J.eps);
}
__global__ void __launch_bounds__(256) k_adam_all(const AdamJobs J)
{
    pdl_wait();
    int q = 0;
    while (q + 1 < J.njobs && blockIdx.x >= J.block0[q + 1]) ++q;
    const unsigned e = (blockIdx.x - J.block0[q]) * ADAM_BLOCK + threadIdx.x * 4, n = J.n[q];
    const float wd = J.wd[q];
    if (e + 4 <= n) {
        float4 w = *reinterpret_cast<float4 *>(J.w[q] + e), m = *reinterpret_cast<float4 *>(J.m[q] + e),
               v = *reinterpret_cast<float4 *>(J.v[q] + e);
        const float4 g = *reinterpret_cast<const float4 *>(J.g[q] + e);
        adam_one(J, wd, w.x, m.x, v.x, g.x);
        adam_one(J, wd, w.y, m.y, v.y, g.y);
        adam_one(J, wd, w.z, m.z, v.z, g.z);
        adam_one(J, wd, w.w, m.w, v.w, g.w);
        *reinterpret_cast<float4 *>(J.w[q] + e) = w;
        *reinterpret_cast<float4 *>(J.m[q] + e) = m;
        *reinterpret_cast<float4 *>(J.v[q] + e) = v;
        if (J.wb[q]) {
            __nv_bfloat162 o[2] = {__floats2bfloat162_rn(w.x, w.y), __floats2bfloat162_rn(w.z, w.w)};
            *reinterpret_cast<uint2 *>(J.wb[q] + e) = *reinterpret_cast<uint2 *>(o);
        }
    } else {
        for (unsigned k = e; k < n; ++k) {
            adam_one(J, wd, J.w[q][k], J.m[q][k], J.v[q][k], J.g[q][k]);
            if (J.wb[q]) J.wb[q][k] = __float2bfloat16_rn(J.w[q][k]);
        }
    }
}

unsigned blocks_for(size_t n) { return (unsigned)((n + 255) / 256 < 152 * 32 ? (n + 255) / 256 : 152 * 32); }

// Mixing of a sample's nin input traces into nout output traces.  Bound by memory (4 (nin + nout) bytes
// per time sample) when each input is read once: a thread holds all its inputs of VEC times in
// registers and runs over the outputs, the mixing matrix sits in shared memory (one 16-byte read feeds
// 4 VEC products).  The sums keep their order, input by input from zero.  8192 samples x 1024 times, 10 -> 18:
// 537 us with a time per thread re-reading its inputs for every output, 140 now (138 at the copy rate).
constexpr int COMBINE_MAX = 2048;   // elements of a sample's matrix
constexpr int COMBINE_REGS = 16;    // inputs held in registers
template <int NIN, int VEC>
__global__ void __launch_bounds__(128) k_combine(const float *__restrict__ R, const float *__restrict__ G, float *__restrict__ out,
                                                 int nout, int T)
{
    constexpr int P = (NIN + 3) / 4 * 4;  // padded row of the matrix
    extern __shared__ __align__(16) float r[];
    const long long m = blockIdx.y;
    for (int e = threadIdx.x; e < nout * P; e += blockDim.x) r[e] = e % P < NIN ? R[m * nout * NIN + e / P * NIN + e % P] : 0.f;
    __syncthreads();
    const int t = (blockIdx.x * blockDim.x + threadIdx.x) * VEC;
    if (t >= T) return;
    float g[NIN][VEC];
    const float *gp = G + m * NIN * T + t;
#pragma unroll
    for (int f = 0; f < NIN; ++f) {
        if constexpr (VEC == 4) *reinterpret_cast<float4 *>(g[f]) = __ldcs(reinterpret_cast<const float4 *>(gp + (long long)f * T));
        else g[f][0] = __ldcs(gp + (long long)f * T);
    }
    float *o = out + m * nout * T + t;
#pragma unroll 2
    for (int a = 0; a < nout; ++a) {
        float acc[VEC];
#pragma unroll
        for (int v = 0; v < VEC; ++v) acc[v] = 0.f;
#pragma unroll
        for (int f = 0; f < NIN; f += 4) {
            const float4 q = *reinterpret_cast<const float4 *>(&r[a * P + f]);
            const float c[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (f + e < NIN)
#pragma unroll
                    for (int v = 0; v < VEC; ++v) acc[v] += c[e] * g[f + e][v];
        }
        if constexpr (VEC == 4) __stcs(reinterpret_cast<float4 *>(o + (long long)a * T), make_float4(acc[0], acc[1], acc[2], acc[3]));
        else __stcs(o + (long long)a * T, acc[0]);
    }
}

// More inputs than fit in registers: a time per thread, the inputs from L1 for every output.
__global__ void k_combine_any(const float *__restrict__ R, const float *__restrict__ G, float *__restrict__ out, int nout, int nin, int T)
{
    __shared__ float r[COMBINE_MAX];
    const long long m = blockIdx.y;
    for (int e = threadIdx.x; e < nout * nin; e += blockDim.x) r[e] = R[m * nout * nin + e];
    __syncthreads();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= T) return;
    const float *g = G + m * nin * T + t;
    float *o = out + m * nout * T + t;
    for (int a = 0; a < nout; ++a) {
        float acc = 0.f;
        for (int f = 0; f < nin; ++f) acc += r[a * nin + f] * g[(long long)f * T];
        o[(long long)a * T] = acc;
    }
}

template <int NIN>
void launch_combine(const float *R, const float *G, float *out, int M, int nout, int nin, int T, cudaStream_t stream)
{
    if constexpr (NIN > COMBINE_REGS) {
        k_combine_any<<<dim3((T + 255) / 256, M), 256, 0, stream>>>(R, G, out, nout, nin, T);
    } else {
        if (nin != NIN) return launch_combine<NIN + 1>(R, G, out, M, nout, nin, T, stream);
        const size_t smem = (size_t)nout * ((NIN + 3) / 4 * 4) * sizeof(float);  // at most 4 x 2048 elements
        if (T % 4 == 0 && !(((uintptr_t)G | (uintptr_t)out) & 15))
            k_combine<NIN, 4><<<dim3((T + 511) / 512, M), 128, smem, stream>>>(R, G, out, nout, T);
        else
            k_combine<NIN, 1><<<dim3((T + 127) / 128, M), 128, smem, stream>>>(R, G, out, nout, T);
    }
}

int check(cudaError_t e, const char *what)
{
    if (e != cudaSuccess) return ewf_fail(EWF_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
    return EWF_OK;
}

}  // namespace

extern "C" int ewf_mlp_gemm(const void *A, const void *B, const float *bias, float *Cf, void *Cb, float *pre, int32_t M,
                            int32_t N, int32_t K, int32_t act, void *stream)
{
    if (!A || !B || (!Cf && !Cb && !pre)) return ewf_fail(EWF_ERR_ARG, "gemm: NULL operand");
    if (M <= 0 || N <= 0 || K <= 0 || M % 128 || N % 128 || K % 32)
        return ewf_fail(EWF_ERR_ARG, "gemm: M, N must be multiples of 128 and K of 32 (got %d %d %d)", M, N, K);
    if (act != 0 && act != 1) return ewf_fail(EWF_ERR_ARG, "gemm: act must be 0 or 1");
    if (((uintptr_t)A | (uintptr_t)B) & 15) return ewf_fail(EWF_ERR_ARG, "gemm: A and B must be 16-byte aligned");
    if (((uintptr_t)Cf | (uintptr_t)pre) & 15 || (uintptr_t)Cb & 3) return ewf_fail(EWF_ERR_ARG, "gemm: outputs misaligned");
    Product p;
    p.A = A;
    p.B = B;
    p.M = M;
    p.N = N;
    p.K = K;
    p.f32 = Cf;
    p.bf16 = Cb;
    p.pre = pre;
    p.bias = bias;
    p.act = act == 1 ? ACT_GELU : 0;
    return gemm_one(p, (cudaStream_t)stream);
}

// ---------------------------------------------------------------------------------------------
// The network's passes, one call each
// ---------------------------------------------------------------------------------------------
namespace {
// rows: the gradients' row count has to be a multiple of 128, as ewf_mlp_gemm's
int check_net(const char *what, int32_t n, const int32_t *sizes, int32_t M, int in_mult)
{
    if (n < 1 || !sizes || M <= 0) return ewf_fail(EWF_ERR_ARG, "%s: bad network or batch", what);
    if (sizes[0] <= 0 || sizes[0] % in_mult) return ewf_fail(EWF_ERR_ARG, "%s: the input width must be a multiple of %d", what, in_mult);
    for (int l = 1; l <= n; ++l)
        if (sizes[l] <= 0 || sizes[l] % 128) return ewf_fail(EWF_ERR_ARG, "%s: layer widths must be multiples of 128 (got %d)", what, sizes[l]);
    return EWF_OK;
}
bool misaligned(const void *p) { return ((uintptr_t)p & 15) != 0; }
}  // namespace

extern "C" int ewf_mlp_forward(int32_t n, const int32_t *sizes, const void *X, const void *const *W, const float *const *b,
                               void *const *H, float *const *P, float *Y, int32_t M, void *stream)
{
    int st = check_net("forward", n, sizes, M, 32);
    if (st) return st;
    if (!X || !W || !b || !Y || (n > 1 && !H)) return ewf_fail(EWF_ERR_ARG, "forward: NULL argument");
    for (int l = 0; l < n; ++l) {
        const void *in = l ? H[l - 1] : X;
        const bool last = l == n - 1;
        Product o;
        o.A = in;
        o.B = W[l];
        o.M = M;
        o.N = sizes[l + 1];
        o.K = sizes[l];
        o.bias = b[l];
        o.f32 = last ? Y : nullptr;
        o.bf16 = last ? nullptr : H[l];
        o.pre = last || !P ? nullptr : P[l];
        o.act = last ? 0 : ACT_GELU;
        if (!in || !W[l] || (!last && (!H[l] || (P && !P[l])))) return ewf_fail(EWF_ERR_ARG, "forward: NULL buffer of layer %d", l);
        if (misaligned(in) || misaligned(W[l]) || misaligned(o.f32) || misaligned(o.bf16) || misaligned(o.pre))
            return ewf_fail(EWF_ERR_ARG, "forward: buffers of layer %d must be 16-byte aligned", l);
        if ((st = gemm_one(o, (cudaStream_t)stream))) return st;
    }
    return EWF_OK;
}

extern "C" int ewf_mlp_backward(int32_t n, const int32_t *sizes, const void *const *H, const void *const *W, const float *const *P,
                                void *const *dY, float *const *gW, float *const *gb, int32_t M, void *stream)
{
    int st = check_net("backward", n, sizes, M, 128);
    if (st) return st;
    if (M % 128) return ewf_fail(EWF_ERR_ARG, "backward: the batch must be a multiple of 128 (got %d)", M);
    if (!H || !W || !dY || !gW || !gb || (n > 1 && !P)) return ewf_fail(EWF_ERR_ARG, "backward: NULL argument");
    for (int l = 0; l < n; ++l) {
        if (!H[l] || !W[l] || !dY[l] || !gW[l] || !gb[l] || (l < n - 1 && !P[l])) return ewf_fail(EWF_ERR_ARG, "backward: NULL buffer of layer %d", l);
        if (misaligned(H[l]) || misaligned(W[l]) || misaligned(dY[l]) || misaligned(gW[l]) || (l < n - 1 && misaligned(P[l])))
            return ewf_fail(EWF_ERR_ARG, "backward: buffers of layer %d must be 16-byte aligned", l);
    }
    const cudaStream_t s = (cudaStream_t)stream;
    for (int l = n - 1; l >= 0; --l) {
        Product gw;  // gW[nout, nin] = dY[M, nout]^T . H[M, nin]
        gw.A = dY[l];
        gw.B = H[l];
        gw.ta = gw.tb = true;
        gw.M = sizes[l + 1];
        gw.N = sizes[l];
        gw.K = M;
        gw.f32 = gW[l];
        if (l == 0) {
            if ((st = gemm_one(gw, s))) return st;
            break;
        }
        Product dh;  // dY of the layer before: (dY[M, nout] . W[nout, nin]) GELU'(P)
        dh.A = dY[l];
        dh.B = W[l];
        dh.tb = true;
        dh.M = M;
        dh.N = sizes[l];
        dh.K = sizes[l + 1];
        dh.bf16 = dY[l - 1];
        dh.gpre = P[l - 1];
        dh.act = ACT_GRAD;
        if ((st = gemm_pair(dh, gw, s))) return st;
    }
    // every layer's bias gradient, BIAS_GROUP layers at a time
    for (int l0 = 0; l0 < n; l0 += BIAS_GROUP) {
        BiasJobs bj;
        memset(&bj, 0, sizeof(bj));
        int blocks = 0;
        bj.n = n - l0 < BIAS_GROUP ? n - l0 : BIAS_GROUP;
        bj.M = M;
        for (int q = 0; q < bj.n; ++q) {
            bj.dy[q] = (const __nv_bfloat16 *)dY[l0 + q];
            bj.db[q] = gb[l0 + q];
            bj.N[q] = sizes[l0 + q + 1];
            bj.block0[q] = blocks;
            blocks += sizes[l0 + q + 1] / 64;
        }
        if ((st = launch_pdl("bias_grad launch", k_bias_grads, dim3(blocks), dim3(1024), 0, s, bj))) return st;
    }
    return EWF_OK;
}

extern "C" int ewf_mlp_mse_loss(const float *y, const float *t, void *dy, size_t n, float scale, float *part, int32_t nblocks, void *done,
                                float *loss, void *stream)
{
    if (!y || !t || !dy || !part || !done || !loss || nblocks < 1 || n == 0 || n % 4) return ewf_fail(EWF_ERR_ARG, "mse_loss: bad argument");
    if (misaligned(y) || misaligned(t) || ((uintptr_t)dy & 7)) return ewf_fail(EWF_ERR_ARG, "mse_loss: misaligned");
    return launch_pdl("mse_loss launch", k_mse_loss, dim3(nblocks), dim3(256), 0, (cudaStream_t)stream, (const float4 *)y, (const float4 *)t,
                      (uint2 *)dy, n / 4, scale, part, (unsigned *)done, loss);
}

extern "C" int ewf_mlp_adam_all(int32_t count, float *const *w, float *const *m, float *const *v, const float *const *g, void *const *wb,
                                const size_t *n, const float *wd, float lr, float b1, float b2, float eps, int32_t step, void *stream)
{
    if (count < 1 || !w || !m || !v || !g || !wb || !n || !wd || step < 1) return ewf_fail(EWF_ERR_ARG, "adam: bad argument");
    for (int q = 0; q < count; ++q) {
        if (!w[q] || !m[q] || !v[q] || !g[q]) return ewf_fail(EWF_ERR_ARG, "adam: NULL tensor %d", q);
    }
    // tensors off 16 bytes (parameters that are views into one buffer), or of 2^31 elements and more, by the kernel of one element a thread
    auto alone = [&](int q) {
        return misaligned(w[q]) || misaligned(m[q]) || misaligned(v[q]) || misaligned(g[q]) || ((uintptr_t)wb[q] & 7) || n[q] >= (1ull << 31);
    };
    for (int q0 = 0; q0 < count;) {
        if (alone(q0)) {
            const int st = n[q0] ? ewf_mlp_adam(w[q0], m[q0], v[q0], g[q0], wb[q0], n[q0], lr, b1, b2, eps, step, wd[q0], stream) : EWF_OK;
            if (st) return st;
            ++q0;
            continue;
        }
        AdamJobs J;
        memset(&J, 0, sizeof(J));
        unsigned blocks = 0;
        int q = q0;
        for (; q < count && J.njobs < ADAM_GROUP && !alone(q); ++q) {
            const int e = J.njobs++;
            J.w[e] = w[q];
            J.m[e] = m[q];
            J.v[e] = v[q];
            J.g[e] = g[q];
            J.wb[e] = (__nv_bfloat16 *)wb[q];
            J.n[e] = (unsigned)n[q];
            J.wd[e] = wd[q];
            J.block0[e] = blocks;
            blocks += (unsigned)((n[q] + ADAM_BLOCK - 1) / ADAM_BLOCK);
        }
        J.lr = lr;
        J.b1 = b1;
        J.b2 = b2;
        J.eps = eps;
        J.c1 = 1.f - powf(b1, (float)step);
        J.c2 = 1.f - powf(b2, (float)step);
        q0 = q;
        if (blocks == 0) continue;
        const int st = launch_pdl("adam launch", k_adam_all, dim3(blocks), dim3(256), 0, (cudaStream_t)stream, J);
        if (st) return st;
    }
    return EWF_OK;
}

extern "C" int ewf_mlp_status(void)
{
    int e = 0;
    cudaError_t ce = cudaMemcpyFromSymbol(&e, g_umma_err, sizeof(int));
    if (ce != cudaSuccess) return check(ce, "gemm status");
    if (e) {
        const int zero = 0;
        cudaMemcpyToSymbol(g_umma_err, &zero, sizeof(int));
        return ewf_fail(EWF_ERR_CUDA, "gemm: an mbarrier wait gave up (outputs of that launch are invalid)");
    }
    return EWF_OK;
}

extern "C" int ewf_mlp_test_hold(int32_t tile, int32_t polls)
{
    const int h = tile >= 0 ? tile : -1;
    const int v = (tile >= 0 && polls > 0) ? polls : kWaitPolls;
    int st = check(cudaMemcpyToSymbol(g_umma_wait_limit, &v, sizeof(int)), "gemm wait limit");
    if (!st) st = check(cudaMemcpyToSymbol(g_umma_hold, &h, sizeof(int)), "gemm hold");
    return st;
}

extern "C" int ewf_mlp_transpose(const void *in, void *out, int32_t rows, int32_t cols, void *stream)
{
    if (!in || !out || rows <= 0 || cols <= 0) return ewf_fail(EWF_ERR_ARG, "transpose: bad argument");
    k_transpose<<<dim3((cols + 31) / 32, (rows + 31) / 32), dim3(32, 8), 0, (cudaStream_t)stream>>>(
        (const __nv_bfloat16 *)in, (__nv_bfloat16 *)out, rows, cols);
    return check(cudaGetLastError(), "transpose launch");
}

extern "C" int ewf_mlp_gelu_grad(const void *dy, const float *pre, void *dx, size_t n, void *stream)
{
    if (!dy || !pre || !dx) return ewf_fail(EWF_ERR_ARG, "gelu_grad: NULL");
    k_gelu_grad<<<blocks_for(n), 256, 0, (cudaStream_t)stream>>>((const __nv_bfloat16 *)dy, pre, (__nv_bfloat16 *)dx, n);
    return check(cudaGetLastError(), "gelu_grad launch");
}

extern "C" int ewf_mlp_bias_grad(const void *dy, float *db, int32_t M, int32_t N, void *stream)
{
    if (!dy || !db || M <= 0 || N <= 0) return ewf_fail(EWF_ERR_ARG, "bias_grad: bad argument");
    k_bias_grad<<<(N + 255) / 256, 256, 0, (cudaStream_t)stream>>>((const __nv_bfloat16 *)dy, db, M, N);
    return check(cudaGetLastError(), "bias_grad launch");
}

// part must hold `nblocks` floats: one partial sum of squared differences per block
extern "C" int ewf_mlp_mse_grad(const float *y, const float *t, void *dy, size_t n, float scale, float *part, int32_t nblocks,
                                void *stream)
{
    if (!y || !t || !dy || !part || nblocks < 1) return ewf_fail(EWF_ERR_ARG, "mse_grad: bad argument");
    k_mse_grad<<<nblocks, 256, 0, (cudaStream_t)stream>>>(y, t, (__nv_bfloat16 *)dy, n, scale, part);
    return check(cudaGetLastError(), "mse_grad launch");
}

extern "C" int ewf_mlp_adam(float *w, float *m, float *v, const float *g, void *wb, size_t n, float lr, float b1, float b2,
                            float eps, int32_t step, float weight_decay, void *stream)
{
    if (!w || !m || !v || !g || step < 1) return ewf_fail(EWF_ERR_ARG, "adam: bad argument");
    const float c1 = 1.f - powf(b1, (float)step), c2 = 1.f - powf(b2, (float)step);
    k_adam<<<blocks_for(n), 256, 0, (cudaStream_t)stream>>>(w, m, v, g, (__nv_bfloat16 *)wb, n, lr, b1, b2, eps, c1, c2,
                                                            weight_decay);
    return check(cudaGetLastError(), "adam launch");
}

extern "C" int ewf_mlp_combine(const float *R, const float *G, float *out, int32_t M, int32_t nout, int32_t nin, int32_t T,
                               void *stream)
{
    if (!R || !G || !out || M <= 0 || nout <= 0 || nin <= 0 || T <= 0) return ewf_fail(EWF_ERR_ARG, "combine: bad argument");
    if (M > 65535) return ewf_fail(EWF_ERR_ARG, "combine: at most 65535 samples per call (got %d)", M);
    if ((long long)nout * nin > COMBINE_MAX)
        return ewf_fail(EWF_ERR_ARG, "combine: nout * nin must be <= %d (got %d x %d)", COMBINE_MAX, nout, nin);
    launch_combine<1>(R, G, out, M, nout, nin, T, (cudaStream_t)stream);
    return check(cudaGetLastError(), "combine launch");
}
