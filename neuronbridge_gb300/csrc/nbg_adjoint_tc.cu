// nbg_adjoint_tc.cu -- the recurrent product of the adjoint on tcgen05
// (C ABI in include/nbg_adjoint.h).
//
// Each adjoint step needs g_ext[b][i] = sum_j dI[b][j] W_rec[i][j], a GEMM of
// B = 128 rows by N by N.  As cuBLAS FP32 it takes about 24 us at N = 1024;
// here it runs on the tensor cores in split BF16:
//   x = x_hi + x_lo,  x_hi = bf16(x),  x_lo = bf16(x - x_hi)
//   dI W^T ~= dI_hi W_hi^T + dI_hi W_lo^T + dI_lo W_hi^T      (FP32 accumulation)
// which keeps about 16 mantissa bits of each operand (the dropped term
// dI_lo W_lo^T is below 2^-16 of the product).
//
// Operands use the UMMA blocked K-major layout of nbg_umma.cuh: A = W (rows
// i, K = j), tiled once per backward by nbg_adjoint_rec_prepare; B = dI
// (rows b, K = j), written tiled by the adjoint step itself
// (nbg_lif_adjoint_step_split).  One CTA owns 128 rows i and all 128 batch
// rows (UMMA M = N = 128, a 128-column TMEM accumulator) over one K range;
// the split-K partials go to g_parts[ks] and the next adjoint step adds them
// in a fixed order, so the backward stays deterministic.
//
// The weight gradients of a checkpoint segment, dW_rec = sum_t S_{t-1}^T dI_t
// and dW_in = sum_t X_t^T dI_t, are the same kind of product with K = the
// segment's (step, batch row) pairs: D[j][n] = sum_K dI^T[j][K] B[n][K] with
// dI^T split (two products) and B = S^T or X^T exact in BF16 (spikes are 0 or
// 1).  nbg_adjoint_blocked_t lays the [L][B][R] FP32 arrays out transposed
// and blocked, nbg_adjoint_wgrad runs the tcgen05 product (UMMA M = 128 rows
// j, N = 256 columns n, split-K partials stored as [split][n][j] so the
// stores are coalesced along j), and nbg_adjoint_reduce_add adds the
// partials into the gradient in a fixed order.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "nbg_adjoint.h"
#include "nbg_common.cuh"
#include "nbg_lif_grad.cuh"
#include "nbg_umma.cuh"

namespace {

using namespace umma;

constexpr int kAdjM = 128, kAdjN = 128;
constexpr int kAdjStages = 3;
constexpr int kAdjBlockA = kAdjM * kKChunk * 2; // 16 KiB per operand block
constexpr int kAdjBlockB = kAdjN * kKChunk * 2;
constexpr int kAdjStageBytes = 2 * kAdjBlockA + 2 * kAdjBlockB; // A_hi A_lo B_hi B_lo
constexpr int kAdjSmemBytes = kAdjStages * kAdjStageBytes + 1024 + 256;
constexpr int kAdjTmemCols = 128;
constexpr int kThreads = 256; // of a product whose result is stored

// kind::f16 instruction descriptor: BF16 x BF16 -> F32, K-major, M = N = 128.
constexpr uint32_t kAdjIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kAdjN >> 3) << 17) |
                               ((uint32_t)(kAdjM >> 4) << 24);

// Element (r, c) of a rows x cols matrix in the blocked layout of 128-row x
// 64-column blocks, block (r / 128, c / 64) at ((r / 128) * (cols / 64) +
// c / 64) blocks.
__device__ __forceinline__ size_t blocked_index(int r, int c, int cols) {
    const size_t blk = (size_t)(r >> 7) * (size_t)(cols >> 6) + (size_t)(c >> 6);
    return blk * (size_t)(kAdjM * kKChunk) + block_offset(r & 127, c & 63) / 2;
}

__device__ __forceinline__ void split_bf16(float x, __nv_bfloat16 &hi, __nv_bfloat16 &lo) {
    hi = __float2bfloat16_rn(x);
    lo = __float2bfloat16_rn(x - __bfloat162float(hi));
}

__global__ void k_split_blocked(const float *__restrict__ x, __nv_bfloat16 *__restrict__ hi,
                                __nv_bfloat16 *__restrict__ lo, int rows, int cols) {
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (long long)rows * cols) return;
    const int r = (int)(idx / cols), c = (int)(idx % cols);
    const size_t o = blocked_index(r, c, cols);
    split_bf16(x[idx], hi[o], lo[o]);
}

// The adjoint step of k_lif_adj (nbg_adjoint.cu) with g_ext the fixed-order
// sum of the split-K partials, writing dI also as the split BF16 B operand.
__global__ void __launch_bounds__(256) k_lif_adj_split(
    const float *__restrict__ g_parts, int n_parts, const float *__restrict__ g_read, float c_t,
    const float *__restrict__ u, const float *__restrict__ s, const unsigned char *__restrict__ m,
    const float *__restrict__ vprev, float *__restrict__ lam_v, float *__restrict__ dI,
    __nv_bfloat16 *__restrict__ dI_hi, __nv_bfloat16 *__restrict__ dI_lo, float *__restrict__ g_theta,
    float *__restrict__ g_alpha, const float *__restrict__ alpha, const float *__restrict__ theta,
    nbg_lif_grad_params p, int N, int total) {
    // programmatic dependent launch: the product that follows may start its
    // prologue (and its W tiles) while this step runs; this step reads
    // g_parts and lam_v only after the product before it has finished
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= total) return;
    const int j = idx % N;
    const float uu = u[idx], ss = s[idx], lv = lam_v[idx];
    const float th = theta[j];
    const float dsdu = p.smooth ? p.slope * ss * (1.0f - ss) : surrogate(uu - th, p.slope);
    float gs = c_t * g_read[idx] - lv * (uu - p.v_reset);
    if (g_parts) {
        float ge = g_parts[idx];
        for (int q = 1; q < n_parts; ++q) ge = ge + g_parts[(size_t)q * total + idx];
        gs = gs + ge;
    }
    const float gu = gs * dsdu + lv * (1.0f - ss);
    const float gm = m[idx] ? gu : 0.0f;
    dI[idx] = gm;
    const size_t o = blocked_index(idx / N, j, N);
    split_bf16(gm, dI_hi[o], dI_lo[o]);
    lam_v[idx] = gm * (1.0f - alpha[j]);
    g_theta[idx] = g_theta[idx] - gs * dsdu;
    g_alpha[idx] = g_alpha[idx] + gm * (p.v_rest - vprev[idx]);
}

// g_parts[ks][b][i] = sum over the K chunks of split ks of the three split
// products.  Grid (N / 128, split), 256 threads: warp 0 lane 0 produces
// (bulk copies into kAdjStages stages), warp 1 lane 0 issues the MMAs, warp 2
// owns the TMEM allocation, all 8 warps run the epilogue.  Every mbarrier
// wait is bounded; on expiry the CTA records kUmmaTimeout in *err, stops,
// frees its TMEM and returns.
__global__ void __launch_bounds__(kThreads, 1)
    k_adj_umma(const __nv_bfloat16 *__restrict__ w_hi, const __nv_bfloat16 *__restrict__ w_lo,
               const __nv_bfloat16 *__restrict__ d_hi, const __nv_bfloat16 *__restrict__ d_lo,
               float *__restrict__ g_parts, int n, int split, int *__restrict__ err) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t *stages = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t *full = (uint64_t *)(stages + kAdjStages * kAdjStageBytes);
    uint64_t *empty = full + kAdjStages;
    uint64_t *done = empty + kAdjStages;
    uint32_t *tmem_slot = (uint32_t *)(done + 1);
    volatile int *abort = (volatile int *)(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int mt = blockIdx.x, ks = blockIdx.y;
    const int kchunks = n / kKChunk;
    const int per = kchunks / split;
    const int kc0 = ks * per;
    const int iters = (ks == split - 1) ? kchunks - kc0 : per;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kAdjStages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        mbar_init(done, 1);
        *abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 2) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tmem_slot)),
                     "r"(kAdjTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = *tmem_slot;

    // Programmatic dependent launch: the set-up above overlaps the launch
    // before, whatever that is (the adjoint step that writes dI, or the kernel
    // that writes W); only the wait makes what it wrote visible.
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (warp == 0 && lane == 0) { // producer
        for (int it = 0; it < iters; ++it) {
            const int s = it % kAdjStages;
            if (it >= kAdjStages && !mbar_wait(&empty[s], ((it / kAdjStages) & 1) ^ 1, abort)) break;
            uint8_t *st = stages + s * kAdjStageBytes;
            const int kc = kc0 + it;
            const size_t a_blk = (size_t)mt * kchunks + kc;
            mbar_expect_tx(&full[s], kAdjStageBytes);
            bulk_copy(st, (const uint8_t *)w_hi + a_blk * kAdjBlockA, kAdjBlockA, &full[s]);
            bulk_copy(st + kAdjBlockA, (const uint8_t *)w_lo + a_blk * kAdjBlockA, kAdjBlockA, &full[s]);
            bulk_copy(st + 2 * kAdjBlockA, (const uint8_t *)d_hi + (size_t)kc * kAdjBlockB, kAdjBlockB, &full[s]);
            bulk_copy(st + 2 * kAdjBlockA + kAdjBlockB, (const uint8_t *)d_lo + (size_t)kc * kAdjBlockB, kAdjBlockB,
                      &full[s]);
        }
    } else if (warp == 1 && lane == 0) { // MMA issuer
        for (int it = 0; it < iters; ++it) {
            const int s = it % kAdjStages;
            if (!mbar_wait(&full[s], (it / kAdjStages) & 1, abort)) break;
            fence_after();
            const uint32_t a_hi = smem_addr(stages + s * kAdjStageBytes);
            const uint32_t a_lo = a_hi + kAdjBlockA;
            const uint32_t b_hi = a_hi + 2 * kAdjBlockA;
            const uint32_t b_lo = b_hi + kAdjBlockB;
#pragma unroll
            for (int k = 0; k < kKChunk / 16; ++k) {
                mma(tmem, make_desc(a_hi + 256 * k), make_desc(b_hi + 256 * k), kAdjIdesc, (it | k) != 0);
                mma(tmem, make_desc(a_lo + 256 * k), make_desc(b_hi + 256 * k), kAdjIdesc, 1u);
                mma(tmem, make_desc(a_hi + 256 * k), make_desc(b_lo + 256 * k), kAdjIdesc, 1u);
            }
            commit(&empty[s]);
        }
        commit(done);
    }
    __syncwarp();
    // epilogue: warp w reads TMEM lanes 32*(w%4).. (rows i) and columns
    // 64*(w/4).. (batch rows b)
    mbar_wait(done, 0, abort);
    __syncthreads();
    fence_after();
    const int q = warp & 3, h = warp >> 2;
    const int i = mt * kAdjM + 32 * q + lane;
    if (!*abort) {
        float *out = g_parts + (size_t)ks * kAdjN * n;
#pragma unroll
        for (int c16 = 0; c16 < 4; ++c16) {
            float acc[16];
            tmem_ld16(tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)(64 * h + 16 * c16), acc);
#pragma unroll
            for (int c = 0; c < 16; ++c) out[(size_t)(64 * h + 16 * c16 + c) * n + i] = acc[c];
        }
    }
    fence_before();
    __syncthreads();
    if (threadIdx.x == 0 && *abort) atomicOr(err, kUmmaTimeout);
    if (warp == 2) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kAdjTmemCols)
                     : "memory");
    }
}

// One adjoint step in one launch: the recurrent product of step t + 1 and
// the adjoint step t that consumes it.  Grid (N / 128, kAdjCluster) in
// clusters of kAdjCluster CTAs along y: the CTAs of a cluster split the K
// range of one 128-row tile of W exactly as k_adj_umma's split-K does
// (cluster rank = split index) and run the same three split products into
// TMEM.  Rank r owns batch rows [16 r, 16 r + 16) of the tile: every CTA
// stores its partial of those rows into rank r's part of the workspace (kParts)
// or straight into its receive buffer through distributed shared memory, which
// waits for nothing.  After one cluster barrier rank r adds the partials of ranks
// 0..7 in order -- the sum k_lif_adj_split forms from g_parts, so the result is
// the same bit for bit -- and runs the
// adjoint step on those elements, writing dI_t as the split
// BF16 operand of the next step's product into the other of two buffers
// (the next launch reads this one while writing its own), in FP32 (when dI
// is given) and as the split BF16 operand of the weight gradients (when dT_hi
// is given: dI^T, row i, column k_off + b of a k_cols-column blocked matrix,
// four consecutive b of one i per 8-byte store).  No CTA reads another's
// shared memory, so none waits for its peers before it exits.  Waits on
// mbarriers are bounded as in k_adj_umma; a CTA that gives up still takes
// part in the cluster barrier, and the error word marks the step's results
// invalid.  Without kParts, two pipeline stages (a CTA has two K chunks at
// N = 1024) leave room for the receive buffer.
//
// What bounds it: the chain from the operands to the next step's (1,000 dependent
// steps in a sweep of 1,000): at N = 1024 hand-over 1.2 us, copies and products
// 1.7, the exchange, the tail.  With eight warps, eight rows a thread, and all of
// the step's arithmetic behind the products, the tail was 1.4 us and a forward and
// backward of 1,000 steps of 128 x 1,024 took 11.24 ms; as below 10.85.  An SM
// moves about 12 bytes a clock through distributed shared memory, so the exchange
// of 64 KiB a CTA took 3.3 us; through the L2 (4 MiB of partials, which stay
// there) 9.95 ms; half of it either way 10.05.
constexpr int kAdjCluster = 8;
// pipeline stages, and the shared memory: with the partials in global memory
// (kParts) there is no receive buffer
template <bool kParts> constexpr int adj_stages() { return kParts ? 3 : 2; }
// sixteen warps run the step's tail, four batch rows a thread; the producer and
// the issuer are warps of their own
constexpr int kAdjTailWarps = 16, kAdjStepThreads = 32 * (kAdjTailWarps + 2);
// receive buffer [source rank][row / 4][i][row % 4]: a thread's sixteen
// partials of one i are four 16-byte stores, and a warp's 32 of one of them are
// contiguous (stores of the same size 80 bytes apart, free of bank conflicts
// but scattered over packets, cost 2.6 us a step)
constexpr int kAdjRecvBytes = kAdjN * kAdjM * 4;
template <bool kParts> constexpr int adj_smem() {
    return adj_stages<kParts>() * kAdjStageBytes + (kParts ? 0 : kAdjRecvBytes) + 1024 + 256;
}

template <bool kParts>
__global__ void __cluster_dims__(1, kAdjCluster, 1) __launch_bounds__(kAdjStepThreads, 1) k_adj_step_umma(
    const __nv_bfloat16 *__restrict__ w_hi, const __nv_bfloat16 *__restrict__ w_lo,
    const __nv_bfloat16 *__restrict__ d_hi_in, const __nv_bfloat16 *__restrict__ d_lo_in,
    __nv_bfloat16 *__restrict__ d_hi_out, __nv_bfloat16 *__restrict__ d_lo_out, const float *__restrict__ g_read,
    float c_t, const float *__restrict__ u, const float *__restrict__ s, const unsigned char *__restrict__ m,
    const float *__restrict__ vprev, float *__restrict__ lam_v, float *__restrict__ dI, float *__restrict__ g_theta,
    float *__restrict__ g_alpha, const float *__restrict__ alpha, const float *__restrict__ theta,
    nbg_lif_grad_params p, int n, __nv_bfloat16 *__restrict__ dT_hi, __nv_bfloat16 *__restrict__ dT_lo,
    long long k_off, long long k_cols, float4 *parts, int *__restrict__ err) {
    constexpr int kStages = adj_stages<kParts>();
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t *stages = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    float4 *recv = reinterpret_cast<float4 *>(stages + kStages * kAdjStageBytes); // kAdjRecvBytes, or parts
    uint64_t *full = (uint64_t *)((uint8_t *)recv + (kParts ? 0 : kAdjRecvBytes));
    uint64_t *empty = full + kStages;
    uint64_t *done = empty + kStages;
    uint32_t *tmem_slot = (uint32_t *)(done + 1);
    volatile int *abort = (volatile int *)(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint32_t rank;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    const int mt = blockIdx.x, ks = (int)rank;
    const int kchunks = n / kKChunk;
    const int per = kchunks / kAdjCluster;
    const int kc0 = ks * per;
    const int iters = (ks == kAdjCluster - 1) ? kchunks - kc0 : per;

    if (threadIdx.x == 0) {
        for (int st = 0; st < kStages; ++st) {
            mbar_init(&full[st], 1);
            mbar_init(&empty[st], 1);
        }
        mbar_init(done, 1);
        *abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 2) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tmem_slot)),
                     "r"(kAdjTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = *tmem_slot;

    // Programmatic dependent launch of a step that follows another of its sweep
    // (`chained` on the host): W is constant during the sweep, so the first
    // stages' W tiles are requested before the wait for the previous step (which
    // writes dI_{t+1}, lam_v and the gradients).  The kernels that write W and
    // the record have ended before a sweep's or a replayed segment's first step
    // starts, since that one is launched without the attribute.
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if constexpr (!kParts) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    if (warp == kAdjTailWarps && lane == 0) { // producer
        const int pre = iters < kStages ? iters : kStages;
        for (int it = 0; it < pre; ++it) {
            uint8_t *st = stages + it * kAdjStageBytes;
            const size_t a_blk = (size_t)mt * kchunks + kc0 + it;
            mbar_expect_tx(&full[it], kAdjStageBytes);
            bulk_copy(st, (const uint8_t *)w_hi + a_blk * kAdjBlockA, kAdjBlockA, &full[it]);
            bulk_copy(st + kAdjBlockA, (const uint8_t *)w_lo + a_blk * kAdjBlockA, kAdjBlockA, &full[it]);
        }
        asm volatile("griddepcontrol.wait;" ::: "memory");
        for (int it = 0; it < pre; ++it) {
            uint8_t *st = stages + it * kAdjStageBytes;
            const int kc = kc0 + it;
            bulk_copy(st + 2 * kAdjBlockA, (const uint8_t *)d_hi_in + (size_t)kc * kAdjBlockB, kAdjBlockB, &full[it]);
            bulk_copy(st + 2 * kAdjBlockA + kAdjBlockB, (const uint8_t *)d_lo_in + (size_t)kc * kAdjBlockB,
                      kAdjBlockB, &full[it]);
        }
        for (int it = pre; it < iters; ++it) {
            const int st_i = it % kStages;
            if (!mbar_wait(&empty[st_i], ((it / kStages) & 1) ^ 1, abort)) break;
            uint8_t *st = stages + st_i * kAdjStageBytes;
            const int kc = kc0 + it;
            const size_t a_blk = (size_t)mt * kchunks + kc;
            mbar_expect_tx(&full[st_i], kAdjStageBytes);
            bulk_copy(st, (const uint8_t *)w_hi + a_blk * kAdjBlockA, kAdjBlockA, &full[st_i]);
            bulk_copy(st + kAdjBlockA, (const uint8_t *)w_lo + a_blk * kAdjBlockA, kAdjBlockA, &full[st_i]);
            bulk_copy(st + 2 * kAdjBlockA, (const uint8_t *)d_hi_in + (size_t)kc * kAdjBlockB, kAdjBlockB, &full[st_i]);
            bulk_copy(st + 2 * kAdjBlockA + kAdjBlockB, (const uint8_t *)d_lo_in + (size_t)kc * kAdjBlockB,
                      kAdjBlockB, &full[st_i]);
        }
    } else if (warp == kAdjTailWarps + 1 && lane == 0) { // MMA issuer
        for (int it = 0; it < iters; ++it) {
            const int st_i = it % kStages;
            if (!mbar_wait(&full[st_i], (it / kStages) & 1, abort)) break;
            fence_after();
            const uint32_t a_hi = smem_addr(stages + st_i * kAdjStageBytes);
            const uint32_t a_lo = a_hi + kAdjBlockA;
            const uint32_t b_hi = a_hi + 2 * kAdjBlockA;
            const uint32_t b_lo = b_hi + kAdjBlockB;
#pragma unroll
            for (int k = 0; k < kKChunk / 16; ++k) {
                mma(tmem, make_desc(a_hi + 256 * k), make_desc(b_hi + 256 * k), kAdjIdesc, (it | k) != 0);
                mma(tmem, make_desc(a_lo + 256 * k), make_desc(b_hi + 256 * k), kAdjIdesc, 1u);
                mma(tmem, make_desc(a_hi + 256 * k), make_desc(b_lo + 256 * k), kAdjIdesc, 1u);
            }
            commit(&empty[st_i]);
        }
        commit(done);
    }
    __syncwarp();
    // this thread's share of the adjoint step: batch rows 16 ks + 4 bsub + k
    // of column i (four consecutive rows: one 8-byte store of dI^T).  What needs
    // no product is done while the products run: first what no adjoint step
    // writes (the forward's record, g_read and the parameters, all complete
    // before the first step of the sweep), before the wait for the previous
    // step, then the accumulators that step updated.
    const bool tail = warp < kAdjTailWarps;
    const int il = threadIdx.x & 127, bsub = threadIdx.x >> 7;
    const int i = mt * kAdjM + il;
    constexpr int kRows = 4;
    float op_u[kRows], op_ds[kRows], op_ns[kRows], op_lv[kRows], op_gr[kRows], op_gt[kRows], op_ga[kRows], op_vp[kRows];
    unsigned char op_m[kRows];
    float th = 0.0f, al = 0.0f;
    if (tail) {
        th = theta[i];
        al = alpha[i];
#pragma unroll
        for (int k = 0; k < kRows; ++k) {
            const size_t idx = (size_t)(16 * ks + 4 * bsub + k) * n + i;
            op_u[k] = u[idx];
            op_ns[k] = s[idx];
            op_gr[k] = g_read[idx];
            op_vp[k] = vprev[idx];
            op_m[k] = m[idx];
        }
#pragma unroll
        for (int k = 0; k < kRows; ++k) {
            const float ss = op_ns[k];
            op_ds[k] = p.smooth ? p.slope * ss * (1.0f - ss) : surrogate(op_u[k] - th, p.slope);
            op_ns[k] = 1.0f - ss;
            op_gr[k] = c_t * op_gr[k];
            op_u[k] = op_u[k] - p.v_reset;
            op_vp[k] = p.v_rest - op_vp[k];
        }
    }
    asm volatile("griddepcontrol.wait;" ::: "memory"); // the previous step's writes are visible
    if (tail) {
#pragma unroll
        for (int k = 0; k < kRows; ++k) {
            const size_t idx = (size_t)(16 * ks + 4 * bsub + k) * n + i;
            op_lv[k] = lam_v[idx];
            op_gt[k] = g_theta[idx];
            op_ga[k] = g_alpha[idx];
        }
#pragma unroll
        for (int k = 0; k < kRows; ++k) {
            op_gr[k] = op_gr[k] - op_lv[k] * op_u[k];
            op_ns[k] = op_lv[k] * op_ns[k];
        }
    }
    mbar_wait(done, 0, abort);
    __syncthreads();
    fence_after();
    if constexpr (!kParts) asm volatile("barrier.cluster.wait.aligned;" ::: "memory"); // the receiving CTAs have started
    // the partial accumulator to the rows' owners: warp w holds rows
    // i = 32 (w % 4) + lane and batch columns b = 32 (w / 4) + 16 c16 + c,
    // which rank 2 (w / 4) + c16 owns; they land in its receive buffer at
    // [this rank][c][i]
    constexpr int kRecv = kAdjCluster * 4 * kAdjM; // 16-byte pieces a rank receives
    if (tail && !*abort) {
        const int q = warp & 3, g = warp >> 2;
        const int mine = ks * 4 * kAdjM + il;
#pragma unroll
        for (int c16 = 0; c16 < 2; ++c16) {
            float acc[16];
            tmem_ld16(tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)(32 * g + 16 * c16), acc);
            const int to = 2 * g + c16;
            if constexpr (kParts) {
                float4 *out = parts + ((size_t)mt * kAdjCluster + to) * kRecv + mine;
#pragma unroll
                for (int c = 0; c < 16; c += 4)
                    __stcg(out + c / 4 * kAdjM, make_float4(acc[c], acc[c + 1], acc[c + 2], acc[c + 3]));
            } else {
                uint32_t ra;
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(smem_addr(recv + mine)), "r"(to));
#pragma unroll
                for (int c = 0; c < 16; c += 4)
                    asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(ra + (uint32_t)(c / 4 * kAdjM * 16)),
                                 "f"(acc[c]), "f"(acc[c + 1]), "f"(acc[c + 2]), "f"(acc[c + 3])
                                 : "memory");
            }
        }
    }
    fence_before();
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    // reduce this rank's batch rows over the cluster's partials, in rank
    // order, and run the adjoint step on them
    if (tail) {
        // every partial of the thread's rows, loaded back to back, then added
        // in rank order
        float x[kAdjCluster][kRows];
#pragma unroll
        for (int r = 0; r < kAdjCluster; ++r) {
            const int at = (r * 4 + bsub) * kAdjM + il;
            *reinterpret_cast<float4 *>(x[r]) =
                kParts ? __ldcg(parts + ((size_t)mt * kAdjCluster + ks) * kRecv + at) : recv[at];
        }
        uint32_t t_hi[kRows / 2], t_lo[kRows / 2]; // dI^T of the rows, split, packed in pairs
#pragma unroll
        for (int k = 0; k < kRows; ++k) {
            const int b = 16 * ks + 4 * bsub + k;
            float ge = x[0][k];
#pragma unroll
            for (int r = 1; r < kAdjCluster; ++r) ge = ge + x[r][k];
            const size_t idx = (size_t)b * n + i;
            const float gs = op_gr[k] + ge;
            const float gu = gs * op_ds[k] + op_ns[k];
            const float gm = op_m[k] ? gu : 0.0f;
            if (dI) dI[idx] = gm;
            const size_t o = blocked_index(b, i, n);
            __nv_bfloat16 h, l;
            split_bf16(gm, h, l);
            d_hi_out[o] = h;
            d_lo_out[o] = l;
            const uint32_t hb = __bfloat16_as_ushort(h), lb = __bfloat16_as_ushort(l);
            if (k & 1) {
                t_hi[k >> 1] |= hb << 16;
                t_lo[k >> 1] |= lb << 16;
            } else {
                t_hi[k >> 1] = hb;
                t_lo[k >> 1] = lb;
            }
            lam_v[idx] = gm * (1.0f - al);
            g_theta[idx] = op_gt[k] - gs * op_ds[k];
            g_alpha[idx] = op_ga[k] + gm * op_vp[k];
        }
        if (dT_hi) {
            const size_t o = blocked_index(i, (int)(k_off + 16 * ks + 4 * bsub), (int)k_cols);
            reinterpret_cast<uint2 *>(dT_hi + o)[0] = make_uint2(t_hi[0], t_hi[1]);
            reinterpret_cast<uint2 *>(dT_lo + o)[0] = make_uint2(t_lo[0], t_lo[1]);
        }
    }
    if (threadIdx.x == 0 && *abort) atomicOr(err, kUmmaTimeout);
    if (warp == 2) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kAdjTmemCols)
                     : "memory");
    }
}

// The adjoint steps of a whole segment in one cooperative launch: the products,
// partial sums and step of k_adj_step_umma, so the same results bit for bit, with
// the loop over the steps inside.  Between two launches a step waited for the last
// CTA of the one before, for its writes and for its own set-up; here the CTAs
// stay: lam_v and the gradients are registers, W stays in shared memory where a
// CTA's chunks have a stage each, the next step's operands are on their way during
// this one, and a CTA's product waits only for the dI that its K range reads.
//
// Split: 32 batch rows of a 128-row tile of W are a chain of their own, run by a
// cluster of four CTAs with two of the eight K ranges each (two accumulators): at
// N = 1024 32 clusters, of which 36 fit on 152 SMs (15 of eight CTAs).  Below 512
// neurons there are as many ranges as chunks, as in the two-launch form.  A CTA sends
// its peers 24 KiB of partials a step through distributed shared memory and reads
// 32 KiB of dI, half of what the step launch moves.
//
// What bounds it: the latency of two exchanges a step, that of the partials in the
// cluster and that of dI through the L2 (publish, poll, copy: about 2 us).  Forward
// and backward of 1,000 steps of 128 x 1,024: 9.97 ms with a launch a step, 9.45
// in one launch with clusters of eight (64 CTAs, partials through the L2), 9.53 as
// here but through the L2, 9.31 as here.  400 steps at 384 neurons: 3.94 ms with two
// launches a step, 3.02 as here.
//
// Order.  The product of step j overwrites the accumulators after `exchanged` of
// step j - 1, which comes after their last read.  The receive buffers alternate,
// since a CTA may be a step ahead of a peer that still reads; it cannot be two
// ahead (`exchanged` between).  `exchanged` alternates too: its arrivals are
// counted, not named, and a CTA that has all of step j may arrive for step j + 1
// at a peer that still lacks a third one's of step j (at once where it has no K
// range to wait for), so with one barrier it could stand in for that one.  With
// two, its next arrival at the same barrier is that of step j + 2, after the wait
// for step j + 1, so after the peer's arrival for step j + 1, which the peer makes
// when it has all of step j.  dI alternates likewise: a CTA writes step j's into
// the buffer of step j - 2 after `exchanged` of step j, so after dI of step j - 1 of
// every tile (a cluster's K ranges cover all of them), which their CTAs wrote after
// their products had read it.
//
// The launch is cooperative, so all CTAs run at once; every wait is bounded all the
// same.  A CTA that gives up goes through the remaining steps without waiting,
// reading or publishing anything, its peers' waits run out once, and the error
// word marks the results.
constexpr int kSweepN = 32, kSweepCluster = 4, kSweepStages = 4; // batch rows of a CTA; CTAs of a cluster; pipeline stages
constexpr int kSweepParts = kAdjN / kSweepN;
constexpr int kSweepBlockB = kSweepN * kKChunk * 2; // 4 KiB
constexpr int kSweepStageBytes = 2 * kAdjBlockA + 2 * kSweepBlockB;
constexpr int kSweepTailWarps = 8, kSweepThreads = 32 * (kSweepTailWarps + 2);
constexpr uint32_t kSweepIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kSweepN >> 3) << 17) |
                                 ((uint32_t)(kAdjM >> 4) << 24);
constexpr int kReadyStride = 32; // a count has a line of its own
constexpr int kExchangeBarriers = 2; // step j's: j % 2
constexpr int kSweepRecv = kAdjCluster * 2 * kAdjM; // 16-byte pieces that a rank receives in a step
constexpr int kSweepSmemBytes = kSweepStages * kSweepStageBytes + 2 * kSweepRecv * 16 + 1024 + 256;
static_assert(kSweepSmemBytes <= 232448, "shared memory of a CTA");

__device__ __forceinline__ bool sweep_ready(const int *flag, int want, volatile int *abort) {
    const long long t0 = clock64();
    for (;;) {
        int x;
        asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(x) : "l"(flag) : "memory");
        if (x >= want) return true;
        if (*abort) return false;
        if (clock64() - t0 > kWaitCycles) {
            *abort = 1;
            return false;
        }
    }
}

// mbar_wait for what the cluster's other CTAs wrote before they arrived.
__device__ __forceinline__ bool mbar_wait_cluster(uint64_t *bar, uint32_t parity, volatile int *abort) {
    const long long t0 = clock64();
    for (;;) {
        uint32_t ok;
        asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
                     " selp.u32 %0, 1, 0, p;\n}"
                     : "=r"(ok)
                     : "r"(smem_addr(bar)), "r"(parity)
                     : "memory");
        if (ok) return true;
        if (*abort) return false;
        if (clock64() - t0 > kWaitCycles) {
            *abort = 1;
            return false;
        }
    }
}

// Waits (bounded) for a phase although the CTA has given up.
__device__ __forceinline__ void mbar_drain(uint64_t *bar, uint32_t parity) {
    const long long t0 = clock64();
    while (!mbar_try(bar, parity) && clock64() - t0 < kWaitCycles) {
    }
}

__global__ void __launch_bounds__(kSweepThreads, 1) k_adj_sweep_umma(
    const __nv_bfloat16 *__restrict__ w_hi, const __nv_bfloat16 *__restrict__ w_lo, __nv_bfloat16 *d_hi0,
    __nv_bfloat16 *d_lo0, __nv_bfloat16 *d_hi1, __nv_bfloat16 *d_lo1, const float *__restrict__ g_read,
    const float *__restrict__ coef, const float *__restrict__ u, const float *__restrict__ s,
    const unsigned char *__restrict__ m, const float *__restrict__ vprev, float *__restrict__ lam_v,
    float *__restrict__ g_theta, float *__restrict__ g_alpha, const float *__restrict__ alpha,
    const float *__restrict__ theta, nbg_lif_grad_params p, int n, int steps, int t0, int ends_run,
    __nv_bfloat16 *__restrict__ dT_hi, __nv_bfloat16 *__restrict__ dT_lo, long long k_off, long long k_cols, int *ready,
    int *__restrict__ err) {
    constexpr int kStages = kSweepStages, kRows = 4;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t *stages = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    float4 *recv = reinterpret_cast<float4 *>(stages + kStages * kSweepStageBytes); // of the even and the odd steps
    uint64_t *full_w = (uint64_t *)(recv + 2 * kSweepRecv);
    uint64_t *full_d = full_w + kStages;
    uint64_t *empty = full_d + kStages;
    uint64_t *done = empty + kStages, *exchanged = done + 1;
    uint32_t *tmem_slot = (uint32_t *)(exchanged + kExchangeBarriers);
    volatile int *abort = (volatile int *)(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint32_t rank, ranks;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(ranks));
    if (ranks != kSweepCluster) { // launched without its cluster (as a profiler may): no peer to send to
        if (threadIdx.x == 0) atomicOr(err, kUmmaTimeout);
        return;
    }
    const int mt = blockIdx.x / kSweepParts, bq = blockIdx.x % kSweepParts, ks = (int)rank;
    const int kchunks = n / kKChunk;
    // two of the K ranges, eight or as many as there are chunks; the last CTA that
    // has any takes the rest, one without runs its rows of the step alone
    const int ranges = kchunks < kAdjCluster ? kchunks : kAdjCluster;
    const int per = kchunks / ranges;
    const int kc0 = 2 * ks * per;
    const int iters = 2 * ks >= ranges ? 0 : 2 * ks + 2 == ranges ? kchunks - kc0 : 2 * per;
    const int pre = iters < kStages ? iters : kStages;

    if (threadIdx.x == 0) {
        for (int st = 0; st < kStages; ++st) {
            mbar_init(&full_w[st], 1);
            mbar_init(&full_d[st], 1);
            mbar_init(&empty[st], 1);
        }
        mbar_init(done, 1);
        for (int k = 0; k < kExchangeBarriers; ++k) mbar_init(&exchanged[k], kSweepCluster);
        *abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 2) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tmem_slot)),
                     "r"(kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = *tmem_slot;
    // the cluster's barriers are initialised
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");

    // Chunk c of step j is piece g = j * iters + c.  Where a CTA's chunks have a
    // stage each, W stays there; else piece g passes through stage g % kStages.
    const bool stay = iters <= kStages;
    auto stage = [&](int j, int c) { return stay ? c : (int)(((long long)j * iters + c) % kStages); };
    auto phase = [&](int j, int c) { return stay ? (uint32_t)j & 1u : (uint32_t)(((long long)j * iters + c) / kStages) & 1u; };
    auto exchange_phase = [](int j) { return (uint32_t)(j / kExchangeBarriers) & 1u; };
    long long sent_w = 0, sent_d = 0; // producer: pieces requested
    auto send_w = [&](int j, int c) { // once the products on the stage's last piece are done
        const long long g = (long long)j * iters + c;
        const int st_i = stage(j, c);
        if ((stay ? j > 0 : g >= kStages) && !mbar_wait(&empty[st_i], phase(j, c) ^ 1u, abort)) return false;
        sent_w = g + 1;
        if (stay && j > 0) return true;
        uint8_t *st = stages + st_i * kSweepStageBytes;
        const size_t a_blk = ((size_t)mt * kchunks + kc0 + c) * kAdjBlockA;
        mbar_expect_tx(&full_w[st_i], 2 * kAdjBlockA);
        bulk_copy(st, (const uint8_t *)w_hi + a_blk, kAdjBlockA, &full_w[st_i]);
        bulk_copy(st + kAdjBlockA, (const uint8_t *)w_lo + a_blk, kAdjBlockA, &full_w[st_i]);
        return true;
    };
    const bool tail = warp < kSweepTailWarps;
    const int il = threadIdx.x & 127, bsub = threadIdx.x >> 7;
    const int i = mt * kAdjM + il, b0 = bq * kSweepN + 8 * ks + 4 * bsub;
    float gr[kRows], lv[kRows], gt[kRows], ga[kRows], op_u[kRows], op_s[kRows], op_vp[kRows];
    unsigned char op_m[kRows];
    float th = 0.0f, al = 0.0f;
    const size_t at0 = (size_t)b0 * n + i, per_step = (size_t)kAdjN * n;
    auto operands = [&](int k) { // of step t0 + k
        const size_t at = (size_t)k * per_step + at0;
#pragma unroll
        for (int r = 0; r < kRows; ++r) {
            op_u[r] = u[at + (size_t)r * n];
            op_s[r] = s[at + (size_t)r * n];
            op_vp[r] = vprev[at + (size_t)r * n];
            op_m[r] = m[at + (size_t)r * n];
        }
    };
    if (tail) {
        th = theta[i];
        al = alpha[i];
#pragma unroll
        for (int r = 0; r < kRows; ++r) {
            gr[r] = g_read[at0 + (size_t)r * n];
            lv[r] = lam_v[at0 + (size_t)r * n];
            gt[r] = g_theta[at0 + (size_t)r * n];
            ga[r] = g_alpha[at0 + (size_t)r * n];
        }
        operands(steps - 1);
    } else if (warp == kSweepTailWarps && lane == 0) {
        for (int c = 0; c < pre; ++c) send_w(0, c);
    }
    for (int j = 0; j < steps; ++j) {
        const int k = steps - 1 - j, t = t0 + k;
        __nv_bfloat16 *const out_hi = t & 1 ? d_hi1 : d_hi0, *const out_lo = t & 1 ? d_lo1 : d_lo0;
        float4 *const got = recv + (j & 1) * kSweepRecv;
        if (warp == kSweepTailWarps) {
            if (lane == 0) { // producer
                const uint8_t *in_hi = (const uint8_t *)(t & 1 ? d_hi0 : d_hi1);
                const uint8_t *in_lo = (const uint8_t *)(t & 1 ? d_lo0 : d_lo1);
                const long long g0 = (long long)j * iters;
                for (int c = 0; c < iters && !*abort; ++c) {
                    if (g0 + c >= sent_w && !send_w(j, c)) break;
                    const int kc = kc0 + c, st_i = stage(j, c);
                    if (j > 0 && (c == 0 || kc % 2 == 0)) { // the tile's CTAs of these rows have written step j - 1's dI
                        if (!sweep_ready(ready + (kc / 2 * kSweepParts + bq) * kReadyStride, kSweepCluster * j, abort)) break;
                        asm volatile("fence.proxy.async.global;" ::: "memory");
                    }
                    uint8_t *st = stages + st_i * kSweepStageBytes;
                    const size_t d_at = (size_t)kc * kAdjBlockB + (size_t)bq * kSweepBlockB;
                    mbar_expect_tx(&full_d[st_i], 2 * kSweepBlockB);
                    bulk_copy(st + 2 * kAdjBlockA, in_hi + d_at, kSweepBlockB, &full_d[st_i]);
                    bulk_copy(st + 2 * kAdjBlockA + kSweepBlockB, in_lo + d_at, kSweepBlockB, &full_d[st_i]);
                    sent_d = g0 + c + 1;
                }
                if (j + 1 < steps) // the next step's W, as its stages get free
                    for (int c = 0; c < pre && !*abort; ++c)
                        if (!send_w(j + 1, c)) break;
            }
            __syncwarp();
        } else if (warp == kSweepTailWarps + 1) {
            if (lane == 0 && j > 0 && // the accumulator has been read
                mbar_wait_cluster(&exchanged[(j - 1) % kExchangeBarriers], exchange_phase(j - 1), abort))
                fence_after();
            if (lane == 0 && !*abort) { // MMA issuer
                for (int c = 0; c < iters; ++c) {
                    const int st_i = stage(j, c);
                    const uint32_t ph = phase(j, c);
                    if (!mbar_wait(&full_w[st_i], stay ? 0u : ph, abort) || !mbar_wait(&full_d[st_i], ph, abort)) break;
                    fence_after();
                    const uint32_t a_hi = smem_addr(stages + st_i * kSweepStageBytes);
                    const uint32_t a_lo = a_hi + kAdjBlockA;
                    const uint32_t b_hi = a_hi + 2 * kAdjBlockA;
                    const uint32_t b_lo = b_hi + kSweepBlockB;
                    const bool second = c >= per; // of the CTA's two K ranges
                    const uint32_t acc = tmem + (second ? kSweepN : 0u);
                    const bool first = c == (second ? per : 0);
#pragma unroll
                    for (int q = 0; q < kKChunk / 16; ++q) {
                        mma(acc, make_desc(a_hi + 256 * q), make_desc(b_hi + 256 * q), kSweepIdesc, !first || q != 0);
                        mma(acc, make_desc(a_lo + 256 * q), make_desc(b_hi + 256 * q), kSweepIdesc, 1u);
                        mma(acc, make_desc(a_hi + 256 * q), make_desc(b_lo + 256 * q), kSweepIdesc, 1u);
                    }
                    commit(&empty[st_i]);
                }
                commit(done);
                if (*abort) mbar_drain(done, j & 1);
            }
            __syncwarp();
        }
        float ds[kRows], gs0[kRows], gu0[kRows], dv[kRows];
        bool keep[kRows];
        if (tail) {
            const float c_t = coef[k];
#pragma unroll
            for (int r = 0; r < kRows; ++r) {
                const float ss = op_s[r];
                ds[r] = p.smooth ? p.slope * ss * (1.0f - ss) : surrogate(op_u[r] - th, p.slope);
                gs0[r] = c_t * gr[r] - lv[r] * (op_u[r] - p.v_reset);
                gu0[r] = lv[r] * (1.0f - ss);
                dv[r] = p.v_rest - op_vp[r];
                keep[r] = op_m[r];
            }
            mbar_wait(done, j & 1, abort);
            __syncwarp();
            fence_after();
            if (__all_sync(0xffffffffu, !*abort) && iters > 0) {
                const int q = warp & 3, g = warp >> 2;
                // K range 2 ks + g, rows i = 32 q + lane, batch columns 8 o + c of rank o
                const uint32_t mine = smem_addr(got + (2 * ks + g) * 2 * kAdjM + il);
#pragma unroll
                for (int c16 = 0; c16 < 2; ++c16) {
                    float acc[16];
                    tmem_ld16(tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)(32 * g + 16 * c16), acc);
#pragma unroll
                    for (int c = 0; c < 16; c += 4) {
                        uint32_t ra;
                        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(mine), "r"(2 * c16 + c / 8));
                        asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(ra + (uint32_t)((c / 4 & 1) * kAdjM * 16)),
                                     "f"(acc[c]), "f"(acc[c + 1]), "f"(acc[c + 2]), "f"(acc[c + 3])
                                     : "memory");
                    }
                }
            }
            fence_before();
            // the partials are in place and the accumulator read: one arrival at each of the cluster's CTAs
            asm volatile("bar.sync 1, %0;" ::"n"(32 * kSweepTailWarps) : "memory");
            if (threadIdx.x < kSweepCluster && !*abort) {
                uint32_t ra;
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(smem_addr(&exchanged[j % kExchangeBarriers])), "r"(threadIdx.x));
                asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(ra) : "memory");
            }
            __syncwarp();
            mbar_wait_cluster(&exchanged[j % kExchangeBarriers], exchange_phase(j), abort);
            float x[kAdjCluster][kRows];
#pragma unroll
            for (int r = 0; r < kAdjCluster; ++r)
                if (r < ranges)
                    *reinterpret_cast<float4 *>(x[r]) = got[(r * 2 + bsub) * kAdjM + il];
            uint32_t t_hi[kRows / 2], t_lo[kRows / 2]; // dI^T of the rows, split, packed in pairs
#pragma unroll
            for (int r = 0; r < kRows; ++r) {
                float ge = x[0][r];
#pragma unroll
                for (int c = 1; c < kAdjCluster; ++c)
                    if (c < ranges) ge = ge + x[c][r];
                // a run's last step has no recurrent term; the product of its zero operand is NaN where W is not finite
                const float gs = j == 0 && ends_run ? gs0[r] : gs0[r] + ge;
                const float gu = gs * ds[r] + gu0[r];
                const float gm = keep[r] ? gu : 0.0f;
                const size_t o = blocked_index(b0 + r, i, n);
                __nv_bfloat16 h, l;
                split_bf16(gm, h, l);
                out_hi[o] = h;
                out_lo[o] = l;
                const uint32_t hb = __bfloat16_as_ushort(h), lb = __bfloat16_as_ushort(l);
                if (r & 1) {
                    t_hi[r >> 1] |= hb << 16;
                    t_lo[r >> 1] |= lb << 16;
                } else {
                    t_hi[r >> 1] = hb;
                    t_lo[r >> 1] = lb;
                }
                lv[r] = gm * (1.0f - al);
                gt[r] = gt[r] - gs * ds[r];
                ga[r] = ga[r] + gm * dv[r];
            }
            // publish: all of this CTA's dI, then one count
            asm volatile("bar.sync 1, %0;" ::"n"(32 * kSweepTailWarps) : "memory");
            if (threadIdx.x == 0 && !*abort)
                asm volatile("red.release.gpu.global.add.s32 [%0], 1;" ::"l"(ready + blockIdx.x * kReadyStride) : "memory");
            if (k > 0) operands(k - 1);
            const size_t o = blocked_index(i, (int)(k_off + (long long)k * kAdjN + b0), (int)k_cols);
            reinterpret_cast<uint2 *>(dT_hi + o)[0] = make_uint2(t_hi[0], t_hi[1]);
            reinterpret_cast<uint2 *>(dT_lo + o)[0] = make_uint2(t_lo[0], t_lo[1]);
        }
    }
    if (tail) {
#pragma unroll
        for (int r = 0; r < kRows; ++r) {
            lam_v[at0 + (size_t)r * n] = lv[r];
            g_theta[at0 + (size_t)r * n] = gt[r];
            g_alpha[at0 + (size_t)r * n] = ga[r];
        }
    } else if (warp == kSweepTailWarps && lane == 0 && *abort) { // its own copies in flight
        for (int c = 0; c < kStages; ++c) {
            const long long gw = sent_w - 1 - c, gd = sent_d - 1 - c;
            if (gw >= 0)
                mbar_drain(&full_w[stage((int)(gw / iters), (int)(gw % iters))],
                           stay ? 0u : phase((int)(gw / iters), (int)(gw % iters)));
            if (gd >= 0)
                mbar_drain(&full_d[stage((int)(gd / iters), (int)(gd % iters))], phase((int)(gd / iters), (int)(gd % iters)));
        }
    }
    __syncthreads();
    // no CTA leaves before its peers have arrived at its barrier
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (threadIdx.x == 0 && *abort) atomicOr(err, kUmmaTimeout);
    if (warp == 2) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols)
                     : "memory");
    }
}

// [L][B][R] FP32 -> the R x (L*B) matrix (row r, K = l*B + b) in the blocked
// layout, split into hi and lo (lo may be null: the values are exact in BF16).
// [L][B][R] FP32 -> the R_pad x (L*B) matrix (row r, K = l*B + b) in the
// blocked layout, split into hi and lo (lo may be null: the values are exact
// in BF16); rows R .. R_pad - 1 are zero (padding to the product's tile).
// One CTA per 128-row x 64-K output block: the 64 x 128 source tile is read
// with coalesced loads into shared memory, and the block -- 16 KiB,
// contiguous in the blocked layout -- is written one 16-byte core-matrix row
// (8 K values of one row) per store.
constexpr int kBtThreads = 256;
__global__ void __launch_bounds__(kBtThreads) k_blocked_t(const float *__restrict__ src, int L, int B, int R,
                                                          int R_pad, __nv_bfloat16 *__restrict__ hi,
                                                          __nv_bfloat16 *__restrict__ lo) {
    __shared__ float tile[kKChunk][kAdjM + 1];
    const int rb = blockIdx.x, kb = blockIdx.y, KK = L * B;
    for (int e = threadIdx.x; e < kKChunk * kAdjM; e += kBtThreads) {
        const int kk = e / kAdjM, rr = e % kAdjM; // r fastest: coalesced along the source row
        const int r = rb * kAdjM + rr;
        tile[kk][rr] = r < R ? src[(size_t)(kb * kKChunk + kk) * R + r] : 0.0f;
    }
    __syncthreads();
    const size_t blk = ((size_t)rb * (size_t)(KK / kKChunk) + (size_t)kb) * (size_t)(kAdjM * kKChunk);
    // 1,024 core-matrix rows of 8 values; element e of the block:
    //   k & 7 = e & 7, row & 7 = (e >> 3) & 7, k >> 3 = (e >> 6) & 7, row >> 3 = e >> 9
    for (int c = threadIdx.x; c < kAdjM * kKChunk / 8; c += kBtThreads) {
        const int e0 = c * 8;
        const int row = ((e0 >> 9) << 3) | ((e0 >> 3) & 7), k0 = ((e0 >> 6) & 7) << 3;
        __align__(16) __nv_bfloat16 h[8], l[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const float v = tile[k0 + q][row];
            if (lo) split_bf16(v, h[q], l[q]);
            else h[q] = __float2bfloat16_rn(v);
        }
        reinterpret_cast<uint4 *>(hi + blk)[c] = *reinterpret_cast<const uint4 *>(h);
        if (lo) reinterpret_cast<uint4 *>(lo + blk)[c] = *reinterpret_cast<const uint4 *>(l);
    }
}

constexpr int kWgN = 256; // UMMA N of the weight-gradient product
constexpr int kWgBlockB = kWgN * kKChunk * 2; // 32 KiB
// stages: 3 of A_hi A_lo B (64 KiB), or 2 of A_hi A_lo B_hi B_lo (96 KiB)
template <bool kSplitB> struct WgShape {
    static constexpr int stages = kSplitB ? 2 : 3;
    static constexpr int stage_bytes = 2 * kAdjBlockA + (kSplitB ? 2 : 1) * kWgBlockB;
    static constexpr int smem_bytes = stages * stage_bytes + 1024 + 256;
};
constexpr int kWgTmemCols = 256;
constexpr uint32_t kWgIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kWgN >> 3) << 17) |
                              ((uint32_t)(kAdjM >> 4) << 24);

// part[ks][n][j] = sum over the K chunks of split ks of (a_hi + a_lo)[j][K]
// (b_hi + b_lo)[n][K], the lo x lo product dropped (b_lo absent when b is
// exact in BF16).  a: M x K blocked (128-row tiles), b: Nc x K blocked (its
// 256-row tile n0 = blockIdx.y * 256 is two 128-row block rows).  Grid
// (M / 128, Nc / 256, split); roles as in k_adj_umma.
template <bool kSplitB>
__global__ void __launch_bounds__(kThreads, 1)
    k_wgrad_umma(const __nv_bfloat16 *__restrict__ a_hi, const __nv_bfloat16 *__restrict__ a_lo,
                 const __nv_bfloat16 *__restrict__ b, const __nv_bfloat16 *__restrict__ b_lo,
                 float *__restrict__ part, int M, int Nc, int K, int split, int *__restrict__ err) {
    constexpr int kWgStages = WgShape<kSplitB>::stages;
    constexpr int kWgStageBytes = WgShape<kSplitB>::stage_bytes;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t *stages = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t *full = (uint64_t *)(stages + kWgStages * kWgStageBytes);
    uint64_t *empty = full + kWgStages;
    uint64_t *done = empty + kWgStages;
    uint32_t *tmem_slot = (uint32_t *)(done + 1);
    volatile int *abort = (volatile int *)(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int mt = blockIdx.x, nt = blockIdx.y, ks = blockIdx.z;
    const int kchunks = K / kKChunk;
    const int per = kchunks / split;
    const int kc0 = ks * per;
    const int iters = (ks == split - 1) ? kchunks - kc0 : per;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kWgStages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        mbar_init(done, 1);
        *abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 2) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tmem_slot)),
                     "r"(kWgTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp == 0 && lane == 0) { // producer
        for (int it = 0; it < iters; ++it) {
            const int s = it % kWgStages;
            if (it >= kWgStages && !mbar_wait(&empty[s], ((it / kWgStages) & 1) ^ 1, abort)) break;
            uint8_t *st = stages + s * kWgStageBytes;
            const int kc = kc0 + it;
            const size_t a_blk = (size_t)mt * kchunks + kc;
            const size_t b_blk0 = (size_t)(2 * nt) * kchunks + kc, b_blk1 = (size_t)(2 * nt + 1) * kchunks + kc;
            mbar_expect_tx(&full[s], kWgStageBytes);
            bulk_copy(st, (const uint8_t *)a_hi + a_blk * kAdjBlockA, kAdjBlockA, &full[s]);
            bulk_copy(st + kAdjBlockA, (const uint8_t *)a_lo + a_blk * kAdjBlockA, kAdjBlockA, &full[s]);
            // the two 128-row halves of the B tile, one after the other: rows
            // 128..255 continue the 8-row core-matrix groups at byte 16384
            bulk_copy(st + 2 * kAdjBlockA, (const uint8_t *)b + b_blk0 * kAdjBlockA, kAdjBlockA, &full[s]);
            bulk_copy(st + 3 * kAdjBlockA, (const uint8_t *)b + b_blk1 * kAdjBlockA, kAdjBlockA, &full[s]);
            if constexpr (kSplitB) {
                bulk_copy(st + 4 * kAdjBlockA, (const uint8_t *)b_lo + b_blk0 * kAdjBlockA, kAdjBlockA, &full[s]);
                bulk_copy(st + 5 * kAdjBlockA, (const uint8_t *)b_lo + b_blk1 * kAdjBlockA, kAdjBlockA, &full[s]);
            }
        }
    } else if (warp == 1 && lane == 0) { // MMA issuer
        for (int it = 0; it < iters; ++it) {
            const int s = it % kWgStages;
            if (!mbar_wait(&full[s], (it / kWgStages) & 1, abort)) break;
            fence_after();
            const uint32_t ah = smem_addr(stages + s * kWgStageBytes);
            const uint32_t al = ah + kAdjBlockA;
            const uint32_t bb = ah + 2 * kAdjBlockA;
#pragma unroll
            for (int k = 0; k < kKChunk / 16; ++k) {
                mma(tmem, make_desc(ah + 256 * k), make_desc(bb + 256 * k), kWgIdesc, (it | k) != 0);
                mma(tmem, make_desc(al + 256 * k), make_desc(bb + 256 * k), kWgIdesc, 1u);
                if constexpr (kSplitB)
                    mma(tmem, make_desc(ah + 256 * k), make_desc(bb + kWgBlockB + 256 * k), kWgIdesc, 1u);
            }
            commit(&empty[s]);
        }
        commit(done);
    }
    __syncwarp();
    mbar_wait(done, 0, abort);
    __syncthreads();
    fence_after();
    // epilogue: warp w reads TMEM lanes 32*(w%4).. (rows j) and columns
    // 128*(w/4).. (n); stores are coalesced along j
    const int q = warp & 3, h = warp >> 2;
    const int j = mt * kAdjM + 32 * q + lane;
    if (!*abort) {
        float *out = part + (size_t)ks * Nc * M;
        for (int c16 = 0; c16 < 8; ++c16) {
            float acc[16];
            tmem_ld16(tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)(128 * h + 16 * c16), acc);
            const int n0 = nt * kWgN + 128 * h + 16 * c16;
#pragma unroll
            for (int c = 0; c < 16; ++c) out[(size_t)(n0 + c) * M + j] = acc[c];
        }
    }
    fence_before();
    __syncthreads();
    if (threadIdx.x == 0 && *abort) atomicOr(err, kUmmaTimeout);
    if (warp == 2) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kWgTmemCols)
                     : "memory");
    }
}

__global__ void k_reduce_add(float *__restrict__ g, const float *__restrict__ part, int split, long long count,
                             long long stride) {
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= count) return;
    float acc = part[idx];
    for (int q = 1; q < split; ++q) acc = acc + part[(size_t)q * stride + idx];
    g[idx] = g[idx] + acc;
}

bool adj_shape_ok(int B, int N) { return B == kAdjN && N > 0 && N % kAdjM == 0; }

} // namespace

template <bool kParts>
static nbg_status adj_step(const char *name, bool chained, float *parts, const void *w_hi, const void *w_lo, const void *dI_hi_in, const void *dI_lo_in,
                                      void *dI_hi_out, void *dI_lo_out, const float *g_read, float c_t,
                                      const float *u, const float *s, const uint8_t *m, const float *vprev,
                                      float *lam_v, float *dI, float *g_theta, float *g_alpha, const float *alpha,
                                      const float *theta, const nbg_lif_grad_params *p, int B, int N, void *dT_hi,
                                      void *dT_lo, int64_t k_off, int64_t k_cols, int *err, void *stream) {
    if (!w_hi || !w_lo || !dI_hi_in || !dI_lo_in || !dI_hi_out || !dI_lo_out || !g_read || !u || !s || !m ||
        !vprev || !lam_v || !g_theta || !g_alpha || !alpha || !theta || !p || !err || !adj_shape_ok(B, N) ||
        N / kKChunk < kAdjCluster || dI_hi_in == dI_hi_out || dI_lo_in == dI_lo_out)
        return nbg_fail(NBG_ERR_INVALID, "%s: bad arguments (B must be %d, N a multiple of %d "
                        "and at least %d, distinct in and out operand buffers)", name, kAdjN, kAdjM,
                        kAdjCluster * kKChunk);
    if (dT_hi && (!dT_lo || k_off < 0 || k_off % kAdjN || k_cols % kKChunk || k_off + kAdjN > k_cols ||
                  k_cols > 0x7fffffff))
        return nbg_fail(NBG_ERR_INVALID, "%s: dT needs dT_lo, k_off a multiple of %d with "
                        "k_off + %d <= k_cols, k_cols a multiple of %d below 2^31", name, kAdjN, kAdjN, kKChunk);
    static bool attr_set = false;
    if (!attr_set) {
        NBG_CUDA(cudaFuncSetAttribute(k_adj_step_umma<kParts>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      adj_smem<kParts>()));
        attr_set = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(N / kAdjM, kAdjCluster);
    cfg.blockDim = dim3(kAdjStepThreads);
    cfg.dynamicSmemBytes = adj_smem<kParts>();
    cfg.stream = (cudaStream_t)stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = chained ? 1 : 0;
    NBG_CUDA(cudaLaunchKernelEx(&cfg, k_adj_step_umma<kParts>, (const __nv_bfloat16 *)w_hi, (const __nv_bfloat16 *)w_lo,
                                (const __nv_bfloat16 *)dI_hi_in, (const __nv_bfloat16 *)dI_lo_in,
                                (__nv_bfloat16 *)dI_hi_out, (__nv_bfloat16 *)dI_lo_out, g_read, c_t, u, s, m, vprev,
                                lam_v, dI, g_theta, g_alpha, alpha, theta, *p, N, (__nv_bfloat16 *)dT_hi,
                                (__nv_bfloat16 *)dT_lo, (long long)k_off, (long long)k_cols, (float4 *)parts, err));
    NBG_CUDA(cudaGetLastError());
    return NBG_OK;
}

static void sweep_config(cudaLaunchConfig_t &cfg, cudaLaunchAttribute (&attr)[2], int N, void *stream) {
    cfg = {};
    cfg.gridDim = dim3(N / kAdjM * kSweepParts, kSweepCluster);
    cfg.blockDim = dim3(kSweepThreads);
    cfg.dynamicSmemBytes = kSweepSmemBytes;
    cfg.stream = (cudaStream_t)stream;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1;
    attr[0].val.clusterDim.y = kSweepCluster;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeCooperative;
    attr[1].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
}

extern "C" {

nbg_status nbg_adjoint_rec_prepare(const float *w_rec, void *w_hi, void *w_lo, int N, void *stream) {
    if (!w_rec || !w_hi || !w_lo || N <= 0 || N % kAdjM)
        return nbg_fail(NBG_ERR_INVALID, "nbg_adjoint_rec_prepare: N must be a positive multiple of %d", kAdjM);
    const long long total = (long long)N * N;
    k_split_blocked<<<(unsigned)((total + 255) / 256), 256, 0, (cudaStream_t)stream>>>(
        w_rec, (__nv_bfloat16 *)w_hi, (__nv_bfloat16 *)w_lo, N, N);
    NBG_CUDA(cudaGetLastError());
    return NBG_OK;
}

nbg_status nbg_lif_adjoint_step_split(const float *g_parts, int n_parts, const float *g_read, float c_t,
                                      const float *u, const float *s, const uint8_t *m, const float *vprev,
                                      float *lam_v, float *dI, void *dI_hi, void *dI_lo, float *g_theta,
                                      float *g_alpha, const float *alpha, const float *theta,
                                      const nbg_lif_grad_params *p, int B, int N, void *stream) {
    if (!g_read || !u || !s || !m || !vprev || !lam_v || !dI || !dI_hi || !dI_lo || !g_theta || !g_alpha || !alpha ||
        !theta || !p || (g_parts && n_parts <= 0) || !adj_shape_ok(B, N))
        return nbg_fail(NBG_ERR_INVALID, "nbg_lif_adjoint_step_split: bad arguments (B must be %d, N a multiple of %d)",
                        kAdjN, kAdjM);
    const int total = B * N;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((total + 255) / 256);
    cfg.blockDim = dim3(256);
    cfg.stream = (cudaStream_t)stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    NBG_CUDA(cudaLaunchKernelEx(&cfg, k_lif_adj_split, g_parts, n_parts, g_read, c_t, u, s, m, vprev, lam_v, dI,
                                (__nv_bfloat16 *)dI_hi, (__nv_bfloat16 *)dI_lo, g_theta, g_alpha, alpha, theta, *p,
                                N, total));
    NBG_CUDA(cudaGetLastError());
    return NBG_OK;
}

nbg_status nbg_adjoint_rec_grad(const void *w_hi, const void *w_lo, const void *dI_hi, const void *dI_lo,
                                float *g_parts, int split, int B, int N, int *err, void *stream) {
    if (!w_hi || !w_lo || !dI_hi || !dI_lo || !g_parts || !err || !adj_shape_ok(B, N) || split <= 0 ||
        split > N / kKChunk)
        return nbg_fail(NBG_ERR_INVALID, "nbg_adjoint_rec_grad: bad arguments (B must be %d, N a multiple of %d, "
                        "1 <= split <= N / %d)", kAdjN, kAdjM, kKChunk);
    static bool attr_set = false;
    if (!attr_set) {
        NBG_CUDA(cudaFuncSetAttribute(k_adj_umma, cudaFuncAttributeMaxDynamicSharedMemorySize, kAdjSmemBytes));
        attr_set = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(N / kAdjM, split);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = kAdjSmemBytes;
    cfg.stream = (cudaStream_t)stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    NBG_CUDA(cudaLaunchKernelEx(&cfg, k_adj_umma, (const __nv_bfloat16 *)w_hi, (const __nv_bfloat16 *)w_lo,
                                (const __nv_bfloat16 *)dI_hi, (const __nv_bfloat16 *)dI_lo, g_parts, N, split, err));
    NBG_CUDA(cudaGetLastError());
    return NBG_OK;
}

nbg_status nbg_lif_adjoint_step_fused(const void *w_hi, const void *w_lo, const void *dI_hi_in, const void *dI_lo_in,
                                      void *dI_hi_out, void *dI_lo_out, const float *g_read, float c_t,
                                      const float *u, const float *s, const uint8_t *m, const float *vprev,
                                      float *lam_v, float *dI, float *g_theta, float *g_alpha, const float *alpha,
                                      const float *theta, const nbg_lif_grad_params *p, int B, int N, void *dT_hi,
                                      void *dT_lo, int64_t k_off, int64_t k_cols, int *err, void *stream) {
    return adj_step<false>("nbg_lif_adjoint_step_fused", false, nullptr, w_hi, w_lo, dI_hi_in, dI_lo_in, dI_hi_out, dI_lo_out, g_read, c_t, u, s, m, vprev, lam_v,
                           dI, g_theta, g_alpha, alpha, theta, p, B, N, dT_hi, dT_lo, k_off, k_cols, err, stream);
}

nbg_status nbg_lif_adjoint_step_parts(const void *w_hi, const void *w_lo, const void *dI_hi_in, const void *dI_lo_in,
                                      void *dI_hi_out, void *dI_lo_out, const float *g_read, float c_t,
                                      const float *u, const float *s, const uint8_t *m, const float *vprev,
                                      float *lam_v, float *dI, float *g_theta, float *g_alpha, const float *alpha,
                                      const float *theta, const nbg_lif_grad_params *p, int B, int N, void *dT_hi,
                                      void *dT_lo, int64_t k_off, int64_t k_cols, float *parts, int *err, void *stream) {
    if (!parts) return nbg_fail(NBG_ERR_INVALID, "nbg_lif_adjoint_step_parts: parts is NULL");
    return adj_step<true>("nbg_lif_adjoint_step_parts", false, parts, w_hi, w_lo, dI_hi_in, dI_lo_in, dI_hi_out, dI_lo_out, g_read, c_t, u, s, m, vprev, lam_v,
                           dI, g_theta, g_alpha, alpha, theta, p, B, N, dT_hi, dT_lo, k_off, k_cols, err, stream);
}

nbg_status nbg_lif_adjoint_step_chained(const void *w_hi, const void *w_lo, const void *dI_hi_in, const void *dI_lo_in,
                                        void *dI_hi_out, void *dI_lo_out, const float *g_read, float c_t,
                                        const float *u, const float *s, const uint8_t *m, const float *vprev,
                                        float *lam_v, float *dI, float *g_theta, float *g_alpha, const float *alpha,
                                        const float *theta, const nbg_lif_grad_params *p, int B, int N, void *dT_hi,
                                        void *dT_lo, int64_t k_off, int64_t k_cols, float *parts, int *err, void *stream) {
    if (!parts) return nbg_fail(NBG_ERR_INVALID, "nbg_lif_adjoint_step_chained: parts is NULL");
    return adj_step<true>("nbg_lif_adjoint_step_chained", true, parts, w_hi, w_lo, dI_hi_in, dI_lo_in, dI_hi_out, dI_lo_out, g_read, c_t, u, s, m, vprev, lam_v,
                           dI, g_theta, g_alpha, alpha, theta, p, B, N, dT_hi, dT_lo, k_off, k_cols, err, stream);
}

int64_t nbg_lif_adjoint_sweep_work(int B, int N) {
    if (!adj_shape_ok(B, N)) return 0;
    if (cudaFuncSetAttribute(k_adj_sweep_umma, cudaFuncAttributeMaxDynamicSharedMemorySize, kSweepSmemBytes) !=
        cudaSuccess) {
        (void)cudaGetLastError();
        return 0;
    }
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[2];
    sweep_config(cfg, attr, N, nullptr);
    cfg.numAttrs = 1; // the cluster's
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, k_adj_sweep_umma, &cfg) != cudaSuccess) {
        (void)cudaGetLastError();
        return 0;
    }
    const int tiles = N / kAdjM * kSweepParts;
    return clusters >= tiles ? tiles * kReadyStride : 0;
}

static nbg_status adj_sweep(const char *name, bool ends_run, const void *w_hi, const void *w_lo, void *d_hi0, void *d_lo0, void *d_hi1, void *d_lo1,
                                 const float *g_read, const float *coef, const float *u, const float *s,
                                 const uint8_t *m, const float *vprev, float *lam_v, float *g_theta, float *g_alpha,
                                 const float *alpha, const float *theta, const nbg_lif_grad_params *p, int steps, int t0,
                                 int B, int N, void *dT_hi, void *dT_lo, int64_t k_off, int64_t k_cols, float *work,
                                 int *err, void *stream) {
    if (!w_hi || !w_lo || !d_hi0 || !d_lo0 || !d_hi1 || !d_lo1 || !g_read || !coef || !u || !s || !m || !vprev || !lam_v ||
        !g_theta || !g_alpha || !alpha || !theta || !p || !dT_hi || !dT_lo || !work || !err || steps <= 0 || t0 < 0 ||
        d_hi0 == d_hi1 || d_lo0 == d_lo1 || k_off < 0 || k_off % kAdjN || k_cols % kKChunk ||
        k_off + (int64_t)steps * B > k_cols || k_cols > 0x7fffffff || steps > 0x7fffffff / kAdjCluster)
        return nbg_fail(NBG_ERR_INVALID, "%s: bad arguments", name);
    if (!nbg_lif_adjoint_sweep_work(B, N))
        return nbg_fail(NBG_ERR_INVALID, "%s: B must be %d, N a multiple of %d and not more than the "
                        "device holds at once", name, kAdjN, kAdjM);
    int *ready = (int *)work;
    NBG_CUDA(cudaMemsetAsync(ready, 0, (size_t)(N / kAdjM * kSweepParts) * kReadyStride * sizeof(int), (cudaStream_t)stream));
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[2];
    sweep_config(cfg, attr, N, stream);
    NBG_CUDA(cudaLaunchKernelEx(&cfg, k_adj_sweep_umma, (const __nv_bfloat16 *)w_hi, (const __nv_bfloat16 *)w_lo,
                                (__nv_bfloat16 *)d_hi0, (__nv_bfloat16 *)d_lo0, (__nv_bfloat16 *)d_hi1,
                                (__nv_bfloat16 *)d_lo1, g_read, coef, u, s, (const unsigned char *)m, vprev, lam_v, g_theta,
                                g_alpha, alpha, theta, *p, N, steps, t0, ends_run ? 1 : 0, (__nv_bfloat16 *)dT_hi, (__nv_bfloat16 *)dT_lo,
                                (long long)k_off, (long long)k_cols, ready, err));
    NBG_CUDA(cudaGetLastError());
    return NBG_OK;
}

nbg_status nbg_lif_adjoint_sweep(const void *w_hi, const void *w_lo, void *d_hi0, void *d_lo0, void *d_hi1, void *d_lo1,
                                 const float *g_read, const float *coef, const float *u, const float *s,
                                 const uint8_t *m, const float *vprev, float *lam_v, float *g_theta, float *g_alpha,
                                 const float *alpha, const float *theta, const nbg_lif_grad_params *p, int steps, int t0,
                                 int B, int N, void *dT_hi, void *dT_lo, int64_t k_off, int64_t k_cols, float *work,
                                 int *err, void *stream) {
    return adj_sweep("nbg_lif_adjoint_sweep", false, w_hi, w_lo, d_hi0, d_lo0, d_hi1, d_lo1, g_read, coef, u, s, m, vprev, lam_v, g_theta, g_alpha, alpha,
                     theta, p, steps, t0, B, N, dT_hi, dT_lo, k_off, k_cols, work, err, stream);
}

nbg_status nbg_lif_adjoint_sweep_end(const void *w_hi, const void *w_lo, void *d_hi0, void *d_lo0, void *d_hi1, void *d_lo1,
                                 const float *g_read, const float *coef, const float *u, const float *s,
                                 const uint8_t *m, const float *vprev, float *lam_v, float *g_theta, float *g_alpha,
                                 const float *alpha, const float *theta, const nbg_lif_grad_params *p, int steps, int t0,
                                 int B, int N, void *dT_hi, void *dT_lo, int64_t k_off, int64_t k_cols, float *work,
                                 int *err, void *stream) {
    return adj_sweep("nbg_lif_adjoint_sweep_end", true, w_hi, w_lo, d_hi0, d_lo0, d_hi1, d_lo1, g_read, coef, u, s, m, vprev, lam_v, g_theta, g_alpha, alpha,
                     theta, p, steps, t0, B, N, dT_hi, dT_lo, k_off, k_cols, work, err, stream);
}

nbg_status nbg_adjoint_blocked_t(const float *src, int L, int B, int R, int R_pad, void *hi, void *lo,
                                 void *stream) {
    if (!src || !hi || L <= 0 || B <= 0 || R <= 0 || R_pad < R || R_pad % kAdjM || ((long long)L * B) % kKChunk)
        return nbg_fail(NBG_ERR_INVALID, "nbg_adjoint_blocked_t: R_pad must be >= R and a multiple of %d, L*B a "
                        "multiple of %d", kAdjM, kKChunk);
    const dim3 grid(R_pad / kAdjM, (unsigned)(((long long)L * B) / kKChunk));
    k_blocked_t<<<grid, kBtThreads, 0, (cudaStream_t)stream>>>(src, L, B, R, R_pad, (__nv_bfloat16 *)hi,
                                                               (__nv_bfloat16 *)lo);
    NBG_CUDA(cudaGetLastError());
    return NBG_OK;
}

nbg_status nbg_adjoint_wgrad(const void *a_hi, const void *a_lo, const void *b, const void *b_lo, int M, int Nc,
                             int K, float *part, int split, int *err, void *stream) {
    if (!a_hi || !a_lo || !b || !part || !err || M <= 0 || M % kAdjM || Nc <= 0 || Nc % kWgN || K <= 0 ||
        K % kKChunk || split <= 0 || split > K / kKChunk)
        return nbg_fail(NBG_ERR_INVALID, "nbg_adjoint_wgrad: M must be a multiple of %d, Nc of %d, K of %d, "
                        "1 <= split <= K / %d", kAdjM, kWgN, kKChunk, kKChunk);
    static bool attr_set[2] = {false, false};
    const dim3 grid(M / kAdjM, Nc / kWgN, split);
    const __nv_bfloat16 *ah = (const __nv_bfloat16 *)a_hi, *al = (const __nv_bfloat16 *)a_lo;
    if (b_lo) {
        if (!attr_set[1]) {
            NBG_CUDA(cudaFuncSetAttribute(k_wgrad_umma<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          WgShape<true>::smem_bytes));
            attr_set[1] = true;
        }
        k_wgrad_umma<true><<<grid, kThreads, WgShape<true>::smem_bytes, (cudaStream_t)stream>>>(
            ah, al, (const __nv_bfloat16 *)b, (const __nv_bfloat16 *)b_lo, part, M, Nc, K, split, err);
    } else {
        if (!attr_set[0]) {
            NBG_CUDA(cudaFuncSetAttribute(k_wgrad_umma<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          WgShape<false>::smem_bytes));
            attr_set[0] = true;
        }
        k_wgrad_umma<false><<<grid, kThreads, WgShape<false>::smem_bytes, (cudaStream_t)stream>>>(
            ah, al, (const __nv_bfloat16 *)b, nullptr, part, M, Nc, K, split, err);
    }
    NBG_CUDA(cudaGetLastError());
    return NBG_OK;
}

nbg_status nbg_adjoint_reduce_add(float *g, const float *part, int split, int64_t count, int64_t stride,
                                  void *stream) {
    if (!g || !part || split <= 0 || count <= 0 || stride < count)
        return nbg_fail(NBG_ERR_INVALID, "nbg_adjoint_reduce_add: bad arguments");
    k_reduce_add<<<(unsigned)((count + 255) / 256), 256, 0, (cudaStream_t)stream>>>(g, part, split, (long long)count,
                                                                                 (long long)stride);
    NBG_CUDA(cudaGetLastError());
    return NBG_OK;
}

} // extern "C"
