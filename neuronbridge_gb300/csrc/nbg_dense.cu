// nbg_dense.cu -- dense all-to-all spike delivery for many LIF populations
// sharing one weight matrix (C ABI in include/nbg_dense.h).
//
// Per step t (instances B = 64, neurons N):
//   delivery   I_t = S_{t-1} W          S binary, W N x N FP32
//   update     voltage-jump LIF over B x N neurons, writes S_t
//
// Delivery paths:
//   * NBG_DENSE_SPLIT_BF16 -- tcgen05 (nbg_umma.cuh): the same split-K GEMM
//     with the accumulator in tensor memory and operands in the UMMA blocked
//     layout, moved by bulk copies; W is tiled once at create time and the
//     update kernel writes S blocked.
//   * NBG_DENSE_SPLIT_BF16_SYNC -- the legacy mma.sync tensor path.  W = W_hi + W_lo with both parts
//     BF16 (W_hi = bf16(W), W_lo = bf16(W - W_hi)); a binary spike is exact in
//     BF16, so S W_hi + S W_lo accumulated in FP32 carries ~16 mantissa bits
//     of W.  The GEMM is "swap-AB": M = post-synaptic neurons (128 per CTA),
//     N = the 64 instances, K = pre-synaptic neurons, with W stored transposed
//     (K-major) so that both operands stream K-contiguous.  Split-K = 2 gives
//     128 CTAs; the two partial sums are added in a fixed order by the update
//     kernel, so results are deterministic.  At M = 64 instances the GEMM
//     streams 2 x N^2 BF16 per step and is HBM-bound.
//   * NBG_DENSE_FP32 -- CUDA cores (k_dense_gather): each post neuron sums W[i][j] over the
//     spiking pre-synaptic i of its instance in ascending i, in FP32, which is
//     the exact sequential sum the CPU oracle computes.

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <vector>

#include "nbg_common.cuh"
#include "nbg_dense.h"
#include "nbg_umma.cuh"

namespace {

constexpr int kInstances = 64; // GEMM N
constexpr int kBM = 128;       // post neurons per CTA (GEMM M)
constexpr int kBK = 64;        // pre neurons per pipeline stage
constexpr int kStages = 4;
constexpr int kSplitK = 2;
constexpr int kGemmThreads = 256;
constexpr int kStageA = kBM * kBK;              // bf16 elements of one A (W^T) tile
constexpr int kStageB = kInstances * kBK;       // bf16 elements of the S tile
constexpr int kStageElems = 2 * kStageA + kStageB;
constexpr size_t kGemmSmem = (size_t)kStages * kStageElems * sizeof(__nv_bfloat16); // 160 KiB

// ------------------------------------------------------------ preprocessing

// W (pre x post, FP32) -> W_hi^T, W_lo^T (post x pre, BF16): 32 x 32 tiles
// transposed through shared memory.
__global__ void k_split_transpose(const float *__restrict__ w, __nv_bfloat16 *__restrict__ hi,
                                  __nv_bfloat16 *__restrict__ lo, int n) {
    __shared__ float tile[32][33];
    const int i0 = blockIdx.y * 32, j0 = blockIdx.x * 32;
    for (int r = threadIdx.y; r < 32; r += blockDim.y) tile[r][threadIdx.x] = w[(size_t)(i0 + r) * n + j0 + threadIdx.x];
    __syncthreads();
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        const float x = tile[threadIdx.x][r]; // W[i0 + tx][j0 + r]
        const __nv_bfloat16 h = __float2bfloat16_rn(x);
        const __nv_bfloat16 l = __float2bfloat16_rn(x - __bfloat162float(h));
        const size_t o = (size_t)(j0 + r) * n + i0 + threadIdx.x;
        hi[o] = h;
        lo[o] = l;
    }
}

// W (pre x post, FP32) -> W_hi^T, W_lo^T in the UMMA blocked layout: block
// (m tile, k chunk) of 128 post x 64 pre at ((mt * kchunks + kc) * 16 KiB).
__global__ void k_split_tile(const float *__restrict__ w, __nv_bfloat16 *__restrict__ hi,
                             __nv_bfloat16 *__restrict__ lo, int n) {
    const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (size_t)n * n) return;
    const int k = (int)(idx / n), j = (int)(idx % n); // W[k][j]: pre k, post j
    const float x = w[idx];
    const __nv_bfloat16 h = __float2bfloat16_rn(x);
    const __nv_bfloat16 l = __float2bfloat16_rn(x - __bfloat162float(h));
    const int kchunks = n / umma::kKChunk;
    const size_t byte = ((size_t)(j / umma::kM) * kchunks + k / umma::kKChunk) * umma::kBlockA +
                        umma::block_offset(j % umma::kM, k % umma::kKChunk);
    hi[byte / 2] = h;
    lo[byte / 2] = l;
}

// offset (elements) of S[b][k] in the blocked S of the tcgen05 path
__device__ __host__ __forceinline__ size_t s_blocked(int b, int k) {
    return ((size_t)(k / umma::kKChunk) * umma::kBlockB + umma::block_offset(b, k % umma::kKChunk)) / 2;
}

// ------------------------------------------------------- spikes in and out
//
// The caller's spikes are bytes [instance][neuron]; the delivery paths hold
// them as BF16 in the blocked layout, BF16 rows or bit words.  One thread
// converts eight neighbouring neurons: a 16-byte core-matrix row, 16 bytes of a
// row or one byte of a word.  Done on the host, element by element, this took
// 1.5 ms of a read-out of 64 x 8,192 and most of a small delivery; the copies
// of the bytes (512 KiB) and this kernel (memory-bound, 1.6 MB) about 40 us.
enum { kLayoutBlocked = 0, kLayoutRows = 1, kLayoutBits = 2 };

template <int kLayout> __device__ __forceinline__ size_t spikes8_at(int b, int k, int n) { // element of the group's first neuron
    return kLayout == kLayoutBlocked ? s_blocked(b, k) : (size_t)b * n + k;
}

template <int kLayout>
__global__ void k_spikes_out(const void *__restrict__ s, uint8_t *__restrict__ out, int n, int groups) {
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= groups) return;
    const int b = g / (n / 8), k = (g - b * (n / 8)) * 8;
    unsigned bits = 0u;
    if constexpr (kLayout == kLayoutBits) {
        bits = reinterpret_cast<const uint8_t *>(s)[g];
    } else {
        const uint4 q = *reinterpret_cast<const uint4 *>(reinterpret_cast<const __nv_bfloat16 *>(s) + spikes8_at<kLayout>(b, k, n));
        const unsigned w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int i = 0; i < 8; ++i) bits |= ((w[i >> 1] >> (16 * (i & 1)) & 0x7fffu) ? 1u : 0u) << i;
    }
    uint2 o = make_uint2(0u, 0u);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        o.x |= (bits >> i & 1u) << (8 * i);
        o.y |= (bits >> (i + 4) & 1u) << (8 * i);
    }
    reinterpret_cast<uint2 *>(out)[g] = o;
}

template <int kLayout>
__global__ void k_spikes_in(const uint8_t *__restrict__ in, void *__restrict__ s, int n, int groups) {
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= groups) return;
    const int b = g / (n / 8), k = (g - b * (n / 8)) * 8;
    const uint2 q = reinterpret_cast<const uint2 *>(in)[g];
    unsigned bits = 0u;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        bits |= (q.x >> (8 * i) & 0xffu ? 1u : 0u) << i;
        bits |= (q.y >> (8 * i) & 0xffu ? 1u : 0u) << (i + 4);
    }
    if constexpr (kLayout == kLayoutBits) {
        reinterpret_cast<uint8_t *>(s)[g] = (uint8_t)bits;
    } else {
        const unsigned one = 0x3f80u; // 1.0 in BF16
        unsigned w[4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
            w[i] = (bits >> (2 * i) & 1u ? one : 0u) | (bits >> (2 * i + 1) & 1u ? one << 16 : 0u);
        *reinterpret_cast<uint4 *>(reinterpret_cast<__nv_bfloat16 *>(s) + spikes8_at<kLayout>(b, k, n)) =
            make_uint4(w[0], w[1], w[2], w[3]);
    }
}

// out = partial[0] + partial[1]: the same fixed order as the update kernels
__global__ void k_sum_split_partials(const float *__restrict__ part, float *__restrict__ out, int total) {
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx < total) out[idx] = part[idx] + part[(size_t)total + idx];
}

// ------------------------------------------------------------- GEMM (mma.sync)

__device__ __forceinline__ unsigned smem_u32(const void *p) {
    return (unsigned)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void cp_async16(void *smem, const void *gmem) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(smem_u32(smem)), "l"(gmem));
}

// element offset of (row, col) in a [rows][64] BF16 tile whose 16-byte chunks
// are XOR-swizzled by row so that ldmatrix reads are bank-conflict free
__device__ __forceinline__ int swz(int row, int col) {
    return row * kBK + ((((col >> 3) ^ (row & 7)) << 3) | (col & 7));
}

__device__ __forceinline__ void ldsm_x4(unsigned &r0, unsigned &r1, unsigned &r2, unsigned &r3, const void *p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
                 : "r"(smem_u32(p)));
}

__device__ __forceinline__ void mma_bf16(float *c, const unsigned *a, unsigned b0, unsigned b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// One stage: W_hi^T rows [m0, m0+128) x K [k0, k0+64), W_lo^T likewise, and
// S rows [0, 64) x K [k0, k0+64).  16-byte cp.async chunks, 10 per thread.
__device__ __forceinline__ void load_stage(__nv_bfloat16 *st, const __nv_bfloat16 *__restrict__ whi,
                                           const __nv_bfloat16 *__restrict__ wlo,
                                           const __nv_bfloat16 *__restrict__ s, int n, int m0, int k0) {
    const int tid = threadIdx.x;
    // A tiles: 128 rows x 8 chunks = 1024 chunks each
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int c = tid + q * kGemmThreads;
        const int row = c >> 3, ch = c & 7;
        const size_t g = (size_t)(m0 + row) * n + k0 + ch * 8;
        cp_async16(st + swz(row, ch * 8), whi + g);
        cp_async16(st + kStageA + swz(row, ch * 8), wlo + g);
    }
    // B tile: 64 rows x 8 chunks = 512 chunks
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const int c = tid + q * kGemmThreads;
        const int row = c >> 3, ch = c & 7;
        cp_async16(st + 2 * kStageA + swz(row, ch * 8), s + (size_t)row * n + k0 + ch * 8);
    }
}

// partial[ks][b][j] = sum over k in split ks of S[b][k] * (W_hi[k][j] + W_lo[k][j])
__global__ void __launch_bounds__(kGemmThreads, 1)
    k_dense_gemm(const __nv_bfloat16 *__restrict__ whi, const __nv_bfloat16 *__restrict__ wlo,
                 const __nv_bfloat16 *__restrict__ s, float *__restrict__ partial, int n) {
    extern __shared__ __align__(128) __nv_bfloat16 smem[];
    const int m0 = blockIdx.x * kBM;
    const int ks = blockIdx.y;
    const int kper = n / kSplitK;
    const int kbeg = ks * kper;
    const int iters = kper / kBK;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    float acc[8][4];
#pragma unroll
    for (int a = 0; a < 8; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) acc[a][b] = 0.0f;

#pragma unroll
    for (int p = 0; p < kStages - 1; ++p) {
        if (p < iters) load_stage(smem + p * kStageElems, whi, wlo, s, n, m0, kbeg + p * kBK);
        asm volatile("cp.async.commit_group;\n");
    }
    for (int it = 0; it < iters; ++it) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(kStages - 2));
        __syncthreads();
        // prefetch stage it + kStages - 1 into the buffer freed by iteration it-1
        const int nx = it + kStages - 1;
        if (nx < iters) load_stage(smem + (nx % kStages) * kStageElems, whi, wlo, s, n, m0, kbeg + nx * kBK);
        asm volatile("cp.async.commit_group;\n");

        const __nv_bfloat16 *st = smem + (it % kStages) * kStageElems;
        const __nv_bfloat16 *sa_hi = st, *sa_lo = st + kStageA, *sb = st + 2 * kStageA;
#pragma unroll
        for (int kk = 0; kk < kBK; kk += 16) {
            unsigned ahi[4], alo[4];
            {
                const int row = warp * 16 + (lane & 7) + 8 * ((lane >> 3) & 1);
                const int col = kk + 8 * (lane >> 4);
                ldsm_x4(ahi[0], ahi[1], ahi[2], ahi[3], sa_hi + swz(row, col));
                ldsm_x4(alo[0], alo[1], alo[2], alo[3], sa_lo + swz(row, col));
            }
#pragma unroll
            for (int nt = 0; nt < 8; nt += 2) {
                unsigned b0, b1, b2, b3;
                const int row = nt * 8 + (lane & 7) + 8 * (lane >> 4);
                const int col = kk + 8 * ((lane >> 3) & 1);
                ldsm_x4(b0, b1, b2, b3, sb + swz(row, col));
                mma_bf16(acc[nt], ahi, b0, b1);
                mma_bf16(acc[nt], alo, b0, b1);
                mma_bf16(acc[nt + 1], ahi, b2, b3);
                mma_bf16(acc[nt + 1], alo, b2, b3);
            }
        }
    }
    asm volatile("cp.async.wait_group 0;\n");
    // D[j][b] fragments -> partial[ks][b][j]
    const int g = lane >> 2, t4 = lane & 3;
    float *out = partial + (size_t)ks * kInstances * n;
#pragma unroll
    for (int nt = 0; nt < 8; ++nt) {
        const int b = nt * 8 + 2 * t4;
        const int j = m0 + warp * 16 + g;
        out[(size_t)b * n + j] = acc[nt][0];
        out[(size_t)(b + 1) * n + j] = acc[nt][1];
        out[(size_t)b * n + j + 8] = acc[nt][2];
        out[(size_t)(b + 1) * n + j + 8] = acc[nt][3];
    }
}

// -------------------------------------------------------------- LIF update

struct LifParams {
    float v_rest, tau, v_th, r, v_reset, i_ext, dt, drive_w, drive_p;
    int t_ref;
};

// Whether the drive spikes at element idx of the instance-major state (its hash index).
__device__ __forceinline__ bool lif_drive(const LifParams &P, int t, int idx) {
    return t >= 1 && nbg_hash_uniform01(idx, t - 1) < P.drive_p;
}

// One neuron's update: summed arrival `a`, the drive's spike, refractory-gated
// voltage jump, forward-Euler voltage-jump LIF
// (TimeDrivenLIF_Voltage_jump.cpp:49-86), state vv, ls in registers.
__device__ __forceinline__ bool lif_apply(const LifParams &P, float a, bool drive, float &vv, int &ls) {
    if (drive) a = a + P.drive_w;
    if (ls > P.t_ref) vv = vv + a;
    float cur = 0.0f;
    cur = cur + P.r * P.i_ext / P.tau;
    const float aux = (ls > P.t_ref) ? cur + (P.v_rest - vv) / P.tau : 0.0f;
    vv = vv + aux * P.dt;
    ls += 1;
    bool spk = false;
    if (vv > P.v_th) {
        vv = P.v_reset;
        ls = 0;
        spk = true;
    }
    return spk;
}

// --------------------------------------------------------- FP32 CUDA cores

// One step on the FP32 path: cur[b][j] = the sum over i ascending with bit i
// of instance b's spike words set of W[i][j] (kLif = false: the result), then
// the neuron update on it, writing the next step's spike words.
//
// What bounds it: every instance reads the rows of its own spikes (131 of 32
// KiB at 8,192 neurons firing 1.6 % of the steps; 270 MB a step for the 64),
// so the L2, and below that the latency of dependent loads: the kernel before
// this one kept one 4-byte load a thread in flight (13.0 us a step at 2,048
// neurons, 152 at 8,192, and 2.6 more for the update in its own launch).  Here
// a CTA ranks the instance's spikes into a list once, each thread owns two
// neighbouring columns and asks for kGatherRows rows before it adds the first.
// The instances of one column slice are neighbours in the grid, so a row that
// several of them need is read from memory once.  Measured, update included:
// 154 -> 29.0 us a step at 8,192 neurons (9.3 TB/s of row reads), 100 steps
// and their read-out at 2,048 neurons 2.59 -> 0.63 ms.
//
// The external spikes are drawn before the wait for the step before.  Registers
// (kCtas, the CTAs an SM is to hold): where the grid has at most three CTAs an SM
// the 73 that the loads in flight want, else 62 for four: 5.79 -> 4.95 us a step at
// 2,048 neurons (5.65 with 62), 7.35 -> 5.97 (7.17) at 3,072, 8.81 -> 8.63 (9.57
// with 73) at 4,096, 29.1 -> 29.0 (33.7) at 8,192.
constexpr int kGatherThreads = 256;
constexpr int kGatherCols = 2 * kGatherThreads; // columns of a CTA
constexpr int kGatherWords = 256;               // spike words listed at a time (8,192 neurons)
constexpr int kGatherRows = 16;

// bits 0..15 of x to the even bits of the result
__device__ __forceinline__ unsigned spread16(unsigned x) {
    x = (x | x << 8) & 0x00ff00ffu;
    x = (x | x << 4) & 0x0f0f0f0fu;
    x = (x | x << 2) & 0x33333333u;
    return (x | x << 1) & 0x55555555u;
}

template <bool kLif, int kCtas>
__global__ void __launch_bounds__(kGatherThreads, kCtas) k_dense_gather(const float *__restrict__ w,
                                                                 const unsigned *__restrict__ sbits,
                                                                 float *__restrict__ cur, LifParams P, float *v,
                                                                 int *last, unsigned *__restrict__ bits_out,
                                                                 int *__restrict__ counts, int t, int n) {
    __shared__ __align__(16) int list[kGatherWords * 32 + 4];
    __shared__ int warp_cnt[kGatherThreads / 32];
    const int b = blockIdx.x, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int j = blockIdx.y * kGatherCols + 2 * tid;
    const bool has = j < n; // n is a multiple of 128: whole warps
    const float *const col = w + (has ? j : 0);
    const int nw = n / 32;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const size_t at = (size_t)b * n + j;
    // this step's external spikes do not depend on the step before
    const bool d0 = kLif && has && lif_drive(P, t, (int)at), d1 = kLif && has && lif_drive(P, t, (int)at + 1);
    asm volatile("griddepcontrol.wait;" ::: "memory"); // the previous step's spikes, v and last
    float2 vv = make_float2(0.0f, 0.0f);
    int2 ls = make_int2(0, 0);
    if (kLif && has) {
        vv = *reinterpret_cast<const float2 *>(v + at);
        ls = *reinterpret_cast<const int2 *>(last + at);
    }
    float2 sum = make_float2(0.0f, 0.0f);
    for (int w0 = 0; w0 < nw; w0 += kGatherWords) {
        // this chunk's spikes, ascending: one word a thread, ranked by a scan
        unsigned word = tid < kGatherWords && w0 + tid < nw ? __ldcg(sbits + (size_t)b * nw + w0 + tid) : 0u;
        int incl = __popc(word);
        const int own = incl;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        __syncthreads(); // the list and the counts of the chunk before have been read
        if (lane == 31) warp_cnt[wid] = incl;
        __syncthreads();
        int pos = incl - own, total = 0;
#pragma unroll
        for (int k = 0; k < kGatherThreads / 32; ++k) {
            const int q = warp_cnt[k];
            if (k < wid) pos += q;
            total += q;
        }
        for (; word; word &= word - 1u) list[pos++] = (w0 + tid) * 32 + __ffs(word) - 1;
        if (tid < 4) list[total + tid] = 0; // padding: row 0, not added
        __syncthreads();
        for (int k0 = 0; k0 < total; k0 += kGatherRows) {
            float2 x[kGatherRows];
#pragma unroll
            for (int g = 0; g < kGatherRows; g += 4)
                if (k0 + g < total) {
                    const int4 q = *reinterpret_cast<const int4 *>(list + k0 + g);
                    x[g] = __ldg(reinterpret_cast<const float2 *>(col + (size_t)q.x * n));
                    x[g + 1] = __ldg(reinterpret_cast<const float2 *>(col + (size_t)q.y * n));
                    x[g + 2] = __ldg(reinterpret_cast<const float2 *>(col + (size_t)q.z * n));
                    x[g + 3] = __ldg(reinterpret_cast<const float2 *>(col + (size_t)q.w * n));
                }
#pragma unroll
            for (int g = 0; g < kGatherRows; ++g)
                if (k0 + g < total) {
                    sum.x = sum.x + x[g].x;
                    sum.y = sum.y + x[g].y;
                }
        }
    }
    if constexpr (!kLif) {
        if (has) *reinterpret_cast<float2 *>(cur + at) = sum;
    } else {
        bool s0 = false, s1 = false;
        if (has) {
            s0 = lif_apply(P, sum.x, d0, vv.x, ls.x);
            s1 = lif_apply(P, sum.y, d1, vv.y, ls.y);
            *reinterpret_cast<float2 *>(v + at) = vv;
            *reinterpret_cast<int2 *>(last + at) = ls;
        }
        const unsigned even = __ballot_sync(0xffffffffu, s0), odd = __ballot_sync(0xffffffffu, s1);
        if (has && (lane & 15) == 0) // a word is sixteen lanes' pairs
            bits_out[at >> 5] = spread16(even >> lane & 0xffffu) | spread16(odd >> lane & 0xffffu) << 1;
        if (lane == 0 && (even | odd)) atomicAdd(counts, __popc(even) + __popc(odd));
    }
}

__global__ void __launch_bounds__(256) k_dense_lif(LifParams P, const float *__restrict__ partial, int nparts,
                                                   float *__restrict__ v, int *__restrict__ last,
                                                   __nv_bfloat16 *__restrict__ s_out, int *__restrict__ counts, int t,
                                                   int total) {
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    bool spk = false;
    if (idx < total) {
        float a = partial[idx];
        for (int k = 1; k < nparts; ++k) a = a + partial[(size_t)k * total + idx];
        float vv = v[idx];
        int ls = last[idx];
        spk = lif_apply(P, a, lif_drive(P, t, idx), vv, ls);
        v[idx] = vv;
        last[idx] = ls;
        s_out[idx] = __float2bfloat16_rn(spk ? 1.0f : 0.0f);
    }
    const unsigned bal = __ballot_sync(0xffffffffu, spk);
    if ((threadIdx.x & 31) == 0 && bal) atomicAdd(&counts[0], __popc(bal));
}

// The step's neuron update fused into the tcgen05 delivery: the same update
// as k_dense_lif for the elements a CTA completes, with their state loaded
// while the products run; S_t is written in the blocked
// layout the next delivery reads.
struct LifFinish {
    static constexpr bool kActive = true;
    LifParams P;
    float *v;
    int *last;
    __nv_bfloat16 *s_out;
    int *counts;
    int t;
    __device__ void load(int idx, float &vv, int &ls) const {
        vv = v[idx];
        ls = last[idx];
    }
    __device__ bool drive(int idx) const { return lif_drive(P, t, idx); }
    __device__ bool update(int b, int j, int idx, float a, bool drive, float &vv, int &ls) const {
        const bool spk = lif_apply(P, a, drive, vv, ls);
        v[idx] = vv;
        last[idx] = ls;
        s_out[s_blocked(b, j)] = __float2bfloat16_rn(spk ? 1.0f : 0.0f);
        return spk;
    }
    __device__ void count(int k) const {
        if (k) atomicAdd(counts, k);
    }
};

} // namespace

struct nbg_dense {
    int device = 0, B = 64, N = 0, precision = 0;
    bool half_tiles = false; // tcgen05 step: tiles of 64 post neurons instead of 128
    bool few_ctas = false;   // FP32 step: at most three CTAs an SM
    LifParams P{};
    DevBuf<float> w, partial, v;
    DevBuf<__nv_bfloat16> whi, wlo, s[2];
    DevBuf<unsigned> bits[2];
    DevBuf<int> last, err;
    // conversions and deliveries outside the step loop: the caller's bytes, the
    // spikes in the path's layout, the partial sums and the result.  Made at
    // first use, one call at a time (io_mu), apart from the simulation's state
    std::mutex io_mu;
    DevBuf<uint8_t> io_bytes;
    DevBuf<__nv_bfloat16> io_s;
    DevBuf<float> io_part, io_out;
    DevBuf<int> cnt; // spikes per step of a run call
    std::vector<cudaEvent_t> dev_pool; // delivery start/stop events, 2 per step
    int next_t = 0;
    bool ran = false;
    std::vector<int> counts_host;
    cudaStream_t stream = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr, evd0 = nullptr, evd1 = nullptr;
    double last_ms = 0.0, last_delivery_ms = 0.0;
    int64_t last_launches = 0;
};

namespace {

__global__ void k_dense_reset(float *__restrict__ v, int *__restrict__ last, float v0, int total) {
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= total) return;
    v[idx] = v0;
    last[idx] = 10000;
}

// On the engine's stream, which nothing on the default stream is ordered with,
// and done on return.
nbg_status dense_reset(nbg_dense *d) {
    const int total = d->B * d->N;
    cudaStream_t st = d->stream;
    k_dense_reset<<<(total + 255) / 256, 256, 0, st>>>(d->v.p, d->last.p, d->P.v_reset, total); // V_reset + random_mu (legacy init)
    NBG_CUDA(cudaGetLastError());
    for (int k = 0; k < 2; ++k) {
        NBG_CUDA(cudaMemsetAsync(d->s[k].p, 0, d->s[k].n * sizeof(__nv_bfloat16), st));
        NBG_CUDA(cudaMemsetAsync(d->bits[k].p, 0, d->bits[k].n * sizeof(unsigned), st));
    }
    NBG_CUDA(cudaStreamSynchronize(st));
    d->next_t = 0;
    d->ran = false;
    d->counts_host.clear();
    return NBG_OK;
}

int layout_of(const nbg_dense *d) {
    return d->precision == NBG_DENSE_SPLIT_BF16 ? kLayoutBlocked
           : d->precision == NBG_DENSE_FP32     ? kLayoutBits
                                                : kLayoutRows;
}

dim3 gather_grid(const nbg_dense *d) { return dim3(d->B, (d->N + kGatherCols - 1) / kGatherCols); }

// A step's launch configuration, overlapping the step before (programmatic
// dependent launch).
cudaLaunchConfig_t step_config(const nbg_dense *d, dim3 grid, int threads, size_t smem, cudaLaunchAttribute (&attr)[2],
                               int cluster_y = 1) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = d->stream;
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = attr[1].val.clusterDim.z = 1;
    attr[1].val.clusterDim.y = (unsigned)cluster_y;
    cfg.attrs = attr;
    cfg.numAttrs = cluster_y > 1 ? 2 : 1;
    return cfg;
}

} // namespace

extern "C" {

nbg_status nbg_dense_create(int instances, int neurons, const float *w, const nbg_layer_desc *lif,
                            float drive_rate_hz, float drive_weight, float dt_ms, int precision, int device,
                            nbg_dense **out) {
    if (!out || !w || !lif) return nbg_fail(NBG_ERR_INVALID, "null argument");
    *out = nullptr;
    if (instances != kInstances) return nbg_fail(NBG_ERR_UNSUPPORTED, "instances must be %d", kInstances);
    if (neurons <= 0 || neurons % kBM != 0 || (neurons / kSplitK) % kBK != 0)
        return nbg_fail(NBG_ERR_INVALID, "neurons must be a positive multiple of %d", kBM);
    if (lif->model != NBG_MODEL_LIF_VJ) return nbg_fail(NBG_ERR_UNSUPPORTED, "the dense engine runs the voltage-jump LIF");
    if (precision != NBG_DENSE_SPLIT_BF16 && precision != NBG_DENSE_FP32 && precision != NBG_DENSE_SPLIT_BF16_SYNC)
        return nbg_fail(NBG_ERR_INVALID, "unknown precision %d", precision);
    if (!(dt_ms > 0.0f) || !(lif->f[1] != 0.0f)) return nbg_fail(NBG_ERR_INVALID, "dt and tau must be non-zero");
    auto *d = new nbg_dense();
    auto bail = [&](nbg_status st) {
        delete d;
        return st;
    };
    d->device = device;
    d->B = instances;
    d->N = neurons;
    d->precision = precision;
    d->P.v_rest = lif->f[0];
    d->P.tau = lif->f[1];
    d->P.v_th = lif->f[2];
    d->P.r = lif->f[3];
    d->P.v_reset = lif->f[4] + lif->f[5];
    d->P.i_ext = lif->f[6];
    d->P.t_ref = lif->ip[0];
    d->P.dt = dt_ms;
    d->P.drive_w = drive_weight;
    {
        float rate = drive_rate_hz > 0.0f ? drive_rate_hz : 0.0f;
        float p = rate * dt_ms * 0.001f;
        d->P.drive_p = p < 1.0f ? p : 1.0f;
    }
    if (cudaSetDevice(device) != cudaSuccess) return bail(nbg_fail(NBG_ERR_CUDA, "cudaSetDevice(%d) failed", device));
    const size_t nn = (size_t)neurons * neurons, tot = (size_t)instances * neurons;
    cudaError_t ce = cudaSuccess;
    auto chk = [&](cudaError_t x) {
        if (ce == cudaSuccess) ce = x;
    };
    int sms = 0;
    chk(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    const dim3 gg = gather_grid(d);
    d->few_ctas = (int)(gg.x * gg.y) <= 3 * sms;
    d->half_tiles = neurons / 64 * kSplitK <= sms;
    chk(cudaStreamCreateWithFlags(&d->stream, cudaStreamNonBlocking));
    chk(cudaEventCreate(&d->ev0));
    chk(cudaEventCreate(&d->ev1));
    chk(cudaEventCreate(&d->evd0));
    chk(cudaEventCreate(&d->evd1));
    chk(d->v.alloc(tot));
    chk(d->last.alloc(tot));
    chk(d->err.alloc(1));
    if (ce == cudaSuccess) chk(cudaMemsetAsync(d->err.p, 0, sizeof(int), d->stream));
    if (precision == NBG_DENSE_SPLIT_BF16_SYNC) chk(d->partial.alloc((size_t)kSplitK * tot));
    for (int k = 0; k < 2; ++k) {
        chk(d->s[k].alloc(tot));
        chk(d->bits[k].alloc(tot / 32));
    }
    if (precision == NBG_DENSE_FP32) {
        chk(d->w.alloc(nn));
        if (ce == cudaSuccess) chk(cudaMemcpyAsync(d->w.p, w, nn * sizeof(float), cudaMemcpyHostToDevice, d->stream));
    } else {
        DevBuf<float> tmp;
        chk(tmp.alloc(nn));
        chk(d->whi.alloc(nn));
        chk(d->wlo.alloc(nn));
        if (ce == cudaSuccess) chk(cudaMemcpy(tmp.p, w, nn * sizeof(float), cudaMemcpyHostToDevice));
        if (ce == cudaSuccess && precision == NBG_DENSE_SPLIT_BF16) {
            k_split_tile<<<(unsigned)((nn + 255) / 256), 256>>>(tmp.p, d->whi.p, d->wlo.p, neurons);
            chk(cudaGetLastError());
            chk(cudaDeviceSynchronize());
            if (ce == cudaSuccess)
                chk(cudaFuncSetAttribute(umma::k_dense_umma<umma::NoFinish>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, umma::kSmemBytes));
            // of the fused step only the tile this engine runs: an attribute loads its kernel
            if (ce == cudaSuccess)
                chk(d->half_tiles ? cudaFuncSetAttribute(umma::k_dense_umma<LifFinish, 64>,
                                                         cudaFuncAttributeMaxDynamicSharedMemorySize, umma::Tile<64>::fused_smem)
                                  : cudaFuncSetAttribute(umma::k_dense_umma<LifFinish, 128>,
                                                         cudaFuncAttributeMaxDynamicSharedMemorySize, umma::Tile<128>::fused_smem));
        } else if (ce == cudaSuccess) {
            dim3 grid(neurons / 32, neurons / 32), block(32, 8);
            k_split_transpose<<<grid, block>>>(tmp.p, d->whi.p, d->wlo.p, neurons);
            chk(cudaGetLastError());
            chk(cudaDeviceSynchronize());
        }
        if (ce == cudaSuccess)
            chk(cudaFuncSetAttribute(k_dense_gemm, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGemmSmem));
    }
    if (ce != cudaSuccess)
        return bail(nbg_fail(ce == cudaErrorMemoryAllocation ? NBG_ERR_OOM : NBG_ERR_CUDA, "dense create: %s",
                             cudaGetErrorString(ce)));
    nbg_status st = dense_reset(d);
    if (st != NBG_OK) return bail(st);
    *out = d;
    return NBG_OK;
}

nbg_status nbg_dense_destroy(nbg_dense *d) {
    if (!d) return NBG_OK;
    cudaSetDevice(d->device);
    if (d->stream) cudaStreamSynchronize(d->stream);
    for (cudaEvent_t e : {d->ev0, d->ev1, d->evd0, d->evd1})
        if (e) cudaEventDestroy(e);
    for (cudaEvent_t e : d->dev_pool) cudaEventDestroy(e);
    if (d->stream) cudaStreamDestroy(d->stream);
    delete d;
    return NBG_OK;
}

nbg_status nbg_dense_reset(nbg_dense *d) {
    if (!d) return nbg_fail(NBG_ERR_INVALID, "null engine");
    NBG_CUDA(cudaSetDevice(d->device));
    NBG_CUDA(cudaStreamSynchronize(d->stream));
    return dense_reset(d);
}

nbg_status nbg_dense_run(nbg_dense *d, int steps) {
    if (!d) return nbg_fail(NBG_ERR_INVALID, "null engine");
    if (steps <= 0) return nbg_fail(NBG_ERR_INVALID, "steps must be positive");
    NBG_CUDA(cudaSetDevice(d->device));
    const int count = d->ran ? steps : steps + 1;
    const int total = d->B * d->N;
    std::vector<int> cnt((size_t)count, 0);
    if (d->cnt.n < (size_t)count) NBG_CUDA(d->cnt.alloc((size_t)count));
    DevBuf<int> &dcnt = d->cnt;
    NBG_CUDA(cudaMemsetAsync(dcnt.p, 0, count * sizeof(int), d->stream));
    // event pairs bracketing every delivery launch of the two-launch path (reused across calls)
    const bool sync_path = d->precision == NBG_DENSE_SPLIT_BF16_SYNC;
    const int chunk = 256;
    while (sync_path && (int)d->dev_pool.size() < 2 * chunk) {
        cudaEvent_t ev;
        NBG_CUDA(cudaEventCreate(&ev));
        d->dev_pool.push_back(ev);
    }
    double dms = 0.0;
    NBG_CUDA(cudaEventRecord(d->ev0, d->stream));
    cudaLaunchAttribute attr[2];
    const int kept = umma::kept_iters(d->N, kSplitK);
    for (int k0 = 0; k0 < count; k0 += chunk) {
        const int k1 = std::min(count, k0 + chunk);
        for (int k = k0; k < k1; ++k) {
            const int t = d->next_t + k;
            const int in = (t + 1) & 1, outp = t & 1; // S_{t-1} lives in buffer (t-1)&1
            if (d->precision == NBG_DENSE_SPLIT_BF16) { // tcgen05: delivery and update in one launch
                const LifFinish fin{d->P, d->v.p, d->last.p, d->s[outp].p, dcnt.p + k, t};
                const int m = d->half_tiles ? 64 : 128;
                const cudaLaunchConfig_t cfg =
                    step_config(d, dim3(d->N / m, kSplitK), umma::threads<LifFinish>(),
                                d->half_tiles ? umma::Tile<64>::fused_smem : umma::Tile<128>::fused_smem, attr, kSplitK);
                NBG_CUDA(cudaLaunchKernelEx(
                    &cfg, d->half_tiles ? umma::k_dense_umma<LifFinish, 64> : umma::k_dense_umma<LifFinish, 128>,
                    (const __nv_bfloat16 *)d->whi.p, (const __nv_bfloat16 *)d->wlo.p, (const __nv_bfloat16 *)d->s[in].p,
                    (float *)nullptr, d->N, (int)kSplitK, t & 1, kept, d->err.p, fin));
                continue;
            }
            if (d->precision == NBG_DENSE_FP32) { // gather and update in one launch
                const cudaLaunchConfig_t cfg = step_config(d, gather_grid(d), kGatherThreads, 0, attr);
                NBG_CUDA(cudaLaunchKernelEx(&cfg, d->few_ctas ? k_dense_gather<true, 1> : k_dense_gather<true, 4>,
                                            (const float *)d->w.p, (const unsigned *)d->bits[in].p, (float *)nullptr,
                                            d->P, d->v.p, d->last.p, d->bits[outp].p, dcnt.p + k, t, d->N));
                continue;
            }
            NBG_CUDA(cudaEventRecord(d->dev_pool[2 * (k - k0)], d->stream));
            k_dense_gemm<<<dim3(d->N / kBM, kSplitK), kGemmThreads, kGemmSmem, d->stream>>>(d->whi.p, d->wlo.p, d->s[in].p,
                                                                                          d->partial.p, d->N);
            NBG_CUDA(cudaEventRecord(d->dev_pool[2 * (k - k0) + 1], d->stream));
            k_dense_lif<<<(total + 255) / 256, 256, 0, d->stream>>>(d->P, d->partial.p, kSplitK, d->v.p, d->last.p,
                                                                    d->s[outp].p, dcnt.p + k, t, total);
        }
        NBG_CUDA(cudaGetLastError());
        if (!sync_path) continue; // one launch per step, no per-step events (they would break the overlap)
        NBG_CUDA(cudaEventSynchronize(d->dev_pool[2 * (k1 - 1 - k0) + 1]));
        for (int k = k0; k < k1; ++k) {
            float x = 0.0f;
            NBG_CUDA(cudaEventElapsedTime(&x, d->dev_pool[2 * (k - k0)], d->dev_pool[2 * (k - k0) + 1]));
            dms += x;
        }
    }
    NBG_CUDA(cudaEventRecord(d->ev1, d->stream));
    NBG_CUDA(cudaStreamSynchronize(d->stream));
    float ms = 0.0f;
    NBG_CUDA(cudaEventElapsedTime(&ms, d->ev0, d->ev1));
    d->last_ms = ms;
    d->last_delivery_ms = sync_path ? dms : ms; // else the whole step is the delivery launch
    d->last_launches = (sync_path ? 2LL : 1LL) * count;
    NBG_CUDA(cudaMemcpy(cnt.data(), dcnt.p, count * sizeof(int), cudaMemcpyDeviceToHost));
    int errv = 0;
    NBG_CUDA(cudaMemcpy(&errv, d->err.p, sizeof(int), cudaMemcpyDeviceToHost));
    if (errv) return nbg_fail(NBG_ERR_TIMEOUT, "tensor-core delivery gave up waiting on a pipeline barrier");
    d->counts_host.insert(d->counts_host.end(), cnt.begin(), cnt.end());
    d->next_t += count;
    d->ran = true;
    return NBG_OK;
}

nbg_status nbg_dense_get_state(nbg_dense *d, float *v, int32_t *last) {
    if (!d) return nbg_fail(NBG_ERR_INVALID, "null engine");
    NBG_CUDA(cudaSetDevice(d->device));
    NBG_CUDA(cudaStreamSynchronize(d->stream));
    const size_t tot = (size_t)d->B * d->N;
    if (v) NBG_CUDA(cudaMemcpy(v, d->v.p, tot * sizeof(float), cudaMemcpyDeviceToHost));
    if (last) NBG_CUDA(cudaMemcpy(last, d->last.p, tot * sizeof(int), cudaMemcpyDeviceToHost));
    return NBG_OK;
}

nbg_status nbg_dense_num_steps(nbg_dense *d, int64_t *n) {
    if (!d || !n) return nbg_fail(NBG_ERR_INVALID, "null argument");
    *n = (int64_t)d->counts_host.size();
    return NBG_OK;
}

nbg_status nbg_dense_spike_counts(nbg_dense *d, int32_t *counts) {
    if (!d || !counts) return nbg_fail(NBG_ERR_INVALID, "null argument");
    if (!d->counts_host.empty())
        std::memcpy(counts, d->counts_host.data(), d->counts_host.size() * sizeof(int32_t));
    return NBG_OK;
}

nbg_status nbg_dense_get_spikes(nbg_dense *d, uint8_t *s) {
    if (!d || !s) return nbg_fail(NBG_ERR_INVALID, "null argument");
    NBG_CUDA(cudaSetDevice(d->device));
    NBG_CUDA(cudaStreamSynchronize(d->stream));
    const size_t tot = (size_t)d->B * d->N;
    const int par = (d->next_t - 1) & 1;
    if (d->next_t == 0) {
        std::memset(s, 0, tot);
        return NBG_OK;
    }
    std::lock_guard<std::mutex> lock(d->io_mu);
    if (d->io_bytes.n < tot) NBG_CUDA(d->io_bytes.alloc(tot));
    const int groups = (int)(tot / 8), grid = (groups + 255) / 256;
    switch (layout_of(d)) {
    case kLayoutBlocked: k_spikes_out<kLayoutBlocked><<<grid, 256, 0, d->stream>>>(d->s[par].p, d->io_bytes.p, d->N, groups); break;
    case kLayoutRows: k_spikes_out<kLayoutRows><<<grid, 256, 0, d->stream>>>(d->s[par].p, d->io_bytes.p, d->N, groups); break;
    default: k_spikes_out<kLayoutBits><<<grid, 256, 0, d->stream>>>(d->bits[par].p, d->io_bytes.p, d->N, groups); break;
    }
    NBG_CUDA(cudaGetLastError());
    NBG_CUDA(cudaMemcpyAsync(s, d->io_bytes.p, tot, cudaMemcpyDeviceToHost, d->stream));
    NBG_CUDA(cudaStreamSynchronize(d->stream));
    return NBG_OK;
}

nbg_status nbg_dense_deliver(nbg_dense *d, const uint8_t *s, float *out) {
    if (!d || !s || !out) return nbg_fail(NBG_ERR_INVALID, "null argument");
    NBG_CUDA(cudaSetDevice(d->device));
    const size_t tot = (size_t)d->B * d->N;
    std::lock_guard<std::mutex> lock(d->io_mu);
    if (d->io_bytes.n < tot) NBG_CUDA(d->io_bytes.alloc(tot));
    if (d->io_s.n < tot) NBG_CUDA(d->io_s.alloc(tot));
    if (d->io_out.n < tot) NBG_CUDA(d->io_out.alloc(tot));
    const bool split = d->precision != NBG_DENSE_FP32;
    if (split && d->io_part.n < (size_t)kSplitK * tot) NBG_CUDA(d->io_part.alloc((size_t)kSplitK * tot));
    const int groups = (int)(tot / 8), grid8 = (groups + 255) / 256;
    cudaStream_t st = d->stream;
    NBG_CUDA(cudaMemcpyAsync(d->io_bytes.p, s, tot, cudaMemcpyHostToDevice, st));
    if (d->precision == NBG_DENSE_SPLIT_BF16) {
        k_spikes_in<kLayoutBlocked><<<grid8, 256, 0, st>>>(d->io_bytes.p, d->io_s.p, d->N, groups);
        umma::k_dense_umma<umma::NoFinish><<<dim3(d->N / umma::kM, kSplitK), umma::threads<umma::NoFinish>(), umma::kSmemBytes, st>>>(
            d->whi.p, d->wlo.p, d->io_s.p, d->io_part.p, d->N, kSplitK, 0, 0, d->err.p, umma::NoFinish{});
    } else if (d->precision == NBG_DENSE_SPLIT_BF16_SYNC) {
        k_spikes_in<kLayoutRows><<<grid8, 256, 0, st>>>(d->io_bytes.p, d->io_s.p, d->N, groups);
        k_dense_gemm<<<dim3(d->N / kBM, kSplitK), kGemmThreads, kGemmSmem, st>>>(d->whi.p, d->wlo.p, d->io_s.p,
                                                                               d->io_part.p, d->N);
    } else {
        unsigned *const bits = reinterpret_cast<unsigned *>(d->io_s.p);
        k_spikes_in<kLayoutBits><<<grid8, 256, 0, st>>>(d->io_bytes.p, bits, d->N, groups);
        k_dense_gather<false, 1><<<gather_grid(d), kGatherThreads, 0, st>>>(d->w.p, bits, d->io_out.p, d->P, nullptr, nullptr,
                                                                         nullptr, nullptr, 0, d->N);
    }
    if (split) k_sum_split_partials<<<(unsigned)((tot + 255) / 256), 256, 0, st>>>(d->io_part.p, d->io_out.p, (int)tot);
    NBG_CUDA(cudaGetLastError());
    NBG_CUDA(cudaMemcpyAsync(out, d->io_out.p, tot * sizeof(float), cudaMemcpyDeviceToHost, st));
    int errv = 0;
    if (d->precision == NBG_DENSE_SPLIT_BF16) // the only path that waits
        NBG_CUDA(cudaMemcpyAsync(&errv, d->err.p, sizeof(int), cudaMemcpyDeviceToHost, st));
    NBG_CUDA(cudaStreamSynchronize(st));
    if (errv) return nbg_fail(NBG_ERR_TIMEOUT, "tensor-core delivery gave up waiting on a pipeline barrier");
    return NBG_OK;
}

nbg_status nbg_dense_profile(nbg_dense *d, double *total_ms, double *delivery_ms, int64_t *launches) {
    if (!d) return nbg_fail(NBG_ERR_INVALID, "null engine");
    if (total_ms) *total_ms = d->last_ms;
    if (delivery_ms) *delivery_ms = d->last_delivery_ms;
    if (launches) *launches = d->last_launches;
    return NBG_OK;
}

} // extern "C"

// ---------------------------------------------------------------------------
// Delivery without allocation (nbg_dense_deliver_noalloc): the split-K
// partial sums go to a file-scope device array instead of a buffer the
// library allocates.  Host code must not use `g_noalloc_partial` as a device
// address: it is a host-side stand-in for the symbol.  The real address is
// looked up once per device with cudaGetSymbolAddress.

static __device__ __align__(256) float g_noalloc_partial[kSplitK * kInstances * NBG_DENSE_NOALLOC_MAX_NEURONS];

namespace {

constexpr int kNoAllocMaxDevices = 64;
std::mutex g_noalloc_mu;
float *g_noalloc_scratch[kNoAllocMaxDevices] = {};

} // namespace

extern "C" nbg_status nbg_dense_deliver_noalloc(const void *w_hi_t, const void *w_lo_t, const void *spikes,
                                                float *out, int neurons, void *stream) {
    if (!w_hi_t || !w_lo_t || !spikes || !out) return nbg_fail(NBG_ERR_INVALID, "null argument");
    // the GEMM reads all three inputs with 16-byte cp.async copies
    if (((uintptr_t)w_hi_t | (uintptr_t)w_lo_t | (uintptr_t)spikes) & 15u)
        return nbg_fail(NBG_ERR_INVALID, "w_hi_t, w_lo_t and spikes must be 16-byte aligned");
    if ((uintptr_t)out & 3u) return nbg_fail(NBG_ERR_INVALID, "out must be 4-byte aligned");
    if (neurons <= 0 || neurons % kBM != 0 || (neurons / kSplitK) % kBK != 0)
        return nbg_fail(NBG_ERR_INVALID, "neurons must be a positive multiple of %d", kBM);
    if (neurons > NBG_DENSE_NOALLOC_MAX_NEURONS)
        return nbg_fail(NBG_ERR_INVALID, "neurons = %d exceeds the no-allocation limit of %d", neurons,
                        NBG_DENSE_NOALLOC_MAX_NEURONS);
    int dev = 0;
    NBG_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kNoAllocMaxDevices) return nbg_fail(NBG_ERR_UNSUPPORTED, "device ordinal %d too large", dev);
    float *scratch = nullptr;
    {
        std::lock_guard<std::mutex> lock(g_noalloc_mu);
        if (!g_noalloc_scratch[dev]) { // first call on this device: set-up, with `dev` current
            void *p = nullptr;
            NBG_CUDA(cudaGetSymbolAddress(&p, g_noalloc_partial));
            NBG_CUDA(cudaFuncSetAttribute(k_dense_gemm, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGemmSmem));
            g_noalloc_scratch[dev] = static_cast<float *>(p);
        }
        scratch = g_noalloc_scratch[dev];
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    dim3 grid(neurons / kBM, kSplitK);
    k_dense_gemm<<<grid, kGemmThreads, kGemmSmem, st>>>(static_cast<const __nv_bfloat16 *>(w_hi_t),
                                                         static_cast<const __nv_bfloat16 *>(w_lo_t),
                                                         static_cast<const __nv_bfloat16 *>(spikes), scratch, neurons);
    const int total = kInstances * neurons;
    k_sum_split_partials<<<(total + 255) / 256, 256, 0, st>>>(scratch, out, total);
    NBG_CUDA(cudaGetLastError());
    return NBG_OK;
}
