// nbg_adjoint_f32.cu -- FP32 products of the recurrent LIF on the CUDA cores,
// for the shapes the split-BF16 tensor-core path does not take (C ABI in
// include/nbg_adjoint.h): the recurrent product fused with the forward or
// adjoint step that consumes it, a plain product of the same form, and the
// weight-gradient products.
//
// Before these, every such product was nbg_small_gemm: one warp per output,
// each term two loads from L1/L2 -- and, where an operand's K index is its
// row index (S^T dI), one sector per lane and load.
#include <cuda_runtime.h>

#include <algorithm>

#include "nbg_adjoint.h"
#include "nbg_common.cuh"
#include "nbg_lif_grad.cuh"

namespace {

// (d.x, d.y) += (a.x * b.x, a.y * b.y), each a fused multiply-add rounded
// once: one packed instruction for two terms.
__device__ __forceinline__ void fma2(unsigned long long &d, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ void add2(unsigned long long &d, unsigned long long a) {
    asm("add.rn.f32x2 %0, %0, %1;" : "+l"(d) : "l"(a));
}
__device__ __forceinline__ unsigned long long pack2(float x, float y) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ float2 unpack2(unsigned long long v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}

// The sum of eight values in pairs (of fewer: the others zero).
__device__ __forceinline__ float tree8(const float (&x)[8]) {
    return ((x[0] + x[1]) + (x[2] + x[3])) + ((x[4] + x[5]) + (x[6] + x[7]));
}

// Asynchronous copy global -> shared of kBytes (4 or 16), zero-filled when
// !valid (src must still be a valid address).
template <int kBytes>
__device__ __forceinline__ void copy_async(void *dst, const void *src, bool valid) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    const int n = valid ? kBytes : 0;
    if constexpr (kBytes == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int kLeft> __device__ __forceinline__ void copy_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(kLeft) : "memory");
}

// ------------------------------------------------------------- A times W^T
//
// P[r][j] = sum over k of A[r][k] W[j][k], both operands contiguous in k, and
// an epilogue on every P: a plain store, the smoothed forward step or the
// adjoint step.
//
// What bounds it: a backward is one such product per time step, each waiting
// for the one before, of a few rows (32 x 512 by 512 x 512: 8 MFLOP), so the
// chip is filled by splitting K, not by tiles.  A CTA of eight warps owns a
// 32 x 32 tile over one K range; its warps take the K granules of four in
// turn (4 x 8 outputs a thread, pairs of k packed), the eight partial tiles
// are added in shared memory, and up to eight CTAs of a cluster split K
// further, each sending every owner its rows through distributed shared
// memory.  The sums are chains of at most K / 16 terms over the splits, then
// trees in pairs, in an order that the shape alone fixes.  W does not change
// during a sweep: its tiles are requested before the wait for the step before
// (programmatic dependent launch).
//
// Measured: the steps of a training step of 32 rows, 512 neurons, 250 steps
// (forward by gather) 21.2 -> 1.66 ms in all; smoothed, 12 rows, 300 neurons,
// 60 steps each way, 1,241 -> 545 us.  Error against 64 bits at 64 x 1000 x
// 1000: 1.23e-7 -> 1.05e-7 of the norm.
constexpr int kTile = 32;
constexpr int kNtThreads = 256, kNtWarps = kNtThreads / 32;
constexpr int kNtChunk = 256;              // k per stage at most
constexpr int kRedLd = 36;                 // partial tiles: 32 lanes of a store in 32 banks
constexpr int kRecvFloats = kTile * kTile; // partials of this rank's rows from every rank

__host__ __device__ constexpr int nt_ld(int kc) { return kc + 4; } // kc a multiple of 8: rows 16 bytes apart mod 128
constexpr size_t nt_smem_bytes(int stages, int kc) {
    const int ops = stages * 2 * kTile * nt_ld(kc), red = kNtWarps * kTile * kRedLd;
    return (size_t)(kRecvFloats + (ops > red ? ops : red)) * sizeof(float);
}

struct NtShape {
    int M, N, K;
    int ranks; // CTAs of a cluster along K
    int per;   // k per rank, a multiple of 8
    int kc;    // k per stage, a multiple of 8
    int stages;
    int vec;   // operand rows are 16-byte aligned and K % 4 == 0
};

template <int kBytes>
__device__ __forceinline__ void nt_load(float *dst, const float *src, int row0, int rows, int k0, int k_end, int ld,
                                        int kc) {
    constexpr int kF = kBytes / 4;
    const int pieces = kc / kF;
    for (int e = threadIdx.x; e < kTile * pieces; e += kNtThreads) {
        const int r = e / pieces, c = (e - r * pieces) * kF;
        const bool ok = row0 + r < rows && k0 + c < k_end;
        copy_async<kBytes>(dst + r * nt_ld(kc) + c, ok ? src + (size_t)(row0 + r) * ld + k0 + c : src, ok);
    }
}

// kE: elements of the tile a thread finishes, at most (4 / ranks, at least
// 1).  With K split (kE <= 2) their operands are loaded ahead of the product;
// an unsplit K has enough tiles to hide them behind.
template <class Epi, int kE>
__global__ void __launch_bounds__(kNtThreads, 2) k_product_nt(const float *__restrict__ A, const float *__restrict__ W,
                                                           const NtShape sh, const Epi epi) {
    extern __shared__ __align__(16) float nt_smem[];
    const int kc = sh.kc, ld = nt_ld(kc);
    float *const recv = nt_smem;
    float *const ops = nt_smem + kRecvFloats; // [stage][A tile, W tile], then the partial tiles
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int rank = sh.ranks > 1 ? (int)(blockIdx.x % (unsigned)sh.ranks) : 0; // = %cluster_ctarank
    const int j0 = (int)(blockIdx.x / (unsigned)sh.ranks) * kTile;
    const long long row_tile = (long long)blockIdx.z * gridDim.y + blockIdx.y; // of a cluster's CTAs the same
    if (row_tile * kTile >= sh.M) return;
    const int r0 = (int)row_tile * kTile;
    const int k_beg = min(rank * sh.per, sh.K), k_end = min(k_beg + sh.per, sh.K);
    const int chunks = A ? (k_end - k_beg + kc - 1) / kc : 0;
    const int stage_floats = 2 * kTile * ld;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (sh.ranks > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    auto load = [&](float *dst, const float *src, int row0, int rows, int c) {
        const int k0 = k_beg + c * kc;
        if (sh.vec) nt_load<16>(dst, src, row0, rows, k0, k_end, sh.K, kc);
        else nt_load<4>(dst, src, row0, rows, k0, k_end, sh.K, kc);
    };
    const int ahead = min(sh.stages, chunks);
    for (int c = 0; c < ahead; ++c) load(ops + c * stage_floats + kTile * ld, W, j0, sh.N, c);
    // this thread's elements of the tile: rank's rows [rank * 32 / ranks, ...)
    const int own = kRecvFloats / sh.ranks;
    constexpr bool kEarly = kE <= 2;
    typename Epi::Regs er[kE];
    auto mine = [&](int q, int &r, int &j) { // element q of this thread: its row and column, false if it has none
        const int e = tid + q * kNtThreads, g = rank * own + e;
        r = r0 + (g >> 5);
        j = j0 + (g & 31);
        return e < own && r < sh.M && j < sh.N;
    };
    int r, j;
    if constexpr (kEarly) {
#pragma unroll
        for (int q = 0; q < kE; ++q)
            if (mine(q, r, j)) epi.before(er[q], r, j);
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    for (int c = 0; c < ahead; ++c) {
        load(ops + c * stage_floats, A, r0, sh.M, c);
        copy_commit();
    }
    if constexpr (kEarly) {
#pragma unroll
        for (int q = 0; q < kE; ++q)
            if (mine(q, r, j)) epi.after(er[q], r, j);
    }
    // rows bg + 8 r, columns jg + 4 q: the eight (four) rows that a warp reads
    // together are neighbours, in different banks
    const int bg = lane & 7, jg = lane >> 3;
    unsigned long long acc[4][8];
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int q = 0; q < 8; ++q) acc[r][q] = 0ull;
    for (int c = 0; c < chunks; ++c) {
        if (c + 1 < chunks && sh.stages > 1) copy_wait<1>();
        else copy_wait<0>();
        __syncthreads();
        const float *const as = ops + (c % sh.stages) * stage_floats, *const ws = as + kTile * ld;
        const int len = min(kc, k_end - k_beg - c * kc);
        for (int k = warp * 4; k < len; k += kNtWarps * 4) {
            ulonglong2 a[4], w[8];
#pragma unroll
            for (int r = 0; r < 4; ++r) a[r] = *reinterpret_cast<const ulonglong2 *>(as + (bg + 8 * r) * ld + k);
#pragma unroll
            for (int q = 0; q < 8; ++q) w[q] = *reinterpret_cast<const ulonglong2 *>(ws + (jg + 4 * q) * ld + k);
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    fma2(acc[r][q], a[r].x, w[q].x);
                    fma2(acc[r][q], a[r].y, w[q].y);
                }
        }
        __syncthreads();
        if (c + sh.stages < chunks) {
            float *const st = ops + (c % sh.stages) * stage_floats;
            load(st, A, r0, sh.M, c + sh.stages);
            load(st + kTile * ld, W, j0, sh.N, c + sh.stages);
            copy_commit();
        }
    }
    // the warps' partial tiles, added in pairs
    float *const red = ops;
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const float2 x = unpack2(acc[r][q]);
            red[(warp * kTile + bg + 8 * r) * kRedLd + jg + 4 * q] = x.x + x.y;
        }
    __syncthreads();
    float sum[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int e = tid + q * kNtThreads;
        const float *p = red + (e >> 5) * kRedLd + (e & 31);
        float x[kNtWarps];
#pragma unroll
        for (int w = 0; w < kNtWarps; ++w) x[w] = p[w * kTile * kRedLd];
        sum[q] = tree8(x);
    }
    if (sh.ranks > 1) { // every CTA's sums to the owners of their rows
        asm volatile("barrier.cluster.wait.aligned;" ::: "memory"); // the peers have started
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int e = tid + q * kNtThreads, to = e / own;
            uint32_t ra;
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
                         : "=r"(ra)
                         : "r"((uint32_t)__cvta_generic_to_shared(recv + rank * own + (e - to * own))), "r"(to));
            asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(ra), "f"(sum[q]) : "memory");
        }
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
#pragma unroll
    for (int q = 0; q < kE; ++q) {
        if (!mine(q, r, j)) continue;
        if constexpr (!kEarly) {
            epi.before(er[q], r, j);
            epi.after(er[q], r, j);
        }
        float x = sum[q];
        if (sh.ranks > 1) {
            const int e = tid + q * kNtThreads;
            float y[8];
#pragma unroll
            for (int s = 0; s < 8; ++s) y[s] = s < sh.ranks ? recv[s * own + e] : 0.0f;
            x = tree8(y);
        }
        epi.apply(er[q], x, r, j);
    }
}

struct StoreEpi {
    float *C;
    int N;
    struct Regs {};
    __device__ void before(Regs &, int, int) const {}
    __device__ void after(Regs &, int, int) const {}
    __device__ void apply(const Regs &, float x, int r, int j) const { C[(size_t)r * N + j] = x; }
};

// The smoothed forward step of nbg_lif_forward_step with I = product + xi.
struct SmoothStepEpi {
    const float *xi;
    float *v, *s_out, *u_rec, *vprev_rec, *z;
    unsigned char *m_rec;
    float c_t;
    const float *alpha, *theta;
    nbg_lif_grad_params p;
    int N;
    struct Regs {
        float xi, al, th, v, z;
    };
    __device__ void before(Regs &g, int r, int j) const {
        g.xi = xi[(size_t)r * N + j];
        g.al = alpha[j];
        g.th = theta[j];
    }
    __device__ void after(Regs &g, int r, int j) const {
        g.v = v[(size_t)r * N + j];
        g.z = z ? z[(size_t)r * N + j] : 0.0f;
    }
    __device__ void apply(const Regs &g, float x, int r, int j) const {
        const size_t idx = (size_t)r * N + j;
        const float I = x + g.xi;
        const float u = g.v + g.al * (p.v_rest - g.v) + I;
        const float s = 1.0f / (1.0f + expf(-p.slope * (u - g.th)));
        v[idx] = u - s * (u - p.v_reset);
        s_out[idx] = s;
        if (u_rec) u_rec[idx] = u;
        if (m_rec) m_rec[idx] = 1;
        if (vprev_rec) vprev_rec[idx] = g.v;
        if (z) z[idx] = g.z + c_t * s;
    }
};

// The adjoint step of nbg_lif_adjoint_step with g_ext = product (none in the
// sweep's first step).
struct AdjointEpi {
    const float *g_read;
    float c_t;
    const float *u, *s, *vprev;
    const unsigned char *m;
    float *lam_v, *dI, *g_theta, *g_alpha;
    const float *alpha, *theta;
    nbg_lif_grad_params p;
    int N, has_ext;
    struct Regs {
        float gr, u, s, vp, al, th, lv, gt, ga;
        unsigned char m;
    };
    __device__ void before(Regs &g, int r, int j) const { // what no step of the sweep writes
        const size_t idx = (size_t)r * N + j;
        g.gr = g_read[idx];
        g.u = u[idx];
        g.s = s[idx];
        g.vp = vprev[idx];
        g.m = m[idx];
        g.al = alpha[j];
        g.th = theta[j];
    }
    __device__ void after(Regs &g, int r, int j) const {
        const size_t idx = (size_t)r * N + j;
        g.lv = lam_v[idx];
        g.gt = g_theta[idx];
        g.ga = g_alpha[idx];
    }
    __device__ void apply(const Regs &g, float x, int r, int j) const {
        const size_t idx = (size_t)r * N + j;
        const float dsdu = p.smooth ? p.slope * g.s * (1.0f - g.s) : surrogate(g.u - g.th, p.slope);
        float gs = c_t * g.gr - g.lv * (g.u - p.v_reset);
        if (has_ext) gs = gs + x;
        const float gu = gs * dsdu + g.lv * (1.0f - g.s);
        const float gm = g.m ? gu : 0.0f;
        dI[idx] = gm;
        lam_v[idx] = gm * (1.0f - g.al);
        g_theta[idx] = g.gt - gs * dsdu;
        g_alpha[idx] = g.ga + gm * (p.v_rest - g.vp);
    }
};

int sm_count() {
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    return n > 0 ? n : 1;
}

// The K split of an M x N x K product: CTAs are added while tiles times ranks
// leave SMs without one and a rank keeps 32 k (four rounds of its eight
// warps' granules; fewer and the exchange costs more than it shortens).  Above
// K = 128 there are two at least: sixteen chains of K / 16 terms, as one CTA
// keeps, leave a larger error than the 32 lane sums of nbg_small_gemm, which
// these products replaced (1000 x 1024 outputs of K = 1,000: 1.53e-7 of the norm
// against 1.23e-7, in two ranks 1.19e-7).
NtShape nt_shape(const float *A, const float *W, int M, int N, int K) {
    NtShape sh{};
    sh.M = M;
    sh.N = N;
    sh.K = K;
    const long long tiles = (long long)((M + kTile - 1) / kTile) * ((N + kTile - 1) / kTile);
    const int sms = sm_count();
    sh.ranks = 1;
    while (sh.ranks < 8 && (tiles * sh.ranks < sms || (sh.ranks == 1 && K > 128)) && K >= 64 * sh.ranks) sh.ranks *= 2;
    sh.per = ((K + sh.ranks - 1) / sh.ranks + 7) & ~7;
    sh.kc = std::min(sh.per, kNtChunk);
    sh.stages = sh.per > sh.kc ? 2 : 1;
    sh.vec = K % 4 == 0 && (((uintptr_t)A | (uintptr_t)W) & 15u) == 0;
    return sh;
}

template <class Epi>
nbg_status launch_nt(const float *A, const float *W, NtShape sh, const Epi &epi, bool chained, cudaStream_t stream) {
    void (*const kernel)(const float *, const float *, NtShape, Epi) =
        sh.ranks >= 4 ? k_product_nt<Epi, 1> : sh.ranks == 2 ? k_product_nt<Epi, 2> : k_product_nt<Epi, 4>;
    const size_t smem = nt_smem_bytes(sh.stages, sh.kc);
    // the limit is the kernel's, for every thread: always what its largest shape needs, never lowered to this one's
    if (smem > 48 * 1024)
        NBG_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)nt_smem_bytes(2, kNtChunk)));
    const long long rows = ((long long)sh.M + kTile - 1) / kTile, y = std::min<long long>(rows, 65535);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)((sh.N + kTile - 1) / kTile * sh.ranks), (unsigned)y, (unsigned)((rows + y - 1) / y));
    cfg.blockDim = dim3(kNtThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (sh.ranks > 1) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = (unsigned)sh.ranks;
        attr[n].val.clusterDim.y = attr[n].val.clusterDim.z = 1;
        ++n;
    }
    if (chained) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n].val.programmaticStreamSerializationAllowed = 1;
        ++n;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    NBG_CUDA(cudaLaunchKernelEx(&cfg, kernel, A, W, sh, epi));
    NBG_CUDA(cudaGetLastError());
    return NBG_OK;
}

// out[c][r] = in[r][c]
__global__ void __launch_bounds__(256) k_transpose(const float *__restrict__ in, float *__restrict__ out, int R,
                                                   int C) {
    __shared__ float tile[32][33];
    const int c0 = blockIdx.x * 32, x = threadIdx.x & 31, y = threadIdx.x >> 5;
    for (long long r0 = (long long)blockIdx.y * 32; r0 < R; r0 += (long long)gridDim.y * 32) {
#pragma unroll
        for (int k = 0; k < 32; k += 8)
            if (r0 + y + k < R && c0 + x < C) tile[y + k][x] = in[(size_t)(r0 + y + k) * C + c0 + x];
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 32; k += 8)
            if (c0 + y + k < C && r0 + x < R) out[(size_t)(c0 + y + k) * R + r0 + x] = tile[x][y + k];
        __syncthreads();
    }
}

// -------------------------------------------------------------- A^T times B
//
// part[q][m][n] = sum over the k of split q of A[k][m] B[k][n], A: K x M,
// B: K x N, both row major: S^T dI and X^T dI with K = the (step, row) pairs.
// Compute-bound (2 M N K operations on (M + N) K values): 64 x 64 tiles, 128
// threads of 8 x 4 outputs, pairs of m packed, three cp.async stages of 32 k,
// split K to fill the SMs.  Sixteen terms are one chain, their sums another, the
// splits a third (nbg_adjoint_reduce_add).  In a split of at most 128 terms the
// sixteen are four chains of four, added in pairs: one chain leaves a larger error
// there than the lane sums of nbg_small_gemm, which this product replaced (512 x
// 512 outputs of K = 100: 8.7e-8 of the norm against 7.5e-8, in pairs 7.3e-8).  In a
// long split the chain of the sums decides (chains of eight, 512 x 512 x 8000:
// 2.2e-7 against 1.7e-7), and the additions would cost.
//
// Measured, 512 x 512 x 8000 in 8 splits: 13.5 ms -> 113 us (37 TFLOP/s);
// error against 64 bits 2.9e-7 -> 1.7e-7 of the norm.
constexpr int kTnTile = 64, kTnThreads = 128, kTnK = 32, kTnStages = 3;

template <int kBytes>
__device__ __forceinline__ void tn_load(float *dst, const float *src, int c0, int cols, int k0, int k_end) {
    constexpr int kF = kBytes / 4, kPieces = kTnTile / kF;
#pragma unroll 4
    for (int e = threadIdx.x; e < kTnK * kPieces; e += kTnThreads) {
        const int k = e / kPieces, c = (e % kPieces) * kF;
        const bool ok = k0 + k < k_end && c0 + c < cols;
        copy_async<kBytes>(dst + k * kTnTile + c, ok ? src + (size_t)(k0 + k) * cols + c0 + c : src, ok);
    }
}

// acc = the kN terms from k0 of a stage, in one chain
template <int kN>
__device__ __forceinline__ void tn_chain(unsigned long long (&acc)[4][4], const float *as, const float *bs, int k0) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
#pragma unroll
    for (int k = k0; k < k0 + kN; ++k) {
        const ulonglong2 a01 = *reinterpret_cast<const ulonglong2 *>(as + k * kTnTile);
        const ulonglong2 a23 = *reinterpret_cast<const ulonglong2 *>(as + k * kTnTile + 4);
        const float4 b = *reinterpret_cast<const float4 *>(bs + k * kTnTile);
        const unsigned long long bb[4] = {pack2(b.x, b.x), pack2(b.y, b.y), pack2(b.z, b.z), pack2(b.w, b.w)};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            fma2(acc[0][j], a01.x, bb[j]);
            fma2(acc[1][j], a01.y, bb[j]);
            fma2(acc[2][j], a23.x, bb[j]);
            fma2(acc[3][j], a23.y, bb[j]);
        }
    }
}
__device__ __forceinline__ void tn_add(unsigned long long (&d)[4][4], const unsigned long long (&a)[4][4]) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) add2(d[i][j], a[i][j]);
}

template <bool kPairs>
__global__ void __launch_bounds__(kTnThreads) k_product_tn(const float *__restrict__ A, const float *__restrict__ B,
                                                           float *__restrict__ part, int M, int N, int K, int per,
                                                           int vec_a, int vec_b) {
    __shared__ __align__(16) float st[kTnStages][2][kTnK * kTnTile];
    const unsigned n_tiles = (unsigned)((N + kTnTile - 1) / kTnTile); // tiles of n first, then of m
    const int n0 = (int)(blockIdx.x % n_tiles) * kTnTile, m0 = (int)(blockIdx.x / n_tiles) * kTnTile;
    const int k_beg = (int)min((long long)blockIdx.z * per, (long long)K), k_end = k_beg + min(per, K - k_beg);
    const int chunks = (k_end - k_beg + kTnK - 1) / kTnK;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int ml = (warp >> 1) * 32 + (lane >> 3) * 8, nl = (warp & 1) * 32 + (lane & 7) * 4;
    auto load = [&](int c) {
        float(*s)[kTnK * kTnTile] = st[c % kTnStages];
        const int k0 = k_beg + c * kTnK;
        if (vec_a) tn_load<16>(s[0], A, m0, M, k0, k_end);
        else tn_load<4>(s[0], A, m0, M, k0, k_end);
        if (vec_b) tn_load<16>(s[1], B, n0, N, k0, k_end);
        else tn_load<4>(s[1], B, n0, N, k0, k_end);
    };
    unsigned long long total[4][4]; // rows 2 i and 2 i + 1 of a column
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) total[i][j] = 0ull;
    for (int c = 0; c < kTnStages - 1; ++c) {
        if (c < chunks) load(c);
        copy_commit();
    }
    for (int c = 0; c < chunks; ++c) {
        copy_wait<kTnStages - 2>();
        __syncthreads(); // chunk c is here, and every warp has left chunk c - 1's stage
        if (c + kTnStages - 1 < chunks) load(c + kTnStages - 1);
        copy_commit();
        const float *const as = st[c % kTnStages][0] + ml, *const bs = st[c % kTnStages][1] + nl;
#pragma unroll 1
        for (int h = 0; h < kTnK; h += 16) {
            unsigned long long acc[4][4];
            if constexpr (kPairs) {
                unsigned long long x[4][4], y[4][4];
                tn_chain<4>(acc, as, bs, h);
                tn_chain<4>(x, as, bs, h + 4);
                tn_add(acc, x);
                tn_chain<4>(x, as, bs, h + 8);
                tn_chain<4>(y, as, bs, h + 12);
                tn_add(x, y);
                tn_add(acc, x);
            } else {
                tn_chain<16>(acc, as, bs, h);
            }
            tn_add(total, acc);
        }
    }
    float *const out = part + (size_t)blockIdx.z * M * N;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int m = m0 + ml + i;
        if (m >= M) break;
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (n0 + nl + j < N) {
                const float2 x = unpack2(total[i >> 1][j]);
                out[(size_t)m * N + n0 + nl + j] = i & 1 ? x.y : x.x;
            }
    }
}

} // namespace

extern "C" {

nbg_status nbg_transpose(const float *in, float *out, int rows, int cols, void *stream) {
    if (!in || !out || in == out || rows <= 0 || cols <= 0) return nbg_fail(NBG_ERR_INVALID, "nbg_transpose: bad arguments");
    const unsigned y = (unsigned)std::min(((long long)rows + 31) / 32, 65535LL);
    k_transpose<<<dim3((unsigned)(((long long)cols + 31) / 32), y), 256, 0, (cudaStream_t)stream>>>(in, out, rows, cols);
    NBG_CUDA(cudaGetLastError());
    return NBG_OK;
}

nbg_status nbg_product_nt(const float *A, const float *W, float *C, int M, int N, int K, void *stream) {
    if (!A || !W || !C || M <= 0 || N <= 0 || K <= 0) return nbg_fail(NBG_ERR_INVALID, "nbg_product_nt: bad arguments");
    return launch_nt(A, W, nt_shape(A, W, M, N, K), StoreEpi{C, N}, false, (cudaStream_t)stream);
}

nbg_status nbg_lif_forward_step_smooth(const float *s_prev, const float *w_rec_t, const float *xi, float *v,
                                       float *s_out, float *u_rec, uint8_t *m_rec, float *vprev_rec, float *z,
                                       float c_t, const float *alpha, const float *theta,
                                       const nbg_lif_grad_params *p, int chained, int B, int N, void *stream) {
    if (!s_prev || !w_rec_t || !xi || !v || !s_out || s_out == s_prev || !alpha || !theta || !p || B <= 0 || N <= 0)
        return nbg_fail(NBG_ERR_INVALID, "nbg_lif_forward_step_smooth: bad arguments");
    if (!p->smooth) return nbg_fail(NBG_ERR_UNSUPPORTED, "nbg_lif_forward_step_smooth runs the smoothed mode");
    const SmoothStepEpi epi{xi, v, s_out, u_rec, vprev_rec, z, m_rec, c_t, alpha, theta, *p, N};
    return launch_nt(s_prev, w_rec_t, nt_shape(s_prev, w_rec_t, B, N, N), epi, chained != 0, (cudaStream_t)stream);
}

nbg_status nbg_lif_adjoint_step_product(const float *dI_next, const float *w_rec, const float *g_read, float c_t,
                                        const float *u, const float *s, const uint8_t *m, const float *vprev,
                                        float *lam_v, float *dI, float *g_theta, float *g_alpha, const float *alpha,
                                        const float *theta, const nbg_lif_grad_params *p, int chained, int B, int N,
                                        void *stream) {
    if (!w_rec || !g_read || !u || !s || !m || !vprev || !lam_v || !dI || dI == dI_next || !g_theta || !g_alpha ||
        !alpha || !theta || !p || B <= 0 || N <= 0)
        return nbg_fail(NBG_ERR_INVALID, "nbg_lif_adjoint_step_product: bad arguments");
    const AdjointEpi epi{g_read, c_t, u, s, vprev, m, lam_v, dI, g_theta, g_alpha, alpha, theta, *p, N, dI_next != nullptr};
    return launch_nt(dI_next, w_rec, nt_shape(dI_next, w_rec, B, N, N), epi, chained != 0, (cudaStream_t)stream);
}

int nbg_product_tn_split(int M, int N, int K) {
    if (M <= 0 || N <= 0 || K <= 0) return 1;
    // four CTAs of 48 KiB fit an SM, three in flight keep its FMA pipes busy;
    // a split keeps at least 32 k, a stage (300 x 300 x 720 took 19 us in 2
    // splits of 360, its CTAs' serial stages, on 50 of 152 SMs)
    const long long tiles = (long long)((M + kTnTile - 1) / kTnTile) * ((N + kTnTile - 1) / kTnTile);
    const long long want = (3LL * sm_count() + tiles - 1) / tiles;
    return (int)std::max<long long>(1, std::min<long long>({want, (long long)K / 32, 64LL}));
}

nbg_status nbg_product_tn(const float *A, const float *B, float *part, int split, int M, int N, int K,
                          void *stream) {
    if (!A || !B || !part || split <= 0 || split > 65535 || M <= 0 || N <= 0 || K <= 0)
        return nbg_fail(NBG_ERR_INVALID, "nbg_product_tn: bad arguments");
    const long long tiles = (((long long)M + kTnTile - 1) / kTnTile) * (((long long)N + kTnTile - 1) / kTnTile);
    if (tiles > 0x7fffffff) return nbg_fail(NBG_ERR_UNSUPPORTED, "nbg_product_tn: %d x %d outputs", M, N);
    const int per = (int)std::min<long long>((((long long)K + split - 1) / split + kTnK - 1) / kTnK * kTnK, 0x7fffffe0);
    const dim3 grid((unsigned)tiles, 1, (unsigned)split);
    const int vec_a = M % 4 == 0 && ((uintptr_t)A & 15u) == 0, vec_b = N % 4 == 0 && ((uintptr_t)B & 15u) == 0;
    (per <= 128 ? k_product_tn<true> : k_product_tn<false>)<<<grid, kTnThreads, 0, (cudaStream_t)stream>>>(A, B, part, M, N, K,
                                                                                               per, vec_a, vec_b);
    NBG_CUDA(cudaGetLastError());
    return NBG_OK;
}

} // extern "C"
