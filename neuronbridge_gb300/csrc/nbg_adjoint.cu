// nbg_adjoint.cu -- forward and adjoint step kernels of the differentiable
// recurrent LIF (C ABI and equations in include/nbg_adjoint.h).  The dense
// products (x W_in, s W_rec, dI W_rec^T and the weight gradients) are plain
// library GEMMs issued by the caller; everything elementwise of a step --
// leak, jump, threshold, surrogate, reset, refractory, readout weighting and
// the parameter gradients -- is one fused kernel each way.

#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "nbg_adjoint.h"
#include "nbg_lif_grad.cuh"
#include "nbg_common.cuh"

namespace {


__global__ void __launch_bounds__(256) k_lif_fwd(const float *__restrict__ I, float *__restrict__ v,
                                                 int *__restrict__ ref, float *__restrict__ s_out,
                                                 float *__restrict__ u_rec, unsigned char *__restrict__ m_rec,
                                                 float *__restrict__ vprev_rec, float *__restrict__ z, float c_t,
                                                 const float *__restrict__ alpha, const float *__restrict__ theta,
                                                 nbg_lif_grad_params p, int N, int total) {
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= total) return;
    const int j = idx % N;
    const float vp = v[idx];
    const int rf = p.smooth ? 0 : ref[idx];
    const bool m = rf == 0;
    const float a = alpha[j], th = theta[j];
    const float u = m ? vp + a * (p.v_rest - vp) + I[idx] : p.v_reset;
    float s;
    if (p.smooth) s = 1.0f / (1.0f + expf(-p.slope * (u - th)));
    else s = u > th ? 1.0f : 0.0f;
    v[idx] = u - s * (u - p.v_reset);
    if (!p.smooth) ref[idx] = s > 0.0f ? p.t_ref : (rf > 0 ? rf - 1 : 0);
    s_out[idx] = s;
    if (u_rec) u_rec[idx] = u;
    if (m_rec) m_rec[idx] = m ? 1 : 0;
    if (vprev_rec) vprev_rec[idx] = vp;
    if (z) z[idx] = z[idx] + c_t * s;
}

__global__ void __launch_bounds__(256) k_lif_adj(const float *__restrict__ g_ext, const float *__restrict__ g_read,
                                                 float c_t, const float *__restrict__ u, const float *__restrict__ s,
                                                 const unsigned char *__restrict__ m, const float *__restrict__ vprev,
                                                 float *__restrict__ lam_v, float *__restrict__ dI,
                                                 float *__restrict__ g_theta, float *__restrict__ g_alpha,
                                                 const float *__restrict__ alpha, const float *__restrict__ theta,
                                                 nbg_lif_grad_params p, int N, int total) {
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= total) return;
    const int j = idx % N;
    const float uu = u[idx], ss = s[idx], lv = lam_v[idx];
    const float th = theta[j];
    const float dsdu = p.smooth ? p.slope * ss * (1.0f - ss) : surrogate(uu - th, p.slope);
    // dL/ds_t: recurrent path + readout + the reset's dependence on s
    float gs = c_t * g_read[idx] - lv * (uu - p.v_reset);
    if (g_ext) gs = gs + g_ext[idx];
    // dL/du_t through the spike and through v_t = u - s (u - V_reset)
    const float gu = gs * dsdu + lv * (1.0f - ss);
    const float gm = m[idx] ? gu : 0.0f;
    dI[idx] = gm;
    lam_v[idx] = gm * (1.0f - alpha[j]);
    g_theta[idx] = g_theta[idx] - gs * dsdu;
    g_alpha[idx] = g_alpha[idx] + gm * (p.v_rest - vprev[idx]);
}

// Spike-driven forward step (spiking mode, binary s): one CTA per instance
// row b.  I = xi + the sum of the W_rec rows of the previous step's spikes in
// ascending neuron order (the spike list of row b), then the same update as
// k_lif_fwd, then the row's new spike list in ascending order (block-wide
// ballot prefix).  Each thread owns columns j = threadIdx.x + q * blockDim.x.
constexpr int kSparseThreads = 256;
constexpr int kSparseCols = 8; // columns per thread: N <= 2048

__global__ void __launch_bounds__(kSparseThreads) k_lif_fwd_sparse(
    const float *__restrict__ xi, const float *__restrict__ w, const int *__restrict__ idx_in,
    const int *__restrict__ cnt_in, int *__restrict__ idx_out, int *__restrict__ cnt_out, float *__restrict__ v,
    int *__restrict__ ref, float *__restrict__ s_out, float *__restrict__ u_rec, unsigned char *__restrict__ m_rec,
    float *__restrict__ vprev_rec, float *__restrict__ z, float c_t, const float *__restrict__ alpha,
    const float *__restrict__ theta, nbg_lif_grad_params p, int N) {
    __shared__ int warp_base[kSparseThreads / 32 + 1];
    const int b = blockIdx.x, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const size_t row = (size_t)b * N;
    const int nq = (N + kSparseThreads - 1) / kSparseThreads;
    float acc[kSparseCols];
#pragma unroll
    for (int q = 0; q < kSparseCols; ++q) {
        const int j = tid + q * kSparseThreads;
        acc[q] = (q < nq && j < N) ? xi[row + j] : 0.0f;
    }
    const int cnt = cnt_in[b];
    const int *list = idx_in + row;
    for (int k = 0; k < cnt; ++k) {
        const float *wr = w + (size_t)__ldg(&list[k]) * N;
#pragma unroll
        for (int q = 0; q < kSparseCols; ++q) {
            const int j = tid + q * kSparseThreads;
            if (q < nq && j < N) acc[q] = acc[q] + __ldg(&wr[j]);
        }
    }
    int base = 0; // spikes of this row in earlier column chunks
    for (int q = 0; q < nq; ++q) {
        const int j = tid + q * kSparseThreads;
        bool spk = false;
        if (j < N) {
            const size_t i = row + j;
            const float vp = v[i];
            const int rf = ref[i];
            const bool m = rf == 0;
            float a_q = acc[0];
#pragma unroll
            for (int r = 1; r < kSparseCols; ++r)
                if (q == r) a_q = acc[r];
            const float u = m ? vp + alpha[j] * (p.v_rest - vp) + a_q : p.v_reset;
            const float sv = u > theta[j] ? 1.0f : 0.0f;
            v[i] = u - sv * (u - p.v_reset);
            ref[i] = sv > 0.0f ? p.t_ref : (rf > 0 ? rf - 1 : 0);
            s_out[i] = sv;
            if (u_rec) u_rec[i] = u;
            if (m_rec) m_rec[i] = m ? 1 : 0;
            if (vprev_rec) vprev_rec[i] = vp;
            if (z) z[i] = z[i] + c_t * sv;
            spk = sv > 0.0f;
        }
        // ordered compaction of this chunk's spikes
        const unsigned bal = __ballot_sync(0xffffffffu, spk);
        if (lane == 0) warp_base[wid] = __popc(bal);
        __syncthreads();
        if (tid == 0) {
            int sum = 0;
            for (int k = 0; k < kSparseThreads / 32; ++k) {
                const int c = warp_base[k];
                warp_base[k] = sum;
                sum += c;
            }
            warp_base[kSparseThreads / 32] = sum;
        }
        __syncthreads();
        if (spk) idx_out[row + base + warp_base[wid] + __popc(bal & ((1u << lane) - 1u))] = j;
        base += warp_base[kSparseThreads / 32];
        __syncthreads();
    }
    if (tid == 0) cnt_out[b] = base;
}

// A whole checkpoint segment of the spike-driven forward for more than
// kRowsMaxInputs input channels (k_lif_fwd_rows below takes the others, whose
// inputs fit its shared-memory ring): one CTA per row, the lists of a step's
// nonzero inputs and of the spikes in shared memory.
//
// acc[q] (column tid + q * kSparseThreads) += the rows idx[0..n) of w (N
// columns), in ascending k, each scaled by val[k] when kScaled.  The rows are
// fetched kRowBatch at a time before any is added, so a batch costs one L2
// round trip instead of one per row; the additions keep their order.
constexpr int kRowBatch = 4;
template <bool kScaled>
__device__ __forceinline__ void gather_rows(float (&acc)[kSparseCols], const float *__restrict__ w,
                                            const int *idx, const float *val, int n, int tid, int nq, int N) {
    for (int k0 = 0; k0 < n; k0 += kRowBatch) {
        float x[kRowBatch][kSparseCols];
#pragma unroll
        for (int r = 0; r < kRowBatch; ++r) {
            const float *wr = w + (size_t)(k0 + r < n ? idx[k0 + r] : 0) * N;
#pragma unroll
            for (int q = 0; q < kSparseCols; ++q) {
                const int j = tid + q * kSparseThreads;
                x[r][q] = (k0 + r < n && q < nq && j < N) ? __ldg(&wr[j]) : 0.0f;
            }
        }
#pragma unroll
        for (int r = 0; r < kRowBatch; ++r) {
            if (k0 + r >= n) break;
            const float v = kScaled ? val[k0 + r] : 1.0f;
#pragma unroll
            for (int q = 0; q < kSparseCols; ++q) {
                const int j = tid + q * kSparseThreads;
                if (q < nq && j < N) acc[q] = kScaled ? acc[q] + v * x[r][q] : acc[q] + x[r][q];
            }
        }
    }
}

// At every step the CTA lists row b's nonzero inputs x_t[b][c] (ascending c,
// with their values) and starts the sum from them: I_t = (sum over listed c
// of x_t[b][c] * W_in[c]) + (the W_rec rows of the previous step's spikes),
// each term added in ascending order.
__global__ void __launch_bounds__(kSparseThreads) k_lif_fwd_segment(
    const float *__restrict__ x, const float *__restrict__ w_in, int C,
    const float *__restrict__ w, int *__restrict__ spk, int *__restrict__ cnt,
    float *__restrict__ v, int *__restrict__ ref, float *__restrict__ s_out, float *__restrict__ s_last,
    float *__restrict__ u_rec, unsigned char *__restrict__ m_rec, float *__restrict__ vprev_rec,
    float *__restrict__ z, const float *__restrict__ c, const float *__restrict__ alpha,
    const float *__restrict__ theta, nbg_lif_grad_params p, int L, int B, int N) {
    extern __shared__ int seg_lists[]; // [2][N], then in_idx[C], in_val[C]
    __shared__ int warp_base[kSparseThreads / 32 + 1];
    __shared__ int list_cnt[2];
    int *in_idx = seg_lists + 2 * N;
    float *in_val = reinterpret_cast<float *>(in_idx + C);
    const int b = blockIdx.x, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const size_t row = (size_t)b * N, plane = (size_t)B * N;
    const int nq = (N + kSparseThreads - 1) / kSparseThreads;
    float vv[kSparseCols], zz[kSparseCols];
    int rr[kSparseCols];
#pragma unroll
    for (int q = 0; q < kSparseCols; ++q) {
        const int j = tid + q * kSparseThreads;
        vv[q] = zz[q] = 0.0f;
        rr[q] = 0;
        if (q < nq && j < N) {
            vv[q] = v[row + j];
            rr[q] = ref[row + j];
            if (z) zz[q] = z[row + j];
        }
    }
    if (tid == 0) list_cnt[0] = cnt[b];
    __syncthreads();
    for (int k = tid; k < list_cnt[0]; k += kSparseThreads) seg_lists[k] = spk[row + k];
    __syncthreads();
    int cur = 0;
    for (int step = 0; step < L; ++step) {
        float acc[kSparseCols];
        // row b's nonzero inputs of this step, ascending
        const float *xr = x + ((size_t)step * B + b) * C;
        int nin = 0;
        for (int c0 = 0; c0 < C; c0 += kSparseThreads) {
            const int ch = c0 + tid;
            const float xv = ch < C ? xr[ch] : 0.0f;
            const bool nz = xv != 0.0f;
            const unsigned bal = __ballot_sync(0xffffffffu, nz);
            if (lane == 0) warp_base[wid] = __popc(bal);
            __syncthreads();
            if (tid == 0) {
                int sum = 0;
                for (int k = 0; k < kSparseThreads / 32; ++k) {
                    const int cc = warp_base[k];
                    warp_base[k] = sum;
                    sum += cc;
                }
                warp_base[kSparseThreads / 32] = sum;
            }
            __syncthreads();
            if (nz) {
                const int at = nin + warp_base[wid] + __popc(bal & ((1u << lane) - 1u));
                in_idx[at] = ch;
                in_val[at] = xv;
            }
            nin += warp_base[kSparseThreads / 32];
            __syncthreads();
        }
#pragma unroll
        for (int q = 0; q < kSparseCols; ++q) acc[q] = 0.0f;
        gather_rows<true>(acc, w_in, in_idx, in_val, nin, tid, nq, N);
        const int *list = seg_lists + cur * N;
        gather_rows<false>(acc, w, list, nullptr, list_cnt[cur], tid, nq, N);
        int *out_list = seg_lists + (cur ^ 1) * N;
        int base = 0;
        const float ct = z ? c[step] : 0.0f;
#pragma unroll
        for (int q = 0; q < kSparseCols; ++q) {
            if (q >= nq) break;
            const int j = tid + q * kSparseThreads;
            bool sp = false;
            if (j < N) {
                const size_t i = row + j, o = (size_t)step * plane + i;
                const float vp = vv[q];
                const int rf = rr[q];
                const bool m = rf == 0;
                const float u = m ? vp + alpha[j] * (p.v_rest - vp) + acc[q] : p.v_reset;
                const float sv = u > theta[j] ? 1.0f : 0.0f;
                vv[q] = u - sv * (u - p.v_reset);
                rr[q] = sv > 0.0f ? p.t_ref : (rf > 0 ? rf - 1 : 0);
                if (s_out) s_out[o] = sv;
                if (s_last && step == L - 1) s_last[i] = sv;
                if (u_rec) u_rec[o] = u;
                if (m_rec) m_rec[o] = m ? 1 : 0;
                if (vprev_rec) vprev_rec[o] = vp;
                if (z) zz[q] = zz[q] + ct * sv;
                sp = sv > 0.0f;
            }
            // ordered compaction of this chunk's spikes into the next list
            const unsigned bal = __ballot_sync(0xffffffffu, sp);
            if (lane == 0) warp_base[wid] = __popc(bal);
            __syncthreads();
            if (tid == 0) {
                int sum = 0;
                for (int k = 0; k < kSparseThreads / 32; ++k) {
                    const int cc = warp_base[k];
                    warp_base[k] = sum;
                    sum += cc;
                }
                warp_base[kSparseThreads / 32] = sum;
            }
            __syncthreads();
            if (sp) out_list[base + warp_base[wid] + __popc(bal & ((1u << lane) - 1u))] = j;
            base += warp_base[kSparseThreads / 32];
            __syncthreads();
        }
        if (tid == 0) list_cnt[cur ^ 1] = base;
        __syncthreads();
        cur ^= 1;
    }
#pragma unroll
    for (int q = 0; q < kSparseCols; ++q) {
        const int j = tid + q * kSparseThreads;
        if (q < nq && j < N) {
            v[row + j] = vv[q];
            ref[row + j] = rr[q];
            if (z) z[row + j] = zz[q];
        }
    }
    const int nl = list_cnt[cur];
    for (int k = tid; k < nl; k += kSparseThreads) spk[row + k] = seg_lists[cur * N + k];
    if (tid == 0) cnt[b] = nl;
}

// ------------------------------------------------ rows through a segment
//
// The spike-driven forward of a checkpoint segment, one CTA per batch row
// (rows are independent), for up to kRowsMaxInputs input channels.  Per step:
//   I = (x_t[c] * W_in[c] over the nonzero inputs c) + (the W_rec rows of the
//       spikes of step t - 1), every term added in ascending order,
// then the update of k_lif_fwd_sparse in the same operations.
//
// What bounds it: the spikes of a step must be known before the next step's
// rows (about 28 of 4 KiB at 1,024 neurons firing 2 % of the steps, from L2)
// can be asked for, so a step is one chain -- spike list, row loads, sums,
// threshold, list -- and a warp's own instructions on it weigh as much as the
// loads' latency.  So:
//   * a thread owns four neighbouring columns (two, or single ones, where N or
//     a pointer is not aligned), adds them packed, and has up to 24 rows in
//     flight; the list holds byte offsets of rows, read four at a time, padded
//     to whole groups of four;
//   * the input rows of step t + 1 do not depend on the spikes of step t: they
//     are requested behind the recurrent rows of step t and summed into the
//     next step's start value;
//   * inputs come through a ring of kRing rows in shared memory, copied
//     asynchronously, and one warp (another each step) lists the nonzero
//     channels of step t + 2 from it while the rows are in flight;
//   * the new spikes are ranked by ballots and one exchange of the warps'
//     counts: two block barriers a step.
// The kernel before it listed, summed and ranked one after the other with
// about twenty barriers a step.  Measured, 500 steps of 64 rows, 1,000
// neurons, 200 inputs, 2.2 % firing: 6.2 -> 2.2 us a step, the call with its
// inputs and readout 3.14 -> 1.13 ms.  (With eight warps of four unpacked columns
// 4.9 us: 1,506 instructions a warp and step, few of them waiting for memory; with
// sixteen warps of two packed columns 2.5.)
constexpr int kRing = 8, kHalfRing = kRing / 2;
constexpr int kRowsMaxInputs = 4096;
constexpr int kRowsMaxNeurons = 2048;
// the lists of two steps' nonzero inputs and the ring of C channels
constexpr size_t rows_smem_bytes(int C) {
    return 2 * ((size_t)(C + 5) & ~(size_t)1) * sizeof(uint2) + (size_t)kRing * C * sizeof(float);
}

__device__ __forceinline__ void ring_copy(float *dst, const float *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}

// A thread's columns of a row, and sums of them: V neighbouring columns (2 or
// 4, as packed pairs) or NC single ones (V = 1).  Packed or not, every
// addition and product is rounded once.
template <int V, int NC> struct Cols {
    static constexpr int kN = V == 1 ? NC : V / 2;
    typename std::conditional<V == 1, float, unsigned long long>::type d[kN];
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int i = 0; i < kN; ++i) d[i] = 0;
    }
    // at: byte offsets of this thread's columns (one per column group)
    __device__ __forceinline__ void load(const float *base, unsigned row, const unsigned (&at)[V == 1 ? NC : 1]) {
        if constexpr (V == 1) {
#pragma unroll
            for (int i = 0; i < NC; ++i) d[i] = __ldg(reinterpret_cast<const float *>((const char *)base + (row + at[i])));
        } else if constexpr (V == 2) {
            d[0] = __ldg(reinterpret_cast<const unsigned long long *>((const char *)base + (row + at[0])));
        } else {
            const ulonglong2 q = __ldg(reinterpret_cast<const ulonglong2 *>((const char *)base + (row + at[0])));
            d[0] = q.x;
            d[1] = q.y;
        }
    }
    __device__ __forceinline__ void add(const Cols &o) {
#pragma unroll
        for (int i = 0; i < kN; ++i) {
            if constexpr (V == 1) d[i] = d[i] + o.d[i];
            else asm("add.rn.f32x2 %0, %0, %1;" : "+l"(d[i]) : "l"(o.d[i]));
        }
    }
    __device__ __forceinline__ void add_scaled(float x, const Cols &o) {
#pragma unroll
        for (int i = 0; i < kN; ++i) {
            if constexpr (V == 1) {
                d[i] = d[i] + x * o.d[i];
            } else {
                // single products: a packed product and sum would be fused into one rounding
                unsigned long long q;
                asm("mov.b64 %0, {%1, %2};" : "=l"(q) : "f"(__fmul_rn(x, o.get(2 * i))), "f"(__fmul_rn(x, o.get(2 * i + 1))));
                asm("add.rn.f32x2 %0, %0, %1;" : "+l"(d[i]) : "l"(q));
            }
        }
    }
    __device__ __forceinline__ float get(int i) const {
        if constexpr (V == 1) {
            return d[i];
        } else {
            float x, y;
            asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(d[i >> 1]));
            return i & 1 ? y : x;
        }
    }
};

template <bool kGather, int V, int NC, int kMaxThreads>
__global__ void __launch_bounds__(kMaxThreads) k_lif_fwd_rows(
    const float *__restrict__ xi, const float *__restrict__ x, const float *__restrict__ w_in, int C,
    const float *__restrict__ w, int *__restrict__ spk, int *__restrict__ cnt, float *__restrict__ v,
    int *__restrict__ ref, float *__restrict__ s_out, float *__restrict__ s_last, float *__restrict__ u_rec,
    unsigned char *__restrict__ m_rec, float *__restrict__ vprev_rec, float *__restrict__ z,
    const float *__restrict__ c, const float *__restrict__ alpha, const float *__restrict__ theta,
    nbg_lif_grad_params p, int L, int B, int N) {
    static_assert(V == 1 || NC == V, "a group is the thread's neighbouring columns");
    // groups of four rows in flight: 96 registers at most, 48 where 512 threads share them
    constexpr int kGroups = kMaxThreads <= 256 ? 24 / NC : NC == 4 ? 3 : NC == 2 ? 6 : 8;
    constexpr int kSegs = V == 1 ? NC : 1;                 // segments of the ascending order: (column group, warp)
    __shared__ __align__(16) unsigned list[kRowsMaxNeurons + 4]; // ascending spikes of the step before: row offsets
    __shared__ int seg_cnt[64];                                  // spikes per (column group, warp)
    __shared__ int in_cnt[2];
    extern __shared__ __align__(16) uint2 rows_smem[]; // kGather: lists [2][C + 4 rounded to even] (row offset, value), ring [kRing][C]
    const int Cl = (C + 5) & ~1;
    uint2 *const in_list = rows_smem;
    float *const ring = reinterpret_cast<float *>(rows_smem + 2 * Cl);
    const int b = blockIdx.x, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int T = blockDim.x, nw = T >> 5;
    const unsigned row_bytes = (unsigned)N * 4u;
    const size_t row = (size_t)b * N, plane = (size_t)B * N;
    int col[NC];
    bool has[NC]; // V > 1: N is a multiple of V, so all or none
    unsigned at[kSegs]; // a thread without columns reads the row's first ones and drops them
#pragma unroll
    for (int i = 0; i < NC; ++i) {
        col[i] = V == 1 ? i * T + tid : tid * V + i;
        has[i] = col[i] < N;
    }
#pragma unroll
    for (int i = 0; i < kSegs; ++i) at[i] = has[i] ? (unsigned)col[i] * 4u : 0u;
    float vv[NC], zz[NC], al[NC], th[NC];
    int rr[NC];
#pragma unroll
    for (int i = 0; i < NC; ++i) {
        vv[i] = zz[i] = al[i] = th[i] = 0.0f;
        rr[i] = 0;
        if (has[i]) {
            vv[i] = v[row + col[i]];
            rr[i] = ref[row + col[i]];
            if (z) zz[i] = z[row + col[i]];
            al[i] = alpha[col[i]];
            th[i] = theta[col[i]];
        }
    }
    using Row = Cols<V, NC>;
    // four rows of the spike list from k on, and their sum in order
    auto request = [&](Row (&d)[4], int k) {
        const uint4 o = *reinterpret_cast<const uint4 *>(list + k);
        d[0].load(w, o.x, at);
        d[1].load(w, o.y, at);
        d[2].load(w, o.z, at);
        d[3].load(w, o.w, at);
    };
    auto add = [&](Row &acc, const Row (&d)[4], int left) {
        acc.add(d[0]);
        if (left >= 4) {
            acc.add(d[1]);
            acc.add(d[2]);
            acc.add(d[3]);
        } else {
            if (left > 1) acc.add(d[1]);
            if (left > 2) acc.add(d[2]);
        }
    };
    auto request_in = [&](Row (&d)[4], float (&xv)[4], int at_list) {
        const uint4 p0 = *reinterpret_cast<const uint4 *>(in_list + at_list);
        const uint4 p1 = *reinterpret_cast<const uint4 *>(in_list + at_list + 2);
        d[0].load(w_in, p0.x, at);
        d[1].load(w_in, p0.z, at);
        d[2].load(w_in, p1.x, at);
        d[3].load(w_in, p1.z, at);
        xv[0] = __uint_as_float(p0.y);
        xv[1] = __uint_as_float(p0.w);
        xv[2] = __uint_as_float(p1.y);
        xv[3] = __uint_as_float(p1.w);
    };
    auto add_in = [&](Row &acc, const Row (&d)[4], const float (&xv)[4], int left) {
#pragma unroll
        for (int r = 0; r < 4; ++r)
            if (left > r) acc.add_scaled(xv[r], d[r]);
    };
    auto ring_load = [&](int step, int rows) { // rows step .. step + rows - 1 of the inputs
        for (int ch = tid; ch < C; ch += T) {
            const float *xr = x + ((size_t)step * B + b) * C + ch;
            float *d = ring + (step % kRing) * C + ch;
            for (int k = 0; k < rows && step + k < L; ++k) ring_copy(d + k * C, xr + (size_t)k * B * C);
        }
    };
    auto list_inputs = [&](int step) { // one warp: the nonzero channels of `step`, ascending
        const float *xr = ring + (step % kRing) * C;
        uint2 *const out = in_list + (step & 1) * Cl;
        int n = 0;
#pragma unroll 4
        for (int c0 = 0; c0 < C; c0 += 32) {
            const float xv = c0 + lane < C ? xr[c0 + lane] : 0.0f;
            const bool nz = xv != 0.0f;
            const unsigned bal = __ballot_sync(0xffffffffu, nz);
            if (nz) out[n + __popc(bal & ((1u << lane) - 1u))] = make_uint2((unsigned)(c0 + lane) * row_bytes, __float_as_uint(xv));
            n += __popc(bal);
        }
        if (lane < 4) out[n + lane] = make_uint2(0u, 0u); // the last group's padding: row 0, not added
        if (lane == 0) in_cnt[step & 1] = n;
    };
    int n_spk = cnt[b];
    for (int k = tid; k < n_spk + 4; k += T) list[k] = k < n_spk ? (unsigned)spk[row + k] * row_bytes : 0u;
    if constexpr (kGather) {
        ring_load(0, kRing);
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        if (wid == 0) {
            list_inputs(0);
            if (L > 1) list_inputs(1);
        }
    }
    __syncthreads();
    Row start; // the sum the next step starts from: its input term
    start.zero();
    if constexpr (kGather) {
        for (int k = 0; k < in_cnt[0]; k += 4) {
            Row d[4];
            float xv[4];
            request_in(d, xv, k);
            add_in(start, d, xv, in_cnt[0] - k);
        }
        __syncthreads(); // step 0 lists the inputs of step 2 over those of step 0
    } else {
        start.load(xi + row, 0u, at);
    }
    int lister = 0; // the warp that lists next
    size_t o = row; // this step's row of the record
    for (int step = 0; step < L; ++step) {
        Row acc = start;
        const float ct = z ? c[step] : 0.0f;
        const bool more = step + 1 < L;
        const int slot = (step + 1) & 1;
        Row d[kGroups][4];
#pragma unroll
        for (int g = 0; g < kGroups; ++g)
            if (4 * g < n_spk) request(d[g], 4 * g);
        int n_in = 0;
        Row di[2][4];
        float xv[2][4];
        if constexpr (kGather) {
            if (more) {
                n_in = in_cnt[slot];
#pragma unroll
                for (int g = 0; g < 2; ++g)
                    if (4 * g < n_in) request_in(di[g], xv[g], slot * Cl + 4 * g);
            }
            if (wid == lister && step + 2 < L) list_inputs(step + 2);
            lister = lister + 1 == nw ? 0 : lister + 1;
            // half the ring at a time, over rows listed two steps ago and before
            if (step > 0 && step % kHalfRing == 0) ring_load(step + kHalfRing, kHalfRing);
        } else {
            if (more) start.load(xi + o + plane, 0u, at);
        }
        for (int k = 0;;) {
#pragma unroll
            for (int g = 0; g < kGroups; ++g)
                if (k + 4 * g < n_spk) add(acc, d[g], n_spk - k - 4 * g);
            k += 4 * kGroups;
            if (k >= n_spk) break;
#pragma unroll
            for (int g = 0; g < kGroups; ++g)
                if (k + 4 * g < n_spk) request(d[g], k + 4 * g);
        }
        float uu[NC], vp[NC];
        unsigned bal[NC];
        bool integ[NC], sp[NC];
#pragma unroll
        for (int i = 0; i < NC; ++i) {
            vp[i] = vv[i];
            const int rf = rr[i];
            integ[i] = rf == 0;
            uu[i] = integ[i] ? vp[i] + al[i] * (p.v_rest - vp[i]) + acc.get(i) : p.v_reset;
            sp[i] = has[i] && uu[i] > th[i];
            const float sv = sp[i] ? 1.0f : 0.0f;
            vv[i] = uu[i] - sv * (uu[i] - p.v_reset);
            rr[i] = sp[i] ? p.t_ref : (rf > 0 ? rf - 1 : 0);
            if (z) zz[i] = zz[i] + ct * sv;
            bal[i] = __ballot_sync(0xffffffffu, sp[i]);
        }
        // ranks: within the warp by ballots, across warps by their counts
        if (lane == 0) {
            if constexpr (V == 1) {
#pragma unroll
                for (int i = 0; i < NC; ++i) seg_cnt[i * nw + wid] = __popc(bal[i]);
            } else {
                int k = 0;
#pragma unroll
                for (int i = 0; i < NC; ++i) k += __popc(bal[i]);
                seg_cnt[wid] = k;
            }
        }
        if constexpr (kGather) // rows asked for a step ago, the first of them listed next step
            if (step % kHalfRing == 1) asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads(); // counts; everyone has read the list
        const unsigned lt = (1u << lane) - 1u;
        int total = 0;
#pragma unroll
        for (int s = 0; s < kSegs; ++s) {
            // spikes before segment s * nw + wid (low half) and in all (high half): both at most 2,048
            unsigned both = 0u;
#pragma unroll
            for (int h = 0; h < (kSegs > 1 ? 2 : 1); ++h) {
                const int k = lane + 32 * h;
                const unsigned q = k < kSegs * nw ? (unsigned)seg_cnt[k] : 0u;
                both += q << 16 | (k < s * nw + wid ? q : 0u);
            }
            both = __reduce_add_sync(0xffffffffu, both);
            int pos = (int)(both & 0xffffu);
            total = (int)(both >> 16);
            if constexpr (V == 1) {
                if (sp[s]) list[pos + __popc(bal[s] & lt)] = (unsigned)col[s] * row_bytes;
            } else {
#pragma unroll
                for (int i = 0; i < NC; ++i) pos += __popc(bal[i] & lt);
#pragma unroll
                for (int i = 0; i < NC; ++i)
                    if (sp[i]) list[pos++] = (unsigned)col[i] * row_bytes;
            }
        }
        n_spk = total;
        if (tid < 4) list[total + tid] = 0u; // the last group's padding: row 0, not added
        // the record, and the next step's input term, off the spikes' chain
        {
            float sv[NC];
#pragma unroll
            for (int i = 0; i < NC; ++i) sv[i] = sp[i] ? 1.0f : 0.0f;
            if constexpr (V == 4) {
                if (has[0]) {
                    const size_t q = (o >> 2) + tid; // rows are multiples of four
                    if (s_out) reinterpret_cast<float4 *>(s_out)[q] = make_float4(sv[0], sv[1], sv[2], sv[3]);
                    if (s_last && !more)
                        reinterpret_cast<float4 *>(s_last)[(row >> 2) + tid] = make_float4(sv[0], sv[1], sv[2], sv[3]);
                    if (u_rec) reinterpret_cast<float4 *>(u_rec)[q] = make_float4(uu[0], uu[1], uu[2], uu[3]);
                    if (m_rec)
                        reinterpret_cast<uchar4 *>(m_rec)[q] = make_uchar4(integ[0], integ[1], integ[2], integ[3]);
                    if (vprev_rec) reinterpret_cast<float4 *>(vprev_rec)[q] = make_float4(vp[0], vp[1], vp[2], vp[3]);
                }
            } else if constexpr (V == 2) {
                if (has[0]) {
                    const size_t q = (o >> 1) + tid;
                    if (s_out) reinterpret_cast<float2 *>(s_out)[q] = make_float2(sv[0], sv[1]);
                    if (s_last && !more) reinterpret_cast<float2 *>(s_last)[(row >> 1) + tid] = make_float2(sv[0], sv[1]);
                    if (u_rec) reinterpret_cast<float2 *>(u_rec)[q] = make_float2(uu[0], uu[1]);
                    if (m_rec) reinterpret_cast<uchar2 *>(m_rec)[q] = make_uchar2(integ[0], integ[1]);
                    if (vprev_rec) reinterpret_cast<float2 *>(vprev_rec)[q] = make_float2(vp[0], vp[1]);
                }
            } else {
#pragma unroll
                for (int i = 0; i < NC; ++i)
                    if (has[i]) {
                        const size_t q = o + col[i];
                        if (s_out) s_out[q] = sv[i];
                        if (s_last && !more) s_last[row + col[i]] = sv[i];
                        if (u_rec) u_rec[q] = uu[i];
                        if (m_rec) m_rec[q] = integ[i] ? 1 : 0;
                        if (vprev_rec) vprev_rec[q] = vp[i];
                    }
            }
        }
        if constexpr (kGather) {
            start.zero();
#pragma unroll
            for (int g = 0; g < 2; ++g)
                if (4 * g < n_in) add_in(start, di[g], xv[g], n_in - 4 * g);
            for (int k = 8; k < n_in; k += 4) {
                request_in(di[0], xv[0], slot * Cl + k);
                add_in(start, di[0], xv[0], n_in - k);
            }
        }
        o += plane;
        __syncthreads(); // the list; the input list of step + 2
    }
#pragma unroll
    for (int i = 0; i < NC; ++i) {
        if (!has[i]) continue;
        v[row + col[i]] = vv[i];
        ref[row + col[i]] = rr[i];
        if (z) z[row + col[i]] = zz[i];
    }
    for (int k = tid; k < n_spk; k += T) spk[row + k] = (int)(list[k] / row_bytes);
    if (tid == 0) cnt[b] = n_spk;
}

// Launch k_lif_fwd_rows: four (two) neighbouring columns a thread where N is a
// multiple of them and every matrix aligned, else single columns.  Eight warps
// of four columns, 24 rows in flight, were faster than sixteen of two (1,000
// neurons: 2.3 against 2.5 us a step): few more instructions a warp, half the
// warps in each other's way.
template <bool kGather>
nbg_status launch_rows(const float *xi, const float *x, const float *w_in, int C, const float *w, int *spk, int *cnt,
                       float *v, int *ref, float *s_out, float *s_last, float *u_rec, unsigned char *m_rec,
                       float *vprev_rec, float *z, const float *c, const float *alpha, const float *theta,
                       const nbg_lif_grad_params &p, int L, int B, int N, cudaStream_t stream) {
    using Kernel = void (*)(const float *, const float *, const float *, int, const float *, int *, int *, float *,
                            int *, float *, float *, float *, unsigned char *, float *, float *, const float *,
                            const float *, const float *, nbg_lif_grad_params, int, int, int);
    const uintptr_t bits = (uintptr_t)xi | (uintptr_t)w_in | (uintptr_t)w | (uintptr_t)s_out | (uintptr_t)s_last |
                           (uintptr_t)u_rec | (uintptr_t)vprev_rec | (uintptr_t)m_rec * 4u;
    Kernel k;
    int threads;
    if (N % 4 == 0 && (bits & 15u) == 0) {
        threads = (N / 4 + 31) & ~31;
        k = threads <= 256 ? k_lif_fwd_rows<kGather, 4, 4, 256> : k_lif_fwd_rows<kGather, 4, 4, 512>;
    } else if (N % 2 == 0 && N <= 1024 && (bits & 7u) == 0) {
        threads = (N / 2 + 31) & ~31;
        k = k_lif_fwd_rows<kGather, 2, 2, 512>;
    } else {
        threads = std::min(512, (N + 31) & ~31);
        const int nc = (N + threads - 1) / threads;
        k = nc == 1   ? k_lif_fwd_rows<kGather, 1, 1, 512>
            : nc == 2 ? k_lif_fwd_rows<kGather, 1, 2, 512>
                      : k_lif_fwd_rows<kGather, 1, 4, 512>;
    }
    const size_t smem = kGather ? rows_smem_bytes(C) : 0;
    // the limit is the kernel's, for every thread: always what its largest shape needs, never lowered to this one's
    if (smem > 32 * 1024)
        NBG_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)rows_smem_bytes(kRowsMaxInputs)));
    k<<<B, threads, smem, stream>>>(xi, x, w_in, C, w, spk, cnt, v, ref, s_out, s_last, u_rec, m_rec, vprev_rec, z, c,
                                    alpha, theta, p, L, B, N);
    NBG_CUDA(cudaGetLastError());
    return NBG_OK;
}

// Ascending spike list of each row of a 0/1 matrix (segment restarts).
__global__ void __launch_bounds__(kSparseThreads) k_spike_list(const float *__restrict__ s, int *__restrict__ idx,
                                                               int *__restrict__ cnt, int N) {
    __shared__ int warp_base[kSparseThreads / 32 + 1];
    const int b = blockIdx.x, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const size_t row = (size_t)b * N;
    int base = 0;
    for (int c0 = 0; c0 < N; c0 += kSparseThreads) {
        const int j = c0 + tid;
        const bool spk = j < N && s[row + j] > 0.0f;
        const unsigned bal = __ballot_sync(0xffffffffu, spk);
        if (lane == 0) warp_base[wid] = __popc(bal);
        __syncthreads();
        if (tid == 0) {
            int sum = 0;
            for (int k = 0; k < kSparseThreads / 32; ++k) {
                const int c = warp_base[k];
                warp_base[k] = sum;
                sum += c;
            }
            warp_base[kSparseThreads / 32] = sum;
        }
        __syncthreads();
        if (spk) idx[row + base + warp_base[wid] + __popc(bal & ((1u << lane) - 1u))] = j;
        base += warp_base[kSparseThreads / 32];
        __syncthreads();
    }
    if (tid == 0) cnt[b] = base;
}

// x[t][b][c]: a spike where the PoissonRate hash of (b C + c + seed, t) is below
// the channel's probability.  Bound by the stores; V (4 or 1) neighbouring
// channels a thread and one 16-byte store where C is a multiple of four and x
// aligned, time steps along y, so that no element needs a 64-bit division (which
// took four times the stores' time: 25.6 MB in 22 us, now 5.9).
template <int V>
__global__ void __launch_bounds__(256) k_poisson(float *__restrict__ x, const float *__restrict__ rates, int T,
                                                 long long BC, int C, float dt, int seed) {
    const long long bc = ((long long)blockIdx.x * 256 + threadIdx.x) * V;
    if (bc >= BC) return;
    const int c = (int)(bc % C);
    float prob[V];
#pragma unroll
    for (int k = 0; k < V; ++k) {
        float r = rates[c + k];
        r = r > 0.0f ? r : 0.0f;
        prob[k] = r * dt * 0.001f;
        prob[k] = prob[k] < 1.0f ? prob[k] : 1.0f;
    }
    for (int t = blockIdx.y; t < T; t += gridDim.y) {
        float *const o = x + (size_t)t * BC + bc;
        float s[V];
#pragma unroll
        for (int k = 0; k < V; ++k) s[k] = nbg_hash_uniform01((int)bc + k + seed, t) < prob[k] ? 1.0f : 0.0f;
        if constexpr (V == 4) *reinterpret_cast<float4 *>(o) = make_float4(s[0], s[1], s[2], s[3]);
        else o[0] = s[0];
    }
}

} // namespace

// C[i][j] = sum over k of A[i][k] B[k][j] (element (r, c) of A at
// A[r * a_rs + c * a_cs], likewise B), for the readout's small products
// (B x N by N x O and the like).  Short sums (K < kSmallGemmWarpK): one
// thread per output, k ascending.  Long ones: one warp per output, lane l
// adding k = l, l + 32, ... in order, then the 32 lane sums in a fixed tree.
// Either way the order depends only on K, so the result does not depend on
// the launch.
constexpr int kSmallGemmWarpK = 64;

__global__ void k_small_gemm(const float *__restrict__ A, int a_rs, int a_cs, const float *__restrict__ Bm, int b_rs,
                             int b_cs, float *__restrict__ Cm, int M, int N, int K) {
    const long long o = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (o >= (long long)M * N) return;
    const int i = (int)(o / N), j = (int)(o % N);
    float acc = 0.0f;
    for (int k = 0; k < K; ++k) acc = acc + A[(size_t)i * a_rs + (size_t)k * a_cs] * Bm[(size_t)k * b_rs + (size_t)j * b_cs];
    Cm[o] = acc;
}

// kAhead: the loop unrolled eight times, for the loads of eight terms in flight.
// Where few warps run (the readout z W_out) they wait for each other's latency:
// 64 x 10 outputs of K = 1,000 8.2 -> 6.0 us.  From about 4,096 outputs on the
// SMs have warps enough, and the longer loop only costs (40 x 2,500 of 1,000: 158
// us, unrolled 172), as its remainder does below K = 256 (64 x 10 of 128: 2.3,
// unrolled 2.4).
template <bool kAhead>
__global__ void k_small_gemm_warp(const float *__restrict__ A, int a_rs, int a_cs, const float *__restrict__ Bm,
                                  int b_rs, int b_cs, float *__restrict__ Cm, int M, int N, int K) {
    const long long o = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (o >= (long long)M * N) return; // whole warps: o is the same for all 32 lanes
    const int i = (int)(o / N), j = (int)(o % N);
    float acc = 0.0f;
    auto term = [&](int k) { acc = acc + A[(size_t)i * a_rs + (size_t)k * a_cs] * Bm[(size_t)k * b_rs + (size_t)j * b_cs]; };
    if constexpr (kAhead) {
#pragma unroll 8
        for (int k = lane; k < K; k += 32) term(k);
    } else {
        for (int k = lane; k < K; k += 32) term(k);
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) acc = acc + __shfl_down_sync(0xffffffffu, acc, d);
    if (lane == 0) Cm[o] = acc;
}

extern "C" {

nbg_status nbg_small_gemm(const float *A, int a_rs, int a_cs, const float *B, int b_rs, int b_cs, float *C, int M,
                          int N, int K, void *stream) {
    if (!A || !B || !C || M <= 0 || N <= 0 || K <= 0) return nbg_fail(NBG_ERR_INVALID, "nbg_small_gemm: bad arguments");
    const long long total = (long long)M * N;
    if (K >= kSmallGemmWarpK)
        (K >= 256 && total < 4096 ? k_small_gemm_warp<true> : k_small_gemm_warp<false>)<<<(unsigned)((total + 3) / 4), 128, 0,
                                                                                       (cudaStream_t)stream>>>(
            A, a_rs, a_cs, B, b_rs, b_cs, C, M, N, K);
    else
        k_small_gemm<<<(unsigned)((total + 127) / 128), 128, 0, (cudaStream_t)stream>>>(A, a_rs, a_cs, B, b_rs, b_cs,
                                                                                       C, M, N, K);
    NBG_CUDA(cudaGetLastError());
    return NBG_OK;
}

nbg_status nbg_lif_forward_step(const float *I, float *v, int32_t *ref, float *s_out, float *u_rec, uint8_t *m_rec,
                                float *vprev_rec, float *z, float c_t, const float *alpha, const float *theta,
                                const nbg_lif_grad_params *p, int B, int N, void *stream) {
    if (!I || !v || !ref || !s_out || !alpha || !theta || !p || B <= 0 || N <= 0)
        return nbg_fail(NBG_ERR_INVALID, "nbg_lif_forward_step: bad arguments");
    const int total = B * N;
    k_lif_fwd<<<(total + 255) / 256, 256, 0, (cudaStream_t)stream>>>(I, v, ref, s_out, u_rec, m_rec, vprev_rec, z,
                                                                      c_t, alpha, theta, *p, N, total);
    NBG_CUDA(cudaGetLastError());
    return NBG_OK;
}

nbg_status nbg_lif_adjoint_step(const float *g_ext, const float *g_read, float c_t, const float *u, const float *s,
                                const uint8_t *m, const float *vprev, float *lam_v, float *dI, float *g_theta,
                                float *g_alpha, const float *alpha, const float *theta, const nbg_lif_grad_params *p,
                                int B, int N, void *stream) {
    if (!g_read || !u || !s || !m || !vprev || !lam_v || !dI || !g_theta || !g_alpha || !alpha || !theta || !p ||
        B <= 0 || N <= 0)
        return nbg_fail(NBG_ERR_INVALID, "nbg_lif_adjoint_step: bad arguments");
    const int total = B * N;
    k_lif_adj<<<(total + 255) / 256, 256, 0, (cudaStream_t)stream>>>(g_ext, g_read, c_t, u, s, m, vprev, lam_v, dI,
                                                                      g_theta, g_alpha, alpha, theta, *p, N, total);
    NBG_CUDA(cudaGetLastError());
    return NBG_OK;
}

nbg_status nbg_lif_forward_step_sparse(const float *xi, const float *w_rec, const int32_t *spk_in,
                                       const int32_t *cnt_in, int32_t *spk_out, int32_t *cnt_out, float *v,
                                       int32_t *ref, float *s_out, float *u_rec, uint8_t *m_rec, float *vprev_rec,
                                       float *z, float c_t, const float *alpha, const float *theta,
                                       const nbg_lif_grad_params *p, int B, int N, void *stream) {
    if (!xi || !w_rec || !spk_in || !cnt_in || !spk_out || !cnt_out || !v || !ref || !s_out || !alpha || !theta ||
        !p || B <= 0 || N <= 0)
        return nbg_fail(NBG_ERR_INVALID, "nbg_lif_forward_step_sparse: bad arguments");
    if (p->smooth) return nbg_fail(NBG_ERR_UNSUPPORTED, "the spike-driven step needs binary spikes (smooth = 0)");
    if (N > kSparseThreads * kSparseCols)
        return nbg_fail(NBG_ERR_UNSUPPORTED, "the spike-driven step supports up to %d neurons",
                        kSparseThreads * kSparseCols);
    k_lif_fwd_sparse<<<B, kSparseThreads, 0, (cudaStream_t)stream>>>(xi, w_rec, spk_in, cnt_in, spk_out, cnt_out, v,
                                                                      ref, s_out, u_rec, m_rec, vprev_rec, z, c_t,
                                                                      alpha, theta, *p, N);
    NBG_CUDA(cudaGetLastError());
    return NBG_OK;
}

nbg_status nbg_lif_forward_segment_sparse(const float *xi, const float *w_rec, int32_t *spk, int32_t *cnt, float *v,
                                          int32_t *ref, float *s_out, float *s_last, float *u_rec, uint8_t *m_rec,
                                          float *vprev_rec, float *z, const float *c, const float *alpha,
                                          const float *theta, const nbg_lif_grad_params *p, int L, int B, int N,
                                          void *stream) {
    if (!xi || !w_rec || !spk || !cnt || !v || !ref || !alpha || !theta || !p || (z && !c) || L <= 0 || B <= 0 ||
        N <= 0)
        return nbg_fail(NBG_ERR_INVALID, "nbg_lif_forward_segment_sparse: bad arguments");
    if (p->smooth) return nbg_fail(NBG_ERR_UNSUPPORTED, "the spike-driven step needs binary spikes (smooth = 0)");
    if (N > kSparseThreads * kSparseCols)
        return nbg_fail(NBG_ERR_UNSUPPORTED, "the spike-driven step supports up to %d neurons",
                        kSparseThreads * kSparseCols);
    return launch_rows<false>(xi, nullptr, nullptr, 0, w_rec, spk, cnt, v, ref, s_out, s_last, u_rec, m_rec, vprev_rec,
                              z, c, alpha, theta, *p, L, B, N, (cudaStream_t)stream);
}

nbg_status nbg_lif_forward_segment_gather(const float *x, const float *w_in, int C, const float *w_rec, int32_t *spk,
                                          int32_t *cnt, float *v, int32_t *ref, float *s_out, float *s_last,
                                          float *u_rec, uint8_t *m_rec, float *vprev_rec, float *z, const float *c,
                                          const float *alpha, const float *theta, const nbg_lif_grad_params *p,
                                          int L, int B, int N, void *stream) {
    if (!x || !w_in || C <= 0 || !w_rec || !spk || !cnt || !v || !ref || !alpha || !theta || !p || (z && !c) ||
        L <= 0 || B <= 0 || N <= 0)
        return nbg_fail(NBG_ERR_INVALID, "nbg_lif_forward_segment_gather: bad arguments");
    if (p->smooth) return nbg_fail(NBG_ERR_UNSUPPORTED, "the spike-driven step needs binary spikes (smooth = 0)");
    if (N > kSparseThreads * kSparseCols)
        return nbg_fail(NBG_ERR_UNSUPPORTED, "the spike-driven step supports up to %d neurons",
                        kSparseThreads * kSparseCols);
    if (C <= kRowsMaxInputs)
        return launch_rows<true>(nullptr, x, w_in, C, w_rec, spk, cnt, v, ref, s_out, s_last, u_rec, m_rec, vprev_rec,
                                 z, c, alpha, theta, *p, L, B, N, (cudaStream_t)stream);
    const size_t smem = (2 * (size_t)N + 2 * (size_t)C) * sizeof(int);
    constexpr size_t most = 200 * 1024;
    if (smem > most) return nbg_fail(NBG_ERR_UNSUPPORTED, "too many inputs for the gather form (C = %d)", C);
    if (smem > 32 * 1024) // as in launch_rows
        NBG_CUDA(cudaFuncSetAttribute(k_lif_fwd_segment, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most));
    k_lif_fwd_segment<<<B, kSparseThreads, smem, (cudaStream_t)stream>>>(
        x, w_in, C, w_rec, spk, cnt, v, ref, s_out, s_last, u_rec, m_rec, vprev_rec, z, c, alpha, theta,
        *p, L, B, N);
    NBG_CUDA(cudaGetLastError());
    return NBG_OK;
}

nbg_status nbg_spike_lists(const float *s, int32_t *spk, int32_t *cnt, int B, int N, void *stream) {
    if (!s || !spk || !cnt || B <= 0 || N <= 0) return nbg_fail(NBG_ERR_INVALID, "nbg_spike_lists: bad arguments");
    k_spike_list<<<B, kSparseThreads, 0, (cudaStream_t)stream>>>(s, spk, cnt, N);
    NBG_CUDA(cudaGetLastError());
    return NBG_OK;
}

nbg_status nbg_poisson_inputs(float *x, const float *rates_hz, int T, int B, int C, float dt_ms, int seed,
                              void *stream) {
    if (!x || !rates_hz || T <= 0 || B <= 0 || C <= 0) return nbg_fail(NBG_ERR_INVALID, "nbg_poisson_inputs: bad arguments");
    const long long BC = (long long)B * C;
    const int V = C % 4 == 0 && ((uintptr_t)x & 15u) == 0 ? 4 : 1;
    const unsigned gx = (unsigned)((BC + 256 * V - 1) / (256 * V));
    // enough CTAs for every SM eight times over, each then running through its share of the steps
    const unsigned gy = (unsigned)std::min<long long>({(long long)T, 65535LL, std::max<long long>(1, 1216 * 2 / gx)});
    if (V == 4) k_poisson<4><<<dim3(gx, gy), 256, 0, (cudaStream_t)stream>>>(x, rates_hz, T, BC, C, dt_ms, seed);
    else k_poisson<1><<<dim3(gx, gy), 256, 0, (cudaStream_t)stream>>>(x, rates_hz, T, BC, C, dt_ms, seed);
    NBG_CUDA(cudaGetLastError());
    return NBG_OK;
}

} // extern "C"
