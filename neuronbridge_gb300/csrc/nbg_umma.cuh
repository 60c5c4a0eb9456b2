// nbg_umma.cuh -- Blackwell (sm_103a) tensor-core GEMM for split-precision
// dense spike delivery: tcgen05.mma with the accumulator in tensor memory,
// operands staged in shared memory by bulk (TMA) copies, an mbarrier
// producer/consumer pipeline.  Included by nbg_dense.cu.
//
//   D[j][b] = sum_k W_hi^T[j][k] S[b][k] + W_lo^T[j][k] S[b][k]
//
// One CTA owns 128 post-synaptic neurons (UMMA M = 128, or 64: below) and all 64 instances
// (UMMA N = 64) over one K range (split-K).  Per 64-wide K chunk it copies
// three pre-tiled blocks (W_hi^T 16 KiB, W_lo^T 16 KiB, S 8 KiB) with
// cp.async.bulk into one of the stages; one elected thread issues
// 4 k-steps x 2 (hi, lo) tcgen05.mma of K = 16 into the same TMEM
// accumulator and commits the stage back to the producer.  The epilogue
// reads the 128 x 64 FP32 accumulator with tcgen05.ld.
//
// Operand layout (both operands K-major, no swizzle): an operand block of R
// rows x 64 K is made of 8-row x 16-byte core matrices; core matrix (row
// group i, K chunk c) sits at byte c * 128 + i * 1024, row r of it at r * 16.
// So the leading-dimension (K) byte offset is 128 and the stride-dimension
// (M/N) byte offset is 1024; k-step s of a chunk starts at byte 256 * s.
// W is stored in HBM already in this blocked order (nbg_dense.cu tiles it
// once at create time) and the update kernel writes S in it, so every stage
// is three contiguous bulk copies.
//
// Every wait on an mbarrier is bounded (clock64 deadline); on expiry the CTA
// records kUmmaTimeout in the error word, stops issuing, waits (bounded) for
// the MMAs it already issued, frees its TMEM and returns.
//
// Tiles of 64 post neurons (M = 64, half of a W block: its first or last eight
// row groups, which are contiguous) where all of them get an SM at once: up to
// 4,864 neurons on 152 SMs.  A step's tail is then half as long: 4.12 us against
// 5.02 with tiles of 128 at 128 neurons, 10.2 against 11.1 at 2,048, 19.5 against
// 19.9 at 4,864.  Above, the last of them would wait for the first.
//
// Fused step (split = 2): with an active `Finish` functor the two split-K CTAs
// of a tile form a cluster.  CTA r finishes instances [32 r, 32 r + 32): each
// sends the other its partial of the other's instances through distributed
// shared memory (16 KiB), and after one cluster barrier adds what it received
// to the accumulator it holds (two-term float addition is commutative, so the
// sum equals partial 0 + partial 1 in both) and runs the functor on each of its
// elements -- the neuron update of the step -- whose state it loaded while the
// products ran.
//
// What bounds a step: the stream of W above about 5,000 neurons, and the way
// from the last product to the next step's first operand at every size.  With
// the partials in global memory, the second CTA to arrive (found by an atomic)
// reading the other's and updating the whole tile alone, a step took 46.9 us at
// 8,192 neurons, 23.1 at 4,096 and 13.3 at 1,024; with the exchange and 16
// instances a thread 39.5, 18.9 and 9.4.  Now sixteen warps finish, eight
// instances a thread (four with M = 64), and draw the step's external spikes
// before they wait for the step before, which they do not depend on; the
// producer and the issuer have warps of their own, so that neither's work is
// behind that: 37.9, 16.8 and 7.0.
//
// W larger than the L2: the chunks of a step's last iterations (about 34 MB in
// all) are the next step's first ones and are kept (evict_last), the others
// pass through (evict_first): 46.9 -> 43.5 us at 8,192 neurons and 32.7 -> 30.5
// at 6,144 without the change above.  Kept shares of 17 to 50 MB are within 0.5
// us of it, 100 MB gives 45.6; below 100 MB of W nothing is marked (no
// difference at 4,096 neurons, 67 MB).
#pragma once

#include <cuda_bf16.h>
#include <cstdint>

namespace umma {

constexpr int kM = 128, kN = 64, kKChunk = 64;
constexpr int kUStages = 4;
constexpr int kBlockA = kM * kKChunk * 2;  // 16 KiB
constexpr int kBlockB = kN * kKChunk * 2;  // 8 KiB
constexpr int kStageBytes = 2 * kBlockA + kBlockB;
// stages (aligned up to 1024 B inside the allocation) + barrier block
constexpr int kSmemBytes = kUStages * kStageBytes + 1024 + 256;
// a tile of M = 128 or 64 post neurons (half of a W block): its stages, and the
// fused step's receive buffer (the other CTA's partial of this one's instances)
template <int M> struct Tile {
    static_assert(M == 128 || M == 64, "UMMA M");
    static constexpr int block_a = M * kKChunk * 2, stage_bytes = 2 * block_a + kBlockB;
    static constexpr int stages = M == 128 ? kUStages : 6;
    static constexpr int recv_bytes = M * (kN / 2) * 4;
    static constexpr int fused_smem = stages * stage_bytes + recv_bytes + 1024 + 256;
};
constexpr long long kKeepBytes = 34000000, kKeepAbove = 100000000; // of W, see above

// Iterations at a step's end whose chunks of W are kept in L2 (0: nothing is
// marked) for n neurons in `split` K ranges.
inline int kept_iters(int n, int split) {
    const long long w = 4ll * n * n, iters = n / kKChunk / split;
    return w > kKeepAbove ? (int)((iters * kKeepBytes + w / 2) / w) : 0;
}
// the warps that finish (16 for the fused step, 8 for partials), the producer's and the issuer's
constexpr int kFinishWarps = 16, kPartialWarps = 8;
template <class Finish> constexpr int threads() { return 32 * ((Finish::kActive ? kFinishWarps : kPartialWarps) + 2); }
constexpr int kTmemCols = 64;
constexpr int kUmmaTimeout = 4;
constexpr long long kWaitCycles = 2000000000ll; // ~1 s at 2 GHz

// byte offset of element (row, k) inside a blocked R x 64 operand block
__host__ __device__ __forceinline__ uint32_t block_offset(int row, int k) {
    return (uint32_t)((k >> 3) * 128 + (row >> 3) * 1024 + (row & 7) * 16 + (k & 7) * 2);
}

__device__ __forceinline__ uint32_t smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// UMMA shared-memory descriptor: K-major, no swizzle, sm100 version bits.
__device__ __forceinline__ uint64_t make_desc(uint32_t saddr) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr >> 4) & 0x3FFF);          // start address
    d |= (uint64_t)((128u >> 4) & 0x3FFF) << 16;     // leading-dimension byte offset (K)
    d |= (uint64_t)((1024u >> 4) & 0x3FFF) << 32;    // stride-dimension byte offset (M/N)
    d |= (uint64_t)1 << 46;                          // descriptor version for sm100
    return d;                                        // base offset 0, layout type 0 = no swizzle
}

// UMMA instruction descriptor, kind::f16: BF16 x BF16 -> F32, K-major A/B.
template <int M> __host__ __device__ constexpr uint32_t make_idesc() {
    return (1u << 4)                 // D format F32
           | (1u << 7)               // A format BF16
           | (1u << 10)              // B format BF16
           | ((uint32_t)(kN >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count));
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes)
                 : "memory");
}

// True when the phase with `parity` has completed; waits for it in hardware,
// up to a limit of the implementation's.
__device__ __forceinline__ bool mbar_try(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
                 : "=r"(ok)
                 : "r"(smem_addr(bar)), "r"(parity)
                 : "memory");
    return ok != 0;
}

// Bounded wait: true when the phase with `parity` completed, false on timeout
// or when another role of the CTA already gave up.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, volatile int *abort) {
    const long long t0 = clock64();
    while (!mbar_try(bar, parity)) {
        if (*abort) return false;
        if (clock64() - t0 > kWaitCycles) {
            *abort = 1;
            return false;
        }
    }
    return true;
}

__device__ __forceinline__ void bulk_copy(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            smem_addr(dst)),
        "l"(src), "r"(bytes), "r"(smem_addr(bar))
        : "memory");
}

// bulk_copy with an L2 eviction policy (createpolicy).
__device__ __forceinline__ void bulk_copy(void *dst, const void *src, uint32_t bytes, uint64_t *bar, uint64_t policy) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;" ::"r"(
            smem_addr(dst)),
        "l"(src), "r"(bytes), "r"(smem_addr(bar)), "l"(policy)
        : "memory");
}

__device__ __forceinline__ void mma(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(acc));
}

__device__ __forceinline__ void commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(bar))
                 : "memory");
}

__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// 8 / 16 consecutive FP32 columns of this warp's 32 TMEM lanes.
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float (&v)[8]) {
    uint32_t r[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// partial[ks][b][j] for the CTA's 128 post neurons and K range (split ks).
// wt_hi / wt_lo: blocked W^T, block (m tile, k chunk) at ((mt * kchunks + kc) * kBlockA);
// s_blk: blocked S, block kc at kc * kBlockB.
// No fused update: the partial sums are the result.
struct NoFinish {
    static constexpr bool kActive = false;
    __device__ bool drive(int) const { return false; }
    __device__ void load(int, float &, int &) const {}
    __device__ bool update(int, int, int, float, bool, float &, int &) const { return false; }
    __device__ void count(int) const {}
};

// M: post neurons of a tile (M = 64: the two halves of a 128-row block of W).
template <class Finish, int M = kM>
__global__ void __launch_bounds__(threads<Finish>(), 1)
    k_dense_umma(const __nv_bfloat16 *__restrict__ wt_hi, const __nv_bfloat16 *__restrict__ wt_lo,
                 const __nv_bfloat16 *__restrict__ s_blk, float *__restrict__ partial, int n, int split,
                 int reverse, int kept, int *__restrict__ err, const Finish fin) {
    using T = Tile<M>;
    constexpr int kStages = T::stages;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t *stages = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t *full = (uint64_t *)(stages + kStages * T::stage_bytes);
    uint64_t *empty = full + kStages;
    uint64_t *done = empty + kStages;
    uint32_t *tmem_slot = (uint32_t *)(done + 1);
    volatile int *abort = (volatile int *)(tmem_slot + 1);
    float4 *recv = reinterpret_cast<float4 *>(stages + kStages * T::stage_bytes + 256); // Finish: [16 columns / 4][j][4]

    constexpr int kProducer = threads<Finish>() / 32 - 2, kIssuer = kProducer + 1; // warps
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int mt = blockIdx.x, ks = blockIdx.y;
    const int kchunks = n / kKChunk;
    const int per = kchunks / split;
    const int kc0 = ks * per;
    const int iters = (ks == split - 1) ? kchunks - kc0 : per;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        mbar_init(done, 1);
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

    // Programmatic dependent launch: the next step's grid may be scheduled
    // as soon as every CTA of this one has started; W does not depend on the
    // previous step, so its first stages are requested before the grid
    // dependency wait (a no-op without a programmatic launch), and S and all
    // state after it.
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if constexpr (Finish::kActive) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    // K chunks in ascending order, or descending when `reverse`: the chunks a
    // step streams last are still in L2 when the next step, run in the other
    // direction, streams them first
    auto chunk = [&](int it) { return reverse ? kc0 + iters - 1 - it : kc0 + it; };
    if (warp == kProducer && lane == 0) { // producer: bulk copies into free stages
        uint64_t keep, pass;
        asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(keep));
        asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pass));
        auto copy_w = [&](int it, uint8_t *st, uint64_t *bar) {
            const size_t at = M == kM ? ((size_t)mt * kchunks + chunk(it)) * kBlockA
                                      : ((size_t)(mt >> 1) * kchunks + chunk(it)) * kBlockA + (size_t)(mt & 1) * T::block_a;
            if (kept == 0) {
                bulk_copy(st, (const uint8_t *)wt_hi + at, T::block_a, bar);
                bulk_copy(st + T::block_a, (const uint8_t *)wt_lo + at, T::block_a, bar);
            } else {
                const uint64_t p = it >= iters - kept ? keep : pass;
                bulk_copy(st, (const uint8_t *)wt_hi + at, T::block_a, bar, p);
                bulk_copy(st + T::block_a, (const uint8_t *)wt_lo + at, T::block_a, bar, p);
            }
        };
        const int pre = iters < kStages ? iters : kStages;
        for (int it = 0; it < pre; ++it) {
            mbar_expect_tx(&full[it], T::stage_bytes);
            copy_w(it, stages + it * T::stage_bytes, &full[it]);
        }
        asm volatile("griddepcontrol.wait;" ::: "memory");
        for (int it = 0; it < pre; ++it)
            bulk_copy(stages + it * T::stage_bytes + 2 * T::block_a, (const uint8_t *)s_blk + (size_t)chunk(it) * kBlockB,
                      kBlockB, &full[it]);
        for (int it = pre; it < iters; ++it) {
            const int s = it % kStages;
            if (!mbar_wait(&empty[s], ((it / kStages) & 1) ^ 1, abort)) break;
            uint8_t *st = stages + s * T::stage_bytes;
            mbar_expect_tx(&full[s], T::stage_bytes);
            copy_w(it, st, &full[s]);
            bulk_copy(st + 2 * T::block_a, (const uint8_t *)s_blk + (size_t)chunk(it) * kBlockB, kBlockB, &full[s]);
        }
    } else if (warp == kIssuer && lane == 0) { // MMA issuer
        constexpr uint32_t idesc = make_idesc<M>();
        int issued = 0;
        for (int it = 0; it < iters; ++it) {
            const int s = it % kStages;
            if (!mbar_wait(&full[s], (it / kStages) & 1, abort)) break;
            fence_after();
            const uint32_t a_hi = smem_addr(stages + s * T::stage_bytes);
            const uint32_t a_lo = a_hi + T::block_a;
            const uint32_t b = a_hi + 2 * T::block_a;
#pragma unroll
            for (int k = 0; k < kKChunk / 16; ++k) {
                mma(tmem, make_desc(a_hi + 256 * k), make_desc(b + 256 * k), idesc, (it | k) != 0);
                mma(tmem, make_desc(a_lo + 256 * k), make_desc(b + 256 * k), idesc, 1u);
            }
            commit(&empty[s]); // frees the stage once these MMAs have read it
            ++issued;
        }
        commit(done); // arrives when every MMA issued above has completed
        (void)issued;
    }
    __syncwarp();
    if constexpr (Finish::kActive) {
        // warp w finishes the post neurons of TMEM lanes 32*(w%4).. and instances
        // 32*ks + 8*(w/4)..; with M = 64 a quarter of the lanes holds sixteen rows in
        // its first half, and the two halves of the warp share the eight instances
        constexpr int kOwn = M == kM ? 8 : 4;
        const bool finishes = warp < kFinishWarps;
        const int q = warp & 3, g = warp >> 2;
        const int jl = M == kM ? 32 * q + lane : 16 * q + (lane & 15), j = mt * M + jl;
        const int c0 = M == kM ? 0 : lane >> 4 << 2;
        const int b0 = 32 * ks + 8 * g, sent = 32 * (ks ^ 1) + 8 * g;
        float vv[kOwn];
        int ls[kOwn];
        unsigned drive = 0u; // this step's external spikes do not depend on the step before
        if (finishes) {
#pragma unroll
            for (int c = 0; c < kOwn; ++c) drive |= fin.drive((b0 + c0 + c) * n + j) ? 1u << c : 0u;
        }
        asm volatile("griddepcontrol.wait;" ::: "memory"); // before touching anything the previous step wrote
        if (finishes) {
#pragma unroll
            for (int c = 0; c < kOwn; ++c) fin.load((b0 + c0 + c) * n + j, vv[c], ls[c]); // while the products run
        }
        mbar_wait(done, 0, abort);
        // uniform across the block before the warp-collective tcgen05.ld
        __syncthreads();
        fence_after();
        const bool ok = finishes && !*abort;
        float own[8], oth[8];
        asm volatile("barrier.cluster.wait.aligned;" ::: "memory"); // the other CTA has started
        if (ok) {
            const uint32_t lanes = tmem + ((uint32_t)(32 * q) << 16);
            tmem_ld8(lanes + (uint32_t)sent, oth);
            uint32_t ra;
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
                         : "=r"(ra)
                         : "r"(smem_addr(recv + 2 * g * M + jl)), "r"(ks ^ 1));
            if (M == kM || lane < 16) {
#pragma unroll
                for (int c = 0; c < 8; c += 4)
                    asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(ra + (uint32_t)(c / 4 * M * 16)),
                                 "f"(oth[c]), "f"(oth[c + 1]), "f"(oth[c + 2]), "f"(oth[c + 3])
                                 : "memory");
            }
            tmem_ld8(lanes + (uint32_t)b0, own);
            if constexpr (M != kM) {
#pragma unroll
                for (int c = 0; c < kOwn; ++c) {
                    const float x = __shfl_sync(0xffffffffu, own[c + 4], lane & 15);
                    own[c] = lane < 16 ? own[c] : x;
                }
            }
        }
        fence_before();
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
        if (ok) {
#pragma unroll
            for (int c = 0; c < kOwn; c += 4) {
                const float4 x = recv[(2 * g + (c0 + c) / 4) * M + jl];
                oth[c] = x.x;
                oth[c + 1] = x.y;
                oth[c + 2] = x.z;
                oth[c + 3] = x.w;
            }
            int spikes = 0;
#pragma unroll
            for (int c = 0; c < kOwn; ++c)
                spikes += fin.update(b0 + c0 + c, j, (b0 + c0 + c) * n + j, own[c] + oth[c], drive >> c & 1u, vv[c], ls[c])
                              ? 1
                              : 0;
            for (int o = 16; o > 0; o >>= 1) spikes += __shfl_down_sync(0xffffffffu, spikes, o);
            if (lane == 0) fin.count(spikes);
        }
    } else {
        static_assert(M == kM, "partials are written for whole blocks");
        asm volatile("griddepcontrol.wait;" ::: "memory");
        const int q = warp & 3, h = warp >> 2, j = mt * M + 32 * q + lane;
        // warp w reads TMEM lanes 32*(w%4).. (post neurons) and columns 32*(w/4).. (instances)
        mbar_wait(done, 0, abort);
        __syncthreads();
        fence_after();
        if (warp < kPartialWarps && !*abort) {
            float acc[2][16];
            float *out = partial + (size_t)ks * kN * n;
            tmem_ld16(tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)(32 * h), acc[0]);
            tmem_ld16(tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)(32 * h + 16), acc[1]);
#pragma unroll
            for (int c = 0; c < 32; ++c) out[(size_t)(32 * h + c) * n + j] = acc[c >> 4][c & 15];
        }
        fence_before();
    }
    __syncthreads();
    if (threadIdx.x == 0 && *abort) atomicOr(err, kUmmaTimeout);
    if (warp == 2) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
    }
}

} // namespace umma
