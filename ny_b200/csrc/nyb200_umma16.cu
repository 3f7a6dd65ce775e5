// tcgen05 contraction of the bound, adjoint and attack passes: C[M x N] = A[M x K] * W[K x N], fp32 in and out, computed
// as three fp16 products of split operands (kind::f16, fp32 accumulators in tensor memory).
//
// Operands: a = 2^-s (ah + 2^-11 al) with fp16 parts, 22 bits together, the same a TF32 pair holds; kind::f16 takes twice
// the products per cycle of kind::tf32 and half the operand bytes.  fp16 has five exponent bits, so A is scaled by a
// power of two per row and K chunk of 64 (largest magnitude in [2^14, 2^15)), W by one per layer; a chunk is one
// accumulation chain, and the epilogue undoes its scale in the multiply-add that joins it to the row's fp32 sums.
//
// What bounds it: shared memory and the L2 port.  A 128 x 256 product step reads 12 KB of operands in 128 tensor cycles,
// and with the tiles' arrival (64 KB of weights, 32 KB of A per chunk of 1536 cycles) that is more than a single SM's 128
// bytes per cycle.  So wide products run on CTA pairs (cta_group::2, 256 x 256 tiles): either CTA holds its own
// 128 rows and half of the weights, which halves the weights' bytes on every path.  Small products take single CTAs and
// tiles of 128 or 64 columns, spread over more SMs (pick_tile).
//
// Persistent CTAs, one per SM, 640 threads:
//   warp 0      TMA: the weight tiles Wh^T, Wl^T (K-major, 128-byte swizzle, 64-row boxes) and the fp32 tile of A, which
//               lands where its fp16 parts will lie; the first weights before the previous kernel of the stream has ended
//               (no kernel writes weights);
//   warp 1      the pair's first CTA: issues the products, the whole warp with one elected lane; per chunk Al*Wh + Ah*Wl first,
//               then Ah*Wh with the accumulator scaled by 2^-11 at its first step (scale-input-d): the cross terms round at
//               their own magnitude and join exactly.  The second CTA: reports its operands, weights and split rows, to the first;
//   warp 2      owns the tensor memory (two accumulators of BN columns);
//   warps 4-11  epilogue: thread = one row, BN / 2 columns in registers; results leave by TMA through 4 KB per warp (row
//               per thread, direct stores took 32 lines per instruction and 10 of a tile's 25 thousand cycles);
//   warps 12-19 split the fp32 tile in place: eight lanes hold 64 values of a row, whose largest magnitude is three
//               shuffles, and the parts of a row's 256 bytes lie in the same 256 bytes, so a warp synchronises with itself
//               alone.  Operands a tensor map cannot describe are loaded directly.
// Across a pair: split rows and weights are reported to the first CTA by one thread (arrive_first; its memory barrier is on the
// way of every chunk: the optimisation of 2048 cells takes 45.1 ms with it, 43.4 with an arrival that orders nothing beyond its
// CTA), drained accumulators by every epilogue warp (arrive_first_relaxed; one thread with a barrier there too: 45.9 ms).
// The scales an epilogue warp has read go back to its own CTA's splitting warps by a barrier of theirs.
// A long contraction with few tiles is cut into K segments, each an output of its own, added in a fixed order by
// k_sum_segments.
//
// Rounding against S = |A||W| (f16_eps): operand split 0.75 * 2^-20; at most one fp32 ulp of the accumulated magnitude per
// MMA step, eight of size 2^-10 S and four of size S per chunk; one fp32 rounding per chunk and segment.  An element more
// than 2^29 times smaller than its chunk's largest loses low bits to the exponent range, an absolute error of at most
// 2^-50 of that largest: q carries it (NetView::qfl).  A layer whose weights span more than that keeps its TF32 form.
// tests/test_gpu_rates.py holds every element of a product against that rate.
#include <cuda.h>
#include <cuda_fp16.h>

#include <algorithm>

#include "nyb200_internal.cuh"
#include "nyb200_tcgen05.cuh"

namespace nyb {

namespace f16 {

constexpr int BM = 128, BK = 64, THREADS = 640;
constexpr int A_PART = BM * BK * 2, A_BYTES = 2 * A_PART;       // 16 KB per part; the fp32 tile is two boxes of 32 columns of that size
constexpr int RING_BYTES = 192 * 1024, SCALES = 5;              // operand stages; chunks whose scales are kept
constexpr int OUT_BYTES = 32 * 32 * 4;                          // per epilogue warp: 32 rows of 32 columns
constexpr int SMEM_BYTES = RING_BYTES + 8 * OUT_BYTES + SCALES * BM * 4 + 512 /*barriers*/;
static_assert(SMEM_BYTES <= 232448, "more than the 227 KB a CTA can opt into");
constexpr int REGS_LAUNCH = 96, REGS_CONTROL = 40, REGS_EPILOGUE = 160, REGS_PRODUCER = 56;   // see nyb200_umma.cu
static_assert(4 * 32 * REGS_CONTROL + 8 * 32 * REGS_EPILOGUE + 8 * 32 * REGS_PRODUCER <= THREADS * REGS_LAUNCH, "setmaxnreg targets exceed the CTA's registers");

struct Params {
    const float *A;
    float *C;
    long lda, ldc, seg_stride;    // seg_stride: distance of two segments' outputs
    int M, N, K, chunks, segs, per_seg;
    int a_tma, c_tma;             // A and C by TMA, or directly
    float w_inv;
    int *err;
};

}  // namespace f16

using namespace umma;
using namespace f16;

// An arrival at a barrier of the pair's first CTA: a release to the cluster, so that what this thread has written or has seen
// written by its own CTA's warps is ordered before what the first CTA does after the barrier's phase.  It is a full memory
// barrier; one thread per chunk does it for all warps, which report to a barrier of their own CTA.
__device__ __forceinline__ void arrive_first(unsigned bar) {
    asm volatile(
        "{\n\t.reg .b32 r;\n\t"
        "mapa.shared::cluster.u32 r, %0, 0;\n\t"
        "mbarrier.arrive.release.cluster.shared::cluster.b64 _, [r];\n\t}" ::"r"(bar) : "memory");
}
// The same for tensor memory alone, which has an order of its own: what was loaded before tcgen05.fence::before_thread_sync and
// this arrival is out of the accumulator before the products that follow the wait and tcgen05.fence::after_thread_sync.
__device__ __forceinline__ void arrive_first_relaxed(unsigned bar) {
    asm volatile(
        "{\n\t.reg .b32 r;\n\t"
        "mapa.shared::cluster.u32 r, %0, 0;\n\t"
        "mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [r];\n\t}" ::"r"(bar) : "memory");
}
// The waits that go with them.
template <bool ACQUIRE>
__device__ __forceinline__ bool wait_second(unsigned bar, unsigned parity) {
    const long long t0 = clock64();
    for (;;) {
        unsigned ok;
        if constexpr (ACQUIRE)
            asm volatile(
                "{\n\t.reg .pred p;\n\t"
                "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
                "selp.u32 %0, 1, 0, p;\n\t}"
                : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
        else
            asm volatile(
                "{\n\t.reg .pred p;\n\t"
                "mbarrier.try_wait.parity.relaxed.cluster.shared::cta.b64 p, [%1], %2;\n\t"
                "selp.u32 %0, 1, 0, p;\n\t}"
                : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
        if (ok) return true;
        if (clock64() - t0 > WAIT_LIMIT_CYCLES) return false;
    }
}
template <int CG>
__device__ __forceinline__ void mma_elect(unsigned d, unsigned long long a, unsigned long long b, unsigned idesc, unsigned accumulate) {
    if constexpr (CG == 1) mma_f16_elect(d, a, b, idesc, accumulate);
    else
        asm volatile(
            "{\n\t.reg .pred p, q;\n\t"
            "elect.sync _|q, 0xffffffff;\n\t"
            "setp.ne.b32 p, %4, 0;\n\t"
            "@q tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
            ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}
// The accumulator scaled by 2^-11 before the products are added.
template <int CG>
__device__ __forceinline__ void mma_scaled_elect(unsigned d, unsigned long long a, unsigned long long b, unsigned idesc) {
    if constexpr (CG == 1)
        asm volatile(
            "{\n\t.reg .pred p, q;\n\t"
            "elect.sync _|q, 0xffffffff;\n\t"
            "setp.ne.b32 p, 1, 0;\n\t"
            "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p, 11;\n\t}"
            ::"r"(d), "l"(a), "l"(b), "r"(idesc) : "memory");
    else
        asm volatile(
            "{\n\t.reg .pred p, q;\n\t"
            "elect.sync _|q, 0xffffffff;\n\t"
            "setp.ne.b32 p, 1, 0;\n\t"
            "@q tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p, 11;\n\t}"
            ::"r"(d), "l"(a), "l"(b), "r"(idesc) : "memory");
}
// Arrives at the barrier (of both CTAs of a pair) when the products issued so far are done.
template <int CG>
__device__ __forceinline__ void commit_elect(unsigned bar) {
    if constexpr (CG == 1) mma_commit_elect(bar);
    else
        asm volatile(
            "{\n\t.reg .pred q;\n\t"
            "elect.sync _|q, 0xffffffff;\n\t"
            "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n\t}" ::"r"(bar), "h"((unsigned short)3)
            : "memory");
}
__device__ __forceinline__ void tma_store_2d(const CUtensorMap *tm, int x, int y, unsigned src) {
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];" ::"l"(tm), "r"(x), "r"(y), "r"(src) : "memory");
}

// Two fp32 operations per instruction (the split and the drain are bound by issue slots).
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
    float2 r;
    asm("{\n\t.reg .b64 x, y;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmul.rn.f32x2 x, x, y;\n\tmov.b64 {%0, %1}, x;\n\t}"
        : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return r;
}
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    float2 r;
    asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmov.b64 z, {%6, %7};\n\tfma.rn.f32x2 x, x, y, z;\n\tmov.b64 {%0, %1}, x;\n\t}"
        : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return r;
}
__device__ __forceinline__ float max3_abs(float a, float b, float c) {
    float r;
    asm("max.abs.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// CG: CTAs that share a tile of CG * 128 rows and BN columns.
template <int BN, int CG>
__global__ void __launch_bounds__(f16::THREADS, 1)
k_umma_f16(const __grid_constant__ CUtensorMap tm_hi, const __grid_constant__ CUtensorMap tm_lo, const __grid_constant__ CUtensorMap tm_a,
           const __grid_constant__ CUtensorMap tm_c, const __grid_constant__ f16::Params P, const __grid_constant__ ConcFuse cf) {
    constexpr int W_ROWS = BN / CG, W_PART = W_ROWS * BK * 2, STAGE = A_BYTES + 2 * W_PART, STAGES = 3, COLS = BN / 2;
    static_assert(STAGES * STAGE <= RING_BYTES, "operand stages");
    static_assert(STAGES + 2 <= SCALES, "a chunk's scales outlive its stage by two chunks");
    extern __shared__ unsigned char smem_raw[];
    // No room to align it here: a kernel without static shared memory starts at a multiple of 1024 (checked below).
    unsigned char *smem = smem_raw;
    unsigned char *out_base = smem + RING_BYTES;
    float *scales = (float *)(out_base + 8 * OUT_BYTES);
    unsigned long long *bars = (unsigned long long *)(scales + SCALES * BM);
    unsigned long long *b_a = bars, *b_raw = b_a + STAGES, *b_w = b_raw + STAGES, *b_w2 = b_w + STAGES, *b_empty = b_w2 + STAGES,
                       *b_full = b_empty + STAGES, *b_drained = b_full + 2, *b_scales = b_drained + 2;
    unsigned *tmem_slot = (unsigned *)(b_scales + SCALES);
    volatile int *abort_flag = (volatile int *)(tmem_slot + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = CG == 1 ? 0 : (int)(blockIdx.x & 1);
    pdl_trigger();
    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(smem_u32(&b_a[s]), 8); mbar_init(smem_u32(&b_raw[s]), 1); mbar_init(smem_u32(&b_w[s]), 1);
            mbar_init(smem_u32(&b_w2[s]), 1); mbar_init(smem_u32(&b_empty[s]), 1);
        }
        for (int b = 0; b < 2; ++b) { mbar_init(smem_u32(&b_full[b]), 1); mbar_init(smem_u32(&b_drained[b]), 8 * CG); }
        for (int s = 0; s < SCALES; ++s) mbar_init(smem_u32(&b_scales[s]), 8);
        *abort_flag = 0;
        if (smem_u32(smem) & 1023u) atomicExch(P.err, 38);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 2) {
        if constexpr (CG == 1) {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(tmem_slot)) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(tmem_slot)) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        }
    }
    auto meet = [&]() {   // all threads of the tile's CTAs
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncthreads();
        if constexpr (CG == 2) {
            asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
            asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    };
    meet();
    const unsigned tmem_base = *tmem_slot;
    const int n_tiles = (P.N + BN - 1) / BN, tiles = ((P.M + CG * BM - 1) / (CG * BM)) * n_tiles * P.segs;
    const int t_first = (smem_u32(smem) & 1023u) ? tiles : (int)blockIdx.x / CG, t_step = gridDim.x / CG;
    // tile t: row block, column block, segment (consecutive tiles share the rows of A)
    auto chunks_of = [&](int t, int &c0) { c0 = (t % P.segs) * P.per_seg; return min(P.per_seg, P.chunks - c0); };
    auto row_of = [&](int t) { return ((t / P.segs / n_tiles) * CG + rank) * BM; };
    // a partial column tile only multiplies the columns it has (rounded up to the granule of 16 per CTA)
    auto width_of = [&](int t) { return min(BN, (P.N - (t / P.segs) % n_tiles * BN + 16 * CG - 1) / (16 * CG) * (16 * CG)); };

    if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REGS_CONTROL));
        if (warp == 0 && lane == 0) {
            // ------------------------------------------------------------ loads
            auto load_w = [&](int t, int c, unsigned s) {
                const int w = width_of(t) / CG, n0 = (t / P.segs) % n_tiles * BN + rank * w, boxes = (w + 63) / 64;
                unsigned char *dst = smem + s * STAGE + A_BYTES;
                const unsigned bar = smem_u32(&b_w[s]);
                mbar_expect_tx(bar, (unsigned)(boxes * 2 * 64 * BK * 2));
                for (int b = 0; b < boxes; ++b) {
                    tma_load_2d(smem_u32(dst + b * 64 * BK * 2), &tm_hi, c * BK, n0 + b * 64, bar);
                    tma_load_2d(smem_u32(dst + W_PART + b * 64 * BK * 2), &tm_lo, c * BK, n0 + b * 64, bar);
                }
            };
            auto load_a = [&](int t, int c, unsigned s) {
                if (!P.a_tma) return;
                const unsigned bar = smem_u32(&b_raw[s]);
                const int row = row_of(t);
                mbar_expect_tx(bar, (unsigned)A_BYTES);
                tma_load_2d(smem_u32(smem + s * STAGE), &tm_a, c * BK, row, bar);
                tma_load_2d(smem_u32(smem + s * STAGE + A_PART), &tm_a, c * BK + 32, row, bar);
            };
            // the first stages' weights, then, once the earlier kernels are done, their rows of A
            int t = t_first, c = 0, c0 = 0, nc = t < tiles ? chunks_of(t, c0) : 0;
            auto next = [&]() { if (++c == nc) { c = 0; t += t_step; if (t < tiles) nc = chunks_of(t, c0); } };
            for (int s = 0; s < STAGES && t < tiles; ++s, next()) load_w(t, c0 + c, s);
            pdl_wait();
            t = t_first; c = 0; nc = t < tiles ? chunks_of(t, c0) : 0;
            for (int s = 0; s < STAGES && t < tiles; ++s, next()) load_a(t, c0 + c, s);
            unsigned s = 0, ph = 0;
            for (; t < tiles && !*abort_flag; next()) {
                if (!mbar_wait_soon(smem_u32(&b_empty[s]), ph)) { atomicExch(P.err, 31); *abort_flag = 1; break; }
                load_w(t, c0 + c, s);
                load_a(t, c0 + c, s);
                if (++s == STAGES) { s = 0; ph ^= 1; }
            }
        } else if (warp == 1 && rank == 0) {
            // ------------------------------------------------------------ products
            unsigned s = 0, ph = 0, buf = 0, bph = 1;
            bool ok = true;
            const unsigned long long d0 = make_desc(smem_u32(smem));
            for (int t = t_first; t < tiles && ok && !*abort_flag; t += t_step) {
                int c0;
                const int nc = chunks_of(t, c0);
                const unsigned idesc = make_idesc_f16(BM * CG, width_of(t));
                for (int c = 0; c < nc; ++c) {
                    ok = CG == 1 ? mbar_wait_soon(smem_u32(&b_drained[buf]), bph) : wait_second<false>(smem_u32(&b_drained[buf]), bph);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) { if (lane == 0) { atomicExch(P.err, 32); *abort_flag = 1; } break; }
                    ok = mbar_wait_soon(smem_u32(&b_w[s]), ph) && mbar_wait_soon(smem_u32(&b_a[s]), ph) && (CG == 1 || wait_second<true>(smem_u32(&b_w2[s]), ph));
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) { if (lane == 0) { atomicExch(P.err, 33); *abort_flag = 1; } break; }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const int steps = min(BK / 16, (P.K - (c0 + c) * BK + 15) / 16);
                    const unsigned long long ah = d0 + (s * STAGE >> 4), al = ah + (A_PART >> 4), wh = ah + (A_BYTES >> 4), wl = wh + (W_PART >> 4);
                    const unsigned d = tmem_base + buf * BN;
                    for (int k = 0; k < steps; ++k) {   // 16 values = 32 bytes = two 16-byte units
                        mma_elect<CG>(d, al + 2 * k, wh + 2 * k, idesc, k > 0 ? 1u : 0u);
                        mma_elect<CG>(d, ah + 2 * k, wl + 2 * k, idesc, 1u);
                    }
                    mma_scaled_elect<CG>(d, ah, wh, idesc);
                    for (int k = 1; k < steps; ++k) mma_elect<CG>(d, ah + 2 * k, wh + 2 * k, idesc, 1u);
                    commit_elect<CG>(smem_u32(&b_empty[s]));
                    commit_elect<CG>(smem_u32(&b_full[buf]));
                    if (++s == STAGES) { s = 0; ph ^= 1; }
                    if ((buf ^= 1) == 0) bph ^= 1;
                }
            }
        } else if (CG == 2 && warp == 1 && lane == 0) {
            // ------------------------------------------------------------ the second CTA's operands are ready
            unsigned s = 0, ph = 0;
            bool ok = true;
            for (int t = t_first; t < tiles && ok && !*abort_flag; t += t_step) {
                int c0;
                for (int c = 0, nc = chunks_of(t, c0); c < nc; ++c) {
                    ok = mbar_wait_soon(smem_u32(&b_w[s]), ph) && mbar_wait_soon(smem_u32(&b_a[s]), ph);
                    if (!ok) { atomicExch(P.err, 37); *abort_flag = 1; break; }
                    arrive_first(smem_u32(&b_w2[s]));
                    if (++s == STAGES) { s = 0; ph ^= 1; }
                }
            }
        }
    } else if (warp < 12) {
        // ---------------------------------------------------------------- epilogue
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(REGS_EPILOGUE));
        pdl_wait();   // C may still be read by an earlier kernel
        const int q = warp & 3, half = (warp - 4) >> 2, r = q * 32 + lane;
        unsigned char *out = out_base + (warp - 4) * OUT_BYTES;
        unsigned buf = 0, bph = 0, slot = 0;
        bool dead = false;
        for (int t = t_first; t < tiles && !dead; t += t_step) {
            int c0;
            const int nc = chunks_of(t, c0), tn = (t / P.segs) % n_tiles;
            const int col0 = tn * BN + half * COLS, ncols = min(COLS, P.N - col0);
            float2 acc[COLS / 2];
#pragma unroll
            for (int j = 0; j < COLS / 2; ++j) acc[j] = make_float2(0.f, 0.f);
            for (int c = 0; c < nc; ++c) {
                const bool ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&b_full[buf]), bph));
                if (!ok) { if (lane == 0) { atomicExch(P.err, 34); *abort_flag = 1; } dead = true; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const float inv = scales[slot * BM + r];
                const unsigned addr = tmem_base + ((unsigned)(q * 32) << 16) + (unsigned)(buf * BN + half * COLS);
                if (ncols > 0) {
#pragma unroll
                    for (int j = 0; j < COLS; j += 16) {
                        unsigned v[16];
                        tmem_ld16(addr + j, v);
                        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                        for (int i = 0; i < 8; ++i)
                            acc[j / 2 + i] = fma2(make_float2(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1])), make_float2(inv, inv), acc[j / 2 + i]);
                    }
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) {
                    if constexpr (CG == 1) mbar_arrive(smem_u32(&b_drained[buf]));
                    else { arrive_first_relaxed(smem_u32(&b_drained[buf])); mbar_arrive(smem_u32(&b_scales[slot])); }
                }
                if (++slot == SCALES) slot = 0;
                if ((buf ^= 1) == 0) bph ^= 1;
            }
            if (dead) break;
#pragma unroll
            for (int j = 0; j < COLS / 2; ++j) acc[j] = mul2(acc[j], make_float2(P.w_inv, P.w_inv));
            auto sum = [&](int j) { return j & 1 ? acc[j / 2].y : acc[j / 2].x; };
            const int row0 = row_of(t) + q * 32, row = row0 + lane;
            if (cf.on && row < P.M) {
                // fused concretisation: this thread's columns of the finished row against the input box
                double s = 0.0;
                float sa = 0.f;   // magnitude sum, rounded upwards: it only scales the charge of the additions
                bool bad = false;
                if (ncols > 0) {
                    const int d = row / cf.R, rr = row - d * cf.R;
                    const bool upper = rr >= cf.S;
                    const float *xl = cf.in_lo + (long)d * cf.box_ds + col0, *xu = cf.in_hi + (long)d * cf.box_ds + col0;
                    const bool vec = ncols == COLS && (((reinterpret_cast<uintptr_t>(xl) | reinterpret_cast<uintptr_t>(xu)) & 15) == 0);
                    auto term = [&](float a, float l, float u) {
                        const bool nonneg = !(__float_as_uint(a) >> 31) || (__float_as_uint(a) & 0x7fffffffu) == 0;
                        const float x = (nonneg != upper) ? l : u;
                        bad |= !(fabsf(a) < 1e10f);  // is_crown_coeff_safe, crates/ny-core/src/gemm.rs:127
                        // a zero factor contributes nothing, whatever the other one is (no 0 * inf)
                        if (a != 0.f && x != 0.f) {
                            s = fma((double)a, (double)x, s);
                            sa = __fmaf_ru(fabsf(a), fabsf(x), sa);
                        }
                    };
                    if (vec) {
#pragma unroll
                        for (int j = 0; j < COLS; j += 4) {
                            const float4 l = *(const float4 *)(xl + j), u = *(const float4 *)(xu + j);
                            term(sum(j), l.x, u.x); term(sum(j + 1), l.y, u.y); term(sum(j + 2), l.z, u.z); term(sum(j + 3), l.w, u.w);
                        }
                    } else {
#pragma unroll
                        for (int j = 0; j < COLS; ++j) if (j < ncols) term(sum(j), xl[j], xu[j]);
                    }
                }
                double *part = cf.part + ((long)row * cf.slots + tn * 2 + half) * 2;
                part[0] = s; part[1] = (double)sa;
                if (bad) cf.bad[row] = 1;
            }
            if (ncols <= 0 || (cf.on && !cf.store)) continue;
            if (P.c_tma) {   // rows and columns past the end are clipped by the tensor map
                if (row0 < P.M)
#pragma unroll
                    for (int j = 0; j < COLS; j += 32) {
                        if (j >= ncols) break;
                        if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                        __syncwarp();
#pragma unroll
                        for (int u = 0; u < 8; ++u)   // 128-byte swizzle: eight lanes' 16-byte units cover all banks
                            *(float4 *)(out + lane * 128 + ((u ^ (lane & 7)) << 4)) = make_float4(sum(j + 4 * u), sum(j + 4 * u + 1), sum(j + 4 * u + 2), sum(j + 4 * u + 3));
                        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                        __syncwarp();
                        if (lane == 0) {
                            tma_store_2d(&tm_c, col0 + j, row0, smem_u32(out));
                            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                        }
                    }
            } else if (row < P.M) {
                float *crow = P.C + (long)(t % P.segs) * P.seg_stride + (long)row * P.ldc + col0;
#pragma unroll
                for (int j = 0; j < COLS; ++j) if (j < ncols) crow[j] = sum(j);
            }
        }
        if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    } else {
        // ---------------------------------------------------------------- operand split
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REGS_PRODUCER));
        pdl_wait();
        const int w = warp - 12, l8 = lane & 7, rsub = lane >> 3;
        // group g of eight rows: rows 2 g + {0, 4, 1, 5}, so that a store's sixteen lanes reach both halves of the swizzled lines
        const int r0 = w * 16 + (rsub & 1) * 4 + (rsub >> 1);
        // byte offsets in the tile: the fp32 values read, the parts written; group g: ^ 32 g, + 256 g; the parts' second box: ^ 64
        const unsigned off_r = r0 * 128 + ((l8 ^ (r0 & 7)) << 4), off_w = r0 * 128 + (((l8 >> 1) ^ (r0 & 7)) << 4) + (l8 & 1) * 8;
        unsigned s = 0, ph = 0, slot = 0, sph = 1;
        bool dead = false;
        for (int t = t_first; t < tiles && !dead; t += t_step) {
            int c0;
            const int nc = chunks_of(t, c0), row_base = row_of(t);
            for (int c = 0; c < nc; ++c) {
                const bool ok = __all_sync(0xffffffffu, (P.a_tma ? mbar_wait(smem_u32(&b_raw[s]), ph) : mbar_wait(smem_u32(&b_empty[s]), ph ^ 1)) &&
                                                            (CG == 1 || mbar_wait(smem_u32(&b_scales[slot]), sph)));
                if (!ok) { if (lane == 0) { atomicExch(P.err, 35); *abort_flag = 1; } dead = true; break; }
                unsigned char *ah = smem + s * STAGE;
                float *sc_row = scales + slot * BM + r0;
#pragma unroll
                for (int h = 0; h < 2; ++h) {   // eight rows at a time, a lane's two of them in registers
                    float4 v[4];
                    if (P.a_tma) {
#pragma unroll
                        for (int g = 0; g < 2; ++g) {
                            const unsigned char *src = ah + (off_r ^ (g << 5)) + h * 1024 + g * 256;
                            v[2 * g] = *(const float4 *)src;
                            v[2 * g + 1] = *(const float4 *)(src + A_PART);
                        }
                        __syncwarp();   // the warp's eight rows have been read: their parts take their place
                    } else {
                        const int k = (c0 + c) * BK + l8 * 4;
#pragma unroll
                        for (int g = 0; g < 2; ++g) {
                            // rows past the last one read it again: their results are not stored
                            const float *src = P.A + (long)min(row_base + r0 + h * 8 + g * 2, P.M - 1) * P.lda + k;
#pragma unroll
                            for (int p = 0; p < 2; ++p)
                                v[2 * g + p] = make_float4(k + p * 32 < P.K ? src[p * 32] : 0.f, k + p * 32 + 1 < P.K ? src[p * 32 + 1] : 0.f,
                                                           k + p * 32 + 2 < P.K ? src[p * 32 + 2] : 0.f, k + p * 32 + 3 < P.K ? src[p * 32 + 3] : 0.f);
                        }
                    }
#pragma unroll
                    for (int g = 0; g < 2; ++g) {
                        const float4 x0 = v[2 * g], x1 = v[2 * g + 1];
                        float m = fmaxf(max3_abs(max3_abs(x0.x, x0.y, x0.z), x0.w, x1.x), max3_abs(x1.y, x1.z, x1.w));
                        m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 1));
                        m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 2));
                        m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 4));
                        // exponent field of the power of two that brings m into [2^14, 2^15), within fp32's range (an
                        // infinite m stays infinite, a zero one zero)
                        const unsigned f = (unsigned)min(268 - (int)(__float_as_uint(m) >> 23), 253);
                        const float sc = __uint_as_float(f << 23);
                        if (l8 == 0) sc_row[h * 8 + g * 2] = __uint_as_float((254 - f) << 23);
#pragma unroll
                        for (int p = 0; p < 2; ++p) {
                            const float4 x = p ? x1 : x0;
                            const float2 a = mul2(make_float2(x.x, x.y), make_float2(sc, sc)), b = mul2(make_float2(x.z, x.w), make_float2(sc, sc));
                            const __half2 h0 = __floats2half2_rn(a.x, a.y), h1 = __floats2half2_rn(b.x, b.y);
                            // 2048 (a - high part), exact
                            const float2 k2 = make_float2(2048.f, 2048.f), kn = make_float2(-2048.f, -2048.f);
                            const float2 la = fma2(__half22float2(h0), kn, mul2(a, k2)), lb = fma2(__half22float2(h1), kn, mul2(b, k2));
                            const __half2 q0 = __floats2half2_rn(la.x, la.y), q1 = __floats2half2_rn(lb.x, lb.y);
                            unsigned char *dst = ah + (off_w ^ (g << 5) ^ (p << 6)) + h * 1024 + g * 256;
                            *(uint2 *)dst = make_uint2(*(const unsigned *)&h0, *(const unsigned *)&h1);
                            *(uint2 *)(dst + A_PART) = make_uint2(*(const unsigned *)&q0, *(const unsigned *)&q1);
                        }
                    }
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&b_a[s]));
                if (++s == STAGES) { s = 0; ph ^= 1; }
                if (++slot == SCALES) { slot = 0; sph ^= 1; }
            }
        }
    }
    meet();   // the other CTA's last products read this one's shared memory
    if (warp == 2) {
        if constexpr (CG == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem_base) : "memory");
        else asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(tmem_base) : "memory");
    }
}

// C[m][n] = the segments' outputs, added in order.
__global__ void __launch_bounds__(256)
k_sum_segments(long total, int N, int segs, const float *__restrict__ part, float *__restrict__ C, long ldc) {
    pdl_trigger();
    pdl_wait();
    const long t = (long)blockIdx.x * 256 + threadIdx.x;
    if (t >= total) return;
    float s = part[t];
    for (int i = 1; i < segs; ++i) s += part[(long)i * total + t];
    C[t / N * ldc + t % N] = s;
}

// An operand [K x N] scaled by 2^e into fp16 high and low parts, transposed and K-padded: [2][N][kpad].
__global__ void k_split_weights_f16(WeightSource src, int K, int N, int kpad, float scale, __half *__restrict__ out) {
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x, n_el = (long)N * kpad;
    if (t >= n_el) return;
    const int n = (int)(t / kpad), k = (int)(t % kpad);
    const float w = k < K ? weight_at(src, k, n, K, N) * scale : 0.f;
    const __half h = __float2half_rn(w);
    out[t] = h;
    out[n_el + t] = __float2half_rn((w - __half2float(h)) * 2048.f);
}

// ---------------------------------------------------------------- host side
// Segments of a contraction: at least one per 64 chunks (4096 values), which bounds the fp32 additions of a row's sums;
// at most one per eight chunks.
static int seg_min(int chunks) { return (chunks + 63) / 64; }
static int seg_max(int chunks) { return std::max(seg_min(chunks), std::min(64, chunks / 8)); }
int f16_segments(int K) { return seg_min((K + BK - 1) / BK); }

double f16_eps(int K) {
    const int chunks = (K + BK - 1) / BK, steps = std::min(4, (K + 15) / 16);
    const double u23 = 1.1920928955078125e-07, u24 = 5.9604644775390625e-08;
    auto adds = [&](int n) { return (chunks + n - 1) / n + (n > 1 ? n : 0); };   // convex in n: largest at an end
    return 0.75 * 9.5367431640625e-07 + steps * u23 + 2 * steps * u23 * 9.765625e-04 * 1.001 +
           std::max(adds(seg_min(chunks)), adds(seg_max(chunks))) * u24;
}

typedef CUresult (*EncodeFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                             const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// Map over a row-major matrix (rows of `cols` elements, `ld` elements apart).
static bool make_map(void *out, CUtensorMapDataType type, int size, const void *base, int cols, int rows, long ld, int box_cols, int box_rows, CUtensorMapSwizzle sw) {
    static EncodeFn enc = nullptr;
    if (!enc) {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult qr;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qr) != cudaSuccess || !p) return false;
        enc = (EncodeFn)p;
    }
    const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)ld * size};
    const cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows}, es[2] = {1, 1};
    return enc((CUtensorMap *)out, type, 2, const_cast<void *>(base), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, sw,
               CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// The fp16 operand [K x N] of `src`; wmax: its largest magnitude (net.wmax, positive: the layer qualifies).
int umma_prepare_f16(nyb200_engine *e, const WeightSource &src, int K, int N, float wmax, UmmaLayer *out, Carve &c) {
    const int kpad = (K + BK - 1) / BK * BK;
    const size_t n_el = (size_t)N * kpad;
    __half *block = (__half *)c.take(2 * n_el * 2);
    if (!c.block) return NYB200_OK;
    out->f16 = block;
    out->K = K; out->N = N;
    int ex;
    frexpf(wmax, &ex);                       // wmax in [2^(ex-1), 2^ex)
    const float scale = ldexpf(1.f, std::max(-126, std::min(15 - ex, 126)));
    out->w_inv = 1.f / scale;
    k_split_weights_f16<<<(unsigned)((n_el + 255) / 256), 256, 0, e->stream>>>(src, K, N, kpad, scale, block);
    e->launches++;
    for (int i = 0; i < 2; ++i)
        if (!make_map(i ? out->tm16_lo : out->tm16_hi, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, block + i * n_el, kpad, N, kpad, BK, 64, CU_TENSOR_MAP_SWIZZLE_128B))
            return set_err(e, NYB200_ERR_INTERNAL, "cuTensorMapEncodeTiled failed for a contraction operand");
    return NYB200_OK;
}

// Tile width (256: CTA pairs) and number of K segments: the cheapest by SM cycles.  A chunk takes 6 tensor cycles per column
// and not less than the 900 its operand split does; a tile's start and its stores about 2500; a wave costs its slowest
// tile.  Segments only for contractions of 16 chunks and more that leave half of the SMs idle.
static void pick_tile(int M, int N, int chunks, int sms, bool fixed, int &bn, int &segs) {
    bn = 256; segs = seg_min(chunks);
    if (fixed) return;
    long best = -1;
    for (int b : {256, 128, 64}) {
        if (b == 256 && M <= BM) continue;
        if (b < 128 && b >= 2 * N && best >= 0) continue;
        const int cg = b == 256 ? 2 : 1, slots = sms / cg;
        const long tiles = (long)((M + cg * BM - 1) / (cg * BM)) * ((N + b - 1) / b);
        int sg = seg_min(chunks);
        if (chunks >= 16 && tiles * 2 * sg <= slots) sg = std::max(sg, std::min<int>(seg_max(chunks), (int)(slots / tiles)));
        const long cost = ((tiles * sg + slots - 1) / slots) * ((long)((chunks + sg - 1) / sg) * std::max(6 * std::min(b, (N + 15) & ~15), 900) + 2500);
        if (best < 0 || cost < best) { best = cost; bn = b; segs = sg; }
    }
}

int launch_umma_f16(nyb200_engine *e, const UmmaLayer &L, int M, const float *A, int lda, float *C, int ldc, int *err, const ConcFuse *cf) {
    const int sms = usable_sms(e);
    f16::Params P;
    P.A = A; P.lda = lda; P.M = M; P.N = L.N; P.K = L.K; P.chunks = (L.K + BK - 1) / BK;
    P.w_inv = L.w_inv; P.err = err;
    int bn, segs;
    pick_tile(M, L.N, P.chunks, sms, cf != nullptr, bn, segs);
    if (cf && segs > 1) return set_err(e, NYB200_ERR_INTERNAL, "fused concretisation of a segmented contraction");
    P.per_seg = (P.chunks + segs - 1) / segs;
    P.segs = (P.chunks + P.per_seg - 1) / P.per_seg;
    P.C = C; P.ldc = ldc; P.seg_stride = 0;
    const long total = (long)M * L.N;
    if (P.segs > 1) {
        NYB_WS(part, float *, e, "umma_segments", (size_t)P.segs * total * 4);
        P.C = part; P.ldc = L.N; P.seg_stride = total;
    }
    // A and C through TMA where a tensor map can describe them: base and row stride multiples of 16 bytes
    const CUtensorMap &th = *(const CUtensorMap *)L.tm16_hi, &tl = *(const CUtensorMap *)L.tm16_lo;
    alignas(64) CUtensorMap ta = th, tc = th;
    P.a_tma = (reinterpret_cast<uintptr_t>(A) & 15) == 0 && (lda & 3) == 0 && lda >= L.K;
    P.c_tma = P.segs == 1 && (reinterpret_cast<uintptr_t>(C) & 15) == 0 && (ldc & 3) == 0 && ldc >= L.N && !(cf && !cf->store);
    if ((P.a_tma && !make_map(&ta, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, A, L.K, M, lda, 32, BM, CU_TENSOR_MAP_SWIZZLE_128B)) ||
        (P.c_tma && !make_map(&tc, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, C, L.N, M, ldc, 32, 32, CU_TENSOR_MAP_SWIZZLE_128B)))
        return set_err(e, NYB200_ERR_INTERNAL, "cuTensorMapEncodeTiled failed for a contraction's rows");
    const int cg = bn == 256 ? 2 : 1;
    const long tiles = (long)((M + cg * BM - 1) / (cg * BM)) * ((L.N + bn - 1) / bn) * P.segs;
    const dim3 grid((unsigned)(std::min<long>(tiles, sms / cg) * cg));
    ConcFuse none;
    cudaError_t st = cudaSuccess;
#define NYB_F16(B, G)                                                                                                           \
    if (bn == B) {                                                                                                              \
        NYB_CUDA(e, cudaFuncSetAttribute(k_umma_f16<B, G>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));           \
        st = launch_pdl_cluster(k_umma_f16<B, G>, grid, dim3(f16::THREADS), G, SMEM_BYTES, e, th, tl, ta, tc, P, cf ? *cf : none); \
    }
    NYB_F16(256, 2) NYB_F16(128, 1) NYB_F16(64, 1)
#undef NYB_F16
    if (st != cudaSuccess) return set_err(e, NYB200_ERR_INTERNAL, "contraction kernel launch failed");
    e->launches++;
    if (P.segs > 1) {
        NYB_CUDA(e, launch_pdl(k_sum_segments, dim3((unsigned)((total + 255) / 256)), dim3(256), 0, e, total, L.N, P.segs, (const float *)P.C, C, (long)ldc));
        e->launches++;
    }
    return NYB200_OK;
}

}  // namespace nyb
