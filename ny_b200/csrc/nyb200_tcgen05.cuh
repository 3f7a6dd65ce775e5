// Inline-PTX building blocks shared by the tcgen05 kernels: bounded mbarrier waits, TMA tile loads, shared-memory
// operand and instruction descriptors for kind::tf32, MMA issue / commit, tensor-memory loads, TF32 rounding.
#pragma once

#include <cuda.h>
#include <stdint.h>

namespace nyb {
namespace umma {

constexpr unsigned WAIT_HINT_NS = 20000;                 // per probe: up to 20 us parked
constexpr long long WAIT_LIMIT_CYCLES = 4000000000LL;    // per wait: about two seconds of SM clock

__device__ __forceinline__ unsigned smem_u32(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(unsigned bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(unsigned bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(unsigned bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// Bounded wait: returns false when the limit expires.  Every probe carries a suspend-time hint, so a waiting warp is
// parked by the hardware until the phase completes (or the hint runs out) instead of competing for issue slots with
// the warps that do the work; the bound is on elapsed SM cycles (about two seconds), read only between probes.
__device__ __forceinline__ bool mbar_probe(unsigned bar, unsigned parity, unsigned hint_ns) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity), "r"(hint_ns)
        : "memory");
    return ok != 0;
}
// sleep_ns > 0: the caller is a role that runs ahead of the work (a producer, the MMA issuer waiting for operands);
// after a failed probe it sleeps that long, so that it does not take issue slots from the warps it is waiting for.
__device__ __forceinline__ bool mbar_wait(unsigned bar, unsigned parity, unsigned sleep_ns = 0) {
    if (mbar_probe(bar, parity, WAIT_HINT_NS)) return true;
    const long long t0 = clock64();
    for (;;) {
        if (sleep_ns) __nanosleep(sleep_ns);
        if (mbar_probe(bar, parity, WAIT_HINT_NS)) return true;
        if (clock64() - t0 > WAIT_LIMIT_CYCLES) return false;
    }
}

// The same without a suspend-time hint: the waiter is back within the hardware's own (short) time slice.
__device__ __forceinline__ bool mbar_wait_soon(unsigned bar, unsigned parity) {
    const long long t0 = clock64();
    for (;;) {
        unsigned ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
        if (ok) return true;
        if (clock64() - t0 > WAIT_LIMIT_CYCLES) return false;
    }
}

// The wait of a converged warp that issues products.  Every exit is a vote, so the warp stays converged in the compiler's eyes
// too and its loops' descriptors live in uniform registers, where tcgen05.mma wants them.  After a wait, or a look at a flag in
// shared memory, that lets lanes leave one by one, they are vector values that each product first moves over: 130 SM cycles a
// product where the tensor core takes 48 (128 x 64 x 16, operands in shared memory) to 64 (128 columns); from a single-lane
// branch 95 to 105, and 169 instead of 128 for 256 columns.
__device__ __forceinline__ bool mbar_wait_warp(unsigned bar, unsigned parity) {
    long long t0 = 0;
    for (;;) {
        unsigned ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
        if (__all_sync(0xffffffffu, ok)) return true;
        const long long now = clock64();
        if (t0 == 0) t0 = now;
        if (__any_sync(0xffffffffu, now - t0 > WAIT_LIMIT_CYCLES)) return false;
    }
}
// A flag in shared memory, read by a converged warp.
__device__ __forceinline__ bool flag_warp(const volatile int *flag) { return __any_sync(0xffffffffu, *flag); }

__device__ __forceinline__ void tma_load_2d(unsigned dst, const CUtensorMap *tm, int x, int y, unsigned bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(dst), "l"(tm), "r"(x), "r"(y), "r"(bar)
        : "memory");
}

// K-major, 128-byte swizzle shared-memory operand descriptor: start address >> 4 in bits [0,14),
// leading byte offset (unused for this layout) = 1 in [16,30), stride byte offset = 1024 B (8 rows of
// 128 B) >> 4 in [32,46), descriptor version 1 in [46,48), layout type 2 (128B swizzle) in [61,64).
__device__ __forceinline__ unsigned long long make_desc(unsigned smem_addr) {
    unsigned long long d = 0;
    d |= (unsigned long long)((smem_addr & 0x3FFFF) >> 4);
    d |= 1ull << 16;
    d |= (unsigned long long)(1024 >> 4) << 32;
    d |= 1ull << 46;
    d |= 2ull << 61;
    return d;
}

// Instruction descriptor: D fp32 (bits [4,6) = 1), A and B TF32 (format 2 at [7,10) and [10,13)),
// both K-major, N >> 3 at [17,23), M >> 4 at [24,29).
__device__ __forceinline__ unsigned make_idesc(int m, int n) {
    return (1u << 4) | (2u << 7) | (2u << 10) | ((unsigned)(n >> 3) << 17) | ((unsigned)(m >> 4) << 24);
}

__device__ __forceinline__ void mma_tf32(unsigned d_tmem, unsigned long long adesc, unsigned long long bdesc,
                                         unsigned idesc, unsigned accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void mma_commit(unsigned bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_ld32(unsigned taddr, unsigned (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}

// ---- fp16 operands (kind::f16, fp32 accumulation, K = 16 per instruction)
__device__ __forceinline__ void tma_load_4d(unsigned dst, const CUtensorMap *tm, int x, int y, int z, int w, unsigned bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];"
        ::"r"(dst), "l"(tm), "r"(x), "r"(y), "r"(z), "r"(w), "r"(bar)
        : "memory");
}
// K-major operand whose rows are `sw` bytes (32, 64 or 128: the swizzle span), eight-row groups `sbo` bytes apart.  The
// swizzle is a function of the shared-memory address, so a start address may lie any whole number of rows behind the
// (aligned) start of the pattern: a window over an image is the same tile read from another row.
__device__ __forceinline__ unsigned long long make_desc_sw(unsigned smem_addr, int sw, unsigned sbo) {
    const unsigned long long type = sw == 128 ? 2ull : sw == 64 ? 4ull : 6ull;
    return (unsigned long long)((smem_addr & 0x3FFFF) >> 4) | (1ull << 16) | ((unsigned long long)(sbo >> 4) << 32) | (1ull << 46) | (type << 61);
}
// D fp32, A and B fp16 (format 0), both K-major.
__device__ __forceinline__ unsigned make_idesc_f16(int m, int n) {
    return (1u << 4) | ((unsigned)(n >> 3) << 17) | ((unsigned)(m >> 4) << 24);
}
// A product of fp16 operands, issued by a whole converged warp with one elected lane doing it: with every lane in the loop the descriptors are
// warp-uniform values and stay in uniform registers, where the instruction wants them; from a single-lane branch every
// product costs some ninety cycles of moving them there, which is what a product of few columns takes.
__device__ __forceinline__ void mma_f16_elect(unsigned d_tmem, unsigned long long adesc, unsigned long long bdesc, unsigned idesc,
                                              unsigned accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "elect.sync _|q, 0xffffffff;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// KS products along K (each 32 bytes further in both operands) of one elected lane; the first one adds to what the accumulator
// holds or starts it.  One election and no descriptor arithmetic between them: the issuing warp shares its scheduler.
template <int KS>
__device__ __forceinline__ void mma_f16_group(unsigned d, unsigned long long a, unsigned long long b, unsigned idesc, unsigned accumulate) {
    if constexpr (KS == 4)
        asm volatile(
            "{\n\t.reg .pred p, q, t;\n\t.reg .b64 a1, a2, a3, b1, b2, b3;\n\t"
            "add.s64 a1, %1, 2;\n\tadd.s64 a2, %1, 4;\n\tadd.s64 a3, %1, 6;\n\tadd.s64 b1, %2, 2;\n\tadd.s64 b2, %2, 4;\n\tadd.s64 b3, %2, 6;\n\t"
            "setp.ne.b32 p, %4, 0;\n\tsetp.eq.b32 t, 0, 0;\n\t"
            "elect.sync _|q, 0xffffffff;\n\t"
            "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t"
            "@q tcgen05.mma.cta_group::1.kind::f16 [%0], a1, b1, %3, t;\n\t"
            "@q tcgen05.mma.cta_group::1.kind::f16 [%0], a2, b2, %3, t;\n\t"
            "@q tcgen05.mma.cta_group::1.kind::f16 [%0], a3, b3, %3, t;\n\t}"
            ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
    else if constexpr (KS == 2)
        asm volatile(
            "{\n\t.reg .pred p, q, t;\n\t.reg .b64 a1, b1;\n\t"
            "add.s64 a1, %1, 2;\n\tadd.s64 b1, %2, 2;\n\t"
            "setp.ne.b32 p, %4, 0;\n\tsetp.eq.b32 t, 0, 0;\n\t"
            "elect.sync _|q, 0xffffffff;\n\t"
            "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t"
            "@q tcgen05.mma.cta_group::1.kind::f16 [%0], a1, b1, %3, t;\n\t}"
            ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
    else mma_f16_elect(d, a, b, idesc, accumulate);
}
__device__ __forceinline__ void mma_commit_elect(unsigned bar) {
    asm volatile(
        "{\n\t.reg .pred q;\n\t"
        "elect.sync _|q, 0xffffffff;\n\t"
        "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_ld16(unsigned taddr, unsigned (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
          "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}

// Round an fp32 value to the nearest TF32 value (10 explicit mantissa bits), ties away from zero.
__device__ __forceinline__ float rn_tf32(float x) {
    // Half an ulp of the 10-bit mantissa added to the magnitude bits, then the 13 low bits cleared: the value
    // cvt.rna.tf32.f32 returns (a carry into the exponent is the correct rounding to the next binade or to
    // infinity; infinities and NaNs keep their class), in two full-rate integer instructions instead of one
    // conversion-pipe instruction.
    return __uint_as_float((__float_as_uint(x) + 0x1000u) & 0xFFFFE000u);
}


}  // namespace umma
}  // namespace nyb
