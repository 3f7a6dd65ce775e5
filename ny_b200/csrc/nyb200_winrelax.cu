// The ReLU step between two convolutions of a backward pass on the tensor path: coefficient rows that a window convolution
// left (or a fully connected layer) through the relaxation, straight into the operand pairs that the next window convolution
// reads (nyb200_convwin.cu).  Per coefficient it is relax_coeff; the row sums and charges are k_relax_dom's.
//
// What it replaces: the relaxation pass over the fp32 rows, the row maxima, the split (a transposition of channel planes into
// pixels through shared memory), and around an identity branch a copy of the rows and a pass that adds them: nine passes over
// memory for a residual block's layer, 2.1 ms for 4608 rows of 65536.  Here rows are read once, in the pixel-major order the
// convolution leaves them in, and written once, as pairs.
//
// What bounds it: instructions and the latency of the loads, at half of the copy rate (1152 rows of 65536: 187 us where the bytes
// take 92).  A batch of rows is on its way while the last one is worked on: 214 us without, and with four rows at a time and
// three blocks an SM; lanes over eight pixels and sixteen channels, half lines of the rows, 246.  256 domains of a residual
// network 45.3 -> 32.9 ms a call, 1024 of a classifier of two strided convolutions 2.76 -> 2.21.
//
// The scale of a row's pairs has to be known before its first coefficient is split.  The convolution reports the largest
// magnitude of every row; slopes lie in [0, 1], so behind the ReLU no coefficient is larger than that, one rounding step and
// the domain's largest split multiplier of the layer (RowBound).  A pair holds its 22 bits down to 2^-28 of the scale's reference,
// and what is lost below is charged against that reference.
#include <cuda_fp16.h>

#include "nyb200_internal.cuh"
#include "nyb200_relax.cuh"

namespace nyb {

namespace {

constexpr int kRows = 64;   // rows whose sums a block holds at a time
// Rows in flight together: nine specification rows are three whole batches.  Other numbers of rows, us a call, passes of their own /
// this: 1024 domains of the classifier 1 row 1364 / 1339, 2 1571 / 1438, 4 1978 / 1666, 5 2211 / 1766, 7 2616 / 1990, 8 2870 / 2088,
// 9 3107 / 2190; 64 of a residual network with two blocks 1 row 6983 / 4335, 3 5424 / 4782, 4 5913 / 5081, 7 7423 / 5813, 8 7855 / 6049,
// 9 8457 / 6271 (the window convolutions of both sides as they were with that form).
constexpr int kBatch = 3;

struct ImageArgs {
    int C, plane, Cp, R, S, vec;     // vec: rows are pixel-major, C channels a pixel; otherwise channel planes
    const float *A;
    long lda;
    const unsigned *row_max;         // [rows] largest magnitude of A's rows (bits)
    const float *beta_max;           // [D] largest multiplier of the layer's splits
    const float *J, *j_max;          // identity branch that joins: rows (pixel-major), their largest magnitudes; or null
    const float *zl, *zu;            // the joining variable's interval
    float *stash, *stash_max;        // rows kept for another identity branch (pixel-major), or null
    long lds, ldk;                   // row strides of J and stash
    long nps, q_ds;
    int off;
    const float4 *tab;
    const float *zabs, *q, *bias;
    float eps;
    __half *hi, *lo;                 // the pairs, or null: the rows go to `stash` alone
    float *row_inv;
    double *rb, *rpen;
};

__device__ __forceinline__ void pair_scale(float bound, float &s, float &inv) {   // as win_scale (nyb200_convwin.cu)
    const int e = (int)((__float_as_uint(bound) & 0x7fffffffu) >> 23);
    if (e == 0 || e == 255) { s = inv = 1.f; return; }
    const int k = min(max(14 - (e - 127), -126), 126);
    s = __uint_as_float((unsigned)(k + 127) << 23);
    inv = __uint_as_float((unsigned)(127 - k) << 23);
}

// Two fp32 operations per instruction.
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

// A thread's coefficients of a batch of rows, on their way from memory.
template <bool JOIN>
struct Batch3 { float4 a[kBatch], j[JOIN ? kBatch : 1]; };

template <bool JOIN>
__device__ __forceinline__ void load_batch(const ImageArgs &P, const float *a, const float *j, int n, bool live, Batch3<JOIN> &b) {
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
        b.a[u] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (JOIN) b.j[u] = b.a[u];
        if (live && u < n) {
            const float *src = a + u * P.lda;
            if (P.vec) b.a[u] = __ldcs((const float4 *)src);
            else b.a[u] = make_float4(src[0], src[P.plane], src[2 * P.plane], src[3 * P.plane]);
            if (JOIN) b.j[u] = __ldcs((const float4 *)(j + u * P.lds));
        }
    }
}

struct Columns { float4 t[4], zg, cj, zm, bias; };   // of a thread's pixel and four channels

// n rows, all lower or all upper ones, of this thread's pixel and four channels; the warp's sums to part.
template <bool UPPER, bool JOIN>
__device__ __forceinline__ void image_batch(const ImageArgs &P, const Batch3<JOIN> &in, int n, bool live, bool put, const Columns &c, const float *scale,
                                            float *keep, __half *hi, __half *lo, long half_row, double (*part)[2], int lane) {
    double sb[kBatch];
    float sp[kBatch];
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
        sb[u] = 0.0; sp[u] = 0.f;
        if (u >= n) continue;   // uniform in the warp
        float4 a = in.a[u];
        if (JOIN) {   // the branch joins: the exact residual of each rounded sum is charged (k_skip_coeff)
            auto add = [&](float &x, float y, float z) {
                const float s = x + y, bb = s - x, err = (x - (s - bb)) + (y - bb);
                sp[u] = __fmaf_ru(fabsf(err), z, sp[u]);
                x = s;
            };
            add(a.x, in.j[u].x, c.zm.x); add(a.y, in.j[u].y, c.zm.y); add(a.z, in.j[u].z, c.zm.z); add(a.w, in.j[u].w, c.zm.w);
        }
        float4 o;
        o.x = relax_prepared<UPPER, true>(a.x, c.t[0], c.zg.x, c.cj.x, c.bias.x, sb[u], sp[u]);
        o.y = relax_prepared<UPPER, true>(a.y, c.t[1], c.zg.y, c.cj.y, c.bias.y, sb[u], sp[u]);
        o.z = relax_prepared<UPPER, true>(a.z, c.t[2], c.zg.z, c.cj.z, c.bias.z, sb[u], sp[u]);
        o.w = relax_prepared<UPPER, true>(a.w, c.t[3], c.zg.w, c.cj.w, c.bias.w, sb[u], sp[u]);
        if (P.stash && live) __stcs((float4 *)(keep + u * P.ldk), o);
        if (put) {   // (channels past the last one: zeros)
            // the low part from the scaled value: the scale alone may lie within 2^11 of fp32's end (rows below 2^-102)
            const float s = scale[u];
            const float2 k2 = make_float2(2048.f, 2048.f), kn = make_float2(-2048.f, -2048.f);
            const float2 v0 = mul2(make_float2(o.x, o.y), make_float2(s, s)), v1 = mul2(make_float2(o.z, o.w), make_float2(s, s));
            const __half2 h0 = __floats2half2_rn(v0.x, v0.y), h1 = __floats2half2_rn(v1.x, v1.y);
            const float2 w0 = fma2(__half22float2(h0), kn, mul2(v0, k2)), w1 = fma2(__half22float2(h1), kn, mul2(v1, k2));   // exact
            const __half2 l0 = __floats2half2_rn(w0.x, w0.y), l1 = __floats2half2_rn(w1.x, w1.y);
            *(uint2 *)(hi + u * half_row) = make_uint2(*(const unsigned *)&h0, *(const unsigned *)&h1);
            *(uint2 *)(lo + u * half_row) = make_uint2(*(const unsigned *)&l0, *(const unsigned *)&l1);
        }
    }
    // the rows' sums reduced together: each step halves the rows a lane holds (as relax_dom_batch)
    const bool hi16 = lane & 16, hi8 = lane & 8;
    double b0 = (hi16 ? sb[2] : sb[0]) + __shfl_xor_sync(0xffffffffu, hi16 ? sb[0] : sb[2], 16);
    double b1 = (hi16 ? 0.0 : sb[1]) + __shfl_xor_sync(0xffffffffu, hi16 ? sb[1] : 0.0, 16);
    float p0 = __fadd_ru(hi16 ? sp[2] : sp[0], __shfl_xor_sync(0xffffffffu, hi16 ? sp[0] : sp[2], 16));
    float p1 = __fadd_ru(hi16 ? 0.f : sp[1], __shfl_xor_sync(0xffffffffu, hi16 ? sp[1] : 0.f, 16));
    b0 = (hi8 ? b1 : b0) + __shfl_xor_sync(0xffffffffu, hi8 ? b0 : b1, 8);
    p0 = __fadd_ru(hi8 ? p1 : p0, __shfl_xor_sync(0xffffffffu, hi8 ? p0 : p1, 8));
#pragma unroll
    for (int o2 = 4; o2 > 0; o2 >>= 1) {
        b0 += __shfl_xor_sync(0xffffffffu, b0, o2);
        p0 = __fadd_ru(p0, __shfl_xor_sync(0xffffffffu, p0, o2));
    }
    const int u = lane >> 3;
    if ((lane & 7) == 0 && u < n) { part[u][0] = b0; part[u][1] = (double)p0; }
}

// One block: 1024 / Cp pixels of a domain, all channels, all rows.  A warp owns four pixels and 32 channels (eight and sixteen
// where there are no more), a lane one pixel and four channels, whose tables stay in registers for the domain's rows: 128-byte
// pieces of the rows, 64-byte ones of the tables.
template <bool JOIN>
__global__ void __launch_bounds__(256, 2)
k_relax_image(const __grid_constant__ ImageArgs P) {
    __shared__ double s_part[8][kRows][2];
    __shared__ float s_scale[kRows], s_bound[kRows], s_q[8], s_z[8];
    pdl_trigger();
    pdl_wait();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int quads = P.Cp >= 32 ? 8 : 4, groups = P.Cp / (4 * quads);   // channel quads of a warp, warps of a pixel
    const int d = blockIdx.y, px = (int)blockIdx.x * (1024 / P.Cp) + (warp / groups) * (32 / quads) + lane / quads, c0 = ((warp % groups) * quads + lane % quads) * 4;
    const bool put = P.hi && px < P.plane, live = px < P.plane && c0 < P.C;
    const long m0 = (long)d * P.R, in_row = (long)px * P.C + c0;
    const float *a_at = P.A + m0 * P.lda + (P.vec ? in_row : (long)c0 * P.plane + px), *j_at = JOIN ? P.J + m0 * P.lds + in_row : nullptr;
    auto batch_of = [&](int r) { return min(min(kBatch, (r < P.S ? P.S : P.R) - r), kRows - r % kRows); };   // lower rows, then upper ones
    Batch3<JOIN> ahead;
    load_batch<JOIN>(P, a_at, j_at, batch_of(0), live, ahead);
    Columns c;
    c.zg = c.cj = c.zm = c.bias = make_float4(0.f, 0.f, 0.f, 0.f);
    float qs = 0.f, zs = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        c.t[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (!live) continue;
        const long j = (long)(c0 + i) * P.plane + px, at = (long)d * P.nps + P.off + j;
        c.t[i] = P.tab[at];
        const float za = P.zabs[at], qv = P.q[(long)d * P.q_ds + P.off + j], bk = P.bias ? P.bias[j] : 0.f;
        (&c.bias.x)[i] = bk;
        qs = __fadd_ru(qs, qv);
        zs = __fadd_ru(zs, za);
        (&c.cj.x)[i] = __fmaf_ru(9.1e-13f, __fadd_ru(za, fabsf(bk)), __fmul_ru(P.eps, qv));
        (&c.zg.x)[i] = (c.t[i].y == 1.f && c.t[i].z == 0.f) ? 0.f : za;   // see relax_coeff
        if (JOIN) (&c.zm.x)[i] = fmaxf(fabsf(P.zl[at]), fabsf(P.zu[at]));
    }
    for (int o = 16; o > 0; o >>= 1) {
        qs = __fadd_ru(qs, __shfl_xor_sync(0xffffffffu, qs, o));
        zs = __fadd_ru(zs, __shfl_xor_sync(0xffffffffu, zs, o));
    }
    if (lane == 0) { s_q[warp] = qs; s_z[warp] = zs; }
    const long half_row = (long)P.plane * P.Cp * (P.Cp <= 32 ? 2 : 1), in_pair = m0 * half_row + (long)px * P.Cp * (P.Cp <= 32 ? 2 : 1) + c0;
    float *keep = P.stash + m0 * P.ldk + in_row;
    __half *hi = P.hi + in_pair, *lo = P.Cp <= 32 ? hi + P.Cp : P.lo + in_pair;
    for (int first = 0; first < P.R; first += kRows) {
        const int end = min(P.R, first + kRows);
        if (P.hi && threadIdx.x < end - first) {
            const long m = m0 + first + threadIdx.x;
            float b = __uint_as_float(P.row_max[m]);
            if (JOIN) b = __fadd_ru(b, P.j_max[m]);
            b = __fmaf_ru(b, 1.000001f, __fadd_ru(P.beta_max[d], 1e-44f));
            float s, inv;
            pair_scale(b, s, inv);
            s_scale[threadIdx.x] = s; s_bound[threadIdx.x] = b;
            if (blockIdx.x == 0) {
                P.row_inv[m] = inv;
                if (P.stash_max) P.stash_max[m] = b;
            }
        }
        __syncthreads();
        for (int r = first; r < end; ) {
            const int n = batch_of(r), next = r + n;
            const Batch3<JOIN> now = ahead;
            a_at += n * P.lda;
            if (JOIN) j_at += n * P.lds;
            if (next < P.R) load_batch<JOIN>(P, a_at, j_at, batch_of(next), live, ahead);   // while this batch is worked on
            if (r < P.S) image_batch<false, JOIN>(P, now, n, live, put, c, s_scale + (r - first), keep, hi, lo, half_row, s_part[warp] + (r - first), lane);
            else image_batch<true, JOIN>(P, now, n, live, put, c, s_scale + (r - first), keep, hi, lo, half_row, s_part[warp] + (r - first), lane);
            keep += n * P.ldk;
            hi += n * half_row; lo += n * half_row;
            r = next;
        }
        __syncthreads();
        if (threadIdx.x < end - first) {
            const long m = m0 + first + threadIdx.x;
            double b = 0.0, p = 0.0, qq = 0.0, zz = 0.0;
            for (int w = 0; w < 8; ++w) { b += s_part[w][threadIdx.x][0]; p += s_part[w][threadIdx.x][1]; qq += (double)s_q[w]; zz += (double)s_z[w]; }
            atomicAdd(&P.rb[m], b);
            // 1.000002: the fp32 sums' roundings (k_relax_dom); then the exponent-range share of the pairs (k_split_image)
            atomicAdd(&P.rpen[m], p * 1.000002 + kUnderflow * zz + (P.hi ? (3.5527137e-15 * (double)s_bound[threadIdx.x] + 1e-37) * qq : 0.0));
        }
        __syncthreads();
    }
}

}  // namespace

// Coefficient rows behind layer `lin`'s ReLU (C channels a pixel, padded to Cp in the operand) as the operand of its window
// convolution, or with hi null as pixel-major rows of their own, keep->rows, one behind the other.
int launch_relax_image(nyb200_engine *e, const Net &net, int lin, const BatchPtrs &p, int D, int R, int S, const float *A, bool pixel_major, const unsigned *row_max,
                       long q_ds, double eps, const ImageBranch *join, const ImageBranch *keep, void *hi, void *lo, float *row_inv) {
    const NetView &nv = net.v;
    const ConvGeom &g = net.geom[lin];
    ImageArgs a;
    memset(&a, 0, sizeof(a));
    a.C = g.oc; a.plane = g.oh * g.ow; a.Cp = hi ? net.win_bwd[lin].in_cp : g.oc <= 16 ? 16 : g.oc <= 32 ? 32 : g.oc <= 64 ? 64 : 128;
    a.R = R; a.S = S; a.vec = pixel_major ? 1 : 0;
    a.A = A; a.lda = p.lda; a.row_max = row_max; a.beta_max = p.beta_max + (size_t)lin * D;
    if (join) { a.J = join->rows; a.j_max = join->max; a.zl = p.zl; a.zu = p.zu; }
    if (keep) { a.stash = keep->rows; a.stash_max = keep->max; }
    a.lds = p.lda; a.ldk = hi ? (long)p.lda : (long)a.plane * a.C;
    a.nps = nv.nps; a.q_ds = q_ds; a.off = nv.pre_off[lin];
    a.tab = p.tab; a.zabs = p.zabs; a.q = p.q; a.bias = nv.b[lin];
    a.eps = (float)(eps * 1.0000002);
    a.hi = (__half *)hi; a.lo = (__half *)lo; a.row_inv = row_inv; a.rb = p.rb; a.rpen = p.rpen;
    const int per = 1024 / a.Cp;
    const dim3 grid((unsigned)((a.plane + per - 1) / per), (unsigned)D);
    NYB_CUDA(e, join ? launch_pdl(k_relax_image<true>, grid, dim3(256), 0, e, a) : launch_pdl(k_relax_image<false>, grid, dim3(256), 0, e, a));
    e->launches++;
    return NYB200_OK;
}

}  // namespace nyb
