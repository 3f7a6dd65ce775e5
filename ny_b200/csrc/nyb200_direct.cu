// Direct binary64 evaluation of fully connected networks: a whole backward pass in ONE kernel, a whole interval pass in
// another.  Plain CROWN with CROWN-IBP intermediate bounds (the pipeline of nyb200_crown.cu, two launches per layer), the
// beta-CROWN bound of small batches, and the binary64 re-evaluation of flagged domains run on it.  Rows of a backward
// pass never mix, so a warp takes eight rows from the layer they start at down to the input box: contraction, relaxation,
// bias and penalty sums, concretisation.  The coefficients stay in shared memory in binary64, the products run on the
// binary64 tensor instruction (mma.sync m8n8k4.f64, round to nearest per step: the gamma_{K+2} model of k_gemm_f64
// covers any order of its additions) and the row sums stay in registers until the end.
//
// Why: launched layer by layer a 5 -> 6x50 -> 5 network takes 251 launches of 2-10 us for one box, and twice the work,
// because nearly every box of that size is flagged by the 3xTF32 pass and evaluated again in binary64; the arithmetic of
// one box is 5.5 MFLOP.  One box 1.59 -> 0.2 ms.  Many small boxes are bound by the instructions around the products, so
// the per-coefficient step reads one 48-byte table entry and does most of its bookkeeping in fp32.
//
// Rounding.  Coefficients are rounded as the layer-by-layer form rounds them (binary64 product sums cast to fp32, slope
// products stepped one ulp outward), so both forms return the same bounds; the charges are its charges, the small ones
// accumulated in fp32 rounded upwards.  The binary64 sums of the bias terms err by at most 2^-40 of their magnitudes
// (fewer than 2^13 additions per partial sum), and those magnitudes are bounded by |nw| |bias| and |a * intercept| <=
// |nw| max|z| (1 + 2^-21) (an intercept only applies on the upper line, where intercept / slope = -l up to rounding and
// the step moves nw away from zero), which joins the contraction's charge: |nw| * cj with
//   cj = eps64(K) q + 2^-39 (max|z| + |bias|),   q = |W| max|z'| of the contraction that follows.
#include <cooperative_groups.h>
#include <math.h>
#include <string.h>

#include "nyb200_internal.cuh"
#include "nyb200_relax.cuh"

namespace nyb {

namespace {

constexpr size_t kPassMaxSmem = 220 * 1024;
constexpr int kRing = 6;                 // groups of weights in flight per warp (k_direct_pass)
constexpr int kDirectMaxNeurons = 16384; // split codes and multipliers of a domain in shared memory
constexpr int kSweepMaxWidth = 3072;     // two buffers of two binary64 vectors of that width fit in shared memory

struct PackedNet {
    NetView nv;
    const float4 *w[kMaxLinear];   // fragment order, see k_pack_fragments
};

// Per (box, neuron): what a pass reads.  zg: magnitude the gap of the outward step is charged against (zero where the
// pre-activation cannot be negative: the step alone is sound); zhi / zlo: the post-activation interval, a hair outside
// and inside, against which the error of a cast is charged or, where it helps, credited.  sbeta: signed split multiplier.
// lsu: the upper rows' own lower slope (dual alpha), equal to ls otherwise.
struct __align__(16) PassEntry { float ls, us, zg, zhi; float zlo, sbeta; double cj; float ui, lsu; double bias; };

__device__ __forceinline__ float step_up(float x) {
    unsigned b = __float_as_uint(x), mag = b & 0x7fffffffu;
    if (mag >= 0x7f800000u) return x;
    if (mag == 0) return __uint_as_float(1u);
    return (b & 0x80000000u) ? __uint_as_float(b - 1) : __uint_as_float(b + 1);
}

// Brings a line into L1: a load whose result nothing waits for (prefetch.global.L1 left the lines in L2: a table entry was
// another 700 cycles away, for each of a warp's tiles in turn).
__device__ __forceinline__ void touch(const void *p) {
    unsigned v;
    asm volatile("ld.global.ca.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    (void)v;
}

__device__ __forceinline__ double eps64(int K) { return (double)(K + 2) * 1.1102230246251565e-16 * 1.000001; }

// W [K x N] row-major -> float4 groups [n-tile][k-group of 16][lane]: component c of lane l is
// W[16 g + 4 c + l % 4][8 t + l / 4], the B operand of the c-th m8n8k4 step of the group; zero outside the matrix.
__global__ void k_pack_fragments(const float *__restrict__ W, int K, int N, int kg, int nt, float4 *__restrict__ out) {
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long)nt * kg * 32) return;
    const int lane = (int)(t & 31), g = (int)((t >> 5) % kg), tile = (int)((t >> 5) / kg);
    const int n = tile * 8 + (lane >> 2);
    float v[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const int k = g * 16 + c * 4 + (lane & 3);
        v[c] = (k < K && n < N) ? W[(long)k * N + n] : 0.f;
    }
    out[t] = make_float4(v[0], v[1], v[2], v[3]);
}

__device__ __forceinline__ void dmma(double &c0, double &c1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(c0), "+d"(c1) : "d"(a), "d"(b));
}

// Interval image of outputs [o0, o1) of one layer for the CTA's box: finish(o, lo, hi, q, early(o)) is called once per
// output by one lane, with lo = W+ zl + W- zu, hi = W+ zu + W- zl, q = |W| max|z| in binary64 (the bounds' arithmetic is
// k_ibp_linear's); early(o) runs before the sums, so that what finish reads from memory is on its way meanwhile.
// The box comes in shared memory, already in binary64 (converting it for every output would cost three times the
// multiply-adds): behind a ReLU as centre and radius, which needs no selection by the weight's sign
// (lo, hi = W c -+ |W| r, q = |W| c + |W| r), in front as the two ends.  Eight lanes share an output and take OPT outputs
// at a time, so that a value is read once for OPT weights.
template <int OPT, class Early, class Finish>
__device__ __forceinline__ void interval_sweep(const float *__restrict__ W, int n_in, int o0, int o1, const double *za, const double *zb,
                                               bool centred, Early early, Finish finish) {
    const int sub = threadIdx.x & 7, grp = threadIdx.x >> 3, ngrp = blockDim.x >> 3;
    const bool vec = (n_in & 3) == 0;
    for (int base = o0; base < o1; base += ngrp * OPT) {   // every lane takes part in the shuffles
        double s0[OPT], s1[OPT], s2[OPT];
        const float *w[OPT];
#pragma unroll
        for (int u = 0; u < OPT; ++u) {
            s0[u] = s1[u] = s2[u] = 0.0;
            const int o = base + grp + u * ngrp;
            w[u] = W + (long)(o < o1 ? o : o1 - 1) * n_in;
        }
        const int mine = base + grp + sub * ngrp;   // OPT <= 8: lane u of the group closes output u
        auto held = early(sub < OPT && mine < o1 ? mine : o1 - 1);
        auto mac = [&](int u, float wf, double a, double b) {
            const double wv = wf;
            if (centred) {
                s0[u] = fma(wv, a, s0[u]);
                s1[u] = fma(fabs(wv), b, s1[u]);
                s2[u] = fma(fabs(wv), a, s2[u]);
            } else {
                const bool pos = wf > 0.f;
                s0[u] = fma(wv, pos ? a : b, s0[u]);
                s1[u] = fma(wv, pos ? b : a, s1[u]);
                s2[u] = fma(fabs(wv), fmax(fabs(a), fabs(b)), s2[u]);
            }
        };
        if (vec) {
#pragma unroll 4
            for (int i = sub * 4; i < n_in; i += 32) {
                const double2 a0 = *(const double2 *)(za + i), a1 = *(const double2 *)(za + i + 2);
                const double2 b0 = *(const double2 *)(zb + i), b1 = *(const double2 *)(zb + i + 2);
#pragma unroll
                for (int u = 0; u < OPT; ++u) {
                    const float4 wv = __ldg((const float4 *)(w[u] + i));
                    mac(u, wv.x, a0.x, b0.x); mac(u, wv.y, a0.y, b0.y); mac(u, wv.z, a1.x, b1.x); mac(u, wv.w, a1.y, b1.y);
                }
            }
        } else {
#pragma unroll 4
            for (int i = sub; i < n_in; i += 8) {
                const double a = za[i], b = zb[i];
#pragma unroll
                for (int u = 0; u < OPT; ++u) mac(u, __ldg(w[u] + i), a, b);
            }
        }
#pragma unroll
        for (int u = 0; u < OPT; ++u) {
#pragma unroll
            for (int s = 4; s > 0; s >>= 1) {
                s0[u] += __shfl_xor_sync(0xffffffffu, s0[u], s);
                s1[u] += __shfl_xor_sync(0xffffffffu, s1[u], s);
                s2[u] += __shfl_xor_sync(0xffffffffu, s2[u], s);
            }
        }
        double lo = s0[0], hi = s1[0], qq = s2[0];
#pragma unroll
        for (int u = 1; u < OPT; ++u)
            if (sub == u) { lo = s0[u]; hi = s1[u]; qq = s2[u]; }
        if (sub < OPT && mine < o1) {
            if (centred) finish(mine, lo - hi, lo + hi, qq + hi, held);
            else finish(mine, lo, hi, qq, held);
        }
    }
}

// A post-activation interval [pl, pu], pl >= 0, as centre and radius.
__device__ __forceinline__ void centre(float pl, float pu, double &c, double &r) {
    c = 0.5 * ((double)pl + (double)pu);
    r = 0.5 * ((double)pu - (double)pl);
}

// Rounding rate of the interval sums: n products and their additions, the centre, the radius and the closing additions.
__device__ __forceinline__ double gam_sweep(int n) { return eps64(n + 4); }

// Weights that fit in L1 on their way there ahead of their use; a layer's reads are a chain of L2 latencies otherwise.
__device__ __forceinline__ void warm_weights(const float *W, int n) {
    if (n > 16384) return;
    for (int i = threadIdx.x * 32; i < n; i += blockDim.x * 32) touch(W + i);
}

struct NoEarly { __device__ int operator()(int) const { return 0; } };

// Outward rounding of an interval product and its bias: slack for the binary64 sums, directed casts.
__device__ __forceinline__ void outward(double lo, double hi, double qq, double gam, const float *bias, int o, float &l, float &u, float &q) {
    const double bv = bias ? (double)bias[o] : 0.0, slack = gam * (qq + fabs(bv));
    l = __double2float_rd(lo + bv - slack); u = __double2float_ru(hi + bv + slack);
    if (isnan(l) || isnan(u)) { l = -INFINITY; u = INFINITY; }
    q = __double2float_ru(qq * (1.0 + gam));
}

// Interval pass of the whole network, one CTA per box; code: the box's split codes (clamps), or null.
__global__ void __launch_bounds__(512)
k_crown_ibp(NetView nv, int zdim, const float *__restrict__ in_lo, const float *__restrict__ in_hi, long box_ds, float *raw_lo, float *raw_hi,
            float *__restrict__ q, float *__restrict__ zl, float *__restrict__ zu, float *__restrict__ ibp_lo, float *__restrict__ ibp_hi,
            const signed char *__restrict__ code, int *__restrict__ flags) {
    pdl_trigger();
    warm_weights(nv.W[0], nv.dims[0] * nv.dims[1]);
    pdl_wait();
    extern __shared__ double s_z[];   // two buffers of zl, zu
    const int d = blockIdx.x;
    const long row = (long)d * nv.nps;
    int bad = 0;
    double *zc = s_z, *zn = s_z + 2 * zdim;
    for (int i = threadIdx.x; i < nv.dims[0]; i += blockDim.x) { zc[i] = in_lo[(long)d * box_ds + i]; zc[zdim + i] = in_hi[(long)d * box_ds + i]; }
    __syncthreads();
    for (int k = 0; k < nv.L; ++k) {
        const long o = row + nv.pre_off[k];
        const double gam = gam_sweep(nv.dims[k]);
        if (k + 1 < nv.L) warm_weights(nv.W[k + 1], nv.dims[k + 1] * nv.dims[k + 2]);
        interval_sweep<2>(nv.W[k], nv.dims[k], 0, nv.dims[k + 1], zc, zc + zdim, k > 0, NoEarly(), [&](int j, double lo, double hi, double qq, int) {
            float l, u, qf;
            outward(lo, hi, qq, gam, nv.b[k], j, l, u, qf);
            if (k == 0) { raw_lo[o + j] = l; raw_hi[o + j] = u; q[o + j] = qf; }   // (k_crown_layer has its own image of the others)
            const int sc = (code && k < nv.L - 1) ? code[o + j] : 0;
            if (sc > 0) l = fmaxf(l, 0.f);
            else if (sc < 0) u = fminf(u, 0.f);
            if (sc != 0) { if (l > u) bad |= kFlagInfeasible; }
            else if (k < nv.L - 1 && (isinf(l) || isinf(u))) bad |= kFlagDegraded;   // a hidden bound overflowed
            ibp_lo[o + j] = l; ibp_hi[o + j] = u;
            const float pl = sc < 0 ? 0.f : fmaxf(l, 0.f), pu = sc < 0 ? 0.f : fmaxf(u, 0.f);
            zl[o + j] = pl; zu[o + j] = pu;
            if (k < nv.L - 1) centre(pl, pu, zn[j], zn[zdim + j]);
        });
        __syncthreads();
        double *sw = zc; zc = zn; zn = sw;
    }
    if (bad) atomicOr(&flags[d], bad);   // cleared before this kernel; the split scatter may have set its own bit
}

// One coefficient of a row through a ReLU's relaxation (the step of k_relax): the coefficient behind it, with the
// intercept's, the bias's and the charge's sums.
__device__ __forceinline__ double relax_step(float a, bool upper, const float4 &f, float sbeta, double cj, const float4 &ib, double &rb,
                                             double &rp, float &gp) {
    const bool pos = a > 0.f;
    const float slope = (pos != upper) ? (upper ? ib.y : f.x) : f.y;
    const float prod = __fmul_rn(a, slope);
    const int pb = __float_as_int(prod), dir = upper ? 1 : -1;
    // one ulp outward on the bit pattern; an underflowed product steps to the smallest denormal, an exact zero stays
    int nb = (pb << 1) ? pb + dir + 2 * dir * (pb >> 31) : (upper ? 1 : (int)0x80000001u);
    if (a == 0.f || slope == 0.f) nb = 0;
    if (a != a) nb = 0x7fc00000;
    float nw = __int_as_float(nb);
    gp = __fmaf_ru(fabsf(fmaf(a, slope, -nw)), f.z, gp);
    if (pos == upper) rb = fma((double)a, (double)ib.x, rb);
    nw = upper ? nw + sbeta : nw - sbeta;   // signed beta (zero for unsplit neurons), relu_backward.rs:156-175
    const double nwd = nw;
    rb = fma(nwd, __hiloint2double(__float_as_int(ib.w), __float_as_int(ib.z)), rb);
    rp = fma(fabs(nwd), cj, rp);
    return nwd;
}

// A contraction's result: rounded to fp32, the cast's exact error charged against the variable's interval [zlo, zhi],
// zlo >= 0 (the signed charge of k_gemm_f64: an error that helps the row's side takes the smaller end off again).
__device__ __forceinline__ float cast_coeff(double v, bool upper, const float4 &f, float zlo, float &gp) {
    const float c = (float)v;
    const float e = (float)(v - (double)c);
    const bool hurts = (e > 0.f) == upper;
    gp = __fmaf_ru(hurts ? fabsf(e) : -fabsf(e), hurts ? f.w : zlo, gp);
    return c;
}

// One partial (or the final) pass: rows = 2 n_rows per box, lower ones first.  CTA = MT groups of eight rows x NW warps
// that share a group's columns.  seed [n_rows x dims[top]]: for a layer that feeds a ReLU its weights (the identity times
// W_top is exact), and the pass goes on with ReLU top-1; for the specification rows (spec) they sit at the network's
// output, top = L, where the table holds the identity.  a_out, ckpt (optional): the coefficients on the input box and, one
// block of rows per ReLU, those that enter it.  idx: the boxes' places in the per-box arrays, or null.  NT: column tiles of eight per warp and sweep.
// C > 1: a cluster of C CTAs shares a group's columns (the row sums meet at the end, the coefficients are written to every
// CTA's shared memory).  RING: the weights run ahead through a ring of kRing groups in shared memory, one per warp, every
// lane fetching what it will read itself (cp.async, no barriers): across layers and epilogues, because they depend on
// nothing.  A wide network's layer does not stay in L1, and with one group in flight the L2 latency was three quarters
// of the pass (37 domains of 784 -> 8x256 -> 10: 163 us); small networks' weights do stay, and need no ring.
template <int NT, bool RING>
__global__ void __launch_bounds__(256, RING ? 1 : NT >= 6 ? 2 : 3)
k_direct_pass(const __grid_constant__ PackedNet pn, int top, int boxes, const int *__restrict__ idx, int n_rows, int MT, int NW, int pitch, int bufs,
             const float *__restrict__ seed, const float *__restrict__ seed_bias, const float *__restrict__ in_lo,
             const float *__restrict__ in_hi, long box_ds, const PassEntry *__restrict__ ptab, float *__restrict__ out_lo,
             float *__restrict__ out_hi, float *__restrict__ a_out, int lda, float *__restrict__ ckpt, long ckpt_stride) {
    extern __shared__ double s_coef[];
    __shared__ double s_red[64][4];
    __shared__ int s_bad[64];
    constexpr int KA = NT == 1 ? 4 : NT == 2 ? 2 : 1;
    cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
    const int C = (int)cl.num_blocks(), rank = (int)cl.block_rank();
    const NetView &nv = pn.nv;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, lr = lane >> 2, lq = lane & 3;
    const int nw1 = NW / C;   // this CTA's share of the NW warps of a group
    const int mi = warp / nw1, ni = rank * nw1 + warp - mi * nw1;
    float4 *ring = (float4 *)(s_coef + bufs * MT * 8 * pitch) + warp * (kRing * NT * 32) + lane;
    // Next group to fetch.  Where it lies is worked out once a layer: looking the layer up for every group, in parameters
    // indexed by it, took longer than the group's products.
    struct { int lay, nb, g, slot, kg, nt; const float4 *src; } ahead = {top, 0, 0, 0, 0, 0, nullptr};
    auto next_layer = [&]() {
        if (--ahead.lay < 0) return;
        ahead.nb = 0;
        ahead.kg = (nv.dims[ahead.lay + 1] + 15) >> 4; ahead.nt = (nv.dims[ahead.lay] + 7) >> 3;
        ahead.src = pn.w[ahead.lay] + (long)ni * ahead.kg * 32 + lane;
    };
    if (RING) next_layer();
    auto fetch_group = [&]() {
        if (!RING) return;
        if (ahead.lay >= 0) {
            const unsigned dst = (unsigned)__cvta_generic_to_shared(ring + ahead.slot * (NT * 32));
#pragma unroll
            for (int t = 0; t < NT; ++t)
                if (ahead.nb + ni + t * NW < ahead.nt)
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + t * 512), "l"(ahead.src + (long)t * NW * ahead.kg * 32) : "memory");
            ahead.slot = ahead.slot + 1 == kRing ? 0 : ahead.slot + 1;
            ahead.src += 32;
            if (++ahead.g == ahead.kg) {
                ahead.g = 0;
                ahead.nb += NW * NT;
                if (ahead.nb >= ahead.nt) next_layer();
                else ahead.src += (long)(NW * NT - 1) * ahead.kg * 32;   // (from the end of this tile's groups)
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    pdl_trigger();
    if (RING) {   // the packed weights were complete before the kernels of this call began
#pragma unroll 1
        for (int i = 0; i < kRing - 1; ++i) fetch_group();
    }
    // rows of all boxes one behind the other: a group of eight may span two boxes
    const int gr = ((int)(blockIdx.x / C) * MT + mi) * 8 + lr;
    const bool live = gr < boxes * 2 * n_rows;
    const int box = live ? gr / (2 * n_rows) : 0, r = live ? gr - box * 2 * n_rows : 0;
    const bool upper = r >= n_rows;
    const int rr = upper ? r - n_rows : r;
    if (NW > 1)   // a small launch: the rows it starts from (weights, or uploaded before the call's first kernel) into L1
        for (int j = lq * 32; j < nv.dims[top]; j += 128) touch(seed + (long)rr * nv.dims[top] + j);
    pdl_wait();
    const int d = idx ? idx[box] : box;
    const PassEntry *dom = ptab + (long)d * nv.nps;
    double *cur = s_coef + (mi * 8 + lr) * pitch, *nxt = cur + (bufs > 1 ? MT * 8 * pitch : 0);
    int slot = 0;
    const bool alone = NW == 1;
    auto meet_rows = [&]() { if (alone) __syncwarp(); else if (C > 1) cl.sync(); else __syncthreads(); };
    auto put2 = [&](double *at, double2 v) {
        if (C == 1) { *(double2 *)at = v; return; }
        for (int p = 0; p < C; ++p) *(double2 *)cl.map_shared_rank(at, p) = v;
    };
    double rb = 0.0, rp = 0.0, cs = 0.0, ca = 0.0;
    float gp = 0.f;   // fp32 share of the penalty: gaps and casts
    bool bad = false;
    {
        const int n = nv.dims[top], np16 = (n + 15) & ~15;
        const bool spec = top == nv.L;   // rows at the network's output: no ReLU in front of the first contraction
        const PassEntry *t = dom + nv.pre_off[top - 1];
        // every CTA of a cluster holds all columns; the sums count a column once
        for (int j = (ni - rank * nw1) * 4 + lq; j < np16; j += 4 * nw1) {
            double v = 0.0, xb = 0.0, xp = 0.0;
            float xg = 0.f;
            if (live && j < n) {
                const float a = seed[(long)rr * n + j];
                if (spec) { v = a; xb = v * t[j].bias; xp = fabs(v) * t[j].cj; }
                else v = relax_step(a, upper, *(const float4 *)&t[j].ls, t[j].sbeta, t[j].cj, *(const float4 *)&t[j].ui, xb, xp, xg);
                if (rank == 0) { rb += xb; rp += xp; gp = __fadd_ru(gp, xg); }
            }
            cur[j] = v;
        }
        if (live && seed_bias && ni == 0 && lq == 0) { const double c = seed_bias[rr]; rb += c; rp += 1.8189894035458565e-12 * fabs(c); }
    }
    meet_rows();
    for (int lay = top - 1; lay >= 0; --lay) {
        const int K = nv.dims[lay + 1], N = nv.dims[lay], kg = (K + 15) >> 4, nt = (N + 7) >> 3;
        const int tail = (K - (kg - 1) * 16 + 3) >> 2;   // m8n8k4 steps of the last group
        const float4 *__restrict__ w = pn.w[lay] + lane;
        const PassEntry *t4 = lay > 0 ? dom + nv.pre_off[lay - 1] : nullptr;
        const float *xl = in_lo + (long)d * box_ds, *xu = in_hi + (long)d * box_ds;
        for (int nb = 0; nb < nt; nb += NW * NT) {
            // a narrow warp's products would be one dependent chain: it is cut into KA, added at the end
            double acc[KA][NT][2];
#pragma unroll
            for (int c = 0; c < KA; ++c)
#pragma unroll
                for (int t = 0; t < NT; ++t) acc[c][t][0] = acc[c][t][1] = 0.0;
            const double *arow = cur + lq;
            if (lay > 0) {   // the epilogue's table entries into L1 while the products run
#pragma unroll
                for (int t = 0; t < NT; ++t) {
                    const int j = (nb + ni + t * NW) * 8;
#pragma unroll
                    for (int i = 0; i < 3; ++i) {   // eight entries: twelve sectors, shared by the row's four lanes
                        const char *at = (const char *)(t4 + j) + (lq + 4 * i) * 32;
                        if (at < (const char *)(t4 + N)) touch(at);
                    }
                }
            }
            const int have = (nt - nb - ni + NW - 1) >> (31 - __clz(NW));   // live tiles of this warp in this sweep (NW: a power of two)
            const float4 *wt = w + (long)(nb + ni) * kg * 32;
            const long ws = (long)NW * kg * 32;
            if (RING) {
                for (int g = 0; g < kg; ++g) {
                    asm volatile("cp.async.wait_group %0;" ::"n"(kRing - 2) : "memory");
                    const float4 *mine = ring + slot * (NT * 32);
                    slot = slot + 1 == kRing ? 0 : slot + 1;
                    const double a0 = arow[g * 16], a1 = arow[g * 16 + 4], a2 = arow[g * 16 + 8], a3 = arow[g * 16 + 12];
                    if (have >= NT) {
                        float4 b[NT];
#pragma unroll
                        for (int t = 0; t < NT; ++t) b[t] = mine[t * 32];
                        fetch_group();
#pragma unroll
                        for (int t = 0; t < NT; ++t) dmma(acc[0 % KA][t][0], acc[0 % KA][t][1], a0, (double)b[t].x);
#pragma unroll
                        for (int t = 0; t < NT; ++t) dmma(acc[1 % KA][t][0], acc[1 % KA][t][1], a1, (double)b[t].y);
#pragma unroll
                        for (int t = 0; t < NT; ++t) dmma(acc[2 % KA][t][0], acc[2 % KA][t][1], a2, (double)b[t].z);
#pragma unroll
                        for (int t = 0; t < NT; ++t) dmma(acc[3 % KA][t][0], acc[3 % KA][t][1], a3, (double)b[t].w);
                    } else {
#pragma unroll
                        for (int t = 0; t < NT; ++t) {
                            if (t >= have) break;
                            const float4 b = mine[t * 32];
                            dmma(acc[0 % KA][t][0], acc[0 % KA][t][1], a0, (double)b.x);
                            dmma(acc[1 % KA][t][0], acc[1 % KA][t][1], a1, (double)b.y);
                            dmma(acc[2 % KA][t][0], acc[2 % KA][t][1], a2, (double)b.z);
                            dmma(acc[3 % KA][t][0], acc[3 % KA][t][1], a3, (double)b.w);
                        }
                        fetch_group();
                    }
                }
            } else if (have >= NT) {
                for (int g = 0; g < kg; ++g) {
                    float4 b[NT];
#pragma unroll
                    for (int t = 0; t < NT; ++t) b[t] = __ldg(wt + t * ws + g * 32);
                    const double a0 = arow[g * 16], a1 = arow[g * 16 + 4], a2 = arow[g * 16 + 8], a3 = arow[g * 16 + 12];
                    const int steps = g + 1 < kg ? 4 : tail;
#pragma unroll
                    for (int t = 0; t < NT; ++t) dmma(acc[0 % KA][t][0], acc[0 % KA][t][1], a0, (double)b[t].x);
                    if (steps < 2) break;
#pragma unroll
                    for (int t = 0; t < NT; ++t) dmma(acc[1 % KA][t][0], acc[1 % KA][t][1], a1, (double)b[t].y);
                    if (steps < 3) break;
#pragma unroll
                    for (int t = 0; t < NT; ++t) dmma(acc[2 % KA][t][0], acc[2 % KA][t][1], a2, (double)b[t].z);
                    if (steps < 4) break;
#pragma unroll
                    for (int t = 0; t < NT; ++t) dmma(acc[3 % KA][t][0], acc[3 % KA][t][1], a3, (double)b[t].w);
                }
            } else {   // fewer tiles than the kernel is built for (a narrow layer, the last sweep)
                for (int g = 0; g < kg; ++g) {
                    const double a0 = arow[g * 16], a1 = arow[g * 16 + 4], a2 = arow[g * 16 + 8], a3 = arow[g * 16 + 12];
#pragma unroll
                    for (int t = 0; t < NT; ++t) {
                        if (t >= have) break;
                        const float4 b = __ldg(wt + t * ws + g * 32);
                        dmma(acc[0 % KA][t][0], acc[0 % KA][t][1], a0, (double)b.x);
                        dmma(acc[1 % KA][t][0], acc[1 % KA][t][1], a1, (double)b.y);
                        dmma(acc[2 % KA][t][0], acc[2 % KA][t][1], a2, (double)b.z);
                        dmma(acc[3 % KA][t][0], acc[3 % KA][t][1], a3, (double)b.w);
                    }
                }
            }
#pragma unroll
            for (int c = KA / 2; c > 0; c /= 2)
#pragma unroll
                for (int u = 0; u < c; ++u)
#pragma unroll
                    for (int t = 0; t < NT; ++t) { acc[u][t][0] += acc[u + c][t][0]; acc[u][t][1] += acc[u + c][t][1]; }
            if (bufs == 1 && lay > 0) meet_rows();   // the rows are written in place
            // The usual case without a branch, so that the coefficients' chains of conversions and table reads overlap (a row past
            // the last one has zero coefficients and a valid table; its sums are not read): 5 of a layer's 18 thousand cycles
            // at 256 columns, four tiles a warp, with a branch at every coefficient; 37 domains 249 -> 235 us a call.
            if (lay > 0 && !ckpt && have >= NT && (nb + ni + (NT - 1) * NW) * 8 + 8 <= N) {
#pragma unroll
                for (int t = 0; t < NT; ++t) {
                    const int j0 = (nb + ni + t * NW) * 8 + lq * 2;
                    const float4 *e0 = (const float4 *)(t4 + j0), *e1 = (const float4 *)(t4 + j0 + 1);
                    const float4 f0 = e0[0], g0 = e0[1], i0 = e0[2], f1 = e1[0], g1 = e1[1], i1 = e1[2];
                    const float c0 = cast_coeff(acc[0][t][0], upper, f0, g0.x, gp), c1 = cast_coeff(acc[0][t][1], upper, f1, g1.x, gp);
                    double2 v;
                    v.x = relax_step(c0, upper, f0, g0.y, __hiloint2double(__float_as_int(g0.w), __float_as_int(g0.z)), i0, rb, rp, gp);
                    v.y = relax_step(c1, upper, f1, g1.y, __hiloint2double(__float_as_int(g1.w), __float_as_int(g1.z)), i1, rb, rp, gp);
                    put2(nxt + j0, v);
                }
                continue;
            }
#pragma unroll
            for (int t = 0; t < NT; ++t) {
                if (t >= have) break;
                const int j0 = (nb + ni + t * NW) * 8 + lq * 2;
                if (lay > 0) {
                    double2 v = make_double2(0.0, 0.0);
                    if (live && j0 < N) {
                        const PassEntry *te = t4 + j0;
                        const float4 f = *(const float4 *)&te->ls, g2 = *(const float4 *)&te->zlo;
                        const double cj = __hiloint2double(__float_as_int(g2.w), __float_as_int(g2.z));
                        const float c = cast_coeff(acc[0][t][0], upper, f, g2.x, gp);
                        if (ckpt) ckpt[(lay - 1) * ckpt_stride + ((long)d * 2 * n_rows + r) * lda + j0] = c;
                        v.x = relax_step(c, upper, f, g2.y, cj, *(const float4 *)&te->ui, rb, rp, gp);
                    }
                    if (live && j0 + 1 < N) {
                        const PassEntry *te = t4 + j0 + 1;
                        const float4 f = *(const float4 *)&te->ls, g2 = *(const float4 *)&te->zlo;
                        const double cj = __hiloint2double(__float_as_int(g2.w), __float_as_int(g2.z));
                        const float c = cast_coeff(acc[0][t][1], upper, f, g2.x, gp);
                        if (ckpt) ckpt[(lay - 1) * ckpt_stride + ((long)d * 2 * n_rows + r) * lda + j0 + 1] = c;
                        v.y = relax_step(c, upper, f, g2.y, cj, *(const float4 *)&te->ui, rb, rp, gp);
                    }
                    put2(nxt + j0, v);
                } else {
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const int j = j0 + h;
                        if (!live || j >= N) continue;
                        const float c = (float)acc[0][t][h];
                        const double e = acc[0][t][h] - (double)c, l = xl[j], u = xu[j];
                        const double el = e * l, eu = e * u;   // the box may have any sign: k_gemm_f64's charge as it stands
                        rp += (upper ? fmax(el, eu) : fmax(-el, -eu)) + 2.9e-14 * fabs(e) * fmax(fabs(l), fabs(u));
                        if (!(fabsf(c) < 1e10f)) bad = true;   // is_crown_coeff_safe, crates/ny-core/src/gemm.rs:127
                        const double x = ((c >= 0.f) != upper) ? l : u;
                        if (c != 0.f && x != 0.0) { const double p = (double)c * x; cs += p; ca += fabs(p); }
                        if (a_out) a_out[((long)d * 2 * n_rows + r) * lda + j] = c;
                    }
                }
            }
        }
        if (lay > 0) {
            if ((nt & 1) && ni == 0) put2(nxt + nt * 8 + lq * 2, make_double2(0.0, 0.0));   // the groups of sixteen are read whole
            meet_rows();
            double *sw = cur; cur = nxt; nxt = sw;
        }
    }
    // row sums: the four lanes of a row, then the warps that share it, in a fixed order
    double v[4] = {rb, rp + (double)gp, cs, ca};
    int anybad = bad ? 1 : 0;
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) {
#pragma unroll
        for (int i = 0; i < 4; ++i) v[i] += __shfl_xor_sync(0xffffffffu, v[i], o);
        anybad |= __shfl_xor_sync(0xffffffffu, anybad, o);
    }
    if (NW > 1) {   // the warps' sums in their order, by the row's lane of the group's first warp
        if (lq == 0) {
#pragma unroll
            for (int i = 0; i < 4; ++i) s_red[warp * 8 + lr][i] = v[i];
            s_bad[warp * 8 + lr] = anybad;
        }
        if (C > 1) cl.sync(); else __syncthreads();
#pragma unroll
        for (int i = 0; i < 4; ++i) v[i] = 0.0;
        anybad = 0;
        if (ni == 0 && lq == 0)
            for (int p = 0; p < C; ++p)
                for (int w2 = 0; w2 < nw1; ++w2) {
                    const int at = (mi * nw1 + w2) * 8 + lr;
                    const double *o = C > 1 ? cl.map_shared_rank(&s_red[at][0], p) : &s_red[at][0];
#pragma unroll
                    for (int i = 0; i < 4; ++i) v[i] += o[i];
                    anybad |= C > 1 ? *cl.map_shared_rank(&s_bad[at], p) : s_bad[at];
                }
    }
    if (ni == 0 && lq == 0 && live) {
        // 2^-40 >> (number of binary64 additions) * 2^-53, as k_concretize; the last term encloses underflowed products
        const double slack = (v[3] + fabs(v[0])) * 9.094947017729282e-13 + 1e-200;
        if (!upper) { const double x = v[0] + v[2] - v[1] - slack; out_lo[(long)d * n_rows + rr] = (anybad || isnan(x)) ? -INFINITY : __double2float_rd(x); }
        else { const double x = v[0] + v[2] + v[1] + slack; out_hi[(long)d * n_rows + rr] = (anybad || isnan(x)) ? INFINITY : __double2float_ru(x); }
    }
    if (RING) asm volatile("cp.async.wait_all;" ::: "memory");
    if (C > 1) cl.sync();   // the sums have been read before their CTA leaves
}

// k_direct_pass for many rows of narrow layers (up to 64 columns): a warp alone takes two groups of eight rows, so that a weight is
// loaded and converted once for both and twice the products are in flight.  What bounds the one-group form there is their
// latency and the conversions, not the tensor instruction (1024 boxes of 5 -> 6x50 -> 5: 816 us of passes where the products take
// 190).  A call on those boxes 1147 -> 1033 us, 512 of them 648 -> 600.
template <int NT>
__global__ void __launch_bounds__(128, 3)
k_direct_rows(const __grid_constant__ PackedNet pn, int top, int boxes, const int *__restrict__ idx, int n_rows, int pitch, const float *__restrict__ seed,
              const float *__restrict__ seed_bias, const float *__restrict__ in_lo, const float *__restrict__ in_hi, long box_ds,
              const PassEntry *__restrict__ ptab, float *__restrict__ out_lo, float *__restrict__ out_hi, float *__restrict__ a_out, int lda) {
    constexpr int MG = 2;
    extern __shared__ double s_coef[];
    const NetView &nv = pn.nv;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, lr = lane >> 2, lq = lane & 3;
    pdl_trigger();
    pdl_wait();
    int d[MG], r[MG], rr[MG];
    bool live[MG], upper[MG], bad[MG];
    double rb[MG], rp[MG], cs[MG], ca[MG];
    float gp[MG];
    double *cur[MG];
#pragma unroll
    for (int m = 0; m < MG; ++m) {   // rows of all boxes one behind the other: a group may span boxes
        const int gr = (((int)blockIdx.x * 4 + warp) * MG + m) * 8 + lr;
        live[m] = gr < boxes * 2 * n_rows;
        const int box = live[m] ? gr / (2 * n_rows) : 0;
        r[m] = live[m] ? gr - box * 2 * n_rows : 0;
        d[m] = idx ? idx[box] : box;
        upper[m] = r[m] >= n_rows;
        rr[m] = upper[m] ? r[m] - n_rows : r[m];
        rb[m] = rp[m] = cs[m] = ca[m] = 0.0;
        gp[m] = 0.f; bad[m] = false;
        cur[m] = s_coef + ((warp * MG + m) * 8 + lr) * pitch;
        const int n = nv.dims[top], np16 = (n + 15) & ~15;
        const bool spec = top == nv.L;   // rows at the network's output: no ReLU in front of the first contraction
        const PassEntry *t = ptab + (long)d[m] * nv.nps + nv.pre_off[top - 1];
        for (int j = lq; j < np16; j += 4) {
            double v = 0.0;
            if (live[m] && j < n) {
                const float a = seed[(long)rr[m] * n + j];
                if (spec) { v = a; rb[m] += v * t[j].bias; rp[m] += fabs(v) * t[j].cj; }
                else v = relax_step(a, upper[m], *(const float4 *)&t[j].ls, t[j].sbeta, t[j].cj, *(const float4 *)&t[j].ui, rb[m], rp[m], gp[m]);
            }
            cur[m][j] = v;
        }
        if (live[m] && seed_bias && lq == 0) { const double c = seed_bias[rr[m]]; rb[m] += c; rp[m] += 1.8189894035458565e-12 * fabs(c); }
    }
    __syncwarp();
    for (int lay = top - 1; lay >= 0; --lay) {
        const int K = nv.dims[lay + 1], N = nv.dims[lay], kg = (K + 15) >> 4, nt = (N + 7) >> 3;
        const int tail = (K - (kg - 1) * 16 + 3) >> 2;   // m8n8k4 steps of the last group
        const float4 *__restrict__ w = pn.w[lay] + lane;
        for (int nb = 0; nb < nt; nb += NT) {   // (one sweep unless this is the input layer)
            const int have = nt - nb;
            double acc[MG][NT][2];
#pragma unroll
            for (int m = 0; m < MG; ++m)
#pragma unroll
                for (int t = 0; t < NT; ++t) acc[m][t][0] = acc[m][t][1] = 0.0;
            const float4 *wt = w + (long)nb * kg * 32;
            const long ws = (long)kg * 32;
            for (int g = 0; g < kg; ++g) {
                float4 b[NT];
#pragma unroll
                for (int t = 0; t < NT; ++t)
                    if (t < have) b[t] = __ldg(wt + t * ws + g * 32);
                const int steps = g + 1 < kg ? 4 : tail;
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    if (c >= steps) break;
                    double a[MG];
#pragma unroll
                    for (int m = 0; m < MG; ++m) a[m] = cur[m][g * 16 + c * 4 + lq];
#pragma unroll
                    for (int t = 0; t < NT; ++t) {
                        if (t >= have) break;
                        const double bd = (double)(c == 0 ? b[t].x : c == 1 ? b[t].y : c == 2 ? b[t].z : b[t].w);
#pragma unroll
                        for (int m = 0; m < MG; ++m) dmma(acc[m][t][0], acc[m][t][1], a[m], bd);
                    }
                }
            }
            if (lay > 0) {
                __syncwarp();   // the rows are written in place
#pragma unroll
                for (int t = 0; t < NT; ++t) {
                    if (t >= have) break;
                    const int j0 = (nb + t) * 8 + lq * 2;
                    const bool whole = (nb + t) * 8 + 8 <= N;
#pragma unroll
                    for (int m = 0; m < MG; ++m) {
                        const PassEntry *te = ptab + (long)d[m] * nv.nps + nv.pre_off[lay - 1] + j0;
                        double2 v = make_double2(0.0, 0.0);
                        auto one = [&](const PassEntry *at, double sum) {
                            const float4 f = *(const float4 *)&at->ls, g2 = *(const float4 *)&at->zlo, ib = *(const float4 *)&at->ui;
                            const float c = cast_coeff(sum, upper[m], f, g2.x, gp[m]);
                            return relax_step(c, upper[m], f, g2.y, __hiloint2double(__float_as_int(g2.w), __float_as_int(g2.z)), ib, rb[m], rp[m], gp[m]);
                        };
                        if (whole) { v.x = one(te, acc[m][t][0]); v.y = one(te + 1, acc[m][t][1]); }   // (dead rows: see k_direct_pass)
                        else {
                            if (j0 < N) v.x = one(te, acc[m][t][0]);
                            if (j0 + 1 < N) v.y = one(te + 1, acc[m][t][1]);
                        }
                        *(double2 *)(cur[m] + j0) = v;
                    }
                }
            } else {
#pragma unroll
                for (int t = 0; t < NT; ++t) {
                    if (t >= have) break;
#pragma unroll
                    for (int m = 0; m < MG; ++m)
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            const int j = (nb + t) * 8 + lq * 2 + h;
                            if (!live[m] || j >= N) continue;
                            const float c = (float)acc[m][t][h];
                            const double e = acc[m][t][h] - (double)c, l = in_lo[(long)d[m] * box_ds + j], u = in_hi[(long)d[m] * box_ds + j];
                            const double el = e * l, eu = e * u;   // the box may have any sign: k_gemm_f64's charge as it stands
                            rp[m] += (upper[m] ? fmax(el, eu) : fmax(-el, -eu)) + 2.9e-14 * fabs(e) * fmax(fabs(l), fabs(u));
                            if (!(fabsf(c) < 1e10f)) bad[m] = true;   // is_crown_coeff_safe, crates/ny-core/src/gemm.rs:127
                            const double x = ((c >= 0.f) != upper[m]) ? l : u;
                            if (c != 0.f && x != 0.0) { const double p = (double)c * x; cs[m] += p; ca[m] += fabs(p); }
                            if (a_out) a_out[((long)d[m] * 2 * n_rows + r[m]) * lda + j] = c;
                        }
                }
            }
        }
        if (lay > 0) {
            if (nt & 1)   // the groups of sixteen are read whole
#pragma unroll
                for (int m = 0; m < MG; ++m) *(double2 *)(cur[m] + nt * 8 + lq * 2) = make_double2(0.0, 0.0);
            __syncwarp();
        }
    }
#pragma unroll
    for (int m = 0; m < MG; ++m) {
        double v[4] = {rb[m], rp[m] + (double)gp[m], cs[m], ca[m]};
        int anybad = bad[m] ? 1 : 0;
#pragma unroll
        for (int o = 1; o < 4; o <<= 1) {
#pragma unroll
            for (int i = 0; i < 4; ++i) v[i] += __shfl_xor_sync(0xffffffffu, v[i], o);
            anybad |= __shfl_xor_sync(0xffffffffu, anybad, o);
        }
        if (lq == 0 && live[m]) {
            const double slack = (v[3] + fabs(v[0])) * 9.094947017729282e-13 + 1e-200;   // as k_direct_pass
            if (!upper[m]) { const double x = v[0] + v[2] - v[1] - slack; out_lo[(long)d[m] * n_rows + rr[m]] = (anybad || isnan(x)) ? -INFINITY : __double2float_rd(x); }
            else { const double x = v[0] + v[2] + v[1] + slack; out_hi[(long)d[m] * n_rows + rr[m]] = (anybad || isnan(x)) ? INFINITY : __double2float_ru(x); }
        }
    }
}

__device__ __forceinline__ void meet(float &l, float &u, float bl, float bu) {
    const float tl = fmaxf(l, bl), tu = fminf(u, bu);
    if (tl <= tu) { l = tl; u = tu; }
    else { l = fminf(l, bl); u = fmaxf(u, bu); }
}

// Domain flags and repair rule of k_finalize on one row's bounds.
__device__ __forceinline__ void repair(int f, float &l, float &u) {
    if (f || !isfinite(l) || !isfinite(u) || l > u) { l = -INFINITY; u = INFINITY; }
}

// Layer k's forward image of the tightened input, then the merge rule of k_crown_flags / k_crown_merge
// (nyb200_crown.cu) and the pass table, one CTA per box.  c_lo null: no CROWN bounds for this layer (the first layer,
// where the pass would repeat the interval image, and the last one, which takes the forward shortcut).
__global__ void __launch_bounds__(512)
k_crown_layer(NetView nv, int k, int zdim, const float *__restrict__ ibp_lo, const float *__restrict__ ibp_hi, const float *__restrict__ raw_lo, const float *__restrict__ raw_hi,
              const float *__restrict__ q, const float *__restrict__ c_lo, const float *__restrict__ c_hi, float *__restrict__ t_lo,
              float *__restrict__ t_hi, float *zl, float *zu, PassEntry *__restrict__ ptab, const signed char *__restrict__ code,
              int *__restrict__ dflags, float *__restrict__ inter_lo, float *__restrict__ inter_hi) {
    // The box's values in shared memory: what earlier kernels left, on its way while the image is summed, and the image.
    extern __shared__ double s_z[];
    float *s_ibl = (float *)(s_z + 2 * zdim), *s_ibu = s_ibl + zdim, *s_rl = s_ibu + zdim, *s_ru = s_rl + zdim, *s_q = s_ru + zdim, *s_cl = s_q + zdim,
          *s_cu = s_cl + zdim;
    pdl_trigger();
    const int d = blockIdx.x, n = nv.dims[k + 1];
    if (k > 0) warm_weights(nv.W[k], nv.dims[k] * n);
    pdl_wait();
    const bool relu = k < nv.L - 1;
    const long o = (long)d * nv.nps + nv.pre_off[k];
    for (int j = threadIdx.x; j < n; j += blockDim.x) {
        s_ibl[j] = ibp_lo[o + j]; s_ibu[j] = ibp_hi[o + j];
        if (c_lo) { s_cl[j] = c_lo[(long)d * n + j]; s_cu[j] = c_hi[(long)d * n + j]; }
        if (k == 0) { s_rl[j] = raw_lo[o + j]; s_ru[j] = raw_hi[o + j]; s_q[j] = q[o + j]; }
    }
    const int dfl = dflags[d];
    if (k > 0) {
        const long in = (long)d * nv.nps + nv.pre_off[k - 1];
        const int n_in = nv.dims[k];
        for (int i = threadIdx.x; i < n_in; i += blockDim.x) centre(zl[in + i], zu[in + i], s_z[i], s_z[zdim + i]);
        __syncthreads();
        const double gam = gam_sweep(n_in);
        interval_sweep<2>(nv.W[k], n_in, 0, n, s_z, s_z + zdim, true, NoEarly(), [&](int j, double lo, double hi, double qq, int) {
            outward(lo, hi, qq, gam, nv.b[k], j, s_rl[j], s_ru[j], s_q[j]);
        });
    }
    __syncthreads();
    int unstable = 0, n_unst = 0;
    for (int j = threadIdx.x; j < n; j += blockDim.x) {
        if (!(s_ibl[j] >= 0.f || s_ibu[j] <= 0.f)) unstable = 1;
        if (s_rl[j] < 0.f && s_ru[j] > 0.f) ++n_unst;
    }
    __shared__ int s_cnt;
    if (threadIdx.x == 0) s_cnt = 0;
    const bool all_stable = !__syncthreads_or(unstable);
    if (n_unst) atomicAdd(&s_cnt, n_unst);
    __syncthreads();
    const bool sparse = s_cnt > 0 && !(1.0f - (float)s_cnt / (float)n < 0.9f);
    auto second = [&](int j, float &cl, float &cu) {
        const float l = s_rl[j], u = s_ru[j];
        if (c_lo == nullptr || (sparse && !(l < 0.f && u > 0.f))) { cl = l; cu = u; return; }
        cl = s_cl[j]; cu = s_cu[j];
        repair(dfl, cl, cu);
    };
    int nan = 0;
    for (int j = threadIdx.x; j < n; j += blockDim.x) {
        float cl, cu;
        second(j, cl, cu);
        if (isnan(s_ibl[j]) || isnan(s_ibu[j]) || isnan(cl) || isnan(cu)) nan = 1;
    }
    const bool any_nan = __syncthreads_or(nan);
    int found = 0;
    const double eps = eps64(n);
    for (int j = threadIdx.x; j < n; j += blockDim.x) {
        const float il = s_ibl[j], iu = s_ibu[j];
        float l = il, u = iu;
        if (!(relu && all_stable) && !any_nan) {
            float cl, cu;
            second(j, cl, cu);
            meet(l, u, cl, cu);
        }
        // pre-activation clamp of a ReLU split (constraints/lookups.rs:138-185); an emptied interval marks the domain
        const int sc = (relu && code) ? code[o + j] : 0;
        if (sc > 0 && !isnan(l)) l = fmaxf(l, 0.f);
        if (sc < 0 && !isnan(u)) u = fminf(u, 0.f);
        if (sc != 0 && l > u) found |= kFlagInfeasible;
        t_lo[o + j] = l; t_hi[o + j] = u;
        const long io = (long)d * nv.n_pre + nv.pre_off[k] + j;
        inter_lo[io] = l; inter_hi[io] = u;
        const double bias = nv.b[k] ? (double)nv.b[k][j] : 0.0, qv = s_q[j];
        PassEntry pe;
        pe.bias = bias; pe.sbeta = pe.zg = pe.zhi = pe.zlo = 0.f; pe.ui = 0.f; pe.lsu = 1.f;
        if (!relu) {   // the specification rows pass through unchanged
            zl[o + j] = l; zu[o + j] = u;
            pe.ls = pe.us = 1.f; pe.cj = eps * qv + 1.8189894035458565e-12 * fabs(bias);
            ptab[o + j] = pe;
            continue;
        }
        float ls, us, ui;
        if (isnan(l) || isnan(u) || ((isinf(l) || isinf(u)) && l < 0.f && u > 0.f)) { found |= kFlagDegraded; ls = us = ui = 0.f; }
        else if (l >= 0.f) { ls = 1.f; us = 1.f; ui = 0.f; }
        else if (u <= 0.f) { ls = us = ui = 0.f; }
        else {   // plain-CROWN chord in binary64, slope and intercept stepped up
            us = step_up((float)((double)u / ((double)u - (double)l)));
            ui = step_up((float)(-(double)us * (double)l));
            ls = (u > -l) ? 1.f : 0.f;
        }
        float pl = isnan(il) ? il : fmaxf(il, 0.f), pu = isnan(iu) ? iu : fmaxf(iu, 0.f);
        if (!any_nan) meet(pl, pu, fmaxf(l, 0.f), fmaxf(u, 0.f));
        if (sc < 0) { pl = 0.f; pu = 0.f; }
        const float za = fmaxf(fabsf(l), fabsf(u));
        pe.ls = pe.lsu = ls; pe.us = us; pe.ui = ui;
        pe.zg = (us == 1.f && ui == 0.f) ? 0.f : za;
        pe.zhi = __fmul_ru(pu, 1.000001f); pe.zlo = __fmul_rd(pl, 0.999999f);
        pe.cj = eps * qv + 1.8189894035458565e-12 * ((double)za + fabs(bias));   // 2^-39
        ptab[o + j] = pe;
        zl[o + j] = pl; zu[o + j] = pu;
    }
    if (found) atomicOr(&dflags[d], found);
}

// Specification rows: interval images of the network's IBP output and of its tightened output, merge with the final
// pass (the rules of k_spec_interval and k_crown_final), one warp per box.
__global__ void __launch_bounds__(256)
k_crown_spec(int D, int S, int nL, const float *__restrict__ spec, const float *__restrict__ ibp_lo, const float *__restrict__ ibp_hi,
             const float *__restrict__ t_lo, const float *__restrict__ t_hi, long stride, int off, const float *__restrict__ c_lo,
             const float *__restrict__ c_hi, const int *__restrict__ dflags, float *__restrict__ out_lo, float *__restrict__ out_hi,
             float4 *__restrict__ scratch) {
    pdl_trigger();
    pdl_wait();
    const int d = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (d >= D) return;
    const int fl = dflags[d];
    const double g = eps64(nL);
    auto image = [&](int s, const float *l, const float *u, float &lo, float &hi) {
        double a = 0.0, b = 0.0, qq = 0.0;
        for (int j = 0; j < nL; ++j) {
            const double w = spec[s * nL + j];
            const bool pos = w > 0.0;
            a = fma(w, pos ? (double)l[j] : (double)u[j], a);
            b = fma(w, pos ? (double)u[j] : (double)l[j], b);
            qq = fma(fabs(w), fmax(fabs((double)l[j]), fabs((double)u[j])), qq);
        }
        lo = __double2float_rd(a - g * qq); hi = __double2float_ru(b + g * qq);
        if (isnan(lo) || isnan(hi)) { lo = -INFINITY; hi = INFINITY; }
    };
    int n_unst = 0;
    const long row = (long)d * stride + off;
    for (int s = lane; s < S; s += 32) {
        float4 v;
        image(s, ibp_lo + row, ibp_hi + row, v.x, v.y);
        image(s, t_lo + row, t_hi + row, v.z, v.w);
        scratch[(long)d * S + s] = v;
        if (v.z < 0.f && v.w > 0.f) ++n_unst;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) n_unst += __shfl_xor_sync(0xffffffffu, n_unst, o);
    const bool sparse = n_unst > 0 && !(1.0f - (float)n_unst / (float)S < 0.9f);
    bool nan = false, cnan = false;
    for (int s = lane; s < S; s += 32) {
        const float4 v = scratch[(long)d * S + s];
        float cl = c_lo[(long)d * S + s], cu = c_hi[(long)d * S + s];
        repair(fl, cl, cu);
        const bool use_f = sparse && !(v.z < 0.f && v.w > 0.f);
        const float sl = use_f ? v.z : cl, su = use_f ? v.w : cu;
        nan |= isnan(v.x) || isnan(v.y) || isnan(sl) || isnan(su);
        cnan |= isnan(cl) || isnan(cu);
    }
    nan = __any_sync(0xffffffffu, nan);
    cnan = __any_sync(0xffffffffu, cnan);
    for (int s = lane; s < S; s += 32) {
        const float4 v = scratch[(long)d * S + s];
        float cl = c_lo[(long)d * S + s], cu = c_hi[(long)d * S + s];
        repair(fl, cl, cu);
        if (!(fl & (kFlagDegraded | kFlagInvalid | kFlagInfeasible))) {
            float l = v.x, u = v.y;
            if (!nan) {
                const bool use_f = sparse && !(v.z < 0.f && v.w > 0.f);
                meet(l, u, use_f ? v.z : cl, use_f ? v.w : cu);
            }
            if (cnan) { cl = l; cu = u; }
            else if (!(isnan(l) || isnan(u))) meet(cl, cu, l, u);
        }
        if (fl & kFlagInfeasible) { cl = INFINITY; cu = -INFINITY; }
        out_lo[(long)d * S + s] = cl; out_hi[(long)d * S + s] = cu;
    }
}

// Interval pass of a batch of split domains (modes 0 and 1 of run_forward), one cluster of CTAs per domain through all
// layers (a small batch spreads every domain's outputs over up to eight SMs; the CTAs hand each other the intervals of a
// layer through distributed shared memory): split
// lists, interval images, inherited bounds, clamps, relaxation tables, post-activation intervals.  Launched layer by
// layer the same work is 2 L + 4 launches of 5-11 us each whatever the batch.  idx: the domains' places in the per-domain
// arrays, or null (then the run's minimum and counters are cleared here too).  raw_lo / raw_hi / q0: the first layer's
// image when all domains share the input box, or null.
__global__ void __launch_bounds__(512)
k_direct_forward(NetView nv, int mode, int zdim, const int *__restrict__ idx, const float *__restrict__ in_lo,
                 const float *__restrict__ in_hi, long box_ds, const float *__restrict__ raw_lo, const float *__restrict__ raw_hi,
                 const float *__restrict__ q0, const float *__restrict__ inh_lo, const float *__restrict__ inh_hi, long inh_ds,
                 const nyb200_split *__restrict__ splits, const int *__restrict__ nsplits, int max_splits,
                 const float *__restrict__ alpha, signed char *__restrict__ code, float *__restrict__ sbeta,
                 float *__restrict__ pre_lo, float *__restrict__ pre_hi, float *__restrict__ zl, float *__restrict__ zu,
                 float4 *__restrict__ tab, float *__restrict__ zabs, float *__restrict__ q, int *__restrict__ flags,
                 float *__restrict__ min_words) {
    extern __shared__ double s_z[];
    __shared__ int s_flags;
    cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
    const int C = (int)cl.num_blocks(), rank = (int)cl.block_rank();
    pdl_trigger();
    pdl_wait();
    const int d = idx ? idx[blockIdx.x / C] : blockIdx.x / C;
    const long row = (long)d * nv.nps;
    if (!idx && blockIdx.x == 0 && threadIdx.x < 8) min_words[threadIdx.x] = threadIdx.x == 0 ? INFINITY : 0.f;
    if (threadIdx.x == 0) s_flags = 0;
    signed char *s_code = (signed char *)(s_z + 4 * zdim);   // split codes and multipliers of the domain, every CTA its copy
    float *s_beta = (float *)(s_code + nv.nps);
    for (int i = threadIdx.x; i < nv.nps; i += blockDim.x) { s_code[i] = 0; s_beta[i] = 0.f; }
    double *zc = s_z, *zn = s_z + 2 * zdim;
    if (!raw_lo)
        for (int i = threadIdx.x; i < nv.dims[0]; i += blockDim.x) { zc[i] = in_lo[(long)d * box_ds + i]; zc[zdim + i] = in_hi[(long)d * box_ds + i]; }
    if (C > 1) cl.sync(); else __syncthreads();   // (every CTA of the cluster runs before another one writes to it)
    int bad = 0;
    const int ns = max_splits > 0 ? nsplits[d] : 0;
    for (int i = threadIdx.x; i < ns; i += blockDim.x) {   // as k_scatter_splits
        const nyb200_split c = splits[(long)d * max_splits + i];
        if (c.relu < 0 || c.relu >= nv.L - 1 || c.neuron < 0 || c.neuron >= nv.dims[c.relu + 1] || (c.sign != 1 && c.sign != -1)) { bad |= kFlagInvalid; continue; }
        const int o = nv.pre_off[c.relu] + c.neuron;
        s_code[o] = (signed char)c.sign;
        s_beta[o] = isfinite(c.beta) ? c.beta * (float)c.sign : 0.0f;
    }
    __syncthreads();
    for (int i = rank * blockDim.x + threadIdx.x; i < nv.nps; i += C * blockDim.x) { code[row + i] = s_code[i]; sbeta[row + i] = s_beta[i]; }
    float *s_l = s_beta + nv.nps, *s_u = s_l + zdim, *s_q = s_u + zdim;
    struct Held { float il, iu, bias; };
    for (int k = 0; k < nv.L; ++k) {
        const int off = nv.pre_off[k], n = nv.dims[k + 1];
        const long o = row + off;
        const bool last = k == nv.L - 1;
        const double gam = gam_sweep(nv.dims[k]);
        auto early = [&](int j) {
            Held h;
            const long io = (long)d * inh_ds + off + j;
            h.il = inh_lo[io]; h.iu = inh_hi[io];
            h.bias = nv.b[k] ? nv.b[k][j] : 0.f;
            return h;
        };
        const int per = (n + C - 1) / C, j0 = min(n, rank * per), j1 = min(n, j0 + per);
        // The interval the next layer reads goes to every CTA at once; what only later kernels read is kept here and
        // stored while the cluster is already in the next layer.
        auto image = [&](int j, float l, float u, float qf, const Held &h) {
            inherit_bounds(mode, &h.il, &h.iu, 0, l, u);
            s_l[j - j0] = l; s_u[j - j0] = u; s_q[j - j0] = qf;
            if (last) return;
            const int sc = s_code[off + j];
            if (sc > 0) l = isnan(l) ? l : fmaxf(l, 0.f);
            else if (sc < 0) u = isnan(u) ? u : fminf(u, 0.f);
            float pl = fmaxf(l, 0.f), pu = fmaxf(u, 0.f);   // as relax_neuron
            if (sc > 0) pu = u;
            else if (sc < 0) { pl = 0.f; pu = 0.f; }
            if (isnan(l)) pl = l;
            if (isnan(u)) pu = u;
            double c, r;
            centre(pl, pu, c, r);
            for (int p = 0; p < C; ++p) {
                double *z = cl.map_shared_rank(zn, p);
                z[j] = c; z[zdim + j] = r;
            }
        };
        if (k == 0 && raw_lo) {
            for (int j = j0 + threadIdx.x; j < j1; j += blockDim.x) image(j, raw_lo[j], raw_hi[j], q0[j], early(j));
        } else if (j0 < j1) {
            interval_sweep<2>(nv.W[k], nv.dims[k], j0, j1, zc, zc + zdim, k > 0, early, [&](int j, double lo, double hi, double qq, const Held &h) {
                float l, u, qf;
                outward(lo, hi, qq, gam, &h.bias, 0, l, u, qf);
                image(j, l, u, qf, h);
            });
        }
        __syncthreads();
        if (C > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        for (int j = j0 + threadIdx.x; j < j1; j += blockDim.x) {
            float l = s_l[j - j0], u = s_u[j - j0];
            q[o + j] = s_q[j - j0];
            if (!last) {
                float4 t;
                float pl, pu;
                bad |= relax_neuron(s_code[off + j], alpha, o + j, l, u, t, pl, pu);
                t.w = s_beta[off + j];
                tab[o + j] = t;
                zabs[o + j] = charge_magnitude(l, u);
                zl[o + j] = pl; zu[o + j] = pu;
            }
            pre_lo[o + j] = l; pre_hi[o + j] = u;
        }
        if (C > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        __syncthreads();
        double *sw = zc; zc = zn; zn = sw;
    }
    int *flag0 = C > 1 ? cl.map_shared_rank(&s_flags, 0) : &s_flags;
    if (bad) atomicOr(flag0, bad);
    if (C > 1) cl.sync(); else __syncthreads();
    if (rank == 0 && threadIdx.x == 0) flags[d] = s_flags;
}

// Pass table of a batch from its relaxation tables, intervals and charge weights.  shared: all domains have one box, and the general
// interval pass leaves the first layer's charge weights in the first domain's row alone.
__global__ void __launch_bounds__(256)
k_pass_table(NetView nv, int boxes, bool shared, const int *__restrict__ idx, const float4 *__restrict__ tab, const float *__restrict__ zabs,
             const float *__restrict__ q, const float *__restrict__ zl, const float *__restrict__ zu, const float *__restrict__ alpha_up,
             PassEntry *__restrict__ ptab) {
    pdl_trigger();
    pdl_wait();
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long)boxes * nv.n_pre) return;
    const int box = (int)(t / nv.n_pre), i = (int)(t - (long)box * nv.n_pre);
    int k = 0;
    while (k + 1 < nv.L && i >= nv.pre_off[k + 1]) ++k;
    const int j = i - nv.pre_off[k];
    const long o = (long)(idx ? idx[box] : box) * nv.nps + i;
    PassEntry pe;
    pe.bias = nv.b[k] ? (double)nv.b[k][j] : 0.0;
    pe.cj = eps64(nv.dims[k + 1]) * (double)q[shared && k == 0 ? i : o] + 1.8189894035458565e-12 * fabs(pe.bias);   // 2^-39
    if (k == nv.L - 1) {   // the specification rows pass through unchanged
        pe.ls = pe.us = pe.lsu = 1.f; pe.zg = pe.zhi = pe.zlo = pe.sbeta = pe.ui = 0.f;
    } else {
        const float4 r = tab[o];
        const float za = zabs[o];
        pe.ls = r.x; pe.us = r.y; pe.ui = r.z; pe.sbeta = r.w;
        pe.lsu = alpha_up ? alpha_up[o] : r.x;
        pe.zg = (r.y == 1.f && r.z == 0.f) ? 0.f : za;
        // tables uploaded by the caller come with magnitudes only: the post-activation lies in [0, max|z|]
        pe.zhi = __fmul_ru(zu ? zu[o] : za, 1.000001f); pe.zlo = zl ? __fmul_rd(zl[o], 0.999999f) : 0.f;
        pe.cj += 1.8189894035458565e-12 * (double)za;
    }
    ptab[o] = pe;
}

int prepare_fragments(nyb200_engine *e, Net &net) {
    const NetView &nv = net.v;
    if (!net.frag.empty()) return NYB200_OK;
    std::vector<float *> frag((size_t)nv.L);
    NYB_TRY(build_operands(e, net, [&](Carve &c) {
        for (int k = 0; k < nv.L; ++k) {
            const int K = nv.dims[k + 1], N = nv.dims[k], kg = (K + 15) / 16, nt = (N + 7) / 8;
            const long n = (long)nt * kg * 32;
            frag[k] = (float *)c.take((size_t)n * 16);
            if (!c.block) continue;
            k_pack_fragments<<<(unsigned)((n + 255) / 256), 256, 0, e->stream>>>(nv.W[k], K, N, kg, nt, (float4 *)frag[k]);
            e->launches++;
        }
        return (int)NYB200_OK;
    }));
    net.frag = std::move(frag);
    return NYB200_OK;
}

PackedNet packed(const Net &net) {
    PackedNet pn;
    memset(&pn, 0, sizeof(pn));
    pn.nv = net.v;
    for (int k = 0; k < net.v.L; ++k) pn.w[k] = (const float4 *)net.frag[k];
    return pn;
}

int allow_smem(nyb200_engine *e, const void *kernel, size_t bytes) {
    if (bytes <= 40 * 1024) return NYB200_OK;
    NYB_CUDA(e, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPassMaxSmem));
    return NYB200_OK;
}

constexpr int kPassMaxWidth = 1536;      // two buffers of eight binary64 rows of that width fit in shared memory

int launch_pass(nyb200_engine *e, const PackedNet &pn, int top, int n_rows, int D, const int *idx, const float *seed, const float *seed_bias,
                const BatchPtrs &p, long box_ds, const PassEntry *ptab, float *c_lo, float *c_hi, float *a_out, float *ckpt = nullptr,
                long ckpt_stride = 0) {
    const NetView &nv = pn.nv;
    int wide = nv.dims[top], written = 0;   // widest row held; widest row a contraction writes
    for (int k = 1; k < top; ++k) { wide = nv.dims[k] > wide ? nv.dims[k] : wide; written = nv.dims[k] > written ? nv.dims[k] : written; }
    const int pitch = ((wide + 15) & ~15) + 4;   // rows start four 8-byte banks apart: a fragment load is free of conflicts
    const int groups = (int)(((long)D * 2 * n_rows + 7) / 8), tiles = (wide + 7) / 8;
    // Warps per group of rows: enough that a warp's columns fit its accumulators, and while the launch is small (fewer
    // than eight warps per SM) more of them, down to one tile each: a group's products are a serial chain.
    const int sms = usable_sms(e);
    int NW = 1;
    while (NW < 8 && (tiles > NW * 8 || ((long)groups * NW < (long)sms * 8 && tiles > NW))) NW *= 2;
    // a launch that leaves SMs idle all the same: clusters of two to eight CTAs of eight warps each
    int C = 1;
    while (NW >= 8 && C < 8 && groups * C * 2 <= sms && tiles >= NW * 2) { C *= 2; NW *= 2; }
    // Warps alone with all columns of their rows, six tiles of them and more: two groups of rows each (k_direct_rows), three CTAs of
    // eight groups an SM where the one-group form has two.  It pays where that saves a wave of CTAs and costs where it does not:
    // 5 -> 6x50 -> 5, us a call, one group / two, at n groups an SM: 16 311/347  20 429/357  24 442/406  26 458/505  32 484/525
    // 34 580/532  48 676/627  56 833/789  72 991/883  96 1216/1110; 4x64: 24 263/238  32 278/316  36 329/331  48 367/362  72 538/522.
    // Up to five tiles both have three CTAs: 4x20 and 5x33 within 2 % of each other from 8 to 96 groups an SM.
    auto waves = [&](long per_sm) { return ((long)groups + per_sm * sms - 1) / (per_sm * sms); };
    if (NW == 1 && C == 1 && !ckpt && tiles >= 6 && waves(24) < waves(16)) {
        const size_t rows_smem = (size_t)4 * 2 * 8 * pitch * 8;
        const dim3 rows_grid((unsigned)((groups + 7) / 8));
#define NYB_ROWS_PASS(NT) case NT:                                                                                              \
        NYB_TRY(allow_smem(e, (const void *)k_direct_rows<NT>, rows_smem));                                                     \
        NYB_CUDA(e, launch_pdl(k_direct_rows<NT>, rows_grid, dim3(128), rows_smem, e, pn, top, D, idx, n_rows, pitch, seed, seed_bias, \
                               (const float *)p.in_lo, (const float *)p.in_hi, box_ds, ptab, c_lo, c_hi, a_out, p.lda)); break;
        switch (tiles) { NYB_ROWS_PASS(6) NYB_ROWS_PASS(7) NYB_ROWS_PASS(8) }
#undef NYB_ROWS_PASS
        e->launches++;
        return NYB200_OK;
    }
    const int per = (tiles + NW - 1) / NW;
    int MT = 8 / (NW / C);
    const int bufs = C > 1 || (written + 7) / 8 > NW * 8 ? 2 : 1;   // one sweep per layer: the rows are replaced in place
    while (MT > 1 && (size_t)MT * 8 * pitch * 8 * bufs > kPassMaxSmem / 2) MT /= 2;
    size_t weights = 0;
    for (int k = 0; k < top; ++k) weights += (size_t)nv.dims[k] * nv.dims[k + 1] * 4;
    const size_t coef = (size_t)bufs * MT * 8 * pitch * 8;
    const int NTq = per > 8 ? 8 : per;
    const size_t ringb = (size_t)(NW / C) * MT * kRing * NTq * 512;
    // weights that L1 keeps (shared memory takes its share of it) need no ring, unless every CTA of the launch is the first on
    // its SM and meets an empty L1 (one box of 5 -> 6x50 -> 5: 173 -> 162 us a call)
    const bool ring = NTq <= 4 && (weights > 96 * 1024 || (groups + MT - 1) / MT * C <= sms) && coef + ringb <= kPassMaxSmem;
    const size_t smem = coef + (ring ? ringb : 0);
    dim3 grid((unsigned)((groups + MT - 1) / MT * C)), block((unsigned)(MT * (NW / C) * 32));
#define NYB_PASS_AS(NT, RING)                                                                                                 \
    NYB_TRY(allow_smem(e, (const void *)k_direct_pass<NT, RING>, smem));                                                      \
    NYB_CUDA(e, launch_pdl_cluster(k_direct_pass<NT, RING>, grid, block, C, smem, e, pn, top, D, idx, n_rows, MT, NW, pitch,  \
                                   bufs, seed, seed_bias, (const float *)p.in_lo, (const float *)p.in_hi, box_ds, ptab, c_lo, \
                                   c_hi, a_out, p.lda, ckpt, ckpt_stride))
#define NYB_PASS(NT) case NT: NYB_PASS_AS(NT, false); break;
#define NYB_PASS_RING(NT) case NT: if (ring) { NYB_PASS_AS(NT, true); } else { NYB_PASS_AS(NT, false); } break;
    switch (NTq) {
        NYB_PASS_RING(1) NYB_PASS_RING(2) NYB_PASS_RING(3) NYB_PASS_RING(4) NYB_PASS(5) NYB_PASS(6) NYB_PASS(7) NYB_PASS(8)
    }
#undef NYB_PASS
#undef NYB_PASS_RING
#undef NYB_PASS_AS
    e->launches++;
    return NYB200_OK;
}

}  // namespace

// Which calls take this form: fully connected networks without residual connections, hidden widths that fit, and no
// more binary64 work than some 60 ms of it: beyond that the 3xTF32 passes of the general pipeline are the faster ones
// when they are not flagged.
bool direct_eligible(const Net &net) {
    const NetView &nv = net.v;
    if (net.has_skip() || nv.dims[0] > kSweepMaxWidth || nv.nps > kDirectMaxNeurons) return false;
    for (int k = 0; k < nv.L; ++k)
        if (net.is_conv(k) || nv.dims[k + 1] > kPassMaxWidth) return false;
    return true;
}

bool crown_direct_eligible(const nyb200_engine *e, const Net &net, int S, int D) {
    const NetView &nv = net.v;
    if (!e->fuse_chain || (e->path == NYB200_PATH_TF32X3 && !e->small_direct)) return false;   // the caller asks for the per-layer or the tensor form
    if (e->error_channel == NYB200_ERRCH_REFERENCE || nv.L < 2 || !direct_eligible(net)) return false;
    double down = 0.0, macs = 0.0;
    for (int k = 0; k < nv.L; ++k) {
        macs += 2.0 * (k < nv.L - 1 ? nv.dims[k + 1] : 0) * down;
        down += (double)nv.dims[k] * nv.dims[k + 1];
    }
    macs += 2.0 * S * down;
    return macs * D <= 5e11;
}

int crown_direct(nyb200_engine *e, int net_id, const float *spec, int S, const float *in_lo, const float *in_hi, int box_stride,
                 int D, float *out_lo, float *out_hi, float *inter_lo, float *inter_hi, const CrownSplits *cs) {
    Net *net;
    NYB_TRY(find_net(e, net_id, &net));
    const NetView &nv = net->v;
    const int L = nv.L;
    const size_t np = nv.nps, n_res = (size_t)D * S, n_int = (size_t)D * nv.n_pre;
    NYB_TRY(prepare_fragments(e, *net));
    Batch b;
    const bool split = cs && cs->max_splits > 0;
    b.net_id = net_id; b.D = D; b.mode = 1; b.box_stride = box_stride; b.S = S; b.R = 2 * S; b.max_splits = split ? cs->max_splits : 0;
    BatchPtrs p;
    NYB_TRY(batch_ptrs(e, *net, b, p));
    e->batch = Batch();  // the resident batch's buffers are being reused
    int widest = S;
    for (int k = 1; k < L; ++k) widest = nv.dims[k] > widest ? nv.dims[k] : widest;
    NYB_WS(ibp_lo, float *, e, "ibp_lo", (size_t)D * np * 4);
    NYB_WS(ibp_hi, float *, e, "ibp_hi", (size_t)D * np * 4);
    NYB_WS(ptab, PassEntry *, e, "crown_ptab", (size_t)D * np * sizeof(PassEntry));
    NYB_WS(c_lo, float *, e, "crown_c", (size_t)2 * D * widest * 4);
    float *c_hi = c_lo + (size_t)D * widest;
    NYB_WS(scratch, float4 *, e, "crown_spec", n_res * 16);
    // results in the order of the caller's arrays: one copy to the host
    NYB_WS(res, float *, e, "crown_result", (2 * n_res + 2 * n_int) * 4);
    float *r_il = res + 2 * n_res, *r_iu = r_il + n_int;
    const size_t box = (size_t)nv.dims[0] * (box_stride ? (size_t)D : 1) * 4, bs = (size_t)S * nv.dims[L] * 4;
    const UploadPiece up[5] = {{p.in_lo, in_lo, box}, {p.in_hi, in_hi, box}, {p.nsplits, split ? cs->n_splits : nullptr, split ? (size_t)D * 4 : 0},
                               {p.splits, split ? cs->splits : nullptr, (size_t)D * b.max_splits * sizeof(nyb200_split)}, {p.spec, spec, bs}};
    NYB_TRY(staged_upload(e, up, 5));
    NYB_CUDA(e, cudaMemsetAsync(p.flags, 0, (size_t)D * 4, e->stream));
    if (split) {
        NYB_CUDA(e, cudaMemsetAsync(p.code, 0, (size_t)D * np, e->stream));
        launch_scatter_splits(e, nv, p.splits, p.nsplits, b.max_splits, D, p.code, p.sbeta, p.flags);   // the multipliers stay unused
    }
    const signed char *code = split ? p.code : nullptr;
    const PackedNet pn = packed(*net);
    // few boxes: a wide CTA shortens the serial chain over the layers; many: smaller ones share an SM
    const dim3 per_box((unsigned)D), box_threads(D < usable_sms(e) ? 512 : 256);
    int zdim = 0;
    for (int k = 0; k <= L; ++k) zdim = nv.dims[k] > zdim ? nv.dims[k] : zdim;
    zdim = (zdim + 1) & ~1;
    NYB_TRY(allow_smem(e, (const void *)k_crown_ibp, (size_t)zdim * 32));
    NYB_TRY(allow_smem(e, (const void *)k_crown_layer, (size_t)zdim * 44));
    NYB_CUDA(e, launch_pdl(k_crown_ibp, per_box, box_threads, (size_t)zdim * 32, e, nv, zdim, (const float *)p.in_lo, (const float *)p.in_hi, (long)box_stride,
                           p.raw_lo, p.raw_hi, p.q, p.zl, p.zu, ibp_lo, ibp_hi, code, p.flags));
    e->launches++;
    for (int k = 0; k < L; ++k) {
        NYB_DEADLINE(e, "plain CROWN");
        const bool pass = k > 0 && k < L - 1;
        if (pass) NYB_TRY(launch_pass(e, pn, k, nv.dims[k + 1], D, nullptr, nv.W[k], nv.b[k], p, box_stride, ptab, c_lo, c_hi, nullptr));
        NYB_CUDA(e, launch_pdl(k_crown_layer, per_box, box_threads, (size_t)zdim * 44, e, nv, k, zdim, (const float *)ibp_lo, (const float *)ibp_hi, (const float *)p.raw_lo,
                               (const float *)p.raw_hi, (const float *)p.q, (const float *)(pass ? c_lo : nullptr), (const float *)(pass ? c_hi : nullptr), p.pre_lo,
                               p.pre_hi, p.zl, p.zu, ptab, code, p.flags, r_il, r_iu));
        e->launches++;
    }
    NYB_TRY(launch_pass(e, pn, L, S, D, nullptr, p.spec, nullptr, p, box_stride, ptab, c_lo, c_hi, p.A0));
    NYB_CUDA(e, launch_pdl(k_crown_spec, dim3((unsigned)((D * 32L + 255) / 256)), dim3(256), 0, e, D, S, nv.dims[L], (const float *)p.spec,
                           (const float *)ibp_lo, (const float *)ibp_hi, (const float *)p.pre_lo, (const float *)p.pre_hi, (long)np,
                           nv.pre_off[L - 1], (const float *)c_lo, (const float *)c_hi, (const int *)p.flags, res, res + n_res, scratch));
    e->launches++;
    NYB_CUDA(e, cudaGetLastError());
    const FetchPiece fp[4] = {{out_lo, n_res * 4}, {out_hi, n_res * 4}, {inter_lo, n_int * 4}, {inter_hi, n_int * 4}};
    NYB_TRY(staged_fetch(e, res, fp, 4));
    if (cs && cs->infeasible) {
        NYB_CUDA(e, cudaMemcpyAsync(cs->infeasible, p.flags, (size_t)D * 4, cudaMemcpyDeviceToHost, e->stream));
        NYB_CUDA(e, cudaStreamSynchronize(e->stream));
        for (int d = 0; d < D; ++d) {
            if (cs->infeasible[d] & kFlagInvalid) return set_err(e, NYB200_ERR_INVALID, "split entry out of range");
            cs->infeasible[d] = (cs->infeasible[d] & kFlagInfeasible) ? 1 : 0;
        }
    }
    e->batch.crown_a = p.A0;
    e->batch.crown_lda = p.lda; e->batch.crown_D = D; e->batch.crown_S = S; e->batch.crown_n0 = nv.dims[0];
    return NYB200_OK;
}

// Is a batch evaluated directly instead of on the tensor path (whose rounding charges its caller would then have to check)?
//
// Fewer than 64 domains: the interval pass of so few is binary64 on either path, so the slopes are the same ones; from 64 on
// they are those of TF32 products, and a batch must not take other lower lines because another form is faster for it (784 ->
// 8x256 -> 10, 9 rows: 390 us directly and 399 on the tensor path at 128 domains, 592 and 415 at 256).
// Below that, time per call directly / on the tensor path in us, 9 rows unless said otherwise, nothing flagged:
//   784->8x256->10     16 domains 240/302   37 246/332   63 252/353       64->9x256->10 63 242/397   784->9x128->10 63 199/280
//   784->9x400->10      4 253/369   16 348/408   37 620/464              784->9x301->10 16 313/425   37 517/469   63 523/521
//   784->9x512->10      4 276/387   16 481/432   37 725/509              1 row: 63 domains 376/600
// So up to 256 columns (a warp's tiles stay in its ring of weights) it is the work of all layers that decides, and the line
// lies where 8e12 multiply-adds a second would take the tensor path's 40 us and 20 more per layer, 147 domains of the first
// network if there were no other limit; wider layers are slower, and their line is the work of the widest one: 5e7 products.
bool direct_pays(const nyb200_engine *e, const Net &net, int S, int D) {
    if (e->path != NYB200_PATH_TF32X3 || !e->small_direct || !e->fuse_chain || D >= 64 || !direct_eligible(net)) return false;
    const NetView &nv = net.v;
    double macs = 0.0, wide = 0.0;
    for (int k = 0; k < nv.L; ++k) {
        macs += (double)nv.dims[k] * nv.dims[k + 1];
        if (k > 0) wide = nv.dims[k] > wide ? (double)nv.dims[k] : wide;
    }
    const double rows = 2.0 * S * D;
    return rows * macs <= 8e12 * (40e-6 + 20e-6 * nv.L) && (wide <= 256.0 || rows * wide * wide <= 5e7);
}

// Interval pass of the n domains idx (null: all b.D) of the resident batch, modes 0 and 1.
int run_forward_direct(nyb200_engine *e, Net &net, const Batch &b, BatchPtrs &p, int mode, const int *idx, int n) {
    const NetView &nv = net.v;
    NYB_DEADLINE(e, "interval pass");
    const bool shared = b.box_stride == 0 && n > 1;   // one image of the shared box serves every domain
    if (shared) launch_ibp_linear(e, nv, 0, 1, p.in_lo, p.in_hi, 0, p.raw_lo, p.raw_hi, p.raw_lo + nv.nps, 0);
    int zdim = 0;
    for (int k = shared ? 1 : 0; k <= nv.L; ++k) zdim = nv.dims[k] > zdim ? nv.dims[k] : zdim;
    zdim = (zdim + 1) & ~1;
    // Few domains: a cluster of CTAs per domain spreads its outputs over the idle SMs, and wide CTAs shorten the serial
    // chain over the layers; many: one small CTA per domain, several to an SM.
    const int sms = usable_sms(e);
    int C = 1;
    while (C < 8 && n * C * 2 <= sms * 7 / 8) C *= 2;   // (clusters live inside a GPC: not every SM can be used)
    const int threads = n * C <= sms ? 512 : 256;
    const size_t smem = (size_t)zdim * (32 + 12) + (size_t)nv.nps * 5;
    NYB_TRY(allow_smem(e, (const void *)k_direct_forward, smem));
    NYB_CUDA(e, launch_pdl_cluster(k_direct_forward, dim3((unsigned)(n * C)), dim3(threads), C, smem, e, nv, mode, zdim, idx,
                           (const float *)p.in_lo, (const float *)p.in_hi, (long)b.box_stride,
                           (const float *)(shared ? p.raw_lo : nullptr), (const float *)p.raw_hi, (const float *)(p.raw_lo + nv.nps),
                           (const float *)p.inh_lo, (const float *)p.inh_hi, (long)b.inh_stride, (const nyb200_split *)p.splits,
                           (const int *)p.nsplits, b.max_splits, (const float *)(b.has_alpha ? p.alpha : nullptr), p.code, p.sbeta, p.pre_lo,
                           p.pre_hi, p.zl, p.zu, p.tab, p.zabs, p.q, p.flags, p.min_lower));
    e->launches++;
    return NYB200_OK;
}

// Backward pass and concretisation of the same domains with the batch's tables as they stand.  The bounds of idx's
// domains are replaced; flags, repair rule and the global minimum are applied to the whole batch.
// ckpt: one block of D x 2S rows (stride p.lda) per ReLU for the coefficients that enter it, or null.
int run_backward_direct(nyb200_engine *e, Net &net, const Batch &b, BatchPtrs &p, const int *idx, int n, float *ckpt) {
    const NetView &nv = net.v;
    NYB_DEADLINE(e, "backward pass");
    NYB_TRY(prepare_fragments(e, net));
    NYB_WS(ptab, PassEntry *, e, "crown_ptab", (size_t)b.D * nv.nps * sizeof(PassEntry));
    const long tot = (long)n * nv.n_pre;
    NYB_CUDA(e, launch_pdl(k_pass_table, dim3((unsigned)((tot + 255) / 256)), dim3(256), 0, e, nv, n, b.box_stride == 0, idx, (const float4 *)p.tab,
                           (const float *)p.zabs, (const float *)p.q, (const float *)(b.external_tables ? nullptr : p.zl),
                           (const float *)(b.external_tables ? nullptr : p.zu), (const float *)p.alpha_up, ptab));
    e->launches++;
    NYB_TRY(launch_pass(e, packed(net), nv.L, b.S, n, idx, p.spec, nullptr, p, b.box_stride, ptab, p.out_lo, p.out_hi,
                        p.keep_final || ckpt ? p.A0 : nullptr, ckpt, (long)b.D * b.R * p.lda));
    p.a_final = p.A0;
    if (idx) launch_fill_f32(e, p.min_lower, 1, INFINITY);
    launch_finalize(e, b.D, b.S, p.flags, p.out_lo, p.out_hi, p.min_lower);
    NYB_CUDA(e, cudaGetLastError());
    return NYB200_OK;
}

namespace {
// Places of the domains whose rounding charge is visible (and that are worth another evaluation), in order; one block.
__global__ void __launch_bounds__(1024) k_flagged(int D, const int *__restrict__ flags, int *__restrict__ idx) {
    __shared__ int s_warp[32];
    __shared__ int s_base;
    if (threadIdx.x == 0) s_base = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int b0 = 0; b0 < D; b0 += 1024) {
        const int d = b0 + threadIdx.x;
        const int f = d < D ? flags[d] : 0;
        const bool take = (f & (kFlagLoose | kFlagLooseFwd)) && !(f & (kFlagInfeasible | kFlagDegraded | kFlagInvalid));
        const unsigned m = __ballot_sync(0xffffffffu, take);
        if (lane == 0) s_warp[warp] = __popc(m);
        __syncthreads();
        int at = s_base + __popc(m & ((1u << lane) - 1u));
        for (int w = 0; w < warp; ++w) at += s_warp[w];
        if (take) idx[at] = d;
        __syncthreads();
        if (threadIdx.x == 0) for (int w = 0; w < 32; ++w) s_base += s_warp[w];
        __syncthreads();
    }
}
}  // namespace

// The n flagged domains of the resident batch as an index list on the device.
int flagged_domains(nyb200_engine *e, int D, const int *flags, int n, int **out) {
    NYB_WS(idx, int *, e, "sub_idx", (size_t)(n > D ? n : D) * 4);
    k_flagged<<<1, 1024, 0, e->stream>>>(D, flags, idx);
    e->launches++;
    *out = idx;
    return NYB200_OK;
}

}  // namespace nyb
