// The per-coefficient step of the beta-CROWN ReLU relaxation pass, shared by the stand-alone relaxation kernels and
// by the fused backward chain so that both produce the same coefficient bits.
#pragma once

namespace nyb {

constexpr float kMinWidth = 1e-8f;   // RELU_RELAX_MIN_WIDTH, relu/mod.rs:24

// One coefficient `a` of a row (`upper`: the row bounds from above) through ReLU's relaxation
// t = (lower slope, upper slope, upper intercept, signed beta), then the charges of the contraction that follows.
// au: the upper path's own lower slope (dual alpha, activations/relu/mod.rs:570-1128); equals t.x otherwise.
// za = max|pre-activation|, qv = |W| max|z| of the next contraction, bk its bias entry, eps its rounding rate.
// Accumulates the row's bias (sb, binary64), bias magnitude (sa) and rounding penalty (sp), both rounded upwards.
// `upper` may be a compile-time constant (the selects fold) or a per-thread value (no divergence either way).
template <bool RELAX, bool BIAS>
__device__ __forceinline__ float relax_coeff(const bool upper, float a, float4 t, float au, float za, float qv, float bk,
                                             float eps, double &sb, float &sa, float &sp) {
    float nw = a;
    if (RELAX) {
        const bool pos = a > 0.f;
        // lower rows: a > 0 takes the lower line (slope ls, no intercept), a < 0 the upper line (us, ui);
        // upper rows mirror it (relu_backward.rs:105-153)
        const float slope = (pos != upper) ? (upper ? au : t.x) : t.y;
        const float icp = ((pos == upper) && a != 0.f) ? t.z : 0.f;
        // the reference's rounding: round to nearest, then one ulp outward (relu_backward.rs:105-153); an exact
        // zero product (a == 0 or slope == 0) needs no step.  A directed product would be up to one ulp tighter,
        // which is visible on bounds that cancel to almost nothing; staying on the reference's values is worth
        // more here than that ulp.
        const float prod = __fmul_rn(a, slope);
        const unsigned pb = __float_as_uint(prod);
        const int neg = (int)pb >> 31;  // 0 or -1: one ulp outward is +-1 on the bit pattern, mirrored for negatives
        const unsigned step = 1u + 2u * (unsigned)neg;
        const float stepped = __uint_as_float(upper ? pb + step : pb - step);
        // a product that underflowed to zero takes the directed product instead (the bit step would wrap); an
        // overflowed one steps into a NaN pattern, which the concretisation turns into [-inf, +inf] for the row
        nw = stepped;
        if (prod == 0.f) nw = upper ? __fmul_ru(a, slope) : __fmul_rd(a, slope);
        nw = (a == 0.f || slope == 0.f) ? 0.f : nw;
        // The step above is outward in the coefficient.  That alone is sound where the variable it multiplies cannot
        // be negative: a neuron that is active on the whole domain (table (1, 1, 0): pre-activation lower bound >= 0,
        // by its interval or by a split).  Everywhere else the pre-activation may be negative and the gap between the
        // exact product and the stepped one is charged against its magnitude.
        const bool nonneg = (t.y == 1.f) && (t.z == 0.f);
        sp = __fmaf_ru(nonneg ? 0.f : fabsf(fmaf(a, slope, -nw)), za, sp);
        sb = fma((double)a, (double)icp, sb);
        sa = __fmaf_ru(fabsf(a), fabsf(icp), sa);
        nw = upper ? nw + t.w : nw - t.w;  // signed beta (zero for unsplit neurons), relu_backward.rs:156-175
    }
    if (BIAS) {
        sb = fma((double)nw, (double)bk, sb);
        sa = __fmaf_ru(fabsf(nw), fabsf(bk), sa);
    }
    sp = __fmaf_ru(__fmul_ru(eps, fabsf(nw)), qv, sp);
    return nw;
}

// What the charges take for a neuron's max|z|.  The intercepts' sums are charged through the coefficients behind them: an intercept
// only applies on the upper line, where |nw| >= |a| slope, and intercept / slope is the chord's -l up to rounding, so that
// |a icp| <= |nw| max|z| (1 + 2^-21).  Where relax_neuron holds the chord's width at 1e-8 the slope is u / 1e-8 and the intercept up to
// u, whatever small value u has: there it is that width.  (The factor covers the roundings of both and of the constant.)
__device__ __forceinline__ float charge_magnitude(float l, float u) {
    const float m = fmaxf(fabsf(l), fabsf(u));
    return l < 0.f && u > 0.f && u - l < kMinWidth ? fmaxf(m, kMinWidth * 1.0000005f) : m;
}

// relax_coeff with its charges prepared per column: zg = max|z| where the outward step is charged (zero where z cannot be
// negative), cj = eps q + 2^-40 (max|z| + |bias|), which bounds the contraction's rounding and (charge_magnitude) that of the
// two binary64 sums.  A zero product stays zero; one that underflowed (at most 2^-150) is covered by a charge of the caller's, kUnderflow
// times the sum of max|z|.
constexpr double kUnderflow = 1e-45;
template <bool UPPER, bool BIAS>
__device__ __forceinline__ float relax_prepared(float a, const float4 &t, float zg, float cj, float bias, double &sb, float &sp) {
    const bool pos = a > 0.f;
    const float slope = (pos != UPPER) ? t.x : t.y;
    const float prod = __fmul_rn(a, slope);
    const int pb = __float_as_int(prod), away = (pb >> 31) | 1;   // a step on the bit pattern away from zero, signed
    float nw = __int_as_float(UPPER ? pb + away : pb - away);     // one ulp up, or down
    if (prod == 0.f) nw = 0.f;
    sp = __fmaf_ru(fabsf(fmaf(a, slope, -nw)), zg, sp);
    if (pos == UPPER) sb = fma((double)a, (double)t.z, sb);
    nw = UPPER ? nw + t.w : nw - t.w;
    if (BIAS) sb = fma((double)nw, (double)bias, sb);
    sp = __fmaf_ru(fabsf(nw), cj, sp);
    return nw;
}

// The same coefficient step for the fused backward chain, with the row sums arranged for issue rate: the coefficient
// bits are those of relax_coeff (same product, same outward step, same beta addition); what differs is the
// bookkeeping around them.
//   * One charge per coefficient, |nw| * cj, with cj prepared once per (domain, column) by the caller:
//         cj = eps * q + (1.6 * 2^-23 + kappa) * max|z| + kappa * |bias|.
//     1.6 * 2^-23 |nw| bounds the gap between the exact product and the stepped one (within 1.5 ulp); it is charged
//     for neurons that cannot be negative as well (at most 3% more than the contraction's own charge).  kappa covers
//     the fp32 accumulation of the two dot products below: a run of n fused multiply-adds errs by at most
//     n * 2^-24 times the run's magnitude sum, and that sum is bounded term by term: |nw bias| directly, and
//     |a * intercept| <= |nw| * max|z| * (1 + 2^-21): see charge_magnitude.
//     A product that underflows to zero stays zero; the floor of the charge encloses it.
//   * The intercept and bias dot products are accumulated in fp32 (gi, gb: one fused multiply-add per term) over a
//     short run of columns; the caller adds each run to the row's binary64 bias.
// dir = +1 for an upper row, -1 for a lower row; dirf the same as a float.
__device__ __forceinline__ float relax_coeff_fast(const bool upper, const int dir, const float dirf, float a, float4 t, float au,
                                                  float cj, float bk, float &gi, float &gb, float &sp) {
    const bool pos = a > 0.f;
    const float slope = (pos != upper) ? (upper ? au : t.x) : t.y;
    const float icp = (pos == upper) ? t.z : 0.f;   // times a == 0 it adds nothing
    const float prod = __fmul_rn(a, slope);
    const int pb = __float_as_int(prod);
    // one ulp outward on the bit pattern: +dir for a positive product, -dir for a negative one; a zero product (zero
    // slope or zero coefficient: common, every stably inactive neuron has one) stays zero without a branch
    // A zero product stays zero: exactly zero when the coefficient or the slope is zero (no step: every stably inactive
    // neuron has one); a product that underflowed (|a * slope| <= 2^-150) is enclosed by the floor of the charge below.
    float nw = __int_as_float((pb << 1) ? pb + dir + 2 * dir * (pb >> 31) : 0);
    gi = fmaf(a, icp, gi);
    nw = fmaf(t.w, dirf, nw);   // signed beta: nw + t.w on upper rows, nw - t.w on lower rows (t.w * +-1 is exact)
    gb = fmaf(nw, bk, gb);
    // the floor covers the underflow case, where the coefficient is taken as zero and the exact product is at most
    // 2^-150: 2^-148 max|z| <= 1.6e-38 cj because cj >= 1.9e-7 max|z| (and cj >= kappa |bias| for the bias product)
    sp = __fmaf_ru(fmaxf(fabsf(nw), 1.6e-38f), cj, sp);
    return nw;
}

// A neuron's bounds from its interval image: what k_ibp_finish does once the image is known, shared with the direct
// interval pass.  mode 0: bounds = inherited (clamp only: beta_crown/engine/domain/child.rs:51-118); mode 1: image
// intersected with inherited (graph/propagation/constraints/mod.rs:738-741); others: the image.  Then the split clamp
// (constraints/lookups.rs:160-175), the beta-CROWN relaxation (beta_crown/engine/backward/relu_backward.rs:63-101) and
// the post-activation interval (:428-548).
__device__ __forceinline__ void inherit_bounds(int mode, const float *inh_lo, const float *inh_hi, long io, float &l, float &u) {
    if (!inh_lo) return;
    if (mode == 0) { l = inh_lo[io]; u = inh_hi[io]; }
    else if (mode == 1) {
        const float il = inh_lo[io], iu = inh_hi[io];
        if (!(isnan(l) || isnan(u) || isnan(il) || isnan(iu))) {
            const float tl = fmaxf(l, il), tu = fminf(u, iu);
            if (tl <= tu) { l = tl; u = tu; } else { l = fminf(l, il); u = fmaxf(u, iu); }
        }
    }
}

// s: split code; l, u: clamped in place; t: relaxation table entry (slopes, intercept; the multiplier is the caller's);
// pl, pu: post-activation interval.  Returns the domain flags it raises.
__device__ __forceinline__ int relax_neuron(int s, const float *alpha, long o, float &l, float &u, float4 &t, float &pl, float &pu) {
    int flag = 0;
    if (s > 0) l = (isnan(l)) ? l : fmaxf(l, 0.f);
    else if (s < 0) u = (isnan(u)) ? u : fminf(u, 0.f);
    if (s != 0 && l > u) flag |= kFlagInfeasible;
    float ls, us, ui;
    if (s > 0) { ls = 1.f; us = 1.f; ui = 0.f; }
    else if (s < 0) { ls = 0.f; us = 0.f; ui = 0.f; }
    else if (isnan(l) || isnan(u) || isinf(l) || isinf(u)) {
        // The reference has closed forms for these arms (relu_backward.rs:75-93); a domain that reaches
        // them is returned as [-inf, +inf] here, which every one of those arms also implies or encloses.
        flag |= kFlagDegraded;
        ls = 0.f; us = 0.f; ui = 0.f;
    } else if (l >= 0.f) { ls = 1.f; us = 1.f; ui = 0.f; }
    else if (u <= 0.f) { ls = 0.f; us = 0.f; ui = 0.f; }
    else {
        float w = fmaxf(u - l, kMinWidth);
        us = __fdiv_rn(u, w);
        // The reference uses ui = -l*u/w in round-to-nearest.  The chord is only a valid upper line if
        // us*l + ui >= 0 and us*u + ui >= u, so the intercept is taken as the smallest fp32 that
        // provably satisfies both; it differs from the reference value by at most a few ulps.
        float i1 = __fmul_ru(us, -l);
        float i2 = __fsub_ru(u, __fmul_rd(us, u));
        ui = fmaxf(fmaxf(i1, i2), 0.f);
        if (alpha) { float a = alpha[o]; ls = isnan(a) ? 0.f : fminf(fmaxf(a, 0.f), 1.f); }
        else ls = (u > -l) ? 1.f : 0.f;  // beta_crown/state/alpha/domain.rs:161
    }
    t.x = ls; t.y = us; t.z = ui;
    pl = fmaxf(l, 0.f); pu = fmaxf(u, 0.f);
    if (s > 0) { pu = u; }
    else if (s < 0) { pl = 0.f; pu = 0.f; }
    if (isnan(l)) pl = l;
    if (isnan(u)) pu = u;
    return flag;
}

}  // namespace nyb
