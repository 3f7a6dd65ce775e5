// PGD attack batched over restarts: concrete forward pass, exact gradient of the worst specification row and
// the AdamClipping step, all K restarts in lock-step on the device.
//
// The forward products Z * W_k^T and the backward products G * W_k run on the same contraction kernels as the
// bound propagation (tcgen05 3xTF32, or binary64 when that path is selected); convolutions use the plain
// forward convolution and the transposed-convolution path.  The attack only proposes points: the value
// returned for each restart comes from a final evaluation of its best point with binary64 contractions.
#include <cmath>

#include "nyb200_internal.cuh"

namespace nyb {

namespace {

struct PgdStep {
    float step, beta1, beta2, epsilon, bc2;
};

// The element-wise kernels.  Large launches: one row a grid row, four columns a thread where the row allows it (VEC); an index
// division per element and one column a thread held them to a third of the copy rate (bias and ReLU of 1024 x 4096: 15.4 -> 7
// us).  Small ones, a few hundred values an SM, take one value a thread and few blocks, rows one behind the other: 16 restarts x 40
// steps on 30 -> 4x60 -> 10, some 25 launches a step, 3.88 ms by rows, 3.82 so; on 784 -> 4x256 -> 10 6.04 and 5.97; 64 restarts on the
// convolutional classifier of side 28 4.76 and 4.70.
#define NYB_ROWS(rows, n, vec) (vec) ? dim3((unsigned)(((n) + 1023) / 1024), (unsigned)(rows)) : dim3((unsigned)(((long)(rows) * (n) + 255) / 256)), 256
template <class F>
__device__ __forceinline__ void over_rows(int rows, int n, bool vec, F f) {   // f(row, column, columns from there: 4 or 1)
    if (vec) {
        const int j = (blockIdx.x * 256 + threadIdx.x) * 4;
        if (j < n) f((int)blockIdx.y, j, 4);
    } else {
        const unsigned t = blockIdx.x * 256 + threadIdx.x, r = t / (unsigned)n;
        if (t < (unsigned)rows * (unsigned)n) f((int)r, (int)(t - r * n), 1);
    }
}
static int rows_most(int n) { return std::min(65535, 0x7fffffff / n); }   // of one launch: grid, 32-bit index
static bool vec4(int rows, int n, long ld, const void *a, const void *b = nullptr, const void *c = nullptr, const void *d = nullptr) {
    return (long)rows * n >= 65536 && n % 4 == 0 && ld % 4 == 0 &&
           ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(c) | reinterpret_cast<uintptr_t>(d)) & 15) == 0;
}

// z += bias; optionally ReLU.  Post-activations are kept: z > 0 afterwards is exactly the gradient mask.
__global__ void __launch_bounds__(256) k_bias_act(int rows, int n, float *__restrict__ Z, long ld, const float *__restrict__ bias, int relu, bool vec) {
    auto one = [&](float x, float b) { const float v = x + b; return relu ? fmaxf(v, 0.f) : v; };
    over_rows(rows, n, vec, [&](int r, int j, int w) {
        float *z = Z + (long)r * ld + j;
        if (w == 4) {
            float4 x = *(float4 *)z;
            const float4 b = bias ? *(const float4 *)(bias + j) : make_float4(0.f, 0.f, 0.f, 0.f);
            *(float4 *)z = make_float4(one(x.x, b.x), one(x.y, b.y), one(x.z, b.z), one(x.w, b.w));
        } else *z = one(*z, bias ? bias[j] : 0.f);
    });
}

// Per restart: margins spec[s] . y, the smallest one and its row.  `track`: the step's point competes for the
// restart's best objective (improved[r] tells k_keep_best to copy the point).  `seed`: G[r] = spec[row].
__global__ void __launch_bounds__(256) k_pgd_objective(int K, int S, int nL, const float *__restrict__ Y, int ldy, const float *__restrict__ spec,
                                float *__restrict__ best, int *__restrict__ improved, float *__restrict__ G, int ldg,
                                float *__restrict__ value_out) {
    // one warp per restart, a lane per specification row (one thread per restart was a chain of S * nL loads: 17.7 us for 1024)
    const int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (r >= K) return;
    const float *y = Y + (long)r * ldy;
    float mv = INFINITY;
    int ms = 0;
    bool bad = false;
    for (int s = lane; s < S; s += 32) {
        double acc = 0.0;
        for (int j = 0; j < nL; ++j) acc = fma((double)spec[s * nL + j], (double)y[j], acc);
        float m = (float)acc;
        if (isnan(m)) bad = true;
        if (m < mv) { mv = m; ms = s; }
    }
    for (int o = 16; o > 0; o >>= 1) {   // the smallest margin, the first row that has it
        const float om = __shfl_xor_sync(0xffffffffu, mv, o);
        const int os = __shfl_xor_sync(0xffffffffu, ms, o);
        if (om < mv || (om == mv && om < INFINITY && os < ms)) { mv = om; ms = os; }
    }
    ms = mv < INFINITY ? ms : 0;
    bad = __any_sync(0xffffffffu, bad);
    if (bad) mv = NAN;
    if (lane == 0) {
        if (value_out) value_out[r] = mv;
        if (best) {
            int imp = (!bad && mv < best[r]) ? 1 : 0;
            if (imp) best[r] = mv;
            improved[r] = imp;
        }
    }
    if (G)
        for (int j = lane; j < nL; j += 32) G[(long)r * ldg + j] = spec[ms * nL + j];
}

__global__ void __launch_bounds__(256) k_keep_best(int rows, int n0, const float *__restrict__ X, long ldx, const int *__restrict__ improved, float *__restrict__ best_x, bool vec) {
    over_rows(rows, n0, vec, [&](int r, int j, int w) {
        if (!improved[r]) return;
        const float *x = X + (long)r * ldx + j;
        float *b = best_x + (long)r * n0 + j;
        if (w == 4) *(float4 *)b = *(const float4 *)x; else *b = *x;
    });
}

// G *= [Zpost > 0]
__global__ void __launch_bounds__(256) k_relu_mask(int rows, int n, float *__restrict__ G, long ld, const float *__restrict__ Z, bool vec) {
    over_rows(rows, n, vec, [&](int r, int j, int w) {
        float *g = G + (long)r * ld + j;
        const float *z = Z + (long)r * ld + j;
        if (w == 4) {
            float4 v = *(float4 *)g;
            const float4 m = *(const float4 *)z;
            *(float4 *)g = make_float4(m.x > 0.f ? v.x : 0.f, m.y > 0.f ? v.y : 0.f, m.z > 0.f ? v.z : 0.f, m.w > 0.f ? v.w : 0.f);
        } else if (!(*z > 0.f)) *g = 0.f;
    });
}

// AdamClipping step (pgd_attack/adam_state.rs:46-88), descending the objective.  A restart whose gradient
// holds a NaN skips the step (attacker/batched.rs:93-104): rows flagged in nan_row are left alone.  x_max (optional, cleared by
// k_nan_rows): the stepped rows' largest magnitudes (bits), for the first convolution's split.
__global__ void __launch_bounds__(256) k_pgd_step(int rows, int n0, float *__restrict__ X, long ld, const float *__restrict__ G,
                           float *__restrict__ mom, float *__restrict__ var, const float *__restrict__ lo,
                           const float *__restrict__ hi, const int *__restrict__ nan_row, unsigned *__restrict__ x_max, PgdStep h, bool vec) {
    float most = 0.f;
    int row = -1;
    auto one = [&](float g, float &m, float &v, float &x, float l, float u) {
        m = h.beta1 * m + (1.f - h.beta1) * g;
        v = h.beta2 * v + (1.f - h.beta2) * g * g;
        float denom = sqrtf(v / h.bc2) + h.epsilon;
        float dir = 0.f;
        if (isfinite(denom) && isfinite(m)) {
            float q = m / denom;
            dir = isnan(q) ? 0.f : copysignf(1.f, q);  // sign(+0) = +1, sign(-0) = -1
        }
        x = x - dir * h.step;
        x = isnan(x) ? l : fminf(fmaxf(x, l), u);
        most = fmaxf(most, fabsf(x));
    };
    over_rows(rows, n0, vec, [&](int r, int j, int w) {
        if (nan_row[r]) return;
        row = r;
        float *x_at = X + (long)r * ld + j, *m_at = mom + (long)r * n0 + j, *v_at = var + (long)r * n0 + j;
        const float *g_at = G + (long)r * ld + j;
        if (w == 4) {
            const float4 g = *(const float4 *)g_at, l = *(const float4 *)(lo + j), u = *(const float4 *)(hi + j);
            float4 m = *(float4 *)m_at, v = *(float4 *)v_at, x = *(float4 *)x_at;
            one(g.x, m.x, v.x, x.x, l.x, u.x); one(g.y, m.y, v.y, x.y, l.y, u.y); one(g.z, m.z, v.z, x.z, l.z, u.z); one(g.w, m.w, v.w, x.w, l.w, u.w);
            *(float4 *)m_at = m; *(float4 *)v_at = v; *(float4 *)x_at = x;
        } else one(*g_at, *m_at, *v_at, *x_at, lo[j], hi[j]);
    });
    if (x_max) {   // (a warp may span rows, and lanes of it have none)
        const int first = __shfl_sync(0xffffffffu, row, 0);
        if (__all_sync(0xffffffffu, row == first)) {
            const unsigned w = __reduce_max_sync(0xffffffffu, __float_as_uint(most));
            if ((threadIdx.x & 31) == 0 && w) atomicMax(x_max + first, w);
        } else if (most > 0.f) atomicMax(x_max + row, __float_as_uint(most));
    }
}

__global__ void __launch_bounds__(256) k_nan_rows(int n0, const float *__restrict__ G, long ld, int *__restrict__ nan_row, unsigned *__restrict__ x_max) {
    const float *g = G + (long)blockIdx.x * ld;
    int bad = 0;
    for (int j = threadIdx.x; j < n0; j += 256) bad |= isnan(g[j]) ? 1 : 0;
    bad = __syncthreads_or(bad);
    if (threadIdx.x == 0) {
        nan_row[blockIdx.x] = bad;
        if (x_max && !bad) x_max[blockIdx.x] = 0;   // (a row that is not stepped keeps its own)
    }
}

// Y[r, j] += X[r, j]
__global__ void k_add_rows(long rows, int n, float *__restrict__ Y, int ldy, const float *__restrict__ X, int ldx) {
    long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= rows * n) return;
    long r = t / n;
    int j = (int)(t - r * n);
    Y[r * ldy + j] += X[r * ldx + j];
}

// out[r] = X[r, :] . Y[r, :], one warp per row, binary64 accumulation
__global__ void k_row_dot(int rows, int n, const float *__restrict__ X, int ldx, const float *__restrict__ Y, int ldy,
                          float *__restrict__ out) {
    int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (warp >= rows) return;
    double acc = 0.0;
    for (int j = lane; j < n; j += 32) acc = fma((double)X[(long)warp * ldx + j], (double)Y[(long)warp * ldy + j], acc);
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) out[warp] = (float)acc;
}

__global__ void k_fill_f32(float *p, long n, float v) {
    long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) p[t] = v;
}

}  // namespace

// Concrete forward pass of `rows` points X [rows x ldx] through the network; act[k] receives layer k's
// post-activation output (row stride ld), act[L-1] the network output.
static int pgd_forward(nyb200_engine *e, Net &net, bool tensor, int rows, const float *X, int ldx, float *const *act, int ld,
                       int *derr, const unsigned *x_rows = nullptr) {
    const NetView &nv = net.v;
    const float *cur = X;
    int ldc = ldx;
    bool pending = false;   // cur is a convolution's result without its bias and ReLU: the next one's split adds them
    for (int k = 0; k < nv.L; ++k) {
        int K = nv.dims[k], N = nv.dims[k + 1];
        // (a layer that is alone between two window convolutions: its row maxima come with the products)
        const bool defer = tensor && k + 1 < nv.L && net.is_conv(k) && net.win_fwd[k].ok && net.skip_of(k) < 0 && net.is_conv(k + 1) && net.win_fwd[k + 1].ok && nv.b[k];
        if (net.is_conv(k) && tensor && net.win_fwd[k].ok) {
            WinWith with;
            if (pending) {
                with.bias = nv.b[k - 1]; with.bias_max = net.bmax[k - 1]; with.keep = act[k - 1]; with.keep_ld = ld;
                with.has_max = true;
            } else if (k == 0 && x_rows) {   // the points' maxima are known
                void *hi, *lo;
                float *row_inv;
                unsigned *row_max;
                NYB_TRY(win_operand(e, net.win_fwd[0], rows, &hi, &lo, &row_inv, &row_max));
                NYB_CUDA(e, cudaMemcpyAsync(row_max, x_rows, (size_t)rows * 4, cudaMemcpyDeviceToDevice, e->stream));
                with.has_max = true;
            }
            NYB_TRY(conv_win(e, net.win_fwd[k], rows, cur, ldc, act[k], ld, nullptr, nullptr, 1, derr, false, defer, &with));
        } else if (net.is_conv(k) && tensor) NYB_TRY(conv_forward_tensor(e, net, k, rows, cur, ldc, act[k], ld, derr));
        else if (net.is_conv(k)) launch_conv_plain(e, net.geom[k], rows, cur, ldc, nv.W[k], act[k], ld);
        else if (tensor) NYB_TRY(launch_umma(e, net.umma_adj[k], rows, cur, ldc, act[k], ld, derr));
        else launch_gemm_f64(e, rows, N, K, cur, ldc, net.wt[k], N, act[k], ld, 1, nullptr, nullptr, 0, nullptr);
        pending = defer;
        if (net.skip_of(k) >= 0) {  // residual: the block's input joins before the bias and the ReLU
            long tot = (long)rows * N;
            k_add_rows<<<(unsigned)((tot + 255) / 256), 256, 0, e->stream>>>(rows, N, act[k], ld, act[net.skip_of(k)], ld);
            e->launches++;
        }
        if (!pending)
            for (int r0 = 0, most = rows_most(N); r0 < rows; r0 += most) {
                const int n = std::min(rows - r0, most);
                const bool vec = vec4(n, N, ld, act[k], nv.b[k]);
                k_bias_act<<<NYB_ROWS(n, N, vec), 0, e->stream>>>(n, N, act[k] + (size_t)r0 * ld, ld, nv.b[k], k < nv.L - 1 ? 1 : 0, vec);
                e->launches++;
            }
        cur = act[k];
        ldc = ld;
    }
    return NYB200_OK;
}

// Exact gradient chain of K rows: G_k = (G_{k+1} . [mask_k > 0]) W_k from the output down to the input, where
// mask_k is act[k] (a concrete forward pass's activations, or caller-supplied 0/1 masks).  G0 holds the output
// cotangents on entry; *result points at the buffer (G0 or G1) that holds the input gradients.
static int pgd_backward(nyb200_engine *e, Net &net, bool tensor, int K, float *G0, float *G1, float *const *act, int ld,
                        int *derr, float **result) {
    const NetView &nv = net.v;
    const int L = nv.L;
    cudaStream_t st = e->stream;
    double *cols64 = nullptr;
    float *g = G0, *gn = G1;
    bool reported = false;   // the rows' maxima came with the products that left g
    struct OpenGrad { float *buf; int src; };   // gradients kept for identity branches (blocks may nest)
    std::vector<OpenGrad> open_grad;
    auto grad_slot = [&](size_t slot) -> float * {
        const std::string name = slot == 0 ? std::string("pgd_skip") : "pgd_skip_" + std::to_string(slot);
        return (float *)ws_get(e, name.c_str(), (size_t)K * ld * 4);
    };
    for (int k = L - 1; k >= 0; --k) {
        int Kd = nv.dims[k + 1], N = nv.dims[k];
        for (size_t oi = 0; oi < open_grad.size();) {  // g is the gradient of relu(pre_k): identity branches join here
            if (open_grad[oi].src != k) { ++oi; continue; }
            long tot = (long)K * Kd;
            k_add_rows<<<(unsigned)((tot + 255) / 256), 256, 0, st>>>(K, Kd, g, ld, open_grad[oi].buf, ld);
            e->launches++;
            open_grad.erase(open_grad.begin() + (long)oi);
        }
        // a window convolution's split masks its rows itself where nothing else reads them
        const bool window = net.is_conv(k) && tensor && net.win_bwd[k].ok, masks = k < L - 1 && window && net.skip_of(k) < 0;
        if (k < L - 1 && !masks)
            for (int r0 = 0, most = rows_most(Kd); r0 < K; r0 += most) {
                const int n = std::min(K - r0, most);
                const bool vec = vec4(n, Kd, ld, g, act[k]);
                k_relu_mask<<<NYB_ROWS(n, Kd, vec), 0, st>>>(n, Kd, g + (size_t)r0 * ld, ld, act[k] + (size_t)r0 * ld, vec);
                e->launches++;
            }
        if (net.skip_of(k) >= 0) {  // the gradient of pre_k also reaches relu(pre_j) directly
            size_t slot = 0;
            for (bool taken = true; taken; ) {
                taken = false;
                for (const OpenGrad &o : open_grad) if (o.buf == grad_slot(slot)) { taken = true; ++slot; break; }
            }
            float *gstash = grad_slot(slot);
            if (!gstash) return NYB200_ERR_OOM;
            NYB_CUDA(e, cudaMemcpyAsync(gstash, g, (size_t)K * ld * 4, cudaMemcpyDeviceToDevice, st));
            open_grad.push_back({gstash, net.skip_of(k)});
        }
        if (window) {
            WinWith with;
            if (masks) { with.mask = act[k]; with.mask_ld = ld; }
            with.has_max = reported;
            // does the next layer's split want this result's maxima?  (an identity branch that joins in between changes them)
            reported = k > 0 && net.is_conv(k - 1) && net.win_bwd[k - 1].ok;
            for (const OpenGrad &o : open_grad) if (o.src == k - 1) reported = false;
            NYB_TRY(conv_win(e, net.win_bwd[k], K, g, ld, gn, ld, nullptr, nullptr, 1, derr, false, reported, &with));
        } else if (net.is_conv(k) && tensor) {
            const ConvGeom &cg = net.geom[k];
            const int plane = cg.oh * cg.ow, taps = cg.ic * cg.kh * cg.kw;
            float *cols = (float *)ws_get(e, "conv_cols", (size_t)K * plane * taps * 4);
            if (!cols) return NYB200_ERR_OOM;
            NYB_TRY(launch_umma(e, net.umma[k], K * plane, g, ld, cols, taps, derr, plane));
            launch_col2im(e, cg, K, cols, gn, ld);
        } else if (net.is_conv(k)) {
            const ConvGeom &cg = net.geom[k];
            cols64 = (double *)ws_get(e, "conv_cols", (size_t)K * cg.oh * cg.ow * cg.ic * cg.kh * cg.kw * 8);
            if (!cols64) return NYB200_ERR_OOM;
            launch_conv_transpose(e, cg, K, g, ld, gn, ld, nv.W[k], 1, nullptr, nullptr, 0, nullptr, cols64);
        } else if (tensor) {
            NYB_TRY(launch_umma(e, net.umma[k], K, g, ld, gn, ld, derr));
        } else {
            launch_gemm_f64(e, K, N, Kd, g, ld, nv.W[k], N, gn, ld, 1, nullptr, nullptr, 0, nullptr);
        }
        if (!window) reported = false;
        float *tmp = g; g = gn; gn = tmp;
    }
    *result = g;
    return NYB200_OK;
}

int pgd_attack(nyb200_engine *e, int net_id, const float *spec, int S, const float *in_lo, const float *in_hi,
               const float *x0, int K, const nyb200_pgd_config &cfg, float *best_margin, float *best_x, int *counterexample) {
    Net *net;
    NYB_TRY(find_net(e, net_id, &net));
    const NetView &nv = net->v;
    if (S <= 0 || K <= 0) return set_err(e, NYB200_ERR_SHAPE, "S and K must be positive");
    if (cfg.steps < 0 || !(cfg.step_size >= 0.f)) return set_err(e, NYB200_ERR_INVALID, "steps and step_size must be >= 0");
    const int L = nv.L, n0 = nv.dims[0], nL = nv.dims[L];
    const bool tensor = e->path == NYB200_PATH_TF32X3;
    const float b1 = cfg.beta1 > 0.f ? cfg.beta1 : 0.9f, b2 = cfg.beta2 > 0.f ? cfg.beta2 : 0.999f;
    const float eps = cfg.epsilon > 0.f ? cfg.epsilon : 1e-8f, decay = cfg.lr_decay > 0.f ? cfg.lr_decay : 0.99f;
    const int ld = (net->max_dim + 7) & ~7;
    e->batch = Batch();  // workspace names are shared with the resident batch

    NYB_TRY(prepare_transposed(e, *net, tensor));
    if (tensor) NYB_TRY(prepare_backward_operands(e, *net, false));
    NYB_WS(dspec, float *, e, "spec", (size_t)S * nL * 4);
    NYB_WS(dlo, float *, e, "in_lo", (size_t)n0 * 4);
    NYB_WS(dhi, float *, e, "in_hi", (size_t)n0 * 4);
    NYB_WS(X, float *, e, "pgd_x", (size_t)K * ld * 4);
    NYB_WS(acts, float *, e, "pgd_act", (size_t)L * K * ld * 4);
    NYB_WS(G0, float *, e, "pgd_g0", (size_t)K * ld * 4);
    NYB_WS(G1, float *, e, "pgd_g1", (size_t)K * ld * 4);
    NYB_WS(mom, float *, e, "pgd_m", (size_t)K * n0 * 4);
    NYB_WS(var, float *, e, "pgd_v", (size_t)K * n0 * 4);
    NYB_WS(dbest, float *, e, "pgd_best", (size_t)K * 4);
    NYB_WS(dbx, float *, e, "pgd_best_x", (size_t)K * n0 * 4);
    NYB_WS(dimp, int *, e, "pgd_improved", (size_t)K * 4);
    NYB_WS(dnan, int *, e, "pgd_nan", (size_t)K * 4);
    int *derr = nullptr;
    if (tensor) {
        derr = (int *)ws_get(e, "umma_err", 256);
        if (!derr) return NYB200_ERR_OOM;
        NYB_CUDA(e, cudaMemsetAsync(derr, 0, 4, e->stream));
    }
    std::vector<float *> act((size_t)L);
    for (int k = 0; k < L; ++k) act[k] = acts + (size_t)k * K * ld;
    cudaStream_t st = e->stream;
    NYB_CUDA(e, cudaMemcpyAsync(dspec, spec, (size_t)S * nL * 4, cudaMemcpyHostToDevice, st));
    NYB_CUDA(e, cudaMemcpyAsync(dlo, in_lo, (size_t)n0 * 4, cudaMemcpyHostToDevice, st));
    NYB_CUDA(e, cudaMemcpyAsync(dhi, in_hi, (size_t)n0 * 4, cudaMemcpyHostToDevice, st));
    NYB_CUDA(e, cudaMemcpy2DAsync(X, (size_t)ld * 4, x0, (size_t)n0 * 4, (size_t)n0 * 4, (size_t)K, cudaMemcpyHostToDevice, st));
    NYB_CUDA(e, cudaMemcpy2DAsync(dbx, (size_t)n0 * 4, x0, (size_t)n0 * 4, (size_t)n0 * 4, (size_t)K, cudaMemcpyHostToDevice, st));
    NYB_CUDA(e, cudaMemsetAsync(mom, 0, (size_t)K * n0 * 4, st));
    NYB_CUDA(e, cudaMemsetAsync(var, 0, (size_t)K * n0 * 4, st));
    k_fill_f32<<<(K + 255) / 256, 256, 0, st>>>(dbest, K, INFINITY);
    e->launches++;
    const unsigned gw = (unsigned)(((long)K * 32 + 255) / 256);
    // The points' largest magnitudes, kept up to date by the steps.
    unsigned *x_rows = nullptr;
    if (tensor && net->is_conv(0) && net->win_fwd[0].ok) {
        x_rows = (unsigned *)ws_get(e, "pgd_xmax", (size_t)K * 4);
        if (!x_rows) return NYB200_ERR_OOM;
        NYB_TRY(row_maxima(e, K, n0, X, ld, x_rows));
    }

    for (int t = 1; t <= cfg.steps + 1; ++t) {
        NYB_DEADLINE(e, "attack");
        NYB_TRY(pgd_forward(e, *net, tensor, K, X, ld, act.data(), ld, derr, x_rows));
        const bool last = t == cfg.steps + 1;
        k_pgd_objective<<<gw, 256, 0, st>>>(K, S, nL, act[L - 1], ld, dspec, dbest, dimp, last ? nullptr : G0, ld, nullptr);
        for (int r0 = 0, most = rows_most(n0); r0 < K; r0 += most) {
            const int n = std::min(K - r0, most);
            const bool vec = vec4(n, n0, ld, X, dbx);
            k_keep_best<<<NYB_ROWS(n, n0, vec), 0, st>>>(n, n0, X + (size_t)r0 * ld, ld, dimp + r0, dbx + (size_t)r0 * n0, vec);
        }
        e->launches += 2;
        if (last) break;
        float *g = nullptr;
        NYB_TRY(pgd_backward(e, *net, tensor, K, G0, G1, act.data(), ld, derr, &g));
        k_nan_rows<<<(unsigned)K, 256, 0, st>>>(n0, g, ld, dnan, x_rows);
        PgdStep h;
        float bc1 = 1.f - powf(b1, (float)t);
        h.bc2 = 1.f - powf(b2, (float)t);
        h.step = cfg.step_size * powf(decay, (float)(t - 1)) / bc1;
        h.beta1 = b1; h.beta2 = b2; h.epsilon = eps;
        for (int r0 = 0, most = rows_most(n0); r0 < K; r0 += most) {
            const int n = std::min(K - r0, most);
            const bool vec = vec4(n, n0, ld, X, g, mom, var) && vec4(n, n0, ld, dlo, dhi);
            k_pgd_step<<<NYB_ROWS(n, n0, vec), 0, st>>>(n, n0, X + (size_t)r0 * ld, ld, g + (size_t)r0 * ld, mom + (size_t)r0 * n0, var + (size_t)r0 * n0, dlo, dhi,
                                                        dnan + r0, x_rows ? x_rows + r0 : nullptr, h, vec);
        }
        e->launches += 2;
    }
    // independent evaluation of every restart's best point with binary64 contractions
    NYB_TRY(prepare_transposed(e, *net, false));
    NYB_TRY(pgd_forward(e, *net, false, K, dbx, n0, act.data(), ld, derr));
    k_pgd_objective<<<gw, 256, 0, st>>>(K, S, nL, act[L - 1], ld, dspec, nullptr, nullptr, nullptr, 0, dbest);
    e->launches++;
    NYB_CUDA(e, cudaGetLastError());
    NYB_CUDA(e, cudaMemcpyAsync(best_margin, dbest, (size_t)K * 4, cudaMemcpyDeviceToHost, st));
    if (best_x) NYB_CUDA(e, cudaMemcpyAsync(best_x, dbx, (size_t)K * n0 * 4, cudaMemcpyDeviceToHost, st));
    int herr = 0;
    if (derr) NYB_CUDA(e, cudaMemcpyAsync(&herr, derr, 4, cudaMemcpyDeviceToHost, st));
    NYB_CUDA(e, cudaStreamSynchronize(st));
    if (herr) return set_err(e, NYB200_ERR_INTERNAL, "tcgen05 pipeline wait expired (code " + std::to_string(herr) + ")");
    int arg = -1;
    float mv = INFINITY;
    for (int r = 0; r < K; ++r)
        if (best_margin[r] < mv) { mv = best_margin[r]; arg = r; }
    if (counterexample) *counterexample = (arg >= 0 && mv <= 0.f) ? arg : -1;
    return NYB200_OK;
}


// Exact point gradients of K restarts: spec_rows[k] . df/dx, ReLU derivatives from the forward pass at x or from
// caller-supplied masks.
int point_vjp(nyb200_engine *e, int net_id, int K, const float *x, const float *masks, const float *spec_rows, float *grads,
              float *values) {
    Net *net;
    NYB_TRY(find_net(e, net_id, &net));
    const NetView &nv = net->v;
    if (K <= 0) return set_err(e, NYB200_ERR_SHAPE, "K must be positive");
    if ((x != nullptr) == (masks != nullptr)) return set_err(e, NYB200_ERR_INVALID, "exactly one of x and masks must be given");
    if (values && !x) return set_err(e, NYB200_ERR_INVALID, "values need the points x");
    const int L = nv.L, n0 = nv.dims[0], nL = nv.dims[L];
    const bool tensor = e->path == NYB200_PATH_TF32X3;
    const int ld = (net->max_dim + 7) & ~7;
    e->batch = Batch();  // workspace names are shared with the resident batch
    NYB_TRY(prepare_transposed(e, *net, tensor));
    if (tensor) NYB_TRY(prepare_backward_operands(e, *net, false));
    NYB_WS(X, float *, e, "pgd_x", (size_t)K * ld * 4);
    NYB_WS(acts, float *, e, "pgd_act", (size_t)L * K * ld * 4);
    NYB_WS(G0, float *, e, "pgd_g0", (size_t)K * ld * 4);
    NYB_WS(G1, float *, e, "pgd_g1", (size_t)K * ld * 4);
    NYB_WS(dval, float *, e, "pgd_best", (size_t)K * 4);
    int *derr = nullptr;
    if (tensor) {
        derr = (int *)ws_get(e, "umma_err", 256);
        if (!derr) return NYB200_ERR_OOM;
        NYB_CUDA(e, cudaMemsetAsync(derr, 0, 4, e->stream));
    }
    std::vector<float *> act((size_t)L);
    for (int k = 0; k < L; ++k) act[k] = acts + (size_t)k * K * ld;
    cudaStream_t st = e->stream;
    NYB_CUDA(e, cudaMemcpy2DAsync(G0, (size_t)ld * 4, spec_rows, (size_t)nL * 4, (size_t)nL * 4, (size_t)K, cudaMemcpyHostToDevice, st));
    if (x) {
        NYB_CUDA(e, cudaMemcpy2DAsync(X, (size_t)ld * 4, x, (size_t)n0 * 4, (size_t)n0 * 4, (size_t)K, cudaMemcpyHostToDevice, st));
        NYB_TRY(pgd_forward(e, *net, tensor, K, X, ld, act.data(), ld, derr));
        if (values) {
            k_row_dot<<<(unsigned)(((long)K * 32 + 255) / 256), 256, 0, st>>>(K, nL, act[L - 1], ld, G0, ld, dval);
            e->launches++;
        }
    } else {
        for (int k = 0; k < L - 1; ++k)  // layer k's mask block of every restart's [n_pre] row
            NYB_CUDA(e, cudaMemcpy2DAsync(act[k], (size_t)ld * 4, masks + nv.pre_off[k], (size_t)nv.n_pre * 4,
                                          (size_t)nv.dims[k + 1] * 4, (size_t)K, cudaMemcpyHostToDevice, st));
    }
    float *g = nullptr;
    NYB_TRY(pgd_backward(e, *net, tensor, K, G0, G1, act.data(), ld, derr, &g));
    NYB_CUDA(e, cudaGetLastError());
    NYB_CUDA(e, cudaMemcpy2DAsync(grads, (size_t)n0 * 4, g, (size_t)ld * 4, (size_t)n0 * 4, (size_t)K, cudaMemcpyDeviceToHost, st));
    if (values) NYB_CUDA(e, cudaMemcpyAsync(values, dval, (size_t)K * 4, cudaMemcpyDeviceToHost, st));
    int herr = 0;
    if (derr) NYB_CUDA(e, cudaMemcpyAsync(&herr, derr, 4, cudaMemcpyDeviceToHost, st));
    NYB_CUDA(e, cudaStreamSynchronize(st));
    if (herr) return set_err(e, NYB200_ERR_INTERNAL, "tcgen05 pipeline wait expired (code " + std::to_string(herr) + ")");
    for (long i = 0; i < (long)K * n0; ++i)  // never a silently wrong gradient batch
        if (!(grads[i] == grads[i]) || grads[i] - grads[i] != 0.f) return set_err(e, NYB200_ERR_NUMERICAL, "non-finite point gradient");
    return NYB200_OK;
}

}  // namespace nyb

extern "C" int32_t nyb200_point_vjp_batched(nyb200_engine *e, int32_t net_id, int32_t K, const float *x, const float *masks,
                                            const float *spec_rows, float *grads, float *values) {
    if (!e || !spec_rows || !grads) return NYB200_ERR_INVALID;
    std::lock_guard<std::mutex> g(e->mu);
    cudaError_t st = cudaSetDevice(e->device);
    if (st != cudaSuccess) return nyb::check_cuda(e, st, "cudaSetDevice");
    return nyb::point_vjp(e, net_id, K, x, masks, spec_rows, grads, values);
}

extern "C" int32_t nyb200_pgd_attack(nyb200_engine *e, int32_t net_id, const float *spec, int32_t S, const float *in_lo,
                                     const float *in_hi, const float *x0, int32_t K, const nyb200_pgd_config *cfg,
                                     float *best_margin, float *best_x, int32_t *counterexample) {
    if (!e || !spec || !in_lo || !in_hi || !x0 || !cfg || !best_margin) return NYB200_ERR_INVALID;
    std::lock_guard<std::mutex> g(e->mu);
    cudaError_t st = cudaSetDevice(e->device);
    if (st != cudaSuccess) return nyb::check_cuda(e, st, "cudaSetDevice");
    return nyb::pgd_attack(e, net_id, spec, S, in_lo, in_hi, x0, K, *cfg, best_margin, best_x, counterexample);
}
