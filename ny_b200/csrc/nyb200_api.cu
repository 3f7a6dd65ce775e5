// Host side of the C ABI declared in include/nyb200.h: engine lifecycle, network residency,
// workspace management and the launch sequences.  No CPU arithmetic path exists here: every
// numeric result is produced by the kernels in this directory.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <algorithm>
#include <atomic>
#include <thread>
#if defined(__SSE2__)
#include <emmintrin.h>
#endif

#include "nyb200_internal.cuh"

using namespace nyb;

namespace nyb {

int set_err(nyb200_engine *e, int code, const std::string &msg) {
    if (e) e->err = msg;
    return code;
}

int check_cuda(nyb200_engine *e, cudaError_t st, const char *what) {
    if (st == cudaSuccess) return NYB200_OK;
    std::string m = std::string(what) + ": " + cudaGetErrorString(st);
    int code = (st == cudaErrorMemoryAllocation) ? NYB200_ERR_OOM : NYB200_ERR_INTERNAL;
    return set_err(e, code, m);
}

void *ws_get(nyb200_engine *e, const char *name, size_t bytes) {
    DevBuf &b = e->ws[name];
    if (b.bytes >= bytes && b.p) return b.p;
    if (b.p) { cudaFree(b.p); b.p = nullptr; b.bytes = 0; }
    size_t want = bytes < 256 ? 256 : bytes;
    void *p = nullptr;
    cudaError_t st = cudaMalloc(&p, want);
    if (st != cudaSuccess) { check_cuda(e, st, (std::string("cudaMalloc ") + name).c_str()); return nullptr; }
    b.p = p; b.bytes = want;
    return p;
}

// Releases every device allocation a registered network owns.
void free_net(Net &net) {
    for (void *p : net.owned) cudaFree(p);
    net.owned.clear(); net.umma.clear(); net.umma_chain.clear(); net.umma_fwd.clear(); net.umma_adj.clear(); net.wt.clear(); net.frag.clear();
    net.win_bwd.clear(); net.win_fwd.clear(); net.umma_whole = false;
}

}  // namespace nyb


extern "C" {

const char *nyb200_backend_provenance(void) {
    return "nyb200 sm_100a engine (hand-written CUDA kernels; no library GEMM; no CPU fallback)";
}

int32_t nyb200_create(int32_t device_ordinal, nyb200_engine **out) {
    if (!out) return NYB200_ERR_INVALID;
    *out = nullptr;
    int count = 0;
    cudaError_t st = cudaGetDeviceCount(&count);
    if (st != cudaSuccess || count <= 0) return NYB200_ERR_UNSUPPORTED;
    if (device_ordinal < 0 || device_ordinal >= count) return NYB200_ERR_INVALID;
    if (cudaSetDevice(device_ordinal) != cudaSuccess) return NYB200_ERR_UNSUPPORTED;
    cudaDeviceProp prop;
    if (cudaGetDeviceProperties(&prop, device_ordinal) != cudaSuccess) return NYB200_ERR_UNSUPPORTED;
    if (prop.major != 10) return NYB200_ERR_UNSUPPORTED;  // kernels are built for sm_100a only
    nyb200_engine *e = new nyb200_engine();
    e->device = device_ordinal;
    e->sms = prop.multiProcessorCount;
    for (int i = 0; i < 3; ++i) cudaEventCreate(&e->timing.ev[i]);
    *out = e;
    return NYB200_OK;
}

void nyb200_destroy(nyb200_engine *e) {
    if (!e) return;
    cudaSetDevice(e->device);
    cudaStreamSynchronize(e->stream);
    for (auto &kv : e->ws) if (kv.second.p) cudaFree(kv.second.p);
    for (auto &kv : e->nets) free_net(kv.second);
    if (e->status_host) cudaFreeHost(e->status_host);
    if (e->stage) cudaFreeHost(e->stage);
    if (e->stage_in_done) cudaEventDestroy(e->stage_in_done);
    if (e->lanes) cudaFreeHost(e->lanes);
    for (cudaEvent_t ev : e->lane_done) if (ev) cudaEventDestroy(ev);
    if (e->frontier) nyb::frontier_free(e->frontier);
    if (e->frontier_spare) nyb::frontier_free(e->frontier_spare);
    if (e->own_stream) cudaStreamDestroy(e->own_stream);
    if (e->side) cudaStreamDestroy(e->side);
    for (cudaEvent_t ev : e->side_ev) if (ev) cudaEventDestroy(ev);
    for (int i = 0; i < 3; ++i) if (e->timing.ev[i]) cudaEventDestroy(e->timing.ev[i]);
    for (cudaEvent_t ev : e->timing.kev) cudaEventDestroy(ev);
    for (int i = 0; i < 2; ++i) if (e->timing.cev[i]) cudaEventDestroy(e->timing.cev[i]);
    delete e;
}

const char *nyb200_last_error(const nyb200_engine *e) { return e ? e->err.c_str() : "null engine"; }

int32_t nyb200_set_stream(nyb200_engine *e, void *cuda_stream) {
    if (!e) return NYB200_ERR_INVALID;
    std::lock_guard<std::mutex> g(e->mu);
    e->stream = (cudaStream_t)cuda_stream;
    return NYB200_OK;
}

int32_t nyb200_set_launch_overlap(nyb200_engine *e, int32_t on) {
    if (!e) return NYB200_ERR_INVALID;
    std::lock_guard<std::mutex> g(e->mu);
    e->launch_overlap = on != 0;
    return NYB200_OK;
}

int32_t nyb200_set_reserved_sms(nyb200_engine *e, int32_t n) {
    if (!e || n < 0 || n > 64) return NYB200_ERR_INVALID;
    std::lock_guard<std::mutex> g(e->mu);
    e->reserve_sms = n;
    return NYB200_OK;
}

int32_t nyb200_use_own_stream(nyb200_engine *e) {
    if (!e) return NYB200_ERR_INVALID;
    std::lock_guard<std::mutex> g(e->mu);
    NYB_CUDA(e, cudaSetDevice(e->device));
    if (!e->own_stream) NYB_CUDA(e, cudaStreamCreateWithFlags(&e->own_stream, cudaStreamNonBlocking));
    NYB_CUDA(e, cudaStreamSynchronize(e->stream));   // work queued on the previous stream is complete before the switch
    e->stream = e->own_stream;
    return NYB200_OK;
}

int32_t nyb200_set_path(nyb200_engine *e, int32_t path) {
    if (!e) return NYB200_ERR_INVALID;
    if (path != NYB200_PATH_F64 && path != NYB200_PATH_TF32X3 && path != NYB200_PATH_AUTO) return set_err(e, NYB200_ERR_INVALID, "unknown path");
    std::lock_guard<std::mutex> g(e->mu);
    e->path = path == NYB200_PATH_F64 ? NYB200_PATH_F64 : NYB200_PATH_TF32X3;
    e->small_direct = path == NYB200_PATH_AUTO;
    return NYB200_OK;
}

int64_t nyb200_launch_count(const nyb200_engine *e) { return e ? e->launches : 0; }

int32_t nyb200_clear_working_set(nyb200_engine *e) {
    if (!e) return NYB200_ERR_INVALID;
    std::lock_guard<std::mutex> g(e->mu);
    cudaSetDevice(e->device);
    cudaStreamSynchronize(e->stream);
    for (auto &kv : e->ws) if (kv.second.p) cudaFree(kv.second.p);
    e->ws.clear();
    e->batch = Batch();
    if (e->frontier_spare) { nyb::frontier_free(e->frontier_spare); e->frontier_spare = nullptr; }
    // networks registered on behalf of the reference-shaped calls (their weight cache)
    for (auto &kv : e->boundary_nets) {
        auto it = e->nets.find(kv.second);
        if (it != e->nets.end()) { free_net(it->second); e->nets.erase(it); }
    }
    e->boundary_nets.clear();
    return NYB200_OK;
}

// Expands a per-channel bias to one value per output element (GpuCrownLayer::Conv2d::bias_expanded).
static void expand_bias(const float *b, int oc, int plane, std::vector<float> &out) {
    out.resize((size_t)oc * plane);
    for (int c = 0; c < oc; ++c)
        for (int i = 0; i < plane; ++i) out[(size_t)c * plane + i] = b[c];
}

}  // extern "C"

namespace nyb {

// What create_net asks about a layer's weights: largest magnitude and smallest non-zero one (as bits, the latter as its
// distance from infinity, so that zeroed words are the start of both), largest sum of magnitudes of a row (binary64 bits).
struct LayerStats { unsigned long long l1_bits; unsigned max_bits, inv_min_bits; };
struct LayerRows { const float *W[kMaxLinear]; int n[kMaxLinear], len[kMaxLinear]; };

static float bits_float(unsigned b) { float f; memcpy(&f, &b, 4); return f; }

// One block per row (grid x) of every layer (grid y).  A walk over all weights in one dependent binary64 sum on the host took
// two milliseconds for a network of 0.7 million.
__global__ void __launch_bounds__(256) k_layer_stats(LayerRows rows, LayerStats *__restrict__ out) {
    const int k = blockIdx.y;
    if ((int)blockIdx.x >= rows.n[k]) return;
    const float *w = rows.W[k] + (long)blockIdx.x * rows.len[k];
    unsigned mx = 0, inv = 0;
    double sum = 0.0;
    for (int i = threadIdx.x; i < rows.len[k]; i += 256) {
        const unsigned b = __float_as_uint(w[i]) & 0x7fffffffu;   // ordered as the magnitudes are, NaN above infinity
        mx = max(mx, b);
        if (b > 0 && b < 0x7f800000u) inv = max(inv, 0x7f800000u - b);
        sum += (double)__uint_as_float(b);
    }
    __shared__ double part[8];
    mx = __reduce_max_sync(0xffffffffu, mx);
    inv = __reduce_max_sync(0xffffffffu, inv);
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if ((threadIdx.x & 31) == 0) {
        part[threadIdx.x >> 5] = sum;
        atomicMax(&out[k].max_bits, mx);
        atomicMax(&out[k].inv_min_bits, inv);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int i = 1; i < 8; ++i) sum += part[i];
        if (mx < 0x7f800000u) atomicMax(&out[k].l1_bits, (unsigned long long)__double_as_longlong(sum));   // (not of a row with a NaN in it)
    }
}

int create_net(nyb200_engine *e, int32_t n_layers, const nyb200_layer_desc *ld, const float *wflat,
               const float *bflat, int32_t *net_id) {
    if (n_layers < 1 || n_layers > kMaxLinear) return set_err(e, NYB200_ERR_UNSUPPORTED, "layer count out of range");
    NYB_CUDA(e, cudaSetDevice(e->device));
    Net net;
    memset(&net.v, 0, sizeof(net.v));
    net.v.L = n_layers;
    net.kind.resize(n_layers);
    net.geom.resize(n_layers);
    net.skip.assign(n_layers, -1);
    int off = 0;
    for (int k = 0; k < n_layers; ++k) {
        const nyb200_layer_desc &l = ld[k];
        if (l.in_features <= 0 || l.out_features <= 0) return set_err(e, NYB200_ERR_SHAPE, "non-positive layer width");
        if (k > 0 && l.in_features != ld[k - 1].out_features) return set_err(e, NYB200_ERR_SHAPE, "layer widths do not chain");
        if (l.kind == NYB200_LAYER_CONV2D) {
            ConvGeom g{l.in_channels, l.in_h, l.in_w, l.out_channels, l.out_h, l.out_w,
                       l.kernel_h, l.kernel_w, l.stride_h, l.stride_w, l.pad_h, l.pad_w};
            if (g.ic <= 0 || g.oc <= 0 || g.ih <= 0 || g.iw <= 0 || g.kh <= 0 || g.kw <= 0 || g.sh <= 0 || g.sw <= 0 ||
                g.ph < 0 || g.pw < 0)
                return set_err(e, NYB200_ERR_SHAPE, "conv2d: non-positive geometry (zero stride or kernel)");
            if (g.ih + 2 * g.ph < g.kh || g.iw + 2 * g.pw < g.kw) return set_err(e, NYB200_ERR_SHAPE, "conv2d: kernel larger than the padded input");
            if (g.oh != (g.ih + 2 * g.ph - g.kh) / g.sh + 1 || g.ow != (g.iw + 2 * g.pw - g.kw) / g.sw + 1)
                return set_err(e, NYB200_ERR_SHAPE, "conv2d: output size does not match the geometry");
            if ((long)g.ic * g.ih * g.iw != l.in_features || (long)g.oc * g.oh * g.ow != l.out_features)
                return set_err(e, NYB200_ERR_SHAPE, "conv2d: flattened sizes do not match the geometry");
            net.geom[k] = g;
        } else if (l.kind != NYB200_LAYER_LINEAR) {
            return set_err(e, NYB200_ERR_UNSUPPORTED, "unknown layer kind");
        }
        net.kind[k] = l.kind;
        if (l.skip_from != 0) {
            int j = l.skip_from - 1;
            if (j < 0 || j > k - 2) return set_err(e, NYB200_ERR_INVALID, "skip_from must name a layer at least two before this one");
            if (ld[j].out_features != l.out_features) return set_err(e, NYB200_ERR_SHAPE, "residual branch widths differ");
            if (k == n_layers - 1) return set_err(e, NYB200_ERR_UNSUPPORTED, "the last layer cannot take a residual connection");
            net.skip[k] = j;
        }
        if (k == 0) { net.v.dims[0] = l.in_features; net.max_dim = l.in_features; }
        net.v.dims[k + 1] = l.out_features;
        if (l.out_features > net.max_dim) net.max_dim = l.out_features;
        net.v.pre_off[k] = off;
        off += l.out_features;
    }
    net.v.pre_off[n_layers] = off;
    net.v.n_pre = off;
    net.v.nps = (off + 3) & ~3;
    // Weights, biases and the layers' statistics in one block; a failed upload releases it
    struct Guard { Net &n; bool armed = true; ~Guard() { if (armed) free_net(n); } } guard{net};
    Carve c;
    float *bias[kMaxLinear] = {};
    LayerStats *stats = nullptr;
    LayerRows rows;
    auto weights_of = [&](int k) {
        const nyb200_layer_desc &l = ld[k];
        return net.kind[k] == NYB200_LAYER_CONV2D ? (size_t)l.out_channels * l.in_channels * l.kernel_h * l.kernel_w : (size_t)l.in_features * l.out_features;
    };
    for (int pass = 0; pass < 2; ++pass) {
        c.used = 0;
        int most_rows = 0;
        for (int k = 0; k < n_layers; ++k) {
            const size_t nw = weights_of(k);
            net.v.W[k] = (const float *)c.take(nw * 4);
            bias[k] = ld[k].has_bias ? (float *)c.take((size_t)ld[k].out_features * 4) : nullptr;
            net.v.b[k] = bias[k];
            rows.W[k] = net.v.W[k];
            rows.n[k] = net.kind[k] == NYB200_LAYER_CONV2D ? ld[k].out_channels : ld[k].out_features;   // one output's weights each
            rows.len[k] = (int)(nw / (size_t)rows.n[k]);
            most_rows = std::max(most_rows, rows.n[k]);
        }
        stats = (LayerStats *)c.take((size_t)n_layers * sizeof(LayerStats));
        if (pass == 0) {
            void *block = nullptr;
            NYB_CUDA(e, cudaMalloc(&block, c.used));
            net.owned.push_back(block);
            c.block = (char *)block;
            continue;
        }
        size_t wo = 0, bo = 0;
        std::vector<float> expanded;
        for (int k = 0; k < n_layers; ++k) {
            const nyb200_layer_desc &l = ld[k];
            const bool conv = l.kind == NYB200_LAYER_CONV2D;
            const size_t nw = weights_of(k);
            NYB_CUDA(e, cudaMemcpyAsync(const_cast<float *>(net.v.W[k]), wflat + wo, nw * 4, cudaMemcpyHostToDevice, e->stream));
            wo += nw;
            net.bmax.push_back(0.f);
            if (!l.has_bias) continue;
            if (!bflat) return set_err(e, NYB200_ERR_INVALID, "has_bias set but bflat is null");
            const size_t nb = conv ? (size_t)l.out_channels : (size_t)l.out_features;
            for (size_t i = 0; i < nb; ++i) {
                if (!std::isfinite(bflat[bo + i])) return set_err(e, NYB200_ERR_NUMERICAL, "non-finite bias");
                net.bmax.back() = std::max(net.bmax.back(), bflat[bo + i]);
            }
            const float *src = bflat + bo;
            if (conv) { expand_bias(bflat + bo, l.out_channels, l.out_h * l.out_w, expanded); src = expanded.data(); }
            NYB_CUDA(e, cudaMemcpyAsync(bias[k], src, (size_t)l.out_features * 4, cudaMemcpyHostToDevice, e->stream));
            if (conv) NYB_CUDA(e, cudaStreamSynchronize(e->stream));   // the next layer's bias is expanded in the same place
            bo += nb;
        }
        NYB_CUDA(e, cudaMemsetAsync(stats, 0, (size_t)n_layers * sizeof(LayerStats), e->stream));
        k_layer_stats<<<dim3((unsigned)most_rows, (unsigned)n_layers), 256, 0, e->stream>>>(rows, stats);
        e->launches++;
        NYB_CUDA(e, cudaGetLastError());
    }
    std::vector<LayerStats> ls((size_t)n_layers);
    NYB_CUDA(e, cudaMemcpyAsync(ls.data(), stats, ls.size() * sizeof(LayerStats), cudaMemcpyDeviceToHost, e->stream));
    NYB_CUDA(e, cudaStreamSynchronize(e->stream));   // (the caller's arrays may go away, too)
    for (int k = 0; k < n_layers; ++k) {
        // a fp16 pair holds a weight's 22 bits unless it is more than 2^27 times smaller than the largest: such a layer keeps
        // its TF32 operands
        const float wmax = bits_float(ls[k].max_bits), wmin = bits_float(0x7f800000u - ls[k].inv_min_bits);
        if (!std::isfinite(wmax)) return set_err(e, NYB200_ERR_NUMERICAL, "non-finite weight");
        net.wmax.push_back(wmin < wmax * 7.450580596923828e-09f ? -wmax : wmax);
        // sum over a chunk of 64 of 2^-50 max|a| q_j <= eps |a| * 64 * 2^-50 / eps * (row sum of |W|) max|z|, eps >= 7.1e-7
        double l1;
        memcpy(&l1, &ls[k].l1_bits, 8);
        net.v.qfl[k] = net.kind[k] == NYB200_LAYER_LINEAR && net.wmax[k] > 0.f ? (float)(64.0 * kWinFloor / 7.1e-7 * l1 * 1.0001) : 0.f;
    }
    int id = e->next_net++;
    e->nets[id] = net;
    guard.armed = false;
    *net_id = id;
    return NYB200_OK;
}

}  // namespace nyb

extern "C" {

int32_t nyb200_net_create(nyb200_engine *e, int32_t n_linear, const int32_t *dims, const float *wflat,
                          const float *bflat, const int32_t *has_bias, int32_t *net_id) {
    if (!e || !dims || !wflat || !has_bias || !net_id) return NYB200_ERR_INVALID;
    if (n_linear < 1 || n_linear > kMaxLinear) return set_err(e, NYB200_ERR_UNSUPPORTED, "layer count out of range");
    std::lock_guard<std::mutex> g(e->mu);
    std::vector<nyb200_layer_desc> ld((size_t)n_linear);
    for (int k = 0; k < n_linear; ++k) {
        memset(&ld[k], 0, sizeof(ld[k]));
        ld[k].kind = NYB200_LAYER_LINEAR;
        ld[k].in_features = dims[k];
        ld[k].out_features = dims[k + 1];
        ld[k].has_bias = has_bias[k];
    }
    return create_net(e, n_linear, ld.data(), wflat, bflat, net_id);
}

int32_t nyb200_net_create_layers(nyb200_engine *e, int32_t n_layers, const nyb200_layer_desc *layers,
                                 const float *wflat, const float *bflat, int32_t *net_id) {
    if (!e || !layers || !wflat || !net_id) return NYB200_ERR_INVALID;
    std::lock_guard<std::mutex> g(e->mu);
    return create_net(e, n_layers, layers, wflat, bflat, net_id);
}

int32_t nyb200_net_destroy(nyb200_engine *e, int32_t net_id) {
    if (!e) return NYB200_ERR_INVALID;
    std::lock_guard<std::mutex> g(e->mu);
    auto it = e->nets.find(net_id);
    if (it == e->nets.end()) return set_err(e, NYB200_ERR_INVALID, "unknown net id");
    cudaSetDevice(e->device);
    cudaStreamSynchronize(e->stream);
    free_net(it->second);
    e->nets.erase(it);
    if (e->batch.net_id == net_id) e->batch = Batch();
    return NYB200_OK;
}

// The trait's precision contract for gemm_f32 is the error model of round-to-nearest fp32 arithmetic in any summation
// order, |c - a.b| <= gamma_k sum|a||b| with gamma_k = k u / (1 - k u), u = 2^-24 (crates/ny-core/src/gemm.rs:318-324);
// verdict-feeding callers certify their results with it.  The 3xTF32 product's certified rate (umma_eps) is below
// gamma_k from k = 21 on; shorter contractions take the binary64-accumulating kernel (exact sum, one rounding).
static bool tensor_product_meets_rn_model(int k) {
    const double u = 5.9604644775390625e-08;
    return umma_eps(k) * 1.000001 <= (double)k * u / (1.0 - (double)k * u);
}

static int32_t gemm_f32_impl(nyb200_engine *e, int32_t m, int32_t k, int32_t n, const float *a, const float *b, float *c_out,
                             bool fast) {
    if (!e || !a || !b || !c_out) return NYB200_ERR_INVALID;
    std::lock_guard<std::mutex> g(e->mu);
    if (m <= 0 || k <= 0 || n <= 0) return set_err(e, NYB200_ERR_SHAPE, "gemm_f32: non-positive dimension");
    NYB_CUDA(e, cudaSetDevice(e->device));
    NYB_WS(da, float *, e, "gemm_a", (size_t)m * k * 4);
    NYB_WS(db, float *, e, "gemm_b", (size_t)k * n * 4);
    NYB_WS(dc, float *, e, "gemm_c", (size_t)m * n * 4);
    NYB_CUDA(e, cudaMemcpyAsync(da, a, (size_t)m * k * 4, cudaMemcpyHostToDevice, e->stream));
    NYB_CUDA(e, cudaMemcpyAsync(db, b, (size_t)k * n * 4, cudaMemcpyHostToDevice, e->stream));
    if (e->path == NYB200_PATH_TF32X3 && (fast || tensor_product_meets_rn_model(k))) {
        NYB_WS(derr, int *, e, "umma_err", 256);
        NYB_CUDA(e, cudaMemsetAsync(derr, 0, 4, e->stream));
        UmmaLayer ul;
        Carve c;
        NYB_TRY(umma_prepare_layer(e, WeightSource{db}, k, n, &ul, c));
        NYB_WS(op, char *, e, "gemm_operand", c.used);
        c.block = op; c.used = 0;
        NYB_TRY(umma_prepare_layer(e, WeightSource{db}, k, n, &ul, c));
        int st = launch_umma(e, ul, m, da, k, dc, n, derr);
        int herr = 0;
        cudaError_t cs = cudaGetLastError();
        if (cs == cudaSuccess) cs = cudaMemcpyAsync(&herr, derr, 4, cudaMemcpyDeviceToHost, e->stream);
        if (cs == cudaSuccess) cs = cudaMemcpyAsync(c_out, dc, (size_t)m * n * 4, cudaMemcpyDeviceToHost, e->stream);
        if (cs == cudaSuccess) cs = cudaStreamSynchronize(e->stream);
        NYB_TRY(st);
        NYB_CUDA(e, cs);
        if (herr) return set_err(e, NYB200_ERR_INTERNAL, "tcgen05 pipeline wait expired (code " + std::to_string(herr) + ")");
        return NYB200_OK;
    }
    launch_gemm_f64(e, m, n, k, da, k, db, n, dc, n, 1, nullptr, nullptr, 0, nullptr);
    NYB_CUDA(e, cudaGetLastError());
    NYB_CUDA(e, cudaMemcpyAsync(c_out, dc, (size_t)m * n * 4, cudaMemcpyDeviceToHost, e->stream));
    NYB_CUDA(e, cudaStreamSynchronize(e->stream));
    return NYB200_OK;
}

int32_t nyb200_gemm_f32(nyb200_engine *e, int32_t m, int32_t k, int32_t n, const float *a, const float *b, float *c_out) {
    return gemm_f32_impl(e, m, k, n, a, b, c_out, false);
}

int32_t nyb200_gemm_f32_fast(nyb200_engine *e, int32_t m, int32_t k, int32_t n, const float *a, const float *b, float *c_out) {
    return gemm_f32_impl(e, m, k, n, a, b, c_out, true);
}

}  // extern "C"

// ------------------------------------------------------------------ batch plumbing
namespace nyb {

// Adds the finished run's event intervals to the accumulators.
void fold_timing(nyb::Timing &t) {
    if (!t.pending) return;
    if (cudaEventSynchronize(t.ev[2]) == cudaSuccess) {
        float f = 0, bw = 0;
        cudaEventElapsedTime(&f, t.ev[0], t.ev[1]);
        cudaEventElapsedTime(&bw, t.ev[1], t.ev[2]);
        t.fwd_ms += f; t.bwd_ms += bw; t.tot_ms += f + bw; t.runs++;
        for (int i = 0; i + 1 < t.kev_used; i += 2) {
            float g = 0;
            if (cudaEventElapsedTime(&g, t.kev[i], t.kev[i + 1]) == cudaSuccess) t.gemm_ms += g;
        }
        if (t.cev_used) {
            float g = 0;
            if (cudaEventElapsedTime(&g, t.cev[0], t.cev[1]) == cudaSuccess) t.chain_ms += g;
        }
    }
    t.kev_used = 0;
    t.cev_used = false;
    t.pending = false;
}

cudaEvent_t next_kev(nyb::Timing &t) {
    if (t.kev_used == (int)t.kev.size()) { cudaEvent_t ev; cudaEventCreate(&ev); t.kev.push_back(ev); }
    return t.kev[t.kev_used++];
}


// Pinned staging of at least kStageIn + out_bytes bytes (grow-only; growing waits for the stream).
static int ensure_stage(nyb200_engine *e, size_t out_bytes) {
    const size_t need = kStageIn + out_bytes;
    if (e->stage && e->stage_bytes >= need) return NYB200_OK;
    NYB_CUDA(e, cudaStreamSynchronize(e->stream));
    if (e->stage) cudaFreeHost(e->stage);
    e->stage = nullptr; e->stage_bytes = 0; e->stage_out_valid = false;
    const size_t sz = need + need / 2;
    if (cudaHostAlloc((void **)&e->stage, sz, cudaHostAllocDefault) != cudaSuccess) return set_err(e, NYB200_ERR_OOM, "pinned staging allocation failed");
    e->stage_bytes = sz;
    if (!e->stage_in_done) NYB_CUDA(e, cudaEventCreateWithFlags(&e->stage_in_done, cudaEventDisableTiming));
    return NYB200_OK;
}

// Copy into pinned memory past the caches (dst 16-byte aligned): a transfer whose source lies in a core's cache is served
// by that cache, at a third of the bus's rate.
static void copy_past_caches(unsigned char *dst, const unsigned char *src, size_t n) {
    size_t i = 0;
#if defined(__SSE2__)
    for (; i + 64 <= n; i += 64) {
        __m128i v[4];
        for (int k = 0; k < 4; ++k) v[k] = _mm_loadu_si128((const __m128i *)(src + i + 16 * k));
        for (int k = 0; k < 4; ++k) _mm_stream_si128((__m128i *)(dst + i + 16 * k), v[k]);
    }
#endif
    memcpy(dst + i, src + i, n - i);
#if defined(__SSE2__)
    _mm_sfence();
#endif
}

// Rows of `width` bytes, one after the other on the host, to rows dst_pitch apart on the device; the source may be reused
// when the call returns.  The driver stages a pageable source with one thread (14 MB of slopes: 0.92 ms, half of the call
// they belong to, the device idle); here kLanes threads each copy blocks of rows into two pinned slots in turn, at the
// device's pitch so that a block is one plain transfer, past the caches: 0.40 ms (0.85 with cached stores; 0.27 is the
// bus).  More threads only share the same memory bandwidth; below one slot their start (60 us) costs what they save.
int upload_rows(nyb200_engine *e, void *dst, size_t dst_pitch, const void *src, size_t width, size_t rows, cudaStream_t stream) {
    const size_t per = std::min(kLaneSlot / dst_pitch, std::max<size_t>(1, (rows + 2 * kLanes - 1) / (2 * kLanes)));
    bool direct = per == 0 || rows * width < kLaneSlot || (dst_pitch & 15);
    if (!direct) {   // a pinned source needs no staging
        cudaPointerAttributes at;
        direct = cudaPointerGetAttributes(&at, src) != cudaSuccess || at.type != cudaMemoryTypeUnregistered;
        cudaGetLastError();
    }
    if (!direct && !e->lanes) {
        if (cudaHostAlloc((void **)&e->lanes, 2 * kLanes * kLaneSlot, cudaHostAllocDefault) != cudaSuccess) { cudaGetLastError(); e->lanes = nullptr; direct = true; }
        for (int i = 0; i < 2 * kLanes && !direct; ++i)
            if (!e->lane_done[i]) NYB_CUDA(e, cudaEventCreateWithFlags(&e->lane_done[i], cudaEventDisableTiming));
    }
    if (direct) {
        if (dst_pitch == width) NYB_CUDA(e, cudaMemcpyAsync(dst, src, width * rows, cudaMemcpyHostToDevice, stream));
        else NYB_CUDA(e, cudaMemcpy2DAsync(dst, dst_pitch, src, width, width, rows, cudaMemcpyHostToDevice, stream));
        return NYB200_OK;
    }
    const size_t blocks = (rows + per - 1) / per;
    std::atomic<int> failed{(int)cudaSuccess};
    auto lane = [&](int t) {
        cudaError_t st = cudaSetDevice(e->device);
        int i = 0;
        for (size_t b = t; b < blocks && st == cudaSuccess; b += kLanes, i ^= 1) {
            unsigned char *slot = e->lanes + (2 * t + i) * kLaneSlot;
            st = cudaEventSynchronize(e->lane_done[2 * t + i]);   // the slot's last transfer, of this call or an earlier one
            if (st != cudaSuccess) break;
            const size_t r0 = b * per, n = std::min(per, rows - r0);
            const unsigned char *from = (const unsigned char *)src + r0 * width;
            if (dst_pitch == width) copy_past_caches(slot, from, n * width);
            else for (size_t r = 0; r < n; ++r) copy_past_caches(slot + r * dst_pitch, from + r * width, width);
            // (the last row without its padding: it may end the allocation)
            st = cudaMemcpyAsync((char *)dst + r0 * dst_pitch, slot, (n - 1) * dst_pitch + width, cudaMemcpyHostToDevice, stream);
            if (st == cudaSuccess) st = cudaEventRecord(e->lane_done[2 * t + i], stream);
        }
        if (st != cudaSuccess) failed = (int)st;
    };
    std::thread th[kLanes - 1];
    int started = 0;
    try {
        for (; started < kLanes - 1; ++started) th[started] = std::thread(lane, started + 1);
    } catch (...) {}   // no thread to be had: the caller takes its share
    lane(0);
    for (int t = started + 1; t < kLanes; ++t) lane(t);
    for (int t = 0; t < started; ++t) th[t].join();
    return check_cuda(e, (cudaError_t)failed.load(), "upload of a large host array");
}

// Host arrays to the device through the pinned input region: one host copy each, and one transfer for every run of
// pieces that lie next to each other on the device (an asynchronous copy costs a few microseconds on both sides however
// small it is).  Pieces that do not fit go by upload_rows.
int staged_upload(nyb200_engine *e, const UploadPiece *pc, int n) {
    size_t total = 0;
    for (int i = 0; i < n; ++i) total += (pc[i].bytes + 255) & ~(size_t)255;
    if (total > kStageIn || ensure_stage(e, 0) != NYB200_OK) {
        const size_t row = 4096;
        for (int i = 0; i < n; ++i) {
            const size_t whole = pc[i].bytes / row * row;
            if (whole) NYB_TRY(upload_rows(e, pc[i].dst, row, pc[i].src, row, whole / row, e->stream));
            if (pc[i].bytes > whole)
                NYB_CUDA(e, cudaMemcpyAsync((char *)pc[i].dst + whole, (const char *)pc[i].src + whole, pc[i].bytes - whole, cudaMemcpyHostToDevice, e->stream));
        }
        return NYB200_OK;
    }
    NYB_CUDA(e, cudaEventSynchronize(e->stage_in_done));   // the previous upload has left the region
    size_t h = 0;
    for (int i = 0; i < n;) {
        if (!pc[i].bytes) { ++i; continue; }
        char *d0 = (char *)pc[i].dst;
        const size_t h0 = h;
        size_t end = 0;   // bytes of the run so far
        for (; i < n; ++i) {
            if (!pc[i].bytes) continue;
            const long off = (char *)pc[i].dst - d0;
            if (off < (long)end || off - (long)end >= 256) break;   // not the next piece of this run
            memcpy(e->stage + h0 + off, pc[i].src, pc[i].bytes);
            end = (size_t)off + pc[i].bytes;
        }
        NYB_CUDA(e, cudaMemcpyAsync(d0, e->stage + h0, end, cudaMemcpyHostToDevice, e->stream));
        h = h0 + ((end + 255) & ~(size_t)255);
    }
    NYB_CUDA(e, cudaEventRecord(e->stage_in_done, e->stream));
    return NYB200_OK;
}

// One contiguous device block to several host arrays (dst null: skipped), through the pinned output region; waits.
int staged_fetch(nyb200_engine *e, const void *src, const FetchPiece *pc, int n) {
    size_t total = 0;
    for (int i = 0; i < n; ++i) total += pc[i].bytes;
    const char *s = (const char *)src;
    if (total > kStageOutMost || ensure_stage(e, total) != NYB200_OK) {
        for (int i = 0; i < n; ++i) {
            if (pc[i].dst && pc[i].bytes) NYB_CUDA(e, cudaMemcpyAsync(pc[i].dst, s, pc[i].bytes, cudaMemcpyDeviceToHost, e->stream));
            s += pc[i].bytes;
        }
        NYB_CUDA(e, cudaStreamSynchronize(e->stream));
        return NYB200_OK;
    }
    unsigned char *h = e->stage + kStageIn;
    e->stage_out_valid = false;
    NYB_CUDA(e, cudaMemcpyAsync(h, s, total, cudaMemcpyDeviceToHost, e->stream));
    NYB_CUDA(e, cudaStreamSynchronize(e->stream));
    for (int i = 0; i < n; ++i) {
        if (pc[i].dst) memcpy(pc[i].dst, h, pc[i].bytes);
        h += pc[i].bytes;
    }
    return NYB200_OK;
}

// Size of the block of results: 256 bytes of words, flags (padded), lower and upper bounds.
static size_t result_bytes(size_t D, size_t S) { return 256 + ((D * 4 + 255) & ~(size_t)255) + 2 * D * S * 4; }

int batch_ptrs(nyb200_engine *e, const Net &net, const Batch &b, BatchPtrs &p) {
    const NetView &nv = net.v;
    size_t D = (size_t)b.D, np = (size_t)nv.nps;
    size_t M = D * b.R;
    p.lda = (net.max_dim + 7) & ~7;
    size_t box = (size_t)nv.dims[0] * (b.box_stride ? D : 1);
#define GET_RAW(var, type, name, bytes)                                 \
    var = (type)ws_get(e, name, (bytes));                                \
    if (!var) return NYB200_ERR_OOM;
#define GET(field, type, name, bytes) GET_RAW(p.field, type, name, bytes)
    // What a call uploads sits in one block, so that a batch of small arrays is one transfer: box, shared inherited
    // bounds, split lists, specification rows.  The rows come last: the partial passes of one call ask for different
    // row counts and must find everything else where it was.
    auto pad = [](size_t v) { return (v + 255) & ~(size_t)255; };
    const size_t b_box = pad(box * 4), b_inh = pad(np * 4), b_ns = pad(D * 4);
    const size_t b_sp = pad(D * (size_t)(b.max_splits > 0 ? b.max_splits : 1) * sizeof(nyb200_split));
    char *in_block;
    GET_RAW(in_block, char *, "inputs", 2 * b_box + 2 * b_inh + b_ns + b_sp + (size_t)b.S * nv.dims[nv.L] * 4)
    p.in_lo = (float *)in_block; p.in_hi = (float *)(in_block + b_box);
    p.inh_lo = (float *)(in_block + 2 * b_box); p.inh_hi = (float *)(in_block + 2 * b_box + b_inh);
    p.nsplits = (int *)(in_block + 2 * b_box + 2 * b_inh);
    p.splits = (nyb200_split *)(in_block + 2 * b_box + 2 * b_inh + b_ns);
    p.spec = (float *)(in_block + 2 * b_box + 2 * b_inh + b_ns + b_sp);
    if (b.inh_stride) {
        GET(inh_lo, float *, "inh_lo", D * np * 4)
        GET(inh_hi, float *, "inh_hi", D * np * 4)
    }
    GET(alpha, float *, "alpha", b.has_alpha ? D * np * 4 : 4)
    // What a run returns sits in one block too: the run's words (minimum, counters), flags, bounds.
    char *out_block;
    GET_RAW(out_block, char *, "results", result_bytes(D, b.S))
    p.min_lower = (float *)out_block;
    p.flags = (int *)(out_block + 256);
    p.out_lo = (float *)(out_block + 256 + b_ns); p.out_hi = p.out_lo + D * b.S;
    GET(code, signed char *, "code", D * np)
    GET(sbeta, float *, "sbeta", D * (np + (size_t)nv.L) * 4)   // and beta_max (run_forward) behind it: one fill clears both
    GET(raw_lo, float *, "raw_lo", D * np * 4)
    GET(raw_hi, float *, "raw_hi", D * np * 4)
    GET(q, float *, "q", D * np * 4)
    GET(pre_lo, float *, "pre_lo", D * np * 4)
    GET(pre_hi, float *, "pre_hi", D * np * 4)
    GET(zl, float *, "zlu", 2 * D * np * 4)  // lower ends, then upper ends: one [2D x nps] operand
    p.zu = p.zl + D * np;
    GET(zabs, float *, "zabs", D * np * 4)
    GET(tab, float4 *, "tab", D * np * 16)
    GET(A0, float *, "A0", M * p.lda * 4)
    GET(A1, float *, "A1", M * p.lda * 4)
    // the per-row scalars share one block so that a pass clears them with one fill: bias, magnitude sum, rounding
    // penalty (binary64 each), then the coefficient-safety flags of the fused concretisation
    GET(rb, double *, "row_scalars", M * 28)
    p.rabs = p.rb + M;
    p.rpen = p.rb + 2 * M;
    p.row_bad = (int *)(p.rb + 3 * M);
    p.alpha_up = nullptr;
    if (b.dual_alpha) { GET(alpha_up, float *, "alpha_up", D * np * 4) }
#undef GET
#undef GET_RAW
    return NYB200_OK;
}

int find_net(nyb200_engine *e, int net_id, Net **out) {
    auto it = e->nets.find(net_id);
    if (it == e->nets.end()) return set_err(e, NYB200_ERR_INVALID, "unknown net id");
    *out = &it->second;
    return NYB200_OK;
}

// Scratch of one slice of an interval convolution.  Slices that fit in L2 are no faster: their launches fill the SMs less well
// (residual network, 256 domains: 50.1 ms in whole layers, 52.6 in slices of 192 MB, 53.3 of 64).
constexpr size_t kConvColsMost = (size_t)4 << 30;

// Interval forward pass for the resident batch.  fwd_mode: 0 clamp-only, 1 constrained, 2 plain IBP.
// The slope of an unstable neuron's lower line is a step function of its interval (relax_neuron: u > -l), so a bound jumps
// where a rounding of this pass decides a tie: its products are TF32 pairs, and fp16 pairs, as exact and faster, are for the
// backward pass alone, where a rounding moves a bound by no more than itself.  (With fp16 pairs here 4096 domains of
// 784 -> 8x256 -> 10 took 1.19 ms instead of 1.21, 1024 of a convolutional classifier 2.38 instead of 3.09 and 256 of a
// residual network 41.8 instead of 49.9, and up to three choices of such a batch, 2345 of a small residual network's, were
// others: single bounds moved by 0.8 %.)
int run_forward(nyb200_engine *e, Net &net, const Batch &b, BatchPtrs &p, int fwd_mode) {
    const NetView &nv = net.v;
    int D = b.D;
    if (e->path == NYB200_PATH_F64 && e->fuse_chain && fwd_mode < 2 && p.inh_lo && direct_eligible(net)) return run_forward_direct(e, net, b, p, fwd_mode, nullptr, D);
    // The tcgen05 path covers every layer whose input is a post-ReLU interval (lower end >= 0) of a
    // per-domain batch; the first layer (arbitrary-sign box, usually shared) stays on the binary64 kernel.
    const bool tensor = (e->path == NYB200_PATH_TF32X3) && D >= 64 && nv.L > 1;
    float *Fl = nullptr;
    int ldf = 0;
    int *derr = nullptr;
    if (tensor) {
        if (net.umma_fwd.empty()) {
            std::vector<UmmaLayer> fwd((size_t)nv.L);
            NYB_TRY(build_operands(e, net, [&](Carve &c) -> int {
                for (int k = 1; k < nv.L; ++k) {
                    const ConvGeom &g = net.geom[k];
                    if (!net.is_conv(k)) NYB_TRY(umma_prepare_signed(e, nv.W[k], 1, nv.dims[k], nv.dims[k + 1], &fwd[k], c));
                    else NYB_TRY(umma_prepare_signed(e, nv.W[k], g.kh * g.kw, g.ic, g.oc, &fwd[k], c));
                }
                return NYB200_OK;
            }));
            net.umma_fwd = std::move(fwd);
        }
        int mo = 0;
        for (int k = 1; k < nv.L; ++k)
            if (!net.is_conv(k)) mo = nv.dims[k + 1] > mo ? nv.dims[k + 1] : mo;
        if (mo == 0) mo = 8;
        ldf = (2 * mo + 7) & ~7;
        Fl = (float *)ws_get(e, "fwd", (size_t)2 * D * ldf * 4);
        derr = (int *)ws_get(e, "umma_err", 256);
        if (!Fl || !derr) return NYB200_ERR_OOM;
    }
    size_t np = nv.nps;
    unsigned *zmax_rows = nullptr;   // largest input magnitude of every (layer, domain), for the charges of fp16 contractions
    if (tensor) {
        zmax_rows = (unsigned *)ws_get(e, "fwd_zmax", (size_t)nv.L * D * 4);
        if (!zmax_rows) return NYB200_ERR_OOM;
        NYB_CUDA(e, cudaMemsetAsync(zmax_rows, 0, (size_t)nv.L * D * 4, e->stream));
    }
    // a slack-to-width ratio above this marks the domain for the binary64 re-evaluation (same switch as the
    // penalty criterion: 0 disables)
    const float fwd_tol = b.decision_thr ? 0.f : e->refine_tol;   // a verdict-only round does not flag on the interval slack
    // When the backward pass of this run will be the fused chain, the finish kernel also leaves the chain's charge
    // weights (one fused multiply-add per table entry here instead of a pass of its own over three arrays).
    float *cj = nullptr;
    if (e->path == NYB200_PATH_TF32X3 && e->fuse_chain && fwd_mode < 2 && chain_eligible(net, nv.L) && (nv.nps % 4 == 0)) {
        cj = (float *)ws_get(e, "chain_cj", (size_t)D * nv.nps * 4);
        if (!cj) return NYB200_ERR_OOM;
    }
    p.cj = cj;
    NYB_CUDA(e, cudaMemsetAsync(p.flags, 0, (size_t)D * 4, e->stream));
    NYB_CUDA(e, cudaMemsetAsync(p.code, 0, (size_t)D * np, e->stream));
    const bool bounded = e->path == NYB200_PATH_TF32X3 && fwd_mode < 2 && net.has_conv();   // what k_relax_image bounds its rows with
    NYB_CUDA(e, cudaMemsetAsync(p.sbeta, 0, ((size_t)D * np + (bounded ? (size_t)nv.L * D : 0)) * 4, e->stream));
    p.beta_max = bounded ? p.sbeta + (size_t)D * np : nullptr;
    if (fwd_mode != 2 && b.max_splits > 0)
        launch_scatter_splits(e, nv, p.splits, p.nsplits, b.max_splits, D, p.code, p.sbeta, p.flags, p.beta_max);
    for (int k = 0; k < nv.L; ++k) {
        NYB_DEADLINE(e, "interval pass");
        const float *zl, *zu;
        long in_ds;
        int Deff;
        if (k == 0) { zl = p.in_lo; zu = p.in_hi; in_ds = b.box_stride; Deff = b.box_stride ? D : 1; }
        else { zl = p.zl + nv.pre_off[k - 1]; zu = p.zu + nv.pre_off[k - 1]; in_ds = (long)np; Deff = D; }
        const bool tk = tensor && k >= 1 && !net.is_conv(k) && net.skip_of(k) < 0;
        const bool tconv = tensor && k >= 1 && net.is_conv(k);
        // does a contraction through layer i take fp16 pairs, and the products in front of it know nothing of its inputs' size?
        auto wants_zmax = [&](int i) { return tensor && i >= 1 && i < nv.L && !net.is_conv(i) && net.skip_of(i) < 0 && nv.qfl[i] > 0.f; };
        if (tk) NYB_TRY(launch_umma(e, net.umma_fwd[k], 2 * D, zl, (int)np, Fl, ldf, derr));   // zl rows, then zu rows
        else if (tconv) {
            // per-pixel products of the lower-end rows, then the upper-end rows, with [W+ | W-]; then the gather.  Slices of
            // domains bound the product space, which grows with the batch.
            const ConvGeom &g = net.geom[k];
            const int plane = g.ih * g.iw, N = 2 * g.oc * g.kh * g.kw;
            const size_t per = (size_t)2 * plane * N * 4;
            const int most = (int)std::min<size_t>({(size_t)D, std::max<size_t>(1, kConvColsMost / per), 0x7fffffffUL / (2UL * plane), 65535UL});   // (the gather's grid)
            float *cols = (float *)ws_get(e, "conv_cols", (size_t)most * per);
            if (!cols) return NYB200_ERR_OOM;
            for (int d0 = 0; d0 < D; d0 += most) {
                const int n = std::min(most, D - d0);
                const size_t at = (size_t)d0 * np;
                if (n == D) NYB_TRY(launch_umma(e, net.umma_fwd[k], 2 * D * plane, zl, (int)np, cols, N, derr, plane));
                else {
                    NYB_TRY(launch_umma(e, net.umma_fwd[k], n * plane, zl + at, (int)np, cols, N, derr, plane));
                    NYB_TRY(launch_umma(e, net.umma_fwd[k], n * plane, zu + at, (int)np, cols + (size_t)n * plane * N, N, derr, plane));
                }
                launch_ibp_conv_gather(e, nv, g, k, n, cols, umma_eps(g.ic, 1) * 1.000001, p.raw_lo + at, p.raw_hi + at, p.q + at, (long)np);
            }
        }
        else if (net.is_conv(k)) launch_ibp_conv(e, nv, net.geom[k], k, Deff, zl, zu, in_ds, p.raw_lo, p.raw_hi, p.q, (long)np);
        else launch_ibp_linear(e, nv, k, Deff, zl, zu, in_ds, p.raw_lo, p.raw_hi, p.q, (long)np);
        long raw_ds = (Deff == 1 && D > 1) ? 0 : (long)np;
        if (net.skip_of(k) >= 0)  // pre_k = W z + b + relu(pre_j): interval sum, outward
            launch_skip_interval(e, D, nv.dims[k + 1], (long)np, p.raw_lo, p.raw_hi, nv.pre_off[k], p.zl, p.zu,
                                 nv.pre_off[net.skip_of(k)]);
        launch_ibp_finish(e, nv, k, D, fwd_mode, p.raw_lo, p.raw_hi, raw_ds, fwd_mode >= 2 ? nullptr : p.inh_lo,
                          fwd_mode >= 2 ? nullptr : p.inh_hi, (long)b.inh_stride, p.code, p.sbeta, b.has_alpha ? p.alpha : nullptr, p.pre_lo,
                          p.pre_hi, p.zl, p.zu, p.tab, p.zabs, p.flags, tk ? Fl : nullptr, ldf,
                          tk ? umma_eps(nv.dims[k], 1) * 1.000001 : 0.0, p.q, tk ? fwd_tol : 0.f, cj, cj ? chain_cj_eps(net, nv.L, k) : 0.f, chain_kappa(),
                          wants_zmax(k) ? zmax_rows + (size_t)k * D : nullptr, wants_zmax(k + 1) ? zmax_rows + (size_t)(k + 1) * D : nullptr);
    }
    NYB_CUDA(e, cudaGetLastError());
    return NYB200_OK;
}

// Operands of the backward products A * W_k.  chain: what the fused chain and the contraction behind it read (every hidden
// layer that a chain can start at or pass, as TF32 pairs, and the first layer's own form); otherwise the own form of every
// layer, a convolution's being its window or the im2col-space operand W_col [oc x ic*kh*kw].
int prepare_backward_operands(nyb200_engine *e, Net &net, bool chain) {
    const NetView &nv = net.v;
    if (chain ? !net.umma_chain.empty() : net.umma_whole) return NYB200_OK;
    std::vector<UmmaLayer> own = net.umma, hidden((size_t)nv.L);
    std::vector<WinOp> win = net.win_bwd;
    own.resize(nv.L);
    win.resize(nv.L);
    NYB_TRY(build_operands(e, net, [&](Carve &c) -> int {
        for (int k = 0; k < nv.L; ++k) {
            const int K = nv.dims[k + 1], N = nv.dims[k];
            if (chain && k > 0) {
                if (chain_eligible(net, k + 1)) NYB_TRY(umma_prepare_layer(e, WeightSource{nv.W[k]}, K, N, &hidden[k], c));
                continue;
            }
            if (!net.umma.empty() && net.umma[k].ready()) continue;   // the first layer's, of an earlier set
            if (!net.is_conv(k)) { NYB_TRY(umma_prepare_own(e, WeightSource{nv.W[k]}, K, N, net.wmax[k], &own[k], c)); continue; }
            const ConvGeom &g = net.geom[k];
            NYB_TRY(win_prepare(e, nv.W[k], net.wmax[k], g, 0, &win[k], c));
            if (!win[k].ok) NYB_TRY(umma_prepare_layer(e, WeightSource{nv.W[k]}, g.oc, g.ic * g.kh * g.kw, &own[k], c));
        }
        return NYB200_OK;
    }));
    net.umma = std::move(own);
    net.win_bwd = std::move(win);
    if (chain) net.umma_chain = std::move(hidden);
    else net.umma_whole = true;
    return NYB200_OK;
}

int run_backward(nyb200_engine *e, Net &net, const Batch &b, BatchPtrs &p, float *const *ckpt, int ld_ckpt, int top) {
    const NetView &nv = net.v;
    const bool tensor = (e->path == NYB200_PATH_TF32X3);
    if (!tensor && e->fuse_chain && !ckpt && top < 0 && direct_eligible(net)) {
        const float clear[8] = {INFINITY, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        NYB_CUDA(e, cudaMemcpyAsync(p.min_lower, clear, sizeof(clear), cudaMemcpyHostToDevice, e->stream));
        return run_backward_direct(e, net, b, p, nullptr, b.D);
    }
    // top < 0: the whole network, seeded with the spec rows.  top >= 0: the pass starts at Linear_top's output
    // with one identity row per neuron (b.S = dims[top + 1]): the partial pass of the CROWN-IBP collection.
    const bool partial = top >= 0;
    int D = b.D, S = b.S, R = b.R, L = partial ? top + 1 : nv.L;
    // Fused chain: seed, identity pass and the contractions L-1 .. 1 with their relaxations run as one kernel that
    // keeps the rows on the SM; what is left for the loop below is Linear_0's (wide) contraction.
    const bool fused = tensor && e->fuse_chain && !ckpt && !b.steep && chain_eligible(net, L) && (nv.nps % 4 == 0) && (p.lda % 4 == 0);
    int *derr = nullptr;
    if (tensor) {
        NYB_TRY(prepare_backward_operands(e, net, fused));
        derr = (int *)ws_get(e, "umma_err", 256);
        if (!derr) return NYB200_ERR_OOM;
    }
    int M = D * R;
    long np = nv.nps;
    bool shared_box = (b.box_stride == 0 && D > 1);
    // rb, rabs, rpen and the safety flags: one fill when they lie back to back for this row count (they do unless the
    // pointers were taken over from a larger batch, as the re-evaluation of a subset does)
    if (p.rabs == p.rb + M && p.rpen == p.rb + 2 * (size_t)M && p.row_bad == (int *)(p.rb + 3 * (size_t)M)) {
        NYB_CUDA(e, cudaMemsetAsync(p.rb, 0, (size_t)M * 28, e->stream));
    } else {
        NYB_CUDA(e, cudaMemsetAsync(p.rb, 0, (size_t)M * 8, e->stream));
        NYB_CUDA(e, cudaMemsetAsync(p.rabs, 0, (size_t)M * 8, e->stream));
        NYB_CUDA(e, cudaMemsetAsync(p.rpen, 0, (size_t)M * 8, e->stream));
        NYB_CUDA(e, cudaMemsetAsync(p.row_bad, 0, (size_t)M * 4, e->stream));
    }
    static const float init_words[8] = {INFINITY, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};  // min lower; loose-domain counter at word 4
    NYB_CUDA(e, cudaMemcpyAsync(p.min_lower, init_words, sizeof(init_words), cudaMemcpyHostToDevice, e->stream));
    float *cur = p.A0, *nxt = p.A1;
    // Open identity branches (blocks may nest or overlap, several may start at the same variable): the coefficient
    // rows kept at a joining layer until the pass reaches the variable the branch starts from, one buffer per slot.
    struct OpenSkip { float *buf; int src; float *max; };
    std::vector<OpenSkip> open_skips;
    auto stash_slot = [&](size_t slot) -> float * {
        const std::string name = slot == 0 ? std::string("skip_coeff") : "skip_coeff_" + std::to_string(slot);
        return (float *)ws_get(e, name.c_str(), (size_t)M * p.lda * 4);
    };
    auto free_slot = [&]() {   // the first buffer no open branch is using
        size_t slot = 0;
        for (bool taken = true; taken; ) {
            taken = false;
            for (const OpenSkip &o : open_skips) if (o.buf == stash_slot(slot)) { taken = true; ++slot; break; }
        }
        return slot;
    };
    // Layers whose rows go through the relaxation straight into their convolution's operand (nyb200_winrelax.cu), 1: a window's
    // pairs, 2: pixel-major rows of an im2col-space product: the tables are the interval pass's (slopes in [0, 1], multipliers
    // the uploaded ones), nothing else reads the rows, and an identity branch is kept and joined in the same pixel order.  The second
    // form is for layers that a branch starts from, whose partner wants that order (the stem of a residual network): elsewhere planar
    // rows through k_relax_dom are as fast or faster (convolutional classifiers, 16 -> 32 channels, side 16: 512 domains 669 us a call
    // in pixels, 649 in planes, 1024 1054 / 1011; 8 -> 16, side 28: 512 domains 2948 / 2900, 16 domains 522 / 525).
    std::vector<char> image((size_t)L, 0);
    if (tensor && !fused && !ckpt && !partial && p.beta_max && !b.external_tables && !p.alpha_up && D <= 65535) {   // (grid)
        auto same_image = [&](int i, int j) { const ConvGeom &x = net.geom[i], &y = net.geom[j]; return net.is_conv(i) && net.is_conv(j) && x.oc == y.oc && x.oh == y.oh && x.ow == y.ow; };
        for (int k = 0; k < L - 1; ++k) {
            if (!net.is_conv(k) || net.geom[k].oc % 4 != 0 || net.geom[k].oc > 128) continue;
            if (net.win_bwd[k].ok) image[k] = net.win_bwd[k].in_cp <= 128 ? 1 : 0;
            else image[k] = net.skip_of(k) < 0 && std::find(net.skip.begin(), net.skip.end(), k) != net.skip.end() ? 2 : 0;
        }
        for (bool again = true; again; ) {
            again = false;
            std::vector<int> joins((size_t)L, 0);
            for (int k = 0; k < L; ++k) if (net.skip_of(k) >= 0) ++joins[net.skip_of(k)];
            for (int k = 0; k < L; ++k) {
                const int j = net.skip_of(k);
                if (j < 0 || (!image[k] && !image[j])) continue;
                if (image[k] && image[j] && joins[j] == 1 && same_image(k, j)) continue;
                image[k] = image[j] = 0;
                again = true;
            }
        }
    }
    // can layer k's window convolution leave its result in the order layer k - 1's image wants?
    auto pixel_result = [&](int k) {
        if (k == 0 || !image[k - 1] || !net.is_conv(k) || !net.win_bwd[k].ok || !net.win_bwd[k].pixel_out) return false;
        const ConvGeom &g = net.geom[k], &h = net.geom[k - 1];
        return g.ic == h.oc && g.ih == h.oh && g.iw == h.ow;
    };
    if (!fused) {
        if (partial) launch_seed_identity(e, S, D, p.lda, cur);
        else launch_seed(e, p.spec, S, nv.dims[L], D, p.lda, cur);
    }
    // rounding rate of the contraction through layer `lin` (accumulation length dims[lin + 1]); convolutions
    // accumulate in binary64 on both paths
    auto eps_for = [&](int lin) {
        // a transposed convolution on the tensor path accumulates oc products per im2col entry, adds the few
        // entries of an output in binary64 and casts the sum once: the contraction's rate at K = oc plus 2^-24
        int K = nv.dims[lin + 1];
        if (tensor && net.is_conv(lin) && net.win_bwd[lin].ok) return win_eps(net.win_bwd[lin]);
        if (tensor && net.is_conv(lin)) return (umma_eps(net.geom[lin].oc) + 5.97e-8) * 1.000001;
        if (tensor) return layer_eps(net.umma[lin], K) * 1.000001;
        return (double)(K + 2) * 1.1102230246251565e-16 * 1.000001;
    };
    auto q_ds = [&](int lin_k) { return (lin_k == 0 && shared_box) ? 0L : np; };
    // The concretisation rides in the epilogue of Linear_0's contraction when that contraction is a plain tensor-core
    // launch and nothing joins its result afterwards (no checkpoint, no identity branch ending at the input).
    const bool fuse_conc = tensor && e->fuse_chain && !ckpt && !net.is_conv(0) && (!net.umma[0].f16 || f16_segments(nv.dims[1]) == 1);
    int conc_slots = 0;
    double *conc_part = nullptr;
    int *conc_bad = nullptr;
    int k_start = L - 1;
    if (fused) {
        const bool timed = e->timing.per_kernel && !e->timing.cev_used;
        if (timed) {
            for (int i = 0; i < 2; ++i) if (!e->timing.cev[i]) cudaEventCreate(&e->timing.cev[i]);
            cudaEventRecord(e->timing.cev[0], e->stream);
        }
        NYB_TRY(launch_chain(e, net, b, p, L, partial, shared_box, cur, eps_for(0), derr));
        if (timed) { cudaEventRecord(e->timing.cev[1], e->stream); e->timing.cev_used = true; }
        k_start = 0;
    } else
        launch_relax(e, nv, -1, L - 1, M, R, S, cur, p.lda, p.tab, p.zabs, p.q, q_ds(L - 1), eps_for(L - 1), p.rb,
                     p.rabs, p.rpen, nullptr, 0);
    for (int k = k_start; k >= 0; --k) {
        NYB_DEADLINE(e, "backward pass");
        int K = nv.dims[k + 1], N = nv.dims[k];
        const float *zin_lo, *zin_hi;
        long zin_ds;
        if (k > 0) { zin_lo = p.zl + nv.pre_off[k - 1]; zin_hi = p.zu + nv.pre_off[k - 1]; zin_ds = np; }
        else { zin_lo = p.in_lo; zin_hi = p.in_hi; zin_ds = b.box_stride; }
        // With checkpoints the product (the coefficients entering ReLU k-1) is kept in its own buffer and
        // the relaxation writes its result into the ping-pong buffer instead of over its input.
        float *dst = (ckpt && k > 0) ? ckpt[k - 1] : nxt;
        int ldd = (ckpt && k > 0) ? ld_ckpt : p.lda;
        if (net.skip_of(k) >= 0 && !image[k]) {
            // residual block: these coefficients also multiply relu(pre_j) directly; keep them until the pass
            // reaches that variable (iteration j + 1 below)
            float *stash = stash_slot(free_slot());
            if (!stash) return NYB200_ERR_OOM;
            NYB_CUDA(e, cudaMemcpy2DAsync(stash, (size_t)p.lda * 4, cur, (size_t)p.lda * 4, (size_t)K * 4, (size_t)M,
                                          cudaMemcpyDeviceToDevice, e->stream));
            open_skips.push_back({stash, net.skip_of(k), nullptr});
        }
        const bool pixel = pixel_result(k), report = k > 0 && image[k - 1] == 1 && net.is_conv(k) && tensor && net.win_bwd[k].ok;
        if (e->timing.per_kernel) cudaEventRecord(next_kev(e->timing), e->stream);
        if (image[k] == 1) {   // its operand is there already (below, one layer earlier)
            void *hi, *lo;
            float *row_inv;
            unsigned *row_max;
            NYB_TRY(win_operand(e, net.win_bwd[k], M, &hi, &lo, &row_inv, &row_max));
            if (report) NYB_CUDA(e, cudaMemsetAsync(row_max, 0, (size_t)M * 4, e->stream));
            NYB_TRY(launch_win(e, net.win_bwd[k], M, hi, lo, row_inv, dst, ldd, derr, pixel, report ? row_max : nullptr));
        } else if (net.is_conv(k) && tensor && net.win_bwd[k].ok) {
            // window form: the row sum of the charge weights carries the share of fp16's exponent range
            NYB_WS(qsum, float *, e, "win_qsum", (size_t)D * 4);
            const bool one = q_ds(k) == 0;
            NYB_TRY(launch_sum_weights(e, one ? 1 : D, K, p.q + nv.pre_off[k], np, qsum));
            NYB_TRY(conv_win(e, net.win_bwd[k], M, cur, p.lda, dst, ldd, p.rpen, qsum, one ? M : R, derr, pixel, report));
        } else if (net.is_conv(k) && tensor) {
            // reshape (implicit: channel-strided operand) + GEMM with W_col on the tensor cores + col2im gather
            const ConvGeom &g = net.geom[k];
            const int plane = g.oh * g.ow, taps = g.ic * g.kh * g.kw;
            if ((long)M * plane > 0x7fffffffL) return set_err(e, NYB200_ERR_UNSUPPORTED, "batch too large for the convolution's im2col space");
            float *cols = (float *)ws_get(e, "conv_cols", (size_t)M * plane * taps * 4);
            if (!cols) return NYB200_ERR_OOM;
            if (image[k]) NYB_TRY(launch_umma(e, net.umma[k], M * plane, cur, g.oc, cols, taps, derr, plane, nullptr, true));
            else NYB_TRY(launch_umma(e, net.umma[k], M * plane, cur, p.lda, cols, taps, derr, plane));
            launch_col2im(e, g, M, cols, dst, ldd);
        } else if (net.is_conv(k)) {
            const ConvGeom &g = net.geom[k];
            size_t cols_bytes = (size_t)M * g.oh * g.ow * g.ic * g.kh * g.kw * 8;
            double *cols = nullptr;  // scratch for the GEMM form when it is affordable, else the direct kernel
            if ((long)M * g.oh * g.ow <= 0x7fffffffL && cols_bytes <= ((size_t)8 << 30)) {
                cols = (double *)ws_get(e, "conv_cols", cols_bytes);
                if (!cols) return NYB200_ERR_OOM;
            }
            launch_conv_transpose(e, g, M, cur, p.lda, dst, ldd, nv.W[k], R, zin_lo, zin_hi, zin_ds, p.rpen, cols);
        } else if (tensor && k == 0 && fuse_conc) {
            // the last contraction concretises in its epilogue: the finished rows are never written unless asked for
            ConcFuse cf;
            cf.on = 1; cf.store = p.keep_final ? 1 : 0; cf.R = R; cf.S = S;
            cf.slots = 2 * ((N + 255) / 256);
            cf.in_lo = p.in_lo; cf.in_hi = p.in_hi; cf.box_ds = b.box_stride;
            cf.part = (double *)ws_get(e, "conc_part", (size_t)M * cf.slots * 16);
            cf.bad = p.row_bad;   // cleared with the row scalars at the start of the pass
            if (!cf.part) return NYB200_ERR_OOM;
            NYB_TRY(launch_umma(e, net.umma[k], M, cur, p.lda, dst, ldd, derr, 0, &cf));
            conc_slots = cf.slots; conc_part = cf.part; conc_bad = cf.bad;
        } else if (tensor) {
            NYB_TRY(launch_umma(e, net.umma[k], M, cur, p.lda, dst, ldd, derr));
        } else {
            launch_gemm_f64(e, M, N, K, cur, p.lda, nv.W[k], N, dst, ldd, R, zin_lo, zin_hi, zin_ds, p.rpen);
        }
        if (e->timing.per_kernel) cudaEventRecord(next_kev(e->timing), e->stream);
        if (k > 0 && image[k - 1]) {
            const bool pairs = image[k - 1] == 1;
            ImageBranch join{nullptr, nullptr}, keep{nullptr, nullptr};
            for (size_t oi = 0; oi < open_skips.size(); ++oi)
                if (open_skips[oi].src == k - 1) { join = {open_skips[oi].buf, open_skips[oi].max}; break; }
            if (net.skip_of(k - 1) >= 0) {
                const size_t slot = free_slot();
                keep.rows = stash_slot(slot);
                keep.max = (float *)ws_get(e, ("skip_max_" + std::to_string(slot)).c_str(), (size_t)M * 4);
                if (!keep.rows || !keep.max) return NYB200_ERR_OOM;
            }
            void *hi = nullptr, *lo = nullptr;
            float *row_inv = nullptr;
            unsigned *row_max = nullptr;
            if (pairs) {
                NYB_TRY(win_operand(e, net.win_bwd[k - 1], M, &hi, &lo, &row_inv, &row_max));
                if (!report) NYB_TRY(row_maxima(e, M, N, dst, ldd, row_max));
            } else
                keep.rows = cur;   // (its rows have been read)
            NYB_TRY(launch_relax_image(e, net, k - 1, p, D, R, S, dst, pixel, row_max, q_ds(k - 1), eps_for(k - 1), join.rows ? &join : nullptr,
                                       keep.rows ? &keep : nullptr, hi, lo, row_inv));
            for (size_t oi = 0; oi < open_skips.size(); ++oi)
                if (open_skips[oi].src == k - 1) { open_skips.erase(open_skips.begin() + (long)oi); break; }
            if (!pairs) continue;   // the rows are in `cur`
            if (keep.rows) open_skips.push_back({keep.rows, net.skip_of(k - 1), keep.max});
            float *t = cur; cur = nxt; nxt = t;
            continue;
        }
        for (size_t oi = 0; oi < open_skips.size();) {  // dst holds the coefficients of relu(pre_{k-1}): add the identity branches
            if (open_skips[oi].src != k - 1) { ++oi; continue; }
            launch_skip_coeff(e, M, N, dst, ldd, open_skips[oi].buf, p.lda, R, p.zl, p.zu, np, nv.pre_off[k - 1], p.rpen);
            open_skips.erase(open_skips.begin() + (long)oi);
        }
        if (k > 0)
            launch_relax(e, nv, k - 1, k - 1, M, R, S, nxt, p.lda, p.tab, p.zabs, p.q, q_ds(k - 1), eps_for(k - 1), p.rb, p.rabs,
                         p.rpen, dst == nxt ? nullptr : dst, ldd, p.alpha_up, b.steep);
        float *t = cur; cur = nxt; nxt = t;
    }
    p.a_final = cur;
    if (conc_part)
        launch_concretize_fused(e, M, R, S, conc_slots, conc_part, conc_bad, p.rb, p.rabs, p.rpen, p.flags, p.out_lo, p.out_hi,
                                p.min_lower, tensor ? e->refine_tol : 0.f);
    else
        launch_concretize(e, M, R, S, nv.dims[0], cur, p.lda, p.in_lo, p.in_hi, b.box_stride, p.rb, p.rabs, p.rpen, p.flags,
                          p.out_lo, p.out_hi, p.min_lower, tensor ? e->refine_tol : 0.f);
    NYB_CUDA(e, cudaGetLastError());
    return NYB200_OK;
}

}  // namespace nyb

namespace {

int upload_batch(nyb200_engine *e, int32_t net_id, const float *spec, int32_t S, const float *in_lo, const float *in_hi,
                 int32_t box_stride, const float *inh_lo, const float *inh_hi, const nyb200_split *splits,
                 const int32_t *n_splits, int32_t max_splits, int32_t D, int32_t mode, const float *alpha, bool alpha_later = false) {
    Net *net;
    NYB_TRY(find_net(e, net_id, &net));
    const NetView &nv = net->v;
    if (D <= 0 || S <= 0) return set_err(e, NYB200_ERR_SHAPE, "D and S must be positive");
    if (!spec || !in_lo || !in_hi) return set_err(e, NYB200_ERR_INVALID, "null spec or input box");
    if (box_stride != 0 && box_stride != nv.dims[0]) return set_err(e, NYB200_ERR_SHAPE, "box_stride must be 0 or dims[0]");
    if (mode != 0 && mode != 1) return set_err(e, NYB200_ERR_INVALID, "mode must be 0 or 1");
    if (!inh_lo || !inh_hi) return set_err(e, NYB200_ERR_INVALID, "inherited bounds are required");
    if (max_splits < 0 || (max_splits > 0 && (!splits || !n_splits))) return set_err(e, NYB200_ERR_INVALID, "bad split list");
    if ((long)D * 2 * S > 0x7fffffffL / 64) return set_err(e, NYB200_ERR_UNSUPPORTED, "batch too large for one call");
    for (int d = 0; d < D && n_splits; ++d)
        if (n_splits[d] < 0 || n_splits[d] > max_splits) return set_err(e, NYB200_ERR_INVALID, "n_splits out of range");
    NYB_CUDA(e, cudaSetDevice(e->device));
    Batch b;
    b.net_id = net_id; b.S = S; b.R = 2 * S; b.D = D; b.mode = mode; b.box_stride = box_stride; b.max_splits = max_splits;
    b.has_alpha = alpha != nullptr;
    BatchPtrs p;
    NYB_TRY(batch_ptrs(e, *net, b, p));
    size_t np = nv.n_pre;
    size_t box = (size_t)nv.dims[0] * (box_stride ? (size_t)D : 1);
    const UploadPiece up[7] = {{p.in_lo, in_lo, box * 4}, {p.in_hi, in_hi, box * 4}, {p.inh_lo, inh_lo, np * 4}, {p.inh_hi, inh_hi, np * 4},
                               {p.nsplits, n_splits, max_splits > 0 ? (size_t)D * 4 : 0},
                               {p.splits, splits, (size_t)D * max_splits * sizeof(nyb200_split)},
                               {p.spec, spec, (size_t)S * nv.dims[nv.L] * 4}};
    NYB_TRY(staged_upload(e, up, 7));
    e->stage_out_valid = false;
    if (alpha && !alpha_later)
        NYB_TRY(upload_rows(e, p.alpha, (size_t)nv.nps * 4, alpha, np * 4, (size_t)D, e->stream));
    b.valid = true;
    e->batch = b;
    return NYB200_OK;
}

// Last kernel of a batch run: folds the run's pipeline error word and flagged-domain count into the engine's sticky
// accumulators and publishes them, then the run's sequence number, to mapped host memory (writes only: the device
// never reads across the bus).
__global__ void k_publish_status(const int *__restrict__ derr, const int *__restrict__ loose, int *__restrict__ acc,
                                 volatile int *status, int seq, int *__restrict__ err_word) {
    pdl_wait();
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    const int h = derr ? *derr : 0, l = loose ? *loose : 0;
    *err_word = h;   // travels to the host with the results
    if (h) acc[0] = h;
    acc[1] += l;
    status[1] = acc[0];
    status[2] = acc[1];
    __threadfence_system();
    status[0] = seq;
}

// late_alpha: the batch's slopes, still in the caller's array.  Bounds do not depend on them: they cross the bus beside the interval
// pass, on a stream of their own, and are put into its tables when both are done (777 domains of 9 x 512, 14 MB: 1460 -> 1260 us a call).
int run_batch(nyb200_engine *e, const float *late_alpha = nullptr) {
    if (!e->batch.valid) return set_err(e, NYB200_ERR_INVALID, "no batch uploaded");
    if (!e->status_host) {
        NYB_CUDA(e, cudaHostAlloc((void **)&e->status_host, 64, cudaHostAllocMapped));
        memset(e->status_host, 0, 64);
        NYB_CUDA(e, cudaHostGetDevicePointer((void **)&e->status_dev, e->status_host, 0));
        int *acc0 = (int *)ws_get(e, "status_acc", 256);
        if (!acc0) return NYB200_ERR_OOM;
        NYB_CUDA(e, cudaMemsetAsync(acc0, 0, 8, e->stream));
    }
    Net *net;
    NYB_TRY(find_net(e, e->batch.net_id, &net));
    BatchPtrs p;
    NYB_TRY(batch_ptrs(e, *net, e->batch, p));
    Timing &t = e->timing;
    fold_timing(t);  // the previous run's events are about to be reused
    const bool direct = !e->batch.external_tables && ((e->path == NYB200_PATH_F64 && e->fuse_chain && direct_eligible(*net)) || direct_pays(e, *net, e->batch.S, e->batch.D));
    const bool tensor = e->path == NYB200_PATH_TF32X3 && !direct;
    if (tensor) {
        int *derr = (int *)ws_get(e, "umma_err", 256);
        if (!derr) return NYB200_ERR_OOM;
        NYB_CUDA(e, cudaMemsetAsync(derr, 0, 4, e->stream));
    }
    cudaEventRecord(t.ev[0], e->stream);
    if (direct) NYB_TRY(run_forward_direct(e, *net, e->batch, p, e->batch.mode, nullptr, e->batch.D));
    else if (late_alpha) {
        if (!e->side) {
            NYB_CUDA(e, cudaStreamCreateWithFlags(&e->side, cudaStreamNonBlocking));
            for (cudaEvent_t &ev : e->side_ev) NYB_CUDA(e, cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
        }
        NYB_CUDA(e, cudaEventRecord(e->side_ev[0], e->stream));   // the slopes' place may still be read by earlier work
        NYB_CUDA(e, cudaStreamWaitEvent(e->side, e->side_ev[0], 0));
        Batch plain = e->batch;
        plain.has_alpha = false;
        NYB_TRY(run_forward(e, *net, plain, p, e->batch.mode));
        NYB_TRY(upload_rows(e, p.alpha, (size_t)net->v.nps * 4, late_alpha, (size_t)net->v.n_pre * 4, (size_t)e->batch.D, e->side));
        NYB_CUDA(e, cudaEventRecord(e->side_ev[1], e->side));
        NYB_CUDA(e, cudaStreamWaitEvent(e->stream, e->side_ev[1], 0));
        launch_apply_alpha(e, net->v, e->batch.D, p.alpha, p.code, p.pre_lo, p.pre_hi, p.tab);
    } else NYB_TRY(run_forward(e, *net, e->batch, p, e->batch.mode));
    cudaEventRecord(t.ev[1], e->stream);
    if (direct) NYB_TRY(run_backward_direct(e, *net, e->batch, p, nullptr, e->batch.D));
    else NYB_TRY(run_backward(e, *net, e->batch, p, nullptr, 0));
    cudaEventRecord(t.ev[2], e->stream);
    e->batch.direct = direct;
    {
        int *acc = (int *)ws_get(e, "status_acc", 256);
        launch_pdl(k_publish_status, dim3(1), dim3(32), 0, e, tensor ? (const int *)ws_get(e, "umma_err", 256) : (const int *)nullptr,
                   tensor && e->refine_tol > 0.f ? (const int *)p.min_lower + 4 : (const int *)nullptr, acc, (volatile int *)e->status_dev,
                   ++e->run_seq, (int *)p.min_lower + 5);
        e->launches++;
        NYB_CUDA(e, cudaGetLastError());
    }
    t.pending = true;
    e->batch.ran = true;
    e->batch.finished = false;
    e->batch.optimized = false;
    e->batch.dual_alpha = false;
    e->batch.refined = 0;
    return NYB200_OK;
}

// Binary64 re-evaluation of the flagged domains only.  Their inputs (split lists, slopes, boxes) are gathered into
// a compact sub-batch that runs through the same scratch arrays; the arrays of the full batch that later calls
// read (bounds, flags, pre-activation bounds, split codes) are saved first, receive the sub-batch's rows, and are
// put back.
int refine_subset(nyb200_engine *e, Net &net, BatchPtrs &p) {
    const Batch &b = e->batch;
    const NetView &nv = net.v;
    const int D = b.D, S = b.S;
    const size_t np = nv.nps;
    cudaStream_t st = e->stream;
    std::vector<int> flags((size_t)D), idx;
    NYB_CUDA(e, cudaMemcpyAsync(flags.data(), p.flags, (size_t)D * 4, cudaMemcpyDeviceToHost, st));
    NYB_CUDA(e, cudaStreamSynchronize(st));
    for (int d = 0; d < D; ++d)
        if ((flags[d] & (kFlagLoose | kFlagLooseFwd)) && !(flags[d] & (kFlagInfeasible | kFlagDegraded | kFlagInvalid))) idx.push_back(d);
    const int Ds = (int)idx.size();
    if (Ds == 0) return NYB200_OK;
    const int ms = b.max_splits > 0 ? b.max_splits : 0;
    NYB_WS(didx, int *, e, "sub_idx", (size_t)Ds * 4);
    NYB_WS(keep_lo, float *, e, "keep_out_lo", (size_t)D * S * 4);
    NYB_WS(keep_hi, float *, e, "keep_out_hi", (size_t)D * S * 4);
    NYB_WS(keep_fl, int *, e, "keep_flags", (size_t)D * 4);
    NYB_WS(keep_pl, float *, e, "keep_pre_lo", (size_t)D * np * 4);
    NYB_WS(keep_pu, float *, e, "keep_pre_hi", (size_t)D * np * 4);
    NYB_WS(keep_code, signed char *, e, "keep_code", (size_t)D * np);
    NYB_WS(keep_tab, float4 *, e, "keep_tab", (size_t)D * np * 16);
    NYB_WS(sub_ns, int *, e, "sub_nsplits", (size_t)Ds * 4);
    NYB_WS(sub_sp, nyb200_split *, e, "sub_splits", (size_t)Ds * (ms > 0 ? ms : 1) * sizeof(nyb200_split));
    NYB_CUDA(e, cudaMemcpyAsync(didx, idx.data(), (size_t)Ds * 4, cudaMemcpyHostToDevice, st));
    NYB_CUDA(e, cudaMemcpyAsync(keep_lo, p.out_lo, (size_t)D * S * 4, cudaMemcpyDeviceToDevice, st));
    NYB_CUDA(e, cudaMemcpyAsync(keep_hi, p.out_hi, (size_t)D * S * 4, cudaMemcpyDeviceToDevice, st));
    NYB_CUDA(e, cudaMemcpyAsync(keep_fl, p.flags, (size_t)D * 4, cudaMemcpyDeviceToDevice, st));
    NYB_CUDA(e, cudaMemcpyAsync(keep_pl, p.pre_lo, (size_t)D * np * 4, cudaMemcpyDeviceToDevice, st));
    NYB_CUDA(e, cudaMemcpyAsync(keep_pu, p.pre_hi, (size_t)D * np * 4, cudaMemcpyDeviceToDevice, st));
    NYB_CUDA(e, cudaMemcpyAsync(keep_code, p.code, (size_t)D * np, cudaMemcpyDeviceToDevice, st));
    NYB_CUDA(e, cudaMemcpyAsync(keep_tab, p.tab, (size_t)D * np * 16, cudaMemcpyDeviceToDevice, st));
    BatchPtrs ps = p;
    Batch bs = b;
    bs.D = Ds;
    launch_gather_rows(e, sub_ns, p.nsplits, didx, Ds, 1);
    ps.nsplits = sub_ns;
    if (ms > 0) {
        launch_gather_rows(e, sub_sp, p.splits, didx, Ds, (long)ms * (long)(sizeof(nyb200_split) / 4));
        ps.splits = sub_sp;
    }
    if (b.has_alpha) {
        NYB_WS(sub_alpha, float *, e, "sub_alpha", (size_t)Ds * np * 4);
        launch_gather_rows(e, sub_alpha, p.alpha, didx, Ds, (long)np);
        ps.alpha = sub_alpha;
    }
    if (b.inh_stride) {
        NYB_WS(sub_il, float *, e, "sub_inh_lo", (size_t)Ds * np * 4);
        NYB_WS(sub_iu, float *, e, "sub_inh_hi", (size_t)Ds * np * 4);
        launch_gather_rows(e, sub_il, p.inh_lo, didx, Ds, (long)np);
        launch_gather_rows(e, sub_iu, p.inh_hi, didx, Ds, (long)np);
        ps.inh_lo = sub_il; ps.inh_hi = sub_iu;
    }
    if (b.box_stride) {
        NYB_WS(sub_lo, float *, e, "sub_in_lo", (size_t)Ds * nv.dims[0] * 4);
        NYB_WS(sub_hi, float *, e, "sub_in_hi", (size_t)Ds * nv.dims[0] * 4);
        launch_gather_rows(e, sub_lo, p.in_lo, didx, Ds, nv.dims[0]);
        launch_gather_rows(e, sub_hi, p.in_hi, didx, Ds, nv.dims[0]);
        ps.in_lo = sub_lo; ps.in_hi = sub_hi;
    }
    e->path = NYB200_PATH_F64;
    int rc = run_forward(e, net, bs, ps, bs.mode);
    if (rc == NYB200_OK) rc = run_backward(e, net, bs, ps, nullptr, 0);
    e->path = NYB200_PATH_TF32X3;
    NYB_TRY(rc);
    // rows of the sub-batch go to their places in the saved arrays, which then replace the scratch arrays
    launch_scatter_rows(e, keep_lo, ps.out_lo, didx, Ds, S);
    launch_scatter_rows(e, keep_hi, ps.out_hi, didx, Ds, S);
    launch_scatter_rows(e, keep_fl, ps.flags, didx, Ds, 1);
    launch_scatter_rows(e, keep_pl, ps.pre_lo, didx, Ds, (long)np);
    launch_scatter_rows(e, keep_pu, ps.pre_hi, didx, Ds, (long)np);
    launch_scatter_rows(e, keep_tab, ps.tab, didx, Ds, (long)np * 4);
    NYB_CUDA(e, cudaMemcpyAsync(p.out_lo, keep_lo, (size_t)D * S * 4, cudaMemcpyDeviceToDevice, st));
    NYB_CUDA(e, cudaMemcpyAsync(p.out_hi, keep_hi, (size_t)D * S * 4, cudaMemcpyDeviceToDevice, st));
    NYB_CUDA(e, cudaMemcpyAsync(p.flags, keep_fl, (size_t)D * 4, cudaMemcpyDeviceToDevice, st));
    NYB_CUDA(e, cudaMemcpyAsync(p.pre_lo, keep_pl, (size_t)D * np * 4, cudaMemcpyDeviceToDevice, st));
    NYB_CUDA(e, cudaMemcpyAsync(p.pre_hi, keep_pu, (size_t)D * np * 4, cudaMemcpyDeviceToDevice, st));
    NYB_CUDA(e, cudaMemcpyAsync(p.code, keep_code, (size_t)D * np, cudaMemcpyDeviceToDevice, st));
    NYB_CUDA(e, cudaMemcpyAsync(p.tab, keep_tab, (size_t)D * np * 16, cudaMemcpyDeviceToDevice, st));
    launch_min_lower(e, D, S, p.out_lo, p.flags, p.min_lower);
    NYB_CUDA(e, cudaGetLastError());
    return NYB200_OK;
}

// Completes the last run: waits for it and, if the fast path reported domains whose rounding penalty
// is visible at the requested tolerance, evaluates the batch again with binary64 contractions.
// prefetch: the caller is about to read the bounds and flags; they travel to the pinned output region ahead of the
// synchronisation (and stay valid there unless a re-evaluation replaces them).
int finish_batch(nyb200_engine *e, bool prefetch = false) {
    if (!e->batch.valid || !e->batch.ran) return set_err(e, NYB200_ERR_INVALID, "no batch has been run");
    if (e->batch.finished) return NYB200_OK;
    Net *net;
    NYB_TRY(find_net(e, e->batch.net_id, &net));
    BatchPtrs p;
    NYB_TRY(batch_ptrs(e, *net, e->batch, p));
    const size_t nout = result_bytes(e->batch.D, e->batch.S);
    int local[8] = {0};
    const bool staged = ensure_stage(e, 256 + nout) == NYB200_OK;
    int *hw = staged ? (int *)(e->stage + kStageIn) : local;   // the run's words: [4] flagged domains, [5] pipeline error
    e->stage_out_valid = false;
    NYB_CUDA(e, cudaMemcpyAsync(hw, p.min_lower, staged && prefetch ? nout : 32, cudaMemcpyDeviceToHost, e->stream));
    int opt_err = 0;
    if (e->path == NYB200_PATH_TF32X3 && e->batch.optimized)   // an optimisation's last kernel does not leave the error word there
        if (int *derr = (int *)ws_get(e, "umma_err", 256)) NYB_CUDA(e, cudaMemcpyAsync(&opt_err, derr, 4, cudaMemcpyDeviceToHost, e->stream));
    NYB_CUDA(e, cudaStreamSynchronize(e->stream));
    int loose = 0, herr = 0;
    if (e->path == NYB200_PATH_TF32X3) {
        if (!e->batch.direct) loose = hw[4];
        herr = e->batch.optimized ? opt_err : hw[5];   // (a direct optimisation's adjoint products are the tensor path's)
    }
    const bool will_refine = loose > 0 && e->path == NYB200_PATH_TF32X3 && e->refine_tol > 0.f;
    e->stage_out_valid = staged && prefetch && !herr && !will_refine;
    if (e->status_host) {  // the stream is idle: whatever earlier runs latched is handled by this call
        int *acc = (int *)ws_get(e, "status_acc", 256);
        if (acc) NYB_CUDA(e, cudaMemsetAsync(acc, 0, 8, e->stream));
        e->status_host[1] = e->status_host[2] = 0;
    }
    if (herr) return set_err(e, NYB200_ERR_INTERNAL, "tcgen05 pipeline wait expired (code " + std::to_string(herr) + ")");
    if (loose > 0 && e->path == NYB200_PATH_TF32X3 && e->refine_tol > 0.f && e->batch.optimized) {
        NYB_TRY(refine_optimized(e, *net, e->batch, p, loose));
        NYB_CUDA(e, cudaStreamSynchronize(e->stream));
        e->batch.refined = loose;
    } else if (loose > 0 && e->path == NYB200_PATH_TF32X3 && e->refine_tol > 0.f) {
        const Batch &b = e->batch;
        int st;
        if (direct_eligible(*net)) {   // in place: only the flagged domains' rows are touched
            int *idx = nullptr;
            st = flagged_domains(e, b.D, p.flags, loose, &idx);
            if (st == NYB200_OK) st = run_forward_direct(e, *net, b, p, b.mode, idx, loose);
            if (st == NYB200_OK) st = run_backward_direct(e, *net, b, p, idx, loose);
        } else if (2 * loose >= b.D) {  // most of the batch is flagged: evaluate all of it again
            e->path = NYB200_PATH_F64;
            st = run_forward(e, *net, b, p, b.mode);
            if (st == NYB200_OK) st = run_backward(e, *net, b, p, nullptr, 0);
            e->path = NYB200_PATH_TF32X3;
        } else {
            st = refine_subset(e, *net, p);
        }
        NYB_TRY(st);
        NYB_CUDA(e, cudaStreamSynchronize(e->stream));
        e->batch.refined = loose;
    }
    if (e->batch.direct && e->path == NYB200_PATH_TF32X3 && e->refine_tol > 0.f && !e->batch.decision_thr) e->batch.refined = e->batch.D;
    e->batch.finished = true;
    return NYB200_OK;
}

int download_batch(nyb200_engine *e, float *out_lo, float *out_hi, int32_t *infeasible) {
    NYB_TRY(finish_batch(e, true));
    if (e->stage_out_valid) {   // the results are already on the host
        const size_t nres = (size_t)e->batch.D * e->batch.S * 4, nfl = (size_t)e->batch.D * 4;
        const unsigned char *o = e->stage + kStageIn + 256, *r = e->stage + kStageIn + result_bytes(e->batch.D, 0);
        if (out_lo) memcpy(out_lo, r, nres);
        if (out_hi) memcpy(out_hi, r + nres, nres);
        if (infeasible) {
            memcpy(infeasible, o, nfl);
            for (int d = 0; d < e->batch.D; ++d) {
                if (infeasible[d] & kFlagInvalid) return set_err(e, NYB200_ERR_INVALID, "split entry out of range");
                infeasible[d] = (infeasible[d] & kFlagInfeasible) ? 1 : 0;
            }
        }
        return NYB200_OK;
    }
    Net *net;
    NYB_TRY(find_net(e, e->batch.net_id, &net));
    BatchPtrs p;
    NYB_TRY(batch_ptrs(e, *net, e->batch, p));
    size_t n = (size_t)e->batch.D * e->batch.S;
    if (out_lo) NYB_CUDA(e, cudaMemcpyAsync(out_lo, p.out_lo, n * 4, cudaMemcpyDeviceToHost, e->stream));
    if (out_hi) NYB_CUDA(e, cudaMemcpyAsync(out_hi, p.out_hi, n * 4, cudaMemcpyDeviceToHost, e->stream));
    if (infeasible) NYB_CUDA(e, cudaMemcpyAsync(infeasible, p.flags, (size_t)e->batch.D * 4, cudaMemcpyDeviceToHost, e->stream));
    NYB_CUDA(e, cudaStreamSynchronize(e->stream));
    if (infeasible) {
        for (int d = 0; d < e->batch.D; ++d) {
            if (infeasible[d] & kFlagInvalid) return set_err(e, NYB200_ERR_INVALID, "split entry out of range");
            infeasible[d] = (infeasible[d] & kFlagInfeasible) ? 1 : 0;
        }
    }
    return NYB200_OK;
}

}  // namespace

namespace nyb {
int finish_batch_public(nyb200_engine *e) { return finish_batch(e); }
int run_batch_public(nyb200_engine *e) { return run_batch(e); }
}

extern "C" {

int32_t nyb200_batch_upload(nyb200_engine *e, int32_t net_id, const float *spec, int32_t S, const float *in_lo,
                            const float *in_hi, int32_t box_stride, const float *inh_lo, const float *inh_hi,
                            const nyb200_split *splits, const int32_t *n_splits, int32_t max_splits, int32_t D,
                            int32_t mode, const float *alpha) {
    if (!e) return NYB200_ERR_INVALID;
    std::lock_guard<std::mutex> g(e->mu);
    return upload_batch(e, net_id, spec, S, in_lo, in_hi, box_stride, inh_lo, inh_hi, splits, n_splits, max_splits, D, mode,
                        alpha);
}

int32_t nyb200_batch_set_thresholds(nyb200_engine *e, const float *thresholds, int32_t S) {
    if (!e) return NYB200_ERR_INVALID;
    std::lock_guard<std::mutex> g(e->mu);
    NYB_CUDA(e, cudaSetDevice(e->device));
    if (!thresholds) { e->batch.decision_thr = nullptr; return NYB200_OK; }
    if (!e->batch.valid) return set_err(e, NYB200_ERR_INVALID, "no batch uploaded");
    if (S != e->batch.S) return set_err(e, NYB200_ERR_SHAPE, "one threshold per specification row of the batch");
    NYB_WS(dt, float *, e, "decision_thr", (size_t)S * 4);
    NYB_CUDA(e, cudaMemcpyAsync(dt, thresholds, (size_t)S * 4, cudaMemcpyHostToDevice, e->stream));
    NYB_CUDA(e, cudaStreamSynchronize(e->stream));   // the caller's array may go away
    e->batch.decision_thr = dt;
    return NYB200_OK;
}

int32_t nyb200_batch_set_inherited(nyb200_engine *e, const float *inh_lo, const float *inh_hi) {
    if (!e || !inh_lo || !inh_hi) return NYB200_ERR_INVALID;
    std::lock_guard<std::mutex> g(e->mu);
    NYB_CUDA(e, cudaSetDevice(e->device));
    if (!e->batch.valid) return set_err(e, NYB200_ERR_INVALID, "no batch uploaded");
    Net *net;
    NYB_TRY(find_net(e, e->batch.net_id, &net));
    const NetView &nv = net->v;
    e->batch.inh_stride = nv.nps;
    BatchPtrs p;
    NYB_TRY(batch_ptrs(e, *net, e->batch, p));
    const size_t w = (size_t)nv.n_pre * 4, pitch = (size_t)nv.nps * 4;
    NYB_CUDA(e, cudaMemsetAsync(p.inh_lo, 0, (size_t)e->batch.D * pitch, e->stream));
    NYB_CUDA(e, cudaMemsetAsync(p.inh_hi, 0, (size_t)e->batch.D * pitch, e->stream));
    NYB_TRY(upload_rows(e, p.inh_lo, pitch, inh_lo, w, (size_t)e->batch.D, e->stream));
    NYB_TRY(upload_rows(e, p.inh_hi, pitch, inh_hi, w, (size_t)e->batch.D, e->stream));
    NYB_CUDA(e, cudaStreamSynchronize(e->stream));
    e->batch.ran = false;
    e->batch.finished = false;
    return NYB200_OK;
}

int32_t nyb200_batch_run(nyb200_engine *e) {
    if (!e) return NYB200_ERR_INVALID;
    std::lock_guard<std::mutex> g(e->mu);
    NYB_CUDA(e, cudaSetDevice(e->device));
    return run_batch(e);
}

int32_t nyb200_batch_download(nyb200_engine *e, float *out_lo, float *out_hi, int32_t *infeasible) {
    if (!e) return NYB200_ERR_INVALID;
    std::lock_guard<std::mutex> g(e->mu);
    NYB_CUDA(e, cudaSetDevice(e->device));
    return download_batch(e, out_lo, out_hi, infeasible);
}

int32_t nyb200_bab_bound_batch(nyb200_engine *e, int32_t net_id, const float *spec, int32_t S, const float *in_lo,
                               const float *in_hi, int32_t box_stride, const float *inh_lo, const float *inh_hi,
                               const nyb200_split *splits, const int32_t *n_splits, int32_t max_splits, int32_t D,
                               int32_t mode, const float *alpha, float *out_lo, float *out_hi, int32_t *infeasible) {
    if (!e || !out_lo || !out_hi) return NYB200_ERR_INVALID;
    std::lock_guard<std::mutex> g(e->mu);
    // many slopes on the tensor path: after the interval pass (run_batch); fewer than a slot of the upload's lanes cost less than the
    // second stream
    Net *net;
    NYB_TRY(find_net(e, net_id, &net));
    const bool later = alpha && D > 0 && S > 0 && (size_t)D * net->v.n_pre * 4 >= kLaneSlot && e->path == NYB200_PATH_TF32X3 && !direct_pays(e, *net, S, D);
    NYB_TRY(upload_batch(e, net_id, spec, S, in_lo, in_hi, box_stride, inh_lo, inh_hi, splits, n_splits, max_splits, D, mode,
                         alpha, later));
    const int st = run_batch(e, later ? alpha : nullptr);
    if (later && st != NYB200_OK) {
        // A run that was given up (a deadline) leaves the batch resident, as where the slopes went ahead of it: they follow now, from
        // an array that may go away behind this call.
        const std::string why = e->err;
        BatchPtrs p;
        const bool there = (!e->side || cudaStreamSynchronize(e->side) == cudaSuccess) && batch_ptrs(e, *net, e->batch, p) == NYB200_OK &&
                           upload_rows(e, p.alpha, (size_t)net->v.nps * 4, alpha, (size_t)net->v.n_pre * 4, (size_t)D, e->stream) == NYB200_OK &&
                           cudaStreamSynchronize(e->stream) == cudaSuccess;
        if (!there) e->batch.valid = false;
        return set_err(e, st, why);
    }
    NYB_TRY(st);
    return download_batch(e, out_lo, out_hi, infeasible);
}

int32_t nyb200_batch_min_lower_device(nyb200_engine *e, void **dev_ptr) {
    if (!e || !dev_ptr) return NYB200_ERR_INVALID;
    std::lock_guard<std::mutex> g(e->mu);
    if (!e->batch.valid) return set_err(e, NYB200_ERR_INVALID, "no batch uploaded");
    void *p = ws_get(e, "results", 256);   // the first word of the results
    if (!p) return NYB200_ERR_OOM;
    *dev_ptr = p;
    return NYB200_OK;
}

int32_t nyb200_batch_min_lower(nyb200_engine *e, float *min_lower) {
    if (!e || !min_lower) return NYB200_ERR_INVALID;
    std::lock_guard<std::mutex> g(e->mu);
    NYB_CUDA(e, cudaSetDevice(e->device));
    NYB_TRY(finish_batch(e));
    void *p = ws_get(e, "results", 256);
    if (!p) return NYB200_ERR_OOM;
    NYB_CUDA(e, cudaMemcpyAsync(min_lower, p, 4, cudaMemcpyDeviceToHost, e->stream));
    NYB_CUDA(e, cudaStreamSynchronize(e->stream));
    return NYB200_OK;
}

int32_t nyb200_batch_download_pre_bounds(nyb200_engine *e, float *pre_lo, float *pre_hi) {
    if (!e || !pre_lo || !pre_hi) return NYB200_ERR_INVALID;
    std::lock_guard<std::mutex> g(e->mu);
    NYB_CUDA(e, cudaSetDevice(e->device));
    NYB_TRY(finish_batch(e));
    Net *net;
    NYB_TRY(find_net(e, e->batch.net_id, &net));
    BatchPtrs p;
    NYB_TRY(batch_ptrs(e, *net, e->batch, p));
    size_t w = (size_t)net->v.n_pre * 4, ws = (size_t)net->v.nps * 4;
    NYB_CUDA(e, cudaMemcpy2DAsync(pre_lo, w, p.pre_lo, ws, w, (size_t)e->batch.D, cudaMemcpyDeviceToHost, e->stream));
    NYB_CUDA(e, cudaMemcpy2DAsync(pre_hi, w, p.pre_hi, ws, w, (size_t)e->batch.D, cudaMemcpyDeviceToHost, e->stream));
    NYB_CUDA(e, cudaStreamSynchronize(e->stream));
    return NYB200_OK;
}

int32_t nyb200_batch_verdicts(nyb200_engine *e, float threshold, int32_t *status) {
    if (!e || !status) return NYB200_ERR_INVALID;
    std::lock_guard<std::mutex> g(e->mu);
    NYB_CUDA(e, cudaSetDevice(e->device));
    NYB_TRY(finish_batch(e));
    Net *net;
    NYB_TRY(find_net(e, e->batch.net_id, &net));
    BatchPtrs p;
    NYB_TRY(batch_ptrs(e, *net, e->batch, p));
    int D = e->batch.D;
    NYB_WS(ds, int *, e, "verdicts", (size_t)D * 4);
    launch_verdicts(e, D, e->batch.S, p.out_lo, p.out_hi, p.flags, threshold, ds);
    NYB_CUDA(e, cudaGetLastError());
    NYB_CUDA(e, cudaMemcpyAsync(status, ds, (size_t)D * 4, cudaMemcpyDeviceToHost, e->stream));
    NYB_CUDA(e, cudaStreamSynchronize(e->stream));
    return NYB200_OK;
}

int32_t nyb200_batch_select_branch(nyb200_engine *e, int32_t *relu, int32_t *neuron, float *width) {
    return nyb200_batch_select_branch_scored(e, NYB200_BRANCH_WIDTH, relu, neuron, width);
}

int32_t nyb200_batch_select_branch_scored(nyb200_engine *e, int32_t kind, int32_t *relu, int32_t *neuron, float *width) {
    if (!e || !relu || !neuron) return NYB200_ERR_INVALID;
    std::lock_guard<std::mutex> g(e->mu);
    if (kind != NYB200_BRANCH_WIDTH && kind != NYB200_BRANCH_INTERCEPT && kind != NYB200_BRANCH_BABSR)
        return set_err(e, NYB200_ERR_INVALID, "unknown branching score");
    NYB_CUDA(e, cudaSetDevice(e->device));
    NYB_TRY(finish_batch(e));
    Net *net;
    NYB_TRY(find_net(e, e->batch.net_id, &net));
    BatchPtrs p;
    NYB_TRY(batch_ptrs(e, *net, e->batch, p));
    int D = e->batch.D;
    NYB_WS(dr, int *, e, "br_relu", (size_t)D * 4);
    NYB_WS(dn, int *, e, "br_neuron", (size_t)D * 4);
    NYB_WS(dw, float *, e, "br_width", (size_t)D * 4);
    if (kind == NYB200_BRANCH_BABSR) NYB_TRY(babsr_select(e, *net, e->batch, p, dr, dn, dw, nullptr));
    else launch_select_branch(e, net->v, D, p.pre_lo, p.pre_hi, p.code, dr, dn, dw, kind);
    NYB_CUDA(e, cudaGetLastError());
    NYB_CUDA(e, cudaMemcpyAsync(relu, dr, (size_t)D * 4, cudaMemcpyDeviceToHost, e->stream));
    NYB_CUDA(e, cudaMemcpyAsync(neuron, dn, (size_t)D * 4, cudaMemcpyDeviceToHost, e->stream));
    if (width) NYB_CUDA(e, cudaMemcpyAsync(width, dw, (size_t)D * 4, cudaMemcpyDeviceToHost, e->stream));
    NYB_CUDA(e, cudaStreamSynchronize(e->stream));
    return NYB200_OK;
}

int32_t nyb200_batch_download_branch_scores(nyb200_engine *e, float *scores, float *backup) {
    if (!e || !scores) return NYB200_ERR_INVALID;
    std::lock_guard<std::mutex> g(e->mu);
    NYB_CUDA(e, cudaSetDevice(e->device));
    if (!e->batch.valid || !e->batch.ran) return set_err(e, NYB200_ERR_INVALID, "no batch has been run");
    Net *net;
    NYB_TRY(find_net(e, e->batch.net_id, &net));
    auto it = e->ws.find("babsr_score");
    const NetView &nv = net->v;
    if (it == e->ws.end() || it->second.bytes < (size_t)2 * e->batch.D * nv.nps * 4)
        return set_err(e, NYB200_ERR_INVALID, "no BaBSR selection has been made for this batch");
    size_t w = (size_t)nv.n_pre * 4;
    NYB_CUDA(e, cudaMemcpy2DAsync(scores, w, it->second.p, (size_t)nv.nps * 4, w, (size_t)e->batch.D, cudaMemcpyDeviceToHost, e->stream));
    if (backup)
        NYB_CUDA(e, cudaMemcpy2DAsync(backup, w, (const float *)it->second.p + (size_t)e->batch.D * nv.nps, (size_t)nv.nps * 4, w,
                                      (size_t)e->batch.D, cudaMemcpyDeviceToHost, e->stream));
    NYB_CUDA(e, cudaStreamSynchronize(e->stream));
    return NYB200_OK;
}

int32_t nyb200_ibp_forward(nyb200_engine *e, int32_t net_id, int32_t D, const float *in_lo, const float *in_hi,
                           int32_t box_stride, float *pre_lo, float *pre_hi) {
    if (!e || !in_lo || !in_hi || !pre_lo || !pre_hi) return NYB200_ERR_INVALID;
    std::lock_guard<std::mutex> g(e->mu);
    Net *net;
    NYB_TRY(find_net(e, net_id, &net));
    const NetView &nv = net->v;
    if (D <= 0) return set_err(e, NYB200_ERR_SHAPE, "D must be positive");
    if (box_stride != 0 && box_stride != nv.dims[0]) return set_err(e, NYB200_ERR_SHAPE, "box_stride must be 0 or dims[0]");
    NYB_CUDA(e, cudaSetDevice(e->device));
    Batch b;
    b.net_id = net_id; b.S = 1; b.R = 2; b.D = D; b.mode = 1; b.box_stride = box_stride; b.max_splits = 0;
    BatchPtrs p;
    NYB_TRY(batch_ptrs(e, *net, b, p));
    size_t box = (size_t)nv.dims[0] * (box_stride ? (size_t)D : 1);
    NYB_CUDA(e, cudaMemcpyAsync(p.in_lo, in_lo, box * 4, cudaMemcpyHostToDevice, e->stream));
    NYB_CUDA(e, cudaMemcpyAsync(p.in_hi, in_hi, box * 4, cudaMemcpyHostToDevice, e->stream));
    e->batch = Batch();  // the resident batch's buffers are being reused
    // This entry point returns the interval bounds themselves, so it always uses the binary64 interval products:
    // the tensor-core products widen every interval by their rounding slack, which compounds with depth to a few
    // 1e-5 of the bound - accounted for inside the batch calls (flags + binary64 re-evaluation of the bounds that
    // show it), but visible to a caller who compares these numbers with the CPU path's.
    const int saved_path = e->path;
    e->path = NYB200_PATH_F64;
    int fst = run_forward(e, *net, b, p, 2);
    e->path = saved_path;
    NYB_TRY(fst);
    size_t w = (size_t)nv.n_pre * 4, ws = (size_t)nv.nps * 4;
    NYB_CUDA(e, cudaMemcpy2DAsync(pre_lo, w, p.pre_lo, ws, w, (size_t)D, cudaMemcpyDeviceToHost, e->stream));
    NYB_CUDA(e, cudaMemcpy2DAsync(pre_hi, w, p.pre_hi, ws, w, (size_t)D, cudaMemcpyDeviceToHost, e->stream));
    NYB_CUDA(e, cudaStreamSynchronize(e->stream));
    return NYB200_OK;
}

int32_t nyb200_set_fusion(nyb200_engine *e, int32_t on) {
    if (!e) return NYB200_ERR_INVALID;
    std::lock_guard<std::mutex> g(e->mu);
    e->fuse_chain = on != 0;
    return NYB200_OK;
}

int32_t nyb200_set_refine_tolerance(nyb200_engine *e, float tol) {
    if (!e || !(tol >= 0.f)) return NYB200_ERR_INVALID;
    std::lock_guard<std::mutex> g(e->mu);
    e->refine_tol = tol;
    return NYB200_OK;
}

int32_t nyb200_batch_refined(nyb200_engine *e, int32_t *n_domains) {
    if (!e || !n_domains) return NYB200_ERR_INVALID;
    std::lock_guard<std::mutex> g(e->mu);
    NYB_CUDA(e, cudaSetDevice(e->device));
    NYB_TRY(finish_batch(e));
    *n_domains = e->batch.refined;
    return NYB200_OK;
}

int32_t nyb200_batch_poll(nyb200_engine *e, int32_t *completed, int32_t *attention) {
    if (!e || !completed || !attention) return NYB200_ERR_INVALID;
    std::lock_guard<std::mutex> g(e->mu);
    if (!e->batch.valid || !e->batch.ran || !e->status_host) return set_err(e, NYB200_ERR_INVALID, "no batch has been run");
    const volatile int *s = e->status_host;
    const int seq = s[0], herr = s[1], loose = s[2];
    *completed = seq == e->run_seq ? 1 : 0;
    *attention = (herr != 0 || loose > 0) ? 1 : 0;
    if (herr) return set_err(e, NYB200_ERR_INTERNAL, "tcgen05 pipeline wait expired (code " + std::to_string(herr) + ")");
    return NYB200_OK;
}

int32_t nyb200_timing_enable(nyb200_engine *e, int32_t per_kernel) {
    if (!e) return NYB200_ERR_INVALID;
    std::lock_guard<std::mutex> g(e->mu);
    e->timing.per_kernel = per_kernel != 0;
    return NYB200_OK;
}

int32_t nyb200_timing_reset(nyb200_engine *e) {
    if (!e) return NYB200_ERR_INVALID;
    std::lock_guard<std::mutex> g(e->mu);
    if (e->timing.pending) { cudaEventSynchronize(e->timing.ev[2]); e->timing.pending = false; e->timing.kev_used = 0; e->timing.cev_used = false; }
    e->timing.fwd_ms = e->timing.bwd_ms = e->timing.tot_ms = e->timing.gemm_ms = e->timing.chain_ms = 0;
    e->timing.runs = 0;
    return NYB200_OK;
}

int32_t nyb200_timing_read(nyb200_engine *e, const char *phase, double *avg_ms, int32_t *n_runs) {
    if (!e || !phase || !avg_ms) return NYB200_ERR_INVALID;
    std::lock_guard<std::mutex> g(e->mu);
    Timing &t = e->timing;
    fold_timing(t);
    double tot = 0;
    if (!strcmp(phase, "forward")) tot = t.fwd_ms;
    else if (!strcmp(phase, "backward")) tot = t.bwd_ms;
    else if (!strcmp(phase, "total")) tot = t.tot_ms;
    else if (!strcmp(phase, "gemm")) tot = t.gemm_ms;
    else if (!strcmp(phase, "chain")) tot = t.chain_ms;
    else return set_err(e, NYB200_ERR_INVALID, "unknown phase");
    *avg_ms = t.runs ? tot / t.runs : 0.0;
    if (n_runs) *n_runs = t.runs;
    return NYB200_OK;
}

}  // extern "C"
