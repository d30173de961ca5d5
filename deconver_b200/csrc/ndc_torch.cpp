// The host path in native code: one autograd node for the whole `Deconv` layer (parameters ->
// float32, 1x1 projection, multiplicative updates), and one each for its neighbours in a block
// (1x1 projection with bias, bias + GELU, instance norm), on the C ABI of libndc_b200.so and cuBLAS.
//
// What bounds the layer at the deep stages and on single images is not the GPU: at 512 channels
// x 8^3 a forward and backward are 0.16 ms of kernels, and issuing them from Python through
// separate autograd nodes took 0.60 ms.  One node, one pass over the parameters in each
// direction, and no intermediate tensor that the update kernels do not read.  The neighbours the same:
// see the figures at their section.
#include <ATen/Context.h>
#include <ATen/cuda/CUDAContext.h>
#include <ATen/ops/convolution_backward.h>
#include <ATen/ops/empty.h>
#include <ATen/ops/relu.h>
#include <c10/cuda/CUDAGuard.h>
#include <cublas_v2.h>
#include <torch/csrc/autograd/functions/basic_ops.h>
#include <torch/extension.h>

#include <algorithm>
#include <mutex>
#include <tuple>
#include <vector>

#include "ndc_b200.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

int dtype_code(const Tensor& t) { return t.scalar_type() == at::kBFloat16 ? NDC_BF16 : NDC_F32; }
bool kernel_dtype(const Tensor& t) { return t.scalar_type() == at::kFloat || t.scalar_type() == at::kBFloat16; }
// The tensor's memory.  A tensor may have none though it has elements (FakeTensor and other wrappers): library
// calls would read at address zero.
void* ptr(const Tensor& t) {
    if (!t.defined()) return nullptr;
    void* p = t.data_ptr();
    TORCH_CHECK(p || !t.numel(), "deconver_b200: a tensor of ", t.sizes(), " has no memory; the kernels need one that does");
    return p;
}
float* fptr(const Tensor& t) { return static_cast<float*>(ptr(t)); }
void* stream() { return at::cuda::getCurrentCUDAStream().stream(); }

void check(int status, const char* message) {
    TORCH_CHECK(status == NDC_OK, "ndc_b200 status ", status, ": ", message);
}

// The nodes have no forward-mode derivative.  Their own `apply` says so, but calls without reverse-mode
// gradients do not go through it, and would drop the tangents.
void refuse_tangents(std::initializer_list<const Tensor*> tensors) {
    for (const Tensor* t : tensors)
        TORCH_CHECK(!t->defined() || !t->_fw_grad(0).defined(), "deconver_b200: forward-mode differentiation is not implemented");
}

// ---- optional CUDA-event timing of ndc_fwd / ndc_bwd on the stream they are issued on ----------
struct Timing {
    std::mutex mu;
    bool enabled = false;
    std::vector<std::pair<cudaEvent_t, cudaEvent_t>> spans[2];   // forward, backward
} g_timing;

struct Span {
    cudaEvent_t start = nullptr, stop = nullptr;
    int kind;
    explicit Span(int k) : kind(k) {
        if (!g_timing.enabled) return;
        C10_CUDA_CHECK(cudaEventCreate(&start));
        C10_CUDA_CHECK(cudaEventCreate(&stop));
        C10_CUDA_CHECK(cudaEventRecord(start, (cudaStream_t)stream()));
    }
    ~Span() {
        if (!start) return;
        (void)cudaEventRecord(stop, (cudaStream_t)stream());
        std::lock_guard<std::mutex> lock(g_timing.mu);
        g_timing.spans[kind].emplace_back(start, stop);
    }
};

void timing_enable() {
    std::lock_guard<std::mutex> lock(g_timing.mu);
    for (auto& v : g_timing.spans) {
        for (auto& s : v) { (void)cudaEventDestroy(s.first); (void)cudaEventDestroy(s.second); }
        v.clear();
    }
    g_timing.enabled = true;
}

// Stops collecting; the caller has synchronised.  {forward ms, backward ms}
std::vector<std::vector<float>> timing_collect() {
    std::lock_guard<std::mutex> lock(g_timing.mu);
    g_timing.enabled = false;
    std::vector<std::vector<float>> out(2);
    for (int k = 0; k < 2; ++k) {
        for (auto& s : g_timing.spans[k]) {
            float ms = 0.0f;
            C10_CUDA_CHECK(cudaEventElapsedTime(&ms, s.first, s.second));
            out[k].push_back(ms);
            (void)cudaEventDestroy(s.first);
            (void)cudaEventDestroy(s.second);
        }
        g_timing.spans[k].clear();
    }
    return out;
}

// ---- 1x1 projections -------------------------------------------------------------------------
// The precision the framework gives convolutions of float32 tensors: TF32 unless switched off.
bool conv_tf32() { return at::globalContext().allowTF32CuDNN(at::Float32Op::CONV); }

// y[b] = op(w) x[b] (+ y[b] if `accumulate`) for a (Co, Ci) matrix `w`, op = transpose if
// `transpose`, and contiguous (B, channels, N) tensors: one strided batched library GEMM with the
// matrix repeated by a zero batch stride; no tensor is converted or copied.
void channel_gemm(const Tensor& w, bool transpose, const Tensor& x, Tensor& y, int64_t batch, int64_t n,
                  bool accumulate) {
    const int64_t co = w.size(0), ci = w.size(1);
    const int64_t out = transpose ? ci : co, in = transpose ? co : ci;
    if (!batch || !n || !out || !in) return;
    const bool bf16 = x.scalar_type() == at::kBFloat16;
    const bool tf32 = !bf16 && conv_tf32();
    const float one = 1.0f, beta = accumulate ? 1.0f : 0.0f;
    const cudaDataType_t type = bf16 ? CUDA_R_16BF : CUDA_R_32F;
    const cublasComputeType_t compute = tf32 ? CUBLAS_COMPUTE_32F_FAST_TF32 : CUBLAS_COMPUTE_32F;
    at::NoTF32Guard plain;   // the handle's own mode; `compute` says what this product uses
    cublasHandle_t handle = at::cuda::getCurrentCUDABlasHandle();
    // column-major view: (n x out) = (n x in) * (in x out)
    const cublasStatus_t st = cublasGemmStridedBatchedEx(
        handle, CUBLAS_OP_N, transpose ? CUBLAS_OP_T : CUBLAS_OP_N, (int)n, (int)out, (int)in, &one, ptr(x),
        type, (int)n, (long long)(in * n), ptr(w), type, (int)ci, 0LL, &beta, ptr(y), type, (int)n,
        (long long)(out * n), (int)batch, compute, CUBLAS_GEMM_DEFAULT);
    TORCH_CHECK(st == CUBLAS_STATUS_SUCCESS, "deconver_b200: projection GEMM failed (cuBLAS status ", (int)st, ")");
}

// The weight gradient of a 1x1 projection is a product of two wide matrices along their positions, and no
// one way is the fastest over the channels, batches and positions that occur:
//   Kernel       ndc_proj_wgrad: any row length; its MMAs' rate and tiles of 128 x 64 bound it for many channels
//   Product      one library product per sample, where samples and tiles of 128 x 128 fill the GPU
//   Slices       a sample's positions in 32 or 16 slices (more were slower: 2 x (256 + 64) x 262144 takes 136 us
//                with 32, 157 with 74), one batched library product per sample
//   Convolution  the library's convolution backward, for rows that are not whole vectors and many channels
// (Slices and Product are views of the tensors as they lie, float32 partial products, summed by ndc_proj_sum.)
enum WgradRoute { kKernel = 0, kProduct = 1, kSlices = 2, kConvolution = 3 };
struct WgradPlan { WgradRoute route; int64_t slices; };

// Whole vectors: the least expected time, microseconds, of the first three, by constants fitted to 1481
// float32 and 1317 bfloat16 shapes (16 to 2048 channels, 1 to 16 samples of 343 to 262144 positions).  On 400
// other shapes of either type the choice takes 42 and 51 ms together, the library's convolution 88 and
// 94, fixed limits on channels and batches (before) 55 and 57; by more than a tenth the convolution is
// faster on 39 and 7 (before: 135 and 76), but it is up to 50 times slower on others, which cannot be foreseen.
// Others (672 shapes): below the limit the kernel takes 0.05 - 0.9 times the library's convolution on the
// average of a class of widths and batches, above it 1.0 - 3.5; a single sample is a plain product for the
// library (1.3 - 3.8 from 20000 on).
// `exact` (float32 without TF32): the kernel throughout.  On 350 shapes it takes 0.42 times the library's
// convolution, and is off by 2.8e-7 of the result against 64 bits where the convolution is by 5.5e-7, slices by 7.2e-7
// and one product per sample, a single chain along its positions, by 1.4e-6 (1e-5 at most).
WgradPlan plan_weight_grad(int64_t batch, int64_t co, int64_t ci, int64_t n, bool bf16, bool exact, int sms) {
    if (exact) return {kKernel, 1};
    if (n % (bf16 ? 8 : 4)) {
        const int64_t limit = batch == 1 ? 20000 : batch <= 8 ? 200000 : bf16 ? 100000 : 30000;
        return {co * ci >= limit ? kConvolution : kKernel, 1};
    }
    const auto tiles = [](int64_t v, int64_t t) { return (v + t - 1) / t; };
    const double e = bf16 ? 2 : 4, bytes = (double)(co + ci) * n * e;                       // of a sample
    const int64_t square = tiles(co, 128) * tiles(ci, 128);
    // the library's products: CTAs of 128 x 128 outputs, each one chain along its positions
    const double rate = bf16 ? 1180.0 : n % 8 ? 455.0 : 525.0;                              // positions per us
    const double product = 14.0 + std::max((double)tiles(batch * square, sms) * n / rate, batch * bytes / 3.9e6);
    const int64_t slices = std::min<int64_t>(square < 4 ? 32 : 16, n / 1024);
    const double sliced = slices < 2 ? product + 1.0
                                     : 9.0 + (n % (8 * slices) ? 8.0 : 0.0) +
                                           batch * (5.5 + std::max(bytes / 5.0e6, 2.0 * co * ci * n / (bf16 ? 600e6 : 370e6)));
    // ndc_proj_wgrad: see plan_wgrad there
    const int64_t t = tiles(co, 128) * tiles(ci, 64), parts = std::max<int64_t>(1, std::min(tiles(4 * sms, t * batch), tiles(n, 512)));
    const double flops = 2.0 * batch * n * t * 128 * 64, read = ((double)co * tiles(ci, 64) + (double)ci * tiles(co, 128)) * batch * n * e;
    const double kernel = 7.3 + std::max(flops / (bf16 ? 272e6 : 134e6) / std::min(1.0, t * batch * parts / (2.0 * sms)), read / (bf16 ? 5.7e6 : 4.1e6)) +
                          batch * parts * co * ci * 8 / (bf16 ? 1.8e6 : 1.4e6);
    if (kernel <= product && kernel <= sliced) return {kKernel, 1};
    return product <= sliced ? WgradPlan{kProduct, 1} : WgradPlan{kSlices, slices};
}

Tensor weight_grad(const Tensor& gy, const Tensor& x, const Tensor& w, int64_t batch, int64_t n) {
    Tensor gw = at::empty(w.sizes(), w.options());
    const int64_t co = w.size(0), ci = w.size(1);
    if (!batch || !n || !co || !ci) return gw.zero_();
    const bool bf16 = gy.scalar_type() == at::kBFloat16;
    const WgradPlan plan = plan_weight_grad(batch, co, ci, n, bf16, !bf16 && !conv_tf32(), at::cuda::getCurrentDeviceProperties()->multiProcessorCount);
    if (plan.route == kConvolution)
        return std::get<1>(at::convolution_backward(gy.view({batch, co, n}), x.view({batch, ci, n}), w.view({co, ci, 1}), at::nullopt, {1}, {0},
                                                    {1}, false, {0}, 1, {false, true, false})).view(w.sizes());
    if (plan.route == kKernel) {
        const size_t bytes = ndc_proj_wgrad_workspace_bytes((int)batch, (int)co, (int)ci, n);
        Tensor ws = at::empty({(int64_t)bytes}, w.options().dtype(at::kByte));
        check(ndc_proj_wgrad((int)batch, (int)co, (int)ci, n, dtype_code(gy), conv_tf32() ? 1 : 0, ptr(gy), ptr(x),
                             ptr(gw), ptr(ws), bytes, stream()), ndc_proj_last_error());
        return gw;
    }
    // slices of whole vectors, and what they leave
    const int64_t slices = plan.slices, length = slices > 1 ? n / slices / 8 * 8 : n, rest = n - slices * length;
    Tensor partial = at::empty({batch * slices, co, ci}, w.options().dtype(at::kFloat));
    const cudaDataType_t type = bf16 ? CUDA_R_16BF : CUDA_R_32F;
    const cublasComputeType_t compute = bf16 ? CUBLAS_COMPUTE_32F : CUBLAS_COMPUTE_32F_FAST_TF32;
    at::NoTF32Guard plain;
    cublasHandle_t handle = at::cuda::getCurrentCUDABlasHandle();
    // `count` products along `k` positions, the first from position `at` of sample b on, the others
    // further on in it (`length` apart) or in the samples after it
    auto products = [&](int64_t b, int64_t at, int64_t k, bool samples, int64_t count, float beta) {
        const float one = 1.0f;
        const size_t e = bf16 ? 2 : 4;
        const int64_t sx = samples ? ci * n : length, sy = samples ? co * n : length, out_step = samples ? slices : 1;
        const cublasStatus_t st = cublasGemmStridedBatchedEx(
            handle, CUBLAS_OP_T, CUBLAS_OP_N, (int)ci, (int)co, (int)k, &one, static_cast<const char*>(ptr(x)) + (b * ci * n + at) * e, type,
            (int)n, (long long)sx, static_cast<const char*>(ptr(gy)) + (b * co * n + at) * e, type, (int)n, (long long)sy, &beta,
            fptr(partial) + b * slices * co * ci, CUDA_R_32F, (int)ci, (long long)(out_step * co * ci), (int)count, compute, CUBLAS_GEMM_DEFAULT);
        TORCH_CHECK(st == CUBLAS_STATUS_SUCCESS, "deconver_b200: projection gradient failed (cuBLAS status ", (int)st, ")");
    };
    if (slices == 1) products(0, 0, n, true, batch, 0.0f);
    else
        for (int64_t b = 0; b < batch; ++b) products(b, 0, length, false, slices, 0.0f);
    if (rest) products(0, slices * length, rest, true, batch, 1.0f);
    if (batch * slices == 1 && !bf16) return partial.view(w.sizes());
    check(ndc_proj_sum((int)(batch * slices), co * ci, dtype_code(gy), fptr(partial), ptr(gw), stream()), ndc_proj_last_error());
    return gw;
}

// ---- the layer -------------------------------------------------------------------------------
struct Config {
    int64_t groups, m, sc;
    double eps;
    int64_t iters, grad_iters, flags;
    bool bf16_params = false;          // filter and bias are bfloat16 values
};

bool bf16_params(const Tensor& h0, const Tensor& bias) {
    return h0.scalar_type() == at::kBFloat16 && (!bias.defined() || bias.scalar_type() == at::kBFloat16);
}

NdcDesc make_desc(const Tensor& x, const Tensor& h0, const Config& c, bool relu) {
    NdcDesc d;
    int64_t sp[3] = {1, 1, 1}, k[3] = {1, 1, 1};
    const int64_t rank = x.dim() - 2;
    for (int64_t i = 0; i < rank; ++i) { sp[3 - rank + i] = x.size(2 + i); k[3 - rank + i] = h0.size(2 + i); }
    d.batch = (int)x.size(0); d.groups = (int)c.groups; d.m = (int)c.m; d.sc = (int)c.sc;
    d.D = (int)sp[0]; d.H = (int)sp[1]; d.W = (int)sp[2];
    d.kD = (int)k[0]; d.kH = (int)k[1]; d.kW = (int)k[2];
    d.eps = (float)c.eps; d.relu_input = relu ? 1 : 0; d.dtype = dtype_code(x); d.flags = (int)c.flags;
    if (c.bf16_params) d.flags |= NDC_FLAG_BF16_PARAMS;
    return d;
}

// relu(h0) and the bias as the kernels take them
void prepare_params(const Tensor& h0, const Tensor& bias, Tensor& h, Tensor& b) {
    const auto f32 = h0.options().dtype(at::kFloat);
    const bool same = !bias.defined() || bias.scalar_type() == h0.scalar_type();
    if (kernel_dtype(h0) && same) {
        h = at::empty(h0.sizes(), f32);
        const bool convert = bias.defined() && bias.scalar_type() != at::kFloat;
        b = convert ? at::empty(bias.sizes(), f32) : bias;
        check(ndc_params_prepare(dtype_code(h0), ptr(h0), h0.numel(), fptr(h), convert ? ptr(bias) : nullptr,
                                 convert ? bias.numel() : 0, convert ? fptr(b) : nullptr, stream()),
              ndc_proj_last_error());
        return;
    }
    h = at::relu(h0).to(at::kFloat);
    b = bias.defined() ? bias.to(at::kFloat) : bias;
}

struct Saved {
    Tensor x;                          // the input, rows padded where that pays
    Tensor h, b;                       // float32 filter and bias
    std::vector<Tensor> z, t1;         // per update that has gradients: its source and K(source)
    int64_t first = 0;                 // index of the first such update
};

Tensor run_forward(const Tensor& x, const Tensor& h0, const Tensor& w, const Tensor& bias, const Config& config,
                   Saved* saved) {
    Saved local;
    Saved& sv = saved ? *saved : local;
    Config c = config;
    c.bf16_params = bf16_params(h0, bias);
    // Without gradients float32 parameters need no pass of their own: the depthwise kernels rectify the
    // filter on load (one launch of three less on a single small image).
    bool raw = !saved && c.m == 1 && c.sc == 4 && h0.scalar_type() == at::kFloat &&
               (!bias.defined() || bias.scalar_type() == at::kFloat) && !(c.flags & NDC_FLAG_FORCE_GENERIC);
    if (raw) { sv.h = h0; sv.b = bias; }
    else prepare_params(h0, bias, sv.h, sv.b);
    auto out_shape = x.sizes().vec();
    out_shape[1] = c.groups * c.sc;
    // Rows that are not whole vectors: the layer owns everything between its input and its output
    // (projection, t1, gradients), so it keeps them with padded rows.  One copy of x (a tenth of
    // the forward's traffic) buys vector loads in every kernel and aligned GEMMs.
    const int W = x.numel() ? (int)x.size(-1) : 0;
    int pitch = W;
    sv.x = x;
    if (x.numel()) {
        const NdcDesc d = make_desc(x, h0, c, true);
        pitch = ndc_row_pitch(&d);
        if (pitch != W) {
            auto xs = x.sizes().vec();
            xs.back() = pitch;
            sv.x = at::empty(xs, x.options());
            check(ndc_pad_rows(x.numel() / W, W, pitch, d.dtype, ptr(x), ptr(sv.x), stream()), ndc_proj_last_error());
        }
    }
    auto shape = out_shape;
    if (W) shape.back() = pitch;
    const int64_t n = sv.x.numel() ? sv.x.numel() / (x.size(0) * x.size(1)) : 0;
    Tensor s = at::empty(shape, x.options());
    channel_gemm(w, false, sv.x, s, x.size(0), n, false);
    sv.first = c.iters > c.grad_iters ? c.iters - c.grad_iters : 0;
    Tensor t1;
    for (int64_t it = 0; it < c.iters; ++it) {
        const bool keep = saved && it >= sv.first;
        const bool last = it + 1 == c.iters;
        Tensor out = at::empty(last ? out_shape : shape, x.options());
        if (keep || !t1.defined()) t1 = at::empty(sv.x.sizes(), x.options());
        if (x.numel()) {
            NdcDesc d = make_desc(x, h0, c, it == 0);
            Span span(0);
            auto update = [&](int flag) {
                d.flags = (int)c.flags | (c.bf16_params ? NDC_FLAG_BF16_PARAMS : 0) | flag;
                return ndc_fwd_rows(&d, pitch, last ? W : pitch, ptr(sv.x), ptr(s), fptr(sv.h), it == 0 ? fptr(sv.b) : nullptr,
                                    ptr(out), ptr(t1), stream());
            };
            int status = update(raw ? NDC_FLAG_RELU_FILTER : 0);
            if (raw && status == NDC_ERR_UNSUPPORTED) {   // not the depthwise kernels
                raw = false;
                prepare_params(h0, bias, sv.h, sv.b);
                status = update(0);
            }
            check(status, ndc_last_error());
        }
        if (keep) { sv.z.push_back(s); sv.t1.push_back(t1); }
        s = out;
    }
    return s;
}

struct LayerNode : public torch::autograd::Function<LayerNode> {
    static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& h0, const Tensor& w,
                          const std::optional<Tensor>& bias, int64_t groups, int64_t m, int64_t sc, double eps,
                          int64_t iters, int64_t grad_iters, int64_t flags) {
        const Config c{groups, m, sc, eps, iters, grad_iters, flags};
        Saved sv;
        const Tensor b = bias ? *bias : Tensor();
        Tensor out = run_forward(x, h0, w, b, c, &sv);
        variable_list keep = {sv.x, h0, w, b, sv.h, sv.b};
        keep.insert(keep.end(), sv.z.begin(), sv.z.end());
        keep.insert(keep.end(), sv.t1.begin(), sv.t1.end());
        ctx->save_for_backward(keep);
        auto& d = ctx->saved_data;
        d["cfg"] = std::vector<int64_t>{groups, m, sc, iters, grad_iters, flags, sv.first, x.size(-1)};
        d["eps"] = eps;
        return out;
    }

    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        TORCH_CHECK(!at::GradMode::is_enabled(), "double backward through the fused Deconv update is not supported");
        const variable_list kept = ctx->get_saved_variables();
        const auto cfg = ctx->saved_data["cfg"].toIntVector();
        Config c{cfg[0], cfg[1], cfg[2], ctx->saved_data["eps"].toDouble(), cfg[3], cfg[4], cfg[5]};
        const int64_t first = cfg[6], count = c.iters - first, W = cfg[7];
        const Tensor &x = kept[0], &h0 = kept[1], &w = kept[2], &bias = kept[3], &h = kept[4], &b = kept[5];
        c.bf16_params = bf16_params(h0, bias);
        const bool need_x = ctx->needs_input_grad(0), need_h = ctx->needs_input_grad(1);
        const bool whole = first == 0;                   // gradients reach the projection
        const bool need_w = whole && ctx->needs_input_grad(2);
        const bool need_b = whole && bias.defined() && ctx->needs_input_grad(3);
        c10::cuda::CUDAGuard guard(x.device());
        const auto f32 = h.options();

        Tensor g = grads[0].contiguous();
        if (g.scalar_type() != x.scalar_type()) g = g.to(x.scalar_type());
        Tensor gx, gh, gb, ws;
        const int64_t n = x.numel() ? x.numel() / (x.size(0) * x.size(1)) : 0;
        for (int64_t i = count - 1; i >= 0; --i) {
            const Tensor &z = kept[6 + i], &t1 = kept[6 + count + i];
            const bool it0 = first + i == 0;
            const bool need_z = i > 0 || (it0 && (need_x || need_w || need_b));
            Tensor gx_i, gz, gh_i;
            if (need_x) gx_i = at::empty(x.sizes(), x.options());
            if (need_z) gz = at::empty(z.sizes(), z.options());
            if (need_h) gh_i = at::empty(h.sizes(), f32);
            if (need_b && it0) gb = at::empty(bias.sizes(), f32);
            if (x.numel()) {
                NdcDesc d = make_desc(x, h0, c, it0);
                const int pitch = d.W;
                d.W = (int)W;
                const size_t bytes = ndc_bwd_rows_workspace_bytes(&d, pitch);
                if (!ws.defined()) ws = at::empty({(int64_t)bytes}, x.options().dtype(at::kByte));
                Span span(1);
                check(ndc_bwd_rows(&d, pitch, i == count - 1 ? (int)W : pitch, ptr(x), ptr(z), ptr(t1), fptr(h),
                                   it0 ? fptr(b) : nullptr, ptr(g), ptr(gx_i), ptr(gz), fptr(gh_i),
                                   it0 ? fptr(gb) : nullptr, ptr(ws), bytes, stream()), ndc_last_error());
            } else {
                for (Tensor* t : {&gx_i, &gz, &gh_i, &gb}) if (t->defined()) t->zero_();
            }
            if (need_x) { if (gx.defined()) gx.add_(gx_i); else gx = gx_i; }
            if (need_h) { if (gh.defined()) gh.add_(gh_i); else gh = gh_i; }
            g = gz;
        }
        ws.reset();
        Tensor gw, gh0, gbias;
        if (whole) {
            // gz of the first update: W^T gz is added to the update's own input gradient
            if (need_x) channel_gemm(w, true, g, gx, x.size(0), n, true);
            if (need_w) gw = weight_grad(g, x, w, x.size(0), n);
        }
        if (need_x && x.numel() && x.size(-1) != W) {
            auto xs = x.sizes().vec();
            xs.back() = W;
            Tensor plain = at::empty(xs, x.options());
            check(ndc_unpad_rows(plain.numel() / W, (int)W, (int)x.size(-1), dtype_code(x), ptr(gx), ptr(plain), stream()),
                  ndc_proj_last_error());
            gx = plain;
        }
        const bool same = !need_b || !need_h || bias.scalar_type() == h0.scalar_type();
        if ((need_h || need_b) && kernel_dtype(need_h ? h0 : bias) && same) {
            if (need_h) gh0 = at::empty(h0.sizes(), h0.options());
            const bool convert = need_b && bias.scalar_type() != at::kFloat;
            gbias = convert ? at::empty(bias.sizes(), bias.options()) : gb;
            if (need_h || convert)
                check(ndc_params_grad(dtype_code(need_h ? h0 : bias), need_h ? ptr(h0) : nullptr, fptr(gh),
                                      need_h ? h0.numel() : 0, ptr(gh0), convert ? fptr(gb) : nullptr,
                                      convert ? bias.numel() : 0, convert ? ptr(gbias) : nullptr, stream()),
                      ndc_proj_last_error());
        } else {
            if (need_h) gh0 = gh.mul_(h0 > 0).to(h0.scalar_type());
            if (need_b) gbias = gb.to(bias.scalar_type());
        }
        variable_list out(11);
        out[0] = gx; out[1] = gh0; out[2] = gw; out[3] = gbias;
        return out;
    }
};

// s of the layer.  `h0` (C, sc, *k), `w` (groups*sc, C, 1), `bias` (groups*sc) or None.
Tensor layer(const Tensor& x_in, const Tensor& h0_in, const Tensor& w_in, const std::optional<Tensor>& bias_in,
             int64_t groups, int64_t m, int64_t sc, double eps, int64_t iters, int64_t grad_iters, int64_t flags) {
    TORCH_CHECK(w_in.scalar_type() == x_in.scalar_type(), "deconver_b200: the input is ", x_in.scalar_type(),
                " but the projection's weight is ", w_in.scalar_type());
    for (const Tensor* t : {&h0_in, &w_in})
        TORCH_CHECK(t->device() == x_in.device(), "deconver_b200: input on ", x_in.device(), ", parameters on ", t->device());
    TORCH_CHECK(x_in.size(1) == groups * m && w_in.size(0) == groups * sc && w_in.size(1) == x_in.size(1) &&
                h0_in.dim() == x_in.dim() && h0_in.size(0) == groups * m && h0_in.size(1) == sc,
                "deconver_b200: input ", x_in.sizes(), ", filter ", h0_in.sizes(), " and projection ", w_in.sizes(),
                " do not match groups=", groups, ", m=", m, ", sc=", sc);
    TORCH_CHECK(!bias_in || (bias_in->device() == x_in.device() && bias_in->numel() == groups * sc),
                "deconver_b200: the bias does not match the projection");
    c10::cuda::CUDAGuard guard(x_in.device());
    refuse_tangents({&x_in, &h0_in, &w_in});
    if (bias_in) refuse_tangents({&*bias_in});
    const Tensor x = x_in.contiguous(), h0 = h0_in.contiguous(), w = w_in.contiguous();
    const std::optional<Tensor> bias = bias_in ? std::optional<Tensor>(bias_in->contiguous()) : std::nullopt;
    const bool grad = at::GradMode::is_enabled() &&
                      (x.requires_grad() || h0.requires_grad() || w.requires_grad() || (bias && bias->requires_grad()));
    if (grad && grad_iters > 0)
        return LayerNode::apply(x, h0, w, bias, groups, m, sc, eps, iters, grad_iters, flags);
    at::AutoDispatchBelowADInplaceOrView below;
    return run_forward(x, h0, w, bias ? *bias : Tensor(), Config{groups, m, sc, eps, iters, grad_iters, flags}, nullptr);
}

// ---- the layer's neighbours in a block ---------------------------------------------------------
// Small blocks are bound by the host here too: with one Python autograd node each and their parameters
// converted one by one, a training step of a bf16 block of 32 channels x 16^3 took 1.44 - 2.16 ms for
// 0.22 ms of kernels; from here it takes 0.72.  float32 projections lose the convolution route's copies
// to channels-last as well (8 x 32 x 40^3: 11.4 -> 3.4 ms).

// A vector of parameters as float32, and a float32 gradient in the parameters' type: one launch.
Tensor as_f32(const Tensor& t) {
    if (!t.defined() || t.scalar_type() == at::kFloat) return t.defined() ? t.contiguous() : t;
    if (t.scalar_type() != at::kBFloat16 || !t.numel()) return t.to(at::kFloat).contiguous();
    const Tensor in = t.contiguous();
    Tensor out = at::empty(in.sizes(), in.options().dtype(at::kFloat));
    check(ndc_params_prepare(NDC_BF16, nullptr, 0, nullptr, ptr(in), in.numel(), fptr(out), stream()), ndc_proj_last_error());
    return out;
}
Tensor from_f32(const Tensor& g, at::ScalarType type) {
    if (!g.defined() || type == at::kFloat) return g;
    if (type != at::kBFloat16 || !g.numel()) return g.to(type);
    Tensor out = at::empty(g.sizes(), g.options().dtype(type));
    check(ndc_params_grad(NDC_BF16, nullptr, nullptr, 0, nullptr, fptr(g), g.numel(), ptr(out), stream()), ndc_proj_last_error());
    return out;
}

// The gradients of a node whose backward is not itself differentiable: they are computed without a
// graph, and differentiating them raises an error.  What torch.autograd.function.once_differentiable does
// for Python nodes, which these were, message included.
variable_list once(const variable_list& grads, variable_list out) {
    bool any = false;
    for (const Tensor& g : grads) any = any || (g.defined() && g.requires_grad());
    if (!at::GradMode::is_enabled() || !any) return out;
    auto error = std::make_shared<torch::autograd::DelayedError>(
        "trying to differentiate twice a function that was marked with @once_differentiable", (int64_t)out.size());
    for (Tensor& t : out)
        if (t.defined()) t = t.detach().requires_grad_();
    return (*error)(std::move(out));
}

struct Slabs { int batch, channels; int64_t n; };
Slabs slabs(const Tensor& x) {
    const int64_t bc = x.size(0) * x.size(1);
    int64_t n = 1;
    for (int64_t i = 2; i < x.dim(); ++i) n *= x.size(i);
    return {(int)x.size(0), (int)x.size(1), bc ? n : 0};
}
Tensor like(const Tensor& g, const Tensor& x) {
    Tensor c = g.contiguous();
    return c.scalar_type() == x.scalar_type() ? c : c.to(x.scalar_type());
}
Tensor bias_scratch(const Slabs& s, const Tensor& x) {
    return at::empty({(int64_t)ndc_bias_grad_workspace_bytes(s.batch, s.channels)}, x.options().dtype(at::kByte));
}

// y = w x (+ bias) over the channel axis; `w` (Co, Ci, 1)
struct LinearNode : public torch::autograd::Function<LinearNode> {
    static Tensor run(const Tensor& x, const Tensor& w, const Tensor& bias) {
        auto shape = x.sizes().vec();
        shape[1] = w.size(0);
        Tensor y = at::empty(shape, x.options());
        const Slabs s = slabs(y), in = slabs(x);
        if (!y.numel()) return y;
        if (!in.channels) y.zero_();
        else channel_gemm(w, false, x, y, s.batch, s.n, false);
        if (bias.defined()) {
            const Tensor b = as_f32(bias);
            check(ndc_bias_add(s.batch, s.channels, s.n, dtype_code(y), ptr(y), fptr(b), stream()), ndc_bias_last_error());
        }
        return y;
    }

    static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w, const std::optional<Tensor>& bias) {
        const Tensor b = bias ? *bias : Tensor();
        ctx->save_for_backward({x, w});
        ctx->saved_data["bias"] = b.defined();
        ctx->saved_data["type"] = (int64_t)(b.defined() ? b.scalar_type() : at::kFloat);
        return run(x, w, b);
    }

    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        variable_list out(3);
        {
            at::AutoGradMode off(false);
            const variable_list kept = ctx->get_saved_variables();
            const Tensor &x = kept[0], &w = kept[1];
            c10::cuda::CUDAGuard guard(x.device());
            const Tensor g = like(grads[0], x);
            const Slabs s = slabs(g);
            if (ctx->needs_input_grad(0)) {
                out[0] = at::empty(x.sizes(), x.options());
                if (s.n) channel_gemm(w, true, g, out[0], s.batch, s.n, false);
                else out[0].zero_();
            }
            if (ctx->needs_input_grad(1)) out[1] = weight_grad(g, x, w, s.batch, s.n);
            if (ctx->saved_data["bias"].toBool() && ctx->needs_input_grad(2)) {
                Tensor gb = at::empty({s.channels}, x.options().dtype(at::kFloat));
                if (s.n) {
                    Tensor ws = bias_scratch(s, x);
                    check(ndc_bias_grad(s.batch, s.channels, s.n, dtype_code(g), ptr(g), fptr(gb), ptr(ws), ws.numel(), stream()),
                          ndc_bias_last_error());
                } else {
                    gb.zero_();
                }
                out[2] = from_f32(gb, (at::ScalarType)ctx->saved_data["type"].toInt());
            }
        }
        return once(grads, out);
    }
};

bool wants_grad(std::initializer_list<const Tensor*> tensors) {
    if (!at::GradMode::is_enabled()) return false;
    for (const Tensor* t : tensors)
        if (t->defined() && t->requires_grad()) return true;
    return false;
}

Tensor linear(const Tensor& x_in, const Tensor& w_in, const std::optional<Tensor>& bias_in) {
    TORCH_CHECK(kernel_dtype(x_in) && w_in.scalar_type() == x_in.scalar_type() && w_in.device() == x_in.device() &&
                x_in.dim() >= 3 && w_in.dim() == 3 && w_in.size(2) == 1 && w_in.size(1) == x_in.size(1),
                "deconver_b200: input ", x_in.sizes(), " (", x_in.scalar_type(), ", ", x_in.device(), ") and 1x1 weight ",
                w_in.sizes(), " (", w_in.scalar_type(), ", ", w_in.device(), ") do not match");
    TORCH_CHECK(!bias_in || (bias_in->device() == x_in.device() && bias_in->numel() == w_in.size(0)),
                "deconver_b200: the bias does not match the projection");
    c10::cuda::CUDAGuard guard(x_in.device());
    const Tensor x = x_in.contiguous(), w = w_in.contiguous(), b = bias_in ? *bias_in : Tensor();
    refuse_tangents({&x, &w, &b});
    if (wants_grad({&x, &w, &b})) return LinearNode::apply(x, w, bias_in);
    at::AutoDispatchBelowADInplaceOrView below;
    return LinearNode::run(x, w, b);
}

// gelu(h + bias[c]), erf form
struct BiasGeluNode : public torch::autograd::Function<BiasGeluNode> {
    static Tensor run(const Tensor& h, const Tensor& b) {
        Tensor out = at::empty(h.sizes(), h.options());
        const Slabs s = slabs(h);
        if (h.numel())
            check(ndc_bias_gelu_fwd(s.batch, s.channels, s.n, dtype_code(h), ptr(h), fptr(b), ptr(out), stream()), ndc_bias_last_error());
        return out;
    }

    static Tensor forward(AutogradContext* ctx, const Tensor& h, const std::optional<Tensor>& bias) {
        const Tensor b = as_f32(bias ? *bias : Tensor());
        ctx->save_for_backward({h, b});
        ctx->saved_data["bias"] = (int64_t)(bias ? bias->scalar_type() : at::kFloat);
        return run(h, b);
    }

    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        variable_list out(2);
        {
            at::AutoGradMode off(false);
            const variable_list kept = ctx->get_saved_variables();
            const Tensor &h = kept[0], &b = kept[1];
            c10::cuda::CUDAGuard guard(h.device());
            const Tensor g = like(grads[0], h);
            const Slabs s = slabs(h);
            const bool want_bias = b.defined() && ctx->needs_input_grad(1);
            out[0] = at::empty(h.sizes(), h.options());
            Tensor gb, ws;
            if (want_bias) {
                gb = at::empty({s.channels}, h.options().dtype(at::kFloat));
                ws = bias_scratch(s, h);
            }
            if (s.n)
                check(ndc_bias_gelu_bwd(s.batch, s.channels, s.n, dtype_code(h), ptr(g), ptr(h), fptr(b), ptr(out[0]), fptr(gb),
                                        ptr(ws), want_bias ? ws.numel() : 0, stream()), ndc_bias_last_error());
            else if (want_bias)
                gb.zero_();
            if (want_bias) out[1] = from_f32(gb, (at::ScalarType)ctx->saved_data["bias"].toInt());
        }
        return once(grads, out);
    }
};

Tensor bias_gelu(const Tensor& h_in, const std::optional<Tensor>& bias) {
    TORCH_CHECK(kernel_dtype(h_in) && h_in.is_cuda() && h_in.dim() >= 2 &&
                (!bias || (bias->device() == h_in.device() && bias->numel() == h_in.size(1))),
                "deconver_b200: the bias does not match the tensor");
    c10::cuda::CUDAGuard guard(h_in.device());
    const Tensor h = h_in.contiguous(), b = bias ? *bias : Tensor();
    refuse_tangents({&h, &b});
    if (wants_grad({&h, &b})) return BiasGeluNode::apply(h, bias);
    at::AutoDispatchBelowADInplaceOrView below;
    return BiasGeluNode::run(h, as_f32(b));
}

// (x - mean) / sqrt(var + eps) [* weight + bias] per (sample, channel)
struct NormNode : public torch::autograd::Function<NormNode> {
    static Tensor run(const Tensor& x, const Tensor& w, const Tensor& b, double eps, Tensor& stats) {
        Tensor y = at::empty(x.sizes(), x.options());
        const Slabs s = slabs(x);
        stats = at::empty({(int64_t)s.batch * s.channels * 2}, x.options().dtype(at::kFloat));
        if (x.numel()) {
            const size_t bytes = ndc_inorm_workspace_bytes(s.batch, s.channels);
            Tensor ws = at::empty({(int64_t)bytes}, x.options().dtype(at::kByte));
            check(ndc_inorm_fwd(s.batch, s.channels, s.n, dtype_code(x), ptr(x), fptr(w), fptr(b), (float)eps, ptr(y), fptr(stats),
                                ptr(ws), bytes, stream()), ndc_inorm_last_error());
        }
        return y;
    }

    static Tensor forward(AutogradContext* ctx, const Tensor& x, const std::optional<Tensor>& weight,
                          const std::optional<Tensor>& bias, double eps) {
        const Tensor w = weight ? *weight : Tensor();
        Tensor stats;
        Tensor y = run(x, as_f32(w), as_f32(bias ? *bias : Tensor()), eps, stats);
        ctx->save_for_backward({x, w, stats});
        // a bias without a weight keeps its gradient in float32
        ctx->saved_data["type"] = (int64_t)(w.defined() ? w.scalar_type() : at::kFloat);
        ctx->saved_data["bias"] = bias.has_value();
        return y;
    }

    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        variable_list out(4);
        {
            at::AutoGradMode off(false);
            const variable_list kept = ctx->get_saved_variables();
            const Tensor &x = kept[0], &w = kept[1], &stats = kept[2];
            c10::cuda::CUDAGuard guard(x.device());
            const Tensor g = like(grads[0], x);
            const Slabs s = slabs(x);
            const auto f32 = x.options().dtype(at::kFloat);
            Tensor gx = at::empty(x.sizes(), x.options()), gw, gb;
            if (w.defined() && ctx->needs_input_grad(1)) gw = at::empty({s.channels}, f32);
            // (gradients are counted over the tensors that are there)
            if (ctx->saved_data["bias"].toBool() && ctx->needs_input_grad(w.defined() ? 2 : 1)) gb = at::empty({s.channels}, f32);
            if (x.numel()) {
                const Tensor wf = as_f32(w);
                const size_t bytes = ndc_inorm_workspace_bytes(s.batch, s.channels);
                Tensor ws = at::empty({(int64_t)bytes}, x.options().dtype(at::kByte));
                check(ndc_inorm_bwd(s.batch, s.channels, s.n, dtype_code(x), ptr(x), ptr(g), fptr(wf), fptr(stats), ptr(gx), fptr(gw),
                                    fptr(gb), ptr(ws), bytes, stream()), ndc_inorm_last_error());
            } else {
                for (Tensor* t : {&gw, &gb}) if (t->defined()) t->zero_();
            }
            const auto type = (at::ScalarType)ctx->saved_data["type"].toInt();
            if (ctx->needs_input_grad(0)) out[0] = gx;
            out[1] = from_f32(gw, type);
            out[2] = from_f32(gb, type);
        }
        return once(grads, out);
    }
};

Tensor instance_norm(const Tensor& x_in, const std::optional<Tensor>& weight, const std::optional<Tensor>& bias, double eps) {
    for (const auto* t : {&weight, &bias})
        TORCH_CHECK(!*t || ((*t)->device() == x_in.device() && (*t)->numel() == x_in.size(1)),
                    "deconver_b200: instance norm parameters do not match the input ", x_in.sizes());
    c10::cuda::CUDAGuard guard(x_in.device());
    const Tensor x = x_in.contiguous(), w = weight ? *weight : Tensor(), b = bias ? *bias : Tensor();
    refuse_tangents({&x, &w, &b});
    if (wants_grad({&x, &w, &b})) return NormNode::apply(x, weight, bias, eps);
    at::AutoDispatchBelowADInplaceOrView below;
    Tensor stats;
    return NormNode::run(x, as_f32(w), as_f32(b), eps, stats);
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, mod) {
    mod.def("layer", &layer, py::call_guard<py::gil_scoped_release>());
    mod.def("linear", &linear, py::call_guard<py::gil_scoped_release>());
    mod.def("bias_gelu", &bias_gelu, py::call_guard<py::gil_scoped_release>());
    mod.def("instance_norm", &instance_norm, py::call_guard<py::gil_scoped_release>());
    mod.def("weight_grad_route", [](int64_t batch, int64_t co, int64_t ci, int64_t n, bool bf16, bool exact, int sms) {
        return (int)plan_weight_grad(batch, co, ci, n, bf16, exact, sms).route;
    });
    mod.def("timing_enable", &timing_enable);
    mod.def("timing_collect", &timing_collect);
}
