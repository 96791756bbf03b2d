// Native host path: the autograd functions of the operator library, from Python call to kernel launch.
//
// A small PAM call is bounded by its host side: described, checked, recorded for autograd and launched
// from Python, one 32 x 512 x 512 linear layer took 46 us around 8 us of GPU time, and a LayerNorm
// forward and backward 146 us around 27 us.  This module does the same work in C++: one call from
// Python per operator, arguments read straight from the interpreter (no argument tuples or
// keyword dictionaries), outputs and scratch from PyTorch's caching allocator, the gradient recorded
// as a torch::autograd::Node whose backward pass runs without the interpreter.  The kernels are those
// of libpam_b200.so, reached through its C ABI like the Python layer reaches them.
//
// Every entry point takes the common form of its operator (fp32 CUDA tensors on one device) and
// returns None for anything else; the caller then goes on in Python, which converts types, expands
// exotic broadcasts or raises the error that describes the mistake.
//
// Scratch is allocated per call: the caching allocator orders its reuse on the stream, keeps calls
// from several threads and streams apart, and takes it back.
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/autograd/variable.h>
#include <torch/csrc/dynamo/compiled_autograd.h>

#include <ATen/ATen.h>
#include <ATen/ExpandUtils.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>

#include <dlfcn.h>
#include <nvtx3/nvToolsExt.h>

#include <array>
#include <atomic>
#include <map>
#include <mutex>
#include <optional>
#include <string>
#include <vector>

#include "../../include/pam_b200.h"

namespace {

using at::Tensor;
using torch::autograd::edge_list;
using torch::autograd::Node;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;

// ---- the kernel library ---------------------------------------------------------------------------

// Entry points used here, bound by name from the library that the Python layer loaded: those that only answer, and
// those that launch.
#define PAMK_QUERIES(X)                                                                                   \
    X(pamk_status_string) X(pamk_last_cuda_error) X(pamk_matmul_auto_split) X(pamk_matmul_bwd_auto_split) \
    X(pamk_matmul_scratch_bytes) X(pamk_column_sum_workspace_bytes) X(pamk_layer_norm_max_width) X(pamk_layer_norm_stats_per_row)      \
    X(pamk_layer_norm_bwd_workspace_bytes) X(pamk_softmax_max_len) X(pamk_softmax_workspace_bytes)
#define PAMK_LAUNCHES(X)                                                                                  \
    X(pamk_pam_fwd) X(pamk_pad_fwd) X(pamk_pam_grad) X(pamk_pad_grad) X(pamk_matmul_bias)                 \
    X(pamk_matmul_strided) X(pamk_matmul_bwd) X(pamk_column_sum) X(pamk_layer_norm_fwd)                   \
    X(pamk_layer_norm_fwd_save) X(pamk_layer_norm_bwd) X(pamk_layer_norm_bwd_saved) X(pamk_softmax_fwd)   \
    X(pamk_softmax_fwd_save) X(pamk_softmax_bwd) X(pamk_softmax_bwd_saved) X(pamk_adam_step)

std::atomic<bool> g_nvtx{false};         // set_nvtx

// A launching entry point, inside an NVTX range of its name while those are on.
template <class F>
struct Launch {
    F* fn = nullptr;
    const char* label = "";
    template <class... A>
    int operator()(A&&... a) const {
        if (!g_nvtx.load(std::memory_order_relaxed)) return fn(std::forward<A>(a)...);
        nvtxRangePushA(label);
        const int status = fn(std::forward<A>(a)...);
        nvtxRangePop();
        return status;
    }
};

struct Library {
#define PAMK_MEMBER(name) decltype(&::name) name = nullptr;
    PAMK_QUERIES(PAMK_MEMBER)
#undef PAMK_MEMBER
#define PAMK_MEMBER(name) Launch<decltype(::name)> name;
    PAMK_LAUNCHES(PAMK_MEMBER)
#undef PAMK_MEMBER
};

Library lib;
PyObject* g_kernel_error = nullptr;      // the Python layer's PamKernelError
std::atomic<bool> g_strict{false};       // set_strict_k_order

// (a PyTorchError is what torch's own handlers, the autograd engine's included, turn into an exception of its Python type)
struct KernelError : torch::PyTorchError {
    using torch::PyTorchError::PyTorchError;
    PyObject* python_type() override { return g_kernel_error ? g_kernel_error : PyExc_RuntimeError; }
};

void check(int status, const char* what) {
    if (status == PAMK_OK) return;
    std::string msg = std::string(what) + ": " + lib.pamk_status_string(status);
    if (status == PAMK_ERR_CUDA) msg += " [cudaError " + std::to_string(lib.pamk_last_cuda_error()) + "]";
    throw KernelError(msg);
}

void* stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

Tensor empty_on(at::IntArrayRef shape, const Tensor& like) {
    return at::detail::empty_cuda(shape, at::kFloat, like.device(), std::nullopt);
}

Tensor scratch_bytes(size_t bytes, const Tensor& like) {
    return at::detail::empty_cuda({(int64_t)bytes}, at::kByte, like.device(), std::nullopt);
}

float* ptr(const Tensor& t) { return t.defined() ? static_cast<float*>(t.data_ptr()) : nullptr; }

// Whether forward-mode AD gave the tensor a tangent.  (Almost none ever had one: that is read from the tensor without a call,
// which an Adam step over 250 parameters asks a thousand times.)
bool has_tangent(const Tensor& t) {
    const auto* meta = static_cast<const torch::autograd::AutogradMeta*>(t.unsafeGetTensorImpl()->autograd_meta());
    return meta != nullptr && meta->fw_grad_ != nullptr && t._fw_grad(0).defined();
}

// fp32 CUDA data that the kernels may read in place: strided, no wrapper of other tensors (functorch, fake, functional), no
// lazy negation or zero.  A tensor with a tangent is for the Python layer, which refuses it: here the tangent
// would be lost without a word.
bool usable(const Tensor& t) {
    using K = c10::DispatchKey;
    constexpr c10::DispatchKeySet special({K::Python, K::PythonTLSSnapshot, K::FuncTorchBatched, K::FuncTorchGradWrapper, K::Batched,
                                           K::Functionalize, K::Conjugate, K::Negative, K::ZeroTensor, K::Sparse, K::SparseCsr, K::NestedTensor});
    return t.defined() && t.is_cuda() && t.scalar_type() == at::kFloat && !t.key_set().has_any(special) && !has_tangent(t);
}

bool wants_grad(const Tensor& t) { return t.defined() && t.requires_grad(); }

// Whether scratch that a call can do without is there to be had, in a cached block or from the device: asked for in vain, it would make torch's
// allocator give its whole cache back first, on every call.  (A cached block may turn out to be another stream's.)  A capture does
// not touch the cache and may not ask.  Other allocators than torch's own keep no such cache, and some refuse the questions (pluggable ones)
// or answer them by taking all memory that is free (cudaMallocAsync): they are just asked for the scratch.
bool room_for(size_t bytes, c10::DeviceIndex device) {
    c10::cuda::CUDAGuard guard(device);
    if (c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None) return true;
    auto* allocator = c10::cuda::CUDACachingAllocator::get();
    if (allocator->name() != "native") return true;
    size_t largest = 1;                   // (zero would stand for the device's free memory)
    allocator->cacheInfo(device, &largest);
    if (largest >= bytes) return true;
    constexpr size_t kUnit = size_t(2) << 20;                 // of the allocator's requests
    const size_t request = (bytes + kUnit - 1) / kUnit * kUnit;
    const auto [free, total] = allocator->getMemoryInfo(device);
    const auto reserved = allocator->getDeviceStats(device).reserved_bytes[0].current;
    return free >= request && (double)reserved + (double)request <= allocator->getMemoryFraction(device) * (double)total;
}

// ---- matrix products ----------------------------------------------------------------------------------

struct Mat {                              // element strides of one operand: batch, row, column
    const float* p;
    int64_t sb, sr, sc;
    Mat t() const { return {p, sb, sc, sr}; }
};

// A matrix whose last or second-to-last stride is 1 is used as it lies, any other is copied
// (pam/cuda_bindings.py:106-115); `t` keeps the copy alive.
Mat matrix(Tensor& t) {
    const int64_t d = t.dim();
    if (t.stride(d - 1) != 1 && t.stride(d - 2) != 1) t = t.contiguous();
    return {ptr(t), d == 3 ? t.stride(0) : 0, t.stride(d - 2), t.stride(d - 1)};
}

Tensor product(const Mat& a, const Mat& b, const Tensor& bias, int64_t batch, int64_t M, int64_t N, int64_t K, double offset,
               at::IntArrayRef out_shape, const Tensor& like) {
    Tensor out = empty_on(out_shape, like);
    const int split = g_strict.load(std::memory_order_relaxed) ? 1 : lib.pamk_matmul_auto_split(batch, M, N, K);
    Tensor ws;
    size_t bytes = split > 1 ? (size_t)split * batch * M * N * sizeof(float) : 0;
    if ((double)batch * (double)M * (double)N * (double)K > PAMK_PACKED_PRODUCTS) {
        // scratch for packed operands too; a product that cannot have it runs without
        const size_t packed = lib.pamk_matmul_scratch_bytes(batch, M, N, K, split);
        if (packed > bytes && room_for(packed, like.device().index())) {
            try {
                ws = scratch_bytes(packed, like);
                bytes = packed;
            } catch (const c10::OutOfMemoryError&) {
            }
        }
    }
    if (!ws.defined() && bytes != 0) ws = scratch_bytes(bytes, like);
    check(lib.pamk_matmul_bias(PAMK_MUL_PAM, a.p, b.p, ptr(bias), ptr(out), batch, M, N, K, a.sb, a.sr, a.sc, b.sb, b.sr, b.sc,
                               (float)offset, split, ws.defined() ? ws.data_ptr() : nullptr, bytes, stream_of(like)),
          "pamk_matmul");
    return out;
}

Tensor product_bwd(const Mat& l, const Mat& r, const Mat& d, bool delta_l, int64_t batch, int64_t M, int64_t N, int64_t K,
                   double offset, at::IntArrayRef out_shape, const Tensor& like) {
    Tensor out = empty_on(out_shape, like);
    const int split = g_strict.load(std::memory_order_relaxed) ? 1 : lib.pamk_matmul_bwd_auto_split(batch, M, N, K);
    Tensor ws;
    size_t bytes = 0;
    if (split > 1) {
        bytes = (size_t)split * batch * M * N * sizeof(float);
        ws = scratch_bytes(bytes, like);
    }
    check(lib.pamk_matmul_bwd(l.p, r.p, d.p, ptr(out), batch, M, N, K, l.sb, l.sr, l.sc, r.sb, r.sr, r.sc, d.sb, d.sr, d.sc,
                              delta_l, (float)offset, split, ws.defined() ? ws.data_ptr() : nullptr, bytes, stream_of(like)),
          "pamk_matmul_bwd");
    return out;
}

Tensor column_sum(const Tensor& x, int64_t rows, int64_t cols) {
    Tensor out = empty_on({cols}, x);
    const size_t bytes = lib.pamk_column_sum_workspace_bytes(rows, cols);
    Tensor ws = scratch_bytes(bytes, x);
    check(lib.pamk_column_sum(ptr(x), ptr(out), rows, cols, ws.data_ptr(), bytes, stream_of(x)), "pamk_column_sum");
    return out;
}

// One product of the attention path: the split is the plain product's of the same shape (none in strict k order).
void strided(const float* a, const float* b, float* c, int64_t outer, int64_t inner, int64_t M, int64_t N, int64_t K,
             const std::array<int64_t, 4>& sa, const std::array<int64_t, 4>& sb, const std::array<int64_t, 3>& sc,
             double offset, std::optional<double> post, const Tensor& like) {
    const int split = g_strict.load(std::memory_order_relaxed) ? 1 : lib.pamk_matmul_auto_split(outer * inner, M, N, K);
    Tensor ws;
    size_t bytes = 0;
    if (split > 1) {
        bytes = (size_t)split * outer * inner * M * N * sizeof(float);
        ws = scratch_bytes(bytes, like);
    }
    check(lib.pamk_matmul_strided(a, b, c, outer, inner, M, N, K, sa[0], sa[1], sa[2], sa[3], sb[0], sb[1], sb[2], sb[3],
                                  sc[0], sc[1], sc[2], (float)offset, post.has_value(), (float)post.value_or(0.0), split,
                                  ws.defined() ? ws.data_ptr() : nullptr, bytes, stream_of(like)),
          "pamk_matmul_strided");
}

// ---- elementwise operands --------------------------------------------------------------------------------

struct Operand {                          // (pointer, kind, immediate) of the C ABI; `keep` holds the data
    Tensor keep;
    int kind = PAMK_IMM;
    float imm = 0.0f;
    int64_t inner = 0;                    // row length of a ROW / COL operand
    const float* p() const { return ptr(keep); }
};

Operand number(double v) {
    Operand o;
    o.imm = (float)v;
    return o;
}

Operand full(const Tensor& t, at::IntArrayRef shape) {
    Operand o;
    o.keep = t.expand(shape).contiguous();
    o.kind = PAMK_FULL;
    return o;
}

// How a tensor is broadcast to `shape`, read in place where the kernels have a form for it.
Operand describe(const Tensor& given, at::IntArrayRef shape) {
    Operand o;
    if (given.sizes() == shape && given.is_contiguous()) {
        o.keep = given;
        o.kind = given.numel() == 1 ? PAMK_SCALAR : PAMK_FULL;
        return o;
    }
    Tensor t = given;
    for (int64_t d = 0; d < t.dim(); ++d)                 // expanded dimensions back to size 1
        if (t.stride(d) == 0 && t.size(d) > 1) t = t.narrow(d, 0, 1);
    if (t.numel() == 1) {
        o.keep = t;
        o.kind = PAMK_SCALAR;
        return o;
    }
    const int64_t nd = (int64_t)shape.size(), lead = nd - t.dim();
    auto size = [&](int64_t d) { return d < lead ? 1 : t.size(d - lead); };
    bool same = true;
    for (int64_t d = 0; d < nd; ++d) same = same && size(d) == shape[d];
    if (same) {
        o.keep = t.contiguous();
        o.kind = PAMK_FULL;
        return o;
    }
    for (int64_t j = 1; j < nd; ++j) {
        bool head_one = true, tail_one = true, head_same = true, tail_same = true;
        int64_t inner = 1;
        for (int64_t d = 0; d < nd; ++d) {
            (d < j ? head_one : tail_one) &= size(d) == 1;
            (d < j ? head_same : tail_same) &= size(d) == shape[d];
            if (d >= j) inner *= shape[d];
        }
        if ((head_one && tail_same) || (tail_one && head_same)) {
            o.keep = t.contiguous();
            o.kind = head_one && tail_same ? PAMK_ROW : PAMK_COL;
            o.inner = inner;
            return o;
        }
    }
    return full(t, shape);
}

// The operands of one launch share one row length; an operand that splits the output elsewhere is expanded.
int64_t shared_inner(std::initializer_list<Operand*> ops, at::IntArrayRef shape) {
    int64_t inner = 0;
    for (Operand* o : ops) {
        if (!o->inner) continue;
        if (!inner) {
            inner = o->inner;
        } else if (o->inner != inner) {
            // (its data are the compact ones: back to a view that broadcasts, then to full size)
            std::vector<int64_t> v;
            int64_t tail = 1;
            for (auto it = shape.rbegin(); it != shape.rend(); ++it) {
                const bool in_tail = tail < o->inner;
                v.insert(v.begin(), in_tail == (o->kind == PAMK_ROW) ? *it : 1);
                if (in_tail) tail *= *it;
            }
            *o = full(o->keep.reshape(v), shape);
        }
    }
    return inner;
}

Tensor reduce_to(const Tensor& g, at::IntArrayRef shape) { return g.sizes() == shape ? g : at::sum_to(g, shape); }

enum class Ew { kMul, kDiv };

Tensor ew_forward(Ew op, const Operand& a, const Operand& b, int64_t inner, at::IntArrayRef shape, double offset, const Tensor& like) {
    Tensor out = empty_on(shape, like);
    auto fn = op == Ew::kMul ? lib.pamk_pam_fwd : lib.pamk_pad_fwd;
    check(fn(a.p(), a.kind, a.imm, b.p(), b.kind, b.imm, ptr(out), out.numel(), inner, (float)offset, stream_of(like)),
          op == Ew::kMul ? "pamk_pam_fwd" : "pamk_pad_fwd");
    return out;
}

// ---- gradients ------------------------------------------------------------------------------------------------

// Which of its inputs' gradients a backward pass asks a rule for.
struct Wanted {
    uint32_t bits = 0;
    bool operator()(size_t k) const { return bits >> k & 1; }
};

// The backward pass of one operator: a rule holds the settings of the call, `kept` is what the forward pass kept.
template <class Rule>
variable_list backward_pass(const Rule& rule, const variable_list& kept, const Tensor& grad, const Wanted& wanted) {
    at::AutoGradMode no_grad(false);
    c10::cuda::CUDAGuard guard(grad.device());
    return rule.grads(kept, grad.scalar_type() == at::kFloat ? grad : grad.to(at::kFloat), wanted);
}

// The bytes of a rule's settings, which tell one compiled backward pass from another.
template <class... T>
std::string bytes_of(const T&... v) {
    std::string out;
    (out.append(reinterpret_cast<const char*>(&v), sizeof v), ...);
    return out;
}

std::string bytes_of_list(at::IntArrayRef v) { return bytes_of(v.size()).append(reinterpret_cast<const char*>(v.data()), v.size() * sizeof(int64_t)); }

// A node keeps its saved tensors until the engine releases them; apply() runs on an engine thread, without
// the interpreter, on the stream of the forward pass.
template <class Rule>
struct RuleNode : Node {
    Rule rule;
    std::vector<SavedVariable> saved;

    explicit RuleNode(Rule r) : rule(std::move(r)) {}
    std::string name() const override { return rule.name(); }
    void keep(std::initializer_list<Tensor> ts) {
        for (const Tensor& t : ts) saved.emplace_back(t, false);
    }
    void release_variables() override {
        std::lock_guard<std::mutex> lock(mutex_);
        for (auto& s : saved) s.reset_data();
    }
    variable_list unpacked() {
        variable_list kept;
        kept.reserve(saved.size());
        for (SavedVariable& s : saved) kept.push_back(s.unpack());
        return kept;
    }
    variable_list apply(variable_list&& in) override {
        std::lock_guard<std::mutex> lock(mutex_);
        const variable_list kept = unpacked();            // (unpack hooks run in the grad mode of the backward pass)
        Wanted wanted;
        for (size_t k = 0; k < num_outputs(); ++k) wanted.bits |= (uint32_t)task_should_compute_output(k) << k;
        // (a gradient that never came counts as zeros, as autograd.Function has it: the inputs get theirs)
        return backward_pass(rule, kept, in[0].defined() ? in[0] : input_metadata(0).zeros_like(), wanted);
    }

    // Compiled autograd: the backward pass becomes one opaque call in the graph, bound to the rule's settings.
    std::vector<int64_t> output_shape() const {
        std::vector<int64_t> shape;
        for (const c10::SymInt& n : input_metadata(0).shape_as_dim_vector()) shape.push_back(n.guard_int(__FILE__, __LINE__));
        return shape;
    }
    Wanted reachable() const {
        Wanted wanted;
        for (size_t k = 0; k < num_outputs(); ++k) wanted.bits |= (uint32_t)should_compute_output(k) << k;
        return wanted;
    }
    void compiled_args(torch::dynamo::autograd::CompiledNodeArgs& args) const override {
        args.collect(rule.name() + rule.key() + bytes_of_list(output_shape()) + bytes_of(reachable().bits));
        args.collect(saved, false);
    }
    variable_list apply_with_saved(const variable_list& inputs, torch::dynamo::autograd::SwapSavedVariables& swap) override {
        namespace ca = torch::dynamo::autograd;
        swap.before(saved);
        ca::PackedArgs args;
        args.pack(unpacked());
        const auto call = [rule = rule, wanted = reachable(), shape = output_shape(), options = input_metadata(0).options()](
                              const variable_list& in, const std::vector<c10::IValue>& packed) {
            const variable_list kept = ca::PackedArgs(packed).template unpack<variable_list>();
            return backward_pass(rule, kept, in[0].defined() ? in[0] : at::zeros(shape, options), wanted);
        };
        const auto& compiler = ca::getPyCompilerInterface();
        const std::string fn = compiler->bind_function(swap.get_py_compiler(), rule.name(), call, {c10::ListType::ofTensors()},
                                                       /*is_custom_function*/ true, /*is_traceable*/ false);
        const auto metadata = ca::IValuePacker<std::vector<std::optional<ca::InputMetadata>>>::pack(ca::get_input_metadata(next_edges()));
        variable_list out = compiler->call_function(swap.get_py_compiler(), "apply_functional", fn, inputs, args.vec(), metadata);
        swap.after(saved);
        return out;
    }
};

template <class Rule, class... Inputs>
std::shared_ptr<RuleNode<Rule>> node(Rule rule, const Inputs&... inputs) {
    std::shared_ptr<RuleNode<Rule>> fn(new RuleNode<Rule>(std::move(rule)), torch::autograd::deleteNode);
    fn->set_next_edges(torch::autograd::collect_next_edges(inputs...));
    return fn;
}

bool recording() { return at::GradMode::is_enabled(); }

struct EwRule {
    Ew op;
    double offset;
    bool approx_a, approx_b, has_a, has_b;
    double num_a = 0.0, num_b = 0.0;
    std::string name() const { return op == Ew::kMul ? "PamMulBackward" : "PamDivBackward"; }
    std::string key() const { return bytes_of(op, offset, approx_a, approx_b, has_a, has_b, num_a, num_b); }
    variable_list grads(const variable_list& kept, const Tensor& g, const Wanted& wanted) const {
        Tensor a, b;
        size_t k = 0;
        if (has_a) a = kept[k++];
        if (has_b) b = kept[k++];
        variable_list out(2);
        const bool na = has_a && wanted(0), nb = has_b && wanted(1);
        if (!na && !nb) return out;
        const auto shape = g.sizes();
        Operand oa = has_a ? describe(a, shape) : number(num_a), ob = has_b ? describe(b, shape) : number(num_b);
        Operand og = describe(g, shape);
        const int64_t inner = shared_inner({&oa, &ob, &og}, shape);
        Tensor da = na ? empty_on(shape, g) : Tensor(), db = nb ? empty_on(shape, g) : Tensor();
        auto fn = op == Ew::kMul ? lib.pamk_pam_grad : lib.pamk_pad_grad;
        check(fn(oa.p(), oa.kind, oa.imm, ob.p(), ob.kind, ob.imm, og.p(), og.kind, og.imm, ptr(da), ptr(db), g.numel(), inner,
                 (float)offset, approx_a, approx_b, stream_of(g)),
              op == Ew::kMul ? "pamk_pam_grad" : "pamk_pad_grad");
        if (na) out[0] = reduce_to(da, a.sizes());
        if (nb) out[1] = reduce_to(db, b.sizes());
        return out;
    }
};

// X [.., in] x W [out, in] (+ bias).  The weight gradient is formed as [out, in] like the weight itself (g^T X:
// the terms and the order over the tokens of X^T g), so nothing transposes it afterwards.
struct LinearRule {
    double offset;
    bool approx_x, approx_w, has_bias;
    std::string name() const { return "PamLinearBackward"; }
    std::string key() const { return bytes_of(offset, approx_x, approx_w, has_bias); }
    variable_list grads(const variable_list& kept, const Tensor& grad, const Wanted& wanted) const {
        Tensor x = kept[0], w = kept[1];
        const int64_t in = w.size(1), out_f = w.size(0), rows = x.numel() / in;
        Tensor g2 = grad.reshape({rows, out_f}), x2 = x.reshape({rows, in});
        const Mat g = matrix(g2), mx = matrix(x2), mw = matrix(w);
        variable_list out(has_bias ? 3 : 2);
        if (wanted(0))
            out[0] = approx_x ? product(g, mw, Tensor(), 1, rows, in, out_f, offset, x.sizes(), x)
                              : product_bwd(g, mw, mx, true, 1, rows, in, out_f, offset, x.sizes(), x);
        if (wanted(1))
            out[1] = approx_w ? product(g.t(), mx, Tensor(), 1, out_f, in, rows, offset, w.sizes(), x)
                              : product_bwd(g.t(), mx, mw, true, 1, out_f, in, rows, offset, w.sizes(), x);
        if (has_bias && wanted(2)) out[2] = column_sum(g2.contiguous(), rows, out_f);
        return out;
    }
};

struct MatMulRule {
    double offset;
    bool approx_a, approx_b;
    std::string name() const { return "PamMatMulBackward"; }
    std::string key() const { return bytes_of(offset, approx_a, approx_b); }
    variable_list grads(const variable_list& kept, const Tensor& grad, const Wanted& wanted) const {
        Tensor a = kept[0], b = kept[1], g2 = grad;
        const int64_t d = a.dim(), batch = d == 3 ? a.size(0) : 1, M = a.size(d - 2), K = a.size(d - 1), N = b.size(d - 1);
        const Mat ma = matrix(a), mb = matrix(b), g = matrix(g2);
        variable_list out(2);
        if (wanted(0))
            out[0] = approx_a ? product(g, mb.t(), Tensor(), batch, M, K, N, offset, a.sizes(), a)
                              : product_bwd(g, mb.t(), ma, true, batch, M, K, N, offset, a.sizes(), a);
        if (wanted(1))
            out[1] = approx_b ? product(ma.t(), g, Tensor(), batch, K, N, M, offset, b.sizes(), a)
                              : product_bwd(ma.t(), g, mb, false, batch, K, N, M, offset, b.sizes(), a);
        return out;
    }
};

// The approximate backward pass works from eight scalars per row that the forward pass kept.
struct LayerNormRule {
    double eps, offset;
    bool approx, has_w, has_b;
    int64_t width;
    std::vector<int64_t> b_shape;
    std::string name() const { return "PamLayerNormBackward"; }
    std::string key() const { return bytes_of(eps, offset, approx, has_w, has_b, width) + bytes_of_list(b_shape); }
    variable_list grads(const variable_list& kept, const Tensor& grad, const Wanted& wanted) const {
        size_t k = 0;
        Tensor x = kept[k++], w, stats;
        if (has_w) w = kept[k++];
        if (approx) stats = kept[k++];
        const Tensor g = grad.contiguous();
        const int64_t rows = x.numel() / width;
        Tensor dx = empty_on(x.sizes(), x);
        const bool nw = has_w && wanted(1), nb = has_b && wanted(has_w ? 2 : 1);
        Tensor dw = nw ? empty_on(w.sizes(), x) : Tensor(), db = nb ? empty_on(b_shape, x) : Tensor();
        Tensor ws;
        size_t bytes = 0;
        if (nw || nb) {
            bytes = lib.pamk_layer_norm_bwd_workspace_bytes(rows, width);
            ws = scratch_bytes(bytes, x);
        }
        void* wsp = ws.defined() ? ws.data_ptr() : nullptr;
        check(approx ? lib.pamk_layer_norm_bwd_saved(ptr(x), ptr(w), ptr(g), ptr(stats), ptr(dx), ptr(dw), ptr(db), rows, width,
                                                     (float)offset, wsp, bytes, stream_of(x))
                     : lib.pamk_layer_norm_bwd(ptr(x), ptr(w), ptr(g), ptr(dx), ptr(dw), ptr(db), rows, width, (float)eps,
                                               (float)offset, 0, wsp, bytes, stream_of(x)),
              "pamk_layer_norm_bwd");
        variable_list out(1 + has_w + has_b);
        out[0] = dx;
        if (has_w) out[1] = dw;
        if (has_b) out[1 + has_w] = db;
        return out;
    }
};

void softmax_forward(const Tensor& x, const Tensor& y, const Tensor& e, int64_t rows, int64_t len, double offset) {
    const size_t bytes = lib.pamk_softmax_workspace_bytes(rows, len);
    Tensor ws = scratch_bytes(bytes, x);
    check(e.defined() ? lib.pamk_softmax_fwd_save(ptr(x), ptr(y), ptr(e), rows, len, (float)offset, ws.data_ptr(), bytes, stream_of(x))
                      : lib.pamk_softmax_fwd(ptr(x), ptr(y), rows, len, (float)offset, ws.data_ptr(), bytes, stream_of(x)),
          "pamk_softmax_fwd");
}

Tensor softmax_backward_saved(const Tensor& e, const Tensor& g, int64_t rows, int64_t len, double offset, std::optional<double> post,
                              at::IntArrayRef shape) {
    Tensor dx = empty_on(shape, e);
    check(lib.pamk_softmax_bwd_saved(ptr(e), ptr(g), ptr(dx), rows, len, (float)offset, post.has_value(), (float)post.value_or(0.0),
                                     stream_of(e)),
          "pamk_softmax_bwd_saved");
    return dx;
}

// With the approximate backward the forward pass keeps its exponentials instead of its input.
struct SoftmaxRule {
    double offset;
    bool approx;
    std::string name() const { return "PamSoftmaxBackward"; }
    std::string key() const { return bytes_of(offset, approx); }
    variable_list grads(const variable_list& kept, const Tensor& grad, const Wanted& wanted) const {
        const Tensor &from = kept[0], g = grad.contiguous();
        const int64_t len = from.size(-1), rows = from.numel() / len;
        if (approx) return {softmax_backward_saved(from, g, rows, len, offset, std::nullopt, from.sizes())};
        Tensor dx = empty_on(from.sizes(), from);
        const size_t bytes = lib.pamk_softmax_workspace_bytes(rows, len);
        Tensor ws = scratch_bytes(bytes, from);
        check(lib.pamk_softmax_bwd(ptr(from), ptr(g), ptr(dx), rows, len, (float)offset, 0, ws.data_ptr(), bytes, stream_of(from)),
              "pamk_softmax_bwd");
        return {dx};
    }
};

// softmax(pam(q k^T, scale)) v on the heads of a fused projection [B, N, 3, heads, head_dim] read in place, the
// context written token-major; the approximate gradients (see fused.py for the correspondence with the chain).
struct AttentionQkvRule {
    int64_t heads;
    double scale, offset;
    std::string name() const { return "PamAttentionQkvBackward"; }
    std::string key() const { return bytes_of(heads, scale, offset); }
    variable_list grads(const variable_list& kept, const Tensor& grad, const Wanted& wanted) const {
        const Tensor qkv = kept[0], expo = kept[1], probs = kept[2], g = grad.contiguous();
        const int64_t B = qkv.size(0), N = qkv.size(1), C3 = qkv.size(2), C = C3 / 3, hd = C / heads;
        const float *q = ptr(qkv), *k = q + C, *v = q + 2 * C;
        Tensor dqkv = empty_on(qkv.sizes(), qkv);
        float *dq = ptr(dqkv), *dv = dq + 2 * C;
        const int64_t H = heads * N * N, NN = N * N;
        Tensor dprobs = empty_on({B * heads, N, N}, qkv);
        strided(ptr(g), v, ptr(dprobs), B, heads, N, N, hd, {N * C, hd, C, 1}, {N * C3, hd, 1, C3}, {H, NN, N}, offset, std::nullopt, qkv);
        strided(ptr(probs), ptr(g), dv, B, heads, N, hd, N, {H, NN, 1, N}, {N * C, hd, C, 1}, {N * C3, hd, C3}, offset, std::nullopt, qkv);
        Tensor ds = softmax_backward_saved(expo, dprobs, B * heads * N, N, offset, scale, dprobs.sizes());
        strided(ptr(ds), k, dq, B, heads, N, hd, N, {H, NN, N, 1}, {N * C3, hd, C3, 1}, {N * C3, hd, C3}, offset, std::nullopt, qkv);
        // d k = (d scores)^T q, where d k lives in d qkv: the terms and the order of the chain's q^T d scores
        strided(ptr(ds), q, dq + C, B, heads, N, hd, N, {H, NN, 1, N}, {N * C3, hd, C3, 1}, {N * C3, hd, C3}, offset, std::nullopt, qkv);
        return {dqkv};
    }
};

// The same for separate projections q [B, T, d], k, v [B, S, d] and an additive mask.
struct AttentionHeadsRule {
    int64_t heads;
    double offset;
    std::string name() const { return "PamAttentionHeadsBackward"; }
    std::string key() const { return bytes_of(heads, offset); }
    variable_list grads(const variable_list& kept, const Tensor& grad, const Wanted& wanted) const {
        const Tensor q = kept[0], k = kept[1], v = kept[2], expo = kept[3], probs = kept[4], g = grad.contiguous();
        const int64_t B = q.size(0), T = q.size(1), d = q.size(2), S = k.size(1), hd = d / heads;
        const int64_t H = heads * T * S, TS = T * S;
        variable_list out(3);
        Tensor dprobs = empty_on({B * heads, T, S}, q);
        strided(ptr(g), ptr(v), ptr(dprobs), B, heads, T, S, hd, {T * d, hd, d, 1}, {S * d, hd, 1, d}, {H, TS, S}, offset, std::nullopt, q);
        out[2] = empty_on(v.sizes(), v);
        strided(ptr(probs), ptr(g), ptr(out[2]), B, heads, S, hd, T, {H, TS, 1, S}, {T * d, hd, d, 1}, {S * d, hd, d}, offset, std::nullopt, q);
        Tensor ds = softmax_backward_saved(expo, dprobs, B * heads * T, S, offset, std::nullopt, dprobs.sizes());
        out[0] = empty_on(q.sizes(), q);
        strided(ptr(ds), ptr(k), ptr(out[0]), B, heads, T, hd, S, {H, TS, S, 1}, {S * d, hd, d, 1}, {T * d, hd, d}, offset, std::nullopt, q);
        out[1] = empty_on(k.sizes(), k);
        strided(ptr(ds), ptr(q), ptr(out[1]), B, heads, S, hd, T, {H, TS, 1, S}, {T * d, hd, d, 1}, {S * d, hd, d}, offset, std::nullopt, q);
        return out;
    }
};

// ---- operators -----------------------------------------------------------------------------------------------

std::optional<Tensor> op_linear(const Tensor& x, const Tensor& w, const Tensor& bias, double offset, bool approx_x, bool approx_w) {
    if (!usable(x) || !usable(w) || x.dim() < 1 || w.dim() != 2 || x.size(-1) != w.size(1) || w.device() != x.device()) return {};
    if (bias.defined() && !(usable(bias) && bias.device() == x.device() && bias.dim() == 1 && bias.size(0) == w.size(0) && bias.is_contiguous()))
        return {};
    if (x.numel() == 0 || w.numel() == 0) return {};
    c10::cuda::CUDAGuard guard(x.device());
    const int64_t in = w.size(1), out_f = w.size(0), rows = x.numel() / in;
    at::DimVector shape(x.sizes());
    shape.back() = out_f;
    Tensor y;
    {
        at::AutoGradMode no_grad(false);
        Tensor x2 = x.dim() == 2 ? x : x.reshape({rows, in}), w2 = w;
        const Mat mx = matrix(x2), mw = matrix(w2);
        y = product(mx, mw.t(), bias, 1, rows, out_f, in, offset, shape, x);
    }
    if (recording() && (wants_grad(x) || wants_grad(w) || wants_grad(bias))) {
        const LinearRule rule{offset, approx_x, approx_w, bias.defined()};
        auto fn = bias.defined() ? node(rule, x, w, bias) : node(rule, x, w);
        fn->keep({x, w});
        torch::autograd::set_history(y, fn);
    }
    return y;
}

std::optional<Tensor> op_matmul(const Tensor& a, const Tensor& b, double offset, bool approx_a, bool approx_b, int64_t dims) {
    if (!usable(a) || !usable(b) || a.device() != b.device() || a.dim() != dims || b.dim() != dims) return {};
    if (a.size(-1) != b.size(-2) || (dims == 3 && a.size(0) != b.size(0)) || a.numel() == 0 || b.numel() == 0) return {};
    c10::cuda::CUDAGuard guard(a.device());
    const int64_t batch = dims == 3 ? a.size(0) : 1, M = a.size(-2), K = a.size(-1), N = b.size(-1);
    Tensor y;
    {
        at::AutoGradMode no_grad(false);
        Tensor a2 = a, b2 = b;
        const Mat ma = matrix(a2), mb = matrix(b2);
        const int64_t shape[3] = {batch, M, N};
        y = product(ma, mb, Tensor(), batch, M, N, K, offset, at::IntArrayRef(shape + (3 - dims), dims), a);
    }
    if (recording() && (wants_grad(a) || wants_grad(b))) {
        auto fn = node(MatMulRule{offset, approx_a, approx_b}, a, b);
        fn->keep({a, b});
        torch::autograd::set_history(y, fn);
    }
    return y;
}

// a and b: tensors, or numbers where undefined
std::optional<Tensor> op_elementwise(Ew op, const Tensor& a, double num_a, const Tensor& b, double num_b, double offset, bool approx_a, bool approx_b) {
    const bool has_a = a.defined(), has_b = b.defined();
    const Tensor& like = has_a ? a : b;
    if ((has_a && !usable(a)) || (has_b && !usable(b)) || (!has_a && !has_b)) return {};
    if (has_a && has_b && a.device() != b.device()) return {};
    if (like.numel() == 0 || (has_b && b.numel() == 0)) return {};
    if (!has_a && op == Ew::kDiv && like.dim() == 0) return {};      // (Python gives number / 0-d tensor one dimension)
    c10::cuda::CUDAGuard guard(like.device());
    Tensor y;
    {
        at::AutoGradMode no_grad(false);
        at::DimVector shape(like.sizes());
        if (has_a && has_b && a.sizes() != b.sizes()) {
            // (shapes that do not broadcast: Python raises)
            const int64_t nd = std::max(a.dim(), b.dim());
            for (int64_t d = 1; d <= std::min(a.dim(), b.dim()); ++d)
                if (a.size(-d) != b.size(-d) && a.size(-d) != 1 && b.size(-d) != 1) return {};
            shape.resize(nd);
            for (int64_t d = 1; d <= nd; ++d) {
                const int64_t u = d <= a.dim() ? a.size(-d) : 1, v = d <= b.dim() ? b.size(-d) : 1;
                shape[nd - d] = u == 1 ? v : u;
            }
        }
        Operand oa = has_a ? describe(a, shape) : number(num_a), ob = has_b ? describe(b, shape) : number(num_b);
        const int64_t inner = shared_inner({&oa, &ob}, shape);
        y = ew_forward(op, oa, ob, inner, shape, offset, like);
    }
    if (recording() && (wants_grad(a) || wants_grad(b))) {
        auto fn = node(EwRule{op, offset, approx_a, approx_b, has_a, has_b, num_a, num_b}, a, b);
        if (has_a) fn->keep({a});
        if (has_b) fn->keep({b});
        torch::autograd::set_history(y, fn);
    }
    return y;
}

std::optional<Tensor> op_layer_norm(const Tensor& x, int64_t width, const Tensor& w, const Tensor& b, double eps, double offset, bool approx) {
    if (!usable(x) || width <= 0 || width > lib.pamk_layer_norm_max_width() || x.numel() == 0) return {};
    for (const Tensor* p : {&w, &b})
        if (p->defined() && !(usable(*p) && p->device() == x.device() && p->numel() == width && p->is_contiguous())) return {};
    c10::cuda::CUDAGuard guard(x.device());
    const int64_t rows = x.numel() / width;
    const bool keep = recording() && (wants_grad(x) || wants_grad(w) || wants_grad(b));
    Tensor xc, y, stats;
    {
        at::AutoGradMode no_grad(false);
        xc = x.contiguous();
        y = empty_on(x.sizes(), x);
        if (keep && approx) stats = empty_on({rows, lib.pamk_layer_norm_stats_per_row()}, x);
        check(stats.defined() ? lib.pamk_layer_norm_fwd_save(ptr(xc), ptr(w), ptr(b), ptr(y), ptr(stats), rows, width, (float)eps,
                                                             (float)offset, stream_of(x))
                              : lib.pamk_layer_norm_fwd(ptr(xc), ptr(w), ptr(b), ptr(y), rows, width, (float)eps, (float)offset, stream_of(x)),
              "pamk_layer_norm_fwd");
    }
    if (keep) {
        LayerNormRule rule{eps, offset, approx, w.defined(), b.defined(), width, {}};
        if (b.defined()) rule.b_shape = b.sizes().vec();
        auto fn = w.defined() ? (b.defined() ? node(rule, x, w, b) : node(rule, x, w)) : (b.defined() ? node(rule, x, b) : node(rule, x));
        fn->keep({xc});
        if (w.defined()) fn->keep({w});
        if (approx) fn->keep({stats});
        torch::autograd::set_history(y, fn);
    }
    return y;
}

std::optional<Tensor> op_softmax(const Tensor& x, double offset, bool approx) {
    if (!usable(x) || x.dim() == 0 || x.numel() == 0 || x.size(-1) > lib.pamk_softmax_max_len()) return {};
    c10::cuda::CUDAGuard guard(x.device());
    const int64_t len = x.size(-1), rows = x.numel() / len;
    const bool keep = recording() && wants_grad(x);
    Tensor xc, y, e;
    {
        at::AutoGradMode no_grad(false);
        xc = x.contiguous();
        y = empty_on(x.sizes(), x);
        if (keep && approx) e = empty_on(x.sizes(), x);
        softmax_forward(xc, y, e, rows, len, offset);
    }
    if (keep) {
        auto fn = node(SoftmaxRule{offset, approx}, x);
        fn->keep({approx ? e : xc});
        torch::autograd::set_history(y, fn);
    }
    return y;
}

std::optional<Tensor> op_attention_qkv(const Tensor& given, int64_t heads, double scale, double offset) {
    if (!usable(given) || given.dim() != 3 || given.numel() == 0 || heads <= 0 || given.size(2) % (3 * heads)) return {};
    if (given.size(1) > lib.pamk_softmax_max_len() || given.size(0) * heads > 65535) return {};
    c10::cuda::CUDAGuard guard(given.device());
    const bool keep = recording() && wants_grad(given);
    Tensor qkv, out, probs, expo;
    {
        at::AutoGradMode no_grad(false);
        qkv = given.contiguous();
        const int64_t B = qkv.size(0), N = qkv.size(1), C3 = qkv.size(2), C = C3 / 3, hd = C / heads;
        const float *q = ptr(qkv), *k = q + C, *v = q + 2 * C;
        Tensor scores = empty_on({B * heads, N, N}, qkv);
        strided(q, k, ptr(scores), B, heads, N, N, hd, {N * C3, hd, C3, 1}, {N * C3, hd, 1, C3}, {heads * N * N, N * N, N}, offset, scale, qkv);
        probs = empty_on(scores.sizes(), qkv);
        if (keep) expo = empty_on(scores.sizes(), qkv);
        softmax_forward(scores, probs, expo, B * heads * N, N, offset);
        out = empty_on({B, N, C}, qkv);
        strided(ptr(probs), v, ptr(out), B, heads, N, hd, N, {heads * N * N, N * N, N, 1}, {N * C3, hd, C3, 1}, {N * C, hd, C}, offset,
                std::nullopt, qkv);
    }
    if (keep) {
        auto fn = node(AttentionQkvRule{heads, scale, offset}, given);
        fn->keep({qkv, expo, probs});
        torch::autograd::set_history(out, fn);
    }
    return out;
}

std::optional<Tensor> op_attention_heads(const Tensor& gq, const Tensor& gk, const Tensor& gv, const Tensor& mask, int64_t heads, double offset) {
    for (const Tensor* t : {&gq, &gk, &gv})
        if (!usable(*t) || t->dim() != 3 || t->device() != gq.device() || t->numel() == 0) return {};
    if (gk.sizes() != gv.sizes() || gq.size(0) != gk.size(0) || gq.size(2) != gk.size(2) || heads <= 0 || gq.size(2) % heads) return {};
    if (gq.size(0) * heads > 65535 || gk.size(1) > lib.pamk_softmax_max_len()) return {};
    if (mask.defined() && (!usable(mask) || mask.device() != gq.device() || mask.requires_grad())) return {};
    c10::cuda::CUDAGuard guard(gq.device());
    const bool keep = recording() && (wants_grad(gq) || wants_grad(gk) || wants_grad(gv));
    Tensor q, k, v, out, probs, expo;
    {
        at::AutoGradMode no_grad(false);
        q = gq.contiguous();
        k = gk.contiguous();
        v = gv.contiguous();
        const int64_t B = q.size(0), T = q.size(1), d = q.size(2), S = k.size(1), hd = d / heads;
        Tensor scores = empty_on({B * heads, T, S}, q);
        strided(ptr(q), ptr(k), ptr(scores), B, heads, T, S, hd, {T * d, hd, d, 1}, {S * d, hd, 1, d}, {heads * T * S, T * S, S}, offset,
                std::nullopt, q);
        if (mask.defined()) scores.add_(mask);
        probs = empty_on(scores.sizes(), q);
        if (keep) expo = empty_on(scores.sizes(), q);
        softmax_forward(scores, probs, expo, B * heads * T, S, offset);
        out = empty_on({B, T, d}, q);
        strided(ptr(probs), ptr(v), ptr(out), B, heads, T, hd, S, {heads * T * S, T * S, S, 1}, {S * d, hd, d, 1}, {T * d, hd, d}, offset,
                std::nullopt, q);
    }
    if (keep) {
        auto fn = node(AttentionHeadsRule{heads, offset}, gq, gk, gv);
        fn->keep({q, k, v, expo, probs});
        torch::autograd::set_history(out, fn);
    }
    return out;
}

// ---- Python entry points -----------------------------------------------------------------------------------------

// Reads a tensor argument: undefined for None, false for anything that is neither (a subclass other than
// Parameter included: it may override operators that the Python layer calls).
bool as_tensor(PyObject* o, Tensor& t) {
    if (o == Py_None) return true;
    if (!THPVariable_CheckExact(o)) return false;
    t = THPVariable_Unpack(o);
    return true;
}

bool as_number(PyObject* o, double& v) {
    if (PyFloat_Check(o)) { v = PyFloat_AS_DOUBLE(o); return true; }
    if (PyLong_Check(o)) {
        v = PyLong_AsDouble(o);
        if (v == -1.0 && PyErr_Occurred()) { PyErr_Clear(); return false; }
        return true;
    }
    return false;
}

// offset: None turns it off (1.0), as cuda_bindings.py:31-32
bool as_offset(PyObject* o, double& v) {
    if (o == Py_None) { v = 1.0; return true; }
    return as_number(o, v);
}

// approx_bwd: one flag, or a (first, second) pair
bool as_pair(PyObject* o, bool& a, bool& b) {
    if (o == Py_True || o == Py_False) { a = b = o == Py_True; return true; }
    if ((PyTuple_Check(o) || PyList_Check(o)) && PySequence_Fast_GET_SIZE(o) == 2) {
        const int x = PyObject_IsTrue(PySequence_Fast_GET_ITEM(o, 0)), y = PyObject_IsTrue(PySequence_Fast_GET_ITEM(o, 1));
        if (x < 0 || y < 0) { PyErr_Clear(); return false; }
        a = x != 0;
        b = y != 0;
        return true;
    }
    return false;
}

bool as_int(PyObject* o, int64_t& v) {
    if (!PyLong_Check(o)) return false;
    v = PyLong_AsLongLong(o);
    if (v == -1 && PyErr_Occurred()) { PyErr_Clear(); return false; }
    return true;
}

PyObject* none() { Py_RETURN_NONE; }

// Gives the interpreter's lock away while other Python threads exist: an allocation or a launch may wait for the GPU, and they
// go on meanwhile.  (A program of one thread keeps it: giving it away and taking it back costs 0.3 us.)
struct Unlocked {
    PyThreadState* mine = nullptr;
    Unlocked() {
        const PyThreadState* me = PyThreadState_Get();
        if (me->next != nullptr || me->prev != nullptr) mine = PyEval_SaveThread();
    }
    ~Unlocked() {
        if (mine != nullptr) PyEval_RestoreThread(mine);
    }
    Unlocked(const Unlocked&) = delete;
};

template <class F>
PyObject* wrapped(F&& op) {
    std::optional<Tensor> t;
    {
        const Unlocked others_may_run;
        t = op();
    }
    return t ? THPVariable_Wrap(std::move(*t)) : none();
}

// Whether nothing watches or transforms the operators that run.  A trace would keep an answer of this path as a constant,
// a dispatch mode would not see its allocations, and functorch's transforms refuse autograd functions like
// these whether or not an operand is wrapped: the Python layer's functions take such a call.
bool unwatched() {
    using K = c10::DispatchKey;
    constexpr c10::DispatchKeySet watching({K::Tracer, K::Python, K::PythonTLSSnapshot, K::FuncTorchDynamicLayerFrontMode,
                                            K::Functionalize});
    return !c10::impl::tls_local_dispatch_key_set().included_.has_any(watching);
}

// Torch's translation of exceptions: one raised by Python code further down (a saved-tensor hook) goes on as it
// is, an allocation that fails is an OutOfMemoryError.
template <class F>
PyObject* guarded(F&& body) {
    try {
        return body();
    } catch (...) {
        torch::translate_exception_to_python(std::current_exception());
        return nullptr;
    }
}

// An operator's entry: `body`, or None where the call is for the Python layer.
template <class F>
PyObject* operator_call(F&& body) {
    return unwatched() ? guarded(std::forward<F>(body)) : none();
}

#define PAMK_ARGS(count)                                                                            \
    if (nargs != (count)) {                                                                         \
        PyErr_SetString(PyExc_TypeError, "wrong number of arguments");                              \
        return nullptr;                                                                             \
    }

// linear(x, weight, bias | None, offset, approx_bwd)
PyObject* py_linear(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
    PAMK_ARGS(5)
    return operator_call([&]() -> PyObject* {
        Tensor x, w, b;
        double off;
        bool p, q;
        if (!as_tensor(a[0], x) || !as_tensor(a[1], w) || !as_tensor(a[2], b) || !as_offset(a[3], off) || !as_pair(a[4], p, q)) return none();
        return wrapped([&] { return op_linear(x, w, b, off, p, q); });
    });
}

// matmul(a, b, offset, approx_bwd, dims)
PyObject* py_matmul(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
    PAMK_ARGS(5)
    return operator_call([&]() -> PyObject* {
        Tensor x, y;
        double off;
        bool p, q;
        int64_t dims;
        if (!as_tensor(a[0], x) || !as_tensor(a[1], y) || !as_offset(a[2], off) || !as_pair(a[3], p, q) || !as_int(a[4], dims)) return none();
        return wrapped([&] { return op_matmul(x, y, off, p, q, dims); });
    });
}

template <Ew OP>
PyObject* py_elementwise(PyObject*, PyObject* const* a, Py_ssize_t nargs) {   // (a, b, offset, approx_bwd)
    PAMK_ARGS(4)
    return operator_call([&]() -> PyObject* {
        Tensor x, y;
        double nx = 0.0, ny = 0.0, off;
        bool p, q;
        if (!(as_number(a[0], nx) || (as_tensor(a[0], x) && x.defined())) || !(as_number(a[1], ny) || (as_tensor(a[1], y) && y.defined())))
            return none();
        if (!as_offset(a[2], off) || !as_pair(a[3], p, q)) return none();
        return wrapped([&] { return op_elementwise(OP, x, nx, y, ny, off, p, q); });
    });
}

// layer_norm(x, width, weight | None, bias | None, eps, offset, approx_bwd)
PyObject* py_layer_norm(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
    PAMK_ARGS(7)
    return operator_call([&]() -> PyObject* {
        Tensor x, w, b;
        int64_t width;
        double eps, off;
        bool p, q;
        if (!as_tensor(a[0], x) || !as_int(a[1], width) || !as_tensor(a[2], w) || !as_tensor(a[3], b) || !as_number(a[4], eps) ||
            !as_offset(a[5], off) || !as_pair(a[6], p, q) || p != q)
            return none();
        return wrapped([&] { return op_layer_norm(x, width, w, b, eps, off, p); });
    });
}

// softmax(x, offset, approx_bwd) over the last dimension
PyObject* py_softmax(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
    PAMK_ARGS(3)
    return operator_call([&]() -> PyObject* {
        Tensor x;
        double off;
        bool p, q;
        if (!as_tensor(a[0], x) || !as_offset(a[1], off) || !as_pair(a[2], p, q) || p != q) return none();
        return wrapped([&] { return op_softmax(x, off, p); });
    });
}

// attention_qkv(qkv, heads, scale, offset)
PyObject* py_attention_qkv(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
    PAMK_ARGS(4)
    return operator_call([&]() -> PyObject* {
        Tensor x;
        int64_t heads;
        double scale, off;
        if (!as_tensor(a[0], x) || !as_int(a[1], heads) || !as_number(a[2], scale) || !as_offset(a[3], off)) return none();
        return wrapped([&] { return op_attention_qkv(x, heads, scale, off); });
    });
}

// attention_heads(q, k, v, mask | None, heads, offset)
PyObject* py_attention_heads(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
    PAMK_ARGS(6)
    return operator_call([&]() -> PyObject* {
        Tensor q, k, v, m;
        int64_t heads;
        double off;
        if (!as_tensor(a[0], q) || !as_tensor(a[1], k) || !as_tensor(a[2], v) || !as_tensor(a[3], m) || !as_int(a[4], heads) ||
            !as_offset(a[5], off))
            return none();
        return wrapped([&] { return op_attention_heads(q, k, v, m, heads, off); });
    });
}

// One parameter's part of an Adam step.
struct AdamEntry {
    Tensor p, g, m, v;
    PyObject* state;      // borrowed: the optimizer's dict of this parameter
    int64_t step;         // before the update
};

// adam_collect(params, state): for one parameter group, whether every parameter with a gradient is in the form that
// the fused update takes and has its state; then [(step, capsule of tensors)] comes back, one entry for each
// distinct step count and device.  Nothing is changed: adam_apply counts the steps, once they are taken.
struct AdamBatch {
    std::vector<Tensor> keep;
    std::vector<PyObject*> states;      // the optimizer's dicts, held
    PyObject* step = nullptr;           // the count that they get
    AdamBatch() = default;
    AdamBatch(const AdamBatch&) = delete;
    ~AdamBatch() {
        for (PyObject* st : states) Py_DECREF(st);
        Py_XDECREF(step);
    }
    std::vector<float*> p, m, v;
    std::vector<const float*> g;
    std::vector<int64_t> n;
};
const char* kAdamCapsule = "pam_b200.adam_batch";

PyObject* step_key() {
    static PyObject* key = PyUnicode_InternFromString("step");
    return key;
}

PyObject* py_adam_collect(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
    PAMK_ARGS(2)
    static PyObject *k_m = PyUnicode_InternFromString("exp_avg"), *k_v = PyUnicode_InternFromString("exp_avg_sq");
    return guarded([&]() -> PyObject* {
        if (!PyList_Check(a[0]) || !PyDict_Check(a[1])) return none();
        std::vector<AdamEntry> found;
        const Py_ssize_t count = PyList_GET_SIZE(a[0]);
        found.reserve(count);
        for (Py_ssize_t i = 0; i < count; ++i) {
            PyObject* po = PyList_GET_ITEM(a[0], i);
            if (!THPVariable_Check(po)) return none();
            AdamEntry e;
            e.p = THPVariable_Unpack(po);
            e.g = e.p.grad();
            if (!e.g.defined()) continue;
            PyObject* st = PyDict_GetItemWithError(a[1], po);
            if (st == nullptr) {
                if (PyErr_Occurred()) return nullptr;
                return none();
            }
            if (!PyDict_Check(st)) return none();
            PyObject *step = PyDict_GetItem(st, step_key()), *m = PyDict_GetItem(st, k_m), *v = PyDict_GetItem(st, k_v);
            if (step == nullptr || m == nullptr || v == nullptr || !PyLong_CheckExact(step) || !THPVariable_Check(m) || !THPVariable_Check(v)) return none();
            e.m = THPVariable_Unpack(m);
            e.v = THPVariable_Unpack(v);
            for (const Tensor* t : {&e.p, &e.g, &e.m, &e.v})
                if (!usable(*t) || !t->is_contiguous() || t->device() != e.p.device() || t->numel() != e.p.numel()) return none();
            e.state = st;
            if (!as_int(step, e.step)) return none();
            found.push_back(std::move(e));
        }
        // A parameter that is listed twice takes two steps, one after the other: one launch would run both at once.
        // (a hash table of the states: sorting them took a tenth of the collection)
        size_t slots = 16;
        while (slots < 2 * found.size()) slots *= 2;
        std::vector<PyObject*> seen(slots, nullptr);
        for (const AdamEntry& e : found) {
            size_t at = (reinterpret_cast<uintptr_t>(e.state) >> 4) * 0x9e3779b97f4a7c15ull >> 32 & (slots - 1);
            while (seen[at] != nullptr && seen[at] != e.state) at = (at + 1) & (slots - 1);
            if (seen[at] == e.state) return none();
            seen[at] = e.state;
        }
        std::map<std::pair<int64_t, int>, std::unique_ptr<AdamBatch>> batches;
        for (AdamEntry& e : found) {
            auto& b = batches[{e.step + 1, e.p.device().index()}];
            if (!b) {
                b = std::make_unique<AdamBatch>();
                b->step = PyLong_FromLongLong(e.step + 1);
                if (b->step == nullptr) return nullptr;
                b->keep.reserve(4 * found.size());
                b->states.reserve(found.size());
                b->n.reserve(found.size());
                b->g.reserve(found.size());
                for (auto* list : {&b->p, &b->m, &b->v}) list->reserve(found.size());
            }
            Py_INCREF(e.state);
            b->states.push_back(e.state);
            b->p.push_back(ptr(e.p));
            b->g.push_back(ptr(e.g));
            b->m.push_back(ptr(e.m));
            b->v.push_back(ptr(e.v));
            b->n.push_back(e.p.numel());
            for (Tensor* t : {&e.p, &e.g, &e.m, &e.v}) b->keep.push_back(std::move(*t));
        }
        PyObject* out = PyList_New(0);
        for (auto& [key, b] : batches) {
            PyObject* capsule = PyCapsule_New(b.get(), kAdamCapsule, [](PyObject* c) { delete static_cast<AdamBatch*>(PyCapsule_GetPointer(c, kAdamCapsule)); });
            if (capsule == nullptr) { Py_DECREF(out); return nullptr; }
            b.release();
            PyObject* item = Py_BuildValue("(LN)", (long long)key.first, capsule);
            if (item == nullptr || PyList_Append(out, item) < 0) { Py_XDECREF(item); Py_DECREF(out); return nullptr; }
            Py_DECREF(item);
        }
        return out;
    });
}

// adam_apply(capsule, beta1, 1 - beta1, beta2, 1 - beta2, eps, decay, step_size)
PyObject* py_adam_apply(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
    PAMK_ARGS(8)
    return guarded([&]() -> PyObject* {
        auto* b = static_cast<AdamBatch*>(PyCapsule_GetPointer(a[0], kAdamCapsule));
        if (b == nullptr) return nullptr;
        double s[7];                    // (anything that converts: a learning rate may be a NumPy scalar or a tensor)
        for (int i = 0; i < 7; ++i) {
            s[i] = PyFloat_AsDouble(a[i + 1]);
            if (s[i] == -1.0 && PyErr_Occurred()) return nullptr;
        }
        {
            const Unlocked others_may_run;
            const Tensor& like = b->keep[0];
            c10::cuda::CUDAGuard guard(like.device());
            check(lib.pamk_adam_step(b->p.data(), b->g.data(), b->m.data(), b->v.data(), b->n.data(), (int)b->n.size(), (float)s[0], (float)s[1],
                                     (float)s[2], (float)s[3], (float)s[4], (float)s[5], (float)s[6], 1.0f, stream_of(like)),
                  "pamk_adam_step");
        }
        for (PyObject* st : b->states)
            if (PyDict_SetItem(st, step_key(), b->step) < 0) return nullptr;
        return none();
    });
}

PyObject* py_set_strict(PyObject*, PyObject* flag) {
    const int v = PyObject_IsTrue(flag);
    if (v < 0) return nullptr;
    g_strict.store(v != 0, std::memory_order_relaxed);
    return none();
}

PyObject* py_set_nvtx(PyObject*, PyObject* flag) {
    const int v = PyObject_IsTrue(flag);
    if (v < 0) return nullptr;
    g_nvtx.store(v != 0, std::memory_order_relaxed);
    return none();
}

// room_for(bytes, device index)
PyObject* py_room_for(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
    PAMK_ARGS(2)
    return guarded([&]() -> PyObject* {
        const size_t bytes = PyLong_AsSize_t(a[0]);
        if (bytes == (size_t)-1 && PyErr_Occurred()) return nullptr;
        const long device = PyLong_AsLong(a[1]);
        if (device == -1 && PyErr_Occurred()) return nullptr;
        return PyBool_FromLong(room_for(bytes, (c10::DeviceIndex)device));
    });
}

// setup(library path, error class)
PyObject* py_setup(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
    PAMK_ARGS(2)
    const char* path = PyUnicode_AsUTF8(a[0]);
    if (path == nullptr) return nullptr;
    void* h = dlopen(path, RTLD_NOW | RTLD_LOCAL);
    if (h == nullptr) {
        PyErr_Format(PyExc_RuntimeError, "cannot load %s: %s", path, dlerror());
        return nullptr;
    }
#define PAMK_BIND(name, to)                                                                  \
    to = reinterpret_cast<decltype(to)>(dlsym(h, #name));                                    \
    if (to == nullptr) {                                                                     \
        PyErr_Format(PyExc_RuntimeError, "%s does not export " #name, path);                 \
        return nullptr;                                                                      \
    }
#define PAMK_BIND_QUERY(name) PAMK_BIND(name, lib.name)
#define PAMK_BIND_LAUNCH(name) PAMK_BIND(name, lib.name.fn) lib.name.label = #name;
    PAMK_QUERIES(PAMK_BIND_QUERY)
    PAMK_LAUNCHES(PAMK_BIND_LAUNCH)
#undef PAMK_BIND_QUERY
#undef PAMK_BIND_LAUNCH
#undef PAMK_BIND
    Py_INCREF(a[1]);
    Py_XDECREF(g_kernel_error);
    g_kernel_error = a[1];
    return none();
}

#define PAMK_FAST(name, fn) {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(fn)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    PAMK_FAST("setup", py_setup),
    {"set_strict", py_set_strict, METH_O, nullptr},
    {"set_nvtx", py_set_nvtx, METH_O, nullptr},
    PAMK_FAST("room_for", py_room_for),
    PAMK_FAST("linear", py_linear),
    PAMK_FAST("matmul", py_matmul),
    PAMK_FAST("mul", py_elementwise<Ew::kMul>),
    PAMK_FAST("div", py_elementwise<Ew::kDiv>),
    PAMK_FAST("layer_norm", py_layer_norm),
    PAMK_FAST("softmax", py_softmax),
    PAMK_FAST("attention_qkv", py_attention_qkv),
    PAMK_FAST("attention_heads", py_attention_heads),
    PAMK_FAST("adam_collect", py_adam_collect),
    PAMK_FAST("adam_apply", py_adam_apply),
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", "Native host path of pam_b200's operators.", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host() { return PyModule_Create(&module); }
