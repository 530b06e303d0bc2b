// The operator API's path from torch tensors to libsparsedrop.so, in native code: argument checks, the casts under
// autocast, the mask draw, the launches and the autograd nodes of a SparseDrop linear, of the convolution
// and of the LayerNorm in front of them.
//
// A small layer is bound by the host: its four kernels take 31 us at 512^3 while the same sequence issued from Python
// (ctypes calls, a Python autograd.Function, tensor bookkeeping) took 197 us per forward + backward.  Everything between
// the Python entry points and the C ABI therefore runs here; the C-ABI library itself stays free of torch.
//
// Replaces the glue of flash_dropout/functional/blockwise_dropout_matmul_cuda.py:7-59 and
// flash_dropout/cuda/src/gemm_binding.cu:44-141.
#include <ATen/ATen.h>
#include <ATen/TensorSubclassLikeUtils.h>
#include <ATen/autocast_mode.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAException.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/python_cpp_function.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/autograd/variable.h>
#include <torch/csrc/utils/pybind.h>

#include <pybind11/stl.h>

#include <array>
#include <mutex>
#include <optional>
#include <unordered_map>
#include <vector>

#include "../../include/sparsedrop.h"

namespace py = pybind11;
using at::Tensor;
using torch::autograd::Node;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;

namespace {

constexpr int TILE = 128;
inline int64_t tiles_of(int64_t n) { return (n + TILE - 1) / TILE; }

// Raised as flash_dropout._lib.SparseDropError (a RuntimeError).
struct SdError : std::runtime_error {
    using std::runtime_error::runtime_error;
};
inline void check_rc(int rc) {
    if (rc != 0) throw SdError("libsparsedrop error " + std::to_string(rc) + ": " + sd_last_error());
}
[[noreturn]] inline void bad(const std::string& msg) { throw std::runtime_error(msg); }

// The Python error that is set (GIL held), as the exception that autograd's engine carries from its threads to the caller
// of backward() with its type; any other exception arrives there as a plain RuntimeError.
[[noreturn]] void throw_python() {
    python_error e;
    e.persist();
    throw std::move(e);
}
void set_python_error(const SdError& err) {
    static PyObject* type = py::module_::import("flash_dropout._lib").attr("SparseDropError").cast<py::object>().release().ptr();
    PyErr_SetString(type, err.what());
}
// The body of a node's apply().
template <class F>
variable_list backward_call(F&& body) {
    try {
        return body();
    } catch (const SdError& err) {
        py::gil_scoped_acquire gil;
        set_python_error(err);
        throw_python();
    }
}

// These nodes have no forward-mode derivative: a dual tensor is refused, as by a torch.autograd.Function without a jvp.
void no_forward_ad(const char* what, std::initializer_list<std::reference_wrapper<const Tensor>> inputs) {
    for (const Tensor& t : inputs)
        if (torch::autograd::isFwGradDefined(t))
            bad(std::string("Trying to use forward AD with ") + what + " that does not support it because it has not been implemented yet.");
}

int dtype_code(at::ScalarType t) {
    if (t == at::kHalf) return SD_F16;
    if (t == at::kBFloat16) return SD_BF16;
    throw SdError(std::string("operands must be half or bfloat16, got ") + c10::toString(t));
}

inline Tensor empty2(int64_t a, int64_t b, at::ScalarType t, const at::Device& d) {
    return at::detail::empty_cuda({a, b}, t, d, std::nullopt);
}
inline Tensor empty_bytes(int64_t n, const at::Device& d) { return at::detail::empty_cuda({n}, at::kByte, d, std::nullopt); }

// ---------------------------------------------------------------- per-device state
// The failure-detection words of a device, and the split-schedule workspaces of the streams that have launched products on it:
// launches that can overlap on the GPU must not share a workspace.  Live until the process exits.
//
// A CUDA graph has workspaces of its own: they come from its memory pool and are cleared by the graph itself, at every replay.
// Only the last capture's are held on to here, for as long as the capture asks for them; the pool keeps their memory with the
// graph.  One shared by the graphs captured on a stream would be cleared by the first of them only, and used by two replays
// at once on different streams.
struct Captured {
    unsigned long long id = 0;
    Tensor workspace;
};
struct DeviceState {
    Tensor status;
    std::unordered_map<cudaStream_t, Tensor> workspaces;
    std::unordered_map<cudaStream_t, Captured> captured;
};
std::mutex& state_mutex() { static auto* m = new std::mutex; return *m; }
std::unordered_map<int, DeviceState>& states() { static auto* s = new std::unordered_map<int, DeviceState>; return *s; }

// Which capture the stream is in; 0: none.
unsigned long long capture_of(cudaStream_t stream) {
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    unsigned long long id = 0;
    if (cudaStreamGetCaptureInfo(stream, &status, &id) != cudaSuccess) {
        (void)cudaGetLastError();
        return 0;
    }
    return status == cudaStreamCaptureStatusActive ? id : 0;
}

Tensor status_tensor(int dev) {
    std::lock_guard<std::mutex> lock(state_mutex());
    DeviceState& s = states()[dev];
    if (s.status.defined()) return s.status;
    const at::Device d(at::kCUDA, c10::DeviceIndex(dev));
    const auto ints = at::TensorOptions().dtype(at::kInt).device(d);
    if (!capture_of(c10::cuda::getCurrentCUDAStream(d.index()).stream())) {
        s.status = at::zeros({4}, ints);
        return s.status;
    }
    // The first launch of all is being captured.  The words outlive the graph, and must be zero before any replay of it.
    c10::cuda::CUDAGuard guard(d);
    c10::cuda::CUDAStreamCaptureModeGuard relaxed(cudaStreamCaptureModeRelaxed);
    void* p = nullptr;
    cudaStream_t own = nullptr;
    C10_CUDA_CHECK(cudaMalloc(&p, 4 * sizeof(int)));
    C10_CUDA_CHECK(cudaStreamCreateWithFlags(&own, cudaStreamNonBlocking));
    C10_CUDA_CHECK(cudaMemsetAsync(p, 0, 4 * sizeof(int), own));
    C10_CUDA_CHECK(cudaStreamSynchronize(own));
    C10_CUDA_CHECK(cudaStreamDestroy(own));
    s.status = at::from_blob(p, {4}, ints);
    return s.status;
}
Tensor workspace_tensor(int dev, cudaStream_t stream) {
    const unsigned long long capture = capture_of(stream);
    std::lock_guard<std::mutex> lock(state_mutex());
    DeviceState& s = states()[dev];
    Captured* c = capture ? &s.captured[stream] : nullptr;
    Tensor& ws = c ? c->workspace : s.workspaces[stream];
    if (!ws.defined() || (c && c->id != capture)) {
        const at::Device d(at::kCUDA, c10::DeviceIndex(dev));
        c10::cuda::CUDAGuard guard(d);
        Tensor t = empty_bytes(int64_t(sd_workspace_bytes()), d);
        check_rc(sd_workspace_init(t.data_ptr(), stream));
        ws = t;
        if (c) c->id = capture;
    }
    return ws;
}

// What every launch needs besides its operands.  The two pointers are looked up once per thread, device, stream and capture.
struct Launch {
    cudaStream_t stream;
    int* status;
    void* ws;
    explicit Launch(const at::Device& d) {
        struct Cached {
            int dev = -1;
            cudaStream_t stream = nullptr;
            unsigned long long capture = 0;
            int* status = nullptr;
            void* ws = nullptr;
        };
        static thread_local Cached c;
        stream = c10::cuda::getCurrentCUDAStream(d.index()).stream();
        const unsigned long long capture = capture_of(stream);
        if (c.dev != d.index() || c.stream != stream || c.capture != capture) {
            c.dev = -1;                            // (nothing is cached if one of the two throws)
            c.status = status_tensor(d.index()).data_ptr<int>();
            c.ws = workspace_tensor(d.index(), stream).data_ptr();
            c.dev = d.index();
            c.stream = stream;
            c.capture = capture;
        }
        status = c.status;
        ws = c.ws;
    }
};

struct Mat { void* p; int64_t rs, cs; };
inline Mat mat(const Tensor& t) { return {t.data_ptr(), t.stride(0), t.stride(1)}; }
inline Mat mat_t(const Tensor& t) { return {t.data_ptr(), t.stride(1), t.stride(0)}; }

// Row- or column-major with a TMA-compatible leading stride, else a contiguous copy.
Tensor operand(const Tensor& x) {
    if (reinterpret_cast<uintptr_t>(x.data_ptr()) % 16 == 0) {
        const int64_t r = x.size(0), c = x.size(1), sr = x.stride(0), sc = x.stride(1);
        if (sc == 1 && (sr % 8 == 0 || r == 1) && sr >= c) return x;
        if (sr == 1 && (sc % 8 == 0 || c == 1) && sc >= r) return x;
    }
    Tensor y = x.contiguous();
    // a contiguous view that starts off a 16-byte boundary is copied as well
    return reinterpret_cast<uintptr_t>(y.data_ptr()) % 16 == 0 ? y : y.clone();
}

// A saved tensor that came back for backward.  Hooks (torch.autograd.graph.saved_tensors_hooks) may return any tensor: the
// kernels take its memory as it is, so one of another type, device or shape is refused.  Its strides are the caller's matter.
Tensor came_back(Tensor t, at::IntArrayRef sizes, at::ScalarType type, const at::Device& dev) {
    if (t.scalar_type() != type || t.device() != dev || t.sizes() != sizes || t.layout() != at::kStrided)
        bad("a saved tensor came back from its hooks with another type, device or shape");
    return t;
}
Tensor dense16(const Tensor& t) {                  // contiguous, on a 16-byte boundary
    const Tensor c = t.contiguous();
    return reinterpret_cast<uintptr_t>(c.data_ptr()) % 16 ? c.clone() : c;
}

// ---------------------------------------------------------------- block plans
// How the mask of one call comes about: a plan that exists, or a draw from (seed, offset), the offset optionally
// advanced by a counter in device memory.
struct Draw {
    uint64_t seed = 0, offset = 0;
    uint64_t* counter = nullptr;
    int rep_r = 1, rep_c = 1;
    float p = 0;
};
Tensor draw_plan(const Draw& d, int64_t M, int64_t K, const at::Device& dev, cudaStream_t stream) {
    const int R = int(tiles_of(M)), C = int(tiles_of(K));
    Tensor buf = empty_bytes(int64_t(sd_plan_bytes(R, C)), dev);
    if (d.counter)
        check_rc(sd_plan_from_seed_counter(buf.data_ptr(), R, C, d.rep_r, d.rep_c, d.seed, d.offset, d.counter, d.p, nullptr, stream));
    else
        check_rc(sd_plan_from_seed(buf.data_ptr(), R, C, d.rep_r, d.rep_c, d.seed, d.offset, d.p, nullptr, stream));
    return buf;
}

void check_plan_device(const std::optional<Tensor>& plan, const at::Device& dev) {
    if (plan && plan->defined() && plan->device() != dev) bad("the plan must be on the device of the operands");
}

// ---------------------------------------------------------------- casts under autocast
inline bool flat_f32(const Tensor& t) {
    return t.scalar_type() == at::kFloat && t.is_contiguous() && reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0;
}

// 16-bit copies of a and, if given, b: one launch where both are contiguous fp32.
void cast_pair(const Tensor& a, Tensor& a16, const Tensor& b, Tensor& b16, at::ScalarType dt, cudaStream_t stream) {
    const bool fa = a.defined() && flat_f32(a), fb = b.defined() && flat_f32(b);
    if (a.defined()) a16 = fa ? Tensor(at::detail::empty_cuda(a.sizes(), dt, a.device(), std::nullopt)) : a.to(dt);
    if (b.defined()) b16 = fb ? Tensor(at::detail::empty_cuda(b.sizes(), dt, b.device(), std::nullopt)) : b.to(dt);
    if (fa || fb)
        check_rc(sd_cast16(fa ? a.data_ptr<float>() : nullptr, fa ? a16.data_ptr() : nullptr, fa ? a.numel() : 0,
                           fb ? b.data_ptr<float>() : nullptr, fb ? b16.data_ptr() : nullptr, fb ? b.numel() : 0,
                           dtype_code(dt), stream));
}

// ---------------------------------------------------------------- a SparseDrop linear
struct PyCallback {
    PyObject* f;
    explicit PyCallback(PyObject* f_) : f(f_) { Py_INCREF(f); }
    PyCallback(const PyCallback&) = delete;
    ~PyCallback() {
        if (Py_IsInitialized()) {
            py::gil_scoped_acquire gil;
            Py_DECREF(f);
        }
    }
    void operator()() const {
        py::gil_scoped_acquire gil;
        PyObject* r = PyObject_CallNoArgs(f);
        if (!r) throw_python();
        Py_DECREF(r);
    }
};

struct Options {
    bool relu = false, input_relu = false, premasked = false;
    Tensor wgrad;                                  // [out, in], fp32 or the operands' type: takes the weight gradient
    bool wgrad_acc = false;
    std::shared_ptr<PyCallback> notify;
};

struct SparseDropLinearBackward : public Node {
    SavedVariable x, w, y;                         // 16-bit operands of the forward product; y: its ReLU'd result
    Tensor plan;                                   // undefined: drawn again from `draw` (recompute_plan)
    Draw draw;
    int64_t block_m = 0, block_k = 0;
    bool pair_block = false;
    int64_t M = 0, K = 0, N = 0;
    at::ScalarType type = at::kHalf;               // of the saved tensors
    at::Device dev = at::Device(at::kCUDA, 0);
    std::vector<int64_t> lead;                     // shape of an input that is not 2-D
    double p = 0, draw_p = 0;                      // of the scale, and of the draw
    bool x_f32 = false, w_f32 = false;             // the layer's own tensors are fp32: their gradients leave in fp32
    Options opt;

    std::string name() const override { return "SparseDropLinearBackward"; }
    void release_variables() override {
        x.reset_data();
        w.reset_data();
        y.reset_data();
    }
    variable_list apply(variable_list&& grads) override;
    variable_list gradients(variable_list&& grads);
};

variable_list SparseDropLinearBackward::apply(variable_list&& grads) { return backward_call([&] { return gradients(std::move(grads)); }); }
variable_list SparseDropLinearBackward::gradients(variable_list&& grads) {
    at::NoGradGuard no_grad;
    c10::cuda::OptionalCUDAGuard guard(dev);
    Tensor x16 = x.unpack();
    x16 = x16.dim() == 2 ? came_back(x16, {M, K}, type, dev) : came_back(x16, lead, type, dev).reshape({M, K});
    x16 = operand(x16);
    const Tensor w16 = operand(came_back(w.unpack(), {N, K}, type, dev));
    if (opt.input_relu && x16.stride(1) != 1) x16 = dense16(x16);
    const Launch L(dev);
    const float scale = float(1.0 / (1.0 - p));
    const int dt = dtype_code(type);
    const Tensor pl = plan.defined() ? plan : draw_plan(draw, M, K, dev, L.stream);
    Tensor dy = grads[0].defined() ? grads[0] : at::zeros({M, N}, x16.options());     // (any rank: only the element count matters)
    if (dy.scalar_type() != x16.scalar_type()) dy = dy.to(x16.scalar_type());
    if (opt.relu && !opt.premasked) dy = at::threshold_backward(dy, came_back(y.unpack(shared_from_this()), dy.sizes(), type, dev), 0);
    dy = operand(dy.dim() == 2 ? dy : dy.reshape({M, N}));
    const Mat mdy = mat(dy), mx = mat(x16), mdyt = mat_t(dy), mxt = mat_t(x16), mwt = mat_t(w16);
    Tensor dx, dw;
    if (task_should_compute_output(0)) {
        // dx (M, K) = keep o (dy (M, N) . W (N, K)) * scale
        const at::ScalarType t = x_f32 ? at::kFloat : x16.scalar_type();
        dx = lead.empty() ? empty2(M, K, t, dev) : Tensor(at::detail::empty_cuda(lead, t, dev, std::nullopt));
        void* mask = opt.input_relu ? mx.p : nullptr;
        if (x_f32)
            check_rc(sd_gemm_sdd_f32(mdy.p, mdy.rs, mdy.cs, mwt.p, mwt.rs, mwt.cs, dx.data_ptr<float>(), K, 1, int(M), int(K), int(N),
                                     pl.data_ptr(), mask, mx.rs, scale, dt, L.ws, L.status, L.stream));
        else if (mask)
            check_rc(sd_gemm_sdd_relu_mask(mdy.p, mdy.rs, mdy.cs, mwt.p, mwt.rs, mwt.cs, dx.data_ptr(), K, 1, int(M), int(K), int(N),
                                           pl.data_ptr(), mask, mx.rs, scale, dt, L.ws, L.status, L.stream));
        else
            check_rc(sd_gemm_sdd(mdy.p, mdy.rs, mdy.cs, mwt.p, mwt.rs, mwt.cs, dx.data_ptr(), K, 1, int(M), int(K), int(N),
                                 pl.data_ptr(), scale, dt, L.ws, L.status, L.stream));
    }
    // dW^T (K, N) = (keep o x)^T (K, M) . dy (M, N) * scale, stored straight into dW (N, K)
    Tensor target = opt.wgrad;
    if (!target.defined() && task_should_compute_output(1)) target = dw = empty2(N, K, w_f32 ? at::kFloat : type, dev);
    if (target.defined()) {
        const Mat out = mat_t(target);
        if (target.scalar_type() == at::kFloat)
            check_rc(sd_gemm_dsd_f32(mxt.p, mxt.rs, mxt.cs, mdyt.p, mdyt.rs, mdyt.cs, static_cast<float*>(out.p), out.rs, out.cs, int(K),
                                     int(N), int(M), pl.data_ptr(), SD_PLAN_COLS, scale, dt, int(opt.wgrad.defined() && opt.wgrad_acc),
                                     L.ws, L.status, L.stream));
        else
            check_rc(sd_gemm_dsd(mxt.p, mxt.rs, mxt.cs, mdyt.p, mdyt.rs, mdyt.cs, out.p, out.rs, out.cs, int(K), int(N), int(M),
                                 pl.data_ptr(), SD_PLAN_COLS, scale, dt, L.ws, L.status, L.stream));
    }
    if (opt.wgrad.defined() && opt.notify) (*opt.notify)();
    return {dx, dw};
}

// y = (keep o input) . weight^T / (1 - p) of 2-D CUDA tensors, see blockwise_dropout_matmul in
// functional/blockwise_dropout_matmul_cuda.py for the meaning of the arguments.  `plan` with its grid, or none: drawn from
// (seed, offset) and the optional device counter with blocks of rep_r x rep_c tiles at draw_p.  `recompute`: what it is drawn
// from is all that is kept for backward.  `p` is the scale's.
Tensor linear(const Tensor& input_, const Tensor& weight_, const std::optional<Tensor>& plan_, int64_t plan_R, int64_t plan_C,
              int64_t rep_r, int64_t rep_c, bool pair_block, double p, uint64_t seed, uint64_t offset,
              const std::optional<Tensor>& counter, bool relu, bool input_relu, bool premasked,
              const std::optional<Tensor>& wgrad, bool wgrad_acc, py::handle notify, bool recompute,
              const std::optional<Tensor>& weight_lowp, bool any_rank, double draw_p) {
    Options opt;
    opt.relu = relu;
    opt.input_relu = input_relu;
    opt.premasked = premasked;
    if (wgrad && wgrad->defined()) {
        opt.wgrad = *wgrad;
        opt.wgrad_acc = wgrad_acc;
        if (!notify.is_none()) opt.notify = std::make_shared<PyCallback>(notify.ptr());
    }
    py::gil_scoped_release no_gil;
    if (!input_.is_cuda() || !weight_.is_cuda()) bad("input and weight must be CUDA");   // no CPU path, as gemm_binding.cu:19
    if ((any_rank ? input_.dim() < 1 : input_.dim() != 2) || weight_.dim() != 2) bad("input and weight must be 2D");
    if (input_.device() != weight_.device()) bad("A and B must be on the same device");
    no_forward_ad("SparseDropLinear", {input_, weight_});
    const at::Device dev = input_.device();
    const bool amp = at::autocast::is_autocast_enabled(at::kCUDA);
    const at::ScalarType amp_t = amp ? at::autocast::get_autocast_dtype(at::kCUDA) : at::kFloat;
    const bool lowp =
        amp && weight_lowp && opt.wgrad.defined() && weight_lowp->scalar_type() == amp_t && weight_lowp->sizes() == weight_.sizes();
    if (lowp && weight_lowp->device() != dev) bad("A and B must be on the same device");
    check_plan_device(plan_, dev);
    c10::cuda::OptionalCUDAGuard guard(dev);
    const Launch L(dev);

    // operands in 16 bits; fp32 ones are cast here, outside autograd, and their gradients leave in fp32
    Tensor input = input_, weight = weight_, x16, w16;
    if (amp) {
        const at::ScalarType dt = amp_t;
        if (input.scalar_type() != dt && input.scalar_type() != at::kFloat) input = input.to(dt);
        if (!lowp && weight.scalar_type() != dt && weight.scalar_type() != at::kFloat) weight = weight.to(dt);
        at::NoGradGuard no_grad;
        const bool cast_x = input.scalar_type() != dt, cast_w = !lowp && weight.scalar_type() != dt;
        x16 = input;
        w16 = lowp ? *weight_lowp : weight;
        // Every call casts for itself: a copy kept from an earlier call could not be known to be current, as a CUDA graph's
        // replay rewrites tensors without a sign that the host could see, and a copy made during a capture holds nothing yet.
        if (cast_x || cast_w) cast_pair(cast_x ? input : Tensor(), x16, cast_w ? weight : Tensor(), w16, dt, L.stream);
    } else {
        x16 = input;
        w16 = weight;
    }
    if (x16.scalar_type() != w16.scalar_type())
        bad(std::string("input (") + c10::toString(x16.scalar_type()) + ") and weight (" + c10::toString(w16.scalar_type()) +
            ") must have the same dtype");
    const int dt = dtype_code(x16.scalar_type());
    const int64_t K = x16.size(-1), M = K ? x16.numel() / K : 0, N = w16.size(0);
    if (K % 8 || N % 8) bad("in_features and out_features must be multiples of 8 (16-byte TMA rows)");
    if (w16.size(1) != K)
        bad("reduction dimensions differ: A is (" + std::to_string(M) + ", " + std::to_string(K) + "), B is (" + std::to_string(N) +
            ", " + std::to_string(w16.size(1)) + ")");
    if (opt.wgrad.defined()) {
        const Tensor& t = opt.wgrad;
        if (t.dim() != 2 || t.size(0) != N || t.size(1) != K || t.device() != dev || !(t.stride(0) == 1 || t.stride(1) == 1) ||
            (t.scalar_type() != at::kFloat && t.scalar_type() != x16.scalar_type()))
            bad("out has the wrong shape, dtype, device or strides");
        if (opt.wgrad_acc && t.scalar_type() != at::kFloat) bad("accumulate needs an fp32 out");
    }
    const bool needs_grad = torch::autograd::compute_requires_grad(input, weight);
    Tensor xs, ws, out, plan;
    Draw d;
    {
        at::NoGradGuard no_grad;
        // leading dimensions are rows: no view goes through autograd for them
        xs = operand(x16.dim() == 2 ? x16 : x16.reshape({M, K}));
        ws = operand(w16);
        if (input_relu && xs.stride(1) != 1) xs = xs.contiguous();
        if (plan_ && plan_->defined()) {
            if (plan_R != tiles_of(M) || plan_C != tiles_of(K))
                bad("plan grid (" + std::to_string(plan_R) + ", " + std::to_string(plan_C) + ") does not match operand A (" +
                    std::to_string(M) + ", " + std::to_string(K) + ")");
            plan = *plan_;
        }
        d.seed = seed;
        d.offset = offset;
        d.counter = counter && counter->defined() ? static_cast<uint64_t*>(counter->data_ptr()) : nullptr;
        d.rep_r = int(rep_r);
        d.rep_c = int(rep_c);
        d.p = float(draw_p);
        if (!plan.defined()) plan = draw_plan(d, M, K, dev, L.stream);
        if (input.dim() == 2)
            out = empty2(M, N, xs.scalar_type(), dev);
        else {
            std::vector<int64_t> shape = input.sizes().vec();
            shape.back() = N;
            out = at::detail::empty_cuda(shape, xs.scalar_type(), dev, std::nullopt);
        }
        const Mat a = mat(xs), b = mat(ws);
        check_rc((relu ? sd_gemm_dsd_relu : sd_gemm_dsd)(a.p, a.rs, a.cs, b.p, b.rs, b.cs, out.data_ptr(), N, 1, int(M), int(N), int(K),
                                                         plan.data_ptr(), SD_PLAN_ROWS, float(1.0 / (1.0 - p)), dt, L.ws, L.status,
                                                         L.stream));
    }
    if (!needs_grad) return out;
    std::shared_ptr<SparseDropLinearBackward> node(new SparseDropLinearBackward(), torch::autograd::deleteNode);
    node->set_next_edges(torch::autograd::collect_next_edges(input, weight));
    // an input that went to the kernel as it is (possibly as a 2-D view of itself) is saved as the variable it is
    const bool own = x16.is_same(input) && xs.data_ptr() == input.data_ptr() && (input.dim() == 2 ? xs.is_same(x16) : input.is_contiguous());
    node->x = SavedVariable(own ? input : xs, false);
    node->w = SavedVariable(ws.is_same(w16) && w16.is_same(weight) ? weight : ws, false);
    node->draw = d;
    node->block_m = rep_r * TILE;
    node->block_k = rep_c * TILE;
    node->pair_block = pair_block;
    node->draw_p = draw_p;
    if (!recompute || d.counter) node->plan = plan;
    node->M = M;
    node->K = K;
    node->N = N;
    node->type = xs.scalar_type();
    node->dev = dev;
    node->p = p;
    if (input.dim() != 2) node->lead = input.sizes().vec();
    node->x_f32 = input.scalar_type() == at::kFloat;
    node->w_f32 = weight.scalar_type() == at::kFloat;
    node->opt = std::move(opt);
    torch::autograd::set_history(out, node);
    if (relu && !premasked) node->y = SavedVariable(out, true);
    return out;
}

// Python attributes of the node: the mask it holds (`plan`: the plan buffer, or None when it is drawn again in backward)
// and what it is drawn from (`origin`: rows, columns, block size, p, seed, offset).
SparseDropLinearBackward* node_of(PyObject* self) {
    return static_cast<SparseDropLinearBackward*>(reinterpret_cast<torch::autograd::THPCppFunction*>(self)->cdata.get());
}
PyObject* get_plan(PyObject* self, void*) {
    const auto* n = node_of(self);
    if (!n->plan.defined()) Py_RETURN_NONE;
    return THPVariable_Wrap(n->plan);
}
PyObject* get_origin(PyObject* self, void*) {
    const auto* n = node_of(self);
    if (n->plan.defined()) Py_RETURN_NONE;
    py::object block = n->pair_block ? py::object(py::make_tuple(n->block_m, n->block_k)) : py::object(py::int_(n->block_m));
    return py::make_tuple(n->M, n->K, block, n->draw_p, n->draw.seed, n->draw.offset).release().ptr();
}
void register_node() {
    using namespace torch::autograd;
    static PyGetSetDef properties[] = {THP_FUNCTION_DEFAULT_PROPERTIES,
                                       {(char*)"plan", get_plan, nullptr, nullptr, nullptr},
                                       {(char*)"origin", get_origin, nullptr, nullptr, nullptr},
                                       {nullptr}};
    static PyTypeObject type;
    _initFunctionPyTypeObject(type, "SparseDropLinearBackward", properties, nullptr);
    Py_INCREF(&type);
    registerCppFunction(typeid(SparseDropLinearBackward), &type);
}

// ---------------------------------------------------------------- the extension-style products
std::string shape_text(int64_t a, int64_t b) { return "(" + std::to_string(a) + ", " + std::to_string(b) + ")"; }
void check_operand(const Tensor& x, const char* name) {      // flash_dropout/cuda/src/gemm_binding.cu:18-22
    if (!x.is_cuda()) bad(std::string(name) + " must be CUDA");
    if (x.dim() != 2) bad(std::string(name) + " must be 2D");
    if (!(x.stride(0) == 1 || x.stride(1) == 1)) bad(std::string(name) + " must be row or column major");
}
int check_pair(const Tensor& A, const Tensor& B) {
    check_operand(A, "A");
    check_operand(B, "B");
    if (A.scalar_type() != B.scalar_type()) bad("A and B must have the same dtype");
    if (A.size(1) != B.size(1))
        bad("reduction dimensions differ: A is " + shape_text(A.size(0), A.size(1)) + ", B is " + shape_text(B.size(0), B.size(1)));
    if (A.device() != B.device()) bad("A and B must be on the same device");
    return dtype_code(A.scalar_type());
}
void check_mask_device(const Tensor& mask, const Tensor& A) {
    if (mask.is_cuda() && mask.device() != A.device()) bad("Mask must be on the operands' device");
}
Tensor plan_from_mask(const Tensor& mask, int64_t rows, int64_t cols, int64_t rep_r, int64_t rep_c, cudaStream_t stream) {
    if (mask.scalar_type() != at::kBool) bad("Mask must be bool");
    if (!mask.is_cuda() || mask.dim() != 2) bad("Mask must be a 2D CUDA tensor");
    const int64_t R = tiles_of(rows), C = tiles_of(cols), wr = (R + rep_r - 1) / rep_r, wc = (C + rep_c - 1) / rep_c;
    if (mask.size(0) != wr || mask.size(1) != wc)
        bad("mask shape " + shape_text(mask.size(0), mask.size(1)) + " does not match " + shape_text(wr, wc) + " blocks of " +
            shape_text(rep_r * TILE, rep_c * TILE));
    Tensor buf = empty_bytes(int64_t(sd_plan_bytes(int(R), int(C))), mask.device());
    check_rc(sd_plan_from_mask(buf.data_ptr(), int(R), int(C), int(rep_r), int(rep_c), static_cast<const uint8_t*>(mask.data_ptr()),
                               mask.stride(0), mask.stride(1), stream));
    return buf;
}

Tensor gemm_dense(const Tensor& A, const Tensor& B) {
    py::gil_scoped_release no_gil;
    at::NoGradGuard no_grad;
    const int dt = check_pair(A, B);
    c10::cuda::OptionalCUDAGuard guard(A.device());
    const Launch L(A.device());
    Tensor C = empty2(A.size(0), B.size(0), A.scalar_type(), A.device());
    const Mat a = mat(A), b = mat(B);
    check_rc(sd_gemm(a.p, a.rs, a.cs, b.p, b.rs, b.cs, C.data_ptr(), C.size(1), 1, int(A.size(0)), int(B.size(0)), int(A.size(1)), 1.0f,
                     dt, L.ws, L.status, L.stream));
    return C;
}
Tensor gemm_dsd(const Tensor& A, const Tensor& B, const Tensor& mask, int64_t rep_r, int64_t rep_c, double scale) {
    py::gil_scoped_release no_gil;
    at::NoGradGuard no_grad;
    check_operand(A, "A");
    check_mask_device(mask, A);
    c10::cuda::OptionalCUDAGuard guard(A.device());
    const Launch L(A.device());
    const Tensor plan = plan_from_mask(mask, A.size(0), A.size(1), rep_r, rep_c, L.stream);
    const int dt = check_pair(A, B);
    Tensor C = empty2(A.size(0), B.size(0), A.scalar_type(), A.device());
    const Mat a = mat(A), b = mat(B);
    check_rc(sd_gemm_dsd(a.p, a.rs, a.cs, b.p, b.rs, b.cs, C.data_ptr(), C.size(1), 1, int(A.size(0)), int(B.size(0)), int(A.size(1)),
                         plan.data_ptr(), SD_PLAN_ROWS, float(scale), dt, L.ws, L.status, L.stream));
    return C;
}
Tensor gemm_sdd(const Tensor& A, const Tensor& B, const Tensor& mask, int64_t rep_r, int64_t rep_c, double scale) {
    py::gil_scoped_release no_gil;
    at::NoGradGuard no_grad;
    check_operand(A, "A");
    check_operand(B, "B");
    check_mask_device(mask, A);
    c10::cuda::OptionalCUDAGuard guard(A.device());
    const Launch L(A.device());
    const Tensor plan = plan_from_mask(mask, A.size(0), B.size(0), rep_r, rep_c, L.stream);
    const int dt = check_pair(A, B);
    Tensor C = empty2(A.size(0), B.size(0), A.scalar_type(), A.device());
    const Mat a = mat(A), b = mat(B);
    check_rc(sd_gemm_sdd(a.p, a.rs, a.cs, b.p, b.rs, b.cs, C.data_ptr(), C.size(1), 1, int(A.size(0)), int(B.size(0)), int(A.size(1)),
                         plan.data_ptr(), float(scale), dt, L.ws, L.status, L.stream));
    return C;
}

// ---------------------------------------------------------------- a SparseDrop convolution
// Blockwise dropout on the im2col matrix (M = N*P*Q rows, K = C*R*S columns in unfold order); see
// functional/blockwise_dropout_conv2d.py for the stages and the semantics.
struct ConvGeometry {
    int N, C, H, W, R, S, ph, pw, sh, sw, dh, dw, P, Q, Ko;
    int M, K, Kg, Kog;                             // Kg, Kog: K and Ko rounded up to what the kernels take
};
#define SD_CONV_GEOM(g) g.N, g.C, g.H, g.W, g.R, g.S, g.ph, g.pw, g.sh, g.sw, g.dh, g.dw

Tensor im2col_panels(const Tensor& x, const ConvGeometry& g, const Tensor& plan, cudaStream_t stream) {
    Tensor col = at::detail::empty_cuda({tiles_of(g.M), g.Kg, TILE}, x.scalar_type(), x.device(), std::nullopt);
    if (g.Kg > g.K) col.slice(1, g.K).zero_();
    check_rc(sd_im2col_kept_panels(x.data_ptr(), SD_CONV_GEOM(g), col.data_ptr(), g.Kg, plan.data_ptr(), stream));
    return col;
}

struct SparseDropConv2dBackward : public Node {
    SavedVariable x, w2d, cols;
    Tensor plan;
    ConvGeometry g;
    at::ScalarType t = at::kHalf;                  // of the saved tensors
    at::Device dev = at::Device(at::kCUDA, 0);
    double p = 0;
    bool fused = false, has_cols = false, x_f32 = false, w_f32 = false;

    std::string name() const override { return "SparseDropConv2dBackward"; }
    void release_variables() override {
        x.reset_data();
        w2d.reset_data();
        cols.reset_data();
    }
    variable_list apply(variable_list&& grads) override { return backward_call([&] { return gradients(std::move(grads)); }); }
    variable_list gradients(variable_list&& grads) {
        at::NoGradGuard no_grad;
        c10::cuda::OptionalCUDAGuard guard(dev);
        const Tensor x16 = dense16(came_back(x.unpack(), {g.N, g.C, g.H, g.W}, t, dev));
        const Tensor w = operand(came_back(w2d.unpack(), {g.Kog, g.Kg}, t, dev));
        const Launch L(dev);
        const int dt = dtype_code(t);
        const float scale = float(1.0 / (1.0 - p));
        Tensor dy = grads[0].defined() ? grads[0] : at::zeros({g.N, g.Ko, g.P, g.Q}, x16.options());
        if (dy.scalar_type() != t) dy = dy.to(t);
        dy = dy.permute({0, 2, 3, 1}).reshape({g.M, g.Ko});          // free for channels-last gradients
        if (g.Kog != g.Ko) dy = at::constant_pad_nd(dy, {0, g.Kog - g.Ko});
        dy = dy.contiguous();
        if (reinterpret_cast<uintptr_t>(dy.data_ptr()) % 16) dy = dy.clone();
        const Mat mdy = mat(dy);
        Tensor dx, dwt;
        if (task_should_compute_output(1)) {
            Tensor dw = empty2(g.Kog, g.Kg, t, dev);
            if (fused)
                check_rc(sd_conv_dsd_dw(x16.data_ptr(), SD_CONV_GEOM(g), mdy.p, mdy.rs, mdy.cs, dw.data_ptr(), g.Kg, 1, g.Kog,
                                        plan.data_ptr(), scale, dt, L.ws, L.status, L.stream));
            else {
                const Tensor col = has_cols ? dense16(came_back(cols.unpack(), {tiles_of(g.M), g.Kg, TILE}, t, dev))
                                            : im2col_panels(x16, g, plan, L.stream);
                check_rc(sd_gemm_dsd_panels(col.data_ptr(), g.M, g.Kg, mdy.p, mdy.cs, mdy.rs, dw.data_ptr(), 1, g.Kg, g.Kog,
                                            plan.data_ptr(), SD_PLAN_COLS, scale, dt, L.ws, L.status, L.stream));
            }
            if (g.Kog != g.Ko || g.Kg != g.K) dw = dw.slice(0, 0, g.Ko).slice(1, 0, g.K);
            if (w_f32) dw = dw.to(at::kFloat);
            dwt = dw.reshape({g.Ko, g.C, g.R, g.S});
        }
        if (task_should_compute_output(0)) {
            // kept blocks of dcolP = W2d^T . dY^T, then the adjoint gather
            Tensor dcol = at::detail::empty_cuda({tiles_of(g.M), g.Kg, TILE}, t, dev, std::nullopt);
            const Mat mwt = mat_t(w);
            check_rc(sd_gemm_sdd_kept_t_panels(mwt.p, mwt.rs, mwt.cs, mdy.p, mdy.rs, mdy.cs, dcol.data_ptr(), g.Kg, g.M, g.Kog,
                                               plan.data_ptr(), scale, dt, L.ws, L.status, L.stream));
            dx = at::detail::empty_cuda({g.N, g.C, g.H, g.W}, x_f32 ? at::kFloat : t, dev, std::nullopt);
            if (x_f32)
                check_rc(sd_col2im_kept_panels_f32(dcol.data_ptr(), g.Kg, SD_CONV_GEOM(g), dx.data_ptr<float>(), plan.data_ptr(), dt, L.stream));
            else
                check_rc(sd_col2im_kept_panels(dcol.data_ptr(), g.Kg, SD_CONV_GEOM(g), dx.data_ptr(), plan.data_ptr(), dt, L.stream));
        }
        return {dx, dwt};
    }
};

Tensor conv2d(const Tensor& input_, const Tensor& kernel_, const std::optional<Tensor>& plan_, int64_t plan_R, int64_t plan_C,
              int64_t rep_r, int64_t rep_c, double p, uint64_t seed, uint64_t offset, const std::optional<Tensor>& counter,
              std::array<int64_t, 2> padding, std::array<int64_t, 2> stride, std::array<int64_t, 2> dilation, bool recompute_cols,
              bool want_fused) {
    py::gil_scoped_release no_gil;
    if (!input_.is_cuda() || !kernel_.is_cuda()) bad("input and kernel must be CUDA");
    if (input_.device() != kernel_.device()) bad("input and kernel must be on the same device");
    check_plan_device(plan_, input_.device());
    no_forward_ad("SparseDropConv2d", {input_, kernel_});
    const Tensor &input = input_, &kernel = kernel_;
    const bool amp = at::autocast::is_autocast_enabled(at::kCUDA);
    const at::ScalarType t = amp ? at::autocast::get_autocast_dtype(at::kCUDA) : input.scalar_type();
    if (!amp && input.scalar_type() != kernel.scalar_type())
        bad(std::string("input (") + c10::toString(input.scalar_type()) + ") and kernel (" + c10::toString(kernel.scalar_type()) +
            ") must have the same dtype");
    const int dt = dtype_code(t);
    if (input.dim() != 4 || kernel.dim() != 4) bad("input must be NCHW and kernel [out, in, R, S]");
    ConvGeometry g;
    g.N = int(input.size(0)); g.C = int(input.size(1)); g.H = int(input.size(2)); g.W = int(input.size(3));
    g.Ko = int(kernel.size(0)); g.R = int(kernel.size(2)); g.S = int(kernel.size(3));
    if (kernel.size(1) != g.C) bad("kernel expects " + std::to_string(kernel.size(1)) + " input channels, input has " + std::to_string(g.C));
    g.ph = int(padding[0]); g.pw = int(padding[1]); g.sh = int(stride[0]); g.sw = int(stride[1]); g.dh = int(dilation[0]); g.dw = int(dilation[1]);
    if (g.sh <= 0 || g.sw <= 0 || g.dh <= 0 || g.dw <= 0) bad("stride and dilation must be positive");
    // rows and columns that the filter can move over; negative: it is larger than the padded input
    const int64_t over_h = int64_t(g.H) + 2 * int64_t(g.ph) - int64_t(g.dh) * (g.R - 1) - 1;
    const int64_t over_w = int64_t(g.W) + 2 * int64_t(g.pw) - int64_t(g.dw) * (g.S - 1) - 1;
    if (over_h < 0 || over_w < 0) bad("the filter does not fit the padded input");
    g.P = int(over_h / g.sh + 1);
    g.Q = int(over_w / g.sw + 1);
    const int64_t M = int64_t(g.N) * g.P * g.Q, K = int64_t(g.C) * g.R * g.S;
    if (M > (1ll << 30) || K > (1ll << 30)) bad("the im2col matrix is too large");
    g.M = int(M);
    g.K = int(K);
    g.Kg = (g.K + 63) & ~63;                        // the im2col matrix is kept in panels: k extent a multiple of 64
    g.Kog = (g.Ko + 7) & ~7;
    const at::Device dev = input.device();
    c10::cuda::OptionalCUDAGuard guard(dev);
    const Launch L(dev);
    Tensor plan, x16, w2d, y2d, cols;
    bool fused;
    {
        at::NoGradGuard no_grad;
        if (plan_ && plan_->defined()) {
            if (plan_R != tiles_of(g.M) || plan_C != tiles_of(g.Kg))
                bad("plan grid (" + std::to_string(plan_R) + ", " + std::to_string(plan_C) + ") does not match the " + std::to_string(g.M) +
                    " x " + std::to_string(g.Kg) + " im2col matrix");
            plan = *plan_;
        } else {
            Draw d;
            d.seed = seed;
            d.offset = offset;
            d.counter = counter && counter->defined() ? static_cast<uint64_t*>(counter->data_ptr()) : nullptr;
            d.rep_r = int(rep_r);
            d.rep_c = int(rep_c);
            d.p = float(p);
            plan = draw_plan(d, g.M, g.Kg, dev, L.stream);
        }
        // 16-byte rows for TMA; zero padding changes nothing
        const bool pad_w2d = g.Kg != g.K || g.Kog != g.Ko, cast_x = input.scalar_type() != t, cast_w = kernel.scalar_type() != t;
        x16 = input;
        Tensor kflat = kernel.reshape({g.Ko, g.K}), k16 = kflat;
        if (cast_x || (cast_w && !pad_w2d)) cast_pair(cast_x ? input : Tensor(), x16, cast_w && !pad_w2d ? kflat : Tensor(), k16, t, L.stream);
        if (pad_w2d) {
            w2d = at::zeros({g.Kog, g.Kg}, kernel.options().dtype(t));
            w2d.slice(0, 0, g.Ko).slice(1, 0, g.K).copy_(kflat);
        } else
            w2d = k16.contiguous();
        x16 = x16.contiguous();
        if (reinterpret_cast<uintptr_t>(x16.data_ptr()) % 16) x16 = x16.clone();
        if (reinterpret_cast<uintptr_t>(w2d.data_ptr()) % 16) w2d = w2d.clone();
        y2d = empty2(g.M, g.Kog, t, dev);
        const Mat mw = mat(w2d);
        const float scale = float(1.0 / (1.0 - p));
        fused = want_fused && sd_conv_fused_supported(SD_CONV_GEOM(g));
        if (fused)
            check_rc(sd_conv_dsd_fwd(x16.data_ptr(), SD_CONV_GEOM(g), mw.p, mw.rs, mw.cs, y2d.data_ptr(), g.Kog, 1, g.Kog, plan.data_ptr(),
                                     scale, dt, L.ws, L.status, L.stream));
        else {
            cols = im2col_panels(x16, g, plan, L.stream);
            check_rc(sd_gemm_dsd_panels(cols.data_ptr(), g.M, g.Kg, mw.p, mw.rs, mw.cs, y2d.data_ptr(), g.Kog, 1, g.Kog, plan.data_ptr(),
                                        SD_PLAN_ROWS, scale, dt, L.ws, L.status, L.stream));
        }
    }
    // an NCHW-shaped view of y2d with channels-last strides
    Tensor out;
    {
        at::AutoDispatchBelowADInplaceOrView below;
        out = y2d.as_strided({g.N, g.Ko, g.P, g.Q}, {int64_t(g.P) * g.Q * g.Kog, 1, int64_t(g.Q) * g.Kog, g.Kog});
    }
    if (!torch::autograd::compute_requires_grad(input, kernel)) return out;
    std::shared_ptr<SparseDropConv2dBackward> node(new SparseDropConv2dBackward(), torch::autograd::deleteNode);
    node->set_next_edges(torch::autograd::collect_next_edges(input, kernel));
    node->x = SavedVariable(x16.is_same(input) ? input : x16, false);
    node->w2d = SavedVariable(w2d, false);
    node->has_cols = !fused && !recompute_cols;
    if (node->has_cols) node->cols = SavedVariable(cols, false);
    node->plan = plan;
    node->g = g;
    node->t = t;
    node->dev = dev;
    node->p = p;
    node->fused = fused;
    node->x_f32 = input.scalar_type() == at::kFloat;
    node->w_f32 = kernel.scalar_type() == at::kFloat;
    torch::autograd::set_history(out, node);
    return out;
}

// ---------------------------------------------------------------- LayerNorm
int norm_code(at::ScalarType t) { return t == at::kHalf ? SD_F16 : t == at::kBFloat16 ? SD_BF16 : SD_F32; }

struct SparseDropLayerNormBackward : public Node {
    SavedVariable x, weight;
    Tensor mean, rstd;
    bool has_bias = false;
    std::vector<int64_t> shape;

    std::string name() const override { return "SparseDropLayerNormBackward"; }
    void release_variables() override {
        x.reset_data();
        weight.reset_data();
        mean.reset();
        rstd.reset();
    }
    variable_list apply(variable_list&& grads) override { return backward_call([&] { return gradients(std::move(grads)); }); }
    variable_list gradients(variable_list&& grads) {
        at::NoGradGuard no_grad;
        Tensor x2 = x.unpack(), g = weight.unpack();
        const at::Device dev = rstd.device();
        c10::cuda::OptionalCUDAGuard guard(dev);
        const int64_t n = shape.back(), rows = rstd.numel();
        x2 = dense16(came_back(x2, shape, at::kFloat, dev));
        g = dense16(came_back(g, {n}, at::kFloat, dev));
        cudaStream_t st = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
        Tensor dy = grads[0].defined() ? grads[0] : at::zeros(shape, x2.options());
        const at::ScalarType t = dy.scalar_type();
        if (t != at::kFloat && t != at::kHalf && t != at::kBFloat16) dy = dy.to(at::kFloat);
        dy = dy.contiguous();
        Tensor dx = at::detail::empty_cuda(shape, at::kFloat, dev, std::nullopt);
        Tensor dg = at::detail::empty_cuda({n}, at::kFloat, dev, std::nullopt), db;
        if (has_bias) db = at::detail::empty_cuda({n}, at::kFloat, dev, std::nullopt);
        Tensor ws = empty_bytes(int64_t(sd_layernorm_bwd_workspace_bytes(int(rows), int(n))), dev);
        check_rc(sd_layernorm_bwd(x2.data_ptr<float>(), dy.data_ptr(), norm_code(dy.scalar_type()), g.data_ptr<float>(),
                                  mean.data_ptr<float>(), rstd.data_ptr<float>(), int(rows), int(n), dx.data_ptr<float>(),
                                  dg.data_ptr<float>(), has_bias ? db.data_ptr<float>() : nullptr, 0, ws.data_ptr(), st));
        return {dx, dg, db};
    }
};

// Nothing if the kernels do not serve these tensors: fp32 rows of up to 1024 elements, a multiple of 4, on a CUDA device.
std::optional<Tensor> layer_norm(const Tensor& x, const Tensor& weight, const std::optional<Tensor>& bias_, double eps) {
    py::gil_scoped_release no_gil;
    {
        const int64_t w = x.dim() ? x.size(-1) : 0;
        const auto plain = [&](const Tensor& t) {
            return t.scalar_type() == at::kFloat && t.is_contiguous() && t.dim() == 1 && t.size(0) == w && t.device() == x.device();
        };
        if (!x.is_cuda() || x.scalar_type() != at::kFloat || w % 4 || w <= 0 || w > 1024 || x.numel() == 0 || x.numel() / w >= (1ll << 31) ||
            !plain(weight) || (bias_ && !plain(*bias_)))
            return std::nullopt;
    }
    at::ScalarType out_t = at::kFloat;
    if (at::autocast::is_autocast_enabled(at::kCUDA)) {
        const at::ScalarType dt = at::autocast::get_autocast_dtype(at::kCUDA);
        if (dt == at::kHalf || dt == at::kBFloat16) out_t = dt;
    }
    const Tensor bias = bias_ ? *bias_ : Tensor();
    no_forward_ad("SparseDropLayerNorm", {x, weight, bias});
    const at::Device dev = x.device();
    c10::cuda::OptionalCUDAGuard guard(dev);
    cudaStream_t st = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
    const int64_t n = x.size(-1), rows = x.numel() / n;
    Tensor xc, y, mean, rstd;
    {
        at::NoGradGuard no_grad;
        xc = x.contiguous();
        y = at::detail::empty_cuda(x.sizes(), out_t, dev, std::nullopt);
        mean = at::detail::empty_cuda({rows}, at::kFloat, dev, std::nullopt);
        rstd = at::detail::empty_cuda({rows}, at::kFloat, dev, std::nullopt);
        check_rc(sd_layernorm_fwd(xc.data_ptr<float>(), int(rows), int(n), weight.data_ptr<float>(),
                                  bias.defined() ? bias.data_ptr<float>() : nullptr, float(eps), y.data_ptr(), norm_code(out_t),
                                  mean.data_ptr<float>(), rstd.data_ptr<float>(), st));
    }
    if (!torch::autograd::compute_requires_grad(x, weight, bias)) return y;
    std::shared_ptr<SparseDropLayerNormBackward> node(new SparseDropLayerNormBackward(), torch::autograd::deleteNode);
    node->set_next_edges(torch::autograd::collect_next_edges(x, weight, bias));
    node->x = SavedVariable(xc.is_same(x) ? x : xc, false);
    node->weight = SavedVariable(weight, false);
    node->mean = mean;
    node->rstd = rstd;
    node->has_bias = bias.defined();
    node->shape = x.sizes().vec();
    torch::autograd::set_history(y, node);
    return y;
}

// ---------------------------------------------------------------- GELU
inline bool aligned16(const Tensor& t) { return reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0; }

struct SparseDropGeluBackward : public Node {
    SavedVariable x;
    at::ScalarType type = at::kHalf;

    std::string name() const override { return "SparseDropGeluBackward"; }
    void release_variables() override { x.reset_data(); }
    variable_list apply(variable_list&& grads) override { return backward_call([&] { return gradients(std::move(grads)); }); }
    variable_list gradients(variable_list&& grads) {
        if (!grads[0].defined()) return {Tensor()};
        const Tensor h = x.unpack();
        // the gradient's own graph is wanted, or it carries a batch dimension or a tangent that only torch's operators follow
        if (at::GradMode::is_enabled() || at::isTensorSubclassLike(grads[0]) || at::isTensorSubclassLike(h) ||
            torch::autograd::isFwGradDefined(grads[0]))
            return {at::gelu_backward(grads[0], h)};
        Tensor dy = grads[0];
        const at::Device dev = dy.device();
        const Tensor hc = dense16(came_back(h, dy.sizes(), type, dev));
        if (dy.scalar_type() != type) dy = dy.to(type);
        dy = dense16(dy);
        c10::cuda::OptionalCUDAGuard guard(dev);
        Tensor dx = at::detail::empty_cuda(hc.sizes(), hc.scalar_type(), dev, std::nullopt);
        check_rc(sd_gelu_bwd(dy.data_ptr(), hc.data_ptr(), dx.data_ptr(), hc.numel(), dtype_code(hc.scalar_type()),
                             c10::cuda::getCurrentCUDAStream(dev.index()).stream()));
        return {dx};
    }
};

// Nothing if the kernels do not serve this tensor: a plain contiguous 16-bit one on a CUDA device.
std::optional<Tensor> gelu(const Tensor& x) {
    py::gil_scoped_release no_gil;
    const at::ScalarType t = x.scalar_type();
    if (!x.is_cuda() || (t != at::kHalf && t != at::kBFloat16) || at::isTensorSubclassLike(x) || !x.is_contiguous() || !x.numel() ||
        !aligned16(x) || torch::autograd::isFwGradDefined(x))
        return std::nullopt;
    const at::Device dev = x.device();
    c10::cuda::OptionalCUDAGuard guard(dev);
    Tensor y = at::detail::empty_cuda(x.sizes(), t, dev, std::nullopt);
    check_rc(sd_gelu_fwd(x.data_ptr(), y.data_ptr(), x.numel(), dtype_code(t), c10::cuda::getCurrentCUDAStream(dev.index()).stream()));
    if (!torch::autograd::compute_requires_grad(x)) return y;
    std::shared_ptr<SparseDropGeluBackward> node(new SparseDropGeluBackward(), torch::autograd::deleteNode);
    node->set_next_edges(torch::autograd::collect_next_edges(x));
    node->x = SavedVariable(x, false);
    node->type = t;
    torch::autograd::set_history(y, node);
    return y;
}

// ---------------------------------------------------------------- residual sum
struct SparseDropResidualBackward : public Node {
    at::ScalarType r_type = at::kHalf;

    std::string name() const override { return "SparseDropResidualBackward"; }
    variable_list apply(variable_list&& grads) override {
        const Tensor& dy = grads[0];
        if (!dy.defined()) return {Tensor(), Tensor()};
        return {dy, task_should_compute_output(1) ? dy.to(r_type) : Tensor()};
    }
};

// x + r, or nothing if the kernel does not serve these tensors: plain contiguous ones of one shape, x in fp32, r in 16 bits.
std::optional<Tensor> residual_add(const Tensor& x, const Tensor& r) {
    py::gil_scoped_release no_gil;
    const at::ScalarType t = r.scalar_type();
    if (!x.is_cuda() || x.scalar_type() != at::kFloat || (t != at::kHalf && t != at::kBFloat16) || r.device() != x.device() ||
        at::isTensorSubclassLike(x) || at::isTensorSubclassLike(r) || x.sizes() != r.sizes() || !x.numel() || !x.is_contiguous() ||
        !r.is_contiguous() || !aligned16(x) || !aligned16(r) || torch::autograd::isFwGradDefined(x) || torch::autograd::isFwGradDefined(r))
        return std::nullopt;
    const at::Device dev = x.device();
    c10::cuda::OptionalCUDAGuard guard(dev);
    Tensor y = at::detail::empty_cuda(x.sizes(), at::kFloat, dev, std::nullopt);
    check_rc(sd_residual_add(x.data_ptr<float>(), r.data_ptr(), y.data_ptr<float>(), x.numel(), dtype_code(t),
                             c10::cuda::getCurrentCUDAStream(dev.index()).stream()));
    if (!torch::autograd::compute_requires_grad(x, r)) return y;
    std::shared_ptr<SparseDropResidualBackward> node(new SparseDropResidualBackward(), torch::autograd::deleteNode);
    node->set_next_edges(torch::autograd::collect_next_edges(x, r));
    node->r_type = t;
    torch::autograd::set_history(y, node);
    return y;
}

// ---------------------------------------------------------------- AdamW
// The tensors of one optimizer, described to the kernel once; a step checks that none of them has moved since.  Only weak
// references are held: parameters lead back to whoever holds this object (their gradient hooks), and Python's collector
// cannot look through it.
struct AdamW {
    std::vector<std::array<c10::weak_intrusive_ptr<c10::TensorImpl>, 5>> tensors;    // p, g, m, v, step
    std::vector<std::array<void*, 5>> where;
    Tensor table;
    int64_t chunks = 0;

    AdamW(const std::vector<std::array<Tensor, 5>>& t, const std::vector<int64_t>& groups) {
        std::vector<sd_adamw_entry> e;
        for (size_t i = 0; i < t.size(); ++i) {
            std::array<void*, 5> at;
            for (int j = 0; j < 5; ++j) {
                const Tensor& x = t[i][j];
                if (!x.is_cuda() || x.scalar_type() != at::kFloat || !x.is_contiguous() || x.device() != t[0][0].device() ||
                    x.numel() != (j < 4 ? t[i][0].numel() : 1))
                    bad("AdamW: contiguous fp32 CUDA tensors of one device are needed");
                at[j] = x.data_ptr();
            }
            where.push_back(at);
            using Weak = c10::weak_intrusive_ptr<c10::TensorImpl>;
            tensors.push_back({Weak(t[i][0].getIntrusivePtr()), Weak(t[i][1].getIntrusivePtr()), Weak(t[i][2].getIntrusivePtr()),
                               Weak(t[i][3].getIntrusivePtr()), Weak(t[i][4].getIntrusivePtr())});
            e.push_back({static_cast<float*>(at[0]), static_cast<const float*>(at[1]), static_cast<float*>(at[2]),
                         static_cast<float*>(at[3]), static_cast<float*>(at[4]), t[i][0].numel(), int32_t(groups[i]), 0});
            chunks += (e.back().n + SD_ADAMW_CHUNK - 1) / SD_ADAMW_CHUNK;
        }
        const int n = int(e.size());
        std::vector<char> host(sd_adamw_table_bytes(e.data(), n));
        check_rc(sd_adamw_table_fill(host.data(), e.data(), n));
        table = at::from_blob(host.data(), {int64_t(host.size())}, at::kByte).to(t[0][0].device());
    }
    // false, with nothing done, if a tensor is gone or no longer where the table says
    bool step(const std::vector<double>& hyper) {
        py::gil_scoped_release no_gil;
        std::vector<Tensor> held;
        held.reserve(5 * tensors.size());
        for (size_t i = 0; i < tensors.size(); ++i)
            for (int j = 0; j < 5; ++j) {
                auto t = tensors[i][j].lock();
                if (!t) return false;
                held.emplace_back(std::move(t));
                if (held.back().data_ptr() != where[i][j]) return false;
            }
        const at::Device dev = table.device();
        c10::cuda::OptionalCUDAGuard guard(dev);
        check_rc(sd_adamw_step(table.data_ptr(), chunks, hyper.data(), int(hyper.size() / 5),
                               c10::cuda::getCurrentCUDAStream(dev.index()).stream()));
        for (size_t i = 0; i < held.size(); ++i)   // in-place updates, as autograd sees them
            if (i % 5 != 1) held[i].unsafeGetTensorImpl()->bump_version();
        return true;
    }
};

}  // namespace

PYBIND11_MODULE(sd_torch, m) {
    m.doc() = "Native host path of the SparseDrop operator API";
    py::register_exception_translator([](std::exception_ptr e) {
        try {
            if (e) std::rethrow_exception(e);
        } catch (const SdError& err) {
            set_python_error(err);
        }
    });
    register_node();
    m.def("linear", &linear);
    m.def("conv2d", &conv2d);
    m.def("gemm", &gemm_dense);
    m.def("gemm_dsd", &gemm_dsd);
    m.def("gemm_sdd", &gemm_sdd);
    m.def("layer_norm", &layer_norm);
    m.def("gelu", &gelu);
    m.def("residual_add", &residual_add);
    py::class_<AdamW>(m, "AdamW")
        .def(py::init<const std::vector<std::array<Tensor, 5>>&, const std::vector<int64_t>&>())
        .def("step", &AdamW::step);
    m.def("status_word", [](int dev) { return status_tensor(dev); });
    m.def("has_status_word", [](int dev) {
        std::lock_guard<std::mutex> lock(state_mutex());
        auto it = states().find(dev);
        return it != states().end() && it->second.status.defined();
    });
    m.def("workspace", [](int dev, uint64_t stream) { return workspace_tensor(dev, reinterpret_cast<cudaStream_t>(stream)); });
    m.def("workspaces", [](int dev) {
        std::lock_guard<std::mutex> lock(state_mutex());
        std::vector<Tensor> all;
        for (auto& w : states()[dev].workspaces) all.push_back(w.second);
        return all;
    });
}
