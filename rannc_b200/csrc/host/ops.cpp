// The fused operators' host side: argument checks, output allocation, kernel launches and autograd nodes.
//
// An operator of a small batch is bound by the host: as Python autograd functions over ctypes, the forward and
// backward of a linear layer of 32 rows took 155 us for 40 us of device time -- filling a ctypes structure and
// re-reading strides per GEMM, two trips through the Python autograd machinery, and a hand-over of the interpreter
// lock to the backward thread.  The nodes here are plain autograd nodes: backward runs without the interpreter
// unless a gradient listener is installed.
//
// Kernels are called through the C ABI of _kernels.so; their addresses are handed over once by ops/_lib.py, so that
// the regular and the checked build of the library serve the same code.
// Reference counterpart: the interpreter loop of src/torch/TorchDriver.cpp:566.
#include <ATen/Context.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/forward_grad.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/accumulate_grad.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/extension.h>

#include <array>
#include <atomic>
#include <optional>
#include <unordered_map>

#include "../cuda/attn.h"
#include "../cuda/gemm_tcgen05.h"
#include "../cuda/sparse_rows.h"

namespace {

using at::Tensor;
using torch::autograd::Node;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;
using OptTensor = std::optional<Tensor>;

// ------------------------------------------------------------------------------------------------ C ABI
struct Api {
    int (*gemm)(const RbGemmArgs*, void*);
    int (*gemm_splits)(long long, long long, long long);
    int (*unstack3)(const void*, int, const float*, void* const*, void* const*, long long, long long, int, void*);
    int (*gelu)(const void*, const void*, void*, long long, int, int, void*);
    int (*colsum)(const void*, float*, int, int, long long, int, void*);
    int (*ln_fwd)(const void*, const void*, const void*, const void*, void*, void*, float*, float*, int, int, float,
                  float, uint64_t, uint64_t, int, void*);
    int (*ln_bwd)(const void*, const void*, const void*, const float*, const float*, void*, void*, float*, float*,
                  float*, int, int, float, uint64_t, uint64_t, int, int, void*);
    int (*ln_bwd16)(const void*, const void*, const void*, const float*, const float*, void*, void*, void*, void*, float*,
                    int, int, float, uint64_t, uint64_t, int, void*);
    int (*ln_bwd_grid)(int);
    int (*embed_fwd)(const long long*, const void*, void*, int, int, long long, int, void*);
    int (*embed_bwd)(const long long*, const void*, float*, int, int, long long, long long, int, void*);
    int (*xent_fwd)(const void*, const long long*, float*, float*, float*, int, int, long long, long long, float, int,
                    void*);
    int (*xent_bwd)(const void*, const long long*, const float*, const float*, const float*, void*, int, int, int, long long,
                    long long, float, int, void*);
    int (*attn_fwd)(const RbAttnArgs*, void*);
    int (*attn_bwd)(const RbAttnArgs*, void*);
    int (*attn_bwd_adds)(const RbAttnArgs*);
    int (*bn_fwd)(const void*, const void*, const float*, const float*, void*, float*, float*, float*, float*, float*,
                  long long, int, float, float, int, int, void*);
    int (*bn_bwd)(const void*, const void*, const void*, const float*, const float*, const float*, float*, float*, float*,
                  void*, void*, long long, int, int, int, void*);
    long long (*bn_part_floats)(long long, int);
    int (*gemm_pairs)();
    decltype(&rb_rows_plan) rows_plan;
    decltype(&rb_rows_gather) rows_gather;
    decltype(&rb_rows_scatter_parts) rows_scatter;
} api;
std::atomic<long long> launches{0};
PyObject* error_class = nullptr;   // ops._lib.KernelLibraryError
PyObject* listener = nullptr;      // called with the parameters whose gradients were just written (under the GIL)
std::atomic<bool> has_listener{false};

void check(int rc, const char* what, int kernels = 1) {
    if (rc == 0) {
        launches.fetch_add(kernels, std::memory_order_relaxed);
        return;
    }
    py::gil_scoped_acquire gil;
    PyErr_Format(error_class ? error_class : PyExc_RuntimeError, "%s failed with code %d", what, rc);
    python_error e;
    e.persist();
    throw e;
}

void* cur_stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

int dt_code(const Tensor& t) {
    if (t.scalar_type() == at::kBFloat16) return 1;
    if (t.scalar_type() == at::kHalf) return 0;
    TORCH_CHECK_TYPE(false, "unsupported dtype ", t.scalar_type());
}
const void* cptr(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }
template <typename T = void>
T* mptr(const Tensor& t) { return t.defined() ? static_cast<T*>(t.data_ptr()) : nullptr; }
Tensor opt(const OptTensor& t) { return t.has_value() ? *t : Tensor(); }
Tensor f32(at::IntArrayRef sizes, const Tensor& like) { return at::empty(sizes, like.options().dtype(at::kFloat)); }
bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }
Tensor dense(const Tensor& t) { return !t.defined() || t.is_contiguous() ? t : t.contiguous(); }
// contiguous and on a 16-byte boundary, for kernels that read whole vectors (a view may start at any element)
Tensor dense16(const Tensor& t) {
    return !t.defined() || (t.is_contiguous() && aligned16(t.data_ptr())) ? t : t.clone(at::MemoryFormat::Contiguous);
}

// ------------------------------------------------------------------------------------------------ operand checks
// Kernels get bare addresses: they read an operand in the type, and as many elements of it, as the call's other operands
// say.  What would be misread is refused here, before anything is launched.
void same_type(const char* op, const Tensor& x, std::initializer_list<const Tensor*> others) {
    for (const Tensor* t : others)
        if (t->defined())
            TORCH_CHECK_TYPE(t->scalar_type() == x.scalar_type() && t->device() == x.device(), op,
                             ": the operands' types or devices differ (", x.scalar_type(), " on ", x.device(), " and ",
                             t->scalar_type(), " on ", t->device(), ")");
}
void length(const char* op, const Tensor& t, int64_t n) {
    TORCH_CHECK_VALUE(!t.defined() || t.numel() == n, op, ": ", n, " elements expected, not ", t.numel());
}
// a parameter's gradient buffer: fp32 and dense, as many elements as the parameter
Tensor grad_buffer(const char* op, const OptTensor& buffer, const Tensor& param) {
    if (!buffer.has_value() || !buffer->defined()) return Tensor();
    length(op, *buffer, param.numel());
    TORCH_CHECK_TYPE(buffer->scalar_type() == at::kFloat && buffer->device() == param.device(), op,
                     ": gradient buffers are fp32, on the parameter's device");
    TORCH_CHECK_VALUE(buffer->is_contiguous(), op, ": gradient buffers are contiguous");
    return *buffer;
}
// a matrix that a GEMM adds to: rows of any stride, in fp32 or in the parameter's own type
Tensor weight_grad_buffer(const char* op, const OptTensor& buffer, const Tensor& w) {
    if (!buffer.has_value() || !buffer->defined()) return Tensor();
    TORCH_CHECK_TYPE((buffer->scalar_type() == at::kFloat || buffer->scalar_type() == w.scalar_type()) &&
                         buffer->device() == w.device(),
                     op, ": a weight's gradient buffer is fp32 or of the weight's type, on its device");
    TORCH_CHECK_VALUE(buffer->sizes() == w.sizes() && buffer->stride(1) == 1, op,
                      ": a weight's gradient buffer has the weight's sizes and dense rows");
    return *buffer;
}

// ------------------------------------------------------------------------------------------------ GEMM
// A matrix as the copy engine wants it: 16-byte aligned base, unit column stride, row stride a multiple of 8.  One
// that does not qualify is copied into rows padded to 8 elements; the padding is never read as data.
struct Mat {
    Tensor keep;
    const void* p = nullptr;
    int64_t rows = 0, cols = 0, ld = 0;
};
Mat mat(const Tensor& t) {
    Mat m;
    m.rows = t.size(0);
    m.cols = t.size(1);
    if (aligned16(t.data_ptr()) && t.stride(1) == 1 && t.stride(0) % 8 == 0) {
        m.keep = t;
    } else {
        m.keep = at::zeros({m.rows, (m.cols + 7) / 8 * 8}, t.options()).narrow(1, 0, m.cols);
        m.keep.copy_(t);
    }
    m.p = m.keep.data_ptr();
    m.ld = m.keep.stride(0);
    return m;
}
// the [rows, last dimension] matrix of a contiguous tensor, whatever its other dimensions
Mat rows_of(const Tensor& t) {
    const int64_t c = t.size(-1);
    if (aligned16(t.data_ptr()) && c % 8 == 0) {
        Mat m;
        m.keep = t;
        m.p = t.data_ptr();
        m.cols = m.ld = c;
        m.rows = c ? t.numel() / c : 0;
        return m;
    }
    return mat(t.reshape({-1, c}));
}
Mat columns(const Mat& m, int64_t first, int64_t n) {   // n columns of m (first a multiple of 8)
    Mat r = m;
    r.p = static_cast<const char*>(m.p) + first * 2;
    r.cols = n;
    return r;
}
struct Epi {
    const void* bias = nullptr;
    const void* aux_in = nullptr;
    void* aux_out = nullptr;
    bool gelu = false, dgelu = false, accumulate = false;
    float* a_colsum = nullptr;   // the column sums of a stored [K, M] are added here
    int32_t* rows_ctl = nullptr;   // see RbGemmArgs
    int rows_mode = 0, rows_out = 0;
};
// out [M, N] = epilogue(op(a) op(b)), rows ldd apart (0: N)
void gemm(const Mat& a, const Mat& b, bool trans_a, bool trans_b, void* out, bool out_fp32, int dtype, const Epi& e,
          int64_t ldd = 0) {
    RbGemmArgs g;
    memset(&g, 0, sizeof(g));
    g.A = a.p;
    g.B = b.p;
    g.D = out;
    g.bias = e.bias;
    g.aux_in = e.aux_in;
    g.aux_out = e.aux_out;
    g.M = trans_a ? a.cols : a.rows;
    g.K = trans_a ? a.rows : a.cols;
    g.N = trans_b ? b.rows : b.cols;
    const int64_t kb = trans_b ? b.cols : b.rows;
    TORCH_CHECK_VALUE(kb == g.K, "gemm: inner dimensions differ (", g.K, " vs ", kb, ")");
    g.batch = 1;
    g.lda = a.ld;
    g.ldb = b.ld;
    g.ldd = ldd ? ldd : g.N;
    g.a_major = trans_a ? 1 : 0;
    g.b_major = trans_b ? 0 : 1;
    g.in_dtype = dtype;
    g.out_dtype = out_fp32 ? 1 : 0;
    g.flags = (e.bias ? RB_GEMM_BIAS : 0) | (e.gelu ? RB_GEMM_GELU : 0) | (e.dgelu ? RB_GEMM_DGELU : 0) |
              (e.accumulate ? RB_GEMM_ACCUM : 0) | (e.aux_out ? RB_GEMM_AUX_OUT : 0);
    g.alpha = 1.f;
    g.a_colsum = e.a_colsum;
    g.rows_ctl = e.rows_ctl;
    g.rows_mode = e.rows_mode;
    g.rows_out = e.rows_out;
    g.in_order = at::globalContext().deterministicAlgorithms() ? 1 : 0;
    check(api.gemm(&g, cur_stream()), "rb_gemm");
}
// ---- rows of zeros in the gradient of a wide output layer (cuda/sparse_rows.cu) ----
// The rows that count are gathered on the device, and each product is launched in two forms of which the device runs one.
struct Rows {
    Tensor keep;   // all of it: one allocation
    int32_t *idx = nullptr, *pos = nullptr, *ctl = nullptr;
    float* dx32 = nullptr;   // the input gradient's parts, rows_out rows
    Mat dy, x;
    int64_t rows_out = 0;
};
// Worth a look at the rows: a wide output layer (the rows of hidden layers' gradients are not zero), and products long enough
// that the look costs next to nothing where every row counts.  Backward of the layer (us), one B200, over all rows ->
// gathered, by the share of rows that count (up to three quarters are gathered):
//     rows x inputs x outputs     2 %          15 %         30 %         45 %         60 %         80 %         100 %
//     8192 x 1024 x 30528         637 -> 217   649 -> 272   674 -> 381   708 -> 491   720 -> 620   747 -> 686   781 -> 690
//     6144 x 1024 x 30528         560 -> 207   564 -> 247   570 -> 311   592 -> 385   617 -> 467   627 -> 587   637 -> 569
//     4096 x  768 x 30528         308 -> 153   310 -> 170   312 -> 203   312 -> 237   314 -> 276   318 -> 321   320 -> 300
//     4096 x 4096 x 32000        1377 -> 380  1444 -> 464  1479 -> 628  1561 -> 822  1580 ->1132  1668 ->1502  1723 ->1541
// (all rows: before the look existed; what both sides do at 80 and 100 % differs by the clock under the power cap.)
// Rows of zeros are read to find them (425 MB at 15 % of 8192 x 30528: 81 us), which is lost where a few rows more than
// three quarters count: the look is 3 to 8 % of the backward there.  Both products use the kernel of CTA pairs whichever
// form runs, so an input gradient of fewer tiles than 0.64 of the pairs stays out (2048 x 1024 x 30528, where all rows
// count: 235 -> 281; 1024 x 1024 x 30528 gains at 15 %, 181 -> 132, and loses at 100 %, 189 -> 238).
// Where one of the two products is not wanted the other has to be as long as both (4249 x 736 x 30336, 80 % of the rows, the
// weight's gradient alone: 158 -> 186 us).
// `pairs`: of SMs that work on 256 x 256 tiles at once (rb_gemm_pairs).  Returns how many rows there is room for, in steps
// of 64 (few rows leave none: 0, as where the look is not worth it).
int64_t gather_room(int64_t rows, int64_t cols, int64_t inputs, int64_t pairs, int64_t products) {
    auto tiles = [](int64_t m, int64_t n) { return (m + 255) / 256 * ((n + 255) / 256); };
    if (pairs <= 0 || cols < 4 * inputs || cols % 8 || inputs % 8 || cols > (1 << 22) || rows >= (1 << 30) ||
        tiles(cols, inputs) < pairs || 25 * tiles(rows, inputs) < 16 * pairs ||
        static_cast<double>(products) * rows * cols * inputs < 1.8e11)
        return 0;
    return std::min<int64_t>(rows / 4 * 3, (int64_t{1} << 30) / cols) / 64 * 64;   // (2 GiB at most)
}
int64_t gather_room(const Mat& dy, const Mat& x, int64_t products) {
    if (dy.cols < 4 * x.cols || at::globalContext().deterministicAlgorithms()) return 0;   // (most layers, before any call)
    return gather_room(dy.rows, dy.cols, x.cols, api.gemm_pairs(), products);
}
// Scratch: three quarters of dy and of x, and 77 MB or three quarters of x in fp32, whatever the number of rows that count
// (the host does not know it): 470 MB for 8192 x 1024 x 30528.  Where there is no memory for it, `keep` stays empty.
Rows gather_rows(const Mat& dy, const Mat& x, int64_t room, bool want_dx, int dtype, const at::TensorOptions& o) {
    Rows r;
    // The input gradient's product is cut into parts along K, each in rows of its own and added up in their order (as
    // reductions into one matrix they came in any, and dx did not repeat): room for four waves of tiles.
    if (want_dx) r.rows_out = (std::max(room, 4 * api.gemm_pairs() * 256 / ((x.cols + 255) / 256)) + 255) / 256 * 256;
    int64_t bytes = 0;
    auto take = [&](int64_t n) {
        const int64_t at = bytes;
        bytes += (n + 255) / 256 * 256;
        return at;
    };
    const int64_t ctl = take(16), idx = take(room * 4), pos = take(dy.rows * 4), live = take(dy.rows),
                  dy_at = take(room * dy.cols * 2), x_at = take(room * x.cols * 2), dx_at = take(r.rows_out * x.cols * 4);
    try {
        r.keep = at::empty({bytes}, o.dtype(at::kByte));
    } catch (const c10::OutOfMemoryError&) {
        return r;   // the products over all rows need none of it
    }
    char* base = static_cast<char*>(r.keep.data_ptr());
    r.ctl = reinterpret_cast<int32_t*>(base + ctl);
    r.idx = reinterpret_cast<int32_t*>(base + idx);
    r.pos = reinterpret_cast<int32_t*>(base + pos);
    if (want_dx) r.dx32 = reinterpret_cast<float*>(base + dx_at);
    auto gathered = [&](int64_t at, const Mat& of) {
        Mat m;
        m.keep = r.keep;
        m.p = base + at;
        m.rows = room;
        m.cols = m.ld = of.cols;
        return m;
    };
    r.dy = gathered(dy_at, dy);
    r.x = gathered(x_at, x);
    check(api.rows_plan(dy.p, dy.ld, x.p, x.ld, static_cast<int>(dy.rows), static_cast<int>(dy.cols), static_cast<int>(x.cols),
                        static_cast<int>(room), reinterpret_cast<uint8_t*>(base + live), r.idx, r.pos, r.ctl, dtype, cur_stream()),
          "rb_rows_plan", 2);
    check(api.rows_gather(dy.p, dy.ld, x.p, x.ld, static_cast<int>(dy.cols), static_cast<int>(x.cols), r.idx, r.ctl, base + dy_at,
                          base + x_at, nullptr, cur_stream()),
          "rb_rows_gather");
    return r;
}

// Gradients of one weight and its bias: dW = dy^T x and, from the same pass over dy, db = its column sums.  Each is added
// to the fp32 buffer the parameter has, or returned in the parameter's own type.
struct Grads {
    Tensor w, b;
};
// Whether an [m, n] weight gradient over `rows` rows, wanted in the parameter's 16-bit type, is added up in fp32 first.
// A long product with few 256 x 256 tiles leaves most of the GPU idle unless K is split, which takes an fp32 result to
// add to: clearing it and rounding it are two more passes over the weight.  Measured, one 16-bit product against clear +
// split + round (us, weight at rows): 256 x 256 at 2048 14.9 / 9.0; 768 x 768 at 1024 10.0 / 10.9, at 8192 46.7 / 19.6;
// 1024 x 1024 at 2048 15.8 / 16.5, at 4096 26.7 / 21.5; 3072 x 768 at 16384 104.5 / 66.6; 4096 x 1024 at 8192
// 71.9 / 73.3, at 16384 134 / 121: the line lies at 256 rows per tile.  Where the tiles fill the GPU the fp32 result
// would gain nothing.  The parts are added in the order they arrive, so the last bits differ from run to run: not when
// torch.use_deterministic_algorithms asks otherwise.
bool in_parts(int64_t m, int64_t n, int64_t rows) {
    return rows >= std::max<int64_t>(2048, 256 * ((m + 255) / 256) * ((n + 255) / 256)) &&
           !at::globalContext().deterministicAlgorithms() && api.gemm_splits(m, n, rows) > 1;
}
Grads param_grads(const Mat& dy, const Mat& x, const Tensor& w, const Tensor& w_mg, bool want_w, const Tensor& bias,
                  const Tensor& b_mg, bool want_b, int dtype, const Rows* rows = nullptr, const Tensor& w_out = Tensor()) {
    Grads out;
    // dW = dy^T x, over all rows or (whichever the device finds) over the gathered ones
    auto product = [&](void* to, bool fp32, Epi e, int64_t ldd) {
        if (rows) {
            e.rows_ctl = rows->ctl;
            e.rows_mode = RB_GEMM_ROWS_K;
            gemm(rows->dy, rows->x, true, false, to, fp32, dtype, e, ldd);
            e.rows_mode = RB_GEMM_ROWS_ALL;
        }
        gemm(dy, x, true, false, to, fp32, dtype, e, ldd);
    };
    Tensor db;
    if (bias.defined() && want_b) db = b_mg.defined() ? b_mg : at::zeros({dy.cols}, bias.options().dtype(at::kFloat));
    if (want_w) {
        Epi e;
        e.a_colsum = mptr<float>(db);
        if (w_mg.defined()) {
            e.accumulate = true;
            product(w_mg.data_ptr(), w_mg.scalar_type() == at::kFloat, e, w_mg.stride(0));
        } else if (in_parts(dy.cols, x.cols, dy.rows)) {
            Tensor w32 = at::zeros({dy.cols, x.cols}, w.options().dtype(at::kFloat));
            e.accumulate = true;
            gemm(dy, x, true, false, w32.data_ptr(), true, dtype, e);
            out.w = w32.to(w.scalar_type());
        } else {
            out.w = w_out.defined() ? w_out : at::empty({dy.cols, x.cols}, w.options());
            product(out.w.data_ptr(), false, e, 0);
        }
    } else if (db.defined()) {
        check(api.colsum(dy.p, mptr<float>(db), static_cast<int>(dy.rows), static_cast<int>(dy.cols), dy.ld, dtype,
                         cur_stream()),
              "rb_colsum");
    }
    if (db.defined() && !b_mg.defined()) out.b = db.to(bias.scalar_type());
    return out;
}

// The gradients of three projections whose dy lie side by side in the columns of `dy`: one product, whose row blocks leave
// as tensors of their own (views of one would share its storage and version).
std::array<Grads, 3> stacked_grads(const Mat& dy, const Mat& x, const Tensor& w, const Tensor& bias, int dtype) {
    const bool parts = in_parts(dy.cols, x.cols, dy.rows);
    const auto wide = w.options().dtype(at::kFloat);
    Tensor all = parts ? at::zeros({dy.cols, x.cols}, wide) : at::empty({dy.cols, x.cols}, w.options()), db;
    if (bias.defined()) db = at::zeros({dy.cols}, wide);
    Epi e;
    e.accumulate = parts;
    e.a_colsum = mptr<float>(db);
    gemm(dy, x, true, false, all.data_ptr(), parts, dtype, e);
    std::array<Grads, 3> out;
    const int64_t n = dy.cols / 3;
    void *wd[3], *bd[3];
    for (int i = 0; i < 3; ++i) {
        out[i].w = at::empty({n, x.cols}, w.options());
        if (db.defined()) out[i].b = at::empty({n}, w.options());
        wd[i] = mptr(out[i].w);
        bd[i] = mptr(out[i].b);
    }
    check(api.unstack3(all.data_ptr(), parts ? 1 : 0, mptr<float>(db), wd, bd, n * x.cols, n, dtype, cur_stream()),
          "rb_unstack3");
    return out;
}

// ------------------------------------------------------------------------------------------------ autograd plumbing
bool wants_grad(std::initializer_list<const Tensor*> ts) {
    bool any = false;
    for (const Tensor* t : ts) {
        if (!t->defined()) continue;
        TORCH_CHECK_NOT_IMPLEMENTED(!torch::autograd::isFwGradDefined(*t),
                                    "the fused operators have no forward-mode derivative");
        any = any || t->requires_grad();
    }
    return any && at::GradMode::is_enabled();
}
template <typename N>
std::shared_ptr<N> new_node() { return std::shared_ptr<N>(new N(), torch::autograd::deleteNode); }

// Tells the listener, when there is one, which parameters' gradients are in their buffers now.
void notify(std::initializer_list<std::pair<const Tensor*, const Tensor*>> param_and_buffer) {
    if (!has_listener.load(std::memory_order_acquire)) return;
    py::gil_scoped_acquire gil;
    if (!listener) return;
    py::list ps;
    for (auto& pb : param_and_buffer)
        if (pb.first->defined() && pb.second->defined()) ps.append(py::cast(*pb.first));
    PyObject* r = PyObject_CallOneArg(listener, ps.ptr());
    if (!r) {
        python_error e;
        e.persist();
        throw e;
    }
    Py_DECREF(r);
}
// A gradient that never arrived counts as zero: the parameters' buffers are complete and reported all the same, which is
// what a gradient reducer waits for.
#define RB_NODE(NAME)                                                              \
    std::string name() const override { return NAME; }                             \
    variable_list apply(variable_list&& grads) override {                          \
        std::lock_guard<std::mutex> lock(mutex_);                                   \
        if (!grads[0].defined()) grads[0] = input_metadata(0).zeros_like();        \
        return run(std::move(grads));                                               \
    }

// ------------------------------------------------------------------------------------------------ linear
struct LinearNode : Node {
    SavedVariable x, w, pre;
    Tensor w_ref, bias, w_mg, b_mg;
    RB_NODE("RbLinearBackward")
    void release_variables() override {
        std::lock_guard<std::mutex> lock(mutex_);
        x.reset_data();
        w.reset_data();
        pre.reset_data();
    }
    variable_list run(variable_list&& grads) {
        const Tensor X = x.unpack(), W = w.unpack(), P = pre.unpack();
        Tensor dy = P.defined() ? dense16(grads[0]) : dense(grads[0]);
        const int dt = dt_code(X);
        if (P.defined()) {
            Tensor d = at::empty(dy.sizes(), dy.options());
            check(api.gelu(P.data_ptr(), dy.data_ptr(), d.data_ptr(), d.numel(), 1, dt, cur_stream()), "rb_gelu");
            dy = d;
        }
        const Mat d = rows_of(dy), xm = rows_of(X);
        const bool want_dx = task_should_compute_output(0), want_w = task_should_compute_output(1);
        Tensor dx, dw;
        if (want_dx) dx = at::empty(X.sizes(), X.options());
        Rows rows;
        if (const int64_t room = P.defined() ? 0 : gather_room(d, xm, want_dx + want_w)) {
            if (want_w && !w_mg.defined()) dw = at::empty({d.cols, xm.cols}, W.options());   // (before the look's scratch)
            rows = gather_rows(d, xm, room, want_dx, dt, X.options());
        }
        const bool look = rows.keep.defined();
        if (want_dx) {
            const Mat wm = mat(W);
            Epi e;
            if (look) {
                e.rows_ctl = rows.ctl;
                e.rows_mode = RB_GEMM_ROWS_M;
                e.rows_out = static_cast<int>(rows.rows_out);
                gemm(rows.dy, wm, false, false, rows.dx32, true, dt, e);
                check(api.rows_scatter(rows.dx32, dx.data_ptr(), static_cast<int>(d.rows), static_cast<int>(xm.cols), rows.pos,
                                       rows.ctl, dt, cur_stream()),
                      "rb_rows_scatter");
                e.rows_mode = RB_GEMM_ROWS_ALL;
            }
            gemm(d, wm, false, false, dx.data_ptr(), false, dt, e);
        }
        const Grads gr = param_grads(d, xm, W, w_mg, want_w, bias, b_mg, bias.defined() && task_should_compute_output(2), dt,
                                     look ? &rows : nullptr, dw);
        notify({{&w_ref, &w_mg}, {&bias, &b_mg}});
        return {dx, gr.w, gr.b};
    }
};

// `owner`: the parameter whose gradient is reported when w is a view of one
Tensor linear(const Tensor& x, const Tensor& w, const OptTensor& bias_, bool gelu, const OptTensor& w_mg,
              const OptTensor& b_mg, const OptTensor& owner) {
    const Tensor bias = opt(bias_);
    same_type("linear", x, {&w, &bias});
    TORCH_CHECK_VALUE(w.dim() == 2, "linear: the weight is a matrix");
    length("linear bias", bias, w.size(0));
    const bool req = wants_grad({&x, &w, &bias});
    Tensor y, pre, xc, bc;
    {
        at::NoGradGuard off;
        xc = dense(x);
        auto sizes = x.sizes().vec();
        sizes.back() = w.size(0);
        y = at::empty(sizes, x.options());
        Epi e;
        bc = dense(bias);
        e.bias = cptr(bc);
        e.gelu = gelu;
        if (gelu && req) {   // (what the backward needs)
            pre = at::empty(sizes, x.options());
            e.aux_out = pre.data_ptr();
        }
        gemm(rows_of(xc), mat(w), false, true, y.data_ptr(), false, dt_code(x), e);
    }
    if (req) {
        auto n = new_node<LinearNode>();
        n->set_next_edges(torch::autograd::collect_next_edges(x, w, bias));
        n->x = SavedVariable(xc, false);
        n->w = SavedVariable(w, false);
        n->pre = SavedVariable(pre, false);
        n->w_ref = owner.has_value() ? *owner : w;
        n->bias = bias;
        n->w_mg = weight_grad_buffer("linear", w_mg, w);
        n->b_mg = grad_buffer("linear", b_mg, bias);
        torch::autograd::set_history(y, n);
    }
    return y;
}

// ------------------------------------------------------------------------------------------------ mlp
// y = gelu(x W1^T + b1) W2^T + b2; the GELU derivative rides in the epilogue of the dgrad GEMM
struct MlpNode : Node {
    SavedVariable x, w1, w2, pre, h;
    Tensor w1_ref, w2_ref, b1, b2, w1_mg, b1_mg, w2_mg, b2_mg;
    RB_NODE("RbMlpBackward")
    void release_variables() override {
        std::lock_guard<std::mutex> lock(mutex_);
        for (SavedVariable* s : {&x, &w1, &w2, &pre, &h}) s->reset_data();
    }
    variable_list run(variable_list&& grads) {
        const Tensor X = x.unpack(), W1 = w1.unpack(), W2 = w2.unpack(), P = pre.unpack(), Hh = h.unpack();
        const Tensor dy = dense(grads[0]);
        const int dt = dt_code(X);
        const Mat d = rows_of(dy), hm = rows_of(Hh);
        const Grads g2 = param_grads(d, hm, W2, w2_mg, true, b2, b2_mg, true, dt);
        Tensor dpre = at::empty(P.sizes(), P.options());
        Epi e;
        e.dgelu = true;
        e.aux_in = P.data_ptr();
        gemm(d, mat(W2), false, false, dpre.data_ptr(), false, dt, e);
        const Mat dp = rows_of(dpre);
        const Grads g1 = param_grads(dp, rows_of(X), W1, w1_mg, true, b1, b1_mg, true, dt);
        Tensor dx;
        if (task_should_compute_output(0)) {
            dx = at::empty(X.sizes(), X.options());
            gemm(dp, mat(W1), false, false, dx.data_ptr(), false, dt, Epi());
        }
        notify({{&w1_ref, &w1_mg}, {&b1, &b1_mg}, {&w2_ref, &w2_mg}, {&b2, &b2_mg}});
        return {dx, g1.w, g1.b, g2.w, g2.b};
    }
};

Tensor mlp(const Tensor& x, const Tensor& w1, const OptTensor& b1_, const Tensor& w2, const OptTensor& b2_,
           const OptTensor& w1_mg, const OptTensor& b1_mg, const OptTensor& w2_mg, const OptTensor& b2_mg) {
    const Tensor b1 = opt(b1_), b2 = opt(b2_);
    same_type("mlp", x, {&w1, &b1, &w2, &b2});
    TORCH_CHECK_VALUE(w1.dim() == 2 && w2.dim() == 2, "mlp: the weights are matrices");
    length("mlp bias", b1, w1.size(0));
    length("mlp bias", b2, w2.size(0));
    const bool req = wants_grad({&x, &w1, &b1, &w2, &b2});
    Tensor xc, pre, h, y, b1c, b2c;
    {
        at::NoGradGuard off;
        xc = dense(x);
        auto sizes = x.sizes().vec();
        sizes.back() = w1.size(0);
        if (req) pre = at::empty(sizes, x.options());   // (what the backward needs)
        h = at::empty(sizes, x.options());
        sizes.back() = w2.size(0);
        y = at::empty(sizes, x.options());
        const int dt = dt_code(x);
        b1c = dense(b1);
        b2c = dense(b2);
        Epi e;
        e.bias = cptr(b1c);
        e.gelu = true;
        e.aux_out = mptr(pre);
        gemm(rows_of(xc), mat(w1), false, true, h.data_ptr(), false, dt, e);
        Epi e2;
        e2.bias = cptr(b2c);
        gemm(rows_of(h), mat(w2), false, true, y.data_ptr(), false, dt, e2);
    }
    if (req) {
        auto n = new_node<MlpNode>();
        n->set_next_edges(torch::autograd::collect_next_edges(x, w1, b1, w2, b2));
        n->x = SavedVariable(xc, false);
        n->w1 = SavedVariable(w1, false);
        n->w2 = SavedVariable(w2, false);
        n->pre = SavedVariable(pre, false);
        n->h = SavedVariable(h, false);
        n->w1_ref = w1;
        n->w2_ref = w2;
        n->b1 = b1;
        n->b2 = b2;
        n->w1_mg = weight_grad_buffer("mlp", w1_mg, w1);
        n->b1_mg = grad_buffer("mlp", b1_mg, b1);
        n->w2_mg = weight_grad_buffer("mlp", w2_mg, w2);
        n->b2_mg = grad_buffer("mlp", b2_mg, b2);
        torch::autograd::set_history(y, n);
    }
    return y;
}

// ------------------------------------------------------------------------------------------------ layer norm
struct LnNode : Node {
    SavedVariable z, gamma, mean, rstd;
    Tensor g_ref, b_ref, g_mg, b_mg;
    double p = 0;
    uint64_t seed = 0, offset = 0;
    RB_NODE("RbLayerNormBackward")
    void release_variables() override {
        std::lock_guard<std::mutex> lock(mutex_);
        for (SavedVariable* s : {&z, &gamma, &mean, &rstd}) s->reset_data();
    }
    variable_list run(variable_list&& grads) {
        const Tensor Z = z.unpack(), G = dense16(gamma.unpack()), M = mean.unpack(), R = rstd.unpack();
        const Tensor dy = dense16(grads[0]);
        const int H = static_cast<int>(Z.size(-1)), rows = static_cast<int>(Z.numel() / H);
        const bool flat = g_mg.defined() && b_mg.defined();
        Tensor dz = at::empty(Z.sizes(), Z.options()), dx = dz;
        // One tensor for both inputs, unless one of them is a leaf: it would copy a gradient that it does not own alone, in
        // a launch of its own, where the kernel writes a second one beside the first (387 x 4096, two leaves, forward and
        // backward: 90.6 -> 82.6 us).
        auto leaf = [&](size_t i) {
            return dynamic_cast<torch::autograd::AccumulateGrad*>(next_edge(i).function.get()) != nullptr;
        };
        // (not where both are the same one, whose gradients the engine adds up)
        const bool both = task_should_compute_output(0) && task_should_compute_output(1) && !(next_edge(0) == next_edge(1));
        if (p > 0 || (both && (leaf(0) || leaf(1)))) dx = at::empty(Z.sizes(), Z.options());
        Tensor partial = f32({static_cast<int64_t>(api.ln_bwd_grid(rows)) * 2 * H}, Z);
        void* dx_own = dx.is_same(dz) ? nullptr : dx.data_ptr();
        if (flat) {
            check(api.ln_bwd(dy.data_ptr(), Z.data_ptr(), G.data_ptr(), mptr<float>(M), mptr<float>(R), dz.data_ptr(), dx_own,
                             mptr<float>(g_mg), mptr<float>(b_mg), mptr<float>(partial), rows, H, static_cast<float>(p),
                             seed, offset, 1, dt_code(Z), cur_stream()),
                  "rb_ln_bwd", 2);
            notify({{&g_ref, &g_mg}, {&b_ref, &b_mg}});
            return {dx, dz, Tensor(), Tensor()};
        }
        // gradients in the parameters' own type, rounded once from the fp32 sums by the reducing kernel
        Tensor dg = at::empty({H}, G.options()), db = at::empty({H}, G.options());
        check(api.ln_bwd16(dy.data_ptr(), Z.data_ptr(), G.data_ptr(), mptr<float>(M), mptr<float>(R), dz.data_ptr(), dx_own,
                           dg.data_ptr(), db.data_ptr(), mptr<float>(partial), rows, H, static_cast<float>(p), seed, offset,
                           dt_code(Z), cur_stream()),
              "rb_ln_bwd16", 2);
        return {dx, dz, dg, db};
    }
};

Tensor layer_norm(const Tensor& x, const OptTensor& res_, const Tensor& gamma, const Tensor& beta, double p, double eps,
                  uint64_t seed, uint64_t offset, const OptTensor& g_mg, const OptTensor& b_mg) {
    const Tensor res = opt(res_);
    same_type("layer_norm", x, {&res, &gamma, &beta});
    length("layer_norm weight", gamma, x.size(-1));
    length("layer_norm bias", beta, x.size(-1));
    TORCH_CHECK_VALUE(!res.defined() || res.sizes() == x.sizes(), "layer_norm: the residual's sizes differ from x's");
    const bool req = wants_grad({&x, &res, &gamma, &beta});
    Tensor xc, y, z, mean, rstd;
    {
        at::NoGradGuard off;
        xc = dense16(x);
        const Tensor rc = dense16(res), gc = dense16(gamma), bc = dense16(beta);
        const int H = static_cast<int>(x.size(-1)), rows = static_cast<int>(x.numel() / H);
        y = at::empty(xc.sizes(), xc.options());
        if (res.defined() || p > 0) z = at::empty(xc.sizes(), xc.options());
        mean = f32({rows}, x);
        rstd = f32({rows}, x);
        check(api.ln_fwd(xc.data_ptr(), cptr(rc), gc.data_ptr(), bc.data_ptr(), y.data_ptr(), mptr(z),
                         mptr<float>(mean), mptr<float>(rstd), rows, H, static_cast<float>(eps), static_cast<float>(p), seed,
                         offset, dt_code(x), cur_stream()),
              "rb_ln_fwd");
        if (!z.defined()) z = xc;
    }
    if (req) {
        auto n = new_node<LnNode>();
        n->set_next_edges(torch::autograd::collect_next_edges(x, res, gamma, beta));
        n->z = SavedVariable(z, false);
        n->gamma = SavedVariable(gamma, false);
        n->mean = SavedVariable(mean, false);
        n->rstd = SavedVariable(rstd, false);
        n->g_ref = gamma;
        n->b_ref = beta;
        n->g_mg = grad_buffer("layer_norm", g_mg, gamma);
        n->b_mg = grad_buffer("layer_norm", b_mg, beta);
        n->p = p;
        n->seed = seed;
        n->offset = offset;
        torch::autograd::set_history(y, n);
    }
    return y;
}

// ------------------------------------------------------------------------------------------------ embedding
struct EmbeddingNode : Node {
    SavedVariable ids;
    Tensor weight, w_mg;
    int64_t padding = -1;
    RB_NODE("RbEmbeddingBackward")
    void release_variables() override {
        std::lock_guard<std::mutex> lock(mutex_);
        ids.reset_data();
    }
    variable_list run(variable_list&& grads) {
        const Tensor I = ids.unpack();
        const Tensor dy = dense(grads[0]);
        Tensor acc = w_mg.defined() ? w_mg : at::zeros(weight.sizes(), weight.options().dtype(at::kFloat).requires_grad(false));
        check(api.embed_bwd(static_cast<const long long*>(I.data_ptr()), dy.data_ptr(), mptr<float>(acc),
                            static_cast<int>(I.numel()), static_cast<int>(dy.size(-1)), weight.size(0), padding, dt_code(dy),
                            cur_stream()),
              "rb_embed_bwd");
        if (w_mg.defined()) {
            notify({{&weight, &w_mg}});
            return {Tensor()};
        }
        return {acc.to(weight.scalar_type())};
    }
};

Tensor embedding(const Tensor& w, const Tensor& ids, int64_t padding, const OptTensor& w_mg) {
    TORCH_CHECK_TYPE(ids.scalar_type() == at::kLong && ids.device() == w.device(),
                     "embedding: the ids are 64-bit integers on the table's device");
    TORCH_CHECK_VALUE(w.dim() == 2 && w.is_contiguous(), "embedding: the table is a contiguous matrix");
    const bool req = wants_grad({&w});
    Tensor out, idc;
    {
        at::NoGradGuard off;
        idc = dense(ids);
        auto sizes = ids.sizes().vec();
        sizes.push_back(w.size(1));
        out = at::empty(sizes, w.options().requires_grad(false));
        const Tensor table = dense16(w);
        check(api.embed_fwd(static_cast<const long long*>(idc.data_ptr()), table.data_ptr(), out.data_ptr(),
                            static_cast<int>(ids.numel()), static_cast<int>(w.size(1)), w.size(0), dt_code(w), cur_stream()),
              "rb_embed_fwd");
    }
    if (req) {
        auto n = new_node<EmbeddingNode>();
        n->set_next_edges(torch::autograd::collect_next_edges(w));
        n->ids = SavedVariable(idc, false);
        n->weight = w;
        n->w_mg = grad_buffer("embedding", w_mg, w);
        n->padding = padding;
        torch::autograd::set_history(out, n);
    }
    return out;
}

// ------------------------------------------------------------------------------------------------ cross entropy
struct XentNode : Node {
    SavedVariable logits, labels, lse, acc;
    int64_t V = 0, ignore = 0;
    double weight = 1;
    RB_NODE("RbCrossEntropyBackward")
    void release_variables() override {
        std::lock_guard<std::mutex> lock(mutex_);
        for (SavedVariable* s : {&logits, &labels, &lse, &acc}) s->reset_data();
    }
    variable_list run(variable_list&& grads) {
        const Tensor L = logits.unpack(), lab = labels.unpack(), ls = lse.unpack(), ac = acc.unpack();
        const Tensor g = grads[0].to(at::kFloat).contiguous();
        // the logits are dead after the loss: their buffer receives the gradient
        Tensor d = L.detach();
        check(api.xent_bwd(L.data_ptr(), static_cast<const long long*>(lab.data_ptr()), mptr<float>(ls), mptr<float>(ac),
                           mptr<float>(g), d.data_ptr(), static_cast<int>(L.size(0)), static_cast<int>(V),
                           static_cast<int>(L.size(1)), L.stride(0), ignore, static_cast<float>(weight), dt_code(L), cur_stream()),
              "rb_xent_bwd");
        return {d};
    }
};

Tensor cross_entropy(const Tensor& logits, const Tensor& labels, int64_t V, int64_t ignore, double weight) {
    TORCH_CHECK_TYPE(labels.scalar_type() == at::kLong && labels.device() == logits.device(),
                     "cross_entropy: the labels are 64-bit integers on the logits' device");
    TORCH_CHECK_VALUE(logits.dim() == 2 && logits.stride(1) == 1 && labels.is_contiguous() &&
                          (logits.size(0) <= 1 || logits.stride(0) >= logits.size(1)) &&
                          labels.numel() == logits.size(0) && V > 0 && V <= logits.size(1),
                      "cross_entropy: one label per row of logits, and no more classes than columns");
    const bool req = wants_grad({&logits});
    Tensor lse, acc, loss;
    {
        at::NoGradGuard off;
        lse = f32({logits.size(0)}, logits);
        acc = at::zeros({2}, lse.options());
        loss = at::empty({}, lse.options());
        check(api.xent_fwd(logits.data_ptr(), static_cast<const long long*>(labels.data_ptr()), mptr<float>(lse),
                           mptr<float>(acc), mptr<float>(loss), static_cast<int>(logits.size(0)), static_cast<int>(V),
                           logits.stride(0), ignore, static_cast<float>(weight), dt_code(logits), cur_stream()),
              "rb_xent_fwd", 2);
    }
    if (req) {
        auto n = new_node<XentNode>();
        n->set_next_edges(torch::autograd::collect_next_edges(logits));
        n->logits = SavedVariable(logits, false);
        n->labels = SavedVariable(labels, false);
        n->lse = SavedVariable(lse, false);
        n->acc = SavedVariable(acc, false);
        n->V = V;
        n->ignore = ignore;
        n->weight = weight;
        torch::autograd::set_history(loss, n);
    }
    return loss;
}

// ------------------------------------------------------------------------------------------------ QKV + attention
// Three tensors that lie back to back in one storage, in this order, seen as one (what the parameter storage does
// with the projections of a block): the address they start at, or null.
const void* adjacent(const Tensor* t) {
    const char* p = static_cast<const char*>(t[0].data_ptr());
    const char* next = p;
    for (int i = 0; i < 3; ++i) {
        if (!t[i].defined() || !t[i].is_contiguous() || t[i].scalar_type() != t[0].scalar_type() ||
            t[i].sizes().slice(1) != t[0].sizes().slice(1) || !t[i].storage().is_alias_of(t[0].storage()) ||
            static_cast<const char*>(t[i].data_ptr()) != next)
            return nullptr;
        next += t[i].nbytes();
    }
    return p;
}
// The three projection weights as one [3 Ho, hid] matrix: in place where they lie back to back, else a stack made for
// this use (`copied`).  A stack is never kept from one call for another: nothing tells when the values it was made of
// change (an update through .data or by a kernel leaves no trace on the parameter).
Mat stacked(const Tensor* w, bool& copied) {
    const void* p = adjacent(w);
    copied = !(p && aligned16(p) && w[0].size(1) % 8 == 0);
    if (copied) return mat(at::cat({w[0].detach(), w[1].detach(), w[2].detach()}, 0));
    Mat m;
    m.keep = w[0];
    m.p = p;
    m.rows = 3 * w[0].size(0);
    m.cols = m.ld = w[0].size(1);
    return m;
}
void attn_args(RbAttnArgs& a, const Tensor& qkv, const Tensor& o, const Tensor& lse, const Tensor& bias, int64_t B, int64_t S,
               int64_t H, double scale, double p, uint64_t seed, uint64_t offset) {
    memset(&a, 0, sizeof(a));
    const char* base = static_cast<const char*>(qkv.data_ptr());
    const int64_t Ho = H * 64;
    a.Q = base;
    a.K = base + Ho * 2;
    a.V = base + 2 * Ho * 2;
    a.q_sb = a.k_sb = a.v_sb = S * 3 * Ho;
    a.q_ss = a.k_ss = a.v_ss = 3 * Ho;
    a.q_sh = a.k_sh = a.v_sh = 64;
    a.O = o.data_ptr();
    a.o_sb = S * Ho;
    a.o_ss = Ho;
    a.o_sh = 64;
    a.lse = mptr<float>(lse);
    a.key_bias = mptr<float>(bias);
    a.B = static_cast<int32_t>(B);
    a.S = static_cast<int32_t>(S);
    a.H = static_cast<int32_t>(H);
    a.D = 64;
    a.dtype = dt_code(qkv);
    a.scale = static_cast<float>(scale);
    a.p_drop = static_cast<float>(p);
    a.seed = seed;
    a.offset = offset;
}
struct QkvNode : Node {
    SavedVariable x, qkv, o, lse, bias, stack;   // stack: the weights, where the forward had to copy them together
    Tensor w[3], b[3], w_mg[3], b_mg[3];
    int64_t B = 0, S = 0, H = 0;
    double p = 0, scale = 1;
    uint64_t seed = 0, offset = 0;
    RB_NODE("RbQkvAttentionBackward")
    void release_variables() override {
        std::lock_guard<std::mutex> lock(mutex_);
        for (SavedVariable* s : {&x, &qkv, &o, &lse, &bias, &stack}) s->reset_data();
    }
    variable_list run(variable_list&& grads) {
        const Tensor X = x.unpack(), Q = qkv.unpack(), O = o.unpack(shared_from_this()), L = lse.unpack(), kb = bias.unpack();
        const Tensor dO = dense16(grads[0]);
        const int dt = dt_code(X);
        const int64_t Ho = H * 64;
        Tensor dqkv = at::empty(Q.sizes(), Q.options());
        Tensor delta = f32({B, H, S}, Q), dq_acc;
        RbAttnArgs a;
        attn_args(a, Q, O, L, kb, B, S, H, scale, p, seed, offset);
        a.dO = dO.data_ptr();
        a.do_sb = S * Ho;
        a.do_ss = Ho;
        a.do_sh = 64;
        char* d = static_cast<char*>(dqkv.data_ptr());
        a.dQ = d;
        a.dK = d + Ho * 2;
        a.dV = d + 2 * Ho * 2;
        a.dq_sb = a.dk_sb = a.dv_sb = S * 3 * Ho;
        a.dq_ss = a.dk_ss = a.dv_ss = 3 * Ho;
        a.dq_sh = a.dk_sh = a.dv_sh = 64;
        a.delta = mptr<float>(delta);
        const bool adds = api.attn_bwd_adds(&a);
        if (adds) dq_acc = f32({B, S, H, 64}, Q);
        a.dq_accum = mptr<float>(dq_acc);
        check(api.attn_bwd(&a, cur_stream()), "rb_attn_bwd", adds ? 3 : 2);
        Mat dm;
        dm.keep = dqkv;
        dm.p = d;
        dm.rows = B * S;
        dm.cols = dm.ld = 3 * Ho;
        const Mat xm = rows_of(X);
        Tensor dx, dw[3], db[3];
        if (task_should_compute_output(0)) {
            dx = at::empty(X.sizes(), X.options());
            const Tensor st = stack.unpack();
            bool copied;
            gemm(dm, st.defined() ? mat(st) : stacked(w, copied), false, false, dx.data_ptr(), false, dt, Epi());
        }
        // adjacent fp32 gradient buffers: one weight-gradient GEMM (with the column sums of the biases) serves all three
        // projections
        auto all = [](const Tensor* t) { return t[0].defined() && t[1].defined() && t[2].defined(); };
        const void* wm = all(w_mg) && w_mg[0].scalar_type() == at::kFloat ? adjacent(w_mg) : nullptr;
        const void* bm = b[0].defined() && all(b_mg) ? adjacent(b_mg) : nullptr;
        if (wm && (bm || !b[0].defined())) {
            Epi e;
            e.accumulate = true;
            e.a_colsum = static_cast<float*>(const_cast<void*>(bm));
            gemm(dm, xm, true, false, const_cast<void*>(wm), true, dt, e);
        } else if (!w_mg[0].defined() && !w_mg[1].defined() && !w_mg[2].defined() && !b_mg[0].defined() &&
                   !b_mg[1].defined() && !b_mg[2].defined()) {
            const auto gr = stacked_grads(dm, xm, w[0], b[0], dt);
            for (int i = 0; i < 3; ++i) dw[i] = gr[i].w, db[i] = gr[i].b;
        } else {
            for (int i = 0; i < 3; ++i) {
                const Grads gr = param_grads(columns(dm, i * Ho, Ho), xm, w[i], w_mg[i], true, b[i], b_mg[i], true, dt);
                dw[i] = gr.w;
                db[i] = gr.b;
            }
        }
        notify({{&w[0], &w_mg[0]}, {&w[1], &w_mg[1]}, {&w[2], &w_mg[2]},
                {&b[0], &b_mg[0]}, {&b[1], &b_mg[1]}, {&b[2], &b_mg[2]}});
        return {dx, dw[0], db[0], dw[1], db[1], dw[2], db[2]};
    }
};

// streamed: parameters that come and go; when they have to be stacked, the backward does it again instead of keeping the
// forward's copy on the device in between
Tensor qkv_attention(const Tensor& x, const std::vector<Tensor>& ws, const std::vector<OptTensor>& bs, const OptTensor& key_bias,
                     double p, double scale, int64_t H, uint64_t seed, uint64_t offset, const std::vector<OptTensor>& w_mgs,
                     const std::vector<OptTensor>& b_mgs, bool streamed) {
    TORCH_CHECK_VALUE(x.dim() == 3 && ws.size() == 3 && bs.size() == 3 && w_mgs.size() == 3 && b_mgs.size() == 3,
                      "qkv_attention: three-dimensional input, three projections");
    const Tensor w[3] = {ws[0], ws[1], ws[2]}, b[3] = {opt(bs[0]), opt(bs[1]), opt(bs[2])};
    same_type("qkv_attention", x, {&w[0], &w[1], &w[2], &b[0], &b[1], &b[2]});
    for (int i = 0; i < 3; ++i) {
        TORCH_CHECK_VALUE(w[i].dim() == 2 && w[i].sizes() == w[0].sizes() && w[0].size(0) == 64 * H &&
                              b[i].defined() == b[0].defined(),
                          "qkv_attention: three projections of one shape, 64 rows a head");
        length("qkv_attention bias", b[i], w[0].size(0));
    }
    const bool req = wants_grad({&x, &w[0], &b[0], &w[1], &b[1], &w[2], &b[2]});
    const int64_t B = x.size(0), S = x.size(1), Ho = w[0].size(0);
    Tensor xc, qkv, o, lse, bias_cat, kb = opt(key_bias);
    if (kb.defined()) {
        TORCH_CHECK_TYPE(kb.scalar_type() == at::kFloat && kb.device() == x.device(), "qkv_attention: the key bias is fp32");
        TORCH_CHECK_VALUE(kb.is_contiguous(), "qkv_attention: the key bias is contiguous");
        length("qkv_attention key bias", kb, B * S);
    }
    Mat wm;
    bool copied;
    {
        at::NoGradGuard off;
        xc = dense(x);
        qkv = at::empty({B, S, 3 * Ho}, x.options());
        o = at::empty({B, S, Ho}, x.options());
        lse = f32({B, H, S}, x);
        Epi e;
        if (b[0].defined()) {
            e.bias = adjacent(b);
            if (!e.bias) {
                bias_cat = at::cat({b[0].detach(), b[1].detach(), b[2].detach()}, 0);
                e.bias = bias_cat.data_ptr();
            }
        }
        wm = stacked(w, copied);
        gemm(rows_of(xc), wm, false, true, qkv.data_ptr(), false, dt_code(x), e);
        RbAttnArgs a;
        attn_args(a, qkv, o, lse, kb, B, S, H, scale, p, seed, offset);
        check(api.attn_fwd(&a, cur_stream()), "rb_attn_fwd");
    }
    if (req) {
        auto n = new_node<QkvNode>();
        n->set_next_edges(torch::autograd::collect_next_edges(x, w[0], b[0], w[1], b[1], w[2], b[2]));
        torch::autograd::set_history(o, n);
        n->x = SavedVariable(xc, false);
        n->qkv = SavedVariable(qkv, false);
        n->o = SavedVariable(o, true);
        n->lse = SavedVariable(lse, false);
        n->bias = SavedVariable(kb, false);
        for (int i = 0; i < 3; ++i) {
            n->w[i] = w[i];
            n->b[i] = b[i];
            n->w_mg[i] = weight_grad_buffer("qkv_attention", w_mgs[i], w[i]);
            n->b_mg[i] = grad_buffer("qkv_attention", b_mgs[i], b[i]);
        }
        if (copied && !streamed) n->stack = SavedVariable(wm.keep, false);
        n->B = B;
        n->S = S;
        n->H = H;
        n->p = p;
        n->scale = scale;
        n->seed = seed;
        n->offset = offset;
    }
    return o;
}

// ------------------------------------------------------------------------------------------------ batch norm
Tensor nhwc(const Tensor& t) {   // channels-last on a 16-byte boundary
    return t.is_contiguous(at::MemoryFormat::ChannelsLast) && aligned16(t.data_ptr()) ? t : t.clone(at::MemoryFormat::ChannelsLast);
}
// A 1x1 convolution: the linear layer over the pixels of a channels-last activation.  As that layer between views (the pixels
// of x, the filter as a matrix, the result as an image again) it was four autograd nodes, and 512 to 2048 channels at
// 32 x 14 x 14 with batch norm, forward and backward, were bound by the host: 164 -> 135 us.
Mat pixels(const Tensor& t) {
    Mat m;
    m.keep = t;
    m.p = t.data_ptr();
    m.cols = m.ld = t.size(1);
    m.rows = t.numel() / m.cols;
    return m;
}
Mat filter(const Tensor& w) {
    if (!aligned16(w.data_ptr()) || w.stride(1) != 1 || w.stride(0) % 8)
        return mat(w.detach().reshape({w.size(0), w.size(1)}));
    Mat m;
    m.keep = w;
    m.p = w.data_ptr();
    m.rows = w.size(0);
    m.cols = w.size(1);
    m.ld = w.stride(0);
    return m;
}
struct Conv1x1Node : Node {
    SavedVariable x, w;
    Tensor bias, w_ref, w_mg, b_mg;
    RB_NODE("RbConv1x1Backward")
    void release_variables() override {
        std::lock_guard<std::mutex> lock(mutex_);
        x.reset_data();
        w.reset_data();
    }
    variable_list run(variable_list&& grads) {
        const Tensor X = x.unpack(), W = w.unpack(), dy = nhwc(grads[0]);
        const int dt = dt_code(X);
        const Mat d = pixels(dy), wm = filter(W);
        Tensor dx;
        if (task_should_compute_output(0)) {
            dx = at::empty_like(X);
            gemm(d, wm, false, false, dx.data_ptr(), false, dt, Epi());
        }
        Grads gr = param_grads(d, pixels(X), W, w_mg, task_should_compute_output(1), bias, b_mg,
                               bias.defined() && task_should_compute_output(2), dt);
        if (gr.w.defined()) gr.w = gr.w.view(W.sizes());
        notify({{&w_ref, &w_mg}, {&bias, &b_mg}});
        return {dx, gr.w, gr.b};
    }
};
Tensor conv1x1(const Tensor& x, const Tensor& w, const OptTensor& bias_, const OptTensor& w_mg, const OptTensor& b_mg) {
    const Tensor bias = opt(bias_);
    same_type("conv1x1", x, {&w, &bias});
    TORCH_CHECK_VALUE(x.dim() == 4 && w.dim() == 4 && w.size(2) == 1 && w.size(3) == 1 && x.size(1) == w.size(1) &&
                          x.size(1) % 8 == 0 && w.size(0) % 8 == 0 && x.size(1) > 0,
                      "conv1x1: images and 1x1 filters of channels that are multiples of 8");
    length("conv1x1 bias", bias, w.size(0));
    const bool req = wants_grad({&x, &w, &bias});
    Tensor xc, y;
    {
        at::NoGradGuard off;
        xc = nhwc(x);
        y = at::empty({x.size(0), w.size(0), x.size(2), x.size(3)}, x.options(), at::MemoryFormat::ChannelsLast);
        const Tensor bc = dense(bias);
        Epi e;
        e.bias = cptr(bc);
        gemm(pixels(xc), filter(w), false, true, y.data_ptr(), false, dt_code(x), e);
    }
    if (req) {
        auto n = new_node<Conv1x1Node>();
        n->set_next_edges(torch::autograd::collect_next_edges(x, w, bias));
        n->x = SavedVariable(xc, false);
        n->w = SavedVariable(w, false);
        n->w_ref = w;
        n->bias = bias;
        const Tensor mg = opt(w_mg);
        if (mg.defined()) {
            TORCH_CHECK_VALUE(mg.numel() == w.numel(), "conv1x1: a filter's gradient buffer has the filter's size");
            n->w_mg = weight_grad_buffer("conv1x1", mg.view({w.size(0), w.size(1)}), w.detach().reshape({w.size(0), w.size(1)}));
        }
        n->b_mg = grad_buffer("conv1x1", b_mg, bias);
        torch::autograd::set_history(y, n);
    }
    return y;
}

struct BnNode : Node {
    SavedVariable x, y, mean, rstd, g32;
    Tensor gamma, beta, g_mg, b_mg;
    bool relu = false, has_res = false;
    RB_NODE("RbBatchNormBackward")
    void release_variables() override {
        std::lock_guard<std::mutex> lock(mutex_);
        for (SavedVariable* s : {&x, &y, &mean, &rstd, &g32}) s->reset_data();
    }
    variable_list run(variable_list&& grads) {
        const Tensor X = x.unpack(), Y = y.unpack(shared_from_this()), M = mean.unpack(), R = rstd.unpack(), G = g32.unpack();
        const Tensor dy = nhwc(grads[0]);
        const int64_t C = X.size(1);
        Tensor dx = at::empty_like(X), dres = has_res ? at::empty_like(X) : Tensor();
        Tensor part = f32({api.bn_part_floats(X.numel() / C, static_cast<int>(C))}, X);
        // fp32 gradient buffers take the sums inside the kernel
        auto acc = [](const Tensor& mg) {
            return mg.defined() && mg.scalar_type() == at::kFloat && mg.is_contiguous() ? mptr<float>(mg) : nullptr;
        };
        float *ga = acc(g_mg), *ba = acc(b_mg);
        check(api.bn_bwd(X.data_ptr(), dy.data_ptr(), Y.data_ptr(), mptr<float>(M), mptr<float>(R), mptr<float>(G),
                         mptr<float>(part), ga, ba, dx.data_ptr(), mptr(dres), X.numel() / C, static_cast<int>(C), relu ? 1 : 0,
                         dt_code(X), cur_stream()),
              "rb_bn_bwd", 3);
        Tensor dg, db;
        if (g_mg.defined()) {
            if (!ga) g_mg.add_(part.narrow(0, C, C));
        } else {
            dg = part.narrow(0, C, C).to(gamma.scalar_type());
        }
        if (b_mg.defined()) {
            if (!ba) b_mg.add_(part.narrow(0, 0, C));
        } else {
            db = part.narrow(0, 0, C).to(beta.scalar_type());
        }
        notify({{&gamma, &g_mg}, {&beta, &b_mg}});
        return {dx, dres, dg, db};
    }
};

Tensor batch_norm_act(const Tensor& x, const OptTensor& res_, const Tensor& gamma, const Tensor& beta,
                      const OptTensor& run_mean_, const OptTensor& run_var_, double momentum, double eps, bool relu,
                      const OptTensor& g_mg, const OptTensor& b_mg) {
    const Tensor res = opt(res_), run_mean = opt(run_mean_), run_var = opt(run_var_);
    same_type("batch_norm", x, {&res});
    TORCH_CHECK_VALUE(x.dim() == 4 && (!res.defined() || res.sizes() == x.sizes()),
                      "batch_norm: the residual's sizes differ from x's");
    for (const Tensor* t : {&gamma, &beta, &run_mean, &run_var}) length("batch_norm parameter", *t, x.size(1));
    const bool req = wants_grad({&x, &res, &gamma, &beta});
    Tensor xc, y, mean, rstd, g32;
    {
        at::NoGradGuard off;
        const int64_t C = x.size(1), R = x.numel() / C;
        xc = nhwc(x);
        const Tensor rc = res.defined() ? nhwc(res) : Tensor();
        g32 = dense(gamma.detach().to(at::kFloat));
        const Tensor b32 = dense(beta.detach().to(at::kFloat));
        auto fp32 = [](const Tensor& t) { return t.defined() && t.scalar_type() == at::kFloat && t.is_contiguous(); };
        const bool in_kernel = fp32(run_mean) && fp32(run_var);
        y = at::empty_like(xc);
        Tensor part = f32({api.bn_part_floats(R, static_cast<int>(C))}, x);
        mean = f32({C}, x);
        rstd = f32({C}, x);
        check(api.bn_fwd(xc.data_ptr(), cptr(rc), mptr<float>(g32), mptr<float>(b32), y.data_ptr(), mptr<float>(part),
                         mptr<float>(mean), mptr<float>(rstd), in_kernel ? mptr<float>(run_mean) : nullptr,
                         in_kernel ? mptr<float>(run_var) : nullptr, R, static_cast<int>(C), static_cast<float>(eps),
                         static_cast<float>(momentum), relu ? 1 : 0, dt_code(x), cur_stream()),
              "rb_bn_fwd", 3);
        if (run_mean.defined() && !in_kernel) {
            // statistics kept in 16 bits, or strided: update them with a few tiny element-wise operations
            const Tensor var = (1.0 / (rstd * rstd) - eps) * (static_cast<double>(R) / std::max<int64_t>(R - 1, 1));
            run_mean.mul_(1 - momentum).add_((momentum * mean).to(run_mean.scalar_type()));
            run_var.mul_(1 - momentum).add_((momentum * var).to(run_var.scalar_type()));
        }
    }
    if (req) {
        auto n = new_node<BnNode>();
        n->set_next_edges(torch::autograd::collect_next_edges(x, res, gamma, beta));
        torch::autograd::set_history(y, n);
        n->x = SavedVariable(xc, false);
        n->y = SavedVariable(y, true);
        n->mean = SavedVariable(mean, false);
        n->rstd = SavedVariable(rstd, false);
        n->g32 = SavedVariable(g32, false);
        n->gamma = gamma;
        n->beta = beta;
        n->g_mg = opt(g_mg);
        n->b_mg = opt(b_mg);
        n->relu = relu;
        n->has_res = res.defined();
    }
    return y;
}

// ------------------------------------------------------------------------------------------------ plain products
// out = epilogue(alpha op(a) op(b)) for 2-D operands
Tensor product(const Tensor& a, const Tensor& b, bool trans_a, bool trans_b, const OptTensor& bias, const OptTensor& residual,
               const OptTensor& aux_in, const OptTensor& aux_out, bool gelu, bool dgelu, const OptTensor& out_, bool accumulate,
               bool fp32_out, double alpha, int64_t max_ctas) {
    at::NoGradGuard off;
    const Mat A = mat(a), B = mat(b);
    RbGemmArgs g;
    memset(&g, 0, sizeof(g));
    g.M = trans_a ? A.cols : A.rows;
    g.K = trans_a ? A.rows : A.cols;
    g.N = trans_b ? B.rows : B.cols;
    const int64_t kb = trans_b ? B.cols : B.rows;
    TORCH_CHECK_VALUE(kb == g.K, "gemm: inner dimensions differ (", g.K, " vs ", kb, ")");
    Tensor out = out_.has_value() ? *out_ : at::empty({g.M, g.N}, fp32_out ? a.options().dtype(at::kFloat) : a.options());
    const Tensor bv = dense(opt(bias)), rv = opt(residual), ai = opt(aux_in), ao = opt(aux_out);
    same_type("gemm", a, {&b, &bv, &rv, &ai, &ao});
    length("gemm bias", bv, g.N);
    TORCH_CHECK_TYPE(out.scalar_type() == (fp32_out ? at::kFloat : a.scalar_type()) && out.device() == a.device(),
                     "gemm: the output is of the operands' type or fp32, on their device");
    // the matrices beside the output share its row stride
    for (const Tensor* t : {static_cast<const Tensor*>(&out), &rv, &ai, &ao})
        TORCH_CHECK_VALUE(!t->defined() || (t->dim() == 2 && t->size(0) == g.M && t->size(1) == g.N &&
                                            (g.N <= 1 || t->stride(1) == 1) && (g.M <= 1 || t->stride(0) == out.stride(0))),
                          "gemm: the output and the matrices beside it are [", g.M, ", ", g.N, "] with one row stride");
    g.A = A.p;
    g.B = B.p;
    g.D = out.data_ptr();
    g.bias = cptr(bv);
    g.residual = cptr(rv);
    g.aux_in = cptr(ai);
    g.aux_out = mptr(ao);
    g.batch = 1;
    g.lda = A.ld;
    g.ldb = B.ld;
    g.ldd = out.stride(-2);
    g.a_major = trans_a ? 1 : 0;
    g.b_major = trans_b ? 0 : 1;
    g.in_dtype = dt_code(a);
    g.out_dtype = fp32_out ? 1 : 0;
    g.flags = (g.bias ? RB_GEMM_BIAS : 0) | (gelu ? RB_GEMM_GELU : 0) | (dgelu ? RB_GEMM_DGELU : 0) |
              (g.residual ? RB_GEMM_RESIDUAL : 0) | (accumulate ? RB_GEMM_ACCUM : 0) | (g.aux_out ? RB_GEMM_AUX_OUT : 0);
    g.alpha = static_cast<float>(alpha);
    g.max_ctas = static_cast<int32_t>(max_ctas);
    g.in_order = at::globalContext().deterministicAlgorithms() ? 1 : 0;
    check(api.gemm(&g, cur_stream()), "rb_gemm");
    return out;
}

// ------------------------------------------------------------------------------------------------ bindings
void init(const std::unordered_map<std::string, uintptr_t>& fns, py::object error) {
    auto set = [&](auto& slot, const char* name) {
        slot = reinterpret_cast<std::remove_reference_t<decltype(slot)>>(fns.at(name));
    };
    set(api.gemm, "rb_gemm");
    set(api.gemm_splits, "rb_gemm_splits");
    set(api.unstack3, "rb_unstack3");
    set(api.gelu, "rb_gelu");
    set(api.colsum, "rb_colsum");
    set(api.ln_fwd, "rb_ln_fwd");
    set(api.ln_bwd, "rb_ln_bwd");
    set(api.ln_bwd16, "rb_ln_bwd16");
    set(api.ln_bwd_grid, "rb_ln_bwd_grid");
    set(api.embed_fwd, "rb_embed_fwd");
    set(api.embed_bwd, "rb_embed_bwd");
    set(api.xent_fwd, "rb_xent_fwd");
    set(api.xent_bwd, "rb_xent_bwd");
    set(api.attn_fwd, "rb_attn_fwd");
    set(api.attn_bwd, "rb_attn_bwd");
    set(api.attn_bwd_adds, "rb_attn_bwd_adds");
    set(api.bn_fwd, "rb_bn_fwd");
    set(api.bn_bwd, "rb_bn_bwd");
    set(api.bn_part_floats, "rb_bn_part_floats");
    set(api.gemm_pairs, "rb_gemm_pairs");
    set(api.rows_plan, "rb_rows_plan");
    set(api.rows_gather, "rb_rows_gather");
    set(api.rows_scatter, "rb_rows_scatter_parts");
    error_class = error.release().ptr();
}
void set_listener(py::object fn) {
    Py_XDECREF(listener);
    listener = fn.is_none() ? nullptr : fn.release().ptr();
    has_listener.store(listener != nullptr, std::memory_order_release);
}

// Errors cross the boundary as the exceptions they are (the library's own error class, ValueError, TypeError, ...).  The
// interpreter lock is released meanwhile, as PyTorch's own operators do it: an allocation that has to wait, or a launch
// into a full queue, must not stop the other Python threads.  (What needs the interpreter takes the lock itself: errors,
// gradient listeners, saved-tensor hooks.)
template <typename F>
struct Guarded;
template <typename R, typename... A>
struct Guarded<R (*)(A...)> {
    template <R (*F)(A...)>
    static R call(A... a) {
        R result{};
        auto body = [&]() -> bool {
            HANDLE_TH_ERRORS
            py::gil_scoped_release unlocked;
            result = F(std::forward<A>(a)...);
            return true;
            END_HANDLE_TH_ERRORS_RET(false)
        };
        if (!body()) throw py::error_already_set();
        return result;
    }
};
#define RB_DEF(NAME) m.def(#NAME, &Guarded<decltype(&NAME)>::call<&NAME>)

}  // namespace

PYBIND11_MODULE(_host, m) {
    m.doc() = "Host side of the fused operators";
    m.def("init", &init);
    m.def("set_listener", &set_listener);
    m.def("launch_count", [] { return launches.load(std::memory_order_relaxed); });
    RB_DEF(product);
    RB_DEF(linear);
    RB_DEF(mlp);
    RB_DEF(layer_norm);
    RB_DEF(embedding);
    RB_DEF(cross_entropy);
    RB_DEF(qkv_attention);
    RB_DEF(batch_norm_act);
    RB_DEF(conv1x1);
    m.def("gather_room", py::overload_cast<int64_t, int64_t, int64_t, int64_t, int64_t>(&gather_room));
}
