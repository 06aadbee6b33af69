// Host path of the hot operators: argument checks, output and workspace allocation, the C-ABI
// calls and the autograd nodes of the convolution and the ragged layer norm, compiled.
//
// The kernels live behind the C ABI (include/pointelligence_b200.h).  What this file replaces is the
// interpreter between a layer's forward() and those entry points: a training pass of one layer
// through Python operators, Python autograd and ctypes marshalling cost 0.5-0.6 ms of host time on
// B200 boxes (150 000 points, 64 channels: 0.54 ms per pass for 0.29 ms of kernels); small layers and
// whole networks on small scenes were bound by it.  The policy that needs Python objects -- which
// engine a rulebook takes, the plans remembered per rulebook -- stays in Python and is asked through
// two hooks (set_hooks), once per convolution pass.
#include <torch/csrc/autograd/custom_function.h>
#include <torch/extension.h>

#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/CUDAEvent.h>
#include <c10/cuda/CUDAGuard.h>

#include "../../include/pointelligence_b200.h"

namespace py = pybind11;
using at::Tensor;
using OptTensor = std::optional<Tensor>;

namespace {

// ------------------------------------------------------------------ helpers ----
PyObject *g_plan_hook = nullptr;       // (scatter, gather, seg, K, n_out, out_width, in_width, forced, split, capturing) -> None | plan tuple
PyObject *g_symmetric_hook = nullptr;  // (i, j, K) -> bool
PyObject *g_ascending_hook = nullptr;  // (scatter, gather, seg, K) -> bool: rows are known to ascend inside every tap
PyObject *g_fullest_hook = nullptr;    // (index, index, seg, K) -> triplets of the fullest tap, or None
PyObject *g_double_backward = nullptr; // differentiable backward of the convolution (create_graph)

[[noreturn]] void raise(PyObject *type, const std::string &msg) {
    PyErr_SetString(type, msg.c_str());
    throw py::error_already_set();
}

// C-ABI status -> the exception type the ctypes binding raises for it
void check(int rc) {
    if (rc == PCX_OK) return;
    PyObject *type = PyExc_RuntimeError;
    if (rc == PCX_E_ARG || rc == PCX_E_ALIGN) type = PyExc_ValueError;
    else if (rc == PCX_E_DTYPE) type = PyExc_TypeError;
    else if (rc == PCX_E_UNSUPPORTED) type = PyExc_NotImplementedError;
    const std::string msg = std::string(pcx_last_error_string()) + " [pcx status " + std::to_string(rc) + "]";
    py::gil_scoped_acquire gil;
    raise(type, msg);
}

void require_cuda(const Tensor &t) {
    if (t.defined() && !t.is_cuda()) {
        py::gil_scoped_acquire gil;
        raise(PyExc_RuntimeError, "pointelligence_b200 operators run on CUDA tensors only (no CPU fallback); got a tensor on " +
                                      t.device().str());
    }
}
void require_cuda(const OptTensor &t) {
    if (t) require_cuda(*t);
}

// `message` makes the text, once it is needed
template <typename F>
void require(bool ok, PyObject *type, F message) {
    if (ok) return;
    py::gil_scoped_acquire gil;
    raise(type, message());
}
std::string str(at::IntArrayRef sizes) {
    std::ostringstream s;
    s << sizes;
    return s.str();
}

int dtype_code(at::ScalarType t) {
    switch (t) {
        case at::kFloat: return PCX_F32;
        case at::kHalf: return PCX_F16;
        case at::kBFloat16: return PCX_BF16;
        default: break;
    }
    py::gil_scoped_acquire gil;
    raise(PyExc_TypeError, std::string("unsupported feature dtype torch.") + c10::toString(t) +
                               "; expected float32, float16 or bfloat16");
}

Tensor as_i32(const Tensor &t) { return t.scalar_type() == at::kInt ? t.contiguous() : t.to(at::kInt).contiguous(); }
Tensor as_i64(const Tensor &t) { return t.scalar_type() == at::kLong ? t.contiguous() : t.to(at::kLong).contiguous(); }

Tensor workspace(size_t bytes, const Tensor &like) {
    return at::empty({(int64_t)std::max<size_t>(bytes, 256)}, at::TensorOptions().dtype(at::kByte).device(like.device()));
}
void *stream() { return (void *)at::cuda::getCurrentCUDAStream().stream(); }
void *ptr(const Tensor &t) { return t.defined() ? t.data_ptr() : nullptr; }
template <typename T>
T *ptr_as(const Tensor &t) { return t.defined() ? static_cast<T *>(t.data_ptr()) : nullptr; }

// --------------------------------------------------------------------- MVMR ----
// Plan of the output-stationary kernel as the hook returns it.
struct Plan {
    Tensor buffer;
    int64_t group = 0, multi = 0;
    bool valid = false;
};

Plan ask_plan(const Tensor &scatter, const Tensor &gather, const Tensor &seg, int64_t K, int64_t n_out, int64_t outw,
              int64_t inw, bool forced, bool split, bool capturing) {
    Plan plan;
    py::gil_scoped_acquire gil;
    py::object r = py::reinterpret_borrow<py::object>(g_plan_hook)(scatter, gather, seg, K, n_out, outw, inw, forced, split, capturing);
    if (!r.is_none()) {
        py::tuple t = py::cast<py::tuple>(r);
        plan.buffer = py::cast<Tensor>(t[0]);
        plan.group = py::cast<int64_t>(t[1]);
        plan.multi = py::cast<int64_t>(t[2]);
        plan.valid = true;
    }
    return plan;
}

// Channels the tensor engines work on for a row of `width`: parts of at most 256 channels, multiples of 16.
int64_t padded(int64_t width) {
    const int64_t unit = 16 * ((width + 255) / 256);
    return (width + unit - 1) / unit * unit;
}
bool is_half(at::ScalarType t) { return t == at::kHalf || t == at::kBFloat16; }

// `outer` matrices (rows x cols) of 16-bit elements in another shape, zeros where the source has nothing
Tensor reshape16(const Tensor &src, int64_t outer, int64_t rows, int64_t cols, int64_t rows_out, int64_t cols_out, at::IntArrayRef shape) {
    Tensor dst = at::empty(shape, src.options());
    check(pcx_reshape16(ptr(src), ptr(dst), outer, (int)rows, (int)cols, (int)rows_out, (int)cols_out, stream()));
    return dst;
}

// Shapes and types the output-stationary kernel takes (16-bit elements, widths in sixteens).
bool plan_fits(at::ScalarType dtype, int64_t T, int64_t n_out, int64_t K, int64_t G, int64_t inw, int64_t outw, bool has_seg) {
    if (!has_seg || !is_half(dtype) || n_out <= 0) return false;
    if (inw != padded(inw) || outw != padded(outw) || inw > 1024 || G * inw > 2048 || K > 512 || G * ((outw + 255) / 256) > 64) return false;
    const int64_t nblocks = (n_out + 127) / 128;
    return T < (int64_t(1) << 31) && nblocks * K * 128 <= (int64_t(1) << 32);
}

constexpr int ENGINE_PLANNED = 3;
constexpr int64_t NO_PLAN = 0x200;   // internal flag of an engine: the automatic choice is between the scatter engines
// ... and of the automatic choice: a layer of widths that have to be padded takes the engines of the padded widths, the
// output-stationary kernel included (the caller's operands are bf16 copies, whose sums it may round)
constexpr int64_t PLAN_PADDED = 0x400;

// Shapes the automatic choice may give to the output-stationary kernel.  It rounds the sums of (row, tap) buckets to 16
// bits; grouped, padded and wider layers multiply their operands as they are unless the caller asks for that kernel.
bool plan_unasked(int64_t K, int64_t G, int64_t outw) { return K > 1 && G == 1 && outw <= 256; }
// ... and those it may be given with the sums in two parts (bf16: as exact as the scatter kernels once a row is rounded; in
// fp16 a sum could leave the type's range, which the scatter kernels' products do not).  The scatter kernels have to take
// them too: they follow where an operand is not finite.
bool plan_split(at::ScalarType dtype, int64_t K, int64_t G, int64_t inw, int64_t outw) {
    return K > 1 && (G > 1 || outw > 256) && dtype == at::kBFloat16 && G * ((inw + 255) / 256) * ((outw + 255) / 256) <= 64;
}
constexpr int SPLIT_SUMS = PCX_MVMR_SPLIT_SUMS;

Tensor mvmr_planned(const Tensor &weight, const Tensor &feat, const Plan &plan, int64_t T, int64_t n_out, int flags,
                    const Tensor &bias) {
    const int64_t K = weight.size(0), G = weight.size(1), C = weight.size(2), M = weight.size(3);
    const bool transpose = flags & 1;
    const int64_t inw = transpose ? M : C, outw = transpose ? C : M;
    Tensor out = at::empty({n_out, G * outw}, feat.options());
    const size_t bytes = pcx_mvmr_planned_scratch_bytes(plan.multi, (int)inw * (flags & SPLIT_SUMS ? 2 : 1), n_out, (int)outw, (int)K, (int)G);
    Tensor ws = workspace(bytes, feat);
    check(pcx_mvmr_planned_bias(ptr(weight), ptr(feat), ptr(plan.buffer), plan.buffer.numel(), ptr(bias), ptr(out), T, feat.size(0),
                                n_out, (int)K, (int)G, (int)C, (int)M, flags, dtype_code(feat.scalar_type()), (int)plan.group, plan.multi,
                                ptr(ws), ws.numel(), stream()));
    return out;
}

// (undefined where the device has no room for its scratch)
Tensor mvmr_split(const Tensor &weight, const Tensor &feat, const Tensor &gather_, const Tensor &scatter_, const Tensor &seg_,
                  const Plan &plan, int64_t n_out, int flags, const Tensor &bias) {
    const int64_t K = weight.size(0), G = weight.size(1), C = weight.size(2), M = weight.size(3);
    const int transpose = flags & 1;
    const Tensor gather = as_i32(gather_), scatter = as_i32(scatter_), seg = as_i64(seg_);
    Tensor out = at::empty({n_out, G * (transpose ? C : M)}, feat.options());
    Tensor ws;
    try {
        ws = workspace(pcx_mvmr_split_workspace_bytes(plan.multi, n_out, (int)K, (int)G, (int)C, (int)M, transpose), feat);
    } catch (const c10::OutOfMemoryError &) {
        return Tensor();
    }
    check(pcx_mvmr_split(ptr(weight), ptr(feat), ptr_as<int32_t>(gather), ptr_as<int32_t>(scatter), ptr_as<int64_t>(seg), ptr(plan.buffer),
                         plan.buffer.numel(), ptr(bias), ptr(out), gather.numel(), feat.size(0), n_out, (int)K, (int)G, (int)C, (int)M,
                         flags, (int)plan.group, plan.multi, ptr(ws), ws.numel(), stream()));
    return out;
}

// Layers of up to 8 channels of the contraction on rulebooks of the geometry path (pcx_mvmr_thin: rows known to ascend
// inside every tap).  That kernel takes its steps one after the other, a microsecond each, in up to 444 blocks at once: for every tile
// of 128 rows x 64 output channels and every eight taps as many as the fullest (row, tap) has triplets, up to eight, of which only the
// average over all is known here.  The scatter kernel adds fp32 sums at a steady rate, the faster one for rows of 64 channels.  The two
// lines below are fitted to 760 calls (rooms, sweeps, uniform clouds of 300 to 400 000 points, 2 to 250 triplets a row, 27 and
// 125 taps, 16 to 256 output channels): the choice is 2.4 % slower than the better of the two (geometric mean), 18 % faster than the
// scatter kernel alone, and more than 10 % slower than that in 14 of them (sweeps, whose points crowd: at worst 198 us for 122).
// Until there was a term for steps and for blocks that are too few, it was 25 % slower than the better one.  us, scatter / this:
//
//   27 taps    1000 points, 40 a row     -> 64   21 / 37    10 000, 40  -> 64   38 / 65     60 000, 15  -> 64   68 / 55
//             100 000, 40                -> 32  199 / 100   200 000, 6  -> 128  225 / 110
//   125 taps   30 000, 80                -> 32  121 / 75    100 000, 30 -> 32  144 / 114    200 000, 5   -> 32   63 / 129
//
// A layer that may round sums (`or_planned`) would get a plan of a dense rulebook instead of the scatter kernel: that takes 150 us and
// more, for a rulebook that is mostly used once.  Only where most (row, tap) hold several triplets is it left to the plan, which adds
// them up beforehand (32 000 points of a sweep with 124 triplets a row, 8 -> 256 channels: 49 us a pass on a plan, 240 here).
bool thin_pays(at::ScalarType dtype, int64_t T, int64_t n_in, int64_t n_out, int64_t K, int64_t G, int64_t inw, int64_t outw, bool or_planned) {
    if (!is_half(dtype) || G != 1 || K <= 1 || K > 512 || inw <= 0 || inw > 8 || outw <= 0 || outw > 1024 || T <= 0 || T >= (int64_t(1) << 27) - 1 ||
        n_in <= 0 || n_out <= 0)
        return false;
    const int64_t tiles = (n_out + 127) / 128, parts = (outw + 63) / 64, eights = (K + 7) / 8, width = (outw + 15) / 16 * 16;
    if (tiles * eights * parts >= int64_t(1) << 31) return false;
    const double triplets = 1e-6 * (double)T, a_cell = (double)T / ((double)n_out * (double)K);
    if (or_planned && T >= 12 * n_out && a_cell >= 0.18) return a_cell < 1.;
    const double thin = 30. + 17.3 * triplets + 0.14 * 512e-6 * (double)(tiles * K) +
                        1.06 * std::max(1., (double)(tiles * parts) / 444.) * (double)eights * std::min(8., 1.3 + 2.05 * a_cell);
    const double a_triplet = width == 64 ? 53. : width <= 32 ? 2.6 + 1.3 * (double)width : 1.35 * (double)width - 4.;
    return thin < 17. + a_triplet * triplets + (width > 32 ? 1e-6 * (double)(n_out * width) : 0.);
}
bool rows_ascend(const Tensor &scatter, const Tensor &gather, const Tensor &seg, int64_t K) {
    py::gil_scoped_acquire gil;
    return py::cast<bool>(py::reinterpret_borrow<py::object>(g_ascending_hook)(scatter, gather, seg, K));
}

// (undefined where its table, a number for every row and tap, is beyond 4 GB or finds no room: the scatter kernels need less)
constexpr size_t THIN_MAX_SCRATCH = size_t(4) << 30;
Tensor mvmr_thin(const Tensor &weight, const Tensor &feat, const Tensor &gather_, const Tensor &scatter_, const Tensor &seg_, int64_t n_out,
                 int flags, const Tensor &bias) {
    const int64_t K = weight.size(0), C = weight.size(2), M = weight.size(3), T = gather_.numel();
    const int transpose = flags & 1;
    // (a sum of triplets, 48 bytes, is made of nine or more)
    const size_t bytes = pcx_mvmr_thin_workspace_bytes(feat.size(0), n_out, (int)K, (int)C, (int)M, transpose) + 48 * std::max<int64_t>(T / 9 - n_out, 0);
    if (bytes > THIN_MAX_SCRATCH) return Tensor();
    Tensor ws;
    try {
        ws = workspace(bytes, feat);
    } catch (const c10::OutOfMemoryError &) {
        return Tensor();
    }
    const Tensor gather = as_i32(gather_), scatter = as_i32(scatter_), seg = as_i64(seg_);
    Tensor out = at::empty({n_out, transpose ? C : M}, feat.options());
    check(pcx_mvmr_thin(ptr(weight), ptr(feat), ptr_as<int32_t>(gather), ptr_as<int32_t>(scatter), ptr_as<int64_t>(seg), ptr(bias), ptr(out), T,
                        feat.size(0), n_out, (int)K, (int)C, (int)M, flags, dtype_code(feat.scalar_type()), ptr(ws), ws.numel(), stream()));
    return out;
}

// out[scatter[t]] += feat[gather[t]] @ W[tap(t)] (+ bias).  flags: 1 = W transposed, 2 = taps of the weight
// in reverse order.  Rows of the result are (G * out width) in feat's type.
Tensor mvmr_impl(Tensor weight, Tensor feat, const Tensor &gather_, const Tensor &scatter_, const OptTensor &seg_,
                 const OptTensor &tap_, int64_t n_out, int flags, int64_t engine, const Tensor &bias) {
    require_cuda(weight), require_cuda(feat), require_cuda(gather_), require_cuda(scatter_);
    require_cuda(seg_), require_cuda(tap_);
    const int code = dtype_code(feat.scalar_type());
    require(weight.dim() == 4, PyExc_ValueError,
            [&] { return "expected a weight (taps, groups, inputs, outputs), got " + str(weight.sizes()); });
    require(weight.scalar_type() == feat.scalar_type(), PyExc_AssertionError, [] { return std::string("weight and features differ in type"); });
    weight = weight.contiguous(), feat = feat.contiguous();
    const int64_t K = weight.size(0), G = weight.size(1), C = weight.size(2), M = weight.size(3);
    const bool transpose = flags & 1;
    const int64_t inw = transpose ? M : C, outw = transpose ? C : M, T = gather_.numel();
    c10::cuda::CUDAGuard guard(feat.device());
    const bool plan_padded = engine & PLAN_PADDED && padded(C) == (C + 15) / 16 * 16 && padded(M) == (M + 15) / 16 * 16;
    engine &= ~PLAN_PADDED;
    if (engine == 0 && seg_ && thin_pays(feat.scalar_type(), T, feat.size(0), n_out, K, G, inw, outw, plan_padded) &&
        // (a captured pass is replayed on whatever the index tensors hold then: on the kernels that take any order)
        c10::cuda::currentStreamCaptureStatusMayInitCtx() == c10::cuda::CaptureStatus::None && rows_ascend(scatter_, gather_, *seg_, K)) {
        const Tensor y = mvmr_thin(weight, feat, gather_, scatter_, *seg_, n_out, flags, bias);
        if (y.defined()) return y;
    }
    if ((engine & 0xff) == 0 && is_half(feat.scalar_type()) && seg_ && T > 0 && n_out > 0 && K <= 1024 && G <= 64 &&
        (C != padded(C) || M != padded(M))) {
        // channel counts the tensor engines do not take (the 3 or 6 channels of an input, 20 classes): zero columns make
        // them up.  60 000 points, 420 000 triplets, forward here / on the CUDA-core engine: 6 -> 32 42 / 56 us, 20 -> 20
        // 52 / 66, 8 groups of 8 129 / 317, 64 groups of 1 1207 / 2474 (these take sixteen times the memory of their rows,
        // 471 MB); 2000 points: 20 / 19, 26 / 19, 32 / 28, 55 / 96
        const int64_t Cp = padded(C), Mp = padded(M), inp = transpose ? Mp : Cp, outp = transpose ? Cp : Mp;
        const Tensor w = reshape16(weight, K * G, C, M, Cp, Mp, {K, G, Cp, Mp});
        const Tensor x = inp == inw ? feat : reshape16(feat, feat.size(0) * G, 1, inw, 1, inp, {feat.size(0), G * inp});
        const Tensor b = !bias.defined() || outp == outw ? bias : reshape16(bias, G, 1, outw, 1, outp, {G * outp});
        const Tensor y = mvmr_impl(w, x, gather_, scatter_, seg_, tap_, n_out, flags, plan_padded ? engine : engine | NO_PLAN, b);
        return outp == outw ? y : reshape16(y, n_out * G, 1, outp, 1, outw, {n_out, G * outw});
    }
    if (engine == 0 || engine == ENGINE_PLANNED) {
        const bool fits = plan_fits(feat.scalar_type(), T, n_out, K, G, inw, outw, seg_.has_value());
        if (engine == ENGINE_PLANNED && !fits) {
            py::gil_scoped_acquire gil;
            raise(PyExc_NotImplementedError,
                  "the output-stationary engine needs fp16/bf16 features, tap-sorted triplets of at most 512 taps, channel "
                  "counts that are multiples of 16 (of 32 beyond 256, of 48 beyond 512 ...) and at most 1024 input "
                  "channels a group");
        }
        const bool aligned = ((uintptr_t)ptr(weight) | (uintptr_t)ptr(feat)) % 16 == 0;   // else the CUDA-core engine
        const bool forced = engine == ENGINE_PLANNED, split = !forced && plan_split(feat.scalar_type(), K, G, inw, outw);
        if (fits && (forced || (aligned && (split || plan_unasked(K, G, outw))))) {
            const bool capturing = c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None;
            const Plan plan = ask_plan(scatter_, gather_, *seg_, K, n_out, G * outw, G * inw, forced, split, capturing);
            if (plan.valid && !split) return mvmr_planned(weight, feat, plan, T, n_out, flags, bias);
            if (plan.valid) {
                const Tensor out = mvmr_split(weight, feat, gather_, scatter_, *seg_, plan, n_out, flags, bias);
                if (out.defined()) return out;
            }
        }
        engine = 0;
    }
    engine &= ~NO_PLAN;
    const Tensor gather = as_i32(gather_), scatter = as_i32(scatter_);
    const Tensor tap = tap_ ? as_i32(*tap_) : Tensor(), seg = seg_ ? as_i64(*seg_) : Tensor();
    Tensor out = at::empty({n_out, G * outw}, feat.options());
    Tensor ws = workspace(pcx_mvmr_workspace_bytes(n_out, (int)K, (int)G, (int)C, (int)M, transpose, code), feat);
    check(pcx_mvmr_bias(ptr(weight), ptr(feat), ptr_as<int32_t>(gather), ptr_as<int32_t>(scatter), ptr_as<int64_t>(seg),
                        ptr_as<int32_t>(tap), ptr(bias), ptr(out), T, feat.size(0), n_out, (int)K, (int)G, (int)C, (int)M, flags,
                        code, (int)engine, ptr(ws), ws.numel(), stream()));
    return out;
}

Tensor mvmr(const Tensor &weight, const Tensor &feat, const Tensor &gather, const Tensor &scatter, const OptTensor &seg,
            const OptTensor &tap, int64_t n_out, bool transpose, int64_t engine) {
    return mvmr_impl(weight, feat, gather, scatter, seg, tap, n_out, transpose ? 1 : 0, engine, Tensor());
}

// --------------------------------------------------------------------- VVOR ----
// Triplets of the fullest tap where that decides the kernel and a search has counted them, else -1.
int64_t fullest_tap(const Tensor &a_idx, const Tensor &b_idx, const Tensor &seg, int64_t n_o, int64_t G, int64_t Ma, int64_t Cb) {
    const int64_t T = a_idx.numel(), limit = pcx_vvor_store_limit(n_o, (int)G, (int)Ma, (int)Cb);
    if (T <= limit || n_o <= 0 || T / n_o > limit) return -1;   // (stored, or summed, whatever it is)
    py::gil_scoped_acquire gil;
    py::object n = py::reinterpret_borrow<py::object>(g_fullest_hook)(a_idx, b_idx, seg, n_o);
    return n.is_none() ? -1 : py::cast<int64_t>(n);
}

Tensor vvor(Tensor a, const Tensor &a_idx_, Tensor b, const Tensor &b_idx_, const OptTensor &seg_, const OptTensor &o_idx_,
            int64_t n_o, int64_t engine) {
    require_cuda(a), require_cuda(b), require_cuda(a_idx_), require_cuda(b_idx_), require_cuda(seg_), require_cuda(o_idx_);
    const int code = dtype_code(a.scalar_type());
    require(a.scalar_type() == b.scalar_type(), PyExc_AssertionError, [] { return std::string("operands differ in type"); });
    a = a.contiguous(), b = b.contiguous();
    const int64_t G = a.size(1), Ma = a.size(2), Cb = b.size(2);
    c10::cuda::CUDAGuard guard(a.device());
    if (engine == 0 && is_half(a.scalar_type()) && seg_ && a_idx_.numel() > 0 && n_o <= 1024 && G <= 64 &&
        (Ma != padded(Ma) || Cb != padded(Cb))) {
        const int64_t Mp = padded(Ma), Cp = padded(Cb);
        const Tensor ap = Mp == Ma ? a : reshape16(a, a.size(0) * G, 1, Ma, 1, Mp, {a.size(0), G, Mp});
        const Tensor bp = Cp == Cb ? b : reshape16(b, b.size(0) * G, 1, Cb, 1, Cp, {b.size(0), G, Cp});
        return reshape16(vvor(ap, a_idx_, bp, b_idx_, seg_, o_idx_, n_o, engine), n_o * G, Mp, Cp, Ma, Cb, {n_o, G, Ma, Cb});
    }
    const Tensor a_idx = as_i32(a_idx_), b_idx = as_i32(b_idx_), o_idx = o_idx_ ? as_i32(*o_idx_) : Tensor(),
                 seg = seg_ ? as_i64(*seg_) : Tensor();
    Tensor out = at::empty({n_o, G, Ma, Cb}, a.options());
    Tensor ws = workspace(pcx_vvor_workspace_bytes(n_o, (int)G, (int)Ma, (int)Cb, code), a);
    const int64_t fullest = engine != 1 && is_half(a.scalar_type()) && seg_ ? fullest_tap(a_idx_, b_idx_, *seg_, n_o, G, Ma, Cb) : -1;
    check(pcx_vvor_known(ptr(a), ptr_as<int32_t>(a_idx), ptr(b), ptr_as<int32_t>(b_idx), ptr_as<int64_t>(seg), ptr_as<int32_t>(o_idx),
                         ptr(out), a_idx.numel(), a.size(0), b.size(0), n_o, (int)G, (int)Ma, (int)Cb, code, (int)engine, fullest, ptr(ws),
                         ws.numel(), stream()));
    return out;
}

Tensor column_sums(const Tensor &x_) {
    const Tensor x = x_.contiguous();
    c10::cuda::CUDAGuard guard(x.device());
    const int64_t N = x.size(0), C = x.size(1);
    Tensor out = at::empty({C}, x.options());
    Tensor ws = workspace(pcx_column_sums_workspace_bytes(N, (int)C), x);
    check(pcx_column_sums(ptr(x), ptr(out), N, (int)C, dtype_code(x.scalar_type()), ptr(ws), ws.numel(), stream()));
    return out;
}

// ------------------------------------------------------- convolution (autograd) ----
std::atomic<int> g_engine{0};   // engine of the current dispatch mode (0 automatic, 1 CUDA cores)

constexpr int64_t FAN_IN_ONE = PCX_ENGINE_FLAG_FAN_IN_ONE;

bool is_symmetric(const Tensor &i, const Tensor &j, int64_t K) {
    py::gil_scoped_acquire gil;
    return py::cast<bool>(py::reinterpret_borrow<py::object>(g_symmetric_hook)(i, j, K));
}

void match(Tensor &w, Tensor &x) {
    if (w.scalar_type() == x.scalar_type()) return;
    const auto t = c10::promoteTypes(w.scalar_type(), x.scalar_type());
    w = w.to(t), x = x.to(t);
}

struct ConvSizes {
    int64_t n_out, n_in, K;
    bool cover_out, cover_in, plan_padded;
    int64_t engine() const { return plan_padded && g_engine == 0 ? PLAN_PADDED : (int64_t)g_engine; }
};

Tensor as4(const Tensor &w) { return w.dim() == 4 ? w : w.unsqueeze(1); }

Tensor conv_forward(const Tensor &weight, const Tensor &feat, const Tensor &bias, const Tensor &i, const Tensor &j,
                    const Tensor &seg, const ConvSizes &s) {
    Tensor w = as4(weight), x = feat;
    require(w.dim() == 4, PyExc_ValueError,
            [&] { return "expected a weight (taps, groups, inputs, outputs), got " + str(weight.sizes()); });
    require(w.size(0) == s.K && x.dim() == 2 && x.size(1) == w.size(1) * w.size(2), PyExc_AssertionError, [&] {
        return "features " + str(x.sizes()) + " do not fit a weight " + str(weight.sizes()) + " of " + std::to_string(s.K) + " taps";
    });
    require(x.size(0) == s.n_in, PyExc_AssertionError,
            [&] { return "feat rows " + std::to_string(x.size(0)) + " != index.N_in " + std::to_string(s.n_in); });
    match(w, x);
    require(!bias.defined() || (bias.dim() == 1 && bias.numel() == w.size(1) * w.size(3) && bias.device() == x.device() &&
                                bias.scalar_type() == x.scalar_type()),   // the kernels read it by address
            PyExc_ValueError, [&] { return "the bias does not fit a weight " + str(weight.sizes()); });
    int64_t engine = s.engine();
    if (s.cover_out && i.numel() == s.n_out) engine |= FAN_IN_ONE;   // one triplet per output row: stored, not reduced
    return mvmr_impl(w, x, j, i, seg, std::nullopt, s.n_out, 0, engine, bias.defined() ? bias.contiguous() : bias)
        .to(feat.scalar_type());
}

Tensor conv_grad_input(const Tensor &weight, const Tensor &grad, const Tensor &i, const Tensor &j, const Tensor &seg,
                       const ConvSizes &s) {
    Tensor w = as4(weight), g = grad;
    match(w, g);
    int64_t engine = s.engine();
    // a self-search rulebook holds (j, i, K - 1 - k) with every (i, j, k): the input gradient is the forward
    // schedule over the same rulebook (and the same plan) with the taps of the weight in reverse order
    if (s.n_out == s.n_in && is_symmetric(i, j, s.K))
        return mvmr_impl(w, g, j, i, seg, std::nullopt, s.n_in, 3, engine, Tensor()).to(grad.scalar_type());
    if (s.cover_in && i.numel() == s.n_in) engine |= FAN_IN_ONE;
    return mvmr_impl(w, g, i, j, seg, std::nullopt, s.n_in, 1, engine, Tensor()).to(grad.scalar_type());
}

Tensor conv_grad_weight(const Tensor &feat, const Tensor &grad, const Tensor &i, const Tensor &j, const Tensor &seg,
                        at::IntArrayRef weight_shape, const ConvSizes &s) {
    const int64_t G = weight_shape.size() == 4 ? weight_shape[1] : 1;
    Tensor x = feat, g = grad;
    match(x, g);
    return vvor(x.view({x.size(0), G, -1}), j, g.view({g.size(0), G, -1}), i, seg, std::nullopt, s.K, g_engine)
        .to(feat.scalar_type())
        .view(weight_shape);
}

// out[i] += feat[j] @ W[k] (+ bias), with its three gradients; one node of the autograd graph.
struct Conv : public torch::autograd::Function<Conv> {
    static Tensor forward(torch::autograd::AutogradContext *ctx, const Tensor &weight, const Tensor &feat, const OptTensor &bias,
                          const Tensor &i, const Tensor &j, const Tensor &seg, int64_t n_out, int64_t n_in, int64_t K,
                          bool cover_out, bool cover_in, bool plan_padded) {
        ctx->save_for_backward({weight, feat, i, j, seg});
        ctx->saved_data["sizes"] = std::vector<int64_t>{n_out, n_in, K, cover_out, cover_in, bias.has_value(), plan_padded};
        return conv_forward(weight, feat, bias ? *bias : Tensor(), i, j, seg, {n_out, n_in, K, cover_out, cover_in, plan_padded});
    }

    static torch::autograd::variable_list backward(torch::autograd::AutogradContext *ctx, torch::autograd::variable_list grads) {
        const auto saved = ctx->get_saved_variables();
        const Tensor &weight = saved[0], &feat = saved[1], &i = saved[2], &j = saved[3], &seg = saved[4];
        const auto v = ctx->saved_data["sizes"].toIntVector();
        const ConvSizes s{v[0], v[1], v[2], v[3] != 0, v[4] != 0, v[6] != 0};
        torch::autograd::variable_list out(12);
        if (!grads[0].defined()) return out;
        const Tensor &go = grads[0];
        const bool want_w = ctx->needs_input_grad(0), want_x = ctx->needs_input_grad(1), want_b = v[5] && ctx->needs_input_grad(2);
        if (at::GradMode::is_enabled()) {   // create_graph: the gradients themselves have to be differentiable
            py::gil_scoped_acquire gil;
            py::tuple r = py::cast<py::tuple>(py::reinterpret_borrow<py::object>(g_double_backward)(
                weight, feat, go, i, j, seg, s.n_out, s.n_in, s.K, s.cover_out, s.cover_in, want_w, want_x, want_b));
            for (int q = 0; q < 3; ++q)
                if (!r[q].is_none()) out[q] = py::cast<Tensor>(r[q]);
            return out;
        }
        const Tensor g = go.contiguous();
        c10::cuda::CUDAGuard guard(g.device());
        if (want_b) out[2] = column_sums(g);
        if (want_w) out[0] = conv_grad_weight(feat, g, i, j, seg, weight.sizes(), s).to(weight.scalar_type());
        if (want_x) out[1] = conv_grad_input(weight, g, i, j, seg, s).to(feat.scalar_type());
        return out;
    }
};

Tensor conv(const Tensor &weight, const Tensor &feat, const OptTensor &bias, const Tensor &i, const Tensor &j, const Tensor &seg,
            int64_t n_out, int64_t n_in, int64_t K, bool cover_out, bool cover_in, bool plan_padded) {
    if (!at::GradMode::is_enabled() ||
        !(weight.requires_grad() || feat.requires_grad() || (bias && bias->requires_grad())))
        return conv_forward(weight, feat, bias ? *bias : Tensor(), i, j, seg, {n_out, n_in, K, cover_out, cover_in, plan_padded});
    return Conv::apply(weight, feat, bias, i, j, seg, n_out, n_in, K, cover_out, cover_in, plan_padded);
}

// --------------------------------------------------- ragged layer norm (autograd) ----
Tensor f32_or_none(const OptTensor &t) { return t ? t->detach().to(at::kFloat).contiguous() : Tensor(); }

std::tuple<Tensor, Tensor, Tensor> layer_norm_forward(Tensor x, const Tensor &lengths_, const OptTensor &weight_,
                                                      const OptTensor &bias_, const OptTensor &residual_, double eps, bool relu) {
    require(x.dim() == 2, PyExc_ValueError, [&] { return "expected rows (points, channels), got " + str(x.sizes()); });
    require_cuda(x), require_cuda(lengths_), require_cuda(weight_), require_cuda(bias_), require_cuda(residual_);
    const int code = dtype_code(x.scalar_type());
    c10::cuda::CUDAGuard guard(x.device());
    x = x.contiguous();
    const Tensor lengths = as_i64(lengths_), weight = f32_or_none(weight_), bias = f32_or_none(bias_);
    const Tensor residual = residual_ ? residual_->to(x.scalar_type()).contiguous() : Tensor();
    const int64_t N = x.size(0), C = x.size(1), S = lengths.numel();
    Tensor y = at::empty_like(x);
    Tensor stats = at::empty({2, S}, x.options().dtype(at::kFloat));
    Tensor mean = stats.select(0, 0), rstd = stats.select(0, 1);
    Tensor ws = workspace(pcx_ragged_layer_norm_workspace_bytes(N, S), x);
    check(pcx_ragged_layer_norm(ptr(x), ptr_as<int64_t>(lengths), ptr_as<float>(weight), ptr_as<float>(bias), ptr(residual), ptr(y),
                                ptr_as<float>(mean), ptr_as<float>(rstd), N, S, (int)C, eps, relu, code, ptr(ws), ws.numel(),
                                stream()));
    return {y, mean, rstd};
}

std::tuple<Tensor, Tensor, Tensor, Tensor> layer_norm_backward(Tensor grad_y, Tensor x, const Tensor &y, const Tensor &lengths_,
                                                               const OptTensor &weight_, const Tensor &mean, const Tensor &rstd,
                                                               bool relu, bool want_affine, bool want_residual) {
    require_cuda(grad_y), require_cuda(x), require_cuda(lengths_);
    const int code = dtype_code(x.scalar_type());
    c10::cuda::CUDAGuard guard(x.device());
    grad_y = grad_y.contiguous(), x = x.contiguous();
    const Tensor lengths = as_i64(lengths_), weight = f32_or_none(weight_);
    const int64_t N = x.size(0), C = x.size(1), S = lengths.numel();
    Tensor gx = at::empty_like(x), gw, gb, gres;
    if (want_affine) {
        gw = at::empty({C}, x.options().dtype(at::kFloat));
        gb = at::empty({C}, x.options().dtype(at::kFloat));
    }
    if (want_residual) gres = at::empty_like(x);
    Tensor ws = workspace(pcx_ragged_layer_norm_workspace_bytes(N, S), x);
    check(pcx_ragged_layer_norm_backward(ptr(grad_y), ptr(x), ptr(y), ptr_as<int64_t>(lengths), ptr_as<float>(weight),
                                         ptr_as<float>(mean), ptr_as<float>(rstd), ptr(gx), ptr_as<float>(gw), ptr_as<float>(gb),
                                         ptr(gres), N, S, (int)C, relu, code, ptr(ws), ws.numel(), stream()));
    return {gx, gw, gb, gres};
}

struct LayerNorm : public torch::autograd::Function<LayerNorm> {
    static Tensor forward(torch::autograd::AutogradContext *ctx, const Tensor &x, const Tensor &lengths, const OptTensor &weight,
                          const OptTensor &bias, const OptTensor &residual, double eps, bool relu) {
        auto [y, mean, rstd] = layer_norm_forward(x, lengths, weight, bias, residual, eps, relu);
        ctx->save_for_backward({x, y, lengths, weight ? *weight : Tensor(), mean, rstd});
        ctx->saved_data["relu"] = relu;
        // edges of the node exist for the tensors that were given: remember where theirs are (-1: none)
        const int64_t at_weight = weight ? 2 : -1, at_bias = bias ? 2 + (weight ? 1 : 0) : -1;
        const int64_t at_residual = residual ? 2 + (weight ? 1 : 0) + (bias ? 1 : 0) : -1;
        ctx->saved_data["edges"] = std::vector<int64_t>{at_weight, at_bias, at_residual};
        ctx->saved_data["bias_type"] = (int64_t)(bias ? bias->scalar_type() : at::kFloat);
        ctx->saved_data["residual_type"] = (int64_t)(residual ? residual->scalar_type() : x.scalar_type());
        return y;
    }

    static torch::autograd::variable_list backward(torch::autograd::AutogradContext *ctx, torch::autograd::variable_list grads) {
        const auto saved = ctx->get_saved_variables();
        torch::autograd::variable_list out(7);
        if (!grads[0].defined()) return out;
        // as the Python node did: once differentiable (its backward is opaque to autograd)
        at::AutoGradMode no_graph(false);
        const auto edges = ctx->saved_data["edges"].toIntVector();
        const auto needs = [&](int q) { return edges[q] >= 0 && ctx->needs_input_grad((size_t)edges[q]); };
        const bool affine = saved[3].defined() && (needs(0) || needs(1));
        auto [gx, gw, gb, gres] =
            layer_norm_backward(grads[0], saved[0], saved[1], saved[2], saved[3].defined() ? OptTensor(saved[3]) : std::nullopt,
                                saved[4], saved[5], ctx->saved_data["relu"].toBool(), affine, needs(2));
        out[0] = gx;
        if (affine) {
            out[2] = gw.to(saved[3].scalar_type());
            if (edges[1] >= 0) out[3] = gb.to((at::ScalarType)ctx->saved_data["bias_type"].toInt());
        }
        if (gres.defined()) out[4] = gres.to((at::ScalarType)ctx->saved_data["residual_type"].toInt());
        return out;
    }
};

Tensor layer_norm(const Tensor &x, const Tensor &lengths, const OptTensor &weight, const OptTensor &bias,
                  const OptTensor &residual, double eps, bool relu) {
    // the node refuses torch.func transforms and forward-mode tangents; the kernels alone would drop them
    const bool transforms = c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::FuncTorchDynamicLayerFrontMode);
    const auto wants = [](const OptTensor &t) {
        return t && ((at::GradMode::is_enabled() && t->requires_grad()) || t->_fw_grad(0).defined());
    };
    if (!transforms && !wants(x) && !wants(weight) && !wants(bias) && !wants(residual))
        return std::get<0>(layer_norm_forward(x, lengths, weight, bias, residual, eps, relu));
    return LayerNorm::apply(x, lengths, weight, bias, residual, eps, relu);
}

// ----------------------------------------------------------------- geometry ----
// Sample ids as the searches and the down-sampling read them: 64-bit ones by their low words, where they lie.
Tensor ids(const Tensor &t) { return t.scalar_type() == at::kLong ? t.contiguous() : as_i32(t); }

// Tap-segmented search: enqueue, fill into buffers sized from `ratio` (pairs per query of earlier searches
// of this kind; negative: count first) and one hand-over.  Returns
// (i, j, k | undefined, seg, num_neighbors, total, queries without neighbour, device status, pairs of the fullest tap).
std::tuple<Tensor, Tensor, OptTensor, Tensor, Tensor, int64_t, int64_t, int64_t, int64_t> radius_taps(
    const Tensor &points_, const Tensor &queries_, double radius, const OptTensor &ps_, const OptTensor &qs_, int64_t distance_type,
    int64_t kernel_size, double grid, bool want_k, double ratio) {
    require_cuda(points_), require_cuda(queries_), require_cuda(ps_), require_cuda(qs_);
    c10::cuda::CUDAGuard guard(points_.device());
    const Tensor points = points_.contiguous(), queries = queries_.contiguous();
    const Tensor ps = ps_ ? ids(*ps_) : Tensor();
    const Tensor qs = !qs_ ? Tensor() : (ps_ && qs_->is_same(*ps_)) ? ps : ids(*qs_);
    if (ps.defined() && ps.scalar_type() == at::kLong) distance_type |= PCX_RADIUS_WIDE_POINT_IDS;
    if (qs.defined() && qs.scalar_type() == at::kLong) distance_type |= PCX_RADIUS_WIDE_QUERY_IDS;
    const int64_t P = points.size(0), Q = queries.size(0), k3 = kernel_size * kernel_size * kernel_size;
    const auto i32 = at::TensorOptions().dtype(at::kInt).device(points.device());
    const auto i64 = i32.dtype(at::kLong);
    Tensor ws = workspace(pcx_radius_taps_workspace_bytes(P, Q, (int)kernel_size), points);
    Tensor num_neighbors = at::empty({Q}, i64), seg = at::empty({k3 + 1}, i64);
    check(pcx_radius_taps_count(ptr_as<float>(points), ptr_as<float>(queries), ptr_as<int32_t>(ps), ptr_as<int32_t>(qs), P, Q, radius,
                                (int)distance_type, (int)kernel_size, grid, ptr_as<int64_t>(num_neighbors), ptr_as<int64_t>(seg),
                                ptr(ws), ws.numel(), stream()));
    int64_t total[4] = {0, 0, 0, 0}, capacity;
    if (ratio < 0) {
        check(pcx_radius_taps_total(P, Q, (int)kernel_size, total, ptr(ws), ws.numel(), stream()));
        capacity = total[0];
    } else {
        capacity = std::min<int64_t>((int64_t)(ratio * (double)Q * 1.25) + 4096, ((int64_t)1 << 31) - 1);
    }
    Tensor i, j, k;
    for (int attempt = 0; attempt < 2; ++attempt) {
        i = at::empty({capacity}, i32), j = at::empty({capacity}, i32);
        if (want_k) k = at::empty({capacity}, i32);
        const int rc = pcx_radius_taps_fill(ptr_as<float>(queries), ptr_as<int32_t>(ps), ptr_as<int32_t>(qs), P, Q, radius,
                                            (int)distance_type | PCX_RADIUS_FULLEST_TAP, (int)kernel_size, grid, capacity, ptr_as<int32_t>(i),
                                            ptr_as<int32_t>(j), ptr_as<int32_t>(k), total, ptr(ws), ws.numel(), stream());
        if (rc == PCX_E_CAPACITY && attempt == 0 && total[0] > capacity) {
            capacity = total[0];   // the estimate was too small: exact size, fill pass only
            continue;
        }
        check(rc);
        break;
    }
    const int64_t n = total[0];
    return {i.narrow(0, 0, n), j.narrow(0, 0, n), want_k ? OptTensor(k.narrow(0, 0, n)) : std::nullopt, seg, num_neighbors, n, total[1],
            total[2], total[3]};
}

// (indices, points, sample | undefined, mapping | undefined, points per sample | undefined) of the centre-nearest
// point of every occupied cell
std::tuple<Tensor, Tensor, OptTensor, OptTensor, OptTensor> grid_sample(const Tensor &points_, double cell, const OptTensor &sample_,
                                                             bool want_mapping) {
    require_cuda(points_), require_cuda(sample_);
    c10::cuda::CUDAGuard guard(points_.device());
    const Tensor points = points_.contiguous(), sample = sample_ ? ids(*sample_) : Tensor();
    const bool wide = sample.defined() && sample.scalar_type() == at::kLong;
    const int64_t N = points.size(0);
    const auto i64 = at::TensorOptions().dtype(at::kLong).device(points.device());
    Tensor ws = workspace(pcx_grid_sample_workspace_bytes(N), points);
    int64_t info[3] = {0, 0, 0};
    if (wide) check(pcx_grid_sample_count_ids(ptr_as<float>(points), ptr_as<int64_t>(sample), N, cell, info, ptr(ws), ws.numel(), stream()));
    else check(pcx_grid_sample_count_samples(ptr_as<float>(points), ptr_as<int32_t>(sample), N, cell, info, ptr(ws), ws.numel(), stream()));
    const int64_t cells = info[0];
    Tensor indices = at::empty({cells}, i64), out = at::empty({cells, 3}, i64.dtype(at::kFloat));
    Tensor out_sample = sample_ ? at::empty({cells}, wide ? i64 : i64.dtype(at::kInt)) : Tensor();
    Tensor mapping = want_mapping ? at::empty({N}, i64) : Tensor();
    OptTensor sizes;
    // cells come in ascending sample order; ids far beyond the number of points (hashes) are not worth an array
    if (sample_ && info[1] >= 0 && info[2] < std::max<int64_t>(N, 4096)) sizes = at::empty({info[2] + 1}, i64);
    if (wide) {
        check(pcx_grid_sample_select_ids(ptr_as<float>(points), ptr_as<int64_t>(sample), N, cell, cells, ptr_as<int64_t>(indices), ptr_as<float>(out),
                                         ptr_as<int64_t>(out_sample), ptr_as<int64_t>(mapping), sizes ? ptr_as<int64_t>(*sizes) : nullptr,
                                         info[2] + 1, ptr(ws), ws.numel(), stream()));
        return {indices, out, OptTensor(out_sample), want_mapping ? OptTensor(mapping) : std::nullopt, sizes};
    }
    check(pcx_grid_sample_select(ptr_as<float>(points), ptr_as<int32_t>(sample), N, cell, cells, ptr_as<int64_t>(indices),
                                 ptr_as<float>(out), ptr_as<int32_t>(out_sample), ptr_as<int64_t>(mapping), ptr(ws), ws.numel(),
                                 stream()));
    if (sizes) check(pcx_sample_sizes(ptr_as<int32_t>(out_sample), cells, info[2] + 1, ptr_as<int64_t>(*sizes), stream()));
    return {indices, out, sample_ ? OptTensor(out_sample) : std::nullopt, want_mapping ? OptTensor(mapping) : std::nullopt, sizes};
}

// (plan buffer, number of buckets with several triplets, null or page-locked words).  A rulebook whose rows are known
// to ascend inside every tap needs no wait: the number is a bound then, and the true one and the builder's verdict on
// the rows replace the words' -1 when the plan is ready.
std::tuple<Tensor, int64_t, OptTensor> plan_build(const Tensor &scatter_, const Tensor &gather_, const Tensor &seg_, int64_t K,
                                                  int64_t n_out, int64_t group, bool ordered) {
    require_cuda(scatter_), require_cuda(gather_), require_cuda(seg_);
    c10::cuda::CUDAGuard guard(scatter_.device());
    const Tensor scatter = as_i32(scatter_), gather = as_i32(gather_), seg = as_i64(seg_);
    const int64_t T = scatter.numel();
    const size_t bytes = pcx_mvmr_plan_bytes(T, n_out, (int)K, (int)group);
    if (bytes == 0) {
        py::gil_scoped_acquire gil;
        raise(PyExc_NotImplementedError, "no output-stationary plan for T=" + std::to_string(T) + " n_out=" + std::to_string(n_out) +
                                             " K=" + std::to_string(K) + " group=" + std::to_string(group));
    }
    Tensor buf = workspace(bytes, scatter), ws = workspace(pcx_mvmr_plan_workspace_bytes(T, n_out, (int)K, (int)group), scatter);
    int64_t multi = 0;
    ordered = ordered && T > 0 && c10::cuda::currentStreamCaptureStatusMayInitCtx() == c10::cuda::CaptureStatus::None;
    check(pcx_mvmr_plan_build_counted(ptr_as<int32_t>(scatter), ptr_as<int32_t>(gather), ptr_as<int64_t>(seg), T, (int)K, n_out, (int)group,
                                      ptr(buf), buf.numel(), ptr(ws), ws.numel(), ordered ? nullptr : &multi, stream()));
    if (!ordered) return {buf, multi, std::nullopt};
    Tensor words = at::empty({2}, at::TensorOptions().dtype(at::kInt).pinned_memory(true));
    for (int n = 0; n < 2; ++n) static_cast<volatile int32_t *>(words.data_ptr<int32_t>())[n] = -1;
    words.copy_(buf.narrow(0, 4 * PCX_PLAN_MULTI_WORD, 8).view(at::kInt), true);
    return {buf, std::min(T / 2, n_out * K), words};
}

// The words of a plan that was not waited for: the number of buckets, -1 until it is known, -2 for rows out of order.
int64_t peek(const Tensor &words) {
    const volatile int32_t *w = static_cast<volatile int32_t *>(words.data_ptr<int32_t>());
    const int32_t multi = w[0], unsorted = w[1];
    return multi == -1 || unsorted == -1 ? -1 : unsorted ? -2 : multi;
}

Tensor planned(const Tensor &weight, const Tensor &feat, const Tensor &buffer, int64_t group, int64_t multi, int64_t T, int64_t n_out,
               bool transpose, bool split) {
    require_cuda(weight), require_cuda(feat);
    c10::cuda::CUDAGuard guard(feat.device());
    Plan plan;
    plan.buffer = buffer, plan.group = group, plan.multi = multi;
    return mvmr_planned(weight.contiguous(), feat.contiguous(), plan, T, n_out, (transpose ? 1 : 0) | (split ? SPLIT_SUMS : 0), Tensor());
}

// Geometry on a stream of its own: from here on the calling thread's work on `device` goes to the given stream ...
std::tuple<int64_t, int64_t, int64_t> side_begin(int64_t stream_id, int64_t device, int64_t type) {
    const auto before = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)device).pack3();
    c10::cuda::setCurrentCUDAStream(c10::cuda::CUDAStream::unpack3(stream_id, (c10::DeviceIndex)device, (c10::DeviceType)type));
    return {before.stream_id, before.device_index, (int64_t)before.device_type};
}
// ... and back: the stream before waits for what was enqueued meanwhile.
void side_end(int64_t stream_id, int64_t device, int64_t type) {
    const auto before = c10::cuda::CUDAStream::unpack3(stream_id, (c10::DeviceIndex)device, (c10::DeviceType)type);
    at::cuda::CUDAEvent event;
    event.record(c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)device));
    event.block(before);
    c10::cuda::setCurrentCUDAStream(before);
}
// The tensors are used on the calling thread's current stream from now on.
void record_streams(const std::vector<Tensor> &tensors) {
    for (const Tensor &t : tensors)
        if (t.is_cuda()) t.record_stream(c10::cuda::getCurrentCUDAStream(t.device().index()).unwrap());
}

void set_hooks(py::object plan, py::object symmetric, py::object ascending, py::object fullest, py::object double_backward) {
    g_plan_hook = plan.release().ptr();
    g_symmetric_hook = symmetric.release().ptr();
    g_ascending_hook = ascending.release().ptr();
    g_fullest_hook = fullest.release().ptr();
    g_double_backward = double_backward.release().ptr();
}

}  // namespace

PYBIND11_MODULE(_pcx_host, m) {
    m.def("set_hooks", &set_hooks);
    m.def("side_begin", &side_begin);
    m.def("side_end", &side_end);
    m.def("record_streams", &record_streams);
    m.def("set_engine", [](int e) { g_engine = e; });
    m.def("mvmr", &mvmr);
    m.def("vvor", &vvor);
    m.def("conv", &conv, py::arg("weight"), py::arg("feat"), py::arg("bias"), py::arg("i"), py::arg("j"), py::arg("seg"), py::arg("n_out"),
          py::arg("n_in"), py::arg("K"), py::arg("cover_out"), py::arg("cover_in"), py::arg("plan_padded") = false);
    m.def("column_sums", &column_sums);
    m.def("layer_norm", &layer_norm);
    m.def("radius_taps", &radius_taps, py::call_guard<py::gil_scoped_release>());
    m.def("grid_sample", &grid_sample, py::call_guard<py::gil_scoped_release>());
    m.def("peek", &peek);
    m.def("plan_build", &plan_build, py::call_guard<py::gil_scoped_release>());
    m.def("planned", &planned);
}
