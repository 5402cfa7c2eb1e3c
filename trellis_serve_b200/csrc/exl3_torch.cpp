// Torch side of the library: the `exl3_b200::linear` operator, the load-time preparation of a fused group and the scratch
// the eager entry points share, in C++ over the C ABI (include/exl3_b200.h).
//
// An eager decode step calls the operator a few hundred times per token on matrices whose kernels take 5 to 40 us, so the
// host side of a call has to stay below that: dispatch, output allocation and launch are native.  The operator written in
// Python (argument handling, two context managers, a dozen ctypes conversions) took 38 us of host time per call whatever the
// size; through the dispatcher it takes 9 to 11 us, of which two thirds are the dispatcher's schema matching and boxing of eleven
// arguments (a call with no rows, which launches nothing, takes 10.8 of 15.9 us on a slow host), so plain eager calls come in through
// `direct_linear` below: 9.1 -> 4.5 us of host time at one row of 1024 x 640.
#include <Python.h>

#include <mutex>
#include <string>
#include <vector>

#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/core/dispatch/Dispatcher.h>
#include <ATen/record_function.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/library.h>

#include "../../include/exl3_b200.h"

namespace {

void check(int status, const char* where)
{
    if (status == EXL3_OK) return;
    std::string msg = std::string(where) + ": " + exl3_status_str(status);
    if (status == EXL3_ERR_CUDA) msg += " (cudaError " + std::to_string(exl3_last_cuda_error()) + ")";
    TORCH_CHECK(false, msg, " (status ", status, ")");
}

// Per-device set-up, once; must precede any CUDA-graph capture.
int device_sms(int device)
{
    static std::mutex m;
    static int sms[64] = {};
    TORCH_CHECK(device >= 0 && device < 64, "device index out of range");
    std::lock_guard<std::mutex> lock(m);
    if (sms[device] == 0) {
        check(exl3_init_device(device), "exl3_init_device");
        sms[device] = exl3_device_sm_count(device);
    }
    return sms[device];
}

// Scratch that calls without a workspace of their own share, one zero-filled tensor per device and kind (0: decode kernels,
// 1: many-row kernels), grown when a larger call comes.
std::mutex g_scratch_mutex;
at::Tensor g_scratch[2][64];

at::Tensor scratch(int64_t kind, int64_t device, int64_t nbytes)
{
    TORCH_CHECK(kind >= 0 && kind < 2 && device >= 0 && device < 64, "no such scratch");
    std::lock_guard<std::mutex> lock(g_scratch_mutex);
    at::Tensor& t = g_scratch[kind][device];
    if (nbytes > 0 && (!t.defined() || t.numel() < nbytes))
        t = at::zeros({nbytes}, at::TensorOptions().dtype(at::kByte).device(at::Device(at::kCUDA, (c10::DeviceIndex)device)));
    return t.defined() ? t : at::empty({0}, at::TensorOptions().dtype(at::kByte));
}

void scratch_clear(int64_t kind)
{
    TORCH_CHECK(kind >= 0 && kind < 2, "no such scratch");
    std::lock_guard<std::mutex> lock(g_scratch_mutex);
    for (auto& t : g_scratch[kind]) t = at::Tensor();
}

// Measurement knobs of runtime/ops.py: [0] row count from which the many-row path is taken (0: exl3_prefers_decode), [1] 1: the many-row
// path decodes the weights and calls the library GEMM.
int64_t g_knob[2] = {0, 0};
int64_t knob(int64_t which, int64_t value)
{
    TORCH_CHECK(which >= 0 && which < 2, "no such knob");
    if (value >= 0) g_knob[which] = value;
    return g_knob[which];
}

int dtype_code(const at::Tensor& t)
{
    if (t.scalar_type() == at::kHalf) return EXL3_F16;
    TORCH_CHECK(t.scalar_type() == at::kBFloat16, "activations must be fp16 or bf16");
    return EXL3_BF16;
}

const uint16_t* u16(const at::Tensor& t) { return static_cast<const uint16_t*>(t.const_data_ptr()); }

// Contiguous copy of columns [a, a + w) of every matrix of the group, logical widths beyond the stored ones read as zeros.
at::Tensor trim(const at::Tensor& y, const std::vector<int64_t>& bounds, at::IntArrayRef widths)
{
    int64_t total = 0;
    bool wider = false;
    for (size_t i = 0; i < widths.size(); i++) {
        total += widths[i];
        wider = wider || widths[i] > bounds[i + 1] - bounds[i];
    }
    at::Tensor out = wider ? at::zeros({y.size(0), total}, y.options()) : at::empty({y.size(0), total}, y.options());
    int64_t col = 0;
    for (size_t i = 0; i < widths.size(); i++) {
        const int64_t keep = std::min(widths[i], bounds[i + 1] - bounds[i]);
        if (keep > 0) out.narrow(1, col, keep).copy_(y.narrow(1, bounds[i], keep));
        col += widths[i];
    }
    return out;
}

at::Tensor linear(const at::Tensor& x, at::TensorList trellis, at::TensorList suh, at::TensorList svh, at::TensorList dense,
                  at::TensorList sliced, int64_t sliced_min_rows, at::TensorList marlin_w, at::IntArrayRef marlin_ends,
                  at::IntArrayRef codebooks, at::IntArrayRef out_widths)
{
    TORCH_CHECK(marlin_w.size() == 3, "marlin_w must be [packed, suh_cat, svh_cat] from kernels.linear.prepare");
    TORCH_CHECK(!codebooks.empty(), "one codebook per fused group");
    for (int64_t c : codebooks) TORCH_CHECK(c == codebooks[0], "one codebook per fused group");
    const at::Tensor &packed = marlin_w[0], &suh_cat = marlin_w[1], &svh_cat = marlin_w[2];
    TORCH_CHECK(packed.dim() == 6, "packed weights are [n/128, k/128, 8, 2, K, 32]");
    const int64_t k = packed.size(1) * 128, n_total = packed.size(0) * 128;
    const int K = (int)packed.size(4), cb = (int)codebooks[0], shards = (int)marlin_ends.size() + 1;
    TORCH_CHECK(shards <= 8, "too many matrices in one group");
    TORCH_CHECK(x.dim() >= 1, "x needs a last dimension");
    const c10::cuda::CUDAGuard guard(x.device());
    const int sms = device_sms(x.device().index());

    at::Tensor h = x.dim() == 2 ? x : x.reshape({-1, x.size(-1)});
    if (h.scalar_type() != at::kHalf && h.scalar_type() != at::kBFloat16) h = h.to(at::kHalf);
    TORCH_CHECK(h.size(1) <= k, "input width ", h.size(1), " exceeds the stored width ", k);
    const int64_t rows = h.size(0);
    std::vector<int64_t> bounds(shards + 1, 0);
    int ends[8], widths[8];
    for (int s = 0; s + 1 < shards; s++) {
        bounds[s + 1] = marlin_ends[s];
        ends[s] = (int)marlin_ends[s];
    }
    bounds[shards] = n_total;
    bool whole = (int)out_widths.size() == shards, wider = !whole;
    int64_t n_out = 0;
    for (int s = 0; s < shards && s < (int)out_widths.size(); s++) {
        whole = whole && out_widths[s] == bounds[s + 1] - bounds[s];
        wider = wider || out_widths[s] > bounds[s + 1] - bounds[s] || out_widths[s] < 0;
        widths[s] = (int)out_widths[s];
        n_out += out_widths[s];
    }
    TORCH_CHECK((int)out_widths.size() <= shards, "more output widths than matrices");

    const bool decode = g_knob[0] > 0 ? rows < g_knob[0] : exl3_prefers_decode((int)rows, (int)k, (int)n_total, sms) != 0;
    const bool library = !decode && (!dense.empty() || g_knob[1] != 0);
    // Stored input width is padded to 128: the kernels read rows of the true width (the many-row one in steps of eight columns).
    h = h.contiguous();
    if (h.size(1) < k && (library || h.size(1) == 0 || (!decode && (h.size(1) % 8 != 0 || reinterpret_cast<uintptr_t>(h.const_data_ptr()) % 16 != 0))))
        h = at::constant_pad_nd(h, {0, k - h.size(1)});
    const int x_cols = (int)h.size(1);
    at::Tensor y;
    bool trimmed = whole;                                    // y has the true output columns
    if (library) {
        // resident decoded weights, or the decode + library GEMM sequence asked for: runtime/ops.py
        static auto op = c10::Dispatcher::singleton().findSchemaOrThrow("exl3_b200::dense_linear", "");
        y = op.typed<at::Tensor(const at::Tensor&, at::TensorList, at::TensorList, at::IntArrayRef, int64_t)>().call(h, dense, marlin_w, marlin_ends, cb);
    } else {
        const bool ragged = decode && !wider && !whole && n_out > 0;
        y = at::empty({rows, ragged ? n_out : n_total}, h.options());
        if (ragged) trimmed = true;
        if (rows > 0) {
            void* st = c10::cuda::getCurrentCUDAStream(x.device().index()).stream();
            const size_t need = decode ? exl3_linear_workspace_bytes((int)rows, (int)k, (int)n_total, shards)
                                       : exl3_gemm_tc_workspace_bytes((int)rows, (int)k, (int)n_total, shards);
            const at::Tensor ws = scratch(decode ? 0 : 1, x.device().index(), (int64_t)need);
            const uint32_t* w = static_cast<const uint32_t*>(packed.const_data_ptr());
            if (decode) {
                if (!ragged)
                    for (int s = 0; s < shards; s++) widths[s] = (int)(bounds[s + 1] - bounds[s]);
                check(exl3_linear_ragged(h.const_data_ptr(), dtype_code(h), x_cols, w, K, cb, u16(suh_cat), u16(svh_cat), ends, widths, shards, (int)rows,
                                         (int)k, (int)n_total, y.mutable_data_ptr(), dtype_code(y), ws.mutable_data_ptr(), (size_t)ws.numel(), st),
                      "exl3_linear");
            } else {
                check(exl3_linear_tc_padded(h.const_data_ptr(), dtype_code(h), x_cols, w, K, cb, u16(suh_cat), u16(svh_cat), ends, shards, (int)rows,
                                            (int)k, (int)n_total, y.mutable_data_ptr(), dtype_code(y), ws.mutable_data_ptr(), (size_t)ws.numel(), st),
                      "exl3_linear_tc");
            }
        }
    }
    if (!trimmed) y = trim(y, bounds, out_widths);
    if (y.scalar_type() != x.scalar_type()) y = y.to(x.scalar_type());
    if (x.dim() == 2) return y;
    std::vector<int64_t> shape(x.sizes().begin(), x.sizes().end());
    shape.back() = y.size(1);
    return y.view(shape);
}

// Stored matrices of a fused group -> (resident weights [n_total/128, k/128, 8, 2, K, 32], suh [shards, k], svh [n_total]).
// Every matrix is repacked straight into its column blocks (no second pass over the weights); the small copies are enqueued
// while those kernels run.  Returns once the results are complete: the run path fetches weights and sign vectors before the
// kernel ahead of it in the stream has finished (programmatic dependent launch).
std::tuple<at::Tensor, at::Tensor, at::Tensor> prepare_group(at::TensorList trellis, at::TensorList suh, at::TensorList svh, int64_t max_rows)
{
    const at::Device device = trellis[0].device();
    const c10::cuda::CUDAGuard guard(device);
    device_sms(device.index());
    const int64_t kt = trellis[0].size(0), words = trellis[0].size(2);
    int64_t nt = 0;
    for (const at::Tensor& t : trellis) {
        TORCH_CHECK(t.size(0) == kt && t.size(2) == words, "the matrices of a fused group share input width and bitrate");
        nt += t.size(1);
    }
    at::Tensor packed = at::empty({nt / 8, kt / 8, 8, 2, words / 16, 32}, trellis[0].options().dtype(at::kInt));
    const auto stream = c10::cuda::getCurrentCUDAStream(device.index());
    uint32_t* dst = static_cast<uint32_t*>(packed.mutable_data_ptr());
    // Vectors as the kernel can copy them: 16-bit, contiguous, one per matrix; anything else goes through torch.
    const int64_t count = (int64_t)trellis.size();
    bool plain = count <= 8 && (int64_t)suh.size() == count && (int64_t)svh.size() == count;
    for (int64_t i = 0; plain && i < count; i++) {
        const auto fits = [&](const at::Tensor& v, int64_t n) {
            return v.device() == device && v.dim() == 1 && v.size(0) == n && v.is_contiguous() && v.element_size() == 2 && v.scalar_type() == suh[0].scalar_type();
        };
        plain = fits(suh[i], kt * 16) && fits(svh[i], trellis[i].size(1) * 16);
    }
    at::Tensor suh_cat, svh_cat;
    if (plain) {
        const uint16_t *t[8], *u[8], *v[8];
        int ns[8];
        std::vector<at::Tensor> keep;
        suh_cat = at::empty({count, kt * 16}, suh[0].options());
        svh_cat = at::empty({nt * 16}, svh[0].options());
        for (int64_t i = 0; i < count; i++) {
            keep.push_back(trellis[i].contiguous());
            t[i] = u16(keep.back());
            u[i] = u16(suh[i]);
            v[i] = u16(svh[i]);
            ns[i] = (int)trellis[i].size(1) * 16;
        }
        check(exl3_repack_group(t, u, v, ns, (int)count, (int)kt * 16, (int)(words / 16), dst, static_cast<uint16_t*>(suh_cat.mutable_data_ptr()),
                                static_cast<uint16_t*>(svh_cat.mutable_data_ptr()), stream.stream()),
              "exl3_repack_group");
    } else {
        for (const at::Tensor& t : trellis) {
            const at::Tensor c = t.contiguous();
            check(exl3_repack(u16(c), (int)kt * 16, (int)c.size(1) * 16, (int)(words / 16), dst, stream.stream()), "exl3_repack");
            dst += c.numel() / 2;
        }
        suh_cat = at::stack(suh);
        svh_cat = at::cat(svh);
    }
    scratch(0, device.index(), (int64_t)exl3_linear_workspace_bytes((int)max_rows, (int)kt * 16, (int)nt * 16, (int)trellis.size()));
    stream.synchronize();
    return {packed, suh_cat, svh_cat};
}

// Stored matrices of one projection, one per expert, into column blocks nb0 .. of out [E, n/128, k/128, 8, 2, K, 32].
void repack_experts(at::TensorList trellis, at::Tensor& out, int64_t nb0)
{
    const c10::cuda::CUDAGuard guard(out.device());
    device_sms(out.device().index());
    void* st = c10::cuda::getCurrentCUDAStream(out.device().index()).stream();
    TORCH_CHECK(out.dim() == 7 && out.is_contiguous() && (int64_t)trellis.size() == out.size(0), "out is [E, n/128, k/128, 8, 2, K, 32]");
    const int64_t k = out.size(2) * 128, K = out.size(5);
    for (size_t e = 0; e < trellis.size(); e++) {
        const at::Tensor t = trellis[e].to(out.device()).contiguous();
        TORCH_CHECK(t.dim() == 3 && t.size(0) * 16 == k && t.size(2) == 16 * K && t.size(1) / 8 + nb0 <= out.size(1),
                    "experts must share one shape and bitrate");
        uint32_t* dst = static_cast<uint32_t*>(out.mutable_data_ptr()) + (int64_t)e * out.stride(0) + nb0 * out.stride(1);
        check(exl3_repack(u16(t), (int)k, (int)t.size(1) * 16, (int)K, dst, st), "exl3_repack");
    }
}

// ------------------------------------------------------------------------------------------------ plain eager calls

// A dense CUDA tensor that asks nothing of the dispatcher: no subclass, no wrapper or lazy negation (keys beyond the ordinary ones), no
// gradient wanted.
bool plain_tensor(PyObject* o)
{
    if (!THPVariable_CheckExact(o)) return false;
    using c10::DispatchKey;
    static const uint64_t plain =
        c10::DispatchKeySet({DispatchKey::CUDA, DispatchKey::AutogradCUDA, DispatchKey::ADInplaceOrView, DispatchKey::AutocastCUDA}).raw_repr();
    const at::Tensor& t = THPVariable_Unpack(o);
    return t.is_cuda() && (t.key_set().raw_repr() & ~plain) == 0 && !(t.requires_grad() && c10::GradMode::is_enabled());
}

bool unpack_tensors(PyObject* o, std::vector<at::Tensor>& out)
{
    if (!PyList_CheckExact(o)) return false;
    const Py_ssize_t n = PyList_GET_SIZE(o);
    out.reserve(n);
    for (Py_ssize_t i = 0; i < n; i++) {
        if (!plain_tensor(PyList_GET_ITEM(o, i))) return false;
        out.push_back(THPVariable_Unpack(PyList_GET_ITEM(o, i)));
    }
    return true;
}

bool unpack_ints(PyObject* o, std::vector<int64_t>& out)
{
    if (!PyList_CheckExact(o)) return false;
    const Py_ssize_t n = PyList_GET_SIZE(o);
    out.reserve(n);
    for (Py_ssize_t i = 0; i < n; i++) {
        PyObject* v = PyList_GET_ITEM(o, i);
        if (!PyLong_CheckExact(v)) return false;
        int overflow = 0;
        out.push_back(PyLong_AsLongLongAndOverflow(v, &overflow));
        if (overflow) return false;
    }
    return true;
}

// The operator for what eager code passes: positional plain CUDA tensors, lists and ints, no gradients, and nothing that wants to see
// the call: dispatch modes, tracing and functional transforms (thread-local dispatch keys), modes over torch functions, profiler and
// other record-function callbacks.  None: not such a call, take the operator.
PyObject* direct_linear(PyObject*, PyObject* const* args, Py_ssize_t n)
{
    HANDLE_TH_ERRORS
    if (n != 11 || !plain_tensor(args[0]) || !PyLong_CheckExact(args[6])) Py_RETURN_NONE;
    if (!(c10::impl::tls_local_dispatch_key_set().included_ - c10::default_included_set).empty()) Py_RETURN_NONE;
    if (at::impl::torch_function_mode_enabled() || at::hasCallbacks()) Py_RETURN_NONE;
    const at::Tensor x = THPVariable_Unpack(args[0]);
    std::vector<at::Tensor> trellis, suh, svh, dense, sliced, weights;
    std::vector<int64_t> ends, codebooks, widths;
    if (!unpack_tensors(args[1], trellis) || !unpack_tensors(args[2], suh) || !unpack_tensors(args[3], svh) || !unpack_tensors(args[4], dense) ||
        !unpack_tensors(args[5], sliced) || !unpack_tensors(args[7], weights) || !unpack_ints(args[8], ends) || !unpack_ints(args[9], codebooks) ||
        !unpack_ints(args[10], widths))
        Py_RETURN_NONE;
    if (!dense.empty()) Py_RETURN_NONE;
    at::Tensor y;
    {
        const at::AutoDispatchBelowAutograd below;
        PyThreadState* state = PyEval_SaveThread();
        try {
            y = linear(x, trellis, suh, svh, dense, sliced, 0, weights, ends, codebooks, widths);
        } catch (...) {
            PyEval_RestoreThread(state);
            throw;
        }
        PyEval_RestoreThread(state);
    }
    return THPVariable_Wrap(std::move(y));
    END_HANDLE_TH_ERRORS
}

PyMethodDef direct_methods[] = {{"linear", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(direct_linear)), METH_FASTCALL, nullptr},
                                {nullptr, nullptr, 0, nullptr}};
PyModuleDef direct_module = {PyModuleDef_HEAD_INIT, "exl3_b200_direct", nullptr, -1, direct_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_exl3_b200_direct() { return PyModule_Create(&direct_module); }

TORCH_LIBRARY_FRAGMENT(exl3_b200, m)
{
    m.def("scratch(int kind, int device, int nbytes) -> Tensor", scratch);
    m.def("scratch_clear(int kind) -> ()", scratch_clear);
    m.def("knob(int which, int value) -> int", knob);
    m.def("prepare_group(Tensor[] trellis, Tensor[] suh, Tensor[] svh, int max_rows) -> (Tensor, Tensor, Tensor)");
    m.def("repack_experts(Tensor[] trellis, Tensor(a!) out, int nb0) -> ()");
    m.def("linear(Tensor x, Tensor[] trellis, Tensor[] suh, Tensor[] svh, Tensor[] dense, Tensor[] sliced, int sliced_min_rows, "
          "Tensor[] marlin_w, int[] marlin_ends, int[] codebooks, int[] out_widths) -> Tensor");
}

TORCH_LIBRARY_IMPL(exl3_b200, CUDA, m)
{
    m.impl("linear", linear);
    m.impl("prepare_group", prepare_group);
    m.impl("repack_experts", repack_experts);
}
