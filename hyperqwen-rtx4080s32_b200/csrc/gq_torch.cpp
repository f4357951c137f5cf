// Native call path of a packed run: the Python extension module `_gq_torch`.
//
// GGUFLinearMethod.apply is called once per linear layer and token step.  Going through the torch custom op and ctypes
// costs 46 us of host time per call on an idle GPU (boxing nine arguments, three of them lists of tensors, a Python
// kernel, two allocations from Python and a ctypes call with fifteen arguments), six times what the GPU needs for a small
// layer.  A Run keeps what does not change between calls — the packed buffer, the descriptor tables, the split per
// row count — and does the call's host work here: output and scratch from torch's caching allocator on the current
// stream, then the C ABI of include/gq_b200.h.
//
// forward() answers None for whatever is not the plain case (dtype, layout, device, autograd, torch modes, tracing, function
// transforms, a call of zero rows); the caller then takes the general path, which also states the errors.
#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <pybind11/pybind11.h>
#include <pybind11/stl.h>
#include <torch/csrc/utils/pybind.h>
#include <torch/csrc/autograd/python_variable.h>
#include <string>
#include <vector>
#include "../../include/gq_b200.h"

namespace py = pybind11;

namespace {

const char *error_text(int rc) {
    switch (rc) {
        case GQ_ERR_TYPE: return "unsupported GGML type";
        case GQ_ERR_SHAPE: return "bad shape (K not a multiple of 256, negative size, or M over the limit)";
        case GQ_ERR_ARG: return "bad argument (null or misaligned pointer, inconsistent sizes)";
        case GQ_ERR_WORKSPACE: return "workspace too small";
        case GQ_ERR_CUDA: return "CUDA runtime error";
        case GQ_ERR_LIMIT: return "size beyond a fixed maximum";
        default: return "unknown error";
    }
}
PyObject *g_error = PyExc_RuntimeError;      // GqError of _lib.py, kept for the life of the process

void raise_if(int64_t rc, const char *what) {
    if (rc >= 0) return;
    std::string msg = std::string(what) + " failed (" + std::to_string(rc) + "): " + error_text((int)rc);
    if (rc == GQ_ERR_CUDA) msg += std::string(": ") + gq_last_cuda_error();
    PyErr_SetString(g_error, msg.c_str());
    throw py::error_already_set();
}

// what a call of the C ABI returned, kept until the GIL is held again
struct Status {
    int64_t rc = 0;
    const char *what = "";
    void check() const { raise_if(rc, what); }
};

// Whether nothing stands between a torch call and its kernel on this thread: no dispatch or function mode, no tracer, no
// function transform (vmap, jvp).  Each of them shows in the thread's own dispatch keys or as a function mode.
inline bool plain_thread() {
    const uint64_t keys = c10::impl::tls_local_dispatch_key_set().included_.raw_repr();
    return !(keys & ~c10::default_included_set.raw_repr()) && !at::impl::torch_function_mode_enabled();
}
// Whether a tensor is what its memory says: a dense CUDA tensor with no key beside the usual ones (negative view, zero tensor,
// a transform's or a mode's wrapper)
inline bool plain_tensor(const at::Tensor &t) {
    constexpr c10::DispatchKeySet usual({c10::DispatchKey::CUDA, c10::DispatchKey::AutogradCUDA, c10::DispatchKey::ADInplaceOrView,
                                         c10::DispatchKey::AutocastCUDA});
    return t.is_cuda() && !(t.key_set().raw_repr() & ~usual.raw_repr()) && !t.has_names();
}
inline bool plain_cuda(const at::Tensor &t, int device) { return plain_tensor(t) && t.get_device() == device && !t.requires_grad(); }

// Whether two sets of bf16 rows may share memory: `cols` columns each, rows and row strides of their own.  Rows of one stride that lie beside each
// other, as two column ranges of one buffer do, do not.
inline bool may_overlap(const void *a, int64_t rows_a, int64_t ld_a, const void *b, int64_t rows_b, int64_t ld_b, int64_t cols) {
    const int64_t pa = (int64_t)((uintptr_t)a / 2), pb = (int64_t)((uintptr_t)b / 2);
    if (pa + (rows_a - 1) * ld_a + cols <= pb || pb + (rows_b - 1) * ld_b + cols <= pa) return false;
    if (ld_a != ld_b) return true;
    const int64_t off = ((pb - pa) % ld_a + ld_a) % ld_a;
    return off < cols || ld_a - off < cols;
}

class Run {
  public:
    Run(at::Tensor packed, std::vector<at::Tensor> descs, std::vector<int64_t> splits, std::vector<int64_t> n_outs, std::vector<int64_t> types,
        int64_t nb, std::vector<int64_t> split_of_rows, int64_t decode_rows, int64_t pre_rows)
        : packed_(std::move(packed)), descs_(std::move(descs)), splits_(std::move(splits)), K_(nb * 256), decode_rows_(decode_rows),
          pre_rows_(pre_rows), device_(packed_.get_device()) {
        std::vector<int32_t> t32(types.begin(), types.end());
        raise_if(info_ = gq_run_info((int)t32.size(), t32.data()), "gq_run_info");
        const int order = t32.size() == n_outs.size() ? gq_run_order((int)t32.size(), t32.data(), n_outs.data()) : 0;      // a hint
        raise_if(order, "gq_run_order");
        info_ |= order;
        for (int64_t n : n_outs) n_total_ += n;
        one_ = index_of(1);
        for (int64_t s : split_of_rows) by_rows_.push_back(index_of(s));
        TORCH_CHECK((int64_t)by_rows_.size() > decode_rows_, "split_of_rows covers 0..decode_rows");
    }

    // x [..., K] -> [..., n_total]; None: not the plain case
    PyObject *forward(py::handle x) { return call(x, 0, nullptr, nullptr, nullptr, 0.0f); }
    PyObject *forward_silu_mul(py::handle x) { return call(x, 1, nullptr, nullptr, nullptr, 0.0f); }
    PyObject *forward_add_rms_norm(py::handle x, const at::Tensor &weight, c10::optional<at::Tensor> residual,
                                   c10::optional<at::Tensor> residual_out, double eps) {
        return call(x, 2, &weight, residual.has_value() ? &*residual : nullptr, residual_out.has_value() ? &*residual_out : nullptr, (float)eps);
    }

  private:
    // the table of a split, or of the largest below it that there is (split 1 always is)
    int index_of(int64_t split) const {
        int best = -1;
        for (size_t i = 0; i < splits_.size(); ++i)
            if (splits_[i] <= split && (best < 0 || splits_[i] > splits_[best])) best = (int)i;
        return best < 0 ? 0 : best;
    }
    static PyObject *none() { Py_RETURN_NONE; }

    PyObject *call(py::handle xh, int pre, const at::Tensor *weight, const at::Tensor *residual, const at::Tensor *residual_out, float eps) {
        if (!THPVariable_CheckExact(xh.ptr()) || !plain_thread()) return none();
        const at::Tensor x = THPVariable_Unpack(xh.ptr());      // a reference of its own: the GIL is released below
        const int64_t width = pre == 1 ? 2 * K_ : K_, nd = x.dim();
        if (nd < 1 || !plain_cuda(x, device_) || x.scalar_type() != at::kBFloat16 || x.size(-1) != width || x.stride(-1) != 1) return none();
        int64_t m = 1, ldx = width;
        if (nd == 2) { m = x.size(0); ldx = x.stride(0); if (m == 1 && ldx < width) ldx = width; }
        else { if (!x.is_contiguous()) return none(); for (int64_t i = 0; i + 1 < nd; ++i) m *= x.size(i); }
        if (m <= 0 || n_total_ == 0 || ldx < width) return none();
        if (pre) {
            if (pre == 2) {
                if (!plain_cuda(*weight, device_) || weight->scalar_type() != at::kBFloat16 || weight->numel() != K_ || !weight->is_contiguous()) return none();
                if ((residual == nullptr) != (residual_out == nullptr)) return none();
                if (residual) {
                    for (const at::Tensor *r : {residual, residual_out})
                        if (!plain_cuda(*r, device_) || r->scalar_type() != at::kBFloat16 || r->dim() != 2 || r->size(0) != m || r->size(1) != K_ ||
                            r->stride(1) != 1) return none();
                    if (residual->stride(0) != residual_out->stride(0)) return none();
                }
            }
        }
        const bool wide = m > decode_rows_, apart = pre && m > pre_rows_;       // apart: the op is a launch of its own
        if (apart && residual) {
            // the new residual may take the old one's place; where it shares other memory that the kernel reads, the general path reads all of it first
            const void *out = residual_out->data_ptr();
            const int64_t ld = residual_out->stride(0);
            if (ld < K_ || (out != residual->data_ptr() && may_overlap(out, m, ld, residual->data_ptr(), m, ld, K_)) ||
                may_overlap(out, m, ld, x.data_ptr(), m, ldx, K_) || may_overlap(out, m, ld, weight->data_ptr(), 1, K_, K_)) return none();
        }
        if (wide && !apart && ((ldx & 7) || (reinterpret_cast<uintptr_t>(x.data_ptr()) & 15))) return none();
        at::Tensor y;
        Status status;
        {
            // the allocator and a full launch queue can keep the caller waiting: other Python threads go on meanwhile
            py::gil_scoped_release unlocked;
            status = launch(x, m, ldx, pre, weight, residual, residual_out, eps, y);
        }
        status.check();
        return THPVariable_Wrap(std::move(y));
    }

    // the call itself, without the GIL: output and scratch, then the C ABI
    Status launch(const at::Tensor &x, int64_t m, int64_t ldx, int pre, const at::Tensor *weight, const at::Tensor *residual,
                  const at::Tensor *residual_out, float eps, at::Tensor &y) const {
        const bool wide = m > decode_rows_;
        const void *in = x.data_ptr();
        c10::DataPtr pre_out;
        c10::cuda::CUDAGuard guard((c10::DeviceIndex)device_);
        void *stream = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)device_).stream();
        at::DimVector sizes(x.sizes().begin(), x.sizes().end());
        sizes.back() = n_total_;
        y = at::detail::empty_cuda(sizes, at::kBFloat16, x.device(), c10::nullopt);
        auto *alloc = c10::cuda::CUDACachingAllocator::get();
        if (pre && m > pre_rows_) {
            pre_out = alloc->allocate((size_t)(m * K_ * 2));
            const int rc = gq_pre_op(in, m, K_, ldx, pre, weight ? weight->data_ptr() : nullptr, residual ? residual->data_ptr() : nullptr,
                                     residual_out ? residual_out->data_ptr() : nullptr, residual ? residual->stride(0) : 0, eps, pre_out.get(), K_, stream);
            if (rc < 0) return {rc, "gq_pre_op"};
            in = pre_out.get(); ldx = K_; pre = 0;
        }
        if (wide) {
            const int64_t n_desc = descs_[one_].size(0), need = gq_prefill_workspace_bytes(m, K_, n_total_, n_desc);
            if (need < 0) return {need, "gq_prefill_workspace_bytes"};
            c10::DataPtr ws = alloc->allocate((size_t)need + 1024);
            const uintptr_t base = (reinterpret_cast<uintptr_t>(ws.get()) + 1023) & ~(uintptr_t)1023;
            return {gq_gemm_prefill(in, m, K_, ldx, packed_.data_ptr(), (const int32_t *)descs_[one_].data_ptr(), n_desc, info_, y.data_ptr(),
                                    n_total_, n_total_, (void *)base, need, stream), "gq_gemm_prefill"};
        }
        const int i = by_rows_[m];
        const int split = (int)splits_[i];
        const at::Tensor &d = descs_[i];
        const int64_t need = gq_workspace_bytes(m, K_, n_total_, split);
        if (need < 0) return {need, "gq_workspace_bytes"};
        c10::DataPtr ws = alloc->allocate((size_t)need);
        if (pre)
            return {gq_gemv_grouped_pre(x.data_ptr(), m, K_, ldx, pre, weight ? weight->data_ptr() : nullptr, residual ? residual->data_ptr() : nullptr,
                                        residual_out ? residual_out->data_ptr() : nullptr, residual ? residual->stride(0) : 0, eps, packed_.data_ptr(),
                                        (const int32_t *)d.data_ptr(), d.size(0), split, info_, y.data_ptr(), n_total_, n_total_, ws.get(), need, stream),
                    "gq_gemv_grouped_pre"};
        // 15: nobody reads this workspace's status word, so a small launch may do without the preparation kernel
        return {gq_gemv_grouped_phases(in, m, K_, ldx, packed_.data_ptr(), (const int32_t *)d.data_ptr(), d.size(0), split, info_,
                                       y.data_ptr(), n_total_, n_total_, ws.get(), need, stream, 15), "gq_gemv_grouped"};
    }

    at::Tensor packed_;
    std::vector<at::Tensor> descs_;
    std::vector<int64_t> splits_;
    std::vector<int> by_rows_;       // rows -> index into descs_
    int64_t K_, n_total_ = 0, decode_rows_, pre_rows_;
    int device_, info_ = 0, one_ = 0;
};

// The load-time calls, on arguments that ops.py has checked: device and stream of the tensor, then the C ABI.
void *stream_of(const at::Tensor &t) { return c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)t.get_device()).stream(); }

void repack(const at::Tensor &raw, int64_t n_out, int64_t type, int64_t nb, const at::Tensor &out) {
    Status status;
    {
        py::gil_scoped_release unlocked;
        c10::cuda::CUDAGuard guard((c10::DeviceIndex)raw.get_device());
        status = {gq_repack((int)type, raw.data_ptr(), n_out, nb * 256, raw.stride(0), out.data_ptr(), stream_of(raw)), "gq_repack"};
    }
    status.check();
}
at::Tensor dequantize(const at::Tensor &tiles, int64_t n_out, int64_t k, int64_t type, bool bf16) {
    Status status;
    at::Tensor out;
    {
        py::gil_scoped_release unlocked;
        c10::cuda::CUDAGuard guard((c10::DeviceIndex)tiles.get_device());
        out = at::detail::empty_cuda({n_out, k}, bf16 ? at::kBFloat16 : at::kFloat, tiles.device(), c10::nullopt);
        status = {gq_dequant((int)type, tiles.data_ptr(), n_out, k, out.data_ptr(), bf16 ? 1 : 0, k, stream_of(tiles)), "gq_dequant"};
    }
    status.check();
    return out;
}
// waits for the caller's stream on the tensor's device; one that is being captured has nothing to wait for
void finish(const at::Tensor &t) {
    py::gil_scoped_release unlocked;
    c10::cuda::CUDAGuard guard((c10::DeviceIndex)t.get_device());
    if (c10::cuda::currentStreamCaptureStatusMayInitCtx() == c10::cuda::CaptureStatus::None)
        c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)t.get_device()).synchronize();
}
void build_descs(const std::vector<int32_t> &types, const std::vector<int64_t> &n_outs, int64_t k, const std::vector<int32_t> &splits, const at::Tensor &out) {
    Status status;
    {
        py::gil_scoped_release unlocked;
        c10::cuda::CUDAGuard guard((c10::DeviceIndex)out.get_device());
        status = {gq_build_descs_device((int)types.size(), types.data(), n_outs.data(), k, (int)splits.size(), splits.data(), (int32_t *)out.data_ptr(),
                                        stream_of(out)), "gq_build_descs_device"};
    }
    status.check();
}

// rows `ids` of a raw table -> weights; None: not the plain case
PyObject *dequantize_rows(py::handle rawh, int64_t type, py::handle idsh, bool bf16) {
    if (!THPVariable_CheckExact(rawh.ptr()) || !THPVariable_CheckExact(idsh.ptr()) || !plain_thread()) Py_RETURN_NONE;
    const at::Tensor raw = THPVariable_Unpack(rawh.ptr()), ids = THPVariable_Unpack(idsh.ptr());
    const int B = gq_bytes_per_256((int)type);
    if (!plain_tensor(raw) || !plain_tensor(ids) || raw.scalar_type() != at::kByte || raw.dim() != 2 || raw.stride(1) != 1 || raw.stride(0) < raw.size(1) || raw.size(0) == 0 || B == 0 || raw.size(1) == 0 ||
        raw.size(1) % B || ids.get_device() != raw.get_device() || !ids.is_contiguous() || ids.numel() == 0 ||
        (ids.scalar_type() != at::kLong && ids.scalar_type() != at::kInt)) Py_RETURN_NONE;
    const int64_t K = raw.size(1) / B * 256;
    at::DimVector sizes(ids.sizes().begin(), ids.sizes().end());
    sizes.push_back(K);
    at::Tensor out;
    Status status;
    {
        py::gil_scoped_release unlocked;
        c10::cuda::CUDAGuard guard((c10::DeviceIndex)raw.get_device());
        out = at::detail::empty_cuda(sizes, bf16 ? at::kBFloat16 : at::kFloat, raw.device(), c10::nullopt);
        status = {gq_dequant_rows((int)type, raw.data_ptr(), raw.size(0), K, raw.stride(0), ids.data_ptr(), ids.scalar_type() == at::kLong ? 8 : 4,
                                  ids.numel(), out.data_ptr(), bf16 ? 1 : 0, K, stream_of(raw)), "gq_dequant_rows"};
    }
    status.check();
    return THPVariable_Wrap(std::move(out));
}

}  // namespace

PYBIND11_MODULE(_gq_torch, m) {
    m.def("set_error_type", [](py::object e) { g_error = e.release().ptr(); });
    m.def("repack", &repack);
    m.def("dequantize", &dequantize);
    m.def("build_descs", &build_descs);
    m.def("finish", &finish);
    m.def("dequantize_rows", [](py::handle raw, int64_t type, py::handle ids, bool bf16) {
        return py::reinterpret_steal<py::object>(dequantize_rows(raw, type, ids, bf16));
    });
    py::class_<Run>(m, "Run")
        .def(py::init<at::Tensor, std::vector<at::Tensor>, std::vector<int64_t>, std::vector<int64_t>, std::vector<int64_t>, int64_t, std::vector<int64_t>,
                      int64_t, int64_t>())
        .def("forward", [](Run &r, py::handle x) { return py::reinterpret_steal<py::object>(r.forward(x)); })
        .def("forward_silu_mul", [](Run &r, py::handle x) { return py::reinterpret_steal<py::object>(r.forward_silu_mul(x)); })
        .def("forward_add_rms_norm", [](Run &r, py::handle x, const at::Tensor &w, c10::optional<at::Tensor> res, c10::optional<at::Tensor> out, double eps) {
            return py::reinterpret_steal<py::object>(r.forward_add_rms_norm(x, w, res, out, eps));
        });
}
