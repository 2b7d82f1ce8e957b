// Host side of the operators in C++: argument checks, allocation of results and scratch, and the call into
// the C ABI, one Python call per operator. The same steps through ctypes cost 20 to 60 us of interpreter
// time an operator (a twenty-argument foreign call, a workspace lookup, tensor attribute reads), which is
// more than most kernels of a mini-batch run for.
//
// Scratch comes from PyTorch's caching allocator on the current stream, so that calls on several streams
// or threads never share it.
#include <ATen/ATen.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/utils/pybind.h>

#include <optional>

#include "../../include/apt_b200.h"

namespace py = pybind11;
using at::Tensor;
using OptTensor = std::optional<Tensor>;

namespace {

struct AptFailure {
  int status;
};

void check(int status) {
  if (status != APT_OK) throw AptFailure{status};
}

void* stream() { return (void*)c10::cuda::getCurrentCUDAStream().stream(); }

[[noreturn]] void fail(const std::string& text) { throw std::runtime_error(text); }

int dtype_code(at::ScalarType t) {
  return t == at::kFloat ? APT_F32 : t == at::kBFloat16 ? APT_BF16 : t == at::kHalf ? APT_F16 : -1;
}

std::string dtype_name(const Tensor& t) {
  return std::string("torch.") + (t.scalar_type() == at::kDouble ? "float64" : t.scalar_type() == at::kFloat ? "float32"
         : t.scalar_type() == at::kLong ? "int64" : t.scalar_type() == at::kInt ? "int32" : t.scalar_type() == at::kHalf ? "float16"
         : t.scalar_type() == at::kBFloat16 ? "bfloat16" : c10::toString(t.scalar_type()));
}

// A contiguous CUDA tensor, of a given type where one is asked for.
Tensor cuda(const Tensor& t, const char* name) {
  if (!t.is_cuda()) fail(std::string(name) + " must be a CUDA tensor (apt_b200 has no CPU path)");
  return t.contiguous();
}
Tensor cuda(const Tensor& t, const char* name, at::ScalarType want, const char* want_name) {
  if (!t.is_cuda()) fail(std::string(name) + " must be a CUDA tensor (apt_b200 has no CPU path)");
  if (t.scalar_type() != want) fail(std::string(name) + " must have dtype " + want_name + ", got " + dtype_name(t));
  return t.contiguous();
}
Tensor ids(const Tensor& t, const char* name) { return cuda(t, name, at::kLong, "torch.int64"); }

const int64_t* ptr(const Tensor& t) { return t.numel() ? t.const_data_ptr<int64_t>() : nullptr; }
const void* data(const Tensor& t) { return t.numel() ? t.const_data_ptr() : nullptr; }
void* mut(const Tensor& t) { return t.numel() ? t.mutable_data_ptr() : nullptr; }

Tensor scratch(const Tensor& like, size_t bytes) { return at::empty({(int64_t)bytes}, like.options().dtype(at::kByte)); }

// ------------------------------------------------------------------------------------------ SpMM / SDDMM
Tensor spmm(int op, const Tensor& coo_row, const Tensor& coo_col, const OptTensor& input, const OptTensor& edata,
            const Tensor& coo_offset, const OptTensor& input_offset, const Tensor& output_offset) {
  const Tensor& given = input ? *input : *edata;
  const int code = dtype_code(given.scalar_type());
  if (code < 0) fail("spmm: unsupported dtype " + dtype_name(given));
  const Tensor row = ids(coo_row, "coo_row"), col = ids(coo_col, "coo_col");
  const Tensor eoff = ids(coo_offset, "coo_offset"), ooff = ids(output_offset, "output_offset");
  Tensor ioff, in, ed;
  if (input_offset) ioff = ids(*input_offset, "input_offset");
  if (input) in = cuda(*input, "input");
  if (edata) ed = input ? cuda(*edata, "edata", given.scalar_type(), dtype_name(given).c_str()) : cuda(*edata, "input");
  const int64_t edges = row.numel();
  // edge values may be [E, D], [E, H] or [E, H, 1]: one value per column or per head
  const int64_t per_edge = edata ? ed.numel() / std::max<int64_t>(edges, 1) : 0;
  const int64_t dim = input ? in.size(1) : per_edge;
  const int64_t edim = edata && edges ? per_edge : dim;
  int64_t shape[3];
  {
    py::gil_scoped_release nogil;   // other threads run while this one waits for the stream
    check(apt_spmm_probe(ptr(col), edges, ptr(eoff), ptr(ooff), (int)eoff.numel() - 1, shape, stream()));
  }
  Tensor out = at::empty({shape[0], dim}, given.options());
  Tensor ws;
  size_t bytes = 0;
  if (shape[1] != 0 && edges > 0 && shape[0] > 0) {
    bytes = apt_spmm_workspace_bytes(shape[0], edges);
    ws = scratch(out, bytes);
  }
  check(apt_spmm_sum_known(op, code, ptr(row), ptr(col), edges, input ? data(in) : nullptr, edata ? data(ed) : nullptr, edim,
                           dim, ptr(eoff), input_offset ? ptr(ioff) : nullptr, ptr(ooff), (int)eoff.numel() - 1, shape[0],
                           (int)shape[1], (int)shape[2], mut(out), bytes ? ws.mutable_data_ptr() : nullptr, bytes, stream()));
  return out;
}

Tensor sddmm(int op, const Tensor& coo_row, const Tensor& coo_col, const Tensor& lhs_in, const Tensor& rhs_in,
             const Tensor& coo_offset, const Tensor& lhs_offset, const Tensor& rhs_offset) {
  const int code = dtype_code(lhs_in.scalar_type());
  if (code < 0 || rhs_in.scalar_type() != lhs_in.scalar_type())
    fail("sddmm: unsupported dtypes " + dtype_name(lhs_in) + "/" + dtype_name(rhs_in));
  const Tensor row = ids(coo_row, "coo_row"), col = ids(coo_col, "coo_col");
  const Tensor lhs = cuda(lhs_in, "lhs"), rhs = cuda(rhs_in, "rhs");
  const Tensor eoff = ids(coo_offset, "coo_offset"), loff = ids(lhs_offset, "lhs_offset"), roff = ids(rhs_offset, "rhs_offset");
  Tensor out = at::empty({row.numel(), lhs.size(1)}, lhs.options());
  check(apt_sddmm(op, code, ptr(row), ptr(col), row.numel(), data(lhs), data(rhs), lhs.size(1), ptr(eoff), ptr(loff),
                  ptr(roff), (int)eoff.numel() - 1, mut(out), stream()));
  return out;
}

}  // namespace

PYBIND11_MODULE(_native, m) {
  m.doc() = "operators of apt_b200 over libapt_b200's C ABI";
  py::register_exception_translator([](std::exception_ptr p) {
    try {
      if (p) std::rethrow_exception(p);
    } catch (const AptFailure& e) {
      // _lib.AptError(status, text), what the ctypes path raises
      py::object cls = py::module_::import("apt_b200._lib").attr("AptError");
      py::object err = cls(e.status, py::bytes(apt_last_error()).attr("decode")("utf-8", "replace"));
      PyErr_SetObject(cls.ptr(), err.ptr());
    }
  });
  m.def("spmm", &spmm);
  m.def("sddmm", &sddmm);
}
