// Host side of the operators in C++: argument checks, allocation of results and scratch, and the call into
// the C ABI, one Python call per operator. The same steps through ctypes cost 20 to 60 us of interpreter
// time an operator (a twenty-argument foreign call, a workspace lookup, tensor attribute reads), which is
// more than most kernels of a mini-batch run for.
//
// Scratch comes from PyTorch's caching allocator on the current stream, so that calls on several streams
// or threads never share it.
#include <ATen/ATen.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/utils/pybind.h>

#include <optional>

#include "../../include/apt_b200.h"

namespace py = pybind11;
using at::Tensor;
using OptTensor = std::optional<Tensor>;

namespace {

// A std::exception: the autograd engine's threads carry nothing else over to the caller.
struct AptFailure : std::runtime_error {
  AptFailure(int code, const char* text) : std::runtime_error(text), status(code) {}
  int status;
};

void check(int status) {
  if (status != APT_OK) throw AptFailure(status, apt_last_error());
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

// The status flags are the last word of the state's word block.
int32_t* status_word(const Tensor& words) { return (int32_t*)(words.mutable_data_ptr<int64_t>() + words.numel() - 1); }

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

// ------------------------------------------------------------------------------------------ row movers
// Rows of the device cache or of the page-locked host table (`column` is the host table's column offset in elements).
Tensor gather(const Tensor& node_id, const Tensor& pos_map, const Tensor& dev_feats, const Tensor& uva_feats, int64_t num_nodes,
              int64_t column, const Tensor& words) {
  const Tensor id = ids(node_id, "node_id");
  const int64_t n = id.numel(), size = dev_feats.element_size(), dim = dev_feats.size(1);
  Tensor out = at::empty({n, dim}, dev_feats.options());
  if (n == 0) return out;
  const size_t bytes = apt_gather_workspace_bytes(n);
  const Tensor ws = scratch(out, bytes);
  check(apt_gather_rows(ptr(id), n, nullptr, ptr(pos_map), num_nodes, data(dev_feats), dev_feats.size(0), dim * size,
                        data(uva_feats), uva_feats.size(0), uva_feats.size(1) * size, column * size, mut(out),
                        ws.mutable_data_ptr(), bytes, status_word(words), stream()));
  return out;
}

Tensor rows_gather(const Tensor& inp, const Tensor& index) {
  const Tensor in = cuda(inp, "inp"), at = ids(index, "index");
  Tensor out = at::empty({at.numel(), in.size(1)}, in.options());
  check(apt_rows_gather(data(in), ptr(at), at.numel(), in.size(1) * in.element_size(), mut(out), stream()));
  return out;
}

Tensor rows_scatter(const Tensor& inp, const Tensor& index, int64_t num_out_rows) {
  const Tensor in = cuda(inp, "inp"), at = ids(index, "index");
  Tensor out = at.numel() == num_out_rows ? at::empty({num_out_rows, in.size(1)}, in.options())
                                          : at::zeros({num_out_rows, in.size(1)}, in.options());
  check(apt_rows_scatter(data(in), ptr(at), at.numel(), in.size(1) * in.element_size(), mut(out), stream()));
  return out;
}

// ---------------------------------------------------------------------------------------- attention block
struct GatShape {
  int code;
  int64_t edges, num_src, num_dst, heads, head_dim;
};

GatShape gat_shape(const char* who, const Tensor& row, const Tensor& ft, const Tensor& el, const Tensor& er, int64_t num_dst) {
  const int code = dtype_code(ft.scalar_type());
  if (code < 0 || el.scalar_type() != ft.scalar_type() || er.scalar_type() != ft.scalar_type())
    fail(std::string(who) + ": unsupported dtypes " + dtype_name(ft) + "/" + dtype_name(el) + "/" + dtype_name(er));
  const int64_t num_src = ft.size(0);
  const int64_t heads = num_src ? el.numel() / std::max<int64_t>(num_src, 1) : er.numel() / std::max<int64_t>(num_dst, 1);
  return {code, row.numel(), num_src, num_dst, heads, ft.numel() / std::max<int64_t>(num_src * heads, 1)};
}

// Results of the forward: sums, attention (when asked for) and the edge buffer that a backward of the same block can use.
std::tuple<Tensor, Tensor, Tensor> gat_forward(const Tensor& coo_row, const Tensor& coo_col, const Tensor& ft_in, const Tensor& el_in,
                                               const Tensor& er_in, int64_t num_dst, double slope, bool want_attention,
                                               const Tensor& words) {
  const Tensor row = ids(coo_row, "coo_row"), col = ids(coo_col, "coo_col");
  const Tensor ft = cuda(ft_in, "ft"), el = cuda(el_in, "el"), er = cuda(er_in, "er");
  const GatShape g = gat_shape("gat_edge_softmax_sum", row, ft, el, er, num_dst);
  Tensor out = at::empty({num_dst, g.heads, g.head_dim}, ft.options()), attn;
  if (want_attention) attn = at::empty({g.edges, g.heads, 1}, ft.options());
  const size_t bytes = apt_gat_edges_bytes(num_dst, g.edges, (int)g.heads);
  const Tensor edges = scratch(ft, bytes);
  check(apt_gat_forward(g.code, ptr(row), ptr(col), g.edges, data(ft), data(el), data(er), (int)g.heads, g.head_dim, (float)slope,
                        num_dst, mut(out), want_attention ? mut(attn) : nullptr, edges.mutable_data_ptr(), bytes,
                        status_word(words), stream()));
  return {out, attn, edges};
}

std::tuple<Tensor, Tensor, Tensor> gat_backward(const Tensor& coo_row, const Tensor& coo_col, const Tensor& ft_in,
                                                const Tensor& el_in, const Tensor& er_in, const Tensor& grad_in, double slope,
                                                const Tensor& words, const OptTensor& edges_of_forward) {
  const Tensor row = ids(coo_row, "coo_row"), col = ids(coo_col, "coo_col");
  const Tensor ft = cuda(ft_in, "ft"), el = cuda(el_in, "el"), er = cuda(er_in, "er"), grad = cuda(grad_in, "grad_out");
  if (grad.scalar_type() != ft.scalar_type()) fail("gat_edge_softmax_sum_backward: unsupported or mixed dtypes");
  const GatShape g = gat_shape("gat_edge_softmax_sum_backward", row, ft, el, er, grad.size(0));
  Tensor grad_ft = at::empty(ft.sizes(), ft.options()), grad_el = at::empty(el.sizes(), el.options()),
         grad_er = at::empty(er.sizes(), er.options());
  const size_t edges_bytes = apt_gat_edges_bytes(g.num_dst, g.edges, (int)g.heads);
  const Tensor edges = edges_of_forward ? *edges_of_forward : scratch(ft, edges_bytes);
  const size_t bytes = apt_gat_backward_workspace_bytes(g.num_src, g.edges, (int)g.heads);
  const Tensor ws = scratch(ft, bytes);
  check(apt_gat_backward(g.code, ptr(row), ptr(col), g.edges, data(ft), data(el), data(er), data(grad), (int)g.heads, g.head_dim,
                         (float)slope, g.num_src, g.num_dst, mut(grad_ft), mut(grad_el), mut(grad_er), edges.mutable_data_ptr(),
                         edges_bytes, edges_of_forward ? 1 : 0, ws.mutable_data_ptr(), bytes, status_word(words), stream()));
  return {grad_ft, grad_el, grad_er};
}

// The forward's ranges and weights are saved with its inputs: the backward of a training step starts from them.
struct GatFunction : public torch::autograd::Function<GatFunction> {
  static Tensor forward(torch::autograd::AutogradContext* ctx, const Tensor& row, const Tensor& col, const Tensor& ft,
                        const Tensor& el, const Tensor& er, int64_t num_dst, double slope, const Tensor& words) {
    auto [out, attn, edges] = gat_forward(row, col, ft, el, er, num_dst, slope, false, words);
    ctx->save_for_backward({row, col, ft, el, er});
    ctx->saved_data["slope"] = slope;
    ctx->saved_data["words"] = words;
    ctx->saved_data["edges"] = edges;
    return out;
  }
  static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx, torch::autograd::variable_list grads) {
    const auto v = ctx->get_saved_variables();
    auto [g_ft, g_el, g_er] = gat_backward(v[0], v[1], v[2], v[3], v[4], grads[0], ctx->saved_data["slope"].toDouble(),
                                           ctx->saved_data["words"].toTensor(), ctx->saved_data["edges"].toTensor());
    return {Tensor(), Tensor(), g_ft, g_el, g_er, Tensor(), Tensor(), Tensor()};
  }
};

}  // namespace

PYBIND11_MODULE(_native, m) {
  m.doc() = "operators of apt_b200 over libapt_b200's C ABI";
  py::register_exception_translator([](std::exception_ptr p) {
    try {
      if (p) std::rethrow_exception(p);
    } catch (const AptFailure& e) {
      // _lib.AptError(status, text), what the ctypes path raises
      py::object cls = py::module_::import("apt_b200._lib").attr("AptError");
      py::object err = cls(e.status, py::bytes(e.what()).attr("decode")("utf-8", "replace"));
      PyErr_SetObject(cls.ptr(), err.ptr());
    }
  });
  m.def("spmm", &spmm);
  m.def("sddmm", &sddmm);
  m.def("gather", &gather);
  m.def("rows_gather", &rows_gather);
  m.def("rows_scatter", &rows_scatter);
  m.def("gat_forward", [](const Tensor& row, const Tensor& col, const Tensor& ft, const Tensor& el, const Tensor& er,
                          int64_t num_dst, double slope, bool want_attention, const Tensor& words) {
    auto [out, attn, edges] = gat_forward(row, col, ft, el, er, num_dst, slope, want_attention, words);
    return std::make_tuple(out, attn);
  });
  m.def("gat_backward", [](const Tensor& row, const Tensor& col, const Tensor& ft, const Tensor& el, const Tensor& er,
                           const Tensor& grad, double slope, const Tensor& words) {
    return gat_backward(row, col, ft, el, er, grad, slope, words, std::nullopt);
  });
  m.def("gat_apply", [](const Tensor& row, const Tensor& col, const Tensor& ft, const Tensor& el, const Tensor& er,
                        int64_t num_dst, double slope, const Tensor& words) {
    return GatFunction::apply(row, col, ft, el, er, num_dst, slope, words);
  });
}
