// Host side of the operators in C++: argument checks, allocation of results and scratch, and the call into
// the C ABI, one Python call per operator. The same steps through ctypes cost 20 to 60 us of interpreter
// time an operator (a twenty-argument foreign call, a workspace lookup, tensor attribute reads), which is
// more than most kernels of a mini-batch run for.
//
// Scratch comes from PyTorch's caching allocator on the current stream, so that calls on several streams
// or threads never share it.
#include <ATen/ATen.h>
#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime_api.h>
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
// Scratch that a call does without where there is none: undefined then.
Tensor room_for(const Tensor& like, size_t bytes) {
  if (!bytes) return Tensor();
  try {
    return scratch(like, bytes);
  } catch (const c10::OutOfMemoryError&) {
    return Tensor();
  }
}

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
  int64_t shape[4] = {0, -1, 0, 0};
  if (ooff.numel() > eoff.numel()) {
    shape[0] = ooff[-1].item<int64_t>();        // further rows behind the last segment's: the block is looked over with them
  } else {
    py::gil_scoped_release nogil;   // other threads run while this one waits for the stream
    const bool may_widen = op == 0 && input && apt_spmm_widened_bytes(code, edges, in.size(0), dim, 2) > 0;
    check(apt_spmm_probe_rows(ptr(col), edges, ptr(eoff), ptr(ooff), (int)eoff.numel() - 1, may_widen, shape, stream()));
  }
  Tensor out = at::empty({shape[0], dim}, given.options());
  Tensor ws;
  size_t bytes = 0;
  if (shape[1] != 0 && edges > 0 && shape[0] > 0) {
    bytes = apt_spmm_workspace_bytes(shape[0], edges);
    ws = scratch(out, bytes);
  }
  const int mode = shape[1] == 2 && !shape[3] ? 3 : (int)shape[1];      // 3: in no order, and no row with very many of the edges
  const size_t wide_bytes = op == 0 && input && shape[0] > 0 ? apt_spmm_widened_bytes(code, edges, in.size(0), dim, mode) : 0;
  const Tensor wide = room_for(out, wide_bytes);
  if (wide.defined()) {
    check(apt_spmm_copy_u_widened(code, ptr(row), ptr(col), edges, data(in), in.size(0), dim, ptr(eoff), ptr(ioff), ptr(ooff),
                                  (int)eoff.numel() - 1, shape[0], mode, (int)shape[2], mut(out), wide.mutable_data_ptr(),
                                  wide_bytes, bytes ? ws.mutable_data_ptr() : nullptr, bytes, stream()));
    return out;
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
  if (n <= apt_gather_static_max_rows()) {      // the same launch without a workspace, which it does not use
    check(apt_gather_rows_static(ptr(id), n, ptr(pos_map), num_nodes, data(dev_feats), dev_feats.size(0), dim * size, data(uva_feats),
                                 uva_feats.size(0), uva_feats.size(1) * size, column * size, mut(out), status_word(words), stream()));
    return out;
  }
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

// ---------------------------------------------------------------------------- feature shuffles of a world of one
void cuda_ok(cudaError_t e, const char* what) {
  if (e != cudaSuccess) fail(std::string(what) + ": " + cudaGetErrorString(e));
}

// What travels nowhere still changes its order.
Tensor feat_shuffle_local(const Tensor& inputs, const Tensor& recv_offset, const Tensor& permutation, int64_t feat_dim, bool fwd) {
  if (dtype_code(inputs.scalar_type()) < 0) fail("feat_shuffle: unsupported dtype " + dtype_name(inputs));
  const Tensor in = cuda(inputs, "inputs");
  ids(permutation, "permutation");
  const int64_t rows = in.numel() / feat_dim;
  const Tensor flat = in.dim() == 2 && in.size(1) == feat_dim ? in : in.view({rows, feat_dim});
  return fwd ? rows_gather(flat, permutation) : rows_scatter(flat, permutation, recv_offset[-1].item<int64_t>());
}

// The parts' sizes are checked and each part is one copy.
Tensor sp_feat_shuffle_local(const Tensor& inputs, const Tensor& send_sizes, const Tensor& recv_sizes, int64_t total_recv,
                             int64_t expand, bool with_dst) {
  if (dtype_code(inputs.scalar_type()) < 0) fail("sp_feat_shuffle: unsupported dtype " + dtype_name(inputs));
  const Tensor in = cuda(inputs, "inputs");
  const int64_t rows = in.numel() / expand;
  if (rows * expand != in.numel()) fail("sp_feat_shuffle: the input is no whole number of rows");
  Tensor out = at::empty({total_recv, expand}, in.options());
  const Tensor send = send_sizes.to(at::kCPU, at::kLong).contiguous(), recv = recv_sizes.to(at::kCPU, at::kLong).contiguous();
  const auto sum = [](const Tensor& t, int64_t first, int64_t step) {
    const int64_t* const v = t.const_data_ptr<int64_t>();
    int64_t total = 0;
    for (int64_t k = first; k < t.numel(); k += step) total += v[k];
    return total;
  };
  const int64_t step = with_dst ? 3 : 2;
  const int64_t sent_dst = with_dst ? sum(send, 0, step) : 0, got_dst = with_dst ? sum(recv, 0, step) : 0;
  const int64_t sent = sum(send, step - 1, step), got = sum(recv, step - 1, step);
  if (sent_dst + sent != rows || got_dst + got != total_recv) fail("sp_feat_shuffle: sizes do not add up to the rows given");
  if (sent_dst != got_dst || sent != got) fail("sp_feat_shuffle: one rank receives what it sends");
  if (in.nbytes())      // the parts follow one another on both sides
    cuda_ok(cudaMemcpyAsync(out.mutable_data_ptr(), in.const_data_ptr(), in.nbytes(), cudaMemcpyDeviceToDevice,
                            (cudaStream_t)stream()), "cudaMemcpyAsync");
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

// Results of the forward: sums, attention (when asked for) and, for a backward of the same block, the edge buffer. Without one
// to come, narrow rows are summed in one kernel that leaves no weights.
std::tuple<Tensor, Tensor, Tensor> gat_forward(const Tensor& coo_row, const Tensor& coo_col, const Tensor& ft_in, const Tensor& el_in,
                                               const Tensor& er_in, int64_t num_dst, double slope, bool want_attention,
                                               const Tensor& words, bool want_edges) {
  const Tensor row = ids(coo_row, "coo_row"), col = ids(coo_col, "coo_col");
  const Tensor ft = cuda(ft_in, "ft"), el = cuda(el_in, "el"), er = cuda(er_in, "er");
  const GatShape g = gat_shape("gat_edge_softmax_sum", row, ft, el, er, num_dst);
  Tensor out = at::empty({num_dst, g.heads, g.head_dim}, ft.options()), attn;
  if (want_attention) attn = at::empty({g.edges, g.heads, 1}, ft.options());
  const int64_t size = ft.element_size(), row_bytes = g.heads * g.head_dim * size;
  if (!want_edges && row_bytes <= APT_GAT_NARROW_BYTES && g.head_dim * size % 16 == 0 && (uintptr_t)data(ft) % 16 == 0) {
    const size_t bytes = apt_spmm_workspace_bytes(num_dst, 0);
    const Tensor ws = scratch(ft, bytes);
    check(apt_gat_edge_softmax_sum(g.code, ptr(row), ptr(col), g.edges, data(ft), data(el), data(er), (int)g.heads, g.head_dim,
                                   (float)slope, num_dst, mut(out), want_attention ? mut(attn) : nullptr, ws.mutable_data_ptr(),
                                   bytes, status_word(words), stream()));
    return {out, attn, Tensor()};
  }
  const size_t bytes = apt_gat_edges_bytes(num_dst, g.edges, (int)g.heads);
  const Tensor edges = scratch(ft, bytes);
  const size_t wide_bytes = apt_gat_widened_bytes(g.code, g.edges, g.num_src, 0, (int)g.heads, g.head_dim);
  const Tensor wide = room_for(ft, wide_bytes);
  check(apt_gat_forward_widened(g.code, ptr(row), ptr(col), g.edges, data(ft), data(el), data(er), (int)g.heads, g.head_dim, (float)slope,
                                g.num_src, num_dst, mut(out), want_attention ? mut(attn) : nullptr, edges.mutable_data_ptr(), bytes,
                                wide.defined() ? wide.mutable_data_ptr() : nullptr, wide_bytes, status_word(words), stream()));
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
  const size_t wide_bytes = g.num_dst ? apt_gat_widened_bytes(g.code, g.edges, g.num_src, g.num_dst, (int)g.heads, g.head_dim) : 0;
  const Tensor wide = room_for(ft, wide_bytes);
  check(apt_gat_backward_widened(g.code, ptr(row), ptr(col), g.edges, data(ft), data(el), data(er), data(grad), (int)g.heads, g.head_dim,
                                 (float)slope, g.num_src, g.num_dst, mut(grad_ft), mut(grad_el), mut(grad_er), edges.mutable_data_ptr(),
                                 edges_bytes, edges_of_forward ? 1 : 0, ws.mutable_data_ptr(), bytes,
                                 wide.defined() ? wide.mutable_data_ptr() : nullptr, wide_bytes, status_word(words), stream()));
  return {grad_ft, grad_el, grad_er};
}

// The forward's ranges and weights are saved with its inputs: the backward of a training step starts from them, and they
// go when the inputs go.
struct GatFunction : public torch::autograd::Function<GatFunction> {
  static Tensor forward(torch::autograd::AutogradContext* ctx, const Tensor& row, const Tensor& col, const Tensor& ft,
                        const Tensor& el, const Tensor& er, int64_t num_dst, double slope, const Tensor& words, bool backward) {
    auto [out, attn, edges] = gat_forward(row, col, ft, el, er, num_dst, slope, false, words, backward);
    ctx->save_for_backward({row, col, ft, el, er, edges});
    ctx->saved_data["slope"] = slope;
    ctx->saved_data["words"] = words;
    return out;
  }
  static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx, torch::autograd::variable_list grads) {
    const auto v = ctx->get_saved_variables();
    auto [g_ft, g_el, g_er] = gat_backward(v[0], v[1], v[2], v[3], v[4], grads[0], ctx->saved_data["slope"].toDouble(),
                                           ctx->saved_data["words"].toTensor(), v[5].defined() ? OptTensor(v[5]) : std::nullopt);
    return {Tensor(), Tensor(), g_ft, g_el, g_er, Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

// ------------------------------------------------------------------------------------------------ samplers
// Page-locked words, also while some stream is being captured.
Tensor pinned_words(int64_t count) {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  cuda_ok(cudaThreadExchangeStreamCaptureMode(&mode), "cudaThreadExchangeStreamCaptureMode");
  Tensor words;
  try {
    words = at::zeros({count}, at::TensorOptions().dtype(at::kLong).pinned_memory(true));
  } catch (...) {
    cudaThreadExchangeStreamCaptureMode(&mode);
    throw;
  }
  cudaThreadExchangeStreamCaptureMode(&mode);
  return words;
}

// Copies a word block to the host (one kernel, polled for), the last word, the status flags, from the end of `status`, and
// returns the flags.
int64_t read_words(const Tensor& words, const Tensor& status, const Tensor& host, int64_t sequence) {
  const int count = (int)words.numel();
  void* const s = stream();
  int64_t* const h = host.mutable_data_ptr<int64_t>();
  py::gil_scoped_release nogil;
  check(apt_publish_tagged(words.const_data_ptr<int64_t>(), count, status.const_data_ptr<int64_t>() + status.numel() - 1, nullptr, sequence,
                           h, s));
  check(apt_wait_tagged(h, count, sequence, s));
  return (h[count - 1] & 0xffffffff) | apt_pending_flags();
}

// One captured mini-batch: launches its graph, waits for its counts, orders other streams behind its last kernel.
class Plan {
 public:
  // replay_in: device words [call-id base, sequence]; host_words: page-locked, count words (apt_publish_tagged); own_stream:
  // 0 for the caller's current stream.
  Plan(uintptr_t exec, Tensor seeds_buf, Tensor replay_in, Tensor host_words, uintptr_t own_stream)
      : exec_((cudaGraphExec_t)exec), seeds_buf_(std::move(seeds_buf)), replay_in_(std::move(replay_in)),
        host_words_(std::move(host_words)), own_((cudaStream_t)own_stream) {
    cuda_ok(cudaEventCreateWithFlags(&done_, cudaEventDisableTiming), "cudaEventCreate");
    cuda_ok(cudaEventCreateWithFlags(&ready_, cudaEventDisableTiming), "cudaEventCreate");
  }
  ~Plan() {
    cudaEventDestroy(done_);
    cudaEventDestroy(ready_);
  }
  Plan(const Plan&) = delete;

  void launch(const Tensor& seeds, int64_t call_base) {
    if (seeds.scalar_type() != at::kLong || !seeds.is_contiguous() || seeds.numel() != seeds_buf_.numel())
      fail("sampler plan: seeds must be contiguous int64 of the plan's length");
    const cudaStream_t cur = (cudaStream_t)stream();
    const cudaStream_t s = own_ ? own_ : cur;
    const int64_t* from = seeds.const_data_ptr<int64_t>();
    int64_t* const to = seeds_buf_.mutable_data_ptr<int64_t>();
    int64_t count = from != to ? seeds.numel() : 0;
    py::gil_scoped_release nogil;
    // a launch nobody waited for (its iterator was given up): its seeds, which go below, may still be read
    if (!waited_) cuda_ok(cudaEventSynchronize(done_), "cudaEventSynchronize");
    if (own_) {
      // behind everything the caller's stream holds so far: the seeds' producer, the consumer of the last results
      cuda_ok(cudaEventRecord(ready_, cur), "cudaEventRecord");
      cuda_ok(cudaStreamWaitEvent(own_, ready_, 0), "cudaStreamWaitEvent");
    } else if (launched_ && stream_ != cur) {
      cuda_ok(cudaStreamWaitEvent(cur, done_, 0), "cudaStreamWaitEvent");
    }
    if (count && !(seeds.is_cuda() && seeds.device() == seeds_buf_.device())) {
      cuda_ok(cudaMemcpyAsync(to, from, count * 8, cudaMemcpyDefault, s), "cudaMemcpyAsync");
      count = 0;
    }
    check(apt_stage_replay(from, count, to, call_base, ++sequence_, replay_in_.mutable_data_ptr<int64_t>(), s));
    cuda_ok(cudaGraphLaunch(exec_, s), "cudaGraphLaunch");
    cuda_ok(cudaEventRecord(done_, s), "cudaEventRecord");
    stream_ = s;
    launched_ = true;
    waited_ = false;
    seeds_ = seeds;       // the copy reads it when the stream gets there
  }
  // Until the counts of the last launch are in host_words; returns the status flags.
  int64_t wait() {
    const int count = (int)host_words_.numel();
    int64_t* const h = host_words_.mutable_data_ptr<int64_t>();
    py::gil_scoped_release nogil;
    if (!waited_) check(apt_wait_tagged(h, count, sequence_, stream_));      // (which takes the tags off)
    waited_ = true;
    return (h[count - 1] & 0xffffffff) | apt_pending_flags();
  }
  void finish() {
    py::gil_scoped_release nogil;
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;      // a plan may go while some stream is being captured
    cudaThreadExchangeStreamCaptureMode(&mode);
    if (launched_) cudaEventSynchronize(done_);
    cudaThreadExchangeStreamCaptureMode(&mode);
  }
  // The current stream runs on behind everything the last launch enqueued (the gathered rows among it).
  void order_current_stream() {
    const cudaStream_t cur = (cudaStream_t)stream();
    if (launched_ && stream_ != cur) cuda_ok(cudaStreamWaitEvent(cur, done_, 0), "cudaStreamWaitEvent");
  }

 private:
  cudaGraphExec_t exec_;
  Tensor seeds_buf_, replay_in_, host_words_, seeds_;
  cudaStream_t own_, stream_ = nullptr;      // the default stream is a null handle too: launched_ says whether there is one
  cudaEvent_t done_, ready_;
  int64_t sequence_ = 0;
  bool launched_ = false, waited_ = true;
};

// The first n rows. Below autograd: a sampler's buffers have no history to carry on, and the view costs half as much.
Tensor front(const Tensor& t, int64_t n) {
  at::AutoDispatchBelowADInplaceOrView below;
  return t.narrow(0, 0, n);
}

Tensor offsets_cpu(const int64_t* v, int64_t n, bool sum) {
  Tensor t = at::empty({n}, at::TensorOptions().dtype(at::kLong));
  int64_t* const o = t.mutable_data_ptr<int64_t>();
  int64_t run = 0;
  for (int64_t k = 0; k < n; ++k) o[k] = sum ? (run += v[k]) : v[k];
  return t;
}

// A view of all of `t` that is cut to its real length once that is known: the views, their Python objects and the blocks
// around them (10 to 15 us a mini-batch) are made while the GPU is still sampling.
Tensor whole(const Tensor& t) { return front(t, t.size(0)); }
void cut(const Tensor& t, int64_t n) {
  if (n < 0 || n > t.size(0)) fail("sampler: a count of " + std::to_string(n) + " exceeds a buffer of " + std::to_string(t.size(0)));
  c10::SmallVector<int64_t, 4> sizes(t.sizes().begin(), t.sizes().end());
  sizes[0] = n;
  t.unsafeGetTensorImpl()->set_sizes_contiguous(sizes);
}

// The hops of a mini-batch, innermost first: (relabelled rows, unique ids, columns, fanout, count slot) each. `blocks`
// lists them outermost first.
class Hops {
 public:
  Hops(const py::list& layers, const py::object& block) {
    for (const auto& item : layers) {
      const py::tuple l = item.cast<py::tuple>();
      Hop h{whole(l[0].cast<Tensor>()), whole(l[1].cast<Tensor>()), whole(l[2].cast<Tensor>()), py::none(),
            l[3].cast<int64_t>(), l[4].cast<int64_t>()};
      h.block = block(h.rows, h.cols, 0, 0, h.ids, h.fanout);
      blocks.insert(0, h.block);
      hops_.push_back(std::move(h));
    }
  }
  // Cuts everything to the counts `w`; returns the number of nodes of the last frontier.
  int64_t fill(const int64_t* w, int64_t num_dst) {
    for (Hop& h : hops_) {
      const int64_t num_src = w[h.slot];
      cut(h.rows, num_dst * h.fanout);
      cut(h.cols, num_dst * h.fanout);
      cut(h.ids, num_src);
      h.block.attr("num_src") = num_src;
      h.block.attr("num_dst") = num_dst;
      num_dst = num_src;
    }
    return num_dst;
  }
  // Tensors much longer than their views (hops that meet the same nodes again and again) are replaced by copies of the views:
  // a caller that keeps its mini-batches keeps what they consist of, within a factor of two.
  void compact() {
    std::vector<const int64_t*> src;
    std::vector<int64_t*> dst;
    std::vector<int64_t> counts;
    for (Hop& h : hops_)
      for (const auto& [name, t] : {std::pair<const char*, Tensor*>{"coo_row", &h.rows}, {"coo_col", &h.cols}, {"src_ids", &h.ids}}) {
        if ((int64_t)t->storage().nbytes() <= 2 * (int64_t)t->nbytes() + kSlackBytes) continue;
        Tensor own = at::empty(t->sizes(), t->options());
        src.push_back(t->const_data_ptr<int64_t>());
        dst.push_back(own.mutable_data_ptr<int64_t>());
        counts.push_back(own.numel());
        left_.push_back(std::move(*t));      // until the copy is enqueued
        *t = std::move(own);
        h.block.attr(name) = *t;
      }
    check(apt_copy_words(src.data(), dst.data(), counts.data(), (int)src.size(), stream()));
    left_.clear();
  }
  py::list blocks;

 private:
  static constexpr int64_t kSlackBytes = 1 << 20;
  struct Hop {
    Tensor rows, ids, cols;
    py::object block;
    int64_t fanout, slot;
  };
  std::vector<Hop> hops_;
  std::vector<Tensor> left_;
};

// What sample() of a chained sampler returns, (input nodes, seeds, blocks, permutation, ids received per peer, bucket
// offsets[, inverse]) and the gathered rows, but for the lengths. `layers`: the inner hops, `outer` the outermost. The words
// hold [0..] hop counts, [16..] ids received per peer, [64..] bucket offsets.
//   node-partitioned        the outermost hop starts from w[frontier_slot] nodes and its sources are the input nodes
//   source-split, attention it starts from the inner hops' frontier; the input nodes are a buffer of their own
class Outline {
 public:
  Outline(const Tensor& seeds, const py::list& layers, const py::tuple& outer, const Tensor& perm, const OptTensor& inverse,
          const OptTensor& input, const OptTensor& rows, int64_t world_size, int64_t frontier_slot, int64_t unique_slot,
          int64_t input_slot, const py::object& block)
      : inner_(layers, block), outer_(only(outer), block), world_(world_size), frontier_slot_(frontier_slot),
        unique_slot_(unique_slot), input_slot_(input_slot), seeds_(seeds.numel()) {
    const auto longs = at::TensorOptions().dtype(at::kLong);
    perm_ = whole(perm);
    input_ = whole(input ? *input : outer[1].cast<Tensor>());
    recv_ = at::empty({world_size}, longs);
    sent_ = at::empty({world_size}, longs);
    inner_.blocks.insert(0, outer_.blocks[0]);
    if (inverse) {
      inverse_ = whole(*inverse);
      got_ = py::make_tuple(input_, seeds, inner_.blocks, perm_, recv_, sent_, inverse_);
    } else {
      got_ = py::make_tuple(input_, seeds, inner_.blocks, perm_, recv_, sent_);
    }
    if (rows) {
      rows_ = whole(*rows);
      row_view_ = py::cast(rows_);
    }
  }
  py::tuple finish(const Tensor& host) {
    const int64_t* const w = host.const_data_ptr<int64_t>();
    int64_t* const recv = recv_.mutable_data_ptr<int64_t>();
    int64_t received = 0;
    for (int64_t k = 0; k < world_; ++k) recv[k] = received += w[16 + k];
    std::copy_n(w + 64, world_, sent_.mutable_data_ptr<int64_t>());
    const int64_t frontier = inner_.fill(w, seeds_);
    const bool np = inverse_.defined();
    if (np ? received > inverse_.numel() : w[input_slot_] > input_.numel())
      fail(std::string(np ? "chained NP sampler" : "chained SNP-GAT sampler") + ": more ids received than the buffer sized from "
           "this rank's own batch holds; use chained=False for batches that differ this much between the ranks");
    const int64_t sources = outer_.fill(w, np ? w[frontier_slot_] : frontier), num_in = np ? sources : w[input_slot_];
    cut(input_, num_in);
    cut(perm_, np ? frontier : w[unique_slot_]);
    if (np) cut(inverse_, received);
    if (rows_.defined()) cut(rows_, num_in);
    return py::make_tuple(got_, row_view_);
  }

 private:
  static py::list only(const py::tuple& layer) {
    py::list l;
    l.append(layer);
    return l;
  }
  Hops inner_, outer_;
  int64_t world_, frontier_slot_, unique_slot_, input_slot_, seeds_;
  Tensor perm_, input_, inverse_, rows_, recv_, sent_;
  py::object row_view_ = py::none();
  py::tuple got_;
};

// Rows of a tensor of its own that a stream has been asked for: orders other streams behind that, and tells the allocator
// of them.
class PendingRows {
 public:
  explicit PendingRows(Tensor rows) : rows_(std::move(rows)), stream_((cudaStream_t)stream()) {
    cuda_ok(cudaEventCreateWithFlags(&done_, cudaEventDisableTiming), "cudaEventCreate");
    const cudaError_t e = cudaEventRecord(done_, stream_);
    if (e != cudaSuccess) {
      cudaEventDestroy(done_);
      cuda_ok(e, "cudaEventRecord");
    }
  }
  ~PendingRows() { cudaEventDestroy(done_); }
  PendingRows(const PendingRows&) = delete;
  void order_current_stream() {
    const auto cur = c10::cuda::getCurrentCUDAStream();
    if (cur.stream() == stream_) return;
    cuda_ok(cudaStreamWaitEvent(cur.stream(), done_, 0), "cudaStreamWaitEvent");
    if (rows_.numel()) rows_.record_stream(cur.unwrap());
  }

 private:
  Tensor rows_;
  cudaStream_t stream_;
  cudaEvent_t done_;
};

// Data-parallel: every hop sampled and relabelled on this GPU behind one read of the counts. All results are tensors of their
// own. The rows of the input nodes are gathered after that read, into as many rows as there are: gathered behind the
// counts without it, they took a buffer for the case of no node met twice (554 MB instead of 74 for 1024 seeds x (15, 10, 5)
// at 512 bytes a row) and a length from a device word that operators on other streams write too.
py::tuple dp_sample(const Tensor& seeds, const std::vector<int64_t>& fanouts, const OptTensor& adj_pos_map, int64_t num_nodes,
                    const OptTensor& dev_indptr, const OptTensor& dev_indices, const Tensor& uva_indptr, const Tensor& uva_indices,
                    int64_t key, int64_t call, const Tensor& relabel_ws, const Tensor& words, const Tensor& host, int64_t sequence,
                    const py::object& features, int64_t row_limit_bytes, const py::object& block) {
  const auto opt = [](const OptTensor& t) { return t ? ptr(*t) : nullptr; };
  Tensor pos_map, dev_feats, uva_feats;
  int64_t feat_nodes = 0, column = 0;
  const bool look_up = !features.is_none();
  if (look_up) {
    const py::tuple f = features.cast<py::tuple>();
    pos_map = f[0].cast<Tensor>(), dev_feats = f[1].cast<Tensor>(), uva_feats = f[2].cast<Tensor>();
    feat_nodes = f[3].cast<int64_t>(), column = f[4].cast<int64_t>();
  }
  int64_t* const word = words.mutable_data_ptr<int64_t>();
  int64_t* const h = host.mutable_data_ptr<int64_t>();
  const int count = (int)words.numel();
  void* const s = stream();
  py::list layers;
  Tensor cur = seeds;
  const auto ids_like = [&](int64_t n) { return at::empty({n}, seeds.options()); };
  for (size_t k = 0; k < fanouts.size(); ++k) {
    const int64_t n = cur.numel(), f = fanouts[k];
    Tensor rel = ids_like(n * f), uniq = ids_like(n * (1 + f)), col = ids_like(n * f);
    const bool last = look_up && k + 1 == fanouts.size();
    check(apt_sample_relabel_block(ptr(cur), n, k ? word + k - 1 : nullptr, (int)f, opt(adj_pos_map), num_nodes, opt(dev_indptr),
                                   opt(dev_indices), ptr(uva_indptr), ptr(uva_indices), (uint64_t)key,
                                   (uint32_t)(call + (int64_t)k), nullptr, relabel_ws.mutable_data_ptr(), relabel_ws.numel(),
                                   nullptr, uniq.mutable_data_ptr<int64_t>(), rel.mutable_data_ptr<int64_t>(),
                                   col.mutable_data_ptr<int64_t>(), word + k, last ? ptr(pos_map) : nullptr, feat_nodes,
                                   last ? dev_feats.size(0) : 0, last ? uva_feats.size(0) : 0, status_word(words), s));
    cur = uniq;
    layers.append(py::make_tuple(rel, uniq, col, f, (int64_t)k));
  }
  check(apt_publish_tagged(word, count, word + count - 1, nullptr, sequence, h, s));
  Hops hops(layers, block);
  {
    py::gil_scoped_release nogil;
    check(apt_wait_tagged(h, count, sequence, s));
  }
  const int64_t num_in = h[fanouts.size() - 1], flags = (h[count - 1] & 0xffffffff) | apt_pending_flags();
  py::object rows = py::none(), pending = py::none();
  if (look_up && num_in * dev_feats.size(1) * (int64_t)dev_feats.element_size() <= row_limit_bytes) {
    if (num_in > cur.size(0)) fail("sampler: more input nodes than were drawn");
    const Tensor got = gather(front(cur, num_in), pos_map, dev_feats, uva_feats, feat_nodes, column, words);
    rows = py::cast(got);
    pending = py::cast(std::make_unique<PendingRows>(got));
  }
  hops.fill(h, seeds.numel());
  hops.compact();
  return py::make_tuple(hops.blocks, rows, pending, flags);
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
      py::object err = cls(e.status, py::bytes(e.what()).attr("decode")("utf-8", "replace"));
      PyErr_SetObject(cls.ptr(), err.ptr());
    }
  });
  m.def("spmm", &spmm);
  m.def("sddmm", &sddmm);
  py::class_<Plan>(m, "Plan")
      .def(py::init<uintptr_t, Tensor, Tensor, Tensor, uintptr_t>())
      .def("launch", &Plan::launch)
      .def("wait", &Plan::wait)
      .def("finish", &Plan::finish)
      .def("order_current_stream", &Plan::order_current_stream);
  m.def("pinned_words", &pinned_words);
  m.def("read_words", &read_words);
  py::class_<Hops>(m, "Hops")
      .def(py::init<const py::list&, const py::object&>())
      .def_readonly("blocks", &Hops::blocks)
      .def("fill", [](Hops& hops, const Tensor& host, int64_t num_dst) { return hops.fill(host.const_data_ptr<int64_t>(), num_dst); });
  py::class_<Outline>(m, "Outline")
      .def(py::init<const Tensor&, const py::list&, const py::tuple&, const Tensor&, const OptTensor&, const OptTensor&,
                    const OptTensor&, int64_t, int64_t, int64_t, int64_t, const py::object&>())
      .def("finish", &Outline::finish);
  m.def("wholes", [](const std::vector<Tensor>& tensors) {
    std::vector<Tensor> out;
    for (const Tensor& t : tensors) out.push_back(whole(t));
    return out;
  });
  m.def("cut", [](const std::vector<Tensor>& tensors, const std::vector<int64_t>& sizes) {
    for (size_t k = 0; k < tensors.size(); ++k) cut(tensors[k], sizes.at(k));
  });
  m.def("pick", [](const Tensor& host, const std::vector<int64_t>& at) {
    std::vector<int64_t> out;
    for (const int64_t k : at) out.push_back(host.const_data_ptr<int64_t>()[k]);
    return out;
  });
  m.def("sizes", [](const std::vector<int64_t>& v) { return offsets_cpu(v.data(), (int64_t)v.size(), false); });
  m.def("feat_shuffle_local", &feat_shuffle_local);
  m.def("sp_feat_shuffle_local", &sp_feat_shuffle_local);
  py::class_<PendingRows>(m, "PendingRows").def("order_current_stream", &PendingRows::order_current_stream);
  m.def("dp_sample", &dp_sample);
  m.def("gather", &gather);
  m.def("rows_gather", &rows_gather);
  m.def("rows_scatter", &rows_scatter);
  m.def("gat_forward", [](const Tensor& row, const Tensor& col, const Tensor& ft, const Tensor& el, const Tensor& er,
                          int64_t num_dst, double slope, bool want_attention, const Tensor& words) {
    auto [out, attn, edges] = gat_forward(row, col, ft, el, er, num_dst, slope, want_attention, words, false);
    return std::make_tuple(out, attn);
  });
  m.def("gat_backward", [](const Tensor& row, const Tensor& col, const Tensor& ft, const Tensor& el, const Tensor& er,
                           const Tensor& grad, double slope, const Tensor& words) {
    return gat_backward(row, col, ft, el, er, grad, slope, words, std::nullopt);
  });
  m.def("gat_apply", [](const Tensor& row, const Tensor& col, const Tensor& ft, const Tensor& el, const Tensor& er,
                        int64_t num_dst, double slope, const Tensor& words) {
    const bool backward = at::GradMode::is_enabled() && (ft.requires_grad() || el.requires_grad() || er.requires_grad());
    return GatFunction::apply(row, col, ft, el, er, num_dst, slope, words, backward);
  });
}
