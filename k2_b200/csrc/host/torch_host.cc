// The host side of a CTC training step as native code: transcripts to graphs, the layout of a
// DenseFsaVec, and the band-graph loss as one node of torch's autograd graph.
//
// A step of one short utterance keeps the GPU busy for 80 us; the same step through numpy,
// ctypes and Python autograd functions took the host 500.  Nothing here computes on the host:
// the functions size and allocate outputs, call the C-ABI (include/k2b200.h) and hand tensors
// back.  Python keeps k2's names and contracts (k2/python/k2/ctc_loss.py:28-208,
// k2/python/k2/fsa_algo.py:1160-1249, k2/python/k2/dense_fsa_vec.py:43-145).
#include <c10/cuda/CUDAException.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/python_cpp_function.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <pybind11/numpy.h>
#include <torch/extension.h>

#include <algorithm>
#include <map>
#include <memory>
#include <mutex>
#include <vector>

#include "../../../include/k2b200.h"
#include "python_ints.h"

namespace py = pybind11;

namespace {

using IntArray = py::array_t<int32_t, py::array::c_style>;

// The reference raises a C++ exception that Python sees as RuntimeError
// (k2/csrc/log.h:196-203); a non-zero status is surfaced the same way.
void Check(int32_t status) {
  if (status != 0) throw std::runtime_error(k2b200_last_error());
}

[[noreturn]] void AssertionFailed(const char *what) {
  PyErr_SetString(PyExc_AssertionError, what);
  throw py::error_already_set();
}

at::TensorOptions On(at::ScalarType type, at::Device device) {
  return at::TensorOptions().dtype(type).device(device);
}

// ---------------------------------------------------------------------------
// Workspaces.  Those of a loss are a gigabyte or more and live from a forward to its backward.
// Handed back to torch's caching allocator they get split for smaller tensors, after which the
// next step needs a fresh cudaMalloc, which waits for the whole device.  So the last few are
// kept here, per device and stream: what comes back may still be read by kernels queued on
// that stream, and the next user queues behind them.  A call that is captured takes memory of
// its graph instead, which stays the graph's for every replay.
// ---------------------------------------------------------------------------
constexpr int64_t kPoolMinBytes = 32 << 20;  // smaller ones go through torch's allocator
constexpr size_t kPoolKeep = 3;              // idle workspaces per (device, stream)

struct Pool {
  std::mutex mutex;
  std::map<std::pair<int, cudaStream_t>, std::vector<at::Tensor>> idle;
};
Pool &ThePool() {
  static Pool *pool = new Pool;  // never destroyed: the CUDA context may be gone by then
  return *pool;
}

struct Workspace {
  at::Tensor tensor;
  std::pair<int, cudaStream_t> key{-1, nullptr};
  Workspace(int64_t bytes, at::Device device, cudaStream_t stream) {
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    if (bytes >= kPoolMinBytes) C10_CUDA_CHECK(cudaStreamIsCapturing(stream, &capture));
    if (bytes < kPoolMinBytes || capture != cudaStreamCaptureStatusNone) {
      tensor = at::empty({std::max<int64_t>(bytes, 1)}, On(at::kByte, device));
      return;
    }
    key = {device.index(), stream};
    {
      std::lock_guard<std::mutex> lock(ThePool().mutex);
      auto &idle = ThePool().idle[key];
      size_t best = idle.size();
      for (size_t k = 0; k < idle.size(); ++k)
        if (idle[k].numel() >= bytes && idle[k].numel() <= 2 * bytes &&
            (best == idle.size() || idle[k].numel() < idle[best].numel()))
          best = k;
      if (best < idle.size()) {
        tensor = idle[best];
        idle.erase(idle.begin() + best);
        return;
      }
    }
    // some headroom, so that a slightly larger batch still fits
    tensor = at::empty({bytes + bytes / 8}, On(at::kByte, device));
  }
  ~Workspace() {
    if (key.first < 0) return;
    at::Tensor drop;  // freed outside the lock
    std::lock_guard<std::mutex> lock(ThePool().mutex);
    auto &idle = ThePool().idle[key];
    idle.push_back(std::move(tensor));
    if (idle.size() > kPoolKeep) {
      auto least = std::min_element(
          idle.begin(), idle.end(),
          [](const at::Tensor &a, const at::Tensor &b) { return a.numel() < b.numel(); });
      drop = *least;
      idle.erase(least);
    }
  }
  Workspace(const Workspace &) = delete;
};

void ReleaseWorkspaces() {
  std::map<std::pair<int, cudaStream_t>, std::vector<at::Tensor>> drop;
  std::lock_guard<std::mutex> lock(ThePool().mutex);
  drop.swap(ThePool().idle);
}

// ---------------------------------------------------------------------------
// Band graphs: what the loss needs of an FsaVec, kept with it.
// ---------------------------------------------------------------------------
struct BandGraph {
  at::Tensor row_splits2, states, arcs;  // device
  std::vector<int32_t> h_row_splits1, h_arc_splits;
  int32_t num_states = 0;
};

std::shared_ptr<BandGraph> MakeBandGraph(at::Tensor row_splits2, at::Tensor states, at::Tensor arcs,
                                         IntArray h_row_splits1, IntArray h_arc_splits) {
  auto g = std::make_shared<BandGraph>();
  g->row_splits2 = std::move(row_splits2);
  g->states = std::move(states);
  g->arcs = std::move(arcs);
  g->h_row_splits1.assign(h_row_splits1.data(), h_row_splits1.data() + h_row_splits1.size());
  g->h_arc_splits.assign(h_arc_splits.data(), h_arc_splits.data() + h_arc_splits.size());
  g->num_states = g->h_row_splits1.back();
  return g;
}

// CTC graphs of a batch of transcripts with their band tables: (values, row_splits1,
// row_splits2, aux_labels, scores, labels, host row_splits1, host arc splits, BandGraph), or
// None when the transcripts are not sequences of Python integers.
py::object CtcGraph(py::handle symbols, bool modified, int device_index) {
  // (what has no length is refused, iterators among it)
  if (PyObject_Size(symbols.ptr()) < 0) throw py::error_already_set();
  py::object outer = py::reinterpret_steal<py::object>(
      PySequence_Fast(symbols.ptr(), "symbols must be a list of lists"));
  if (!outer) throw py::error_already_set();
  const Py_ssize_t n = PySequence_Fast_GET_SIZE(outer.ptr());
  if (n == 0) return py::none();
  std::vector<py::object> rows(n);
  int64_t tot = 0;
  for (Py_ssize_t i = 0; i < n; ++i) {
    PyObject *row = PySequence_Fast_GET_ITEM(outer.ptr(), i);
    if (PyObject_Size(row) < 0) throw py::error_already_set();
    rows[i] = py::reinterpret_steal<py::object>(
        PySequence_Fast(row, "a transcript must be a list"));
    if (!rows[i]) throw py::error_already_set();
    tot += PySequence_Fast_GET_SIZE(rows[i].ptr());
  }
  if (tot > (int64_t)1 << 28) return py::none();
  // first symbol of every graph, first arc of every graph, symbols
  std::vector<int32_t> meta(2 * (n + 1) + tot);
  IntArray h_row_splits1(n + 1), h_arc_splits(n + 1);
  int32_t *first = meta.data(), *arc0 = first + n + 1, *sym = arc0 + n + 1;
  int32_t *rs1 = h_row_splits1.mutable_data();
  int64_t at = 0, arcs = 0;
  bool blank_free = true;
  for (Py_ssize_t i = 0; i < n; ++i) {
    const Py_ssize_t len = PySequence_Fast_GET_SIZE(rows[i].ptr());
    int32_t *mine = sym + at;
    if (!Int32sOf(rows[i].ptr(), len, mine)) return py::none();
    first[i] = (int32_t)at;
    arc0[i] = (int32_t)arcs;
    rs1[i] = (int32_t)(2 * at + 2 * i);
    // symbol states have a third arc unless the next symbol is the same
    int32_t same = 0;
    for (Py_ssize_t k = 0; k < len; ++k) {
      blank_free &= mine[k] != -1;
      same += k + 1 < len && mine[k] == mine[k + 1];
    }
    arcs += 5 * (int64_t)len + 2 - (modified ? 0 : same);
    at += len;
  }
  if (!blank_free) AssertionFailed("symbols must not contain -1");
  first[n] = (int32_t)at;
  arc0[n] = (int32_t)arcs;
  const int32_t states = (int32_t)(2 * at + 2 * n), num_arcs = (int32_t)arcs;
  rs1[n] = states;
  std::copy(arc0, arc0 + n + 1, h_arc_splits.mutable_data());

  const at::Device device(at::kCUDA, (c10::DeviceIndex)device_index);
  c10::cuda::CUDAGuard guard(device);
  at::Tensor values = at::empty({num_arcs, 4}, On(at::kInt, device));
  at::Tensor ints = at::empty({n + 1 + states + 1 + num_arcs + (int64_t)meta.size()},
                              On(at::kInt, device));
  size_t state_bytes = 0, arc_bytes = 0;
  Check(k2b200_band_tables_bytes(states, &state_bytes, &arc_bytes));
  at::Tensor tables = at::empty({(int64_t)(state_bytes + arc_bytes)}, On(at::kByte, device));
  int32_t *d = ints.data_ptr<int32_t>();
  int32_t *d_rs1 = d, *d_rs2 = d_rs1 + n + 1, *d_aux = d_rs2 + states + 1, *d_meta = d_aux + num_arcs;
  char *d_tables = static_cast<char *>(tables.data_ptr());
  Check(k2b200_ctc_graph_host(meta.data(), (int32_t)n, (int32_t)tot, modified, d_rs1, d_rs2,
                              values.data_ptr(), d_aux, d_tables, d_tables + state_bytes, d_meta,
                              c10::cuda::getCurrentCUDAStream(device.index()).stream()));
  auto g = std::make_shared<BandGraph>();
  g->row_splits2 = ints.narrow(0, n + 1, states + 1);
  g->states = tables;
  g->arcs = tables.narrow(0, (int64_t)state_bytes, (int64_t)arc_bytes);
  g->h_row_splits1.assign(rs1, rs1 + n + 1);
  g->h_arc_splits.assign(arc0, arc0 + n + 1);
  g->num_states = states;
  return py::make_tuple(values, ints.narrow(0, 0, n + 1), g->row_splits2,
                        ints.narrow(0, n + 1 + states + 1, num_arcs),
                        values.select(1, 3).view(at::kFloat), values.select(1, 2), h_row_splits1,
                        h_arc_splits, g);
}

// Layout of a DenseFsaVec over N sequences of T frames: (row_splits, first row of every
// segment in the [N * T, C] log-probs, segments after truncation, do segments overlap).
py::tuple DenseLayout(const at::Tensor &segments, int64_t N, int64_t T, int64_t allow_truncate) {
  if (segments.dim() != 2 || (segments.size(0) > 0 && segments.size(1) != 3))
    AssertionFailed("supervision_segments must be [num_segs, 3]");
  const at::Tensor seg = segments.contiguous();
  const int64_t n = seg.size(0);
  const int32_t *s = seg.data_ptr<int32_t>();
  IntArray row_splits(n + 1), first(n);
  IntArray effective(std::vector<py::ssize_t>{(py::ssize_t)n, 3});
  int32_t *rs = row_splits.mutable_data(), *fr = first.mutable_data(), *eff = effective.mutable_data();
  rs[0] = 0;
  bool one_each = true;
  std::vector<char> seen(N, 0);
  for (int64_t k = 0; k < n; ++k) {
    const int32_t seq = s[3 * k], start = s[3 * k + 1], dur = s[3 * k + 2];
    if (seq < 0 || start < 0 || dur < 0 || seq >= N || start >= T)
      AssertionFailed("a supervision segment lies outside the log-probs");
    const int64_t end = (int64_t)start + dur;
    if (end > T + allow_truncate) AssertionFailed("a supervision segment ends after the last frame");
    const int32_t d = (int32_t)(std::min(end, T) - start);
    rs[k + 1] = rs[k] + d + 1;
    fr[k] = (int32_t)((int64_t)seq * T + start);
    eff[3 * k] = seq;
    eff[3 * k + 1] = start;
    eff[3 * k + 2] = d;
    one_each &= !seen[seq];
    seen[seq] = 1;
  }
  bool overlapping = false;
  if (!one_each) {  // only segments of one sequence can touch the same frame
    std::vector<std::pair<int64_t, int64_t>> spans(n);
    for (int64_t k = 0; k < n; ++k) {
      const int64_t b = (int64_t)eff[3 * k] * T + eff[3 * k + 1];
      spans[k] = {b, b + eff[3 * k + 2]};
    }
    std::sort(spans.begin(), spans.end());
    for (int64_t k = 0; k + 1 < n; ++k) overlapping |= spans[k].second > spans[k + 1].first;
  }
  return py::make_tuple(row_splits, first, effective, overlapping);
}

// ---------------------------------------------------------------------------
// The band-graph loss.
// ---------------------------------------------------------------------------
enum Mode : int32_t { kTotals = 0, kNegSum = 1, kMean = 2 };

// k2b200_band_loss_args and everything its pointers refer to.
struct BandCall {
  k2b200_band_loss_args args{};
  std::shared_ptr<BandGraph> graph;
  std::vector<int32_t> first, frames;
  at::Tensor log_probs;  // what the kernels read (normalised when the user gave logits)
  std::shared_ptr<Workspace> workspace;
  size_t bytes = 0;
};

struct BandLossNode : public torch::autograd::Node {
  BandCall call;
  torch::autograd::SavedVariable saved_lens;  // complains if they were changed in the meantime
  std::vector<int64_t> input_sizes;
  int64_t num_arcs = 0;
  int32_t mode = kTotals, lens_type = 0;
  bool logits = false;

  torch::autograd::variable_list apply(torch::autograd::variable_list &&grads) override {
    torch::autograd::variable_list out(2);
    at::Tensor g = grads[0];
    if (!g.defined()) return out;
    TORCH_CHECK(call.workspace != nullptr,
                "the loss was already differentiated and its buffers freed (retain_graph=True "
                "keeps them)");
    const at::Device device = call.log_probs.device();
    c10::cuda::CUDAGuard guard(device);
    if (g.scalar_type() != at::kFloat && g.scalar_type() != at::kDouble) g = g.to(at::kDouble);
    k2b200_band_upstream up{};
    up.grad = g.data_ptr();
    up.is_double = g.scalar_type() == at::kDouble;
    // the gradient of a reduction arrives expanded: element stride may be 0
    up.stride = mode == kTotals && g.numel() > 0 ? (int32_t)g.stride(0) : 0;
    up.negate = mode != kTotals;
    up.lens_type = lens_type;
    const at::Tensor lens = lens_type ? saved_lens.unpack() : at::Tensor();
    up.lens = lens_type ? lens.data_ptr() : nullptr;
    if (task_should_compute_output(0)) out[0] = at::empty(input_sizes, On(at::kFloat, device));
    if (task_should_compute_output(1)) out[1] = at::zeros({num_arcs}, On(at::kFloat, device));
    Check(k2b200_band_loss_backward_dense(
        &call.args, call.workspace->tensor.data_ptr(), call.bytes, &up,
        out[1].defined() ? out[1].data_ptr<float>() : nullptr,
        out[0].defined() ? out[0].data_ptr<float>() : nullptr, logits,
        c10::cuda::getCurrentCUDAStream(device.index()).stream()));
    return out;
  }
  void release_variables() override {
    call.workspace.reset();
    saved_lens.reset_data();
  }
};

// One class per mode, so that `grad_fn` of a result says in Python what it is.
struct BandTotScoresNode : public BandLossNode {};
struct BandNegSumNode : public BandLossNode {};
struct BandMeanNode : public BandLossNode {};

std::shared_ptr<BandLossNode> NewNode(int32_t mode) {
  BandLossNode *node = mode == kTotals   ? static_cast<BandLossNode *>(new BandTotScoresNode())
                       : mode == kNegSum ? static_cast<BandLossNode *>(new BandNegSumNode())
                                         : new BandMeanNode();
  return std::shared_ptr<BandLossNode>(node, torch::autograd::deleteNode);
}

template <typename T>
void NameNode(const char *name) {
  using namespace torch::autograd;  // the properties below are named without it
  static PyTypeObject type;
  static PyMethodDef methods[] = {
      {"register_hook", THPCppFunction_register_hook, METH_O, nullptr},
      {"register_prehook", THPCppFunction_register_prehook, METH_O, nullptr},
      {"name", THPCppFunction_name, METH_NOARGS, nullptr},
      {nullptr}};
  static PyGetSetDef properties[] = {THP_FUNCTION_DEFAULT_PROPERTIES, {nullptr}};
  _initFunctionPyTypeObject(type, name, properties, methods);
  registerCppFunction(typeid(T), &type);
}

int32_t LensType(const at::Tensor &t) {
  switch (t.scalar_type()) {
    case at::kInt: return 1;
    case at::kLong: return 2;
    case at::kFloat: return 3;
    case at::kDouble: return 4;
    default: return 0;
  }
}

// Total scores (mode 0) or the loss of them (1: -sum, 2: mean of -tot / target length) of band
// graphs against log-probs or logits, or None when the band kernels do not take these inputs.
// first: row of every sequence's first frame; row_splits: of the DenseFsaVec.
py::object BandLoss(const std::shared_ptr<BandGraph> &graph, const at::Tensor &scores_a,
                    const at::Tensor &input, bool logits, const IntArray &first,
                    const IntArray &row_splits, const py::object &a_to_b, double beam,
                    int64_t max_states, int64_t max_arcs, int32_t mode, bool use_double,
                    const c10::optional<at::Tensor> &lens, double delay_penalty,
                    const c10::optional<at::Tensor> &symbols) {
  if (!input.is_cuda() || input.scalar_type() != at::kFloat || input.dim() != 3 ||
      !input.is_contiguous() || graph->states.device() != input.device())
    return py::none();
  // forward-mode derivatives are refused, which the Python autograd functions do
  if (input._fw_grad(0).defined() || scores_a._fw_grad(0).defined()) return py::none();
  const int32_t n = (int32_t)graph->h_row_splits1.size() - 1, seqs = (int32_t)first.size();
  BandCall call;
  call.graph = graph;
  call.first.resize(n);
  call.frames.resize(n);
  const int32_t *rs = row_splits.data(), *fr = first.data();
  if (a_to_b.is_none()) {
    if (n != seqs) return py::none();
    for (int32_t i = 0; i < n; ++i) {
      call.first[i] = fr[i];
      call.frames[i] = rs[i + 1] - rs[i] - 1;
    }
  } else {
    const IntArray to_seq = a_to_b.cast<IntArray>();
    if (to_seq.size() != n) return py::none();
    for (int32_t i = 0; i < n; ++i) {
      const int32_t j = to_seq.data()[i];
      if (j < 0 || j >= seqs || (i > 0 && j < to_seq.data()[i - 1])) return py::none();
      call.first[i] = fr[j];
      call.frames[i] = rs[j + 1] - rs[j] - 1;
    }
  }
  int32_t lens_type = 0;
  if (mode == kMean) {
    if (!lens.has_value() || !lens->is_cuda() || lens->device() != input.device() ||
        lens->dim() != 1 || lens->numel() != n || !lens->is_contiguous() ||
        (lens_type = LensType(*lens)) == 0 ||
        // (no derivative with respect to the lengths here)
        torch::autograd::compute_requires_grad(*lens) || lens->_fw_grad(0).defined())
      return py::none();
  }
  // the gradient of the arc scores does not know of the penalty
  const bool delayed = delay_penalty > 0.0;
  if (delayed && (!symbols.has_value() || !symbols->is_cuda() ||
                  symbols->device() != input.device() || symbols->dim() != 1 ||
                  !symbols->is_contiguous() || symbols->numel() != graph->h_arc_splits.back() ||
                  (symbols->scalar_type() != at::kInt && symbols->scalar_type() != at::kBool) ||
                  torch::autograd::compute_requires_grad(scores_a)))
    return py::none();
  k2b200_band_loss_args &a = call.args;
  const int64_t classes = input.size(2);
  if (classes > (int64_t)1 << 24) return py::none();
  a.num_fsas = n;
  a.num_states = graph->num_states;
  a.a_row_splits2 = graph->row_splits2.data_ptr<int32_t>();
  a.h_a_row_splits1 = graph->h_row_splits1.data();
  a.h_a_arc_splits = graph->h_arc_splits.data();
  a.band_states = graph->states.data_ptr();
  a.band_arcs = graph->arcs.data_ptr();
  a.log_probs = input.data_ptr<float>();
  a.log_prob_rows = input.size(0) * input.size(1);
  a.num_classes = (int32_t)classes;
  a.h_first_row = call.first.data();
  a.h_frames = call.frames.data();
  a.output_beam = (float)beam;
  a.max_states = (int32_t)std::min<int64_t>(max_states, INT32_MAX);
  a.max_arcs = (int32_t)std::min<int64_t>(max_arcs, INT32_MAX);
  int32_t supported = 0, exclusive = 0;
  Check(k2b200_band_loss_plan(&a, &supported, &exclusive, &call.bytes));
  const bool graded = torch::autograd::compute_requires_grad(input, scores_a);
  if (!supported || (!exclusive && (logits || graded))) return py::none();

  const at::Device device = input.device();
  c10::cuda::CUDAGuard guard(device);
  const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(device.index()).stream();
  at::Tensor out;
  {
    at::AutoDispatchBelowADInplaceOrView below_autograd;
    call.log_probs = logits ? at::empty(input.sizes(), On(at::kFloat, device)) : input.detach();
    a.log_probs = call.log_probs.data_ptr<float>();
    call.workspace = std::make_shared<Workspace>((int64_t)call.bytes, device, stream);
    at::Tensor tot = at::empty({n}, On(at::kDouble, device));
    k2b200_band_reduce reduce{};
    reduce.mode = mode;
    reduce.lens_type = lens_type;
    reduce.lens = lens_type ? lens->data_ptr() : nullptr;
    reduce.logits = logits ? input.data_ptr<float>() : nullptr;
    if (delayed) {
      reduce.delay_penalty = (float)delay_penalty;
      if (symbols->scalar_type() == at::kBool)
        reduce.arc_repeat = reinterpret_cast<const uint8_t *>(symbols->data_ptr<bool>());
      else
        reduce.arc_aux = symbols->data_ptr<int32_t>();
    }
    if (mode != kTotals) {
      out = at::empty({}, On(at::kFloat, device));
      reduce.loss = out.data_ptr<float>();
    }
    {
      py::gil_scoped_release release;  // the call may wait for the counts of the beam reduction
      Check(k2b200_band_loss_forward_reduce(&a, call.workspace->tensor.data_ptr(), call.bytes,
                                            stream, tot.data_ptr<double>(), nullptr, &reduce));
    }
    if (mode == kTotals) out = use_double ? tot : tot.to(at::kFloat);
  }
  if (graded) {
    std::shared_ptr<BandLossNode> node = NewNode(mode);
    node->set_next_edges(torch::autograd::collect_next_edges(input, scores_a));
    node->input_sizes = input.sizes().vec();
    node->num_arcs = scores_a.size(0);
    node->mode = mode;
    node->lens_type = lens_type;
    if (lens_type) node->saved_lens = torch::autograd::SavedVariable(*lens, false);
    node->logits = logits;
    node->call = std::move(call);
    // the argument block points into the vectors, which have moved
    node->call.args.h_first_row = node->call.first.data();
    node->call.args.h_frames = node->call.frames.data();
    torch::autograd::set_history(out, node);
  }
  return py::cast(out);
}

}  // namespace

PYBIND11_MODULE(_host, m) {
  NameNode<BandTotScoresNode>("_BandTotScoresBackward");
  NameNode<BandNegSumNode>("_BandNegSumBackward");
  NameNode<BandMeanNode>("_BandMeanBackward");
  py::class_<Workspace, std::shared_ptr<Workspace>>(m, "Workspace")
      .def(py::init([](int64_t bytes, int device_index) {
        const at::Device device(at::kCUDA, (c10::DeviceIndex)device_index);
        return std::make_shared<Workspace>(
            bytes, device, c10::cuda::getCurrentCUDAStream(device.index()).stream());
      }))
      .def_readonly("tensor", &Workspace::tensor);
  py::class_<BandGraph, std::shared_ptr<BandGraph>>(m, "BandGraph")
      .def(py::init(&MakeBandGraph))
      .def_property_readonly("states_ptr",
                             [](const BandGraph &g) { return (uintptr_t)g.states.data_ptr(); })
      .def_property_readonly("arcs_ptr",
                             [](const BandGraph &g) { return (uintptr_t)g.arcs.data_ptr(); });
  m.def("ctc_graph", &CtcGraph);
  m.def("dense_layout", &DenseLayout);
  m.def("band_loss", &BandLoss);
  m.def("release_workspaces", &ReleaseWorkspaces);
}
