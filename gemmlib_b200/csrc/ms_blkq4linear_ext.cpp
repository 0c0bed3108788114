// PyTorch extension `ms_blkq4linear_ext`: the host-side mirror of the reference's
// python/ms_blkq4linear_ext/ms_blkq4linear.cpp (quant :13-72, forward :74-117,
// module definition :120-123).  Same function names, argument order and checks;
// tensors are reduced to device pointers and byte sizes and handed to the C ABI in
// include/ms_blkq4gemm.h.  Differences, all additive:
//   - work is enqueued on PyTorch's current CUDA stream (the reference passes the
//     legacy default stream), so the calls compose with CUDA graphs and side streams;
//   - with has_offsets == false `quant` returns an empty uint8 tensor for the zero
//     points (the reference returns an undefined tensor, which its own `forward`
//     cannot accept);
//   - `forward_out` writes into a caller-provided output tensor and takes an optional fp16 bias
//     (added in the kernel epilogue, bit-identical to `output += bias`) and the flags of
//     blkq4_fp16_gemm_sm100.
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/extension.h>

#include <algorithm>
#include <atomic>
#include <cstddef>
#include <cstdint>
#include <map>
#include <mutex>
#include <utility>
#include <vector>

#include <cuda_runtime.h>

#include "ms_blkq4gemm.h"

namespace {

constexpr size_t kHalfBytes = 2;

std::vector<torch::Tensor> blkq4linear_quant(int block_size, bool col_wise, bool has_offsets,
                                             torch::Tensor weights) {
  TORCH_CHECK(weights.scalar_type() == torch::kFloat16, "blkq4linear_quant only supports float16 weights");
  TORCH_CHECK(weights.numel() > 0, "blkq4linear_quant only supports non-empty tensors");
  TORCH_CHECK(weights.is_contiguous(), "blkq4linear_quant only supports contiguous tensors");
  TORCH_CHECK(weights.dim() == 2, "blkq4linear_quant only supports 2D tensors");
  TORCH_CHECK(weights.device().type() == at::kCUDA,
              "blkq4linear_quant only supports CUDA tensors, instead got ", weights.device().str());
  const int64_t out_features = weights.size(0);
  const int64_t in_features = weights.size(1);

  std::string err;
  int64_t w_size = 0, meta_size = 0;
  int rc = blkq4_fp16_quant_size_sm80(block_size, col_wise, int(in_features), int(out_features), w_size,
                                      meta_size, &err);
  TORCH_CHECK(rc == 0, err);

  const c10::cuda::CUDAGuard guard(weights.device());
  auto u8 = torch::TensorOptions().dtype(torch::kUInt8).device(weights.device());
  auto f16 = torch::TensorOptions().dtype(torch::kFloat16).device(weights.device());
  torch::Tensor q_weights = torch::empty({w_size}, u8);
  torch::Tensor q_scales = torch::empty({meta_size}, f16);
  torch::Tensor q_zp = torch::empty({has_offsets ? meta_size : 0}, u8);

  rc = blkq4_fp16_quant_sm80(block_size, col_wise, int(in_features), int(out_features), int(in_features),
                             c10::cuda::getCurrentCUDAStream().stream(), weights.data_ptr(),
                             size_t(weights.numel()) * kHalfBytes, q_weights.data_ptr(), size_t(w_size),
                             q_scales.data_ptr(), size_t(meta_size) * kHalfBytes,
                             has_offsets ? q_zp.data_ptr() : nullptr, has_offsets ? size_t(meta_size) : 0,
                             &err);
  TORCH_CHECK(rc == 0, err);
  return {q_weights, q_scales, q_zp};
}

torch::Tensor blkq4linear_forward_out(int block_size, bool col_wise, int in_features, int out_features,
                                      const torch::Tensor& input, const torch::Tensor& q_weights,
                                      const torch::Tensor& q_scales, const torch::Tensor& q_zp,
                                      const torch::Tensor& output, const c10::optional<torch::Tensor>& bias,
                                      int64_t flags, const c10::optional<torch::Tensor>& workspace) {
  TORCH_CHECK(input.scalar_type() == torch::kFloat16, "blkq4linear_forward only supports float16 inputs");
  TORCH_CHECK(input.dim() == 2 && input.size(1) == in_features,
              "Activation shape is not compatible with the weights");
  TORCH_CHECK(input.device().type() == torch::kCUDA, "blkq4linear_forward only supports CUDA inputs");
  TORCH_CHECK(input.is_contiguous(), "blkq4linear_forward only supports contiguous inputs");
  const auto dev = input.device();
  TORCH_CHECK(q_weights.device() == dev && q_scales.device() == dev &&
                  (!q_zp.defined() || q_zp.numel() == 0 || q_zp.device() == dev) && output.device() == dev,
              "blkq4linear_forward requires all tensors on the same device");
  TORCH_CHECK(output.scalar_type() == torch::kFloat16 && output.is_contiguous() && output.dim() == 2 &&
                  output.size(0) == input.size(0) && output.size(1) == out_features,
              "Output tensor must be a contiguous float16 [batch, out_features] tensor");

  const bool has_bias = bias.has_value() && bias->defined() && bias->numel() > 0;
  if (has_bias)
    TORCH_CHECK(bias->scalar_type() == torch::kFloat16 && bias->is_contiguous() && bias->device() == dev &&
                    bias->numel() == out_features,
                "Fused bias must be a contiguous float16 [out_features] tensor on the input's device");

  const c10::cuda::CUDAGuard guard(dev);
  const bool has_zp = q_zp.defined() && q_zp.numel() > 0;
  std::string err;
  const bool has_ws = workspace.has_value() && workspace->defined() && workspace->numel() > 0;
  if (has_ws)
    TORCH_CHECK(workspace->device() == dev && workspace->is_contiguous(),
                "The split-K workspace must be a contiguous tensor on the input's device");
  int rc = blkq4_fp16_gemm_ws_sm100(block_size, col_wise, int(input.size(0)), out_features, in_features,
                                 c10::cuda::getCurrentCUDAStream().stream(), input.data_ptr(),
                                 size_t(input.numel()) * kHalfBytes, q_weights.data_ptr(),
                                size_t(q_weights.numel()), q_scales.data_ptr(),
                                size_t(q_scales.numel()) * kHalfBytes, has_zp ? q_zp.data_ptr() : nullptr,
                                has_zp ? size_t(q_zp.numel()) : 0, output.data_ptr(),
                                size_t(output.numel()) * kHalfBytes, has_bias ? bias->data_ptr() : nullptr,
                                has_bias ? size_t(bias->numel()) * kHalfBytes : 0, unsigned(flags),
                                has_ws ? workspace->data_ptr() : nullptr,
                                has_ws ? size_t(workspace->numel()) * workspace->element_size() : 0, &err);
  TORCH_CHECK(rc == 0, err);
  return output;
}

torch::Tensor blkq4linear_forward(int block_size, bool col_wise, int in_features, int out_features,
                                  torch::Tensor input, torch::Tensor q_weights, torch::Tensor q_scales,
                                  torch::Tensor q_zp) {
  TORCH_CHECK(input.dim() == 2, "Activation shape is not compatible with the weights");
  auto output = torch::empty({input.size(0), out_features},
                             torch::TensorOptions().dtype(torch::kFloat16).device(input.device()));
  return blkq4linear_forward_out(block_size, col_wise, in_features, out_features, input, q_weights, q_scales,
                                 q_zp, output, c10::nullopt, 0, c10::nullopt);
}

// Layers that read the same activations, as one launch (blkq4_fp16_gemm_group_sm100): their packed tensors, zero points
// (all or none), fp16 biases or None, and the [rows, out_features] outputs to write.
void blkq4linear_group(int block_size, bool col_wise, int in_features, const torch::Tensor& input,
                       const std::vector<torch::Tensor>& q_weights, const std::vector<torch::Tensor>& q_scales,
                       const std::vector<torch::Tensor>& q_zp, const std::vector<c10::optional<torch::Tensor>>& bias,
                       const std::vector<torch::Tensor>& outputs, int64_t flags,
                       const c10::optional<torch::Tensor>& workspace) {
  const size_t count = q_weights.size();
  TORCH_CHECK(count >= 2 && count <= 4 && q_scales.size() == count && q_zp.size() == count && bias.size() == count &&
                  outputs.size() == count,
              "A group has two to four layers");
  TORCH_CHECK(input.scalar_type() == torch::kFloat16 && input.dim() == 2 && input.size(1) == in_features &&
                  input.is_contiguous() && input.device().type() == torch::kCUDA,
              "Activations must be a contiguous float16 CUDA tensor [rows, in_features]");
  const auto dev = input.device();
  blkq4_gemm_part parts[4] = {};
  for (size_t i = 0; i < count; ++i) {
    const bool has_bias = bias[i].has_value() && bias[i]->defined() && bias[i]->numel() > 0;
    TORCH_CHECK(q_weights[i].device() == dev && q_scales[i].device() == dev && outputs[i].device() == dev &&
                    (q_zp[i].numel() == 0 || q_zp[i].device() == dev) && (!has_bias || bias[i]->device() == dev),
                "A group requires all tensors on the same device");
    TORCH_CHECK(outputs[i].scalar_type() == torch::kFloat16 && outputs[i].is_contiguous() && outputs[i].dim() == 2 &&
                    outputs[i].size(0) == input.size(0),
                "Outputs must be contiguous float16 [rows, out_features] tensors");
    TORCH_CHECK(!has_bias || (bias[i]->scalar_type() == torch::kFloat16 && bias[i]->is_contiguous()),
                "Fused biases must be contiguous float16 tensors");
    auto& p = parts[i];
    p.n = int(outputs[i].size(1));
    p.weights = q_weights[i].data_ptr();
    p.weights_size = size_t(q_weights[i].numel());
    p.scales = q_scales[i].data_ptr();
    p.scales_size = size_t(q_scales[i].numel()) * kHalfBytes;
    if (q_zp[i].numel() > 0) {
      p.offsets = q_zp[i].data_ptr();
      p.offsets_size = size_t(q_zp[i].numel());
    }
    p.output = outputs[i].data_ptr();
    p.output_size = size_t(outputs[i].numel()) * kHalfBytes;
    if (has_bias) {
      p.bias = bias[i]->data_ptr();
      p.bias_size = size_t(bias[i]->numel()) * kHalfBytes;
    }
  }
  const bool has_ws = workspace.has_value() && workspace->defined() && workspace->numel() > 0;
  TORCH_CHECK(!has_ws || (workspace->device() == dev && workspace->is_contiguous()),
              "The split-K workspace must be a contiguous tensor on the input's device");
  const c10::cuda::CUDAGuard guard(dev);
  std::string err;
  const int rc = blkq4_fp16_gemm_group_sm100(block_size, col_wise, int(input.size(0)), in_features,
                                             c10::cuda::getCurrentCUDAStream().stream(), input.data_ptr(),
                                             size_t(input.numel()) * kHalfBytes, int(count), parts, unsigned(flags),
                                             has_ws ? workspace->data_ptr() : nullptr, has_ws ? workspace->nbytes() : 0, &err);
  TORCH_CHECK(rc == 0, err);
}

// ---- workspaces of calls that are being captured into a CUDA graph ----
// The graph keeps the buffer's address, so the graph keeps the buffer: a user object of the graph holds the tensor
// until the graph and everything instantiated from it are gone.  One buffer per capture and stream, its flag words
// zeroed by a node of the same graph, so that graphs share nothing and may replay side by side.
std::mutex g_dropped_mutex;
std::vector<torch::Tensor>& g_dropped = *new std::vector<torch::Tensor>;  // outlives static destruction
std::atomic<bool> g_any_dropped{false};
std::atomic<int> g_graph_workspaces{0};

// Gives the buffers of graphs that are gone back to the allocator.
int free_dropped_workspaces(void*) {
  std::vector<torch::Tensor> dropped;
  std::lock_guard<std::mutex> lock(g_dropped_mutex);
  dropped.swap(g_dropped);
  g_any_dropped.store(false);
  return 0;  // the lock goes first, then the tensors
}

// A user object's destructor may run on any thread and may not call CUDA, so it leaves the buffer to the
// interpreter's next pending calls, or, should that queue be full, to the next call of graph_workspace.
void drop_graph_workspace(void* held) {
  auto* buffer = static_cast<torch::Tensor*>(held);
  {
    std::lock_guard<std::mutex> lock(g_dropped_mutex);
    g_dropped.push_back(std::move(*buffer));
    g_any_dropped.store(true);
  }
  delete buffer;
  --g_graph_workspaces;
  if (Py_IsInitialized()) Py_AddPendingCall(free_dropped_workspaces, nullptr);
}

// The workspace of at least `nbytes` for the capture that is under way on the device's current stream (`stream`);
// nothing when none is, an empty tensor when the graph cannot take one.  Called with the GIL held.
c10::optional<torch::Tensor> graph_workspace(int device, uintptr_t stream_handle, int64_t nbytes) {
  if (g_any_dropped.load()) free_dropped_workspaces(nullptr);
  const auto stream = reinterpret_cast<cudaStream_t>(stream_handle);
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  unsigned long long id = 0;
  cudaGraph_t graph = nullptr;
  if (cudaStreamGetCaptureInfo(stream, &status, &id, &graph) != cudaSuccess) {
    cudaGetLastError();
    return c10::nullopt;
  }
  if (status == cudaStreamCaptureStatusNone) return c10::nullopt;
  const c10::cuda::CUDAGuard guard(static_cast<c10::DeviceIndex>(device));
  const auto u8 = torch::TensorOptions().dtype(torch::kUInt8).device(torch::kCUDA, static_cast<c10::DeviceIndex>(device));
  if (status != cudaStreamCaptureStatusActive) return torch::empty({0}, u8);

  // the last capture of each stream; its tensor is there as long as that capture is under way (ids are never reused)
  static auto& last = *new std::map<std::pair<int, cudaStream_t>, std::pair<unsigned long long, torch::Tensor*>>;
  auto& slot = last[{device, stream}];
  if (slot.first == id && slot.second && slot.second->numel() >= nbytes) return *slot.second;
  auto* held = new torch::Tensor(torch::empty({nbytes}, u8));
  ++g_graph_workspaces;
  torch::Tensor buffer = *held;
  cudaUserObject_t object = nullptr;
  if (cudaUserObjectCreate(&object, held, drop_graph_workspace, 1, cudaUserObjectNoDestructorSync) != cudaSuccess) {
    cudaGetLastError();
    drop_graph_workspace(held);
    return torch::empty({0}, u8);
  }
  // flag words: at most one per SM, far below 64 KB; the partial tiles behind them need no clearing
  if (cudaGraphRetainUserObject(graph, object, 1, cudaGraphUserObjectMove) != cudaSuccess) {
    cudaGetLastError();
    cudaUserObjectRelease(object, 1);
    return torch::empty({0}, u8);
  }
  slot = {id, held};
  C10_CUDA_CHECK(cudaMemsetAsync(buffer.data_ptr(), 0, size_t(std::min<int64_t>(nbytes, 64 << 10)), stream));
  return buffer;
}

// ---- BlkQ4Linear.forward ----
// Where split-K workspaces come from: `eager` is the module's dict (device, stream) -> tensor, `provide(device, nbytes)`
// its function for every other case, both null until somebody imports that module; `owners` counts the blocks in which somebody else provides them, in any thread.
PyObject* g_eager_workspaces = nullptr;
PyObject* g_provide_workspace = nullptr;
std::atomic<int> g_workspace_owners{0};

// The workspace of a call on the device's current stream; none without a source of them.  The common case, an eager call on
// a stream that has a buffer of the size, is answered here.
c10::optional<torch::Tensor> split_k_workspace(int device, int64_t nbytes) {
  if (!g_eager_workspaces || !g_provide_workspace) return c10::nullopt;
  const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(device)).stream();
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(stream, &status) != cudaSuccess) {
    cudaGetLastError();
    status = cudaStreamCaptureStatusInvalidated;
  }
  if (status == cudaStreamCaptureStatusNone && g_workspace_owners.load() == 0 && !g_any_dropped.load()) {
    const py::tuple key = py::make_tuple(device, reinterpret_cast<uintptr_t>(stream));
    PyObject* found = PyDict_GetItemWithError(g_eager_workspaces, key.ptr());  // borrowed
    if (found && THPVariable_Check(found)) {
      const torch::Tensor& ws = THPVariable_Unpack(found);
      if (ws.numel() >= nbytes) return ws;
    }
    if (!found && PyErr_Occurred()) throw py::error_already_set();
  }
  const py::object ws = py::reinterpret_borrow<py::object>(g_provide_workspace)(device, nbytes);
  if (ws.is_none()) return c10::nullopt;
  return ws.cast<torch::Tensor>();
}

// The whole of BlkQ4Linear.forward but a bias that cannot be fused: leading dimensions flattened, the split-K workspace
// found, the output allocated unless the caller brought one, the launch, the leading dimensions restored.  In one call
// because at decode sizes the Python calls around the launch took longer than the kernel, and with CPython's vectorcall
// signature because pybind11 took about 1 us to convert the arguments.  Measured, host time per call: one token 6.7 -> 6.1 us,
// with a split-K workspace (M = 333) 12.7 -> 7.8.
constexpr int kLinearArgs = 12;
constexpr const char* kLinearNames[kLinearArgs] = {"block_size", "col_wise", "in_features", "out_features", "input", "q_weights",
                                                   "q_scales", "q_zp", "bias", "flags", "workspace", "out"};

PyObject* linear_positional(PyObject* const* args) {
  HANDLE_TH_ERRORS
  auto integer = [&](int i) {
    const long v = PyLong_AsLong(args[i]);
    if (v == -1 && PyErr_Occurred()) throw python_error();
    return v;
  };
  auto small = [&](int i) {
    const long v = integer(i);
    TORCH_CHECK_TYPE(v == long(int(v)), "linear: ", kLinearNames[i], " = ", v, " is out of range");
    return int(v);
  };
  auto truth = [&](int i) {
    const int v = PyObject_IsTrue(args[i]);
    if (v < 0) throw python_error();
    return v == 1;
  };
  auto tensor = [&](int i) -> const torch::Tensor& {
    TORCH_CHECK_TYPE(THPVariable_Check(args[i]), "linear: ", kLinearNames[i], " must be a tensor");
    return THPVariable_Unpack(args[i]);
  };
  const int block_size = small(0), in_features = small(2), out_features = small(3);
  const bool col_wise = truth(1);
  const torch::Tensor &input = tensor(4), &q_weights = tensor(5), &q_scales = tensor(6), &q_zp = tensor(7);
  c10::optional<torch::Tensor> bias, workspace;
  if (args[8] != Py_None) bias = tensor(8);
  int64_t flags = integer(9);
  // the caller's workspace, or whether to find one (a bool first: asking whether one is a tensor takes 0.1 us)
  bool split_k = args[10] == Py_True;
  if (!split_k && args[10] != Py_False && args[10] != Py_None) {
    if (THPVariable_Check(args[10])) workspace = tensor(10);
    else split_k = truth(10);
  }
  torch::Tensor output;
  {
    const bool flat = input.dim() == 2 && input.size(1) == in_features && input.is_contiguous();
    const torch::Tensor x = flat ? input : input.reshape({-1, in_features});
    const int64_t rows = x.size(0);
    if (split_k && x.is_cuda() && (rows > 16 || block_size < 64 || !col_wise)) {  // the others never use one
      const c10::cuda::CUDAGuard guard(x.device());
      const size_t need = blkq4_gemm_workspace_size_sm100(block_size, col_wise, int(rows), out_features, in_features);
      if (need > 0) {
        workspace = split_k_workspace(x.device().index(), int64_t(need));
        flags |= BLKQ4_GEMM_SKINNY_WORKSPACE;
      }
    }
    const bool brought = args[11] != Py_None;
    output = brought ? tensor(11).view({-1, out_features})
                     : torch::empty({rows, out_features}, torch::TensorOptions().dtype(torch::kFloat16).device(x.device()));
    blkq4linear_forward_out(block_size, col_wise, in_features, out_features, x, q_weights, q_scales, q_zp, output, bias,
                            flags, workspace);
    if (!flat || brought) {
      auto shape = input.sizes().vec();
      shape.back() = out_features;
      output = output.view(shape);
    }
  }
  return THPVariable_Wrap(output);
  END_HANDLE_TH_ERRORS
}

// The arguments by position; `named`: where those given by keyword are put.
PyObject* const* linear_arguments(PyObject* const* given, Py_ssize_t nargs, PyObject* kwnames, PyObject** named) {
  const Py_ssize_t nkw = kwnames ? PyTuple_GET_SIZE(kwnames) : 0;
  TORCH_CHECK_TYPE(nargs + nkw == kLinearArgs,
                   "linear(block_size, col_wise, in_features, out_features, input, q_weights, q_scales, q_zp, bias, flags, workspace, out)");
  std::copy(given, given + nargs, named);
  for (Py_ssize_t k = 0; k < nkw; ++k) {
    int i = 0;
    while (i < kLinearArgs && PyUnicode_CompareWithASCIIString(PyTuple_GET_ITEM(kwnames, k), kLinearNames[i]) != 0) ++i;
    TORCH_CHECK_TYPE(i < kLinearArgs && !named[i], "linear: a keyword that it does not have, or an argument given twice");
    named[i] = given[nargs + k];
  }
  return named;
}

PyObject* linear_fastcall(PyObject*, PyObject* const* args, Py_ssize_t nargs, PyObject* kwnames) {
  if (nargs == kLinearArgs && !kwnames) return linear_positional(args);
  HANDLE_TH_ERRORS
  PyObject* named[kLinearArgs] = {};
  return linear_positional(linear_arguments(args, nargs, kwnames, named));
  END_HANDLE_TH_ERRORS
}

PyMethodDef g_methods[] = {
    {"linear", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(linear_fastcall)), METH_FASTCALL | METH_KEYWORDS,
     "BlkQ4Linear.forward: any leading dimensions, the output allocated unless given; workspace: a tensor, or whether to find one"},
    {nullptr, nullptr, 0, nullptr}};

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  m.def("quant", &blkq4linear_quant, "Quantize float 16 weights");
  m.def("forward", &blkq4linear_forward, "Forward pass for block quantized linear layer");
  m.def("forward_out", &blkq4linear_forward_out, "Forward pass into a caller-provided output tensor",
        py::arg("block_size"), py::arg("col_wise"), py::arg("in_features"), py::arg("out_features"),
        py::arg("input"), py::arg("q_weights"), py::arg("q_scales"), py::arg("q_zp"), py::arg("output"),
        py::arg("bias") = py::none(), py::arg("flags") = 0, py::arg("workspace") = py::none());
  if (PyModule_AddFunctions(m.ptr(), g_methods) != 0) throw py::error_already_set();
  m.def("workspace_source",
        [](py::dict eager, py::function provide) {
          g_eager_workspaces = eager.release().ptr();
          g_provide_workspace = provide.release().ptr();
        },
        "Where linear takes split-K workspaces from");
  m.def("workspace_owners", [](int change) { g_workspace_owners += change; },
        "Counts the blocks in which workspaces come from somewhere else");
  m.def("linear_group", &blkq4linear_group, "Layers that read the same activations, as one launch");
  m.def("linear_group_supported",
        [](int block, bool col_wise, int m_, int k_, const std::vector<int>& n_) {
          return blkq4_gemm_group_supported_sm100(block, col_wise, m_, k_, int(n_.size()), n_.data()) != 0;
        },
        "Whether one launch takes layers of these widths");
  m.def("linear_group_keeps_bits",
        [](int block, bool col_wise, int m_, int k_, const std::vector<int>& n_) {
          return blkq4_gemm_group_keeps_bits_sm100(block, col_wise, m_, k_, int(n_.size()), n_.data()) != 0;
        },
        "Whether linear_group with its workspace gives every bit of the layers' own calls with theirs");
  m.def("gemm_plan",
        [](int m_, int n_, int k_) {
          int plan[6];
          blkq4_gemm_plan(m_, n_, k_, 0, plan);
          return py::make_tuple(plan[0], plan[2]);
        },
        "Kernel and output tiles of a call without a workspace (blkq4_gemm_plan)");
  m.def("linear_group_workspace_size",
        [](int block, bool col_wise, int m_, int k_, const std::vector<int>& n_) {
          return int64_t(blkq4_gemm_group_workspace_size_sm100(block, col_wise, m_, k_, int(n_.size()), n_.data()));
        },
        "Bytes of zeroed workspace with which linear_group splits K (0: it does not)");
  m.def("gemm_workspace_size_blocked",
        [](int block, bool col_wise, int m_, int n_, int k_) {
          return int64_t(blkq4_gemm_workspace_size_sm100(block, col_wise, m_, n_, k_));
        },
        "Bytes of workspace of a call with SKINNY_WORKSPACE, for any row count");
  m.def("gemm_workspace_size", [](int m_, int n_, int k_) { return int64_t(blkq4_gemm_workspace_size(m_, n_, k_)); },
        "Bytes of zeroed workspace with which the tensor-core kernel splits K (0: it does not)");
  m.def("graph_workspace", &graph_workspace,
        "Workspace owned by the CUDA graph that the device's current stream is being captured into, else None",
        py::arg("device"), py::arg("stream"), py::arg("nbytes"));
  m.def("graph_workspaces", [] { return g_graph_workspaces.load(); }, "Workspaces that CUDA graphs hold at present");
  m.attr("EARLY_WEIGHT_FETCH") = int(BLKQ4_GEMM_EARLY_WEIGHT_FETCH);
  m.attr("SKINNY_WORKSPACE") = int(BLKQ4_GEMM_SKINNY_WORKSPACE);
  m.def("library_version", []() { return std::string(blkq4_version()); });
}
