// Native host side of the eager calls: argument checks, output and scratch allocation and the launches of one call, without
// the interpreter in between. A small decode call occupies the GPU for ten to twenty microseconds; the same steps in Python
// (a dozen attribute reads, checks and conversions per launch) took 25 to 120, so the calls were bound by the host.
// The functions take positional arguments only and are called by the package's own Python layer.
#include <Python.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/torch.h>

#include <map>
#include <memory>
#include <mutex>
#include <string>
#include <utility>
#include <vector>

#include "../../include/inkling_b200.h"

namespace {

// Errors keep the types that the Python layer's calls have: AssertionError for an argument of the wrong form, RuntimeError for
// what the library refuses and for tensors that are not on the GPU, torch's own (out of memory, say) for what torch throws.
struct Failure {
  std::string what;
  PyObject* type = nullptr;   // null: the interpreter's error is set already
};
[[noreturn]] void fail(const std::string& what) { throw Failure{what, PyExc_RuntimeError}; }
void check(int code) {
  if (code != 0) fail("inkling_b200: " + std::string(ink_last_error()) + " (code " + std::to_string(code) + ")");
}

const at::Tensor& tensor_at(PyObject* const* args, Py_ssize_t i) {
  if (!THPVariable_Check(args[i])) throw Failure{"argument " + std::to_string(i) + " is not a tensor", PyExc_TypeError};
  return THPVariable_Unpack(args[i]);
}
bool given(PyObject* const* args, Py_ssize_t i) { return args[i] != Py_None; }
long long int_at(PyObject* const* args, Py_ssize_t i) {
  const long long v = PyLong_AsLongLong(args[i]);
  if (v == -1 && PyErr_Occurred()) throw Failure{};
  return v;
}
double float_at(PyObject* const* args, Py_ssize_t i) {
  const double v = PyFloat_AsDouble(args[i]);
  if (v == -1.0 && PyErr_Occurred()) throw Failure{};
  return v;
}
void require(bool ok, const char* what) {
  if (!ok) throw Failure{what, PyExc_AssertionError};
}
void require_cuda(const at::Tensor& t) {
  if (!t.is_cuda()) fail("inkling_b200 kernels run on CUDA tensors only (no CPU path)");
}
void require_reshape(bool ok, const char* what) {   // (what torch's reshape refuses, and with its type)
  if (!ok) fail(what);
}
// a contiguous BF16 tensor on the GPU, its data on a 16-byte boundary
at::Tensor bf16_rows(const at::Tensor& t, const char* what) {
  require(t.scalar_type() == at::kBFloat16, what);
  require_cuda(t);
  at::Tensor c = t.is_contiguous() ? t : t.contiguous();
  return (reinterpret_cast<uintptr_t>(c.data_ptr()) & 15) ? c.clone() : c;
}
// Allocation and launches run without the interpreter's lock: a launch waits while the stream's queue is full, and the other
// threads, or a host function that a stream is waiting for, may need the interpreter meanwhile. (The caller's frame holds the
// arguments.)
struct WithoutGil {
  PyThreadState* const state = PyEval_SaveThread();
  ~WithoutGil() { PyEval_RestoreThread(state); }
};
at::Tensor new_tensor(at::IntArrayRef sizes, at::ScalarType type, const at::Device& device) {
  return at::empty(sizes, at::TensorOptions().dtype(type).device(device));
}

// ------------------------------------------------------------------------------------------------ attention
// The join's workspace starts with counters that are zero between launches. An eager call keeps one for its stream (made
// again, zeroed, when the sizes change; at most kMostWorkspaces, then the pool starts anew -- the memory goes back to the
// allocator, which hands it out on the same stream only). A call under capture gets its own from the graph's pool, its
// counters cleared by the graph: graphs may be replayed in any order, on any stream. (`joins`: the call counts at all. A
// node that clears memory between two kernels costs 8 us.)
at::Tensor attention_workspace(const at::Device& device, cudaStream_t stream, size_t bytes, size_t counters, bool joins) {
  const auto options = at::TensorOptions().dtype(at::kByte).device(device);
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(stream, &capture) != cudaSuccess || capture != cudaStreamCaptureStatusNone) {
    const at::Tensor t = at::empty({(int64_t)bytes}, options);
    if (joins && cudaMemsetAsync(t.data_ptr(), 0, counters, stream) != cudaSuccess) fail("decode_attention: the workspace could not be cleared");
    return t;
  }
  struct Workspace {
    size_t counters = 0;
    at::Tensor t;
  };
  constexpr size_t kMostWorkspaces = 64;
  static std::mutex mutex;
  static auto* pool = new std::map<std::pair<int, cudaStream_t>, Workspace>();   // (not destroyed at exit: the CUDA context may be gone)
  const std::lock_guard<std::mutex> lock(mutex);
  if (pool->size() >= kMostWorkspaces && !pool->count({device.index(), stream})) pool->clear();
  Workspace& kept = (*pool)[{device.index(), stream}];
  if (!kept.t.defined() || kept.counters != counters || (size_t)kept.t.numel() < bytes) {
    kept.t = at::Tensor();
    kept.t = at::zeros({(int64_t)bytes}, options);
    kept.counters = counters;
  }
  return kept.t;
}

// (query, relative_states, proj, k_cache, v_cache, position, pad_counts, window, n_floor, alpha, scale, out, new_key, new_value)
PyObject* decode_attention(PyObject* const* args) {
  const at::Tensor &query = tensor_at(args, 0), &states = tensor_at(args, 1), &proj = tensor_at(args, 2), &k = tensor_at(args, 3), &v = tensor_at(args, 4);
  require(THPVariable_Check(args[5]) && tensor_at(args, 5).scalar_type() == at::kLong, "decode_attention: int64 position on the device");
  const at::Tensor& position = tensor_at(args, 5);
  for (const at::Tensor* t : {&query, &states, &proj, &k, &v}) require(t->scalar_type() == at::kBFloat16, "decode_attention: BF16 query, relative states, proj and caches");
  require(query.dim() >= 3 && k.dim() == 4 && proj.dim() == 2, "decode_attention: query [bs, h, (1,) c], caches [bs, hk, slots, c], proj [d_rel, extent]");
  const int64_t bs = query.size(0), h = query.size(1), c = query.size(-1), hk = k.size(1), slots = k.size(2), d_rel = proj.size(0);
  require(proj.is_contiguous() && k.is_contiguous() && v.is_contiguous() && k.sizes() == v.sizes(), "decode_attention: contiguous proj and caches of one shape");
  require(k.size(0) == bs && k.size(3) == c, "decode_attention: caches of the query's batch and head width");
  require_reshape(query.numel() == bs * h * c, "decode_attention: one query per sequence and head");
  require(states.numel() == bs * h * d_rel, "decode_attention: one relative state per sequence and head");
  const void* pads = nullptr;
  if (given(args, 6)) {
    const at::Tensor& p = tensor_at(args, 6);
    require(p.scalar_type() == at::kLong && p.numel() == bs && p.is_contiguous(), "decode_attention: int64 pad_counts [bs]");
    require_cuda(p);
    pads = p.data_ptr();
  }
  for (const at::Tensor* t : {&states, &proj, &k, &v, &position}) require_cuda(*t);
  at::Tensor out, new_k, new_v;
  if (given(args, 11)) {
    out = tensor_at(args, 11);
    require_cuda(out);
  }
  if (given(args, 12)) {
    require(given(args, 13), "decode_attention: new_key and new_value come together");
    new_k = tensor_at(args, 12);
    new_v = tensor_at(args, 13);
    require_reshape(new_k.numel() == bs * hk * c && new_v.numel() == bs * hk * c, "decode_attention: one new key and value per sequence and key/value head");
  }
  const int window = (int)int_at(args, 7), n_floor = (int)int_at(args, 8);
  const float alpha = (float)float_at(args, 9), scale = (float)float_at(args, 10);
  {
    const WithoutGil unlocked;
    const at::Tensor q = bf16_rows(query, "decode_attention: BF16 query");
    const at::Tensor r = states.is_contiguous() ? states : states.contiguous();
    if (new_k.defined()) {
      new_k = bf16_rows(new_k, "decode_attention: BF16 new_key");
      new_v = bf16_rows(new_v, "decode_attention: BF16 new_value");
    }
    const c10::cuda::CUDAGuard guard(q.device());
    const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(q.device().index()).stream();
    if (!out.defined()) out = new_tensor({bs, h, 1, c}, at::kBFloat16, q.device());
    const size_t need = ink_decode_attention_workspace_bytes((int)bs, (int)h, (int)c, (int)slots);
    at::Tensor workspace;
    if (need) workspace = attention_workspace(q.device(), stream, need, ink_decode_attention_counter_bytes((int)bs, (int)h),
                                              ink_decode_attention_joins((int)bs, (int)h, (int)hk, (int)c, (int)slots) != 0);
    check(ink_decode_attention(q.data_ptr(), r.data_ptr(), proj.data_ptr(), k.data_ptr(), v.data_ptr(), (const int64_t*)position.data_ptr(), (const int64_t*)pads,
                               out.data_ptr(), (int)bs, (int)h, (int)hk, (int)c, (int)d_rel, (int)proj.size(1), (int)slots, window, n_floor, alpha, scale, new_k.defined() ? new_k.data_ptr() : nullptr,
                               new_v.defined() ? new_v.data_ptr() : nullptr, need ? workspace.data_ptr() : nullptr, need, stream));
  }
  return THPVariable_Wrap(out);
}

// ------------------------------------------------------------------------------------------------ blocks
// What the calls need of a module, taken down once (the module makes a new record when one of its tensors is replaced).
// The record holds the tensors themselves beside what was found of them: a tensor whose storage, type, sizes or strides were
// exchanged underneath shows, and the call then returns NotImplemented for the module to check it and make a new record.
struct Kept {
  int field;
  at::Tensor t;
  at::ScalarType type;
  at::DimVector sizes, strides;
};
struct Block {
  long long v[48] = {};
  std::vector<Kept> kept;
  std::shared_ptr<std::mutex> launching;   // see launch_lock
  bool current() const {
    for (const Kept& k : kept)
      if ((long long)(uintptr_t)k.t.data_ptr() != v[k.field] || k.t.scalar_type() != k.type || k.t.sizes() != at::IntArrayRef(k.sizes) ||
          k.t.strides() != at::IntArrayRef(k.strides))
        return false;
    return true;
  }
};
enum Field {
  kHidden, kWidth, kTopK, kShared, kStart, kLocal, kStride, kCapacity, kMaxExpert, kQuantized, kTokens, kRouted,
  kSources, kPointers, kExperts, kCounts, kRows, kActivated, kDown, kStatus, kBankMaps,
  kRouterWeight, kRouterBias, kGlobalScale, kSharedMaps, kTopkWeights, kTopkIndices, kGammas, kWorkspace, kWorkspaceBytes, kPartial,
  kTable, kScratch, kScratchBytes, kStackFlags, kStackStatus, kRouteScaleBits, kSharedGate, kSharedUp, kSharedDown, kFields
};
const char* const kFieldNames[kFields] = {
    "hidden", "width", "top_k", "shared", "start", "local", "stride", "capacity", "max_expert", "quantized", "tokens", "routed",
    "sources", "pointers", "experts", "counts", "rows", "activated", "down", "status", "bank_maps",
    "router_weight", "router_bias", "global_scale", "shared_maps", "topk_weights", "topk_indices", "gammas", "workspace", "workspace_bytes", "partial",
    "table", "scratch", "scratch_bytes", "stack_flags", "stack_status", "route_scale_bits", "shared_gate", "shared_up", "shared_down"};
template <typename T>
T* at_field(const Block& b, Field f) {
  return reinterpret_cast<T*>((uintptr_t)b.v[f]);
}

// The launches of a call hand buffers of the module from one to the next, so they go to their stream as one sequence although
// the interpreter is free meanwhile: one lock per pointer table, i.e. for a module of experts and every block that uses it.
std::shared_ptr<std::mutex> launch_lock(long long pointers) {
  if (!pointers) return std::make_shared<std::mutex>();   // (a record for one token: a single launch)
  static std::mutex mutex;
  static auto* locks = new std::map<long long, std::weak_ptr<std::mutex>>();
  const std::lock_guard<std::mutex> lock(mutex);
  for (auto it = locks->begin(); it != locks->end();) it = it->second.expired() ? locks->erase(it) : std::next(it);
  std::shared_ptr<std::mutex> found = (*locks)[pointers].lock();
  if (!found) (*locks)[pointers] = found = std::make_shared<std::mutex>();
  return found;
}

PyObject* make_block(PyObject* const* args) {
  auto block = std::make_unique<Block>();
  for (int f = 0; f < kFields; ++f) {
    PyObject* item = PyDict_GetItemString(args[0], kFieldNames[f]);
    if (!item) continue;
    if (THPVariable_Check(item)) {
      const at::Tensor& t = THPVariable_Unpack(item);
      block->v[f] = (long long)(uintptr_t)t.data_ptr();
      block->kept.push_back({f, t, t.scalar_type(), at::DimVector(t.sizes()), at::DimVector(t.strides())});
      continue;
    }
    block->v[f] = PyLong_AsLongLong(item);
    if (block->v[f] == -1 && PyErr_Occurred()) throw Failure{};
  }
  block->launching = launch_lock(block->v[kPointers]);
  PyObject* capsule = PyCapsule_New(block.get(), "inkling_block", [](PyObject* c) { delete (Block*)PyCapsule_GetPointer(c, "inkling_block"); });
  if (capsule) (void)block.release();
  return capsule;
}
const Block& block_at(PyObject* const* args) {
  auto* block = (const Block*)PyCapsule_GetPointer(args[0], "inkling_block");
  if (!block) throw Failure{};
  return *block;
}
struct Rows {   // the block's input as [tokens, hidden]
  at::Tensor x;
  int tokens;
};
Rows rows_of(const Block& b, const at::Tensor& t) {
  require(t.dim() >= 1 && t.size(-1) == b.v[kHidden], "input of another width than the block's");
  Rows r{bf16_rows(t, "BF16 input expected"), 0};
  r.tokens = (int)(t.numel() / b.v[kHidden]);
  return r;
}

// Tokens of a many-token call that are planned and projected at a time: the images of the tokens take about 85 KB a token
// at full width (2.7 GB), the banks are read once per 32 768 tokens (0.5 of about 20 ms), and the kernels' 32-bit work
// counters hold sixteen times as many with the router's most choices (32).
constexpr int kMostTokens = 32768;
void grouped(const Block& b, const Rows& r, int t0, int tokens, const int64_t* indices, const char* weights, const char* gammas, float* partial, void* out,
             int n_shared, cudaStream_t stream) {
  const int top_k = (int)b.v[kTopK], hidden = (int)b.v[kHidden];
  const int routes = tokens * top_k, groups = routes < b.v[kLocal] ? routes : (int)b.v[kLocal];
  const size_t need = ink_moe_grouped_scratch_bytes(tokens, top_k, n_shared, hidden, (int)b.v[kWidth], groups, (int)b.v[kQuantized]);
  const at::Tensor scratch = new_tensor({(int64_t)need}, at::kByte, r.x.device());   // (of this stream, or of the graph being captured)
  const size_t before = (size_t)t0 * hidden;
  check(ink_moe_grouped((const char*)r.x.data_ptr() + 2 * before, indices, weights, at_field<int64_t>(b, kPointers), at_field<int32_t>(b, kExperts),
                        at_field<int32_t>(b, kRows), at_field<int32_t>(b, kCounts), at_field<void>(b, kBankMaps),
                        n_shared ? at_field<void>(b, kSharedMaps) : nullptr, n_shared ? gammas : nullptr, at_field<void>(b, kActivated), at_field<void>(b, kDown),
                        partial ? partial + before : nullptr, out ? (char*)out + 2 * before : nullptr, tokens, top_k, n_shared, hidden, (int)b.v[kWidth], groups,
                        (int)b.v[kStart], (int)b.v[kLocal], (int)b.v[kCapacity], (int)b.v[kMaxExpert], (int)b.v[kQuantized], scratch.data_ptr(), need,
                        at_field<int32_t>(b, kStatus), stream));
}

at::Tensor block_forward(const Block& b, const at::Tensor& input, bool want_partial) {
  const Rows r = rows_of(b, input);
  require(r.tokens <= b.v[kTokens] && (r.tokens == 1 || std::min(r.tokens, kMostTokens) * b.v[kTopK] <= b.v[kCapacity]), "more tokens than the block's buffers hold");
  const c10::cuda::CUDAGuard guard(r.x.device());
  const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(r.x.device().index()).stream();
  const std::lock_guard<std::mutex> one_call(*b.launching);
  at::Tensor out;
  if (!want_partial) out = new_tensor(input.sizes(), at::kBFloat16, r.x.device());
  if (r.tokens == 1 && b.v[kTable]) {
    check(ink_moe_stack_decode(at_field<void>(b, kTable), 1, r.x.data_ptr(), nullptr, want_partial ? nullptr : out.data_ptr(), at_field<float>(b, kPartial),
                               (int)b.v[kStackFlags], 1e-6f, (int)b.v[kHidden], (int)b.v[kWidth], (int)b.v[kRouted], (int)b.v[kShared], (int)b.v[kTopK],
                               at_field<void>(b, kScratch), (size_t)b.v[kScratchBytes], at_field<int32_t>(b, kStackStatus), stream));
  } else if (r.tokens > 0) {
    require(b.v[kBankMaps] != 0, "a record for one token only");
    float route_scale;
    const uint32_t bits = (uint32_t)b.v[kRouteScaleBits];
    memcpy(&route_scale, &bits, sizeof(route_scale));
    for (int t0 = 0; t0 < r.tokens; t0 += kMostTokens) {
      const int tokens = std::min(kMostTokens, r.tokens - t0);
      const size_t routes0 = (size_t)t0 * b.v[kTopK];
      char *weights = at_field<char>(b, kTopkWeights) + 2 * routes0, *gammas = at_field<char>(b, kGammas) + 2 * (size_t)t0 * b.v[kShared];
      int64_t* indices = at_field<int64_t>(b, kTopkIndices) + routes0;
      check(ink_router_plan_forward((const char*)r.x.data_ptr() + 2 * (size_t)t0 * b.v[kHidden], at_field<void>(b, kRouterWeight), at_field<float>(b, kRouterBias),
                                    at_field<void>(b, kGlobalScale), route_scale, tokens, (int)b.v[kHidden], (int)b.v[kRouted], (int)b.v[kShared], (int)b.v[kTopK],
                                    nullptr, weights, indices, gammas, at_field<void>(b, kWorkspace), (size_t)b.v[kWorkspaceBytes], at_field<int64_t>(b, kSources),
                                    at_field<int64_t>(b, kPointers), at_field<int32_t>(b, kExperts), at_field<int32_t>(b, kCounts), at_field<int32_t>(b, kRows),
                                    (int)b.v[kStart], (int)b.v[kLocal], (int)b.v[kStride], (int)b.v[kCapacity], stream));
      grouped(b, r, t0, tokens, indices, weights, gammas, want_partial ? at_field<float>(b, kPartial) : nullptr, want_partial ? nullptr : out.data_ptr(),
              (int)b.v[kShared], stream);
    }
  }
  return out;
}
// (block, x, want_partial) -> BF16 like x; with want_partial the FP32 output goes to the block's own buffer, None is returned
PyObject* run_block(PyObject* const* args) {
  const Block& b = block_at(args);
  if (!b.current()) Py_RETURN_NOTIMPLEMENTED;
  const at::Tensor& input = tensor_at(args, 1);
  const bool want_partial = args[2] == Py_True;
  at::Tensor out;
  {
    const WithoutGil unlocked;
    out = block_forward(b, input, want_partial);
  }
  if (want_partial) Py_RETURN_NONE;
  return THPVariable_Wrap(out);
}

at::Tensor experts_forward(const Block& b, const at::Tensor& input, const at::Tensor& i, const at::Tensor& w) {
  const Rows r = rows_of(b, input);
  const at::Tensor weights = bf16_rows(w, "BF16 router weights expected");
  require(i.scalar_type() == at::kLong && i.numel() == r.tokens * b.v[kTopK] && weights.numel() == i.numel(), "int64 indices and BF16 weights [tokens, top_k]");
  require_cuda(i);
  const at::Tensor indices = i.is_contiguous() ? i : i.contiguous();
  require(indices.numel() <= b.v[kCapacity], "more routes than the module's buffers hold");
  const c10::cuda::CUDAGuard guard(r.x.device());
  const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(r.x.device().index()).stream();
  const std::lock_guard<std::mutex> one_call(*b.launching);
  const at::Tensor out = new_tensor(input.sizes(), at::kBFloat16, r.x.device());
  for (int t0 = 0; t0 < r.tokens; t0 += kMostTokens) {
    const int tokens = std::min(kMostTokens, r.tokens - t0);
    const size_t routes0 = (size_t)t0 * b.v[kTopK];
    const int64_t* here = (const int64_t*)indices.data_ptr() + routes0;
    check(ink_expert_plan(here, at_field<int64_t>(b, kSources), at_field<int64_t>(b, kPointers), at_field<int32_t>(b, kExperts), at_field<int32_t>(b, kCounts),
                          at_field<int32_t>(b, kRows), (int)b.v[kStart], (int)b.v[kLocal], (int)b.v[kStride], tokens * (int)b.v[kTopK], (int)b.v[kCapacity], stream));
    grouped(b, r, t0, tokens, here, (const char*)weights.data_ptr() + 2 * routes0, nullptr, nullptr, out.data_ptr(), 0, stream);
  }
  return out;
}
// (block, x, indices, weights) -> BF16 like x: the routed experts alone, plan and projections
PyObject* run_experts(PyObject* const* args) {
  const Block& b = block_at(args);
  if (!b.current()) Py_RETURN_NOTIMPLEMENTED;
  const at::Tensor &input = tensor_at(args, 1), &indices = tensor_at(args, 2), &weights = tensor_at(args, 3);
  at::Tensor out;
  {
    const WithoutGil unlocked;
    out = experts_forward(b, input, indices, weights);
  }
  return THPVariable_Wrap(out);
}

template <PyObject* (*F)(PyObject* const*), Py_ssize_t N>
PyObject* entry(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != N) {
    PyErr_Format(PyExc_TypeError, "expected %zd arguments, got %zd", N, n);
    return nullptr;
  }
  try {
    return F(args);
  } catch (const Failure& f) {
    if (f.type) PyErr_SetString(f.type, f.what.c_str());
  } catch (...) {
    torch::translate_exception_to_python(std::current_exception());
  }
  return nullptr;
}

PyMethodDef kMethods[] = {
    {"decode_attention", (PyCFunction)(void*)&entry<decode_attention, 14>, METH_FASTCALL, nullptr},
    {"make_block", (PyCFunction)(void*)&entry<make_block, 1>, METH_FASTCALL, nullptr},
    {"run_block", (PyCFunction)(void*)&entry<run_block, 3>, METH_FASTCALL, nullptr},
    {"run_experts", (PyCFunction)(void*)&entry<run_experts, 4>, METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "inkling_b200_host", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_inkling_b200_host() { return PyModule_Create(&kModule); }
