// The host path of the package in native code: what a forward pass does between two kernel launches.
//
// The kernels of one Pairformer block at N = 128 take some 200 us; launched one by one from Python, with the checks, the
// weight look-ups and a foreign-function call for each, a block cost the host 700 us and a LayerNorm of the single
// representation 18 us for a 3 us kernel.  Here a module keeps a `Params` object: the places of its parameters (the
// module's own `_parameters` dictionaries), what was seen there last, and the forms the kernels want (fp32 vectors,
// 16-bit matrices, the split planes of the single branch), renewed when a parameter, its storage, its version or a
// submodule has changed (what is written past the version counter has to be announced: weights.py).  A call checks its
// tensors, looks the parameters over (some tens of pointer comparisons) and issues the launches through the C ABI of
// px_b200.h, whose functions are taken from the library handle that the Python side has loaded.  Workspaces come from the
// caching allocator on each call.
#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/CUDAEvent.h>
#include <ATen/ops/dropout.h>
#include <ATen/ops/empty.h>
#include <ATen/ops/empty_like.h>
#include <ATen/ops/full.h>
#include <ATen/ops/mm.h>
#include <ATen/ops/ones.h>
#include <c10/cuda/CUDAException.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <c10/util/SmallVector.h>
#include <dlfcn.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/pybind.h>

#include <algorithm>
#include <atomic>
#include <mutex>
#include <stdexcept>
#include <string>
#include <tuple>
#include <vector>

#include "../../include/px_b200.h"

namespace py = pybind11;
using at::Tensor;
typedef c10::optional<Tensor> OptTensor;

namespace {

constexpr int64_t kCz = 128, kCs = 384, kHeadsSingle = 16, kHeads = 4, kHeadDim = 32;

[[noreturn]] void fail(const std::string& what) { throw std::runtime_error(what); }

// ---- the C ABI, by the handle of the loaded library ------------------------------------------------------------------
#define PX_FUNCTIONS(X)                                                                                                  \
  X(px_status_string) X(px_ld) X(px_ld_mask) X(px_layer_norm_fwd_params) X(px_layer_norm_bwd_params)                     \
  X(px_scale_add_rowwise) X(px_standardise_rows) X(px_trimul_in_folded_bytes) X(px_trimul_in_fold)                       \
  X(px_trimul_in_proj_folded) X(px_trimul_contract) X(px_trimul_out_folded_bytes) X(px_trimul_out_fold)                  \
  X(px_trimul_out_folded) X(px_trimul_workspace_bytes) X(px_triatt_in_folded_bytes) X(px_triatt_in_fold)                 \
  X(px_triatt_in_proj_folded) X(px_triatt_flash) X(px_triatt_out_folded_bytes)                                           \
  X(px_triatt_out_fold) X(px_triatt_out_folded) X(px_triatt_workspace_bytes) X(px_transition)                            \
  X(px_pair_bias_folded_bytes) X(px_pair_bias_fold) X(px_pair_bias_proj_folded) X(px_single_weights_bytes)               \
  X(px_single_workspace_bytes) X(px_single_prepare) X(px_single_project) X(px_single_finish) X(px_opm_outer)             \
  X(px_opm_out) X(px_msa_opm_prep) X(px_msa_values) X(px_msa_weights) X(px_msa_average) X(px_msa_gate_out)               \
  X(px_msa_rows_weights_bytes) X(px_msa_rows_prepare) X(px_msa_transition_weights_bytes) X(px_msa_transition_prepare) X(px_msa_transition)
struct Abi {
#define X(f) decltype(&::f) f = nullptr;
  PX_FUNCTIONS(X)
#undef X
} abi;

void bind_library(uintptr_t handle) {
#define X(f)                                                                   \
  abi.f = reinterpret_cast<decltype(abi.f)>(dlsym((void*)handle, #f));         \
  if (!abi.f) fail(std::string("the kernel library lacks ") + #f);
  PX_FUNCTIONS(X)
#undef X
}

// ---- launches: counted, and timed with event pairs while a timer is on -----------------------------------------------
std::atomic<int64_t> g_launches{0};
std::atomic<bool> g_timing{false};
std::mutex g_timer_mutex;
struct Timed {
  const char* name;
  at::cuda::CUDAEvent start{cudaEventDefault}, stop{cudaEventDefault};
};
std::vector<Timed> g_timed;

template <typename F>
void launch(const char* name, cudaStream_t st, F f) {
  int32_t status;
  if (g_timing.load(std::memory_order_relaxed)) {
    Timed t;
    t.name = name;
    const auto stream = c10::cuda::getStreamFromExternal(st, c10::cuda::current_device());
    t.start.record(stream);
    status = f();
    t.stop.record(stream);
    std::lock_guard<std::mutex> lock(g_timer_mutex);
    g_timed.push_back(std::move(t));
  } else {
    status = f();
  }
  ++g_launches;
  if (status != PX_OK)
    fail(std::string(name) + " failed: " + abi.px_status_string(status) + " (status " + std::to_string(status) + ")");
}

std::vector<std::pair<std::string, double>> timer_collect() {
  std::lock_guard<std::mutex> lock(g_timer_mutex);
  std::vector<std::pair<std::string, double>> out;
  for (auto& t : g_timed) {
    t.stop.synchronize();
    out.emplace_back(t.name, (double)t.start.elapsed_time(t.stop));
  }
  g_timed.clear();
  return out;
}

// ---- tensors ----------------------------------------------------------------------------------------------------------
void need_cuda(const Tensor& t, const char* name) {
  if (!t.is_cuda()) fail(std::string(name) + " must be a CUDA tensor: this package has no CPU path");
}
// The kernels of a call run on one device, and an address of another one may not be mapped there.
void need_on(const Tensor& t, const at::Device& dev, const char* name) {
  need_cuda(t, name);
  if (t.device() != dev) fail(std::string(name) + " must be on the device of the other tensors");
}
int dtype_code(const Tensor& t, const char* name) {
  switch (t.scalar_type()) {
    case at::kFloat: return PX_F32;
    case at::kBFloat16: return PX_BF16;
    case at::kHalf: return PX_F16;
    default: fail(std::string(name) + " must be float32, bfloat16 or float16");
  }
}
Tensor bytes_like(const Tensor& t, int64_t n) { return at::empty({n}, t.options().dtype(at::kByte)); }

// [N, N, 128] or [1, N, N, 128] -> contiguous [N, N, 128]; batch says whether there was a leading 1.
Tensor pair_tensor(const Tensor& z, bool& batch) {
  if (!z.is_cuda()) fail("pair tensor must live on a CUDA device: this package has no CPU path");
  batch = z.dim() == 4;
  if (batch && z.size(0) != 1) fail("leading batch dimensions other than 1 are not supported");
  const Tensor t = batch ? z.select(0, 0) : z;
  if (t.dim() != 3) fail("expected [N, N, C] or [1, N, N, C]");
  if (t.size(0) != t.size(1) || t.size(2) != kCz) fail("pair tensor must have shape [N, N, 128]");
  if (t.scalar_type() != at::kFloat && t.scalar_type() != at::kBFloat16) fail("pair tensor must be float32 or bfloat16");
  return t.contiguous();
}
Tensor pair_mask(const OptTensor& mask, const Tensor& z) {
  if (!mask.has_value() || !mask->defined()) return Tensor();
  Tensor m = mask->dim() == 3 ? mask->select(0, 0) : *mask;
  if (m.device() != z.device() || m.scalar_type() != at::kFloat) m = m.to(z.device(), at::kFloat);
  if (m.dim() != 2 || m.size(0) != z.size(0) || m.size(1) != z.size(0)) fail("mask must be [N, N]");
  return m.contiguous();
}
const float* fptr(const Tensor& t) { return t.defined() ? (const float*)t.data_ptr() : nullptr; }

// ---- parameters of a module -----------------------------------------------------------------------------------------
// What a parameter becomes: 'f' an fp32 vector, 'z' a matrix in the format of the pair tensor's rows (bf16 rows: bf16, fp32
// rows: fp16), 'h' an fp16 matrix, 's' an fp32 matrix.  What the group becomes then: kMul, kAtt and kBias the folded weights
// of their row kernels (in, out), kSingle and kMsa the laid-out matrices of the single branch and of the MSA stack behind what comes before them, kOpm the
// outer product's two projections laid out as one,
// kPlain nothing more.
enum Group { kPlain, kMul, kAtt, kBias, kSingle, kMsa, kOpm };
struct Prepared {
  std::vector<Tensor> t[2];          // by format of z: 0 fp32, 1 bf16; complete, and no aliases of the parameters
  std::vector<const void*> p[2];
  std::vector<float> scalars;
  at::Device dev = at::kCPU;         // where the parameters are
  bool have[2] = {false, false};
  std::vector<cudaStream_t> streams[2];   // that calls have used it on: its memory is not given out again before they are through
};
typedef std::shared_ptr<const Prepared> Ready;

// Where a call runs: the device, its current stream, and the graph that this stream is being captured into, if any.
struct Use {
  at::Device dev;
  c10::cuda::CUDAStream stream;
  cudaGraph_t graph = nullptr;
  explicit Use(const at::Device& d) : dev(d), stream(at::cuda::getCurrentCUDAStream(d.index())) {
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    cudaGraph_t g = nullptr;
    if (cudaStreamGetCaptureInfo(stream, &status, nullptr, &g, nullptr, nullptr) != cudaSuccess) {
      cudaGetLastError();            // the legacy stream beside somebody else's capture: not being captured itself
      return;
    }
    if (status == cudaStreamCaptureStatusActive) graph = g;
  }
};

// A graph launches the kernels of its capture with the addresses of that time, however often the weights have been laid out
// anew since: it holds the set it was captured with until it is destroyed.  The graph lets go of it on a thread of the driver that may
// not call CUDA, so the set waits in a list and is freed by the next call that looks up weights (the list outlives the process'
// other objects: it is never destroyed).
class GraphHeld {
 public:
  static void keep(cudaGraph_t graph, const Ready& set) {
    Ready* const box = new Ready(set);
    cudaUserObject_t object;
    if (cudaUserObjectCreate(&object, box, &GraphHeld::let_go, 1, cudaUserObjectNoDestructorSync) != cudaSuccess) {
      cudaGetLastError();
      delete box;
      fail("the graph cannot hold the weights of its capture");
    }
    if (cudaGraphRetainUserObject(graph, object, 1, cudaGraphUserObjectMove) != cudaSuccess) {
      cudaGetLastError();
      cudaUserObjectRelease(object, 1);
      fail("the graph cannot hold the weights of its capture");
    }
  }
  static void free_released() {
    if (!any_.load(std::memory_order_acquire)) return;
    std::vector<Ready*> now;
    {
      std::lock_guard<std::mutex> lock(mutex_);
      now.swap(list());
      any_ = false;
    }
    for (Ready* r : now) delete r;
  }

 private:
  static void CUDART_CB let_go(void* box) {
    std::lock_guard<std::mutex> lock(mutex_);
    list().push_back((Ready*)box);
    any_.store(true, std::memory_order_release);
  }
  static std::vector<Ready*>& list() {
    static auto* const l = new std::vector<Ready*>;
    return *l;
  }
  static std::mutex mutex_;
  static std::atomic<bool> any_;
};
std::mutex GraphHeld::mutex_;
std::atomic<bool> GraphHeld::any_{false};

class Params {
 public:
  // root: the module this is kept for; checks: (dict, name) of submodules; params: (dict, name, kind, shape, module);
  // scalars: (module, name).  Modules and their __dict__ are held weakly or not at all: they hold this, and the garbage collector
  // does not see through it.
  Params(const std::string& group, const py::object& root, const py::list& checks, const py::list& params, const py::list& scalars)
      : root_(py::weakref(root)) {
    const char* names[] = {"plain", "mul", "att", "bias", "single", "msa", "opm"};
    int g = 0;
    while (g < 7 && group != names[g]) ++g;
    if (g == 7) fail("unknown parameter group " + group);
    group_ = (Group)g;
    for (const auto& c : checks) {
      const auto t = c.cast<py::tuple>();
      checks_.push_back({t[0].cast<py::dict>(), t[1].cast<py::object>(), py::none(), py::none()});
    }
    for (const auto& c : params) {
      const auto t = c.cast<py::tuple>();
      params_.push_back({t[0].cast<py::dict>(), t[1].cast<py::object>(), py::none(), py::weakref(t[4])});
      kind_.push_back(t[2].cast<std::string>()[0]);
      shape_.push_back(t[3].cast<std::vector<int64_t>>());
    }
    for (const auto& c : scalars) {
      const auto t = c.cast<py::tuple>();
      scalars_.push_back({py::dict(), t[1].cast<py::object>(), py::none(), py::weakref(t[0])});
    }
    for (auto& s : checks_) s.seen = py::reinterpret_borrow<py::object>(find(s));
  }

  // False for another module than the one it was made for (a replica or a shallow copy of it, which took over its attributes), and
  // when a submodule has been replaced: the object has to be made again from the module.
  bool current(const py::handle& module) const {
    if (PyWeakref_GetObject(root_.ptr()) != module.ptr()) return false;
    for (const auto& s : checks_)
      if (find(s) != s.seen.ptr()) return false;
    return true;
  }

  // The kernels' forms of the parameters for z of format zf; needs the GIL.  What it returns is complete: the host has waited for
  // it, so every stream may use it.  Inside a capture nothing can be laid out, since the graph's replays alone would write it.
  Ready get(int zf, const Use& use) {
    GraphHeld::free_released();
    c10::SmallVector<py::object, 16> objects;      // held, since a computed one runs Python code, and other threads with it
    for (const auto& s : params_) objects.push_back(parameter(s));
    c10::SmallVector<float, 4> scalars;
    for (const auto& s : scalars_) scalars.push_back(py::getattr(PyWeakref_GetObject(s.owner.ptr()), s.key).cast<float>());
    bool same = prepared_ != nullptr && std::equal(scalars.begin(), scalars.end(), prepared_->scalars.begin());
    c10::SmallVector<Seen, 16> now(params_.size());
    for (size_t i = 0; i < params_.size(); ++i) {
      PyObject* const o = objects[i].ptr();
      if (o != Py_None) {
        if (!THPVariable_Check(o)) fail("a module parameter is not a tensor");
        const Tensor& t = THPVariable_Unpack(o);
        now[i] = {o, t.data_ptr(), t.storage().unsafeGetStorageImpl(), (uint32_t)t._version(), t.scalar_type()};
      }
      same = same && now[i] == seen_[i];
    }
    if (use.graph && !(same && prepared_->have[zf]))
      fail("the weights are new to this module, or have changed, and cannot be laid out inside a graph capture: call the module once "
           "with inputs of this type before capturing");
    if (!same) {                     // calls in flight hold the set they were given
      prepared_ = std::make_shared<Prepared>();
      prepared_->scalars.assign(scalars.begin(), scalars.end());
      seen_.assign(now.begin(), now.end());
      params_hold_.assign(objects.begin(), objects.end());
      storages_.clear();
      for (const Seen& n : now)
        if (n.object) storages_.push_back(THPVariable_Unpack(n.object).storage().getWeakStorageImpl());
    }
    if (!prepared_->have[zf]) make(*prepared_, zf, use);
    if (prepared_->dev != use.dev) fail("parameters and inputs must be on the same device");
    if (use.graph) GraphHeld::keep(use.graph, prepared_);
    else used_on(*prepared_, zf, use.stream);
    return prepared_;
  }

 private:
  struct Slot {
    py::dict dict;
    py::object key, seen, owner;     // owner: weak reference to the module
  };
  struct Seen {
    PyObject* object = nullptr;
    void* data = nullptr;
    const void* storage = nullptr;
    uint32_t version = 0;
    at::ScalarType type = at::kFloat;
    bool operator==(const Seen& o) const {
      return object == o.object && data == o.data && storage == o.storage && version == o.version && type == o.type;
    }
  };
  static PyObject* find(const Slot& s) {
    PyObject* o = PyDict_GetItem(s.dict.ptr(), s.key.ptr());
    return o ? o : Py_None;
  }
  // A parameter as the module's attribute gives it: registered (the usual case, looked up directly), or a plain attribute or a property
  // (flattened, replicated and parametrised modules).
  static py::object parameter(const Slot& s) {
    if (PyObject* o = PyDict_GetItemWithError(s.dict.ptr(), s.key.ptr())) return py::reinterpret_borrow<py::object>(o);
    if (PyErr_Occurred()) throw py::error_already_set();
    return py::getattr(PyWeakref_GetObject(s.owner.ptr()), s.key);
  }

  // The allocator knows the stream of make(); every other one is told to it once, and asked of when the set is freed.
  static void used_on(Prepared& p, int zf, const c10::cuda::CUDAStream& stream) {
    for (const cudaStream_t s : p.streams[zf])
      if (s == stream.stream()) return;
    for (const Tensor& t : p.t[zf])
      if (t.defined()) t.record_stream(stream.unwrap());
    p.streams[zf].push_back(stream.stream());
  }

  void make(Prepared& p, int zf, const Use& use) {
    at::NoGradGuard no_grad;
    const at::Device& dev = use.dev;
    std::vector<Tensor> t;
    for (size_t i = 0; i < params_.size(); ++i) {
      PyObject* o = params_hold_[i].ptr();
      Tensor v;
      if (o != Py_None) {
        v = THPVariable_Unpack(o).detach();
        need_cuda(v, "parameters");
        if (v.device() != dev) fail("parameters and inputs must be on the same device");
        if (!v.sizes().equals(shape_[i]) || !v.is_floating_point())
          fail("a parameter must be a floating-point tensor of the shape the kernels are built for");
        const auto want = kind_[i] == 'f' || kind_[i] == 's' ? at::kFloat
                          : kind_[i] == 'z' && zf == 1       ? at::kBFloat16
                                                             : at::kHalf;
        v = v.to(want).contiguous();
        if (((uintptr_t)v.data_ptr() & 15) != 0) v = v.clone();
      }
      t.push_back(v);
    }
    const cudaStream_t st = use.stream;
    const int rows = zf == 1 ? PX_BF16 : PX_F16;
    const auto byte = at::TensorOptions().device(dev).dtype(at::kByte);
    auto f = [&](int i) { return t[i].defined() ? (const float*)t[i].data_ptr() : nullptr; };
    auto w = [&](int i) { return (const px_w16*)t[i].data_ptr(); };
    auto msa_rows = [&](const Tensor& a, const Tensor& b) {          // b: the second half of the outputs
      const Tensor out = at::empty({abi.px_msa_rows_weights_bytes()}, byte);
      launch("px_msa_rows_prepare", st, [&] {
        return abi.px_msa_rows_prepare((const float*)a.data_ptr(), b.defined() ? (const float*)b.data_ptr() : nullptr, out.data_ptr(), st);
      });
      return out;
    };
    if (group_ == kMul) {
      const Tensor in = at::empty({abi.px_trimul_in_folded_bytes()}, byte), out = at::empty({abi.px_trimul_out_folded_bytes()}, byte);
      launch("px_trimul_in_fold", st, [&] {
        return abi.px_trimul_in_fold(f(0), f(1), w(4), w(5), w(6), w(7), rows, in.data_ptr(), st);
      });
      launch("px_trimul_out_fold", st, [&] {
        return abi.px_trimul_out_fold(f(0), f(1), f(2), f(3), w(8), w(9), rows, out.data_ptr(), st);
      });
      t = {in, out};
    } else if (group_ == kAtt) {
      const Tensor in = at::empty({abi.px_triatt_in_folded_bytes()}, byte), out = at::empty({abi.px_triatt_out_folded_bytes()}, byte);
      launch("px_triatt_in_fold", st, [&] {
        return abi.px_triatt_in_fold(f(0), f(1), w(3), w(4), w(5), w(2), rows, in.data_ptr(), st);
      });
      launch("px_triatt_out_fold", st, [&] { return abi.px_triatt_out_fold(f(0), f(1), w(6), w(7), rows, out.data_ptr(), st); });
      t = {in, out};
    } else if (group_ == kBias) {
      const Tensor out = at::empty({abi.px_pair_bias_folded_bytes()}, byte);
      launch("px_pair_bias_fold", st, [&] {
        return abi.px_pair_bias_fold(f(0), f(1), w(2), (int32_t)shape_[2][0], rows, out.data_ptr(), st);
      });
      t = {out};
    } else if (group_ == kSingle) {
      const Tensor out = at::empty({abi.px_single_weights_bytes()}, byte);
      launch("px_single_prepare", st, [&] {
        return abi.px_single_prepare(f(5), f(6), f(7), f(8), f(9), f(10), f(11), f(12), out.data_ptr(), st);
      });
      t.resize(5);
      t.push_back(out);
    } else if (group_ == kMsa) {
      const Tensor out = at::empty({abi.px_msa_transition_weights_bytes()}, byte);
      launch("px_msa_transition_prepare", st, [&] { return abi.px_msa_transition_prepare(f(7), f(8), f(9), out.data_ptr(), st); });
      t.resize(7);
      t.push_back(out);
      for (int i = 2; i < 5; ++i) t[i] = msa_rows(t[i], Tensor());
    } else if (group_ == kOpm) {
      t[2] = msa_rows(t[2], t[3]);
    }
    for (Tensor& v : t)              // a set of its own: what a graph reads outlives the parameters, and the whole set changes at once
      for (const auto& o : params_hold_)
        if (v.defined() && !o.is_none() && v.is_alias_of(THPVariable_Unpack(o.ptr()))) {
          v = v.clone();
          break;
        }
    p.t[zf] = t;
    p.p[zf].clear();
    for (const Tensor& v : t) p.p[zf].push_back(v.defined() ? v.data_ptr() : nullptr);
    // The row kernels fetch folded weights before the kernels in front of them are complete (programmatic launch), and other
    // streams use the set too: once per change of the weights, the host waits for it.
    C10_CUDA_CHECK(cudaStreamSynchronize(st));
    p.streams[zf] = {st};
    p.dev = dev;
    p.have[zf] = true;
  }

  Group group_;
  py::object root_;                          // weak reference
  std::vector<Slot> checks_, params_, scalars_;
  std::vector<char> kind_;
  std::vector<std::vector<int64_t>> shape_;
  std::vector<Seen> seen_;
  // The parameter objects seen last, and their storages, these without the memory: the addresses of neither can be reused, so that
  // another object or storage is told from them even where its memory lies where the old one's did.
  std::vector<py::object> params_hold_;
  std::vector<c10::weak_intrusive_ptr<c10::StorageImpl>> storages_;
  std::shared_ptr<Prepared> prepared_;
};

int64_t al(int64_t n) { return (n + 255) / 256 * 256; }
int zformat(const Tensor& z) { return z.scalar_type() == at::kBFloat16 ? 1 : 0; }

// ---- the pair updates ------------------------------------------------------------------------------------------------
struct PairCall {
  int64_t n;
  int zf, dt;                    // format index and dtype code of z
  const float* mask;
  unsigned char* ws;             // shared by the updates, which run one after the other
  cudaStream_t st;
};
// as laid out by tri_mul and tri_att, and behind that the standardised rows
int64_t pair_workspace(int64_t n) { return std::max(abi.px_trimul_workspace_bytes(n), abi.px_triatt_workspace_bytes(n)); }

// The standardised copy of the rows of z that the updates of an fp32 z read: where it lies, and whether it holds the current z,
// made with which eps.
struct Rows {
  px_f16* zn = nullptr;
  bool valid = false;
  float eps = 0.f;
  void need(const PairCall& c, const void* z, float want) {
    if (valid && eps == want) return;
    launch("px_standardise_rows", c.st, [&] { return abi.px_standardise_rows((const float*)z, zn, c.n * c.n, want, c.st); });
    valid = true, eps = want;
  }
};

void tri_mul(const PairCall& c, const Prepared& pr, const void* z_in, void* z_out, bool incoming, bool add, Rows& rows) {
  const auto& p = pr.p[c.zf];
  const float eps = pr.scalars[0];
  const int64_t n = c.n, ld = abi.px_ld(n), per = kCz * n * ld * 2;
  px_f16 *a = (px_f16*)c.ws, *b = (px_f16*)(c.ws + per), *x = (px_f16*)(c.ws + 2 * per);
  const bool fp32 = c.dt == PX_F32;      // the projection and the output stage normalise the same z: one standardised copy
  if (fp32) rows.need(c, z_in, eps);
  launch("px_trimul_in_proj", c.st, [&] {
    return abi.px_trimul_in_proj_folded(fp32 ? rows.zn : z_in, fp32 ? PX_F16 : c.dt, c.mask, p[0], a, b, n, n, ld, incoming, eps, c.st);
  });
  launch("px_trimul_contract", c.st, [&] { return abi.px_trimul_contract(a, b, x, kCz, n, ld, c.st); });
  rows.valid = false;
  launch("px_trimul_out", c.st, [&] {
    return abi.px_trimul_out_folded(x, z_in, rows.zn, z_out, c.dt, p[1], n, n, ld, add, eps, c.st);
  });
}

// before_core(): called when everything in front of the attention core has been launched.
template <typename F>
void tri_att(const PairCall& c, const Prepared& pr, const void* z_in, void* z_out, bool ending, bool add, Rows& rows, F before_core) {
  const auto& p = pr.p[c.zf];
  const float eps = pr.scalars[0], inf = pr.scalars[1];
  const int64_t n = c.n, ldm = abi.px_ld_mask(n);
  const int64_t qkv = al(n * kHeads * abi.px_ld(n) * kHeadDim * 2);   // v is [n][4][32][ld(n)], q and k fit as well
  px_f16 *q = (px_f16*)c.ws, *k = (px_f16*)(c.ws + qkv), *v = (px_f16*)(c.ws + 2 * qkv), *o = (px_f16*)(c.ws + 3 * qkv);
  unsigned char* bias = (unsigned char*)o + al(n * n * kCz * 2);
  unsigned char* mbias = bias + al(kHeads * n * ldm * 4);
  const bool fp32 = c.dt == PX_F32;
  if (fp32) rows.need(c, z_in, eps);
  launch("px_triatt_in_proj", c.st, [&] {
    return abi.px_triatt_in_proj_folded(fp32 ? rows.zn : z_in, fp32 ? PX_F16 : c.dt, c.mask, p[0], q, k, v, (float*)bias, (float*)mbias, n,
                                        n, ldm, ending, eps, inf, c.st);
  });
  before_core();
  launch("px_triatt_flash", c.st, [&] {
    return abi.px_triatt_flash(q, k, v, (const float*)bias, (const float*)mbias, o, n, n, ldm, c.st);
  });
  rows.valid = false;
  launch("px_triatt_out", c.st, [&] {
    return abi.px_triatt_out_folded(o, z_in, rows.zn, z_out, c.dt, p[1], n, n, ending, add, eps, c.st);
  });
}

void transition_rows(cudaStream_t st, const Prepared& pr, int zf, int dt, const void* x_in, void* x_out, int64_t rows, bool add) {
  const auto& p = pr.p[zf];
  launch("px_transition", st, [&] {
    return abi.px_transition(x_in, x_out, dt, (const float*)p[0], (const float*)p[1], (const px_f16*)p[2], (const px_f16*)p[3],
                             (const px_f16*)p[4], rows, add, pr.scalars[0], st);
  });
}

// The standardised rows at the end of a workspace of the size that the library asks for.
Rows own_rows(const PairCall& c, const Tensor& ws) {
  Rows r;
  if (c.dt == PX_F32) r.zn = (px_f16*)(c.ws + ws.numel() - al(c.n * c.n * kCz * 2));
  return r;
}

Tensor tri_mul_forward(Params& params, const Tensor& z, const OptTensor& mask, bool incoming, bool inplace_add) {
  bool batch;
  const Tensor zc = pair_tensor(z, batch);
  c10::cuda::CUDAGuard guard(zc.device());
  at::NoGradGuard no_grad;
  const Tensor m = pair_mask(mask, zc);
  const Ready pr = params.get(zformat(zc), Use(zc.device()));
  py::gil_scoped_release release;
  const Tensor out = inplace_add && zc.data_ptr() == z.data_ptr() ? zc : at::empty_like(zc);
  const Tensor ws = bytes_like(zc, abi.px_trimul_workspace_bytes(zc.size(0)));
  const PairCall c{zc.size(0), zformat(zc), dtype_code(zc, "z"), fptr(m), (unsigned char*)ws.data_ptr(), at::cuda::getCurrentCUDAStream()};
  Rows rows = own_rows(c, ws);
  tri_mul(c, *pr, zc.data_ptr(), out.data_ptr(), incoming, inplace_add, rows);
  return batch ? out.unsqueeze(0) : out;
}

Tensor tri_att_forward(Params& params, const Tensor& z, const OptTensor& mask, bool ending, bool inplace_add) {
  bool batch;
  const Tensor zc = pair_tensor(z, batch);
  c10::cuda::CUDAGuard guard(zc.device());
  at::NoGradGuard no_grad;
  const Tensor m = pair_mask(mask, zc);
  const Ready pr = params.get(zformat(zc), Use(zc.device()));
  py::gil_scoped_release release;
  const Tensor out = inplace_add && zc.data_ptr() == z.data_ptr() ? zc : at::empty_like(zc);
  const Tensor ws = bytes_like(zc, abi.px_triatt_workspace_bytes(zc.size(0)));
  const PairCall c{zc.size(0), zformat(zc), dtype_code(zc, "z"), fptr(m), (unsigned char*)ws.data_ptr(), at::cuda::getCurrentCUDAStream()};
  Rows rows = own_rows(c, ws);
  tri_att(c, *pr, zc.data_ptr(), out.data_ptr(), ending, inplace_add, rows, [] {});
  return batch ? out.unsqueeze(0) : out;
}

Tensor transition_forward(Params& params, const Tensor& x, bool inplace_add) {
  need_cuda(x, "x");
  if (x.dim() < 1 || x.size(-1) != kCz) fail("transition kernel handles [..., 128] rows");
  c10::cuda::CUDAGuard guard(x.device());
  at::NoGradGuard no_grad;
  const Tensor xc = x.contiguous();
  const Ready pr = params.get(zformat(xc), Use(xc.device()));
  py::gil_scoped_release release;
  const Tensor out = inplace_add && xc.data_ptr() == x.data_ptr() ? xc : at::empty_like(xc);
  transition_rows(at::cuda::getCurrentCUDAStream(), *pr, zformat(xc), dtype_code(xc, "x"), xc.data_ptr(), out.data_ptr(),
                  xc.numel() / kCz, inplace_add);
  return out;
}

// ---- blocks ----------------------------------------------------------------------------------------------------------
struct Block {
  std::shared_ptr<Params> mul_out, mul_in, att_start, att_end, transition, pair_bias, single;   // the last two: s branch
  bool current(const py::handle& module) const {
    for (const auto& p : {mul_out, mul_in, att_start, att_end, transition, pair_bias, single})
      if (p && !p->current(module)) return false;
    return true;
  }
};
struct BlockReady {
  Ready mul_out, mul_in, att_start, att_end, transition, pair_bias, single;
};

// The single branch: what needs s alone, then s_in -> s_out given the block's pair bias.
void single_project(cudaStream_t st, const Prepared& pr, int zf, const Tensor& s, const Tensor& ws) {
  const auto& p = pr.p[zf];
  launch("px_single_update", st, [&] {
    return abi.px_single_project(s.data_ptr(), dtype_code(s, "s"), p.back(), (const float*)p[0], (const float*)p[1], (const float*)p[2],
                                 ws.data_ptr(), ws.numel(), s.numel() / kCs, pr.scalars[0], st);
  });
}
void single_finish(cudaStream_t st, const Prepared& pr, int zf, const Tensor& s_in, const Tensor& s_out, const Tensor& bias,
                   const Tensor& ws) {
  const auto& p = pr.p[zf];
  launch("px_single_update", st, [&] {
    return abi.px_single_finish(s_in.data_ptr(), s_out.data_ptr(), dtype_code(s_in, "s"), p.back(), (const float*)p[3],
                                (const float*)p[4], (const float*)bias.data_ptr(), ws.data_ptr(), ws.numel(), s_in.numel() / kCs,
                                pr.scalars[1], st);
  });
}

// One side stream per device for plain calls and one for captures: work of another thread's plain call must not meet a stream that is
// being captured.
c10::cuda::CUDAStream side_stream(const Use& use) {
  static std::mutex mutex;
  static std::vector<c10::optional<c10::cuda::CUDAStream>> streams;
  const size_t i = 2 * (size_t)use.dev.index() + (use.graph ? 1 : 0);
  std::lock_guard<std::mutex> lock(mutex);
  if (i >= streams.size()) streams.resize(i + 1);
  if (!streams[i]) streams[i] = c10::cuda::getStreamFromPool(false, use.dev.index());
  return *streams[i];
}

// The blocks one after the other.  The pair path never reads s, and the single branch takes nothing from z but the pair
// bias of the block's final z: the branch of a block runs on a side stream beside the pair path of the next block, which writes another
// pair-bias buffer.  It is let go when the next block comes to its first attention core.  Beside row kernels, whose tiles are dealt out in
// advance, each of its kernels holds up the tile of some SM, and with it the whole kernel.  So it does beside the core, whose units are dealt
// out in advance as well from 129 to 1024 tokens, but by a smaller part of its far longer time.  us per block, fp32 z, in order | beside from the
// block's start on | from its first attention core | from its second: N = 64 155 | 115 | 112 | 113, 128 182 | 151 | 145 | 148, 150 234 | 202 | 195 |
// 198, 200 292 | 260 | 254 | 260, 256 353 | 323 | 324 | 324, 300 510 | 482 | 479 | 477, 384 743 | 693 | 695 | 695, 437 1059 | 1023 | 1010 | 1005,
// 512 1352 | 1332 | 1305 | 1312, 640 2251 | 2240 | 2210 | 2226, 768 3405 | 3397 | 3367 | 3358, 1024 6783 | 6838 | 6747 | 6697, 1280 level;
// bf16 200 274 | 242 | 238 | 243, 384 648 | 609 | 600 | 609, 768 3017 | 3008 | 2939 | 2988 (from 384 tokens on the runs of one side differ by 1
// to 3 %).  Its transition only beside the second core, while the core had a CTA for each unit: 145 at N = 128, 276 against 278 at 200, 720
// against 719 at 384.
// One block alone: its projections of s, which need no bias, beside its own pair path (224 | 216 at N = 128, no difference from 200 on).
// Everything is allocated on the caller's stream, which waits for the side stream before this returns.
// Where the main stream waits for the side stream before it writes a pair-bias buffer anew, the launch behind does not overlap the kernel
// before.  Up to kManyBiasUpTo tokens there are eight buffers (together as large as an fp32 z) and one such wait in four blocks.  Two buffers |
// eight, us per block: N = 24 105.3 | 103.9, 64 110.5 | 109.3, 128 146.3 | 144.8, 200 256.9 | 255.6, 300 478.5 | 474.4, 384 691.0 | 690.9, 437
// 1002 | 1017, 512 1312 | 1310, 640 2197 | 2202; bf16 200 235.5 | 234.3, 384 598.6 | 596.1.
constexpr int64_t kBesideBelow = 1281, kProjectFirstUpTo = 256, kManyBiasUpTo = 384;
std::tuple<OptTensor, Tensor> stack_forward(const std::vector<std::shared_ptr<Block>>& blocks, const OptTensor& s_in,
                                            const Tensor& z, const OptTensor& mask, bool inplace) {
  bool batch;
  const Tensor zi = pair_tensor(z, batch);
  c10::cuda::CUDAGuard guard(zi.device());
  at::NoGradGuard no_grad;
  const Tensor m = pair_mask(mask, zi);
  const int zf = zformat(zi);
  const int64_t n = zi.size(0);
  Tensor s = s_in.has_value() ? *s_in : Tensor();
  bool singles = false;
  const Use use(zi.device());
  std::vector<BlockReady> ready;
  for (const auto& b : blocks) {
    BlockReady r{b->mul_out->get(zf, use), b->mul_in->get(zf, use), b->att_start->get(zf, use), b->att_end->get(zf, use),
                 b->transition->get(zf, use), nullptr, nullptr};
    if (b->single && s.defined()) {
      r.pair_bias = b->pair_bias->get(zf, use), r.single = b->single->get(zf, use);
      singles = true;
    }
    ready.push_back(r);
  }
  if (singles) {
    need_on(s, zi.device(), "s");
    if (s.dim() < 2 || s.size(-1) != kCs || s.size(-2) != n || s.numel() != n * kCs) fail("s must be [N, 384]");
    dtype_code(s, "s");
    s = s.contiguous();
  }
  py::gil_scoped_release release;
  // z is copied only if there is no block to write it anew: the first update reads z and writes the result's tensor
  const bool own = inplace || zi.data_ptr() != z.data_ptr();
  const Tensor zc = own ? zi : blocks.empty() ? zi.clone() : at::empty_like(zi);
  const Tensor ws = bytes_like(zc, pair_workspace(n));
  const auto main = at::cuda::getCurrentCUDAStream();
  const PairCall c{n, zf, dtype_code(zc, "z"), fptr(m), (unsigned char*)ws.data_ptr(), main};
  const bool fp32 = c.dt == PX_F32;
  Rows rows = own_rows(c, ws);
  const bool first = n <= kProjectFirstUpTo;       // projections of s beside the pair path of the first block from its start on
  const bool aside = singles && (blocks.size() > 1 ? n < kBesideBelow : first);
  const auto side = aside ? side_stream(use) : main;
  // update k of s has bias buffer k % (2 * per_wait); the main stream waits before every per_wait-th for those of the round before
  const int64_t per_wait = n <= kManyBiasUpTo ? 4 : 1;
  std::vector<Tensor> bias;
  Tensor sb[2], sws;
  at::cuda::CUDAEvent gate, side_done[2];
  int64_t waiting = -1;             // block whose bias is made and whose update, number k - 1, is still to be issued
  if (singles) {
    for (int64_t i = 0; i < std::min<int64_t>(blocks.size(), 2 * per_wait); ++i)
      bias.push_back(at::empty({kHeadsSingle, n, n}, zc.options().dtype(at::kFloat)));
    for (int i = 0; i < (blocks.size() > 1 ? 2 : 1); ++i) sb[i] = at::empty_like(s);
    sws = bytes_like(zc, abi.px_single_workspace_bytes(n));
    if (aside) {
      side_done[0].record(main);
      side_done[0].block(side);
    }
  }
  struct Join {                     // the caller's stream goes on when the side stream is through, after an error too
    bool on;
    c10::cuda::CUDAStream side, main;
    ~Join() {
      if (!on) return;
      at::cuda::CUDAEvent e;
      e.record(side);
      e.block(main);
    }
  } join{aside, side, main};
  int64_t k = 0, last = -1;         // single updates so far; the last block that has one
  for (size_t b = 0; b < ready.size(); ++b)
    if (ready[b].single) last = b;
  for (size_t b = 0; b < ready.size(); ++b) {
    const BlockReady& r = ready[b];
    if (r.single && first && (b == 0 || !aside)) single_project(side, *r.single, zf, s, sws);
    void* const z = zc.data_ptr();
    tri_mul(c, *r.mul_out, b == 0 ? zi.data_ptr() : z, z, false, true, rows);
    tri_mul(c, *r.mul_in, z, z, true, true, rows);
    tri_att(c, *r.att_start, z, z, false, true, rows, [&] {
      if (!aside || (waiting < 0 && !r.single)) return;
      gate.record(main);
      gate.block(side);
      if (waiting >= 0) {
        const int64_t done = k - 1;
        single_finish(side, *ready[waiting].single, zf, s, sb[done & 1], bias[done % bias.size()], sws);
        if (k % per_wait == 0) side_done[(k / per_wait) & 1].record(side);      // updates up to k - 1
        s = sb[done & 1];
        waiting = -1;
      }
      if (r.single && !(first && b == 0)) single_project(side, *r.single, zf, s, sws);
    });
    tri_att(c, *r.att_end, z, z, true, true, rows, [] {});
    rows.valid = false;
    transition_rows(c.st, *r.transition, zf, c.dt, z, z, n * n, true);
    if (!r.single) continue;
    const Tensor& pair_bias = bias[k % bias.size()];
    // the copy for the pair bias also serves the next block's first update
    if (fp32) rows.need(c, z, r.pair_bias->scalars[0]);
    // the updates that read this and the next buffers last, up to number k - per_wait - 1, are through
    if (aside && k >= 2 * per_wait && k % per_wait == 0) side_done[(k / per_wait - 1) & 1].block(main);
    const auto& p = r.pair_bias->p[zf];
    launch("px_pair_bias_proj", c.st, [&] {
      return abi.px_pair_bias_proj_folded(fp32 ? rows.zn : z, fp32 ? PX_F16 : PX_BF16, p[0], (float*)pair_bias.data_ptr(), n * n, kHeadsSingle,
                                          r.pair_bias->scalars[0], c.st);
    });
    if (aside && (int64_t)b != last) {
      waiting = b;
      ++k;
      continue;
    }
    if (aside) {                                   // the last block's rest has nothing to run beside
      gate.record(side);
      gate.block(main);
    } else if (!first) {
      single_project(main, *r.single, zf, s, sws);
    }
    single_finish(main, *r.single, zf, s, sb[k & 1], pair_bias, sws);
    s = sb[k & 1];
    ++k;
  }
  return {s.defined() ? OptTensor(s) : OptTensor(), batch ? zc.unsqueeze(0) : zc};
}

// ---- MSA module ------------------------------------------------------------------------------------------------------
// z_out = [z_in +] OuterProductMean(m) for m [S, N, 64] fp32; x_bytes bounds the outer products formed at a time.
Tensor opm_forward(Params& params, const Tensor& m, const OptTensor& mask, const OptTensor& z_in, const Tensor& z_out, int64_t x_bytes) {
  need_cuda(m, "m");
  c10::cuda::CUDAGuard guard(m.device());
  at::NoGradGuard no_grad;
  const int64_t s_rows = m.size(0), n = m.size(1), ld = (s_rows + 7) / 8 * 8;
  if (m.dim() != 3 || m.size(2) != 64 || m.scalar_type() != at::kFloat || !m.is_contiguous()) fail("m must be a contiguous float32 [S, N, 64] tensor");
  if (n > 32768 || n < 1 || s_rows < 1) fail("outer_product_mean supports 1 <= N <= 32768 tokens");
  const bool residual = z_in.has_value() && z_in->defined();
  for (const Tensor& z : {z_out, residual ? *z_in : z_out}) {
    need_on(z, m.device(), "z");
    if (z.dim() != 3 || z.size(0) != n || z.size(1) != n || z.size(2) != kCz || !z.is_contiguous() || z.scalar_type() != z_out.scalar_type())
      fail("z must be contiguous [N, N, 128] with N = m.shape[1]");
  }
  Tensor mk;
  if (mask.has_value() && mask->defined()) {
    need_on(*mask, m.device(), "msa_mask");
    if (mask->dim() != 2 || mask->size(0) != s_rows || mask->size(1) != n) fail("msa_mask must be [N_seq, N_res]");
    mk = mask->to(at::kFloat).contiguous();
  }
  const Ready pr = params.get(0, Use(m.device()));
  py::gil_scoped_release release;
  const auto& p = pr->p[0];
  const float eps = pr->scalars[0], ln_eps = pr->scalars[1];
  const auto opt = m.options();
  const Tensor ab = at::empty({2, n * 32, ld}, opt.dtype(at::kHalf));
  px_f16 *a = (px_f16*)ab.data_ptr(), *b = a + n * 32 * ld;
  const Tensor inv = mk.defined() ? at::mm(mk.t(), mk).add_(eps).reciprocal_() : at::full({n, n}, 1.0f / ((float)s_rows + eps), opt);
  const int64_t n_blk = std::max<int64_t>(1, std::min(n, x_bytes / (2048 * n)));   // rows i of x = [32 n_i][32 N] fp16
  const Tensor x = at::empty({n_blk * 32, n * 32}, opt.dtype(at::kHalf));
  const cudaStream_t st = at::cuda::getCurrentCUDAStream();
  launch("px_msa_opm_prep", st, [&] {
    return abi.px_msa_opm_prep((const float*)m.data_ptr(), fptr(mk), (const float*)p[0], (const float*)p[1], p[2], a, b, s_rows, n, ld, ln_eps, st);
  });
  const int64_t row = z_out.element_size() * n * kCz;
  for (int64_t i0 = 0; i0 < n; i0 += n_blk) {
    const int64_t ni = std::min(n_blk, n - i0);
    launch("px_opm_outer", st, [&] { return abi.px_opm_outer(a + i0 * 32 * ld, b, (px_f16*)x.data_ptr(), ni * 32, n * 32, ld, st); });
    launch("px_opm_out", st, [&] {
      return abi.px_opm_out((const px_f16*)x.data_ptr(), (const px_f16*)p[4], (const float*)p[5], (const float*)inv.data_ptr() + i0 * n,
                            residual ? (const char*)z_in->data_ptr() + i0 * row : nullptr, (char*)z_out.data_ptr() + i0 * row,
                            dtype_code(z_out, "z"), ni, n, residual, st);
    });
  }
  return z_out;
}

// m += PairWeightedAveraging(m, z), m += Transition(m) in place over chunks of sequences: m [S, N, 64] fp32, 8 heads x 8.
void msa_stack_forward(Params& params, Params& bias_params, const Tensor& m, const Tensor& z_, int64_t chunk) {
  need_cuda(m, "m");
  bool batch;
  const Tensor z = pair_tensor(z_, batch);
  need_on(z, m.device(), "z");
  c10::cuda::CUDAGuard guard(m.device());
  at::NoGradGuard no_grad;
  const int64_t s_all = m.size(0), n = m.size(1), heads = 8;
  if (m.dim() != 3 || m.size(2) != 64 || n != z.size(0) || m.scalar_type() != at::kFloat || !m.is_contiguous())
    fail("m must be a contiguous float32 [S, N, 64] tensor with z [N, N, 128]");
  const int zf = zformat(z);
  const Use use(m.device());
  const Ready pr = params.get(0, use), br = bias_params.get(zf, use);
  py::gil_scoped_release release;
  const auto& p = pr->p[0];
  const cudaStream_t st = at::cuda::getCurrentCUDAStream();
  const auto opt = m.options();
  const int64_t ld = (n + 7) / 8 * 8;
  const Tensor logits = at::empty({heads, n, n}, opt), w = at::empty({heads, 3, n, ld}, opt.dtype(at::kBFloat16));
  Tensor zn;
  const void* rows = z.data_ptr();
  if (zf == 0) {
    zn = at::empty(z.sizes(), opt.dtype(at::kHalf));
    launch("px_standardise_rows", st, [&] {
      return abi.px_standardise_rows((const float*)z.data_ptr(), (px_f16*)zn.data_ptr(), n * n, br->scalars[0], st);
    });
    rows = zn.data_ptr();
  }
  launch("px_pair_bias_proj", st, [&] {
    return abi.px_pair_bias_proj_folded(rows, zf ? PX_BF16 : PX_F16, br->p[zf][0], (float*)logits.data_ptr(), n * n, (int32_t)heads, br->scalars[0], st);
  });
  launch("px_msa_weights", st, [&] { return abi.px_msa_weights((const float*)logits.data_ptr(), (px_bf16*)w.data_ptr(), n, ld, st); });
  auto f = [&](int i) { return (const float*)p[i]; };
  for (int64_t s0 = 0; s0 < s_all; s0 += chunk) {
    const int64_t s = std::min(chunk, s_all - s0);
    float* part = (float*)m.data_ptr() + s0 * n * 64;
    const Tensor v = at::empty({heads, 3, n, s * 8}, opt.dtype(at::kBFloat16)), wv = at::empty({heads, n, s * 8}, opt);
    launch("px_msa_values", st, [&] { return abi.px_msa_values(part, f(0), f(1), p[2], (px_bf16*)v.data_ptr(), s, n, pr->scalars[0], st); });
    launch("px_msa_average", st, [&] {
      return abi.px_msa_average((const px_bf16*)w.data_ptr(), (const px_bf16*)v.data_ptr(), (float*)wv.data_ptr(), s, n, ld, st);
    });
    launch("px_msa_gate_out", st, [&] {
      return abi.px_msa_gate_out(part, (const float*)wv.data_ptr(), f(0), f(1), p[3], p[4], s, n, pr->scalars[0], st);
    });
    launch("px_msa_transition", st, [&] { return abi.px_msa_transition(part, p[7], f(5), f(6), s * n, pr->scalars[1], st); });
  }
}

// ---- LayerNorm -------------------------------------------------------------------------------------------------------
struct LnParams {
  Tensor w, b;     // as the kernels take them: of the type of x, or fp32 (rounded to the type of x inside)
  int code;        // dtype code of both
};
bool has(const OptTensor& t) { return t.has_value() && t->defined(); }
LnParams ln_params(const Tensor& x, const OptTensor& weight, const OptTensor& bias) {
  LnParams r;
  const bool fp32 = (!has(weight) || weight->scalar_type() == at::kFloat) && (!has(bias) || bias->scalar_type() == at::kFloat);
  const auto type = fp32 ? at::kFloat : x.scalar_type();
  auto fit = [&](const OptTensor& p, const char* name, Tensor& to) {
    if (!has(p)) return;
    need_on(*p, x.device(), name);
    if (p->numel() != x.size(-1)) fail(std::string(name) + " must have as many elements as the last axis");
    to = p->scalar_type() == type && p->is_contiguous() ? *p : p->detach().to(type).contiguous();
  };
  fit(weight, "weight", r.w);
  fit(bias, "bias", r.b);
  r.code = fp32 ? PX_F32 : dtype_code(x, "input");
  return r;
}
void ln_check(const Tensor& x, int64_t width) {
  need_cuda(x, "input");
  if (x.dim() < 1 || x.size(-1) != width) {
    std::string s;
    for (int64_t d : x.sizes()) s += (s.empty() ? "" : ", ") + std::to_string(d);
    fail("Expected input with last dimension " + std::to_string(width) + ", got (" + s + ")");
  }
  dtype_code(x, "input");
}
Tensor ln_forward(const Tensor& x, const LnParams& p, double eps, Tensor* mean, Tensor* invvar) {
  c10::cuda::CUDAGuard guard(x.device());
  const Tensor y = at::empty_like(x);
  const int64_t cols = x.size(-1), rows = cols ? x.numel() / cols : 0;
  if (mean) {
    *mean = at::empty({rows}, x.options().dtype(at::kFloat));
    *invvar = at::empty({rows}, x.options().dtype(at::kFloat));
  }
  const cudaStream_t st = at::cuda::getCurrentCUDAStream();
  launch("px_layer_norm_fwd", st, [&] {
    return abi.px_layer_norm_fwd_params(x.data_ptr(), p.w.defined() ? p.w.data_ptr() : nullptr, p.b.defined() ? p.b.data_ptr() : nullptr,
                                        y.data_ptr(), mean ? (float*)mean->data_ptr() : nullptr,
                                        mean ? (float*)invvar->data_ptr() : nullptr, rows, cols, (float)eps, dtype_code(x, "input"),
                                        p.code, st);
  });
  return y;
}

// y = LayerNorm(x); keeps x and the fp32 row statistics for the backward.
struct LayerNormFunction : torch::autograd::Function<LayerNormFunction> {
  static Tensor forward(torch::autograd::AutogradContext* ctx, const Tensor& x, const OptTensor& weight, const OptTensor& bias,
                        double eps) {
    const Tensor xc = x.contiguous();
    const LnParams p = ln_params(xc, weight, bias);
    Tensor mean, invvar;
    const Tensor y = ln_forward(xc, p, eps, &mean, &invvar);
    ctx->save_for_backward({xc, p.w, mean, invvar});
    const int64_t w_type = (int64_t)(has(weight) ? weight->scalar_type() : at::kFloat);
    const int64_t b_type = (int64_t)(has(bias) ? bias->scalar_type() : at::kFloat);
    // one entry: dtype code, types of the parameters, which gradients are wanted
    ctx->saved_data["f"] = (int64_t)p.code | w_type << 8 | b_type << 16 | (int64_t)(has(weight) && weight->requires_grad()) << 24 |
                           (int64_t)(has(bias) && bias->requires_grad()) << 25 | (int64_t)x.requires_grad() << 26;
    return y;
  }
  static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx, torch::autograd::variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &x = saved[0], &w = saved[1], &mean = saved[2], &invvar = saved[3];
    c10::cuda::CUDAGuard guard(x.device());
    const Tensor dy = grads[0].contiguous();
    const int64_t flags = ctx->saved_data["f"].toInt();
    const int code = (int)(flags & 255);
    const bool want_w = flags >> 24 & 1, want_b = flags >> 25 & 1;
    const int64_t cols = x.size(-1), rows = cols ? x.numel() / cols : 0;
    const auto grad_type = code == PX_F32 ? at::kFloat : x.scalar_type();
    const Tensor dx = at::empty_like(x);
    Tensor dw, db, scratch;
    if (want_w) dw = at::empty({cols}, x.options().dtype(grad_type));
    if (want_b) db = at::empty({cols}, x.options().dtype(grad_type));
    if (want_w || want_b) scratch = at::empty({2 * cols}, x.options().dtype(at::kFloat));
    const cudaStream_t st = at::cuda::getCurrentCUDAStream();
    launch("px_layer_norm_bwd", st, [&] {
      return abi.px_layer_norm_bwd_params(dy.data_ptr(), x.data_ptr(), (const float*)mean.data_ptr(), (const float*)invvar.data_ptr(),
                                          w.defined() ? w.data_ptr() : nullptr, dx.data_ptr(), want_w ? dw.data_ptr() : nullptr,
                                          want_b ? db.data_ptr() : nullptr, scratch.defined() ? (float*)scratch.data_ptr() : nullptr,
                                          rows, cols, dtype_code(x, "x"), code, st);
    });
    auto as = [&](const Tensor& t, int shift) {
      const auto type = (at::ScalarType)(flags >> shift & 255);
      return !t.defined() || t.scalar_type() == type ? t : t.to(type);
    };
    return {flags >> 26 & 1 ? dx : Tensor(), as(dw, 8), as(db, 16), Tensor()};
  }
};

Tensor layer_norm(const Tensor& x, const OptTensor& weight, const OptTensor& bias, int64_t width, double eps) {
  ln_check(x, width);
  auto wants = [](const OptTensor& t) { return has(t) && t->requires_grad(); };
  if (at::GradMode::is_enabled() && (x.requires_grad() || wants(weight) || wants(bias)))
    return LayerNormFunction::apply(x, weight, bias, eps);
  const Tensor xc = x.contiguous();
  return ln_forward(xc, ln_params(xc, weight, bias), eps, nullptr, nullptr);
}

// ---- residual + row-shared dropout -----------------------------------------------------------------------------------
// residual + x * mask with mask [..., 1, C, D] shared over axis -3 (residual undefined: x * mask)
Tensor scale_add(const Tensor& residual, const Tensor& x_, const Tensor& mask) {
  c10::cuda::CUDAGuard guard(x_.device());
  const Tensor x = x_.contiguous(), r = residual.defined() ? residual.contiguous() : residual;
  const Tensor out = at::empty_like(x);
  const int64_t rows = x.size(-3), cd = x.size(-2) * x.size(-1), batches = rows * cd ? x.numel() / (rows * cd) : 0;
  const cudaStream_t st = at::cuda::getCurrentCUDAStream();
  launch("px_scale_add_rowwise", st, [&] {
    return abi.px_scale_add_rowwise(r.defined() ? r.data_ptr() : nullptr, x.data_ptr(), mask.data_ptr(), out.data_ptr(), batches, rows,
                                    cd, dtype_code(x, "x"), st);
  });
  return out;
}

struct DropoutAddFunction : torch::autograd::Function<DropoutAddFunction> {
  static Tensor forward(torch::autograd::AutogradContext* ctx, const Tensor& residual, const Tensor& x, const Tensor& mask) {
    ctx->save_for_backward({mask});
    ctx->saved_data["f"] = (int64_t)residual.requires_grad() | (int64_t)x.requires_grad() << 1;
    return scale_add(residual, x, mask);
  }
  static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx, torch::autograd::variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const int64_t flags = ctx->saved_data["f"].toInt();
    return {flags & 1 ? grads[0] : Tensor(), flags & 2 ? scale_add(Tensor(), grads[0], saved[0]) : Tensor(), Tensor()};
  }
};

Tensor dropout_add(const Tensor& residual, const Tensor& x, double p) {
  need_cuda(x, "x");
  if (x.dim() < 3) fail("x must be [..., R, C, D]");
  dtype_code(x, "x");
  need_on(residual, x.device(), "residual");
  if (residual.sizes() != x.sizes() || residual.scalar_type() != x.scalar_type()) fail("residual must match x");
  auto shape = x.sizes().vec();
  shape[shape.size() - 3] = 1;
  Tensor mask;
  {
    // drawn as a dropout of ones: the same generator calls, so that a seed gives the same mask
    at::AutoDispatchBelowAutograd below;
    mask = at::dropout(at::ones(shape, x.options()), p, true);
  }
  if (!at::GradMode::is_enabled() || !(residual.requires_grad() || x.requires_grad())) return scale_add(residual, x, mask);
  return DropoutAddFunction::apply(residual, x, mask);
}

}  // namespace

PYBIND11_MODULE(_C, m) {
  m.def("bind_library", &bind_library);
  m.def("layer_norm", &layer_norm);
  m.def("dropout_add", &dropout_add);
  py::class_<Params, std::shared_ptr<Params>>(m, "Params")
      .def(py::init<std::string, py::object, py::list, py::list, py::list>())
      .def("current", &Params::current)
      // kept in a module's __dict__: a copy or an unpickled module makes its own
      .def("__deepcopy__", [](const Params&, py::dict) { return py::none(); })
      .def("__reduce__", [](const Params&) { return py::make_tuple(py::type::of(py::none()), py::tuple()); });
  py::class_<Block, std::shared_ptr<Block>>(m, "Block")
      .def(py::init([](std::vector<std::shared_ptr<Params>> p) {
        if (p.size() != 7) fail("a block has seven parameter groups");
        return std::make_shared<Block>(Block{p[0], p[1], p[2], p[3], p[4], p[5], p[6]});
      }))
      .def("current", &Block::current)
      .def("__deepcopy__", [](const Block&, py::dict) { return py::none(); })
      .def("__reduce__", [](const Block&) { return py::make_tuple(py::type::of(py::none()), py::tuple()); });
  m.def("tri_mul_forward", &tri_mul_forward);
  m.def("tri_att_forward", &tri_att_forward);
  m.def("transition_forward", &transition_forward);
  m.def("stack_forward", &stack_forward);
  m.def("opm_forward", &opm_forward);
  m.def("msa_stack_forward", &msa_stack_forward);
  m.def("launches", [](bool reset) { return reset ? g_launches.exchange(0) : g_launches.load(); });
  m.def("timer", [](bool on) { g_timing = on; });
  m.def("timer_collect", &timer_collect);
}
