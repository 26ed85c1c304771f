// Host path of the operators: argument checks, output allocation and the call of the C ABI, natively.
//
// One product of a served layer takes 3 - 15 us on the GPU; the same call written in Python (ctypes structure filled
// field by field, device guards, property reads) took 17 - 20 us of host time, so the stream ran dry between calls.
// Everything here ends in the entry points of include/void_b200.h; nothing computes on the CPU.  Functions take their
// arguments by position (METH_FASTCALL) from the Python operators, which keep the public signatures.
#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/autograd/saved_variable.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <memory>
#include <mutex>
#include <optional>
#include <string>
#include <vector>

#include "../../include/void_b200.h"

namespace {

PyObject* g_error = nullptr;  // void_b200._lib.VoidB200Error

// Raised as VoidB200Error; caught at the boundary of every function of the module.
struct Failure {
  std::string text;
};
[[noreturn]] void fail(const std::string& text) { throw Failure{text}; }
void check(int status, const char* what) {
  if (status != VOID_OK)
    fail(std::string("void_b200 ") + what + " failed: " + void_strerror(status) + " (status " + std::to_string(status) + ")");
}

bool none(PyObject* o) { return o == Py_None || o == nullptr; }
const at::Tensor& tensor(PyObject* o, const char* what) {
  if (!THPVariable_Check(o)) throw torch::TypeError(std::string(what) + " must be a tensor");
  return THPVariable_Unpack(o);
}
const at::Tensor& cuda_tensor(PyObject* o, const char* what) {
  const at::Tensor& t = tensor(o, what);
  if (!t.is_cuda())
    fail("void_b200 runs on a B200 GPU only: got a tensor on " + t.device().str() + " (there is no CPU path)");
  return t;
}
int64_t integer(PyObject* o) {
  const long long v = PyLong_AsLongLong(o);
  if (v == -1 && PyErr_Occurred()) throw python_error();
  return v;
}
double real(PyObject* o) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) throw python_error();
  return v;
}
int out_code(at::ScalarType t) {
  switch (t) {
    case at::kFloat: return VOID_OUT_F32;
    case at::kHalf: return VOID_OUT_F16;
    case at::kBFloat16: return VOID_OUT_BF16;
    default: fail(std::string("unsupported output dtype ") + c10::toString(t));
  }
}
int elem_bytes(int kind) { return kind == VOID_KIND_TF32 ? 4 : ((kind == VOID_KIND_F16 || kind == VOID_KIND_BF16) ? 2 : 1); }
at::Tensor new_cuda(at::IntArrayRef size, at::ScalarType type, c10::Device dev) {
  return at::Tensor(at::detail::empty_cuda(size, type, dev, std::nullopt));
}
at::Tensor as_type(const at::Tensor& t, at::ScalarType type) { return t.scalar_type() == type ? t : t.to(type); }
void_stream_t stream_of(c10::DeviceIndex dev) { return c10::cuda::getCurrentCUDAStream(dev).stream(); }

// The streams that have read the arrays of a store.  The allocator knows the stream an array was allocated on; that another
// one reads it has to be said, or the memory is handed out again when the tensor is dropped while that stream's kernel still
// runs.  Callers cannot say it for arrays they never see.
class Readers {
 public:
  // the stream all arrays were allocated on, where that is known
  void home(cudaStream_t stream) { seen_.push_back(stream); }
  void add(c10::cuda::CUDAStream stream, std::initializer_list<const at::Tensor*> arrays) {
    const intptr_t key = reinterpret_cast<intptr_t>(stream.stream());
    if (last_.load(std::memory_order_acquire) == key) return;
    const std::lock_guard<std::mutex> lock(mutex_);
    if (std::find(seen_.begin(), seen_.end(), stream.stream()) == seen_.end()) {
      for (const at::Tensor* t : arrays)
        if (t->defined()) c10::cuda::CUDACachingAllocator::recordStream(t->storage().data_ptr(), stream);
      seen_.push_back(stream.stream());
    }
    last_.store(key, std::memory_order_release);
  }

 private:
  std::atomic<intptr_t> last_{-1};   // the last one added
  std::mutex mutex_;
  std::vector<cudaStream_t> seen_;
};

#define NATIVE_BEGIN                                    \
  HANDLE_TH_ERRORS                                      \
  try {
#define NATIVE_END                                      \
  }                                                     \
  catch (const Failure& f) {                            \
    PyErr_SetString(g_error, f.text.c_str());           \
    return nullptr;                                     \
  }                                                     \
  END_HANDLE_TH_ERRORS

// ------------------------------------------------------------------------------------------ packed A
// What a store was made from, so that it is made again when its tensor has changed: the storage (held weakly, so that its
// address cannot come back as another one's), the version of its contents and how the tensor lies in it.
struct Identity {
  std::optional<c10::weak_intrusive_ptr<c10::StorageImpl>> storage;   // none: no tensor
  const void* ptr = nullptr;
  int64_t version = 0;
  at::ScalarType type = at::kFloat;
  c10::SmallVector<int64_t, 6> layout;   // sizes, then strides

  Identity() = default;
  explicit Identity(PyObject* o) {
    if (none(o)) return;
    const at::Tensor& t = tensor(o, "operand");
    storage = t.storage().getWeakStorageImpl();
    ptr = t.const_data_ptr();
    version = t.is_inference() ? -1 : (int64_t)t._version();
    type = t.scalar_type();
    layout.append(t.sizes().begin(), t.sizes().end());
    layout.append(t.strides().begin(), t.strides().end());
  }
  // Inference tensors have no version: their contents may have changed at any time.
  bool still(PyObject* o) const {
    if (none(o)) return !storage.has_value();
    const at::Tensor& t = tensor(o, "operand");
    const size_t dims = (size_t)t.dim();
    return storage.has_value() && storage->_unsafe_get_target() == t.storage().unsafeGetStorageImpl() && ptr == t.const_data_ptr() &&
           !t.is_inference() && version == (int64_t)t._version() && type == t.scalar_type() && layout.size() == 2 * dims &&
           std::equal(t.sizes().begin(), t.sizes().end(), layout.begin()) &&
           std::equal(t.strides().begin(), t.strides().end(), layout.begin() + (std::ptrdiff_t)dims);
  }
};
// The tiles of a packed tensor laid out once more for products of groups of tile rows (csrc/group.cu).
struct GroupStore {
  at::Tensor index, blob;
  void_group_store store = {};
  cudaEvent_t built = nullptr;   // behind the kernels that write it; null once it is known to be complete
  bool captured = false;         // a graph reads it
  Readers readers;
  GroupStore() = default;
  GroupStore(const GroupStore&) = delete;
  GroupStore& operator=(const GroupStore&) = delete;
  ~GroupStore() {
    if (built != nullptr) cudaEventDestroy(built);
  }
};
constexpr int kMaxGroupStores = 2;
struct Packed {
  void_spmm_args args = {};   // the fields of A; everything of a launch is filled into a copy
  at::Tensor tiles, tile_cols, tile_scales, row_ptr, row_scale_array, row_order_array;   // what those fields point into
  const int32_t* row_order = nullptr;
  const float* row_scale = nullptr;
  Identity made_from[4];      // values, scales, block rows, block columns
  int64_t M = 0, K = 0;
  int32_t kind = 0;
  int32_t stable = 0;
  c10::DeviceIndex device = 0;
  Readers readers;
  std::unique_ptr<GroupStore> groups[kMaxGroupStores];   // null: not built
  int32_t group_calls = 0;    // products a group store would have served since the last build; -1: there was no room for one
  bool grouped = true;        // whether group stores may be built and used
  bool captured = false;      // a graph was captured that reads these arrays, and may be replayed as long as the tensor lives
  std::vector<std::unique_ptr<GroupStore>> retired;   // group stores that are no longer used, but read by a graph
};
struct PackedObject {
  PyObject_HEAD
  Packed* packed;
};
PyTypeObject* g_packed_type = nullptr;

Packed* packed_of(PyObject* o) {
  if (Py_TYPE(o) != g_packed_type) throw torch::TypeError("expected a packed tensor handle");
  return reinterpret_cast<PackedObject*>(o)->packed;
}
template <typename T>
T* data_or_null(PyObject* o) {
  return none(o) ? nullptr : static_cast<T*>(tensor(o, "operand").data_ptr());
}
bool capturing(void_stream_t st);
// The stream a product of this store is launched on, noted as one of its readers.
void_stream_t launch_stream(Packed* p) {
  const c10::cuda::CUDAStream stream = c10::cuda::getCurrentCUDAStream(p->device);
  p->readers.add(stream, {&p->tiles, &p->tile_cols, &p->tile_scales, &p->row_ptr, &p->row_scale_array, &p->row_order_array});
  if (capturing(stream.stream())) p->captured = true;
  return stream.stream();
}

// packed_handle(M, K, kind, terms, nnz, stable, status, tiles, tile_cols, tile_scales, row_ptr, row_scale, row_order, home | None)
PyObject* packed_handle(PyObject*, PyObject* const* a, Py_ssize_t n) {
  NATIVE_BEGIN
  if (n != 14) throw torch::TypeError("packed_handle takes 14 arguments");
  std::unique_ptr<Packed> p(new Packed);
  p->M = integer(a[0]);
  p->K = integer(a[1]);
  p->kind = (int32_t)integer(a[2]);
  p->args.tile_terms = (int32_t)integer(a[3]);
  p->args.nnz = integer(a[4]);
  p->stable = (int32_t)integer(a[5]);
  p->args.status = data_or_null<int32_t>(a[6]);
  at::Tensor* arrays[6] = {&p->tiles, &p->tile_cols, &p->tile_scales, &p->row_ptr, &p->row_scale_array, &p->row_order_array};
  for (int i = 0; i < 6; ++i)
    if (!none(a[7 + i])) *arrays[i] = cuda_tensor(a[7 + i], "packed array");
  p->args.tiles = data_or_null<void>(a[7]);
  p->args.tile_cols = data_or_null<int32_t>(a[8]);
  p->args.tile_scales = data_or_null<float>(a[9]);
  p->args.row_ptr = data_or_null<int32_t>(a[10]);
  p->row_scale = data_or_null<float>(a[11]);
  p->row_order = data_or_null<int32_t>(a[12]);
  p->args.nbr = (int32_t)((p->M + 31) / 32);
  p->args.nbc = (int32_t)((p->K + 31) / 32);
  p->args.M = (int32_t)p->M;
  p->args.K = (int32_t)p->K;
  p->device = p->tiles.device().index();
  if (!none(a[13])) p->readers.home(reinterpret_cast<cudaStream_t>((intptr_t)integer(a[13])));
  PyObject* self = PyType_GenericAlloc(g_packed_type, 0);
  if (self == nullptr) return nullptr;
  reinterpret_cast<PackedObject*>(self)->packed = p.release();
  return self;
  NATIVE_END
}

// packed_made_from(handle, values, scales, block_rows, block_cols): note what the store was packed from
PyObject* packed_made_from(PyObject*, PyObject* const* a, Py_ssize_t n) {
  NATIVE_BEGIN
  if (n != 5) throw torch::TypeError("packed_made_from takes 5 arguments");
  Packed* p = packed_of(a[0]);
  for (int i = 0; i < 4; ++i) p->made_from[i] = Identity(a[1 + i]);
  Py_RETURN_NONE;
  NATIVE_END
}
// packed_is_current(handle, values, scales, block_rows, block_cols, shape): the store still belongs to these tensors
bool is_current(const Packed* p, PyObject* values, PyObject* scales, PyObject* rows, PyObject* cols, PyObject* shape) {
  PyObject* const from[4] = {values, scales, rows, cols};
  for (int i = 0; i < 4; ++i)
    if (!p->made_from[i].still(from[i])) return false;
  return PyTuple_Check(shape) && PyTuple_GET_SIZE(shape) == 2 && integer(PyTuple_GET_ITEM(shape, 0)) == p->M &&
         integer(PyTuple_GET_ITEM(shape, 1)) == p->K;
}
PyObject* packed_is_current(PyObject*, PyObject* const* a, Py_ssize_t n) {
  NATIVE_BEGIN
  if (n != 6) throw torch::TypeError("packed_is_current takes 6 arguments");
  return PyBool_FromLong(is_current(packed_of(a[0]), a[1], a[2], a[3], a[4], a[5]));
  NATIVE_END
}

// identity(tensor | None, ...) -> what the tensors are now; unchanged(identity, tensor | None, ...) -> whether they still are:
// for what the Python layer derives from a tensor's fields and keeps
constexpr const char* kIdentityName = "void_b200.identity";
PyObject* identity(PyObject*, PyObject* const* a, Py_ssize_t n) {
  NATIVE_BEGIN
  std::unique_ptr<std::vector<Identity>> ids(new std::vector<Identity>);
  for (Py_ssize_t i = 0; i < n; ++i) ids->emplace_back(a[i]);
  PyObject* c = PyCapsule_New(ids.get(), kIdentityName, [](PyObject* o) {
    delete static_cast<std::vector<Identity>*>(PyCapsule_GetPointer(o, kIdentityName));
  });
  if (c != nullptr) ids.release();
  return c;
  NATIVE_END
}
PyObject* unchanged(PyObject*, PyObject* const* a, Py_ssize_t n) {
  NATIVE_BEGIN
  if (n < 1) throw torch::TypeError("unchanged takes an identity and its tensors");
  const auto* ids = static_cast<const std::vector<Identity>*>(PyCapsule_GetPointer(a[0], kIdentityName));
  if (ids == nullptr) return nullptr;
  bool same = ids->size() == (size_t)n - 1;
  for (Py_ssize_t i = 1; same && i < n; ++i) same = (*ids)[(size_t)i - 1].still(a[i]);
  return PyBool_FromLong(same);
  NATIVE_END
}

// packed_captured(handle) -> whether a graph reads this store: then it is kept when another takes its place
PyObject* packed_captured(PyObject*, PyObject* const* a, Py_ssize_t n) {
  NATIVE_BEGIN
  if (n != 1) throw torch::TypeError("packed_captured takes 1 argument");
  return PyBool_FromLong(packed_of(a[0])->captured);
  NATIVE_END
}

// packed_grouped(handle, allowed | None) -> (allowed, group stores, of them complete): whether products may use tiles laid out
// for groups of tile rows; the stores there are, are given back when they may not (those a graph reads with the tensor)
PyObject* packed_grouped(PyObject*, PyObject* const* a, Py_ssize_t n) {
  NATIVE_BEGIN
  if (n != 2) throw torch::TypeError("packed_grouped takes 2 arguments");
  Packed* p = packed_of(a[0]);
  if (!none(a[1])) {
    p->grouped = PyObject_IsTrue(a[1]) == 1;
    if (!p->grouped) {
      for (std::unique_ptr<GroupStore>& g : p->groups) {
        if (g != nullptr && g->captured) p->retired.push_back(std::move(g));
        g.reset();
      }
      p->group_calls = 0;
    }
  }
  int stores = 0, done = 0;
  for (const std::unique_ptr<GroupStore>& g : p->groups)
    if (g != nullptr) {
      ++stores;
      done += g->built == nullptr ? 1 : 0;
    }
  return Py_BuildValue("Oii", p->grouped ? Py_True : Py_False, stores, done);
  NATIVE_END
}

// ------------------------------------------------------------------------------------------ products
// Elements between the rows of an operand that is allocated here, rows on 64 bytes: 128-byte pieces of rows that start anywhere
// touch a sector more (N = 1000, 60 %, 4096 x 1024: fp16 16.7 -> 13.9 us, INT8 10.9 -> 9.4).
int64_t padded_pitch(int64_t cols, int es) { return (cols * es + 63) / 64 * 64 / es; }
// B with unit column stride and rows on 16-byte boundaries, as the copy engine needs them; others are copied (one pass).
// A single row has no pitch, so only its start matters.  Whole panels (products: the (tile, 128 columns) pairs that read one) of
// rows that start on 16 bytes but not on 32 load slower, by 0.17 ns a pair for 16-bit and 0.12 for 8-bit elements, so large
// products have them copied too: N = 1000, 8192^2, 80 %: fp16 98 -> 75 us and 6.5 for the copy, INT8 49 -> 36 and 6.
at::Tensor kernel_operand(const at::Tensor& b, int es, int64_t products = 0) {
  if (b.element_size() != es)
    fail("B must have " + std::to_string(es) + "-byte elements to match A, got " + c10::toString(b.scalar_type()));
  const int64_t rows = b.size(0), cols = b.size(1), per16 = 16 / es;
  const bool unit = b.stride(1) == 1 || cols <= 1;
  if (unit && (reinterpret_cast<uintptr_t>(b.const_data_ptr()) & 15u) == 0 &&
      (rows == 1 || (b.stride(0) % per16 == 0 && b.stride(0) >= cols))) {
    const double saves = products * (es == 1 ? 0.12 : (es == 2 ? 0.17 : 0.0)), costs = 3500.0 + 2.0 * rows * cols * es / 4500.0;
    if (rows == 1 || b.stride(0) * es % 32 == 0 || saves < costs) return b;
  }
  const int64_t ld = padded_pitch(cols, es);
  at::Tensor padded = new_cuda({rows, ld}, b.scalar_type(), b.device());
  at::Tensor view = padded.narrow(1, 0, cols);
  if (unit && b.stride(0) >= cols)
    check(void_copy_rows(b.const_data_ptr(), b.stride(0) * es, padded.data_ptr(), ld * es, es, rows, (int32_t)cols,
                         stream_of(b.device().index())),
          "void_copy_rows");
  else
    view.copy_(b);
  return view;
}
// Bytes between the rows of a kernel operand.
int64_t row_pitch(const at::Tensor& b, int es) {
  return b.size(0) == 1 ? (b.size(1) * es + 15) / 16 * 16 : b.stride(0) * es;
}
// A linear layer on x [N, K] either reads x as it lies (its 32-element pieces of rows load at a fraction of the rate of
// whole panels) or has it transposed to [K, N] first and its result written transposed.  The copy costs two passes over x
// and a launch that nothing overlaps; what it saves grows with the (tile, 128 columns) products: INT8 0.36 ns each (8192^2,
// N = 1024, 80 %: 73.4 -> 40.6 us), 16 bits 0.15 (16384 rows of 13 / 26 / 51 tiles, N = 2048: 83.6 -> 78.0, 142 -> 130, 260 -> 233;
// 8192 rows, N = 4096: 85.4 -> 83.0, 150 -> 150, 270 -> 259), fp32 no more than the copy takes (8192^2, N = 1024, 50 %: 298.5
// against 298.8).
double copy_saves_ns(int kind, int64_t nnz, int64_t N) {
  const double per = kind == VOID_KIND_I8 ? 0.36 : (kind == VOID_KIND_TF32 ? 0.0 : 0.15);
  return per * (double)nnz * (double)((N + 127) / 128);
}
double copy_costs_ns(int64_t N, int64_t K, int es) { return 5000.0 + 2.0 * (double)N * (double)K * es / 4500.0; }
bool copy_pays(int kind, int64_t nnz, int64_t N, int64_t K) {
  return N > 128 && copy_saves_ns(kind, nnz, N) > copy_costs_ns(N, K, elem_bytes(kind));
}
// A matrix with rows on 16-byte boundaries whose contents are to be written.
at::Tensor pitched(int64_t rows, int64_t cols, at::ScalarType type, int es, c10::Device dev) {
  const int64_t ld = padded_pitch(cols, es);
  const at::Tensor t = new_cuda({rows, ld}, type, dev);
  return ld == cols ? t : t.narrow(1, 0, cols);
}
at::Tensor transposed_copy(const at::Tensor& x_in, int es) {
  if (x_in.element_size() != es)
    fail("B must have " + std::to_string(es) + "-byte elements to match A, got " + c10::toString(x_in.scalar_type()));
  const at::Tensor x = x_in.stride(1) == 1 && x_in.stride(0) >= x_in.size(1) ? x_in : x_in.contiguous();
  const at::Tensor out = pitched(x.size(1), x.size(0), x.scalar_type(), es, x.device());
  check(void_transpose(x.const_data_ptr(), x.stride(0) * es, out.data_ptr(), out.stride(0) * es, es, (int32_t)x.size(0),
                       (int32_t)x.size(1), stream_of(x.device().index())),
        "void_transpose");
  return out;
}
at::Tensor fp32_vector(PyObject* o, c10::Device dev, const char* what, int64_t at_least = 0) {
  const at::Tensor& t = tensor(o, what);
  if (t.numel() < at_least)
    fail(std::string(what) + " must have " + std::to_string(at_least) + " elements, got " + std::to_string(t.numel()));
  if (t.scalar_type() == at::kFloat && t.device() == dev && t.is_contiguous()) return t;
  return t.to(dev, at::kFloat).contiguous();
}

// ------------------------------------------------------------------------------------------ groups of tile rows
// How the tile rows are dealt to groups for N columns, and what that saves.  In units of a row-accumulate launch's bytes: a
// CTA slot (two per SM) takes `turns` groups, each the panels of the block columns that any of its rows stores and its tiles;
// the other kernel takes a panel with every tile.  More than four rows leave no second accumulator set, which costs where a
// slot has more than one group (16384 x 4096, N = 2048, fp16, 7 and 4 rows, us: 70 % 131 133, 80 % 102 100, 85 % 86 80; fp32 70 % 255 -,
// 80 % 199 211); with up to four there is still the end of each.
struct GroupShape {
  int groups = 0;
  double saves = 0.0;
};
double group_saves(const Packed* p, int64_t N, int groups, int slots) {
  const int es = elem_bytes(p->kind);
  const double chunks = (double)((N + 127) / 128), nbr = p->args.nbr, nbc = p->args.nbc, nnz = (double)p->args.nnz;
  const double d = nnz / (nbr * nbc), panel = 4.0 * es, tile = es;
  const double rows = std::ceil(nbr / groups), turns = std::ceil(groups * chunks / slots);
  double cost = turns * nbc * ((1.0 - std::pow(1.0 - d, rows)) * panel + d * rows * tile);
  if (turns > 1) cost *= rows > 4 ? (es == 4 ? 1.2 : 1.3) : 1.05;
  return nnz * chunks / slots * (panel + tile) / cost;
}
// What a stage holds: the split of a CTA's shared memory into stages of E block columns and T tiles with which the ring holds the
// most block columns, T / (tiles that a column's panel serves) or E of them per stage.  Of equal ones that with three stages: a
// stage costs the same chain of waits whatever is in it.  (8192^2, N = 1024, us: fp16 80 % 3 x (3 + 5) 46.2, 2 x (4 + 8) 49, 4 x (2 + 4) 49;
// INT8 50 % 3 x (4 + 18) 42.0, 2 x (6 + 21) 43.6.)  The room is that beside staged results, which those of fp32 tiles are with an operand of 16
// bits only; with all of it fp32 stages would hold a tile more: chosen and best seen, 50 % 3 x (1 + 4) 166, 3 x (1 + 5) 157, 70 % 4 x (1 + 2) 129,
// 3 x (1 + 5) 117, 80 % 4 x (1 + 2) 93, 2 x (2 + 5) 90, but 16-bit results 3 x (1 + 4) 164, (1 + 5), of which two are left beside the staging, 185.
void stage_shape(void_group_store& s, double tiles_per_column, int es) {
  const int room = 116736 - 3072 - 8192;   // half of an SM's shared memory less the kernel's own and the staging of its results
  double most = 0.0;
  for (int n : {3, 4, 5, 6, 2}) {
    const int bytes = room / n / 1024 * 1024;
    for (int e = 1; e <= 6; ++e) {
      const int t = std::min((bytes - e * 4096 * es) / (1024 * es), 32);
      if (t < 1) break;
      const double columns = n * std::min((double)e, t / tiles_per_column);
      if (columns > 1.01 * most) {
        most = columns;
        s.max_entries = e;
        s.max_tiles = t;
      }
    }
  }
}
GroupShape group_shape(const Packed* p, int64_t N, int slots) {
  GroupShape best;
  const int64_t chunks = (N + 127) / 128, nbr = p->args.nbr;
  for (int64_t turns = 1; turns <= 256; ++turns) {
    const int64_t groups = turns * slots / chunks;
    if (groups < 1) continue;
    const int64_t rows = (nbr + groups - 1) / groups;
    if (rows > 8) continue;
    if (rows < 2) break;
    const double saves = group_saves(p, N, (int)groups, slots);
    if (saves > best.saves) {
      best.saves = saves;
      best.groups = (int)groups;
    }
  }
  return best;
}
// The saving from which the grouped kernel is the faster one; swept at 4096^2, 8192^2 (N = 1024), 16384 x 4096 and 4096 x 16384 (N = 2048),
// 50 - 90 % sparsity.  Predicted saving and measured gain, fp16: 1.06 0.99 - 1.07, 1.09 1.01, 1.12 1.06 - 1.15, 1.12 1.10, 1.22 1.07, 1.36 1.14,
// 1.52 1.24, 2.32 1.53; fp32 0.97 0.99, 1.03 1.08, 1.06 0.95, 1.09 1.19, 1.12 1.15, 1.15 1.15, 1.22 1.22, 1.24 1.12, 1.26 1.20,
// 1.38 1.18, 1.40 1.24, 1.50 1.27 - 1.31, 1.52 1.25, 1.68 1.24, 1.80 1.32, 1.93 1.72, 2.17 1.70, 2.32 1.67; INT8 1.36 - 1.38 0.99 - 1.01, 1.50 1.13, 1.52 1.06,
// 1.80 1.21, and with rows of 100 tiles 1.26 1.07, 1.40 1.11.
double group_line(const Packed* p) {
  switch (p->kind) {
    case VOID_KIND_I8: return p->args.nnz >= 96ll * p->args.nbr ? 1.3 : 1.45;
    case VOID_KIND_TF32: return 1.12;
    default: return 1.1;
  }
}
// Whether the kernels that write the store are through.  Asked without waiting; not while the stream is captured, where the
// store then is not used.  (Another thread may be capturing: relaxed mode keeps the question from ending its capture.)
bool complete(GroupStore* g, void_stream_t st) {
  if (g->built == nullptr) return true;
  if (capturing(st)) return false;
  const c10::cuda::CUDAStreamCaptureModeGuard relaxed(cudaStreamCaptureModeRelaxed);
  if (cudaEventQuery(g->built) != cudaSuccess) {
    (void)cudaGetLastError();   // "not ready" is no error of the launch that follows
    return false;
  }
  cudaEventDestroy(g->built);
  g->built = nullptr;
  return true;
}
int64_t group_blob_bytes(const Packed* p) { return p->args.nnz * (1024 * (int64_t)elem_bytes(p->kind) + VOID_GROUP_HEAD_BYTES); }
// Queues the kernels that lay the tiles out for G groups; null where there is no memory for it.
std::unique_ptr<GroupStore> build_group_store(const Packed* p, int64_t G, void_stream_t st) {
  std::unique_ptr<GroupStore> g(new GroupStore);
  const int64_t nnz = p->args.nnz, es = elem_bytes(p->kind);
  at::Tensor ws;
  try {
    const c10::Device dev(c10::kCUDA, p->device);
    g->index = new_cuda({16 * G + (G + 4) / 4 * 4 + 8 * nnz}, at::kInt, dev);
    g->blob = new_cuda({group_blob_bytes(p) + 128}, at::kByte, dev);
    ws = new_cuda({2 * G + nnz}, at::kInt, dev);
  } catch (const c10::OutOfMemoryError&) {
    return nullptr;
  }
  int32_t *rows = g->index.data_ptr<int32_t>(), *stages = rows + 16 * G, *records = stages + (G + 4) / 4 * 4;
  uint8_t* blob = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(g->blob.data_ptr()) + 127) & ~uintptr_t(127));
  g->store.blob = blob;
  g->store.records = records;
  g->store.stage_ptr = stages;
  g->store.group_rows = rows;
  g->store.n_groups = (int32_t)G;
  const double d = (double)nnz / ((double)p->args.nbr * p->args.nbc), in_group = std::ceil((double)p->args.nbr / (double)G);
  stage_shape(g->store, in_group * d / (1.0 - std::pow(1.0 - d, in_group)), (int)es);
  if (cudaEventCreateWithFlags(&g->built, cudaEventDisableTiming) != cudaSuccess) return nullptr;
  check(void_group_build(p->args.row_ptr, p->row_order, p->args.tile_cols, p->args.tiles, p->args.nbr, nnz, (int32_t)es, (int32_t)G,
                         g->store.max_entries, g->store.max_tiles, rows, stages, records, blob, ws.data_ptr<int32_t>(), st),
        "void_group_build");
  if (cudaEventRecord(g->built, reinterpret_cast<cudaStream_t>(st)) != cudaSuccess) throw std::runtime_error("CUDA error: recording an event failed");
  return g;
}
// The group store that serves this product, or null.  Its build is queued behind the third product it would have served - a
// tensor that is multiplied once or twice does not pay for it - once for each of up to two widths.  Nothing waits for it:
// products go to the other kernel until it is complete, and then read it on any stream and ahead of their stream's order.
GroupStore* group_store(Packed* p, int64_t N, void_stream_t st) {
  if (!p->grouped || N <= 64 || p->args.nnz < 4096 || p->kind == VOID_KIND_F8E4M3) return nullptr;   // (FP8 of two terms: within 5 % either way)
  const int slots = 2 * void_device_sm_count();
  if ((int64_t)p->args.nbr * ((N + 127) / 128) < 2ll * slots) return nullptr;
  const double line = group_line(p);
  const GroupShape shape = group_shape(p, N, slots);
  if (shape.saves < line) return nullptr;
  GroupStore* hit = nullptr;
  double hit_saves = 0.0, best = 0.0;   // best: of those that are still being built, too
  int n = 0;
  for (; n < kMaxGroupStores && p->groups[n] != nullptr; ++n) {
    const double saves = group_saves(p, N, p->groups[n]->store.n_groups, slots);
    best = std::max(best, saves);
    if (saves > hit_saves && complete(p->groups[n].get(), st)) { hit = p->groups[n].get(); hit_saves = saves; }
  }
  if (best < 0.93 * shape.saves && n < kMaxGroupStores && p->stable && group_blob_bytes(p) <= (4ll << 30) && p->group_calls >= 0 && !capturing(st) &&
      ++p->group_calls >= 3) {
    p->group_calls = -1;   // for good, if there is no room for it
    p->groups[n] = build_group_store(p, shape.groups, st);
    if (p->groups[n] != nullptr) p->group_calls = 0;
  }
  return hit_saves >= line ? hit : nullptr;
}
// A plain product with everything filled in.
void launch_product(Packed* p, const void_spmm_args& s, void_stream_t st) {
  if (s.transposed != 1 && s.scale_mode == VOID_SCALE_ROW_MEAN) {
    GroupStore* g = group_store(p, s.N, st);
    if (g != nullptr) {
      g->readers.add(c10::cuda::getCurrentCUDAStream(p->device), {&g->index, &g->blob});
      if (p->captured && capturing(st)) g->captured = true;
      check(void_spmm_grouped(&s, &g->store, p->kind, st), "void_spmm_grouped");
      return;
    }
  }
  if (elem_bytes(p->kind) > 1) check(void_spmm_fp(&s, p->kind, st), "void_spmm_fp");
  else check(p->kind == VOID_KIND_I8 ? void_spmm_i8(&s, st) : void_spmm_f8(&s, st), "void_spmm");
}

// An array for raw sums of four bytes each; null for None.
void* raw_sums(PyObject* o, c10::Device dev, int64_t at_least, const char* what) {
  if (none(o)) return nullptr;
  const at::Tensor& t = cuda_tensor(o, what);
  if (t.device() != dev || t.element_size() != 4 || !t.is_contiguous() || t.numel() < at_least)
    fail(std::string(what) + " must be a contiguous tensor of at least " + std::to_string(at_least) + " 32-bit elements on B's device");
  return t.data_ptr();
}

// spmm(handle, b, out | None, out_dtype | None, per_tile, col_scale | None, b_scale, bias | None, row_bias | None, act,
//      transposed, options | None) -> out
// options: (plan | None, acc_out, worker_partials, panels, stages, grid, tiles_per_stage, cta_shape, trace, flags,
//           test_hooks, sorted_rows | None, use_row_scale); plan: (segs, cta_seg_ptr, n_cta, partials | None, counters, panels)
PyObject* spmm(PyObject*, PyObject* const* a, Py_ssize_t n) {
  NATIVE_BEGIN
  if (n != 12) throw torch::TypeError("spmm takes 12 arguments");
  Packed* pk = packed_of(a[0]);
  const at::Tensor& b_in = cuda_tensor(a[1], "B");
  const c10::Device dev = b_in.device();
  const bool tr = PyObject_IsTrue(a[10]) == 1;
  if (b_in.dim() != 2) fail("B must be a matrix");
  if (b_in.size(tr ? 1 : 0) != pk->K)
    fail("shape mismatch: A is (" + std::to_string(pk->M) + ", " + std::to_string(pk->K) + "), B is (" +
         std::to_string(b_in.size(0)) + ", " + std::to_string(b_in.size(1)) + ")");
  if (dev.index() != pk->device) fail("A and B are on different devices");
  const int64_t N = b_in.size(tr ? 0 : 1);
  const int64_t rows = tr ? N : pk->M, cols = tr ? pk->M : N;
  const int es = elem_bytes(pk->kind);
  c10::cuda::OptionalCUDAGuard guard;
  if (c10::cuda::current_device() != dev.index()) guard.set_device(dev);

  at::Tensor out;
  if (none(a[2])) {
    const at::ScalarType type = none(a[3]) ? at::kFloat : reinterpret_cast<THPDtype*>(a[3])->scalar_type;
    out_code(type);
    out = new_cuda({rows, cols}, type, dev);
  } else {
    out = cuda_tensor(a[2], "out");
    if (out.dim() != 2 || out.size(0) != rows || out.size(1) != cols || out.stride(1) != 1)
      fail("out must be a row-major [" + std::to_string(rows) + ", " + std::to_string(cols) + "] tensor");
    if (out.device() != dev) fail("out and B are on different devices");
  }
  const bool copied = tr && none(a[11]) && copy_pays(pk->kind, pk->args.nnz, N, pk->K);
  const at::Tensor b = copied ? transposed_copy(b_in, es) : kernel_operand(b_in, es, tr ? 0 : pk->args.nnz * ((N + 127) / 128));

  void_spmm_args s = pk->args;
  const bool per_tile = PyObject_IsTrue(a[4]) == 1;
  s.scale_mode = per_tile ? VOID_SCALE_PER_TILE : VOID_SCALE_ROW_MEAN;
  bool use_row_scale = true;
  s.b = b.const_data_ptr();
  s.ldb = row_pitch(b, es);
  s.N = (int32_t)N;
  at::Tensor col_scale, bias, row_bias;   // keep converted copies alive until the launch is queued
  if (!none(a[5])) {
    col_scale = fp32_vector(a[5], dev, "col_scale", N);
    s.col_scale = col_scale.const_data_ptr<float>();
  }
  s.b_scale = (float)real(a[6]);
  if (!none(a[7])) {
    bias = fp32_vector(a[7], dev, "bias", N);
    s.bias = bias.const_data_ptr<float>();
  }
  if (!none(a[8])) {
    row_bias = fp32_vector(a[8], dev, "row bias");
    if (row_bias.numel() != pk->M)
      fail("row bias must have " + std::to_string(pk->M) + " elements, got " + std::to_string(row_bias.numel()));
    s.row_bias = row_bias.const_data_ptr<float>();
  }
  s.out = out.data_ptr();
  s.ldc = out.stride(0);
  s.out_dtype = out_code(out.scalar_type());
  s.act = (int32_t)integer(a[9]);
  s.transposed = copied ? 2 : (tr ? 1 : 0);
  // Tile rows taken by falling tile count: measured at the 4096^2 sweep and at 16384^2, INT8 gains 3 - 5 %
  // (6.80 -> 6.58 us at 90 %, 10.33 -> 10.02 at 70 %, 72.7 -> 68.7 at 16384^2); FP8 tiles stored as two terms gain at
  // 90 % (7.88 -> 7.57) and lose at 70 % (13.55 -> 13.76): the balance it buys weighs less, and the scattered order of A
  // more, the more bytes a tile row holds.  The 16- and 32-bit kinds run two CTAs per SM, where balance is worth more
  // (4096^2, 90 %: fp32 14.2 -> 13.1 us, fp16 9.3 -> 8.8).
  bool sorted_rows = pk->kind != VOID_KIND_F8E4M3 || s.nnz <= 16ll * s.nbr;
  int64_t flags = 0;
  if (!none(a[11])) {
    PyObject* o = a[11];
    if (!PyTuple_Check(o) || PyTuple_GET_SIZE(o) != 13) throw torch::TypeError("spmm: options is a tuple of 13");
    PyObject* plan = PyTuple_GET_ITEM(o, 0);
    s.panels_per_item = (int32_t)integer(PyTuple_GET_ITEM(o, 3));
    if (!none(plan)) {
      if (!PyTuple_Check(plan) || PyTuple_GET_SIZE(plan) != 6) throw torch::TypeError("spmm: a plan is a tuple of 6");
      s.segs = data_or_null<int32_t>(PyTuple_GET_ITEM(plan, 0));
      s.cta_seg_ptr = data_or_null<int32_t>(PyTuple_GET_ITEM(plan, 1));
      s.n_cta = (int32_t)integer(PyTuple_GET_ITEM(plan, 2));
      if (!none(PyTuple_GET_ITEM(plan, 3))) {
        const at::Tensor& parts = tensor(PyTuple_GET_ITEM(plan, 3), "partials");
        s.partials = parts.data_ptr();
        s.partials_bytes = parts.numel() * 4;
      }
      s.counters = data_or_null<int32_t>(PyTuple_GET_ITEM(plan, 4));
      s.panels_per_item = (int32_t)integer(PyTuple_GET_ITEM(plan, 5));
    }
    s.acc_out = raw_sums(PyTuple_GET_ITEM(o, 1), dev, (int64_t)pk->args.nbr * 32 * N, "acc_out");
    s.worker_partials = raw_sums(PyTuple_GET_ITEM(o, 2), dev, 0, "worker_partials");
    s.stages = (int32_t)integer(PyTuple_GET_ITEM(o, 4));
    s.grid = (int32_t)integer(PyTuple_GET_ITEM(o, 5));
    s.tiles_per_stage = (int32_t)integer(PyTuple_GET_ITEM(o, 6));
    s.cta_shape = (int32_t)integer(PyTuple_GET_ITEM(o, 7));
    s.trace = data_or_null<void>(PyTuple_GET_ITEM(o, 8));
    flags = integer(PyTuple_GET_ITEM(o, 9));
    s.test_hooks = (int32_t)integer(PyTuple_GET_ITEM(o, 10));
    if (!none(PyTuple_GET_ITEM(o, 11))) sorted_rows = PyObject_IsTrue(PyTuple_GET_ITEM(o, 11)) == 1;
    use_row_scale = PyObject_IsTrue(PyTuple_GET_ITEM(o, 12)) == 1;
  }
  if (use_row_scale && !per_tile && es == 1) s.row_scale = pk->row_scale;
  if (s.segs == nullptr && sorted_rows) s.row_order = pk->row_order;
  // bit 2: the packed store (and the plan, whose builder synchronises) is complete, so the kernel may read it
  // before it waits for the previous kernel; bit 30 (measurements) keeps it from doing so
  s.flags = (int32_t)(flags & 0xffff) | ((pk->stable && !(flags & (1ll << 30))) ? 4 : 0);
  const void_stream_t st = launch_stream(pk);
  if (none(a[11])) launch_product(pk, s, st);
  else if (es > 1) check(void_spmm_fp(&s, pk->kind, st), "void_spmm_fp");
  else check(pk->kind == VOID_KIND_I8 ? void_spmm_i8(&s, st) : void_spmm_f8(&s, st), "void_spmm");
  if (!none(a[2])) {
    Py_INCREF(a[2]);
    return a[2];
  }
  return THPVariable_Wrap(out);
  NATIVE_END
}

// act(x A1^T + b1) A2^T + b2 [N, M2] of x [N, K], in x's type
// The activations in between have the layout that suits the products: [N, M1] where the layers read them as they lie, or
// [M1, N] where copying x pays, which then serves both layers.
at::Tensor two_layers(Packed* first, Packed* second, const at::Tensor& x, PyObject* bias1, int32_t act, PyObject* bias2) {
  Packed* pk[2] = {first, second};
  PyObject* const given[2] = {bias1, bias2};
  const c10::Device dev = x.device();
  if (x.dim() != 2 || x.size(1) != pk[0]->K || pk[1]->K != pk[0]->M) fail("shape mismatch between the layers and their input");
  if (dev.index() != pk[0]->device || dev.index() != pk[1]->device) fail("A and B are on different devices");
  if (pk[0]->kind != pk[1]->kind || elem_bytes(pk[0]->kind) == 1) fail("mlp takes two floating layers of one type");
  c10::cuda::OptionalCUDAGuard guard;
  if (c10::cuda::current_device() != dev.index()) guard.set_device(dev);
  const int kind = pk[0]->kind, es = elem_bytes(kind);
  const int64_t N = x.size(0);
  const bool columns = N > 128 && copy_saves_ns(kind, pk[0]->args.nnz + pk[1]->args.nnz, N) > copy_costs_ns(N, pk[0]->K, es);
  const void_stream_t st = launch_stream(pk[0]);
  launch_stream(pk[1]);
  at::Tensor in = columns ? transposed_copy(x, es) : kernel_operand(x, es), bias[2], out;
  for (int layer = 0; layer < 2; ++layer) {
    Packed* p = pk[layer];
    void_spmm_args s = p->args;
    s.scale_mode = VOID_SCALE_ROW_MEAN;
    s.row_order = p->row_order;
    s.b = in.const_data_ptr();
    s.ldb = row_pitch(in, es);
    s.N = (int32_t)N;
    s.b_scale = 1.0f;
    if (!none(given[layer])) {
      bias[layer] = fp32_vector(given[layer], dev, "bias");
      if (bias[layer].numel() != p->M) fail("bias must have " + std::to_string(p->M) + " elements, got " + std::to_string(bias[layer].numel()));
      s.row_bias = bias[layer].const_data_ptr<float>();
    }
    if (layer == 1) out = new_cuda({N, p->M}, x.scalar_type(), dev);
    else out = columns ? pitched(p->M, N, x.scalar_type(), es, dev) : pitched(N, p->M, x.scalar_type(), es, dev);
    s.out = out.data_ptr();
    s.ldc = out.stride(0);
    s.out_dtype = out_code(out.scalar_type());
    s.act = layer == 0 ? act : VOID_ACT_NONE;
    s.transposed = columns ? (layer == 0 ? 0 : 2) : 1;
    s.flags = p->stable ? 4 : 0;
    launch_product(p, s, st);
    in = out;
  }
  return out;
}
// mlp(handle1, handle2, x [N, K], bias1 | None, act, bias2 | None) -> y
PyObject* mlp(PyObject*, PyObject* const* a, Py_ssize_t n) {
  NATIVE_BEGIN
  if (n != 6) throw torch::TypeError("mlp takes 6 arguments");
  return THPVariable_Wrap(two_layers(packed_of(a[0]), packed_of(a[1]), cuda_tensor(a[2], "x"), a[3], (int32_t)integer(a[4]), a[5]));
  NATIVE_END
}
// mlp_packed(handle1, values1, block_rows1, block_cols1, shape1, the same of the second layer, x, bias1 | None, act, bias2 | None)
//   -> y, or None where a store is not current or an operand is not what two packed layers of one type take
// One call with all checks: a decode step's kernels take less time than the interpreter would for them (8192 x 2048 and back,
// eight tokens: kernels 8.8 us, the host 8.2, with a call for each check 10.2).
PyObject* mlp_packed(PyObject*, PyObject* const* a, Py_ssize_t n) {
  NATIVE_BEGIN
  if (n != 14) throw torch::TypeError("mlp_packed takes 14 arguments");
  Packed* pk[2] = {packed_of(a[0]), packed_of(a[5])};
  const at::Tensor& x = tensor(a[10], "x");
  bool ok = x.is_cuda() && x.dim() == 2;
  for (int layer = 0; ok && layer < 2; ++layer) {
    PyObject* const* own = a + 5 * layer;
    PyObject* b = a[layer == 0 ? 11 : 13];
    ok = is_current(pk[layer], own[1], Py_None, own[2], own[3], own[4]) && x.scalar_type() == pk[layer]->made_from[0].type &&
         (none(b) || (tensor(b, "bias").dim() == 1 && tensor(b, "bias").size(0) == pk[layer]->M));
  }
  if (!ok || x.size(1) != pk[0]->K || pk[0]->M != pk[1]->K) Py_RETURN_NONE;
  return THPVariable_Wrap(two_layers(pk[0], pk[1], x, a[11], (int32_t)integer(a[12]), a[13]));
  NATIVE_END
}

// spmv(handle, x [K], out [M] | None, out_dtype) -> y = A x
PyObject* spmv(PyObject*, PyObject* const* a, Py_ssize_t n) {
  NATIVE_BEGIN
  if (n != 4) throw torch::TypeError("spmv takes 4 arguments");
  Packed* pk = packed_of(a[0]);
  at::Tensor x = cuda_tensor(a[1], "x");
  const c10::Device dev = x.device();
  const int es = elem_bytes(pk->kind);
  if (dev.index() != pk->device) fail("A and x are on different devices");
  if (x.dim() != 1 || x.size(0) != pk->K || x.element_size() != es) fail("x must be a vector of K elements of A's type");
  c10::cuda::OptionalCUDAGuard guard;
  if (c10::cuda::current_device() != dev.index()) guard.set_device(dev);
  if (x.stride(0) != 1 || (reinterpret_cast<uintptr_t>(x.const_data_ptr()) & 15u) != 0) x = x.clone(at::MemoryFormat::Contiguous);
  at::Tensor out = none(a[2]) ? new_cuda({pk->M}, reinterpret_cast<THPDtype*>(a[3])->scalar_type, dev) : cuda_tensor(a[2], "out");
  if (out.dim() != 1 || out.size(0) != pk->M || out.stride(0) != 1) fail("out must be a contiguous vector of M elements");
  if (out.device() != dev) fail("out and x are on different devices");
  void_spmm_args s = pk->args;
  s.scale_mode = VOID_SCALE_ROW_MEAN;
  s.b = x.const_data_ptr();
  s.ldb = (pk->K * es + 15) / 16 * 16;
  s.N = 1;
  s.b_scale = 1.0f;
  s.out = out.data_ptr();
  s.ldc = pk->M;
  s.out_dtype = out_code(out.scalar_type());
  s.transposed = 1;
  s.flags = pk->stable ? 4 : 0;
  check(void_spmm_fp(&s, pk->kind, launch_stream(pk)), "void_spmm_fp");
  if (!none(a[2])) {
    Py_INCREF(a[2]);
    return a[2];
  }
  return THPVariable_Wrap(out);
  NATIVE_END
}

// ------------------------------------------------------------------------------------------ quantisers
// quant_cols(b, kind) -> (q [K, N], scale [N], scale_inv [N] | None): per-column INT8 or E4M3 of a matrix
PyObject* quant_cols(PyObject*, PyObject* const* a, Py_ssize_t n) {
  NATIVE_BEGIN
  if (n != 2) throw torch::TypeError("quant_cols takes 2 arguments");
  const at::Tensor& in = cuda_tensor(a[0], "b");
  const int kind = (int)integer(a[1]);
  if (in.dim() != 2) fail("quantising columns needs a matrix");
  const c10::Device dev = in.device();
  c10::cuda::OptionalCUDAGuard guard;
  if (c10::cuda::current_device() != dev.index()) guard.set_device(dev);
  at::Tensor b = in.scalar_type() == at::kFloat ? in : in.to(at::kFloat);
  if (!b.is_contiguous()) b = b.contiguous();
  const int64_t K = b.size(0), N = b.size(1), ld = N % 16 == 0 ? N : padded_pitch(N, 1);
  const bool i8 = kind == VOID_KIND_I8;
  at::Tensor q = new_cuda({K, ld}, i8 ? at::kChar : at::kFloat8_e4m3fn, dev);
  at::Tensor scale = new_cuda({N}, at::kFloat, dev);
  at::Tensor inv;
  if (!i8) inv = new_cuda({N}, at::kFloat, dev);
  check(void_quant_cols(b.const_data_ptr<float>(), b.stride(0), (int32_t)K, (int32_t)N, kind, q.data_ptr(), ld,
                        scale.data_ptr<float>(), i8 ? nullptr : inv.data_ptr<float>(), stream_of(dev.index())),
        "void_quant_cols");
  if (ld != N) q = q.narrow(1, 0, N);
  PyObject* res = PyTuple_New(3);
  if (res == nullptr) return nullptr;
  PyTuple_SET_ITEM(res, 0, THPVariable_Wrap(q));
  PyTuple_SET_ITEM(res, 1, THPVariable_Wrap(scale));
  if (i8) {
    Py_INCREF(Py_None);
    PyTuple_SET_ITEM(res, 2, Py_None);
  } else {
    PyTuple_SET_ITEM(res, 2, THPVariable_Wrap(inv));
  }
  return res;
  NATIVE_END
}

// ------------------------------------------------------------------------------------------ set-up of a tensor
// Waits for the stream with the interpreter free to run other threads.
void wait_for(void_stream_t st) {
  cudaError_t rc;
  Py_BEGIN_ALLOW_THREADS
  rc = cudaStreamSynchronize(reinterpret_cast<cudaStream_t>(st));
  Py_END_ALLOW_THREADS
  if (rc != cudaSuccess) throw std::runtime_error(std::string("CUDA error: ") + cudaGetErrorString(rc));
}
bool capturing(void_stream_t st) {
  if (st == nullptr) return false;   // the legacy default stream is never captured; asking costs 0.3 us
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  return cudaStreamIsCapturing(reinterpret_cast<cudaStream_t>(st), &status) == cudaSuccess && status != cudaStreamCaptureStatusNone;
}
// launch_key(device) -> the current stream, as a key for what belongs to one stream; -1 while it is being captured
PyObject* launch_key(PyObject*, PyObject* const* a, Py_ssize_t n) {
  NATIVE_BEGIN
  if (n != 1) throw torch::TypeError("launch_key takes 1 argument");
  const void_stream_t st = stream_of((c10::DeviceIndex)integer(a[0]));
  return PyLong_FromLongLong(capturing(st) ? -1 : (long long)reinterpret_cast<intptr_t>(st));
  NATIVE_END
}
// zeroed_words(n, device) -> int32 [n], zero before the call returns, whatever the current stream is capturing: it is
// allocated and cleared on another stream
PyObject* zeroed_words(PyObject*, PyObject* const* a, Py_ssize_t n) {
  NATIVE_BEGIN
  if (n != 2) throw torch::TypeError("zeroed_words takes 2 arguments");
  const int64_t words = integer(a[0]);
  const c10::Device dev(c10::kCUDA, (c10::DeviceIndex)integer(a[1]));
  c10::cuda::CUDAStream side = c10::cuda::getStreamFromPool(false, dev.index());
  for (int i = 0; i < 64 && capturing(side.stream()); ++i) side = c10::cuda::getStreamFromPool(false, dev.index());
  const c10::cuda::CUDAStreamGuard on_side(side);
  const c10::cuda::CUDAStreamCaptureModeGuard relaxed(cudaStreamCaptureModeRelaxed);
  const at::Tensor t = new_cuda({words}, at::kInt, dev);
  if (cudaMemsetAsync(t.data_ptr(), 0, (size_t)words * 4, side.stream()) != cudaSuccess || cudaStreamSynchronize(side.stream()) != cudaSuccess)
    throw std::runtime_error("CUDA error: clearing scratch memory failed");
  return THPVariable_Wrap(t);
  NATIVE_END
}
// Host memory the GPU writes a few integers to (the caching host allocator hands the same block out again).
at::Tensor host_words(int64_t n) {
  return at::empty({n}, at::TensorOptions().dtype(at::kLong).pinned_memory(true));
}
at::Tensor as_index(PyObject* o, const char* what) {
  const at::Tensor& t = cuda_tensor(o, what);
  return as_type(t, at::kInt).contiguous();
}
PyObject* pack_tuple(std::initializer_list<at::Tensor> ts) {
  PyObject* res = PyTuple_New((Py_ssize_t)ts.size());
  if (res == nullptr) throw python_error();
  Py_ssize_t i = 0;
  for (const at::Tensor& t : ts) {
    if (t.defined()) {
      PyTuple_SET_ITEM(res, i++, THPVariable_Wrap(t));
    } else {
      Py_INCREF(Py_None);
      PyTuple_SET_ITEM(res, i++, Py_None);
    }
  }
  return res;
}

// dense_build(matrix, threshold) -> (values, block_rows, block_cols, morton_codes, n_blocks, nonzeros)
PyObject* dense_build(PyObject*, PyObject* const* a, Py_ssize_t n) {
  NATIVE_BEGIN
  if (n != 2) throw torch::TypeError("dense_build takes 2 arguments");
  const at::Tensor& in = cuda_tensor(a[0], "matrix");
  const float threshold = (float)real(a[1]);
  const c10::Device dev = in.device();
  c10::cuda::OptionalCUDAGuard guard(dev);
  const int64_t M = in.size(0), N = in.size(1);
  const at::Tensor m = (N == 0 || (in.stride(1) == 1 && in.stride(0) >= N)) ? in : in.contiguous();
  const int elem = out_code(m.scalar_type());
  const int64_t ld = M > 1 ? m.stride(0) : std::max<int64_t>(N, 1);
  const int32_t nbr = (int32_t)((M + 31) / 32), nbc = (int32_t)((N + 31) / 32);
  const size_t ws_bytes = void_format_ws_bytes(nbr, nbc);
  if (ws_bytes == 0)
    fail("block grid " + std::to_string(nbr) + " x " + std::to_string(nbc) + " is too large for the device format builder");
  const void_stream_t st = stream_of(dev.index());
  const at::Tensor ws = new_cuda({(int64_t)ws_bytes}, at::kByte, dev);
  const at::Tensor counts = host_words(2);
  check(void_dense_mark(m.const_data_ptr(), elem, ld, (int32_t)M, (int32_t)N, threshold, ws.data_ptr(), ws_bytes,
                        counts.data_ptr<int64_t>(), st),
        "void_dense_mark");
  wait_for(st);   // the one synchronisation, like .nonzero(): the outputs' sizes
  const int64_t kept = counts.data_ptr<int64_t>()[0], nonzeros = counts.data_ptr<int64_t>()[1];
  at::Tensor values = new_cuda({kept, 32, 32}, m.scalar_type(), dev);
  at::Tensor rows = new_cuda({kept}, at::kInt, dev), cols = new_cuda({kept}, at::kInt, dev);
  at::Tensor codes = new_cuda({kept}, at::kLong, dev);
  check(void_dense_emit(ws.const_data_ptr(), m.const_data_ptr(), elem, ld, (int32_t)M, (int32_t)N, kept, rows.data_ptr<int32_t>(),
                        cols.data_ptr<int32_t>(), codes.data_ptr<int64_t>(), values.data_ptr(), st),
        "void_dense_emit");
  return Py_BuildValue("NNNNLL", THPVariable_Wrap(values), THPVariable_Wrap(rows), THPVariable_Wrap(cols), THPVariable_Wrap(codes),
                       (long long)kept, (long long)nonzeros);
  NATIVE_END
}

// quant_tiles_i8(values [n, 32, 32], block_rows, block_cols) -> (q, scales, zero_points, block_rows copy, block_cols copy)
PyObject* quant_tiles_i8(PyObject*, PyObject* const* a, Py_ssize_t n) {
  NATIVE_BEGIN
  if (n != 3) throw torch::TypeError("quant_tiles_i8 takes 3 arguments");
  const at::Tensor& in = cuda_tensor(a[0], "values");
  const c10::Device dev = in.device();
  c10::cuda::OptionalCUDAGuard guard(dev);
  const at::ScalarType t = in.scalar_type();
  at::Tensor v = (t == at::kFloat || t == at::kHalf || t == at::kBFloat16 ? in : in.to(at::kFloat)).contiguous();
  if ((reinterpret_cast<uintptr_t>(v.const_data_ptr()) & 15u) != 0) v = v.clone();   // the kernel loads 16 bytes at a time
  const int64_t count = v.size(0);
  if (v.dim() != 3 || v.numel() != count * 1024) fail("void_b200 kernels are built for 32x32 tiles");
  at::Tensor q = new_cuda(v.sizes(), at::kChar, dev), scales = new_cuda({count}, at::kFloat, dev);
  at::Tensor zeros = new_cuda({count}, at::kChar, dev);
  at::Tensor copy[2];
  const int32_t* from[2] = {nullptr, nullptr};
  int32_t* to[2] = {nullptr, nullptr};
  for (int i = 0; i < 2; ++i) {
    const at::Tensor& c = tensor(a[1 + i], "block coordinates");
    if (c.scalar_type() == at::kInt && c.is_contiguous() && c.device() == dev && c.numel() == count) {
      copy[i] = new_cuda(c.sizes(), at::kInt, dev);
      from[i] = c.const_data_ptr<int32_t>();
      to[i] = copy[i].data_ptr<int32_t>();
    } else {
      copy[i] = c.clone();
    }
  }
  check(void_quant_tiles(v.const_data_ptr(), out_code(v.scalar_type()), count, VOID_KIND_I8, q.data_ptr(), scales.data_ptr<float>(),
                         nullptr, nullptr, zeros.data_ptr<int8_t>(), from[0], from[1], to[0], to[1], stream_of(dev.index())),
        "void_quant_tiles");
  return pack_tuple({q, scales, zeros, copy[0], copy[1]});
  NATIVE_END
}

// A tile list names every stored tile once; kernels read as many coordinates as there are tiles.
void check_list(const at::Tensor& rows, const at::Tensor& cols, int64_t tiles) {
  TORCH_CHECK_VALUE(rows.numel() == tiles && cols.numel() == tiles, "invalid VOID tile list: ", rows.numel(), " block rows and ",
                    cols.numel(), " block columns for ", tiles, " tiles");
}
void check_index(const at::Tensor& row_ptr, const at::Tensor& block_indices, int64_t nbr, int64_t tiles) {
  TORCH_CHECK_VALUE(row_ptr.is_cuda() && block_indices.is_cuda() && row_ptr.scalar_type() == at::kInt && block_indices.scalar_type() == at::kInt &&
                        row_ptr.is_contiguous() && block_indices.is_contiguous() && row_ptr.numel() == nbr + 1 && block_indices.numel() == tiles,
                    "invalid VOID tile index: it does not belong to ", tiles, " tiles in ", nbr, " tile rows");
}
constexpr int32_t kMaxOrderRows = 4096;   // tile rows that are put in order by comparing all pairs
// order: null, or the tile rows by falling tile count (left undefined for more rows than that)
void build_index(const at::Tensor& rows, const at::Tensor& cols, int32_t nbr, int32_t nbc, at::Tensor& row_ptr, at::Tensor& block_indices,
                 at::Tensor* order, void_stream_t st) {
  const c10::Device dev = rows.device();
  const int64_t count = rows.numel();
  row_ptr = new_cuda({nbr + 1}, at::kInt, dev);
  block_indices = new_cuda({count}, at::kInt, dev);
  const size_t ws_bytes = void_tile_index_ws_bytes(nbr, nbc);
  const at::Tensor ws = new_cuda({(int64_t)ws_bytes}, at::kByte, dev);
  const int32_t *r = rows.const_data_ptr<int32_t>(), *c = cols.const_data_ptr<int32_t>();
  if (order != nullptr && nbr > 0 && nbr <= kMaxOrderRows) {
    *order = new_cuda({nbr}, at::kInt, dev);
    check(void_build_tile_index_order(r, c, count, nbr, nbc, row_ptr.data_ptr<int32_t>(), block_indices.data_ptr<int32_t>(),
                                      order->data_ptr<int32_t>(), ws.data_ptr(), ws_bytes, st),
          "void_build_tile_index_order");
  } else {
    check(void_build_tile_index(r, c, count, nbr, nbc, row_ptr.data_ptr<int32_t>(), block_indices.data_ptr<int32_t>(), ws.data_ptr(),
                                ws_bytes, st),
          "void_build_tile_index");
  }
}
// Waits for the index and reads how many tiles it holds: one read of one integer per built index.
long long indexed_tiles(const at::Tensor& row_ptr, int32_t nbr, void_stream_t st) {
  const at::Tensor last = host_words(1);
  if (cudaMemcpyAsync(last.data_ptr(), row_ptr.const_data_ptr<int32_t>() + nbr, 4, cudaMemcpyDeviceToHost,
                      reinterpret_cast<cudaStream_t>(st)) != cudaSuccess)
    throw std::runtime_error("CUDA error: reading the tile index failed");
  wait_for(st);
  return *static_cast<const int32_t*>(last.data_ptr());
}

// tile_index(block_rows, block_cols, nbr, nbc) -> (row_ptr, block_indices, indexed tiles)
PyObject* tile_index(PyObject*, PyObject* const* a, Py_ssize_t n) {
  NATIVE_BEGIN
  if (n != 4) throw torch::TypeError("tile_index takes 4 arguments");
  const at::Tensor rows = as_index(a[0], "block_rows"), cols = as_index(a[1], "block_cols");
  c10::cuda::OptionalCUDAGuard guard(rows.device());
  const void_stream_t st = stream_of(rows.device().index());
  const int32_t nbr = (int32_t)integer(a[2]), nbc = (int32_t)integer(a[3]);
  check_list(rows, cols, rows.numel());
  at::Tensor row_ptr, block_indices;
  build_index(rows, cols, nbr, nbc, row_ptr, block_indices, nullptr, st);
  const long long indexed = indexed_tiles(row_ptr, nbr, st);
  return Py_BuildValue("NNL", THPVariable_Wrap(row_ptr), THPVariable_Wrap(block_indices), indexed);
  NATIVE_END
}

// pack_store(values, scales | None, block_rows, block_cols, M, K, kind, terms, row_ptr | None, block_indices | None)
//   -> (tiles, tile_cols, tile_scales, row_ptr, block_indices, row_scale, row_order, home): row_order where it came with the
//   index, else None; home is the stream all of them were allocated on, None with an index that was given
// The packed store of a tensor, its tile index built on the way when it is not given.  The caller waits for it
// and checks the index (finish_store); until then a list that is not valid is packed without leaving its arrays.
PyObject* pack_store(PyObject*, PyObject* const* a, Py_ssize_t n) {
  NATIVE_BEGIN
  if (n != 10) throw torch::TypeError("pack_store takes 10 arguments");
  const at::Tensor values = cuda_tensor(a[0], "values").contiguous();
  const at::Tensor rows = as_index(a[2], "block_rows"), cols = as_index(a[3], "block_cols");
  const c10::Device dev = values.device();
  c10::cuda::OptionalCUDAGuard guard(dev);
  const void_stream_t st = stream_of(dev.index());
  const int64_t M = integer(a[4]), K = integer(a[5]), count = values.size(0);
  const int kind = (int)integer(a[6]), terms = (int)integer(a[7]), es = elem_bytes(kind);
  const int32_t nbr = (int32_t)((M + 31) / 32), nbc = (int32_t)((K + 31) / 32);
  check_list(rows, cols, count);
  at::Tensor row_ptr, block_indices, order, scales;
  if (none(a[8]) || none(a[9])) {
    build_index(rows, cols, nbr, nbc, row_ptr, block_indices, &order, st);
  } else {
    row_ptr = tensor(a[8], "row_ptr");
    block_indices = tensor(a[9], "block_indices");
    check_index(row_ptr, block_indices, nbr, count);
  }
  if (!none(a[1])) scales = as_type(tensor(a[1], "scales"), at::kFloat).contiguous();
  const float* sc = scales.defined() ? scales.const_data_ptr<float>() : nullptr;
  const int64_t n_sc = scales.defined() ? scales.numel() : 0;
  const int64_t room = std::max<int64_t>(count, 1);
  const at::Tensor raw = new_cuda({room * 1024 * es * terms + 1024}, at::kByte, dev);
  const int64_t off = -reinterpret_cast<intptr_t>(raw.data_ptr()) & 1023;   // tiles start on a 1024-byte boundary
  const at::Tensor tiles = raw.narrow(0, off, room * 1024 * es * terms);
  const at::Tensor tile_cols = new_cuda({room}, at::kInt, dev), tile_scales = new_cuda({room}, at::kFloat, dev);
  const at::Tensor row_scale = new_cuda({std::max<int64_t>(nbr, 1)}, at::kFloat, dev);
  const int32_t *rp = row_ptr.const_data_ptr<int32_t>(), *bi = block_indices.const_data_ptr<int32_t>();
  const int32_t *br = rows.const_data_ptr<int32_t>(), *bc = cols.const_data_ptr<int32_t>();
  int32_t* tc = tile_cols.data_ptr<int32_t>();
  float *ts = tile_scales.data_ptr<float>(), *rs = row_scale.data_ptr<float>();
  if (es > 1)
    check(void_pack_tiles_fp(values.const_data_ptr(), es, bc, bi, count, tiles.data_ptr(), tc, st), "void_pack_tiles_fp");
  else if (terms > 1)
    check(void_pack_tiles_f8_split(values.const_data_ptr(), sc, n_sc, br, bc, bi, rp, count, nbr, terms, tiles.data_ptr(), tc, ts, rs, st),
          "void_pack_tiles_f8_split");
  else
    check(void_pack_tiles(values.const_data_ptr(), sc, n_sc, bc, bi, rp, count, nbr, tiles.data_ptr(), tc, ts, rs, st), "void_pack_tiles");
  PyObject* home = Py_None;
  if (none(a[8]) || none(a[9])) home = PyLong_FromLongLong((long long)reinterpret_cast<intptr_t>(st));
  else Py_INCREF(home);
  PyObject* by_length = Py_None;
  if (order.defined()) by_length = THPVariable_Wrap(order);
  else Py_INCREF(by_length);
  return Py_BuildValue("NNNNNNNN", THPVariable_Wrap(tiles), THPVariable_Wrap(tile_cols), THPVariable_Wrap(tile_scales), THPVariable_Wrap(row_ptr),
                       THPVariable_Wrap(block_indices), THPVariable_Wrap(row_scale), by_length, home);
  NATIVE_END
}

// finish_store(row_ptr, nbr, row_order | None) -> (row_order, indexed tiles | None): the order of the tile rows, unless there is
// one, then - outside a stream capture, where nothing can be waited for - the wait until the store is complete and the size of
// its index
PyObject* finish_store(PyObject*, PyObject* const* a, Py_ssize_t n) {
  NATIVE_BEGIN
  if (n != 3) throw torch::TypeError("finish_store takes 3 arguments");
  const at::Tensor& row_ptr = cuda_tensor(a[0], "row_ptr");
  const int32_t nbr = (int32_t)integer(a[1]);
  const c10::Device dev = row_ptr.device();
  c10::cuda::OptionalCUDAGuard guard(dev);
  const void_stream_t st = stream_of(dev.index());
  at::Tensor order;
  if (!none(a[2])) {
    order = cuda_tensor(a[2], "row_order");
  } else if (nbr > 0 && nbr <= kMaxOrderRows) {
    order = new_cuda({nbr}, at::kInt, dev);
    check(void_row_order(row_ptr.const_data_ptr<int32_t>(), nbr, order.data_ptr<int32_t>(), st), "void_row_order");
  } else if (nbr > 0) {   // beyond a few thousand rows a sort does less work than comparing all pairs
    order = at::argsort(row_ptr.narrow(0, 1, nbr) - row_ptr.narrow(0, 0, nbr), /*stable=*/true, 0, /*descending=*/true).to(at::kInt);
  }
  PyObject* o = Py_None;
  if (order.defined()) o = THPVariable_Wrap(order);
  else Py_INCREF(o);
  if (capturing(st)) return Py_BuildValue("NO", o, Py_None);
  return Py_BuildValue("NL", o, indexed_tiles(row_ptr, nbr, st));
  NATIVE_END
}

// ------------------------------------------------------------------------------------------ training
// The index arrays of one sparsity structure, both ways round; they outlive the values that train over them.
struct Structure {
  at::Tensor row_ptr[2], block_indices[2], tile_cols[2], row_order[2];   // of A, of A^T
  at::Tensor items, status;
  int64_t M = 0, K = 0, nnz = 0;
  mutable Readers readers;
  mutable std::atomic<bool> captured{false};   // a graph reads these arrays
};
struct StructureObject {
  PyObject_HEAD
  std::shared_ptr<const Structure> st;
};
PyTypeObject* g_structure_type = nullptr;

// structure(row_ptr, block_indices, tile_cols, row_ptr_t, block_indices_t, tile_cols_t, items, status, M, K, n_blocks,
//           row_order | None, row_order_t | None)
PyObject* structure(PyObject*, PyObject* const* a, Py_ssize_t n) {
  NATIVE_BEGIN
  if (n != 13) throw torch::TypeError("structure takes 13 arguments");
  auto st = std::make_shared<Structure>();
  for (int i = 0; i < 2; ++i) {
    st->row_ptr[i] = cuda_tensor(a[3 * i], "row_ptr");
    st->block_indices[i] = cuda_tensor(a[3 * i + 1], "block_indices");
    st->tile_cols[i] = cuda_tensor(a[3 * i + 2], "tile_cols");
    if (!none(a[11 + i])) st->row_order[i] = cuda_tensor(a[11 + i], "row_order");
  }
  st->items = cuda_tensor(a[6], "items");
  st->status = cuda_tensor(a[7], "status");
  st->M = integer(a[8]);
  st->K = integer(a[9]);
  st->nnz = integer(a[10]);
  check_index(st->row_ptr[0], st->block_indices[0], (st->M + 31) / 32, st->nnz);
  check_index(st->row_ptr[1], st->block_indices[1], (st->K + 31) / 32, st->nnz);
  PyObject* self = PyType_GenericAlloc(g_structure_type, 0);
  if (self == nullptr) return nullptr;
  new (&reinterpret_cast<StructureObject*>(self)->st) std::shared_ptr<const Structure>(std::move(st));
  return self;
  NATIVE_END
}
void_stream_t launch_stream(const Structure& st, c10::Device dev) {
  const c10::cuda::CUDAStream stream = c10::cuda::getCurrentCUDAStream(dev.index());
  st.readers.add(stream, {&st.row_ptr[0], &st.row_ptr[1], &st.block_indices[0], &st.block_indices[1], &st.tile_cols[0], &st.tile_cols[1],
                          &st.row_order[0], &st.row_order[1], &st.items});
  if (capturing(stream.stream())) st.captured.store(true, std::memory_order_relaxed);
  return stream.stream();
}
std::shared_ptr<const Structure> structure_of(PyObject* o) {
  if (Py_TYPE(o) != g_structure_type) throw torch::TypeError("expected a structure handle");
  return reinterpret_cast<StructureObject*>(o)->st;
}
// structure_captured(structure) -> whether a graph reads its arrays
PyObject* structure_captured(PyObject*, PyObject* const* a, Py_ssize_t n) {
  NATIVE_BEGIN
  if (n != 1) throw torch::TypeError("structure_captured takes 1 argument");
  return PyBool_FromLong(structure_of(a[0])->captured.load(std::memory_order_relaxed));
  NATIVE_END
}
int common_kind(at::ScalarType a, at::ScalarType b) {   // their common 16-bit type, else fp32 operands (TF32)
  if (a == b && a == at::kHalf) return VOID_KIND_F16;
  if (a == b && a == at::kBFloat16) return VOID_KIND_BF16;
  return VOID_KIND_TF32;
}
at::ScalarType kind_type(int kind) { return kind == VOID_KIND_F16 ? at::kHalf : (kind == VOID_KIND_BF16 ? at::kBFloat16 : at::kFloat); }

void check_tiles(const Structure& st, const at::Tensor& values) {
  if (values.dim() != 3 || values.size(0) != st.nnz || values.size(1) != 32 || values.size(2) != 32)
    fail("the sparse matrix stores " + std::to_string(st.nnz) + " tiles of 32x32, got values of another shape");
}
// Product with tiles that change from call to call: they are packed (their transposes for A^T) and multiplied at once.
// linear: b is x [N, K] and the result x A^T [N, M]; otherwise b is [K, N] and the result A b [M, N].
at::Tensor product_of_values(const Structure& st, bool a_transposed, const at::Tensor& values_in, const at::Tensor& b_in,
                             bool linear, const at::Tensor* row_bias) {
  const c10::Device dev = b_in.device();
  const int kind = common_kind(values_in.scalar_type(), b_in.scalar_type());
  const int es = elem_bytes(kind);
  const at::Tensor values = as_type(values_in, kind_type(kind)).contiguous();
  const int64_t M = a_transposed ? st.K : st.M, K = a_transposed ? st.M : st.K;
  const int64_t N = b_in.size(linear ? 0 : 1);
  if (b_in.dim() != 2 || b_in.size(linear ? 1 : 0) != K) fail("shape mismatch between the sparse matrix and the dense operand");
  check_tiles(st, values);
  const bool copied = linear && copy_pays(kind, st.nnz, N, K);
  const at::Tensor b_typed = as_type(b_in, kind_type(kind));
  const at::Tensor b = copied ? transposed_copy(b_typed, es) : kernel_operand(b_typed, es, linear ? 0 : st.nnz * ((N + 127) / 128));
  at::Tensor out = new_cuda({linear ? N : M, linear ? M : N}, b_in.scalar_type(), dev);
  at::Tensor store = new_cuda({std::max<int64_t>(st.nnz, 1) * 1024 * es + 1024}, at::kByte, dev);
  uint8_t* tiles = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(store.data_ptr()) + 1023) & ~uintptr_t(1023));
  const void_stream_t stream = launch_stream(st, dev);
  const int way = a_transposed ? 1 : 0;
  check(void_repack_tiles_fp(values.const_data_ptr(), es, st.block_indices[way].const_data_ptr<int32_t>(), st.nnz, way, tiles, stream),
        "void_repack_tiles_fp");
  void_spmm_args s = void_spmm_args();
  s.tiles = tiles;
  s.tile_cols = st.tile_cols[way].const_data_ptr<int32_t>();
  s.row_ptr = st.row_ptr[way].const_data_ptr<int32_t>();
  if (st.row_order[way].defined()) s.row_order = st.row_order[way].const_data_ptr<int32_t>();
  s.nbr = (int32_t)((M + 31) / 32);
  s.nbc = (int32_t)((K + 31) / 32);
  s.nnz = st.nnz;
  s.b = b.const_data_ptr();
  s.ldb = row_pitch(b, es);
  s.K = (int32_t)K;
  s.N = (int32_t)N;
  s.b_scale = 1.0f;
  at::Tensor bias;
  if (row_bias != nullptr) {
    bias = row_bias->to(dev, at::kFloat).contiguous();
    if (bias.numel() != M) fail("row bias must have " + std::to_string(M) + " elements, got " + std::to_string(bias.numel()));
    s.row_bias = bias.const_data_ptr<float>();
  }
  s.out = out.data_ptr();
  s.ldc = out.stride(0);
  s.M = (int32_t)M;
  s.out_dtype = out_code(out.scalar_type());
  s.scale_mode = VOID_SCALE_ROW_MEAN;
  s.status = st.status.data_ptr<int32_t>();
  s.transposed = copied ? 2 : (linear ? 1 : 0);
  check(void_spmm_fp(&s, kind, stream), "void_spmm_fp");
  return out;
}

// dL/dA for the stored tiles; linear: g [N, M], x [N, K], otherwise g [M, N], x [K, N]
at::Tensor gradient_of_values(const Structure& st, const at::Tensor& g_in, const at::Tensor& x_in, at::ScalarType type, bool linear) {
  const c10::Device dev = x_in.device();
  const int64_t N = x_in.size(linear ? 0 : 1);
  if (g_in.dim() != 2 || x_in.dim() != 2 || g_in.size(linear ? 0 : 1) != N || g_in.size(linear ? 1 : 0) != st.M || x_in.size(linear ? 1 : 0) != st.K)
    fail("shape mismatch between the gradient, the dense operand and the sparse matrix");
  if (st.nnz == 0 || N == 0) return at::zeros({st.nnz, 32, 32}, x_in.options().dtype(type));
  const int kind = common_kind(g_in.scalar_type(), x_in.scalar_type());
  const int es = elem_bytes(kind);
  const at::Tensor g = kernel_operand(as_type(g_in, kind_type(kind)), es);
  const at::Tensor x = kernel_operand(as_type(x_in, kind_type(kind)), es);
  at::Tensor grad = new_cuda({st.nnz, 32, 32}, type, dev);   // every stored tile is written
  check((linear ? void_linear_tile_grad : void_spmm_tile_grad)(
            g.const_data_ptr(), row_pitch(g, es), x.const_data_ptr(), row_pitch(x, es), (int32_t)st.M, (int32_t)st.K, (int32_t)N,
            kind, st.items.const_data_ptr<int32_t>(), (int32_t)st.items.size(0), st.tile_cols[0].const_data_ptr<int32_t>(),
            st.block_indices[0].const_data_ptr<int32_t>(), grad.data_ptr(), out_code(type), st.status.data_ptr<int32_t>(),
            launch_stream(st, dev)),
        "void_spmm_tile_grad");
  return grad;
}

at::Tensor column_sums(const at::Tensor& m) {
  at::Tensor out = new_cuda({m.size(1)}, m.scalar_type(), m.device());
  check(void_column_sum(m.const_data_ptr(), out_code(m.scalar_type()), std::max<int64_t>(m.stride(0), m.size(1)), (int32_t)m.size(0),
                        (int32_t)m.size(1), out.data_ptr(), stream_of(m.device().index())),
        "void_column_sum");
  return out;
}

// The gradients of A b (or of x A^T + bias): an autograd node of its own, so that a backward pass runs in the engine's
// thread without taking the interpreter's lock.
struct ProductBackward : torch::autograd::Node {
  torch::autograd::SavedVariable values, dense;
  std::shared_ptr<const Structure> st;
  bool linear = false;

  std::string name() const override { return "VOIDProductBackward"; }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    values.reset_data();
    dense.reset_data();
  }
  torch::autograd::variable_list apply(torch::autograd::variable_list&& grads) override {
    std::lock_guard<std::mutex> lock(mutex_);
    torch::autograd::variable_list out(3);
    if (!grads[0].defined()) return out;
    // Unpacked with autograd on: a hook may run the user's code here, such as a checkpoint's second forward pass.
    const at::Tensor v = values.unpack(), b = dense.unpack(), g = grads[0].contiguous();
    c10::cuda::OptionalCUDAGuard guard(b.device());
    // (a backward pass that is recorded itself gets the bias gradient from an operator that can be differentiated)
    if (task_should_compute_output(2) && at::GradMode::is_enabled()) out[2] = g.sum(0);
    at::AutoDispatchBelowADInplaceOrView below;
    try {
      if (task_should_compute_output(1))
        out[1] = st->nnz ? product_of_values(*st, true, v, as_type(g, b.scalar_type()), linear, nullptr) : at::zeros_like(b);
      if (task_should_compute_output(0)) out[0] = gradient_of_values(*st, g, b, v.scalar_type(), linear);
      if (task_should_compute_output(2) && !out[2].defined()) out[2] = column_sums(g);
    } catch (const Failure& f) {
      TORCH_CHECK(false, f.text);
    }
    return out;
  }
};

// values_product(structure, values, b, linear, bias | None) -> A b, or x A^T + bias; differentiable in all three
PyObject* values_product(PyObject*, PyObject* const* a, Py_ssize_t n) {
  NATIVE_BEGIN
  if (n != 5) throw torch::TypeError("values_product takes 5 arguments");
  std::shared_ptr<const Structure> st = structure_of(a[0]);
  const at::Tensor& values = cuda_tensor(a[1], "values");
  const at::Tensor& b = cuda_tensor(a[2], "the dense operand");
  c10::cuda::OptionalCUDAGuard guard(b.device());
  const bool linear = PyObject_IsTrue(a[3]) == 1;
  const at::Tensor none_given;
  const at::Tensor& bias = none(a[4]) ? none_given : tensor(a[4], "bias");
  for (const at::Tensor* t : {&values, &b, &bias})
    TORCH_CHECK_NOT_IMPLEMENTED(!torch::autograd::isFwGradDefined(*t),
                                "the sparse product has no forward-mode derivative: an operand carries a tangent");
  at::Tensor out;
  {
    at::AutoDispatchBelowADInplaceOrView below;
    out = product_of_values(*st, false, values, b, linear, bias.defined() ? &bias : nullptr);
  }
  if (torch::autograd::compute_requires_grad(values, b, bias)) {
    auto node = std::shared_ptr<ProductBackward>(new ProductBackward(), torch::autograd::deleteNode);
    node->set_next_edges(torch::autograd::collect_next_edges(values, b, bias));
    node->values = torch::autograd::SavedVariable(values, false);
    node->dense = torch::autograd::SavedVariable(b, false);
    node->st = std::move(st);
    node->linear = linear;
    torch::autograd::set_history(out, node);
  }
  return THPVariable_Wrap(out);
  NATIVE_END
}

// tile_gradient(structure, grad, b, linear, dtype) -> dL/dA_values
PyObject* tile_gradient(PyObject*, PyObject* const* a, Py_ssize_t n) {
  NATIVE_BEGIN
  if (n != 5) throw torch::TypeError("tile_gradient takes 5 arguments");
  const std::shared_ptr<const Structure> st = structure_of(a[0]);
  const at::Tensor& b = cuda_tensor(a[2], "the dense operand");
  c10::cuda::OptionalCUDAGuard guard(b.device());
  at::AutoDispatchBelowADInplaceOrView below;
  return THPVariable_Wrap(gradient_of_values(*st, cuda_tensor(a[1], "the gradient"), b, reinterpret_cast<THPDtype*>(a[4])->scalar_type,
                                             PyObject_IsTrue(a[3]) == 1));
  NATIVE_END
}

PyObject* set_error(PyObject*, PyObject* cls) {
  Py_INCREF(cls);
  g_error = cls;
  Py_RETURN_NONE;
}

#define FAST(name) {#name, (PyCFunction)(void (*)(void))name, METH_FASTCALL, nullptr}
PyMethodDef kMethods[] = {
    {"set_error", set_error, METH_O, nullptr},
    FAST(packed_handle),
    FAST(packed_made_from),
    FAST(packed_is_current),
    FAST(packed_captured),
    FAST(packed_grouped),
    FAST(identity),
    FAST(launch_key),
    FAST(zeroed_words),
    FAST(unchanged),
    FAST(spmm),
    FAST(spmv),
    FAST(mlp),
    FAST(mlp_packed),
    FAST(quant_cols),
    FAST(dense_build),
    FAST(quant_tiles_i8),
    FAST(tile_index),
    FAST(pack_store),
    FAST(finish_store),
    FAST(structure),
    FAST(structure_captured),
    FAST(values_product),
    FAST(tile_gradient),
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

void packed_dealloc(PyObject* self) {
  delete reinterpret_cast<PackedObject*>(self)->packed;
  PyTypeObject* type = Py_TYPE(self);
  type->tp_free(self);
  Py_DECREF(type);
}
void structure_dealloc(PyObject* self) {
  PyTypeObject* type = Py_TYPE(self);
  reinterpret_cast<StructureObject*>(self)->st.~shared_ptr();
  type->tp_free(self);
  Py_DECREF(type);
}
PyType_Slot kStructureSlots[] = {{Py_tp_dealloc, (void*)structure_dealloc}, {0, nullptr}};
PyType_Spec kStructureSpec = {"_native.Structure", (int)sizeof(StructureObject), 0, Py_TPFLAGS_DEFAULT, kStructureSlots};
PyType_Slot kPackedSlots[] = {{Py_tp_dealloc, (void*)packed_dealloc}, {0, nullptr}};
PyType_Spec kPackedSpec = {"_native.Packed", (int)sizeof(PackedObject), 0, Py_TPFLAGS_DEFAULT, kPackedSlots};

}  // namespace

PyMODINIT_FUNC PyInit__native(void) {
  g_packed_type = reinterpret_cast<PyTypeObject*>(PyType_FromSpec(&kPackedSpec));
  g_structure_type = reinterpret_cast<PyTypeObject*>(PyType_FromSpec(&kStructureSpec));
  if (g_packed_type == nullptr || g_structure_type == nullptr) return nullptr;
  return PyModule_Create(&kModule);
}
