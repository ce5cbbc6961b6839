// Native host path of the Python operators: argument checks, output and scratch allocation, the
// parameter block and the launch of one attention call, as a CPython extension over the C ABI of
// include/fa4_nvfp4.h.
//
// Why it exists: a decode step is 5-10 us of GPU time, and the same checks, attribute reads and
// ctypes assignments written in Python took 35-60 us per call (B200, 76 us per pass of a
// one-token call with linear scales), so the GPU waited for the host.  Here they take 5-8 us.
//
// The functions take their arguments positionally (METH_FASTCALL); interface.py and varlen.py own
// the signatures, defaults and documentation.  Each reads its Python arguments into plain values first and
// then works without the interpreter lock: allocations, launches, reads of a value that is still on the
// device and copies of pageable memory may all wait for the GPU, and other Python threads run meanwhile.
// Error types and messages are those of the reference's host code (flash_attn/cute/interface.py:231-236,
// 384-398): AssertionError for malformed tensors, NotImplementedError for what is not built, ValueError
// for bad numbers.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/CachingHostAllocator.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Device.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <memory>
#include <mutex>
#include <string>
#include <utility>
#include <vector>

#include "../../include/fa4_nvfp4.h"

namespace {

// What travels to the boundary: a Python exception that has been set; one to be set there (thrown with or
// without the interpreter lock); a return code of the C ABI.
struct PyErrorSet {};
struct Failure {
  PyObject* type;       // a built-in exception type
  std::string message;
};
struct CallFailed {
  int rc;
  const char* what;
};

[[noreturn]] __attribute__((format(printf, 2, 3))) void fail(PyObject* type, const char* fmt, ...) {
  char msg[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(msg, sizeof msg, fmt, ap);
  va_end(ap);
  throw Failure{type, msg};
}
void check_rc(int rc, const char* what) {
  if (rc != 0) throw CallFailed{rc, what};
}

// The calling thread without the interpreter lock.  No Python object is touched while one is alive.
class NoGil {
 public:
  NoGil() : state_(PyEval_SaveThread()) {}
  ~NoGil() { PyEval_RestoreThread(state_); }
  NoGil(const NoGil&) = delete;
  NoGil& operator=(const NoGil&) = delete;

 private:
  PyThreadState* state_;
};
#define FA4_ASSERT(cond, ...) \
  do { if (!(cond)) fail(PyExc_AssertionError, __VA_ARGS__); } while (0)

std::string dims_of(at::IntArrayRef s) {
  std::string r = "(";
  for (size_t i = 0; i < s.size(); ++i) r += (i ? ", " : "") + std::to_string(s[i]);
  return r + ")";
}

const at::Tensor& tensor_of(PyObject* o, const char* name) {
  if (!THPVariable_Check(o)) fail(PyExc_TypeError, "%s must be a torch.Tensor, got %s", name, Py_TYPE(o)->tp_name);
  return THPVariable_Unpack(o);
}
bool is_none(PyObject* o) { return o == nullptr || o == Py_None; }
at::Tensor optional_tensor(PyObject* o, const char* name) { return is_none(o) ? at::Tensor() : tensor_of(o, name); }

// packed bytes arrive as uint8, float8_e4m3fn or float4_e2m1fn_x2
at::Tensor as_u8(PyObject* o, const char* name) {
  const at::Tensor& t = tensor_of(o, name);
  const auto st = t.scalar_type();
  if (st == at::kByte) return t;
  if (st == at::ScalarType::Float8_e4m3fn || st == at::ScalarType::Float4_e2m1fn_x2) return t.view(at::kByte);
  fail(PyExc_AssertionError, "%s must be uint8 / float8_e4m3fn / float4_e2m1fn_x2, got %s", name,
       c10::toString(st));
}

void validate(const at::Tensor& t, const char* name, at::IntArrayRef shape, at::ScalarType dtype,
              const at::Device& device) {
  FA4_ASSERT(t.sizes() == shape, "%s shape %s != expected %s", name, dims_of(t.sizes()).c_str(), dims_of(shape).c_str());
  FA4_ASSERT(t.scalar_type() == dtype, "%s dtype %s != expected %s", name, c10::toString(t.scalar_type()),
             c10::toString(dtype));
  FA4_ASSERT(t.device() == device, "%s device %s != expected %s", name, t.device().str().c_str(), device.str().c_str());
  FA4_ASSERT(t.is_cuda(), "%s must be on CUDA", name);
}

at::Tensor inner_contiguous(at::Tensor t) { return t.stride(-1) == 1 ? t : t.contiguous(); }

double number_of(PyObject* o) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) throw PyErrorSet();
  return v;
}
long integer_of(PyObject* o) {
  PyObject* n = PyNumber_Long(o);
  if (n == nullptr) throw PyErrorSet();
  const long v = PyLong_AsLong(n);
  Py_DECREF(n);
  if (v == -1 && PyErr_Occurred()) throw PyErrorSet();
  return v;
}
bool truth_of(PyObject* o) {
  if (o == Py_True) return true;
  if (o == Py_False) return false;
  const int v = PyObject_IsTrue(o);
  if (v < 0) throw PyErrorSet();
  return v != 0;
}
// ---- per-tensor scales that are still on their way ------------------------------------------------
// What quantize_qkv hands out for a scale: the quantiser leaves it on the device, and an attention call
// on the quantiser's stream reads it there, so quantising and attending never wait on the host.
// float(scale) copies all three back and waits for the stream, once; calls after that take the values.
struct ScaleState {
  c10::DataPtr device;              // three floats
  cudaStream_t stream;
  std::atomic<bool> known{false};
  std::mutex fetching;
  float value[3];
  const float* ptr(int i) const { return static_cast<const float*>(device.get()) + i; }
  void fetch() {                    // without the interpreter lock
    if (known) return;
    std::lock_guard<std::mutex> lock(fetching);
    if (known) return;
    c10::cuda::CUDAGuard guard(device.device().index());
    // another stream may be capturing (a call outside of this one's stream takes the values)
    c10::cuda::CUDAStreamCaptureModeGuard relaxed(cudaStreamCaptureModeRelaxed);
    float v[3];
    C10_CUDA_CHECK(cudaMemcpyAsync(v, device.get(), sizeof v, cudaMemcpyDeviceToHost, stream));
    C10_CUDA_CHECK(cudaStreamSynchronize(stream));
    std::copy_n(v, 3, value);
    known = true;
  }
};
struct LazyScale {
  PyObject_HEAD
  std::shared_ptr<ScaleState>* state;
  int which;
};
PyObject* lazy_float(PyObject* self) {
  HANDLE_TH_ERRORS
  const std::shared_ptr<ScaleState> state = *reinterpret_cast<LazyScale*>(self)->state;
  if (!state->known) {
    NoGil nogil;
    state->fetch();
  }
  return PyFloat_FromDouble(state->value[reinterpret_cast<LazyScale*>(self)->which]);
  END_HANDLE_TH_ERRORS
}
void lazy_dealloc(PyObject* self) {
  delete reinterpret_cast<LazyScale*>(self)->state;
  Py_TYPE(self)->tp_free(self);
}
PyNumberMethods lazy_number = {};
PyTypeObject lazy_type = {PyVarObject_HEAD_INIT(nullptr, 0)};
bool is_lazy(PyObject* o) { return Py_TYPE(o) == &lazy_type; }
PyObject* new_lazy(const std::shared_ptr<ScaleState>& st, int which) {
  PyObject* o = lazy_type.tp_alloc(&lazy_type, 0);
  if (o == nullptr) throw PyErrorSet();
  reinterpret_cast<LazyScale*>(o)->state = new std::shared_ptr<ScaleState>(st);
  reinterpret_cast<LazyScale*>(o)->which = which;
  return o;
}
// A per-tensor scale as it was passed: a number, a one-element tensor, or one on its way.
struct Scale {
  double number = 0.0;
  at::Tensor tensor;
  std::shared_ptr<ScaleState> lazy;
  int which = 0;
  // its value (waits for one that lives on the device)
  float value(const char* name) const {
    if (lazy) {
      lazy->fetch();
      return lazy->value[which];
    }
    if (!tensor.defined()) return static_cast<float>(number);
    FA4_ASSERT(tensor.numel() == 1, "%s must be a python float or a 1-element tensor", name);
    return static_cast<float>(tensor.item<double>());
  }
};
Scale scale_of(PyObject* o) {
  Scale s;
  if (is_lazy(o)) {
    s.lazy = *reinterpret_cast<LazyScale*>(o)->state;
    s.which = reinterpret_cast<LazyScale*>(o)->which;
  } else if (THPVariable_Check(o)) {
    s.tensor = THPVariable_Unpack(o);
  } else {
    s.number = number_of(o);
  }
  return s;
}
// The device copies of three scales for a call on `stream`; false: take their values instead (they are known,
// or have to be fetched).
bool device_scales(const Scale (&s)[3], const at::Device& device, cudaStream_t stream, const float** ptr) {
  for (int i = 0; i < 3; ++i) {
    if (!s[i].lazy || s[i].lazy->known || s[i].lazy->stream != stream || s[i].lazy->device.device() != device) return false;
    ptr[i] = s[i].lazy->ptr(s[i].which);
  }
  return true;
}

// The status word of a device (see DeviceStatus in interface.py, which owns it): address kept here.
uint32_t* status_word(const at::Device& device) {
  static PyObject* kept[64] = {};
  static uint32_t* ptr[64] = {};
  const int idx = device.index();
  TORCH_CHECK(idx >= 0 && idx < 64, "device index out of range");
  if (ptr[idx] == nullptr) {
    PyObject* mod = PyImport_ImportModule("flash_attention_b200.interface");
    if (mod == nullptr) throw PyErrorSet();
    PyObject* cls = PyObject_GetAttrString(mod, "DeviceStatus");
    Py_DECREF(mod);
    if (cls == nullptr) throw PyErrorSet();
    PyObject* dev = THPDevice_New(device);
    PyObject* w = dev ? PyObject_CallMethod(cls, "word", "O", dev) : nullptr;
    Py_XDECREF(dev);
    Py_DECREF(cls);
    if (w == nullptr) throw PyErrorSet();
    kept[idx] = w;   // never freed: one word per device
    ptr[idx] = static_cast<uint32_t*>(THPVariable_Unpack(w).data_ptr());
  }
  return ptr[idx];
}

// ---- rules on sizes (interface.py documents them) ------------------------------------------------

// Causal and window arguments after the reference's rules (flash_attn/cute/interface.py:256-276).
struct Window {
  bool causal = false;
  int left = -1, right = -1;      // -1: no limit
};
Window resolve_window(bool causal, PyObject* left_o, PyObject* right_o) {
  bool has_l = !is_none(left_o), has_r = !is_none(right_o);
  long l = has_l ? integer_of(left_o) : 0, r = has_r ? integer_of(right_o) : 0;
  if (causal) { has_r = true; r = 0; }
  if (has_l && has_r && l + r < 0) has_l = has_r = false;
  if ((has_l && l < 0) || (has_r && r < 0))
    fail(PyExc_NotImplementedError, "negative window limits (a band shifted off the diagonal) are not built");
  Window w;
  w.left = has_l ? static_cast<int>(std::min<long>(l, 0x7fffffff)) : -1;
  w.right = has_r ? static_cast<int>(std::min<long>(r, 0x7fffffff)) : -1;
  w.causal = has_r && r == 0 && !has_l;
  return w;
}

int64_t cdiv(int64_t a, int64_t b) { return (a + b - 1) / b; }

int64_t decode_splits(int64_t B, int64_t Hkv, int64_t Sk, int64_t sms) {
  const int64_t blocks = cdiv(Sk, 128), units = std::max<int64_t>(1, B * Hkv);
  if (units > 3 * sms) {
    int64_t best = 1, best_cost = -1;
    for (int64_t ns = 1; ns < 5 && ns <= std::max<int64_t>(1, blocks / 2); ++ns) {
      const int64_t cost = cdiv(ns * units, 3 * sms) * (cdiv(blocks, ns) + 4);
      if (best_cost < 0 || cost < best_cost) { best = ns; best_cost = cost; }
    }
    return best;
  }
  const int64_t want = std::max<int64_t>(1, (2 * sms + units / 2) / units);
  return std::max<int64_t>(1, std::min({int64_t{128}, want, std::max<int64_t>(1, blocks / 2)}));
}

int64_t prefill_splits(int64_t B, int64_t Sq, int64_t Sk, int64_t Hq, int64_t sms) {
  const int64_t tiles = B * Hq * cdiv(Sq, 128), blocks = cdiv(Sk, 128);
  if (tiles * 2 > sms || blocks < 8) return 1;
  int64_t best = 1, best_cost = -1;
  for (int64_t n = 1; n <= std::min<int64_t>(blocks / 4, 128); ++n) {
    const int64_t per = cdiv(blocks, n);
    if (n > 1 && per * (n - 1) >= blocks) continue;   // the last split would be empty
    const int64_t cost = cdiv(tiles * n, sms) * (per + 2);
    if (best_cost < 0 || cost < best_cost) { best = n; best_cost = cost; }
  }
  return best;
}

// Up to this many keys (times kv heads, over the batch) a decode call reads linear scales itself instead of having
// them tiled by a launch of their own; the results are the same bits.  A lane fetches the eight bytes of a row, 32
// bytes of a sector, so the line depends on how far apart the rows of K are (`row_stride` bytes; V's, whose
// neighbouring blocks share the sector, cost the same in every shape):
//  * up to 16 bytes (one or two kv heads) two to four rows share a sector and reading is faster at any length -- but
//    for five to eight query rows, whose instantiations have no registers to spare (`tight`);
//  * from 256 bytes on (32 kv heads; `tight`: 128) the line is 128 k keys, between those 160 k.
// Tiling goes over the whole of a page pool, reading only over the pages in use: a pool of two or three times the keys
// of the table (`pool_ratio`) moves the line fourfold each time, beyond that reading is always faster.
// us, tiled first / read linear, one token, inputs from HBM (kv heads x query heads each):
//   8 x 4, 160 k keys x heads as 1, 4, 16, 32 entries 15.1 / 14.4, 14.7 / 13.9, 15.1 / 14.4, 14.0 / 13.1; 256 k 17.6 /
//     17.1, 17.3 / 17.2, 17.1 / 20.4, 16.0 / 17.6; 1 M 43.5 / 43.7, 43.3 / 44.0, 42.8 / 54.6, 42.2 / 54.9
//   32 x 1, 128 k, 1, 4, 16 entries 13.5 / 13.1, 13.8 / 13.6, 15.7 / 16.2, 160 k 14.6 / 14.7, 15.1 / 15.7, 18.0 / 18.3
//   16 x 1, 8 tokens, 128 k, 1, 8, 32 entries 15.1 / 15.8, 14.7 / 14.3, 17.4 / 17.8, 160 k 16.6 / 18.1, 15.9 / 16.7,
//     19.8 / 19.9; 16 x 4, 4 tokens, 160 k 17.5 / 17.4, 17.0 / 17.3, 22.1 / 20.7
//   2 x 4, 1 M, 4, 16, 32 entries 46.5 / 41.3, 46.1 / 41.7, 45.2 / 45.4; 1 x 16, 1 M, 8 entries 56.1 / 43.5
//   1 x 8, 384 k, 4, 16, 32 entries 26.4 / 27.1, 27.8 / 28.3, 25.2 / 25.4; 2 x 8, 1 M, 8 entries 47.7 / 52.0
//   pool of 2, 3 times the table, 8 x 4, 512 k 28.3 / 24.6, 32.9 / 24.7; 16 ragged entries 24.8 / 24.0, 28.2 / 23.8;
//     1 M 39.7 / 43.6, 47.9 / 43.8; of 16 times, 1 x 8, 256 k 122 / 19
// A call that is dealt by the lengths of its entries (fa4_nvfp4_decode_is_balanced, and a split count that is left open) reads them at any
// length: the key counts are on the device, so tiling goes over every slot of the cache.  us, tiled first / read linear, lengths spread over
// the logarithm down to a 64th: 8 x 4, 800 k slots x heads as 4, 12 entries 27.9 / 24.8, 32.4 / 27.9; 1.6 M as 4, 12, 40
//   38.7 / 29.8, 41.1 / 31.9, 36.2 / 27.3; 3.2 M 78.5 / 57.0, 79.8 / 45.2, 63.2 / 43.4; 32 x 1, 800 k as 4 28.8 / 29.4, 1.6 M
//   as 4, 12 43.9 / 38.8, 43.9 / 42.7, 3.2 M 81.7 / 64.8, 107 / 108; 8 x 4, four tokens, 800 k as 4, 12 31.6 / 27.3, 37.0 / 30.4.
int64_t linear_keys_limit(int64_t rows, int64_t row_stride, int64_t pool_ratio) {
  const bool tight = rows > 4 && rows <= 8;
  if (pool_ratio > 3 || (row_stride <= 16 && !tight)) return INT64_MAX;
  const int64_t line = row_stride >= (tight ? 128 : 256) ? 128 * 1024 : 160 * 1024;
  return line << (2 * (std::max<int64_t>(pool_ratio, 1) - 1));
}

int64_t sm_count(const at::Device& d) { return at::cuda::getDeviceProperties(d.index())->multiProcessorCount; }

bool head_dims_built(int64_t D, int64_t Dv) {
  return (D == Dv && (D == 64 || D == 128)) || (D == 192 && Dv == 128);
}

// The learnable sink as Hq contiguous fp32 values on the device.
at::Tensor sink_of(const at::Tensor& t, int64_t Hq, const at::Device& device) {
  if (!t.defined()) return {};
  FA4_ASSERT(t.dim() == 1 && t.size(0) == Hq, "learnable_sink must have one entry per query head");
  if (t.device() == device && t.scalar_type() == at::kFloat && t.is_contiguous()) return t;
  return t.to(device, at::kFloat).contiguous();
}

// ---- allocation ---------------------------------------------------------------------------------------
// (at::empty goes through the dispatcher, 2-4 us a call on the hosts of these GPUs; these do not)
at::Tensor new_tensor(at::IntArrayRef sizes, at::ScalarType dtype, const at::Device& device) {
  return at::detail::empty_cuda(sizes, dtype, device, std::nullopt);
}
// Scratch of the current stream, given back to it when the launches that use it have been issued.
c10::DataPtr scratch_bytes(int64_t bytes) { return c10::cuda::CUDACachingAllocator::get()->allocate((size_t)bytes); }

// ---- linear scales -> the tiled layout, the three tensors of a call in one launch ------------------
// One job: (outer, inner) matrices of rows x cols bytes.
fa4_nvfp4_sf_job sf_job(const at::Tensor& sf, int64_t outer, int64_t inner, int64_t rows, int64_t cols,
                        int64_t stride_outer, int64_t stride_inner, int64_t stride_row, int64_t mult) {
  fa4_nvfp4_sf_job j = {};
  j.src = sf.data_ptr();
  j.n_outer = (int32_t)outer; j.n_inner = (int32_t)inner; j.rows = (int32_t)rows; j.cols = (int32_t)cols;
  j.stride_outer = stride_outer; j.stride_inner = stride_inner; j.stride_row = stride_row;
  j.col_tile_multiple = (int32_t)mult;
  return j;
}
fa4_nvfp4_sf_job sf_job(const at::Tensor& sf, int rows_dim, int head_dim, int64_t mult) {
  return sf_job(sf, sf.size(0), sf.size(head_dim), sf.size(rows_dim), sf.size(3), sf.stride(0), sf.stride(head_dim),
                sf.stride(rows_dim), mult);
}
// Allocates the tiles of all jobs as one buffer and launches; the tiles of job i are at jobs[i].dst.
c10::DataPtr tile_scales(fa4_nvfp4_sf_job (&jobs)[3], void* stream) {
  int64_t bytes[3], total = 0;
  for (int i = 0; i < 3; ++i) {
    const fa4_nvfp4_sf_job& j = jobs[i];
    const int64_t ct = cdiv(cdiv(j.cols, 4), j.col_tile_multiple) * j.col_tile_multiple;
    bytes[i] = (int64_t)j.n_outer * j.n_inner * cdiv(j.rows, 128) * ct * 512;
    total += bytes[i];
  }
  c10::DataPtr out = scratch_bytes(total);
  uint8_t* at_byte = static_cast<uint8_t*>(out.get());
  for (int i = 0; i < 3; at_byte += bytes[i++]) jobs[i].dst = at_byte;
  check_rc(fa4_nvfp4_sf_tile_jobs(jobs, 3, stream), "fa4_nvfp4_sf_tile_jobs");
  return out;
}

PyObject* pair_of(PyObject* out_o, const at::Tensor& out, PyObject* lse_o, const at::Tensor& lse) {
  PyObject* a;
  if (!is_none(out_o)) { a = out_o; Py_INCREF(a); } else a = THPVariable_Wrap(out);
  PyObject* b;
  if (!is_none(lse_o)) { b = lse_o; Py_INCREF(b); }
  else if (lse.defined()) b = THPVariable_Wrap(lse);
  else { b = Py_None; Py_INCREF(b); }
  PyObject* r = PyTuple_New(2);
  PyTuple_SET_ITEM(r, 0, a);
  PyTuple_SET_ITEM(r, 1, b);
  return r;
}

// ---- flash_attn_fp4_func ------------------------------------------------------------------------
// q k v q_sf k_sf v_sf q_scale k_scale v_scale softmax_scale causal return_lse out lse sf_layout
// variant num_splits window_left window_right learnable_sink softcap seqused_k page_table
struct Call {
  at::Tensor q, k, v, q_sf, k_sf, v_sf, out, lse, sink, used, table;
  Scale scale[3];
  bool default_softmax_scale = true, want_lse = true, tiled = false;
  double softmax_scale = 0.0, softcap = 0.0;
  int variant = FA4_VARIANT_AUTO;
  long num_splits = 1;
  Window win;
  uint32_t* status = nullptr;
};

// Checks, allocates (out and lse where they are not given) and launches; no Python.
void run(Call& c) {
  at::Tensor &q = c.q, &k = c.k, &v = c.v, &q_sf = c.q_sf, &k_sf = c.k_sf, &v_sf = c.v_sf, &out = c.out, &lse = c.lse;
  FA4_ASSERT(q.dim() == 4 && k.dim() == 4 && v.dim() == 4, "q, k, v must be 4-D");
  FA4_ASSERT(q.is_cuda() && k.is_cuda() && v.is_cuda(), "inputs must be on CUDA");
  q = inner_contiguous(std::move(q));
  k = inner_contiguous(std::move(k));
  v = inner_contiguous(std::move(v));
  const int64_t B = q.size(0), Sq = q.size(1), Hq = q.size(2), D = 2 * q.size(3);
  const int64_t B_kv = k.size(0), Sk_kv = k.size(1), Hkv = k.size(2), Dv = v.size(2);
  const at::Device device = q.device();
  const bool paged = c.table.defined();
  int64_t Sk = Sk_kv, pages_per_seq = 0;
  at::Tensor table, used;
  if (paged) {
    // k / v are a pool of B_kv pages of Sk_kv (= page_size) keys; Sk is the logical key length
    const at::Tensor& t = c.table;
    FA4_ASSERT(t.dim() == 2 && t.size(0) == B && t.scalar_type() == at::kInt && t.is_cuda(),
               "page_table must be a (B, pages_per_seq) int32 CUDA tensor");
    FA4_ASSERT(v.size(0) == B_kv, "k and v pools differ in their number of pages");
    if (Sk_kv % 128 != 0)
      fail(PyExc_NotImplementedError, "page_size must be a multiple of 128 (whole K/V blocks per page)");
    table = t.contiguous();
    pages_per_seq = t.size(1);
    Sk = pages_per_seq * Sk_kv;
  } else {
    FA4_ASSERT(B_kv == B && v.size(0) == B, "batch size mismatch");
  }
  if (c.used.defined()) {
    const at::Tensor& t = c.used;
    FA4_ASSERT(t.dim() == 1 && t.size(0) == B && t.scalar_type() == at::kInt && t.is_cuda(),
               "seqused_k must be a (B,) int32 CUDA tensor");
    used = t.contiguous();
  }
  FA4_ASSERT(2 * k.size(3) == D, "q and k head dims differ");
  const int64_t Sk_pad = cdiv(Sk_kv, 32) * 32;   // V's key axis is padded to whole 32-key groups (zeros)
  FA4_ASSERT(v.size(1) == Hkv && 2 * v.size(3) == Sk_pad,
             "v must be (B, Hkv, Dv, Skp/2) with Skp = seqlen_k rounded up to a multiple of 32, got %s",
             dims_of(v.sizes()).c_str());
  FA4_ASSERT(Hkv > 0 && Hq % Hkv == 0, "num_head must be divisible by num_head_kv");
  if (!head_dims_built(D, Dv))
    fail(PyExc_NotImplementedError,
         "head dims (D=%lld, Dv=%lld) not built; supported: (128, 128), (64, 64) and (192, 128)", (long long)D,
         (long long)Dv);
  const double softmax_scale = c.default_softmax_scale ? 1.0 / std::sqrt((double)D) : c.softmax_scale;

  c10::cuda::OptionalCUDAGuard guard;
  if (device.index() != c10::cuda::current_device()) guard.set_device(device);
  void* stream = c10::cuda::getCurrentCUDAStream(device.index()).stream();

  const Window win = c.win;
  const double softcap = c.softcap;
  // A handful of query rows per kv head (decode, append): the transposed kernel, which always
  // splits the keys over CTAs and merges with the combine kernel.
  const bool decode_ok = D == 128 && Dv == 128 && Sq * (Hq / Hkv) <= 32 && win.left < 0 && win.right <= 0 &&
                         !c.sink.defined() && softcap == 0.0;
  const bool decode = c.variant == FA4_VARIANT_DECODE || (c.variant == FA4_VARIANT_AUTO && decode_ok);

  c10::DataPtr tiles;                     // scratch for tiled copies of linear scales
  const void* sf_ptr[3];
  fa4_nvfp4_linear_sf linear = {};
  if (!c.tiled) {
    validate(q_sf, "q_sf", {B, Sq, Hq, D / 16}, at::kByte, device);
    validate(k_sf, "k_sf", {B_kv, Sk_kv, Hkv, D / 16}, at::kByte, device);
    validate(v_sf, "v_sf", {B_kv, Hkv, Dv, Sk_pad / 16}, at::kByte, device);
    q_sf = inner_contiguous(std::move(q_sf));
    k_sf = inner_contiguous(std::move(k_sf));
    v_sf = inner_contiguous(std::move(v_sf));
    const int64_t pool_ratio = paged ? B_kv * Sk_kv / std::max<int64_t>(1, B * Sk) : 1;
    const bool dealt = c.num_splits == 0 && used.defined() && fa4_nvfp4_decode_is_balanced((int32_t)B, (int32_t)Sq, (int32_t)Sk, (int32_t)Hq, (int32_t)Hkv);
    if (decode && decode_ok && (dealt || B * Hkv * Sk <= linear_keys_limit(Sq * (Hq / Hkv), k_sf.stride(1), pool_ratio))) {
      // the decode kernel reads them as they are
      linear.struct_size = sizeof linear;
      linear.q_stride_b = q_sf.stride(0); linear.q_stride_s = q_sf.stride(1); linear.q_stride_h = q_sf.stride(2);
      linear.k_stride_b = k_sf.stride(0); linear.k_stride_s = k_sf.stride(1); linear.k_stride_h = k_sf.stride(2);
      linear.v_stride_b = v_sf.stride(0); linear.v_stride_h = v_sf.stride(1); linear.v_stride_d = v_sf.stride(2);
      sf_ptr[0] = q_sf.data_ptr();
      sf_ptr[1] = k_sf.data_ptr();
      sf_ptr[2] = v_sf.data_ptr();
    } else {
      fa4_nvfp4_sf_job jobs[3] = {sf_job(q_sf, 1, 2, 1), sf_job(k_sf, 1, 2, 1), sf_job(v_sf, 2, 1, 2)};
      tiles = tile_scales(jobs, stream);
      for (int i = 0; i < 3; ++i) sf_ptr[i] = jobs[i].dst;
    }
  } else {
    validate(q_sf, "q_sf", {B, Hq, cdiv(Sq, 128), D / 64, 512}, at::kByte, device);
    validate(k_sf, "k_sf", {B_kv, Hkv, cdiv(Sk_kv, 128), D / 64, 512}, at::kByte, device);
    validate(v_sf, "v_sf", {B_kv, Hkv, cdiv(Dv, 128), 2 * cdiv(Sk_kv, 128), 512}, at::kByte, device);
    FA4_ASSERT(q_sf.is_contiguous() && k_sf.is_contiguous() && v_sf.is_contiguous(),
               "tiled scale factors must be contiguous");
    sf_ptr[0] = q_sf.data_ptr();
    sf_ptr[1] = k_sf.data_ptr();
    sf_ptr[2] = v_sf.data_ptr();
  }

  if (!out.defined()) {
    out = new_tensor({B, Sq, Hq, Dv}, at::kBFloat16, device);
  } else {
    validate(out, "out", {B, Sq, Hq, Dv}, at::kBFloat16, device);
    FA4_ASSERT(out.stride(-1) == 1, "out's last dimension must be contiguous");
  }
  if (lse.defined()) {
    validate(lse, "lse", {B, Hq, Sq}, at::kFloat, device);
    FA4_ASSERT(lse.is_contiguous(), "lse must be contiguous");
  } else if (c.want_lse) {
    lse = new_tensor({B, Hq, Sq}, at::kFloat, device);
  }

  fa4_nvfp4_params p = {};
  p.struct_size = sizeof p;
  p.variant = c.variant;
  p.q = q.data_ptr();
  p.k = k.data_ptr();
  p.v = v.data_ptr();
  p.q_sf = sf_ptr[0];
  p.k_sf = sf_ptr[1];
  p.v_sf = sf_ptr[2];
  p.out = out.data_ptr();
  p.lse = lse.defined() ? lse.data_ptr<float>() : nullptr;
  p.status = c.status;
  p.q_stride_b = q.stride(0); p.q_stride_s = q.stride(1); p.q_stride_h = q.stride(2);
  p.k_stride_b = k.stride(0); p.k_stride_s = k.stride(1); p.k_stride_h = k.stride(2);
  p.v_stride_b = v.stride(0); p.v_stride_h = v.stride(1); p.v_stride_d = v.stride(2);
  p.o_stride_b = out.stride(0); p.o_stride_s = out.stride(1); p.o_stride_h = out.stride(2);
  p.B = (int32_t)B; p.Sq = (int32_t)Sq; p.Sk = (int32_t)Sk; p.Hq = (int32_t)Hq; p.Hkv = (int32_t)Hkv;
  p.D = (int32_t)D; p.Dv = (int32_t)Dv;
  const float* scales[3];
  const bool lazy = device_scales(c.scale, device, static_cast<cudaStream_t>(stream), scales);
  if (!lazy) {
    p.q_scale = c.scale[0].value("q_scale");
    p.k_scale = c.scale[1].value("k_scale");
    p.v_scale = c.scale[2].value("v_scale");
  }
  p.softmax_scale = (float)softmax_scale;

  long num_splits = c.num_splits;
  if (num_splits < 0 || num_splits > 128) fail(PyExc_ValueError, "num_splits must be in 0..128");
  const bool auto_splits = num_splits == 0;
  p.causal = win.causal ? 1 : 0;
  if (!(softcap >= 0.0) || !std::isfinite(softcap)) fail(PyExc_ValueError, "softcap must be a finite number >= 0");
  const at::Tensor sink = sink_of(c.sink, Hq, device);
  if (p.variant == FA4_VARIANT_DECODE && !decode_ok)
    fail(PyExc_NotImplementedError,
         "the decode kernel takes D = Dv = 128, Sq * (Hq / Hkv) <= 32, no window / sink / softcap");
  if (decode) p.variant = FA4_VARIANT_DECODE;
  if (auto_splits)
    num_splits = decode ? decode_splits(B, Hkv, Sk, sm_count(device)) : prefill_splits(B, Sq, Sk, Hq, sm_count(device));

  if (num_splits == 1 && !sink.defined() && win.left < 0 && win.right <= 0 && softcap == 0.0 && !used.defined() &&
      !paged && !decode && !lazy) {
    check_rc(fa4_nvfp4_fwd(&p, stream), "fa4_nvfp4_fwd");
  } else {
    fa4_nvfp4_ext x = {};
    x.struct_size = sizeof x;
    x.num_splits = (int32_t)num_splits;
    x.window_left = win.left;
    x.window_right = win.right;
    x.sink = sink.defined() ? sink.data_ptr<float>() : nullptr;
    x.softcap = (float)softcap;
    x.seqused_k = used.defined() ? used.data_ptr<int32_t>() : nullptr;
    if (paged) {
      x.page_table = table.data_ptr<int32_t>();
      x.page_size = (int32_t)Sk_kv;
      x.pages_per_seq = (int32_t)pages_per_seq;
      x.num_pages = (int32_t)B_kv;
    }
    c10::DataPtr workspace;
    // (a split count that the caller chose is kept to: the result of an entry then does not depend on the others)
    const int64_t bytes = auto_splits ? fa4_nvfp4_fwd_ex_workspace_bytes(&p, &x)
                                      : fa4_nvfp4_splitkv_workspace_bytes(&p, (int32_t)num_splits);
    if (bytes < 0) check_rc((int)bytes, "workspace of fa4_nvfp4_fwd_ex");
    if (bytes > 0) {
      workspace = scratch_bytes(bytes);
      x.workspace = workspace.get();
      x.workspace_bytes = (uint64_t)bytes;
    }
    if (linear.struct_size != 0) {
      if (lazy) linear.q_scale = scales[0], linear.k_scale = scales[1], linear.v_scale = scales[2];
      check_rc(fa4_nvfp4_fwd_decode_linear_sf(&p, &x, &linear, stream), "fa4_nvfp4_fwd_decode_linear_sf");
    } else if (lazy)
      check_rc(fa4_nvfp4_fwd_device_scales(&p, &x, scales[0], scales[1], scales[2], stream), "fa4_nvfp4_fwd_device_scales");
    else
      check_rc(fa4_nvfp4_fwd_ex(&p, &x, stream), "fa4_nvfp4_fwd_ex");
  }
}

PyObject* fwd(PyObject* const* a) {
  Call c;
  c.q = as_u8(a[0], "q"), c.k = as_u8(a[1], "k"), c.v = as_u8(a[2], "v");
  c.q_sf = as_u8(a[3], "q_sf"), c.k_sf = as_u8(a[4], "k_sf"), c.v_sf = as_u8(a[5], "v_sf");
  for (int i = 0; i < 3; ++i) c.scale[i] = scale_of(a[6 + i]);
  c.default_softmax_scale = is_none(a[9]);
  if (!c.default_softmax_scale) c.softmax_scale = number_of(a[9]);
  c.want_lse = truth_of(a[11]);
  c.out = optional_tensor(a[12], "out");
  c.lse = optional_tensor(a[13], "lse");
  const char* layout = PyUnicode_Check(a[14]) ? PyUnicode_AsUTF8(a[14]) : nullptr;
  c.tiled = layout != nullptr && !strcmp(layout, "tiled");
  if (!c.tiled && (layout == nullptr || strcmp(layout, "linear") != 0)) {
    PyErr_Format(PyExc_ValueError, "sf_layout must be 'linear' or 'tiled', got %R", a[14]);
    throw PyErrorSet();
  }
  c.variant = (int)integer_of(a[15]);
  c.num_splits = integer_of(a[16]);
  c.win = resolve_window(truth_of(a[10]), a[17], a[18]);
  c.sink = optional_tensor(a[19], "learnable_sink");
  if (!is_none(a[20])) c.softcap = number_of(a[20]);
  c.used = optional_tensor(a[21], "seqused_k");
  c.table = optional_tensor(a[22], "page_table");
  if (c.q.is_cuda()) c.status = status_word(c.q.device());
  {
    NoGil nogil;
    run(c);
  }
  return pair_of(a[12], c.out, a[13], c.lse);
}

// ---- flash_attn_varlen_fp4_func -------------------------------------------------------------------
at::Tensor offsets_of(const at::Tensor& t, const char* name, const at::Device& device) {
  if (!t.defined()) return {};
  FA4_ASSERT(t.dim() == 1, "%s must be one-dimensional", name);
  if (t.device() == device && t.scalar_type() == at::kInt && t.is_contiguous()) return t;
  return t.to(device, at::kInt).contiguous();
}

// the longest sequence of a packed batch: one synchronising read
int64_t longest_of(const at::Tensor& cu) { return cu.diff().max().item<int64_t>(); }

// q k v q_sf k_sf v_sf q_scale k_scale v_scale cu_q cu_k seqused_k cu_v max_q max_k softmax_scale causal
// window_left window_right learnable_sink softcap return_lse
struct VarlenCall : Call {
  at::Tensor cu_q, cu_k, cu_v;
  bool known = false;              // max_q and max_k are given
  int64_t max_q = 0, max_k = 0;
};

void run_varlen(VarlenCall& c) {
  at::Tensor &q = c.q, &k = c.k, &v = c.v, &q_sf = c.q_sf, &k_sf = c.k_sf, &v_sf = c.v_sf, &out = c.out, &lse = c.lse;
  FA4_ASSERT(q.dim() == 3 && k.dim() == 3 && v.dim() == 3, "packed operands are 3-D");
  FA4_ASSERT(q.is_cuda() && k.is_cuda() && v.is_cuda(), "inputs must be on CUDA");
  q = inner_contiguous(std::move(q));
  k = inner_contiguous(std::move(k));
  v = inner_contiguous(std::move(v));
  const at::Device device = q.device();
  c10::cuda::OptionalCUDAGuard guard;
  if (device.index() != c10::cuda::current_device()) guard.set_device(device);
  void* stream = c10::cuda::getCurrentCUDAStream(device.index()).stream();
  q_sf = q_sf.contiguous();
  k_sf = k_sf.contiguous();
  v_sf = v_sf.contiguous();
  const int64_t total_q = q.size(0), Hq = q.size(1), D = 2 * q.size(2);
  const int64_t total_k = k.size(0), Hkv = k.size(1), Dv = v.size(1);
  const bool has_cu_v = c.cu_v.defined();
  const int64_t total_kp = has_cu_v ? 2 * v.size(2) : cdiv(total_k, 32) * 32;
  FA4_ASSERT(2 * k.size(2) == D && v.size(0) == Hkv && Hkv > 0 && Hq % Hkv == 0,
             "head counts / head dims of q, k, v do not fit");
  FA4_ASSERT(2 * v.size(2) == total_kp && total_kp % 32 == 0 && total_kp >= total_k,
             "v must be (Hkv, Dv, total_kp/2) with total_kp = %lld, got %s", (long long)total_kp,
             dims_of(v.sizes()).c_str());
  FA4_ASSERT(q_sf.sizes() == at::IntArrayRef({total_q, Hq, D / 16}) &&
                 k_sf.sizes() == at::IntArrayRef({total_k, Hkv, D / 16}) &&
                 v_sf.sizes() == at::IntArrayRef({Hkv, Dv, total_kp / 16}),
             "scale factors must be the packed linear layouts");
  if (!head_dims_built(D, Dv))
    fail(PyExc_NotImplementedError, "head dims (D=%lld, Dv=%lld) not built", (long long)D, (long long)Dv);
  const at::Tensor cu_q = offsets_of(c.cu_q, "cu_seqlens_q", device), cu_k = offsets_of(c.cu_k, "cu_seqlens_k", device);
  FA4_ASSERT(cu_q.numel() == cu_k.numel() && cu_q.numel() >= 2, "cu_seqlens_q / cu_seqlens_k describe different batches");
  const int64_t seqs = cu_q.numel() - 1;
  const at::Tensor cu_v = offsets_of(c.cu_v, "cu_seqlens_v", device), used = offsets_of(c.used, "seqused_k", device);
  FA4_ASSERT(!cu_v.defined() || cu_v.numel() == seqs + 1, "cu_seqlens_v has another batch size");
  FA4_ASSERT(!used.defined() || used.numel() == seqs, "seqused_k has another batch size");
  // without both maxima one synchronising read; pass them to stay asynchronous, as the reference's callers do
  int64_t max_q = c.known ? c.max_q : longest_of(cu_q), max_k = c.known ? c.max_k : longest_of(cu_k);
  max_q = std::min(std::max<int64_t>(1, max_q), total_q);
  max_k = std::min(std::max<int64_t>(1, max_k), total_k);
  const double softmax_scale = c.default_softmax_scale ? 1.0 / std::sqrt((double)D) : c.softmax_scale;
  const Window win = c.win;
  const at::Tensor sink = sink_of(c.sink, Hq, device);

  // per-sequence tiles of the packed scales, padded to the longest sequence
  const int64_t cols = D / 16, ckp = total_kp / 16;
  fa4_nvfp4_sf_job jobs[3] = {sf_job(q_sf, seqs, Hq, max_q, cols, 0, cols, Hq * cols, 1),
                              sf_job(k_sf, seqs, Hkv, max_k, cols, 0, cols, Hkv * cols, 1),
                              sf_job(v_sf, seqs, Hkv, Dv, cdiv(max_k, 16), 0, Dv * ckp, ckp, 2)};
  jobs[0].cu_seqlens = cu_q.data_ptr<int32_t>();
  jobs[1].cu_seqlens = cu_k.data_ptr<int32_t>();
  jobs[2].cu_seqlens = (cu_v.defined() ? cu_v : cu_k).data_ptr<int32_t>();
  jobs[0].packed_rows = jobs[1].packed_rows = 1;
  const c10::DataPtr tiles = tile_scales(jobs, stream);
  out = new_tensor({total_q, Hq, Dv}, at::kBFloat16, device);
  if (c.want_lse) lse = new_tensor({Hq, total_q}, at::kFloat, device);

  fa4_nvfp4_params p = {};
  p.struct_size = sizeof p;
  p.q = q.data_ptr(); p.k = k.data_ptr(); p.v = v.data_ptr();
  p.q_sf = jobs[0].dst; p.k_sf = jobs[1].dst; p.v_sf = jobs[2].dst;
  p.out = out.data_ptr();
  p.lse = lse.defined() ? lse.data_ptr<float>() : nullptr;
  p.status = c.status;
  p.q_stride_s = q.stride(0); p.q_stride_h = q.stride(1); p.q_stride_b = q.stride(0) * std::max<int64_t>(1, total_q);
  p.k_stride_s = k.stride(0); p.k_stride_h = k.stride(1); p.k_stride_b = k.stride(0) * std::max<int64_t>(1, total_k);
  p.v_stride_h = v.stride(0); p.v_stride_d = v.stride(1); p.v_stride_b = v.stride(0) * Hkv;
  p.o_stride_s = out.stride(0); p.o_stride_h = out.stride(1); p.o_stride_b = out.stride(0) * std::max<int64_t>(1, total_q);
  p.B = (int32_t)seqs; p.Sq = (int32_t)max_q; p.Sk = (int32_t)max_k; p.Hq = (int32_t)Hq; p.Hkv = (int32_t)Hkv;
  p.D = (int32_t)D; p.Dv = (int32_t)Dv;
  p.causal = win.causal ? 1 : 0;
  p.q_scale = c.scale[0].value("q_scale");
  p.k_scale = c.scale[1].value("k_scale");
  p.v_scale = c.scale[2].value("v_scale");
  p.softmax_scale = (float)softmax_scale;

  fa4_nvfp4_varlen x = {};
  x.struct_size = sizeof x;
  x.num_seqs = (int32_t)seqs;
  x.cu_seqlens_q = cu_q.data_ptr<int32_t>();
  x.cu_seqlens_k = cu_k.data_ptr<int32_t>();
  x.seqused_k = used.defined() ? used.data_ptr<int32_t>() : nullptr;
  x.total_q = (int32_t)total_q;
  x.total_k = (int32_t)total_k;
  x.max_seqlen_q = (int32_t)max_q;
  x.max_seqlen_k = (int32_t)max_k;
  x.window_left = win.left;
  x.window_right = win.right;
  x.sink = sink.defined() ? sink.data_ptr<float>() : nullptr;
  x.softcap = (float)c.softcap;
  x.cu_seqlens_v = cu_v.defined() ? cu_v.data_ptr<int32_t>() : nullptr;
  x.total_v = cu_v.defined() ? (int32_t)total_kp : 0;
  check_rc(fa4_nvfp4_fwd_varlen(&p, &x, stream), "fa4_nvfp4_fwd_varlen");
}

PyObject* varlen_fwd(PyObject* const* a) {
  VarlenCall c;
  c.q = as_u8(a[0], "q"), c.k = as_u8(a[1], "k"), c.v = as_u8(a[2], "v");
  c.q_sf = as_u8(a[3], "q_sf"), c.k_sf = as_u8(a[4], "k_sf"), c.v_sf = as_u8(a[5], "v_sf");
  for (int i = 0; i < 3; ++i) c.scale[i] = scale_of(a[6 + i]);
  c.cu_q = tensor_of(a[9], "cu_seqlens_q");
  c.cu_k = tensor_of(a[10], "cu_seqlens_k");
  c.used = optional_tensor(a[11], "seqused_k");
  c.cu_v = optional_tensor(a[12], "cu_seqlens_v");
  c.known = !is_none(a[13]) && !is_none(a[14]);
  if (c.known) c.max_q = integer_of(a[13]), c.max_k = integer_of(a[14]);
  c.default_softmax_scale = is_none(a[15]);
  if (!c.default_softmax_scale) c.softmax_scale = number_of(a[15]);
  c.win = resolve_window(truth_of(a[16]), a[17], a[18]);
  c.sink = optional_tensor(a[19], "learnable_sink");
  if (!is_none(a[20])) c.softcap = number_of(a[20]);
  c.want_lse = truth_of(a[21]);
  if (c.q.is_cuda()) c.status = status_word(c.q.device());
  {
    NoGil nogil;
    run_varlen(c);
  }
  return pair_of(nullptr, c.out, nullptr, c.lse);
}

// ---- quantize_qkv_fused ----------------------------------------------------------------------------
// Allocates the results and launches; no Python.
void quantize(const at::Tensor (&in)[3], bool linear, at::Tensor (&packed)[3], at::Tensor (&lin)[3],
              at::Tensor (&tiled)[3], ScaleState& state) {
  const at::Device device = in[0].device();
  fa4_nvfp4_quant_job jobs[3] = {};
  c10::DataPtr scratch, scales;
  c10::cuda::OptionalCUDAGuard guard;
  for (int i = 0; i < 3; ++i) {
    const at::Tensor& x = in[i];
    FA4_ASSERT(x.is_cuda() && x.scalar_type() == at::kBFloat16 && x.dim() == 4 && x.stride(-1) == 1 &&
                   x.device() == device,
               "quantize_qkv_fused takes CUDA bf16 (B, S, H, D) tensors, last dim contiguous");
    if (i == 0) {
      if (device.index() != c10::cuda::current_device()) guard.set_device(device);
      scales = scratch_bytes(3 * sizeof(float));
      scratch = scratch_bytes(FA4_QUANT_SCRATCH_FLOATS * sizeof(float));
    }
    const int64_t B = x.size(0), S = x.size(1), H = x.size(2), D = x.size(3);
    // V is blocked along its key axis, stored padded with zeros to whole 32-key groups
    const int64_t s_out = i == 2 ? cdiv(S, 32) * 32 : S;
    if (i == 2) {
      packed[i] = new_tensor({B, H, D, s_out / 2}, at::kByte, device);
      if (linear) lin[i] = new_tensor({B, H, D, s_out / 16}, at::kByte, device);
      tiled[i] = new_tensor({B, H, cdiv(D, 128), 2 * cdiv(s_out, 128), 512}, at::kByte, device);
    } else {
      packed[i] = new_tensor({B, S, H, D / 2}, at::kByte, device);
      if (linear) lin[i] = new_tensor({B, S, H, D / 16}, at::kByte, device);
      tiled[i] = new_tensor({B, H, cdiv(S, 128), D / 64, 512}, at::kByte, device);
    }
    fa4_nvfp4_quant_job& j = jobs[2 - i];   // V first: its tiles take longest
    j.x = x.data_ptr();
    j.stride_b = x.stride(0); j.stride_s = x.stride(1); j.stride_h = x.stride(2);
    j.B = (int32_t)B; j.S = (int32_t)S; j.H = (int32_t)H; j.D = (int32_t)D;
    j.is_v = i == 2;
    j.S_out = (int32_t)s_out;
    j.packed = packed[i].data_ptr();
    j.sf_linear = linear ? lin[i].data_ptr() : nullptr;
    j.sf_tiled = tiled[i].data_ptr();
    j.scale_out = static_cast<float*>(scales.get()) + i;
  }
  const c10::cuda::CUDAStream stream = c10::cuda::getCurrentCUDAStream(device.index());
  check_rc(fa4_nvfp4_quantize_jobs_bf16(jobs, 3, static_cast<float*>(scratch.get()), stream.stream()), "fa4_nvfp4_quantize_jobs_bf16");
  state.device = std::move(scales);
  state.stream = stream.stream();
}

// q k v linear_sf -> (packed, linear scales or None, tiled scales, LazyScale) x 3
PyObject* quantize_qkv(PyObject* const* a) {
  static const char* names[3] = {"q", "k", "v"};
  const bool linear = truth_of(a[3]);
  at::Tensor in[3], packed[3], lin[3], tiled[3];
  for (int i = 0; i < 3; ++i) in[i] = tensor_of(a[i], names[i]);
  auto state = std::make_shared<ScaleState>();
  {
    NoGil nogil;
    quantize(in, linear, packed, lin, tiled, *state);
  }
  PyObject* res = PyTuple_New(3);
  for (int i = 0; i < 3; ++i) {
    PyObject* t = PyTuple_New(4);
    PyTuple_SET_ITEM(t, 0, THPVariable_Wrap(packed[i]));
    PyObject* l = linear ? THPVariable_Wrap(lin[i]) : (Py_INCREF(Py_None), Py_None);
    PyTuple_SET_ITEM(t, 1, l);
    PyTuple_SET_ITEM(t, 2, THPVariable_Wrap(tiled[i]));
    PyTuple_SET_ITEM(t, 3, new_lazy(state, i));
    PyTuple_SET_ITEM(res, i, t);
  }
  return res;
}

// ---- HostPipeline.run: the pieces of a call on operands in host memory -----------------------------
// q k v q_sf k_sf v_sf (host) | the same on the device | out lse (device) | out_host lse_host | q_scale k_scale
// v_scale softmax_scale causal | ranges [(s0, s1), ...] | streams in, compute, out (cudaStream_t as integers)
//
// Issued from Python a piece cost 140 us of host time against 155 us of its copy-out, so the loads went out
// late; here it is about 45.  Tried and not kept: K and V by range as well, more and smaller pieces
// (each copy beside a copy-out costs 30-40 us whatever its size), and loads by a kernel that reads the
// pinned memory (no faster beside a copy-out, and it slows the kernels it runs next to).
struct Event {
  cudaEvent_t e = nullptr;
  Event() { C10_CUDA_CHECK(cudaEventCreateWithFlags(&e, cudaEventDisableTiming)); }
  ~Event() { cudaEventDestroy(e); }
  // what `then` is given next runs after what `first` holds now
  void order(cudaStream_t first, cudaStream_t then) {
    C10_CUDA_CHECK(cudaEventRecord(e, first));
    C10_CUDA_CHECK(cudaStreamWaitEvent(then, e, 0));
  }
};

void issue_pieces(PyObject* const* a) {
  at::Tensor host[6], dev[6];
  static const char* names[6] = {"q", "k", "v", "q_sf", "k_sf", "v_sf"};
  for (int i = 0; i < 6; ++i) {
    host[i] = tensor_of(a[i], names[i]);
    dev[i] = tensor_of(a[6 + i], names[i]);
    FA4_ASSERT(host[i].element_size() == 1 && host[i].is_cpu() && host[i].is_contiguous() && dev[i].is_contiguous() &&
                   host[i].sizes() == dev[i].sizes(),
               "%s: packed bytes in a contiguous CPU tensor of the pipeline's shape expected", names[i]);
  }
  const at::Tensor out = tensor_of(a[12], "out"), lse = tensor_of(a[13], "lse"), out_host = tensor_of(a[14], "out_host");
  at::Tensor lse_host;
  if (!is_none(a[15])) lse_host = tensor_of(a[15], "lse_host");
  const bool causal = truth_of(a[20]);
  const at::Device device = dev[0].device();
  Call call;                       // what the pieces share
  for (int i = 0; i < 3; ++i) call.scale[i] = scale_of(a[16 + i]);
  call.default_softmax_scale = is_none(a[19]);
  if (!call.default_softmax_scale) call.softmax_scale = number_of(a[19]);
  call.win = resolve_window(causal, nullptr, nullptr);
  call.status = status_word(device);
  std::vector<std::pair<int64_t, int64_t>> ranges;
  for (Py_ssize_t n = 0; n < PyList_GET_SIZE(a[21]); ++n) {
    PyObject* r = PyList_GET_ITEM(a[21], n);
    const int64_t s0 = integer_of(PyTuple_GET_ITEM(r, 0)), s1 = integer_of(PyTuple_GET_ITEM(r, 1));
    ranges.emplace_back(s0, s1);
  }
  cudaStream_t raw[3];
  for (int i = 0; i < 3; ++i) {
    raw[i] = static_cast<cudaStream_t>(PyLong_AsVoidPtr(a[22 + i]));
    if (raw[i] == nullptr && PyErr_Occurred()) throw PyErrorSet();
  }
  const c10::cuda::CUDAStream s_in = c10::cuda::getStreamFromExternal(raw[0], device.index()),
                              s_compute = c10::cuda::getStreamFromExternal(raw[1], device.index()),
                              s_out = c10::cuda::getStreamFromExternal(raw[2], device.index());
  const int64_t B = dev[0].size(0), Sq = dev[0].size(1), Hq = dev[0].size(2), Sk = dev[1].size(1);
  NoGil nogil;                     // (copies from and to pageable memory wait for themselves and for what is before them)
  c10::cuda::CUDAGuard device_guard(device);
  Event in_done, compute_done;
  // rows [r0, r1) of batch entry b (contiguous byte tensors, both sides)
  auto load = [&](int i, int64_t b, int64_t r0, int64_t r1) {
    const int64_t row = dev[i].stride(1), at_byte = b * dev[i].stride(0) + r0 * row;
    C10_CUDA_CHECK(cudaMemcpyAsync(dev[i].data_ptr<uint8_t>() + at_byte,
                                   static_cast<const uint8_t*>(host[i].data_ptr()) + at_byte, (r1 - r0) * row,
                                   cudaMemcpyHostToDevice, raw[0]));
  };
  auto store = [&](const at::Tensor& to, const at::Tensor& from, int64_t b, int64_t r0, int64_t r1) {
    if (to.is_contiguous() && to.scalar_type() == from.scalar_type() && to.sizes() == from.sizes()) {
      const int64_t size = from.element_size(), row = from.stride(1) * size, at_byte = b * from.stride(0) * size + r0 * row;
      C10_CUDA_CHECK(cudaMemcpyAsync(static_cast<uint8_t*>(to.data_ptr()) + at_byte,
                                     static_cast<const uint8_t*>(from.data_ptr()) + at_byte, (r1 - r0) * row,
                                     cudaMemcpyDeviceToHost, raw[2]));
    } else {
      c10::cuda::CUDAStreamGuard g(s_out);
      to.select(0, b).narrow(0, r0, r1 - r0).copy_(from.select(0, b).narrow(0, r0, r1 - r0), /*non_blocking=*/true);
    }
  };
  // pinned blocks go back to their pool no earlier than the copies issued here have run, also after an error
  auto keep = [](const at::Tensor& t, const c10::cuda::CUDAStream& s) {
    if (t.is_pinned()) at::getHostAllocator(at::kCUDA)->record_event(t.data_ptr(), t.storage().data_ptr().get_context(), s.unwrap());
  };
  auto keep_all = [&] {
    for (const at::Tensor& t : host) keep(t, s_in);
    keep(out_host, s_out);
    if (lse_host.defined()) keep(lse_host, s_out);
  };
  try {
    for (int64_t b = 0; b < B; ++b) {
      // Few, large loads: while a copy-out runs, PCIe lets about 16 GB/s in, and each copy waits its turn.
      // The query rows of the first entry come by range, so that its first piece starts early.
      for (int i : {3, 4, 5, 1, 2}) load(i, b, 0, dev[i].size(1));
      if (b > 0) load(0, b, 0, Sq);
      for (const auto& [s0, s1] : ranges) {
        const int64_t sk = causal ? s1 : Sk;     // s1 is a multiple of 128, or Sq == Sk for the last range
        if (b == 0) load(0, b, s0, s1);
        in_done.order(raw[0], raw[1]);
        {
          // one range of query rows against its keys, through the same entry as any other call.  The LSE of
          // a partial range is a strided slice of (Hq, Sq): written compactly, then moved into place
          c10::cuda::CUDAStreamGuard g(s_compute);
          const bool whole = s1 - s0 == Sq;
          const int64_t kp = cdiv(sk, 32) * 32;
          Call c = call;
          c.q = dev[0].narrow(0, b, 1).narrow(1, s0, s1 - s0);
          c.k = dev[1].narrow(0, b, 1).narrow(1, 0, sk);
          c.v = dev[2].narrow(0, b, 1).narrow(3, 0, kp / 2);
          c.q_sf = dev[3].narrow(0, b, 1).narrow(1, s0, s1 - s0);
          c.k_sf = dev[4].narrow(0, b, 1).narrow(1, 0, sk);
          c.v_sf = dev[5].narrow(0, b, 1).narrow(3, 0, kp / 16);
          c.out = out.narrow(0, b, 1).narrow(1, s0, s1 - s0);
          if (whole) c.lse = lse.narrow(0, b, 1);
          run(c);
          if (!whole) {
            C10_CUDA_CHECK(cudaMemcpy2DAsync(lse.data_ptr<float>() + b * Hq * Sq + s0, Sq * 4, c.lse.data_ptr<float>(),
                                             (s1 - s0) * 4, (s1 - s0) * 4, Hq, cudaMemcpyDeviceToDevice, raw[1]));
          }
        }
        compute_done.order(raw[1], raw[2]);
        store(out_host, out, b, s0, s1);
      }
      if (lse_host.defined()) store(lse_host, lse, b, 0, Hq);
    }
  } catch (...) {
    try {
      keep_all();
    } catch (const std::exception&) {      // (the first error is the one to report)
    }
    throw;
  }
  keep_all();
}

PyObject* host_pieces(PyObject* const* a) {
  issue_pieces(a);
  Py_RETURN_NONE;
}

// ---- the module -----------------------------------------------------------------------------------
PyObject* choose_decode_splits(PyObject* const* a) {
  return PyLong_FromLongLong(decode_splits(integer_of(a[0]), integer_of(a[1]), integer_of(a[2]), integer_of(a[3])));
}
PyObject* choose_num_splits(PyObject* const* a) {
  return PyLong_FromLongLong(
      prefill_splits(integer_of(a[0]), integer_of(a[1]), integer_of(a[2]), integer_of(a[3]), integer_of(a[4])));
}
PyObject* choose_linear_keys(PyObject* const* a) {
  return PyLong_FromLongLong(linear_keys_limit(integer_of(a[0]), integer_of(a[1]), integer_of(a[2])));
}
PyObject* window_of(PyObject* const* a) {
  const Window w = resolve_window(truth_of(a[0]), a[1], a[2]);
  PyObject *t = w.causal ? Py_True : Py_False, *l = w.left < 0 ? nullptr : PyLong_FromLong(w.left),
           *r = w.right < 0 ? nullptr : PyLong_FromLong(w.right);
  PyObject* res = PyTuple_Pack(3, t, l ? l : Py_None, r ? r : Py_None);
  Py_XDECREF(l);
  Py_XDECREF(r);
  return res;
}

// Sets the exception _lib.check raises for a return code of the C ABI.
void raise_for(const CallFailed& f) {
  PyObject* mod = PyImport_ImportModule("flash_attention_b200._lib");
  if (mod == nullptr) return;
  PyObject* r = PyObject_CallMethod(mod, "check", "is", f.rc, f.what);
  Py_DECREF(mod);
  Py_XDECREF(r);
}

template <PyObject* (*fn)(PyObject* const*), int kArgs>
PyObject* entry(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != kArgs) {
    PyErr_Format(PyExc_TypeError, "expected %d positional arguments, got %zd", kArgs, n);
    return nullptr;
  }
  HANDLE_TH_ERRORS
  try {
    return fn(args);
  } catch (const PyErrorSet&) {
    return nullptr;
  } catch (const Failure& f) {
    PyErr_SetString(f.type, f.message.c_str());
    return nullptr;
  } catch (const CallFailed& f) {
    raise_for(f);
    return nullptr;
  }
  END_HANDLE_TH_ERRORS
}
template <PyObject* (*fn)(PyObject* const*), int kArgs>
PyMethodDef method(const char* name) {
  return {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(&entry<fn, kArgs>)), METH_FASTCALL, nullptr};
}
PyMethodDef methods[] = {method<fwd, 23>("fwd"),
                         method<varlen_fwd, 22>("varlen_fwd"),
                         method<choose_decode_splits, 4>("choose_decode_splits"),
                         method<choose_num_splits, 5>("choose_num_splits"),
                         method<choose_linear_keys, 3>("choose_linear_keys"),
                         method<quantize_qkv, 4>("quantize_qkv"),
                         method<host_pieces, 25>("host_pieces"),
                         method<window_of, 3>("resolve_window"),
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_host", "Native host path of flash_attention_b200.", -1, methods,
                          nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) {
  lazy_number.nb_float = lazy_float;
  lazy_type.tp_name = "flash_attention_b200._host.LazyScale";
  lazy_type.tp_doc = "A per-tensor scale on its way from the quantiser; float() waits for it.";
  lazy_type.tp_basicsize = sizeof(LazyScale);
  lazy_type.tp_flags = Py_TPFLAGS_DEFAULT;
  lazy_type.tp_as_number = &lazy_number;
  lazy_type.tp_dealloc = lazy_dealloc;
  if (PyType_Ready(&lazy_type) < 0) return nullptr;
  PyObject* m = PyModule_Create(&module_def);
  if (m != nullptr) PyModule_AddObjectRef(m, "LazyScale", reinterpret_cast<PyObject*>(&lazy_type));
  return m;
}
