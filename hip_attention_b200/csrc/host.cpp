// Host path of the operator: argument checks, device memory, launches and the returned metadata of one hip_attention_12
// call (dual_stage_quadratic_hip_attention, attention_extend.py:1918-3133), as a CPython extension over torch tensors.
//
// A decode call on a cached mask is ~15 us of kernels and is made once per layer and token; in Python its checks, parameter
// structs, allocations and launches took 100 us.  Here an attribute read is 40 ns, an allocation from torch's caching
// allocator half a microsecond, and what the call returns besides the context (copies of a cached mask, widened chunk
// bounds, query positions, constants) is written by kernels that run anyway or by one launch for all of it.
//
// Device work goes through the functions of libhipattn_sm100.so; memory and streams are torch's.  The module is stateless
// but for references to the package's Python classes and the per-device status words.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cmath>
#include <cstdarg>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <string>
#include <unordered_map>
#include <vector>

#include "../../include/hipattn.h"
#include "host_kernels.h"

namespace {

// ---------------------------------------------------------------------------------------------------------------------
// Python plumbing
// ---------------------------------------------------------------------------------------------------------------------
struct PyError {};   // a Python exception is set

[[noreturn]] void fail(PyObject* type, const char* fmt, ...) {
  char msg[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(msg, sizeof(msg), fmt, ap);
  va_end(ap);
  PyErr_SetString(type, msg);
  throw PyError{};
}
#define VALUE_ERROR(...) fail(PyExc_ValueError, __VA_ARGS__)
#define NOT_BUILT(...) fail(PyExc_NotImplementedError, __VA_ARGS__)

class Ref {   // owned reference
 public:
  Ref() = default;
  explicit Ref(PyObject* o) : o_(o) {}
  Ref(Ref&& r) noexcept : o_(r.o_) { r.o_ = nullptr; }
  Ref& operator=(Ref&& r) noexcept { std::swap(o_, r.o_); return *this; }
  Ref(const Ref&) = delete;
  ~Ref() { Py_XDECREF(o_); }
  PyObject* get() const { return o_; }
  PyObject* release() { PyObject* o = o_; o_ = nullptr; return o; }
  bool none() const { return o_ == nullptr || o_ == Py_None; }
  static Ref borrow(PyObject* o) { Py_XINCREF(o); return Ref(o); }

 private:
  PyObject* o_ = nullptr;
};
Ref checked(PyObject* o) {
  if (!o) throw PyError{};
  return Ref(o);
}

// interned attribute names
#define NAMES(X)                                                                                                              \
  X(offload_cache) X(online_update_cache) X(using_extend) X(need_apply_rope) X(rope_cos) X(rope_sin) X(sa_extend_backend)       \
  X(stages) X(scan_extend_backend) X(low_percent) X(low_k_ratio) X(is_causal) X(stage_early_terminate)                         \
  X(sliding_window_indices) X(second_stage_k) X(q_mask) X(k_mask) X(k_cache) X(v_cache) X(block_table) X(cache_seq_lens)       \
  X(position_ids) X(extend_context_length) X(sliding_window_size) X(sink_token_size) X(block_size_k) X(require_stage_caches)   \
  X(require_cache_statistics) X(mask_only) X(block_sparse_block_size_q) X(model_context_length) X(disable_flashdecode)         \
  X(logit_softcap) X(using_paged_cache) X(update_flags) X(stage_block_size_q) X(stage_block_stride_q) X(stage_chunk_size)      \
  X(stage_k) X(stage_stride) X(stage_extend_backend) X(require_realign_index) X(require_reset_score) X(require_post_sort)      \
  X(indices) X(ks) X(ks_count) X(ks_start_end) X(stage_caches) X(indices_left) X(indices_right) X(out_scores) X(mark)          \
  X(_heads_share) X(_left32) X(_right32) X(current_stream) X(wait_event)
struct Names {
#define X(n) PyObject* n;
  NAMES(X)
#undef X
} N;

// the package's classes (set by bind())
struct Classes {
  PyObject *ScanStage, *Metadata, *StageCache, *Statistics, *LibError, *torch_cuda;
} K;

Ref attr(PyObject* o, PyObject* name) { return checked(PyObject_GetAttr(o, name)); }
// the attribute, or an empty reference when there is none
Ref attr_opt(PyObject* o, PyObject* name) {
  PyObject* r = PyObject_GetAttr(o, name);
  if (!r) {
    if (!PyErr_ExceptionMatches(PyExc_AttributeError)) throw PyError{};
    PyErr_Clear();
  }
  return Ref(r);
}
bool truth(const Ref& r) {
  const int t = PyObject_IsTrue(r.get());
  if (t < 0) throw PyError{};
  return t != 0;
}
bool attr_true(PyObject* o, PyObject* name) { return truth(attr(o, name)); }
int64_t as_int(const Ref& r) {
  Ref i = checked(PyNumber_Index(r.get()));
  const long long v = PyLong_AsLongLong(i.get());
  if (v == -1 && PyErr_Occurred()) throw PyError{};
  return v;
}
int64_t attr_int(PyObject* o, PyObject* name) { return as_int(attr(o, name)); }
double attr_num(PyObject* o, PyObject* name) {
  const double v = PyFloat_AsDouble(attr(o, name).get());
  if (v == -1.0 && PyErr_Occurred()) throw PyError{};
  return v;
}
const char* as_text(const Ref& r) {
  if (r.none()) return "None";
  const char* s = PyUnicode_Check(r.get()) ? PyUnicode_AsUTF8(r.get()) : "?";
  if (!s) throw PyError{};
  return s;
}
// a tensor attribute or argument, or an undefined tensor for None
at::Tensor tensor_of(PyObject* o, const char* what) {
  if (o == nullptr || o == Py_None) return at::Tensor();
  if (!THPVariable_Check(o)) fail(PyExc_TypeError, "%s must be a torch.Tensor or None", what);
  return THPVariable_Unpack(o);
}
at::Tensor attr_tensor(PyObject* o, PyObject* name, const char* what) { return tensor_of(attr(o, name).get(), what); }
PyObject* wrap(const at::Tensor& t) {
  if (!t.defined()) Py_RETURN_NONE;
  return THPVariable_Wrap(t);
}

// ---------------------------------------------------------------------------------------------------------------------
// small helpers
// ---------------------------------------------------------------------------------------------------------------------
int64_t cdiv(int64_t a, int64_t b) { return (a + b - 1) / b; }
int64_t next_pow2(int64_t x) {
  int64_t p = 1;
  while (p < x) p <<= 1;
  return p;
}
void check(int rc, const char* what) {
  if (rc == HIPATTN_OK) return;
  const char* msg = hipattn_error_string();
  if (rc == HIPATTN_ERR_INVALID) VALUE_ERROR("%s: %s", what, msg);
  if (rc == HIPATTN_ERR_UNSUPPORTED) NOT_BUILT("%s: %s", what, msg);
  fail(K.LibError, "%s: %s (code %d)", what, msg, rc);
}
const char* env(const char* name, const char* otherwise) {
  const char* v = getenv(name);
  return v ? v : otherwise;
}
bool is_fp8(at::ScalarType t) { return t == at::kFloat8_e5m2 || t == at::kByte; }
int dtype_of(at::ScalarType t) {
  switch (t) {
    case at::kFloat: return HIPATTN_F32;
    case at::kHalf: return HIPATTN_F16;
    case at::kBFloat16: return HIPATTN_BF16;
    default: return -1;
  }
}
std::string shape_text(const at::Tensor& t) {
  std::string s = "(";
  for (int64_t i = 0; i < t.dim(); ++i) s += (i ? ", " : "") + std::to_string(t.size(i));
  return s + ")";
}
float round_to(float x, int dt) {
  if (dt == HIPATTN_F16) return (float)c10::Half(x);
  if (dt == HIPATTN_BF16) return (float)c10::BFloat16(x);
  return x;
}

struct Device {
  c10::Device dev;
  std::vector<at::Tensor>* keep = nullptr;   // a call beside the current stream: holds its memory until the streams have joined
  at::Tensor empty(at::IntArrayRef sizes, at::ScalarType t) const {
    at::Tensor x = at::detail::empty_cuda(sizes, t, dev, c10::nullopt);
    if (keep) keep->push_back(x);
    return x;
  }
};

// Calls that do not depend on one another run beside the current stream: fork() marks the point they start from, forward()
// with the fork launches on a stream of the pool, join() makes the current stream wait for all of them.  Memory still
// belongs to the current stream; what the calls allocate is held until the join, so nothing is reused under them.
struct Fork {
  c10::Device dev{at::kCUDA, 0};
  c10::cuda::CUDAStream main;
  cudaEvent_t start = nullptr;
  std::vector<cudaEvent_t> done;
  std::vector<at::Tensor> keep;
  explicit Fork(c10::Device d) : dev(d), main(c10::cuda::getCurrentCUDAStream(d.index())) {}
  ~Fork() {
    join();
    if (start) cudaEventDestroy(start);
  }
  void join() {
    for (cudaEvent_t e : done) {
      cudaStreamWaitEvent(main.stream(), e, 0);
      cudaEventDestroy(e);
    }
    done.clear();
    keep.clear();
  }
};
void cuda_ok(cudaError_t e, const char* what) {
  if (e != cudaSuccess) fail(PyExc_RuntimeError, "%s: %s", what, cudaGetErrorString(e));
}
const char* kForkName = "hip_attention_b200.fork";
void drop_fork(PyObject* o) { delete (Fork*)PyCapsule_GetPointer(o, kForkName); }
// the launches of one call on a stream of the pool; the end is marked however the call ends
struct Beside {
  Fork* fork = nullptr;
  cudaStream_t stream = nullptr;
  void begin(Fork* f) {
    stream = c10::cuda::getStreamFromPool(false, f->dev.index()).stream();
    cuda_ok(cudaStreamWaitEvent(stream, f->start, 0), "cudaStreamWaitEvent");
    fork = f;
  }
  // work given to the current stream in between comes first
  void after_current() {
    if (!fork) return;
    cudaEvent_t e;
    cuda_ok(cudaEventCreateWithFlags(&e, cudaEventDisableTiming), "cudaEventCreate");
    cudaEventRecord(e, fork->main.stream());
    cudaStreamWaitEvent(stream, e, 0);
    cudaEventDestroy(e);
  }
  ~Beside() {
    if (!fork) return;
    cudaEvent_t e;
    if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess) {
      cudaEventRecord(e, stream);
      fork->done.push_back(e);
    } else {
      cudaStreamSynchronize(stream);
    }
  }
};

// Device status word (one int32 per device) the kernels OR their HIPATTN_STATUS_* bits into.
std::mutex g_status_mutex;
std::unordered_map<int, at::Tensor> g_status;
at::Tensor status_word(int index) {
  std::lock_guard<std::mutex> lock(g_status_mutex);
  at::Tensor& t = g_status[index];
  if (!t.defined()) t = at::zeros({1}, at::TensorOptions().dtype(at::kInt).device(at::kCUDA, index));
  return t;
}

hipattn_tokens_t tokens(const at::Tensor& dense, const at::Tensor& cache, const at::Tensor& table, const at::Tensor& lens, const char* what) {
  hipattn_tokens_t t;
  memset(&t, 0, sizeof(t));
  if (cache.defined()) {
    if (cache.dim() != 4 || cache.stride(3) != 1) VALUE_ERROR("%s_cache must be [n_pages, page_size, kv_heads, head_dim] with a contiguous last dim", what);
    if (!table.defined() || table.dim() != 2 || !lens.defined() || lens.dim() != 1)
      VALUE_ERROR("paged KV needs block_table [B, pages] and cache_seq_lens [B]");
    for (const at::Tensor* x : {&table, &lens})
      if (x->scalar_type() != at::kInt && x->scalar_type() != at::kLong) VALUE_ERROR("block_table and cache_seq_lens must be int32 or int64");
    if (table.stride(1) != 1) VALUE_ERROR("block_table rows must be contiguous");
    if (!lens.is_contiguous()) VALUE_ERROR("cache_seq_lens must be contiguous");
    t.cache = cache.data_ptr();
    t.fp8_e5m2 = is_fp8(cache.scalar_type());
    t.stride_page = cache.stride(0);
    t.stride_off = cache.stride(1);
    t.stride_ch = cache.stride(2);
    t.block_table = table.data_ptr();
    t.table_stride_b = table.stride(0);
    t.cache_seq_lens = lens.data_ptr();
    t.n_pages = cache.size(0);
    t.table_width = (int32_t)table.size(1);
    t.table_is_i64 = table.scalar_type() == at::kLong;
    t.seq_lens_is_i64 = lens.scalar_type() == at::kLong;
    t.page_size = (int32_t)cache.size(1);
  } else {
    if (!dense.defined()) VALUE_ERROR("%s is None and no %s_cache was given", what, what);
    if (dense.dim() != 4 || dense.stride(3) != 1) VALUE_ERROR("%s must be [B, T, kv_heads, head_dim] with a contiguous last dim", what);
    t.dense = dense.data_ptr();
    t.fp8_e5m2 = is_fp8(dense.scalar_type());
    t.stride_b = dense.stride(0);
    t.stride_t = dense.stride(1);
    t.stride_h = dense.stride(2);
  }
  return t;
}

struct StageArgs {
  int64_t bq, stride, chunk, k;   // k: tokens kept before this stage (-1: None)
  int rope_mode;
};
int rope_mode_of(const Ref& name) {
  const char* s = as_text(name);
  if (!strcmp(s, "relative")) return HIPATTN_ROPE_RELATIVE;
  if (!strcmp(s, "streaming")) return HIPATTN_ROPE_STREAMING;
  NOT_BUILT("scan_extend_backend '%s' is not built (relative, streaming)", s);
}

int scan_mode() {
  const char* m = env("HIPATTN_SCAN_MODE", "auto");
  if (!strcmp(m, "auto")) return HIPATTN_SCAN_AUTO;
  if (!strcmp(m, "strict")) return HIPATTN_SCAN_STRICT;
  if (!strcmp(m, "check")) return HIPATTN_SCAN_CHECK;
  VALUE_ERROR("HIPATTN_SCAN_MODE='%s': expected auto, strict or check", m);
}

// several tensors copied (and converted) in one launch
int copy_type(at::ScalarType t) {
  switch (t) {
    case at::kLong: return hipattn::COPY_I64;
    case at::kInt: return hipattn::COPY_I32;
    case at::kUInt32: return hipattn::COPY_U32;
    case at::kFloat: return hipattn::COPY_F32;
    case at::kBFloat16: return hipattn::COPY_BF16;
    default: return -1;
  }
}
struct Copies {
  hipattn::CopyList list{};
  cudaStream_t stream;
  explicit Copies(cudaStream_t s) : stream(s) {}
  void add(const hipattn::CopySeg& s) {
    if (s.n0 * s.n1 * s.n2 == 0) return;
    if (list.count == hipattn::kMaxCopies) flush();
    list.seg[list.count++] = s;
  }
  // contiguous dst <- src of the same shape
  void add(const at::Tensor& src, const at::Tensor& dst) {
    hipattn::CopySeg s{};
    s.src = src.data_ptr();
    s.dst = dst.data_ptr();
    s.src_type = copy_type(src.scalar_type());
    s.dst_type = copy_type(dst.scalar_type());
    if (s.src_type < 0 || s.dst_type < 0) fail(PyExc_TypeError, "metadata tensors must be int32, int64, uint32, float32 or bfloat16");
    if (src.is_contiguous()) {
      s.n0 = s.n1 = 1;
      s.n2 = src.numel();
      s.plain = 1;
      add(s);
      return;
    }
    std::vector<int64_t> n, st;   // outer dimensions of equal stride merged
    for (int64_t i = 0; i < src.dim(); ++i) {
      if (src.size(i) == 1) continue;
      if (!n.empty() && st.back() == src.stride(i) * src.size(i)) { n.back() *= src.size(i); st.back() = src.stride(i); }
      else { n.push_back(src.size(i)); st.push_back(src.stride(i)); }
    }
    while (n.size() < 3) { n.insert(n.begin(), 1); st.insert(st.begin(), 0); }
    strided(s, src.element_size(), dst.element_size(), n.data(), st.data(), n.size());
  }
  // a segment takes three dimensions: more are dealt out slice by slice (no copy in between, which would have to outlive the launch)
  void strided(hipattn::CopySeg s, int64_t src_bytes, int64_t dst_bytes, const int64_t* n, const int64_t* st, size_t dims) {
    if (dims > 3) {
      int64_t inner = 1;
      for (size_t i = 1; i < dims; ++i) inner *= n[i];
      for (int64_t i = 0; i < n[0]; ++i) {
        strided(s, src_bytes, dst_bytes, n + 1, st + 1, dims - 1);
        s.src = (const char*)s.src + st[0] * src_bytes;
        s.dst = (char*)s.dst + inner * dst_bytes;
      }
      return;
    }
    s.n0 = n[0]; s.n1 = n[1]; s.n2 = n[2];
    for (int i = 0; i < 3; ++i) s.src_s[i] = st[i];
    s.dst_s[0] = n[1] * n[2]; s.dst_s[1] = n[2]; s.dst_s[2] = 1;
    add(s);
  }
  void flush(bool early = false) {
    if (list.count) check(hipattn::multi_copy(list, stream, early), "multi_copy");
    list.count = 0;
  }
};

// ---------------------------------------------------------------------------------------------------------------------
// one call
// ---------------------------------------------------------------------------------------------------------------------
struct Call {
  PyObject *args, *debug, *reduce, *timer;
  at::Tensor q, q_attn, k, v, k_scan, k_cache, v_cache, table, lens, pos, rope_cos, rope_sin;
  std::vector<StageArgs> stages;
  int64_t B, TQ, H, D, T, HKV, sink, sw, second_k;
  int dt;
  bool using_extend;
  Device dv{c10::Device(at::kCUDA, 0)};
  cudaStream_t stream;
  uint32_t* status;
  // Calls that a prefill chunk is split into read the same keys: what they prepare from them is handed on in this dict
  // (None: a call of its own), valid for the positions and the windows it names.
  PyObject* shared = Py_None;
  hipattn::QueryPositions where{};   // positions that prepared tables and keys have to reach
  at::Tensor last_pos;               // [B] largest of them

  at::Tensor shared_get(const char* name) const {
    PyObject* v = shared == Py_None ? nullptr : PyDict_GetItemString(shared, name);
    return v ? tensor_of(v, name) : at::Tensor();
  }
  void shared_set(const char* name, const at::Tensor& t) const {
    if (shared == Py_None || !t.defined()) return;
    Ref v = checked(wrap(t));
    if (PyDict_SetItemString(shared, name, v.get()) < 0) throw PyError{};
  }

  void mark(const char* name) {
    if (timer == Py_None) return;
    Ref r = checked(PyObject_CallMethod(timer, "mark", "s", name));
  }
};

void read_stages(Call& c) {
  Ref list = attr(c.args, N.stages);
  Ref seq = checked(PySequence_Fast(list.get(), "args.stages must be a list"));
  const Py_ssize_t n = PySequence_Fast_GET_SIZE(seq.get());
  if (n == 0) VALUE_ERROR("args.stages is empty");
  Ref scan_backend = attr(c.args, N.scan_extend_backend);
  if (c.using_extend) {
    if (attr(c.args, N.rope_cos).none() || attr(c.args, N.rope_sin).none()) VALUE_ERROR("using_extend needs rope_cos and rope_sin");
    Ref sa = attr(c.args, N.sa_extend_backend);
    if (strcmp(as_text(sa), "streaming")) NOT_BUILT("sa_extend_backend '%s' is not built (streaming)", as_text(sa));
  }
  for (Py_ssize_t i = 0; i < n; ++i) {
    PyObject* st = PySequence_Fast_GET_ITEM(seq.get(), i);
    StageArgs s;
    s.rope_mode = HIPATTN_ROPE_NONE;
    if (c.using_extend) {
      Ref own = attr_opt(st, N.stage_extend_backend);
      s.rope_mode = rope_mode_of(own.none() || !truth(own) ? scan_backend : own);
    }
    const int is = PyObject_IsInstance(st, K.ScanStage);
    if (is < 0) throw PyError{};
    if (!is) NOT_BUILT("stage %d: only ScanStage is built (%s given)", (int)i, Py_TYPE(st)->tp_name);
    if (attr_num(st, N.stage_stride) != 1) NOT_BUILT("stage_stride != 1 is not built");
    // the selection kernel always realigns, resets the scores and sorts by position; the reference does each only when
    // the stage asks for it (attention_extend.py:2075-2090, 2638)
    if (i > 0 && !(attr_true(st, N.require_realign_index) && attr_true(st, N.require_reset_score) && attr_true(st, N.require_post_sort)))
      NOT_BUILT("stage %d: require_realign_index / require_reset_score / require_post_sort = False is not built", (int)i);
    s.bq = attr_int(st, N.stage_block_size_q);
    s.stride = attr_int(st, N.stage_block_stride_q);
    s.chunk = attr_int(st, N.stage_chunk_size);
    Ref k = attr(st, N.stage_k);
    s.k = k.none() ? -1 : as_int(k);
    if (s.bq <= 0 || s.stride <= 0 || s.chunk <= 0) VALUE_ERROR("stage %d: block size, stride and chunk size must be positive", (int)i);
    if (i > 0 && s.bq != c.stages[0].bq) NOT_BUILT("all stages must use the same stage_block_size_q");
    if (s.bq % s.stride) VALUE_ERROR("stage %d: stage_block_size_q must be a multiple of stage_block_stride_q", (int)i);
    c.stages.push_back(s);
  }
  if (c.stages[0].k >= 0) VALUE_ERROR("first stage always quadratic: stages[0].stage_k must be None");
  for (size_t i = 1; i < c.stages.size(); ++i) {
    const StageArgs &p = c.stages[i - 1], &s = c.stages[i];
    if (s.k < 0 || s.k % p.chunk) VALUE_ERROR("stage %d: stage_k %lld must be a multiple of the previous chunk size", (int)i, (long long)s.k);
    if (p.chunk % s.chunk) VALUE_ERROR("stage %d: chunk size %lld must divide %lld", (int)i, (long long)s.chunk, (long long)p.chunk);
  }
  c.second_k = attr_int(c.args, N.second_stage_k);
  if (c.second_k % c.stages.back().chunk) VALUE_ERROR("second_stage_k must be a multiple of the last stage_chunk_size");
}

// what the build does not have is refused before anything is launched
void reject_unsupported(Call& c) {
  PyObject* a = c.args;
  if (!attr(a, N.offload_cache).none() || attr_true(a, N.online_update_cache))
    NOT_BUILT("host-offloaded KV (offload_cache / online_update_cache) is not part of this build");
  c.using_extend = attr_true(a, N.using_extend);
  if (c.using_extend != attr_true(a, N.need_apply_rope))
    NOT_BUILT("using_extend and need_apply_rope must be set together (rotation of already rotated q / k, attention_extend.py:299-323, is not built)");
  if (attr_num(a, N.low_percent) > 0 && attr_num(a, N.low_k_ratio) < 1) NOT_BUILT("low_percent / low_k_ratio is dead code in the reference and is not built");
  if (!attr_true(a, N.is_causal)) NOT_BUILT("is_causal=False is not built");
  if (attr_num(a, N.stage_early_terminate) != 1) NOT_BUILT("stage_early_terminate != 1 is not built");
  if (!attr(a, N.sliding_window_indices).none()) NOT_BUILT("sliding_window_indices is not built");
  if (strcmp(env("HIP_HEAD_REDUCE", "1"), "1")) NOT_BUILT("HIP_HEAD_REDUCE=0 (per-head masks) is not built");
  for (const char* name : {"HIP_DEBUG_TOPKMEAN", "HIP_DEBUG_UNION_HEAD", "HIP_DEBUG_ADD_DELAY_WINDOW", "HIP_DEBUG_SNAP_KV", "APPLY_V_DOT", "HIP_CUMSUM"})
    if (!strcmp(env(name, "0"), "1")) NOT_BUILT("%s=1 selects a research branch of the reference that is not built", name);
  read_stages(c);
}

void check_inputs(Call& c, const at::Tensor& q_mask, const at::Tensor& k_mask) {
  const at::Tensor& q = c.q;
  if (!q.is_cuda())
    fail(PyExc_RuntimeError, "hip_attention_12 runs on a CUDA device only (B200, sm_100a); q is on %s", q.device().str().c_str());
  c.dt = dtype_of(q.scalar_type());
  if (c.dt < 0) NOT_BUILT("q dtype %s is not built (float32, float16, bfloat16)", c10::toString(q.scalar_type()));
  if (q.stride(3) != 1) VALUE_ERROR("q must have a contiguous last dim");
  if (c.k.defined() != c.v.defined()) VALUE_ERROR("k and v must both be given or both be None");
  struct { const char* name; const at::Tensor* t; bool kv; } all[] = {{"k", &c.k, true}, {"v", &c.v, true}, {"k_cache", &c.k_cache, true},
                                                                      {"v_cache", &c.v_cache, true}, {"q_mask", &q_mask, false}, {"k_mask", &k_mask, false}};
  for (auto& x : all) {
    if (!x.t->defined()) continue;
    if (is_fp8(x.t->scalar_type()) && x.kv) {
      if (c.dt == HIPATTN_F32) NOT_BUILT("an fp8 (e5m2) KV cache needs float16 or bfloat16 queries");
    } else if (x.t->scalar_type() != q.scalar_type()) {
      NOT_BUILT("%s dtype %s differs from q dtype %s", x.name, c10::toString(x.t->scalar_type()), c10::toString(q.scalar_type()));
    }
    if (x.t->device() != q.device()) VALUE_ERROR("%s is on %s, q on %s", x.name, x.t->device().str().c_str(), q.device().str().c_str());
  }
  if (c.k.defined() && c.k.sizes() != c.v.sizes()) VALUE_ERROR("k and v must have the same shape");
  if (c.k.defined() && is_fp8(c.k.scalar_type()) != is_fp8(c.v.scalar_type())) NOT_BUILT("k and v must both be fp8 or both be q's dtype");
  if (c.k_cache.defined() && c.v_cache.defined() && is_fp8(c.k_cache.scalar_type()) != is_fp8(c.v_cache.scalar_type()))
    NOT_BUILT("k_cache and v_cache must both be fp8 or both be q's dtype");
  if (!c.k.defined() && !c.k_cache.defined()) VALUE_ERROR("k is None and args.k_cache is None");
  if (c.k_cache.defined() && !c.v_cache.defined()) VALUE_ERROR("k_cache without v_cache");
}

const int32_t* last_positions(Call& c) {
  if (!c.last_pos.defined()) c.last_pos = c.shared_get("last_pos");
  if (!c.last_pos.defined()) {
    c.last_pos = c.dv.empty({c.where.B}, at::kInt);
    check(hipattn::last_positions(c.where, c.last_pos.data_ptr<int32_t>(), c.stream), "last_positions");
    c.shared_set("last_pos", c.last_pos);
  }
  return c.last_pos.data_ptr<int32_t>();
}

// cos / sin [rows, >= D / 2] in q's element type, rows of whole 16-byte pieces (the kernels cast the tables to the
// element type before use, attention_extend.py:308-321; doing it once here is the same arithmetic)
at::Tensor rope_table(const Call& c, const at::Tensor& given) {
  at::Tensor t = given;
  if (t.dim() != 2 || t.size(1) < c.D / 2) VALUE_ERROR("rope tables must be [positions, >= head_dim / 2], got %s", shape_text(t).c_str());
  if (t.device() != c.q.device()) VALUE_ERROR("rope table on %s, q on %s", t.device().str().c_str(), c.q.device().str().c_str());
  t = t.to(c.q.scalar_type());
  if (t.stride(1) != 1 || t.stride(0) % 8 || (uintptr_t)t.data_ptr() % 16) {
    t = t.contiguous();
    if (t.size(1) % 8) {
      at::Tensor pad = at::zeros({t.size(0), cdiv(t.size(1), 8) * 8}, t.options());
      pad.narrow(1, 0, t.size(1)).copy_(t);
      t = pad;
    }
  }
  return t;
}

// The call's rope tables.  fp32 tables with 16-bit queries, the usual case, are converted as far as the call can reach into
// them: a query or key is never rotated to a position beyond the largest query position, except by the scan, whose
// positions end at the number of chunks of a stage + the window.
void set_rope_tables(Call& c, int64_t restart_chunks) {
  c.rope_cos = c.shared_get("rope_cos");
  c.rope_sin = c.shared_get("rope_sin");
  if (c.rope_cos.defined()) return;
  const at::Tensor cos = attr_tensor(c.args, N.rope_cos, "rope_cos"), sin = attr_tensor(c.args, N.rope_sin, "rope_sin");
  auto plain = [&](const at::Tensor& t) {
    return t.defined() && t.dim() == 2 && t.size(1) >= c.D / 2 && t.scalar_type() == at::kFloat && t.device() == c.q.device() && t.stride(1) == 1 &&
           t.stride(0) % 4 == 0 && (uintptr_t)t.data_ptr() % 16 == 0 && t.size(0) > 0 && t.size(0) < (1 << 30);
  };
  if (c.dt == HIPATTN_F32 || c.D % 16 || !plain(cos) || !plain(sin) || cos.size(0) != sin.size(0) || cos.stride(0) != sin.stride(0)) {
    c.rope_cos = rope_table(c, cos);
    c.rope_sin = rope_table(c, sin);
  } else {
    auto reach = [&](int64_t sw) {   // last row of a scan with this window
      const int64_t c0 = c.stages[0].chunk;
      int64_t n = cdiv(std::max<int64_t>(0, c.T - c.sink - sw), c0), most = std::max(n, restart_chunks);
      for (size_t i = 1; i < c.stages.size(); ++i) {
        n = std::min(c.stages[i].k / c.stages[i - 1].chunk, n) * (c.stages[i - 1].chunk / c.stages[i].chunk);
        most = std::max(most, n);
      }
      return most + std::max<int64_t>(0, sw - c0) + 1;
    };
    int64_t floor = reach(c.sw);
    if (PyObject* windows = c.shared == Py_None ? nullptr : PyDict_GetItemString(c.shared, "windows")) {   // of the calls that use these tables
      Ref all = checked(PySequence_Fast(windows, "windows must be a list"));
      for (Py_ssize_t i = 0; i < PySequence_Fast_GET_SIZE(all.get()); ++i)
        floor = std::max(floor, reach(as_int(Ref::borrow(PySequence_Fast_GET_ITEM(all.get(), i)))));
    }
    at::Tensor both = c.dv.empty({2, cos.size(0), c.D / 2}, c.q.scalar_type());
    hipattn::RopeTables t{};
    t.cos = cos.data_ptr<float>();
    t.sin = sin.data_ptr<float>();
    t.row_stride = cos.stride(0);
    t.rows = (int)cos.size(0);
    t.cols = (int)c.D / 2;
    t.dtype = c.dt;
    t.floor = (int)std::min<int64_t>(floor, 1 << 30);
    t.q = c.where;
    if (c.last_pos.defined() || c.where.B * (int64_t)c.where.TQ > 2048) t.last_pos = last_positions(c);
    t.dst = both.data_ptr();
    check(hipattn::convert_rope_tables(t, c.stream), "convert_rope_tables");
    c.rope_cos = both.select(0, 0);
    c.rope_sin = both.select(0, 1);
  }
  c.shared_set("rope_cos", c.rope_cos);
  c.shared_set("rope_sin", c.rope_sin);
}

struct Mask {
  at::Tensor indices, ks, kse;
  std::vector<at::Tensor> left32, right32, left64, right64;   // inputs of stage i (empty for stage 0 and cached stages)
  at::Tensor consts;
  bool heads_share;
};

// Runs the scan stages (attention_extend.py:2012-2776).
Mask estimate_mask(Call& c, const hipattn_tokens_t& ktok, int64_t first, at::Tensor left, at::Tensor right, bool want_inputs,
                   const at::Tensor& access, hipattn::BeginCall& begin) {
  const Device& dv = c.dv;
  const int64_t bq = c.stages[0].bq, BDST = cdiv(c.TQ, bq), rows = c.B * BDST;
  const int64_t c0 = c.stages[0].chunk, scan_window = std::max<int64_t>(0, c.sw - c0);
  const size_t n_st = c.stages.size();
  Mask out;
  out.left32.resize(n_st); out.right32.resize(n_st); out.left64.resize(n_st); out.right64.resize(n_st);
  int64_t n;
  at::Tensor score;
  if (first > 0) {
    n = left.size(1);
  } else {
    n = cdiv(std::max<int64_t>(0, c.T - c.sink - c.sw), c0);
    at::Tensor two = dv.empty({2, rows, n}, at::kInt);
    left = two.select(0, 0);
    right = two.select(0, 1);
    begin.left = left.data_ptr<int32_t>();
    begin.right = right.data_ptr<int32_t>();
  }
  if (n > HIPATTN_MAX_CHUNKS) NOT_BUILT("%lld chunks per query block exceed the on-chip selection limit of %d", (long long)n, HIPATTN_MAX_CHUNKS);
  score = dv.empty({rows, n}, at::kInt);
  begin.score_max = score.data_ptr<int32_t>();
  begin.rows = rows;
  begin.n = n;
  begin.sink = (int)c.sink; begin.chunk = (int)c0; begin.T = (int)c.T; begin.scan_window = (int)scan_window;
  if (want_inputs) {
    out.consts = dv.empty({(int64_t)n_st}, at::kFloat);
    begin.consts = out.consts.data_ptr<float>();
    begin.n_const = (int64_t)n_st;
  }
  check(hipattn::begin_call(begin, c.stream), "begin_call");

  // Query / key scales of the scan (attention_extend.py:924-940), rounded to the element type
  const float s_ = std::sqrt((float)c.D), ss_ = std::sqrt(s_);
  const float q_scale = round_to(s_ / ss_, c.dt), k_scale = round_to(1.0f / ss_, c.dt);
  const int mode = scan_mode();

  // scaled keys and their magnitudes (error radius) for the tensor-core scan (16-bit prefill only), once per call.
  // With in-kernel RoPE the stages whose backend is "relative" get two copies (keys rotated to table position 0 / 1 for
  // the left / right candidate); "streaming" stages (a key is rotated to its chunk's index, which changes from stage to
  // stage) get the keys as they are in a head-major copy, and the scan kernel rotates and scales them in its operand
  // tile (head dim 128; other shapes stay on the strict kernel).
  at::Tensor key_abs, k_scaled, key_abs_plain, k_plain;
  bool rows16 = true, any_relative = false, any_streaming = false;
  for (const StageArgs& s : c.stages) rows16 = rows16 && (s.bq / s.stride) % 16 == 0 && s.bq / s.stride >= 16;
  for (size_t i = first; i < n_st; ++i) {
    any_relative |= c.stages[i].rope_mode == HIPATTN_ROPE_RELATIVE;
    any_streaming |= c.stages[i].rope_mode == HIPATTN_ROPE_STREAMING;
  }
  bool tensor_scan = c.dt != HIPATTN_F32 && (c.D == 64 || c.D == 128) && std::min(c.TQ, bq) > 1 && mode != HIPATTN_SCAN_STRICT && rows16 && n > 0;
  int sides = 1;
  bool want_plain = false;
  const int64_t key_rows = c.B * c.T * c.HKV, limit = (1ll << 31) - 1;
  if (tensor_scan && c.using_extend) {
    sides = 2;
    want_plain = c.D == 128 && any_streaming && key_rows < limit;
    tensor_scan = any_relative && 2 * key_rows < limit;
  }
  if (tensor_scan || want_plain) {
    c.mark("start");
    // Tokens up to the last query position and the rest of its chunk (a server hands over its model's whole context length);
    // a restart's first list is the caller's, so all of them.
    check(hipattn::validate_tokens(ktok, 2, (int)c.D, "k"), "scan_prepare_keys");
    auto prepare = [&](const char* abs_name, const char* copy_name, at::Tensor& abs, at::Tensor& copy, int copies, bool rope, float scale) {
      abs = c.shared_get(abs_name);
      copy = c.shared_get(copy_name);
      if (abs.defined()) return;
      abs = dv.empty({copies, c.B, c.HKV, c.T}, at::kFloat);
      if (copies * key_rows < limit) copy = dv.empty({copies, c.B, c.HKV, c.T, c.D}, c.q.scalar_type());
      // (table position -1: both copies, rotated to positions 0 and 1, from one read of the keys)
      check(hipattn::scan_prepare_keys(ktok, c.dt, (int)c.D, (int)c.B, (int)c.T, (int)c.HKV, scale, abs.data_ptr<float>(),
                                       copy.defined() ? copy.data_ptr() : nullptr, c.status, c.stream, rope ? c.rope_cos.data_ptr() : nullptr,
                                       rope ? c.rope_sin.data_ptr() : nullptr, rope ? c.rope_cos.stride(0) : 0, rope ? (int)c.rope_cos.size(0) : 0, -1,
                                       first == 0 ? last_positions(c) : nullptr, (int)c0), "scan_prepare_keys");
      c.shared_set(abs_name, abs);
      c.shared_set(copy_name, copy);
    };
    if (tensor_scan) prepare("key_abs", "k_scaled", key_abs, k_scaled, sides, c.using_extend, k_scale);
    // scale 1: the copy holds the keys' own values
    if (want_plain) prepare("key_abs_plain", "k_plain", key_abs_plain, k_plain, 1, false, 1.0f);
    c.mark("prep");
  }

  int64_t block_chunk = attr_int(c.args, N.block_size_k);
  const int64_t c_last = c.stages.back().chunk;
  const bool per_head_final = c.sink % c_last != 0;
  const bool debug = c.debug != Py_None;
  uint64_t* stats = nullptr;
  at::Tensor stats_t;
  if (debug) {
    PyObject* st = PyDict_GetItemString(c.debug, "scan_stats");
    if (st) { stats_t = tensor_of(st, "scan_stats"); stats = (uint64_t*)stats_t.data_ptr(); }
  }
  out.heads_share = !per_head_final;
  if (n == 0) {   // nothing to scan: K shorter than sink + window
    out.indices = dv.empty({c.B * c.H, BDST, 0}, at::kLong);
    out.ks = at::zeros({c.B * c.H, BDST}, out.indices.options());
    out.kse = at::zeros({c.B * c.H, BDST, 2}, out.indices.options().dtype(at::kInt));
    return out;
  }
  for (size_t i = first; i < n_st; ++i) {
    const StageArgs& st = c.stages[i];
    if (i > (size_t)first && want_inputs) { out.left32[i] = left; out.right32[i] = right; }
    block_chunk = std::max<int64_t>(16, next_pow2(std::min(n, block_chunk)));
    const bool last = i + 1 == n_st;
    at::Tensor left_out, right_out, score_out;
    if ((last && per_head_final) || debug) left_out = dv.empty({rows, c.H, n}, at::kInt);
    if (debug) {
      right_out = dv.empty({rows, c.H, n}, at::kInt);
      score_out = dv.empty({rows, c.H, n}, at::kFloat);
    }
    hipattn_scan_params_t sp;
    memset(&sp, 0, sizeof(sp));
    sp.q = c.q.data_ptr();
    sp.q_stride_b = c.q.stride(0); sp.q_stride_t = c.q.stride(1); sp.q_stride_h = c.q.stride(2);
    sp.pos = c.pos.data_ptr<int64_t>();
    sp.pos_stride_b = c.pos.stride(0); sp.pos_stride_t = c.pos.stride(1);
    sp.k = ktok;
    sp.left = left.data_ptr<int32_t>();
    sp.right = right.data_ptr<int32_t>();
    sp.score_max = score.data_ptr<int32_t>();
    if (left_out.defined()) sp.left_out = left_out.data_ptr<int32_t>();
    if (right_out.defined()) sp.right_out = right_out.data_ptr<int32_t>();
    if (score_out.defined()) sp.score_out = score_out.data_ptr<float>();
    sp.status = c.status;
    if (st.rope_mode != HIPATTN_ROPE_STREAMING) {
      if (key_abs.defined()) sp.key_abs = key_abs.data_ptr<float>();
      if (k_scaled.defined()) { sp.k_scaled = k_scaled.data_ptr(); sp.k_scaled_sides = sides; }
    } else if (k_plain.defined()) {   // the plain copy, rotated and scaled inside the scan kernel
      sp.key_abs = key_abs_plain.data_ptr<float>();
      sp.k_scaled = k_plain.data_ptr();
      sp.k_scaled_sides = 1;
    }
    sp.dtype = c.dt; sp.D = (int)c.D; sp.B = (int)c.B; sp.TQ = (int)c.TQ; sp.H = (int)c.H; sp.HKV = (int)c.HKV; sp.T = (int)c.T;
    sp.block_size_q = (int)bq; sp.stride_q = (int)st.stride;
    sp.n_chunks = (int)n; sp.block_chunk = (int)block_chunk; sp.scan_window = (int)scan_window;
    sp.q_scale = q_scale; sp.k_scale = k_scale;
    sp.mode = mode;
    sp.chunk_size = (int)st.chunk;
    if (access.defined()) {
      sp.access_counter = access.data_ptr<int32_t>();
      sp.access_n = (int)access.size(2);
      sp.access_stride_b = access.stride(0); sp.access_stride_h = access.stride(1);
    }
    if (c.using_extend) {
      sp.rope_cos = c.rope_cos.data_ptr(); sp.rope_sin = c.rope_sin.data_ptr();
      sp.rope_stride = c.rope_cos.stride(0); sp.rope_rows = (int)c.rope_cos.size(0);
      sp.rope_mode = st.rope_mode;
    }
    sp.stats = stats;
    c.mark("start");
    // (a caller's own list, which a restart begins with, may hold a chunk twice, and so may what is selected from it)
    const int64_t scratch_bytes = i > 0 && first == 0 ? hipattn::scan_key_tiles_scratch(sp, (int)c.sink, (int)c.stages[i - 1].chunk) : 0;
    at::Tensor scratch;
    if (scratch_bytes > 0) {
      try {
        scratch = dv.empty({scratch_bytes}, at::kByte);
      } catch (const c10::OutOfMemoryError&) {   // the general scan needs none
      }
    }
    if (scratch.defined()) {
      check(hipattn::scan_key_tiles(sp, (int)c.sink, (int)c.stages[i - 1].chunk, scratch.data_ptr(), c.stream), ("scan_stage[" + std::to_string(i) + "]").c_str());
    } else {
      check(hipattn_scan_stage(&sp, c.stream), ("scan_stage[" + std::to_string(i) + "]").c_str());
    }
    c.mark(("scan" + std::to_string(i)).c_str());
    if (c.reduce != Py_None) {
      Ref s = checked(wrap(score));
      Ref r = checked(PyObject_CallOneArg(c.reduce, s.get()));
      c.mark("reduce");
    }
    if (debug) {
      PyObject* list = PyDict_GetItemString(c.debug, "stages");
      if (!list) {
        Ref l = checked(PyList_New(0));
        if (PyDict_SetItemString(c.debug, "stages", l.get()) < 0) throw PyError{};
        list = l.get();
      }
      Ref d = checked(PyDict_New());
      struct { const char* k; at::Tensor* t; } items[] = {{"left_in", &left}, {"right_in", &right}, {"left", &left_out}, {"right", &right_out},
                                                          {"score", &score_out}, {"score_max", &score}};
      for (auto& x : items) {
        Ref v = checked(wrap(*x.t));
        if (PyDict_SetItemString(d.get(), x.k, v.get()) < 0) throw PyError{};
      }
      Ref bc = checked(PyLong_FromLongLong(block_chunk));
      if (PyDict_SetItemString(d.get(), "block_chunk", bc.get()) < 0 || PyList_Append(list, d.get()) < 0) throw PyError{};
    }
    if (!last) {
      const StageArgs& nx = c.stages[i + 1];
      const int64_t keep = std::min(nx.k / st.chunk, n), split = st.chunk / nx.chunk, n2 = keep * split;
      if (n2 > HIPATTN_MAX_CHUNKS) NOT_BUILT("%lld chunks per query block exceed the on-chip selection limit of %d", (long long)n2, HIPATTN_MAX_CHUNKS);
      at::Tensor three = dv.empty({3, rows, n2}, at::kInt), wide;
      int32_t* p3 = three.data_ptr<int32_t>();
      int64_t* pw = nullptr;
      if (want_inputs) {
        wide = dv.empty({2, rows, n2}, at::kLong);
        pw = wide.data_ptr<int64_t>();
      }
      check(hipattn::select_stage(score.data_ptr<int32_t>(), left.data_ptr<int32_t>(), rows, (int)n, (int)keep, (int)c.sink, (int)st.chunk, (int)nx.chunk,
                                  p3, p3 + rows * n2, p3 + 2 * rows * n2, pw, pw ? pw + rows * n2 : nullptr, c.stream),
            ("select_stage[" + std::to_string(i) + "]").c_str());
      c.mark("select");
      left = three.select(0, 0);
      right = three.select(0, 1);
      score = three.select(0, 2);
      if (want_inputs) { out.left64[i + 1] = wide.select(0, 0); out.right64[i + 1] = wide.select(0, 1); }
      n = n2;
    } else {
      const int64_t Kk = std::min(c.second_k / c_last, n);
      out.indices = dv.empty({c.B * c.H, BDST, Kk}, at::kLong);
      out.ks = dv.empty({c.B * c.H, BDST}, at::kLong);
      out.kse = dv.empty({c.B * c.H, BDST, 2}, at::kInt);
      const at::Tensor& lh = per_head_final ? left_out : left;
      check(hipattn_finalize_indices(score.data_ptr<int32_t>(), lh.data_ptr<int32_t>(), per_head_final ? c.H * n : n, per_head_final ? n : 0,
                                     c.pos.data_ptr<int64_t>(), c.pos.stride(0), c.pos.stride(1), (int)c.B, (int)BDST, (int)c.H, (int)n, (int)Kk, (int)c_last,
                                     (int)bq, out.indices.data_ptr<int64_t>(), out.ks.data_ptr<int64_t>(), out.kse.data_ptr<int32_t>(), c.stream),
            "finalize_indices");
      c.mark("select");
    }
  }
  return out;
}

struct AttentionArgs {
  int64_t window, block_k, bsa_bq, index_bq;
  bool heads_share, decode, want_lse, own_mask;
  bool beside;   // the launch before is an early multi_copy that the attention does not depend on
  float softcap;
};

// The attention over {sink, selected blocks, window}; fills out [B, TQ, H, D] and, on request, the base-2 log-sum-exp.
void attention(Call& c, const hipattn_tokens_t& ktok, const hipattn_tokens_t& vtok, const at::Tensor& indices, const at::Tensor& ks,
               const AttentionArgs& a, const at::Tensor& access, at::Tensor& out, at::Tensor& lse) {
  const Device& dv = c.dv;
  if (!out.defined()) out = dv.empty({c.B, c.TQ, c.H, c.D}, c.q_attn.scalar_type());
  if (a.want_lse && !lse.defined()) lse = dv.empty({c.B, c.TQ, c.H}, at::kFloat);
  const int64_t Kk = indices.size(2);
  hipattn_bsa_params_t bp;
  memset(&bp, 0, sizeof(bp));
  bp.q = c.q_attn.data_ptr();
  bp.q_stride_b = c.q_attn.stride(0); bp.q_stride_t = c.q_attn.stride(1); bp.q_stride_h = c.q_attn.stride(2);
  bp.out = out.data_ptr();
  bp.o_stride_b = out.stride(0); bp.o_stride_t = out.stride(1); bp.o_stride_h = out.stride(2);
  bp.pos = c.pos.data_ptr<int64_t>();
  bp.pos_stride_b = c.pos.stride(0); bp.pos_stride_t = c.pos.stride(1);
  bp.k = ktok; bp.v = vtok;
  // (an empty selection has no storage; ks is zero then and no entry is read)
  bp.indices = Kk ? indices.data_ptr<int64_t>() : ks.data_ptr<int64_t>();
  bp.idx_stride_n = Kk ? indices.stride(0) : 0; bp.idx_stride_d = Kk ? indices.stride(1) : 0;
  bp.ks = ks.data_ptr<int64_t>();
  bp.ks_stride_n = ks.stride(0); bp.ks_stride_d = ks.stride(1);
  bp.status = c.status;
  bp.dtype = c.dt; bp.D = (int)c.D; bp.B = (int)c.B; bp.TQ = (int)c.TQ; bp.H = (int)c.H; bp.HKV = (int)c.HKV; bp.T = (int)c.T;
  bp.block_size_q = (int)a.bsa_bq; bp.index_block_q = (int)a.index_bq; bp.block_size_k = (int)a.block_k; bp.K = (int)Kk;
  bp.sink = (int)c.sink; bp.window = (int)a.window;
  bp.heads_share_mask = a.heads_share || a.decode;
  bp.logit_softcap = a.softcap;
  at::Tensor order;
  bp.indices_ascending = 1;
  if (!a.own_mask) {   // a mask handed in may be a caller's own, its blocks in any order (decode takes them as they come)
    bp.indices_ascending = c.TQ > 1 && Kk > 0;
    if (bp.indices_ascending) {
      order = dv.empty({1}, at::kInt);
      bp.indices_order = order.data_ptr<int32_t>();
      check(hipattn::zero_memory(order.data_ptr(), 4, c.stream), "zero_memory");
      check(hipattn::check_order(bp.indices, bp.idx_stride_n, bp.idx_stride_d, bp.ks, bp.ks_stride_n, bp.ks_stride_d, (int)indices.size(0),
                                 (int)indices.size(1), (int)Kk, order.data_ptr<int32_t>(), c.stream), "check_order");
    }
  }
  if (c.using_extend) {
    bp.rope_cos = c.rope_cos.data_ptr(); bp.rope_sin = c.rope_sin.data_ptr();
    bp.rope_stride = c.rope_cos.stride(0); bp.rope_rows = (int)c.rope_cos.size(0);
  }
  if (access.defined())   // which tokens / pages the attention loads (require_cache_statistics)
    check(hipattn_mark_attention_access(&bp, access.data_ptr<int32_t>(), access.stride(0), access.stride(1), (int)access.size(2),
                                        a.decode ? 1 : (int)a.bsa_bq, c.stream), "mark_attention_access");
  // key ranges: a single query row that is not a decode call keeps one (its heads may have masks of their own)
  bp.n_splits = a.decode || c.TQ > 1 ? hipattn_attention_splits(&bp) : 1;
  if (bp.n_splits > 1) {
    const int64_t rows = c.B * c.TQ * c.H;
    at::Tensor part = dv.empty({rows * bp.n_splits * (c.D + 1)}, at::kFloat);
    bp.part_o = part.data_ptr<float>();
    bp.part_lse = bp.part_o + rows * bp.n_splits * c.D;
    check(hipattn_bsa_attention(&bp, c.stream), "bsa_attention");
    check(hipattn::merge_partials(bp.part_o, bp.part_lse, rows, bp.n_splits, (int)c.D, c.dt, out.data_ptr(), c.D,
                                  lse.defined() ? lse.data_ptr<float>() : nullptr, c.TQ * c.H, out.stride(0), c.stream), "merge_partials");
  } else {
    bp.lse_out = lse.defined() ? lse.data_ptr<float>() : nullptr;
    check(hipattn::bsa_attention(&bp, c.stream, a.beside), "bsa_attention");
  }
}

// Reference layout of a stage-input cache: int64 [B, BDST, H, n], identical for every head.
Ref stage_cache(const Call& c, const Mask& m, size_t i, int64_t BDST) {
  Ref none = Ref::borrow(Py_None);
  if (i >= m.left64.size() || !m.left64[i].defined()) {
    PyObject* a[] = {Py_None, Py_None, Py_None};
    return checked(PyObject_Vectorcall(K.StageCache, a, 3, nullptr));
  }
  const int64_t n = m.left64[i].size(1), H = c.H;
  auto view = [&](const at::Tensor& t) { return t.as_strided({c.B, BDST, H, n}, {BDST * n, n, 0, 1}, t.storage_offset()); };
  Ref l = checked(wrap(view(m.left64[i]))), r = checked(wrap(view(m.right64[i])));
  Ref s = checked(wrap(m.consts.as_strided({c.B, BDST, H, n}, {0, 0, 0, 0}, (int64_t)i)));
  PyObject* a[] = {l.get(), r.get(), s.get()};
  Ref entry = checked(PyObject_Vectorcall(K.StageCache, a, 3, nullptr));
  // private: lets a restart skip the narrowing copy
  Ref l32 = checked(wrap(m.left32[i])), r32 = checked(wrap(m.right32[i]));
  if (PyObject_SetAttr(entry.get(), N._left32, l32.get()) < 0 || PyObject_SetAttr(entry.get(), N._right32, r32.get()) < 0) throw PyError{};
  return entry;
}

// the chunk lists a restart begins with (foreign caches, e.g. the reference's: per-head lists are identical under the
// head max-reduce)
void restart_inputs(Call& c, PyObject* entry, int64_t rows, at::Tensor& left, at::Tensor& right, Beside& beside) {
  Ref l32 = attr_opt(entry, N._left32);
  if (!l32.none()) {
    left = tensor_of(l32.get(), "_left32");
    right = attr_tensor(entry, N._right32, "_right32");
    if (left.size(0) == rows && left.is_contiguous() && right.is_contiguous()) return;
  }
  at::Tensor l = attr_tensor(entry, N.indices_left, "indices_left"), r = attr_tensor(entry, N.indices_right, "indices_right");
  if (!l.defined() || !r.defined() || l.dim() != 4 || r.sizes() != l.sizes() || l.size(0) * l.size(1) != rows || l.size(2) < 1)
    VALUE_ERROR("a stage cache must hold indices_left / indices_right [B, blocks, H, n] of this call's shape");
  const int64_t n = l.size(3);
  at::Tensor two = c.dv.empty({2, rows, n}, at::kInt);
  left = two.select(0, 0);
  right = two.select(0, 1);
  if (l.device() != c.q.device() || r.device() != c.q.device()) VALUE_ERROR("stage caches must be on q's device");
  for (at::Tensor* t : {&l, &r}) {
    const int type = copy_type(t->scalar_type());
    if (type >= 0 && type <= hipattn::COPY_U32) continue;
    *t = t->to(at::kLong);     // (a caller's own type; a torch operation, on the current stream)
    beside.after_current();
    if (c.dv.keep) c.dv.keep->push_back(*t);
  }
  Copies cp(c.stream);
  cp.add(l.select(2, 0), left);
  cp.add(r.select(2, 0), right);
  cp.flush();
}

PyObject* forward(PyObject* const* argv) {
  Call c;
  PyObject* q_obj = argv[0];
  c.args = argv[3];
  PyObject* cached = argv[4];
  const bool return_lse = PyObject_IsTrue(argv[5]) == 1;
  c.debug = argv[6];
  c.reduce = argv[7];
  c.timer = argv[8];
  PyObject* v_ready = argv[9];
  c.shared = argv[10];
  at::Tensor context = tensor_of(argv[11], "out"), lse = tensor_of(argv[12], "lse");
  Fork* fork = argv[13] == Py_None ? nullptr : (Fork*)PyCapsule_GetPointer(argv[13], kForkName);
  if (argv[13] != Py_None && !fork) throw PyError{};

  if (!THPVariable_Check(q_obj) || THPVariable_Unpack(q_obj).dim() != 4) VALUE_ERROR("q must be a tensor [B, TQ, H, D]");
  c.q = THPVariable_Unpack(q_obj);
  c.k = tensor_of(argv[1], "k");
  c.v = tensor_of(argv[2], "v");
  c.k_cache = attr_tensor(c.args, N.k_cache, "k_cache");
  c.v_cache = attr_tensor(c.args, N.v_cache, "v_cache");
  const at::Tensor q_mask = attr_tensor(c.args, N.q_mask, "q_mask"), k_mask = attr_tensor(c.args, N.k_mask, "k_mask");
  check_inputs(c, q_mask, k_mask);
  reject_unsupported(c);
  if (attr_true(c.args, N.using_paged_cache) != c.k_cache.defined()) {   // k_cache was changed behind the flags' back
    Ref r = checked(PyObject_CallMethodNoArgs(c.args, N.update_flags));
  }
  if (c.k_cache.defined() && c.k_cache.dim() == 4 && c.k_cache.size(1) <= 0)
    VALUE_ERROR("k_cache must be [n_pages, page_size, kv_heads, head_dim] with page_size > 0");
  c.q_attn = c.q;
  if (q_mask.defined()) {
    c.q = q_mask;
    if (c.q.sizes() != c.q_attn.sizes() || c.q.stride(3) != 1) VALUE_ERROR("q_mask must have q's shape and a contiguous last dim");
  }
  c.k_scan = k_mask.defined() ? k_mask : c.k;
  c.B = c.q.size(0); c.TQ = c.q.size(1); c.H = c.q.size(2); c.D = c.q.size(3);
  if (c.k.defined()) {
    if (c.k.dim() != 4) VALUE_ERROR("k must be [B, T, kv_heads, head_dim] with a contiguous last dim");
    c.T = c.k.size(1);
    c.HKV = c.k.size(2);
    if (c.k.size(0) != c.B || c.k.size(3) != c.D) VALUE_ERROR("k shape %s does not match q shape %s", shape_text(c.k).c_str(), shape_text(c.q).c_str());
  } else {
    Ref length = attr(c.args, N.extend_context_length);     // (whatever int() takes: configuration files write 1e5)
    c.T = as_int(checked(PyNumber_Long(length.get())));
    if (c.k_cache.dim() != 4) VALUE_ERROR("k_cache must be [n_pages, page_size, kv_heads, head_dim] with a contiguous last dim");
    c.HKV = c.k_cache.size(2);
    if (c.k_cache.size(3) != c.D) VALUE_ERROR("k_cache head_dim differs from q");
  }
  if (c.HKV <= 0 || c.H % c.HKV) VALUE_ERROR("%lld query heads are not a multiple of %lld KV heads", (long long)c.H, (long long)c.HKV);
  c.sink = attr_int(c.args, N.sink_token_size);
  c.sw = attr_int(c.args, N.sliding_window_size);

  const c10::cuda::CUDAGuard guard(c.q.device());
  c.dv.dev = c.q.device();
  c.stream = c10::cuda::getCurrentCUDAStream(c.q.device().index()).stream();
  at::Tensor status = status_word(c.q.device().index());
  c.status = (uint32_t*)status.data_ptr();
  Beside beside;
  // (a decode call with something to scan and no rope tables: nothing on its way is a torch operation)
  if (fork) {
    c.dv.keep = &fork->keep;    // (memory that a call on the current stream gives back could be handed to one beside it)
    if (PyObject_IsTrue(argv[14]) == 1 && c.TQ == 1 && !c.using_extend && c.T - c.sink - c.sw > 0 && c.q.device() == fork->dev) {
      beside.begin(fork);
      c.stream = beside.stream;
    }
  }

  hipattn::BeginCall begin{};
  Ref pos_obj = attr(c.args, N.position_ids);
  bool own_pos = false;
  if (!pos_obj.none()) {
    c.pos = tensor_of(pos_obj.get(), "position_ids");
    if (c.pos.dim() != 2 || c.pos.size(0) != c.B || c.pos.size(1) != c.TQ)
      VALUE_ERROR("position_ids shape %s != (%lld, %lld)", shape_text(c.pos).c_str(), (long long)c.B, (long long)c.TQ);
    if (c.pos.scalar_type() != at::kLong) c.pos = c.pos.to(at::kLong);
  } else {
    cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
    cudaStreamIsCapturing(c.stream, &capturing);
    // (the sequence shards hand over a `shared` dict: theirs are the last positions at every replay)
    if (capturing != cudaStreamCaptureStatusNone && c.shared == Py_None) VALUE_ERROR("position_ids must be given under CUDA graph capture");
    own_pos = true;
    at::Tensor row = c.dv.empty({c.TQ}, at::kLong);
    begin.pos = row.data_ptr<int64_t>();
    begin.n_pos = c.TQ;
    begin.pos0 = c.T - c.TQ;
    c.pos = row.as_strided({c.B, c.TQ}, {0, 1});
  }
  {
    const at::Tensor all = c.shared_get("positions");   // of the whole chunk
    const at::Tensor& w = all.defined() ? all : c.pos;
    const bool given = all.defined() || !own_pos;
    c.where = {given ? w.data_ptr<int64_t>() : nullptr, given ? w.stride(0) : 0, given ? w.stride(1) : 0, c.T - c.TQ, (int)c.B, given ? (int)w.size(1) : (int)c.TQ};
  }
  if (context.defined() && (context.sizes() != c.q_attn.sizes() || context.scalar_type() != c.q_attn.scalar_type() || context.stride(3) != 1 ||
                            context.stride(2) != c.D || context.stride(1) != c.H * c.D))
    VALUE_ERROR("out must have q's shape and type, its rows contiguous");
  const int64_t bq = c.stages.back().bq, BDST = cdiv(c.TQ, bq), rows = c.B * BDST;
  const int64_t c0 = c.stages[0].chunk, c_last = c.stages.back().chunk;
  int64_t sw_attn = std::max<int64_t>(0, c.sw - c0) + c0;   // attention_extend.py:1976-1978, 2901

  c.table = attr_tensor(c.args, N.block_table, "block_table");
  c.lens = attr_tensor(c.args, N.cache_seq_lens, "cache_seq_lens");
  const at::Tensor undef;
  // attention reads the page pool whenever one is given (attention_extend_bsa.py:1756)
  const bool paged = c.k_cache.defined();
  const hipattn_tokens_t ktok = tokens(paged ? undef : c.k, c.k_cache, c.table, c.lens, "k");
  const hipattn_tokens_t vtok = tokens(paged ? undef : c.v, c.v_cache, c.table, c.lens, "v");

  // metadata in hand
  Ref cached_caches = cached == Py_None ? Ref::borrow(Py_None) : attr(cached, N.stage_caches);
  const bool fresh = cached == Py_None || attr(cached, N.indices).none();
  Ref stage_caches = Ref::borrow(Py_None);
  if (attr_true(c.args, N.require_stage_caches))
    stage_caches = cached_caches.none() ? checked(PyList_New(0)) : Ref::borrow(cached_caches.get());   // extended in place, like the reference

  // Access statistics (attention_extend.py:1988-2010): one int32 per key position (dense) or page.  No offload cache
  // exists here, so the miss counters stay zero: views of one zero.
  at::Tensor mask_stats, sa_stats, miss;
  if (attr_true(c.args, N.require_cache_statistics)) {
    const int64_t slots = paged ? c.k_cache.size(0) : c.T, per = c.B * c.HKV * slots, sets = fresh ? 2 : 1;
    at::Tensor all = c.dv.empty({sets * per + 4}, at::kInt);
    check(hipattn::zero_memory(all.data_ptr(), (sets * per + 4) * 4, c.stream), "zero_memory");
    auto view = [&](int64_t off) { return all.as_strided({c.B, c.HKV, slots}, {c.HKV * slots, slots, 1}, off); };
    sa_stats = view(0);
    if (fresh) mask_stats = view(per);
    miss = all.as_strided({c.B, c.HKV, slots}, {0, 0, 0}, sets * per);
  }

  at::Tensor indices, ks, ks_count, kse, read_indices, read_ks;
  bool heads_share, copies_first = false;
  int64_t index_bq;
  Ref bsq = attr(c.args, N.block_sparse_block_size_q);
  int64_t bsa_bq = bsq.none() ? bq : as_int(bsq);
  if (bsa_bq == 0) bsa_bq = bq;
  bsa_bq = std::min(bsa_bq, bq);
  if (fresh) {
    int64_t first = 0;
    at::Tensor left, right;
    if (!stage_caches.none() && !cached_caches.none()) {
      const Py_ssize_t have = PyList_Check(stage_caches.get()) ? PyList_GET_SIZE(stage_caches.get()) : PySequence_Size(stage_caches.get());
      if (have < 0) throw PyError{};
      if (have > 1) {
        if (have > (Py_ssize_t)c.stages.size()) VALUE_ERROR("more stage caches than stages");
        first = have - 1;
        Ref entry = checked(PySequence_GetItem(stage_caches.get(), first));
        restart_inputs(c, entry.get(), rows, left, right, beside);
      }
    }
    if (c.using_extend) set_rope_tables(c, first > 0 ? left.size(1) : 0);
    // scan reads dense K when it is given, else the page pool (attention_extend.py:2524)
    const hipattn_tokens_t kscan = c.k_scan.defined() ? tokens(c.k_scan, undef, undef, undef, "k") : ktok;
    Mask m = estimate_mask(c, kscan, first, left, right, !stage_caches.none(), mask_stats, begin);
    if (!stage_caches.none()) {
      const Py_ssize_t have = PySequence_Size(stage_caches.get());
      for (size_t i = (size_t)have; i < c.stages.size(); ++i) {
        Ref e = stage_cache(c, m, i, BDST);
        if (PyList_Check(stage_caches.get())) {
          if (PyList_Append(stage_caches.get(), e.get()) < 0) throw PyError{};
        } else {
          Ref r = checked(PyObject_CallMethod(stage_caches.get(), "append", "O", e.get()));
        }
      }
    }
    indices = m.indices; ks = m.ks; kse = m.kse;
    ks_count = ks.unsqueeze(-1);
    heads_share = m.heads_share;
    index_bq = bq;
    if (attr_true(c.args, N.mask_only)) return PyTuple_Pack(2, Py_None, Py_None);
  } else {
    if (own_pos) check(hipattn::begin_call(begin, c.stream), "begin_call");
    if (c.using_extend) set_rope_tables(c, 0);
    const at::Tensor ci = attr_tensor(cached, N.indices, "indices"), cks = attr_tensor(cached, N.ks, "ks"),
                     ckc = attr_tensor(cached, N.ks_count, "ks_count"), cse = attr_tensor(cached, N.ks_start_end, "ks_start_end");
    if (!cks.defined() || !ckc.defined() || !cse.defined()) VALUE_ERROR("cached metadata with indices needs ks, ks_count and ks_start_end");
    if (ci.dim() != 3 || cks.dim() != 2) VALUE_ERROR("cached indices shape %s does not fit this call", shape_text(ci).c_str());
    // the returned metadata holds copies; int64 is what the kernels read
    auto like = [&](const at::Tensor& t, at::ScalarType type) { return c.dv.empty(t.sizes(), type); };
    Ref shared = attr_opt(cached, N._heads_share);
    heads_share = !shared.none() && truth(shared);
    // cached rows may already be broken down to the attention block size: the fresh path returns BDST * (bq / bsa_bq)
    // rows (repeat-interleave, attention_extend.py:3036-3051), of which a ragged last block uses only the first
    // cdiv(TQ, bsa_bq)
    const int64_t have = ci.size(1);
    index_bq = have == BDST ? bq : bsa_bq;
    if ((have != BDST && have != cdiv(c.TQ, bsa_bq) && have != BDST * (bq / bsa_bq)) || ci.size(0) != c.B * c.H)
      VALUE_ERROR("cached indices shape %s does not fit this call", shape_text(ci).c_str());
    if (cks.size(0) != ci.size(0) || cks.size(1) != have) VALUE_ERROR("cached ks shape %s does not fit this call", shape_text(cks).c_str());
    bool fast = true;
    for (const at::Tensor* t : {&ci, &cks, &ckc, &cse})
      fast = fast && t->device() == c.q.device() && copy_type(t->scalar_type()) >= 0 && copy_type(t->scalar_type()) <= hipattn::COPY_U32;
    if (fast) {
      indices = like(ci, at::kLong); ks = like(cks, at::kLong); ks_count = like(ckc, ckc.scalar_type()); kse = like(cse, cse.scalar_type());
      Copies cp(c.stream);
      cp.add(ci, indices); cp.add(cks, ks); cp.add(ckc, ks_count); cp.add(cse, kse);
      // A decode call's attention may read the mask that it was given and run beside the copies, as long as nothing else comes
      // between the two on the stream.
      copies_first = cp.list.count > 0 && c.TQ == 1 && ci.scalar_type() == at::kLong && cks.scalar_type() == at::kLong && ci.stride(2) == 1 &&
                     v_ready == Py_None && c.debug == Py_None && !sa_stats.defined();
      if (copies_first) { read_indices = ci; read_ks = cks; }
      cp.flush(copies_first);
    } else {
      indices = ci.clone().to(at::kLong).contiguous(); ks = cks.clone().to(at::kLong).contiguous(); ks_count = ckc.clone(); kse = cse.clone();
      if (indices.device() != c.q.device() || ks.device() != c.q.device()) VALUE_ERROR("cached metadata is on another device than q");
      beside.after_current();
      if (c.dv.keep) c.dv.keep->insert(c.dv.keep->end(), {indices, ks});
    }
  }

  bsa_bq = std::min(bsa_bq, next_pow2(c.TQ));
  if (bsa_bq <= 0 || bq % bsa_bq) VALUE_ERROR("block_sparse_block_size_q must divide stage_block_size_q");
  if (sw_attn == 777) {
    // window sentinel of the serving adapter (attention_extend.py:3070-3076): these queries see everything the model
    // context has room for beside the sink, the selected keys and their own block
    sw_attn = attr_int(c.args, N.model_context_length) - c.sink - c.second_k - bsa_bq;
    if (sw_attn < 0) VALUE_ERROR("the window sentinel 777 needs model_context_length > sink + second_stage_k + query block");
  }
  AttentionArgs a;
  a.window = sw_attn;
  a.block_k = c_last;
  a.bsa_bq = bsa_bq;
  a.index_bq = index_bq;
  a.heads_share = heads_share;
  a.own_mask = fresh;
  a.decode = c.TQ == 1 && !attr_true(c.args, N.disable_flashdecode) && strcmp(env("HIP_DISABLE_FLASHDECODE", "0"), "1");
  a.want_lse = return_lse;
  Ref cap = attr(c.args, N.logit_softcap);
  a.softcap = cap.none() ? 0.f : (float)PyFloat_AsDouble(cap.get());
  if (PyErr_Occurred()) throw PyError{};
  a.beside = copies_first && a.decode;
  c.mark("start");
  if (v_ready != Py_None) {
    Ref dev = checked(PyLong_FromLong(c.q.device().index()));
    Ref s = checked(PyObject_CallMethodOneArg(K.torch_cuda, N.current_stream, dev.get()));
    Ref r = checked(PyObject_CallMethodOneArg(s.get(), N.wait_event, v_ready));
  }
  if (lse.defined() && (lse.scalar_type() != at::kFloat || lse.numel() != c.B * c.TQ * c.H || !lse.is_contiguous()))
    VALUE_ERROR("lse must be a contiguous float32 tensor [B, TQ, H]");
  attention(c, ktok, vtok, a.beside ? read_indices : indices, a.beside ? read_ks : ks, a, sa_stats, context, lse);
  c.mark("attention");

  if (fresh && cdiv(c.TQ, bsa_bq) != BDST) {
    // break the mask down to the attention block size (attention_extend.py:3036-3051)
    const int64_t rep = bq / bsa_bq;
    indices = indices.repeat_interleave(rep, 1);
    ks = ks.repeat_interleave(rep, 1);
    ks_count = ks_count.repeat_interleave(rep, 1);
    kse = kse.repeat_interleave(rep, 1);
  }
  auto stats = [&](const at::Tensor& t) {
    Ref x = checked(wrap(t)), y = checked(wrap(t.defined() ? miss : t));
    PyObject* v[] = {x.get(), y.get()};
    return checked(PyObject_Vectorcall(K.Statistics, v, 2, nullptr));
  };
  Ref mi = checked(wrap(indices)), mk = checked(wrap(ks)), mc = checked(wrap(ks_count)), me = checked(wrap(kse));
  Ref ms = fresh ? stats(mask_stats) : Ref::borrow(Py_None), ss = stats(sa_stats);
  PyObject* v[] = {mi.get(), mk.get(), mc.get(), me.get(), ms.get(), ss.get(), stage_caches.get()};
  Ref md = checked(PyObject_Vectorcall(K.Metadata, v, 7, nullptr));
  if (PyObject_SetAttr(md.get(), N._heads_share, heads_share ? Py_True : Py_False) < 0) throw PyError{};
  Ref ctx = checked(wrap(context));
  if (return_lse) {
    Ref l = checked(wrap(lse));
    return PyTuple_Pack(3, ctx.get(), md.get(), l.get());
  }
  return PyTuple_Pack(2, ctx.get(), md.get());
}

// ---------------------------------------------------------------------------------------------------------------------
// metadata pool: buffers [rows, ...] or [batch, 1, heads, ...] to fresh tensors and back, one launch for all of them
// ---------------------------------------------------------------------------------------------------------------------
// pool_read([(buffer, rows, int64?)...]): contiguous leading rows of every buffer as int64 (integers) or float32 tensors
PyObject* pool_read(PyObject* list) {
  const Py_ssize_t n = PyList_GET_SIZE(list);
  Ref out = checked(PyList_New(n));
  std::unique_ptr<c10::cuda::CUDAGuard> guard;
  std::unique_ptr<Copies> cp;
  for (Py_ssize_t i = 0; i < n; ++i) {
    PyObject* e = PyList_GET_ITEM(list, i);
    const at::Tensor& buf = THPVariable_Unpack(PyTuple_GET_ITEM(e, 0));
    const int64_t rows = PyLong_AsLongLong(PyTuple_GET_ITEM(e, 1));
    if (!cp) {
      guard.reset(new c10::cuda::CUDAGuard(buf.device()));
      cp.reset(new Copies(c10::cuda::getCurrentCUDAStream(buf.device().index()).stream()));
    }
    std::vector<int64_t> sizes = buf.sizes().vec();
    sizes[0] = rows;
    const int t = copy_type(buf.scalar_type());
    at::Tensor dst = at::detail::empty_cuda(sizes, t >= hipattn::COPY_F32 ? at::kFloat : at::kLong, buf.device(), c10::nullopt);
    hipattn::CopySeg s{};
    s.src = buf.data_ptr();
    s.dst = dst.data_ptr();
    s.src_type = t;
    s.dst_type = copy_type(dst.scalar_type());
    s.n0 = s.n1 = 1;
    s.n2 = dst.numel();
    s.plain = 1;
    cp->add(s);
    PyList_SET_ITEM(out.get(), i, wrap(dst));
  }
  if (cp) cp->flush();
  return out.release();
}

// pool_write([(buffer, value or None, rows)...]): value into the leading rows of its buffer, zeros for None; returns the
// places in the list of the values it does not take (another layout, type or device, too many rows)
PyObject* pool_write(PyObject* list) {
  const Py_ssize_t n = PyList_GET_SIZE(list);
  Ref left = checked(PyList_New(0));
  std::unique_ptr<c10::cuda::CUDAGuard> guard;
  std::unique_ptr<Copies> cp;
  for (Py_ssize_t i = 0; i < n; ++i) {
    PyObject* e = PyList_GET_ITEM(list, i);
    const at::Tensor& buf = THPVariable_Unpack(PyTuple_GET_ITEM(e, 0));
    PyObject* val = PyTuple_GET_ITEM(e, 1);
    if (!cp) {
      guard.reset(new c10::cuda::CUDAGuard(buf.device()));
      cp.reset(new Copies(c10::cuda::getCurrentCUDAStream(buf.device().index()).stream()));
    }
    if (val == Py_None) {
      hipattn::CopySeg s{};
      s.src = nullptr;
      s.dst = buf.data_ptr();
      s.src_type = hipattn::COPY_ZERO;
      s.dst_type = copy_type(buf.scalar_type());
      s.n0 = s.n1 = 1;
      s.n2 = PyLong_AsLongLong(PyTuple_GET_ITEM(e, 2)) * buf.stride(0);
      s.plain = 1;
      cp->add(s);
    } else {
      const at::Tensor v = tensor_of(val, "value");
      const int ts = copy_type(v.scalar_type()), td = copy_type(buf.scalar_type());
      if (ts < 0 || (ts >= hipattn::COPY_F32) != (td >= hipattn::COPY_F32) || v.device() != buf.device() || v.dim() != buf.dim() || v.dim() < 1 ||
          v.size(0) > buf.size(0) || v.sizes().slice(1) != buf.sizes().slice(1)) {
        Ref at = checked(PyLong_FromSsize_t(i));
        if (PyList_Append(left.get(), at.get()) < 0) throw PyError{};
        continue;
      }
      cp->add(v, buf);
    }
  }
  if (cp) cp->flush();
  return left.release();
}

// ---------------------------------------------------------------------------------------------------------------------
// module
// ---------------------------------------------------------------------------------------------------------------------
template <typename F>
PyObject* guarded(F f) {
  try {
    return f();
  } catch (const PyError&) {
    return nullptr;
  } catch (const c10::OutOfMemoryError& e) {
    PyObject* type = PyObject_GetAttrString(K.torch_cuda, "OutOfMemoryError");
    PyErr_SetString(type ? type : PyExc_RuntimeError, e.what_without_backtrace());
    Py_XDECREF(type);
    return nullptr;
  } catch (const c10::Error& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what_without_backtrace());
    return nullptr;
  } catch (const std::exception& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
    return nullptr;
  }
}

PyObject* py_forward(PyObject*, PyObject* const* argv, Py_ssize_t n) {
  if (n != 15) {
    PyErr_SetString(PyExc_TypeError, "forward takes fifteen arguments");
    return nullptr;
  }
  return guarded([&] { return forward(argv); });
}
// gather_table(table [*, width], rows [n], lens [n]) -> [n, width]: the rows' first lens[i] entries (the rest is not written)
PyObject* gather_table(PyObject* const* argv) {
  const at::Tensor table = tensor_of(argv[0], "req_to_tokens"), rows = tensor_of(argv[1], "req_pool_indices"), lens = tensor_of(argv[2], "seq_lens");
  auto ints = [](const at::Tensor& t) { return t.defined() && (t.scalar_type() == at::kInt || t.scalar_type() == at::kLong); };
  if (!ints(table) || !ints(rows) || !ints(lens) || !table.is_cuda() || rows.device() != table.device() || lens.device() != table.device() ||
      table.dim() != 2 || rows.dim() != 1 || lens.dim() != 1 || lens.size(0) != rows.size(0) || table.stride(1) != 1 || !rows.is_contiguous() ||
      !lens.is_contiguous() || rows.size(0) > 65535 || table.size(0) < 1)
    Py_RETURN_NONE;
  const c10::cuda::CUDAGuard guard(table.device());
  at::Tensor out = at::detail::empty_cuda({rows.size(0), table.size(1)}, table.scalar_type(), table.device(), c10::nullopt);
  const at::Tensor status = status_word(table.device().index());
  check(hipattn::gather_table(table.data_ptr(), table.size(0), table.stride(0), (uint32_t*)status.data_ptr(), (int)table.element_size(),
                              rows.data_ptr(), rows.scalar_type() == at::kLong, lens.data_ptr(), lens.scalar_type() == at::kLong,
                              (int)rows.size(0), (int)table.size(1), out.data_ptr(),
                              c10::cuda::getCurrentCUDAStream(table.device().index()).stream()), "gather_table");
  return wrap(out);
}
// fork(tensor): the point of the current stream of its device that calls beside it start from
PyObject* py_fork(PyObject*, PyObject* x) {
  return guarded([&]() -> PyObject* {
    const at::Tensor t = tensor_of(x, "q");
    const c10::cuda::CUDAGuard guard(t.device());
    status_word(t.device().index());
    std::unique_ptr<Fork> f(new Fork(t.device()));
    cuda_ok(cudaEventCreateWithFlags(&f->start, cudaEventDisableTiming), "cudaEventCreate");
    cuda_ok(cudaEventRecord(f->start, f->main.stream()), "cudaEventRecord");
    PyObject* o = PyCapsule_New(f.get(), kForkName, drop_fork);
    if (o) f.release();
    return o;
  });
}
PyObject* py_join(PyObject*, PyObject* o) {
  return guarded([&]() -> PyObject* {
    Fork* f = (Fork*)PyCapsule_GetPointer(o, kForkName);
    if (!f) return nullptr;
    const c10::cuda::CUDAGuard guard(f->dev);
    f->join();
    Py_RETURN_NONE;
  });
}
// stack_rows([[tensors...], ...]): every list of [rows, ...] tensors one below the other, in one launch
PyObject* stack_rows(PyObject* lists) {
  const Py_ssize_t n = PyList_GET_SIZE(lists);
  Ref out = checked(PyList_New(n));
  std::unique_ptr<c10::cuda::CUDAGuard> guard;
  std::unique_ptr<Copies> cp;
  for (Py_ssize_t i = 0; i < n; ++i) {
    PyObject* l = PyList_GET_ITEM(lists, i);
    const Py_ssize_t m = PyList_GET_SIZE(l);
    const at::Tensor first = tensor_of(PyList_GET_ITEM(l, 0), "rows");
    if (!cp) {
      guard.reset(new c10::cuda::CUDAGuard(first.device()));
      cp.reset(new Copies(c10::cuda::getCurrentCUDAStream(first.device().index()).stream()));
    }
    std::vector<int64_t> sizes = first.sizes().vec();
    int64_t rows = 0;
    at::ScalarType type = first.scalar_type();      // int32 and int64 side by side: int64
    for (Py_ssize_t j = 0; j < m; ++j) {
      const at::Tensor t = tensor_of(PyList_GET_ITEM(l, j), "rows");
      if ((t.scalar_type() != at::kInt && t.scalar_type() != at::kLong) || t.device() != first.device() || t.dim() != first.dim() || t.dim() < 1 ||
          t.sizes().slice(1) != first.sizes().slice(1))
        VALUE_ERROR("shards of one page pool must have int32 or int64 block tables and lengths of the same width on one device");
      type = at::promoteTypes(type, t.scalar_type());
      rows += t.size(0);
    }
    sizes[0] = rows;
    at::Tensor dst = at::detail::empty_cuda(sizes, type, first.device(), c10::nullopt);
    int64_t at_row = 0;
    for (Py_ssize_t j = 0; j < m; ++j) {
      const at::Tensor t = tensor_of(PyList_GET_ITEM(l, j), "rows");
      cp->add(t, dst.narrow(0, at_row, t.size(0)));
      at_row += t.size(0);
    }
    PyList_SET_ITEM(out.get(), i, wrap(dst));
  }
  if (cp) cp->flush();
  return out.release();
}
PyObject* py_stack_rows(PyObject*, PyObject* lists) {
  return guarded([&] { return stack_rows(lists); });
}
// merge_shards(outs [S, B, 1, H, D], lses [S, B, 1, H]) -> [B, 1, H, D]
PyObject* py_merge_shards(PyObject*, PyObject* const* argv, Py_ssize_t n) {
  if (n != 2) {
    PyErr_SetString(PyExc_TypeError, "merge_shards takes two arguments");
    return nullptr;
  }
  return guarded([&]() -> PyObject* {
    const at::Tensor o = tensor_of(argv[0], "outs"), l = tensor_of(argv[1], "lses");
    if (dtype_of(o.scalar_type()) < 0 || o.dim() != 5 || l.dim() != 4 || !o.is_contiguous() || !l.is_contiguous() || l.numel() * o.size(4) != o.numel())
      VALUE_ERROR("merge_shards: outs [S, B, 1, H, D] and lses [S, B, 1, H] must be contiguous");
    const c10::cuda::CUDAGuard guard(o.device());
    at::Tensor out = at::detail::empty_cuda(o.sizes().slice(1), o.scalar_type(), o.device(), c10::nullopt);
    check(hipattn::merge_shards(o.data_ptr(), l.data_ptr<float>(), l.numel() / l.size(0), (int)l.size(0), (int)o.size(4), dtype_of(o.scalar_type()),
                                out.data_ptr(), c10::cuda::getCurrentCUDAStream(o.device().index()).stream()), "merge_shards");
    return wrap(out);
  });
}
PyObject* py_gather_table(PyObject*, PyObject* const* argv, Py_ssize_t n) {
  if (n != 3) {
    PyErr_SetString(PyExc_TypeError, "gather_table takes three arguments");
    return nullptr;
  }
  return guarded([&] { return gather_table(argv); });
}
PyObject* py_status_word(PyObject*, PyObject* index) {
  return guarded([&] { return wrap(status_word((int)PyLong_AsLong(index))); });
}
PyObject* py_pool_read(PyObject*, PyObject* list) {
  return guarded([&] { return pool_read(list); });
}
PyObject* py_pool_write(PyObject*, PyObject* list) {
  return guarded([&] { return pool_write(list); });
}
// bind(ScanStage, HiPAttentionOutputMetadata, HiPAttentionStageInputCache, HiPAttentionCacheAccessStatistics, HipAttnError, torch.cuda)
PyObject* py_bind(PyObject*, PyObject* const* argv, Py_ssize_t n) {
  if (n != 6) {
    PyErr_SetString(PyExc_TypeError, "bind takes six arguments");
    return nullptr;
  }
  for (Py_ssize_t i = 0; i < n; ++i) Py_INCREF(argv[i]);
  K = Classes{argv[0], argv[1], argv[2], argv[3], argv[4], argv[5]};
  Py_RETURN_NONE;
}

PyMethodDef methods[] = {
    {"forward", (PyCFunction)(void*)py_forward, METH_FASTCALL, "q, k, v, args, cached_metadata, return_lse, debug, score_reduce, timer, v_ready, shared, out, lse, fork, beside"},
    {"gather_table", (PyCFunction)(void*)py_gather_table, METH_FASTCALL, "table, rows, lens -> rows of the table, or None when it does not take them"},
    {"fork", py_fork, METH_O, "tensor -> fork of the current stream"},
    {"join", py_join, METH_O, "fork"},
    {"stack_rows", py_stack_rows, METH_O, "[[tensors], ...] -> [tensor, ...]"},
    {"merge_shards", (PyCFunction)(void*)py_merge_shards, METH_FASTCALL, "outs, lses -> context"},
    {"status_word", py_status_word, METH_O, "device index -> int32 tensor [1]"},
    {"pool_read", py_pool_read, METH_O, "[(buffer, rows), ...] -> list of tensors"},
    {"pool_write", py_pool_write, METH_O, "[(buffer, value or None, rows), ...]"},
    {"bind", (PyCFunction)(void*)py_bind, METH_FASTCALL, "classes of the package"},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", "Host path of hip_attention_12.", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host() {
#define X(n) \
  if (!(N.n = PyUnicode_InternFromString(#n))) return nullptr;
  NAMES(X)
#undef X
  return PyModule_Create(&module);
}
