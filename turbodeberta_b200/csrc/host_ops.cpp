// Host side of the operators: argument checks, output allocation, the launch and the read of the status words, in one
// native call.  A short attention call takes about 10 us on the GPU; the same steps issued from Python (eight tensor calls,
// forty ctypes arguments, a device-to-host copy of the status words) took 57 us around it.
//
// Status words.  Every call gets a slot of a per-device pool: 16 bytes of pinned host memory that the kernels report into
// (only when something is wrong, so they stay zero and reading them after a stream synchronisation costs nothing), and
// 16 bytes of device memory with the tensor-core kernel's work counter, which the kernel leaves at zero.  No launch and no
// copy per call.  A slot belongs to one call from its launch until its words have been read after the stream was
// synchronised, so calls of several threads and streams never share one.  When all slots of a device are taken (calls with
// deferred checks that nobody collects) or a stream capture is in progress (the recorded launch outlives the call), the
// call gets zeroed words of its own from torch's allocator instead.
#include <torch/extension.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/CUDAGraphsUtils.cuh>
#include <cublasLt.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <map>
#include <mutex>
#include <unordered_map>
#include <utility>
#include <vector>

#include "tdb_internal.h"

namespace py = pybind11;
using at::Tensor;
using OptTensor = std::optional<Tensor>;

namespace {

constexpr int MAX_DEV = 64, SLOTS = 256, SLOT_WORDS = 4;

// Whether the stream is a caller's (cudaStreamCreate, handed to torch) and not one of torch's or the legacy one.
bool is_external(c10::cuda::CUDAStream s) {
  return s.stream() && c10::cuda::getStreamFromExternal(s.stream(), s.device_index()).id() == s.id();
}

// The end of what a stream holds now.  torch never destroys its own streams, so their handle stays good to wait for; one that a
// caller made and handed to torch may be gone by then, and is marked with an event instead.
class Mark {
 public:
  explicit Mark(c10::cuda::CUDAStream s) : stream_(s.stream()) {
    if (!is_external(s)) return;
    own_ = false;
    if (cudaEventCreateWithFlags(&event_, cudaEventDisableTiming) != cudaSuccess) event_ = nullptr;
    renew();
  }
  Mark(Mark&& o) noexcept : stream_(o.stream_), own_(o.own_), event_(std::exchange(o.event_, nullptr)) {}
  Mark& operator=(Mark&& o) noexcept {
    std::swap(stream_, o.stream_); std::swap(own_, o.own_); std::swap(event_, o.event_);
    return *this;
  }
  ~Mark() {
    if (event_) cudaEventDestroy(event_);
  }
  // Called while the stream is the current one: move the mark behind what it holds by now.
  void renew() {
    if (own_ || (event_ && cudaEventRecord(event_, stream_) == cudaSuccess)) return;
    (void)cudaGetLastError();
    cudaStreamSynchronize(stream_);                  // no event to be had: nothing left to wait for later
    if (event_) cudaEventDestroy(std::exchange(event_, nullptr));
  }
  bool on(cudaStream_t s) const { return own_ && stream_ == s; }
  cudaError_t wait() const { return own_ ? cudaStreamSynchronize(stream_) : event_ ? cudaEventSynchronize(event_) : cudaSuccess; }
  cudaStream_t stream() const { return stream_; }    // to compare with, not to use

 private:
  cudaStream_t stream_;
  bool own_ = true;                                  // torch's own, or the legacy stream
  cudaEvent_t event_ = nullptr;
};

struct StatusPool {
  std::mutex mu;
  int32_t* host = nullptr;        // SLOTS x 4 words, pinned and mapped
  int32_t* ctl = nullptr;         // SLOTS x 4 words on the device: work counter, gave-up flag
  std::vector<int> free;
  struct Pending { int slot; Mark mark; bool keep; };             // keep: the slot stays its owner's
  std::vector<Pending> pending;   // launches whose check was deferred
};
StatusPool g_pools[MAX_DEV];

void cuda_ok(cudaError_t e, const char* what) {
  if (e != cudaSuccess) { (void)cudaGetLastError(); TORCH_CHECK(false, what, ": ", cudaGetErrorString(e)); }
}

// A free slot of the current device, or -1.
int acquire(int dev) {
  if (dev < 0 || dev >= MAX_DEV) return -1;
  StatusPool& p = g_pools[dev];
  std::lock_guard<std::mutex> lock(p.mu);
  if (!p.host) {
    int32_t *h = nullptr, *d = nullptr;
    cuda_ok(cudaHostAlloc(reinterpret_cast<void**>(&h), SLOTS * SLOT_WORDS * 4, cudaHostAllocMapped | cudaHostAllocPortable), "cudaHostAlloc(status words)");
    memset(h, 0, SLOTS * SLOT_WORDS * 4);
    if (cudaMalloc(reinterpret_cast<void**>(&d), SLOTS * SLOT_WORDS * 4) != cudaSuccess || cudaMemset(d, 0, SLOTS * SLOT_WORDS * 4) != cudaSuccess ||
        cudaDeviceSynchronize() != cudaSuccess) {
      const cudaError_t e = cudaGetLastError();
      cudaFreeHost(h);
      if (d) cudaFree(d);
      cuda_ok(e == cudaSuccess ? cudaErrorMemoryAllocation : e, "status pool");
    }
    p.host = h; p.ctl = d;
    p.free.reserve(SLOTS);
    for (int i = SLOTS - 1; i >= 0; --i) p.free.push_back(i);
  }
  if (p.free.empty()) return -1;
  const int s = p.free.back();
  p.free.pop_back();
  return s;
}

// What a launch has reported: 0 = code of a wait that gave up, 1 = malformed offsets, 3 = a token id outside the vocabulary.
struct Words {
  int w[SLOT_WORDS] = {};
  bool any() const { return w[0] || w[1] || w[2] || w[3]; }
  void merge(const Words& o) {
    for (int i = 0; i < SLOT_WORDS; ++i) w[i] = std::max(w[i], o.w[i]);
  }
  py::object to_python() const { return any() ? py::object(py::make_tuple(w[0], w[1], w[2], w[3])) : py::none(); }
};

// Read the words of a slot whose launch has finished, and hand the slot back clean.
Words collect(int dev, int slot, bool keep = false) {
  StatusPool& p = g_pools[dev];
  volatile int32_t* w = p.host + slot * SLOT_WORDS;
  Words r;
  for (int i = 0; i < SLOT_WORDS; ++i) r.w[i] = w[i];
  if (r.any()) {
    for (int i = 0; i < SLOT_WORDS; ++i) w[i] = 0;
    // a launch that gave up may have left its work counter and flag set
    cudaMemset(p.ctl + slot * SLOT_WORDS, 0, SLOT_WORDS * 4);
    cudaDeviceSynchronize();
  }
  if (keep) return r;
  std::lock_guard<std::mutex> lock(p.mu);
  p.free.push_back(slot);
  return r;
}

// A Python warning; as an error, where the caller's filters ask for that.
void warn(const std::string& text) {
  py::gil_scoped_acquire gil;
  if (PyErr_WarnEx(PyExc_RuntimeWarning, text.c_str(), 1) < 0) throw py::error_already_set();
}

// Scratch for long sequences (see AttnParams::part_o), 264 bytes per query row and head, if the device has room for it.  The call
// works without it too, on the kernel that takes near and far key tiles, and says so.
Tensor partial_scratch(tdb::AttnParams& p, int dtype, int kernel, const Tensor& like) {
  const int64_t n = tdb_partial_floats(&p, dtype, kernel);
  if (n == 0) return {};
  Tensor t;
  try {
    t = at::empty({n}, like.options().dtype(at::kFloat));
  } catch (const c10::OutOfMemoryError&) {
    warn("turbodeberta_b200: no room for " + std::to_string(n * 4 >> 20) + " MB of scratch for long sequences; the call takes a kernel that "
         "needs none and is up to 1.5 times slower (and torch's allocator has given its cached blocks back)");
    return {};
  }
  p.part_o = t.data_ptr<float>();
  p.part_ml = p.part_o + n / 66 * 64;
  return t;
}

void release_unused(int dev, int slot) {
  if (slot < 0) return;
  std::lock_guard<std::mutex> lock(g_pools[dev].mu);
  g_pools[dev].free.push_back(slot);
}

// Where one call reports: a pool slot, or words of its own.  The slot goes back by itself if the call ends (by an exception of
// the allocator, say) before anything was launched with it.
struct Status {
  int dev, slot = -1;
  Tensor own;
  Status(int device, tdb::AttnParams& p) : dev(device) {
    if (at::cuda::currentStreamCaptureStatusMayInitCtx() == at::cuda::CaptureStatus::None) slot = acquire(dev);
    if (slot >= 0) {
      p.status = g_pools[dev].host + slot * SLOT_WORDS;
      p.counter = g_pools[dev].ctl + slot * SLOT_WORDS;
      p.gave_up = p.counter + 1;
    } else {
      own = at::zeros({8}, at::TensorOptions().dtype(at::kInt).device(at::kCUDA, (c10::DeviceIndex)dev));
      p.status = own.data_ptr<int32_t>();
      p.counter = p.status + 4;
      p.gave_up = p.status + 5;
    }
  }
  Status(const Status&) = delete;
  Status& operator=(const Status&) = delete;
  ~Status() { release_unused(dev, slot); }
  // The launch failed.  One of its kernels may be running all the same, and then reports into the slot until it ends.
  void failed(cudaStream_t stream) {
    if (slot < 0) return;
    cudaStreamSynchronize(stream);
    (void)cudaGetLastError();
    collect(dev, std::exchange(slot, -1));
  }
  // Leave the check to drain_pending(); words of the call's own go to `words`.  Needs no interpreter lock.
  void defer(c10::cuda::CUDAStream stream, std::vector<Tensor>& words) {
    if (slot < 0) { words.push_back(own.narrow(0, 0, SLOT_WORDS)); return; }
    Mark mark(stream);
    std::lock_guard<std::mutex> lock(g_pools[dev].mu);
    g_pools[dev].pending.push_back({std::exchange(slot, -1), std::move(mark), false});
  }
  // Leave the check to the holder of the report, or of the tensor of words.
  py::object report(c10::cuda::CUDAStream stream);
  // What the caller in Python gets to see: None (fine, or deferred into the pool), the words, or the tensor of words.
  py::object finish(bool check, c10::cuda::CUDAStream stream) {
    if (slot < 0) return py::cast(own.narrow(0, 0, SLOT_WORDS));
    if (!check) {
      Mark mark(stream);
      std::lock_guard<std::mutex> lock(g_pools[dev].mu);
      g_pools[dev].pending.push_back({std::exchange(slot, -1), std::move(mark), false});
      return py::none();
    }
    cudaError_t e;
    {
      py::gil_scoped_release nogil;
      e = cudaStreamSynchronize(stream.stream());
    }
    const Words r = collect(dev, std::exchange(slot, -1));
    cuda_ok(e, "cudaStreamSynchronize");
    return r.to_python();
  }
};

// The words of one launch that its caller reads, and nobody else: what a check finds in the pool's list may belong to another thread.
class Report {
 public:
  Report(int dev, int slot, c10::cuda::CUDAStream stream) : dev_(dev), slot_(slot), mark_(stream) {}
  Report(const Report&) = delete;
  Report& operator=(const Report&) = delete;
  ~Report() {                                        // its caller has met an error before the check
    if (slot_ < 0) return;
    py::gil_scoped_release nogil;
    mark_.wait();
    (void)cudaGetLastError();
    int before = 0;
    cudaGetDevice(&before);
    cudaSetDevice(dev_);
    collect(dev_, slot_);
    cudaSetDevice(before);
  }
  int device() const { return slot_ < 0 ? -1 : dev_; }
  const Mark& mark() const { return mark_; }
  Words take() { return slot_ < 0 ? Words() : collect(dev_, std::exchange(slot_, -1)); }       // the mark has been waited for

 private:
  int dev_, slot_;
  Mark mark_;
};

py::object Status::report(c10::cuda::CUDAStream stream) {
  if (slot < 0) return py::cast(own.narrow(0, 0, SLOT_WORDS));
  auto r = std::make_unique<Report>(dev, slot, stream);
  slot = -1;
  return py::cast(std::move(r));
}

// Words of every launch with a deferred check, all devices, and of the caller's own report: None, or the largest of each word.
py::object drain_pending(Report* own) {
  Words all;
  for (int dev = 0; dev < MAX_DEV; ++dev) {
    StatusPool& p = g_pools[dev];
    std::vector<StatusPool::Pending> take;
    {
      std::lock_guard<std::mutex> lock(p.mu);
      take.swap(p.pending);
    }
    const bool with_own = own && own->device() == dev;
    if (take.empty() && !with_own) continue;
    c10::cuda::CUDAGuard guard((c10::DeviceIndex)dev);
    cudaError_t e = cudaSuccess;
    {
      py::gil_scoped_release nogil;
      const Mark* last = nullptr;
      for (const auto& t : take) {
        if (last && t.mark.on(last->stream()) && last->on(t.mark.stream())) continue;
        last = &t.mark;
        if ((e = t.mark.wait()) != cudaSuccess) break;
      }
      if (with_own && e == cudaSuccess && !(last && own->mark().on(last->stream()) && last->on(own->mark().stream()))) e = own->mark().wait();
    }
    for (const auto& t : take) all.merge(collect(dev, t.slot, t.keep));
    if (with_own) all.merge(own->take());
    cuda_ok(e, "synchronisation");
  }
  return all.to_python();
}

// ------------------------------------------------------------------------------------------------- argument checks
int device_of(std::initializer_list<const Tensor*> ts) {
  int dev = -1;
  for (const Tensor* t : ts) {
    if (!t || !t->defined()) continue;
    if (!t->is_cuda()) throw std::runtime_error("turbodeberta_b200 runs on CUDA tensors only; there is no CPU path");
    if (dev >= 0 && t->get_device() != dev) throw py::value_error("all tensors must live on the same device");
    dev = t->get_device();
  }
  return dev;
}

int dtype_code(const Tensor& t) {
  if (t.scalar_type() == at::kFloat) return TDB_DTYPE_F32;
  if (t.scalar_type() == at::kBFloat16) return TDB_DTYPE_BF16;
  throw py::value_error(std::string("unsupported dtype ") + c10::toString(t.scalar_type()) + ": the kernels take float32 or bfloat16");
}

void check_qkv(const Tensor& q, const Tensor& k, const Tensor& v, int64_t dim, const char* shape) {
  if (q.dim() != dim || k.sizes() != q.sizes() || v.sizes() != q.sizes())
    throw py::value_error(std::string("q, k, v must share the shape ") + shape);
  if (k.scalar_type() != q.scalar_type() || v.scalar_type() != q.scalar_type()) throw py::value_error("q, k, v must share a dtype");
}

void check_rows(const Tensor& q, const Tensor& k, const Tensor& v) {
  if (q.stride(-1) != 1 || k.stride(-1) != 1 || v.stride(-1) != 1) throw py::value_error("the head dimension must be contiguous");
}

void* ptr(const OptTensor& t) { return t.has_value() && t->defined() ? t->data_ptr() : nullptr; }

// One layer's position tables (the fields of relpos.RelPosTables).
struct Tables {
  OptTensor kr, qr, idx, kr_exp, qr_exp;
  int two_span, idx_delta_max, exp_delta_max, exp_rows;
  bool one_call = false;                             // made for one call, whose kernel decides whether they have to be expanded
  void fill(tdb::AttnParams& p, const Tensor& q) const {
    for (const OptTensor* t : {&kr, &qr})
      if (t->has_value() && (*t)->scalar_type() != q.scalar_type()) throw py::value_error("relative tables must have the dtype of q");
    p.kr = ptr(kr); p.qr = ptr(qr); p.two_span = two_span;
    p.idx = static_cast<const int16_t*>(ptr(idx)); p.idx_delta_max = idx_delta_max;
    p.kr_exp = ptr(kr_exp); p.qr_exp = ptr(qr_exp);
    p.exp_delta_max = exp_delta_max; p.exp_rows = exp_rows;
    p.flags = (p.kr ? TDB_FLAG_C2P : 0) | (p.qr ? TDB_FLAG_P2C : 0);
  }
};

struct Strides { int64_t b, t, h; };
Strides fixed_strides(const Tensor& t) { return {t.stride(0), t.stride(2), t.stride(1)}; }

void set_qkvo_fixed(tdb::AttnParams& p, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& o) {
  Strides s;
  p.q = q.data_ptr(); s = fixed_strides(q); p.q_sb = s.b; p.q_st = s.t; p.q_sh = s.h;
  p.k = k.data_ptr(); s = fixed_strides(k); p.k_sb = s.b; p.k_st = s.t; p.k_sh = s.h;
  p.v = v.data_ptr(); s = fixed_strides(v); p.v_sb = s.b; p.v_st = s.t; p.v_sh = s.h;
  p.o = o.data_ptr(); s = fixed_strides(o); p.o_sb = s.b; p.o_st = s.t; p.o_sh = s.h;
}

void set_qkvo_packed(tdb::AttnParams& p, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& o) {
  p.q = q.data_ptr(); p.q_st = q.stride(0); p.q_sh = q.stride(1);
  p.k = k.data_ptr(); p.k_st = k.stride(0); p.k_sh = k.stride(1);
  p.v = v.data_ptr(); p.v_st = v.stride(0); p.v_sh = v.stride(1);
  p.o = o.data_ptr(); p.o_st = o.stride(0); p.o_sh = o.stride(1);
}

int int_size(int64_t n) {
  if (n > INT_MAX) throw py::value_error("size exceeds 2^31 - 1");
  return (int)n;
}

// o is (B, H, L, D) over [B, L, H, D] memory.
Tensor fixed_output(const Tensor& q) {
  const int64_t B = q.size(0), H = q.size(1), L = q.size(2), D = q.size(3);
  return at::empty_strided({B, H, L, D}, {L * H * D, D, H * D, 1}, q.options());
}

Tensor lens_on_device(const Tensor& seqlens, int64_t B, const Tensor& q) {
  Tensor s = seqlens.to(q.device(), at::kInt).contiguous();
  if (s.numel() != B) throw py::value_error("seqlens must have one entry per batch row");
  return s;
}

using Result = std::tuple<Tensor, py::object, py::object>;      // o, lse or None, status (see Status::finish) or an error code

Result launch(tdb::AttnParams& p, int dtype, int kernel, int dev, Tensor o, const Tensor& lse, bool check) {
  const c10::cuda::CUDAStream stream = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)dev);
  Status st(dev, p);
  const Tensor partial = partial_scratch(p, dtype, kernel, o);
  const int rc = tdb_run_attn(&p, dtype, kernel, stream);
  py::object lse_out = lse.defined() ? py::cast(lse) : py::none();
  if (rc) {
    st.failed(stream);
    return {o, lse_out, py::int_(rc)};
  }
  return {o, lse_out, st.finish(check, stream)};
}

// Distance-expanded copies of both tables (bf16, head_dim 64) with one allocation and one launch: [1 or 2, H, rows, 64].
Tensor expand_both(const OptTensor& kr, const OptTensor& qr, const Tensor& idx, int64_t exp_delta_max) {
  const Tensor& some = kr ? *kr : *qr;
  const int64_t H = some.size(0), two_span = some.size(1), exp_rows = (2 * exp_delta_max + 1 + 7) / 8 * 8;
  c10::cuda::CUDAGuard guard(some.device());
  const int n = (kr ? 1 : 0) + (qr ? 1 : 0);
  Tensor both = at::empty({n, H, exp_rows, 64}, some.options());
  char* e = static_cast<char*>(both.data_ptr());
  const int rc = tdb_expand_pair(ptr(kr), ptr(qr), idx.data_ptr<int16_t>(), (int)((idx.numel() - 1) / 2), (int)H, (int)two_span,
                                 (int)exp_delta_max, (int)exp_rows, kr ? e : nullptr, qr ? e + (kr ? both.nbytes() / 2 : 0) : nullptr,
                                 c10::cuda::getCurrentCUDAStream().stream());
  if (rc) throw std::runtime_error(std::string("libtdb_b200: ") + tdb_last_error());
  return both;
}
// Tables of one call are expanded only for a kernel that reads them so (the CUDA-core kernel does not, in either type).  Returns the
// expanded ones, for p to point into.
Tensor expand_for(tdb::AttnParams& p, const Tables* tables, int dtype, int kernel) {
  if (!tables || !tables->one_call || dtype != TDB_DTYPE_BF16 || kernel == TDB_KERNEL_SIMT) return {};
  p.direct_tables = tdb_takes_direct_tables(&p, dtype, kernel);
  if (p.direct_tables) return {};
  const Tensor both = expand_both(tables->kr, tables->qr, *tables->idx, tables->exp_delta_max);
  char* e = static_cast<char*>(both.data_ptr());
  p.kr_exp = tables->kr ? e : nullptr;
  p.qr_exp = tables->qr ? e + (tables->kr ? both.nbytes() / 2 : 0) : nullptr;
  return both;
}

Result attn_fixed(const Tensor& q, const Tensor& k, const Tensor& v, const Tables* tables, const OptTensor& seqlens,
                  double sm_scale, int kernel, bool return_lse, bool check) {
  const int dev = device_of({&q, &k, &v, seqlens ? &*seqlens : nullptr});
  check_qkv(q, k, v, 4, "(B, H, L, D); cross-attention lengths are not supported");
  const int code = dtype_code(q);
  check_rows(q, k, v);
  c10::cuda::CUDAGuard guard((c10::DeviceIndex)dev);
  const int64_t B = q.size(0), H = q.size(1), L = q.size(2);
  Tensor o = fixed_output(q), lse;
  if (return_lse) lse = at::empty({B, H, L}, q.options().dtype(at::kFloat));
  if (B == 0 || L == 0) return {o, lse.defined() ? py::cast(lse) : py::none(), py::none()};
  Tensor lens;
  if (seqlens) lens = lens_on_device(*seqlens, B, q);
  tdb::AttnParams p{};
  set_qkvo_fixed(p, q, k, v, o);
  if (tables) tables->fill(p, q);
  p.seqlens = lens.defined() ? lens.data_ptr<int32_t>() : nullptr;
  p.n_seqs = int_size(B); p.L = int_size(L); p.total_tokens = B * L; p.H = int_size(H); p.D = int_size(q.size(3));
  p.sm_scale = (float)sm_scale;
  if (return_lse) { p.lse = lse.data_ptr<float>(); p.lse_sb = H * L; p.lse_sh = L; }
  const Tensor expanded = expand_for(p, tables, code, kernel);
  return launch(p, code, kernel, dev, o, lse, check);
}

void check_offsets(const Tensor& cu) {
  if (cu.scalar_type() != at::kInt || cu.dim() != 1 || cu.numel() < 1)
    throw py::value_error("cu_seqlens must be a 1-D int32 tensor of n_seqs + 1 offsets");
}

Result attn_packed(const Tensor& q, const Tensor& k, const Tensor& v, const Tables* tables, const Tensor& cu_seqlens,
                   int64_t max_seqlen, double sm_scale, int kernel, bool return_lse, bool check) {
  const int dev = device_of({&q, &k, &v, &cu_seqlens});
  check_qkv(q, k, v, 3, "(T, H, D)");
  const int code = dtype_code(q);
  check_rows(q, k, v);
  check_offsets(cu_seqlens);
  c10::cuda::CUDAGuard guard((c10::DeviceIndex)dev);
  const Tensor cu = cu_seqlens.contiguous();
  const int64_t T = q.size(0), H = q.size(1), n_seqs = cu.numel() - 1;
  Tensor o = at::empty({T, H, q.size(2)}, q.options()), lse;
  if (return_lse) lse = at::empty({H, T}, q.options().dtype(at::kFloat));
  if (T == 0 || n_seqs == 0) return {o, lse.defined() ? py::cast(lse) : py::none(), py::none()};
  tdb::AttnParams p{};
  set_qkvo_packed(p, q, k, v, o);
  if (tables) tables->fill(p, q);
  p.cu_seqlens = cu.data_ptr<int32_t>(); p.varlen = 1; p.n_seqs = int_size(n_seqs);
  p.L = int_size(max_seqlen); p.total_tokens = T; p.H = int_size(H); p.D = int_size(q.size(2));
  p.sm_scale = (float)sm_scale;
  if (return_lse) { p.lse = lse.data_ptr<float>(); p.lse_sh = T; }
  p.workspace_bytes = tdb_attn_workspace_bytes(p.n_seqs, T);
  const Tensor ws = at::empty({(int64_t)std::max<size_t>(p.workspace_bytes, 16)}, q.options().dtype(at::kByte));
  p.workspace = ws.data_ptr();
  const Tensor expanded = expand_for(p, tables, code, kernel);
  return launch(p, code, kernel, dev, o, lse, check);
}

// The materialised form: c2p / p2c have the leading shape of q and two_span columns.
void set_scores(tdb::AttnParams& p, const Tensor& q, const OptTensor& c2p, const OptTensor& p2c, const Tensor& idx, bool mirrored) {
  const int64_t two_span = (c2p ? *c2p : *p2c).size(-1);
  for (const OptTensor* t : {&c2p, &p2c}) {
    if (!*t) continue;
    const Tensor& x = **t;
    const bool fits = x.dim() == q.dim() && x.sizes().slice(0, x.dim() - 1) == q.sizes().slice(0, q.dim() - 1) && x.size(-1) == two_span;
    if (!fits || x.scalar_type() != q.scalar_type() || x.stride(-1) != 1)
      throw py::value_error(std::string(t == &c2p ? "q_pos" : "k_pos") + " must have q's leading shape, 2*span contiguous columns and q's dtype");
  }
  p.two_span = int_size(two_span);
  p.idx = idx.data_ptr<int16_t>(); p.idx_delta_max = (int)((idx.numel() - 1) / 2);
  p.c2p_scores = ptr(c2p); p.p2c_scores = ptr(p2c);
  p.flags = (c2p ? TDB_FLAG_C2P : 0) | (p2c ? TDB_FLAG_P2C : 0) | (mirrored ? TDB_FLAG_P2C_MIRRORED : 0);
}

Result attn_fixed_scores(const Tensor& q, const Tensor& k, const Tensor& v, const OptTensor& c2p, const OptTensor& p2c,
                         const Tensor& idx, bool mirrored, const OptTensor& seqlens, double sm_scale, bool return_lse, bool check) {
  const int dev = device_of({&q, &k, &v, seqlens ? &*seqlens : nullptr});
  check_qkv(q, k, v, 4, "(B, H, L, D)");
  const int code = dtype_code(q);
  c10::cuda::CUDAGuard guard((c10::DeviceIndex)dev);
  const int64_t B = q.size(0), H = q.size(1), L = q.size(2);
  tdb::AttnParams p{};
  set_scores(p, q, c2p, p2c, idx, mirrored);
  check_rows(q, k, v);
  Tensor o = fixed_output(q), lse;
  if (return_lse) lse = at::empty({B, H, L}, q.options().dtype(at::kFloat));
  if (B == 0 || L == 0) return {o, lse.defined() ? py::cast(lse) : py::none(), py::none()};
  Tensor lens;
  if (seqlens) lens = lens_on_device(*seqlens, B, q);
  set_qkvo_fixed(p, q, k, v, o);
  Strides s;
  if (c2p) { s = fixed_strides(*c2p); p.c2p_sb = s.b; p.c2p_st = s.t; p.c2p_sh = s.h; }
  if (p2c) { s = fixed_strides(*p2c); p.p2c_sb = s.b; p.p2c_st = s.t; p.p2c_sh = s.h; }
  p.seqlens = lens.defined() ? lens.data_ptr<int32_t>() : nullptr;
  p.n_seqs = int_size(B); p.L = int_size(L); p.total_tokens = B * L; p.H = int_size(H); p.D = int_size(q.size(3));
  p.sm_scale = (float)sm_scale;
  if (return_lse) { p.lse = lse.data_ptr<float>(); p.lse_sb = H * L; p.lse_sh = L; }
  return launch(p, code, TDB_KERNEL_SIMT, dev, o, lse, check);
}

Result attn_packed_scores(const Tensor& q, const Tensor& k, const Tensor& v, const OptTensor& c2p, const OptTensor& p2c,
                          const Tensor& idx, bool mirrored, const Tensor& cu_seqlens, int64_t max_seqlen, double sm_scale,
                          bool return_lse, bool check) {
  const int dev = device_of({&q, &k, &v, &cu_seqlens});
  check_qkv(q, k, v, 3, "(T, H, D)");
  const int code = dtype_code(q);
  c10::cuda::CUDAGuard guard((c10::DeviceIndex)dev);
  tdb::AttnParams p{};
  set_scores(p, q, c2p, p2c, idx, mirrored);
  check_rows(q, k, v);
  check_offsets(cu_seqlens);
  const Tensor cu = cu_seqlens.contiguous();
  const int64_t T = q.size(0), H = q.size(1), n_seqs = cu.numel() - 1;
  Tensor o = at::empty({T, H, q.size(2)}, q.options()), lse;
  if (return_lse) lse = at::empty({H, T}, q.options().dtype(at::kFloat));
  if (T == 0 || n_seqs == 0) return {o, lse.defined() ? py::cast(lse) : py::none(), py::none()};
  set_qkvo_packed(p, q, k, v, o);
  if (c2p) { p.c2p_st = c2p->stride(0); p.c2p_sh = c2p->stride(1); }
  if (p2c) { p.p2c_st = p2c->stride(0); p.p2c_sh = p2c->stride(1); }
  p.cu_seqlens = cu.data_ptr<int32_t>(); p.varlen = 1; p.n_seqs = int_size(n_seqs);
  p.L = int_size(max_seqlen); p.total_tokens = T; p.H = int_size(H); p.D = int_size(q.size(2));
  p.sm_scale = (float)sm_scale;
  if (return_lse) { p.lse = lse.data_ptr<float>(); p.lse_sh = T; }
  return launch(p, code, TDB_KERNEL_SIMT, dev, o, lse, check);
}

std::pair<OptTensor, OptTensor> expand_pair(const OptTensor& kr, const OptTensor& qr, const Tensor& idx, int64_t exp_delta_max) {
  const OptTensor k = kr ? OptTensor(kr->contiguous()) : std::nullopt, r = qr ? OptTensor(qr->contiguous()) : std::nullopt;
  const Tensor both = expand_both(k, r, idx, exp_delta_max);
  OptTensor ko, qo;
  if (kr) ko = both.select(0, 0);
  if (qr) qo = both.select(0, both.size(0) - 1);
  return {ko, qo};
}

// ------------------------------------------------------------------------------------------------------- the encoder
Tensor mask_bytes(const Tensor& mask) {
  if (mask.scalar_type() == at::kLong || mask.scalar_type() == at::kBool || mask.scalar_type() == at::kByte) return mask.contiguous();
  return mask.ne(0).contiguous();
}

// A set of modules whose forward the native encoder stands in for, as it was when the plan was made.  The plan holds as long
// as nobody has put a hook, a new child or parameter, or another forward on any of them, and all are in eval mode.  Checked
// on every forward, so it follows pointers instead of looking names up: a module keeps its hook, child and parameter dicts.
// settings: (module, names of attributes) pairs of what else the plan was made from (a norm's eps, an attention's position terms).
class Watch {
 public:
  Watch(const py::list& modules, const py::list& settings) {
    training_ = py::str("training");
    forward_ = py::str("forward");
    const py::object list_type = py::module_::import("torch.nn").attr("ModuleList");
    std::unordered_map<PyObject*, size_t> at;
    at.reserve(modules.size());
    entries_.reserve(modules.size());
    for (py::handle m : modules) {
      Entry e;
      e.module = py::reinterpret_borrow<py::object>(m);
      e.type = Py_TYPE(m.ptr());
      e.runs = (PyObject*)e.type != list_type.ptr();
      e.dict = m.attr("__dict__");
      for (const char* n : {"_forward_hooks", "_forward_pre_hooks"})       // no gradients here, so no backward hooks
        if (e.dict.contains(n)) e.hooks.push_back(e.dict[n]);
      for (const char* part : {"_modules", "_parameters"}) {
        py::dict d = e.dict[part];
        std::vector<py::object> values;
        for (auto kv : d) values.push_back(py::reinterpret_borrow<py::object>(kv.second));
        e.parts.emplace_back(d, std::move(values));
      }
      at[m.ptr()] = entries_.size();
      entries_.push_back(std::move(e));
    }
    for (py::handle s : settings) {
      const py::tuple of = py::reinterpret_borrow<py::tuple>(s), names = of[1];
      const auto found = at.find(of[0].ptr());
      TORCH_CHECK(found != at.end(), "settings of a module that is not watched");
      Entry& e = entries_[found->second];
      e.settings.reserve(names.size());
      for (py::handle name : names) {
        PyObject* now = PyDict_GetItem(e.dict.ptr(), name.ptr());               // null where the attribute is absent
        py::object value = py::reinterpret_borrow<py::object>(now);
        if (now && PyList_Check(now)) value = py::reinterpret_steal<py::object>(PyList_GetSlice(now, 0, PyList_Size(now)));       // may be changed in place
        e.settings.emplace_back(py::reinterpret_borrow<py::object>(name), std::move(value));
      }
    }
  }
  bool holds() const {
    // Some two hundred modules whose objects the last forward has long pushed out of the core's caches: fetched side by side
    // first, since one after the other they cost 95 us.
    for (const Entry& e : entries_) {
      __builtin_prefetch(e.module.ptr());
      prefetch_dict(e.dict.ptr());
      for (const py::dict& h : e.hooks) prefetch_dict(h.ptr());
      for (const auto& part : e.parts) prefetch_dict(part.first.ptr());
    }
    for (const Entry& e : entries_) {
      prefetch_keys(e.dict.ptr());
      if (!e.settings.empty()) prefetch_values(e.dict.ptr());
      for (const auto& part : e.parts)
        if (!part.second.empty()) prefetch_keys(part.first.ptr());
    }
    for (const Entry& e : entries_) {
      if (Py_TYPE(e.module.ptr()) != e.type) return false;
      PyObject* d = e.dict.ptr();
      if (e.runs && (PyDict_GetItem(d, training_.ptr()) != Py_False || PyDict_Contains(d, forward_.ptr()))) return false;
      for (const auto& [name, value] : e.settings) {
        PyObject* now = PyDict_GetItem(d, name.ptr());
        if (now == value.ptr()) continue;
        const int same = now && value ? PyObject_RichCompareBool(now, value.ptr(), Py_EQ) : 0;
        if (same < 0) PyErr_Clear();                 // a value that does not compare is not the one of the plan
        if (same != 1) return false;
      }
      for (const py::dict& h : e.hooks)
        if (PyDict_Size(h.ptr()) != 0) return false;
      for (const auto& [dict, values] : e.parts) {
        if ((size_t)PyDict_Size(dict.ptr()) != values.size()) return false;
        Py_ssize_t pos = 0;
        PyObject *k, *v;
        for (size_t i = 0; PyDict_Next(dict.ptr(), &pos, &k, &v); ++i)
          if (v != values[i].ptr()) return false;
      }
    }
    return true;
  }

 private:
  static void prefetch_dict(PyObject* d) { __builtin_prefetch(&reinterpret_cast<PyDictObject*>(d)->ma_used); }
  static void prefetch_keys(PyObject* d) {
    const char* k = reinterpret_cast<const char*>(reinterpret_cast<PyDictObject*>(d)->ma_keys);
    for (int i = 0; i < 8; ++i) __builtin_prefetch(k + 64 * i);
    if (reinterpret_cast<PyDictObject*>(d)->ma_values) __builtin_prefetch(reinterpret_cast<PyDictObject*>(d)->ma_values);
  }
  static void prefetch_values(PyObject* d) {         // the first line: above
    const char* v = reinterpret_cast<const char*>(reinterpret_cast<PyDictObject*>(d)->ma_values);
    for (int i = 1; v && i < 4; ++i) __builtin_prefetch(v + 64 * i);
  }
  struct Entry {
    py::object module;
    PyTypeObject* type;
    bool runs;                                       // a list has no forward, and its mode means nothing (a new one trains)
    py::dict dict;
    std::vector<std::pair<py::object, py::object>> settings;     // name, value
    std::vector<py::dict> hooks;
    std::vector<std::pair<py::dict, std::vector<py::object>>> parts;
  };
  std::vector<Entry> entries_;
  py::object training_, forward_;
};

bool misaligned(const Tensor& t) { return reinterpret_cast<uintptr_t>(t.data_ptr()) & 15; }

// x itself where the kernels can read it as it is, a copy otherwise (a slice of wider rows, or one that starts anywhere).
Tensor rows_of_16_bytes(const Tensor& x) {
  const Tensor c = x.contiguous();
  return misaligned(c) ? c.clone() : c;
}

int64_t version_of(const Tensor& t) { return t.is_inference() ? 0 : (int64_t)t._version(); }

// y = x W^T + b for bf16, straight through cuBLASLt: the library picks the kernel as it does behind torch's linear, but the
// choice is kept per shape and alignment and nothing else is looked up per call (about 3 us of host time instead of 9).
class Linear {
 public:
  // One per run, with a workspace that nobody else uses on another stream meanwhile.  recording: `stream` is not torch's
  // current one, so what torch would have to do cannot be done.
  Linear(const Tensor& x, cudaStream_t stream, Tensor ws = {}, bool recording = false) : stream_(stream), recording_(recording) {
    own_ = applies(x);
    if (!own_) return;
    handle_ = at::cuda::getCurrentCUDABlasLtHandle();
    ws_ = ws.defined() ? ws : at::empty({(int64_t)WORKSPACE}, x.options().dtype(at::kByte));
  }
  static bool applies(const Tensor& x) {
    return x.scalar_type() == at::kBFloat16 && at::globalContext().allowBF16ReductionCuBLAS() == at::CuBLASReductionOption::AllowReducedPrecisionWithSplitK;
  }
  // False: the caller's torch has to do it.
  bool try_run(Tensor& y, const Tensor& x, const Tensor& w, const Tensor& b) {
    const uintptr_t addresses = reinterpret_cast<uintptr_t>(x.data_ptr()) | reinterpret_cast<uintptr_t>(w.data_ptr()) |
                                reinterpret_cast<uintptr_t>(b.data_ptr()) | reinterpret_cast<uintptr_t>(y.data_ptr());
    if (!own_ || addresses & 15) return false;
    const int64_t T = x.size(0), k = x.size(1), n = w.size(0);
    Plan& p = plan(T, k, n, addresses & 255 ? 16 : 256);
    if (!p.usable) return false;
    const void* bias = b.data_ptr();
    const float one = 1.f, zero = 0.f;
    bool good = cublasLtMatmulDescSetAttribute(p.op, CUBLASLT_MATMUL_DESC_BIAS_POINTER, &bias, sizeof(bias)) == CUBLAS_STATUS_SUCCESS;
    good = good && cublasLtMatmul(handle_, p.op, &one, w.data_ptr(), p.w, x.data_ptr(), p.x, &zero, y.data_ptr(), p.y, y.data_ptr(), p.y, &p.algo,
                                  ws_.data_ptr(), WORKSPACE, stream_) == CUBLAS_STATUS_SUCCESS;
    return good;
  }
  // gelu: y goes through it.  early: see tdb_skinny.
  void operator()(Tensor& y, const Tensor& x, const Tensor& w, const Tensor& b, bool gelu = false, bool early = true) {
    const int64_t T = x.size(0), k = x.size(1), n = w.size(0);
    if (own_ && !(misaligned(x) | misaligned(w) | misaligned(b) | misaligned(y)) && tdb_skinny_applies(T, k, n)) {
      check(tdb_skinny(x.data_ptr(), w.data_ptr(), b.data_ptr(), (int)T, (int)k, (int)n, gelu, early, y.data_ptr(), stream_));
      return;
    }
    product(y, x, w, b);
    if (gelu) check(tdb_gelu(y.data_ptr(), y.numel(), dtype_code(y), stream_));
  }
  static constexpr size_t WORKSPACE = 32u << 20;

 private:
  static void check(int rc) { TORCH_CHECK(rc == 0, "libtdb_b200: ", tdb_last_error(), " (code ", rc, ")"); }
  void product(Tensor& y, const Tensor& x, const Tensor& w, const Tensor& b) {
    if (try_run(y, x, w, b)) return;
    TORCH_CHECK(!recording_, "not recordable");
    at::addmm_out(y, b, x, w.t());
  }
  struct Plan {
    bool usable = false;
    cublasLtMatmulDesc_t op = nullptr;
    cublasLtMatrixLayout_t w = nullptr, x = nullptr, y = nullptr;
    cublasLtMatmulAlgo_t algo;
    ~Plan() {
      if (op) cublasLtMatmulDescDestroy(op);
      for (auto l : {w, x, y})
        if (l) cublasLtMatrixLayoutDestroy(l);
    }
  };
  // alignment: of all four addresses, 256 (what the library takes for granted unless told otherwise, and what an allocation of
  // torch's has) or 16 (parameters that are views of one flat buffer).
  Plan& plan(int64_t T, int64_t k, int64_t n, uint32_t alignment) {
    // per thread (a descriptor is written to before each launch), and bounded: a packed batch brings a new T each time
    thread_local std::map<std::tuple<int, int64_t, int64_t, int64_t, uint32_t>, std::unique_ptr<Plan>> plans;
    int dev = 0;
    cudaGetDevice(&dev);
    const auto key = std::make_tuple(dev, T, k, n, alignment);
    auto it = plans.find(key);
    if (it != plans.end()) return *it->second;
    if (plans.size() >= 256) plans.clear();
    auto p = std::make_unique<Plan>();
    const cublasOperation_t trans = CUBLAS_OP_T;
    const cublasLtEpilogue_t epilogue = CUBLASLT_EPILOGUE_BIAS;
    cublasLtMatmulPreference_t pref = nullptr;
    cublasLtMatmulHeuristicResult_t found{};
    int count = 0;
    bool good = cublasLtMatmulDescCreate(&p->op, CUBLAS_COMPUTE_32F, CUDA_R_32F) == CUBLAS_STATUS_SUCCESS &&
                cublasLtMatmulDescSetAttribute(p->op, CUBLASLT_MATMUL_DESC_TRANSA, &trans, sizeof(trans)) == CUBLAS_STATUS_SUCCESS &&
                cublasLtMatmulDescSetAttribute(p->op, CUBLASLT_MATMUL_DESC_EPILOGUE, &epilogue, sizeof(epilogue)) == CUBLAS_STATUS_SUCCESS &&
                cublasLtMatrixLayoutCreate(&p->w, CUDA_R_16BF, k, n, k) == CUBLAS_STATUS_SUCCESS &&
                cublasLtMatrixLayoutCreate(&p->x, CUDA_R_16BF, k, T, k) == CUBLAS_STATUS_SUCCESS &&
                cublasLtMatrixLayoutCreate(&p->y, CUDA_R_16BF, n, T, n) == CUBLAS_STATUS_SUCCESS &&
                cublasLtMatmulPreferenceCreate(&pref) == CUBLAS_STATUS_SUCCESS &&
                cublasLtMatmulPreferenceSetAttribute(pref, CUBLASLT_MATMUL_PREF_MAX_WORKSPACE_BYTES, &WORKSPACE_BYTES, sizeof(WORKSPACE_BYTES)) == CUBLAS_STATUS_SUCCESS;
    for (auto which : {CUBLASLT_MATMUL_PREF_MIN_ALIGNMENT_A_BYTES, CUBLASLT_MATMUL_PREF_MIN_ALIGNMENT_B_BYTES,
                       CUBLASLT_MATMUL_PREF_MIN_ALIGNMENT_C_BYTES, CUBLASLT_MATMUL_PREF_MIN_ALIGNMENT_D_BYTES})
      good = good && cublasLtMatmulPreferenceSetAttribute(pref, which, &alignment, sizeof(alignment)) == CUBLAS_STATUS_SUCCESS;
    good = good && cublasLtMatmulAlgoGetHeuristic(handle_, p->op, p->w, p->x, p->y, p->y, pref, 1, &found, &count) == CUBLAS_STATUS_SUCCESS && count == 1;
    if (pref) cublasLtMatmulPreferenceDestroy(pref);
    if (good) { p->algo = found.algo; p->usable = true; }
    return *(plans[key] = std::move(p));
  }
  static constexpr uint64_t WORKSPACE_BYTES = WORKSPACE;
  bool own_, recording_;
  cublasLtHandle_t handle_ = nullptr;
  cudaStream_t stream_;
  Tensor ws_;
};

// What is made from a layer's weights.  Never changed once made: a pass that runs without the interpreter lock works from the
// ones it started with, whatever another thread replaces meanwhile.
struct Derived {
  Tensor qkv_w, qkv_b;
  std::optional<Tables> tables;
};
struct AllDerived {
  std::vector<std::shared_ptr<const Derived>> layers;
  uint64_t version = 0;                              // goes up whenever one of them is made anew
  const Derived& operator[](size_t i) const { return *layers[i]; }
};

struct Layer {
  Tensor out_w, out_b, ln1_w, ln1_b, up_w, up_b, down_w, down_b, ln2_w, ln2_b;
  double eps1, eps2, sm_scale;
  std::vector<Tensor> sources;                       // what the derived tensors were made from
  std::vector<std::pair<void*, int64_t>> seen;
  std::shared_ptr<const Derived> derived;
};

// The encoder's layer loop on a token-major [T, hidden] stream: four library matrix products per layer, the fused attention,
// and two residual + LayerNorm kernels and a GELU in between.
class Encoder {
 public:
  Encoder(int heads) : heads_(heads) {}
  ~Encoder() {
    if (ready_) cudaEventDestroy(ready_);
  }
  void add_layer(std::vector<Tensor> w, double eps1, double eps2, double sm_scale, std::vector<Tensor> sources) {
    TORCH_CHECK(w.size() == 10);
    layers_.push_back(Layer{w[0], w[1], w[2], w[3], w[4], w[5], w[6], w[7], w[8], w[9], eps1, eps2, sm_scale, std::move(sources), {}, {}});
  }
  // Layers whose derived tensors are missing, or older than what they were made from.
  std::vector<int> stale() const {
    std::vector<int> r;
    for (size_t i = 0; i < layers_.size(); ++i)
      if (!current(layers_[i])) r.push_back((int)i);
    return r;
  }
  // False: not tensors that the loop can take for inputs like x.
  bool set_derived(int i, const Tensor& x, Tensor qkv_w, Tensor qkv_b, py::object tables) {
    const int64_t hidden = 64 * heads_;
    if (qkv_w.scalar_type() != x.scalar_type() || qkv_w.device() != x.device() || qkv_w.sizes() != at::IntArrayRef{3 * hidden, hidden} ||
        qkv_b.numel() != 3 * hidden)
      return false;
    Layer& l = layers_.at(i);
    auto d = std::make_shared<Derived>(Derived{std::move(qkv_w), std::move(qkv_b), std::nullopt});
    if (!tables.is_none()) d->tables = *tables.cast<const Tables*>();
    l.derived = std::move(d);
    l.seen = stamp(l);
    ++derived_version_;
    return true;
  }
  // The derived tensors for inputs like x were made on the current stream, which may not be done with that.
  void set_ready(const Tensor& x) {
    c10::cuda::CUDAGuard guard(x.device());
    const cudaStream_t stream = c10::cuda::getCurrentCUDAStream().stream();
    if (ready_) {                                                 // of others, made on another stream perhaps
      cuda_ok(cudaStreamWaitEvent(stream, ready_, 0), "cudaStreamWaitEvent");
      cudaEventDestroy(std::exchange(ready_, nullptr));
    }
    if (cudaEventCreateWithFlags(&ready_, cudaEventDisableTiming) == cudaSuccess && cudaEventRecord(ready_, stream) == cudaSuccess) return;
    (void)cudaGetLastError();
    if (ready_) cudaEventDestroy(std::exchange(ready_, nullptr));
    cuda_ok(cudaStreamSynchronize(stream), "cudaStreamSynchronize");
  }
  // Whether the loop can run on x ([.., hidden]) with the parameters as they are now: sizes are taken from x below, vectors of the
  // norms are read 16 bytes at a time, and a parameter's data may have been replaced by another tensor's.
  bool fits(const Tensor& x) const {
    const int64_t hidden = 64 * heads_;
    if (x.size(-1) != hidden) return false;
    for (const Layer& l : layers_) {
      const int64_t inner = l.up_b.numel();
      if (l.out_w.sizes() != at::IntArrayRef{hidden, hidden} || l.up_w.sizes() != at::IntArrayRef{inner, hidden} ||
          l.down_w.sizes() != at::IntArrayRef{hidden, inner})
        return false;
      for (const Tensor* t : {&l.out_b, &l.ln1_w, &l.ln1_b, &l.down_b, &l.ln2_w, &l.ln2_b})
        if (t->numel() != hidden) return false;
      for (const Tensor* t : {&l.ln1_w, &l.ln1_b, &l.ln2_w, &l.ln2_b})
        if (misaligned(*t)) return false;
      for (const Tensor* t : {&l.out_w, &l.out_b, &l.ln1_w, &l.ln1_b, &l.up_w, &l.up_b, &l.down_w, &l.down_b, &l.ln2_w, &l.ln2_b})
        if (t->scalar_type() != x.scalar_type() || t->device() != x.device() || !t->is_contiguous()) return false;
    }
    return true;
  }
  int64_t recordings() const { return recordings_; }
  // x: [T, hidden].  Packed form: cu_seqlens; padded form: batch rows of `length` tokens, all valid.  Returns the outputs of
  // all layers (or of the last one), and the status words that the caller has to look at (see Status).
  std::pair<std::vector<Tensor>, std::vector<Tensor>> run(const Tensor& given, const OptTensor& cu_seqlens, int64_t length, bool every) {
    std::pair<std::vector<Tensor>, std::vector<Tensor>> r;
    auto& [outs, words] = r;
    AllDerived all;
    all.version = derived_version_;
    all.layers.reserve(layers_.size());
    for (const Layer& l : layers_) all.layers.push_back(l.derived);
    c10::cuda::CUDAGuard guard(given.device());
    if (ready_ && at::cuda::currentStreamCaptureStatusMayInitCtx() == at::cuda::CaptureStatus::None) {       // this stream may be another
      const cudaError_t e = cudaEventQuery(ready_);
      if (e == cudaSuccess) {
        cudaEventDestroy(std::exchange(ready_, nullptr));
      } else {
        (void)cudaGetLastError();
        cuda_ok(cudaStreamWaitEvent(c10::cuda::getCurrentCUDAStream().stream(), ready_, 0), "cudaStreamWaitEvent");
      }
    }
    py::gil_scoped_release nogil;
    at::AutoDispatchBelowAutograd below;
    const Tensor x = rows_of_16_bytes(given);
    const c10::cuda::CUDAStream torch_stream = c10::cuda::getCurrentCUDAStream();
    const cudaStream_t stream = torch_stream.stream();
    if (!every) {
      Tensor y = short_stack(all, x, cu_seqlens, length, torch_stream, words);
      if (!y.defined()) y = replay(all, x, cu_seqlens, length, torch_stream);
      if (y.defined()) {
        outs.push_back(y);
        return r;
      }
    }
    Scratch s(*this, x, cu_seqlens);
    Linear linear(x, stream);
    const int dev = x.get_device();
    Tensor in = x;
    for (size_t i = 0; i < layers_.size(); ++i) {
      Tensor out = every || i + 1 == layers_.size() ? at::empty_like(x) : s.z[i & 1];
      layer(layers_[i], all[i], in, out, s, cu_seqlens, length, linear, stream, i > 0, [&](tdb::AttnParams& p) {
        Status st(dev, p);
        const Tensor partial = partial_scratch(p, dtype_code(x), TDB_KERNEL_AUTO, x);
        const int rc = tdb_run_attn(&p, dtype_code(x), TDB_KERNEL_AUTO, stream);
        if (rc) st.failed(stream);
        ok(rc);
        st.defer(torch_stream, words);
      });
      in = out;
      if (every) outs.push_back(out);
    }
    if (!every) outs.push_back(in);
    return r;
  }

 private:
  static std::vector<std::pair<void*, int64_t>> stamp(const Layer& l) {
    std::vector<std::pair<void*, int64_t>> s;
    s.reserve(l.sources.size());
    for (const Tensor& t : l.sources) s.emplace_back(t.data_ptr(), version_of(t));
    return s;
  }
  static bool current(const Layer& l) {
    if (l.seen.size() != l.sources.size()) return false;
    for (size_t i = 0; i < l.seen.size(); ++i)
      if (l.seen[i].first != l.sources[i].data_ptr() || l.seen[i].second != version_of(l.sources[i])) return false;
    return true;
  }
  static void ok(int rc) { TORCH_CHECK(rc == 0, "libtdb_b200: ", tdb_last_error(), " (code ", rc, ")"); }
  static void add_norm(Tensor& x, const Tensor& res, const Tensor& w, const Tensor& b, double eps, int code, cudaStream_t stream) {
    ok(tdb_add_layernorm(x.data_ptr(), res.data_ptr(), w.data_ptr(), b.data_ptr(), (float)eps, x.size(0), (int)x.size(1), code, x.data_ptr(), 1, stream));
  }
  // The buffers of one pass: every layer writes over those of the layer before it.
  struct Scratch {
    Tensor qkv, ctx, y, u, z[2], tiles;
    Scratch(const Encoder& e, const Tensor& x, const OptTensor& cu) {
      const int64_t T = x.size(0), hidden = x.size(1);
      qkv = at::empty({T, 3 * hidden}, x.options());
      ctx = at::empty({T, hidden}, x.options());
      y = at::empty({T, hidden}, x.options());
      u = at::empty({T, e.layers_[0].up_w.size(0)}, x.options());
      z[0] = at::empty({T, hidden}, x.options());
      z[1] = at::empty({T, hidden}, x.options());
      if (cu) tiles = at::empty({(int64_t)tdb_attn_workspace_bytes((int)(cu->numel() - 1), T)}, x.options().dtype(at::kByte));
    }
  };

  template <typename Attention>
  void layer(const Layer& l, const Derived& d, const Tensor& x, Tensor& out, Scratch& s, const OptTensor& cu_seqlens, int64_t length, Linear& linear,
             cudaStream_t stream, bool not_first, Attention attention) {
    const int code = dtype_code(x);
    const int64_t T = x.size(0), hidden = x.size(1), e = x.element_size();
    linear(s.qkv, x, d.qkv_w, d.qkv_b, false, not_first);      // a pass's first kernel starts behind all that came before
    tdb::AttnParams p{};
    char* base = static_cast<char*>(s.qkv.data_ptr());
    p.q = base; p.k = base + e * hidden; p.v = base + 2 * e * hidden; p.o = s.ctx.data_ptr();
    p.q_st = p.k_st = p.v_st = 3 * hidden; p.q_sh = p.k_sh = p.v_sh = p.o_sh = hidden / heads_; p.o_st = hidden;
    if (d.tables) d.tables->fill(p, x);
    p.H = heads_; p.D = (int)(hidden / heads_); p.sm_scale = (float)l.sm_scale; p.total_tokens = T;
    if (cu_seqlens) {
      p.varlen = 1; p.cu_seqlens = cu_seqlens->data_ptr<int32_t>(); p.n_seqs = (int)(cu_seqlens->numel() - 1); p.L = (int)length;
      p.workspace = s.tiles.data_ptr(); p.workspace_bytes = s.tiles.numel(); p.tiles_listed = not_first; p.lengths_known = 1;
    } else {
      p.n_seqs = (int)(T / length); p.L = (int)length;
      p.q_sb = p.k_sb = p.v_sb = 3 * hidden * length; p.o_sb = hidden * length;
    }
    attention(p);
    linear(s.y, s.ctx, l.out_w, l.out_b);
    add_norm(s.y, x, l.ln1_w, l.ln1_b, l.eps1, code, stream);
    linear(s.u, s.y, l.up_w, l.up_b, true);
    linear(out, s.u, l.down_w, l.down_b);
    add_norm(out, s.y, l.ln2_w, l.ln2_b, l.eps2, code, stream);
  }

  // All layers in one kernel (see encoder_short.cu), or nothing where it does not apply.  It needs no recording: it is one launch.
  Tensor short_stack(const AllDerived& all, const Tensor& x, const OptTensor& cu_seqlens, int64_t length, c10::cuda::CUDAStream stream,
                     std::vector<Tensor>& words) {
    const int64_t T = x.size(0), hidden = x.size(1);
    if (!Linear::applies(x) || !tdb_short_stack_applies(T, hidden, layers_[0].up_w.size(0), (int64_t)layers_.size())) return {};
    tdb::ShortStack p{};
    for (size_t i = 0; i < layers_.size(); ++i) {
      const Layer& l = layers_[i];
      const Derived& d = all[i];
      if (l.up_w.size(0) != 4 * hidden) return {};
      for (const Tensor* t : {&d.qkv_w, &d.qkv_b, &l.out_w, &l.out_b, &l.up_w, &l.up_b, &l.down_w, &l.down_b})      // the norms': see fits()
        if (misaligned(*t) || !t->is_contiguous()) return {};
      tdb::AttnParams a{};
      if (d.tables) d.tables->fill(a, x);
      auto b = [](const Tensor& t) { return reinterpret_cast<const __nv_bfloat16*>(t.data_ptr()); };
      p.layer[i] = {b(d.qkv_w), b(d.qkv_b), b(l.out_w), b(l.out_b), b(l.ln1_w), b(l.ln1_b), b(l.up_w), b(l.up_b), b(l.down_w), b(l.down_b),
                    b(l.ln2_w), b(l.ln2_b), static_cast<const __nv_bfloat16*>(a.kr_exp), static_cast<const __nv_bfloat16*>(a.qr_exp),
                    (float)l.eps1, (float)l.eps2, (float)l.sm_scale, a.exp_delta_max, a.exp_rows};
    }
    const Tensor y = at::empty_like(x), scratch = at::empty({10 * T * hidden}, x.options());
    __nv_bfloat16* at = reinterpret_cast<__nv_bfloat16*>(scratch.data_ptr());
    auto take = [&](int64_t columns) { return std::exchange(at, at + T * columns); };
    p.qkv = take(3 * hidden); p.ctx = take(hidden); p.y = take(hidden); p.u = take(4 * hidden); p.z = take(hidden);
    p.x = reinterpret_cast<const __nv_bfloat16*>(x.data_ptr());
    p.out = reinterpret_cast<__nv_bfloat16*>(y.data_ptr());
    p.n_layers = (int)layers_.size(); p.tokens = (int)T;
    p.n_seqs = (int)(cu_seqlens ? cu_seqlens->numel() - 1 : T / length); p.length = (int)length;
    p.cu_seqlens = cu_seqlens ? cu_seqlens->data_ptr<int32_t>() : nullptr;
    tdb::AttnParams reports{};
    Status st(x.get_device(), reports);
    p.status = reports.status; p.counter = reports.counter; p.gave_up = reports.gave_up;
    p.limit_ns = 1000ull * 1000ull * 1000ull;
    if (const int rc = tdb_short_stack(&p, (int)hidden, stream.stream())) {
      st.failed(stream.stream());
      if (rc == TDB_ERR_UNSUPPORTED) return {};      // a part of the device that is too small for all of its blocks
      ok(rc);
    }
    st.defer(stream, words);
    return y;
  }

  // Small passes that the one kernel does not take are bound by the host: eight launches per layer of some 4 us each, for kernels of
  // 2 to 8 us.  A shape that comes a second time on a stream is recorded into a CUDA graph, which belongs to that stream (its buffers are in use until
  // the replay is over), as long as the weights stay where they are.  At most GRAPHS of them.  A shape then has to come COMEBACKS
  // times while the longest unused recording does not come once: only then does it take that one's place.  With any number of
  // shapes in turn the first GRAPHS stay recorded and the others stay eager.
  // us per pass, eager and replayed, and what the pass that records costs beyond an eager one: base model, 128 tokens 659, 562, 730; 2048
  // tokens 1027, 899, 700; large model, 128 tokens 1271, 1086, 1150; 2048 tokens 2337, 2081, 1040.  So a recording has paid for itself after
  // six to eight replays (COMEBACKS).  Twelve shapes in turn of some 30 tokens each, before the one kernel took those: 502 us per pass; 40 shapes 574; all new ones
  // 632 (when every shape that came back pushed the oldest out: 1070 and 1277).  Beyond GRAPH_MAX_ELEMENTS the gain falls (6 M elements 5 %, 9 to 12 M 1 to 2 %) and the
  // buffers grow: a recording at the limit holds 52 MB, and each stream with one 32 MB of workspace.
  static constexpr int GRAPHS = 8, COMEBACKS = 8, SEEN = 64, BLOCK = 128;
  static constexpr int64_t GRAPH_MAX_ELEMENTS = 2048 * 1024;      // T * hidden, see above
  struct Graph {
    int dev = 0, slot = -1;
    Tensor x, out, cu, lt_ws, partial;
    std::unique_ptr<Scratch> scratch;
    std::vector<const void*> weights;
    cudaGraphExec_t exec = nullptr;
    uint64_t used = 0;
    bool refused = false;                                         // could not be recorded: stays eager until the weights move
    ~Graph() {
      if (!exec && slot < 0) return;
      int before = 0;
      cudaGetDevice(&before);
      cudaSetDevice(dev);
      cudaDeviceSynchronize();                                    // it may still be running
      if (exec) cudaGraphExecDestroy(exec);
      cudaSetDevice(before);
      (void)cudaGetLastError();
      if (slot < 0) return;
      StatusPool& p = g_pools[dev];
      std::lock_guard<std::mutex> lock(p.mu);
      bool listed = false;
      for (auto& t : p.pending)
        if (t.slot == slot) {                                     // an unread report: reading it frees the slot
          t.keep = listed;                                        // (once, should two streams have listed it)
          listed = true;
        }
      if (!listed) p.free.push_back(slot);
    }
  };
  // Of a stream, and of no other later (as a caller's handle may be): torch's own id, or CUDA's for a caller's stream.
  using StreamId = std::pair<bool, uint64_t>;
  using Key = std::tuple<int, StreamId, int64_t, int64_t, int64_t>;        // device, stream, tokens, sequences (0: padded form), length

  // A shape without a recording: when it last came with these derived tensors, in passes, the latest at (n - 1) % COMEBACKS.
  struct Seen {
    uint64_t at[COMEBACKS] = {}, n = 0, derived = 0;
    void came(uint64_t pass, uint64_t with) {
      if (std::exchange(derived, with) != with) n = 0;
      at[n++ % COMEBACKS] = pass;
    }
    uint64_t last() const { return at[(n - 1) % COMEBACKS]; }
    bool came_often_since(uint64_t pass) const { return n >= COMEBACKS && at[n % COMEBACKS] > pass; }
  };

  // The recording of this shape for these weights (one to be made, if it has none yet), or null if it is not worth one so far.
  // What has to make room goes to `gone`.
  Graph* recording_of(const Key& key, const AllDerived& all, std::vector<std::unique_ptr<Graph>>& gone) {
    const auto it = graphs_.find(key);
    if (it != graphs_.end()) {
      if (it->second->weights == weight_pointers(all)) return it->second.get();
      gone.push_back(std::move(it->second));                      // weights that change with every pass are not worth another
      graphs_.erase(it);
    }
    Seen& s = seen_[key];
    s.came(++uses_, all.version);
    auto older = [](const auto& a, const auto& b) { return a.second->used < b.second->used; };
    const auto oldest = std::min_element(graphs_.begin(), graphs_.end(), older);
    const bool room = graphs_.size() < GRAPHS;
    if (room ? s.n < 2 : !s.came_often_since(oldest->second->used)) {
      if (seen_.size() > SEEN)
        seen_.erase(std::min_element(seen_.begin(), seen_.end(), [](const auto& a, const auto& b) { return a.second.last() < b.second.last(); }));
      return nullptr;
    }
    seen_.erase(key);
    if (!room) {
      gone.push_back(std::move(oldest->second));
      graphs_.erase(oldest);
    }
    Graph& g = *graphs_.emplace(key, std::make_unique<Graph>()).first->second;
    g.weights = weight_pointers(all);
    return &g;
  }

  std::vector<const void*> weight_pointers(const AllDerived& all) const {
    std::vector<const void*> w;
    w.reserve(layers_.size() * 15);
    for (size_t i = 0; i < layers_.size(); ++i) {
      const Layer& l = layers_[i];
      const Derived& d = all[i];
      for (const Tensor* t : {&d.qkv_w, &d.qkv_b, &l.out_w, &l.out_b, &l.ln1_w, &l.ln1_b, &l.up_w, &l.up_b, &l.down_w, &l.down_b, &l.ln2_w, &l.ln2_b})
        w.push_back(t->data_ptr());
      w.push_back(reinterpret_cast<const void*>(l.up_w.size(0)));        // with the addresses, all that can differ
      w.push_back(d.tables ? ptr(d.tables->kr_exp) : nullptr);
      w.push_back(d.tables ? ptr(d.tables->qr_exp) : nullptr);
    }
    return w;
  }

  Tensor replay(const AllDerived& all, const Tensor& x, const OptTensor& cu_seqlens, int64_t length, c10::cuda::CUDAStream stream) {
    if (x.numel() > GRAPH_MAX_ELEMENTS || !Linear::applies(x) || !x.is_contiguous() ||
        at::cuda::currentStreamCaptureStatusMayInitCtx() != at::cuda::CaptureStatus::None)
      return {};
    const int dev = x.get_device();
    StreamId id(is_external(stream), (uint64_t)stream.id());
    if (id.first) {
      unsigned long long unique = 0;
      if (cudaStreamGetId(stream.stream(), &unique) != cudaSuccess) {
        (void)cudaGetLastError();
        return {};
      }
      id.second = unique;
    }
    const Key key(dev, id, x.size(0), cu_seqlens ? cu_seqlens->numel() - 1 : 0, length);
    std::vector<std::unique_ptr<Graph>> gone;                     // destroyed, which waits for the GPU, without the lock
    std::lock_guard<std::mutex> lock(graph_mu_);
    Graph* g = recording_of(key, all, gone);
    if (!g || g->refused) return {};
    const Tensor y = at::empty_like(x);                           // before a recording takes its buffers
    if (!g->exec) {
      bool recorded;
      try {
        recorded = record(*g, all, x, cu_seqlens, length, id);
      } catch (const c10::OutOfMemoryError&) {                    // a recording's buffers are its own: the pass may fit without
        graphs_.erase(key);
        drop_idle_workspaces();
        return {};
      }
      if (!recorded) {
        auto note = std::make_unique<Graph>();                    // without the buffers
        note->refused = true;
        note->weights = g->weights;
        note->used = ++uses_;
        gone.push_back(std::exchange(graphs_.at(key), std::move(note)));
        return {};
      }
      ++recordings_;
    }
    launch_graph(*g, x, cu_seqlens, y, stream);
    return y;
  }

  // Those of streams whose last graph is gone.
  void drop_idle_workspaces() {
    for (auto w = lt_workspaces_.begin(); w != lt_workspaces_.end();)
      w = w->second.use_count() == 1 ? lt_workspaces_.erase(w) : std::next(w);
  }

  bool record(Graph& g, const AllDerived& all, const Tensor& x, const OptTensor& cu_seqlens, int64_t length, const StreamId& stream_id) {
    g.dev = x.get_device();
    g.slot = acquire(g.dev);
    if (g.slot < 0) return false;
    g.x = at::empty_like(x);
    g.out = at::empty_like(x);
    OptTensor cu;
    if (cu_seqlens) cu = g.cu = at::empty_like(*cu_seqlens);
    g.scratch = std::make_unique<Scratch>(*this, x, cu_seqlens);
    drop_idle_workspaces();
    Tensor& ws = lt_workspaces_[{g.dev, stream_id}];
    if (!ws.defined()) ws = at::empty({(int64_t)Linear::WORKSPACE}, x.options().dtype(at::kByte));
    g.lt_ws = ws;
    if (length > 2 * BLOCK) {                                     // long enough for far key tiles
      const int64_t n = cu_seqlens ? cu_seqlens->numel() - 1 : x.size(0) / length;
      g.partial = at::empty({(x.size(0) / BLOCK + 2 * n + 1) * BLOCK * heads_ * 66}, x.options().dtype(at::kFloat));
    }
    cudaStream_t side = nullptr;
    cudaGraph_t graph = nullptr;
    if (cudaStreamCreateWithFlags(&side, cudaStreamNonBlocking) != cudaSuccess) return false;
    Linear linear(x, side, g.lt_ws, true);                        // makes the library handle, which a capture would not allow
    bool good = cudaStreamBeginCapture(side, cudaStreamCaptureModeThreadLocal) == cudaSuccess;
    if (good) {
      try {
        Tensor in = g.x;
        for (size_t i = 0; good && i < layers_.size(); ++i) {
          Tensor out = i + 1 == layers_.size() ? g.out : g.scratch->z[i & 1];
          layer(layers_[i], all[i], in, out, *g.scratch, cu, length, linear, side, i > 0, [&](tdb::AttnParams& p) {
            p.status = g_pools[g.dev].host + g.slot * SLOT_WORDS;
            p.counter = g_pools[g.dev].ctl + g.slot * SLOT_WORDS;
            p.gave_up = p.counter + 1;
            const int64_t n = tdb_partial_floats(&p, dtype_code(x), TDB_KERNEL_AUTO);
            if (n > 0 && g.partial.defined() && n <= g.partial.numel()) {
              p.part_o = g.partial.data_ptr<float>();
              p.part_ml = p.part_o + n / 66 * 64;
            }
            ok(tdb_run_attn(&p, dtype_code(x), TDB_KERNEL_AUTO, side));
          });
          in = out;
        }
      } catch (const std::exception&) {
        good = false;                                             // e.g. a shape that cuBLASLt leaves to torch: stays eager
      }
      good = (cudaStreamEndCapture(side, &graph) == cudaSuccess) && good && graph;
    }
    good = good && cudaGraphInstantiate(&g.exec, graph, 0) == cudaSuccess;
    if (graph) cudaGraphDestroy(graph);
    cudaStreamDestroy(side);
    if (!good) (void)cudaGetLastError();
    return good;
  }

  void launch_graph(Graph& g, const Tensor& x, const OptTensor& cu_seqlens, const Tensor& y, c10::cuda::CUDAStream torch_stream) {
    const cudaStream_t stream = torch_stream.stream();
    g.used = ++uses_;
    cuda_ok(cudaMemcpyAsync(g.x.data_ptr(), x.data_ptr(), x.nbytes(), cudaMemcpyDeviceToDevice, stream), "copy of the encoder's input");
    if (cu_seqlens) cuda_ok(cudaMemcpyAsync(g.cu.data_ptr(), cu_seqlens->data_ptr(), cu_seqlens->nbytes(), cudaMemcpyDeviceToDevice, stream), "copy of the offsets");
    cuda_ok(cudaGraphLaunch(g.exec, stream), "cudaGraphLaunch");
    cuda_ok(cudaMemcpyAsync(y.data_ptr(), g.out.data_ptr(), y.nbytes(), cudaMemcpyDeviceToDevice, stream), "copy of the encoder's output");
    StatusPool& p = g_pools[g.dev];
    std::lock_guard<std::mutex> lock(p.mu);
    bool listed = false;
    for (auto& t : p.pending)
      if (t.slot == g.slot && t.keep) {                           // the graph is one stream's, so there is one entry at most
        t.mark.renew();
        listed = true;
      }
    if (!listed) p.pending.push_back({g.slot, Mark(torch_stream), true});
  }

  int heads_;
  std::vector<Layer> layers_;
  std::mutex graph_mu_;
  std::map<Key, std::unique_ptr<Graph>> graphs_;
  std::map<Key, Seen> seen_;                                      // the last SEEN of them
  std::map<std::pair<int, StreamId>, Tensor> lt_workspaces_;
  uint64_t uses_ = 0;                                             // passes that looked for a recording
  int64_t recordings_ = 0;
  uint64_t derived_version_ = 0;
  cudaEvent_t ready_ = nullptr;                                   // behind what made them; used with the interpreter lock held
};


// (all ones, right padded, tokens, longest, seqlens, cu_seqlens) of a [B, L] padding mask; one synchronisation.
py::object mask_rows(const Tensor& mask) {
  const Tensor m = mask_bytes(mask);
  const int dev = m.get_device();
  c10::cuda::CUDAGuard guard((c10::DeviceIndex)dev);
  cudaStream_t stream = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)dev).stream();
  const int64_t B = m.size(0), L = m.size(1);
  struct Slot {
    int dev, i;
    ~Slot() { release_unused(dev, i); }
  } slot{dev, acquire(dev)};
  if (slot.i < 0) return py::none();
  int32_t* out = g_pools[dev].host + slot.i * SLOT_WORDS;
  Tensor both;
  int rc;
  cudaError_t e = cudaSuccess;
  int32_t w[4];
  {
    py::gil_scoped_release nogil;
    both = at::empty({2 * B + 1}, m.options().dtype(at::kInt));
    int32_t* lens = both.data_ptr<int32_t>();
    rc = tdb_mask_rows(m.data_ptr(), (int)m.element_size(), (int)B, (int)L, lens, lens + B, g_pools[dev].ctl + slot.i * SLOT_WORDS, out, stream);
    if (!rc) e = cudaStreamSynchronize(stream);
    for (int i = 0; i < 4; ++i) { w[i] = reinterpret_cast<volatile int32_t*>(out)[i]; out[i] = 0; }
  }
  TORCH_CHECK(rc == 0, "libtdb_b200: ", tdb_last_error());
  cuda_ok(e, "cudaStreamSynchronize");
  return py::make_tuple((bool)w[0], (bool)w[1], w[2], w[3], both.narrow(0, 0, B), both.narrow(0, B, B + 1));
}

// A model's input from ids [B, L]: LayerNorm of their embeddings, times the padding mask.  (output, words that somebody has to look at
// or None), or None where the kernel does not take the tensors.  own: ids and mask of any layout, and the words come as a Report, or a tensor, for the
// caller's own check.
py::object embed(const Tensor& given_ids, const Tensor& table, const Tensor& w, const Tensor& b, double eps, const Tensor& given_mask, bool own) {
  const Tensor ids = own ? given_ids.contiguous() : given_ids, mask = own ? given_mask.contiguous() : given_mask;
  const at::ScalarType t = table.scalar_type();
  const int64_t hidden = table.size(1);
  const bool types = (t == at::kFloat || t == at::kBFloat16) && w.scalar_type() == t && b.scalar_type() == t &&
                     (ids.scalar_type() == at::kLong || ids.scalar_type() == at::kInt) &&
                     (mask.scalar_type() == at::kLong || mask.scalar_type() == at::kBool || mask.scalar_type() == at::kByte);
  if (!types || hidden % 8 || hidden > (t == at::kFloat ? 1024 : 2048) || w.numel() != hidden || b.numel() != hidden || ids.numel() == 0 || mask.sizes() != ids.sizes())
    return py::none();
  for (const Tensor* x : {&ids, &table, &w, &b, &mask})
    if (!x->is_cuda() || x->get_device() != ids.get_device() || !x->is_contiguous()) return py::none();
  if (misaligned(table) | misaligned(w) | misaligned(b)) return py::none();
  c10::cuda::CUDAGuard guard(ids.device());
  at::AutoDispatchBelowAutograd below;
  const c10::cuda::CUDAStream stream = c10::cuda::getCurrentCUDAStream();
  Tensor out = at::empty({ids.size(0), ids.size(1), hidden}, table.options());
  tdb::AttnParams reports{};
  Status st(ids.get_device(), reports);
  const int rc = tdb_embed(ids.data_ptr(), (int)ids.element_size(), table.data_ptr(), table.size(0), w.data_ptr(), b.data_ptr(), (float)eps,
                           mask.data_ptr(), (int)mask.element_size(), ids.numel(), (int)hidden, dtype_code(table), out.data_ptr(), reports.status, stream);
  if (rc) st.failed(stream);
  TORCH_CHECK(rc == 0, "libtdb_b200: ", tdb_last_error());
  return py::make_tuple(out, own ? st.report(stream) : st.finish(false, stream));
}

// The valid rows of x [B, L, hidden] back to back, and each token's place in that stream (-1: padding).
std::pair<Tensor, Tensor> pack_rows(const Tensor& x, const Tensor& mask, const Tensor& cu, int64_t tokens) {
  c10::cuda::CUDAGuard guard(x.device());
  cudaStream_t stream = c10::cuda::getCurrentCUDAStream().stream();
  const Tensor m = mask_bytes(mask), xc = rows_of_16_bytes(x);
  const int64_t B = x.size(0), L = x.size(1), hidden = x.size(2);
  Tensor pos = at::empty({B * L}, cu.options()), out = at::empty({tokens, hidden}, x.options());
  int rc = tdb_mask_positions(m.data_ptr(), (int)m.element_size(), cu.data_ptr<int32_t>(), (int)B, (int)L, pos.data_ptr<int32_t>(), stream);
  if (!rc) rc = tdb_repack(1, xc.data_ptr(), pos.data_ptr<int32_t>(), B * L, (int)(hidden * x.element_size()), out.data_ptr(), stream);
  TORCH_CHECK(rc == 0, "libtdb_b200: ", tdb_last_error());
  return {out, pos};
}

// The inverse: [B, L, hidden] with zeros at the padding.
Tensor unpack_rows(const Tensor& x, const Tensor& pos, int64_t B, int64_t L) {
  c10::cuda::CUDAGuard guard(x.device());
  Tensor out = at::empty({B, L, x.size(1)}, x.options());
  const int rc = tdb_repack(0, x.data_ptr(), pos.data_ptr<int32_t>(), B * L, (int)(x.size(1) * x.element_size()), out.data_ptr(),
                            c10::cuda::getCurrentCUDAStream().stream());
  TORCH_CHECK(rc == 0, "libtdb_b200: ", tdb_last_error());
  return out;
}

// The tables of one call from its projected tables (rows of 64), in the call's dtype.
Tables* call_tables(const OptTensor& kr, const OptTensor& qr, const Tensor& q, const Tensor& idx, int64_t exp_delta_max) {
  auto fit = [&](const OptTensor& t) -> OptTensor {
    if (!t) return std::nullopt;
    device_of({&q, &*t});
    if (t->scalar_type() == q.scalar_type() && t->is_contiguous()) return t;
    return t->to(q.scalar_type()).contiguous();
  };
  const OptTensor k = fit(kr), r = fit(qr);
  return new Tables{k, r, idx, {}, {}, (int)(k ? *k : *r).size(1), (int)((idx.numel() - 1) / 2), (int)exp_delta_max,
                    (int)((2 * exp_delta_max + 1 + 7) / 8 * 8), true};
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  py::class_<Tables>(m, "Tables")
      .def(py::init([](OptTensor kr, OptTensor qr, OptTensor idx, OptTensor kr_exp, OptTensor qr_exp, int two_span, int idx_delta_max,
                       int exp_delta_max, int exp_rows) {
        return new Tables{kr, qr, idx, kr_exp, qr_exp, two_span, idx_delta_max, exp_delta_max, exp_rows, false};
      }));
  m.def("attn_fixed", &attn_fixed);
  m.def("attn_packed", &attn_packed);
  m.def("attn_fixed_scores", &attn_fixed_scores);
  m.def("attn_packed_scores", &attn_packed_scores);
  m.def("expand_pair", &expand_pair);
  m.def("call_tables", &call_tables);
  py::class_<Report>(m, "Report");
  m.def("drain_pending", &drain_pending, py::arg("own") = py::none());
  py::class_<Watch>(m, "Watch").def(py::init<const py::list&, const py::list&>(), py::arg("modules"), py::arg("settings") = py::list()).def("holds", &Watch::holds);
  py::class_<Encoder>(m, "Encoder")
      .def(py::init<int>())
      .def("add_layer", &Encoder::add_layer)
      .def("stale", &Encoder::stale)
      .def("set_derived", &Encoder::set_derived)
      .def("set_ready", &Encoder::set_ready)
      .def("fits", &Encoder::fits)
      .def_property_readonly("recordings", &Encoder::recordings)
      .def("run", &Encoder::run);
  m.def("add_layernorm", [](const Tensor& x, const Tensor& res, const Tensor& w, const Tensor& b, double eps, const Tensor& out) {
    c10::cuda::CUDAGuard guard(x.device());
    return tdb_add_layernorm(x.data_ptr(), res.data_ptr(), w.data_ptr(), b.data_ptr(), (float)eps, x.size(0), (int)x.size(1), dtype_code(x),
                             out.data_ptr(), 0, c10::cuda::getCurrentCUDAStream().stream());
  });
  m.def("skinny", [](const Tensor& x, const Tensor& w, const Tensor& b, bool gelu, const Tensor& y) {
    c10::cuda::CUDAGuard guard(x.device());
    if (!tdb_skinny_applies(x.size(0), x.size(1), w.size(0))) return (int)TDB_ERR_SHAPE;
    return tdb_skinny(x.data_ptr(), w.data_ptr(), b.data_ptr(), (int)x.size(0), (int)x.size(1), (int)w.size(0), gelu, 0, y.data_ptr(),
                      c10::cuda::getCurrentCUDAStream().stream());
  });
  m.def("gelu_", [](const Tensor& x) {
    c10::cuda::CUDAGuard guard(x.device());
    return tdb_gelu(x.data_ptr(), x.numel(), dtype_code(x), c10::cuda::getCurrentCUDAStream().stream());
  });
  m.def("embed", &embed, py::arg("ids"), py::arg("table"), py::arg("w"), py::arg("b"), py::arg("eps"), py::arg("mask"), py::arg("own") = false);
  m.def("mask_rows", &mask_rows);
  m.def("pack_rows", &pack_rows);
  m.def("unpack_rows", &unpack_rows);
}
