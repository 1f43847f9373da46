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
#include <cuda_runtime.h>

#include <mutex>
#include <vector>

#include "tdb_internal.h"

namespace py = pybind11;
using at::Tensor;
using OptTensor = std::optional<Tensor>;

namespace {

constexpr int MAX_DEV = 64, SLOTS = 256, SLOT_WORDS = 4;

struct StatusPool {
  std::mutex mu;
  int32_t* host = nullptr;        // SLOTS x 4 words, pinned and mapped
  int32_t* ctl = nullptr;         // SLOTS x 4 words on the device: work counter, gave-up flag
  std::vector<int> free;
  struct Pending { int slot; cudaStream_t stream; };
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

// Read the words of a slot whose launch has finished, and hand the slot back clean.
std::pair<int, int> collect(int dev, int slot) {
  StatusPool& p = g_pools[dev];
  volatile int32_t* w = p.host + slot * SLOT_WORDS;
  const std::pair<int, int> r(w[0], w[1]);
  if (r.first || r.second) {
    for (int i = 0; i < SLOT_WORDS; ++i) w[i] = 0;
    // a launch that gave up may have left its work counter and flag set
    cudaMemset(p.ctl + slot * SLOT_WORDS, 0, SLOT_WORDS * 4);
    cudaDeviceSynchronize();
  }
  std::lock_guard<std::mutex> lock(p.mu);
  p.free.push_back(slot);
  return r;
}

void release_unused(int dev, int slot) {
  if (slot < 0) return;
  std::lock_guard<std::mutex> lock(g_pools[dev].mu);
  g_pools[dev].free.push_back(slot);
}

// Where one call reports: a pool slot, or words of its own.
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
      own = at::zeros({4}, at::TensorOptions().dtype(at::kInt).device(at::kCUDA, (c10::DeviceIndex)dev));
      p.status = own.data_ptr<int32_t>();
    }
  }
  // What the caller in Python gets to see: None (fine, or deferred into the pool), (word 0, word 1), or the tensor of words.
  py::object finish(bool check, cudaStream_t stream) {
    if (slot < 0) return py::cast(own);
    if (!check) {
      std::lock_guard<std::mutex> lock(g_pools[dev].mu);
      g_pools[dev].pending.push_back({slot, stream});
      return py::none();
    }
    cudaError_t e;
    {
      py::gil_scoped_release nogil;
      e = cudaStreamSynchronize(stream);
    }
    const auto r = collect(dev, slot);
    cuda_ok(e, "cudaStreamSynchronize");
    if (r.first || r.second) return py::make_tuple(r.first, r.second);
    return py::none();
  }
};

// Words of every launch with a deferred check, all devices: None, or the largest of each word.
py::object drain_pending() {
  int w0 = 0, w1 = 0;
  for (int dev = 0; dev < MAX_DEV; ++dev) {
    StatusPool& p = g_pools[dev];
    std::vector<StatusPool::Pending> take;
    {
      std::lock_guard<std::mutex> lock(p.mu);
      take.swap(p.pending);
    }
    if (take.empty()) continue;
    c10::cuda::CUDAGuard guard((c10::DeviceIndex)dev);
    cudaError_t e = cudaSuccess;
    {
      py::gil_scoped_release nogil;
      cudaStream_t last = nullptr;
      bool any = false;
      for (const auto& t : take) {
        if (any && t.stream == last) continue;
        last = t.stream; any = true;
        if (cudaStreamSynchronize(t.stream) == cudaSuccess) continue;
        (void)cudaGetLastError();                       // e.g. a stream that its owner has destroyed
        if ((e = cudaDeviceSynchronize()) != cudaSuccess) break;
      }
    }
    for (const auto& t : take) {
      const auto r = collect(dev, t.slot);
      w0 = std::max(w0, r.first); w1 = std::max(w1, r.second);
    }
    cuda_ok(e, "synchronisation");
  }
  if (w0 || w1) return py::make_tuple(w0, w1);
  return py::none();
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
  void fill(tdb::AttnParams& p, const Tensor& q) const {
    for (const OptTensor* t : {&kr, &qr})
      if (t->has_value() && (*t)->scalar_type() != q.scalar_type()) throw py::value_error("relative tables must have the dtype of q");
    p.kr = ptr(kr); p.qr = ptr(qr); p.two_span = two_span;
    p.idx = static_cast<const int16_t*>(ptr(idx)); p.idx_delta_max = idx_delta_max;
    p.kr_exp = ptr(kr_exp); p.qr_exp = ptr(qr_exp); p.exp_delta_max = exp_delta_max; p.exp_rows = exp_rows;
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
  cudaStream_t stream = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)dev).stream();
  Status st(dev, p);
  const int rc = tdb_run_attn(&p, dtype, kernel, stream);
  py::object lse_out = lse.defined() ? py::cast(lse) : py::none();
  if (rc) {
    release_unused(dev, st.slot);
    return {o, lse_out, py::int_(rc)};
  }
  return {o, lse_out, st.finish(check, stream)};
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

// Distance-expanded copies of both tables (bf16, head_dim 64) with one allocation and one launch.
std::pair<OptTensor, OptTensor> expand_pair(const OptTensor& kr, const OptTensor& qr, const Tensor& idx, int64_t exp_delta_max) {
  const Tensor& some = kr ? *kr : *qr;
  const int64_t H = some.size(0), two_span = some.size(1), exp_rows = (2 * exp_delta_max + 1 + 7) / 8 * 8;
  c10::cuda::CUDAGuard guard(some.device());
  const int n = (kr ? 1 : 0) + (qr ? 1 : 0);
  Tensor both = at::empty({n, H, exp_rows, 64}, some.options());
  OptTensor ko, qo;
  if (kr) ko = both.select(0, 0);
  if (qr) qo = both.select(0, n - 1);
  const int rc = tdb_expand_pair(ptr(kr), ptr(qr), idx.data_ptr<int16_t>(), (int)((idx.numel() - 1) / 2), (int)H, (int)two_span,
                                 (int)exp_delta_max, (int)exp_rows, ptr(ko), ptr(qo), c10::cuda::getCurrentCUDAStream().stream());
  if (rc) throw std::runtime_error(std::string("libtdb_b200: ") + tdb_last_error());
  return {ko, qo};
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  py::class_<Tables>(m, "Tables")
      .def(py::init([](OptTensor kr, OptTensor qr, OptTensor idx, OptTensor kr_exp, OptTensor qr_exp, int two_span, int idx_delta_max,
                       int exp_delta_max, int exp_rows) {
        return new Tables{kr, qr, idx, kr_exp, qr_exp, two_span, idx_delta_max, exp_delta_max, exp_rows};
      }));
  m.def("attn_fixed", &attn_fixed);
  m.def("attn_packed", &attn_packed);
  m.def("attn_fixed_scores", &attn_fixed_scores);
  m.def("attn_packed_scores", &attn_packed_scores);
  m.def("expand_pair", &expand_pair);
  m.def("drain_pending", &drain_pending);
}
