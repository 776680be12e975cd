// Host path of the fused attention operators: one dispatcher operator for the whole forward of an attention layer and one for its
// backward, registered with C++ autograd, over the C ABI of libllsa_b200.so.
//
//   llsa_b200::layer_fwd   (RMSNorm, rotation,) pooling, selection, attention  -> [o, saved] or [o, saved, q', k']
//   llsa_b200::layer_bwd   index transpose, attention backward(, rotation and norm backwards) -> [dq, dk, dv(, dwq, dwk)]
//   llsa_b200::attn_fwd / attn_bwd   the attention core alone, for callers that pool and select themselves
//
// A small layer is bound by the host: some ten kernel launches of 2 us each, next to what the operator layer in front of them
// costs.  The same sequence driven from Python (torch.library custom operators with a Python autograd formula, ctypes descriptors)
// took 0.19 ms forward and 0.75 ms forward + backward whatever the size; B=1 H=2 N=1024 fp32 forward + backward has 0.29 ms of
// kernels.  Here an operator makes three or four allocations (the tensors of a call that live equally long share one), builds the
// descriptors on the stack and issues the launches.
#include <ATen/ATen.h>
#include <ATen/core/dispatch/Dispatcher.h>
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/CUDAEvent.h>
#include <c10/cuda/CUDAGuard.h>
#include <pybind11/pybind11.h>
#include <torch/csrc/autograd/autograd_not_implemented_fallback.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/library.h>

#include <array>
#include <atomic>
#include <mutex>
#include <optional>

#include "../../include/llsa_b200.h"

namespace {

using at::Tensor;
using OptTensor = std::optional<Tensor>;
using torch::autograd::variable_list;

// ------------------------------------------------------------------ settings (mirrored from ops.py)
enum Flag : int {
  kForceGeneric = 1,    // every stage on the scalar kernels
  kNoTcgen05 = 2,       // pooled stages on the mma.sync kernels
  kExactGrad = 4,       // one level: token weight kept in the pooled-key gradients
  kTwoPass = 8,         // long pooled lists: two passes over the keys for every row
  kDeviceChecks = 16,   // read the status word back after every operator
  kNoOverlap = 32,      // index transpose on the main stream
};
std::atomic<int> g_flags{0}, g_wait_limit{0};
std::atomic<bool> g_has_hook{false};
PyObject* g_hook = nullptr;      // guarded by the GIL

bool flag(Flag f) { return g_flags.load(std::memory_order_relaxed) & f; }

void mark(const char* name) {
  if (!g_has_hook.load(std::memory_order_relaxed)) return;
  pybind11::gil_scoped_acquire gil;
  if (g_hook) pybind11::reinterpret_borrow<pybind11::object>(g_hook)(name);
}

// The marks of the most recent forward that was asked to leave them (which rows its second round redid; undefined if it made none): the
// debug forms of the operators ask, every other call's marks end with the call.
thread_local bool t_keep_marks = false;
std::mutex g_redo_mutex;
Tensor& last_redo() {
  static Tensor* t = new Tensor();      // not destroyed at exit: the CUDA context may be gone by then
  return *t;
}

// ------------------------------------------------------------------ descriptors
int dtype_code(at::ScalarType t) {
  switch (t) {
    case at::kFloat: return LLSA_F32;
    case at::kBFloat16: return LLSA_BF16;
    case at::kInt: return LLSA_I32;
    case at::kLong: return LLSA_I64;
    default: TORCH_CHECK_TYPE(false, "llsa_b200 supports float32 and bfloat16 tensors, got ", t);
  }
}

LlsaTensor desc(const Tensor& t) {
  LlsaTensor d;
  d.ptr = t.data_ptr();
  d.dtype = dtype_code(t.scalar_type());
  d.ndim = (int32_t) t.dim();
  TORCH_CHECK(t.dim() <= 4, "llsa_b200: tensors of at most 4 dimensions, got ", t.dim());
  for (int i = 0; i < d.ndim; ++i) {
    d.shape[i] = t.size(i);
    d.stride[i] = t.stride(i);
  }
  return d;
}

LlsaTensor packed(void* p, int dtype, std::initializer_list<int64_t> shape) {
  LlsaTensor d;
  d.ptr = p;
  d.dtype = dtype;
  d.ndim = (int32_t) shape.size();
  int i = 0;
  for (int64_t s : shape) d.shape[i++] = s;
  int64_t st = 1;
  for (i = d.ndim - 1; i >= 0; --i) {
    d.stride[i] = st;
    st *= d.shape[i];
  }
  return d;
}

void ok(int rc, const char* what) {
  TORCH_CHECK(rc == 0, "llsa_b200.", what, " failed (code ", rc, "): ", llsa_last_error_string());
}

void need_cuda(const Tensor& t) {
  TORCH_CHECK(t.is_cuda(), "llsa_b200 runs on CUDA tensors only (got a ", t.device().type(), " tensor); there is no CPU path");
}

// Operands the caller may leave out are undefined tensors here.  A host pointer in a descriptor would be read by a kernel.
void need_cuda(std::initializer_list<Tensor> ts) {
  for (const Tensor& t : ts)
    if (t.defined()) need_cuda(t);
}
Tensor or_none(const OptTensor& t) { return t.value_or(Tensor()); }

void check_float(std::initializer_list<const Tensor*> ts) {
  const at::ScalarType dt = (*ts.begin())->scalar_type();
  TORCH_CHECK_TYPE(dt == at::kFloat || dt == at::kBFloat16, "llsa_b200 supports float32 and bfloat16 tensors, got ", dt);
  for (const Tensor* t : ts) TORCH_CHECK_TYPE(t->scalar_type() == dt, "llsa_b200: all floating-point operands must share one dtype");
}

// Unit channel stride; bf16 rows on 32-byte boundaries (256-bit loads of the tensor-core kernels), fp32 rows on 16-byte ones; no rows that
// overlap, such as those of an expanded tensor: tensor maps are specified for strides that reach past a row.
bool rows_ok(const Tensor& t) {
  const int64_t align = t.scalar_type() == at::kBFloat16 ? 32 : 16, per = align / t.element_size();
  if (t.stride(-1) != 1 || (uintptr_t) t.data_ptr() % align) return false;
  for (int64_t i = 0; i + 1 < t.dim(); ++i)
    if (t.size(i) != 1 && (t.stride(i) % per || t.stride(i) < t.size(-1))) return false;
  return true;
}
Tensor prep(const Tensor& t) { return rows_ok(t) ? t : t.contiguous(); }
Tensor cont(const Tensor& t) { return t.is_contiguous() ? t : t.contiguous(); }
bool table_ok(const Tensor& f) {
  return f.stride(-1) == 1 && (uintptr_t) f.data_ptr() % 16 == 0 && (f.stride(0) * f.element_size()) % 16 == 0;
}

// Blocks carved out of one allocation, every one on a 256-byte boundary.
struct Carver {
  int64_t off = 0;
  int64_t take(int64_t bytes) {
    const int64_t at = off;
    off += (bytes + 255) / 256 * 256;
    return at;
  }
};
Tensor byte_buffer(int64_t n, const Tensor& like) {
  return at::empty({n}, at::TensorOptions().dtype(at::kByte).device(like.device()));
}

// ------------------------------------------------------------------ status word
struct Status {
  Tensor word;
  explicit Status(const Tensor& like) {
    if (flag(kDeviceChecks)) word = at::zeros({1}, at::TensorOptions().dtype(at::kInt).device(like.device()));
  }
  int32_t* ptr() const { return word.defined() ? (int32_t*) word.data_ptr() : nullptr; }
  void check(const char* what) const {
    if (word.defined()) ok(llsa_status_check(word.item<int32_t>()), what);
  }
};

// ------------------------------------------------------------------ sizes of one problem
struct Dims {
  int64_t B, H, N, Nq, n1, n2, nq1, nq2;
  int bs;
  Dims(const Tensor& q, const Tensor& k, int64_t block) {
    TORCH_CHECK(q.dim() == 4 && k.dim() == 4, "llsa_b200: q, k, v must be [B,H,N,D]");
    TORCH_CHECK(block >= 1, "llsa_b200: bad block size ", block);
    bs = (int) block;
    B = q.size(0); H = q.size(1); Nq = q.size(2); N = k.size(2);
    n1 = N / bs; n2 = n1 / bs; nq1 = Nq / bs; nq2 = nq1 / bs;
  }
};

// What the backward of a layer needs beside q, k, v and o, in one buffer.  ops.py unpacks the same layout (_saved_specs).
struct Saved {
  int64_t lse, indices, p_indices = 0, pk, pv, pk2 = 0, pv2 = 0, bytes;
  Saved(const Dims& d, int64_t D, int64_t esize, int64_t topk1, int64_t topk2, int levels) {
    Carver c;
    const int64_t BH = d.B * d.H;
    lse = c.take(BH * d.Nq * 4);
    indices = c.take(BH * d.nq1 * topk1 * 4);
    if (levels == 2) p_indices = c.take(BH * d.nq2 * topk2 * 4);
    pk = c.take(BH * d.n1 * D * esize);
    pv = c.take(BH * d.n1 * D * esize);
    if (levels == 2) {
      pk2 = c.take(BH * d.n2 * D * esize);
      pv2 = c.take(BH * d.n2 * D * esize);
    }
    bytes = c.off;
  }
};

// ------------------------------------------------------------------ attention core
struct Core {      // operands common to forward and backward
  LlsaTensor q, k, v, pk, pv, pk2, pv2, indices, p_indices, o, lse;
  bool two = false;
  LlsaAttnArgs args(int topk, int topk_p, int bs, double w1, double w2) const {
    LlsaAttnArgs a;
    memset(&a, 0, sizeof(a));
    a.q = &q; a.k = &k; a.v = &v; a.pk = &pk; a.pv = &pv;
    if (two) { a.pk2 = &pk2; a.pv2 = &pv2; a.p_indices = &p_indices; }
    a.indices = &indices; a.o = &o; a.lse = &lse;
    a.topk = topk; a.topk_p = topk_p; a.block_size = bs;
    a.token_weight = (float) w1; a.token_weight_2 = (float) w2;
    a.force_generic = flag(kForceGeneric);
    a.no_tcgen05 = flag(kNoTcgen05);
    a.wait_limit = g_wait_limit.load(std::memory_order_relaxed);
    return a;
  }
};

void keep_redo(const Tensor& t) {
  std::lock_guard<std::mutex> lock(g_redo_mutex);
  last_redo() = t;
}

void run_fwd(const Core& c, int topk, int topk_p, int bs, double w1, double w2, const Tensor& like, const Status& status, cudaStream_t st) {
  LlsaAttnArgs a = c.args(topk, topk_p, bs, w1, w2);
  LlsaTensor r, rd;
  Tensor redo, rem;
  const int64_t n_redo = flag(kTwoPass) ? 0 : llsa_attn_fwd_redo_elems(&a);      // marks of the one-pass form (include/llsa_b200.h: fwd_redo)
  if (n_redo) {
    redo = at::empty({n_redo}, like.options().dtype(at::kInt));
    r = desc(redo);
    a.fwd_redo = &r;
  }
  if (llsa_attn_remainder_elems(&a, 0)) {
    rem = at::empty({c.q.shape[0], c.q.shape[1], c.q.shape[2], c.q.shape[3]}, like.options());
    rd = desc(rem);
    a.remainder = &rd;
  }
  a.status = status.ptr();
  mark("attn_fwd");
  ok(llsa_attn_fwd(&a, st), "attn_fwd");
  mark("end");
  status.check("attn_fwd");
  if (t_keep_marks) keep_redo(redo);
}

// The values' share of the pooling pass runs beside the two-level selection, which reads little and leaves SMs idle, instead of in front of it: one launch
// more.  Below the first line the host is the pace of an eager forward + backward; above the second the refinement fills the SMs one and a half times and
// more, and only its end is left for the values.  us, in front / beside, forward + backward, the same in a graph, forward alone: B=1 H=6 N=4096 (1,536
// query blocks) 112.7 / 115.8, 80.0 / 78.7, 25.2 / 24.5; B=3 H=5 N=5376 (5,040) 142.8 / 138.5, 140.3 / 138.8, 39.3 / 39.4; B=1 H=6 N=16384 (6,144) 165.3 / 160.1, 164.3 /
// 160.2, 45.3 / 44.9; B=2 H=6 N=16384 (12,288) 278.0 / 270.1, 275.7 / 271.0, 78.9 / 75.4; B=4 H=6 N=16384 (24,576) 505 / 499, 507 / 501, 153 / 146; B=2 H=4 N=65536
// (32,768) 791 / 795, 781 / 781, 228.8 / 225.5; B=8 H=6 N=16384 (49,152) 951 / 960 eager; B=1 H=6 N=262144 (98,304) forward 1034 / 1045.
// One level: no gain (B=2 H=4 N=16384 323 / 325).  With a norm or a rotation the values are a fifth of the pass: B=1 H=6 N=16384 57.9 / 59.1.
constexpr int64_t kValuesBesideFrom = 4096, kValuesBesideTo = 24576;
bool values_beside(const Dims& d, int64_t D, at::ScalarType dt, bool two, bool transformed) {
  const int64_t blocks = d.B * d.H * d.nq1;
  return two && !transformed && dt == at::kBFloat16 && D == 64 && d.bs == 16 && blocks >= kValuesBesideFrom && blocks <= kValuesBesideTo &&
         !g_has_hook.load(std::memory_order_relaxed);      // a stage hook's stages do not overlap
}

// One side stream per device: the index transpose is needed only by the last stage of the backward and leaves most SMs idle.  Of high priority: its
// CTAs take the place of the first ones of the dQ stage that end, not of the last.
at::cuda::CUDAStream side_stream(c10::DeviceIndex dev) {
  static std::mutex mu;
  static std::array<std::optional<at::cuda::CUDAStream>, C10_COMPILE_TIME_MAX_GPUS> streams;
  std::lock_guard<std::mutex> lock(mu);
  auto& s = streams[dev];
  if (!s) s = at::cuda::getStreamFromPool(true, dev);
  return *s;
}

// Work on the side stream between two points of the current one.  The second point is there whatever happens in between: a call that
// fails half way gives its scratch back to the allocator of the current stream, which may hand it out while the side stream still writes,
// and a capture cannot end with an open fork.
struct Fork {
  const at::cuda::CUDAStream cur, side;
  at::cuda::CUDAEvent done;
  bool recorded = false, open = true;
  Fork(const at::cuda::CUDAStream& c, const at::cuda::CUDAStream& s) : cur(c), side(s) {
    at::cuda::CUDAEvent start;
    start.record(cur);
    start.block(side);
  }
  void record() {
    done.record(side);
    recorded = true;
  }
  void join() {
    open = false;
    if (!recorded) record();
    done.block(cur);
  }
  ~Fork() {
    if (!open) return;
    try {
      join();
    } catch (...) {      // an error of the call itself is on its way out
    }
  }
};

// dq, dk, dv are written, and dpk, dpv(, dpk2, dpv2) in fp32 at acc (nullptr: in the call's scratch).
void run_bwd(Core& c, const Dims& d, const LlsaTensor& d_o, const LlsaTensor& dq, const LlsaTensor& dk, const LlsaTensor& dv, int topk,
             int topk_p, double w1, double w2, double kvw1, double kvw2, bool fold, bool bf16, float* const* acc, const Tensor& like) {
  const int64_t BH = d.B * d.H, E = d.nq1 * topk, D = d.B * d.H ? c.q.shape[3] : 0;
  const bool tensor_core = bf16 && !flag(kForceGeneric);
  const int S = llsa_transpose_range_entries(d.B, d.H, d.nq1, topk);
  const int64_t R = (E + S - 1) / S;
  const int64_t n_partial = tensor_core ? llsa_attn_bwd_partial_elems(d.B, d.H, d.Nq, topk) : 0;
  const int64_t acc1 = BH * d.n1 * D, acc2 = c.two ? BH * d.n2 * D : 0;
  LlsaAttnArgs a = c.args(topk, topk_p, d.bs, w1, w2);
  const int64_t n_rem = llsa_attn_remainder_elems(&a, 1);
  Carver cv;
  const int64_t o_off = cv.take(BH * (d.n1 + 1) * 4), o_flat = cv.take(BH * E * 4), o_ranges = cv.take(BH * R * 8), o_delta = cv.take(BH * d.Nq * 4),
                o_acc = cv.take(acc ? 0 : (2 * acc1 + 2 * acc2) * 4), o_partial = cv.take(n_partial * 4), o_rem = cv.take(n_rem * 2);
  const Tensor ws = byte_buffer(cv.off, like);
  char* p = (char*) ws.data_ptr();
  float* const scratch = (float*) (p + o_acc);
  float* const inside[4] = {scratch, scratch + acc1, scratch + 2 * acc1, scratch + 2 * acc1 + acc2};
  float* const* const at = acc ? acc : inside;
  const LlsaTensor offsets = packed(p + o_off, LLSA_I32, {d.B, d.H, d.n1 + 1}), flat = packed(p + o_flat, LLSA_I32, {d.B, d.H, E}),
                   ranges = packed(p + o_ranges, LLSA_I32, {d.B, d.H, R, 2}),
                   delta = packed(p + o_delta, LLSA_F32, {d.B, d.H, d.Nq}), dpk = packed(at[0], LLSA_F32, {d.B, d.H, d.n1, D}),
                   dpv = packed(at[1], LLSA_F32, {d.B, d.H, d.n1, D}), dpk2 = packed(at[2], LLSA_F32, {d.B, d.H, d.n2, D}),
                   dpv2 = packed(at[3], LLSA_F32, {d.B, d.H, d.n2, D}),
                   partial = packed(p + o_partial, LLSA_F32, {d.B, d.H, BH ? n_partial / (BH * 4096) : 0, 4096}),
                   rem = packed(p + o_rem, LLSA_BF16, {d.B, d.H, d.Nq, D});
  const Status t_status(like), status(like);

  const at::cuda::CUDAStream cur = at::cuda::getCurrentCUDAStream(like.device().index());
  const bool hooked = g_has_hook.load(std::memory_order_relaxed);      // a stage hook times every stage on ONE stream
  // Up to some thousand query blocks the host is the pace of an eager call: two events, four stream operations and a second launch call are
  // worth more there than the 5 us of the transpose.  Forward + backward, us a pass with the side stream / on one stream: one level, N = 1024,
  // 128 query blocks fp32 108 / 97, bf16 117 / 108, 1,024 blocks 118 / 108; two levels, 512 blocks (N = 4096) 119 / 113, 1,024 blocks
  // (N = 16384) 114 / 111; from 2,048 blocks on the GPU is the pace and the two are equal (119 / 119 at one level, 150 / 150 at 4,096 blocks of
  // two).  In a graph the host's time does not count.
  auto capturing = [&] {
    cudaStreamCaptureStatus s = cudaStreamCaptureStatusNone;
    C10_CUDA_CHECK(cudaStreamIsCapturing(cur, &s));
    return s != cudaStreamCaptureStatusNone;
  };
  const bool overlap = !hooked && !flag(kNoOverlap) && (BH * d.nq1 > 1024 || capturing());
  auto transpose = [&](cudaStream_t st) {
    mark("transpose_indices");
    ok(llsa_transpose_indices_pairs(&c.indices, &offsets, &flat, nullptr, tensor_core ? &ranges : nullptr, d.n1, nullptr, 0, t_status.ptr(), st),
       "transpose_indices");
  };
  a.d_o = &d_o; a.dq = &dq; a.dk = &dk; a.dv = &dv;
  a.offsets = &offsets; a.flat = &flat; a.delta = &delta;
  a.dpk_acc = &dpk; a.dpv_acc = &dpv;
  if (c.two) { a.dpk2_acc = &dpk2; a.dpv2_acc = &dpv2; }
  if (tensor_core) { a.dkv_partial = &partial; a.flat_ranges = &ranges; }
  if (n_rem) a.remainder = &rem;
  a.fold_pool_bwd = fold;
  a.kv_weight = (float) kvw1; a.kv_weight_2 = (float) kvw2;
  a.status = status.ptr();
  if (overlap) {
    // the scratch belongs to the current stream; the side stream works between the two events
    const at::cuda::CUDAStream side = side_stream(like.device().index());
    Fork fork(cur, side);
    // The lists are transposed next to the dQ stage, which does not need them.  The transpose is first in line: its CTAs find no room once those of
    // the dQ stage have filled the SMs.  The scalar dQ stage has the accumulators cleared here too.
    transpose(side);
    if (!tensor_core && !acc) {
      if (acc1) C10_CUDA_CHECK(cudaMemsetAsync(scratch, 0, (2 * acc1 + 2 * acc2) * 4, side));
    } else if (!tensor_core) {
      for (int i = 0; i < (c.two ? 4 : 2); ++i) C10_CUDA_CHECK(cudaMemsetAsync(acc[i], 0, (i < 2 ? acc1 : acc2) * 4, side));
    }
    fork.record();
    a.stage_mask = tensor_core ? 1 : 1 | 8;
    ok(llsa_attn_bwd(&a, cur), "attn_bwd");
    fork.join();
    a.stage_mask = 2 | 4;
    ok(llsa_attn_bwd(&a, cur), "attn_bwd");
  } else {
    transpose(cur);
    static const char* const names[3] = {"attn_bwd_dq", "attn_bwd_dkv_pooled", "attn_bwd_dkv_fine"};
    if (!hooked) ok(llsa_attn_bwd(&a, cur), "attn_bwd");
    else
      for (int i = 0; i < 3; ++i) {
        mark(names[i]);
        a.stage_mask = 1 << i;
        ok(llsa_attn_bwd(&a, cur), names[i]);
      }
    mark("end");
  }
  t_status.check("transpose_indices");
  status.check("attn_bwd");
}

Core make_core(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& pk, const Tensor& pv, const OptTensor& pk2, const OptTensor& pv2,
               const Tensor& indices, const OptTensor& p_indices, const Tensor& o, const Tensor& lse) {
  Core c;
  c.q = desc(q); c.k = desc(k); c.v = desc(v); c.pk = desc(pk); c.pv = desc(pv);
  c.two = pk2.has_value();
  if (c.two) { c.pk2 = desc(*pk2); c.pv2 = desc(*pv2); c.p_indices = desc(*p_indices); }
  c.indices = desc(indices); c.o = desc(o); c.lse = desc(lse);
  return c;
}

std::vector<Tensor> attn_fwd(const Tensor& q_, const Tensor& k_, const Tensor& v_, const Tensor& pk, const Tensor& pv, const OptTensor& pk2,
                             const OptTensor& pv2, const Tensor& indices, const OptTensor& p_indices, int64_t topk, int64_t topk_p,
                             int64_t block_size, double w1, double w2) {
  need_cuda({q_, k_, v_, pk, pv, or_none(pk2), or_none(pv2), indices, or_none(p_indices)});
  check_float({&q_, &k_, &v_, &pk, &pv});
  const c10::cuda::CUDAGuard guard(q_.device());
  const Tensor q = prep(q_), k = prep(k_), v = prep(v_), pkc = cont(pk), pvc = cont(pv), ic = cont(indices);
  OptTensor pk2c, pv2c, pic;
  if (pk2) {
    TORCH_CHECK(pv2 && p_indices, "llsa_b200: pv2 / p_indices missing for the two-level form");
    pk2c = cont(*pk2); pv2c = cont(*pv2); pic = cont(*p_indices);
  }
  const Dims d(q, k, block_size);
  Tensor o = at::empty_like(q), lse = at::empty({d.B, d.H, d.Nq}, q.options().dtype(at::kFloat));
  const Status status(q);
  const Core c = make_core(q, k, v, pkc, pvc, pk2c, pv2c, ic, pic, o, lse);
  run_fwd(c, (int) topk, (int) topk_p, (int) block_size, w1, w2, q, status, at::cuda::getCurrentCUDAStream(q.device().index()));
  return {o, lse};
}

std::vector<Tensor> attn_bwd(const Tensor& d_o_, const Tensor& q_, const Tensor& k_, const Tensor& v_, const Tensor& pk, const Tensor& pv,
                             const OptTensor& pk2, const OptTensor& pv2, const Tensor& o_, const Tensor& lse, const Tensor& indices,
                             const OptTensor& p_indices, int64_t topk, int64_t topk_p, int64_t block_size, double w1, double w2, double kvw1,
                             double kvw2, bool fold) {
  need_cuda({d_o_, q_, k_, v_, pk, pv, or_none(pk2), or_none(pv2), o_, lse, indices, or_none(p_indices)});
  const c10::cuda::CUDAGuard guard(q_.device());
  const Tensor d_o = prep(d_o_), q = prep(q_), k = prep(k_), v = prep(v_), o = prep(o_), pkc = cont(pk), pvc = cont(pv), ic = cont(indices),
               lc = cont(lse);
  OptTensor pk2c, pv2c, pic;
  if (pk2) {
    TORCH_CHECK(pv2 && p_indices, "llsa_b200: pv2 / p_indices missing for the two-level form");
    pk2c = cont(*pk2); pv2c = cont(*pv2); pic = cont(*p_indices);
  }
  TORCH_CHECK(ic.dim() == 4 && ic.size(3) == topk, "llsa_b200: indices must be [B,H,N/block,topk=", topk, "], got ", ic.sizes());
  const Dims d(q, k, block_size);
  // tensors of their own, not views of one: outputs of an operator must not share memory
  std::vector<Tensor> out = {at::empty_like(q), at::empty_like(k), at::empty_like(v)};
  float* acc[4] = {nullptr, nullptr, nullptr, nullptr};
  for (int i = 0; i < (pk2 ? 4 : 2); ++i) {
    out.push_back(at::empty({d.B, d.H, i < 2 ? d.n1 : d.n2, q.size(3)}, q.options().dtype(at::kFloat)));
    acc[i] = (float*) out.back().data_ptr();
  }
  Core c = make_core(q, k, v, pkc, pvc, pk2c, pv2c, ic, pic, o, lc);
  run_bwd(c, d, desc(d_o), desc(out[0]), desc(out[1]), desc(out[2]), (int) topk, (int) topk_p, w1, w2, kvw1, kvw2, fold,
          q.scalar_type() == at::kBFloat16, acc, q);
  return out;
}

// ------------------------------------------------------------------ the fused layer
std::vector<Tensor> layer_fwd(const Tensor& q_, const Tensor& k_, const Tensor& v_, const OptTensor& freq_, const OptTensor& wq, const OptTensor& wk,
                              double eps, int64_t topk1_, int64_t topk2_, int64_t block_size, int64_t levels) {
  need_cuda({q_, k_, v_, or_none(freq_), or_none(wq), or_none(wk)});
  check_float({&q_, &k_, &v_});
  const c10::cuda::CUDAGuard guard(q_.device());
  const cudaStream_t st = at::cuda::getCurrentCUDAStream(q_.device().index());
  Tensor q = prep(q_), k = prep(k_), v = prep(v_);
  const Dims d(q, k, block_size);
  TORCH_CHECK(k.sizes() == v.sizes() && k.sizes() == q.sizes(), "llsa_b200: q, k, v must have the same shape");
  const at::ScalarType dt = q.scalar_type();
  const bool two = levels == 2, norm = wq.has_value() || wk.has_value();
  const int64_t D = q.size(3), es = q.element_size(), BH = d.B * d.H;
  const int code = dtype_code(dt);
  const int topk1 = (int) (two ? topk1_ : std::min<int64_t>(topk1_, d.n1)), topk2 = two ? (int) std::min<int64_t>(topk2_, d.n2) : 0;
  const Saved sv(d, D, es, topk1, topk2, (int) levels);
  const Tensor saved = byte_buffer(sv.bytes, q);
  char* sp = (char*) saved.data_ptr();
  Carver cv;      // what only this call needs: the pooled queries
  const int64_t o_pq = cv.take(BH * d.nq1 * D * es), o_pq2 = cv.take(two ? BH * d.nq2 * D * es : 0);
  const Tensor tmp = byte_buffer(cv.off, q);
  char* tp = (char*) tmp.data_ptr();
  const LlsaTensor y1[3] = {packed(tp + o_pq, code, {d.B, d.H, d.nq1, D}), packed(sp + sv.pk, code, {d.B, d.H, d.n1, D}),
                            packed(sp + sv.pv, code, {d.B, d.H, d.n1, D})};
  const LlsaTensor y2[3] = {packed(tp + o_pq2, code, {d.B, d.H, d.nq2, D}), packed(sp + sv.pk2, code, {d.B, d.H, d.n2, D}),
                            packed(sp + sv.pv2, code, {d.B, d.H, d.n2, D})};

  // ---- preparation of q and k, pooling
  std::vector<Tensor> out(2);
  Tensor freq;
  if (freq_) {
    freq = *freq_;
    if (norm && freq.scalar_type() != dt) freq = freq.to(dt);
    else if (freq.scalar_type() == at::kDouble || (dt == at::kFloat && freq.scalar_type() == at::kBFloat16)) freq = freq.to(at::kFloat);
    if (!table_ok(freq)) freq = freq.contiguous();
  }
  const bool v_beside = values_beside(d, D, dt, two, freq.defined() || norm);
  mark("pool_pyramid");
  if (!freq.defined() && !norm) {
    const LlsaTensor x[3] = {desc(q), desc(k), desc(v)};
    ok(llsa_pool_pyramid_fwd(v_beside ? 2 : 3, x, y1, two ? y2 : nullptr, (int) block_size, st), "pool_pyramid_fwd");
  } else {
    LlsaTensor x[3] = {desc(q), desc(k), desc(v)}, xr[3], f;
    // without a table a tensor that has no norm passes unchanged: a copy, since an output of the operator must not be its input
    Tensor qr = freq.defined() || wq ? at::empty_like(q) : q.clone(), kr = freq.defined() || wk ? at::empty_like(k) : k.clone();
    xr[0] = desc(qr); xr[1] = desc(kr); xr[2] = x[2];
    if (freq.defined()) f = desc(freq);
    if (freq.defined() && freq.scalar_type() != dt) {      // a table wider than the data: rotate first, then pool
      ok(llsa_rope_fwd(&x[0], &f, &xr[0], st), "rope");
      ok(llsa_rope_fwd(&x[1], &f, &xr[1], st), "rope");
      ok(llsa_pool_pyramid_fwd(3, xr, y1, two ? y2 : nullptr, (int) block_size, st), "pool_pyramid_fwd");
    } else if (!norm) {
      ok(llsa_rope_pool_pyramid_fwd(3, x, &f, 3, xr, y1, two ? y2 : nullptr, (int) block_size, st), "rope_pool_pyramid_fwd");
    } else {
      const Tensor w[2] = {wq ? cont(wq->to(at::kFloat)) : Tensor(), wk ? cont(wk->to(at::kFloat)) : Tensor()};
      LlsaTensor wd[2];
      const LlsaTensor* wp[3] = {nullptr, nullptr, nullptr};
      int mask = 0;
      for (int i = 0; i < 2; ++i)
        if (w[i].defined()) { wd[i] = desc(w[i]); wp[i] = &wd[i]; mask |= 1 << i; }
      ok(llsa_rms_rope_pool_pyramid_fwd(3, x, wp, mask, (float) eps, freq.defined() ? &f : nullptr, freq.defined() ? 3 : 0, xr, y1,
                                        two ? y2 : nullptr, (int) block_size, st),
         "rms_rope_pool_pyramid_fwd");
    }
    q = qr; k = kr;
    out.push_back(qr);
    out.push_back(kr);
  }
  // ---- selection
  Core c;
  c.two = two;
  c.q = desc(q); c.k = desc(k); c.v = desc(v);
  c.pk = y1[1]; c.pv = y1[2];
  c.indices = packed(sp + sv.indices, LLSA_I32, {d.B, d.H, d.nq1, topk1});
  c.lse = packed(sp + sv.lse, LLSA_F32, {d.B, d.H, d.Nq});
  if (two) {
    c.pk2 = y2[1]; c.pv2 = y2[2];
    c.p_indices = packed(sp + sv.p_indices, LLSA_I32, {d.B, d.H, d.nq2, topk2});
    mark("select_two_level");
    ok(llsa_select_two_level(&y1[0], &y1[1], &y2[0], &y2[1], &c.p_indices, &c.indices, topk1, topk2, (int) block_size, st), "select_two_level");
  } else {
    mark("coarse_topk");
    ok(llsa_coarse_topk(&y1[0], &y1[1], &c.indices, topk1, st), "coarse_topk");
  }
  if (v_beside) ok(llsa_pool_pyramid_beside_fwd(1, &c.v, &y1[2], two ? &y2[2] : nullptr, (int) block_size, st), "pool_pyramid_beside_fwd");
  // ---- attention
  Tensor o = at::empty_like(q);
  c.o = desc(o);
  const Status status(q);
  run_fwd(c, topk1, topk2, (int) block_size, (double) block_size, two ? (double) (block_size * block_size) : 1.0, q, status, st);
  out[0] = o;
  out[1] = saved;
  return out;
}

// q, k: what the attention kernels saw (after preparation); xq, xk: what went into the norm (given with wq / wk)
std::vector<Tensor> layer_bwd(const Tensor& d_o_, const Tensor& q_, const Tensor& k_, const Tensor& v_, const Tensor& o_, const Tensor& saved,
                              const OptTensor& freq_, const OptTensor& xq, const OptTensor& xk, const OptTensor& wq, const OptTensor& wk, double eps,
                              int64_t topk1_, int64_t topk2_, int64_t block_size, int64_t levels, bool want_dw) {
  need_cuda({d_o_, q_, k_, v_, o_, saved, or_none(freq_), or_none(xq), or_none(xk), or_none(wq), or_none(wk)});
  check_float({&q_, &k_, &v_, &d_o_});
  const c10::cuda::CUDAGuard guard(q_.device());
  const cudaStream_t st = at::cuda::getCurrentCUDAStream(q_.device().index());
  const Tensor d_o = prep(d_o_), q = prep(q_), k = prep(k_), v = prep(v_), o = prep(o_);
  const Dims d(q, k, block_size);
  const at::ScalarType dt = q.scalar_type();
  const bool two = levels == 2, norm = wq.has_value() || wk.has_value();
  const int64_t D = q.size(3);
  const int code = dtype_code(dt);
  const int topk1 = (int) (two ? topk1_ : std::min<int64_t>(topk1_, d.n1)), topk2 = two ? (int) std::min<int64_t>(topk2_, d.n2) : 0;
  const Saved sv(d, D, q.element_size(), topk1, topk2, (int) levels);
  TORCH_CHECK(saved.numel() == sv.bytes && saved.is_contiguous(), "llsa_b200.layer_bwd: `saved` is not from the matching layer_fwd");
  char* sp = (char*) saved.data_ptr();
  Core c;
  c.two = two;
  c.q = desc(q); c.k = desc(k); c.v = desc(v); c.o = desc(o);
  c.pk = packed(sp + sv.pk, code, {d.B, d.H, d.n1, D});
  c.pv = packed(sp + sv.pv, code, {d.B, d.H, d.n1, D});
  c.indices = packed(sp + sv.indices, LLSA_I32, {d.B, d.H, d.nq1, topk1});
  c.lse = packed(sp + sv.lse, LLSA_F32, {d.B, d.H, d.Nq});
  if (two) {
    c.pk2 = packed(sp + sv.pk2, code, {d.B, d.H, d.n2, D});
    c.pv2 = packed(sp + sv.pv2, code, {d.B, d.H, d.n2, D});
    c.p_indices = packed(sp + sv.p_indices, LLSA_I32, {d.B, d.H, d.nq2, topk2});
  }
  const double w1 = (double) block_size, w2 = two ? w1 * w1 : 1.0;
  const double kvw1 = two || flag(kExactGrad) ? w1 : 1.0;      // the reference's one-level backward drops the weight (sparse_attention_res_1.py:389)
  Tensor dq = at::empty_like(q), dk = at::empty_like(k), dv = at::empty_like(v);
  run_bwd(c, d, desc(d_o), desc(dq), desc(dk), desc(dv), topk1, topk2, w1, w2, kvw1, w2, true, dt == at::kBFloat16, nullptr, q);
  std::vector<Tensor> out = {dq, dk, dv};
  if (freq_ || norm) {
    Tensor freq;
    LlsaTensor f;
    if (freq_) {
      freq = *freq_;
      // a table wider than the data stays: the backward has always rotated with the table as it was given
      if (freq.scalar_type() != dt && freq.scalar_type() != at::kFloat) freq = freq.to(at::kFloat);
      if (!table_ok(freq)) freq = freq.contiguous();
      f = desc(freq);
    }
    const LlsaTensor dy[2] = {desc(dq), desc(dk)};
    LlsaTensor x[2], wd[2], dwd[2], part;
    Tensor xs[2], w[2], dw[2], partial;
    const LlsaTensor *wp[2] = {nullptr, nullptr}, *dwp[2] = {nullptr, nullptr};
    int mask = 0;
    if (norm) {
      const OptTensor *ws[2] = {&wq, &wk}, *xo[2] = {&xq, &xk};
      for (int i = 0; i < 2; ++i) {
        x[i] = dy[i];
        if (!ws[i]->has_value()) continue;
        TORCH_CHECK(xo[i]->has_value(), "llsa_b200.layer_bwd: the input of the norm is missing");
        xs[i] = prep(**xo[i]);
        x[i] = desc(xs[i]);
        w[i] = cont((*ws[i])->to(at::kFloat));
        wd[i] = desc(w[i]);
        wp[i] = &wd[i];
        mask |= 1 << i;
      }
      if (want_dw) {
        partial = at::empty({llsa_rms_rope_bwd_partial_elems(2)}, q.options().dtype(at::kFloat));
        part = desc(partial);
        for (int i = 0; i < 2; ++i)
          if (wp[i]) {
            dw[i] = at::empty({D}, q.options().dtype(at::kFloat));
            dwd[i] = desc(dw[i]);
            dwp[i] = &dwd[i];
          }
      }
    }
    ok(llsa_rms_rope_bwd(2, dy, norm ? x : nullptr, wp, mask, (float) eps, freq.defined() ? &f : nullptr, dy, partial.defined() ? &part : nullptr,
                         dwp, st),
       "rms_rope_bwd");
    for (int i = 0; i < 2; ++i)
      if (dw[i].defined()) out.push_back(dw[i].to((i ? wk : wq)->scalar_type()));
  }
  return out;
}

// ------------------------------------------------------------------ autograd
using FwdSig = std::vector<Tensor>(const Tensor&, const Tensor&, const Tensor&, const OptTensor&, const OptTensor&, const OptTensor&, double,
                                   int64_t, int64_t, int64_t, int64_t);
using BwdSig = std::vector<Tensor>(const Tensor&, const Tensor&, const Tensor&, const Tensor&, const Tensor&, const Tensor&, const OptTensor&,
                                   const OptTensor&, const OptTensor&, const OptTensor&, const OptTensor&, double, int64_t, int64_t, int64_t,
                                   int64_t, bool);

const c10::TypedOperatorHandle<FwdSig>& fwd_op() {
  static const auto op = c10::Dispatcher::singleton().findSchemaOrThrow("llsa_b200::layer_fwd", "").typed<FwdSig>();
  return op;
}
const c10::TypedOperatorHandle<BwdSig>& bwd_op() {
  static const auto op = c10::Dispatcher::singleton().findSchemaOrThrow("llsa_b200::layer_bwd", "").typed<BwdSig>();
  return op;
}

OptTensor opt(const Tensor& t) { return t.defined() ? OptTensor(t) : std::nullopt; }

struct LayerFunction : torch::autograd::Function<LayerFunction> {
  static variable_list forward(torch::autograd::AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, const OptTensor& freq,
                               const OptTensor& wq, const OptTensor& wk, double eps, int64_t topk1, int64_t topk2, int64_t block_size,
                               int64_t levels) {
    variable_list out;
    {
      at::AutoDispatchBelowADInplaceOrView below;
      out = fwd_op().call(q, k, v, freq, wq, wk, eps, topk1, topk2, block_size, levels);
    }
    const bool front = out.size() == 4, norm = wq.has_value() || wk.has_value();
    ctx->set_materialize_grads(false);      // only o carries a gradient
    if (front) ctx->mark_non_differentiable({out[1], out[2], out[3]});
    else ctx->mark_non_differentiable({out[1]});
    const Tensor none;
    ctx->save_for_backward({front ? out[2] : q, front ? out[3] : k, v, out[0], out[1], freq.value_or(none), norm ? q : none, norm ? k : none,
                            wq.value_or(none), wk.value_or(none)});
    auto& s = ctx->saved_data;
    s["eps"] = eps;
    s["cfg"] = std::vector<int64_t>{topk1, topk2, block_size, levels};
    return out;
  }

  static variable_list backward(torch::autograd::AutogradContext* ctx, variable_list grads) {
    variable_list g(11);
    if (!grads[0].defined()) return g;
    const variable_list s = ctx->get_saved_variables();
    const std::vector<int64_t> cfg = ctx->saved_data["cfg"].toIntVector();
    const double eps = ctx->saved_data["eps"].toDouble();
    // needs_input_grad counts the tensors that were given: an absent table or weight has no edge
    size_t edge = 3 + (s[5].defined() ? 1 : 0);
    const bool want_wq = s[8].defined() && ctx->needs_input_grad(edge++), want_wk = s[9].defined() && ctx->needs_input_grad(edge);
    const bool want_dw = want_wq || want_wk;
    std::vector<Tensor> r;
    auto call = [&] {
      r = bwd_op().call(grads[0], s[0], s[1], s[2], s[3], s[4], opt(s[5]), opt(s[6]), opt(s[7]), opt(s[8]), opt(s[9]), eps, cfg[0], cfg[1], cfg[2],
                        cfg[3], want_dw);
    };
    if (at::GradMode::is_enabled()) {
      call();      // create_graph: the operator's own node raises if it is differentiated again
    } else {
      at::AutoDispatchBelowADInplaceOrView below;
      call();
    }
    g[0] = r[0]; g[1] = r[1]; g[2] = r[2];
    size_t at = 3;
    if (want_dw) {
      if (s[8].defined()) g[4] = r[at++];
      if (s[9].defined()) g[5] = r[at++];
    }
    return g;
  }
};

std::vector<Tensor> layer_fwd_autograd(const Tensor& q, const Tensor& k, const Tensor& v, const OptTensor& freq, const OptTensor& wq,
                                       const OptTensor& wk, double eps, int64_t topk1, int64_t topk2, int64_t block_size, int64_t levels) {
  auto wants = [](const Tensor& t) { return t.requires_grad(); };
  if (wq || wk)      // the tangent would be dropped without a word
    for (const Tensor& t : {q, k, v, or_none(wq), or_none(wk)})
      TORCH_CHECK_NOT_IMPLEMENTED(!t.defined() || !t._fw_grad(0).defined(), "llsa_b200: no forward-mode derivative of the layer with norms in front");
  if (at::GradMode::is_enabled() && (wants(q) || wants(k) || wants(v) || (wq && wants(*wq)) || (wk && wants(*wk))))
    return LayerFunction::apply(q, k, v, freq, wq, wk, eps, topk1, topk2, block_size, levels);
  at::AutoDispatchBelowADInplaceOrView below;
  return fwd_op().call(q, k, v, freq, wq, wk, eps, topk1, topk2, block_size, levels);
}

}  // namespace

TORCH_LIBRARY_FRAGMENT(llsa_b200, m) {
  m.def("layer_fwd(Tensor q, Tensor k, Tensor v, Tensor? freq, Tensor? wq, Tensor? wk, float eps, int topk1, int topk2, int block_size, "
        "int levels) -> Tensor[]");
  m.def("layer_bwd(Tensor d_o, Tensor q, Tensor k, Tensor v, Tensor o, Tensor saved, Tensor? freq, Tensor? xq, Tensor? xk, Tensor? wq, "
        "Tensor? wk, float eps, int topk1, int topk2, int block_size, int levels, bool want_dw) -> Tensor[]");
  m.def("last_fwd_redo() -> Tensor");
  m.def("attn_fwd(Tensor q, Tensor k, Tensor v, Tensor pk, Tensor pv, Tensor? pk2, Tensor? pv2, Tensor indices, Tensor? p_indices, int topk, "
        "int topk_p, int block_size, float w1, float w2) -> Tensor[]");
  m.def("attn_bwd(Tensor d_o, Tensor q, Tensor k, Tensor v, Tensor pk, Tensor pv, Tensor? pk2, Tensor? pv2, Tensor o, Tensor lse, "
        "Tensor indices, Tensor? p_indices, int topk, int topk_p, int block_size, float w1, float w2, float kvw1, float kvw2, bool fold) "
        "-> Tensor[]");
}
TORCH_LIBRARY_IMPL(llsa_b200, CompositeExplicitAutograd, m) {
  m.impl("last_fwd_redo", [] {
    std::lock_guard<std::mutex> lock(g_redo_mutex);
    return last_redo();
  });
}
TORCH_LIBRARY_IMPL(llsa_b200, CUDA, m) {
  m.impl("layer_fwd", layer_fwd);
  m.impl("layer_bwd", layer_bwd);
  m.impl("attn_fwd", attn_fwd);
  m.impl("attn_bwd", attn_bwd);
}
TORCH_LIBRARY_IMPL(llsa_b200, CPU, m) {      // refuse with the library's own words
  m.impl("layer_fwd", layer_fwd);
  m.impl("layer_bwd", layer_bwd);
  m.impl("attn_fwd", attn_fwd);
  m.impl("attn_bwd", attn_bwd);
}
TORCH_LIBRARY_IMPL(llsa_b200, Autograd, m) {
  m.impl("layer_fwd", layer_fwd_autograd);
  m.impl("layer_bwd", torch::autograd::autogradNotImplementedFallback());
  m.impl("attn_fwd", torch::autograd::autogradNotImplementedFallback());
  m.impl("attn_bwd", torch::autograd::autogradNotImplementedFallback());
}

PYBIND11_MODULE(_host, m) {
  m.def("configure", [](int flags, int wait_limit) {
    g_flags.store(flags);
    g_wait_limit.store(wait_limit);
  });
  m.def("keep_marks", [](bool keep) { t_keep_marks = keep; });      // of this thread's forwards
  m.def("set_stage_hook", [](pybind11::object fn) {
    PyObject* old = g_hook;
    g_hook = fn.is_none() ? nullptr : fn.inc_ref().ptr();
    g_has_hook.store(g_hook != nullptr);
    Py_XDECREF(old);
  });
}
