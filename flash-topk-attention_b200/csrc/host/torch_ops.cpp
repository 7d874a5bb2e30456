// Native host layer between the Python operators and the C ABI: allocation of
// outputs and scratch, views of the inputs, launches, and the autograd node of
// the attention.
//
// What it is for: at short sequences the path is bound by host time.  One
// training pass (score, select, merge, attention, backward) at N = 256, H = 2
// spent 490 us in Python: ctypes conversions, one torch call per buffer, a
// pinned copy and an event per operator for the status word, and a Python
// autograd function whose backward needs the interpreter lock, around 91 us of
// kernels.  Nothing here waits for the device or keeps state between calls but
// the status words.
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/CUDAEvent.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/extension.h>

#include <atomic>
#include <cmath>
#include <mutex>
#include <string>
#include <tuple>
#include <vector>

#include "../../../include/ftk_api.h"

namespace {

using at::Tensor;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;

struct Unsupported : std::runtime_error {
  using std::runtime_error::runtime_error;
};

// C-ABI return code -> the exception the reference raises for that class of problem
void check(int code, const char* what) {
  if (code == 0) return;
  const std::string msg =
      std::string(what) + ": " + ftk_error_string(code) + " (code " + std::to_string(code) + ")";
  if (code == -2) throw Unsupported(msg);
  if (code == -1) throw py::value_error(msg);
  throw std::runtime_error(msg);
}

// ------------------------------------------------------------- status words
// One sticky word per device in pinned host memory that every launch may write
// (the device reaches it through unified addressing, and only ever writes it on
// a failure).  The host reads it directly: no copy, event or synchronisation.
constexpr int MAX_DEVICES = 64;
std::mutex g_status_mutex;
Tensor g_status[MAX_DEVICES];
std::atomic<int*> g_status_ptr[MAX_DEVICES];
std::atomic<bool> g_deferred{true}, g_debug{false};

int* status_ptr(int dev) {
  TORCH_CHECK(dev >= 0 && dev < MAX_DEVICES, "device index out of range");
  int* p = g_status_ptr[dev].load(std::memory_order_acquire);
  if (p) return p;
  std::lock_guard<std::mutex> lock(g_status_mutex);
  p = g_status_ptr[dev].load(std::memory_order_relaxed);
  if (!p) {
    g_status[dev] =
        at::zeros({1}, at::TensorOptions().dtype(at::kInt).device(at::kCPU).pinned_memory(true));
    p = g_status[dev].data_ptr<int>();
    g_status_ptr[dev].store(p, std::memory_order_release);
  }
  return p;
}

Tensor status_word(int dev) {
  status_ptr(dev);
  return g_status[dev];
}

// code of a failure reported since the last look (and forget it), 0 if none
int take_status(int dev) {
  volatile int* p = status_ptr(dev);
  const int code = *p;
  if (code != 0) *p = 0;
  return code;
}

// raises what an earlier launch reported
void look(int dev) {
  if (!g_deferred.load(std::memory_order_relaxed)) return;
  if (const int code = take_status(dev))
    throw std::runtime_error(std::string("flash_topk_attn_v2 device error in an earlier call: ") +
                             ftk_error_string(code) + " (status " + std::to_string(code) + ")");
}

// ------------------------------------------------------------------- timing
std::atomic<bool> g_timing{false};
std::mutex g_timing_mutex;
struct Timed {
  std::string name;
  at::cuda::CUDAEvent begin{cudaEventDefault}, end{cudaEventDefault};
};
std::vector<std::unique_ptr<Timed>> g_timed;

// brackets a C-ABI call with events on its stream when timing is switched on
class TimedCall {
 public:
  TimedCall(const char* name, const c10::cuda::CUDAStream& st) : st_(st) {
    if (!g_timing.load(std::memory_order_relaxed)) return;
    t_ = std::make_unique<Timed>();
    t_->name = name;
    t_->begin.record(st_);
  }
  ~TimedCall() {
    if (!t_) return;
    try {
      t_->end.record(st_);
      std::lock_guard<std::mutex> lock(g_timing_mutex);
      g_timed.push_back(std::move(t_));
    } catch (...) {
    }
  }

 private:
  c10::cuda::CUDAStream st_;
  std::unique_ptr<Timed> t_;
};

void set_timing(bool on) {
  std::lock_guard<std::mutex> lock(g_timing_mutex);
  g_timed.clear();
  g_timing = on;
}

std::vector<std::pair<std::string, double>> take_times() {
  std::lock_guard<std::mutex> lock(g_timing_mutex);
  std::vector<std::pair<std::string, double>> out;
  for (auto& t : g_timed) out.emplace_back(t->name, t->begin.elapsed_time(t->end));
  return out;
}

// ------------------------------------------------------------ device memory
// Outputs, straight from the allocator's tensor factory (a dispatched at::empty
// takes about twice as long).
Tensor new_cuda(at::IntArrayRef sizes, at::ScalarType dtype, const at::Device& device) {
  return Tensor(at::detail::empty_cuda(sizes, dtype, device, std::nullopt));
}
// Scratch of one call: memory of the caching allocator without a tensor around it.
// Freed at the end of the scope, for reuse in stream order, like a tensor would be.
struct Scratch {
  at::DataPtr p;
  size_t bytes;
  explicit Scratch(size_t n) : bytes(n) {
    p = c10::cuda::CUDACachingAllocator::get()->allocate(std::max<size_t>(n, 16));
  }
  void* get() const { return p.get(); }
};

// ------------------------------------------------------------------- layouts
// A tensor addressed as [b][n][h][d]: d dense, 16-byte aligned base, strides
// multiples of 8 elements, no dimension repeated (an expanded tensor, such as the
// gradient of a sum over tokens, has stride 0, which a tensor map cannot have).
// Copies only what cannot be addressed in place.
struct View {
  Tensor t;
  int64_t sb = 0, sn = 0, sh = 0;

  static bool strides(const Tensor& x, bool four_d, int64_t D, View* v) {
    if (x.stride(-1) != 1) return false;
    for (int64_t i = 0; i + 1 < x.dim(); i++)
      if (x.size(i) > 1 && x.stride(i) <= 0) return false;
    v->sb = x.stride(0);
    v->sn = four_d ? x.stride(2) : x.stride(1);
    v->sh = four_d ? x.stride(1) : D;
    return (reinterpret_cast<uintptr_t>(x.data_ptr()) & 15) == 0 &&
           ((v->sb | v->sn | v->sh) & 7) == 0;
  }
  View() = default;
  View(const Tensor& x, bool four_d, int64_t D) {
    t = x;
    if (strides(t, four_d, D, this)) return;
    t = x.contiguous();
    if (strides(t, four_d, D, this)) return;
    t = x.clone(at::MemoryFormat::Contiguous);
    if (!strides(t, four_d, D, this))
      throw py::value_error(
          "tensor cannot be aligned to 16 bytes (head dim must be a multiple of 8)");
  }
};

int dtype_code(const Tensor& t) { return t.scalar_type() == at::kHalf ? FTK_F16 : FTK_BF16; }

// bf16 copies of float32 tensors, one launch for all
template <size_t N>
void cast_bf16(Tensor (&x)[N], const c10::cuda::CUDAStream& st) {
  static_assert(N <= 3, "");
  const float* src[3] = {nullptr, nullptr, nullptr};
  int64_t n[3] = {0, 0, 0};
  void* dst[3] = {nullptr, nullptr, nullptr};
  Tensor keep[3];
  for (size_t i = 0; i < N; i++) {
    Tensor s = x[i].contiguous();
    if (reinterpret_cast<uintptr_t>(s.data_ptr()) & 15) s = s.clone();
    keep[i] = s;
    x[i] = at::empty(s.sizes(), s.options().dtype(at::kBFloat16));
    src[i] = s.const_data_ptr<float>();
    n[i] = s.numel();
    dst[i] = x[i].data_ptr();
  }
  check(ftk_cast_bf16(src[0], n[0], dst[0], src[1], n[1], dst[1], src[2], n[2], dst[2], st.stream()),
        "ftk_cast_bf16");
}

// -------------------------------------------------------------- score + select
// Slices b0 .. b0 + count - 1.  `outs` = {idx, raw, avg} of an earlier chunk of
// the same call, or empty: allocated here.  float32 q and k are computed in bf16.
std::vector<Tensor> score_topk(Tensor q, Tensor k, bool four_d, int64_t H, int64_t block,
                               int64_t topk, int64_t pad_head, int64_t pad_tail, double threshold,
                               double scale, int64_t b0, int64_t count, std::vector<Tensor> outs) {
  const at::Device device = q.device();
  c10::cuda::CUDAGuard guard(device);
  look(device.index());
  const auto st = c10::cuda::getCurrentCUDAStream(device.index());
  const int64_t B = q.size(0), N = four_d ? q.size(2) : q.size(1),
                D = four_d ? q.size(3) : q.size(2) / H;
  const int64_t M = (pad_head + N + pad_tail) / block;
  if (q.scalar_type() == at::kFloat) {
    Tensor x[2] = {q, k};
    cast_bf16(x, st);
    q = x[0];
    k = x[1];
  }
  const View vq(q, four_d, D), vk(k, four_d, D);
  if (outs.empty()) {
    const int64_t width = topk > 0 ? std::min(topk, M) : M;
    outs.reserve(3);
    outs.push_back(new_cuda({B, H, N, width}, at::kInt, device));
    outs.push_back(new_cuda({B, H, N, width}, at::kFloat, device));
    outs.push_back(new_cuda({B, H, N, width}, at::kFloat, device));
  }
  const int64_t first = b0 * N * outs[0].size(3);
  const Scratch ws(ftk_score_topk_workspace(count, N, M));
  check(ftk_score_topk(vq.t.data_ptr(), vk.t.data_ptr(), dtype_code(vq.t), B, H, N, D, vq.sb, vq.sn,
                       vq.sh, vk.sb, vk.sn, vk.sh, b0, count, block, pad_head, pad_tail, scale,
                       topk, threshold, outs[0].data_ptr<int>() + first,
                       outs[1].data_ptr<float>() + first, outs[2].data_ptr<float>() + first,
                       ws.get(), ws.bytes, status_ptr(device.index()), st.stream()),
        "ftk_score_topk");
  return outs;
}

// ----------------------------------------------------------------------- merge
std::tuple<Tensor, std::optional<Tensor>, Tensor> qblock_merge(
    const Tensor& topk_idx, const std::optional<Tensor>& topk_scores, int64_t q_block,
    int64_t pad_head, int64_t pad_tail, int64_t blocks, int64_t width, bool want_scores) {
  const at::Device device = topk_idx.device();
  c10::cuda::CUDAGuard guard(device);
  look(device.index());
  const auto st = c10::cuda::getCurrentCUDAStream(device.index());
  const int64_t B = topk_idx.size(0), H = topk_idx.size(1), N = topk_idx.size(2);
  const int64_t QM = (pad_head + N + pad_tail) / q_block;
  auto dense = [](const Tensor& t, at::ScalarType dtype) {
    return t.scalar_type() == dtype && t.is_contiguous() ? t : t.to(dtype).contiguous();
  };
  const Tensor idx = dense(topk_idx, at::kInt);
  Tensor scr;
  if (topk_scores) scr = dense(*topk_scores, at::kFloat);
  Tensor merged = new_cuda({B, H, QM, width}, at::kInt, device);
  Tensor counts = new_cuda({B, H, QM}, at::kInt, device);
  std::optional<Tensor> scores;
  if (want_scores) scores = new_cuda({B, H, QM, width}, at::kFloat, device);
  check(ftk_qblock_merge(idx.data_ptr<int>(), scr.defined() ? scr.data_ptr<float>() : nullptr,
                         B * H, N, topk_idx.size(3), q_block, pad_head, pad_tail, blocks, width,
                         merged.data_ptr<int>(), scores ? scores->data_ptr<float>() : nullptr,
                         counts.data_ptr<int>(), status_ptr(device.index()), st.stream()),
        "ftk_qblock_merge");
  return {merged, scores, counts};
}

// ------------------------------------------------------------------- attention
struct AttnMeta {
  int64_t H, Hkv, q_block, kv_block, q_pad_head, kv_pad_head;
  double scale;
};

ftk_attn describe(const AttnMeta& m, const View& q, const View& k, const View& v,
                  const Tensor& lists, bool out_f32) {
  ftk_attn a{};
  a.q = q.t.data_ptr();
  a.k = k.t.data_ptr();
  a.v = v.t.data_ptr();
  a.dtype = dtype_code(q.t);
  a.out_f32 = out_f32;
  a.B = q.t.size(0);
  a.H = m.H;
  a.Hkv = m.Hkv;
  a.N = q.t.size(1);
  a.D = q.t.size(2) / m.H;
  a.sq_b = q.sb;
  a.sq_n = q.sn;
  a.sq_h = q.sh;
  a.sk_b = k.sb;
  a.sk_n = k.sn;
  a.sk_h = k.sh;
  a.sv_b = v.sb;
  a.sv_n = v.sn;
  a.sv_h = v.sh;
  a.lists = lists.data_ptr<int>();
  a.list_rows = lists.size(2);
  a.W = lists.size(3);
  a.q_block = m.q_block;
  a.kv_block = m.kv_block;
  a.q_pad_head = m.q_pad_head;
  a.kv_pad_head = m.kv_pad_head;
  a.scale = m.scale;
  return a;
}

struct Forward {
  Tensor q, k, v, lists, o, lse;   // q, k, v, lists: what the kernels read
};

Forward attn_forward(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& merged,
                     const AttnMeta& m) {
  const at::Device device = q.device();
  c10::cuda::CUDAGuard guard(device);
  look(device.index());
  const auto st = c10::cuda::getCurrentCUDAStream(device.index());
  const bool f32 = q.scalar_type() == at::kFloat;
  Tensor x[3] = {q, k, v};
  if (f32) cast_bf16(x, st);
  const int64_t D = q.size(2) / m.H;
  const View vq(x[0], false, D), vk(x[1], false, D), vv(x[2], false, D);
  Forward f{vq.t, vk.t, vv.t, merged.contiguous(), Tensor(), Tensor()};
  f.o = new_cuda(q.sizes(), q.scalar_type(), device);
  f.lse = new_cuda({q.size(0), m.H, q.size(1)}, at::kFloat, device);
  const ftk_attn a = describe(m, vq, vk, vv, f.lists, f32);
  const Scratch ws(ftk_attn_fwd_workspace(&a));
  {
    TimedCall timed("ftk_sparse_fwd", st);
    check(ftk_attn_fwd(&a, f.o.data_ptr(), f.o.stride(0), f.o.stride(1), D,
                       f.lse.data_ptr<float>(), ws.get(), ws.bytes, status_ptr(device.index()),
                       st.stream()),
          "ftk_attn_fwd");
  }
  return f;
}

// Backward of the gathered-KV attention (reference: FlashSparseAttnFunc,
// flash_topk_attn_v2/sparse_attn.py:130-224).  A node of its own instead of a
// torch::autograd::Function, whose context and wrapping of outputs cost some 6 us
// per pass.
struct SparseAttnBackward : torch::autograd::Node {
  AttnMeta m{};
  SavedVariable q, k, v, o, lse, lists;

  std::string name() const override { return "SparseAttnBackward"; }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    for (SavedVariable* x : {&q, &k, &v, &o, &lse, &lists}) x->reset_data();
  }

  variable_list apply(variable_list&& grads) override {
    std::lock_guard<std::mutex> lock(mutex_);
    variable_list out(3);
    if (!grads[0].defined()) return out;
    at::AutoDispatchBelowADInplaceOrView below;
    const Tensor tq = q.unpack(), tk = k.unpack(), tv = v.unpack(),
                 to = o.unpack(shared_from_this()), tl = lse.unpack(), tm = lists.unpack();
    const at::Device device = to.device();
    c10::cuda::CUDAGuard guard(device);
    look(device.index());
    const auto st = c10::cuda::getCurrentCUDAStream(device.index());
    const bool f32 = to.scalar_type() == at::kFloat;
    const int64_t D = to.size(2) / m.H;
    const View vq(tq, false, D), vk(tk, false, D), vv(tv, false, D);
    Tensor g[1] = {grads[0]};
    if (f32) cast_bf16(g, st);
    else if (g[0].scalar_type() != tq.scalar_type()) g[0] = g[0].to(tq.scalar_type());
    const View vg(g[0], false, D);
    const ftk_attn a = describe(m, vq, vk, vv, tm, f32);
    const Scratch ws(ftk_attn_bwd_workspace(&a));
    Tensor dq = new_cuda(to.sizes(), to.scalar_type(), device);
    int* status = status_ptr(device.index());
    {
      TimedCall timed("ftk_sparse_bwd_dq", st);
      check(ftk_attn_bwd_dq(&a, to.data_ptr(), to.stride(0), to.stride(1), D, vg.t.data_ptr(), vg.sb,
                            vg.sn, vg.sh, tl.data_ptr<float>(), ws.get(), ws.bytes, dq.data_ptr(),
                            dq.stride(0), dq.stride(1), D, status, st.stream()),
            "ftk_attn_bwd_dq");
    }
    out[0] = dq;
    if (task_should_compute_output(1) || task_should_compute_output(2)) {
      Tensor dk = new_cuda({a.B, a.N, m.Hkv * D}, to.scalar_type(), device);
      Tensor dv = new_cuda({a.B, a.N, m.Hkv * D}, to.scalar_type(), device);
      TimedCall timed("ftk_sparse_bwd_dkv", st);
      check(ftk_attn_bwd_dkv(&a, vg.t.data_ptr(), vg.sb, vg.sn, vg.sh, tl.data_ptr<float>(),
                             ws.get(), ws.bytes, dk.data_ptr(), dk.stride(0), dk.stride(1), D,
                             dv.data_ptr(), dv.stride(0), dv.stride(1), D, status, st.stream()),
            "ftk_attn_bwd_dkv");
      out[1] = dk;
      out[2] = dv;
    }
    if (g_debug.load(std::memory_order_relaxed) &&
        c10::cuda::currentStreamCaptureStatusMayInitCtx() == c10::cuda::CaptureStatus::None) {
      st.synchronize();
      if (const int code = take_status(device.index()))
        throw std::runtime_error(std::string("flash_topk_attn_v2 device error: ") +
                                 ftk_error_string(code) + " (status " + std::to_string(code) + ")");
    }
    return out;
  }
};

std::tuple<Tensor, Tensor> sparse_attn(const Tensor& q, const Tensor& k, const Tensor& v,
                                       const Tensor& merged, int64_t H, int64_t Hkv,
                                       int64_t q_block, int64_t kv_block, int64_t q_pad_head,
                                       int64_t kv_pad_head, double scale) {
  const AttnMeta m{H, Hkv, q_block, kv_block, q_pad_head, kv_pad_head, scale};
  // the outputs would silently carry no tangent
  for (const Tensor* t : {&q, &k, &v})
    if (torch::autograd::isFwGradDefined(*t))
      throw Unsupported("flash_sparse_attn has no forward-mode derivative");
  if (!at::GradMode::is_enabled() || !(q.requires_grad() || k.requires_grad() || v.requires_grad())) {
    const Forward f = attn_forward(q, k, v, merged, m);
    return {f.o, f.lse};
  }
  auto node = std::shared_ptr<SparseAttnBackward>(new SparseAttnBackward(),
                                                  torch::autograd::deleteNode);
  node->set_next_edges(torch::autograd::collect_next_edges(q, k, v));
  Forward f;
  {
    at::AutoDispatchBelowADInplaceOrView below;
    f = attn_forward(q, k, v, merged, m);
  }
  node->m = m;
  node->q = SavedVariable(f.q, false);
  node->k = SavedVariable(f.k, false);
  node->v = SavedVariable(f.v, false);
  node->lse = SavedVariable(f.lse, false);
  node->lists = SavedVariable(f.lists, false);
  torch::autograd::set_history(f.o, node);
  node->o = SavedVariable(f.o, true);
  return {f.o, f.lse};
}

// ----------------------------------------------------------- the ordinary call
// The Python operators check their arguments one by one, as the reference does, to
// raise its exceptions: 5 to 8 us per call.  These entry points take a call that
// passes all of the checks (and needs no special handling) straight through and
// return nothing for any other, which the Python code then deals with.
using Pads = std::pair<int64_t, int64_t>;

bool pads_fit(const Pads& p, int64_t n, int64_t block) {
  return p.first >= 0 && p.second >= 0 && p.first < block && p.second < block &&
         (p.first + n + p.second) % block == 0;
}
bool float_type(const Tensor& t) {
  const auto d = t.scalar_type();
  return d == at::kHalf || d == at::kBFloat16 || d == at::kFloat;
}

std::optional<std::tuple<Tensor, Tensor, Tensor, int64_t>> plain_score(
    const Tensor& q, const Tensor& k, std::optional<int64_t> num_heads, int64_t block, int64_t topk,
    const Pads& pad, double threshold, int64_t scratch) {
  const bool four_d = q.dim() == 4;
  if (!q.is_cuda() || q.device() != k.device() || (!four_d && (q.dim() != 3 || !num_heads)))
    return std::nullopt;
  const int64_t H = four_d ? q.size(1) : *num_heads;
  if (H <= 0 || (num_heads && *num_heads != H)) return std::nullopt;
  const int64_t N = q.size(four_d ? 2 : 1), C = four_d ? H * q.size(3) : q.size(2), D = C / H;
  if (k.sizes() != q.sizes() || q.scalar_type() != k.scalar_type() || !float_type(q) || C % H ||
      D % 8 || D > 256 || D <= 0 || q.size(0) <= 0 || N <= 0)
    return std::nullopt;
  if (block <= 0 || topk < 0 || !pads_fit(pad, N, block)) return std::nullopt;
  const int64_t M = (pad.first + N + pad.second) / block, slices = q.size(0) * H;
  if (M > 4096 || slices > 32768 ||
      slices * static_cast<int64_t>(ftk_score_topk_workspace(1, N, M)) > scratch)
    return std::nullopt;
  auto r = score_topk(q, k, four_d, H, block, topk, pad.first, pad.second, threshold,
                      1.0 / std::sqrt(static_cast<double>(D)), 0, slices, {});
  return std::make_tuple(std::move(r[0]), std::move(r[1]), std::move(r[2]), M);
}

std::optional<std::tuple<Tensor, Tensor>> plain_merge(const Tensor& idx,
                                                      const std::optional<Tensor>& scores,
                                                      int64_t q_block, const Pads& pad,
                                                      std::optional<int64_t> width, int64_t blocks) {
  if (!idx.is_cuda() || idx.dim() != 4 || q_block <= 0 || blocks <= 0 || blocks > 4096 ||
      (scores && (scores->sizes() != idx.sizes() || scores->device() != idx.device())) ||
      !pads_fit(pad, idx.size(2), q_block))
    return std::nullopt;
  const int64_t w = width ? *width : q_block * idx.size(3);
  if (w <= 0) return std::nullopt;
  auto r = qblock_merge(idx, scores, q_block, pad.first, pad.second, blocks, w, false);
  return std::make_tuple(std::move(std::get<0>(r)), std::move(std::get<2>(r)));
}

std::optional<std::tuple<Tensor, Tensor>> plain_attn(
    const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& merged, int64_t H,
    int64_t q_block, int64_t kv_block, std::optional<double> scale, const Pads& q_pad,
    const Pads& kv_pad, std::optional<int64_t> kv_heads) {
  if (!q.is_cuda() || q.dim() != 3 || H <= 0 || !float_type(q)) return std::nullopt;
  const int64_t B = q.size(0), N = q.size(1), D = q.size(2) / H, Hkv = kv_heads ? *kv_heads : H;
  if (q.size(2) != H * D || D <= 0 || D % 16 || D > 256 || Hkv <= 0 || H % Hkv || B <= 0 || N <= 0)
    return std::nullopt;
  for (const Tensor* t : {&k, &v})
    if (t->dim() != 3 || t->size(0) != B || t->size(1) != N || t->size(2) != Hkv * D ||
        t->scalar_type() != q.scalar_type() || t->device() != q.device())
      return std::nullopt;
  for (const int64_t b : {q_block, kv_block})
    if (b <= 0 || b > 128 || (b > 64 && b % 32)) return std::nullopt;
  if (!pads_fit(q_pad, N, q_block) || !pads_fit(kv_pad, N, kv_block)) return std::nullopt;
  if (merged.dim() != 4 || merged.scalar_type() != at::kInt || merged.device() != q.device() ||
      merged.size(0) != B || merged.size(1) != H ||
      merged.size(2) != (q_pad.first + N + q_pad.second) / q_block || merged.size(3) <= 0)
    return std::nullopt;
  // block sizes that every gradient kernel takes
  auto usual = [](int64_t b) { return b == 16 || b == 32 || b == 64 || b == 128; };
  if (!usual(q_block) || !usual(kv_block)) return std::nullopt;
  return sparse_attn(q, k, v, merged, H, Hkv, q_block, kv_block, q_pad.first, kv_pad.first,
                     scale ? *scale : 1.0 / std::sqrt(static_cast<double>(D)));
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  using release = py::call_guard<py::gil_scoped_release>;
  py::register_exception_translator([](std::exception_ptr p) {
    try {
      if (p) std::rethrow_exception(p);
    } catch (const Unsupported& e) {
      PyErr_SetString(PyExc_NotImplementedError, e.what());
    }
  });
  m.attr("built_for") = FTK_BUILT_FOR;   // build.py
  m.def("in_place", [](const Tensor& x, bool four_d, int64_t D) {
    View v;
    return View::strides(x, four_d, D, &v);
  }, "whether the kernels can address a tensor as it is");
  m.def("score_topk", &score_topk, release());
  m.def("score_topk_workspace", &ftk_score_topk_workspace);
  m.def("qblock_merge", &qblock_merge, release());
  m.def("sparse_attn", &sparse_attn, release());
  m.def("plain_score", &plain_score, release());
  m.def("plain_merge", &plain_merge, release());
  m.def("plain_attn", &plain_attn, release());
  m.def("status_word", &status_word, "the device's status word, a pinned host tensor");
  m.def("take_status", &take_status);
  m.def("look", &look);
  m.def("set_deferred", [](bool on) { g_deferred = on; });
  m.def("set_debug", [](bool on) { g_debug = on; });
  m.def("set_timing", &set_timing);
  m.def("take_times", &take_times, release());
}
