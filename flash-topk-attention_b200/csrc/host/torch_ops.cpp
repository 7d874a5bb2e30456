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
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/extension.h>

#include <atomic>
#include <mutex>
#include <string>
#include <tuple>
#include <vector>

#include "../../../include/ftk_api.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
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

// ------------------------------------------------- launch counts and timing
std::atomic<long> g_launches{0};
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

// ------------------------------------------------------------------- layouts
// A tensor addressed as [b][n][h][d]: d dense, 16-byte aligned base, strides
// multiples of 8 elements.  Copies only what cannot be addressed in place.
struct View {
  Tensor t;
  int64_t sb = 0, sn = 0, sh = 0;

  static bool strides(const Tensor& x, bool four_d, int64_t D, View* v) {
    if (x.stride(-1) != 1) return false;
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
  g_launches++;
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
    const auto opt = at::TensorOptions().device(device);
    outs.push_back(at::empty({B, H, N, width}, opt.dtype(at::kInt)));
    outs.push_back(at::empty({B, H, N, width}, opt.dtype(at::kFloat)));
    outs.push_back(at::empty({B, H, N, width}, opt.dtype(at::kFloat)));
  }
  const int64_t first = b0 * N * outs[0].size(3);
  const size_t bytes = ftk_score_topk_workspace(count, N, M);
  const Tensor ws = at::empty({static_cast<int64_t>(bytes)},
                              at::TensorOptions().device(device).dtype(at::kByte));
  check(ftk_score_topk(vq.t.data_ptr(), vk.t.data_ptr(), dtype_code(vq.t), B, H, N, D, vq.sb, vq.sn,
                       vq.sh, vk.sb, vk.sn, vk.sh, b0, count, block, pad_head, pad_tail, scale,
                       topk, threshold, outs[0].data_ptr<int>() + first,
                       outs[1].data_ptr<float>() + first, outs[2].data_ptr<float>() + first,
                       ws.data_ptr(), bytes, status_ptr(device.index()), st.stream()),
        "ftk_score_topk");
  g_launches += 2;
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
  const Tensor idx = topk_idx.to(at::kInt).contiguous();
  Tensor scr;
  if (topk_scores) scr = topk_scores->to(at::kFloat).contiguous();
  const auto opt = at::TensorOptions().device(device);
  Tensor merged = at::empty({B, H, QM, width}, opt.dtype(at::kInt));
  Tensor counts = at::empty({B, H, QM}, opt.dtype(at::kInt));
  std::optional<Tensor> scores;
  if (want_scores) scores = at::empty({B, H, QM, width}, opt.dtype(at::kFloat));
  check(ftk_qblock_merge(idx.data_ptr<int>(), scr.defined() ? scr.data_ptr<float>() : nullptr,
                         B * H, N, topk_idx.size(3), q_block, pad_head, pad_tail, blocks, width,
                         merged.data_ptr<int>(), scores ? scores->data_ptr<float>() : nullptr,
                         counts.data_ptr<int>(), status_ptr(device.index()), st.stream()),
        "ftk_qblock_merge");
  g_launches += 1;
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
  f.o = at::empty(q.sizes(), q.options().memory_format(at::MemoryFormat::Contiguous));
  f.lse = at::empty({q.size(0), m.H, q.size(1)}, q.options().dtype(at::kFloat));
  const ftk_attn a = describe(m, vq, vk, vv, f.lists, f32);
  const size_t bytes = ftk_attn_fwd_workspace(&a);
  const Tensor ws =
      at::empty({static_cast<int64_t>(std::max<size_t>(bytes, 4))}, q.options().dtype(at::kByte));
  {
    TimedCall timed("ftk_sparse_fwd", st);
    check(ftk_attn_fwd(&a, f.o.data_ptr(), f.o.stride(0), f.o.stride(1), D,
                       f.lse.data_ptr<float>(), ws.data_ptr(), bytes, status_ptr(device.index()),
                       st.stream()),
          "ftk_attn_fwd");
  }
  g_launches += 2;
  return f;
}

// Forward and backward of the gathered-KV attention (reference:
// FlashSparseAttnFunc, flash_topk_attn_v2/sparse_attn.py:130-224).
struct SparseAttn : torch::autograd::Function<SparseAttn> {
  static variable_list forward(AutogradContext* ctx, const Tensor& q, const Tensor& k,
                               const Tensor& v, const Tensor& merged, int64_t H, int64_t Hkv,
                               int64_t q_block, int64_t kv_block, int64_t q_pad_head,
                               int64_t kv_pad_head, double scale) {
    const AttnMeta m{H, Hkv, q_block, kv_block, q_pad_head, kv_pad_head, scale};
    Forward f = attn_forward(q, k, v, merged, m);
    ctx->save_for_backward({f.q, f.k, f.v, f.o, f.lse, f.lists});
    ctx->saved_data["meta"] = std::vector<int64_t>{H, Hkv, q_block, kv_block, q_pad_head, kv_pad_head};
    ctx->saved_data["scale"] = scale;
    ctx->mark_non_differentiable({f.lse});
    ctx->set_materialize_grads(false);
    return {f.o, f.lse};
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    variable_list out(11);
    if (!grads[0].defined()) return out;
    const variable_list saved = ctx->get_saved_variables();
    const std::vector<int64_t> i = ctx->saved_data["meta"].toIntVector();
    const AttnMeta m{i[0], i[1], i[2], i[3], i[4], i[5], ctx->saved_data["scale"].toDouble()};
    const Tensor &o = saved[3], &lse = saved[4];
    const at::Device device = o.device();
    c10::cuda::CUDAGuard guard(device);
    look(device.index());
    const auto st = c10::cuda::getCurrentCUDAStream(device.index());
    const bool f32 = o.scalar_type() == at::kFloat;
    const int64_t D = o.size(2) / m.H;
    const View vq(saved[0], false, D), vk(saved[1], false, D), vv(saved[2], false, D);
    Tensor g[1] = {grads[0]};
    if (f32) cast_bf16(g, st);
    else if (g[0].scalar_type() != vq.t.scalar_type()) g[0] = g[0].to(vq.t.scalar_type());
    const View vg(g[0], false, D);
    const ftk_attn a = describe(m, vq, vk, vv, saved[5], f32);
    const size_t bytes = ftk_attn_bwd_workspace(&a);
    const Tensor ws = at::empty({static_cast<int64_t>(std::max<size_t>(bytes, 4))},
                                o.options().dtype(at::kByte));
    Tensor dq = at::empty_like(o);
    int* status = status_ptr(device.index());
    {
      TimedCall timed("ftk_sparse_bwd_dq", st);
      check(ftk_attn_bwd_dq(&a, o.data_ptr(), o.stride(0), o.stride(1), D, vg.t.data_ptr(), vg.sb,
                            vg.sn, vg.sh, lse.data_ptr<float>(), ws.data_ptr(), bytes,
                            dq.data_ptr(), dq.stride(0), dq.stride(1), D, status, st.stream()),
            "ftk_attn_bwd_dq");
    }
    g_launches += 1;
    out[0] = dq;
    if (ctx->needs_input_grad(1) || ctx->needs_input_grad(2)) {
      Tensor dk = at::empty({a.B, a.N, m.Hkv * D}, o.options());
      Tensor dv = at::empty({a.B, a.N, m.Hkv * D}, o.options());
      TimedCall timed("ftk_sparse_bwd_dkv", st);
      check(ftk_attn_bwd_dkv(&a, vg.t.data_ptr(), vg.sb, vg.sn, vg.sh, lse.data_ptr<float>(),
                             ws.data_ptr(), bytes, dk.data_ptr(), dk.stride(0), dk.stride(1), D,
                             dv.data_ptr(), dv.stride(0), dv.stride(1), D, status, st.stream()),
            "ftk_attn_bwd_dkv");
      g_launches += 1;
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
  if (at::GradMode::is_enabled() && (q.requires_grad() || k.requires_grad() || v.requires_grad())) {
    variable_list r = SparseAttn::apply(q, k, v, merged, H, Hkv, q_block, kv_block, q_pad_head,
                                        kv_pad_head, scale);
    return {r[0], r[1]};
  }
  const Forward f =
      attn_forward(q, k, v, merged, {H, Hkv, q_block, kv_block, q_pad_head, kv_pad_head, scale});
  return {f.o, f.lse};
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
  m.def("score_topk", &score_topk, release());
  m.def("score_topk_workspace", &ftk_score_topk_workspace);
  m.def("qblock_merge", &qblock_merge, release());
  m.def("sparse_attn", &sparse_attn, release());
  m.def("status_word", &status_word, "the device's status word, a pinned host tensor");
  m.def("take_status", &take_status);
  m.def("look", &look);
  m.def("set_deferred", [](bool on) { g_deferred = on; });
  m.def("set_debug", [](bool on) { g_debug = on; });
  m.def("launch_count", []() { return g_launches.load(); });
  m.def("set_timing", &set_timing);
  m.def("take_times", &take_times, release());
}
