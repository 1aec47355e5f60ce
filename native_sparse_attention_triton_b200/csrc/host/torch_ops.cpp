// Host side of the operators: argument checks, output and workspace allocation, autograd nodes and the calls into the C
// interface of libnsa_b200.so, in C++.
//
// What this file is bound by is the host's time per call.  A training pass over short samples launches some sixty kernels
// that take 540 us on the device; issued from Python (autograd.Function, ctypes, attribute reads of tensors and streams) it
// took 1100-1300 us of host time per pass, and a decode step of eight launches 300 us.  Here an operator costs its
// allocations, its tensor maps and its launches.
//
// Backward passes are plain autograd nodes (no Python object on the graph); they run on the engine's thread without the GIL.
// Kernels are launched on the current stream of the tensors' device, which is made current for the duration of a call.
#include <ATen/cuda/EmptyTensor.h>
#include <ATen/core/grad_mode.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/extension.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <memory>
#include <mutex>
#include <optional>
#include <unordered_map>
#include <vector>

#include "nsa_b200.h"

namespace {

using at::Tensor;
using torch::autograd::Node;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;
using OptTensor = std::optional<Tensor>;

// ------------------------------------------------------------------------------------------------------------- checks
[[noreturn]] void raise_python(PyObject* type, const char* what) {
  PyErr_SetString(type, what);
  throw py::error_already_set();
}
#define NSA_ASSERT(cond, what) \
  do {                         \
    if (!(cond)) raise_python(PyExc_AssertionError, what); \
  } while (0)

void check_rc(int rc, const char* name) {
  if (rc == 0) return;
  std::string why = rc == -1   ? "invalid argument"
                    : rc == -2 ? "unsupported configuration"
                    : rc == -3 ? "scratch buffer too small"
                    : rc == -4 ? "device status raised"
                    : rc >= 1000 ? "CUDA error " + std::to_string(rc - 1000)
                                 : "unknown";
  throw std::runtime_error(std::string(name) + " failed: code " + std::to_string(rc) + " (" + why + ")");
}

void require_cuda(const Tensor& t) {
  if (!t.is_cuda()) throw std::runtime_error("native_sparse_attention_triton_b200 ops run on CUDA tensors only (no CPU path)");
}
template <typename... Ts>
void require_cuda(const Tensor& t, const Ts&... more) {
  require_cuda(t);
  require_cuda(more...);
}

bool is_16bit(const Tensor& t) { return t.scalar_type() == at::kBFloat16 || t.scalar_type() == at::kHalf; }
int dtype_code(const Tensor& t) {
  if (t.scalar_type() == at::kBFloat16) return NSA_DTYPE_BF16;
  NSA_ASSERT(t.scalar_type() == at::kHalf, "only bfloat16 and float16 tensors are supported");
  return NSA_DTYPE_FP16;
}
void check_qkv_dtypes(const Tensor& q, const Tensor& k, const Tensor& v) {
  NSA_ASSERT(is_16bit(q), "q must be bfloat16 or float16");
  NSA_ASSERT(q.scalar_type() == k.scalar_type() && k.scalar_type() == v.scalar_type(), "q, k and v must have the same dtype");
}
bool is_int32(const Tensor& t) { return t.scalar_type() == at::kInt; }

// ------------------------------------------------------------------------------------------------- tensors and streams
template <typename T = void>
T* ptr(const Tensor& t) { return static_cast<T*>(t.data_ptr()); }
void* ptr(const OptTensor& t) { return t.has_value() ? t->data_ptr() : nullptr; }

Tensor empty(at::IntArrayRef sizes, at::ScalarType type, const at::Device& device) {
  return at::detail::empty_cuda(sizes, type, device, std::nullopt);
}
Tensor empty_like_rows(const Tensor& t) { return empty(t.sizes(), t.scalar_type(), t.device()); }

// Kernels need a unit innermost stride and 16-byte aligned rows; copied only when that does not hold.
Tensor inner_contiguous(const Tensor& t) {
  bool ok = t.stride(-1) == 1 && reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0;
  for (int64_t i = 0; ok && i + 1 < t.dim(); ++i) ok = t.stride(i) % 8 == 0;
  return ok ? t : t.contiguous();
}

// An output gradient as the kernels read it: also copied where it is a contiguous view at an odd offset.
Tensor gradient_rows(const Tensor& t) {
  const Tensor rows = inner_contiguous(t);
  return reinterpret_cast<uintptr_t>(rows.data_ptr()) % 16 ? rows.clone() : rows;
}

// The tensors' device made current, and its current stream.
struct Launch {
  c10::cuda::CUDAGuard guard;
  void* stream;
  explicit Launch(const Tensor& t) : guard(t.device()), stream(c10::cuda::getCurrentCUDAStream(t.device().index()).stream()) {}
};

double default_scale(int64_t head_dim) { return 1.0 / std::sqrt(static_cast<double>(head_dim)); }

// ---------------------------------------------------------------------------------------------------- sequence lengths
// Host copies of cu_seqlens tensors and what is derived from them.  Reading one costs a device-to-host copy (a
// synchronisation); it is remembered for as long as that tensor lives and is not written to (its version counter), so a
// training loop that passes the same cu_seqlens every step synchronises once.  The weak reference keeps the address from
// being reused while the entry exists.
struct Layout {
  int ks, st;
  int total, longest;  // compressed rows in all and of the longest sequence
  Tensor cu;           // their prefix sum on the device
  uint32_t version;
};
struct SeqInfo {
  c10::weak_intrusive_ptr<c10::TensorImpl, c10::UndefinedTensorImpl> key;
  uint32_t version;
  std::vector<int> cu;
  int longest = 0;
  std::mutex mu;
  std::vector<Layout> layouts;
  explicit SeqInfo(const Tensor& t) : key(t.getIntrusivePtr()), version(0) {}
};

std::mutex g_seq_mu;
std::unordered_map<c10::TensorImpl*, std::shared_ptr<SeqInfo>> g_seq;
constexpr size_t kSeqEntries = 64;

bool version_of(const Tensor& t, uint32_t& out) {
  const auto& vc = t.unsafeGetTensorImpl()->version_counter();
  if (!vc.enabled()) return false;  // inference tensors do not count their writes: never remembered
  out = vc.current_version();
  return true;
}

std::shared_ptr<SeqInfo> seq_info(const Tensor& cu) {
  uint32_t version = 0;
  const bool counted = version_of(cu, version);
  if (counted) {
    std::lock_guard<std::mutex> lk(g_seq_mu);
    auto it = g_seq.find(cu.unsafeGetTensorImpl());
    if (it != g_seq.end() && it->second->version == version) return it->second;
  }
  auto info = std::make_shared<SeqInfo>(cu);
  info->version = version;
  Tensor host;
  {
    py::gil_scoped_release nogil;
    host = cu.detach().to(at::kCPU).contiguous();
  }
  const int* p = host.data_ptr<int>();
  info->cu.assign(p, p + host.numel());
  for (size_t i = 0; i + 1 < info->cu.size(); ++i) info->longest = std::max(info->longest, info->cu[i + 1] - info->cu[i]);
  if (counted) {
    std::lock_guard<std::mutex> lk(g_seq_mu);
    if (g_seq.size() >= kSeqEntries) {
      for (auto it = g_seq.begin(); it != g_seq.end();) it = it->second->key.expired() ? g_seq.erase(it) : std::next(it);
      if (g_seq.size() >= kSeqEntries) g_seq.clear();
    }
    g_seq[cu.unsafeGetTensorImpl()] = info;
  }
  return info;
}

// The longest sequence where that is known without a synchronisation, else the bound `total`.
int longest_if_known(const Tensor& cu, int64_t total) {
  uint32_t version = 0;
  if (version_of(cu, version)) {
    std::lock_guard<std::mutex> lk(g_seq_mu);
    auto it = g_seq.find(cu.unsafeGetTensorImpl());
    if (it != g_seq.end() && it->second->version == version) return it->second->longest;
  }
  return (int)total;
}

Layout layout_of(SeqInfo& info, int ks, int st, const at::Device& device) {
  std::lock_guard<std::mutex> lk(info.mu);
  for (const auto& l : info.layouts) {
    uint32_t version = 0;
    if (l.ks == ks && l.st == st && l.cu.device() == device && version_of(l.cu, version) && version == l.version) return l;
  }
  Layout l;
  l.ks = ks; l.st = st; l.total = 0; l.longest = 0;
  std::vector<int> y(info.cu.size(), 0);
  for (size_t i = 0; i + 1 < info.cu.size(); ++i) {
    const int len = info.cu[i + 1] - info.cu[i];
    const int n = len < ks ? 0 : (len - ks) / st + 1;
    l.total += n;
    l.longest = std::max(l.longest, n);
    y[i + 1] = l.total;
  }
  l.cu = at::tensor(y, at::TensorOptions().dtype(at::kInt)).to(device);
  if (version_of(l.cu, l.version)) {
    if (info.layouts.size() >= 8) info.layouts.clear();
    info.layouts.push_back(l);
  }
  return l;
}

// ----------------------------------------------------------------------------------------------------- autograd nodes
// Saved tensors behind one lock, freed with the graph like those of torch's own nodes (a second backward without
// retain_graph raises).  They are unpacked with autograd's dispatch keys in place: an unpack hook may run operators that have to be
// recorded (activation checkpointing computes the forward again in there).
struct SavingNode : Node {
  std::vector<SavedVariable> saved;
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    for (auto& s : saved) s.reset_data();
  }
  std::vector<Tensor> unpack() {
    std::vector<Tensor> out;
    out.reserve(saved.size());
    for (auto& s : saved) out.push_back(s.unpack(shared_from_this()));
    return out;
  }
};

bool needs_graph(std::initializer_list<Tensor> inputs) {
  for (const auto& t : inputs)  // a tangent would be dropped in silence below the autograd dispatch keys
    if (t.defined() && t._fw_grad(/*level=*/0).defined())
      throw std::runtime_error("forward-mode differentiation is not implemented for native_sparse_attention_triton_b200 operators");
  if (!at::GradMode::is_enabled()) return false;
  for (const auto& t : inputs)
    if (t.defined() && t.requires_grad()) return true;
  return false;
}

template <typename N, typename... In>
std::shared_ptr<N> make_node(const In&... inputs) {
  std::shared_ptr<N> n(new N(), torch::autograd::deleteNode);
  n->set_next_edges(torch::autograd::collect_next_edges(inputs...));
  return n;
}
SavedVariable save_input(const Tensor& t) { return SavedVariable(t, /*is_output=*/false); }

// ------------------------------------------------------------------------------------------------------- compression
enum CompressMode : int { kLinear = 0, kWeighted = 1, kAverage = 2 };

struct CompressMeta {
  int mode, ks, st, batch, total_y, longest_x;
};

Tensor compress_forward(const Tensor& x, const Tensor& w, const Tensor& pe, const Tensor& cu, const Layout& l, const CompressMeta& m) {
  const int64_t H = x.size(1), D = x.size(2);
  Tensor y = empty({l.total, H, D}, x.scalar_type(), x.device());
  Tensor bias;
  if (pe.defined()) bias = empty({H, D}, x.scalar_type(), x.device());
  Launch run(x);
  const auto p = [](const Tensor& t) -> void* { return t.defined() ? t.data_ptr() : nullptr; };
  auto fn = m.mode == kLinear ? nsa_linear_compress_fwd : nsa_pool_compress_fwd;
  check_rc(fn(p(x), p(w), p(pe), ptr<int>(cu), ptr<int>(l.cu), p(y), p(bias), (int)x.size(0), m.batch, l.total, l.longest, (int)H, (int)D,
              m.ks, m.st, x.stride(0), x.stride(1), dtype_code(x), run.stream),
           m.mode == kLinear ? "nsa_linear_compress_fwd" : "nsa_pool_compress_fwd");
  return y;
}

struct CompressBackward final : SavingNode {
  CompressMeta m;
  bool has_w, has_pe;
  std::string name() const override { return "CompressBackward"; }
  variable_list apply(variable_list&& grads) override {
    std::lock_guard<std::mutex> lock(mutex_);
    variable_list out(3);
    if (!grads[0].defined()) return out;
    const auto s = unpack();
    at::AutoDispatchBelowADInplaceOrView guard;
    const Tensor &x = s[0], &w = s[1], &pe = s[2], &cu = s[3], &ycu = s[4];
    const int64_t N = x.size(0), H = x.size(1), D = x.size(2);
    const Tensor dy = gradient_rows(grads[0].contiguous());
    Tensor dx = empty({N, H, D}, x.scalar_type(), x.device()), dw, dpe;
    if (has_w) dw = empty(w.sizes(), w.scalar_type(), w.device());
    if (has_pe) dpe = empty(pe.sizes(), pe.scalar_type(), pe.device());
    const auto p = [](const Tensor& t) -> void* { return t.defined() ? t.data_ptr() : nullptr; };
    Launch run(x);
    if (m.mode == kLinear) {
      Tensor dbias;
      if (has_pe) dbias = empty({H, D}, at::kFloat, x.device());
      check_rc(nsa_linear_compress_bwd(p(x), p(w), p(pe), p(dy), ptr<int>(cu), ptr<int>(ycu), p(dx), p(dw), p(dpe),
                                       static_cast<float*>(p(dbias)), (int)N, m.batch, m.total_y, m.longest_x, (int)H, (int)D, m.ks, m.st,
                                       x.stride(0), x.stride(1), dtype_code(x), run.stream),
               "nsa_linear_compress_bwd");
    } else {
      // column sums of dy, then the streaming pass's partial rows
      const long long n = nsa_pool_compress_bwd_workspace_floats((int)N, m.batch, m.longest_x, (int)H, (int)D, m.ks, m.st);
      Tensor ws = empty({n}, at::kFloat, x.device());
      check_rc(nsa_pool_compress_bwd(p(x), p(w), p(pe), p(dy), ptr<int>(cu), ptr<int>(ycu), p(dx), p(dw), p(dpe), ptr<float>(ws), n,
                                     (int)N, m.batch, m.total_y, m.longest_x, (int)H, (int)D, m.ks, m.st, x.stride(0), x.stride(1),
                                     dtype_code(x), run.stream),
               "nsa_pool_compress_bwd");
    }
    out[0] = dx;
    out[1] = dw;
    out[2] = dpe;
    return out;
  }
};

// Argument checks of a compression; the weight and the position embedding, undefined where there is none.
std::pair<Tensor, Tensor> check_compress(const Tensor& x_in, const OptTensor& w_in, const Tensor& cu, int ks, int st, const OptTensor& pe_in,
                                         int mode) {
  NSA_ASSERT(is_16bit(x_in), "x must be float16 or bfloat16");
  NSA_ASSERT(is_int32(cu), "cu_seqlens must be int32");
  NSA_ASSERT(st > 0 && ks % st == 0, "kernel_size must be a multiple of kernel_stride");
  NSA_ASSERT(ks == 16 || ks == 32 || ks == 64 || ks == 128, "kernel_size must be 16, 32, 64 or 128");
  const Tensor w = w_in.value_or(Tensor()), pe = pe_in.value_or(Tensor());
  if (pe.defined()) {
    NSA_ASSERT(pe.scalar_type() == x_in.scalar_type() && pe.device() == x_in.device(), "pe must have x's dtype and device");
    NSA_ASSERT(pe.dim() == 3 && pe.size(0) == x_in.size(1) && pe.size(1) == ks && pe.size(2) == x_in.size(2),
               "pe must be [num_heads, kernel_size, head_dim]");
  }
  if (mode != kAverage) {
    NSA_ASSERT(w.defined() && x_in.scalar_type() == w.scalar_type(), "w must have x's dtype");
    if (mode == kLinear)
      NSA_ASSERT(w.size(0) == x_in.size(1) && w.size(1) == ks * x_in.size(2) && w.size(2) == x_in.size(2) && x_in.size(2) % 8 == 0,
                 "w must be [num_heads, kernel_size * head_dim, head_dim]");
    else
      NSA_ASSERT(w.size(0) == x_in.size(1) && w.size(1) == ks, "w must be [num_heads, kernel_size]");
    require_cuda(w);
  } else {
    NSA_ASSERT(!w.defined(), "don't need additional weight for avgpool");
  }
  require_cuda(x_in, cu);
  if (pe.defined()) require_cuda(pe);
  return {w, pe};
}

std::tuple<Tensor, Tensor> compress(const Tensor& x_in, const OptTensor& w_in, const Tensor& cu, int ks, int st, const OptTensor& pe_in,
                                    int mode) {
  const auto [w, pe] = check_compress(x_in, w_in, cu, ks, st, pe_in, mode);
  auto info = seq_info(cu);
  const Layout l = layout_of(*info, ks, st, x_in.device());
  const CompressMeta m{mode, ks, st, (int)info->cu.size() - 1, l.total, info->longest};
  const bool graph = needs_graph({x_in, w, pe});
  Tensor x, wc, pec, y;
  {
    at::AutoDispatchBelowADInplaceOrView guard;
    x = inner_contiguous(x_in);
    if (w.defined()) wc = w.contiguous();
    if (pe.defined()) pec = pe.contiguous();
    y = compress_forward(x, wc, pec, cu, l, m);
  }
  if (graph) {
    auto node = make_node<CompressBackward>(x_in, w, pe);
    node->m = m;
    node->has_w = wc.defined();
    node->has_pe = pec.defined();
    for (const Tensor& t : {x, wc, pec, cu, l.cu}) node->saved.push_back(save_input(t));
    torch::autograd::set_history(y, node);
  }
  return {y, l.cu};
}

// One row per sequence from staging buffers: every sequence is one window of ks rows, cu and y_cu are its caller's device tensors, and
// nothing is read on the host or remembered.
Tensor compress_staged(const Tensor& x, const OptTensor& w_in, const Tensor& cu, const Tensor& y_cu, int ks, int st, const OptTensor& pe_in,
                       int mode) {
  at::NoGradGuard no_grad;
  at::AutoDispatchBelowADInplaceOrView guard;
  const auto [w, pe] = check_compress(x, w_in, cu, ks, st, pe_in, mode);
  require_cuda(y_cu);
  const int batch = (int)cu.size(0) - 1;
  NSA_ASSERT(is_int32(y_cu) && y_cu.size(0) == cu.size(0) && x.size(0) == (int64_t)batch * ks, "kernel_size rows per sequence");
  const Layout l{ks, st, /*total=*/batch, /*longest=*/1, y_cu, 0};
  return compress_forward(inner_contiguous(x), w.defined() ? w.contiguous() : w, pe.defined() ? pe.contiguous() : pe, cu, l,
                          CompressMeta{mode, ks, st, batch, batch, ks});
}

// ------------------------------------------------------------------------------------- dense varlen and window attention
struct DenseMeta {
  int max_q, max_k, causal, window, stride, left;  // left >= 0: sliding window
  double scale;
};

struct QkvStrides {
  long long s[19];
  int n = 0;
  QkvStrides& add(const Tensor& t) {
    s[n++] = t.stride(0);
    s[n++] = t.stride(1);
    return *this;
  }
};

std::pair<Tensor, Tensor> dense_forward(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& cu_q, const Tensor& cu_k,
                                        const DenseMeta& m) {
  const int64_t N = q.size(0), Hq = q.size(1), D = q.size(2), Nk = k.size(0), Hkv = k.size(1);
  if (Nk == 0)
    return {at::zeros(q.sizes(), q.options()), at::full({N, Hq}, -INFINITY, q.options().dtype(at::kFloat))};
  Tensor o = empty({N, Hq, D}, q.scalar_type(), q.device()), lse = empty({N, Hq}, at::kFloat, q.device());
  QkvStrides st;
  st.add(q).add(k).add(v).add(o);
  const int batch = (int)cu_q.size(0) - 1;
  Launch run(q);
  if (m.left >= 0)
    check_rc(nsa_window_attn_fwd(ptr(q), ptr(k), ptr(v), ptr<int>(cu_q), ptr(o), ptr<float>(lse), (int)N, batch, m.max_q, (int)Hq, (int)Hkv,
                                 (int)D, m.left, st.s, (float)m.scale, dtype_code(q), run.stream),
             "nsa_window_attn_fwd");
  else
    check_rc(nsa_varlen_attn_fwd(ptr(q), ptr(k), ptr(v), ptr<int>(cu_q), ptr<int>(cu_k), ptr(o), ptr<float>(lse), (int)N, (int)Nk, batch,
                                 m.max_q, (int)Hq, (int)Hkv, (int)D, m.causal, m.window, m.stride, st.s, (float)m.scale, dtype_code(q),
                                 run.stream),
             "nsa_varlen_attn_fwd");
  return {o, lse};
}

struct DenseAttentionBackward final : SavingNode {
  DenseMeta m;
  std::string name() const override { return m.left >= 0 ? "SlidingWindowAttentionBackward" : "VarlenAttentionBackward"; }
  variable_list apply(variable_list&& grads) override {
    std::lock_guard<std::mutex> lock(mutex_);
    variable_list out(3);
    if (!grads[0].defined()) return out;
    const auto s = unpack();
    at::AutoDispatchBelowADInplaceOrView guard;
    const Tensor &q = s[0], &k = s[1], &v = s[2], &o = s[3], &lse = s[4], &cu_q = s[5], &cu_k = s[6];
    const int64_t N = q.size(0), Hq = q.size(1), D = q.size(2), Nk = k.size(0), Hkv = k.size(1);
    Tensor dq = empty({N, Hq, D}, q.scalar_type(), q.device()), dk = empty({Nk, Hkv, D}, q.scalar_type(), q.device()),
           dv = empty({Nk, Hkv, D}, q.scalar_type(), q.device());
    if (Nk == 0) {
      out = {dq.zero_(), dk, dv};
      return out;
    }
    const Tensor dout = gradient_rows(grads[0]);
    const int batch = (int)cu_q.size(0) - 1;
    const long long least = nsa_varlen_attn_bwd_workspace((int)N, (int)Nk, (int)Hq, (int)Hkv, (int)D);
    // one pass adds dQ up in the order in which CTAs arrive, the dQ pass in a fixed one
    long long bytes = m.left >= 0 || at::globalContext().deterministicAlgorithms()
                          ? least
                          : nsa_varlen_attn_bwd_workspace_one_pass((int)N, (int)Nk, batch, m.max_k, (int)Hq, (int)Hkv, (int)D);
    Tensor ws;
    try {
      ws = empty({std::max<long long>(bytes, 16)}, at::kByte, q.device());
    } catch (const c10::OutOfMemoryError&) {
      // one pass asks for an fp32 dq more (2.1 GB for 65 536 tokens of 64 heads): where that does not fit, two passes are the way
      if (bytes == least) throw;
      bytes = least;
      ws = empty({std::max<long long>(bytes, 16)}, at::kByte, q.device());
    }
    QkvStrides st;
    st.add(q).add(k).add(v).add(o).add(dout).add(dq).add(dk).add(dv);
    Launch run(q);
    if (m.left >= 0)
      check_rc(nsa_window_attn_bwd(ptr(q), ptr(k), ptr(v), ptr(o), ptr(dout), ptr<float>(lse), ptr<int>(cu_q), ptr(dq), ptr(dk), ptr(dv),
                                   ptr(ws), bytes, (int)N, batch, m.max_q, (int)Hq, (int)Hkv, (int)D, m.left, st.s, (float)m.scale,
                                   dtype_code(q), run.stream),
               "nsa_window_attn_bwd");
    else
      check_rc(nsa_varlen_attn_bwd(ptr(q), ptr(k), ptr(v), ptr(o), ptr(dout), ptr<float>(lse), ptr<int>(cu_q), ptr<int>(cu_k), ptr(dq),
                                   ptr(dk), ptr(dv), ptr(ws), bytes, (int)N, (int)Nk, batch, m.max_q, m.max_k, (int)Hq, (int)Hkv, (int)D,
                                   m.causal, m.window, m.stride, st.s, (float)m.scale, dtype_code(q), run.stream),
               "nsa_varlen_attn_bwd");
    out = {dq, dk, dv};
    return out;
  }
};

// (output on the autograd graph, log-sum-exp, the row-contiguous q and k the kernels read)
struct DenseResult {
  Tensor o, lse, q, k;
};
DenseResult dense_attention(const Tensor& q_in, const Tensor& k_in, const Tensor& v_in, const Tensor& cu_q, const Tensor& cu_k,
                            const DenseMeta& m) {
  const bool graph = needs_graph({q_in, k_in, v_in});
  DenseResult r;
  Tensor v;
  {
    at::AutoDispatchBelowADInplaceOrView guard;
    r.q = inner_contiguous(q_in);
    r.k = inner_contiguous(k_in);
    v = inner_contiguous(v_in);
    std::tie(r.o, r.lse) = dense_forward(r.q, r.k, v, cu_q, cu_k, m);
  }
  if (graph) {
    auto node = make_node<DenseAttentionBackward>(q_in, k_in, v_in);
    node->m = m;
    torch::autograd::set_history(r.o, node);
    for (const Tensor& t : {r.q, r.k, v}) node->saved.push_back(save_input(t));
    node->saved.push_back(SavedVariable(r.o, /*is_output=*/true));
    for (const Tensor& t : {r.lse, cu_q, cu_k}) node->saved.push_back(save_input(t));
  }
  return r;
}

Tensor select_topk_blocks(const Tensor& q, const Tensor& k, const Tensor& lse, int ks, int st, int block_size, int topk, const Tensor& cu_q,
                          const Tensor& cu_k, int max_q, double scale, int init_blocks, int local_blocks) {
  const int64_t N = q.size(0), Hq = q.size(1), D = q.size(2), Hkv = k.size(1);
  const int max_blocks = (max_q + block_size - 1) / block_size;
  Tensor idx = empty({Hkv, N, std::min(topk, max_blocks)}, at::kInt, q.device());
  const long long strides[7] = {q.stride(0), q.stride(1), k.stride(0), k.stride(1), idx.stride(0), idx.stride(1), idx.stride(2)};
  Launch run(q);
  check_rc(nsa_compressed_attn_topk(ptr(q), ptr(k), ptr<float>(lse), ptr<int>(cu_q), ptr<int>(cu_k), ptr<int>(idx), (int)N, (int)k.size(0),
                                    (int)cu_q.size(0) - 1, max_q, (int)Hq, (int)Hkv, (int)D, ks, st, block_size, topk, init_blocks,
                                    local_blocks, strides, (float)scale, dtype_code(q), run.stream),
           "nsa_compressed_attn_topk");
  return idx;
}

std::tuple<Tensor, OptTensor> compressed_attention(const Tensor& q, const Tensor& k, const Tensor& v, int ks, int st, int block_size,
                                                   int topk, const Tensor& cu_q, const Tensor& cu_k, std::optional<int64_t> max_q,
                                                   std::optional<int64_t> max_k, std::optional<double> sm_scale, int init_blocks,
                                                   int local_blocks) {
  require_cuda(q, k, v, cu_q, cu_k);
  if (!max_q) max_q = seq_info(cu_q)->longest;
  if (!max_k) max_k = seq_info(cu_k)->longest;
  NSA_ASSERT(k.size(0) == v.size(0) && q.size(0) > k.size(0), "k and v need as many rows, and fewer than q");
  NSA_ASSERT(k.size(1) == v.size(1) && q.size(1) % k.size(1) == 0, "query heads must be a multiple of the key/value heads");
  check_qkv_dtypes(q, k, v);
  NSA_ASSERT(is_int32(cu_q) && is_int32(cu_k), "cu_seqlens must be int32");
  const DenseMeta m{(int)*max_q, (int)*max_k, 1, ks, st, -1, sm_scale.value_or(default_scale(q.size(2)))};
  DenseResult r = dense_attention(q, k, v, cu_q, cu_k, m);
  if (topk <= 0) return {r.o, std::nullopt};
  NSA_ASSERT(topk >= init_blocks + local_blocks, "topk must be at least init_blocks + local_blocks");
  NSA_ASSERT(block_size % st == 0 && ks % st == 0, "block_size and kernel_size must be multiples of kernel_stride");
  at::AutoDispatchBelowADInplaceOrView guard;
  // no compressed key anywhere: scores are all zero, only forced blocks and the lowest ids are taken
  const Tensor keys = k.size(0) ? r.k : at::zeros({1, k.size(1), k.size(2)}, q.options());
  return {r.o, select_topk_blocks(r.q, keys, r.lse, ks, st, block_size, topk, cu_q, cu_k, m.max_q, m.scale, init_blocks, local_blocks)};
}

Tensor flash_attention_varlen(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& cu_q, const Tensor& cu_k, int64_t max_q,
                              int64_t max_k, bool causal, std::optional<double> sm_scale) {
  require_cuda(q, k, v, cu_q, cu_k);
  check_qkv_dtypes(q, k, v);
  NSA_ASSERT(is_int32(cu_q) && is_int32(cu_k), "cu_seqlens must be int32");
  NSA_ASSERT(q.size(1) % k.size(1) == 0 && k.size(1) == v.size(1), "query heads must be a multiple of the key/value heads");
  return dense_attention(q, k, v, cu_q, cu_k, DenseMeta{(int)max_q, (int)max_k, causal, 1, 1, -1, sm_scale.value_or(default_scale(q.size(2)))}).o;
}

Tensor sliding_window_attention(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& cu, int64_t max_seqlen, int64_t window,
                                std::optional<double> sm_scale) {
  require_cuda(q, k, v, cu);
  check_qkv_dtypes(q, k, v);
  NSA_ASSERT(is_int32(cu), "cu_seqlens must be int32");
  NSA_ASSERT(q.size(0) == k.size(0) && k.size(0) == v.size(0), "q, k and v need as many rows");
  NSA_ASSERT(q.size(1) % k.size(1) == 0 && k.size(1) == v.size(1), "query heads must be a multiple of the key/value heads");
  NSA_ASSERT(q.size(2) == 128, "sliding_window_attention supports head_dim 128");
  NSA_ASSERT(window >= 0, "window_size must not be negative");
  return dense_attention(q, k, v, cu, cu,
                         DenseMeta{(int)max_seqlen, (int)max_seqlen, 1, 1, 1, (int)std::min<int64_t>(window, INT_MAX / 2),
                                   sm_scale.value_or(default_scale(q.size(2)))}).o;
}

// --------------------------------------------------------------------------------------------- selected-block attention
struct SparseAttentionBackward final : SavingNode {
  int block_size;
  double scale;
  std::string name() const override { return "TopkSparseAttentionBackward"; }
  variable_list apply(variable_list&& grads) override {
    std::lock_guard<std::mutex> lock(mutex_);
    variable_list out(3);
    if (!grads[0].defined()) return out;
    const auto s = unpack();
    at::AutoDispatchBelowADInplaceOrView guard;
    const Tensor &q = s[0], &k = s[1], &v = s[2], &o = s[3], &lse = s[4], &cu = s[5], &idx = s[6];
    const int64_t N = q.size(0), Hq = q.size(1), D = q.size(2), Hkv = k.size(1), topk = idx.size(2);
    const int batch = (int)cu.size(0) - 1;
    Tensor dq = empty({N, Hq, D}, q.scalar_type(), q.device()), dk = empty({N, Hkv, D}, q.scalar_type(), q.device()),
           dv = empty({N, Hkv, D}, q.scalar_type(), q.device());
    const Tensor dout = gradient_rows(grads[0]);
    const long long bytes = nsa_topk_sparse_attn_bwd_workspace((int)N, batch, (int)Hq, (int)Hkv, (int)D, (int)topk, block_size);
    Tensor ws = empty({std::max<long long>(bytes, 16)}, at::kByte, q.device());
    QkvStrides st;
    st.add(q).add(k).add(v).add(o).add(dout).add(dq).add(dk).add(dv);
    for (int i = 0; i < 3; ++i) st.s[st.n++] = idx.stride(i);
    Launch run(q);
    check_rc(nsa_topk_sparse_attn_bwd(ptr(q), ptr(k), ptr(v), ptr(o), ptr(dout), ptr<float>(lse), ptr<int>(idx), ptr<int>(cu), nullptr,
                                      ptr(dq), ptr(dk), ptr(dv), ptr(ws), bytes, (int)N, batch, (int)Hq, (int)Hkv, (int)D, (int)topk,
                                      block_size, st.s, (float)scale, dtype_code(q), run.stream),
             "nsa_topk_sparse_attn_bwd");
    out = {dq, dk, dv};
    return out;
  }
};

Tensor topk_sparse_attention(const Tensor& q_in, const Tensor& k_in, const Tensor& v_in, const Tensor& idx, int block_size, const Tensor& cu,
                             std::optional<double> sm_scale) {
  require_cuda(q_in, k_in, v_in, idx, cu);
  NSA_ASSERT(block_size == 32 || block_size == 64 || block_size == 128 || block_size == 256, "block_size must be 32, 64, 128 or 256");
  if (block_size == 32)
    raise_python(PyExc_NotImplementedError, "block_size 32 is not built: the kernels work on 64-key tiles (use 64, 128 or 256)");
  if (idx.size(-1) * (block_size / 64) > 64)
    raise_python(PyExc_NotImplementedError, "at most 64 tiles of 64 keys per query (topk * block_size / 64 <= 64)");
  NSA_ASSERT(q_in.size(1) % k_in.size(1) == 0 && k_in.size(1) == v_in.size(1) && k_in.size(1) == idx.size(0),
             "query heads must be a multiple of the key/value heads, and topk_idx have one row set per key/value head");
  check_qkv_dtypes(q_in, k_in, v_in);
  NSA_ASSERT(is_int32(idx), "topk_idx must be int32");
  NSA_ASSERT(is_int32(cu), "cu_seqlens must be int32");
  const double scale = sm_scale.value_or(default_scale(q_in.size(2)));
  const bool graph = needs_graph({q_in, k_in, v_in});
  Tensor q, k, v, o, lse;
  {
    at::AutoDispatchBelowADInplaceOrView guard;
    q = inner_contiguous(q_in);
    k = inner_contiguous(k_in);
    v = inner_contiguous(v_in);
    const int64_t N = q.size(0), Hq = q.size(1), D = q.size(2);
    o = empty({N, Hq, D}, q.scalar_type(), q.device());
    lse = empty({N, Hq}, at::kFloat, q.device());
    QkvStrides st;
    st.add(q).add(k).add(v).add(o);
    for (int i = 0; i < 3; ++i) st.s[st.n++] = idx.stride(i);
    Launch run(q);
    check_rc(nsa_topk_sparse_attn_fwd_bounded(ptr(q), ptr(k), ptr(v), ptr<int>(idx), ptr<int>(cu), ptr(o), ptr<float>(lse), (int)N,
                                      (int)cu.size(0) - 1, std::max(1, longest_if_known(cu, N)), (int)Hq, (int)k.size(1), (int)D, (int)idx.size(2), block_size, st.s, (float)scale,
                                      dtype_code(q), run.stream),
             "nsa_topk_sparse_attn_fwd");
  }
  if (graph) {
    auto node = make_node<SparseAttentionBackward>(q_in, k_in, v_in);
    node->block_size = block_size;
    node->scale = scale;
    torch::autograd::set_history(o, node);
    for (const Tensor& t : {q, k, v}) node->saved.push_back(save_input(t));
    node->saved.push_back(SavedVariable(o, /*is_output=*/true));
    for (const Tensor& t : {lse, cu, idx}) node->saved.push_back(save_input(t));
  }
  return o;
}

// ----------------------------------------------------------------------------------------------------------- gated sum
struct GateCombineBackward final : SavingNode {
  std::string name() const override { return "GateCombineBackward"; }
  variable_list apply(variable_list&& grads) override {
    std::lock_guard<std::mutex> lock(mutex_);
    variable_list out(4);
    if (!grads[0].defined()) return out;
    const auto s = unpack();
    at::AutoDispatchBelowADInplaceOrView guard;
    const Tensor& gate = s[0];
    const Tensor dout = gradient_rows(grads[0]);
    for (int i = 0; i < 4; ++i) out[i] = empty_like_rows(s[i]);
    QkvStrides st;
    st.add(gate).add(s[1]).add(s[2]).add(s[3]).add(dout).add(out[0]).add(out[1]).add(out[2]).add(out[3]);
    Launch run(dout);
    check_rc(nsa_gate_combine_bwd(ptr(gate), ptr(s[1]), ptr(s[2]), ptr(s[3]), ptr(dout), ptr(out[0]), ptr(out[1]), ptr(out[2]), ptr(out[3]),
                                  (int)s[1].size(0), (int)s[1].size(1), (int)s[1].size(2), st.s, dtype_code(dout), run.stream),
             "nsa_gate_combine_bwd");
    return out;
  }
};

Tensor gate_combine_forward(const Tensor& gate, const Tensor& a, const Tensor& b, const Tensor& c) {
  Tensor o = empty_like_rows(a);
  QkvStrides st;
  st.add(gate).add(a).add(b).add(c).add(o);
  Launch run(o);
  check_rc(nsa_gate_combine_fwd(ptr(gate), ptr(a), ptr(b), ptr(c), ptr(o), (int)a.size(0), (int)a.size(1), (int)a.size(2), st.s,
                                dtype_code(o), run.stream),
           "nsa_gate_combine_fwd");
  return o;
}

Tensor gate_combine(const Tensor& gate, const Tensor& o_cmp, const Tensor& o_sel, const Tensor& o_win) {
  require_cuda(gate, o_cmp, o_sel, o_win);
  NSA_ASSERT(is_16bit(o_cmp), "the branch outputs must be bfloat16 or float16");
  NSA_ASSERT(o_sel.scalar_type() == o_cmp.scalar_type() && o_win.scalar_type() == o_cmp.scalar_type() &&
                 gate.scalar_type() == o_cmp.scalar_type(), "gate and branch outputs must have the same dtype");
  NSA_ASSERT(o_cmp.sizes() == o_sel.sizes() && o_sel.sizes() == o_win.sizes() && o_cmp.dim() == 3, "the branch outputs must have the same shape");
  NSA_ASSERT(gate.dim() == 3 && gate.size(0) == o_cmp.size(0) && gate.size(1) == o_cmp.size(1) && gate.size(2) == 3,
             "gate must be [rows, num_heads, 3]");
  NSA_ASSERT(o_cmp.size(2) == 64 || o_cmp.size(2) == 128, "gate_combine supports head_dim 64 and 128");
  const bool graph = needs_graph({gate, o_cmp, o_sel, o_win});
  Tensor t[4], o;
  {
    at::AutoDispatchBelowADInplaceOrView guard;
    t[0] = gate.contiguous();
    t[1] = inner_contiguous(o_cmp);
    t[2] = inner_contiguous(o_sel);
    t[3] = inner_contiguous(o_win);
    o = gate_combine_forward(t[0], t[1], t[2], t[3]);
  }
  if (graph) {
    auto node = make_node<GateCombineBackward>(gate, o_cmp, o_sel, o_win);
    for (const Tensor& x : t) node->saved.push_back(save_input(x));
    torch::autograd::set_history(o, node);
  }
  return o;
}

// ----------------------------------------------------------------------------------------------------- rotary embedding
struct RopeMeta {
  int step, stride;
  double scaling;
};
Tensor rope_launch(const Tensor& x, const Tensor& inv_freq, const Tensor& cu, const RopeMeta& m, int inverse) {
  Tensor y = empty_like_rows(x);
  Launch run(x);
  check_rc(nsa_rope(ptr(x), ptr(y), ptr<float>(inv_freq), ptr<int>(cu), (int)x.size(0), (int)cu.size(0) - 1, (int)x.size(1), (int)x.size(2),
                    m.step, m.stride, (float)m.scaling, inverse, x.stride(0), x.stride(1), y.stride(0), y.stride(1), dtype_code(x),
                    run.stream),
           "nsa_rope");
  return y;
}
struct RopeBackward final : SavingNode {
  RopeMeta m;
  std::string name() const override { return "RopeBackward"; }
  variable_list apply(variable_list&& grads) override {
    std::lock_guard<std::mutex> lock(mutex_);
    variable_list out(1);
    if (!grads[0].defined()) return out;
    const auto s = unpack();
    at::AutoDispatchBelowADInplaceOrView guard;
    out[0] = rope_launch(gradient_rows(grads[0]), s[0], s[1], m, 1);
    return out;
  }
};

Tensor rope(const Tensor& x, const Tensor& inv_freq, const Tensor& cu, int64_t step, int64_t stride, double scaling) {
  require_cuda(x, inv_freq, cu);
  NSA_ASSERT(is_16bit(x), "x must be bfloat16 or float16");
  NSA_ASSERT(x.dim() == 3 && (x.size(2) == 64 || x.size(2) == 128), "rope supports head_dim 64 and 128");
  NSA_ASSERT(inv_freq.scalar_type() == at::kFloat && inv_freq.dim() == 1 && inv_freq.size(0) == x.size(2) / 2 && inv_freq.is_contiguous(),
             "inv_freq must be a contiguous float32 [head_dim / 2]");
  NSA_ASSERT(is_int32(cu) && cu.dim() == 1 && cu.is_contiguous(), "cu_seqlens must be a contiguous int32 vector");
  NSA_ASSERT(step >= 0 && stride >= 1, "step must not be negative and stride at least 1");
  if (step > 0) NSA_ASSERT(x.size(0) == cu.size(0) - 1, "a decode step has one row per sequence");
  const RopeMeta m{(int)step, (int)stride, scaling};
  const bool graph = needs_graph({x});
  Tensor y;
  {
    at::AutoDispatchBelowADInplaceOrView guard;
    y = rope_launch(inner_contiguous(x), inv_freq, cu, m, 0);
  }
  if (graph) {
    auto node = make_node<RopeBackward>(x);
    node->m = m;
    node->saved.push_back(save_input(inv_freq));
    node->saved.push_back(save_input(cu));
    torch::autograd::set_history(y, node);
  }
  return y;
}

// -------------------------------------------------------------------------------------------------- single-token operators
// Split-KV scratch, one buffer per (device, stream): calls on one stream cannot overlap.  The kernels leave the control words
// at the front at zero when they finish, so a buffer zeroed once serves every later call on that stream; it is regrown (and
// zeroed again) when a call needs more.  At most kScratchBuffers are kept.  A CUDA-graph capture takes none of them: a replay
// finds its buffer by address, after other calls on the stream may have outgrown it, dirtied control words beyond their own, or had
// it given back.  It gets one of the graph's pool, zeroed by a captured kernel at every replay.
struct Scratch {
  Tensor buf;
  long long ctrl = 0;
};
std::mutex g_scratch_mu;
std::unordered_map<uint64_t, Scratch> g_scratch;
constexpr size_t kScratchBuffers = 64;

uint64_t scratch_key(const at::Device& d, const c10::cuda::CUDAStream& s) {
  return (reinterpret_cast<uint64_t>(s.stream()) << 6) ^ (uint64_t)(d.index() & 63);
}

// `pairs`: (sequence, KV head) pairs; `n`: floats
Tensor take_scratch(long long pairs, long long n, const at::Device& device, uint64_t key) {
  const long long ctrl = (pairs + 1 + 63) / 64 * 64;
  const auto fresh = [&] {
    Tensor t = empty({n}, at::kFloat, device);
    t.narrow(0, 0, ctrl).zero_();
    return t;
  };
  if (c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None) return fresh();
  std::lock_guard<std::mutex> lk(g_scratch_mu);
  auto it = g_scratch.find(key);
  if (it == g_scratch.end() || it->second.buf.numel() < n) {
    if (it == g_scratch.end() && g_scratch.size() >= kScratchBuffers) g_scratch.clear();  // their tensors go back to the allocator
    return (g_scratch[key] = Scratch{fresh(), ctrl}).buf;
  }
  // the control region grows with the pairs; beyond the previous call's region lie that call's partial results
  if (it->second.ctrl < ctrl) it->second.buf.narrow(0, 0, ctrl).zero_();
  it->second.ctrl = ctrl;
  return it->second.buf;
}

// A decode entry point, call(scratch, floats, splits): first without scratch, which the cluster kernels do not need and for want of
// which the split-KV kernel's route answers -3 before it launches anything; then with it.
template <typename Call>
void with_scratch(const char* name, int batch, int hkv, int d, int cache_len, bool compressed, const at::Device& device, Call call) {
  const int splits = nsa_decode_num_splits(batch, hkv, (cache_len + 63) / 64);
  int rc = call(static_cast<float*>(nullptr), 0ll, splits);
  if (rc == -3) {
    const long long n = compressed ? nsa_compressed_decode_scratch_floats(batch, hkv, d, splits, cache_len)
                                   : nsa_decode_scratch_floats(batch, hkv, d, splits);
    const uint64_t key = scratch_key(device, c10::cuda::getCurrentCUDAStream(device.index()));
    const Tensor buf = take_scratch((long long)batch * hkv, n, device, key);
    rc = call(buf.data_ptr<float>(), n, splits);
    if (rc) {  // a failed call may have left control words that are not zero
      std::lock_guard<std::mutex> lk(g_scratch_mu);
      g_scratch.erase(key);
    }
  }
  check_rc(rc, name);
}

void check_decode(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& seqlens) {
  require_cuda(q, k, v, seqlens);
  check_qkv_dtypes(q, k, v);
  NSA_ASSERT(is_int32(seqlens), "seqlens must be int32");
  NSA_ASSERT(k.size(1) == v.size(1) && q.size(0) == seqlens.size(0), "k and v need as many rows, seqlens one entry per query");
  NSA_ASSERT(k.size(2) == v.size(2) && q.size(1) % k.size(2) == 0, "query heads must be a multiple of the key/value heads");
}

struct DecodeStrides {
  long long s[13] = {0};
  DecodeStrides(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& o, const Tensor* idx = nullptr) {
    s[0] = q.stride(0); s[1] = q.stride(1);
    for (int i = 0; i < 3; ++i) { s[2 + i] = k.stride(i); s[5 + i] = v.stride(i); }
    s[8] = o.stride(0); s[9] = o.stride(1);
    if (idx)
      for (int i = 0; i < 3; ++i) s[10 + i] = idx->stride(i);
  }
};

Tensor flash_attention_decode(const Tensor& q_in, const Tensor& k_in, const Tensor& v_in, const Tensor& seqlens,
                              std::optional<double> sm_scale) {
  check_decode(q_in, k_in, v_in, seqlens);
  at::NoGradGuard no_grad;
  at::AutoDispatchBelowADInplaceOrView guard;
  const Tensor q = inner_contiguous(q_in), k = inner_contiguous(k_in), v = inner_contiguous(v_in);
  const int64_t B = q.size(0), Hq = q.size(1), D = q.size(2), L = k.size(1), Hkv = k.size(2);
  if (L == 0) return at::zeros_like(q);
  Tensor o = empty_like_rows(q);  // every row is written: a sequence without visible rows gets zeros from the kernel
  Launch run(q);
  const DecodeStrides st(q, k, v, o);
  with_scratch("nsa_flash_attn_decode", (int)B, (int)Hkv, (int)D, (int)L, /*compressed=*/false, q.device(),
               [&](float* scratch, long long floats, int splits) {
                 return nsa_flash_attn_decode(ptr(q), ptr(k), ptr(v), ptr<int>(seqlens), ptr(o), scratch, floats, splits, (int)B, (int)L,
                                              (int)Hq, (int)Hkv, (int)D, st.s, (float)sm_scale.value_or(default_scale(D)), dtype_code(q),
                                              run.stream);
               });
  return o;
}

Tensor topk_sparse_attention_decode(const Tensor& q_in, const Tensor& k_in, const Tensor& v_in, const Tensor& idx_in, int block_size,
                                    const Tensor& seqlens, std::optional<double> sm_scale) {
  check_decode(q_in, k_in, v_in, seqlens);
  NSA_ASSERT(k_in.size(2) == idx_in.size(0) && q_in.size(0) == idx_in.size(1), "topk_idx must be [num_kv_heads, batch, topk]");
  at::NoGradGuard no_grad;
  at::AutoDispatchBelowADInplaceOrView guard;
  const Tensor q = inner_contiguous(q_in), k = inner_contiguous(k_in), v = inner_contiguous(v_in);
  const Tensor idx = is_int32(idx_in) ? idx_in : idx_in.to(at::kInt);
  const int64_t B = q.size(0), Hq = q.size(1), D = q.size(2), L = k.size(1), Hkv = k.size(2), T = idx.size(-1);
  if (L == 0) return at::zeros_like(q);
  Tensor o = empty_like_rows(q);
  Launch run(q);
  const DecodeStrides st(q, k, v, o, &idx);
  check_rc(nsa_topk_sparse_attn_decode(ptr(q), ptr(k), ptr(v), ptr<int>(idx), ptr<int>(seqlens), ptr(o), nullptr, 0, 1, (int)B, (int)L, (int)Hq,
                                       (int)Hkv, (int)D, (int)T, block_size, st.s, (float)sm_scale.value_or(default_scale(D)), dtype_code(q),
                                       run.stream),
           "nsa_topk_sparse_attn_decode");
  return o;
}

std::tuple<Tensor, Tensor> compressed_attention_decode(const Tensor& q_in, const Tensor& k_in, const Tensor& v_in, const Tensor& seqlens_in,
                                                       const Tensor& comp_in, int ks, int st_, int block_size, int topk, int init_blocks,
                                                       int local_blocks, std::optional<double> sm_scale, std::optional<int64_t> max_seqlen) {
  NSA_ASSERT(block_size % ks == 0 && ks % st_ == 0, "block_size must be a multiple of kernel_size, kernel_size of kernel_stride");
  require_cuda(q_in, k_in, v_in, seqlens_in, comp_in);
  at::NoGradGuard no_grad;
  at::AutoDispatchBelowADInplaceOrView guard;
  const int64_t B = q_in.size(0), Hq = q_in.size(1), D = q_in.size(2), L = k_in.size(1), Hkv = k_in.size(2);
  if (L == 0)  // input is too short to have a compressed block
    return {at::zeros_like(q_in), at::zeros({Hkv, B, 1}, q_in.options().dtype(at::kInt))};
  const Tensor q = inner_contiguous(q_in), k = inner_contiguous(k_in), v = inner_contiguous(v_in);
  const Tensor seqlens = is_int32(seqlens_in) ? seqlens_in : seqlens_in.to(at::kInt), comp = is_int32(comp_in) ? comp_in : comp_in.to(at::kInt);
  const int longest = max_seqlen ? (int)*max_seqlen : (int)seqlens.max().item<int>();
  const int max_blocks = (longest + block_size - 1) / block_size;
  Tensor o = empty_like_rows(q), idx = empty({Hkv, B, std::min(topk, max_blocks)}, at::kInt, q.device());
  Launch run(q);
  const DecodeStrides st(q, k, v, o, &idx);
  with_scratch("nsa_compressed_attn_decode", (int)B, (int)Hkv, (int)D, (int)L, /*compressed=*/true, q.device(),
               [&](float* scratch, long long floats, int splits) {
                 return nsa_compressed_attn_decode(ptr(q), ptr(k), ptr(v), ptr<int>(seqlens), ptr<int>(comp), ptr(o), ptr<int>(idx), scratch,
                                                   floats, splits, (int)B, (int)L, longest, (int)Hq, (int)Hkv, (int)D, ks, st_, block_size,
                                                   topk, init_blocks, local_blocks, st.s, (float)sm_scale.value_or(default_scale(D)),
                                                   dtype_code(q), run.stream);
               });
  return {o, idx};
}

// ------------------------------------------------------------------------------------------------------- inference step
// The caches of a layer as NSACache holds them: [2, batch, rows, heads, d] tensors and int32 counters.
struct CacheRefs {
  Tensor sel, sel_len, cmp, cmp_len, stage, stage_len, win, win_len, ticket;
};
CacheRefs cache_refs(const std::vector<Tensor>& c) {
  NSA_ASSERT(c.size() == 9, "nine cache tensors");
  return CacheRefs{c[0], c[1], c[2], c[3], c[4], c[5], c[6], c[7], c[8]};
}

// One decode step of nsa_infer in one launch (two for linear compression).  Returns nothing when the shapes are not the fused
// kernel's, before anything has been launched; the caller then takes the operators one by one.
std::optional<Tensor> decode_step(const Tensor& q_in, const Tensor& k_in, const Tensor& v_in, const Tensor& gate_in,
                                  const std::vector<Tensor>& caches, const OptTensor& w_k, const OptTensor& w_v, const OptTensor& pe,
                                  int mode_k, int mode_v, const Tensor& inv_freq, double rope_scaling, int ks, int st, int block_size,
                                  int topk, int init_blocks, int local_blocks, const OptTensor& out) {
  const CacheRefs c = cache_refs(caches);
  require_cuda(q_in, k_in, v_in, gate_in, inv_freq);
  at::NoGradGuard no_grad;
  at::AutoDispatchBelowADInplaceOrView guard;
  const int64_t B = k_in.size(0), Hkv = k_in.size(1), D = k_in.size(2), Hq = q_in.size(1);
  NSA_ASSERT(q_in.size(0) == B && k_in.sizes() == v_in.sizes() && B <= c.sel.size(1), "one row per sequence, no more than the cache holds");
  NSA_ASSERT(Hkv == c.sel.size(3) && D == c.sel.size(4) && q_in.size(2) == D && Hq % Hkv == 0, "heads and head_dim must be the cache's");
  NSA_ASSERT(is_16bit(q_in) && q_in.scalar_type() == k_in.scalar_type() && q_in.scalar_type() == v_in.scalar_type() &&
                 q_in.scalar_type() == gate_in.scalar_type() && q_in.scalar_type() == c.sel.scalar_type(),
             "query, key, value, gate and caches must have the same 16-bit dtype");
  NSA_ASSERT(gate_in.size(0) == B && gate_in.size(1) == Hq && gate_in.size(2) == 3, "gate must be [batch, query heads, 3]");
  NSA_ASSERT(block_size % ks == 0 && ks % st == 0, "block_size must be a multiple of kernel_size, kernel_size of kernel_stride");
  if ((D != 64 && D != 128) || Hq / Hkv > 16 || c.cmp.size(2) == 0 || c.win.size(2) == 0) return std::nullopt;
  if (inv_freq.scalar_type() != at::kFloat || inv_freq.dim() != 1 || inv_freq.size(0) != D / 2 || !inv_freq.is_contiguous()) return std::nullopt;
  NSA_ASSERT((mode_k == kLinear) == (mode_v == kLinear), "linear and pooling compression take separate launches");
  const bool linear = mode_k == kLinear;
  const auto weight = [&](const OptTensor& w, int mode) {  // of the keys or the values; average pooling has none
    if (mode == kAverage) return Tensor();
    NSA_ASSERT(w.has_value(), "this compression needs weights");
    require_cuda(*w);
    NSA_ASSERT(w->scalar_type() == c.sel.scalar_type(), "w must have the caches' dtype");
    NSA_ASSERT(w->size(0) == Hkv && w->numel() == Hkv * ks * (linear ? D * D : 1), "w must be [num_heads, kernel_size * head_dim, head_dim] or [num_heads, kernel_size]");
    return w->contiguous();
  };
  const Tensor wk = weight(w_k, mode_k), wv = weight(w_v, mode_v);
  if (pe) {
    require_cuda(*pe);
    NSA_ASSERT(pe->scalar_type() == c.sel.scalar_type() && pe->numel() == Hkv * ks * D, "pe must be [num_heads, kernel_size, head_dim] of the caches' dtype");
  }
  const Tensor q = inner_contiguous(q_in), k = inner_contiguous(k_in), v = inner_contiguous(v_in), gate = gate_in.contiguous();
  Launch run(q);
  const int fits = nsa_decode_step_supported((int)B, (int)Hq, (int)Hkv, (int)D, ks, st, block_size, topk, init_blocks, local_blocks,
                                             (int)c.sel.size(2), (int)c.cmp.size(2), (int)c.win.size(2), dtype_code(q));
  if (fits == -2) return std::nullopt;
  check_rc(fits, "nsa_decode_step");
  Tensor pec;
  if (pe) pec = pe->contiguous();
  const auto p = [](const Tensor& t) -> void* { return t.defined() ? t.data_ptr() : nullptr; };
  Tensor o = out ? *out : empty_like_rows(q);
  Tensor taps;
  if (linear) {
    taps = empty({ks, B, 2, Hkv, D}, at::kFloat, q.device());
    const long long s[8] = {k.stride(0), k.stride(1), v.stride(0), v.stride(1), c.stage.stride(0), c.stage.stride(1), c.stage.stride(2),
                            c.stage.stride(3)};
    check_rc(nsa_linear_decode_taps(ptr(k), ptr(v), ptr(wk), ptr(wv), p(pec), ptr(c.stage), ptr<int>(c.stage_len), ptr<float>(taps), (int)B, (int)Hkv,
                                    (int)D, ks, st, s, dtype_code(q), run.stream),
             "nsa_linear_decode_taps");
  }
  QkvStrides s;
  long long strides[26];
  s.add(q).add(k).add(v).add(gate).add(o);
  std::copy(s.s, s.s + 10, strides);
  int n = 10;
  for (const Tensor* t : {&c.sel, &c.cmp, &c.stage, &c.win})
    for (int i = 0; i < 4; ++i) strides[n++] = t->stride(i);
  check_rc(nsa_decode_step(ptr(q), ptr(k), ptr(v), ptr(gate), ptr(o), ptr(c.sel), ptr<int>(c.sel_len), ptr(c.cmp), ptr<int>(c.cmp_len),
                           ptr(c.stage), ptr<int>(c.stage_len), ptr(c.win), ptr<int>(c.win_len), ptr<int>(c.ticket), p(wk), p(wv),
                           p(pec), static_cast<float*>(p(taps)), ptr<float>(inv_freq), (float)rope_scaling, (int)B, (int)Hq, (int)Hkv,
                           (int)D, ks, st, block_size, topk, init_blocks, local_blocks, (int)c.sel.size(2), (int)c.cmp.size(2),
                           (int)c.win.size(2), strides, (float)default_scale(D), dtype_code(q), run.stream),
           "nsa_decode_step");
  return o;
}

void cache_fill(const Tensor& cache, const Tensor& len, const Tensor& key, const Tensor& value, const Tensor& cu, int mode, int window, int hop,
                void* stream) {
  const long long s[8] = {cache.stride(0), cache.stride(1), cache.stride(2), cache.stride(3), key.stride(0), key.stride(1), value.stride(0),
                          value.stride(1)};
  check_rc(nsa_kv_cache_fill(ptr(cache), ptr<int>(len), ptr(key), ptr(value), ptr<int>(cu), mode, window, hop, (int)key.size(0),
                             (int)cu.size(0) - 1, (int)cache.size(2), (int)key.size(1), (int)key.size(2), s, stream),
           "nsa_kv_cache_fill");
}

// The prefill of nsa_infer with the library's own compression and rotary embedding.  The lengths come from the host copy of
// cu_seqlens, so nothing waits for the device once that tensor has been seen.
Tensor prefill(const Tensor& cu, const Tensor& q_in, const Tensor& k_in, const Tensor& v_in, const Tensor& gate, const std::vector<Tensor>& caches,
               const OptTensor& w_k, const OptTensor& w_v, const OptTensor& pe, int mode_k, int mode_v, const Tensor& inv_freq,
               double rope_scaling, int ks, int st, int block_size, int topk, int init_blocks, int local_blocks, int window) {
  const CacheRefs c = cache_refs(caches);
  at::NoGradGuard no_grad;
  require_cuda(q_in, k_in, v_in, gate, cu);
  NSA_ASSERT(k_in.sizes() == v_in.sizes() && k_in.scalar_type() == c.sel.scalar_type() && v_in.scalar_type() == c.sel.scalar_type(),
             "key and value must have the same shape and the cache's dtype");
  NSA_ASSERT(k_in.size(1) == c.sel.size(3) && k_in.size(2) == c.sel.size(4), "heads and head_dim must be the cache's");
  NSA_ASSERT(is_int32(cu) && cu.size(0) - 1 <= c.sel.size(1), "cu_seqlens must be int32, with no more sequences than the cache holds");
  const Tensor k = inner_contiguous(k_in), v = inner_contiguous(v_in);
  const auto info = seq_info(cu);
  const Layout l = layout_of(*info, ks, st, k.device());
  Launch run(k);
  cache_fill(c.stage, c.stage_len, k, v, cu, 2, ks, st, run.stream);
  auto [ck, cu_k] = compress(k, w_k, cu, ks, st, pe, mode_k);
  const Tensor cv = std::get<0>(compress(v, w_v, cu, ks, st, std::nullopt, mode_v));
  const Tensor q = rope(q_in, inv_freq, cu, 0, 1, rope_scaling);
  ck = rope(ck, inv_freq, cu_k, 0, st, rope_scaling);
  const Tensor kr = rope(k, inv_freq, cu, 0, 1, rope_scaling);
  cache_fill(c.cmp, c.cmp_len, ck, cv, cu_k, 0, 0, 0, run.stream);
  cache_fill(c.sel, c.sel_len, kr, v, cu, 0, 0, 0, run.stream);
  cache_fill(c.win, c.win_len, kr, v, cu, 1, window, 0, run.stream);
  auto [o_cmp, idx] = compressed_attention(q, ck, cv, ks, st, block_size, topk, cu, cu_k, info->longest, l.longest, std::nullopt, init_blocks,
                                           local_blocks);
  NSA_ASSERT(idx.has_value(), "topk must be positive");
  const Tensor o_sel = topk_sparse_attention(q, kr, v, *idx, block_size, cu, std::nullopt);
  const Tensor o_win = sliding_window_attention(q, kr, v, cu, info->longest, window, std::nullopt);
  return gate_combine(gate, o_cmp, o_sel, o_win);
}

}  // namespace

PYBIND11_MODULE(_nsa_host, m) {
  m.doc() = "Host side of the native_sparse_attention_triton_b200 operators.";
  m.def("compress", &compress);
  m.def("compress_staged", &compress_staged);
  m.def("compressed_attention", &compressed_attention);
  m.def("flash_attention_varlen", &flash_attention_varlen);
  m.def("sliding_window_attention", &sliding_window_attention);
  m.def("topk_sparse_attention", &topk_sparse_attention);
  m.def("gate_combine", &gate_combine);
  m.def("rope", &rope);
  m.def("flash_attention_decode", &flash_attention_decode);
  m.def("topk_sparse_attention_decode", &topk_sparse_attention_decode);
  m.def("compressed_attention_decode", &compressed_attention_decode);
  m.def("decode_step", &decode_step);
  m.def("prefill", &prefill);
}
