// Host path of the layers: one call from Python per forward.
//
// A plan (LinearPlan, MoEPlan) is built once after loading and owns everything a forward needs - the
// C-ABI weight descriptors, references to the tensors behind them, slot buffers, workspaces.  Its
// call picks the route, allocates the outputs and one workspace with torch's allocator and launches
// the library's kernels on the current stream.  The same sequence from Python (custom-op dispatch,
// ctypes structs rebuilt per call, one torch.empty per intermediate) cost 40 us for the one launch of
// a 4096 x 4096 decode row and 70 to 100 us for the seven of a routed layer, several times what
// their kernels take.
//
// The library is reached through dlsym on the path the ctypes loader uses, so that both bind the
// same file and a missing symbol fails closed.
#include <ATen/ATen.h>
#include <ATen/cuda/CUDAEvent.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <pybind11/stl.h>
#include <torch/csrc/utils/pybind.h>

#include <atomic>
#include <dlfcn.h>
#include <map>
#include <memory>
#include <mutex>
#include <stdexcept>
#include <string>
#include <tuple>
#include <vector>

#include "../../include/gridbook_b200.h"

namespace py = pybind11;

namespace {

// The library's entries used here.
#define GB_ENTRIES(F) \
  F(gb_last_error) F(gb_gemv_hinted_workspace_bytes) F(gb_gemv) F(gb_gemv_row_batch_max) F(gb_gemv_tab) \
  F(gb_gemv_tab_slots_bytes) F(gb_fp4_act_qdq) F(gb_fp8_act_qdq) F(gb_fp8_quantize_rows) F(gb_nvfp4_sf_bytes) \
  F(gb_nvfp4_quantize_rows) F(gb_expand_fp4_nvfp4) F(gb_expand_fp4_bf16) F(gb_expand_fp8) F(gb_expand_fp8_bf16) \
  F(gb_gemv_shared) F(gb_gemv_shared_applies) F(gb_expand_fp4_nvfp4_beside) F(gb_expand_fp8_beside) F(gb_gemm_fp4) F(gb_gemm_tn) F(gb_gemm_tn_grouped) F(gb_moe_route_ws) F(gb_moe_route_workspace_bytes) \
  F(gb_moe_gather_rows) F(gb_moe_swiglu_rows) F(gb_moe_gemv) F(gb_moe_gemv_sorted) F(gb_moe_mlp_pairs) \
  F(gb_moe_mlp_pairs_workspace_bytes) F(gb_moe_combine) F(gb_gemv_hinted) F(gb_scales_e4m3) F(gb_moe_route_inv) \
  F(gb_moe_fp4_pass_rows) F(gb_moe_fp4_operand_bytes) F(gb_moe_fp4_rows) F(gb_moe_fp4_swiglu_rows) \
  F(gb_moe_gemv_fp4) F(gb_moe_gemm_fp4)

struct Lib {
#define GB_FN(name) decltype(&::name) name = nullptr;
  GB_ENTRIES(GB_FN)
#undef GB_FN
};
Lib L;

void bind(const std::string& path) {
  void* h = dlopen(path.c_str(), RTLD_NOW | RTLD_LOCAL);
  if (!h) throw std::runtime_error("cannot load " + path + ": " + dlerror());
#define GB_FN(name)                                              \
  L.name = reinterpret_cast<decltype(L.name)>(dlsym(h, #name));  \
  if (!L.name) throw std::runtime_error(path + " lacks the required symbol " #name);
  GB_ENTRIES(GB_FN)
#undef GB_FN
}

void check(int rc) {
  if (rc != GB_OK)
    throw std::runtime_error(std::string("gridbook_b200: ") + L.gb_last_error() + " (status " + std::to_string(rc) + ")");
}

using Opt = c10::optional<at::Tensor>;

// A weight as the kernels see it, and the tensors that keep its pointers valid.
struct Weight {
  gb_weight w{};
  int64_t expert_stride = 0, experts = 1;
  bool scales_e4m3 = false;      // two-tier: every composed scale is an exact E4M3 value
  std::vector<at::Tensor> keep;
  bool fp4() const { return w.fmt.grid == GB_GRID_FP4; }
  int act() const { return fp4() ? GB_ACT_FP4_GROUP16 : GB_ACT_FP8_TOKEN; }
};

Weight make_weight(const at::Tensor& qw, const at::Tensor& codebook, std::array<int, 6> fmt, int64_t K, int64_t rows,
                   int64_t row_stride, const Opt& off, const Opt& compose, const Opt& scale, double global_scale,
                   int64_t expert_stride, int64_t experts) {
  Weight r;
  r.w.qw = static_cast<const uint8_t*>(qw.data_ptr());
  r.w.row_stride = row_stride;
  r.w.codebook = codebook.data_ptr();
  r.keep = {qw, codebook};
  auto hold = [&](const Opt& t) -> void* {
    if (!t.has_value() || !t->defined()) return nullptr;
    r.keep.push_back(*t);
    return t->data_ptr();
  };
  r.w.cb_row_offset = static_cast<const int32_t*>(hold(off));
  r.w.compose = static_cast<const float*>(hold(compose));
  r.w.weight_scale = static_cast<const float*>(hold(scale));
  r.w.global_scale = (float)global_scale;
  r.w.rows = rows;
  r.w.K = K;
  r.w.fmt = {fmt[0], fmt[1], fmt[2], fmt[3], fmt[4], fmt[5]};
  r.expert_stride = expert_stride;
  r.experts = experts;
  if (r.w.fmt.scale_coding == GB_SCALE_V2) {               // looked at once, here: the kernels may then rely on it
    const c10::cuda::CUDAGuard guard(qw.device());
    at::Tensor flag = at::empty({1}, qw.options().dtype(at::kInt));
    check(L.gb_scales_e4m3(&r.w, experts * rows, flag.data_ptr<int32_t>(), c10::cuda::getCurrentCUDAStream().stream()));
    r.scales_e4m3 = flag.item<int32_t>() == 0;
  }
  return r;
}

// Everything one forward needs between its kernels, cut from a single allocation.
struct Arena {
  std::vector<int64_t> at;
  int64_t total = 0;
  at::Tensor buf;
  uint8_t* base = nullptr;
  int add(int64_t bytes) {
    at.push_back(total);
    total += (bytes + 255) & ~int64_t(255);
    return (int)at.size() - 1;
  }
  void alloc(const at::Tensor& like) {
    buf = at::empty({total > 0 ? total : 1}, like.options().dtype(at::kByte));
    base = static_cast<uint8_t*>(buf.data_ptr());
  }
  template <typename T = void>
  T* ptr(int i) const { return reinterpret_cast<T*>(base + at[i]); }
};

void need_cuda(const at::Tensor& t) {
  if (!t.is_cuda()) throw std::runtime_error("gridbook_b200 kernels take CUDA tensors only (no CPU path exists)");
}

void need_bf16(const at::Tensor& t, const char* what) {
  if (t.scalar_type() != at::kBFloat16) throw py::type_error(std::string(what) + " takes bf16 activations");
}

bool capturing() { return c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None; }

// A tensor that later calls read too, and the kernels that filled it.  Not made under capture: they would be
// recorded instead of run, and a call outside the graph would find the tensor unfilled.
struct Kept {
  at::Tensor t;
  c10::cuda::CUDAStream stream;
  at::cuda::CUDAEvent filled;
  explicit Kept(at::Tensor tensor) : t(std::move(tensor)), stream(c10::cuda::getCurrentCUDAStream()) { filled.record(stream); }
  // for the current stream; what a capture starts from has run
  const at::Tensor& ready() {
    const auto now = c10::cuda::getCurrentCUDAStream();
    if (now != stream && !capturing()) filled.block(now);
    return t;
  }
};

// A number that the runtime gives no second stream, as it may a handle; 0 under capture.  The default stream, which is never
// captured, is told without asking the runtime (two calls, 0.25 of the 7.2 us of a 4096 x 4096 row).
unsigned long long number_of(cudaStream_t stream) {
  if (stream == nullptr) return ~0ull;
  if (capturing()) return 0;
  unsigned long long id = 0;
  C10_CUDA_CHECK(cudaStreamGetId(stream, &id));
  return id + 1;
}

// Armed slots of the table kernel (gb_gemv_tab): calls that may overlap on the GPU need a buffer each, so every stream has
// its own.  Graphs have one more, armed outside any capture, for a replay may run beside eager calls; replays of graphs
// that hold the same layers must not overlap.
struct ArmedSlots {
  static constexpr size_t kMostStreams = 8;        // past these, and for a set whose first call is captured: armed on each call
  std::mutex mutex;
  at::Tensor captured;
  std::vector<std::pair<unsigned long long, at::Tensor>> of_stream;

  static at::Tensor armed(int64_t bytes, const at::Tensor& like) { return at::full({bytes}, 0xFF, like.options().dtype(at::kByte)); }
  at::Tensor get(int64_t bytes, const at::Tensor& like, cudaStream_t stream) {
    const unsigned long long id = number_of(stream);
    std::lock_guard<std::mutex> lock(mutex);
    if (id == 0) return captured.defined() ? captured : armed(bytes, like);
    if (!captured.defined()) captured = armed(bytes, like);
    for (const auto& s : of_stream)
      if (s.first == id) return s.second;
    at::Tensor t = armed(bytes, like);
    if (of_stream.size() < kMostStreams) of_stream.emplace_back(id, t);
    return t;
  }
};

constexpr int64_t kDecodeMaxRows = 16;
// Routed rows per expert from which a stack is decoded once into its NVFP4 view and multiplied by the grouped GEMM,
// instead of decoded in every pass of up to 64 rows.  The larger an expert, the later: its decoded copy is written
// and read once whatever the rows, while the passes lose less to their hand-overs.  Whole layer, us, passes / once,
// literal and K16: hidden 1024, intermediate 512, 64 experts, 112 rows 109 / 108, 117 / 115; 2048 x 768, 128 experts,
// 128 rows 400 / 400, 431 / 431; 2048 x 1536, 32 experts, 144 rows 209 / 201, 231 / 217; 4096 x 1536, 64 experts,
// 208 rows 800 / 831, 883 / 876; 7168 x 2048, 32 experts, 128 rows 510 / 705, 572 / 768 and 320 rows 1108 / 1197,
// 1279 / 1296; 4096 x 4096, 16 experts, 352 rows 700 / 735, 849 / 779.
// K20 and K24 hold one superblock per raw stage, take 16 rows a pass and cross over earlier and alike: 16 rows 306 / 312
// (2048 x 768), 467 / 580 (7168 x 2048), 95 / 95 (1024 x 512), 24 rows 365 / 320, 571 / 580, 108 / 99.
int64_t fp4_gemm_min_rows(const gb_weight& w, int64_t expert_weights) {
  return w.fmt.k_bits >= 20 ? 20 : 100 + expert_weights / 65536;
}
constexpr float kNvfp4ActRange = 448.0f;      // a row's largest group scale factor: the top of the UE4M3 range

// Routes a plan has taken, reported to the host code by number.
enum { kRouteNone = 0, kRouteNvfp4 = 1, kRouteBf16 = 2, kRouteFp8 = 3 };
enum { kMoePrefill = 1, kMoeSorted = 2, kMoePairs = 3, kMoeGrouped = 4 };

struct LinearPlan : std::enable_shared_from_this<LinearPlan> {
  Weight w;
  // Scratch of decode calls on the stream that loaded the layer, one call at a time; elsewhere, and in a graph, where it may
  // be another call's at the same time, a call brings its own.
  at::Tensor workspace;
  unsigned long long home = 0;
  bool tables = false;                             // the table kernel takes the layer
  ArmedSlots slots;
  int64_t row_batch_max = 16;
  gb_hints hints{};
  std::atomic<int> prefill_route{kRouteNone};
  const int64_t serial = next_serial++;            // never given twice, as an address is
  std::mutex mutex, scratch_mutex;
  std::map<std::vector<int64_t>, ArmedSlots> shared_slots;   // by the serials of the plans that share a row
  static std::atomic<int64_t> next_serial;

  // `role_rows`: row counts of the parts with a codebook of their own (empty: one codebook)
  LinearPlan(Weight weight, at::Tensor ws, const Opt& armed, const std::vector<int64_t>& role_rows)
      : w(std::move(weight)), workspace(std::move(ws)) {
    hints.scales_e4m3 = w.scales_e4m3 ? 1 : 0;
    if (role_rows.size() <= GB_MAX_ROLES) {                // more parts than that: the per-row offsets alone speak
      hints.n_roles = (int32_t)role_rows.size();
      for (size_t i = 0; i < role_rows.size(); ++i) hints.role_rows[i] = role_rows[i];
    }
    if (workspace.defined() && workspace.is_cuda()) home = number_of(c10::cuda::getCurrentCUDAStream(workspace.get_device()));
    if (armed.has_value() && armed->defined()) {
      const c10::cuda::CUDAGuard guard(armed->device());
      slots.of_stream.emplace_back(number_of(c10::cuda::getCurrentCUDAStream()), *armed);
      slots.captured = ArmedSlots::armed(armed->numel(), *armed);
      tables = true;
    }
    row_batch_max = L.gb_gemv_row_batch_max(&w.w);
  }

  at::Tensor forward(const at::Tensor& x, int rule, bool nvfp4, int64_t midm_max) {
    const int64_t N = w.w.rows, K = w.w.K;
    if (x.dim() < 1) throw std::runtime_error("activations are rows of " + std::to_string(K) + " values, got a scalar");
    std::vector<int64_t> shape(x.sizes().begin(), x.sizes().end());
    int64_t M = 1;
    for (size_t i = 0; i + 1 < shape.size(); ++i) M *= shape[i];
    // the output has M rows: an input of another width, whatever its element count, would make the kernels write others
    if (M > 0 && shape.back() != K)
      throw std::runtime_error("activations are rows of " + std::to_string(K) + " values, got rows of " + std::to_string(shape.back()));
    need_cuda(x);
    shape.back() = N;
    if (M == 0) return at::empty(shape, x.options());
    need_bf16(x, "the codebook linear");
    const c10::cuda::CUDAGuard guard(x.device());
    const cudaStream_t stream = c10::cuda::getCurrentCUDAStream().stream();
    const at::Tensor xc = x.is_contiguous() ? x : x.contiguous();
    at::Tensor out = at::empty(shape, x.options());
    if (M == 1 && tables) {
      const gb_weight* ws[1] = {&w.w};
      void* ys[1] = {out.data_ptr()};
      const at::Tensor armed = slots.get(L.gb_gemv_tab_slots_bytes(ws, 1), x, stream);
      const int rc = L.gb_gemv_tab(xc.data_ptr(), ws, ys, 1, w.act(), rule, armed.data_ptr(), armed.numel(), stream);
      if (rc == GB_OK) return out;
      if (rc != GB_EUNSUPPORTED) check(rc);
    }
    if (M <= kDecodeMaxRows || M <= std::min(midm_max, row_batch_max)) {
      const int64_t need = L.gb_gemv_hinted_workspace_bytes(M, N, K);
      at::Tensor ws;
      std::unique_lock<std::mutex> lock(scratch_mutex, std::defer_lock);
      if (workspace.defined() && workspace.numel() >= need && home != 0 && number_of(stream) == home) {
        lock.lock();                                       // until both launches of the call are on the stream
        ws = workspace;
      } else {
        ws = at::empty({need}, x.options().dtype(at::kByte));
      }
      check(L.gb_gemv_hinted(xc.data_ptr(), M, &w.w, &hints, rule, out.data_ptr(), ws.data_ptr(), ws.numel(), stream));
      return out;
    }
    prefill(xc, M, out, rule, nvfp4, stream);
    return out;
  }

  // M > 16: the layer is expanded once into a transient decoded operand and multiplied on the tensor
  // cores.  fp4 grid: native NVFP4 activations x the native NVFP4 view of the layer, block-scaled MMA
  // (the reference's fused FP4 prefill lane, gridbook/csrc/cb_fused_fp4_gemm.cu:758-903; its
  // activation bucket is NOT the decode contract's), or with nvfp4 off the decode contract kept:
  // bucketed bf16 rows x bf16(value * scale) (gridbook/linear.py:983-1023,1146-1152).  fp8 grid:
  // per-token E4M3 activations x the E4M3 value plane, both scales on the fp32 accumulator
  // (gridbook/linear.py:1221-1264; epilogue of gridbook/csrc/cb_fused_gemm.cu:476-486).
  void prefill(const at::Tensor& x, int64_t M, at::Tensor& out, int rule, bool nvfp4, void* stream) {
    const int64_t N = w.w.rows, K = w.w.K;
    Arena a;
    if (w.fp4() && nvfp4) {
      const int qa = a.add(M * K / 2), sa = a.add(L.gb_nvfp4_sf_bytes(M, K)), as = a.add(M * 4);
      const int qb = a.add(N * K / 2), sb = a.add(L.gb_nvfp4_sf_bytes(N, K));
      a.alloc(x);
      check(L.gb_nvfp4_quantize_rows(x.data_ptr(), M, K, kNvfp4ActRange, a.ptr(qa), a.ptr(sa), a.ptr<float>(as), stream));
      // scale factors of the rows past N stay unset: they only reach columns that are not stored
      check(L.gb_expand_fp4_nvfp4_beside(&w.w, 0, N, a.ptr(qb), a.ptr(sb), 2, stream));
      check(L.gb_gemm_fp4(a.ptr(qa), a.ptr(sa), a.ptr(qb), a.ptr(sb), out.data_ptr(), M, N, K, a.ptr<float>(as),
                          w.w.global_scale, stream));
      prefill_route = kRouteNvfp4;
    } else if (w.fp4()) {
      const int xq = a.add(M * K * 2), wt = a.add(N * K * 2);
      a.alloc(x);
      check(L.gb_fp4_act_qdq(x.data_ptr(), a.ptr(xq), M, K, rule, stream));
      check(L.gb_expand_fp4_bf16(&w.w, 0, N, a.ptr(wt), stream));
      check(L.gb_gemm_tn(a.ptr(xq), a.ptr(wt), out.data_ptr(), M, N, K, GB_GEMM_BF16, nullptr, nullptr, w.w.global_scale, stream));
      prefill_route = kRouteBf16;
    } else {
      const int q = a.add(M * K), as = a.add(M * 4), wt = a.add(N * K);
      a.alloc(x);
      check(L.gb_fp8_quantize_rows(x.data_ptr(), a.ptr(q), a.ptr<float>(as), M, K, rule, stream));
      check(L.gb_expand_fp8_beside(&w.w, 0, N, a.ptr(wt), stream));
      check(L.gb_gemm_tn(a.ptr(q), a.ptr(wt), out.data_ptr(), M, N, K, GB_GEMM_E4M3, a.ptr<float>(as), w.w.weight_scale,
                         w.w.global_scale, stream));
      prefill_route = kRouteFp8;
    }
  }
};

std::atomic<int64_t> LinearPlan::next_serial{0};

// Whether a layer's prefill of the fp4 grid quantises its rows to NVFP4, and its largest decode batch.
using Route = std::pair<bool, int64_t>;

// Several linears that read the same rows: the rows are bucketed or quantised once, and the decode batches of the fp4 formats
// go out as one launch (two layers of K16 at 16 rows 137 -> 127 us, one literal layer at 64 rows 91 -> 81).  None: one by one.
py::object shared_rows(const std::vector<std::shared_ptr<LinearPlan>>& plans, const at::Tensor& x, int rule, const std::vector<Route>& routes) {
  const size_t n = plans.size();
  const int64_t K = plans[0]->w.w.K, M = x.numel() / K;
  if (x.size(-1) != K || M < 1 || routes.size() != n || x.scalar_type() != at::kBFloat16) return py::none();
  bool decode = true, prefill = true;
  for (size_t i = 0; i < n; ++i) {
    const LinearPlan& p = *plans[i];
    if (p.w.w.K != K || p.w.fp4() != plans[0]->w.fp4() || routes[i].first != routes[0].first) return py::none();
    const bool few = M <= kDecodeMaxRows || M <= std::min(routes[i].second, p.row_batch_max);
    decode = decode && few && p.hints.n_roles <= 1 && p.w.w.cb_row_offset == nullptr && p.w.scales_e4m3 == plans[0]->w.scales_e4m3;
    prefill = prefill && !few;
  }
  const bool fp4 = plans[0]->w.fp4();
  if (!decode && !(prefill && (routes[0].first || !fp4))) return py::none();
  // decided before anything is allocated: layers that go one by one allocate again
  const gb_weight* ws[4];
  for (size_t i = 0; i < n; ++i) ws[i] = &plans[i]->w.w;
  // rows off the vector alignment (as they lie: a copy starts on it) are the layers' to take or to refuse
  if (x.is_contiguous() && ((uintptr_t)x.data_ptr() & 15u) != 0) return py::none();
  if (decode && fp4 && L.gb_gemv_shared_applies(ws, (int)n, plans[0]->w.scales_e4m3 ? 1 : 0) == 0) return py::none();
  const c10::cuda::CUDAGuard guard(x.device());
  void* stream = c10::cuda::getCurrentCUDAStream().stream();
  const at::Tensor xc = x.is_contiguous() ? x : x.contiguous();
  void* ys[4];
  std::vector<at::Tensor> outs;
  for (size_t i = 0; i < n; ++i) {
    std::vector<int64_t> shape(x.sizes().begin(), x.sizes().end());
    shape.back() = plans[i]->w.w.rows;
    outs.push_back(at::empty(shape, x.options()));
    ys[i] = outs.back().data_ptr();
  }
  Arena a;
  if (decode && fp4) {
    const int scratch = a.add(L.gb_gemv_hinted_workspace_bytes(M, ws[0]->rows, K));
    a.alloc(xc);
    const int rc = L.gb_gemv_shared(xc.data_ptr(), M, ws, (int)n, plans[0]->w.scales_e4m3 ? 1 : 0, rule, ys, a.ptr(scratch),
                                    L.gb_gemv_hinted_workspace_bytes(M, ws[0]->rows, K), stream);
    if (rc == GB_EUNSUPPORTED) return py::none();
    check(rc);
  } else if (decode) {
    int64_t need = 0;
    for (size_t i = 0; i < n; ++i) need = std::max(need, L.gb_gemv_hinted_workspace_bytes(M, ws[i]->rows, K));
    const int xq = a.add(M * K * 2), scratch = a.add(need);
    a.alloc(xc);
    check(L.gb_fp8_act_qdq(xc.data_ptr(), a.ptr(xq), M, K, rule, stream));
    for (size_t i = 0; i < n; ++i) check(L.gb_gemv(a.ptr(xq), M, ws[i], GB_ACT_NONE, rule, ys[i], a.ptr(scratch), need, stream));
  } else {
    const int q = a.add(fp4 ? M * K / 2 : M * K), sf = a.add(fp4 ? L.gb_nvfp4_sf_bytes(M, K) : 0), as = a.add(M * 4);
    // one decoded copy at a time, in the place of the largest: multiplied while it lies in L2, and no more memory than one by one
    int64_t rows = 0;
    for (size_t i = 0; i < n; ++i) rows = std::max(rows, ws[i]->rows);
    const int wq = a.add(fp4 ? rows * K / 2 : rows * K), wsf = a.add(fp4 ? L.gb_nvfp4_sf_bytes(rows, K) : 0);
    a.alloc(xc);
    if (fp4) check(L.gb_nvfp4_quantize_rows(xc.data_ptr(), M, K, kNvfp4ActRange, a.ptr(q), a.ptr(sf), a.ptr<float>(as), stream));
    else check(L.gb_fp8_quantize_rows(xc.data_ptr(), a.ptr(q), a.ptr<float>(as), M, K, rule, stream));
    for (size_t i = 0; i < n; ++i) {                       // the first expander right behind the quantiser, beside it
      if (fp4) {
        check((i == 0 ? L.gb_expand_fp4_nvfp4_beside : L.gb_expand_fp4_nvfp4)(ws[i], 0, ws[i]->rows, a.ptr(wq), a.ptr(wsf), 2, stream));
        check(L.gb_gemm_fp4(a.ptr(q), a.ptr(sf), a.ptr(wq), a.ptr(wsf), ys[i], M, ws[i]->rows, K, a.ptr<float>(as), ws[i]->global_scale, stream));
      } else {
        check((i == 0 ? L.gb_expand_fp8_beside : L.gb_expand_fp8)(ws[i], 0, ws[i]->rows, a.ptr(wq), stream));
        check(L.gb_gemm_tn(a.ptr(q), a.ptr(wq), ys[i], M, ws[i]->rows, K, GB_GEMM_E4M3, a.ptr<float>(as), ws[i]->weight_scale,
                           ws[i]->global_scale, stream));
      }
      plans[i]->prefill_route = fp4 ? kRouteNvfp4 : kRouteFp8;
    }
  }
  return py::cast(outs);
}

// Several linears that read the same activation row, one launch; None when they have no such kernel.  `routes`: called for the
// layers' routes where their calls may be replaced by more than the table kernel; none or empty: they may not.
py::object shared_row(const std::vector<std::shared_ptr<LinearPlan>>& plans, const at::Tensor& x, int rule, const py::object& routes) {
  const size_t n = plans.size();
  if (n < 2 || n > 4 || !x.is_cuda() || x.dim() < 1) return py::none();
  const int64_t K = plans[0]->w.w.K;
  bool tables = x.numel() == K;
  for (const auto& p : plans) tables = tables && p->tables;
  if (!tables) return routes.is_none() ? py::none() : shared_rows(plans, x, rule, routes().cast<std::vector<Route>>());
  if (x.numel() != K || x.size(-1) != K) return py::none();   // another width: refused where the layers are called one by one
  for (const auto& p : plans)
    if (!p->tables || p->w.w.K != K) return py::none();
  need_bf16(x, "the table GEMV");
  const c10::cuda::CUDAGuard guard(x.device());
  const gb_weight* ws[4];
  void* ys[4];
  std::vector<int64_t> key;
  for (size_t i = 0; i < n; ++i) {
    ws[i] = &plans[i]->w.w;
    key.push_back(plans[i]->serial);
  }
  ArmedSlots* kept;
  {
    std::lock_guard<std::mutex> lock(plans[0]->mutex);
    kept = &plans[0]->shared_slots[key];                   // a node of the map: it stays where it is
  }
  const cudaStream_t stream = c10::cuda::getCurrentCUDAStream().stream();
  const at::Tensor slots = kept->get(L.gb_gemv_tab_slots_bytes(ws, (int)n), x, stream);
  const at::Tensor xc = x.is_contiguous() ? x : x.contiguous();
  std::vector<at::Tensor> outs;
  for (size_t i = 0; i < n; ++i) {
    std::vector<int64_t> shape(x.sizes().begin(), x.sizes().end());
    shape.back() = ws[i]->rows;
    outs.push_back(at::empty(shape, x.options()));
    ys[i] = outs.back().data_ptr();
  }
  const int rc = L.gb_gemv_tab(xc.data_ptr(), ws, ys, (int)n, plans[0]->w.act(), rule, slots.data_ptr(), slots.numel(), stream);
  if (rc == GB_EUNSUPPORTED) return py::none();
  check(rc);
  return py::cast(outs);
}

struct MoEPlan {
  Weight w13, w2;
  Weight rows13, rows2;          // the stacks seen as one matrix of E * rows rows (for the expanders)
  int64_t E, hidden, inter;
  bool sorted13, sorted2, pair_ok;   // per projection: a kernel that takes rows in expert order
  std::atomic<int> route{kRouteNone};
  std::mutex mutex;
  std::map<int64_t, std::vector<Kept>> x_rows;   // per top-k, each at least twice the last: a batch reads the front of one

  MoEPlan(Weight a, Weight b, Weight ra, Weight rb, int64_t E_, int64_t hidden_, int64_t inter_, bool sorted_13, bool sorted_2, bool pair_)
      : w13(std::move(a)), w2(std::move(b)), rows13(std::move(ra)), rows2(std::move(rb)), E(E_), hidden(hidden_),
        inter(inter_), sorted13(L.gb_moe_fp4_pass_rows(&w13.w, w13.scales_e4m3, 1, E_) > 0 || sorted_13),
        sorted2(L.gb_moe_fp4_pass_rows(&w2.w, w2.scales_e4m3, 1, E_) > 0 || sorted_2), pair_ok(pair_) {}

  // both projections on the block-scaled FP4 tensor cores
  bool fp4() const {
    return L.gb_moe_fp4_pass_rows(&w13.w, w13.scales_e4m3, 1, E) > 0 && L.gb_moe_fp4_pass_rows(&w2.w, w2.scales_e4m3, 1, E) > 0;
  }

  // Token of every routed pair.  Earlier, shorter tensors stay: a captured graph may read them.
  at::Tensor x_row(int64_t T, int64_t topk, const at::Tensor& like) {
    auto make = [&](int64_t pairs) { return at::arange(pairs, like.options().dtype(at::kInt)).floor_divide(topk).to(at::kInt).contiguous(); };
    std::lock_guard<std::mutex> lock(mutex);
    std::vector<Kept>& kept = x_rows[topk];
    for (Kept& k : kept)
      if (k.t.numel() >= T * topk) return k.ready();
    if (capturing()) return make(T * topk);
    kept.emplace_back(make(std::max(T * topk, kept.empty() ? 64 * topk : 2 * kept.back().t.numel())));
    return kept.back().t;
  }

  struct Limits { int64_t pair_max, sorted_per_expert, sorted_other, prefill_per_expert, prefill_other, fused_bucket_max; };

  at::Tensor forward(const at::Tensor& x, const at::Tensor& topk_weights, const at::Tensor& topk_ids, int rule,
                     std::array<int64_t, 6> limits) {
    const Limits lim{limits[0], limits[1], limits[2], limits[3], limits[4], limits[5]};
    // the kernels take their extents from the ids: everything else has to fit them
    if (topk_ids.dim() != 2) throw std::runtime_error("routed layer: expert ids of shape [tokens, top-k] expected");
    const int64_t T = topk_ids.size(0), topk = topk_ids.size(1);
    if (T > 0 && x.numel() != T * hidden) throw std::runtime_error("routed layer: " + std::to_string(T) + " tokens of " +
                                                                   std::to_string(hidden) + " values expected");
    if (topk_weights.numel() != T * topk) throw std::runtime_error("routed layer: " + std::to_string(T) + " x " + std::to_string(topk) +
                                                                   " router weights expected");
    need_cuda(x);
    need_cuda(topk_ids);
    need_cuda(topk_weights);
    if (T == 0) return at::empty_like(x);
    const c10::cuda::CUDAGuard guard(x.device());
    Call c;
    c.x = x.to(at::kBFloat16).contiguous();
    if (((uintptr_t)c.x.data_ptr() & 15u) != 0) c.x = c.x.clone();   // a view into the middle of another tensor
    c.ids = topk_ids.to(at::kInt).contiguous();
    c.tw = topk_weights.to(at::kFloat).contiguous();
    c.T = T; c.topk = topk; c.P = T * topk; c.rule = rule;
    c.stream = c10::cuda::getCurrentCUDAStream().stream();
    c.out = at::empty({T, hidden}, c.x.options());
    c.plan = this;
    const bool sorted_ok = sorted13 && sorted2;
    const int64_t prefill_min = sorted_ok ? lim.prefill_per_expert : std::min(lim.prefill_per_expert, lim.prefill_other);
    if (c.P >= prefill_min * E) prefill(c);
    else if (sorted_ok && c.P >= (pair_ok ? lim.sorted_per_expert * E : lim.sorted_other)) sorted(c);
    else if (!(c.P <= lim.pair_max && w13.fp4() && w2.fp4() && pairs(c))) grouped(c, c.P <= lim.fused_bucket_max);
    at::Tensor out = c.out;
    if (x.scalar_type() != at::kBFloat16) out = out.to(x.scalar_type());
    return out.reshape(x.sizes());
  }

 private:
  struct Call {
    at::Tensor x, ids, tw, out, tokens;
    MoEPlan* plan;
    const int32_t* x_row() {
      if (!tokens.defined()) tokens = plan->x_row(T, topk, x);
      return tokens.data_ptr<int32_t>();
    }
    int64_t T, topk, P;
    int rule;
    void* stream;
  };

  struct Routing { int counts, offsets, order, inv, pair_w, ws; int64_t ws_bytes; };
  Routing plan_routing(Arena& a, const Call& c) const {
    Routing r;
    r.counts = a.add(E * 4);
    r.offsets = a.add((E + 1) * 4);
    r.order = a.add(c.P * 4);
    r.inv = a.add(c.P * 4);
    r.pair_w = a.add(c.P * 4);
    r.ws_bytes = L.gb_moe_route_workspace_bytes(c.T, c.topk, E);
    r.ws = a.add(r.ws_bytes);
    return r;
  }
  void run_routing(const Arena& a, const Routing& r, const Call& c) const {
    check(L.gb_moe_route_inv(c.ids.data_ptr<int32_t>(), c.T, c.topk, E, 0, a.ptr<int32_t>(r.counts), a.ptr<int32_t>(r.offsets),
                             a.ptr<int32_t>(r.order), a.ptr<int32_t>(r.inv), c.tw.data_ptr<float>(), a.ptr<float>(r.pair_w),
                             r.ws_bytes ? a.ptr(r.ws) : nullptr, r.ws_bytes, c.stream));
  }
  static void bucket(const Weight& w, const void* in, void* out, int64_t rows, const Call& c) {
    check(w.fp4() ? L.gb_fp4_act_qdq(in, out, rows, w.w.K, c.rule, c.stream)
                  : L.gb_fp8_act_qdq(in, out, rows, w.w.K, c.rule, c.stream));
  }
  void combine(const void* y, const float* pair_w, const Call& c, bool round) const {
    check(L.gb_moe_combine(y, pair_w, c.ids.data_ptr<int32_t>(), E, c.T, c.topk, hidden, round ? 1 : 0, c.out.data_ptr(),
                           c.stream));
  }

  // Small batches of the literal format: every routed pair is its own M = 1 linear through the
  // inner-product-table kernel (bucket fused; the down projection sums the gate/up K slices and
  // applies SwiGLU while it stages its rows), then the combine.  False when there is no such kernel.
  bool pairs(Call& c) {
    if (!pair_ok) return false;
    Arena a;
    const int64_t need = L.gb_moe_mlp_pairs_workspace_bytes(c.P, w13.w.K, w2.w.K);
    const int y = a.add(c.P * hidden * 2), ws = a.add(need);
    a.alloc(c.x);
    const int rc = L.gb_moe_mlp_pairs(c.x.data_ptr(), c.x_row(), &w13.w, w13.expert_stride, &w2.w,
                                      w2.expert_stride, E, 0, c.ids.data_ptr<int32_t>(), c.P, 0, GB_ACT_FP4_GROUP16, c.rule,
                                      a.ptr(y), nullptr, a.ptr(ws), std::max<int64_t>(need, 16), c.stream);
    if (rc == GB_EUNSUPPORTED) return false;
    check(rc);
    combine(a.ptr(y), c.tw.data_ptr<float>(), c, true);
    route = kMoePairs;
    return true;
  }

  // Route -> bucket -> grouped gate/up GEMV with SwiGLU -> bucket -> grouped down GEMV -> combine.  Any
  // format and token count: an expert's tokens are taken in passes of up to sixteen rows, its weights
  // stream once per pass.  `fuse`: the fp4 bucket runs inside the grouped kernel while it stages the
  // rows (two launches fewer for small batches; for large ones every row tile would repeat it).
  void grouped(Call& c, bool fuse) {
    Arena a;
    const Routing r = plan_routing(a, c);
    const bool fuse13 = fuse && w13.fp4(), fuse2 = fuse && w2.fp4();
    const int xq = a.add(fuse13 ? 0 : c.T * hidden * 2), h = a.add(c.P * inter * 2);
    const int hq = a.add(fuse2 ? 0 : c.P * inter * 2), y = a.add(c.P * hidden * 2);
    a.alloc(c.x);
    run_routing(a, r, c);
    const int32_t *off = a.ptr<int32_t>(r.offsets), *ord = a.ptr<int32_t>(r.order);
    const void* in = c.x.data_ptr();
    if (!fuse13) {
      bucket(w13, in, a.ptr(xq), c.T, c);
      in = a.ptr(xq);
    }
    check(L.gb_moe_gemv(in, c.x_row(), &w13.w, w13.expert_stride, E, off, ord, c.P, 1,
                        fuse13 ? GB_ACT_FP4_GROUP16 : GB_ACT_NONE, c.rule, a.ptr(h), nullptr, nullptr, 0, c.stream));
    in = a.ptr(h);
    if (!fuse2) {
      bucket(w2, in, a.ptr(hq), c.P, c);
      in = a.ptr(hq);
    }
    check(L.gb_moe_gemv(in, nullptr, &w2.w, w2.expert_stride, E, off, ord, c.P, 0,
                        fuse2 ? GB_ACT_FP4_GROUP16 : GB_ACT_NONE, c.rule, a.ptr(y), nullptr, nullptr, 0, c.stream));
    combine(a.ptr(y), a.ptr<float>(r.pair_w), c, false);
    route = kMoeGrouped;
  }

  // SwiGLU over the sorted rows and the down projection's bucket on top.
  void swiglu(const Arena& a, const Call& c, const Routing& r, int h13, int hs, int h) const {
    const int32_t* off = a.ptr<int32_t>(r.offsets);
    if (w2.fp4() && inter % 16 == 0) {
      check(L.gb_moe_swiglu_rows(a.ptr(h13), off, E, c.P, inter, GB_ACT_FP4_GROUP16, c.rule, a.ptr(h), c.stream));
      return;
    }
    check(L.gb_moe_swiglu_rows(a.ptr(h13), off, E, c.P, inter, GB_ACT_NONE, c.rule, a.ptr(hs), c.stream));
    bucket(w2, a.ptr(hs), a.ptr(h), c.P, c);
  }

  // The rows in expert order, then per projection one launch in which every (expert, 128-row tile)
  // decodes its packed rows into tensor memory and multiplies them with the expert's rows on the
  // tensor cores; the down projection stores its rows back in pair order.  A stack of the fp4 grid runs
  // on the block-scaled FP4 cores, its activations written as that kernel's operand in one launch (bucket
  // and gather, or SwiGLU and bucket); the others bucket to bf16 rows.  The two stacks may be of
  // different grids: each projection's rows go through its own grid's bucket.
  void sorted(Call& c) {
    Arena a;
    const Routing r = plan_routing(a, c);
    const int fp13 = L.gb_moe_fp4_pass_rows(&w13.w, w13.scales_e4m3, c.P, E), fp2 = L.gb_moe_fp4_pass_rows(&w2.w, w2.scales_e4m3, c.P, E);
    // decoded once and multiplied by the grouped GEMM (pass rows 0) where several passes would decode every weight again
    auto once = [&](const Weight& w, int fp) {
      return fp > 0 && E <= 1024 && c.P >= E * fp4_gemm_min_rows(w.w, hidden * inter);
    };
    const bool once13 = once(w13, fp13), once2 = once(w2, fp2);
    const int pr13 = once13 ? 0 : fp13, pr2 = once2 ? 0 : fp2;
    const int64_t flat13 = once13 ? E * w13.w.rows : 0, flat2 = once2 ? E * w2.w.rows : 0;
    const int wq = a.add(std::max(flat13 * w13.w.K, flat2 * w2.w.K) / 2);
    const int wsf = a.add(std::max(L.gb_nvfp4_sf_bytes(flat13, w13.w.K), L.gb_nvfp4_sf_bytes(flat2, w2.w.K)));
    const int64_t op13 = L.gb_moe_fp4_operand_bytes(c.P, E, hidden, pr13), op2 = L.gb_moe_fp4_operand_bytes(c.P, E, inter, pr2);
    const int xq = a.add(fp13 ? 0 : c.T * hidden * 2), xs = a.add(fp13 ? op13 : c.P * hidden * 2), h13 = a.add(c.P * 2 * inter * 2);
    const int hs = a.add(fp2 || w2.fp4() ? 0 : c.P * inter * 2), h = a.add(fp2 ? op2 : c.P * inter * 2), y = a.add(c.P * hidden * 2);
    a.alloc(c.x);
    run_routing(a, r, c);
    const int32_t *off = a.ptr<int32_t>(r.offsets), *ord = a.ptr<int32_t>(r.order), *ids = c.ids.data_ptr<int32_t>();
    auto multiply = [&](const Weight& w, const Weight& flat, bool once_w, int pr, int operand, const int32_t* map, void* to) {
      if (!once_w) {
        check(L.gb_moe_gemv_fp4(a.ptr(operand), &w.w, w.scales_e4m3, w.expert_stride, E, off, map, c.P, pr, to, c.stream));
        return;
      }
      check(L.gb_expand_fp4_nvfp4_beside(&flat.w, 0, flat.w.rows, a.ptr(wq), a.ptr(wsf), 2, c.stream));   // behind the rows' launch
      check(L.gb_moe_gemm_fp4(a.ptr(operand), a.ptr(wq), a.ptr(wsf), w.w.rows, w.w.K, E, off, map, c.P, w.w.global_scale, to, c.stream));
    };
    if (fp13) {
      check(L.gb_moe_fp4_rows(c.x.data_ptr(), ids, a.ptr<int32_t>(r.inv), off, c.T, c.topk, E, hidden, pr13, c.rule, a.ptr(xs), c.stream));
      multiply(w13, rows13, once13, pr13, xs, nullptr, a.ptr(h13));
    } else {
      bucket(w13, c.x.data_ptr(), a.ptr(xq), c.T, c);
      check(L.gb_moe_gather_rows(a.ptr(xq), c.x_row(), ord, off, E, c.P, hidden, a.ptr(xs), c.stream));
      check(L.gb_moe_gemv_sorted(a.ptr(xs), &w13.w, w13.expert_stride, E, off, nullptr, c.P, a.ptr(h13), nullptr, c.stream));
    }
    if (fp2) {
      check(L.gb_moe_fp4_swiglu_rows(a.ptr(h13), ids, ord, off, c.P, E, inter, pr2, c.rule, a.ptr(h), c.stream));
      multiply(w2, rows2, once2, pr2, h, ord, a.ptr(y));
    } else {
      swiglu(a, c, r, h13, hs, h);
      check(L.gb_moe_gemv_sorted(a.ptr(h), &w2.w, w2.expert_stride, E, off, ord, c.P, a.ptr(y), nullptr, c.stream));
    }
    combine(a.ptr(y), a.ptr<float>(r.pair_w), c, false);
    route = kMoeSorted;
  }

  // (Stacks that the FP4 cores take come here only when a caller has set the limit: their default is never.)
  // Many tokens per expert: each stack decoded once into a transient bf16 tile of the exact served
  // weights, one grouped tensor-core GEMM over the expert segments per projection - the reference's
  // grouped bf16 route (gridbook/moe.py:2388-2504 with gridbook/ops.py:137-306).  Both grids keep the
  // decode contract: the buckets between the two projections are coarse enough to turn a last-place
  // difference of the first projection into whole quantisation steps, so the fp8 grid does not take
  // the scales-in-the-epilogue E4M3 GEMM of the dense prefill.
  void prefill(Call& c) {
    Arena a;
    const Routing r = plan_routing(a, c);
    const int64_t tile13 = E * w13.w.rows * w13.w.K * 2, tile2 = E * w2.w.rows * w2.w.K * 2;
    const int tile = a.add(std::max(tile13, tile2));
    const int xq = a.add(c.T * hidden * 2), xs = a.add(c.P * hidden * 2), h13 = a.add(c.P * 2 * inter * 2);
    const int hs = a.add(w2.fp4() && inter % 16 == 0 ? 0 : c.P * inter * 2), h = a.add(c.P * inter * 2);
    const int y = a.add(c.P * hidden * 2);
    a.alloc(c.x);
    run_routing(a, r, c);
    const int32_t *off = a.ptr<int32_t>(r.offsets), *ord = a.ptr<int32_t>(r.order);
    auto stage = [&](const Weight& stack, const Weight& one, const void* in, void* out, const int32_t* map) {
      check(stack.fp4() ? L.gb_expand_fp4_bf16(&stack.w, 0, stack.w.rows, a.ptr(tile), c.stream)
                        : L.gb_expand_fp8_bf16(&stack.w, 0, stack.w.rows, a.ptr(tile), c.stream));
      check(L.gb_gemm_tn_grouped(in, a.ptr(tile), out, c.P, one.w.rows, one.w.K, GB_GEMM_BF16, E, off, map, nullptr, nullptr,
                                 one.w.global_scale, c.stream));
    };
    bucket(w13, c.x.data_ptr(), a.ptr(xq), c.T, c);
    check(L.gb_moe_gather_rows(a.ptr(xq), c.x_row(), ord, off, E, c.P, hidden, a.ptr(xs), c.stream));
    stage(rows13, w13, a.ptr(xs), a.ptr(h13), nullptr);
    swiglu(a, c, r, h13, hs, h);
    stage(rows2, w2, a.ptr(h), a.ptr(y), ord);             // rows back in pair order
    combine(a.ptr(y), a.ptr<float>(r.pair_w), c, false);
    route = kMoePrefill;
  }
};

}  // namespace

PYBIND11_MODULE(_gb_torch, m) {
  m.def("bind", &bind);
  m.def("abi_version", [] { return GB_ABI_VERSION; });
  py::class_<Weight>(m, "Weight").def(py::init(&make_weight));
  py::class_<LinearPlan, std::shared_ptr<LinearPlan>>(m, "LinearPlan")
      .def(py::init<Weight, at::Tensor, const Opt&, const std::vector<int64_t>&>())
      .def("__call__", &LinearPlan::forward, py::call_guard<py::gil_scoped_release>())
      .def_property_readonly("serial", [](const LinearPlan& p) { return p.serial; })
      .def_property_readonly("prefill_route", [](const LinearPlan& p) { return p.prefill_route.load(); });
  py::class_<MoEPlan, std::shared_ptr<MoEPlan>>(m, "MoEPlan")
      .def(py::init<Weight, Weight, Weight, Weight, int64_t, int64_t, int64_t, bool, bool, bool>())
      .def_property_readonly("fp4", &MoEPlan::fp4)
      .def("__call__", &MoEPlan::forward, py::call_guard<py::gil_scoped_release>())
      .def_property_readonly("route", [](const MoEPlan& p) { return p.route.load(); });
  m.def("shared_row", &shared_row, py::arg("plans"), py::arg("x"), py::arg("rule"), py::arg("routes") = py::none());
}
