// Python bindings: translate torch tensors into the raw tables the kernels consume.
// Kernels live in the .cu files and know nothing about torch; this file owns all torch-facing glue.
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/extension.h>

#include <ATen/MemoryOverlap.h>

#include <algorithm>
#include <optional>
#include <string>
#include <string_view>
#include <unordered_map>
#include <vector>

#include "chol_qr.h"
#include "colsum.h"
#include "cross_entropy.h"
#include "fused_chain.h"
#include "gelu.h"
#include "layer_norm.h"
#include "matrix_passes.h"
#include "ns_gemm.h"
#include "peer_sync.h"
#include "power_iteration.h"
#include "skinny.h"
#include "split16_gemm.h"
#include "tf32_gemm.h"

namespace py = pybind11;
using OptT = std::optional<at::Tensor>;
using TList = std::vector<OptT>;

namespace {

void check(cudaError_t e, const char* what) {
  TORCH_CHECK(e == cudaSuccess, what, ": ", cudaGetErrorString(e));
}

void* ptr_or_null(const TList& l, size_t i) {
  if (l.empty() || !l[i].has_value() || !l[i]->defined()) return nullptr;
  return l[i]->data_ptr();
}

bool aligned16(const void* p) { return p == nullptr || (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

struct Table {
  at::Tensor device_blob;  // metas followed by the chunk prefix
  const hb::TensorMeta* metas;
  const int* prefix;
  int total_chunks;
  int n;
  int chunk;
};

std::vector<int> chunk_prefix(const std::vector<hb::TensorMeta>& metas, int chunk) {
  std::vector<int> prefix(metas.size() + 1, 0);
  for (size_t i = 0; i < metas.size(); ++i) prefix[i + 1] = prefix[i] + (int)((metas[i].numel + chunk - 1) / chunk);
  return prefix;
}

// The settings of a fused-chain launch, collected in one walk over the dict (a lookup by name builds a string object each time, and
// there are forty of them).
struct ChainConfig {
  enum Key { algo, out_mode, n_state, dt_p, dt_g, dt_u, dt_s, u_is_input, mars, cautious_wd, caution_apply, use_tensor_scale, accum_sumsq, u_op,
             post_state, g_clip_mode, g_clip_at, g_clip_numel, lr, wd, eps, b1, b2, b3, alpha, mars_a, seed, g_delta, g_scale, p_delta, g_mc_delta,
             p_mc_delta, count_caution, scale_stride, gsq_stride, kKeys };
  py::handle values[kKeys];
  explicit ChainConfig(const py::dict& cfg) {
    static const std::unordered_map<std::string_view, int> index = {
        {"algo", algo}, {"out_mode", out_mode}, {"n_state", n_state}, {"dt_p", dt_p}, {"dt_g", dt_g}, {"dt_u", dt_u}, {"dt_s", dt_s},
        {"u_is_input", u_is_input}, {"mars", mars}, {"cautious_wd", cautious_wd}, {"caution_apply", caution_apply},
        {"use_tensor_scale", use_tensor_scale}, {"accum_sumsq", accum_sumsq}, {"u_op", u_op}, {"post_state", post_state},
        {"g_clip_mode", g_clip_mode}, {"g_clip_at", g_clip_at}, {"g_clip_numel", g_clip_numel}, {"lr", lr}, {"wd", wd}, {"eps", eps}, {"b1", b1},
        {"b2", b2}, {"b3", b3}, {"alpha", alpha}, {"mars_a", mars_a}, {"seed", seed}, {"g_delta", g_delta}, {"g_scale", g_scale},
        {"p_delta", p_delta}, {"g_mc_delta", g_mc_delta}, {"p_mc_delta", p_mc_delta}, {"count_caution", count_caution},
        {"scale_stride", scale_stride}, {"gsq_stride", gsq_stride}};
    for (const auto& item : cfg) {
      Py_ssize_t len = 0;
      const char* name = PyUnicode_AsUTF8AndSize(item.first.ptr(), &len);
      if (name == nullptr) throw py::error_already_set();
      const auto it = index.find(std::string_view(name, (size_t)len));
      if (it != index.end()) values[it->second] = item.second;
    }
  }
  bool has(Key k) const { return values[k].ptr() != nullptr; }
  template <class T>
  T get(Key k, T otherwise) const { return has(k) ? values[k].cast<T>() : otherwise; }
  int i(Key k) const { return get<int>(k, 0); }
  float f(Key k) const { return get<float>(k, 0.f); }
};

// Builds the per-tensor table and uploads it with one async copy on the current stream.
Table upload(std::vector<hb::TensorMeta>& metas, const at::Device& dev, int chunk = hb::chain_chunk_elems()) {
  const int n = (int)metas.size();
  const std::vector<int> prefix = chunk_prefix(metas, chunk);
  const size_t meta_bytes = sizeof(hb::TensorMeta) * n, prefix_bytes = sizeof(int) * (n + 1);
  std::vector<uint8_t> host(meta_bytes + prefix_bytes);
  memcpy(host.data(), metas.data(), meta_bytes);
  memcpy(host.data() + meta_bytes, prefix.data(), prefix_bytes);
  Table t;
  t.device_blob = at::empty({(int64_t)host.size()}, at::TensorOptions().dtype(at::kByte).device(dev));
  auto stream = at::cuda::getCurrentCUDAStream();
  check(cudaMemcpyAsync(t.device_blob.data_ptr(), host.data(), host.size(), cudaMemcpyHostToDevice, stream), "table upload");
  t.metas = reinterpret_cast<const hb::TensorMeta*>(t.device_blob.data_ptr());
  t.prefix = reinterpret_cast<const int*>((uint8_t*)t.device_blob.data_ptr() + meta_bytes);
  t.total_chunks = prefix[n];
  t.n = n;
  t.chunk = chunk;
  return t;
}

}  // namespace

// One fused pass over a param group.  Every list is either empty or has one entry per tensor.
// `cfg`: algo, out_mode, n_state, dt_p, dt_g, dt_u, dt_s, u_is_input, mars, cautious_wd, caution_apply,
// use_tensor_scale, count_caution (ints); lr, wd, eps, b1, b2, b3, alpha, mars_a (floats); seed.
void fused_chain(const TList& p, const TList& pe, const TList& g, const TList& u, const TList& s0, const TList& s0e,
                 const TList& s1, const TList& s1e, const TList& s2, const TList& s2e, const TList& mars,
                 const TList& marse, const OptT& scale, const OptT& masked, const OptT& gsq, const py::dict& settings) {
  const size_t n = !g.empty() ? g.size() : (!u.empty() ? u.size() : p.size());
  if (n == 0) return;
  const at::Tensor& ref = !g.empty() ? *g[0] : (!u.empty() ? *u[0] : *p[0]);
  c10::cuda::CUDAGuard guard(ref.device());
  using Key = ChainConfig;
  const ChainConfig cfg(settings);
  const int scale_stride = std::max(1, cfg.i(Key::scale_stride));
  const int gsq_stride = std::max(1, cfg.i(Key::gsq_stride));
  {  // the kernel trusts the table: every buffer must be a contiguous CUDA tensor of the element count and storage
     // kind its slot is declared with, on the device of the launch
    // storage kinds as in common.cuh: 0 fp32, 1 bf16, 2 fp16, 3 bf16+8, 4 bf16+16, 5 fp16+8, 6 fp16+16, 7 none
    auto primary_bytes = [](int dt) { return dt == 0 ? 4 : (dt == 7 ? 0 : 2); };
    auto residual_bytes = [](int dt) { return (dt == 3 || dt == 5) ? 1 : ((dt == 4 || dt == 6) ? 2 : 0); };
    struct Slot { const TList* list; const char* name; int dt; bool residual; };
    const int dp = cfg.i(Key::dt_p), dg = cfg.i(Key::dt_g), du = cfg.i(Key::dt_u), ds = cfg.i(Key::dt_s);
    const Slot slots[] = {{&p, "p", dp, false}, {&pe, "pe", dp, true}, {&g, "g", dg, false}, {&u, "u", du, false},
                          {&s0, "s0", ds, false}, {&s0e, "s0e", ds, true}, {&s1, "s1", ds, false}, {&s1e, "s1e", ds, true},
                          {&s2, "s2", ds, false}, {&s2e, "s2e", ds, true}, {&mars, "mars", ds, false}, {&marse, "marse", ds, true}};
    for (const Slot& sl : slots) {
      if (sl.list->empty()) continue;
      TORCH_CHECK(sl.list->size() == n, "fused_chain: list '", sl.name, "' has ", std::to_string(sl.list->size()), " entries, expected ", std::to_string(n));
      const int want = sl.residual ? residual_bytes(sl.dt) : primary_bytes(sl.dt);
      for (size_t i = 0; i < n; ++i) {
        const OptT& t = (*sl.list)[i];
        TORCH_CHECK(t.has_value() && t->defined(), "fused_chain: '", sl.name, "'[", std::to_string(i), "] is missing");
        TORCH_CHECK(t->is_cuda() && t->device() == ref.device() && t->is_contiguous(), "fused_chain: '", sl.name, "'[", std::to_string(i),
                    "] must be a contiguous CUDA tensor on the launch device");
        TORCH_CHECK(want != 0 && (int)t->element_size() == want, "fused_chain: '", sl.name, "'[", std::to_string(i), "] has ", std::to_string(t->element_size()),
                    "-byte elements, its storage kind needs ", std::to_string(want));
      }
    }
    for (const at::Tensor* aux : {scale.has_value() ? &*scale : nullptr, masked.has_value() ? &*masked : nullptr}) {
      if (aux == nullptr) continue;
      const size_t per = aux == (scale.has_value() ? &*scale : nullptr) ? (size_t)scale_stride : 1;
      TORCH_CHECK(aux->is_cuda() && aux->is_contiguous() && (size_t)aux->numel() >= n * per && aux->element_size() == 4,
                  "fused_chain: per-tensor scalars need ", std::to_string(per), " 4-byte entries per tensor");
    }
    if (gsq.has_value())
      TORCH_CHECK(gsq->is_cuda() && gsq->is_contiguous() && gsq->scalar_type() == at::kFloat &&
                      (gsq->numel() == 1 || (size_t)gsq->numel() >= n * (size_t)gsq_stride),
                  "fused_chain: gsq needs one fp32 entry, or gsq_stride per tensor");
    const int clip_mode = cfg.i(Key::g_clip_mode);
    TORCH_CHECK(clip_mode != hb::kClipOrtho || (gsq.has_value() && gsq_stride == 3 && !p.empty()),
                "fused_chain: the OrthoGrad projection needs the parameters and three dot products per tensor");
    const int uop = cfg.i(Key::u_op);
    const int acc = cfg.i(Key::accum_sumsq);
    TORCH_CHECK((uop != hb::kUopSignGraft && acc != 2) || (scale.has_value() && scale_stride == 2),
                "fused_chain: sign grafting keeps two sums per tensor in `scale`");
  }
  std::vector<hb::TensorMeta> metas(n);
  for (size_t i = 0; i < n; ++i) {
    hb::TensorMeta& m = metas[i];
    m.p = ptr_or_null(p, i); m.pe = ptr_or_null(pe, i); m.g = ptr_or_null(g, i); m.u = ptr_or_null(u, i);
    m.s0 = ptr_or_null(s0, i); m.s0e = ptr_or_null(s0e, i); m.s1 = ptr_or_null(s1, i); m.s1e = ptr_or_null(s1e, i);
    m.s2 = ptr_or_null(s2, i); m.s2e = ptr_or_null(s2e, i); m.mars = ptr_or_null(mars, i); m.marse = ptr_or_null(marse, i);
    m.scale = scale.has_value() ? scale->data_ptr<float>() + (int64_t)i * scale_stride : nullptr;
    m.masked = masked.has_value() ? masked->data_ptr<int>() + i : nullptr;
    m.gsq = gsq.has_value() ? gsq->data_ptr<float>() + (gsq->numel() == 1 ? 0 : (int64_t)i * gsq_stride) : nullptr;
    const at::Tensor& any = !g.empty() && g[i].has_value() ? *g[i] : (!u.empty() && u[i].has_value() ? *u[i] : *p[i]);
    m.numel = any.numel();
    for (const TList* l : {&p, &pe, &g, &u, &s0, &s0e, &s1, &s1e, &s2, &s2e, &mars, &marse})
      TORCH_CHECK(l->empty() || (*l)[i]->numel() == m.numel, "fused_chain: buffers of tensor ", std::to_string(i), " differ in element count");
    bool ok = true;
    for (void* q : {m.p, m.pe, m.g, m.u, m.s0, m.s0e, m.s1, m.s1e, m.s2, m.s2e, m.mars, m.marse}) ok = ok && aligned16(q);
    m.vec_ok = ok ? 1 : 0;
    m.pad = 0;
  }
  hb::ChainParams P{};
  P.algo = cfg.i(Key::algo); P.out_mode = cfg.i(Key::out_mode); P.n_state = cfg.i(Key::n_state);
  P.dt_p = cfg.i(Key::dt_p); P.dt_g = cfg.i(Key::dt_g); P.dt_u = cfg.i(Key::dt_u); P.dt_s = cfg.i(Key::dt_s);
  P.u_is_input = cfg.i(Key::u_is_input); P.mars = cfg.i(Key::mars); P.cautious_wd = cfg.i(Key::cautious_wd);
  P.caution_apply = cfg.i(Key::caution_apply); P.use_tensor_scale = cfg.i(Key::use_tensor_scale);
  P.accum_sumsq = cfg.i(Key::accum_sumsq); P.u_op = cfg.i(Key::u_op); P.post_state = cfg.i(Key::post_state);
  TORCH_CHECK(P.post_state != hb::kPostMsam || (!s0.empty() && !s2.empty() && P.n_state == 3),
              "fused_chain: Momentum-SAM keeps its momentum in s0 and the unperturbed weights in s2");
  TORCH_CHECK(P.post_state != hb::kPostDecayIn || !p.empty(), "fused_chain: decay folded into the update reads the parameters");
  P.g_clip_mode = cfg.i(Key::g_clip_mode); P.g_clip_at = cfg.f(Key::g_clip_at); P.g_clip_numel = cfg.f(Key::g_clip_numel);
  P.lr = cfg.f(Key::lr); P.wd = cfg.f(Key::wd); P.eps = cfg.f(Key::eps);
  P.b1 = cfg.f(Key::b1); P.b2 = cfg.f(Key::b2); P.b3 = cfg.f(Key::b3); P.alpha = cfg.f(Key::alpha); P.mars_a = cfg.f(Key::mars_a);
  P.seed = cfg.get<uint64_t>(Key::seed, 0);
  if (cfg.has(Key::g_delta)) {
    auto d = cfg.get<std::vector<int64_t>>(Key::g_delta, {});
    TORCH_CHECK((int)d.size() <= hb::kMaxPeers, "too many gradient sources");
    P.n_src = (int)d.size();
    for (size_t i = 0; i < d.size(); ++i) P.g_delta[i] = d[i];
    P.g_scale = cfg.f(Key::g_scale);
  }
  if (cfg.has(Key::p_delta)) {
    auto d = cfg.get<std::vector<int64_t>>(Key::p_delta, {});
    TORCH_CHECK((int)d.size() <= hb::kMaxPeers, "too many parameter destinations");
    P.n_dst = (int)d.size();
    for (size_t i = 0; i < d.size(); ++i) P.p_delta[i] = d[i];
  }
  P.g_mc_delta = cfg.get<int64_t>(Key::g_mc_delta, 0);
  P.p_mc_delta = cfg.get<int64_t>(Key::p_mc_delta, 0);
  const bool count = cfg.i(Key::count_caution) != 0;
  int64_t elems = 0;
  for (const hb::TensorMeta& m : metas) elems += m.numel;
  const int chunk = hb::chain_chunk_elems_for(P, count, elems);
  if (hb::chain_takes_inline(P, count, (int)n, elems)) {
    const std::vector<int> prefix = chunk_prefix(metas, chunk);
    P.n_tensors = (int)n;
    P.chunk = chunk;
    check(hb::launch_fused_chain_inline(metas.data(), prefix.data(), prefix[n], P, count, at::cuda::getCurrentCUDAStream()), "fused_chain launch");
    return;
  }
  Table t = upload(metas, ref.device(), chunk);
  P.n_tensors = t.n;
  P.chunk = t.chunk;
  check(hb::launch_fused_chain(t.metas, t.prefix, t.total_chunks, P, count, at::cuda::getCurrentCUDAStream()),
        "fused_chain launch");
}

// out[i] = sum(x_i^2) in fp32.
at::Tensor sumsq(const std::vector<at::Tensor>& xs, int dt) {
  TORCH_CHECK(!xs.empty(), "sumsq: empty list");
  c10::cuda::CUDAGuard guard(xs[0].device());
  std::vector<hb::TensorMeta> metas(xs.size());
  for (size_t i = 0; i < xs.size(); ++i) {
    memset(&metas[i], 0, sizeof(hb::TensorMeta));
    metas[i].u = xs[i].data_ptr();
    metas[i].numel = xs[i].numel();
    metas[i].vec_ok = aligned16(metas[i].u) ? 1 : 0;
  }
  Table t = upload(metas, xs[0].device());
  at::Tensor out = at::zeros({(int64_t)xs.size()}, xs[0].options().dtype(at::kFloat));
  check(hb::launch_sumsq(t.metas, t.prefix, t.total_chunks, t.n, dt, out.data_ptr<float>(),
                         at::cuda::getCurrentCUDAStream()), "sumsq launch");
  return out;
}

// out[i] = sum(x_i * y_i) (op 0) or max |x_i| (op 1, `ys` empty) in fp32; all tensors contiguous, one storage kind.
at::Tensor segmented_reduce(const std::vector<at::Tensor>& xs, const std::vector<at::Tensor>& ys, int dt, int op) {
  TORCH_CHECK(!xs.empty(), "segmented_reduce: empty list");
  TORCH_CHECK(op == hb::kReduceAbsMax ? ys.empty() : ys.size() == xs.size(), "segmented_reduce: one y per x for the dot product");
  c10::cuda::CUDAGuard guard(xs[0].device());
  std::vector<hb::TensorMeta> metas(xs.size());
  for (size_t i = 0; i < xs.size(); ++i) {
    TORCH_CHECK(xs[i].is_cuda() && xs[i].is_contiguous() && xs[i].scalar_type() == xs[0].scalar_type(), "segmented_reduce: contiguous CUDA tensors of one dtype");
    memset(&metas[i], 0, sizeof(hb::TensorMeta));
    metas[i].u = xs[i].data_ptr();
    metas[i].numel = xs[i].numel();
    bool ok = aligned16(metas[i].u);
    if (!ys.empty()) {
      TORCH_CHECK(ys[i].is_cuda() && ys[i].is_contiguous() && ys[i].scalar_type() == xs[0].scalar_type() &&
                      ys[i].numel() == xs[i].numel(), "segmented_reduce: y like x");
      metas[i].g = ys[i].data_ptr();
      ok = ok && aligned16(metas[i].g);
    }
    metas[i].vec_ok = ok ? 1 : 0;
  }
  Table t = upload(metas, xs[0].device());
  at::Tensor out = at::zeros({(int64_t)xs.size()}, xs[0].options().dtype(at::kFloat));
  check(hb::launch_segmented_reduce(t.metas, t.prefix, t.total_chunks, t.n, dt, op, out.data_ptr<float>(),
                                    at::cuda::getCurrentCUDAStream()), "segmented_reduce launch");
  return out;
}

// D = A * B^T (bf16, K-major operands, batched) with the fused epilogues described in ns_gemm.h.
void ns_gemm(const at::Tensor& A, int64_t lda, int64_t strideA, const at::Tensor& B, int64_t ldb, int64_t strideB,
             int64_t M, int64_t N, int64_t K, int64_t batch, int mode, bool symmetric, const OptT& C, int64_t ldc,
             int64_t strideC, const OptT& CT, int64_t ldct, int64_t strideCT, const OptT& F, int64_t ldf, int64_t strideF,
             bool f_transposed, double f_scale, const OptT& S, int64_t lds, int64_t strideS, double ca, double cb,
             double cc, const at::Tensor& status) {
  c10::cuda::CUDAGuard guard(A.device());
  hb::GemmParams P{};
  P.M = (int)M; P.N = (int)N; P.K = (int)K; P.batch = (int)batch; P.mode = mode; P.symmetric = symmetric ? 1 : 0;
  P.C = C.has_value() ? (__nv_bfloat16*)C->data_ptr() : nullptr; P.ldc = ldc; P.strideC = strideC;
  P.CT = CT.has_value() ? (__nv_bfloat16*)CT->data_ptr() : nullptr; P.ldct = ldct; P.strideCT = strideCT;
  P.F = F.has_value() ? F->data_ptr<float>() : nullptr; P.ldf = ldf; P.strideF = strideF;
  P.f_transposed = f_transposed ? 1 : 0; P.f_scale = (float)f_scale;
  P.S = S.has_value() ? (const __nv_bfloat16*)S->data_ptr() : nullptr; P.lds = lds; P.strideS = strideS;
  P.ca = (float)ca; P.cb = (float)cb; P.cc = (float)cc;
  P.status = status.data_ptr<int>();
  const hb::NsProduct X{A.data_ptr(), lda, strideA, B.data_ptr(), ldb, strideB, P};
  check(hb::launch_ns_products(&X, 1, nullptr, at::cuda::getCurrentCUDAStream()), "ns_gemm launch");
}

// The whole Newton-Schulz iteration of several shape buckets: one launch normalises and rounds every matrix, then each step is
// a Gram, a polynomial and an apply product of all buckets together (the last apply writes fp32 into `outs`, in the caller's
// orientation).  mats[g]: the matrices of bucket g, contiguous, one shape and dtype per bucket (one dtype for all);
// sumsq / sumsq_at[g][j]: fp32 squared Frobenius norms and where matrix j of bucket g has its own; seeds[g]: rounding noise.
// Returns the number of kernel launches.
int64_t ns_orthogonalize(const std::vector<std::vector<at::Tensor>>& mats, int src_dt, const at::Tensor& sumsq,
                         const std::vector<std::vector<int64_t>>& sumsq_at, const std::vector<at::Tensor>& outs,
                         const std::vector<double>& out_scales, const std::vector<uint64_t>& seeds,
                         const std::vector<std::vector<double>>& coeffs, double eps, const at::Tensor& status) {
  const size_t n = mats.size();
  TORCH_CHECK(n > 0 && sumsq_at.size() == n && outs.size() == n && out_scales.size() == n && seeds.size() == n,
              "ns_orthogonalize: one entry per bucket");
  TORCH_CHECK(sumsq.is_cuda() && sumsq.scalar_type() == at::kFloat && sumsq.is_contiguous(), "ns_orthogonalize: fp32 norms");
  const at::Device dev = sumsq.device();
  c10::cuda::CUDAGuard guard(dev);
  auto stream = at::cuda::getCurrentCUDAStream();
  struct Bucket { int64_t batch, R, C, m, n, ldx, lds; __nv_bfloat16 *x[2], *s, *y; };
  std::vector<Bucket> buckets(n);
  auto up8 = [](int64_t v) { return (v + 7) / 8 * 8; };
  auto room = [](int64_t elems) { return (elems + 127) / 128 * 128; };  // buffers start on 256-byte boundaries
  int64_t elems = 0;
  size_t total_mats = 0;
  for (size_t g = 0; g < n; ++g) {
    Bucket& b = buckets[g];
    TORCH_CHECK(!mats[g].empty() && mats[g][0].dim() == 2 && sumsq_at[g].size() == mats[g].size(), "ns_orthogonalize: empty bucket");
    b.batch = (int64_t)mats[g].size(); b.R = mats[g][0].size(0); b.C = mats[g][0].size(1);
    b.m = std::min(b.R, b.C); b.n = std::max(b.R, b.C); b.ldx = up8(b.n); b.lds = up8(b.m);
    const at::Tensor& o = outs[g];
    TORCH_CHECK(o.device() == dev && o.scalar_type() == at::kFloat && o.is_contiguous() && o.numel() == b.batch * b.R * b.C,
                "ns_orthogonalize: out must be contiguous fp32 [batch, R, C]");
    elems += 2 * room(b.batch * b.m * b.ldx) + 2 * room(b.batch * b.m * b.lds);
    total_mats += mats[g].size();
  }
  at::Tensor slab = at::empty({elems}, sumsq.options().dtype(at::kBFloat16));
  auto* cursor = (__nv_bfloat16*)slab.data_ptr();
  std::vector<hb::NsSource> src;
  std::vector<int> first(1, 0);
  src.reserve(total_mats);
  for (size_t g = 0; g < n; ++g) {
    Bucket& b = buckets[g];
    for (auto** p : {&b.x[0], &b.x[1]}) { *p = cursor; cursor += room(b.batch * b.m * b.ldx); }
    for (auto** p : {&b.s, &b.y}) { *p = cursor; cursor += room(b.batch * b.m * b.lds); }
    for (int64_t j = 0; j < b.batch; ++j) {
      const at::Tensor& t = mats[g][j];
      TORCH_CHECK(t.device() == dev && t.is_contiguous() && t.scalar_type() == mats[0][0].scalar_type() && t.dim() == 2 &&
                      t.size(0) == b.R && t.size(1) == b.C, "ns_orthogonalize: contiguous matrices of one shape per bucket");
      TORCH_CHECK(sumsq_at[g][j] >= 0 && sumsq_at[g][j] < sumsq.numel(), "ns_orthogonalize: norm index out of range");
      src.push_back({t.data_ptr(), sumsq.data_ptr<float>() + sumsq_at[g][j], b.x[0] + j * b.m * b.ldx, seeds[g], b.ldx, (int)b.R,
                     (int)b.C, b.R > b.C ? 1 : 0, (int)j});
      first.push_back(first.back() + (int)(((b.R + 63) / 64) * ((b.C + 63) / 64)));
    }
  }
  const size_t src_bytes = src.size() * sizeof(hb::NsSource), first_bytes = first.size() * sizeof(int);
  std::vector<uint8_t> host(src_bytes + first_bytes);
  memcpy(host.data(), src.data(), src_bytes);
  memcpy(host.data() + src_bytes, first.data(), first_bytes);
  at::Tensor table = at::empty({(int64_t)host.size()}, sumsq.options().dtype(at::kByte));
  check(cudaMemcpyAsync(table.data_ptr(), host.data(), host.size(), cudaMemcpyHostToDevice, stream), "matrix table upload");
  check(hb::launch_ns_prepare((const hb::NsSource*)table.data_ptr(), (const int*)((uint8_t*)table.data_ptr() + src_bytes),
                              (int)src.size(), first.back(), src_dt, (float)eps, stream), "ns_prepare launch");
  int launches = 1;
  std::vector<hb::NsProduct> stage(n);
  // the products of one kind for every bucket, reading iterate `cur`; the last apply writes the results
  const auto plan = [&](int mode, int cur, bool last) {
    for (size_t g = 0; g < n; ++g) {
      const Bucket& b = buckets[g];
      hb::NsProduct& X = stage[g];
      hb::GemmParams P{};
      P.mode = mode; P.batch = (int)b.batch; P.status = status.data_ptr<int>(); P.M = (int)b.m; P.f_scale = 1.f;
      if (mode == hb::kModeApply) {  // X' = Y X
        X = {b.y, b.lds, b.m * b.lds, b.x[cur], b.ldx, b.m * b.ldx, {}};
        P.N = (int)b.n; P.K = (int)b.m; P.b_mn = 1;
        if (!last) {
          P.C = b.x[1 - cur]; P.ldc = b.ldx; P.strideC = b.m * b.ldx;
        } else {
          P.F = outs[g].data_ptr<float>(); P.ldf = b.C; P.strideF = b.R * b.C; P.f_transposed = b.R > b.C ? 1 : 0;
          P.f_scale = (float)out_scales[g];
        }
      } else {  // S = X X^T,  Y = c S S + b S + a I
        const bool poly = mode == hb::kModePoly;
        if (poly)
          X = {b.s, b.lds, b.m * b.lds, b.s, b.lds, b.m * b.lds, {}};
        else
          X = {b.x[cur], b.ldx, b.m * b.ldx, b.x[cur], b.ldx, b.m * b.ldx, {}};
        P.N = (int)b.m; P.K = (int)(poly ? b.m : b.n); P.symmetric = 1;
        P.C = P.CT = poly ? b.y : b.s; P.ldc = P.ldct = b.lds; P.strideC = P.strideCT = b.m * b.lds;
        if (poly) { P.S = b.s; P.lds = b.lds; P.strideS = b.m * b.lds; }
      }
      X.P = P;
    }
    hb::NsPlan made;
    check(hb::prepare_ns_products(stage.data(), (int)n, &made), "ns_orthogonalize products");
    return made;
  };
  hb::NsPlan gram[2], poly, apply[2];
  int cur = 0;
  for (size_t step = 0; step < coeffs.size(); ++step, cur = 1 - cur) {
    TORCH_CHECK(coeffs[step].size() == 3, "ns_orthogonalize: (a, b, c) per step");
    const bool last = step + 1 == coeffs.size();
    if (!gram[cur].launches) gram[cur] = plan(hb::kModeGram, cur, false);
    if (!poly.launches) poly = plan(hb::kModePoly, cur, false);
    if (last || !apply[cur].launches) apply[cur] = plan(hb::kModeApply, cur, last);
    hb::set_ns_coefficients(poly, (float)coeffs[step][0], (float)coeffs[step][1], (float)coeffs[step][2]);
    for (const hb::NsPlan* p : {&gram[cur], &poly, &apply[cur]}) check(hb::launch_ns_plan(*p, &launches, stream), "ns_orthogonalize launch");
  }
  return launches;
}

// Store `epoch` into slot[rank] of every peer's flag array (after a system-scope fence).
void peer_signal(const std::vector<int64_t>& flag_ptrs, int slot, int rank, int epoch) {
  hb::PeerPtrs ptrs{};
  TORCH_CHECK((int)flag_ptrs.size() <= hb::kMaxWorld, "world size above kMaxWorld");
  for (size_t i = 0; i < flag_ptrs.size(); ++i) ptrs.ptr[i] = (uint64_t)flag_ptrs[i];
  check(hb::launch_peer_signal(ptrs, slot, rank, (int)flag_ptrs.size(), epoch, at::cuda::getCurrentCUDAStream()),
        "peer_signal launch");
}

// Wait (bounded) until every rank has stored `epoch` into `slot` of this rank's flag array.
void peer_wait(const at::Tensor& my_flags, int slot, int world, int epoch, double timeout_s, const at::Tensor& status) {
  c10::cuda::CUDAGuard guard(my_flags.device());
  check(hb::launch_peer_wait(my_flags.data_ptr<int>(), slot, world, epoch, timeout_s, status.data_ptr<int>(),
                             at::cuda::getCurrentCUDAStream()), "peer_wait launch");
}

// In-place softmax cross-entropy: `logits` ([rows, ld] bf16) becomes the gradient of sum(loss) * scale[0];
// returns the per-row losses.
at::Tensor cross_entropy_(at::Tensor& logits, const at::Tensor& targets, const at::Tensor& scale, int64_t vocab,
                          int64_t ignore_index) {
  TORCH_CHECK(logits.is_cuda() && logits.dim() == 2 && logits.scalar_type() == at::kBFloat16, "logits: 2-D bf16 CUDA tensor");
  TORCH_CHECK(logits.is_contiguous() && logits.size(1) % 8 == 0 && aligned16(logits.data_ptr()),
              "logits must be contiguous with a row length that is a multiple of 8 (pad the vocabulary)");
  TORCH_CHECK(vocab > 0 && vocab <= logits.size(1), "vocab out of range");
  TORCH_CHECK(targets.is_cuda() && targets.scalar_type() == at::kLong && targets.is_contiguous() &&
                  targets.numel() == logits.size(0), "targets: contiguous int64, one per row");
  TORCH_CHECK(scale.is_cuda() && scale.scalar_type() == at::kFloat && scale.numel() == 1, "scale: fp32 device scalar");
  c10::cuda::CUDAGuard guard(logits.device());
  at::Tensor loss = at::empty({logits.size(0)}, logits.options().dtype(at::kFloat));
  check(hb::launch_cross_entropy(logits.data_ptr(), reinterpret_cast<const long long*>(targets.data_ptr<int64_t>()),
                                 loss.data_ptr<float>(), scale.data_ptr<float>(), logits.size(0), (int)vocab,
                                 (int)logits.size(1), ignore_index, at::cuda::getCurrentCUDAStream()),
        "cross_entropy launch");
  return loss;
}

// x *= s[0] in place for a contiguous fp32 or bf16 tensor; s: one fp32 value on the same device.
void scale_(const at::Tensor& x, const at::Tensor& s) {
  TORCH_CHECK(x.is_cuda() && x.is_contiguous() && (x.scalar_type() == at::kFloat || x.scalar_type() == at::kBFloat16) && aligned16(x.data_ptr()),
              "scale_: contiguous fp32 or bf16 CUDA tensor");
  TORCH_CHECK(s.device() == x.device() && s.scalar_type() == at::kFloat && s.numel() == 1, "scale_: fp32 device scalar");
  c10::cuda::CUDAGuard guard(x.device());
  check(hb::launch_scale(x.data_ptr(), x.scalar_type() == at::kBFloat16, x.numel(), s.data_ptr<float>(), at::cuda::getCurrentCUDAStream()), "scale launch");
}

// Split-tf32 operands of a contiguous fp32 [batch, R, C] tensor: rows of [hi | lo] (see tf32_gemm.h).  Returns
// (same, trans): same = [batch, R, 2 kp(C)] (operand rows = rows of x), trans = [batch, C, 2 kp(R)] (operand rows =
// columns of x); an orientation that was not asked for comes back undefined.
std::vector<at::Tensor> tf32_split(const at::Tensor& x, bool want_same, bool want_trans) {
  // views are welcome: any row and batch stride, unit inner stride
  TORCH_CHECK(x.is_cuda() && x.scalar_type() == at::kFloat && x.dim() == 3 && x.stride(2) == 1 && x.size(0) >= 1 && x.size(1) >= 1 &&
                  x.size(2) >= 1, "tf32_split: fp32 [batch, rows, cols] CUDA tensor with unit inner stride");
  c10::cuda::CUDAGuard guard(x.device());
  const int64_t batch = x.size(0), R = x.size(1), C = x.size(2);
  at::Tensor same = want_same ? at::empty({batch, R, 2 * hb::tf32_split_kp(C)}, x.options().memory_format(at::MemoryFormat::Contiguous)) : at::Tensor();
  at::Tensor trans = want_trans ? at::empty({batch, C, 2 * hb::tf32_split_kp(R)}, x.options().memory_format(at::MemoryFormat::Contiguous)) : at::Tensor();
  check(hb::launch_tf32_split(x.data_ptr<float>(), x.stride(1), x.stride(0), (int)R, (int)C, (int)batch,
                              want_same ? same.data_ptr<float>() : nullptr, want_trans ? trans.data_ptr<float>() : nullptr,
                              at::cuda::getCurrentCUDAStream()), "tf32 split");
  return {same, trans};
}

// epilogue(A * B^T) over split operands a2: [batch, M, 2 kp(K)], b2: [batch, N, 2 kp(K)] (see tf32_gemm.h).
//   mode 0 store, 1 lerp into `c` with weight w, 2 Adam / 3 LaProp on the moments m, v ([batch, M, N] fp32, in place).
//   c: fp32 [batch, M, >= N] output (optional unless mode 1).  split_out: 0 none, 1 also / instead write the result as
//   a split operand with rows = output rows, 2 with rows = output columns; it is returned (undefined when 0).
at::Tensor tf32_gemm(const at::Tensor& a2, const at::Tensor& b2, int64_t K, int mode, double alpha, double w, double b1,
                     double b2c, double eps, const OptT& c, int split_out, const OptT& m, const OptT& v,
                     const at::Tensor& status) {
  TORCH_CHECK(a2.is_cuda() && b2.is_cuda() && a2.scalar_type() == at::kFloat && b2.scalar_type() == at::kFloat &&
                  a2.dim() == 3 && b2.dim() == 3 && a2.is_contiguous() && b2.is_contiguous() && a2.size(0) == b2.size(0),
              "tf32_gemm: contiguous fp32 split operands [batch, rows, 2 kp]");
  const int64_t batch = a2.size(0), M = a2.size(1), N = b2.size(1), kp = hb::tf32_split_kp(K);
  TORCH_CHECK(a2.size(2) == 2 * kp && b2.size(2) == 2 * kp, "tf32_gemm: operands were not split for K = ", std::to_string(K));
  c10::cuda::CUDAGuard guard(a2.device());
  hb::Tf32Epilogue E{};
  E.mode = mode; E.alpha = (float)alpha; E.w = (float)w; E.b1 = (float)b1; E.b2 = (float)b2c; E.eps = (float)eps;
  if (c.has_value() && c->defined()) {
    TORCH_CHECK(c->is_cuda() && c->scalar_type() == at::kFloat && c->dim() == 3 && c->size(0) == batch && c->size(1) == M &&
                    c->size(2) >= N && c->stride(2) == 1 && c->stride(1) >= N && c->device() == a2.device(),
                "tf32_gemm: c must be fp32 [batch, M, >= N] with unit inner stride");
    E.C = c->data_ptr<float>(); E.ldc = c->stride(1); E.strideC = c->stride(0);
  }
  at::Tensor s;
  if (split_out != 0) {
    const int64_t rows = split_out == 1 ? M : N, kps = hb::tf32_split_kp(split_out == 1 ? N : M);
    s = at::empty({batch, rows, 2 * kps}, a2.options());
    E.S = s.data_ptr<float>(); E.kpS = kps; E.strideS = rows * 2 * kps; E.s_transposed = split_out == 2 ? 1 : 0;
  }
  if (mode == hb::kEpiAdam || mode == hb::kEpiLaProp) {
    TORCH_CHECK(m.has_value() && v.has_value(), "tf32_gemm: moment buffers required");
    for (const at::Tensor* t : {&*m, &*v})
      TORCH_CHECK(t->is_cuda() && t->scalar_type() == at::kFloat && t->is_contiguous() && t->numel() == batch * M * N &&
                      t->device() == a2.device(), "tf32_gemm: moments must be contiguous fp32 [batch, M, N]");
    E.m = m->data_ptr<float>(); E.v = v->data_ptr<float>();
  }
  TORCH_CHECK(E.C != nullptr || E.S != nullptr, "tf32_gemm: no output requested");
  // X X^T (one buffer as both operands): upper tiles only, mirrored on store.  An in-place lerp target is then
  // symmetric by construction (it only ever receives symmetric increments).
  E.symmetric = (a2.data_ptr() == b2.data_ptr() && M == N && E.C != nullptr && E.S == nullptr &&
                 (mode == hb::kEpiStore || mode == hb::kEpiLerp || mode == hb::kEpiAdd)) ? 1 : 0;
  check(hb::launch_tf32_gemm(a2.data_ptr<float>(), b2.data_ptr<float>(), (int)M, (int)N, (int)K, (int)batch, E,
                             status.data_ptr<int>(), at::cuda::getCurrentCUDAStream()), "tf32 gemm");
  return s;
}

void check_split16_source(const at::Tensor& x) {
  TORCH_CHECK(x.is_cuda() && x.scalar_type() == at::kFloat && x.dim() == 3 && x.stride(2) == 1 && x.size(0) >= 1 && x.size(1) >= 1 &&
                  x.size(2) >= 1 && x.size(0) <= 65535, "split16: fp32 [batch, rows, cols] CUDA tensor with unit inner stride");
}

// The matrix x behind an operand whose rows are the rows (trans: the columns) of x.
hb::Split16Source source_of(const at::Tensor& x, bool trans) {
  return {x.data_ptr<float>(), x.stride(0), trans ? x.stride(2) : x.stride(1), trans ? x.stride(1) : x.stride(2)};
}

// Operands of the fp16-pair product of an fp32 [batch, R, C] tensor (see split16_gemm.h): (same, same_unit, trans, trans_unit); an
// orientation that was not asked for comes back undefined.
std::vector<at::Tensor> split16(const at::Tensor& x, bool want_same, bool want_trans) {
  check_split16_source(x);
  c10::cuda::CUDAGuard guard(x.device());
  const int64_t batch = x.size(0), R = x.size(1), C = x.size(2);
  std::vector<at::Tensor> out(4);
  hb::Split16Operand op[2] = {};
  for (int i = 0; i < 2; ++i) {
    if (!(i == 0 ? want_same : want_trans)) continue;
    const int64_t rows = i == 0 ? R : C, K = i == 0 ? C : R;
    out[2 * i] = at::empty({batch, rows, 2 * hb::split16_kp(K)}, x.options().dtype(at::kHalf).memory_format(at::MemoryFormat::Contiguous));
    out[2 * i + 1] = at::empty({batch, hb::split16_units(rows)}, x.options().memory_format(at::MemoryFormat::Contiguous));
    op[i] = {out[2 * i].data_ptr(), out[2 * i + 1].data_ptr<float>(), source_of(x, i == 1)};
  }
  const hb::Split16Pass pass{x.data_ptr<float>(), x.stride(1), x.stride(0), (int)R, (int)C, op[0], op[1]};
  check(hb::launch_split16(&pass, 1, (int)batch, at::cuda::getCurrentCUDAStream()), "split16");
  return out;
}

// Results may be computed from the matrices after others have been stored.  (Interleaved views of one buffer pass: whether they share
// entries is the caller's business.)
void check_split16_overlap(const at::Tensor& out, const at::Tensor& source) {
  const at::MemOverlapStatus overlap = at::get_overlap_status(out, source);
  TORCH_CHECK(overlap != at::MemOverlapStatus::Full && overlap != at::MemOverlapStatus::Partial,
              "split16: an output lies over the matrix that an operand was made from");
}

// epilogue(A * B^T) over operands of split16; arguments as for tf32_gemm.  Both operands being one buffer makes the product symmetric.
// xa, xb: the tensors the operands were made from, with their columns (ta, tb) or rows as operand rows; neither may be written here.
void split16_gemm(const at::Tensor& a, const at::Tensor& ua, const at::Tensor& xa, bool ta, const at::Tensor& b, const at::Tensor& ub,
                  const at::Tensor& xb, bool tb, int64_t K, int mode, double alpha, double w, double b1, double b2c, double eps, const OptT& c,
                  const OptT& m, const OptT& v, bool upper_upper, const at::Tensor& status) {
  TORCH_CHECK(a.is_cuda() && b.is_cuda() && a.scalar_type() == at::kHalf && b.scalar_type() == at::kHalf && a.dim() == 3 && b.dim() == 3 &&
                  a.is_contiguous() && b.is_contiguous() && a.size(0) == b.size(0) && K >= 1,
              "split16_gemm: contiguous fp16 operands [batch, rows, 2 kp]");
  const int64_t batch = a.size(0), M = a.size(1), N = b.size(1), kp = hb::split16_kp(K);
  TORCH_CHECK(a.size(2) == 2 * kp && b.size(2) == 2 * kp, "split16_gemm: operands were not split for K = ", std::to_string(K));
  struct Side { const at::Tensor &u, &x; bool trans; int64_t rows; };
  for (const Side& s : {Side{ua, xa, ta, M}, Side{ub, xb, tb, N}}) {
    TORCH_CHECK(s.u.is_cuda() && s.u.scalar_type() == at::kFloat && s.u.is_contiguous() && s.u.numel() == batch * hb::split16_units(s.rows) &&
                    s.u.device() == a.device(), "split16_gemm: units of another operand");
    TORCH_CHECK(s.x.device() == a.device() && s.x.scalar_type() == at::kFloat && s.x.dim() == 3 && s.x.size(0) == batch && s.x.stride(2) == 1 &&
                    s.x.size(s.trans ? 2 : 1) == s.rows && s.x.size(s.trans ? 1 : 2) == K, "split16_gemm: the source of another operand");
    for (const OptT* out : {&c, &m, &v})
      if (out->has_value() && (*out)->defined()) check_split16_overlap(**out, s.x);
  }
  c10::cuda::CUDAGuard guard(a.device());
  hb::Tf32Epilogue E{};
  E.mode = mode; E.alpha = (float)alpha; E.w = (float)w; E.b1 = (float)b1; E.b2 = (float)b2c; E.eps = (float)eps;
  if (c.has_value() && c->defined()) {
    TORCH_CHECK(c->is_cuda() && c->scalar_type() == at::kFloat && c->dim() == 3 && c->size(0) == batch && c->size(1) == M &&
                    c->size(2) >= N && c->stride(2) == 1 && c->stride(1) >= N && c->device() == a.device(),
                "split16_gemm: c must be fp32 [batch, M, >= N] with unit inner stride");
    E.C = c->data_ptr<float>(); E.ldc = c->stride(1); E.strideC = c->stride(0);
  }
  if (mode == hb::kEpiAdam || mode == hb::kEpiLaProp) {
    TORCH_CHECK(m.has_value() && v.has_value(), "split16_gemm: moment buffers required");
    for (const at::Tensor* t : {&*m, &*v})
      TORCH_CHECK(t->is_cuda() && t->scalar_type() == at::kFloat && t->is_contiguous() && t->numel() == batch * M * N &&
                      t->device() == a.device(), "split16_gemm: moments must be contiguous fp32 [batch, M, N]");
    E.m = m->data_ptr<float>(); E.v = v->data_ptr<float>();
  }
  TORCH_CHECK(E.C != nullptr, "split16_gemm: no output requested");
  TORCH_CHECK(!upper_upper || (M == N && M == K && a.data_ptr() != b.data_ptr()), "split16_gemm: upper_upper needs two square matrices of one size");
  E.tri = upper_upper ? 1 : 0;
  E.symmetric = (a.data_ptr() == b.data_ptr() && M == N && (mode == hb::kEpiStore || mode == hb::kEpiLerp || mode == hb::kEpiAdd)) ? 1 : 0;
  check(hb::launch_split16_gemm({a.data_ptr(), ua.data_ptr<float>(), source_of(xa, ta)}, {b.data_ptr(), ub.data_ptr<float>(), source_of(xb, tb)},
                                (int)M, (int)N, (int)K, (int)batch, E, status.data_ptr<int>(), at::cuda::getCurrentCUDAStream()), "split16 gemm");
}

// c <- alpha op(a) op(b), or c + alpha op(a) op(b) (kEpiAdd): both operand passes and the product.  The operands share one allocation: a
// captured region cannot use blocks of the memory outside it, and what it pays for its own goes by their number.
void split16_product(const at::Tensor& a, const at::Tensor& b, bool ta, bool tb, int mode, double alpha, const at::Tensor& c, bool upper_upper,
                     const at::Tensor& status) {
  const int64_t batch = a.size(0), M = ta ? a.size(2) : a.size(1), K = ta ? a.size(1) : a.size(2), N = tb ? b.size(1) : b.size(2);
  TORCH_CHECK(b.device() == a.device() && b.size(0) == batch && (tb ? b.size(2) : b.size(1)) == K, "split16: batches or inner dimensions differ");
  const bool one = a.data_ptr() == b.data_ptr() && a.sizes() == b.sizes() && a.strides() == b.strides() && ta != tb;  // X X^T or X^T X
  TORCH_CHECK(!upper_upper || (M == N && M == K && !one), "split16: upper_upper needs two square matrices of one size");
  c10::cuda::CUDAGuard guard(a.device());
  const auto stream = at::cuda::getCurrentCUDAStream();
  // rows of pairs are multiples of 256 bytes, units of 1 KiB
  const int64_t kp = hb::split16_kp(K), a_bytes = batch * M * 4 * kp, b_bytes = one ? 0 : batch * N * 4 * kp;
  const int64_t a_units = batch * hb::split16_units(M) * 4, b_units = one ? 0 : batch * hb::split16_units(N) * 4;
  const at::Tensor memory = at::empty({a_bytes + b_bytes + a_units + b_units}, a.options().dtype(at::kByte).memory_format(at::MemoryFormat::Contiguous));
  uint8_t* const p = memory.data_ptr<uint8_t>();
  const hb::Split16Operand none{};
  const hb::Split16Operand A{p, (float*)(p + a_bytes + b_bytes), source_of(a, ta)};
  // B as the K-major [N, K] operand: b given as [K, N] must be transposed, b given as [N, K] is used as it is
  const hb::Split16Operand B = one ? A : hb::Split16Operand{p + a_bytes, (float*)(p + a_bytes + b_bytes + a_units), source_of(b, !tb)};
  const auto pass_of = [&](const at::Tensor& t, bool as_rows, const hb::Split16Operand& to) {
    return hb::Split16Pass{t.data_ptr<float>(), t.stride(1), t.stride(0), (int)t.size(1), (int)t.size(2), as_rows ? to : none, as_rows ? none : to};
  };
  const hb::Split16Pass passes[2] = {pass_of(a, !ta, A), pass_of(b, tb, B)};
  check(hb::launch_split16(passes, one ? 1 : 2, (int)batch, stream), "split16 of a product's operands");
  hb::Tf32Epilogue E{};
  E.mode = mode; E.alpha = (float)alpha;
  E.C = c.data_ptr<float>(); E.ldc = c.stride(1); E.strideC = c.stride(0);
  E.tri = upper_upper ? 1 : 0;
  E.symmetric = one ? 1 : 0;
  check(hb::launch_split16_gemm(A, B, (int)M, (int)N, (int)K, (int)batch, E, status.data_ptr<int>(), stream), "split16 gemm");
}

// op(a) @ op(b) for batched fp32 matrices from fp16 pairs; arguments and result as for tf32x3_matmul.
at::Tensor split16_matmul(const at::Tensor& a, const at::Tensor& b, bool ta, bool tb, double alpha, const at::Tensor& status,
                          bool upper_upper) {
  check_split16_source(a);
  check_split16_source(b);
  const int64_t M = ta ? a.size(2) : a.size(1), N = tb ? b.size(1) : b.size(2), ldc = (N + 3) / 4 * 4;
  c10::cuda::CUDAGuard guard(a.device());
  const at::Tensor c = at::empty({a.size(0), M, ldc}, a.options().memory_format(at::MemoryFormat::Contiguous));
  const at::Tensor view = ldc == N ? c : c.narrow(2, 0, N);
  split16_product(a, b, ta, tb, hb::kEpiStore, alpha, view, upper_upper, status);
  return view;
}

// c <- c + alpha a op(b), in place on the view c (unit inner stride), which neither operand may overlap.
void split16_accumulate(const at::Tensor& c, const at::Tensor& a, const at::Tensor& b, bool tb, double alpha, const at::Tensor& status) {
  check_split16_source(a);
  check_split16_source(b);
  TORCH_CHECK(c.device() == a.device() && c.scalar_type() == at::kFloat && c.dim() == 3 && c.stride(2) == 1 && c.size(0) == a.size(0) &&
                  c.size(1) == a.size(1) && c.size(2) == (tb ? b.size(1) : b.size(2)) && c.stride(1) >= c.size(2),
              "split16_accumulate: c must be fp32 [batch, M, N] with unit inner stride");
  check_split16_overlap(c, a);
  check_split16_overlap(c, b);
  split16_product(a, b, false, tb, hb::kEpiAdd, alpha, c, false, status);
}

// op(a) @ op(b) for batched fp32 matrices on the split-tf32 tensor-core path.  a: [batch, R, C]; ta = 0 uses a as
// [M, K], ta = 1 as [K, M]; likewise b is [K, N] for tb = 0 and [N, K] for tb = 1.  Returns [batch, M, N].
// upper_upper: op(a) and op(b) are both upper triangular (square, same size): only the non-zero K range of every tile
// is walked and the part below the diagonal comes back as zeros.
at::Tensor tf32x3_matmul(const at::Tensor& a, const at::Tensor& b, bool ta, bool tb, double alpha, const at::Tensor& status,
                         bool upper_upper) {
  TORCH_CHECK(a.is_cuda() && b.is_cuda() && a.scalar_type() == at::kFloat && b.scalar_type() == at::kFloat &&
                  a.dim() == 3 && b.dim() == 3 && a.is_contiguous() && b.is_contiguous() && a.size(0) == b.size(0),
              "tf32x3_matmul: contiguous fp32 [batch, rows, cols] CUDA tensors");
  const int64_t batch = a.size(0);
  const int64_t M = ta ? a.size(2) : a.size(1), K = ta ? a.size(1) : a.size(2);
  const int64_t N = tb ? b.size(1) : b.size(2), Kb = tb ? b.size(2) : b.size(1);
  TORCH_CHECK(K == Kb, "tf32x3_matmul: inner dimensions differ");
  c10::cuda::CUDAGuard guard(a.device());
  auto stream = at::cuda::getCurrentCUDAStream();
  const int64_t kp = hb::tf32_split_kp(K), ldc = (N + 3) / 4 * 4;
  at::Tensor a2 = at::empty({batch, M, 2 * kp}, a.options());
  const bool same_operand = a.data_ptr() == b.data_ptr() && a.sizes() == b.sizes() && ta != tb;  // X X^T or X^T X
  at::Tensor b2 = same_operand ? a2 : at::empty({batch, N, 2 * kp}, a.options());
  at::Tensor c = at::empty({batch, M, ldc}, a.options());
  check(hb::launch_tf32_split(a.data_ptr<float>(), a.size(2), a.size(1) * a.size(2), (int)a.size(1), (int)a.size(2),
                              (int)batch, ta ? nullptr : a2.data_ptr<float>(), ta ? a2.data_ptr<float>() : nullptr, stream),
        "tf32 split A");
  // B as the K-major [N, K] operand: b given as [K, N] must be transposed, b given as [N, K] is used as it is
  if (!same_operand)
    check(hb::launch_tf32_split(b.data_ptr<float>(), b.size(2), b.size(1) * b.size(2), (int)b.size(1), (int)b.size(2),
                                (int)batch, tb ? b2.data_ptr<float>() : nullptr, tb ? nullptr : b2.data_ptr<float>(), stream),
          "tf32 split B");
  hb::Tf32Epilogue E{};
  E.mode = hb::kEpiStore; E.alpha = (float)alpha; E.C = c.data_ptr<float>(); E.ldc = ldc; E.strideC = M * ldc;
  E.symmetric = same_operand ? 1 : 0;  // X X^T / X^T X: upper tiles, mirrored on store
  if (upper_upper) {
    TORCH_CHECK(M == N && M == K && !same_operand, "tf32x3_matmul: upper_upper needs two square matrices of one size");
    E.tri = 1;
  }
  check(hb::launch_tf32_gemm(a2.data_ptr<float>(), b2.data_ptr<float>(), (int)M, (int)N, (int)K, (int)batch, E,
                             status.data_ptr<int>(), stream), "tf32 gemm");
  return ldc == N ? c : c.narrow(2, 0, N);
}

// Partial products X^T W over the long dimension: x = first `m` columns of the contiguous [batch, n, k] tensor `base`,
// w: contiguous [batch, n, p], p <= 32.  Returns [splits, batch, m, p]; sum over dim 0 for the product.
at::Tensor tall_t_mul(const at::Tensor& base, int64_t m, const at::Tensor& w) {
  TORCH_CHECK(base.is_cuda() && w.is_cuda() && base.scalar_type() == at::kFloat && w.scalar_type() == at::kFloat &&
                  base.dim() == 3 && w.dim() == 3 && base.is_contiguous() && w.is_contiguous() &&
                  base.size(0) == w.size(0) && base.size(1) == w.size(1) && w.size(2) <= 32 && m >= 0 && m <= base.size(2),
              "tall_t_mul: contiguous fp32 [batch, n, k] and [batch, n, p <= 32]");
  c10::cuda::CUDAGuard guard(base.device());
  const int64_t batch = base.size(0), n = base.size(1), k = base.size(2), p = w.size(2);
  at::Tensor c = at::empty({hb::tall_splits((int)n), batch, m, p}, base.options());
  check(hb::launch_tall_t_mul(base.data_ptr<float>(), k, n * k, w.data_ptr<float>(), p, n * p, (int)batch, (int)n, (int)m,
                              (int)p, c.data_ptr<float>(), at::cuda::getCurrentCUDAStream()), "tall_t_mul launch");
  return c;
}

// Inverses of the 128 x 128 diagonal blocks of a batch of upper-triangular fp32 matrices q: [batch, n, n] (unit inner
// stride).  Returns [batch, ceil(n / 128), 128, 128]; entries below the diagonal of q are ignored.
at::Tensor tri_inv_blocks(const at::Tensor& q) {
  TORCH_CHECK(q.is_cuda() && q.scalar_type() == at::kFloat && q.dim() == 3 && q.size(1) == q.size(2) && q.stride(2) == 1,
              "tri_inv_blocks: fp32 [batch, n, n] CUDA tensor with unit inner stride");
  c10::cuda::CUDAGuard guard(q.device());
  const int64_t batch = q.size(0), n = q.size(1), nb = (n + hb::kTriBlock - 1) / hb::kTriBlock;
  at::Tensor x = at::empty({batch, nb, hb::kTriBlock, hb::kTriBlock}, q.options());
  check(hb::launch_tri_inv_blocks(q.data_ptr<float>(), q.stride(1), q.stride(0), (int)batch, (int)n, x.data_ptr<float>(),
                                  at::cuda::getCurrentCUDAStream()), "tri_inv_blocks launch");
  return x;
}

// Columns of the contiguous fp32 [batch, n, k] tensor x in the order of the permutations `order` (contiguous int64 [batch, k]), or put
// back from it (inverse).
at::Tensor permute_columns(const at::Tensor& x, const at::Tensor& order, bool inverse) {
  TORCH_CHECK(x.is_cuda() && x.scalar_type() == at::kFloat && x.dim() == 3 && x.is_contiguous() && x.size(2) <= hb::kMaxPermuted && x.size(0) <= 65535,
              "permute_columns: contiguous fp32 [batch, n, k] CUDA tensor, k <= 12288");
  TORCH_CHECK(order.device() == x.device() && order.scalar_type() == at::kLong && order.is_contiguous() && order.dim() == 2 &&
                  order.size(0) == x.size(0) && order.size(1) == x.size(2), "permute_columns: contiguous int64 [batch, k] order");
  c10::cuda::CUDAGuard guard(x.device());
  at::Tensor out = at::empty_like(x);
  check(hb::launch_permute_columns(x.data_ptr<float>(), reinterpret_cast<const long long*>(order.data_ptr<int64_t>()), out.data_ptr<float>(),
                                   (int)x.size(0), (int)x.size(1), (int)x.size(2), inverse ? 1 : 0, at::cuda::getCurrentCUDAStream()),
        "permute_columns launch");
  return out;
}

// bad[b] |= 1 where the fp32 [batch, k, k] matrix g[b] (unit inner stride) is further than `limit` from the identity, or not finite.
void identity_defect(const at::Tensor& g, double limit, at::Tensor& bad) {
  TORCH_CHECK(g.is_cuda() && g.scalar_type() == at::kFloat && g.dim() == 3 && g.size(1) == g.size(2) && g.stride(2) == 1 && g.size(0) <= 65535,
              "identity_defect: fp32 [batch, k, k] CUDA tensor with unit inner stride");
  TORCH_CHECK(bad.device() == g.device() && bad.scalar_type() == at::kInt && bad.is_contiguous() && bad.numel() == g.size(0),
              "identity_defect: one int32 flag per matrix");
  c10::cuda::CUDAGuard guard(g.device());
  check(hb::launch_identity_defect(g.data_ptr<float>(), g.stride(1), g.stride(0), (int)g.size(0), (int)g.size(1), (float)limit, bad.data_ptr<int>(),
                                   at::cuda::getCurrentCUDAStream()), "identity_defect launch");
}

// Factors the diagonal leaf [lo, lo + size) of the batched symmetric positive definite fp32 matrices g ([batch, n, n], unit
// inner stride) as R^T R: writes R's block into r (same layout as g) and the block's inverse into inv[:, lo / 128]
// (inv: contiguous [batch, ceil(n / 128), 128, 128]); info: int32 [batch], incremented per matrix with a bad pivot.
void chol_inv_leaf(const at::Tensor& g, at::Tensor& r, at::Tensor& inv, int64_t lo, int64_t size, at::Tensor& info) {
  TORCH_CHECK(g.is_cuda() && g.scalar_type() == at::kFloat && g.dim() == 3 && g.size(1) == g.size(2) && g.stride(2) == 1 &&
                  r.is_cuda() && r.scalar_type() == at::kFloat && r.sizes() == g.sizes() && r.stride(2) == 1 &&
                  r.device() == g.device(), "chol_inv_leaf: fp32 [batch, n, n] CUDA tensors with unit inner stride");
  const int64_t batch = g.size(0), n = g.size(1), nb = (n + hb::kTriBlock - 1) / hb::kTriBlock;
  TORCH_CHECK(lo >= 0 && size >= 1 && size <= hb::kTriBlock && lo + size <= n && lo % hb::kTriBlock == 0,
              "chol_inv_leaf: leaf [lo, lo + size) must start on a multiple of 128 and hold at most 128 rows");
  TORCH_CHECK(inv.is_cuda() && inv.scalar_type() == at::kFloat && inv.is_contiguous() && inv.dim() == 4 && inv.size(0) == batch &&
                  inv.size(1) == nb && inv.size(2) == hb::kTriBlock && inv.size(3) == hb::kTriBlock && inv.device() == g.device(),
              "chol_inv_leaf: inv must be contiguous fp32 [batch, ceil(n / 128), 128, 128]");
  TORCH_CHECK(info.is_cuda() && info.scalar_type() == at::kInt && info.is_contiguous() && info.numel() == batch &&
                  info.device() == g.device(), "chol_inv_leaf: info must be int32 [batch]");
  c10::cuda::CUDAGuard guard(g.device());
  const int64_t blk = hb::kTriBlock * hb::kTriBlock;
  check(hb::launch_chol_inv_leaf(g.data_ptr<float>() + lo * g.stride(1) + lo, g.stride(1), g.stride(0),
                                 r.data_ptr<float>() + lo * r.stride(1) + lo, r.stride(1), r.stride(0),
                                 inv.data_ptr<float>() + (lo / hb::kTriBlock) * blk, nb * blk, (int)batch, (int)size,
                                 info.data_ptr<int>(), at::cuda::getCurrentCUDAStream()), "chol_inv_leaf launch");
}

// One round of Cholesky QR (chol_qr.h): a <- a R^-1 with R^T R = gram, which is overwritten.  Contiguous fp32, a: [batch, n, k], n a multiple of
// 64, k of 128; info: int32 [batch], incremented per leaf with a bad pivot.  Returns the split-tf32 operand of the new a^T (when asked) and the
// number of launches.
std::tuple<OptT, int> chol_qr_round(const at::Tensor& gram, const at::Tensor& a, bool want_trans, const at::Tensor& info,
                                                const at::Tensor& status) {
  for (const at::Tensor* t : {&gram, &a})
    TORCH_CHECK(t->is_cuda() && t->device() == a.device() && t->scalar_type() == at::kFloat && t->dim() == 3 && t->is_contiguous() && aligned16(t->data_ptr()),
                "chol_qr_round: contiguous fp32 [batch, n, k] CUDA tensors");
  const int64_t batch = a.size(0), n = a.size(1), k = a.size(2);
  TORCH_CHECK(n >= 1 && k >= 1 && n % hb::kQrRows == 0 && k % hb::kQrBlock == 0 && batch <= 65535 && gram.size(0) == batch && gram.size(1) == k && gram.size(2) == k,
              "chol_qr_round: a of n x k, n a multiple of 64 and k of 128, with its k x k Gram matrix");
  TORCH_CHECK(at::get_overlap_status(gram, a) == at::MemOverlapStatus::No, "chol_qr_round: two tensors");
  TORCH_CHECK(info.device() == a.device() && info.scalar_type() == at::kInt && info.is_contiguous() && info.numel() == batch, "chol_qr_round: info must be int32 [batch]");
  c10::cuda::CUDAGuard guard(a.device());
  const auto options = a.options().memory_format(at::MemoryFormat::Contiguous);
  const at::Tensor x_same = at::empty({batch, n, 2 * k}, options), l = at::empty({batch, k, 2 * k}, options);
  const at::Tensor inv = at::empty({batch, k / hb::kQrBlock, hb::kQrBlock, hb::kQrBlock}, options);
  OptT trans;
  if (want_trans) trans = at::empty({batch, k, 2 * n}, options);
  int launches = 0;
  const hb::QrRound round{gram.data_ptr<float>(), a.data_ptr<float>(), want_trans ? trans->data_ptr<float>() : nullptr, l.data_ptr<float>(),
                          inv.data_ptr<float>(), x_same.data_ptr<float>(), (int)n, (int)k, (int)batch, info.data_ptr<int>(), status.data_ptr<int>()};
  check(hb::launch_chol_qr_round(round, &launches, at::cuda::getCurrentCUDAStream()), "chol_qr_round");
  return {trans, launches};
}

// (x / norm, split-tf32 operand of its transpose) for contiguous fp32 x: [batch, n, k] and norm: [batch, 1, k]; n a multiple of 64, k of 128.
// `in_place`: x itself is divided.
std::tuple<at::Tensor, at::Tensor> qr_unit_columns(const at::Tensor& x, const at::Tensor& norm, bool in_place) {
  for (const at::Tensor* t : {&x, &norm})
    TORCH_CHECK(t->is_cuda() && t->device() == x.device() && t->scalar_type() == at::kFloat && t->dim() == 3 && t->is_contiguous() && aligned16(t->data_ptr()),
                "qr_unit_columns: contiguous fp32 CUDA tensors");
  const int64_t batch = x.size(0), n = x.size(1), k = x.size(2);
  TORCH_CHECK(n >= 1 && k >= 1 && n % 64 == 0 && k % hb::kQrBlock == 0 && batch <= 65535 && norm.size(0) == batch && norm.size(1) == 1 && norm.size(2) == k,
              "qr_unit_columns: x of n x k, n a multiple of 64 and k of 128, and one norm per column");
  c10::cuda::CUDAGuard guard(x.device());
  const auto options = x.options().memory_format(at::MemoryFormat::Contiguous);
  const at::Tensor a = in_place ? x : at::empty({batch, n, k}, options), trans = at::empty({batch, k, 2 * n}, options);
  check(hb::launch_qr_unit_columns(x.data_ptr<float>(), norm.data_ptr<float>(), a.data_ptr<float>(), trans.data_ptr<float>(), (int)batch, (int)n, (int)k,
                                   at::cuda::getCurrentCUDAStream()), "qr_unit_columns launch");
  return {a, trans};
}

void check_matrices(const at::Tensor& x, const char* name) {
  TORCH_CHECK(x.is_cuda() && x.scalar_type() == at::kFloat && x.dim() == 3 && x.is_contiguous() && x.size(0) <= 65535 && x.size(1) < (1 << 22) && x.size(2) < (1 << 22),
              name, ": contiguous fp32 [batch <= 65535, rows, cols] CUDA tensors");
}

// Contiguous [batch, C, R] copy of the transposes of x: [batch, R, C].
at::Tensor transposed(const at::Tensor& x) {
  check_matrices(x, "transposed");
  c10::cuda::CUDAGuard guard(x.device());
  at::Tensor out = at::empty({x.size(0), x.size(2), x.size(1)}, x.options().memory_format(at::MemoryFormat::Contiguous));
  check(hb::launch_transpose(x.data_ptr<float>(), out.data_ptr<float>(), (int)x.size(0), (int)x.size(1), (int)x.size(2), at::cuda::getCurrentCUDAStream()),
        "transpose launch");
  return out;
}

// a <- a + b, b <- triu(a - b), in place.
void sum_triu_diff_(const at::Tensor& a, const at::Tensor& b) {
  check_matrices(a, "sum_triu_diff_");
  check_matrices(b, "sum_triu_diff_");
  TORCH_CHECK(a.sizes() == b.sizes() && a.size(1) == a.size(2) && a.device() == b.device() && at::get_overlap_status(a, b) == at::MemOverlapStatus::No,
              "sum_triu_diff_: two batches of square matrices of one size");
  c10::cuda::CUDAGuard guard(a.device());
  check(hb::launch_sum_triu_diff(a.data_ptr<float>(), b.data_ptr<float>(), (int)a.size(0), (int)a.size(1), at::cuda::getCurrentCUDAStream()), "sum_triu_diff launch");
}

// Estimates of the largest eigenvalues of contiguous fp32 symmetric positive semi-definite matrices [batch, n, n] (power_iteration.h).
at::Tensor power_iteration(const at::Tensor& a, int64_t iterations) {
  check_matrices(a, "power_iteration");
  TORCH_CHECK(a.size(1) == a.size(2) && a.size(1) >= 1 && a.size(1) <= hb::kMaxPowerSize && iterations >= 0 && iterations < (1 << 20),
              "power_iteration: square matrices of at most 2048 rows");
  c10::cuda::CUDAGuard guard(a.device());
  at::Tensor out = at::empty({a.size(0)}, a.options().memory_format(at::MemoryFormat::Contiguous));
  check(hb::launch_power_iteration(a.data_ptr<float>(), (int)a.size(0), (int)a.size(1), (int)iterations, out.data_ptr<float>(),
                                   at::cuda::getCurrentCUDAStream()), "power_iteration launch");
  return out;
}

// x[b] *= by[b] in place; x: contiguous fp32, first dimension the batch.
void scale_matrices_(const at::Tensor& x, const at::Tensor& by) {
  TORCH_CHECK(x.is_cuda() && x.scalar_type() == at::kFloat && x.dim() >= 1 && x.is_contiguous() && x.size(0) >= 1 && x.size(0) <= 65535,
              "scale_matrices_: contiguous fp32 CUDA tensor");
  TORCH_CHECK(by.device() == x.device() && by.scalar_type() == at::kFloat && by.is_contiguous() && by.numel() == x.size(0) &&
                  at::get_overlap_status(x, by) == at::MemOverlapStatus::No, "scale_matrices_: one fp32 value per matrix");
  c10::cuda::CUDAGuard guard(x.device());
  check(hb::launch_scale_matrices(x.data_ptr<float>(), by.data_ptr<float>(), (int)x.size(0), x.numel() / x.size(0), at::cuda::getCurrentCUDAStream()),
        "scale_matrices launch");
}

// X = B T^-1 for 128 columns: b, x: fp32 [batch, rows, 128] with unit inner stride and rows on 16-byte boundaries, rows a multiple of 64; inv:
// [batch, blocks, 128, 128] contiguous, inverses of upper-triangular blocks, of which `block` is used.  x may not overlap b.
void leaf_solve(const at::Tensor& b, const at::Tensor& inv, int64_t block, const at::Tensor& x) {
  const int64_t batch = b.size(0), rows = b.dim() == 3 ? b.size(1) : 0;
  for (const at::Tensor* t : {&b, &x})
    TORCH_CHECK(t->is_cuda() && t->device() == b.device() && t->scalar_type() == at::kFloat && t->dim() == 3 && t->size(0) == batch && t->size(1) == rows &&
                    t->size(2) == hb::kQrBlock && t->stride(2) == 1 && t->stride(1) % 4 == 0 && t->stride(0) % 4 == 0 && aligned16(t->data_ptr()),
                "leaf_solve: fp32 [batch, rows, 128] CUDA tensors with rows on 16-byte boundaries");
  TORCH_CHECK(rows >= 1 && rows % hb::kQrRows == 0 && batch <= 65535, "leaf_solve: a multiple of 64 rows");
  TORCH_CHECK(inv.device() == b.device() && inv.scalar_type() == at::kFloat && inv.is_contiguous() && inv.dim() == 4 && inv.size(0) == batch && block >= 0 &&
                  block < inv.size(1) && inv.size(2) == hb::kQrBlock && inv.size(3) == hb::kQrBlock, "leaf_solve: contiguous fp32 inverses [batch, blocks, 128, 128]");
  const at::MemOverlapStatus overlap = at::get_overlap_status(b, x);
  TORCH_CHECK(overlap != at::MemOverlapStatus::Full && overlap != at::MemOverlapStatus::Partial, "leaf_solve: not in place");
  c10::cuda::CUDAGuard guard(b.device());
  hb::QrLeafSolve S{};
  S.src = b.data_ptr<float>(); S.ld = b.stride(1); S.stride = b.stride(0);
  S.inv = inv.data_ptr<float>() + block * hb::kQrBlock * hb::kQrBlock; S.stride_inv = inv.stride(0);
  S.out = x.data_ptr<float>(); S.ld_out = x.stride(1); S.stride_out = x.stride(0);
  check(hb::launch_qr_leaf_solve(S, (int)rows, (int)batch, at::cuda::getCurrentCUDAStream()), "leaf_solve launch");
}

// g + (damp + eps |g|) v for contiguous fp32 tensors of one shape.
at::Tensor dampen(const at::Tensor& g, const at::Tensor& v, double damp, double eps) {
  for (const at::Tensor* t : {&g, &v})
    TORCH_CHECK(t->is_cuda() && t->scalar_type() == at::kFloat && t->is_contiguous() && t->sizes() == g.sizes() && t->device() == g.device(),
                "dampen: contiguous fp32 CUDA tensors of one shape");
  c10::cuda::CUDAGuard guard(g.device());
  at::Tensor out = at::empty_like(g);
  check(hb::launch_dampen(g.data_ptr<float>(), v.data_ptr<float>(), out.data_ptr<float>(), g.numel(), (float)damp, (float)eps, at::cuda::getCurrentCUDAStream()),
        "dampen launch");
  return out;
}

// line -= packed upper triangle of step / ell * lr, in place.  line: contiguous fp32 [batch, n (n + 1) / 2], ell: contiguous fp32 [batch].
void triu_step_(const at::Tensor& line, const at::Tensor& step, const at::Tensor& ell, double lr) {
  check_matrices(step, "triu_step_");
  const int64_t batch = step.size(0), n = step.size(1);
  TORCH_CHECK(step.size(2) == n && line.device() == step.device() && line.scalar_type() == at::kFloat && line.is_contiguous() && line.dim() == 2 &&
                  line.size(0) == batch && line.size(1) == n * (n + 1) / 2, "triu_step_: packed triangles of the matrices' size");
  TORCH_CHECK(ell.device() == step.device() && ell.scalar_type() == at::kFloat && ell.is_contiguous() && ell.numel() == batch, "triu_step_: one fp32 divisor per matrix");
  c10::cuda::CUDAGuard guard(step.device());
  check(hb::launch_triu_step(step.data_ptr<float>(), ell.data_ptr<float>(), line.data_ptr<float>(), (int)batch, (int)n, (float)lr, at::cuda::getCurrentCUDAStream()),
        "triu_step launch");
}

// Row-major upper triangles of contiguous [batch, n, n] matrices (2- or 4-byte elements) as [batch, n (n + 1) / 2].
at::Tensor triu_pack(const at::Tensor& dense) {
  TORCH_CHECK(dense.is_cuda() && dense.dim() == 3 && dense.size(1) == dense.size(2) && dense.is_contiguous() &&
                  (dense.element_size() == 2 || dense.element_size() == 4) && dense.size(0) <= 65535,
              "triu_pack: contiguous [batch <= 65535, n, n] CUDA tensor with 2- or 4-byte elements");
  c10::cuda::CUDAGuard guard(dense.device());
  const int64_t n = dense.size(1);
  at::Tensor line = at::empty({dense.size(0), n * (n + 1) / 2}, dense.options());
  check(hb::launch_triu_pack(dense.data_ptr(), line.data_ptr(), (int)dense.element_size(), (int)dense.size(0), (int)n,
                             at::cuda::getCurrentCUDAStream()), "triu_pack launch");
  return line;
}

// Inverse of triu_pack; entries below the diagonal are zero.
at::Tensor triu_unpack(const at::Tensor& line, int64_t n) {
  TORCH_CHECK(line.is_cuda() && line.dim() == 2 && line.size(1) == n * (n + 1) / 2 && line.is_contiguous() &&
                  (line.element_size() == 2 || line.element_size() == 4) && line.size(0) <= 65535,
              "triu_unpack: contiguous [batch <= 65535, n (n + 1) / 2] CUDA tensor with 2- or 4-byte elements");
  c10::cuda::CUDAGuard guard(line.device());
  at::Tensor dense = at::empty({line.size(0), n, n}, line.options());
  check(hb::launch_triu_unpack(line.data_ptr(), dense.data_ptr(), (int)line.element_size(), (int)line.size(0), (int)n,
                               at::cuda::getCurrentCUDAStream()), "triu_unpack launch");
  return dense;
}

// fp32 column sums of a contiguous bf16 matrix [rows, cols] (cols % 8 == 0).
at::Tensor colsum_bf16(const at::Tensor& x) {
  TORCH_CHECK(x.is_cuda() && x.dim() == 2 && x.scalar_type() == at::kBFloat16 && x.is_contiguous() &&
                  x.size(1) % 8 == 0 && aligned16(x.data_ptr()), "colsum_bf16: contiguous bf16 [rows, cols], cols % 8 == 0");
  c10::cuda::CUDAGuard guard(x.device());
  at::Tensor out = at::empty({x.size(1)}, x.options().dtype(at::kFloat));
  at::Tensor partial = at::empty({hb::colsum_splits(), x.size(1)}, out.options());
  check(hb::launch_colsum_bf16(x.data_ptr(), x.size(0), (int)x.size(1), partial.data_ptr<float>(), out.data_ptr<float>(),
                               at::cuda::getCurrentCUDAStream()), "colsum launch");
  return out;
}

// Concatenated fp32 column sums of up to four contiguous bf16 matrices of one shape: out[i * cols + c].
at::Tensor colsum_bf16_batch(const std::vector<at::Tensor>& xs) {
  TORCH_CHECK(!xs.empty() && xs.size() <= (size_t)hb::kColsumMaxBatch, "colsum_bf16_batch: one to four matrices");
  const void* ptrs[hb::kColsumMaxBatch];
  for (size_t i = 0; i < xs.size(); ++i) {
    const at::Tensor& x = xs[i];
    TORCH_CHECK(x.is_cuda() && x.dim() == 2 && x.scalar_type() == at::kBFloat16 && x.is_contiguous() && x.size(1) % 8 == 0 &&
                    aligned16(x.data_ptr()) && x.sizes() == xs[0].sizes() && x.device() == xs[0].device(),
                "colsum_bf16_batch: contiguous bf16 [rows, cols] of one shape, cols % 8 == 0");
    ptrs[i] = x.data_ptr();
  }
  c10::cuda::CUDAGuard guard(xs[0].device());
  const int64_t n = (int64_t)xs.size(), cols = xs[0].size(1);
  at::Tensor out = at::empty({n * cols}, xs[0].options().dtype(at::kFloat));
  at::Tensor partial = at::empty({n, hb::colsum_splits(), cols}, out.options());
  check(hb::launch_colsum_bf16_batch(ptrs, (int)n, xs[0].size(0), (int)cols, partial.data_ptr<float>(), out.data_ptr<float>(),
                                     at::cuda::getCurrentCUDAStream()), "colsum batch launch");
  return out;
}

// y = gelu_tanh(u) for a contiguous bf16 tensor whose element count is a multiple of 8.
at::Tensor gelu_fwd(const at::Tensor& u) {
  TORCH_CHECK(u.is_cuda() && u.scalar_type() == at::kBFloat16 && u.is_contiguous() && u.numel() % 8 == 0 &&
                  aligned16(u.data_ptr()), "gelu_fwd: contiguous bf16, numel % 8 == 0");
  c10::cuda::CUDAGuard guard(u.device());
  at::Tensor y = at::empty_like(u);
  check(hb::launch_gelu_fwd(u.data_ptr(), y.data_ptr(), u.numel(), at::cuda::getCurrentCUDAStream()), "gelu_fwd launch");
  return y;
}

// (du, dbias) = (dy * gelu_tanh'(u), column sums of that product in fp32) for contiguous bf16 [rows, cols], cols % 8 == 0.
std::vector<at::Tensor> gelu_bwd(const at::Tensor& dy, const at::Tensor& u) {
  TORCH_CHECK(u.is_cuda() && u.dim() == 2 && u.scalar_type() == at::kBFloat16 && u.is_contiguous() && u.size(1) % 8 == 0 &&
                  aligned16(u.data_ptr()), "gelu_bwd: u contiguous bf16 [rows, cols], cols % 8 == 0");
  TORCH_CHECK(dy.is_cuda() && dy.scalar_type() == at::kBFloat16 && dy.is_contiguous() && dy.sizes() == u.sizes() &&
                  dy.device() == u.device() && aligned16(dy.data_ptr()), "gelu_bwd: dy like u");
  c10::cuda::CUDAGuard guard(u.device());
  const int64_t rows = u.size(0), cols = u.size(1);
  at::Tensor du = at::empty_like(u);
  at::Tensor dbias = rows > 0 ? at::empty({cols}, u.options().dtype(at::kFloat)) : at::zeros({cols}, u.options().dtype(at::kFloat));
  if (rows > 0 && cols > 0) {
    at::Tensor partial = at::empty({hb::gelu_bwd_splits(rows, (int)cols), cols}, dbias.options());
    check(hb::launch_gelu_bwd(dy.data_ptr(), u.data_ptr(), du.data_ptr(), rows, (int)cols, partial.data_ptr<float>(),
                              dbias.data_ptr<float>(), at::cuda::getCurrentCUDAStream()), "gelu_bwd launch");
  }
  return {du, dbias};
}

// LayerNorm over the last dimension of a contiguous fp32 tensor.  With `res` (same shape, bf16 or fp32) the normalised
// tensor is x + res, which is returned as a fourth tensor.  Returns (y, mean, rstd[, x + res]); y is bf16 when asked.
std::vector<at::Tensor> layer_norm_fwd(const at::Tensor& x, const OptT& res, const at::Tensor& gamma, const at::Tensor& beta,
                                       double eps, bool out_bf16) {
  const int64_t D = x.size(-1);
  TORCH_CHECK(x.is_cuda() && x.scalar_type() == at::kFloat && x.is_contiguous(), "x: contiguous fp32 CUDA tensor");
  TORCH_CHECK(hb::layer_norm_supported((int)D), "row length must be a multiple of 128, at most 1024");
  TORCH_CHECK(gamma.scalar_type() == at::kFloat && beta.scalar_type() == at::kFloat && gamma.numel() == D &&
                  beta.numel() == D && gamma.is_contiguous() && beta.is_contiguous(), "gamma / beta: fp32 [D]");
  const bool has_res = res.has_value() && res->defined();
  if (has_res)
    TORCH_CHECK(res->is_cuda() && res->is_contiguous() && res->numel() == x.numel() &&
                    (res->scalar_type() == at::kFloat || res->scalar_type() == at::kBFloat16), "res: contiguous fp32 / bf16 like x");
  c10::cuda::CUDAGuard guard(x.device());
  const int64_t rows = x.numel() / D;
  at::Tensor y = at::empty(x.sizes(), x.options().dtype(out_bf16 ? at::kBFloat16 : at::kFloat));
  at::Tensor mean = at::empty({rows}, x.options()), rstd = at::empty({rows}, x.options());
  at::Tensor xsum = has_res ? at::empty_like(x) : at::Tensor();
  check(hb::launch_layer_norm_fwd(x.data_ptr<float>(), has_res ? res->data_ptr() : nullptr,
                                  has_res && res->scalar_type() == at::kBFloat16, has_res ? xsum.data_ptr<float>() : nullptr,
                                  gamma.data_ptr<float>(), beta.data_ptr<float>(), y.data_ptr(), out_bf16,
                                  mean.data_ptr<float>(), rstd.data_ptr<float>(), rows, (int)D, (float)eps,
                                  at::cuda::getCurrentCUDAStream()), "layer_norm_fwd launch");
  if (has_res) return {y, mean, rstd, xsum};
  return {y, mean, rstd};
}

// Returns (dx, dgamma, dbeta[, bf16 copy of dx]) for dy in fp32 or bf16; `dres` (fp32, optional) is added to dx.
std::vector<at::Tensor> layer_norm_bwd(const at::Tensor& dy, const at::Tensor& x, const at::Tensor& gamma,
                                       const at::Tensor& mean, const at::Tensor& rstd, const OptT& dres, bool dx_bf16) {
  const int64_t D = x.size(-1);
  TORCH_CHECK(dy.is_cuda() && dy.is_contiguous() && dy.numel() == x.numel() &&
                  (dy.scalar_type() == at::kFloat || dy.scalar_type() == at::kBFloat16), "dy: contiguous fp32 / bf16");
  TORCH_CHECK(x.scalar_type() == at::kFloat && x.is_contiguous() && hb::layer_norm_supported((int)D), "x: contiguous fp32");
  const bool has_dres = dres.has_value() && dres->defined();
  if (has_dres)
    TORCH_CHECK(dres->is_cuda() && dres->is_contiguous() && dres->scalar_type() == at::kFloat && dres->numel() == x.numel(),
                "dres: contiguous fp32 like x");
  c10::cuda::CUDAGuard guard(x.device());
  const int64_t rows = x.numel() / D;
  const int n_cta = hb::layer_norm_partial_ctas(rows);
  at::Tensor dx = at::empty_like(x), dgamma = at::empty_like(gamma), dbeta = at::empty_like(gamma);
  at::Tensor partial = at::empty({n_cta, 2 * D}, x.options());
  at::Tensor dx16 = dx_bf16 ? at::empty(x.sizes(), x.options().dtype(at::kBFloat16)) : at::Tensor();
  check(hb::launch_layer_norm_bwd(dy.data_ptr(), dy.scalar_type() == at::kBFloat16, x.data_ptr<float>(),
                                  gamma.data_ptr<float>(), mean.data_ptr<float>(), rstd.data_ptr<float>(),
                                  has_dres ? dres->data_ptr<float>() : nullptr, dx.data_ptr<float>(),
                                  dx_bf16 ? dx16.data_ptr() : nullptr, dgamma.data_ptr<float>(), dbeta.data_ptr<float>(), partial.data_ptr<float>(), n_cta, rows,
                                  (int)D, at::cuda::getCurrentCUDAStream()), "layer_norm_bwd launch");
  if (dx_bf16) return {dx, dgamma, dbeta, dx16};
  return {dx, dgamma, dbeta};
}

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  m.def("tf32x3_matmul", &tf32x3_matmul);
  m.def("tf32_split", &tf32_split);
  m.def("tf32_gemm", &tf32_gemm);
  m.def("split16", &split16);
  m.def("split16_matmul", &split16_matmul);
  m.def("split16_accumulate", &split16_accumulate);
  m.def("split16_gemm", &split16_gemm);
  m.def("set_split16_gemm_tile", &hb::set_split16_gemm_tile_override);
  m.def("colsum_bf16", &colsum_bf16);
  m.def("colsum_bf16_batch", &colsum_bf16_batch);
  m.def("gelu_fwd", &gelu_fwd);
  m.def("gelu_bwd", &gelu_bwd);
  m.def("tall_t_mul", &tall_t_mul);
  m.def("tri_inv_blocks", &tri_inv_blocks);
  m.def("permute_columns", &permute_columns);
  m.def("identity_defect", &identity_defect);
  m.def("layer_norm_fwd", &layer_norm_fwd);
  m.def("layer_norm_bwd", &layer_norm_bwd);
  m.def("layer_norm_supported", &hb::layer_norm_supported);
  m.def("cross_entropy_", &cross_entropy_);
  m.def("scale_", &scale_);
  m.def("peer_signal", &peer_signal);
  m.def("peer_wait", &peer_wait);
  m.attr("MAX_WORLD") = hb::kMaxWorld;
  m.def("fused_chain", &fused_chain);
  m.def("sumsq", &sumsq);
  m.def("segmented_reduce", &segmented_reduce);
  m.def("ns_gemm", &ns_gemm);
  m.def("ns_orthogonalize", &ns_orthogonalize);
  m.def("set_ns_gemm_tile", &hb::set_ns_gemm_tile_override);
  m.def("set_tf32_gemm_tile", &hb::set_tf32_gemm_tile_override);
  m.def("tf32_gemm_tiles", [](int M, int N, int K, int batch, bool symmetric) {
    int choice = 0;
    check(hb::tf32_gemm_tiles(M, N, K, batch, symmetric, &choice), "tf32 tile choice");
    return choice;
  });
  m.def("chol_inv_leaf", &chol_inv_leaf);
  m.def("chol_qr_round", &chol_qr_round);
  m.def("qr_unit_columns", &qr_unit_columns);
  m.def("transposed", &transposed);
  m.def("sum_triu_diff_", &sum_triu_diff_);
  m.def("dampen", &dampen);
  m.def("power_iteration", &power_iteration);
  m.def("scale_matrices_", &scale_matrices_);
  m.def("leaf_solve", &leaf_solve);
  m.def("triu_step_", &triu_step_);
  m.def("triu_pack", &triu_pack);
  m.def("triu_unpack", &triu_unpack);
  m.def("chunk_elems", &hb::chain_chunk_elems);
}
