// A decoder layer on one GPU as one call each way: the kernels that its blocks launch one Python call at a time, in the same order on
// the same values.  For short sequences, whose layers finish sooner than the host can launch them (two layers of width 1024,
// 512 tokens: 20 autograd nodes and 78 launches at about 17 us each).  What the backward needs lies in one buffer, what either
// direction needs in between in another.  That step 1303 -> 943 us, logits of 128 tokens 256 -> 134.
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/extension.h>
namespace py = pybind11;

#include <algorithm>
#include <stdexcept>
#include <string>

#include "ody_kernels.h"
#include "scratch.h"

int* ody_status_ptr(const at::Tensor& like);
void ody_count_launches(int64_t n);

namespace {

typedef std::vector<at::Tensor> Tensors;
enum { W_IN, W_QKV, W_O, W_POST, W_GU, W_DOWN, N_WEIGHTS };      // in the order of the forward; W_IN and W_POST are the norms'

void req(bool c, const char* what) {
  if (!c) throw std::runtime_error(std::string("odysseus_transformer_b200: decoder layer: ") + what);
}
void check(int rc, const char* what) {
  if (rc != 0) throw std::runtime_error(std::string("odysseus_transformer_b200: decoder layer: ") + what + " failed with code " + std::to_string(rc));
}

// Byte ranges of one allocation, each on a 256-byte boundary
struct Carver {
  int64_t size = 0;
  int64_t take(int64_t bytes) {
    const int64_t at = size;
    size += (bytes + 255) / 256 * 256;
    return at;
  }
};

struct Layer {
  int64_t T, d, hq, hkv, q, n, I;      // tokens, width, heads, columns of q, of q|k|v, of the MLP
  // offsets in what the backward takes
  int64_t h1, rstd1, qkv, o, lse, x2, h2, rstd2, gu, act, kept_bytes;
  const at::Tensor& x;
  const Tensors& w;
  const float *cos, *sin;
  cudaStream_t st;
  int* err;

  Layer(const at::Tensor& x_, const Tensors& w_, const at::Tensor& cos_, const at::Tensor& sin_, int64_t hq_, int64_t hkv_) : x(x_), w(w_) {
    req(x.is_cuda() && x.scalar_type() == at::kBFloat16 && x.dim() == 2 && x.is_contiguous() && x.size(0) > 0 && x.size(1) > 0,
        "x must be a contiguous bfloat16 CUDA tensor [tokens, width]");
    req(w.size() == N_WEIGHTS && hq_ > 0 && hkv_ > 0 && hq_ % hkv_ == 0, "six weights, query heads a multiple of kv heads");
    T = x.size(0); d = x.size(1); hq = hq_; hkv = hkv_; q = hq * 128; n = (hq + 2 * hkv) * 128;
    req(w[W_GU].dim() == 2 && w[W_GU].size(0) % 2 == 0 && w[W_GU].size(0) > 0, "gate|up weight [2 i, width]");
    I = w[W_GU].size(0) / 2;
    const int64_t rows[N_WEIGHTS] = {d, n, d, d, 2 * I, d}, cols[N_WEIGHTS] = {0, d, q, 0, d, I};
    for (int i = 0; i < N_WEIGHTS; ++i)
      req(w[i].is_cuda() && w[i].get_device() == x.get_device() && w[i].scalar_type() == at::kBFloat16 && w[i].dim() == (cols[i] ? 2 : 1) &&
          rows_of(w[i]) && w[i].size(0) == rows[i] && (!cols[i] || w[i].size(1) == cols[i]),
          "a weight has the wrong shape, type, layout or device");
    for (const at::Tensor* t : {&cos_, &sin_})
      req(t->is_cuda() && t->get_device() == x.get_device() && t->scalar_type() == at::kFloat && t->is_contiguous() && t->dim() == 2 &&
          t->size(0) == T && t->size(1) == 64, "rope tables must be contiguous fp32 [tokens, 64] on x's device");
    req(T < (int64_t(1) << 31) && n < (int64_t(1) << 31) && 2 * I < (int64_t(1) << 31), "too large");
    Carver c;
    h1 = c.take(T * d * 2); rstd1 = c.take(T * 4); qkv = c.take(T * n * 2); o = c.take(T * q * 2); lse = c.take(hq * T * 4);
    x2 = c.take(T * d * 2); h2 = c.take(T * d * 2); rstd2 = c.take(T * 4); gu = c.take(T * 2 * I * 2); act = c.take(T * I * 2);
    kept_bytes = c.size;
    cos = cos_.data_ptr<float>();
    sin = sin_.data_ptr<float>();
    st = at::cuda::getCurrentCUDAStream().stream();
    err = ody_status_ptr(x);
  }

  // a norm's weight is packed; a projection's rows are, and may lie apart (a slice of a wider matrix)
  static bool rows_of(const at::Tensor& t) { return t.dim() == 2 ? t.stride(1) == 1 : t.is_contiguous(); }

  at::Tensor bytes(int64_t size) const { return at::empty({size}, x.options().dtype(at::kByte)); }

  static int64_t gemm_scratch(int64_t M, int64_t N, int64_t K, bool rope = false) {
    int bn, s;
    return ody_gemm_cluster_plan((int)M, (int)N, (int)K, rope, &bn, &s) ? 0 : ody_gemm_split_bytes((int)M, (int)N, (int)K);
  }
  // C = A B in `layout`, rows of B and C ldb and ldc apart, those of A packed
  void gemm(const void* A, const void* B, void* C, int64_t M, int64_t N, int64_t K, int64_t ldb, int64_t ldc, int layout, bool accumulate,
            const OdyEpilogue* epi, const ody::OptionalScratch& ws) const {
    const int64_t need = gemm_scratch(M, N, K, epi != nullptr && epi->rope_cos != nullptr);
    const bool split = need > 0 && ws.bytes >= need;
    check(ody_gemm_bf16_ws(A, B, C, (int)M, (int)N, (int)K, layout == 2 ? M : K, ldb, ldc, layout, accumulate ? 1 : 0, epi,
                           split ? ws.ptr() : nullptr, split ? ws.bytes : 0, err, st), "gemm");
    ody_count_launches(split ? 2 : 1);
  }
};

std::pair<at::Tensor, c10::optional<at::Tensor>> decoder_layer_fwd(const at::Tensor& x, const Tensors& w, const at::Tensor& cos,
                                                                   const at::Tensor& sin, int64_t hq, int64_t hkv, double eps,
                                                                   double scale, bool keep) {
  c10::cuda::CUDAGuard guard(x.device());
  const Layer L(x, w, cos, sin, hq, hkv);
  const int64_t T = L.T, d = L.d;
  at::Tensor y = at::empty_like(x), kept = L.bytes(L.kept_bytes);
  char* k = (char*)kept.data_ptr();
  const ody::OptionalScratch ws(std::max({Layer::gemm_scratch(T, L.n, d, true), Layer::gemm_scratch(T, d, L.q),
                                          Layer::gemm_scratch(T, 2 * L.I, d), Layer::gemm_scratch(T, d, L.I)}), x);
  const ody::OptionalScratch parts(ody_flash_fwd_split_bytes((int)T, (int)T, (int)hq, 1), x);
  OdyEpilogue rope = {}, res = {};
  rope.rope_cos = L.cos;
  rope.rope_sin = L.sin;
  rope.rope_rot_cols = (int)((hq + hkv) * 128);
  rope.rope_period_cols = (int)L.n;
  res.residual_ld = d;

  check(ody_rmsnorm_fwd(x.data_ptr(), nullptr, w[W_IN].data_ptr(), nullptr, k + L.h1, (float*)(k + L.rstd1), T, (int)d, (float)eps, L.st), "norm");
  auto project = [&](const void* in, int i, void* dst, const OdyEpilogue* epi) {
    L.gemm(in, w[i].data_ptr(), dst, T, w[i].size(0), w[i].size(1), w[i].stride(0), w[i].size(0), 0, false, epi, ws);
  };
  project(k + L.h1, W_QKV, k + L.qkv, &rope);
  char* q = k + L.qkv;
  check(ody_flash_fwd_parts(q, q + L.q * 2, q + (L.q + hkv * 128) * 2, k + L.o, (float*)(k + L.lse), (int)T, (int)T, (int)hq, (int)hkv, L.n, L.n,
                            L.n, L.q, 1, (float)scale, nullptr, nullptr, 0, 0, 0, parts.ptr(), parts.bytes, L.err, L.st), "attention");
  res.residual = x.data_ptr();
  project(k + L.o, W_O, k + L.x2, &res);
  check(ody_rmsnorm_fwd(k + L.x2, nullptr, w[W_POST].data_ptr(), nullptr, k + L.h2, (float*)(k + L.rstd2), T, (int)d, (float)eps, L.st), "norm");
  project(k + L.h2, W_GU, k + L.gu, nullptr);
  check(ody_swiglu_fwd(k + L.gu, k + L.act, T, L.I, L.st), "swiglu");
  res.residual = k + L.x2;
  project(k + L.act, W_DOWN, y.data_ptr(), &res);
  ody_count_launches(3 + (parts.bytes > 0 ? 2 : 1));
  if (!keep) return {y, c10::nullopt};
  return {y, kept};
}

// dx, then the weights' gradients.  out[i]: where weight i's goes (added to it with accumulate[i]; norms: written, bf16); without
// one it is returned (norms: fp32), else None.
Tensors decoder_layer_bwd(const at::Tensor& dy, const at::Tensor& x, const Tensors& w, const at::Tensor& cos, const at::Tensor& sin,
                          const at::Tensor& kept, int64_t hq, int64_t hkv, double scale, const std::vector<c10::optional<at::Tensor>>& out,
                          const std::vector<bool>& accumulate) {
  c10::cuda::CUDAGuard guard(x.device());
  const Layer L(x, w, cos, sin, hq, hkv);
  const int64_t T = L.T, d = L.d;
  req(dy.is_cuda() && dy.get_device() == x.get_device() && dy.scalar_type() == at::kBFloat16 && dy.is_contiguous() && dy.sizes() == x.sizes(),
      "the incoming gradient must match x");
  req(kept.is_cuda() && kept.get_device() == x.get_device() && kept.scalar_type() == at::kByte && kept.is_contiguous() &&
      kept.numel() == L.kept_bytes && ((uintptr_t)kept.data_ptr() & 15) == 0, "what the forward kept does not fit these sizes");
  req(out.size() == N_WEIGHTS && accumulate.size() == N_WEIGHTS, "six destinations");
  Tensors r(1 + N_WEIGHTS);
  void* dw[N_WEIGHTS];
  int64_t ld_dw[N_WEIGHTS];
  for (int i = 0; i < N_WEIGHTS; ++i) {
    const bool norm = i == W_IN || i == W_POST;
    if (out[i].has_value()) {
      const at::Tensor& t = out[i].value();
      req(t.is_cuda() && t.get_device() == x.get_device() && t.scalar_type() == at::kBFloat16 && t.sizes() == w[i].sizes() && Layer::rows_of(t),
          "a gradient's destination has the wrong shape, type, layout or device");
      dw[i] = t.data_ptr();
      ld_dw[i] = t.stride(0);
    } else {
      r[1 + i] = at::empty(w[i].sizes(), norm ? x.options().dtype(at::kFloat) : x.options());
      dw[i] = r[1 + i].data_ptr();
      ld_dw[i] = r[1 + i].stride(0);
    }
  }
  r[0] = at::empty_like(x);
  const char* k = (const char*)kept.data_ptr();
  Carver c;
  const int64_t o_dgu = c.take(T * 2 * L.I * 2), o_t1 = c.take(T * std::max(L.I, L.q) * 2), o_t2 = c.take(T * d * 2), o_dx2 = c.take(T * d * 2),
                o_dqkv = c.take(T * L.n * 2), o_norm = c.take((int64_t)ody_rmsnorm_bwd_blocks(T, (int)d) * d * 4),
                o_attn = c.take(ody_flash_bwd_workspace_bytes((int)T, (int)hq));
  const at::Tensor scratch = L.bytes(c.size);
  char* s = (char*)scratch.data_ptr();
  const ody::OptionalScratch ws(std::max({Layer::gemm_scratch(T, L.I, d), Layer::gemm_scratch(d, L.I, T), Layer::gemm_scratch(T, d, 2 * L.I),
                                          Layer::gemm_scratch(2 * L.I, d, T), Layer::gemm_scratch(T, L.q, d), Layer::gemm_scratch(d, L.q, T),
                                          Layer::gemm_scratch(T, d, L.n), Layer::gemm_scratch(L.n, d, T)}), x);
  const ody::OptionalScratch parts(ody_flash_bwd_split_bytes((int)T, (int)T, (int)hq, (int)hkv, 1), x);
  auto dgrad = [&](const void* g, int i, void* dst) {
    L.gemm(g, w[i].data_ptr(), dst, T, w[i].size(1), w[i].size(0), w[i].stride(0), w[i].size(1), 1, false, nullptr, ws);
  };
  auto wgrad = [&](const void* g, int i, const void* in) {
    L.gemm(g, in, dw[i], w[i].size(0), w[i].size(1), T, w[i].size(1), ld_dw[i], 2, out[i].has_value() && accumulate[i], nullptr, ws);
  };
  auto norm = [&](int i, const void* g, const void* in, const void* rstd, const void* ds, void* dst) {
    check(ody_rmsnorm_bwd_to(g, in, w[i].data_ptr(), (const float*)rstd, ds, dst, dw[i], out[i].has_value() ? 1 : 0, (float*)(s + o_norm), T,
                             (int)d, L.st), "norm backward");
  };
  dgrad(dy.data_ptr(), W_DOWN, s + o_t1);
  wgrad(dy.data_ptr(), W_DOWN, k + L.act);
  check(ody_swiglu_bwd(s + o_t1, k + L.gu, s + o_dgu, T, L.I, L.st), "swiglu backward");
  dgrad(s + o_dgu, W_GU, s + o_t2);
  wgrad(s + o_dgu, W_GU, k + L.h2);
  norm(W_POST, s + o_t2, k + L.x2, k + L.rstd2, dy.data_ptr(), s + o_dx2);
  dgrad(s + o_dx2, W_O, s + o_t1);
  wgrad(s + o_dx2, W_O, k + L.o);
  const char* q = k + L.qkv;
  char* dq = s + o_dqkv;
  const int64_t kc = L.q * 2, vc = (L.q + hkv * 128) * 2;
  check(ody_flash_bwd_parts(s + o_t1, q, q + kc, q + vc, k + L.o, (const float*)(k + L.lse), dq, dq + kc, dq + vc, s + o_attn, (int)T, (int)T,
                            (int)hq, (int)hkv, L.q, L.n, L.n, L.n, L.q, L.n, L.n, L.n, 1, (float)scale, nullptr, nullptr, nullptr, 0, 0,
                            parts.ptr(), parts.bytes, L.err, L.st), "attention backward");
  check(ody_rope_inplace(dq, L.cos, L.sin, T, (int)(hq + hkv), 128, L.n, 1, L.st), "rotation backward");
  dgrad(dq, W_QKV, s + o_t2);
  wgrad(dq, W_QKV, k + L.h1);
  norm(W_IN, s + o_t2, x.data_ptr(), k + L.rstd1, s + o_dx2, r[0].data_ptr());
  ody_count_launches(6 + ody_flash_bwd_launches((int)T, (int)T, (int)hq, (int)hkv, 1, parts.bytes > 0 ? 1 : 0));
  return r;
}

}  // namespace

void ody_register_layer(pybind11::module& m) {
  m.def("decoder_layer_fwd", &decoder_layer_fwd);
  m.def("decoder_layer_bwd", &decoder_layer_bwd);
}
