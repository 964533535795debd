// The training layers' autograd functions: allocation, routing and launches of the tensor-core, normalisation and attention
// kernels, forward and backward, without Python between them.
//
// One BERT layer is 12 function calls and about 25 launches; as Python autograd functions with ctypes launches that was
// 1.1 ms of host time forward and backward, five times the device time of a small batch. The arithmetic, the kernels and
// their order are those of the Python functions these replace (ops/kernels.py keeps the less used ones).
#include "layers.h"

#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/autograd/saved_variable.h>

#include <array>
#include <atomic>
#include <cstdlib>
#include <cstring>
#include <initializer_list>
#include <mutex>

extern "C" {
int gcow_gemm2_max_pairs();
int gcow_wgrad_slabs(int64_t M, int64_t N, int64_t K);
int gcow_gemm2_wgrad_slices(int M, int N, int K);
int gcow_gemm2_wgrad_sums(int N);
int gcow_gemm2_wgrad(const void* A, const void* B, float* parts, float* sums, int M, int N, int K, int lda, int ldb, int slices,
                     uint32_t* error, void* stream);
int gcow_gemm2_bf16(const void* A, const void* B, void* C, int M, int N, int K, int lda, int ldb, int ldc, const float* bias,
                    const void* residual, void* aux, int flags, uint32_t* error, int b_mn, void* stream);
int gcow_gemm_bf16(const void* A, const void* B, void* C, int M, int N, int K, int lda, int ldb, int ldc, const float* bias,
                   const void* residual, int flags, uint32_t* error, int max_ctas, int a_mn, int b_mn, int tile_rows, void* stream);
int gcow_gemm_bf16_aux(const void* A, const void* B, void* C, int M, int N, int K, int lda, int ldb, int ldc, const float* bias,
                       const void* residual, void* aux, int flags, uint32_t* error, int a_mn, int b_mn, int tile_rows, void* stream);
int gcow_gemm_bf16_batched(const void* A, const void* B, void* C, int M, int N, int K, int lda, int ldb, int ldc, int batch,
                           long long stride_a, long long stride_b, long long stride_c, const float* bias, const void* residual,
                           int flags, uint32_t* error, int a_mn, int b_mn, int tile_rows, void* stream);
int gcow_reduce_partials(const float* part, float* out, int parts, int64_t n, void* stream);
int gcow_reduce_weight_bias(const float* part, float* out, int parts, int64_t n, const float* bias_part, float* bias_out, int bias_parts,
                            int bias_n, void* stream);
int gcow_colsum_parts(int rows);
int gcow_colsum_launches(const void* g, int rows, int cols, int ld);
int gcow_colsum(const void* g, float* part, float* out, int rows, int cols, int ld, void* stream);
int gcow_cast_bf16(const float* x, void* y, uint64_t n, void* stream);
int gcow_layernorm_fwd(const void* x, const float* gamma, const float* beta, void* y, float* mean, float* rstd, int rows, int H,
                       float eps, void* stream);
int gcow_layernorm_bwd_parts(int rows);
int gcow_layernorm_bwd(const void* dy, const void* x, const float* gamma, const float* mean, const float* rstd, void* dx,
                       float* part, float* dgb, int rows, int H, void* stream);
int gcow_attention_fwd(const void* qkv, void* out, float* lse, int B, int S, int H, int d, float scale, uint32_t* error, void* stream);
int gcow_attention_bwd(const void* qkv, const void* out, const void* dout, const float* lse, float* delta, void* dqkv, int B, int S,
                       int H, int d, float scale, uint32_t* error, void* stream);
int gcow_softmax_fwd(const void* x, void* y, int64_t rows, int S, float scale, void* stream);
int gcow_softmax_bwd(const void* dp, const void* p, void* ds, int64_t rows, int S, float scale, void* stream);
int gcow_bn_parts(int64_t R, int C);
int gcow_bn_launches(int64_t R, int C, int backward, int extra);
int gcow_bn_fwd_train(const void* x, const void* residual, void* y, void* mask, const float* gamma, const float* beta, float* run_mean,
                      float* run_var, float* stats, float* part, int64_t R, int C, float eps, float momentum, int relu, void* stream);
int gcow_bn_bwd3(const void* dy, const void* dy2, const void* mask, const void* x, const float* gamma, const float* stats, void* dx,
                 void* dres, float* dgamma, float* dbeta, float* part, int64_t R, int C, int relu, void* stream);
int gcow_conv_fwd(const void* x, const void* w, void* y, const float* bias, int N, int Hin, int Win, int Ci, int Co, int kh, int kw,
                  int pad_h, int pad_w, uint32_t* error, void* stream);
int gcow_conv_fwd_strided(const void* x, const void* w, void* y, const float* bias, int N, int Hin, int Win, int Ci, int Co, int kh,
                          int kw, int pad_h, int pad_w, int stride, uint32_t* error, void* stream);
int gcow_conv_fwd_ws(const void* x, const void* w, void* y, const float* bias, int N, int H, int W, uint32_t* error, void* stream);
int gcow_conv_fwd_halo(const void* x, const void* w, void* y, const float* bias, int N, int H, int W, int Ci, uint32_t* error,
                       void* stream);
int gcow_conv_ws_usable(int N, int H, int W);
int gcow_conv_halo_usable(int N, int H, int W, int Ci);
int gcow_conv_flip_weights(const void* w, void* wt, int Co, int kh, int kw, int Ci, void* stream);
int gcow_conv_wgrad_ws_split(int N, int H, int W);
int gcow_conv_wgrad_ws(const void* dy, const void* x, float* part, int N, int H, int W, uint32_t* error, void* stream);
int gcow_conv_wgrad_halo_split(int N, int H, int W, int Ci, int Co);
int gcow_conv_wgrad_halo(const void* dy, const void* x, float* part, int N, int H, int W, int Ci, int Co, uint32_t* error,
                         void* stream);
int gcow_conv_wgrad_split(int N, int Hin, int Win, int Ci, int Co, int kh, int kw, int pad_h, int pad_w);
int gcow_conv_wgrad(const void* dy, const void* x, float* part, int N, int Hin, int Win, int Ci, int Co, int kh, int kw, int pad_h,
                    int pad_w, uint32_t* error, void* stream);
int gcow_conv_wgrad_split_strided(int N, int Hin, int Win, int Ci, int Co, int kh, int kw, int pad_h, int pad_w, int stride);
int gcow_conv_wgrad_strided(const void* dy, const void* x, float* part, int N, int Hin, int Win, int Ci, int Co, int kh, int kw,
                            int pad_h, int pad_w, int stride, uint32_t* error, void* stream);
int gcow_conv_dgrad_1x1_s2(const void* dy, const void* wt, void* dx, int N, int Hin, int Win, int Ci, int Co, uint32_t* error,
                           void* stream);
int gcow_conv_dgrad_s2(const void* dy, const void* w, void* wp, void* dx, int N, int Hin, int Win, int Ci, int Co, uint32_t* error,
                       void* stream);
}

namespace gcow_ext {

using at::Tensor;
using torch::autograd::variable_list;

namespace {

std::atomic<int64_t> g_launches{0}, g_view_hits{0};
std::mutex g_error_mu;
Tensor g_error[64];

constexpr int kOutF32 = 1, kBias = 2, kGelu = 4, kResidual = 8, kAccumulate = 16, kAuxOut = 32, kGeluGrad = 64;

void check(int err, const char* what) {
  TORCH_CHECK(err == 0, what, " refused the call: ", err);
}
inline bool env_off(const char* name) {
  const char* e = getenv(name);
  return e && !strcmp(e, "0");
}
// The current stream of a tensor's device; the guard makes that device current.
struct On {
  c10::cuda::CUDAGuard guard;
  void* stream;
  uint32_t* error;
  explicit On(const Tensor& t)
      : guard(t.device()), stream(c10::cuda::getCurrentCUDAStream(t.device().index()).stream()),
        error((uint32_t*)error_word(t.device().index()).mutable_data_ptr()) {}
};
inline Tensor empty(c10::IntArrayRef shape, at::ScalarType t, const Tensor& like) {
  return at::detail::empty_cuda(shape, t, like.device(), std::nullopt);
}
inline Tensor empty_nhwc(int64_t N, int64_t C, int64_t H, int64_t W, const Tensor& like) {
  return at::detail::empty_cuda({N, C, H, W}, at::kBFloat16, like.device(), at::MemoryFormat::ChannelsLast);
}
inline float* f32(const Tensor& t) { return t.defined() ? (float*)t.data_ptr() : nullptr; }
inline void* raw(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }
inline Tensor bf16_rows(const Tensor& t) {                  // contiguous bf16, copied only where it is not
  return (t.scalar_type() == at::kBFloat16 ? t : t.to(at::kBFloat16)).contiguous();
}
inline Tensor bf16_rows16(const Tensor& t) {                // and from a 16-byte boundary on, as the tensor maps want it
  const Tensor r = bf16_rows(t);
  return (uintptr_t)r.data_ptr() & 15 ? r.clone(at::MemoryFormat::Contiguous) : r;
}
inline Tensor float_vector(const Tensor& t) {
  return !t.defined() ? t : (t.scalar_type() == at::kFloat ? t : t.to(at::kFloat)).contiguous();
}
inline Tensor nhwc_bf16(const Tensor& t) {
  if (t.scalar_type() == at::kBFloat16 && t.is_contiguous(at::MemoryFormat::ChannelsLast)) return t;
  return t.to(at::kBFloat16).contiguous(at::MemoryFormat::ChannelsLast);
}

// ------------------------------------------------------------------------ operands
// The kernels take bare pointers: every operand has to be where x is and as long as x says, or they would read and write
// past its end.
void on_device_of(const Tensor& x, std::initializer_list<const Tensor*> others) {
  for (const Tensor* t : others)
    TORCH_CHECK(!t->defined() || t->device() == x.device(), "expected every operand on ", x.device(), ", got one on ", t->device());
}
void length(const char* what, const Tensor& t, int64_t n) {
  TORCH_CHECK(!t.defined() || t.numel() == n, what, " has ", t.numel(), " elements, expected ", n);
}
void matrix(const char* what, const Tensor& t, int64_t rows, int64_t cols) {
  TORCH_CHECK(t.dim() == 2 && t.size(0) == rows && t.size(1) == cols, what, " has shape ", t.sizes(), ", expected [", rows, ", ", cols, "]");
}
void dims(const char* what, const Tensor& t, int64_t n) {
  TORCH_CHECK(t.dim() == n, what, " has ", t.dim(), " dimensions, expected ", n);
}

// ------------------------------------------------------------------------ products
// Whether the device can co-schedule clusters of two CTAs with the pair kernel's shared memory, and GCOW_GEMM2 is not 0.
bool pair_gemm_enabled() {
  static const bool on = !env_off("GCOW_GEMM2") && gcow_gemm2_max_pairs() > 0;
  return on;
}

struct GemmOpts {
  Tensor bias, residual, pre_gelu_out, gelu_grad_of, out;
  bool gelu = false, a_t = false, b_t = false, out_f32 = false, accumulate = false;
  int max_ctas = 0, tile_rows = 0;       // of the one-CTA kernel; 0: chosen from the sizes
  int pair = -1;                         // 1: the CTA-pair kernel wherever it can, 0: never, -1: by the rule below
};

// C[M,N] = op(A) op(B)^T with the epilogues of the tcgen05 kernels.
Tensor gemm(const Tensor& a, const Tensor& b, const GemmOpts& o, const On& on) {
  TORCH_CHECK(a.dim() == 2 && b.dim() == 2 && a.scalar_type() == at::kBFloat16 && b.scalar_type() == at::kBFloat16 && a.stride(1) == 1 &&
              b.stride(1) == 1, "gemm: the operands have to be bf16 matrices with contiguous rows");
  const int64_t M = o.a_t ? a.size(1) : a.size(0), K = o.a_t ? a.size(0) : a.size(1);
  const int64_t N = o.b_t ? b.size(1) : b.size(0), Kb = o.b_t ? b.size(0) : b.size(1);
  TORCH_CHECK(K == Kb, "gemm: reduction lengths differ");
  Tensor out = o.out.defined() ? o.out : empty({M, N}, o.out_f32 ? at::kFloat : at::kBFloat16, a);
  const Tensor& aux = o.pre_gelu_out.defined() ? o.pre_gelu_out : o.gelu_grad_of;
  TORCH_CHECK(out.dim() == 2 && out.size(0) == M && out.size(1) == N, "gemm: the result has another shape than the product");
  TORCH_CHECK(out.scalar_type() == at::kFloat || out.scalar_type() == at::kBFloat16, "gemm: the result has to be float32 or bf16");
  TORCH_CHECK(!o.bias.defined() || (o.bias.numel() == N && o.bias.scalar_type() == at::kFloat && o.bias.is_contiguous()),
              "gemm: the bias has to be a float32 vector as long as the product's rows");
  TORCH_CHECK(!o.residual.defined() || (o.residual.sizes() == out.sizes() && o.residual.strides() == out.strides() &&
                                        o.residual.scalar_type() == out.scalar_type()),
              "gemm: the residual has another shape or type than the product");
  TORCH_CHECK(!(o.pre_gelu_out.defined() && o.gelu_grad_of.defined()), "gemm: one side tensor of the GELU at a time");
  TORCH_CHECK(!aux.defined() || (aux.scalar_type() == at::kBFloat16 && aux.sizes() == out.sizes() && aux.strides() == out.strides()),
              "gemm: the GELU's side tensor has another shape or type than the product");
  on_device_of(a, {&b, &out, &o.bias, &o.residual, &aux});
  int flags = (out.scalar_type() == at::kFloat ? kOutF32 : 0) | (o.bias.defined() ? kBias : 0) | (o.gelu ? kGelu : 0) |
              (o.residual.defined() ? kResidual : 0) | (o.accumulate ? kAccumulate : 0);
  if (aux.defined()) flags |= o.pre_gelu_out.defined() ? kAuxOut : kGeluGrad;
  const int lda = (int)a.stride(0), ldb = (int)b.stride(0), ldc = (int)out.stride(0);
  // A large product goes to CTA pairs: two SMs per 256 x 256 tile have the one-CTA tile's traffic per flop and an overlapped
  // epilogue as well. Where nothing but a bias follows, the one-CTA tile's main loop is the faster one the longer the reduction, so the pairs
  // need the finer rounds that they come with (74 tiles at twice the pace instead of 148). `even`: they have none. One-CTA tile, pairs, each
  // by itself, us, single launches / back to back:
  //   pairs: 16384 x 1024 x 4096 107.6, 100.4 / 116.3, 116.7; x 768 x 3072 79.9, 63.5 / 80.9, 69.7; 4096^3 106.5, 99.3 / 112.4, 110.2;
  //   4096 x 8192 x 5120 243.7, 217.1 / 276, 254; 16384 x 2048 x 8192 377, 358 / 435, 433; even, 8192 x 8192 x 4096 363, 367 / 432, 425; with at most
  //   two rounds, 16384 x 1024 x 6144 152, 144 / 170, 171;
  //   one-CTA: even, 8192 x 8192 x 5120 451, 469 / 535, 533, x 6144 543, 569 / 639, 652, x 8192 713, 770 / 843, 875; 4096 x 4096 x 8192 194.6, 192.5 / 220, 227;
  //   a single round, 2048 x 4096 x 4096 57, 57 / 56.0, 57.5.
  // A single round that leaves pairs idle, short and wide, plain or with a bias, stays there too: 1024 x 4096 x 512 6.9, 7.7, 2048 x 2048 x 768 8.4, 9.1, 4096 x
  // 768 x 768 8.8, 9.2; from 1536 rows of reduction on, or with 512 columns, the two are even (8192 x 512 x 768 10.5, 10.3).
  // Shorter, narrower and lower products (K < 512, N < 256, M < 1024; one-CTA tile, pairs in a graph). A residual, a kept argument or a GELU' factor, which
  // the one-CTA kernel's lanes read and write themselves: pairs from 64 columns on, 1 x 1024 x 1024 with a residual 12.1, 7.1, 300 x 1024 x 1024
  // 15.4, 7.9, 16384 x 1024 x 256 46.5, 18.0, 200704 x 512 x 128 261, 84; 32 columns 16384 x 32 x 64 5.5, 6.4. Others, whose results leave by the TMA
  // on both: pairs where a round's tiles are few (a pair fetches twice as much at once: 128 x 1024 x 1024 9.4, 6.6, 1024 x 256 x 64 5.0, 4.4; up to 8
  // tiles with 64 columns, 24 with 128, 37 with 256) and where there are several rounds of 256 columns (50176 x 1024 x 256 32.7, 28.7, with a bias
  // 38.0, 33.0; 12544 x 2048 x 256 19.1, 15.9); a single round of more than 37 tiles is one of twice as many CTAs without pairs' start (16384 x 256 x 64 5.2,
  // 6.2, 4096 x 768 x 256 6.3, 6.6). On one CTA: plain, 64 columns deep in few rounds 8192 x 1024 x 64 7.0, 7.2; plain with 524288 rows and more, where the two
  // are uneven (524288 x 256 x 256 88.1, 90.5, 802816 x 256 x 256 134.9, 140.5, 1204224 x 256 x 128 152, 159, but 602112 x 256 x 256 120.6, 105.0, 802816 x 256 x 128 147, 116, x 64 84.4, 90.7
  // and 136.6, 125.7 on two days; 401408 x 256 x 256 73.3, 70.5); a single row of 4096 columns or more (x 1024 9.5, 9.8; 8192 x 4096 23.3, 32.5).
  // Few rows of a wide result (`wide`). Up to 128 rows, and from 257 to 384, half of a pair, or of one pair in two, has no rows, while the one-CTA kernel's tiles
  // of 128 rows fit: 64 x 30528 x 768 12.1, 15.4, 128 x 50304 x 256 12.0, 13.6, 300 x 50304 x 256 with a bias 20.7, 25.9; where those are one round of CTAs, pairs need two: 300
  // x 12288 x 4096 32.4, 43.6. Pairs all the same: deep and wide 128 x 50304 x 2048 55, 45, and with a residual, a kept argument or a GELU' factor 64 x 30528 x 768 19.2, 16.5.
  // Up to 16 rows pairs wait for their short A (less than 64 K elements of it): 2 x 6144 x 4096 27.4, 32.1, 8 x 30528 x 4096 with a residual 55.9, 76.6; 16 x 8192 x 4096
  // 28.1, 21.5.
  const bool can_pair = pair_gemm_enabled() && !o.a_t && !(flags & (kOutF32 | kAccumulate)) && !o.max_ctas && !o.tile_rows;
  const int64_t tiles = ((M + 255) / 256) * ((N + 255) / 256);
  const bool even = 2 * ((tiles + 147) / 148) <= (tiles + 73) / 74;
  const bool one_cta = !(flags & (kGelu | kResidual | kGeluGrad)) && tiles >= 118 && even &&
                       (K >= 8192 || (K > 4096 && tiles > 296) || (K >= 2048 && tiles <= 148));
  const bool fits = K % 64 == 0 && N % (o.b_t ? 64 : 32) == 0 && lda % 8 == 0 && ldb % 8 == 0 && ldc % 8 == 0;
  const bool bare = !(flags & (kGelu | kResidual | kGeluGrad | kAuxOut)), plain = bare && !(flags & kBias), short_round = tiles > 37 && tiles <= 74;
  const bool side = flags & (kResidual | kGeluGrad | kAuxOut), low = M <= 128 || (M > 256 && M <= 384);
  const bool wide = M >= 1024 || tiles <= 16 ? false
                    : tiles <= 37            ? M <= 16 && M * K < 65536 && (K >= 2048 || (bare && (K >= 512 || tiles > 24)))
                    : side                   ? M <= 8 || (M * K < 65536 && K >= 1536)
                    : tiles <= 74            ? false
                    : M <= 128               ? tiles <= 148 || K < 2048 || M * K < 65536
                                             : ((M + 127) / 128) * ((N + 255) / 256) <= 148 || (low && K < 2048 && K >= (bare ? 128 : 1024));
  const bool by_rule = fits && (M > 1 || N <= 3072) &&
                       (K >= 512 && M >= 1024 && N >= 256 ? !one_cta && !(bare && short_round && K <= 768 && N >= 768)
                        : wide                            ? false
                        : side                            ? N >= 64
                        : tiles <= 8                      ? N >= 64
                        : tiles <= 24                     ? N >= 128
                        : tiles <= 37                     ? N >= 256 && K >= 128
                                                          : !short_round && N >= 256 && !(plain && (M >= 524288 || (K < 128 && tiles <= 148))));
  if (can_pair && (o.pair < 0 ? by_rule : o.pair > 0)) {
    const int err = gcow_gemm2_bf16(a.data_ptr(), b.data_ptr(), out.data_ptr(), (int)M, (int)N, (int)K, lda, ldb, ldc, f32(o.bias),
                                    raw(o.residual), raw(aux), flags, on.error, o.b_t, on.stream);
    if (err == 0) { g_launches++; return out; }
    TORCH_CHECK(err == -2, "gcow_gemm2_bf16 refused the call: ", err);
  }
  if (aux.defined())
    check(gcow_gemm_bf16_aux(a.data_ptr(), b.data_ptr(), out.data_ptr(), (int)M, (int)N, (int)K, lda, ldb, ldc, f32(o.bias),
                             raw(o.residual), raw(aux), flags, on.error, o.a_t, o.b_t, o.tile_rows, on.stream), "gcow_gemm_bf16_aux");
  else
    check(gcow_gemm_bf16(a.data_ptr(), b.data_ptr(), out.data_ptr(), (int)M, (int)N, (int)K, lda, ldb, ldc, f32(o.bias),
                         raw(o.residual), flags, on.error, o.max_ctas, o.a_t, o.b_t, o.tile_rows, on.stream), "gcow_gemm_bf16");
  g_launches++;
  return out;
}

// Ordered sum of `parts` fp32 partial results into `out` (allocated when undefined).
Tensor add_parts(const Tensor& part, int64_t parts, c10::IntArrayRef shape, Tensor out, const On& on) {
  if (!out.defined()) out = empty(shape, at::kFloat, part);
  check(gcow_reduce_partials(f32(part), f32(out), (int)parts, out.numel(), on.stream), "gcow_reduce_partials");
  g_launches++;
  return out;
}

// dW[N,K] = g^T x, fp32, for g [M,N] and x [M,K], both stored with the reduction dimension M outermost. The result has few tiles
// while M is long, so the rows are cut into slices whose products are added in order: on CTA pairs in one launch, else as
// slabs of one batched launch. With `bias` CTA pairs add up the columns of g as they pass (*bias: the result, which stays undefined otherwise).
Tensor wgrad(const Tensor& g, const Tensor& x, const Tensor& out, const On& on, Tensor* bias = nullptr) {
  TORCH_CHECK(g.dim() == 2 && x.dim() == 2 && g.size(0) == x.size(0) && g.scalar_type() == at::kBFloat16 && x.scalar_type() == at::kBFloat16 &&
              g.stride(1) == 1 && x.stride(1) == 1, "wgrad: expected two bf16 matrices with contiguous rows, as many in each");
  const int64_t M = g.size(0), N = g.size(1), K = x.size(1);
  TORCH_CHECK(!out.defined() || (out.dim() == 2 && out.size(0) == N && out.size(1) == K && out.scalar_type() == at::kFloat && out.is_contiguous()),
              "wgrad: the result has to be a contiguous float32 matrix of the product's shape");
  on_device_of(g, {&x, &out});
  const int slices = pair_gemm_enabled() && M <= 0x7fffffff && N <= 0x7fffffff && K <= 0x7fffffff && g.stride(0) % 8 == 0 && x.stride(0) % 8 == 0 &&
                             !((uintptr_t)g.data_ptr() & 15) && !((uintptr_t)x.data_ptr() & 15) && !(out.defined() && ((uintptr_t)out.data_ptr() & 15))
                         ? gcow_gemm2_wgrad_slices((int)N, (int)K, (int)M) : 0;
  if (slices > 0) {                                          // CTA pairs, which cut the rows themselves
    const Tensor to = slices == 1 && out.defined() ? out : empty({slices, N, K}, at::kFloat, g);
    const int64_t bias_parts = bias ? slices * gcow_gemm2_wgrad_sums((int)K) : 0;
    if (!bias_parts) bias = nullptr;
    const Tensor sums = bias ? empty({bias_parts, N}, at::kFloat, g) : Tensor();
    check(gcow_gemm2_wgrad(g.data_ptr(), x.data_ptr(), f32(to), f32(sums), (int)N, (int)K, (int)M, (int)g.stride(0), (int)x.stride(0), slices,
                           on.error, on.stream), "gcow_gemm2_wgrad");
    g_launches++;
    if (bias) {                                              // N and K are multiples of 64
      const Tensor dw = slices > 1 && !out.defined() ? empty({N, K}, at::kFloat, g) : out;
      *bias = empty({N}, at::kFloat, g);
      check(gcow_reduce_weight_bias(f32(to), slices > 1 ? f32(dw) : nullptr, slices > 1 ? slices : 0, slices > 1 ? N * K : 0, f32(sums), f32(*bias), (int)bias_parts,
                                    (int)N, on.stream), "gcow_reduce_weight_bias");
      g_launches++;
      return slices > 1 || out.defined() ? dw : to.view({N, K});
    }
    return slices > 1 ? add_parts(to, slices, {N, K}, out, on) : out.defined() ? out : to.view({N, K});
  }
  const int64_t s = gcow_wgrad_slabs(N, K, M);
  if (s == 1 || g.stride(0) != N || x.stride(0) != K) {
    GemmOpts o;
    o.a_t = o.b_t = o.out_f32 = true;
    o.out = out;
    return gemm(g, x, o, on);
  }
  const Tensor part = empty({s, N, K}, at::kFloat, g);
  const int64_t m = M / s;
  check(gcow_gemm_bf16_batched(g.data_ptr(), x.data_ptr(), part.data_ptr(), (int)N, (int)K, (int)m, (int)N, (int)K, (int)K, (int)s,
                               m * N, m * K, N * K, nullptr, nullptr, kOutF32, on.error, 1, 1, 0, on.stream), "gcow_gemm_bf16_batched");
  g_launches++;
  return add_parts(part, s, {N, K}, out, on);
}

// fp32 column sums of a bf16 matrix (bias gradient)
Tensor colsum(const Tensor& g, const On& on) {
  const int64_t rows = g.size(0), cols = g.size(1);
  if (cols % 2 || g.stride(1) != 1 || g.stride(0) % 2) return g.to(at::kFloat).sum(0);
  TORCH_CHECK(g.dim() == 2 && g.scalar_type() == at::kBFloat16, "colsum: expected a bf16 matrix");
  const int launches = gcow_colsum_launches(g.data_ptr(), (int)rows, (int)cols, (int)g.stride(0));
  const Tensor part = launches > 1 ? empty({gcow_colsum_parts((int)rows) * cols}, at::kFloat, g) : Tensor(), out = empty({cols}, at::kFloat, g);
  check(gcow_colsum(g.data_ptr(), f32(part), f32(out), (int)rows, (int)cols, (int)g.stride(0), on.stream), "gcow_colsum");
  g_launches += launches;
  return out;
}

// ------------------------------------------------------- weights: bf16 copies, gradient targets
PyObject* name_bf16() { static PyObject* s = PyUnicode_InternFromString("_gcow_bf16"); return s; }
PyObject* name_version() { static PyObject* s = PyUnicode_InternFromString("_gcow_bf16_version"); return s; }
PyObject* name_view() { static PyObject* s = PyUnicode_InternFromString("_gcow_grad_view"); return s; }

// An attribute of a parameter object, or null (no error set) where there is none.
PyObject* attr(PyObject* o, PyObject* name) {
  PyObject* v = PyObject_GetAttr(o, name);
  if (!v) PyErr_Clear();
  return v;
}

// A weight in bf16, in its own element order. Not counted in g_launches: whether a layer needs it depends on whether an optimiser keeps the
// copy, or which types torch casts, and the count is of the layers' own work.
Tensor cast_bf16(const Tensor& d) {
  if (d.scalar_type() != at::kFloat || !d.is_non_overlapping_and_dense()) return d.to(at::kBFloat16);
  const Tensor out = at::detail::empty_strided_cuda(d.sizes(), d.strides(), at::TensorOptions(d.device()).dtype(at::kBFloat16));
  check(gcow_cast_bf16((const float*)d.const_data_ptr(), out.mutable_data_ptr(), (uint64_t)d.numel(),
                       c10::cuda::getCurrentCUDAStream(d.device().index()).stream()), "gcow_cast_bf16");
  return out;
}

// ops/kernels.py::bf16_weight, for the weights of the layers below
Tensor bf16_weight(PyObject* obj) {
  const Tensor& w = THPVariable_Unpack(obj);
  PyObject* sh = attr(obj, name_bf16());
  if (!sh || !THPVariable_Check(sh) || w.scalar_type() != at::kFloat || THPVariable_Unpack(sh).sizes() != w.sizes() ||
      THPVariable_Unpack(sh).device() != w.device()) {
    Py_XDECREF(sh);
    const Tensor d = w.detach();
    return d.scalar_type() == at::kBFloat16 ? d : cast_bf16(d);
  }
  Tensor copy = THPVariable_Unpack(sh);
  Py_DECREF(sh);
  PyObject* ver = attr(obj, name_version());
  const long have = ver ? PyLong_AsLong(ver) : -1;
  Py_XDECREF(ver);
  PyErr_Clear();
  const long now = (long)w._version();
  if (have != now) {
    at::NoGradGuard no_grad;
    copy.copy_(w.detach());
    PyObject* v = PyLong_FromLong(now);
    if (PyObject_SetAttr(obj, name_version(), v)) PyErr_Clear();
    Py_DECREF(v);
  }
  return copy;
}

// The float32 tensor this step's gradient of a weight may be written into, or none. A trainer that knows where the gradient
// will end up (DDP's bucket view, i.e. last step's .grad) leaves it in the weight's _gcow_grad_view before it drops the
// gradients; the first layer to use the weight in a forward pass takes it, so two uses of one weight never share it. The
// weight-gradient kernels then write there and the backward returns an alias of that memory: autograd adopts it as the
// weight's .grad and DDP, seeing its own bucket memory, copies nothing.
Tensor take_grad_view(PyObject* obj) {
  const Tensor& w = THPVariable_Unpack(obj);
  if (w.scalar_type() != at::kFloat) return Tensor();
  PyObject* v = attr(obj, name_view());
  if (!v || v == Py_None || !THPVariable_Check(v)) { Py_XDECREF(v); return Tensor(); }
  Tensor gv = THPVariable_Unpack(v);
  Py_DECREF(v);
  if (PyObject_SetAttr(obj, name_view(), Py_None)) PyErr_Clear();
  if (gv.scalar_type() != at::kFloat || gv.sizes() != w.sizes() || gv.device() != w.device()) return Tensor();
  return gv;
}

// A gradient target held by a backward function. `w` is the weight itself: its .grad tells whether gradients accumulate.
struct Target { Tensor view, weight; };

// The [rows, cols] fp32 matrix to write (undefined where there is none) and the tensor to return as the gradient. `align`: what
// the writing kernel needs of the address (the GEMM and convolution epilogues store 16 bytes at a time).
Tensor target_matrix(const Target& t, int64_t rows, int64_t cols, uintptr_t align, Tensor* result) {
  if (!t.view.defined() || t.weight.grad().defined()) return Tensor();
  const Tensor flat = t.view.dim() == 4 ? t.view.permute({0, 2, 3, 1}) : t.view;
  if (!flat.is_contiguous() || flat.numel() != rows * cols || (uintptr_t)t.view.data_ptr() % align) return Tensor();
  g_view_hits++;
  *result = t.view.as_strided(t.view.sizes(), t.view.strides());
  return flat.view({rows, cols});
}

// ---------------------------------------------------------------------- autograd nodes
// A tensor kept for the backward pass. SavedVariable runs the saved-tensor hooks in force (activation offload and
// checkpointing work through them), catches in-place writes in between and breaks the cycle between a node and its output.
struct Kept {
  torch::autograd::SavedVariable saved;
  void set(const Tensor& x, bool is_output = false) { saved = torch::autograd::SavedVariable(x, is_output); }
};
constexpr int kKeep = 6;
using Saved = std::array<Tensor, kKeep>;                    // what a node kept, unpacked

// Backward nodes: `kept` holds the saved tensors, inputs are numbered in the order given to record().
struct LayerNode : torch::autograd::Node {
  Kept kept[kKeep];
  Target target[2];
  bool released = false;
  void release_variables() override {
    for (auto& k : kept) k.saved.reset_data();
    for (auto& t : target) { t.view.reset(); t.weight.reset(); }
    released = true;
  }
  bool wants(size_t i) { return task_should_compute_output(i); }
  // At least one of g is defined; `had`: the saved tensors.
  virtual variable_list grads(variable_list&& g, const Saved& had) = 0;
  variable_list apply(variable_list&& g) override {
    bool any = false;
    for (const Tensor& t : g) any = any || t.defined();
    if (!any) return variable_list(num_outputs());
    TORCH_CHECK(!released, torch::autograd::ERR_BACKWARD_TWICE);
    // Before the guards: an unpack hook is the user's code, and a checkpoint's reruns the forward pass of its region, whose
    // operators have to record their history.
    Saved had;
    for (int i = 0; i < kKeep; i++) had[i] = kept[i].saved.unpack(shared_from_this());
    at::NoGradGuard no_grad;
    at::AutoDispatchBelowADInplaceOrView below;
    return grads(std::move(g), had);
  }
};

template <class N, class... In>
std::shared_ptr<N> record(const In&... in) {
  const Tensor* const all[] = {&in...};
  for (const Tensor* t : all)
    TORCH_CHECK_NOT_IMPLEMENTED(!t->defined() || !t->_fw_grad(0).defined(), "forward-mode AD is not implemented for this layer function");
  if (!at::GradMode::is_enabled() || !torch::autograd::compute_requires_grad(in...)) return nullptr;
  std::shared_ptr<N> n(new N(), torch::autograd::deleteNode);
  n->set_next_edges(torch::autograd::collect_next_edges(in...));
  return n;
}
// Everything up to the history of the result runs without gradients, as in the forward of a Python function; views are
// still tracked, so that a saved view of an input shares the input's version counter.
struct Below {
  at::NoGradGuard no_grad;
};
template <class N>
PyObject* finish(Tensor out, const std::shared_ptr<N>& n) {
  if (n) torch::autograd::set_history(out, n);
  return THPVariable_Wrap(std::move(out));
}
inline Tensor arg(PyObject* o) {                            // None: undefined
  TORCH_CHECK_TYPE(o == Py_None || THPVariable_Check(o), "expected a tensor, got ", Py_TYPE(o)->tp_name);
  return o == Py_None ? Tensor() : in_memory(THPVariable_Unpack(o));
}
inline Tensor need(PyObject* o) {
  TORCH_CHECK_TYPE(o != Py_None, "expected a tensor, got None");
  return arg(o);
}
inline Tensor rows_of(const Tensor& x) { return bf16_rows(x.reshape({-1, x.size(-1)})); }
inline Tensor as_rows(const Tensor& x) { return x.view({-1, x.size(-1)}); }
inline std::vector<int64_t> with_last(const Tensor& x, int64_t last) {
  std::vector<int64_t> s = x.sizes().vec();
  s.back() = last;
  return s;
}

// The gradients of a linear layer's weight, into the trainer's target where there is one, else a new tensor, and of its bias, as far as they are
// wanted.
void linear_wgrad(const Target& t, const Tensor& g, const Tensor& x, bool want_weight, bool want_bias, Tensor* weight, Tensor* bias, const On& on) {
  if (want_weight) {
    Tensor result;
    const Tensor flat = target_matrix(t, g.size(1), x.size(1), 16, &result), dw = wgrad(g, x, flat, on, want_bias ? bias : nullptr);
    *weight = flat.defined() ? result : dw;
  }
  if (want_bias && !bias->defined()) *bias = colsum(g, on);
}

// ---------------------------------------------------------------------- linear layers
struct LinearNode : LayerNode {                             // inputs: x, w, b, residual; outputs: y and, forked, x again
  std::vector<int64_t> x_shape;
  bool has_bias = false, has_res = false;
  std::string name() const override { return "GcowLinearBackward"; }
  variable_list grads(variable_list&& in, const Saved& had) override {
    variable_list out(4);
    const Tensor &xb = had[0], &wb = had[1];
    const On on(xb);
    const Tensor other = in.size() > 1 ? in[1] : Tensor();  // x's other gradient
    if (!in[0].defined()) {
      if (wants(0)) out[0] = other;
      return out;
    }
    const Tensor g = rows_of(in[0]);
    if (wants(0)) {                                         // dx[M,K] = g[M,N] W[N,K] (+ other): W is stored [reduction N][K]
      GemmOpts o;
      o.b_t = true;
      if (other.defined()) o.residual = as_rows(bf16_rows16(other));
      o.out = empty(x_shape, at::kBFloat16, g);
      Tensor full = o.out;
      o.out = as_rows(full);
      gemm(g, wb, o, on);
      out[0] = std::move(full);
    }
    linear_wgrad(target[0], g, xb, wants(1), has_bias && wants(2), &out[1], &out[2], on);
    if (has_res && wants(3)) out[3] = in[0];
    return out;
  }
};

// linear(x, w, b or None, residual or None): x W^T + b (+ residual, in the epilogue)
// linear(x, w, b or None, None, True): that and a second tensor on x's memory, for the other consumer of a bf16 x. The two gradients then come
// to this layer's node, and the data gradient's epilogue adds the other one; autograd would add them with a kernel of its own.
PyObject* linear(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  TORCH_CHECK(nargs == 4 || nargs == 5, "linear: bad arguments");
  const Tensor x = need(args[0]), w = need(args[1]), b = arg(args[2]), r = arg(args[3]);
  const bool fork = nargs == 5 && PyObject_IsTrue(args[4]) == 1;
  TORCH_CHECK(!fork || (!r.defined() && x.scalar_type() == at::kBFloat16), "linear: the second result goes with a bf16 input and no residual");
  TORCH_CHECK(x.dim() >= 1, "linear: the input has no dimensions");
  on_device_of(x, {&w, &b, &r});
  dims("linear: the weight", w, 2);
  matrix("linear: the weight", w, w.size(0), x.size(-1));
  length("linear: the bias", b, w.size(0));
  TORCH_CHECK(!r.defined() || (r.dim() >= 1 && r.size(-1) == w.size(0)), "linear: the residual's rows have another length than the result's");
  auto node = record<LinearNode>(x, w, b, r);
  Tensor out;
  {
    Below below;
    const On on(x);
    const Tensor xb = rows_of(x), wb = bf16_weight(args[1]).contiguous();
    out = empty(r.defined() ? r.sizes().vec() : with_last(x, w.size(0)), at::kBFloat16, x);
    GemmOpts o;
    o.bias = float_vector(b);
    if (r.defined()) o.residual = rows_of(r);
    o.out = as_rows(out);
    gemm(xb, wb, o, on);
    if (node) {
      node->kept[0].set(xb);
      node->kept[1].set(wb);
      node->x_shape = x.sizes().vec();
      node->has_bias = b.defined();
      node->has_res = r.defined();
      node->target[0] = {take_grad_view(args[1]), w};
    }
  }
  if (fork) {
    Tensor again = x.variable_data();                       // the same memory, no autograd view of x
    torch::autograd::impl::set_version_counter(again, torch::autograd::impl::version_counter(x));   // a change of it is one of the saved input
    if (node) {
      torch::autograd::set_history(out, node);
      torch::autograd::set_history(again, node);
    }
    PyObject *y = THPVariable_Wrap(std::move(out)), *z = THPVariable_Wrap(std::move(again));
    PyObject* pair = y && z ? PyTuple_Pack(2, y, z) : nullptr;
    Py_XDECREF(y);
    Py_XDECREF(z);
    return pair;
  }
  return finish(std::move(out), node);
  END_HANDLE_TH_ERRORS
}

struct FfnNode : LayerNode {                                // inputs: x, w1, b1, w2, b2
  std::vector<int64_t> shape;
  std::string name() const override { return "GcowFfnBackward"; }
  variable_list grads(variable_list&& in, const Saved& had) override {
    variable_list out(5);
    const Tensor &xb = had[0], &w1b = had[1], &w2b = had[2], &pre = had[3], &act = had[4];
    const On on(xb);
    const Tensor g = rows_of(in[0]);
    GemmOpts o;
    o.b_t = true;
    o.gelu_grad_of = pre;
    const Tensor dpre = gemm(g, w2b, o, on);                // (g W2) * GELU'(pre)
    linear_wgrad(target[1], g, act, wants(3), wants(4), &out[3], &out[4], on);
    if (wants(0)) {
      Tensor full = empty(shape, at::kBFloat16, g);
      GemmOpts q;
      q.b_t = true;
      q.residual = g;
      q.out = as_rows(full);
      gemm(dpre, w1b, q, on);
      out[0] = std::move(full);
    }
    linear_wgrad(target[0], dpre, xb, wants(1), wants(2), &out[1], &out[2], on);
    return out;
  }
};

// ffn_residual(x, w1, b1, w2, b2): x + GELU(x W1^T + b1) W2^T + b2
PyObject* ffn_residual(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  TORCH_CHECK(nargs == 5, "ffn_residual: bad arguments");
  const Tensor x = need(args[0]), w1 = need(args[1]), b1 = need(args[2]), w2 = need(args[3]), b2 = need(args[4]);
  TORCH_CHECK(x.dim() >= 1, "ffn_residual: the input has no dimensions");
  on_device_of(x, {&w1, &b1, &w2, &b2});
  dims("ffn_residual: the first weight", w1, 2);
  matrix("ffn_residual: the first weight", w1, w1.size(0), x.size(-1));
  matrix("ffn_residual: the second weight", w2, x.size(-1), w1.size(0));
  length("ffn_residual: the first bias", b1, w1.size(0));
  length("ffn_residual: the second bias", b2, w2.size(0));
  auto node = record<FfnNode>(x, w1, b1, w2, b2);
  Tensor out;
  {
    Below below;
    const On on(x);
    const Tensor xb = rows_of(x), w1b = bf16_weight(args[1]).contiguous(), w2b = bf16_weight(args[3]).contiguous();
    GemmOpts o;
    o.bias = float_vector(b1);
    o.gelu = true;
    o.pre_gelu_out = empty({xb.size(0), w1b.size(0)}, at::kBFloat16, x);
    const Tensor act = gemm(xb, w1b, o, on);
    out = empty(x.sizes(), at::kBFloat16, x);
    GemmOpts q;
    q.bias = float_vector(b2);
    q.residual = xb;
    q.out = as_rows(out);
    gemm(act, w2b, q, on);
    if (node) {
      const Tensor all[5] = {xb, w1b, w2b, o.pre_gelu_out, act};
      for (int i = 0; i < 5; i++) node->kept[i].set(all[i]);
      node->shape = x.sizes().vec();
      node->target[0] = {take_grad_view(args[1]), w1};
      node->target[1] = {take_grad_view(args[3]), w2};
    }
  }
  return finish(std::move(out), node);
  END_HANDLE_TH_ERRORS
}

// ---------------------------------------------------------------------- LayerNorm
struct LayerNormNode : LayerNode {                          // inputs: x, gamma, beta
  std::vector<int64_t> shape;
  at::ScalarType ptype = at::kFloat;
  std::string name() const override { return "GcowLayerNormBackward"; }
  variable_list grads(variable_list&& in, const Saved& had) override {
    variable_list out(3);
    const Tensor &xb = had[0], &g32 = had[1], &mean = had[2], &rstd = had[3];
    const On on(xb);
    const int64_t rows = xb.size(0), H = xb.size(1);
    const Tensor g = rows_of(in[0]);
    Tensor dx = empty(shape, at::kBFloat16, xb);
    const Tensor part = empty({gcow_layernorm_bwd_parts((int)rows) * 2 * H}, at::kFloat, xb), dgb = empty({2 * H}, at::kFloat, xb);
    check(gcow_layernorm_bwd(g.data_ptr(), xb.data_ptr(), f32(g32), f32(mean), f32(rstd), dx.data_ptr(), f32(part), f32(dgb), (int)rows,
                             (int)H, on.stream), "gcow_layernorm_bwd");
    g_launches += 2;
    out[0] = std::move(dx);
    out[1] = dgb.narrow(0, 0, H).to(ptype);
    out[2] = dgb.narrow(0, H, H).to(ptype);
    return out;
  }
};

PyObject* layernorm(PyObject*, PyObject* const* args, Py_ssize_t nargs) {      // (x, gamma, beta, eps)
  HANDLE_TH_ERRORS
  TORCH_CHECK(nargs == 4, "layernorm: bad arguments");
  const Tensor x = need(args[0]), gamma = need(args[1]), beta = need(args[2]);
  const double eps = PyFloat_AsDouble(args[3]);
  if (PyErr_Occurred()) return nullptr;
  TORCH_CHECK(x.dim() >= 1, "layernorm: the input has no dimensions");
  on_device_of(x, {&gamma, &beta});
  length("layernorm: gamma", gamma, x.size(-1));
  length("layernorm: beta", beta, x.size(-1));
  auto node = record<LayerNormNode>(x, gamma, beta);
  Tensor out;
  {
    Below below;
    const On on(x);
    const Tensor xb = rows_of(x), g32 = float_vector(gamma), b32 = float_vector(beta);
    const int64_t rows = xb.size(0), H = xb.size(1);
    out = empty(x.sizes(), at::kBFloat16, x);
    const Tensor mean = empty({rows}, at::kFloat, x), rstd = empty({rows}, at::kFloat, x);
    check(gcow_layernorm_fwd(xb.data_ptr(), f32(g32), f32(b32), out.data_ptr(), f32(mean), f32(rstd), (int)rows, (int)H, (float)eps,
                             on.stream), "gcow_layernorm_fwd");
    g_launches++;
    if (node) {
      const Tensor all[4] = {xb, g32, mean, rstd};
      for (int i = 0; i < 4; i++) node->kept[i].set(all[i]);
      node->shape = x.sizes().vec();
      node->ptype = gamma.scalar_type();
    }
  }
  return finish(std::move(out), node);
  END_HANDLE_TH_ERRORS
}

// ---------------------------------------------------------------------- attention
struct FusedAttentionNode : LayerNode {                     // input: qkv
  float scale = 1;
  std::string name() const override { return "GcowAttentionBackward"; }
  variable_list grads(variable_list&& in, const Saved& had) override {
    variable_list out(1);
    const Tensor &q = had[0], &o = had[1], &lse = had[2];
    const On on(q);
    const int B = (int)q.size(0), S = (int)q.size(1), H = (int)q.size(3), D = (int)q.size(4);
    const Tensor g = bf16_rows16(in[0]);
    Tensor dqkv = at::empty_like(q);
    const Tensor delta = empty({B, H, S}, at::kFloat, q);
    check(gcow_attention_bwd(q.data_ptr(), o.data_ptr(), g.data_ptr(), f32(lse), f32(delta), dqkv.data_ptr(), B, S, H, D, scale, on.error,
                             on.stream), "gcow_attention_bwd");
    g_launches += 2;
    out[0] = std::move(dqkv);
    return out;
  }
};

PyObject* fused_attention(PyObject*, PyObject* const* args, Py_ssize_t nargs) {   // (qkv [B, S, 3, H, 64], scale)
  HANDLE_TH_ERRORS
  TORCH_CHECK(nargs == 2, "fused_attention: bad arguments");
  const Tensor qkv = need(args[0]);
  const double scale = PyFloat_AsDouble(args[1]);
  if (PyErr_Occurred()) return nullptr;
  dims("fused_attention: the input", qkv, 5);
  TORCH_CHECK(qkv.size(2) == 3, "fused_attention: expected [batch, positions, 3, heads, 64], got ", qkv.sizes());
  auto node = record<FusedAttentionNode>(qkv);
  Tensor out;
  {
    Below below;
    const On on(qkv);
    const int64_t B = qkv.size(0), S = qkv.size(1), H = qkv.size(3), D = qkv.size(4);
    const Tensor q = bf16_rows16(qkv);
    out = empty({B, S, H * D}, at::kBFloat16, q);
    const Tensor lse = empty({B, H, S}, at::kFloat, q);
    check(gcow_attention_fwd(q.data_ptr(), out.data_ptr(), f32(lse), (int)B, (int)S, (int)H, (int)D, (float)scale, on.error, on.stream),
          "gcow_attention_fwd");
    g_launches++;
    if (node) {
      node->kept[0].set(q);
      node->kept[2].set(lse);
      node->scale = (float)scale;
    }
  }
  if (node) {
    torch::autograd::set_history(out, node);
    node->kept[1].set(out, true);
  }
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// C[i] = op(A[i]) op(B[i])^T for [batch, rows, cols] operands with contiguous rows
Tensor bmm(const Tensor& a, const Tensor& b, bool a_t, bool b_t, const On& on, bool out_f32 = false) {
  TORCH_CHECK(a.dim() == 3 && b.dim() == 3 && a.size(0) == b.size(0) && a.scalar_type() == at::kBFloat16 && b.scalar_type() == at::kBFloat16 &&
              a.stride(2) == 1 && b.stride(2) == 1, "bmm: expected two bf16 batches of matrices with contiguous rows, as many in each");
  const int64_t batch = a.size(0), M = a_t ? a.size(2) : a.size(1), K = a_t ? a.size(1) : a.size(2), N = b_t ? b.size(2) : b.size(1);
  TORCH_CHECK(K == (b_t ? b.size(1) : b.size(2)), "bmm: reduction lengths differ");
  on_device_of(a, {&b});
  Tensor out = empty({batch, M, N}, out_f32 ? at::kFloat : at::kBFloat16, a);
  check(gcow_gemm_bf16_batched(a.data_ptr(), b.data_ptr(), out.data_ptr(), (int)M, (int)N, (int)K, (int)a.stride(1), (int)b.stride(1),
                               (int)N, (int)batch, a.stride(0), b.stride(0), M * N, nullptr, nullptr, out_f32 ? kOutF32 : 0, on.error, a_t, b_t, 128, on.stream),
        "gcow_gemm_bf16_batched");
  g_launches++;
  return out;
}

struct AttentionNode : LayerNode {                          // inputs: q, k, v
  float scale = 1;
  std::string name() const override { return "GcowUnfusedAttentionBackward"; }
  variable_list grads(variable_list&& in, const Saved& had) override {
    variable_list out(3);
    const Tensor &q = had[0], &k = had[1], &v = had[2], &p = had[3];
    const On on(q);
    const Tensor go = bf16_rows(in[0]);
    out[2] = bmm(p, go, true, true, on);                    // P^T dO
    const Tensor dp = bmm(go, v, false, false, on);         // dO V^T
    const Tensor ds = at::empty_like(p);
    check(gcow_softmax_bwd(dp.data_ptr(), p.data_ptr(), ds.data_ptr(), p.size(0) * p.size(1), (int)p.size(2), scale, on.stream),
          "gcow_softmax_bwd");
    g_launches++;
    out[0] = bmm(ds, k, false, true, on);                   // dS K
    out[1] = bmm(ds, q, true, true, on);                    // dS^T Q
    return out;
  }
};

PyObject* attention(PyObject*, PyObject* const* args, Py_ssize_t nargs) {      // (q, k, v [batch * heads, S, D] bf16, scale)
  HANDLE_TH_ERRORS
  TORCH_CHECK(nargs == 4, "attention: bad arguments");
  const Tensor q = need(args[0]), k = need(args[1]), v = need(args[2]);
  const double scale = PyFloat_AsDouble(args[3]);
  if (PyErr_Occurred()) return nullptr;
  on_device_of(q, {&k, &v});
  for (const Tensor* t : {&q, &k, &v})
    TORCH_CHECK(t->dim() == 3 && t->sizes() == q.sizes() && t->scalar_type() == at::kBFloat16 && t->is_contiguous(),
                "attention: expected three contiguous bf16 tensors [batch * heads, positions, dimensions] of one shape");
  auto node = record<AttentionNode>(q, k, v);
  Tensor out;
  {
    Below below;
    const On on(q);
    const Tensor s = bmm(q, k, false, false, on), p = at::empty_like(s);
    check(gcow_softmax_fwd(s.data_ptr(), p.data_ptr(), s.size(0) * s.size(1), (int)s.size(2), (float)scale, on.stream), "gcow_softmax_fwd");
    g_launches++;
    out = bmm(p, v, false, true, on);
    if (node) {
      const Tensor all[4] = {q, k, v, p};
      for (int i = 0; i < 4; i++) node->kept[i].set(all[i]);
      node->scale = (float)scale;
    }
  }
  return finish(std::move(out), node);
  END_HANDLE_TH_ERRORS
}

// ---------------------------------------------------------------------- convolutions (NHWC bf16)
struct ConvShape { int N, C, H, W, Co, KH, KW, OH, OW, ph, pw; };

// 64 -> 64 channels, 3x3, stride 1, padding 1: the weight-stationary kernel (pixels as the MMA's N).
bool conv_ws(const ConvShape& s) {
  return s.C == 64 && s.Co == 64 && s.KH == 3 && s.KW == 3 && s.ph == 1 && s.pw == 1 && !env_off("GCOW_CONV_WS") &&
         gcow_conv_ws_usable(s.N, s.H, s.W);
}
// Ci -> 128 channels, 3x3, stride 1, padding 1, tiles that fit the shared memory: the halo-tile kernel.
bool conv_halo(const ConvShape& s) {
  return s.Co == 128 && s.KH == 3 && s.KW == 3 && s.ph == 1 && s.pw == 1 && !env_off("GCOW_CONV_HALO") &&
         gcow_conv_halo_usable(s.N, s.H, s.W, s.C);
}
// The stride-1 forward kernel for these extents: weight-stationary or halo-tile where they apply, else the general one.
void conv_forward(const Tensor& x, const Tensor& w, const Tensor& y, const Tensor& bias, const ConvShape& s, const On& on) {
  if (conv_ws(s)) check(gcow_conv_fwd_ws(x.data_ptr(), w.data_ptr(), y.data_ptr(), f32(bias), s.N, s.H, s.W, on.error, on.stream), "gcow_conv_fwd_ws");
  else if (conv_halo(s)) check(gcow_conv_fwd_halo(x.data_ptr(), w.data_ptr(), y.data_ptr(), f32(bias), s.N, s.H, s.W, s.C, on.error, on.stream), "gcow_conv_fwd_halo");
  else check(gcow_conv_fwd(x.data_ptr(), w.data_ptr(), y.data_ptr(), f32(bias), s.N, s.H, s.W, s.C, s.Co, s.KH, s.KW, s.ph, s.pw, on.error, on.stream), "gcow_conv_fwd");
  g_launches++;
}

// The weight gradient [Co, KH * KW * C] from `parts` partial results that launch(float* part) writes.
template <class Launch>
Tensor conv_wgrad(const Target& t, const ConvShape& s, int parts, const Tensor& like, const On& on, Launch launch) {
  const int64_t cols = (int64_t)s.KH * s.KW * s.C;
  Tensor result;
  const Tensor flat = target_matrix(t, s.Co, cols, 16, &result);
  Tensor out = flat;
  if (parts > 1) {
    const Tensor part = empty({parts, s.Co, cols}, at::kFloat, like);
    launch(f32(part));
    out = add_parts(part, parts, {s.Co, cols}, flat, on);
  } else {
    if (!out.defined()) out = empty({s.Co, cols}, at::kFloat, like);
    launch(f32(out));
  }
  g_launches++;
  return flat.defined() ? result : out.view({s.Co, s.KH, s.KW, s.C}).permute({0, 3, 1, 2});
}
Tensor conv_bias_grad(const Tensor& gy, int Co, const On& on) { return colsum(gy.permute({0, 2, 3, 1}).reshape({-1, Co}), on); }

struct ConvNode : LayerNode {                               // inputs: x, w, b
  ConvShape s;
  int kind = 0, halo_min_w = 15;                            // kind: 0 stride 1, 1 1x1 stride 2, 2 3x3 stride 2
  bool has_bias = false;
  std::string name() const override { return "GcowConvBackward"; }
  variable_list grads(variable_list&& in, const Saved& had) override {
    variable_list out(3);
    const Tensor &x = had[0], &wr = had[1];
    const On on(x);
    const Tensor gy = nhwc_bf16(in[0]);
    const void* const g = gy.data_ptr();
    if (wants(0)) {
      Tensor gx = empty_nhwc(s.N, s.C, s.H, s.W, x);
      if (kind == 2) {
        const Tensor wp = empty({9 * (int64_t)s.C * s.Co}, at::kBFloat16, x);
        check(gcow_conv_dgrad_s2(g, wr.data_ptr(), wp.data_ptr(), gx.data_ptr(), s.N, s.H, s.W, s.C, s.Co, on.error, on.stream), "gcow_conv_dgrad_s2");
        g_launches += 5;
      } else {
        const Tensor wt = empty({s.C, s.KH, s.KW, s.Co}, at::kBFloat16, x);
        check(gcow_conv_flip_weights(wr.data_ptr(), wt.data_ptr(), s.Co, s.KH, s.KW, s.C, on.stream), "gcow_conv_flip_weights");
        g_launches++;
        if (kind == 1) {
          check(gcow_conv_dgrad_1x1_s2(g, wt.data_ptr(), gx.data_ptr(), s.N, s.H, s.W, s.C, s.Co, on.error, on.stream), "gcow_conv_dgrad_1x1_s2");
          g_launches++;
        } else {
          const ConvShape back{s.N, s.Co, s.OH, s.OW, s.C, s.KH, s.KW, s.H, s.W, s.KH - 1 - s.ph, s.KW - 1 - s.pw};
          conv_forward(gy, wt, gx, Tensor(), back, on);
        }
      }
      out[0] = std::move(gx);
    }
    if (wants(1)) {
      if (kind) {
        const int parts = gcow_conv_wgrad_split_strided(s.N, s.H, s.W, s.C, s.Co, s.KH, s.KW, s.ph, s.pw, 2);
        out[1] = conv_wgrad(target[0], s, parts, x, on, [&](float* part) {
          check(gcow_conv_wgrad_strided(g, x.data_ptr(), part, s.N, s.H, s.W, s.C, s.Co, s.KH, s.KW, s.ph, s.pw, 2, on.error, on.stream), "gcow_conv_wgrad_strided");
        });
      } else {
        // 64 -> 64 channels, 3x3, padding 1: the halo-tile kernel, when the image rows fit its slot pitch; channel counts
        // that are multiples of 128, 3x3, padding 1, rows of at least halo_min_w pixels: the one with a CTA group per
        // (filter row, 128 x 128 channels); else the general one (the line is explained in ops/kernels.py)
        const int ws = conv_ws(s) && !env_off("GCOW_CONV_WS_WGRAD") ? gcow_conv_wgrad_ws_split(s.N, s.H, s.W) : 0;
        const int halo = s.C % 128 == 0 && s.Co % 128 == 0 && s.KH == 3 && s.KW == 3 && s.ph == 1 && s.pw == 1 && s.W >= halo_min_w &&
                         !env_off("GCOW_CONV_HALO_WGRAD") ? gcow_conv_wgrad_halo_split(s.N, s.H, s.W, s.C, s.Co) : 0;
        const int parts = ws > 0 ? ws : halo > 0 ? halo : gcow_conv_wgrad_split(s.N, s.H, s.W, s.C, s.Co, s.KH, s.KW, s.ph, s.pw);
        out[1] = conv_wgrad(target[0], s, parts, x, on, [&](float* part) {
          if (ws > 0) check(gcow_conv_wgrad_ws(g, x.data_ptr(), part, s.N, s.H, s.W, on.error, on.stream), "gcow_conv_wgrad_ws");
          else if (halo > 0) check(gcow_conv_wgrad_halo(g, x.data_ptr(), part, s.N, s.H, s.W, s.C, s.Co, on.error, on.stream), "gcow_conv_wgrad_halo");
          else check(gcow_conv_wgrad(g, x.data_ptr(), part, s.N, s.H, s.W, s.C, s.Co, s.KH, s.KW, s.ph, s.pw, on.error, on.stream), "gcow_conv_wgrad");
        });
      }
    }
    if (has_bias && wants(2)) out[2] = conv_bias_grad(gy, s.Co, on);
    return out;
  }
};

// conv(x, w, b or None, kind, pad_h, pad_w, halo_min_w): implicit-GEMM convolutions; kind as in ConvNode
PyObject* conv(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  TORCH_CHECK(nargs == 7, "conv: bad arguments");
  const Tensor xin = need(args[0]), w = need(args[1]), b = arg(args[2]);
  int v[4];
  for (int i = 0; i < 4; i++) v[i] = (int)PyLong_AsLong(args[3 + i]);
  if (PyErr_Occurred()) return nullptr;
  on_device_of(xin, {&w, &b});
  dims("conv: the input", xin, 4);
  dims("conv: the weight", w, 4);
  TORCH_CHECK(w.size(1) == xin.size(1), "conv: the weight has ", w.size(1), " input channels, the input ", xin.size(1));
  TORCH_CHECK(v[0] == 0 || (v[0] == 1 ? w.size(2) == 1 && w.size(3) == 1 : w.size(2) == 3 && w.size(3) == 3),
              "conv: the stride-2 kernels take filters of 1 x 1 and of 3 x 3");
  length("conv: the bias", b, w.size(0));
  auto node = record<ConvNode>(xin, w, b);
  Tensor out;
  {
    Below below;
    const On on(xin);
    const Tensor x = nhwc_bf16(xin), wr = bf16_weight(args[1]).permute({0, 2, 3, 1}).contiguous(), bias = float_vector(b);   // [Co, kh, kw, Ci]
    ConvShape s{(int)x.size(0), (int)x.size(1), (int)x.size(2), (int)x.size(3), (int)w.size(0), (int)w.size(2), (int)w.size(3), 0, 0, v[1], v[2]};
    s.OH = v[0] ? (s.H - 1) / 2 + 1 : s.H + 2 * s.ph - s.KH + 1;
    s.OW = v[0] ? (s.W - 1) / 2 + 1 : s.W + 2 * s.pw - s.KW + 1;
    out = empty_nhwc(s.N, s.Co, s.OH, s.OW, x);
    if (v[0]) {
      check(gcow_conv_fwd_strided(x.data_ptr(), wr.data_ptr(), out.data_ptr(), f32(bias), s.N, s.H, s.W, s.C, s.Co, s.KH, s.KW, s.ph, s.pw, 2,
                                  on.error, on.stream), "gcow_conv_fwd_strided");
      g_launches++;
    } else {
      conv_forward(x, wr, out, bias, s, on);
    }
    if (node) {
      node->kept[0].set(x);
      node->kept[1].set(wr);
      node->s = s;
      node->kind = v[0];
      node->halo_min_w = v[3];
      node->has_bias = b.defined();
      node->target[0] = {take_grad_view(args[1]), w};
    }
  }
  return finish(std::move(out), node);
  END_HANDLE_TH_ERRORS
}

struct Conv1x1Node : LayerNode {                            // inputs: x, w, b
  int64_t N = 0, C = 0, H = 0, W = 0, Co = 0;
  at::ScalarType wtype = at::kFloat;
  bool has_bias = false;
  std::string name() const override { return "GcowConv1x1Backward"; }
  variable_list grads(variable_list&& in, const Saved& had) override {
    variable_list out(3);
    const Tensor &xm = had[0], &wb = had[1];
    const On on(xm);
    const Tensor g = bf16_rows(in[0].permute({0, 2, 3, 1})).view({-1, Co});
    if (wants(0)) {
      GemmOpts o;
      o.b_t = true;
      out[0] = gemm(g, wb, o, on).view({N, H, W, C}).permute({0, 3, 1, 2});
    }
    if (wants(1)) {
      Tensor result;
      const Tensor flat = target_matrix(target[0], Co, C, 16, &result);
      if (flat.defined()) { wgrad(g, xm, flat, on); out[1] = result; }
      else out[1] = wgrad(g, xm, Tensor(), on).view({Co, C, 1, 1}).to(wtype).contiguous(at::MemoryFormat::ChannelsLast);
    }
    if (has_bias && wants(2)) out[2] = colsum(g, on);
    return out;
  }
};

PyObject* conv1x1(PyObject*, PyObject* const* args, Py_ssize_t nargs) {        // (x, w, b or None): a GEMM over the pixels
  HANDLE_TH_ERRORS
  TORCH_CHECK(nargs == 3, "conv1x1: bad arguments");
  const Tensor x = need(args[0]), w = need(args[1]), b = arg(args[2]);
  on_device_of(x, {&w, &b});
  dims("conv1x1: the input", x, 4);
  length("conv1x1: the weight", w, w.size(0) * x.size(1));
  length("conv1x1: the bias", b, w.size(0));
  auto node = record<Conv1x1Node>(x, w, b);
  Tensor out;
  {
    Below below;
    const On on(x);
    const int64_t N = x.size(0), C = x.size(1), H = x.size(2), W = x.size(3), Co = w.size(0);
    const Tensor xm = bf16_rows(x.permute({0, 2, 3, 1})).view({-1, C}), wb = bf16_weight(args[1]).reshape({Co, C}).contiguous();
    GemmOpts o;
    o.bias = float_vector(b);
    out = empty_nhwc(N, Co, H, W, x);
    o.out = out.permute({0, 2, 3, 1}).view({-1, Co});
    gemm(xm, wb, o, on);
    if (node) {
      node->kept[0].set(xm);
      node->kept[1].set(wb);
      node->N = N; node->C = C; node->H = H; node->W = W; node->Co = Co;
      node->wtype = w.scalar_type();
      node->has_bias = b.defined();
      node->target[0] = {take_grad_view(args[1]), w};
    }
  }
  return finish(std::move(out), node);
  END_HANDLE_TH_ERRORS
}

// ---------------------------------------------------------------------- BatchNorm (+ add) (+ ReLU)
struct BatchNormNode : LayerNode {                          // inputs: x, gamma, beta, residual; outputs: y and, forked, y again
  int64_t R = 0, C = 0;
  bool relu = false, has_res = false;
  at::ScalarType ptype = at::kFloat;
  std::string name() const override { return "GcowBatchNormBackward"; }
  variable_list grads(variable_list&& in, const Saved& had) override {
    variable_list out(4);
    Tensor gy = in[0], gy2 = in.size() > 1 ? in[1] : Tensor();
    if (!gy.defined()) std::swap(gy, gy2);
    const Tensor &x = had[0], &g32 = had[1], &stats = had[2];
    const Tensor& mask = had[3];
    const On on(x);
    gy = nhwc_bf16(gy);
    if (gy2.defined()) gy2 = nhwc_bf16(gy2);
    Tensor dx = empty_nhwc(x.size(0), C, x.size(2), x.size(3), x);
    // the masked (summed) gradient: the residual input's gradient, and what the second sweep reads
    Tensor dres;
    if (has_res || gy2.defined()) dres = empty_nhwc(x.size(0), C, x.size(2), x.size(3), x);
    const int launches = gcow_bn_launches(R, (int)C, 1, (dres.defined() ? 1 : 0) | (relu ? 2 : 0));
    const Tensor part = launches > 1 ? empty({(int64_t)gcow_bn_parts(R, (int)C) * 2 * C}, at::kFloat, x) : Tensor();
    // dgamma and dbeta go straight into the two parameters' gradient tensors when the trainer pointed at them
    Tensor dgamma, dbeta, flat_g = target_matrix(target[0], 1, C, 4, &dgamma), flat_b;
    if (flat_g.defined()) flat_b = target_matrix(target[1], 1, C, 4, &dbeta);
    float *pg, *pb;
    if (flat_b.defined()) {
      pg = f32(flat_g);
      pb = f32(flat_b);
    } else {
      const Tensor dgb = empty({2 * C}, at::kFloat, x);
      pg = f32(dgb);
      pb = pg + C;
      dgamma = dgb.narrow(0, 0, C);
      dbeta = dgb.narrow(0, C, C);
    }
    check(gcow_bn_bwd3(gy.data_ptr(), raw(gy2), raw(mask), x.data_ptr(), f32(g32), f32(stats), dx.data_ptr(), raw(dres), pg, pb, f32(part),
                       R, (int)C, relu, on.stream), "gcow_bn_bwd3");
    g_launches += launches;
    out[0] = std::move(dx);
    out[1] = flat_b.defined() ? dgamma : dgamma.to(ptype);
    out[2] = flat_b.defined() ? dbeta : dbeta.to(ptype);
    if (has_res) out[3] = std::move(dres);
    return out;
  }
};

// batchnorm_act(x, gamma, beta, run_mean or None, run_var or None, residual or None, relu, momentum, eps, fork)
PyObject* batchnorm_act(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  TORCH_CHECK(nargs == 10, "batchnorm_act: bad arguments");
  const Tensor x = need(args[0]), gamma = need(args[1]), beta = need(args[2]), rm = arg(args[3]), rv = arg(args[4]), res = arg(args[5]);
  const bool relu = PyObject_IsTrue(args[6]) == 1, fork = PyObject_IsTrue(args[9]) == 1;
  const double momentum = PyFloat_AsDouble(args[7]), eps = PyFloat_AsDouble(args[8]);
  if (PyErr_Occurred()) return nullptr;
  on_device_of(x, {&gamma, &beta, &rm, &rv, &res});
  dims("batchnorm_act: the input", x, 4);
  for (const Tensor* t : {&x, &res})
    TORCH_CHECK(!t->defined() || (t->sizes() == x.sizes() && t->scalar_type() == at::kBFloat16 && t->is_contiguous(at::MemoryFormat::ChannelsLast)),
                "batchnorm_act: expected input and residual as channels-last bf16 tensors of one shape");
  length("batchnorm_act: gamma", gamma, x.size(1));
  length("batchnorm_act: beta", beta, x.size(1));
  for (const Tensor* t : {&rm, &rv}) {
    length("batchnorm_act: the running statistics", *t, x.size(1));
    TORCH_CHECK(!t->defined() || (t->scalar_type() == at::kFloat && t->is_contiguous()),
                "batchnorm_act: the running statistics have to be contiguous float32");
  }
  auto node = record<BatchNormNode>(x, gamma, beta, res);
  Tensor y, y2;
  {
    Below below;
    const On on(x);
    const int64_t C = x.size(1), R = x.size(0) * x.size(2) * x.size(3);
    y = empty_nhwc(x.size(0), C, x.size(2), x.size(3), x);
    const int launches = gcow_bn_launches(R, (int)C, 0, (res.defined() ? 1 : 0) | (relu ? 2 : 0));
    const Tensor stats = empty({4 * C}, at::kFloat, x),
                 part = launches > 1 ? empty({(int64_t)gcow_bn_parts(R, (int)C) * 2 * C}, at::kFloat, x) : Tensor();
    const Tensor g32 = float_vector(gamma), b32 = float_vector(beta);
    const Tensor mask = relu ? empty({R * C / 8}, at::kByte, x) : Tensor();
    check(gcow_bn_fwd_train(x.data_ptr(), raw(res), y.data_ptr(), raw(mask), f32(g32), f32(b32), f32(rm), f32(rv), f32(stats), f32(part), R,
                            (int)C, (float)eps, (float)momentum, relu, on.stream), "gcow_bn_fwd_train");
    g_launches += launches;
    if (node) {                                             // the ReLU bit mask stands in for y in the backward
      node->kept[0].set(x);
      node->kept[1].set(g32);
      node->kept[2].set(stats);
      node->kept[3].set(mask);
      node->R = R; node->C = C;
      node->relu = relu;
      node->has_res = res.defined();
      node->ptype = gamma.scalar_type();
      if (gamma.scalar_type() == at::kFloat) {
        node->target[0] = {take_grad_view(args[1]), gamma};
        node->target[1] = {take_grad_view(args[2]), beta};
      }
    }
    if (fork) {                                             // a second tensor on the same storage (not an autograd view of the first)
      y2 = empty({0}, at::kBFloat16, x);
      y2.set_(y.storage(), y.storage_offset(), y.sizes(), y.strides());
      torch::autograd::impl::set_version_counter(y2, torch::autograd::impl::version_counter(y));   // a change of either is one of both
    }
  }
  if (node) torch::autograd::set_history(y, node);
  if (!fork) return THPVariable_Wrap(std::move(y));
  if (node) torch::autograd::set_history(y2, node);
  PyObject *a = THPVariable_Wrap(std::move(y)), *c = THPVariable_Wrap(std::move(y2));
  PyObject* r = PyTuple_Pack(2, a, c);
  Py_DECREF(a);
  Py_DECREF(c);
  return r;
  END_HANDLE_TH_ERRORS
}

// ---------------------------------------------------------------------- the products and rules by themselves
// gemm(a, b, bias, residual, gelu, out, out_f32, accumulate, max_ctas, a_t, b_t, tile_rows, pre_gelu_out, gelu_grad_of, pair)
PyObject* py_gemm(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  TORCH_CHECK(nargs == 15, "gemm: bad arguments");
  const Tensor a = need(args[0]), b = need(args[1]);
  GemmOpts o;
  o.bias = arg(args[2]);
  o.residual = arg(args[3]);
  o.gelu = PyObject_IsTrue(args[4]) == 1;
  o.out = arg(args[5]);
  o.out_f32 = PyObject_IsTrue(args[6]) == 1;
  o.accumulate = PyObject_IsTrue(args[7]) == 1;
  o.max_ctas = (int)PyLong_AsLong(args[8]);
  o.a_t = PyObject_IsTrue(args[9]) == 1;
  o.b_t = PyObject_IsTrue(args[10]) == 1;
  o.tile_rows = (int)PyLong_AsLong(args[11]);
  o.pre_gelu_out = arg(args[12]);
  o.gelu_grad_of = arg(args[13]);
  if (args[14] != Py_None) o.pair = PyObject_IsTrue(args[14]) == 1;
  if (PyErr_Occurred()) return nullptr;
  const On on(a);
  return THPVariable_Wrap(gemm(a, b, o, on));
  END_HANDLE_TH_ERRORS
}
PyObject* py_wgrad(PyObject*, PyObject* const* args, Py_ssize_t nargs) {       // (g, x, out or None)
  HANDLE_TH_ERRORS
  TORCH_CHECK(nargs == 3, "wgrad: bad arguments");
  const Tensor g = need(args[0]), x = need(args[1]), out = arg(args[2]);
  const On on(g);
  return THPVariable_Wrap(wgrad(g, x, out, on));
  END_HANDLE_TH_ERRORS
}
PyObject* py_bmm(PyObject*, PyObject* const* args, Py_ssize_t nargs) {         // (a, b, a_t, b_t, out_f32)
  HANDLE_TH_ERRORS
  TORCH_CHECK(nargs == 5, "bmm: bad arguments");
  const Tensor a = need(args[0]), b = need(args[1]);
  const On on(a);
  return THPVariable_Wrap(bmm(a, b, PyObject_IsTrue(args[2]) == 1, PyObject_IsTrue(args[3]) == 1, on, PyObject_IsTrue(args[4]) == 1));
  END_HANDLE_TH_ERRORS
}
PyObject* py_colsum(PyObject*, PyObject* g) {
  HANDLE_TH_ERRORS
  const Tensor t = need(g);
  at::NoGradGuard no_grad;
  const On on(t);
  return THPVariable_Wrap(colsum(t, on));
  END_HANDLE_TH_ERRORS
}
PyObject* py_take_grad_view(PyObject*, PyObject* w) {                          // the view, or None
  HANDLE_TH_ERRORS
  need(w);
  Tensor v = take_grad_view(w);
  if (!v.defined()) Py_RETURN_NONE;
  return THPVariable_Wrap(std::move(v));
  END_HANDLE_TH_ERRORS
}
PyObject* py_grad_target(PyObject*, PyObject* const* args, Py_ssize_t nargs) { // (view, weight, rows, cols, align) -> (matrix, gradient)
  HANDLE_TH_ERRORS
  TORCH_CHECK(nargs == 5, "grad_target: bad arguments");
  const Target t{need(args[0]), need(args[1])};
  const int64_t rows = PyLong_AsLongLong(args[2]), cols = PyLong_AsLongLong(args[3]), align = PyLong_AsLongLong(args[4]);
  if (PyErr_Occurred()) return nullptr;
  TORCH_CHECK(align > 0, "grad_target: bad alignment");
  Tensor result;
  Tensor flat = target_matrix(t, rows, cols, (uintptr_t)align, &result);
  if (!flat.defined()) return PyTuple_Pack(2, Py_None, Py_None);
  PyObject *a = THPVariable_Wrap(std::move(flat)), *b = THPVariable_Wrap(std::move(result));
  PyObject* r = a && b ? PyTuple_Pack(2, a, b) : nullptr;
  Py_XDECREF(a);
  Py_XDECREF(b);
  return r;
  END_HANDLE_TH_ERRORS
}
// conv_rules(N, H, W, C, Co, KH, KW, pad_h, pad_w) -> (weight-stationary, halo-tile): which of the two stride-1 kernels apply
PyObject* conv_rules(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  TORCH_CHECK(nargs == 9, "conv_rules: bad arguments");
  int v[9];
  for (int i = 0; i < 9; i++) v[i] = (int)PyLong_AsLong(args[i]);
  if (PyErr_Occurred()) return nullptr;
  const ConvShape s{v[0], v[3], v[1], v[2], v[4], v[5], v[6], 0, 0, v[7], v[8]};
  return PyTuple_Pack(2, conv_ws(s) ? Py_True : Py_False, conv_halo(s) ? Py_True : Py_False);
  END_HANDLE_TH_ERRORS
}

// ---------------------------------------------------------------------- bookkeeping
PyObject* launches(PyObject*, PyObject*) { return PyLong_FromLongLong(g_launches.load()); }
PyObject* view_hits(PyObject*, PyObject*) { return PyLong_FromLongLong(g_view_hits.load()); }
PyObject* py_error_word(PyObject*, PyObject* index) {       // the kernels' error word of a device
  HANDLE_TH_ERRORS
  const long i = PyLong_AsLong(index);
  if (PyErr_Occurred()) return nullptr;
  return THPVariable_Wrap(error_word((int)i));
  END_HANDLE_TH_ERRORS
}
PyObject* error_words(PyObject*, PyObject*) {               // those that exist
  HANDLE_TH_ERRORS
  PyObject* list = PyList_New(0);
  std::lock_guard<std::mutex> lock(g_error_mu);
  for (const Tensor& t : g_error) {
    if (!t.defined()) continue;
    PyObject* o = THPVariable_Wrap(t);
    PyList_Append(list, o);
    Py_DECREF(o);
  }
  return list;
  END_HANDLE_TH_ERRORS
}

}  // namespace

Tensor error_word(int device) {
  TORCH_CHECK(device >= 0 && device < 64, "device index out of range");
  std::lock_guard<std::mutex> lock(g_error_mu);
  Tensor& t = g_error[device];
  if (!t.defined()) {
    // below every dispatch mode: the word outlives a mode that would make it a tensor of its own kind
    at::AutoDispatchBelowADInplaceOrView below;
    const c10::impl::ExcludeDispatchKeyGuard no_modes(c10::DispatchKeySet({c10::DispatchKey::Python, c10::DispatchKey::PythonTLSSnapshot}));
    t = at::zeros({1}, at::TensorOptions().dtype(at::kInt).device(at::Device(at::kCUDA, (at::DeviceIndex)device)));
  }
  return t;
}

#define GCOW_FAST(name) {#name, (PyCFunction)(void (*)())name, METH_FASTCALL, nullptr}
PyMethodDef layer_methods[] = {
    GCOW_FAST(linear), GCOW_FAST(ffn_residual), GCOW_FAST(layernorm), GCOW_FAST(fused_attention), GCOW_FAST(attention),
    GCOW_FAST(conv), GCOW_FAST(conv1x1), GCOW_FAST(batchnorm_act), GCOW_FAST(conv_rules),
    {"gemm", (PyCFunction)(void (*)())py_gemm, METH_FASTCALL, nullptr},
    {"wgrad", (PyCFunction)(void (*)())py_wgrad, METH_FASTCALL, nullptr},
    {"bmm", (PyCFunction)(void (*)())py_bmm, METH_FASTCALL, nullptr},
    {"colsum", py_colsum, METH_O, nullptr},
    {"take_grad_view", py_take_grad_view, METH_O, nullptr},
    {"grad_target", (PyCFunction)(void (*)())py_grad_target, METH_FASTCALL, nullptr},
    {"launches", launches, METH_NOARGS, nullptr},
    {"view_hits", view_hits, METH_NOARGS, nullptr},
    {"error_word", py_error_word, METH_O, nullptr},
    {"error_words", error_words, METH_NOARGS, nullptr},
    {nullptr, nullptr, 0, nullptr},
};

}  // namespace gcow_ext
