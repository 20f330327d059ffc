// Inference over a packed batch: the rows of all sequences lie one behind the other, nothing is
// padded, and only the last position of every sequence leaves the network (move prediction and the
// prompts of a search need no other).
//
//   gather_rows : the last rows of the residual stream and of the attention output, after the last
//                 layer's attention; everything behind it runs on one row per sequence
//   ab_infer_last : the schedule of one such pass.  It is native because a pass of the medium model is
//                 170 launches: about 15 us each from Python against 3 us from here, and a single short
//                 game needs less than that on the GPU.
// Padding cost: with games of 4 to 300 tokens half of the rows of a padded batch are padding.
#include "gemm_tc.cuh"
#include "ptx.cuh"

namespace ab {

__global__ void __launch_bounds__(128)
gather_rows_kernel(const float* __restrict__ x, const __nv_bfloat16* __restrict__ y, const int* __restrict__ last,
                   float* __restrict__ x_out, __nv_bfloat16* __restrict__ y_out, int d) {
  griddep_enter();
  const long long src = last[blockIdx.x], dst = blockIdx.x;
  for (int i = threadIdx.x; i < d / 8; i += 128) {
    reinterpret_cast<uint4*>(y_out + dst * d)[i] = reinterpret_cast<const uint4*>(y + src * d)[i];
    reinterpret_cast<float4*>(x_out + dst * d)[2 * i] = reinterpret_cast<const float4*>(x + src * d)[2 * i];
    reinterpret_cast<float4*>(x_out + dst * d)[2 * i + 1] = reinterpret_cast<const float4*>(x + src * d)[2 * i + 1];
  }
}

}  // namespace ab

extern "C" {

struct AbInferLayer {
  const float *ln1_w, *ln1_b, *ln2_w, *ln2_b;
  const void* qkv_w; const float* qkv_b;
  const void* o_w;   const float* o_b;
  const void* fc_w;  const float* fc_b;
  const void* pr_w;  const float* pr_b;
};

struct AbInfer {
  // model
  int n_layer, d, H, hd, F, V, rms;
  float eps;
  const float *wte, *wpe, *ctrl, *lnf_w, *lnf_b;
  const void* wte_bf16;
  const float *wv, *bv, *wt, *bt;            // scalar heads, null without them
  // batch: n sequences, M rows in all, T rows the longest
  int n, M, T;
  const int *ids, *pos, *row0, *last;        // [M], [M], [n + 1], [n]
  // scratch ([M, .]; the *_last ones [n, .])
  float* x; void *ln, *qkv, *att, *act;
  float* x_last; void* att_last;
  // results, one row per sequence
  void *h, *logits;
  float *value, *time;
  // key/value cache of the search ([layer][tree][head][slot][hd]), or null
  void *kc, *vc;
  long long kv_layer;                        // elements between layers
  int S;
  int max_ctas;
  int* status;
};

int ab_layernorm_fwd(const float*, const float*, const float*, void*, float*, float*, int, int, float, int, cudaStream_t);
int ab_layernorm_fwd_ahead(const float*, const float*, const float*, void*, float*, float*, int, int, float, int,
                           cudaStream_t);
int ab_embed_fwd(const int*, const int*, const float*, const float*, const float*, float*, int, int, int,
                 unsigned long long, unsigned int, unsigned int, cudaStream_t);
int ab_heads_fwd(const void*, const float*, const float*, const float*, const float*, const float*, const float*,
                 const int*, float, float, float*, float*, float*, float*, float*, int, int, cudaStream_t);
int ab_heads_fwd_ahead(const void*, const float*, const float*, const float*, const float*, float*, float*, int, int,
                       cudaStream_t);
int ab_attn_fwd_packed_kv(const void* qkv, void* out, const int* row0, int B, int T, int rows, int H, int hd, float scale,
                          void* kc, void* vc, int slots, int dependent, int* status, cudaStream_t stream);

// Returns the number of kernels launched, or a negative number / minus a cudaError_t.
int ab_infer_last(const AbInfer* p, const AbInferLayer* layers, cudaStream_t stream) {
  using namespace ab;
  const AbInfer& a = *p;
  if (a.n < 1 || a.M < a.n || a.T < 1 || a.n > 65535 || a.d % 128 || a.d > 2048 || a.H * a.hd != a.d) return -1;
  if (a.kc && (a.T > a.S)) return -1;
  int launched = 0, rc = 0;
  // Few rows: launch latencies are what the pass waits for, so every kernel is a programmatic
  // dependent of the one before it (its set-up and first weight tiles overlap that kernel).
  const int dep = a.M <= 256;
  auto norm = [&](const float* x, const float* w, const float* b, void* y, int M) {
    ++launched;
    return (dep ? ab_layernorm_fwd_ahead : ab_layernorm_fwd)(x, w, b, y, nullptr, nullptr, M, a.d, a.eps, a.rms, stream);
  };
  // No contraction is split: each output is one chain of products whatever the batch, so a game's
  // evaluation does not depend on the games beside it.
  auto gemm = [&](const void* A, int K, const void* B, int b_mn, const float* bias, int act, void* out, int fp32,
                  int M, int N, const void* next = nullptr, long long next_size = 0) {
    AbGemmEpilogue ep = {};
    if (dep && next) { ep.next_b = next; ep.next_bytes = next_size * 2 / 16 * 16; }
    ep.out = out; ep.ldo = N; ep.out_fp32 = fp32; ep.bias = bias; ep.act = act; ep.alpha = 1.f; ep.pdl = dep;
    if (fp32) { ep.resid = static_cast<const float*>(out); ep.ldr = N; }    // residual update in place
    ++launched;
    return ab_gemm_bf16(A, 0, K, B, b_mn, b_mn ? N : K, M, N, K, &ep, 1, a.max_ctas, a.status, stream);
  };
#define AB_TRY(call) if ((rc = (call)) != 0) return rc < 0 ? rc : -rc
  AB_TRY(ab_embed_fwd(a.ids, a.pos, a.wte, a.wpe, a.ctrl, a.x, a.M, a.d, a.V, 0, 0, 0, stream));
  ++launched;
  float* x = a.x;
  const void* att = a.att;
  int M = a.M;
  for (int l = 0; l < a.n_layer; ++l) {
    const AbInferLayer& L = layers[l];
    AB_TRY(norm(x, L.ln1_w, L.ln1_b, a.ln, M));
    const long long dd = static_cast<long long>(a.d) * a.d, df = static_cast<long long>(a.d) * a.F;
    AB_TRY(gemm(a.ln, a.d, L.qkv_w, 1, L.qkv_b, 0, a.qkv, 0, M, 3 * a.d, L.o_w, dd));
    // the keys and values of a search's prompts go on to its cache from the attention's shared memory (a kernel of
    // its own took 59 us per layer for 39000 rows of 1024)
    __nv_bfloat16* kc = a.kc ? static_cast<__nv_bfloat16*>(a.kc) + l * a.kv_layer : nullptr;
    __nv_bfloat16* vc = a.kc ? static_cast<__nv_bfloat16*>(a.vc) + l * a.kv_layer : nullptr;
    AB_TRY(ab_attn_fwd_packed_kv(a.qkv, a.att, a.row0, a.n, a.T, M, a.H, a.hd, 1.f / sqrtf((float)a.hd), kc, vc, a.S, dep,
                                 a.status, stream));
    ++launched;
    if (l == a.n_layer - 1) {
      launch_chained(gather_rows_kernel, dim3(a.n), dim3(128), 0, stream, (const float*)x,
                     (const __nv_bfloat16*)a.att, a.last, a.x_last, (__nv_bfloat16*)a.att_last, a.d);
      AB_TRY((int)cudaGetLastError());
      ++launched;
      x = a.x_last;
      att = a.att_last;
      M = a.n;
    }
    AB_TRY(gemm(att, a.d, L.o_w, 1, L.o_b, 0, x, 1, M, a.d, L.fc_w, df));
    AB_TRY(norm(x, L.ln2_w, L.ln2_b, a.ln, M));
    AB_TRY(gemm(a.ln, a.d, L.fc_w, 1, L.fc_b, 3, a.act, 0, M, a.F, L.pr_w, df));
    const bool more = l + 1 < a.n_layer;
    AB_TRY(gemm(a.act, a.F, L.pr_w, 1, L.pr_b, 0, x, 1, M, a.d, more ? layers[l + 1].qkv_w : a.wte_bf16,
                more ? 3 * dd : static_cast<long long>(a.V) * a.d));
  }
  AB_TRY(norm(x, a.lnf_w, a.lnf_b, a.h, M));
  AB_TRY(gemm(a.h, a.d, a.wte_bf16, 0, nullptr, 0, a.logits, 0, M, a.V));
  if (a.wv) {
    AB_TRY(dep ? ab_heads_fwd_ahead(a.h, a.wv, a.bv, a.wt, a.bt, a.value, a.time, M, a.d, stream)
               : ab_heads_fwd(a.h, a.wv, a.bv, a.wt, a.bt, nullptr, nullptr, nullptr, 0.f, 0.f, a.value, a.time, nullptr,
                              nullptr, nullptr, M, a.d, stream));
    ++launched;
  }
#undef AB_TRY
  return launched;
}
}
