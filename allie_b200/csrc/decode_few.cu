// All layers of a search step for at most 16 trees as ONE cooperative kernel.
//
// One new token per tree: a step reads every weight once (604 MB for the medium model: 92 us at memory
// speed) and computes next to nothing.  As a chain of kernels (seven per layer; even as programmatic
// dependents a link costs 5 to 9 us: launch, descriptors, first loads, accumulator hand-over, last
// stores) the step took 1.2 ms.  Here one CTA per SM stays for the whole step:
//   * a producer warp streams the CTA's share of ALL layers' weights through a shared-memory ring of
//     112 KB with asynchronous copies.  It knows nothing of the phases, so weights keep arriving while
//     the other warps wait for a phase to end;
//   * eight warps compute the five phases of a layer: LayerNorm + QKV, attention, output projection,
//     LayerNorm + FC, GELU + projection.  Between phases all CTAs meet at a counter in memory (bounded
//     wait; the launch is cooperative, so all CTAs are resident);
//   * a work unit is 64 output columns (whole 128-byte lines of W; with 16 columns the copies of 32-byte
//     pieces took ten times as long) and a slice of the contraction.  A warp owns a share of the contraction and
//     multiplies with m16n8k16 MMAs (a 128-row tensor-core tile would be 7/8 padding); the warps' products
//     meet in shared memory and the slices are added in memory with fp32 reductions, into the residual
//     stream or into accumulators that the next phase rounds as the chain of kernels does;
//   * every CTA normalises the residual rows for itself (n x d values through L2);
//   * attention: a CTA takes a (tree, head), its warps split the keys;
//   * what does not belong to a phase (clearing accumulators, prefetches, the next norm's vectors) is done by
//     seven warps while the eighth watches a meeting.
// Measured (24 layers of 1024 / 4096, cold weights): 455 us with one tree, 476 with 4, 523 with 8, 708 with 16
// (626, 636, - and 837 with the norm's vectors and the requests read through L2 by every phase, a warp per row
// and eight columns per warp); 367 us at width 128, where only the meetings and the first loads behind each are
// left.  A meeting takes 2600 clocks: 1000 until a CTA's additions are known to be done, 1600 until all have seen
// the last arrival.  That is 13000 of a layer's 35000 and bounds it now.  Attention and output projection as one
// phase (each head's attention by every CTA of its projection rows) saves a meeting and loses it again to the
// size of the code.  From 17 trees on the chain of kernels is used: its tiles hold 128 rows.
#include "ptx.cuh"

namespace ab {

constexpr int DF_MAX_N = 16;
constexpr int DF_COLS = 64;                        // columns of a unit
constexpr int DF_CHUNK = 64;                       // rows of W per ring slot
constexpr int DF_SLOT = DF_CHUNK * DF_COLS * 2;    // 8 KB
constexpr int DF_STAGES = 14;
constexpr int DF_MAX_K = 1280;                     // widest operand in shared memory
constexpr int DF_MAX_LAYERS = 64;
constexpr int DF_WARPS = 8;
constexpr int DF_THREADS = (DF_WARPS + 1) * 32;
constexpr int DF_WORK_HEAD = 256;                  // words in front of the accumulators; the first counts arrivals

struct DecodeLayer {
  const float *ln1_w, *ln1_b, *ln2_w, *ln2_b, *qkv_b, *o_b, *fc_b, *pr_b;
  const __nv_bfloat16 *qkv_w, *o_w, *fc_w, *pr_w;  // [K][N]
  __nv_bfloat16 *kc, *vc;                          // [tree][head][slot][hd]
};

// What the search asks for, copied to shared memory once per step: every layer reads it, through L2 each time
// otherwise (the meetings void L1), one dependent trip after the other.
constexpr int DF_ANC = 128;                        // entries of a tree's ancestor list kept there
struct DfTrees {
  int active[DF_MAX_N], slot[DF_MAX_N], prefix[DF_MAX_N], n_anc[DF_MAX_N];
  int anc[DF_MAX_N][DF_ANC];
};

struct DecodeFewArgs {
  const DecodeLayer* layers;
  int n_layer, n, d, H, F, S, rms;
  float eps, scale;
  float* x;                                        // [n, d] residual stream, updated in place
  __nv_bfloat16* att;                              // [n, d]
  float *qkv, *fc;                                 // [n, 3d], [n, F] accumulators, zero at launch
  const int *active, *slot, *prefix_len, *anc, *n_anc;
  int anc_stride;
  int slices[4];                                   // of the contraction, per matrix
  int pitch;                                       // bytes per row of the operand buffer
  unsigned int* arrivals;                          // zero at launch
  long long max_wait;                              // clock cycles at a meeting
  int* status;
};

constexpr int DF_PART = DF_COLS + 8;               // floats per row of partial products: rows on different banks

// matrix m: 0 QKV, 1 output projection, 2 FC, 3 projection
struct DfMat {
  int N, K, k, blocks, units;
  const __nv_bfloat16* w;
};
__device__ __forceinline__ DfMat df_mat(const DecodeFewArgs& g, const DecodeLayer& L, int m) {
  DfMat p;
  p.N = m == 0 ? 3 * g.d : m == 2 ? g.F : g.d;
  p.K = m == 3 ? g.F : g.d;
  p.w = m == 0 ? L.qkv_w : m == 1 ? L.o_w : m == 2 ? L.fc_w : L.pr_w;
  p.k = p.K / g.slices[m];
  p.blocks = p.N / DF_COLS;
  p.units = p.blocks * g.slices[m];
  return p;
}

__device__ __forceinline__ void df_ldsm4(uint32_t* r, uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void df_ldsm4_t(uint32_t* r, uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void df_mma(float* c, const uint32_t* a, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
               "{%0, %1, %2, %3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void df_sync() {        // the eight computing warps
  asm volatile("bar.sync 1, %0;" ::"n"(DF_WARPS * 32) : "memory");
}
__device__ __forceinline__ void df_red2(float* p, float a, float b) {
  asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(p), "f"(a), "f"(b) : "memory");
}
// eight accumulators (+ bias, + GELU) rounded to bf16; they come from other SMs, so through L2
template <bool GELU>
__device__ __forceinline__ uint4 df_round8(const float* acc, const float* bias) {
  float4 a = __ldcg(reinterpret_cast<const float4*>(acc)), b = __ldcg(reinterpret_cast<const float4*>(acc) + 1);
  if (bias) {
    const float4 p = __ldg(reinterpret_cast<const float4*>(bias)), q = __ldg(reinterpret_cast<const float4*>(bias) + 1);
    a.x += p.x; a.y += p.y; a.z += p.z; a.w += p.w;
    b.x += q.x; b.y += q.y; b.z += q.z; b.w += q.w;
  }
  if (GELU) {
    a.x = gelu_tanh(a.x); a.y = gelu_tanh(a.y); a.z = gelu_tanh(a.z); a.w = gelu_tanh(a.w);
    b.x = gelu_tanh(b.x); b.y = gelu_tanh(b.y); b.z = gelu_tanh(b.z); b.w = gelu_tanh(b.w);
  }
  return make_uint4(pack_bf16x2(a.x, a.y), pack_bf16x2(a.z, a.w), pack_bf16x2(b.x, b.y), pack_bf16x2(b.z, b.w));
}

// LayerNorm / RMSNorm of the residual rows -> operand buffer (bf16).  The eight warps share the rows: eight, four
// or two warps to a row for one, two and up to four trees (their sums meet in `sR`), else one, which takes a
// second row from nine trees on.  `sN` holds the weights and, behind DF_MAX_K of them, the offsets.  (Read from
// global in the last loop, they cost a trip to L2 per 128 columns: 8000 of a phase's 14000 clocks at d = 1024.)
template <int W>
__device__ __forceinline__ void df_norm(const DecodeFewArgs& g, const float* sN, uint8_t* sA, float* sR, int warp,
                                        int lane) {
  constexpr int NV = DF_MAX_K / 128 / W + (DF_MAX_K / 128 % W != 0);      // float4s of a lane
  const int part = warp % W, c_first = part * 32 + lane, n4 = g.d >> 2;   // n4 is a multiple of 32
  auto all_sum = [&](float s, int k) {             // over the row; `k`: which of its two sums
#pragma unroll
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (W == 1) return s;
    if (lane == 0) sR[k * DF_WARPS + warp] = s;
    df_sync();
    s = 0.f;
#pragma unroll
    for (int i = 0; i < W; ++i) s += sR[k * DF_WARPS + warp - part + i];
    return s;
  };
#pragma unroll 1
  for (int row = warp / W; W > 1 ? row < DF_WARPS / W : row < g.n; row += DF_WARPS) {
    const bool live = row < g.n;                   // every warp takes part in the meetings
    const float4* xr = reinterpret_cast<const float4*>(g.x + static_cast<long long>(row) * g.d);
    float4 v[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (live && c_first + 32 * W * i < n4) v[i] = __ldcg(xr + c_first + 32 * W * i);
    }
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) s += v[i].x + v[i].y + v[i].z + v[i].w;
    s = all_sum(s, 0);
    const float mean = g.rms ? 0.f : s / g.d;
    float q = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i)
      if (c_first + 32 * W * i < n4) {
        const float a = v[i].x - mean, c = v[i].y - mean, e = v[i].z - mean, f = v[i].w - mean;
        q += a * a + c * c + e * e + f * f;
      }
    q = all_sum(q, 1);
    const float rstd = rsqrtf(q / g.d + g.eps);
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int c4 = c_first + 32 * W * i;
      if (live && c4 < n4) {
        const float4 ww = reinterpret_cast<const float4*>(sN)[c4], bb = reinterpret_cast<const float4*>(sN + DF_MAX_K)[c4];
        *reinterpret_cast<uint2*>(sA + row * g.pitch + c4 * 8) =
            make_uint2(pack_bf16x2((v[i].x - mean) * rstd * ww.x + bb.x, (v[i].y - mean) * rstd * ww.y + bb.y),
                       pack_bf16x2((v[i].z - mean) * rstd * ww.z + bb.z, (v[i].w - mean) * rstd * ww.w + bb.w));
      }
    }
  }
}

// Attention of one (tree, head): the eight warps split the keys (eight keys per warp and round, four
// lanes per key, ROUNDS rounds of loads in flight) and merge through shared memory.
template <int HD>
__device__ __forceinline__ void df_attention(const DecodeFewArgs& g, const DecodeLayer& L, const DfTrees& tr, int t,
                                             int h, float* sM, int warp, int lane) {
  constexpr int DPL = HD / 4, U = DPL / 8, ROUNDS = HD == 64 ? 2 : 1;
  const int c4 = lane & 3, kg = lane >> 2;
  const float* row = g.qkv + static_cast<long long>(t) * 3 * g.d + h * HD;       // this token's q; k, v d and 2d on
  const float* bias = L.qkv_b ? L.qkv_b + h * HD : nullptr;
  auto own = [&](int part, int c) {                // eight values of q (0), k (1) or v (2) from column c
    return df_round8<false>(row + part * g.d + c, bias ? bias + part * g.d + c : nullptr);
  };
  const long long base = (static_cast<long long>(t) * g.H + h) * g.S * HD;
  const int P = tr.prefix[t], n = P + tr.n_anc[t];
  auto anc = [&](int k) { return k < DF_ANC ? tr.anc[t][k] : g.anc[static_cast<long long>(t) * g.anc_stride + k]; };
  // every load of the first round is on its way before any is waited for
  uint4 qw[U], kv[ROUNDS][U], vv[ROUNDS][U];
  auto fetch = [&](int j0) {
#pragma unroll
    for (int r = 0; r < ROUNDS; ++r) {
      const int j = j0 + r * 64 + kg;
#pragma unroll
      for (int u = 0; u < U; ++u) {
        kv[r][u] = make_uint4(0u, 0u, 0u, 0u);
        vv[r][u] = kv[r][u];
      }
      if (j < n && (j < P || j < n - 1)) {
        const long long off = base + static_cast<long long>(j < P ? j : anc(j - P)) * HD + c4 * DPL;
#pragma unroll
        for (int u = 0; u < U; ++u) {
          kv[r][u] = __ldcg(reinterpret_cast<const uint4*>(L.kc + off + u * 8));
          vv[r][u] = __ldcg(reinterpret_cast<const uint4*>(L.vc + off + u * 8));
        }
      } else if (j == n - 1) {                     // the last entry of the list is the token itself
#pragma unroll
        for (int u = 0; u < U; ++u) {
          kv[r][u] = own(1, c4 * DPL + u * 8);
          vv[r][u] = own(2, c4 * DPL + u * 8);
        }
      }
    }
  };
  if (warp * 8 < n) fetch(warp * 8);
#pragma unroll
  for (int u = 0; u < U; ++u) qw[u] = own(0, c4 * DPL + u * 8);
  if (warp == 0 && lane < HD / 8) {                // this token's key / value go into the cache
    const long long dst = base + static_cast<long long>(tr.slot[t]) * HD + lane * 8;
    *reinterpret_cast<uint4*>(L.kc + dst) = own(1, lane * 8);
    *reinterpret_cast<uint4*>(L.vc + dst) = own(2, lane * 8);
  }
  float q[DPL], acc[DPL];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const uint4 w = qw[u];
    q[u * 8 + 0] = bf16_lo(w.x) * g.scale; q[u * 8 + 1] = bf16_hi(w.x) * g.scale;
    q[u * 8 + 2] = bf16_lo(w.y) * g.scale; q[u * 8 + 3] = bf16_hi(w.y) * g.scale;
    q[u * 8 + 4] = bf16_lo(w.z) * g.scale; q[u * 8 + 5] = bf16_hi(w.z) * g.scale;
    q[u * 8 + 6] = bf16_lo(w.w) * g.scale; q[u * 8 + 7] = bf16_hi(w.w) * g.scale;
  }
#pragma unroll
  for (int e = 0; e < DPL; ++e) acc[e] = 0.f;
  float m = -INFINITY, l = 0.f;
  for (int j0 = warp * 8; j0 < n; j0 += 64 * ROUNDS) {
    if (j0 != warp * 8) fetch(j0);
#pragma unroll
    for (int r = 0; r < ROUNDS; ++r) {
      if (j0 + r * 64 >= n) break;                 // warp-uniform
      const bool live = j0 + r * 64 + kg < n;
      float dot = 0.f;
#pragma unroll
      for (int u = 0; u < U; ++u)
        dot += q[u * 8 + 0] * bf16_lo(kv[r][u].x) + q[u * 8 + 1] * bf16_hi(kv[r][u].x) +
               q[u * 8 + 2] * bf16_lo(kv[r][u].y) + q[u * 8 + 3] * bf16_hi(kv[r][u].y) +
               q[u * 8 + 4] * bf16_lo(kv[r][u].z) + q[u * 8 + 5] * bf16_hi(kv[r][u].z) +
               q[u * 8 + 6] * bf16_lo(kv[r][u].w) + q[u * 8 + 7] * bf16_hi(kv[r][u].w);
      dot += __shfl_xor_sync(0xffffffffu, dot, 1);
      dot += __shfl_xor_sync(0xffffffffu, dot, 2);
      if (live) {
        const float m_new = fmaxf(m, dot);
        const float a = __expf(m - m_new), p = __expf(dot - m_new);
        l = l * a + p;
        m = m_new;
#pragma unroll
        for (int u = 0; u < U; ++u) {
          acc[u * 8 + 0] = acc[u * 8 + 0] * a + p * bf16_lo(vv[r][u].x); acc[u * 8 + 1] = acc[u * 8 + 1] * a + p * bf16_hi(vv[r][u].x);
          acc[u * 8 + 2] = acc[u * 8 + 2] * a + p * bf16_lo(vv[r][u].y); acc[u * 8 + 3] = acc[u * 8 + 3] * a + p * bf16_hi(vv[r][u].y);
          acc[u * 8 + 4] = acc[u * 8 + 4] * a + p * bf16_lo(vv[r][u].z); acc[u * 8 + 5] = acc[u * 8 + 5] * a + p * bf16_hi(vv[r][u].z);
          acc[u * 8 + 6] = acc[u * 8 + 6] * a + p * bf16_lo(vv[r][u].w); acc[u * 8 + 7] = acc[u * 8 + 7] * a + p * bf16_hi(vv[r][u].w);
        }
      }
    }
  }
  // merge the eight key groups of the warp, then the warps
#pragma unroll
  for (int o = 4; o < 32; o <<= 1) {
    const float m_o = __shfl_xor_sync(0xffffffffu, m, o), l_o = __shfl_xor_sync(0xffffffffu, l, o);
    const float m_new = fmaxf(m, m_o);
    const float fa = m == -INFINITY ? 0.f : __expf(m - m_new), fb = m_o == -INFINITY ? 0.f : __expf(m_o - m_new);
    l = l * fa + l_o * fb;
    m = m_new;
#pragma unroll
    for (int e = 0; e < DPL; ++e) acc[e] = acc[e] * fa + __shfl_xor_sync(0xffffffffu, acc[e], o) * fb;
  }
  float* mine = sM + warp * (HD + 2);
  if (kg == 0) {
#pragma unroll
    for (int e = 0; e < DPL; ++e) mine[c4 * DPL + e] = acc[e];
    if (c4 == 0) { mine[HD] = m; mine[HD + 1] = l; }
  }
  df_sync();
  const int c = warp * 32 + lane;
  if (c < HD) {
    float mx = -INFINITY;
#pragma unroll
    for (int w = 0; w < DF_WARPS; ++w) mx = fmaxf(mx, sM[w * (HD + 2) + HD]);
    float lt = 0.f, ot = 0.f;
#pragma unroll
    for (int w = 0; w < DF_WARPS; ++w) {
      const float mw = sM[w * (HD + 2) + HD], f = mw == -INFINITY ? 0.f : __expf(mw - mx);
      lt += sM[w * (HD + 2) + HD + 1] * f;
      ot += sM[w * (HD + 2) + c] * f;
    }
    g.att[static_cast<long long>(t) * g.d + h * HD + c] = __float2bfloat16_rn(ot / lt);
  }
  df_sync();                                       // sM may be overwritten
}

// NB: trees, rounded up to 1, 2, 4, 8 or 16
template <int HD, int NB>
__global__ void __launch_bounds__(DF_THREADS, 1)
decode_few_kernel(const DecodeFewArgs g) {
  extern __shared__ __align__(128) uint8_t df_smem[];
  uint8_t* ring = df_smem;
  uint8_t* sA = ring + DF_STAGES * DF_SLOT;                          // DF_MAX_N rows of g.pitch bytes
  float* sP = reinterpret_cast<float*>(sA + DF_MAX_N * g.pitch);     // the warps' partial products
  float* sM = sP + DF_WARPS * DF_MAX_N * DF_PART;                    // 8 x (HD + 2): attention's merge
  DecodeLayer* sL = reinterpret_cast<DecodeLayer*>(sM + DF_WARPS * (HD + 2));
  DfTrees& sT = *reinterpret_cast<DfTrees*>(sL + g.n_layer);
  __shared__ float sR[2 * DF_WARPS];                                 // sums of a row's parts
  __shared__ __align__(16) float sN[2 * DF_MAX_K];                   // the next norm's weights and offsets
  __shared__ uint64_t full[DF_STAGES], empty[DF_STAGES];
  __shared__ int abort_word, met;
  volatile int* abort_flag = &abort_word;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int cta = blockIdx.x, ctas = gridDim.x;

  if (tid == 0) {
    for (int i = 0; i < DF_STAGES; ++i) { mbar_init(&full[i], 32); mbar_init(&empty[i], DF_WARPS / 2); }
    abort_word = 0;
    mbar_fence_init();
  }
  for (int i = tid * 16; i < DF_MAX_N * g.pitch; i += DF_THREADS * 16)     // rows past n stay zero
    *reinterpret_cast<uint4*>(sA + i) = make_uint4(0u, 0u, 0u, 0u);
  for (int i = tid; i < g.n_layer * static_cast<int>(sizeof(DecodeLayer) / 8); i += DF_THREADS)
    reinterpret_cast<unsigned long long*>(sL)[i] = reinterpret_cast<const unsigned long long*>(g.layers)[i];
  if (tid < g.n) {
    sT.active[tid] = g.active[tid];
    sT.slot[tid] = g.slot[tid];
    sT.prefix[tid] = g.prefix_len[tid];
    sT.n_anc[tid] = g.n_anc[tid];
  }
  for (int i = tid; i < g.n * DF_ANC; i += DF_THREADS) {
    const int t = i / DF_ANC, k = i % DF_ANC;
    if (k < g.anc_stride) sT.anc[t][k] = g.anc[static_cast<long long>(t) * g.anc_stride + k];
  }
  __syncthreads();

  if (warp == DF_WARPS) {
    // ------------------------------------------------------------------ producer
    int slot = 0;
    uint32_t par = 1;
    bool ok = true;
    for (int l = 0; l < g.n_layer && ok; ++l) {
      for (int m = 0; m < 4 && ok; ++m) {
        const DfMat p = df_mat(g, sL[l], m);
        for (int u = cta; u < p.units && ok; u += ctas) {
          const __nv_bfloat16* src = p.w + static_cast<long long>((u / p.blocks) * p.k + (lane >> 3)) * p.N +
                                     (u % p.blocks) * DF_COLS + (lane & 7) * 8;
          for (int c = 0; c < p.k / DF_CHUNK; ++c) {
            int w = 1;
            if (lane == 0) w = mbar_wait(&empty[slot], par, abort_flag) ? 1 : 0;
            w = __shfl_sync(0xffffffffu, w, 0);
            if (!w) { ok = false; break; }
            // row r, 16-byte chunk h at r * 128 + 16 * (h ^ (r & 7)): conflict-free for ldmatrix
            const uint32_t dst = smem_u32(ring + slot * DF_SLOT);
#pragma unroll
            for (int i = 0; i < DF_CHUNK / 4; ++i) {
              const int r = i * 4 + (lane >> 3);
              asm volatile("cp.async.cg.shared.global [%0], [%1], 16;"
                           ::"r"(dst + r * 128 + (((lane & 7) ^ (r & 7)) << 4)), "l"(src + static_cast<long long>(i) * 4 * p.N)
                           : "memory");
            }
            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(&full[slot])) : "memory");
            src += static_cast<long long>(DF_CHUNK) * p.N;
            if (++slot == DF_STAGES) { slot = 0; par ^= 1; }
          }
        }
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    if (!ok && lane == 0) { *abort_flag = ST_TIMEOUT_EMPTY; atomicCAS(g.status, 0, ST_TIMEOUT_EMPTY); }
    return;
  }

  // ------------------------------------------------------------------- computing warps
  int slot = 0;
  uint32_t par = 0;
  unsigned int target = 0;
  bool ok = true;       // uniform over the computing warps
  bool good = true;     // of this lane: after a wait that ran out it goes through the motions up to the meeting
  // All CTAs have finished the phase and see its results (read through L2 afterwards).  One addition and
  // one watching thread per CTA; the release and the acquire order the CTA's other accesses.  (A flag per
  // CTA that threads of all CTAs watch keeps 148 x 148 loads in flight and takes longer.)  The verdict is one
  // thread's: were each warp to read the abort flag, which the producer may set at any time, those that saw
  // it would leave and the others wait at the next df_sync for good.
  // `spare`: what the other warps do meanwhile.
  auto grid_barrier = [&](auto spare) {
    target += ctas;
    df_sync();
    if (warp > 0) {
      spare(tid - 32);
      asm volatile("cp.async.wait_all;" ::: "memory");     // load_norm's copies
    }
    if (tid == 0) {
      asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(g.arrivals) : "memory");
      const long long t0 = clock64();
      unsigned int seen, spins = 0;
      while (true) {
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(g.arrivals) : "memory");
        if (static_cast<int>(seen - target) >= 0) break;
        if ((++spins & 0xf) == 0 && (*abort_flag || clock64() - t0 > g.max_wait)) {
          *abort_flag = ST_TIMEOUT_MISC;
          atomicCAS(g.status, 0, ST_TIMEOUT_MISC);
          break;
        }
      }
      met = *abort_flag == 0;
    }
    df_sync();
    return met != 0;                               // rewritten behind the next meeting's first df_sync
  };
  // Vectors (norms, biases) and cached keys / values are read once per step, so they come from memory:
  // a latency in the middle of a phase, unless they are asked for a phase or a layer ahead.
  auto prefetch = [](const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); };
  constexpr int SPARE = (DF_WARPS - 1) * 32;       // threads that `spare` runs on
  auto prefetch_vectors = [&](int l, int st) {
    const float* v[8] = {sL[l].ln1_w, sL[l].ln1_b, sL[l].ln2_w, sL[l].ln2_b, sL[l].o_b, sL[l].pr_b, sL[l].qkv_b, sL[l].fc_b};
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int lines = (k < 6 ? g.d : k == 6 ? 3 * g.d : g.F) / 32;      // 128 bytes each, dealt out to the CTAs
      for (int i = st * ctas + cta; v[k] && i < lines; i += SPARE * ctas) prefetch(v[k] + i * 32);
    }
  };
  auto prefetch_keys = [&](const DecodeLayer& L, int st) {
    constexpr int LINES = HD / 64;
    for (int i = cta; i < g.n * g.H; i += ctas) {
      const int t = i / g.H;
      if (!sT.active[t]) continue;
      const long long base = static_cast<long long>(i) * g.S * HD;
      for (int j = st; j < sT.prefix[t] * LINES; j += SPARE) {
        prefetch(L.kc + base + j * 64);
        prefetch(L.vc + base + j * 64);
      }
    }
  };
  auto load_norm = [&](const float* w, const float* b, int st) {
    for (int i = st; i < g.d / 4; i += SPARE) {
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(sN + i * 4)), "l"(w + i * 4) : "memory");
      if (b)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(sN + DF_MAX_K + i * 4)), "l"(b + i * 4) : "memory");
      else
        *reinterpret_cast<float4*>(sN + DF_MAX_K + i * 4) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  };
  auto clear = [&](float* p, int count, int st) {  // this CTA's share
    for (int i = (cta * SPARE + st) * 4; i < count; i += ctas * SPARE * 4)
      __stcg(reinterpret_cast<float4*>(p + i), make_float4(0.f, 0.f, 0.f, 0.f));
  };
  // While the CTAs meet behind phase m of layer l: vectors of the next norm, accumulators that everybody has read
  // and that are added to behind the next meeting or later, and what the next layer will read, into L2.  (At
  // the start of a phase it was 600 to 2000 of the phase's clocks.)
  auto spare_work = [&](int l, int m, int st) {
    const bool more = l + 1 < g.n_layer;
    if (m == 0) {                                  // QKV done, FC's sums read by the phase before it
      load_norm(sL[l].ln2_w, sL[l].ln2_b, st);
      if (l > 0) clear(g.fc, g.n * g.F, st);
    } else if (m == 1) {                           // output projection done
      if (more) prefetch_vectors(l + 1, st);
    } else if (m == 2) {                           // FC done, QKV's sums read by attention
      if (more) load_norm(sL[l + 1].ln1_w, sL[l + 1].ln1_b, st);
      clear(g.qkv, g.n * 3 * g.d, st);
    } else if (more) {
      prefetch_keys(sL[l + 1], st);
    }
  };
  if (warp > 0) {
    prefetch_vectors(0, tid - 32);
    load_norm(sL[0].ln1_w, sL[0].ln1_b, tid - 32);
    prefetch_keys(sL[0], tid - 32);
    asm volatile("cp.async.wait_all;" ::: "memory");
  }
  df_sync();

  for (int l = 0; l < g.n_layer && ok; ++l) {
    const DecodeLayer& L = sL[l];
    for (int m = 0; m < 4 && ok; ++m) {
      if (m == 1) {
        for (int i = cta; i < g.n * g.H; i += ctas) {
          const int t = i / g.H;
          if (sT.active[t]) df_attention<HD>(g, L, sT, t, i - t * g.H, sM, warp, lane);
        }
        if (!(ok = grid_barrier([](int) {}))) break;
      }
      const DfMat p = df_mat(g, L, m);
      if (cta < p.units && m < 3) {                // the operand, all of its columns
        if (m == 1) {
          const int c8 = g.d >> 3;
          for (int i = tid; i < g.n * c8; i += DF_WARPS * 32) {
            const int r = i / c8, c = i - r * c8;
            *reinterpret_cast<uint4*>(sA + r * g.pitch + c * 16) =
                __ldcg(reinterpret_cast<const uint4*>(g.att + static_cast<long long>(r) * g.d) + c);
          }
        } else {
          df_norm<NB <= 4 ? 8 / NB : 1>(g, sN, sA, sR, warp, lane);
        }
        df_sync();
      }
      for (int u = cta; u < p.units; u += ctas) {
        const int ks = u / p.blocks;
        int a_col = ks * p.k;                      // first operand column in shared memory
        if (u != cta) df_sync();                   // operand and partial products of the unit before have been read
        if (m == 3) {                              // GELU of this slice of the FC accumulators
          const int c8 = p.k >> 3;
          for (int i = tid; i < g.n * c8; i += DF_WARPS * 32) {
            const int r = i / c8, c = (i - r * c8) * 8;
            *reinterpret_cast<uint4*>(sA + r * g.pitch + c * 2) =
                df_round8<true>(g.fc + static_cast<long long>(r) * g.F + a_col + c, L.fc_b ? L.fc_b + a_col + c : nullptr);
          }
          a_col = 0;
          df_sync();
        }
        // A warp multiplies 16 of a slot's 64 rows with all columns: warps 0 to 3 in the unit's even slots,
        // 4 to 7 in the odd ones.  (With all rows and eight of the columns every warp loads the whole operand,
        // 24 KB of shared memory per slot: 340 clocks a slot.)  The columns of W are the MMA's 16 rows and the
        // trees its eight columns: half the MMAs of the other way round for up to eight trees, and these are
        // what a slot's time goes into.
        constexpr int NT = NB > 8 ? 2 : 1;         // blocks of eight trees
        float acc[DF_COLS / 16][NT][4] = {};
        const int step = warp & 3, chunks = p.k / DF_CHUNK;
        // operand rows (trees) as the MMA's second operand: lanes 0 to 7 its first eight k, 8 to 15 the others, and
        // with 16 to 31 the same for the next eight trees
        const uint32_t a_addr = smem_u32(sA) + ((lane & 7) + (lane >> 4) * 8) * g.pitch + ((lane >> 3) & 1) * 16 +
                                (a_col + step * 16) * 2;
        const int w_k = (lane & 7) + (lane >> 4) * 8;        // row of the slot, of this warp's 16
        const uint32_t w_row = (step * 16 + w_k) * 128;
        for (int c = 0; c < chunks; ++c) {
          if ((c & 1) == (warp >> 2)) {            // warp-uniform
            // After a wait that ran out a lane goes on like the others, with whatever the slot holds: ldmatrix and
            // the MMAs are the whole warp's.  (A vote on the answer cost a step 7 us.)
            if (good && !mbar_wait(&full[slot], par, abort_flag)) {
              good = false;
              *abort_flag = ST_TIMEOUT_FULL;
              atomicCAS(g.status, 0, ST_TIMEOUT_FULL);
            }
            __syncwarp();
            const uint32_t w_addr = smem_u32(ring + slot * DF_SLOT) + w_row;
            uint32_t x[4], w[DF_COLS / 16][4];
            df_ldsm4(x, a_addr + c * DF_CHUNK * 2);
#pragma unroll
            for (int t = 0; t < DF_COLS / 16; ++t)           // 16 columns: two blocks of eight
              df_ldsm4_t(w[t], w_addr + (((2 * t + ((lane >> 3) & 1)) ^ (w_k & 7)) << 4));
#pragma unroll
            for (int t = 0; t < DF_COLS / 16; ++t)
#pragma unroll
              for (int j = 0; j < NT; ++j) df_mma(acc[t][j], w[t], x[2 * j], x[2 * j + 1]);
            __syncwarp();
            if (lane == 0) mbar_arrive(&empty[slot]);
          }
          if (++slot == DF_STAGES) { slot = 0; par ^= 1; }
        }
#pragma unroll
        for (int t = 0; t < DF_COLS / 16; ++t)
#pragma unroll
          for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const int r = j * 8 + (lane & 3) * 2 + (e & 1);
              if (r < g.n) sP[(warp * DF_MAX_N + r) * DF_PART + t * 16 + (lane >> 2) + (e >> 1) * 8] = acc[t][j][e];
            }
        df_sync();
        const int col = (u % p.blocks) * DF_COLS + lane * 2;
        float b0 = 0.f, b1 = 0.f;                  // the first slice carries the bias into the residual stream
        const float* bias = m == 1 ? L.o_b : L.pr_b;
        if ((m & 1) && ks == 0 && bias) { b0 = __ldg(bias + col); b1 = __ldg(bias + col + 1); }
        float* out = (m == 0 ? g.qkv : m == 2 ? g.fc : g.x) + col;
        for (int r = warp; r < g.n; r += DF_WARPS) {
          float s0 = b0, s1 = b1;
#pragma unroll
          for (int w = 0; w < DF_WARPS; ++w) {
            const float2 v = *reinterpret_cast<const float2*>(sP + (w * DF_MAX_N + r) * DF_PART + lane * 2);
            s0 += v.x;
            s1 += v.y;
          }
          df_red2(out + static_cast<long long>(r) * p.N, s0, s1);
        }
      }
      if (l + 1 < g.n_layer || m < 3) ok = grid_barrier([&](int st) { spare_work(l, m, st); });     // false for all warps once a wait ran out
    }
  }
}

}  // namespace ab

// Layers of one search step for n <= 16 trees.  `layers`: device array of DecodeLayer.  `work`: device
// scratch of 256 + n * (3 * d + F) words, cleared here.  `max_wait`: clock cycles after which a CTA gives up
// at a meeting (0: the usual second).  Returns 1, with no kernel launched, for shapes that the chain of
// kernels serves and where max_ctas CTAs cannot all be resident (a process that has part of the SMs).
extern "C" int ab_decode_few(const void* layers, int n_layer, int n, int d, int H, int F, int S, int rms, float eps,
                             float* x, void* att, const int* active, const int* slot, const int* prefix_len,
                             const int* anc, int anc_stride, const int* n_anc, void* work, int max_ctas,
                             long long max_wait, int* status, cudaStream_t stream) {
  using namespace ab;
  const int hd = H > 0 ? d / H : 0;
  if (n < 1 || n > DF_MAX_N || n_layer < 1 || n_layer > DF_MAX_LAYERS || d % 128 || F % 128 || d > DF_MAX_K ||
      H * hd != d || (hd != 64 && hd != 128) || max_ctas < 1)
    return 1;
  DecodeFewArgs g;
  // slices of a contraction: the fewest rows of W that the busiest CTA has to read, a unit's own cost
  // (operand, reductions) counted as 64 rows
  auto slices = [&](int K, int N) {
    int best = 0;
    long long cost = 0;
    for (int s = 1; s <= 32 && s * DF_CHUNK <= K; ++s) {
      if (K % (s * DF_CHUNK) || K / s > DF_MAX_K) continue;
      const long long units = static_cast<long long>(N / DF_COLS) * s, c = (units + max_ctas - 1) / max_ctas * (K / s + 64);
      if (!best || c < cost) { best = s; cost = c; }
    }
    return best;
  };
  g.slices[0] = slices(d, 3 * d);
  g.slices[1] = slices(d, d);
  g.slices[2] = slices(d, F);
  g.slices[3] = slices(F, d);
  if (!g.slices[0] || !g.slices[1] || !g.slices[2] || !g.slices[3]) return 1;
  const int longest = d > F / g.slices[3] ? d : F / g.slices[3];
  g.layers = static_cast<const DecodeLayer*>(layers);
  g.n_layer = n_layer; g.n = n; g.d = d; g.H = H; g.F = F; g.S = S; g.rms = rms; g.eps = eps;
  g.scale = 1.f / sqrtf(static_cast<float>(hd));
  g.x = x;
  g.att = static_cast<__nv_bfloat16*>(att);
  g.arrivals = static_cast<unsigned int*>(work);
  g.qkv = static_cast<float*>(work) + DF_WORK_HEAD;
  g.fc = g.qkv + static_cast<long long>(n) * 3 * d;
  g.active = active; g.slot = slot; g.prefix_len = prefix_len; g.anc = anc; g.anc_stride = anc_stride; g.n_anc = n_anc;
  g.pitch = longest * 2 + 16;                      // eight rows fall on different banks
  g.max_wait = max_wait > 0 ? max_wait : AB_SPIN_CYCLES;
  g.status = status;
  const int smem = DF_STAGES * DF_SLOT + DF_MAX_N * g.pitch + DF_WARPS * (DF_MAX_N * DF_PART + hd + 2) * 4 +
                   n_layer * (int)sizeof(DecodeLayer) + (int)sizeof(DfTrees);
  using Kernel = void (*)(const DecodeFewArgs);
  static const Kernel kernels[2][5] = {
      {decode_few_kernel<64, 1>, decode_few_kernel<64, 2>, decode_few_kernel<64, 4>, decode_few_kernel<64, 8>, decode_few_kernel<64, 16>},
      {decode_few_kernel<128, 1>, decode_few_kernel<128, 2>, decode_few_kernel<128, 4>, decode_few_kernel<128, 8>, decode_few_kernel<128, 16>}};
  const int nb = n == 1 ? 0 : n == 2 ? 1 : n <= 4 ? 2 : n <= 8 ? 3 : 4;
  const Kernel kern = kernels[hd == 128][nb];
  // the most any model needs, once: set to each call's own size, one thread's call lowers the limit between
  // another's setting and its launch
  constexpr int SMEM_MAX = DF_STAGES * DF_SLOT + DF_MAX_N * (DF_MAX_K * 2 + 16) +
                           DF_WARPS * (DF_MAX_N * DF_PART + 128 + 2) * 4 +
                           DF_MAX_LAYERS * (int)sizeof(DecodeLayer) + (int)sizeof(DfTrees);
  static PerDeviceOnce attr[2][5];
  PerDeviceOnce& once = attr[hd == 128][nb];
  cudaError_t e = cudaSuccess;
  if (once.first_use_on_device()) {
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_MAX);
    if (e != cudaSuccess) return -static_cast<int>(e);
    once.mark_device();
  }
  int per_sm = 0, sms = 0, dev = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, DF_THREADS, smem);
  if (e == cudaSuccess) e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return -static_cast<int>(e);
  if (per_sm * sms < max_ctas) return 1;
  e = cudaMemsetAsync(work, 0, sizeof(float) * (DF_WORK_HEAD + static_cast<size_t>(n) * (3 * d + F)), stream);
  if (e != cudaSuccess) return -static_cast<int>(e);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(max_ctas);
  cfg.blockDim = dim3(DF_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;       // all CTAs resident, or the launch is refused
  at[0].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  e = cudaLaunchKernelEx(&cfg, kern, g);
  if (e == cudaErrorCooperativeLaunchTooLarge) {   // nothing was launched, and nothing is wrong otherwise
    cudaGetLastError();
    return 1;
  }
  return -static_cast<int>(e);
}
