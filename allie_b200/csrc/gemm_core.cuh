// Device-side pieces shared by the tcgen05 GEMM kernels (gemm_tc.cu: plain and CTA-pair kernels;
// gemm_grouped.cu: the grouped CTA-pair kernel of the MoE expert layers): tile constants, the
// kernel argument block, the fused epilogue math and the routines with which an epilogue warp
// drains its part of a finished accumulator.
#pragma once
#include "gemm_tc.cuh"
#include "ptx.cuh"

namespace ab {

constexpr int BM = 128;
constexpr int BK = 64;
constexpr int UMMA_K = 16;
constexpr int NUM_EPI_WARPS = 16;
constexpr int NUM_THREADS = 64 + 32 * NUM_EPI_WARPS;

// CTA-pair kernels (cta_group::2, 256 x 256 tiles)
constexpr int PAIR_STAGES = 5;
constexpr int PAIR_WARP_STAGING = 4096;   // one wide staging tile per epilogue warp
constexpr int PAIR_BN = 256;      // instruction N; each CTA stages PAIR_BN / 2 columns of B

// Equal shares of an accumulation for all CTA pairs: `waves` rounds of whole tiles, then `rest` tiles that are cut
// along the contraction into `slices` parts of `q` steps, a pair each, and what is left of each, `r` steps; the
// pairs that are over take these, `extra_q` steps each of them all laid end to end.
struct EvenShare {
  int on, pairs, waves, rest, slices, q, r, extra_q;
};
// i-th unit of a pair: steps [kb0, kb1) of a tile; false when it has no more
__host__ __device__ inline bool even_unit(const EvenShare& s, int steps, int pair, int i, int& tile, int& kb0, int& kb1) {
  if (i < s.waves) {
    tile = i * s.pairs + pair; kb0 = 0; kb1 = steps;
    return true;
  }
  i -= s.waves;
  const int first = s.waves * s.pairs, main = s.slices * s.rest;
  if (pair < main) {
    tile = first + pair % s.rest;
    kb0 = pair / s.rest * s.q;
    kb1 = kb0 + s.q < steps ? kb0 + s.q : steps;
    return i == 0 && kb0 < kb1;
  }
  if (s.r == 0) return false;
  const int x0 = (pair - main) * s.extra_q, all = s.rest * s.r, x1 = x0 + s.extra_q < all ? x0 + s.extra_q : all;
  const int t = x0 / s.r + i;
  const int a = t * s.r > x0 ? t * s.r : x0, b = (t + 1) * s.r < x1 ? (t + 1) * s.r : x1;
  tile = first + t;
  kb0 = s.slices * s.q + a - t * s.r;
  kb1 = s.slices * s.q + b - t * s.r;
  return a < b;
}

struct GemmArgs {
  int M, N, K;
  int k_splits;
  int pdl;            // launched as a programmatic dependent: B (weights) may be fetched before griddep_wait
  int aux_tma;        // CTA-pair kernel: a second epilogue operand arrives by TMA in the warp's staging tile
                      // (tmAux is a load map) instead of by row loads.  1: the aux tile of act == 2,
                      // 64 bf16 columns; 2: the residual, 32 fp32 columns at a time
  EvenShare even;     // CTA-pair kernel, EPI_ACCUM
  int accum_steps;    // likewise: steps that one accumulator sums up
  AbGemmEpilogue ep;
  const unsigned long long* salt;   // seed_salt_ptr() at launch: folded into ep.drop_seed when not null
  int* status;
};

// Fused epilogue math for 8 adjacent columns n..n+7 of row m.  `v` comes in as the raw fp32
// accumulators and leaves as the final values; `pre` receives the bf16 pre-activation when
// act == 1.  Reads (bias, aux for act == 2, residual) are predicated by the caller's `ok`.
// `bias_off` shifts the bias vector (grouped GEMMs: one bias row per group).
__device__ __forceinline__ void epilogue_math8(const GemmArgs& g, float* v, uint4& pre, int m, int n,
                                               bool ok, bool add_bias, int bias_off = 0,
                                               const uint4* aux_staged = nullptr) {
  const AbGemmEpilogue& ep = g.ep;
  if (ep.alpha != 1.f) {
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] *= ep.alpha;
  }
  if (!ok) return;
  if (ep.bias && add_bias) {      // with split-K only the first split carries the bias
    const float4 b0 = __ldg(reinterpret_cast<const float4*>(ep.bias + bias_off + n));
    const float4 b1 = __ldg(reinterpret_cast<const float4*>(ep.bias + bias_off + n + 4));
    v[0] += b0.x; v[1] += b0.y; v[2] += b0.z; v[3] += b0.w;
    v[4] += b1.x; v[5] += b1.y; v[6] += b1.z; v[7] += b1.w;
  }
  if (ep.act == 1 && ep.aux_grad) {
    // the second output is gelu'(pre-activation): the backward epilogue only multiplies by it
    float d[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = gelu_tanh_with_grad(v[j], d[j]);
    pre.x = pack_bf16x2(d[0], d[1]); pre.y = pack_bf16x2(d[2], d[3]);
    pre.z = pack_bf16x2(d[4], d[5]); pre.w = pack_bf16x2(d[6], d[7]);
  } else if (ep.act == 1) {
    pre.x = pack_bf16x2(v[0], v[1]); pre.y = pack_bf16x2(v[2], v[3]);
    pre.z = pack_bf16x2(v[4], v[5]); pre.w = pack_bf16x2(v[6], v[7]);
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = gelu_tanh(v[j]);
  } else if (ep.act == 3) {        // GELU without keeping the pre-activation (inference)
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = gelu_tanh(v[j]);
  } else if (ep.act == 2) {
    // the eight aux values: from the staged tile in shared memory, or straight from global
    const uint4 q = aux_staged ? *aux_staged
                               : *reinterpret_cast<const uint4*>(
                                     static_cast<const __nv_bfloat16*>(ep.aux) + (long long)m * ep.ldaux + n);
    if (ep.aux_grad) {        // aux already holds the derivative (written by an act == 1 launch with aux_grad)
      v[0] *= bf16_lo(q.x); v[1] *= bf16_hi(q.x); v[2] *= bf16_lo(q.y); v[3] *= bf16_hi(q.y);
      v[4] *= bf16_lo(q.z); v[5] *= bf16_hi(q.z); v[6] *= bf16_lo(q.w); v[7] *= bf16_hi(q.w);
    } else {
    v[0] *= gelu_tanh_grad(bf16_lo(q.x)); v[1] *= gelu_tanh_grad(bf16_hi(q.x));
    v[2] *= gelu_tanh_grad(bf16_lo(q.y)); v[3] *= gelu_tanh_grad(bf16_hi(q.y));
    v[4] *= gelu_tanh_grad(bf16_lo(q.z)); v[5] *= gelu_tanh_grad(bf16_hi(q.z));
    v[6] *= gelu_tanh_grad(bf16_lo(q.w)); v[7] *= gelu_tanh_grad(bf16_hi(q.w));
    }
  }
  if (ep.resid) {
    if (ep.drop_thr16) {
      const uint64_t group = (static_cast<uint64_t>(m) * g.N + n) >> 3;
      const uint32_t keep = dropout_keep8(salted(ep.drop_seed, g.salt), ep.drop_stream, group, ep.drop_thr16);
      const float s = dropout_scale(ep.drop_thr16);
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = ((keep >> j) & 1u) ? v[j] * s : 0.f;
    }
    const float4 r0 = *reinterpret_cast<const float4*>(ep.resid + (long long)m * ep.ldr + n);
    const float4 r1 = *reinterpret_cast<const float4*>(ep.resid + (long long)m * ep.ldr + n + 4);
    v[0] += r0.x; v[1] += r0.y; v[2] += r0.z; v[3] += r0.w;
    v[4] += r1.x; v[5] += r1.y; v[6] += r1.z; v[7] += r1.w;
  }
}

// One epilogue warp drains its 32 rows x COLS columns of a finished accumulator: TMEM -> registers
// -> fused math -> swizzled staging tile -> TMA store (or reduce-add), 16 columns per round.
template <int COLS>
__device__ __forceinline__ void epilogue_drain(const GemmArgs& g, const CUtensorMap& tmOut,
                                               const CUtensorMap& tmAux, uint32_t taddr, int m,
                                               int m0w, int nbase, bool row_ok, uint8_t* my_stage,
                                               int lane, bool add_bias) {
#pragma unroll 1
  for (int rd = 0; rd < COLS / 16; ++rd) {      // rounds of 16 columns
    const int n0 = nbase + rd * 16;
    if (n0 >= g.N) break;                                 // warp-uniform
    uint32_t r[16];
    tmem_ld16(taddr + rd * 16, r);
    if (lane == 0) tma_store_wait_read<0>();              // staging tile free again
    __syncwarp();
    tmem_ld_wait();
#pragma unroll
    for (int grp = 0; grp < 2; ++grp) {
      const int n = n0 + grp * 8;
      float v[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = __uint_as_float(r[grp * 8 + j]);
      uint4 pre = make_uint4(0, 0, 0, 0);
      epilogue_math8(g, v, pre, m, n, row_ok && n < g.N, add_bias);
      if (g.ep.out_fp32) {
        // 16 fp32 columns = 64-byte rows, 64B swizzle: 16-byte chunk index ^= (row >> 1) & 3
        uint8_t* rowp = my_stage + lane * 64;
        const int sw = (lane >> 1) & 3;
        *reinterpret_cast<float4*>(rowp + (((2 * grp) ^ sw) << 4)) = make_float4(v[0], v[1], v[2], v[3]);
        *reinterpret_cast<float4*>(rowp + (((2 * grp + 1) ^ sw) << 4)) = make_float4(v[4], v[5], v[6], v[7]);
      } else {
        // 16 bf16 columns = 32-byte rows, 32B swizzle: chunk index ^= (row >> 2) & 1
        const uint32_t off = lane * 32 + ((grp ^ ((lane >> 2) & 1)) << 4);
        uint4 o;
        o.x = pack_bf16x2(v[0], v[1]); o.y = pack_bf16x2(v[2], v[3]);
        o.z = pack_bf16x2(v[4], v[5]); o.w = pack_bf16x2(v[6], v[7]);
        *reinterpret_cast<uint4*>(my_stage + off) = o;
        if (g.ep.act == 1) *reinterpret_cast<uint4*>(my_stage + 1024 + off) = pre;
      }
    }
    fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0) {
      if (g.ep.accumulate) tma_reduce_add_2d(&tmOut, my_stage, n0, m0w);
      else                 tma_store_2d(&tmOut, my_stage, n0, m0w);
      if (g.ep.act == 1) tma_store_2d(&tmAux, my_stage + 1024, n0, m0w);
      tma_store_commit();
    }
  }
}

// ------------------------------------------------------------------------------------------
// Specialised drains of the CTA-pair kernels.  The general routine below decides per eight columns
// what an output needs; at 256 x 256 tiles and K = 1024 its branches cost as many issue slots as
// the tensor core leaves (32768 x 4096 x 1024, bf16 output: 227 us against 191 us with the stores
// and the math taken out).  The kernels of the training and inference schedule therefore know at
// compile time which of these they are; everything else takes EPI_ANY.
enum EpiKind : int {
  EPI_ANY = 0,
  EPI_BF16,        // bf16 out (+ bias)
  EPI_GELU,        // bf16 out = gelu(. + bias), nothing kept
  EPI_GELU_GRAD,   // bf16 out = gelu(. + bias), second bf16 output = gelu'
  EPI_MUL,         // bf16 out = . * aux tile (aux_grad), aux staged by TMA
  EPI_RESID,       // fp32 out = dropout(. + bias) + residual, residual staged by TMA
  EPI_ACCUM,       // fp32 out += .
  EPI_DOT,         // bf16 out, and per row and 64 columns its product with the aux tile (staged by TMA)
};

// which specialised drain an epilogue description fits (aux_tma as chosen by the launcher)
inline EpiKind epi_kind(const GemmArgs& g) {
  const AbGemmEpilogue& ep = g.ep;
  if (ep.alpha != 1.f) return EPI_ANY;
  if (ep.accumulate) return (!ep.bias && !ep.act && !ep.resid) ? EPI_ACCUM : EPI_ANY;
  if (ep.resid) return g.aux_tma == 2 ? EPI_RESID : EPI_ANY;
  if (ep.out_fp32) return EPI_ANY;
  if (ep.act == 0) return EPI_BF16;
  if (ep.act == 3) return EPI_GELU;
  if (ep.act == 4) return EPI_DOT;       // the entry point has checked the rest
  if (ep.act == 1 && ep.aux_grad) return EPI_GELU_GRAD;
  if (ep.act == 2 && ep.aux_grad && g.aux_tma == 1 && !ep.bias) return EPI_MUL;
  return EPI_ANY;
}

// eight accumulators (+ bias) as four packed pairs; `n` and `has` are warp-uniform
__device__ __forceinline__ void epi_load8(const uint32_t* r, uint64_t* v, const float* bias, int n, bool has) {
#pragma unroll
  for (int j = 0; j < 4; ++j) v[j] = f2_pack(__uint_as_float(r[2 * j]), __uint_as_float(r[2 * j + 1]));
  if (has) {
    const float4 b0 = __ldg(reinterpret_cast<const float4*>(bias + n));
    const float4 b1 = __ldg(reinterpret_cast<const float4*>(bias + n + 4));
    v[0] = f2_add(v[0], f2_pack(b0.x, b0.y)); v[1] = f2_add(v[1], f2_pack(b0.z, b0.w));
    v[2] = f2_add(v[2], f2_pack(b1.x, b1.y)); v[3] = f2_add(v[3], f2_pack(b1.z, b1.w));
  }
}
__device__ __forceinline__ uint4 epi_pack8(const uint64_t* v) {
  return make_uint4(f2_to_bf16x2(v[0]), f2_to_bf16x2(v[1]), f2_to_bf16x2(v[2]), f2_to_bf16x2(v[3]));
}

// EPI_ACCUM: a warp's 32 rows x 64 columns of sums, two to a register pair, are added to the output by the TMA unit;
// 32 fp32 columns at a time = 128-byte rows, 128B swizzle
__device__ __forceinline__ void epilogue_add_sums(const CUtensorMap& tmOut, const uint64_t* sum, int nbase, int m0w, int N,
                                                  uint8_t* stg, int lane) {
#pragma unroll
  for (int grp = 0; grp < 2; ++grp) {
    if (nbase + grp * 32 >= N) break;      // warp-uniform
    if (lane == 0) tma_store_wait_read<0>();
    __syncwarp();
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      float4 v;
      f2_unpack(sum[grp * 16 + c * 2], v.x, v.y);
      f2_unpack(sum[grp * 16 + c * 2 + 1], v.z, v.w);
      *reinterpret_cast<float4*>(stg + lane * 128 + ((c ^ (lane & 7)) << 4)) = v;
    }
    fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0) {
      tma_reduce_add_2d(&tmOut, stg, nbase + grp * 32, m0w);
      tma_store_commit();
    }
  }
}

// One epilogue warp drains its 32 rows x 64 columns.  Rows past the end of the output are clipped by
// the TMA store.  `wait_tile` / `next_tile`: see EPI_RESID.  Returns false when a wait ran out.
template <int EPI, typename Wait, typename Next>
__device__ __forceinline__ bool epilogue_drain_kind(const GemmArgs& g, const CUtensorMap& tmOut,
                                                    const CUtensorMap& tmAux, uint32_t taddr, int m, int m0w,
                                                    int nbase, uint8_t* stg, int lane, Wait wait_tile,
                                                    Next next_tile) {
  const float* bias = g.ep.bias;
  const bool has_bias = bias != nullptr;
  if constexpr (EPI == EPI_BF16 || EPI == EPI_GELU || EPI == EPI_MUL || EPI == EPI_DOT) {
    // one store group: 64 bf16 columns = 128-byte rows, 128B swizzle.  The aux tile of EPI_MUL and
    // EPI_DOT lies in the staging tile already, in the same layout.
    constexpr bool AUX = EPI == EPI_MUL || EPI == EPI_DOT;
    uint8_t* rowp = stg + lane * 128;
    const int sw = lane & 7;
    uint64_t dot = 0;                    // EPI_DOT: two partial sums
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      uint32_t r[32];
      tmem_ld32(taddr + half * 32, r);
      if (half == 0) {
        if constexpr (AUX) {
          if (!wait_tile()) return false;
        } else {
          if (lane == 0) tma_store_wait_read<0>();        // staging tile free again
          __syncwarp();
        }
      }
      tmem_ld_wait();
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int n = nbase + half * 32 + c * 8;
        uint64_t v[4];
        epi_load8(r + c * 8, v, bias, n, !AUX && has_bias && n < g.N);
        uint4* chunk = reinterpret_cast<uint4*>(rowp + (((half * 4 + c) ^ sw) << 4));
        if constexpr (EPI == EPI_GELU) {
#pragma unroll
          for (int j = 0; j < 4; ++j) v[j] = f2_gelu_tanh(v[j]);
        }
        if constexpr (EPI == EPI_MUL) {
          const uint4 q = *chunk;
          v[0] = f2_mul(v[0], f2_pack(bf16_lo(q.x), bf16_hi(q.x)));
          v[1] = f2_mul(v[1], f2_pack(bf16_lo(q.y), bf16_hi(q.y)));
          v[2] = f2_mul(v[2], f2_pack(bf16_lo(q.z), bf16_hi(q.z)));
          v[3] = f2_mul(v[3], f2_pack(bf16_lo(q.w), bf16_hi(q.w)));
        }
        const uint4 o = epi_pack8(v);
        if constexpr (EPI == EPI_DOT) {
          const uint4 q = *chunk;
          dot = f2_fma(f2_pack(bf16_lo(o.x), bf16_hi(o.x)), f2_pack(bf16_lo(q.x), bf16_hi(q.x)), dot);
          dot = f2_fma(f2_pack(bf16_lo(o.y), bf16_hi(o.y)), f2_pack(bf16_lo(q.y), bf16_hi(q.y)), dot);
          dot = f2_fma(f2_pack(bf16_lo(o.z), bf16_hi(o.z)), f2_pack(bf16_lo(q.z), bf16_hi(q.z)), dot);
          dot = f2_fma(f2_pack(bf16_lo(o.w), bf16_hi(o.w)), f2_pack(bf16_lo(q.w), bf16_hi(q.w)), dot);
        }
        *chunk = o;
      }
    }
    fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0) {
      tma_store_2d(&tmOut, stg, nbase, m0w);
      tma_store_commit();
    }
    if constexpr (EPI == EPI_MUL) {
      if (g.ep.colsum) {
        // Column sums of the tile just staged (rows past M are zeros): each lane adds up two columns, a
        // row of shared memory per load, while the store leaves.  The issue slots are free: the tensor
        // core needs 8192 clocks per 256 x 256 tile at K = 1024, this takes 600 of the epilogue's.  A
        // pass of its own over 32768 x 4096 took 55 us.
        uint64_t s2[2] = {0ull, 0ull};
#pragma unroll 8
        for (int row = 0; row < 32; ++row) {
          const uint32_t w = *reinterpret_cast<const uint32_t*>(
              stg + row * 128 + (((lane >> 2) ^ (row & 7)) << 4) + (lane & 3) * 4);
          s2[row & 1] = f2_add(s2[row & 1], f2_pack(bf16_lo(w), bf16_hi(w)));
        }
        float a0, a1;
        f2_unpack(f2_add(s2[0], s2[1]), a0, a1);
        const int n = nbase + lane * 2;
        if (n < g.N)
          asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(g.ep.colsum + n), "f"(a0), "f"(a1) : "memory");
        __syncwarp();                      // all lanes have read the tile
      }
    }
    if constexpr (EPI == EPI_DOT) {
      float a0, a1;
      f2_unpack(dot, a0, a1);
      if (m < g.M) {
        const int seq = m / g.ep.dot_T;
        g.ep.dot_out[(static_cast<long long>(seq) * (g.N >> 6) + (nbase >> 6)) * g.ep.dot_T + (m - seq * g.ep.dot_T)] = a0 + a1;
      }
    }
    if constexpr (AUX) {
      if (lane == 0) {
        tma_store_wait_read<0>();          // the store has read the staging tile
        next_tile(0);
      }
    }
  } else if constexpr (EPI == EPI_GELU_GRAD) {
    // two bf16 outputs share the staging tile: 32 columns each = 64-byte rows, 64B swizzle
    const int sw = (lane >> 1) & 3;
#pragma unroll
    for (int grp = 0; grp < 2; ++grp) {
      const int gn0 = nbase + grp * 32;
      if (gn0 >= g.N) break;               // warp-uniform
      uint32_t r[32];
      tmem_ld32(taddr + grp * 32, r);
      if (lane == 0) tma_store_wait_read<0>();
      __syncwarp();
      tmem_ld_wait();
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int n = gn0 + c * 8;
        uint64_t v[4], d[4];
        epi_load8(r + c * 8, v, bias, n, has_bias && n < g.N);
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] = f2_gelu_tanh_with_grad(v[j], d[j]);
        uint8_t* dst = stg + lane * 64 + ((c ^ sw) << 4);
        *reinterpret_cast<uint4*>(dst) = epi_pack8(v);
        *reinterpret_cast<uint4*>(dst + 2048) = epi_pack8(d);
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        tma_store_2d(&tmOut, stg, gn0, m0w);
        tma_store_2d(&tmAux, stg + 2048, gn0, m0w);
        tma_store_commit();
      }
    }
  } else {
    static_assert(EPI == EPI_RESID, "no drain for this epilogue kind");
    // fp32 output with a residual.  A lane owns a row, so residual loads straight from global would
    // touch 32 rows per instruction and keep the load unit busy for longer than the tensor core
    // needs at K <= 1024 (12136 x 768 x 768: 35.5 us; 27.9 us with the tiles by TMA).  The 32 x 32
    // residual tile of a column group lies in the staging tile, in the layout of the output tile,
    // and each lane replaces its values by the results before the tile leaves.  `wait_tile()` waits
    // for the current group's tile; `next_tile(grp)` is called by lane 0 once group grp has been
    // stored and the staging tile is free again.
    uint8_t* rowp = stg + lane * 128;
    const int sw = lane & 7;
    const uint32_t thr16 = g.ep.drop_thr16;
    const uint64_t s2 = f2_bcast(dropout_scale(thr16));
#pragma unroll 1
    for (int grp = 0; grp < 2; ++grp) {
      const int gn0 = nbase + grp * 32;
      if (gn0 >= g.N) break;               // warp-uniform
      uint32_t r[32];
      tmem_ld32(taddr + grp * 32, r);
      uint32_t keep = 0xffffffffu;         // does not depend on the accumulator: drawn under the load
      if (thr16) {
        const uint64_t seed = uniform64(salted(g.ep.drop_seed, g.salt));
        const uint64_t group0 = (static_cast<uint64_t>(m) * g.N + gn0) >> 3;
        keep = dropout_keep32(seed, g.ep.drop_stream, group0, thr16);
      }
      if (!wait_tile()) return false;
      tmem_ld_wait();
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int n = gn0 + c * 8;
        uint64_t v[4];
        epi_load8(r + c * 8, v, bias, n, has_bias && n < g.N);
        float4* s0 = reinterpret_cast<float4*>(rowp + (((2 * c) ^ sw) << 4));
        float4* s1 = reinterpret_cast<float4*>(rowp + (((2 * c + 1) ^ sw) << 4));
        const float4 r0 = *s0, r1 = *s1;
        const uint64_t res[4] = {f2_pack(r0.x, r0.y), f2_pack(r0.z, r0.w), f2_pack(r1.x, r1.y), f2_pack(r1.z, r1.w)};
        float o[8];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (thr16) {               // selected, not multiplied by zero: a dropped Inf or NaN is a zero
            float x0, x1;
            f2_unpack(f2_mul(v[j], s2), x0, x1);
            v[j] = f2_pack(((keep >> (c * 8 + 2 * j)) & 1u) ? x0 : 0.f, ((keep >> (c * 8 + 2 * j + 1)) & 1u) ? x1 : 0.f);
          }
          f2_unpack(f2_add(v[j], res[j]), o[2 * j], o[2 * j + 1]);
        }
        *s0 = make_float4(o[0], o[1], o[2], o[3]);
        *s1 = make_float4(o[4], o[5], o[6], o[7]);
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        tma_store_2d(&tmOut, stg, gn0, m0w);
        tma_store_commit();
        tma_store_wait_read<0>();
        next_tile(grp);
      }
    }
  }
  return true;
}

// General drain of the CTA-pair kernels (EPI_ANY, and the grouped kernel): the same per-round math as
// epilogue_drain, but several 16-column rounds are staged side by side in one 4 KB tile per warp and
// leave in one TMA store with 128-byte rows (64 bf16 or 32 fp32 columns; 64-byte rows when a second
// bf16 output shares the tile).  Wide rows matter: the store path costs per row segment, not per byte.
template <int COLS>
__device__ __forceinline__ void epilogue_drain_wide(const GemmArgs& g, const CUtensorMap& tmOut,
                                                    const CUtensorMap& tmAux, uint32_t taddr, int m,
                                                    int m0w, int nbase, bool row_ok, uint8_t* stg,
                                                    int lane, bool add_bias, int bias_off = 0,
                                                    bool aux_in_stage = false) {
  // aux_in_stage (act == 2, one bf16 output, COLS == 64): the staging tile already holds the aux
  // tile in the layout of the output tile (same box, same swizzle), so a lane reads its eight aux
  // values from the very chunk it then overwrites with its eight results.
  const bool two = g.ep.act == 1, f32 = g.ep.out_fp32 != 0;
  const int gcols = (f32 || two) ? 32 : 64;             // columns per TMA store (warp-uniform)
#pragma unroll 1
  for (int g0 = 0; g0 < COLS; g0 += gcols) {
    const int gn0 = nbase + g0;
    if (gn0 >= g.N) break;                              // warp-uniform
    if (lane == 0) tma_store_wait_read<0>();            // staging tile free again
    __syncwarp();
#pragma unroll 1
    for (int rd = 0; rd < gcols / 16; ++rd) {
      const int n0 = gn0 + rd * 16;
      if (n0 >= g.N) break;
      uint32_t r[16];
      tmem_ld16(taddr + g0 + rd * 16, r);
      tmem_ld_wait();
#pragma unroll
      for (int grp = 0; grp < 2; ++grp) {
        const int n = n0 + grp * 8;
        float v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = __uint_as_float(r[grp * 8 + j]);
        uint4 pre = make_uint4(0, 0, 0, 0);
        const uint4* staged = aux_in_stage
            ? reinterpret_cast<const uint4*>(stg + lane * 128 + (((rd * 2 + grp) ^ (lane & 7)) << 4)) : nullptr;
        epilogue_math8(g, v, pre, m, n, row_ok && n < g.N, add_bias, bias_off, staged);
        if (f32) {
          // 32 fp32 columns = 128-byte rows, 128B swizzle: 16-byte chunk index ^= row & 7
          uint8_t* rowp = stg + lane * 128;
          const int c = rd * 4 + grp * 2, sw = lane & 7;
          *reinterpret_cast<float4*>(rowp + ((c ^ sw) << 4)) = make_float4(v[0], v[1], v[2], v[3]);
          *reinterpret_cast<float4*>(rowp + (((c + 1) ^ sw) << 4)) = make_float4(v[4], v[5], v[6], v[7]);
        } else {
          uint4 o;
          o.x = pack_bf16x2(v[0], v[1]); o.y = pack_bf16x2(v[2], v[3]);
          o.z = pack_bf16x2(v[4], v[5]); o.w = pack_bf16x2(v[6], v[7]);
          const int c = rd * 2 + grp;
          if (two) {   // 32 bf16 columns = 64-byte rows, 64B swizzle; pre-activation tile 2 KB further
            const uint32_t off = lane * 64 + ((c ^ ((lane >> 1) & 3)) << 4);
            *reinterpret_cast<uint4*>(stg + off) = o;
            *reinterpret_cast<uint4*>(stg + 2048 + off) = pre;
          } else {     // 64 bf16 columns = 128-byte rows, 128B swizzle
            *reinterpret_cast<uint4*>(stg + lane * 128 + ((c ^ (lane & 7)) << 4)) = o;
          }
        }
      }
    }
    fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0) {
      if (g.ep.accumulate) tma_reduce_add_2d(&tmOut, stg, gn0, m0w);
      else                 tma_store_2d(&tmOut, stg, gn0, m0w);
      if (two) tma_store_2d(&tmAux, stg + 2048, gn0, m0w);
      tma_store_commit();
    }
  }
}

}  // namespace ab
