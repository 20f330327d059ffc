// Fused output-embedding GEMM + cross entropy for training (forward and the gradient of the
// logits in one launch; the logits themselves never reach memory).
//
//   logits[m, :] = h[m, :] . wte^T        (bf16 operands, fp32 accumulation in TMEM)
//   loss        += sum over rows with label >= 0 of  logsumexp(logits[m, :]) - logits[m, label[m]]
//   dlogits[m, n] = (softmax(logits[m, :])[n] - [n == label[m]]) * coef / n_valid   (0 for ignored rows)
//
// Up to 4096 columns (lmhead_ce_cluster_kernel): a cluster of CTAs owns 128 rows, each CTA 512 columns of the
// vocabulary, which is what TMEM holds.  The CTAs exchange every row's maximum, sum of exponentials and label
// logit through distributed shared memory and turn the accumulators, still in place, into the gradient.
// Larger vocabularies (lmhead_ce_kernel): a CTA walks the vocabulary in tiles of 256 columns, TWICE: the first
// sweep keeps a running maximum and sum of exponentials per row (online softmax across the N tiles) and picks
// up the label's logit; the second recomputes every tile on the tensor cores.  2048 columns, rows x width, that
// form (as it was before the cluster, its loads and MMAs issued by one lane) and the cluster: 300 x 512 70 and 25 us,
// 2048 x 256 53 and 21, 12136 x 768 99 and 72, 32768 x 1024 248 and 202.  Where the line lies, both as they
// are: 2048 x 256 with 4096 columns by cluster 39 us, with 4104 by two sweeps 98.
//
// Same pipeline as the plain GEMM (gemm_tc.cu): warp 0 TMA producer, warp 1 MMA issuer, 16 epilogue
// warps (four per TMEM lane quarter, 64 columns each), two accumulators in TMEM so the epilogue of
// tile i overlaps the MMAs of tile i + 1.  Every wait is bounded and reports through `status`.
#include "gemm_core.cuh"

namespace ab {

constexpr int LC_BN = 256;
constexpr int LC_STAGES = 3;      // 3 x 48 KB operand stages leave room for the row statistics

struct LmCeArgs {
  int M, V, K;
  const int* labels;      // [M], < 0 = ignored
  const int* n_valid;     // device scalar: rows with a label
  float coef;
  float* loss_acc;        // += sum of the rows' negative log likelihoods
  int* status;
};

__global__ void __launch_bounds__(NUM_THREADS, 1)
lmhead_ce_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                 const __grid_constant__ CUtensorMap tmOut, const LmCeArgs g) {
  griddep_enter();
  constexpr int BN = LC_BN, STAGES = LC_STAGES;
  constexpr int A_BYTES = BM * BK * 2;
  constexpr int B_BYTES = BN * BK * 2;
  constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  constexpr int TMEM_COLS = 2 * BN;
  constexpr float L2E = 1.4426950408889634f;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* stage_out = smem + STAGES * STAGE_BYTES;                 // 2 KB per epilogue warp
  // row statistics shared between the sweeps: [2 unit parities][3: max, sum, label logit][4 parts][128 rows]
  float* s_stat = reinterpret_cast<float*>(stage_out + NUM_EPI_WARPS * 2048);
  uint64_t* bars = reinterpret_cast<uint64_t*>(s_stat + 2 * 3 * 4 * BM);
  uint64_t* full_bar = bars;
  uint64_t* empty_bar = bars + STAGES;
  uint64_t* tfull_bar = bars + 2 * STAGES;
  uint64_t* tempty_bar = bars + 2 * STAGES + 2;
  uint64_t* stat_bar = bars + 2 * STAGES + 4;       // the 16 epilogue warps meet here once per unit
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 5);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = warp_number();
  const int lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(&tfull_bar[i], 1); mbar_init(&tempty_bar[i], NUM_EPI_WARPS); }
    mbar_init(stat_bar, NUM_EPI_WARPS);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
    tma_prefetch_desc(&tmOut);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  const int m_tiles = (g.M + BM - 1) / BM;
  const int n_tiles = (g.V + BN - 1) / BN;
  const int kb_total = (g.K + BK - 1) / BK;
  const int tiles_per_unit = 2 * n_tiles;                  // two sweeps over the vocabulary

  if (warp == 0) {
    // ------------------------------------------------------- TMA producer
    {
      const uint32_t lead = elect_one();
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int u = blockIdx.x; u < m_tiles && ok; u += gridDim.x) {
        const int m0 = u * BM;
        for (int t = 0; t < tiles_per_unit && ok; ++t) {
          const int n0 = (t % n_tiles) * BN;
          for (int kb = 0; kb < kb_total; ++kb) {
            if (!mbar_wait_warp(&empty_bar[stage], phase ^ 1, abort_flag)) {
              *abort_flag = ST_TIMEOUT_EMPTY;
              if (lead) atomicCAS(g.status, 0, ST_TIMEOUT_EMPTY);
              ok = false;
              break;
            }
            uint8_t* sa = smem + stage * STAGE_BYTES;
            mbar_expect_tx(&full_bar[stage], STAGE_BYTES, lead);
            tma_load_2d(sa, &tmA, &full_bar[stage], kb * BK, m0, lead);
            tma_load_2d(sa + A_BYTES, &tmB, &full_bar[stage], kb * BK, n0, lead);
            if (++stage == STAGES) { stage = 0; phase ^= 1; }
          }
        }
      }
    }
  } else if (warp == 1) {
    // --------------------------------------------------------- MMA issuer
    {
      const uint32_t lead = elect_one();
      constexpr uint32_t idesc = make_idesc_bf16(BM, BN, 0, 0);
      int stage = 0;
      uint32_t phase = 0;
      uint32_t acc_phase[2] = {0, 0};
      int it = 0;
      bool ok = true;
      for (int u = blockIdx.x; u < m_tiles && ok; u += gridDim.x) {
        for (int t = 0; t < tiles_per_unit && ok; ++t, ++it) {
          const int ab = it & 1;
          if (!mbar_wait_warp(&tempty_bar[ab], acc_phase[ab] ^ 1, abort_flag)) {
            *abort_flag = ST_TIMEOUT_TMEM_EMPTY;
            if (lead) atomicCAS(g.status, 0, ST_TIMEOUT_TMEM_EMPTY);
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t d_tmem = tmem_base + ab * BN;
          for (int kb = 0; kb < kb_total; ++kb) {
            if (!mbar_wait_warp(&full_bar[stage], phase, abort_flag)) {
              *abort_flag = ST_TIMEOUT_FULL;
              if (lead) atomicCAS(g.status, 0, ST_TIMEOUT_FULL);
              ok = false;
              break;
            }
            tc_fence_after();
            const uint32_t sa = smem_u32(smem + stage * STAGE_BYTES);
            const uint32_t sb = sa + A_BYTES;
#pragma unroll
            for (int k = 0; k < BK / UMMA_K; ++k) {
              const uint64_t adesc = make_sdesc_sw128(sa, k * UMMA_K * 2, 16, 1024);
              const uint64_t bdesc = make_sdesc_sw128(sb, k * UMMA_K * 2, 16, 1024);
              umma_bf16(d_tmem, adesc, bdesc, idesc, (kb > 0 || k > 0) ? 1u : 0u, lead);
            }
            umma_commit(&empty_bar[stage], lead);
            if (++stage == STAGES) { stage = 0; phase ^= 1; }
          }
          if (!ok) break;
          umma_commit(&tfull_bar[ab], lead);
          acc_phase[ab] ^= 1;
        }
      }
    }
  } else {
    // ----------------------------------------------------------- epilogue
    const int e = warp - 2;
    const int quad = warp & 3;           // TMEM lane quarter this warp may read
    const int part = e >> 2;             // which 64 of the tile's 256 columns
    constexpr int COLS_PER_WARP = BN / 4;
    uint8_t* my_stage = stage_out + e * 2048;
    const int rloc = quad * 32 + lane;   // row inside the 128-row tile
    uint32_t acc_phase[2] = {0, 0};
    int it = 0;
    const int nval = __ldg(g.n_valid);
    const float gscale = nval > 0 ? g.coef / static_cast<float>(nval) : 0.f;
    float loss_local = 0.f;
    bool ok = true;
    uint32_t unit_it = 0;
    for (int u = blockIdx.x; u < m_tiles && ok; u += gridDim.x, ++unit_it) {
      float* s_m = s_stat + (unit_it & 1) * (3 * 4 * BM);     // double-buffered by unit parity: a warp can
      float* s_l = s_m + 4 * BM;                              // only overwrite a buffer after every warp
      float* s_lab = s_l + 4 * BM;                            // has passed the meeting that follows its use
      const int m = u * BM + rloc;
      const int m0w = u * BM + quad * 32;
      const bool row_in = m < g.M;
      const int label = row_in ? __ldg(g.labels + m) : -1;
      float rm = -INFINITY, rl = 0.f, rlab = -INFINITY, lse = 0.f;
      for (int t = 0; t < tiles_per_unit; ++t, ++it) {
        const int ab = it & 1;
        const int sweep = t / n_tiles;
        const int nbase = (t % n_tiles) * BN + part * COLS_PER_WARP;
        if (sweep == 1 && t == n_tiles) {
          // between the sweeps: the four column parts of a row share their statistics
          s_m[part * BM + rloc] = rm;
          s_l[part * BM + rloc] = rl;
          s_lab[part * BM + rloc] = rlab;
          __syncwarp();
          if (lane == 0) mbar_arrive(stat_bar);
          if (!mbar_wait_warp(stat_bar, unit_it & 1, abort_flag)) {     // bounded, and it sees another warp's abort
            *abort_flag = ST_TIMEOUT_MISC;
            atomicCAS(g.status, 0, ST_TIMEOUT_MISC);
            ok = false;
            break;
          }
          float M4 = -INFINITY;
#pragma unroll
          for (int p = 0; p < 4; ++p) M4 = fmaxf(M4, s_m[p * BM + rloc]);
          float L4 = 0.f, lab = -INFINITY;
#pragma unroll
          for (int p = 0; p < 4; ++p) {
            const float mp = s_m[p * BM + rloc];
            if (mp != -INFINITY) L4 += s_l[p * BM + rloc] * ex2_fast((mp - M4) * L2E);
            lab = fmaxf(lab, s_lab[p * BM + rloc]);
          }
          lse = M4 + logf(L4);
          if (part == 0 && label >= 0) loss_local += lse - lab;
        }
        if (!mbar_wait_warp(&tfull_bar[ab], acc_phase[ab], abort_flag)) {
          *abort_flag = ST_TIMEOUT_TMEM_FULL;
          atomicCAS(g.status, 0, ST_TIMEOUT_TMEM_FULL);
          ok = false;
          break;
        }
        acc_phase[ab] ^= 1;
        tc_fence_after();
        const uint32_t taddr =
            tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + ab * BN + part * COLS_PER_WARP;
#pragma unroll 1
        for (int rd = 0; rd < COLS_PER_WARP / 16; ++rd) {
          const int n0 = nbase + rd * 16;
          if (n0 >= g.V) break;                             // warp-uniform
          uint32_t r[16];
          tmem_ld16(taddr + rd * 16, r);
          if (sweep == 1 && lane == 0) tma_store_wait_read<0>();   // staging tile free again
          __syncwarp();
          tmem_ld_wait();
          if (sweep == 0) {
            float tm = -INFINITY;
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              const float v = (n0 + j < g.V) ? __uint_as_float(r[j]) : -INFINITY;
              tm = fmaxf(tm, v);
              if (n0 + j == label) rlab = v;
            }
            const float m_new = fmaxf(rm, tm);
            float s = 0.f;
#pragma unroll
            for (int j = 0; j < 16; ++j)
              if (n0 + j < g.V) s += ex2_fast((__uint_as_float(r[j]) - m_new) * L2E);
            rl = rl * ex2_fast((rm - m_new) * L2E) + s;
            rm = m_new;
          } else {
#pragma unroll
            for (int grp = 0; grp < 2; ++grp) {
              float p[8];
#pragma unroll
              for (int j = 0; j < 8; ++j) {
                const int n = n0 + grp * 8 + j;
                float v = 0.f;
                if (label >= 0 && n < g.V) {
                  v = ex2_fast((__uint_as_float(r[grp * 8 + j]) - lse) * L2E) * gscale;
                  if (n == label) v -= gscale;
                }
                p[j] = v;
              }
              // 16 bf16 columns = 32-byte rows, 32B swizzle: chunk index ^= (row >> 2) & 1
              const uint32_t off = lane * 32 + ((grp ^ ((lane >> 2) & 1)) << 4);
              uint4 o;
              o.x = pack_bf16x2(p[0], p[1]); o.y = pack_bf16x2(p[2], p[3]);
              o.z = pack_bf16x2(p[4], p[5]); o.w = pack_bf16x2(p[6], p[7]);
              *reinterpret_cast<uint4*>(my_stage + off) = o;
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
              tma_store_2d(&tmOut, my_stage, n0, m0w);
              tma_store_commit();
            }
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&tempty_bar[ab]);
      }
    }
    if (lane == 0) tma_store_wait<0>();
    // loss: only the part-0 warps hold row losses
#pragma unroll
    for (int o = 16; o; o >>= 1) loss_local += __shfl_xor_sync(0xffffffffu, loss_local, o);
    if (lane == 0 && part == 0 && loss_local != 0.f) atomicAdd(g.loss_acc, loss_local);
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

// ------------------------------------------------------------------------------------------
constexpr int LX_TILES = 2;                                 // accumulators of a CTA
constexpr int LX_COLS = LX_TILES * LC_BN;                   // columns of a CTA
constexpr int LX_MAX_CTAS = 8;
constexpr int LX_STAGING = 4096;                            // 32 rows x 64 bf16 columns per epilogue warp

template <int C>
__global__ void __cluster_dims__(C, 1, 1) __launch_bounds__(NUM_THREADS, 1)
lmhead_ce_cluster_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                         const __grid_constant__ CUtensorMap tmOut, const LmCeArgs g) {
  griddep_enter();
  constexpr int BN = LC_BN, STAGES = LC_STAGES;
  constexpr int A_BYTES = BM * BK * 2;
  constexpr int B_BYTES = BN * BK * 2;
  constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  constexpr float L2E = 1.4426950408889634f;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* stage_out = smem + STAGES * STAGE_BYTES;
  // [3: max, sum, label logit][4 parts][128 rows]; read for the last time before the staging tiles are used
  float* s_stat = reinterpret_cast<float*>(stage_out);
  // [C][3][128 rows], written by the CTAs of the cluster
  float* s_all = reinterpret_cast<float*>(stage_out + NUM_EPI_WARPS * LX_STAGING);
  uint64_t* bars = reinterpret_cast<uint64_t*>(s_all + C * 3 * BM);
  uint64_t* full_bar = bars;
  uint64_t* empty_bar = bars + STAGES;
  uint64_t* tfull_bar = bars + 2 * STAGES;
  uint64_t* stat_bar = bars + 2 * STAGES + LX_TILES;        // this CTA's epilogue warps meet
  uint64_t* all_bar = stat_bar + 1;                         // four warps of every CTA have written s_all
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(all_bar + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = warp_number();
  const int lane = threadIdx.x & 31;
  const int rank = static_cast<int>(cluster_ctarank());
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    for (int i = 0; i < LX_TILES; ++i) mbar_init(&tfull_bar[i], 1);
    mbar_init(stat_bar, NUM_EPI_WARPS);
    mbar_init(all_bar, 4 * C);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
    tma_prefetch_desc(&tmOut);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, LX_TILES * BN);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();           // the barriers of all CTAs are initialised before any is signalled
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  const int m0 = static_cast<int>(blockIdx.x) / C * BM;
  const int first = rank * LX_COLS;                         // first column of this CTA
  const int tiles = min(LX_TILES, (g.V - first + BN - 1) / BN);      // may be none (or negative)
  const int kb_total = (g.K + BK - 1) / BK;

  if (warp == 0) {
    // ------------------------------------------------------- TMA producer
    {
      const uint32_t lead = elect_one();
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int t = 0; t < tiles && ok; ++t) {
        for (int kb = 0; kb < kb_total; ++kb) {
          if (!mbar_wait_warp(&empty_bar[stage], phase ^ 1, abort_flag)) {
            *abort_flag = ST_TIMEOUT_EMPTY;
            if (lead) atomicCAS(g.status, 0, ST_TIMEOUT_EMPTY);
            ok = false;
            break;
          }
          uint8_t* sa = smem + stage * STAGE_BYTES;
          mbar_expect_tx(&full_bar[stage], STAGE_BYTES, lead);
          tma_load_2d(sa, &tmA, &full_bar[stage], kb * BK, m0, lead);
          tma_load_2d(sa + A_BYTES, &tmB, &full_bar[stage], kb * BK, first + t * BN, lead);
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    // --------------------------------------------------------- MMA issuer
    {
      const uint32_t lead = elect_one();
      constexpr uint32_t idesc = make_idesc_bf16(BM, BN, 0, 0);
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int t = 0; t < tiles && ok; ++t) {
        for (int kb = 0; kb < kb_total; ++kb) {
          if (!mbar_wait_warp(&full_bar[stage], phase, abort_flag)) {
            *abort_flag = ST_TIMEOUT_FULL;
            if (lead) atomicCAS(g.status, 0, ST_TIMEOUT_FULL);
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t sa = smem_u32(smem + stage * STAGE_BYTES);
          const uint32_t sb = sa + A_BYTES;
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k)
            umma_bf16(tmem_base + t * BN, make_sdesc_sw128(sa, k * UMMA_K * 2, 16, 1024),
                      make_sdesc_sw128(sb, k * UMMA_K * 2, 16, 1024), idesc, (kb > 0 || k > 0) ? 1u : 0u, lead);
          umma_commit(&empty_bar[stage], lead);
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
        if (ok) umma_commit(&tfull_bar[t], lead);
      }
    }
  } else {
    // ----------------------------------------------------------- epilogue
    const int e = warp - 2;
    const int quad = warp & 3;           // TMEM lane quarter this warp may read
    const int part = e >> 2;             // which 64 of a tile's 256 columns
    constexpr int COLS_PER_WARP = BN / 4;
    uint8_t* stg = stage_out + e * LX_STAGING;
    const int rloc = quad * 32 + lane;   // row inside the 128-row tile
    const int m = m0 + rloc;
    const int label = m < g.M ? __ldg(g.labels + m) : -1;
    const int nval = __ldg(g.n_valid);
    const float gscale = nval > 0 ? g.coef / static_cast<float>(nval) : 0.f;
    const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + part * COLS_PER_WARP;
    float rm = -INFINITY, rl = 0.f, rlab = -INFINITY;
    bool ok = true;
    for (int t = 0; t < tiles && ok; ++t) {
      if (!mbar_wait_warp(&tfull_bar[t], 0, abort_flag)) {
        *abort_flag = ST_TIMEOUT_TMEM_FULL;
        atomicCAS(g.status, 0, ST_TIMEOUT_TMEM_FULL);
        ok = false;
        break;
      }
      tc_fence_after();
#pragma unroll 1
      for (int h = 0; h < 2; ++h) {
        const int n0 = first + t * BN + part * COLS_PER_WARP + h * 32;
        if (n0 >= g.V) break;                               // warp-uniform
        uint32_t r[32];
        tmem_ld32(taddr + t * BN + h * 32, r);
        tmem_ld_wait();
        float tm = -INFINITY;
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          const float v = (n0 + j < g.V) ? __uint_as_float(r[j]) : -INFINITY;
          tm = fmaxf(tm, v);
          if (n0 + j == label) rlab = v;
        }
        const float m_new = fmaxf(rm, tm);
        float s = 0.f;
#pragma unroll
        for (int j = 0; j < 32; ++j)
          if (n0 + j < g.V) s += ex2_fast((__uint_as_float(r[j]) - m_new) * L2E);
        rl = rl * ex2_fast((rm - m_new) * L2E) + s;
        rm = m_new;
      }
    }
    // the four column parts of a row share their statistics, and then the CTAs of the cluster
    s_stat[part * BM + rloc] = rm;
    s_stat[(4 + part) * BM + rloc] = rl;
    s_stat[(8 + part) * BM + rloc] = rlab;
    __syncwarp();
    if (lane == 0) mbar_arrive(stat_bar);
    if (ok && !mbar_wait_warp(stat_bar, 0, abort_flag)) {
      *abort_flag = ST_TIMEOUT_MISC;
      atomicCAS(g.status, 0, ST_TIMEOUT_MISC);
      ok = false;
    }
    // of n statistics `stride` floats apart: maximum, sum of exponentials below it, label logit
    auto merge = [&](const float* pm, const float* pl, const float* pb, int n, int stride, float& M, float& L, float& lab) {
      M = lab = -INFINITY;
      L = 0.f;
      for (int i = 0; i < n; ++i) M = fmaxf(M, pm[i * stride]);
      for (int i = 0; i < n; ++i) {
        const float mi = pm[i * stride];
        if (mi != -INFINITY) L += pl[i * stride] * ex2_fast((mi - M) * L2E);
        lab = fmaxf(lab, pb[i * stride]);
      }
    };
    if (part == 0) {                     // four warps tell every CTA of the cluster, this one included
      float M, L, lab;
      merge(s_stat + rloc, s_stat + 4 * BM + rloc, s_stat + 8 * BM + rloc, 4, BM, M, L, lab);
      const uint32_t mine = smem_u32(s_all + rank * 3 * BM + rloc);
#pragma unroll
      for (int c = 0; c < C; ++c) {
        const uint32_t dst = mapa_shared(mine, c);
        asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(dst), "f"(M) : "memory");
        asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(dst + BM * 4), "f"(L) : "memory");
        asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(dst + BM * 8), "f"(lab) : "memory");
      }
      asm volatile("fence.acq_rel.cluster;" ::: "memory");
      __syncwarp();
      if (lane == 0) {
#pragma unroll
        for (int c = 0; c < C; ++c) mbar_arrive_cluster(mapa_shared(smem_u32(all_bar), c));
      }
    }
    if (ok && !mbar_wait_warp(all_bar, 0, abort_flag)) {
      *abort_flag = ST_TIMEOUT_MISC;
      atomicCAS(g.status, 0, ST_TIMEOUT_MISC);
      ok = false;
    }
    asm volatile("fence.acq_rel.cluster;" ::: "memory");
    if (ok) {
      float M, L, lab;
      merge(s_all + rloc, s_all + BM + rloc, s_all + 2 * BM + rloc, C, 3 * BM, M, L, lab);
      const float lse = M + logf(L);
      for (int t = 0; t < tiles; ++t) {
        const int nbase = first + t * BN + part * COLS_PER_WARP;
        if (nbase >= g.V || m0 + quad * 32 >= g.M) break;   // warp-uniform
        if (t > 0) {
          if (lane == 0) tma_store_wait_read<0>();          // staging tile free again
          __syncwarp();
        }
#pragma unroll 1
        for (int h = 0; h < 2; ++h) {
          uint32_t r[32];
          tmem_ld32(taddr + t * BN + h * 32, r);
          tmem_ld_wait();
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            float p[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              float v = 0.f;
              if (label >= 0) {
                v = ex2_fast((__uint_as_float(r[c * 8 + j]) - lse) * L2E) * gscale;
                if (nbase + h * 32 + c * 8 + j == label) v -= gscale;
              }
              p[j] = v;                                     // columns past V are clipped by the store
            }
            *reinterpret_cast<uint4*>(stg + lane * 128 + (((h * 4 + c) ^ (lane & 7)) << 4)) =
                make_uint4(pack_bf16x2(p[0], p[1]), pack_bf16x2(p[2], p[3]), pack_bf16x2(p[4], p[5]), pack_bf16x2(p[6], p[7]));
          }
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          tma_store_2d(&tmOut, stg, nbase, m0 + quad * 32);
          tma_store_commit();
        }
      }
      if (lane == 0) tma_store_wait<0>();
      if (rank == 0 && part == 0) {      // one warp of the cluster per 32 rows
        float loss = label >= 0 ? lse - lab : 0.f;
#pragma unroll
        for (int o = 16; o; o >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, o);
        if (lane == 0 && loss != 0.f) atomicAdd(g.loss_acc, loss);
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  cluster_sync_all();           // nobody writes into another CTA's shared memory after this point
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, LX_TILES * BN);
  }
}

template <int C>
static int launch_lmhead_cluster(const CUtensorMap& tmA, const CUtensorMap& tmB, const CUtensorMap& tmOut,
                                 const LmCeArgs& g, cudaStream_t stream) {
  if constexpr (C < LX_MAX_CTAS) {
    if (g.V > C * LX_COLS) return launch_lmhead_cluster<2 * C>(tmA, tmB, tmOut, g, stream);
  }
  constexpr int SMEM = 1024 + LC_STAGES * (BM * BK * 2 + LC_BN * BK * 2) + NUM_EPI_WARPS * LX_STAGING +
                       C * 3 * BM * 4 + 256;
  static_assert(SMEM <= 227 * 1024, "shared memory");
  static PerDeviceOnce attr_set;
  auto kern = lmhead_ce_cluster_kernel<C>;
  if (attr_set.first_use_on_device()) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
    if (e != cudaSuccess) return static_cast<int>(e);
    attr_set.mark_device();
  }
  launch_chained(kern, dim3((g.M + BM - 1) / BM * C), dim3(NUM_THREADS), SMEM, stream, tmA, tmB, tmOut, g);
  return static_cast<int>(cudaGetLastError());
}

}  // namespace ab

// h: [M, K] bf16 (final hidden states), wte: [V, K] bf16, labels: [M] int (already shifted, < 0 =
// ignored), dlogits: [M, V] bf16 out.  K, V multiples of 8.  max_ctas bounds the CTAs of the two-sweep form; the
// clusters, one per 128 rows, are launched all at once.
extern "C" int ab_lmhead_ce(const void* h, long long ldh, const void* wte, long long ldw, const int* labels,
                            const int* n_valid, float coef, void* dlogits, long long ldo, float* loss_acc,
                            int M, int V, int K, int max_ctas, int* status, cudaStream_t stream) {
  using namespace ab;
  if (M <= 0 || V <= 0 || K <= 0 || (V & 7) || (K & 7) || (ldh & 7) || (ldw & 7) || (ldo & 7) || !status) return -1;
  if ((reinterpret_cast<uintptr_t>(h) | reinterpret_cast<uintptr_t>(wte) | reinterpret_cast<uintptr_t>(dlogits)) & 15)
    return -3;
  CUtensorMap tmA, tmB, tmOut;
  int rc = make_tmap_2d(&tmA, h, M, K, ldh, BM, BK, 2, true);
  if (rc) return rc;
  rc = make_tmap_2d(&tmB, wte, V, K, ldw, LC_BN, BK, 2, true);
  if (rc) return rc;
  LmCeArgs g;
  g.M = M; g.V = V; g.K = K; g.labels = labels; g.n_valid = n_valid; g.coef = coef; g.loss_acc = loss_acc;
  g.status = status;
  if (V <= LX_MAX_CTAS * LX_COLS) {
    rc = make_tmap_2d_sw(&tmOut, dlogits, M, V, ldo, 32, 64, 2, 128);
    return rc ? rc : launch_lmhead_cluster<1>(tmA, tmB, tmOut, g, stream);
  }
  rc = make_tmap_2d_sw(&tmOut, dlogits, M, V, ldo, 32, 16, 2, 32);
  if (rc) return rc;
  constexpr int SMEM = 1024 + LC_STAGES * (BM * BK * 2 + LC_BN * BK * 2) + NUM_EPI_WARPS * 2048 + 2 * 3 * 4 * BM * 4 + 256;
  static PerDeviceOnce attr_set;
  if (attr_set.first_use_on_device()) {
    cudaError_t e = cudaFuncSetAttribute(lmhead_ce_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
    if (e != cudaSuccess) return static_cast<int>(e);
    attr_set.mark_device();
  }
  if (max_ctas <= 0) max_ctas = 148;
  const int m_tiles = (M + BM - 1) / BM;
  const int grid = m_tiles < max_ctas ? m_tiles : max_ctas;
  launch_chained(lmhead_ce_kernel, dim3(grid), dim3(NUM_THREADS), SMEM, stream, tmA, tmB, tmOut, g);
  return static_cast<int>(cudaGetLastError());
}
