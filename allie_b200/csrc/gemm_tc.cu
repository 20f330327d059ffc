// Persistent, warp-specialised bf16 GEMM for sm_100a.
//
//   warp 0      : TMA producer   (cp.async.bulk.tensor into a STAGES-deep smem ring)
//   warp 1      : MMA issuer     (one thread issues tcgen05.mma; accumulators live in TMEM)
//   warps 2..17 : epilogue       (tcgen05.ld TMEM -> registers -> fused epilogue -> global);
//                 four warps per TMEM lane quarter, each owning a quarter of the tile's columns
//
// The 512 TMEM columns hold two 128 x BN fp32 accumulators, so the epilogue of
// work unit i overlaps the main loop of unit i+1.  Work units are
// (output tile, K split) pairs handed out round-robin to a grid of at most one
// CTA per SM.  Operands may be K-major or MN-major in memory (the UMMA
// descriptors express both), which covers forward (X*W), dgrad (dY*W^T) and
// wgrad (X^T*dY) of a layer whose weight is stored [in][out] without any
// transposed copies.  No TMA multicast is used anywhere.
#include "gemm_core.cuh"
#include <cstdlib>

namespace ab {

EncodeTiledFn get_encode_tiled() {
  static EncodeTiledFn fn = nullptr;
  static bool tried = false;
  if (!tried) {
    tried = true;
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  }
  return fn;
}

int make_tmap_2d(CUtensorMap* out, const void* base, uint64_t rows, uint64_t cols, uint64_t ld,
                 uint32_t box_rows, uint32_t box_cols, int elem_bytes, bool swizzle128) {
  return make_tmap_2d_sw(out, base, rows, cols, ld, box_rows, box_cols, elem_bytes,
                         swizzle128 ? 128 : 0);
}

int make_tmap_2d_sw(CUtensorMap* out, const void* base, uint64_t rows, uint64_t cols, uint64_t ld,
                    uint32_t box_rows, uint32_t box_cols, int elem_bytes, int swizzle_bytes) {
  EncodeTiledFn enc = get_encode_tiled();
  if (!enc) return -100;
  cuuint64_t dims[2] = {cols, rows};
  cuuint64_t strides[1] = {ld * static_cast<uint64_t>(elem_bytes)};
  cuuint32_t box[2] = {box_cols, box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUtensorMapDataType dt = elem_bytes == 2   ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16
                           : elem_bytes == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32
                                             : CU_TENSOR_MAP_DATA_TYPE_UINT8;
  CUresult r = enc(out, dt, 2, const_cast<void*>(base), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE,
                   swizzle_bytes == 128  ? CU_TENSOR_MAP_SWIZZLE_128B
                   : swizzle_bytes == 64 ? CU_TENSOR_MAP_SWIZZLE_64B
                   : swizzle_bytes == 32 ? CU_TENSOR_MAP_SWIZZLE_32B
                                         : CU_TENSOR_MAP_SWIZZLE_NONE,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -200 - static_cast<int>(r);
}

// KSUB: 64-wide steps of the contraction per stage.  Two for the 64-column tiles, whose four MMAs a step take no longer
// than the waits and commits around them (chain of 90 x 1024 x 1024 launches: 5.8 us with one, 5.45 with two).
template <int TM, int BN, int STAGES, int KSUB, bool A_MN, bool B_MN>
__global__ void __launch_bounds__(NUM_THREADS, 1)
gemm_bf16_tcgen05_kernel(const __grid_constant__ CUtensorMap tmA,
                         const __grid_constant__ CUtensorMap tmB,
                         const __grid_constant__ CUtensorMap tmOut,
                         const __grid_constant__ CUtensorMap tmAux, const GemmArgs g) {
  static_assert(TM == 128 || (TM == 64 && !A_MN), "rows of a tile");
  constexpr int A_BYTES = TM * BK * 2;
  constexpr int B_BYTES = BN * BK * 2;
  constexpr int SUB_BYTES = A_BYTES + B_BYTES, STAGE_BYTES = KSUB * SUB_BYTES;
  constexpr int BKS = KSUB * BK;          // contraction columns of a stage
  constexpr int TMEM_COLS = 2 * BN;  // 256 or 512, power of two
  static_assert(TMEM_COLS == 256 || TMEM_COLS == 512 || TMEM_COLS == 128 || TMEM_COLS == 64, "bad BN");
  // 32 columns of an MN-major B: rows of 64 bytes, swizzled over 64 (else panels of 64 columns, over 128)
  constexpr bool B_HALF_PANEL = B_MN && BN == 32;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  // per-epilogue-warp staging tiles for the TMA stores: 2 KB each (32 rows x 16 columns of
  // fp32, or 32 x 16 bf16 output + 32 x 16 bf16 pre-activation)
  uint8_t* stage_out = smem + STAGES * STAGE_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(stage_out + NUM_EPI_WARPS * 2048);
  uint64_t* full_bar = bars;
  uint64_t* empty_bar = bars + STAGES;
  uint64_t* tfull_bar = bars + 2 * STAGES;
  uint64_t* tempty_bar = bars + 2 * STAGES + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = warp_number();
  const int lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&tfull_bar[i], 1);
      mbar_init(&tempty_bar[i], NUM_EPI_WARPS);
    }
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
    tma_prefetch_desc(&tmOut);
    if (g.ep.act == 1) tma_prefetch_desc(&tmAux);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, TMEM_COLS);
    tmem_relinquish();
  }
  // the kernel behind this one in the stream may begin its own set-up now
  if (threadIdx.x == 0) griddep_launch_dependents();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  // As a programmatic dependent this kernel may be running before its predecessor has finished:
  // only the weight operand B (and the set-up above) is touched before griddep_wait.  m_limit /
  // k_limit are device values of earlier kernels, so such launches are never made dependent.
  if (warp >= 2) {
    // the bias is a weight: brought near while the kernel before is still running, its first use comes when the
    // accumulator is ready and would wait for memory
    if (g.pdl && g.ep.bias) {
      const int n_tiles = (g.N + BN - 1) / BN, n = (blockIdx.x % n_tiles) * BN + (warp - 2) * 32 + lane;
      if (warp - 2 < BN / 32 && n < g.N) asm volatile("prefetch.global.L2 [%0];" ::"l"(g.ep.bias + n));
    }
    griddep_wait();                       // epilogue: residual / aux reads and every store come after
  }

  const int Meff = g.ep.m_limit ? min(g.M, __ldg(g.ep.m_limit)) : g.M;
  const int Keff = g.ep.k_limit ? min(g.K, __ldg(g.ep.k_limit)) : g.K;
  const int m_tiles = (Meff + TM - 1) / TM;
  const int n_tiles = (g.N + BN - 1) / BN;
  const int kb_total = (Keff + BKS - 1) / BKS;
  const int kb_per = (kb_total + g.k_splits - 1) / g.k_splits;
  const int num_tiles = m_tiles * n_tiles;
  // units are ordered K-split-major: CTAs running at the same time work on the same K range of
  // different output tiles, so each operand slab is fetched from HBM once and shared through L2
  const int num_units = num_tiles * g.k_splits;

  if (warp == 0) {
    // ------------------------------------------------------- TMA producer
    const uint32_t lead = elect_one();
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    auto load_b = [&](uint8_t* sb, uint64_t* bar, int k0, int n0) {
      if constexpr (!B_MN) {
        tma_load_2d(sb, &tmB, bar, k0, n0, lead);
      } else {
#pragma unroll
        for (int i = 0; i < (BN + 63) / 64; ++i) tma_load_2d(sb + i * (BK * 128), &tmB, bar, n0 + i * 64, k0, lead);
      }
    };
    // dependent launch: the first ring-full of weight tiles of my first unit goes out while the
    // kernel before this one is still running; the activations follow after griddep_wait
    int prefetched = 0;
    if (g.pdl) {
      const int u = blockIdx.x;
      if (u < num_units) {
        const int ks = u / num_tiles, tile = u % num_tiles;
        const int n0 = (tile % n_tiles) * BN;
        const int kb0 = ks * kb_per, kb1 = min(kb_total, kb0 + kb_per);
        for (int kb = kb0; kb < kb1 && prefetched < STAGES; ++kb, ++prefetched) {
          mbar_expect_tx(&full_bar[prefetched], STAGE_BYTES, lead);      // the stages are all free at start
#pragma unroll
          for (int j = 0; j < KSUB; ++j)
            load_b(smem + prefetched * STAGE_BYTES + j * SUB_BYTES + A_BYTES, &full_bar[prefetched], kb * BKS + j * BK, n0);
        }
      }
    }
    // A chain of launches over a few rows streams the weights of a whole model, and none of them is long or
    // wide enough to keep memory busy by itself: each asks for the weights of the next into L2.
    if (g.pdl && g.ep.next_b) {
      const long long per = ((g.ep.next_bytes + gridDim.x - 1) / gridDim.x + 127) & ~127ll;
      const long long end = min(g.ep.next_bytes, (blockIdx.x + 1) * per);
      for (long long o = blockIdx.x * per; o < end; o += 16384)
        if (lead) bulk_prefetch_l2(static_cast<const uint8_t*>(g.ep.next_b) + o, static_cast<uint32_t>(min(16384ll, end - o)));
    }
    griddep_wait();       // no-op unless launched as a dependent (decode step, captured training step)
    for (int u = blockIdx.x; u < num_units && ok; u += gridDim.x) {
      const int ks = u / num_tiles;
      const int tile = u % num_tiles;
      const int m0 = (tile / n_tiles) * TM;
      const int n0 = (tile % n_tiles) * BN;
      const int kb0 = ks * kb_per;
      const int kb1 = min(kb_total, kb0 + kb_per);
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!mbar_wait_warp(&empty_bar[stage], phase ^ 1, abort_flag)) {
          *abort_flag = ST_TIMEOUT_EMPTY;
          if (lead) atomicCAS(g.status, 0, ST_TIMEOUT_EMPTY);
          ok = false;
          break;
        }
        const bool b_done = prefetched > 0;       // this stage's B tiles and byte count are already out
        if (b_done) --prefetched;
        else mbar_expect_tx(&full_bar[stage], STAGE_BYTES, lead);
#pragma unroll
        for (int j = 0; j < KSUB; ++j) {
          uint8_t* sa = smem + stage * STAGE_BYTES + j * SUB_BYTES;
          const int k0 = kb * BKS + j * BK;
          if constexpr (!A_MN) {
            tma_load_2d(sa, &tmA, &full_bar[stage], k0, m0, lead);
          } else {
#pragma unroll
            for (int i = 0; i < TM / 64; ++i)
              tma_load_2d(sa + i * (BK * 128), &tmA, &full_bar[stage], m0 + i * 64, k0, lead);
          }
          if (!b_done) load_b(sa + A_BYTES, &full_bar[stage], k0, n0);
        }
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
      }
    }
  } else if (warp == 1) {
    // --------------------------------------------------------- MMA issuer
    const uint32_t lead = elect_one();
    constexpr uint32_t idesc = make_idesc_bf16(TM, BN, A_MN ? 1 : 0, B_MN ? 1 : 0);
    constexpr uint32_t A_LBO = A_MN ? BK * 128 : 16;
    constexpr uint32_t B_LBO = B_MN ? BK * 128 : 16;
    constexpr uint32_t A_KADV = A_MN ? UMMA_K * 128 : UMMA_K * 2;  // bytes per UMMA_K step
    constexpr uint32_t B_KADV = B_HALF_PANEL ? UMMA_K * 64 : B_MN ? UMMA_K * 128 : UMMA_K * 2;
    int stage = 0;
    uint32_t phase = 0;
    uint32_t acc_phase = 0;             // bit ab: phase of accumulator ab
    int it = 0;
    bool ok = true;
    for (int u = blockIdx.x; u < num_units && ok; u += gridDim.x, ++it) {
      const int ks = u / num_tiles;
      const int kb0 = ks * kb_per;
      const int kb1 = min(kb_total, kb0 + kb_per);
      if (kb0 >= kb1) continue;
      const int ab = it & 1;
      if (!mbar_wait_warp(&tempty_bar[ab], ((acc_phase >> ab) & 1) ^ 1, abort_flag)) {
        *abort_flag = ST_TIMEOUT_TMEM_EMPTY;
        if (lead) atomicCAS(g.status, 0, ST_TIMEOUT_TMEM_EMPTY);
        break;
      }
      tc_fence_after();
      const uint32_t d_tmem = tmem_base + ab * BN;
      for (int kb = kb0; kb < kb1; ++kb) {
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
        for (int k = 0; k < BKS / UMMA_K; ++k) {
          const int sub = k / (BK / UMMA_K) * SUB_BYTES, kk = k % (BK / UMMA_K);
          const uint64_t adesc = make_sdesc_sw128(sa, sub + kk * A_KADV, A_LBO, 1024);
          const uint64_t bdesc = B_HALF_PANEL ? make_sdesc<4>(sb, sub + kk * B_KADV, B_LBO, 512)
                                              : make_sdesc_sw128(sb, sub + kk * B_KADV, B_LBO, 1024);
          umma_bf16(d_tmem, adesc, bdesc, idesc, (kb > kb0 || k > 0) ? 1u : 0u, lead);
        }
        umma_commit(&empty_bar[stage], lead);  // frees the smem stage once these MMAs retire
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
      }
      if (!ok) break;
      umma_commit(&tfull_bar[ab], lead);  // accumulator complete -> epilogue
      acc_phase ^= 1u << ab;
    }
  } else {
    // ----------------------------------------------------------- epilogue
    const int e = warp - 2;
    const int quad = warp & 3;           // TMEM lane quarter this warp may read
    const int part = e >> 2;             // which quarter of the BN columns
    constexpr int COLS_PER_WARP = BN > 64 ? BN / 4 : 16;      // with 32 columns half of the warps have none
    constexpr int ROWS = TM / 4;         // of the tile in a TMEM lane quarter, from its first lane on
    uint8_t* my_stage = stage_out + e * 2048;
    uint32_t acc_phase = 0;             // bit ab: phase of accumulator ab
    int it = 0;
    for (int u = blockIdx.x; u < num_units; u += gridDim.x, ++it) {
      const int ks = u / num_tiles;
      const int tile = u % num_tiles;
      const int kb0 = ks * kb_per;
      const int kb1 = min(kb_total, kb0 + kb_per);
      if (kb0 >= kb1) continue;
      const int ab = it & 1;
      const int m0w = (tile / n_tiles) * TM + quad * ROWS, m = m0w + lane;   // first row of this warp's block
      const int nbase = (tile % n_tiles) * BN + part * COLS_PER_WARP;
      if (!mbar_wait_warp(&tfull_bar[ab], (acc_phase >> ab) & 1, abort_flag)) {
        *abort_flag = ST_TIMEOUT_TMEM_FULL;
        atomicCAS(g.status, 0, ST_TIMEOUT_TMEM_FULL);
        break;
      }
      acc_phase ^= 1u << ab;
      tc_fence_after();
      const uint32_t taddr =
          tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + ab * BN + part * COLS_PER_WARP;
      const bool row_ok = lane < ROWS && m < Meff;
      if (part * COLS_PER_WARP < BN)
        epilogue_drain<COLS_PER_WARP>(g, tmOut, tmAux, taddr, m, m0w, nbase, row_ok, my_stage, lane, ks == 0);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tempty_bar[ab]);
    }
    if (lane == 0) tma_store_wait<0>();   // all of this warp's bulk stores have landed
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

// ------------------------------------------------------------------------------------------
// CTA-pair variant: a cluster of two CTAs computes a 256 x 256 output tile with
// tcgen05.mma.cta_group::2 (instruction shape 256 x 256 x 16).  CTA r of the pair stages rows
// [r*128, r*128+128) of the A tile and columns [r*128, r*128+128) of the B tile in its own shared
// memory (32 KB per stage instead of 48 KB, so the ring is five stages deep and each B byte is
// fetched by one SM instead of two) and owns accumulator rows [r*128, r*128+128) in its own TMEM.
// Only the leader (rank 0) issues MMAs.  Barrier protocol:
//   full[s]    leader only, 1 arrival (leader producer's expect_tx) + the bytes of both CTAs' loads
//   empty[s]   one per CTA, 1 arrival: the leader commits to its own and to the partner's
//   tfull[b]   one per CTA, 1 arrival: committed by the leader to both
//   tempty[b]  leader only, 2 x NUM_EPI_WARPS arrivals: the epilogue warps of both CTAs
// Loads are plain unicast TMA loads whose completion is counted on the leader's barrier.

// An accumulation (EPI_ACCUM) hands its accumulator over every few 64-wide steps (GemmArgs::accum_steps), and the
// epilogue warps add these up in registers.  The tensor core cuts its sums off after every 16 products instead of
// rounding them, so the error of a chain grows with its length: 1024 x 4096 outputs over 32768 rows, 2-norm
// against 64 bits, one chain 3.8e-5, of 64 steps 4.4e-6, of 32 2.1e-6, of 16 1.0e-6, of 8 4.8e-7.  It costs 0.5 % of the
// time every 32 steps and 2.5 % every 8, and is never longer than a part of `k_splits` equal ones.
constexpr int ACCUM_STEPS = 32;

template <bool A_MN, bool B_MN, int EPI>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(NUM_THREADS, 1)
gemm_bf16_tcgen05_pair_kernel(const __grid_constant__ CUtensorMap tmA,
                              const __grid_constant__ CUtensorMap tmB,
                              const __grid_constant__ CUtensorMap tmOut,
                              const __grid_constant__ CUtensorMap tmAux, const GemmArgs g) {
  constexpr int STAGES = PAIR_STAGES;
  constexpr int BN = PAIR_BN;
  constexpr int HALF_N = BN / 2;
  constexpr int A_BYTES = BM * BK * 2;
  constexpr int B_BYTES = HALF_N * BK * 2;
  constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  constexpr int TMEM_COLS = 2 * BN;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* stage_out = smem + STAGES * STAGE_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(stage_out + NUM_EPI_WARPS * PAIR_WARP_STAGING);
  uint64_t* full_bar = bars;
  uint64_t* empty_bar = bars + STAGES;
  uint64_t* tfull_bar = bars + 2 * STAGES;
  uint64_t* tempty_bar = bars + 2 * STAGES + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  uint64_t* aux_bar = bars + 2 * STAGES + 5;      // one per epilogue warp: its staged aux tile
  static_assert((2 * STAGES + 5 + NUM_EPI_WARPS) * 8 <= 256, "barrier block outgrew its 256 bytes");

  const int warp = warp_number();
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const bool leader = rank == 0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&tfull_bar[i], 1);
      mbar_init(&tempty_bar[i], 2 * NUM_EPI_WARPS);
    }
    for (int i = 0; i < NUM_EPI_WARPS; ++i) mbar_init(&aux_bar[i], 1);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
    tma_prefetch_desc(&tmOut);
    if (g.ep.act == 1 || g.aux_tma) tma_prefetch_desc(&tmAux);
  }
  if (warp == 1) {
    tmem_alloc_pair(tmem_slot, TMEM_COLS);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();     // both CTAs' barriers are initialised before either signals the other
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  // link of a programmatic chain (captured training step): the set-up above may have run while the
  // kernel before this one was draining; loads, the epilogue's reads and all stores come after
  if (threadIdx.x == 0) griddep_launch_dependents();
  griddep_wait();

  const int m_tiles = (g.M + 2 * BM - 1) / (2 * BM);
  const int n_tiles = (g.N + BN - 1) / BN;
  const int kb_total = (g.K + BK - 1) / BK;
  const int kb_per = (kb_total + g.k_splits - 1) / g.k_splits;
  const int num_tiles = m_tiles * n_tiles;
  const int num_units = num_tiles * g.k_splits;
  const int pair_id = blockIdx.x >> 1;
  const int num_pairs = gridDim.x >> 1;
  // i-th work unit of this pair, for accumulations: steps [kb0, kb1) of an output tile
  auto accum_unit = [&](int i, int& tile, int& kb0, int& kb1) {
    if (g.even.on) return even_unit(g.even, kb_total, pair_id, i, tile, kb0, kb1);
    const int u = pair_id + i * num_pairs, ks = u / num_tiles;
    tile = u - ks * num_tiles;
    kb0 = ks * kb_per;
    kb1 = min(kb_total, kb0 + kb_per);
    return u < num_units;
  };

  if (warp == 0) {
    // ------------------------------------------------------- TMA producer (both CTAs)
    const uint32_t lead = elect_one();
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    auto load_unit = [&](int tile, int kb0, int kb1) {
      const int m0 = (tile / n_tiles) * (2 * BM) + rank * BM;
      const int n0 = (tile % n_tiles) * BN + rank * HALF_N;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!mbar_wait_warp(&empty_bar[stage], phase ^ 1, abort_flag)) {
          *abort_flag = ST_TIMEOUT_EMPTY;
          if (lead) atomicCAS(g.status, 0, ST_TIMEOUT_EMPTY);
          ok = false;
          break;
        }
        uint8_t* sa = smem + stage * STAGE_BYTES;
        uint8_t* sb = sa + A_BYTES;
        const uint32_t fb = mapa_shared(smem_u32(&full_bar[stage]), 0);
        if (leader) mbar_expect_tx(&full_bar[stage], 2 * STAGE_BYTES, lead);
        const int k0 = kb * BK;
        if constexpr (!A_MN) {
          tma_load_2d_pair(sa, &tmA, fb, k0, m0, lead);
        } else {
#pragma unroll
          for (int i = 0; i < BM / 64; ++i)
            tma_load_2d_pair(sa + i * (BK * 128), &tmA, fb, m0 + i * 64, k0, lead);
        }
        if constexpr (!B_MN) {
          tma_load_2d_pair(sb, &tmB, fb, k0, n0, lead);
        } else {
#pragma unroll
          for (int i = 0; i < HALF_N / 64; ++i)
            tma_load_2d_pair(sb + i * (BK * 128), &tmB, fb, n0 + i * 64, k0, lead);
        }
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
      }
    };
    if constexpr (EPI == EPI_ACCUM) {
      int tile, kb0, kb1;
      for (int i = 0; ok && accum_unit(i, tile, kb0, kb1); ++i) load_unit(tile, kb0, kb1);
    } else {
      for (int u = pair_id; u < num_units && ok; u += num_pairs) {
        const int ks = u / num_tiles, kb0 = ks * kb_per;
        load_unit(u % num_tiles, kb0, min(kb_total, kb0 + kb_per));
      }
    }
  } else if (warp == 1) {
    // --------------------------------------------------------- MMA issuer (leader only)
    if (leader) {
      const uint32_t lead = elect_one();
      constexpr uint32_t idesc = make_idesc_bf16(2 * BM, BN, A_MN ? 1 : 0, B_MN ? 1 : 0);
      constexpr uint32_t A_LBO = A_MN ? BK * 128 : 16;
      constexpr uint32_t B_LBO = B_MN ? BK * 128 : 16;
      constexpr uint32_t A_KADV = A_MN ? UMMA_K * 128 : UMMA_K * 2;
      constexpr uint32_t B_KADV = B_MN ? UMMA_K * 128 : UMMA_K * 2;
      int stage = 0;
      uint32_t phase = 0;
      uint32_t n_acc = 0;                 // accumulators handed over, the two in turn
      auto accumulate = [&](int kb0, int kb1) {
        const int ab = n_acc & 1;
        if (!mbar_wait_warp(&tempty_bar[ab], ((n_acc >> 1) & 1) ^ 1, abort_flag)) {
          *abort_flag = ST_TIMEOUT_TMEM_EMPTY;
          if (lead) atomicCAS(g.status, 0, ST_TIMEOUT_TMEM_EMPTY);
          return false;
        }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + ab * BN;
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait_warp(&full_bar[stage], phase, abort_flag)) {
            *abort_flag = ST_TIMEOUT_FULL;
            if (lead) atomicCAS(g.status, 0, ST_TIMEOUT_FULL);
            return false;
          }
          tc_fence_after();
          const uint32_t sa = smem_u32(smem + stage * STAGE_BYTES);
          const uint32_t sb = sa + A_BYTES;
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k) {
            const uint64_t adesc = make_sdesc_sw128(sa, k * A_KADV, A_LBO, 1024);
            const uint64_t bdesc = make_sdesc_sw128(sb, k * B_KADV, B_LBO, 1024);
            umma_bf16_pair(d_tmem, adesc, bdesc, idesc, (kb > kb0 || k > 0) ? 1u : 0u, lead);
          }
          const uint32_t eb = smem_u32(&empty_bar[stage]);
          umma_commit_pair(mapa_shared(eb, 0), lead);   // frees this stage in both CTAs
          umma_commit_pair(mapa_shared(eb, 1), lead);
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
        const uint32_t tb = smem_u32(&tfull_bar[ab]);
        umma_commit_pair(mapa_shared(tb, 0), lead);     // accumulator complete -> both epilogues
        umma_commit_pair(mapa_shared(tb, 1), lead);
        ++n_acc;
        return true;
      };
      bool ok = true;
      if constexpr (EPI == EPI_ACCUM) {
        int tile, kb0, kb1;
        for (int i = 0; ok && accum_unit(i, tile, kb0, kb1); ++i)
          for (; ok && kb0 < kb1; kb0 += g.accum_steps) ok = accumulate(kb0, min(kb1, kb0 + g.accum_steps));
      } else {
        for (int u = pair_id; u < num_units && ok; u += num_pairs) {
          const int kb0 = u / num_tiles * kb_per, kb1 = min(kb_total, kb0 + kb_per);
          if (kb0 < kb1) ok = accumulate(kb0, kb1);
        }
      }
    }
  } else {
    // ----------------------------------------------------------- epilogue (both CTAs)
    const int e = warp - 2;
    const int quad = warp & 3;
    const int part = e >> 2;
    constexpr int COLS_PER_WARP = BN / 4;
    uint8_t* my_stage = stage_out + e * PAIR_WARP_STAGING;
    uint32_t n_acc = 0;                 // accumulators taken over, the two in turn
    // GELU backward (aux_tma == 1): the warp's 32 x 64 tile of aux values is fetched by TMA into its
    // staging tile one unit ahead (right after the store of the unit before has read the tile), so
    // the loads that the epilogue math depends on are in flight while the accumulator is still
    // being computed instead of being issued, row by row, once it is ready.  Residual outputs
    // (aux_tma == 2) do the same with 32 x 32 fp32 tiles: the second of a unit's two tiles follows
    // when the first has left, the next unit's first one unit ahead.
    static_assert(COLS_PER_WARP == 64, "the staged aux tile is one 64-column store group");
    const bool stage_aux = EPI == EPI_RESID || EPI == EPI_MUL || EPI == EPI_DOT || (EPI == EPI_ANY && g.aux_tma != 0);
    uint32_t aux_phase = 0;
    if constexpr (EPI == EPI_ACCUM) {
      int tile, kb0, kb1;
      bool ok = true;
      for (int i = 0; ok && accum_unit(i, tile, kb0, kb1); ++i) {
        if (kb0 >= kb1) continue;
        const int m0w = (tile / n_tiles) * (2 * BM) + rank * BM + quad * 32;
        const int nbase = (tile % n_tiles) * BN + part * COLS_PER_WARP;
        const bool live = m0w < g.M && nbase < g.N;
        uint64_t sum[COLS_PER_WARP / 2];
#pragma unroll
        for (int c = 0; c < COLS_PER_WARP / 2; ++c) sum[c] = 0;
        for (; kb0 < kb1; kb0 += g.accum_steps) {
          const int ab = n_acc & 1;
          if (!mbar_wait_warp(&tfull_bar[ab], (n_acc >> 1) & 1, abort_flag)) {
            *abort_flag = ST_TIMEOUT_TMEM_FULL;
            atomicCAS(g.status, 0, ST_TIMEOUT_TMEM_FULL);
            ok = false;
            break;
          }
          ++n_acc;
          tc_fence_after();
          if (live) {
#pragma unroll
            for (int c = 0; c < COLS_PER_WARP / 16; ++c) {
              uint32_t r[16];
              tmem_ld16(tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + ab * BN + part * COLS_PER_WARP + c * 16, r);
              tmem_ld_wait();
#pragma unroll
              for (int k = 0; k < 8; ++k)
                sum[c * 8 + k] = f2_add(sum[c * 8 + k], f2_pack(__uint_as_float(r[2 * k]), __uint_as_float(r[2 * k + 1])));
            }
          }
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster(mapa_shared(smem_u32(&tempty_bar[ab]), 0));
        }
        if (ok && live) epilogue_add_sums(tmOut, sum, nbase, m0w, g.N, my_stage, lane);
      }
    } else {
      auto fetch_aux = [&](int u, int grp) {          // lane 0; the staging tile must be free
        if (u >= num_units) return;
        const int tile = u % num_tiles;
        const int m0w = (tile / n_tiles) * (2 * BM) + rank * BM + quad * 32;
        const int n = (tile % n_tiles) * BN + part * COLS_PER_WARP + grp * 32;
        if (m0w >= g.M || n >= g.N) return;           // the same test skips the drain below
        mbar_expect_tx(&aux_bar[e], 32 * 128);
        tma_load_2d(my_stage, &tmAux, &aux_bar[e], n, m0w);
      };
      if (stage_aux && lane == 0) fetch_aux(pair_id, 0);
      for (int u = pair_id; u < num_units; u += num_pairs) {
        const int ks = u / num_tiles;
        const int tile = u % num_tiles;
        const int kb0 = ks * kb_per;
        const int kb1 = min(kb_total, kb0 + kb_per);
        if (kb0 >= kb1) continue;
        const int ab = n_acc & 1;
        const int m0w = (tile / n_tiles) * (2 * BM) + rank * BM + quad * 32;
        const int m = m0w + lane;
        const int nbase = (tile % n_tiles) * BN + part * COLS_PER_WARP;
        const bool staged = stage_aux && m0w < g.M && nbase < g.N;
        if (!mbar_wait_warp(&tfull_bar[ab], (n_acc >> 1) & 1, abort_flag)) {
          *abort_flag = ST_TIMEOUT_TMEM_FULL;
          atomicCAS(g.status, 0, ST_TIMEOUT_TMEM_FULL);
          if (staged) mbar_wait_landed(&aux_bar[e], aux_phase);     // before the warp leaves
          break;
        }
        ++n_acc;
        tc_fence_after();
        const uint32_t taddr =
            tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + ab * BN + part * COLS_PER_WARP;
        auto wait_aux = [&]() {
          if (!mbar_wait_warp(&aux_bar[e], aux_phase, abort_flag)) {
            *abort_flag = ST_TIMEOUT_FULL;
            atomicCAS(g.status, 0, ST_TIMEOUT_FULL);
            mbar_wait_landed(&aux_bar[e], aux_phase);
            return false;
          }
          aux_phase ^= 1;
          return true;
        };
        // a warp whose 32 rows lie entirely past M has nothing to store (its accumulator rows came
        // from zero-filled loads); it still hands the buffer back
        if constexpr (EPI == EPI_ANY) {
          if (staged && !wait_aux()) break;
          if (m0w < g.M)
            epilogue_drain_wide<COLS_PER_WARP>(g, tmOut, tmAux, taddr, m, m0w, nbase, m < g.M, my_stage, lane,
                                               ks == 0, 0, staged);
        } else {
          // past the last staged tile of this unit: the first one of the next
          auto next_tile = [&](int grp) {
            if (EPI == EPI_RESID && grp == 0 && nbase + 32 < g.N) fetch_aux(u, 1);
            else fetch_aux(u + num_pairs, 0);
          };
          if (m0w < g.M && nbase < g.N) {
            if (!epilogue_drain_kind<EPI>(g, tmOut, tmAux, taddr, m, m0w, nbase, my_stage, lane, wait_aux, next_tile))
              break;
          } else if ((EPI == EPI_RESID || EPI == EPI_MUL || EPI == EPI_DOT) && lane == 0) {
            fetch_aux(u + num_pairs, 0);
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(mapa_shared(smem_u32(&tempty_bar[ab]), 0));
        if (EPI == EPI_ANY && stage_aux && lane == 0) {
          tma_store_wait_read<0>();           // the store just issued has read the staging tile
          fetch_aux(u + num_pairs, 0);
        }
      }
    }
    if (lane == 0) tma_store_wait<0>();
  }

  tc_fence_before();
  __syncthreads();
  cluster_sync_all();     // nobody signals the partner's barriers or reads TMEM after this point
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, TMEM_COLS);
  }
}

// What an epilogue warp of the pair kernel fetches by TMA (GemmArgs::aux_tma)
static int pair_aux_tma(const AbGemmEpilogue& ep, int k_splits) {
  if (ep.act == 1 || ep.accumulate || k_splits != 1) return 0;
  // aux tiles travel in the geometry of the output tiles (see the kernel)
  if ((ep.act == 2 || ep.act == 4) && !ep.out_fp32)
    return (reinterpret_cast<uintptr_t>(ep.aux) & 15) == 0 && (ep.ldaux * 2) % 16 == 0 ? 1 : 0;
  // residual tiles likewise, in the geometry of the fp32 output tiles
  if (ep.resid && ep.out_fp32 && ep.act == 0)
    return (reinterpret_cast<uintptr_t>(ep.resid) & 15) == 0 && (ep.ldr & 3) == 0 ? 2 : 0;
  return 0;
}

// The specialised drain that an epilogue takes where it is compiled.  Forward layers: [in][out] weights;
// input gradients: the same weights read K-major; weight gradients: both operands MN-major.
static EpiKind pair_kind(bool a_mn, bool b_mn, const GemmArgs& g) {
  const EpiKind kind = epi_kind(g);
  switch (kind) {
    case EPI_BF16: return !a_mn ? kind : EPI_ANY;
    case EPI_GELU: case EPI_GELU_GRAD: case EPI_RESID: return !a_mn && b_mn ? kind : EPI_ANY;
    case EPI_MUL: case EPI_DOT: return !a_mn && !b_mn ? kind : EPI_ANY;
    case EPI_ACCUM: return a_mn && b_mn ? kind : EPI_ANY;
    default: return EPI_ANY;
  }
}

// Cuts an accumulation into work units for `max_pairs` CTA pairs: either every tile into `splits` equal parts
// (`on` = 0), or equal shares of it all.  A unit ends with a pass over its tile that adds 256 KB of fp32 in L2; it runs
// under the next unit's main loop, which has to be EVEN_COVER steps long for that, and the last one under
// none.  The cheapest way by that count is taken, a number of equal parts where it is level with the shares (its CTAs
// read the same rows of the operands at the same time).  us, the equal parts taken before (balanced within 2 %,
// whatever their length) and now, at 16384 rows: 1280 x 3840 181 and 112, 1280 x 1280 69 and 44, 1280 x 5120 166 and 156;
// at 32768: 1024 x 4096 206 and 194, 1024 x 1024 67 and 56, 2048 x 1024 109 and 100; 1024 x 3072 (three equal parts
// either way) 148, and at 12136 rows 768 x 3072 45 and 46, 768 x 768 22.
constexpr int EVEN_MIN_STEPS = 8;      // of a part
constexpr int EVEN_COVER = 16;
constexpr int EVEN_UNIT = 2;           // steps that any unit costs beside its own
static EvenShare even_share(int tiles, int steps, int max_pairs, int* splits) {
  auto unit_cost = [](long long n) { return (n > EVEN_COVER ? n : EVEN_COVER) + EVEN_UNIT; };
  if (max_pairs < 1) max_pairs = 1;
  const int most = steps / EVEN_MIN_STEPS > 1 ? steps / EVEN_MIN_STEPS : 1;
  long long best = 0;
  for (int s = 1; s <= most && s <= 32; ++s) {
    const long long rounds = (static_cast<long long>(tiles) * s + max_pairs - 1) / max_pairs;
    const long long len = (steps + s - 1) / s, cost = (rounds - 1) * unit_cost(len) + len + EVEN_UNIT;
    if (s == 1 || cost < best) { best = cost; *splits = s; }
  }
  EvenShare b = {};
  b.pairs = max_pairs;
  b.waves = tiles / max_pairs;
  b.rest = tiles % max_pairs;
  if (b.rest == 0) return b;
  const long long before = b.waves * unit_cost(steps);
  auto take = [&](int q, int r, int extra_q, long long cost) {
    if ((before + cost) * 65 >= best * 64) return;
    best = before + cost;
    b.on = 1; b.q = q; b.r = r; b.extra_q = extra_q;
  };
  b.slices = max_pairs / b.rest < most ? max_pairs / b.rest : most;
  take((steps + b.slices - 1) / b.slices, 0, 0, (steps + b.slices - 1) / b.slices + EVEN_UNIT);
  const int extra = max_pairs - b.slices * b.rest;
  if (extra == 0) return b;
  // a longer main part leaves the other pairs less to do, and these have more and shorter units
  const int q0 = static_cast<int>((static_cast<long long>(b.rest) * steps + max_pairs - 1) / max_pairs);
  const int q1 = (steps + b.slices - 1) / b.slices, by = steps / 128 > 1 ? steps / 128 : 1;
  for (int q = q0; q < q1; q += by) {
    const int r = steps - b.slices * q;
    if (r < EVEN_MIN_STEPS) break;
    const int xq = (b.rest * r + extra - 1) / extra, whole = xq / r, part = xq % r;
    // part of a tile lies across two more often than not
    long long cost = part ? whole * unit_cost(r) + part + unit_cost(0) : (whole - 1) * unit_cost(r) + r + EVEN_UNIT;
    if (q + EVEN_UNIT > cost) cost = q + EVEN_UNIT;
    take(q, r, xq, cost);
  }
  return b;
}

template <bool A_MN, bool B_MN>
static int launch_pair(const void* A, long long lda, const void* B, long long ldb, const GemmArgs& g,
                       int max_ctas, cudaStream_t stream) {
  constexpr int HALF_N = PAIR_BN / 2;
  CUtensorMap tmA, tmB;
  int rc;
  if (!A_MN) rc = make_tmap_2d(&tmA, A, g.M, g.K, lda, BM, BK, 2, true);
  else       rc = make_tmap_2d(&tmA, A, g.K, g.M, lda, BK, 64, 2, true);
  if (rc) return rc;
  if (!B_MN) rc = make_tmap_2d(&tmB, B, g.N, g.K, ldb, HALF_N, BK, 2, true);
  else       rc = make_tmap_2d(&tmB, B, g.K, g.N, ldb, BK, 64, 2, true);
  if (rc) return rc;
  CUtensorMap tmOut, tmAux;
  const AbGemmEpilogue& ep = g.ep;
  // store boxes of 32 rows with 128-byte rows (64-byte rows when two bf16 outputs share the tile)
  if (ep.out_fp32)       rc = make_tmap_2d_sw(&tmOut, ep.out, g.M, g.N, ep.ldo, 32, 32, 4, 128);
  else if (ep.act == 1)  rc = make_tmap_2d_sw(&tmOut, ep.out, g.M, g.N, ep.ldo, 32, 32, 2, 64);
  else                   rc = make_tmap_2d_sw(&tmOut, ep.out, g.M, g.N, ep.ldo, 32, 64, 2, 128);
  if (rc) return rc;
  GemmArgs ga = g;
  ga.aux_tma = pair_aux_tma(ep, g.k_splits);
  if (ep.act == 1)            rc = make_tmap_2d_sw(&tmAux, ep.aux, g.M, g.N, ep.ldaux, 32, 32, 2, 64);
  else if (ga.aux_tma == 1)   rc = make_tmap_2d_sw(&tmAux, ep.aux, g.M, g.N, ep.ldaux, 32, 64, 2, 128);
  else if (ga.aux_tma == 2)   rc = make_tmap_2d_sw(&tmAux, ep.resid, g.M, g.N, ep.ldr, 32, 32, 4, 128);
  else                        tmAux = tmOut;
  if (rc) return rc;
  constexpr int SMEM = 1024 + PAIR_STAGES * (BM * BK * 2 + HALF_N * BK * 2) +
                       NUM_EPI_WARPS * PAIR_WARP_STAGING + 256;
  const int m_tiles = (g.M + 2 * BM - 1) / (2 * BM), n_tiles = (g.N + PAIR_BN - 1) / PAIR_BN;
  const int steps = (g.K + BK - 1) / BK;
  ga.accum_steps = (steps + g.k_splits - 1) / g.k_splits;
  if (ga.accum_steps > ACCUM_STEPS) ga.accum_steps = ACCUM_STEPS;
  ga.even.on = 0;
  if (ep.even_k && pair_kind(A_MN, B_MN, ga) == EPI_ACCUM)
    ga.even = even_share(m_tiles * n_tiles, steps, max_ctas / 2, &ga.k_splits);
  const int units = m_tiles * n_tiles * ga.k_splits;
  int pairs = max_ctas / 2;
  if (pairs > units && !ga.even.on) pairs = units;
  if (pairs < 1) pairs = 1;
  auto go = [&](auto kern, PerDeviceOnce& attr_set) {
    if (attr_set.first_use_on_device()) {
      cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
      if (e != cudaSuccess) return static_cast<int>(e);
      attr_set.mark_device();
    }
    launch_chained(kern, dim3(2 * pairs), dim3(NUM_THREADS), SMEM, stream, tmA, tmB, tmOut, tmAux, ga);
    return static_cast<int>(cudaGetLastError());
  };
  static PerDeviceOnce attr[EPI_DOT + 1];      // one per kernel of this operand layout
  const EpiKind kind = pair_kind(A_MN, B_MN, ga);
  if constexpr (!A_MN) {
    if (kind == EPI_BF16) return go(gemm_bf16_tcgen05_pair_kernel<A_MN, B_MN, EPI_BF16>, attr[EPI_BF16]);
  }
  if constexpr (!A_MN && B_MN) {
    if (kind == EPI_GELU) return go(gemm_bf16_tcgen05_pair_kernel<A_MN, B_MN, EPI_GELU>, attr[EPI_GELU]);
    if (kind == EPI_GELU_GRAD) return go(gemm_bf16_tcgen05_pair_kernel<A_MN, B_MN, EPI_GELU_GRAD>, attr[EPI_GELU_GRAD]);
    if (kind == EPI_RESID) return go(gemm_bf16_tcgen05_pair_kernel<A_MN, B_MN, EPI_RESID>, attr[EPI_RESID]);
  }
  if constexpr (!A_MN && !B_MN) {
    if (kind == EPI_MUL) return go(gemm_bf16_tcgen05_pair_kernel<A_MN, B_MN, EPI_MUL>, attr[EPI_MUL]);
    if (kind == EPI_DOT) return go(gemm_bf16_tcgen05_pair_kernel<A_MN, B_MN, EPI_DOT>, attr[EPI_DOT]);
  }
  if constexpr (A_MN && B_MN) {
    if (kind == EPI_ACCUM) return go(gemm_bf16_tcgen05_pair_kernel<A_MN, B_MN, EPI_ACCUM>, attr[EPI_ACCUM]);
  }
  if (ep.colsum) return -7;                      // only EPI_MUL adds column sums
  if (ga.aux_tma == 2) ga.aux_tma = 0;           // EPI_ANY reads the residual row by row
  return go(gemm_bf16_tcgen05_pair_kernel<A_MN, B_MN, EPI_ANY>, attr[EPI_ANY]);
}

template <int TM, int BN, int STAGES, int KSUB, bool A_MN, bool B_MN>
static int launch(const void* A, long long lda, const void* B, long long ldb, const GemmArgs& g,
                  int max_ctas, cudaStream_t stream) {
  CUtensorMap tmA, tmB;
  int rc;
  if (!A_MN) rc = make_tmap_2d(&tmA, A, g.M, g.K, lda, TM, BK, 2, true);
  else       rc = make_tmap_2d(&tmA, A, g.K, g.M, lda, BK, 64, 2, true);
  if (rc) return rc;
  if (!B_MN) rc = make_tmap_2d(&tmB, B, g.N, g.K, ldb, BN, BK, 2, true);
  else       rc = make_tmap_2d_sw(&tmB, B, g.K, g.N, ldb, BK, BN < 64 ? BN : 64, 2, BN < 64 ? 64 : 128);
  if (rc) return rc;
  // output / pre-activation maps for the epilogue's TMA stores: boxes of a warp's rows x 16 columns
  CUtensorMap tmOut, tmAux;
  const AbGemmEpilogue& ep = g.ep;
  if (ep.out_fp32) rc = make_tmap_2d_sw(&tmOut, ep.out, g.M, g.N, ep.ldo, TM / 4, 16, 4, 64);
  else             rc = make_tmap_2d_sw(&tmOut, ep.out, g.M, g.N, ep.ldo, TM / 4, 16, 2, 32);
  if (rc) return rc;
  if (ep.act == 1) {
    rc = make_tmap_2d_sw(&tmAux, ep.aux, g.M, g.N, ep.ldaux, TM / 4, 16, 2, 32);
    if (rc) return rc;
  } else {
    tmAux = tmOut;
  }
  constexpr int SMEM = 1024 + STAGES * KSUB * (TM * BK * 2 + BN * BK * 2) + NUM_EPI_WARPS * 2048 + 256;
  auto kern = gemm_bf16_tcgen05_kernel<TM, BN, STAGES, KSUB, A_MN, B_MN>;
  static PerDeviceOnce attr_set;
  if (attr_set.first_use_on_device()) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
    if (e != cudaSuccess) return static_cast<int>(e);
    attr_set.mark_device();
  }
  const int m_tiles = (g.M + TM - 1) / TM, n_tiles = (g.N + BN - 1) / BN;
  const int units = m_tiles * n_tiles * g.k_splits;
  int grid = units < max_ctas ? units : max_ctas;
  if (grid < 1) grid = 1;
  if (g.pdl) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(NUM_THREADS);
    cfg.dynamicSmemBytes = SMEM;
    cfg.stream = stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return static_cast<int>(cudaLaunchKernelEx(&cfg, kern, tmA, tmB, tmOut, tmAux, g));
  }
  launch_chained(kern, dim3(grid), dim3(NUM_THREADS), SMEM, stream, tmA, tmB, tmOut, tmAux, g);
  return static_cast<int>(cudaGetLastError());
}

}  // namespace ab

extern "C" int ab_colsum_bf16(const void* x, long long ld, int M, int N, float* out, const int* m_limit,
                              cudaStream_t stream);
extern "C" int ab_attn_delta(const void* o, const void* dout, float* delta, int B, int T, int H, int hd,
                             cudaStream_t stream);

namespace ab {

// Which kernel serves a problem, and whether column sums or head products come from passes of their own
struct GemmPlan {
  int kernel;                  // columns of the single-CTA kernel's tile (64, 128, 256), PLAN_64X32 or PLAN_PAIR
  bool dot_pass, colsum_pass;
};
constexpr int PLAN_PAIR = 512;
constexpr int PLAN_64X32 = 32;          // 64 rows

static GemmPlan gemm_plan(int a_mn, int b_mn, int M, int N, const AbGemmEpilogue& ep, int k_splits, int max_ctas) {
  // CTA pairs for the large shapes; the single-CTA kernel keeps the device-sized problems
  // (m_limit / k_limit) and anything a caller pins with AB_GEMM_NO_PAIR=1 in the environment
  static const bool no_pair = [] {
    const char* v = getenv("AB_GEMM_NO_PAIR");
    return v && v[0] == '1';
  }();
  bool pair = !no_pair && !ep.m_limit && !ep.k_limit && M >= 512 && N >= 256 && max_ctas >= 2;
  const bool aux_by_tma = pair && ep.aux && pair_aux_tma(ep, k_splits) == 1 && !a_mn && !b_mn && ep.alpha == 1.f && !ep.bias;
  const bool dot = ep.act == 4 && aux_by_tma;
  const bool sums = ep.colsum && aux_by_tma && ep.act == 2 && ep.aux_grad && !ep.resid;
  GemmPlan p = {0, ep.act == 4 && !dot, ep.colsum && !sums};
  // A problem that fits one wave of smaller tiles takes them: a 256 x 256 tile keeps two SMs for the whole
  // contraction and its epilogue while the others are idle.  128 x 64 tiles where they fit, else 128 x 128
  // (2048 x 256 x 256 with residual and dropout: 11.7 us on pairs, 9.4 with 128 x 128, 7.3 with 128 x 64;
  // 2048 x 1024 x 256: 11.9, 9.6, 9.8 in two waves; 4096 x 1024 x 1024, two waves: 16.3, 19.9, 27.7).
  // Over M 512 to 4096, N 256 to 4096, K 128 to 4096 with bias, GELU, residual or plain outputs, wherever the rule
  // holds: 0.64 to 0.77 of the pairs' time on average, 0.89 at most.
  auto tiles = [&](int bn) { return static_cast<long long>((M + 127) / 128) * ((N + bn - 1) / bn); };
  const bool one_wave = pair && !a_mn && !sums && !dot && k_splits == 1 && tiles(128) <= max_ctas;
  // narrow tiles also for skinny problems (decode steps with a few hundred rows): twice the CTAs
  const bool narrow = (N <= 128) || (M <= 256);
  // A few hundred rows against a wide weight matrix (decode steps): the time goes into streaming
  // the weights, so the columns are cut into 64-wide tiles to put twice as many SMs on them.  Not for a
  // contraction whose length is a device value: it ends with a whole stage, and here that is 128 columns instead of 64
  // that have to be zero past the limit.
  if (M <= 256 && N >= 1024 && !a_mn && !ep.k_limit) p.kernel = 64;
  else if (one_wave) p.kernel = tiles(64) <= max_ctas ? 64 : 128;
  else if (narrow)   p.kernel = 128;
  else               p.kernel = pair ? PLAN_PAIR : 256;
  // 64 x 32 tiles wherever they fit a wave: a step of the contraction takes 165 clocks (12 KB of operands) instead of
  // 320 (24 KB, and MMAs of 128 rows that take 67 clocks whatever their columns).  128 x 64 tiles leave three quarters of
  // the SMs idle there with more than 64 rows, and half of them and more with up to 64.  Per launch of a chain, us, with
  // 128 x 64 and with 64 x 32: 90 x 1024 x 4096 14.7 and 10.7, 90 x 1024 x 1024 with residual 6.5 and 5.4, 200 x 1024 x
  // 4096 15.0 and 11.2; 1 row x 2048 x 1024 6.2 and 5.3, x 3072 6.8 and 6.2, x 4096 7.5 and 6.7, x 4608 7.9 and 7.1;
  // 32 rows x 3072 x 1024 6.2 and 5.4, x 4096 7.0 and 6.0; 64 rows x 4096 x 1024 5.4 both, x 4608 5.6 both.  Whole
  // passes of up to 64 rows, never, only where a quarter of the SMs would have 128 x 64 tiles, and as it is: one game
  // of 20 tokens (24 layers of 1024) 1163, 1133 and 1058 us, of 768 columns 646, 656 and 638; 32 trees 6697, 6684 and
  // 6310, of 1280 columns 4265, 4220 and 3868.
  // Problems of one wave: 512 to 1100 rows x 256 to 576 columns x 64 to 4096, plain, GELU or residual, 0.72 to 0.98 of the time
  // with 128 x 64 (512 x 256 x 1024 with residual and dropout 8.3 and 6.5).
  // With 64 x 64 tiles as well where 64 x 32 are too many (90 x 3072 x 1024 5.9 and 5.6) neighbouring launches of a
  // pass no longer fit the SMs together, and their set-up waits: one game 1230 us as it was, 1250 so, 1180 without.
  if (p.kernel == 64 && k_splits == 1 && !ep.m_limit && !ep.k_limit &&
      static_cast<long long>((M + 63) / 64) * ((N + 31) / 32) <= max_ctas)
    p.kernel = PLAN_64X32;
  return p;
}

template <bool A_MN, bool B_MN>
static int launch_plan(int kernel, const void* A, long long lda, const void* B, long long ldb, const GemmArgs& g,
                       int max_ctas, cudaStream_t stream) {
  if (kernel == PLAN_PAIR) return launch_pair<A_MN, B_MN>(A, lda, B, ldb, g, max_ctas, stream);
  if (kernel == 256) return launch<128, 256, 4, 1, A_MN, B_MN>(A, lda, B, ldb, g, max_ctas, stream);
  if constexpr (!A_MN) {
    if (kernel == 64) return launch<128, 64, 4, 2, A_MN, B_MN>(A, lda, B, ldb, g, max_ctas, stream);
    if (kernel == PLAN_64X32) return launch<64, 32, 8, 2, A_MN, B_MN>(A, lda, B, ldb, g, max_ctas, stream);
  }
  return launch<128, 128, 6, 1, A_MN, B_MN>(A, lda, B, ldb, g, max_ctas, stream);
}

}  // namespace ab

extern "C" int ab_gemm_bf16(const void* A, int a_mn, long long lda, const void* B, int b_mn,
                            long long ldb, int M, int N, int K, const AbGemmEpilogue* ep,
                            int k_splits, int max_ctas, int* status, cudaStream_t stream) {
  using namespace ab;
  if (M <= 0 || N <= 0 || K <= 0 || (N & 7) || (lda & 7) || (ldb & 7) || !ep || !ep->out ||
      !status)
    return -1;
  if (k_splits < 1) k_splits = 1;
  if (k_splits > 1 && !(ep->out_fp32 && ep->accumulate)) return -2;
  if ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B) |
       reinterpret_cast<uintptr_t>(ep->out) | reinterpret_cast<uintptr_t>(ep->aux)) & 15)
    return -3;
  if ((ep->ldo * (ep->out_fp32 ? 4 : 2)) & 15) return -4;   // TMA row pitch: multiple of 16 bytes
  if (ep->act == 1 && (ep->ldaux & 7)) return -4;
  if (max_ctas <= 0) max_ctas = 148;
  if (ep->next_b && ((reinterpret_cast<uintptr_t>(ep->next_b) | ep->next_bytes) & 15)) return -3;
  const GemmPlan plan = gemm_plan(a_mn, b_mn, M, N, *ep, k_splits, max_ctas);
  if (ep->act == 4) {
    if (!ep->aux || !ep->dot_out || ep->dot_T < 1 || M % ep->dot_T || (N & 63) || ep->out_fp32 || ep->ldo != N ||
        ep->ldaux != N || ep->m_limit || ep->resid)
      return -5;
    if (plan.dot_pass) {
      AbGemmEpilogue plain = *ep;
      plain.act = 0;
      const int rc = ab_gemm_bf16(A, a_mn, lda, B, b_mn, ldb, M, N, K, &plain, k_splits, max_ctas, status, stream);
      if (rc) return rc;
      if (ep->passes) ++*ep->passes;
      return ab_attn_delta(ep->aux, ep->out, ep->dot_out, M / ep->dot_T, ep->dot_T, N / 64, 64, stream);
    }
  }
  if (plan.colsum_pass) {
    if (ep->out_fp32) return -6;
    AbGemmEpilogue plain = *ep;
    plain.colsum = nullptr;
    const int rc = ab_gemm_bf16(A, a_mn, lda, B, b_mn, ldb, M, N, K, &plain, k_splits, max_ctas, status, stream);
    if (rc) return rc;
    if (ep->passes) ++*ep->passes;
    return ab_colsum_bf16(ep->out, ep->ldo, M, N, ep->colsum, ep->m_limit, stream);
  }
  GemmArgs g;
  g.M = M; g.N = N; g.K = K; g.k_splits = k_splits; g.ep = *ep; g.status = status; g.salt = seed_salt_ptr(); g.aux_tma = 0;
  // programmatic dependent launch: single-CTA kernels only, never with device-side limits (those
  // are values of earlier kernels, read before any wait)
  g.pdl = (ep->pdl && !ep->m_limit && !ep->k_limit) ? 1 : 0;
  if (!a_mn && !b_mn) return launch_plan<false, false>(plan.kernel, A, lda, B, ldb, g, max_ctas, stream);
  if (!a_mn && b_mn) return launch_plan<false, true>(plan.kernel, A, lda, B, ldb, g, max_ctas, stream);
  if (a_mn && !b_mn) return launch_plan<true, false>(plan.kernel, A, lda, B, ldb, g, max_ctas, stream);
  return launch_plan<true, true>(plan.kernel, A, lda, B, ldb, g, max_ctas, stream);
}

// For tests: the units that `pairs` CTA pairs get of `tiles` output tiles of `steps` steps with even_k, four numbers
// each (pair, tile, first step, end).  Returns how many (no more than `room` are written), or minus the number of
// equal parts per tile.
extern "C" int ab_gemm_even_units(int tiles, int steps, int pairs, int* out, int room) {
  int splits = 1, n = 0, tile, kb0, kb1;
  const ab::EvenShare s = ab::even_share(tiles, steps, pairs, &splits);
  if (!s.on) return -splits;
  for (int p = 0; p < s.pairs; ++p)
    for (int i = 0; ab::even_unit(s, steps, p, i, tile, kb0, kb1); ++i, ++n)
      if (n < room) { out[4 * n] = p; out[4 * n + 1] = tile; out[4 * n + 2] = kb0; out[4 * n + 3] = kb1; }
  return n;
}

// What ab_gemm_bf16 would run for the same arguments, without running it: the columns of the single-CTA
// kernel's tile (32: of 64 rows, else of 128), or 512 + EpiKind on CTA pairs.  Passes beside the GEMM: see `passes`.
extern "C" int ab_gemm_route(const void*, int a_mn, long long, const void*, int b_mn, long long, int M, int N, int,
                             const AbGemmEpilogue* ep, int k_splits, int max_ctas, int*, cudaStream_t) {
  using namespace ab;
  if (k_splits < 1) k_splits = 1;
  if (max_ctas <= 0) max_ctas = 148;
  AbGemmEpilogue e = *ep;
  GemmPlan plan = gemm_plan(a_mn, b_mn, M, N, e, k_splits, max_ctas);
  if (plan.dot_pass) { e.act = 0; plan = gemm_plan(a_mn, b_mn, M, N, e, k_splits, max_ctas); }
  if (plan.colsum_pass) { e.colsum = nullptr; plan = gemm_plan(a_mn, b_mn, M, N, e, k_splits, max_ctas); }
  if (plan.kernel != PLAN_PAIR) return plan.kernel;
  GemmArgs g;
  g.ep = e;
  g.aux_tma = pair_aux_tma(e, k_splits);
  return PLAN_PAIR + pair_kind(a_mn, b_mn, g);
}
