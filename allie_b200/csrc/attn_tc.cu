// Causal flash attention on tcgen05 (forward; the backward kernels follow further down).
//
// An item is one 128-row query tile of one (batch, head); two CTAs share an SM.  In launches of many items CTAs stay: one
// that has asked for an item's tiles takes the place of a block of the grid that has not started
// (`grid_take_block`) and goes on with that one's item, so that loads run ahead of the items and blocks with short
// ones do more of them.  In launches of few, and in programmatic chains, a CTA does its own item and leaves (ONE;
// `fwd_takes_over` has the rule).  Per 128-row key/value tile:
//   warp 9              : S = Q K^T          -> TMEM (128 lanes = query rows, 128 fp32 columns)
//   warps 0-7           : two threads per query row, 64 keys each: S in registers, maximum (exchanged
//                         through shared memory), exponentials, dropout, P -> TMEM as packed bf16 (the A
//                         operand of the second product)
//   warp 9              : O += P V           -> TMEM
//   warp 8              : items; TMA loads of Q and of K/V tiles (through rings that go on from item to item)
// Q, K and V are read straight out of the packed [B*T, 3*d] QKV activation with 2-D TMA boxes
// (64 columns x 128 rows), and O is written in the [B*T, d] layout the projection GEMM reads.
// V is consumed MN-major (rows = keys), so no transposes exist anywhere.
//
// What bounds it: with dropout, instruction issue (the generator takes 45 of 150 us at 64 x 512 x 16 x 64) and how
// much of it the warps of an SM can overlap; without, latencies and then the exponential unit (16 per SM
// and clock).  So: sixteen math warps per SM (with one thread per row, eight, issue was 39 % busy), S
// is read once, P never passes through shared memory, O stays in TMEM and is rescaled there when the
// maximum of one of a warp's rows has grown, and unrolled code stays small (fetching instructions was
// a fifth of the stalls with 128 keys per thread).  Keeping the old scale until the maximum has grown
// by 2^8 saves little at these lengths and gives up that the largest probability of a row is exactly
// one: error against 64 bits 0.00195 instead of 0.00181.  The reciprocal of the keep probability is
// applied at the end.
// With a CTA per item (and blocks past the end of their sequence that only leave) an SM had 1.3 of its two CTAs at
// work and 4700 of a CTA's 7900 clocks over one key tile were set-up, first loads and the way out.  Cold L2, heads of
// 64, us, a CTA per item and now: 256 prompts of 4 to 300 tokens x 16 heads 192 and 111, 64 of them 58 and 41,
// 256 x 128 tokens 86 and 61, 64 x 512 x 16 117 and 97, with dropout (and with the generator's keys in uniform
// registers and its bits by carry) 176 and 150, 37 x 328 x 12 with dropout 57 and 51; heads of 128, 256 prompts x 8
// 121 and 90.  A tile takes 1650 clocks per SM, of which the exponential unit needs 1024.
#include <algorithm>

#include "attn_common.cuh"

namespace ab {

constexpr int FWD_MATH_WARPS = 8;
constexpr int FWD_TMA_WARP = FWD_MATH_WARPS;
constexpr int FWD_MMA_WARP = FWD_MATH_WARPS + 1;
constexpr int FWD_THREADS = (FWD_MATH_WARPS + 2) * 32;

template <int HD>
struct FwdCfg {
  static constexpr int PANELS = HD / 64;               // 64-column panels per Q/K/V tile
  static constexpr int TILE_BYTES = 128 * HD * 2;      // one Q / K / V tile
  // head_dim 64: S, P and O side by side in 256 TMEM columns, two K/V stages.  head_dim 128: P takes
  // the place of S (already in registers by then) and one K/V stage, so that two CTAs still fit an SM;
  // the partner's math covers what this CTA's tensor work waits for.
  static constexpr bool P_IN_S = HD == 128;
  static constexpr int STAGES = HD == 128 ? 1 : 2;       // of Q and of K / V
  static constexpr int TM_P = P_IN_S ? 0 : 128;
  static constexpr int TM_O = 256 - HD;
  static constexpr int SMEM = 3 * STAGES * TILE_BYTES + 512 + 2048;
};
constexpr int FWD_QUEUE = 4;             // items between the producer and the warps that work on them

// One query tile of one (sequence, head).  The producer hands them on through a ring in shared memory.
struct FwdItem {
  int qt, h, b;                          // qt < 0: no more
  int first, T;                          // the sequence's first activation row and length
};

// 16 AND-masks (one per packed bf16 pair) of 32 keep bits: the bit of each element is shifted into
// the sign of its byte and spread over a half-word by the byte permute's sign mode.
__device__ __forceinline__ void keep_masks16(uint32_t word, uint32_t* m) {
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const uint32_t x = word << (7 - 2 * q), y = word << (6 - 2 * q);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const uint32_t sel = (8u | k) * 0x11u | (8u | (4 + k)) * 0x1100u;
      asm("prmt.b32 %0, %1, %2, %3;" : "=r"(m[4 * k + q]) : "r"(x), "r"(y), "r"(sel));
    }
  }
}

// The caches that keys and values also go to.  A kernel of its own: as an option of the one without, its maps and code
// cost a pass over one short game 25 of 1180 us.
template <bool KV>
struct KvMaps {
  CUtensorMap k, v;
};
template <>
struct KvMaps<false> {};

// ONE: a block does its own item and leaves, without the ring of items, the hand-back of Q tiles and the end marker, which
// cost a launch of few items half a microsecond (us so and with them: 64 items of 128 keys 5.6 and 6.1, 108 of three
// key tiles 8.2 and 8.9).
template <int HD, bool KV, bool ONE>
__global__ void __launch_bounds__(FWD_THREADS, 2)
attn_fwd_kernel(const __grid_constant__ CUtensorMap tmQKV, const __grid_constant__ CUtensorMap tmO,
                const __grid_constant__ KvMaps<KV> cache, const AttnArgs a) {
  using C = FwdCfg<HD>;
  constexpr int PANELS = C::PANELS, TILE_BYTES = C::TILE_BYTES, STAGES = C::STAGES;
  constexpr uint32_t IDESC_S = make_idesc_bf16(128, 128, 0, 0);
  constexpr uint32_t IDESC_PV = make_idesc_bf16(128, HD, 0, 1);

  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = smem_raw;
  if (smem_u32(smem) & 1023) {  // swizzled tiles need a 1024-byte aligned base
    if (threadIdx.x == 0) atomicCAS(a.status, 0, ST_BAD_ARGUMENT);
    return;
  }
  uint8_t* sQ = smem;
  uint8_t* sK = sQ + STAGES * TILE_BYTES;
  uint8_t* sV = sK + STAGES * TILE_BYTES;
  uint8_t* tail = sV + STAGES * TILE_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(tail);
  uint64_t* q_full = bars;                  // STAGES (two reserved)
  uint64_t* q_empty = bars + 2;
  uint64_t* k_full = bars + 4;
  uint64_t* v_full = bars + 6;
  uint64_t* k_empty = bars + 8;
  uint64_t* v_empty = bars + 10;
  uint64_t* s_full = bars + 12;
  uint64_t* s_empty = bars + 13;
  uint64_t* p_full = bars + 14;
  uint64_t* pv_full = bars + 15;
  uint64_t* xchg = bars + 16;               // 4: the two warps of a TMEM lane quarter
  uint64_t* item_full = bars + 20;          // FWD_QUEUE
  uint64_t* item_empty = bars + 24;
  uint64_t* grid_bar = bars + 28;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 29);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  uint4* grid_next = reinterpret_cast<uint4*>(bars + 30);
  FwdItem* items = reinterpret_cast<FwdItem*>(bars + 32);
  static_assert(32 * 8 + FWD_QUEUE * sizeof(FwdItem) <= 512, "barriers and items outgrew their 512 bytes");
  float* s_row = reinterpret_cast<float*>(tail + 512);       // [2][2 halves][128] row values

  const int warp = warp_number(), lane = threadIdx.x & 31;
  const int d_model = a.H * HD;

  auto item_of = [&](uint3 block) {
    FwdItem it;
    it.qt = (a.T + AT_BM - 1) / AT_BM - 1 - static_cast<int>(block.x);       // heaviest tiles first
    it.h = block.y; it.b = block.z;
    // packed batch: sequence b owns rows [row0[b], row0[b + 1]) of the activation
    it.first = a.row0 ? __ldg(a.row0 + it.b) : it.b * a.T;
    it.T = a.row0 ? __ldg(a.row0 + it.b + 1) - it.first : a.T;
    return it;
  };
  // The set-up may run under the kernel before; the producer asks for the first item's rows as soon as that is done.
  FwdItem it = {};
  if (warp == FWD_TMA_WARP) {
    griddep_wait();
    it = item_of(make_uint3(blockIdx.x, blockIdx.y, blockIdx.z));
    if (ONE && lane == 0) {
      items[0] = it;
      if (it.qt * AT_BM >= it.T) items[0].qt = -1;
    }
  }
  if (warp == 0) {                           // a barrier per lane
    const uint64_t* bar = bars + lane;
    const uint32_t count = bar == s_empty || bar == p_full || (bar >= q_empty && bar < k_full) ? FWD_MATH_WARPS
                           : bar >= xchg && bar < item_full       ? 2
                           : bar >= item_empty && bar < grid_bar ? FWD_MATH_WARPS + 1 : 1;
    if (bar <= grid_bar) mbar_init(bars + lane, count);
    __syncwarp();
  }
  if (threadIdx.x == 0) {
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmQKV);
  }
  if (warp == FWD_MMA_WARP) { tmem_alloc(tmem_slot, 256); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  // only now: a dependent GEMM's CTA must not take the TMEM columns that this grid still has to allocate
  if (threadIdx.x == 0) griddep_launch_dependents();
  griddep_wait();                            // all else that is read or written comes after this
  const uint32_t tS = tmem_base, tP = tmem_base + C::TM_P, tO = tmem_base + C::TM_O;

  // n-th item of this CTA, for a whole warp (bounded; null when a wait ran out).  It stays until item_done.
  auto next_item = [&](int n) -> const volatile FwdItem* {
    if (ONE) return &items[0];
    return mbar_wait_warp(&item_full[n % FWD_QUEUE], (n / FWD_QUEUE) & 1, abort_flag) ? &items[n % FWD_QUEUE] : nullptr;
  };
  auto item_done = [&](int n) {
    if (ONE) return;
    __syncwarp();
    if (lane == 0) mbar_arrive(&item_empty[n % FWD_QUEUE]);
  };

  if (warp == FWD_TMA_WARP) {
    // ------------------------------------------------------------ TMA producer
    const uint32_t lead = elect_one();
    int g = 0, n = 0, nq = 0, nk = 0, nv = 0;    // key tiles, items; tiles asked for
    bool ok = true;
    // An item's last key tile is its own rows' keys and values: they go on to the cache from where they lie, before
    // the tile's place is loaded again.  32 rows per TMA store; the last rows of a sequence one by one, the
    // slots behind them belong to others.
    int keep = -1, keep_rows = 0;                // that tile (keep < 0: none), its rows in the sequence
    long long keep_slot = 0;                     // and the first one's row of the cache
    [[maybe_unused]] auto store_kept = [&]() {
      if constexpr (KV) {
        const int st = keep % STAGES, par = (keep / STAGES) & 1, whole = keep_rows & ~31;
        keep = -1;
        if (!mbar_wait_warp(&k_full[st], par, abort_flag) || !mbar_wait_warp(&v_full[st], par, abort_flag)) return false;
        const uint8_t* k = sK + st * TILE_BYTES;
        const uint8_t* v = sV + st * TILE_BYTES;
        if (lead) {
          for (int r = 0; r < whole; r += 32)
#pragma unroll
            for (int p = 0; p < PANELS; ++p) {
              tma_store_2d(&cache.k, k + p * 16384 + r * 128, p * 64, static_cast<int>(keep_slot) + r);
              tma_store_2d(&cache.v, v + p * 16384 + r * 128, p * 64, static_cast<int>(keep_slot) + r);
            }
          tma_store_commit();
        }
        for (int i = lane; i < (keep_rows - whole) * 8 * PANELS; i += 32) {
          const int r = whole + i / (8 * PANELS), c = i % (8 * PANELS);          // row, 16-byte chunk of it
          const uint32_t off = (c >> 3) * 16384 + sw128_chunk(r, c & 7);
          const long long dst = (keep_slot + r) * HD + c * 8;
          *reinterpret_cast<uint4*>(a.kc + dst) = *reinterpret_cast<const uint4*>(k + off);
          *reinterpret_cast<uint4*>(a.vc + dst) = *reinterpret_cast<const uint4*>(v + off);
        }
        if (lead) tma_store_wait_read<0>();
        __syncwarp();
      }
      return true;
    };
    auto push = [&](const FwdItem& it) {
      if (ONE) return true;
      const int s = n % FWD_QUEUE;
      if (!mbar_wait_warp(&item_empty[s], ((n / FWD_QUEUE) & 1) ^ 1, abort_flag)) return false;
      if (lead) { items[s] = it; mbar_arrive(&item_full[s]); }
      __syncwarp();
      return true;
    };
    for (int asked = 0; ok; ++asked) {
      // the place of a block that has not started yet; the answer is needed when this one's loads are out
      if (!ONE) {
        mbar_expect_tx(grid_bar, 16, lead);
        grid_take_block(grid_next, grid_bar, lead);
      }
      if (it.qt * AT_BM < it.T) {
        const int qs = n % STAGES;
        if (ONE || (ok = mbar_wait_warp(&q_empty[qs], ((n / STAGES) & 1) ^ 1, abort_flag))) {
          mbar_expect_tx(&q_full[qs], TILE_BYTES, lead);
#pragma unroll
          for (int p = 0; p < PANELS; ++p)
            tma_load_2d(sQ + qs * TILE_BYTES + p * 16384, &tmQKV, &q_full[qs], it.h * HD + p * 64, it.first + it.qt * AT_BM, lead);
          nq = n + 1;
          ok = push(it);
          ++n;
        }
        for (int j = 0; j <= it.qt && ok; ++j, ++g) {                          // causal: key tiles 0..qt
          const int st = g % STAGES;
          const uint32_t par = ((g / STAGES) & 1) ^ 1;
          const int row_k = it.first + j * AT_BN;
          if (KV && keep >= 0 && keep % STAGES == st && !(ok = store_kept())) break;
          if (!(ok = mbar_wait_warp(&k_empty[st], par, abort_flag))) break;
          mbar_expect_tx(&k_full[st], TILE_BYTES, lead);
#pragma unroll
          for (int p = 0; p < PANELS; ++p)
            tma_load_2d(sK + st * TILE_BYTES + p * 16384, &tmQKV, &k_full[st], d_model + it.h * HD + p * 64, row_k, lead);
          nk = g + 1;
          if (!(ok = mbar_wait_warp(&v_empty[st], par, abort_flag))) break;
          mbar_expect_tx(&v_full[st], TILE_BYTES, lead);
#pragma unroll
          for (int p = 0; p < PANELS; ++p)
            tma_load_2d(sV + st * TILE_BYTES + p * 16384, &tmQKV, &v_full[st], 2 * d_model + it.h * HD + p * 64, row_k, lead);
          nv = g + 1;
        }
        if (KV && ok) {
          if (keep >= 0) ok = store_kept();
          keep = g - 1;
          keep_rows = min(AT_BM, it.T - it.qt * AT_BM);
          keep_slot = (static_cast<long long>(it.b) * a.H + it.h) * a.slots + it.qt * AT_BM;
        }
      }
      if (ONE) break;
      // before the block leaves, too: the answer is written to its shared memory
      ok = __all_sync(0xffffffffu, mbar_wait_landed(grid_bar, asked & 1)) && ok;
      uint3 block;
      if (!ok || !grid_taken_block(grid_next, block)) break;      // none left, and none may be asked for after that
      it = item_of(block);
      fence_proxy_async_smem();
      __syncwarp();
    }
    if (!ONE && ok) { FwdItem end = {-1, 0, 0, 0, 0}; ok = push(end); }
    if (KV && ok && keep >= 0) ok = store_kept();
    if (!ok) { *abort_flag = ST_TIMEOUT_EMPTY; if (lead) atomicCAS(a.status, 0, ST_TIMEOUT_EMPTY); }
    // when a wait ran out, nobody has waited for these: they land before the block leaves
    for (int i = nq > STAGES ? nq - STAGES : 0; i < nq; ++i) mbar_wait_landed(&q_full[i % STAGES], (i / STAGES) & 1);
    for (int i = nk > STAGES ? nk - STAGES : 0; i < nk; ++i) mbar_wait_landed(&k_full[i % STAGES], (i / STAGES) & 1);
    for (int i = nv > STAGES ? nv - STAGES : 0; i < nv; ++i) mbar_wait_landed(&v_full[i % STAGES], (i / STAGES) & 1);
  } else if (warp == FWD_MMA_WARP) {
    // -------------------------------------------------------------- MMA issuer
    const uint32_t lead = elect_one();
    bool ok = true;
    int g = 0;                                   // key tiles of the items before
    for (int n = 0;; ++n) {
      const volatile FwdItem* it = next_item(n);
      if (!(ok = it != nullptr)) break;
      const int qs = n % STAGES, nkv = it->qt + 1;
      item_done(n);
      if (nkv == 0) break;
      if (!(ok = mbar_wait_warp(&q_full[qs], (n / STAGES) & 1, abort_flag))) break;
      const uint32_t q0 = smem_u32(sQ + qs * TILE_BYTES);
      // S of key tile t.  With P in the place of S the product P V of the tile before was issued earlier (MMAs
      // of one thread execute in order); otherwise the math warps must have read the S before.
      auto issue_qk = [&](int t) {
        const int st = t % STAGES;
        if (!mbar_wait_warp(&k_full[st], (t / STAGES) & 1, abort_flag)) return false;
        if (!C::P_IN_S && t > 0 && !mbar_wait_warp(s_empty, (t - 1) & 1, abort_flag)) return false;
        tc_fence_after();
        const uint32_t k0 = smem_u32(sK + st * TILE_BYTES);
#pragma unroll
        for (int k = 0; k < HD / 16; ++k) {
          const uint32_t off = (k >> 2) * 16384 + (k & 3) * 32;
          umma_bf16(tS, make_sdesc_sw128(q0, off, 16, 1024), make_sdesc_sw128(k0, off, 16, 1024),
                    IDESC_S, k > 0, lead);
        }
        umma_commit(&k_empty[st], lead);
        umma_commit(s_full, lead);
        return true;
      };
      if (!(ok = issue_qk(g))) break;
      for (int j = 0; j < nkv; ++j) {
        const int t = g + j, st = t % STAGES;
        if (!C::P_IN_S && j + 1 < nkv && !(ok = issue_qk(t + 1))) break;
        if (!(ok = mbar_wait_warp(&v_full[st], (t / STAGES) & 1, abort_flag))) break;
        // also: every math warp has read O of the item before (it does so before it writes P of this one)
        if (!(ok = mbar_wait_warp(p_full, t & 1, abort_flag))) break;
        tc_fence_after();
        const uint32_t v0 = smem_u32(sV + st * TILE_BYTES);
#pragma unroll
        for (int k = 0; k < 8; ++k)    // 128 keys = 8 UMMA_K steps of 8 TMEM columns each
          umma_bf16_ts(tO, tP + k * 8, make_sdesc_sw128(v0, k * 2048, 16384, 1024), IDESC_PV, (j > 0 || k > 0), lead);
        umma_commit(&v_empty[st], lead);
        umma_commit(pv_full, lead);
        if (C::P_IN_S && j + 1 < nkv && !(ok = issue_qk(t + 1))) break;
      }
      if (!ok || ONE) break;
      g += nkv;
    }
    if (!ok) { *abort_flag = ST_TIMEOUT_FULL; if (lead) atomicCAS(a.status, 0, ST_TIMEOUT_FULL); }
  } else {
    // ---------------------------------------------------- softmax / output warps
    const int quad = warp & 3, hf = warp >> 2;    // TMEM lane quarter; half of the keys and of O's columns
    const int r = quad * 32 + lane;               // query row inside the tile = TMEM lane
    const uint32_t lane_addr = static_cast<uint32_t>(quad * 32) << 16;
    constexpr int OC = HD / 2;
    // meeting of the two warps of a lane quarter (bounded, one arrival per warp)
    uint32_t met = 0, tile = 0;                   // parities: meetings, key tiles
    auto pair_sync = [&]() {
      __syncwarp();
      if (lane == 0) mbar_arrive(&xchg[quad]);
      met ^= 1;
      return mbar_wait_warp(&xchg[quad], met ^ 1, abort_flag);
    };
    const float sl2 = a.scale * LOG2E;
    const uint64_t sl2_2 = f2_bcast(sl2);
    const uint64_t seed = uniform64(a.thr16 ? salted(a.seed, a.salt) : 0);
    bool ok = true;
    bool leaving = false;                         // output of the item before, out of its Q tile
    for (int n = 0;; ++n) {
      const volatile FwdItem* it = next_item(n);
      if (!(ok = it != nullptr) || it->qt < 0) break;
      const int qt = it->qt, q_idx = qt * AT_BM + r, qs = n % STAGES;
      float m_ref = 0.f;                          // running maximum, which P and O are scaled to
      float l_run = 0.f;                          // row sum of this half's keys
      for (int j = 0; j <= qt; ++j, tile ^= 1) {
        // dropout keep bits of this thread's 64 keys; they are also what the backward pass reads back
        uint32_t keep[2] = {0u, 0u};
        if (a.thr16) {
          const uint64_t e0 = (static_cast<uint64_t>(it->b * a.H + it->h) * a.T + q_idx) * a.T + hf * 64 + j * AT_BN;
#pragma unroll
          for (int c = 0; c < 2; ++c)              // zeros where all 32 rows of the warp are before these keys
            if (j < qt || hf * 64 + c * 32 < quad * 32 + 32)
              keep[c] = dropout_keep32(seed, a.stream_id, (e0 >> 3) + c * 4, a.thr16);
          const int T = a.T;                       // packed batches have no dropout
          if (a.drop_mask && q_idx < T) {
            uint32_t* dst = a.drop_mask + (e0 >> 5);
            if ((T & 63) == 0) {
              if (j * AT_BN + hf * 64 < T) *reinterpret_cast<uint2*>(dst) = make_uint2(keep[0], keep[1]);
            } else {
#pragma unroll
              for (int c = 0; c < 2; ++c)
                if (j * AT_BN + hf * 64 + c * 32 < T) dst[c] = keep[c];
            }
          }
        }
        if (!(ok = mbar_wait_warp(s_full, tile, abort_flag))) break;
        tc_fence_after();
        uint32_t v[64];
#pragma unroll
        for (int c = 0; c < 2; ++c) tmem_ld32(tS + lane_addr + hf * 64 + c * 32, v + c * 32);
        tmem_ld_wait();
        if (!C::P_IN_S) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(s_empty);     // the next S may be computed
        }
        if (j == qt) {                             // diagonal tile: keys after the row's own position
#pragma unroll
          for (int i = 0; i < 64; ++i) v[i] = hf * 64 + i <= r ? v[i] : 0xff800000u;
        }
        float mx4[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) mx4[k] = __uint_as_float(v[k]);
#pragma unroll
        for (int i = 4; i < 64; ++i) mx4[i & 3] = fmaxf(mx4[i & 3], __uint_as_float(v[i]));
        float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
        // the other half's maximum (slots alternate: one is rewritten only after the meeting in between, which
        // its reader has passed)
        float* slot = s_row + met * 256;
        slot[hf * 128 + r] = mx;
        if (!(ok = pair_sync())) break;
        mx = fmaxf(mx, slot[(hf ^ 1) * 128 + r]);  // finite: key 0 is never masked
        float grow = 1.f;                          // what sums and O are multiplied by
        if (j == 0) {
          m_ref = mx;
        } else if (__any_sync(0xffffffffu, mx > m_ref)) {
          if (!(ok = mbar_wait_warp(pv_full, tile ^ 1, abort_flag))) break;
          tc_fence_after();
          const float m_new = fmaxf(m_ref, mx);
          grow = ex2_fast((m_ref - m_new) * sl2);
          const uint64_t f = f2_bcast(grow);
          m_ref = m_new;
#pragma unroll 1
          for (int c = 0; c < OC / 16; ++c) {
            uint32_t o[16];
            tmem_ld16(tO + lane_addr + hf * OC + c * 16, o);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              float lo, hi;
              f2_unpack(f2_mul(f2_pack(__uint_as_float(o[2 * i]), __uint_as_float(o[2 * i + 1])), f), lo, hi);
              o[2 * i] = __float_as_uint(lo);
              o[2 * i + 1] = __float_as_uint(hi);
            }
            tmem_st16(tO + lane_addr + hf * OC + c * 16, o);
          }
        }
        const uint64_t mb = f2_bcast(-m_ref * sl2);
        float rs = 0.f;                            // added up in column order
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          uint32_t w[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            float x0, x1;
            f2_unpack(f2_fma(f2_pack(__uint_as_float(v[c * 32 + 2 * i]), __uint_as_float(v[c * 32 + 2 * i + 1])), sl2_2, mb),
                      x0, x1);
            x0 = ex2_fast(x0);
            x1 = ex2_fast(x1);
            rs += x0;
            rs += x1;
            w[i] = pack_bf16x2(x0, x1);
          }
          if (a.thr16) {
            uint32_t m[16];
            keep_masks16(keep[c], m);
#pragma unroll
            for (int i = 0; i < 16; ++i) w[i] &= m[i];
          }
          // P of the tile before is read by its product until that completes
          if (c == 0 && j > 0 && !(ok = mbar_wait_warp(pv_full, tile ^ 1, abort_flag))) break;
          if (c == 0) tc_fence_after();
          tmem_st16(tP + lane_addr + hf * 32 + c * 16, w);
        }
        if (!ok) break;
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(p_full);                     // one arrival per warp
          if (!ONE && leaving) {                   // that has been read by now
            tma_store_wait_read<0>();
            mbar_arrive(&q_empty[qs ^ 1]);
          }
        }
        leaving = false;
        l_run = l_run * grow + rs;
      }
      if (!ok) break;
      const int T = it->T, h = it->h, b = it->b, row = it->first + qt * AT_BM + quad * 32;    // this warp's first row
      item_done(n);
      if (!(ok = mbar_wait_warp(pv_full, tile ^ 1, abort_flag))) break;
      tc_fence_after();
      float* slot = s_row + met * 256;
      slot[hf * 128 + r] = l_run;
      if (!(ok = pair_sync())) break;
      const float l = slot[r] + slot[128 + r];
      const float inv = dropout_scale(a.thr16) / l;
      // The warps' 32 rows leave through the (now idle) Q tile with one TMA store per 64 columns; warps
      // with rows past the end of the sequence store row by row.
      const bool whole = qt * AT_BM + quad * 32 + 32 <= T;
      uint8_t* out_tile = sQ + qs * TILE_BYTES;
      __nv_bfloat16* orow = a.out + (static_cast<long long>(row) + lane) * d_model + h * HD + hf * OC;
#pragma unroll
      for (int c = 0; c < OC / 32; ++c) {
        uint32_t o[32];
        tmem_ld32(tO + lane_addr + hf * OC + c * 32, o);
        tmem_ld_wait();
        const int col8 = (hf * OC + c * 32) / 8;                  // first 16-byte chunk of the row
        uint8_t* rowp = out_tile + (col8 >> 3) * 16384 + quad * 4096 + lane * 128;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          uint4 w;
          w.x = pack_bf16x2(__uint_as_float(o[k * 8 + 0]) * inv, __uint_as_float(o[k * 8 + 1]) * inv);
          w.y = pack_bf16x2(__uint_as_float(o[k * 8 + 2]) * inv, __uint_as_float(o[k * 8 + 3]) * inv);
          w.z = pack_bf16x2(__uint_as_float(o[k * 8 + 4]) * inv, __uint_as_float(o[k * 8 + 5]) * inv);
          w.w = pack_bf16x2(__uint_as_float(o[k * 8 + 6]) * inv, __uint_as_float(o[k * 8 + 7]) * inv);
          if (whole) *reinterpret_cast<uint4*>(rowp + ((((col8 & 7) + k) ^ (lane & 7)) << 4)) = w;
          else if (q_idx < T) *reinterpret_cast<uint4*>(orow + c * 32 + k * 8) = w;
        }
      }
      if (a.lse && hf == 0 && q_idx < T)
        a.lse[(static_cast<long long>(b) * a.H + h) * a.T + q_idx] = m_ref * a.scale + logf(l);
      if (whole) {
        fence_proxy_async_smem();
        if (!(ok = pair_sync())) break;
        // head_dim 64: one panel of both halves; 128: each half filled a panel of its own
        leaving = hf < PANELS;
        if (leaving && lane == 0) {
          tma_store_2d(&tmO, out_tile + hf * 16384 + quad * 4096, h * HD + hf * 64, row);
          tma_store_commit();
        }
      }
      if (ONE) break;
      // The tile may be loaded again once the stores have read it: with two tiles that is said behind the first
      // keys of the next item, with one the next item's Q waits for it.
      if (STAGES == 1 || !leaving) {
        __syncwarp();
        if (lane == 0) {
          if (leaving) tma_store_wait_read<0>();
          mbar_arrive(&q_empty[qs]);
        }
        leaving = false;
      }
    }
    if (lane == 0) tma_store_wait_read<0>();       // the staging tile outlives the read
    if (!ok) { *abort_flag = ST_TIMEOUT_TMEM_FULL; atomicCAS(a.status, 0, ST_TIMEOUT_TMEM_FULL); }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == FWD_MMA_WARP) { tc_fence_after(); tmem_dealloc(tmem_base, 256); }
}

}  // namespace ab

// =================================================================================================
// Backward.  Two launches of one templated kernel, both with threads = query rows:
//   MODE 0 (key/value-stationary): CTA owns key tile j, streams query tiles i >= j, accumulates
//           dV_j += P^T dO_i and dK_j += dS^T Q_i in TMEM.
//   MODE 1 (query-stationary)    : CTA owns query tile i, streams key tiles j <= i, accumulates
//           dQ_i += dS K_j in TMEM.
// Both recompute S = Q K^T and dP = dO V^T per tile pair, so no atomics and no fp32 dQ buffer
// are needed.  P and dS are written once to shared memory as [query row][key] bf16 panels; that
// one layout is the K-major A operand of dS*K and the MN-major A operand of P^T*dO / dS^T*Q.
// delta[b,h,t] = sum_c dO*O is produced by a small pre-kernel.
namespace ab {


// One thread per 16-byte chunk of O / dO (hd / 8 adjacent lanes share one (row, head)), so a
// warp reads 512 contiguous bytes of each tensor; the lanes of a (row, head) fold their partial
// dot products with shuffles.
__global__ void __launch_bounds__(256)
attn_delta_kernel(const __nv_bfloat16* __restrict__ o, const __nv_bfloat16* __restrict__ dout,
                  float* __restrict__ delta, int B, int T, int H, int hd) {
  griddep_enter();
  const int cpr = hd >> 3;                                    // chunks per (row, head): 8 or 16
  const long long total = static_cast<long long>(B) * T * H * cpr;
  const long long gid = blockIdx.x * 256ll + threadIdx.x;
  float s = 0.f;
  if (gid < total) {
    const uint4 x = __ldcs(reinterpret_cast<const uint4*>(o) + gid);
    const uint4 y = __ldcs(reinterpret_cast<const uint4*>(dout) + gid);
    s = bf16_lo(x.x) * bf16_lo(y.x) + bf16_hi(x.x) * bf16_hi(y.x);
    s += bf16_lo(x.y) * bf16_lo(y.y) + bf16_hi(x.y) * bf16_hi(y.y);
    s += bf16_lo(x.z) * bf16_lo(y.z) + bf16_hi(x.z) * bf16_hi(y.z);
    s += bf16_lo(x.w) * bf16_lo(y.w) + bf16_hi(x.w) * bf16_hi(y.w);
  }
  for (int off = 1; off < cpr; off <<= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
  if (gid < total && (gid & (cpr - 1)) == 0) {
    const long long rh = gid / cpr;                           // row * H + head
    const int hh = static_cast<int>(rh % H);
    const long long row = rh / H;
    const int bb = static_cast<int>(row / T), t = static_cast<int>(row % T);
    delta[(static_cast<long long>(bb) * H + hh) * T + t] = s;
  }
}

constexpr int BWD_MATH_WARPS = 16;
constexpr int BWD_MATH_THREADS = BWD_MATH_WARPS * 32;
constexpr int BWD_TMA_WARP = BWD_MATH_WARPS;
constexpr int BWD_MMA_WARP = BWD_MATH_WARPS + 1;
constexpr int BWD_THREADS = (BWD_MATH_WARPS + 2) * 32;

template <int HD, int MODE>
__global__ void __launch_bounds__(BWD_THREADS, 1)
attn_bwd_kernel(const __grid_constant__ CUtensorMap tmQKV, const __grid_constant__ CUtensorMap tmDO,
                const AttnBwdArgs a) {
  griddep_enter();
  constexpr int STAGES = HD <= 64 ? 2 : 1;
  constexpr int PANELS = HD / 64;
  constexpr int TILE_BYTES = 128 * HD * 2;
  constexpr int P_BYTES = 128 * 128 * 2;
  constexpr uint32_t IDESC_S = make_idesc_bf16(128, 128, 0, 0);     // Q K^T and dO V^T
  constexpr uint32_t IDESC_T = make_idesc_bf16(128, HD, 1, 1);      // P^T dO, dS^T Q (both MN-major)
  constexpr uint32_t IDESC_DQ = make_idesc_bf16(128, HD, 0, 1);     // dS K

  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = smem_raw;
  if (smem_u32(smem) & 1023) {
    if (threadIdx.x == 0) atomicCAS(a.status, 0, ST_BAD_ARGUMENT);
    return;
  }
  uint8_t* sStatA = smem;                                  // MODE 0: K_j   MODE 1: Q_i
  uint8_t* sStatB = sStatA + TILE_BYTES;                   // MODE 0: V_j   MODE 1: dO_i
  uint8_t* sStrX = sStatB + TILE_BYTES;                    // MODE 0: Q_i   MODE 1: K_j   (STAGES)
  uint8_t* sStrY = sStrX + STAGES * TILE_BYTES;            // MODE 0: dO_i  MODE 1: V_j   (STAGES)
  uint8_t* sP = sStrY + STAGES * TILE_BYTES;
  uint8_t* sDS = sP + P_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sDS + P_BYTES);
  uint64_t* stat_full = bars;
  uint64_t* full = bars + 1;        // STAGES
  uint64_t* empty = bars + 3;       // STAGES
  uint64_t* sdp_full = bars + 5;
  uint64_t* sdp_empty = bars + 6;
  uint64_t* pds_full = bars + 7;
  uint64_t* pds_empty = bars + 8;
  uint64_t* acc_full = bars + 9;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 10);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = warp_number(), lane = threadIdx.x & 31;
  const int nt = (a.T + 127) / 128;
  const int h = blockIdx.y, b = blockIdx.z;
  // MODE 0: own key tile `own`, iterate query tiles own..nt-1 (heaviest = small own first)
  // MODE 1: own query tile `own`, iterate key tiles 0..own (heaviest = large own first)
  const int own = MODE == 0 ? static_cast<int>(blockIdx.x) : nt - 1 - static_cast<int>(blockIdx.x);
  const int n_iter = MODE == 0 ? nt - own : own + 1;
  const int d_model = a.H * HD;

  if (threadIdx.x == 0) {
    mbar_init(stat_full, 1);
    for (int i = 0; i < STAGES; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], 1); }
    mbar_init(sdp_full, 1); mbar_init(sdp_empty, BWD_MATH_WARPS);
    mbar_init(pds_full, BWD_MATH_WARPS); mbar_init(pds_empty, 1); mbar_init(acc_full, 1);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmQKV);
    tma_prefetch_desc(&tmDO);
  }
  if (warp == BWD_MMA_WARP) { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tS = tmem_base, tDP = tmem_base + 128, tAcc0 = tmem_base + 256,
                 tAcc1 = tmem_base + 256 + HD;

  if (warp == BWD_TMA_WARP) {
    // ------------------------------------------------------------ TMA producer
    {
      const uint32_t lead = elect_one();
      const int row_own = b * a.T + own * 128;
      mbar_expect_tx(stat_full, 2 * TILE_BYTES, lead);
#pragma unroll
      for (int p = 0; p < PANELS; ++p) {
        if (MODE == 0) {
          tma_load_2d(sStatA + p * 16384, &tmQKV, stat_full, d_model + h * HD + p * 64, row_own, lead);
          tma_load_2d(sStatB + p * 16384, &tmQKV, stat_full, 2 * d_model + h * HD + p * 64, row_own, lead);
        } else {
          tma_load_2d(sStatA + p * 16384, &tmQKV, stat_full, h * HD + p * 64, row_own, lead);
          tma_load_2d(sStatB + p * 16384, &tmDO, stat_full, h * HD + p * 64, row_own, lead);
        }
      }
      for (int it = 0; it < n_iter; ++it) {
        const int st = it % STAGES;
        const uint32_t use = it / STAGES;
        const int tile = MODE == 0 ? own + it : it;
        const int row = b * a.T + tile * 128;
        if (!mbar_wait_warp(&empty[st], (use & 1) ^ 1, abort_flag)) {
          *abort_flag = ST_TIMEOUT_EMPTY; if (lead) atomicCAS(a.status, 0, ST_TIMEOUT_EMPTY); break;
        }
        mbar_expect_tx(&full[st], 2 * TILE_BYTES, lead);
#pragma unroll
        for (int p = 0; p < PANELS; ++p) {
          if (MODE == 0) {
            tma_load_2d(sStrX + st * TILE_BYTES + p * 16384, &tmQKV, &full[st], h * HD + p * 64, row, lead);
            tma_load_2d(sStrY + st * TILE_BYTES + p * 16384, &tmDO, &full[st], h * HD + p * 64, row, lead);
          } else {
            tma_load_2d(sStrX + st * TILE_BYTES + p * 16384, &tmQKV, &full[st],
                        d_model + h * HD + p * 64, row, lead);
            tma_load_2d(sStrY + st * TILE_BYTES + p * 16384, &tmQKV, &full[st],
                        2 * d_model + h * HD + p * 64, row, lead);
          }
        }
      }
    }
  } else if (warp == BWD_MMA_WARP) {
    // -------------------------------------------------------------- MMA issuer
    {
      const uint32_t lead = elect_one();
      bool ok = mbar_wait_warp(stat_full, 0, abort_flag);
      // group 1: S = Q K^T, dP = dO V^T
      auto issue_sdp = [&](int it) {
        const int st = it % STAGES;
        if (!mbar_wait_warp(&full[st], (it / STAGES) & 1, abort_flag)) return false;
        if (it > 0 && !mbar_wait_warp(sdp_empty, (it - 1) & 1, abort_flag)) return false;
        tc_fence_after();
        const uint32_t x = smem_u32(sStrX + st * TILE_BYTES), y = smem_u32(sStrY + st * TILE_BYTES);
        const uint32_t sa = smem_u32(sStatA), sb = smem_u32(sStatB);
        const uint32_t q = MODE == 0 ? x : sa, kk = MODE == 0 ? sa : x;
        const uint32_t dO = MODE == 0 ? y : sb, vv = MODE == 0 ? sb : y;
#pragma unroll
        for (int k = 0; k < HD / 16; ++k) {
          const uint32_t off = (k >> 2) * 16384 + (k & 3) * 32;
          umma_bf16(tS, make_sdesc_sw128(q, off, 16, 1024), make_sdesc_sw128(kk, off, 16, 1024),
                    IDESC_S, k > 0, lead);
        }
#pragma unroll
        for (int k = 0; k < HD / 16; ++k) {
          const uint32_t off = (k >> 2) * 16384 + (k & 3) * 32;
          umma_bf16(tDP, make_sdesc_sw128(dO, off, 16, 1024), make_sdesc_sw128(vv, off, 16, 1024),
                    IDESC_S, k > 0, lead);
        }
        umma_commit(sdp_full, lead);
        return true;
      };
      // group 2: the accumulating products
      auto issue_acc = [&](int it) {
        const int st = it % STAGES;
        if (!mbar_wait_warp(pds_full, it & 1, abort_flag)) return false;
        tc_fence_after();
        const uint32_t x = smem_u32(sStrX + st * TILE_BYTES), y = smem_u32(sStrY + st * TILE_BYTES);
        const uint32_t p0 = smem_u32(sP), ds0 = smem_u32(sDS);
        if (MODE == 0) {
#pragma unroll
          for (int k = 0; k < 8; ++k) {   // contraction over 128 query rows
            umma_bf16(tAcc0, make_sdesc_sw128(p0, k * 2048, 16384, 1024),
                      make_sdesc_sw128(y, k * 2048, 16384, 1024), IDESC_T, (it > 0 || k > 0), lead);
          }
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            umma_bf16(tAcc1, make_sdesc_sw128(ds0, k * 2048, 16384, 1024),
                      make_sdesc_sw128(x, k * 2048, 16384, 1024), IDESC_T, (it > 0 || k > 0), lead);
          }
        } else {
#pragma unroll
          for (int k = 0; k < 8; ++k) {   // contraction over 128 keys
            umma_bf16(tAcc0, make_sdesc_sw128(ds0, (k >> 2) * 16384 + (k & 3) * 32, 16, 1024),
                      make_sdesc_sw128(x, k * 2048, 16384, 1024), IDESC_DQ, (it > 0 || k > 0), lead);
          }
        }
        umma_commit(&empty[st], lead);
        umma_commit(pds_empty, lead);
        return true;
      };
      if (ok) ok = issue_sdp(0);
      for (int it = 0; it < n_iter && ok; ++it) {
        if (STAGES > 1 && it + 1 < n_iter) { ok = issue_sdp(it + 1); if (!ok) break; }
        ok = issue_acc(it);
        if (!ok) break;
        if (STAGES == 1 && it + 1 < n_iter) ok = issue_sdp(it + 1);
      }
      if (ok) umma_commit(acc_full, lead);
      else { *abort_flag = ST_TIMEOUT_FULL; if (lead) atomicCAS(a.status, 0, ST_TIMEOUT_FULL); }
    }
  } else {
    // ------------------------------------------------------------ math warps
    // warp w: TMEM lane quarter w & 3 (query rows 32*(w&3)..), key columns 32*(w>>2)..+31
    const int r = (warp & 3) * 32 + lane;
    const int cb = warp >> 2;
    const uint32_t lane_addr = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const float sl2 = a.scale * LOG2E;
    const uint64_t seed = uniform64(a.thr16 ? salted(a.seed, a.salt) : 0);
    const float dscale = dropout_scale(a.thr16);
    const long long bh = static_cast<long long>(b) * a.H + h;
    bool ok = true;
    for (int it = 0; it < n_iter && ok; ++it) {
      const int qi = MODE == 0 ? own + it : own;     // query tile
      const int kj = MODE == 0 ? own : it;           // key tile
      const int q_idx = qi * 128 + r;
      const bool q_ok = q_idx < a.T;
      const float lse_l2 = q_ok ? a.lse[bh * a.T + q_idx] * LOG2E : 0.f;
      const float dlt = q_ok ? a.delta[bh * a.T + q_idx] : 0.f;
      const bool diag = (qi == kj);
      const uint64_t row_elem0 = (static_cast<uint64_t>(bh) * a.T + q_idx) * a.T + kj * 128 + cb * 32;
      if (!mbar_wait_warp(sdp_full, it & 1, abort_flag)) { ok = false; break; }
      if (it > 0 && !mbar_wait_warp(pds_empty, (it - 1) & 1, abort_flag)) { ok = false; break; }
      tc_fence_after();
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) {      // two 16-column pieces keep the register count low
        const int col0 = cb * 32 + hf * 16;
        uint32_t sv[16], dv[16];
        tmem_ld16(tS + lane_addr + col0, sv);
        tmem_ld16(tDP + lane_addr + col0, dv);
        tmem_ld_wait();
        float p[16], ds[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const bool live = q_ok && (!diag || (col0 + i) <= r);
          p[i] = live ? ex2_fast(__uint_as_float(sv[i]) * sl2 - lse_l2) : 0.f;
          ds[i] = __uint_as_float(dv[i]);
        }
        if (a.thr16) {
#pragma unroll
          for (int g = 0; g < 2; ++g) {
            const uint64_t e0 = row_elem0 + hf * 16 + g * 8;
            // keys past the end of the sequence have no bits: their words are the next row's, or past the mask
            const uint32_t keep = a.drop_mask
                ? (q_ok && kj * 128 + col0 < a.T ? (a.drop_mask[e0 >> 5] >> (e0 & 31)) & 0xffu : 0u)
                : dropout_keep8(seed, a.stream_id, e0 >> 3, a.thr16);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const bool kp = (keep >> i) & 1u;
              const float pd = kp ? p[g * 8 + i] * dscale : 0.f;          // dropped P (for dV)
              const float dpe = kp ? ds[g * 8 + i] * dscale : 0.f;        // grad wrt softmax prob
              ds[g * 8 + i] = p[g * 8 + i] * (dpe - dlt) * a.scale;
              p[g * 8 + i] = pd;
            }
          }
        } else {
#pragma unroll
          for (int i = 0; i < 16; ++i) ds[i] = p[i] * (ds[i] - dlt) * a.scale;
        }
        const uint32_t poff = (col0 >> 6) * 16384;
#pragma unroll
        for (int g = 0; g < 2; ++g) {
          const uint32_t off = poff + sw128_chunk(r, ((col0 & 63) >> 3) + g);
          uint4 w;
          if (MODE == 0) {
            w.x = pack_bf16x2(p[g * 8 + 0], p[g * 8 + 1]); w.y = pack_bf16x2(p[g * 8 + 2], p[g * 8 + 3]);
            w.z = pack_bf16x2(p[g * 8 + 4], p[g * 8 + 5]); w.w = pack_bf16x2(p[g * 8 + 6], p[g * 8 + 7]);
            *reinterpret_cast<uint4*>(sP + off) = w;
          }
          w.x = pack_bf16x2(ds[g * 8 + 0], ds[g * 8 + 1]); w.y = pack_bf16x2(ds[g * 8 + 2], ds[g * 8 + 3]);
          w.z = pack_bf16x2(ds[g * 8 + 4], ds[g * 8 + 5]); w.w = pack_bf16x2(ds[g * 8 + 6], ds[g * 8 + 7]);
          *reinterpret_cast<uint4*>(sDS + off) = w;
        }
      }
      // one arrival per warp: hundreds of threads arriving on one mbarrier serialise on it
      tc_fence_before();
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) { mbar_arrive(sdp_empty); mbar_arrive(pds_full); }
    }
    if (ok && !mbar_wait_warp(acc_full, 0, abort_flag)) ok = false;
    if (!ok) { *abort_flag = ST_TIMEOUT_TMEM_FULL; atomicCAS(a.status, 0, ST_TIMEOUT_TMEM_FULL); }
    if (ok) {
      tc_fence_after();
      const int t_idx = own * 128 + r;   // row of the owned tile (key row in MODE 0, query row in MODE 1)
      __nv_bfloat16* base = a.dqkv + (static_cast<long long>(b) * a.T + t_idx) * (3 * d_model) + h * HD;
      constexpr int NACC = MODE == 0 ? 2 : 1;
      constexpr int CH = HD / 32;        // 32-column chunks per accumulator
      // MODE 0: acc0 = dV -> third block, acc1 = dK -> second block.  MODE 1: acc0 = dQ -> first.
      for (int g = cb; g < NACC * CH; g += 4) {
        const int which = g / CH, c = g % CH;
        const uint32_t tacc = which == 0 ? tAcc0 : tAcc1;
        __nv_bfloat16* dst = base + (MODE == 0 ? (which == 0 ? 2 * d_model : d_model) : 0);
        uint32_t v[32];
        tmem_ld32(tacc + lane_addr + c * 32, v);
        tmem_ld_wait();
        if (t_idx < a.T) {
#pragma unroll
          for (int q4 = 0; q4 < 4; ++q4) {
            uint4 w;
            w.x = pack_bf16x2(__uint_as_float(v[q4 * 8 + 0]), __uint_as_float(v[q4 * 8 + 1]));
            w.y = pack_bf16x2(__uint_as_float(v[q4 * 8 + 2]), __uint_as_float(v[q4 * 8 + 3]));
            w.z = pack_bf16x2(__uint_as_float(v[q4 * 8 + 4]), __uint_as_float(v[q4 * 8 + 5]));
            w.w = pack_bf16x2(__uint_as_float(v[q4 * 8 + 6]), __uint_as_float(v[q4 * 8 + 7]));
            *reinterpret_cast<uint4*>(dst + c * 32 + q4 * 8) = w;
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == BWD_MMA_WARP) { tc_fence_after(); tmem_dealloc(tmem_base, 512); }
}

}  // namespace ab

// ------------------------------------------------------------------------------------ host side
namespace ab {
int launch_attn_bwd_fused64(const CUtensorMap& tq, const CUtensorMap& td, const AttnBwdArgs& a,
                            int* launched, cudaStream_t stream);   // attn_bwd_fused.cu

template <int HD, bool KV, bool ONE>
static int launch_attn_fwd_kernel(const CUtensorMap& tm, const CUtensorMap& tmo, const KvMaps<KV>& cache, dim3 grid,
                                  const AttnArgs& a, int dependent, cudaStream_t stream) {
  constexpr int SMEM = FwdCfg<HD>::SMEM;
  auto kern = attn_fwd_kernel<HD, KV, ONE>;
  static PerDeviceOnce attr;
  if (attr.first_use_on_device()) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
    if (e != cudaSuccess) return (int)e;
    // two CTAs per SM only fit when the SM is configured for its largest shared-memory carve-out
    e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout,
                             cudaSharedmemCarveoutMaxShared);
    if (e != cudaSuccess) return (int)e;
    attr.mark_device();
  }
  if (dependent) return (int)launch_dependent(kern, grid, dim3(FWD_THREADS), SMEM, stream, tm, tmo, cache, a);
  launch_chained(kern, grid, dim3(FWD_THREADS), SMEM, stream, tm, tmo, cache, a);
  return (int)cudaGetLastError();
}

// Whether blocks are taken over.  An item is then tied to a CTA when that one starts on the item before, heaviest items
// first, while the grid gives it to whoever is free; so it takes more rounds of the resident CTAs to pay the longer
// the items are, and with heads of 128, whose one Q tile lets the next item's loads wait for the output, two at
// least.  us, a block per item and taken over, from 150 sizes between 16 and 12000 items, heads of 64: 320 items of
// 128 keys 10.0 and 8.7, 900 18.9 and 14.6; 320 of 512 keys 14.9 and 16.9, 600 21.5 and 21.8, 900 29.2 and 27.9,
// 1500 46.6 and 40.5; 600 of 1000 keys 33.0 and 34.6, 900 44.0 and 44.0, 1500 68.4 and 63.2.  The rule's choice is
// 0.5 % from the better of the two on average, 11 % at worst (450 items of two key tiles fill a wave and a
// half).
static bool fwd_takes_over(long long items, int tiles, int hd, int sms) {
  return 2 * items > 2ll * sms * std::max(hd == 128 ? 4 : 2, tiles);
}

template <int HD, bool KV>
static int launch_attn_fwd(const CUtensorMap& tm, const AttnArgs& a, uint64_t rows, int dependent,
                           cudaStream_t stream) {
  // output map: boxes of 32 rows x 64 columns (half a math warp's rows at head_dim 128)
  CUtensorMap tmo;
  int rc = make_tmap_2d_sw(&tmo, a.out, rows, (uint64_t)a.H * HD, (uint64_t)a.H * HD, 32, 64, 2, 128);
  if (rc) return rc;
  KvMaps<KV> cache;
  if constexpr (KV) {                            // rows of HD
    const uint64_t slots = (uint64_t)a.B * a.H * a.slots;
    if (slots > 0x7fffffffull) return -1;
    if ((rc = make_tmap_2d_sw(&cache.k, a.kc, slots, HD, HD, 32, 64, 2, 128)) != 0) return rc;
    if ((rc = make_tmap_2d_sw(&cache.v, a.vc, slots, HD, HD, 32, 64, 2, 128)) != 0) return rc;
  }
  dim3 grid((a.T + 127) / 128, a.H, a.B);
  int sms = 0;
  if (const cudaError_t e = device_sms(&sms)) return (int)e;
  // Not in programmatic chains, as a precaution: when a grid whose blocks are taken over releases its dependents was
  // not established, and a wait for it has no limit.  No fault was traced to it.
  const bool chain = dependent || g_pdl_chain;
  const bool take_over = !chain && fwd_takes_over(static_cast<long long>(grid.x) * grid.y * grid.z, grid.x, HD, sms);
  return take_over ? launch_attn_fwd_kernel<HD, KV, false>(tm, tmo, cache, grid, a, dependent, stream)
                   : launch_attn_fwd_kernel<HD, KV, true>(tm, tmo, cache, grid, a, dependent, stream);
}

template <int HD, int MODE>
static int launch_attn_bwd(const CUtensorMap& tq, const CUtensorMap& td, const AttnBwdArgs& a,
                           cudaStream_t stream) {
  constexpr int STAGES = HD <= 64 ? 2 : 1;
  constexpr int SMEM = (2 + 2 * STAGES) * 128 * HD * 2 + 2 * 128 * 128 * 2 + 256;
  auto kern = attn_bwd_kernel<HD, MODE>;
  static PerDeviceOnce attr;
  if (attr.first_use_on_device()) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
    if (e != cudaSuccess) return (int)e;
    attr.mark_device();
  }
  dim3 grid((a.T + 127) / 128, a.H, a.B);
  launch_chained(kern, grid, dim3(BWD_THREADS), SMEM, stream, tq, td, a);
  return (int)cudaGetLastError();
}
}  // namespace ab

extern "C" {

int ab_colsum_bf16(const void* x, long long ld, int M, int N, float* out, const int* m_limit, cudaStream_t stream);

// delta[b][h][t] = sum over the head's columns of dO * O (o, dout: bf16 [B*T, H*hd])
int ab_attn_delta(const void* o, const void* dout, float* delta, int B, int T, int H, int hd, cudaStream_t stream) {
  using namespace ab;
  if ((hd != 64 && hd != 128) || B <= 0 || T <= 0 || H <= 0) return -1;
  const long long n = (long long)B * T * H * (hd / 8);
  launch_chained(attn_delta_kernel, dim3((unsigned)((n + 255) / 256)), dim3(256), 0, stream,
                 (const __nv_bfloat16*)o, (const __nv_bfloat16*)dout, delta, B, T, H, hd);
  return (int)cudaGetLastError();
}

// qkv: bf16 [B*T, 3*H*hd]; out: bf16 [B*T, H*hd]; lse: fp32 [B,H,T] (may be null).
// hd must be 64 or 128.  With dropout (thr16 > 0) T must be a multiple of 8.
// drop_mask (optional): uint32 [B,H,T,T/32], receives the dropout keep bits (needs T % 32 == 0).
int ab_attn_fwd(const void* qkv, void* out, float* lse, unsigned int* drop_mask, int B, int T, int H,
                int hd, float scale, unsigned long long seed, unsigned int stream_id,
                unsigned int thr16, int* status, cudaStream_t stream) {
  using namespace ab;
  if ((hd != 64 && hd != 128) || B <= 0 || T <= 0 || (thr16 && (T & 7))) return -1;
  if (drop_mask && (T & 31)) return -1;
  CUtensorMap tm;
  int rc = make_tmap_2d(&tm, qkv, (uint64_t)B * T, 3ull * H * hd, 3ull * H * hd, 128, 64, 2, true);
  if (rc) return rc;
  AttnArgs a;
  a.B = B; a.T = T; a.H = H; a.hd = hd; a.scale = scale; a.seed = seed; a.stream_id = stream_id;
  a.thr16 = thr16; a.out = (__nv_bfloat16*)out; a.lse = lse; a.status = status; a.salt = seed_salt_ptr();
  a.drop_mask = drop_mask; a.row0 = nullptr; a.kc = a.vc = nullptr; a.slots = 0;
  const uint64_t rows = (uint64_t)B * T;
  return hd == 64 ? launch_attn_fwd<64, false>(tm, a, rows, 0, stream) : launch_attn_fwd<128, false>(tm, a, rows, 0, stream);
}

// For tests: whether blocks are taken over in a launch of `items` items of up to `tiles` key tiles, outside chains
int ab_attn_fwd_takes_over(int items, int tiles, int hd, int sms) { return ab::fwd_takes_over(items, tiles, hd, sms); }

// The same over a packed batch without padding (inference: no dropout, no log-sum-exp): sequence b is
// rows [row0[b], row0[b+1]) of qkv [rows, 3*H*hd]; T = longest sequence.  `dependent`: launched as a
// programmatic dependent of the kernel before it.  kc, vc (optional, bf16 [B, H, slots, hd], 16-byte aligned): receive
// the keys and values of every sequence in slots 0, 1, ...; T <= slots.
int ab_attn_fwd_packed_kv(const void* qkv, void* out, const int* row0, int B, int T, int rows, int H, int hd, float scale,
                          void* kc, void* vc, int slots, int dependent, int* status, cudaStream_t stream) {
  using namespace ab;
  if ((hd != 64 && hd != 128) || B <= 0 || T <= 0 || rows < B || !row0) return -1;
  if ((kc == nullptr) != (vc == nullptr) || (kc && T > slots)) return -1;
  CUtensorMap tm;
  int rc = make_tmap_2d(&tm, qkv, (uint64_t)rows, 3ull * H * hd, 3ull * H * hd, 128, 64, 2, true);
  if (rc) return rc;
  AttnArgs a = {};
  a.B = B; a.T = T; a.row0 = row0; a.H = H; a.hd = hd; a.scale = scale; a.out = (__nv_bfloat16*)out; a.status = status;
  a.kc = (__nv_bfloat16*)kc; a.vc = (__nv_bfloat16*)vc; a.slots = slots;
  if (kc)
    return hd == 64 ? launch_attn_fwd<64, true>(tm, a, rows, dependent, stream)
                    : launch_attn_fwd<128, true>(tm, a, rows, dependent, stream);
  return hd == 64 ? launch_attn_fwd<64, false>(tm, a, rows, dependent, stream)
                  : launch_attn_fwd<128, false>(tm, a, rows, dependent, stream);
}
int ab_attn_fwd_packed(const void* qkv, void* out, const int* row0, int B, int T, int rows, int H, int hd, float scale,
                       int dependent, int* status, cudaStream_t stream) {
  return ab_attn_fwd_packed_kv(qkv, out, row0, B, T, rows, H, hd, scale, nullptr, nullptr, 0, dependent, status, stream);
}

// delta: fp32 scratch [B,H,T] owned by the caller.  drop_mask (optional): the keep bits the forward
// pass wrote.  dq_acc (optional, hd == 64): fp32 [B*T, H*hd] accumulator that must be all zero on
// entry and is all zero again on return; when given, the single-kernel backward runs.
// dbias (optional, fp32 [3*H*hd]): the column sums of dqkv are added to it (the bias gradient of the
// QKV projection).  delta_ready: delta already holds the row sums of dO * O.  launched (optional, host):
// receives the number of kernels launched.
int ab_attn_bwd(const void* qkv, const void* out, const float* lse, const void* dout, void* dqkv,
                float* delta, const unsigned int* drop_mask, float* dq_acc, int B, int T, int H, int hd,
                float scale, unsigned long long seed, unsigned int stream_id, unsigned int thr16,
                float* dbias, int delta_ready, int* launched, int* status, cudaStream_t stream) {
  using namespace ab;
  int count = 0;
  if (!launched) launched = &count;
  *launched = 0;
  if ((hd != 64 && hd != 128) || B <= 0 || T <= 0 || (thr16 && (T & 7))) return -1;
  if (drop_mask && (T & 31)) return -1;
  CUtensorMap tq, td;
  int rc = make_tmap_2d(&tq, qkv, (uint64_t)B * T, 3ull * H * hd, 3ull * H * hd, 128, 64, 2, true);
  if (rc) return rc;
  rc = make_tmap_2d(&td, dout, (uint64_t)B * T, (uint64_t)H * hd, (uint64_t)H * hd, 128, 64, 2, true);
  if (rc) return rc;
  if (!delta_ready) {
    if ((rc = ab_attn_delta(out, dout, delta, B, T, H, hd, stream)) != 0) return rc;
    ++*launched;
  }
  AttnBwdArgs a;
  a.B = B; a.T = T; a.H = H; a.hd = hd; a.scale = scale; a.seed = seed; a.stream_id = stream_id;
  a.thr16 = thr16; a.lse = lse; a.delta = delta; a.dqkv = (__nv_bfloat16*)dqkv; a.status = status;
  a.salt = seed_salt_ptr();
  a.drop_mask = drop_mask; a.dq_acc = dq_acc; a.dbias = dbias;
  if (hd == 64 && dq_acc) return launch_attn_bwd_fused64(tq, td, a, launched, stream);
  rc = hd == 64 ? launch_attn_bwd<64, 0>(tq, td, a, stream) : launch_attn_bwd<128, 0>(tq, td, a, stream);
  if (rc) return rc;
  rc = hd == 64 ? launch_attn_bwd<64, 1>(tq, td, a, stream) : launch_attn_bwd<128, 1>(tq, td, a, stream);
  if (rc) return rc;
  *launched += 2;
  if (!dbias) return 0;
  ++*launched;
  return ab_colsum_bf16(dqkv, 3ll * H * hd, B * T, 3 * H * hd, dbias, nullptr, stream);
}
}

// ------------------------------------------------------------------------------------------------
// Allocation-free variant (see attn_static.cuh for who needs it and why).
#include <atomic>

#include "attn_static.cuh"

namespace ab {
// Scratch for `delta`.  In host code this name is only a handle; the device address is looked up
// per device below.
static __device__ __align__(256) float g_attn_static_delta[AB_ATTN_STATIC_MAX_ROWS];
// Per-device cache of the array's device address.  Host threads may fill an entry concurrently;
// they all store the same value, and the atomic keeps the store and the loads untorn.
static std::atomic<float*> g_attn_static_ptr[64];
}  // namespace ab

extern "C" int ab_attn_bwd_static(const void* qkv, const void* out, const float* lse,
                                  const void* dout, void* dqkv, const unsigned int* drop_mask, int B,
                                  int T, int H, int hd, float scale, unsigned long long seed,
                                  unsigned int stream_id, unsigned int thr16, int* status,
                                  cudaStream_t stream) {
  using namespace ab;
  if (B <= 0 || T <= 0 || H <= 0) return -1;
  if (static_cast<long long>(B) * H * T > AB_ATTN_STATIC_MAX_ROWS) return -10;
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return (int)e;
  if (dev < 0 || dev >= 64) return -11;
  float* scratch = g_attn_static_ptr[dev].load(std::memory_order_acquire);
  if (!scratch) {
    // once per device, with that device current: turn the symbol into a device pointer
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_attn_static_delta);
    if (e != cudaSuccess) return (int)e;
    scratch = static_cast<float*>(p);
    g_attn_static_ptr[dev].store(scratch, std::memory_order_release);
  }
  return ab_attn_bwd(qkv, out, lse, dout, dqkv, scratch, drop_mask, nullptr, B, T, H, hd,
                     scale, seed, stream_id, thr16, nullptr, 0, nullptr, status, stream);
}
