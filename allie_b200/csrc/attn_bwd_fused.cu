// Single-kernel attention backward for head_dim 64 (the medium / large configurations).
//
// A CTA owns one 128-row key/value tile j of one (batch, head) and streams the query tiles
// i >= j.  Per pair (i, j) the tensor core runs five products, S and dP into TMEM, then
// dV += P^T dO, dK += dS^T Q (accumulated over i in TMEM) and dQ_ij = dS K_j (fresh each time,
// double-buffered).  The 16 math warps turn S/dP into P/dS exactly once per pair - half the
// exponentials and dropout work of the two-kernel scheme - and push each dQ_ij tile to an fp32
// accumulator in global memory with TMA reduce-add, one 32x16 box per warp, so no atomics are
// issued by threads.  With one key tile per CTA a trailing kernel converts the fp32 dQ to bf16
// into the packed dQKV activation and the accumulator is cleared for the next layer; the persistent
// walk does both by itself.
//
// TMEM columns (512): S 0-127 | dP 128-255 | dV 256-319 | dK 320-383 | dQ 384-447, 448-511.
#include "attn_common.cuh"
#include <algorithm>
#include <cstdlib>

extern "C" int ab_colsum_bf16(const void* x, long long ld, int M, int N, float* out, const int* m_limit,
                              cudaStream_t stream);

namespace ab {


constexpr int FB_MATH_WARPS = 16;
constexpr int FB_MATH_THREADS = FB_MATH_WARPS * 32;
constexpr int FB_TMA_WARP = FB_MATH_WARPS;
constexpr int FB_MMA_WARP = FB_MATH_WARPS + 1;
constexpr int FB_THREADS = (FB_MATH_WARPS + 2) * 32;
constexpr int FB_TILE = 128 * 64 * 2;       // one 128 x 64 bf16 tile
constexpr int FB_P = 128 * 128 * 2;

// P and dS for 16 adjacent keys of one query row.
//   p_i  = exp2(s_i * sl2 - lse_l2)                       (0 on masked keys)
//   P_i  = keep_i ? p_i * dscale : 0                      (what multiplies dO in dV)
//   dS_i = p_i * ((keep_i ? dP_i * dscale : 0) - delta) * scale
// A row outside the sequence passes lse_l2 = +inf, which makes every p_i zero without a select;
// the dropout decision is applied as a multiplication by m_i = keep_i ? dscale : 0.
// Two values per instruction where there is one (packed fp32): the math warps are bound by how much they
// issue (20 instructions per element before, of which 9 here; now 7).
template <bool DIAG, bool DROP>
__device__ __forceinline__ void fb_math16(const uint32_t* sv, const uint32_t* dv, uint32_t* pw, uint32_t* dw,
                                          int r, int col0, float sl2, float lse_l2,
                                          float dlt_s, float scale, float dscale, uint32_t keep16) {
  const uint64_t sl2_2 = f2_bcast(sl2), lse_2 = f2_bcast(-lse_l2), dlt_2 = f2_bcast(-dlt_s);
  const float ms = dscale * scale;
#pragma unroll
  for (int i = 0; i < 16; i += 2) {
    float e0, e1;
    f2_unpack(f2_fma(f2_pack(__uint_as_float(sv[i]), __uint_as_float(sv[i + 1])), sl2_2, lse_2), e0, e1);
    e0 = ex2_fast(e0);
    e1 = ex2_fast(e1);
    if (DIAG) {
      e0 = (col0 + i) <= r ? e0 : 0.f;
      e1 = (col0 + i + 1) <= r ? e1 : 0.f;
    }
    const uint64_t e = f2_pack(e0, e1), dp = f2_pack(__uint_as_float(dv[i]), __uint_as_float(dv[i + 1]));
    if (DROP) {
      const bool k0 = (keep16 >> i) & 1u, k1 = (keep16 >> (i + 1)) & 1u;
      pw[i >> 1] = f2_to_bf16x2(f2_mul(e, f2_pack(k0 ? dscale : 0.f, k1 ? dscale : 0.f)));
      dw[i >> 1] = f2_to_bf16x2(f2_mul(e, f2_fma(dp, f2_pack(k0 ? ms : 0.f, k1 ? ms : 0.f), dlt_2)));
    } else {
      pw[i >> 1] = f2_to_bf16x2(e);
      dw[i >> 1] = f2_to_bf16x2(f2_mul(e, f2_fma(dp, f2_bcast(scale), dlt_2)));
    }
  }
}

__global__ void __launch_bounds__(FB_THREADS, 1)
attn_bwd_fused64_kernel(const __grid_constant__ CUtensorMap tmQKV,
                        const __grid_constant__ CUtensorMap tmDO,
                        const __grid_constant__ CUtensorMap tmDQ, const AttnBwdArgs a) {
  griddep_enter();
  constexpr int HD = 64;
  constexpr uint32_t IDESC_S = make_idesc_bf16(128, 128, 0, 0);
  constexpr uint32_t IDESC_T = make_idesc_bf16(128, HD, 1, 1);
  constexpr uint32_t IDESC_DQ = make_idesc_bf16(128, HD, 0, 1);

  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = smem_raw;
  if (smem_u32(smem) & 1023) {
    if (threadIdx.x == 0) atomicCAS(a.status, 0, ST_BAD_ARGUMENT);
    return;
  }
  uint8_t* sK = smem;
  uint8_t* sV = sK + FB_TILE;
  uint8_t* sQ = sV + FB_TILE;            // 2 stages
  uint8_t* sDO = sQ + 2 * FB_TILE;       // 2 stages
  uint8_t* sP = sDO + 2 * FB_TILE;
  uint8_t* sDS = sP + FB_P;
  uint8_t* sDQ = sDS + FB_P;             // 16 warps x 2 KB staging for the dQ reduce-adds
  uint64_t* bars = reinterpret_cast<uint64_t*>(sDQ + FB_MATH_WARPS * 2048);
  uint64_t* stat_full = bars;
  uint64_t* full = bars + 1;       // 2
  uint64_t* empty = bars + 3;      // 2
  uint64_t* sdp_full = bars + 5;
  uint64_t* sdp_empty = bars + 6;
  uint64_t* pds_full = bars + 7;
  uint64_t* pds_empty = bars + 8;
  uint64_t* dq_full = bars + 9;    // 2
  uint64_t* dq_empty = bars + 11;  // 2
  uint64_t* acc_full = bars + 13;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 14);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = warp_number(), lane = threadIdx.x & 31;
  const int nt = (a.T + 127) / 128;
  const int h = blockIdx.y, b = blockIdx.z;
  const int own = static_cast<int>(blockIdx.x);     // key tile; small index = most query tiles first
  const int n_iter = nt - own;
  const int d_model = a.H * HD;

  if (threadIdx.x == 0) {
    mbar_init(stat_full, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&full[i], 1); mbar_init(&empty[i], 1);
      mbar_init(&dq_full[i], 1); mbar_init(&dq_empty[i], FB_MATH_WARPS);
    }
    mbar_init(sdp_full, 1); mbar_init(sdp_empty, FB_MATH_WARPS);
    mbar_init(pds_full, FB_MATH_WARPS); mbar_init(pds_empty, 1); mbar_init(acc_full, 1);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmQKV);
    tma_prefetch_desc(&tmDO);
    tma_prefetch_desc(&tmDQ);
  }
  if (warp == FB_MMA_WARP) { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tS = tmem_base, tDP = tmem_base + 128, tDV = tmem_base + 256, tDK = tmem_base + 320,
                 tDQ = tmem_base + 384;

  if (warp == FB_TMA_WARP) {
    {
      const uint32_t lead = elect_one();
      const int row_own = b * a.T + own * 128;
      mbar_expect_tx(stat_full, 2 * FB_TILE, lead);
      tma_load_2d(sK, &tmQKV, stat_full, d_model + h * HD, row_own, lead);
      tma_load_2d(sV, &tmQKV, stat_full, 2 * d_model + h * HD, row_own, lead);
      for (int it = 0; it < n_iter; ++it) {
        const int st = it & 1;
        const int row = b * a.T + (own + it) * 128;
        if (!mbar_wait_warp(&empty[st], ((it >> 1) & 1) ^ 1, abort_flag)) {
          *abort_flag = ST_TIMEOUT_EMPTY; if (lead) atomicCAS(a.status, 0, ST_TIMEOUT_EMPTY); break;
        }
        mbar_expect_tx(&full[st], 2 * FB_TILE, lead);
        tma_load_2d(sQ + st * FB_TILE, &tmQKV, &full[st], h * HD, row, lead);
        tma_load_2d(sDO + st * FB_TILE, &tmDO, &full[st], h * HD, row, lead);
      }
    }
  } else if (warp == FB_MMA_WARP) {
    {
      const uint32_t lead = elect_one();
      bool ok = mbar_wait_warp(stat_full, 0, abort_flag);
      const uint32_t k0 = smem_u32(sK), v0 = smem_u32(sV), p0 = smem_u32(sP), ds0 = smem_u32(sDS);
      auto issue_sdp = [&](int it) {
        const int st = it & 1;
        if (!mbar_wait_warp(&full[st], (it >> 1) & 1, abort_flag)) return false;
        if (it > 0 && !mbar_wait_warp(sdp_empty, (it - 1) & 1, abort_flag)) return false;
        tc_fence_after();
        const uint32_t q = smem_u32(sQ + st * FB_TILE), dO = smem_u32(sDO + st * FB_TILE);
#pragma unroll
        for (int k = 0; k < 4; ++k)
          umma_bf16(tS, make_sdesc_sw128(q, k * 32, 16, 1024), make_sdesc_sw128(k0, k * 32, 16, 1024),
                    IDESC_S, k > 0, lead);
#pragma unroll
        for (int k = 0; k < 4; ++k)
          umma_bf16(tDP, make_sdesc_sw128(dO, k * 32, 16, 1024), make_sdesc_sw128(v0, k * 32, 16, 1024),
                    IDESC_S, k > 0, lead);
        umma_commit(sdp_full, lead);
        return true;
      };
      auto issue_acc = [&](int it) {
        const int st = it & 1;
        if (!mbar_wait_warp(pds_full, it & 1, abort_flag)) return false;
        if (it >= 2 && !mbar_wait_warp(&dq_empty[it & 1], ((it - 2) >> 1) & 1, abort_flag)) return false;
        tc_fence_after();
        const uint32_t q = smem_u32(sQ + st * FB_TILE), dO = smem_u32(sDO + st * FB_TILE);
        // dQ_ij = dS K_j first: its consumers (the math warps) can start draining it earliest
#pragma unroll
        for (int k = 0; k < 8; ++k)
          umma_bf16(tDQ + (it & 1) * 64, make_sdesc_sw128(ds0, (k >> 2) * 16384 + (k & 3) * 32, 16, 1024),
                    make_sdesc_sw128(k0, k * 2048, 16384, 1024), IDESC_DQ, k > 0, lead);
        umma_commit(&dq_full[it & 1], lead);
#pragma unroll
        for (int k = 0; k < 8; ++k)
          umma_bf16(tDV, make_sdesc_sw128(p0, k * 2048, 16384, 1024),
                    make_sdesc_sw128(dO, k * 2048, 16384, 1024), IDESC_T, (it > 0 || k > 0), lead);
#pragma unroll
        for (int k = 0; k < 8; ++k)
          umma_bf16(tDK, make_sdesc_sw128(ds0, k * 2048, 16384, 1024),
                    make_sdesc_sw128(q, k * 2048, 16384, 1024), IDESC_T, (it > 0 || k > 0), lead);
        umma_commit(&empty[st], lead);
        umma_commit(pds_empty, lead);
        return true;
      };
      if (ok) ok = issue_sdp(0);
      for (int it = 0; it < n_iter && ok; ++it) {
        if (it + 1 < n_iter) { ok = issue_sdp(it + 1); if (!ok) break; }
        ok = issue_acc(it);
      }
      if (ok) umma_commit(acc_full, lead);
      else { *abort_flag = ST_TIMEOUT_FULL; if (lead) atomicCAS(a.status, 0, ST_TIMEOUT_FULL); }
    }
  } else {
    // ------------------------------------------------------------ math warps
    const int quad = warp & 3, cb = warp >> 2;
    const int r = quad * 32 + lane;
    const uint32_t lane_addr = static_cast<uint32_t>(quad * 32) << 16;
    const float sl2 = a.scale * LOG2E;
    const float dscale = dropout_scale(a.thr16);
    const long long bh = static_cast<long long>(b) * a.H + h;
    uint8_t* my_dq = sDQ + warp * 2048;
    const uint64_t seed = uniform64(a.thr16 ? salted(a.seed, a.salt) : 0);
    bool ok = true;

    // drains dQ tile `it` (rows of query tile own+it, this warp's 16 columns) into the global
    // fp32 accumulator with one TMA reduce-add
    auto drain_dq = [&](int it) {
      if (!mbar_wait_warp(&dq_full[it & 1], (it >> 1) & 1, abort_flag)) return false;
      tc_fence_after();
      uint32_t v[16];
      tmem_ld16(tDQ + (it & 1) * 64 + lane_addr + cb * 16, v);
      if (lane == 0) tma_store_wait_read<0>();
      __syncwarp();
      tmem_ld_wait();
      tc_fence_before();
      // 16 fp32 columns = 64-byte rows, 64B swizzle
      uint8_t* rowp = my_dq + lane * 64;
      const int sw = (lane >> 1) & 3;
#pragma unroll
      for (int c = 0; c < 4; ++c)
        *reinterpret_cast<float4*>(rowp + ((c ^ sw) << 4)) =
            make_float4(__uint_as_float(v[c * 4 + 0]), __uint_as_float(v[c * 4 + 1]),
                        __uint_as_float(v[c * 4 + 2]), __uint_as_float(v[c * 4 + 3]));
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&dq_empty[it & 1]);
        tma_reduce_add_2d(&tmDQ, my_dq, h * HD + cb * 16, b * a.T + (own + it) * 128 + quad * 32);
        tma_store_commit();
      }
      return true;
    };

    for (int it = 0; it < n_iter && ok; ++it) {
      const int qi = own + it;
      const int q_idx = qi * 128 + r;
      const bool q_ok = q_idx < a.T;
      const float lse_l2 = q_ok ? a.lse[bh * a.T + q_idx] * LOG2E : INFINITY;
      const float dlt = q_ok ? a.delta[bh * a.T + q_idx] : 0.f;
      const bool diag = it == 0;
      const uint64_t row_elem0 = (static_cast<uint64_t>(bh) * a.T + q_idx) * a.T + own * 128 + cb * 32;
      uint32_t keep32 = 0xffffffffu;
      if (a.thr16) {
        if (a.drop_mask) {
          keep32 = q_ok && own * 128 + cb * 32 < a.T ? a.drop_mask[row_elem0 >> 5] : 0u;
        } else {
          keep32 = dropout_keep32(seed, a.stream_id, row_elem0 >> 3, a.thr16);
        }
      }
      if (!mbar_wait_warp(sdp_full, it & 1, abort_flag)) { ok = false; break; }
      tc_fence_after();
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) {
        const int col0 = cb * 32 + hf * 16;
        uint32_t sv[16], dv[16];
        tmem_ld16(tS + lane_addr + col0, sv);
        tmem_ld16(tDP + lane_addr + col0, dv);
        tmem_ld_wait();
        if (hf == 1) {
          // S and dP are in registers: handed back before the math of the second half, so the tensor
          // core computes the next pair's under it
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(sdp_empty);
        }
        uint32_t pw[8], dw[8];
        const uint32_t k16 = keep32 >> (hf * 16);
        if (a.thr16) {
          if (diag) fb_math16<true, true>(sv, dv, pw, dw, r, col0, sl2, lse_l2, dlt * a.scale, a.scale, dscale, k16);
          else      fb_math16<false, true>(sv, dv, pw, dw, r, col0, sl2, lse_l2, dlt * a.scale, a.scale, dscale, k16);
        } else {
          if (diag) fb_math16<true, false>(sv, dv, pw, dw, r, col0, sl2, lse_l2, dlt * a.scale, a.scale, dscale, k16);
          else      fb_math16<false, false>(sv, dv, pw, dw, r, col0, sl2, lse_l2, dlt * a.scale, a.scale, dscale, k16);
        }
        // the shared P / dS tiles feed the previous pair's products until pds_empty completes
        if (hf == 0 && it > 0 && !mbar_wait_warp(pds_empty, (it - 1) & 1, abort_flag)) { ok = false; break; }
        const uint32_t poff = (col0 >> 6) * 16384;
#pragma unroll
        for (int g = 0; g < 2; ++g) {
          const uint32_t off = poff + sw128_chunk(r, ((col0 & 63) >> 3) + g);
          *reinterpret_cast<uint4*>(sP + off) = make_uint4(pw[g * 4], pw[g * 4 + 1], pw[g * 4 + 2], pw[g * 4 + 3]);
          *reinterpret_cast<uint4*>(sDS + off) = make_uint4(dw[g * 4], dw[g * 4 + 1], dw[g * 4 + 2], dw[g * 4 + 3]);
        }
      }
      if (!ok) break;
      // one arrival per warp: hundreds of threads arriving on one mbarrier serialise on it
      tc_fence_before();
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(pds_full);
      // the previous pair's dQ tile finished long ago: drain it while the tensor core works
      if (it > 0) ok = drain_dq(it - 1);
    }
    if (ok) ok = drain_dq(n_iter - 1);
    if (ok && !mbar_wait_warp(acc_full, 0, abort_flag)) ok = false;
    if (!ok) { *abort_flag = ST_TIMEOUT_TMEM_FULL; atomicCAS(a.status, 0, ST_TIMEOUT_TMEM_FULL); }
    if (ok) {
      tc_fence_after();
      const int t_idx = own * 128 + r;
      __nv_bfloat16* base = a.dqkv + (static_cast<long long>(b) * a.T + t_idx) * (3 * d_model) + h * HD;
      // 4 chunks of 32 columns: dV chunks 0,1 then dK chunks 0,1; warp group cb takes chunk cb
      const uint32_t tacc = (cb < 2 ? tDV : tDK) + (cb & 1) * 32;
      __nv_bfloat16* dst = base + (cb < 2 ? 2 * d_model : d_model) + (cb & 1) * 32;
      uint32_t v[32];
      tmem_ld32(tacc + lane_addr, v);
      tmem_ld_wait();
      if (t_idx < a.T) {
#pragma unroll
        for (int q4 = 0; q4 < 4; ++q4) {
          uint4 w;
          w.x = pack_bf16x2(__uint_as_float(v[q4 * 8 + 0]), __uint_as_float(v[q4 * 8 + 1]));
          w.y = pack_bf16x2(__uint_as_float(v[q4 * 8 + 2]), __uint_as_float(v[q4 * 8 + 3]));
          w.z = pack_bf16x2(__uint_as_float(v[q4 * 8 + 4]), __uint_as_float(v[q4 * 8 + 5]));
          w.w = pack_bf16x2(__uint_as_float(v[q4 * 8 + 6]), __uint_as_float(v[q4 * 8 + 7]));
          *reinterpret_cast<uint4*>(dst + q4 * 8) = w;
        }
      }
    }
    if (lane == 0) tma_store_wait<0>();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == FB_MMA_WARP) { tc_fence_after(); tmem_dealloc(tmem_base, 512); }
}

// ------------------------------------------------------------------------------------------
// Persistent form of the kernel above: one CTA per SM walks (batch*head) = blockIdx.x,
// blockIdx.x + gridDim.x, ... and, for each, the key tiles 0..nt-1, as ONE pipeline over
// (query tile, key tile) pairs.  K/V are double-buffered across key tiles, the Q/dO ring and the
// S/dP, P/dS and dQ hand-offs run on a pair counter that never restarts, and the end-of-tile work
// of key tile w (last dQ drain, dV/dK read-out and store) runs beside the first pair of key tile w + 1.
// So the per-key-tile prologue (TMEM allocation, barrier set-up, first loads) and tail, which cost
// as much as two pairs in the one-tile-per-CTA kernel, are paid once per CTA.
// Four warps of their own, one per TMEM lane quarter, take the results out: the dQ tile of every pair, and dV / dK
// where a key tile ends.  Done by the math warps between pairs this was 1100 of a pair's 5000 clocks, and these are
// what a pair waits for (the tensor core is done early, nobody waits for it).  us with
// dropout 0.1, before and now: 64 x 512 x 16 heads 258 and 187, 32 x 512 x 20 188 and 137, 37 x 328 x 12 90 and 68,
// 16 x 1000 x 16 267 and 197 (these two draw the keep bits again).

constexpr int FBP_DRAIN_WARPS = 4;
constexpr int FBP_THREADS = FB_THREADS + FBP_DRAIN_WARPS * 32;

struct FbWalk {
  int bh, own, it, nt, bh_end, step;
  int w, g;      // key tiles and pairs done so far by this CTA
  __host__ __device__ __forceinline__ bool valid() const { return bh < bh_end; }
  __host__ __device__ __forceinline__ bool first() const { return it == 0; }
  __host__ __device__ __forceinline__ bool last() const { return it == nt - own - 1; }
  __host__ __device__ __forceinline__ void next() {
    ++g;
    if (++it == nt - own) {
      it = 0; ++w;
      if (++own == nt) { own = 0; bh += step; }
    }
  }
};

// A drain warp's bulk operations on a dQ place are ordered by waits only: groups of one thread may be performed in any
// order, whatever they were issued in.  How many of its latest groups may be under way still
// - when the sum of query tile `own` is read (the diagonal pair of key tile own > 0).  The last addition to it was for the
//   second pair of key tile own - 1; behind that came nt - own - 1 pairs and, before the last of these, that tile's
//   dV / dK, a group each.
__host__ __device__ constexpr int fb_open_at_sum(int nt, int own) { return nt - own >= 3 ? 3 : nt - own == 2 ? 2 : 0; }
// - when key tile own > 0 adds to a query tile (it > 0).  At its first addition everything up to the key tile before is
//   complete: what that one stored (own == 1) or added there comes first, so the sums are always taken in the same order.
//   All that came since is this key tile's diagonal pair (a pair's time ago) and, if this pair is its last, dV / dK.
constexpr int FB_NO_WAIT = -1;
__host__ __device__ constexpr int fb_open_at_add(int it) { return it == 1 ? 1 : FB_NO_WAIT; }

__device__ __forceinline__ void fb_wait_groups(int open) {
  if (open >= 3) tma_store_wait<3>();
  else if (open == 2) tma_store_wait<2>();
  else if (open == 1) tma_store_wait<1>();
  else if (open == 0) tma_store_wait<0>();
}

// RAGGED: T is no multiple of 128; the last 32-row blocks of a sequence are stored row by row
template <bool RAGGED>
__global__ void __launch_bounds__(FBP_THREADS, 1)
attn_bwd_fused64_persistent_kernel(const __grid_constant__ CUtensorMap tmQKV,
                                   const __grid_constant__ CUtensorMap tmDO,
                                   const __grid_constant__ CUtensorMap tmDQ,
                                   const __grid_constant__ CUtensorMap tmOut, const AttnBwdArgs a) {
  griddep_enter();
  constexpr int HD = 64;
  constexpr uint32_t IDESC_S = make_idesc_bf16(128, 128, 0, 0);
  constexpr uint32_t IDESC_T = make_idesc_bf16(128, HD, 1, 1);
  constexpr uint32_t IDESC_DQ = make_idesc_bf16(128, HD, 0, 1);

  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = smem_raw;
  if (smem_u32(smem) & 1023) {
    if (threadIdx.x == 0) atomicCAS(a.status, 0, ST_BAD_ARGUMENT);
    return;
  }
  uint8_t* sK = smem;                    // 2 stages
  uint8_t* sV = sK + 2 * FB_TILE;        // 2 stages
  uint8_t* sQ = sV + 2 * FB_TILE;        // 2 stages
  uint8_t* sDO = sQ + 2 * FB_TILE;       // 2 stages
  uint8_t* sP = sDO + 2 * FB_TILE;
  uint8_t* sDS = sP + FB_P;
  uint8_t* sDQ = sDS + FB_P;             // staging of the drain warps, 8 KB each
  uint64_t* bars = reinterpret_cast<uint64_t*>(sDQ + FBP_DRAIN_WARPS * 8192);
  uint64_t* kv_full = bars;        // 2
  uint64_t* kv_empty = bars + 2;   // 2
  uint64_t* full = bars + 4;       // 2
  uint64_t* empty = bars + 6;      // 2
  uint64_t* sdp_full = bars + 8;
  uint64_t* sdp_empty = bars + 9;
  uint64_t* pds_full = bars + 10;
  uint64_t* pds_empty = bars + 11;
  uint64_t* dq_full = bars + 12;   // 2
  uint64_t* dq_empty = bars + 14;  // 2
  uint64_t* acc_full = bars + 16;
  uint64_t* acc_empty = bars + 17;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 18);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = warp_number(), lane = threadIdx.x & 31;
  const int nt = (a.T + 127) / 128;
  const int d_model = a.H * HD;

  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(&kv_full[i], 1); mbar_init(&kv_empty[i], 1);
      mbar_init(&full[i], 1); mbar_init(&empty[i], 1);
      mbar_init(&dq_full[i], 1); mbar_init(&dq_empty[i], FBP_DRAIN_WARPS);
    }
    mbar_init(sdp_full, 1); mbar_init(sdp_empty, FB_MATH_WARPS);
    mbar_init(pds_full, FB_MATH_WARPS); mbar_init(pds_empty, 1);
    mbar_init(acc_full, 1); mbar_init(acc_empty, FBP_DRAIN_WARPS);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmQKV);
    tma_prefetch_desc(&tmDO);
    tma_prefetch_desc(&tmDQ);
    tma_prefetch_desc(&tmOut);
  }
  if (warp == FB_MMA_WARP) { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tS = tmem_base, tDP = tmem_base + 128, tDV = tmem_base + 256, tDK = tmem_base + 320,
                 tDQ = tmem_base + 384;
  FbWalk start;
  start.bh = static_cast<int>(blockIdx.x); start.own = 0; start.it = 0; start.nt = nt;
  start.bh_end = a.B * a.H; start.step = static_cast<int>(gridDim.x); start.w = 0; start.g = 0;

  if (warp == FB_TMA_WARP) {
    {
      const uint32_t lead = elect_one();
      for (FbWalk p = start; p.valid(); p.next()) {
        const int b = p.bh / a.H, h = p.bh % a.H;
        if (p.first()) {
          const int s = p.w & 1;
          if (!mbar_wait_warp(&kv_empty[s], ((p.w >> 1) & 1) ^ 1, abort_flag)) {
            *abort_flag = ST_TIMEOUT_EMPTY; if (lead) atomicCAS(a.status, 0, ST_TIMEOUT_EMPTY); break;
          }
          const int row_own = b * a.T + p.own * 128;
          mbar_expect_tx(&kv_full[s], 2 * FB_TILE, lead);
          tma_load_2d(sK + s * FB_TILE, &tmQKV, &kv_full[s], d_model + h * HD, row_own, lead);
          tma_load_2d(sV + s * FB_TILE, &tmQKV, &kv_full[s], 2 * d_model + h * HD, row_own, lead);
        }
        const int st = p.g & 1;
        const int row = b * a.T + (p.own + p.it) * 128;
        if (!mbar_wait_warp(&empty[st], ((p.g >> 1) & 1) ^ 1, abort_flag)) {
          *abort_flag = ST_TIMEOUT_EMPTY; if (lead) atomicCAS(a.status, 0, ST_TIMEOUT_EMPTY); break;
        }
        mbar_expect_tx(&full[st], 2 * FB_TILE, lead);
        tma_load_2d(sQ + st * FB_TILE, &tmQKV, &full[st], h * HD, row, lead);
        tma_load_2d(sDO + st * FB_TILE, &tmDO, &full[st], h * HD, row, lead);
      }
    }
  } else if (warp == FB_MMA_WARP) {
    {
      const uint32_t lead = elect_one();
      const uint32_t p0 = smem_u32(sP), ds0 = smem_u32(sDS);
      auto issue_sdp = [&](const FbWalk& p) {
        const int st = p.g & 1;
        if (p.first() && !mbar_wait_warp(&kv_full[p.w & 1], (p.w >> 1) & 1, abort_flag)) return false;
        if (!mbar_wait_warp(&full[st], (p.g >> 1) & 1, abort_flag)) return false;
        if (p.g > 0 && !mbar_wait_warp(sdp_empty, (p.g - 1) & 1, abort_flag)) return false;
        tc_fence_after();
        const uint32_t k0 = smem_u32(sK + (p.w & 1) * FB_TILE), v0 = smem_u32(sV + (p.w & 1) * FB_TILE);
        const uint32_t q = smem_u32(sQ + st * FB_TILE), dO = smem_u32(sDO + st * FB_TILE);
#pragma unroll
        for (int k = 0; k < 4; ++k)
          umma_bf16(tS, make_sdesc_sw128(q, k * 32, 16, 1024), make_sdesc_sw128(k0, k * 32, 16, 1024),
                    IDESC_S, k > 0, lead);
#pragma unroll
        for (int k = 0; k < 4; ++k)
          umma_bf16(tDP, make_sdesc_sw128(dO, k * 32, 16, 1024), make_sdesc_sw128(v0, k * 32, 16, 1024),
                    IDESC_S, k > 0, lead);
        umma_commit(sdp_full, lead);
        return true;
      };
      auto issue_acc = [&](const FbWalk& p) {
        const int st = p.g & 1;
        if (!mbar_wait_warp(pds_full, p.g & 1, abort_flag)) return false;
        if (p.g >= 2 && !mbar_wait_warp(&dq_empty[p.g & 1], ((p.g - 2) >> 1) & 1, abort_flag)) return false;
        // dV / dK of the previous key tile must have been read out before they are overwritten
        if (p.first() && p.w > 0 && !mbar_wait_warp(acc_empty, (p.w - 1) & 1, abort_flag)) return false;
        tc_fence_after();
        const uint32_t k0 = smem_u32(sK + (p.w & 1) * FB_TILE);
        const uint32_t q = smem_u32(sQ + st * FB_TILE), dO = smem_u32(sDO + st * FB_TILE);
#pragma unroll
        for (int k = 0; k < 8; ++k)
          umma_bf16(tDQ + (p.g & 1) * 64, make_sdesc_sw128(ds0, (k >> 2) * 16384 + (k & 3) * 32, 16, 1024),
                    make_sdesc_sw128(k0, k * 2048, 16384, 1024), IDESC_DQ, k > 0, lead);
        umma_commit(&dq_full[p.g & 1], lead);
#pragma unroll
        for (int k = 0; k < 8; ++k)
          umma_bf16(tDV, make_sdesc_sw128(p0, k * 2048, 16384, 1024),
                    make_sdesc_sw128(dO, k * 2048, 16384, 1024), IDESC_T, (p.it > 0 || k > 0), lead);
#pragma unroll
        for (int k = 0; k < 8; ++k)
          umma_bf16(tDK, make_sdesc_sw128(ds0, k * 2048, 16384, 1024),
                    make_sdesc_sw128(q, k * 2048, 16384, 1024), IDESC_T, (p.it > 0 || k > 0), lead);
        umma_commit(&empty[st], lead);
        umma_commit(pds_empty, lead);
        if (p.last()) {
          umma_commit(acc_full, lead);                 // dV / dK of this key tile complete
          umma_commit(&kv_empty[p.w & 1], lead);       // and its K / V stage is free
        }
        return true;
      };
      FbWalk cur = start, nxt = start;
      bool ok = true;
      if (cur.valid()) { nxt.next(); ok = issue_sdp(cur); }
      while (ok && cur.valid()) {
        if (nxt.valid()) { ok = issue_sdp(nxt); if (!ok) break; }
        ok = issue_acc(cur);
        cur = nxt;
        if (nxt.valid()) nxt.next();
      }
      if (!ok) { *abort_flag = ST_TIMEOUT_FULL; if (lead) atomicCAS(a.status, 0, ST_TIMEOUT_FULL); }
    }
  } else if (warp > FB_MMA_WARP) {
    // ----------------------------------------------------------- drain warps
    const int quad = warp & 3, r = quad * 32 + lane;
    const uint32_t lane_addr = static_cast<uint32_t>(quad * 32) << 16;
    // Staging: two tiles of 32 rows of 128 bytes (128B swizzle), 32 fp32 or 64 bf16 columns.  A lane reads and
    // writes its own row.
    uint8_t* stg = sDQ + quad * 8192;
    uint8_t* my_row = stg + lane * 128;
    auto at = [&](int k) { return ((k ^ (lane & 7)) << 4); };           // 16-byte chunk k of it
    bool ok = true;

    // The dQ sums of the slice that this CTA works on live in a place of its own in dq_acc (nt - 1 tiles of 128
    // rows of 64 columns: query tile 0 has one pair and needs none) and nowhere else, so 148 slices stay in L2 instead of every slice passing through
    // memory twice, and no pass converts or clears them: key tile 0 stores its contributions, later ones
    // add, and the last one of a query tile (its diagonal pair) reads the sum back, adds its own part from
    // TMEM and stores bf16 into dQKV.  The same warp does all of it for its rows.
    const int s_row0 = (static_cast<int>(blockIdx.x) * (nt - 1) - 1) * 128 + quad * 32;    // of query tile 0, if it had one
    // rows past the end of a sequence are the next one's: P and dS, and so dQ, dK and dV, are zeros there
    auto whole_rows = [&](int row) { return !RAGGED || row + 32 <= a.T; };
    // adds the column sums of a staged tile of 64 bf16 columns to dst: a lane takes two columns
    auto add_colsum = [&](const uint8_t* tile, float* dst) {
      uint64_t sum[4] = {0ull, 0ull, 0ull, 0ull};
#pragma unroll
      for (int k = 0; k < 32; ++k) {
        const uint32_t w = *reinterpret_cast<const uint32_t*>(tile + k * 128 + (((lane >> 2) ^ (k & 7)) << 4) + (lane & 3) * 4);
        sum[k & 3] = f2_add(sum[k & 3], f2_pack(bf16_lo(w), bf16_hi(w)));
      }
      float s0, s1;
      f2_unpack(f2_add(f2_add(sum[0], sum[1]), f2_add(sum[2], sum[3])), s0, s1);
      asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(dst + lane * 2), "f"(s0), "f"(s1) : "memory");
    };

    // The sum so far of query tile `own`, into the staging tiles, while
    // the pair that completes it is still computed: behind it, the wait for this warp's earlier contributions and
    // the trip to L2 were 6000 of 7500 clocks.
    auto fetch_sum = [&](int own) {
      if (lane == 0) {
        fb_wait_groups(fb_open_at_sum(nt, own)); // the additions are complete,
        tma_store_wait_read<0>();                // and the staging tiles free
        asm volatile("fence.proxy.async;" ::: "memory");
      }
      __syncwarp();
      const float* src = a.dq_acc + (static_cast<long long>(s_row0) + own * 128) * HD;
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const int row = i * 2 + (lane >> 4), k = lane & 15;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;"
                     ::"r"(smem_u32(stg + (k >> 3) * 4096 + row * 128 + (((k & 7) ^ (row & 7)) << 4))), "l"(src + row * HD + k * 4)
                     : "memory");
      }
    };
    // the dQ tile of pair g (query tile own + it of head h of sequence b)
    auto drain_dq = [&](int g, int b, int h, int own, int it) {
      const bool last = it == 0, summed = last && own > 0;
      if (summed) fetch_sum(own);
      const bool there = mbar_wait_warp(&dq_full[g & 1], (g >> 1) & 1, abort_flag);
      asm volatile("cp.async.wait_all;" ::: "memory");
      if (!there) return false;
      tc_fence_after();
      if (lane == 0 && !summed) tma_store_wait_read<0>();
      __syncwarp();
      const int qrow = (own + it) * 128;
      const bool rows_whole = whole_rows(qrow + quad * 32);            // warp-uniform
#pragma unroll 1
      for (int hf = 0; hf < 2; ++hf) {           // 32 columns
        uint32_t v[32];
        tmem_ld32(tDQ + (g & 1) * 64 + lane_addr + hf * 32, v);
        float4 x[8];                             // the sum so far
#pragma unroll
        for (int k = 0; k < 8; ++k)
          x[k] = summed ? *reinterpret_cast<const float4*>(my_row + hf * 4096 + at(k)) : make_float4(0.f, 0.f, 0.f, 0.f);
        tmem_ld_wait();
        if (hf == 1) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&dq_empty[g & 1]);
        }
        if (last) {
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const float4 lo = x[2 * k], hi = x[2 * k + 1];
            const uint32_t* f = v + k * 8;
            auto f_ = [&](int i) { return __uint_as_float(f[i]); };
            const uint4 w = make_uint4(pack_bf16x2(f_(0) + lo.x, f_(1) + lo.y), pack_bf16x2(f_(2) + lo.z, f_(3) + lo.w),
                                       pack_bf16x2(f_(4) + hi.x, f_(5) + hi.y), pack_bf16x2(f_(6) + hi.z, f_(7) + hi.w));
            *reinterpret_cast<uint4*>(my_row + at(hf * 4 + k)) = w;
            if (!rows_whole && qrow + r < a.T)
              *reinterpret_cast<uint4*>(a.dqkv + (static_cast<long long>(b) * a.T + qrow + r) * (3 * d_model) + h * HD + hf * 32 + k * 8) = w;
          }
        } else {
#pragma unroll
          for (int k = 0; k < 8; ++k)
            *reinterpret_cast<uint4*>(my_row + hf * 4096 + at(k)) = make_uint4(v[k * 4], v[k * 4 + 1], v[k * 4 + 2], v[k * 4 + 3]);
        }
      }
      // the first store into the slice's place: behind the reads of what was there for the slice before
      if (own == 0 && it == 1) asm volatile("fence.proxy.async;" ::: "memory");
      else fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        if (last) {
          if (rows_whole) tma_store_2d(&tmOut, stg, h * HD, b * a.T + qrow + quad * 32);
        } else if (own == 0) {
          tma_store_2d(&tmDQ, stg, 0, s_row0 + qrow);
          tma_store_2d(&tmDQ, stg + 4096, 32, s_row0 + qrow);
        } else {
          fb_wait_groups(fb_open_at_add(it));
          tma_reduce_add_2d(&tmDQ, stg, 0, s_row0 + qrow);
          tma_reduce_add_2d(&tmDQ, stg + 4096, 32, s_row0 + qrow);
        }
        tma_store_commit();
      }
      if (last && a.dbias) add_colsum(stg, a.dbias + h * HD);
      return true;
    };
    // reads the finished dV / dK of key tile w out of TMEM, frees them, and stores them
    auto finish_tile = [&](int w, int b, int h, int own) {
      if (!mbar_wait_warp(acc_full, w & 1, abort_flag)) return false;
      tc_fence_after();
      const bool rows_whole = whole_rows(own * 128 + quad * 32);       // warp-uniform
      const int t_idx = own * 128 + r;
      // dV, then dK, one TMA store each.  (Plain stores of 64-byte row pieces 6 KB apart kept the load/store unit
      // busy for thousands of cycles per key tile and delayed every other warp's shared-memory traffic with them.)
#pragma unroll 1
      for (int m = 0; m < 2; ++m) {
        uint32_t w[32];                                                // 64 columns as bf16 pairs
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          uint32_t v[32];
          tmem_ld32((m ? tDK : tDV) + c * 32 + lane_addr, v);
          tmem_ld_wait();
#pragma unroll
          for (int k = 0; k < 16; ++k) w[c * 16 + k] = pack_bf16x2(__uint_as_float(v[2 * k]), __uint_as_float(v[2 * k + 1]));
        }
        if (m == 1) tc_fence_before();
        else if (lane == 0) tma_store_wait_read<0>();                  // the staging tiles are free
        __syncwarp();                                                  // (and their column sums taken)
        if (m == 1 && lane == 0) mbar_arrive(acc_empty);
        const int col = (m ? d_model : 2 * d_model) + h * HD;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const uint4 wv = make_uint4(w[k * 4], w[k * 4 + 1], w[k * 4 + 2], w[k * 4 + 3]);
          *reinterpret_cast<uint4*>(my_row + m * 4096 + at(k)) = wv;
          if (!rows_whole && t_idx < a.T)
            *reinterpret_cast<uint4*>(a.dqkv + (static_cast<long long>(b) * a.T + t_idx) * (3 * d_model) + col + k * 8) = wv;
        }
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        if (rows_whole) {
          tma_store_2d(&tmOut, stg, 2 * d_model + h * HD, b * a.T + own * 128 + quad * 32);
          tma_store_2d(&tmOut, stg + 4096, d_model + h * HD, b * a.T + own * 128 + quad * 32);
        }
        tma_store_commit();
      }
      if (a.dbias) {
        add_colsum(stg, a.dbias + 2 * d_model + h * HD);
        add_colsum(stg + 4096, a.dbias + d_model + h * HD);
      }
      return true;
    };
    int b = 0, h = 0;
    for (FbWalk p = start; p.valid() && ok; p.next()) {
      if (p.it == 0 && p.own == 0) { b = p.bh / a.H; h = p.bh - b * a.H; }
      // dV / dK first: the next key tile's products wait for their place, dQ has two.  (Slices of one tile are bound
      // by these warps, which would only wait for dV / dK.)
      if (nt == 1) ok = drain_dq(p.g, b, h, p.own, p.it);
      if (ok && p.last()) ok = finish_tile(p.w, b, h, p.own);
      if (ok && nt > 1) ok = drain_dq(p.g, b, h, p.own, p.it);
      __syncwarp();                                // the staging tiles have been read by all lanes
    }
    if (ok && start.valid() && nt > 1) {
      // hand the accumulator back all zero (query tile 0 never went through it)
      if (lane == 0) tma_store_wait_read<0>();
      __syncwarp();
#pragma unroll
      for (int k = 0; k < 8; ++k) *reinterpret_cast<float4*>(my_row + k * 16) = make_float4(0.f, 0.f, 0.f, 0.f);
      asm volatile("fence.proxy.async;" ::: "memory");
      __syncwarp();
      if (lane == 0) {
        for (int i = 1; i < nt; ++i)
          for (int hf = 0; hf < 2; ++hf) tma_store_2d(&tmDQ, stg, hf * 32, s_row0 + i * 128);
        tma_store_commit();
      }
    }
    if (!ok) { *abort_flag = ST_TIMEOUT_TMEM_FULL; atomicCAS(a.status, 0, ST_TIMEOUT_TMEM_FULL); }
    if (lane == 0) tma_store_wait<0>();
  } else {
    // ------------------------------------------------------------ math warps
    const int quad = warp & 3, cb = warp >> 2;
    const int r = quad * 32 + lane;
    const uint32_t lane_addr = static_cast<uint32_t>(quad * 32) << 16;
    const float sl2 = a.scale * LOG2E;
    const float dscale = dropout_scale(a.thr16);
    const uint64_t seed = uniform64(a.thr16 ? salted(a.seed, a.salt) : 0);
    bool ok = true;

    // per-row inputs of a pair: log-sum-exp, delta and the 32 dropout keep bits of this thread's
    // columns.  They are fetched one pair ahead so their latency never sits in the pair's chain.
    // Addresses advance by fixed strides from one query tile to the next, so they are rebuilt from
    // the indices only at the first pair of a key tile.
    long long row_off = 0;          // (batch*head) * T + query index of this thread's row
    long long keep_off = 0;         // word index of its 32 keep bits
    // (fetch only issues the loads: no arithmetic on the loaded values here, so nothing waits for
    // them before the next pair needs them)
    auto fetch = [&](const FbWalk& w, float& lse_raw, float& dlt, uint32_t& keep32) {
      const int q_idx = (w.own + w.it) * 128 + r;
      const bool q_ok = q_idx < a.T;
      if (w.it == 0) {
        row_off = static_cast<long long>(w.bh) * a.T + q_idx;
        keep_off = (row_off * a.T + w.own * 128 + cb * 32) >> 5;
      } else {
        row_off += 128;
        keep_off += 4ll * a.T;      // 128 rows of T / 32 words
      }
      lse_raw = INFINITY;
      dlt = 0.f;
      if (q_ok) { lse_raw = a.lse[row_off]; dlt = a.delta[row_off]; }
      keep32 = 0xffffffffu;
      if (a.thr16) {
        if (a.drop_mask) {
          keep32 = 0u;
          if (q_ok && (!RAGGED || w.own * 128 + cb * 32 < a.T)) keep32 = a.drop_mask[keep_off];
        } else {
          const uint64_t row_elem0 = static_cast<uint64_t>(row_off) * a.T + w.own * 128 + cb * 32;
          keep32 = dropout_keep32(seed, a.stream_id, row_elem0 >> 3, a.thr16);
        }
      }
    };
    FbWalk p = start;
    float lse_raw = 0.f, dlt = 0.f;
    uint32_t keep32 = 0xffffffffu;
    if (p.valid()) fetch(p, lse_raw, dlt, keep32);
    for (; p.valid() && ok; p.next()) {
      const bool diag = p.it == 0;
      float n_lse = 0.f, n_dlt = 0.f;
      uint32_t n_keep = 0xffffffffu;
      {
        FbWalk q = p;
        q.next();
        if (q.valid()) fetch(q, n_lse, n_dlt, n_keep);
      }
      if (!mbar_wait_warp(sdp_full, p.g & 1, abort_flag)) { ok = false; break; }
      tc_fence_after();
      const float lse_l2 = lse_raw * LOG2E;          // +inf for rows outside the sequence
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) {
        const int col0 = cb * 32 + hf * 16;
        uint32_t sv[16], dv[16];
        tmem_ld16(tS + lane_addr + col0, sv);
        tmem_ld16(tDP + lane_addr + col0, dv);
        tmem_ld_wait();
        if (hf == 1) {
          // S and dP are in registers: handed back before the math of the second half, so the tensor
          // core computes the next pair's under it
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(sdp_empty);
        }
        uint32_t pw[8], dw[8];
        const uint32_t k16 = keep32 >> (hf * 16);
        if (a.thr16) {
          if (diag) fb_math16<true, true>(sv, dv, pw, dw, r, col0, sl2, lse_l2, dlt * a.scale, a.scale, dscale, k16);
          else      fb_math16<false, true>(sv, dv, pw, dw, r, col0, sl2, lse_l2, dlt * a.scale, a.scale, dscale, k16);
        } else {
          if (diag) fb_math16<true, false>(sv, dv, pw, dw, r, col0, sl2, lse_l2, dlt * a.scale, a.scale, dscale, k16);
          else      fb_math16<false, false>(sv, dv, pw, dw, r, col0, sl2, lse_l2, dlt * a.scale, a.scale, dscale, k16);
        }
        if (hf == 0) {
          // the shared P / dS tiles feed the previous pair's dV / dK / dQ products until
          // pds_empty completes; the first half of this pair's math has run under them
          if (p.g > 0 && !mbar_wait_warp(pds_empty, (p.g - 1) & 1, abort_flag)) { ok = false; break; }
        }
        const uint32_t poff = (col0 >> 6) * 16384;
#pragma unroll
        for (int g2 = 0; g2 < 2; ++g2) {
          const uint32_t off = poff + sw128_chunk(r, ((col0 & 63) >> 3) + g2);
          *reinterpret_cast<uint4*>(sP + off) = make_uint4(pw[g2 * 4], pw[g2 * 4 + 1], pw[g2 * 4 + 2], pw[g2 * 4 + 3]);
          *reinterpret_cast<uint4*>(sDS + off) = make_uint4(dw[g2 * 4], dw[g2 * 4 + 1], dw[g2 * 4 + 2], dw[g2 * 4 + 3]);
        }
      }
      if (!ok) break;
      tc_fence_before();
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(pds_full);
      lse_raw = n_lse; dlt = n_dlt; keep32 = n_keep;
    }
    if (!ok) { *abort_flag = ST_TIMEOUT_TMEM_FULL; atomicCAS(a.status, 0, ST_TIMEOUT_TMEM_FULL); }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == FB_MMA_WARP) { tc_fence_after(); tmem_dealloc(tmem_base, 512); }
}


// dqkv[:, 0:d] = bf16(dq_acc).  A block walks whole rows (thread = one float4 column group), so
// every access is a contiguous row segment.  The accumulator is cleared by a separate memset:
// overwriting each element right after loading it in the same kernel measured ten times slower
// on B200 than the read-only conversion plus a memset.
__global__ void __launch_bounds__(256)
attn_dq_convert_kernel(const float* __restrict__ acc, __nv_bfloat16* __restrict__ dqkv, int rows, int d) {
  griddep_enter();
  const int d4 = d >> 2;
  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    const float4* src = reinterpret_cast<const float4*>(acc + static_cast<long long>(row) * d);
    uint2* dst = reinterpret_cast<uint2*>(dqkv + static_cast<long long>(row) * 3 * d);
    for (int c4 = threadIdx.x; c4 < d4; c4 += 256) {
      const float4 v = src[c4];
      uint2 o;
      o.x = pack_bf16x2(v.x, v.y);
      o.y = pack_bf16x2(v.z, v.w);
      dst[c4] = o;
    }
  }
}

// 0 = choose by problem shape, 1 = one key tile per CTA, 2 = persistent walk
static int g_attn_bwd_schedule = -1;
static int attn_bwd_schedule_mode() {
  if (g_attn_bwd_schedule < 0) {
    const char* v = getenv("AB_ATTN_BWD_SCHEDULE");
    g_attn_bwd_schedule = (v && v[0] >= '0' && v[0] <= '2') ? v[0] - '0' : 0;
  }
  return g_attn_bwd_schedule;
}

// The walk hands whole slices to CTAs (each has a place for the sums of one in dq_acc: nt - 1 tiles of 128 rows, fewer
// than T); few, long ones leave SMs idle, which the grid of key tiles does not.  us, from launches of 1 to 320 slices
// of 1 to 8 tiles in a replayed graph: a slice of nt (nt + 1) / 2 pairs of tiles takes the walk 2.2 a pair and 8 in
// all; the grid 12 with the conversion, clearing and column sums behind it, and the longer of its longest CTA (1.7 a
// query tile) and of all its CTAs' work (4 a pair, one and a half pairs' worth per key tile to start and end).  Of the 190 sizes
// measured none loses more than 3 % to the other form.  Grid and walk: 16 slices of 1 tile 14.8 and 7.7, of 2 17.6 and
// 14.8, of 3 19.9 and 21.7, of 4 22.5 and 30; 32 of 4 26 and 30; 148 of 2 36 and 17, of 4 73 and 33; 200 of 1000 keys
// 244 and 186.
static bool fb_walks(int bh, int nt, int sms) {
  const double slice = 0.5 * nt * (nt + 1);
  const double walk_us = 8.0 + 2.2 * ((bh + sms - 1) / sms) * slice;
  const double grid_us = 12.0 + std::max(1.7 * nt, 4.0 * bh * (slice + 1.5 * nt) / sms);
  return walk_us <= grid_us;
}

int launch_attn_bwd_fused64(const CUtensorMap& tq, const CUtensorMap& td, const AttnBwdArgs& a,
                            int* launched, cudaStream_t stream) {
  CUtensorMap tdq;
  const long long rows = static_cast<long long>(a.B) * a.T;
  const int d = a.H * 64;
  int rc = make_tmap_2d_sw(&tdq, a.dq_acc, rows, d, d, 32, 16, 4, 64);
  if (rc) return rc;
  const int mode = attn_bwd_schedule_mode();
  const bool ragged = (a.T & 127) != 0;
  int sms = 0;
  if (const cudaError_t e = device_sms(&sms)) return (int)e;
  const int bh = a.B * a.H, ctas = bh < sms ? bh : sms, nt = (a.T + 127) / 128;
  if (mode == 1 || (mode == 0 && !fb_walks(bh, nt, sms))) {
    constexpr int SMEM = 6 * FB_TILE + 2 * FB_P + FB_MATH_WARPS * 2048 + 256;
    static PerDeviceOnce attr;
    if (attr.first_use_on_device()) {
      cudaError_t e = cudaFuncSetAttribute(attn_bwd_fused64_kernel,
                                           cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
      if (e != cudaSuccess) return (int)e;
      attr.mark_device();
    }
    dim3 grid((a.T + 127) / 128, a.H, a.B);
    launch_chained(attn_bwd_fused64_kernel, dim3(grid), dim3(FB_THREADS), SMEM, stream, tq, td, tdq, a);
    ++*launched;
  } else {
    constexpr int SMEM = 8 * FB_TILE + 2 * FB_P + FBP_DRAIN_WARPS * 8192 + 256;
    auto kern = ragged ? attn_bwd_fused64_persistent_kernel<true> : attn_bwd_fused64_persistent_kernel<false>;
    static PerDeviceOnce attr[2];
    if (attr[ragged].first_use_on_device()) {
      cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
      if (e != cudaSuccess) return (int)e;
      attr[ragged].mark_device();
    }
    CUtensorMap tout;     // the packed dQKV activation, boxes of 32 rows x 64 columns
    rc = make_tmap_2d_sw(&tout, a.dqkv, rows, 3 * d, 3 * d, 32, 64, 2, 128);
    if (rc) return rc;
    CUtensorMap tplace;   // dq_acc as rows of 64 columns, boxes of 32 rows x 32 columns
    rc = make_tmap_2d_sw(&tplace, a.dq_acc, rows * a.H, 64, 64, 32, 32, 4, 128);
    if (rc) return rc;
    launch_chained(kern, dim3(ctas), dim3(FBP_THREADS), SMEM, stream, tq, td, tplace, tout, a);
    ++*launched;
    return (int)cudaGetLastError();                  // dQ, its bias sums and the clearing are done
  }
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return (int)e;
  launch_chained(attn_dq_convert_kernel, dim3(148 * 16), dim3(256), 0, stream, a.dq_acc, a.dqkv, (int)rows, d);
  ++*launched;
  e = cudaGetLastError();
  if (e != cudaSuccess) return (int)e;
  e = cudaMemsetAsync(a.dq_acc, 0, sizeof(float) * rows * d, stream);
  if (e != cudaSuccess || !a.dbias) return (int)e;
  ++*launched;
  return ab_colsum_bf16(a.dqkv, 3 * d, (int)rows, 3 * d, a.dbias, nullptr, stream);
}

}  // namespace ab

// Schedule of the head_dim-64 backward: 0 = by problem shape (default; also read once from the
// environment variable AB_ATTN_BWD_SCHEDULE), 1 = one key tile per CTA, 2 = persistent walk.
extern "C" int ab_attn_bwd_schedule(int mode) {
  if (mode < 0 || mode > 2) return -1;
  ab::g_attn_bwd_schedule = mode;
  return 0;
}

// For tests: whether schedule 0 walks `slices` (batch, head) slices of T keys on a GPU of `sms` SMs
extern "C" int ab_attn_bwd_walks(int slices, int T, int sms) { return ab::fb_walks(slices, (T + 127) / 128, sms); }

// For tests: what a drain warp of the walk does to the dQ places over `slices` slices of nt tiles, in its order; four
// numbers each: what (0 store, 1 add, 2 read, 3 dQ out, 4 dV / dK out; all but reads are a bulk group), slice, query tile (of
// 3 and 4: 0), and how many of the groups before may be under way still (-1: any number).  Returns how many (no
// more than `room` are written).
extern "C" int ab_attn_bwd_walk_order(int nt, int slices, int* out, int room) {
  using namespace ab;
  int n = 0;
  auto put = [&](int what, int slice, int tile, int open) {
    if (n < room) { out[4 * n] = what; out[4 * n + 1] = slice; out[4 * n + 2] = tile; out[4 * n + 3] = open; }
    ++n;
  };
  auto drain_dq = [&](const FbWalk& p) {
    if (p.it == 0 && p.own > 0) put(2, p.bh, p.own, fb_open_at_sum(nt, p.own));
    if (p.it == 0) put(3, p.bh, 0, FB_NO_WAIT);
    else if (p.own == 0) put(0, p.bh, p.it, FB_NO_WAIT);
    else put(1, p.bh, p.own + p.it, fb_open_at_add(p.it));
  };
  FbWalk p = {};
  p.nt = nt; p.bh_end = slices; p.step = 1;
  for (; p.valid(); p.next()) {
    if (nt == 1) drain_dq(p);
    if (p.last()) put(4, p.bh, 0, FB_NO_WAIT);
    if (nt > 1) drain_dq(p);
  }
  for (int i = 1; i < nt; ++i) put(0, slices, i, FB_NO_WAIT);      // handed back all zero
  return n;
}

// Stand-alone entry to the dQ conversion (bf16 copy into the packed dQKV activation, then clear).
extern "C" int ab_attn_dq_convert(float* acc, void* dqkv, int rows, int d, cudaStream_t stream) {
  ab::launch_chained(ab::attn_dq_convert_kernel, dim3(148 * 16), dim3(256), 0, stream, acc, (__nv_bfloat16*)dqkv, rows, d);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return (int)e;
  return (int)cudaMemsetAsync(acc, 0, sizeof(float) * (size_t)rows * d, stream);
}
