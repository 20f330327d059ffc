// LayerNorm / RMSNorm forward and backward for the fp32 residual stream.
//
// forward : x fp32 [M,d] -> y bf16 [M,d] (the A operand of the next GEMM), mean/rstd fp32 [M]
// backward: dy bf16 (+ optional rank-2 term from the scalar heads) -> dx fp32, added to the
//           incoming residual gradient; optionally also emits the bf16, dropout-masked copy of
//           dx that the previous branch's projection GEMMs consume, and accumulates
//           dgamma/dbeta into the fp32 gradient buffers with one atomic per column per block.
// Forward: one warp owns one row; a lane owns float4 columns lane*4 + 128*i.  Backward: see ln_bwd_kernel.
#include "ptx.cuh"

namespace ab {

constexpr int LN_WARPS = 8;

// NV = d / 128 float4s per lane, known at compile time: with a bound checked per float4 every load waited for
// the one before it.  AHEAD (dependent launches of a few hundred rows whose caller says that the kernel before does not
// write gamma and beta): these, which may lie in memory, are fetched while that kernel is still running.
template <int NV, bool AHEAD>
__global__ void __launch_bounds__(LN_WARPS * 32)
ln_fwd_kernel(const float* __restrict__ x, const float* __restrict__ gamma,
              const float* __restrict__ beta, __nv_bfloat16* __restrict__ y,
              float* __restrict__ mean_out, float* __restrict__ rstd_out, int M, float eps, int rms) {
  constexpr int d = NV * 128;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  if (threadIdx.x == 0) griddep_launch_dependents();   // a dependent GEMM may start fetching its weights
  float4 g[NV], b[NV];
  auto fetch_weights = [&]() {
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      g[i] = __ldg(reinterpret_cast<const float4*>(gamma) + lane + 32 * i);
      b[i] = beta ? __ldg(reinterpret_cast<const float4*>(beta) + lane + 32 * i) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  };
  if (AHEAD) fetch_weights();
  griddep_wait();       // launched as a dependent itself: x comes from the kernel before (no-op otherwise)

  for (int row = blockIdx.x * warps + warp; row < M; row += gridDim.x * warps) {
    const float4* xr = reinterpret_cast<const float4*>(x + (long long)row * d);
    float4 v[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) v[i] = xr[lane + 32 * i];
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) s += v[i].x + v[i].y + v[i].z + v[i].w;
#pragma unroll
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    const float mean = rms ? 0.f : s / d;
    float q = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const float a = v[i].x - mean, e = v[i].y - mean, c = v[i].z - mean, f = v[i].w - mean;
      q += a * a + e * e + c * c + f * f;
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
    const float rstd = rsqrtf(q / d + eps);
    if (lane == 0) {
      if (mean_out) mean_out[row] = mean;
      if (rstd_out) rstd_out[row] = rstd;
    }
    if (!AHEAD) fetch_weights();
    uint2* yr = reinterpret_cast<uint2*>(y + (long long)row * d);
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      uint2 o;
      o.x = pack_bf16x2((v[i].x - mean) * rstd * g[i].x + b[i].x, (v[i].y - mean) * rstd * g[i].y + b[i].y);
      o.y = pack_bf16x2((v[i].z - mean) * rstd * g[i].z + b[i].z, (v[i].w - mean) * rstd * g[i].w + b[i].w);
      yr[lane + 32 * i] = o;
    }
  }
}

struct LnBwdArgs {
  const __nv_bfloat16* dy;   // [M,d] grad wrt normalised output (may be null if only heads feed)
  const float* x;            // [M,d] forward input
  const float* mean;         // [M]
  const float* rstd;         // [M]
  const float* gamma;        // [d]
  const float* dres_in;      // [M,d] incoming residual gradient or null
  float* dx;                 // [M,d] out (may alias dres_in)
  __nv_bfloat16* dbranch;    // [M,d] out or null: bf16(dropout_mask * dx)
  float* dgamma;             // [d] accumulated
  float* dbeta;              // [d] accumulated or null
  float* dbias;              // [d] accumulated or null: column sums of the masked copy (the bias
                             // gradient of the projection whose output that copy is the gradient of)
  // optional rank-2 term: dy_eff[m,c] = dy[m,c] + s0[m]*w0[c] + s1[m]*w1[c]
  const float* s0; const float* w0; const float* s1; const float* w1;
  int M, d, rms;
  unsigned long long drop_seed; unsigned int drop_stream, drop_thr16;
  const unsigned long long* salt;   // seed_salt_ptr() at launch: folded into drop_seed when not null
  int* status;
};

// Backward kernel.  A group of threads owns a row and every thread of it the same eight columns of
// each row it meets (float4 columns t and t + d/8), so the column sums dgamma / dbeta / dbias stay in
// 24 registers per thread from the first row to the last and no shared-memory accumulator limits how
// many rows are in flight: bound by bytes (16 per element with a residual and a masked copy).  The
// form before kept a warp per row and the sums of every warp in shared memory (96 bytes per column of
// a block): 16 warps per SM at d <= 1024, 8 above.
//   LNB_ROWS rows are handled together (one exchange of row sums through shared memory for all of them).
//   They come in by bulk copies, LNB_STAGES pairs of rows ahead per group (160 KB in flight on an SM): with
//   loads into registers nothing was on its way while a block computed (32768 x 1024: 113 us, now 105).
//   RING = false is the form with plain loads, for tensors that bulk copies cannot address (16 bytes).
//   A block holds as many groups as fit 512 threads (the registers of an SM) and folds their sums before
//   its atomics: with a block per group, 740 blocks adding to the same 2304 addresses cost 12136 x 768
//   more than the register sums gain.
// The eight columns of a thread belong to two dropout groups of eight; neighbouring lanes share both,
// so each lane draws one and they swap.
constexpr int LNB_ROWS = 2;
constexpr int LNB_THREADS = 512;
constexpr int LNB_STAGES = 2;

__device__ __forceinline__ float4 ln_unpack4(uint2 p) {
  return make_float4(bf16_lo(p.x), bf16_hi(p.x), bf16_lo(p.y), bf16_hi(p.y));
}
__device__ __forceinline__ void ln_red4(float* dst, const float4& v) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w)
               : "memory");
}

__device__ __forceinline__ void ln_bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}

template <bool RING>
__global__ void __launch_bounds__(LNB_THREADS, 1)
ln_bwd_kernel(const LnBwdArgs a) {
  griddep_enter();
  constexpr int R = LNB_ROWS;
  // RING: [groups][stages][R rows of x | dres_in | dy]; at the end, and without it, [groups][3][d]
  extern __shared__ __align__(16) float ln_fold[];
  __shared__ uint64_t full[LNB_THREADS / 32][LNB_STAGES];
  __shared__ int abort_word;
  __shared__ int late[LNB_THREADS / 32][3];                 // first wait of a group's thread 0 that ran out
  __shared__ __align__(16) float red[2][LNB_THREADS / 32][2 * R];
  const int gt = blockDim.x;                                // threads of a row group (multiple of 32)
  const int t = threadIdx.x, grp = threadIdx.y, groups = blockDim.y;
  const int lane = t & 31, gwarps = gt >> 5, warp = grp * gwarps + (t >> 5);
  const int d = a.d, n = d >> 3;                            // n threads carry columns
  const bool own = t < n;
  const int c[2] = {own ? t : 0, own ? t + n : 0};          // float4 columns
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  const bool has_dy = a.dy != nullptr, has_r = a.dres_in != nullptr;
  const bool want_bias = a.dgamma != nullptr && a.dbias != nullptr && a.dbranch != nullptr;
  const float dscale = dropout_scale(a.drop_thr16);
  const uint64_t seed = a.drop_thr16 ? salted(a.drop_seed, a.salt) : 0;
  const float inv_d = 1.f / d;
  float4 gam[2], sg[2] = {zero, zero}, sb[2] = {zero, zero}, sc[2] = {zero, zero};
#pragma unroll
  for (int u = 0; u < 2; ++u) gam[u] = own ? __ldg(reinterpret_cast<const float4*>(a.gamma) + c[u]) : zero;

  int par = 0;
  const int step = gridDim.x * groups * R, first = (blockIdx.x * groups + grp) * R;
  uint8_t* ring = reinterpret_cast<uint8_t*>(ln_fold) + static_cast<size_t>(grp) * LNB_STAGES * R * 10 * d;
  // rows row0 .. row0 + R - 1 (those below M) into stage st; one thread of the group
  auto fetch = [&](int row0, int st) {
    if (row0 >= a.M) return;
    uint8_t* dst = ring + static_cast<size_t>(st) * R * 10 * d;
    const uint32_t n = (a.M - row0 < R ? a.M - row0 : R) * d;           // elements
    const long long off = static_cast<long long>(row0) * d;
    mbar_expect_tx(&full[grp][st], n * (4 + (has_r ? 4 : 0) + (has_dy ? 2 : 0)));
    ln_bulk_load(dst, a.x + off, n * 4, &full[grp][st]);
    if (has_r) ln_bulk_load(dst + R * 4 * d, a.dres_in + off, n * 4, &full[grp][st]);
    if (has_dy) ln_bulk_load(dst + R * 8 * d, a.dy + off, n * 2, &full[grp][st]);
  };
  if (RING) {
    if (t == 0) {
      for (int i = 0; i < LNB_STAGES; ++i) mbar_init(&full[grp][i], 1);
      if (grp == 0) abort_word = 0;
      late[grp][0] = -1;
      mbar_fence_init();
    }
    __syncthreads();
    if (t == 0)
      for (int i = 0; i < LNB_STAGES; ++i) fetch(first + i * step, i);
  }
  int stage = 0;
  uint32_t phase = 0;
  for (int row0 = first; row0 < a.M; row0 += step, par ^= 1) {
    const uint8_t* src = ring + static_cast<size_t>(stage) * R * 10 * d;
    if (RING && !mbar_wait(&full[grp][stage], phase, &abort_word)) {
      // every thread goes on (the group meets at barriers); the waits that follow end at once
      *static_cast<volatile int*>(&abort_word) = 1;
      if (a.status) atomicCAS(a.status, 0, ST_TIMEOUT_FULL);
      if (t == 0 && late[grp][0] < 0) { late[grp][0] = row0; late[grp][1] = stage; late[grp][2] = phase; }
    }
    float4 xh[R][2], rv[R][2], dy[R][2];
    uint2 dyp[R][2];
    float mean[R], rstd[R];
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int row = row0 + i;
      const bool live = own && row < a.M;
      mean[i] = 0.f;
      rstd[i] = 0.f;
      if (row < a.M) {
        rstd[i] = a.rstd[row];
        if (!a.rms) mean[i] = a.mean[row];
      }
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        xh[i][u] = zero; rv[i][u] = zero; dyp[i][u] = make_uint2(0u, 0u);
        if (live) {
          if (RING) {
            xh[i][u] = reinterpret_cast<const float4*>(src + i * 4 * d)[c[u]];
            if (has_r) rv[i][u] = reinterpret_cast<const float4*>(src + (R + i) * 4 * d)[c[u]];
            if (has_dy) dyp[i][u] = reinterpret_cast<const uint2*>(src + R * 8 * d + i * 2 * d)[c[u]];
          } else {
            xh[i][u] = reinterpret_cast<const float4*>(a.x + (long long)row * d)[c[u]];
            if (has_dy) dyp[i][u] = reinterpret_cast<const uint2*>(a.dy + (long long)row * d)[c[u]];
            if (has_r) rv[i][u] = reinterpret_cast<const float4*>(a.dres_in + (long long)row * d)[c[u]];
          }
        }
      }
    }
    float part[2 * R];
#pragma unroll
    for (int i = 0; i < R; ++i) {
      float s1 = 0.f, s2 = 0.f;
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        float4 g = ln_unpack4(dyp[i][u]);
        if (a.s0 && own && row0 + i < a.M) {                // rank-2 term of the scalar heads
          const float k = a.s0[row0 + i];
          const float4 w = __ldg(reinterpret_cast<const float4*>(a.w0) + c[u]);
          g.x += k * w.x; g.y += k * w.y; g.z += k * w.z; g.w += k * w.w;
        }
        if (a.s1 && own && row0 + i < a.M) {
          const float k = a.s1[row0 + i];
          const float4 w = __ldg(reinterpret_cast<const float4*>(a.w1) + c[u]);
          g.x += k * w.x; g.y += k * w.y; g.z += k * w.z; g.w += k * w.w;
        }
        const float4 x = xh[i][u];
        const float4 h = make_float4((x.x - mean[i]) * rstd[i], (x.y - mean[i]) * rstd[i],
                                     (x.z - mean[i]) * rstd[i], (x.w - mean[i]) * rstd[i]);
        xh[i][u] = h;
        dy[i][u] = g;
        s1 += g.x * gam[u].x + g.y * gam[u].y + g.z * gam[u].z + g.w * gam[u].w;
        s2 += g.x * gam[u].x * h.x + g.y * gam[u].y * h.y + g.z * gam[u].z * h.z + g.w * gam[u].w * h.w;
        sg[u].x += g.x * h.x; sg[u].y += g.y * h.y; sg[u].z += g.z * h.z; sg[u].w += g.w * h.w;
        sb[u].x += g.x; sb[u].y += g.y; sb[u].z += g.z; sb[u].w += g.w;
      }
      part[2 * i] = s1;
      part[2 * i + 1] = s2;
    }
#pragma unroll
    for (int o = 16; o; o >>= 1)
#pragma unroll
      for (int k = 0; k < 2 * R; ++k) part[k] += __shfl_xor_sync(0xffffffffu, part[k], o);
    if (gwarps > 1) {
      // the slot written two rounds ago is free: its readers passed the barrier of the round between
      if (lane == 0)
#pragma unroll
        for (int k = 0; k < 2 * R; ++k) red[par][warp][k] = part[k];
      asm volatile("bar.sync %0, %1;" ::"r"(grp + 1), "r"(gt) : "memory");
#pragma unroll
      for (int k = 0; k < 2 * R; ++k) part[k] = 0.f;
      for (int w = 0; w < gwarps; ++w)
#pragma unroll
        for (int k = 0; k < 2 * R; ++k) part[k] += red[par][grp * gwarps + w][k];
    } else {
      __syncwarp();
    }
    if (RING) {                                             // the group has read the stage
      if (t == 0 && late[grp][0] < 0) fetch(row0 + LNB_STAGES * step, stage);
      if (++stage == LNB_STAGES) { stage = 0; phase ^= 1; }
    }
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int row = row0 + i;
      const float m1 = a.rms ? 0.f : part[2 * i] * inv_d, m2 = part[2 * i + 1] * inv_d;
      uint32_t keep = 0xffu;                                // low 4 bits: column c[0], high 4: c[1]
      if (a.drop_thr16 && a.dbranch) {
        const uint64_t f4 = static_cast<uint64_t>(row) * (d >> 2) + ((lane & 1) ? t - 1 + n : t);
        const uint32_t mine = dropout_keep8(seed, a.drop_stream, f4 >> 1, a.drop_thr16);
        const uint32_t other = __shfl_xor_sync(0xffffffffu, mine, 1);
        keep = (lane & 1) ? ((other >> 4) & 0xfu) | (mine & 0xf0u) : (mine & 0xfu) | ((other & 0xfu) << 4);
      }
      if (!own || row >= a.M) continue;
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const float4 g = dy[i][u], h = xh[i][u];
        float4 o;
        o.x = (g.x * gam[u].x - m1 - h.x * m2) * rstd[i] + rv[i][u].x;
        o.y = (g.y * gam[u].y - m1 - h.y * m2) * rstd[i] + rv[i][u].y;
        o.z = (g.z * gam[u].z - m1 - h.z * m2) * rstd[i] + rv[i][u].z;
        o.w = (g.w * gam[u].w - m1 - h.w * m2) * rstd[i] + rv[i][u].w;
        reinterpret_cast<float4*>(a.dx + (long long)row * d)[c[u]] = o;
        if (a.dbranch) {
          if (a.drop_thr16) {
            const uint32_t k4 = keep >> (4 * u);
            o.x = (k4 & 1u) ? o.x * dscale : 0.f;
            o.y = (k4 & 2u) ? o.y * dscale : 0.f;
            o.z = (k4 & 4u) ? o.z * dscale : 0.f;
            o.w = (k4 & 8u) ? o.w * dscale : 0.f;
          }
          reinterpret_cast<uint2*>(a.dbranch + (long long)row * d)[c[u]] =
              make_uint2(pack_bf16x2(o.x, o.y), pack_bf16x2(o.z, o.w));
          sc[u].x += o.x; sc[u].y += o.y; sc[u].z += o.z; sc[u].w += o.w;
        }
      }
    }
  }
  if (RING && t == 0 && late[grp][0] >= 0) {
    // The thread that fetches has stopped there; what it had under way lands before the block reuses or
    // leaves its shared memory.
    for (int i = 0; i < LNB_STAGES; ++i) {
      const int row0 = late[grp][0] + i * step, st = (late[grp][1] + i) % LNB_STAGES;
      if (row0 < a.M) mbar_wait_landed(&full[grp][st], late[grp][2] ^ (late[grp][1] + i >= LNB_STAGES));
    }
  }
  if (!a.dgamma) return;
  if (groups > 1) {                                         // block-uniform
    if (RING) __syncthreads();                              // the sums take the place of the ring
    float4* f = reinterpret_cast<float4*>(ln_fold);
    const int d4 = d >> 2;
    if (own && grp > 0)
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        f[(grp * 3 + 0) * d4 + c[u]] = sg[u];
        f[(grp * 3 + 1) * d4 + c[u]] = sb[u];
        f[(grp * 3 + 2) * d4 + c[u]] = sc[u];
      }
    __syncthreads();
    if (grp > 0) return;
    for (int g = 1; g < groups; ++g)
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const float4 x = f[(g * 3 + 0) * d4 + c[u]], y = f[(g * 3 + 1) * d4 + c[u]], z = f[(g * 3 + 2) * d4 + c[u]];
        sg[u].x += x.x; sg[u].y += x.y; sg[u].z += x.z; sg[u].w += x.w;
        sb[u].x += y.x; sb[u].y += y.y; sb[u].z += y.z; sb[u].w += y.w;
        sc[u].x += z.x; sc[u].y += z.y; sc[u].z += z.z; sc[u].w += z.w;
      }
  }
  if (!own) return;
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    ln_red4(a.dgamma + c[u] * 4, sg[u]);
    if (a.dbeta) ln_red4(a.dbeta + c[u] * 4, sb[u]);
    if (want_bias) ln_red4(a.dbias + c[u] * 4, sc[u]);
  }
}

}  // namespace ab

// rows spread over all SMs before a block takes more than one
static int ln_block_warps(int M) {
  const int want = (M + 147) / 148;
  return want < ab::LN_WARPS ? want : ab::LN_WARPS;
}

// dependent: 1 = programmatic dependent, 2 = and gamma and beta may be read before the kernel before has finished
template <int NV>
static int launch_ln_fwd(int dependent, const float* x, const float* gamma, const float* beta, void* y, float* mean,
                         float* rstd, int M, int d, float eps, int rms, cudaStream_t stream) {
  using namespace ab;
  if constexpr (NV < 16) {
    if (d > NV * 128)
      return launch_ln_fwd<NV + 1>(dependent, x, gamma, beta, y, mean, rstd, M, d, eps, rms, stream);
  }
  const int warps = ln_block_warps(M);
  int grid = (M + warps - 1) / warps;
  if (grid > 148 * 8) grid = 148 * 8;
  if (!dependent) {
    launch_chained(ln_fwd_kernel<NV, false>, dim3(grid), dim3(warps * 32), 0, stream, x, gamma, beta,
                   (__nv_bfloat16*)y, mean, rstd, M, eps, rms);
    return (int)cudaGetLastError();
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(warps * 32);
  cfg.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  auto kern = dependent == 2 ? ln_fwd_kernel<NV, true> : ln_fwd_kernel<NV, false>;
  return (int)cudaLaunchKernelEx(&cfg, kern, x, gamma, beta, (__nv_bfloat16*)y, mean, rstd, M, eps, rms);
}

extern "C" {

// d must be a multiple of 128 and at most 2048.
// Same as ab_layernorm_fwd, launched as a programmatic dependent of the kernel before it in the
// stream (its launch overlaps that kernel's tail; it waits for it before reading anything).
int ab_layernorm_fwd_dependent(const float* x, const float* gamma, const float* beta, void* y, float* mean,
                               float* rstd, int M, int d, float eps, int rms, cudaStream_t stream) {
  if (d < 128 || d % 128 != 0 || d > 2048 || M <= 0) return -1;
  return launch_ln_fwd<1>(1, x, gamma, beta, y, mean, rstd, M, d, eps, rms, stream);
}

// The same for gamma and beta that the kernel before does not write: they are read while it is still running.
int ab_layernorm_fwd_ahead(const float* x, const float* gamma, const float* beta, void* y, float* mean, float* rstd,
                           int M, int d, float eps, int rms, cudaStream_t stream) {
  if (d < 128 || d % 128 != 0 || d > 2048 || M <= 0) return -1;
  return launch_ln_fwd<1>(2, x, gamma, beta, y, mean, rstd, M, d, eps, rms, stream);
}

int ab_layernorm_fwd(const float* x, const float* gamma, const float* beta, void* y, float* mean,
                     float* rstd, int M, int d, float eps, int rms, cudaStream_t stream) {
  if (d < 128 || d % 128 != 0 || d > 2048 || M <= 0) return -1;
  return launch_ln_fwd<1>(0, x, gamma, beta, y, mean, rstd, M, d, eps, rms, stream);
}

int ab_layernorm_bwd(const void* dy, const float* x, const float* mean, const float* rstd,
                     const float* gamma, const float* dres_in, float* dx, void* dbranch,
                     float* dgamma, float* dbeta, float* dbias, const float* s0, const float* w0,
                     const float* s1, const float* w1, int M, int d, int rms,
                     unsigned long long drop_seed, unsigned int drop_stream,
                     unsigned int drop_thr16, int* status, cudaStream_t stream) {
  using namespace ab;
  if (d % 128 != 0 || d > 2048 || M <= 0) return -1;
  LnBwdArgs a;
  a.dy = (const __nv_bfloat16*)dy; a.x = x; a.mean = mean; a.rstd = rstd; a.gamma = gamma;
  a.dres_in = dres_in; a.dx = dx; a.dbranch = (__nv_bfloat16*)dbranch; a.dgamma = dgamma;
  a.dbeta = dbeta; a.dbias = dbias; a.s0 = s0; a.w0 = w0; a.s1 = s1; a.w1 = w1; a.M = M; a.d = d; a.rms = rms;
  a.drop_seed = drop_seed; a.drop_stream = drop_stream; a.drop_thr16 = drop_thr16; a.salt = seed_salt_ptr(); a.status = status;
  const int gt = ((d >> 3) + 31) / 32 * 32;                 // threads of a row group
  // groups per block: what 512 threads hold, but no more than leaves every SM a block
  const int want = (M + 148 * LNB_ROWS - 1) / (148 * LNB_ROWS);
  const int groups = want < LNB_THREADS / gt ? want : LNB_THREADS / gt;
  const int rows = groups * LNB_ROWS;
  int grid = (M + rows - 1) / rows;
  if (grid > 148) grid = 148;
  const bool ring = ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(dy) | reinterpret_cast<uintptr_t>(dres_in)) & 15) == 0;
  const size_t smem = ring ? (size_t)groups * LNB_STAGES * LNB_ROWS * 10 * d : groups > 1 ? sizeof(float) * groups * 3 * d : 0;
  auto kern = ring ? ln_bwd_kernel<true> : ln_bwd_kernel<false>;
  static PerDeviceOnce attr_set[2];
  if (attr_set[ring].first_use_on_device()) {
    // groups * d <= LNB_THREADS / gt * 8 * gt columns
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         LNB_THREADS * 8 * (ring ? LNB_STAGES * LNB_ROWS * 10 : 3 * (int)sizeof(float)));
    if (e != cudaSuccess) return (int)e;
    attr_set[ring].mark_device();
  }
  launch_chained(kern, dim3(grid), dim3(gt, groups), smem, stream, a);
  return (int)cudaGetLastError();
}
}
