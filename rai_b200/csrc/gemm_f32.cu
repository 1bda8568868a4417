// float32 Linear (the float32 models' rb_linear and rb_gated_linear) on CUDA cores: every product and sum is a float32 FMA.
//
// gemv_f32_kernel   M <= 8 rows (single-token steps): bound by the weight stream.  A feature's weight row is shared out among
//                   1 to 8 warps, so that narrow layers, too, put enough warps on the GPU, and a lane requests 64 to 128 bytes of
//                   the row (a warp 2 to 4 KB) before it multiplies any of them.
// gemm_f32_kernel   more rows (prompts): bound by the FMA pipe.  Tiles of 16 TM rows x 64 features, TM chosen so that few rows
//                   are padding; where the tiles alone do not fill the GPU, K is cut among the blocks of a cluster, which add
//                   their sums through distributed shared memory in the order of K.
#include <algorithm>

#include "ctx.h"

namespace rb {

namespace {

bool rows_of_pieces(const GemmArgs& a) {
  auto al16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  return a.k % 4 == 0 && al16(a.x) && al16(a.w) && (!a.w2 || al16(a.w2));
}

// ---- few rows ---------------------------------------------------------------------------------------------------------------
// MR: rows computed (m <= MR).  Blocks of 8 warps, `share` of them per feature.
template <int MR, bool GATED>
__global__ void __launch_bounds__(256) gemv_f32_kernel(const float* __restrict__ x, const float* __restrict__ w,
                                                       const float* __restrict__ w2, const float* __restrict__ bias,
                                                       const float* __restrict__ residual, float* __restrict__ out, int m, int n, int k,
                                                       int act, const float* __restrict__ act_params, int share, int vec) {
  constexpr int U = GATED || MR > 4 ? 4 : 8;   // 16-byte pieces of a weight row that a lane has in flight
  constexpr int G = GATED ? 2 : 1;
  __shared__ float part[8][G * MR];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int col = blockIdx.x * (8 / share) + warp / share, piece = warp % share;
  float acc[G * MR];
#pragma unroll
  for (int r = 0; r < G * MR; ++r) acc[r] = 0.f;
  const float* wr = w + (size_t)col * k;
  const float* wr2 = GATED ? w2 + (size_t)col * k : nullptr;
  if (col < n && !vec) {   // rows that are not made of 16-byte pieces
    for (int i = piece * 32 + lane; i < k; i += share * 32) {
      const float a = wr[i], b = GATED ? wr2[i] : 0.f;
#pragma unroll
      for (int r = 0; r < MR; ++r) {
        if (MR > 1 && r >= m) break;
        const float xv = x[(size_t)r * k + i];
        acc[r] = fmaf(a, xv, acc[r]);
        if (GATED) acc[MR + r] = fmaf(b, xv, acc[MR + r]);
      }
    }
  } else if (col < n) {
    for (int i0 = piece * (128 * U); i0 < k; i0 += share * (128 * U)) {
      float4 a[U], b[GATED ? U : 1];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int i = i0 + u * 128 + lane * 4;
        a[u] = i < k ? __ldcs(reinterpret_cast<const float4*>(wr + i)) : make_float4(0.f, 0.f, 0.f, 0.f);
        if (GATED) b[u] = i < k ? __ldcs(reinterpret_cast<const float4*>(wr2 + i)) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
#pragma unroll
      for (int r = 0; r < MR; ++r) {
        if (MR > 1 && r >= m) break;
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int i = i0 + u * 128 + lane * 4;
          if (i >= k) break;
          const float4 xv = *reinterpret_cast<const float4*>(x + (size_t)r * k + i);
          acc[r] = fmaf(a[u].w, xv.w, fmaf(a[u].z, xv.z, fmaf(a[u].y, xv.y, fmaf(a[u].x, xv.x, acc[r]))));
          if (GATED) acc[MR + r] = fmaf(b[u].w, xv.w, fmaf(b[u].z, xv.z, fmaf(b[u].y, xv.y, fmaf(b[u].x, xv.x, acc[MR + r]))));
        }
      }
    }
  }
#pragma unroll
  for (int r = 0; r < G * MR; ++r) {
    const float v = warp_sum(acc[r]);
    if (lane == 0) part[warp][r] = v;
  }
  __syncthreads();
  if (piece != 0 || lane >= m || col >= n) return;   // lane r of a feature's first warp finishes row r
  float v = 0.f, v2 = 0.f;
  for (int s = 0; s < share; ++s) {
    v += part[warp + s][lane];
    if (GATED) v2 += part[warp + s][MR + lane];
  }
  const size_t at = (size_t)lane * n + col;
  if (GATED) {
    v = act_apply(act, v) * v2;
  } else {
    if (bias) v += bias[col];
    v = act_apply(act, v, act == RB_ACT_XIELU ? xielu_consts(act_params) : make_float2(0.f, 0.f));
    if (residual) v += residual[at];
  }
  out[at] = v;
}

// ---- many rows --------------------------------------------------------------------------------------------------------------
constexpr int kBN = 64, kBK = 32, kPitch = kBK + 4;   // floats; the pad keeps 16-byte reads of neighbouring rows apart
constexpr int kStages = 3;

template <int TM, bool GATED>
constexpr int gemm_f32_smem() {
  return std::max(kStages * (16 * TM + (GATED ? 2 : 1) * kBN) * kPitch, (GATED ? 2 : 1) * 16 * TM * kBN) * (int)sizeof(float);
}

__device__ __forceinline__ void copy16(float* dst, const float* src, bool real) {   // zeros where the tile sticks out
  const int bytes = real ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes)
               : "memory");
}

template <int TM, bool GATED>
__global__ void __launch_bounds__(128) gemm_f32_kernel(const float* __restrict__ x, const float* __restrict__ w,
                                                       const float* __restrict__ w2, const float* __restrict__ bias,
                                                       const float* __restrict__ residual, float* __restrict__ out, int m, int n, int k,
                                                       int act, const float* __restrict__ act_params) {
  constexpr int BM = 16 * TM, G = GATED ? 2 : 1;
  constexpr int kStageFloats = (BM + G * kBN) * kPitch;
  extern __shared__ __align__(16) float smem_f32[];
  uint32_t rank, shares;   // of the cluster that cuts K
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(shares));
  const int row0 = blockIdx.y * BM, col0 = blockIdx.x / (int)shares * kBN;
  const int num_kb = (k + kBK - 1) / kBK;
  const int kb0 = (int)((long long)num_kb * rank / shares), kb1 = (int)((long long)num_kb * (rank + 1) / shares);
  const int tx = threadIdx.x & 7, ty = threadIdx.x >> 3;   // columns tx + 8 j, rows ty + 16 i

  auto load = [&](int kb) {
    float* st = smem_f32 + (kb - kb0) % kStages * kStageFloats;
    const int c4 = threadIdx.x & 7, kc = kb * kBK + c4 * 4;
    for (int r = threadIdx.x >> 3; r < BM; r += 16) {
      const bool real = row0 + r < m && kc < k;
      copy16(st + r * kPitch + c4 * 4, real ? x + (size_t)(row0 + r) * k + kc : x, real);
    }
    for (int r = threadIdx.x >> 3; r < kBN; r += 16) {
      const bool real = col0 + r < n && kc < k;
      copy16(st + (BM + r) * kPitch + c4 * 4, real ? w + (size_t)(col0 + r) * k + kc : w, real);
      if (GATED) copy16(st + (BM + kBN + r) * kPitch + c4 * 4, real ? w2 + (size_t)(col0 + r) * k + kc : w2, real);
    }
  };
  float acc[G][TM][8] = {};
#pragma unroll
  for (int s = 0; s < kStages - 1; ++s) {
    if (kb0 + s < kb1) load(kb0 + s);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  for (int kb = kb0; kb < kb1; ++kb) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
    __syncthreads();   // the stage is there for all, and the one before it has been read by all
    if (kb + kStages - 1 < kb1) load(kb + kStages - 1);
    asm volatile("cp.async.commit_group;" ::: "memory");
    const float* xs = smem_f32 + (kb - kb0) % kStages * kStageFloats;
    const float* ws = xs + BM * kPitch;
#pragma unroll
    for (int c = 0; c < kBK; c += 4) {
      float4 a[TM], b[8];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = *reinterpret_cast<const float4*>(xs + (ty + 16 * i) * kPitch + c);
#pragma unroll
      for (int g = 0; g < G; ++g) {
#pragma unroll
        for (int j = 0; j < 8; ++j) b[j] = *reinterpret_cast<const float4*>(ws + (g * kBN + tx + 8 * j) * kPitch + c);
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
          for (int j = 0; j < 8; ++j)
            acc[g][i][j] = fmaf(a[i].w, b[j].w, fmaf(a[i].z, b[j].z, fmaf(a[i].y, b[j].y, fmaf(a[i].x, b[j].x, acc[g][i][j]))));
      }
    }
  }
  __syncthreads();
  // the tile's sums in shared memory, [G][BM][64]; each block of the cluster finishes a share of the rows
#pragma unroll
  for (int g = 0; g < G; ++g)
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) smem_f32[(g * BM + ty + 16 * i) * kBN + tx + 8 * j] = acc[g][i][j];
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  const float2 ac = act == RB_ACT_XIELU ? xielu_consts(act_params) : make_float2(0.f, 0.f);
  const int r_end = min(BM, m - row0);
  const uint32_t base = (uint32_t)__cvta_generic_to_shared(smem_f32);
  for (int id = threadIdx.x + (int)rank * 128; id < r_end * (kBN / 4); id += 128 * (int)shares) {
    const int r = id / (kBN / 4), c = id % (kBN / 4) * 4;
    float v[G][4] = {};
    for (uint32_t s = 0; s < shares; ++s)
#pragma unroll
      for (int g = 0; g < G; ++g) {
        uint32_t at;
        float4 t;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(base + (uint32_t)((g * BM + r) * kBN + c) * 4u), "r"(s));
        asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(t.x), "=f"(t.y), "=f"(t.z), "=f"(t.w) : "r"(at) : "memory");
        v[g][0] += t.x; v[g][1] += t.y; v[g][2] += t.z; v[g][3] += t.w;
      }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int col = col0 + c + j;
      if (col >= n) break;
      const size_t o = (size_t)(row0 + r) * n + col;
      float y = v[0][j];
      if (GATED) {
        y = act_apply(act, y) * v[G - 1][j];
      } else {
        if (bias) y += bias[col];
        y = act_apply(act, y, ac);
        if (residual) y += residual[o];
      }
      out[o] = y;
    }
  }
  // no block leaves while another may still read its sums
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <int MR, bool GATED>
void gemv_launch(rb_ctx* ctx, const GemmArgs& a) {
  // as many warps per feature as put about 32 warps on every SM, as long as each has a piece of the row
  constexpr int U = GATED || MR > 4 ? 4 : 8;
  const int vec = rows_of_pieces(a);
  int share = 1;
  while (share < 8 && a.n * share * 2 <= (int64_t)ctx->sm_count * 32 && (int64_t)share * 128 * U < a.k) share *= 2;
  const int cols = 8 / share;
  gemv_f32_kernel<MR, GATED><<<(unsigned)((a.n + cols - 1) / cols), 256, 0, ctx->stream>>>(
      (const float*)a.x, (const float*)a.w, (const float*)a.w2, GATED ? nullptr : (const float*)a.bias,
      GATED ? nullptr : (const float*)a.residual, (float*)a.out, (int)a.m, (int)a.n, (int)a.k, a.act, (const float*)a.act_params, share, vec);
}

template <int TM, bool GATED>
int gemm_launch(rb_ctx* ctx, const GemmArgs& a) {
  auto kern = gemm_f32_kernel<TM, GATED>;
  constexpr int smem = gemm_f32_smem<TM, GATED>();
  static bool attr_set[64] = {};
  const int dv = ctx->device & 63;
  if (smem > 48 * 1024 && !attr_set[dv]) {
    RB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    attr_set[dv] = true;
  }
  const int64_t nt = (a.n + kBN - 1) / kBN, mt = (a.m + 16 * TM - 1) / (16 * TM), num_kb = (a.k + kBK - 1) / kBK;
  RB_REQUIRE(mt <= 65535, "gemm: %lld rows", (long long)a.m);
  unsigned shares = 1;   // two blocks per SM, and at least four slices of K each
  while (shares < 8 && nt * mt * shares * 2 <= (int64_t)ctx->sm_count * 2 && num_kb >= (int64_t)shares * 8) shares *= 2;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)nt * shares, (unsigned)mt);
  cfg.blockDim = dim3(128);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = ctx->stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = shares;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  RB_CUDA(cudaLaunchKernelEx(&cfg, kern, (const float*)a.x, (const float*)a.w, (const float*)a.w2, (const float*)(GATED ? nullptr : a.bias),
                             (const float*)(GATED ? nullptr : a.residual), (float*)a.out, (int)a.m, (int)a.n, (int)a.k, a.act,
                             (const float*)a.act_params));
  return RB_OK;
}

template <bool GATED>
int dispatch(rb_ctx* ctx, const GemmArgs& a) {
  if (a.m <= 8) {
    if (a.m == 1) gemv_launch<1, GATED>(ctx, a);
    else if (a.m <= 2) gemv_launch<2, GATED>(ctx, a);
    else if (a.m <= 4) gemv_launch<4, GATED>(ctx, a);
    else gemv_launch<8, GATED>(ctx, a);
    return RB_OK;
  }
  // rows per thread: a slice of K costs a thread TM rows' products and about two rows' worth of reading the features
  // (a gated tile holds two sets of sums, so it stays smaller).  Where K is too short to be cut, tiles may not fill the GPU, and
  // what counts is how long one of them takes and how many follow it on an SM (us: 128 x 2048 x 100 with a residual 31 -> 12.5, 1000 x 64 x 64
  // 25 -> 8.3, 512 x 2048 x 100 33 -> 22, gated 200 x 2048 x 100 30 -> 21).
  constexpr int most = GATED ? 5 : 8;
  const int64_t r16 = (a.m + 15) / 16;
  const int64_t nt = (a.n + kBN - 1) / kBN, slots = 2 * (int64_t)ctx->sm_count;
  const bool short_k = (a.k + kBK - 1) / kBK < 8;
  auto cost = [&](int t) {
    const int64_t tiles = (r16 + t - 1) / t;
    return (short_k ? (tiles * nt + slots - 1) / slots : tiles) * (t + 2);
  };
  int best = 1;
  for (int t = 2; t <= most; ++t)
    if (cost(t) <= cost(best)) best = t;
  switch (best) {
    case 1: return gemm_launch<1, GATED>(ctx, a);
    case 2: return gemm_launch<2, GATED>(ctx, a);
    case 3: return gemm_launch<3, GATED>(ctx, a);
    case 4: return gemm_launch<4, GATED>(ctx, a);
    case 5: return gemm_launch<5, GATED>(ctx, a);
  }
  if constexpr (!GATED) {
    if (best == 6) return gemm_launch<6, false>(ctx, a);
    if (best == 7) return gemm_launch<7, false>(ctx, a);
    return gemm_launch<8, false>(ctx, a);
  }
  return RB_OK;
}

}  // namespace

// false: the general kernel takes this call
bool gemm_f32_takes(const GemmArgs& a) {
  return !a.partials && (a.m <= 8 || (a.k > 0 && rows_of_pieces(a) && a.m <= 65535 * 16));
}

int gemm_f32(rb_ctx* ctx, const GemmArgs& a) {
  RB_TRY(a.w2 ? dispatch<true>(ctx, a) : dispatch<false>(ctx, a));
  ctx->launches++;
  return launch_status("gemm_f32");
}

}  // namespace rb
