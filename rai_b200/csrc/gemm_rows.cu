// The products of a decode step with at most eight rows: C[M,N] = X[M,K] . W[N,K]^T, bound by the stream of W and, on small
// models, by how long each of a layer's launches takes from its predecessor's last store to its own.  So the whole of what
// lies between two products is in here: the norm of the rows on the way in; bias, activation, gate or the residual sum on the
// way out.  A layer is five launches: [norm, q/k/v], attention, [o, residual], [norm, gate/up, activation], [down, residual].
//
// One block of eight warps per SM.  Eight rows of W make a tile; its K is shared out among 1, 2, 4 or 8 warps, so that an SM works on
// all its tiles at once.  Each warp streams its own share: lane l copies 16 bytes of row l / 4 per slice of 32 K (cp.async) to
// where it will read them itself, which are the B operand of two m16n8k16 products if X is read in the same order (16 bytes of
// a row of shared memory).  So the stream needs no barriers, and 12 KB a warp are on their way.  The first of them do not depend
// on the kernel before this one and are requested while that is still running; where X leaves room, two blocks fit an SM.
// (Measured against it: the same reads held in registers, too few on their way, 1.8 TB/s; bulk copies of rows into a ring that all
// warps share, 2.9 TB/s, each stage costing every warp a wait, an arrival and half of a chain of products.)
// Tensor cores of the fifth generation would not help: a tile of 128 rows of W per SM leaves most SMs without work here (a
// layer of 896 features has seven), and splitting K over blocks is what costs the extra launches.
//
// Sums are float32; rows are normalised from, and the residual sum is rounded to, the model's type, as in the kernels with
// more rows.
#include <algorithm>

#include "ctx.h"
#include "ptx.cuh"

namespace rb {

using bf16 = __nv_bfloat16;

namespace {

constexpr int kWarps = 8;
// 16-byte pieces of a row that a lane normalises at most.  With 12 (a row's warps shared out among eight rows of more than 1024) a layer
// was slower than on the kernels for more rows: 16 layers of 1536 x 6144, eight rows 764 -> 826 us, of 2048 x 5000 838 -> 977.
constexpr int kNormPieces = 4;
constexpr int kTurns = 3, kTurnSlices = 8; // a warp's ring: turns of eight slices (gated: four of gate and four of up)
constexpr int kRingBytes = kWarps * kTurns * kTurnSlices * 512;
constexpr int kMostBytes = 212 * 1024;     // of shared memory (beside 8 KB of sums)

struct RowsParams {
  const bf16 *x, *w, *w2, *bias, *residual, *norm_w, *norm_b;
  bf16* out;
  float* out_f;
  int m, n, k, act, norm, pitch, share;    // norm: an rb norm kind, or -1; pitch: bytes of a row of X; share: warps per tile
  float eps;
};

__device__ __forceinline__ void copy16(uint32_t dst, const bf16* src, bool real) {   // zeros where W ends
  const int bytes = real ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
template <int N>
__device__ __forceinline__ void copies_left() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void copies_end() { asm volatile("cp.async.commit_group;" ::: "memory"); }

// c (rows 0-7 of X, 8 rows of W) += X (16 k, rows 8-15 are zero) . W^T
__device__ __forceinline__ void mma_rows(float (&c)[4], uint32_t a0, uint32_t a2, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(0u), "r"(a2), "r"(0u), "r"(b0), "r"(b1));
}

template <bool GATED>
__global__ void __launch_bounds__(kWarps * 32, 2) gemm_rows_kernel(const RowsParams p) {
  constexpr int G = GATED ? 2 : 1, U = kTurnSlices / G;   // slices per turn
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ float red[2][kWarps][G][64];  // [turn][warp][..][row of X * 8 + row of W]
  __shared__ float sums[2][kWarps];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int share = p.share, group = warp / share, part = warp % share;
  const int r = lane >> 2, q = lane & 3;
  const int tiles = (p.n + 7) / 8, step = (int)gridDim.x * (kWarps / share);
  const int slices = (p.k + 31) / 32, mine = (slices + share - 1) / share, first = part * mine, limit = min(slices, first + mine);
  const int turns = (mine + U - 1) / U;    // per tile
  uint8_t* x_s = smem + kRingBytes;
  const uint32_t ring = ptx::smem_u32(smem) + (uint32_t)(warp * kTurns * kTurnSlices * 512 + lane * 16);
  const uint8_t* ring_p = smem + warp * kTurns * kTurnSlices * 512 + lane * 16;

  // the copies run kTurns turns ahead of the products
  int c_tile = (int)blockIdx.x + group * (int)gridDim.x, c_turn = 0, c_slot = 0;
  auto request = [&] {
    if (c_tile < tiles) {
      const int row = c_tile * 8 + r, k0 = (first + c_turn * U) * 32 + q * 8;
      const size_t at = (size_t)row * p.k + k0;
      const int stop = row < p.n ? min(p.k, limit * 32) : 0;
      const uint32_t dst = ring + (uint32_t)(c_slot * kTurnSlices * 512);
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const bool real = k0 + u * 32 < stop;
        copy16(dst + u * 512, real ? p.w + at + u * 32 : p.w, real);
        if (GATED) copy16(dst + (U + u) * 512, real ? p.w2 + at + u * 32 : p.w2, real);
      }
      if (++c_turn == turns) { c_turn = 0; c_tile += step; }
      if (++c_slot == kTurns) c_slot = 0;
    }
    copies_end();
  };
  pdl_launch_dependents();
#pragma unroll
  for (int i = 0; i < kTurns; ++i) request();
  pdl_wait();

  // ---- X into shared memory, normalised on the way; what sticks out of K is zero
  const int pieces = p.k >> 3, padded = (p.k + 31) / 32 * 4;
  if (p.norm < 0) {
    for (int i = threadIdx.x; i < p.m * padded; i += kWarps * 32) {
      const int row = i / padded, c = i % padded;
      uint4* dst = reinterpret_cast<uint4*>(x_s + row * p.pitch + c * 16);
      if (c < pieces)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(ptx::smem_u32(dst)), "l"(p.x + (size_t)row * p.k + c * 8) : "memory");
      else *dst = make_uint4(0, 0, 0, 0);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");   // (the ring, requested earlier, is there then, too)
  } else {
    const int per_row = kWarps / p.m, row = warp / per_row, at = (warp % per_row) * 32 + lane, stride = per_row * 32;
    const bool work = row < p.m;
    uint4 v[kNormPieces];
    float s = 0.f;
    const float inv_sqrt_h = 1.0f / sqrtf((float)p.k);
#pragma unroll
    for (int i = 0; i < kNormPieces; ++i)
      if (work && at + i * stride < pieces) v[i] = *reinterpret_cast<const uint4*>(p.x + (size_t)row * p.k + (at + i * stride) * 8);
#pragma unroll
    for (int i = 0; i < kNormPieces; ++i)
      if (work && at + i * stride < pieces) {
        float t[8];
        load8(reinterpret_cast<const bf16*>(&v[i]), t);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          if (p.norm == RB_NORM_LAYER) s += t[j];
          else if (p.norm == RB_NORM_RMS) { const float u = t[j] * inv_sqrt_h; s += u * u; }
          else s += t[j] * t[j];
        }
      }
    auto row_sum = [&](float a, int turn) {   // over the warps of a row
      a = warp_sum(a);
      if (lane == 0) sums[turn][warp] = a;
      __syncthreads();
      a = 0.f;
      for (int i = 0; i < per_row; ++i) a += work ? sums[turn][row * per_row + i] : 0.f;
      return a;
    };
    s = row_sum(s, 0);
    float mean = 0.f, scale;
    if (p.norm == RB_NORM_LAYER) {
      mean = s / (float)p.k;
      float d2 = 0.f;
#pragma unroll
      for (int i = 0; i < kNormPieces; ++i)
        if (work && at + i * stride < pieces) {
          float t[8];
          load8(reinterpret_cast<const bf16*>(&v[i]), t);
#pragma unroll
          for (int j = 0; j < 8; ++j) d2 += (t[j] - mean) * (t[j] - mean);
        }
      scale = 1.0f / sqrtf(row_sum(d2, 1) / (float)p.k + p.eps);
    } else {
      scale = 1.0f / sqrtf((p.norm == RB_NORM_RMS ? s : s / (float)p.k) + p.eps);
    }
#pragma unroll
    for (int i = 0; i < kNormPieces; ++i) {
      const int c = at + i * stride;
      if (!work || c >= padded) continue;
      float y[8] = {};
      if (c < pieces) {
        float t[8], g[8], o[8] = {};
        load8(reinterpret_cast<const bf16*>(&v[i]), t);
        load8(p.norm_w + c * 8, g);
        if (p.norm_b) load8(p.norm_b + c * 8, o);
#pragma unroll
        for (int j = 0; j < 8; ++j)
          y[j] = p.norm == RB_NORM_LAYER ? g[j] * ((t[j] - mean) * scale) + o[j]
                 : p.norm == RB_NORM_RMS ? g[j] * t[j] * scale : t[j] * scale * (g[j] + 1.0f);
      }
      store8(reinterpret_cast<bf16*>(x_s + row * p.pitch + c * 16), y);
    }
  }
  __syncthreads();

  // ---- tiles
  const uint8_t* x_row = x_s + r * p.pitch + q * 16;
  const bool have = r < p.m;
  int slot = 0, flip = 0;
  for (int tile = (int)blockIdx.x + group * (int)gridDim.x; tile < tiles; tile += step, flip ^= 1) {
    // what the end of the tile needs, while its products run: lane e (of the tile's warps) finishes sum e
    const int e0 = part * 32 + lane, stride = share * 32;
    float extra[2] = {0.f, 0.f};
    if (!GATED) {
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int e = e0 + j * stride, col = tile * 8 + (e & 7);
        if (e < p.m * 8 && col < p.n) {
          if (p.residual) extra[j] = __bfloat162float(p.residual[(size_t)(e >> 3) * p.n + col]);
        }
      }
    }
    float acc[2][G][4] = {};   // two chains
    for (int t = 0; t < turns; ++t) {
      copies_left<kTurns - 1>();
      const uint8_t* w_s = ring_p + slot * kTurnSlices * 512;
      const int s0 = first + t * U;
      auto product = [&](int u) {
        uint4 x = make_uint4(0, 0, 0, 0);
        if (have) x = *reinterpret_cast<const uint4*>(x_row + (s0 + u) * 64);
#pragma unroll
        for (int g = 0; g < G; ++g) {
          const uint4 b = *reinterpret_cast<const uint4*>(w_s + (g * U + u) * 512);
          mma_rows(acc[0][g], x.x, x.y, b.x, b.y);
          mma_rows(acc[1][g], x.z, x.w, b.z, b.w);
        }
      };
      if (s0 + U <= limit) {
#pragma unroll
        for (int u = 0; u < U; ++u) product(u);
      } else {
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (s0 + u < limit) product(u);
      }
      request();
      if (++slot == kTurns) slot = 0;
    }
    // the warps of a tile add their sums in a fixed order; the slots are free again two tiles later
#pragma unroll
    for (int g = 0; g < G; ++g) {
      red[flip][warp][g][r * 8 + q * 2] = acc[0][g][0] + acc[1][g][0];
      red[flip][warp][g][r * 8 + q * 2 + 1] = acc[0][g][1] + acc[1][g][1];
    }
    if (share > 1) asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "r"(share * 32) : "memory");
    else __syncwarp();
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int e = e0 + j * stride, row = e >> 3, col = tile * 8 + (e & 7);
      if (e >= p.m * 8 || col >= p.n) continue;
      float v = 0.f, v2 = 0.f;
      for (int s = 0; s < share; ++s) {
        v += red[flip][group * share + s][0][e];
        if (GATED) v2 += red[flip][group * share + s][G - 1][e];
      }
      const size_t o = (size_t)row * p.n + col;
      if (p.out_f) { p.out_f[o] = v; continue; }
      if (GATED) {
        v = act_apply(p.act, v) * v2;
      } else {
        if (p.bias) v += __bfloat162float(p.bias[col]);
        v = act_apply(p.act, v) + extra[j];
      }
      p.out[o] = __float2bfloat16_rn(v);
    }
    if (share == 1) __syncwarp();
  }
  copies_left<0>();
}

int pitch_of(int64_t k) {   // rows of X: two neighbours' 16-byte reads fall on different banks
  const int bytes = (int)((k + 31) / 32 * 64);
  return bytes % 128 == 64 ? bytes : bytes + 64;
}

}  // namespace

// Rows of 16-byte pieces, X in shared memory, and (with a norm) a row in the registers of its warps.
bool gemm_rows_takes(int64_t m, int64_t k, bool norm) {
  return m >= 1 && m <= 8 && k >= 8 && k % 8 == 0 && m * pitch_of(k) + kRingBytes <= kMostBytes &&
         (!norm || (k + 31) / 32 * 4 <= (int64_t)kNormPieces * 32 * (kWarps / m));
}

// Layered designs' products, by their size.  With the norm that reads it, alone in a chain of its like, a product of 2 MB takes 4.5 us
// against 6.0 with split K and slabs for the consumer to sum, of 8 MB 5.2 against 6.5, of 20 MB 8.9 against 9.6, of 36 MB 15.3
// against 14.3 (one row).  Between larger products that split K, one of one to three rows and many features either way costs more than
// that: a step of malasun-2k (2048 x 2048, 8 MB) with one row 618 -> 632 us at 128 keys, 641 -> 667 at 1500, of votapel-2k 824 -> 852.  From
// four rows on it gains: malasun-2k, six rows at 1500 keys, 691 -> 673, fizadra-2k, four rows, 915 -> 893, kufulix-2k 973 -> 948.
bool gemm_rows_pays(const rb_ctx* ctx, int64_t m, int64_t n, int64_t k) {
  return !ctx->debug_simple && !ctx->debug_simple_gemm && gemm_rows_takes(m, k, false) && n * k * 2 <= (20 << 20) &&
         (m >= 4 || std::min(n, k) <= 1024);
}

int gemm_rows(rb_ctx* ctx, const RowsArgs& a) {
  RB_REQUIRE(gemm_rows_takes(a.m, a.k, a.norm >= 0) && a.n > 0, "GEMM: %lld rows of %lld", (long long)a.m, (long long)a.k);
  RowsParams p{};
  p.x = (const bf16*)a.x; p.w = (const bf16*)a.w; p.w2 = (const bf16*)a.w2; p.bias = (const bf16*)a.bias;
  p.residual = (const bf16*)a.residual; p.norm_w = (const bf16*)a.norm_w; p.norm_b = (const bf16*)a.norm_b;
  p.out = (bf16*)a.out; p.out_f = a.out_f;
  p.m = (int)a.m; p.n = (int)a.n; p.k = (int)a.k; p.act = a.act; p.norm = a.norm; p.eps = a.eps;
  p.pitch = pitch_of(a.k);
  const int tiles = (p.n + 7) / 8, grid = std::min(tiles, ctx->sm_count), each = (tiles + grid - 1) / grid;
  p.share = each >= 5 ? 1 : each >= 3 ? 2 : each == 2 ? 4 : 8;   // all of an SM's tiles at once, up to eight
  const size_t smem = (size_t)kRingBytes + p.m * p.pitch;
  auto kern = a.w2 ? gemm_rows_kernel<true> : gemm_rows_kernel<false>;
  static bool attr_set[2][64] = {};  // the attribute belongs to the (kernel, device) pair
  bool& set = attr_set[a.w2 ? 1 : 0][ctx->device & 63];
  if (!set) {
    RB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kMostBytes));
    set = true;
  }
  RB_CUDA(launch_kernel(kern, dim3((unsigned)grid), dim3(kWarps * 32), smem, ctx->stream, ctx->pdl, p));
  ctx->launches++;
  return RB_OK;
}

}  // namespace rb
