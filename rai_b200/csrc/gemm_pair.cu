// bf16 GEMM of prompts (M > 256): C[M,N] = X[M,K] . W[N,K]^T on pairs of SMs (tcgen05, cta_group::2).
//
// A cluster of two CTAs works on one tile of MT (256 or 512) rows of X by 256 rows of W.  Each CTA brings MT / 2 rows of X and
// half of the W rows into its own shared memory; the tensor cores of both SMs read both halves of W.  What bounds this product
// is the traffic of a CTA's shared memory: per 128 cycles of the tensor cores (256 x 256 x 16 over the pair) it is read 8 KB
// and written 8 KB with MT = 256, 6 KB with MT = 512 (two products share a slice of W); one SM alone on a 128 x 256 tile is
// read and written 12 KB each.
//
// The roles are those of gemm_tc.cu: warp 0 of each CTA is its TMA producer (both CTAs' copies are counted on the barrier of
// the leader, CTA 0), warp 1 of the leader issues the MMAs, warps 2-9 are each CTA's epilogue for its own rows.  Two
// accumulators of 256 columns fill the tensor memory: the two halves of a 512-row tile, or two tiles of 256 rows.  An epilogue
// warp has 32 rows x 128 columns and gives the accumulator back once the last of them are in registers; with MT = 512 the
// products of the first half run ahead while the second half is still drained.
//
// Persistent: 74 clusters stride over the tiles.  Where the tiles do not fill the last round and the caller has lent a workspace
// (ctx.h), that round's tiles are cut along K in equal shares for all clusters and done first: a cluster's share is the end of one
// tile and perhaps the start of the next.  Which tiles are cut, and so the order of their sums, depends on the sizes alone.  Whoever has a tile's end finishes it, with the float32 sums that the others (all of them clusters before it, none of which
// waits for anyone, and each does the start of a tile first) left in global memory, added in a fixed order.
//
// GATED computes act(X.Wg^T) * (X.Wu^T): a CTA's half of the W rows is 64 gate rows above the same 64 up rows, so one MMA
// covers both and a column's gate and up sums lie 64 apart in the same lane.
//
// Measured against the one-SM kernel before it, a cool chip each time (M x N x K, us): 32768 x 3584 x 18944 3530 -> 2924, gated
// 32768 x 18944 x 3584 7980 -> 6061 (1468 TFLOP/s of 1636 measured in bursts), 8192 x 9216 x 3072 350 -> 326, 4096 x 2560 x 10240 204 -> 159,
// gated 3003 x 16384 x 2048 353 -> 290, 1000 x 896 x 896 25 -> 12.5.
//
// The epilogue turns rows into whole 128-byte pieces through shared memory, residual rows on their way in and results on
// their way out; sums stay in float32 until the one rounding.
#include <math.h>

#include <algorithm>

#include "ctx.h"
#include "gemm_epilogue.cuh"
#include "ptx.cuh"

namespace rb {

using bf16 = __nv_bfloat16;

namespace {

constexpr int kBN = 256, kHalfM = 128, kBK = 64;
constexpr int kEpiWarps = 8;
constexpr int kThreads = 64 + kEpiWarps * 32;
constexpr int kTurnBytes = 32 * 128;      // per epilogue warp: 32 rows of 128 bytes
constexpr int kBBytes = kBN / 2 * kBK * 2;
constexpr int kRingBytes = 192 * 1024;
constexpr int kSmemBytes = kRingBytes + kEpiWarps * kTurnBytes + 1024;
constexpr int kTmemCols = 512;

struct PairParams {
  int m, n;
  int n_p, n_q, tiles;   // tiles of MT rows, tiles of 256 W rows
  int num_kb;
  int cut_tiles, cut_clusters;  // the first cut_tiles tiles are shared out among that many clusters
  const bf16* bias;
  const bf16* residual;
  bf16* out;
  int act;
  const bf16* act_params;
  float* slabs;          // [cluster][rank][MT / 256][epilogue warp][128 columns][32 rows]
  uint32_t* flags;       // [cluster][rank][MT / 256][epilogue warp]
  long long wait_cycles;
  uint32_t* status;
};

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// the address of the same variable in the leader's shared memory
__device__ __forceinline__ uint32_t leader_addr(const void* p) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(ptx::smem_u32(p)));
  return r;
}
__device__ __forceinline__ void arrive_remote(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void load_2d_pair(void* dst, const CUtensorMap* m, uint32_t bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(
          ptx::smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(m)), "r"(bar), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void umma_pair(uint32_t d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t"
      "}\n" ::"r"(d),
      "l"(da), "l"(db), "r"(idesc), "r"(accumulate)
      : "memory");
}
// arrives on the barrier of both CTAs once every MMA issued so far has completed
__device__ __forceinline__ void commit_both(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
                   ptx::smem_u32(bar)),
               "h"((uint16_t)3)
               : "memory");
}

// A stretch of K blocks of one tile.
struct Work {
  int tile, kb0, kb1;
  int first_helper, last_helper;   // clusters whose sums of the tile's earlier K blocks are to be added: [first, last)
  bool help;                       // not the tile's end: the sums go to this cluster's slab
};

// The i-th stretch of a cluster: its share of the tiles that are cut, then whole tiles.  False: there is none.
__device__ __forceinline__ bool work_item(const PairParams& p, int cluster, int n_clusters, int i, Work& w) {
  w.first_helper = w.last_helper = 0;
  w.help = false;
  int done = 0;
  if (cluster < p.cut_clusters) {
    const int units = p.cut_tiles * p.num_kb;
    auto start = [&](int c) { return (int)((long long)c * units / p.cut_clusters); };
    const int u0 = start(cluster), u1 = start(cluster + 1), tile = u0 / p.num_kb, end = (tile + 1) * p.num_kb;
    const bool next = u1 > end;
    done = next ? 2 : 1;
    if (i < done) {
      if (next && i == 0) {           // the start of the next tile goes first: others wait for it
        w.tile = tile + 1; w.kb0 = 0; w.kb1 = u1 - end; w.help = true;
        return true;
      }
      w.tile = tile; w.kb0 = u0 - tile * p.num_kb; w.kb1 = min(u1, end) - tile * p.num_kb;
      w.help = u1 < end;
      if (!w.help && w.kb0 > 0) {
        w.last_helper = cluster;
        w.first_helper = cluster - 1;
        while (start(w.first_helper) > tile * p.num_kb) --w.first_helper;
      }
      return true;
    }
  }
  w.tile = p.cut_tiles + cluster + (i - done) * n_clusters;
  w.kb0 = 0;
  w.kb1 = p.num_kb;
  return w.tile < p.tiles;
}

// Tiles along P are grouped so that clusters at work share operand tiles in L2 (about as many rows of X as of W).
template <int MT>
__device__ __forceinline__ void tile_at(const PairParams& p, int tile, int& pt, int& qt) {
  constexpr int G = MT == 512 ? 6 : 8;
  const int per_group = G * p.n_q;
  const int group = tile / per_group, first = group * G, in_group = tile % per_group;
  const int gsz = min(p.n_p - first, G);
  pt = first + in_group % gsz;
  qt = in_group / gsz;
}

template <int MT, bool GATED>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_w,
                 const __grid_constant__ CUtensorMap tm_w2, const PairParams p) {
  constexpr int MB = MT / 256;                      // accumulators per tile
  constexpr int kABytes = MB * kHalfM * kBK * 2;
  constexpr int kStageBytes = kABytes + kBBytes;
  constexpr int kStages = kRingBytes / kStageBytes;
  constexpr int kOut = GATED ? kBN / 2 : kBN;       // output columns of a tile
  constexpr int kChunks = GATED ? 1 : 2;            // 64 output columns per turn of an epilogue warp
  constexpr int kCols = 128 / kChunks;              // out of so many accumulator columns
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t full_bar[kStages];    // the leader's count both CTAs' copies
  __shared__ __align__(8) uint64_t empty_bar[kStages];
  __shared__ __align__(8) uint64_t acc_full[2];
  __shared__ __align__(8) uint64_t acc_empty[2];         // the leader's count both CTAs' epilogue warps
  __shared__ uint32_t tmem_base_slot;
  __shared__ volatile uint32_t abort_flag;
  __shared__ uint32_t issued_count;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  const int cluster = blockIdx.x >> 1, n_clusters = gridDim.x >> 1;
  uint8_t* tiles = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) { ptx::mbar_init(&full_bar[s], 1); ptx::mbar_init(&empty_bar[s], 1); }
    for (int a = 0; a < 2; ++a) { ptx::mbar_init(&acc_full[a], 1); ptx::mbar_init(&acc_empty[a], 2 * kEpiWarps); }
    abort_flag = 0;
    issued_count = 0;
    ptx::fence_barrier_init();
    ptx::fence_proxy_async();
    ptx::tma_prefetch_desc(&tm_x);
    ptx::tma_prefetch_desc(&tm_w);
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(ptx::smem_u32(&tmem_base_slot)),
                 "r"((uint32_t)kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  ptx::tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // the leader's barriers exist before the other CTA's copies are counted on them
  ptx::tc_fence_after();
  const uint32_t tmem_base = tmem_base_slot;
  pdl_launch_dependents();

  Work w;
  int pt, qt;
  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer of this CTA's operand rows
    if (lane == 0) {
      auto load_w = [&](uint8_t* st, uint32_t bar, int kb) {
        uint8_t* b = st + kABytes;
        if (GATED) {
          const int row = qt * kOut + (int)rank * (kBN / 4);
          load_2d_pair(b, &tm_w, bar, kb * kBK, row);
          load_2d_pair(b + kBBytes / 2, &tm_w2, bar, kb * kBK, row);
        } else {
          load_2d_pair(b, &tm_w, bar, kb * kBK, qt * kBN + (int)rank * (kBN / 2));
        }
      };
      // the first ring of weights does not wait for the kernel before this one
      int n_pre = 0;
      for (int i = 0; n_pre < kStages && work_item(p, cluster, n_clusters, i, w); ++i) {
        tile_at<MT>(p, w.tile, pt, qt);
        for (int kb = w.kb0; kb < w.kb1 && n_pre < kStages; ++kb, ++n_pre) {
          if (rank == 0) ptx::mbar_expect_tx(&full_bar[n_pre], 2 * kStageBytes);
          load_w(tiles + (size_t)n_pre * kStageBytes, leader_addr(&full_bar[n_pre]), kb);
        }
      }
      pdl_wait();
      int stage = 0, issued = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int i = 0; ok && work_item(p, cluster, n_clusters, i, w); ++i) {
        tile_at<MT>(p, w.tile, pt, qt);
        const int row = pt * MT + (int)rank * kHalfM;
        for (int kb = w.kb0; kb < w.kb1; ++kb) {
          uint8_t* st = tiles + (size_t)stage * kStageBytes;
          const uint32_t bar = leader_addr(&full_bar[stage]);
          if (issued >= n_pre) {
            if (!ptx::mbar_wait(&empty_bar[stage], phase ^ 1u, &abort_flag, p.wait_cycles)) { ok = false; break; }
            if (rank == 0) ptx::mbar_expect_tx(&full_bar[stage], 2 * kStageBytes);
            load_w(st, bar, kb);
          }
#pragma unroll
          for (int b = 0; b < MB; ++b) load_2d_pair(st + b * kHalfM * kBK * 2, &tm_x, bar, kb * kBK, row + b * 256);
          ++issued;
          if (++stage == kStages) { stage = 0; phase ^= 1u; }
        }
      }
      issued_count = (uint32_t)issued;
      // the leader's commits of the last ring are counted in this CTA's shared memory, and nothing else waits for them
      for (int i = 0; ok && i < kStages; ++i) {   // (a stage that was never filled: its barrier's phase before the first)
        ok = ptx::mbar_wait(&empty_bar[stage], phase ^ 1u, &abort_flag, p.wait_cycles);
        if (++stage == kStages) { stage = 0; phase ^= 1u; }
      }
      if (!ok) { p.status[0] = (uint32_t)(-RB_ERR_TIMEOUT); p.status[1] = 0x6E11u; p.status[2] = blockIdx.x; }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (the leader's)
    if (rank == 0 && lane == 0) {
      constexpr uint32_t idesc = ptx::umma_idesc_bf16(256, kBN);
      int stage = 0, as = 0;
      uint32_t phase = 0, aphase = 0;
      bool ok = true;
      auto products = [&](int st_i, int b, uint32_t d, bool first) {
        const uint32_t st = ptx::smem_u32(tiles + (size_t)st_i * kStageBytes), x = st + b * kHalfM * kBK * 2, wt = st + kABytes;
#pragma unroll
        for (int j = 0; j < kBK / 16; ++j)
          umma_pair(d, ptx::umma_desc_k_sw128(x + j * 32), ptx::umma_desc_k_sw128(wt + j * 32), idesc, (!first || j > 0) ? 1u : 0u);
      };
      auto wait_full = [&](int st_i, uint32_t ph) {
        if (!ptx::mbar_wait(&full_bar[st_i], ph, &abort_flag, p.wait_cycles)) return false;
        ptx::tc_fence_after();
        return true;
      };
      for (int i = 0; ok && work_item(p, cluster, n_clusters, i, w); ++i) {
        if (MB == 1) {
          if (!ptx::mbar_wait(&acc_empty[as], aphase ^ 1u, &abort_flag, p.wait_cycles)) { ok = false; break; }
          ptx::tc_fence_after();
          for (int kb = w.kb0; kb < w.kb1; ++kb) {
            if (!wait_full(stage, phase)) { ok = false; break; }
            products(stage, 0, tmem_base + (uint32_t)(as * kBN), kb == w.kb0);
            commit_both(&empty_bar[stage]);
            if (++stage == kStages) { stage = 0; phase ^= 1u; }
          }
          if (!ok) break;
          commit_both(&acc_full[as]);
          if (++as == 2) { as = 0; aphase ^= 1u; }
        } else {
          if (!ptx::mbar_wait(&acc_empty[0], aphase ^ 1u, &abort_flag, p.wait_cycles)) { ok = false; break; }
          ptx::tc_fence_after();
          // the first half's products of a ring of stages, then, its accumulator free, the second half's
          const int head = min(w.kb1 - w.kb0, kStages);
          int s2 = stage;
          uint32_t ph2 = phase;
          for (int k = 0; k < head; ++k) {
            if (!wait_full(s2, ph2)) { ok = false; break; }
            products(s2, 0, tmem_base, k == 0);
            if (++s2 == kStages) { s2 = 0; ph2 ^= 1u; }
          }
          if (!ok) break;
          if (!ptx::mbar_wait(&acc_empty[1], aphase ^ 1u, &abort_flag, p.wait_cycles)) { ok = false; break; }
          ptx::tc_fence_after();
          for (int k = 0; k < head; ++k) {
            products(stage, 1, tmem_base + kBN, k == 0);
            commit_both(&empty_bar[stage]);
            if (++stage == kStages) { stage = 0; phase ^= 1u; }
          }
          for (int kb = w.kb0 + head; kb < w.kb1; ++kb) {
            if (!wait_full(stage, phase)) { ok = false; break; }
            products(stage, 0, tmem_base, false);
            if (kb == w.kb1 - 1) commit_both(&acc_full[0]);
            products(stage, 1, tmem_base + kBN, false);
            commit_both(&empty_bar[stage]);
            if (++stage == kStages) { stage = 0; phase ^= 1u; }
          }
          if (!ok) break;
          if (head == w.kb1 - w.kb0) commit_both(&acc_full[0]);
          commit_both(&acc_full[1]);
          aphase ^= 1u;
        }
      }
      if (!ok) { p.status[0] = (uint32_t)(-RB_ERR_TIMEOUT); p.status[1] = 0x6E12u; p.status[2] = blockIdx.x; }
    }
  } else {
    // ------------------------------------------------------------------ epilogue of this CTA's rows
    pdl_wait();
    const int quarter = warp & 3;           // the 32 TMEM lanes this warp may read
    const int half = (warp - 2) >> 2;       // which 128 of the accumulator's columns it takes
    uint8_t* turn = tiles + kRingBytes + (warp - 2) * kTurnBytes;
    auto slot = [&](int row, int piece) { return reinterpret_cast<uint4*>(turn + row * 128 + ((piece ^ (row & 7)) << 4)); };
    const float2 ac = p.act == RB_ACT_XIELU ? xielu_consts(p.act_params) : make_float2(0.f, 0.f);
    const bool vec_ok = (p.n % 8) == 0;
    const bool add_residual = !GATED && p.residual && vec_ok;
    // residual pieces of the next 64 columns, on their way while the accumulator is waited for
    auto fetch = [&](int row0, int gn0) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int r = i * 4 + lane / 8, c = gn0 + lane % 8 * 8;
        if (row0 + r < p.m && c < p.n)
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(ptx::smem_u32(slot(r, lane % 8))),
                       "l"(p.residual + (size_t)(row0 + r) * p.n + c)
                       : "memory");
      }
    };
    auto slab_of = [&](int c, size_t place) {
      return reinterpret_cast<float4*>(p.slabs) + ((size_t)c * 2 * MB * kEpiWarps + place) * (32 * 32) + lane;
    };
    auto flag_of = [&](int c, size_t place) { return p.flags + (size_t)c * 2 * MB * kEpiWarps + place; };
    const uint32_t acc_empty_leader[2] = {leader_addr(&acc_empty[0]), leader_addr(&acc_empty[1])};
    int as = 0;
    uint32_t aphase = 0;
    bool ok = true;
    for (int i = 0; ok && work_item(p, cluster, n_clusters, i, w); ++i) {
      tile_at<MT>(p, w.tile, pt, qt);
#pragma unroll 1
      for (int b = 0; b < MB; ++b) {
        const int row0 = pt * MT + b * 256 + (int)rank * kHalfM + quarter * 32;   // first of this warp's rows
        const int col0 = qt * kOut + half * (kOut / 2);                           // and of its columns
        const bool wanted = row0 < p.m && col0 < p.n;
        if (add_residual && wanted && !w.help) fetch(row0, col0);
        ok = ptx::mbar_wait(&acc_full[as], aphase, &abort_flag, p.wait_cycles);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        ptx::tc_fence_after();
        const uint32_t at = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(as * kBN + half * 128);
        const size_t place = ((size_t)rank * MB + b) * kEpiWarps + (warp - 2);   // of this warp's sums in a cluster's slab
        const int gm = row0 + lane;
#pragma unroll 1
        for (int ch = 0; ch < kChunks; ++ch) {
          float v[kCols];
#pragma unroll
          for (int c = 0; c < kCols; c += 32) ptx::tmem_ld_32x32(at + ch * kCols + c, reinterpret_cast<uint32_t(&)[32]>(v[c]));
          ptx::tmem_wait_ld();
          if (ch == kChunks - 1) {
            ptx::tc_fence_before();
            __syncwarp();
            if (lane == 0) arrive_remote(acc_empty_leader[as]);
          }
          if (w.help) {
            float4* s = slab_of(cluster, place) + ch * (kCols / 4) * 32;
#pragma unroll
            for (int c = 0; c < kCols / 4; ++c) __stcg(s + c * 32, make_float4(v[c * 4], v[c * 4 + 1], v[c * 4 + 2], v[c * 4 + 3]));
            continue;
          }
          for (int h = w.first_helper; h < w.last_helper; ++h) {
            uint32_t* flag = flag_of(h, place);
            if (ch == 0 && lane == 0) {
              uint32_t seen = 0;
              const long long t0 = clock64();
              while (true) {
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(flag) : "memory");
                if (seen || abort_flag) break;
                if (clock64() - t0 > p.wait_cycles) { abort_flag = 1u; break; }
              }
              ok = seen != 0;
              *flag = 0;
            }
            __syncwarp();   // what lane 0 acquired is there for the other lanes' loads (a shuffle orders no memory)
            ok = __shfl_sync(0xffffffffu, ok, 0);
            if (!ok) break;
            const float4* s = slab_of(h, place) + ch * (kCols / 4) * 32;
#pragma unroll
            for (int c0 = 0; c0 < kCols / 4; c0 += 8) {
              float4 t[8];
#pragma unroll
              for (int c = 0; c < 8; ++c) t[c] = __ldcg(s + (c0 + c) * 32);
#pragma unroll
              for (int c = 0; c < 8; ++c) {
                float* a = v + (c0 + c) * 4;
                a[0] += t[c].x; a[1] += t[c].y; a[2] += t[c].z; a[3] += t[c].w;
              }
            }
          }
          const int gn0 = col0 + ch * 64;
          if (!ok || !wanted || gn0 >= p.n) continue;
          // (each step over all 64 columns: the selectors between them are branched on once)
          if constexpr (GATED) {
            act_inplace(p.act, reinterpret_cast<float(&)[64]>(v), ac);
#pragma unroll
            for (int j = 0; j < 64; ++j) v[j] *= v[kCols - 64 + j];
          } else {
            if (p.bias) {
#pragma unroll
              for (int j8 = 0; j8 < 64; j8 += 8) {
                if (vec_ok) {
                  float b8[8] = {};
                  if (gn0 + j8 < p.n) unpack8(*reinterpret_cast<const uint4*>(p.bias + gn0 + j8), b8);
#pragma unroll
                  for (int j = 0; j < 8; ++j) v[j8 + j] += b8[j];
                } else {
#pragma unroll
                  for (int j = 0; j < 8; ++j)
                    if (gn0 + j8 + j < p.n) v[j8 + j] += __bfloat162float(p.bias[gn0 + j8 + j]);
                }
              }
            }
            if (p.act != RB_ACT_NONE) act_inplace(p.act, reinterpret_cast<float(&)[64]>(v), ac);
          }
          if (!vec_ok) {   // rows that are not made of 16-byte pieces
            if (gm < p.m) {
#pragma unroll
              for (int j = 0; j < 64; ++j) {
                if (gn0 + j >= p.n) break;
                const size_t o = (size_t)gm * p.n + gn0 + j;
                p.out[o] = __float2bfloat16_rn(!GATED && p.residual ? v[j] + __bfloat162float(p.residual[o]) : v[j]);
              }
            }
            continue;
          }
          if (add_residual) {
            if (ch > 0) fetch(row0, gn0);
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncwarp();
#pragma unroll
            for (int j8 = 0; j8 < 64; j8 += 8) {
              float r8[8];
              unpack8(*slot(lane, j8 / 8), r8);
#pragma unroll
              for (int j = 0; j < 8; ++j) v[j8 + j] += r8[j];
            }
          }
#pragma unroll
          for (int j8 = 0; j8 < 64; j8 += 8) *slot(lane, j8 / 8) = pack8(v + j8);
          __syncwarp();
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const int r = j * 4 + lane / 8, c = lane % 8;
            if (row0 + r < p.m && gn0 + c * 8 < p.n)
              *reinterpret_cast<uint4*>(p.out + (size_t)(row0 + r) * p.n + gn0 + c * 8) = *slot(r, c);
          }
          __syncwarp();
        }
        if (w.help) {
          __threadfence();
          __syncwarp();
          if (lane == 0) asm volatile("st.release.gpu.global.u32 [%0], 1;" ::"l"(flag_of(cluster, place)) : "memory");
        }
        if (++as == 2) { as = 0; aphase ^= 1u; }
        if (!ok) break;
      }
    }
    if (!ok && lane == 0) { p.status[0] = (uint32_t)(-RB_ERR_TIMEOUT); p.status[1] = 0x6E13u; p.status[2] = blockIdx.x; }
  }

  // ------------------------------------------------------------------ teardown
  ptx::tc_fence_before();
  __syncthreads();
  if (abort_flag && threadIdx.x == 0) {
    // copies already handed to the copy engine get a bounded time to land: the leader can see its stages fill, the other CTA
    // (whose copies the leader's barriers count) only waits
    volatile uint32_t never = 0;
    const uint32_t issued = issued_count;
    for (uint32_t i = (issued > kStages ? issued - kStages : 0); rank == 0 && i < issued; ++i)
      ptx::mbar_wait(&full_bar[i % kStages], (i / kStages) & 1u, &never, p.wait_cycles);
    const long long t0 = clock64();
    while (clock64() - t0 < 1000000) {}
  }
  __syncthreads();
  cluster_sync_all();  // neither CTA leaves while the other may still reach its memory; every wait before this one is bounded
  if (warp == 1) {
    __syncwarp();
    ptx::tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)kTmemCols) : "memory");
  }
}

int most_clusters(const rb_ctx* ctx) { return std::min(ctx->sm_count / 2, kPairClusters); }

// How a product is shared out with tiles of mt rows, and what that costs in K blocks of a 256-row tile (about 0.25 us alone,
// 0.45 us with the whole GPU at work).  A 512-row tile's block costs 1.9 of them, and its second accumulator's epilogue about 10.
// The round that the tiles do not fill is cut along K when that is cheaper than a round of whole tiles: a helper's sums
// cost about 2.5 blocks to move, and waiting for them 10, or 30 where no whole tile follows that hides it.  Measured
// (us, whole tiles only -> with the cut): 4096 x 2560 x 2560 71 -> 55, 8192 x 3072 x 8192 345 -> 313, 3003 x 2048 x 16384
// 185 -> 161, 300 x 3584 x 18944 106 -> 61; 1000 x 3584 x 3584, where the rule keeps whole tiles, 28 -> 32.
// 256- against 512-row tiles: 32768 x 2 x 18944 x 3584 (gated) 7190 / 6370, 9000 x 2048 x 8192 260 / 237, 8192 x 3072 x 8192 346 / 313,
// but 2100 x 4608 x 3584 62 / 93 and 4096 x 2560 x 10240 175 / 217.
struct Split {
  int n_q = 0, cut = 0, shares = 0;   // tiles of W rows; tiles that are cut, and among how many clusters
  double cost = 0.0;
};
Split plan_split(const rb_ctx* ctx, int m, int n_out, int out_cols, int num_kb, int mt) {
  Split s;
  const int most = most_clusters(ctx);
  s.n_q = (n_out + out_cols - 1) / out_cols;
  const int64_t tiles = (int64_t)((m + mt - 1) / mt) * s.n_q;
  const int left = (int)(tiles % most);
  const int64_t rounds = tiles / most;
  double last = left > 0 ? num_kb : 0.0;
  if (left > 0 && ctx->pair_space) {
    const double move = 2.5, wait = (rounds > 0 ? 10.0 : 30.0) * 256 / mt;
    const double each = std::max(1.0, std::min((double)most / left, sqrt(num_kb / move)));   // clusters per cut tile
    const int shares = std::min(most, (int)(left * each));
    const double cut = (double)left * num_kb / shares + move * (shares / left) + wait;
    if (shares > left && cut < last) {
      s.cut = left;
      s.shares = shares;
      last = cut;
    }
  }
  s.cost = ((double)rounds * num_kb + last) * (mt == 512 ? 1.9 : 1.0) + (mt == 512 ? 10.0 : 0.0);
  return s;
}

template <int MT, bool GATED>
int launch_pair(rb_ctx* ctx, const GemmArgs& a, PairParams& p, const Split& split) {
  CUtensorMap tx, tw, tw2;
  constexpr int w_box = GATED ? kBN / 4 : kBN / 2;
  RB_TRY(tmap_2d_bf16(ctx, a.x, a.m, a.k, a.k, kHalfM, &tx));
  RB_TRY(tmap_2d_bf16(ctx, a.w, a.n, a.k, a.k, w_box, &tw));
  RB_TRY(tmap_2d_bf16(ctx, GATED ? a.w2 : a.w, a.n, a.k, a.k, w_box, &tw2));
  auto kern = gemm_pair_kernel<MT, GATED>;
  static bool attr_set[64] = {};  // the attribute belongs to the (kernel, device) pair
  const int dv = ctx->device & 63;
  if (!attr_set[dv]) {
    RB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes));
    attr_set[dv] = true;
  }
  p.n_p = (p.m + MT - 1) / MT;
  p.n_q = split.n_q;
  p.tiles = p.n_p * p.n_q;
  int clusters = std::min(p.tiles, most_clusters(ctx));
  p.cut_tiles = split.cut;
  p.cut_clusters = split.shares;
  if (split.shares > 0) {
    p.slabs = ctx->pair_space->slabs;
    p.flags = ctx->pair_space->flags;
    clusters = std::max(clusters, split.shares);
  }
  RB_CUDA(launch_kernel(kern, dim3((unsigned)(2 * clusters)), dim3(kThreads), kSmemBytes, ctx->stream, ctx->pdl, tx, tw, tw2, p));
  ctx->launches++;
  return RB_OK;
}

}  // namespace

int gemm_pair_bf16(rb_ctx* ctx, const GemmArgs& a, int tile_rows) {
  PairParams p{};
  p.m = (int)a.m;
  p.n = (int)a.n;
  p.num_kb = (int)((a.k + kBK - 1) / kBK);
  p.bias = (const bf16*)a.bias;
  p.residual = (const bf16*)a.residual;
  p.out = (bf16*)a.out;
  p.act = a.act;
  p.act_params = (const bf16*)a.act_params;
  p.status = ctx->status_dev;
  p.wait_cycles = ctx->local_wait_cycles();
  const int out_cols = a.w2 ? kBN / 2 : kBN;
  const Split narrow = plan_split(ctx, p.m, p.n, out_cols, p.num_kb, 256), wide = plan_split(ctx, p.m, p.n, out_cols, p.num_kb, 512);
  if (tile_rows == 512 || (tile_rows == 0 && wide.cost < narrow.cost))
    return a.w2 ? launch_pair<512, true>(ctx, a, p, wide) : launch_pair<512, false>(ctx, a, p, wide);
  return a.w2 ? launch_pair<256, true>(ctx, a, p, narrow) : launch_pair<256, false>(ctx, a, p, narrow);
}

}  // namespace rb
