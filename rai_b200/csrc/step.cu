// One kernel for all layers of a single-token step of at most eight sequences: Model::fwd of rai-models/src/llm/{qwen2,phi2,phi3,
// gemma}.rs at sequence length 1, from the embedded rows to the logits.
//
// What bounds such a step beside its bytes is the hand-overs between the products, the attention and the norms of a layer: as
// launches of their own each costs 4 to 8 us from the last store of one to the first product of the next, seven to nine times a
// layer.  Here one CTA stays on every SM and the phases of a layer follow one another through grid-wide barriers (five a layer, about 2 us
// each by themselves), while the copies of weights and cached keys and values, which depend on nothing, run ahead through
// all of them: a ring of shared memory (190 KB an SM, 4.5 us of HBM over the GPU) takes the tiles of the next phase while this one
// waits.  us per step of 8 layers and a vocabulary of 1024, seven launches a layer -> here: phi2 (157 MB a layer) 1 x 17 keys 473 -> 349, 8 x 512
// 528 -> 470; phi3-mini (226 MB) 1 x 3500 597 -> 507, 4 x 2048 662 -> 574; qwen2-7b (466 MB) 1 x 17 782 -> 743.  A layer of phi3-mini
// takes 54 us with 17 keys, 35 of them its weights at the copy rate, and 72 with 4 x 2048 keys (50); a further MB of weights costs what HBM
// takes for it (97 -> 145 MB a layer), a further MB of keys and values 5.6 TB/s (8 x 200 -> 8 x 1600).  DRAM reads are 0.5 to 2.5 % above the bytes.
//
//   warp 8      weights, keys and values: TMA tiles into the ring in the order of the program, whatever phase the rest is in
//   warps 9, 10 wait at the barriers; then the activations that belong to each weight tile (a few KB from L2) into the same slot
//   warps 0-7   products (mma.sync), attention, epilogues
//
// Rows of a weight matrix are shared out evenly over the CTAs (3072 rows are 21 each for 147 of 148), so no product is cut along K over CTAs and no
// sums travel between SMs.  (In what order the eight warps' sums meet depends on the rows of the call, and into what pieces the attention is
// cut on all its lengths, so a sequence's last bits may.)  That is also why the products are mma.sync: a
// tile of 128 rows, which tcgen05 wants, would leave most SMs without work or cut K sixfold, and at eight rows of X the tensor cores
// have nothing to do anyway (active 7 to 9 % of the time).  With more rows the activations' way through L2 costs more than the launches did (see step_takes).
//
// A CTA owns the same few columns of the residual stream all through the step and keeps them in shared memory.  The RMS norms need no
// phase of their own: whoever finishes a column of the stream also writes it times the next norm's weight, and its square joins a
// sum per CTA and row; the product that reads the row is scaled afterwards.  (A LayerNorm is a phase: row by row, as its own kernel does it.)
//
// Attention: a pair (sequence, KV head) is walked by one CTA or, where that is shorter, in pieces by several; the one that arrives last
// adds them up, in the order of the pieces.
//
// Tried and left out: the next 40 MB of tiles brought into L2 ahead of the ring by a warp of its own (phi3-mini 4 x 2048 16.2 -> 16.9 ms
// for seven steps); activations asked for by the warp that works on the slot (the same 16.2 -> 16.8); all warps sharing every slot's
// rows (350 ns a slot, whatever was in it); slots of exactly the bytes needed (the account of them costs 300 ns a slot on one thread).
#include <algorithm>
#include <type_traits>

#include "ctx.h"
#include "model.h"
#include "ptx.cuh"
#include "step.h"
#include "step_rule.h"

namespace rb {

using bf16 = __nv_bfloat16;

namespace {

constexpr int kRows = 8;                     // sequences at most: the narrow side of a tensor-core product
constexpr int kMaxSlots = 14;
constexpr int kSlotBytes = 20 * 1024;        // of the ring at most (a tile of 128 rows of W and 8 of X is 17 KB, one of 64 keys 16)
constexpr int kWorkWarps = 8, kThreads = (kWorkWarps + 3) * 32;
constexpr int kReleases = 4;                 // arrivals that free a slot
constexpr int kTiles = 8;                    // of 16 rows of W per slot at most
constexpr int kMergeFloats = 6144;           // at least
constexpr int kMostSmem = 232448 - 3072;      // dynamic; the rest is Shared, aligned
constexpr int kOwnColumns = 64;              // of the stream per CTA at most

// What happens in a layer, in the order of the program: [q/k/v, attention, output projection, up, down], or, where the MLP stands beside
// the attention (phi2), [q/k/v, up, attention, down and output projection].  A step ends with the product with the vocabulary.
enum Op : int { kQkv, kOut, kUp, kDown, kHead, kAttend };
__device__ __forceinline__ int op_at(bool serial, int i) { return (serial ? 0x32150 : 0xf3520) >> (4 * i) & 15; }   // 15: none

struct StepLayerPtrs {
  const bf16 *qkv_b, *o_b, *fc_b, *down_b, *norm1_w, *norm1_b, *norm2_w;
};
// How the rows of a weight matrix are shared out: `passes` tiles of `rows` rows per CTA (gated: of gate and of up each, `parts` 2), `slices`
// times 64 of the `blocks` times 64 columns per slot, `stages` slots in all.
struct StepShare {
  int n, rows, passes, parts, slices, blocks, stages;
};
struct StepParams {
  CUtensorMap w[kStepLayers][4];             // by Op
  CUtensorMap head, k, v;
  CUtensorMap x[5];                          // by Op: what it multiplies
  StepLayerPtrs layer[kStepLayers];
  const bf16 *head_norm_w, *head_norm_b, *head_b;
  StepShare share[5];                        // by Op
  int m, layers, hidden, inter, nqkv, vocab, q_heads, kv_heads, group, rot, max_seq, act, norm, slots, slot_bytes, merge_floats, most_pieces;
  int pages_per_seq, cache_rows;             // cache_rows: rows of 64-key pages per layer
  size_t layer_stride;                       // elements of one layer's pages
  bool want_head;
  float eps, scale_log2;
  float squares_of, squares_over;            // what a column is multiplied by before it is squared, and the sum divided by
  bf16 *h, *hw, *attn, *inner, *logits;
  float *qkv_out, *squares, *part_o, *part_ml;
  bf16 *cache_k, *cache_v;
  const float *cos_t, *sin_t;
  const int32_t *block_table, *seq_lens;
  uint32_t *flags, *split_count, *status;
  long long wait_cycles;
};

__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* m, uint64_t* bar, int x, int y, int z) {
  asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
               ::"r"(dst), "l"(reinterpret_cast<uint64_t>(m)), "r"(ptx::smem_u32(bar)), "r"(x), "r"(y), "r"(z) : "memory");
}
__device__ __forceinline__ void tma_load_3d_hint(uint32_t dst, const CUtensorMap* m, uint64_t* bar, int x, int y, int z, uint64_t policy) {
  asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%3, %4, %5}], [%2], %6;"
               ::"r"(dst), "l"(reinterpret_cast<uint64_t>(m)), "r"(ptx::smem_u32(bar)), "r"(x), "r"(y), "r"(z), "l"(policy) : "memory");
}
__device__ __forceinline__ void ldsm_x4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm_x4_t(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ float ex2(float x) {   // 2^x; what is too small for a normal number is zero
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ void work_sync() { asm volatile("bar.sync 1, 256;" ::: "memory"); }
__device__ __forceinline__ float ldcg(const float* p) { return __ldcg(p); }
__device__ __forceinline__ void ldcg8(const float* p, float* v) {
  const float4 a = __ldcg(reinterpret_cast<const float4*>(p)), b = __ldcg(reinterpret_cast<const float4*>(p) + 1);
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
__device__ __forceinline__ float round_bf16(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }

template <int D>
struct Cfg {
  static constexpr int kKeys = kPageTokens;                // per slot
  static constexpr int kBlocks = (D + 63) / 64;
  static constexpr int kTileBytes = kKeys * kBlocks * 128;
  static constexpr int kWarpsPerTile = kKeys / 16, kGroups = kWorkWarps / kWarpsPerTile;
  static constexpr int kQRow = (D + 8) * 2;                // conflict-free ldmatrix
  static_assert(kTileBytes <= kSlotBytes && kTileBytes % 1024 == 0 && kReleases % kWarpsPerTile == 0, "stage");
};

// The pieces that a CTA walks: piece i of (sequence b, KV head kvh), and how many are left
struct Walk {
  int b, kvh, i, left;
};

// The next slot of the ring: every role counts along for itself.
struct Ring {
  int slot = 0;
  uint32_t parity = 0;
  __device__ __forceinline__ void pass(int slots) {
    if (++slot == slots) { slot = 0; parity ^= 1u; }
  }
  __device__ __forceinline__ void pass(int n, int slots) {
    const int to = slot + n, rounds = to / slots;
    slot = to - rounds * slots;
    parity ^= (uint32_t)rounds & 1u;
  }
};

struct Shared {
  uint64_t full[kMaxSlots], empty[kMaxSlots], go;
  uint32_t abort, last;
  int len[kRows], tiles[kRows], pieces[kRows], piece_tiles[kRows], each;   // pieces of a pair of this sequence, and of a CTA
  float rstd[kRows], sums[2][kWorkWarps], extra[128];
  float mm[kWorkWarps][16], ml[kWorkWarps][16], row_m[16], row_l[16];
};

static_assert(sizeof(Shared) <= 3072, "static shared memory");

// Where a CTA begins its way along K.  (All of them at the same place would ask the same few lines of X of L2 at the same time.)
__device__ __forceinline__ int first_stage(int cta, int ctas, int stages) { return cta * stages / ctas; }
__device__ __forceinline__ void release_slot(uint64_t* bar, int n) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0], %1;" ::"r"(ptx::smem_u32(bar)), "r"(n) : "memory");
}
template <int D>
__global__ void __launch_bounds__(kThreads, 1) step_kernel(const __grid_constant__ StepParams p) {
  using C = Cfg<D>;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  __shared__ Shared sh;
  uint8_t* ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint32_t ring_a = ptx::smem_u32(ring);
  float* merge = reinterpret_cast<float*>(ring + p.slots * p.slot_bytes);   // sums of products, pieces of attention
  float* own = merge + p.merge_floats;                                      // the CTA's columns of the stream [row][column]
  bf16* new_kv = reinterpret_cast<bf16*>(own + kRows * p.share[kOut].rows); // the new token's k row, then its v row
  uint8_t* q_s = reinterpret_cast<uint8_t*>(new_kv + 2 * D);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int cta = blockIdx.x, ctas = gridDim.x;
  const bool serial = p.norm != RB_NORM_LAYER;     // not phi2: RMS norms and a gated MLP behind the attention
  const int slots = p.slots, slot_bytes = p.slot_bytes, m_rows = p.m;
  volatile uint32_t* abort_flag = &sh.abort;

  if (threadIdx.x == 0) {
    for (int s = 0; s < slots; ++s) { ptx::mbar_init(&sh.full[s], 2); ptx::mbar_init(&sh.empty[s], kReleases); }
    ptx::mbar_init(&sh.go, 1);
    sh.abort = 0;
    ptx::fence_barrier_init();
    ptx::fence_proxy_async();
  }
  if (threadIdx.x < kRows) {
    int len = (int)threadIdx.x < p.m ? __ldcg(p.seq_lens + threadIdx.x) : 0;
    if ((int)threadIdx.x < p.m && (len < 1 || len > p.max_seq)) {   // (the guard of the kernels that append to a cache)
      p.status[0] = (uint32_t)(-RB_ERR_INVALID); p.status[1] = 0x57E1u; p.status[2] = (uint32_t)(len - 1);
      len = 0;
    }
    sh.len[threadIdx.x] = len;
    sh.tiles[threadIdx.x] = (len + C::kKeys - 1) / C::kKeys;
  }
  __syncthreads();

  // ---- how the keys are shared out (step_pieces of step_rule.h does the same on the host): all pairs (sequence, KV head) in pieces of at
  // most `most / (lane + 1)` tiles, in a line, the same number of pieces for every CTA.  The cheapest of 16 ways, in units of 0.1 us: a
  // tile 4, a piece 35 (rows in, parts out), cut pairs 25.
  if (warp == 0) {
    int most = 0;
    for (int b = 0; b < m_rows; ++b) most = max(most, sh.tiles[b]);
    const int ways = lane & 15, q = max(1, (most + ways) / (ways + 1));
    int line = 0, widest = 0;
#pragma unroll 1
    for (int b = 0; b < m_rows; ++b) {
      const int t = sh.tiles[b], n = (t + q - 1) / q;
      line += n * p.kv_heads;
      if (n) widest = max(widest, (t + n - 1) / n);
    }
    const int each = (line + ctas - 1) / ctas;
    unsigned cost = (unsigned)(each * (widest * 4 + 35) + (q < most ? 25 : 0));
    if (line > p.most_pieces) cost = 1u << 24;
    const unsigned best = __reduce_min_sync(0xffffffffu, cost << 4 | (unsigned)ways);
    const int q_best = max(1, (most + (int)(best & 15u)) / ((int)(best & 15u) + 1));
    line = 0;
    if (lane < m_rows) {
      const int t = sh.tiles[lane], n = (t + q_best - 1) / q_best;
      sh.pieces[lane] = n;
      sh.piece_tiles[lane] = n ? (t + n - 1) / n : 0;
      line = n * p.kv_heads;
    }
    line = __reduce_add_sync(0xffffffffu, line);
    if (lane == 0) sh.each = (line + ctas - 1) / ctas;
  }
  __syncthreads();
  Walk start{0, 0, 0, 0};
  int stretch = 0;   // tiles
  auto piece_of = [&](const Walk& w, int& first) {   // its first tile and how many there are
    first = w.i * sh.piece_tiles[w.b];
    return min(sh.piece_tiles[w.b], sh.tiles[w.b] - first);
  };
  auto next_piece = [&](Walk& w) {
    --w.left;
    if (++w.i < sh.pieces[w.b]) return;
    w.i = 0;
    if (++w.kvh < p.kv_heads) return;
    w.kvh = 0;
    do ++w.b; while (w.b < m_rows && sh.tiles[w.b] == 0);
  };
  {
    int rem = cta * sh.each;
#pragma unroll 1
    for (int b = 0; b < m_rows; ++b) {
      const int span = sh.pieces[b] * p.kv_heads;
      if (start.left == 0 && rem < span) {
        start.b = b; start.kvh = rem / sh.pieces[b]; start.i = rem % sh.pieces[b];
        start.left = span - rem;
      } else if (start.left > 0) {
        start.left += span;
      }
      rem -= span;
    }
    start.left = min(start.left, sh.each);
    Walk w = start;
    while (w.left > 0) {
      int first;
      stretch += piece_of(w, first);
      next_piece(w);
    }
  }

  Ring r;
  bool ok = true;

  // ================================================================ weights, keys and values
  if (warp == kWorkWarps) {
    if (lane == 0) {
      const uint64_t policy = ptx::policy_evict_first();
      auto acquire = [&]() { return ok = ptx::mbar_wait(&sh.empty[r.slot], r.parity ^ 1u, abort_flag, p.wait_cycles); };
#pragma unroll 1
      for (int l = 0; l <= p.layers && ok; ++l) {
#pragma unroll 1
        for (int i = 0; i < 5 && ok; ++i) {
          const int op = l < p.layers ? op_at(serial, i) : i == 0 && p.want_head ? kHead : 15;
          if (op == 15) break;
          if (op != kAttend) {
            // (the output projection of phi2 follows its down projection)
#pragma unroll 1
            for (int now = op;; now = kOut) {
              const StepShare s = p.share[now];
              const CUtensorMap* map = now == kHead ? &p.head : &p.w[l][now];
              const int stages = s.stages, part = s.slices * s.rows * 128;
#pragma unroll 1
              for (int pass = 0; pass < s.passes; ++pass) {
                const int y = (cta * s.passes + pass) * s.rows;
                if (y >= s.n) break;
                int at = first_stage(cta, ctas, stages);
#pragma unroll 1
                for (int k = 0; k < stages && ok; ++k) {
                  if (!acquire()) break;
                  const uint32_t dst = ring_a + (uint32_t)(r.slot * slot_bytes);
                  uint64_t* bar = &sh.full[r.slot];
                  ptx::mbar_expect_tx(bar, s.parts * part);
                  tma_load_3d_hint(dst, map, bar, 0, y, at * s.slices, policy);
                  if (s.parts > 1) tma_load_3d_hint(dst + (uint32_t)part, map, bar, 0, y + s.n, at * s.slices, policy);
                  r.pass(slots);
                  if (++at == stages) at = 0;
                }
              }
              if (serial || now != kDown) break;
            }
            continue;
          }
          Walk w = start;
          while (w.left > 0 && ok) {
            int first;
            const int n = piece_of(w, first);
            const int32_t* pages = p.block_table + (size_t)w.b * p.pages_per_seq;
            int page = pages[first];
#pragma unroll 1
            for (int j = 0; j < 2 * n && ok; ++j) {   // K and V of a tile in turn
              const int t = first + (j >> 1);
              const int y = l * p.cache_rows + (page * p.kv_heads + w.kvh) * kPageTokens;
              if ((j & 1) && j + 1 < 2 * n) page = pages[t + 1];
              if (!acquire()) break;
              uint64_t* bar = &sh.full[r.slot];
              ptx::mbar_expect_tx(bar, C::kTileBytes);
#pragma unroll
              for (int cb = 0; cb < C::kBlocks; ++cb)   // (read once a step: L2 is for what the CTAs share, 8 x 512 keys of phi2 521 -> 508 us)
                ptx::tma_load_2d_hint(ring + r.slot * slot_bytes + cb * (C::kKeys * 128), j & 1 ? &p.v : &p.k, bar, cb * 64, y, policy);
              ptx::mbar_arrive(bar);   // (in the place of the activations)
              r.pass(slots);
            }
            next_piece(w);
          }
        }
      }
    }
  }
  // ================================================================ barriers and activations
  else if (warp > kWorkWarps) {
    const int turn = warp - kWorkWarps - 1;   // two warps, each for every other slot (there is an even number of them): one alone needs 200 ns for each
    uint32_t target = 0;                      // arrivals at all barriers so far
    auto barrier = [&]() {
      target += (uint32_t)ctas;
      if (ok) {
        const long long t0 = clock64();
        uint32_t spins = 0, f;
        while (true) {
          asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(f) : "l"(p.flags) : "memory");
          if ((int32_t)(f - target) >= 0) break;
          if ((++spins & 0xffu) == 0 && (*abort_flag != 0 || clock64() - t0 > p.wait_cycles)) { ok = false; *abort_flag = 1u; break; }
        }
      }
      if (turn == 0) ptx::mbar_arrive(&sh.go);
    };
    if (lane == 0) {
#pragma unroll 1
      for (int l = 0; l <= p.layers; ++l) {
#pragma unroll 1
        for (int i = 0; i < 5; ++i) {
          const int op = l < p.layers ? op_at(serial, i) : i == 0 && p.want_head ? kHead : 15;
          if (op == 15) break;
          // (before the first slot behind it: attention's may be several times around the ring, and a slot's parity means nothing
          // before they are through)
          if (serial || op != kUp) barrier();
          if (op == kAttend) {
            r.pass(2 * stretch, slots);
            continue;
          }
#pragma unroll 1
          for (int now = op;; now = kOut) {
            const StepShare s = p.share[now];
            const uint32_t from = (uint32_t)(s.parts * s.slices * s.rows) * 128u, bytes = (uint32_t)(s.slices * m_rows) * 128u;
            const int stages = s.stages;
#pragma unroll 1
            for (int pass = 0; pass < s.passes; ++pass) {
              if ((cta * s.passes + pass) * s.rows >= s.n) break;
              int at = first_stage(cta, ctas, stages);
#pragma unroll 1
              for (int k = 0; k < stages; ++k) {
                if ((r.slot & 1) == turn && ok) {
                  ok = ptx::mbar_wait(&sh.empty[r.slot], r.parity ^ 1u, abort_flag, p.wait_cycles);
                  uint64_t* bar = &sh.full[r.slot];
                  if (ok) {
                    ptx::mbar_expect_tx(bar, bytes);
                    tma_load_3d(ring_a + (uint32_t)(r.slot * slot_bytes) + from, &p.x[now], bar, 0, 0, at * s.slices);
                  }
                }
                r.pass(slots);
                if (++at == stages) at = 0;
              }
            }
            if (serial || now != kDown) break;
          }
        }
        if (!serial && l < p.layers) barrier();   // the LayerNorm's
      }
    }
  }
  // ================================================================ products, attention, epilogues
  else {
    uint32_t gone = 0;
    const int tid = threadIdx.x;
    const int row_e = warp, col_e = lane;   // of an epilogue into the stream: a warp per row
    const bool row_ok = row_e < m_rows;
    const int spread = m_rows <= 1 ? 256 : m_rows <= 2 ? 128 : m_rows <= 4 ? 64 : 32;   // threads per row
    const int own_rows = p.share[kOut].rows, own0 = cta * own_rows, own_n = max(0, min(own_rows, p.hidden - own0));

    auto arrive = [&]() {   // this CTA's part of the phase is in memory, for copies to read, too
      asm volatile("fence.proxy.async.global;" ::: "memory");
      work_sync();
      // (A CTA that has given up waits for nothing more, and must not be counted: other CTAs' barriers would open before their own attention is
      // through, and activations asked for then would arrive on barriers of slots in an older use.)
      if (tid == 0 && *abort_flag == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(p.flags) : "memory");
    };
    auto wait_go = [&]() { ptx::mbar_wait(&sh.go, gone & 1u, abort_flag, p.wait_cycles); ++gone; };
    // (A parity tells a slot's use from the one before it, not from the one before that: who does not read every slot in turn first sees that
    // the slot has been left by its last user.  The use before that one has been: copies go round in order, and either this warp has had
    // the slot eight places before this one, or all warps have met since.)
    // What has not come (somebody gave up) is not given back: its barrier still expects a copy, and nobody may arm it again.
    auto wait_slot = [&](const Ring& at) {
      return ptx::mbar_wait(&sh.empty[at.slot], at.parity ^ 1u, abort_flag, p.wait_cycles) &&
             ptx::mbar_wait(&sh.full[at.slot], at.parity, abort_flag, p.wait_cycles);
    };
    auto leave_slot = [&](const Ring& at, int n, bool came) {
      came = __all_sync(0xffffffffu, came);
      if (lane == 0 && came) release_slot(&sh.empty[at.slot], n);
    };
    // acc += W . X^T over the slots of one pass.  A slot belongs to one warp, which takes all its rows: a byte of it is read once from
    // shared memory, and eight slots are at work at a time.  (With a slot's rows shared out among the warps each of them waited for
    // every slot and read the rows of X for itself: 350 ns a slot, whatever was in it.)  T: tiles of 16 rows; with few of them S sums
    // per tile run side by side.
    auto product = [&](auto tiles_c, float (&acc)[kTiles][4], const StepShare& s) {
      constexpr int T = decltype(tiles_c)::value, S = T == 8 ? 1 : 2;
      const int nt = (s.rows + 15) >> 4, tiles = nt * s.parts, stages = s.stages, rows = s.rows, slices = s.slices;
      int w_q[T];
#pragma unroll
      for (int t = 0; t < T; ++t) {
        const int part = t >= nt && tiles > nt ? 1 : 0;
        w_q[t] = (min((t - part * nt) * 16 + (lane & 15), rows - 1) + part * slices * rows) * 128;
      }
      const int x_q = (s.parts * slices * rows + min(lane & 7, m_rows - 1)) * 128;
      const int whole = s.blocks;
      int at = first_stage(cta, ctas, stages) + warp;
      Ring mine = r;
      mine.pass(warp, slots);
      if (at >= stages) at -= stages;
      const bool whole_ring = *abort_flag == 0;   // (no slot that only some warps of an attention gave back: four more would be too many)
#pragma unroll 1
      for (int turn = warp; turn < stages; turn += kWorkWarps) {
        const bool came = wait_slot(mine) && whole_ring;
        const int n = min(slices, whole - at * slices);
        const uint32_t base = ring_a + (uint32_t)(mine.slot * slot_bytes);
#pragma unroll T == 2 ? 2 : 1
        for (int k = 0; k < 2 * n; ++k) {     // 32 columns
          const int c0 = (k & 1) * 4;
          const uint32_t w_base = base + (uint32_t)((k >> 1) * rows) * 128u, x_row = base + (uint32_t)(x_q + (k >> 1) * m_rows * 128);
          uint32_t x[4];                      // 16 columns in two, the next 16 in two
          ldsm_x4(x, x_row + (((uint32_t)(c0 + (lane >> 3)) ^ ((x_row >> 7) & 7u)) << 4));
          uint32_t from[T];
#pragma unroll
          for (int t = 0; t < T; ++t) {
            const uint32_t row = w_base + (uint32_t)w_q[t];
            from[t] = row + (((uint32_t)(c0 + (lane >> 4)) ^ ((row >> 7) & 7u)) << 4);   // (the second 16 columns: bit 5 the other way)
          }
#pragma unroll
          for (int h0 = 0; h0 < 2; h0 += S) {
            uint32_t w[S * T][4];
#pragma unroll
            for (int h = 0; h < S; ++h)
#pragma unroll
              for (int t = 0; t < T; ++t) ldsm_x4(w[h * T + t], h0 + h ? from[t] ^ 32u : from[t]);
#pragma unroll
            for (int h = 0; h < S; ++h)
#pragma unroll
              for (int t = 0; t < T; ++t) mma16816(acc[h * T + t], w[h * T + t], x[2 * (h0 + h)], x[2 * (h0 + h) + 1]);
          }
        }
        leave_slot(mine, kReleases, came);
        mine.slot += kWorkWarps;
        if (mine.slot >= slots) { mine.slot -= slots; mine.parity ^= 1u; }   // (there are at least as many slots as warps)
        at += kWorkWarps;
        while (at >= stages) at -= stages;
      }
      r.pass(stages, slots);
    };
    // 1 / root of the mean square of every row, from the CTAs' sums: asked for before a product, added up behind it
    constexpr int kShares = 10;   // of 16 lanes; there are at most 160 CTAs
    auto ask_squares = [&](float (&part)[kShares]) {
      const float* from = p.squares + (tid >> 4) * ctas + (tid & 15);
#pragma unroll
      for (int i = 0; i < kShares; ++i) part[i] = (tid >> 4) < m_rows && (tid & 15) + i * 16 < ctas ? ldcg(from + i * 16) : 0.f;
    };
    auto row_scales = [&](const float (&part)[kShares]) {
      float s = 0.f;
#pragma unroll
      for (int i = 0; i < kShares; ++i) s += part[i];
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if ((tid & 15) == 0 && (tid >> 4) < m_rows) sh.rstd[tid >> 4] = 1.0f / sqrtf(s / p.squares_over + p.eps);
    };
    // what the next norm needs of a finished column of the stream: times its weight, and the square
    auto publish = [&](int c, float v, float gain) {
      p.hw[(size_t)row_e * p.hidden + own0 + c] = __float2bfloat16_rn(v * (p.norm == RB_NORM_RMS_ONE_PLUS ? gain + 1.0f : gain));
    };
    auto square = [&](float v) {   // (as the norm's own kernel takes it: RMS divides by the root of the width first, and a mean is in range where a sum is not)
      v *= p.squares_of;
      return v * v;
    };
    auto publish_squares = [&](float s) {   // of this thread's columns
      s = warp_sum(s);
      if (row_ok && lane == 0) p.squares[row_e * ctas + cta] = s;
    };
    // LayerNorm of row `cta` of the stream
    auto layer_norm = [&](const bf16* w, const bf16* b) {
      if (cta >= m_rows) return;
      const bf16* src = p.h + (size_t)cta * p.hidden;
      const int pieces = p.hidden >> 3;
      auto total = [&](float v, int turn) {
        v = warp_sum(v);
        if (lane == 0) sh.sums[turn][warp] = v;
        work_sync();
        v = 0.f;
#pragma unroll
        for (int i = 0; i < kWorkWarps; ++i) v += sh.sums[turn][i];
        return v;
      };
      auto piece = [&](int i, float* t) {
        const uint4 u = __ldcg(reinterpret_cast<const uint4*>(src) + i);
        load8(reinterpret_cast<const bf16*>(&u), t);
      };
      float s = 0.f, t[8];
#pragma unroll 1
      for (int i = tid; i < pieces; i += 256) {
        piece(i, t);
#pragma unroll
        for (int j = 0; j < 8; ++j) s += t[j];
      }
      const float mean = total(s, 0) / (float)p.hidden;
      s = 0.f;
#pragma unroll 1
      for (int i = tid; i < pieces; i += 256) {
        piece(i, t);
#pragma unroll
        for (int j = 0; j < 8; ++j) s += (t[j] - mean) * (t[j] - mean);
      }
      const float scale = 1.0f / sqrtf(total(s, 1) / (float)p.hidden + p.eps);
#pragma unroll 1
      for (int i = tid; i < pieces; i += 256) {
        float g[8], o[8], y[8];
        piece(i, t);
        load8(w + i * 8, g);
        load8(b + i * 8, o);
#pragma unroll
        for (int j = 0; j < 8; ++j) y[j] = g[j] * ((t[j] - mean) * scale) + o[j];
        store8(p.hw + (size_t)cta * p.hidden + i * 8, y);
      }
    };

    auto attend = [&](int l) {
      Walk w = start;
      const int grp = warp / C::kWarpsPerTile, kw0 = (warp % C::kWarpsPerTile) * 16;
      const int g = lane >> 2, t4 = lane & 3;
      const int half = p.rot >> 1;
      // Whoever gave up has no row to append: what it would write (not a number, maybe) lies behind the cached length, where it is masked out of
      // later prompts' products as zero times that.
      const bool sound = *abort_flag == 0;
      while (w.left > 0) {
        int first_tile;
        const int n = piece_of(w, first_tile), b = w.b, kvh = w.kvh, head = kvh * p.group, len = sh.len[b], pos = len - 1;
        const bool newest = first_tile + n == sh.tiles[b];
        // q heads of this KV head, its k head and its v head out of the projection, rotated
        {
          const float* src = p.qkv_out + (size_t)b * p.nqkv;
          const int pairs = half >> 3, rest = (D - p.rot) >> 3, per_head = pairs + rest, turned = (p.group + 1) * per_head;
          const int total = newest ? turned + (D >> 3) : p.group * per_head;
          const int page = p.block_table[(size_t)b * p.pages_per_seq + pos / kPageTokens];
          const size_t new_row = (size_t)l * p.layer_stride + (((size_t)page * p.kv_heads + kvh) * kPageTokens + pos % kPageTokens) * D;
          auto emit = [&](int r, int at, const float* v) {
            if (r < p.group) { store8(reinterpret_cast<bf16*>(q_s + r * C::kQRow) + at, v); return; }
            bf16* keep = new_kv + (r - p.group) * D + at;
            store8(keep, v);
            if (sound) *reinterpret_cast<uint4*>((r == p.group ? p.cache_k : p.cache_v) + new_row + at) = *reinterpret_cast<const uint4*>(keep);
          };
#pragma unroll 1
          for (int it = tid; it < total; it += 256) {
            if (it < turned) {
              const int r = it / per_head, j = it % per_head;
              const float* from = src + (size_t)(r < p.group ? head + r : p.q_heads + kvh) * D;
              if (j < pairs) {
                const int i0 = j * 8;
                float lo[8], hi[8], cs[8], sn[8], ylo[8], yhi[8];
                ldcg8(from + i0, lo);
                ldcg8(from + i0 + half, hi);
                load8(p.cos_t + (size_t)pos * half + i0, cs);
                load8(p.sin_t + (size_t)pos * half + i0, sn);
                rope_rotate8(lo, hi, cs, sn, ylo, yhi);
                emit(r, i0, ylo);
                emit(r, i0 + half, yhi);
              } else {
                const int i0 = p.rot + (j - pairs) * 8;
                float v[8];
                ldcg8(from + i0, v);
                emit(r, i0, v);
              }
            } else {
              const int i0 = (it - turned) * 8;
              float v[8];
              ldcg8(src + (size_t)(p.q_heads + p.kv_heads + kvh) * D + i0, v);
              emit(p.group + 1, i0, v);
            }
          }
        }
        work_sync();
        uint32_t qf[D / 16][4];
        const uint32_t q_a = ptx::smem_u32(q_s) + (uint32_t)(min(lane & 15, p.group - 1) * C::kQRow + (lane >> 4) * 16);
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) ldsm_x4(qf[kk], q_a + kk * 32);
        float o[D / 8][4];
#pragma unroll
        for (int i = 0; i < D / 8; ++i) { o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f; }
        float m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.f, 0.f};
        auto tile_at = [&](uint32_t base, int key, int dc) {
          return base + (uint32_t)((dc >> 6) * (C::kKeys * 128) + key * 128 + ((((dc & 63) >> 3) ^ (key & 7)) << 4));
        };
        // the copy of the newest tile may be older than the new token's row: it is put in place
        auto patch = [&](int kv, int at) {
          const int key = pos % C::kKeys, i = tid % (C::kWarpsPerTile * 32);
          if (i < D / 8)
            *reinterpret_cast<uint4*>(ring + at + tile_at(0, key, i * 8)) = *reinterpret_cast<const uint4*>(new_kv + kv * D + i * 8);
          asm volatile("bar.sync %0, %1;" ::"r"(3 + grp), "r"(C::kWarpsPerTile * 32) : "memory");
        };
#pragma unroll 1
        for (int i = 0; i < n; ++i) {
          if (i % C::kGroups != grp) {
            r.pass(slots);
            r.pass(slots);
            continue;
          }
          const int at_k = r.slot * slot_bytes;
          const int first = (first_tile + i) * C::kKeys + kw0;
          const bool has_new = newest && i == n - 1, active = first < len;
          bool came = wait_slot(r);
          if (has_new) patch(0, at_k);
          float s[2][4] = {};
          uint32_t pa[4] = {};
          if (active) {
            const uint32_t ks = ring_a + (uint32_t)at_k;
            float odd[2][4] = {};     // two chains of products
#pragma unroll
            for (int k2 = 0; k2 < D / 16; k2 += 2) {
              uint32_t bb[2][4];
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                const int kk = k2 + h;
                if (kk >= D / 16) break;
                ldsm_x4(bb[h], tile_at(ks, kw0 + (lane & 7) + ((lane >> 4) << 3), kk * 16 + (((lane >> 3) & 1) << 3)));
              }
              mma16816(s[0], qf[k2], bb[0][0], bb[0][1]);
              mma16816(s[1], qf[k2], bb[0][2], bb[0][3]);
              if (k2 + 1 < D / 16) {
                mma16816(odd[0], qf[k2 + 1 < D / 16 ? k2 + 1 : 0], bb[1][0], bb[1][1]);
                mma16816(odd[1], qf[k2 + 1 < D / 16 ? k2 + 1 : 0], bb[1][2], bb[1][3]);
              }
            }
#pragma unroll
            for (int nt = 0; nt < 2; ++nt)
#pragma unroll
              for (int e = 0; e < 4; ++e) s[nt][e] += odd[nt][e];
          }
          if (has_new) ptx::fence_proxy_async();
          leave_slot(r, kReleases / C::kWarpsPerTile, came);
          r.pass(slots);
          if (active) {
            float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
            for (int nt = 0; nt < 2; ++nt)
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const float v = first + nt * 8 + 2 * t4 + (e & 1) < len ? s[nt][e] * p.scale_log2 : -INFINITY;
                s[nt][e] = v;
                mx[e >> 1] = fmaxf(mx[e >> 1], v);
              }
            float corr[2], use[2];
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
              mx[hf] = fmaxf(mx[hf], __shfl_xor_sync(0xffffffffu, mx[hf], 1));
              mx[hf] = fmaxf(mx[hf], __shfl_xor_sync(0xffffffffu, mx[hf], 2));
              const float m_new = fmaxf(m_run[hf], mx[hf]);
              use[hf] = m_new == -INFINITY ? 0.f : m_new;
              corr[hf] = ex2(m_run[hf] - use[hf]);
              m_run[hf] = m_new;
              l_run[hf] *= corr[hf];
            }
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) {
              const float p0 = ex2(s[nt][0] - use[0]), p1 = ex2(s[nt][1] - use[0]);
              const float p2 = ex2(s[nt][2] - use[1]), p3 = ex2(s[nt][3] - use[1]);
              l_run[0] += p0 + p1;
              l_run[1] += p2 + p3;
              pa[nt * 2] = pack_bf16(p0, p1);
              pa[nt * 2 + 1] = pack_bf16(p2, p3);
            }
            if (__any_sync(0xffffffffu, corr[0] != 1.f || corr[1] != 1.f)) {   // some row has a new maximum
#pragma unroll
              for (int j = 0; j < D / 8; ++j) { o[j][0] *= corr[0]; o[j][1] *= corr[0]; o[j][2] *= corr[1]; o[j][3] *= corr[1]; }
            }
          }
          came = wait_slot(r);
          const int at_v = r.slot * slot_bytes;
          if (has_new) patch(1, at_v);
          if (active) {
            const uint32_t vs = ring_a + (uint32_t)at_v;
#pragma unroll
            for (int dp = 0; dp < D / 16; ++dp) {
              uint32_t bb[4];
              ldsm_x4_t(bb, tile_at(vs, kw0 + (lane & 7) + (((lane >> 3) & 1) << 3), dp * 16 + ((lane >> 4) << 3)));
              mma16816(o[2 * dp], pa, bb[0], bb[1]);
              mma16816(o[2 * dp + 1], pa, bb[2], bb[3]);
            }
          }
          if (has_new) ptx::fence_proxy_async();
          leave_slot(r, kReleases / C::kWarpsPerTile, came);
          r.pass(slots);
        }
        // ---- the warps' parts of the piece: one scale, then one sum per element in the order of the warps
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
          l_run[hf] += __shfl_xor_sync(0xffffffffu, l_run[hf], 1);
          l_run[hf] += __shfl_xor_sync(0xffffffffu, l_run[hf], 2);
          if (t4 == 0) { sh.mm[warp][g + hf * 8] = m_run[hf]; sh.ml[warp][g + hf * 8] = l_run[hf]; }
        }
        work_sync();
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
          float M = -INFINITY;
#pragma unroll
          for (int i = 0; i < kWorkWarps; ++i) M = fmaxf(M, sh.mm[i][g + hf * 8]);
          const float f = exp2f(m_run[hf] - (M == -INFINITY ? 0.f : M));
          if (warp == hf && t4 == 0) {   // the piece's maximum and sum of this row
            float L = 0.f;
#pragma unroll
            for (int i = 0; i < kWorkWarps; ++i) L += sh.ml[i][g + hf * 8] * exp2f(sh.mm[i][g + hf * 8] - (M == -INFINITY ? 0.f : M));
            sh.row_m[g + hf * 8] = M;
            sh.row_l[g + hf * 8] = L;
          }
#pragma unroll
          for (int j = 0; j < D / 8; ++j) { o[j][hf * 2] *= f; o[j][hf * 2 + 1] *= f; }
        }
        const int size = p.group * D;
        // as many warps at a time as there is room for: the last ones hand theirs to the first
        int parts = kWorkWarps;
#pragma unroll 1
        while (true) {
          const bool fits = parts * size <= p.merge_floats;
          const int k = fits ? 0 : min(p.merge_floats / size, parts >> 1), rest = parts - k, low = fits ? 0 : rest;   // (one piece always fits)
          if (warp >= low && warp < parts) {
            float* dst = merge + (warp - low) * size + 2 * t4;
#pragma unroll
            for (int hf = 0; hf < 2; ++hf)
              if (g + hf * 8 < p.group)
#pragma unroll
                for (int j = 0; j < D / 8; ++j)
                  *reinterpret_cast<float2*>(dst + (g + hf * 8) * D + j * 8) = make_float2(o[j][hf * 2], o[j][hf * 2 + 1]);
          }
          work_sync();
          if (fits) break;
          if (warp < k) {
            const float* from = merge + warp * size + 2 * t4;
#pragma unroll
            for (int hf = 0; hf < 2; ++hf)
              if (g + hf * 8 < p.group)
#pragma unroll
                for (int j = 0; j < D / 8; ++j) {
                  const float2 v = *reinterpret_cast<const float2*>(from + (g + hf * 8) * D + j * 8);
                  o[j][hf * 2] += v.x;
                  o[j][hf * 2 + 1] += v.y;
                }
          }
          work_sync();
          parts = rest;
        }
        const int pieces = sh.pieces[b], pair = b * p.kv_heads + kvh;
        int id0 = kvh * pieces;            // the pair's first piece in the line
        for (int i = 0; i < b; ++i) id0 += sh.pieces[i] * p.kv_heads;
#pragma unroll 1
        for (int i = tid; i < size; i += 256) {
          const int r = i / D;
          const float M = sh.row_m[r], L = sh.row_l[r];
          float v = 0.f, part[kWorkWarps];
#pragma unroll
          for (int k = 0; k < kWorkWarps; ++k) part[k] = k < parts ? merge[k * size + i] : 0.f;
#pragma unroll
          for (int k = 0; k < kWorkWarps; ++k) v += part[k];
          if (pieces == 1) {
            p.attn[((size_t)b * p.q_heads + head) * D + i] = __float2bfloat16_rn(v / L);
          } else {
            const size_t at = (size_t)(id0 + w.i) * p.group;
            p.part_o[at * D + i] = v;
            if (i % D == 0) { p.part_ml[(at + r) * 2] = M; p.part_ml[(at + r) * 2 + 1] = L; }
          }
        }
        if (pieces > 1) {
          __threadfence();
          work_sync();
          if (tid == 0) {
            uint32_t* cnt = p.split_count + pair;
            const uint32_t last = atomicAdd(cnt, 1u) == (uint32_t)pieces - 1u ? 1u : 0u;
            if (last) *cnt = 0u;
            __threadfence();
            sh.last = last;
          }
          work_sync();
          if (sh.last) {
            const int rows = pieces * p.group;            // [piece][head of the group]
            const size_t at = (size_t)id0 * p.group;
            auto from = [&](int i) { return at + (size_t)(i / p.group) * p.group + i % p.group; };
#pragma unroll 1
            for (int i = tid; i < rows; i += 256) {
              merge[2 * i] = ldcg(p.part_ml + from(i) * 2);
              merge[2 * i + 1] = ldcg(p.part_ml + from(i) * 2 + 1);
            }
            work_sync();
#pragma unroll 1
            for (int i = tid; i < size; i += 256) {
              const int r = i / D, dd = i % D;
              float M = -INFINITY;
#pragma unroll 1
              for (int k = 0; k < pieces; ++k) M = fmaxf(M, merge[2 * (k * p.group + r)]);
              float L = 0.f, O = 0.f;
#pragma unroll 1
              for (int k0 = 0; k0 < pieces; k0 += 8) {
                float part[8];
#pragma unroll
                for (int k = 0; k < 8; ++k)
                  part[k] = k0 + k < pieces ? ldcg(p.part_o + (at + (size_t)(k0 + k) * p.group + r) * D + dd) : 0.f;
#pragma unroll
                for (int k = 0; k < 8; ++k)
                  if (k0 + k < pieces) {
                    const float f = exp2f(merge[2 * ((k0 + k) * p.group + r)] - M);
                    L += merge[2 * ((k0 + k) * p.group + r) + 1] * f;
                    O += part[k] * f;
                  }
              }
              p.attn[((size_t)b * p.q_heads + head) * D + i] = __float2bfloat16_rn(O / L);
            }
          }
        }
        work_sync();   // q_s, the sums and the shared flags are free again
        next_piece(w);
      }
    };

    // the bias of this thread's column, or the weight of the norm behind it: from HBM, so asked for before the wait for the other CTAs
    auto ask_extra = [&](int l, int op, int y, const StepShare& s) {
      float extra = 0.f;
      if (tid < s.rows && y + tid < s.n) {
        const bf16 *e = nullptr, *e2 = nullptr;
        if (op == kHead) e = p.head_b;
        else if (op == kQkv) e = p.layer[l].qkv_b;
        else if (op == kUp) e = p.layer[l].fc_b;
        else if (!serial) { e = p.layer[l].o_b; e2 = p.layer[l].down_b; }
        else e = op == kOut ? p.layer[l].norm2_w : l + 1 == p.layers ? p.head_norm_w : p.layer[l + 1].norm1_w;
        if (e) extra = __bfloat162float(e[y + tid]);
        if (e2) extra += __bfloat162float(e2[y + tid]);
      }
      return extra;
    };

    // ---- the program
    {
      float squares = 0.f;
      for (int c = col_e; row_ok && c < own_n; c += 32) {
        const float v = __bfloat162float(p.h[(size_t)row_e * p.hidden + own0 + c]);
        own[row_e * own_rows + c] = v;
        if (serial) { publish(c, v, __bfloat162float(p.layer[0].norm1_w[own0 + c])); squares += square(v); }
      }
      if (serial) { publish_squares(squares); arrive(); }
    }
#pragma unroll 1
    for (int l = 0; l <= p.layers; ++l) {
      if (!serial) {
        if (l) wait_go();
        if (l < p.layers) layer_norm(p.layer[l].norm1_w, p.layer[l].norm1_b);
        else layer_norm(p.head_norm_w, p.head_norm_b);
        arrive();
      }
#pragma unroll 1
      for (int i = 0; i < 5; ++i) {
        const int op = l < p.layers ? op_at(serial, i) : i == 0 && p.want_head ? kHead : 15;
        if (op == 15) break;
        float extra = op == kAttend ? 0.f : ask_extra(l, op, cta * p.share[op].passes * p.share[op].rows, p.share[op]);
        if (serial || op != kUp) wait_go();
        if (op == kAttend) {
          attend(l);
          arrive();
          continue;
        }
        const bool into = op == kOut || op == kDown, last = l + 1 == p.layers;
        float part[kShares];
        if (serial && !into) ask_squares(part);
        const StepShare s = p.share[op];
        float squares = 0.f;
#pragma unroll 1
        for (int pass = 0; pass < s.passes; ++pass) {
          const int y = (cta * s.passes + pass) * s.rows;
          if (y >= s.n) break;
          if (pass > 0) extra = ask_extra(l, op, y, s);
          float acc[kTiles][4] = {};
#pragma unroll 1
          for (int now = op;; now = kOut) {
            const StepShare of = p.share[now];
            const int n = ((of.rows + 15) >> 4) * of.parts;
            if (n <= 2) product(std::integral_constant<int, 2>(), acc, of);
            else if (n <= 4) product(std::integral_constant<int, 4>(), acc, of);
            else product(std::integral_constant<int, 8>(), acc, of);
            if (serial || now != kDown) break;
            work_sync();   // (see wait_slot: between two products every warp has left its slots)
          }
          // ---- the warps' sums meet in shared memory: as many at a time as there is room for
          const int nt = (s.rows + 15) >> 4, tiles = nt * s.parts;
          const int pitch = ((tiles * 16 + 31) & ~31) + 4, size = m_rows * pitch;   // conflict-free
          if (tiles <= 4) {   // the sums that ran side by side
            const bool two = tiles <= 2;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
#pragma unroll
              for (int t = 0; t < 2; ++t) acc[t][e] += two ? acc[t + 2][e] : acc[t + 4][e];
              if (!two) { acc[2][e] += acc[6][e]; acc[3][e] += acc[7][e]; }
            }
          }
          int parts = kWorkWarps;
          work_sync();   // the space is free
          if (tid < s.rows) sh.extra[tid] = extra;
          if (serial && !into && pass == 0) row_scales(part);
#pragma unroll 1
          while (true) {
            const bool fits = parts * size <= p.merge_floats;
            const int k = fits ? 0 : min(p.merge_floats / size, parts >> 1), rest = parts - k, low = fits ? 0 : rest;
            if (warp >= low && warp < parts) {
              float* at = merge + (warp - low) * size + (lane >> 2) + (lane & 3) * 2 * pitch;
#pragma unroll
              for (int t = 0; t < kTiles; ++t) {
                if (t >= tiles) break;
#pragma unroll
                for (int e = 0; e < 4; ++e)
                  if ((lane & 3) * 2 + (e & 1) < m_rows) at[(e & 1) * pitch + t * 16 + (e >> 1) * 8] = acc[t][e];
              }
            }
            work_sync();
            if (fits) break;
            if (warp < k) {
              const float* at = merge + warp * size + (lane >> 2) + (lane & 3) * 2 * pitch;
#pragma unroll
              for (int t = 0; t < kTiles; ++t) {
                if (t >= tiles) break;
#pragma unroll
                for (int e = 0; e < 4; ++e)
                  if ((lane & 3) * 2 + (e & 1) < m_rows) acc[t][e] += at[(e & 1) * pitch + t * 16 + (e >> 1) * 8];
              }
            }
            work_sync();
            parts = rest;
          }
          // (into the stream: the columns that a thread has there; else all threads share a row's columns)
          const int lanes = into ? 32 : spread, row = tid / lanes;
#pragma unroll 1
          for (int c = tid % lanes; row < m_rows && c < s.rows && y + c < s.n; c += lanes) {
            const float* at = merge + row * pitch + c;
            const float e = sh.extra[c];
            float v = 0.f, u = 0.f, va[kWorkWarps], ua[kWorkWarps];
#pragma unroll
            for (int k = 0; k < kWorkWarps; ++k) {
              va[k] = k < parts ? at[k * size] : 0.f;
              ua[k] = k < parts && s.parts > 1 ? at[k * size + nt * 16] : 0.f;
            }
#pragma unroll
            for (int k = 0; k < kWorkWarps; ++k) { v += va[k]; u += ua[k]; }
            if (into) {
              float& mine = own[row_e * own_rows + c];
              v = round_bf16((serial ? v : v + e) + mine);
              mine = v;
              if (serial) { publish(c, v, e); squares += square(v); }
              if (!serial || (last && op == kDown)) p.h[(size_t)row_e * p.hidden + y + c] = __float2bfloat16_rn(v);
              continue;
            }
            const float scale = serial ? sh.rstd[row] : 1.0f;
            v = v * scale + e;
            if (op == kQkv) p.qkv_out[(size_t)row * p.nqkv + y + c] = v;
            else if (op == kHead) p.logits[(size_t)row * p.vocab + y + c] = __float2bfloat16_rn(v);
            else p.inner[(size_t)row * p.inter + y + c] = __float2bfloat16_rn(act_apply(p.act, v) * (serial ? u * scale : 1.0f));
          }
        }
        if (serial && into) publish_squares(squares);
        if (op != kHead && (serial || op != kQkv)) arrive();
      }
    }
  }
  __syncwarp();
  __syncthreads();   // no role asks for a copy any more
  if (threadIdx.x == 0 && sh.abort) {
    // Whoever gave up, the others went on without waiting: copies that any of the three asking warps had issued may be under way.  They
    // end within microseconds, and the CTA must not leave before them.
    p.status[0] = (uint32_t)(-RB_ERR_TIMEOUT); p.status[1] = 0x57E9u; p.status[2] = (uint32_t)cta;
    const long long t0 = clock64();
    while (clock64() - t0 < 2000000) {}
  }
  // the last CTA to leave, when nobody waits any more, puts the barriers' count back
  if (threadIdx.x == 0 && atomicInc(p.flags + 32, (uint32_t)ctas - 1u) == (uint32_t)ctas - 1u) *p.flags = 0u;
}


StepShare share_rows(int n, int k, bool two, int ctas) {
  StepShare s{};
  const int per = (n + ctas - 1) / ctas, most = two ? 64 : 128;
  s.n = n;
  s.passes = (per + most - 1) / most;
  s.rows = (per + s.passes - 1) / s.passes;
  s.parts = two ? 2 : 1;
  s.blocks = k / 64;
  // columns for a slot, but no fewer slots than warps
  const int fit = std::min(s.blocks, kSlotBytes / 128 / (s.parts * s.rows + kRows));
  s.slices = std::max(1, std::min(fit, (s.blocks + kWorkWarps - 1) / kWorkWarps));
  s.stages = (s.blocks + s.slices - 1) / s.slices;
  return s;
}

template <int D>
int blocks_per_sm(size_t smem, int* n) {
  RB_CUDA(cudaFuncSetAttribute(step_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMostSmem));
  RB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(n, step_kernel<D>, kThreads, smem));
  return RB_OK;
}

template <int D>
cudaError_t launch(rb_ctx* ctx, const StepParams& p, size_t smem) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)ctx->sm_count);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = ctx->stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;   // its blocks wait for one another: all of them or none
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, step_kernel<D>, p);
}

}  // namespace

// What is the same for every step of a model: tensor maps of its weights and pages, shares, pointers.
struct StepPlan {
  StepParams p{};
  size_t smem = 0;
  bool refused = false;                      // (test hook)
  double layer_bytes = 0, token_bytes = 0;   // weights of a layer; keys and values of a token in it
};
void step_plan_free(StepPlan* plan) { delete plan; }

int step_reserve(rb_model* m) {
  const rb_model_config& c = m->cfg;
  rb_ctx* ctx = m->ctx;
  const int H = c.hidden_size, I = m->inter_l, d = m->d, K = m->nq_l * d, group = m->nq_l / m->nkv_l, ctas = ctx->sm_count;
  const bool phi2 = c.arch == RB_ARCH_PHI2;
  rb_kv_cache* kv = m->cache;
  const int64_t cache_rows = (int64_t)kv->num_pages * kv->kv_heads * kPageTokens;
  const double layer_bytes = 2.0 * ((double)m->nqkv_l * H + (double)H * K + (phi2 ? 2.0 : 3.0) * I * H);
  // Models of up to 96 MB a layer have faster steps as five launches a layer (gemm_rows.cu): 24 layers of 28 MB, one row, 0.66 ms against
  // 0.69 here.  (Layers of 97, 110, 125 and 145 MB take 0.72 to 0.93 of the launches' time here, 24 points each; between 28 and 97 nothing was measured.)  Heads of 256 (gemma-2b, 8 layers, 8 x 1024 keys: 805 us as launches, 883 here) would want two slots for a tile.
  if (c.dtype != RB_BF16 || c.tp_size != 1 || layer_bytes <= (double)(96 << 20) || c.num_hidden_layers > kStepLayers || H % 64 || I % 64 ||
      K % 64 || c.hidden_act == RB_ACT_XIELU || group > 16 || !(d == 64 || d == 80 || d == 96 || d == 128) || c.rotary_dim % 16 ||
      c.rotary_dim > d || (d - c.rotary_dim) % 8 || (H + ctas - 1) / ctas > kOwnColumns || cache_rows * c.num_hidden_layers >= (1LL << 31) ||
      ctas > 160 || ctx->debug_simple || ctx->debug_simple_gemm || ctx->debug_simple_attn || ctx->debug_no_fuse)
    return RB_OK;
  StepPlan* plan = m->step_plan = new StepPlan();
  StepParams& p = plan->p;
  plan->layer_bytes = layer_bytes;
  plan->token_bytes = 4.0 * m->nkv_l * d;
  p.layers = c.num_hidden_layers; p.hidden = H; p.inter = I; p.nqkv = m->nqkv_l; p.vocab = m->vocab_l;
  p.q_heads = m->nq_l; p.kv_heads = m->nkv_l; p.group = group; p.rot = c.rotary_dim; p.act = c.hidden_act; p.eps = (float)c.norm_eps;
  p.norm = phi2 ? RB_NORM_LAYER : c.arch == RB_ARCH_GEMMA ? RB_NORM_RMS_ONE_PLUS : RB_NORM_RMS;
  p.squares_of = p.norm == RB_NORM_RMS ? 1.0f / sqrtf((float)H) : 1.0f;
  p.squares_over = p.norm == RB_NORM_RMS ? 1.0f : (float)H;
  const int64_t n[5] = {p.nqkv, H, I, H, p.vocab}, k[5] = {H, K, H, I, H};
  int most = kPageTokens * ((d + 63) / 64) * 128;
  for (int op = 0; op < 5; ++op) {
    StepShare& s = p.share[op];
    s = share_rows((int)n[op], (int)k[op], op == kUp && !phi2, ctas);
    most = std::max(most, (s.parts * s.rows + kRows) * s.slices * 128);
  }
  p.slot_bytes = (most + 1023) & ~1023;
  p.merge_floats = kMergeFloats;
  // what the ring leaves: sums, the CTA's columns of the stream, rows for the attention
  const size_t rest = (size_t)p.merge_floats * 4 + (size_t)kRows * p.share[kOut].rows * 4 + 4 * d + (size_t)group * (d + 8) * 2 + 1024;
  p.slots = std::min<int>(kMaxSlots, (int)((kMostSmem - rest) / p.slot_bytes)) & ~1;
  plan->smem = rest + (size_t)p.slots * p.slot_bytes;
  // (a LayerNorm is a row per CTA; the launch is all of the grid or nothing, so a device, or a share of one, without room for it has no plan)
  int cooperative = 0, per_sm = 0;
  RB_CUDA(cudaDeviceGetAttribute(&cooperative, cudaDevAttrCooperativeLaunch, ctx->device));
  switch (d) {
    case 64: RB_TRY(blocks_per_sm<64>(plan->smem, &per_sm)); break;
    case 80: RB_TRY(blocks_per_sm<80>(plan->smem, &per_sm)); break;
    case 96: RB_TRY(blocks_per_sm<96>(plan->smem, &per_sm)); break;
    default: RB_TRY(blocks_per_sm<128>(plan->smem, &per_sm));
  }
  if (p.slots < kWorkWarps || ctas < kRows || !cooperative || per_sm < 1) { delete plan; m->step_plan = nullptr; return RB_OK; }
  for (int l = 0; l < p.layers; ++l) {
    const LayerW& w = m->layers[l];
    p.layer[l] = {(const bf16*)w.qkv_b, (const bf16*)w.o_b, (const bf16*)w.fc1_b, (const bf16*)w.down_b,
                  (const bf16*)w.ln1_w, (const bf16*)w.ln1_b, (const bf16*)w.ln2_w};
    const void* base[4] = {w.qkv, w.o, w.gate, w.down};
    for (int op = 0; op < 4; ++op)
      RB_TRY(tmap_slices_bf16(base[op], n[op] * p.share[op].parts, k[op], p.share[op].rows, p.share[op].slices, &p.w[l][op]));
  }
  RB_TRY(tmap_slices_bf16(m->lm_head ? m->lm_head : m->embed, p.vocab, H, p.share[kHead].rows, p.share[kHead].slices, &p.head));
  p.cache_rows = (int)cache_rows;
  p.layer_stride = kv->layer_stride_elems();
  RB_TRY(tmap_2d_bf16(ctx, kv->k, cache_rows * p.layers, d, d, kPageTokens, &p.k));
  RB_TRY(tmap_2d_bf16(ctx, kv->v, cache_rows * p.layers, d, d, kPageTokens, &p.v));
  p.head_norm_w = (const bf16*)m->norm_w; p.head_norm_b = (const bf16*)m->norm_b; p.head_b = (const bf16*)m->lm_head_b;
  p.pages_per_seq = kv->pages_per_seq;
  p.max_seq = std::min<int>(kv->max_seq, c.max_position_embeddings);
  p.scale_log2 = (float)(1.4426950408889634 / sqrt((double)d));
  p.h = (bf16*)m->h; p.hw = (bf16*)m->xn; p.attn = (bf16*)m->attn; p.inner = (bf16*)m->act; p.logits = (bf16*)m->logits;
  p.qkv_out = m->scratch;
  p.cache_k = (bf16*)kv->k; p.cache_v = (bf16*)kv->v;
  p.cos_t = m->rope_cos; p.sin_t = m->rope_sin;
  p.block_table = kv->block_table; p.seq_lens = kv->seq_lens; p.split_count = kv->split_count;
  p.status = ctx->status_dev;
  const size_t pieces = (size_t)std::min<int>(kRows, c.max_batch) * p.kv_heads + 2 * ctas;
  p.most_pieces = (int)pieces;
  RB_TRY(dev_alloc(m, pieces * group * d * sizeof(float), (void**)&p.part_o, false));
  RB_TRY(dev_alloc(m, pieces * group * 2 * sizeof(float), (void**)&p.part_ml, false));
  RB_TRY(dev_alloc(m, (size_t)ctas * kRows * sizeof(float), (void**)&p.squares, false));
  RB_TRY(dev_alloc(m, kStepFlagBytes, (void**)&p.flags, true));
  m->step_flags = p.flags;
  ctx->step_flags.push_back(p.flags);
  return RB_OK;
}

// Up to eight sequences, no more cached bytes than three quarters of the weights' (a step of more streams as fast in launches of its own), and an
// attention phase that is not longer than the launches' by more than those lose between kernels (step_rule.h).  us per step of 8 layers, as launches -> here,
// and cached bytes to weights: phi3-mini 1 x 3500 keys 597 -> 507 (0.19), 4 x 2048 662 -> 574 (0.44), 8 x 200 566 -> 503 (0.09), 8 x 1700 721 -> 705 (0.74); phi2
// 1 x 17 473 -> 349, 8 x 512 528 -> 470 (0.27), 8 x 1400 608 -> 594 (0.73); qwen2-7b 1 x 17 782 -> 743, 8 x 4500 928 -> 903 (0.16); layers of 97 MB,
// 1 x 100 and 8 x 500 keys: qwen2 400 -> 294 and 455 -> 336, phi3 374 -> 289 and 431 -> 390.  With sixteen sequences (two eights per product)
// every one of these was slower: phi3-mini 16 x 200 675 -> 706, qwen2-7b 16 x 2048 1086 -> 1164.
// (Under a per-launch profile the steps are launches of their own: a launch belongs to one class there.)
bool step_takes(const rb_model* m, int batch) {
  const StepPlan* plan = m->step_plan;
  if (!plan || m->ctx->profiling || batch > kRows || (size_t)batch * m->nqkv_l > m->scratch_floats) return false;
  const int32_t* lens = m->cache->host_lens.data();
  double tokens = 0;
  for (int b = 0; b < batch; ++b) tokens += lens[b];
  const StepParams& p = plan->p;
  return tokens * plan->token_bytes <= 0.75 * plan->layer_bytes &&
         step_attention_pays(lens, batch, p.kv_heads, p.group, m->d, m->ctx->sm_count, p.most_pieces);
}

int step_spoil(rb_model* m) {
  RB_REQUIRE(m->step_plan, "this model has no resident steps");
  // (behind by more than all arrivals of a step, 160 x 5 x 40 and some.  Never ahead: a barrier that opens early lets activations into
  // slots of an older use, and an arrival that a mbarrier does not expect is a launch failure.)
  const uint32_t far = 0u - (1u << 20);
  RB_CUDA(cudaStreamSynchronize(m->ctx->stream));
  RB_CUDA(cudaMemcpy(m->step_flags, &far, sizeof(far), cudaMemcpyHostToDevice));
  return RB_OK;
}

int step_refuse(rb_model* m) {
  RB_REQUIRE(m->step_plan, "this model has no resident steps");
  m->step_plan->refused = true;
  return RB_OK;
}

int step_forward(rb_model* m, int batch, bool want_head, bool* ran) {
  rb_ctx* ctx = m->ctx;
  StepParams& p = m->step_plan->p;
  const size_t smem = m->step_plan->smem;
  p.m = batch;
  p.want_head = want_head;
  p.wait_cycles = ctx->local_wait_cycles();
  const rb_model_config& c = m->cfg;
  const int H = c.hidden_size, I = m->inter_l, K = m->nq_l * m->d;
  const void* x[5] = {p.hw, p.attn, p.hw, p.inner, p.hw};
  const int k[5] = {H, K, H, I, H};
  for (int op = 0; op < 5; ++op) RB_TRY(tmap_slices_bf16(x[op], batch, k[op], batch, p.share[op].slices, &p.x[op]));
  cudaError_t e = cudaErrorCooperativeLaunchTooLarge;
  if (!m->step_plan->refused) {
    switch (m->d) {
      case 64: e = launch<64>(ctx, p, smem); break;
      case 80: e = launch<80>(ctx, p, smem); break;
      case 96: e = launch<96>(ctx, p, smem); break;
      default: e = launch<128>(ctx, p, smem);
    }
  }
  *ran = e == cudaSuccess;
  if (e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorLaunchOutOfResources || e == cudaErrorNotSupported) {
    // fewer SMs than the device has (a stream of a part of them): nothing has run, and this model's steps are launches from now on
    cudaGetLastError();
    step_plan_free(m->step_plan);
    m->step_plan = nullptr;
    return RB_OK;
  }
  RB_CUDA(e);
  ctx->launches++;
  return RB_OK;
}

}  // namespace rb
