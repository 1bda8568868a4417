// Head split of prompts (bf16), where thousands of rows are there and what counts is how many bytes are on their way.
#include <algorithm>

#include "ctx.h"

namespace rb {

using bf16 = __nv_bfloat16;

namespace {

// rb_rope_kv_append out of a finished projection: a block has a row; a thread turns the same eight dimensions of up to four heads,
// whose angles it loads once and whose eight loads are in flight together, and what is not turned moves four pieces at a time.
// (One item per thread,
// angles loaded for each, took 205 us for 32768 x 4608, 111 for 8192 x 9216, 64 for 4096 x 7680 and 13 for 3003 x 2560; this 136, 68, 57, 11.)
__global__ void __launch_bounds__(256) rope_rows_kernel(const bf16* __restrict__ qkv, const float* __restrict__ cos_t,
                                                        const float* __restrict__ sin_t, int rot, int s_new, int q_heads, int kv_heads,
                                                        int d, bf16* __restrict__ q_out, bf16* __restrict__ k_cache,
                                                        bf16* __restrict__ v_cache, const int32_t* __restrict__ block_table,
                                                        const int32_t* __restrict__ seq_lens, int pages_per_seq, int max_seq,
                                                        uint32_t* status, const Packed pk) {
  pdl_launch_dependents();
  pdl_wait();
  const int m = blockIdx.x;
  const int b = pk.seq ? pk.seq[m] : m / s_new;
  const int pos = seq_lens[b] - rows_of(pk.start, b, s_new) + m - first_row(pk.start, b, s_new);
  if (pos < 0 || pos >= max_seq) {
    if (threadIdx.x == 0) { status[0] = (uint32_t)(-RB_ERR_INVALID); status[1] = 0x20BEu; status[2] = (uint32_t)pos; }
    return;
  }
  const int half = rot >> 1, pairs = half >> 3, rot_heads = q_heads + kv_heads;
  const bf16* row = qkv + (size_t)m * (rot_heads + kv_heads) * d;
  const int page = block_table[(size_t)b * pages_per_seq + pos / kPageTokens], slot = pos % kPageTokens;
  auto place = [&](int head) -> bf16* {   // where a head of the row goes
    if (head < q_heads) return q_out + ((size_t)m * q_heads + head) * d;
    const int kvh = head < rot_heads ? head - q_heads : head - rot_heads;
    return (head < rot_heads ? k_cache : v_cache) + (((size_t)page * kv_heads + kvh) * kPageTokens + slot) * d;
  };
  for (int u = threadIdx.x; u < pairs * ((rot_heads + 3) / 4); u += blockDim.x) {
    const int i0 = u % pairs * 8, h0 = u / pairs * 4;
    uint4 lo[4], hi[4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (h0 + k < rot_heads) {
        lo[k] = *reinterpret_cast<const uint4*>(row + (h0 + k) * d + i0);
        hi[k] = *reinterpret_cast<const uint4*>(row + (h0 + k) * d + i0 + half);
      }
    float cs[8], sn[8];
    load8(cos_t + (size_t)pos * half + i0, cs);
    load8(sin_t + (size_t)pos * half + i0, sn);
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (h0 + k < rot_heads) {
        float a[8], c[8], ya[8], yc[8];
        load8(reinterpret_cast<const bf16*>(&lo[k]), a);
        load8(reinterpret_cast<const bf16*>(&hi[k]), c);
        rope_rotate8(a, c, cs, sn, ya, yc);
        bf16* dst = place(h0 + k) + i0;
        store8(dst, ya);
        store8(dst + half, yc);
      }
  }
  const int pass = (d - rot) >> 3, whole = d >> 3, passed = rot_heads * pass, moves = passed + kv_heads * whole;
  for (int id0 = threadIdx.x; id0 < moves; id0 += 4 * blockDim.x) {
    uint4 v[4];
    int head[4], at[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int id = id0 + k * blockDim.x;
      if (id >= moves) continue;
      head[k] = id < passed ? id / pass : rot_heads + (id - passed) / whole;
      at[k] = id < passed ? rot + id % pass * 8 : (id - passed) % whole * 8;
      v[k] = *reinterpret_cast<const uint4*>(row + head[k] * d + at[k]);
    }
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (id0 + k * (int)blockDim.x < moves) *reinterpret_cast<uint4*>(place(head[k]) + at[k]) = v[k];
  }
}

// Several rows for every SM, and rows wide enough that a block has work for more than its smallest 64 threads.  us, one item per thread -> this: 1024 rows
// of 4608 columns 6.0 -> 5.2, of 2560 (one key head of 256) 5.9 -> 5.3; 16384 of 3072 56 -> 50, of 2560 (heads of 128) 50 -> 49, but of 1152
// (qwen2-0.5b) 22 -> 38, of 2048 37 -> 48; 256 to 768 rows within 0.3 of one another but for heads of 80 and 96, where 512 gain already.
constexpr int64_t kManyRows = 1024, kWideRow = 2560;

}  // namespace

// The caller has checked that rows are made of aligned 16-byte pieces.  false: its own kernel takes the call.
bool rope_prompt(rb_ctx* ctx, const void* qkv, const float* cos_t, const float* sin_t, int rot, int rows, int s_new, int q_heads, rb_kv_cache* c,
                 void* k, void* v, void* q_out, const Packed* pk, cudaError_t* status) {
  const int d = c->head_dim, rot_heads = q_heads + c->kv_heads;
  if (rows < kManyRows || (rot_heads + c->kv_heads) * d < kWideRow) return false;
  const int work = std::max(rot / 16 * ((rot_heads + 3) / 4), (rot_heads * ((d - rot) / 8) + c->kv_heads * (d / 8) + 3) / 4);
  const int threads = std::max(64, std::min(256, (work + 31) / 32 * 32));
  *status = launch_kernel(rope_rows_kernel, dim3((unsigned)rows), dim3((unsigned)threads), 0, ctx->stream, ctx->pdl, (const bf16*)qkv, cos_t, sin_t,
                          rot, s_new, q_heads, c->kv_heads, d, (bf16*)q_out, (bf16*)k, (bf16*)v, (const int32_t*)c->block_table,
                          (const int32_t*)c->seq_lens, c->pages_per_seq, c->max_seq, ctx->status_dev, pk ? *pk : Packed());
  return true;
}

}  // namespace rb
