// Causal grouped-query attention over the paged cache: two warps a query head and token or four warps up to four heads of a group, or (heads
// of more than 128 entries or no multiple of 4) one warp per (query token, query head).
//
// This is the plain kernel: it serves the whole 32-bit path (prompts and single tokens alike) and any
// shape the faster bfloat16 kernels refuse.  A query at absolute position p of the sequence in `slot`
// sees key j of the same slot iff j <= p, and with a window w only iff j > p - w
// (engine/engine.py:781-787 for the rule that causality follows absolute positions, not the number of
// queries in the step).  Query head h reads key/value head h / (heads / kv_heads)
// (engine/kernels/fused.py:263-266).  Scores, the running maximum and sum, and the accumulator are
// float (fused.py:288-312); the result is rounded to the working type once.
#include "common.cuh"

#define SB_ROW_MAX_D 8  // head_dim <= 256

template <typename T>
__global__ void attention_rowwise_kernel(const T* __restrict__ q, T* __restrict__ out,
                                         const T* __restrict__ k_store, const T* __restrict__ v_store,
                                         const int* __restrict__ block_table, int table_stride,
                                         const int* __restrict__ tok_slot,
                                         const int* __restrict__ tok_pos, int n_tokens, int heads,
                                         int kv_heads, int head_dim, float scale, int window) {
  const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (warp >= (long long)n_tokens * heads) return;
  const int token = (int)(warp / heads);
  const int h = (int)(warp - (long long)token * heads);
  const int kvh = h / (heads / kv_heads);
  const int pos = tok_pos[token];
  const int* pages = block_table + (size_t)tok_slot[token] * table_stride;
  const T* qr = q + ((size_t)token * heads + h) * head_dim;

  float qv[SB_ROW_MAX_D], acc[SB_ROW_MAX_D];
#pragma unroll
  for (int i = 0; i < SB_ROW_MAX_D; ++i) {
    const int d = lane + 32 * i;
    qv[i] = d < head_dim ? to_f<T>(qr[d]) * scale : 0.f;
    acc[i] = 0.f;
  }
  float m = -INFINITY, l = 0.f;
  int first = 0;
  if (window > 0 && pos - window + 1 > 0) first = pos - window + 1;

  for (int j0 = first; j0 <= pos; j0 += 4) {
    float s[4];
    const T* vrow[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int j = j0 + u;
      s[u] = 0.f;
      vrow[u] = nullptr;
      if (j <= pos) {
        const int page = pages[j / SB_PAGE_TOKENS];
        const size_t off = page_row(page, kvh, j % SB_PAGE_TOKENS, kv_heads, head_dim);
        const T* kr = k_store + off;
        vrow[u] = v_store + off;
#pragma unroll
        for (int i = 0; i < SB_ROW_MAX_D; ++i) {
          const int d = lane + 32 * i;
          if (d < head_dim) s[u] += qv[i] * to_f<T>(kr[d]);
        }
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) s[u] = warp_sum(s[u]);
    float m_new = m;
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (j0 + u <= pos) m_new = fmaxf(m_new, s[u]);
    const float alpha = expf(m - m_new);
    l *= alpha;
#pragma unroll
    for (int i = 0; i < SB_ROW_MAX_D; ++i) acc[i] *= alpha;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (j0 + u <= pos) {
        const float p = expf(s[u] - m_new);
        l += p;
#pragma unroll
        for (int i = 0; i < SB_ROW_MAX_D; ++i) {
          const int d = lane + 32 * i;
          if (d < head_dim) acc[i] += p * to_f<T>(vrow[u][d]);
        }
      }
    }
    m = m_new;
  }
  T* orow = out + ((size_t)token * heads + h) * head_dim;
  const float inv = 1.f / l;
#pragma unroll
  for (int i = 0; i < SB_ROW_MAX_D; ++i) {
    const int d = lane + 32 * i;
    if (d < head_dim) orow[d] = from_f<T>(acc[i] * inv);
  }
}

// Heads of up to 128 entries, a multiple of 4, in 16- or 8-byte pieces: a lane holds four entries of a row, and 16 keys, then their
// values, are asked for together (four keys a round, each round a chain of page number, keys, sums, exponential and values: 75 us for
// 141 tokens of 16 heads over up to 77 keys).  The sums of 16 scores share their shuffles: lane l ends with key l / 2.
#define ROW_KEYS 16
template <typename T> struct RowPiece;
template <> struct RowPiece<float> {
  typedef float4 type;
  static __device__ __forceinline__ float4 open(const float4& v) { return v; }
  static __device__ __forceinline__ float4 zero() { return make_float4(0.f, 0.f, 0.f, 0.f); }
};
template <> struct RowPiece<bf16> {
  typedef uint2 type;
  static __device__ __forceinline__ float4 open(const uint2& v) {
    return make_float4(__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xffff0000u), __uint_as_float(v.y << 16),
                       __uint_as_float(v.y & 0xffff0000u));
  }
  static __device__ __forceinline__ uint2 zero() { return make_uint2(0u, 0u); }
};

// W warps have HB query heads of one key/value head and a token (a unit): a warp takes every W-th sixteen keys, which serve all HB heads,
// and the warps' sums meet in shared memory.  What bounds a step of few tokens here is the chain of rounds a warp walks, one of many its
// issue slots and the keys' way from L2.  HB 1, W 2, two units a block: half the rounds of a warp a head and token, three blocks an SM (145
// registers, no spills; four an SM spill 52 bytes).  HB 4, W 4: keys and values are asked for once for four heads, four blocks an SM (spills of
// 192 bytes; three an SM are slower: 154 tokens 151.9 for 150.3), from 1,184 heads of tokens on, when its blocks fill half the SMs' places.
// Measured, a float32 layer, us, a warp a head / HB 1 / HB 4, groups of four (16 heads): 20 tokens 77.4 / 76.0 / 79.2, 40 behind 150 113.7 / 94.2 /
// 96.5, 100 108.6 / 106.5 / 104.2, 120 behind 100 144.0 / 131.8 / 119.0, 2 x 77 126.2 / 125.4 / 125.5, 2 x 150 244.8 / 241.5 / 231.7; of six (12
// heads) 100 100.6 / 94.4 / 96.0, 2 x 77 113.4 / 113.1 / 115.6, 2 x 110 183.2 / 182.3 / 180.9; of eight 20 76.1 / 74.8 / 78.2, 100 106.6 / 104.3 /
// 102.5, 2 x 110 196.0 / 195.4 / 189.2.  Smaller groups, a warp a head / HB 1 / four warps up to four heads: of one 2 x 77 152.0 / 151.3 / 154.6,
// 40 behind 150 129.4 / 111.1 / 114.3; of two 2 x 77 129.0 / 129.4 / 133.7, 40 behind 150 116.6 / 98.2 / 104.1, 2 x 150 251.5 / 250.8 / 253.0; of three
// 2 x 77 114.9 / 115.0 / 117.6, 40 behind 150 101.2 / 87.7 / 90.4, 2 x 150 224.0 / 221.3 / 219.2.
#define ROW_UNIT_WARPS(HB) ((HB) == 1 ? 2 : 4)
template <typename T, int HB>
__global__ void __launch_bounds__(128, HB == 1 ? 3 : 4)
attention_rowwise_group_kernel(const T* __restrict__ q, T* __restrict__ out, const T* __restrict__ k_store,
                               const T* __restrict__ v_store, const int* __restrict__ block_table, int table_stride,
                               const int* __restrict__ tok_slot, const int* __restrict__ tok_pos, int heads,
                               int kv_heads, int head_dim, float scale, int window, unsigned units) {
  typedef RowPiece<T> Piece;
  typedef typename Piece::type Raw;
  constexpr int W = ROW_UNIT_WARPS(HB);
  __shared__ __align__(16) float sums[4][HB][128];
  __shared__ float most[4][HB], total[4][HB];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int group = heads / kv_heads, shares = (group + HB - 1) / HB;
  const int turn = warp % W;
  const unsigned unit = min(blockIdx.x * (4 / W) + warp / W, units - 1);           // (an odd last one is done twice)
  const int token = unit / (unsigned)(kv_heads * shares), rest = unit - token * (unsigned)(kv_heads * shares);
  const int kvh = rest / shares, h0 = kvh * group + (rest - kvh * shares) * HB, here = min(HB, (kvh + 1) * group - h0);
  const int pos = tok_pos[token];
  const int* pages = block_table + (size_t)tok_slot[token] * table_stride;
  const int d = 4 * lane;
  const bool in = d < head_dim;
  const T* own = q + ((size_t)token * heads + h0) * head_dim + d;
  float4 qv[HB], acc[HB];
  float m[HB], l[HB];                               // l: this lane's own keys' weights
#pragma unroll
  for (int i = 0; i < HB; ++i) {
    qv[i] = in && i < here ? Piece::open(*reinterpret_cast<const Raw*>(own + (size_t)i * head_dim)) : make_float4(0.f, 0.f, 0.f, 0.f);
    qv[i].x *= scale; qv[i].y *= scale; qv[i].z *= scale; qv[i].w *= scale;
    acc[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    m[i] = -INFINITY;
    l[i] = 0.f;
  }
  int first = 0;
  if (window > 0 && pos - window + 1 > 0) first = pos - window + 1;
#pragma unroll 1
  for (int j0 = first + turn * ROW_KEYS; j0 <= pos; j0 += W * ROW_KEYS) {
    // a lane a key looks up its page
    const int mine = min(j0 + (lane & (ROW_KEYS - 1)), pos);
    const long long at = (long long)page_row(pages[mine / SB_PAGE_TOKENS], kvh, mine % SB_PAGE_TOKENS, kv_heads, head_dim);
    Raw raw[ROW_KEYS];
#pragma unroll
    for (int u = 0; u < ROW_KEYS; ++u) {
      const long long row = __shfl_sync(0xffffffffu, at, u) + d;
      raw[u] = in ? *reinterpret_cast<const Raw*>(k_store + row) : Piece::zero();
    }
    const bool seen = j0 + (lane >> 1) <= pos;
    float p[HB];
#pragma unroll
    for (int i = 0; i < HB; ++i) {
      float s[ROW_KEYS];
#pragma unroll
      for (int u = 0; u < ROW_KEYS; ++u) {
        const float4 k = Piece::open(raw[u]);
        s[u] = qv[i].x * k.x + qv[i].y * k.y + qv[i].z * k.z + qv[i].w * k.w;
      }
      if (i == HB - 1) {
        // the keys are used: their values take their place
#pragma unroll
        for (int u = 0; u < ROW_KEYS; ++u) {
          const long long row = __shfl_sync(0xffffffffu, at, u) + d;
          raw[u] = in && j0 + u <= pos ? *reinterpret_cast<const Raw*>(v_store + row) : Piece::zero();
        }
      }
#pragma unroll
      for (int w = ROW_KEYS / 2; w >= 1; w >>= 1) {
        const bool upper = (lane & (2 * w)) != 0;
#pragma unroll
        for (int c = 0; c < w; ++c) {
          const float send = upper ? s[c] : s[c + w], keep = upper ? s[c + w] : s[c];
          s[c] = keep + __shfl_xor_sync(0xffffffffu, send, 2 * w);
        }
      }
      s[0] += __shfl_xor_sync(0xffffffffu, s[0], 1);
      const float m_new = fmaxf(m[i], warp_max(seen ? s[0] : -INFINITY));
      // (scores of minus infinity alone, so far: they weigh nothing, whatever the other warps have)
      const float m_use = m_new == -INFINITY ? 0.f : m_new, alpha = expf(m[i] - m_use);
      p[i] = seen ? expf(s[0] - m_use) : 0.f;
      l[i] = l[i] * alpha + p[i];
      acc[i].x *= alpha; acc[i].y *= alpha; acc[i].z *= alpha; acc[i].w *= alpha;
      m[i] = m_new;
    }
#pragma unroll
    for (int u = 0; u < ROW_KEYS; ++u) {
      const float4 v = Piece::open(raw[u]);          // (zeros past the last key)
#pragma unroll
      for (int i = 0; i < HB; ++i) {
        const float pu = __shfl_sync(0xffffffffu, p[i], 2 * u);
        acc[i].x += pu * v.x; acc[i].y += pu * v.y; acc[i].z += pu * v.z; acc[i].w += pu * v.w;
      }
    }
  }
#pragma unroll
  for (int i = 0; i < HB; ++i) {
    const float sum = warp_sum((lane & 1) ? 0.f : l[i]);
    *reinterpret_cast<float4*>(&sums[warp][i][d]) = acc[i];
    if (lane == 0) {
      most[warp][i] = m[i];
      total[warp][i] = sum;
    }
  }
  __syncthreads();
  const int w0 = warp - turn;
  for (int i = turn; i < here; i += W) {
    // (a warp without keys has minus infinity and zeros)
    float top = most[w0][i];
#pragma unroll
    for (int w = 1; w < W; ++w) top = fmaxf(top, most[w0 + w][i]);
    float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
    float sum = 0.f;
#pragma unroll
    for (int w = 0; w < W; ++w) {
      const float by = expf(most[w0 + w][i] - top);
      const float4 a = *reinterpret_cast<const float4*>(&sums[w0 + w][i][d]);
      sum += by * total[w0 + w][i];
      o.x += by * a.x; o.y += by * a.y; o.z += by * a.z; o.w += by * a.w;
    }
    if (in) {
      const float inv = 1.f / sum;
      T* to = out + ((size_t)token * heads + h0 + i) * head_dim + d;
      to[0] = from_f<T>(o.x * inv);
      to[1] = from_f<T>(o.y * inv);
      to[2] = from_f<T>(o.z * inv);
      to[3] = from_f<T>(o.w * inv);
    }
  }
}

template <typename T>
static int rowwise_group(const void* q, void* out, const void* k_store, const void* v_store, const int* block_table, int table_stride,
                         const int* tok_slot, const int* tok_pos, int n_tokens, int heads, int kv_heads, int head_dim, float scale,
                         int window, cudaStream_t s) {
  const int group = heads / kv_heads;
  const long long fours = (long long)n_tokens * kv_heads * ((group + 3) / 4), ones = (long long)n_tokens * heads;
  if (group >= 4 && ones >= 8 * 148)
    attention_rowwise_group_kernel<T, 4><<<(unsigned)fours, 128, 0, s>>>(
        (const T*)q, (T*)out, (const T*)k_store, (const T*)v_store, block_table, table_stride, tok_slot, tok_pos, heads, kv_heads, head_dim,
        scale, window, (unsigned)fours);
  else
    attention_rowwise_group_kernel<T, 1><<<(unsigned)((ones + 1) / 2), 128, 0, s>>>(
        (const T*)q, (T*)out, (const T*)k_store, (const T*)v_store, block_table, table_stride, tok_slot, tok_pos, heads, kv_heads, head_dim,
        scale, window, (unsigned)ones);
  return SB_LAUNCH_RESULT();
}

extern "C" {

// q, out: [n_tokens, heads * head_dim].  window <= 0 means all keys.
int sb_attention_rowwise(int dtype, const void* q, void* out, const void* k_store, const void* v_store,
                         const int* block_table, int table_stride, const int* tok_slot,
                         const int* tok_pos, int n_tokens, int heads, int kv_heads, int head_dim,
                         float scale, int window, cudaStream_t s) {
  if (head_dim > 32 * SB_ROW_MAX_D || kv_heads <= 0 || heads % kv_heads) return -2;
  const long long warps = (long long)n_tokens * heads;
  if (warps == 0) return 0;
  const int threads = 128;
  const long long blocks = (warps * 32 + threads - 1) / threads;
  if (head_dim <= 128 && head_dim % 4 == 0 && !(((uintptr_t)q | (uintptr_t)k_store | (uintptr_t)v_store) % 16)) {
    return dtype == 0 ? rowwise_group<float>(q, out, k_store, v_store, block_table, table_stride, tok_slot, tok_pos, n_tokens, heads,
                                             kv_heads, head_dim, scale, window, s)
                      : rowwise_group<bf16>(q, out, k_store, v_store, block_table, table_stride, tok_slot, tok_pos, n_tokens, heads,
                                            kv_heads, head_dim, scale, window, s);
  }
  if (dtype == 0)
    attention_rowwise_kernel<float><<<(unsigned)blocks, threads, 0, s>>>(
        (const float*)q, (float*)out, (const float*)k_store, (const float*)v_store, block_table,
        table_stride, tok_slot, tok_pos, n_tokens, heads, kv_heads, head_dim, scale, window);
  else
    attention_rowwise_kernel<bf16><<<(unsigned)blocks, threads, 0, s>>>(
        (const bf16*)q, (bf16*)out, (const bf16*)k_store, (const bf16*)v_store, block_table,
        table_stride, tok_slot, tok_pos, n_tokens, heads, kv_heads, head_dim, scale, window);
  return SB_LAUNCH_RESULT();
}

}  // extern "C"
