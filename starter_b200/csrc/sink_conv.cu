// The short convolution over [q | k | v] of a window attention, the RMS norms of its query and key rows, their rotation (neighbouring
// pairs) and the write of keys and values into the cache, in one pass (short_conv.cu and sink_prepare_norm of attention_sink.cu
// are the same in two, with the convolved rows in memory between them).
//
// A thread owns four neighbouring channels of CH consecutive tokens of a sequence: its taps, biases and gains are read once, its
// tokens' inputs (and the K - 1 in front of them) are in flight together, the convolved values stay in registers as the bfloat16 that the
// separate kernels would have filed, and the rows' squares of all CH tokens meet behind one barrier, with the angles and pages on their way.
// Queries and the keys and values are blocks of their own, so that two of them share an SM and one's loads run beside the other's sums (a
// block of all 3,072 channels: 22 us of a pass).  In two kernels 2,048 tokens of 24 heads of 128 spend 7 and 15 us, most of it issue slots
// for indexes, partners and small loads; here 14.  At the 64 registers that two blocks of 512 threads leave, eight tokens a thread spill 52 to
// 100 bytes of stores and as many to 164 of loads (three taps 80 and 144), two tokens none.
// A layer, two kernels / two tokens a thread / eight (us): captured, single tokens of 1 sequence 27.8 / 26.8 / 29.4, of 30 43.3 / 39.2 / 41.3, 256
// tokens 35.0 / 30.9 / 33.8, 600 55.1 / 52.0 / 52.8; 900 66.9 / 63.2 / 61.8, 1,184 85.3 / 83.6 / 80.7, 2 x 700 77.2 / 75.4 / 76.6, 1,500 93.4 / 90.8 /
// 91.3, 2,048 104.9 / 104.0 / 101.5.
#include "common.cuh"

struct SinkConvArgs {
  const bf16* x;                 // [tokens, ldx]
  int ldx;
  const float *taps, *in_bias;   // [channels][K], [channels] or null
  float* state;                  // a slot's K - 1 rows of `channels`, or null with one tap
  long long slot_stride;
  const int *seq_slot, *seq_q_start, *seq_q_len, *tok_pos, *block_table;
  int table_stride, chunks;
  const float *q_gain, *k_gain;  // [heads dim], [kv_heads dim], or both null
  float eps;
  const float *cos_t, *sin_t;    // [positions, rot / 2]
  int rot, heads, kv_heads, dim, vdim;
  bf16 *q, *k_store, *v_store;   // q: [tokens, heads dim]
};

__device__ __forceinline__ void sink_unpack4(const uint2& v, float* f) {
  f[0] = __uint_as_float(v.x << 16);
  f[1] = __uint_as_float(v.x & 0xffff0000u);
  f[2] = __uint_as_float(v.y << 16);
  f[3] = __uint_as_float(v.y & 0xffff0000u);
}
__device__ __forceinline__ uint2 sink_pack4(const float* f) {
  const __nv_bfloat162 p = __floats2bfloat162_rn(f[0], f[1]), q = __floats2bfloat162_rn(f[2], f[3]);
  return make_uint2(*reinterpret_cast<const uint32_t*>(&p), *reinterpret_cast<const uint32_t*>(&q));
}
__device__ __forceinline__ void sink_four(float* f, const float4& v) { f[0] = v.x; f[1] = v.y; f[2] = v.z; f[3] = v.w; }

template <int K, int CH>
__global__ void __launch_bounds__(512, 2)
sink_conv_kernel(const SinkConvArgs args) {
  constexpr int B = K - 1;
  static_assert(B <= CH, "only a sequence's first chunk reads what earlier steps left");
  __shared__ float shares[CH][17];
  __shared__ float inverse[CH];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int q_size = args.heads * args.dim, k_size = args.kv_heads * args.dim;
  const int channels = q_size + k_size + args.kv_heads * args.vdim;
  const int c = (blockIdx.y ? q_size : 0) + tid * 4;      // (a grid row each: queries, keys and values)
  const int kind = c < q_size ? 0 : c < q_size + k_size ? 1 : 2;            // (the same in a whole warp)
  const bool mine = blockIdx.y ? c < channels : c < q_size;
  // ---- weights, ahead of the wait
  float tap[4 * K] = {}, ib[4] = {0.f, 0.f, 0.f, 0.f};                          // tap[K e + j]: channel e, the input K - 1 - j tokens back
#pragma unroll
  for (int n = 0; n < K && mine; ++n) sink_four(tap + 4 * n, *reinterpret_cast<const float4*>(args.taps + (size_t)c * K + 4 * n));
  if (args.in_bias && mine) sink_four(ib, *reinterpret_cast<const float4*>(args.in_bias + c));
  const bool normed = args.q_gain && kind < 2;
  pdl_trigger_small();
  pdl_wait();
  const bf16* x = args.x;
  float* state = args.state;
  const int *slots = args.seq_slot, *starts = args.seq_q_start, *lens = args.seq_q_len, *places = args.tok_pos, *table = args.block_table;
  SB_BEHIND_WAIT(x); SB_BEHIND_WAIT(state); SB_BEHIND_WAIT(slots); SB_BEHIND_WAIT(starts); SB_BEHIND_WAIT(lens);
  SB_BEHIND_WAIT(places); SB_BEHIND_WAIT(table);
  const int seq = blockIdx.x / args.chunks, chunk = blockIdx.x - seq * args.chunks;
  const int q_len = lens[seq], t0 = chunk * CH;
  if (t0 >= q_len) return;                          // (the whole block)
  const int here = min(CH, q_len - t0), slot = slots[seq];
  const size_t row0 = (size_t)starts[seq] + t0;
  const bf16* xc = x + row0 * args.ldx + c;
  uint2 raw[B + CH];                                                      // from B tokens in front of the chunk on
#pragma unroll
  for (int i = 0; i < B + CH; ++i)
    raw[i] = mine && t0 + i - B >= 0 && i - B < here ? *reinterpret_cast<const uint2*>(xc + (long long)(i - B) * args.ldx) : make_uint2(0u, 0u);
  float in[K][4];                                                         // in[i % K]: token t0 + i - B
#pragma unroll
  for (int i = 0; i < B; ++i) {
    sink_unpack4(raw[i], in[i]);
#pragma unroll
    for (int e = 0; e < 4; ++e) in[i][e] += ib[e];
  }
  if (chunk == 0 && B > 0 && mine) {
    // what earlier steps left in front of the sequence, and what the next one will find (row j: the input j + 1 tokens back)
    float* st = state + (size_t)slot * args.slot_stride + c;
    float old[B > 0 ? B : 1][4];
#pragma unroll
    for (int j = 0; j < B; ++j) sink_four(old[j], *reinterpret_cast<const float4*>(st + (size_t)j * channels));
#pragma unroll
    for (int j = 0; j < B; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) in[B - 1 - j][e] = old[j][e];
#pragma unroll
    for (int j = 0; j < B; ++j) {
      const int t = q_len - 1 - j;
      float v[4];
      if (t >= 0) {
        sink_unpack4(*reinterpret_cast<const uint2*>(xc + (long long)t * args.ldx), v);
#pragma unroll
        for (int e = 0; e < 4; ++e) v[e] += ib[e];
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          v[e] = 0.f;
#pragma unroll
          for (int o = 0; o < B; ++o)
            if (o == -t - 1) v[e] = old[o][e];
        }
      }
      *reinterpret_cast<float4*>(st + (size_t)j * channels) = make_float4(v[0], v[1], v[2], v[3]);
    }
  }
  uint2 y[CH];
#pragma unroll
  for (int i = 0; i < CH; ++i) {
    float a[4], *now = in[(B + i) % K];
    sink_unpack4(raw[B + i], now);
    float sq = 0.f;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      now[e] += ib[e];
      a[e] = __fmul_rn(tap[K * e + B], now[e]);
#pragma unroll
      for (int j = 1; j < K; ++j) a[e] = fmaf(tap[K * e + B - j], in[(B + i - j) % K][e], a[e]);
    }
    y[i] = sink_pack4(a);
    if (normed) {
      sink_unpack4(y[i], a);
#pragma unroll
      for (int e = 0; e < 4; ++e) sq += a[e] * a[e];
      sq = warp_sum(sq);
      if (lane == 0) shares[i][warp] = sq;
    }
  }
  const int of_kind = kind == 0 ? c : kind == 1 ? c - q_size : c - q_size - k_size, size = kind == 2 ? args.vdim : args.dim;
  const int h = of_kind / size, d = of_kind - h * size;
  const bool turns = kind < 2 && d < args.rot;
  // the tokens' places and angles, all asked for at once (positions of a sequence's tokens follow each other)
  const int pos0 = __ldg(places + row0);
  float gain[4] = {1.f, 1.f, 1.f, 1.f};
  if (normed && mine) sink_four(gain, *reinterpret_cast<const float4*>(kind == 0 ? args.q_gain + c : args.k_gain + (c - q_size)));
  float2 co[CH], si[CH];
#pragma unroll
  for (int i = 0; i < CH; ++i) {
    const size_t at = (size_t)(pos0 + min(i, here - 1)) * (args.rot / 2) + d / 2;
    co[i] = turns ? __ldg(reinterpret_cast<const float2*>(args.cos_t + at)) : make_float2(1.f, 1.f);
    si[i] = turns ? __ldg(reinterpret_cast<const float2*>(args.sin_t + at)) : make_float2(0.f, 0.f);
  }
  int page[2] = {0, 0};                             // (CH tokens lie on two pages at most)
  if (kind) {
    const int* row = table + (size_t)slot * args.table_stride;
    page[0] = __ldg(row + pos0 / SB_PAGE_TOKENS);
    page[1] = __ldg(row + (pos0 + here - 1) / SB_PAGE_TOKENS);
  }
  if (args.q_gain) {                                // the rows' squares: a warp a token, over the block's warps of queries, or of keys
    __syncthreads();
    const int from = (blockIdx.y ? k_size : q_size) / 128;
    for (int i = warp; i < CH; i += blockDim.x >> 5) {
      const float sum = warp_sum(lane < from ? shares[i][lane] : 0.f);
      if (lane == 0) inverse[i] = 1.f / sqrtf(sum / (float)(blockIdx.y ? k_size : q_size) + args.eps);
    }
    __syncthreads();
  }
  if (!mine) return;
#pragma unroll
  for (int i = 0; i < CH; ++i) {
    if (i >= here) break;
    bf16* to;
    if (kind == 0) {
      to = args.q + (row0 + i) * q_size + c;
    } else {
      const int pos = pos0 + i;
      const int p = pos / SB_PAGE_TOKENS == pos0 / SB_PAGE_TOKENS ? page[0] : page[1];
      to = (kind == 1 ? args.k_store : args.v_store) + page_row(p, h, pos % SB_PAGE_TOKENS, args.kv_heads, size) + d;
    }
    if (normed || turns) {
      float a[4];
      sink_unpack4(y[i], a);
      if (normed) {
        const float inv = inverse[i];
#pragma unroll
        for (int e = 0; e < 4; ++e) a[e] *= inv * gain[e];
      }
      if (turns) {
        const float u0 = a[0] * co[i].x - a[1] * si[i].x, u1 = a[1] * co[i].x + a[0] * si[i].x;
        const float v0 = a[2] * co[i].y - a[3] * si[i].y, v1 = a[3] * co[i].y + a[2] * si[i].y;
        a[0] = u0; a[1] = u1; a[2] = v0; a[3] = v1;
      }
      y[i] = sink_pack4(a);
    }
    *reinterpret_cast<uint2*>(to) = y[i];
  }
}

extern "C" {

// x: [n_tokens, ldx] bfloat16, a row = [q (heads * dim) | k (kv_heads * dim) | v (kv_heads * vdim) | ..]; taps float [channels, K] and
// in_bias float [channels] or null over those channels; state: float, a slot's K - 1 rows of them start at the pointer (as sb_short_conv's,
// no activation); gains, tables and stores as sb_sink_prepare_norm's (pairs of neighbours; keys and values are filed); q: [n_tokens,
// heads * dim].  tok_pos: a sequence's positions follow each other (the first of every chunk of tokens is read).  -2: not taken (the separate kernels take anything): whole warps of queries, keys and values, up to 2,048 channels of queries
// and of keys and values, 1 to 4 taps, everything on 16 bytes.
int sb_sink_conv(const void* x, int ldx, const float* taps, int K, const float* in_bias, float* state, long long slot_stride,
                 const int* seq_slot, const int* seq_q_start, const int* seq_q_len, int n_seqs, int max_q_len, const int* tok_pos,
                 const int* block_table, int table_stride, const float* q_gain, const float* k_gain, float eps, const float* cos_t,
                 const float* sin_t, int rot, int heads, int kv_heads, int dim, int vdim, void* q, void* k_store, void* v_store,
                 cudaStream_t s) {
  if (n_seqs == 0) return 0;
  if (heads < 1 || kv_heads < 1 || dim < 8 || vdim < 8 || K < 1 || K > 4 || max_q_len < 1) return -2;
  const long long channels = (long long)heads * dim + (long long)kv_heads * (dim + vdim);
  if ((heads * dim) % 128 || (kv_heads * dim) % 128 || (kv_heads * vdim) % 128 || dim % 8 || vdim % 8 || heads * dim > 2048 || channels - heads * dim > 2048)
    return -2;
  if (rot < 0 || rot > dim || rot % 8 || (rot && (!cos_t || !sin_t)) || (!q_gain != !k_gain) || (K > 1 && !state)) return -2;
  if (ldx % 8 || ldx < channels || slot_stride % 4) return -2;
  if (((uintptr_t)x | (uintptr_t)taps | (uintptr_t)in_bias | (uintptr_t)state | (uintptr_t)q_gain | (uintptr_t)k_gain | (uintptr_t)cos_t |
       (uintptr_t)sin_t | (uintptr_t)q | (uintptr_t)k_store | (uintptr_t)v_store) % 16) return -2;
  // eight tokens a thread once that gives every SM a block, else two (which have to reach over the taps): measured above, within 4 %
  // of each other from 600 to 1,500 tokens
  const bool many = K > 3 || (long long)n_seqs * ((max_q_len + 7) / 8) >= 148;
  const int chunk = many ? 8 : 2, chunks = (max_q_len + chunk - 1) / chunk;
  const int kv_size = kv_heads * (dim + vdim), threads = (heads * dim > kv_size ? heads * dim : kv_size) / 4;
  const SinkConvArgs args = {(const bf16*)x, ldx, taps, in_bias, state, slot_stride, seq_slot, seq_q_start, seq_q_len, tok_pos, block_table,
                             table_stride, chunks, q_gain, k_gain, eps, cos_t, sin_t, rot, heads, kv_heads, dim, vdim, (bf16*)q,
                             (bf16*)k_store, (bf16*)v_store};
  const dim3 grid((unsigned)(n_seqs * chunks), 2);
#define CONV_GO(TAPS) case TAPS: return launch_dependent(many ? sink_conv_kernel<TAPS, 8> : sink_conv_kernel<TAPS, TAPS == 4 ? 8 : 2>, grid, dim3(threads), 0, s, args)
  switch (K) {
    CONV_GO(1);
    CONV_GO(2);
    CONV_GO(3);
    CONV_GO(4);
  }
#undef CONV_GO
  return -2;
}

}  // extern "C"
