// A routed mixture of small gated feed-forward experts, for any number of tokens, without a word
// from the host between its kernels (so that it can sit inside a captured step).
//
//   route    z = W_r h + b in float; the `top` largest (the lower index first among equals); their
//            weights are the softmax over those `top` logits alone (scoring 0), or their sigmoids divided
//            by the sum of those sigmoids (+ 1e-20) and multiplied by a constant (scoring 1), or the plain
//            sigmoids times a constant (scoring 3).
//   align    the (token, choice) pairs grouped by expert: every expert's pairs fill whole tiles of
//            rows (32, or 64 for the tensor-core tiles; padded with -1), `tile_expert` names each tile's expert, `n_tiles` counts them.
//   up       per tile: g = min(gate(h), limit), u = clamp(up(h), -limit, limit),
//            a = g * sigmoid(1.702 g) * (u + 1), for the tile's rows gathered from h (expert kind 1);
//            or, for experts without a gate, a = relu(up(h))^2 (expert kind 2); with limit 0 the gated kind
//            has no clamps and the plain gate: a = silu(gate(h)) * up(h).
//            A weight that belongs in front of an expert (expert(w h) instead of w expert(h)) multiplies the up
//            pass's products, which are linear in the row, ahead of the activation; combine then only sums.
//   down     per tile: the expert's down projection of a, filed at the pair's own place.
//   combine  out[t] = sum_c weight[t][c] * down[t][c], summed in float in the order of the choices.
//
// A second router (route_all) scores by the softmax over ALL its outputs, chooses by score + correction among the
// experts of the best groups, and may have more outputs than there are experts: a choice from `experts` on is
// an identity expert, which has no weights.  align leaves such pairs out of the tiles and combine adds the
// token's own row in their place.  combine also adds a shared expert's output times a gate per token.
//
// Products accumulate in float; gate and up are rounded to the working type before the activation, as
// the projections of the dense feed-forward are.  A token's result depends on nothing but its own row
// and the experts' weights: not on which tile it landed in, nor on who else is in the step.
#include <mma.h>

#include "common.cuh"

#define MOE_BM 32
#define MOE_BN 64
#define MOE_BK 32
#define MOE_MAX_EXPERTS 1024
#define MOE_MAX_TOP 16
#define MOE_STAGE_BYTES 32768

// The gated expert's activation from its (rounded) gate and up products.  limit > 0: the clamped gate,
// min(g, limit) * sigmoid(1.702 min(g, limit)) * (clamp(u, -limit, limit) + 1); limit == 0: no clamps and the
// plain gate silu(g) * u.
__device__ __forceinline__ float moe_gate(float g, float u, float limit) {
  if (limit > 0.f) {
    g = fminf(g, limit);
    u = fminf(fmaxf(u, -limit), limit);
    return g / (1.f + expf(-1.702f * g)) * (u + 1.f);
  }
  return g / (1.f + expf(-g)) * u;
}

// The logits of TOK tokens from `row0` on (rows past `n_tokens` repeat the last one): z[token][output].  A warp takes EXP outputs
// and all TOK tokens at a time: a piece of a router's row serves TOK tokens, a piece of a token EXP outputs (one output a warp and one token
// a block read 128 KB of router from L2 a token with 16 experts of 2,048: 46 us for 2,048 tokens, 18 with four; moe_route_many_kernel 12).  A sum is the
// same whatever EXP and TOK are.
template <typename T, int TOK, int EXP>
__device__ __forceinline__ void moe_logits(const T* __restrict__ h, const float* __restrict__ w, const float* __restrict__ b,
                                           float* z, int ldz, int row0, int n_tokens, int width, int outputs, int rows) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  // (16-byte pieces of the router's rows when the rows allow it)
  const bool wide = width % 4 == 0 && ((uintptr_t)w % 16) == 0 && ((uintptr_t)h % 8) == 0;
  const T* ht[TOK];
#pragma unroll
  for (int t = 0; t < TOK; ++t) ht[t] = h + (size_t)min(row0 + t, n_tokens - 1) * width;
  for (int e0 = warp * EXP; e0 < rows; e0 += warps * EXP) {
    const float* wr[EXP];
#pragma unroll
    for (int e = 0; e < EXP; ++e) wr[e] = w + (size_t)min(e0 + e, rows - 1) * width;
    float a[EXP][TOK];
#pragma unroll
    for (int e = 0; e < EXP; ++e)
#pragma unroll
      for (int t = 0; t < TOK; ++t) a[e][t] = 0.f;
    if (wide && sizeof(T) == 2) {
      // BATCH pieces of every row in flight together (no condition between the loads and the sums, or the compiler moves each
      // load to its use)
      constexpr int BATCH = TOK * EXP == 1 ? 16 : 4;
      const int pieces = width / 4;
      auto add = [](float& sum, const uint2& hv, const float4& wv) {
        sum += __uint_as_float(hv.x << 16) * wv.x + __uint_as_float(hv.x & 0xffff0000u) * wv.y +
               __uint_as_float(hv.y << 16) * wv.z + __uint_as_float(hv.y & 0xffff0000u) * wv.w;
      };
      int c0 = 0;
      for (; c0 + 32 * BATCH <= pieces; c0 += 32 * BATCH) {
        float4 wv[BATCH][EXP];
        uint2 hv[BATCH][TOK];
#pragma unroll
        for (int i = 0; i < BATCH; ++i) {
#pragma unroll
          for (int e = 0; e < EXP; ++e) wv[i][e] = reinterpret_cast<const float4*>(wr[e])[c0 + 32 * i + lane];
#pragma unroll
          for (int t = 0; t < TOK; ++t) hv[i][t] = reinterpret_cast<const uint2*>(ht[t])[c0 + 32 * i + lane];
        }
#pragma unroll
        for (int i = 0; i < BATCH; ++i)
#pragma unroll
          for (int e = 0; e < EXP; ++e)
#pragma unroll
            for (int t = 0; t < TOK; ++t) add(a[e][t], hv[i][t], wv[i][e]);
      }
      for (int c = c0 + lane; c < pieces; c += 32) {
#pragma unroll
        for (int e = 0; e < EXP; ++e) {
          const float4 wv = reinterpret_cast<const float4*>(wr[e])[c];
#pragma unroll
          for (int t = 0; t < TOK; ++t) add(a[e][t], reinterpret_cast<const uint2*>(ht[t])[c], wv);
        }
      }
    } else {
      for (int c = lane; c < width; c += 32)
#pragma unroll
        for (int e = 0; e < EXP; ++e)
#pragma unroll
          for (int t = 0; t < TOK; ++t) a[e][t] += to_f<T>(ht[t][c]) * wr[e][c];
    }
#pragma unroll
    for (int e = 0; e < EXP; ++e)
#pragma unroll
      for (int t = 0; t < TOK; ++t) {
        const float v = warp_sum(a[e][t]);
        if (lane == 0 && e0 + e < rows) z[t * ldz + e0 + e] = v + (b && e0 + e < outputs ? b[e0 + e] : 0.f);
      }
  }
}

// The block's TOK rows of h into shared memory, all pieces in flight at once (a warp that reads them piece by piece beside the
// router's rows waits for memory eight times); returns where they are, or null where they do not fit or come in no whole pieces.
template <typename T, int TOK>
__device__ __forceinline__ const T* moe_stage_rows(const T* __restrict__ h, unsigned char* to, int row0, int n_tokens, int width) {
  if (TOK == 1 || (width * sizeof(T)) % 16 || ((uintptr_t)h % 16) || TOK * width * sizeof(T) > MOE_STAGE_BYTES) return nullptr;
  const int pieces = width * (int)sizeof(T) / 16;
#pragma unroll
  for (int t = 0; t < TOK; ++t) {
    const unsigned char* from = reinterpret_cast<const unsigned char*>(h + (size_t)min(row0 + t, n_tokens - 1) * width);
    for (int c = threadIdx.x; c < pieces; c += blockDim.x) {
      const unsigned d = (unsigned)__cvta_generic_to_shared(to + ((size_t)t * pieces + c) * 16);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(from + (size_t)c * 16) : "memory");
    }
  }
  asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  return reinterpret_cast<const T*>(to);
}

// TOK tokens a block; a warp chooses for a token.
template <typename T, int TOK>
__global__ void __launch_bounds__(512) moe_route_kernel(const T* __restrict__ h, const float* __restrict__ w, const float* __restrict__ b,
                                 int* __restrict__ ids, float* __restrict__ weights, int n_tokens, int width, int experts, int top,
                                 int scoring, float weight_scale) {
  extern __shared__ __align__(16) unsigned char route_smem[];
  float* route_z = reinterpret_cast<float*>(route_smem + (TOK > 1 ? MOE_STAGE_BYTES : 0));
  pdl_trigger();
  pdl_wait();
  SB_BEHIND_WAIT(h);
  const int row0 = blockIdx.x * TOK;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const T* staged = moe_stage_rows<T, TOK>(h, route_smem, row0, n_tokens, width);
  moe_logits<T, TOK, TOK>(staged ? staged : h, w, b, route_z, experts, staged ? 0 : row0, staged ? TOK : n_tokens, width, experts, experts);
  __syncthreads();
  for (int t = warp; t < TOK && row0 + t < n_tokens; t += warps) {
    const int row = row0 + t;
    float* z = route_z + t * experts;
    float best[MOE_MAX_TOP];
    float top_max = 0.f;
    for (int c = 0; c < top; ++c) {
      // the largest logit left, the lowest index among equals
      float v = -INFINITY;
      int at = 0x7fffffff;
      for (int e = lane; e < experts; e += 32)
        if (z[e] > v) { v = z[e]; at = e; }
      for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, v, o);
        const int oa = __shfl_xor_sync(0xffffffffu, at, o);
        if (ov > v || (ov == v && oa < at)) { v = ov; at = oa; }
      }
      if (at >= experts) at = 0;          // no finite logit left: keep the indices inside the table
      if (c == 0) top_max = v;
      best[c] = v;
      __syncwarp();
      if (lane == 0) {
        ids[(size_t)row * top + c] = at;
        z[at] = -INFINITY;
      }
      __syncwarp();
    }
    if (lane == 0) {
      float sum = 0.f;
      for (int c = 0; c < top; ++c) {
        best[c] = scoring != 0 ? 1.f / (1.f + expf(-best[c])) : expf(best[c] - top_max);
        sum += best[c];
      }
      if (scoring == 3) {
        for (int c = 0; c < top; ++c) weights[(size_t)row * top + c] = best[c] * weight_scale;
      } else if (scoring == 1) {
        for (int c = 0; c < top; ++c) weights[(size_t)row * top + c] = best[c] / (sum + 1e-20f) * weight_scale;
      } else {
        for (int c = 0; c < top; ++c) weights[(size_t)row * top + c] = best[c] / sum;
      }
    }
  }
}

// ROUTE_TOKENS tokens a block, bfloat16 rows in whole 16-byte pieces, up to ROUTE_EXPERTS experts.  What bounds the router is the way from
// L2: a block of four tokens brings all router rows for those four (512 blocks times 128 KB with 16 experts of 2,048: 64 MB), a block of
// sixteen a quarter of that; rows and tokens pass through shared memory, 512 entries of each a stage, two stages ahead.  A warp
// keeps the sums of TPW tokens and eight experts (a piece of a router's row serves TPW tokens, a piece of a token eight experts), and
// each sum has the terms and the order that moe_logits gives it: the same bits.  The choice keeps a token's logits in the lanes'
// registers and finds the largest by the warp's integer maximum.
// Both kinds run in waves: 1,184 tokens (more than 16 experts) or 2,368 (up to 16) of four a block, 2,368 of sixteen a block; and a block's
// passes over 16 experts are a chain.  So more than 16 experts want more than a wave of the other kind.  Measured, four tokens a block /
// here, us, width 2,048, in a row (and with the caches emptied in front, as behind other layers): 8 experts 592 tokens 8.6 / 6.6 (18.4 / 12.3);
// 16 592 8.7 / 8.4 (18.4 / 14.3), 2,368 13.1 / 10.9 (20.5 / 16.4), 5,000 31.7 / 27.2 (41 / 33); 32 1,184 10.3 / 14.8 (20.4 / 20.7), 1,400 19.1 /
// 14.8 (30.7 / 22.5), 2,600 28.3 / 28.5 (39 / 35); 48 1,184 15.2 / 20.9 (30.7 / 28.7), 1,400 28.7 / 21.0 (45 / 29), 2,600 42.7 / 40.7 (59 / 49); 64
// 1,184 16.2 / 27.0 (30.7 / 34.8), 1,400 30.8 / 27.3 (45 / 35), 2,600 45.8 / 52.9 (61.4 / 59.4), 8,192 112 / 109 (127 / 115).  Stages of 256 entries,
// four: 13.2 for 12.4 (2,048 tokens of 16 experts).
#define ROUTE_TOKENS 16
#define ROUTE_EXPERTS 64
#define ROUTE_STAGES 3
#define ROUTE_K 512
template <int GROUPS>
__global__ void __launch_bounds__(256) moe_route_many_kernel(const bf16* __restrict__ h, const float* __restrict__ w, const float* __restrict__ b,
                                 int* __restrict__ ids, float* __restrict__ weights, int n_tokens, int width, int experts, int top,
                                 int scoring, float weight_scale) {
  // GROUPS of eight experts at a time, eight warps: 8 / GROUPS warps of TPW tokens each
  constexpr int TPW = ROUTE_TOKENS * GROUPS / 8, EPP = 8 * GROUPS;
  constexpr int W_BYTES = EPP * ROUTE_K * 4, STAGE = W_BYTES + ROUTE_TOKENS * ROUTE_K * 2;
  extern __shared__ __align__(16) unsigned char route_smem[];
  __shared__ float z[ROUTE_TOKENS][ROUTE_EXPERTS];
  pdl_trigger();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, row0 = blockIdx.x * ROUTE_TOKENS;
  const int group = warp % GROUPS, t0 = warp / GROUPS * TPW;
  const int stages = (width + ROUTE_K - 1) / ROUTE_K, all = stages * ((experts + EPP - 1) / EPP);
  const unsigned smem = (unsigned)__cvta_generic_to_shared(route_smem);
  // a stage: the pass's router rows and the block's tokens, zeros behind the width
  auto bring_router = [&](int e0, int k0, int slot) {
#pragma unroll
    for (int i = 0; i < EPP * (ROUTE_K / 4) / 256; ++i) {
      const int c = threadIdx.x + 256 * i, e = min(e0 + c / (ROUTE_K / 4), experts - 1), k = k0 + c % (ROUTE_K / 4) * 4;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem + slot * STAGE + c * 16),
                   "l"(w + (size_t)e * width + min(k, width - 4)), "r"(k < width ? 16 : 0) : "memory");
    }
  };
  auto bring_tokens = [&](int k0, int slot) {
#pragma unroll
    for (int i = 0; i < ROUTE_TOKENS * (ROUTE_K / 8) / 256; ++i) {
      const int c = threadIdx.x + 256 * i, t = min(row0 + c / (ROUTE_K / 8), n_tokens - 1), k = k0 + c % (ROUTE_K / 8) * 8;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem + slot * STAGE + W_BYTES + c * 16),
                   "l"(h + (size_t)t * width + min(k, width - 8)), "r"(k < width ? 16 : 0) : "memory");
    }
  };
  // (the router's rows are weights: the first stages' are asked for in front of the wait)
  int e_ahead = 0, k_ahead = 0;                    // the next stage to ask for
  auto next = [&] {
    if ((k_ahead += ROUTE_K) >= width) { k_ahead = 0; e_ahead += EPP; }
  };
  for (int i = 0; i < ROUTE_STAGES - 1 && i < all; ++i, next()) bring_router(e_ahead, k_ahead, i);
  pdl_wait();
  SB_BEHIND_WAIT(h);
  for (int i = 0, k = 0; i < ROUTE_STAGES - 1; ++i) {
    if (i < all) bring_tokens(k, i);
    asm volatile("cp.async.commit_group;" ::: "memory");
    if ((k += ROUTE_K) >= width) k = 0;
  }
  float a[8][TPW];
  int slot = 0, free_slot = ROUTE_STAGES - 1, left = stages, pass_e = 0;
#pragma unroll 1
  for (int at = 0; at < all; ++at) {
    if (left == stages)
#pragma unroll
      for (int e = 0; e < 8; ++e)
#pragma unroll
        for (int t = 0; t < TPW; ++t) a[e][t] = 0.f;
    asm volatile("cp.async.wait_group %0;" ::"n"(ROUTE_STAGES - 2) : "memory");
    __syncthreads();          // stage `at` is there for all, and nobody reads the stage before any more
    if (at + ROUTE_STAGES - 1 < all) {
      bring_router(e_ahead, k_ahead, free_slot);
      bring_tokens(k_ahead, free_slot);
      next();
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    const unsigned char* stage = route_smem + slot * STAGE;
    slot = slot == ROUTE_STAGES - 1 ? 0 : slot + 1;
    free_slot = free_slot == ROUTE_STAGES - 1 ? 0 : free_slot + 1;
#pragma unroll
    for (int piece = 0; piece < ROUTE_K / 128; ++piece) {
      float hv[TPW][4];
#pragma unroll
      for (int t = 0; t < TPW; ++t) {
        const uint2 v = reinterpret_cast<const uint2*>(stage + W_BYTES + (t0 + t) * ROUTE_K * 2)[piece * 32 + lane];
        hv[t][0] = __uint_as_float(v.x << 16);
        hv[t][1] = __uint_as_float(v.x & 0xffff0000u);
        hv[t][2] = __uint_as_float(v.y << 16);
        hv[t][3] = __uint_as_float(v.y & 0xffff0000u);
      }
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float4 wv = reinterpret_cast<const float4*>(stage + (group * 8 + e) * ROUTE_K * 4)[piece * 32 + lane];
#pragma unroll
        for (int t = 0; t < TPW; ++t) a[e][t] += hv[t][0] * wv.x + hv[t][1] * wv.y + hv[t][2] * wv.z + hv[t][3] * wv.w;
      }
    }
    if (--left == 0) {
      // the lanes' sums, a token's eight at a time: each step hands half of the values over and leaves the same tree as warp_sum's
      const int e0 = pass_e + group * 8;
      left = stages;
      pass_e += EPP;
#pragma unroll
      for (int t = 0; t < TPW; ++t) {
        float v[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) v[e] = a[e][t];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const bool up = lane & 16;
          const float got = __shfl_xor_sync(0xffffffffu, up ? v[e] : v[e + 4], 16);
          v[e] = (up ? v[e + 4] : v[e]) + got;
        }
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const bool up = lane & 8;
          const float got = __shfl_xor_sync(0xffffffffu, up ? v[e] : v[e + 2], 8);
          v[e] = (up ? v[e + 2] : v[e]) + got;
        }
        const bool up = lane & 4;
        const float got = __shfl_xor_sync(0xffffffffu, up ? v[0] : v[1], 4);
        float sum = (up ? v[1] : v[0]) + got;
        sum += __shfl_xor_sync(0xffffffffu, sum, 2);
        sum += __shfl_xor_sync(0xffffffffu, sum, 1);
        const int e = e0 + (lane >> 4) * 4 + (lane >> 3 & 1) * 2 + (lane >> 2 & 1);
        if ((lane & 3) == 0 && e < experts) z[t0 + t][e] = sum + (b ? b[e] : 0.f);
      }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  // a float as an integer of the same order; INT_MIN: nothing to choose (no number, or minus infinity)
  auto key = [](float v) {
    const int i = __float_as_int(v + 0.f);
    return v > -INFINITY ? i ^ (i >> 31 & 0x7fffffff) : (int)0x80000000;
  };
#pragma unroll 1
  for (int t = warp; t < ROUTE_TOKENS && row0 + t < n_tokens; t += 8) {
    const float z0 = lane < experts ? z[t][lane] : -INFINITY, z1 = lane + 32 < experts ? z[t][lane + 32] : -INFINITY;
    int k0 = key(z0), k1 = key(z1), chosen = 0;
    float best = 0.f, first = 0.f;
#pragma unroll 1
    for (int c = 0; c < top; ++c) {
      // the largest logit left, the lowest index among equals; none left: index 0, to keep inside the table
      const int most = __reduce_max_sync(0xffffffffu, max(k0, k1));
      const unsigned low = __ballot_sync(0xffffffffu, k0 == most), high = __ballot_sync(0xffffffffu, k1 == most);
      int at = low ? __ffs(low) - 1 : 31 + __ffs(high);
      float v = __shfl_sync(0xffffffffu, at < 32 ? z0 : z1, at & 31);
      if (most == (int)0x80000000) { at = 0; v = -INFINITY; }
      if (c == 0) first = v;
      if (lane == c) { best = v; chosen = at; }
      if (lane == (at & 31)) (at < 32 ? k0 : k1) = (int)0x80000000;
    }
    if (lane < top) best = scoring != 0 ? 1.f / (1.f + expf(-best)) : expf(best - first);
    float sum = 0.f;
#pragma unroll 1
    for (int c = 0; c < top; ++c) sum += __shfl_sync(0xffffffffu, best, c);
    if (lane < top) {
      const size_t to = (size_t)(row0 + t) * top + lane;
      ids[to] = chosen;
      weights[to] = scoring == 3 ? best * weight_scale : scoring == 1 ? best / (sum + 1e-20f) * weight_scale : best / sum;
    }
  }
}

// The router of the softmax over all outputs (see sb_moe_route_all).  z holds outputs + 1 logits (the last one
// the shared expert's gate, when asked for), then the scores, the choice numbers and the groups' maxima.
template <typename T, int TOK>
__global__ void __launch_bounds__(512) moe_route_all_kernel(const T* __restrict__ h, const float* __restrict__ w,
                                     const float* __restrict__ correction, int* __restrict__ ids,
                                     float* __restrict__ weights, float* __restrict__ gate_out, int n_tokens, int width, int outputs,
                                     int top, int groups, int keep, float weight_scale) {
  extern __shared__ __align__(16) unsigned char route_smem[];
  float* route_z = reinterpret_cast<float*>(route_smem + (TOK > 1 ? MOE_STAGE_BYTES : 0));
  pdl_trigger();
  pdl_wait();
  SB_BEHIND_WAIT(h);
  const int row0 = blockIdx.x * TOK, per_token = 3 * outputs + 1 + groups;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const T* staged = moe_stage_rows<T, TOK>(h, route_smem, row0, n_tokens, width);
  moe_logits<T, TOK, TOK>(staged ? staged : h, w, nullptr, route_z, per_token, staged ? 0 : row0, staged ? TOK : n_tokens, width, outputs,
                          outputs + (gate_out ? 1 : 0));
  __syncthreads();
  for (int t = warp; t < TOK && row0 + t < n_tokens; t += warps) {
    const int row = row0 + t;
    float* z = route_z + t * per_token;
    float* score = z + outputs + 1;
    float* choice = score + outputs;
    float* best_of = choice + outputs;
    if (gate_out && lane == 0) gate_out[row] = 1.f / (1.f + expf(-z[outputs]));
    float top_z = -INFINITY;
    for (int e = lane; e < outputs; e += 32) top_z = fmaxf(top_z, z[e]);
    top_z = warp_max(top_z);
    float sum = 0.f;
    for (int e = lane; e < outputs; e += 32) {
      const float v = expf(z[e] - top_z);
      score[e] = v;
      sum += v;
    }
    sum = warp_sum(sum);
    for (int e = lane; e < outputs; e += 32) {
      score[e] /= sum;
      choice[e] = score[e] + (correction ? correction[e] : 0.f);
    }
    __syncwarp();
    if (groups > 1) {
      const int per = outputs / groups;
      for (int g = lane; g < groups; g += 32) {
        float v = -INFINITY;
        for (int e = g * per; e < (g + 1) * per; ++e) v = fmaxf(v, choice[e]);
        best_of[g] = v;
      }
      __syncwarp();
      // the `keep` best groups are marked with +inf, then every other group's outputs leave the choice
      for (int c = 0; c < keep; ++c) {
        float v = -INFINITY;
        int at = 0x7fffffff;
        for (int g = lane; g < groups; g += 32)
          if (best_of[g] != INFINITY && (best_of[g] > v || at == 0x7fffffff)) { v = best_of[g]; at = g; }
        for (int o = 16; o > 0; o >>= 1) {
          const float ov = __shfl_xor_sync(0xffffffffu, v, o);
          const int oa = __shfl_xor_sync(0xffffffffu, at, o);
          if (oa != 0x7fffffff && (at == 0x7fffffff || ov > v || (ov == v && oa < at))) { v = ov; at = oa; }
        }
        if (lane == 0 && at < groups) best_of[at] = INFINITY;
        __syncwarp();
      }
      for (int e = lane; e < outputs; e += 32)
        if (best_of[e / per] != INFINITY) choice[e] = -INFINITY;
      __syncwarp();
    }
    float picked[MOE_MAX_TOP];
    for (int c = 0; c < top; ++c) {
      float v = -INFINITY;
      int at = 0x7fffffff;
      for (int e = lane; e < outputs; e += 32)
        if (choice[e] > v) { v = choice[e]; at = e; }
      for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, v, o);
        const int oa = __shfl_xor_sync(0xffffffffu, at, o);
        if (ov > v || (ov == v && oa < at)) { v = ov; at = oa; }
      }
      if (at >= outputs) at = 0;          // nothing left to choose from: keep the indices inside the table
      picked[c] = score[at];
      if (lane == 0) {
        ids[(size_t)row * top + c] = at;
        choice[at] = -INFINITY;
      }
      __syncwarp();
    }
    if (lane == 0) {
      float total = 0.f;
      for (int c = 0; c < top; ++c) total += picked[c];
      for (int c = 0; c < top; ++c) weights[(size_t)row * top + c] = picked[c] / (total + 1e-20f) * weight_scale;
    }
  }
}

// The lanes of the warp that hold the same number below 2^bits (a vote a bit; the hardware's own match takes a warp's time a
// distinct number).
__device__ __forceinline__ unsigned moe_same(int e, int bits) {
  unsigned same = 0xffffffffu;
  for (int b = 0; b < bits; ++b) {
    const bool set = (e >> b) & 1;
    const unsigned votes = __ballot_sync(0xffffffffu, set);
    same &= set ? votes : ~votes;
  }
  return same;
}

// One block.  ids: [n_pairs]; sorted: [capacity] receives pair numbers or -1; tile_expert: [max_tiles].
// The lanes of a warp that hold one expert count, and take their places, together (16 experts of 8,192 pairs would otherwise
// queue at 16 counters: 24 us of a prompt's step, 12 with votes, 7 by the cluster below).
__global__ void __launch_bounds__(1024)
moe_align_kernel(const int* __restrict__ ids, int n_pairs, int experts, int* __restrict__ sorted, int capacity,
                 int* __restrict__ tile_expert, int* __restrict__ n_tiles, int bm) {
  __shared__ int count[MOE_MAX_EXPERTS], offset[MOE_MAX_EXPERTS];
  pdl_trigger();
  pdl_wait();
  SB_BEHIND_WAIT(ids);
  const int tid = threadIdx.x, lane = tid & 31, threads = blockDim.x;
  const int bits = 32 - __clz(experts);             // (numbers up to `experts`, which stands for all that have no tile)
  for (int e = tid; e < experts; e += threads) count[e] = 0;
  __syncthreads();
  // (an id from `experts` on names an identity expert: it has no tile)
  // Up to eight pairs a thread keep their experts and the places that the count gave them, one pass in place of two (a layer of 16
  // experts, four a token, 100 tokens: 96.4 -> 95.3 us, 2,048: 219.1 -> 217.6); more walk their pairs a second time.
  const bool once = n_pairs <= 8 * threads;
  int kept[8], place[8];
  for (int b0 = tid - lane; b0 < n_pairs; b0 += 8 * threads) {
#pragma unroll
    for (int n = 0; n < 8; ++n)
      kept[n] = b0 + n * threads + lane < n_pairs ? min((unsigned)ids[b0 + n * threads + lane], (unsigned)experts) : experts;
#pragma unroll
    for (int n = 0; n < 8; ++n) {
      if (b0 + n * threads >= n_pairs) break;
      const unsigned same = moe_same(kept[n], bits);
      const int leader = __ffs(same) - 1;
      int at = 0;
      if (kept[n] < experts && lane == leader) at = atomicAdd(&count[kept[n]], __popc(same));
      place[n] = __shfl_sync(0xffffffffu, at, leader) + __popc(same & ((1u << lane) - 1u));
    }
  }
  __syncthreads();
  // the experts' first tiles: the first warp, 32 experts at a time
  if (tid < 32) {
    int tiles = 0;
    for (int e0 = 0; e0 < experts; e0 += 32) {
      const int e = e0 + lane, mine = e < experts ? (count[e] + bm - 1) / bm : 0;
      int upto = mine;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, upto, o);
        if (lane >= o) upto += v;
      }
      if (e < experts) offset[e] = (tiles + upto - mine) * bm;
      tiles += __shfl_sync(0xffffffffu, upto, 31);
    }
    if (lane == 0) n_tiles[0] = tiles;
  }
  __syncthreads();
  // a warp an expert: its tiles' names, and -1 behind its pairs
  for (int e = tid >> 5; e < experts; e += threads >> 5) {
    const int n = count[e], first = offset[e], nt = (n + bm - 1) / bm;
    for (int t = lane; t < nt; t += 32) tile_expert[first / bm + t] = e;
    for (int i = first + n + lane; i < first + nt * bm && i < capacity; i += 32) sorted[i] = -1;
  }
  if (once) {
#pragma unroll
    for (int n = 0; n < 8; ++n)
      if (n * threads + tid < n_pairs && kept[n] < experts) sorted[offset[kept[n]] + place[n]] = n * threads + tid;
    return;
  }
  __syncthreads();
  for (int e = tid; e < experts; e += threads) count[e] = 0;
  __syncthreads();
  for (int b0 = tid - lane; b0 < n_pairs; b0 += 8 * threads) {
    int e[8];
#pragma unroll
    for (int n = 0; n < 8; ++n) e[n] = b0 + n * threads + lane < n_pairs ? min((unsigned)ids[b0 + n * threads + lane], (unsigned)experts) : experts;
#pragma unroll
    for (int n = 0; n < 8; ++n) {
      if (b0 + n * threads >= n_pairs) break;
      const unsigned same = moe_same(e[n], bits);
      const int leader = __ffs(same) - 1;
      const bool real = e[n] < experts;
      int at = 0;
      if (real && lane == leader) at = atomicAdd(&count[e[n]], __popc(same));
      at = __shfl_sync(0xffffffffu, at, leader);
      if (real) sorted[offset[e[n]] + at + __popc(same & ((1u << lane) - 1u))] = b0 + n * threads + lane;
    }
  }
}

// The same by a cluster of eight blocks, for more than 512 pairs of up to ALIGN_EXPERTS experts: what bounds one block there is its SM's
// issue slots (a vote a bit for every 32 pairs: 9,300 cycles of 8,192 pairs, 16 experts) and code that no cache holds yet, so the pairs
// are dealt to eight SMs and each loop stands once.  Every warp has counts of its own, which nobody queues at; a block's sums reach the
// others through their shared memory.  One block / eight, us, warm: 16 experts
// 512 pairs 3.7 / 3.8, 1,024 4.3 / 3.7, 4,096 5.4 / 4.0, 8,192 8.1 / 4.6, 20,000 22.4 / 9.5; 64 experts 8,192 12.2 / 4.9; a layer of 16 experts and
// 2,048 tokens 215.0 -> 212.5.
#define ALIGN_CTAS 8
#define ALIGN_EXPERTS 64
__device__ __forceinline__ int moe_of_block(const int* at, int rank) {
  unsigned there;
  int v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(there) : "r"((unsigned)__cvta_generic_to_shared(at)), "r"(rank));
  asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(there) : "memory");
  return v;
}
__global__ void __launch_bounds__(256)
moe_align_cluster_kernel(const int* __restrict__ ids, int n_pairs, int experts, int* __restrict__ sorted, int capacity,
                         int* __restrict__ tile_expert, int* __restrict__ n_tiles, int bm) {
  // own: a warp's pairs of an expert so far; first those that it has counted, then its pairs' first place
  __shared__ int own[8][ALIGN_EXPERTS], total[ALIGN_EXPERTS], count[ALIGN_EXPERTS], row[ALIGN_EXPERTS], place0[ALIGN_EXPERTS],
      half_tiles;
  pdl_trigger();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, rank = blockIdx.x;
  const int bits = 32 - __clz(experts);             // (numbers up to `experts`, which stands for all that have no tile)
  constexpr int STEP = ALIGN_CTAS * 256, KEPT = 8;
  int* mine = own[warp];
  mine[lane] = 0;
  mine[lane + 32] = 0;
  __syncwarp();
  // the lane's place among the pairs of its expert that its warp has met
  auto take = [&](int e) {
    const unsigned same = moe_same(e, bits);
    const int leader = __ffs(same) - 1;
    int at = 0;
    if (e < experts && lane == leader) {
      at = mine[e];
      mine[e] = at + __popc(same);
    }
    __syncwarp();
    return __shfl_sync(0xffffffffu, at, leader) + __popc(same & ((1u << lane) - 1u));
  };
  auto expert_of = [&](int pair) { return pair < n_pairs ? (int)min((unsigned)ids[pair], (unsigned)experts) : experts; };
  pdl_wait();
  SB_BEHIND_WAIT(ids);
  // up to eight pairs a thread keep their experts and places, more walk their pairs a second time
  const int pair0 = rank * 256 + tid;
  int kept[KEPT], place[KEPT];
#pragma unroll
  for (int n = 0; n < KEPT; ++n) kept[n] = expert_of(pair0 + n * STEP);
#pragma unroll
  for (int n = 0; n < KEPT; ++n)
    if (n * STEP < n_pairs) place[n] = take(kept[n]);
#pragma unroll 1
  for (int p = KEPT * STEP; p < n_pairs; p += STEP) take(expert_of(pair0 + p));
  __syncthreads();
  if (tid < ALIGN_EXPERTS) {
    int sum = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
      const int v = own[w][tid];
      own[w][tid] = sum;
      sum += v;
    }
    total[tid] = sum;
  }
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
  int all = 0, before = 0, upto = 0, tiles = 0;
  if (tid < ALIGN_EXPERTS) {
#pragma unroll
    for (int r = 0; r < ALIGN_CTAS; ++r) {
      const int v = moe_of_block(&total[tid], r);
      all += v;
      before += r < rank ? v : 0;
    }
    count[tid] = all;
    upto = tiles = (all + bm - 1) / bm;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += v;
    }
    if (tid == 31) half_tiles = upto;
  }
  asm volatile("barrier.cluster.arrive.release;" ::: "memory");       // (this block has read what it needs of the others)
  __syncthreads();
  if (tid < ALIGN_EXPERTS) {
    if (tid >= 32) upto += half_tiles;
    const int first = (upto - tiles) * bm;
    row[tid] = first;
    place0[tid] = first + before;
    if (tid == ALIGN_EXPERTS - 1 && rank == 0) n_tiles[0] = upto;
  }
  __syncthreads();
  // a warp an expert: its tiles' names, and -1 behind its pairs
  const int expert = rank * 8 + warp;
  if (expert < experts) {
    const int first = row[expert], n = count[expert], nt = (n + bm - 1) / bm;
    for (int t = lane; t < nt; t += 32) tile_expert[first / bm + t] = expert;
    for (int i = first + n + lane; i < first + nt * bm && i < capacity; i += 32) sorted[i] = -1;
  }
  if (n_pairs <= KEPT * STEP) {
#pragma unroll
    for (int n = 0; n < KEPT; ++n)
      if (kept[n] < experts) sorted[place0[kept[n]] + mine[kept[n]] + place[n]] = pair0 + n * STEP;
  } else {
    // (the warp's counts stand at its pairs' first places and go on from there)
#pragma unroll 1
    for (int p = 0; p < n_pairs; p += STEP) {
      const int e = expert_of(pair0 + p), at = take(e);
      if (e < experts) sorted[place0[e] + at] = pair0 + p;
    }
  }
  asm volatile("barrier.cluster.wait.acquire;" ::: "memory");         // nobody leaves while another block may read its sums
}

// A tile of MOE_BM rows times MOE_BN outputs in float on the CUDA cores: the 32-bit path, and the
// working-type path for widths the tensor-core kernel does not take.  MODE 1: rows gathered from h by
// pair / top, two weight blocks (gate, up) and the gated activation; MODE 2: rows gathered likewise, one
// weight block, squared relu; MODE 0: rows of `a`, one block, results filed by pair.
template <typename T, int MODE>
__global__ void __launch_bounds__(256)
moe_tile_kernel(const T* __restrict__ x, const T* __restrict__ w, T* __restrict__ y, const int* __restrict__ sorted,
                const int* __restrict__ tile_expert, const int* __restrict__ n_tiles, int k_dim, int n_out, int top,
                float limit, const float* __restrict__ in_scale) {
  __shared__ float xs[MOE_BM][MOE_BK + 1];
  constexpr bool UP = MODE != 0;
  constexpr int NW = MODE == 1 ? 2 : 1;
  __shared__ float ws[NW][MOE_BN][MOE_BK + 1];
  __shared__ int src[MOE_BM];
  // (launch_dependents comes at this kernel's end, not its start: it runs in several waves of large blocks,
  // and a successor that starts early would only sit on the SMs its later waves need)
  pdl_wait();
  SB_BEHIND_WAIT(x);
  SB_BEHIND_WAIT(sorted);
  SB_BEHIND_WAIT(tile_expert);
  SB_BEHIND_WAIT(n_tiles);
  SB_BEHIND_WAIT(in_scale);
  const int tile = blockIdx.x;
  if (tile >= n_tiles[0]) return;
  const int e = tile_expert[tile];
  const int n0 = blockIdx.y * MOE_BN;
  const int tid = threadIdx.x;
  if (tid < MOE_BM) src[tid] = sorted[tile * MOE_BM + tid];
  __syncthreads();
  const T* we = w + (size_t)e * NW * n_out * k_dim;
  const int ty = tid >> 4, tx = tid & 15;
  float acc[NW][2][4];
#pragma unroll
  for (int a = 0; a < NW; ++a)
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[a][i][j] = 0.f;
  for (int k0 = 0; k0 < k_dim; k0 += MOE_BK) {
    for (int i = tid; i < MOE_BM * MOE_BK; i += 256) {
      const int m = i / MOE_BK, kk = i % MOE_BK;
      const int pair = src[m];
      float v = 0.f;
      if (pair >= 0 && k0 + kk < k_dim) {
        const size_t row = UP ? (size_t)(pair / top) : (size_t)tile * MOE_BM + m;
        v = to_f<T>(x[row * k_dim + k0 + kk]);
      }
      xs[m][kk] = v;
    }
    for (int i = tid; i < NW * MOE_BN * MOE_BK; i += 256) {
      const int a = i / (MOE_BN * MOE_BK), rem = i % (MOE_BN * MOE_BK);
      const int n = rem / MOE_BK, kk = rem % MOE_BK;
      float v = 0.f;
      if (n0 + n < n_out && k0 + kk < k_dim) v = to_f<T>(we[((size_t)a * n_out + n0 + n) * k_dim + k0 + kk]);
      ws[a][n][kk] = v;
    }
    __syncthreads();
#pragma unroll 8
    for (int kk = 0; kk < MOE_BK; ++kk) {
      const float x0 = xs[ty * 2][kk], x1 = xs[ty * 2 + 1][kk];
#pragma unroll
      for (int a = 0; a < NW; ++a)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float wv = ws[a][tx + 16 * j][kk];
          acc[a][0][j] += x0 * wv;
          acc[a][1][j] += x1 * wv;
        }
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int m = ty * 2 + i;
    const int pair = src[m];
    const float by = UP && in_scale && pair >= 0 ? in_scale[pair] : 1.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int n = n0 + tx + 16 * j;
      if (n >= n_out) continue;
      if (MODE == 1) {
        const float g = rnd<T>(acc[0][i][j] * by), u = rnd<T>(acc[NW - 1][i][j] * by);
        const float a = pair >= 0 ? moe_gate(g, u, limit) : 0.f;
        y[((size_t)tile * MOE_BM + m) * n_out + n] = from_f<T>(a);
      } else if (MODE == 2) {
        const float u = fmaxf(rnd<T>(acc[0][i][j] * by), 0.f);
        y[((size_t)tile * MOE_BM + m) * n_out + n] = from_f<T>(pair >= 0 ? u * u : 0.f);
      } else if (pair >= 0) {
        y[(size_t)pair * n_out + n] = from_f<T>(acc[0][i][j]);
      }
    }
  }
}

// The same on the tensor cores (bfloat16, k a multiple of 16): tiles of 64 rows times 64 outputs, eight
// warps (four groups of 16 rows times two halves of the outputs), wmma 16 x 16 x 16 with float
// accumulators.  Rows (gathered through `sorted`) and weights arrive in k-slices of 64 through a ring of
// three cp.async stages, so that the copies of the next two slices are in flight while one is multiplied.
#define MOE_TC_BM 64
#define MOE_TC_BK 64
__device__ __forceinline__ void moe_cp16(void* dst, const void* src, bool real) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  const int bytes = real ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}

template <int MODE>
__global__ void __launch_bounds__(256)
moe_tile_tc_kernel(const bf16* __restrict__ x, const bf16* __restrict__ w, bf16* __restrict__ y,
                   const int* __restrict__ sorted, const int* __restrict__ tile_expert,
                   const int* __restrict__ n_tiles, int k_dim, int n_out, int top, float limit,
                   const float* __restrict__ in_scale) {
  using namespace nvcuda;
  constexpr bool UP = MODE != 0;
  constexpr int BK = MOE_TC_BK, LD = BK + 8, NW = MODE == 1 ? 2 : 1, STAGES = 3, CLD = MOE_BN + 4;
  constexpr int PIECES = BK / 8, PASS_ROWS = 256 / PIECES, PASSES = MOE_TC_BM / PASS_ROWS;
  extern __shared__ __align__(128) unsigned char moe_smem[];
  bf16* xs = reinterpret_cast<bf16*>(moe_smem);                          // [STAGES][64][LD]
  bf16* ws = xs + STAGES * MOE_TC_BM * LD;                               // [STAGES][NW][64][LD]
  // [NW][64][CLD], in the ring's place once the last slice is multiplied (the ring is the larger of the two)
  float* cs = reinterpret_cast<float*>(moe_smem);
  static_assert((size_t)NW * MOE_TC_BM * CLD * sizeof(float) <= (size_t)STAGES * (1 + NW) * MOE_TC_BM * LD * sizeof(bf16),
                "the staging tile must fit in the ring");
  __shared__ int src[MOE_TC_BM];
  // (launch_dependents comes at this kernel's end, not its start: it runs in several waves of large blocks,
  // and a successor that starts early would only sit on the SMs its later waves need)
  pdl_wait();
  SB_BEHIND_WAIT(x);
  SB_BEHIND_WAIT(sorted);
  SB_BEHIND_WAIT(tile_expert);
  SB_BEHIND_WAIT(n_tiles);
  SB_BEHIND_WAIT(in_scale);
  const int tile = blockIdx.x;
  if (tile >= n_tiles[0]) return;
  const int e = tile_expert[tile];
  const int n0 = blockIdx.y * MOE_BN;
  const int tid = threadIdx.x, warp = tid >> 5;
  if (tid < MOE_TC_BM) src[tid] = sorted[tile * MOE_TC_BM + tid];
  __syncthreads();
  const bf16* we = w + (size_t)e * NW * n_out * k_dim;
  // this thread's 16-byte piece of PASSES rows (lm, lm + PASS_ROWS, ..) of every slice
  const int lm = tid / PIECES, lc = (tid % PIECES) * 8;
  const bf16* x_row[PASSES];
  const bf16* w_row[PASSES];
  bool x_in[PASSES], w_in[PASSES];
#pragma unroll
  for (int p = 0; p < PASSES; ++p) {
    const int r = lm + PASS_ROWS * p;
    const int pair = src[r];
    x_in[p] = pair >= 0;
    x_row[p] = x + (UP ? (size_t)(pair >= 0 ? pair / top : 0) : (size_t)tile * MOE_TC_BM + r) * k_dim;
    w_in[p] = n0 + r < n_out;
    w_row[p] = we + (size_t)(w_in[p] ? n0 + r : 0) * k_dim;
  }
  const int k_tiles = (k_dim + BK - 1) / BK;
  auto load = [&](int kt, int st) {
    const int kk = kt * BK + lc;
    const bool in_k = kk < k_dim;
#pragma unroll
    for (int p = 0; p < PASSES; ++p) {
      const int r = lm + PASS_ROWS * p;
      moe_cp16(xs + ((size_t)st * MOE_TC_BM + r) * LD + lc, x_row[p] + (in_k ? kk : 0), in_k && x_in[p]);
#pragma unroll
      for (int a = 0; a < NW; ++a)
        moe_cp16(ws + (((size_t)st * NW + a) * MOE_BN + r) * LD + lc, w_row[p] + (size_t)a * n_out * k_dim + (in_k ? kk : 0),
                 in_k && w_in[p]);
    }
  };
  const int wm = warp & 3, wn = warp >> 2;
  wmma::fragment<wmma::accumulator, 16, 16, 16, float> acc[NW][2];
#pragma unroll
  for (int a = 0; a < NW; ++a)
#pragma unroll
    for (int j = 0; j < 2; ++j) wmma::fill_fragment(acc[a][j], 0.f);
#pragma unroll
  for (int st = 0; st < STAGES - 1; ++st) {
    if (st < k_tiles) load(st, st);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  for (int kt = 0; kt < k_tiles; ++kt) {
    asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
    __syncthreads();
    const int nk = kt + STAGES - 1;
    if (nk < k_tiles) load(nk, nk % STAGES);
    asm volatile("cp.async.commit_group;" ::: "memory");
    const int st = kt % STAGES;
#pragma unroll
    for (int kk = 0; kk < BK; kk += 16) {
      wmma::fragment<wmma::matrix_a, 16, 16, 16, bf16, wmma::row_major> fa;
      wmma::load_matrix_sync(fa, xs + ((size_t)st * MOE_TC_BM + wm * 16) * LD + kk, LD);
#pragma unroll
      for (int a = 0; a < NW; ++a)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          wmma::fragment<wmma::matrix_b, 16, 16, 16, bf16, wmma::col_major> fb;
          wmma::load_matrix_sync(fb, ws + (((size_t)st * NW + a) * MOE_BN + wn * 32 + j * 16) * LD + kk, LD);
          wmma::mma_sync(acc[a][j], fa, fb, acc[a][j]);
        }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  pdl_trigger();
  __syncthreads();      // every warp is done with the ring before the staging tile takes its place
#pragma unroll
  for (int a = 0; a < NW; ++a)
#pragma unroll
    for (int j = 0; j < 2; ++j)
      wmma::store_matrix_sync(cs + ((size_t)a * MOE_TC_BM + wm * 16) * CLD + wn * 32 + j * 16, acc[a][j], CLD,
                              wmma::mem_row_major);
  __syncthreads();
  for (int i = tid; i < MOE_TC_BM * MOE_BN; i += 256) {
    const int m = i / MOE_BN, nn = i % MOE_BN;
    const int n = n0 + nn;
    const int row_pair = src[m];
    if (n >= n_out) continue;
    const float by = UP && in_scale && row_pair >= 0 ? in_scale[row_pair] : 1.f;
    if (MODE == 1) {
      const float g = rnd<bf16>(cs[(size_t)m * CLD + nn] * by), u = rnd<bf16>(cs[((size_t)(NW - 1) * MOE_TC_BM + m) * CLD + nn] * by);
      const float a = row_pair >= 0 ? moe_gate(g, u, limit) : 0.f;
      y[((size_t)tile * MOE_TC_BM + m) * n_out + n] = from_f<bf16>(a);
    } else if (MODE == 2) {
      const float u = fmaxf(rnd<bf16>(cs[(size_t)m * CLD + nn] * by), 0.f);
      y[((size_t)tile * MOE_TC_BM + m) * n_out + n] = from_f<bf16>(row_pair >= 0 ? u * u : 0.f);
    } else if (row_pair >= 0) {
      y[(size_t)row_pair * n_out + n] = from_f<bf16>(cs[(size_t)m * CLD + nn]);
    }
  }
}

// The same for steps with many rows an expert (prompts): tiles of 128 rows times 128 outputs, eight warps
// (two groups of 64 rows times four groups of 32 outputs), mma.sync m16n8k16 with operands by ldmatrix.
// A warp's k-step of 16 is four A loads, two B loads and sixteen products (the 64 x 64 wmma tile above has
// three loads for two products and is bound by them).  Rows and weights arrive in k-slices through a ring of
// three cp.async stages; rows are padded by 16 bytes, so the eight 16-byte rows of an ldmatrix fall into
// eight different bank groups.  The epilogue goes from the accumulators to global memory in pairs.
#define MOE_BIG 128
__device__ __forceinline__ void moe_ldm4(const void* p, uint32_t* r) {
  const uint32_t addr = (uint32_t)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void moe_mma(float* c, const uint32_t* a, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

template <int MODE>
__global__ void __launch_bounds__(256)
moe_tile_big_kernel(const bf16* __restrict__ x, const bf16* __restrict__ w, bf16* __restrict__ y,
                    const int* __restrict__ sorted, const int* __restrict__ tile_expert,
                    const int* __restrict__ n_tiles, int k_dim, int n_out, int top, float limit,
                    const float* __restrict__ in_scale) {
  constexpr bool UP = MODE != 0;
  // k-slices of 64 (rows of 144 bytes) with one weight block, of 32 (rows of 80 bytes) with two: three stages
  // of either leave room for two blocks an SM
  constexpr int NW = MODE == 1 ? 2 : 1, BK = NW == 1 ? 64 : 32, LD = BK + 8, STAGES = 3;
  constexpr int PIECES = BK / 8, PASS_ROWS = 256 / PIECES, PASSES = MOE_BIG / PASS_ROWS;
  extern __shared__ __align__(128) unsigned char moe_smem[];
  bf16* xs = reinterpret_cast<bf16*>(moe_smem);                          // [STAGES][128][LD]
  bf16* ws = xs + STAGES * MOE_BIG * LD;                                 // [STAGES][NW][128][LD]
  __shared__ int src[MOE_BIG];
  // (launch_dependents comes at this kernel's end, as in the smaller tile: several waves of large blocks)
  pdl_wait();
  SB_BEHIND_WAIT(x);
  SB_BEHIND_WAIT(sorted);
  SB_BEHIND_WAIT(tile_expert);
  SB_BEHIND_WAIT(n_tiles);
  SB_BEHIND_WAIT(in_scale);
  const int tile = blockIdx.x;
  if (tile >= n_tiles[0]) return;
  const int e = tile_expert[tile];
  const int n0 = blockIdx.y * MOE_BIG;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid < MOE_BIG) src[tid] = sorted[tile * MOE_BIG + tid];
  __syncthreads();
  const bf16* we = w + (size_t)e * NW * n_out * k_dim;
  // this thread copies one 16-byte piece of PASSES rows (lm, lm + PASS_ROWS, ..) of every slice of rows and of weights
  const int lm = tid / PIECES, lc = (tid % PIECES) * 8;
  const bf16* x_row[PASSES];
  const bf16* w_row[PASSES];
  bool x_in[PASSES], w_in[PASSES];
#pragma unroll
  for (int h = 0; h < PASSES; ++h) {
    const int r = lm + PASS_ROWS * h;
    const int pair = src[r];
    x_in[h] = pair >= 0;
    x_row[h] = x + (UP ? (size_t)(pair >= 0 ? pair / top : 0) : (size_t)tile * MOE_BIG + r) * k_dim;
    w_in[h] = n0 + r < n_out;
    w_row[h] = we + (size_t)(w_in[h] ? n0 + r : 0) * k_dim;
  }
  const int k_tiles = (k_dim + BK - 1) / BK;
  auto load = [&](int kt, int st) {
    const int kk = kt * BK + lc;
    const bool in_k = kk < k_dim;
    const int ko = in_k ? kk : 0;
#pragma unroll
    for (int h = 0; h < PASSES; ++h) {
      const int r = lm + PASS_ROWS * h;
      moe_cp16(xs + ((size_t)st * MOE_BIG + r) * LD + lc, x_row[h] + ko, in_k && x_in[h]);
#pragma unroll
      for (int a = 0; a < NW; ++a)
        moe_cp16(ws + (((size_t)st * NW + a) * MOE_BIG + r) * LD + lc, w_row[h] + (size_t)a * n_out * k_dim + ko,
                 in_k && w_in[h]);
    }
  };
  const int wm = warp & 1, wn = warp >> 1;               // rows 64 wm .., outputs 32 wn ..
  float acc[NW][4][4][4];
#pragma unroll
  for (int a = 0; a < NW; ++a)
#pragma unroll
    for (int mb = 0; mb < 4; ++mb)
#pragma unroll
      for (int nb = 0; nb < 4; ++nb)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[a][mb][nb][c] = 0.f;
#pragma unroll
  for (int st = 0; st < STAGES - 1; ++st) {
    if (st < k_tiles) load(st, st);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  const int a_row = wm * 64 + (lane & 15), a_col = (lane >> 4) * 8;
  const int b_row = wn * 32 + (lane & 7) + (lane >> 4) * 8, b_col = ((lane >> 3) & 1) * 8;
  for (int kt = 0; kt < k_tiles; ++kt) {
    asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
    __syncthreads();
    const int nk = kt + STAGES - 1;
    if (nk < k_tiles) load(nk, nk % STAGES);
    asm volatile("cp.async.commit_group;" ::: "memory");
    const int st = kt % STAGES;
    const bf16* xt = xs + (size_t)st * MOE_BIG * LD;
#pragma unroll
    for (int kk = 0; kk < BK; kk += 16) {
      uint32_t af[4][4];
#pragma unroll
      for (int mb = 0; mb < 4; ++mb) moe_ldm4(xt + (size_t)(a_row + mb * 16) * LD + kk + a_col, af[mb]);
#pragma unroll
      for (int a = 0; a < NW; ++a) {
        const bf16* wt = ws + ((size_t)st * NW + a) * MOE_BIG * LD;
#pragma unroll
        for (int nb2 = 0; nb2 < 2; ++nb2) {
          uint32_t bfr[4];
          moe_ldm4(wt + (size_t)(b_row + nb2 * 16) * LD + kk + b_col, bfr);
#pragma unroll
          for (int mb = 0; mb < 4; ++mb) {
            moe_mma(acc[a][mb][nb2 * 2], af[mb], bfr[0], bfr[1]);
            moe_mma(acc[a][mb][nb2 * 2 + 1], af[mb], bfr[2], bfr[3]);
          }
        }
      }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  pdl_trigger();
  // accumulator (mb, nb, c): row 64 wm + 16 mb + lane / 4 + 8 (c / 2), output 32 wn + 8 nb + 2 (lane % 4) + c % 2;
  // n_out is even here (a multiple of 16), so a pair of outputs is inside or outside together
#pragma unroll
  for (int mb = 0; mb < 4; ++mb)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int m = wm * 64 + mb * 16 + (lane >> 2) + 8 * h;
      const int row_pair = src[m];
      if (MODE == 0 && row_pair < 0) continue;
      const float by = UP && in_scale && row_pair >= 0 ? in_scale[row_pair] : 1.f;
      bf16* y_row = y + (MODE == 0 ? (size_t)row_pair : (size_t)tile * MOE_BIG + m) * n_out;
#pragma unroll
      for (int nb = 0; nb < 4; ++nb) {
        const int n = n0 + wn * 32 + nb * 8 + (lane & 3) * 2;
        if (n >= n_out) continue;
        float r0, r1;
        if (MODE == 1) {
          float g0 = rnd<bf16>(acc[0][mb][nb][2 * h] * by), g1 = rnd<bf16>(acc[0][mb][nb][2 * h + 1] * by);
          float u0 = rnd<bf16>(acc[NW - 1][mb][nb][2 * h] * by), u1 = rnd<bf16>(acc[NW - 1][mb][nb][2 * h + 1] * by);
          r0 = row_pair >= 0 ? moe_gate(g0, u0, limit) : 0.f;
          r1 = row_pair >= 0 ? moe_gate(g1, u1, limit) : 0.f;
        } else if (MODE == 2) {
          const float u0 = fmaxf(rnd<bf16>(acc[0][mb][nb][2 * h] * by), 0.f);
          const float u1 = fmaxf(rnd<bf16>(acc[0][mb][nb][2 * h + 1] * by), 0.f);
          r0 = row_pair >= 0 ? u0 * u0 : 0.f;
          r1 = row_pair >= 0 ? u1 * u1 : 0.f;
        } else {
          r0 = acc[0][mb][nb][2 * h];
          r1 = acc[0][mb][nb][2 * h + 1];
        }
        *reinterpret_cast<__nv_bfloat162*>(y_row + n) = __floats2bfloat162_rn(r0, r1);
      }
    }
}

// For steps with a handful of rows an expert (single tokens): a tile is up to MOE_FEW rows of one expert, the columns of an
// m16n8k16 product whose rows are 16 weight rows (16 gate and the matching 16 up rows).  Operands go from global memory to
// registers in 16-byte pieces: lane 4 g + x holds the pieces x, x + 4, .. of weight rows g and g + 8 and of the tile's row g, so
// that every product sees its k entries in one order.  The step is bound by the weights' bytes, which are read once a
// tile, so what counts is that loads never stop: a warp keeps FLY steps of 32 entries in flight and asks for the next one as
// soon as it has used one, and a block has as many warps (1, 2, 4 or 8, which share the k range; their sums meet in shared memory) as
// bring ten and more to every SM: 1,480 to 2,958 warps over the grid from 185 to 1,479 blocks, eight a block and fewer warps in all below, one a
// block above.  (16 fit an SM.  An end at those 16, one round for all, is slower where it bites: 1,296 blocks, gated, 45.3 us a layer -> 49.4, squared
// relu 35.3 -> 37.1; four always 43.3 -> 46.4 and 35.0 -> 37.0 at 1,152.)  The number of warps, and with it the order in which the parts of
// a sum over k join, follows from the step's tiles: a row's last bits depend on how many other rows a step has.
// The weight rows of a tile run along the grid, so that the warps of an SM share the tile's rows in the first cache, in which the
// weights take no place: from memory, where a model's layers are, 16 experts of 2,048 x 2,048, 8 tokens 96 -> 88 us and of 1,024 x 1,024, 4 tokens
// 38.9 -> 36.9; a layer called in a row whose weights stay in L2 loses by it (the latter 25.0 -> 29.7).
// A captured layer of 16 experts of 2,048 x 2,048 at 8 tokens, four each, with blocks of four warps (a round and a half of them) and loads that
// stop between steps 82, now 74 (363 MB are 55); with the caches emptied in front 98 -> 88, one token 57 -> 41, 16 tokens of 1,536 x 1,536 78 -> 66,
// squared relu 70 -> 49.
// The second product reads the tiles' experts and its first weights ahead of its wait.  It may because it stands directly behind the first
// one (sb_moe_few launches both), which lets it start only behind its own wait, when the kernel that made the tiles has completed.
#define MOE_FEW 8
#define MOE_FEW_WARPS 10         // the fewest warps an SM that a grid should bring
#define MOE_FEW_REGS 128         // (16 warps an SM; 6 and 3 steps in flight fill them.  144 registers and 8 and 4: 77.5 -> 90.0 us, 96 and 4 and 2: 88.0)
__device__ __forceinline__ void moe_unpack8(const uint4& v, float* f) {
  f[0] = __uint_as_float(v.x << 16); f[1] = __uint_as_float(v.x & 0xffff0000u);
  f[2] = __uint_as_float(v.y << 16); f[3] = __uint_as_float(v.y & 0xffff0000u);
  f[4] = __uint_as_float(v.z << 16); f[5] = __uint_as_float(v.z & 0xffff0000u);
  f[6] = __uint_as_float(v.w << 16); f[7] = __uint_as_float(v.w & 0xffff0000u);
}


__device__ __forceinline__ uint4 moe_stream16(const uint4* p) {      // (volatile: loads stay where they are asked for)
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}

template <int MODE>
__global__ void __maxnreg__(MOE_FEW_REGS)
moe_few_kernel(const bf16* __restrict__ x, const bf16* __restrict__ w, bf16* __restrict__ y,
               const int* __restrict__ sorted, const int* __restrict__ tile_expert, const int* __restrict__ n_tiles,
               int max_tiles, int k_dim, int n_out, int top, float limit, const float* __restrict__ in_scale) {
  constexpr bool UP = MODE != 0;
  constexpr int NW = MODE == 1 ? 2 : 1, FLY = MODE == 1 ? 3 : 6;
  extern __shared__ float few_part[];                   // [warps][NW * 4][32], with more than one warp
  const int warps = blockDim.x >> 5;
  if (UP) {
    pdl_wait();
    pdl_trigger();
  }
  SB_BEHIND_WAIT(sorted);
  SB_BEHIND_WAIT(tile_expert);
  SB_BEHIND_WAIT(n_tiles);
  const int tile = blockIdx.z * gridDim.y + blockIdx.y;
  if (tile >= max_tiles) {                               // (more tiles than a grid's dimension counts to)
    if (!UP) pdl_wait();
    return;
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, q = lane & 3;
  // (three loads at once; a tile that is not there has garbage in its places and leaves)
  const int expert = tile_expert[tile], own = sorted[tile * MOE_FEW + g];
  if (tile >= n_tiles[0]) {
    if (!UP) pdl_wait();
    return;
  }
  const bf16* we = w + (size_t)expert * NW * n_out * k_dim;
  const int n0 = blockIdx.x * 16;
  // this lane's row of the tile (none: the loads are of the tile's first row, the products are not stored) and its weight rows
  const uint4* wr[NW][2];
#pragma unroll
  for (int a = 0; a < NW; ++a)
#pragma unroll
    for (int r = 0; r < 2; ++r)
      wr[a][r] = reinterpret_cast<const uint4*>(we + ((size_t)a * n_out + min(n0 + g + 8 * r, n_out - 1)) * k_dim) + q;
  const int pieces = k_dim / 8 - q;                     // (pieces from this lane's first on)
  const int steps = (k_dim / 8 + 3) / 4;
  uint4 wv[FLY][NW][2], xv[FLY];
  auto load_w = [&](int i, int s) {
    const bool in = 4 * s < pieces;
#pragma unroll
    for (int a = 0; a < NW; ++a)
#pragma unroll
      for (int r = 0; r < 2; ++r) wv[i][a][r] = in ? moe_stream16(wr[a][r] + 4 * s) : make_uint4(0u, 0u, 0u, 0u);
  };
#pragma unroll
  for (int i = 0; i < FLY; ++i) load_w(i, warp + i * warps);
  if (!UP) {
    pdl_wait();
    pdl_trigger();
  }
  SB_BEHIND_WAIT(x);
  SB_BEHIND_WAIT(in_scale);
  const uint4* xr = reinterpret_cast<const uint4*>(x + (UP ? (size_t)(own >= 0 ? own / top : 0) : (size_t)tile * MOE_FEW + (own >= 0 ? g : 0)) * k_dim) + q;
  auto load_x = [&](int i, int s) { xv[i] = 4 * s < pieces ? xr[4 * s] : make_uint4(0u, 0u, 0u, 0u); };
#pragma unroll
  for (int i = 0; i < FLY; ++i) load_x(i, warp + i * warps);
  float acc[NW][4];
#pragma unroll
  for (int a = 0; a < NW; ++a) acc[a][0] = acc[a][1] = acc[a][2] = acc[a][3] = 0.f;
  for (int s0 = warp; s0 < steps; s0 += FLY * warps) {
#pragma unroll
    for (int i = 0; i < FLY; ++i) {
#pragma unroll
      for (int a = 0; a < NW; ++a) {
        const uint4 u = wv[i][a][0], v = wv[i][a][1];
        const uint32_t lo[4] = {u.x, v.x, u.y, v.y}, hi[4] = {u.z, v.z, u.w, v.w};
        // (a step's own sum, joined by rounded additions: the tensor cores cut what they add to an accumulator)
        float step[4] = {0.f, 0.f, 0.f, 0.f};
        moe_mma(step, lo, xv[i].x, xv[i].y);
        moe_mma(step, hi, xv[i].z, xv[i].w);
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[a][c] += step[c];
      }
      const int next = s0 + (i + FLY) * warps;
      load_w(i, next);
      load_x(i, next);
    }
  }
  if (warps > 1) {
#pragma unroll
    for (int a = 0; a < NW; ++a)
#pragma unroll
      for (int c = 0; c < 4; ++c) few_part[(warp * NW * 4 + a * 4 + c) * 32 + lane] = acc[a][c];
    __syncthreads();
  }
  // accumulator c of a lane: weight row g + 8 (c / 2), the tile's row 2 q + c % 2; warp c finishes it
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    if (warps > 1 && c % warps != warp) continue;
    float v[NW];
#pragma unroll
    for (int a = 0; a < NW; ++a) {
      v[a] = acc[a][c];
      if (warps > 1) {
        v[a] = few_part[(a * 4 + c) * 32 + lane];
        for (int p = 1; p < warps; ++p) v[a] += few_part[(p * NW * 4 + a * 4 + c) * 32 + lane];
      }
    }
    const int n = n0 + g + 8 * (c >> 1), r = 2 * q + (c & 1);
    const int pair = sorted[tile * MOE_FEW + r];
    if (n >= n_out || pair < 0) continue;
    const float by = UP && in_scale ? in_scale[pair] : 1.f;
    if (MODE == 1) {
      y[((size_t)tile * MOE_FEW + r) * n_out + n] = from_f<bf16>(moe_gate(rnd<bf16>(v[0] * by), rnd<bf16>(v[NW - 1] * by), limit));
    } else if (MODE == 2) {
      const float u = fmaxf(rnd<bf16>(v[0] * by), 0.f);
      y[((size_t)tile * MOE_FEW + r) * n_out + n] = from_f<bf16>(u * u);
    } else {
      y[(size_t)pair * n_out + n] = from_f<bf16>(v[0]);
    }
  }
}

// The rows of h in the order of `sorted` (a pair's row is h[pair / top]; zeros where a tile is padded), for a
// product that wants its rows in place: a block MOE_GATHER rows, whose 16-byte pieces are in flight together.  Rows behind the last tile stay unwritten.
// in_scale (float [pairs] or null) multiplies the rows.
#define MOE_GATHER 4
__global__ void __launch_bounds__(256) moe_gather_kernel(const bf16* __restrict__ h, const int* __restrict__ sorted,
                                  const int* __restrict__ n_tiles, int tile_rows, int top, bf16* __restrict__ out,
                                  int width, const float* __restrict__ in_scale) {
  pdl_trigger();
  pdl_wait();
  SB_BEHIND_WAIT(h);
  SB_BEHIND_WAIT(sorted);
  SB_BEHIND_WAIT(n_tiles);
  SB_BEHIND_WAIT(in_scale);
  const int rows = n_tiles[0] * tile_rows, row0 = blockIdx.x * MOE_GATHER;
  if (row0 >= rows) return;
  int pair[MOE_GATHER];
#pragma unroll
  for (int r = 0; r < MOE_GATHER; ++r) pair[r] = row0 + r < rows ? sorted[row0 + r] : -1;
  for (int c = threadIdx.x; c < width / 8; c += blockDim.x) {
    uint4 v[MOE_GATHER];
#pragma unroll
    for (int r = 0; r < MOE_GATHER; ++r)
      v[r] = pair[r] >= 0 ? reinterpret_cast<const uint4*>(h + (size_t)(pair[r] / top) * width)[c] : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
    for (int r = 0; r < MOE_GATHER; ++r) {
      if (in_scale && pair[r] >= 0) {
        const float by = in_scale[pair[r]];
        float f[8];
        moe_unpack8(v[r], f);
        __nv_bfloat162* e = reinterpret_cast<__nv_bfloat162*>(&v[r]);
#pragma unroll
        for (int i = 0; i < 4; ++i) e[i] = __floats2bfloat162_rn(f[2 * i] * by, f[2 * i + 1] * by);
      }
      if (row0 + r < rows) reinterpret_cast<uint4*>(out + (size_t)(row0 + r) * width)[c] = v[r];
    }
  }
}

// weights null: the choices are summed as they are.  ids / h (null: every choice is a real expert): a choice from `experts` on stands for the token's own row h[t].
// shared / shared_gate (null: none): shared_gate[t] * shared[t] is added.
template <typename T>
__global__ void moe_combine_kernel(const T* __restrict__ down, const float* __restrict__ weights, T* __restrict__ out,
                                   int width, int top, const int* __restrict__ ids, int experts, const T* __restrict__ h,
                                   const T* __restrict__ shared, const float* __restrict__ shared_gate) {
  pdl_trigger();
  pdl_wait();
  SB_BEHIND_WAIT(down);
  SB_BEHIND_WAIT(weights);
  SB_BEHIND_WAIT(ids);
  SB_BEHIND_WAIT(h);
  SB_BEHIND_WAIT(shared);
  SB_BEHIND_WAIT(shared_gate);
  const int row = blockIdx.x;
  const float sg = shared ? shared_gate[row] : 0.f;
  for (int c = threadIdx.x; c < width; c += blockDim.x) {
    float a = 0.f;
    for (int j = 0; j < top; ++j) {
      const bool own = ids && ids[(size_t)row * top + j] >= experts;
      a += (weights ? weights[(size_t)row * top + j] : 1.f) *
           to_f<T>(own ? h[(size_t)row * width + c] : down[((size_t)row * top + j) * width + c]);
    }
    if (shared) a += sg * to_f<T>(shared[(size_t)row * width + c]);
    out[(size_t)row * width + c] = from_f<T>(a);
  }
}

// The same for bfloat16 rows of 16-byte pieces: a thread a piece of a token's row, all the choices' loads in flight (a block a
// token and two bytes a load took 16 us for 8 rows of 2,048 and 31 for 2,048, now 3 and 7).
template <bool OWN>
__global__ void __launch_bounds__(128)
moe_combine_vec_kernel(const bf16* __restrict__ down, const float* __restrict__ weights, bf16* __restrict__ out, int width, int top,
                       const int* __restrict__ ids, int experts, const bf16* __restrict__ h, const bf16* __restrict__ shared,
                       const float* __restrict__ shared_gate) {
  pdl_trigger();
  pdl_wait();
  SB_BEHIND_WAIT(down);
  SB_BEHIND_WAIT(weights);
  SB_BEHIND_WAIT(ids);
  SB_BEHIND_WAIT(h);
  SB_BEHIND_WAIT(shared);
  SB_BEHIND_WAIT(shared_gate);
  const size_t row = blockIdx.x;
  const int c = (blockIdx.y * 128 + threadIdx.x) * 8;
  if (c >= width) return;
  float a[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  auto piece = [&](int j, float& by) {
    const size_t at = row * top + j;
    by = weights ? weights[at] : 1.f;
    return *reinterpret_cast<const uint4*>(OWN && ids[at] >= experts ? h + row * width + c : down + at * width + c);
  };
  auto add = [&](const uint4& v, float by) {
    float f[8];
    moe_unpack8(v, f);
#pragma unroll
    for (int i = 0; i < 8; ++i) a[i] += by * f[i];
  };
  int j = 0;
  for (; j + 4 <= top; j += 4) {
    uint4 v[4];
    float by[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = piece(j + i, by[i]);
#pragma unroll
    for (int i = 0; i < 4; ++i) add(v[i], by[i]);
  }
  for (; j < top; ++j) {
    float by;
    const uint4 v = piece(j, by);
    add(v, by);
  }
  if (shared) {
    const float sg = shared_gate[row];
    float f[8];
    moe_unpack8(*reinterpret_cast<const uint4*>(shared + row * width + c), f);
#pragma unroll
    for (int i = 0; i < 8; ++i) a[i] += sg * f[i];
  }
  uint4 o;
  __nv_bfloat162* e = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
  for (int i = 0; i < 4; ++i) e[i] = __floats2bfloat162_rn(a[2 * i], a[2 * i + 1]);
  *reinterpret_cast<uint4*>(out + row * width + c) = o;
}

// up 1: x = h [n_tokens, k_dim], w = [experts, 2 * n_out, k_dim] (gate rows, then up rows), y =
// [capacity, n_out] in the order of `sorted`, the clamped gated activation.  up 2: the same with w =
// [experts, n_out, k_dim] and the squared relu.  up 0: x = that y [capacity, k_dim], w = [experts,
// n_out, k_dim], y = [n_pairs, n_out] by pair.  in_scale (up passes): float [n_pairs] that multiplies the products ahead
// of the activation, or null.
// (tiles of MOE_FEW rows: sb_moe_few)
template <int MODE>
static int moe_tiles_mode(int dtype, int tile_rows, const void* x, const void* w, void* y, const int* sorted,
                          const int* tile_expert, const int* n_tiles, int max_tiles, int k_dim, int n_out, int top,
                          float limit, const float* in_scale, cudaStream_t s) {
  if (tile_rows == MOE_BIG) {
    if (dtype != 1 || k_dim % 16 || n_out % 2 || ((uintptr_t)x % 16) || ((uintptr_t)w % 16) || ((uintptr_t)y % 4)) return -2;
    constexpr int NW = MODE == 1 ? 2 : 1, LD = (NW == 1 ? 64 : 32) + 8;
    const size_t smem = (size_t)3 * (1 + NW) * MOE_BIG * LD * sizeof(bf16);
    cudaFuncSetAttribute(moe_tile_big_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    return launch_dependent(moe_tile_big_kernel<MODE>, dim3(max_tiles, (n_out + MOE_BIG - 1) / MOE_BIG), dim3(256), smem, s,
                            (const bf16*)x, (const bf16*)w, (bf16*)y, sorted, tile_expert, n_tiles, k_dim, n_out, top, limit,
                            in_scale);
  }
  const dim3 grid(max_tiles, (n_out + MOE_BN - 1) / MOE_BN);
  if (tile_rows == MOE_TC_BM) {
    if (dtype != 1 || k_dim % 16 || ((uintptr_t)x % 16) || ((uintptr_t)w % 16)) return -2;
    constexpr int NW = MODE == 1 ? 2 : 1;
    const size_t smem = (size_t)3 * (1 + NW) * 64 * (MOE_TC_BK + 8) * sizeof(bf16);
    cudaFuncSetAttribute(moe_tile_tc_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    return launch_dependent(moe_tile_tc_kernel<MODE>, grid, dim3(256), smem, s, (const bf16*)x, (const bf16*)w,
                            (bf16*)y, sorted, tile_expert, n_tiles, k_dim, n_out, top, limit,
                            in_scale);
  }
  if (tile_rows != MOE_BM) return -2;
  if (dtype == 0)
    return launch_dependent(moe_tile_kernel<float, MODE>, grid, dim3(256), 0, s, (const float*)x, (const float*)w,
                            (float*)y, sorted, tile_expert, n_tiles, k_dim, n_out, top, limit,
                            in_scale);
  return launch_dependent(moe_tile_kernel<bf16, MODE>, grid, dim3(256), 0, s, (const bf16*)x, (const bf16*)w,
                          (bf16*)y, sorted, tile_expert, n_tiles, k_dim, n_out, top, limit,
                            in_scale);
}

// A product of the few-row kernel, bfloat16, k_dim a multiple of 8.
template <int MODE>
static int moe_few(const void* x, const void* w, void* y, const int* sorted, const int* tile_expert, const int* n_tiles, int max_tiles,
                   int k_dim, int n_out, int top, float limit, const float* in_scale, cudaStream_t s) {
  // warps a block: the fewest that bring MOE_FEW_WARPS to every SM, each with two steps and more
  const long long items = (long long)max_tiles * ((n_out + 15) / 16);
  int warps = 1;
  while (warps < 8 && items * warps < 148 * MOE_FEW_WARPS && k_dim >= 32 * 4 * warps) warps *= 2;
  const size_t smem = warps > 1 ? (size_t)warps * (MODE == 1 ? 8 : 4) * 32 * sizeof(float) : 0;
  const int layers = (max_tiles + 65534) / 65535;
  return launch_dependent(moe_few_kernel<MODE>, dim3((n_out + 15) / 16, (max_tiles + layers - 1) / layers, layers), dim3(32 * warps), smem, s,
                          (const bf16*)x, (const bf16*)w, (bf16*)y, sorted, tile_expert, n_tiles, max_tiles, k_dim, n_out, top, limit, in_scale);
}

extern "C" {

// Rows of a tile for these operands: 64 when both products run on the tensor-core tiles (bfloat16, width and
// inner size multiples of 16), else 32.
int sb_moe_tile_rows(int dtype, int width, int inner) {
  return dtype == 1 && width % 16 == 0 && inner % 16 == 0 ? MOE_TC_BM : MOE_BM;
}
// The same for a step of `n_pairs` (row, expert) pairs over `experts` experts, where the caller does not take the grouped tcgen05
// products (more than six rows an expert on average, moe_group_rows in ops.py; it leaves gated experts of odd inner sizes here):
// 8 up to six rows an expert (the few-row kernel), 128 from 128 (the large tiles pay for their padding from there on), 256 from 256 (the grouped prompt product); else as above.
int sb_moe_tile_rows_for(int dtype, int width, int inner, long long n_pairs, int experts) {
  const int rows = sb_moe_tile_rows(dtype, width, inner);
  if (rows != MOE_TC_BM) return rows;
  // 8: the few-row kernel, up to six rows an expert on average (single tokens; beyond, many experts take two tiles of 8, which
  // read the weights twice)
  if (n_pairs <= 6ll * experts) return MOE_FEW;
  // 256: the grouped prompt product (its row tiles), from 256 rows an expert on average
  if (n_pairs >= 256ll * experts) return 256;
  return n_pairs >= (long long)MOE_BIG * experts ? MOE_BIG : rows;
}

// h [.., width] bfloat16 with width a multiple of 8, 16-byte aligned; out [capacity, width].
int sb_moe_gather(const void* h, const int* sorted, const int* n_tiles, int tile_rows, int top, void* out, int capacity,
                  int width, const float* in_scale, cudaStream_t s) {
  if (capacity == 0) return 0;
  if (width % 8 || ((uintptr_t)h % 16) || ((uintptr_t)out % 16) || top < 1) return -2;
  return launch_dependent(moe_gather_kernel, dim3((capacity + MOE_GATHER - 1) / MOE_GATHER), dim3(width / 8 >= 256 ? 256 : 128), 0, s, (const bf16*)h,
                          sorted, n_tiles, tile_rows, top, (bf16*)out, width, in_scale);
}
int sb_moe_max_experts() { return MOE_MAX_EXPERTS; }
int sb_moe_max_top() { return MOE_MAX_TOP; }

// From how many tokens on a block of the router takes sixteen of them (moe_route_many_kernel).
int sb_moe_route_many_from(int experts) {
  return experts > 16 ? 8 * 148 + 1 : 4 * 148;
}

// h: [n_tokens, width]; w: float [experts, width]; b: float [experts] or null; ids: int [n_tokens, top];
// weights: float [n_tokens, top].
// scoring 0: softmax over the chosen logits; 1: sigmoid scores divided by their sum, times weight_scale; 3: plain
// sigmoid scores times weight_scale.
int sb_moe_route(int dtype, const void* h, const float* w, const float* b, int* ids, float* weights, int n_tokens,
                 int width, int experts, int top, int scoring, float weight_scale, cudaStream_t s) {
  if (n_tokens == 0) return 0;
  if (experts < 1 || experts > MOE_MAX_EXPERTS || top < 1 || top > MOE_MAX_TOP || top > experts) return -2;
  if (scoring != 0 && scoring != 1 && scoring != 3) return -2;
  if (dtype == 1 && n_tokens >= sb_moe_route_many_from(experts) && experts <= ROUTE_EXPERTS && width % 8 == 0 && !(((uintptr_t)h | (uintptr_t)w) % 16)) {
    const int groups = experts > 8 ? 2 : 1;
    const int smem = ROUTE_STAGES * (groups * 8 * ROUTE_K * 4 + ROUTE_TOKENS * ROUTE_K * 2);
    const auto kernel = groups == 2 ? moe_route_many_kernel<2> : moe_route_many_kernel<1>;
    // (a device's own setting)
    static bool configured[64][2];
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 64 || !configured[dev][groups - 1]) {
      const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
      if (e != cudaSuccess) return (int)e;
      if (dev < 64) configured[dev][groups - 1] = true;
    }
    return launch_dependent(kernel, dim3((n_tokens + ROUTE_TOKENS - 1) / ROUTE_TOKENS), dim3(256), smem, s, (const bf16*)h, w, b, ids, weights,
                            n_tokens, width, experts, top, scoring, weight_scale);
  }
  // a step of few rows leaves most SMs idle: a token a block and a warp an expert (up to 16) shorten the chain; from 4 tokens
  // an SM on, 4 tokens a block read the router once for all of them (what moe_route_many_kernel does not take)
  const bool many = n_tokens >= 4 * 148 && experts <= 512;
  const int threads = many ? (experts > 16 ? 256 : 128) : experts >= 16 ? 512 : experts > 4 ? 256 : 128;
  const int blocks = many ? (n_tokens + 3) / 4 : n_tokens;
  const size_t smem = (many ? MOE_STAGE_BYTES : 0) + (size_t)(many ? 4 : 1) * experts * sizeof(float);      // (under 48 KB)
#define MOE_ROUTE(T, TOK)                                                                                                  \
  return launch_dependent(moe_route_kernel<T, TOK>, dim3(blocks), dim3(threads), smem, s, (const T*)h, w, b, ids, weights, \
                          n_tokens, width, experts, top, scoring, weight_scale)
  if (dtype == 0) { if (many) MOE_ROUTE(float, 4); MOE_ROUTE(float, 1); }
  if (many) MOE_ROUTE(bf16, 4);
  MOE_ROUTE(bf16, 1);
#undef MOE_ROUTE
}

int sb_moe_align(const int* ids, int n_pairs, int experts, int* sorted, int capacity, int* tile_expert, int* n_tiles,
                 int tile_rows, cudaStream_t s) {
  if (experts < 1 || experts > MOE_MAX_EXPERTS || tile_rows < 1) return -2;
  if (n_pairs > 512 && experts <= ALIGN_EXPERTS)
    return launch_dependent_cluster(moe_align_cluster_kernel, dim3(ALIGN_CTAS), dim3(256), 0, s, dim3(ALIGN_CTAS, 1, 1), ids, n_pairs, experts,
                                    sorted, capacity, tile_expert, n_tiles, tile_rows);
  return launch_dependent(moe_align_kernel, dim3(1), dim3(n_pairs > 1024 ? 1024 : 256), 0, s, ids, n_pairs, experts, sorted, capacity,
                          tile_expert, n_tiles, tile_rows);
}

int sb_moe_tiles(int dtype, int up, int tile_rows, const void* x, const void* w, void* y, const int* sorted,
                 const int* tile_expert, const int* n_tiles, int max_tiles, int k_dim, int n_out, int top, float limit,
                 const float* in_scale, cudaStream_t s) {
  if (max_tiles == 0) return 0;
#define MOE_ARGS dtype, tile_rows, x, w, y, sorted, tile_expert, n_tiles, max_tiles, k_dim, n_out, top, limit, in_scale, s
  if (up == 0) return moe_tiles_mode<0>(MOE_ARGS);
  if (up == 1) return moe_tiles_mode<1>(MOE_ARGS);
  if (up == 2) return moe_tiles_mode<2>(MOE_ARGS);
#undef MOE_ARGS
  return -2;
}

// Both products over tiles of MOE_FEW rows, bfloat16: `up` (1 or 2) of h [.., width] and w [experts, (2 *) inner, width] into act [capacity,
// inner], then down [experts, width, inner] into per_pair [n_pairs, width].  They are one entry because the second reads the tiles in front of
// its wait: nothing may stand between the two.
int sb_moe_few(int up, const void* h, const void* w, void* act, const void* down, void* per_pair, const int* sorted,
               const int* tile_expert, const int* n_tiles, int max_tiles, int width, int inner, int top, float limit,
               const float* in_scale, cudaStream_t s) {
  if (max_tiles == 0) return 0;
  if (up < 1 || up > 2 || top < 1 || width % 8 || inner % 8 || (((uintptr_t)h | (uintptr_t)w | (uintptr_t)act | (uintptr_t)down) % 16)) return -2;
  const int rc = up == 1 ? moe_few<1>(h, w, act, sorted, tile_expert, n_tiles, max_tiles, width, inner, top, limit, in_scale, s)
                         : moe_few<2>(h, w, act, sorted, tile_expert, n_tiles, max_tiles, width, inner, top, limit, in_scale, s);
  if (rc) return rc;
  return moe_few<0>(act, down, per_pair, sorted, tile_expert, n_tiles, max_tiles, inner, width, top, limit, nullptr, s);
}

int sb_moe_combine(int dtype, const void* down, const float* weights, void* out, int n_tokens, int width, int top,
                   const int* ids, int experts, const void* h, const void* shared, const float* shared_gate,
                   cudaStream_t s) {
  if (n_tokens == 0) return 0;
  if ((ids != nullptr) != (h != nullptr) || (shared != nullptr) != (shared_gate != nullptr)) return -2;
  if (dtype == 1 && width % 8 == 0 && !(((uintptr_t)down | (uintptr_t)out | (uintptr_t)h | (uintptr_t)shared) % 16)) {
    const dim3 grid(n_tokens, (width / 8 + 127) / 128);
    return launch_dependent(ids ? moe_combine_vec_kernel<true> : moe_combine_vec_kernel<false>, grid, dim3(128), 0, s,
                            (const bf16*)down, weights, (bf16*)out, width, top, ids, experts, (const bf16*)h, (const bf16*)shared,
                            shared_gate);
  }
  const int threads = width >= 1024 ? 256 : 128;
  if (dtype == 0)
    return launch_dependent(moe_combine_kernel<float>, dim3(n_tokens), dim3(threads), 0, s, (const float*)down,
                            weights, (float*)out, width, top, ids, experts, (const float*)h, (const float*)shared,
                            shared_gate);
  return launch_dependent(moe_combine_kernel<bf16>, dim3(n_tokens), dim3(threads), 0, s, (const bf16*)down, weights,
                          (bf16*)out, width, top, ids, experts, (const bf16*)h, (const bf16*)shared, shared_gate);
}

// The router that scores by the softmax over all `outputs` rows of w (float [outputs (+ 1), width]): the choice
// goes by score + correction (float [outputs] or null) among the outputs of the `keep` of `groups` equal groups
// of neighbours whose largest such number is largest (the lower index first among equals, here and in the
// choice); weights: the chosen plain scores over their sum (+ 1e-20), times weight_scale.  gate_out (null:
// none): w has one row more, and gate_out[t] = sigmoid of that row's product.
int sb_moe_route_all(int dtype, const void* h, const float* w, const float* correction, int* ids, float* weights,
                     float* gate_out, int n_tokens, int width, int outputs, int top, int groups, int keep,
                     float weight_scale, cudaStream_t s) {
  if (n_tokens == 0) return 0;
  if (outputs < 1 || outputs > MOE_MAX_EXPERTS || top < 1 || top > MOE_MAX_TOP) return -2;
  if (groups < 1 || outputs % groups || keep < 1 || keep > groups || top > outputs / groups * keep) return -2;
  // 4 tokens a block (see sb_moe_route), where their numbers fit beside the staged rows into the 48 KB of a plain launch: 256
  // outputs in 256 groups do not
  const size_t token_bytes = (size_t)(3 * outputs + 1 + groups) * sizeof(float);
  const bool many = n_tokens >= 4 * 148 && MOE_STAGE_BYTES + 4 * token_bytes <= 48 * 1024;
  const int threads = many ? (outputs > 16 ? 256 : 128) : outputs >= 16 ? 512 : outputs > 4 ? 256 : 128;
  const int blocks = many ? (n_tokens + 3) / 4 : n_tokens;
  const size_t smem = many ? MOE_STAGE_BYTES + 4 * token_bytes : token_bytes;
#define MOE_ROUTE(T, TOK)                                                                                              \
  return launch_dependent(moe_route_all_kernel<T, TOK>, dim3(blocks), dim3(threads), smem, s, (const T*)h, w, correction, ids, \
                          weights, gate_out, n_tokens, width, outputs, top, groups, keep, weight_scale)
  if (dtype == 0) { if (many) MOE_ROUTE(float, 4); MOE_ROUTE(float, 1); }
  if (many) MOE_ROUTE(bf16, 4);
  MOE_ROUTE(bf16, 1);
#undef MOE_ROUTE
}

}  // extern "C"
