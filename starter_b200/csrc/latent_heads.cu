// The head-wise products around the attention over cached latents (attention_latent.cu) for steps of few tokens, bfloat16:
//
//   fold    qa[t, h] = [q_plain[t, h] uk_h | q_rot[t, h] turned by the token's position]: a query head in latent space
//   unfold  a[t, h] = (summed latents of head h) uv_h^T, times sigmoid(gate) where the layer has one; the summed latents come as the
//           attention's parts (sums, references and sums of weights of every part of the keys), joined here as they are read
//
// A head's matrices are 128 KB and a step has a few rows, so each of these is a chain of latencies, not of bytes.  As library products
// with a rotation, a merge and a gate around them they were five launches of 3 to 6 us; these two have their matrices in shared
// memory before the kernel in front of them has ended.  A layer of 16 heads over a latent of 512: 8
// sequences of about 2,000 tokens at width 2,048 47.5 -> 43.3 us, 2 of 54 at width 1,280 37.2 -> 29.4, 4 of 863 41.3 -> 35.5.
// Products are m16n8k16 with float accumulators of values rounded to bfloat16 where the separate kernels round them: queries, summed
// latents, the product in front of the gate, the gated result.
#include "common.cuh"

#define LH_ROWS 16               // tokens a block

__device__ __forceinline__ void lh_copy16(void* dst, const void* src, bool real) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  const int bytes = real ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void lh_arrive() { asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory"); }
__device__ __forceinline__ void lh_mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void lh_ldsm4(uint32_t (&r)[4], const void* p) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void lh_ldsm4_t(uint32_t (&r)[4], const void* p) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}

// ------------------------------------------------------------------------------------------ fold
// A block of four warps: 64 entries of a head's latent query for 16 tokens, a warp 16 of them.  The blocks of a head's first entries turn
// its rotated part too.
#define LH_FOLD_COLS 64
#define LH_MAX_DIM 256
__global__ void __launch_bounds__(128)
latent_fold_kernel(const bf16* __restrict__ q, const bf16* __restrict__ uk, bf16* __restrict__ qa, const float* __restrict__ cos_t,
                   const float* __restrict__ sin_t, int table_width, const int* __restrict__ tok_pos, int n_tokens, int heads,
                   int dim, int rot, int rot_dims, int rank, int split) {
  extern __shared__ __align__(16) bf16 lh_smem[];
  const int ldw = LH_FOLD_COLS + 8, ldq = dim + 8;
  bf16* w = lh_smem;                                // [dim][64]
  bf16* rows = w + dim * ldw;                       // [16][dim]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, h = blockIdx.y, c0 = blockIdx.x * LH_FOLD_COLS;
  const int t0 = blockIdx.z * LH_ROWS;
  for (int e = tid; e < dim * (LH_FOLD_COLS / 8); e += 128) {        // (weights: no earlier kernel writes them)
    const int k = e >> 3, c = (e & 7) * 8;
    lh_copy16(w + k * ldw + c, uk + ((size_t)h * dim + k) * rank + c0 + c, true);
  }
  pdl_trigger();
  pdl_wait();
  SB_BEHIND_WAIT(q); SB_BEHIND_WAIT(tok_pos);
  const int width = dim + rot;
  for (int e = tid; e < LH_ROWS * (dim / 8); e += 128) {
    const int r = e / (dim / 8), c = (e - r * (dim / 8)) * 8;
    const bool real = t0 + r < n_tokens;
    lh_copy16(rows + r * ldq + c, q + ((size_t)(real ? t0 + r : t0) * heads + h) * width + c, real);
  }
  if (blockIdx.x == 0) {
    const int half = rot_dims / 2, per = half + rot - rot_dims;
    for (int e = tid; e < min(LH_ROWS, n_tokens - t0) * per; e += 128) {
      const int r = e / per, i = e - r * per, t = t0 + r;
      const bf16* src = q + ((size_t)t * heads + h) * width + dim;
      bf16* dst = qa + ((size_t)t * heads + h) * (rank + rot) + rank;
      if (i < half) {
        const int ia = split ? i : 2 * i, ib = split ? i + half : 2 * i + 1, pos = tok_pos[t];
        const float a = to_f<bf16>(src[ia]), b = to_f<bf16>(src[ib]);
        const float c = cos_t[(size_t)pos * table_width + i], s = sin_t[(size_t)pos * table_width + i];
        dst[ia] = from_f<bf16>(a * c - b * s);
        dst[ib] = from_f<bf16>(b * c + a * s);
      } else {
        dst[rot_dims + i - half] = src[rot_dims + i - half];
      }
    }
  }
  lh_arrive();
  __syncthreads();
  float acc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
  const int g = lane >> 2, x = lane & 3, mi = lane >> 3;
#pragma unroll 4
  for (int k = 0; k < dim; k += 16) {
    uint32_t a[4], b[4];
    lh_ldsm4(a, rows + ((lane & 7) + (mi & 1) * 8) * ldq + k + (mi >> 1) * 8);
    lh_ldsm4_t(b, w + (k + (lane & 7) + (mi & 1) * 8) * ldw + 16 * warp + (mi >> 1) * 8);
    lh_mma(acc[0], a, b[0], b[1]);
    lh_mma(acc[1], a, b[2], b[3]);
  }
#pragma unroll
  for (int n = 0; n < 2; ++n)
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int t = t0 + g + 8 * r, c = c0 + 16 * warp + 8 * n + 2 * x;
      if (t < n_tokens)
        *reinterpret_cast<__nv_bfloat162*>(qa + ((size_t)t * heads + h) * (rank + rot) + c) =
            __floats2bfloat162_rn(acc[n][2 * r], acc[n][2 * r + 1]);
    }
}

// ------------------------------------------------------------------------------------------ unfold
// A block of eight warps: 32 entries of a head's output for 16 tokens.  The blocks of a head are a cluster: each joins the parts of its
// share of the latent and takes the others' from their shared memory (every block for itself: 8 tokens in 18 parts are twelve rounds of loads, and a
// layer took 49.3 us).  Then a warp has eight entries and half of the latent, and the halves meet in shared memory.
#define LH_OUT_COLS 32
#define LH_MAX_PARTS 32
__global__ void __launch_bounds__(256)
latent_unfold_kernel(const bf16* __restrict__ summed, const float* __restrict__ part_acc, const float* __restrict__ part_ml,
                     int n_parts, int shares, const float* __restrict__ sink, const bf16* __restrict__ uv, const bf16* __restrict__ gate, int ldg,
                     bf16* __restrict__ out, int n_tokens, int heads, int rank, int vdim) {
  extern __shared__ __align__(16) bf16 lh_smem[];
  __shared__ float factor[LH_ROWS][LH_MAX_PARTS];
  __shared__ float half_sum[4][4][32];
  const int ld = rank + 8;
  bf16* w = lh_smem;                                // [32][rank]
  bf16* rows = w + LH_OUT_COLS * ld;                // [16][rank]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, h = blockIdx.y, c0 = blockIdx.x * LH_OUT_COLS;
  const int t0 = blockIdx.z * LH_ROWS, here = min(LH_ROWS, n_tokens - t0);
  const int pieces = rank / 8;
  for (int e = tid; e < LH_OUT_COLS * pieces; e += 256) {            // (weights: no earlier kernel writes them)
    const int n = e / pieces, c = (e - n * pieces) * 8;
    lh_copy16(w + n * ld + c, uv + ((size_t)h * vdim + min(c0 + n, vdim - 1)) * rank + c, true);
  }
  pdl_trigger();
  pdl_wait();
  SB_BEHIND_WAIT(summed); SB_BEHIND_WAIT(part_acc); SB_BEHIND_WAIT(part_ml); SB_BEHIND_WAIT(gate);
  if (part_acc) {
    const size_t n_rows = (size_t)n_tokens * heads;
    // the parts' factors, a warp a token, as latent_merge_kernel has them
    for (int r = warp; r < here; r += 8) {
      const size_t row = (size_t)(t0 + r) * heads + h;
      const float2 ml = lane < n_parts ? *reinterpret_cast<const float2*>(part_ml + ((size_t)lane * n_rows + row) * 2) : make_float2(-INFINITY, 0.f);
      const float sk = sink ? sink[h] : -INFINITY;
      const float M = fmaxf(warp_max(ml.x), sk);
      const float e = ml.x == -INFINITY ? 0.f : expf(ml.x - M);
      float L = warp_sum(ml.y * e);
      if (sink) L += expf(sk - M);
      factor[r][lane] = e / L;
    }
    __syncthreads();
    // this block's share of the latent, in whole pieces of eight
    const int per = (pieces + shares - 1) / shares, own = shares > 1 ? blockIdx.x : 0;
    const int from = min(own * per, pieces), quads = 2 * (min(from + per, pieces) - from);
    for (int e = tid; e < LH_ROWS * quads; e += 256) {
      const int r = e / quads, c = 8 * from + (e - r * quads) * 4;
      float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
      if (r < here) {
        const float* acc = part_acc + ((size_t)(t0 + r) * heads + h) * rank + c;
        for (int s0 = 0; s0 < n_parts; s0 += 8) {
          float4 v[8];
#pragma unroll
          for (int s = 0; s < 8; ++s)
            v[s] = s0 + s < n_parts ? *reinterpret_cast<const float4*>(acc + (size_t)(s0 + s) * n_rows * rank) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
          for (int s = 0; s < 8; ++s) {
            const float f = s0 + s < n_parts ? factor[r][s0 + s] : 0.f;
            // (a part without keys left zeros; its factor is zero, as that of a part whose weights vanish beside the others')
            a.x += f != 0.f ? v[s].x * f : 0.f;
            a.y += f != 0.f ? v[s].y * f : 0.f;
            a.z += f != 0.f ? v[s].z * f : 0.f;
            a.w += f != 0.f ? v[s].w * f : 0.f;
          }
        }
      }
      __nv_bfloat162* to = reinterpret_cast<__nv_bfloat162*>(rows + r * ld + c);
      to[0] = __floats2bfloat162_rn(a.x, a.y);
      to[1] = __floats2bfloat162_rn(a.z, a.w);
    }
    if (shares > 1) {
      __syncwarp();                                 // (.aligned: a whole warp at once, and the loop above may leave it in two)
      asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
      for (int e = tid; e < here * pieces; e += 256) {
        const int r = e / pieces, piece = e - r * pieces, whose = piece / per;
        if (whose == own) continue;
        bf16* at = rows + r * ld + 8 * piece;
        uint4 v;
        asm volatile("{\n\t.reg .b32 a;\n\tmapa.shared::cluster.u32 a, %4, %5;\n\tld.shared::cluster.v4.u32 {%0, %1, %2, %3}, [a];\n\t}"
                     : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"((unsigned)__cvta_generic_to_shared(at)), "r"(whose) : "memory");
        *reinterpret_cast<uint4*>(at) = v;
      }
    }
  } else {
    for (int e = tid; e < LH_ROWS * pieces; e += 256) {
      const int r = e / pieces, c = (e - r * pieces) * 8;
      lh_copy16(rows + r * ld + c, summed + ((size_t)(t0 + (r < here ? r : 0)) * heads + h) * rank + c, r < here);
    }
  }
  lh_arrive();
  __syncthreads();
  // (nobody leaves while others read from it; the wait stands at the end)
  if (shares > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
  // warp: entries 8 (w % 4) .. and the lower (w < 4) or upper half of the latent, in steps of 16
  const int g = lane >> 2, x = lane & 3, mi = lane >> 3, n0 = 8 * (warp & 3), steps = rank / 16, first = warp < 4 ? 0 : (steps + 1) / 2;
  const int last = warp < 4 ? (steps + 1) / 2 : steps;
  float acc[4] = {0.f, 0.f, 0.f, 0.f};
  for (int s = first; s < last; ++s) {
    uint32_t a[4];
    lh_ldsm4(a, rows + ((lane & 7) + (mi & 1) * 8) * ld + 16 * s + (mi >> 1) * 8);
    const bf16* b = w + (n0 + g) * ld + 16 * s + 2 * x;
    lh_mma(acc, a, *reinterpret_cast<const uint32_t*>(b), *reinterpret_cast<const uint32_t*>(b + 8));
  }
  if (warp >= 4) {
#pragma unroll
    for (int e = 0; e < 4; ++e) half_sum[warp - 4][e][lane] = acc[e];
  }
  __syncthreads();
  if (shares > 1) asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
  if (warp >= 4) return;
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const int t = t0 + g + 8 * r, c = c0 + n0 + 2 * x;
    if (t >= n_tokens || c >= vdim) continue;
    float o[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      o[e] = rnd<bf16>(acc[2 * r + e] + half_sum[warp][2 * r + e][lane]);
      if (gate) o[e] = o[e] / (1.f + expf(-to_f<bf16>(gate[(size_t)t * ldg + h * vdim + c + e])));
    }
    *reinterpret_cast<__nv_bfloat162*>(out + ((size_t)t * heads + h) * vdim + c) = __floats2bfloat162_rn(o[0], o[1]);
  }
}

extern "C" {

// Whether the two kernels take these sizes (bfloat16, 16-byte aligned operands).
int sb_latent_heads_take(int dim, int rot, int rank, int vdim) {
  return dim % 16 == 0 && dim >= 16 && dim <= LH_MAX_DIM && rot % 8 == 0 && rank % 64 == 0 && rank >= 64 && rank <= 512 && vdim % 8 == 0;
}

// q [n_tokens, heads * (dim + rot)], uk [heads, dim, rank], qa [n_tokens, heads, rank + rot]; the tables and `split` as
// sb_latent_rotate_q's.
int sb_latent_fold(const void* q, const void* uk, void* qa, const float* cos_t, const float* sin_t, int table_width, const int* tok_pos,
                   int n_tokens, int heads, int dim, int rot, int rot_dims, int rank, int split, cudaStream_t s) {
  if (n_tokens == 0) return 0;
  if (!sb_latent_heads_take(dim, rot, rank, 8) || (((uintptr_t)q | (uintptr_t)uk | (uintptr_t)qa) & 15) || heads > 65535) return -2;
  const size_t smem = (size_t)(dim * (LH_FOLD_COLS + 8) + LH_ROWS * (dim + 8)) * sizeof(bf16);
  return launch_dependent(latent_fold_kernel, dim3(rank / LH_FOLD_COLS, heads, (n_tokens + LH_ROWS - 1) / LH_ROWS), dim3(128), smem, s,
                          (const bf16*)q, (const bf16*)uk, (bf16*)qa, cos_t, sin_t, table_width, tok_pos, n_tokens, heads, dim, rot,
                          rot_dims, rank, split);
}

// Either summed [n_tokens, heads, rank] (part_acc null) or the parts of sb_latent_attention_tc (n_parts of them, at most 32; sink joins
// here).  uv [heads, vdim, rank]; gate: null or the first of heads * vdim columns of rows of ldg entries; out [n_tokens, heads * vdim].
int sb_latent_unfold(const void* summed, const float* part_acc, const float* part_ml, int n_parts, const float* sink, const void* uv,
                     const void* gate, int ldg, void* out, int n_tokens, int heads, int rank, int vdim, cudaStream_t s) {
  if (n_tokens == 0) return 0;
  if (!sb_latent_heads_take(16, 8, rank, vdim) || n_parts < 1 || n_parts > LH_MAX_PARTS || heads > 65535) return -2;
  if (((uintptr_t)summed | (uintptr_t)part_acc | (uintptr_t)uv | (uintptr_t)out) & 15) return -2;
  const size_t smem = (size_t)((LH_OUT_COLS + LH_ROWS) * (rank + 8)) * sizeof(bf16);
  // (at every call, one limit for all sizes: the attribute is the current device's and other threads launch too)
  const cudaError_t err = cudaFuncSetAttribute(latent_unfold_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 64 * 1024);
  if (err != cudaSuccess) return (int)err;
  const int blocks = (vdim + LH_OUT_COLS - 1) / LH_OUT_COLS;
  const int shares = part_acc && blocks > 1 && blocks <= 8 ? blocks : 1;
  return launch_dependent_cluster(latent_unfold_kernel, dim3(blocks, heads, (n_tokens + LH_ROWS - 1) / LH_ROWS), dim3(256), smem, s,
                                  dim3(shares), (const bf16*)summed, part_acc, part_ml, n_parts, shares, sink, (const bf16*)uv,
                                  (const bf16*)gate, ldg, (bf16*)out, n_tokens, heads, rank, vdim);
}

}  // extern "C"
