// True 32-bit y[m, n] = sum_k x[m, k] * w[n, k] for many rows: FFMA only, no reduced-precision
// matrix mode.  This is the prompt-sized projection of the float32 path (the bfloat16 path uses
// tensor cores instead).
//
// A block makes 64 x 128 outputs with 128 threads, 8 x 8 a thread, from k-slices of 16 in two shared-memory
// buffers (the next slice's 16-byte loads are in flight while one is multiplied).  Bound by the fma pipe: 64 fmas a
// thread and slice entry for 16 floats from shared memory (512 bytes a warp and 16-byte load, 4 of an SM's cycles
// whether lanes share addresses or not; with x kept twice in a row, to spare the copies into the packed fma's
// operands, the loads were the bound: 35.7 TFLOP/s at 4096^3).  Packed fmas (two columns) halve the issue slots.
// 46.7 TFLOP/s at 4096^3 (128 x 128 tiles, slices of 8 and 4-byte loads before: 24.2); 141 x 2048 x 2048: 47 us
// (434 before, when 32 blocks walked all of k), 141 x 8192 x 2048: 172 us (436).
// The k range is cut into parts whose number depends on n_out and k_dim alone.  With few output tiles the parts of a
// tile are the blocks of one cluster, which leave their sums in their shared memory and add them, part by part; with
// enough tiles a block walks the parts itself and adds in the same order.  The sum for one (m, n) is therefore
// the same whatever the other rows of the call are: a chain over k in each part, the parts added in order.
#include "common.cuh"

#define SG_M 64
#define SG_N 128
#define SG_K 16
#define SG_XLD (SG_M + 4)
#define SG_WLD (SG_N + 4)
#define SG_MAX_PARTS 8

struct SgemmTiles {
  float x[2][SG_K][SG_XLD];
  float w[2][SG_K][SG_WLD];
  float sum[SG_M][SG_N];           // a part's sums (cluster), or the parts so far (one block)
};

__device__ __forceinline__ unsigned long long sg_fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}

__device__ __forceinline__ unsigned long long sg_twice(float v) {
  unsigned long long d;
  asm("mov.b64 %0, {%1, %1};" : "=l"(d) : "f"(v));
  return d;
}

// VEC: rows of x and w may be read in 16-byte pieces.
template <bool VEC>
__global__ void __launch_bounds__(128)
sgemm_nt_kernel(const float* __restrict__ x, const float* __restrict__ w, float* __restrict__ y, int rows, int n_out,
                int k_dim, int parts, int part_k) {
  extern __shared__ __align__(16) unsigned char sgemm_smem[];
  SgemmTiles& sm = *reinterpret_cast<SgemmTiles*>(sgemm_smem);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int tiles_n = (n_out + SG_N - 1) / SG_N;
  const int n_base = (int)(blockIdx.x % tiles_n) * SG_N, m_base = (int)(blockIdx.x / tiles_n) * SG_M;
  // a thread's outputs: rows m0 .. m0 + 3 and m0 + 16 .. m0 + 19, columns n0 .. n0 + 3 and n0 + 64 .. n0 + 67
  const int m0 = 4 * (lane & 3) + 32 * (warp & 1), n0 = 4 * ((lane >> 2) + 8 * (warp >> 1));
  const bool split = gridDim.z > 1;                  // a part a block, or all parts
  const int p_begin = split ? blockIdx.z : 0, p_end = split ? blockIdx.z + 1 : parts;

  float4 px[2], pw[4];
  auto piece = [&](const float* from, int limit, int row, int k, int k_end) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (row < limit) {
      const float* at = from + (size_t)row * k_dim + k;
      if (VEC) {
        if (k < k_end) v = *reinterpret_cast<const float4*>(at);       // (k_end is a multiple of 4 here)
      } else {
        if (k < k_end) v.x = at[0];
        if (k + 1 < k_end) v.y = at[1];
        if (k + 2 < k_end) v.z = at[2];
        if (k + 3 < k_end) v.w = at[3];
      }
    }
    return v;
  };
  const int lr = tid >> 2, lk = (tid & 3) * 4;       // rows lr + 32 i, entries lk .. lk + 3 of a slice
  auto fetch = [&](int k0, int k_end) {
#pragma unroll
    for (int i = 0; i < 2; ++i) px[i] = piece(x, rows, m_base + lr + 32 * i, k0 + lk, k_end);
#pragma unroll
    for (int i = 0; i < 4; ++i) pw[i] = piece(w, n_out, n_base + lr + 32 * i, k0 + lk, k_end);
  };
  auto file = [&](int b) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const float v[4] = {px[i].x, px[i].y, px[i].z, px[i].w};
#pragma unroll
      for (int j = 0; j < 4; ++j) sm.x[b][lk + j][lr + 32 * i] = v[j];
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float v[4] = {pw[i].x, pw[i].y, pw[i].z, pw[i].w};
#pragma unroll
      for (int j = 0; j < 4; ++j) sm.w[b][lk + j][lr + 32 * i] = v[j];
    }
  };

  for (int p = p_begin; p < p_end; ++p) {
    const int k_begin = p * part_k, k_end = min(k_dim, k_begin + part_k);
    unsigned long long acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
    fetch(k_begin, k_end);
    file(0);
    __syncthreads();
    int b = 0;
    for (int k0 = k_begin; k0 < k_end; k0 += SG_K, b ^= 1) {
      const bool more = k0 + SG_K < k_end;
      if (more) fetch(k0 + SG_K, k_end);
#pragma unroll
      for (int k = 0; k < SG_K; ++k) {
        unsigned long long a[8], c[4];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const float4 v = *reinterpret_cast<const float4*>(&sm.x[b][k][m0 + 16 * i]);
          a[4 * i] = sg_twice(v.x);
          a[4 * i + 1] = sg_twice(v.y);
          a[4 * i + 2] = sg_twice(v.z);
          a[4 * i + 3] = sg_twice(v.w);
        }
        const ulonglong2 w0 = *reinterpret_cast<const ulonglong2*>(&sm.w[b][k][n0]);
        const ulonglong2 w1 = *reinterpret_cast<const ulonglong2*>(&sm.w[b][k][n0 + 64]);
        c[0] = w0.x; c[1] = w0.y; c[2] = w1.x; c[3] = w1.y;
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[i][j] = sg_fma2(a[i], c[j], acc[i][j]);
      }
      if (more) file(b ^ 1);
      __syncthreads();
    }
    // the part's sums (a thread's own places): left for the cluster, or added to the parts before
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float2* at = reinterpret_cast<float2*>(&sm.sum[m0 + 16 * (i >> 2) + (i & 3)][n0 + (j >> 1) * 64 + (j & 1) * 2]);
        float2 v = make_float2(__uint_as_float((unsigned)acc[i][j]), __uint_as_float((unsigned)(acc[i][j] >> 32)));
        if (p > p_begin) {
          const float2 o = *at;
          v.x = o.x + v.x;
          v.y = o.y + v.y;
        }
        *at = v;
      }
  }
  unsigned rank = 0, size = 1;
  if (split) {
    rank = blockIdx.z;
    size = gridDim.z;
    asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
  } else {
    __syncthreads();
  }
  // block `rank` of the cluster stores the tile's rows rank, rank + size, ..; a warp a row
  for (int m = rank + size * warp; m < SG_M; m += size * 4) {
    if (m_base + m >= rows) break;
    const int n = 4 * lane;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    const unsigned at = (unsigned)__cvta_generic_to_shared(&sm.sum[m][n]);
    for (unsigned r = 0; r < size; ++r) {
      float4 o;
      if (split) {
        unsigned peer;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(peer) : "r"(at), "r"(r));
        asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(o.x), "=f"(o.y), "=f"(o.z), "=f"(o.w) : "r"(peer) : "memory");
      } else {
        o = *reinterpret_cast<const float4*>(&sm.sum[m][n]);
      }
      if (r == 0) v = o;
      else v = make_float4(v.x + o.x, v.y + o.y, v.z + o.z, v.w + o.w);
    }
    float* to = y + (size_t)(m_base + m) * n_out + n_base + n;
    const float e[4] = {v.x, v.y, v.z, v.w};
    if (n_out % 4 == 0) {
      if (n_base + n < n_out) *reinterpret_cast<float4*>(to) = v;
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (n_base + n + j < n_out) to[j] = e[j];
    }
  }
  // no block leaves while a peer may still read its sums
  if (split) asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
}

extern "C" {

// How many parts the k range of a product is cut into: enough that one row of output tiles fills the SMs about
// twice (two to three blocks fit an SM), none shorter than 128 (eight slices: below that a block mostly fills and
// drains its pipeline).  A cluster's blocks take the parts while all tiles' parts are at most a few waves; from four
// waves of tiles on there is nothing to fill and the parts' sums need not travel.
int sb_sgemm_parts(int n_out, int k_dim) {
  const int tiles = (n_out + SG_N - 1) / SG_N;
  int parts = 1;
  while (parts < SG_MAX_PARTS && parts * tiles < 296 && k_dim >= 2 * parts * 128) parts *= 2;
  return parts;
}

int sb_sgemm_nt(const float* x, const float* w, float* y, int rows, int n_out, int k_dim,
                cudaStream_t s) {
  if (rows == 0 || n_out == 0) return 0;
  const int parts = sb_sgemm_parts(n_out, k_dim);
  const int part_k = ((k_dim + parts - 1) / parts + SG_K - 1) / SG_K * SG_K;
  const int tn = (n_out + SG_N - 1) / SG_N, tm = (rows + SG_M - 1) / SG_M;
  const bool vec = k_dim % 4 == 0 && ((uintptr_t)x % 16) == 0 && ((uintptr_t)w % 16) == 0;
  const bool split = parts > 1 && (long long)tn * tm < 4 * 148;      // (an order of work, not of sums: see above)
  auto kernel = vec ? sgemm_nt_kernel<true> : sgemm_nt_kernel<false>;
  cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SgemmTiles));
  if (err != cudaSuccess) return (int)err;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)((long long)tn * tm), 1, split ? parts : 1);
  cfg.blockDim = dim3(128);
  cfg.dynamicSmemBytes = sizeof(SgemmTiles);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = split ? parts : 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  err = cudaLaunchKernelEx(&cfg, kernel, x, w, y, rows, n_out, k_dim, parts, part_k);
  return err == cudaSuccess ? SB_LAUNCH_RESULT() : (int)err;
}

}  // extern "C"
