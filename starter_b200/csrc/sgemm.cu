// y[m, n] = sum_k x[m, k] * w[n, k] of float32 matrices for many rows, in full 32-bit precision, on the
// fifth-generation tensor cores.  This is the prompt-sized projection of the float32 path.
//
// Every operand is cut into three bfloat16 pieces, a = a0 + a1 + a2 to 24 bits, and a product is
// a0 b0 + (a0 b1 + a1 b0) + (a1 b1 + a0 b2 + a2 b0); what is left out is below 2^-26 of it.  The tensor cores truncate
// when they add to an accumulator, so no accumulator lives long: the six products of SG_CHUNK entries of k start a fresh
// one, the small terms first (their truncations are 2^-8 of the others'), and its sum joins the result by rounded
// additions in registers.  Against 64 bits the error is below that of a chain of 32-bit fmas (sizes below).
//
// A block owns 128 rows of w (the MMA's M) and up to 160 of x (its N; equal tiles in steps of 16, so that 141 rows are
// one tile of 144).  Eight warps read 64-entry slices of both as floats (the next slice's 16-byte loads in flight
// while the MMAs of the one before run), cut them and file the pieces in 128-byte swizzled tiles; eight warps empty the
// two accumulators in turn, two of which issue the MMAs.
// Events around a launch, L2 flushed, the multiply-add kernel of 64 x 128 tiles that this replaces -> here: 141 x 2048 x 2048
// 52 -> 30 us, 141 x 8192 x 2048 177 -> 55, 20 x 2048 x 2048 41 -> 22, 4096^3 2,942 -> 1,095 (126 TFLOP/s); nothing
// measured between 17 x 5 x 4097 and 4096^3 is slower.  Error against 64 bits (rms, of the result's): 2.9e-7 -> 1.0e-7 at k = 2048,
// 4.1e-7 -> 1.3e-7 at 4096.  By clock64() a slice at 144 rows is about 3,000 cycles where its MMAs alone are 1,730: issuing
// costs some 90 cycles an MMA, and cutting 2,500 a slice.  Short k is bound by the ends: 5,000 cycles to the first
// accumulator, 6,000 to add eight parts.
//
// The k range is cut into parts whose number depends on n_out and k_dim alone, the blocks of one cluster; they leave
// their sums in shared memory and each adds its share of the tile, part by part.  So the sum for one (m, n) is the same
// whatever the other rows of the call are.
//
// What the pieces cannot hold is computed again as a chain of fmas.  Infinities, NaN and values next to the largest float do not
// survive the cut (inf - inf): a result that is not finite is formed again.  A piece below 2^-133 is lost, which is less than
// 2^-134 of an operand, and only of one below 2^-109: a result below 2^-80 is formed again, and so is every result whose
// one row has such an entry and whose other row has one of 2^20 or more (where it has none, what is lost is under 2^-34 of the smallest
// result that stays).  A product below 2^-126 may come out as zero: a zero is formed again where both rows have entries and one of them
// has some below 2^-63.  The cutters keep the smallest magnitude they see (12 operations beside some 52 of cutting eight entries: a float32
// layer of 141 tokens 147 -> 152 us); only a block that finds one below 2^-63 goes over its rows again and notes what each has: all
// of k if there was one below 2^-109, else up to the first entry that is not zero (4096^3: 1,095 us, 1,180 with entries below
// 2^-63, 2,430 with entries below 2^-109).
#include "tcgen05.cuh"

#define SG_W 128                 // rows of w a block
#define SG_X 160                 // rows of x a block, at most (two slices of both fill the shared memory)
#define SG_K 64                  // entries of k a slice: 128 bytes of bfloat16, one swizzle atom
#define SG_CHUNK 32              // entries of k a fresh accumulator sums: half a slice
#define SG_W_PLANE (SG_W * SG_K * 2)
#define SG_CUTTERS 8             // warps that read and cut
#define SG_DRAINERS 8            // warps that empty the accumulators: a lane quarter and every other 16 columns each
#define SG_THREADS (32 * (SG_CUTTERS + SG_DRAINERS))
#define SG_MAX_PARTS 8
#define SG_MAX_STAGES 4
#define SG_SMEM (224 * 1024)

// What a row of an operand has in the part of k that a block cuts.
#define SG_TINY 1                // entries below 2^-109, which are not cut exactly
#define SG_SMALL 2               // entries below 2^-63, whose products may be below the smallest float
#define SG_LARGE 4               // entries of 2^20 or more
#define SG_ENTRIES 8             // entries that are not zero

struct SgemmArgs {
  const float* x;
  const float* w;
  float* y;
  int* status;
  int rows, n_out, k_dim, tile_rows, parts, stages;
  int withhold;                    // >= 0: the first cutter does not hand over this slice (tests of the give-up path)
  unsigned long long wait_limit_ns;
};

// 16 columns of this warp's lane quarter, or twice 16 that are 32 apart.
__device__ __forceinline__ void sg_tmem_load16(uint32_t taddr, float* v) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n\t"
               "tcgen05.wait::ld.sync.aligned;"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]), "=f"(v[8]), "=f"(v[9]), "=f"(v[10]), "=f"(v[11]), "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15])
               : "r"(taddr) : "memory");
}
__device__ __forceinline__ void sg_tmem_load16x2(uint32_t taddr, float* v) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%32];\n\t"
               "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%33];\n\t"
               "tcgen05.wait::ld.sync.aligned;"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]), "=f"(v[8]), "=f"(v[9]), "=f"(v[10]), "=f"(v[11]), "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15]),
                 "=f"(v[16]), "=f"(v[17]), "=f"(v[18]), "=f"(v[19]), "=f"(v[20]), "=f"(v[21]), "=f"(v[22]), "=f"(v[23]), "=f"(v[24]), "=f"(v[25]), "=f"(v[26]), "=f"(v[27]), "=f"(v[28]), "=f"(v[29]), "=f"(v[30]), "=f"(v[31])
               : "r"(taddr), "r"(taddr + 32) : "memory");
}

// (volatile: the loads stay where they are written, ahead of the wait for a free stage)
__device__ __forceinline__ float4 sg_load4(const float* at) {
  float4 v;
  asm volatile("ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(at));
  return v;
}

// Two floats as three pairs of bfloat16.
__device__ __forceinline__ void sg_cut(float a, float b, uint32_t& hi, uint32_t& mid, uint32_t& low) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  hi = *reinterpret_cast<const uint32_t*>(&h);
  a -= __uint_as_float(hi << 16);
  b -= __uint_as_float(hi & 0xffff0000u);
  const __nv_bfloat162 m = __floats2bfloat162_rn(a, b);
  mid = *reinterpret_cast<const uint32_t*>(&m);
  a -= __uint_as_float(mid << 16);
  b -= __uint_as_float(mid & 0xffff0000u);
  const __nv_bfloat162 l = __floats2bfloat162_rn(a, b);
  low = *reinterpret_cast<const uint32_t*>(&l);
}

// (addresses in shared memory are kept as such: through generic ones a store costs several times as much)
__device__ __forceinline__ void sg_store4(uint32_t at, uint4 v) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}

// The smallest of `least` and the magnitudes of eight entries that are not zero, as twice its bits less one (a zero's are the largest
// number there is).
__device__ __forceinline__ uint32_t sg_least(uint32_t least, const float4 (&v)[2]) {
  auto of = [](float a) { return 2u * __float_as_uint(a) - 1u; };
  least = __vimin3_u32(least, of(v[0].x), of(v[0].y));
  least = __vimin3_u32(least, of(v[0].z), of(v[0].w));
  least = __vimin3_u32(least, of(v[1].x), of(v[1].y));
  return __vimin3_u32(least, of(v[1].z), of(v[1].w));
}
#define SG_LEAST(e) (2u * ((127u - (e)) << 23) - 1u)      // of 2^-e

// What one entry has.
__device__ __forceinline__ uint32_t sg_note(float a) {
  a = fabsf(a);
  return a == 0.f ? 0u : SG_ENTRIES | (a < 0x1p-63f ? SG_SMALL : 0) | (a < 0x1p-109f ? SG_TINY : 0) | (a >= 0x1p20f ? SG_LARGE : 0);
}

__device__ __forceinline__ bool sg_again(float v) {
  const float a = fabsf(v);
  return !(a < INFINITY) || (a < 0x1p-80f && a != 0.f);
}
// Whether what the cut lost, or products below the smallest float, may show in a sum of rows that have `x` and `w`.
__device__ __forceinline__ bool sg_cut_short(uint32_t x, uint32_t w) {
  return ((x & SG_TINY) && (w & SG_LARGE)) || ((w & SG_TINY) && (x & SG_LARGE));
}
__device__ __forceinline__ bool sg_vanished(uint32_t x, uint32_t w) { return ((x | w) & SG_SMALL) && (x & w & SG_ENTRIES); }

__device__ __noinline__ float sg_chain(const float* x, const float* w, int k_dim) {
  float sum = 0.f;
  for (int k = 0; k < k_dim; ++k) sum = fmaf(x[k], w[k], sum);
  return sum;
}

// A word of the same shared variable in block `rank` of the cluster.
__device__ __forceinline__ uint32_t sg_remote(const void* at, int rank) {
  uint32_t v;
  asm volatile("{\n\t.reg .b32 a;\n\tmapa.shared::cluster.u32 a, %1, %2;\n\tld.shared::cluster.u32 %0, [a];\n\t}"
               : "=r"(v) : "r"(smem_u32(at)), "r"(rank) : "memory");
  return v;
}

// VEC: rows of x and w may be read in 16-byte pieces.
template <bool VEC>
__global__ void __launch_bounds__(SG_THREADS, 1) sgemm_tcgen05_kernel(const SgemmArgs args) {
  extern __shared__ uint8_t sgemm_smem[];
  const uint32_t smem = (smem_u32(sgemm_smem) + 1023) & ~1023u;
  __shared__ uint64_t full_bar[SG_MAX_STAGES], empty_bar[SG_MAX_STAGES], sum_full[2], sum_empty[2], done_bar;
  __shared__ uint32_t tmem_holder;
  __shared__ __align__(16) uint32_t notes[SG_W + SG_X];      // what the rows of w, then of x, have in this block's part of k
  __shared__ uint32_t noted;                 // what any row of w has, and any of x above it (0: nothing is noted, nothing is small)
  __shared__ int abort_flag, small_flag;

  const int stages = args.stages, cols = args.tile_rows, k_dim = args.k_dim;
  const int x_plane = cols * SG_K * 2;
  const int stage_bytes = 3 * (SG_W_PLANE + x_plane);
  const uint32_t buffer_cols = cols <= 128 ? 128 : 256;
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int tiles = (args.n_out + SG_W - 1) / SG_W;
  const int n_base = (int)(blockIdx.x % tiles) * SG_W, m_base = (int)(blockIdx.x / tiles) * cols, part = blockIdx.y;
  const int kb_total = (k_dim + SG_K - 1) / SG_K;
  const int kb_part = (kb_total + args.parts - 1) / args.parts;
  const int kb_begin = min(part * kb_part, kb_total);
  const int n_kb = min(kb_begin + kb_part, kb_total) - kb_begin;
  const int rows_here = min(cols, args.rows - m_base);

  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) { mbar_init(&full_bar[s], SG_CUTTERS); mbar_init(&empty_bar[s], 2); }
    for (int b = 0; b < 2; ++b) { mbar_init(&sum_full[b], 1); mbar_init(&sum_empty[b], SG_DRAINERS); }
    mbar_init(&done_bar, 2);
    abort_flag = small_flag = 0;
    noted = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  pdl_trigger();
  if (warp == SG_CUTTERS) tmem_alloc(&tmem_holder, 2 * buffer_cols);
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_holder;
  volatile int* abort = &abort_flag;

  if (warp < SG_CUTTERS) {
    // ---------------- read and cut: eight lanes a row, eight entries a lane, 32 rows a step of all eight warps
    const int row = threadIdx.x >> 3, piece = threadIdx.x & 7;
    const int x_steps = (cols + 31) / 32;
    float4 wv[SG_W / 32][2], xv[SG_X / 32][2];
    auto read = [&](const float* from, int r, int limit, int k0, float4 (&v)[2]) {
      // rows past the end read the last one: what they give is not stored
      const float* at = from + (size_t)min(r, limit - 1) * k_dim + k0 + piece * 8;
      if (VEC && k0 + SG_K <= k_dim) {
        v[0] = sg_load4(at);
        v[1] = sg_load4(at + 4);
      } else {
        float e[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) e[j] = k0 + piece * 8 + j < k_dim ? at[j] : 0.f;
        v[0] = make_float4(e[0], e[1], e[2], e[3]);
        v[1] = make_float4(e[4], e[5], e[6], e[7]);
      }
    };
    auto read_w = [&](int i) {
#pragma unroll
      for (int j = 0; j < SG_W / 32; ++j) read(args.w, n_base + row + 32 * j, args.n_out, (kb_begin + i) * SG_K, wv[j]);
    };
    auto read_x = [&](int i) {
#pragma unroll
      for (int j = 0; j < SG_X / 32; ++j)
        if (j < x_steps) read(args.x, m_base + row + 32 * j, args.rows, (kb_begin + i) * SG_K, xv[j]);
    };
    uint32_t least = 0xffffffffu;
    auto file = [&](uint32_t plane, int plane_bytes, int r, const float4 (&v)[2]) {
      uint4 hi, mid, low;
      sg_cut(v[0].x, v[0].y, hi.x, mid.x, low.x);
      sg_cut(v[0].z, v[0].w, hi.y, mid.y, low.y);
      sg_cut(v[1].x, v[1].y, hi.z, mid.z, low.z);
      sg_cut(v[1].z, v[1].w, hi.w, mid.w, low.w);
      const uint32_t at = plane + r * 128 + ((piece ^ (r & 7)) << 4);
      sg_store4(at, hi);
      sg_store4(at + plane_bytes, mid);
      sg_store4(at + 2 * plane_bytes, low);
    };
    pdl_wait();
    if (n_kb > 0) {
      read_w(0);
      read_x(0);
    }
    int s = 0;
    uint32_t parity = 1;                     // (a fresh barrier's phase before the first counts as completed)
    for (int i = 0; i < n_kb; ++i) {
      if (!__all_sync(0xffffffffu, mbar_wait(&empty_bar[s], parity, abort, args.wait_limit_ns))) break;
      const uint32_t stage = smem + s * stage_bytes;
#pragma unroll
      for (int j = 0; j < SG_W / 32; ++j) {
        least = sg_least(least, wv[j]);
        file(stage, SG_W_PLANE, row + 32 * j, wv[j]);
      }
#pragma unroll
      for (int j = 0; j < SG_X / 32; ++j)
        if (row + 32 * j < cols) {
          least = sg_least(least, xv[j]);
          file(stage + 3 * SG_W_PLANE, x_plane, row + 32 * j, xv[j]);
        }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0 && (i != args.withhold || warp != 0))
        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&full_bar[s])) : "memory");
      if (i + 1 < n_kb) {                    // (behind the fence, which would wait for them)
        read_w(i + 1);
        read_x(i + 1);
      }
      if (++s == stages) { s = 0; parity ^= 1; }
    }
    if (least < SG_LEAST(63)) atomicMax(&small_flag, least < SG_LEAST(109) ? 2 : 1);
    asm volatile("barrier.sync 2, %0;" ::"n"(32 * SG_CUTTERS) : "memory");
    const int small = *(volatile int*)&small_flag;
    if (small) {
      const int k0 = kb_begin * SG_K, k1 = min((kb_begin + n_kb) * SG_K, k_dim);
      for (int r = row; r < SG_W + cols; r += 32) {                   // (whole warps: four rows, eight lanes each)
        const float* at = r < SG_W ? args.w + (size_t)min(n_base + r, args.n_out - 1) * k_dim
                                   : args.x + (size_t)min(m_base + r - SG_W, args.rows - 1) * k_dim;
        uint32_t has = small == 1 ? SG_SMALL : 0u;                    // (which rows have them is not looked for)
        for (int k = k0; k < k1; k += 64) {
          float e[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) e[j] = k + 8 * j + piece < k1 ? __ldg(at + k + 8 * j + piece) : 0.f;
#pragma unroll
          for (int j = 0; j < 8; ++j) has |= sg_note(e[j]);
          if (small == 1) {
            const uint32_t found = __ballot_sync(0xffffffffu, has & SG_ENTRIES);
            if ((found & 0xffu) && (found & 0xff00u) && (found & 0xff0000u) && (found & 0xff000000u)) break;
          }
        }
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) has |= __shfl_xor_sync(0xffffffffu, has, o);
        if (piece == 0) {
          notes[r] = has;
          atomicOr(&noted, r < SG_W ? has : has << 4);
        }
      }
    }
    if (args.parts == 1) asm volatile("barrier.sync 1, %0;" ::"n"(SG_THREADS) : "memory");      // (of a cluster: below)
  } else {
    // ---------------- add up the accumulators: a lane has one row of w, its columns are rows of x.  Two of these warps also
    // issue the MMAs, each those of one accumulator (together, one elected lane), before they empty the other: issuing
    // takes a warp longer than emptying (1,090 cycles of 1,800 a chunk when one warp issued all).
    const int quarter = warp & 3, half = (warp - SG_CUTTERS) >> 2;
    const bool issuer = quarter == 0;
    const uint32_t idesc = instr_desc(cols);
    const int n_chunks = n_kb * (SG_K / SG_CHUNK);
    int s = 0;
    uint32_t parity = 0;
    auto issue = [&](int chunk) -> bool {
      if (!__all_sync(0xffffffffu, mbar_wait(&full_bar[s], parity, abort, args.wait_limit_ns))) return false;
      if (!__all_sync(0xffffffffu, mbar_wait(&sum_empty[half], ((chunk >> 1) & 1) ^ 1, abort, args.wait_limit_ns))) return false;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t at = smem + s * stage_bytes + half * SG_CHUNK * 2;
      const uint32_t d = tmem + half * buffer_cols;
      // (formed by the whole warp, so that they are in uniform registers, as an MMA wants them)
      uint64_t wd[3], xd[3];
#pragma unroll
      for (int p = 0; p < 3; ++p) {
        wd[p] = smem_desc(at + p * SG_W_PLANE);
        xd[p] = smem_desc(at + 3 * SG_W_PLANE + p * x_plane);
      }
      if (elect_one()) {
        // the pieces of w and of x that meet, the smallest products first
        constexpr int PW[6] = {2, 0, 1, 1, 0, 0}, PX[6] = {0, 2, 1, 0, 1, 0};
#pragma unroll
        for (int t = 0; t < 6; ++t)
#pragma unroll
          for (int k = 0; k < SG_CHUNK / 16; ++k)                     // 16 entries of k are 32 bytes: 2 units
            umma_bf16(d, wd[PW[t]] + 2 * k, xd[PX[t]] + 2 * k, idesc, t > 0 || k > 0 ? 1u : 0u);
        umma_commit(&sum_full[half]);
        umma_commit(&empty_bar[s]);
      }
      __syncwarp();
      if (++s == stages) { s = 0; parity ^= 1; }
      return true;
    };
    const int r = quarter * 32 + lane;
    float sum[SG_X / 32][16];
#pragma unroll
    for (int j = 0; j < SG_X / 32; ++j)
#pragma unroll
      for (int c = 0; c < 16; ++c) sum[j][c] = 0.f;
    bool ok = !issuer || half != 0 || n_chunks == 0 || issue(0);
#pragma unroll 1
    for (int chunk = 0; ok && chunk < n_chunks; ++chunk) {
      if (issuer && ((chunk + 1) & 1) == half && chunk + 1 < n_chunks && !issue(chunk + 1)) break;
      if (!__all_sync(0xffffffffu, mbar_wait(&sum_full[chunk & 1], (chunk >> 1) & 1, abort, args.wait_limit_ns))) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t from = tmem + (chunk & 1) * buffer_cols + ((uint32_t)(quarter * 32) << 16);
#pragma unroll
      for (int j = 0; j < SG_X / 32; j += 2) {
        const int c0 = 32 * j + 16 * half;
        if (j + 1 < SG_X / 32 && c0 + 32 < cols) {
          float v[32];
          sg_tmem_load16x2(from + c0, v);
#pragma unroll
          for (int c = 0; c < 32; ++c) sum[j + c / 16][c % 16] += v[c];
        } else if (c0 < cols) {
          float v[16];
          sg_tmem_load16(from + c0, v);
#pragma unroll
          for (int c = 0; c < 16; ++c) sum[j][c] += v[c];
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&sum_empty[chunk & 1])) : "memory");
    }
    if (issuer) {
      // nothing this block issued is in flight when it leaves (it is not, unless a wait ran out)
      if (elect_one()) umma_commit(&done_bar);
      __syncwarp();
      const uint64_t start = now_ns();
      while (!mbar_try(&done_bar, 0) && now_ns() - start < TC_WAIT_LIMIT_NS) {}
    }
    if (args.parts == 1) asm volatile("barrier.sync 1, %0;" ::"n"(SG_THREADS) : "memory");      // the notes are there
    pdl_wait();                              // before the first store: an earlier kernel may still read y's memory
    const int n = n_base + r;
    if (args.parts > 1) {
      // (the ring is idle: every MMA that read it has been waited for)
#pragma unroll
      for (int j = 0; j < SG_X / 32; ++j)
#pragma unroll
        for (int c = 0; c < 16; ++c) {
          const int m = 32 * j + 16 * half + c;
          if (m < rows_here)
            asm volatile("st.shared.f32 [%0], %1;" ::"r"(smem + (m * SG_W + r) * 4), "f"(sum[j][c]) : "memory");
        }
    } else if (n < args.n_out) {
#pragma unroll
      for (int j = 0; j < SG_X / 32; ++j)
#pragma unroll
        for (int c = 0; c < 16; ++c) {
          const int m = 32 * j + 16 * half + c;
          if (m < rows_here) args.y[(size_t)(m_base + m) * args.n_out + n] = sum[j][c];
        }
      const uint32_t any = *(volatile uint32_t*)&noted;
      const bool lost = sg_cut_short(any >> 4, any), vanished = sg_vanished(any >> 4, any);      // (may be)
      bool again = lost || vanished;
#pragma unroll
      for (int j = 0; j < SG_X / 32; ++j)
#pragma unroll
        for (int c = 0; c < 16; ++c) again |= 32 * j + 16 * half + c < rows_here && sg_again(sum[j][c]);
      if (again)
#pragma unroll 1
        for (int m = 16 * half; m < rows_here; m += m % 16 == 15 ? 17 : 1) {
          float* at = args.y + (size_t)(m_base + m) * args.n_out + n;
          if (sg_again(*at) || (lost && sg_cut_short(notes[SG_W + m], notes[r])) ||
              (vanished && *at == 0.f && sg_vanished(notes[SG_W + m], notes[r])))
            *at = sg_chain(args.x + (size_t)(m_base + m) * k_dim, args.w + (size_t)n * k_dim, k_dim);
        }
    }
  }

  if (args.parts > 1) {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
    if (!*abort) {
      const bool vector_store = args.n_out % 4 == 0;
      const int n_items = rows_here * (SG_W / 4);
      uint32_t base[SG_MAX_PARTS];
      bool lost = false, vanished = false;   // (may be, in some part)
#pragma unroll
      for (int p = 0; p < SG_MAX_PARTS; ++p) {
        base[p] = 0;
        if (p < args.parts) {
          asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(base[p]) : "r"(smem), "r"(p));
          const uint32_t any = sg_remote(&noted, p);
          lost |= sg_cut_short(any >> 4, any);
          vanished |= sg_vanished(any >> 4, any);
        }
      }
      // the same of the result `v` of row m of x and row r of w
      auto short_of = [&](float v, int m, int r) -> bool {
        bool again = false;
#pragma unroll 1
        for (int p = 0; p < args.parts; ++p) {
          if (sg_remote(&noted, p) == 0) continue;
          const uint32_t x_has = sg_remote(&notes[SG_W + m], p), w_has = sg_remote(&notes[r], p);
          again |= sg_cut_short(x_has, w_has) || (v == 0.f && sg_vanished(x_has, w_has));
        }
        return again;
      };
      // an item: four neighbouring results; the loads of all parts are in flight together and are added in order
      for (int item = part * SG_THREADS + threadIdx.x; item < n_items; item += args.parts * SG_THREADS) {
        const int m = item >> 5, c = (item & 31) * 4, n = n_base + c;
        float4 v[SG_MAX_PARTS];
#pragma unroll
        for (int p = 0; p < SG_MAX_PARTS; ++p)
          if (p < args.parts)
            asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                         : "=f"(v[p].x), "=f"(v[p].y), "=f"(v[p].z), "=f"(v[p].w) : "r"(base[p] + 16 * item) : "memory");
        float e[4] = {v[0].x, v[0].y, v[0].z, v[0].w};
#pragma unroll
        for (int p = 1; p < SG_MAX_PARTS; ++p)
          if (p < args.parts) { e[0] += v[p].x; e[1] += v[p].y; e[2] += v[p].z; e[3] += v[p].w; }
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (n + j < args.n_out && (sg_again(e[j]) || ((lost || (vanished && e[j] == 0.f)) && short_of(e[j], m, c + j))))
            e[j] = sg_chain(args.x + (size_t)(m_base + m) * k_dim, args.w + (size_t)(n + j) * k_dim, k_dim);
        float* to = args.y + (size_t)(m_base + m) * args.n_out + n;
        if (vector_store) {
          if (n < args.n_out) *reinterpret_cast<float4*>(to) = make_float4(e[0], e[1], e[2], e[3]);
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (n + j < args.n_out) to[j] = e[j];
        }
      }
    }
    // no block leaves while a neighbour may still read its sums
    asm volatile("barrier.cluster.arrive.relaxed;\n\tbarrier.cluster.wait;" ::: "memory");
  }

  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == SG_CUTTERS) tmem_free(tmem, 2 * buffer_cols);
  if (threadIdx.x == 0 && abort_flag && args.status) atomicOr(args.status, 4);
}

// x [rows, k_dim] and w [n_out, k_dim] float32, y [rows, n_out].  Bit 4 of *status (if there is one) is set when a wait
// ran out.  How many parts the k range is cut into: as many as let one row of tiles run at once, each of two slices
// at least.  Clusters do not fill the SMs, whose groups are not multiples of them: how many of p blocks run at once is the
// occupancy query's answer for one block an SM.  One cluster too many is a second round: 16 tiles of 8 parts took 41 us a
// product of 141 x 2048 x 2048, of 6 parts 29.
static int sgemm_launch(const float* x, const float* w, float* y, int rows, int n_out, int k_dim, int* status, int withhold,
                        unsigned long long wait_limit_ns, cudaStream_t s) {
  if (rows == 0 || n_out == 0) return 0;
  const int tiles = (n_out + SG_W - 1) / SG_W, slices = (k_dim + SG_K - 1) / SG_K;
  static const int at_once[SG_MAX_PARTS + 1] = {0, 148, 74, 45, 33, 26, 22, 15, 15};
  int parts = SG_MAX_PARTS;
  while (parts > 1 && (at_once[parts] < tiles || 2 * parts > slices)) --parts;
  const int row_tiles = (rows - 1) / SG_X + 1;
  if ((long long)tiles * row_tiles > 0x7fffffffLL) return -2;
  SgemmArgs args;
  args.x = x; args.w = w; args.y = y; args.status = status;
  args.withhold = withhold; args.wait_limit_ns = wait_limit_ns;
  args.rows = rows; args.n_out = n_out; args.k_dim = k_dim; args.parts = parts;
  args.tile_rows = ((rows - 1) / row_tiles + 16) / 16 * 16;
  const int stage_bytes = 3 * (SG_W_PLANE + args.tile_rows * SG_K * 2);
  args.stages = (SG_SMEM - 1024) / stage_bytes;
  if (args.stages > SG_MAX_STAGES) args.stages = SG_MAX_STAGES;
  const bool vec = k_dim % 4 == 0 && ((uintptr_t)x % 16) == 0 && ((uintptr_t)w % 16) == 0;
  auto kernel = vec ? sgemm_tcgen05_kernel<true> : sgemm_tcgen05_kernel<false>;
  cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SG_SMEM);
  if (err != cudaSuccess) return (int)err;
  const int smem = args.stages * stage_bytes + 1024;
  return launch_dependent_cluster(kernel, dim3(tiles * row_tiles, parts), dim3(SG_THREADS), smem, s, dim3(1, parts, 1), args);
}

extern "C" {

int sb_sgemm_nt(const float* x, const float* w, float* y, int rows, int n_out, int k_dim, int* status, cudaStream_t s) {
  return sgemm_launch(x, w, y, rows, n_out, k_dim, status, -1, TC_WAIT_LIMIT_NS, s);
}

// The same with slice `slice` (64 entries of k) of every block's part not handed over by one of its warps: the waits on it give up
// after wait_limit_ns, the kernel returns, the status bit is set and y is undefined.  For tests.
int sb_sgemm_nt_withheld(const float* x, const float* w, float* y, int rows, int n_out, int k_dim, int* status, int slice,
                         unsigned long long wait_limit_ns, cudaStream_t s) {
  if (slice < 0 || wait_limit_ns == 0) return -2;
  return sgemm_launch(x, w, y, rows, n_out, k_dim, status, slice, wait_limit_ns, s);
}

}  // extern "C"
