// The matrix-state recurrences of state_scan.cu for steps that bring many tokens a sequence (bfloat16, states of 65 to
// 128 rows).  The walk there gives a token's state to 256 threads, eight rows of one column each: every multiply-add
// is paid for with a float from shared memory (which hands a warp 128 bytes a cycle, shared addresses or not), and a
// token's sums are a round of shuffles in the chain of the next.  Here operands stay bfloat16 in shared memory until they are
// used (cp.async brings them three stages ahead, nothing passes through registers on the way) and many tokens share a
// step of the chain.
//
//   blocks (state-space, gated delta): sixteen tokens at a time from the state S the block finds.  With G_t the
//     product of the block's decays up to token t and Gamma(t, i) from i's successor to t,
//       z_t = beta_t (v_t - G_t S^T k_t)  (state-space: v_t),   u = (I + A)^-1 z,  A(t, i) = beta_t Gamma(t, i) k_i . k_t
//       o_t = G_t S^T q_t + sum_{i <= t} Gamma(t, i) (k_i . q_t) u_i,     S <- G S + sum_i Gamma(last, i) k_i u_i^T
//     What does not involve S (the products of keys and queries, the decays, the inverse: the compact form of a product
//     of such updates, Bischof and Van Loan 1987) is one 16 x 16 matrix pair a block and head, made beforehand for
//     all blocks at once by scan_coef_kernel.  The products with S run on the tensor cores, whose other operands, keys and
//     queries, are bfloat16 as they come: S (and the write) is cut into three pieces of 8 bits, so that nothing of its 24 is
//     lost (of an entry below 2^-109 less than 2^-134; S itself is kept whole), and sums are float.  A block's G is applied as
//     S - (1 - G) S, the complement carried as such (state_scan.cu says why), and a block's write is added to S by ordinary adds.
//   walk (forget-write, channel-decay): the decay differs by row, so a token is a step; the state's update is the whole
//     chain, and read-outs of eight tokens are summed together.  A thread keeps 16 entries, so that a loaded vector serves
//     four columns.  forget-write's gates are formed beforehand (scan_gates_kernel): inside the walk every block of 16
//     columns would form them again.  32-bit multiply-adds.
// Measured at 2,048 tokens of one sequence, 16 heads of 128 x 128 (state-space: 32 of 128 x 64), few-token kernel -> here: state-space
// 577 -> 63 us (in one walk of four warps, as the delta rule's: 98), gated delta 673 -> 133, forget-write 414 -> 174,
// channel-decay 400 -> 177; unequal sequences of 801, 712 and 623 tokens: gated delta 598 -> 100, forget-write 382 -> 160,
// channel-decay 377 -> 155.  The error against 64 bits falls or stays (outputs 5.5e-7 -> 2.2e-7, 3.7e-7 -> 2.0e-7, 4.9e-8, 1.2e-7).  With one
// sequence of the delta rule an SM has four warps and the chain's latencies are the bound (about 2,000 cycles a block of sixteen).
#include <type_traits>

#include "common.cuh"

#define SP_N 128                 // rows of the state kept (N up to this; the rest are zeros)
#define SP_CT 16                 // tokens a block (and a stage)
#define SP_STAGES 3
#define SP_COLS 16               // value columns a block: four a warp
// State-space: row B (16: the block's product of queries and keys, below the diagonal), then Gamma(last, t) dt_t, G, 1 - G of the whole
// block, B's diagonal with D added.
#define SP_SCOEF 20
#define SP_COEF(DELTA) ((DELTA) ? 36 : SP_SCOEF)      // floats of a token's coefficients: W row (16, delta rule), B row (16), four scalars

typedef unsigned long long f2;
__device__ __forceinline__ f2 f2_make(float a, float b) { f2 d; asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(a), "f"(b)); return d; }
__device__ __forceinline__ f2 f2_fma(f2 a, f2 b, f2 c) { f2 d; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c)); return d; }
__device__ __forceinline__ f2 f2_mul(f2 a, f2 b) { f2 d; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
__device__ __forceinline__ float f2_sum(f2 a) {
  float x, y;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a));
  return x + y;
}
// Two bfloat16 (low half first) as floats.
__device__ __forceinline__ f2 f2_bf16(uint32_t w) { return f2_make(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u)); }
__device__ __forceinline__ f2 f2_neg(f2 a) { return a ^ 0x8000000080000000ull; }

__device__ __forceinline__ void sp_copy16(void* dst, const void* src, bool real) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  const int bytes = real ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void sp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void sp_wait_one() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }

__device__ __forceinline__ float sp_softplus(float z) { return z > 20.f ? z : log1pf(expf(z)); }

// ------------------------------------------------------------------------------------------ coefficients of the blocks
// A warp a block of sixteen tokens and up to SP_HEADS heads of one key/query group.  k . k and q . k of the block are
// 16 x 16 products of bfloat16 (exact) with float sums; lane 4 g + x holds tokens g and g + 8 (rows), entries 2 x, 2 x + 1 of both
// halves (columns).  Row (token, head) of `coef`, delta rule: [W: mk Gamma(last, t) (I + A)^-1 row t | B: row t times the inverse |
// beta, beta mk G, mq G, 1 - G of the whole block]; state-space: [B: Gamma dt_i (q_t . k_i), D added at i = t | Gamma(last, t) dt_t, 0, G,
// 1 - G of the block].
#define SP_HEADS 4
__device__ __forceinline__ void sp_mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// Two floats as the sums of three pairs of bfloat16.
__device__ __forceinline__ void sp_split(float x, float y, uint32_t (&piece)[3]) {
#pragma unroll
  for (int n = 0; n < 3; ++n) {
    const __nv_bfloat162 p = __floats2bfloat162_rn(x, y);
    const uint32_t w = *reinterpret_cast<const uint32_t*>(&p);
    piece[n] = w;
    x -= __uint_as_float(w << 16);
    y -= __uint_as_float(w & 0xffff0000u);
  }
}

__device__ __forceinline__ void sp_mma8(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
  asm("mma.sync.aligned.m16n8k8.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(b0));
}

// The sequence whose block of T tokens number `left` is (-1: none), and which of its blocks: by a whole warp, 32 sequences' block
// counts at a time.
template <int T>
__device__ __forceinline__ int sp_find_block(const int* seq_q_len, int n_seqs, int left, int lane, int& block) {
  for (int s0 = 0; s0 < n_seqs; s0 += 32) {
    const int s = s0 + lane;
    const int mine = s < n_seqs ? (seq_q_len[s] + T - 1) / T : 0;
    int upto = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += v;
    }
    const unsigned hit = __ballot_sync(0xffffffffu, left < upto);
    if (hit) {
      const int at = __ffs(hit) - 1;
      block = left - (__shfl_sync(0xffffffffu, upto, at) - __shfl_sync(0xffffffffu, mine, at));
      return s0 + at;
    }
    left -= __shfl_sync(0xffffffffu, upto, 31);
  }
  block = 0;
  return -1;
}

template <bool DELTA>
__global__ void __launch_bounds__(128)
scan_coef_kernel(const bf16* __restrict__ q, int ldq, const bf16* __restrict__ k, int ldk, const bf16* __restrict__ a_raw,
                 int lda, const bf16* __restrict__ b_raw, int ldb, const float* __restrict__ A_log,
                 const float* __restrict__ dt_bias, const float* __restrict__ D, float* __restrict__ coef,
                 const int* __restrict__ seq_q_start, const int* __restrict__ seq_q_len, int n_seqs, int H, int G, int N,
                 int per_group) {
  constexpr int COEF = SP_COEF(DELTA);
  __shared__ float sa[4][16][17], sb[4][16][17];
  pdl_wait();
  SB_BEHIND_WAIT(q); SB_BEHIND_WAIT(k); SB_BEHIND_WAIT(a_raw); SB_BEHIND_WAIT(b_raw);
  SB_BEHIND_WAIT(seq_q_start); SB_BEHIND_WAIT(seq_q_len);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int job = blockIdx.y * 4 + warp;            // (group, which SP_HEADS of its heads)
  if (job >= G * per_group) return;                 // (whole warps leave; nothing below waits for the block)
  const int group = job / per_group, h0 = group * (H / G) + (job - group * per_group) * SP_HEADS;
  const int h1 = min(h0 + SP_HEADS, (group + 1) * (H / G));
  int block;
  const int seq = sp_find_block<SP_CT>(seq_q_len, n_seqs, blockIdx.x, lane, block);
  if (seq < 0) return;
  const int first = seq_q_start[seq] + SP_CT * block, ct = min(SP_CT, seq_q_len[seq] - SP_CT * block);
  const int g = lane >> 2, x = lane & 3;
  // element (r, n, e) of a lane: token t = g + 8 r, column i = 8 n + 2 x + e
  float kk[2][4], qk[2][4], qq[2][4];               // [n][2 r + e]
#pragma unroll
  for (int n = 0; n < 2; ++n)
#pragma unroll
    for (int e = 0; e < 4; ++e) kk[n][e] = qk[n][e] = qq[n][e] = 0.f;
  // lane (g, x): 16-byte pieces x, x + 4, .. of the tokens' keys and queries; every product sees its entries in one order
  const bf16* kr[2];
  const bf16* qr[2];
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const size_t row = (size_t)(first + (g + 8 * r < ct ? g + 8 * r : 0));
    kr[r] = k + row * ldk + (size_t)group * N;
    qr[r] = q + row * ldq + (size_t)group * N;
  }
#pragma unroll
  for (int j = 0; j < SP_N / 32; ++j) {
    const int piece = x + 4 * j;
    uint4 kv[2], qv[2];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const bool have = g + 8 * r < ct && piece * 8 < N;
      kv[r] = have ? *reinterpret_cast<const uint4*>(kr[r] + piece * 8) : make_uint4(0u, 0u, 0u, 0u);
      qv[r] = have ? *reinterpret_cast<const uint4*>(qr[r] + piece * 8) : make_uint4(0u, 0u, 0u, 0u);
    }
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      sp_mma(qk[n], qv[0].x, qv[1].x, qv[0].y, qv[1].y, kv[n].x, kv[n].y);
      sp_mma(qk[n], qv[0].z, qv[1].z, qv[0].w, qv[1].w, kv[n].z, kv[n].w);
      if (DELTA) {
        sp_mma(kk[n], kv[0].x, kv[1].x, kv[0].y, kv[1].y, kv[n].x, kv[n].y);
        sp_mma(kk[n], kv[0].z, kv[1].z, kv[0].w, kv[1].w, kv[n].z, kv[n].w);
        sp_mma(qq[n], qv[0].x, qv[1].x, qv[0].y, qv[1].y, qv[n].x, qv[n].y);
        sp_mma(qq[n], qv[0].z, qv[1].z, qv[0].w, qv[1].w, qv[n].z, qv[n].w);
      }
    }
  }
  // unit norms, lane t holding token t's (t < 16): its squares lie on lane 4 (t % 8) + t % 8 / 2, entry t % 2, half t / 8
  float mk = 1.f, mq = 1.f;
  if (DELTA) {
    auto diag = [&](const float (&c)[2][4]) {
      const int j = lane & 7, from = 4 * j + (j >> 1);
      const float a = __shfl_sync(0xffffffffu, c[0][0], from), b = __shfl_sync(0xffffffffu, c[0][1], from);
      const float d = __shfl_sync(0xffffffffu, c[1][2], from), e = __shfl_sync(0xffffffffu, c[1][3], from);
      return (lane & 8) ? ((j & 1) ? e : d) : ((j & 1) ? b : a);
    };
    mk = 1.f / sqrtf(diag(kk) + 1e-6f);
    mq = rsqrtf((float)N) / sqrtf(diag(qq) + 1e-6f);
  }
  for (int h = h0; h < h1; ++h) {
    float d = 0.f, fac = 0.f;             // lane t < 16: token t's 1 - decay and its factor (dt, or beta)
    if (lane < ct) {
      const size_t row = (size_t)(first + lane);
      const float dt = sp_softplus(to_f<bf16>(a_raw[row * lda + h]) + dt_bias[h]);
      d = -expm1f(-expf(A_log[h]) * dt);
      fac = DELTA ? 1.f / (1.f + expf(-to_f<bf16>(b_raw[row * ldb + h]))) : dt;
    }
    float gam[2][4], all = 1.f, last = 1.f, gone = 0.f;    // Gamma(t, i); lane t: G_t, Gamma(end, t); 1 - G
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) gam[n][e] = 1.f;
#pragma unroll
    for (int r = 0; r < SP_CT; ++r) {
      const float dr = __shfl_sync(0xffffffffu, d, r), keep = 1.f - dr;
      gone = fmaf(-gone, dr, gone + dr);
      if (r <= lane) all *= keep;
      else last *= keep;
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (r <= g + 8 * (e >> 1) && r > 8 * n + 2 * x + (e & 1)) gam[n][e] *= keep;
    }
    float* rows = coef + ((size_t)first * H + h) * COEF;
    const size_t next = (size_t)H * COEF;
    if (!DELTA) {
      const float skip = D ? D[h] : 0.f;
#pragma unroll
      for (int n = 0; n < 2; ++n) {
        const int i0 = 8 * n + 2 * x;
        const float f0 = __shfl_sync(0xffffffffu, fac, i0), f1 = __shfl_sync(0xffffffffu, fac, i0 + 1);
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const int t = g + 8 * r;
          float2 b;
          b.x = i0 <= t ? gam[n][2 * r] * f0 * qk[n][2 * r] + (i0 == t ? skip : 0.f) : 0.f;
          b.y = i0 + 1 <= t ? gam[n][2 * r + 1] * f1 * qk[n][2 * r + 1] + (i0 + 1 == t ? skip : 0.f) : 0.f;
          if (t < ct) *reinterpret_cast<float2*>(rows + t * next + i0) = b;
        }
      }
      if (lane < ct) *reinterpret_cast<float4*>(rows + lane * next + SP_CT) = make_float4(last * fac, 0.f, all, gone);
      continue;
    }
    __syncwarp();
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int t = g + 8 * r;
      const float ft = __shfl_sync(0xffffffffu, fac * mk, t), mqt = __shfl_sync(0xffffffffu, mq, t);
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int i = 8 * n + 2 * x + e;
          const float mki = __shfl_sync(0xffffffffu, mk, i);
          sa[warp][t][i] = i < t ? ft * gam[n][2 * r + e] * mki * kk[n][2 * r + e] : 0.f;
          sb[warp][t][i] = i <= t ? mqt * gam[n][2 * r + e] * mki * qk[n][2 * r + e] : 0.f;
        }
    }
    __syncwarp();
    // column j of the inverse of I + A, by lanes j and j + 16; rows of B times it, eight by each
    const int j = lane & 15;
    float inv[SP_CT];
#pragma unroll
    for (int r = 0; r < SP_CT; ++r) {
      float s = r == j ? 1.f : 0.f;
#pragma unroll
      for (int i = 0; i < r; ++i) s = fmaf(-sa[warp][r][i], inv[i], s);
      inv[r] = r < j ? 0.f : s;
    }
    const float wt = mk * last;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int r = 8 * (lane >> 4) + e;
      float s = 0.f;
#pragma unroll
      for (int i = 0; i <= 8 + e; ++i) s = fmaf(sb[warp][r][i], i <= e || (lane >> 4) ? inv[i] : 0.f, s);
      const float own = (lane >> 4) ? inv[8 + e] : inv[e];
      const float wr = __shfl_sync(0xffffffffu, wt, e), wr8 = __shfl_sync(0xffffffffu, wt, e + 8);
      if (r < ct) {
        rows[r * next + j] = ((lane >> 4) ? wr8 : wr) * own;
        rows[r * next + SP_CT + j] = s;
      }
    }
    if (lane < ct) *reinterpret_cast<float4*>(rows + lane * next + 2 * SP_CT) = make_float4(fac, fac * mk * all, mq * all, gone);
  }
}

// ------------------------------------------------------------------------------------------ the chain of blocks
// A block of four warps owns 16 columns of one head's S for one sequence; warp w keeps rows 32 w .. 32 w + 31 as the
// accumulators of m16n8k16 products: S^T in four tiles of 16 columns x 8 rows.  Products with keys and queries, which are bfloat16,
// are exact in the tensor cores but for the float sums when the other operand is cut into three bfloat16 pieces (8 bits
// each, 24 in all): S^T k and S^T q (the tiles as they lie are the other operand's layout), and the write S^T += w^T k.  The
// warps' sums over their rows meet in shared memory; the two small products of the block (z to outputs and writes) are fmas.
// (State-space: where a walk in segments is not the faster one, scan_segments in ops.py.)
template <bool DELTA> struct BlocksStage {
  bf16 k[SP_CT][SP_N + 8], q[SP_CT][SP_N + 8], v[SP_CT][SP_COLS];
  float coef[SP_CT][SP_COEF(DELTA)];
};

__device__ __forceinline__ void sp_ldsm4(uint32_t (&r)[4], const void* p) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void sp_ldsm4_t(uint32_t (&r)[4], const void* p) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}

template <bool DELTA>
__global__ void __launch_bounds__(128)
scan_blocks_kernel(const bf16* __restrict__ q, int ldq, const bf16* __restrict__ k, int ldk, const bf16* __restrict__ v, int ldv,
                   const float* __restrict__ coef, float* __restrict__ state, long long slot_stride, float* __restrict__ out,
                   const int* __restrict__ seq_slot, const int* __restrict__ seq_q_start, const int* __restrict__ seq_q_len,
                   int H, int G, int N, int V) {
  constexpr int COEF = SP_COEF(DELTA), TOKS = DELTA ? 2 * SP_CT : SP_CT;      // read-outs a block: queries (then keys)
  constexpr int B_AT = DELTA ? SP_CT : 0, S_AT = COEF - 4;                    // places in a row of coefficients
  extern __shared__ __align__(16) unsigned char blocks_smem[];
  BlocksStage<DELTA>* stages = reinterpret_cast<BlocksStage<DELTA>*>(blocks_smem);
  __shared__ __align__(16) float part[4][TOKS][SP_COLS + 2], zs[SP_CT][SP_COLS], ws[SP_CT][SP_COLS + 4];
  pdl_wait();
  SB_BEHIND_WAIT(state); SB_BEHIND_WAIT(seq_slot); SB_BEHIND_WAIT(seq_q_start); SB_BEHIND_WAIT(seq_q_len);
  const int seq = blockIdx.x, h = blockIdx.y, col0 = blockIdx.z * SP_COLS;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, x = lane & 3;
  const int group = h / (H / G);
  const int q_start = seq_q_start[seq], q_len = seq_q_len[seq];
  float* sp = state + (size_t)seq_slot[seq] * slot_stride + (size_t)h * N * V + col0;
  // S^T tile j: entries [column g + 8 r][row 32 w + 8 j + 2 x + e] at 2 r + e
  float S[4][4];
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int n = 0; n < 4; ++n) {
      const int row = 32 * warp + 8 * j + 2 * x + (n & 1), c = g + 8 * (n >> 1);
      S[j][n] = row < N && col0 + c < V ? sp[(size_t)row * V + c] : 0.f;
    }
  const bf16* kg = k + (size_t)group * N;
  const bf16* qg = q + (size_t)group * N;
  const bf16* vh = v + (size_t)h * V + col0;
  auto load = [&](int t0) {                         // a block's operands into a stage: 16-byte pieces, zeros where nothing is
    BlocksStage<DELTA>& st = stages[t0 / SP_CT % SP_STAGES];
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      const int e = tid + 128 * n, tt = e >> 4, c = (e & 15) * 8;
      const bool real = t0 + tt < q_len && c < N;
      const size_t row = (size_t)(q_start + (real ? t0 + tt : 0));
      sp_copy16(&st.k[tt][c], kg + row * ldk + (real ? c : 0), real);
      sp_copy16(&st.q[tt][c], qg + row * ldq + (real ? c : 0), real);
    }
    if (tid < 2 * SP_CT) {
      const int tt = tid >> 1, c = (tid & 1) * 8;
      const bool real = t0 + tt < q_len && col0 + c < V;
      sp_copy16(&st.v[tt][c], vh + (size_t)(q_start + (real ? t0 + tt : 0)) * ldv + (real ? c : 0), real);
    }
    for (int e = tid; e < SP_CT * (COEF / 4); e += 128) {
      const int tt = e / (COEF / 4), c = e % (COEF / 4) * 4;
      const bool real = t0 + tt < q_len;
      sp_copy16(&st.coef[tt][c], coef + ((size_t)(q_start + (real ? t0 + tt : 0)) * H + h) * COEF + c, real);
    }
  };
  load(0);
  sp_commit();
  if (SP_CT < q_len) load(SP_CT);
  sp_commit();
  const int mi = lane >> 3;
  const int tok = tid >> 3, c2 = (tid & 7) * 2;     // the small products: a thread a token and two columns
  for (int t0 = 0; t0 < q_len; t0 += SP_CT) {
    sp_wait_one();
    __syncthreads();                                // the block's operands are there, and nobody reads the stage filled next
    if (t0 + 2 * SP_CT < q_len) load(t0 + 2 * SP_CT);
    sp_commit();
    const BlocksStage<DELTA>& st = stages[t0 / SP_CT % SP_STAGES];
    // this warp's rows of S^T q (and S^T k): columns x tokens
    float dots[TOKS / 8][4];
#pragma unroll
    for (int n = 0; n < TOKS / 8; ++n) dots[n][0] = dots[n][1] = dots[n][2] = dots[n][3] = 0.f;
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      uint32_t a[4][3];
#pragma unroll
      for (int r = 0; r < 4; ++r) sp_split(S[2 * s + (r >> 1)][2 * (r & 1)], S[2 * s + (r >> 1)][2 * (r & 1) + 1], a[r]);
      const int tt = (lane & 7) + (mi >> 1) * 8, row = 32 * warp + 16 * s + (mi & 1) * 8;
      uint32_t b[DELTA ? 2 : 1][4];
      sp_ldsm4(b[0], &st.q[tt][row]);
      if constexpr (DELTA) sp_ldsm4(b[1], &st.k[tt][row]);
#pragma unroll
      for (int p = 2; p >= 0; --p)                  // (the small pieces first)
#pragma unroll
        for (int n = 0; n < TOKS / 8; ++n)
          sp_mma(dots[n], a[0][p], a[1][p], a[2][p], a[3][p], b[n >> 1][2 * (n & 1)], b[n >> 1][2 * (n & 1) + 1]);
    }
#pragma unroll
    for (int n = 0; n < TOKS / 8; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) part[warp][8 * n + 2 * x + (e & 1)][g + 8 * (e >> 1)] = dots[n][e];
    auto update = [&](const float (&w)[8]) {        // w: [column g + 8 r][token 2 x + e + 8 u] at 4 u + 2 r + e
      uint32_t a[4][3];
#pragma unroll
      for (int r = 0; r < 4; ++r) sp_split(w[2 * r], w[2 * r + 1], a[r]);
      const float gone = st.coef[0][S_AT + 3];
      const int tt = (lane & 7) + (mi & 1) * 8;
#pragma unroll
      for (int j = 0; j < 4; j += 2) {
        uint32_t b[4];
        sp_ldsm4_t(b, &st.k[tt][32 * warp + 8 * j + (mi >> 1) * 8]);
#pragma unroll
        for (int n = 0; n < 2; ++n) {
          // (the write's own sums, added to the state by rounded adds: the tensor cores' sums are cut, not rounded, which
          // over many blocks is a drift: 2.1e-6 off in place of 5e-7 after 2,048 tokens)
          float add[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
          for (int p = 2; p >= 0; --p) sp_mma(add, a[0][p], a[1][p], a[2][p], a[3][p], b[2 * n], b[2 * n + 1]);
#pragma unroll
          for (int e = 0; e < 4; ++e) S[j + n][e] = fmaf(-gone, S[j + n][e], S[j + n][e]) + add[e];
        }
      }
    };
    if constexpr (!DELTA) {                         // what is written does not depend on what is read
      float w[8];
#pragma unroll
      for (int n = 0; n < 8; ++n) {
        const int t = 2 * x + (n & 1) + 8 * (n >> 2);
        w[n] = st.coef[t][S_AT] * to_f<bf16>(st.v[t][g + 8 * ((n >> 1) & 1)]);
      }
      update(w);
    }
    const uint32_t vv = *reinterpret_cast<const uint32_t*>(&st.v[tok][c2]);
    // Coefficients of later tokens are zero, but 0 * inf would not be: a block with a value that is not finite masks them
    // (the test rides on a barrier that is there anyway, the masked sums stand behind the usual ones: 164 us a layer of 2,048 tokens;
    // masking always, or a branch around the usual sums: 190)
    bool bad = !(fabsf(__uint_as_float(vv << 16)) < INFINITY && fabsf(__uint_as_float(vv & 0xffff0000u)) < INFINITY);
    if constexpr (DELTA) __syncthreads();           // the warps' sums are there
    else bad = __syncthreads_or(bad);
    const float4 s4 = *reinterpret_cast<const float4*>(&st.coef[tok][S_AT]);
    float2 rq = make_float2(0.f, 0.f);
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      const float2 p = *reinterpret_cast<const float2*>(&part[w][tok][c2]);
      rq.x += p.x;
      rq.y += p.y;
    }
    if constexpr (DELTA) {
      float2 rk = make_float2(0.f, 0.f);
#pragma unroll
      for (int w = 0; w < 4; ++w) {
        const float2 p = *reinterpret_cast<const float2*>(&part[w][SP_CT + tok][c2]);
        rk.x += p.x;
        rk.y += p.y;
      }
      const float2 z = make_float2(s4.x * __uint_as_float(vv << 16) - s4.y * rk.x, s4.x * __uint_as_float(vv & 0xffff0000u) - s4.y * rk.y);
      *reinterpret_cast<float2*>(&zs[tok][c2]) = z;
      bad = __syncthreads_or(!(fabsf(z.x) < INFINITY && fabsf(z.y) < INFINITY));
    }
    float2 own = make_float2(0.f, 0.f), w2 = make_float2(0.f, 0.f);
    auto small = [&](auto masked) {
#pragma unroll
      for (int i = 0; i < SP_CT; i += 4) {
        const float4 b = *reinterpret_cast<const float4*>(&st.coef[tok][B_AT + i]);
        const float bb[4] = {b.x, b.y, b.z, b.w};
        float ww[4] = {0.f, 0.f, 0.f, 0.f};
        if constexpr (DELTA) {
          const float4 w = *reinterpret_cast<const float4*>(&st.coef[tok][i]);
          ww[0] = w.x; ww[1] = w.y; ww[2] = w.z; ww[3] = w.w;
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          float2 z;
          if constexpr (DELTA) {
            z = *reinterpret_cast<const float2*>(&zs[i + e][c2]);
          } else {
            const uint32_t raw = *reinterpret_cast<const uint32_t*>(&st.v[i + e][c2]);
            z = make_float2(__uint_as_float(raw << 16), __uint_as_float(raw & 0xffff0000u));
          }
          if (decltype(masked)::value && i + e > tok) z = make_float2(0.f, 0.f);
          own.x = fmaf(bb[e], z.x, own.x);
          own.y = fmaf(bb[e], z.y, own.y);
          if constexpr (DELTA) {
            w2.x = fmaf(ww[e], z.x, w2.x);
            w2.y = fmaf(ww[e], z.y, w2.y);
          }
        }
      }
    };
    small(std::false_type{});
    if (bad) {                                      // (behind, so that the usual way has no branch in it)
      own = w2 = make_float2(0.f, 0.f);
      small(std::true_type{});
    }
    if constexpr (DELTA) *reinterpret_cast<float2*>(&ws[tok][c2]) = w2;
    if (t0 + tok < q_len && col0 + c2 < V)
      *reinterpret_cast<float2*>(out + (size_t)(q_start + t0 + tok) * H * V + (size_t)h * V + col0 + c2) =
          make_float2(fmaf(s4.z, rq.x, own.x), fmaf(s4.z, rq.y, own.y));
    if constexpr (DELTA) {
      __syncthreads();
      float w[8];
#pragma unroll
      for (int n = 0; n < 8; ++n) w[n] = ws[2 * x + (n & 1) + 8 * (n >> 2)][g + 8 * ((n >> 1) & 1)];
      update(w);
    }
  }
  pdl_trigger();
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int n = 0; n < 4; ++n) {
      const int row = 32 * warp + 8 * j + 2 * x + (n & 1), c = g + 8 * (n >> 1);
      if (row < N && col0 + c < V) sp[(size_t)row * V + c] = S[j][n];
    }
}

// ------------------------------------------------------------------------------------------ segments of blocks
// Where what a block of tokens writes does not depend on the state it finds (state-space), a segment of blocks takes S to G S + L
// with L what it writes into zeros.  So every sequence is cut into `segs` segments that are walked at once: scan_prepare_kernel
// walks all but the last without outputs and files the state a sequence starts with (place 0), the state behind its first segment
// (place 1) and the others' L (place of the next segment), beside the blocks' coefficients; scan_segments_kernel puts together the
// state its segment finds and walks it with outputs.
// A block of eight warps owns 64 columns, a warp 16 of them and half the rows: S^T as the accumulators of m16n8k16 products, eight tiles
// of 16 columns x 8 rows.  The two halves' sums over their rows meet in shared memory one step later, behind the barrier that is
// there anyway: each half keeps one half of the tokens.  Measured against one walk by four warps a head and 16 columns (us; segments):
// 2,048 tokens of 32 heads 100 -> 64 (9), of 16 heads 99 -> 45 (16); 700 of 16 heads 41 -> 23 (9); four sequences of 500 tokens and 32 heads
// 73 -> 54, eight of 400 99 -> 73 (1 each).  Few tokens or blocks that do not fill the SMs stay with one walk (64 tokens of 16 heads 9.6, here
// 12.2: two kernels of longer straight code; scan_one_walk in ops.py).  The error against 64 bits, means of 16 seeds (outputs; states;
// slow decays): 2,048 tokens of 32 heads 1.87e-7 -> 1.65e-7; 1.20e-7 the same; 2.54e-7 -> 1.73e-7; 2 x 700 of 16 heads 1.84e-7 -> 1.62e-7;
// 1.16e-7 the same; 1.80e-7 -> 1.62e-7; 200 of 32 heads 1.79e-7 -> 1.58e-7; 1.14e-7 -> 1.12e-7; 1.29e-7 -> 1.19e-7.  At nine segments the walk with outputs takes 31 of the 64 us: its products keep the tensor
// cores busy for half of that, cutting the state into pieces the issue slots for a third.
__device__ __forceinline__ int sp_span(int q_len, int segs) {       // tokens a segment: whole blocks
  const int blocks = (q_len + SP_CT - 1) / SP_CT;
  return (blocks + segs - 1) / segs * SP_CT;
}

#define SP_TILES (SP_N / 16)     // tiles of a warp's S^T
#define SP_SCOLS 64              // columns of a block
#define SP_STHREADS 256
struct __align__(16) SegmentStage {
  bf16 k[SP_CT][SP_N + 8], q[SP_CT][SP_N + 8], v[SP_CT][SP_SCOLS + 8];
  float coef[SP_CT][SP_SCOEF + 4];                  // (rows 24 floats apart: a quarter warp's pairs meet no bank twice)
};
struct __align__(16) WritesStage {
  bf16 k[SP_CT][SP_N + 8], v[SP_CT][SP_SCOLS + 8];
  float c[SP_CT], gone;          // Gamma(last, t) dt_t, 1 - G of the block
};

// The block's coefficients for a head, by a warp: q . k, a 16 x 16 product, then the decays.  (Two or four heads a warp, which
// share q . k, are slower where blocks are few: 200 tokens 16.4 us, 18.5, 24.4; 2,048 tokens 65.8, 65.7, 62.5.)
__device__ __forceinline__ void sp_pairs(const bf16* q, int ldq, const bf16* k, int ldk, const bf16* a_raw, int lda, const float* A_log,
                                         const float* dt_bias, const float* D, float* coef, const int* seq_q_start,
                                         const int* seq_q_len, int n_seqs, int H, int G, int N, int number) {
  const int lane = threadIdx.x & 31;
  const int at = number / H, h = number - at * H, group = h / (H / G);
  int block;
  const int seq = sp_find_block<SP_CT>(seq_q_len, n_seqs, at, lane, block);
  if (seq < 0) return;
  const int first = seq_q_start[seq] + SP_CT * block, ct = min(SP_CT, seq_q_len[seq] - SP_CT * block);
  const int g = lane >> 2, x = lane & 3;
  const float raw = lane < ct ? to_f<bf16>(a_raw[(size_t)(first + lane) * lda + h]) : 0.f;
  // element (r, n, e) of a lane: token t = g + 8 r, column i = 8 n + 2 x + e
  float qk[2][4];                                   // [n][2 r + e]
#pragma unroll
  for (int n = 0; n < 2; ++n) qk[n][0] = qk[n][1] = qk[n][2] = qk[n][3] = 0.f;
  // lane (g, x): 16-byte pieces x, x + 4, .. of the tokens' keys and queries; every product sees its entries in one order
  uint4 kv[SP_N / 32][2], qv[SP_N / 32][2];
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const size_t row = (size_t)(first + (g + 8 * r < ct ? g + 8 * r : 0));
#pragma unroll
    for (int j = 0; j < SP_N / 32; ++j) {
      const int piece = x + 4 * j;
      const bool have = g + 8 * r < ct && piece * 8 < N;
      kv[j][r] = have ? *reinterpret_cast<const uint4*>(k + row * ldk + (size_t)group * N + piece * 8) : make_uint4(0u, 0u, 0u, 0u);
      qv[j][r] = have ? *reinterpret_cast<const uint4*>(q + row * ldq + (size_t)group * N + piece * 8) : make_uint4(0u, 0u, 0u, 0u);
    }
  }
#pragma unroll
  for (int j = 0; j < SP_N / 32; ++j)
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      sp_mma(qk[n], qv[j][0].x, qv[j][1].x, qv[j][0].y, qv[j][1].y, kv[j][n].x, kv[j][n].y);
      sp_mma(qk[n], qv[j][0].z, qv[j][1].z, qv[j][0].w, qv[j][1].w, kv[j][n].z, kv[j][n].w);
    }
  float d = 0.f, dt = 0.f;                          // lane t < 16: token t's 1 - decay and dt
  if (lane < ct) {
    dt = sp_softplus(raw + dt_bias[h]);
    d = -expm1f(-expf(A_log[h]) * dt);
  }
  float gam[2][4], all = 1.f, last = 1.f, gone = 0.f;       // Gamma(t, i); lane t: G_t, Gamma(end, t); 1 - G
#pragma unroll
  for (int n = 0; n < 2; ++n)
#pragma unroll
    for (int e = 0; e < 4; ++e) gam[n][e] = 1.f;
#pragma unroll
  for (int r = 0; r < SP_CT; ++r) {
    const float dr = __shfl_sync(0xffffffffu, d, r), keep = 1.f - dr;
    gone = fmaf(-gone, dr, gone + dr);
    if (r <= lane) all *= keep;
    else last *= keep;
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (r <= g + 8 * (e >> 1) && r > 8 * n + 2 * x + (e & 1)) gam[n][e] *= keep;
  }
  float* rows = coef + ((size_t)first * H + h) * SP_SCOEF;
  const size_t next = (size_t)H * SP_SCOEF;
  const float skip = D ? D[h] : 0.f;
#pragma unroll
  for (int n = 0; n < 2; ++n) {
    const int i0 = 8 * n + 2 * x;
    const float f0 = __shfl_sync(0xffffffffu, dt, i0), f1 = __shfl_sync(0xffffffffu, dt, i0 + 1);
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int t = g + 8 * r;
      float2 b;
      b.x = i0 < t ? gam[n][2 * r] * f0 * qk[n][2 * r] : 0.f;
      b.y = i0 + 1 < t ? gam[n][2 * r + 1] * f1 * qk[n][2 * r + 1] : 0.f;
      if (i0 == t && t < ct) rows[t * next + SP_SCOEF - 1] = f0 * qk[n][2 * r] + skip;
      if (i0 + 1 == t && t < ct) rows[t * next + SP_SCOEF - 1] = f1 * qk[n][2 * r + 1] + skip;
      if (t < ct) *reinterpret_cast<float2*>(rows + t * next + i0) = b;
    }
  }
  if (lane < ct) {
    *reinterpret_cast<float2*>(rows + lane * next + SP_CT) = make_float2(last * dt, all);
    rows[lane * next + SP_CT + 2] = gone;
  }
}

// Sixteen tokens' values of a warp's columns as the A operand [column g + 8 (r & 1)][tokens 2 x + 8 (r >> 1) and the next].
__device__ __forceinline__ void sp_values(uint32_t (&va)[4], const bf16 (*v)[SP_SCOLS + 8], int cw, int lane) {
  sp_ldsm4_t(va, &v[(lane & 7) + (lane >> 4) * 8][16 * cw + (lane >> 3 & 1) * 8]);
}

// S <- S - gone S + sum over the block's tokens of k_t (c_t v_t)^T, c_t at c[LD t].
template <int LD>
__device__ __forceinline__ void sp_write(float (&S)[SP_TILES][4], const uint32_t (&va)[4], const float* c, float gone,
                                         const bf16 (*k)[SP_N + 8], int row0, int lane) {
  const int x = lane & 3;
  uint32_t a[4][3];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const float c0 = c[LD * (8 * h + 2 * x)], c1 = c[LD * (8 * h + 2 * x + 1)];
#pragma unroll
    for (int r = 2 * h; r < 2 * h + 2; ++r)
      sp_split(c0 * __uint_as_float(va[r] << 16), c1 * __uint_as_float(va[r] & 0xffff0000u), a[r]);
  }
  const int tt = (lane & 7) + (lane >> 3 & 1) * 8;
#pragma unroll
  for (int j = 0; j < SP_TILES; j += 4) {           // (four products side by side)
    uint32_t b[2][4];
    sp_ldsm4_t(b[0], &k[tt][row0 + 8 * j + (lane >> 4) * 8]);
    sp_ldsm4_t(b[1], &k[tt][row0 + 8 * j + 16 + (lane >> 4) * 8]);
    // (the write's own sums, added to the state by rounded adds: the tensor cores' sums are cut, not rounded, which over many
    // blocks is a drift: 2.1e-6 off in place of 5e-7 after 2,048 tokens)
    float add[4][4];
#pragma unroll
    for (int n = 0; n < 4; ++n) add[n][0] = add[n][1] = add[n][2] = add[n][3] = 0.f;
#pragma unroll
    for (int p = 2; p >= 0; --p)
#pragma unroll
      for (int n = 0; n < 4; ++n) sp_mma(add[n], a[0][p], a[1][p], a[2][p], a[3][p], b[n >> 1][2 * (n & 1)], b[n >> 1][2 * (n & 1) + 1]);
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) S[j + n][e] = fmaf(-gone, S[j + n][e], S[j + n][e]) + add[n][e];
  }
}

// The first `writers` blocks walk the segments' writes, the others' warps make the coefficients of a block and its heads each: neither
// needs the other, so they run side by side.
__global__ void __launch_bounds__(SP_STHREADS, 2)
scan_prepare_kernel(const bf16* __restrict__ q, int ldq, const bf16* __restrict__ k, int ldk, const bf16* __restrict__ v, int ldv,
                    const bf16* __restrict__ a_raw, int lda, const float* __restrict__ A_log, const float* __restrict__ dt_bias,
                    const float* __restrict__ D, float* __restrict__ coef, const float* __restrict__ state, long long slot_stride,
                    const int* __restrict__ seq_slot, const int* __restrict__ seq_q_start, const int* __restrict__ seq_q_len,
                    int n_seqs, int H, int G, int N, int V, int segs, int writers, float4* __restrict__ carried,
                    float* __restrict__ keeps) {
  constexpr int T = SP_STHREADS;
  extern __shared__ __align__(16) unsigned char writes_smem[];
  WritesStage* stages = reinterpret_cast<WritesStage*>(writes_smem);
  __shared__ float dt_of[T / 32];
  pdl_wait();
  SB_BEHIND_WAIT(q); SB_BEHIND_WAIT(k); SB_BEHIND_WAIT(a_raw); SB_BEHIND_WAIT(state);
  SB_BEHIND_WAIT(seq_slot); SB_BEHIND_WAIT(seq_q_start); SB_BEHIND_WAIT(seq_q_len);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, x = lane & 3;
  if ((int)blockIdx.x >= writers) {
    sp_pairs(q, ldq, k, ldk, a_raw, lda, A_log, dt_bias, D, coef, seq_q_start, seq_q_len, n_seqs, H, G, N,
             (blockIdx.x - writers) * (T / 32) + warp);
    return;
  }
  const int z = (V + SP_SCOLS - 1) / SP_SCOLS;
  int rest = blockIdx.x / z;
  const int zi = blockIdx.x - rest * z, h = rest % H;
  rest /= H;
  const int seq = rest / (segs - 1), seg = rest - seq * (segs - 1), col0 = zi * SP_SCOLS;
  const int cw = warp & 3, row0 = (warp >> 2) * (SP_N / 2);      // the warp's columns and rows
  const int group = h / (H / G);
  const int q_start = seq_q_start[seq], all_len = seq_q_len[seq], span = sp_span(all_len, segs), t_first = seg * span;
  const bool last = t_first + span >= all_len;      // nobody starts behind it
  if (last && seg > 0) return;
  const int q_len = last ? t_first : t_first + span;
  float4* to = carried + ((((size_t)seq * H + h) * z + zi) * segs) * (SP_TILES * T) + tid;
  float S[SP_TILES][4], dt_mine = 0.f;
#pragma unroll
  for (int j = 0; j < SP_TILES; ++j) S[j][0] = S[j][1] = S[j][2] = S[j][3] = 0.f;
  if (seg == 0) {
    const float* sp = state + (size_t)seq_slot[seq] * slot_stride + (size_t)h * N * V;
#pragma unroll
    for (int j = 0; j < SP_TILES; ++j)
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        const int row = row0 + 8 * j + 2 * x + (n & 1), c = col0 + 16 * cw + g + 8 * (n >> 1);
        if (row < N && c < V) S[j][n] = sp[(size_t)row * V + c];
      }
#pragma unroll
    for (int j = 0; j < SP_TILES; ++j) to[j * T] = make_float4(S[j][0], S[j][1], S[j][2], S[j][3]);
    if (last) return;
  }
  // Lane t < 16 of a warp makes token t's factor Gamma(last, t) dt_t; the warps take turns at it, one step ahead.
  const float decay = expf(A_log[h]), bias = dt_bias[h];
  auto factors = [&](int t0) {
    WritesStage& st = stages[t0 / SP_CT % SP_STAGES];
    float dt = 0.f, d = 0.f;
    if (lane < SP_CT && t0 + lane < q_len) {
      dt = sp_softplus(to_f<bf16>(a_raw[(size_t)(q_start + t0 + lane) * lda + h]) + bias);
      d = -expm1f(-decay * dt);
    }
    float suf = 1.f - d, gone = d;                  // the products and the complement from this token to the last
#pragma unroll
    for (int o = 1; o < SP_CT; o <<= 1) {
      const float s2 = __shfl_down_sync(0xffffffffu, suf, o), g2 = __shfl_down_sync(0xffffffffu, gone, o);
      if (lane + o < SP_CT) {
        suf *= s2;
        gone = fmaf(-gone, g2, gone + g2);
      }
    }
    const float behind = __shfl_down_sync(0xffffffffu, suf, 1);
    if (lane < SP_CT) st.c[lane] = dt * (lane < SP_CT - 1 ? behind : 1.f);
    if (lane == 0) st.gone = gone;
    dt_mine += dt;
  };
  const bf16* kg = k + (size_t)group * N;
  const bf16* vh = v + (size_t)h * V + col0;
  auto load = [&](int t0) {
    WritesStage& st = stages[t0 / SP_CT % SP_STAGES];
#pragma unroll
    for (int e = tid; e < SP_CT * SP_N / 8; e += T) {
      const int tt = e >> 4, c = (e & 15) * 8;
      const bool real = t0 + tt < q_len && c < N;
      sp_copy16(&st.k[tt][c], kg + (size_t)(q_start + (real ? t0 + tt : 0)) * ldk + (real ? c : 0), real);
    }
    if (tid < SP_CT * SP_SCOLS / 8) {
      const int tt = tid >> 3, c = (tid & 7) * 8;
      const bool real = t0 + tt < q_len && col0 + c < V;
      sp_copy16(&st.v[tt][c], vh + (size_t)(q_start + (real ? t0 + tt : 0)) * ldv + (real ? c : 0), real);
    }
  };
  load(t_first);
  sp_commit();
  if (t_first + SP_CT < q_len) load(t_first + SP_CT);
  sp_commit();
  if (warp == 0) factors(t_first);
  for (int t0 = t_first; t0 < q_len; t0 += SP_CT) {
    sp_wait_one();
    __syncthreads();                                // the block's operands are there, and nobody reads the stage filled next
    if (t0 + 2 * SP_CT < q_len) load(t0 + 2 * SP_CT);
    sp_commit();
    const WritesStage& st = stages[t0 / SP_CT % SP_STAGES];
    uint32_t va[4];
    sp_values(va, st.v, cw, lane);
    if (t0 + SP_CT < q_len && warp == (t0 / SP_CT + 1) % (T / 32)) factors(t0 + SP_CT);
    if (t0 + SP_CT >= q_len) {                      // (the factors are made: their exponents' sum, beside the last products)
      const float sum = warp_sum(dt_mine);
      if (lane == 0) dt_of[warp] = sum;
    }
    sp_write<1>(S, va, st.c, st.gone, st.k, row0, lane);
  }
  pdl_trigger();
#pragma unroll
  for (int j = 0; j < SP_TILES; ++j) to[((seg + 1) * SP_TILES + j) * T] = make_float4(S[j][0], S[j][1], S[j][2], S[j][3]);
  // What the segment leaves of the state it finds, from the sum of its exponents: products of complements, which every block would round
  // again, had the states 1.158e-7 off after 200 tokens in four segments (one walk 1.138e-7, this 1.118e-7).
  if (zi > 0) return;
  __syncthreads();
  if (tid == 0) {
    float x = 0.f;
    for (int w = 0; w < T / 32; ++w) x += dt_of[w];
    keeps[((size_t)seq * H + h) * segs + seg] = expf(-decay * x);
  }
}

__global__ void __launch_bounds__(SP_STHREADS, 2)
scan_segments_kernel(const bf16* __restrict__ q, int ldq, const bf16* __restrict__ k, int ldk, const bf16* __restrict__ v, int ldv,
                     const float* __restrict__ coef, float* __restrict__ state, long long slot_stride, float* __restrict__ out,
                     const int* __restrict__ seq_slot, const int* __restrict__ seq_q_start, const int* __restrict__ seq_q_len,
                     int H, int G, int N, int V, int segs, const float4* __restrict__ carried, const float* __restrict__ keeps) {
  constexpr int T = SP_STHREADS;
  extern __shared__ __align__(16) unsigned char segments_smem[];
  SegmentStage* stages = reinterpret_cast<SegmentStage*>(segments_smem);
  __shared__ __align__(16) float4 part[2][8][32];
  pdl_wait();
  SB_BEHIND_WAIT(state); SB_BEHIND_WAIT(seq_slot); SB_BEHIND_WAIT(seq_q_start); SB_BEHIND_WAIT(seq_q_len);
  SB_BEHIND_WAIT(carried); SB_BEHIND_WAIT(keeps);
  const int seq = blockIdx.x / segs, seg = blockIdx.x - seq * segs, h = blockIdx.y, col0 = blockIdx.z * SP_SCOLS;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, x = lane & 3;
  const int cw = warp & 3, row0 = (warp >> 2) * (SP_N / 2);      // the warp's columns and rows
  const int group = h / (H / G);
  const int q_start = seq_q_start[seq], all_len = seq_q_len[seq], span = sp_span(all_len, segs), t_first = seg * span;
  if (t_first >= all_len && seg > 0) return;
  const int q_len = min(all_len, t_first + span);   // the segment's tokens: t_first up to here
  const bf16* kg = k + (size_t)group * N;
  const bf16* qg = q + (size_t)group * N;
  const bf16* vh = v + (size_t)h * V + col0;
  auto load = [&](int t0) {                         // a block's operands into a stage: 16-byte pieces, zeros where nothing is
    SegmentStage& st = stages[t0 / SP_CT % SP_STAGES];
#pragma unroll
    for (int e = tid; e < SP_CT * SP_N / 8; e += T) {
      const int tt = e >> 4, c = (e & 15) * 8;
      const bool real = t0 + tt < q_len && c < N;
      const size_t row = (size_t)(q_start + (real ? t0 + tt : 0));
      sp_copy16(&st.k[tt][c], kg + row * ldk + (real ? c : 0), real);
      sp_copy16(&st.q[tt][c], qg + row * ldq + (real ? c : 0), real);
    }
    if (tid < SP_CT * SP_SCOLS / 8) {
      const int tt = tid >> 3, c = (tid & 7) * 8;
      const bool real = t0 + tt < q_len && col0 + c < V;
      sp_copy16(&st.v[tt][c], vh + (size_t)(q_start + (real ? t0 + tt : 0)) * ldv + (real ? c : 0), real);
    } else if (tid < SP_CT * SP_SCOLS / 8 + SP_CT * SP_SCOEF / 4) {
      const int e = tid - SP_CT * SP_SCOLS / 8, tt = e / (SP_SCOEF / 4), c = e % (SP_SCOEF / 4) * 4;
      const bool real = t0 + tt < q_len;
      sp_copy16(&st.coef[tt][c], coef + ((size_t)(q_start + (real ? t0 + tt : 0)) * H + h) * SP_SCOEF + c, real);
    }
  };
  load(t_first);
  sp_commit();
  if (t_first + SP_CT < q_len) load(t_first + SP_CT);
  sp_commit();
  // S^T tile j: entries [column g + 8 r][row 8 j + 2 x + e] at 2 r + e
  float* sp = state + (size_t)seq_slot[seq] * slot_stride + (size_t)h * N * V;
  float S[SP_TILES][4];
  if (segs == 1) {
#pragma unroll
    for (int j = 0; j < SP_TILES; ++j)
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        const int row = row0 + 8 * j + 2 * x + (n & 1), c = col0 + 16 * cw + g + 8 * (n >> 1);
        S[j][n] = row < N && c < V ? sp[(size_t)row * V + c] : 0.f;
      }
  } else {
    const float4* from = carried + ((((size_t)seq * H + h) * gridDim.z + blockIdx.z) * segs) * (SP_TILES * T) + tid;
    const float* kept = keeps + ((size_t)seq * H + h) * segs;
    const int p0 = seg == 0 ? 0 : 1;
#pragma unroll
    for (int j = 0; j < SP_TILES; ++j) {
      const float4 e = from[(p0 * SP_TILES + j) * T];
      S[j][0] = e.x; S[j][1] = e.y; S[j][2] = e.z; S[j][3] = e.w;
    }
    for (int p = 2; p <= seg; ++p) {
      const float d = kept[p - 1];
#pragma unroll
      for (int j = 0; j < SP_TILES; ++j) {
        const float4 e = from[(p * SP_TILES + j) * T];
        S[j][0] = fmaf(d, S[j][0], e.x);
        S[j][1] = fmaf(d, S[j][1], e.y);
        S[j][2] = fmaf(d, S[j][2], e.z);
        S[j][3] = fmaf(d, S[j][3], e.w);
      }
    }
  }
  const int half = warp >> 2;
  float own[4] = {0.f, 0.f, 0.f, 0.f};              // [column g + 8 r][token 8 half + 2 x + e] at 2 r + e
  auto finish = [&](int t0) {                       // the outputs of the block at t0
    const float4 p = part[t0 / SP_CT & 1][warp ^ 4][lane];
    const float o[4] = {own[0] + p.x, own[1] + p.y, own[2] + p.z, own[3] + p.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int t = t0 + 8 * half + 2 * x + (e & 1), col = col0 + 16 * cw + g + 8 * (e >> 1);
      if (t < q_len && col < V) out[(size_t)(q_start + t) * H * V + (size_t)h * V + col] = o[e];
    }
  };
  for (int t0 = t_first; t0 < q_len; t0 += SP_CT) {
    sp_wait_one();
    __syncthreads();                                // the block's operands are there, and nobody reads the stage filled next
    if (t0 + 2 * SP_CT < q_len) load(t0 + 2 * SP_CT);
    sp_commit();
    const SegmentStage& st = stages[t0 / SP_CT % SP_STAGES];
    if (t0 > t_first) finish(t0 - SP_CT);           // the block before: what the other half found lies behind this step's barrier
    // S^T q of the warp's rows, 32 rows' sums at a time: [column g + 8 r][token 8 n + 2 x + e]
    float dots[2][4];
#pragma unroll
    for (int s2 = 0; s2 < SP_N / 64; ++s2) {
      uint32_t a[2][4][3], b[2][4];
#pragma unroll
      for (int s = 0; s < 2; ++s) {
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const float* from = S[2 * (2 * s2 + s) + (r >> 1)] + 2 * (r & 1);
          sp_split(from[0], from[1], a[s][r]);
        }
        sp_ldsm4(b[s], &st.q[(lane & 7) + (lane >> 4) * 8][row0 + 16 * (2 * s2 + s) + (lane >> 3 & 1) * 8]);
      }
      float d[2][4];
#pragma unroll
      for (int n = 0; n < 2; ++n) d[n][0] = d[n][1] = d[n][2] = d[n][3] = 0.f;
#pragma unroll
      for (int p = 2; p >= 0; --p)                  // (all small pieces first: only two sums are cut at the result's size)
#pragma unroll
        for (int s = 0; s < 2; ++s)
#pragma unroll
          for (int n = 0; n < 2; ++n) sp_mma(d[n], a[s][0][p], a[s][1][p], a[s][2][p], a[s][3][p], b[s][2 * n], b[s][2 * n + 1]);
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) dots[n][e] = s2 ? dots[n][e] + d[n][e] : d[n][e];
    }
    uint32_t va[4];
    sp_values(va, st.v, cw, lane);
    sp_write<SP_SCOEF + 4>(S, va, &st.coef[0][SP_CT], st.coef[0][SP_CT + 2], st.k, row0, lane);
    // What the block's own tokens add, for this half's eight.  Coefficients of later tokens are zero, but 0 * inf would not be: values
    // that are not finite are left out of the product and added behind it, to their own and later tokens.
    bool bad = false;
#pragma unroll
    for (int r = 0; r < 4; ++r) bad |= (va[r] & 0x7f80u) == 0x7f80u || (va[r] & 0x7f800000u) == 0x7f800000u;
    bad = __any_sync(0xffffffffu, bad);
    if (bad) {
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        if ((va[r] & 0x7f80u) == 0x7f80u) va[r] &= 0xffff0000u;
        if ((va[r] & 0x7f800000u) == 0x7f800000u) va[r] &= 0xffffu;
      }
    }
    uint32_t b0[3], b1[3];
    const float2 w0 = *reinterpret_cast<const float2*>(&st.coef[8 * half + g][2 * x]);
    const float2 w1 = *reinterpret_cast<const float2*>(&st.coef[8 * half + g][2 * x + 8]);
    sp_split(w0.x, w0.y, b0);
    sp_split(w1.x, w1.y, b1);
    // (the large pieces' products in two sums of eight, added by rounded adds)
    float small[4] = {0.f, 0.f, 0.f, 0.f}, late[4] = {0.f, 0.f, 0.f, 0.f};
    own[0] = own[1] = own[2] = own[3] = 0.f;
    sp_mma(small, va[0], va[1], va[2], va[3], b0[2], b1[2]);
    sp_mma(small, va[0], va[1], va[2], va[3], b0[1], b1[1]);
    sp_mma8(own, va[0], va[1], b0[0]);
    sp_mma8(late, va[2], va[3], b1[0]);
    float mine[4], theirs[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int t = 8 * half + 2 * x + (e & 1);
      own[e] = fmaf(st.coef[t][SP_CT + 3], to_f<bf16>(st.v[t][16 * cw + g + 8 * (e >> 1)]), (own[e] + late[e]) + small[e]);
      mine[e] = half ? dots[1][e] : dots[0][e];
      theirs[e] = half ? dots[0][e] : dots[1][e];
    }
    if (bad) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int t = 8 * half + 2 * x + (e & 1);
        for (int i = 0; i < t; ++i) {
          const float value = to_f<bf16>(st.v[i][16 * cw + g + 8 * (e >> 1)]);
          if (!(fabsf(value) < INFINITY)) own[e] += st.coef[t][i] * value;
        }
      }
    }
    const float m0 = st.coef[8 * half + 2 * x][SP_CT + 1], m1 = st.coef[8 * half + 2 * x + 1][SP_CT + 1];
    const float o0 = st.coef[8 - 8 * half + 2 * x][SP_CT + 1], o1 = st.coef[8 - 8 * half + 2 * x + 1][SP_CT + 1];
#pragma unroll
    for (int e = 0; e < 4; ++e) own[e] = fmaf(e & 1 ? m1 : m0, mine[e], own[e]);
    part[t0 / SP_CT & 1][warp][lane] = make_float4(o0 * theirs[0], o1 * theirs[1], o0 * theirs[2], o1 * theirs[3]);
  }
  if (q_len > t_first) {
    __syncthreads();
    finish((q_len - 1) / SP_CT * SP_CT);
  }
  pdl_trigger();
  if (q_len < all_len) return;                      // (the sequence's last segment files the state)
#pragma unroll
  for (int j = 0; j < SP_TILES; ++j)
#pragma unroll
    for (int n = 0; n < 4; ++n) {
      const int row = row0 + 8 * j + 2 * x + (n & 1), c = col0 + 16 * cw + g + 8 * (n >> 1);
      if (row < N && c < V) sp[(size_t)row * V + c] = S[j][n];
    }
}

// ------------------------------------------------------------------------------------------ a decay per row
// qf = silu(q), d = (1 - lower) sigmoid(-(z + bias)): a thread eight channels of a token (blockIdx.x: a step may bring more
// tokens than the grid's other dimensions count to).
__global__ void __launch_bounds__(256)
scan_gates_kernel(const bf16* __restrict__ q, int ldq, const bf16* __restrict__ z, int ldz, const float* __restrict__ lower,
                  const float* __restrict__ bias, float* __restrict__ qf, float* __restrict__ d, int channels, int wide) {
  const int c = (blockIdx.y * 256 + threadIdx.x) * 8;
  alignas(16) float lo[8], bi[8];                   // (weights: ahead of the wait, in 16-byte loads where they may be)
  if (c < channels) {
    if (wide) {
#pragma unroll
      for (int i = 0; i < 8; i += 4) {
        *reinterpret_cast<float4*>(lo + i) = *reinterpret_cast<const float4*>(lower + c + i);
        *reinterpret_cast<float4*>(bi + i) = *reinterpret_cast<const float4*>(bias + c + i);
      }
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        lo[i] = lower[c + i];
        bi[i] = bias[c + i];
      }
    }
  }
  pdl_wait();
  SB_BEHIND_WAIT(q); SB_BEHIND_WAIT(z);
  if (c >= channels) return;
  const size_t row = blockIdx.x;
  const uint4 qv = *reinterpret_cast<const uint4*>(q + row * ldq + c), zv = *reinterpret_cast<const uint4*>(z + row * ldz + c);
  const uint32_t qw[4] = {qv.x, qv.y, qv.z, qv.w}, zw[4] = {zv.x, zv.y, zv.z, zv.w};
  float a[8], g[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float qe = __uint_as_float(i & 1 ? qw[i / 2] & 0xffff0000u : qw[i / 2] << 16);
    const float ze = __uint_as_float(i & 1 ? zw[i / 2] & 0xffff0000u : zw[i / 2] << 16);
    a[i] = qe / (1.f + expf(-qe));
    g[i] = (1.f - lo[i]) / (1.f + expf(ze + bi[i]));
  }
  float4* qo = reinterpret_cast<float4*>(qf + row * channels + c);
  float4* go = reinterpret_cast<float4*>(d + row * channels + c);
  qo[0] = make_float4(a[0], a[1], a[2], a[3]);
  qo[1] = make_float4(a[4], a[5], a[6], a[7]);
  go[0] = make_float4(g[0], g[1], g[2], g[3]);
  go[1] = make_float4(g[4], g[5], g[6], g[7]);
}

// A block of four warps owns 16 columns; a lane keeps rows 4 l .. 4 l + 3 of its warp's four columns.  FORGET: q (silu
// applied) and d as floats, S <- S + d (v - S); else q and k as bfloat16, d as floats, S <- S - d S + k v, o times q_mult.
struct ForgetStage {
  float q[SP_CT][SP_N], d[SP_CT][SP_N];
  bf16 v[SP_CT][SP_COLS];
};
struct DecayStage {
  bf16 q[SP_CT][SP_N], k[SP_CT][SP_N];
  float d[SP_CT][SP_N];
  bf16 v[SP_CT][SP_COLS];
};
template <bool FORGET> struct RowStage { typedef DecayStage type; };
template <> struct RowStage<true> { typedef ForgetStage type; };

template <bool FORGET>
__global__ void __launch_bounds__(128, 3)
scan_rows_kernel(const void* __restrict__ q, int ldq, const bf16* __restrict__ k, int ldk, const bf16* __restrict__ v, int ldv,
                 const float* __restrict__ d, float* __restrict__ state, long long slot_stride, float* __restrict__ out,
                 const int* __restrict__ seq_slot, const int* __restrict__ seq_q_start, const int* __restrict__ seq_q_len,
                 int H, int N, int V) {
  typedef typename RowStage<FORGET>::type Stage;
  extern __shared__ __align__(16) unsigned char rows_smem[];
  Stage* stages = reinterpret_cast<Stage*>(rows_smem);
  pdl_wait();
  SB_BEHIND_WAIT(state); SB_BEHIND_WAIT(seq_slot); SB_BEHIND_WAIT(seq_q_start); SB_BEHIND_WAIT(seq_q_len);
  const int seq = blockIdx.x, h = blockIdx.y, col0 = blockIdx.z * SP_COLS;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int q_start = seq_q_start[seq], q_len = seq_q_len[seq];
  const int col = col0 + 4 * warp;
  const bool in = col < V;                          // (the warp's four columns: inside or outside together)
  float* sp = state + (size_t)seq_slot[seq] * slot_stride + (size_t)h * N * V;
  f2 S[2][4];                                       // rows 4 l + 2 r and the next
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    float e[2][4];
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      const int row = 4 * lane + 2 * r + x;
#pragma unroll
      for (int c = 0; c < 4; ++c) e[x][c] = in && row < N ? sp[(size_t)row * V + col + c] : 0.f;
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) S[r][c] = f2_make(e[0][c], e[1][c]);
  }
  const size_t ld_rows = (size_t)H * N;
  auto load = [&](int t0) {
    Stage& st = stages[t0 / SP_CT % SP_STAGES];
#pragma unroll
    for (int n = 0; n < 4; ++n) {                   // floats: 32 pieces a row
      const int e = tid + 128 * n, tt = e >> 5, c = (e & 31) * 4;
      const bool real = t0 + tt < q_len && c < N;
      const size_t at = (size_t)(q_start + (real ? t0 + tt : 0)) * ld_rows + (size_t)h * N + (real ? c : 0);
      sp_copy16(&st.d[tt][c], d + at, real);
      if constexpr (FORGET) sp_copy16(&st.q[tt][c], static_cast<const float*>(q) + at, real);
    }
    if constexpr (!FORGET) {
#pragma unroll
      for (int n = 0; n < 2; ++n) {
        const int e = tid + 128 * n, tt = e >> 4, c = (e & 15) * 8;
        const bool real = t0 + tt < q_len && c < N;
        const size_t row = (size_t)(q_start + (real ? t0 + tt : 0));
        sp_copy16(&st.q[tt][c], static_cast<const bf16*>(q) + row * ldq + (size_t)h * N + (real ? c : 0), real);
        sp_copy16(&st.k[tt][c], k + row * ldk + (size_t)h * N + (real ? c : 0), real);
      }
    }
    if (tid < 2 * SP_CT) {
      const int tt = tid >> 1, c = (tid & 1) * 8;
      const bool real = t0 + tt < q_len && col0 + c < V;
      sp_copy16(&st.v[tt][c], v + (size_t)(q_start + (real ? t0 + tt : 0)) * ldv + (size_t)h * V + (real ? col0 + c : 0), real);
    }
  };
  const float q_mult = FORGET ? 1.f : 1.f / sqrtf((float)N);
  const f2 minus = f2_make(-1.f, -1.f);
  load(0);
  sp_commit();
  if (SP_CT < q_len) load(SP_CT);
  sp_commit();
  for (int t0 = 0; t0 < q_len; t0 += SP_CT) {
    sp_wait_one();
    __syncthreads();                                // the chunk is there, and nobody reads the stage filled next
    if (t0 + 2 * SP_CT < q_len) load(t0 + 2 * SP_CT);
    sp_commit();
    const Stage& st = stages[t0 / SP_CT % SP_STAGES];
#pragma unroll 1
    for (int b = 0; b < SP_CT && t0 + b < q_len; b += 8) {
      // (tokens past the sequence's end were filed as zeros: they neither decay nor write)
      float part[32];
#pragma unroll
      for (int t = 0; t < 8; ++t) {
        const uint2 vv = *reinterpret_cast<const uint2*>(&st.v[b + t][4 * warp]);
        const ulonglong2 dv = *reinterpret_cast<const ulonglong2*>(&st.d[b + t][4 * lane]);
        const float x[4] = {__uint_as_float(vv.x << 16), __uint_as_float(vv.x & 0xffff0000u), __uint_as_float(vv.y << 16),
                            __uint_as_float(vv.y & 0xffff0000u)};
        f2 q2[2], k2[2], d2[2];
        if constexpr (FORGET) {
          const ulonglong2 qv = *reinterpret_cast<const ulonglong2*>(&st.q[b + t][4 * lane]);
          q2[0] = qv.x; q2[1] = qv.y;
          d2[0] = dv.x; d2[1] = dv.y;
        } else {
          const uint2 qv = *reinterpret_cast<const uint2*>(&st.q[b + t][4 * lane]);
          const uint2 kv = *reinterpret_cast<const uint2*>(&st.k[b + t][4 * lane]);
          q2[0] = f2_bf16(qv.x); q2[1] = f2_bf16(qv.y);
          k2[0] = f2_bf16(kv.x); k2[1] = f2_bf16(kv.y);
          d2[0] = f2_neg(dv.x); d2[1] = f2_neg(dv.y);
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const f2 xx = f2_make(x[c], x[c]);
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            if constexpr (FORGET) S[r][c] = f2_fma(d2[r], f2_fma(S[r][c], minus, xx), S[r][c]);
            else S[r][c] = f2_fma(k2[r], xx, f2_fma(d2[r], S[r][c], S[r][c]));
          }
          part[4 * t + c] = f2_sum(f2_fma(q2[1], S[1][c], f2_mul(q2[0], S[0][c])));
        }
      }
      // lane l ends with token l / 4, column l % 4
#pragma unroll
      for (int w = 16; w >= 1; w >>= 1) {
        const bool upper = (lane & w) != 0;
#pragma unroll
        for (int i = 0; i < w; ++i) {
          const float send = upper ? part[i] : part[i + w], keep = upper ? part[i + w] : part[i];
          part[i] = keep + __shfl_xor_sync(0xffffffffu, send, w);
        }
      }
      const int t = lane >> 2, c = lane & 3;
      if (in && t0 + b + t < q_len)
        out[(size_t)(q_start + t0 + b + t) * H * V + (size_t)h * V + col + c] = FORGET ? part[0] : part[0] * q_mult;
    }
  }
  pdl_trigger();
#pragma unroll
  for (int r = 0; r < 2; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int row = 4 * lane + 2 * r;
      if (in && row < N) sp[(size_t)row * V + col + c] = __uint_as_float((unsigned)S[r][c]);
      if (in && row + 1 < N) sp[(size_t)(row + 1) * V + col + c] = __uint_as_float((unsigned)(S[r][c] >> 32));
    }
}

template <bool DELTA>
static int scan_blocks(const bf16* q, int ldq, const bf16* k, int ldk, const bf16* v, int ldv, const bf16* a_raw, int lda, const bf16* b_raw,
                       int ldb, const float* A_log, const float* dt_bias, const float* D, float* coef, float* state,
                       long long slot_stride, float* out, const int* seq_slot, const int* seq_q_start, const int* seq_q_len, int n_tokens,
                       int n_seqs, int H, int G, int N, int V, cudaStream_t s) {
  const int per_group = (H / G + SP_HEADS - 1) / SP_HEADS;
  const int rc = launch_dependent(scan_coef_kernel<DELTA>, dim3(n_tokens / SP_CT + n_seqs, (G * per_group + 3) / 4), dim3(128), 0, s, q, ldq, k,
                                  ldk, a_raw, lda, b_raw, ldb, A_log, dt_bias, D, coef, seq_q_start, seq_q_len, n_seqs, H, G, N, per_group);
  if (rc) return rc;
  const size_t smem = SP_STAGES * sizeof(BlocksStage<DELTA>);
  cudaError_t err = cudaFuncSetAttribute(scan_blocks_kernel<DELTA>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (err != cudaSuccess) return (int)err;
  return launch_dependent(scan_blocks_kernel<DELTA>, dim3(n_seqs, H, (V + SP_COLS - 1) / SP_COLS), dim3(128), smem, s, q, ldq, k, ldk, v, ldv,
                          (const float*)coef, state, slot_stride, out, seq_slot, seq_q_start, seq_q_len, H, G, N, V);
}

static int scan_segments(const bf16* q, int ldq, const bf16* k, int ldk, const bf16* v, int ldv, const bf16* a_raw, int lda,
                         const float* A_log, const float* dt_bias, const float* D, float* coef, float* state, long long slot_stride,
                         float* out, const int* seq_slot, const int* seq_q_start, const int* seq_q_len, int n_tokens, int n_seqs, int H, int G, int N, int V, int segs, float* carried, cudaStream_t s) {
  const int z = (V + SP_SCOLS - 1) / SP_SCOLS;
  float* keeps = carried ? carried + (size_t)n_seqs * segs * H * z * (SP_SCOLS * SP_N) : nullptr;
  const size_t wsmem = SP_STAGES * sizeof(WritesStage), alone = 120 * 1024;
  // (blocks that all find an SM of their own ask for more than half its shared memory: two on one SM, the others idle, is up to
  // half again as slow, and happened in every third run)
  const size_t smem = n_seqs * segs * H * z <= 148 ? alone : SP_STAGES * sizeof(SegmentStage);
  cudaError_t err = cudaFuncSetAttribute(scan_segments_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)alone);
  if (err != cudaSuccess) return (int)err;
  const int writers = n_seqs * (segs - 1) * H * z, jobs = (n_tokens / SP_CT + n_seqs) * H;
  const int rc = launch_dependent(scan_prepare_kernel, dim3(writers + (jobs + 7) / 8), dim3(SP_STHREADS), wsmem, s, q, ldq, k, ldk, v,
                                  ldv, a_raw, lda, A_log, dt_bias, D, coef, (const float*)state, slot_stride, seq_slot, seq_q_start,
                                  seq_q_len, n_seqs, H, G, N, V, segs, writers, (float4*)carried, keeps);
  if (rc) return rc;
  return launch_dependent(scan_segments_kernel, dim3(n_seqs * segs, H, z), dim3(SP_STHREADS), smem, s, q, ldq, k, ldk, v, ldv, (const float*)coef,
                          state, slot_stride, out, seq_slot, seq_q_start, seq_q_len, H, G, N, V, segs, (const float4*)carried,
                          (const float*)keeps);
}

extern "C" {

// Floats of scratch a token needs here (mode as in sb_state_scan), or -1 for what these kernels do not take: q, k, v (and
// in mode 2 the gate's logits, in k's place) as 16-byte pieces.
int sb_scan_prompt_floats(int dtype, int mode, const void* q, int ldq, const void* k, int ldk, const void* v, int ldv,
                          const float* row_decay, int H, int G, int N, int V) {
  if (dtype != 1 || mode < 0 || mode > 3 || N <= 64 || N > SP_N || N % 8 || V < 8 || V % 8 || ldq % 8 || ldk % 8 || ldv % 8) return -1;
  if (H < 1 || G < 1 || H % G || (mode >= 2 && G != H)) return -1;
  if (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)row_decay) % 16) return -1;
  return mode < 2 ? H * SP_COEF(mode == 1) : mode == 2 ? 2 * H * N : 0;
}

// Floats of a segment's place in `carried`, per sequence: the state in whole blocks of columns, and its decay.
long long sb_scan_segment_floats(int H, int V) { return (long long)H * ((V + SP_SCOLS - 1) / SP_SCOLS * (SP_SCOLS * SP_N) + 1); }

// Arguments as sb_state_scan's; scratch: float [n_tokens, that many], 16-byte aligned (null where it is 0).  segs: segments a
// sequence (mode 0 only; 0: one walk, the delta rule's kernels), carried: float [n_seqs, segs, sb_scan_segment_floats], 16-byte aligned
// (null up to one).
int sb_state_scan_prompt(int mode, const void* q, int ldq, const void* k, int ldk, const void* v, int ldv,
                         const void* a_raw, int lda, const void* b_raw, int ldb, const float* A_log, const float* dt_bias,
                         const float* D, const float* row_decay, float* state, long long slot_stride, float* out,
                         const int* seq_slot, const int* seq_q_start, const int* seq_q_len, int n_tokens, int n_seqs, int H,
                         int G, int N, int V, float* scratch, int segs, float* carried, cudaStream_t s) {
  if (n_seqs == 0 || n_tokens == 0) return 0;
  if (sb_scan_prompt_floats(1, mode, q, ldq, k, ldk, v, ldv, row_decay, H, G, N, V) < 0 || (mode < 3 && !scratch) ||
      ((uintptr_t)scratch % 16) || segs < 0 || (segs > 1 && (mode != 0 || !carried || (uintptr_t)carried % 16)) || (mode == 1 && !b_raw) ||
      (mode == 3) != (row_decay != nullptr))
    return -2;
  const dim3 grid(n_seqs, H, (V + SP_COLS - 1) / SP_COLS);
  if (mode < 2) {
#define ARGS(...) (const bf16*)q, ldq, (const bf16*)k, ldk, (const bf16*)v, ldv, (const bf16*)a_raw, lda, __VA_ARGS__ A_log, dt_bias, D, scratch, \
                  state, slot_stride, out, seq_slot, seq_q_start, seq_q_len, n_tokens, n_seqs, H, G, N, V
    if (mode == 0 && segs > 0) return scan_segments(ARGS(), segs, carried, s);
    return mode == 1 ? scan_blocks<true>(ARGS((const bf16*)b_raw, ldb,), s) : scan_blocks<false>(ARGS((const bf16*)b_raw, ldb,), s);
#undef ARGS
  }
  if (mode == 2) {
    const int channels = H * N;
    float* qf = scratch;
    float* d = scratch + (size_t)n_tokens * channels;
    int rc = launch_dependent(scan_gates_kernel, dim3(n_tokens, (channels / 8 + 255) / 256), dim3(256), 0, s, (const bf16*)q, ldq,
                              (const bf16*)k, ldk, A_log, dt_bias, qf, d, channels, (int)!(((uintptr_t)A_log | (uintptr_t)dt_bias) % 16));
    if (rc) return rc;
    const size_t smem = SP_STAGES * sizeof(ForgetStage);
    cudaError_t err = cudaFuncSetAttribute(scan_rows_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (err != cudaSuccess) return (int)err;
    return launch_dependent(scan_rows_kernel<true>, grid, dim3(128), smem, s, (const void*)qf, channels, (const bf16*)nullptr, 0,
                            (const bf16*)v, ldv, (const float*)d, state, slot_stride, out, seq_slot, seq_q_start, seq_q_len, H, N,
                            V);
  }
  const size_t smem = SP_STAGES * sizeof(DecayStage);
  cudaError_t err = cudaFuncSetAttribute(scan_rows_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (err != cudaSuccess) return (int)err;
  return launch_dependent(scan_rows_kernel<false>, grid, dim3(128), smem, s, q, ldq, (const bf16*)k, ldk, (const bf16*)v, ldv,
                          row_decay, state, slot_stride, out, seq_slot, seq_q_start, seq_q_len, H, N, V);
}

}  // extern "C"
