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
//     lost (of an entry below 2^-109 less than 2^-134; S itself is kept whole), and sums are float.  G is applied as S - (1 - G) S, the complement carried as such (state_scan.cu says why), and a
//     block's write is added to S by ordinary adds.
//   walk (forget-write, channel-decay): the decay differs by row, so a token is a step; the state's update is the whole
//     chain, and read-outs of eight tokens are summed together.  A thread keeps 16 entries, so that a loaded vector serves
//     four columns.  forget-write's gates are formed beforehand (scan_gates_kernel): inside the walk every block of 16
//     columns would form them again.  32-bit multiply-adds.
// Measured at 2,048 tokens of one sequence, 16 heads of 128 x 128 (state-space: 32 of 128 x 64), few-token kernel -> here: state-space
// 577 -> 102 us (eight tokens a block on multiply-adds: 164), gated delta 673 -> 133 (203), forget-write 414 -> 174,
// channel-decay 400 -> 177; unequal sequences of 801, 712 and 623 tokens: 383 -> 72, 598 -> 100, 382 -> 160, 377 -> 155.  The
// error against 64 bits falls or stays (outputs 5.5e-7 -> 2.2e-7, 3.7e-7 -> 2.0e-7, 4.9e-8, 1.2e-7).  With one sequence
// an SM has four warps and the chain's latencies are the bound (about 1,500 cycles a block of sixteen), not a pipe.
#include <type_traits>

#include "common.cuh"

#define SP_N 128                 // rows of the state kept (N up to this; the rest are zeros)
#define SP_CT 16                 // tokens a block (and a stage)
#define SP_STAGES 3
#define SP_COLS 16               // value columns a block: four a warp
#define SP_COEF(DELTA) ((DELTA) ? 36 : 20)      // floats of a token's coefficients: W row (16, delta rule), B row (16), four scalars

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
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
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
  // the block's sequence: 32 sequences' block counts at a time
  int left = blockIdx.x, seq = -1, block = 0;
  for (int s0 = 0; s0 < n_seqs && seq < 0; s0 += 32) {
    const int s = s0 + lane;
    const int mine = s < n_seqs ? (seq_q_len[s] + SP_CT - 1) / SP_CT : 0;
    int upto = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += v;
    }
    const unsigned hit = __ballot_sync(0xffffffffu, left < upto);
    if (hit) {
      const int at = __ffs(hit) - 1;
      seq = s0 + at;
      block = left - (__shfl_sync(0xffffffffu, upto, at) - __shfl_sync(0xffffffffu, mine, at));
    } else {
      left -= __shfl_sync(0xffffffffu, upto, 31);
    }
  }
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

// ------------------------------------------------------------------------------------------ a decay per row
// qf = silu(q), d = (1 - lower) sigmoid(-(z + bias)): a thread eight channels of a token (blockIdx.x: a step may bring more
// tokens than the grid's other dimensions count to).
__global__ void __launch_bounds__(256)
scan_gates_kernel(const bf16* __restrict__ q, int ldq, const bf16* __restrict__ z, int ldz, const float* __restrict__ lower,
                  const float* __restrict__ bias, float* __restrict__ qf, float* __restrict__ d, int channels) {
  pdl_wait();
  SB_BEHIND_WAIT(q); SB_BEHIND_WAIT(z);
  const int c = (blockIdx.y * 256 + threadIdx.x) * 8;
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
    g[i] = (1.f - lower[c + i]) / (1.f + expf(ze + bias[c + i]));
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

// Arguments as sb_state_scan's; scratch: float [n_tokens, that many], 16-byte aligned (null where it is 0).
int sb_state_scan_prompt(int mode, const void* q, int ldq, const void* k, int ldk, const void* v, int ldv,
                         const void* a_raw, int lda, const void* b_raw, int ldb, const float* A_log, const float* dt_bias,
                         const float* D, const float* row_decay, float* state, long long slot_stride, float* out,
                         const int* seq_slot, const int* seq_q_start, const int* seq_q_len, int n_tokens, int n_seqs, int H,
                         int G, int N, int V, float* scratch, cudaStream_t s) {
  if (n_seqs == 0 || n_tokens == 0) return 0;
  if (sb_scan_prompt_floats(1, mode, q, ldq, k, ldk, v, ldv, row_decay, H, G, N, V) < 0 || (mode < 3 && !scratch) ||
      ((uintptr_t)scratch % 16) || (mode == 1 && !b_raw) || (mode == 3) != (row_decay != nullptr))
    return -2;
  const dim3 grid(n_seqs, H, (V + SP_COLS - 1) / SP_COLS);
  if (mode < 2) {
    const int per_group = (H / G + SP_HEADS - 1) / SP_HEADS;
    const dim3 cgrid(n_tokens / SP_CT + n_seqs, (G * per_group + 3) / 4);
    int rc = mode == 1
        ? launch_dependent(scan_coef_kernel<true>, cgrid, dim3(128), 0, s, (const bf16*)q, ldq, (const bf16*)k, ldk,
                           (const bf16*)a_raw, lda, (const bf16*)b_raw, ldb, A_log, dt_bias, D, scratch, seq_q_start, seq_q_len,
                           n_seqs, H, G, N, per_group)
        : launch_dependent(scan_coef_kernel<false>, cgrid, dim3(128), 0, s, (const bf16*)q, ldq, (const bf16*)k, ldk,
                           (const bf16*)a_raw, lda, (const bf16*)b_raw, ldb, A_log, dt_bias, D, scratch, seq_q_start, seq_q_len,
                           n_seqs, H, G, N, per_group);
    if (rc) return rc;
    const size_t smem = SP_STAGES * (mode == 1 ? sizeof(BlocksStage<true>) : sizeof(BlocksStage<false>));
    auto kernel = mode == 1 ? scan_blocks_kernel<true> : scan_blocks_kernel<false>;
    cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (err != cudaSuccess) return (int)err;
    return launch_dependent(kernel, grid, dim3(128), smem, s, (const bf16*)q, ldq, (const bf16*)k, ldk, (const bf16*)v, ldv,
                            (const float*)scratch, state, slot_stride, out, seq_slot, seq_q_start, seq_q_len, H, G, N, V);
  }
  if (mode == 2) {
    const int channels = H * N;
    float* qf = scratch;
    float* d = scratch + (size_t)n_tokens * channels;
    int rc = launch_dependent(scan_gates_kernel, dim3(n_tokens, (channels / 8 + 255) / 256), dim3(256), 0, s, (const bf16*)q, ldq,
                              (const bf16*)k, ldk, A_log, dt_bias, qf, d, channels);
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
