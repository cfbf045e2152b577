// The matrix-state recurrences of state_scan.cu for steps that bring many tokens a sequence (bfloat16, states of 65 to
// 128 rows).  The walk there gives a token's state to 256 threads, eight rows of one column each: every multiply-add
// is paid for with a float from shared memory (which hands a warp 128 bytes a cycle, shared addresses or not), and a
// token's sums are a round of shuffles in the chain of the next.  Here a thread keeps 16 entries (so that a
// loaded vector serves two or four columns), operands stay bfloat16 in shared memory until they are used (cp.async
// brings them three chunks ahead, nothing passes through registers on the way), and sums over rows are made for eight
// tokens at once.  All arithmetic is 32-bit; bfloat16 inputs are exact.
//
//   blocks (state-space, gated delta): eight tokens at a time from the state S the block finds.  With G_t the
//     product of the block's decays up to token t and Gamma(t, i) from i's successor to t,
//       z_t = beta_t (v_t - G_t S^T k_t)  (state-space: v_t),   u = (I + A)^-1 z,  A(t, i) = beta_t Gamma(t, i) k_i . k_t
//       o_t = G_t S^T q_t + sum_{i <= t} Gamma(t, i) (k_i . q_t) u_i,     S <- G S + sum_i Gamma(last, i) k_i u_i^T
//     What does not involve S (the products of keys and queries, the decays, the inverse: the compact form of a product
//     of such updates, Bischof and Van Loan 1987) is one 8 x 8 matrix pair a block and head, made beforehand for
//     all blocks at once by scan_coef_kernel; the chain over the sequence is one round of sums and two small products
//     for eight tokens.  G is applied as S - (1 - G) S, the complement carried as such (state_scan.cu says why).
//   walk (forget-write, channel-decay): the decay differs by row, so a token is a step; the state's update is the whole
//     chain, and read-outs of eight tokens are summed together.  forget-write's gates are formed beforehand
//     (scan_gates_kernel): inside the walk every block of 16 columns would form them again.
// Measured at 2,048 tokens of one sequence, 16 heads of 128 x 128 (state-space: 32 of 128 x 64), before -> now: state-space 577 ->
// 164 us, gated delta 673 -> 203, forget-write 414 -> 174, channel-decay 400 -> 177; unequal sequences of 801, 712 and 623
// tokens: 383 -> 138, 603 -> 181, 382 -> 160, 377 -> 155.  The error against 64 bits is that of the other kernel or less
// (outputs 5.5e-7 -> 4.2e-7, 3.7e-7 -> 3.1e-7, 4.9e-8, 1.2e-7).  With one sequence a scheduler has one warp, which issues in
// 45 % of its cycles (the rest: waits of a few cycles for the result before); DRAM and shared memory are not the bound.
#include "common.cuh"

#define SP_N 128                 // rows of the state kept (N up to this; the rest are zeros)
#define SP_CT 16                 // tokens a chunk
#define SP_STAGES 3
#define SP_COLS 16               // value columns a block: four a warp
#define SP_COEF 20               // floats of a token's coefficients: W row (8), B row (8), four scalars

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
// A warp a block of eight tokens and up to SP_HEADS heads of one key/query group.  k . k and q . k of the block are one
// 16 x 8 product of bfloat16 (exact) with float sums; lane l holds token l / 4, entries 2 (l % 4) and the next.
// Row (token, head) of `coef`: [W: mk Gamma(last, t) (I + A)^-1 row t | B: row t times the inverse | beta, beta mk G, mq G,
// 1 - G of the whole block] for the delta rule; [unused | B: Gamma dt_i (q_t . k_i), D added at i = t | Gamma(last, t) dt_t, 0, G,
// 1 - G of the block] for the state-space form.
#define SP_HEADS 4
__device__ __forceinline__ void sp_mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

template <bool DELTA>
__global__ void __launch_bounds__(128, 3)
scan_coef_kernel(const bf16* __restrict__ q, int ldq, const bf16* __restrict__ k, int ldk, const bf16* __restrict__ a_raw,
                 int lda, const bf16* __restrict__ b_raw, int ldb, const float* __restrict__ A_log,
                 const float* __restrict__ dt_bias, const float* __restrict__ D, float* __restrict__ coef,
                 const int* __restrict__ seq_q_start, const int* __restrict__ seq_q_len, int n_seqs, int H, int G, int N,
                 int per_group) {
  __shared__ float sa[4][8][9], sb[4][8][9];
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
    const int mine = s < n_seqs ? (seq_q_len[s] + 7) / 8 : 0;
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
  const int first = seq_q_start[seq] + 8 * block, ct = min(8, seq_q_len[seq] - 8 * block);
  const int t = lane >> 2, i0 = 2 * (lane & 3);
  const bool real = t < ct;
  // lane (t, x): 16-byte pieces x, x + 4, .. of token t's key and query; every product sees its entries in one order
  float ck[4] = {0.f, 0.f, 0.f, 0.f}, cq[4] = {0.f, 0.f, 0.f, 0.f};      // k.k | q.k;  k.q | q.q (only the norms are read)
  const bf16* kr = k + (size_t)(first + (real ? t : 0)) * ldk + (size_t)group * N;
  const bf16* qr = q + (size_t)(first + (real ? t : 0)) * ldq + (size_t)group * N;
#pragma unroll
  for (int j = 0; j < SP_N / 32; ++j) {
    const int piece = (lane & 3) + 4 * j;
    const bool have = real && piece * 8 < N;
    uint4 kv = make_uint4(0u, 0u, 0u, 0u), qv = kv;
    if (have) {
      kv = *reinterpret_cast<const uint4*>(kr + piece * 8);
      qv = *reinterpret_cast<const uint4*>(qr + piece * 8);
    }
    sp_mma(ck, kv.x, qv.x, kv.y, qv.y, kv.x, kv.y);
    sp_mma(ck, kv.z, qv.z, kv.w, qv.w, kv.z, kv.w);
    if (DELTA) {
      sp_mma(cq, kv.x, qv.x, kv.y, qv.y, qv.x, qv.y);
      sp_mma(cq, kv.z, qv.z, kv.w, qv.w, qv.z, qv.w);
    }
  }
  // unit norms of the block's tokens: token j's squares lie on lane (j, j / 2), entry j % 2
  float mk_t = 1.f, mq_t = 1.f, mk_i[2] = {1.f, 1.f};
  if (DELTA) {
    auto diag = [&](float even, float odd, int j) {
      const float e = __shfl_sync(0xffffffffu, even, 4 * j + (j >> 1)), o = __shfl_sync(0xffffffffu, odd, 4 * j + (j >> 1));
      return (j & 1) ? o : e;
    };
    const float q_mult = rsqrtf((float)N);
    mk_t = 1.f / sqrtf(diag(ck[0], ck[1], t) + 1e-6f);
    mq_t = q_mult / sqrtf(diag(cq[2], cq[3], t) + 1e-6f);
    mk_i[0] = __shfl_sync(0xffffffffu, mk_t, 4 * i0);
    mk_i[1] = __shfl_sync(0xffffffffu, mk_t, 4 * (i0 + 1));
  }
  for (int h = h0; h < h1; ++h) {
    float d = 0.f, fac = 0.f;             // lanes 0 .. 7: token `lane`'s 1 - decay and its factor (dt, or beta)
    if (lane < ct) {
      const size_t row = (size_t)(first + lane);
      const float dt = sp_softplus(to_f<bf16>(a_raw[row * lda + h]) + dt_bias[h]);
      d = -expm1f(-expf(A_log[h]) * dt);
      fac = DELTA ? 1.f / (1.f + expf(-to_f<bf16>(b_raw[row * ldb + h]))) : dt;
    }
    float gam[2] = {1.f, 1.f}, all = 1.f, last = 1.f, gone = 0.f;    // Gamma(t, i), G_t, Gamma(end, t), 1 - G
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const float dr = __shfl_sync(0xffffffffu, d, r), keep = 1.f - dr;
      gone = fmaf(-gone, dr, gone + dr);
      if (r <= t) all *= keep;
      if (r > t) last *= keep;
      if (r <= t && r > i0) gam[0] *= keep;
      if (r <= t && r > i0 + 1) gam[1] *= keep;
    }
    const float fac_t = __shfl_sync(0xffffffffu, fac, t);
    float* row = coef + ((size_t)(first + t) * H + h) * SP_COEF;
    if (!DELTA) {
      const float fi[2] = {__shfl_sync(0xffffffffu, fac, i0), __shfl_sync(0xffffffffu, fac, i0 + 1)};
      const float skip = D ? D[h] : 0.f;
      if (real) {
        float2 b;
        b.x = i0 <= t ? gam[0] * fi[0] * ck[2] + (i0 == t ? skip : 0.f) : 0.f;
        b.y = i0 + 1 <= t ? gam[1] * fi[1] * ck[3] + (i0 + 1 == t ? skip : 0.f) : 0.f;
        *reinterpret_cast<float2*>(row + 8 + i0) = b;
        if ((lane & 3) == 0) *reinterpret_cast<float4*>(row + 16) = make_float4(last * fac_t, 0.f, all, gone);
      }
      continue;
    }
    __syncwarp();
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      sa[warp][t][i0 + e] = i0 + e < t ? fac_t * gam[e] * mk_t * mk_i[e] * ck[e] : 0.f;
      sb[warp][t][i0 + e] = i0 + e <= t ? gam[e] * mq_t * mk_i[e] * ck[2 + e] : 0.f;
    }
    __syncwarp();
    // column j of the inverse of I + A, by lane j of every eight; rows of B times it
    const int j = lane & 7;
    float x[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      float s = r == j ? 1.f : 0.f;
#pragma unroll
      for (int i = 0; i < r; ++i) s = fmaf(-sa[warp][r][i], x[i], s);
      x[r] = r < j ? 0.f : s;
    }
    // lane's eight: rows 2 (lane / 8) and the next
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int r = 2 * (lane >> 3) + e;
      float s = 0.f, own = 0.f;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        s = fmaf(sb[warp][r][i], x[i], s);
        own = i == r ? x[i] : own;
      }
      const float mk_r = __shfl_sync(0xffffffffu, mk_t, 4 * r), last_r = __shfl_sync(0xffffffffu, last, 4 * r);
      if (r < ct) {
        float* to = coef + ((size_t)(first + r) * H + h) * SP_COEF;
        to[j] = mk_r * last_r * own;
        to[8 + j] = s;
      }
    }
    if (real && (lane & 3) == 0) *reinterpret_cast<float4*>(row + 16) = make_float4(fac_t, fac_t * mk_t * all, mq_t * all, gone);
  }
}

// ------------------------------------------------------------------------------------------ the chain of blocks
// A block of four warps owns 16 columns of one head's S for one sequence; a lane keeps rows 8 p .. 8 p + 7 (p = lane % 16) of
// two columns.  After the sums lane p holds token p / 2, column p % 2 of its half warp's pair.
struct BlocksStage {
  bf16 k[SP_CT][SP_N], q[SP_CT][SP_N], v[SP_CT][SP_COLS];
  float coef[SP_CT][SP_COEF];
};

// The sums over 16 lanes of 16 values each: lane p ends with value p.
__device__ __forceinline__ float sp_sums16(float (&part)[16], int p) {
#pragma unroll
  for (int w = 8; w >= 1; w >>= 1) {
    const bool upper = (p & w) != 0;
#pragma unroll
    for (int i = 0; i < w; ++i) {
      const float send = upper ? part[i] : part[i + w], keep = upper ? part[i + w] : part[i];
      part[i] = keep + __shfl_xor_sync(0xffffffffu, send, w);
    }
  }
  return part[0];
}

template <bool DELTA>
__global__ void __launch_bounds__(128, 3)
scan_blocks_kernel(const bf16* __restrict__ q, int ldq, const bf16* __restrict__ k, int ldk, const bf16* __restrict__ v, int ldv,
                   const float* __restrict__ coef, float* __restrict__ state, long long slot_stride, float* __restrict__ out,
                   const int* __restrict__ seq_slot, const int* __restrict__ seq_q_start, const int* __restrict__ seq_q_len,
                   int H, int G, int N, int V) {
  __shared__ __align__(16) BlocksStage stages[SP_STAGES];
  __shared__ __align__(16) float written[4][2][8][2];
  pdl_wait();
  SB_BEHIND_WAIT(state); SB_BEHIND_WAIT(seq_slot); SB_BEHIND_WAIT(seq_q_start); SB_BEHIND_WAIT(seq_q_len);
  const int seq = blockIdx.x, h = blockIdx.y, col0 = blockIdx.z * SP_COLS;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, p = lane & 15, half = lane >> 4;
  const int group = h / (H / G);
  const int q_start = seq_q_start[seq], q_len = seq_q_len[seq];
  const int col = col0 + 4 * warp + 2 * half;       // this lane's columns: col, col + 1 (inside or outside together)
  const bool in = col < V;
  float* sp = state + (size_t)seq_slot[seq] * slot_stride + (size_t)h * N * V;
  f2 S[4][2];                                       // rows 8 p + 2 r and the next
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    float e[2][2];
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      const int row = 8 * p + 2 * r + x;
      const bool have = in && row < N;
      e[x][0] = have ? sp[(size_t)row * V + col] : 0.f;
      e[x][1] = have ? sp[(size_t)row * V + col + 1] : 0.f;
    }
    S[r][0] = f2_make(e[0][0], e[1][0]);
    S[r][1] = f2_make(e[0][1], e[1][1]);
  }
  const bf16* kg = k + (size_t)group * N;
  const bf16* qg = q + (size_t)group * N;
  const bf16* vh = v + (size_t)h * V + col0;
  auto load = [&](int t0) {                         // a chunk into its stage: 16-byte pieces, zeros where nothing is
    BlocksStage& st = stages[t0 / SP_CT % SP_STAGES];
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
    if (tid < SP_CT * (SP_COEF / 4)) {
      const int tt = tid / (SP_COEF / 4), c = tid % (SP_COEF / 4) * 4;
      const bool real = t0 + tt < q_len;
      sp_copy16(&st.coef[tt][c], coef + ((size_t)(q_start + (real ? t0 + tt : 0)) * H + h) * SP_COEF + c, real);
    }
  };
  load(0);
  sp_commit();
  if (SP_CT < q_len) load(SP_CT);
  sp_commit();
  for (int t0 = 0; t0 < q_len; t0 += SP_CT) {
    sp_wait_one();
    __syncthreads();                                // the chunk is there, and nobody reads the stage filled next
    if (t0 + 2 * SP_CT < q_len) load(t0 + 2 * SP_CT);
    sp_commit();
    const BlocksStage& st = stages[t0 / SP_CT % SP_STAGES];
#pragma unroll 1
    for (int b = 0; b < SP_CT && t0 + b < q_len; b += 8) {
      float pq[16], pk[DELTA ? 16 : 1];
#pragma unroll
      for (int t = 0; t < 8; ++t) {
        const uint4 qv = *reinterpret_cast<const uint4*>(&st.q[b + t][8 * p]);
        const f2 q2[4] = {f2_bf16(qv.x), f2_bf16(qv.y), f2_bf16(qv.z), f2_bf16(qv.w)};
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          f2 a = f2_mul(q2[0], S[0][c]);
#pragma unroll
          for (int r = 1; r < 4; ++r) a = f2_fma(q2[r], S[r][c], a);
          pq[2 * t + c] = f2_sum(a);
        }
        if (DELTA) {
          const uint4 kv = *reinterpret_cast<const uint4*>(&st.k[b + t][8 * p]);
          const f2 k2[4] = {f2_bf16(kv.x), f2_bf16(kv.y), f2_bf16(kv.z), f2_bf16(kv.w)};
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            f2 a = f2_mul(k2[0], S[0][c]);
#pragma unroll
            for (int r = 1; r < 4; ++r) a = f2_fma(k2[r], S[r][c], a);
            pk[2 * t + c] = f2_sum(a);
          }
        }
      }
      const int t = p >> 1, c = p & 1;
      const float* row = st.coef[b + t];
      const float4 s = *reinterpret_cast<const float4*>(row + 16);
      float B[8], own = 0.f;
#pragma unroll
      for (int n = 0; n < 2; ++n) *reinterpret_cast<float4*>(B + 4 * n) = *reinterpret_cast<const float4*>(row + 8 + 4 * n);
      if constexpr (DELTA) {
        float W[8], w = 0.f;
#pragma unroll
        for (int n = 0; n < 2; ++n) *reinterpret_cast<float4*>(W + 4 * n) = *reinterpret_cast<const float4*>(row + 4 * n);
        const float x = to_f<bf16>(st.v[b + t][4 * warp + 2 * half + c]);
        const float z = s.x * x - s.y * sp_sums16(pk, p);
        float zi[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) zi[i] = __shfl_sync(0xffffffffu, z, (lane & 16) | (2 * i + c));
#pragma unroll
        for (int i = 0; i < 8; ++i) w = fmaf(W[i], zi[i], w);
        written[warp][half][t][c] = w;
#pragma unroll
        for (int i = 0; i < 8; ++i) own = fmaf(B[i], zi[i], own);
        __syncwarp();
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) own = fmaf(B[i], to_f<bf16>(st.v[b + i][4 * warp + 2 * half + c]), own);
      }
      const float gone = st.coef[b][19];
      const f2 g2 = f2_make(-gone, -gone);
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int cc = 0; cc < 2; ++cc) S[r][cc] = f2_fma(g2, S[r][cc], S[r][cc]);
#pragma unroll
      for (int tt = 0; tt < 8; ++tt) {
        const uint4 kv = *reinterpret_cast<const uint4*>(&st.k[b + tt][8 * p]);
        const f2 k2[4] = {f2_bf16(kv.x), f2_bf16(kv.y), f2_bf16(kv.z), f2_bf16(kv.w)};
        float2 u;
        if constexpr (DELTA) {
          u = *reinterpret_cast<const float2*>(written[warp][half][tt]);
        } else {
          const uint32_t vv = *reinterpret_cast<const uint32_t*>(&st.v[b + tt][4 * warp + 2 * half]);
          const float by = st.coef[b + tt][16];
          u = make_float2(by * __uint_as_float(vv << 16), by * __uint_as_float(vv & 0xffff0000u));
        }
        const f2 u0 = f2_make(u.x, u.x), u1 = f2_make(u.y, u.y);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          S[r][0] = f2_fma(k2[r], u0, S[r][0]);
          S[r][1] = f2_fma(k2[r], u1, S[r][1]);
        }
      }
      const float done = sp_sums16(pq, p);
      if (in && t0 + b + t < q_len) out[(size_t)(q_start + t0 + b + t) * H * V + (size_t)h * V + col + c] = fmaf(s.z, done, own);
      if (DELTA) __syncwarp();
    }
  }
  pdl_trigger();
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int cc = 0; cc < 2; ++cc) {
      const int row = 8 * p + 2 * r;
      if (in && row < N) sp[(size_t)row * V + col + cc] = __uint_as_float((unsigned)S[r][cc]);
      if (in && row + 1 < N) sp[(size_t)(row + 1) * V + col + cc] = __uint_as_float((unsigned)(S[r][cc] >> 32));
    }
}

// ------------------------------------------------------------------------------------------ a decay per row
// qf = silu(q), d = (1 - lower) sigmoid(-(z + bias)): a thread eight channels of a token.
__global__ void __launch_bounds__(256)
scan_gates_kernel(const bf16* __restrict__ q, int ldq, const bf16* __restrict__ z, int ldz, const float* __restrict__ lower,
                  const float* __restrict__ bias, float* __restrict__ qf, float* __restrict__ d, int channels) {
  pdl_wait();
  SB_BEHIND_WAIT(q); SB_BEHIND_WAIT(z);
  const int c = (blockIdx.x * 256 + threadIdx.x) * 8;
  if (c >= channels) return;
  const size_t row = blockIdx.y;
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
  return mode < 2 ? H * SP_COEF : mode == 2 ? 2 * H * N : 0;
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
    const dim3 cgrid(n_tokens / 8 + n_seqs, (G * per_group + 3) / 4);
    int rc = mode == 1
        ? launch_dependent(scan_coef_kernel<true>, cgrid, dim3(128), 0, s, (const bf16*)q, ldq, (const bf16*)k, ldk,
                           (const bf16*)a_raw, lda, (const bf16*)b_raw, ldb, A_log, dt_bias, D, scratch, seq_q_start, seq_q_len,
                           n_seqs, H, G, N, per_group)
        : launch_dependent(scan_coef_kernel<false>, cgrid, dim3(128), 0, s, (const bf16*)q, ldq, (const bf16*)k, ldk,
                           (const bf16*)a_raw, lda, (const bf16*)b_raw, ldb, A_log, dt_bias, D, scratch, seq_q_start, seq_q_len,
                           n_seqs, H, G, N, per_group);
    if (rc) return rc;
    return mode == 1
        ? launch_dependent(scan_blocks_kernel<true>, grid, dim3(128), 0, s, (const bf16*)q, ldq, (const bf16*)k, ldk,
                           (const bf16*)v, ldv, (const float*)scratch, state, slot_stride, out, seq_slot, seq_q_start, seq_q_len,
                           H, G, N, V)
        : launch_dependent(scan_blocks_kernel<false>, grid, dim3(128), 0, s, (const bf16*)q, ldq, (const bf16*)k, ldk,
                           (const bf16*)v, ldv, (const float*)scratch, state, slot_stride, out, seq_slot, seq_q_start, seq_q_len,
                           H, G, N, V);
  }
  if (mode == 2) {
    const int channels = H * N;
    float* qf = scratch;
    float* d = scratch + (size_t)n_tokens * channels;
    int rc = launch_dependent(scan_gates_kernel, dim3((channels / 8 + 255) / 256, n_tokens), dim3(256), 0, s, (const bf16*)q, ldq,
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
