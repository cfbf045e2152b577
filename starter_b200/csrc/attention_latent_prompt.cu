// Latent attention for prompts (bfloat16) on the fifth-generation tensor cores.
//
// attention_latent.cu scores the cached latents themselves: a query head of rank + rot entries, values of rank.  For a
// step of few tokens that reads each cache row once and multiplies little.  A prompt's queries outnumber what it costs to
// form every head's keys and values once (rows * heads * (dim + vdim) * rank products against pairs of rank + rot and
// rank), so here they are formed: latent_gather_kernel brings the sequences' cache rows behind one another, the library's
// product makes [k of all heads | v of all heads] of them, and this kernel attends with queries and keys of dim + rot and
// values of vdim (192 and 128 in place of 576 and 512: 3.4 times fewer products a pair).  The rotated part of the keys
// is the gathered rows' own, shared by the heads.
//
// The block is attention_prefill_tc.cu's: 256 queries of a head as two tiles of 128, S and O of both in tensor memory, TMA
// brings the operands in 128-byte swizzle, one warp issues the products of each tile, a thread is a query row, the output
// is rescaled only when a row's maximum has grown by more than 2^8.  Three chunks of 64 query entries leave no room for
// steps of 128 keys (2 x 48 KB of queries, 2 x 48 of keys, 32 of values, 2 x 32 of weights): steps are 64 keys, with
// two buffers each of keys, values and S, so that S of the next step is formed while this one's exponentials run.
//
// A layer of width 2048, 16 heads of 128 + 64 over a latent of 512, 2,048 tokens: 517 us a pass with the kernel that scores the latents
// (417 of them in it, mma.sync at 0.11 of the tensor peak; two products of 11 us around it), 156 with these.  The error against
// 64 bits is no larger (keys and values are rounded here, folded queries and summed latents there): 0.00470 against 0.00473 at
// that size, 0.00463 against 0.00464 for four sequences of up to 450 tokens, 0.00482 against 0.00489 for 300 tokens behind 900 (means of
// three seeds; 0.00477, 0.00471 and 0.00482 while the weights were summed before their rounding and relative to the sink).
//
// Few blocks over many keys: a cluster's CTAs walk a part of a block's keys each and merge (attention_tc.cuh): 700 tokens behind 1,200
// 60.1 -> 48.6 us.  Up to a block an SM, of unequal lengths: blocks from `split_from` steps on are shared by the two CTAs of a cluster,
// in front of shorter ones the two take a head's block each; a causal prompt's longest chain gets shorter while short blocks fill the
// SMs (2,048 tokens a layer 147 -> 137 us, 1,300 114 -> 106, 1,200 behind 1,200 136 -> 120; latent_mixed_splits in ops.py).
//
// Gathered rows: a sequence's keys from the first that any of its queries sees, padded to a multiple of 64 with zeros, so
// that a step never reads another sequence's values (their weights are zero, but 0 * inf would not be).
#include <cuda.h>

#include "attention_tc.cuh"
#include "common.cuh"
#include "tensor_map.cuh"

#define LP_BK 64
#define LP_THREADS 352

// The first key that a sequence's queries of this step see.
__device__ __forceinline__ int lp_first_key(int kv_len, int q_len, int window) {
  return window > 0 ? max(0, kv_len - q_len - window + 1) : 0;
}
__device__ __forceinline__ int lp_rows(int kv_len, int q_len, int window) {
  return (kv_len - lp_first_key(kv_len, q_len, window) + LP_BK - 1) / LP_BK * LP_BK;
}
// Where sequence `seq` begins among the gathered rows (whole warp).
__device__ __forceinline__ int lp_row0(const int* seq_kv_len, const int* seq_q_len, int seq, int window, int lane) {
  int rows = 0;
  for (int s = lane; s < seq; s += 32) rows += lp_rows(seq_kv_len[s], seq_q_len[s], window);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) rows += __shfl_xor_sync(0xffffffffu, rows, o);
  return rows;
}

// (The queries' turn beside the gathering and the gate in the attention's last step in place of launches of their own: a layer of 2,048 tokens
// 150.0 -> 146.6 us, 600 behind 1,100 94 -> 91.0, two prompts of 207 captured 52.3 -> 49.9.)
// What turns the queries beside the gathering: pairs of neighbours of a head's last 64 entries, in place, a thread eight of them.
struct LatentTurn {
  bf16* q;                       // [tokens, heads * (dim + 64)], or null: nothing turns
  const float *cos_t, *sin_t;
  const int* tok_pos;
  int table_width, heads, dim;
  long long pieces;
};
__device__ __forceinline__ void latent_turn(const LatentTurn& turn, long long at) {
  if (at >= turn.pieces) return;
  const int per_row = turn.heads * 8;
  const long long row = at / per_row;
  const int e = (int)(at - row * per_row), h = e >> 3, c = (e & 7) * 8;
  bf16* to = turn.q + ((size_t)row * turn.heads + h) * (turn.dim + 64) + turn.dim + c;
  const uint4 v = *reinterpret_cast<const uint4*>(to);
  const size_t angle = (size_t)turn.tok_pos[row] * turn.table_width + c / 2;
  const float4 co = *reinterpret_cast<const float4*>(turn.cos_t + angle), si = *reinterpret_cast<const float4*>(turn.sin_t + angle);
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
  const float cs[4] = {co.x, co.y, co.z, co.w}, sn[4] = {si.x, si.y, si.z, si.w};
  uint4 o;
  __nv_bfloat162* p = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float a = __uint_as_float(w[i] << 16), b = __uint_as_float(w[i] & 0xffff0000u);
    p[i] = __floats2bfloat162_rn(a * cs[i] - b * sn[i], b * cs[i] + a * sn[i]);
  }
  *reinterpret_cast<uint4*>(to) = o;
}

// c [rows, rank] and shared [rows, rot] from the cache rows [pages, 64, rank + rot]: a warp a row, 16-byte pieces.  The grid's rows
// behind the sequences' turn the queries: one launch in place of two that do not need each other.
__global__ void __launch_bounds__(256)
latent_gather_kernel(const bf16* __restrict__ store, const int* __restrict__ block_table, int table_stride,
                     const int* __restrict__ seq_slot, const int* __restrict__ seq_q_len, const int* __restrict__ seq_kv_len,
                     bf16* __restrict__ c, bf16* __restrict__ shared, int rank, int rot, int window, int n_seqs, LatentTurn turn) {
  pdl_trigger();
  pdl_wait();
  SB_BEHIND_WAIT(store); SB_BEHIND_WAIT(block_table); SB_BEHIND_WAIT(seq_slot); SB_BEHIND_WAIT(seq_q_len); SB_BEHIND_WAIT(seq_kv_len);
  SB_BEHIND_WAIT(turn.q); SB_BEHIND_WAIT(turn.tok_pos);
  if ((int)blockIdx.y >= n_seqs) {
    latent_turn(turn, ((long long)(blockIdx.y - n_seqs) * gridDim.x + blockIdx.x) * 256 + threadIdx.x);
    return;
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, seq = blockIdx.y;
  const int kv_len = seq_kv_len[seq], first = lp_first_key(kv_len, seq_q_len[seq], window);
  const int i = blockIdx.x * 8 + warp;
  if (i >= lp_rows(kv_len, seq_q_len[seq], window)) return;
  const size_t row = (size_t)lp_row0(seq_kv_len, seq_q_len, seq, window, lane) + i;
  const int j = first + i;
  const bool real = j < kv_len;
  const int page = block_table[(size_t)seq_slot[seq] * table_stride + (real ? j : first) / SB_PAGE_TOKENS];
  const bf16* from = store + page_row(page, 0, j % SB_PAGE_TOKENS, 1, rank + rot);
  const int pieces = (rank + rot) / 8, own = rank / 8;
  for (int p = lane; p < pieces; p += 32) {
    const uint4 v = real ? *reinterpret_cast<const uint4*>(from + p * 8) : make_uint4(0u, 0u, 0u, 0u);
    if (p < own) *reinterpret_cast<uint4*>(c + row * rank + p * 8) = v;
    else *reinterpret_cast<uint4*>(shared + row * rot + (p - own) * 8) = v;
  }
}

// DC: 64-entry chunks of a head's plain key, VC: of its value; the rotated part is one more chunk.
template <int DC, int VC>
__global__ void __launch_bounds__(LP_THREADS, 1)
latent_prompt_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_kv,
                     const __grid_constant__ CUtensorMap map_rot, bf16* __restrict__ out, const int* __restrict__ seq_q_start,
                     const int* __restrict__ seq_q_len, const int* __restrict__ seq_kv_len, const int* __restrict__ block_seq,
                     const int* __restrict__ block_first, int heads, float scale_log2, int window,
                     const float* __restrict__ sink, int* status, int withhold, int splits, int split_from, const bf16* __restrict__ gate,
                     int gate_ld) {
  constexpr int QC = DC + 1;
  constexpr int QSUB = 128 * 128, KSUB = 64 * 128;  // bytes of 128 (64) rows of 128 bytes
  constexpr int Q_BYTES = QC * QSUB, K_BYTES = QC * KSUB, V_BYTES = VC * KSUB, P_BYTES = QSUB;
  constexpr uint32_t TMEM_COLS = 512;               // S: 2 tiles x 2 buffers x 64; O: 2 x 128 from column 256 on
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* q_sm = smem;                             // 2 tiles
  uint8_t* p_sm = q_sm + 2 * Q_BYTES;               // 2 tiles
  uint8_t* k_sm = p_sm + 2 * P_BYTES;               // 2 buffers
  uint8_t* v_sm = k_sm + 2 * K_BYTES;               // 2 buffers
  __shared__ uint64_t q_full, k_full[2], k_empty[2], v_full[2], v_empty[2], s_ready[2][2], s_free[2][2], p_ready[2], o_ready[2];
  __shared__ uint32_t tmem_holder;
  __shared__ int abort_flag;
  __shared__ __align__(8) float2 ml[2 * TC_BQ];     // keys in parts: the rows' references and sums

  const int seq = block_seq[blockIdx.y], q_first = block_first[blockIdx.y];
  const int q_len = seq_q_len[seq], kv_len = seq_kv_len[seq];
  const int rows_valid = min(2 * TC_BQ, q_len - q_first);
  const int pos0 = kv_len - q_len + q_first;
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  // steps of 64 keys, counted from the sequence's first gathered key; this block's first step
  const int base = lp_first_key(kv_len, q_len, window);
  const int lo = window > 0 ? max(0, pos0 - window + 1) : 0;
  int step0 = (lo - base) / LP_BK;
  int n_tile[2];
  n_tile[0] = (pos0 + min(rows_valid, TC_BQ) - 1 - base) / LP_BK - step0 + 1;
  n_tile[1] = rows_valid > TC_BQ ? (pos0 + rows_valid - 1 - base) / LP_BK - step0 + 1 : 0;
  int n_steps = max(n_tile[0], n_tile[1]);
  // the CTAs of a cluster share a head's block, or, of fewer steps than split_from, take one each
  if (n_steps < split_from) splits = 1;
  const int head = blockIdx.x / splits, part = blockIdx.x - head * splits;
  if (head >= heads) return;
  if (splits > 1) {                                 // this CTA's steps
    const int per = (n_steps + splits - 1) / splits;
    for (int t = 0; t < 2; ++t) n_tile[t] = max(0, min(per, n_tile[t] - part * per));
    n_steps = max(n_tile[0], n_tile[1]);
    step0 += part * per;
    withhold -= part * per;
  }

  if (threadIdx.x == 0) {
    mbar_init(&q_full, 1);
    for (int b = 0; b < 2; ++b) {
      mbar_init(&k_full[b], 1);
      mbar_init(&v_full[b], 1);
      mbar_init(&k_empty[b], 2);
      mbar_init(&v_empty[b], 2);
    }
    for (int t = 0; t < 2; ++t) {
      for (int b = 0; b < 2; ++b) {
        mbar_init(&s_ready[t][b], 1);
        mbar_init(&s_free[t][b], 4);  // one arrival per softmax warp
      }
      mbar_init(&p_ready[t], 4);
      mbar_init(&o_ready[t], 1);
    }
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  pdl_trigger();
  if (warp == 9) tmem_alloc(&tmem_holder, TMEM_COLS);
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = tmem_holder;
  volatile int* abort = &abort_flag;

  if (warp == 8) {
    // ---------------- producer: the warp as a whole, one elected lane issues the copies
    const bool elected = elect_one();
    pdl_wait();
    const int q_row0 = seq_q_start[seq] + q_first;
    const int row0 = lp_row0(seq_kv_len, seq_q_len, seq, window, lane) + step0 * LP_BK;
    const int q_tiles = n_tile[1] ? 2 : n_steps > 0 ? 1 : 0;
    if (elected && q_tiles) mbar_expect_tx(&q_full, q_tiles * Q_BYTES);
    for (int t = 0; t < q_tiles; ++t)
      for (int c = 0; c < QC; ++c)
        if (elected) tma_load_2d(q_sm + t * Q_BYTES + c * QSUB, &map_q, &q_full, head * (QC * 64) + c * 64, q_row0 + t * TC_BQ);
    int loads[4] = {0, 0, 0, 0};                    // copies started, by buffer (keys, values)
    bool ok = true;
    for (int i = 0; i < n_steps && ok; ++i) {
      const int b = i & 1, row = row0 + i * LP_BK;
      if (i >= 2) ok = __all_sync(0xffffffffu, mbar_wait(&k_empty[b], ((i >> 1) - 1) & 1, abort));
      if (!ok) break;
      if (elected) mbar_expect_tx(&k_full[b], K_BYTES);
      for (int c = 0; c < DC; ++c)
        if (elected) tma_load_2d(k_sm + b * K_BYTES + c * KSUB, &map_kv, &k_full[b], (head * DC + c) * 64, row);
      if (elected) tma_load_2d(k_sm + b * K_BYTES + DC * KSUB, &map_rot, &k_full[b], 0, row);
      loads[b]++;
      if (i >= 2) ok = __all_sync(0xffffffffu, mbar_wait(&v_empty[b], ((i >> 1) - 1) & 1, abort));
      if (!ok) break;
      if (elected) mbar_expect_tx(&v_full[b], V_BYTES);
      if (i == withhold) continue;                  // (tests: this step's values never come)
      for (int c = 0; c < VC; ++c)
        if (elected) tma_load_2d(v_sm + b * V_BYTES + c * KSUB, &map_kv, &v_full[b], (heads * DC + head * VC + c) * 64, row);
      loads[2 + b]++;
    }
    if (*abort && elected) {                        // let the copies in flight land before the block ends
      for (int b = 0; b < 4; ++b) {
        uint64_t* bar = b < 2 ? &k_full[b] : &v_full[b - 2];
        const uint64_t start = now_ns();
        while (loads[b] > 0 && !mbar_try(bar, (loads[b] - 1) & 1) && now_ns() - start < WAIT_LIMIT_NS) {}
      }
      const uint64_t start = now_ns();
      while (q_tiles && !mbar_try(&q_full, 0) && now_ns() - start < WAIT_LIMIT_NS) {}
    }
  } else if (warp == 9 || warp == 10) {
    // ---------------- MMA issuers: warp 9 for tile 0, warp 10 for tile 1
    const int t = warp - 9, n_mine = n_tile[t], n_other = n_tile[1 - t];
    if (n_mine > 0) {
      const bool elected = elect_one();
      const uint32_t idesc_s = instr_desc(LP_BK, 0), idesc_o = instr_desc(VC * 64, 1);
      const uint32_t q_addr = smem_u32(q_sm + t * Q_BYTES), p_addr = smem_u32(p_sm + t * P_BYTES);
      const uint32_t tmem_s = tmem_base + t * 2 * LP_BK, tmem_o = tmem_base + 4 * LP_BK + t * 128;
      auto issue_s = [&](int b) {
        if (elected) {
          const uint32_t k_addr = smem_u32(k_sm + b * K_BYTES);
#pragma unroll
          for (int k = 0; k < QC * 4; ++k)
            umma_bf16(tmem_s + b * LP_BK, smem_desc(q_addr + (k >> 2) * QSUB + (k & 3) * 32, 16),
                      smem_desc(k_addr + (k >> 2) * KSUB + (k & 3) * 32, 16), idesc_s, k > 0 ? 1u : 0u);
          umma_commit(&s_ready[t][b]);
        }
      };
      // V's rows are keys (16 keys = 2048 bytes), its 64-wide chunks KSUB bytes apart
      auto issue_pv = [&](int b, bool first) {
        if (elected) {
          const uint32_t v_addr = smem_u32(v_sm + b * V_BYTES);
#pragma unroll
          for (int k = 0; k < LP_BK / 16; ++k)
            umma_bf16(tmem_o, smem_desc(p_addr + k * 32, 16), smem_desc(v_addr + k * 2048, KSUB), idesc_o,
                      (first && k == 0) ? 0u : 1u);
          umma_commit(&o_ready[t]);
        }
      };
      // a buffer is free after two arrivals, one per tile; a tile that is alone in a step makes both
      auto release = [&](uint64_t* bar, bool alone) {
        if (elected) {
          umma_commit(bar);
          if (alone) umma_commit(bar);
        }
        __syncwarp();
      };
      auto wait_for = [&](uint64_t* bar, uint32_t parity) -> bool { return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort)); };
      bool ok = wait_for(&q_full, 0) && wait_for(&k_full[0], 0);
      if (ok) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        issue_s(0);
        release(&k_empty[0], n_other == 0);
      }
      for (int i = 0; i < n_mine && ok; ++i) {
        const int b = i & 1;
        if (i + 1 < n_mine) {                       // S of the next step, in the other buffer
          const int nb = b ^ 1, use = (i + 1) >> 1;
          ok = wait_for(&k_full[nb], use & 1);
          if (ok && use > 0) ok = wait_for(&s_free[t][nb], (use - 1) & 1);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          issue_s(nb);
          release(&k_empty[nb], i + 1 >= n_other);
        }
        ok = wait_for(&v_full[b], (i >> 1) & 1) && wait_for(&p_ready[t], i & 1);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        issue_pv(b, i == 0);
        release(&v_empty[b], i >= n_other);
      }
    }
  } else if (warp < 8) {
    // ---------------- softmax and output: warps 0-3 own tile 0, warps 4-7 tile 1; thread = query row
    const int t = warp >> 2, quarter = warp & 3, r = quarter * 32 + lane;
    const int pos = pos0 + t * TC_BQ + r;
    const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
    const uint32_t tmem_s = tmem_base + t * 2 * LP_BK + lane_addr, tmem_o = tmem_base + 4 * LP_BK + t * 128 + lane_addr;
    uint8_t* p_row = p_sm + t * P_BYTES + r * 128;
    const int n_mine = n_tile[t];
    float m_ref = -INFINITY, l_run = 0.f;
    const int row_first = window > 0 ? pos - window + 1 : 0;
    pdl_wait();
    bool ok = true;
    for (int i = 0; i < n_mine && ok; ++i) {
      const int b = i & 1;
      ok = mbar_wait(&s_ready[t][b], (i >> 1) & 1, abort);
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const int j0 = base + (step0 + i) * LP_BK;
      float sv[64];
      tmem_load64(tmem_s + b * LP_BK, sv);
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&s_free[t][b]);    // S of this step may be overwritten
      if (j0 + LP_BK - 1 > pos0 + t * TC_BQ || (window > 0 && j0 <= pos0 + t * TC_BQ + TC_BQ - window)) {
#pragma unroll
        for (int e = 0; e < 64; ++e)
          if ((j0 + e > pos) | (j0 + e < row_first)) sv[e] = -INFINITY;
      }
      float mx = -INFINITY, mx2 = -INFINITY;
#pragma unroll
      for (int e = 0; e < 64; e += 2) {
        mx = fmaxf(mx, sv[e]);
        mx2 = fmaxf(mx2, sv[e + 1]);
      }
      mx = fmaxf(mx, mx2) * scale_log2;             // scale_log2 > 0: the maximum commutes with it
      const bool outgrown = mx > m_ref + 8.f;       // also the first keys a row sees (m_ref = -inf)
      if (__any_sync(0xffffffffu, outgrown)) {
        // a new reference: rescale what has been accumulated
        const float m_new = fmaxf(m_ref, mx);
        const float alpha = m_ref == -INFINITY ? 1.f : fast_exp2(m_ref - m_new);
        if (i > 0) {
          ok = mbar_wait(&o_ready[t], (i - 1) & 1, abort);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
          for (int c = 0; c < VC * 64; c += 32) {
            float ov[32];
            tmem_load32(tmem_o + c, ov);
#pragma unroll
            for (int e = 0; e < 32; ++e) ov[e] *= alpha;
            tmem_store32(tmem_o + c, ov);
          }
          asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        }
        l_run *= alpha;
        m_ref = m_new;
      }
      const float m_use = m_ref == -INFINITY ? 0.f : m_ref;
      float rs = 0.f, rs_hi = 0.f;
      uint32_t pk[32];
#pragma unroll
      for (int e = 0; e < 32; ++e) {
        float x0, x1;
        fma2(x0, x1, sv[2 * e], sv[2 * e + 1], scale_log2, -m_use);
        __nv_bfloat162 two = __floats2bfloat162_rn(fast_exp2(x0), fast_exp2(x1));
        pk[e] = *reinterpret_cast<uint32_t*>(&two);
        // (the sum is of the weights as they multiply the values, so that their roundings cancel where one key has most of the weight)
        add2(rs, rs_hi, __uint_as_float(pk[e] << 16), __uint_as_float(pk[e] & 0xffff0000u));
      }
      // P's tile is free once PV of the step before has finished
      if (i > 0) ok = mbar_wait(&o_ready[t], (i - 1) & 1, abort);
      if (!ok) break;
      // K-major A operand: 16-byte column c ^ (r % 8) of row r
#pragma unroll
      for (int c = 0; c < 8; ++c)
        *reinterpret_cast<uint4*>(p_row + ((c ^ (r & 7)) << 4)) = make_uint4(pk[4 * c], pk[4 * c + 1], pk[4 * c + 2], pk[4 * c + 3]);
      l_run += rs + rs_hi;
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_ready[t]);
    }
    if (ok && n_mine > 0) ok = mbar_wait(&o_ready[t], (n_mine - 1) & 1, abort);
    if (splits > 1) {
      if constexpr (DC == 2 || VC == 1) {
        ml[t * TC_BQ + r] = n_mine > 0 ? make_float2(m_ref, l_run) : make_float2(-INFINITY, 0.f);
        if (ok && n_mine > 0) {
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
          for (int c = 0; c < VC * 64; c += 32) {
            float ov[32];
            tmem_load32(tmem_o + c, ov);
#pragma unroll
            for (int d = 0; d < 32; d += 4)
              *reinterpret_cast<float4*>(part_piece<32, VC * 64>(p_sm + t * P_BYTES, q_sm + t * Q_BYTES, r, (c + d) / 4)) =
                  make_float4(ov[d], ov[d + 1], ov[d + 2], ov[d + 3]);
          }
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        }
      }
    } else if (ok && n_mine > 0) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const bool valid = t * TC_BQ + r < rows_valid;
      // the sink joins at the end, so that the weights are relative to a key's score: the largest of the first step is one exactly
      float inv = 1.f / l_run;
      if (sink) {
        const float own = sink[head] * 1.4426950408889634f, top = fmaxf(m_ref, own), f = fast_exp2(m_ref - top);
        inv = f / (l_run * f + fast_exp2(own - top));
      }
      const size_t row = (size_t)seq_q_start[seq] + q_first + t * TC_BQ + r;
      bf16* dst = out + row * ((size_t)heads * (VC * 64)) + (size_t)head * (VC * 64);
      const bf16* gate_row = gate + (gate ? row * gate_ld + (size_t)head * (VC * 64) : 0);
#pragma unroll 1
      for (int c = 0; c < VC * 64; c += 32) {
        float ov[32];
        tmem_load32(tmem_o + c, ov);
        if (valid) {
#pragma unroll
          for (int d = 0; d < 32; d += 8) {
#pragma unroll
            for (int e = 0; e < 8; ++e) ov[d + e] *= inv;
            if (gate) gate8(ov + d, gate_row + c + d);
            uint32_t w[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              __nv_bfloat162 two = __floats2bfloat162_rn(ov[d + 2 * e], ov[d + 2 * e + 1]);
              w[e] = *reinterpret_cast<uint32_t*>(&two);
            }
            *reinterpret_cast<uint4*>(dst + c + d) = make_uint4(w[0], w[1], w[2], w[3]);
          }
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    }
  }

  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  if constexpr (DC == 2 || VC == 1) {
    if (splits > 1) {
      cluster_barrier();
      if (threadIdx.x < 2 * TC_BQ) {
        const size_t stride = (size_t)heads * (VC * 64);
        merge_parts<32, VC * 64, Q_BYTES, P_BYTES>(
            q_sm, p_sm, ml, part, splits, rows_valid, VC * 64,
            out + ((size_t)seq_q_start[seq] + q_first) * stride + (size_t)head * (VC * 64), stride, [&](int, float ref, float sum) {
              if (!sink) return 1.f / sum;
              const float own = sink[head] * 1.4426950408889634f, top = fmaxf(ref, own), f = fast_exp2(ref - top);
              return f / (sum * f + fast_exp2(own - top));
            }, gate ? gate + ((size_t)seq_q_start[seq] + q_first) * gate_ld + (size_t)head * (VC * 64) : nullptr, gate_ld);
      }
      cluster_barrier();                            // nobody leaves while others read from it
    }
  }
  __syncthreads();
  if (warp == 9) {
    __syncwarp();
    tmem_free(tmem_holder, TMEM_COLS);
  }
  if (threadIdx.x == 0 && abort_flag && status) atomicOr(status, 16);
}

template <int DC, int VC>
static int lp_launch(const CUtensorMap& mq, const CUtensorMap& mkv, const CUtensorMap& mr, void* out, const int* seq_q_start,
                     const int* seq_q_len, const int* seq_kv_len, const int* block_seq, const int* block_first, int n_blocks,
                     int heads, float scale, int window, const float* sink, int* status, int withhold, int split,
                     const bf16* gate, int gate_ld, cudaStream_t s) {
  const int smem = 2 * (DC + 1) * 128 * 128 + 2 * 128 * 128 + 2 * (DC + 1 + VC) * 64 * 128 + 1024;
  cudaError_t err = cudaFuncSetAttribute(latent_prompt_kernel<DC, VC>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (err != cudaSuccess) return (int)err;
  const int parts = split & 255, splits = DC == 1 && VC == 2 ? 1 : parts >= 4 ? 4 : parts >= 2 ? 2 : 1, split_from = split >> 8;
  return launch_dependent_cluster(latent_prompt_kernel<DC, VC>, dim3(heads * splits, n_blocks), dim3(LP_THREADS), smem, s, dim3(splits),
                                  mq, mkv, mr, (bf16*)out, seq_q_start, seq_q_len, seq_kv_len, block_seq, block_first, heads,
                                  scale * 1.4426950408889634f, window, sink, status, withhold, splits, split_from, gate, gate_ld);
}

static int lp_run(const void* q, const void* kv, const void* shared, void* out, const int* seq_q_start, const int* seq_q_len,
                  const int* seq_kv_len, const int* block_seq, const int* block_first, int n_blocks, int n_tokens, int rows,
                  int heads, int dim, int vdim, float scale, int window, const float* sink, int* status, int withhold,
                  int splits, const bf16* gate, int gate_ld, cudaStream_t s) {
  if (n_blocks == 0 || n_tokens == 0) return 0;
  if ((dim != 64 && dim != 128) || (vdim != 64 && vdim != 128) || !(scale > 0.f) || n_blocks > 65535) return -2;
  if (((uintptr_t)q | (uintptr_t)kv | (uintptr_t)shared | (uintptr_t)out | (uintptr_t)gate) & 15 || gate_ld % 8) return -2;
  CUtensorMap mq, mkv, mr;
  int rc = sb_make_map(&mq, q, n_tokens, (long long)heads * (dim + 64), TC_BQ);
  if (rc) return rc;
  rc = sb_make_map(&mkv, kv, rows, (long long)heads * (dim + vdim), LP_BK);
  if (rc) return rc;
  rc = sb_make_map(&mr, shared, rows, 64, LP_BK);
  if (rc) return rc;
#define ARGS mq, mkv, mr, out, seq_q_start, seq_q_len, seq_kv_len, block_seq, block_first, n_blocks, heads, scale, window, sink, status, withhold, splits, gate, gate_ld, s
  if (dim == 128) return vdim == 128 ? lp_launch<2, 2>(ARGS) : lp_launch<2, 1>(ARGS);
  return vdim == 128 ? lp_launch<1, 2>(ARGS) : lp_launch<1, 1>(ARGS);
#undef ARGS
}

extern "C" {

// c: [rows, rank]; shared: [rows, rot]; rows: over the sequences, the keys from the first that a query of the step sees on (all,
// without a window), each rounded up to a multiple of 64; max_rows: the most of one sequence.  q: null, or [n_tokens, heads * (dim + 64)],
// the last 64 entries of whose heads are turned in place, entry 2 i with 2 i + 1 (16-byte aligned, tables of whole 16-byte pieces).
int sb_latent_gather(const void* store, const int* block_table, int table_stride, const int* seq_slot, const int* seq_q_len,
                     const int* seq_kv_len, int n_seqs, int max_rows, void* c, void* shared, int rank, int rot, int window, void* q,
                     const float* cos_t, const float* sin_t, int table_width, const int* tok_pos, int n_tokens, int heads, int dim,
                     cudaStream_t s) {
  if (n_seqs == 0 || max_rows == 0) return 0;
  if (rank % 8 || rot % 8 || n_seqs > 65535 || (((uintptr_t)store | (uintptr_t)c | (uintptr_t)shared) & 15)) return -2;
  LatentTurn turn = {nullptr, nullptr, nullptr, nullptr, 0, 0, 0, 0};
  const int x = (max_rows + 7) / 8;
  long long extra = 0;
  if (q) {
    if (dim % 8 || table_width % 4 || table_width < 32 || (((uintptr_t)q | (uintptr_t)cos_t | (uintptr_t)sin_t) & 15)) return -2;
    turn = LatentTurn{(bf16*)q, cos_t, sin_t, tok_pos, table_width, heads, dim, (long long)n_tokens * heads * 8};
    extra = ((turn.pieces + 255) / 256 + x - 1) / x;
    if (n_seqs + extra > 65535) return -2;
  }
  return launch_dependent(latent_gather_kernel, dim3(x, (unsigned)(n_seqs + extra)), dim3(256), 0, s, (const bf16*)store, block_table,
                          table_stride, seq_slot, seq_q_len, seq_kv_len, (bf16*)c, (bf16*)shared, rank, rot, window, n_seqs, turn);
}

// q: [n_tokens, heads * (dim + 64)], the last 64 entries of a head turned; kv: [rows, heads * dim + heads * vdim]; shared:
// [rows, 64]; out: [n_tokens, heads * vdim], with a gate (rows of gate_ld entries, those of a head's values in out's order; null: none)
// times its sigmoid; block_seq / block_first: blocks of 256 queries; dim and vdim 64 or 128; scale > 0.  splits: 1, 2 or 4 CTAs that share
// a block's keys, in its higher bytes the least steps of 64 keys of a block that they share (shorter ones go to one CTA).
int sb_latent_prompt(const void* q, const void* kv, const void* shared, void* out, const int* seq_q_start, const int* seq_q_len,
                     const int* seq_kv_len, const int* block_seq, const int* block_first, int n_blocks, int n_tokens, int rows,
                     int heads, int dim, int vdim, float scale, int window, const float* sink, int* status, int splits,
                     const void* gate, int gate_ld, cudaStream_t s) {
  return lp_run(q, kv, shared, out, seq_q_start, seq_q_len, seq_kv_len, block_seq, block_first, n_blocks, n_tokens, rows, heads,
                dim, vdim, scale, window, sink, status, -1, splits, (const bf16*)gate, gate_ld, s);
}

// The same with the values of step `step` (64 keys) of every block left out: the waits on them give up after wait_limit_ns, the
// kernel returns, the status bit is set and out is undefined.  For tests.
int sb_latent_prompt_withheld(const void* q, const void* kv, const void* shared, void* out, const int* seq_q_start, const int* seq_q_len,
                              const int* seq_kv_len, const int* block_seq, const int* block_first, int n_blocks, int n_tokens, int rows,
                              int heads, int dim, int vdim, float scale, int window, const float* sink, int* status, int splits,
                              const void* gate, int gate_ld, int step, unsigned long long wait_limit_ns, cudaStream_t s) {
  if (step < 0 || wait_limit_ns == 0) return -2;
  const unsigned long long usual = WAIT_LIMIT_NS;
  cudaMemcpyToSymbolAsync(tc_wait_limit_ns, &wait_limit_ns, sizeof(usual), 0, cudaMemcpyHostToDevice, s);
  const int rc = lp_run(q, kv, shared, out, seq_q_start, seq_q_len, seq_kv_len, block_seq, block_first, n_blocks, n_tokens, rows,
                        heads, dim, vdim, scale, window, sink, status, step, splits, (const bf16*)gate, gate_ld, s);
  cudaMemcpyToSymbolAsync(tc_wait_limit_ns, &usual, sizeof(usual), 0, cudaMemcpyHostToDevice, s);
  return rc;
}

}  // extern "C"
