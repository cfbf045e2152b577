// Causal grouped-query attention for prompts on the fifth-generation tensor cores (bfloat16).
//
// A block takes 256 consecutive query tokens of one sequence and one query head as two tiles of 128.
// Both products of a tile run as tcgen05.mma with the accumulators in tensor memory:
//     S  = Q K^T     M = 128 queries, N = 128 keys,  K = head_dim   (Q and K K-major)
//     O += P V       M = 128 queries, N = head_dim,  K = 128 keys   (V as it lies in the cache:
//                                                                    keys x head_dim, "MN-major")
// Tensor memory holds S of both tiles (2 x 128 columns) and O of both tiles (2 x 128 columns).
//
// Warps:   0-3 softmax of tile 0, 4-7 softmax of tile 1 (thread = query row = TMEM lane, so the
//          online softmax needs no shuffle: engine/kernels/fused.py:288-312),
//          8 TMA producer, 9 and 10 the MMA issuers of tile 0 and tile 1.
// TMA brings both Q tiles once and, per step of 128 keys (two cache pages), K and V with the
// 128-byte swizzle the tensor core reads; the keys alternate between two buffers and run a step
// ahead of the values, which have one buffer, because S of step i+1 is issued as soon as the softmax
// warps have read S of step i out of tensor memory, while PV of step i has to wait for P.
// The softmax warps write P = exp2(S * scale - m), rounded to bfloat16 (fused.py:699-701), into
// shared memory as the A operand of PV.  O stays in tensor memory and is accumulated by the MMA
// itself: m is the reference of the step before as long as no row's maximum outgrows it by more
// than 2^8 (P stays far inside bfloat16's range, the sum is kept in float); only then is O read,
// rescaled and written back, and the step's P redone.  The result is O / l, as in the exact online
// softmax, up to rounding.
// Keys are read from the cache like in every other attention kernel of this library, so a chunk
// that continues a sequence needs nothing special: a query at absolute position p sees keys j <= p
// (engine/engine.py:781-787) and, with a window w, j > p - w.
//
// The same kernel also serves attention whose positions enter through the scores and the mask (EXT, see
// attention_sink.cu): the penalty r1 log2(1 + r2 (p - j)) is taken off a score as it leaves tensor
// memory (S is unscaled there, so the penalty is divided by the scale first); a row masks the keys
// before its own chunk; the sink is the state a row's softmax starts from (reference = sink log2(e),
// sum = 1); the gate multiplies the row's result; scores may be capped (softcap.cuh); a window may keep the
// sequence's first keys visible, whose pages then come in front of the window's in the walk.  The queries may
// lie at the front of wider rows (a stacked projection): the tensor map of Q covers those rows.
// Keys and values have sizes of their own there, up to 128 each, in shared-memory tiles of one or two 64-entry
// chunks.  Entries of a key or a value behind the real ones arrive as the zeros TMA fills in: they take what lies
// behind a query's own entries (its neighbour's) out of S, and the output columns they give are not stored.
// (Loops over the real sizes would make the one lane that issues the products form every descriptor anew.)
//
// Few blocks of queries over many keys: `splits` CTAs, a cluster, walk a part of a block's keys each and merge (attention_tc.cuh).
//
// Every wait on an mbarrier gives up after WAIT_LIMIT_NS, raises bit 16 of *status and lets the
// block drain its copies, free its tensor memory and return.
#include <cuda.h>

#include "attention_tc.cuh"
#include "common.cuh"
#include "softcap.cuh"
#include "tensor_map.cuh"

#define TC_BK 128
#define TC_THREADS 352
#define TC_RING 3

// What the EXT instance takes besides: r1, r2 (float [heads], both or neither), sink (float [heads] or null),
// gate (float [tokens, heads] or null), chunk (0: none), keep (the first keys a window or chunk keeps visible), the
// cap of the scores as scale / cap and cap / scale (S is scaled after it; 0: none), the entries of a key and a value.
struct TcExtras {
  const float* r1;
  const float* r2;
  const float* sink;
  const float* gate;
  int chunk;
  int keep;
  float cap_in, cap_out;
  int dim, vdim;
};

// EXT 0: plain; 1: the extras without the cap; 2: all of them.
template <int DC, int VC, int EXT, bool PARTS>
__global__ void __launch_bounds__(TC_THREADS, 1)
attention_prefill_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                            const __grid_constant__ CUtensorMap map_v, bf16* __restrict__ out,
                            const int* __restrict__ block_table, int table_stride,
                            const int* __restrict__ seq_slot, const int* __restrict__ seq_q_start,
                            const int* __restrict__ seq_q_len, const int* __restrict__ seq_kv_len,
                            const int* __restrict__ tile_seq, const int* __restrict__ tile_first,
                            int heads, int kv_heads, float scale_log2, int window, int* status, int list_of_blocks,
                            int splits, TcExtras ex) {
  // DC, VC: 64-element (128-byte) chunks of a key and of a value
  constexpr bool CAP = EXT == 2;
  const int dim = EXT ? ex.dim : DC * 64, vdim = EXT ? ex.vdim : VC * 64;
  constexpr int SUB = 128 * 128;                    // bytes of a [128 rows x 128 bytes] sub-tile
  constexpr int Q_BYTES = DC * SUB;                 // one tile of 128 queries
  constexpr int KV_BYTES = (DC > VC ? DC : VC) * SUB;   // room for the keys (or values) of 128 tokens
  constexpr int P_BYTES = 2 * SUB;                  // [128 queries x 128 keys] bfloat16
  constexpr uint32_t TMEM_COLS = 512;               // S of both tiles: 2 x 128; O of both tiles: 2 x 128
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* q_sm = smem;                             // 2 tiles
  uint8_t* p_sm = q_sm + 2 * Q_BYTES;               // 2 tiles
  uint8_t* ring = p_sm + 2 * P_BYTES;               // buffers 0 and 1: keys of even and odd steps; 2: values
  __shared__ uint64_t q_full, full[TC_RING], empty[TC_RING], s_ready[2], s_free[2], p_ready[2], o_ready[2];
  __shared__ uint32_t tmem_holder;
  __shared__ int abort_flag;
  float2 row_state = make_float2(-INFINITY, 0.f);   // keys in parts: a row's reference and sum

  // heads run fastest: the work list's order holds; the CTAs of a cluster share a head's block
  const int tile = blockIdx.y, head = PARTS ? blockIdx.x / splits : blockIdx.x, part = PARTS ? blockIdx.x - head * splits : 0;
  const int q_first = tile_first[tile];
  // the work list is either this kernel's own (one entry per block of 256 queries) or the common
  // one in tiles of 64 queries, of which every fourth starts a block
  if (!list_of_blocks && (q_first & 255)) return;
  const int seq = tile_seq[tile];
  const int q_len = seq_q_len[seq], kv_len = seq_kv_len[seq];
  const int rows_valid = min(2 * TC_BQ, q_len - q_first);
  const int pos0 = kv_len - q_len + q_first;
  const int kvh = head / (heads / kv_heads);
  const int* pages = block_table + (size_t)seq_slot[seq] * table_stride;
  // the warp's number as a value the compiler knows to be the same in every lane
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;

  const int hi = pos0 + rows_valid - 1;
  int lo = 0;
  if (window > 0 && pos0 - window + 1 > 0) lo = pos0 - window + 1;
  if (EXT && ex.chunk > 0 && pos0 / ex.chunk * ex.chunk > lo) lo = pos0 / ex.chunk * ex.chunk;
  const int page_lo = lo / SB_PAGE_TOKENS, page_hi = hi / SB_PAGE_TOKENS;
  // the walk's pages: those of kept keys in front of page_lo, then page_lo and on
  const int kept = EXT && ex.keep > 0 ? min((ex.keep + SB_PAGE_TOKENS - 1) / SB_PAGE_TOKENS, page_lo) : 0;
  auto page_of = [&](int n) { return EXT && n < kept ? n : page_lo + n - kept; };
  // steps of two pages (128 keys) that each tile of 128 queries needs
  int n_tile[2];
  n_tile[0] = ((pos0 + min(rows_valid, TC_BQ) - 1) / SB_PAGE_TOKENS - page_lo + kept) / 2 + 1;
  n_tile[1] = rows_valid > TC_BQ ? (page_hi - page_lo + kept) / 2 + 1 : 0;
  int n_steps = max(n_tile[0], n_tile[1]), first_step = 0;
  if constexpr (PARTS) {                            // this CTA's steps
    const int per = (n_steps + splits - 1) / splits;
    first_step = part * per;
    for (int t = 0; t < 2; ++t) n_tile[t] = max(0, min(per, n_tile[t] - first_step));
    n_steps = max(n_tile[0], n_tile[1]);
  }

  if (threadIdx.x == 0) {
    mbar_init(&q_full, 1);
    for (int s = 0; s < TC_RING; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 2); }
    for (int t = 0; t < 2; ++t) {
      mbar_init(&s_ready[t], 1);
      mbar_init(&s_free[t], 4);       // one arrival per softmax warp
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
    // ---------------- producer: the whole warp walks the schedule, one elected lane issues the
    // copies (addresses and coordinates are then the same in every lane and can live in the uniform
    // registers the copy instructions want; run by one lane inside a branch on the lane number, each
    // copy costs over a hundred cycles to issue)
    {
      const bool elected = elect_one();
      pdl_wait();
      const int q_row0 = seq_q_start[seq] + q_first;
      const int q_tiles = n_tile[1] ? 2 : !PARTS || n_steps > 0 ? 1 : 0;
      if (elected && q_tiles) mbar_expect_tx(&q_full, q_tiles * Q_BYTES);
      for (int t = 0; t < q_tiles; ++t)
        for (int c = 0; c < DC; ++c)
          if (elected) tma_load_2d(q_sm + t * Q_BYTES + c * SUB, &map_q, &q_full, head * dim + c * 64, q_row0 + t * TC_BQ);
      // Keys alternate between buffers 0 and 1 and run a step ahead of the values, which have
      // buffer 2: K0 V0 K1 | K2 V1 | K3 V2 ...  (S of step i+1 is issued early in step i, PV late.)
      auto load = [&](bool is_v, int i) -> bool {
        const int b = is_v ? 2 : (i & 1), use = is_v ? i : (i >> 1);
        if (use > 0 && !__all_sync(0xffffffffu, mbar_wait(&empty[b], (use - 1) & 1, abort))) return false;
        const int chunks = is_v ? VC : DC;
        if (elected) mbar_expect_tx(&full[b], chunks * SUB);
        const bool withheld = is_v && first_step + i == *(volatile int*)&tc_withhold_step;   // tests only
        for (int half = 0; half < (withheld ? 1 : 2); ++half) {
          const int page = pages[min(page_of(2 * (first_step + i) + half), page_hi)];
          const int row = (page * kv_heads + kvh) * SB_PAGE_TOKENS;
          for (int c = 0; c < chunks; ++c)
            if (elected) tma_load_2d(ring + b * KV_BYTES + c * SUB + half * 8192, is_v ? &map_v : &map_k, &full[b], c * 64, row);
        }
        return true;
      };
      int loads[3] = {0, 0, 0};                        // per buffer: how many copies were started
      bool ok = (!PARTS || n_steps > 0) && load(false, 0);
      if (ok) { loads[0]++; ok = load(true, 0); }
      if (ok) loads[2]++;
      if (ok && n_steps > 1) { ok = load(false, 1); if (ok) loads[1]++; }
      for (int i = 1; i < n_steps && ok; ++i) {
        if (i + 1 < n_steps) { ok = load(false, i + 1); if (ok) loads[(i + 1) & 1]++; }
        if (ok) { ok = load(true, i); if (ok) loads[2]++; }
      }
      if (*abort && elected) {                         // let the copies in flight land before the block ends
        for (int b = 0; b < 3; ++b) {
          const uint64_t start = now_ns();
          while (loads[b] > 0 && !mbar_try(&full[b], (loads[b] - 1) & 1) && now_ns() - start < WAIT_LIMIT_NS) {}
        }
      }
    }
  } else if (warp == 9 || warp == 10) {
    // ---------------- MMA issuers: warp 9 for tile 0, warp 10 for tile 1.  Each runs its own chain
    // of waits, so that one tile's waiting does not hold up the other's products.
    const int t = warp - 9, n_mine = n_tile[t], n_other = n_tile[1 - t];
    if (n_mine > 0) {
      // the whole warp waits and computes descriptors; one elected lane issues (see the producer)
      const bool elected = elect_one();
      const uint32_t idesc_s = instr_desc(TC_BK, 0), idesc_o = instr_desc(VC * 64, 1);
      const uint32_t q_addr = smem_u32(q_sm + t * Q_BYTES), p_addr = smem_u32(p_sm + t * P_BYTES);
      // S = Q K^T: k runs over the head in steps of 16 (32 bytes inside a 128-byte chunk)
      auto issue_s = [&](int buf) {
        if (elected) {
#pragma unroll
          for (int k = 0; k < DC * 4; ++k) {
            const uint32_t off = (k >> 2) * SUB + (k & 3) * 32;
            umma_bf16(tmem_base + t * TC_BK, smem_desc(q_addr + off, 16),
                      smem_desc(smem_u32(ring + buf * KV_BYTES) + off, 16), idesc_s, k > 0 ? 1u : 0u);
          }
          umma_commit(&s_ready[t]);
        }
      };
      // O (+)= P V: k runs over the 128 keys in steps of 16; P K-major (two 64-key chunks); V's
      // rows are keys (16 keys = 2048 bytes), its 64-wide chunks of the head are SUB bytes apart
      auto issue_pv = [&](bool first) {
        if (elected) {
#pragma unroll
          for (int k = 0; k < TC_BK / 16; ++k) {
            const uint32_t a_off = (k >> 2) * SUB + (k & 3) * 32;
            umma_bf16(tmem_base + 2 * TC_BK + t * 128, smem_desc(p_addr + a_off, 16),
                      smem_desc(smem_u32(ring + 2 * KV_BYTES) + k * 2048, SUB), idesc_o,
                      (first && k == 0) ? 0u : 1u);
          }
          umma_commit(&o_ready[t]);
        }
      };
      // A buffer is free after two arrivals, one per tile; a tile that is alone in a step makes both.
      auto release = [&](int buf, bool alone) {
        if (elected) {
          umma_commit(&empty[buf]);
          if (alone) umma_commit(&empty[buf]);
        }
        __syncwarp();
      };
      // every lane waits; the warp goes on together or stops together
      auto wait2 = [&](uint64_t* first_bar, uint32_t first_parity, uint64_t* second_bar, uint32_t second_parity) -> bool {
        const bool got = mbar_wait(first_bar, first_parity, abort) && mbar_wait(second_bar, second_parity, abort);
        return __all_sync(0xffffffffu, got);
      };
      bool ok = wait2(&q_full, 0, &full[0], 0);
      if (ok) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        issue_s(0);
        release(0, n_other == 0);
      }
      // Step i: S of step i+1 as soon as the softmax warps have read S of step i out of tensor
      // memory (they are still busy with its exponentials), then PV of step i when P is written.
      for (int i = 0; i < n_mine && ok; ++i) {
        if (i + 1 < n_mine) {
          const int kb = (i + 1) & 1;                  // buffer of K(i+1); V(i) is in buffer 2
          ok = wait2(&full[kb], ((i + 1) >> 1) & 1, &s_free[t], i & 1);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          issue_s(kb);
          release(kb, i + 1 >= n_other);
        }
        ok = wait2(&full[2], i & 1, &p_ready[t], i & 1);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        issue_pv(i == 0);
        release(2, i >= n_other);
      }
    }
  } else if (warp < 8) {
    // ---------------- softmax and output: warps 0-3 own tile 0, warps 4-7 tile 1; thread = query
    // row = TMEM lane.  The running output stays in tensor memory; it is rescaled only when a row's
    // maximum has grown by more than 2^8 since the last rescale, so most steps only produce P.
    const int t = warp >> 2;
    const int quarter = warp & 3;
    const int r = quarter * 32 + lane;
    const int pos = pos0 + t * TC_BQ + r;
    const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
    const uint32_t tmem_s = tmem_base + t * TC_BK + lane_addr;
    const uint32_t tmem_o = tmem_base + 2 * TC_BK + t * 128 + lane_addr;
    uint8_t* p_row = p_sm + t * P_BYTES + r * 128;
    const int n_mine = n_tile[t];
    float m_ref = -INFINITY, l_run = 0.f;
    // EXT: the first key of the row's own chunk, the first key of the chunk of the tile's last row, the
    // penalty's two numbers (the first over the scale, because S is scaled after it), the sink
    int row_lo = 0, tile_lo = 0;
    float pen1 = 0.f, pen2 = 0.f;
    if (EXT) {
      if (ex.chunk > 0) {
        row_lo = pos / ex.chunk * ex.chunk;
        tile_lo = (pos0 + t * TC_BQ + TC_BQ - 1) / ex.chunk * ex.chunk;
      }
      if (ex.r1) {
        pen1 = ex.r1[head] / scale_log2;
        pen2 = ex.r2[head];
      }
      if (ex.sink && part == 0) {
        m_ref = ex.sink[head] * 1.4426950408889634f;
        l_run = 1.f;
      }
    }
    const int row_first = max(row_lo, window > 0 ? pos - window + 1 : 0);
    const uint32_t gap = EXT ? (uint32_t)max(row_first - ex.keep, 0) : 0u;
    float series[6];
    if (CAP) cap_series(ex.cap_in, ex.cap_out, series);
    pdl_wait();
    bool ok = true;
    for (int i = 0; i < n_mine && ok; ++i) {
      ok = mbar_wait(&s_ready[t], i & 1, abort);
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      // the first keys of the step's two pages (neighbours, but for the step between the kept pages and the others)
      const int jp[2] = {page_of(2 * (first_step + i)) * SB_PAGE_TOKENS,
                         page_of(2 * (first_step + i) + 1) * SB_PAGE_TOKENS};
      const bool edge = jp[1] + SB_PAGE_TOKENS - 1 > pos0 + t * TC_BQ ||
                        (window > 0 && jp[0] <= pos0 + t * TC_BQ + TC_BQ - window) || (EXT && jp[0] < tile_lo);
      float sv[64];
      float rs = 0.f, rs_hi = 0.f;                   // the row sum in two halves (packed adds)
      // half h of the row of S from tensor memory, masked where the step touches an edge
      auto load_half = [&](int h) {
        tmem_load64(tmem_s + h * 64, sv);
        const int j0 = h ? jp[1] : jp[0];
        if (CAP) cap64(sv, ex.cap_in, ex.cap_out, series);
        if (EXT && ex.r1) {
          const float far = (float)(pos - j0);                // the distance to this half's first key
#pragma unroll
          for (int e = 0; e < 64; ++e)
            sv[e] -= pen1 * __log2f(fmaf(pen2, fmaxf(far - (float)e, 0.f), 1.f));
        }
        if (edge) {
#pragma unroll
          for (int e = 0; e < 64; ++e) {
            const int j = j0 + e;
            if constexpr (EXT != 0) {
              // hidden: what comes later, and the gap between the kept keys and the row's first key (without a
              // branch: the nested conditions compiled to branches doubled the time of a windowed prompt)
              if ((j > pos) | ((uint32_t)(j - ex.keep) < gap)) sv[e] = -INFINITY;
            } else if (j > pos || (window > 0 && j <= pos - window)) {
              sv[e] = -INFINITY;
            }
          }
        }
      };
      if constexpr (CAP) {
        // Half after half, one piece of code for both and for what is done again.  As straight code (below) the capped kernel spills
        // 230 bytes a thread, and a block's first steps take as long to fetch as to run: 2,048 tokens of window 1,024 47.7 us against
        // 44.5 here, 500 tokens 21.5 / 19.9, 150 tokens 13.3 / 11.8.  Without the cap the exponentials are the bound and the votes
        // between them cost more: 2,000 tokens 35.3 us straight, 39.8 this way.
#pragma unroll 1
        for (int h = 0; h < 2; ++h) {
          load_half(h);
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
              for (int c = 0; c < vdim; c += 32) {
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
            if (h == 1) {                               // the first half again, on the new reference
              rs = rs_hi = 0.f;
              h = -1;
              continue;
            }
          }
          if (h == 1) {                                 // S of this step may be overwritten
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&s_free[t]);
          }
          const float m_use = m_ref == -INFINITY ? 0.f : m_ref;
          uint32_t pk[32];                              // P = exp2(S * scale - m), rounded to bfloat16
#pragma unroll
          for (int e = 0; e < 32; ++e) {
            float x0, x1;
            fma2(x0, x1, sv[2 * e], sv[2 * e + 1], scale_log2, -m_use);
            const float p0 = fast_exp2(x0), p1 = fast_exp2(x1);
            add2(rs, rs_hi, p0, p1);
            __nv_bfloat162 two = __floats2bfloat162_rn(p0, p1);
            pk[e] = *reinterpret_cast<uint32_t*>(&two);
          }
          // P's tile is free once PV of the step before has finished
          if (h == 0 && i > 0) ok = mbar_wait(&o_ready[t], (i - 1) & 1, abort);
          if (!ok) break;
          // K-major A operand: 64-key chunk h, 16-byte column c ^ (r % 8) of row r
#pragma unroll
          for (int c = 0; c < 8; ++c)
            *reinterpret_cast<uint4*>(p_row + h * SUB + ((c ^ (r & 7)) << 4)) =
                make_uint4(pk[4 * c], pk[4 * c + 1], pk[4 * c + 2], pk[4 * c + 3]);
        }
        if (!ok) break;
      } else {
        uint32_t pk[32];
        float mx = -INFINITY, m_use = m_ref == -INFINITY ? 0.f : m_ref;
        // P = exp2(S * scale - m) of 8 keys, rounded to bfloat16: one 16-byte column of the A operand
        auto exp8 = [&](int c, uint32_t* w) {
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            float x0, x1;
            fma2(x0, x1, sv[c * 8 + 2 * e], sv[c * 8 + 2 * e + 1], scale_log2, -m_use);
            const float p0 = fast_exp2(x0), p1 = fast_exp2(x1);
            add2(rs, rs_hi, p0, p1);
            __nv_bfloat162 two = __floats2bfloat162_rn(p0, p1);
            w[e] = *reinterpret_cast<uint32_t*>(&two);
          }
        };
        // K-major A operand: 64-key chunk h, 16-byte column c ^ (r % 8) of row r
        auto store8 = [&](int h, int c, const uint32_t* w) {
          *reinterpret_cast<uint4*>(p_row + h * SUB + ((c ^ (r & 7)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
        };
        auto s_consumed = [&]() {                        // S of this step may be overwritten
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) mbar_arrive(&s_free[t]);
        };
        // One pass in the common case: the exponent's reference is the one of the step before, which
        // is good as long as no row's maximum outgrows it by more than 2^8.
        load_half(0);
#pragma unroll
        for (int e = 0; e < 64; ++e) mx = fmaxf(mx, sv[e]);
#pragma unroll
        for (int c = 0; c < 8; ++c) exp8(c, pk + 4 * c);
        load_half(1);
#pragma unroll
        for (int e = 0; e < 64; ++e) mx = fmaxf(mx, sv[e]);
        mx *= scale_log2;                               // scale_log2 > 0: the maximum commutes with it
        const bool outgrown = mx > m_ref + 8.f;         // also the first keys a row sees (m_ref = -inf)
        if (!__any_sync(0xffffffffu, outgrown)) {
          s_consumed();
          // P's tile and O are free once PV of the step before has finished
          if (i > 0) ok = mbar_wait(&o_ready[t], (i - 1) & 1, abort);
          if (!ok) break;
#pragma unroll
          for (int c = 0; c < 8; ++c) store8(0, c, pk + 4 * c);
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            uint32_t w[4];
            exp8(c, w);
            store8(1, c, w);
          }
        } else {
          // a new reference: rescale what has been accumulated, then redo this step's P
          const float m_new = fmaxf(m_ref, mx);
          const float alpha = m_ref == -INFINITY ? 1.f : fast_exp2(m_ref - m_new);
          if (i > 0) {
            ok = mbar_wait(&o_ready[t], (i - 1) & 1, abort);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
            for (int c = 0; c < vdim; c += 32) {
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
          m_use = m_ref == -INFINITY ? 0.f : m_ref;
          rs = 0.f;
          rs_hi = 0.f;
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            uint32_t w[4];
            exp8(c, w);
            store8(1, c, w);
          }
          load_half(0);
          s_consumed();
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            uint32_t w[4];
            exp8(c, w);
            store8(0, c, w);
          }
        }
      }
      l_run += rs + rs_hi;
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_ready[t]);
    }
    if (ok && n_mine > 0) ok = mbar_wait(&o_ready[t], (n_mine - 1) & 1, abort);
    if constexpr (PARTS) {
      if (n_mine > 0) row_state = make_float2(m_ref, l_run);
      if (ok && n_mine > 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
        for (int c = 0; c < VC * 64; c += 32) {
          float ov[32];
          tmem_load32(tmem_o + c, ov);
#pragma unroll
          for (int d = 0; d < 32; d += 4)
            *reinterpret_cast<float4*>(part_piece<64, VC * 64>(p_sm + t * P_BYTES, q_sm + t * Q_BYTES, r, (c + d) / 4)) =
                make_float4(ov[d], ov[d + 1], ov[d + 2], ov[d + 3]);
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      }
    } else if (ok && n_mine > 0) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const bool valid = t * TC_BQ + r < rows_valid;
      float inv = 1.f / l_run;
      if (EXT && ex.gate && valid)
        inv *= ex.gate[((size_t)seq_q_start[seq] + q_first + t * TC_BQ + r) * heads + head];
      bf16* dst = out + ((size_t)seq_q_start[seq] + q_first + t * TC_BQ + r) * ((size_t)heads * vdim) + (size_t)head * vdim;
#pragma unroll 1
      for (int c = 0; c < vdim; c += 32) {
        float ov[32];
        tmem_load32(tmem_o + c, ov);
        if (valid) {
#pragma unroll
          for (int d = 0; d < 32; d += 8) {
            if (EXT && c + d >= vdim) break;
            uint32_t w[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              __nv_bfloat162 pk = __floats2bfloat162_rn(ov[d + 2 * e] * inv, ov[d + 2 * e + 1] * inv);
              w[e] = *reinterpret_cast<uint32_t*>(&pk);
            }
            *reinterpret_cast<uint4*>(dst + c + d) = make_uint4(w[0], w[1], w[2], w[3]);
          }
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    }
  }

  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  if constexpr (PARTS) {
    // (the rows' states lie where keys were: both tiles are done with them behind the block's barrier)
    float2* ml = reinterpret_cast<float2*>(ring);
    __syncthreads();
    if (threadIdx.x < 2 * TC_BQ) ml[threadIdx.x] = row_state;
    cluster_barrier();
    if (threadIdx.x < 2 * TC_BQ) {
      const size_t row0 = (size_t)seq_q_start[seq] + q_first;
      merge_parts<64, VC * 64, Q_BYTES, P_BYTES>(
          q_sm, p_sm, ml, part, splits, rows_valid, vdim, out + row0 * ((size_t)heads * vdim) + (size_t)head * vdim,
          (size_t)heads * vdim, [&](int row, float, float sum) {
            float inv = 1.f / sum;
            if (EXT && ex.gate) inv *= ex.gate[(row0 + row) * heads + head];
            return inv;
          });
    }
    cluster_barrier();                            // nobody leaves while others read from it
  }
  __syncthreads();
  if (warp == 9) {
    __syncwarp();
    tmem_free(tmem_holder, TMEM_COLS);
  }
  if (threadIdx.x == 0 && abort_flag && status) atomicOr(status, 16);
}

// ------------------------------------------------------------------------------------------ host

// PARTS: keys in parts.  An instance of its own: as a question at run time it cost either form (us, then / now): one CTA a block, 2,048 tokens
// of 16 heads of 128 35.1 / 34.4, of 64 32.1 / 30.7, 4 x 129 of 64 7.8 / 7.4; 700 behind 1,200 in two parts 28.9 / 27.6, of 64 26.3 / 24.6.
// (The formed keys' kernel does not pay: 60.4 / 60.8, 51.7 / 52.7.)
template <int DC, int VC, int EXT, bool PARTS>
static int launch_as(const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv, void* out,
                     const int* block_table, int table_stride, const int* seq_slot, const int* seq_q_start,
                     const int* seq_q_len, const int* seq_kv_len, const int* tile_seq, const int* tile_first,
                     int n_tiles, int heads, int kv_heads, float scale, int window, int* status, int list_of_blocks,
                     int splits, cudaStream_t s, TcExtras ex) {
  const int smem = (2 * DC + 4 + TC_RING * (DC > VC ? DC : VC)) * 128 * 128 + 1024;
  auto kernel = attention_prefill_tc_kernel<DC, VC, EXT, PARTS>;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return (int)e;
    configured = true;
  }
#define ARGS mq, mk, mv, (bf16*)out, block_table, table_stride, seq_slot, seq_q_start, seq_q_len, seq_kv_len, tile_seq, tile_first, heads, \
             kv_heads, scale * 1.4426950408889634f, window, status, list_of_blocks, splits, ex
  if (PARTS)
    return launch_dependent_cluster(kernel, dim3(heads * splits, n_tiles), dim3(TC_THREADS), smem, s, dim3(splits), ARGS);
  return launch_dependent(kernel, dim3(heads, n_tiles), dim3(TC_THREADS), smem, s, ARGS);
#undef ARGS
}

template <int DC, int VC, int EXT>
static int launch(const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv, void* out,
                  const int* block_table, int table_stride, const int* seq_slot, const int* seq_q_start,
                  const int* seq_q_len, const int* seq_kv_len, const int* tile_seq, const int* tile_first,
                  int n_tiles, int heads, int kv_heads, float scale, int window, int* status, int list_of_blocks,
                  int splits, cudaStream_t s, TcExtras ex = TcExtras{nullptr, nullptr, nullptr, nullptr, 0, 0, 0.f, 0.f, DC * 64, VC * 64}) {
#define ARGS(SPLITS) mq, mk, mv, out, block_table, table_stride, seq_slot, seq_q_start, seq_q_len, seq_kv_len, tile_seq, tile_first, n_tiles, \
                     heads, kv_heads, scale, window, status, list_of_blocks, SPLITS, s, ex
  if constexpr (DC == 2 || VC == 1)
    if (splits >= 2) return launch_as<DC, VC, EXT, true>(ARGS(splits >= 4 ? 4 : 2));
  return launch_as<DC, VC, EXT, false>(ARGS(1));
#undef ARGS
}

static unsigned long long next_limit_ns = WAIT_LIMIT_NS;
static int next_withhold_step = -1;

extern "C" {

// For tests of the give-up path: the NEXT sb_attention_prefill_tc launch leaves out half of the
// values of step `step` (128 keys) of every block and its waits give up after `limit_ns`.  The
// blocks cannot finish; the launch must return with bit 16 of *status set.  The switches are set
// and put back by copies on the launch's stream, around that one launch.
void sb_attention_prefill_tc_withhold(int step, unsigned long long limit_ns) {
  next_withhold_step = step;
  next_limit_ns = limit_ns ? limit_ns : WAIT_LIMIT_NS;
}

// How many clusters of `size` CTAs that take an SM each (the prompt attentions' blocks) the current device runs at once, or minus an
// error.  A cluster lies inside one of the chip's processing clusters, whose SMs need not be a multiple of its size.
int sb_prompt_clusters(int size) {
  auto kernel = attention_prefill_tc_kernel<2, 2, 0, true>;
  const int smem = (2 * 2 + 4 + TC_RING * 2) * 128 * 128 + 1024;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return -(int)e;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = size;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(size);
  cfg.blockDim = dim3(TC_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int n = 0;
  e = cudaOccupancyMaxActiveClusters(&n, kernel, &cfg);
  return e == cudaSuccess ? n : -(int)e;
}

// Same contract as sb_attention_prefill; n_tokens rows in q/out, n_pages pages in the stores.
// list_of_blocks: tile_seq/tile_first list blocks of 256 queries (else tiles of 64, see the kernel).  splits: CTAs that share a block's
// keys (1, 2 or 4; 1 where keys of up to 64 entries have values of more).
// head_dim must be 64 or 128 (returns -2 otherwise).
int sb_attention_prefill_tc(const void* q, void* out, const void* k_store, const void* v_store,
                            const int* block_table, int table_stride, const int* seq_slot,
                            const int* seq_q_start, const int* seq_q_len, const int* seq_kv_len,
                            const int* tile_seq, const int* tile_first, int n_tiles, int n_tokens,
                            int n_pages, int heads, int kv_heads, int head_dim, float scale, int window,
                            int* status, int list_of_blocks, int splits, cudaStream_t s) {
  if (n_tiles == 0) return 0;
  if (kv_heads <= 0 || heads % kv_heads) return -2;
  if (head_dim != 64 && head_dim != 128) return -2;
  if (((uintptr_t)q | (uintptr_t)out | (uintptr_t)k_store | (uintptr_t)v_store) & 15) return -2;
  CUtensorMap mq, mk, mv;
  int rc = sb_make_map(&mq, q, n_tokens, (long long)heads * head_dim, TC_BQ);
  if (rc) return rc;
  const long long kv_rows = (long long)n_pages * kv_heads * SB_PAGE_TOKENS;
  rc = sb_make_map(&mk, k_store, kv_rows, head_dim, SB_PAGE_TOKENS);
  if (rc) return rc;
  rc = sb_make_map(&mv, v_store, kv_rows, head_dim, SB_PAGE_TOKENS);
  if (rc) return rc;
#define ARGS mq, mk, mv, out, block_table, table_stride, seq_slot, seq_q_start, seq_q_len, seq_kv_len, \
             tile_seq, tile_first, n_tiles, heads, kv_heads, scale, window, status, list_of_blocks, splits, s
  const bool test_run = next_withhold_step >= 0;
  if (test_run) {
    cudaMemcpyToSymbolAsync(tc_withhold_step, &next_withhold_step, sizeof(int), 0, cudaMemcpyHostToDevice, s);
    cudaMemcpyToSymbolAsync(tc_wait_limit_ns, &next_limit_ns, sizeof(next_limit_ns), 0, cudaMemcpyHostToDevice, s);
    cudaStreamSynchronize(s);
  }
  rc = head_dim == 64 ? launch<1, 1, 0>(ARGS) : launch<2, 2, 0>(ARGS);
  if (test_run) {
    cudaStreamSynchronize(s);
    next_withhold_step = -1;
    next_limit_ns = WAIT_LIMIT_NS;
    cudaMemcpyToSymbolAsync(tc_withhold_step, &next_withhold_step, sizeof(int), 0, cudaMemcpyHostToDevice, s);
    cudaMemcpyToSymbolAsync(tc_wait_limit_ns, &next_limit_ns, sizeof(next_limit_ns), 0, cudaMemcpyHostToDevice, s);
    cudaStreamSynchronize(s);
  }
  return rc;
#undef ARGS
}

// The same for attention with a distance penalty, chunks, a sink and head gates (see attention_sink.cu): q
// points at rows of q_width entries (a multiple of 8) whose first heads * dim are the queries; out is
// [n_tokens, heads * vdim]; dim is a multiple of 16 and vdim of 8, both 16 to 128; scale > 0.  keep: the first keys a
// window or chunk keeps visible; cap: the scores' cap; 0: none.
int sb_sink_attention_tcgen05(const void* q, int q_width, void* out, const void* k_store, const void* v_store,
                              const int* block_table, int table_stride, const int* seq_slot, const int* seq_q_start,
                              const int* seq_q_len, const int* seq_kv_len, const int* tile_seq, const int* tile_first,
                              int n_tiles, int n_tokens, int n_pages, int heads, int kv_heads, int dim, int vdim, float scale,
                              const float* r1, const float* r2, const float* sink, const float* gate, int chunk, int window,
                              int keep, float cap, int* status, int list_of_blocks, int splits, cudaStream_t s) {
  if (n_tiles == 0) return 0;
  if (kv_heads <= 0 || heads % kv_heads || !(scale > 0.f) || keep < 0) return -2;
  if (dim < 16 || dim > 128 || dim % 16 || vdim < 16 || vdim > 128 || vdim % 8) return -2;
  if ((r1 == nullptr) != (r2 == nullptr) || q_width % 8 || q_width < heads * dim) return -2;
  if (((uintptr_t)q | (uintptr_t)out | (uintptr_t)k_store | (uintptr_t)v_store) & 15) return -2;
  CUtensorMap mq, mk, mv;
  int rc = sb_make_map(&mq, q, n_tokens, q_width, TC_BQ);
  if (rc) return rc;
  const long long kv_rows = (long long)n_pages * kv_heads * SB_PAGE_TOKENS;
  rc = sb_make_map(&mk, k_store, kv_rows, dim, SB_PAGE_TOKENS);
  if (rc) return rc;
  rc = sb_make_map(&mv, v_store, kv_rows, vdim, SB_PAGE_TOKENS);
  if (rc) return rc;
  const TcExtras ex{r1, r2, sink, gate, chunk > 0 ? chunk : 0, chunk > 0 || window > 0 ? keep : 0,
                    cap > 0.f ? scale / cap : 0.f, cap > 0.f ? cap / scale : 0.f, dim, vdim};
#define ARGS mq, mk, mv, out, block_table, table_stride, seq_slot, seq_q_start, seq_q_len, seq_kv_len, tile_seq, \
             tile_first, n_tiles, heads, kv_heads, scale, window, status, list_of_blocks, splits, s, ex
  const int kind = (dim > 64) * 2 + (vdim > 64);
  if (ex.cap_out == 0.f)
    return kind == 0 ? launch<1, 1, 1>(ARGS) : kind == 1 ? launch<1, 2, 1>(ARGS) : kind == 2 ? launch<2, 1, 1>(ARGS) : launch<2, 2, 1>(ARGS);
  return kind == 0 ? launch<1, 1, 2>(ARGS) : kind == 1 ? launch<1, 2, 2>(ARGS) : kind == 2 ? launch<2, 1, 2>(ARGS) : launch<2, 2, 2>(ARGS);
#undef ARGS
}

}  // extern "C"
