// One token a sequence of the recurrences of state_scan.cu, with what stands around them: the decays of a channel-decay step formed
// from their low-rank product, the recurrence, and the RMS norm of each head's read-out with its gate.  In three kernels each link
// of that chain waits for the one before, and a step of few sequences is latency: one sequence, 16 heads of 128 x 128, 5.8 + 6.1 + 2.9 us
// behind the projection.  Everything a head needs is the head's own (the norm too, in parts of a head), so here a block is a head of a
// sequence from the logits of its decays to its bfloat16 row.
//
// A warp keeps eight consecutive rows of S a lane: V / 4 lanes of four columns make a row, and where that is less than a warp its parts
// take further rows.  All of S is asked for at once (16 bytes a lane and row; 64 KB a block of 512 threads), the rows' factors are formed
// by the lanes of the warp that needs them while it is on its way, and the warps' sums over their rows meet behind the one barrier.
// (One block reads a head's 64 KB in about a microsecond; two or eight blocks a head would have to meet for the norm, which costs as much.)
//   state-space, gated delta: both read-outs are taken of the state as it is found (state_scan.cu), the delta rule's warps each add all
//     warps' S^T k behind the barrier and then write; forget-write, channel-decay: the state moves first.
// The state-space norm spans the heads, so that mode ends with float read-outs.
// (At the 64 registers that two blocks of 512 threads leave, channel-decay spills 52 bytes of stores and 36 of loads, state-space up to 44,
// the others 12 at most.)
// Measured captured, a whole layer, in separate kernels -> here (us): channel-decay, width 2,048, 16 heads, 1 sequence 27.5 -> 21.5, 32 sequences
// 70.8 -> 41.1 (67 MB of states are 10.5 at the copy rate); gated delta, 1,536, 12 heads, 4 sequences 25.8 -> 20.6, 2,048, 16 heads, 32 71.8 -> 50.1;
// forget-write, 1,536, 12 heads, 4 22.6 -> 16.5; state-space, heads of 128 x 64, 32 of them, 1 20.6 -> 18.6, 24, 16 33.6 -> 24.8, 32,
// 32 63.8 -> 41.1.
#include "common.cuh"

#define STEP_ROWS 8              // rows of S a lane keeps
#define STEP_RANKS 8             // entries of a decay's low rank a lane asks for ahead of the wait (four lanes share a row: ranks up to 32)

__device__ __forceinline__ float step_softplus(float z) { return z > 20.f ? z : log1pf(expf(z)); }
__device__ __forceinline__ float4 step_bf4(const uint2& v) {
  return make_float4(__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xffff0000u), __uint_as_float(v.y << 16),
                     __uint_as_float(v.y & 0xffff0000u));
}
__device__ __forceinline__ float4 step_fma(float a, const float4& x, const float4& y) {
  return make_float4(fmaf(a, x.x, y.x), fmaf(a, x.y, y.y), fmaf(a, x.z, y.z), fmaf(a, x.w, y.w));
}

struct StepArgs {
  const bf16 *q, *k, *v, *a_raw, *b_raw;
  int ldq, ldk, ldv, lda, ldb;
  const float *A_log, *dt_bias, *D;
  const bf16* low;               // channel-decay: the low-rank entries [tokens, ldl]
  const float *a2, *a2_bias;     // [rank][H N], [H N]
  int ldl, rank;
  float inv_tau;
  float* state;
  long long slot_stride;
  const int *seq_slot, *seq_q_start, *seq_q_len;
  int H, G, N;
  const bf16* gate;              // [tokens, ldg], or null
  int ldg;
  const float* gain;             // [wlen], or null: the read-outs go out as floats
  int wlen;
  float eps;
  float* out32;                  // [tokens, H V]
  bf16* out;
};

// LANES: lanes a row of S (V = 4 LANES).
template <int MODE, int LANES>
__global__ void __launch_bounds__(512, 2)
state_step_kernel(const StepArgs args) {
  constexpr int V = 4 * LANES, PARTS = 32 / LANES;
  constexpr bool READ_FIRST = MODE < 2;
  __shared__ __align__(16) float4 part[MODE == 1 ? 2 : 1][16][32];
  const int seq = blockIdx.x, h = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const int N = args.N, H = args.H;
  const int row0 = (warp * PARTS + lane / LANES) * STEP_ROWS, col = (lane % LANES) * 4;
  // the factors of the warp's rows are formed by lanes: lane l those of row PARTS * 8 * warp + (l % 8) + 8 * (part)
  const int mine = (warp * PARTS) * STEP_ROWS + (lane % (STEP_ROWS * PARTS));
  const bool have = mine < N;
  // ---- weights, ahead of the wait
  float rate = 0.f, bias = 0.f, skip = 0.f, a2[STEP_RANKS];
  if (MODE == 2) {
    rate = have ? 1.f - args.A_log[(size_t)h * N + mine] : 0.f;
    bias = have ? args.dt_bias[(size_t)h * N + mine] : 0.f;
  } else if (MODE == 3) {
    bias = have ? args.a2_bias[(size_t)h * N + mine] : 0.f;
#pragma unroll
    for (int i = 0; i < STEP_RANKS; ++i) {
      const int r = lane / (STEP_ROWS * PARTS) + (4 / PARTS) * i;
      a2[i] = have && r < args.rank ? args.a2[(size_t)r * H * N + (size_t)h * N + mine] : 0.f;
    }
  } else {
    rate = expf(args.A_log[h]);
    bias = args.dt_bias[h];
    skip = MODE == 0 && args.D ? args.D[h] : 0.f;
  }
  float4 gain = make_float4(0.f, 0.f, 0.f, 0.f);
  if (args.gain && warp == 0) gain = *reinterpret_cast<const float4*>(args.gain + ((size_t)h * V + col) % args.wlen);
  pdl_trigger();
  pdl_wait();
  const int* slots = args.seq_slot;
  const int* starts = args.seq_q_start;
  const int* lens = args.seq_q_len;
  float* state = args.state;
  const bf16 *qp = args.q, *kp = args.k, *vp = args.v, *ap = args.a_raw, *bp = args.b_raw, *lp = args.low, *zp = args.gate;
  SB_BEHIND_WAIT(slots); SB_BEHIND_WAIT(starts); SB_BEHIND_WAIT(lens); SB_BEHIND_WAIT(state);
  SB_BEHIND_WAIT(qp); SB_BEHIND_WAIT(kp); SB_BEHIND_WAIT(vp); SB_BEHIND_WAIT(ap); SB_BEHIND_WAIT(bp); SB_BEHIND_WAIT(lp); SB_BEHIND_WAIT(zp);
  if (lens[seq] < 1) return;
  const size_t token = starts[seq];
  const int group = h / (H / args.G);
  float* sp = state + (size_t)slots[seq] * args.slot_stride + (size_t)h * N * V;
  float4 S[STEP_ROWS];
#pragma unroll
  for (int r = 0; r < STEP_ROWS; ++r)
    S[r] = row0 + r < N ? *reinterpret_cast<const float4*>(sp + (size_t)(row0 + r) * V + col) : make_float4(0.f, 0.f, 0.f, 0.f);
  const float4 x = step_bf4(*reinterpret_cast<const uint2*>(vp + token * args.ldv + (size_t)h * V + col));
  float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
  if (zp && warp == 0) z = step_bf4(*reinterpret_cast<const uint2*>(zp + token * args.ldg + (size_t)h * V + col));
  // ---- the rows' entries of q and k (state-space, delta rule: k and q themselves), by the lanes
  const bf16* kr = kp + token * args.ldk + (size_t)group * N;
  const bf16* qr = qp + token * args.ldq + (size_t)group * N;
  float qe = have ? to_f<bf16>(qr[mine]) : 0.f, ke = have ? to_f<bf16>(kr[mine]) : 0.f, de = 0.f;
  float gone = 0.f, fac = 0.f, dot = 0.f;          // READ_FIRST: 1 - g, the factor of a write, k . q
  if (MODE == 2) {
    qe = qe / (1.f + expf(-qe));
    de = rate / (1.f + expf(ke + bias));
  } else if (MODE == 3) {
    const bf16* low = lp + token * args.ldl;
    constexpr int SHARE = 4 / PARTS;               // lanes of a row
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < STEP_RANKS; ++i) {
      const int r = lane / (STEP_ROWS * PARTS) + SHARE * i;
      s = fmaf(a2[i], r < args.rank ? to_f<bf16>(low[r]) : 0.f, s);
    }
    for (int r = lane / (STEP_ROWS * PARTS) + SHARE * STEP_RANKS; r < args.rank; r += SHARE)
      if (have) s = fmaf(args.a2[(size_t)r * H * N + (size_t)h * N + mine], to_f<bf16>(low[r]), s);
#pragma unroll
    for (int o = STEP_ROWS * PARTS; o < 32; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    s += bias;
    const float log_sigmoid = fminf(s, 0.f) - log1pf(expf(-fabsf(s)));
    de = -expm1f(log_sigmoid * args.inv_tau);
    qe *= 1.f / sqrtf((float)N);
  } else {
    // k . q and the squares over all rows, by every warp for itself: lane l entries 4 l .. 4 l + 3
    float sq = 0.f, sk = 0.f;
    if (4 * lane < N) {
      const float4 a = step_bf4(*reinterpret_cast<const uint2*>(qr + 4 * lane)), b = step_bf4(*reinterpret_cast<const uint2*>(kr + 4 * lane));
      dot = a.x * b.x + a.y * b.y + a.z * b.z + a.w * b.w;
      sq = a.x * a.x + a.y * a.y + a.z * a.z + a.w * a.w;
      sk = b.x * b.x + b.y * b.y + b.z * b.z + b.w * b.w;
    }
    dot = warp_sum(dot);
    const float dt = step_softplus(to_f<bf16>(ap[token * args.lda + h]) + bias);
    gone = -expm1f(-rate * dt);
    fac = dt;
    if (MODE == 1) {
      sq = warp_sum(sq);
      sk = warp_sum(sk);
      const float mq = rsqrtf((float)N) / sqrtf(sq + 1e-6f), mk = 1.f / sqrtf(sk + 1e-6f);
      qe *= mq;
      ke *= mk;
      dot *= mq * mk;
      fac = 1.f / (1.f + expf(-to_f<bf16>(bp[token * args.ldb + h])));
    }
  }
  // ---- the walk's one step
  float4 o = make_float4(0.f, 0.f, 0.f, 0.f), rk = o;
  const int from = lane / LANES * STEP_ROWS;        // lane from + r holds row row0 + r
#pragma unroll
  for (int r = 0; r < STEP_ROWS; ++r) {
    const float kk = __shfl_sync(0xffffffffu, ke, from + r), qq = __shfl_sync(0xffffffffu, qe, from + r);
    if (READ_FIRST) {
      o = step_fma(qq, S[r], o);
      if (MODE == 1) rk = step_fma(kk, S[r], rk);
    } else {
      const float d = __shfl_sync(0xffffffffu, de, from + r);
      if (MODE == 2) S[r] = step_fma(d, make_float4(x.x - S[r].x, x.y - S[r].y, x.z - S[r].z, x.w - S[r].w), S[r]);
      else S[r] = step_fma(kk, x, step_fma(-d, S[r], S[r]));
      o = step_fma(qq, S[r], o);
    }
  }
  auto file = [&]() {
#pragma unroll
    for (int r = 0; r < STEP_ROWS; ++r)
      if (row0 + r < N) *reinterpret_cast<float4*>(sp + (size_t)(row0 + r) * V + col) = S[r];
  };
  float4 u = make_float4(fac * x.x, fac * x.y, fac * x.z, fac * x.w);
  if (MODE == 0) {                                  // (the write does not depend on what is read)
#pragma unroll
    for (int r = 0; r < STEP_ROWS; ++r) S[r] = step_fma(__shfl_sync(0xffffffffu, ke, from + r), u, step_fma(-gone, S[r], S[r]));
  }
  if (MODE != 1) file();
  part[0][warp][lane] = o;
  if (MODE == 1) part[MODE == 1][warp][lane] = rk;
  __syncthreads();
  auto total = [&](const float4 (*p)[32]) {
    float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int w = 0; w < warps; ++w) {
      const float4 e = p[w][lane];
      t = make_float4(t.x + e.x, t.y + e.y, t.z + e.z, t.w + e.w);
    }
#pragma unroll
    for (int s = LANES; s < 32; s <<= 1) {
      t.x += __shfl_xor_sync(0xffffffffu, t.x, s);
      t.y += __shfl_xor_sync(0xffffffffu, t.y, s);
      t.z += __shfl_xor_sync(0xffffffffu, t.z, s);
      t.w += __shfl_xor_sync(0xffffffffu, t.w, s);
    }
    return t;
  };
  if (MODE == 1) {
    const float4 t = total(part[MODE == 1]);
    u = make_float4(fac * (x.x - fmaf(-gone, t.x, t.x)), fac * (x.y - fmaf(-gone, t.y, t.y)), fac * (x.z - fmaf(-gone, t.z, t.z)),
                    fac * (x.w - fmaf(-gone, t.w, t.w)));
#pragma unroll
    for (int r = 0; r < STEP_ROWS; ++r) S[r] = step_fma(__shfl_sync(0xffffffffu, ke, from + r), u, step_fma(-gone, S[r], S[r]));
    file();
  }
  if (warp != 0) return;
  o = total(part[0]);
  if (READ_FIRST) {
    o = step_fma(dot, u, step_fma(-gone, o, o));
    if (MODE == 0) o = step_fma(skip, x, o);
  }
  const size_t at = token * H * V + (size_t)h * V + col;
  if (!args.gain) {
    if (lane < LANES) *reinterpret_cast<float4*>(args.out32 + at) = o;
    return;
  }
  float sq = o.x * o.x + o.y * o.y + o.z * o.z + o.w * o.w;
#pragma unroll
  for (int s = 1; s < LANES; s <<= 1) sq += __shfl_xor_sync(0xffffffffu, sq, s);
  const float inv = 1.f / sqrtf(sq / (float)V + args.eps);
  float y[4] = {o.x * inv * gain.x, o.y * inv * gain.y, o.z * inv * gain.z, o.w * inv * gain.w};
  if (zp) {
    const float g[4] = {z.x, z.y, z.z, z.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) y[i] *= g[i] / (1.f + expf(-g[i]));
  }
  uint2 w;
  *reinterpret_cast<__nv_bfloat162*>(&w.x) = __floats2bfloat162_rn(y[0], y[1]);
  *reinterpret_cast<__nv_bfloat162*>(&w.y) = __floats2bfloat162_rn(y[2], y[3]);
  if (lane < LANES) *reinterpret_cast<uint2*>(args.out + at) = w;
}

extern "C" {

// Whether the step is one of these kernels': bfloat16 heads of 32, 64 or 128 values and 8 to 128 rows (whole blocks of eight a lane).
int sb_state_step_takes(int mode, int H, int G, int N, int V) {
  if (mode < 0 || mode > 3 || H < 1 || G < 1 || H % G || (mode >= 2 && G != H) || H > 65535) return 0;
  if (V != 32 && V != 64 && V != 128) return 0;
  return N >= 8 && N <= 128 && N % (8 * (128 / V)) == 0;
}

// Arguments as sb_state_scan's (bfloat16 operands; mode 3: the low-rank entries `low` [tokens, ldl], a2 float [rank][H * N] and its
// bias in the decays' place), for sequences that bring at most one token.  gate: [tokens, ldg] or null; gain: float [wlen], then out is
// bfloat16 [tokens, H * V] = rms(o) * gain (* silu(gate)), a head a part; without a gain (and a gate) out32 float gets the read-outs.
// -2: not taken (sizes, or an operand off its alignment: v, gate, q, k in 8-byte pieces, state, gain and outputs in 16).
int sb_state_step(int mode, const void* q, int ldq, const void* k, int ldk, const void* v, int ldv, const void* a_raw, int lda,
                  const void* b_raw, int ldb, const float* A_log, const float* dt_bias, const float* D, const void* low, int ldl,
                  const float* a2, const float* a2_bias, int rank, float inv_tau, float* state, long long slot_stride,
                  const int* seq_slot, const int* seq_q_start, const int* seq_q_len, int n_seqs, int H, int G, int N, int V,
                  const void* gate, int ldg, const float* gain, int wlen, float eps, float* out32, void* out, cudaStream_t s) {
  if (n_seqs == 0) return 0;
  if (!sb_state_step_takes(mode, H, G, N, V)) return -2;
  if ((((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)gate | (uintptr_t)out) % 8) || ldq % 4 || ldk % 4 || ldv % 4 || ldg % 4) return -2;
  if ((((uintptr_t)state | (uintptr_t)gain | (uintptr_t)out32) % 16) || slot_stride % 4) return -2;
  if (gain ? (!out || wlen < 4 || wlen % 4) : (!out32 || gate)) return -2;
  if (mode < 2 ? (!a_raw || !A_log || !dt_bias || (mode == 1 && !b_raw)) : mode == 2 ? (!A_log || !dt_bias) : (!low || !a2 || !a2_bias || rank < 1))
    return -2;
  const StepArgs args = {(const bf16*)q, (const bf16*)k, (const bf16*)v, (const bf16*)a_raw, (const bf16*)b_raw, ldq, ldk, ldv, lda, ldb,
                         A_log, dt_bias, D, (const bf16*)low, a2, a2_bias, ldl, rank, inv_tau, state, slot_stride, seq_slot, seq_q_start,
                         seq_q_len, H, G, N, (const bf16*)gate, ldg, gain, wlen, eps, out32, (bf16*)out};
  const int lanes = V / 4, warps = N / (STEP_ROWS * (32 / lanes));
#define STEP_GO(M)                                                                                                            \
  return lanes == 32 ? launch_dependent(state_step_kernel<M, 32>, dim3(n_seqs, H), dim3(32 * warps), 0, s, args)              \
         : lanes == 16 ? launch_dependent(state_step_kernel<M, 16>, dim3(n_seqs, H), dim3(32 * warps), 0, s, args)            \
                       : launch_dependent(state_step_kernel<M, 8>, dim3(n_seqs, H), dim3(32 * warps), 0, s, args)
  switch (mode) {
    case 0: STEP_GO(0);
    case 1: STEP_GO(1);
    case 2: STEP_GO(2);
    default: STEP_GO(3);
  }
#undef STEP_GO
}

}  // extern "C"
