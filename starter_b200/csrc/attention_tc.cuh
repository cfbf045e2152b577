// What the tcgen05 attention kernels for prompts share: mbarriers with bounded waits, TMA tile loads, tensor memory, packed
// float arithmetic, shared-memory and instruction descriptors.
#pragma once

#include <cuda.h>

#include "common.cuh"

#define TC_BQ 128                // query rows of a tile
#define WAIT_LIMIT_NS 2000000000ull

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
// True in exactly one lane of the (converged) warp.
__device__ __forceinline__ bool elect_one() {
  uint32_t chosen;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(chosen));
  return chosen != 0;
}
__device__ __forceinline__ uint64_t now_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
  return ok != 0;
}
// For tests of the give-up path (sb_attention_prefill_tc_withhold): how long a wait may take, and
// which step's values the producer leaves out (-1: none).  Read only once a wait has spun a while.
__device__ unsigned long long tc_wait_limit_ns = WAIT_LIMIT_NS;
__device__ int tc_withhold_step = -1;

__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* abort) {
#pragma unroll 1
  for (int spin = 0; spin < 2048; ++spin)
    if (mbar_try(bar, parity)) return true;
  const uint64_t start = now_ns();
  const uint64_t limit = *(volatile unsigned long long*)&tc_wait_limit_ns;
#pragma unroll 1
  for (uint32_t spin = 0;; ++spin) {
    if (mbar_try(bar, parity)) return true;
    if ((spin & 63) == 0) {
      if (*abort) return false;
      if (now_ns() - start > limit) { *abort = 1; return false; }
    }
  }
}
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, uint64_t* bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void tmem_alloc(uint32_t* holder, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(holder)), "r"(cols) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_free(uint32_t addr, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(cols) : "memory");
}
__device__ __forceinline__ void umma_bf16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// 32 consecutive float columns of this thread's TMEM lane
__device__ __forceinline__ void tmem_load32(uint32_t taddr, float* v) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

// 64 consecutive 32-bit columns of this thread's TMEM lane
__device__ __forceinline__ void tmem_load64(uint32_t taddr, float* v) {
  uint32_t r[64];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x64.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, "
      "%32, %33, %34, %35, %36, %37, %38, %39, %40, %41, %42, %43, %44, %45, %46, %47, "
      "%48, %49, %50, %51, %52, %53, %54, %55, %56, %57, %58, %59, %60, %61, %62, %63}, [%64];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31]),
        "=r"(r[32]), "=r"(r[33]), "=r"(r[34]), "=r"(r[35]), "=r"(r[36]), "=r"(r[37]), "=r"(r[38]), "=r"(r[39]),
        "=r"(r[40]), "=r"(r[41]), "=r"(r[42]), "=r"(r[43]), "=r"(r[44]), "=r"(r[45]), "=r"(r[46]), "=r"(r[47]),
        "=r"(r[48]), "=r"(r[49]), "=r"(r[50]), "=r"(r[51]), "=r"(r[52]), "=r"(r[53]), "=r"(r[54]), "=r"(r[55]),
        "=r"(r[56]), "=r"(r[57]), "=r"(r[58]), "=r"(r[59]), "=r"(r[60]), "=r"(r[61]), "=r"(r[62]), "=r"(r[63])
      : "r"(taddr)
      : "memory");
#pragma unroll
  for (int i = 0; i < 64; ++i) v[i] = __uint_as_float(r[i]);
}
// 32 columns back into this thread's TMEM lane
__device__ __forceinline__ void tmem_store32(uint32_t taddr, const float* v) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
      ::"r"(taddr), "r"(__float_as_uint(v[0])), "r"(__float_as_uint(v[1])), "r"(__float_as_uint(v[2])),
        "r"(__float_as_uint(v[3])), "r"(__float_as_uint(v[4])), "r"(__float_as_uint(v[5])),
        "r"(__float_as_uint(v[6])), "r"(__float_as_uint(v[7])), "r"(__float_as_uint(v[8])),
        "r"(__float_as_uint(v[9])), "r"(__float_as_uint(v[10])), "r"(__float_as_uint(v[11])),
        "r"(__float_as_uint(v[12])), "r"(__float_as_uint(v[13])), "r"(__float_as_uint(v[14])),
        "r"(__float_as_uint(v[15])), "r"(__float_as_uint(v[16])), "r"(__float_as_uint(v[17])),
        "r"(__float_as_uint(v[18])), "r"(__float_as_uint(v[19])), "r"(__float_as_uint(v[20])),
        "r"(__float_as_uint(v[21])), "r"(__float_as_uint(v[22])), "r"(__float_as_uint(v[23])),
        "r"(__float_as_uint(v[24])), "r"(__float_as_uint(v[25])), "r"(__float_as_uint(v[26])),
        "r"(__float_as_uint(v[27])), "r"(__float_as_uint(v[28])), "r"(__float_as_uint(v[29])),
        "r"(__float_as_uint(v[30])), "r"(__float_as_uint(v[31]))
      : "memory");
}
// Two fused multiply-adds / two adds in one instruction (packed f32x2): half the issue slots.
__device__ __forceinline__ void fma2(float& d0, float& d1, float a0, float a1, float b, float c) {
  asm("{\n\t.reg .b64 ra, rb, rc, rd;\n\t"
      "mov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %4};\n\tmov.b64 rc, {%5, %5};\n\t"
      "fma.rn.f32x2 rd, ra, rb, rc;\n\tmov.b64 {%0, %1}, rd;\n\t}"
      : "=f"(d0), "=f"(d1) : "f"(a0), "f"(a1), "f"(b), "f"(c));
}
__device__ __forceinline__ void add2(float& acc0, float& acc1, float a0, float a1) {
  asm("{\n\t.reg .b64 ra, rb;\n\t"
      "mov.b64 ra, {%0, %1};\n\tmov.b64 rb, {%2, %3};\n\t"
      "add.rn.f32x2 ra, ra, rb;\n\tmov.b64 {%0, %1}, ra;\n\t}"
      : "+f"(acc0), "+f"(acc1) : "f"(a0), "f"(a1));
}
__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Operand tile with rows of 128 bytes and 128-byte swizzle, 8-row groups 1024 bytes apart.  For a
// K-major operand the rows are M/N and `lbo` is unused; for an MN-major operand the rows are k and
// `lbo` is the distance between 64-element chunks along M/N.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo_bytes) {
  uint64_t d = 0;
  d |= (uint64_t)((addr & 0x3FFFF) >> 4);
  d |= (uint64_t)((lbo_bytes >> 4) & 0x3FFF) << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}
// kind::f16, float accumulator, bfloat16 operands, A K-major, M = 128; B K-major or MN-major.
__device__ __forceinline__ uint32_t instr_desc(int n, int b_mn_major) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)b_mn_major << 16) | ((uint32_t)(n >> 3) << 17) |
         ((uint32_t)(TC_BQ >> 4) << 24);
}

// ------------------------------------------------------------------------------------------ keys in parts
// With few blocks of queries the CTAs of a cluster share a block: each walks a part of its keys, files its rows' reference, sum and
// output (float, unscaled) in its own shared memory, and after the cluster's barrier every CTA merges its share of the rows, reading
// the others' through distributed shared memory.  A tile's output lies where its own weights and queries were (nobody else
// reads those): PC columns in P's tile, the rest in Q's, 16-byte pieces swizzled over eight.
template <int PC, int COLS>
__device__ __forceinline__ float* part_piece(uint8_t* p_tile, uint8_t* q_tile, int r, int piece) {
  constexpr int QW = COLS > PC ? COLS - PC : PC;
  return piece * 4 < PC ? reinterpret_cast<float*>(p_tile + r * (PC * 4) + ((piece ^ (r & 7)) << 4))
                        : reinterpret_cast<float*>(q_tile + r * (QW * 4) + (((piece - PC / 4) ^ (r & 7)) << 4));
}
__device__ __forceinline__ void cluster_barrier() {
  __syncwarp();                    // (.aligned: a whole warp at once)
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t peer_u32(const void* p, int rank) {
  uint32_t a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
  return a;
}
__device__ __forceinline__ float4 peer_load4(uint32_t a) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ float2 peer_load2(uint32_t a) {
  float2 v;
  asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a) : "memory");
  return v;
}
// Eight outputs times the sigmoid of their gates.
__device__ __forceinline__ void gate8(float* o, const bf16* gate) {
  const uint4 g = *reinterpret_cast<const uint4*>(gate);
  const uint32_t w[4] = {g.x, g.y, g.z, g.w};
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    const float z = __uint_as_float(e & 1 ? w[e / 2] & 0xffff0000u : w[e / 2] << 16);
    // (rounded to bfloat16 at once: the fast quotient, both sides by a quarter, since it is zero for divisors above 2^126)
    o[e] = __fdividef(0.25f * o[e], fmaf(0.25f, __expf(-z), 0.25f));
  }
}
// The rows of this CTA's share, by its first 256 threads: 16 threads a row, eight columns each.  ml: [2 tiles][128 rows] of (reference,
// sum); finish(t, r, reference, sum) gives the factor of the row's summed outputs; dst: output row 0 of the block, `cols` entries of a
// head, rows `stride` apart.  gate: null, or rows (gate_ld entries apart) of the output's columns, by whose sigmoid it is multiplied.
template <int PC, int COLS, int Q_BYTES, int P_BYTES, typename Finish>
__device__ __forceinline__ void merge_parts(uint8_t* q_sm, uint8_t* p_sm, float2* ml, int rank, int splits, int rows_valid, int cols,
                                            bf16* dst, size_t stride, Finish finish, const bf16* gate = nullptr, size_t gate_ld = 0) {
  const int share = 2 * TC_BQ / splits, c = (threadIdx.x & 15) * 8;
  if (c >= COLS || c >= cols) return;
  for (int n = threadIdx.x >> 4; n < share; n += 16) {
    const int row = rank * share + n, t = row / TC_BQ, r = row % TC_BQ;
    if (row >= rows_valid) return;
    float top = -INFINITY;
    float2 part[4];
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      part[p] = p < splits ? peer_load2(peer_u32(ml + t * TC_BQ + r, p)) : make_float2(-INFINITY, 0.f);
      if (part[p].y != 0.f) top = fmaxf(top, part[p].x);
    }
    float sum = 0.f, o[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    const float* a = part_piece<PC, COLS>(p_sm + t * P_BYTES, q_sm + t * Q_BYTES, r, c / 4);
    const float* b = part_piece<PC, COLS>(p_sm + t * P_BYTES, q_sm + t * Q_BYTES, r, c / 4 + 1);
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      // (a part without keys filed nothing; one whose sum is no number has a score that is none, which is the row's result)
      if (p >= splits || part[p].y == 0.f) continue;
      const float w = fast_exp2(part[p].x - top);
      sum = fmaf(w, part[p].y, sum);
      const float4 x = peer_load4(peer_u32(a, p)), y = peer_load4(peer_u32(b, p));
      o[0] = fmaf(w, x.x, o[0]); o[1] = fmaf(w, x.y, o[1]); o[2] = fmaf(w, x.z, o[2]); o[3] = fmaf(w, x.w, o[3]);
      o[4] = fmaf(w, y.x, o[4]); o[5] = fmaf(w, y.y, o[5]); o[6] = fmaf(w, y.z, o[6]); o[7] = fmaf(w, y.w, o[7]);
    }
    const float inv = finish(row, top, sum);
#pragma unroll
    for (int e = 0; e < 8; ++e) o[e] *= inv;
    if (gate) gate8(o, gate + (size_t)row * gate_ld + c);
    uint32_t w[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const __nv_bfloat162 two = __floats2bfloat162_rn(o[2 * e], o[2 * e + 1]);
      w[e] = *reinterpret_cast<const uint32_t*>(&two);
    }
    *reinterpret_cast<uint4*>(dst + (size_t)row * stride + c) = make_uint4(w[0], w[1], w[2], w[3]);
  }
}
