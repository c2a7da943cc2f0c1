// Device helpers shared by the forward and backward TTT-MLP kernels: the GELU family
// (reference: include/common/base_ops.cuh:465-548 and kernels/ttt_backward/matching.py:42-55),
// bf16 row access to 128-byte-swizzled tiles, and the two MMA forms every contraction of
// the operator reduces to.
#pragma once

#include "sm100_ptx.cuh"
#include <cuda_fp16.h>

namespace tttdev {

using namespace sm100;

constexpr uint32_t TILE = 8192;    // 64 x 64 bf16 tile
constexpr uint32_t BIG = 32768;    // 256 x 64 bf16 tile ("hidden-major": one row per hidden unit)

constexpr float kG0 = 0.79788456f, kG1 = 0.044715f, kG2 = 0.1070322243f;
constexpr float kG01 = kG0 * kG1;      // tanh argument: kG0 x (1 + kG1 x^2) = x (kG0 + kG01 x^2), one multiply less

__device__ __forceinline__ float tanh_fast(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// gelu(x), gelu'(x), gelu''(x), tanh approximation.  With t = tanh(x (kG0 + kG01 x^2)), h = (1 + t) / 2
// and q = kG0 + kG2 x^2 (the argument's derivative):
//   gelu = x h,   gelu' = h + x (1 - t^2) q / 2 = h + (g - g t) q   (since (1 - t^2) / 2 = h (1 - t)),
//   gelu'' = (1 - t^2) (kG0 + 2 kG2 x^2 - x t q^2).
// Two elements at a time in packed fp32: the epilogues that evaluate it are bound by the fp32 pipe, so these forms have
// the fewest operations and no negation (which packed operands do not have): gelu and gelu' from t' = -t = tanh(-u) as
// h = (1 - t') / 2, g = x h, gelu' = h + (g + g t') q; gelu alone from y = x / 2 as y + y t.
__device__ __forceinline__ f32x2 tanh2(f32x2 u) {
  float lo, hi;
  upk(u, lo, hi);
  return pk(tanh_fast(lo), tanh_fast(hi));
}
__device__ __forceinline__ void gelu_pair2(f32x2 x, f32x2& g, f32x2& gp) {
  const f32x2 x2 = mul2(x, x);
  const f32x2 t = tanh2(mul2(x, fma2(x2, pk1(-kG01), pk1(-kG0))));       // -tanh(u)
  const f32x2 h = fma2(t, pk1(-0.5f), pk1(0.5f));
  g = mul2(x, h);
  gp = fma2(fma2(g, t, g), fma2(x2, pk1(kG2), pk1(kG0)), h);
}
// gelu(2 y)
__device__ __forceinline__ f32x2 gelu_half2(f32x2 y) {
  const f32x2 t = tanh2(mul2(y, fma2(mul2(y, y), pk1(8.f * kG01), pk1(2.f * kG0))));
  return fma2(y, t, y);
}

// ---- The same family on two elements at a time in packed fp16 arithmetic.  The tanh-GELU and its
// derivatives are O(1) functions of O(1) arguments, so fp16 (11 significand bits) evaluates them to
// ~5e-4 (gelu'': ~2e-3), below the bf16 rounding (4e-3) every result meets when it is stored as an MMA
// operand; one instruction then serves two elements.  The argument is clamped to +-20, beyond which
// gelu' is 0 or 1 and gelu'' is 0 to fp16 precision (and x^3 would leave the fp16 range); gelu
// itself stays in fp32: on fp32 arguments the conversions cost what the packed arithmetic saves, so
// only the derivatives of Z1, which the recompute keeps as f16 tiles, use this path.
__device__ __forceinline__ __half2 h2c(float v) { return __float2half2_rn(v); }
__device__ __forceinline__ __half2 tanh_h2(__half2 u) {
  uint32_t r;
  asm("tanh.approx.f16x2 %0, %1;" : "=r"(r) : "r"(*reinterpret_cast<const uint32_t*>(&u)));
  return *reinterpret_cast<__half2*>(&r);
}

__device__ __forceinline__ uint32_t f32x2_to_f16x2(f32x2 a) {
  float lo, hi;
  upk(a, lo, hi);
  const __half2 h = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ f32x2 f16x2_to_f32x2(uint32_t w) {
  const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w));
  return pk(f.x, f.y);
}
// gelu'(z) and gelu''(z); a value beyond the f16 range has become infinite and is clamped like one beyond 20
__device__ __forceinline__ void gelu_grad_h2(uint32_t z, uint32_t& gp, uint32_t& gpp) {
  const __half2 x = __hmax2(__hmin2(*reinterpret_cast<const __half2*>(&z), h2c(20.f)), h2c(-20.f));
  const __half2 x2 = __hmul2(x, x);
  const __half2 t = tanh_h2(__hmul2(x, __hfma2(h2c(kG01), x2, h2c(kG0))));
  const __half2 h = __hfma2(h2c(0.5f), t, h2c(0.5f));
  const __half2 q = __hfma2(h2c(kG2), x2, h2c(kG0));
  const __half2 g = __hmul2(x, h);
  const __half2 a = __hfma2(__hfma2(__hneg2(g), t, g), q, h);
  const __half2 c = __hfma2(h2c(2.f * kG2), x2, h2c(kG0));
  const __half2 b = __hmul2(__hfma2(__hneg2(t), t, h2c(1.f)), __hfma2(__hneg2(__hmul2(__hmul2(x, t), q)), q, c));
  gp = *reinterpret_cast<const uint32_t*>(&a);
  gpp = *reinterpret_cast<const uint32_t*>(&b);
}

__device__ __forceinline__ uint4 pack_chunk(const float* v) {
  uint4 w;
  w.x = pack_bf16(v[0], v[1]);
  w.y = pack_bf16(v[2], v[3]);
  w.z = pack_bf16(v[4], v[5]);
  w.w = pack_bf16(v[6], v[7]);
  return w;
}
// 8 consecutive elements (16-byte chunk `chunk`) of row `row` of a swizzled tile
__device__ __forceinline__ void st_chunk(uint8_t* tile, uint32_t row, uint32_t chunk, const float* v) {
  *reinterpret_cast<uint4*>(tile + sw128_off(row, chunk)) = pack_chunk(v);
}
// the four 16-byte chunks of 32 fp32 accumulator columns as bf16, to row `row` of a swizzled tile
__device__ __forceinline__ void st_cols32(uint8_t* tile, int row, int half, const uint32_t (&v)[32]) {
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    uint4 w;
    w.x = pack_bf16(__uint_as_float(v[c * 8 + 0]), __uint_as_float(v[c * 8 + 1]));
    w.y = pack_bf16(__uint_as_float(v[c * 8 + 2]), __uint_as_float(v[c * 8 + 3]));
    w.z = pack_bf16(__uint_as_float(v[c * 8 + 4]), __uint_as_float(v[c * 8 + 5]));
    w.w = pack_bf16(__uint_as_float(v[c * 8 + 6]), __uint_as_float(v[c * 8 + 7]));
    *reinterpret_cast<uint4*>(tile + sw128_off(row, half * 4 + c)) = w;
  }
}
// 32 fp32 accumulator columns as bf16 pairs to 16 columns of tensor memory (an A operand of the MMAs)
__device__ __forceinline__ void st_cols32_tmem(uint32_t taddr, const uint32_t (&v)[32]) {
  uint32_t w[16];
#pragma unroll
  for (int k = 0; k < 16; ++k) w[k] = pack_bf16(__uint_as_float(v[2 * k]), __uint_as_float(v[2 * k + 1]));
  tmem_st16(taddr, w);
}

// the raw 16 bytes of a chunk: requested between a tensor-memory load and its wait, unpacked after
__device__ __forceinline__ uint4 ld_chunk_raw(const uint8_t* tile, uint32_t row, uint32_t chunk) {
  return *reinterpret_cast<const uint4*>(tile + sw128_off(row, chunk));
}

// ---- MMA issue.  The instruction stream around each tcgen05.mma is kept to two integer adds: the descriptors' high
// words are the same constant for every operand (stride byte offset 1024, version 1, 128-byte swizzle) and
// the low words (start address | leading byte offset) advance by a constant per K step.
constexpr uint32_t kDescHi = (1024u >> 4) | (1u << 14) | (2u << 29);
__device__ __forceinline__ uint32_t desc_lo(uint32_t smem_addr, uint32_t lbo_bytes) {
  return ((smem_addr & 0x3FFFFu) >> 4) | ((lbo_bytes >> 4) << 16);
}

// ---- Products issued by single threads (lane 0 of warps 0..3, one product or half each), through one out-of-line loop
// that every product of the kernel shares: n MMAs whose operand descriptors advance by a constant per K step; the first
// one overwrites D unless `acc` is set.  For the one-CTA backward, whose instruction footprint exceeds the instruction
// cache: a tcgen05.mma costs about ten instructions of set-up, so one loop instead of one per product shrinks it by
// roughly a tenth.
__device__ __forceinline__ void mma_issue_rt(uint32_t tmem_d, uint32_t a_lo, uint32_t b_lo, uint32_t idesc,
                                             uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
      "mov.b64 da, {%1, %4};\n\t"
      "mov.b64 db, {%2, %4};\n\t"
      "setp.ne.b32 p, %5, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, p;\n\t}" ::"r"(tmem_d),
      "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(kDescHi), "r"(accumulate)
      : "memory");
}
static __device__ __noinline__ void mma_run(uint32_t tmem_d, uint32_t a_lo, uint32_t b_lo, uint32_t idesc,
                                            uint32_t n, uint32_t astep, uint32_t bstep, uint32_t acc) {
  // n is a multiple of 4 at every call
#pragma unroll 1
  for (uint32_t j = 0; j < n; j += 4) {
    mma_issue_rt(tmem_d, a_lo, b_lo, idesc, acc | j);
    mma_issue_rt(tmem_d, a_lo + astep, b_lo + bstep, idesc, 1u);
    mma_issue_rt(tmem_d, a_lo + 2 * astep, b_lo + 2 * bstep, idesc, 1u);
    mma_issue_rt(tmem_d, a_lo + 3 * astep, b_lo + 3 * bstep, idesc, 1u);
    a_lo += 4 * astep;
    b_lo += 4 * bstep;
  }
}

// "Hidden-major" product: D[256 x 64] (two M=128 blocks, 64 fp32 columns each, at tmem_d and
// tmem_d + 64) (+)= A * B with A a [256][64] bf16 tile read K-major (row = hidden unit) and B a
// [64][64] tile read K-major (row = N index) or MN-major (row = K index).
// One M = 128 block (`blk` = 0 or 1: hidden units 128 blk .. 128 blk + 127) of the product.  The two
// blocks are independent, so two threads may issue one each.  The flags are constants at every call.
__device__ __forceinline__ void mma_hidden_half(uint32_t tmem_d, uint32_t a_smem, uint32_t b_smem, bool b_mn,
                                                bool accumulate, int blk) {
  mma_run(tmem_d + blk * 64, desc_lo(a_smem, 16) + blk * (16384u >> 4), desc_lo(b_smem, b_mn ? 8192 : 16),
          umma_idesc_bf16(128, 64, false, b_mn, false), 4, 2, b_mn ? (2048u >> 4) : (32u >> 4), accumulate ? 1u : 0u);
}
__device__ __forceinline__ void mma_hidden_major(uint32_t tmem_d, uint32_t a_smem, uint32_t b_smem, bool b_mn,
                                                 bool accumulate) {
#pragma unroll 1
  for (int blk = 0; blk < 2; ++blk) mma_hidden_half(tmem_d, a_smem, b_smem, b_mn, accumulate, blk);
}
// "Token-major" product: D[64 tok x 64] (M = 64: row r in TMEM lane (r % 16) + 32 * (r / 16))
// = X[64 x 256] * W[256 x 64], both operands [256][64] tiles read MN-major (row = hidden unit).
__device__ __forceinline__ void mma_token_major(uint32_t tmem_d, uint32_t x_smem, uint32_t w_smem) {
  mma_run(tmem_d, desc_lo(x_smem, BIG), desc_lo(w_smem, BIG), umma_idesc_bf16(64, 64, true, true, false), 16,
          2048u >> 4, 2048u >> 4, 0u);
}

// ---- The same products issued by a whole warp under a predicate: the warp runs the code uniformly, so that the
// descriptors are computed in uniform registers, and only the elected lane's tcgen05.mma is enabled (`lead`).
// Inside an `if (elect_one())` block the operands pass through vector registers instead: 8 MMAs took 390 cycles
// to issue there and take 182 here (16: 537 and 397), against 376 (512) that the tensor pipe needs for them.
template <bool kAccumulate>
__device__ __forceinline__ void mma_lead(uint32_t tmem_d, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint32_t lead) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t.reg .b64 da, db;\n\t"
      "mov.b64 da, {%1, %4};\n\t"
      "mov.b64 db, {%2, %4};\n\t"
      "setp.ne.b32 p, %5, 0;\n\t"
      "setp.ne.b32 q, %6, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, p;\n\t}" ::"r"(tmem_d),
      "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(kDescHi), "n"(kAccumulate ? 1 : 0), "r"(lead)
      : "memory");
}
// ... with the accumulate flag in a register, for rolled issue loops
__device__ __forceinline__ void mma_lead_rt(uint32_t tmem_d, uint32_t a_lo, uint32_t b_lo, uint32_t idesc,
                                            uint32_t accumulate, uint32_t lead) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t.reg .b64 da, db;\n\t"
      "mov.b64 da, {%1, %4};\n\t"
      "mov.b64 db, {%2, %4};\n\t"
      "setp.ne.b32 p, %5, 0;\n\t"
      "setp.ne.b32 q, %6, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, p;\n\t}" ::"r"(tmem_d),
      "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(kDescHi), "r"(accumulate), "r"(lead)
      : "memory");
}
// one 128-row block: D[128 x 64] (+)= A[128][64] B
template <bool kBMn, bool kAccumulate>
__device__ __forceinline__ void mma_hidden_lead(uint32_t tmem_d, uint32_t a_smem, uint32_t b_smem, int blk, uint32_t lead) {
  constexpr uint32_t idesc = umma_idesc_bf16(128, 64, false, kBMn, false);
  const uint32_t a0 = desc_lo(a_smem, 16) + blk * (16384u >> 4);
  const uint32_t b0 = desc_lo(b_smem, kBMn ? 8192 : 16);
  constexpr uint32_t bstep = kBMn ? (2048u >> 4) : (32u >> 4);
  const uint32_t d = tmem_d + blk * 64;
  mma_lead<kAccumulate>(d, a0, b0, idesc, lead);
#pragma unroll
  for (int j = 1; j < 4; ++j) mma_lead<true>(d, a0 + j * 2, b0 + j * bstep, idesc, lead);
}
// The same block with A in tensor memory: bf16 pairs, row = lane, 32 columns for the 64 elements along K.  The MMA
// then reads 2 KB of shared memory instead of 6 KB (32 cycles instead of 47, the tensor pipe's own rate).
template <bool kAccumulate>
__device__ __forceinline__ void mma_lead_ta(uint32_t tmem_d, uint32_t tmem_a, uint32_t b_lo, uint32_t idesc, uint32_t lead) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t.reg .b64 db;\n\t"
      "mov.b64 db, {%2, %4};\n\t"
      "setp.ne.b32 p, %5, 0;\n\t"
      "setp.ne.b32 q, %6, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %3, p;\n\t}" ::"r"(tmem_d),
      "r"(tmem_a), "r"(b_lo), "r"(idesc), "r"(kDescHi), "n"(kAccumulate ? 1 : 0), "r"(lead)
      : "memory");
}
template <bool kBMn, bool kAccumulate>
__device__ __forceinline__ void mma_hidden_ta(uint32_t tmem_d, uint32_t tmem_a, uint32_t b_smem, uint32_t lead) {
  constexpr uint32_t idesc = umma_idesc_bf16(128, 64, false, kBMn, false);
  const uint32_t b0 = desc_lo(b_smem, kBMn ? 8192 : 16);
  constexpr uint32_t bstep = kBMn ? (2048u >> 4) : (32u >> 4);
  mma_lead_ta<kAccumulate>(tmem_d, tmem_a, b0, idesc, lead);
#pragma unroll
  for (int j = 1; j < 4; ++j) mma_lead_ta<true>(tmem_d, tmem_a + j * 8, b0 + j * bstep, idesc, lead);
}
__device__ __forceinline__ void mma_token_lead(uint32_t tmem_d, uint32_t x_smem, uint32_t w_smem, uint32_t lead) {
  constexpr uint32_t idesc = umma_idesc_bf16(64, 64, true, true, false);
  const uint32_t a0 = desc_lo(x_smem, BIG);
  const uint32_t b0 = desc_lo(w_smem, BIG);
  mma_lead<false>(tmem_d, a0, b0, idesc, lead);
#pragma unroll
  for (int j = 1; j < 16; ++j) mma_lead<true>(tmem_d, a0 + j * (2048u >> 4), b0 + j * (2048u >> 4), idesc, lead);
}

// ---- A warp's 32 rows x 32 fp32 columns (lane = row, v = the row's 32 values) -> a row-major global
// matrix with `ld` floats per row, as whole 128-byte lines: written straight from the registers the
// 16-byte stores of a warp would land in 32 different lines (measured: the fp32 W2 checkpoint written
// that way cost 4 % of the forward), so the block is turned through a warp-private staging area
// (32 rows x 144 bytes of shared memory; the 16-byte pad keeps both directions conflict-free).
// `dst` points at the block's first element (row of lane 0, first of the 32 columns).  The caller makes
// sure that no other warp writes the bytes of this warp's staging area while the call runs.
__device__ __forceinline__ void store_rows_coalesced(float* dst, int ld, const uint32_t (&v)[32], uint8_t* stage,
                                                     int lane) {
#pragma unroll
  for (int c = 0; c < 8; ++c)
    *reinterpret_cast<uint4*>(stage + lane * 144 + c * 16) = make_uint4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int r = 4 * i + (lane >> 3), ch = lane & 7;
    const uint4 w = *reinterpret_cast<const uint4*>(stage + r * 144 + ch * 16);
    *reinterpret_cast<uint4*>(dst + static_cast<long>(r) * ld + ch * 4) = w;
  }
  __syncwarp();
}
constexpr uint32_t kRowStageBytes = 32 * 144;     // per warp

// ---- 64 x 64 x 64 products on M = 64 accumulators, issued likewise.  A is a [64][64] tile read K-major (row = M index),
// B one read K-major (row = N index) or MN-major (row = contraction index).
template <bool kBMn, bool kAccumulate>
__device__ __forceinline__ void mma_64_lead(uint32_t tmem_d, uint32_t a_smem, uint32_t b_smem, uint32_t lead) {
  constexpr uint32_t idesc = umma_idesc_bf16(64, 64, false, kBMn, false);
  const uint32_t a0 = desc_lo(a_smem, 16);
  const uint32_t b0 = desc_lo(b_smem, kBMn ? 8192 : 16);
  constexpr uint32_t bstep = kBMn ? (2048u >> 4) : (32u >> 4);
  mma_lead<kAccumulate>(tmem_d, a0, b0, idesc, lead);
#pragma unroll
  for (int j = 1; j < 4; ++j) mma_lead<true>(tmem_d, a0 + j * 2, b0 + j * bstep, idesc, lead);
}
// D += A^T B, both tiles read MN-major (row = contraction index)
__device__ __forceinline__ void mma_64_tn_lead(uint32_t tmem_d, uint32_t a_smem, uint32_t b_smem, uint32_t lead) {
  constexpr uint32_t idesc = umma_idesc_bf16(64, 64, true, true, false);
  const uint32_t a0 = desc_lo(a_smem, TILE);
  const uint32_t b0 = desc_lo(b_smem, TILE);
#pragma unroll
  for (int j = 0; j < 4; ++j) mma_lead<true>(tmem_d, a0 + j * (2048u >> 4), b0 + j * (2048u >> 4), idesc, lead);
}
// A warp's 32 rows x 32 fp32 columns (lane = row) -> a row-major global matrix with 64 floats per row, as whole
// 128-byte lines, turned through the warp's own 4 KB of a hidden-major tile (16-byte chunks XOR-swizzled by row:
// both directions conflict-free).
__device__ __forceinline__ void store_rows_own(float* dst, const uint32_t (&v)[32], uint8_t* stage, int lane) {
  __syncwarp();
#pragma unroll
  for (int c = 0; c < 8; ++c)
    *reinterpret_cast<uint4*>(stage + sw128_off(lane, c)) = make_uint4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int r = 4 * i + (lane >> 3), ch = lane & 7;
    *reinterpret_cast<uint4*>(dst + r * 64 + ch * 4) = *reinterpret_cast<const uint4*>(stage + sw128_off(r, ch));
  }
  __syncwarp();
}


// ---- Token-major 64 x 64 accumulators spread over 8 warps (256 threads).
// A token-major accumulator (M = 64) keeps row r in TMEM lane (r % 16) + 32 * (r / 16): quadrant q
// holds rows 16q .. 16q+15 in its first 16 lanes.  The two warps that may touch quadrant q (q and
// q + 4) each take 32 of the 64 columns with one 16x256b.x4 load, so every thread owns 16 values:
//   rows r0 = 16q + lane/4 and r1 = r0 + 8;  for j = 0..3 the column pair c = 32*colhalf + 8j + 2(lane%4):
//   v[4j], v[4j+1] = (r0, c), (r0, c+1);   v[4j+2], v[4j+3] = (r1, c), (r1, c+1).
// A row is shared by 8 threads: the 4 lanes of a quad in each of the two warps; row sums go through
// two shuffles and one exchange in shared memory between the warp pair (named barrier 1 + q).
struct TokMap {
  int quad, colhalf, l3;
  int r0, r1;
  uint32_t taddr;      // lane/column offset to add to the accumulator's TMEM address
  __device__ __forceinline__ TokMap(int warp, int lane)
      : quad(warp & 3), colhalf(warp >> 2), l3(lane & 3), r0((warp & 3) * 16 + (lane >> 2)),
        r1((warp & 3) * 16 + (lane >> 2) + 8),
        taddr((static_cast<uint32_t>((warp & 3) * 32) << 16) + static_cast<uint32_t>((warp >> 2) * 32)) {}
  __device__ __forceinline__ int col(int j) const { return colhalf * 32 + j * 8 + l3 * 2; }
  // byte offset of the column pair j of row r inside a swizzled [64][64] bf16 tile
  __device__ __forceinline__ uint32_t off(int r, int j) const { return sw128_off(r, colhalf * 4 + j) + l3 * 4; }
};
// three accumulators with one wait (the loads overlap)
__device__ __forceinline__ void tok_ld3(const TokMap& m, uint32_t acc_a, float (&a)[16], uint32_t acc_b,
                                        float (&b)[16], uint32_t acc_c, float (&c)[16]) {
  uint32_t ua[16], ub[16], uc[16];
  tmem_ld_16x256b_x4(acc_a + m.taddr, ua);
  tmem_ld_16x256b_x4(acc_b + m.taddr, ub);
  tmem_ld_16x256b_x4(acc_c + m.taddr, uc);
  tmem_wait_ld();
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    a[i] = __uint_as_float(ua[i]);
    b[i] = __uint_as_float(ub[i]);
    c[i] = __uint_as_float(uc[i]);
  }
}
__device__ __forceinline__ void tok_ld(const TokMap& m, uint32_t tmem_acc, float (&v)[16]) {
  uint32_t u[16];
  tmem_ld_16x256b_x4(tmem_acc + m.taddr, u);
  tmem_wait_ld();
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(u[i]);
}
// the thread's 16 values of a swizzled bf16 tile, same order as the accumulator fragment
__device__ __forceinline__ void tok_ld_tile(const TokMap& m, const uint8_t* tile, float (&v)[16]) {
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const uint32_t w0 = *reinterpret_cast<const uint32_t*>(tile + m.off(m.r0, j));
    const uint32_t w1 = *reinterpret_cast<const uint32_t*>(tile + m.off(m.r1, j));
    v[4 * j] = bf16_lo(w0); v[4 * j + 1] = bf16_hi(w0);
    v[4 * j + 2] = bf16_lo(w1); v[4 * j + 3] = bf16_hi(w1);
  }
}
__device__ __forceinline__ void tok_st_tile(const TokMap& m, uint8_t* tile, const float (&v)[16]) {
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    *reinterpret_cast<uint32_t*>(tile + m.off(m.r0, j)) = pack_bf16(v[4 * j], v[4 * j + 1]);
    *reinterpret_cast<uint32_t*>(tile + m.off(m.r1, j)) = pack_bf16(v[4 * j + 2], v[4 * j + 3]);
  }
}
// All-reduce N per-row partial sums over the 8 threads that share each row.  a[] belongs to row
// r0, b[] to row r1.  xch: fp32[2][64][8] in shared memory; the call uses columns kSlot .. kSlot+N-1
// of it.  There is no barrier after the read-back: the all-reduces of one epilogue phase must use
// disjoint columns, and a CTA barrier must separate phases (every phase ends with one).
template <int N, int kSlot>
__device__ __forceinline__ void tok_row_allreduce(const TokMap& m, float (&a)[N], float (&b)[N], float* xch) {
  static_assert(kSlot >= 0 && kSlot + N <= 8, "the exchange buffer has 8 columns per row");
#pragma unroll
  for (int i = 0; i < N; ++i) {
    a[i] += __shfl_xor_sync(0xffffffffu, a[i], 1);
    b[i] += __shfl_xor_sync(0xffffffffu, b[i], 1);
    a[i] += __shfl_xor_sync(0xffffffffu, a[i], 2);
    b[i] += __shfl_xor_sync(0xffffffffu, b[i], 2);
  }
  if (m.l3 == 0) {
#pragma unroll
    for (int i = 0; i < N; ++i) {
      xch[(m.colhalf * 64 + m.r0) * 8 + kSlot + i] = a[i];
      xch[(m.colhalf * 64 + m.r1) * 8 + kSlot + i] = b[i];
    }
  }
  named_bar_sync(1 + m.quad, 64);
#pragma unroll
  for (int i = 0; i < N; ++i) {
    a[i] += xch[((m.colhalf ^ 1) * 64 + m.r0) * 8 + kSlot + i];
    b[i] += xch[((m.colhalf ^ 1) * 64 + m.r1) * 8 + kSlot + i];
  }
}
// ---- The same fragments as packed fp32 pairs, for kernels whose CTA runs several groups of 8 warps: a[j] is
// the column pair col(j), col(j) + 1 of row r0, b[j] that of row r1.  `bar` = the group's first of four named
// barriers (one per warp pair), `xch` the group's exchange area (kXchBytes).
constexpr uint32_t kXchBytes = 2 * 2 * 64 * 2 * 4;      // two exchanges x two column halves x 64 rows x two values
struct TokFrag {
  f32x2 a[4], b[4];
};
__device__ __forceinline__ void frag_ld(const TokMap& m, uint32_t tmem_acc, TokFrag& f) {
  uint32_t u[16];
  tmem_ld_16x256b_x4(tmem_acc + m.taddr, u);
  tmem_wait_ld();
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    f.a[j] = pk(u[4 * j], u[4 * j + 1]);
    f.b[j] = pk(u[4 * j + 2], u[4 * j + 3]);
  }
}
// the raw bf16 pairs of a swizzled tile: w[2j] row r0, w[2j + 1] row r1
__device__ __forceinline__ void frag_ld_raw(const TokMap& m, const uint8_t* tile, uint32_t (&w)[8]) {
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    w[2 * j] = *reinterpret_cast<const uint32_t*>(tile + m.off(m.r0, j));
    w[2 * j + 1] = *reinterpret_cast<const uint32_t*>(tile + m.off(m.r1, j));
  }
}
__device__ __forceinline__ void frag_st_tile(const TokMap& m, uint8_t* tile, const TokFrag& f) {
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    *reinterpret_cast<uint32_t*>(tile + m.off(m.r0, j)) = f32x2_to_bf16x2(f.a[j]);
    *reinterpret_cast<uint32_t*>(tile + m.off(m.r1, j)) = f32x2_to_bf16x2(f.b[j]);
  }
}
// ... as f16, and raw words as frag_ld_raw gives them
__device__ __forceinline__ void frag_st_tile_h(const TokMap& m, uint8_t* tile, const TokFrag& f) {
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    *reinterpret_cast<uint32_t*>(tile + m.off(m.r0, j)) = f32x2_to_f16x2(f.a[j]);
    *reinterpret_cast<uint32_t*>(tile + m.off(m.r1, j)) = f32x2_to_f16x2(f.b[j]);
  }
}
__device__ __forceinline__ void frag_st_raw(const TokMap& m, uint8_t* tile, const uint32_t (&w)[8]) {
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    *reinterpret_cast<uint32_t*>(tile + m.off(m.r0, j)) = w[2 * j];
    *reinterpret_cast<uint32_t*>(tile + m.off(m.r1, j)) = w[2 * j + 1];
  }
}
// ... straight to a row-major [64][64] bf16 tile in global memory
__device__ __forceinline__ void frag_st_global(const TokMap& m, __nv_bfloat16* tile, const TokFrag& f) {
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    *reinterpret_cast<uint32_t*>(tile + m.r0 * 64 + m.col(j)) = f32x2_to_bf16x2(f.a[j]);
    *reinterpret_cast<uint32_t*>(tile + m.r1 * 64 + m.col(j)) = f32x2_to_bf16x2(f.b[j]);
  }
}
// per-column vector (fp32[64] in shared memory): the thread's four column pairs
__device__ __forceinline__ f32x2 frag_col(const TokMap& m, const float* vec, int j) {
  return *reinterpret_cast<const f32x2*>(vec + m.col(j));
}
// two sums per row over the row's 8 threads; kSlot = 0 or 1 picks the exchange (each once per phase)
template <int kSlot>
__device__ __forceinline__ void frag_allreduce2(const TokMap& m, float (&a)[2], float (&b)[2], float* xch, uint32_t bar) {
#pragma unroll
  for (int s = 1; s <= 2; s <<= 1) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      a[i] += __shfl_xor_sync(0xffffffffu, a[i], s);
      b[i] += __shfl_xor_sync(0xffffffffu, b[i], s);
    }
  }
  float2* x = reinterpret_cast<float2*>(xch) + kSlot * 128;
  if (m.l3 == 0) {
    x[m.colhalf * 64 + m.r0] = make_float2(a[0], a[1]);
    x[m.colhalf * 64 + m.r1] = make_float2(b[0], b[1]);
  }
  named_bar_sync(bar + m.quad, 64);
  const float2 oa = x[(m.colhalf ^ 1) * 64 + m.r0], ob = x[(m.colhalf ^ 1) * 64 + m.r1];
  a[0] += oa.x; a[1] += oa.y;
  b[0] += ob.x; b[1] += ob.y;
}
// LayerNorm of the thread's two rows in place (x -> (x - mean) / std), returns 1/std per row.  Mean and sum of
// squared deviations are merged pairwise (Chan, Golub and LeVeque's update for equal counts): as accurate as a
// second pass about the mean, with one exchange between the warp pair instead of two.  Uses exchange 0.
__device__ __forceinline__ void frag_layernorm(const TokMap& m, TokFrag& f, float eps, float* xch, uint32_t bar,
                                               float& rs0, float& rs1) {
  float m0 = hsum(add2(add2(f.a[0], f.a[1]), add2(f.a[2], f.a[3]))) * 0.125f;
  float m1 = hsum(add2(add2(f.b[0], f.b[1]), add2(f.b[2], f.b[3]))) * 0.125f;
  f32x2 q0 = 0ull, q1 = 0ull;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const f32x2 d0 = add2(f.a[j], pk1(-m0)), d1 = add2(f.b[j], pk1(-m1));
    q0 = fma2(d0, d0, q0);
    q1 = fma2(d1, d1, q1);
  }
  float s0 = hsum(q0), s1 = hsum(q1);
#pragma unroll
  for (int s = 1; s <= 2; s <<= 1) {
    const float n0 = __shfl_xor_sync(0xffffffffu, m0, s), n1 = __shfl_xor_sync(0xffffffffu, m1, s);
    const float t0 = __shfl_xor_sync(0xffffffffu, s0, s), t1 = __shfl_xor_sync(0xffffffffu, s1, s);
    const float d0 = n0 - m0, d1 = n1 - m1;
    m0 = 0.5f * (m0 + n0);
    m1 = 0.5f * (m1 + n1);
    s0 = fmaf(d0 * d0, 4.f * s, s0 + t0);
    s1 = fmaf(d1 * d1, 4.f * s, s1 + t1);
  }
  float2* x = reinterpret_cast<float2*>(xch);
  if (m.l3 == 0) {
    x[m.colhalf * 64 + m.r0] = make_float2(m0, s0);
    x[m.colhalf * 64 + m.r1] = make_float2(m1, s1);
  }
  named_bar_sync(bar + m.quad, 64);
  const float2 o0 = x[(m.colhalf ^ 1) * 64 + m.r0], o1 = x[(m.colhalf ^ 1) * 64 + m.r1];
  {
    const float d0 = o0.x - m0, d1 = o1.x - m1;
    m0 = 0.5f * (m0 + o0.x);
    m1 = 0.5f * (m1 + o1.x);
    s0 = fmaf(d0 * d0, 16.f, s0 + o0.y);
    s1 = fmaf(d1 * d1, 16.f, s1 + o1.y);
  }
  rs0 = rsqrtf(s0 * (1.f / 64.f) + eps);
  rs1 = rsqrtf(s1 * (1.f / 64.f) + eps);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    f.a[j] = mul2(add2(f.a[j], pk1(-m0)), pk1(rs0));
    f.b[j] = mul2(add2(f.b[j], pk1(-m1)), pk1(rs1));
  }
}

// Column sums of fragments over a warp's 16 rows: v[2j], v[2j + 1] hold this lane's sums over its own rows for the
// column pair j.  The eight lanes that share a pair halve the set at every exchange, so that seven shuffles leave every
// lane with the total of one column: col(2 * bit4 + bit3 of the lane) + bit2.
__device__ __forceinline__ float frag_colsum(const f32x2 (&v)[4], int lane) {
  float k[8];
#pragma unroll
  for (int j = 0; j < 4; ++j) upk(v[j], k[2 * j], k[2 * j + 1]);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const bool up = lane & 16;
    const float send = up ? k[i] : k[4 + i], keep = up ? k[4 + i] : k[i];
    k[i] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const bool up = lane & 8;
    const float send = up ? k[i] : k[2 + i], keep = up ? k[2 + i] : k[i];
    k[i] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
  }
  const bool up = lane & 4;
  return (up ? k[1] : k[0]) + __shfl_xor_sync(0xffffffffu, up ? k[0] : k[1], 4);
}
__device__ __forceinline__ int frag_colsum_col(const TokMap& m, int lane) {
  return m.colhalf * 32 + (lane >> 3) * 8 + m.l3 * 2 + ((lane >> 2) & 1);
}

}  // namespace tttdev
