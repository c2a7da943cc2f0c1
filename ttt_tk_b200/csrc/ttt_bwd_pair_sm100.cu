// TTT-MLP backward for sm_100a with two CTAs per (batch, head) stream: one recomputes, one sweeps.
//
// Like ttt_bwd_sm100.cu it replaces the reference's bwd_ttt_mlp_ker (kernels/ttt_backward/ttt.cu:179-1443); the math is
// that of kernels/ttt_backward/matching.py:57-342 (forward with saved intermediates, then the
// hand-derived reverse step), driven like kernels/ttt_backward/matching.py:539-663: for every
// checkpoint group, last to first, recompute the forward from the group's checkpoint, then
// sweep the group in reverse.
//
// Everything that does not depend on the gradient state is done by the recompute, which therefore ends each mini-batch
// with the backward of the output LayerNorm, dL/dZ1_bar and dQ; the sweep is left with the four dependent MMA phases of
// the update rule's backward.  The two run side by side, one CTA each: while one sweeps group g, the other recomputes group
// g - 1.  The sweep frees the slots of its group from the last mini-batch to the first, so every other group numbers its
// slots backwards and the recompute fills them in the order in which they become free.
//
// Layout conventions are those of the forward kernel: every 64x256 / 256x64 quantity is
// "hidden-major" (hidden unit = TMEM lane), every 64x64 quantity "token-major" (token = TMEM lane, M = 64).  A CTA has
// 16 epilogue warps and four helper warps that issue the MMAs and the bulk copies and wait for both, so that no epilogue
// warp spends its issue slots on a product or sits on a buffer's barrier.  Epilogues and helpers hand each other work over
// mbarriers; each completes once per mini-batch (E_5 and E_X once more, at the start) and everyone who waits for one waits for
// all its completions.  tests/kernel_order.py derives the order of all accesses from this source and looks for gaps in it.
//
// Recompute (go = dL/dOut).  The chain group (warps 0..7) works a step ahead of the output group (warps 8..15):
//   MMA1  Z1^T = W1^T K^T                     W2     bf16 copy of the new W2; b2
//   EPI1  Z1, X2 = gelu, G' = gelu'           MMA5   Z1b^T = W1^T Q^T
//   MMA2  Z2 = X2 W2                          EPI5   X2b = gelu, gelu'
//   LN    x_hat_fused, gZ2, U2 = -eta gZ2     MMA6   Z2b = X2b W2
//   MMA3  R^T = W2 gZ2^T                      S4     gZ2b = LNbwd(go gamma; LN(Z2b + b2));  d_gamma, d_beta
//   EPI3  gZ1 = R G'                          G1     gX2b^T = W2 gZ2b^T
//   MMA4  W1^T += gZ1^T (-eta K), b1;         E1     gZ1b^T = gX2b^T gelu'(Z1b^T)
//         W2 += X2^T U2                       G7     dQ = go + gZ1b W1^T
//   EPI4  bf16 copy of the new W1^T
// Tensor memory: W1^T | W2 (fp32) | chain accumulator | output accumulator, 128 columns each.
//
// Scratch.  Per mini-batch the recompute leaves, in the caller's `*_group` tensors, raw images of swizzled shared-memory
// tiles moved by bulk copies in both directions: [256][64 tok] Z1 (f16: the sweep evaluates gelu' and gelu'' of it in
// packed f16), X2, gZ1, X2b (X2_bar_group), gZ1b (Z1_bar_group), bf16 W1^T / W2 before the update (first 32 KB of the
// W*_init_group slots); [64 tok][64] x_hat_fused, gZ2, gZ2b (x_hat_ln_group); fp32 1/std of the fused LayerNorm
// (std_fused_group), its row sums of grad_x_hat x_hat (b2_init_group), column sums of gZ2b (std_ln_group), row sums of
// gZ1b (b1_init_group).
//
// Reverse step for mini-batch i (G* = gradient w.r.t. the state after the update), all 16 warps:
//   E2   (gelu'(Z1), gelu''(Z1) under G15;)  bf16 snapshots of G_W1^T, then of G_W2 (the "last" values of the update rule)
//   G4   A1raw^T = G_W1^T K^T   G8  T1 = gZ1 G_W1
//   E3   A1^T = -eta (A1raw^T + G_b1);  P^T = A1^T gelu'(Z1^T);  S^T = A1^T gelu''(Z1^T), kept in registers to E5
//   G6   acc2 = P W2            G10 G_W2 += P^T gZ2              G5  acc1 = X2 G_W2
//   E4   A2 = -eta (acc1 + G_b2) + acc2, second-order LayerNorm terms -> gZ2in; d_gamma, d_beta, dV, d_eta
//   G12  R^T = W2 gZ2^T         G11b gX2^T = G_W2 (-eta gZ2)^T   (both while E4 computes)
//   G2   G_W2 += X2b^T gZ2b     G3  G_W1^T += gZ1b^T Q           (of mini-batch i - 1, which nothing waits for)
//   G11a gX2^T += W2 gZ2in^T    G14 G_W2 += X2^T gZ2in
//   E5   gZ1in^T = gX2^T gelu'(Z1^T) + R^T S^T;  G_b1 += row sums
//   G15  G_W1^T += gZ1in^T K    G13 dK = partial + gZ1in W1^T    (finished under the next step's G4)
// Tensor memory: G_W1^T | G_W2 (fp32) | A1raw, acc2, R | T1 and acc1, gX2, dK in the place of acc1.
// Five hidden-major buffers: one holds W2, then W1; the other four change roles from step to step (see `turn`).
//
// What bounds it: issue and the fp32 pipe in the epilogues of either role, then instruction fetch: both programs together
// exceed the 128 KB instruction cache that the SMs of a TPC share, which is why the helper warps run tables in loops and
// why two streams share a cluster of four.  Registers come next (104 a thread: E4 runs with E5's 32 in place).  Measured
// per mini-batch: 60 streams in groups of 5 20.2 us with the hidden units split over two CTAs -> 11.7; 32 streams in
// groups of 16 13.2 with four -> 8.5; 4 streams in groups of 4 14.0 with four -> 10.7, most of it the turn from group to
// group (one slot to spare).  Steps on the way, at 60 streams: 21.6 with helpers written out and 860 bytes of spills, 19.3
// with rolled MMA issue, 16.2 with tables, 14.4 with two streams to a cluster, 13.6 with a branch per role, 13.0 with X2
// loaded where Z1 was and products prepared before their waits, 12.7 with -eta in K (no U1) and checkpoints loaded ahead, 12.6 with
// slots freed when their last load has landed (groups of 4: 12.0 -> 11.7).  12.1 with the sweep's products written out and the
// clock left to the helpers (32 streams in groups of 16 9.9 -> 9.4, 4 in groups of 4 11.7 -> 11.0): the issuing warp took 1200
// cycles a product, of which the tensor pipe needs 320 to 500, and with thirteen of them was busy all of a step's 15700; the
// epilogues' waits carried a clock's worth of instructions each (11 KB in all; with them again, and all else as it is, 60 streams x
// 37 430 -> 448 us, 32 x 128 1138 -> 1187, 4 x 32 339 -> 349).  11.7 with a copy's addresses and sizes put
// together before the events that it waits for (8.5 at 32 streams, 10.7 at 4).  Not kept: the sweep running on into the next
// group (64 x 64 in groups of 8 654 -> 679 us for both passes: the recompute is as slow, and the sweep then waits in mid-step);
// the recompute's chain starting a group under the output pass of the last (32 x 128 in groups of 16 1136 -> 1167 us, 128 x 64
// in groups of 4 1518 -> 1492).
//
// Deviations from the reference kernel (see include/ttt_mlp_b200.h): outputs are overwritten,
// not accumulated; `Out` is never touched.  Every wait is bounded.
#include <mutex>
#include <type_traits>

#define TTT_WAIT_INLINE
#include "ttt_cluster.cuh"
#include "ttt_internal.h"

using namespace tttcl;

namespace {

constexpr int kEpi = 512;                    // epilogue threads
constexpr int kGroup = 256;                  // threads of the recompute's chain / output group
constexpr int kThreads = kEpi + 128;         // and four helper warps
// registers per thread: the block is launched with 96 of them
constexpr int kRegsEpi = 104, kRegsHelp = 64;
static_assert(kRegsEpi * kEpi + kRegsHelp * 128 <= 96 * kThreads, "the shares add up to the block's registers at launch");

// named barriers
constexpr uint32_t kBarPairC = 1, kBarPairO = 5, kBarC = 9, kBarO = 10;      // recompute: warp pairs of a group, groups
constexpr uint32_t kBarQuad = 1;                                             // sweep: four warps of a quadrant

// ---- shared memory: five hidden-major buffers and seven token tiles in either role, then vectors
constexpr uint32_t OFF_BIG = 0;
constexpr uint32_t OFF_T = 5 * BIG;
constexpr uint32_t OFF_NETA = OFF_T + 7 * TILE;        // recompute: bf16[64] -eta, a row of a swizzled tile (1024-byte aligned)
constexpr uint32_t OFF_GAMMA = OFF_NETA + 128;
constexpr uint32_t OFF_BETA = OFF_GAMMA + 256;
constexpr uint32_t OFF_BAR = OFF_BETA + 256;
constexpr uint32_t OFF_MISC = OFF_BAR + 512;
constexpr uint32_t OFF_VECS = OFF_MISC + 64;
// recompute
constexpr uint32_t R_W1 = 0, R_W2 = BIG, R_X2 = 2 * BIG;
constexpr uint32_t R_ZG = 3 * BIG;                      // Z1, then gZ1
constexpr uint32_t R_XB = 4 * BIG;                      // X2b, then gZ1b
constexpr uint32_t R_K = OFF_T;                         // + stage
constexpr uint32_t R_V = OFF_T + 2 * TILE;              // V, then x_hat_fused on its way out
constexpr uint32_t R_Q = OFF_T + 3 * TILE;              // Q, then gZ2b
constexpr uint32_t R_GO = OFF_T + 4 * TILE;             // dL/dOut, then dQ on its way out
constexpr uint32_t R_U2 = OFF_T + 5 * TILE, R_GZ2 = OFF_T + 6 * TILE;
constexpr uint32_t R_ETA = OFF_VECS;                    // bf16[2][64]
constexpr uint32_t R_B1 = R_ETA + 256;                  // fp32[256]
constexpr uint32_t R_B2 = R_B1 + 1024;                  // fp32[64]
// fp32[64] 1/std of the fused LayerNorm, fp32[64] sum(grad_x_hat_fused x_hat_fused), on their way out
constexpr uint32_t R_SIG = R_B2 + 256;
constexpr uint32_t R_VEC = R_SIG + 512;                 // fp32[256] row sums of gZ1b, fp32[64] column sums of gZ2b, on their way out
constexpr uint32_t R_CSC = R_VEC + 1280;                // fp32[4][64] column sums per quadrant: chain ...
constexpr uint32_t R_CSO = R_CSC + 1024;                // ... and output group
constexpr uint32_t R_XCHC = R_CSO + 1024;               // row-sum exchanges
constexpr uint32_t R_XCHO = R_XCHC + kXchBytes;
constexpr uint32_t R_END = R_XCHO + kXchBytes;
// sweep
constexpr uint32_t S_K = OFF_T;                         // + parity of the step: K, then dK on its way out
constexpr uint32_t S_GZ2 = OFF_T + 2 * TILE;
constexpr uint32_t S_V = OFF_T + 3 * TILE;              // V, then dV on its way out
constexpr uint32_t S_XF = OFF_T + 4 * TILE;             // x_hat_fused, then gZ2in
constexpr uint32_t S_Q = OFF_T + 5 * TILE;              // Q of the next step, then U2
constexpr uint32_t S_GZB = OFF_T + 6 * TILE;            // gZ2b of the next step
constexpr uint32_t S_ETA = OFF_VECS;                    // bf16[2][64]
constexpr uint32_t S_SIG = S_ETA + 256;                 // fp32[2][64], as R_SIG
constexpr uint32_t S_VEC = S_SIG + 512;                 // fp32[256] row sums of gZ1b, fp32[64] column sums of gZ2b
constexpr uint32_t S_GB1 = S_VEC + 1280;                // fp32[256] dL/db1
constexpr uint32_t S_GB2 = S_GB1 + 1024;                // fp32[64] dL/db2
constexpr uint32_t S_PART = S_GB2 + 256;                // + parity of the step: fp32[2][64] sums over the hidden units of gZ1 G_b1
constexpr uint32_t S_CS = S_PART + 1024;                 // fp32[4][64] column sums of gZ2in per quadrant
constexpr uint32_t S_X1 = S_CS + 1024;                  // float2[4][64] row-sum exchanges
constexpr uint32_t S_X2 = S_X1 + 2048;
constexpr uint32_t S_END = S_X2 + 2048;
constexpr uint32_t SMEM_BYTES = R_END > S_END ? R_END : S_END;
static_assert(SMEM_BYTES <= 232448, "exceeds the 227 KB per-CTA shared memory of sm_100");

// ---- barriers
enum : int {
  // recompute: loads
  RK, RK1, RV, RQ, RGO,
  // products: MMA1, MMA3, MMA4's W1 (one per 128-row block), MMA2, MMA4's W2, MMA5, MMA6, G1, G7
  RA, RA1, RZ, RW2UPD, RB, RBZ, RG1, RG7,
  // epilogues done: a checkpoint in tensor memory, its bf16 W1 and W2 in place, EPI1, LN, EPI3, EPI4, W2 copy, EPI5, S4, E1, dQ
  E_LDT, E_LD1, E_LD2, E_1, E_2, E_3, E_W1, E_W2, E_O5, E_OS4, E_OE1, E_ODQ,
  // images have left shared memory: Z1 and W1^T; X2, gZ1, gZ2; X2b and W2 (and a checkpoint's W2); gZ1b
  F_ZG, F_X, F_XB, F_XB2,
  kRecBars,
  // sweep: loads
  SW2 = kRecBars, SW1, SGZ1, SX2, SZ1, SGZ1B, SX2B, SK, SGZ2, SV, SXF, SQ,
  // products: G4 and G8, G10, G5 and G6, G11b and G2, G11a, G3, G15, G13
  C2, C10, C4, CB, C5, C3, C6, C7,
  // epilogues done: Z1 read, E2 (G_W1), E2 (G_W2, dK), E3, E4's accumulators read and U2, gZ2in, dV, E5 and d_eta's addends;
  // gZ1 G_b1 summed, d_eta's addends read
  E_D, E_S1, E_S2, E_P, E_T, E_Z, E_V, E_5, E_PART, E_X,
  // the scratch slots of a group are written, by parity of the group: where a short first group and the next fit in beside
  // each other, both can be before the sweep has looked
  BGROUP, BGROUP1,
  BDRAIN,      // abort path only
  kBars
};
static_assert(kBars * 8 <= 512 && kRecBars <= 32 && BDRAIN - kRecBars <= 32, "barrier storage, parity masks");

// tensor-memory columns: see the head of the file
constexpr uint32_t TM_S1 = 0;
constexpr uint32_t TM_S2 = 128;
constexpr uint32_t TM_A = 256;
constexpr uint32_t TM_B = 384;
constexpr uint32_t TM_COLS = 512;

// the arrays of a scratch slot
enum : int { A_X2, A_Z1, A_GZ1, A_X2B, A_GZ1B, A_W1, A_W2, A_XHF, A_GZ2, A_GZ2B, A_RS, A_CS, A_SIG, A_S3, A_COUNT };

// ---- programs of the helper warps.  Those of the copies are run by small loops: written out, a step's are 40 KB of code, which
// the instruction cache that two SMs share has no room for; that of the products is, in 20 KB (see `issue`).
// A copy: one lane of the copying warp owns it and issues it when its event has been seen.
enum : uint8_t { R_NONE, R_GZ, R_Z, R_S1, R_S2, R_A };                       // destination: fixed, or a rotating buffer's
enum : uint8_t { K_NONE, K_LOAD, K_TMA, K_STORE };                           // bulk load, tiled load, bulk store
enum : uint8_t { M_Q, M_K, M_V, M_GO };                                      // tensor maps
enum : uint8_t { A_ETA = A_COUNT };                                          // source outside the scratch, indexed by mini-batch
struct CopyOp {
  uint8_t event, kind, src, bar;
  uint8_t role, next, only_next, pad;      // next: of the following mini-batch's slot; only_next: only if there is one
  uint32_t off, par;                       // shared-memory offset, plus par for odd steps
  uint32_t bytes, arm;                     // arm: bytes the barrier is armed with (0: by another copy)
};
// One product of the reverse step: waits, operands (rotating buffer, or offset), commit.
constexpr uint8_t kNo = 255;
enum : uint8_t { P_HID, P_HID_ACC, P_HID_MN, P_TOK };      // hidden-major: B K-major, the same accumulating, B MN-major accumulating
struct MmaOp {
  uint8_t w0, w1, commit, kind;
  uint8_t ra, rb, only_next, pad;
  uint32_t a, b;                           // b: K's parity offset is added if b == S_K
  uint32_t d;
};

struct BwdParams {
  const __nv_bfloat16* eta;
  const float* gamma;
  const float* beta;
  const float* W1c; const float* b1c; const float* W2c; const float* b2c;
  uint8_t* sc[A_COUNT];     // scratch: each array's first slot
  uint32_t stride[A_COUNT]; // and the bytes from slot to slot
  uint8_t* spare[A_COUNT];  // the same of the slots beyond one per mini-batch, which lie 256 KB apart
  // upstream
  const float* gW1_last; const float* gb1_last; const float* gW2_last; const float* gb2_last;
  // outputs
  float* d_gamma; float* d_beta;
  float* gW1; float* gb1; float* gW2; float* gb2;
  __nv_bfloat16* d_eta;
  int H, NC, cgs, nck;
  int first, streams;       // this launch's first stream, and the call's number of them
  int drop_load;            // test only: mini-batch whose recompute inputs stream 0 never loads (-1: none)
  uint32_t* status;
  uint64_t wait_limit_ns;
};

// ---- 64 x 64 token-major tiles spread over 16 warps: a warp takes the 16 rows of its quadrant and 16 of the 64 columns,
// a thread rows r0 and r1 = r0 + 8 and the column pairs col(0), col(1) (the TokMap fragment, halved).
struct TokMap16 {
  int quad, cq, l3;
  int r0, r1;
  uint32_t taddr;
  __device__ __forceinline__ TokMap16(int warp, int lane)
      : quad(warp & 3), cq(warp >> 2), l3(lane & 3), r0((warp & 3) * 16 + (lane >> 2)), r1(r0 + 8),
        taddr((static_cast<uint32_t>((warp & 3) * 32) << 16) + static_cast<uint32_t>((warp >> 2) * 16)) {}
  __device__ __forceinline__ int col(int j) const { return cq * 16 + j * 8 + l3 * 2; }
  __device__ __forceinline__ uint32_t off(int r, int j) const { return sw128_off(r, cq * 2 + j) + l3 * 4; }
};
struct Frag16 {
  f32x2 a[2], b[2];
};
__device__ __forceinline__ void tmem_ld_16x256b_x2(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ Frag16 f16_pack(const uint32_t (&u)[8]) {
  Frag16 f;
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    f.a[j] = pk(u[4 * j], u[4 * j + 1]);
    f.b[j] = pk(u[4 * j + 2], u[4 * j + 3]);
  }
  return f;
}
// the raw bf16 pairs of a swizzled tile: w[2j] row r0, w[2j + 1] row r1
__device__ __forceinline__ void f16_ld_raw(const TokMap16& m, const uint8_t* tile, uint32_t (&w)[4]) {
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    w[2 * j] = *reinterpret_cast<const uint32_t*>(tile + m.off(m.r0, j));
    w[2 * j + 1] = *reinterpret_cast<const uint32_t*>(tile + m.off(m.r1, j));
  }
}
__device__ __forceinline__ void f16_st_tile(const TokMap16& m, uint8_t* tile, const Frag16& f) {
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    *reinterpret_cast<uint32_t*>(tile + m.off(m.r0, j)) = f32x2_to_bf16x2(f.a[j]);
    *reinterpret_cast<uint32_t*>(tile + m.off(m.r1, j)) = f32x2_to_bf16x2(f.b[j]);
  }
}
__device__ __forceinline__ f32x2 f16_col(const TokMap16& m, const float* vec, int j) {
  return *reinterpret_cast<const f32x2*>(vec + m.col(j));
}
// Column sums over a warp's 16 rows, the eight lanes that share a column pair halving the set at every exchange: every
// lane ends with the total of column f16_colsum_col (lanes that differ in bit 2 with the same one).
__device__ __forceinline__ float f16_colsum(f32x2 v0, f32x2 v1, int lane) {
  float k[4];
  upk(v0, k[0], k[1]);
  upk(v1, k[2], k[3]);
  const bool u4 = lane & 16, u3 = lane & 8;
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const float send = u4 ? k[i] : k[2 + i], keep = u4 ? k[2 + i] : k[i];
    k[i] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
  }
  const float s = (u3 ? k[1] : k[0]) + __shfl_xor_sync(0xffffffffu, u3 ? k[0] : k[1], 8);
  return s + __shfl_xor_sync(0xffffffffu, s, 4);
}
__device__ __forceinline__ int f16_colsum_col(const TokMap16& m, int lane) {
  return m.cq * 16 + ((lane >> 4) & 1) * 8 + m.l3 * 2 + ((lane >> 3) & 1);
}
// two sums per row over the row's four lanes and four warps; xch: float2[4][64], bar: the first of four named barriers
__device__ __forceinline__ void f16_row_sums(const TokMap16& m, float (&a)[2], float (&b)[2], float2* xch, uint32_t bar) {
#pragma unroll
  for (int s = 1; s <= 2; s <<= 1) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      a[i] += __shfl_xor_sync(0xffffffffu, a[i], s);
      b[i] += __shfl_xor_sync(0xffffffffu, b[i], s);
    }
  }
  if (m.l3 == 0) {
    xch[m.cq * 64 + m.r0] = make_float2(a[0], a[1]);
    xch[m.cq * 64 + m.r1] = make_float2(b[0], b[1]);
  }
  named_bar_sync(bar + m.quad, 128);
  const float2 a0 = xch[m.r0], a1 = xch[64 + m.r0], a2 = xch[128 + m.r0], a3 = xch[192 + m.r0];
  const float2 b0 = xch[m.r1], b1 = xch[64 + m.r1], b2 = xch[128 + m.r1], b3 = xch[192 + m.r1];
  a[0] = (a0.x + a1.x) + (a2.x + a3.x); a[1] = (a0.y + a1.y) + (a2.y + a3.y);
  b[0] = (b0.x + b1.x) + (b2.x + b3.x); b[1] = (b0.y + b1.y) + (b2.y + b3.y);
}

// D[128 x 16] = A B^T with A in tensor memory (as in mma_hidden_ta) and B 16 rows of 64 bf16 from `b_smem` on (K-major)
__device__ __forceinline__ void mma_rowsum_ta(uint32_t tmem_d, uint32_t tmem_a, uint32_t b_smem, uint32_t lead) {
  constexpr uint32_t idesc = umma_idesc_bf16(128, 16, false, false, false);
  const uint32_t b0 = desc_lo(b_smem, 16);
  mma_lead_ta<false>(tmem_d, tmem_a, b0, idesc, lead);
#pragma unroll
  for (int j = 1; j < 4; ++j) mma_lead_ta<true>(tmem_d, tmem_a + j * 8, b0 + j * (32u >> 4), idesc, lead);
}

// ---- across the two CTAs of a stream
__device__ __forceinline__ void st_release_cluster(uint32_t addr, uint32_t v) {
  asm volatile("st.release.cluster.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ uint32_t ld_acquire_cluster(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.acquire.cluster.shared::cta.u32 %0, [%1];" : "=r"(v) : "r"(smem_u32(p)) : "memory");
  return v;
}
__device__ __forceinline__ float ld_cluster_f32(uint32_t addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void fence_proxy_async_all() { asm volatile("fence.proxy.async;" ::: "memory"); }

enum : uint8_t { V_D, V_S2, V_C2, V_PART, V_C10, V_CB, V_C5, V_V, V_C3, V_C6, V_C7, V_COUNT };      // the sweep copies' events
__constant__ const uint8_t kSweepEvent[V_COUNT] = {E_D, E_S2, C2, E_PART, C10, CB, C5, E_V, C3, C6, C7};
constexpr int kSweepCopies = 19;
__constant__ const CopyOp kSweepCopy[kSweepCopies] = {
    {V_D, K_LOAD, A_X2, SX2, R_Z, 0, 0, 0, 0, 0, BIG, BIG},
    {V_PART, K_LOAD, A_X2B, SX2B, R_GZ, 1, 1, 0, 0, 0, BIG, BIG + TILE + 1280},
    {V_PART, K_LOAD, A_GZ2B, SX2B, R_NONE, 1, 1, 0, S_GZB, 0, TILE, 0},
    {V_PART, K_LOAD, A_RS, SX2B, R_NONE, 1, 1, 0, S_VEC, 0, 1024, 0},
    {V_PART, K_LOAD, A_CS, SX2B, R_NONE, 1, 1, 0, S_VEC + 1024, 0, 256, 0},
    {V_C10, K_LOAD, A_GZ1B, SGZ1B, R_S1, 1, 1, 0, 0, 0, BIG, BIG},
    {V_CB, K_TMA, M_Q, SQ, R_NONE, 1, 1, 0, S_Q, 0, TILE, TILE},
    {V_C5, K_LOAD, A_W1, SW1, R_A, 0, 0, 0, 0, 0, BIG, BIG},
    {V_CB, K_LOAD, A_Z1, SZ1, R_S2, 1, 1, 0, 0, 0, BIG, BIG},
    {V_C5, K_LOAD, A_GZ2, SGZ2, R_NONE, 1, 1, 0, S_GZ2, 0, TILE, TILE},
    {V_V, K_TMA, M_K, SK, R_NONE, 1, 1, 0, S_K, TILE, TILE, TILE + 128},
    {V_V, K_LOAD, A_ETA, SK, R_NONE, 1, 1, 0, S_ETA, 128, 128, 0},
    {V_C3, K_LOAD, A_GZ1, SGZ1, R_S1, 1, 1, 0, 0, 0, BIG, BIG},
    {V_C3, K_LOAD, A_XHF, SXF, R_NONE, 1, 1, 0, S_XF, 0, TILE, TILE + 512},
    {V_C3, K_LOAD, A_SIG, SXF, R_NONE, 1, 1, 0, S_SIG, 0, 256, 0},
    {V_C3, K_LOAD, A_S3, SXF, R_NONE, 1, 1, 0, S_SIG + 256, 0, 256, 0},
    {V_C6, K_TMA, M_V, SV, R_NONE, 1, 1, 0, S_V, 0, TILE, TILE},
    {V_C7, K_LOAD, A_W2, SW2, R_A, 1, 1, 0, 0, 0, BIG, BIG},
    {V_COUNT, K_NONE, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0}};
// Two of these waits are not for an operand, they stand where the tensor pipe is busy or E4 runs: E_PART before G11b is for E5,
// which overwrites gZ1 and adds to G_b1, and E_X before G8 for E4, which writes over the last step's addends to d_eta.
constexpr int kSweepMmas = 13;
constexpr __constant__ const MmaOp kSweepMma[kSweepMmas] = {
    {E_S1, SK, kNo, P_HID, R_S1, R_NONE, 0, 0, 0, S_K, TM_A},                  // G4
    {SGZ1, E_X, C2, P_TOK, R_GZ, R_S1, 0, 0, 0, 0, TM_B},                     // G8
    {E_S2, SX2, kNo, P_TOK, R_Z, R_S2, 0, 0, 0, 0, TM_B + 64},                // G5
    {E_P, SW2, C4, P_TOK, R_S1, R_A, 0, 0, 0, 0, TM_A},                       // G6
    {SGZ2, kNo, C10, P_HID_MN, R_S1, R_NONE, 0, 0, 0, S_GZ2, TM_S2},          // G10
    {E_T, kNo, kNo, P_HID, R_A, R_NONE, 0, 0, 0, S_GZ2, TM_A},                // G12
    {E_PART, kNo, kNo, P_HID, R_S2, R_NONE, 0, 0, 0, S_Q, TM_B},              // G11b
    {SX2B, kNo, CB, P_HID_MN, R_GZ, R_NONE, 1, 0, 0, S_GZB, TM_S2},           // G2 of the next step
    {E_Z, kNo, C5, P_HID_ACC, R_A, R_NONE, 0, 0, 0, S_XF, TM_B},              // G11a
    {kNo, kNo, kNo, P_HID_MN, R_Z, R_NONE, 0, 0, 0, S_XF, TM_S2},             // G14
    {SGZ1B, SQ, C3, P_HID_MN, R_S1, R_NONE, 1, 0, 0, S_Q, TM_S1},             // G3 of the next step
    {E_5, kNo, C6, P_HID_MN, R_GZ, R_NONE, 0, 0, 0, S_K, TM_S1},              // G15
    {SW1, kNo, C7, P_TOK, R_GZ, R_A, 0, 0, 0, 0, TM_B + 64}};                 // G13

// copies of the recompute: chain (loads of K, eta, V; images out) and output group (loads of Q, dL/dOut; images out)
enum : uint8_t { Y_LD, Y_1, Y_2, Y_3, Y_W, Y_LOADS };      // events: checkpoint in place, then the group's epilogues in order
constexpr int kRecCopies = 11;
__constant__ const CopyOp kChainCopy[kRecCopies] = {
    {Y_1, K_STORE, A_X2, 0, 0, 0, 0, 0, R_X2, 0, BIG, 0},
    {Y_1, K_STORE, A_Z1, 0, 0, 0, 0, 0, R_ZG, 0, BIG, 0},
    {Y_2, K_STORE, A_XHF, 0, 0, 0, 0, 0, R_V, 0, TILE, 0},
    {Y_2, K_STORE, A_GZ2, 0, 0, 0, 0, 0, R_GZ2, 0, TILE, 0},
    {Y_2, K_STORE, A_SIG, 0, 0, 0, 0, 0, R_SIG, 0, 256, 0},
    {Y_2, K_STORE, A_S3, 0, 0, 0, 0, 0, R_SIG + 256, 0, 256, 0},
    {Y_3, K_STORE, A_GZ1, 0, 0, 0, 0, 0, R_ZG, 0, BIG, 0},
    {Y_W, K_STORE, A_W1, 0, 0, 1, 1, 0, R_W1, 0, BIG, 0},
    {Y_LOADS, K_TMA, M_K, RK, 0, 0, 0, 0, R_K, TILE, TILE, TILE + 128},
    {Y_LOADS, K_LOAD, A_ETA, RK, 0, 0, 0, 0, R_ETA, 128, 128, 0},
    {Y_LOADS, K_TMA, M_V, RV, 0, 0, 0, 0, R_V, 0, TILE, TILE}};
__constant__ const CopyOp kOutCopy[kRecCopies] = {
    {Y_1, K_STORE, A_X2B, 0, 0, 0, 0, 0, R_XB, 0, BIG, 0},
    {Y_2, K_STORE, A_GZ2B, 0, 0, 0, 0, 0, R_Q, 0, TILE, 0},
    {Y_3, K_STORE, A_GZ1B, 0, 0, 0, 0, 0, R_XB, 0, BIG, 0},
    {Y_3, K_STORE, A_RS, 0, 0, 0, 0, 0, R_VEC, 0, 1024, 0},
    {Y_3, K_STORE, A_CS, 0, 0, 0, 0, 0, R_VEC + 1024, 0, 256, 0},
    {Y_W, K_STORE, A_W2, 0, 0, 1, 1, 0, R_W2, 0, BIG, 0},
    {Y_LOADS, K_TMA, M_Q, RQ, 0, 0, 0, 0, R_Q, 0, TILE, TILE},
    {Y_LOADS, K_TMA, M_GO, RGO, 0, 0, 0, 0, R_GO, 0, TILE, TILE},
    {Y_LOADS, K_NONE, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0},
    {Y_LOADS, K_NONE, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0},
    {Y_LOADS, K_NONE, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0}};
constexpr int kLaneK = 8, kLaneV = 10, kLaneQ = 6, kLaneGo = 7;      // the loads' places in these (K's eta behind it)

// kStreams: streams to a cluster, whose first kStreams CTAs sweep and whose others recompute.  Two where all fit at once: the
// SMs of a TPC then run the same role and share its instructions (60 streams: 16.2 -> 13.6 us per mini-batch; with one of
// each role the two programs evict one another from the instruction cache).
template <int kStreams>
__global__ void __launch_bounds__(kThreads, 1)
ttt_bwd_pair_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
               const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmGo,
               const __grid_constant__ CUtensorMap tmDQ, const __grid_constant__ CUtensorMap tmDK,
               const __grid_constant__ CUtensorMap tmDV, const BwdParams p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  if (smem_u32(smem) & 1023u) {       // the swizzled tiles need it; never seen
    if (threadIdx.x == 0) atomicExch(p.status, static_cast<uint32_t>(TTT_B200_ERR_LAUNCH));
    return;
  }
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);   // same value, known to be warp-uniform
  const uint32_t crank = cluster_ctarank();
  const bool sweeper = crank < kStreams;
  const uint32_t peer = sweeper ? crank + kStreams : crank - kStreams;
  const int sid = p.first + (blockIdx.x / (2 * kStreams)) * kStreams + (crank % kStreams);
  const bool idle = sid >= p.streams;      // the last cluster's second stream, if there is none: it only keeps step
  const int head = sid % p.H;
  const int NC = p.NC, cgs = p.cgs, nck = p.nck;

  float* sGamma = reinterpret_cast<float*>(smem + OFF_GAMMA);
  float* sBeta = reinterpret_cast<float*>(smem + OFF_BETA);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + OFF_BAR);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + OFF_MISC);
  volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(smem + OFF_MISC + 4);
  volatile uint32_t* never_flag = reinterpret_cast<volatile uint32_t*>(smem + OFF_MISC + 8);   // stays 0
  uint32_t* freed = reinterpret_cast<uint32_t*>(smem + OFF_MISC + 12);      // rank 1: slots the sweep has read so far
  const uint64_t limit = p.wait_limit_ns;

  if (tid == kEpi) {
    for (int i = 0; i < kBars; ++i)
      mbar_init(&bars[i], i >= E_LDT && i <= E_ODQ ? 8 : i >= E_D && i <= E_5 ? 16 : i >= E_PART ? 2 : 1);
    fence_mbar_init();
    *abort_flag = 0;
    *never_flag = 0;
    *freed = 0;
    prefetch_tmap(&tmQ);
    prefetch_tmap(&tmK);
    prefetch_tmap(&tmV);
    prefetch_tmap(&tmGo);
    prefetch_tmap(&tmDQ);
    prefetch_tmap(&tmDK);
    prefetch_tmap(&tmDV);
  }
  if (warp == 0) {
    tmem_alloc(tmem_slot, TM_COLS);
    tmem_relinquish();
  }
  if (tid < 64 && !idle) {
    sGamma[tid] = p.gamma[head * 64 + tid];
    sBeta[tid] = p.beta[head * 64 + tid];
  }
  tc_fence_before_sync();
  __syncthreads();
  cluster_arrive();      // the peer's barriers are initialised before anything is sent there
  cluster_wait();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  const uint32_t lead = elect_one() ? 1u : 0u;         // the lane that issues the MMAs

  // ---- waiting and signalling
  uint32_t phR = 0, phS = 0;      // expected parity per barrier, recompute's and sweep's
  // (one small loop: there are some eighty of these, and the instruction cache is short)
  auto bounded = [&](int b, uint32_t parity) -> bool {
    uint64_t t0 = 0;
    uint32_t spins = 0;
    while (!(b >= BGROUP ? mbar_try_wait_cluster(&bars[b], parity) : mbar_try_wait(&bars[b], parity))) {
      if (warp < 16) {      // (whatever holds an epilogue warp up holds a helper warp up that waits for it: the clock is theirs)
        if (*abort_flag) return false;
        continue;
      }
      if (++spins & 31u) continue;
      if (*abort_flag) return false;
      const uint64_t t = globaltimer_ns();
      if (t0 == 0) t0 = t;
      if (t - t0 > limit) {
        *abort_flag = 1;      // (a peer is told when this CTA has left its loops)
        return false;
      }
    }
    return true;
  };
  auto wait = [&](int b) -> bool {
    uint32_t& ph = b < kRecBars ? phR : phS;
    const uint32_t bit = b < kRecBars ? b : b - kRecBars;
    if (!bounded(b, (ph >> bit) & 1u)) return false;
    ph ^= 1u << bit;
    return true;
  };
  auto wait_mma = [&](int b) {      // a product's completion, by the warps that read its accumulator
    wait(b);
    __syncwarp();
    tc_fence_after_sync();
  };
  auto arrive = [&](int b) { mbar_arrive(&bars[b]); };
  auto done = [&](int b) {          // this warp's share of an epilogue: its writes and tensor-memory reads are over
    fence_proxy_async_smem();
    tc_fence_before_sync();
    __syncwarp();
    if (lane == 0) arrive(b);
  };
  auto commit = [&](int b) { if (lead) umma_commit(&bars[b]); };
  // loads issued so far, for the abort path: parity of each barrier's next load, and whether there was one
  uint32_t ldpR = 0, ldpS = 0, ldaR = 0, ldaS = 0;
  auto arm = [&](int b, uint32_t bytes) {
    mbar_expect_tx(&bars[b], bytes);
    if (b < kRecBars) { ldpR ^= 1u << b; ldaR |= 1u << b; }
    else { ldpS ^= 1u << (b - kRecBars); ldaS |= 1u << (b - kRecBars); }
  };

  // ---- group g (0 = the last of the sequence, the first to be processed): first mini-batch, size, slot of mini-batch j
  auto first_of = [&](int g) { return (nck - 1 - g) * cgs; };
  auto size_of = [&](int g) { return g == 0 ? NC - (nck - 1) * cgs : cgs; };
  // Slots: one per mini-batch of a group and one more for every four, in the second halves of the W*_init_group slots
  // (32 KB each, eight to a slot).  Neighbouring groups number them from opposite ends.
  const int nslots = cgs + cgs / 4;
  auto slot_of = [&](int g, int j) { return g & 1 ? nslots - 1 - j : j; };
  auto row_of = [&](int i) { return (sid * NC + i) * 64; };
  // A slot is free once the sweep has read what it held: a mini-batch of the group before, or, if it is one of those at
  // this end that the group before did not use, of the group before that (which the recompute can reach while the sweep is
  // still in it).
  auto steps_before = [&](int g) { return g == 0 ? 0 : size_of(0) + (g - 1) * cgs; };
  auto wait_slot = [&](int g, int j) -> bool {
    if (g == 0) return true;
    const int own = j - (nslots - size_of(g - 1));                    // step of group g - 1 that reads this slot
    int need = steps_before(g - 1) + own + 1;
    if (own < 0) {
      if (g == 1 || j >= size_of(g - 2)) return true;
      need = steps_before(g - 2) + size_of(g - 2) - j;
    }
    uint64_t t0 = 0;
    bool ok = true;
    while (ok && ld_acquire_cluster(freed) < static_cast<uint32_t>(need)) {
      const uint64_t t = globaltimer_ns();
      if (t0 == 0) t0 = t;
      if (*abort_flag) ok = false;
      else if (t - t0 > limit) {
        *abort_flag = 1;
        ok = false;
      }
    }
    fence_proxy_async_all();
    return __all_sync(0xffffffffu, ok);
  };
  // a group's slots are complete: the bulk stores of this warp are, and the sweep may read them
  auto group_written = [&](int g) {
    tma_wait_group<0>();
    fence_proxy_async_all();
    __threadfence();
    __syncwarp();
    if (lane == 0) mbar_arrive_remote(&bars[BGROUP + (g & 1)], peer);
  };
  // A copying warp's lane: its copy, and where that is in global memory.
  struct Lane {
    CopyOp op;
    const CUtensorMap* map;
    uint8_t* mem;      // slot 0 of the array, or mini-batch 0's learning rates
    uint8_t* far;      // first slot beyond the group's
    uint32_t step;
  };
  auto lane_of = [&](const CopyOp* table, int n) {
    Lane c;
    c.op = table[lane < n ? lane : n - 1];
    c.map = c.op.src == M_Q ? &tmQ : c.op.src == M_K ? &tmK : c.op.src == M_V ? &tmV : &tmGo;
    c.mem = const_cast<uint8_t*>(reinterpret_cast<const uint8_t*>(p.eta)) + long{sid} * NC * 128;
    c.far = nullptr;
    c.step = 128;
#pragma unroll
    for (int a = 0; a < A_COUNT; ++a)      // (selected: an index per lane would put the parameters into local memory)
      if (c.op.src == a) {
        c.step = p.stride[a];
        c.mem = p.sc[a] + long{sid} * cgs * p.stride[a];
        c.far = p.spare[a] + long{sid} * cgs * 65536;
      }
    return c;
  };
  auto place = [&](const Lane& c, int slot) { return slot >= cgs ? c.far + (slot - cgs) * 262144L : c.mem + static_cast<long>(slot) * c.step; };
  // one copy, by the lanes for which `act` holds: mini-batch i, slot `slot`, shared-memory offset `off`, parity of its stage
  auto copy = [&](const Lane& c, bool act, int i, int slot, uint32_t off, uint32_t par, bool dropped) {
    if (!act || dropped) return;
    off += par ? c.op.par : 0u;
    const int b = c.op.bar + (c.op.bar == RK ? par : 0);
    if (c.op.arm) arm(b, c.op.arm);
    if (c.op.kind == K_TMA) {
      tma_load_2d(smem + off, c.map, &bars[b], 0, row_of(i));
    } else {
      const uint32_t n = c.op.src == A_ETA ? i : slot;
      uint8_t* mem = c.op.src != A_ETA && slot >= cgs ? c.far + (slot - cgs) * 262144L : c.mem + static_cast<long>(n) * c.step;
      if (c.op.kind == K_STORE) {
        bulk_store_1d(mem, smem + off, c.op.bytes);
        tma_commit_group();
      } else {
        bulk_load_1d(smem + off, mem, c.op.bytes, &bars[b]);
      }
    }
  };
  auto seen_all = [&](int b) -> bool { return __all_sync(0xffffffffu, wait(b)); };      // by a whole helper warp
  auto quad_sum = [&](const float* cs, int f) { return (cs[f] + cs[64 + f]) + (cs[128 + f] + cs[192 + f]); };

  // =====================================================================================================
  //                                             recompute
  // =====================================================================================================
  const int quad = warp & 3;
  const uint32_t lane_base = static_cast<uint32_t>(quad * 32) << 16;
  const int gwarp = warp & 7, wg = gwarp >> 2, gtid = tid & (kGroup - 1);
  const int hrow8 = wg * 128 + quad * 32 + lane;             // hidden unit owned in the 256-row epilogues of a group
  const TokMap tm8(gwarp, lane);
  int nrec = 0;                                              // mini-batches recomputed so far
  float dgam = 0.f, dbet = 0.f;                              // output group: this lane's column of d_gamma / d_beta
  uint8_t* rW1 = smem + R_W1;
  uint8_t* rW2 = smem + R_W2;
  uint8_t* rX2 = smem + R_X2;
  uint8_t* rZG = smem + R_ZG;
  uint8_t* rXB = smem + R_XB;
  float* rB1 = reinterpret_cast<float*>(smem + R_B1);
  float* rB2 = reinterpret_cast<float*>(smem + R_B2);
  float* rVec = reinterpret_cast<float*>(smem + R_VEC);

  // A group's warps meet at named barriers, so they leave the loop by a vote (true: left).  The sweep's never do: once the
  // abort flag is up their waits fail at once, and they run through what is left.
  // A checkpoint into tensor memory, by the chain group: the first one, later ones while the output group is at its last
  // products of the group before (which use the bf16 copies)
  auto load_checkpoint = [&](int g) {
    const long ck = long{sid} * nck + nck - 1 - g;
    const float* W1g = p.W1c + ck * (64 * 256) + hrow8;
#pragma unroll 1
    for (int half = 0; half < 2; ++half) {
      uint32_t v[32];
#pragma unroll
      for (int q = 0; q < 32; ++q) v[q] = __float_as_uint(W1g[(half * 32 + q) * 256]);
      tmem_st32(tmem + lane_base + TM_S1 + wg * 64 + half * 32, v);
    }
    if (g > 0) {      // MMA6 has waited for the last W2 copy
      bounded(RBZ, (nrec - 1) & 1);
      __syncwarp();
      tc_fence_after_sync();
    }
    const float4* W2g = reinterpret_cast<const float4*>(p.W2c + ck * (256 * 64) + hrow8 * 64);
#pragma unroll 1
    for (int half = 0; half < 2; ++half) {
      uint32_t v[32];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const float4 f = W2g[half * 8 + q];
        v[4 * q] = __float_as_uint(f.x); v[4 * q + 1] = __float_as_uint(f.y);
        v[4 * q + 2] = __float_as_uint(f.z); v[4 * q + 3] = __float_as_uint(f.w);
      }
      tmem_st32(tmem + lane_base + TM_S2 + wg * 64 + half * 32, v);
    }
    tmem_wait_st();
    done(E_LDT);
  };
  auto copy_state = [&](uint32_t col, uint8_t* dst) {      // this thread's row as bf16
#pragma unroll 1
    for (int half = 0; half < 2; ++half) {
      uint32_t v[32];
      tmem_ld32(tmem + lane_base + col + wg * 64 + half * 32, v);
      tmem_wait_ld();
      st_cols32(dst, hrow8, half, v);
    }
  };
  auto rec_chain = [&](int g) -> bool {
    const int gsz = size_of(g);
    float b1v = p.b1c[(long{sid} * nck + nck - 1 - g) * 256 + hrow8];
    if (g == 0) load_checkpoint(0);
    __syncwarp();
    copy_state(TM_S1, rW1);
    done(E_LD1);
    for (int j = 0; j < gsz; ++j, ++nrec) {
      const int s = j & 1;
      uint8_t* sK = smem + R_K + s * TILE;
      uint8_t* sV = smem + R_V;
      const __nv_bfloat16* eta = reinterpret_cast<const __nv_bfloat16*>(smem + R_ETA) + s * 64;
      wait(RK + s);
      if (nrec > 0) wait(F_X);
      wait_mma(RA + wg);
      // ---- EPI1: G' = gelu' stays in registers, the thread that needs it in EPI3 is this one
      // (rolled, like every pass over the columns: the values kept for later move down a register half per turn)
      uint32_t gp[32];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
#pragma unroll
        for (int k = 0; k < 16; ++k) gp[k] = gp[16 + k];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          uint32_t v[16];
          tmem_ld16(tmem + lane_base + TM_A + wg * 64 + h * 32 + q * 16, v);
          tmem_wait_ld();
          uint32_t z[8], x2[8];
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            const f32x2 x = add2(pk(v[2 * k], v[2 * k + 1]), pk1(b1v));
            f32x2 y, yp;
            gelu_pair2(x, y, yp);
            z[k] = f32x2_to_f16x2(x);          // f16: the sweep evaluates gelu' and gelu'' of it in f16
            x2[k] = f32x2_to_bf16x2(y);
            gp[16 + q * 8 + k] = f32x2_to_bf16x2(yp);
          }
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            const uint32_t off = sw128_off(hrow8, h * 4 + q * 2 + c);
            *reinterpret_cast<uint4*>(rX2 + off) = make_uint4(x2[4 * c], x2[4 * c + 1], x2[4 * c + 2], x2[4 * c + 3]);
            *reinterpret_cast<uint4*>(rZG + off) = make_uint4(z[4 * c], z[4 * c + 1], z[4 * c + 2], z[4 * c + 3]);
          }
        }
      }
      done(E_1);

      // ---- LN: fused LayerNorm + L2 gradient
      wait(RV);
      wait_mma(RZ);
      {
        float* xch = reinterpret_cast<float*>(smem + R_XCHC);
        TokFrag x, gr;
        uint32_t kk[8], vv[8];
        frag_ld(tm8, tmem + TM_A, x);
        frag_ld_raw(tm8, sK, kk);         // requested before the all-reduces of the LayerNorm, used after them
        frag_ld_raw(tm8, sV, vv);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const f32x2 b = frag_col(tm8, rB2, q);
          x.a[q] = add2(x.a[q], b);
          x.b[q] = add2(x.b[q], b);
        }
        float rs0, rs1;
        frag_layernorm(tm8, x, TTT_LN_EPS, xch, kBarPairC, rs0, rs1);
        f32x2 a0 = 0ull, a1 = 0ull, c0 = 0ull, c1 = 0ull;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const f32x2 gam = frag_col(tm8, sGamma, q), bet = frag_col(tm8, sBeta, q), neg = pk1(-1.f);
          const f32x2 t0 = fma2(bf16x2_to_f32x2(vv[2 * q]), neg, bf16x2_to_f32x2(kk[2 * q]));          // K - V
          const f32x2 t1 = fma2(bf16x2_to_f32x2(vv[2 * q + 1]), neg, bf16x2_to_f32x2(kk[2 * q + 1]));
          gr.a[q] = mul2(fma2(gam, x.a[q], add2(t0, bet)), gam);
          gr.b[q] = mul2(fma2(gam, x.b[q], add2(t1, bet)), gam);
          a0 = add2(a0, gr.a[q]); a1 = fma2(gr.a[q], x.a[q], a1);
          c0 = add2(c0, gr.b[q]); c1 = fma2(gr.b[q], x.b[q], c1);
        }
        // x_hat_fused leaves through the V tile: every thread overwrites exactly the elements it has read
        frag_st_tile(tm8, sV, x);
        float a[2] = {hsum(a0), hsum(a1)}, b[2] = {hsum(c0), hsum(c1)};
        frag_allreduce2<1>(tm8, a, b, xch, kBarPairC);
        const f32x2 sc0 = pk1(rs0 * (1.f / 64.f)), sc1 = pk1(rs1 * (1.f / 64.f));
        const f32x2 ne0 = pk1(-__bfloat162float(eta[tm8.r0])), ne1 = pk1(-__bfloat162float(eta[tm8.r1]));
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          // dl/dZ2, rounded to bf16 once: the update below uses -eta times the rounded value.  The forward rounds the
          // product instead, and adds up b2 from the rounded products (the recompute with four CTAs per stream does so
          // too, this one takes the fp32 ones): the state rebuilt inside a group differs from the
          // forward's by about that rounding, 2e-3 of b2's change since the checkpoint.
          const uint32_t w0 = f32x2_to_bf16x2(mul2(fma2(x.a[q], pk1(-a[1]), fma2(gr.a[q], pk1(64.f), pk1(-a[0]))), sc0));
          const uint32_t w1 = f32x2_to_bf16x2(mul2(fma2(x.b[q], pk1(-b[1]), fma2(gr.b[q], pk1(64.f), pk1(-b[0]))), sc1));
          *reinterpret_cast<uint32_t*>(smem + R_GZ2 + tm8.off(tm8.r0, q)) = w0;
          *reinterpret_cast<uint32_t*>(smem + R_GZ2 + tm8.off(tm8.r1, q)) = w1;
          gr.a[q] = mul2(bf16x2_to_f32x2(w0), ne0);
          gr.b[q] = mul2(bf16x2_to_f32x2(w1), ne1);
          x.a[q] = add2(gr.a[q], gr.b[q]);
        }
        frag_st_tile(tm8, smem + R_U2, gr);
        if (tm8.colhalf == 0 && tm8.l3 == 0) {
          float* sig = reinterpret_cast<float*>(smem + R_SIG);      // 1/std, and sum(grad_x_hat_fused x_hat_fused)
          sig[tm8.r0] = rs0;
          sig[tm8.r1] = rs1;
          sig[64 + tm8.r0] = a[1];
          sig[64 + tm8.r1] = b[1];
        }
        done(E_2);
        // under the product: column sums of U2, and -eta K over K, MMA4's operand (dl/dZ1 then is its other as it stands)
        reinterpret_cast<float*>(smem + R_CSC)[tm8.quad * 64 + frag_colsum_col(tm8, lane)] = frag_colsum(x.a, lane);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          gr.a[q] = mul2(bf16x2_to_f32x2(kk[2 * q]), ne0);
          gr.b[q] = mul2(bf16x2_to_f32x2(kk[2 * q + 1]), ne1);
        }
        frag_st_tile(tm8, sK, gr);
        if (gtid < 32) reinterpret_cast<uint32_t*>(smem + OFF_NETA)[gtid] = reinterpret_cast<const uint32_t*>(eta)[gtid] ^ 0x80008000u;
      }

      // ---- EPI3: dl/dZ1 over Z1 (its image) and over R in tensor memory (the A operand of its MMAs)
      wait(F_ZG);
      wait_mma(RA + wg);
      {
        const uint32_t acc = tmem + lane_base + TM_A + wg * 64;
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          uint32_t v[32], w[16];
          tmem_ld32(acc + half * 32, v);
          tmem_wait_ld();
#pragma unroll
          for (int k = 0; k < 16; ++k)
            w[k] = f32x2_to_bf16x2(mul2(bf16x2_to_f32x2(gp[half * 16 + k]), pk(v[2 * k], v[2 * k + 1])));
#pragma unroll
          for (int c = 0; c < 4; ++c)
            *reinterpret_cast<uint4*>(rZG + sw128_off(hrow8, half * 4 + c)) = make_uint4(w[4 * c], w[4 * c + 1], w[4 * c + 2], w[4 * c + 3]);
          tmem_st16(acc + half * 16, w);
        }
        tmem_wait_st();
      }
      done(E_3);

      // ---- EPI4: bf16 copy of the new W1, and b1, once the output group has used the last ones
      if (j > 0) wait(RG7);
      wait_mma(RA + wg);
      {
        uint32_t v[8];
        tmem_ld8(tmem + lane_base + TM_A + wg * 64 + 32, v);
        tmem_wait_ld();
        b1v += __uint_as_float(v[0]);
      }
      copy_state(TM_S1, rW1);
      rB1[hrow8] = b1v;
      done(E_W1);
      if (named_bar_or(kBarC, kGroup, *abort_flag != 0)) return true;
    }
    if (g + 1 < nck) load_checkpoint(g + 1);
    wait(RG7);
    return false;
  };

  auto rec_out = [&](int g) -> bool {
    const int gsz = size_of(g);
    wait_mma(E_LDT);
    copy_state(TM_S2, rW2);
    if (gtid < 64) rB2[gtid] = p.b2c[(long{sid} * nck + nck - 1 - g) * 64 + gtid];
    done(E_LD2);
    auto finish_dq = [&]() {      // dQ = go + gZ1b W1^T, over the dL/dOut tile
      wait_mma(RG7);
      TokFrag x;
      uint32_t gw[8];
      frag_ld(tm8, tmem + TM_B, x);
      frag_ld_raw(tm8, smem + R_GO, gw);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        x.a[q] = add2(x.a[q], bf16x2_to_f32x2(gw[2 * q]));
        x.b[q] = add2(x.b[q], bf16x2_to_f32x2(gw[2 * q + 1]));
      }
      frag_st_tile(tm8, smem + R_GO, x);
      done(E_ODQ);
    };
    for (int j = 0; j < gsz; ++j, ++nrec) {
      // ---- bf16 copy of the new W2; b2
      if (j == 0) wait(F_XB);                   // the checkpoint's image has left
      wait_mma(RW2UPD);
      copy_state(TM_S2, rW2);
      if (gtid < 64) rB2[gtid] += quad_sum(reinterpret_cast<const float*>(smem + R_CSC), gtid);
      done(E_W2);
      if (j > 0) finish_dq();
      // ---- EPI5
      if (nrec > 0) wait(F_XB2);
      wait_mma(RB);
      uint32_t gp[32];
      {
        const f32x2 bb = pk1(rB1[hrow8]);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
#pragma unroll
          for (int k = 0; k < 16; ++k) gp[k] = gp[16 + k];
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            uint32_t v[16], x2[8];
            tmem_ld16(tmem + lane_base + TM_B + wg * 64 + h * 32 + q * 16, v);
            tmem_wait_ld();
#pragma unroll
            for (int k = 0; k < 8; ++k) {
              f32x2 y, yp;
              gelu_pair2(add2(pk(v[2 * k], v[2 * k + 1]), bb), y, yp);
              x2[k] = f32x2_to_bf16x2(y);
              gp[16 + q * 8 + k] = f32x2_to_bf16x2(yp);
            }
#pragma unroll
            for (int c = 0; c < 2; ++c)
              *reinterpret_cast<uint4*>(rXB + sw128_off(hrow8, h * 4 + q * 2 + c)) =
                  make_uint4(x2[4 * c], x2[4 * c + 1], x2[4 * c + 2], x2[4 * c + 3]);
          }
        }
      }
      done(E_O5);
      // ---- S4: output LayerNorm and its backward
      wait(RGO);
      wait_mma(RBZ);
      {
        float* xch = reinterpret_cast<float*>(smem + R_XCHO);
        TokFrag x, gr;
        uint32_t gw[8];
        frag_ld(tm8, tmem + TM_B, x);
        frag_ld_raw(tm8, smem + R_GO, gw);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const f32x2 b = frag_col(tm8, rB2, q);
          x.a[q] = add2(x.a[q], b);
          x.b[q] = add2(x.b[q], b);
        }
        float rs0, rs1;
        frag_layernorm(tm8, x, TTT_LN_EPS, xch, kBarPairO, rs0, rs1);
        f32x2 a0 = 0ull, a1 = 0ull, c0 = 0ull, c1 = 0ull, sb[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const f32x2 gam = frag_col(tm8, sGamma, q);
          gr.a[q] = mul2(bf16x2_to_f32x2(gw[2 * q]), gam);
          gr.b[q] = mul2(bf16x2_to_f32x2(gw[2 * q + 1]), gam);
          a0 = add2(a0, gr.a[q]); a1 = fma2(gr.a[q], x.a[q], a1);
          c0 = add2(c0, gr.b[q]); c1 = fma2(gr.b[q], x.b[q], c1);
        }
        float a[2] = {hsum(a0), hsum(a1)}, b[2] = {hsum(c0), hsum(c1)};
        frag_allreduce2<1>(tm8, a, b, xch, kBarPairO);
        const f32x2 q0 = pk1(rs0 * (1.f / 64.f)), q1 = pk1(rs1 * (1.f / 64.f));
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          gr.a[q] = mul2(fma2(x.a[q], pk1(-a[1]), fma2(gr.a[q], pk1(64.f), pk1(-a[0]))), q0);
          gr.b[q] = mul2(fma2(x.b[q], pk1(-b[1]), fma2(gr.b[q], pk1(64.f), pk1(-b[0]))), q1);
        }
        frag_st_tile(tm8, smem + R_Q, gr);      // Q was consumed by MMA5
        done(E_OS4);
        // (column sums under the product)
#pragma unroll
        for (int q = 0; q < 4; ++q) sb[q] = add2(gr.a[q], gr.b[q]);
        reinterpret_cast<float*>(smem + R_CSO)[tm8.quad * 64 + frag_colsum_col(tm8, lane)] = frag_colsum(sb, lane);
#pragma unroll
        for (int q = 0; q < 4; ++q) sb[q] = add2(bf16x2_to_f32x2(gw[2 * q]), bf16x2_to_f32x2(gw[2 * q + 1]));
        dbet += frag_colsum(sb, lane);
#pragma unroll
        for (int q = 0; q < 4; ++q)
          sb[q] = fma2(bf16x2_to_f32x2(gw[2 * q]), x.a[q], mul2(bf16x2_to_f32x2(gw[2 * q + 1]), x.b[q]));
        dgam += frag_colsum(sb, lane);
      }
      named_bar_sync(kBarO, kGroup);            // the column sums of all quadrants are in place
      // ---- E1: dL/dZ1_bar over X2b
      wait(F_XB);
      wait_mma(RG1);
      {
        f32x2 bsum = 0ull;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t v[32];
          tmem_ld32(tmem + lane_base + TM_B + wg * 64 + h * 32, v);
          tmem_wait_ld();
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            uint32_t w[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const f32x2 t = mul2(bf16x2_to_f32x2(gp[c * 4 + k]), pk(v[c * 8 + 2 * k], v[c * 8 + 2 * k + 1]));
              bsum = add2(bsum, t);
              w[k] = f32x2_to_bf16x2(t);
            }
            *reinterpret_cast<uint4*>(rXB + sw128_off(hrow8, h * 4 + c)) = make_uint4(w[0], w[1], w[2], w[3]);
          }
#pragma unroll
          for (int k = 0; k < 16; ++k) gp[k] = gp[16 + k];
        }
        rVec[hrow8] = hsum(bsum);
        if (gtid < 64) rVec[256 + gtid] = quad_sum(reinterpret_cast<const float*>(smem + R_CSO), gtid);
      }
      done(E_OE1);
      if (named_bar_or(kBarO, kGroup, *abort_flag != 0)) return true;
    }
    finish_dq();
    return false;
  };

  // ---- MMA issue
  // (rolled by four: unrolled, the sweep's 136 MMAs a step would be 36 KB of code)
  auto hidden = [&](auto bmn, auto acc, uint32_t d, const uint8_t* a, const uint8_t* b) {
    const uint32_t as = smem_u32(a), bs = smem_u32(b);
#pragma unroll 1
    for (int blk = 0; blk < 2; ++blk) mma_hidden_lead<decltype(bmn)::value, decltype(acc)::value>(d, as, bs, blk, lead);
  };
  auto token = [&](uint32_t d, const uint8_t* x, const uint8_t* w) {
    constexpr uint32_t idesc = umma_idesc_bf16(64, 64, true, true, false);
    uint32_t a = desc_lo(smem_u32(x), BIG), b = desc_lo(smem_u32(w), BIG);
#pragma unroll 1
    for (uint32_t k = 0; k < 16; k += 4) {
#pragma unroll
      for (uint32_t i = 0; i < 4; ++i)
        mma_lead_rt(d, a + i * (2048u >> 4), b + i * (2048u >> 4), idesc, k | i, lead);
      a += 4 * (2048u >> 4);
      b += 4 * (2048u >> 4);
    }
  };
  using T = std::true_type;
  using F = std::false_type;
  auto seen = [&](int b) -> bool {      // by a whole helper warp, which goes on or leaves as one
    const bool ok = __all_sync(0xffffffffu, wait(b));
    tc_fence_after_sync();
    return ok;
  };

  auto rec_chain_issue = [&](int g) {
    const int gsz = size_of(g);
    for (int j = 0; j < gsz; ++j) {
      const uint8_t* sK = smem + R_K + (j & 1) * TILE;
      if (!(j == 0 ? seen(E_LD1) : seen(E_W1)) || !seen(RK + (j & 1))) return;
#pragma unroll 1
      for (int blk = 0; blk < 2; ++blk) {
        mma_hidden_lead<false, false>(tmem + TM_A, smem_u32(rW1), smem_u32(sK), blk, lead);
        commit(RA + blk);
      }
      if (!seen(E_1) || !(j == 0 ? seen(E_LD2) : seen(E_W2))) return;
      token(tmem + TM_A, rX2, rW2);
      commit(RZ);
      if (!seen(E_2)) return;
#pragma unroll 1
      for (int blk = 0; blk < 2; ++blk) {
        mma_hidden_lead<false, false>(tmem + TM_A, smem_u32(rW2), smem_u32(smem + R_GZ2), blk, lead);
        commit(RA + blk);
      }
      if (!seen(E_3)) return;
#pragma unroll 1
      for (int blk = 0; blk < 2; ++blk) {
        // W1^T += gZ1^T (-eta K); b1's sums gZ1^T (-eta) to 16 columns behind gZ1, of which the first is used (the others
        // multiply what lies behind -eta)
        mma_hidden_ta<true, true>(tmem + TM_S1 + blk * 64, tmem + TM_A + blk * 64, smem_u32(sK), lead);
        mma_rowsum_ta(tmem + TM_A + blk * 64 + 32, tmem + TM_A + blk * 64, smem_u32(smem + OFF_NETA), lead);
        commit(RA + blk);
      }
      hidden(T{}, T{}, tmem + TM_S2, rX2, smem + R_U2);
      commit(RW2UPD);
    }
    if (!seen(E_W1)) return;
    seen(E_W2);
  };
  auto rec_out_issue = [&](int g) {
    const int gsz = size_of(g);
    for (int j = 0; j < gsz; ++j) {
      if (j > 0 && !seen(E_ODQ)) return;               // the accumulator has been read
      if (!seen(E_W1) || !seen(RQ)) return;
      hidden(F{}, F{}, tmem + TM_B, rW1, smem + R_Q);
      commit(RB);
      if (!seen(E_O5) || !seen(E_W2)) return;
      token(tmem + TM_B, rXB, rW2);
      commit(RBZ);
      if (!seen(E_OS4)) return;
      hidden(F{}, F{}, tmem + TM_B, rW2, smem + R_Q);
      commit(RG1);
      if (!seen(E_OE1)) return;
      token(tmem + TM_B, rXB, rW1);
      commit(RG7);
    }
    seen(E_ODQ);
  };

  // ---- copies of the chain and of the output group, a warp each.  Events of a mini-batch: the group's epilogues in order.
  auto dropped = [&](int i) { return i == p.drop_load && sid == 0; };
  auto rec_chain_copy = [&](int g) {
    const Lane c = lane_of(kChainCopy, kRecCopies);
    const CopyOp& op = c.op;
    const int i0 = first_of(g), gsz = size_of(g);
    const bool mine = lane < kRecCopies, is_k = lane == kLaneK || lane == kLaneK + 1, is_v = lane == kLaneV;
    auto first = [&](int gg) {
      const int i1 = first_of(gg);
#pragma unroll 1
      for (int k = 0; k < 2; ++k)
        copy(c, (is_k && k < size_of(gg)) || (is_v && k == 0), i1 + k, 0, op.off, k, dropped(i1 + k));
      __syncwarp();
    };
    if (g == 0) first(g);
    for (int j = -1; j < gsz; ++j) {
      // this lane's copies of the mini-batch, put together before their events are waited for
      uint8_t* const mem = place(c, slot_of(g, j + op.next));
      const bool store = mine && op.kind == K_STORE && j + op.next < gsz;
      const int ahead = is_v ? 1 : 2, i = i0 + j + ahead;      // the load's mini-batch
      const bool load = (is_v || is_k) && j >= 0 && j + ahead < gsz && !dropped(i);
      const uint32_t off = op.off + (is_k && (j & 1) ? op.par : 0u);
      const int b = op.bar + (is_k ? j & 1 : 0);
      const uint8_t* const src = c.mem + i * 128L;             // eta
#pragma unroll 1
      for (int ev = j < 0 ? Y_W : Y_1; ev <= Y_W; ++ev) {      // j = -1: the checkpoint's W1
        if (!seen_all(j < 0 ? E_LD1 : ev == Y_1 ? E_1 : ev == Y_2 ? E_2 : ev == Y_3 ? E_3 : E_W1)) return;
        if (ev == Y_2 || ev == Y_3) {
          tma_wait_group_read<0>();
          __syncwarp();
          if (ev == Y_2 && lane == 0) arrive(F_ZG);
        }
        // V's tile is free after E_3 (x_hat_fused has left), K's stage after EPI4
        if (load && ev == (is_v ? Y_3 : Y_W)) {
          if (op.arm) arm(b, op.arm);
          if (op.kind == K_TMA) tma_load_2d(smem + off, c.map, &bars[b], 0, row_of(i));
          else bulk_load_1d(smem + off, src, op.bytes, &bars[b]);
        }
        if (ev == Y_W && j + 1 < gsz && !wait_slot(g, j + 1)) return;
        if (store && op.event == ev) {
          bulk_store_1d(mem, smem + op.off, op.bytes);
          tma_commit_group();
        }
        __syncwarp();
        if (ev == Y_3) {
          tma_wait_group_read<0>();
          __syncwarp();
          if (lane == 0) arrive(F_X);
        }
      }
    }
    if (g + 1 < nck) first(g + 1);
    group_written(g);
  };
  auto rec_out_copy = [&](int g) {
    const Lane c = lane_of(kOutCopy, kRecCopies);
    const CopyOp& op = c.op;
    const int i0 = first_of(g), gsz = size_of(g);
    const bool mine = lane < kRecCopies;
    if (g == 0) copy(c, lane == kLaneQ || lane == kLaneGo, i0, 0, op.off, 0, dropped(i0));
    for (int j = -1; j < gsz; ++j) {
      uint8_t* const mem = place(c, slot_of(g, j + op.next));
      const bool store = mine && op.kind == K_STORE && j + op.next < gsz;
      const int when = op.event == Y_W ? Y_LD : op.event;
#pragma unroll 1
      for (int ev = Y_LD; ev <= Y_3; ++ev) {      // Y_LD: the W2 copy (j = -1: the checkpoint's W2)
        if (!seen_all(j < 0 ? E_LD2 : ev == Y_LD ? E_W2 : ev == Y_1 ? E_O5 : ev == Y_2 ? E_OS4 : E_OE1)) return;
        if (ev == Y_LD && j + 1 < gsz && !wait_slot(g, j + 1)) return;
        if (ev == Y_2) {
          tma_wait_group_read<0>();
          __syncwarp();
          if (lane == 0) arrive(F_XB);
        }
        if (store && when == ev) {
          bulk_store_1d(mem, smem + op.off, op.bytes);
          tma_commit_group();
        }
        __syncwarp();
        const bool dq = ev == Y_LD && j > 0;
        if (dq) {
          if (!seen_all(E_ODQ)) return;
          if (lane == 0) {
            tma_store_2d(&tmDQ, smem + R_GO, 0, row_of(i0 + j - 1));
            tma_commit_group();
          }
        }
        if (dq || j < 0 || ev == Y_3) {
          tma_wait_group_read<0>();
          __syncwarp();
          if (!dq && lane == 0) arrive(j < 0 ? F_XB : F_XB2);
        }
        // dL/dOut's tile is free when dQ has left it, Q's when gZ2b has
        const int i = i0 + j + (dq ? 0 : 1);
        if (((dq && lane == kLaneGo) || (ev == Y_3 && lane == kLaneQ && j + 1 < gsz)) && !dropped(i)) {
          arm(op.bar, op.arm);
          tma_load_2d(smem + op.off, c.map, &bars[op.bar], 0, row_of(i));
        }
        __syncwarp();
        if (j < 0) break;
      }
    }
    if (!seen_all(E_ODQ)) return;
    if (lane == 0) {
      tma_store_2d(&tmDQ, smem + R_GO, 0, row_of(i0 + gsz - 1));
      tma_commit_group();
    }
    tma_wait_group_read<0>();
    __syncwarp();
    if (g + 1 < nck) copy(c, lane == kLaneQ || lane == kLaneGo, first_of(g + 1), 0, op.off, 0, dropped(first_of(g + 1)));
    group_written(g);
  };

  // =====================================================================================================
  //                                             reverse sweep
  // =====================================================================================================
  const int cq = warp >> 2;                                  // 0..3: 128-row block and column half of the hidden-major tiles
  const int blk = cq & 1, ch = cq >> 1;
  const int hrow = blk * 128 + quad * 32 + lane;
  const TokMap16 tm(warp, lane);
  int nsw = 0;                                               // steps swept so far
  float dgam_s = 0.f, dbet_s = 0.f;
  float* sGb1 = reinterpret_cast<float*>(smem + S_GB1);
  float* sGb2 = reinterpret_cast<float*>(smem + S_GB2);
  float* sVec = reinterpret_cast<float*>(smem + S_VEC);
  float* sCS = reinterpret_cast<float*>(smem + S_CS);
  // hidden-major buffers: buffer 0 holds W2 then W1; the other four, as offsets, by what they hold first in a step:
  //   gz  gZ1, X2b(i - 1), gZ1in                 -> the next step's G_W2 snapshot
  //   z   Z1, X2                                 -> G_W1 snapshot
  //   s1  G_W1 snapshot, P, gZ1b(i - 1)          -> gZ1
  //   s2  G_W2 snapshot                          -> Z1
  uint32_t o_gz = BIG, o_z = 2 * BIG, o_s1 = 3 * BIG, o_s2 = 4 * BIG;
  auto turn = [&]() {
    const uint32_t g = o_gz, z = o_z, s1 = o_s1, s2 = o_s2;
    o_z = s2; o_gz = s1; o_s1 = z; o_s2 = g;
  };

  auto sweep_epi = [&](int g) {
    const int i0 = first_of(g), gsz = size_of(g);
    const uint32_t hl = lane_base + blk * 64 + ch * 32;      // this thread's lanes and columns of a 256-row matrix
    if (g == 0) {   // dL/dW state: global (fp32) -> tensor memory
      const float* G1 = p.gW1_last + long{sid} * (64 * 256) + hrow;
      const float4* G2 = reinterpret_cast<const float4*>(p.gW2_last + long{sid} * (256 * 64) + hrow * 64 + ch * 32);
      uint32_t v[32];
#pragma unroll
      for (int q = 0; q < 32; ++q) v[q] = __float_as_uint(G1[(ch * 32 + q) * 256]);
      tmem_st32(tmem + TM_S1 + hl, v);
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const float4 f = G2[q];
        v[4 * q] = __float_as_uint(f.x); v[4 * q + 1] = __float_as_uint(f.y);
        v[4 * q + 2] = __float_as_uint(f.z); v[4 * q + 3] = __float_as_uint(f.w);
      }
      tmem_st32(tmem + TM_S2 + hl, v);
      if (ch == 0) sGb1[hrow] = p.gb1_last[long{sid} * 256 + hrow];
      if (tid < 64) sGb2[tid] = p.gb2_last[long{sid} * 64 + tid];
      tmem_wait_st();
      done(E_5);
    }
    Frag16 kp;                // partial dK of the last step
    auto finish_dk = [&]() {  // after C7
      uint32_t u[8];
      tmem_ld_16x256b_x2(tmem + TM_B + 64 + tm.taddr, u);
      tmem_wait_ld();
      Frag16 x = f16_pack(u);
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        x.a[q] = add2(x.a[q], kp.a[q]);
        x.b[q] = add2(x.b[q], kp.b[q]);
      }
      f16_st_tile(tm, smem + S_K + ((nsw - 1) & 1) * TILE, x);
    };
    auto snapshot = [&](uint32_t src, uint8_t* dst) {      // this thread's 32 columns as bf16
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        uint32_t v[16];
        tmem_ld16(src + q * 16, v);
        tmem_wait_ld();
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          uint4 w;
          w.x = pack_bf16(__uint_as_float(v[c * 8 + 0]), __uint_as_float(v[c * 8 + 1]));
          w.y = pack_bf16(__uint_as_float(v[c * 8 + 2]), __uint_as_float(v[c * 8 + 3]));
          w.z = pack_bf16(__uint_as_float(v[c * 8 + 4]), __uint_as_float(v[c * 8 + 5]));
          w.w = pack_bf16(__uint_as_float(v[c * 8 + 6]), __uint_as_float(v[c * 8 + 7]));
          *reinterpret_cast<uint4*>(dst + sw128_off(hrow, ch * 4 + q * 2 + c)) = w;
        }
      }
    };
    for (int j = gsz - 1; j >= 0; --j) {
      const bool first = j == gsz - 1;
      const int par = nsw & 1;
      const __nv_bfloat16* eta = reinterpret_cast<const __nv_bfloat16*>(smem + S_ETA) + par * 64;
      // ---- gelu'(Z1) and gelu''(Z1) in f16: half of them under the last products of the step before, half under G4 and G8
      uint32_t sS[16], sG[16];
      uint4 zr[4];
      wait(SZ1);
#pragma unroll
      for (int q = 0; q < 4; ++q) zr[q] = ld_chunk_raw(smem + o_z, hrow, ch * 4 + q);
      __syncwarp();
      if (lane == 0) arrive(E_D);
      auto derivatives = [&](int q0) {
#pragma unroll
        for (int q = q0; q < q0 + 2; ++q) {
          const uint32_t zw[4] = {zr[q].x, zr[q].y, zr[q].z, zr[q].w};
#pragma unroll
          for (int k = 0; k < 4; ++k) gelu_grad_h2(zw[k], sG[q * 4 + k], sS[q * 4 + k]);
        }
      };
      derivatives(0);
      // ---- E2: bf16 snapshots of the gradient state
      if (first) wait(SX2B);
      wait_mma(C6);
      {
        if (ch == 0) sGb1[hrow] += sVec[hrow];
        if (tid < 64) sGb2[tid] += (first ? 0.f : quad_sum(sCS, tid)) + sVec[256 + tid];
        snapshot(tmem + TM_S1 + hl, smem + o_s1);
      }
      done(E_S1);
      wait_mma(C7);
      snapshot(tmem + TM_S2 + hl, smem + o_s2);
      if (!first) finish_dk();
      done(E_S2);
      derivatives(2);

      // ---- E3: A1, P = A1 gelu'(Z1) over the G_W1 snapshot, which G4 and G8 have read; S = A1 gelu''(Z1) in the place of
      // gelu''(Z1)
      wait(SK);
      wait_mma(C2);
      {
        const f32x2 gb = pk1(sGb1[hrow]);
        uint32_t v[2][16];
        tmem_ld16(tmem + TM_A + hl, v[0]);
        tmem_ld16(tmem + TM_A + hl + 16, v[1]);
        tmem_wait_ld();
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          uint32_t pw[4];
          const uint4 ew = *reinterpret_cast<const uint4*>(eta + ch * 32 + q * 8);     // one broadcast load
          const uint32_t et[4] = {ew.x, ew.y, ew.z, ew.w};
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const uint32_t* w = v[q >> 1] + (q & 1) * 8 + 2 * k;
            const f32x2 a1 = mul2(bf16x2_to_f32x2(et[k] ^ 0x80008000u), add2(pk(w[0], w[1]), gb));
            pw[k] = f32x2_to_bf16x2(mul2(a1, f16x2_to_f32x2(sG[q * 4 + k])));
            sS[q * 4 + k] = f32x2_to_bf16x2(mul2(a1, f16x2_to_f32x2(sS[q * 4 + k])));
          }
          *reinterpret_cast<uint4*>(smem + o_s1 + sw128_off(hrow, ch * 4 + q)) = make_uint4(pw[0], pw[1], pw[2], pw[3]);
        }
      }
      done(E_P);
      wait(SGZ2);
      {   // U2 = -eta gZ2
        uint32_t w[4];
        f16_ld_raw(tm, smem + S_GZ2, w);
        const f32x2 n0 = pk1(-__bfloat162float(eta[tm.r0])), n1 = pk1(-__bfloat162float(eta[tm.r1]));
        Frag16 u;
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          u.a[q] = mul2(bf16x2_to_f32x2(w[2 * q]), n0);
          u.b[q] = mul2(bf16x2_to_f32x2(w[2 * q + 1]), n1);
        }
        f16_st_tile(tm, smem + S_Q, u);
      }

      // ---- E4: second order through the fused LayerNorm + L2 gradient
      wait(SXF);
      wait(SV);
      wait_mma(C4);
      float de0, de1;                      // d_eta's row terms
      {
        uint32_t gzw[4], xw[4], kw[4], vw[4];
        f16_ld_raw(tm, smem + S_GZ2, gzw);
        f16_ld_raw(tm, smem + S_XF, xw);
        f16_ld_raw(tm, smem + S_K + par * TILE, kw);
        const float* sig = reinterpret_cast<const float*>(smem + S_SIG);
        const float eta0 = __bfloat162float(eta[tm.r0]), eta1 = __bfloat162float(eta[tm.r1]);
        const float rs0 = sig[tm.r0], rs1 = sig[tm.r1];      // 1 / std
        Frag16 A2, go;
        f32x2 cl[2];                       // dV's addends to d_beta
        float ra[2], rb[2];                // sum A2, sum A2 x_hat
        {
          uint32_t u0[8], u1[8];
          tmem_ld_16x256b_x2(tmem + TM_B + 64 + tm.taddr, u0);
          tmem_ld_16x256b_x2(tmem + TM_A + tm.taddr, u1);
          tmem_wait_ld();
          const Frag16 acc1 = f16_pack(u0);                         // X2 G_W2
          A2 = f16_pack(u1);                                        // P W2
          f32x2 d0 = 0ull, d1 = 0ull, s0 = 0ull, s1 = 0ull, x0s = 0ull, x1s = 0ull;
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            const f32x2 gb2 = f16_col(tm, sGb2, q);
            const f32x2 w0 = add2(acc1.a[q], gb2), w1 = add2(acc1.b[q], gb2);
            A2.a[q] = fma2(w0, pk1(-eta0), A2.a[q]);
            A2.b[q] = fma2(w1, pk1(-eta1), A2.b[q]);
            s0 = add2(s0, A2.a[q]);
            s1 = add2(s1, A2.b[q]);
            x0s = fma2(A2.a[q], bf16x2_to_f32x2(xw[2 * q]), x0s);
            x1s = fma2(A2.b[q], bf16x2_to_f32x2(xw[2 * q + 1]), x1s);
            d0 = fma2(bf16x2_to_f32x2(gzw[2 * q]), w0, d0);
            d1 = fma2(bf16x2_to_f32x2(gzw[2 * q + 1]), w1, d1);
          }
          tmem_ld_16x256b_x2(tmem + TM_B + tm.taddr, u0);
          tmem_wait_ld();
          done(E_T);
          const Frag16 t1 = f16_pack(u0);                           // gZ1 G_W1
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            d0 = fma2(t1.a[q], bf16x2_to_f32x2(kw[2 * q]), d0);
            d1 = fma2(t1.b[q], bf16x2_to_f32x2(kw[2 * q + 1]), d1);
            kp.a[q] = mul2(t1.a[q], pk1(-eta0));
            kp.b[q] = mul2(t1.b[q], pk1(-eta1));
          }
          de0 = hsum(d0); de1 = hsum(d1);
          ra[0] = hsum(s0); ra[1] = hsum(x0s);
          rb[0] = hsum(s1); rb[1] = hsum(x1s);
        }
        float2* x1 = reinterpret_cast<float2*>(smem + S_X1);
        float2* x2 = reinterpret_cast<float2*>(smem + S_X2);
        f16_row_sums(tm, ra, rb, x1, kBarQuad);
        // (tiles are read again after an exchange rather than held over it: 32 registers are E5's already)
        f16_ld_raw(tm, smem + S_XF, xw);
        f16_ld_raw(tm, smem + S_GZ2, gzw);
        f16_ld_raw(tm, smem + S_K + par * TILE, kw);
        f16_ld_raw(tm, smem + S_V, vw);
#pragma unroll
        for (int q = 0; q < 2; ++q) {   // grad_output_fused = gamma x_hat_fused + beta - (V - K)
          const f32x2 gam = f16_col(tm, sGamma, q), bet = f16_col(tm, sBeta, q), neg = pk1(-1.f);
          go.a[q] = add2(fma2(bf16x2_to_f32x2(vw[2 * q]), neg, bf16x2_to_f32x2(kw[2 * q])),
                         fma2(gam, bf16x2_to_f32x2(xw[2 * q]), bet));
          go.b[q] = add2(fma2(bf16x2_to_f32x2(vw[2 * q + 1]), neg, bf16x2_to_f32x2(kw[2 * q + 1])),
                         fma2(gam, bf16x2_to_f32x2(xw[2 * q + 1]), bet));
        }
        f32x2 cs[2];
        float sa[2], sb[2];                // sums of g_std and of g_xhat of the two rows
        {
          const float s30 = sig[64 + tm.r0], s31 = sig[64 + tm.r1];      // sum(grad_x_hat_fused x_hat_fused)
          const f32x2 n64 = pk1(-1.f / 64.f);
          const f32x2 mA = mul2(pk1(ra[0]), n64), xA = mul2(pk1(ra[1]), n64), mB = mul2(pk1(rb[0]), n64), xB = mul2(pk1(rb[1]), n64);
          const f32x2 fA3 = pk1(-ra[1] * rs0 * (1.f / 64.f)), fA4 = pk1(-s30 * rs0 * (1.f / 64.f));
          const f32x2 fB3 = pk1(-rb[1] * rs1 * (1.f / 64.f)), fB4 = pk1(-s31 * rs1 * (1.f / 64.f));
          f32x2 sa0 = 0ull, sa1 = 0ull, sb0 = 0ull, sb1 = 0ull;
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            const f32x2 gm = f16_col(tm, sGamma, q);
            const f32x2 v0 = bf16x2_to_f32x2(xw[2 * q]), v1 = bf16x2_to_f32x2(xw[2 * q + 1]);
            const f32x2 bt0 = mul2(add2(A2.a[q], fma2(v0, xA, mA)), pk1(rs0));
            const f32x2 bt1 = mul2(add2(A2.b[q], fma2(v1, xB, mB)), pk1(rs1));
            const f32x2 gl0 = mul2(gm, bt0), gl1 = mul2(gm, bt1);
            cs[q] = add2(fma2(go.a[q], bt0, mul2(gl0, v0)), fma2(go.b[q], bt1, mul2(gl1, v1)));
            cl[q] = add2(gl0, gl1);
            kp.a[q] = add2(kp.a[q], gl0);
            kp.b[q] = add2(kp.b[q], gl1);
            // dV, over V
            *reinterpret_cast<uint32_t*>(smem + S_V + tm.off(tm.r0, q)) = f32x2_to_bf16x2(gl0) ^ 0x80008000u;
            *reinterpret_cast<uint32_t*>(smem + S_V + tm.off(tm.r1, q)) = f32x2_to_bf16x2(gl1) ^ 0x80008000u;
            const f32x2 gx0 = fma2(gl0, gm, fma2(mul2(go.a[q], gm), fA3, mul2(A2.a[q], fA4)));
            const f32x2 gx1 = fma2(gl1, gm, fma2(mul2(go.b[q], gm), fB3, mul2(A2.b[q], fB4)));
            sa0 = fma2(gx0, v0, fma2(A2.a[q], bf16x2_to_f32x2(gzw[2 * q]), sa0));
            sb0 = fma2(gx1, v1, fma2(A2.b[q], bf16x2_to_f32x2(gzw[2 * q + 1]), sb0));
            sa1 = add2(sa1, gx0);
            sb1 = add2(sb1, gx1);
            A2.a[q] = gx0;
            A2.b[q] = gx1;
          }
          sa[0] = -hsum(sa0) * rs0; sa[1] = hsum(sa1);
          sb[0] = -hsum(sb0) * rs1; sb[1] = hsum(sb1);
        }
        f16_row_sums(tm, sa, sb, x2, kBarQuad);
        {
          const f32x2 k0 = pk1(sa[0] * (1.f / 64.f)), l0 = pk1(-sa[1] * rs0 * (1.f / 64.f));
          const f32x2 k1 = pk1(sb[0] * (1.f / 64.f)), l1 = pk1(-sb[1] * rs1 * (1.f / 64.f));
#pragma unroll
          for (int q = 0; q < 2; ++q) {      // gZ2in, over x_hat_fused
            A2.a[q] = fma2(A2.a[q], pk1(rs0), fma2(bf16x2_to_f32x2(xw[2 * q]), k0, l0));
            A2.b[q] = fma2(A2.b[q], pk1(rs1), fma2(bf16x2_to_f32x2(xw[2 * q + 1]), k1, l1));
          }
          f16_st_tile(tm, smem + S_XF, A2);
        }
        done(E_Z);
        if (lane == 0) arrive(E_V);
        // ---- what nothing on the chain waits for: column sums, d_eta's rows
        sCS[quad * 64 + f16_colsum_col(tm, lane)] = f16_colsum(add2(A2.a[0], A2.b[0]), add2(A2.a[1], A2.b[1]), lane);
        dgam_s += f16_colsum(cs[0], cs[1], lane);
        dbet_s += f16_colsum(cl[0], cl[1], lane);
#pragma unroll
        for (int sft = 1; sft <= 2; sft <<= 1) {
          de0 += __shfl_xor_sync(0xffffffffu, de0, sft);
          de1 += __shfl_xor_sync(0xffffffffu, de1, sft);
        }
      }

      // ---- E5: gZ1in^T = gX2^T gelu'(Z1^T) + R^T S^T
      wait_mma(C5);
      // (over the first exchange: its last reader is behind E_Z, and E4 of the next step, which writes there again, behind E_X)
      if (tm.l3 == 0) {
        float* xe = reinterpret_cast<float*>(smem + S_X1);
        xe[cq * 64 + tm.r0] = de0;
        xe[cq * 64 + tm.r1] = de1;
      }
      {
        f32x2 bs = 0ull;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          uint32_t v[8], w[8], o[4];
          tmem_ld8(tmem + TM_B + hl + q * 8, v);
          tmem_ld8(tmem + TM_A + hl + q * 8, w);
          tmem_wait_ld();
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const f32x2 t = fma2(pk(v[2 * k], v[2 * k + 1]), f16x2_to_f32x2(sG[q * 4 + k]),
                                 mul2(pk(w[2 * k], w[2 * k + 1]), bf16x2_to_f32x2(sS[q * 4 + k])));
            bs = add2(bs, t);
            o[k] = f32x2_to_bf16x2(t);
          }
          *reinterpret_cast<uint4*>(smem + o_gz + sw128_off(hrow, ch * 4 + q)) = make_uint4(o[0], o[1], o[2], o[3]);
        }
        if (j > 0) wait(SX2B);      // the next step's row sums of gZ1b, which this adds to
        if (ch == 0) sGb1[hrow] += hsum(bs);
        else sVec[hrow] = hsum(bs) + (j > 0 ? sVec[hrow] : 0.f);
      }
      done(E_5);
      turn();
      ++nsw;
    }
    // ---- the group's last step: dK, bias gradients
    wait(C6);
    wait_mma(C7);
    finish_dk();
    if (ch == 0) sGb1[hrow] += sVec[hrow];
    if (tid < 64) sGb2[tid] += quad_sum(sCS, tid);
    done(E_S2);
    if (g == nck - 1) {   // the gradient state: tensor memory -> grad_L_W*_init
      float* G1 = p.gW1 + long{sid} * (64 * 256) + hrow;
      uint32_t v[32];
      tmem_ld32(tmem + TM_S1 + hl, v);
      tmem_wait_ld();
#pragma unroll
      for (int q = 0; q < 32; ++q) G1[(ch * 32 + q) * 256] = __uint_as_float(v[q]);
      tmem_ld32(tmem + TM_S2 + hl, v);
      tmem_wait_ld();
      // whole lines through a staging area in the two buffers that hold nothing an MMA or a copy still reads
      store_rows_own(p.gW2 + long{sid} * (256 * 64) + (hrow - lane) * 64 + ch * 32, v,
                     smem + (warp < 8 ? o_s1 + warp * 4096 : o_z + (warp - 8) * 4096), lane);
      if (ch == 0) p.gb1[long{sid} * 256 + hrow] = sGb1[hrow];
      if (tid < 64) p.gb2[long{sid} * 64 + tid] = sGb2[tid];
    }
  };

  auto role = [&](uint32_t r) { return r == R_GZ ? o_gz : r == R_Z ? o_z : r == R_S1 ? o_s1 : r == R_S2 ? o_s2 : 0u; };
  // One product, written out: the issue is what the sweep waits for, so nothing stands between a product's barriers and its
  // MMAs but two additions to the descriptors.  (The operands' offsets are the same in all lanes, and known to be through the
  // shuffles of a step, so that the descriptors are put together in uniform registers.)
  auto uniform = [&](uint32_t v) { return __shfl_sync(0xffffffffu, v, 0); };
  const uint32_t base = smem_u32(smem);
  auto issue = [&](uint32_t kind, uint32_t d, uint32_t a_off, uint32_t b_off) {
    const bool tok = kind == P_TOK, mn = kind >= P_HID_MN;
    const uint32_t idesc = tok ? umma_idesc_bf16(64, 64, true, true, false)
                               : mn ? umma_idesc_bf16(128, 64, false, true, false) : umma_idesc_bf16(128, 64, false, false, false);
    const uint32_t as = tok ? 2048u >> 4 : 2u, bs = mn || tok ? 2048u >> 4 : 2u;
    uint32_t a = desc_lo(base + a_off, tok ? BIG : 16), b = desc_lo(base + b_off, tok ? BIG : mn ? 8192 : 16), dd = tmem + d;
    uint32_t acc = kind == P_HID_ACC || kind == P_HID_MN ? 1u : 0u;
#pragma unroll 1
    for (uint32_t k = tok ? 4u : 2u; k > 0; --k) {
      mma_lead_rt(dd, a, b, idesc, acc, lead);
      mma_lead_rt(dd, a + as, b + bs, idesc, 1u, lead);
      mma_lead_rt(dd, a + 2 * as, b + 2 * bs, idesc, 1u, lead);
      mma_lead_rt(dd, a + 3 * as, b + 3 * bs, idesc, 1u, lead);
      a += tok ? 4 * (2048u >> 4) : 16384u >> 4;      // the next K steps, or the other 128-row block
      b += tok ? 4 * (2048u >> 4) : 0u;
      dd += tok ? 0u : 64u;
      if (tok) acc = 1u;
    }
  };
  auto sweep_issue = [&](int g) {
    const int gsz = size_of(g);
    if ((g == 0 && !seen(E_5)) || !seen(SX2B) || !seen(SGZ1B) || !seen(SQ)) return;
#pragma unroll 1
    for (int k = 0; k < 2; ++k)       // G2, G3 of the group's first step
      issue(P_HID_MN, k ? TM_S1 : TM_S2, uniform(k ? o_s2 : o_s1), k ? S_Q : S_GZB);
    commit(C6);
    commit(C7);
    for (int j = gsz - 1; j >= 0; --j) {
      const uint32_t u_gz = uniform(o_gz), u_z = uniform(o_z), u_s1 = uniform(o_s1), u_s2 = uniform(o_s2);
      const uint32_t u_k = uniform(S_K + (nsw & 1) * TILE);
#pragma unroll
      for (int o = 0; o < kSweepMmas; ++o) {
        const MmaOp op = kSweepMma[o];
        if (!op.only_next || j > 0) {
          if (op.w0 != kNo && !seen(op.w0)) return;
          if (op.w1 != kNo && !seen(op.w1)) return;
          issue(op.kind, op.d, op.a + (op.ra == R_GZ ? u_gz : op.ra == R_Z ? u_z : op.ra == R_S1 ? u_s1 : op.ra == R_S2 ? u_s2 : 0u),
                op.b == S_K ? u_k : op.b + (op.rb == R_GZ ? u_gz : op.rb == R_Z ? u_z : op.rb == R_S1 ? u_s1 : op.rb == R_S2 ? u_s2 : 0u));
        }
        if (op.commit != kNo) commit(op.commit);
      }
      turn();
      ++nsw;
    }
    seen(E_S2);
  };

  auto sweep_copy = [&](int g) {      // a warp
    const Lane c = lane_of(kSweepCopy, kSweepCopies);
    const CopyOp& op = c.op;
    const int i0 = first_of(g), gsz = size_of(g);
    {   // the first step's: what does not come from the slots, then what does
      const int i = i0 + gsz - 1, slot = slot_of(g, gsz - 1);
      const bool outside = op.kind == K_TMA || op.src == A_ETA, any = op.kind != K_NONE && op.only_next;
      // (buffers as the last step would have found them; gZ1b, loaded beside the others here, to the place of S2)
      const uint32_t r = op.src == A_X2B ? o_s1 : op.src == A_GZ1B ? o_s2 : op.src == A_GZ1 ? o_gz : op.src == A_Z1 ? o_z : 0u;
      const uint32_t off = op.role == R_NONE ? op.off : r;
#pragma unroll 1
      for (int k = 0; k < 2; ++k) {
        if (k == 1) {
          if (!seen_all(BGROUP + (g & 1))) return;
          fence_proxy_async_all();      // the slots were written by the other CTA
        }
        copy(c, any && outside == (k == 0), i, slot, off, nsw & 1, false);
        __syncwarp();
      }
      if (!seen_all(C6) || !seen_all(C7)) return;
    }
    for (int j = gsz - 1; j >= 0; --j) {
      // this lane's copy of the step, put together before its event is waited for
      const int i = i0 + j, par = nsw & 1;
      const bool first = j == gsz - 1, more = j > 0;
      const int slot = slot_of(g, j - op.next);
      const bool act = !op.only_next || more;
      const uint32_t off = op.off + role(op.role) + (par ? 0u : op.par);
      uint8_t* const mem = op.src == A_ETA ? c.mem + (i - op.next) * 128L : place(c, slot);
#pragma unroll 1
      for (int ev = 0; ev < V_COUNT; ++ev) {
        if (!seen_all(kSweepEvent[ev])) return;
        if (lane == 0) {
          if ((ev == V_S2 && !first) || ev == V_V) {
            const bool dk = ev == V_S2;
            tma_store_2d(dk ? &tmDK : &tmDV, smem + (dk ? S_K + (par ^ 1) * TILE : S_V), 0, row_of(dk ? i + 1 : i));
            tma_commit_group();
          }
          if (ev == V_V) tma_wait_group_read<1>();      // the last dK has left its tile
          if (ev == V_C6) tma_wait_group_read<0>();     // dV has
        }
        __syncwarp();
        if (act && op.event == ev) {
          if (op.arm) arm(op.bar, op.arm);
          if (op.kind == K_TMA) tma_load_2d(smem + off, c.map, &bars[op.bar], 0, row_of(i - op.next));
          else bulk_load_1d(smem + off, mem, op.bytes, &bars[op.bar]);
        }
        __syncwarp();
      }
      turn();
      ++nsw;
    }
    if (!seen_all(E_S2)) return;
    if (lane == 0) {
      tma_store_2d(&tmDK, smem + S_K + ((nsw - 1) & 1) * TILE, 0, row_of(i0));      // (its tile's next K waits for it: V_V)
      tma_commit_group();
    }
    __syncwarp();
  };

  // d_eta; its fourth term, gZ1 G_b1, is summed over half of the hidden units by each of two warps: lane l takes the token pair (2 l, 2 l + 1)
  auto sweep_part = [&](int g, int half) {
    const int gsz = size_of(g);
    if (g == 0) {      // the gradient state is in place, and there are no addends yet
      if (!seen(E_5)) return;
      if (lane == 0) arrive(E_X);
    }
    for (int j = gsz - 1; j >= 0; --j) {
      if (!seen(E_S1) || !seen(SGZ1)) return;
      const uint8_t* bg = smem + o_gz + half * 16384 + (lane & 3) * 4;      // (128 rows: the swizzle's phase is the same)
      const float* gb = sGb1 + half * 128;
      const uint32_t chunk = lane >> 2;
      float a0 = 0.f, a1 = 0.f, c0 = 0.f, c1 = 0.f;
#pragma unroll 2
      for (int h = 0; h < 128; h += 8) {
        const float4 g0 = *reinterpret_cast<const float4*>(gb + h), g1 = *reinterpret_cast<const float4*>(gb + h + 4);
        uint32_t w[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) w[k] = *reinterpret_cast<const uint32_t*>(bg + h * 128 + k * 128 + ((chunk ^ k) << 4));
        a0 = fmaf(bf16_lo(w[0]), g0.x, a0); a1 = fmaf(bf16_hi(w[0]), g0.x, a1);
        c0 = fmaf(bf16_lo(w[1]), g0.y, c0); c1 = fmaf(bf16_hi(w[1]), g0.y, c1);
        a0 = fmaf(bf16_lo(w[2]), g0.z, a0); a1 = fmaf(bf16_hi(w[2]), g0.z, a1);
        c0 = fmaf(bf16_lo(w[3]), g0.w, c0); c1 = fmaf(bf16_hi(w[3]), g0.w, c1);
        a0 = fmaf(bf16_lo(w[4]), g1.x, a0); a1 = fmaf(bf16_hi(w[4]), g1.x, a1);
        c0 = fmaf(bf16_lo(w[5]), g1.y, c0); c1 = fmaf(bf16_hi(w[5]), g1.y, c1);
        a0 = fmaf(bf16_lo(w[6]), g1.z, a0); a1 = fmaf(bf16_hi(w[6]), g1.z, a1);
        c0 = fmaf(bf16_lo(w[7]), g1.w, c0); c1 = fmaf(bf16_hi(w[7]), g1.w, c1);
      }
      float* part = reinterpret_cast<float*>(smem + S_PART) + (nsw & 1) * 128;
      *reinterpret_cast<float2*>(part + half * 64 + 2 * lane) = make_float2(a0 + c0, a1 + c1);
      __syncwarp();
      if (lane == 0) arrive(E_PART);
      if (half == 0) {      // all of this step's slot is in shared memory (W1 came last): the recompute may have it
        if (!seen(SW1)) return;
        if (lane == 0) st_release_cluster(mapa(smem_u32(freed), peer), static_cast<uint32_t>(nsw + 1));
      }
      // d_eta of 32 tokens, when the other half of the sums is there and E5 has left the addends
      if (!seen(E_PART) || !seen(E_5)) return;
      const int t = half * 32 + lane;
      p.d_eta[(sid * NC + first_of(g) + j) * 64 + t] =
          __float2bfloat16(-(quad_sum(reinterpret_cast<const float*>(smem + S_X1), t) + (part[t] + part[64 + t])));
      __syncwarp();
      if (lane == 0) arrive(E_X);
      turn();
      ++nsw;
    }
  };

  // (a branch per role and kind of warp, each with its own share of the registers: where the branches meet before the work,
  // the compiler spills several times as much)
  if (warp < 16 && sweeper) {
    reg_take<kRegsEpi>();
    for (int g = idle ? nck : 0; g < nck; ++g) sweep_epi(g);
  } else if (warp < 16) {
    reg_take<kRegsEpi>();
    for (int g = idle ? nck : 0; g < nck; ++g)
      if (warp < 8 ? rec_chain(g) : rec_out(g)) break;
  } else {
    reg_give<kRegsHelp>();
    if (sweeper) {
      for (int g = idle ? nck : 0; g < nck && !*abort_flag; ++g) {
        if (warp == 16) sweep_issue(g);
        else if (warp == 17) sweep_copy(g);
        else sweep_part(g, warp - 18);
        __syncwarp();
      }
    } else {
      for (int g = idle ? nck : 0; g < nck && !*abort_flag; ++g) {
        if (warp == 16) rec_chain_issue(g);
        else if (warp == 17) rec_out_issue(g);
        else if (warp == 18) rec_chain_copy(g);
        else rec_out_copy(g);
        __syncwarp();
      }
    }
  }

  // ---- d_gamma, d_beta: the recompute's and the sweep's addends; teardown
  if (warp >= 16) tma_wait_group<0>();
  __syncwarp();
  float* fin = reinterpret_cast<float*>(smem + OFF_BIG);      // fp32[2][4][64] of the recompute, then of the sweep
  fence_proxy_async_smem();
  tc_fence_before_sync();
  const bool aborted = __syncthreads_or(*abort_flag != 0) != 0;
  tc_fence_after_sync();
  if (aborted && tid == 0) st_cluster_u32(mapa(smem_u32(const_cast<uint32_t*>(abort_flag)), peer), 1u);
  if (warp >= 8 && warp < 16 && !sweeper) {
    fin[tm8.quad * 64 + frag_colsum_col(tm8, lane)] = dgam;
    fin[256 + tm8.quad * 64 + frag_colsum_col(tm8, lane)] = dbet;
  }
  if (warp < 16 && sweeper && !(lane & 4)) {
    fin[512 + quad * 64 + f16_colsum_col(tm, lane)] = dgam_s;
    fin[768 + quad * 64 + f16_colsum_col(tm, lane)] = dbet_s;
  }
  __syncthreads();
  cluster_arrive();
  cluster_wait();
  if (!aborted && !idle && tid < 128 && sweeper) {
    const int f = tid & 63, o = (tid >> 6) * 256;
    const uint32_t a = mapa(smem_u32(fin + o + f), peer);
    const float r = (ld_cluster_f32(a) + ld_cluster_f32(a + 256)) + (ld_cluster_f32(a + 512) + ld_cluster_f32(a + 768));
    (tid < 64 ? p.d_gamma : p.d_beta)[long{sid} * 64 + f] = r + quad_sum(fin + 512 + o, f);
  }
  if (aborted) {
    // everything this CTA still has in flight is waited for (bounded, not cut short by the abort flag) before its shared
    // and tensor memory go away: the tensor-core work of both issuers, and the loads
    if ((warp == 16 || warp == 17) && lead) umma_commit(&bars[BDRAIN]);
    if (warp >= 16) {
      for (int b = 0; b < kRecBars; ++b)
        if ((ldaR >> b) & 1u) mbar_wait_bounded(&bars[b], ((ldpR >> b) & 1u) ^ 1u, never_flag, limit);
      for (int b = 0; b < BDRAIN - kRecBars; ++b)
        if ((ldaS >> b) & 1u) mbar_wait_bounded(&bars[kRecBars + b], ((ldpS >> b) & 1u) ^ 1u, never_flag, limit);
    }
    if (tid == 0) {
      mbar_wait_bounded(&bars[BDRAIN], 0, never_flag, limit);
      atomicExch(p.status, static_cast<uint32_t>(TTT_B200_ERR_TIMEOUT));
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, TM_COLS);
  cluster_arrive();      // the peer reads this CTA's addends, and no CTA leaves while another may still send to it
  cluster_wait();
}

}  // namespace

namespace {

// Once per device: the kernel's dynamic shared memory limit.
template <int kStreams>
int prepare_kernel() {
  static std::once_flag once[64];
  static cudaError_t attr_err[64];
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return ttt_set_error(TTT_B200_ERR_LAUNCH, "device index out of range");
  std::call_once(once[dev], [&] {
    attr_err[dev] = cudaFuncSetAttribute(ttt_bwd_pair_kernel<kStreams>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
  });
  if (attr_err[dev] != cudaSuccess) return ttt_set_error(TTT_B200_ERR_LAUNCH, cudaGetErrorString(attr_err[dev]));
  return TTT_B200_OK;
}

void cluster_attribute(cudaLaunchAttribute* attr, unsigned n) {
  attr->id = cudaLaunchAttributeClusterDimension;
  attr->val.clusterDim.x = n;
  attr->val.clusterDim.y = 1;
  attr->val.clusterDim.z = 1;
}

// How many clusters of kStreams streams the device runs at once (a cluster lives inside one GPC).  0 if the query fails.
template <int kStreams>
int clusters_at_once() {
  static std::once_flag once[64];
  static int cap[64];
  if (prepare_kernel<kStreams>()) return 0;
  int dev = 0;
  cudaGetDevice(&dev);
  std::call_once(once[dev], [&] {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * kStreams * 64);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = SMEM_BYTES;
    cudaLaunchAttribute attr[1];
    cluster_attribute(attr, 2 * kStreams);
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, ttt_bwd_pair_kernel<kStreams>, &cfg) != cudaSuccess) {
      cudaGetLastError();
      n = 0;
    }
    cap[dev] = n;
  });
  return cap[dev];
}

}  // namespace

// How many streams the device runs at once with two CTAs each.
int ttt_backward_pair_capacity() { return clusters_at_once<1>(); }
// ... and with two streams to a cluster, the faster form.
int ttt_backward_pairs_a_turn() { return 2 * clusters_at_once<2>(); }

// The streams from `first` on, to the last.
int ttt_launch_backward_pair(const ttt_b200_bwd_args* a, int first, cudaStream_t stream, uint32_t* status, uint64_t limit_ns,
                             int drop_load) {
  const uint64_t rows = static_cast<uint64_t>(a->B) * a->H * a->NC * 64;
  CUtensorMap tmQ, tmK, tmV, tmGo, tmDQ, tmDK, tmDV;
  if (int rc = ttt_make_tile_map(&tmQ, a->XQ, rows)) return rc;
  if (int rc = ttt_make_tile_map(&tmK, a->XK, rows)) return rc;
  if (int rc = ttt_make_tile_map(&tmV, a->XV, rows)) return rc;
  if (int rc = ttt_make_tile_map(&tmGo, a->grad_L_XQW_mini_batch, rows)) return rc;
  if (int rc = ttt_make_tile_map(&tmDQ, a->grad_L_XQ, rows)) return rc;
  if (int rc = ttt_make_tile_map(&tmDK, a->grad_L_XK, rows)) return rc;
  if (int rc = ttt_make_tile_map(&tmDV, a->grad_L_XV, rows)) return rc;
  BwdParams p;
  p.eta = static_cast<const __nv_bfloat16*>(a->last_eta);
  p.gamma = a->ttt_norm_weight;
  p.beta = a->ttt_norm_bias;
  p.W1c = a->W1_checkpoints; p.b1c = a->b1_checkpoints; p.W2c = a->W2_checkpoints; p.b2c = a->b2_checkpoints;
  uint8_t* const w1 = reinterpret_cast<uint8_t*>(a->W1_init_group);
  uint8_t* const w2 = reinterpret_cast<uint8_t*>(a->W2_init_group);
  void* const sc[A_COUNT] = {a->X2_group, a->Z1_group, a->grad_l_wrt_Z1_group, a->X2_bar_group, a->Z1_bar_group, w1, w2,
                             a->x_hat_fused_group, a->grad_l_wrt_Z2_group, a->x_hat_ln_group, a->b1_init_group,
                             a->std_ln_group, a->std_fused_group, a->b2_init_group};
  const uint32_t stride[A_COUNT] = {BIG, BIG, BIG, BIG, BIG, 65536, 65536, TILE, TILE, TILE, 1024, 256, 256, 256};
  for (int i = 0; i < A_COUNT; ++i) {
    p.sc[i] = static_cast<uint8_t*>(sc[i]);
    p.stride[i] = stride[i];
    // a slot beyond the group's takes the second halves of four W1_init_group and four W2_init_group slots
    p.spare[i] = i < 4 ? w1 + i * 65536 + BIG : i < 7 ? w2 + (i - 4) * 65536 + BIG : w2 + 3 * 65536 + BIG;
  }
  for (int i = A_XHF; i <= A_GZ2B; ++i) p.spare[i] += (i - A_XHF) * TILE;
  const uint32_t vec_off[4] = {0, 1024, 1280, 1536};
  for (int i = A_RS; i <= A_S3; ++i) p.spare[i] += 3 * TILE + vec_off[i - A_RS];
  p.gW1_last = a->grad_L_W1_last; p.gb1_last = a->grad_L_b1_last;
  p.gW2_last = a->grad_L_W2_last; p.gb2_last = a->grad_L_b2_last;
  p.d_gamma = a->grad_L_ttt_norm_weight; p.d_beta = a->grad_L_ttt_norm_bias;
  p.gW1 = a->grad_L_W1_init; p.gb1 = a->grad_L_b1_init; p.gW2 = a->grad_L_W2_init; p.gb2 = a->grad_L_b2_init;
  p.d_eta = static_cast<__nv_bfloat16*>(a->grad_L_last_eta);
  p.first = first; p.streams = a->B * a->H; p.H = a->H; p.NC = a->NC; p.cgs = a->checkpoint_group_size; p.nck = a->num_checkpoints;
  p.drop_load = drop_load;
  p.status = status;
  p.wait_limit_ns = limit_ns;
  const int streams = a->B * a->H - first;
  // streams to a cluster: one only where clusters of one stream hold all streams at once and clusters of two do not
  const int per = streams > 2 * clusters_at_once<2>() && streams <= clusters_at_once<1>() ? 1 : 2;
  if (int rc = per == 1 ? prepare_kernel<1>() : prepare_kernel<2>()) return rc;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>((streams + per - 1) / per * 2 * per));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = SMEM_BYTES;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  cluster_attribute(attr, 2 * per);
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, per == 1 ? ttt_bwd_pair_kernel<1> : ttt_bwd_pair_kernel<2>, tmQ, tmK, tmV, tmGo,
                                           tmDQ, tmDK, tmDV, p);
  if (e != cudaSuccess) return ttt_set_error(TTT_B200_ERR_LAUNCH, cudaGetErrorString(e));
  return TTT_B200_OK;
}
