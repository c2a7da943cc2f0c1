// TTT-MLP backward for sm_100a: one persistent CTA per (batch, head) stream.
//
// Replaces the reference's bwd_ttt_mlp_ker (kernels/ttt_backward/ttt.cu:179-1443); the math is
// that of kernels/ttt_backward/matching.py:57-342 (forward with saved intermediates, then the
// hand-derived reverse step), driven like kernels/ttt_backward/matching.py:539-663: for every
// checkpoint group, last to first, recompute the forward from the group's checkpoint, then
// sweep the group in reverse.
//
// Layout conventions are those of the forward kernel: every 64x256 / 256x64 quantity is
// "hidden-major" (hidden unit = TMEM lane = one thread in the epilogues), every 64x64
// quantity "token-major" (token = TMEM lane, M = 64).  All contractions are one of two MMA
// forms (ttt_device.cuh).  Tensor memory (512 columns):
//   [  0,256)  fp32 state: W1^T | W2 while recomputing, dL/dW1^T | dL/dW2 while sweeping
//              (the gradient state is parked in the grad_L_W*_init output buffers in between)
//   [256,384)  accumulator A (256 x 64, or a 64 x 64 one in its first 64 columns)
//   [384,512)  accumulator B (256 x 64, or two 64 x 64 ones)
//
// Scratch.  The recompute phase writes, per mini-batch slot of the group, into the caller's
// `*_group` tensors (raw images of 128-byte-swizzled shared-memory tiles, so the sweep can
// bring them back with plain bulk copies):
//   X2_group, grad_l_wrt_Z1_group, Z1_bar_group (holds gelu'(Z1_bar)), X2_bar_group : [256][64 tok] bf16
//   Z1_group : [256][64 tok] f16 (the sweep evaluates gelu' and gelu'' of it in packed f16)
//   W1_init_group / W2_init_group (first 32 KB of each slot): bf16 W1^T / W2 before the update
//   x_hat_fused, grad_l_wrt_Z2, x_hat_ln_group : [64 tok][64] bf16
//   std_fused_group, std_ln_group : fp32 [64]
//
// Reverse step for mini-batch i (G* = gradient w.r.t. the state after the update, go = dL/dOut):
//   S4   gZ2b = LNbwd(go * gamma; x_hat_ln, std_ln);  d_gamma, d_beta += column sums
//   G1   gX2b^T = W2+ gZ2b^T          E1  gZ1b^T = gX2b^T * gelu'(Z1b^T);  G_b1 += row sums
//   G2   G_W2 += X2b^T gZ2b     G3  G_W1^T += gZ1b^T Q     G7  dQ = go + gZ1b W1+^T
//   E2   bf16 snapshots of G_W1^T, G_W2 (the "last" values the update-rule terms use)
//   G4   A1raw^T = G_W1^T K^T   G8  T1 = gZ1 G_W1          G5  acc1 = X2 G_W2
//   E3   A1^T = -eta (A1raw^T + G_b1);  P^T = A1^T gelu'(Z1^T);  S^T = A1^T gelu''(Z1^T)
//   G6   acc2 = P W2            G10 G_W2 += P^T gZ2
//   E4   A2 = -eta (acc1 + G_b2) + acc2, second-order LayerNorm terms -> gZ2in, dV, d_gamma,
//        d_beta, d_eta, dK (partial)
//   G11  gX2^T = W2 gZ2in^T + G_W2snap (-eta gZ2)^T        G12 R^T = W2 gZ2^T
//   E5   gZ1in^T = gX2^T gelu'(Z1^T) + R^T S^T;  G_b1 += row sums
//   G13  dK += gZ1in W1^T       G14 G_W2 += X2^T gZ2in     G15 G_W1^T += gZ1in^T K
//
// What bounds it: one chain of 12 MMA phases and as many epilogues on two warps per scheduler (128 streams: tensor pipe
// 15 %, issue slots 30 %, DRAM 38 %; the warps wait for tensor memory, the MMAs and, half a warp per issue, for
// instructions).  The epilogues run on packed fp32 pairs and take column sums from registers.  Measured per mini-batch, 128
// streams of 128: 25.2 -> 21.6 us in groups of 8, 23.6 in groups of 4 (64 mini-batches in groups of 8: 25.1 -> 23.5 by the
// packed pairs; 32 in groups of 4: 25.5 -> 24.0 by shared-space addresses and unrolled column passes).  Sixteen warps
// with the recompute's output pass beside its chain were no faster (24.4-26 us: 128 registers a thread and more code
// than the instruction cache holds).
//
// Deviations from the reference kernel (see include/ttt_mlp_b200.h): outputs are overwritten,
// not accumulated; `Out` is never touched.  Every wait is bounded.
#include <mutex>

#include "ttt_device.cuh"
#include "ttt_internal.h"

using namespace tttdev;

namespace {

constexpr int kThreads = 256;
// The thread that issues the bulk copies and waits for their completion is not one of the four MMA issuers
// (lane 0 of warps 0..3): its bookkeeping between a barrier and the next MMA group stays off the issue path.
constexpr int kProd = 128;

// The MMAs of one phase are issued by lane 0 of warps 0..3: four instruction streams on four
// schedulers instead of one.  Every issuer commits (an issuer without work too), so the MMA
// barrier counts four arrivals per phase.
#define TTT_ISSUE(W0, W1, W2, W3)   \
  if (warp < 4) {                   \
    if (elect_one()) {              \
      tc_fence_after_sync();        \
      if (warp == 0) { W0; }        \
      else if (warp == 1) { W1; }   \
      else if (warp == 2) { W2; }   \
      else { W3; }                  \
      commit();                     \
    }                               \
    __syncwarp();                   \
  }

// ---- shared memory map (offsets from a 1024-byte aligned base)
constexpr uint32_t OFF_BIG = 0;                      // 5 hidden-major buffers of 32 KB
constexpr uint32_t OFF_T = 5 * BIG;                  // 7 token tiles of 8 KB
constexpr uint32_t OFF_B2 = OFF_T + 7 * TILE;        // fp32[64]  b2 (recompute)
constexpr uint32_t OFF_GB2 = OFF_B2 + 256;           // fp32[64]  dL/db2 state
constexpr uint32_t OFF_GAMMA = OFF_GB2 + 256;
constexpr uint32_t OFF_BETA = OFF_GAMMA + 256;
constexpr uint32_t OFF_SIGLN = OFF_BETA + 256;       // fp32[64]
constexpr uint32_t OFF_SIGF = OFF_SIGLN + 256;       // fp32[64]
constexpr uint32_t OFF_GB1 = OFF_SIGF + 256;         // fp32[256] copy of the per-thread dL/db1
constexpr uint32_t OFF_PART = OFF_GB1 + 1024;        // fp32[8][64] partial sums for d_eta (one row per warp)
constexpr uint32_t OFF_ETA = OFF_PART + 2048;        // bf16[2][64]
constexpr uint32_t OFF_BAR = OFF_ETA + 256;          // 17 mbarriers
constexpr uint32_t OFF_MISC = OFF_BAR + 192;
constexpr uint32_t OFF_XCH = OFF_MISC + 64;        // fp32[2][64][8] row-sum exchange between warp pairs
constexpr uint32_t SMEM_USED = OFF_XCH + 4096;
constexpr uint32_t SMEM_BYTES = SMEM_USED + 1024;
static_assert(SMEM_BYTES <= 232448, "exceeds the 227 KB per-CTA shared memory of sm_100");

// barrier indices
constexpr int BAR_BIG = 0;     // +buffer index (0..4)
constexpr int BAR_T = 5;       // +tile index (0..6)
constexpr int BAR_IN = 12;     // +stage (0..1), recompute inputs
constexpr int BAR_MMA = 14;
constexpr int BAR_V = 15;      // recompute: the single V tile
constexpr int BAR_DRAIN = 16;  // abort path only

constexpr uint32_t TM_S1 = 0;      // W1^T / dL/dW1^T
constexpr uint32_t TM_S2 = 128;    // W2   / dL/dW2
constexpr uint32_t TM_A = 256;
constexpr uint32_t TM_B = 384;
constexpr uint32_t TM_COLS = 512;

struct BwdParams {
  const __nv_bfloat16* eta;
  const float* gamma;
  const float* beta;
  const float* W1c; const float* b1c; const float* W2c; const float* b2c;
  // scratch
  uint8_t* sc_W1; uint8_t* sc_W2;                       // w_stride bytes per slot, first 32 KB used
  long w_stride;                                        // 64 KB in the caller's fp32-shaped tensors, 32 KB in the built-in scratch
  uint8_t* sc_Z1; uint8_t* sc_X2; uint8_t* sc_gZ1; uint8_t* sc_Z1b; uint8_t* sc_X2b;   // 32 KB per slot
  uint8_t* sc_xhf; uint8_t* sc_gof; uint8_t* sc_gZ2; uint8_t* sc_xhln;                 // 8 KB per slot
  float* sc_sigf; float* sc_sigln;                      // 64 floats per slot
  // upstream
  const float* gW1_last; const float* gb1_last; const float* gW2_last; const float* gb2_last;
  // outputs
  float* d_gamma; float* d_beta;
  float* gW1; float* gb1; float* gW2; float* gb2;
  __nv_bfloat16* d_eta;
  uint8_t* dXQ; uint8_t* dXK; uint8_t* dXV;              // bf16 [rows][64], row-major
  int H, NC, cgs, nck;
  int drop_load;            // test only: mini-batch whose recompute inputs stream 0 never loads (-1: none)
  uint32_t* status;
  uint64_t wait_limit_ns;
};

__global__ void __launch_bounds__(kThreads, 1)
ttt_bwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
               const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmGo,
               const __grid_constant__ CUtensorMap tmDQ, const __grid_constant__ CUtensorMap tmDK,
               const __grid_constant__ CUtensorMap tmDV, const BwdParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_align_1024(smem_raw);

  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);   // same value, known to be warp-uniform
  const int quad = warp & 3, wg = warp >> 2;
  const int hrow = wg * 128 + quad * 32 + lane;
  const uint32_t lane_base = static_cast<uint32_t>(quad * 32) << 16;
  const TokMap tm(warp, lane);          // this thread's fragment of the 64 x 64 token-major tiles
  const long sid = blockIdx.x;
  const int head = static_cast<int>(sid % p.H);
  const int NC = p.NC, cgs = p.cgs;

  auto big = [&](int i) -> uint8_t* { return smem + OFF_BIG + i * BIG; };
  auto tile = [&](int i) -> uint8_t* { return smem + OFF_T + i * TILE; };
  float* sB2 = reinterpret_cast<float*>(smem + OFF_B2);
  float* sGb2 = reinterpret_cast<float*>(smem + OFF_GB2);
  float* sGamma = reinterpret_cast<float*>(smem + OFF_GAMMA);
  float* sBeta = reinterpret_cast<float*>(smem + OFF_BETA);
  float* sSigLn = reinterpret_cast<float*>(smem + OFF_SIGLN);
  float* sSigF = reinterpret_cast<float*>(smem + OFF_SIGF);
  float* sGb1 = reinterpret_cast<float*>(smem + OFF_GB1);
  float* sPart = reinterpret_cast<float*>(smem + OFF_PART);
  __nv_bfloat16* sEta = reinterpret_cast<__nv_bfloat16*>(smem + OFF_ETA);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + OFF_BAR);
  float* sXch = reinterpret_cast<float*>(smem + OFF_XCH);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + OFF_MISC);
  volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(smem + OFF_MISC + 4);
  volatile uint32_t* never_flag = reinterpret_cast<volatile uint32_t*>(smem + OFF_MISC + 8);   // stays 0
  const uint64_t limit = p.wait_limit_ns;

  if (tid == kProd) {
    for (int i = 0; i < 17; ++i) mbar_init(&bars[i], (i == BAR_MMA || i == BAR_DRAIN) ? 4 : 1);
    fence_mbar_init();
    *abort_flag = 0;
    *never_flag = 0;
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
  if (tid < 64) {
    sGamma[tid] = p.gamma[head * 64 + tid];
    sBeta[tid] = p.beta[head * 64 + tid];
    sGb2[tid] = p.gb2_last[sid * 64 + tid];
  }
  float Gb1 = p.gb1_last[sid * 256 + hrow];
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot;

  // ---- barrier bookkeeping: every thread waits on every barrier use, in program order, or counts it (skip_bar)
  uint32_t ph = 0;        // expected parity per barrier
  uint32_t pending = 0;   // thread 0: loads issued and not yet waited for
  auto wait_bar = [&](int b) {
    if (mbar_wait_bounded(&bars[b], (ph >> b) & 1u, abort_flag, limit)) {
      ph ^= 1u << b;
      pending &= ~(1u << b);
    }
  };
  auto skip_bar = [&](int b) { ph ^= 1u << b; };      // a use that this warp need not wait for
  auto wait_mma = [&]() {
    wait_bar(BAR_MMA);
    __syncwarp();
    tc_fence_after_sync();
  };
  auto publish = [&]() {
    fence_proxy_async_smem();   // generic-proxy writes to shared memory -> async proxy (MMA, bulk copies)
    tc_fence_before_sync();
    __syncthreads();
  };
  auto commit = [&]() { umma_commit(&bars[BAR_MMA]); };   // thread 0
  // thread 0: bulk-load helpers
  auto load_big = [&](int buf, const uint8_t* src) {
    mbar_expect_tx(&bars[BAR_BIG + buf], BIG);
    bulk_load_1d(big(buf), src, BIG, &bars[BAR_BIG + buf]);
    pending |= 1u << (BAR_BIG + buf);
  };

  const long tok_rows0 = sid * NC * 64;      // first row of this stream in the [rows][64] token tensors

  // ---- column sums over the 64 tokens of a token-major quantity are taken from the registers of the epilogue that
  // produces it (frag_colsum: seven shuffles), one row of four per quadrant, added up by threads 0..63 after the next
  // barrier.  (Passes over the bf16 tiles inside the MMA windows outlasted those windows by a thousand cycles.)
  float* sCS = sXch + 512;      // fp32[4][64], behind the row-sum exchange
  auto put_colsum = [&](const f32x2 (&v)[4]) { sCS[tm.quad * 64 + frag_colsum_col(tm, lane)] = frag_colsum(v, lane); };
  auto quad_sum = [&](int f) { return (sCS[f] + sCS[64 + f]) + (sCS[128 + f] + sCS[192 + f]); };
  float dgam = 0.f, dbet = 0.f;      // this lane's column (frag_colsum_col) of d_gamma / d_beta
  // All CTAs reach a group boundary together, and each then reads 132 KB of state: the lines are asked
  // into L2 one step ahead (two 64 KB matrices = 2 x 512 lines, two lines of each per thread).
  auto prefetch_state = [&](const float* m1, const float* m2) {
    const char* a = reinterpret_cast<const char*>(m1) + tid * 128;
    const char* b = reinterpret_cast<const char*>(m2) + tid * 128;
    prefetch_l2(a);
    prefetch_l2(a + 32768);
    prefetch_l2(b);
    prefetch_l2(b + 32768);
  };
  // =====================================================================================
  const float* Gsrc_W1 = p.gW1_last + sid * (64 * 256);
  const float* Gsrc_W2 = p.gW2_last + sid * (256 * 64);
  float* Gdst_W1 = p.gW1 + sid * (64 * 256);
  float* Gdst_W2 = p.gW2 + sid * (256 * 64);
  bool aborted = false;

  for (int ck = p.nck - 1; ck >= 0 && !aborted; --ck) {
    const int i0 = ck * cgs;
    const int gsz = min(cgs, NC - i0);
    const long slot0 = sid * cgs;           // scratch slot of the group's first mini-batch
    // buffer roles during recompute: 0 = W1^T bf16, 1 = W2 bf16, 2 = X2^T / X2_bar^T,
    // 3 = Z1^T -> U1^T -> Z1_bar^T, 4 = G' -> dl/dZ1^T; every one of them also leaves for the
    // scratch slot as a bulk copy.  Token tiles: 0..3 = K, Q of two stages, 4 = V, 5 = gZ2, 6 = U2.
    uint8_t* bW1 = big(0);
    uint8_t* bW2 = big(1);
    uint8_t* bX2 = big(2);
    uint8_t* bZ1 = big(3);
    uint8_t* bGP = big(4);
    uint8_t* tV = tile(4);
    uint8_t* tGZ2 = tile(5);
    uint8_t* tU2 = tile(6);

    auto issue_inputs = [&](int j) {   // thread 0
      if (i0 + j == p.drop_load && sid == 0) return;
      const int s = j & 1;
      const int row0 = static_cast<int>(tok_rows0 + (long)(i0 + j) * 64);
      mbar_expect_tx(&bars[BAR_IN + s], 2 * TILE + 128);
      tma_load_2d(tile(2 * s + 0), &tmK, &bars[BAR_IN + s], 0, row0);
      tma_load_2d(tile(2 * s + 1), &tmQ, &bars[BAR_IN + s], 0, row0);
      bulk_load_1d(sEta + s * 64, p.eta + (sid * NC + i0 + j) * 64, 128, &bars[BAR_IN + s]);
      pending |= 1u << (BAR_IN + s);
    };
    auto issue_v = [&](int j) {        // thread 0
      mbar_expect_tx(&bars[BAR_V], TILE);
      tma_load_2d(tV, &tmV, &bars[BAR_V], 0, static_cast<int>(tok_rows0 + (long)(i0 + j) * 64));
      pending |= 1u << BAR_V;
    };
    if (tid == kProd) {
      issue_inputs(0);
      issue_v(0);
      if (gsz > 1) issue_inputs(1);
    }

    // ---- checkpoint -> tensor memory (fp32) + shared memory (bf16) + scratch slot 0 (bf16)
    float b1v = p.b1c[(sid * p.nck + ck) * 256 + hrow];
    if (tid < 64) sB2[tid] = p.b2c[(sid * p.nck + ck) * 64 + tid];
    {
      const float* W1g = p.W1c + (sid * p.nck + ck) * (64 * 256);
      const float* W2g = p.W2c + (sid * p.nck + ck) * (256 * 64) + hrow * 64;
#pragma unroll 1
      for (int half = 0; half < 2; ++half) {
        uint32_t v[32];
        float f[32];
        float4 q4[8];
        // both matrices' loads of this half go out before either is used (one memory round trip, not two)
#pragma unroll
        for (int j = 0; j < 32; ++j) f[j] = W1g[(half * 32 + j) * 256 + hrow];
#pragma unroll
        for (int j = 0; j < 8; ++j) q4[j] = reinterpret_cast<const float4*>(W2g)[half * 8 + j];
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = __float_as_uint(f[j]);
        tmem_st32(tmem + lane_base + TM_S1 + wg * 64 + half * 32, v);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const uint4 w = pack_chunk(f + c * 8);
          const uint32_t off = sw128_off(hrow, half * 4 + c);
          *reinterpret_cast<uint4*>(bW1 + off) = w;
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          f[j * 4 + 0] = q4[j].x; f[j * 4 + 1] = q4[j].y; f[j * 4 + 2] = q4[j].z; f[j * 4 + 3] = q4[j].w;
        }
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = __float_as_uint(f[j]);
        tmem_st32(tmem + lane_base + TM_S2 + wg * 64 + half * 32, v);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const uint4 w = pack_chunk(f + c * 8);
          const uint32_t off = sw128_off(hrow, half * 4 + c);
          *reinterpret_cast<uint4*>(bW2 + off) = w;
        }
      }
      tmem_wait_st();
    }
    publish();
    if (tid == kProd) {   // bf16 images of the checkpoint = pre-update weights of the group's first mini-batch
      bulk_store_1d(p.sc_W1 + slot0 * p.w_stride, bW1, BIG);
      bulk_store_1d(p.sc_W2 + slot0 * p.w_stride, bW2, BIG);
      tma_commit_group();
    }

    // ================================================================== recompute the group
    for (int j = 0; j < gsz; ++j) {
      const int s = j & 1;
      const long slot = slot0 + j;
      const uint8_t* sK = tile(2 * s + 0);
      const uint8_t* sQ = tile(2 * s + 1);
      const uint8_t* sV = tV;
      const __nv_bfloat16* eta = sEta + s * 64;
      if (j == gsz - 1) prefetch_state(Gsrc_W1, Gsrc_W2);    // read back when the sweep starts
      wait_bar(BAR_IN + s);

      // MMA1: Z1^T = W1^T K^T
      TTT_ISSUE(mma_hidden_half(tmem + TM_A, smem_u32(bW1), smem_u32(sK), false, false, 0),
                mma_hidden_half(tmem + TM_A, smem_u32(bW1), smem_u32(sK), false, false, 1),
                ,
                )
      wait_mma();
      {
        // (this and the other passes over 64 columns are unrolled: one pass's stores run beside the next one's
        // loads, 24.5 -> 24.0 us per mini-batch at 128 streams; all 64 columns loaded at once is slower, 24.2)
#pragma unroll
        for (int half = 0; half < 4; ++half) {   // 16 columns per pass
          uint32_t v[16];
          tmem_ld16(tmem + lane_base + TM_A + wg * 64 + half * 16, v);
          tmem_wait_ld();
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            uint32_t z[4], g[4], gp[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const f32x2 x = add2(pk(v[c * 8 + 2 * k], v[c * 8 + 2 * k + 1]), pk1(b1v));
              f32x2 y, yp;
              gelu_pair2(x, y, yp);
              z[k] = f32x2_to_f16x2(x);          // f16: the sweep evaluates gelu' and gelu'' of it in f16
              g[k] = f32x2_to_bf16x2(y);
              gp[k] = f32x2_to_bf16x2(yp);
            }
            const uint32_t off = sw128_off(hrow, half * 2 + c);
            *reinterpret_cast<uint4*>(bX2 + off) = make_uint4(g[0], g[1], g[2], g[3]);
            *reinterpret_cast<uint4*>(bGP + off) = make_uint4(gp[0], gp[1], gp[2], gp[3]);
            *reinterpret_cast<uint4*>(bZ1 + off) = make_uint4(z[0], z[1], z[2], z[3]);
          }
        }
      }
      if (tid == kProd && j > 0) tma_wait_group_read<0>();     // the previous mini-batch's x_hat_ln has left the U2 tile
      publish();
      if (tid == kProd) {
        bulk_store_1d(p.sc_X2 + slot * BIG, bX2, BIG);
        bulk_store_1d(p.sc_Z1 + slot * BIG, bZ1, BIG);
        tma_commit_group();
      }

      // MMA2: Z2 = X2 W2
      TTT_ISSUE(mma_token_major(tmem + TM_B, smem_u32(bX2), smem_u32(bW2)),
                ,
                ,
                )
      wait_mma();
      wait_bar(BAR_V);
      {
        TokFrag x, g;
        uint32_t kk[8], vv[8];
        frag_ld(tm, tmem + TM_B, x);
        frag_ld_raw(tm, sK, kk);          // requested before the all-reduces of the LayerNorm, used after them
        frag_ld_raw(tm, sV, vv);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const f32x2 b = frag_col(tm, sB2, q);
          x.a[q] = add2(x.a[q], b);
          x.b[q] = add2(x.b[q], b);
        }
        float rs0, rs1;
        frag_layernorm(tm, x, TTT_LN_EPS, sXch, 1, rs0, rs1);
        f32x2 a0 = 0ull, a1 = 0ull, c0 = 0ull, c1 = 0ull;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const f32x2 gam = frag_col(tm, sGamma, q), bet = frag_col(tm, sBeta, q), neg = pk1(-1.f);
          const f32x2 t0 = fma2(bf16x2_to_f32x2(vv[2 * q]), neg, bf16x2_to_f32x2(kk[2 * q]));          // K - V
          const f32x2 t1 = fma2(bf16x2_to_f32x2(vv[2 * q + 1]), neg, bf16x2_to_f32x2(kk[2 * q + 1]));
          g.a[q] = mul2(fma2(gam, x.a[q], add2(t0, bet)), gam);
          g.b[q] = mul2(fma2(gam, x.b[q], add2(t1, bet)), gam);
          a0 = add2(a0, g.a[q]); a1 = fma2(g.a[q], x.a[q], a1);
          c0 = add2(c0, g.b[q]); c1 = fma2(g.b[q], x.b[q], c1);
        }
        // x_hat_fused leaves through the V tile (every thread overwrites exactly the elements it has just
        // read) as a bulk store; grad_output_fused is not kept: the sweep rebuilds it from x_hat_fused, K, V
        frag_st_tile(tm, tV, x);
        float a[2] = {hsum(a0), hsum(a1)}, b[2] = {hsum(c0), hsum(c1)};
        frag_allreduce2<1>(tm, a, b, sXch, 1);
        const f32x2 sc0 = pk1(rs0 * (1.f / 64.f)), sc1 = pk1(rs1 * (1.f / 64.f));
        const f32x2 ne0 = pk1(-__bfloat162float(eta[tm.r0])), ne1 = pk1(-__bfloat162float(eta[tm.r1]));
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          // dl/dZ2, rounded to bf16 once: the update below uses -eta times the rounded value.  The forward rounds the
          // product instead, and adds up b2 from the rounded products (the recompute with four CTAs per stream does so
          // too, this one and that with two take the fp32 ones): the state rebuilt inside a group differs from the
          // forward's by about that rounding, 2e-3 of b2's change since the checkpoint.
          const uint32_t w0 = f32x2_to_bf16x2(mul2(fma2(x.a[q], pk1(-a[1]), fma2(g.a[q], pk1(64.f), pk1(-a[0]))), sc0));
          const uint32_t w1 = f32x2_to_bf16x2(mul2(fma2(x.b[q], pk1(-b[1]), fma2(g.b[q], pk1(64.f), pk1(-b[0]))), sc1));
          *reinterpret_cast<uint32_t*>(tGZ2 + tm.off(tm.r0, q)) = w0;
          *reinterpret_cast<uint32_t*>(tGZ2 + tm.off(tm.r1, q)) = w1;
          g.a[q] = mul2(bf16x2_to_f32x2(w0), ne0);
          g.b[q] = mul2(bf16x2_to_f32x2(w1), ne1);
          x.a[q] = add2(g.a[q], g.b[q]);
        }
        frag_st_tile(tm, tU2, g);
        put_colsum(x.a);
        if (tm.colhalf == 0 && tm.l3 == 0) {
          p.sc_sigf[slot * 64 + tm.r0] = rs0;     // the slot keeps 1/std: the sweep only ever divides by std
          p.sc_sigf[slot * 64 + tm.r1] = rs1;
        }
      }
      if (tid == kProd) tma_wait_group_read<0>();   // Z1 / X2 images have left shared memory
      publish();

      // MMA3: R^T = W2 gZ2^T
      if (tid == kProd) {
        bulk_store_1d(p.sc_xhf + slot * TILE, tV, TILE);
        bulk_store_1d(p.sc_gZ2 + slot * TILE, tGZ2, TILE);
        tma_commit_group();
      }
      TTT_ISSUE(mma_hidden_half(tmem + TM_A, smem_u32(bW2), smem_u32(tGZ2), false, false, 0),
                mma_hidden_half(tmem + TM_A, smem_u32(bW2), smem_u32(tGZ2), false, false, 1),
                ,
                )
      if (tid < 64) sB2[tid] += quad_sum(tid);
      wait_mma();
      {
        f32x2 bsum = 0ull;
#pragma unroll
        for (int half = 0; half < 4; ++half) {   // 16 columns per pass
          uint32_t v[16];
          tmem_ld16(tmem + lane_base + TM_A + wg * 64 + half * 16, v);
          const uint4 gr[2] = {ld_chunk_raw(bGP, hrow, half * 2), ld_chunk_raw(bGP, hrow, half * 2 + 1)};
          tmem_wait_ld();
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            const uint32_t off = sw128_off(hrow, half * 2 + c);
            const uint32_t gw[4] = {gr[c].x, gr[c].y, gr[c].z, gr[c].w};
            const uint4 ew = *reinterpret_cast<const uint4*>(eta + half * 16 + c * 8);     // one broadcast load
            const uint32_t et[4] = {ew.x, ew.y, ew.z, ew.w};
            uint32_t w[4], u[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              w[k] = f32x2_to_bf16x2(mul2(bf16x2_to_f32x2(gw[k]), pk(v[c * 8 + 2 * k], v[c * 8 + 2 * k + 1])));   // dl/dZ1
              const f32x2 t = mul2(bf16x2_to_f32x2(w[k]), bf16x2_to_f32x2(et[k] ^ 0x80008000u));   // -eta dl/dZ1
              bsum = add2(bsum, t);
              u[k] = f32x2_to_bf16x2(t);
            }
            *reinterpret_cast<uint4*>(bGP + off) = make_uint4(w[0], w[1], w[2], w[3]);     // dl/dZ1 in place over G'
            *reinterpret_cast<uint4*>(bZ1 + off) = make_uint4(u[0], u[1], u[2], u[3]);     // U1 over Z1
          }
        }
        b1v += hsum(bsum);
      }
      publish();

      // MMA4: W1^T += U1^T K ; W2 += X2^T U2
      if (tid == kProd) {
        tma_wait_group_read<0>();               // x_hat_fused has left the V tile
        if (j + 1 < gsz) issue_v(j + 1);
        bulk_store_1d(p.sc_gZ1 + slot * BIG, bGP, BIG);
        tma_commit_group();
      }
      TTT_ISSUE(mma_hidden_half(tmem + TM_S1, smem_u32(bZ1), smem_u32(sK), true, true, 0),
                mma_hidden_half(tmem + TM_S1, smem_u32(bZ1), smem_u32(sK), true, true, 1),
                mma_hidden_half(tmem + TM_S2, smem_u32(bX2), smem_u32(tU2), true, true, 0),
                mma_hidden_half(tmem + TM_S2, smem_u32(bX2), smem_u32(tU2), true, true, 1))
      wait_mma();
      {
#pragma unroll
        for (int half = 0; half < 4; ++half) {   // 16 columns per pass
          uint32_t v[16];
          float f[16];
          tmem_ld16(tmem + lane_base + TM_S1 + wg * 64 + half * 16, v);
          tmem_wait_ld();
#pragma unroll
          for (int q = 0; q < 16; ++q) f[q] = __uint_as_float(v[q]);
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            const uint4 w = pack_chunk(f + c * 8);
            const uint32_t off = sw128_off(hrow, half * 2 + c);
            *reinterpret_cast<uint4*>(bW1 + off) = w;
          }
          tmem_ld16(tmem + lane_base + TM_S2 + wg * 64 + half * 16, v);
          tmem_wait_ld();
#pragma unroll
          for (int q = 0; q < 16; ++q) f[q] = __uint_as_float(v[q]);
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            const uint4 w = pack_chunk(f + c * 8);
            const uint32_t off = sw128_off(hrow, half * 2 + c);
            *reinterpret_cast<uint4*>(bW2 + off) = w;
          }
        }
      }
      publish();

      // MMA5: Z1b^T = W1+^T Q^T
      if (tid == kProd) {
        if (j + 1 < gsz) {   // the new weights are the next mini-batch's pre-update weights
          bulk_store_1d(p.sc_W1 + (slot + 1) * p.w_stride, bW1, BIG);
          bulk_store_1d(p.sc_W2 + (slot + 1) * p.w_stride, bW2, BIG);
          tma_commit_group();
        }
      }
      TTT_ISSUE(mma_hidden_half(tmem + TM_A, smem_u32(bW1), smem_u32(sQ), false, false, 0),
                mma_hidden_half(tmem + TM_A, smem_u32(bW1), smem_u32(sQ), false, false, 1),
                ,
                )
      wait_mma();
      {
#pragma unroll
        for (int half = 0; half < 4; ++half) {   // 16 columns per pass
          uint32_t v[16];
          tmem_ld16(tmem + lane_base + TM_A + wg * 64 + half * 16, v);
          tmem_wait_ld();
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            uint32_t z[4], g[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              // the sweep needs gelu'(Z1_bar) only: it is cheaper here, next to gelu, than there from a bf16 copy
              f32x2 y, yp;
              gelu_pair2(add2(pk(v[c * 8 + 2 * k], v[c * 8 + 2 * k + 1]), pk1(b1v)), y, yp);
              g[k] = f32x2_to_bf16x2(y);
              z[k] = f32x2_to_bf16x2(yp);
            }
            const uint32_t off = sw128_off(hrow, half * 2 + c);
            *reinterpret_cast<uint4*>(bX2 + off) = make_uint4(g[0], g[1], g[2], g[3]);
            *reinterpret_cast<uint4*>(bZ1 + off) = make_uint4(z[0], z[1], z[2], z[3]);
          }
        }
      }
      publish();

      // MMA6: Z2b = X2b W2+ ; output LayerNorm statistics
      if (tid == kProd) {
        bulk_store_1d(p.sc_X2b + slot * BIG, bX2, BIG);
        bulk_store_1d(p.sc_Z1b + slot * BIG, bZ1, BIG);
        tma_commit_group();
      }
      TTT_ISSUE(mma_token_major(tmem + TM_B, smem_u32(bX2), smem_u32(bW2)),
                ,
                ,
                )
      wait_mma();
      {
        TokFrag x;
        frag_ld(tm, tmem + TM_B, x);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const f32x2 b = frag_col(tm, sB2, q);
          x.a[q] = add2(x.a[q], b);
          x.b[q] = add2(x.b[q], b);
        }
        float rs0, rs1;
        frag_layernorm(tm, x, TTT_LN_EPS, sXch, 1, rs0, rs1);
        frag_st_tile(tm, tU2, x);     // the U2 tile is dead since MMA4; x_hat_ln leaves through it
        if (tm.colhalf == 0 && tm.l3 == 0) {
          p.sc_sigln[slot * 64 + tm.r0] = rs0;
          p.sc_sigln[slot * 64 + tm.r1] = rs1;
        }
      }
      if (tid == kProd) tma_wait_group_read<0>();   // every big image of this mini-batch has left shared memory
      publish();
      if (tid == kProd) {
        bulk_store_1d(p.sc_xhln + slot * TILE, tU2, TILE);
        tma_commit_group();
        if (j + 2 < gsz && !*abort_flag) issue_inputs(j + 2);
      }
      if (*abort_flag) { aborted = true; break; }
    }
    if (aborted) break;

    // ================================================================== reverse sweep
    // buffer roles: i0b = W1+ (bf16), i1b = W2+, the other three free
    int ib0 = 0, ib1 = 1, ib2 = 2, ib3 = 3, ib4 = 4;
    uint8_t* t_go = tile(0);
    uint8_t* t_a = tile(1);     // x_hat_ln -> grad_output_fused -> d_gamma addends
    uint8_t* t_q = tile(2);     // Q -> gZ2in
    uint8_t* t_g = tile(3);     // gZ2b -> U2 = -eta gZ2
    uint8_t* t_k = tile(4);
    uint8_t* t_gz2 = tile(5);
    uint8_t* t_xf = tile(6);    // x_hat_fused
    // thread 0: loads of sweep step j, in three parts so that each can go out as early as its
    // destination is free (token tiles first: the step starts with them)
    auto issue_tiles_a = [&](int j) {          // dL/dOut, x_hat_ln + std_ln, x_hat_fused + std_fused
      const long slot = slot0 + j;
      const int row0 = static_cast<int>(tok_rows0 + (long)(i0 + j) * 64);
      mbar_expect_tx(&bars[BAR_T + 0], TILE);
      tma_load_2d(t_go, &tmGo, &bars[BAR_T + 0], 0, row0);
      mbar_expect_tx(&bars[BAR_T + 1], TILE + 256);
      bulk_load_1d(t_a, p.sc_xhln + slot * TILE, TILE, &bars[BAR_T + 1]);
      bulk_load_1d(sSigLn, p.sc_sigln + slot * 64, 256, &bars[BAR_T + 1]);
      mbar_expect_tx(&bars[BAR_T + 6], TILE + 256);
      bulk_load_1d(t_xf, p.sc_xhf + slot * TILE, TILE, &bars[BAR_T + 6]);
      bulk_load_1d(sSigF, p.sc_sigf + slot * 64, 256, &bars[BAR_T + 6]);
      pending |= (1u << (BAR_T + 0)) | (1u << (BAR_T + 1)) | (1u << (BAR_T + 6));
    };
    auto issue_rest = [&](int j) {             // Q, K + eta, dl/dZ2 tiles; X2_bar and dl/dZ1
      const long slot = slot0 + j;
      const int row0 = static_cast<int>(tok_rows0 + (long)(i0 + j) * 64);
      mbar_expect_tx(&bars[BAR_T + 2], TILE);
      tma_load_2d(t_q, &tmQ, &bars[BAR_T + 2], 0, row0);
      load_big(ib3, p.sc_X2b + slot * BIG);
      mbar_expect_tx(&bars[BAR_T + 4], TILE + 128);
      tma_load_2d(t_k, &tmK, &bars[BAR_T + 4], 0, row0);
      bulk_load_1d(sEta, p.eta + (sid * NC + i0 + j) * 64, 128, &bars[BAR_T + 4]);
      load_big(ib4, p.sc_gZ1 + slot * BIG);
      pending |= (1u << (BAR_T + 2)) | (1u << (BAR_T + 4));
    };
    // the dl/dZ2 tile of step j: its destination stages the previous step's dK on its way out, so this
    // load goes out one phase into the step, when that store has long read the tile
    auto issue_gz2 = [&](int j) {
      tma_wait_group_read<0>();
      mbar_expect_tx(&bars[BAR_T + 5], TILE);
      bulk_load_1d(t_gz2, p.sc_gZ2 + (slot0 + j) * TILE, TILE, &bars[BAR_T + 5]);
      pending |= 1u << (BAR_T + 5);
    };
    // scratch was written partly with generic-proxy stores by all threads, partly with bulk
    // stores by thread 0: order both before the bulk (async-proxy) copies that read it back
    asm volatile("fence.proxy.async;" ::: "memory");
    if (tid == kProd) tma_wait_group<0>();
    publish();
    if (tid == kProd) {
      issue_tiles_a(gsz - 1);
      load_big(ib2, p.sc_Z1b + (slot0 + gsz - 1) * BIG);
      issue_rest(gsz - 1);
    }
    // (the first step's loads are in flight while the gradient state comes back)
    // dL/dW state: global (fp32) -> tensor memory
    {
#pragma unroll 1
      for (int half = 0; half < 2; ++half) {
        uint32_t v[32];
        float4 q4[8];
        const float4* src = reinterpret_cast<const float4*>(Gsrc_W2 + hrow * 64 + half * 32);
#pragma unroll
        for (int q = 0; q < 32; ++q) v[q] = __float_as_uint(Gsrc_W1[(half * 32 + q) * 256 + hrow]);
#pragma unroll
        for (int q = 0; q < 8; ++q) q4[q] = src[q];
        tmem_st32(tmem + lane_base + TM_S1 + wg * 64 + half * 32, v);
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          v[q * 4 + 0] = __float_as_uint(q4[q].x); v[q * 4 + 1] = __float_as_uint(q4[q].y);
          v[q * 4 + 2] = __float_as_uint(q4[q].z); v[q * 4 + 3] = __float_as_uint(q4[q].w);
        }
        tmem_st32(tmem + lane_base + TM_S2 + wg * 64 + half * 32, v);
      }
      tmem_wait_st();
    }
    tc_fence_before_sync();   // the state columns are read by the MMAs of the first step

    for (int j = gsz - 1; j >= 0; --j) {
      const long slot = slot0 + j;
      const int row0 = static_cast<int>(tok_rows0 + (long)(i0 + j) * 64);   // first token row of this mini-batch
      f32x2 kpa[4], kpb[4];                                                  // partial dK, completed in E6
      if (j == 0 && ck > 0)                                                  // the next group's checkpoint
        prefetch_state(p.W1c + (sid * p.nck + ck - 1) * (64 * 256), p.W2c + (sid * p.nck + ck - 1) * (256 * 64));

      // ---- S4: backward of the output LayerNorm
      wait_bar(BAR_T + 0);
      wait_bar(BAR_T + 1);
      {
        uint32_t gw[8], xw[8];
        frag_ld_raw(tm, t_go, gw);
        frag_ld_raw(tm, t_a, xw);
        TokFrag g;
        f32x2 a0 = 0ull, a1 = 0ull, c0 = 0ull, c1 = 0ull, sb[4], sg[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const f32x2 gam = frag_col(tm, sGamma, q);
          g.a[q] = mul2(bf16x2_to_f32x2(gw[2 * q]), gam);
          g.b[q] = mul2(bf16x2_to_f32x2(gw[2 * q + 1]), gam);
          a0 = add2(a0, g.a[q]); a1 = fma2(g.a[q], bf16x2_to_f32x2(xw[2 * q]), a1);
          c0 = add2(c0, g.b[q]); c1 = fma2(g.b[q], bf16x2_to_f32x2(xw[2 * q + 1]), c1);
          sb[q] = add2(bf16x2_to_f32x2(gw[2 * q]), bf16x2_to_f32x2(gw[2 * q + 1]));
          sg[q] = fma2(bf16x2_to_f32x2(gw[2 * q]), bf16x2_to_f32x2(xw[2 * q]),
                       mul2(bf16x2_to_f32x2(gw[2 * q + 1]), bf16x2_to_f32x2(xw[2 * q + 1])));
        }
        dbet += frag_colsum(sb, lane);
        dgam += frag_colsum(sg, lane);
        float a[2] = {hsum(a0), hsum(a1)}, b[2] = {hsum(c0), hsum(c1)};
        frag_allreduce2<1>(tm, a, b, sXch, 1);
        const f32x2 q0 = pk1(sSigLn[tm.r0] * (1.f / 64.f)), q1 = pk1(sSigLn[tm.r1] * (1.f / 64.f));   // 1 / (64 std)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          g.a[q] = mul2(fma2(bf16x2_to_f32x2(xw[2 * q]), pk1(-a[1]), fma2(g.a[q], pk1(64.f), pk1(-a[0]))), q0);
          g.b[q] = mul2(fma2(bf16x2_to_f32x2(xw[2 * q + 1]), pk1(-b[1]), fma2(g.b[q], pk1(64.f), pk1(-b[0]))), q1);
          sb[q] = add2(g.a[q], g.b[q]);
        }
        frag_st_tile(tm, t_g, g);
        put_colsum(sb);
      }
      publish();
      // G1: gX2b^T = W2+ gZ2b^T
      TTT_ISSUE(mma_hidden_half(tmem + TM_A, smem_u32(big(ib1)), smem_u32(t_g), false, false, 0),
                mma_hidden_half(tmem + TM_A, smem_u32(big(ib1)), smem_u32(t_g), false, false, 1),
                ,
                )
      if (tid < 64) sGb2[tid] += quad_sum(tid);
      wait_mma();
      if (tid == kProd) load_big(ib1, p.sc_X2 + slot * BIG);   // W2+ is consumed (G1 was its only use): X2 for G5
      wait_bar(BAR_BIG + ib2);
      // ---- E1: gZ1b^T = gX2b^T * gelu'(Z1b^T), in place over Z1b^T
      {
        uint8_t* bz = big(ib2);
        f32x2 bsum = 0ull;
#pragma unroll
        for (int half = 0; half < 4; ++half) {   // 16 columns per pass
          uint32_t v[16];
          tmem_ld16(tmem + lane_base + TM_A + wg * 64 + half * 16, v);
          const uint4 zr[2] = {ld_chunk_raw(bz, hrow, half * 2), ld_chunk_raw(bz, hrow, half * 2 + 1)};
          tmem_wait_ld();
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            const uint32_t zw[4] = {zr[c].x, zr[c].y, zr[c].z, zr[c].w};      // gelu'(Z1_bar)
            uint32_t w[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const f32x2 t = mul2(bf16x2_to_f32x2(zw[k]), pk(v[c * 8 + 2 * k], v[c * 8 + 2 * k + 1]));
              bsum = add2(bsum, t);
              w[k] = f32x2_to_bf16x2(t);
            }
            *reinterpret_cast<uint4*>(bz + sw128_off(hrow, half * 2 + c)) = make_uint4(w[0], w[1], w[2], w[3]);
          }
        }
        Gb1 += hsum(bsum);
      }
      publish();
      if (tid == kProd) {   // x_hat_ln and its column sums are consumed: bring V into that tile (E4 rebuilds
                        // grad_output_fused = gamma x_hat_fused + beta - (V - K) from it)
        mbar_expect_tx(&bars[BAR_T + 1], TILE);
        tma_load_2d(t_a, &tmV, &bars[BAR_T + 1], 0, row0);
        pending |= 1u << (BAR_T + 1);
        issue_gz2(j);
      }
      wait_bar(BAR_BIG + ib3);
      wait_bar(BAR_T + 2);
      // G2 // G3 // G7
      TTT_ISSUE(mma_token_major(tmem + TM_B, smem_u32(big(ib2)), smem_u32(big(ib0))),
                mma_hidden_major(tmem + TM_S2, smem_u32(big(ib3)), smem_u32(t_g), true, true),
                mma_hidden_half(tmem + TM_S1, smem_u32(big(ib2)), smem_u32(t_q), true, true, 0),
                mma_hidden_half(tmem + TM_S1, smem_u32(big(ib2)), smem_u32(t_q), true, true, 1))
      wait_mma();
      // gZ1b is consumed: Z1 of this step comes in while E2 runs (X2_bar's buffer takes the W2 snapshot)
      if (tid == kProd) load_big(ib2, p.sc_Z1 + slot * BIG);
      // ---- E2: bf16 snapshots of the gradient state; dQ
      {
        uint8_t* s1b = big(ib0);
        uint8_t* s2b = big(ib3);
#pragma unroll
        for (int half = 0; half < 4; ++half) {   // 16 columns per pass
          uint32_t v[16];
          float f[16];
          tmem_ld16(tmem + lane_base + TM_S1 + wg * 64 + half * 16, v);
          tmem_wait_ld();
#pragma unroll
          for (int q = 0; q < 16; ++q) f[q] = __uint_as_float(v[q]);
#pragma unroll
          for (int c = 0; c < 2; ++c) st_chunk(s1b, hrow, half * 2 + c, f + c * 8);
          tmem_ld16(tmem + lane_base + TM_S2 + wg * 64 + half * 16, v);
          tmem_wait_ld();
#pragma unroll
          for (int q = 0; q < 16; ++q) f[q] = __uint_as_float(v[q]);
#pragma unroll
          for (int c = 0; c < 2; ++c) st_chunk(s2b, hrow, half * 2 + c, f + c * 8);
        }
        sGb1[hrow] = Gb1;
      }
      {   // dQ = go + gZ1b W1+^T, staged over the dL/dOut tile and stored by TMA
        TokFrag x;
        uint32_t gw[8];
        frag_ld(tm, tmem + TM_B, x);
        frag_ld_raw(tm, t_go, gw);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          x.a[q] = add2(x.a[q], bf16x2_to_f32x2(gw[2 * q]));
          x.b[q] = add2(x.b[q], bf16x2_to_f32x2(gw[2 * q + 1]));
        }
        frag_st_tile(tm, t_go, x);
      }
      publish();
      if (tid == kProd) {
        tma_store_2d(&tmDQ, t_go, 0, row0);
        tma_commit_group();
      }
      wait_bar(BAR_BIG + ib4);
      wait_bar(BAR_T + 4);
      // X2, requested two phases ago.  Only those who issue MMAs or the next load wait: nothing would hold that load, of W2
      // into the same buffer, back until a warp without a part in them had seen this one.
      if (warp <= kProd / 32) wait_bar(BAR_BIG + ib1);
      else skip_bar(BAR_BIG + ib1);
      // G4 // G8 // G5
      TTT_ISSUE(mma_token_major(tmem + TM_B, smem_u32(big(ib4)), smem_u32(big(ib0))),
                mma_token_major(tmem + TM_B + 64, smem_u32(big(ib1)), smem_u32(big(ib3))),
                mma_hidden_half(tmem + TM_A, smem_u32(big(ib0)), smem_u32(t_k), false, false, 0),
                mma_hidden_half(tmem + TM_A, smem_u32(big(ib0)), smem_u32(t_k), false, false, 1))
      // ---- while the MMAs run: partial sums over the hidden units of gZ1 * G_b1 (fourth term of d_eta)
      {
        // warp w takes hidden units 32 w .. 32 w + 31, lane l the token pair (2 l, 2 l + 1): one conflict-free
        // 4-byte load per row, four independent accumulators
        const uint8_t* bg = big(ib4) + (lane & 3) * 4;
        const uint32_t chunk = lane >> 2;
        float a0 = 0.f, a1 = 0.f, c0 = 0.f, c1 = 0.f;
#pragma unroll
        for (int hh = 0; hh < 32; hh += 4) {
          const int h = warp * 32 + hh;
          const float4 g = *reinterpret_cast<const float4*>(sGb1 + h);
          const uint32_t w0 = *reinterpret_cast<const uint32_t*>(bg + sw128_off(h, chunk));
          const uint32_t w1 = *reinterpret_cast<const uint32_t*>(bg + sw128_off(h + 1, chunk));
          const uint32_t w2 = *reinterpret_cast<const uint32_t*>(bg + sw128_off(h + 2, chunk));
          const uint32_t w3 = *reinterpret_cast<const uint32_t*>(bg + sw128_off(h + 3, chunk));
          a0 = fmaf(bf16_lo(w0), g.x, a0); a1 = fmaf(bf16_hi(w0), g.x, a1);
          c0 = fmaf(bf16_lo(w1), g.y, c0); c1 = fmaf(bf16_hi(w1), g.y, c1);
          a0 = fmaf(bf16_lo(w2), g.z, a0); a1 = fmaf(bf16_hi(w2), g.z, a1);
          c0 = fmaf(bf16_lo(w3), g.w, c0); c1 = fmaf(bf16_hi(w3), g.w, c1);
        }
        *reinterpret_cast<float2*>(sPart + warp * 64 + 2 * lane) = make_float2(a0 + c0, a1 + c1);
      }
      wait_mma();
      if (tid == kProd) {
        load_big(ib1, p.sc_W2 + slot * p.w_stride);      // X2 is consumed until G14: W2 takes its buffer
        tma_wait_group_read<0>();     // dQ has left the dL/dOut tile (E4 reuses it for dV)
      }
      wait_bar(BAR_BIG + ib2);
      // ---- E3: A1, P = A1 gelu'(Z1), S = A1 gelu''(Z1), gelu'(Z1)
      {
        uint8_t* bz = big(ib2);
        uint8_t* bp = big(ib4);
        uint8_t* bgp = big(ib0);
#pragma unroll
        for (int half = 0; half < 4; ++half) {   // 16 columns per pass
          uint32_t v[16];
          tmem_ld16(tmem + lane_base + TM_A + wg * 64 + half * 16, v);
          const uint4 zr[2] = {ld_chunk_raw(bz, hrow, half * 2), ld_chunk_raw(bz, hrow, half * 2 + 1)};
          tmem_wait_ld();
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            const uint32_t zw[4] = {zr[c].x, zr[c].y, zr[c].z, zr[c].w};
            const uint4 ew = *reinterpret_cast<const uint4*>(sEta + half * 16 + c * 8);     // one broadcast load
            const uint32_t et[4] = {ew.x, ew.y, ew.z, ew.w};
            uint32_t pw[4], sw[4], gw[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const f32x2 a1 = mul2(bf16x2_to_f32x2(et[k] ^ 0x80008000u),
                                    add2(pk(v[c * 8 + 2 * k], v[c * 8 + 2 * k + 1]), pk1(Gb1)));
              uint32_t gp, gpp;
              gelu_grad_h2(zw[k], gp, gpp);
              gw[k] = gp;                                        // kept as f16
              pw[k] = f32x2_to_bf16x2(mul2(a1, f16x2_to_f32x2(gp)));
              sw[k] = f32x2_to_bf16x2(mul2(a1, f16x2_to_f32x2(gpp)));
            }
            const uint32_t off = sw128_off(hrow, half * 2 + c);
            *reinterpret_cast<uint4*>(bp + off) = make_uint4(pw[0], pw[1], pw[2], pw[3]);
            *reinterpret_cast<uint4*>(bz + off) = make_uint4(sw[0], sw[1], sw[2], sw[3]);
            *reinterpret_cast<uint4*>(bgp + off) = make_uint4(gw[0], gw[1], gw[2], gw[3]);
          }
        }
      }
      publish();
      wait_bar(BAR_BIG + ib1);
      wait_bar(BAR_T + 5);
      // G6 // G10
      TTT_ISSUE(mma_token_major(tmem + TM_A, smem_u32(big(ib4)), smem_u32(big(ib1))),
                mma_hidden_half(tmem + TM_S2, smem_u32(big(ib4)), smem_u32(t_gz2), true, true, 0),
                mma_hidden_half(tmem + TM_S2, smem_u32(big(ib4)), smem_u32(t_gz2), true, true, 1),
                )
      wait_mma();
      if (tid == kProd) load_big(ib4, p.sc_W1 + slot * p.w_stride);
      wait_bar(BAR_T + 6);
      wait_bar(BAR_T + 1);   // grad_output_fused
      // ---- E4: second order through the fused LayerNorm + L2 gradient (token-major, all 8 warps)
      {
        TokFrag A2, t1, go;
        uint32_t gzw[8], xhw[8], kw[8];
        frag_ld_raw(tm, t_gz2, gzw);
        frag_ld_raw(tm, t_xf, xhw);
        frag_ld_raw(tm, t_k, kw);
        const float eta0 = __bfloat162float(sEta[tm.r0]), eta1 = __bfloat162float(sEta[tm.r1]);
        const float rs0 = sSigF[tm.r0], rs1 = sSigF[tm.r1];      // 1 / std
        float ra[4], rb[4];       // d_eta's row terms, sum A2, sum A2 xh, sum gxf xh
        {
          TokFrag acc1;
          uint32_t vw[8];
          frag_ld_raw(tm, t_a, vw);
          // X2 G_W2, P W2, gZ1 G_W1
          frag_ld(tm, tmem + TM_B + 64, acc1);
          frag_ld(tm, tmem + TM_A, A2);
          frag_ld(tm, tmem + TM_B, t1);
          f32x2 s0[4] = {0ull, 0ull, 0ull, 0ull}, s1[4] = {0ull, 0ull, 0ull, 0ull};
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const f32x2 gam = frag_col(tm, sGamma, q), bet = frag_col(tm, sBeta, q), gb2 = frag_col(tm, sGb2, q), neg = pk1(-1.f);
            const f32x2 x0 = bf16x2_to_f32x2(xhw[2 * q]), x1 = bf16x2_to_f32x2(xhw[2 * q + 1]);
            const f32x2 k0 = bf16x2_to_f32x2(kw[2 * q]), k1 = bf16x2_to_f32x2(kw[2 * q + 1]);
            // grad_output_fused = gamma x_hat_fused + beta - (V - K)
            go.a[q] = add2(fma2(bf16x2_to_f32x2(vw[2 * q]), neg, k0), fma2(gam, x0, bet));
            go.b[q] = add2(fma2(bf16x2_to_f32x2(vw[2 * q + 1]), neg, k1), fma2(gam, x1, bet));
            const f32x2 u0 = add2(acc1.a[q], gb2), u1 = add2(acc1.b[q], gb2);
            s0[0] = fma2(bf16x2_to_f32x2(gzw[2 * q]), u0, fma2(t1.a[q], k0, s0[0]));
            s1[0] = fma2(bf16x2_to_f32x2(gzw[2 * q + 1]), u1, fma2(t1.b[q], k1, s1[0]));
            A2.a[q] = fma2(u0, pk1(-eta0), A2.a[q]);
            A2.b[q] = fma2(u1, pk1(-eta1), A2.b[q]);
            s0[1] = add2(s0[1], A2.a[q]);
            s1[1] = add2(s1[1], A2.b[q]);
            s0[2] = fma2(A2.a[q], x0, s0[2]);
            s1[2] = fma2(A2.b[q], x1, s1[2]);
            s0[3] = fma2(mul2(go.a[q], gam), x0, s0[3]);
            s1[3] = fma2(mul2(go.b[q], gam), x1, s1[3]);
          }
#pragma unroll
          for (int i = 0; i < 4; ++i) { ra[i] = hsum(s0[i]); rb[i] = hsum(s1[i]); }
        }
        // all-reduce over the row's four lanes and two warps
#pragma unroll
        for (int sft = 1; sft <= 2; sft <<= 1)
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            ra[i] += __shfl_xor_sync(0xffffffffu, ra[i], sft);
            rb[i] += __shfl_xor_sync(0xffffffffu, rb[i], sft);
          }
        float4* x4 = reinterpret_cast<float4*>(sXch);      // 2 KB; the second exchange follows behind the column sums
        if (tm.l3 == 0) {
          x4[tm.colhalf * 64 + tm.r0] = make_float4(ra[0], ra[1], ra[2], ra[3]);
          x4[tm.colhalf * 64 + tm.r1] = make_float4(rb[0], rb[1], rb[2], rb[3]);
        }
        named_bar_sync(1 + tm.quad, 64);
        {
          const float4 o0 = x4[(tm.colhalf ^ 1) * 64 + tm.r0], o1 = x4[(tm.colhalf ^ 1) * 64 + tm.r1];
          ra[0] += o0.x; ra[1] += o0.y; ra[2] += o0.z; ra[3] += o0.w;
          rb[0] += o1.x; rb[1] += o1.y; rb[2] += o1.z; rb[3] += o1.w;
        }
        f32x2 sa0 = 0ull, sa1 = 0ull, sb0 = 0ull, sb1 = 0ull;      // sum g_std, sum g_xhat of the two rows
        f32x2 cs[4];
        {
          const f32x2 n64 = pk1(-1.f / 64.f);
          const f32x2 mA = mul2(pk1(ra[1]), n64), xA = mul2(pk1(ra[2]), n64), mB = mul2(pk1(rb[1]), n64), xB = mul2(pk1(rb[2]), n64);
          const f32x2 fA3 = pk1(-ra[2] * rs0 * (1.f / 64.f)), fA4 = pk1(-ra[3] * rs0 * (1.f / 64.f));
          const f32x2 fB3 = pk1(-rb[2] * rs1 * (1.f / 64.f)), fB4 = pk1(-rb[3] * rs1 * (1.f / 64.f));
          f32x2 cl[4];
          TokFrag dv;
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const f32x2 gm = frag_col(tm, sGamma, q), neg = pk1(-1.f);
            const f32x2 x0 = bf16x2_to_f32x2(xhw[2 * q]), x1 = bf16x2_to_f32x2(xhw[2 * q + 1]);
            const f32x2 bt0 = mul2(add2(A2.a[q], fma2(x0, xA, mA)), pk1(rs0));
            const f32x2 bt1 = mul2(add2(A2.b[q], fma2(x1, xB, mB)), pk1(rs1));
            const f32x2 gl0 = mul2(gm, bt0), gl1 = mul2(gm, bt1);
            cs[q] = add2(fma2(go.a[q], bt0, mul2(gl0, x0)), fma2(go.b[q], bt1, mul2(gl1, x1)));
            cl[q] = add2(gl0, gl1);
            dv.a[q] = mul2(gl0, neg);
            dv.b[q] = mul2(gl1, neg);
            kpa[q] = fma2(t1.a[q], pk1(-eta0), gl0);
            kpb[q] = fma2(t1.b[q], pk1(-eta1), gl1);
            const f32x2 gx0 = fma2(gl0, gm, fma2(mul2(go.a[q], gm), fA3, mul2(A2.a[q], fA4)));
            const f32x2 gx1 = fma2(gl1, gm, fma2(mul2(go.b[q], gm), fB3, mul2(A2.b[q], fB4)));
            sa0 = fma2(gx0, x0, fma2(A2.a[q], bf16x2_to_f32x2(gzw[2 * q]), sa0));
            sb0 = fma2(gx1, x1, fma2(A2.b[q], bf16x2_to_f32x2(gzw[2 * q + 1]), sb0));
            sa1 = add2(sa1, gx0);
            sb1 = add2(sb1, gx1);
            A2.a[q] = gx0;
            A2.b[q] = gx1;
          }
          frag_st_tile(tm, t_go, dv);      // dV: stored by TMA
          dgam += frag_colsum(cs, lane);
          dbet += frag_colsum(cl, lane);
        }
        float sa[2] = {-hsum(sa0) * rs0, hsum(sa1)}, sb[2] = {-hsum(sb0) * rs1, hsum(sb1)};
        frag_allreduce2<0>(tm, sa, sb, sXch + 768, 1);
        {
          const f32x2 k0 = pk1(sa[0] * (1.f / 64.f)), l0 = pk1(-sa[1] * rs0 * (1.f / 64.f));
          const f32x2 k1 = pk1(sb[0] * (1.f / 64.f)), l1 = pk1(-sb[1] * rs1 * (1.f / 64.f));
          TokFrag u2;
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            A2.a[q] = fma2(A2.a[q], pk1(rs0), fma2(bf16x2_to_f32x2(xhw[2 * q]), k0, l0));      // gZ2in
            A2.b[q] = fma2(A2.b[q], pk1(rs1), fma2(bf16x2_to_f32x2(xhw[2 * q + 1]), k1, l1));
            cs[q] = add2(A2.a[q], A2.b[q]);
            u2.a[q] = mul2(bf16x2_to_f32x2(gzw[2 * q]), pk1(-eta0));                           // U2 = -eta gZ2
            u2.b[q] = mul2(bf16x2_to_f32x2(gzw[2 * q + 1]), pk1(-eta1));
          }
          frag_st_tile(tm, t_q, A2);
          frag_st_tile(tm, t_g, u2);
          put_colsum(cs);
        }
        if (tm.colhalf == 0 && tm.l3 == 0) {
          const int r0 = tm.r0, r1 = tm.r1;
          float p0 = 0.f, p1 = 0.f;
#pragma unroll
          for (int w = 0; w < 8; ++w) {
            p0 += sPart[w * 64 + r0];
            p1 += sPart[w * 64 + r1];
          }
          p.d_eta[(sid * NC + i0 + j) * 64 + r0] = __float2bfloat16(-(ra[0] + p0));
          p.d_eta[(sid * NC + i0 + j) * 64 + r1] = __float2bfloat16(-(rb[0] + p1));
        }
      }
      publish();
      // G11
      // + G_W2snap U2^T
      // G12
      if (tid == kProd) {
        tma_store_2d(&tmDV, t_go, 0, row0);
        tma_commit_group();
      }
      TTT_ISSUE(mma_hidden_half(tmem + TM_B, smem_u32(big(ib1)), smem_u32(t_q), false, false, 0); mma_hidden_half(tmem + TM_B, smem_u32(big(ib3)), smem_u32(t_g), false, true, 0),
                mma_hidden_half(tmem + TM_B, smem_u32(big(ib1)), smem_u32(t_q), false, false, 1); mma_hidden_half(tmem + TM_B, smem_u32(big(ib3)), smem_u32(t_g), false, true, 1),
                mma_hidden_half(tmem + TM_A, smem_u32(big(ib1)), smem_u32(t_gz2), false, false, 0),
                mma_hidden_half(tmem + TM_A, smem_u32(big(ib1)), smem_u32(t_gz2), false, false, 1))
      if (tid < 64) sGb2[tid] += quad_sum(tid);
      wait_mma();
      if (tid == kProd) {
        // the W2 state-gradient snapshot is consumed: X2 comes back into its buffer for G14 (it lands while
        // E5 runs); dV has left its tile, the d_gamma addends and x_hat_fused are consumed: the next step's
        // first tiles are requested now, two phases before they are needed
        load_big(ib3, p.sc_X2 + slot * BIG);
        tma_wait_group_read<0>();
        if (j > 0) issue_tiles_a(j - 1);
      }
      // ---- E5: gZ1in^T = gX2^T gelu'(Z1^T) + R^T S^T, in place over S^T
      {
        uint8_t* bs = big(ib2);
        const uint8_t* bgp = big(ib0);
        f32x2 bs2 = 0ull;
#pragma unroll
        for (int half = 0; half < 4; ++half) {   // 16 columns per pass
          uint32_t v[16], w[16];
          tmem_ld16(tmem + lane_base + TM_B + wg * 64 + half * 16, v);
          tmem_ld16(tmem + lane_base + TM_A + wg * 64 + half * 16, w);
          const uint4 gr[2] = {ld_chunk_raw(bgp, hrow, half * 2), ld_chunk_raw(bgp, hrow, half * 2 + 1)};
          const uint4 sr[2] = {ld_chunk_raw(bs, hrow, half * 2), ld_chunk_raw(bs, hrow, half * 2 + 1)};
          tmem_wait_ld();
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            const uint32_t gw[4] = {gr[c].x, gr[c].y, gr[c].z, gr[c].w};      // gelu'(Z1), f16
            const uint32_t sw[4] = {sr[c].x, sr[c].y, sr[c].z, sr[c].w};
            uint32_t o[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const f32x2 t = fma2(pk(v[c * 8 + 2 * k], v[c * 8 + 2 * k + 1]), f16x2_to_f32x2(gw[k]),
                                   mul2(pk(w[c * 8 + 2 * k], w[c * 8 + 2 * k + 1]), bf16x2_to_f32x2(sw[k])));
              bs2 = add2(bs2, t);
              o[k] = f32x2_to_bf16x2(t);
            }
            *reinterpret_cast<uint4*>(bs + sw128_off(hrow, half * 2 + c)) = make_uint4(o[0], o[1], o[2], o[3]);
          }
        }
        Gb1 += hsum(bs2);
      }
      publish();
      // gelu'(Z1) is consumed: the next step's gelu'(Z1_bar) comes into its buffer
      if (tid == kProd && j > 0) load_big(ib0, p.sc_Z1b + (slot - 1) * BIG);
      wait_bar(BAR_BIG + ib4);
      wait_bar(BAR_BIG + ib3);
      // G13 // G15 // G14
      TTT_ISSUE(mma_token_major(tmem + TM_A, smem_u32(big(ib2)), smem_u32(big(ib4))),
                mma_hidden_major(tmem + TM_S1, smem_u32(big(ib2)), smem_u32(t_k), true, true),
                mma_hidden_half(tmem + TM_S2, smem_u32(big(ib3)), smem_u32(t_q), true, true, 0),
                mma_hidden_half(tmem + TM_S2, smem_u32(big(ib3)), smem_u32(t_q), true, true, 1))
      wait_mma();
      // ---- E6: dK = partial + gZ1in W1^T, staged over the dl/dZ2 tile (dead since G12) and stored by TMA;
      // nothing waits for the store here: the tile's next load is issue_gz2's
      {
        TokFrag x;
        frag_ld(tm, tmem + TM_A, x);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          x.a[q] = add2(x.a[q], kpa[q]);
          x.b[q] = add2(x.b[q], kpb[q]);
        }
        frag_st_tile(tm, t_gz2, x);
      }
      publish();
      if (tid == kProd) {
        tma_store_2d(&tmDK, t_gz2, 0, row0);
        tma_commit_group();
      }
      // pre-update weights of this mini-batch are the post-update weights of the previous one
      {
        const int n0 = ib4, n1 = ib1, n2 = ib0, n3 = ib2, n4 = ib3;
        ib0 = n0; ib1 = n1; ib2 = n2; ib3 = n3; ib4 = n4;
      }
      if (tid == kProd && j > 0 && !*abort_flag) issue_rest(j - 1);
      if (*abort_flag) { aborted = true; break; }
    }
    if (aborted) break;
    if (tid == kProd) tma_wait_group_read<0>();   // the last dK has left its tile (the recompute writes it again)

    // ---- park the gradient state (tensor memory -> grad_L_W*_init); the last group leaves the result
    {
      __syncwarp();
#pragma unroll 1
      for (int half = 0; half < 2; ++half) {
        uint32_t v[32];
        tmem_ld32(tmem + lane_base + TM_S1 + wg * 64 + half * 32, v);
        tmem_wait_ld();
#pragma unroll
        for (int q = 0; q < 32; ++q) Gdst_W1[(half * 32 + q) * 256 + hrow] = __uint_as_float(v[q]);
        tmem_ld32(tmem + lane_base + TM_S2 + wg * 64 + half * 32, v);
        tmem_wait_ld();
        // whole lines through a staging area in the first two hidden-major buffers (nothing is in flight
        // into them at the end of a group)
        store_rows_coalesced(Gdst_W2 + (hrow - lane) * 64 + half * 32, 64, v, big(0) + warp * kRowStageBytes, lane);
      }
      Gsrc_W1 = Gdst_W1;
      Gsrc_W2 = Gdst_W2;
    }
    publish();
  }

  // ---- final vector outputs
  if (!aborted) {
    p.gb1[sid * 256 + hrow] = Gb1;
    sXch[tm.quad * 64 + frag_colsum_col(tm, lane)] = dgam;
    sXch[256 + tm.quad * 64 + frag_colsum_col(tm, lane)] = dbet;
    __syncthreads();
    if (tid < 64) {
      p.gb2[sid * 64 + tid] = sGb2[tid];
      p.d_gamma[sid * 64 + tid] = (sXch[tid] + sXch[64 + tid]) + (sXch[128 + tid] + sXch[192 + tid]);
      p.d_beta[sid * 64 + tid] = (sXch[256 + tid] + sXch[320 + tid]) + (sXch[384 + tid] + sXch[448 + tid]);
    }
  }
  if (tid == kProd) tma_wait_group<0>();
  if (aborted) {
    // everything this CTA still has in flight is waited for (bounded, not cut short by the abort flag)
    // before its shared and tensor memory go away: the tensor-core work of the four issuers ...
    if (warp < 4) {
      if (elect_one()) umma_commit(&bars[BAR_DRAIN]);
      __syncwarp();
    }
    if (tid == kProd) {
      mbar_wait_bounded(&bars[BAR_DRAIN], 0, never_flag, limit);
      // ... and its own loads
      for (int b = 0; b < 16; ++b)
        if (pending & (1u << b)) mbar_wait_bounded(&bars[b], (ph >> b) & 1u, never_flag, limit);
      atomicExch(p.status, static_cast<uint32_t>(TTT_B200_ERR_TIMEOUT));
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, TM_COLS);
}

}  // namespace

// The first `streams` of the call's streams.
int ttt_launch_backward(const ttt_b200_bwd_args* a, int streams, cudaStream_t stream, uint32_t* status, uint64_t limit_ns,
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
  p.sc_W1 = reinterpret_cast<uint8_t*>(a->W1_init_group);
  p.sc_W2 = reinterpret_cast<uint8_t*>(a->W2_init_group);
  p.w_stride = 65536;
  p.sc_Z1 = static_cast<uint8_t*>(a->Z1_group);
  p.sc_X2 = static_cast<uint8_t*>(a->X2_group);
  p.sc_gZ1 = static_cast<uint8_t*>(a->grad_l_wrt_Z1_group);
  p.sc_Z1b = static_cast<uint8_t*>(a->Z1_bar_group);
  p.sc_X2b = static_cast<uint8_t*>(a->X2_bar_group);
  p.sc_xhf = static_cast<uint8_t*>(a->x_hat_fused_group);
  p.sc_gof = static_cast<uint8_t*>(a->grad_output_fused_group);
  p.sc_gZ2 = static_cast<uint8_t*>(a->grad_l_wrt_Z2_group);
  p.sc_xhln = static_cast<uint8_t*>(a->x_hat_ln_group);
  p.sc_sigf = a->std_fused_group;
  p.sc_sigln = a->std_ln_group;
  p.gW1_last = a->grad_L_W1_last; p.gb1_last = a->grad_L_b1_last;
  p.gW2_last = a->grad_L_W2_last; p.gb2_last = a->grad_L_b2_last;
  p.d_gamma = a->grad_L_ttt_norm_weight; p.d_beta = a->grad_L_ttt_norm_bias;
  p.gW1 = a->grad_L_W1_init; p.gb1 = a->grad_L_b1_init; p.gW2 = a->grad_L_W2_init; p.gb2 = a->grad_L_b2_init;
  p.d_eta = static_cast<__nv_bfloat16*>(a->grad_L_last_eta);
  p.dXQ = static_cast<uint8_t*>(a->grad_L_XQ);
  p.dXK = static_cast<uint8_t*>(a->grad_L_XK);
  p.dXV = static_cast<uint8_t*>(a->grad_L_XV);
  p.H = a->H; p.NC = a->NC; p.cgs = a->checkpoint_group_size; p.nck = a->num_checkpoints;
  p.drop_load = drop_load;
  p.status = status;
  p.wait_limit_ns = limit_ns;
  static std::once_flag once[64];
  static cudaError_t attr_err[64];
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return ttt_set_error(TTT_B200_ERR_LAUNCH, "device index out of range");
  std::call_once(once[dev], [&] {
    attr_err[dev] = cudaFuncSetAttribute(ttt_bwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
  });
  if (attr_err[dev] != cudaSuccess) return ttt_set_error(TTT_B200_ERR_LAUNCH, cudaGetErrorString(attr_err[dev]));
  ttt_bwd_kernel<<<dim3(streams), dim3(kThreads), SMEM_BYTES, stream>>>(tmQ, tmK, tmV, tmGo, tmDQ, tmDK, tmDV, p);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return ttt_set_error(TTT_B200_ERR_LAUNCH, cudaGetErrorString(e));
  return TTT_B200_OK;
}

// =============================================================================================
// Backward entry point that allocates no device memory.
//
// Some hosts of this library cannot let it call cudaMalloc (or hand it freshly allocated
// scratch): inference servers and training loops that pre-commit all of HBM to their own
// pools at start-up, so a later allocation fails or fragments the pool; and latency-critical
// loops for which the implicit device synchronisation of an allocation is not acceptable.
// For them the per-mini-batch scratch of the backward lives in the fixed array below instead
// of the caller's sixteen `*_group` tensors.  The array is part of the library image: every
// GPU on which the library's kernels are loaded holds it until the process exits.
//
// Capacity: B * H * checkpoint_group_size <= TTT_B200_NOALLOC_MAX_SLOTS scratch slots of
// 262 656 bytes (about 32 MiB in total).  Larger problems are rejected with code 1.
//
// All calls on a device share the array.  Nothing in it has to start at zero (each slot is
// written before it is read within one call) and it keeps the previous call's contents; two
// calls that overlap on the GPU (different streams) race on it and must be serialised by the
// caller.  The first call on each device looks up the array's device address (the name of a
// __device__ array is only a host-side handle in host code), raises the kernel's shared-memory
// limit and resolves the tensor-map encoder; make that first call outside any stream capture.
namespace {

constexpr size_t NA_SLOTS = TTT_B200_NOALLOC_MAX_SLOTS;
constexpr size_t NA_OFF_W1 = 0;
constexpr size_t NA_OFF_W2 = NA_OFF_W1 + NA_SLOTS * BIG;
constexpr size_t NA_OFF_Z1 = NA_OFF_W2 + NA_SLOTS * BIG;
constexpr size_t NA_OFF_X2 = NA_OFF_Z1 + NA_SLOTS * BIG;
constexpr size_t NA_OFF_GZ1 = NA_OFF_X2 + NA_SLOTS * BIG;
constexpr size_t NA_OFF_Z1B = NA_OFF_GZ1 + NA_SLOTS * BIG;
constexpr size_t NA_OFF_X2B = NA_OFF_Z1B + NA_SLOTS * BIG;
constexpr size_t NA_OFF_XHF = NA_OFF_X2B + NA_SLOTS * BIG;
constexpr size_t NA_OFF_GOF = NA_OFF_XHF + NA_SLOTS * TILE;
constexpr size_t NA_OFF_GZ2 = NA_OFF_GOF + NA_SLOTS * TILE;
constexpr size_t NA_OFF_XHLN = NA_OFF_GZ2 + NA_SLOTS * TILE;
constexpr size_t NA_OFF_SIGF = NA_OFF_XHLN + NA_SLOTS * TILE;
constexpr size_t NA_OFF_SIGLN = NA_OFF_SIGF + NA_SLOTS * 256;
constexpr size_t NA_BYTES = NA_OFF_SIGLN + NA_SLOTS * 256;
static_assert(NA_BYTES == NA_SLOTS * 262656, "scratch slot size changed: update the header comment");

static __device__ __align__(256) unsigned char g_noalloc_scratch[NA_BYTES];
static __device__ __align__(16) uint32_t g_noalloc_status;

struct NoAllocDevice {
  uint8_t* scratch = nullptr;
  uint32_t* status = nullptr;
  bool ready = false;
};
NoAllocDevice g_noalloc_dev[64];

// Once per device, with that device current: device addresses of the two symbols.
int noalloc_setup(int dev) {
  NoAllocDevice& d = g_noalloc_dev[dev];
  if (d.ready) return TTT_B200_OK;
  void* ptr = nullptr;
  cudaError_t e = cudaGetSymbolAddress(&ptr, g_noalloc_scratch);
  if (e != cudaSuccess || ptr == nullptr)
    return ttt_set_error(TTT_B200_ERR_LAUNCH, e != cudaSuccess ? cudaGetErrorString(e) : "scratch symbol has no address");
  d.scratch = static_cast<uint8_t*>(ptr);
  e = cudaGetSymbolAddress(&ptr, g_noalloc_status);
  if (e != cudaSuccess || ptr == nullptr)
    return ttt_set_error(TTT_B200_ERR_LAUNCH, e != cudaSuccess ? cudaGetErrorString(e) : "status symbol has no address");
  d.status = static_cast<uint32_t*>(ptr);
  e = cudaFuncSetAttribute(ttt_bwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
  if (e != cudaSuccess) return ttt_set_error(TTT_B200_ERR_LAUNCH, cudaGetErrorString(e));
  d.ready = true;
  return TTT_B200_OK;
}

}  // namespace

extern "C" int ttt_b200_backward_noalloc(const ttt_b200_bwd_noalloc_args* a, void* stream_) {
  if (a == nullptr) return ttt_set_error(TTT_B200_ERR_BAD_ARGS, "args is NULL");
  if (a->B < 1 || a->H < 1 || a->NC < 1 || a->checkpoint_group_size < 1)
    return ttt_set_error(TTT_B200_ERR_BAD_ARGS, "B, H, NC and checkpoint_group_size must be >= 1");
  if (a->num_checkpoints != (a->NC + a->checkpoint_group_size - 1) / a->checkpoint_group_size)
    return ttt_set_error(TTT_B200_ERR_BAD_ARGS,
                         "checkpoint tensors must hold ceil(NC / checkpoint_group_size) states");
  if (static_cast<uint64_t>(a->B) * a->H * a->NC * 64 >= (1ull << 31))
    return ttt_set_error(TTT_B200_ERR_BAD_ARGS, "B*H*NC*64 must be below 2^31");
  const uint64_t slots = static_cast<uint64_t>(a->B) * a->H * a->checkpoint_group_size;
  if (slots > NA_SLOTS)
    return ttt_set_error(TTT_B200_ERR_BAD_ARGS,
                         "B*H*checkpoint_group_size exceeds TTT_B200_NOALLOC_MAX_SLOTS (the built-in scratch); "
                         "use ttt_b200_backward with caller-provided scratch");
  const void* ptrs[] = {a->XQ, a->XK, a->XV, a->last_eta, a->ttt_norm_weight, a->ttt_norm_bias,
                        a->W1_checkpoints, a->b1_checkpoints, a->W2_checkpoints, a->b2_checkpoints,
                        a->grad_L_W1_last, a->grad_L_b1_last, a->grad_L_W2_last, a->grad_L_b2_last,
                        a->grad_L_XQW_mini_batch, a->grad_L_ttt_norm_weight, a->grad_L_ttt_norm_bias,
                        a->grad_L_W1_init, a->grad_L_b1_init, a->grad_L_W2_init, a->grad_L_b2_init,
                        a->grad_L_last_eta, a->grad_L_XQ, a->grad_L_XK, a->grad_L_XV};
  for (const void* q : ptrs) {
    if (q == nullptr) return ttt_set_error(TTT_B200_ERR_BAD_ARGS, "a required tensor pointer is NULL");
    if (reinterpret_cast<uintptr_t>(q) & 15u)
      return ttt_set_error(TTT_B200_ERR_BAD_ARGS, "tensor pointers must be 16-byte aligned");
  }
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return ttt_set_error(TTT_B200_ERR_LAUNCH, cudaGetErrorString(e));
  if (dev < 0 || dev >= 64) return ttt_set_error(TTT_B200_ERR_LAUNCH, "device index out of range");
  static std::mutex mu;
  {
    std::lock_guard<std::mutex> lk(mu);
    if (int rc = noalloc_setup(dev)) return rc;
  }
  const NoAllocDevice& d = g_noalloc_dev[dev];
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);

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
  p.sc_W1 = d.scratch + NA_OFF_W1;
  p.sc_W2 = d.scratch + NA_OFF_W2;
  p.w_stride = BIG;
  p.sc_Z1 = d.scratch + NA_OFF_Z1;
  p.sc_X2 = d.scratch + NA_OFF_X2;
  p.sc_gZ1 = d.scratch + NA_OFF_GZ1;
  p.sc_Z1b = d.scratch + NA_OFF_Z1B;
  p.sc_X2b = d.scratch + NA_OFF_X2B;
  p.sc_xhf = d.scratch + NA_OFF_XHF;
  p.sc_gof = d.scratch + NA_OFF_GOF;
  p.sc_gZ2 = d.scratch + NA_OFF_GZ2;
  p.sc_xhln = d.scratch + NA_OFF_XHLN;
  p.sc_sigf = reinterpret_cast<float*>(d.scratch + NA_OFF_SIGF);
  p.sc_sigln = reinterpret_cast<float*>(d.scratch + NA_OFF_SIGLN);
  p.gW1_last = a->grad_L_W1_last; p.gb1_last = a->grad_L_b1_last;
  p.gW2_last = a->grad_L_W2_last; p.gb2_last = a->grad_L_b2_last;
  p.d_gamma = a->grad_L_ttt_norm_weight; p.d_beta = a->grad_L_ttt_norm_bias;
  p.gW1 = a->grad_L_W1_init; p.gb1 = a->grad_L_b1_init; p.gW2 = a->grad_L_W2_init; p.gb2 = a->grad_L_b2_init;
  p.d_eta = static_cast<__nv_bfloat16*>(a->grad_L_last_eta);
  p.dXQ = static_cast<uint8_t*>(a->grad_L_XQ);
  p.dXK = static_cast<uint8_t*>(a->grad_L_XK);
  p.dXV = static_cast<uint8_t*>(a->grad_L_XV);
  p.H = a->H; p.NC = a->NC; p.cgs = a->checkpoint_group_size; p.nck = a->num_checkpoints;
  p.drop_load = -1;
  // The status word of this entry point is a device word that no launch clears: a kernel that gives up
  // on a bounded wait sets it, and it stays set until a synchronising call or ttt_b200_take_status()
  // reads and clears it (both without allocating anything).
  p.status = d.status;
  p.wait_limit_ns = ttt_wait_limit_ns();
  ttt_bwd_kernel<<<dim3(a->B * a->H), dim3(kThreads), SMEM_BYTES, stream>>>(tmQ, tmK, tmV, tmGo, tmDQ, tmDK, tmDV, p);
  e = cudaGetLastError();
  if (e != cudaSuccess) return ttt_set_error(TTT_B200_ERR_LAUNCH, cudaGetErrorString(e));
  if (a->flags & TTT_B200_FLAG_SYNC) {
    uint32_t st = 0;
    e = cudaMemcpyAsync(&st, d.status, sizeof(uint32_t), cudaMemcpyDeviceToHost, stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
    if (e != cudaSuccess) return ttt_set_error(TTT_B200_ERR_LAUNCH, cudaGetErrorString(e));
    if (st != 0) {
      cudaMemsetAsync(d.status, 0, sizeof(uint32_t), stream);
      cudaStreamSynchronize(stream);
      return ttt_set_error(TTT_B200_ERR_TIMEOUT, "a device-side bounded wait ran out; results are invalid");
    }
  }
  return TTT_B200_OK;
}

// Read and clear the status word of ttt_b200_backward_noalloc on every device it has run on (plain
// synchronous copies from / to the symbol: nothing is allocated).  Called after the caller has
// synchronised, by ttt_b200_take_status().
uint32_t ttt_noalloc_take_status() {
  uint32_t any = 0;
  int cur = 0;
  if (cudaGetDevice(&cur) != cudaSuccess) return 0;
  for (int dev = 0; dev < 64; ++dev) {
    if (!g_noalloc_dev[dev].ready) continue;
    if (cudaSetDevice(dev) != cudaSuccess) continue;
    uint32_t st = 0;
    if (cudaMemcpyFromSymbol(&st, g_noalloc_status, sizeof(st)) == cudaSuccess && st != 0) {
      any = st;
      const uint32_t zero = 0;
      cudaMemcpyToSymbol(g_noalloc_status, &zero, sizeof(zero));
    }
  }
  cudaSetDevice(cur);
  return any;
}
