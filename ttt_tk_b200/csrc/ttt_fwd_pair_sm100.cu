// TTT-MLP forward for sm_100a with two CTAs per (batch, head) stream: one runs the chain, the other the output pass.
//
// Like ttt_fwd_sm100.cu it replaces the reference's fwd_ttt_mlp_ker (kernels/ttt/ttt.cu:85-586); the per-mini-batch math is
// that of kernels/ttt/matching.py:30-125.  Layouts are that kernel's: every 64x256 / 256x64 quantity "hidden-major"
// (hidden unit = TMEM lane), every 64x64 quantity token-major (M = 64).
//
// There the chain (what the next mini-batch waits for) and the output pass share one SM's issue slots, MUFU and tensor
// pipe; here each has an SM of its own:
//
//   chain CTA                                            output CTA
//   MMA1  Z1^T = W1^T K^T                                (X2, U1, U2 there:)
//   EPI1  X2^T = gelu(Z1^T + b1), G' = gelu'(.)          MMA4  W1^T += U1^T K ;  W2 += X2^T U2, on a state of its own
//   MMA2  Z2 = X2 W2                                     COPY  bf16 copies of W1^T and W2; b1, b2; checkpoints
//   LN    U2 = -eta dl/dZ2                               MMA5  Z1b^T = W1^T Q^T
//   MMA3  R^T = W2 U2^T;  W2 += X2^T U2                  EPI5  X2b^T = gelu(Z1b^T + b1)
//   EPI3  U1^T = R^T G'                                  MMA6  Z2b = X2b W2
//   MMA4  W1^T += U1^T K                                 OUT   Q + gamma LN(Z2b + b2) + beta -> TMA store
//   EPI4  bf16 copies of the new W1^T and W2;  b1, b2
//
// Both CTAs hold the fp32 state, and update it with the same products of the same bf16 operands, so only those operands
// cross the SM-to-SM network: 75 KB a mini-batch as bulk copies between the CTAs' shared memories (measured 21 bytes a clock,
// 3500 of the chain's 6900 cycles, beside everything else), and the fp32 state never leaves its SM but as a checkpoint, which
// the output CTA writes while the chain goes on.  X2, which the chain has first, has two buffers there, the rest one.
//
// Sixteen epilogue warps per CTA (32 columns of a 256-row matrix each; the 64 x 64 tiles are the first eight warps') and four
// helper warps, which issue the MMAs and the copies and wait for both.  Hand-overs are mbarriers, each completed once per
// mini-batch (CA three times), waited for at every completion; tests/test_forward_pair_order_cpu.py derives the order of all
// accesses from this source.  Every wait is bounded.
//
// What bounds it: the chain.  Of its 6900 cycles, EPI1 has 1800 (the fp32 pipe alone needs 1150, the MUFU 1000), the LayerNorm
// with its two exchanges 1250, the four products with their hand-overs 2800.  us per mini-batch, against one CTA per stream and
// against four with a quarter of the hidden units each: 48 streams x 32 in groups of 4 4.75 -> 4.3, 32 x 128 in groups of 16
// 4.2 / 4.19 -> 3.73, 4 x 32 in groups of 4 4.65 / 4.36 -> 4.05.  A checkpoint takes the output CTA 4900 cycles (132 KB at 27
// bytes a clock), of which the chain has to wait for about 2500.  Steps on the way, 32 x 128: 4.31 with everything in sixteen
// warps, 4.12 with the LayerNorm in eight and X2 in two buffers, 3.84 with two streams to a cluster, 3.82 with W2's copy beside
// MMA4 and all that needs no Z2 before its wait.  Not kept: G' in a pass of its own under MMA2 (that window is full: 3.94),
// polling with test_wait (it takes issue slots: 4.0), waits with a long suspend hint (3.90).
#include <mutex>

#define TTT_WAIT_INLINE
#include "ttt_cluster.cuh"
#include "ttt_internal.h"

using namespace tttcl;

namespace {

constexpr int kEpi = 512;                    // epilogue threads
constexpr int kThreads = kEpi + 128;         // and four helper warps
// registers per thread: the block is launched with 96 of them
constexpr int kRegsEpi = 104, kRegsHelp = 64;
static_assert(kRegsEpi * kEpi + kRegsHelp * 128 <= 96 * kThreads, "the shares add up to the block's registers at launch");
constexpr uint32_t kBarPair = 1, kBarEpi = 5;      // named barriers: the two warps of a quadrant that work on 64 x 64 tiles; all epilogue warps

// ---- shared memory.  X2, U1, U2 and the vectors have the same offsets in both CTAs: they are copied from one to the other.
constexpr uint32_t OFF_X2 = 0;                          // + parity of the mini-batch
constexpr uint32_t OFF_U1 = 2 * BIG;
constexpr uint32_t OFF_U2 = 3 * BIG;
constexpr uint32_t OFF_W2 = OFF_U2 + TILE;              // bf16 operand copy
constexpr uint32_t OFF_K = OFF_W2 + BIG;                // + stage
constexpr uint32_t OFF_V = OFF_K + 2 * TILE;            // chain: + stage
constexpr uint32_t OFF_Q = OFF_K + 2 * TILE;            // output: + stage; Q, then Out on its way to global memory
constexpr uint32_t OFF_X2B = OFF_Q + 2 * TILE;          // output; also 4 KB for each of eight warps, W2 checkpoints on their way out
constexpr uint32_t OFF_SUM = OFF_X2B + BIG;             // fp32[2][256] row sums of U1 per column half, fp32[4][64] column sums of U2 per quadrant
constexpr uint32_t SUM_BYTES = 2048 + 1024;
constexpr uint32_t OFF_ETA = OFF_SUM + SUM_BYTES;       // bf16[2][64]
constexpr uint32_t OFF_GAMMA = OFF_ETA + 256;
constexpr uint32_t OFF_BETA = OFF_GAMMA + 256;
constexpr uint32_t OFF_XCH = OFF_BETA + 256;            // row-sum exchanges
constexpr uint32_t OFF_BAR = OFF_XCH + kXchBytes;
constexpr uint32_t OFF_MISC = OFF_BAR + 320;
constexpr uint32_t SMEM_BYTES = OFF_MISC + 64;
static_assert(SMEM_BYTES <= 232448, "exceeds the 227 KB per-CTA shared memory of sm_100");

// ---- barriers
enum : int {
  // chain: loads (+ stage); products: MMA1, MMA3, MMA4 (per 128-row block), MMA2, W2 update
  CK, CK1, CV, CV1, CA, CA1, CZ, CW2,
  // chain epilogues done: EPI1 (+ parity of the mini-batch), LN, EPI3 and EPI4 (per block), U1 in shared memory, W2 copy
  E_1, E_11, E_2, E_3, E_31, E_4, E_41, E_U, E_W2,
  // output: loads (+ stage); products: MMA4, MMA5, MMA6
  OKT, OKT1, OQ, OQ1, OUPD, OB, OZ,
  // output epilogues done: bf16 copies, state read, EPI5, Out (+ stage)
  E_C, E_R, E_5, E_OUT, E_OUT1,
  // completed from the other CTA.  Chain: what was sent has arrived there, has been used; output: X2 (+ parity of the
  // mini-batch), the rest
  U_SENT, X_FREE, OX, OX1, OU,
  BDRAIN,      // abort path only
  kBars
};
static_assert(U_SENT <= 32 && BDRAIN <= 64 && kBars * 8 <= 320, "parity masks, barrier storage");

// tensor-memory columns: two 128-lane blocks of 64 fp32 (32 bf16-pair) columns per 256-row matrix
constexpr uint32_t TM_W1 = 0;
constexpr uint32_t TM_W2 = 128;
constexpr uint32_t TM_A = 256;       // chain: Z1; Z2 in its first 64 columns; R.  Output: Z1b
constexpr uint32_t TM_W1B = 384;     // bf16 operand copy of W1^T
constexpr uint32_t TM_U1 = 448;      // chain: U1 (bf16)
constexpr uint32_t TM_ZB = 448;      // output: Z2b
constexpr uint32_t TM_COLS = 512;

struct FwdParams {
  const __nv_bfloat16* eta;
  const float* gamma;
  const float* beta;
  const float* W1; const float* b1; const float* W2; const float* b2;
  float* W1c; float* b1c; float* W2c; float* b2c;
  float* W1f; float* b1f; float* W2f; float* b2f;
  int H, NC, cgs, nck;
  int streams;
  int drop_load;            // test only: mini-batch whose loads stream 0 never issues (-1: none)
  uint32_t* status;
  uint64_t wait_limit_ns;
};

// Streams to a cluster, whose first CTAs are the chains and whose others the output passes: the SMs of a TPC, which share an
// instruction cache, then run the same program (48 streams x 32: 176 -> 141 us; with a stream to a cluster 74 would run at
// once, but at 5.2 us per mini-batch against 4.3 with one CTA each).
constexpr int kStreams = 2;

__global__ void __launch_bounds__(kThreads, 1)
ttt_fwd_pair_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                    const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmOut,
                    const FwdParams p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  if (smem_u32(smem) & 1023u) {       // the swizzled tiles need it; never seen
    if (threadIdx.x == 0) atomicExch(p.status, static_cast<uint32_t>(TTT_B200_ERR_LAUNCH));
    return;
  }
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);   // same value, known to be warp-uniform
  const uint32_t crank = cluster_ctarank();
  const bool chain = crank < kStreams;
  const uint32_t peer = chain ? crank + kStreams : crank - kStreams;
  const long sid = (blockIdx.x / (2 * kStreams)) * kStreams + (crank % kStreams);
  const bool idle = sid >= p.streams;      // the last cluster's second stream, if there is none: it only keeps step
  const int head = static_cast<int>(sid % p.H);
  const int NC = idle ? 0 : p.NC;

  float* sGamma = reinterpret_cast<float*>(smem + OFF_GAMMA);
  float* sBeta = reinterpret_cast<float*>(smem + OFF_BETA);
  float* sRow = reinterpret_cast<float*>(smem + OFF_SUM);             // [2][256]
  float* sCol = reinterpret_cast<float*>(smem + OFF_SUM + 2048);      // [4][64]
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + OFF_BAR);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + OFF_MISC);
  volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(smem + OFF_MISC + 4);
  volatile uint32_t* never_flag = reinterpret_cast<volatile uint32_t*>(smem + OFF_MISC + 8);   // stays 0
  const uint64_t limit = p.wait_limit_ns;

  if (tid == kEpi) {
    for (int i = 0; i < kBars; ++i)
      mbar_init(&bars[i], i == E_1 || i == E_11 || i == E_U || (i >= E_C && i <= E_5) ? 16
                          : (i >= E_2 && i <= E_41) || i == E_W2 || i == E_OUT || i == E_OUT1 ? 8 : i == CW2 || i == BDRAIN ? 2 : 1);
    fence_mbar_init();
    *abort_flag = 0;
    *never_flag = 0;
    prefetch_tmap(&tmQ);
    prefetch_tmap(&tmK);
    prefetch_tmap(&tmV);
    prefetch_tmap(&tmOut);
  }
  if (warp == 0) {
    tmem_alloc(tmem_slot, TM_COLS);
    tmem_relinquish();
  }
  griddep_launch();
  griddep_wait();
  if (tid < 64) {
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
  uint64_t ph = 0;      // expected parity per barrier
  auto bounded = [&](int b, uint32_t parity) -> bool {
    uint64_t t0 = 0;
    uint32_t spins = 0;
    while (!(b >= U_SENT ? mbar_try_wait_cluster(&bars[b], parity) : mbar_try_wait(&bars[b], parity))) {
      if (warp < 16) {      // (whatever holds an epilogue warp up holds a helper warp up that waits for it: the clock is theirs)
        if (*abort_flag) return false;
        continue;
      }
      if (++spins & 31u) continue;
      if (*abort_flag) return false;
      const uint64_t t = globaltimer_ns();
      if (t0 == 0) t0 = t;
      if (t - t0 > limit) {
        *abort_flag = 1;      // (the peer is told when this CTA has left its loops)
        return false;
      }
    }
    return true;
  };
  auto wait = [&](int b) -> bool {
    if (!bounded(b, static_cast<uint32_t>(ph >> b) & 1u)) return false;
    ph ^= 1ull << b;
    return true;
  };
  auto wait_mma = [&](int b) {      // a product's completion, by the warps that read its accumulator
    wait(b);
    __syncwarp();
    tc_fence_after_sync();
  };
  auto seen = [&](int b) -> bool {      // by a whole helper warp, which goes on or leaves as one
    const bool ok = __all_sync(0xffffffffu, wait(b));
    tc_fence_after_sync();
    return ok;
  };
  auto done = [&](int b) {          // this warp's share of an epilogue: its writes and tensor-memory reads are over
    fence_proxy_async_smem();
    tc_fence_before_sync();
    __syncwarp();
    if (lane == 0) mbar_arrive(&bars[b]);
  };
  auto done_tmem = [&](int b) {     // the same where no shared memory was written that a product or a copy reads
    tc_fence_before_sync();
    __syncwarp();
    if (lane == 0) mbar_arrive(&bars[b]);
  };
  auto token = [&](uint32_t d, uint32_t x, uint32_t w) {      // mma_token_lead, rolled by four
    constexpr uint32_t idesc = umma_idesc_bf16(64, 64, true, true, false);
    uint32_t a = desc_lo(x, BIG), b = desc_lo(w, BIG);
#pragma unroll 1
    for (uint32_t k = 0; k < 16; k += 4) {
#pragma unroll
      for (uint32_t i = 0; i < 4; ++i)
        mma_lead_rt(d, a + i * (2048u >> 4), b + i * (2048u >> 4), idesc, k | i, lead);
      a += 4 * (2048u >> 4);
      b += 4 * (2048u >> 4);
    }
  };
  auto commit = [&](int b) { if (lead) umma_commit(&bars[b]); };
  // loads issued so far (by lane 0 of a helper warp), for the abort path: parity of each barrier's next load, and whether there was one
  uint32_t ldp = 0, lda = 0;
  auto arm = [&](int b, uint32_t bytes) {
    mbar_expect_tx(&bars[b], bytes);
    ldp ^= 1u << b;
    lda |= 1u << b;
  };
  auto row_of = [&](int i) { return static_cast<int>((sid * NC + i) * 64); };
  auto dropped = [&](int i) { return i == p.drop_load && sid == 0; };
  auto load_tile = [&](int i, const CUtensorMap* map, uint32_t off, int bar) {
    if (i < NC && !dropped(i)) {
      const int s = i & 1;
      arm(bar + s, TILE);
      tma_load_2d(smem + off + s * TILE, map, &bars[bar + s], 0, row_of(i));
    }
  };

  const int quad = warp & 3, cq = (warp >> 2) & 3;           // 128-row block and column half of the hidden-major matrices
  const int blk = cq & 1, ch = cq >> 1;
  const int hrow = blk * 128 + quad * 32 + lane;
  const uint32_t lane_base = static_cast<uint32_t>(quad * 32) << 16;
  const uint32_t hl = lane_base + blk * 64 + ch * 32;        // this thread's lanes and columns of a 256-row matrix
  const TokMap tm(warp & 7, lane);                           // 64 x 64 tiles are the first eight warps'
  const bool tok = warp < 8;
  const long st_w = sid * (64 * 256);
  float* xch = reinterpret_cast<float*>(smem + OFF_XCH);

  if (warp < 16) {
    reg_take<kRegsEpi>();
    // ---- the initial state into tensor memory; the output CTA also writes it as checkpoint 0
    const long st = idle ? 0 : sid;
    float b1v = p.b1[st * 256 + hrow];
    f32x2 b2r[4];             // this thread's columns of b2
#pragma unroll
    for (int j = 0; j < 4; ++j) b2r[j] = *reinterpret_cast<const f32x2*>(p.b2 + st * 64 + tm.col(j));
    // b1 += row sums of U1, b2 += column sums of U2
    auto add_sums = [&]() {
      b1v += sRow[hrow] + sRow[256 + hrow];
      if (tok) {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          b2r[j] = add2(b2r[j], add2(add2(frag_col(tm, sCol, j), frag_col(tm, sCol + 64, j)),
                                     add2(frag_col(tm, sCol + 128, j), frag_col(tm, sCol + 192, j))));
      }
    };
    if (!idle) {
      const float* W1g = p.W1 + st_w + hrow;
      const float4* W2g = reinterpret_cast<const float4*>(p.W2 + st_w + hrow * 64 + ch * 32);
      uint32_t v[32];
      float4 q4[8];             // (both matrices' loads go out before either is used: one memory round trip, not two)
#pragma unroll
      for (int j = 0; j < 32; ++j) v[j] = __float_as_uint(W1g[(ch * 32 + j) * 256]);
#pragma unroll
      for (int j = 0; j < 8; ++j) q4[j] = W2g[j];
      tmem_st32(tmem + TM_W1 + hl, v);
      if (chain) {
        st_cols32_tmem(tmem + lane_base + TM_W1B + blk * 32 + ch * 16, v);
      } else {
        float* W1k = p.W1c + sid * p.nck * (64 * 256) + hrow;
#pragma unroll
        for (int j = 0; j < 32; ++j) W1k[(ch * 32 + j) * 256] = __uint_as_float(v[j]);
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        v[4 * j] = __float_as_uint(q4[j].x); v[4 * j + 1] = __float_as_uint(q4[j].y);
        v[4 * j + 2] = __float_as_uint(q4[j].z); v[4 * j + 3] = __float_as_uint(q4[j].w);
      }
      tmem_st32(tmem + TM_W2 + hl, v);
      if (chain) {
        st_cols32(smem + OFF_W2, hrow, ch, v);
        tmem_wait_st();
        fence_proxy_async_smem();
        tc_fence_before_sync();
        named_bar_sync(kBarEpi, kEpi);
        if (lane == 0) mbar_arrive(&bars[E_4 + blk]);
        if (lane == 0 && ch == 1) mbar_arrive(&bars[E_W2]);
      } else {
        // (through X2b and the bf16 W2, which nothing uses yet)
        store_rows_own(p.W2c + sid * p.nck * (64 * 256) + (hrow - lane) * 64 + ch * 32, v,
                       smem + (tok ? OFF_X2B : OFF_W2) + (warp & 7) * 4096, lane);
        if (ch == 0) p.b1c[sid * p.nck * 256 + hrow] = b1v;
        if (tid < 64) p.b2c[sid * p.nck * 64 + tid] = p.b2[sid * 64 + tid];
        tmem_wait_st();
        done(E_R);
      }
    }

    if (chain) {
      // ================================================================================== the chain
      for (int it = 0; it < NC; ++it) {
        const int s = it & 1;
        const __nv_bfloat16* eta = reinterpret_cast<const __nv_bfloat16*>(smem + OFF_ETA) + s * 64;
        // ---- EPI1: X2^T = gelu(Z1^T + b1) -> smem; G' = gelu'(Z1^T + b1) stays in registers (the thread that needs it in
        // EPI3 is this one)
        uint8_t* sX2 = smem + OFF_X2 + s * BIG;
        wait_mma(CA + blk);
        // (rolled, like every pass over columns here: the two programs' instructions have to be fetched once per mini-batch and
        // SM pair; the values kept for later move down a register half per turn)
        uint32_t gp[16];
        {
          const f32x2 bb = pk1(b1v);
#pragma unroll 1
          for (int q = 0; q < 2; ++q) {
            uint32_t v[16], g[8];
            tmem_ld16(tmem + TM_A + hl + q * 16, v);
#pragma unroll
            for (int k = 0; k < 8; ++k) gp[k] = gp[8 + k];
            tmem_wait_ld();
#pragma unroll
            for (int k = 0; k < 8; ++k) {
              f32x2 x, y;
              gelu_pair2(add2(pk(v[2 * k], v[2 * k + 1]), bb), x, y);
              g[k] = f32x2_to_bf16x2(x);
              gp[8 + k] = f32x2_to_bf16x2(y);
            }
            *reinterpret_cast<uint4*>(sX2 + sw128_off(hrow, ch * 4 + q * 2)) = make_uint4(g[0], g[1], g[2], g[3]);
            *reinterpret_cast<uint4*>(sX2 + sw128_off(hrow, ch * 4 + q * 2 + 1)) = make_uint4(g[4], g[5], g[6], g[7]);
          }
        }
        done(E_1 + s);

        // ---- LN: fused LayerNorm + L2 gradient, U2 = -eta * dl/dZ2 (eight warps, 16 values a thread: with sixteen warps the
        // exchanges and addresses, which do not shrink, took 1800 cycles instead of 1300)
        if (tok) {
          wait(CK + s);
          wait(CV + s);
          // what needs no Z2 comes before the wait: gamma^2 x_hat + gamma (beta + K - V) is the gradient's first factor
          f32x2 g2[4], ga[4], gb[4];
          {
            uint32_t kk[8], vv[8];
            frag_ld_raw(tm, smem + OFF_K + s * TILE, kk);
            frag_ld_raw(tm, smem + OFF_V + s * TILE, vv);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const f32x2 gam = frag_col(tm, sGamma, j), bet = frag_col(tm, sBeta, j), neg = pk1(-1.f);
              g2[j] = mul2(gam, gam);
              ga[j] = mul2(gam, add2(bet, fma2(bf16x2_to_f32x2(vv[2 * j]), neg, bf16x2_to_f32x2(kk[2 * j]))));
              gb[j] = mul2(gam, add2(bet, fma2(bf16x2_to_f32x2(vv[2 * j + 1]), neg, bf16x2_to_f32x2(kk[2 * j + 1]))));
            }
          }
          const float e0 = -__bfloat162float(eta[tm.r0]) * (1.f / 64.f), e1 = -__bfloat162float(eta[tm.r1]) * (1.f / 64.f);
          wait_mma(CZ);
          TokFrag x, g;
          frag_ld(tm, tmem + TM_A, x);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            x.a[j] = add2(x.a[j], b2r[j]);
            x.b[j] = add2(x.b[j], b2r[j]);
          }
          float rs0, rs1;
          frag_layernorm(tm, x, TTT_LN_EPS, xch, kBarPair, rs0, rs1);
          f32x2 a0 = 0ull, a1 = 0ull, c0 = 0ull, c1 = 0ull;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            g.a[j] = fma2(g2[j], x.a[j], ga[j]);
            g.b[j] = fma2(g2[j], x.b[j], gb[j]);
            a0 = add2(a0, g.a[j]); a1 = fma2(g.a[j], x.a[j], a1);
            c0 = add2(c0, g.b[j]); c1 = fma2(g.b[j], x.b[j], c1);
          }
          float a[2] = {hsum(a0), hsum(a1)}, b[2] = {hsum(c0), hsum(c1)};
          frag_allreduce2<1>(tm, a, b, xch, kBarPair);
          const f32x2 sc0 = pk1(e0 * rs0), sc1 = pk1(e1 * rs1);
          if (it > 0) wait(U_SENT);        // the last X2, U1, U2 and sums have left
          f32x2 cs[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const uint32_t w0 = f32x2_to_bf16x2(mul2(fma2(x.a[j], pk1(-a[1]), fma2(g.a[j], pk1(64.f), pk1(-a[0]))), sc0));
            const uint32_t w1 = f32x2_to_bf16x2(mul2(fma2(x.b[j], pk1(-b[1]), fma2(g.b[j], pk1(64.f), pk1(-b[0]))), sc1));
            *reinterpret_cast<uint32_t*>(smem + OFF_U2 + tm.off(tm.r0, j)) = w0;
            *reinterpret_cast<uint32_t*>(smem + OFF_U2 + tm.off(tm.r1, j)) = w1;
            cs[j] = add2(bf16x2_to_f32x2(w0), bf16x2_to_f32x2(w1));
          }
          done(E_2);
          // under the product: column sums of U2 (bf16 values, the operand the W2 update sees) for b2
          sCol[quad * 64 + frag_colsum_col(tm, lane)] = frag_colsum(cs, lane);
        } else if (it > 0) {
          wait(U_SENT);
        }

        // ---- EPI3: U1^T = R^T * G' (= -eta dl/dZ1), as bf16 to tensor memory, MMA4's operand; its row sums for b1
        wait_mma(CA + blk);
        {
          uint32_t v[32], u[16];
          tmem_ld32(tmem + TM_A + hl, v);
          tmem_wait_ld();
          f32x2 bsum = 0ull;
#pragma unroll
          for (int k = 0; k < 16; ++k) {
            const f32x2 w = mul2(bf16x2_to_f32x2(gp[k]), pk(v[2 * k], v[2 * k + 1]));
            bsum = add2(bsum, w);
            u[k] = f32x2_to_bf16x2(w);
          }
          tmem_st16(tmem + lane_base + TM_U1 + blk * 32 + ch * 16, u);
          sRow[ch * 256 + hrow] = hsum(bsum);
          tmem_wait_st();
          done_tmem(E_3 + blk);
          // while MMA4 runs: U1 to shared memory, for the output CTA
#pragma unroll
          for (int c = 0; c < 4; ++c)
            *reinterpret_cast<uint4*>(smem + OFF_U1 + sw128_off(hrow, ch * 4 + c)) =
                make_uint4(u[4 * c], u[4 * c + 1], u[4 * c + 2], u[4 * c + 3]);
          done(E_U);
        }

        // ---- EPI4: bf16 operand copies of the new state.  The warps of the second column half copy W2 while MMA4 runs, those
        // of the first W1 behind it
        if (ch == 1) {
          wait_mma(CW2);
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            uint32_t v[32];
            tmem_ld32(tmem + lane_base + TM_W2 + blk * 64 + half * 32, v);
            tmem_wait_ld();
            st_cols32(smem + OFF_W2, hrow, half, v);
          }
          done(E_W2);
          wait(CA + blk);
        } else {
          wait_mma(CA + blk);
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            uint32_t v[32];
            tmem_ld32(tmem + lane_base + TM_W1 + blk * 64 + half * 32, v);
            tmem_wait_ld();
            st_cols32_tmem(tmem + lane_base + TM_W1B + blk * 32 + half * 16, v);
          }
          tmem_wait_st();
        }
        done_tmem(E_4 + blk);      // (by those of W2 too: no product may complete on CA again before they have seen MMA4)
        // ---- b1, b2 (the sums are those of this block's warps, which MMA4 waited for)
        add_sums();
      }
    } else {
      // ================================================================================== the output pass
      long ck = sid * p.nck + 1;                         // the next checkpoint, and the mini-batch that it precedes (0: none)
      int next_ck = p.cgs < NC ? p.cgs : 0;
      // the state's fp32 matrices to global memory: W1 by the warps of the first column half, W2 by the others
      auto store_state = [&](float* W1o, float* W2o, float* b1o, float* b2o) {
#pragma unroll 1
        for (int half = 0; half < 2; ++half) {
          uint32_t v[32];
          if (ch == 0) {
            tmem_ld32(tmem + lane_base + TM_W1 + blk * 64 + half * 32, v);
            tmem_wait_ld();
#pragma unroll
            for (int j = 0; j < 32; ++j) W1o[(half * 32 + j) * 256 + hrow] = __uint_as_float(v[j]);
          } else {
            tmem_ld32(tmem + lane_base + TM_W2 + blk * 64 + half * 32, v);
            tmem_wait_ld();
            store_rows_own(W2o + (hrow - lane) * 64 + half * 32, v, smem + OFF_X2B + (warp & 7) * 4096, lane);
          }
        }
        if (ch == 0) b1o[hrow] = b1v;
        if (tok && quad == 0 && lane < 4) {
#pragma unroll
          for (int j = 0; j < 4; ++j) *reinterpret_cast<f32x2*>(b2o + tm.col(j)) = b2r[j];
        }
      };
      for (int it = 0; it < NC; ++it) {
        const int s = it & 1;
        uint8_t* sQ = smem + OFF_Q + s * TILE;
        // ---- COPY: b1, b2, bf16 operand copies of the new W1 and W2
        wait(OU);
        wait_mma(OUPD);
        add_sums();
        {
          uint32_t v[32];
          tmem_ld32(tmem + TM_W1 + hl, v);
          tmem_wait_ld();
          st_cols32_tmem(tmem + lane_base + TM_W1B + blk * 32 + ch * 16, v);
          tmem_ld32(tmem + TM_W2 + hl, v);
          tmem_wait_ld();
          st_cols32(smem + OFF_W2, hrow, ch, v);
          tmem_wait_st();
        }
        done(E_C);
        // ---- the state after this mini-batch is a checkpoint if the next one starts a group
        if (it + 1 == next_ck) {
          store_state(p.W1c + ck * (64 * 256), p.W2c + ck * (64 * 256), p.b1c + ck * 256, p.b2c + ck * 64);
          ck += 1;
          next_ck = it + 1 + p.cgs < NC ? it + 1 + p.cgs : 0;
          named_bar_sync(kBarEpi, kEpi);         // X2b's place is free again
        }
        done(E_R);
        // ---- EPI5: X2b^T = gelu(W1^T Q^T + b1)
        wait_mma(OB);
        {
          const f32x2 bb = pk1(0.5f * b1v);
#pragma unroll 1
          for (int q = 0; q < 2; ++q) {
            uint32_t v[16], g[8];
            tmem_ld16(tmem + TM_A + hl + q * 16, v);
            tmem_wait_ld();
#pragma unroll
            for (int k = 0; k < 8; ++k)
              g[k] = f32x2_to_bf16x2(gelu_half2(fma2(pk(v[2 * k], v[2 * k + 1]), pk1(0.5f), bb)));
            *reinterpret_cast<uint4*>(smem + OFF_X2B + sw128_off(hrow, ch * 4 + q * 2)) = make_uint4(g[0], g[1], g[2], g[3]);
            *reinterpret_cast<uint4*>(smem + OFF_X2B + sw128_off(hrow, ch * 4 + q * 2 + 1)) = make_uint4(g[4], g[5], g[6], g[7]);
          }
        }
        done(E_5);
        // ---- OUT: Q + gamma * LN(Z2b + b2) + beta, over the Q tile (every thread rewrites what it has read)
        if (tok) wait(OQ + s);
        wait_mma(OZ);
        if (tok) {
          TokFrag x;
          uint32_t q[8];
          frag_ld(tm, tmem + TM_ZB, x);
          frag_ld_raw(tm, sQ, q);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            x.a[j] = add2(x.a[j], b2r[j]);
            x.b[j] = add2(x.b[j], b2r[j]);
          }
          float rs0, rs1;
          frag_layernorm(tm, x, TTT_LN_EPS, xch, kBarPair, rs0, rs1);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const f32x2 gam = frag_col(tm, sGamma, j), bet = frag_col(tm, sBeta, j);
            x.a[j] = add2(bf16x2_to_f32x2(q[2 * j]), fma2(gam, x.a[j], bet));
            x.b[j] = add2(bf16x2_to_f32x2(q[2 * j + 1]), fma2(gam, x.b[j], bet));
          }
          frag_st_tile(tm, sQ, x);
          done(E_OUT + s);
        }
      }
      if (p.W1f != nullptr && !idle && __all_sync(0xffffffffu, *abort_flag == 0))
        store_state(p.W1f + st_w, p.W2f + st_w, p.b1f + sid * 256, p.b2f + sid * 64);
    }
  } else {
    reg_give<kRegsHelp>();
    if (chain && warp < 18) {
      // ---- the chain's products: a warp per 128-row block
      const int b = warp - 16;
      for (int it = 0; it < NC; ++it) {
        const uint32_t sK = smem_u32(smem + OFF_K + (it & 1) * TILE), sX2 = smem_u32(smem + OFF_X2 + (it & 1) * BIG);
        if (!seen(CK + (it & 1)) || !seen(E_4 + b)) break;
        mma_hidden_ta<false, false>(tmem + TM_A + b * 64, tmem + TM_W1B + b * 32, sK, lead);                 // MMA1
        commit(CA + b);
        if (b == 0) {
          if (!seen(E_W2) || !seen(E_1 + (it & 1))) break;
          token(tmem + TM_A, sX2, smem_u32(smem + OFF_W2));                    // MMA2
          commit(CZ);
        }
        if (!seen(E_2)) break;
        mma_hidden_lead<false, false>(tmem + TM_A, smem_u32(smem + OFF_W2), smem_u32(smem + OFF_U2), b, lead);      // MMA3
        commit(CA + b);
        mma_hidden_lead<true, true>(tmem + TM_W2, sX2, smem_u32(smem + OFF_U2), b, lead);
        commit(CW2);
        if (!seen(E_3 + b)) break;
        mma_hidden_ta<true, true>(tmem + TM_W1 + b * 64, tmem + TM_U1 + b * 32, sK, lead);                   // MMA4
        commit(CA + b);
      }
    } else if (chain && warp == 18) {
      // ---- the chain's copies: loads, and the output CTA's operands
      auto load_k = [&](int i) {
        if (i < NC && !dropped(i)) {
          const int s = i & 1;
          arm(CK + s, TILE + 128);
          tma_load_2d(smem + OFF_K + s * TILE, &tmK, &bars[CK + s], 0, row_of(i));
          bulk_load_1d(smem + OFF_ETA + s * 128, p.eta + (sid * NC + i) * 64, 128, &bars[CK + s]);
        }
      };
      auto send = [&](uint32_t off, uint32_t bytes, int bar) {
        bulk_copy_peer(mapa(smem_u32(smem + off), peer), smem_u32(smem + off), bytes, mapa(smem_u32(&bars[bar]), peer));
      };
      if (lane == 0) {
#pragma unroll 1
        for (int i = 0; i < 2; ++i) {
          load_k(i);
          load_tile(i, &tmV, OFF_V, CV);
        }
      }
      __syncwarp();
      for (int it = 0; it < NC; ++it) {
        if (!seen(E_1 + (it & 1))) break;
        if (lane == 0 && it > 0) load_k(it + 1);                      // all warps are past the last mini-batch's MMA4, which read K
        __syncwarp();
        if (lane == 0) send(OFF_X2 + (it & 1) * BIG, BIG, OX + (it & 1));      // (its place there: X_FREE of two mini-batches ago)
        __syncwarp();
        if (!seen(E_2)) break;
        if (lane == 0) load_tile(it + 2, &tmV, OFF_V, CV);            // V has been read
        __syncwarp();
        if (it > 0 && !seen(X_FREE)) break;
        if (lane == 0) send(OFF_U2, TILE, OU);
        __syncwarp();
        if (!seen(E_U)) break;
        if (lane == 0) {
          send(OFF_U1, BIG, OU);
          send(OFF_SUM, SUM_BYTES, OU);
        }
        __syncwarp();
      }
      if (NC > 0) seen(X_FREE);                // nothing is on its way from this CTA when it ends
    } else if (!chain && warp == 16) {
      // ---- the output CTA's state update
      for (int it = 0; it < NC; ++it) {
        const uint32_t sK = smem_u32(smem + OFF_K + (it & 1) * TILE), sX2 = smem_u32(smem + OFF_X2 + (it & 1) * BIG);
        if (!seen(E_R) || !seen(OKT + (it & 1)) || !seen(OX + (it & 1))) break;
        if (!seen(OU)) break;
#pragma unroll
        for (int b = 0; b < 2; ++b) {
          mma_hidden_lead<true, true>(tmem + TM_W1, smem_u32(smem + OFF_U1), sK, b, lead);
          mma_hidden_lead<true, true>(tmem + TM_W2, sX2, smem_u32(smem + OFF_U2), b, lead);
        }
        commit(OUPD);
      }
    } else if (!chain && warp == 17) {
      // ---- its other products
      for (int it = 0; it < NC; ++it) {
        const uint32_t sQ = smem_u32(smem + OFF_Q + (it & 1) * TILE);
        if (!seen(OQ + (it & 1)) || !seen(E_C)) break;
#pragma unroll
        for (int b = 0; b < 2; ++b)
          mma_hidden_ta<false, false>(tmem + TM_A + b * 64, tmem + TM_W1B + b * 32, sQ, lead);               // MMA5
        commit(OB);
        if (!seen(E_5)) break;
        token(tmem + TM_ZB, smem_u32(smem + OFF_X2B), smem_u32(smem + OFF_W2));                    // MMA6
        commit(OZ);
      }
    } else if (!chain && warp == 18) {
      // ---- what the chain sends: acknowledged when it has arrived, and its place given back when it has been used
      auto expect = [&](int i) {
        mbar_expect_tx(&bars[OX + (i & 1)], BIG);
      };
      auto expect_u = [&]() { mbar_expect_tx(&bars[OU], BIG + TILE + SUM_BYTES); };
      if (lane == 0) {
        if (NC > 0) expect(0);
        if (NC > 1) expect(1);
        if (NC > 0) expect_u();
        load_tile(0, &tmK, OFF_K, OKT);
        load_tile(1, &tmK, OFF_K, OKT);
      }
      __syncwarp();
      for (int it = 0; it < NC; ++it) {
        if (!seen(OX + (it & 1))) break;
        if (!seen(OU)) break;
        if (lane == 0) mbar_arrive_remote(&bars[U_SENT], peer);
        __syncwarp();
        if (!seen(E_C)) break;                 // (behind MMA4, which it waits for)
        if (lane == 0) {
          load_tile(it + 2, &tmK, OFF_K, OKT);
          if (it + 2 < NC) expect(it + 2);
          if (it + 1 < NC) expect_u();
          mbar_arrive_remote(&bars[X_FREE], peer);
        }
        __syncwarp();
      }
    } else if (!chain) {
      // ---- Q in, Out out
      if (lane == 0) {
        load_tile(0, &tmQ, OFF_Q, OQ);
        load_tile(1, &tmQ, OFF_Q, OQ);
      }
      __syncwarp();
      for (int it = 0; it < NC; ++it) {
        if (!seen(E_OUT + (it & 1))) break;
        if (lane == 0) {
          tma_store_2d(&tmOut, smem + OFF_Q + (it & 1) * TILE, 0, row_of(it));
          tma_commit_group();
          tma_wait_group_read<0>();
          load_tile(it + 2, &tmQ, OFF_Q, OQ);
        }
        __syncwarp();
      }
      if (lane == 0) tma_wait_group<0>();
      __syncwarp();
    }
  }

  // ---- teardown
  tc_fence_before_sync();
  const bool aborted = __syncthreads_or(*abort_flag != 0) != 0;
  tc_fence_after_sync();
  if (aborted && tid == 0) st_cluster_u32(mapa(smem_u32(const_cast<uint32_t*>(abort_flag)), peer), 1u);
  if (aborted) {
    // everything this CTA still has in flight is waited for (bounded, not cut short by the abort flag) before its shared and
    // tensor memory go away: the tensor-core work of both issuers, and the loads
    if ((warp == 16 || warp == 17) && lead) umma_commit(&bars[BDRAIN]);
    if (warp >= 16) {
      for (int b = 0; b < U_SENT; ++b)
        if ((lda >> b) & 1u) mbar_wait_bounded(&bars[b], ((ldp >> b) & 1u) ^ 1u, never_flag, limit);
    }
    if (tid == 0) {
      mbar_wait_bounded(&bars[BDRAIN], 0, never_flag, limit);
      atomicExch(p.status, static_cast<uint32_t>(TTT_B200_ERR_TIMEOUT));
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, TM_COLS);
  if (aborted) {         // copies to the other CTA that the abort cut short may still be on their way: they take a few microseconds
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 50000) {}
    __syncthreads();
  }
  // No CTA leaves while another may still send to it.  One barrier for all of the cluster: whether a CTA aborted is its own
  // affair, and with two streams to a cluster not the other stream's.  (A CTA that sent anything and did not abort has seen it
  // used: X_FREE of the last mini-batch.)
  cluster_arrive();
  cluster_wait();
}

// Once per device: the kernel's dynamic shared memory limit.
int prepare_kernel() {
  static std::once_flag once[64];
  static cudaError_t attr_err[64];
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return ttt_set_error(TTT_B200_ERR_LAUNCH, "device index out of range");
  std::call_once(once[dev], [&] {
    attr_err[dev] = cudaFuncSetAttribute(ttt_fwd_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
  });
  if (attr_err[dev] != cudaSuccess) return ttt_set_error(TTT_B200_ERR_LAUNCH, cudaGetErrorString(attr_err[dev]));
  return TTT_B200_OK;
}

void launch_attributes(cudaLaunchAttribute (&attr)[2]) {
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2 * kStreams;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
}

// How many clusters the device runs at once (a cluster lives inside one GPC).  0 if the query fails.
int clusters_at_once() {
  static std::once_flag once[64];
  static int cap[64];
  if (prepare_kernel()) return 0;
  int dev = 0;
  cudaGetDevice(&dev);
  std::call_once(once[dev], [&] {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * kStreams * 64);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = SMEM_BYTES;
    cudaLaunchAttribute attr[2];
    launch_attributes(attr);
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, ttt_fwd_pair_kernel, &cfg) != cudaSuccess) {
      cudaGetLastError();
      n = 0;
    }
    cap[dev] = n;
  });
  return cap[dev];
}

}  // namespace

// How many streams the device runs at once with two CTAs each.
int ttt_forward_pair_capacity() { return kStreams * clusters_at_once(); }

int ttt_launch_forward_pair(const ttt_b200_fwd_args* a, cudaStream_t stream, uint32_t* status, uint64_t limit_ns, int drop_load) {
  const uint64_t rows = static_cast<uint64_t>(a->B) * a->H * a->NC * 64;
  CUtensorMap tmQ, tmK, tmV, tmOut;
  if (int rc = ttt_make_tile_map(&tmQ, a->XQ, rows)) return rc;
  if (int rc = ttt_make_tile_map(&tmK, a->XK, rows)) return rc;
  if (int rc = ttt_make_tile_map(&tmV, a->XV, rows)) return rc;
  if (int rc = ttt_make_tile_map(&tmOut, a->Out, rows)) return rc;
  FwdParams p;
  p.eta = static_cast<const __nv_bfloat16*>(a->last_eta);
  p.gamma = a->ttt_norm_weight;
  p.beta = a->ttt_norm_bias;
  p.W1 = a->W1; p.b1 = a->b1; p.W2 = a->W2; p.b2 = a->b2;
  p.W1c = a->W1_checkpoints; p.b1c = a->b1_checkpoints; p.W2c = a->W2_checkpoints; p.b2c = a->b2_checkpoints;
  const bool want_final = a->W1_final && a->b1_final && a->W2_final && a->b2_final;
  p.W1f = want_final ? a->W1_final : nullptr;
  p.b1f = a->b1_final; p.W2f = a->W2_final; p.b2f = a->b2_final;
  p.H = a->H; p.NC = a->NC; p.cgs = a->checkpoint_group_size; p.nck = a->num_checkpoints;
  p.streams = a->B * a->H;
  p.drop_load = drop_load;
  p.status = status;
  p.wait_limit_ns = limit_ns;
  if (int rc = prepare_kernel()) return rc;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>((p.streams + kStreams - 1) / kStreams * 2 * kStreams));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = SMEM_BYTES;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  launch_attributes(attr);
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, ttt_fwd_pair_kernel, tmQ, tmK, tmV, tmOut, p);
  if (e != cudaSuccess) return ttt_set_error(TTT_B200_ERR_LAUNCH, cudaGetErrorString(e));
  return TTT_B200_OK;
}
