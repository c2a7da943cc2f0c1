// TTT-MLP forward for sm_100a: one persistent CTA per (batch, head) stream.
//
// Replaces the reference's fwd_ttt_mlp_ker (kernels/ttt/ttt.cu:85-586); the per-mini-batch
// math is that of kernels/ttt/matching.py:30-125.
//
// Orientation.  Every 64x256 / 256x64 quantity is kept "hidden-major": the 256 hidden units
// run along the M dimension of the tensor-core tile (= TMEM lanes, = one thread per hidden
// unit in the epilogues) and the 64 tokens or 64 features along N.  The fp32 master state
//   W1^T [256 x 64]  and  W2 [256 x 64]
// lives in tensor memory as the accumulator of its own update MMA; a bf16 copy in shared
// memory, refreshed once per mini-batch, feeds the other MMAs.  b1 lives in registers (one
// hidden unit per thread), b2 in shared memory.
//
// A mini-batch is a chain of dependent MMA -> epilogue round trips, and only a part of it is needed by the
// next mini-batch: the output pass (the post-update product with Q, GELU, LayerNorm) is not.  So the CTA runs two
// groups of eight warps, each with its own accumulator in tensor memory, its own MMA issuers and barriers:
//
//   chain group                                        output group
//   MMA1  Z1^T = W1^T K^T        [256 x 64 tok]        (U2 there:)    W2 += X2^T U2
//   EPI1  X2^T = gelu(Z1^T + b1), G' = gelu'(.)                       bf16 copy of the new W2 -> smem; b2 += colsum(U2)
//   MMA2  Z2 = X2 W2             [64 tok x 64]         (W1 copied:)   checkpoints;  MMA5  Z1b^T = W1^T Q^T
//   LN    U2 = -eta * dl/dZ2 (fused LN + L2 gradient)  EPI5  X2b^T = gelu(Z1b^T + b1)
//   MMA3  R^T = W2 U2^T                                MMA6  Z2b = X2b W2
//   EPI3  U1^T = R^T * G';  b1 += rowsum               OUT   Q + gamma * LN(Z2b + b2) + beta -> TMA store
//   MMA4  W1^T += U1^T K
//   EPI4  bf16 copy of the new W1^T
//
// The output group works one step behind, on the state the chain group has just left: the chain is four round
// trips per mini-batch instead of six, and each group's MMA latencies are filled with the other's epilogues (four
// warps per scheduler).
//
// What bounds it: the chain's four round trips.  No pipe is full over a mini-batch (128 streams: issue slots 44 %, fp32
// pipe 37 %, tensor pipe 21 %, DRAM 11 %), but within its epilogues the fp32 and MUFU pipes set the pace (EPI1 alone is
// 1300 cycles of fp32 pipe at 9 packed operations and 2 conversions per pair of elements) and within its products the
// shared-memory operands.  So the arithmetic runs on packed fp32 pairs; what only one thread needs stays out of shared
// memory (G' in registers from EPI1 to EPI3, U1 and the bf16 W1 in tensor memory as A operands of their MMAs, which then
// read 2 KB of shared memory instead of 6); and the MMAs are issued from warp-uniform code.  Measured (B200, 128 streams
// of 128 mini-batches, one checkpoint in 8): 8.0 us per mini-batch as one group of 8 warps, 6.0 with the two groups, 4.6
// with the rest, 4.3 with the products of a block issued by the block's own first warp and the W2 update by the output
// group (before, one warp issued all sixteen MMAs of the state update and came 400 cycles late to EPI4, with everyone
// waiting for it); 1536 streams of 64 mini-batches 5.43 -> 3.23 -> 3.00 ms.  In groups of two, where the output group is the
// longer one on average, that made calls of 16 and more mini-batches 1.1 to 1.6 % slower (128 x 32 169.1 -> 171.4 us; in groups
// of one and three as before); with W2's update left to the chain there (167.6) the kernel's other calls lost up to 0.9 %.  The
// copy of W2 rolled again, 1536 x 64 2946 -> 3023 us; checkpoints divided for instead of counted, 2949.  A checkpoint costs about
// 2100 cycles (the output group's 4200 for 132 KB of stores, of which half fit its slack); as bulk copies from a staging area
// it cost more, since W1's turn of the area waits for W2 to leave.
//
// Hand-over between the groups (mbarriers, each completed once per mini-batch):
//   u2rdy   U2 and X2 are in place                             chain -> output group (W2 update)
//   r       MMA3 has read the bf16 W2                          chain's tensor work -> output group (its next copy)
//   w2upd   the W2 update has completed                        output's tensor work -> output group; chain (EPI1: X2)
//   w2rdy   bf16 W2 and b2 are refreshed                       output group -> chain (MMA2, LN)
//   sread   the output group has read the state columns and
//           taken note of w1rdy                                output group -> chain (MMA4)
//   w1rdy   bf16 W1 and the shared copy of b1 are refreshed    chain -> output group (MMA5)
//   w1read  MMA5 has completed: the bf16 W1 may be rewritten   output's tensor work -> chain (EPI4)
// A waiter tells only odd from even completions, so a barrier that the other group waits for must complete once per
// mini-batch and be waited for in every one.  (w1read is apart from accb, the accumulator's own barrier, which completes
// once per 128-row block: with its second use in the place of w1read, the use of the mini-batch before satisfied EPI4
// while an output group held up by its checkpoint stores had not issued MMA5 yet, and Out took a state one step too new.)
//
// All waits are bounded (see sm100_ptx.cuh); on expiry the CTA reports through the status
// word, drains its own copies, frees its tensor memory and returns.
#include <mutex>

#define TTT_WAIT_INLINE
#include "ttt_device.cuh"
#include "ttt_internal.h"

using namespace tttdev;

namespace {

constexpr int kStages = 2;
constexpr int kGroup = 256;          // threads of one group
constexpr int kThreads = 2 * kGroup;
// registers per thread: EPI1 leaves G' in 32 of the chain group's
constexpr int kRegsChain = 152, kRegsOut = 104;
static_assert(kRegsChain + kRegsOut <= 2 * 128, "the block is launched with 128 registers per thread");
// named barriers: one per warp pair of each group, then one per group
constexpr uint32_t kBarPairC = 1, kBarPairO = 5, kBarC = 9, kBarO = 10, kBarBlk = 11;      // kBarBlk: + 128-row block of the chain

constexpr uint32_t OFF_K = 0;
constexpr uint32_t OFF_V = OFF_K + kStages * TILE;
constexpr uint32_t OFF_Q = OFF_V + kStages * TILE;      // Q, then Out on its way to global memory
constexpr uint32_t OFF_W2 = OFF_Q + kStages * TILE;
constexpr uint32_t OFF_X2 = OFF_W2 + BIG;
constexpr uint32_t OFF_X2B = OFF_X2 + BIG;
constexpr uint32_t OFF_STG = OFF_X2B + BIG;             // 4 KB per warp of the output group: W2 checkpoints on their way out
constexpr uint32_t OFF_U2 = OFF_STG + BIG;
constexpr uint32_t OFF_ETA = OFF_U2 + TILE;
constexpr uint32_t OFF_B1 = OFF_ETA + kStages * 128;    // fp32[2][256]: b1 as of odd / even mini-batches
constexpr uint32_t OFF_B2 = OFF_B1 + 2048;              // fp32[2][64]
constexpr uint32_t OFF_GAMMA = OFF_B2 + 512;
constexpr uint32_t OFF_BETA = OFF_GAMMA + 256;
constexpr uint32_t OFF_XCHC = OFF_BETA + 256;           // row-sum exchange of each group
constexpr uint32_t OFF_XCHO = OFF_XCHC + kXchBytes;     // also the partial column sums: fp32[8][64]
constexpr uint32_t OFF_BAR = OFF_XCHO + kXchBytes;
constexpr uint32_t OFF_MISC = OFF_BAR + 192;
constexpr uint32_t SMEM_USED = OFF_MISC + 16;
constexpr uint32_t SMEM_BYTES = SMEM_USED + 1024;       // slack for the 1024-byte alignment
static_assert(SMEM_BYTES <= 232448, "exceeds the 227 KB per-CTA shared memory of sm_100");
static_assert(kXchBytes >= 8 * 64 * 4, "the partial column sums fit the exchange area");

// barrier indices
constexpr int BAR_K = 0, BAR_V = 2, BAR_Q = 4;          // + stage
constexpr int BAR_ACCA = 6;                             // + block (the two 128-row halves of the accumulator)
constexpr int BAR_Z = 8;
constexpr int BAR_ACCB = 9;                             // two uses per mini-batch, within the output group
constexpr int BAR_W1READ = 10;
constexpr int BAR_ZB = 11;
constexpr int BAR_W2UPD = 12, BAR_W2RDY = 13, BAR_SREAD = 14, BAR_W1RDY = 15;
constexpr int BAR_U2RDY = 16, BAR_R = 17;
constexpr int BAR_DRAIN = 18;                           // abort path only
constexpr int kBars = 19;

// tensor-memory columns: two 128-lane blocks of 64 fp32 (32 bf16-pair) columns per 256-row matrix
constexpr uint32_t TM_W1 = 0;
constexpr uint32_t TM_W2 = 128;
constexpr uint32_t TM_A = 256;       // chain: Z1; Z2 in its first 64 columns; R; U1 (bf16) in the first half of each block
constexpr uint32_t TM_W1B = 384;     // bf16 operand copy of W1^T
constexpr uint32_t TM_B = 448;       // output: Z1b, one block after the other; Z2b
constexpr uint32_t TM_COLS = 512;

struct FwdParams {
  const __nv_bfloat16* eta;
  const float* gamma;
  const float* beta;
  const float* W1;
  const float* b1;
  const float* W2;
  const float* b2;
  float* W1c;
  float* b1c;
  float* W2c;
  float* b2c;
  float* W1f;
  float* b1f;
  float* W2f;
  float* b2f;
  int H, NC, cgs, nck;
  int drop_load;            // test only: mini-batch whose loads stream 0 never issues (-1: none)
  uint32_t* status;
  uint64_t wait_limit_ns;
};

__global__ void __launch_bounds__(kThreads, 1)
ttt_fwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
               const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmOut,
               const FwdParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_align_1024(smem_raw);

  const int tid = threadIdx.x, lane = tid & 31;
  const int cta_warp = __shfl_sync(0xffffffffu, tid >> 5, 0);   // same value, known to be warp-uniform
  const int warp = cta_warp & 7;                         // within the group
  const int quad = warp & 3, wg = warp >> 2;
  const int gtid = tid & (kGroup - 1);
  const int hrow = wg * 128 + quad * 32 + lane;          // hidden unit owned in the 256-row epilogues
  const uint32_t lane_base = static_cast<uint32_t>(quad * 32) << 16;
  const TokMap tm(warp, lane);                           // fragment of the 64 x 64 token-major tiles
  const long stream_id = blockIdx.x;
  const int head = static_cast<int>(stream_id % p.H);

  uint8_t* sW2 = smem + OFF_W2;
  uint8_t* sX2 = smem + OFF_X2;
  uint8_t* sX2b = smem + OFF_X2B;
  uint8_t* sU2 = smem + OFF_U2;
  float* sB1 = reinterpret_cast<float*>(smem + OFF_B1);
  float* sB2 = reinterpret_cast<float*>(smem + OFF_B2);
  float* sGamma = reinterpret_cast<float*>(smem + OFF_GAMMA);
  float* sBeta = reinterpret_cast<float*>(smem + OFF_BETA);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + OFF_BAR);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + OFF_MISC);
  volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(smem + OFF_MISC + 4);
  volatile uint32_t* never_flag = reinterpret_cast<volatile uint32_t*>(smem + OFF_MISC + 8);   // stays 0
  volatile uint32_t* stop_flag = reinterpret_cast<volatile uint32_t*>(smem + OFF_MISC + 12);   // the chain group's copy of abort_flag

  const uint64_t limit = p.wait_limit_ns;
  const int NC = p.NC;

  if (tid == 0) {
    for (int i = 0; i < kBars; ++i)
      mbar_init(&bars[i], i == BAR_SREAD ? 8 : i == BAR_W2RDY || i == BAR_DRAIN ? 3 : i == BAR_W1RDY || i == BAR_R ? 2 : 1);
    fence_mbar_init();
    *abort_flag = 0;
    *never_flag = 0;
    prefetch_tmap(&tmQ);
    prefetch_tmap(&tmK);
    prefetch_tmap(&tmV);
    prefetch_tmap(&tmOut);
  }
  if (cta_warp == 0) {
    tmem_alloc(tmem_slot, TM_COLS);
    tmem_relinquish();
  }
  griddep_launch();
  griddep_wait();
  if (tid < 64) {
    sGamma[tid] = p.gamma[head * 64 + tid];
    sBeta[tid] = p.beta[head * 64 + tid];
    sB2[tid] = p.b2[stream_id * 64 + tid];
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot;

  auto wait_bar = [&](int b, uint32_t parity) { mbar_wait_bounded(&bars[b], parity & 1u, abort_flag, limit); };
  // Loads, by one thread of the group that consumes them: K with eta, V (chain group), Q (output group).  Stream
  // 0's loads of mini-batch drop_load are never issued (test of the failure path).
  auto dropped = [&](int i) { return i == p.drop_load && stream_id == 0; };
  auto row_of = [&](int i) { return static_cast<int>((stream_id * NC + i) * 64); };
  auto load_k = [&](int i) {
    if (i >= NC || dropped(i)) return;
    const int s = i & 1;
    mbar_expect_tx(&bars[BAR_K + s], TILE + 128);
    tma_load_2d(smem + OFF_K + s * TILE, &tmK, &bars[BAR_K + s], 0, row_of(i));
    bulk_load_1d(smem + OFF_ETA + s * 128, p.eta + (stream_id * NC + i) * 64, 128, &bars[BAR_K + s]);
  };
  auto load_tile = [&](int i, const CUtensorMap* map, uint32_t off, int bar) {
    if (i >= NC || dropped(i)) return;
    const int s = i & 1;
    mbar_expect_tx(&bars[bar + s], TILE);
    tma_load_2d(smem + off + s * TILE, map, &bars[bar + s], 0, row_of(i));
  };
  // abort path: the loads of mini-batches i and i + 1 or before that may still be in flight, one per stage
  auto drain_loads = [&](int bar, int issued) {
    for (int i = issued > kStages ? issued - kStages : 0; i < issued && i < NC; ++i)
      if (!dropped(i)) mbar_wait_bounded(&bars[bar + (i & 1)], (i >> 1) & 1, never_flag, limit);
  };
  const long st_w = stream_id * (64 * 256);
  const bool chain = cta_warp < 8;
  const uint32_t lead = elect_one() ? 1u : 0u;      // the lane that issues the MMAs (warps 0 and 4 of the chain group, warp 0 of the output group)
  int it = 0;
  int issued = 0;       // loads of this group issued so far (its loading thread), for the abort path

  if (chain) {
    // ================================================================================== chain group
    reg_take<kRegsChain>();
    const bool loader = gtid == 224;      // of a warp that issues no products: its bookkeeping stays off the issue path
    if (loader) {
      for (; issued < kStages; ++issued) {
        load_k(issued);
        load_tile(issued, &tmV, OFF_V, BAR_V);
      }
    }
    auto publish = [&]() {     // shared-memory writes and tensor-memory reads done -> the next MMA may be issued
      fence_proxy_async_smem();
      tc_fence_before_sync();
      named_bar_sync(kBarC, kGroup);
    };
    auto publish_block = [&]() {     // the same, by and for the warps of one 128-row block
      tc_fence_before_sync();
      named_bar_sync(kBarBlk + wg, kGroup / 2);
    };
    const bool issuer = quad == 0;      // warps 0 and 4: each issues its block's products
    // ---- initial W1, b1: global fp32 -> tensor memory (master), shared memory (bf16 operand copy), checkpoint 0
    float b1v = p.b1[stream_id * 256 + hrow];
    {
      const float* W1g = p.W1 + st_w + hrow;
      float* W1k = p.W1c + stream_id * p.nck * (64 * 256) + hrow;
#pragma unroll 1
      for (int half = 0; half < 2; ++half) {
        uint32_t v[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = __float_as_uint(W1g[(half * 32 + j) * 256]);
        tmem_st32(tmem + lane_base + TM_W1 + wg * 64 + half * 32, v);
        st_cols32_tmem(tmem + lane_base + TM_W1B + wg * 32 + half * 16, v);
#pragma unroll
        for (int j = 0; j < 32; ++j) W1k[(half * 32 + j) * 256] = __uint_as_float(v[j]);
      }
      p.b1c[stream_id * p.nck * 256 + hrow] = b1v;
      if (gtid < 64) p.b2c[stream_id * p.nck * 64 + gtid] = sB2[gtid];
      tmem_wait_st();
    }
    publish();

    uint32_t pa = 0;      // parity of the accumulator barriers: three uses per mini-batch
    auto wait_acca = [&]() {
      wait_bar(BAR_ACCA + wg, pa);
      pa ^= 1u;
      __syncwarp();
      tc_fence_after_sync();
    };
    // The two 128-row blocks of a product are issued and committed one by one, each by the first of its four warps: the
    // warps of a block start when theirs is complete, and where only a block's own rows are needed (U1, the bf16 W1) they
    // wait for each other alone.
    for (; it < NC; ++it) {
      const int s = it & 1;
      const uint8_t* sK = smem + OFF_K + s * TILE;
      const uint8_t* sV = smem + OFF_V + s * TILE;
      const __nv_bfloat16* sEta = reinterpret_cast<const __nv_bfloat16*>(smem + OFF_ETA + s * 128);
      const uint32_t par = it & 1, prev = par ^ 1u;      // parity of this / the last mini-batch's hand-overs
      wait_bar(BAR_K + s, it >> 1);

      // ---- MMA1: Z1^T = W1^T K^T
      if (issuer) {
        tc_fence_after_sync();
        mma_hidden_ta<false, false>(tmem + TM_A + wg * 64, tmem + TM_W1B + wg * 32, smem_u32(sK), lead);
        if (lead) umma_commit(&bars[BAR_ACCA + wg]);
      }
      if (it > 0) wait_bar(BAR_W2UPD, prev);             // the W2 update has read X2
      wait_acca();
      // ---- EPI1: X2^T = gelu(Z1^T + b1) -> smem; G' = gelu'(Z1^T + b1) stays in registers (the thread that needs it
      // in EPI3 is this one).  The next 16 columns are requested before these are processed.
      uint32_t gp[32];
      {
        const f32x2 bb = pk1(b1v);
        const uint32_t acc = tmem + lane_base + TM_A + wg * 64;
        uint32_t v[2][16];
        tmem_ld16(acc, v[0]);
        tmem_wait_ld();
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          if (q < 3) tmem_ld16(acc + q * 16 + 16, v[(q + 1) & 1]);
          uint32_t g[8];
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            f32x2 x, y;
            gelu_pair2(add2(pk(v[q & 1][2 * k], v[q & 1][2 * k + 1]), bb), x, y);
            g[k] = f32x2_to_bf16x2(x);
            gp[q * 8 + k] = f32x2_to_bf16x2(y);
          }
          *reinterpret_cast<uint4*>(sX2 + sw128_off(hrow, q * 2)) = make_uint4(g[0], g[1], g[2], g[3]);
          *reinterpret_cast<uint4*>(sX2 + sw128_off(hrow, q * 2 + 1)) = make_uint4(g[4], g[5], g[6], g[7]);
          tmem_wait_ld();
        }
      }
      if (gtid == 0) *stop_flag = *abort_flag;
      publish();
      const bool stop = *stop_flag != 0;
      if (loader && it > 0) {      // MMA4 of the last mini-batch has read K
        load_k(it + 1);
        issued = it + 2;
      }

      // ---- MMA2: Z2 = X2 W2
      wait_bar(BAR_W2RDY, par);                          // also b2, written with it
      if (cta_warp == 0) {
        __syncwarp();
        tc_fence_after_sync();
        mma_token_lead(tmem + TM_A, smem_u32(sX2), smem_u32(sW2), lead);
        if (lead) umma_commit(&bars[BAR_Z]);
      }
      wait_bar(BAR_V + s, it >> 1);
      wait_bar(BAR_Z, par);
      __syncwarp();
      tc_fence_after_sync();
      // ---- LN: fused LayerNorm + L2 gradient, U2 = -eta * dl/dZ2 (all 8 warps, 16 values each)
      {
        float* xch = reinterpret_cast<float*>(smem + OFF_XCHC);
        const float* b2 = sB2 + par * 64;
        TokFrag x;
        uint32_t kk[8], vv[8];
        frag_ld(tm, tmem + TM_A, x);
        frag_ld_raw(tm, sK, kk);         // requested before the all-reduces of the LayerNorm, used after them
        frag_ld_raw(tm, sV, vv);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const f32x2 b = frag_col(tm, b2, j);
          x.a[j] = add2(x.a[j], b);
          x.b[j] = add2(x.b[j], b);
        }
        float rs0, rs1;
        frag_layernorm(tm, x, TTT_LN_EPS, xch, kBarPairC, rs0, rs1);
        TokFrag g;
        f32x2 a0 = 0ull, a1 = 0ull, c0 = 0ull, c1 = 0ull;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const f32x2 gam = frag_col(tm, sGamma, j), bet = frag_col(tm, sBeta, j), neg = pk1(-1.f);
          const f32x2 t0 = fma2(bf16x2_to_f32x2(vv[2 * j]), neg, bf16x2_to_f32x2(kk[2 * j]));          // K - V
          const f32x2 t1 = fma2(bf16x2_to_f32x2(vv[2 * j + 1]), neg, bf16x2_to_f32x2(kk[2 * j + 1]));
          g.a[j] = mul2(fma2(gam, x.a[j], add2(t0, bet)), gam);
          g.b[j] = mul2(fma2(gam, x.b[j], add2(t1, bet)), gam);
          a0 = add2(a0, g.a[j]); a1 = fma2(g.a[j], x.a[j], a1);
          c0 = add2(c0, g.b[j]); c1 = fma2(g.b[j], x.b[j], c1);
        }
        float a[2] = {hsum(a0), hsum(a1)}, b[2] = {hsum(c0), hsum(c1)};
        frag_allreduce2<1>(tm, a, b, xch, kBarPairC);
        const f32x2 sc0 = pk1(-__bfloat162float(sEta[tm.r0]) * rs0 * (1.f / 64.f));
        const f32x2 sc1 = pk1(-__bfloat162float(sEta[tm.r1]) * rs1 * (1.f / 64.f));
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          g.a[j] = mul2(fma2(x.a[j], pk1(-a[1]), fma2(g.a[j], pk1(64.f), pk1(-a[0]))), sc0);
          g.b[j] = mul2(fma2(x.b[j], pk1(-b[1]), fma2(g.b[j], pk1(64.f), pk1(-b[0]))), sc1);
        }
        frag_st_tile(tm, sU2, g);
      }
      publish();

      // ---- MMA3: R^T = W2 U2^T
      if (issuer) {
        tc_fence_after_sync();
        mma_hidden_lead<false, false>(tmem + TM_A, smem_u32(sW2), smem_u32(sU2), wg, lead);
        if (lead) umma_commit(&bars[BAR_ACCA + wg]);
        if (lead) umma_commit(&bars[BAR_R]);
      }
      if (gtid == 64) mbar_arrive(&bars[BAR_U2RDY]);     // the output group updates W2
      if (loader) load_tile(it + kStages, &tmV, OFF_V, BAR_V);      // V has been read
      wait_acca();
      // ---- EPI3: U1^T = R^T * G' (= -eta dl/dZ1), as bf16 over R in tensor memory; b1 += row sum
      {
        f32x2 bsum = 0ull;
        const uint32_t acc = tmem + lane_base + TM_A + wg * 64;
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          uint32_t v[32], u[16];
          tmem_ld32(acc + half * 32, v);
          tmem_wait_ld();
#pragma unroll
          for (int k = 0; k < 16; ++k) {
            const f32x2 w = mul2(bf16x2_to_f32x2(gp[half * 16 + k]), pk(v[2 * k], v[2 * k + 1]));
            bsum = add2(bsum, w);
            u[k] = f32x2_to_bf16x2(w);
          }
          tmem_st16(acc + half * 16, u);
        }
        b1v += hsum(bsum);
        sB1[prev * 256 + hrow] = b1v;      // b1 after this mini-batch
        tmem_wait_st();
      }
      publish_block();

      // ---- MMA4: W1^T += U1^T K
      if (issuer) {
        if (it > 0) wait_bar(BAR_SREAD, prev);
        __syncwarp();
        tc_fence_after_sync();
        mma_hidden_ta<true, true>(tmem + TM_W1 + wg * 64, tmem + TM_A + wg * 64, smem_u32(sK), lead);
        if (lead) umma_commit(&bars[BAR_ACCA + wg]);
      }
      if (it > 0) wait_bar(BAR_W1READ, prev);         // the last mini-batch's MMA5 has read the bf16 W1
      wait_acca();
      // ---- EPI4: bf16 operand copy of the new W1
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        uint32_t v[32];
        tmem_ld32(tmem + lane_base + TM_W1 + wg * 64 + half * 32, v);
        tmem_wait_ld();
        st_cols32_tmem(tmem + lane_base + TM_W1B + wg * 32 + half * 16, v);
      }
      tmem_wait_st();
      publish_block();
      if (lane == 0 && quad == 1) mbar_arrive(&bars[BAR_W1RDY]);
      if (stop) break;
    }
    if (loader && *abort_flag) {
      drain_loads(BAR_K, issued);
      drain_loads(BAR_V, it + kStages + 1);
    }
  } else {
    // ================================================================================= output group
    reg_give<kRegsOut>();
    const bool loader = gtid == 128;
    if (loader)
      for (; issued < kStages; ++issued) load_tile(issued, &tmQ, OFF_Q, BAR_Q);
    auto publish = [&]() {
      fence_proxy_async_smem();
      tc_fence_before_sync();
      named_bar_sync(kBarO, kGroup);
    };
    uint8_t* stage = smem + OFF_STG + warp * 4096;
    long ck = stream_id * p.nck + 1;                   // the next checkpoint, and the mini-batch that it precedes (0: none)
    int next_ck = p.cgs < NC ? p.cgs : 0;
    // ---- initial W2: global fp32 -> tensor memory (master), shared memory (bf16 operand copy), checkpoint 0
    {
      const float4* W2g = reinterpret_cast<const float4*>(p.W2 + st_w + hrow * 64);
      float* W2k = p.W2c + stream_id * p.nck * (64 * 256) + (hrow - lane) * 64;
#pragma unroll 1
      for (int half = 0; half < 2; ++half) {
        uint32_t v[32];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float4 q4 = W2g[half * 8 + j];
          v[4 * j] = __float_as_uint(q4.x); v[4 * j + 1] = __float_as_uint(q4.y);
          v[4 * j + 2] = __float_as_uint(q4.z); v[4 * j + 3] = __float_as_uint(q4.w);
        }
        tmem_st32(tmem + lane_base + TM_W2 + wg * 64 + half * 32, v);
        st_cols32(sW2, hrow, half, v);
        store_rows_own(W2k + half * 32, v, stage, lane);
      }
      tmem_wait_st();
    }
    publish();
    if (gtid < 3) mbar_arrive(&bars[BAR_W2RDY]);

    for (; it < NC; ++it) {
      const int s = it & 1;
      uint8_t* sQ = smem + OFF_Q + s * TILE;
      const uint32_t par = it & 1, next = par ^ 1u;
      // ---- W2 += X2^T U2 (the group's reads of W2 for the last mini-batch's checkpoint are behind its barriers)
      if (warp == 0) {
        wait_bar(BAR_U2RDY, par);
        __syncwarp();
        tc_fence_after_sync();
        mma_hidden_lead<true, true>(tmem + TM_W2, smem_u32(sX2), smem_u32(sU2), 0, lead);
        mma_hidden_lead<true, true>(tmem + TM_W2, smem_u32(sX2), smem_u32(sU2), 1, lead);
        if (lead) umma_commit(&bars[BAR_W2UPD]);
      }
      wait_bar(BAR_W2UPD, par);
      wait_bar(BAR_R, par);                              // MMA3 has read the bf16 W2
      __syncwarp();
      tc_fence_after_sync();
      // ---- b2 += column sums of U2 (bf16 values, the operand the W2 update sees), fp32 accumulate: a thread
      // sums 8 rows of a column pair, threads 0..63 add the eight parts.  bf16 operand copy of the new W2.
      // (The backward's recompute rebuilds the state from another rounding of the same update: see its LN stage.)
      float* part = reinterpret_cast<float*>(smem + OFF_XCHO);
      {
        const int pr = gtid & 31;
        f32x2 acc = 0ull;
#pragma unroll
        for (int r = 0; r < 8; ++r)
          acc = add2(acc, bf16x2_to_f32x2(*reinterpret_cast<const uint32_t*>(
                              sU2 + sw128_off(warp * 8 + r, pr >> 2) + (pr & 3) * 4)));
        *reinterpret_cast<f32x2*>(part + warp * 64 + 2 * pr) = acc;
      }
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        uint32_t v[32];
        tmem_ld32(tmem + lane_base + TM_W2 + wg * 64 + half * 32, v);
        tmem_wait_ld();
        st_cols32(sW2, hrow, half, v);
      }
      publish();
      if (gtid == 128) mbar_arrive(&bars[BAR_W2RDY]);
      if (gtid < 64) {
        float b = sB2[par * 64 + gtid];
#pragma unroll
        for (int k = 0; k < 8; ++k) b += part[k * 64 + gtid];
        sB2[next * 64 + gtid] = b;
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars[BAR_W2RDY]);
      }
      wait_bar(BAR_W1RDY, par);
      __syncwarp();
      // ---- the state after this mini-batch is a checkpoint if the next one starts a group
      if (it + 1 == next_ck) {
        const long ckc = ck;
        ck += 1;
        next_ck = it + 1 + p.cgs < NC ? it + 1 + p.cgs : 0;
        float* W1k = p.W1c + ckc * (64 * 256) + hrow;
        float* W2k = p.W2c + ckc * (256 * 64) + (hrow - lane) * 64;
#pragma unroll 1
        for (int half = 0; half < 2; ++half) {
          uint32_t v[32];
          tmem_ld32(tmem + lane_base + TM_W1 + wg * 64 + half * 32, v);
          tmem_wait_ld();
#pragma unroll
          for (int j = 0; j < 32; ++j) W1k[(half * 32 + j) * 256] = __uint_as_float(v[j]);
          tmem_ld32(tmem + lane_base + TM_W2 + wg * 64 + half * 32, v);
          tmem_wait_ld();
          store_rows_own(W2k + half * 32, v, stage, lane);
        }
        p.b1c[ckc * 256 + hrow] = sB1[next * 256 + hrow];
        if (gtid < 64) p.b2c[ckc * 64 + gtid] = sB2[next * 64 + gtid];
      }
      tc_fence_before_sync();
      if (lane == 0) mbar_arrive(&bars[BAR_SREAD]);
      if (loader && it > 0) {      // the last Out tile has left its stage: Q of the next mini-batch comes in
        tma_wait_group_read<0>();
        load_tile(it + 1, &tmQ, OFF_Q, BAR_Q);
        issued = it + 2;
      }
      wait_bar(BAR_Q + s, it >> 1);

      // ---- MMA5, EPI5: X2b^T = gelu(W1^T Q^T + b1), one 128-row block after the other; the two warps of a quadrant
      // take 32 tokens each.  (Holding EPI5 back until the next mini-batch's EPI1, with which it shares the fp32 and
      // MUFU pipes, has led to MMA2 was 1.5 % slower: it then meets the LayerNorm.)
      auto issue_mma5 = [&](int blk) {
        tc_fence_after_sync();
        mma_hidden_ta<false, false>(tmem + TM_B, tmem + TM_W1B + blk * 32, smem_u32(sQ), lead);
        if (lead) umma_commit(&bars[BAR_ACCB]);
        if (lead && blk == 1) umma_commit(&bars[BAR_W1READ]);
      };
      __syncwarp();
      if (warp == 0) issue_mma5(0);
#pragma unroll
      for (int blk = 0; blk < 2; ++blk) {
        const int row = blk * 128 + quad * 32 + lane;
        const f32x2 bb = pk1(0.5f * sB1[next * 256 + row]);
        wait_bar(BAR_ACCB, blk);
        __syncwarp();
        tc_fence_after_sync();
        uint32_t v[32];
        tmem_ld32(tmem + lane_base + TM_B + wg * 32, v);
        tmem_wait_ld();
        if (blk == 0) {
          tc_fence_before_sync();
          named_bar_sync(kBarO, kGroup);       // the accumulator has been read
          if (warp == 0) issue_mma5(1);
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t g[4];
#pragma unroll
          for (int k = 0; k < 4; ++k)
            g[k] = f32x2_to_bf16x2(gelu_half2(fma2(pk(v[c * 8 + 2 * k], v[c * 8 + 2 * k + 1]), pk1(0.5f), bb)));
          *reinterpret_cast<uint4*>(sX2b + sw128_off(row, wg * 4 + c)) = make_uint4(g[0], g[1], g[2], g[3]);
        }
      }
      publish();

      // ---- MMA6: Z2b = X2b W2
      if (warp == 0) {
        tc_fence_after_sync();
        mma_token_lead(tmem + TM_B, smem_u32(sX2b), smem_u32(sW2), lead);
        if (lead) umma_commit(&bars[BAR_ZB]);
      }
      wait_bar(BAR_ZB, par);
      __syncwarp();
      tc_fence_after_sync();
      // ---- OUT: Q + gamma * LN(Z2b + b2) + beta, over the Q tile (every thread rewrites what it has read)
      {
        TokFrag x;
        uint32_t q[8];
        frag_ld(tm, tmem + TM_B, x);
        frag_ld_raw(tm, sQ, q);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const f32x2 b = frag_col(tm, sB2 + next * 64, j);
          x.a[j] = add2(x.a[j], b);
          x.b[j] = add2(x.b[j], b);
        }
        float rs0, rs1;
        frag_layernorm(tm, x, TTT_LN_EPS, part, kBarPairO, rs0, rs1);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const f32x2 gam = frag_col(tm, sGamma, j), bet = frag_col(tm, sBeta, j);
          x.a[j] = add2(bf16x2_to_f32x2(q[2 * j]), fma2(gam, x.a[j], bet));
          x.b[j] = add2(bf16x2_to_f32x2(q[2 * j + 1]), fma2(gam, x.b[j], bet));
        }
        frag_st_tile(tm, sQ, x);
      }
      fence_proxy_async_smem();
      tc_fence_before_sync();
      const bool stop = named_bar_or(kBarO, kGroup, *abort_flag != 0);
      if (loader) {
        tma_store_2d(&tmOut, sQ, 0, row_of(it));
        tma_commit_group();
      }
      if (stop) break;
    }
    if (loader) {
      if (*abort_flag) drain_loads(BAR_Q, issued);
      tma_wait_group<0>();
    }
  }

  // ---- epilogue: optional final state, then teardown
  tc_fence_before_sync();
  const bool aborted = __syncthreads_or(*abort_flag != 0) != 0;
  tc_fence_after_sync();
  if (!aborted && p.W1f != nullptr) {
    uint32_t v[32];
    if (chain) {
      float* W1o = p.W1f + st_w + hrow;
#pragma unroll 1
      for (int half = 0; half < 2; ++half) {
        tmem_ld32(tmem + lane_base + TM_W1 + wg * 64 + half * 32, v);
        tmem_wait_ld();
#pragma unroll
        for (int j = 0; j < 32; ++j) W1o[(half * 32 + j) * 256] = __uint_as_float(v[j]);
      }
      p.b1f[stream_id * 256 + hrow] = sB1[(NC & 1) * 256 + hrow];
      if (gtid < 64) p.b2f[stream_id * 64 + gtid] = sB2[(NC & 1) * 64 + gtid];
    } else {
      float* W2o = p.W2f + st_w + (hrow - lane) * 64;
#pragma unroll 1
      for (int half = 0; half < 2; ++half) {
        tmem_ld32(tmem + lane_base + TM_W2 + wg * 64 + half * 32, v);
        tmem_wait_ld();
        store_rows_own(W2o + half * 32, v, smem + OFF_STG + warp * 4096, lane);
      }
    }
  }
  if (aborted) {
    // everything this CTA still has in flight is waited for (bounded, not cut short by the abort flag)
    // before its shared and tensor memory go away: the loads above, and the tensor-core work of both issuers
    if ((cta_warp == 0 || cta_warp == 4 || cta_warp == 8) && lead) umma_commit(&bars[BAR_DRAIN]);
    if (tid == 0) {
      mbar_wait_bounded(&bars[BAR_DRAIN], 0, never_flag, limit);
      atomicExch(p.status, static_cast<uint32_t>(TTT_B200_ERR_TIMEOUT));
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (cta_warp == 0) tmem_dealloc(tmem, TM_COLS);
}

}  // namespace

int ttt_launch_forward(const ttt_b200_fwd_args* a, cudaStream_t stream, uint32_t* status, uint64_t limit_ns,
                       int drop_load) {
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
  p.drop_load = drop_load;
  p.status = status;
  p.wait_limit_ns = limit_ns;
  static std::once_flag once[64];
  static cudaError_t attr_err[64];
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return ttt_set_error(TTT_B200_ERR_LAUNCH, "device index out of range");
  std::call_once(once[dev], [&] {
    attr_err[dev] = cudaFuncSetAttribute(ttt_fwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
  });
  if (attr_err[dev] != cudaSuccess) return ttt_set_error(TTT_B200_ERR_LAUNCH, cudaGetErrorString(attr_err[dev]));
  const cudaError_t e = ttt_launch_overlapped(ttt_fwd_kernel, a->B * a->H, kThreads, SMEM_BYTES, stream, tmQ, tmK, tmV, tmOut, p);
  if (e != cudaSuccess) return ttt_set_error(TTT_B200_ERR_LAUNCH, cudaGetErrorString(e));
  return TTT_B200_OK;
}
