// TTT-Linear forward for sm_100a: the operator's mini-batch step with the inner model reduced from the
// two-layer MLP to one linear layer, f(x) = x W + b with W [64 x 64].
//
// The reference ships the TTT-MLP operator only (README.md:18: non-causal, head dimension 64); this
// variant keeps its interface, tensor layouts, checkpoint rule (kernels/ttt/matching.py:223-228) and the
// fused LayerNorm + L2 step of kernels/ttt/matching.py:67-101, and drops the hidden layer.  Per mini-batch
// (K, V, Q: 64 x 64 bf16 tiles, eta: 64 bf16):
//
//   MMA1  Z  = K W                              [64 tok x 64]
//   LN    x = LN(Z + b); e = gamma x + beta - (V - K); U = -eta * dl/dZ (the LayerNorm backward of
//         e * gamma)                            -> smem bf16;  b += column sums of U
//   MMA2  W^T += U^T K                          (accumulated into the fp32 state in tensor memory)
//   EPI   bf16 operand copy of the new W^T      -> smem
//   MMA3  Zb = Q W
//   OUT   Out = Q + gamma * LN(Zb + b) + beta   -> global
//
// Before mini-batch i with i % checkpoint_group_size == 0 the state (W, b) is stored as checkpoint
// i / checkpoint_group_size.  One CTA per (batch, head) stream, in one of two forms
// chosen by the launcher: of two groups of 256 threads when there are no more streams than SMs (namespace pair), else of
// one such group; every tile is 64 x 64, read
// out of tensor memory as the 16x256b fragments of TokMap by all eight warps; up to three CTAs share an SM
// when there are more streams than SMs (72 KB of shared memory with a two-stage input ring, 128
// tensor-memory columns, 80 registers per thread each), which hides the latency of the three dependent MMA
// phases (measured at
// 1536 streams of 64 mini-batches: 1.43 ms with two CTAs per SM and a three-stage ring, 1.34 ms with three, 1.04-1.10 with
// packed epilogues; issue slots 56 %, fp32 pipe 40 %, DRAM 36 %).  All waits are bounded; on expiry the CTA reports
// through the status word, drains its own copies, frees its tensor memory and returns.
#include <mutex>

#include "ttt_cluster.cuh"
#include "ttt_internal.h"

using namespace tttcl;

namespace {

constexpr int kStages = 2;
constexpr int kThreads = 256;
constexpr int kProd = 128;     // issues the bulk copies; not the MMA issuer (lane 0 of warp 0)

constexpr uint32_t OFF_K = 0;
constexpr uint32_t OFF_V = OFF_K + kStages * TILE;
constexpr uint32_t OFF_Q = OFF_V + kStages * TILE;
constexpr uint32_t OFF_W = OFF_Q + kStages * TILE;      // bf16 W^T: row = output feature, column = input feature
constexpr uint32_t OFF_U = OFF_W + TILE;                // bf16 U: row = token
constexpr uint32_t OFF_ETA = OFF_U + TILE;
constexpr uint32_t OFF_B = OFF_ETA + kStages * 128;
constexpr uint32_t OFF_GAMMA = OFF_B + 256;
constexpr uint32_t OFF_BETA = OFF_GAMMA + 256;
constexpr uint32_t OFF_BAR = OFF_BETA + 256;
constexpr uint32_t OFF_MISC = OFF_BAR + 64;
constexpr uint32_t OFF_XCH = OFF_MISC + 64;             // row-sum exchange between warp pairs
constexpr uint32_t OFF_CS = OFF_XCH + kXchBytes;        // fp32[4][64] column sums, one row per quadrant
constexpr uint32_t SMEM_USED = OFF_CS + 1024;
constexpr uint32_t SMEM_BYTES = SMEM_USED + 1024;       // slack for the 1024-byte alignment
static_assert(3 * (SMEM_BYTES + 1024) <= 233472, "three CTAs per SM");

constexpr uint32_t TM_W = 0;
constexpr uint32_t TM_Z = 64;
constexpr uint32_t TM_COLS = 128;

struct LinParams {
  const __nv_bfloat16* eta;
  const float* gamma;
  const float* beta;
  const float* W;
  const float* b;
  float* Wc;
  float* bc;
  float* Wf;
  float* bf;
  __nv_bfloat16* out;
  int H, NC, cgs, nck;
  int drop_load;            // test only: mini-batch whose loads stream 0 never issues (-1: none)
  uint32_t* status;
  uint64_t wait_limit_ns;
};

// LN: fused LayerNorm + L2 gradient of the accumulator at `acc`, U = -eta * dl/dZ, and its column sums, one row of
// `cs` (fp32[4][64]) per quadrant (in registers: four N = 8 MMAs behind the update would cost as much latency as a
// whole product).  `bar`: first of the group's four pair barriers.
__device__ __forceinline__ void lin_ln(const TokMap& tm, int lane, uint32_t acc, const uint8_t* sK, const uint8_t* sV,
                                       const __nv_bfloat16* sEta, const float* b_vec, const float* sGamma, const float* sBeta,
                                       float* xch, uint32_t bar, uint8_t* sU, float* sCS) {
  TokFrag x, g;
  uint32_t kk[8], vv[8];
  frag_ld(tm, acc, x);
  frag_ld_raw(tm, sK, kk);
  frag_ld_raw(tm, sV, vv);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const f32x2 b = frag_col(tm, b_vec, j);
    x.a[j] = add2(x.a[j], b);
    x.b[j] = add2(x.b[j], b);
  }
  float rs0, rs1;
  frag_layernorm(tm, x, TTT_LN_EPS, xch, bar, rs0, rs1);
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
  frag_allreduce2<1>(tm, a, b, xch, bar);
  const f32x2 sc0 = pk1(-__bfloat162float(sEta[tm.r0]) * rs0 * (1.f / 64.f));
  const f32x2 sc1 = pk1(-__bfloat162float(sEta[tm.r1]) * rs1 * (1.f / 64.f));
  f32x2 su[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    g.a[j] = mul2(fma2(x.a[j], pk1(-a[1]), fma2(g.a[j], pk1(64.f), pk1(-a[0]))), sc0);
    g.b[j] = mul2(fma2(x.b[j], pk1(-b[1]), fma2(g.b[j], pk1(64.f), pk1(-b[0]))), sc1);
    su[j] = add2(g.a[j], g.b[j]);
  }
  frag_st_tile(tm, sU, g);
  sCS[tm.quad * 64 + frag_colsum_col(tm, lane)] = frag_colsum(su, lane);
}
// OUT: x = Q + gamma * LN(Zb + b) + beta
__device__ __forceinline__ void lin_out(const TokMap& tm, uint32_t acc, const uint8_t* sQ, const float* b_vec,
                                        const float* sGamma, const float* sBeta, float* xch, uint32_t bar, TokFrag& x) {
  uint32_t q[8];
  frag_ld(tm, acc, x);
  frag_ld_raw(tm, sQ, q);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const f32x2 b = frag_col(tm, b_vec, j);
    x.a[j] = add2(x.a[j], b);
    x.b[j] = add2(x.b[j], b);
  }
  float rs0, rs1;
  frag_layernorm(tm, x, TTT_LN_EPS, xch, bar, rs0, rs1);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const f32x2 gam = frag_col(tm, sGamma, j), bet = frag_col(tm, sBeta, j);
    x.a[j] = add2(bf16x2_to_f32x2(q[2 * j]), fma2(gam, x.a[j], bet));
    x.b[j] = add2(bf16x2_to_f32x2(q[2 * j + 1]), fma2(gam, x.b[j], bet));
  }
}

__global__ void __launch_bounds__(kThreads, 3)
ttt_linear_fwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                      const __grid_constant__ CUtensorMap tmV, const LinParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_align_1024(smem_raw);

  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const TokMap tm(warp, lane);
  const long stream_id = blockIdx.x;
  const int head = static_cast<int>(stream_id % p.H);

  uint8_t* sW = smem + OFF_W;
  uint8_t* sU = smem + OFF_U;
  float* sB = reinterpret_cast<float*>(smem + OFF_B);
  float* sGamma = reinterpret_cast<float*>(smem + OFF_GAMMA);
  float* sBeta = reinterpret_cast<float*>(smem + OFF_BETA);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + OFF_BAR);   // [kStages]
  uint64_t* mma_bar = full + kStages;
  uint64_t* drain_bar = mma_bar + 1;        // abort path only
  float* sXch = reinterpret_cast<float*>(smem + OFF_XCH);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + OFF_MISC);
  volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(smem + OFF_MISC + 4);
  volatile uint32_t* never_flag = reinterpret_cast<volatile uint32_t*>(smem + OFF_MISC + 8);   // stays 0

  const uint64_t limit = p.wait_limit_ns;
  const int NC = p.NC;

  if (tid == kProd) {
    for (int s = 0; s < kStages; ++s) mbar_init(&full[s], 1);
    mbar_init(mma_bar, 1);
    mbar_init(drain_bar, 1);
    fence_mbar_init();
    *abort_flag = 0;
    *never_flag = 0;
    prefetch_tmap(&tmQ);
    prefetch_tmap(&tmK);
    prefetch_tmap(&tmV);
  }
  if (warp == 0) {
    tmem_alloc(tmem_slot, TM_COLS);
    tmem_relinquish();
  }
  if (tid < 64) {
    sGamma[tid] = p.gamma[head * 64 + tid];
    sBeta[tid] = p.beta[head * 64 + tid];
    sB[tid] = p.b[stream_id * 64 + tid];
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot;

  auto issue_loads = [&](int i) {   // thread kProd only
    if (i == p.drop_load && stream_id == 0) return;
    const int s = i % kStages;
    const int row0 = static_cast<int>((stream_id * NC + i) * 64);
    mbar_expect_tx(&full[s], 3 * TILE + 128);
    tma_load_2d(smem + OFF_K + s * TILE, &tmK, &full[s], 0, row0);
    tma_load_2d(smem + OFF_V + s * TILE, &tmV, &full[s], 0, row0);
    tma_load_2d(smem + OFF_Q + s * TILE, &tmQ, &full[s], 0, row0);
    bulk_load_1d(smem + OFF_ETA + s * 128, p.eta + (stream_id * NC + i) * 64, 128, &full[s]);
  };
  int loads_issued = 0;
  if (tid == kProd) {
    for (; loads_issued < kStages && loads_issued < NC; ++loads_issued) issue_loads(loads_issued);
  }

  // ---- state <-> global memory.  W is [64 in][64 out] in global memory; the fragment of W^T holds output
  // features r0 / r1 (rows) and, for j = 0..3, the input-feature pair col(j), col(j) + 1.
  auto load_state = [&](const float* Wg) {
    float w[16];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int c = tm.col(j);
      w[4 * j] = Wg[c * 64 + tm.r0];
      w[4 * j + 1] = Wg[(c + 1) * 64 + tm.r0];
      w[4 * j + 2] = Wg[c * 64 + tm.r1];
      w[4 * j + 3] = Wg[(c + 1) * 64 + tm.r1];
    }
    tok_st_tmem(tm, tmem + TM_W, w);
    tok_st_tile(tm, sW, w);
  };
  auto store_state = [&](float* Wo, float* bo) {
    float w[16];
    tok_ld(tm, tmem + TM_W, w);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int c = tm.col(j);
      Wo[c * 64 + tm.r0] = w[4 * j];
      Wo[(c + 1) * 64 + tm.r0] = w[4 * j + 1];
      Wo[c * 64 + tm.r1] = w[4 * j + 2];
      Wo[(c + 1) * 64 + tm.r1] = w[4 * j + 3];
    }
    if (tid < 64) bo[tid] = sB[tid];
  };
  load_state(p.W + stream_id * 4096);
  tmem_wait_st();
  fence_proxy_async_smem();
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();

  uint32_t mma_phase = 0;
  auto wait_mma = [&]() {
    mbar_wait_bounded(mma_bar, mma_phase, abort_flag, limit);
    mma_phase ^= 1;
    __syncwarp();
    tc_fence_after_sync();
  };
  auto publish = [&]() {
    fence_proxy_async_smem();
    tc_fence_before_sync();
    __syncthreads();
  };
  const uint32_t lead = elect_one() ? 1u : 0u;      // the lane of warp 0 that issues the MMAs
  float* sCS = reinterpret_cast<float*>(smem + OFF_CS);

  int it = 0;
  for (; it < NC; ++it) {
    const int s = it % kStages;
    const uint8_t* sK = smem + OFF_K + s * TILE;
    const uint8_t* sV = smem + OFF_V + s * TILE;
    const uint8_t* sQ = smem + OFF_Q + s * TILE;
    const __nv_bfloat16* sEta = reinterpret_cast<const __nv_bfloat16*>(smem + OFF_ETA + s * 128);
    mbar_wait_bounded(&full[s], (it / kStages) & 1, abort_flag, limit);

    // ---- MMA1: Z = K W
    if (warp == 0) {
      tc_fence_after_sync();
      mma_64_lead<false, false>(tmem + TM_Z, smem_u32(sK), smem_u32(sW), lead);
      if (lead) umma_commit(mma_bar);
    }
    // a checkpoint (the state before this mini-batch) leaves while MMA1 runs: it only reads the state
    if (it % p.cgs == 0) {
      const long ckc = stream_id * p.nck + it / p.cgs;
      store_state(p.Wc + ckc * 4096, p.bc + ckc * 64);
      tc_fence_before_sync();      // the state columns are written by the second MMA group
    }
    wait_mma();
    lin_ln(tm, lane, tmem + TM_Z, sK, sV, sEta, sB, sGamma, sBeta, sXch, 1, sU, sCS);
    publish();

    // ---- MMA2: W^T += U^T K;  b += column sums of U
    if (warp == 0) {
      tc_fence_after_sync();
      mma_64_tn_lead(tmem + TM_W, smem_u32(sU), smem_u32(sK), lead);
      if (lead) umma_commit(mma_bar);
    }
    if (tid < 64) sB[tid] += (sCS[tid] + sCS[64 + tid]) + (sCS[128 + tid] + sCS[192 + tid]);     // read after the barrier below
    wait_mma();
    // ---- EPI: refresh the bf16 operand copy of the state
    {
      TokFrag w;
      frag_ld(tm, tmem + TM_W, w);
      frag_st_tile(tm, sW, w);
    }
    publish();

    // ---- MMA3: Zb = Q W
    if (warp == 0) {
      tc_fence_after_sync();
      mma_64_lead<false, false>(tmem + TM_Z, smem_u32(sQ), smem_u32(sW), lead);
      if (lead) umma_commit(mma_bar);
    }
    wait_mma();
    // ---- OUT, straight to global memory
    {
      TokFrag x;
      lin_out(tm, tmem + TM_Z, sQ, sB, sGamma, sBeta, sXch, 1, x);
      frag_st_global(tm, p.out + (stream_id * NC + it) * 4096, x);
    }
    // every warp has read this stage's tiles and the tensor-memory tile: the stage takes the loads of the
    // mini-batch kStages ahead, and all threads take the same decision on leaving the loop
    tc_fence_before_sync();
    const bool stop = __syncthreads_or(*abort_flag != 0) != 0;
    if (stop) break;
    if (tid == kProd && loads_issued < NC && loads_issued == it + kStages) {
      issue_loads(loads_issued);
      ++loads_issued;
    }
  }

  // ---- epilogue: optional final state, then teardown
  const bool aborted = __syncthreads_or(*abort_flag != 0) != 0;
  if (!aborted && p.Wf != nullptr) store_state(p.Wf + stream_id * 4096, p.bf + stream_id * 64);
  if (aborted) {
    // everything this CTA still has in flight is waited for (bounded, not cut short by the abort flag)
    // before its shared and tensor memory go away: the issuer's tensor-core work ...
    if (warp == 0 && lead) umma_commit(drain_bar);
    if (tid == kProd) {
      mbar_wait_bounded(drain_bar, 0, never_flag, limit);
      // ... and its own loads
      for (int j = it; j < loads_issued; ++j) {
        if (j == p.drop_load && stream_id == 0) continue;
        mbar_wait_bounded(&full[j % kStages], (j / kStages) & 1, never_flag, limit);
      }
      atomicExch(p.status, static_cast<uint32_t>(TTT_B200_ERR_TIMEOUT));
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, TM_COLS);
}

// ---- The form for launches with no more streams than SMs: nothing but the stream itself could fill its SM, so the
// output pass runs on eight warps of its own beside the chain of the other eight (Z -> U -> state -> bf16 copy), one step
// behind, as in the MLP forward (148 streams of 64 mini-batches: 2.8 -> 1.95 us per mini-batch; bound by the latency of
// the chain, two products and the LayerNorm with its two exchanges: issue slots 45 %, tensor pipe 10 %).  Two copies of the
// bf16 state alternate, so that the chain does not wait for the output product; the output group also stores the
// checkpoints.
namespace pair {

constexpr int kGroup = 256;
constexpr uint32_t kBarPairC = 1, kBarPairO = 5, kBarC = 9, kBarO = 10;     // named barriers
constexpr uint32_t OFF_K = 0;
constexpr uint32_t OFF_V = OFF_K + 2 * TILE;
constexpr uint32_t OFF_Q = OFF_V + 2 * TILE;            // Q, then Out on its way to global memory
constexpr uint32_t OFF_W = OFF_Q + 2 * TILE;            // bf16 W^T before / after the update
constexpr uint32_t OFF_U = OFF_W + 2 * TILE;
constexpr uint32_t OFF_ETA = OFF_U + TILE;
constexpr uint32_t OFF_B = OFF_ETA + 256;               // fp32[2][64] likewise
constexpr uint32_t OFF_GAMMA = OFF_B + 512;
constexpr uint32_t OFF_BETA = OFF_GAMMA + 256;
constexpr uint32_t OFF_XC = OFF_BETA + 256;
constexpr uint32_t OFF_XO = OFF_XC + kXchBytes;
constexpr uint32_t OFF_CS = OFF_XO + kXchBytes;
constexpr uint32_t OFF_BAR = OFF_CS + 1024;
constexpr uint32_t OFF_MISC = OFF_BAR + 128;
constexpr uint32_t SMEM_USED = OFF_MISC + 64;
constexpr uint32_t SMEM_BYTES = SMEM_USED + 1024;

constexpr int BAR_KV = 0, BAR_Q = 2;                    // + stage
constexpr int BAR_C = 4;                                // chain's products: two uses per mini-batch
constexpr int BAR_O = 5;                                // output product
constexpr int BAR_WRDY = 6, BAR_SREAD = 7, BAR_DRAIN = 8;
constexpr int kBars = 9;

constexpr uint32_t TM_W = 0, TM_Z = 64, TM_ZB = 128, TM_COLS = 256;

__global__ void __launch_bounds__(2 * kGroup, 1)
ttt_linear_fwd_pair_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                           const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmOut,
                           const LinParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_align_1024(smem_raw);
  const int tid = threadIdx.x, lane = tid & 31;
  const int cta_warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int warp = cta_warp & 7;
  const int gtid = tid & (kGroup - 1);
  const bool loader = gtid == 128;
  const TokMap tm(warp, lane);
  const long stream_id = blockIdx.x;
  const int head = static_cast<int>(stream_id % p.H);
  const int NC = p.NC;
  auto tile = [&](uint32_t off, int s) { return smem + off + s * TILE; };
  auto vec = [&](uint32_t off) { return reinterpret_cast<float*>(smem + off); };
  float* sB = vec(OFF_B);
  float* sGamma = vec(OFF_GAMMA);
  float* sBeta = vec(OFF_BETA);
  float* sCS = vec(OFF_CS);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + OFF_BAR);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + OFF_MISC);
  volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(smem + OFF_MISC + 4);
  volatile uint32_t* never_flag = reinterpret_cast<volatile uint32_t*>(smem + OFF_MISC + 8);   // stays 0
  const uint64_t limit = p.wait_limit_ns;
  const bool chain = cta_warp < 8;

  if (tid == 0) {
    for (int i = 0; i < kBars; ++i) mbar_init(&bars[i], i == BAR_SREAD ? 8 : i == BAR_DRAIN ? 2 : 1);
    fence_mbar_init();
    *abort_flag = 0;
    *never_flag = 0;
    prefetch_tmap(&tmQ);
    prefetch_tmap(&tmK);
    prefetch_tmap(&tmV);
    prefetch_tmap(&tmOut);
  }
  if (cta_warp == 8) {
    tmem_alloc(tmem_slot, TM_COLS);
    tmem_relinquish();
  }
  griddep_launch();
  griddep_wait();
  if (tid < 64) {
    sGamma[tid] = p.gamma[head * 64 + tid];
    sBeta[tid] = p.beta[head * 64 + tid];
    sB[tid] = p.b[stream_id * 64 + tid];
  }
  // the chain group's part of W comes in meanwhile (fragment of W^T: see the other form)
  float w0[16];
  auto store_frag = [&](float* Wo, const float (&w)[16]) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int c = tm.col(j);
      Wo[c * 64 + tm.r0] = w[4 * j];
      Wo[(c + 1) * 64 + tm.r0] = w[4 * j + 1];
      Wo[c * 64 + tm.r1] = w[4 * j + 2];
      Wo[(c + 1) * 64 + tm.r1] = w[4 * j + 3];
    }
  };
  if (chain) {
    const float* Wg = p.W + stream_id * 4096;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int c = tm.col(j);
      w0[4 * j] = Wg[c * 64 + tm.r0];
      w0[4 * j + 1] = Wg[(c + 1) * 64 + tm.r0];
      w0[4 * j + 2] = Wg[c * 64 + tm.r1];
      w0[4 * j + 3] = Wg[(c + 1) * 64 + tm.r1];
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  const uint32_t lead = elect_one() ? 1u : 0u;
  auto wait_bar = [&](int b, uint32_t parity) { mbar_wait_bounded(&bars[b], parity & 1u, abort_flag, limit); };
  auto mma_seen = [&]() {
    __syncwarp();
    tc_fence_after_sync();
  };
  auto dropped = [&](int i) { return i == p.drop_load && stream_id == 0; };
  auto row_of = [&](int i) { return static_cast<int>((stream_id * NC + i) * 64); };
  auto load_kv = [&](int i) {
    if (i >= NC || dropped(i)) return;
    const int s = i & 1;
    mbar_expect_tx(&bars[BAR_KV + s], 2 * TILE + 128);
    tma_load_2d(tile(OFF_K, s), &tmK, &bars[BAR_KV + s], 0, row_of(i));
    tma_load_2d(tile(OFF_V, s), &tmV, &bars[BAR_KV + s], 0, row_of(i));
    bulk_load_1d(smem + OFF_ETA + s * 128, p.eta + (stream_id * NC + i) * 64, 128, &bars[BAR_KV + s]);
  };
  auto load_q = [&](int i) {
    if (i >= NC || dropped(i)) return;
    mbar_expect_tx(&bars[BAR_Q + (i & 1)], TILE);
    tma_load_2d(tile(OFF_Q, i & 1), &tmQ, &bars[BAR_Q + (i & 1)], 0, row_of(i));
  };
  // abort path: the loads that may still be in flight, the last one of each stage
  auto drain_loads = [&](int bar, int issued) {
    for (int i = issued > 2 ? issued - 2 : 0; i < issued && i < NC; ++i)
      if (!dropped(i)) mbar_wait_bounded(&bars[bar + (i & 1)], (i >> 1) & 1, never_flag, limit);
  };
  int it = 0;
  int issued = 2;

  if (chain) {
    if (loader) {
      load_kv(0);
      load_kv(1);
    }
    tok_st_tmem(tm, tmem + TM_W, w0);
    tok_st_tile(tm, tile(OFF_W, 0), w0);
    store_frag(p.Wc + stream_id * p.nck * 4096, w0);
    if (gtid < 64) p.bc[stream_id * p.nck * 64 + gtid] = sB[gtid];
    tmem_wait_st();
    auto publish = [&]() {
      fence_proxy_async_smem();
      tc_fence_before_sync();
      named_bar_sync(kBarC, kGroup);
    };
    publish();
    for (; it < NC; ++it) {
      const int s = it & 1;
      const uint32_t par = it & 1, prev = par ^ 1u;
      wait_bar(BAR_KV + s, it >> 1);
      // ---- MMA1: Z = K W
      if (cta_warp == 0) {
        tc_fence_after_sync();
        mma_64_lead<false, false>(tmem + TM_Z, smem_u32(tile(OFF_K, s)), smem_u32(tile(OFF_W, s)), lead);
        if (lead) umma_commit(&bars[BAR_C]);
      }
      wait_bar(BAR_C, 0);
      mma_seen();
      lin_ln(tm, lane, tmem + TM_Z, tile(OFF_K, s), tile(OFF_V, s), reinterpret_cast<const __nv_bfloat16*>(smem + OFF_ETA) + s * 64,
             sB + par * 64, sGamma, sBeta, vec(OFF_XC), kBarPairC, smem + OFF_U, sCS);
      publish();
      // ---- MMA2: W^T += U^T K;  b += column sums of U.  The output group has read the state of the last
      // step; it was through with the step before, whose b and bf16 copy are written over now.
      if (it > 0) wait_bar(BAR_SREAD, prev);
      if (cta_warp == 0) {
        mma_seen();
        mma_64_tn_lead(tmem + TM_W, smem_u32(smem + OFF_U), smem_u32(tile(OFF_K, s)), lead);
        if (lead) umma_commit(&bars[BAR_C]);
      }
      if (gtid < 64)
        sB[prev * 64 + gtid] = sB[par * 64 + gtid] + ((sCS[gtid] + sCS[64 + gtid]) + (sCS[128 + gtid] + sCS[192 + gtid]));
      wait_bar(BAR_C, 1);
      mma_seen();
      // ---- EPI: bf16 copy of the new state
      {
        TokFrag w;
        frag_ld(tm, tmem + TM_W, w);
        frag_st_tile(tm, tile(OFF_W, s ^ 1), w);
      }
      fence_proxy_async_smem();
      tc_fence_before_sync();
      const bool stop = named_bar_or(kBarC, kGroup, *abort_flag != 0);
      if (gtid == 0) mbar_arrive(&bars[BAR_WRDY]);
      if (stop) break;
      if (loader) {
        load_kv(it + 2);
        issued = it + 3;
      }
    }
    if (loader && *abort_flag) drain_loads(BAR_KV, issued);
  } else {
    if (loader) {
      load_q(0);
      load_q(1);
    }
    for (; it < NC; ++it) {
      const int s = it & 1;
      const uint32_t par = it & 1, next = par ^ 1u;
      uint8_t* sQ = tile(OFF_Q, s);
      wait_bar(BAR_WRDY, par);
      mma_seen();
      if (it + 1 < NC && (it + 1) % p.cgs == 0) {      // the state after this mini-batch is a checkpoint
        const long ckc = stream_id * p.nck + (it + 1) / p.cgs;
        float w[16];
        tok_ld(tm, tmem + TM_W, w);
        store_frag(p.Wc + ckc * 4096, w);
        if (gtid < 64) p.bc[ckc * 64 + gtid] = sB[next * 64 + gtid];
      }
      tc_fence_before_sync();
      if (lane == 0) mbar_arrive(&bars[BAR_SREAD]);
      if (loader && it > 0) {      // the last Out tile has left its stage: Q of the next mini-batch comes in
        tma_wait_group_read<0>();
        load_q(it + 1);
        issued = it + 2;
      }
      wait_bar(BAR_Q + s, it >> 1);
      // ---- MMA3: Zb = Q W
      if (cta_warp == 8) {
        mma_seen();
        mma_64_lead<false, false>(tmem + TM_ZB, smem_u32(sQ), smem_u32(tile(OFF_W, s ^ 1)), lead);
        if (lead) umma_commit(&bars[BAR_O]);
      }
      wait_bar(BAR_O, par);
      mma_seen();
      TokFrag x;
      lin_out(tm, tmem + TM_ZB, sQ, sB + next * 64, sGamma, sBeta, vec(OFF_XO), kBarPairO, x);
      frag_st_tile(tm, sQ, x);       // over Q (every thread rewrites what it has read)
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

  tc_fence_before_sync();
  const bool aborted = __syncthreads_or(*abort_flag != 0) != 0;
  tc_fence_after_sync();
  if (!aborted && p.Wf != nullptr && chain) {
    float w[16];
    tok_ld(tm, tmem + TM_W, w);
    store_frag(p.Wf + stream_id * 4096, w);
    if (gtid < 64) p.bf[stream_id * 64 + gtid] = sB[(NC & 1) * 64 + gtid];
  }
  if (aborted) {
    // everything this CTA still has in flight is waited for (bounded) before its shared and tensor memory go away: the
    // loads above, and the tensor-core work of both issuers
    if (warp == 0 && lead) umma_commit(&bars[BAR_DRAIN]);
    if (tid == 0) {
      mbar_wait_bounded(&bars[BAR_DRAIN], 0, never_flag, limit);
      atomicExch(p.status, static_cast<uint32_t>(TTT_B200_ERR_TIMEOUT));
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (cta_warp == 8) tmem_dealloc(tmem, TM_COLS);
}

}  // namespace pair

}  // namespace

int ttt_launch_linear_forward(const ttt_b200_linear_fwd_args* a, cudaStream_t stream, uint32_t* status,
                              uint64_t limit_ns, int drop_load) {
  const uint64_t rows = static_cast<uint64_t>(a->B) * a->H * a->NC * 64;
  CUtensorMap tmQ, tmK, tmV;
  if (int rc = ttt_make_tile_map(&tmQ, a->XQ, rows)) return rc;
  if (int rc = ttt_make_tile_map(&tmK, a->XK, rows)) return rc;
  if (int rc = ttt_make_tile_map(&tmV, a->XV, rows)) return rc;
  LinParams p;
  p.eta = static_cast<const __nv_bfloat16*>(a->last_eta);
  p.gamma = a->ttt_norm_weight;
  p.beta = a->ttt_norm_bias;
  p.W = a->W1; p.b = a->b1;
  p.Wc = a->W1_checkpoints; p.bc = a->b1_checkpoints;
  const bool want_final = a->W1_final && a->b1_final;
  p.Wf = want_final ? a->W1_final : nullptr;
  p.bf = a->b1_final;
  p.out = static_cast<__nv_bfloat16*>(a->Out);
  p.H = a->H; p.NC = a->NC; p.cgs = a->checkpoint_group_size; p.nck = a->num_checkpoints;
  p.drop_load = drop_load;
  p.status = status;
  p.wait_limit_ns = limit_ns;
  static std::once_flag once[64];
  static cudaError_t attr_err[64];
  static int sms[64];
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return ttt_set_error(TTT_B200_ERR_LAUNCH, "device index out of range");
  std::call_once(once[dev], [&] {
    attr_err[dev] = cudaFuncSetAttribute(ttt_linear_fwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
    if (attr_err[dev] == cudaSuccess)
      attr_err[dev] = cudaFuncSetAttribute(pair::ttt_linear_fwd_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           pair::SMEM_BYTES);
    sms[dev] = 148;
    cudaDeviceGetAttribute(&sms[dev], cudaDevAttrMultiProcessorCount, dev);
  });
  if (attr_err[dev] != cudaSuccess) return ttt_set_error(TTT_B200_ERR_LAUNCH, cudaGetErrorString(attr_err[dev]));
  // no more streams than SMs: one CTA of two groups per stream.  Beyond that two or three plain CTAs share an SM and fill
  // each other's waits (296 streams: 3.5 us per mini-batch of all, against 2 x 1.95 in two turns of the form above).
  cudaError_t e;
  if (a->B * a->H <= sms[dev]) {
    CUtensorMap tmOut;
    if (int rc = ttt_make_tile_map(&tmOut, a->Out, rows)) return rc;
    e = ttt_launch_overlapped(pair::ttt_linear_fwd_pair_kernel, a->B * a->H, 2 * pair::kGroup, pair::SMEM_BYTES, stream, tmQ,
                              tmK, tmV, tmOut, p);
  } else {
    // not overlapped: CTAs placed while the predecessor's still fill most slots would crowd on the SMs that are free first
    ttt_linear_fwd_kernel<<<dim3(a->B * a->H), dim3(kThreads), SMEM_BYTES, stream>>>(tmQ, tmK, tmV, p);
    e = cudaGetLastError();
  }
  if (e != cudaSuccess) return ttt_set_error(TTT_B200_ERR_LAUNCH, cudaGetErrorString(e));
  return TTT_B200_OK;
}
