// TTT-Linear backward for sm_100a: gradients of the TTT-Linear forward (ttt_linear_fwd_sm100.cu) from its
// checkpoints, one persistent CTA of 16 warps per (batch, head) stream.
//
// The reference has no counterpart (it ships the TTT-MLP operator only, README.md:18); the structure is its
// backward's (kernels/ttt_backward/ttt.cu:453-1424, math kernels/ttt_backward/matching.py:173-342) with the
// hidden layer removed: per checkpoint group, last to first, recompute the group's mini-batches from the
// checkpoint, keeping what the reverse sweep needs in the caller's scratch buffer, then sweep the group in
// reverse.  Every tile is 64 x 64: token-major tiles and the 64 x 64 state alike are M = 64 accumulators read
// with the 16x256b fragments of TokMap by eight warps.  The state W^T and the gradient state
// G^T = (dL/dW)^T live side by side in tensor memory as the accumulators of their own update MMAs, b and dL/db in
// shared memory.
//
// The recompute of one group does not depend on the sweep of another, so the two run side by side: eight warps
// recompute group g - 1 while the other eight sweep group g, each a chain of short MMA -> epilogue round trips that
// alone would leave the SM idle most of the time.  One slot of scratch per mini-batch of a group is enough for both:
// the sweep frees the slots of its group from the last mini-batch to the first, so every other group numbers its
// slots backwards and the recompute fills them in the order in which they become free.
//
//   recompute of mini-batch j                              reverse step of mini-batch j, go = dL/dOut
//   MMA1  Z = K W                                          P1  dK(j+1) += gZin W^T;  G^T += gZin^T K   (of step j + 1)
//   LN    x_f = LN(Z + b), e = gamma x_f + beta - (V - K)      G^T += gZb^T Q;  G_b += column sums of gZb
//         gZ = LNbwd(e gamma), U = -eta gZ                 E2  bf16 copy of G^T
//   MMA2  W^T += U^T K, b += colsum U                      P2  K G, T1 = gZ G^T
//   EPI   bf16 copy of W+^T                                E4  A1 = -eta (K G + G_b), second order through the fused
//   MMA3  Zb = Q W+                                            LayerNorm + L2 gradient: Bt, d_gamma, d_beta,
//   LNB   x_l = LN(Zb + b+), gZb = LNbwd(go gamma; x_l),       dV = -gamma Bt, gZin, d_eta; G_b += column sums of gZin
//         d_beta += colsum go, d_gamma += colsum go x_l
//   MMA4  gZb W+^T;  dQ = go + .
//   slot <- bf16 W^T before the update, x_f, gZ, gZb (raw images of the swizzled shared-memory tiles, stored and read
//   back with bulk copies), 1/std of the fused LayerNorm, the column sums of gZb.
//
// What bounds it: the latency of the two chains and their shared issue slots (16.2 k warp-instructions per mini-batch,
// most in token-major epilogues; 128 streams: issue slots 50 %, fp32 pipe 34 %, DRAM 33 %, tensor pipe 12 %).  Measured
// at 128 streams: 8.4 us per mini-batch as one chain of eight warps, 5.3 with the recompute beside the sweep, 4.5 with
// packed epilogues and shared-space addresses.  All waits are bounded; on expiry the CTA
// reports through the status word, drains its own copies, frees its tensor memory and returns.
#include <mutex>

#include "ttt_cluster.cuh"
#include "ttt_internal.h"

using namespace tttcl;

namespace {

constexpr int kGroup = 256;
constexpr int kThreads = 2 * kGroup;
constexpr uint32_t kBarPairR = 1, kBarPairS = 5, kBarR = 9, kBarS = 10;     // named barriers

// scratch slot (one per mini-batch of a checkpoint group and stream)
constexpr uint32_t SL_W = 0;
constexpr uint32_t SL_XF = TILE;
constexpr uint32_t SL_GZ = 2 * TILE;
constexpr uint32_t SL_GZB = 3 * TILE;
constexpr uint32_t SL_VEC = 4 * TILE;          // fp32[64] 1/std of the fused LayerNorm, fp32[64] column sums of gZb
constexpr uint32_t SLOT_BYTES = 4 * TILE + 512;

// shared memory
constexpr uint32_t OFF_RK = 0;                          // recompute: + stage
constexpr uint32_t OFF_RQ = OFF_RK + 2 * TILE;
constexpr uint32_t OFF_RV = OFF_RQ + 2 * TILE;          // V, then x_f on its way out
constexpr uint32_t OFF_RGO = OFF_RV + 2 * TILE;         // dL/dOut, then dQ on its way out
constexpr uint32_t OFF_RW = OFF_RGO + 2 * TILE;         // bf16 W^T before / after the update
constexpr uint32_t OFF_RGZ = OFF_RW + 2 * TILE;
constexpr uint32_t OFF_RU = OFF_RGZ + TILE;             // U, then gZb
constexpr uint32_t OFF_SK = OFF_RU + TILE;              // sweep: + stage
constexpr uint32_t OFF_SQ = OFF_SK + 2 * TILE;
constexpr uint32_t OFF_SV = OFF_SQ + TILE;              // + stage: V, then dV on its way out
constexpr uint32_t OFF_SXF = OFF_SV + 2 * TILE;         // + stage
constexpr uint32_t OFF_SGZ = OFF_SXF + 2 * TILE;        // + stage
constexpr uint32_t OFF_SGZB = OFF_SGZ + 2 * TILE;
constexpr uint32_t OFF_SWP = OFF_SGZB + TILE;           // bf16 W^T before the update
constexpr uint32_t OFF_SG = OFF_SWP + TILE;             // bf16 G^T
constexpr uint32_t OFF_SZIN = OFF_SG + TILE;
constexpr uint32_t OFF_SDK = OFF_SZIN + TILE;           // dK on its way out
constexpr uint32_t OFF_RETA = OFF_SDK + TILE;           // bf16[2][64]
constexpr uint32_t OFF_SETA = OFF_RETA + 256;           // bf16[2][64]
constexpr uint32_t OFF_RVEC = OFF_SETA + 256;           // fp32[2][128]: the slot's vectors on their way out
constexpr uint32_t OFF_SVEC = OFF_RVEC + 1024;          // fp32[2][128]
constexpr uint32_t OFF_B = OFF_SVEC + 1024;
constexpr uint32_t OFF_GB = OFF_B + 256;
constexpr uint32_t OFF_GAMMA = OFF_GB + 256;
constexpr uint32_t OFF_BETA = OFF_GAMMA + 256;
constexpr uint32_t OFF_CSR = OFF_BETA + 256;            // fp32[4][64] column sums, one row per quadrant
constexpr uint32_t OFF_CSS = OFF_CSR + 1024;
constexpr uint32_t OFF_XR = OFF_CSS + 1024;             // row-sum exchange of each group
constexpr uint32_t OFF_XS = OFF_XR + kXchBytes;
constexpr uint32_t OFF_BAR = OFF_XS + 3072;
constexpr uint32_t OFF_MISC = OFF_BAR + 192;
constexpr uint32_t SMEM_USED = OFF_MISC + 64;
constexpr uint32_t SMEM_BYTES = SMEM_USED + 1024;       // slack for the 1024-byte alignment
static_assert(SMEM_BYTES <= 232448, "exceeds the 227 KB per-CTA shared memory of sm_100");

// barriers: loads first (their completion is what an aborting CTA still waits for)
constexpr int BAR_RIN = 0;                              // recompute, + stage: K, eta, Q, V, dL/dOut
constexpr int BAR_SIN = 2;                              // sweep, + stage: K, eta, V, gZ, x_f, vectors
constexpr int BAR_SQB = 4;                              // Q, gZb
constexpr int BAR_SWP = 5;
constexpr int kLoadBars = 6;
constexpr int BAR_RM = 6;                               // the recompute's products: four uses per mini-batch
constexpr int BAR_DK = 7, BAR_P1 = 8, BAR_P2 = 9;       // the sweep's
constexpr int BAR_GROUP = 10;                           // a group's slots are written
constexpr int BAR_TAIL = 11;
constexpr int BAR_DRAIN = 12;                           // abort path only
constexpr int kBars = 13;

// tensor-memory columns
constexpr uint32_t TM_W = 0;
constexpr uint32_t TM_G = 64;
constexpr uint32_t TM_R = 128;        // recompute accumulator
constexpr uint32_t TM_SA = 256;       // sweep accumulators
constexpr uint32_t TM_SB = 320;
constexpr uint32_t TM_COLS = 512;

struct LinBwdParams {
  const __nv_bfloat16* eta;
  const float* gamma;
  const float* beta;
  const float* Wc;
  const float* bc;
  const float* gW_last;
  const float* gb_last;
  uint8_t* scratch;
  float* d_gamma;
  float* d_beta;
  float* gW;
  float* gb;
  __nv_bfloat16* d_eta;
  int H, NC, cgs, nck;
  int drop_load;            // test only: mini-batch whose recompute inputs stream 0 never loads (-1: none)
  uint32_t* status;
  uint64_t wait_limit_ns;
};

__global__ void __launch_bounds__(kThreads, 1)
ttt_linear_bwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                      const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmGo,
                      const __grid_constant__ CUtensorMap tmDQ, const __grid_constant__ CUtensorMap tmDK,
                      const __grid_constant__ CUtensorMap tmDV, const LinBwdParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_align_1024(smem_raw);

  const int tid = threadIdx.x, lane = tid & 31;
  const int cta_warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int warp = cta_warp & 7;                       // within the group
  const bool recompute = cta_warp < 8;
  const int gtid = tid & (kGroup - 1);
  const bool loader = gtid == 128;                     // issues its group's bulk copies; not its MMA issuer (warp 0)
  const TokMap tm(warp, lane);
  const int quad = tm.quad;
  const long sid = blockIdx.x;
  const int head = static_cast<int>(sid % p.H);
  const int NC = p.NC, cgs = p.cgs;
  const bool row_writer = tm.colhalf == 0 && tm.l3 == 0;   // of the 8 threads that share a row, the one that stores per-row values

  auto tile = [&](uint32_t off, int s = 0) { return smem + off + s * TILE; };
  auto vec = [&](uint32_t off) { return reinterpret_cast<float*>(smem + off); };
  float* sGamma = vec(OFF_GAMMA);
  float* sBeta = vec(OFF_BETA);
  float* sB = vec(OFF_B);
  float* sGb = vec(OFF_GB);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + OFF_BAR);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + OFF_MISC);
  volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(smem + OFF_MISC + 4);
  volatile uint32_t* never_flag = reinterpret_cast<volatile uint32_t*>(smem + OFF_MISC + 8);   // stays 0
  volatile uint32_t* freed = reinterpret_cast<volatile uint32_t*>(smem + OFF_MISC + 12);       // slots the sweep has read so far
  // loads issued so far, for the abort path: bit b of word 0 = parity of barrier b's next load, of word 1 = there was one
  uint32_t* loads = reinterpret_cast<uint32_t*>(smem + OFF_MISC + 16);
  const uint64_t limit = p.wait_limit_ns;

  if (tid == 0) {
    for (int i = 0; i < kBars; ++i) mbar_init(&bars[i], i == BAR_DRAIN ? 2 : 1);
    fence_mbar_init();
    *abort_flag = 0;
    *never_flag = 0;
    *freed = 0;
    loads[0] = loads[1] = 0;
    prefetch_tmap(&tmQ);
    prefetch_tmap(&tmK);
    prefetch_tmap(&tmV);
    prefetch_tmap(&tmGo);
    prefetch_tmap(&tmDQ);
    prefetch_tmap(&tmDK);
    prefetch_tmap(&tmDV);
  }
  if (cta_warp == 0) {
    tmem_alloc(tmem_slot, TM_COLS);
    tmem_relinquish();
  }
  if (tid < 64) {
    sGamma[tid] = p.gamma[head * 64 + tid];
    sBeta[tid] = p.beta[head * 64 + tid];
    sGb[tid] = p.gb_last[sid * 64 + tid];
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  const uint32_t lead = elect_one() ? 1u : 0u;         // the lane that issues the MMAs (warp 0 of each group)

  auto wait_bar = [&](int b, uint32_t parity) { mbar_wait_bounded(&bars[b], parity & 1u, abort_flag, limit); };
  auto mma_seen = [&]() {
    __syncwarp();
    tc_fence_after_sync();
  };
  auto commit = [&](int b) { if (lead) umma_commit(&bars[b]); };
  auto expect = [&](int b, uint32_t bytes) {
    mbar_expect_tx(&bars[b], bytes);
    atomicXor(loads, 1u << b);
    atomicOr(loads + 1, 1u << b);
  };
  const long tok_rows0 = sid * NC * 64;
  auto row_of = [&](int i) { return static_cast<int>(tok_rows0 + static_cast<long>(i) * 64); };
  uint8_t* slots = p.scratch + sid * cgs * static_cast<long>(SLOT_BYTES);
  // group g (0 = the last of the sequence, the first to be processed): its first mini-batch, size, slot of mini-batch j
  auto first_of = [&](int g) { return (p.nck - 1 - g) * cgs; };
  auto size_of = [&](int g) { return g == 0 ? NC - (p.nck - 1) * cgs : cgs; };
  auto slot_of = [&](int g, int j) { return slots + static_cast<long>(g & 1 ? cgs - 1 - j : j) * SLOT_BYTES; };
  // W-shaped matrices are [64 in][64 out] in global memory; the fragment of the transposed matrix holds output features
  // r0 / r1 (rows) and the input-feature pairs col(j), col(j) + 1.
  auto load_frag = [&](const float* Wg, float (&w)[16]) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int c = tm.col(j);
      w[4 * j] = Wg[c * 64 + tm.r0];
      w[4 * j + 1] = Wg[(c + 1) * 64 + tm.r0];
      w[4 * j + 2] = Wg[c * 64 + tm.r1];
      w[4 * j + 3] = Wg[(c + 1) * 64 + tm.r1];
    }
  };
  // column sums left by the four quadrants of a group's warps
  auto quad_sum = [&](const float* cs, int f) { return (cs[f] + cs[64 + f]) + (cs[128 + f] + cs[192 + f]); };
  float dgam = 0.f, dbet = 0.f;      // this lane's column (frag_colsum_col) of what its group adds to d_gamma / d_beta
  bool stop = false;

  if (recompute) {
    // ======================================================================================= recompute
    auto publish = [&]() {
      fence_proxy_async_smem();
      tc_fence_before_sync();
      named_bar_sync(kBarR, kGroup);
    };
    uint32_t n = 0, pm = 0;
    auto wait_mma = [&]() {
      wait_bar(BAR_RM, pm);
      pm ^= 1u;
      mma_seen();
    };
    auto issue_inputs = [&](int i, uint32_t cnt) {     // loader
      if (i == p.drop_load && sid == 0) return;
      const int s = cnt & 1;
      expect(BAR_RIN + s, 4 * TILE + 128);
      tma_load_2d(tile(OFF_RK, s), &tmK, &bars[BAR_RIN + s], 0, row_of(i));
      tma_load_2d(tile(OFF_RV, s), &tmV, &bars[BAR_RIN + s], 0, row_of(i));
      tma_load_2d(tile(OFF_RQ, s), &tmQ, &bars[BAR_RIN + s], 0, row_of(i));
      tma_load_2d(tile(OFF_RGO, s), &tmGo, &bars[BAR_RIN + s], 0, row_of(i));
      bulk_load_1d(smem + OFF_RETA + s * 128, p.eta + (sid * NC + i) * 64, 128, &bars[BAR_RIN + s]);
    };
    // The slots of group g that group g - 1 used as well are free once the sweep has read them: wait (bounded) for its count.
    auto wait_slot = [&](int g, int j) {               // loader
      if (g == 0) return;
      const int before = g == 1 ? 0 : size_of(0) + (g - 2) * cgs;       // steps of the groups before g - 1
      const int own = j - (cgs - size_of(g - 1));                       // step of group g - 1 that reads this slot
      if (own < 0) return;
      const uint32_t need = static_cast<uint32_t>(before + own + 1);
      if (*freed >= need) return;
      const uint64_t t0 = globaltimer_ns();
      while (*freed < need) {
        if (*abort_flag) return;
        if (globaltimer_ns() - t0 > limit) {
          *abort_flag = 1;
          return;
        }
      }
    };
    for (int g = 0; g < p.nck && !stop; ++g) {
      const int i0 = first_of(g), gsz = size_of(g);
      if (loader) {
        if (g > 0) tma_wait_group_read<0>();
        issue_inputs(i0, n);
        if (gsz > 1) issue_inputs(i0 + 1, n + 1);
      }
      {   // checkpoint -> tensor memory (fp32) + shared memory (bf16)
        float w[16];
        load_frag(p.Wc + (sid * p.nck + p.nck - 1 - g) * 4096, w);
        tok_st_tmem(tm, tmem + TM_W, w);
        tok_st_tile(tm, tile(OFF_RW, n & 1), w);
        tmem_wait_st();
        if (gtid < 64) sB[gtid] = p.bc[(sid * p.nck + p.nck - 1 - g) * 64 + gtid];
      }
      publish();
      for (int j = 0; j < gsz; ++j, ++n) {
        const int s = n & 1;
        uint8_t* tK = tile(OFF_RK, s);
        uint8_t* tV = tile(OFF_RV, s);
        uint8_t* tGo = tile(OFF_RGO, s);
        uint8_t* tW = tile(OFF_RW, s);
        uint8_t* tWn = tile(OFF_RW, s ^ 1);
        uint8_t* tGZ = tile(OFF_RGZ);
        uint8_t* tU = tile(OFF_RU);
        uint8_t* tGZB = tU;              // U is dead after MMA2
        float* sVec = vec(OFF_RVEC) + s * 128;
        float* xch = vec(OFF_XR);
        const __nv_bfloat16* eta = reinterpret_cast<const __nv_bfloat16*>(smem + OFF_RETA) + s * 64;
        uint8_t* sl = slot_of(g, j);
        wait_bar(BAR_RIN + s, n >> 1);

        // ---- MMA1: Z = K W
        if (cta_warp == 0) {
          tc_fence_after_sync();
          mma_64_lead<false, false>(tmem + TM_R, smem_u32(tK), smem_u32(tW), lead);
          commit(BAR_RM);
        }
        if (loader && j > 0) {         // the last mini-batch's tiles have left: its stage takes the next inputs
          tma_wait_group_read<0>();
          if (j + 1 < gsz) issue_inputs(i0 + j + 1, n + 1);
        }
        wait_mma();
        // ---- LN.  x_f leaves through the V tile (every thread overwrites exactly the elements it has read); dl/dZ is
        // rounded to bf16 once, the update uses -eta times the rounded value.
        {
          TokFrag x, gr;
          uint32_t kk[8], vv[8];
          frag_ld(tm, tmem + TM_R, x);
          frag_ld_raw(tm, tK, kk);
          frag_ld_raw(tm, tV, vv);
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const f32x2 b = frag_col(tm, sB, q);
            x.a[q] = add2(x.a[q], b);
            x.b[q] = add2(x.b[q], b);
          }
          float rs0, rs1;
          frag_layernorm(tm, x, TTT_LN_EPS, xch, kBarPairR, rs0, rs1);
          f32x2 a0 = 0ull, a1 = 0ull, c0 = 0ull, c1 = 0ull;
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const f32x2 gam = frag_col(tm, sGamma, q), bet = frag_col(tm, sBeta, q), neg = pk1(-1.f);
            const f32x2 t0 = fma2(bf16x2_to_f32x2(vv[2 * q]), neg, bf16x2_to_f32x2(kk[2 * q]));          // K - V
            const f32x2 t1 = fma2(bf16x2_to_f32x2(vv[2 * q + 1]), neg, bf16x2_to_f32x2(kk[2 * q + 1]));
            gr.a[q] = mul2(fma2(gam, x.a[q], add2(t0, bet)), gam);
            gr.b[q] = mul2(fma2(gam, x.b[q], add2(t1, bet)), gam);
            a0 = add2(a0, gr.a[q]); a1 = fma2(gr.a[q], x.a[q], a1);
            c0 = add2(c0, gr.b[q]); c1 = fma2(gr.b[q], x.b[q], c1);
          }
          frag_st_tile(tm, tV, x);
          float a[2] = {hsum(a0), hsum(a1)}, b[2] = {hsum(c0), hsum(c1)};
          frag_allreduce2<1>(tm, a, b, xch, kBarPairR);
          const f32x2 sc0 = pk1(rs0 * (1.f / 64.f)), sc1 = pk1(rs1 * (1.f / 64.f));
          const f32x2 ne0 = pk1(-__bfloat162float(eta[tm.r0])), ne1 = pk1(-__bfloat162float(eta[tm.r1]));
          f32x2 su[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const uint32_t w0 = f32x2_to_bf16x2(mul2(fma2(x.a[q], pk1(-a[1]), fma2(gr.a[q], pk1(64.f), pk1(-a[0]))), sc0));
            const uint32_t w1 = f32x2_to_bf16x2(mul2(fma2(x.b[q], pk1(-b[1]), fma2(gr.b[q], pk1(64.f), pk1(-b[0]))), sc1));
            *reinterpret_cast<uint32_t*>(tGZ + tm.off(tm.r0, q)) = w0;
            *reinterpret_cast<uint32_t*>(tGZ + tm.off(tm.r1, q)) = w1;
            gr.a[q] = mul2(bf16x2_to_f32x2(w0), ne0);
            gr.b[q] = mul2(bf16x2_to_f32x2(w1), ne1);
            su[q] = add2(gr.a[q], gr.b[q]);
          }
          frag_st_tile(tm, tU, gr);
          // (column sums in registers: seven shuffles, off the tensor pipe, where four N = 8 MMAs behind the update cost
          // as much latency as a whole product)
          vec(OFF_CSR)[quad * 64 + frag_colsum_col(tm, lane)] = frag_colsum(su, lane);
          if (row_writer) {
            sVec[tm.r0] = rs0;
            sVec[tm.r1] = rs1;
          }
        }
        publish();

        // ---- MMA2: W^T += U^T K
        if (cta_warp == 0) {
          tc_fence_after_sync();
          mma_64_tn_lead(tmem + TM_W, smem_u32(tU), smem_u32(tK), lead);
          commit(BAR_RM);
        }
        if (loader) {
          wait_slot(g, j);
          bulk_store_1d(sl + SL_W, tW, TILE);
          bulk_store_1d(sl + SL_XF, tV, TILE);
          bulk_store_1d(sl + SL_GZ, tGZ, TILE);
          tma_commit_group();
        }
        __syncwarp();
        if (gtid < 64) sB[gtid] += quad_sum(vec(OFF_CSR), gtid);      // its next reader comes after the barrier below
        wait_mma();
        // ---- EPI: bf16 copy of the new W^T
        {
          TokFrag w;
          frag_ld(tm, tmem + TM_W, w);
          frag_st_tile(tm, tWn, w);
        }
        publish();

        // ---- MMA3: Zb = Q W+
        if (cta_warp == 0) {
          tc_fence_after_sync();
          mma_64_lead<false, false>(tmem + TM_R, smem_u32(tile(OFF_RQ, s)), smem_u32(tWn), lead);
          commit(BAR_RM);
        }
        wait_mma();
        // ---- LNB: output LayerNorm and its backward, gZb; its column sums; d_beta += sum go, d_gamma += sum go x_l
        {
          TokFrag x, gr;
          uint32_t go[8];
          frag_ld(tm, tmem + TM_R, x);
          frag_ld_raw(tm, tGo, go);
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const f32x2 b = frag_col(tm, sB, q);
            x.a[q] = add2(x.a[q], b);
            x.b[q] = add2(x.b[q], b);
          }
          float rs0, rs1;
          frag_layernorm(tm, x, TTT_LN_EPS, xch, kBarPairR, rs0, rs1);
          f32x2 a0 = 0ull, a1 = 0ull, c0 = 0ull, c1 = 0ull, sb[4], sg[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const f32x2 gam = frag_col(tm, sGamma, q);
            const f32x2 o0 = bf16x2_to_f32x2(go[2 * q]), o1 = bf16x2_to_f32x2(go[2 * q + 1]);
            sb[q] = add2(o0, o1);
            sg[q] = fma2(o0, x.a[q], mul2(o1, x.b[q]));
            gr.a[q] = mul2(o0, gam);
            gr.b[q] = mul2(o1, gam);
            a0 = add2(a0, gr.a[q]); a1 = fma2(gr.a[q], x.a[q], a1);
            c0 = add2(c0, gr.b[q]); c1 = fma2(gr.b[q], x.b[q], c1);
          }
          dbet += frag_colsum(sb, lane);
          dgam += frag_colsum(sg, lane);
          float a[2] = {hsum(a0), hsum(a1)}, b[2] = {hsum(c0), hsum(c1)};
          frag_allreduce2<1>(tm, a, b, xch, kBarPairR);
          const f32x2 q0 = pk1(rs0 * (1.f / 64.f)), q1 = pk1(rs1 * (1.f / 64.f));
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            gr.a[q] = mul2(fma2(x.a[q], pk1(-a[1]), fma2(gr.a[q], pk1(64.f), pk1(-a[0]))), q0);
            gr.b[q] = mul2(fma2(x.b[q], pk1(-b[1]), fma2(gr.b[q], pk1(64.f), pk1(-b[0]))), q1);
            sb[q] = add2(gr.a[q], gr.b[q]);
          }
          frag_st_tile(tm, tGZB, gr);
          vec(OFF_CSR)[quad * 64 + frag_colsum_col(tm, lane)] = frag_colsum(sb, lane);
        }
        publish();

        // ---- MMA4: gZb W+^T
        if (cta_warp == 0) {
          tc_fence_after_sync();
          mma_64_lead<true, false>(tmem + TM_R, smem_u32(tGZB), smem_u32(tWn), lead);
          commit(BAR_RM);
        }
        if (loader) {
          bulk_store_1d(sl + SL_GZB, tGZB, TILE);
          tma_commit_group();
        }
        __syncwarp();
        if (gtid < 64) sVec[64 + gtid] = quad_sum(vec(OFF_CSR), gtid);
        wait_mma();
        // ---- dQ = go + gZb W+^T, over the dL/dOut tile
        {
          TokFrag x;
          uint32_t go[8];
          frag_ld(tm, tmem + TM_R, x);
          frag_ld_raw(tm, tGo, go);
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            x.a[q] = add2(x.a[q], bf16x2_to_f32x2(go[2 * q]));
            x.b[q] = add2(x.b[q], bf16x2_to_f32x2(go[2 * q + 1]));
          }
          frag_st_tile(tm, tGo, x);
        }
        if (loader) tma_wait_group_read<0>();        // W, x_f, gZ and gZb have left their tiles
        fence_proxy_async_smem();
        tc_fence_before_sync();
        stop = named_bar_or(kBarR, kGroup, *abort_flag != 0);
        if (loader) {
          tma_store_2d(&tmDQ, tGo, 0, row_of(i0 + j));
          bulk_store_1d(sl + SL_VEC, sVec, 512);
          tma_commit_group();
        }
        if (stop) break;
      }
      if (loader && !stop) {       // the group's slots are complete
        tma_wait_group<0>();
        mbar_arrive(&bars[BAR_GROUP]);
      }
    }
    if (loader) tma_wait_group<0>();
  } else {
    // =========================================================================================== sweep
    auto publish = [&]() {
      fence_proxy_async_smem();
      tc_fence_before_sync();
      named_bar_sync(kBarS, kGroup);
    };
    uint8_t* tQ = tile(OFF_SQ);
    uint8_t* tGZB = tile(OFF_SGZB);
    uint8_t* tWP = tile(OFF_SWP);
    uint8_t* tG = tile(OFF_SG);
    uint8_t* tZin = tile(OFF_SZIN);
    uint8_t* tDK = tile(OFF_SDK);
    float* xch = vec(OFF_XS);
    {   // the gradient state starts as dL/d(final state)
      float w[16];
      load_frag(p.gW_last + sid * 4096, w);
      tok_st_tmem(tm, tmem + TM_G, w);
      tmem_wait_st();
    }
    tc_fence_before_sync();
    named_bar_sync(kBarS, kGroup);
    tc_fence_after_sync();

    // loads of one step, in parts, each issued when its tiles are free (loader)
    auto issue_in = [&](int i, const uint8_t* sl, uint32_t cnt) {
      const int s = cnt & 1;
      uint64_t* b = &bars[BAR_SIN + s];
      expect(BAR_SIN + s, 4 * TILE + 128 + 512);
      tma_load_2d(tile(OFF_SK, s), &tmK, b, 0, row_of(i));
      tma_load_2d(tile(OFF_SV, s), &tmV, b, 0, row_of(i));
      bulk_load_1d(tile(OFF_SGZ, s), sl + SL_GZ, TILE, b);
      bulk_load_1d(tile(OFF_SXF, s), sl + SL_XF, TILE, b);
      bulk_load_1d(smem + OFF_SETA + s * 128, p.eta + (sid * NC + i) * 64, 128, b);
      bulk_load_1d(vec(OFF_SVEC) + s * 128, sl + SL_VEC, 512, b);
    };
    auto issue_qb = [&](int i, const uint8_t* sl) {
      expect(BAR_SQB, 2 * TILE);
      tma_load_2d(tQ, &tmQ, &bars[BAR_SQB], 0, row_of(i));
      bulk_load_1d(tGZB, sl + SL_GZB, TILE, &bars[BAR_SQB]);
    };
    auto issue_wp = [&](const uint8_t* sl) {
      expect(BAR_SWP, TILE);
      bulk_load_1d(tWP, sl + SL_W, TILE, &bars[BAR_SWP]);
    };
    f32x2 kpa[4], kpb[4];        // partial dK of the step before: gamma Bt - eta T1
    // what the step of count c adds to the gradient state, and its dK product (MMA issuer)
    auto issue_tail = [&](uint32_t c) {
      wait_bar(BAR_SWP, c);
      mma_seen();
      mma_64_lead<true, false>(tmem + TM_SA, smem_u32(tZin), smem_u32(tWP), lead);
      commit(BAR_DK);
      mma_64_tn_lead(tmem + TM_G, smem_u32(tZin), smem_u32(tile(OFF_SK, c & 1)), lead);
    };
    auto finish_dk = [&](uint32_t c) {
      wait_bar(BAR_DK, c);
      mma_seen();
      TokFrag x;
      frag_ld(tm, tmem + TM_SA, x);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        x.a[q] = add2(x.a[q], kpa[q]);
        x.b[q] = add2(x.b[q], kpb[q]);
      }
      frag_st_tile(tm, tDK, x);
    };

    uint32_t m = 0;
    for (int g = 0; g < p.nck && !stop; ++g) {
      const int i0 = first_of(g), gsz = size_of(g);
      if (loader) {
        wait_bar(BAR_GROUP, g);
        const int j = gsz - 1;
        const uint8_t* sl = slot_of(g, j);
        issue_qb(i0 + j, sl);
        tma_wait_group_read<0>();
        issue_in(i0 + j, sl, m);
      }
      __syncwarp();
      for (int j = gsz - 1; j >= 0; --j, ++m) {
        const uint32_t par = m & 1;
        const bool first = j == gsz - 1;
        uint8_t* tK = tile(OFF_SK, par);
        uint8_t* tV = tile(OFF_SV, par);
        uint8_t* tXF = tile(OFF_SXF, par);
        uint8_t* tGZ = tile(OFF_SGZ, par);
        const float* sVec = vec(OFF_SVEC) + par * 128;
        const __nv_bfloat16* eta = reinterpret_cast<const __nv_bfloat16*>(smem + OFF_SETA) + par * 64;

        // ---- P1: the step before's dK product and state gradient; G^T += gZb^T Q
        if (cta_warp == 8) {
          tc_fence_after_sync();
          if (!first) issue_tail(m - 1);
          wait_bar(BAR_SQB, par);
          mma_seen();
          mma_64_tn_lead(tmem + TM_G, smem_u32(tGZB), smem_u32(tQ), lead);
          commit(BAR_P1);
        }
        if (!first) finish_dk(m - 1);
        wait_bar(BAR_P1, par);
        mma_seen();
        if (loader) {
          if (!first) *freed = m;            // the step before's slot has been read (its last tile, W, just now)
          issue_wp(slot_of(g, j));
          if (j > 0) {
            issue_qb(i0 + j - 1, slot_of(g, j - 1));
            tma_wait_group_read<0>();        // dV of the step before has left the tile V comes into
            issue_in(i0 + j - 1, slot_of(g, j - 1), m + 1);
          }
        }
        // ---- E2: bf16 copy of G^T
        {
          TokFrag w;
          frag_ld(tm, tmem + TM_G, w);
          frag_st_tile(tm, tG, w);
        }
        wait_bar(BAR_SIN + par, m >> 1);
        if (gtid < 64) sGb[gtid] += sVec[64 + gtid];
        publish();

        // ---- P2: K G, T1 = gZ G^T
        if (cta_warp == 8) {
          tc_fence_after_sync();
          mma_64_lead<false, false>(tmem + TM_SA, smem_u32(tK), smem_u32(tG), lead);
          mma_64_lead<true, false>(tmem + TM_SB, smem_u32(tGZ), smem_u32(tG), lead);
          commit(BAR_P2);
        }
        if (loader && !first) {
          tma_store_2d(&tmDK, tDK, 0, row_of(i0 + j + 1));
          tma_commit_group();
        }
        __syncwarp();
        // ---- E4: second order through the fused LayerNorm + L2 gradient
        {
          TokFrag A, t1, go;
          uint32_t gzw[8], xhw[8], kw[8];
          frag_ld_raw(tm, tGZ, gzw);
          frag_ld_raw(tm, tXF, xhw);
          frag_ld_raw(tm, tK, kw);
          {
            uint32_t vw[8];
            frag_ld_raw(tm, tV, vw);
#pragma unroll
            for (int q = 0; q < 4; ++q) {    // grad_output_fused = gamma x_hat_fused + beta - (V - K)
              const f32x2 gam = frag_col(tm, sGamma, q), bet = frag_col(tm, sBeta, q), neg = pk1(-1.f);
              go.a[q] = add2(fma2(bf16x2_to_f32x2(vw[2 * q]), neg, bf16x2_to_f32x2(kw[2 * q])),
                             fma2(gam, bf16x2_to_f32x2(xhw[2 * q]), bet));
              go.b[q] = add2(fma2(bf16x2_to_f32x2(vw[2 * q + 1]), neg, bf16x2_to_f32x2(kw[2 * q + 1])),
                             fma2(gam, bf16x2_to_f32x2(xhw[2 * q + 1]), bet));
            }
          }
          const float eta0 = __bfloat162float(eta[tm.r0]), eta1 = __bfloat162float(eta[tm.r1]);
          const float rs0 = sVec[tm.r0], rs1 = sVec[tm.r1];      // 1 / std
          wait_bar(BAR_P2, par);
          mma_seen();
          frag_ld(tm, tmem + TM_SA, A);
          frag_ld(tm, tmem + TM_SB, t1);
          float ra[4], rb[4];       // d_eta, sum A, sum A xh, sum g xh
          {
            f32x2 s0[4] = {0ull, 0ull, 0ull, 0ull}, s1[4] = {0ull, 0ull, 0ull, 0ull};
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const f32x2 gb = frag_col(tm, sGb, q), gam = frag_col(tm, sGamma, q);
              const f32x2 x0 = bf16x2_to_f32x2(xhw[2 * q]), x1 = bf16x2_to_f32x2(xhw[2 * q + 1]);
              s0[0] = fma2(t1.a[q], bf16x2_to_f32x2(kw[2 * q]), fma2(gb, bf16x2_to_f32x2(gzw[2 * q]), s0[0]));
              s1[0] = fma2(t1.b[q], bf16x2_to_f32x2(kw[2 * q + 1]), fma2(gb, bf16x2_to_f32x2(gzw[2 * q + 1]), s1[0]));
              kpa[q] = mul2(t1.a[q], pk1(-eta0));
              kpb[q] = mul2(t1.b[q], pk1(-eta1));
              A.a[q] = mul2(add2(A.a[q], gb), pk1(-eta0));
              A.b[q] = mul2(add2(A.b[q], gb), pk1(-eta1));
              s0[1] = add2(s0[1], A.a[q]);
              s1[1] = add2(s1[1], A.b[q]);
              s0[2] = fma2(A.a[q], x0, s0[2]);
              s1[2] = fma2(A.b[q], x1, s1[2]);
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
          float4* x4 = reinterpret_cast<float4*>(xch);
          if (tm.l3 == 0) {
            x4[tm.colhalf * 64 + tm.r0] = make_float4(ra[0], ra[1], ra[2], ra[3]);
            x4[tm.colhalf * 64 + tm.r1] = make_float4(rb[0], rb[1], rb[2], rb[3]);
          }
          named_bar_sync(kBarPairS + tm.quad, 64);
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
              const f32x2 bt0 = mul2(add2(A.a[q], fma2(x0, xA, mA)), pk1(rs0));
              const f32x2 bt1 = mul2(add2(A.b[q], fma2(x1, xB, mB)), pk1(rs1));
              const f32x2 gl0 = mul2(gm, bt0), gl1 = mul2(gm, bt1);
              cs[q] = add2(fma2(go.a[q], bt0, mul2(gl0, x0)), fma2(go.b[q], bt1, mul2(gl1, x1)));
              cl[q] = add2(gl0, gl1);
              dv.a[q] = mul2(gl0, neg);
              dv.b[q] = mul2(gl1, neg);
              kpa[q] = add2(kpa[q], gl0);
              kpb[q] = add2(kpb[q], gl1);
              const f32x2 gx0 = fma2(gl0, gm, fma2(mul2(go.a[q], gm), fA3, mul2(A.a[q], fA4)));
              const f32x2 gx1 = fma2(gl1, gm, fma2(mul2(go.b[q], gm), fB3, mul2(A.b[q], fB4)));
              sa0 = fma2(gx0, x0, fma2(A.a[q], bf16x2_to_f32x2(gzw[2 * q]), sa0));
              sb0 = fma2(gx1, x1, fma2(A.b[q], bf16x2_to_f32x2(gzw[2 * q + 1]), sb0));
              sa1 = add2(sa1, gx0);
              sb1 = add2(sb1, gx1);
              A.a[q] = gx0;
              A.b[q] = gx1;
            }
            frag_st_tile(tm, tV, dv);       // over V (every thread overwrites the elements it has read)
            dgam += frag_colsum(cs, lane);
            dbet += frag_colsum(cl, lane);
          }
          float sa[2] = {-hsum(sa0) * rs0, hsum(sa1)}, sb[2] = {-hsum(sb0) * rs1, hsum(sb1)};
          frag_allreduce2<1>(tm, sa, sb, xch + 256, kBarPairS);       // (behind the 2 KB of the exchange above)
          {
            const f32x2 k0 = pk1(sa[0] * (1.f / 64.f)), l0 = pk1(-sa[1] * rs0 * (1.f / 64.f));
            const f32x2 k1 = pk1(sb[0] * (1.f / 64.f)), l1 = pk1(-sb[1] * rs1 * (1.f / 64.f));
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              A.a[q] = fma2(A.a[q], pk1(rs0), fma2(bf16x2_to_f32x2(xhw[2 * q]), k0, l0));      // gZin
              A.b[q] = fma2(A.b[q], pk1(rs1), fma2(bf16x2_to_f32x2(xhw[2 * q + 1]), k1, l1));
              cs[q] = add2(A.a[q], A.b[q]);
            }
            frag_st_tile(tm, tZin, A);
            vec(OFF_CSS)[quad * 64 + frag_colsum_col(tm, lane)] = frag_colsum(cs, lane);
          }
          if (row_writer) {
            p.d_eta[(sid * NC + i0 + j) * 64 + tm.r0] = __float2bfloat16(-ra[0]);
            p.d_eta[(sid * NC + i0 + j) * 64 + tm.r1] = __float2bfloat16(-rb[0]);
          }
        }
        if (loader) tma_wait_group_read<0>();      // dK of the step before has left its tile
        fence_proxy_async_smem();
        tc_fence_before_sync();
        stop = named_bar_or(kBarS, kGroup, *abort_flag != 0);
        if (loader) {
          tma_store_2d(&tmDV, tV, 0, row_of(i0 + j));
          tma_commit_group();
        }
        if (gtid < 64) sGb[gtid] += quad_sum(vec(OFF_CSS), gtid);
        if (stop) break;
      }
      if (stop) break;
      // ---- what the group's last step adds, and its dK
      if (cta_warp == 8) {
        tc_fence_after_sync();
        issue_tail(m - 1);
        commit(BAR_TAIL);
      }
      finish_dk(m - 1);
      wait_bar(BAR_TAIL, g);
      mma_seen();
      if (loader) *freed = m;
      publish();
      if (loader) {
        tma_store_2d(&tmDK, tDK, 0, row_of(i0));
        tma_commit_group();
      }
      __syncwarp();
    }
    // ---- dL/d(initial state)
    if (!stop) {
      float w[16];
      tok_ld(tm, tmem + TM_G, w);
      float* Wo = p.gW + sid * 4096;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int c = tm.col(j);
        Wo[c * 64 + tm.r0] = w[4 * j];
        Wo[(c + 1) * 64 + tm.r0] = w[4 * j + 1];
        Wo[c * 64 + tm.r1] = w[4 * j + 2];
        Wo[(c + 1) * 64 + tm.r1] = w[4 * j + 3];
      }
    }
    if (loader) tma_wait_group<0>();
  }

  // ---- norm gradients of this stream; teardown
  tc_fence_before_sync();
  const bool aborted = __syncthreads_or(stop || *abort_flag != 0) != 0;
  tc_fence_after_sync();
  if (!aborted) {
    float* sum = vec(OFF_RK);      // [2 groups][d_gamma, d_beta][4 quadrants][64]
    const int at = (recompute ? 0 : 512) + quad * 64 + frag_colsum_col(tm, lane);
    sum[at] = dgam;
    sum[at + 256] = dbet;
    __syncthreads();
    if (tid < 64) {
      p.gb[sid * 64 + tid] = sGb[tid];
      p.d_gamma[sid * 64 + tid] = quad_sum(sum, tid) + quad_sum(sum + 512, tid);
      p.d_beta[sid * 64 + tid] = quad_sum(sum + 256, tid) + quad_sum(sum + 768, tid);
    }
  } else {
    // everything this CTA still has in flight is waited for (bounded, not cut short by the abort flag)
    // before its shared and tensor memory go away: the tensor-core work of both issuers, and the loads
    if (warp == 0 && lead) umma_commit(&bars[BAR_DRAIN]);
    if (tid == 0) {
      mbar_wait_bounded(&bars[BAR_DRAIN], 0, never_flag, limit);
      for (int b = 0; b < kLoadBars; ++b)
        if (loads[1] >> b & 1u) mbar_wait_bounded(&bars[b], (loads[0] >> b & 1u) ^ 1u, never_flag, limit);
      atomicExch(p.status, static_cast<uint32_t>(TTT_B200_ERR_TIMEOUT));
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (cta_warp == 0) tmem_dealloc(tmem, TM_COLS);
}

}  // namespace

uint64_t ttt_linear_backward_scratch_bytes(int B, int H, int cgs) {
  return static_cast<uint64_t>(B) * H * cgs * SLOT_BYTES;
}

int ttt_launch_linear_backward(const ttt_b200_linear_bwd_args* a, cudaStream_t stream, uint32_t* status,
                               uint64_t limit_ns, int drop_load) {
  const uint64_t rows = static_cast<uint64_t>(a->B) * a->H * a->NC * 64;
  CUtensorMap tmQ, tmK, tmV, tmGo, tmDQ, tmDK, tmDV;
  if (int rc = ttt_make_tile_map(&tmQ, a->XQ, rows)) return rc;
  if (int rc = ttt_make_tile_map(&tmK, a->XK, rows)) return rc;
  if (int rc = ttt_make_tile_map(&tmV, a->XV, rows)) return rc;
  if (int rc = ttt_make_tile_map(&tmGo, a->grad_L_XQW_mini_batch, rows)) return rc;
  if (int rc = ttt_make_tile_map(&tmDQ, a->grad_L_XQ, rows)) return rc;
  if (int rc = ttt_make_tile_map(&tmDK, a->grad_L_XK, rows)) return rc;
  if (int rc = ttt_make_tile_map(&tmDV, a->grad_L_XV, rows)) return rc;
  LinBwdParams p;
  p.eta = static_cast<const __nv_bfloat16*>(a->last_eta);
  p.gamma = a->ttt_norm_weight;
  p.beta = a->ttt_norm_bias;
  p.Wc = a->W1_checkpoints; p.bc = a->b1_checkpoints;
  p.gW_last = a->grad_L_W1_last; p.gb_last = a->grad_L_b1_last;
  p.scratch = static_cast<uint8_t*>(a->scratch);
  p.d_gamma = a->grad_L_ttt_norm_weight; p.d_beta = a->grad_L_ttt_norm_bias;
  p.gW = a->grad_L_W1_init; p.gb = a->grad_L_b1_init;
  p.d_eta = static_cast<__nv_bfloat16*>(a->grad_L_last_eta);
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
    attr_err[dev] = cudaFuncSetAttribute(ttt_linear_bwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
  });
  if (attr_err[dev] != cudaSuccess) return ttt_set_error(TTT_B200_ERR_LAUNCH, cudaGetErrorString(attr_err[dev]));
  ttt_linear_bwd_kernel<<<dim3(a->B * a->H), dim3(kThreads), SMEM_BYTES, stream>>>(tmQ, tmK, tmV, tmGo, tmDQ, tmDK, tmDV, p);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return ttt_set_error(TTT_B200_ERR_LAUNCH, cudaGetErrorString(e));
  return TTT_B200_OK;
}
