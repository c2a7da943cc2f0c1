// TTT-MLP backward for sm_100a, cluster-sharded: one thread-block cluster of kC = 2 or 4 CTAs per
// (batch, head) stream, each CTA owning 256 / kC of the hidden units.
//
// Replaces the reference's bwd_ttt_mlp_ker with its hidden dimension split over a cluster of four
// CTAs and its tp_reduce (kernels/ttt_backward/ttt.cu:21-69, 179-1443; reductions at :574, :766,
// :1160); the math is that of kernels/ttt_backward/matching.py:57-342.  Structure, phase order,
// buffer rotation and scratch layout are those of the one-CTA kernel (ttt_bwd_sm100.cu), whose
// header lists the reverse step G1..G15 / E1..E6; what changes is the ownership:
//
//   local to the CTA that owns a hidden unit: its rows of W1^T / W2 and of the gradient state
//   dL/dW1^T / dL/dW2 (tensor memory), b1 and dL/db1 (registers), and every [256][64 tok] quantity
//   (Z1, X2, dl/dZ1, gelu', P, S, ... : NB = 4 / kC blocks of 64 rows).  In the scratch slots a CTA
//   writes and reads back only its own rows of the [256][64] images, so scratch written by this
//   kernel has the layout of the one-CTA kernel's.
//
//   summed over the cluster (ttt_cluster.cuh), as fp32 64 x 64 tiles: Z2 and Z2_bar in the
//   recompute; in the reverse step the hidden-unit contractions G7 (dQ), G5 / G6 / G8 (merged into
//   one tile: A2 = -eta acc1 + acc2, plus the two d_eta row sums that are linear in acc1 and T1) and
//   G13 (dK, together with the -eta T1 term).  Three sums per reverse step, two per recomputed
//   mini-batch.  dQ and dK are outputs only: they are summed by reduce-scatter (every CTA finishes and
//   stores the token rows it owns), which sends kC times fewer bytes than an all-reduce.
//
//   the 64 x 64 token stages (LayerNorm stages, second-order terms), in one of two forms:
//
//   kC = 2, replicated: every CTA computes them from the same summed tiles, bit for bit, together with b2,
//   dL/db2, d_gamma, d_beta.  The token-tile scratch (x_hat_fused, dl/dZ2, x_hat_ln, 1/std) is written by
//   every CTA with the same bytes, so that a CTA only ever reads back what it has written itself.  The CTAs
//   take turns storing dV; rank 0 stores d_eta and the per-stream vectors.
//
//   kC = 4, split by rows (RowSplit in ttt_cluster.cuh): every sum is a reduce-scatter to the CTA that owns
//   the 16 token rows, which runs the stage on them (warp = row pair, lane = column pair) and hands the bf16
//   rows that feed MMAs (dl/dZ2, U2, x_hat_ln, gZ2in) to every peer's operand tile.  x_hat_fused and the
//   1/std vectors are needed by the row's owner only: a CTA writes and reads back its own rows of those
//   scratch tiles.  dQ, dK, dV, d_eta are stored by the owner of the row.  b2 and dL/db2 stay replicated
//   (column sums of gathered tiles); the d_gamma / d_beta addends of the second-order stage are summed per
//   CTA over its own rows and added up by rank 0, in rank order, at the end.
//
// Bound by the chain: at four CTAs per stream the work of a phase is a few hundred cycles beside the latencies of MMA,
// exchange, row sums and barriers.  Hence the epilogues work on packed fp32 pairs, take column sums from registers, and
// leave the row sums that only the bias gradients need to the next MMA window.  Measured per mini-batch, 32 streams in
// groups of 4: 15.5 -> 14.9 us (all rows' sums at once), -> 14.0 us (the rest).  Two CTAs per stream run here where there
// are no groups to pipeline (else ttt_bwd_pair_sm100.cu), 48 streams x 32: 17.6 us in one group (one CTA: 20.7), 25.3 in
// groups of one (31.4).  Issue slots are used to 28-29 %, the tensor pipe to 9 % (four CTAs) and 14 % (two).
//
// Every wait is bounded; a wait that runs out raises the abort flag of the whole cluster, the vote on
// leaving a loop is taken CTA-wide at a barrier, and no CTA exits before its peers have reached the
// exit barrier.
#include <mutex>

#include "ttt_cluster.cuh"
#include "ttt_internal.h"

using namespace tttcl;

namespace {

constexpr int kThreads = 256;
// The thread that issues the bulk copies and waits for their completion is not one of the four MMA issuers
// (lane 0 of warps 0..3): its bookkeeping between a barrier and the next MMA group stays off the issue path.
constexpr int kProd = 128;

// barrier indices
constexpr int BAR_BIG = 0;     // +buffer index (0..4)
constexpr int BAR_T = 5;       // +tile index (0..6)
constexpr int BAR_IN = 12;     // +stage (0..1), recompute inputs
constexpr int BAR_MMA = 14;
constexpr int BAR_V = 15;      // recompute: the single V tile
constexpr int BAR_SUM = 16;    // +buffer (0..3; the all-reduce form uses two), cluster sums
constexpr int BAR_DRAIN = 20;  // abort path only
constexpr int BAR_AG = 21;     // row-split form: rows of a stage's result arriving from the peers
constexpr int BAR_AG2 = 22;    // the same for the deferred x_hat_ln
constexpr int NUM_BARS = 23;

template <int kC>
struct Cfg {
  static constexpr int NB = 4 / kC;
  static constexpr int R = 64 * NB;
  static constexpr uint32_t HB = NB * TILE;            // bytes of an [R][64] bf16 tile
  using Sum = ClusterSum<kC, 18432>;                   // a 64 x 64 tile, optionally with two extra values per thread
  // Four CTAs: the token stages are split by rows as well (every CTA runs them on the 16 token rows it owns
  // and hands the bf16 results to its peers).  At two CTAs the row-split form works too (set this to true) but
  // was measured slower than the all-reduce form: 22.9 against 21.2 us per mini-batch at 32 streams.
  static constexpr bool kRowSplit = kC == 4;
  using RS = RowSplit<kC, true>;
  static constexpr uint32_t OFF_BIG = 0;               // 5 hidden-major buffers
  static constexpr uint32_t OFF_T = 5 * HB;            // 8 token tiles of 8 KB
  static constexpr uint32_t OFF_SUM = OFF_T + 8 * TILE;
  static constexpr uint32_t OFF_B2 = OFF_SUM + (kRowSplit ? RS::kBytes : Sum::kBytes);
  static constexpr uint32_t OFF_GB2 = OFF_B2 + 256;
  static constexpr uint32_t OFF_GAMMA = OFF_GB2 + 256;
  static constexpr uint32_t OFF_BETA = OFF_GAMMA + 256;
  static constexpr uint32_t OFF_DG = OFF_BETA + 256;
  static constexpr uint32_t OFF_DB = OFF_DG + 256;
  static constexpr uint32_t OFF_SIGLN = OFF_DB + 256;
  static constexpr uint32_t OFF_SIGF = OFF_SIGLN + 256;
  static constexpr uint32_t OFF_GB1 = OFF_SIGF + 256;       // fp32[R] copy of the per-thread dL/db1
  static constexpr uint32_t OFF_PART = OFF_GB1 + 1024;      // fp32[4][64] partial sums for d_eta (one row per quadrant)
  // fp32[3][4][64] column-sum partials (the row-split form keeps the second-order stage's own-row partials,
  // 2 x [8][64], in the row-sum exchange area, which is not in use between that stage and their sum)
  static constexpr uint32_t OFF_CSUM = OFF_PART + 1024;
  static constexpr uint32_t OFF_ETA = OFF_CSUM + 3072;      // bf16[2][64]
  static constexpr uint32_t OFF_BAR = OFF_ETA + 256;
  static constexpr uint32_t OFF_MISC = OFF_BAR + 192;
  static constexpr uint32_t OFF_XCH = OFF_MISC + 64;        // fp32[2][64][8] row-sum exchange between warp pairs
  // row-split form only: 1/std of x_hat_ln gathered from the row owners; d_gamma / d_beta addends of this
  // CTA's own rows ([2][64])
  static constexpr uint32_t OFF_SIGAG = OFF_XCH + 4096;
  static constexpr uint32_t OFF_DGP = OFF_SIGAG + 256;
  static constexpr uint32_t OFF_ONES = (OFF_DGP + 512 + 1023) & ~1023u;   // bf16[8][64] ones: B operand of the column sums
  static constexpr uint32_t SMEM_USED = OFF_ONES + (NB == 1 ? 1024 : 0);
  static constexpr uint32_t SMEM_BYTES = SMEM_USED + 1024;
  static_assert(SMEM_BYTES <= 232448, "exceeds the 227 KB per-CTA shared memory of sm_100");
  static_assert(NUM_BARS * 8 <= 192, "barrier area");
  // tensor memory: state blocks, accumulator A (NB hidden blocks or one token tile), accumulator B (NB
  // hidden blocks or two token tiles)
  static constexpr uint32_t TM_S1 = 0;
  static constexpr uint32_t TM_S2 = 64 * NB;
  static constexpr uint32_t TM_A = 128 * NB;
  static constexpr uint32_t TM_B = 128 * NB + (NB > 1 ? 64 * NB : 64);
  // four CTAs per stream only (tensor memory is full at two): 8 columns each for column sums taken by the tensor pipe
  static constexpr bool kMmaColsum = NB == 1;
  static constexpr uint32_t TM_CS = TM_B + 128;
  static constexpr uint32_t TM_COLS = 512;
  static_assert(TM_B + 128 + (kMmaColsum ? 16 : 0) <= 512, "tensor memory");
};

struct BwdClParams {
  const __nv_bfloat16* eta;
  const float* gamma;
  const float* beta;
  const float* W1c; const float* b1c; const float* W2c; const float* b2c;
  uint8_t* sc_W1; uint8_t* sc_W2;                       // 64 KB per slot, first 32 KB used
  uint8_t* sc_Z1; uint8_t* sc_X2; uint8_t* sc_gZ1; uint8_t* sc_Z1b; uint8_t* sc_X2b;   // 32 KB per slot
  uint8_t* sc_xhf; uint8_t* sc_gZ2; uint8_t* sc_xhln;                                  // 8 KB per slot
  float* sc_sigf; float* sc_sigln;                      // 64 floats per slot
  const float* gW1_last; const float* gb1_last; const float* gW2_last; const float* gb2_last;
  float* d_gamma; float* d_beta;
  float* gW1; float* gb1; float* gW2; float* gb2;
  __nv_bfloat16* d_eta;
  __nv_bfloat16* dXQ; __nv_bfloat16* dXK; __nv_bfloat16* dXV;   // bf16 [rows][64], row-major
  int H, NC, cgs, nck;
  int drop_load;            // test only: mini-batch whose recompute inputs stream 0 never loads (-1: none)
  uint32_t* status;
  uint64_t wait_limit_ns;
};

template <int kC>
__global__ void __launch_bounds__(kThreads, 1)
ttt_bwd_cluster_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                       const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmGo,
                       const __grid_constant__ CUtensorMap tmDQ, const __grid_constant__ CUtensorMap tmDK,
                       const __grid_constant__ CUtensorMap tmDV, const BwdClParams p) {
  using C = Cfg<kC>;
  constexpr int NB = C::NB;
  constexpr uint32_t HB = C::HB;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_align_1024(smem_raw);

  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const TokMap tm(warp, lane);
  const uint32_t rank = cluster_ctarank();
  const long sid = blockIdx.x / kC;
  const int head = static_cast<int>(sid % p.H);
  const int NC = p.NC, cgs = p.cgs;
  const int hid0 = static_cast<int>(rank) * C::R;
  const uint32_t img0 = rank * HB;            // this CTA's rows inside a [256][64] scratch image
  const bool kp_owner = C::Sum::row_owner(tid) == rank;     // this thread's token rows are this CTA's to finish
  const bool row_writer = tm.colhalf == 0 && tm.l3 == 0;   // of the 8 threads that share a row, the one that stores per-row values

  auto big = [&](int i) -> uint8_t* { return smem + C::OFF_BIG + i * HB; };
  auto tile = [&](int i) -> uint8_t* { return smem + C::OFF_T + i * TILE; };
  float* sB2 = reinterpret_cast<float*>(smem + C::OFF_B2);
  float* sGb2 = reinterpret_cast<float*>(smem + C::OFF_GB2);
  float* sGamma = reinterpret_cast<float*>(smem + C::OFF_GAMMA);
  float* sBeta = reinterpret_cast<float*>(smem + C::OFF_BETA);
  float* sDG = reinterpret_cast<float*>(smem + C::OFF_DG);
  float* sDB = reinterpret_cast<float*>(smem + C::OFF_DB);
  float* sSigLn = reinterpret_cast<float*>(smem + C::OFF_SIGLN);
  float* sSigF = reinterpret_cast<float*>(smem + C::OFF_SIGF);
  float* sGb1 = reinterpret_cast<float*>(smem + C::OFF_GB1);
  float* sPart = reinterpret_cast<float*>(smem + C::OFF_PART);
  float* part = reinterpret_cast<float*>(smem + C::OFF_CSUM);
  __nv_bfloat16* sEta = reinterpret_cast<__nv_bfloat16*>(smem + C::OFF_ETA);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::OFF_BAR);
  float* sXch = reinterpret_cast<float*>(smem + C::OFF_XCH);
  float* sSigAG = reinterpret_cast<float*>(smem + C::OFF_SIGAG);
  float* sDGp = reinterpret_cast<float*>(smem + C::OFF_DGP);       // [0..63] d_gamma, [64..127] d_beta addends of the own rows
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + C::OFF_MISC);
  volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(smem + C::OFF_MISC + 4);
  volatile uint32_t* never_flag = reinterpret_cast<volatile uint32_t*>(smem + C::OFF_MISC + 8);   // stays 0
  const uint64_t limit = p.wait_limit_ns;

  if (tid == kProd) {
    for (int i = 0; i < NUM_BARS; ++i) {
      uint32_t cnt = 1;
      if (i == BAR_MMA || i == BAR_DRAIN) cnt = 4;
      if (i >= BAR_SUM && i < BAR_SUM + 4) cnt = C::kRowSplit ? C::RS::kBarCount : C::Sum::kArrivals;
      mbar_init(&bars[i], cnt);
    }
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
    tmem_alloc(tmem_slot, C::TM_COLS);
    tmem_relinquish();
  }
  if (tid < 64) {
    sGamma[tid] = p.gamma[head * 64 + tid];
    sBeta[tid] = p.beta[head * 64 + tid];
    sGb2[tid] = p.gb2_last[sid * 64 + tid];
    sDG[tid] = 0.f;
    sDB[tid] = 0.f;
    sDGp[tid] = 0.f;
    sDGp[64 + tid] = 0.f;
  }
  if constexpr (C::kMmaColsum) reinterpret_cast<uint32_t*>(smem + C::OFF_ONES)[tid] = 0x3F803F80u;     // 256 x two bf16 ones
  float Gb1[NB][2];
#pragma unroll
  for (int b = 0; b < NB; ++b) {
    Gb1[b][0] = p.gb1_last[sid * 256 + hid0 + 64 * b + tm.r0];
    Gb1[b][1] = p.gb1_last[sid * 256 + hid0 + 64 * b + tm.r1];
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  cluster_arrive();     // the peers' mbarriers and abort flags are initialised before anything is sent to them
  cluster_wait();
  const uint32_t tmem = *tmem_slot;
  const uint32_t lead = elect_one() ? 1u : 0u;      // the lane of an issuing warp whose MMAs are enabled

  typename C::Sum csum;
  csum.bufp = smem + C::OFF_SUM;
  csum.bars = &bars[BAR_SUM];
  csum.n = 0;
  csum.rank = rank;
  csum.abort_flag = abort_flag;
  csum.limit = limit;
  auto cluster_sum = [&](float (&v)[16]) { csum.run(v, tid, lane); };
  typename C::RS rs;
  rs.bufp = smem + C::OFF_SUM;
  rs.bars = &bars[BAR_SUM];
  rs.n = 0;
  rs.rank = rank;
  rs.abort_flag = abort_flag;
  rs.limit = limit;
  constexpr int NR = C::RS::NR;
  using RSx = typename C::RS;

  // ---- barrier bookkeeping: every thread waits on every barrier use, in program order, or counts it (skip_bar)
  uint32_t ph = 0;        // expected parity per barrier
  uint32_t pending = 0;   // thread 0: loads issued and not yet waited for
  auto wait_bar = [&](int b) {
    if (mbar_wait_cl(&bars[b], (ph >> b) & 1u, abort_flag, limit, kC)) {
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
    fence_proxy_async_smem();
    tc_fence_before_sync();
    __syncthreads();
  };
  // the same barrier, also taking the CTA-wide vote on the abort flag (a peer can raise it at any moment)
  auto publish_vote = [&]() -> bool {
    fence_proxy_async_smem();
    tc_fence_before_sync();
    return __syncthreads_or(*abort_flag != 0) != 0;
  };
  auto load_big = [&](int buf, const uint8_t* slot_image) {     // thread 0: this CTA's rows of a scratch image
    mbar_expect_tx(&bars[BAR_BIG + buf], HB);
    bulk_load_1d(big(buf), slot_image + img0, HB, &bars[BAR_BIG + buf]);
    pending |= 1u << (BAR_BIG + buf);
  };
  auto store_big = [&](uint8_t* slot_image, const uint8_t* src) {   // thread 0
    bulk_store_1d(slot_image + img0, src, HB);
  };
#define TTT_ISSUE4(W0, W1_, W2_, W3)  \
  if (warp < 4) {                     \
    tc_fence_after_sync();            \
    if (warp == 0) { W0; }            \
    else if (warp == 1) { W1_; }      \
    else if (warp == 2) { W2_; }      \
    else { W3; }                      \
    if (lead) umma_commit(&bars[BAR_MMA]);        \
  }
  // hidden-major block products over this CTA's NB blocks: D[b] (+)= A[b] * Bt
#define HID_ALL(KBMN, D, A, BT, ACC)                                                          \
  do {                                                                                        \
    _Pragma("unroll") for (int b_ = 0; b_ < NB; ++b_)                                         \
      mma_hid64<KBMN>(tmem + (D) + b_ * 64, smem_u32(A) + b_ * TILE, smem_u32(BT), (ACC), lead);    \
  } while (0)
#define HID_ONE(KBMN, D, A, BT, ACC, B_)                                                      \
  mma_hid64<KBMN>(tmem + (D) + (B_) * 64, smem_u32(A) + (B_) * TILE, smem_u32(BT), (ACC), lead)

  const long tok_rows0 = sid * NC * 64;

  auto part_sum = [&](int k) {
    return (part[k * 256 + tid] + part[k * 256 + 64 + tid]) + (part[k * 256 + 128 + tid] + part[k * 256 + 192 + tid]);
  };
  // -eta of the thread's token column pair q
  auto neg_eta_col = [&](const __nv_bfloat16* e, int q) {
    return bf16x2_to_f32x2(*reinterpret_cast<const uint32_t*>(e + tm.col(q)) ^ 0x80008000u);
  };

  // ---- state <-> global memory (this CTA's rows): W1-shaped matrices are [64 feat][256 hid], W2-shaped
  // ones [256 hid][64 feat]; in the fragment of block b a thread holds hidden units hid0 + 64 b + r0 / r1
  // and, for j = 0..3, the feature pair col(j), col(j) + 1.
  auto w1_index = [&](int b, int r, int c) { return c * 256 + hid0 + 64 * b + r; };
  auto w2_index = [&](int b, int r, int c) { return (hid0 + 64 * b + r) * 64 + c; };
  auto load_w1_frag = [&](const float* W1g, int b, float (&w)[16]) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int c = tm.col(j);
      w[4 * j] = W1g[w1_index(b, tm.r0, c)];
      w[4 * j + 1] = W1g[w1_index(b, tm.r0, c + 1)];
      w[4 * j + 2] = W1g[w1_index(b, tm.r1, c)];
      w[4 * j + 3] = W1g[w1_index(b, tm.r1, c + 1)];
    }
  };
  auto load_w2_frag = [&](const float* W2g, int b, float (&w)[16]) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int c = tm.col(j);
      const float2 a = *reinterpret_cast<const float2*>(W2g + w2_index(b, tm.r0, c));
      const float2 d = *reinterpret_cast<const float2*>(W2g + w2_index(b, tm.r1, c));
      w[4 * j] = a.x; w[4 * j + 1] = a.y; w[4 * j + 2] = d.x; w[4 * j + 3] = d.y;
    }
  };
  auto store_w1_frag = [&](float* W1o, int b, const float (&w)[16]) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int c = tm.col(j);
      W1o[w1_index(b, tm.r0, c)] = w[4 * j];
      W1o[w1_index(b, tm.r0, c + 1)] = w[4 * j + 1];
      W1o[w1_index(b, tm.r1, c)] = w[4 * j + 2];
      W1o[w1_index(b, tm.r1, c + 1)] = w[4 * j + 3];
    }
  };
  auto store_w2_frag = [&](float* W2o, int b, const float (&w)[16]) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int c = tm.col(j);
      *reinterpret_cast<float2*>(W2o + w2_index(b, tm.r0, c)) = make_float2(w[4 * j], w[4 * j + 1]);
      *reinterpret_cast<float2*>(W2o + w2_index(b, tm.r1, c)) = make_float2(w[4 * j + 2], w[4 * j + 3]);
    }
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
    // 3 = Z1^T -> U1^T -> gelu'(Z1_bar^T), 4 = G' -> dl/dZ1^T.  Token tiles: 0..3 = K, Q of two stages,
    // 4 = V, 5 = gZ2, 6 = U2.
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
    float b1v[NB][2];
#pragma unroll
    for (int b = 0; b < NB; ++b) {
      b1v[b][0] = p.b1c[(sid * p.nck + ck) * 256 + hid0 + 64 * b + tm.r0];
      b1v[b][1] = p.b1c[(sid * p.nck + ck) * 256 + hid0 + 64 * b + tm.r1];
    }
    if (tid < 64) sB2[tid] = p.b2c[(sid * p.nck + ck) * 64 + tid];
    {
      const float* W1g = p.W1c + (sid * p.nck + ck) * (64 * 256);
      const float* W2g = p.W2c + (sid * p.nck + ck) * (256 * 64);
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        float w1[16], w2[16];
        load_w1_frag(W1g, b, w1);
        load_w2_frag(W2g, b, w2);
        tok_st_tmem(tm, tmem + C::TM_S1 + b * 64, w1);
        tok_st_tmem(tm, tmem + C::TM_S2 + b * 64, w2);
        tok_st_tile(tm, bW1 + b * TILE, w1);
        tok_st_tile(tm, bW2 + b * TILE, w2);
      }
      tmem_wait_st();
    }
    publish();
    if (tid == kProd) {   // bf16 images of the checkpoint = pre-update weights of the group's first mini-batch
      store_big(p.sc_W1 + slot0 * 65536, bW1);
      store_big(p.sc_W2 + slot0 * 65536, bW2);
      tma_commit_group();
    }

    // ================================================================== recompute the group
    float zb[16];             // a mini-batch's partial Z2b between the send and the receive of its sum
    uint32_t zb_tag = 0;
    long zb_slot = -1;
    uint8_t* tXln = tile(7);  // x_hat_ln on its way to the scratch slot
    auto finish_xhln = [&]() {
      csum.allreduce_recv(zb, tid, zb_tag);
      TokFrag x;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const f32x2 b = frag_col(tm, sB2, q);
        x.a[q] = add2(pk(zb[4 * q], zb[4 * q + 1]), b);
        x.b[q] = add2(pk(zb[4 * q + 2], zb[4 * q + 3]), b);
      }
      float rs0, rs1;
      frag_layernorm(tm, x, TTT_LN_EPS, sXch, 1, rs0, rs1);
      frag_st_tile(tm, tXln, x);
      if (row_writer) {
        p.sc_sigln[zb_slot * 64 + tm.r0] = rs0;
        p.sc_sigln[zb_slot * 64 + tm.r1] = rs1;
      }
    };
    // Row-split form: the sums of the rows this CTA owns are normalised here; the bf16 rows and their 1/std go
    // to every CTA of the cluster (each keeps a whole tile for its scratch slot).
    auto finish_xhln_rows = [&]() {
      if (tid == 0) rs.arm_all_gather(&bars[BAR_AG2], 1, C::RS::ROWS * 4u);
      const float2 b2c = *reinterpret_cast<const float2*>(sB2 + 2 * lane);
      float z[NR][2];
      rs.recv(z, warp, lane, zb_tag);
      float rstd[NR];
      RSx::row_layernorm(z, b2c, TTT_LN_EPS, rstd);
#pragma unroll
      for (int i = 0; i < NR; ++i) {
        const int r = rs.row(i, warp);
        rs.all_gather_store(tXln, &bars[BAR_AG2], r, lane, z[i][0], z[i][1]);
        if (lane == 0) sSigAG[r] = rstd[i];
        else if (lane < kC)
          st_async_f1(mapa(smem_u32(sSigAG + r), rank ^ static_cast<uint32_t>(lane)),
                      mapa(smem_u32(&bars[BAR_AG2]), rank ^ static_cast<uint32_t>(lane)), rstd[i]);
      }
    };
    // after the barrier that follows the wait on BAR_AG2: the gathered tile and its 1/std leave for the slot
    auto store_xhln_rows = [&](long xslot) {
      if (tid < 64) p.sc_sigln[xslot * 64 + tid] = sSigAG[tid];
      if (tid == kProd) bulk_store_1d(p.sc_xhln + xslot * TILE, tXln, TILE);
    };
    for (int j = 0; j < gsz; ++j) {
      const int s = j & 1;
      const long slot = slot0 + j;
      const uint8_t* sK = tile(2 * s + 0);
      const uint8_t* sQ = tile(2 * s + 1);
      const uint8_t* sV = tV;
      const __nv_bfloat16* eta = sEta + s * 64;
      wait_bar(BAR_IN + s);

      // MMA1: Z1^T = W1^T K^T
      TTT_ISSUE4(HID_ONE(false, C::TM_A, bW1, sK, 0u, 0),
                 if (NB > 1) HID_ONE(false, C::TM_A, bW1, sK, 0u, NB - 1),
                 ,
                 )
      long xhln_slot = -1;                     // the previous mini-batch's x_hat_ln, with the b2 it saw
      if constexpr (!C::kRowSplit) {
        xhln_slot = zb_slot;
        if (zb_slot >= 0) {
          finish_xhln();
          zb_slot = -1;
        }
      }
      wait_mma();
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        TokFrag z, g, gp;
        frag_ld(tm, tmem + C::TM_A + b * 64, z);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          z.a[q] = add2(z.a[q], pk1(b1v[b][0]));
          z.b[q] = add2(z.b[q], pk1(b1v[b][1]));
          gelu_pair2(z.a[q], g.a[q], gp.a[q]);
          gelu_pair2(z.b[q], g.b[q], gp.b[q]);
        }
        frag_st_tile(tm, bX2 + b * TILE, g);
        frag_st_tile(tm, bGP + b * TILE, gp);
        frag_st_tile_h(tm, bZ1 + b * TILE, z);      // f16: the sweep evaluates gelu' and gelu'' of it in f16
      }
      publish();
      if (tid == kProd) {
        if (xhln_slot >= 0) bulk_store_1d(p.sc_xhln + xhln_slot * TILE, tXln, TILE);
        store_big(p.sc_X2 + slot * BIG, bX2);
        store_big(p.sc_Z1 + slot * BIG, bZ1);
        tma_commit_group();
      }

      // MMA2: partial Z2 = X2 W2
      TTT_ISSUE4(mma_tok_partial(tmem + C::TM_B, smem_u32(bX2), smem_u32(bW2), NB, lead),
                 ,
                 ,
                 )
      wait_mma();
      wait_bar(BAR_V);
      long xrow_slot = -1;      // row-split form: the x_hat_ln gathered during this phase
      if constexpr (C::kRowSplit) {
        // the partial Z2 tiles are summed by reduce-scatter; the fused LayerNorm + L2 gradient runs on the token
        // rows this CTA owns (warp = row pair, lane = column pair) and its rows of dl/dZ2 and U2 go to every CTA
        float frag[16];
        tok_ld(tm, tmem + C::TM_B, frag);
        const uint32_t tag = rs.send(frag, tid, warp, lane);
        if (tid == 0) rs.arm_all_gather(&bars[BAR_AG], 2);
        const float2 b2c = *reinterpret_cast<const float2*>(sB2 + 2 * lane);
        const float2 gam = *reinterpret_cast<const float2*>(sGamma + 2 * lane);
        const float2 bet = *reinterpret_cast<const float2*>(sBeta + 2 * lane);
        float2 kk[NR], vv[NR];
        float neta[NR];
#pragma unroll
        for (int i = 0; i < NR; ++i) {
          const int r = rs.row(i, warp);
          kk[i] = RSx::ld_pair(sK, r, lane);
          vv[i] = RSx::ld_pair(sV, r, lane);
          neta[i] = -__bfloat162float(eta[r]);
        }
        // while this sum is under way: the previous mini-batch's x_hat_ln, whose sum arrived long ago (b2 has
        // not changed since: its update follows in the next MMA window)
        if (zb_slot >= 0) {
          xrow_slot = zb_slot;
          finish_xhln_rows();
          zb_slot = -1;
        }
        float z[NR][2];
        rs.recv(z, warp, lane, tag);
        float rstd[NR], g[NR][2], a[2 * NR];
        RSx::row_layernorm(z, b2c, TTT_LN_EPS, rstd);
#pragma unroll
        for (int i = 0; i < NR; ++i) {
          g[i][0] = (fmaf(gam.x, z[i][0], bet.x) - (vv[i].x - kk[i].x)) * gam.x;
          g[i][1] = (fmaf(gam.y, z[i][1], bet.y) - (vv[i].y - kk[i].y)) * gam.y;
          a[2 * i] = g[i][0] + g[i][1];
          a[2 * i + 1] = fmaf(g[i][0], z[i][0], g[i][1] * z[i][1]);
        }
        RSx::row_sums(a);
#pragma unroll
        for (int i = 0; i < NR; ++i) {
          const int r = rs.row(i, warp);
          const float x0 = z[i][0], x1 = z[i][1], g0 = g[i][0], g1 = g[i][1], a0 = a[2 * i], a1 = a[2 * i + 1];
          const float sc = rstd[i] * (1.f / 64.f);
          // x_hat_fused leaves through this CTA's rows of the V tile; dl/dZ2 is rounded to bf16 once (the update
          // uses -eta times the rounded value)
          RSx::st_pair(tV, r, lane, x0, x1);
          const float d0 = __bfloat162float(__float2bfloat16((64.f * g0 - a0 - x0 * a1) * sc));
          const float d1 = __bfloat162float(__float2bfloat16((64.f * g1 - a0 - x1 * a1) * sc));
          rs.all_gather_store(tGZ2, &bars[BAR_AG], r, lane, d0, d1);
          rs.all_gather_store(tU2, &bars[BAR_AG], r, lane, neta[i] * d0, neta[i] * d1);
          if (lane == 0) p.sc_sigf[slot * 64 + r] = rstd[i];
        }
        wait_bar(BAR_AG);
        if (xrow_slot >= 0) wait_bar(BAR_AG2);
      } else {
        float zs[16];
        uint32_t kk[8], vv[8];
        tok_ld(tm, tmem + C::TM_B, zs);
        frag_ld_raw(tm, sK, kk);
        frag_ld_raw(tm, sV, vv);
        cluster_sum(zs);
        TokFrag x, g;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const f32x2 b = frag_col(tm, sB2, q);
          x.a[q] = add2(pk(zs[4 * q], zs[4 * q + 1]), b);
          x.b[q] = add2(pk(zs[4 * q + 2], zs[4 * q + 3]), b);
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
        // read) as a bulk store; grad_output_fused is rebuilt in the sweep from x_hat_fused, K, V
        frag_st_tile(tm, tV, x);
        float a[2] = {hsum(a0), hsum(a1)}, bb[2] = {hsum(c0), hsum(c1)};
        frag_allreduce2<1>(tm, a, bb, sXch, 1);
        const f32x2 sc0 = pk1(rs0 * (1.f / 64.f)), sc1 = pk1(rs1 * (1.f / 64.f));
        const f32x2 ne0 = pk1(-__bfloat162float(eta[tm.r0])), ne1 = pk1(-__bfloat162float(eta[tm.r1]));
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          // dl/dZ2, rounded to bf16 once: the update below uses -eta times the rounded value
          kk[2 * q] = f32x2_to_bf16x2(mul2(fma2(x.a[q], pk1(-a[1]), fma2(g.a[q], pk1(64.f), pk1(-a[0]))), sc0));
          kk[2 * q + 1] = f32x2_to_bf16x2(mul2(fma2(x.b[q], pk1(-bb[1]), fma2(g.b[q], pk1(64.f), pk1(-bb[0]))), sc1));
          g.a[q] = mul2(bf16x2_to_f32x2(kk[2 * q]), ne0);
          g.b[q] = mul2(bf16x2_to_f32x2(kk[2 * q + 1]), ne1);
          x.a[q] = add2(g.a[q], g.b[q]);
        }
        frag_st_raw(tm, tGZ2, kk);
        frag_st_tile(tm, tU2, g);
        part[tm.quad * 64 + frag_colsum_col(tm, lane)] = frag_colsum(x.a, lane);
        if (row_writer) {
          p.sc_sigf[slot * 64 + tm.r0] = rs0;     // the slot keeps 1/std: the sweep only ever divides by std
          p.sc_sigf[slot * 64 + tm.r1] = rs1;
        }
      }
      if (tid == kProd) tma_wait_group_read<0>();   // Z1 / X2 images have left shared memory
      publish();

      // MMA3: R^T = W2 gZ2^T
      if constexpr (C::kRowSplit) {
        if (xrow_slot >= 0) store_xhln_rows(xrow_slot);
      }
      if (tid == kProd) {
        if constexpr (C::kRowSplit) {   // only the rows this CTA owns hold x_hat_fused (the others still hold V)
          constexpr uint32_t RB = C::RS::ROWS * 128u;
          bulk_store_1d(p.sc_xhf + slot * TILE + rank * RB, tV + rank * RB, RB);
        } else {
          bulk_store_1d(p.sc_xhf + slot * TILE, tV, TILE);
        }
        bulk_store_1d(p.sc_gZ2 + slot * TILE, tGZ2, TILE);
        tma_commit_group();
      }
      if constexpr (C::kMmaColsum) {
        // b2 += column sums of U2, taken by the tensor pipe in the same phase (the window of these small MMAs is
        // too short to hide a pass over the tile by the warps)
        TTT_ISSUE4(HID_ONE(false, C::TM_A, bW2, tGZ2, 0u, 0),
                   mma_colsum(tmem + C::TM_CS, smem_u32(tU2), smem_u32(smem + C::OFF_ONES), lead),
                   ,
                   )
        wait_mma();
        if (warp < 4) {
          const float cs = colsum_read(tmem + C::TM_CS, warp);
          if (lane < 16) sB2[16 * warp + lane] += cs;
        }
      } else {
        TTT_ISSUE4(HID_ONE(false, C::TM_A, bW2, tGZ2, 0u, 0),
                   if (NB > 1) HID_ONE(false, C::TM_A, bW2, tGZ2, 0u, NB - 1),
                   ,
                   )
        if (tid < 64) sB2[tid] += part_sum(0);
        wait_mma();
      }
      float ra[NB], rb[NB];      // row sums of U1 (for b1): this thread's part, reduced in the next MMA window
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        TokFrag r;
        uint32_t gw[8];
        frag_ld(tm, tmem + C::TM_A + b * 64, r);
        frag_ld_raw(tm, bGP + b * TILE, gw);
        f32x2 s0 = 0ull, s1 = 0ull;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const f32x2 ne = neg_eta_col(eta, q);
          // dl/dZ1 rounded to bf16 (the value the scratch slot and the sweep see), in place over G'; U1 = -eta dl/dZ1
          gw[2 * q] = f32x2_to_bf16x2(mul2(bf16x2_to_f32x2(gw[2 * q]), r.a[q]));
          gw[2 * q + 1] = f32x2_to_bf16x2(mul2(bf16x2_to_f32x2(gw[2 * q + 1]), r.b[q]));
          r.a[q] = mul2(bf16x2_to_f32x2(gw[2 * q]), ne);
          r.b[q] = mul2(bf16x2_to_f32x2(gw[2 * q + 1]), ne);
          s0 = add2(s0, r.a[q]);
          s1 = add2(s1, r.b[q]);
        }
        frag_st_raw(tm, bGP + b * TILE, gw);
        frag_st_tile(tm, bZ1 + b * TILE, r);     // U1, over Z1
        ra[b] = hsum(s0);
        rb[b] = hsum(s1);
      }
      publish();

      // MMA4: W1^T += U1^T K ; W2 += X2^T U2
      if (tid == kProd) {
        tma_wait_group_read<0>();               // x_hat_fused has left the V tile
        if (j + 1 < gsz) issue_v(j + 1);
        store_big(p.sc_gZ1 + slot * BIG, bGP);
        tma_commit_group();
      }
      TTT_ISSUE4(HID_ONE(true, C::TM_S1, bZ1, sK, 1u, 0),
                 HID_ONE(true, C::TM_S2, bX2, tU2, 1u, 0),
                 if (NB > 1) HID_ONE(true, C::TM_S1, bZ1, sK, 1u, NB - 1),
                 if (NB > 1) HID_ONE(true, C::TM_S2, bX2, tU2, 1u, NB - 1))
      tok_row_allreduce<NB, 4>(tm, ra, rb, sXch);
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        b1v[b][0] += ra[b];
        b1v[b][1] += rb[b];
      }
      wait_mma();
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        float w[16];
        tok_ld(tm, tmem + C::TM_S1 + b * 64, w);
        tok_st_tile(tm, bW1 + b * TILE, w);
        tok_ld(tm, tmem + C::TM_S2 + b * 64, w);
        tok_st_tile(tm, bW2 + b * TILE, w);
      }
      publish();

      // MMA5: Z1b^T = W1+^T Q^T
      if (tid == kProd) {
        if (j + 1 < gsz) {   // the new weights are the next mini-batch's pre-update weights
          store_big(p.sc_W1 + (slot + 1) * 65536, bW1);
          store_big(p.sc_W2 + (slot + 1) * 65536, bW2);
          tma_commit_group();
        }
      }
      TTT_ISSUE4(HID_ONE(false, C::TM_A, bW1, sQ, 0u, 0),
                 if (NB > 1) HID_ONE(false, C::TM_A, bW1, sQ, 0u, NB - 1),
                 ,
                 )
      wait_mma();
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        TokFrag z, g;
        frag_ld(tm, tmem + C::TM_A + b * 64, z);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          // the sweep needs gelu'(Z1_bar) only: it is cheaper here, next to gelu, than there from a bf16 copy
          gelu_pair2(add2(z.a[q], pk1(b1v[b][0])), g.a[q], z.a[q]);
          gelu_pair2(add2(z.b[q], pk1(b1v[b][1])), g.b[q], z.b[q]);
        }
        frag_st_tile(tm, bX2 + b * TILE, g);
        frag_st_tile(tm, bZ1 + b * TILE, z);
      }
      publish();

      // MMA6: partial Z2b = X2b W2+ ; output LayerNorm statistics
      if (tid == kProd) {
        store_big(p.sc_X2b + slot * BIG, bX2);
        store_big(p.sc_Z1b + slot * BIG, bZ1);
        tma_commit_group();
      }
      TTT_ISSUE4(mma_tok_partial(tmem + C::TM_B, smem_u32(bX2), smem_u32(bW2), NB, lead),
                 ,
                 ,
                 )
      wait_mma();
      // Z2b only feeds the output LayerNorm statistics the sweep will read back from scratch: nothing in the
      // recompute waits for it.  Its partial tile is sent now; the sum is received and normalised inside the
      // first MMA window of the next mini-batch (or right after the group's last one).
      tok_ld(tm, tmem + C::TM_B, zb);
      if constexpr (C::kRowSplit) zb_tag = rs.send(zb, tid, warp, lane);
      else zb_tag = csum.allreduce_send(zb, tid);
      zb_slot = slot;
      if (tid == kProd) tma_wait_group_read<0>();   // every big image of this mini-batch has left shared memory
      aborted = publish_vote();
      if (tid == kProd && j + 2 < gsz && !aborted) issue_inputs(j + 2);
      if (aborted) break;
    }
    if (aborted) break;
    if constexpr (C::kRowSplit) {   // the group's last x_hat_ln
      finish_xhln_rows();
      wait_bar(BAR_AG2);
      publish();
      store_xhln_rows(zb_slot);
      if (tid == kProd) tma_commit_group();
    } else {
      finish_xhln();
      publish();
      if (tid == kProd) {
        bulk_store_1d(p.sc_xhln + zb_slot * TILE, tXln, TILE);
        tma_commit_group();
      }
    }

    // ================================================================== reverse sweep
    // buffer roles: ib0 = W1+ (bf16), ib1 = W2+, the other three free
    int ib0 = 0, ib1 = 1, ib2 = 2, ib3 = 3, ib4 = 4;
    uint8_t* t_go = tile(0);
    uint8_t* t_a = tile(1);     // x_hat_ln -> V -> d_gamma addends
    uint8_t* t_q = tile(2);     // Q -> gZ2in
    uint8_t* t_g = tile(3);     // gZ2b -> U2 = -eta gZ2
    uint8_t* t_k = tile(4);
    uint8_t* t_gz2 = tile(5);
    uint8_t* t_xf = tile(6);    // x_hat_fused
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
    auto issue_rest = [&](int j) {             // Q, K + eta tiles; X2_bar and dl/dZ1
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
    // dL/dW state: global (fp32) -> tensor memory
#pragma unroll
    for (int b = 0; b < NB; ++b) {
      float w1[16], w2[16];
      load_w1_frag(Gsrc_W1, b, w1);
      load_w2_frag(Gsrc_W2, b, w2);
      tok_st_tmem(tm, tmem + C::TM_S1 + b * 64, w1);
      tok_st_tmem(tm, tmem + C::TM_S2 + b * 64, w2);
    }
    tmem_wait_st();
    tc_fence_before_sync();   // the state columns are read by the MMAs of the first step

    float dk_pend[16];          // a step's share of dK between its send and its receive
    uint32_t dk_tag = 0;
    int dk_row0 = -1;
    float dk_gly[NR][2];        // row-split form: the LayerNorm term of dK for the rows this CTA owns
    auto finish_dk_rows = [&]() {
      float z[NR][2];
      rs.recv(z, warp, lane, dk_tag);
#pragma unroll
      for (int i = 0; i < NR; ++i)
        RSx::st_pair_global(p.dXK + static_cast<long>(dk_row0) * 64, rs.row(i, warp), lane, z[i][0] + dk_gly[i][0],
                            z[i][1] + dk_gly[i][1]);
    };
    for (int j = gsz - 1; j >= 0; --j) {
      const long slot = slot0 + j;
      const int row0 = static_cast<int>(tok_rows0 + (long)(i0 + j) * 64);
      const uint32_t turn = static_cast<uint32_t>(i0 + j);     // whose turn it is to store dQ / dV / dK
      float kp[16];                                            // this CTA's share of dK, completed in E6

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
          const f32x2 go0 = bf16x2_to_f32x2(gw[2 * q]), go1 = bf16x2_to_f32x2(gw[2 * q + 1]);
          const f32x2 x0 = bf16x2_to_f32x2(xw[2 * q]), x1 = bf16x2_to_f32x2(xw[2 * q + 1]);
          g.a[q] = mul2(go0, gam);
          g.b[q] = mul2(go1, gam);
          a0 = add2(a0, g.a[q]); a1 = fma2(g.a[q], x0, a1);
          c0 = add2(c0, g.b[q]); c1 = fma2(g.b[q], x1, c1);
          sb[q] = add2(go0, go1);
          sg[q] = fma2(go0, x0, mul2(go1, x1));
        }
        // column sums over the tokens (d_beta, d_gamma, G_b2) from the registers: a pass over the tiles beside G1 was
        // longer than G1
        const int fc = tm.quad * 64 + frag_colsum_col(tm, lane);
        part[fc] = frag_colsum(sb, lane);
        part[256 + fc] = frag_colsum(sg, lane);
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
        part[512 + fc] = frag_colsum(sb, lane);
      }
      publish();
      // G1: gX2b^T = W2+ gZ2b^T
      TTT_ISSUE4(HID_ONE(false, C::TM_A, big(ib1), t_g, 0u, 0),
                 if (NB > 1) HID_ONE(false, C::TM_A, big(ib1), t_g, 0u, NB - 1),
                 ,
                 )
      if (tid < 64) {
        sDB[tid] += part_sum(0);
        sDG[tid] += part_sum(1);
        sGb2[tid] += part_sum(2);
      }
      if (dk_row0 >= 0) {     // the previous step's dK
        if constexpr (C::kRowSplit) {
          finish_dk_rows();
        } else {
          if (csum.reduce_scatter_recv(dk_pend, tid, dk_tag)) tok_st_global(tm, p.dXK + static_cast<long>(dk_row0) * 64, dk_pend);
        }
        dk_row0 = -1;
      }
      wait_mma();
      if (tid == kProd) load_big(ib1, p.sc_X2 + slot * BIG);   // W2+ is consumed (G1 was its only use): X2 for G5
      wait_bar(BAR_BIG + ib2);
      // ---- E1: gZ1b^T = gX2b^T * gelu'(Z1b^T), in place over the gelu'(Z1_bar) tile
      float ga[NB], gb[NB];      // row sums (for G_b1): this thread's part, reduced in the next MMA window
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        TokFrag v;
        uint32_t zw[8];
        frag_ld(tm, tmem + C::TM_A + b * 64, v);
        frag_ld_raw(tm, big(ib2) + b * TILE, zw);
        f32x2 s0 = 0ull, s1 = 0ull;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          v.a[q] = mul2(bf16x2_to_f32x2(zw[2 * q]), v.a[q]);
          v.b[q] = mul2(bf16x2_to_f32x2(zw[2 * q + 1]), v.b[q]);
          s0 = add2(s0, v.a[q]);
          s1 = add2(s1, v.b[q]);
        }
        frag_st_tile(tm, big(ib2) + b * TILE, v);
        ga[b] = hsum(s0);
        gb[b] = hsum(s1);
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
      // G7 (partial dQ) // G2 // G3
      TTT_ISSUE4(mma_tok_partial(tmem + C::TM_B, smem_u32(big(ib2)), smem_u32(big(ib0)), NB, lead),
                 HID_ALL(true, C::TM_S2, big(ib3), t_g, 1u),
                 HID_ONE(true, C::TM_S1, big(ib2), t_q, 1u, 0),
                 if (NB > 1) HID_ONE(true, C::TM_S1, big(ib2), t_q, 1u, NB - 1))
      tok_row_allreduce<NB, 4>(tm, ga, gb, sXch);
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        Gb1[b][0] += ga[b];
        Gb1[b][1] += gb[b];
      }
      wait_mma();
      // gZ1b is consumed: Z1 of this step comes in while E2 runs (X2_bar's buffer takes the W2 snapshot)
      if (tid == kProd) load_big(ib2, p.sc_Z1 + slot * BIG);
      // ---- E2: bf16 snapshots of the gradient state; dQ
      {
        uint8_t* s1b = big(ib0);
        uint8_t* s2b = big(ib3);
#pragma unroll
        for (int b = 0; b < NB; ++b) {
          float w[16];
          tok_ld(tm, tmem + C::TM_S1 + b * 64, w);
          tok_st_tile(tm, s1b + b * TILE, w);
          tok_ld(tm, tmem + C::TM_S2 + b * 64, w);
          tok_st_tile(tm, s2b + b * TILE, w);
          if (row_writer) {
            sGb1[64 * b + tm.r0] = Gb1[b][0];
            sGb1[64 * b + tm.r1] = Gb1[b][1];
          }
        }
      }
      // dQ = go + sum over the cluster of gZ1b W1+^T: an output only, so the partial tiles are summed by
      // reduce-scatter and every CTA stores the token rows it owns.  The partial tile is sent now and
      // received inside the next MMA window: nobody waits for the exchange.
      float dq[16];
      tok_ld(tm, tmem + C::TM_B, dq);
      uint32_t dq_tag;
      if constexpr (C::kRowSplit) dq_tag = rs.send(dq, tid, warp, lane);
      else dq_tag = csum.reduce_scatter_send(dq, tid);
      publish();
      wait_bar(BAR_BIG + ib4);
      wait_bar(BAR_T + 4);
      // X2, requested two phases ago.  Only those who issue MMAs or the next load wait: nothing would hold that load, of W2
      // into the same buffer, back until a warp without a part in them had seen this one.
      if (warp <= kProd / 32) wait_bar(BAR_BIG + ib1);
      else skip_bar(BAR_BIG + ib1);
      // G8 (partial T1) // G5 (partial acc1) // G4
      TTT_ISSUE4(mma_tok_partial(tmem + C::TM_B, smem_u32(big(ib4)), smem_u32(big(ib0)), NB, lead),
                 mma_tok_partial(tmem + C::TM_B + 64, smem_u32(big(ib1)), smem_u32(big(ib3)), NB, lead),
                 HID_ONE(false, C::TM_A, big(ib0), t_k, 0u, 0),
                 if (NB > 1) HID_ONE(false, C::TM_A, big(ib0), t_k, 0u, NB - 1))
      // ---- while the MMAs run: partial sums over this CTA's hidden units of gZ1 * G_b1 (fourth term of d_eta).  A warp takes
      // the elements of gZ1 that its own fragment of P overwrites in E3: nothing holds another warp's E3 back until here.
      {
        // lane l takes the token pair l % 16 of the warp's 32 tokens and, of the quadrant's 16 rows of a block, 0..3 and
        // 8..11 or, l >= 16, the others: the two half warps read opposite halves of the swizzled lines, without conflicts
        const int sub = (lane >> 4) * 4, pair = lane & 15;
        const uint8_t* bg = big(ib4) + (pair & 3) * 4;
        const uint32_t chunk = tm.colhalf * 4 + (pair >> 2);
        float a0 = 0.f, a1 = 0.f, c0 = 0.f, c1 = 0.f;
#pragma unroll
        for (int hh = 0; hh < 8 * NB; hh += 4) {
          const int h = (hh >> 3) * 64 + tm.quad * 16 + (hh & 4) * 2 + sub;
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
        a0 += c0;
        a1 += c1;
        a0 += __shfl_xor_sync(0xffffffffu, a0, 16);
        a1 += __shfl_xor_sync(0xffffffffu, a1, 16);
        if (lane < 16) *reinterpret_cast<float2*>(sPart + tm.quad * 64 + tm.colhalf * 32 + 2 * pair) = make_float2(a0, a1);
      }
      if constexpr (C::kRowSplit) {
        // finished inside E4's wait for its own sum
      } else if (csum.reduce_scatter_recv(dq, tid, dq_tag)) {
        float go[16];
        tok_ld_tile(tm, t_go, go);
#pragma unroll
        for (int q = 0; q < 16; ++q) go[q] += dq[q];
        tok_st_global(tm, p.dXQ + static_cast<long>(row0) * 64, go);
      }
      wait_mma();
      if (tid == kProd) {
        load_big(ib1, p.sc_W2 + slot * 65536);      // X2 is consumed until G14: W2 takes its buffer
        tma_wait_group_read<0>();     // dQ has left the dL/dOut tile (E4 reuses it for dV)
      }
      wait_bar(BAR_BIG + ib2);
      // ---- E3: A1, P = A1 gelu'(Z1), S = A1 gelu''(Z1), gelu'(Z1) (kept as f16)
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        TokFrag v, sv;
        uint32_t zw[8], gp[8];
        frag_ld(tm, tmem + C::TM_A + b * 64, v);
        frag_ld_raw(tm, big(ib2) + b * TILE, zw);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const f32x2 ne = neg_eta_col(sEta, q);
          uint32_t gpp;
          v.a[q] = mul2(ne, add2(v.a[q], pk1(Gb1[b][0])));
          gelu_grad_h2(zw[2 * q], gp[2 * q], gpp);
          sv.a[q] = mul2(v.a[q], f16x2_to_f32x2(gpp));
          v.a[q] = mul2(v.a[q], f16x2_to_f32x2(gp[2 * q]));
          v.b[q] = mul2(ne, add2(v.b[q], pk1(Gb1[b][1])));
          gelu_grad_h2(zw[2 * q + 1], gp[2 * q + 1], gpp);
          sv.b[q] = mul2(v.b[q], f16x2_to_f32x2(gpp));
          v.b[q] = mul2(v.b[q], f16x2_to_f32x2(gp[2 * q + 1]));
        }
        frag_st_tile(tm, big(ib4) + b * TILE, v);
        frag_st_tile(tm, big(ib2) + b * TILE, sv);
        frag_st_raw(tm, big(ib0) + b * TILE, gp);
      }
      publish();
      wait_bar(BAR_BIG + ib1);
      wait_bar(BAR_T + 5);
      // G6 (partial acc2) // G10
      TTT_ISSUE4(mma_tok_partial(tmem + C::TM_A, smem_u32(big(ib4)), smem_u32(big(ib1)), NB, lead),
                 HID_ONE(true, C::TM_S2, big(ib4), t_gz2, 1u, 0),
                 if (NB > 1) HID_ONE(true, C::TM_S2, big(ib4), t_gz2, 1u, NB - 1),
                 )
      wait_mma();
      if (tid == kProd) load_big(ib4, p.sc_W1 + slot * 65536);
      wait_bar(BAR_T + 6);
      wait_bar(BAR_T + 1);   // V
      // ---- E4: second order through the fused LayerNorm + L2 gradient (token-major, all 8 warps)
      if constexpr (C::kRowSplit) {
        // Row-split form.  Fragment side: this CTA's shares X2 G_W2 (acc1), P W2 (acc2), gZ1 G_W1 (t1); what the
        // step needs from them is linear: A2 = -eta acc1 + acc2 and the d_eta row sums of gz acc1 + t1 K travel
        // to the owner of the rows, -eta t1 stays for dK.  U2 = -eta gZ2 needs no sum: every CTA writes all of it.
        uint32_t a2_tag;
        {
          float A2[16], gz[16], kk[16], acc1[16], acc2[16], t1[16];
          const float eta0 = __bfloat162float(sEta[tm.r0]), eta1 = __bfloat162float(sEta[tm.r1]);
          tok_ld_tile(tm, t_gz2, gz);
          tok_ld_tile(tm, t_k, kk);
          tok_ld3(tm, tmem + C::TM_B + 64, acc1, tmem + C::TM_A, acc2, tmem + C::TM_B, t1);
          float de0 = 0.f, de1 = 0.f;
#pragma unroll
          for (int q = 0; q < 4; ++q) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const int x0 = 4 * q + h, x1 = 4 * q + 2 + h;
              A2[x0] = fmaf(-eta0, acc1[x0], acc2[x0]);
              A2[x1] = fmaf(-eta1, acc1[x1], acc2[x1]);
              de0 = fmaf(gz[x0], acc1[x0], fmaf(t1[x0], kk[x0], de0));
              de1 = fmaf(gz[x1], acc1[x1], fmaf(t1[x1], kk[x1], de1));
              kp[x0] = -eta0 * t1[x0];
              kp[x1] = -eta1 * t1[x1];
              gz[x0] *= -eta0;
              gz[x1] *= -eta1;
            }
          }
          if (row_writer) {     // the partial sums over this CTA's hidden units of gZ1 * G_b1, once per row
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              de0 += sPart[q * 64 + tm.r0];
              de1 += sPart[q * 64 + tm.r1];
            }
          }
          a2_tag = rs.send_x(A2, de0, de1, tid, warp, lane);
          if (tid == 0) rs.arm_all_gather(&bars[BAR_AG], 1);
          tok_st_tile(tm, t_g, gz);
        }
        // Row side: the rows this CTA owns (warp = row pair, lane = column pair)
        const float2 gam = *reinterpret_cast<const float2*>(sGamma + 2 * lane);
        const float2 bet = *reinterpret_cast<const float2*>(sBeta + 2 * lane);
        const float2 gb2 = *reinterpret_cast<const float2*>(sGb2 + 2 * lane);
        float2 gzr[NR], xh[NR], vv[NR], kr[NR];
        float etar[NR], rsd[NR];
#pragma unroll
        for (int i = 0; i < NR; ++i) {
          const int r = rs.row(i, warp);
          gzr[i] = RSx::ld_pair(t_gz2, r, lane);
          xh[i] = RSx::ld_pair(t_xf, r, lane);
          vv[i] = RSx::ld_pair(t_a, r, lane);
          kr[i] = RSx::ld_pair(t_k, r, lane);
          etar[i] = __bfloat162float(sEta[r]);
          rsd[i] = sSigF[r];       // 1 / std
        }
        {   // while the A2 sum is under way: dQ = dL/dOut + the sum sent in E2, on the rows this CTA owns
          float2 go[NR];
#pragma unroll
          for (int i = 0; i < NR; ++i) go[i] = RSx::ld_pair(t_go, rs.row(i, warp), lane);
          float zq[NR][2];
          rs.recv(zq, warp, lane, dq_tag);
#pragma unroll
          for (int i = 0; i < NR; ++i)
            RSx::st_pair_global(p.dXQ + static_cast<long>(row0) * 64, rs.row(i, warp), lane, go[i].x + zq[i][0],
                                go[i].y + zq[i][1]);
        }
        // likewise: the row sums that need no A2.  grad_output_fused = gamma x_hat_fused + beta - (V - K)
        float gof[NR][2], pre[2 * NR];
#pragma unroll
        for (int i = 0; i < NR; ++i) {
          gof[i][0] = fmaf(gam.x, xh[i].x, bet.x) - (vv[i].x - kr[i].x);
          gof[i][1] = fmaf(gam.y, xh[i].y, bet.y) - (vv[i].y - kr[i].y);
          pre[2 * i] = fmaf(gzr[i].x, gb2.x, gzr[i].y * gb2.y);
          pre[2 * i + 1] = fmaf(gof[i][0] * gam.x, xh[i].x, gof[i][1] * gam.y * xh[i].y);
        }
        RSx::row_sums(pre);
        float z[NR][2], ex[NR];
        rs.recv_x(z, ex, warp, lane, a2_tag);
        float ca0 = 0.f, ca1 = 0.f, cv0 = 0.f, cv1 = 0.f;
        float s23[2 * NR], gx[NR][2], sa[2 * NR];
#pragma unroll
        for (int i = 0; i < NR; ++i) {
          // the G_b2 parts of u = acc1 + G_b2
          z[i][0] = fmaf(-etar[i], gb2.x, z[i][0]);
          z[i][1] = fmaf(-etar[i], gb2.y, z[i][1]);
          s23[2 * i] = z[i][0] + z[i][1];
          s23[2 * i + 1] = fmaf(z[i][0], xh[i].x, z[i][1] * xh[i].y);
        }
        RSx::row_sums(s23);
#pragma unroll
        for (int i = 0; i < NR; ++i) {
          const int r = rs.row(i, warp);
          const float rstd = rsd[i], go0 = gof[i][0], go1 = gof[i][1], A0 = z[i][0], A1 = z[i][1];
          const float s2 = s23[2 * i], s3 = s23[2 * i + 1], s4 = pre[2 * i + 1];
          const float bt0 = (A0 - (s2 + xh[i].x * s3) * (1.f / 64.f)) * rstd;
          const float bt1 = (A1 - (s2 + xh[i].y * s3) * (1.f / 64.f)) * rstd;
          const float gly0 = gam.x * bt0, gly1 = gam.y * bt1;
          ca0 += fmaf(go0, bt0, gly0 * xh[i].x);      // d_gamma addends
          ca1 += fmaf(go1, bt1, gly1 * xh[i].y);
          cv0 += gly0;                                // d_beta addends
          cv1 += gly1;
          dk_gly[i][0] = gly0;
          dk_gly[i][1] = gly1;
          RSx::st_pair_global(p.dXV + static_cast<long>(row0) * 64, r, lane, -gly0, -gly1);
          const float gx0 = fmaf(gly0, gam.x, -(go0 * gam.x * s3 + A0 * s4) * rstd * (1.f / 64.f));
          const float gx1 = fmaf(gly1, gam.y, -(go1 * gam.y * s3 + A1 * s4) * rstd * (1.f / 64.f));
          sa[2 * i] = ((-gx0 * xh[i].x - A0 * gzr[i].x) + (-gx1 * xh[i].y - A1 * gzr[i].y)) * rstd;
          sa[2 * i + 1] = gx0 + gx1;
          gx[i][0] = gx0;
          gx[i][1] = gx1;
        }
        RSx::row_sums(sa);
#pragma unroll
        for (int i = 0; i < NR; ++i) {
          const int r = rs.row(i, warp);
          const float rstd = rsd[i], sa0 = sa[2 * i], sa1 = sa[2 * i + 1];
          rs.all_gather_store(t_q, &bars[BAR_AG], r, lane,
                              fmaf(gx[i][0], rstd, (sa0 * xh[i].x - sa1 * rstd) * (1.f / 64.f)),      // gZ2in
                              fmaf(gx[i][1], rstd, (sa0 * xh[i].y - sa1 * rstd) * (1.f / 64.f)));
          if (lane == 0) p.d_eta[(sid * NC + i0 + j) * 64 + r] = __float2bfloat16(-(ex[i] + pre[2 * i]));
        }
        *reinterpret_cast<float2*>(sXch + warp * 64 + 2 * lane) = make_float2(ca0, ca1);
        *reinterpret_cast<float2*>(sXch + 512 + warp * 64 + 2 * lane) = make_float2(cv0, cv1);
        wait_bar(BAR_AG);
      } else {
        TokFrag A2, t1, go;
        uint32_t gzw[8], xhw[8], kw[8], vw[8];
        frag_ld_raw(tm, t_gz2, gzw);
        frag_ld_raw(tm, t_xf, xhw);
        frag_ld_raw(tm, t_k, kw);
        frag_ld_raw(tm, t_a, vw);
        const float eta0 = __bfloat162float(sEta[tm.r0]), eta1 = __bfloat162float(sEta[tm.r1]);
        const float rs0 = sSigF[tm.r0], rs1 = sSigF[tm.r1];      // 1 / std
        float de0, de1;
        {
          // this CTA's shares: X2 G_W2 (acc1), P W2 (acc2), gZ1 G_W1 (t1).  Everything the step needs
          // from them is linear: A2 = -eta acc1 + acc2, the d_eta row sums of gz acc1 and of t1 K, and
          // -eta t1 inside dK; one cluster sum carries the first three, the dK sum the last.
          TokFrag acc1;
          frag_ld(tm, tmem + C::TM_B + 64, acc1);
          frag_ld(tm, tmem + C::TM_A, A2);
          frag_ld(tm, tmem + C::TM_B, t1);
          f32x2 s0 = 0ull, s1 = 0ull;
          float sum[16];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            s0 = fma2(bf16x2_to_f32x2(gzw[2 * q]), acc1.a[q], fma2(t1.a[q], bf16x2_to_f32x2(kw[2 * q]), s0));
            s1 = fma2(bf16x2_to_f32x2(gzw[2 * q + 1]), acc1.b[q], fma2(t1.b[q], bf16x2_to_f32x2(kw[2 * q + 1]), s1));
            upk(fma2(acc1.a[q], pk1(-eta0), A2.a[q]), sum[4 * q], sum[4 * q + 1]);
            upk(fma2(acc1.b[q], pk1(-eta1), A2.b[q]), sum[4 * q + 2], sum[4 * q + 3]);
          }
          de0 = hsum(s0);
          de1 = hsum(s1);
          if (row_writer) {     // the partial sums over this CTA's hidden units of gZ1 * G_b1, once per row
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              de0 += sPart[q * 64 + tm.r0];
              de1 += sPart[q * 64 + tm.r1];
            }
          }
          csum.run_with_extras(sum, de0, de1, tid, lane);
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            A2.a[q] = pk(sum[4 * q], sum[4 * q + 1]);
            A2.b[q] = pk(sum[4 * q + 2], sum[4 * q + 3]);
          }
        }
        float ra[4], rb[4];       // d_eta's row terms, sum A2, sum A2 xh, sum gxf xh
        {
          f32x2 s0[4] = {0ull, 0ull, 0ull, 0ull}, s1[4] = {0ull, 0ull, 0ull, 0ull};
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const f32x2 gam = frag_col(tm, sGamma, q), bet = frag_col(tm, sBeta, q), gb2 = frag_col(tm, sGb2, q), neg = pk1(-1.f);
            const f32x2 x0 = bf16x2_to_f32x2(xhw[2 * q]), x1 = bf16x2_to_f32x2(xhw[2 * q + 1]);
            // grad_output_fused = gamma x_hat_fused + beta - (V - K)
            go.a[q] = add2(fma2(bf16x2_to_f32x2(vw[2 * q]), neg, bf16x2_to_f32x2(kw[2 * q])), fma2(gam, x0, bet));
            go.b[q] = add2(fma2(bf16x2_to_f32x2(vw[2 * q + 1]), neg, bf16x2_to_f32x2(kw[2 * q + 1])), fma2(gam, x1, bet));
            // the G_b2 parts of u = acc1 + G_b2
            s0[0] = fma2(bf16x2_to_f32x2(gzw[2 * q]), gb2, s0[0]);
            s1[0] = fma2(bf16x2_to_f32x2(gzw[2 * q + 1]), gb2, s1[0]);
            A2.a[q] = fma2(gb2, pk1(-eta0), A2.a[q]);
            A2.b[q] = fma2(gb2, pk1(-eta1), A2.b[q]);
            s0[1] = add2(s0[1], A2.a[q]);
            s1[1] = add2(s1[1], A2.b[q]);
            s0[2] = fma2(A2.a[q], x0, s0[2]);
            s1[2] = fma2(A2.b[q], x1, s1[2]);
            s0[3] = fma2(mul2(go.a[q], gam), x0, s0[3]);
            s1[3] = fma2(mul2(go.b[q], gam), x1, s1[3]);
          }
#pragma unroll
          for (int i = 0; i < 4; ++i) { ra[i] = hsum(s0[i]); rb[i] = hsum(s1[i]); }
          ra[0] += de0;
          rb[0] += de1;
        }
        // all-reduce over the row's four lanes and two warps
#pragma unroll
        for (int sft = 1; sft <= 2; sft <<= 1)
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            ra[i] += __shfl_xor_sync(0xffffffffu, ra[i], sft);
            rb[i] += __shfl_xor_sync(0xffffffffu, rb[i], sft);
          }
        float4* x4 = reinterpret_cast<float4*>(sXch);      // 2 KB; the second exchange follows behind
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
        const int fc = tm.quad * 64 + frag_colsum_col(tm, lane);
        f32x2 sa0 = 0ull, sa1 = 0ull, sb0 = 0ull, sb1 = 0ull;      // sum g_std, sum g_xhat of the two rows
        f32x2 cs[4];
        {
          const f32x2 n64 = pk1(-1.f / 64.f);
          const f32x2 mA = mul2(pk1(ra[1]), n64), xA = mul2(pk1(ra[2]), n64), mB = mul2(pk1(rb[1]), n64), xB = mul2(pk1(rb[2]), n64);
          const f32x2 fA3 = pk1(-ra[2] * rs0 * (1.f / 64.f)), fA4 = pk1(-ra[3] * rs0 * (1.f / 64.f));
          const f32x2 fB3 = pk1(-rb[2] * rs1 * (1.f / 64.f)), fB4 = pk1(-rb[3] * rs1 * (1.f / 64.f));
          const f32x2 own = pk1(kp_owner ? 1.f : 0.f);     // gly enters dK once across the cluster: by the row's owner
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
            upk(fma2(t1.a[q], pk1(-eta0), mul2(gl0, own)), kp[4 * q], kp[4 * q + 1]);
            upk(fma2(t1.b[q], pk1(-eta1), mul2(gl1, own)), kp[4 * q + 2], kp[4 * q + 3]);
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
          part[256 + fc] = frag_colsum(cs, lane);
          part[512 + fc] = frag_colsum(cl, lane);
        }
        float sa[2] = {-hsum(sa0) * rs0, hsum(sa1)}, sb[2] = {-hsum(sb0) * rs1, hsum(sb1)};
        frag_allreduce2<0>(tm, sa, sb, sXch + 512, 1);
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
          part[fc] = frag_colsum(cs, lane);
        }
        if (row_writer && rank == 0) {
          p.d_eta[(sid * NC + i0 + j) * 64 + tm.r0] = __float2bfloat16(-ra[0]);
          p.d_eta[(sid * NC + i0 + j) * 64 + tm.r1] = __float2bfloat16(-rb[0]);
        }
      }
      publish();
      // G11 (+ G_W2snap U2^T) // G12
      if constexpr (!C::kRowSplit) {
        if (tid == kProd && (turn + 1) % kC == rank) {
          tma_store_2d(&tmDV, t_go, 0, row0);
          tma_commit_group();
        }
      }
      TTT_ISSUE4(HID_ONE(false, C::TM_B, big(ib1), t_q, 0u, 0); HID_ONE(false, C::TM_B, big(ib3), t_g, 1u, 0),
                 if (NB > 1) { HID_ONE(false, C::TM_B, big(ib1), t_q, 0u, NB - 1); HID_ONE(false, C::TM_B, big(ib3), t_g, 1u, NB - 1); }
                 else if (C::kMmaColsum) mma_colsum(tmem + C::TM_CS + 8, smem_u32(t_q), smem_u32(smem + C::OFF_ONES), lead),
                 HID_ONE(false, C::TM_A, big(ib1), t_gz2, 0u, 0),
                 if (NB > 1) HID_ONE(false, C::TM_A, big(ib1), t_gz2, 0u, NB - 1))
      if constexpr (C::kRowSplit) {
        // the second-order stage's d_gamma / d_beta partials (this CTA's rows only: summed over the cluster at
        // the end) are read out of the row-sum exchange area, which is used again after the next epilogue's barrier.  The
        // column sums of the gathered gZ2in tile (G_b2 stays replicated) come from the tensor pipe after the phase.
        if (tid < 64) {
          float a = 0.f, v = 0.f;
#pragma unroll
          for (int w = 0; w < 8; ++w) {
            a += sXch[w * 64 + tid];
            v += sXch[512 + w * 64 + tid];
          }
          sDGp[tid] += a;
          sDGp[64 + tid] += v;
        }
      } else {
        if (tid < 64) {
          sGb2[tid] += part_sum(0);
          sDG[tid] += part_sum(1);
          sDB[tid] += part_sum(2);
        }
      }
      wait_mma();
      if constexpr (C::kRowSplit) {
        if (warp < 4) {
          const float cs = colsum_read(tmem + C::TM_CS + 8, warp);
          if (lane < 16) sGb2[16 * warp + lane] += cs;
        }
      }
      if (tid == kProd) {
        // the W2 state-gradient snapshot is consumed: X2 comes back into its buffer for G14; dV has left
        // its tile, the d_gamma addends and x_hat_fused are consumed: the next step's first tiles are
        // requested now, two phases before they are needed
        load_big(ib3, p.sc_X2 + slot * BIG);
        tma_wait_group_read<0>();
        if (j > 0) issue_tiles_a(j - 1);
      }
      // ---- E5: gZ1in^T = gX2^T gelu'(Z1^T) + R^T S^T, in place over S^T
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        TokFrag v, w;
        uint32_t gp[8], sw[8];
        frag_ld(tm, tmem + C::TM_B + b * 64, v);
        frag_ld(tm, tmem + C::TM_A + b * 64, w);
        frag_ld_raw(tm, big(ib0) + b * TILE, gp);
        frag_ld_raw(tm, big(ib2) + b * TILE, sw);
        f32x2 s0 = 0ull, s1 = 0ull;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          v.a[q] = fma2(v.a[q], f16x2_to_f32x2(gp[2 * q]), mul2(w.a[q], bf16x2_to_f32x2(sw[2 * q])));
          v.b[q] = fma2(v.b[q], f16x2_to_f32x2(gp[2 * q + 1]), mul2(w.b[q], bf16x2_to_f32x2(sw[2 * q + 1])));
          s0 = add2(s0, v.a[q]);
          s1 = add2(s1, v.b[q]);
        }
        frag_st_tile(tm, big(ib2) + b * TILE, v);
        ga[b] = hsum(s0);
        gb[b] = hsum(s1);
      }
      publish();
      // gelu'(Z1) is consumed: the next step's gelu'(Z1_bar) comes into its buffer
      if (tid == kProd && j > 0) load_big(ib0, p.sc_Z1b + (slot - 1) * BIG);
      wait_bar(BAR_BIG + ib4);
      wait_bar(BAR_BIG + ib3);
      // G13 (partial dK) // G15 // G14
      TTT_ISSUE4(mma_tok_partial(tmem + C::TM_A, smem_u32(big(ib2)), smem_u32(big(ib4)), NB, lead),
                 HID_ALL(true, C::TM_S1, big(ib2), t_k, 1u),
                 HID_ONE(true, C::TM_S2, big(ib3), t_q, 1u, 0),
                 if (NB > 1) HID_ONE(true, C::TM_S2, big(ib3), t_q, 1u, NB - 1))
      tok_row_allreduce<NB, 0>(tm, ga, gb, sXch);
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        Gb1[b][0] += ga[b];
        Gb1[b][1] += gb[b];
      }
      wait_mma();
      // ---- E6: dK = sum over the cluster of (share of dK + gZ1in W1^T): an output only, summed by
      // reduce-scatter; every CTA stores the token rows it owns.  Sent now, received inside the first MMA
      // window of the next step (or right after the group's last step).
      {
        float acc[16];
        tok_ld(tm, tmem + C::TM_A, acc);
#pragma unroll
        for (int q = 0; q < 16; ++q) dk_pend[q] = kp[q] + acc[q];
        if constexpr (C::kRowSplit) dk_tag = rs.send(dk_pend, tid, warp, lane);
        else dk_tag = csum.reduce_scatter_send(dk_pend, tid);
        dk_row0 = row0;
      }
      aborted = publish_vote();
      // pre-update weights of this mini-batch are the post-update weights of the previous one
      {
        const int n0 = ib4, n1 = ib1, n2 = ib0, n3 = ib2, n4 = ib3;
        ib0 = n0; ib1 = n1; ib2 = n2; ib3 = n3; ib4 = n4;
      }
      if (tid == kProd && j > 0 && !aborted) issue_rest(j - 1);
      if (aborted) break;
    }
    if (aborted) break;
    if constexpr (C::kRowSplit) {      // the group's last dK
      if (dk_row0 >= 0) finish_dk_rows();
    } else {
      if (dk_row0 >= 0 && csum.reduce_scatter_recv(dk_pend, tid, dk_tag))
        tok_st_global(tm, p.dXK + static_cast<long>(dk_row0) * 64, dk_pend);
    }
    if (tid == kProd) tma_wait_group_read<0>();   // the last dV has left its tile (the recompute writes it again)

    // ---- park the gradient state (tensor memory -> grad_L_W*_init); the last group leaves the result
    __syncwarp();
#pragma unroll
    for (int b = 0; b < NB; ++b) {
      float w[16];
      tok_ld(tm, tmem + C::TM_S1 + b * 64, w);
      store_w1_frag(Gdst_W1, b, w);
      tok_ld(tm, tmem + C::TM_S2 + b * 64, w);
      store_w2_frag(Gdst_W2, b, w);
    }
    Gsrc_W1 = Gdst_W1;
    Gsrc_W2 = Gdst_W2;
    publish();
  }
#undef TTT_ISSUE4
#undef HID_ALL
#undef HID_ONE

  // ---- final vector outputs
  if (!aborted) {
    if (row_writer) {
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        p.gb1[sid * 256 + hid0 + 64 * b + tm.r0] = Gb1[b][0];
        p.gb1[sid * 256 + hid0 + 64 * b + tm.r1] = Gb1[b][1];
      }
    }
    if constexpr (C::kRowSplit) {
      // d_gamma / d_beta: the replicated addends (output LayerNorm) plus every CTA's own-row addends, summed by
      // rank 0 in rank order.  The peers' addends ([kC][2][64]) land in the exchange buffer after next: the last
      // sum that used it was received by every CTA before the last-but-one was sent.
      float* sFin = reinterpret_cast<float*>(rs.bufp + ((rs.n + 1u) & 3u) * C::RS::kBufBytes);
      if (rank == 0) {
        if (tid == 0) mbar_expect_tx(&bars[BAR_AG], (kC - 1) * 512u);
      } else if (tid < 32) {
        const float4 v = reinterpret_cast<const float4*>(sDGp)[tid];
        st_async_f4(mapa(smem_u32(sFin + rank * 128 + tid * 4), 0), mapa(smem_u32(&bars[BAR_AG]), 0), v.x, v.y, v.z, v.w);
      }
      if (rank == 0) {
        wait_bar(BAR_AG);
        if (tid < 64) {
          float dg = sDG[tid] + sDGp[tid], db = sDB[tid] + sDGp[64 + tid];
#pragma unroll
          for (int r = 1; r < kC; ++r) {
            dg += sFin[r * 128 + tid];
            db += sFin[r * 128 + 64 + tid];
          }
          p.gb2[sid * 64 + tid] = sGb2[tid];
          p.d_gamma[sid * 64 + tid] = dg;
          p.d_beta[sid * 64 + tid] = db;
        }
      }
    } else if (rank == 0 && tid < 64) {
      p.gb2[sid * 64 + tid] = sGb2[tid];
      p.d_gamma[sid * 64 + tid] = sDG[tid];
      p.d_beta[sid * 64 + tid] = sDB[tid];
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
  // no CTA leaves while a peer may still write into its shared memory (exchange area, abort flag)
  cluster_exit(abort_flag);
  if (warp == 0) tmem_dealloc(tmem, C::TM_COLS);
}

// Once per device: the kernel's dynamic shared memory limit.
template <int kC>
int prepare_kernel() {
  using C = Cfg<kC>;
  static std::once_flag once[64];
  static cudaError_t attr_err[64];
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return ttt_set_error(TTT_B200_ERR_LAUNCH, "device index out of range");
  std::call_once(once[dev], [&] {
    attr_err[dev] = cudaFuncSetAttribute(ttt_bwd_cluster_kernel<kC>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES);
  });
  if (attr_err[dev] != cudaSuccess) return ttt_set_error(TTT_B200_ERR_LAUNCH, cudaGetErrorString(attr_err[dev]));
  return TTT_B200_OK;
}

// How many clusters of kC CTAs the device runs at once (a cluster lives inside one GPC, and the GPCs' SM counts
// are not all multiples of kC: fewer than SMs / kC).  0 if the query fails.
template <int kC>
int cluster_capacity() {
  using C = Cfg<kC>;
  static std::once_flag once[64];
  static int cap[64];
  if (prepare_kernel<kC>()) return 0;
  int dev = 0;
  cudaGetDevice(&dev);
  std::call_once(once[dev], [&] {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kC * 64);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = C::SMEM_BYTES;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kC;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, ttt_bwd_cluster_kernel<kC>, &cfg) != cudaSuccess) {
      cudaGetLastError();
      n = 0;
    }
    cap[dev] = n;
  });
  return cap[dev];
}

template <int kC>
int launch_cluster(const CUtensorMap* tm, const BwdClParams& p, int streams, cudaStream_t stream) {
  using C = Cfg<kC>;
  if (int rc = prepare_kernel<kC>()) return rc;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(streams) * kC);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = C::SMEM_BYTES;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = kC;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaError_t e = cudaLaunchKernelEx(&cfg, ttt_bwd_cluster_kernel<kC>, tm[0], tm[1], tm[2], tm[3], tm[4], tm[5], tm[6], p);
  if (e != cudaSuccess) return ttt_set_error(TTT_B200_ERR_LAUNCH, cudaGetErrorString(e));
  return TTT_B200_OK;
}

}  // namespace

int ttt_launch_backward_cluster(const ttt_b200_bwd_args* a, int cluster, cudaStream_t stream, uint32_t* status,
                                uint64_t limit_ns, int drop_load) {
  const uint64_t rows = static_cast<uint64_t>(a->B) * a->H * a->NC * 64;
  CUtensorMap tm[7];
  const void* bases[7] = {a->XQ, a->XK, a->XV, a->grad_L_XQW_mini_batch, a->grad_L_XQ, a->grad_L_XK, a->grad_L_XV};
  for (int i = 0; i < 7; ++i)
    if (int rc = ttt_make_tile_map(&tm[i], bases[i], rows)) return rc;
  BwdClParams p;
  p.eta = static_cast<const __nv_bfloat16*>(a->last_eta);
  p.gamma = a->ttt_norm_weight;
  p.beta = a->ttt_norm_bias;
  p.W1c = a->W1_checkpoints; p.b1c = a->b1_checkpoints; p.W2c = a->W2_checkpoints; p.b2c = a->b2_checkpoints;
  p.sc_W1 = reinterpret_cast<uint8_t*>(a->W1_init_group);
  p.sc_W2 = reinterpret_cast<uint8_t*>(a->W2_init_group);
  p.sc_Z1 = static_cast<uint8_t*>(a->Z1_group);
  p.sc_X2 = static_cast<uint8_t*>(a->X2_group);
  p.sc_gZ1 = static_cast<uint8_t*>(a->grad_l_wrt_Z1_group);
  p.sc_Z1b = static_cast<uint8_t*>(a->Z1_bar_group);
  p.sc_X2b = static_cast<uint8_t*>(a->X2_bar_group);
  p.sc_xhf = static_cast<uint8_t*>(a->x_hat_fused_group);
  p.sc_gZ2 = static_cast<uint8_t*>(a->grad_l_wrt_Z2_group);
  p.sc_xhln = static_cast<uint8_t*>(a->x_hat_ln_group);
  p.sc_sigf = a->std_fused_group;
  p.sc_sigln = a->std_ln_group;
  p.gW1_last = a->grad_L_W1_last; p.gb1_last = a->grad_L_b1_last;
  p.gW2_last = a->grad_L_W2_last; p.gb2_last = a->grad_L_b2_last;
  p.d_gamma = a->grad_L_ttt_norm_weight; p.d_beta = a->grad_L_ttt_norm_bias;
  p.gW1 = a->grad_L_W1_init; p.gb1 = a->grad_L_b1_init; p.gW2 = a->grad_L_W2_init; p.gb2 = a->grad_L_b2_init;
  p.d_eta = static_cast<__nv_bfloat16*>(a->grad_L_last_eta);
  p.dXQ = static_cast<__nv_bfloat16*>(a->grad_L_XQ);
  p.dXK = static_cast<__nv_bfloat16*>(a->grad_L_XK);
  p.dXV = static_cast<__nv_bfloat16*>(a->grad_L_XV);
  p.H = a->H; p.NC = a->NC; p.cgs = a->checkpoint_group_size; p.nck = a->num_checkpoints;
  p.drop_load = drop_load;
  p.status = status;
  p.wait_limit_ns = limit_ns;
  const int streams = a->B * a->H;
  if (cluster == 2) return launch_cluster<2>(tm, p, streams, stream);
  if (cluster == 4) return launch_cluster<4>(tm, p, streams, stream);
  return ttt_set_error(TTT_B200_ERR_BAD_ARGS, "cluster size must be 2 or 4");
}

int ttt_backward_cluster_capacity(int cluster) {
  return cluster == 2 ? cluster_capacity<2>() : cluster == 4 ? cluster_capacity<4>() : 0;
}
