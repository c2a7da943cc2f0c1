// Host side of the C ABI: argument validation, tensor-map construction, status word,
// error text.  Replaces the host launchers of the reference
// (kernels/ttt/ttt.cu:594-721, kernels/ttt_backward/ttt.cu:1451-1917): same checks, made on
// every call (the reference's backward checks only on the first call of the process,
// kernels/ttt_backward/ttt.cu:1507-1508), and errors are returned instead of printed
// (kernels/ttt/ttt.cu:708-718).
#include <cuda.h>
#include <cuda_runtime.h>

#include <atomic>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <string>

#include "ttt_internal.h"

int ttt_launch_forward(const ttt_b200_fwd_args* a, cudaStream_t stream, uint32_t* status, uint64_t limit_ns,
                       int drop_load);
int ttt_launch_forward_pair(const ttt_b200_fwd_args* a, cudaStream_t stream, uint32_t* status, uint64_t limit_ns,
                            int drop_load);
int ttt_launch_backward(const ttt_b200_bwd_args* a, int streams, cudaStream_t stream, uint32_t* status, uint64_t limit_ns,
                        int drop_load);
int ttt_launch_backward_pair(const ttt_b200_bwd_args* a, int first, cudaStream_t stream, uint32_t* status, uint64_t limit_ns,
                             int drop_load);
int ttt_launch_backward_cluster(const ttt_b200_bwd_args* a, int cluster, cudaStream_t stream, uint32_t* status,
                                uint64_t limit_ns, int drop_load);
int ttt_launch_linear_forward(const ttt_b200_linear_fwd_args* a, cudaStream_t stream, uint32_t* status,
                              uint64_t limit_ns, int drop_load);
int ttt_launch_linear_backward(const ttt_b200_linear_bwd_args* a, cudaStream_t stream, uint32_t* status,
                               uint64_t limit_ns, int drop_load);
uint64_t ttt_linear_backward_scratch_bytes(int B, int H, int cgs);
int ttt_forward_cluster_capacity(int cluster);
int ttt_backward_cluster_capacity(int cluster);
int ttt_backward_pair_capacity();
int ttt_backward_pairs_a_turn();
int ttt_forward_pair_capacity();
int ttt_launch_forward_cluster(const ttt_b200_fwd_args* a, cudaStream_t stream, uint32_t* status, uint64_t limit_ns,
                               int drop_load);

namespace {

thread_local std::string g_last_error;

std::mutex g_mu;
uint32_t* g_status_host = nullptr;   // pinned, device-visible
uint32_t* g_status_dev = nullptr;

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

uint64_t wait_limit_ns() { return ttt_wait_limit_ns(); }

// ... of the kernels that recompute a checkpoint group beside the sweep of another (MLP backward with two CTAs per stream,
// TTT-Linear backward): the sweep waits for the first group's whole recompute, which takes 9 to 12 us per mini-batch (MLP;
// TTT-Linear at most 5) on an SM that nothing else uses.  It is allowed 100 on top of the limit.
uint64_t wait_limit_ns(int cgs, int NC) { return wait_limit_ns() + static_cast<uint64_t>(cgs < NC ? cgs : NC) * 100000ull; }

}  // namespace

// Device-side waits give up after this long (nanoseconds).  A healthy launch never waits more than microseconds, but for
// one group's recompute where that is waited for as a whole (wait_limit_ns of a group's size); the limit only decides how
// fast a lost signal is reported.
uint64_t ttt_wait_limit_ns() {
  static uint64_t v = [] {
    const char* e = std::getenv("TTT_B200_WAIT_LIMIT_MS");
    long ms = e ? std::atol(e) : 2000;
    if (ms < 1) ms = 1;
    return static_cast<uint64_t>(ms) * 1000000ull;
  }();
  return v;
}

namespace {

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

}  // namespace

namespace {

// The cluster size that the flags or, failing them, TTT_B200_CLUSTER ask for; 0: neither names one.
int asked_cluster(uint32_t flags, int* cluster) {
  *cluster = static_cast<int>((flags & TTT_B200_FLAG_CLUSTER_MASK) >> TTT_B200_FLAG_CLUSTER_SHIFT);
  if (*cluster == 0) {
    static const int env = [] {
      const char* e = std::getenv("TTT_B200_CLUSTER");
      return e ? std::atoi(e) : 0;
    }();
    *cluster = env;
  }
  if (*cluster != 0 && *cluster != 1 && *cluster != 2 && *cluster != 4)
    return ttt_set_error(TTT_B200_ERR_BAD_ARGS, "cluster size must be 1, 2 or 4");
  return TTT_B200_OK;
}

int capacity(int cluster, bool backward) {
  return backward ? ttt_backward_cluster_capacity(cluster) : ttt_forward_cluster_capacity(cluster);
}

}  // namespace

// How many CTAs share one stream.  The mini-batches of a stream are strictly sequential, so with fewer
// streams than SMs the idle SMs can only help by taking a share of every stream's hidden units, and only while all
// streams are resident at once.  Four CTAs per stream win whenever the device runs that many clusters of four (32 streams
// of 128 mini-batches in groups of 4 on a B200: forward 4.3 against 4.6 us per mini-batch with one CTA, backward 14.0
// against 22.7; of longer calls: forward_ctas, backward_ctas).  Where only clusters of two fit (34 to 74 streams), short
// forwards run one CTA, whose output pass runs beside the chain in two groups of warps, and the backward two (60 streams in groups of 5: 11.7 us per mini-batch against 23.3 with
// one).  Beyond, one.
static int ttt_launch_cluster(int streams, uint32_t flags, bool backward, int* cluster) {
  if (int rc = asked_cluster(flags, cluster)) return rc;
  if (*cluster != 0) return TTT_B200_OK;
  if (streams <= capacity(4, backward)) *cluster = 4;
  else if (backward && streams <= capacity(2, backward)) *cluster = 2;
  else *cluster = 1;
  return TTT_B200_OK;
}

// CTAs per stream of a forward.  Two where the device runs all streams as pairs at once and that is the faster form: against
// one CTA from six mini-batches on (us, one CTA / pair: 34 streams x 4 in groups of 2 27.6 / 27.5, x 6 in groups of 3 35.5 /
// 34.9, x 16 in groups of 4 79 / 72; 66 streams x 6 in one group 34.6 / 34.6; 48 x 32 in groups of 6 147 / 136, in groups of 1 203 / 177), against four, which share
// the writing of the state, from 16 mini-batches in groups of four on (four / pair: 12 streams x 12 in groups of 4 54.8 /
// 56.1, x 16 71.9 / 70.5, 33 streams x 16 72.1 / 71.1; x 32 in groups of 6 138 / 131, x 16 in groups of 2 72.7 / 77.6; 32 x 128 in groups of 16 536 / 489).
// Two are always the chain and the output pass (ttt_fwd_pair_sm100.cu), whatever the call's length: a sequence in chunks, with
// the size named, then has the bits of one call.  (Half of the hidden units each is faster up to three mini-batches, 12 streams
// x 1 10.9 / 14.5 us, but no rule takes two there.)
static int forward_ctas(int streams, int NC, int cgs, uint32_t flags, int* ctas) {
  if (int rc = ttt_launch_cluster(streams, flags, false, ctas)) return rc;
  int asked = 0;
  if (asked_cluster(flags, &asked) != TTT_B200_OK || asked != 0 || streams > ttt_forward_pair_capacity()) return TTT_B200_OK;
  if (*ctas == 4 ? NC >= 16 && cgs >= 4 : NC >= 6) *ctas = 2;
  return TTT_B200_OK;
}

// A backward with two CTAs per stream gives them the recompute and the sweep (ttt_bwd_pair_sm100.cu) where there is
// something to do side by side: groups of several mini-batches, and more than one of them.  Else each takes half of the
// hidden units: a single group is within 4 % either way, groups of one mini-batch (one scratch slot, so that the two CTAs
// of a pair take turns) 26 us per mini-batch against 28.
static bool runs_pair(int ctas, int NC, int cgs) { return ctas == 2 && cgs > 1 && NC > cgs; }

// CTAs per stream of a backward.  Where four would fit, two are faster once a call has two groups of eight mini-batches or
// three of four to pipeline: the first group's recompute runs alone, and a group that has few slots to spare ends with a wait
// for the last of the next (32 streams, pair against four CTAs, us per mini-batch: 256 mini-batches in groups of 16 8.5 / 13.2,
// 48 in groups of 16 10.4 / 13.5, 24 in groups of 8 11.4 / 14.0, 12 in groups of 4 13.0 / 14.8; two groups: 32 in groups of 16
// 11.6 / 13.5, 16 in groups of 8 12.8 / 14.2, 12 streams 11.8 / 13.8, 8 in groups of 4 14.4 / 15.3; a short second group: 12 in
// groups of 8 14.1 / 14.5, 20 in groups of 16 13.9 / 13.9, 9 in groups of 8 16.5 / 15.3; small groups: 32 in groups of 3 13.7 /
// 14.8 and 6 16.4 / 15.7, 32 in groups of 2 16.0 / 15.5).
static int backward_ctas(int streams, int NC, int cgs, uint32_t flags, int* ctas) {
  if (int rc = ttt_launch_cluster(streams, flags, true, ctas)) return rc;
  int asked = 0;
  if (asked_cluster(flags, &asked) == TTT_B200_OK && asked == 0 && *ctas == 4 && cgs >= 4 && NC >= (cgs >= 8 ? 2 : 3) * cgs)
    *ctas = 2;
  return TTT_B200_OK;
}

// Streams of a call for one CTA per stream that two CTAs per stream take, in a launch of their own after the others': those
// beyond a multiple of the SMs, when the device runs them as pairs at once.  A turn over the SMs with one CTA per stream lasts
// 21.7 us per mini-batch however few streams are in it, one of pairs 9 to 13 and some us of launch.  Backward, us, without
// and with it: 176 streams x 64 in groups of 8 2783 / 2025, 192 x 37 in groups of 6 1681 / 1280, 312 x 52 in groups of 7 3454 /
// 2860, 1536 x 16 in groups of 4 4272 / 4141; where pairs are most and have least to pipeline, 222 streams x 8 in groups of 2
// 459 / 421, x 5 309 / 296, x 4 238 / 239, x 3 199 / 201, 370 x 3 300 / 304.  So it gains from five mini-batches on and is
// within 2 % below (149 and 176 streams x 4 in groups of 2 236 / 233 and 235 / 229, x 3 196 / 198 and 195 / 194).
//
// All of them, in two turns, where those hold them and are faster than one turn of single CTAs: per mini-batch two turns of
// pairs take 18 to 20 us, one of single CTAs 21 to 22, but each turn starts with a recompute that nothing runs beside.  So it
// takes groups to pipeline, and groups long enough that the sweep does not wait for the recompute.  Us, one CTA / pairs: 128
// streams x 128 in groups of 8 2770 / 2458, x 64 1397 / 1295, x 64 in groups of 6 1435 / 1395, x 96 in groups of 12 2030 / 1869,
// x 128 in groups of 20 2667 / 2457, 75 streams x 64 in groups of 8 1380 / 1244; 128 streams x 40 in groups of 5 921 / 938, x 64
// in groups of 4 1517 / 1518, of 16 1344 / 1387, x 32 in groups of 6 735 / 769.  On the line itself, 75 / 96 / 112 / 128 / 132
// streams (132 is two full turns): six groups of eight 1043 / 975, 1046 / 993, 1048 / 1007, 1053 / 1015, 1055 / 1023; of nine 1163 /
// 1072, 1166 / 1099, 1167 / 1107, 1172 / 1123, 1174 / 1142; ten of six 1331 / 1279, 1333 / 1290, 1337 / 1309, 1345 / 1335, 1349 / 1353.
static int backward_tail(int streams, int NC, int cgs, uint32_t flags, int ctas) {
  int asked = 0, dev = 0, sms = 0;
  if (ctas != 1 || !runs_pair(2, NC, cgs) || asked_cluster(flags, &asked) != TTT_B200_OK || asked != 0) return 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms < 1)
    return 0;
  if (streams <= 2 * ttt_backward_pairs_a_turn() && (cgs >= 8 ? NC >= 6 * cgs : cgs >= 6 && NC >= 10 * cgs)) return streams;
  const int rest = streams % sms;      // SMs hold one CTA each
  return streams > sms && rest <= ttt_backward_pair_capacity() ? rest : 0;
}

int ttt_set_error(int code, const char* msg) {
  g_last_error = msg ? msg : "";
  return code;
}

int ttt_status_word(uint32_t** dev_ptr) {
  std::lock_guard<std::mutex> lk(g_mu);
  if (!g_status_host) {
    cudaError_t e = cudaHostAlloc(reinterpret_cast<void**>(&g_status_host), sizeof(uint32_t),
                                  cudaHostAllocMapped | cudaHostAllocPortable);
    if (e != cudaSuccess) return ttt_set_error(TTT_B200_ERR_LAUNCH, cudaGetErrorString(e));
    *g_status_host = 0;
    e = cudaHostGetDevicePointer(reinterpret_cast<void**>(&g_status_dev), g_status_host, 0);
    if (e != cudaSuccess) return ttt_set_error(TTT_B200_ERR_LAUNCH, cudaGetErrorString(e));
  }
  *dev_ptr = g_status_dev;
  return TTT_B200_OK;
}

uint32_t ttt_take_status() {
  std::lock_guard<std::mutex> lk(g_mu);
  if (!g_status_host) return 0;
  volatile uint32_t* w = g_status_host;
  const uint32_t v = *w;
  *w = 0;
  return v;
}

int ttt_check_status(cudaStream_t stream) {
  cudaError_t e = cudaStreamSynchronize(stream);
  if (e != cudaSuccess) return ttt_set_error(TTT_B200_ERR_LAUNCH, cudaGetErrorString(e));
  if (ttt_take_status() != 0)
    return ttt_set_error(TTT_B200_ERR_TIMEOUT, "a device-side bounded wait ran out; results are invalid");
  return TTT_B200_OK;
}

// Encoded on every call, nothing is kept by the address of a caller's buffer: an encode takes less than 0.1 us of host
// time.  A forward of one mini-batch, which has four, is enqueued in 4.2 us; with maps kept in a table of 64 searched
// under a lock it took 4.5 us when all four were found and 4.8 us when none was (calls that rotate over 40 sets of
// buffers, as a model's layers do).
int ttt_make_tile_map(CUtensorMap* map, const void* base, uint64_t rows) {
  static std::atomic<EncodeTiledFn> encode{nullptr};
  EncodeTiledFn fn = encode.load(std::memory_order_relaxed);
  if (!fn) {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult qres;
    const cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &qres);
    if (e != cudaSuccess || qres != cudaDriverEntryPointSuccess || !f)
      return ttt_set_error(TTT_B200_ERR_LAUNCH, "cuTensorMapEncodeTiled is not available from the driver");
    fn = reinterpret_cast<EncodeTiledFn>(f);
    encode.store(fn, std::memory_order_relaxed);
  }
  const cuuint64_t dims[2] = {64, rows};
  const cuuint64_t strides[1] = {128};           // bytes between rows
  const cuuint32_t box[2] = {64, 64};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    char buf[96];
    std::snprintf(buf, sizeof buf, "cuTensorMapEncodeTiled failed with CUresult %d", static_cast<int>(r));
    return ttt_set_error(TTT_B200_ERR_LAUNCH, buf);
  }
  return TTT_B200_OK;
}

namespace {

#define TTT_REQUIRE(cond, msg) \
  do {                         \
    if (!(cond)) return ttt_set_error(TTT_B200_ERR_BAD_ARGS, msg); \
  } while (0)

int check_dims(int B, int H, int NC, int cgs, int nck) {
  TTT_REQUIRE(B >= 1 && H >= 1, "B and H must be >= 1");
  TTT_REQUIRE(NC >= 1, "NC (sequence length / 64) must be >= 1");
  TTT_REQUIRE(cgs >= 1, "checkpoint_group_size must be >= 1");
  TTT_REQUIRE(nck == (NC + cgs - 1) / cgs, "checkpoint tensors must hold ceil(NC / checkpoint_group_size) states");
  TTT_REQUIRE(static_cast<uint64_t>(B) * H * NC * 64 < (1ull << 31), "B*H*NC*64 must be below 2^31");
  return TTT_B200_OK;
}

int pre_launch(uint32_t** status) {
  if (int rc = ttt_status_word(status)) return rc;
  if (ttt_take_status() != 0)
    return ttt_set_error(TTT_B200_ERR_TIMEOUT,
                         "an earlier launch reported a device-side wait that ran out; its results are invalid");
  return TTT_B200_OK;
}

}  // namespace

extern "C" int ttt_b200_forward(const ttt_b200_fwd_args* a, void* stream_) {
  TTT_REQUIRE(a != nullptr, "args is NULL");
  if (int rc = check_dims(a->B, a->H, a->NC, a->checkpoint_group_size, a->num_checkpoints)) return rc;
  const void* ptrs[] = {a->XQ, a->XK, a->XV, a->last_eta, a->ttt_norm_weight, a->ttt_norm_bias, a->W1, a->b1,
                        a->W2, a->b2, a->W1_checkpoints, a->b1_checkpoints, a->W2_checkpoints, a->b2_checkpoints,
                        a->Out};
  for (const void* q : ptrs) {
    TTT_REQUIRE(q != nullptr, "a required tensor pointer is NULL");
    TTT_REQUIRE(aligned16(q), "tensor pointers must be 16-byte aligned");
  }
  const int nfinal = (a->W1_final != nullptr) + (a->b1_final != nullptr) + (a->W2_final != nullptr) +
                     (a->b2_final != nullptr);
  TTT_REQUIRE(nfinal == 0 || nfinal == 4, "W1/b1/W2/b2_final must be given together or not at all");
  if (nfinal == 4)
    TTT_REQUIRE(aligned16(a->W1_final) && aligned16(a->b1_final) && aligned16(a->W2_final) && aligned16(a->b2_final),
                "tensor pointers must be 16-byte aligned");
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  uint32_t* status = nullptr;
  if (int rc = pre_launch(&status)) return rc;
  const int streams = a->B * a->H;
  int ctas = 1;
  if (int rc = forward_ctas(streams, a->NC, a->checkpoint_group_size, a->flags, &ctas)) return rc;
  const int drop = (a->flags & TTT_B200_FLAG_TEST_LOST_LOAD) ? (a->NC > 1 ? 1 : 0) : -1;
  if (ctas == 1) {
    if (int rc = ttt_launch_forward(a, stream, status, wait_limit_ns(), drop)) return rc;
  } else if (ctas == 2) {
    if (int rc = ttt_launch_forward_pair(a, stream, status, wait_limit_ns(), drop)) return rc;
  } else if (int rc = ttt_launch_forward_cluster(a, stream, status, wait_limit_ns(), drop)) {
    return rc;
  }
  if (a->flags & TTT_B200_FLAG_SYNC) return ttt_check_status(stream);
  return TTT_B200_OK;
}

extern "C" int ttt_b200_linear_forward(const ttt_b200_linear_fwd_args* a, void* stream_) {
  TTT_REQUIRE(a != nullptr, "args is NULL");
  if (int rc = check_dims(a->B, a->H, a->NC, a->checkpoint_group_size, a->num_checkpoints)) return rc;
  const void* ptrs[] = {a->XQ, a->XK, a->XV, a->last_eta, a->ttt_norm_weight, a->ttt_norm_bias, a->W1, a->b1,
                        a->W1_checkpoints, a->b1_checkpoints, a->Out};
  for (const void* q : ptrs) {
    TTT_REQUIRE(q != nullptr, "a required tensor pointer is NULL");
    TTT_REQUIRE(aligned16(q), "tensor pointers must be 16-byte aligned");
  }
  TTT_REQUIRE((a->W1_final != nullptr) == (a->b1_final != nullptr), "W1_final and b1_final must be given together or not at all");
  if (a->W1_final != nullptr)
    TTT_REQUIRE(aligned16(a->W1_final) && aligned16(a->b1_final), "tensor pointers must be 16-byte aligned");
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  uint32_t* status = nullptr;
  if (int rc = pre_launch(&status)) return rc;
  const int drop = (a->flags & TTT_B200_FLAG_TEST_LOST_LOAD) ? (a->NC > 1 ? 1 : 0) : -1;
  if (int rc = ttt_launch_linear_forward(a, stream, status, wait_limit_ns(), drop)) return rc;
  if (a->flags & TTT_B200_FLAG_SYNC) return ttt_check_status(stream);
  return TTT_B200_OK;
}

extern "C" uint64_t ttt_b200_linear_backward_scratch_bytes(int B, int H, int checkpoint_group_size) {
  if (B < 1 || H < 1 || checkpoint_group_size < 1) return 0;
  return ttt_linear_backward_scratch_bytes(B, H, checkpoint_group_size);
}

extern "C" int ttt_b200_linear_backward(const ttt_b200_linear_bwd_args* a, void* stream_) {
  TTT_REQUIRE(a != nullptr, "args is NULL");
  if (int rc = check_dims(a->B, a->H, a->NC, a->checkpoint_group_size, a->num_checkpoints)) return rc;
  const void* ptrs[] = {a->XQ, a->XK, a->XV, a->last_eta, a->ttt_norm_weight, a->ttt_norm_bias, a->W1_checkpoints,
                        a->b1_checkpoints, a->grad_L_W1_last, a->grad_L_b1_last, a->grad_L_XQW_mini_batch, a->scratch,
                        a->grad_L_ttt_norm_weight, a->grad_L_ttt_norm_bias, a->grad_L_W1_init, a->grad_L_b1_init,
                        a->grad_L_last_eta, a->grad_L_XQ, a->grad_L_XK, a->grad_L_XV};
  for (const void* q : ptrs) {
    TTT_REQUIRE(q != nullptr, "a required tensor pointer is NULL");
    TTT_REQUIRE(aligned16(q), "tensor pointers must be 16-byte aligned");
  }
  TTT_REQUIRE(a->scratch_bytes >= ttt_linear_backward_scratch_bytes(a->B, a->H, a->checkpoint_group_size),
              "scratch is smaller than ttt_b200_linear_backward_scratch_bytes(B, H, checkpoint_group_size)");
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  uint32_t* status = nullptr;
  if (int rc = pre_launch(&status)) return rc;
  // the hook drops the recompute inputs of the last group's second mini-batch (its only one if it has one)
  const int last0 = (a->num_checkpoints - 1) * a->checkpoint_group_size;
  const int drop = (a->flags & TTT_B200_FLAG_TEST_LOST_LOAD) ? (last0 + 1 < a->NC ? last0 + 1 : last0) : -1;
  if (int rc = ttt_launch_linear_backward(a, stream, status, wait_limit_ns(a->checkpoint_group_size, a->NC), drop)) return rc;
  if (a->flags & TTT_B200_FLAG_SYNC) return ttt_check_status(stream);
  return TTT_B200_OK;
}

extern "C" int ttt_b200_backward(const ttt_b200_bwd_args* a, void* stream_) {
  TTT_REQUIRE(a != nullptr, "args is NULL");
  if (int rc = check_dims(a->B, a->H, a->NC, a->checkpoint_group_size, a->num_checkpoints)) return rc;
  const void* ptrs[] = {a->XQ, a->XK, a->XV, a->last_eta, a->ttt_norm_weight, a->ttt_norm_bias,
                        a->W1_checkpoints, a->b1_checkpoints, a->W2_checkpoints, a->b2_checkpoints,
                        a->W1_init_group, a->b1_init_group, a->W2_init_group, a->b2_init_group,
                        a->x_hat_ln_group, a->std_ln_group, a->X2_group, a->Z1_group, a->Z1_bar_group,
                        a->X2_bar_group, a->grad_l_wrt_Z2_group, a->grad_l_wrt_Z1_group, a->x_hat_fused_group,
                        a->grad_x_hat_fused_group, a->grad_output_fused_group, a->std_fused_group,
                        a->grad_L_W1_last, a->grad_L_b1_last, a->grad_L_W2_last, a->grad_L_b2_last,
                        a->grad_L_XQW_mini_batch, a->grad_L_ttt_norm_weight, a->grad_L_ttt_norm_bias,
                        a->grad_L_W1_init, a->grad_L_b1_init, a->grad_L_W2_init, a->grad_L_b2_init,
                        a->grad_L_last_eta, a->grad_L_XQ, a->grad_L_XK, a->grad_L_XV};
  for (const void* q : ptrs) {
    TTT_REQUIRE(q != nullptr, "a required tensor pointer is NULL");
    TTT_REQUIRE(aligned16(q), "tensor pointers must be 16-byte aligned");
  }
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  uint32_t* status = nullptr;
  if (int rc = pre_launch(&status)) return rc;
  int cluster = 1;
  if (int rc = backward_ctas(a->B * a->H, a->NC, a->checkpoint_group_size, a->flags, &cluster)) return rc;
  // the hook drops the recompute inputs of the last group's second mini-batch (its only one if it has one)
  const int last0 = (a->num_checkpoints - 1) * a->checkpoint_group_size;
  const int drop = (a->flags & TTT_B200_FLAG_TEST_LOST_LOAD) ? (last0 + 1 < a->NC ? last0 + 1 : last0) : -1;
  const uint64_t pair_limit = wait_limit_ns(a->checkpoint_group_size, a->NC);
  const int streams = a->B * a->H, tail = backward_tail(streams, a->NC, a->checkpoint_group_size, a->flags, cluster);
  if (cluster == 1) {
    if (tail < streams)
      if (int rc = ttt_launch_backward(a, streams - tail, stream, status, wait_limit_ns(), drop)) return rc;
    if (tail > 0)
      if (int rc = ttt_launch_backward_pair(a, streams - tail, stream, status, pair_limit, drop)) return rc;
  } else if (runs_pair(cluster, a->NC, a->checkpoint_group_size)) {
    if (int rc = ttt_launch_backward_pair(a, 0, stream, status, pair_limit, drop)) return rc;
  } else if (int rc = ttt_launch_backward_cluster(a, cluster, stream, status, wait_limit_ns(), drop)) {
    return rc;
  }
  if (a->flags & TTT_B200_FLAG_SYNC) return ttt_check_status(stream);
  return TTT_B200_OK;
}

extern "C" const char* ttt_b200_last_error(void) { return g_last_error.c_str(); }

extern "C" int ttt_b200_take_status(void) {
  const uint32_t a = ttt_take_status();
  const uint32_t b = ttt_noalloc_take_status();
  return (a | b) ? TTT_B200_ERR_TIMEOUT : TTT_B200_OK;
}

extern "C" int ttt_b200_version(void) { return 1001; }

extern "C" int ttt_b200_cluster_capacity(int cluster, int backward) {
  return backward ? ttt_backward_cluster_capacity(cluster) : ttt_forward_cluster_capacity(cluster);
}

// The widest size whose capacity covers the streams (two in the forward only): a property of the device, kept for its
// callers.  What a call runs is the answer of ttt_b200_forward_ctas and ttt_b200_backward_ctas.
extern "C" int ttt_b200_pick_cluster(int streams, int backward) {
  int c = 0;
  if (streams < 1 || asked_cluster(0u, &c) != TTT_B200_OK) return -1;
  if (c != 0) return c;
  if (streams <= capacity(4, backward != 0)) return 4;
  return !backward && streams <= capacity(2, false) ? 2 : 1;
}

extern "C" int ttt_b200_forward_ctas(int streams, int NC, int checkpoint_group_size, uint32_t flags) {
  int c = 0;
  if (streams < 1 || NC < 1 || checkpoint_group_size < 1) return -1;
  return forward_ctas(streams, NC, checkpoint_group_size, flags, &c) == TTT_B200_OK ? c : -1;
}

extern "C" int ttt_b200_backward_ctas(int streams, int NC, int checkpoint_group_size, uint32_t flags) {
  int c = 0;
  if (streams < 1 || NC < 1 || checkpoint_group_size < 1) return -1;
  return backward_ctas(streams, NC, checkpoint_group_size, flags, &c) == TTT_B200_OK ? c : -1;
}

extern "C" int ttt_b200_backward_tail(int streams, int NC, int checkpoint_group_size, uint32_t flags) {
  const int c = ttt_b200_backward_ctas(streams, NC, checkpoint_group_size, flags);
  return c < 0 ? -1 : backward_tail(streams, NC, checkpoint_group_size, flags, c);
}

extern "C" int ttt_b200_backward_pairs(int streams, int NC, int checkpoint_group_size, uint32_t flags) {
  const int c = ttt_b200_backward_ctas(streams, NC, checkpoint_group_size, flags);
  if (c < 0) return -1;
  return runs_pair(c, NC, checkpoint_group_size) ? streams : backward_tail(streams, NC, checkpoint_group_size, flags, c);
}

extern "C" int ttt_b200_launch_cluster(int streams, uint32_t flags, int backward) {
  int c = 0;
  if (streams < 1 || ttt_launch_cluster(streams, flags, backward != 0, &c) != TTT_B200_OK) return -1;
  return c;
}
