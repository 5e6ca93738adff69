// runtime.h -- host-side runtime of libgeye_dpm: context, plans, pipeline.
#pragma once
#include <cuda_runtime.h>

#include <atomic>
#include <map>
#include <set>
#include <memory>
#include <string>
#include <vector>

#include "internal.h"

// status plumbing shared by the host translation units
#define CUDA_TRY(call)                                                   \
  do {                                                                   \
    cudaError_t e_ = (call);                                             \
    if (e_ != cudaSuccess) {                                             \
      geye::set_error(std::string(#call) + ": " + cudaGetErrorString(e_)); \
      return GEYE_ERR_CUDA;                                              \
    }                                                                    \
  } while (0)
#define GEYE_TRY(call)            \
  do {                            \
    geye_status s_ = (call);      \
    if (s_ != GEYE_OK) return s_; \
  } while (0)
#define ARG_CHECK(cond, msg)   \
  do {                         \
    if (!(cond)) {             \
      geye::set_error(msg);    \
      return GEYE_ERR_ARG;     \
    }                          \
  } while (0)
// a model's filters live on the device of the context that loaded it, and are freed
// with that context: it runs only there, and only while that context lives
#define MODEL_CHECK(m, dev)                                                          \
  do {                                                                               \
    ARG_CHECK((m), "null model");                                                    \
    ARG_CHECK((m)->ctx, "the model's context was destroyed");                        \
    ARG_CHECK((m)->ctx->device == (dev), "the model was loaded on another device");  \
  } while (0)

namespace geye {

// thread-local error text, set by every failing entry point
void set_error(const std::string &msg);

struct DevBuf;
struct Plan;
struct ModelPlan;
// copies n bytes from the host into buf (allocated to fit)
geye_status upload_bytes(geye_ctx *ctx, DevBuf &buf, const void *src, size_t n);
struct ArenaAlloc;
// tensor-core convolution of a plan's models together (conv_tc.cu): tables and
// arena space before the arena exists, bank and tuned chunks after, the launch
geye_status plan_tc(geye_ctx *ctx, Plan &P, ArenaAlloc &A);
geye_status build_tc_plan(geye_ctx *ctx, Plan &P);
geye_status run_conv_tc(geye_ctx *ctx, Plan &P);
// d_small[kNmsNeed + m]: model m's kept set was resolved again in the quicksort's order
constexpr int kNmsNeed = 160;
// *err gets the kernel's error word once the stream has drained (0: no wait ran out)
// tensor-core fconvsMT of one feature map (float planes on the device) for the stage entry point
geye_status conv_tc_maps(geye_ctx *ctx, const float *d_feat, int a0, int a1, const float *const *filters,
                         const int *b_dims, int n_filters, float *d_out, const std::vector<int> &out_off,
                         std::vector<std::unique_ptr<DevBuf>> &tmp, int *err);

// Bump allocator of a plan's float arena (128-byte aligned offsets, in words).
struct ArenaAlloc {
  size_t words = 0;
  int take(size_t n) {
    size_t o = (words + 31) & ~size_t(31);   // 128-byte alignment
    words = o + n;
    return (int)o;
  }
};

// the n-th call of `op` fails by request (geye_debug_inject_fault)
bool injected(geye_ctx *ctx, const char *op);

// cudaMalloc; where there is not enough, the device's idle scratch (below) is given back and it is tried again
cudaError_t device_malloc(void **out, size_t n);

// Device memory of a context's stage calls: handed out piece by piece during a
// call, all of it free again at its end (reset), and kept for the next one
// (up to kScratchKeep bytes; cudaMalloc and cudaFree synchronise and cost more than most stages).
// Between two calls any context's allocation that fails may take it (device_malloc), from any thread.
struct ScratchArena {
  struct Chunk {
    char *p;
    size_t bytes;
  };
  std::vector<Chunk> chunks;   // the last one is being handed out
  size_t used = 0;             // of the last chunk
  size_t total = 0;            // handed out since the last reset
  size_t want = 0;             // the largest call so far
  int device = 0;
  bool busy = false;           // a call has memory of it (changed and, by other threads, read under the list's mutex)
  ~ScratchArena() { release(); }
  void release();
  geye_status take(geye_ctx *ctx, size_t n, void **out);
  void reset();                // the stream has drained
};
constexpr size_t kScratchKeep = 512ull << 20;

// Device buffer owned by a plan or context, or (arena) a piece of a context's scratch.
struct DevBuf {
  void *p = nullptr;
  size_t bytes = 0;
  ScratchArena *arena = nullptr;
  DevBuf() = default;
  explicit DevBuf(ScratchArena *a) : arena(a) {}
  ~DevBuf();
  geye_status alloc(geye_ctx *ctx, size_t n);
  void release();
  template <class T> T *as() const { return reinterpret_cast<T *>(p); }
};

// Host memory handed to callers, who free it with geye_free, or with free() like the reference's
// results: blocks of a megabyte and more that come back through geye_free are kept for the next
// call (kHostKeep bytes in all, until the last context goes or an allocation fails), since fresh
// pages cost more than the copy into them.
void *host_alloc(size_t n);
void host_free(void *p);
void host_pool_ref(int d);   // contexts come (+1) and go (-1)

// Results of a frame in pinned host memory, written by the NMS kernels: ints [0, 32)
// boxes before NMS per model, [32, 64) kept per model, then per model point[4R], or_point[4R], type[R], scale[R], score[R]
constexpr int kHostRes = 2048;
inline size_t res_block_ints(int n_models) { return 64 + (size_t)n_models * 11 * kHostRes; }
// model mi's result of the plan's finished frame (out: geye_result_free); parked: of the frame put aside by park_pending
geye_status read_result(Plan &P, int mi, geye_result *out, bool parked = false);
// A submitted frame's results put aside, in stream order, before another frame runs on its plan (and writes the plan's
// result block) while they have not been collected
geye_status park_pending(geye_ctx *ctx, Plan &P);
void tune_plan(geye_ctx *ctx, Plan &P);

struct LevelInfo {
  int img_h = 0, img_w = 0;   // image of this level (aliases for [interval, 2*interval))
  int img_level = 0;          // level whose image planes are used
  int img_off = -1;           // word offset of the planes (own image only)
  int fs0 = 0, fs1 = 0;       // features
  int sbin = 0;
  float scale = 0.f;          // scales[] entry
  int feat_off = -1;          // float planes
  int feat16_off = -1;        // tensor-core planes, 2-byte units
  int feat16lo_off = -1;      // BF16 remainder planes (root levels, BF16 mode), 2-byte units
  int hist_off = -1;
};

// a model's distance transforms in strips of one size (tuned on the plan's first frame, tune_dt)
struct DtPlan {
  int elems = 0;
  std::vector<DtJob> jobs;
  DtBlocks blocks;
  DevBuf d_jobs, d_chunks, d_strips, d_work;
};

struct ModelPlan {
  geye_model *model = nullptr;
  int LEN = 0;                          // levels this model uses
  std::vector<DtJob> dt_jobs;
  int dt_max_d0 = 0, dt_max_d1 = 0;
  std::vector<ScoreJob> score_jobs;
  int score_max_r = 0;
  int cap = 0;                          // max detections (sum of root map sizes)
  // device copies
  DevBuf d_score_jobs, d_counts;
  std::unique_ptr<DtPlan> dt;
  bool dt_tuned = false;
  float dt_ms[3] = {0, 0, 0};           // the timed launch per kDtElemsChoices entry
  DevBuf d_score_blocks;                // score / box blocks of every map (score_block_list)
  int score_nblocks = 0;
  // per-(level, comp) and per-(L, part) map offsets for stage readback
  std::vector<int> root_map_off, root_r0, root_r1;     // [level*NoC + c], -1 if none
  std::vector<int> part_map_off, part_d0, part_d1;     // [L*NoP + p]
  std::vector<int> skipped;                            // per level
  double conv_flops = 0, conv_bytes = 0, dt_bytes = 0, score_bytes = 0;
  // A_SCORE lookups: [job][image column] score-map column base, [job][image row] score row
  DevBuf d_as_col, d_as_row;
};

// One row of the tensor-core convolution's filter bank (conv_tc.cu): filter
// `filt` of model `mi` (its roots, then its parts), from filter row y0 and
// column x0 on, or the BF16 remainder of those weights; mi < 0: a padding row.
struct BankRowSpec {
  int mi = -1, filt = 0, y0 = 0, x0 = 0, lo = 0;
  float scale = 1.f;   // FP8: the filter's power-of-two scale
};

// The tensor-core convolution of all of a plan's models (conv_tc.cu): bank
// rows, one job per feature level, the epilogue's column tables, the root sums.
struct TcPlan {
  int planes = 0;                       // 4: BF16 planes, 2: e4m3
  int grid_b0 = 0, grid_b1 = 0;         // the bank's tap grid
  int rows = 0, rows_p16 = 0, rows_r16 = 0;
  std::vector<BankRowSpec> bank_rows;
  std::vector<TcJob> jobs;
  std::vector<TcCol> cols;
  std::vector<RootSumJob> sums;
  int sum_max_r = 0;
  DevBuf d_bank, d_jobs, d_chunks, d_cols, d_sums;
  int n_chunks = 0, stages = 0, tps = 1;   // bank stages; taps a stage (0: a filter column, -1: a phase)
  size_t smem = 0;
  int shape = -1;                       // tile-shape candidate the autotuner chose
  float tuned_ms = 0.f;                 // its measured time per launch
  // the persistent form (shape == the candidate after the tile shapes): units, and per CTA
  // its units, bank region and slab buffer bytes
  DevBuf d_units, d_ranges;
  int tcp_ctas = 0;
  uint32_t tcp_colbuf = 0;
};

struct Plan {
  // distinct for every plan a process builds (a rebuilt plan never reuses one)
  const unsigned long long serial = next_plan_serial();
  static unsigned long long next_plan_serial() {
    static std::atomic<unsigned long long> n{0};
    return ++n;
  }
  int width = 0, height = 0;           // frame size (0 when built from features)
  int interval = 0, sbin = 0, LEN = 0;
  bool from_features = false;
  std::vector<LevelInfo> lv;
  // resize phases: each phase is two passes (vertical then horizontal)
  std::vector<std::vector<ResizeJob>> rjobs;
  std::vector<int> r_max_blocks;       // per phase: the largest job's
  std::vector<DevBuf> d_rjobs;
  DevBuf d_tap_start, d_tap_si, d_tap_alpha;
  std::vector<HogJob> hog_jobs;
  DevBuf d_hog_jobs;
  DevBuf d_hog_vote_blocks;             // vote kernel blocks of every level (hog_vote_blocks)
  int hog_vote_nblocks = 0;
  int hog_max_b0 = 0, hog_max_b1 = 0;
  std::vector<HogPixJob> pix_jobs;   // one per image
  DevBuf d_pix_jobs;
  int pix_max_xe = 0;
  std::vector<std::unique_ptr<ModelPlan>> models;
  TcPlan tc;                             // BF16 / FP8 modes
  // FP32 mode: the filter groups of every model and level, one launch
  std::vector<ConvJob> conv_jobs;
  ConvBank conv_bank;
  DevBuf d_conv_jobs, d_conv_blocks, d_conv_bank;
  int conv_nblocks = 0;
  size_t conv_smem = 0;
  // memory
  size_t arena_words = 0, arena16_elems = 0;
  DevBuf arena, arena16;
  DevBuf d_bgr;                          // frame upload buffer
  DevBuf d_nms_f, d_nms_i, d_small, d_ascore, d_result;
  int max_cap = 0;
  // algorithmic bytes per stage (for roofline reporting)
  double bytes_resize = 0, bytes_hog = 0;
  // last-run results (host)
  std::vector<int> last_D, last_K;
  // the frame after its ingest, captured as CUDA graphs keyed by threshold, overlap and timing
  struct FrameGraph {
    cudaGraphExec_t exec = nullptr;
    int kernels = 0;
  };
  std::map<std::string, FrameGraph> graphs;
  void *h_res = nullptr;                // pinned result block (kHostRes)
  void *h_bgr = nullptr;                // pinned copy of a submitted frame (where its upload is not waited for)
  cudaEvent_t ev_done = nullptr;        // asynchronous submission (serve.cu): the frame's completion
  // park_pending: whether the pending frame's results are there, its counts (pinned) and records
  bool parked = false;
  void *h_parked = nullptr;
  DevBuf d_parked;
  ~Plan() {
    for (auto &g : graphs)
      if (g.second.exec) cudaGraphExecDestroy(g.second.exec);
    if (h_res) cudaFreeHost(h_res);
    if (h_bgr) cudaFreeHost(h_bgr);
    if (h_parked) cudaFreeHost(h_parked);
    if (ev_done) cudaEventDestroy(ev_done);
  }
};

}  // namespace geye

struct geye_ctx {
  int device = 0;
  cudaStream_t stream = nullptr;
  bool own_stream = false;
  // A_SCORE runs beside NMS on this stream (forked after the score stage,
  // joined before the frame ends)
  cudaStream_t side = nullptr;
  // captures the body of the frame graph's conditional node (NMS in the quicksort's order)
  cudaStream_t aux = nullptr;
  cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
  geye_conv_mode conv_mode = GEYE_CONV_FP32;
  std::map<std::string, std::unique_ptr<geye::Plan>> plans;
  int next_model_id = 1;
  // timing
  bool timing = false;
  cudaEvent_t ev[GEYE_N_STAGES + 1] = {};
  float stage_ms[GEYE_N_STAGES] = {};
  double stage_bytes[GEYE_N_STAGES] = {};
  double conv_flops = 0;
  int launches = 0;
  bool use_graphs = true;   // replay the frame as a CUDA graph (GEYE_NO_GRAPHS=1 at creation: plain launches)
  int nms_order = geye::kNmsOrderKey;   // geye_ctx_set_nms_order
  // the frame graph runs the NMS in the quicksort's order of all boxes as an if node (a lone
  // frame skips its launches when no model needs it); batch
  // lanes launch it plainly (its kernels return at once there), which measured
  // faster with frames of other contexts in flight
  bool nms_if_node = true;
  bool front_external = false;   // a batch's front end ran ingest, resize and HOG of the frame already
  bool capturing = false;
  // fault injection (host side)
  std::string inject_op;
  int inject_countdown = 0;
  // fallback counters etc. (device)
  geye::DevBuf d_diag;
  geye::ScratchArena scratch;   // stage calls
  // last device-resident run
  geye::Plan *last_plan = nullptr;
  // frame submitted with geye_detect_submit and not collected yet
  geye::Plan *pending = nullptr;
  // live models (detached when the context goes away first)
  std::set<geye_model *> models;
};
