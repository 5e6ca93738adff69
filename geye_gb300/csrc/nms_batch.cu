// nms_batch.cu -- NMS of the pipeline's detections, every model of a frame at once.
//
// Same kept set as nms.cu (CAR_TRACKING/nms.cpp:70-217): the reference's Hoare
// quicksort order for equal scores, greedy suppression by intersection over
// the smaller area or containment, and a box that is alone when its turn comes
// never emitted.
//
//  1. The order: score order from the radix sort (nms_radix.cu), checked for
//     the cases where the quicksort's order among equal scores could change
//     the kept set.  Where a batch's decisions depend on it, the cluster puts the batch's
//     members of those runs in the quicksort's order (nms_quick.h) and decides the batch again.  What a batch cannot settle
//     (a run longer than a batch, the last pick of all tied with another, NaN, ties without end)
//     starts the walk again with every box in the quicksort's order.
//  2. k_nms_greedy, a cluster of kCluster blocks per model, walks the boxes in
//     that order, a chunk at a time:
//       - the cluster tests the chunk's boxes against the picks so far that can
//         suppress them (found by image cell).  Which of several does is of no
//         account, but for the last pick of all (step 3): it counts only for
//         boxes that no earlier one removed;
//       - rounds over the boxes left alive: every block alike takes the first
//         kBatch of them; the blocks share the tests of every pair of those, a
//         bit per pair, written into the first block's shared memory; that
//         block walks them in order, a bit of each in registers: the first
//         undecided one is picked and its row of suppressed members struck out
//         -- the sequential loop's decisions, since every box before the batch
//         is resolved.  Boxes of the chunk still alive are tested against the
//         new picks.
//     A chunk is sized so that about a batch of it survives: a few hundred boxes
//     at the head of the order, most of them at its end.
//     Where there are more than kWhole boxes it stops after the first kPrefix:
//     by then nearly every pick is made.  k_nms_rest tests the others over the
//     whole grid, and a second cluster launch takes the few survivors.
//  3. The first block drops the final pick if it suppressed nothing (the
//     reference's `while (cnum > 0)` with cnum = NUM-1 never takes a box that is
//     alone at its turn) and writes the results in input order.
//
// What bounds it is latency: rounds depend on one another, and so do the steps
// of a round (L2 reads of a thousand cycles, cluster barriers of 1200, the walk's
// 200 a pick).  Tried before, 640x480 car+person, NMS stage: 256 members a round
// resolved by one block, a pass of all alive boxes over the grid, 285 us; 512
// members, the pair tests by 32 blocks handing over by a ticket, 155 us; one
// cluster kernel for all rounds with a pass of all alive boxes each, 147 us;
// this form 160 us (320x240 car: 135 -> 70, 1280x720: 575 -> 403, 1280x720 trained-like:
// 280 -> 170).
// With the whole quicksort over the grid and a second walk wherever a model needed its order (75 launches, in a batch's
// lanes on every frame) 1920x1080 took 1830 us when it did, and a batch of eight mixed frames 3630 us; with the few
// members put in order inside the walk 1010 us, the batch 3140 us.
#include <algorithm>

#include "nms_common.h"
#include "nms_quick.h"
#include "rects.h"

namespace geye {

constexpr int kBatch = kNmsBatch;
constexpr int kBW = kBatch / 32;     // words of a suppression row
constexpr int kPickGroup = 256;      // picks per table of a pass
constexpr int kGW = kPickGroup / 32;
// Boxes that the first launch takes where there are more than kWhole: its first three chunks, after which nearly every pick
// is made; the others meet the picks on all of the chip instead of the cluster's 16 SMs, for two launches more.
// 1013x571 (140 000 boxes) NMS stage 264 us in one launch, 236 so; 1280x720 (240 000) 397 with a prefix of 65 536, 341 so
// and 364 with 4608; 640x480 (66 000) 160 either way.
constexpr int kPrefix = 512 + 4096 + 32768, kWhole = 70000;
constexpr int kWinWords = 4 * kResNT;   // words of a chunk's window
constexpr int kMaxChunk = 32 * (kWinWords - 2);   // with the run at its end
constexpr int kChunkCap = 60000;
// Where a batch's tied members are put in order, and where all boxes are, the walk then starting again (1920x1080,
// 600 000 boxes: 250 us the first time and 150 the next ones, against 1000).  A textured frame ties a few members of one or two
// runs, far down the order; kSettleHead members or more tied in the first 32nd of the order belong to a frame with
// large areas of one colour, and more ties follow (a frame of one colour: 3.5 ms with this line, 4.2 without).
constexpr int kSettle = 4, kSettleHead = 8, kSettleRun = 4096;
static_assert(kBatch == kResNT, "a thread per member");

// cell of a coordinate on one axis of the pick tables (monotone; NaN to cell 0); inv: cells per pixel (.x: y axis, .y: x axis)
__device__ __forceinline__ int nms_cell(float v, float inv) {
  return (int)fminf(fmaxf(v * inv, 0.0f), (float)(kNmsCells - 1));
}

struct PickTable {   // see pick_table
  unsigned covers[2][kGW][kNmsCells];
  unsigned in_span[2][kNmsLevels][kGW][kNmsCells];
};

struct GreedySmem {
  union {
    unsigned adj[kBatch * kBW];   // the members' rows (the first block's)
    PickTable table;
    int idx[kBatch * kBW];        // at the end: the kept boxes
    QuickSmem quick;              // while boxes are put in the quicksort's order
  };
  float4 pk[kBatch];              // the tested picks' boxes and areas
  float pka[kBatch];
  float my[5][kBatch];            // members' boxes
  int item[kBatch + 1], pos[kBatch + 1];   // members' items and sorted positions
  unsigned key[kBatch + 1];       // key order: the candidates' keys
  int pick_mem[kBatch];
  int pick_any[kBatch];           // the pick removed a member alive at its turn
  int wtot[kResWarps];
  int total[kCluster];            // (the first block's) the blocks' survivors
  unsigned tied[kBW];             // the batch's runs to be put in order, by their first member
  SortRuns runs;
  int nb, np, tot;                // np = -1: the batch depends on the order inside R.runs
  int n, c0, c1, chunk, npicks, tested, left, batches, settled;   // the walk's place (walk_boxes)
  int cut, need;                  // a run longer than a batch; a pick that removes a member of its own run
};

// exclusive block scan of c (kResNT threads); *tot gets the sum
__device__ __forceinline__ int block_excl_scan(int c, int *tot, int *wtot) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int inc = c;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += t;
  }
  __syncthreads();   // wtot free
  if (lane == 31) wtot[warp] = inc;
  __syncthreads();
  int before = inc - c, t = 0;
#pragma unroll
  for (int k = 0; k < kResWarps; k++) {
    const int v = wtot[k];
    if (k < warp) before += v;
    t += v;
  }
  *tot = t;
  return before;
}

// ---------------------------------------------------------------------------
// tests against picks
// ---------------------------------------------------------------------------
// Which picks can suppress a box.  With an overlap of a half or more, a pick and a box where one suppresses the other
// share more than half of the smaller one's area, so more than half of its width and of its height, so its centre:
// the pick covers the box's centre, or the box the pick's.  (Boxes of the pipeline are proper, so containment is an
// overlap; two pixels of slack cover the + 1 of the reference's widths and every rounding.)  With a smaller
// overlap they only share a cell on each axis.
//
// The table of np <= kPickGroup picks by cell: `covers` lists a pick on every cell of its widened span, `in_span` what
// a box's span is looked up in (half: the picks' centres; else their spans again) with the unions over 2^l cells,
// so that a span is the union of two entries.  A warp per axis and word of picks, two cells a lane.
__device__ __forceinline__ void pick_table(PickTable &T, const float4 *pk, int np, float2 cell_inv, bool half) {
  const int lane = threadIdx.x & 31;
  static_assert(kNmsCells == 64, "two cells a lane");
  for (int e = threadIdx.x >> 5; e < 2 * ((np + 31) >> 5); e += kResWarps) {
    const int a = e & 1, k = e >> 1;   // a = 0: y (my[0], my[2]); 1: x (my[1], my[3])
    int c0 = kNmsCells, c1 = -1, d0 = kNmsCells, d1 = -1;
    if (32 * k + lane < np) {
      const float4 p = pk[32 * k + lane];
      const float lo = (a ? fminf(p.y, p.w) : fminf(p.x, p.z)) - 2.0f, hi = (a ? fmaxf(p.y, p.w) : fmaxf(p.x, p.z)) + 2.0f;
      const float inv = a ? cell_inv.y : cell_inv.x;
      c0 = nms_cell(lo, inv);
      c1 = nms_cell(hi, inv);
      const float mid = 0.5f * (lo + hi);
      d0 = half ? nms_cell(mid - 2.0f, inv) : c0;
      d1 = half ? nms_cell(mid + 2.0f, inv) : c1;
    }
    unsigned u0 = 0u, u1 = 0u, v0 = 0u, v1 = 0u;   // cells lane and lane + 32
#pragma unroll 8
    for (int b = 0; b < 32; b++) {
      const int lo = __shfl_sync(0xffffffffu, c0, b), hi = __shfl_sync(0xffffffffu, c1, b);
      const int l2 = __shfl_sync(0xffffffffu, d0, b), h2 = __shfl_sync(0xffffffffu, d1, b);
      u0 |= (unsigned)(lo <= lane && lane <= hi) << b;
      u1 |= (unsigned)(lo <= lane + 32 && lane + 32 <= hi) << b;
      v0 |= (unsigned)(l2 <= lane && lane <= h2) << b;
      v1 |= (unsigned)(l2 <= lane + 32 && lane + 32 <= h2) << b;
    }
    T.covers[a][k][lane] = u0;
    T.covers[a][k][lane + 32] = u1;
#pragma unroll
    for (int l = 0; l < kNmsLevels; l++) {
      if (l > 0) {   // the cell 2^(l-1) further, the last one at most
        const int d = 1 << (l - 1);
        const unsigned s0 = __shfl_sync(0xffffffffu, v0, (lane + d) & 31), s1 = __shfl_sync(0xffffffffu, v1, (lane + d) & 31);
        const unsigned top = __shfl_sync(0xffffffffu, v1, 31);
        v0 |= lane + d < 32 ? s0 : s1;
        v1 |= lane + d < 32 ? s1 : top;
      }
      T.in_span[a][l][k][lane] = v0;
      T.in_span[a][l][k][lane + 32] = v1;
    }
  }
}

// One of the table's picks that suppresses a box, or -1; pick `last` only where no other one does.
__device__ __forceinline__ int suppressor(const PickTable &T, const float4 *pk, const float *pka, int np, int last,
                                          float e0, float e1, float e2, float e3, float e4, float overlap,
                                          float2 cell_inv, bool half) {
  const int nwm = (np + 31) >> 5;
  const int cy0 = nms_cell(fminf(e0, e2) - 2.0f, cell_inv.x), cy1 = nms_cell(fmaxf(e0, e2) + 2.0f, cell_inv.x);
  const int cx0 = nms_cell(fminf(e1, e3) - 2.0f, cell_inv.y), cx1 = nms_cell(fmaxf(e1, e3) + 2.0f, cell_inv.y);
  const int ly = 31 - __clz(cy1 - cy0 + 1), lx = 31 - __clz(cx1 - cx0 + 1);
  const unsigned *y0p = &T.in_span[0][ly][0][cy0], *y1p = &T.in_span[0][ly][0][cy1 - (1 << ly) + 1];
  const unsigned *x0p = &T.in_span[1][lx][0][cx0], *x1p = &T.in_span[1][lx][0][cx1 - (1 << lx) + 1];
  const unsigned *cy = &T.covers[0][0][nms_cell(0.5f * (e0 + e2), cell_inv.x)];
  const unsigned *cx = &T.covers[1][0][nms_cell(0.5f * (e1 + e3), cell_inv.y)];
  bool by_last = false;
  for (int k = 0; k < nwm; k++) {
    const int o = k * kNmsCells;
    unsigned cand = (y0p[o] | y1p[o]) & (x0p[o] | x1p[o]);
    if (half) cand |= cy[o] & cx[o];
    while (cand) {
      const int t = (k << 5) + __ffs(cand) - 1;
      cand &= cand - 1;
      const float4 p = pk[t];
      if (supp(p.x, p.y, p.z, p.w, pka[t], e0, e1, e2, e3, e4, overlap)) {
        if (t != last) return t;
        by_last = true;
      }
    }
  }
  return by_last ? last : -1;
}

// Words of the item bitmap [w0, w1], a run of them per warp (gw of nw), against the table's np picks (pick numbers from
// pick_base on), a lane per box, four words' boxes in flight.  first: the alive items are [c0, c1) (nothing is read
// from the bitmap), else the bitmap's.  last: the newest pick's place in the table (its flag is raised when it removes a
// box: only the last of all picks' is read, and any other's would be raised by thousands).  list: the items' sorted positions (null: the item itself).
__device__ __forceinline__ void test_words(const Slots &S, const PickTable &T, const float4 *pk, const float *pka, int np,
                                           int pick_base, int last, const int *list, int w0, int w1, bool first, int c0,
                                           int c1, float overlap, float2 cell_inv, int gw, int nw) {
  const int lane = threadIdx.x & 31;
  const bool half = overlap >= 0.5f;
  const int run = max(1, min(32, (w1 - w0 + nw) / nw));
  for (int wb = w0 + gw * run; wb <= w1; wb += nw * run) {
    const int w = wb + lane;
    unsigned mine = 0u;
    if (lane < run && w <= w1) {
      if (first) {   // items c0 .. c1 of word w
        const int lo = c0 - 32 * w, hi = c1 - 32 * w;
        mine = (lo <= 0 ? ~0u : ~0u << lo) & (hi >= 32 ? ~0u : (1u << hi) - 1u);
      } else {
        mine = __ldcg(&S.bits[w]);
      }
    }
    unsigned some = __ballot_sync(0xffffffffu, mine != 0u), left = mine;
    while (some) {
      int wi[4];
      unsigned alive[4];
      float e[4][5];
#pragma unroll
      for (int u = 0; u < 4; u++) {
        wi[u] = some ? __ffs(some) - 1 : -1;
        some &= some - 1;   // (0 stays 0)
        alive[u] = __shfl_sync(0xffffffffu, mine, wi[u] & 31);
        if (wi[u] >= 0 && ((alive[u] >> lane) & 1u)) {
          const int q = ((wb + wi[u]) << 5) + lane, r = list ? list[q] : q;
          e[u][0] = S.y1[r]; e[u][1] = S.x1[r]; e[u][2] = S.y2[r]; e[u][3] = S.x2[r]; e[u][4] = S.ar[r];
        }
      }
#pragma unroll
      for (int u = 0; u < 4; u++) {
        if (wi[u] < 0) break;
        int k = -1;
        if ((alive[u] >> lane) & 1u)
          k = suppressor(T, pk, pka, np, last, e[u][0], e[u][1], e[u][2], e[u][3], e[u][4], overlap,
                         cell_inv, half);
        const unsigned gone = __ballot_sync(0xffffffffu, k >= 0);
        if (k >= 0 && k == last) S.flag[pick_base + k] = 1;
        if (lane == wi[u]) left &= ~gone;
      }
    }
    if (lane < run && w <= w1 && (first || left != mine)) S.bits[w] = left;
  }
}

// items [c0, c1) (bitmap words w0 .. w1) against the picks [p0, p1), by the warps gw of nw; first: all of
// them are alive before it (else those in the bitmap)
__device__ __forceinline__ void test_chunk(const Slots &S, PickTable &T, float4 *pk, float *pka, int p0, int p1,
                                           const int *list, int w0, int w1, int c0, int c1, float overlap,
                                           float2 cell_inv, int gw, int nw, bool first = true) {
  int k0 = p0;
  do {
    const int np = min(kPickGroup, p1 - k0);
    __syncthreads();   // the last table is free
    if (threadIdx.x < np) {
      pk[threadIdx.x] = __ldcg(&S.pb[k0 + threadIdx.x]);
      pka[threadIdx.x] = __ldcg(&S.pa[k0 + threadIdx.x]);
    }
    __syncthreads();
    if (np > 0) pick_table(T, pk, np, cell_inv, overlap >= 0.5f);
    __syncthreads();
    test_words(S, T, pk, pka, np, k0, p1 - 1 - k0, list, w0, w1, first && k0 == p0, c0, c1, overlap, cell_inv, gw, nw);
    k0 += kPickGroup;
  } while (k0 < p1);
}

// ---------------------------------------------------------------------------
// rounds over a chunk's survivors
// ---------------------------------------------------------------------------
// The batch: the first kBatch alive items of words [w0, w1] with their boxes, by the whole block (R.nb of them; R.tot:
// the alive items).  The bitmap is read past L1: other blocks of the cluster have changed it.
// ordered: the positions are the quicksort's.  Else a run of equal scores never straddles two batches (the batch ends
// before a run that the next alive box continues); a run longer than a batch raises R.cut.
__device__ __forceinline__ void select_members(const Slots &S, GreedySmem &R, const int *list, int w0, int w1, bool ordered) {
  constexpr int want = kBatch + 1;                     // one more, to see the run at the boundary
  const int per = (w1 - w0 + kResNT) / kResNT;         // words per thread: at most four
  unsigned word[4];
  int cnt = 0;
#pragma unroll
  for (int u = 0; u < 4; u++) {
    const int w = w0 + threadIdx.x * per + u;
    word[u] = u < per && w <= w1 ? __ldcg(&S.bits[w]) : 0u;
    cnt += __popc(word[u]);
  }
  int tot;
  int rank = block_excl_scan(cnt, &tot, R.wtot);
#pragma unroll
  for (int u = 0; u < 4; u++)
    for (unsigned rem = word[u]; rem && rank < want; rem &= rem - 1)
      R.item[rank++] = ((w0 + threadIdx.x * per + u) << 5) + __ffs(rem) - 1;
  __syncthreads();
  for (int k = threadIdx.x; k < min(want, tot); k += kResNT) {
    const int r = list ? list[R.item[k]] : R.item[k];
    R.pos[k] = r;
    R.key[k] = S.key[r];
    if (k < kBatch) {
      R.my[0][k] = S.y1[r];
      R.my[1][k] = S.x1[r];
      R.my[2][k] = S.y2[r];
      R.my[3][k] = S.x2[r];
      R.my[4][k] = S.ar[r];
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int nb = min(kBatch, tot);
    R.cut = 0;
    R.runs.n = 0;
    if (!ordered && tot > kBatch && R.key[kBatch - 1] == R.key[kBatch]) {   // end before the run that goes on
      const unsigned kb = R.key[kBatch];
      int lo = 0, hi = kBatch;   // first candidate with key kb (keys ascend)
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (R.key[mid] < kb) lo = mid + 1;
        else hi = mid;
      }
      nb = lo;
      if (nb == 0) {   // a run longer than a batch
        R.cut = 1;
        nb = kBatch;
      }
    }
    R.nb = nb;
    R.tot = tot;
  }
  __syncthreads();
}

// Row i of the pairs (bit j of word w: member j = 32 w + lane > i is suppressed by member i) by one warp
__device__ __forceinline__ void pair_row(const GreedySmem &R, int i, float overlap, unsigned *row) {
  const int lane = threadIdx.x & 31, nb = R.nb;
  const float a0 = R.my[0][i], a1 = R.my[1][i], a2 = R.my[2][i], a3 = R.my[3][i], a4 = R.my[4][i];
  unsigned mine = 0u;
#pragma unroll 4
  for (int w = i >> 5; 32 * w < nb; w++) {
    const int j = 32 * w + lane;
    const bool s = j > i && j < nb &&
                   supp(a0, a1, a2, a3, a4, R.my[0][j], R.my[1][j], R.my[2][j], R.my[3][j], R.my[4][j], overlap);
    const unsigned bal = __ballot_sync(0xffffffffu, s);
    if (lane == w) mine = bal;
  }
  if (lane < kBW) row[lane] = mine;
}

// First of the places [lo, hi) with ascending keys that is not below k (kAbove: that is above k), else hi; by a warp
template <bool kAbove, class F>
__device__ __forceinline__ int key_bound(F key, int lo, int hi, unsigned k) {
  const int lane = threadIdx.x & 31;
  while (lo < hi) {
    const long long len = hi - lo;
    const unsigned v = key(lo + (int)(len * lane / 32));
    const int c = __popc(__ballot_sync(0xffffffffu, kAbove ? v <= k : v < k));   // the first c probes are before it
    if (c < 32) hi = lo + (int)(len * c / 32);
    if (c > 0) lo = lo + (int)(len * (c - 1) / 32) + 1;
  }
  return lo;
}

// Whether a sorted position is inside one of the runs
__device__ __forceinline__ bool in_runs(const SortRuns &runs, int pos) {
  bool in = false;
  for (int q = 0; q < runs.n; q++) in |= pos >= runs.r[q].x && pos <= runs.r[q].y;
  return in;
}

// The batch's runs in R.tied (a bit for the first member of each) into R.runs (their places in the sorted
// order); what is more than kRuns goes into the last, which then holds other runs' places too
__device__ __forceinline__ void tied_runs(GreedySmem &R, const Slots &S, int D) {
  if (threadIdx.x >= 32) return;
  auto key = [&](int q) { return S.key[q]; };
  int n = R.runs.n;
  for (int w = 0; w < kBW; w++)
    for (unsigned rem = R.tied[w]; rem; rem &= rem - 1) {
      const unsigned k = R.key[32 * w + __ffs(rem) - 1];
      const int lo = key_bound<false>(key, 0, D, k), hi = key_bound<true>(key, 0, D, k) - 1;
      if (threadIdx.x == 0) {
        int2 &last = R.runs.r[kRuns - 1];
        if (n < kRuns) R.runs.r[n] = make_int2(lo, hi);
        else last = make_int2(min(last.x, lo), max(last.y, hi));
      }
      n = min(n + 1, kRuns);
    }
  if (threadIdx.x == 0) R.runs.n = n;
}

// The members of the first block's R.tied and R.runs in the quicksort's order, in every block; false where the order of all boxes
// is to be taken instead
__device__ __noinline__ bool settle_members(GreedySmem &R, int *si, float *sf, int m, int cap, int *err) {
  cg::cluster_group cluster = cg::this_cluster();
  const Slots S = slots(si, sf, m, cap);
  const int D = S.st->D;
  const GreedySmem *R0 = cluster.map_shared_rank(&R, 0);
  if (cluster.block_rank() == 0) tied_runs(R, S, D);
  cluster.sync();
  if (threadIdx.x < sizeof(SortRuns) / sizeof(int))
    reinterpret_cast<int *>(&R.runs)[threadIdx.x] = reinterpret_cast<const int *>(&R0->runs)[threadIdx.x];
  if (threadIdx.x == 0) R.settled++;
  cluster.sync();   // every block has its copy: the first block's may be overwritten (split_boxes)
  int places = 0;
  for (int q = 0; q < R.runs.n; q++) places += R.runs.r[q].y - R.runs.r[q].x + 1;
  const int tied = __syncthreads_count((int)threadIdx.x < R.nb && in_runs(R.runs, R.pos[threadIdx.x]));
  if (R.settled > kSettle || places > max(kSettleRun, D / 4) || (tied >= kSettleHead && R.runs.r[0].x < D / 32)) return false;
  quick_sort(R.quick, R.runs, S, false, err);
  const int k = threadIdx.x, nb = R.nb;
  int *rk = R.pick_mem;   // a member's place: a run's members share the run's, the others keep theirs
  static_assert(kBatch == kResNT, "a thread per member");
  int pos = 0, item = 0, at = 0;
  float box[5];
  if (k < nb) {
    pos = R.pos[k];
    item = R.item[k];
    for (int c = 0; c < 5; c++) box[c] = R.my[c][k];
    rk[k] = in_runs(R.runs, pos) ? __ldcg(S.place + S.ord[pos]) : pos;
  }
  __syncthreads();
  if (k < nb)
    for (int j = 0; j < nb; j++) at += rk[j] < rk[k];
  if (k < nb) {
    R.pos[at] = pos;
    R.item[at] = item;
    for (int c = 0; c < 5; c++) R.my[c][at] = box[c];
  }
  __syncthreads();
  return true;
}

// The quicksort of all boxes, as far as the cluster takes it
__device__ __noinline__ void split_boxes(GreedySmem &R, int *si, float *sf, int m, int cap, int *err) {
  const Slots S = slots(si, sf, m, cap);
  const int D = S.st->D;
  __syncthreads();
  if (threadIdx.x == 0) {
    R.runs.n = 1;
    R.runs.r[0] = make_int2(0, D - 1);
  }
  __syncthreads();
  quick_sort(R.quick, R.runs, S, true, err);
}

// The boxes in the quicksort's order, by the cluster
__device__ __noinline__ void gather_boxes(int *si, float *sf, int m, int cap) {
  cg::cluster_group cluster = cg::this_cluster();
  const Slots S = slots(si, sf, m, cap);
  const int D = S.st->D;
#pragma unroll 4
  for (int r = (int)cluster.block_rank() * kResNT + threadIdx.x; r < D; r += (int)cluster.num_blocks() * kResNT) {
    const int i = S.qo[r];
    const float4 b = S.box[i];
    S.ord[r] = i;
    S.y1[r] = b.x; S.x1[r] = b.y; S.y2[r] = b.z; S.x2[r] = b.w;
    S.ar[r] = (b.w - b.y + 1.0) * (b.z - b.x + 1.0);   // nms.cpp's area expression
  }
  cluster.sync();
}

// The batch's decisions from its rows (R.adj), by the first block: R.np picks in R.pick_mem, appended to S.picks
// and S.pb, the members cleared from the bitmap.  check: where the order inside a run of equal scores
// matters (a pick that removes a member of its own run, other than the runs in R.runs, which are in order), nothing of
// that but R.np = -1 and the run in R.tied.
__device__ __forceinline__ void decide_members(const Slots &S, GreedySmem &R, int base, bool check) {
  const int nb = R.nb, lane = threadIdx.x & 31;
  if (threadIdx.x < 32) {
    // the undecided members in registers, every lane alike (one wide broadcast read a pick; warp votes in this
    // loop measured 640 cycles a pick, this 170)
    unsigned und[kBW];
#pragma unroll
    for (int w = 0; w < kBW; w++) und[w] = nb >= 32 * w + 32 ? ~0u : nb > 32 * w ? (1u << (nb - 32 * w)) - 1u : 0u;
    int np = 0;
#pragma unroll
    for (int w = 0; w < kBW; w++)
      while (und[w]) {   // its first member: nobody before it suppresses it
        const int i = 32 * w + __ffs(und[w]) - 1;
        const uint4 *row = reinterpret_cast<const uint4 *>(R.adj + i * kBW);
        unsigned gone = 0u;
#pragma unroll
        for (int q = w / 4; q < kBW / 4; q++) {
          const uint4 v = row[q];
          gone |= (und[4 * q] & v.x) | (und[4 * q + 1] & v.y) | (und[4 * q + 2] & v.z) | (und[4 * q + 3] & v.w);
          und[4 * q] &= ~v.x; und[4 * q + 1] &= ~v.y; und[4 * q + 2] &= ~v.z; und[4 * q + 3] &= ~v.w;
        }
        und[w] &= und[w] - 1u;
        R.pick_mem[np] = i;
        R.pick_any[np++] = gone != 0u;
      }
    if (lane == 0) {
      R.np = np;
      R.need = 0;
    }
    if (lane < kBW) R.tied[lane] = 0u;
  }
  __syncthreads();
  const int np = R.np;
  if (check) {
    for (int k = threadIdx.x; k < np; k += kResNT) {
      // members of the pick's own run that it removed: suppressed by it and by no pick before it
      const int i = R.pick_mem[k];
      if (in_runs(R.runs, R.pos[i])) continue;
      for (int j = i + 1; j < nb && R.key[j] == R.key[i]; j++) {
        if (!((R.adj[i * kBW + (j >> 5)] >> (j & 31)) & 1u)) continue;
        bool alive = true;
        for (int q = 0; q < k && alive; q++) alive = !((R.adj[R.pick_mem[q] * kBW + (j >> 5)] >> (j & 31)) & 1u);
        if (!alive) continue;
        int first = i;
        while (first > 0 && R.key[first - 1] == R.key[i]) first--;
        atomicOr(&R.tied[first >> 5], 1u << (first & 31));
        R.need = 1;
        break;
      }
    }
    __syncthreads();
    if (R.need) {
      if (threadIdx.x == 0) R.np = -1;
      return;
    }
  }
  for (int k = threadIdx.x; k < np; k += kResNT) {
    const int i = R.pick_mem[k];
    S.picks[base + k] = R.pos[i];
    S.flag[base + k] = R.pick_any[k];
    S.pb[base + k] = make_float4(R.my[0][i], R.my[1][i], R.my[2][i], R.my[3][i]);
    S.pa[base + k] = R.my[4][i];
  }
  for (int k = threadIdx.x; k < nb; k += kResNT)   // every member is resolved
    atomicAnd(&S.bits[R.item[k] >> 5], ~(1u << (R.item[k] & 31)));
}

// ---------------------------------------------------------------------------
// final-pick rule, the kept boxes in input order (the model done)
// ---------------------------------------------------------------------------
// The kept boxes' input indices, by the first block: R.tot of them, in R.idx + kRankMax, or in S.Rpos where they are more
constexpr int kRankMax = 2 * kResNT;
__device__ __forceinline__ void rank_kept(const Slots &S, GreedySmem &R, int npk) {
  const int D = S.st->D;
  // (the flags are read past L1: other blocks of the cluster have set them)
  const int K = npk - ((npk > 0 && __ldcg(&S.flag[npk - 1]) == 0) ? 1 : 0);
  // the kept boxes' input indices (all distinct) in ascending order
  int *keep = S.Rpos;
  int *idx = R.idx;   // the round's buffers are free now
  if (K <= kRankMax) {   // ranked in shared memory
    for (int k = threadIdx.x; k < ((K + 3) & ~3); k += kResNT) idx[k] = k < K ? S.ord[__ldcg(&S.picks[k])] : 0x7fffffff;
    __syncthreads();
    keep = idx + kRankMax;
    for (int k = threadIdx.x; k < K; k += kResNT) {
      const int v = idx[k];
      int r = 0;
#pragma unroll 4
      for (int j = 0; j < K; j += 4) {
        const int4 u = *reinterpret_cast<const int4 *>(idx + j);
        r += (u.x < v) + (u.y < v) + (u.z < v) + (u.w < v);
      }
      keep[r] = v;
    }
  } else {   // many: marked by input index, then packed
    int *mark = S.Lpos;   // (the list of items is done with)
    for (int i = threadIdx.x; i < D; i += kResNT) mark[i] = 0;
    __syncthreads();
    for (int k = threadIdx.x; k < K; k += kResNT) mark[S.ord[__ldcg(&S.picks[k])]] = 1;
    __syncthreads();
    int written = 0;
    for (int base = 0; base < D; base += kResNT) {
      const int i = base + threadIdx.x;
      const int f = i < D && mark[i];
      int tot;
      const int r = block_excl_scan(f, &tot, R.wtot);
      if (f) keep[written + r] = i;
      written += tot;
    }
  }
  if (threadIdx.x == 0) R.tot = K;
}

// The results (get_new_rects) of the kept boxes, by the cluster, four threads a box: its parts' corners looked up anew,
// then a side each; on the device, and the first of them in the host's block
__device__ __forceinline__ void write_results(const Slots &S, GreedySmem &R, int m, int cap, const NmsResults &res) {
  cg::cluster_group cluster = cg::this_cluster();
  const GreedySmem *R0 = cluster.map_shared_rank(&R, 0);
  const NmsResults::Model &Q = res.m[m];
  const int K = R0->tot, np = Q.np, ML = 1 + 2 * (1 + np);
  int *out = res.out + (size_t)m * cap * 11, *host = res.host + 64 + (size_t)m * 11 * res.host_cap;
  static_assert(sizeof(R.idx) >= (2 * kRankMax + (kResNT / 4) * (1 + 2 * (1 + kMaxParts))) * sizeof(int) ||
                    sizeof(QuickSmem) >= (2 * kRankMax + (kResNT / 4) * (1 + 2 * (1 + kMaxParts))) * sizeof(int),
                "the ranks and a block's records");
  // [w, (x1, y1) of root and parts] of the thread's box, behind the ranks
  float *vec = reinterpret_cast<float *>(R.idx) + 2 * kRankMax + (threadIdx.x >> 2) * ML;
  const int step = (int)cluster.num_blocks() * kResNT, first = (int)cluster.block_rank() * kResNT;
  for (int e0 = first; e0 < 4 * K; e0 += step) {
    const int e = e0 + threadIdx.x, k = e >> 2, c = e & 3;
    const bool in = k < K;
    int comp = 0, more = 0;
    if (in) {
      const int box = K <= kRankMax ? R0->idx[kRankMax + k] : __ldcg(&S.Rpos[k]), ref = S.ref[box];
      const int2 blk = Q.blocks[ref / kScoreThreads];
      const ScoreJob &J = Q.jobs[blk.x];
      const int i = blk.y * kScoreThreads + ref % kScoreThreads, y = i % J.r0, x = i / J.r0;
      comp = J.comp;
      for (int p = c; p < np; p += 4) {
        const float2 q = part_corner(J, p, x, y, res.arena_i);
        vec[3 + 2 * p] = q.y;
        vec[4 + 2 * p] = q.x;
      }
      if (c == 0) {
        const float4 b = S.box[box];
        vec[0] = b.w - b.y;
        vec[1] = b.y;
        vec[2] = b.x;
      }
      // type, scale, score
      more = c == 0 ? comp : __float_as_int(c == 1 ? J.scale : S.score[box]);
    }
    __syncwarp();
    if (in) {
      const float *w = Q.coef + ((size_t)comp * 4 + c) * ML;
      float sum = 0;
#pragma unroll 8
      for (int q = 0; q < ML; q++) sum += vec[q] * w[q];
      const int v = rect_bound(sum, res.img_w, res.img_h, c), r = (int)((float)v / Q.ratio);
      auto put = [&](int *o, size_t stride) {
        o[e] = v;
        o[4 * stride + e] = r;
        if (c < 3) o[(8 + c) * stride + k] = more;
      };
      put(out, cap);
      if (k < res.host_cap) put(host, res.host_cap);
    }
    __syncwarp();
  }
}

// The first item at or after c1 whose score differs from the one before it, at most hi (every warp alike)
__device__ __forceinline__ int run_end(const Slots &S, const int *list, int c1, int hi) {
  auto key = [&](int q) { return S.key[list ? list[q] : q]; };
  const unsigned k = key(c1 - 1);
  const int q = c1 + (threadIdx.x & 31);
  const unsigned other = __ballot_sync(0xffffffffu, q >= hi || key(q) != k);
  return other ? c1 + __ffs(other) - 1 : key_bound<true>(key, c1 + 32, hi, k);
}

// The walk over the items [R.c0, R.n), with R.npicks picks of which R.tested have been tested against all items (list:
// the items' sorted positions).  kTied: a batch's decisions depend on the order inside runs of equal scores (R.tied of the
// first block); again with resume kBatchReady once its members are in order.  kCut: a run longer than a batch or a chunk.
// Every block alike; its place rests in shared memory between the calls.
enum WalkEnd { kDone, kTied, kCut };
enum WalkResume { kAnew, kChunkTested, kBatchReady };   // in a chunk that has been tested; with a batch that is selected
__device__ __forceinline__ WalkEnd walk_boxes(const Slots &S, GreedySmem &R, const int *list, float overlap, float2 cell_inv,
                                              bool ordered, WalkResume resume) {
  cg::cluster_group cluster = cg::this_cluster();
  GreedySmem *R0 = cluster.map_shared_rank(&R, 0);
  const int rank = (int)cluster.block_rank(), blocks = (int)cluster.num_blocks();
  const int gw = rank * kResWarps + (threadIdx.x >> 5), nw = blocks * kResWarps;
  const int n = R.n;
  int chunk = R.chunk, np = R.npicks, tested = R.tested, batches = R.batches, left = R.left;
  WalkEnd end = kDone;
  for (int c0 = R.c0; c0 < n;) {
    int c1 = resume != kAnew ? R.c1 : min(c0 + chunk, n);
    if (resume == kAnew && n - c1 < chunk / 8 && n - c0 <= kMaxChunk) c1 = n;   // (no round for a short rest: 4 us)
    if (resume == kAnew && !ordered && c1 < n) {   // not inside a run of equal scores
      const int lim = min(n, c0 + kMaxChunk);
      c1 = run_end(S, list, c1, lim);
      if (c1 == lim && c1 < n && run_end(S, list, c1, c1 + 1) > c1) return kCut;   // a run of that length would be cut
    }
    const int w0 = c0 >> 5, w1 = (c1 - 1) >> 5;
    if (resume == kAnew) {
      test_chunk(S, R.table, R.pk, R.pka, tested, np, list, w0, w1, c0, c1, overlap, cell_inv, gw, nw);
      cluster.sync();   // the bitmap is complete
    }
    for (bool first = resume == kAnew;; first = false) {
      if (resume != kBatchReady) select_members(S, R, list, w0, w1, ordered);
      resume = kAnew;
      if (first) left = R.tot;
      if (R.tot == 0) break;
      if (R.cut) {
        end = kCut;
        break;
      }
      for (int k = 0; k * nw < R.nb; k++) {   // rows g, then 2G - 1 - g, ...: long and short ones in turn
        const int i = k * nw + ((k & 1) ? nw - 1 - gw : gw);
        if (i < R.nb) pair_row(R, i, overlap, R0->adj + i * kBW);
      }
      cluster.sync();   // the rows are in the first block
      if (rank == 0) decide_members(S, R, np, !ordered);
      cluster.sync();   // the picks are in the first block and in S, the members cleared
      const int added = R0->np;
      if (added < 0) {
        end = kTied;
        break;
      }
      batches++;
      if (R.tot > R.nb) {   // the rest of the chunk against the new picks
        test_chunk(S, R.table, R.pk, R.pka, np, np + added, list, w0, w1, 0, 0, overlap, cell_inv, gw, nw, false);
        cluster.sync();
      }
      np += added;
      if (R.tot <= R.nb) break;
    }
    cluster.sync();   // (the first block's picks have been read)
    if (end != kDone) {
      if (threadIdx.x == 0) {
        R.c0 = c0;
        R.c1 = c1;
      }
      break;
    }
    // the head leaves about a tenth of what follows alive, and the picks thin every next stretch out further:
    // eight times the chunk leaves a batch or two (twice after one that left more)
    chunk = min((left > 2 * kBatch ? 2 : 8) * chunk, kChunkCap);
    c0 = c1;
  }
  if (threadIdx.x == 0) {
    R.chunk = chunk;
    R.npicks = np;
    R.batches = batches;
    R.left = left;
  }
  __syncthreads();
  return end;
}

// The greedy rounds of a model (see the top of the file).
// kFirst: all the boxes, or the first kPrefix of more than kWhole; kRest: the survivors that k_nms_rest left of
// the others; kOrderedFirst and kOrderedRest: the same in the quicksort's order.
// kFull = false stops where the quicksort is needed and leaves the model to the kFull instance: with the sort's calls in
// it, the rounds' code is 8 % slower (same rounds: 1280x720, NMS stage 433 us against 399).
enum GreedyPass { kFirst, kRest, kOrderedFirst, kOrderedRest };
template <bool kFull>
__global__ void __launch_bounds__(kResNT, 1) k_nms_greedy(int cap, int *si,
                                                       float *sf, float overlap, float2 cell_inv,
                                                       const __grid_constant__ NmsResults res, int *d_kept,
                                                       long long *diag, const int *need, int *err, bool all_ordered,
                                                       GreedyPass pass, cudaGraphConditionalHandle cond, bool has_cond) {
  extern __shared__ __align__(16) unsigned char res_sm[];
  GreedySmem &R = *reinterpret_cast<GreedySmem *>(res_sm);
  cg::cluster_group cluster = cg::this_cluster();
  const int m = blockIdx.y;
  const bool ordered = kFull && pass >= kOrderedFirst, rest = pass & 1;
  bool whole = false;          // the quicksort's order of all boxes is needed (every block alike)
  WalkResume resume = kAnew;
  {
    const BatchState st = *slots(si, sf, m, cap).st;   // (the same in every block: it is written behind a cluster barrier)
    if (kFull) {
      if (pass == kFirst && st.stage == kNmsWhole) whole = true;
      else if ((pass == kFirst && st.stage == kNmsTied) || (pass == kRest && st.stage == kNmsTiedRest)) resume = kChunkTested;
      else if (!((pass == kRest && st.stage == kNmsPrefix) || (pass == kOrderedFirst && st.stage == kNmsSplit) ||
                 (pass == kOrderedRest && st.stage == kNmsOrderedPrefix)))
        return;
    } else {
      if (st.stage != (pass == kFirst ? kNmsStart : kNmsPrefix)) return;
      whole = pass == kFirst && (all_ordered || need[m]);
    }
    if (threadIdx.x == 0) {
      const bool anew = resume == kAnew;
      R.n = anew ? st.D : st.n;
      R.c0 = anew ? 0 : st.c0;
      R.c1 = anew ? 0 : st.c1;
      R.chunk = anew ? kBatch : st.chunk;
      R.npicks = st.npicks;
      R.tested = anew ? 0 : st.tested;
      R.left = anew ? 0 : st.left;
      R.batches = st.batches;
      R.settled = 0;
    }
  }
  cluster.sync();   // every block has started: its shared memory can be written
  if (kFull && pass == kOrderedFirst) gather_boxes(si, sf, m, cap);
  if (resume != kAnew || whole) {
  } else if (!rest) {
    const Slots S = slots(si, sf, m, cap);
    const int D = R.n, n = D <= kWhole ? D : ordered ? kPrefix : run_end(S, nullptr, kPrefix, D);
    __syncthreads();
    if (threadIdx.x == 0) R.n = n;
  } else {
    // the alive bits of the words from st.next on as a list of sorted positions, in order: a stretch of words per block
    const Slots S = slots(si, sf, m, cap);
    const int rank = (int)cluster.block_rank(), blocks = (int)cluster.num_blocks();
    GreedySmem *R0 = cluster.map_shared_rank(&R, 0);
    const int wa = S.st->next >> 5, nwords = ((R.n + 31) >> 5) - wa;
    const int share = (nwords + blocks - 1) / blocks, per = (share + kResNT - 1) / kResNT;
    const int b0 = wa + rank * share, b1 = min(wa + nwords, b0 + share);
    const int t0 = b0 + threadIdx.x * per, t1 = min(b1, t0 + per);
    int cnt = 0, tot;
    for (int w = t0; w < t1; w++) cnt += __popc(__ldcg(&S.bits[w]));
    int at = block_excl_scan(cnt, &tot, R.wtot);
    if (threadIdx.x == 0) R0->total[rank] = tot;
    cluster.sync();
    int n = 0;
    for (int b = 0; b < blocks; b++) {
      const int v = R0->total[b];
      if (b < rank) at += v;
      n += v;
    }
    for (int w = t0; w < t1; w++)
      for (unsigned rem = __ldcg(&S.bits[w]); rem; rem &= rem - 1) S.Lpos[at++] = (w << 5) + __ffs(rem) - 1;
    if (threadIdx.x == 0) {
      R.n = n;
      R.tested = R.npicks;
    }
    cluster.sync();   // the list is complete, the bitmap free
  }
  __syncthreads();
  bool tied = false;
  while (!whole) {
    if (kFull) asm volatile("" : "+l"(si), "+l"(sf));   // (nothing formed of them is kept over the settling)
    const Slots S = slots(si, sf, m, cap);
    const WalkEnd end = walk_boxes(S, R, rest ? S.Lpos : nullptr, overlap, cell_inv, ordered, resume);
    if (end == kDone) break;
    whole = end == kCut;
    if (!kFull) {
      tied = !whole;
      break;
    }
    if (!whole) whole = !settle_members(R, si, sf, m, cap, err);
    resume = kBatchReady;
  }
  if (kFull) asm volatile("" : "+l"(si), "+l"(sf));
  const Slots S = slots(si, sf, m, cap);
  const int np = R.npicks;
  const bool more = !rest && R.n < S.st->D;
  // the last pick of all shares its score with another pick: which of them is last is the quicksort's call
  if (!whole && !tied && !ordered && !more && np >= 2)
    whole = S.key[__ldcg(&S.picks[np - 1])] == S.key[__ldcg(&S.picks[np - 2])];
  if (kFull && whole) split_boxes(R, si, sf, m, cap, err);
  const bool quick = kFull || whole || tied, first = cluster.block_rank() == 0;
  if (whole || tied || more) {
    if (first && threadIdx.x == 0) {
      BatchState &st = *slots(si, sf, m, cap).st;
      st.stage = whole ? (kFull ? kNmsSplit : kNmsWhole) : tied ? (rest ? kNmsTiedRest : kNmsTied)
                 : ordered ? kNmsOrderedPrefix : kNmsPrefix;
      st.quick |= quick;
      st.next = rest ? st.next : R.n;
      st.n = R.n; st.c0 = R.c0; st.c1 = R.c1; st.chunk = R.chunk; st.tested = R.tested; st.left = R.left;
      st.npicks = whole ? 0 : R.npicks;
      st.batches = R.batches;
      if (!kFull && (whole || tied) && has_cond) cudaGraphSetConditional(cond, 1);
    }
    return;
  }
  if (first) rank_kept(S, R, np);
  cluster.sync();   // the kept boxes are in order
  write_results(S, R, m, cap, res);
  if (first && threadIdx.x == 0) {
    S.st->stage = kNmsDone;
    d_kept[m] = res.host[32 + m] = R.tot;
    if (diag) {
      diag[8 * m + 2] = R.batches;
      diag[8 * m + 3] = np;
      diag[8 * m + 5] = quick || S.st->quick;
    }
  }
  cluster.sync();   // (the first block's ranks have been read)
}

// The boxes from st.next on against every pick so far, over the grid
__global__ void __launch_bounds__(kResNT) k_nms_rest(int cap, int *si, float *sf, float overlap, float2 cell_inv, NmsStage stage) {
  __shared__ PickTable T;
  __shared__ float4 pk[kPickGroup];
  __shared__ float pka[kPickGroup];
  Slots S = slots(si, sf, blockIdx.y, cap);
  const BatchState st = *S.st;
  if (st.stage != stage) return;
  const int w0 = st.next >> 5, w1 = (st.D - 1) >> 5;
  test_chunk(S, T, pk, pka, 0, st.npicks, nullptr, w0, w1, st.next, st.D, overlap, cell_inv,
             blockIdx.x * kResWarps + (threadIdx.x >> 5), gridDim.x * kResWarps);
}

// The quicksort of all boxes of a model that needs it, a block per segment: k_quick_mid takes those that the cluster has
// left (S.Lpos) down to those for shared memory (S.picks: the picks start anew), which k_quick_small finishes
__device__ __forceinline__ bool quick_block(const Slots &S, SortRuns &runs) {
  if (S.st->stage != kNmsSplit) return false;
  if (threadIdx.x == 0) {
    runs.n = 1;
    runs.r[0] = make_int2(0, S.st->D - 1);
  }
  __syncthreads();
  return true;
}

__global__ void __launch_bounds__(kResNT) k_quick_mid(int cap, int *si, float *sf, int *err) {
  extern __shared__ __align__(16) unsigned char res_sm[];
  QuickSmem &Q = *reinterpret_cast<QuickSmem *>(res_sm);
  __shared__ SortRuns runs;
  cg::cluster_group cluster = cg::this_cluster();
  const Slots S = slots(si, sf, blockIdx.y, cap);
  if (!quick_block(S, runs)) return;
  const int2 *mid = reinterpret_cast<const int2 *>(S.Lpos);
  int2 *small = reinterpret_cast<int2 *>(S.picks);   // (disjoint segments of two elements or more: they fit)
  for (int e = blockIdx.x; e < S.st->n_mid; e += gridDim.x) {
    auto push = [&](int2 c) {   // by thread 0
      if (c.y - c.x < kQuickSmall) small[atomicAdd(&S.st->n_small, 1)] = c;
      else if (Q.nst < 40) Q.stk[Q.nst++] = c;
      else atomicOr(err, 512);   // impossible: depth <= log2(kQuickMid) + 1
    };
    if (threadIdx.x == 0) {
      Q.nst = 0;
      push(mid[e]);
    }
    __syncthreads();
    while (Q.nst > 0) {
      const int2 seg = Q.stk[Q.nst - 1];
      __syncthreads();   // everyone has read the top entry
      const int2 ij = quick_partition<false>(cluster, Q, S.qv, S.qo, S.qL, S.qR, seg.x, seg.y);
      if (threadIdx.x == 0) {
        Q.nst--;
        quick_children(runs, 0, seg.x, seg.y, ij.x, ij.y, push, [](int2) {});
      }
      __syncthreads();
    }
    __syncthreads();   // everyone has seen the stack empty
  }
}

__global__ void __launch_bounds__(kResNT) k_quick_small(int cap, int *si, float *sf, int *err) {
  extern __shared__ __align__(16) unsigned char res_sm[];
  QuickSmem &Q = *reinterpret_cast<QuickSmem *>(res_sm);
  __shared__ SortRuns runs;
  cg::cluster_group cluster = cg::this_cluster();
  const Slots S = slots(si, sf, blockIdx.y, cap);
  if (!quick_block(S, runs)) return;
  const int2 *small = reinterpret_cast<const int2 *>(S.picks);
  for (int e = blockIdx.x; e < S.st->n_small; e += gridDim.x) {
    const int2 seg = small[e];
    quick_small(cluster, Q, runs, S, seg.x, seg.y, false, err);
  }
}

// Inside a stream capture: a handle for a conditional node of the graph s is
// capturing (its condition reset to init at every launch of the graph)
static cudaError_t cond_handle(cudaStream_t s, unsigned init, cudaGraphConditionalHandle *h) {
  cudaStreamCaptureStatus cs;
  cudaGraph_t g = nullptr;
  cudaError_t e = cudaStreamGetCaptureInfo(s, &cs, nullptr, &g, nullptr, nullptr, nullptr);
  if (e != cudaSuccess) return e;
  if (cs != cudaStreamCaptureStatusActive) return cudaErrorStreamCaptureUnsupported;
  return cudaGraphConditionalHandleCreate(h, g, init, cudaGraphCondAssignDefault);
}

// the conditional node on s's current dependencies, which become the node;
// aux then captures its body (the capture is begun here, end_conditional ends it)
static cudaError_t begin_conditional(cudaStream_t s, cudaStream_t aux, cudaGraphConditionalNodeType type,
                                     cudaGraphConditionalHandle h) {
  cudaStreamCaptureStatus cs;
  cudaGraph_t g = nullptr;
  const cudaGraphNode_t *deps = nullptr;
  const cudaGraphEdgeData *ed = nullptr;
  size_t nd = 0;
  cudaError_t e = cudaStreamGetCaptureInfo(s, &cs, nullptr, &g, &deps, &ed, &nd);
  if (e != cudaSuccess) return e;
  cudaGraphNodeParams p = {};
  p.type = cudaGraphNodeTypeConditional;
  p.conditional.handle = h;
  p.conditional.type = type;
  p.conditional.size = 1;
  cudaGraphNode_t node;
  if ((e = cudaGraphAddNode(&node, g, deps, ed, nd, &p)) != cudaSuccess) return e;
  if ((e = cudaStreamUpdateCaptureDependencies(s, &node, nullptr, 1, cudaStreamSetCaptureDependencies)) != cudaSuccess)
    return e;
  return cudaStreamBeginCaptureToGraph(aux, p.conditional.phGraph_out[0], nullptr, nullptr, 0,
                                       cudaStreamCaptureModeRelaxed);
}

static cudaError_t end_conditional(cudaStream_t aux) {
  cudaGraph_t body = nullptr;
  cudaError_t e = cudaStreamEndCapture(aux, &body);
  if (e != cudaSuccess) return e;
  return cudaGetLastError();   // a launch inside the body
}

// blocks per model: kCluster where the device can place such a cluster, else the portable 8
template <class K>
static int cluster_blocks(K *kernel, size_t smem) {
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
    cudaGetLastError();
    return 8;
  }
  cudaLaunchConfig_t c = {};
  c.gridDim = dim3(kCluster);
  c.blockDim = dim3(kResNT);
  c.dynamicSmemBytes = smem;
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim = {(unsigned)kCluster, 1, 1};
  c.attrs = &at;
  c.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, kernel, &c) != cudaSuccess || n < 1) {
    cudaGetLastError();
    return 8;
  }
  return kCluster;
}

cudaError_t launch_nms_batch(const int *d_num, int n_models, float overlap,
                             int cap, int *si, float *sf, const NmsResults &res, int *d_kept, int *err,
                             long long *diag, int *need, int order, cudaStream_t s, cudaStream_t aux) {
  if (n_models <= 0) return cudaSuccess;
  // cells over the image and a margin for boxes that leave it (any value is exact: what is outside shares the edge cells)
  const float2 cell_inv = make_float2(kNmsCells / (1.15f * std::max(res.img_h, 1)), kNmsCells / (1.15f * std::max(res.img_w, 1)));
  launch_nms_radix(d_num, n_models, cap, si, sf, need, res.host, s);
  static SmemAttr attr[4];
  cudaError_t e = raise_smem(attr[0], k_nms_greedy<false>, sizeof(GreedySmem));
  if (e == cudaSuccess) e = raise_smem(attr[1], k_nms_greedy<true>, sizeof(GreedySmem));
  if (e == cudaSuccess) e = raise_smem(attr[2], k_quick_mid, sizeof(QuickSmem));
  if (e == cudaSuccess) e = raise_smem(attr[3], k_quick_small, sizeof(QuickSmem));
  if (e != cudaSuccess) return e;
  const int blocks = std::min(cluster_blocks(k_nms_greedy<false>, sizeof(GreedySmem)),
                              cluster_blocks(k_nms_greedy<true>, sizeof(GreedySmem)));
  cudaLaunchConfig_t c = {};
  c.gridDim = dim3(blocks, n_models);
  c.blockDim = dim3(kResNT);
  c.dynamicSmemBytes = sizeof(GreedySmem);
  c.stream = s;
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim = {(unsigned)blocks, 1, 1};
  c.attrs = &at;
  c.numAttrs = 1;
  cudaGraphConditionalHandle h = 0;
  if (aux && (e = cond_handle(s, 0u, &h)) != cudaSuccess) return e;
  auto greedy = [&](bool full, GreedyPass pass) {
    if (e != cudaSuccess || ((pass & 1) && cap <= kWhole)) return;
    if (pass & 1)
      k_nms_rest<<<dim3(std::max(304 / n_models, 1), n_models), kResNT, 0, c.stream>>>(
          cap, si, sf, overlap, cell_inv, pass == kRest ? kNmsPrefix : kNmsOrderedPrefix);
    e = cudaLaunchKernelEx(&c, full ? k_nms_greedy<true> : k_nms_greedy<false>, cap, si, sf, overlap, cell_inv,
                           res, d_kept, diag, (const int *)need, err, order == kNmsOrderQuicksort, pass, h, aux != nullptr);
  };
  greedy(false, kFirst);
  greedy(false, kRest);
  // the models that need the quicksort's order, among a batch's members or of all boxes: in a graph captured with aux, an
  // if node that runs only when some model needs it; otherwise launches that return at once where none does
  if (e == cudaSuccess && aux) {
    e = begin_conditional(s, aux, cudaGraphCondTypeIf, h);
    c.stream = aux;
  }
  if (e != cudaSuccess) return e;
  greedy(true, kFirst);
  greedy(true, kRest);
  k_quick_mid<<<dim3(std::max(152 / n_models, 1), n_models), kResNT, sizeof(QuickSmem), c.stream>>>(cap, si, sf, err);
  k_quick_small<<<dim3(std::max(456 / n_models, 1), n_models), kResNT, sizeof(QuickSmem), c.stream>>>(cap, si, sf, err);
  greedy(true, kOrderedFirst);
  greedy(true, kOrderedRest);
  if (aux) {
    const cudaError_t e2 = end_conditional(aux);
    if (e == cudaSuccess) e = e2;
  }
  return e == cudaSuccess ? cudaGetLastError() : e;
}

}  // namespace geye
