// nms_common.h -- scratch layout and device routines shared by the pipeline
// NMS kernels (nms_radix.cu: score order; nms_batch.cu: the greedy suppression;
// nms_quick.h: the reference's quicksort).  Reference: CAR_TRACKING/nms.cpp:70-217.
#pragma once
#include <stdint.h>

#include "internal.h"

namespace geye {

enum NmsStage : int {   // how far a model is (see the launches at the end of nms_batch.cu)
  kNmsStart,     // nothing looked at
  kNmsPrefix,    // the first kPrefix boxes done: the others to be tested
  kNmsTied,      // stopped among these: members to be put in the quicksort's order
  kNmsTiedRest,  // stopped among the others' survivors
  kNmsWhole,     // the quicksort's order of all boxes is needed
  kNmsSplit,     // its first passes done
  kNmsOrderedPrefix,
  kNmsDone
};
struct BatchState {   // greedy rounds, between launches
  int D;
  NmsStage stage;
  int quick;                   // the quicksort's order has been asked for
  int next;                    // the first box not looked at
  int n, c0, c1, chunk, npicks, tested, left, batches;   // the walk's place (walk_boxes in nms_batch.cu)
  int n_mid, n_small;          // segments waiting for a block (in Lpos), and for a block's shared memory (in picks)
  int n_left;                  // the quicksort's segments not in order yet (in hist; 0: it has not begun)
  int pad[1];
};

// per-model scratch: nms_model_words(cap) ints and 16 * cap floats
struct Slots {
  unsigned *key;     // sort keys (nms_radix.cu)
  int *ord;          // sorted position -> box
  int *Lpos, *Rpos;  // the radix sort's second buffers; then Lpos the list of items, Rpos the kept boxes' input indices
  float *qv;         // the quicksort's values, boxes and partition lists
  int *qo, *qL, *qR;
  int *place;        // box -> its place in the quicksort's order
  int *picks;        // sorted positions of the picks, in pick order
  int *flag;         // per pick: it suppressed at least one box
  unsigned *bits;    // alive bitmap (nms_batch.cu)
  BatchState *st;
  int *hist;         // [pass][tile][256] radix-sort digit counts (nms_radix.cu); then the quicksort's segments
  float *y1, *x1, *y2, *x2, *ar;   // boxes in sorted order
  float4 *pb;        // the picks' boxes y1, x1, y2, x2 and areas, in pick order
  float *pa;
  const float4 *box;   // the candidates in input order (NmsCandidates)
  const float *score;
  const int *ref;
};

__device__ __forceinline__ Slots slots(int *si, float *sf, int m, int cap) {
  int *b = si + (size_t)m * nms_model_words(cap);
  float *f = sf + (size_t)m * 16 * cap;
  const size_t n = cap;
  Slots S;
  S.st = reinterpret_cast<BatchState *>(b);
  b += 32;
  S.key = reinterpret_cast<unsigned *>(b);
  S.ord = b + n;
  S.Lpos = b + 2 * n;
  S.Rpos = b + 3 * n;
  S.qv = reinterpret_cast<float *>(b + 4 * n);
  S.qo = b + 5 * n;
  S.qL = b + 6 * n;
  S.qR = S.Rpos;
  S.picks = b + 7 * n;
  S.flag = b + 8 * n;
  S.place = b + 9 * n;
  S.bits = reinterpret_cast<unsigned *>(b + 10 * n);
  S.hist = b + ((10 * n + n / 32 + 2) & ~(size_t)1);
  S.y1 = f;
  S.x1 = f + cap;
  S.y2 = f + 2 * (size_t)cap;
  S.x2 = f + 3 * (size_t)cap;
  S.ar = f + 4 * (size_t)cap;
  S.pb = reinterpret_cast<float4 *>(f + 5 * (size_t)cap);
  S.pa = f + 9 * n;
  S.box = reinterpret_cast<const float4 *>(f + 10 * n);
  S.score = f + 14 * n;
  S.ref = reinterpret_cast<const int *>(f + 15 * n);
  return S;
}

// suppression test (nms.cpp:141-176) for the pipeline's boxes (score.cu's root_box: both extents, with the
// + 1 of the widths, are positive): containment is an overlap, so only the ratio
// of the areas decides.  A is the kept box, B the other one; nms.cpp adds the double 1.0
// and stores a float: one rounding of the exact sum, which is what the float addition gives.
__device__ __forceinline__ bool supp(float Ay1, float Ax1, float Ay2, float Ax2, float aA, float By1, float Bx1,
                                            float By2, float Bx2, float aB, float overlap) {
  const float w = fminf(Ax2, Bx2) - fmaxf(Ax1, Bx1) + 1.0f;
  const float h = fminf(Ay2, By2) - fmaxf(Ay1, By1) + 1.0f;
  const float R_AREA = fminf(aA, aB);
  // w * h / R_AREA > overlap, without the division where the product with the
  // overlap decides: with u = 2^-24, q > p (1 + 2^-21) (each side rounded) puts q / R_AREA
  // above overlap (1 + 2^-22), whose rounding is above overlap; below likewise
  const float q = w * h, p = R_AREA * overlap;
  const bool meet = fminf(w, h) > 0.0f;
  const bool over = q > p * (1.0f + 4.76837158203125e-07f), under = q < p * (1.0f - 4.76837158203125e-07f);
  bool s = meet & over;
  if (meet & !((over | under) & (p > 1e-30f) & (p < 1e30f))) s = q / R_AREA > overlap;
  return s;
}

// key-order sort (nms_radix.cu): key = transformed scores, ord = input index,
// BatchState initialised; need[m] set for a NaN score
void launch_nms_radix(const int *d_num, int n_models, int cap, int *si, float *sf,
                      int *need, int *host, cudaStream_t s);

}  // namespace geye
