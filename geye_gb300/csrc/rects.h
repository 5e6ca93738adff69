// rects.h -- one detection's record (get_boxes.cpp:227-258) and the box regression of a
// kept one (get_new_rects, CAR_TRACKING/tracking.cpp:90-166), shared by the stage
// entry points' kernels (score.cu) and the pipeline's (nms_batch.cu).
#pragma once
#include "internal.h"

namespace geye {

// partbox (get_boxes.cpp:243-258) is written in double; every step of it is
// exact except the final rounding to float, so it is restated in float and
// integer arithmetic with that one rounding (the FP64 pipe is narrow here):
//   q0 = ((py - 2)/2 + 1) * scale  ==  (py * 0.5f) * scale   (exact product, one rounding)
//   q2 = q0 + psize*scale/2 - 1     ==  one rounding of the exact sum (below)

// float(q + h - 1) with the sum taken exactly.  For q, h in [0.5, 2^23) the
// double expression is exact before its rounding to float.  In float:
// s + e = q + h exactly (TwoSum; no contraction), s - 1 is exact for
// 1 <= s < 2^24 (1 is a multiple of s's unit in the last place), so
// (s - 1) + e is one correctly rounded addition of the exact q + h - 1.
// (64-bit integer conversions would run on the narrow FP64 pipe.)
__device__ __forceinline__ float sum_minus_one(float q, float h) {
  if (q >= 0.5f && h >= 0.5f && q < 8388608.0f && h < 8388608.0f) {
    const float s = q + h;
    const float bb = s - q;
    const float e = (q - (s - bb)) + (h - bb);
    return (s - 1.0f) + e;
  }
  return (float)((double)q + (double)h - 1.0);
}

// Part k of the detection at position (x, y): the corner (y1, x1) of its box
__device__ __forceinline__ float2 part_corner(const ScoreJob &J, int k, int x, int y, const int *__restrict__ arena_i) {
  const int probex = (x - 1) * 2 + J.ax[k];
  const int probey = (y - 1) * 2 + J.ay[k];
  long Pi;
  if (const int ci0 = J.part_ci0[k]) {   // compact: every probe is inside and in the stored class
    Pi = (long)(probex >> 1) * ci0 + (probey >> 1);
  } else {
    Pi = probey + (long)probex * J.part_d0[k];
    // the reference reads outside the map here (undefined); use entry 0 instead
    if (Pi < 0 || Pi >= (long)J.part_d0[k] * J.part_d1[k]) Pi = 0;
  }
  const float px = (float)arena_i[J.part_Ix[k] + Pi] + 1.0f;   // an integer: exact
  const float py = (float)arena_i[J.part_Iy[k] + Pi] + 1.0f;
  return make_float2((py * 0.5f) * J.scale, (px * 0.5f) * J.scale);
}

// its box into Q
__device__ __forceinline__ void part_box(const ScoreJob &J, int k, int x, int y, const int *__restrict__ arena_i, float *Q) {
  const float2 q = part_corner(J, k, x, y, arena_i);
  Q[0] = q.x;
  Q[1] = q.y;
  Q[2] = sum_minus_one(q.x, ((float)J.psize0[k] * J.scale) * 0.5f);
  Q[3] = sum_minus_one(q.y, ((float)J.psize1[k] * J.scale) * 0.5f);
}

// A regressed side, clamped to the image
__device__ __forceinline__ int rect_bound(float sum, int img_w, int img_h, int side) {
  if (side < 2) return sum > 0 ? (int)sum : 0;
  const int lim = side == 2 ? img_w : img_h;
  return sum < lim ? (int)sum : lim;
}

// One side of the rectangle of record P (0: x1, 1: y1, 2: x2, 3: y2), clamped to the image;
// coef = [comp][x1, y1, x2, y2][ML]
__device__ __forceinline__ int new_rect_side(const float *__restrict__ P, int GL, int np,
                                             const float *__restrict__ coef, int img_w, int img_h, int side) {
  const int ML = 1 + 2 * (1 + np), LL = GL - 3;
  const int CNUM = (int)P[GL - 3];
  const float *w = coef + ((size_t)CNUM * 4 + side) * ML;
  float sum = 0;
  for (int k0 = 0; k0 < ML; k0 += 8) {   // eight loads ahead of the ordered sum
    float av[8], wv[8];
#pragma unroll
    for (int u = 0; u < 8; u++) {
      const int q = k0 + u - 1, box = q >> 1;   // Avec = [w, (x1, y1) of root and parts]
      const bool in = k0 + u < ML && k0 + u > 0 && 4 * box < LL;
      av[u] = in ? ((q & 1) ? P[4 * box] : P[4 * box + 1]) : 0.f;
      wv[u] = k0 + u < ML ? w[k0 + u] : 0.f;
    }
    if (k0 == 0) av[0] = P[3] - P[1];
#pragma unroll
    for (int u = 0; u < 8; u++)
      if (k0 + u < ML) sum += av[u] * wv[u];
  }
  return rect_bound(sum, img_w, img_h, side);
}

}  // namespace geye
