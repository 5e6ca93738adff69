// rects.h -- box regression of one kept record (get_new_rects,
// CAR_TRACKING/tracking.cpp:90-166), shared by the stage entry point's kernel
// (score.cu) and the pipeline's (nms_batch.cu).
#pragma once
#include "internal.h"

namespace geye {

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
  if (side < 2) return sum > 0 ? (int)sum : 0;
  const int lim = side == 2 ? img_w : img_h;
  return sum < lim ? (int)sum : lim;
}

}  // namespace geye
