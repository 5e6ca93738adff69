// score.cu -- score assembly, detection records, accumulated score map and
// box regression.
//
//   score = root + offw[ridx[c]] - sum_k M_k[(ay_k-1+2y) + (ax_k-1+2x)*d0_k]
//       CAR_TRACKING/get_boxes.cpp:1022-1041 and dt.cpp:38-55, parts in order
//   threshold in column-major scan order, level by level, component by
//   component: get_boxes.cpp:185-220 (get_gmpc), :1497-1569, :1746-1762
//   root / part boxes: get_boxes.cpp:227-258
//   A_SCORE: get_boxes.cpp:265-300 (CPU form), normalised at :1765-1787
//   box regression: CAR_TRACKING/tracking.cpp:90-166 (get_new_rects)
// Records are written in the reference's order: a per-block count pass, an
// exclusive scan, and a write pass that recomputes the same flags.
#include <algorithm>

#include "internal.h"
#include "rects.h"

namespace geye {


__global__ void k_fill(float *__restrict__ p, size_t n, float v) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) p[i] = v;
}

void launch_fill(float *p, size_t n, float v, cudaStream_t s) {
  size_t b = (n + 255) / 256;
  k_fill<<<(unsigned)(b > 4096 ? 4096 : (b ? b : 1)), 256, 0, s>>>(p, n, v);
}

__device__ __forceinline__ float assemble(const ScoreJob &J, const float *__restrict__ arena, int x, int y) {
  const int i = x * J.r0 + y;
  float s = arena[J.root_off + i];
  s += J.off;
  for (int k = 0; k < J.np; k++) {
    // M at (ax - 1 + 2x, ay - 1 + 2y); compact: its class entry ((ax - 1) / 2 + x, (ay - 1) / 2 + y)
    const int cm0 = J.part_cm0[k];
    const int idx = cm0 ? ((J.ax[k] - 1) / 2 + x) * cm0 + ((J.ay[k] - 1) / 2 + y)
                        : (J.ay[k] + 2 * y - 1) + (J.ax[k] - 1 + 2 * x) * J.part_d0[k];
    s -= arena[J.part_M[k] + idx];
  }
  return s;
}

// One block per entry of `blocks` (job, block of 256 positions): exactly the
// blocks the maps need, whatever their sizes across levels.  Its count of
// positions above the threshold goes to block_counts[blockIdx.x]; the list is
// in job order, so the exclusive scan of the counts places every block's
// records in the reference's order.
__global__ void k_score(const ScoreJob *__restrict__ jobs, const int2 *__restrict__ blocks, float thresh,
                        float *__restrict__ arena, int *__restrict__ block_counts) {
  const int2 blk = blocks[blockIdx.x];
  const ScoreJob &J = jobs[blk.x];
  const int n = J.r0 * J.r1;
  const int i = blk.y * kScoreThreads + threadIdx.x;
  int flag = 0;
  if (i < n) {
    const int y = i % J.r0, x = i / J.r0;
    const float s = assemble(J, arena, x, y);
    arena[J.score_off + i] = s;
    flag = s > thresh;
  }
  const int c = __syncthreads_count(flag);
  if (threadIdx.x == 0) block_counts[blockIdx.x] = c;   // block-list order: job, then position
}

void score_block_list(const std::vector<ScoreJob> &jobs, std::vector<int2> &blocks) {
  blocks.clear();
  for (size_t j = 0; j < jobs.size(); j++)
    for (int b = 0; b * kScoreThreads < jobs[j].r0 * jobs[j].r1; b++) blocks.push_back(make_int2((int)j, b));
}

void launch_score(const ScoreJob *d_jobs, const int2 *d_blocks, int n_blocks, float thresh, float *arena,
                  int *block_counts, cudaStream_t s) {
  if (n_blocks <= 0) return;
  k_score<<<n_blocks, kScoreThreads, 0, s>>>(d_jobs, d_blocks, thresh, arena, block_counts);
}

// exclusive scan of n ints in place (one block); *total gets the sum
__global__ void k_scan(int *__restrict__ a, int n, int *__restrict__ total) {
  __shared__ int warp_sums[32];
  __shared__ int carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int base = 0; base < n; base += blockDim.x) {
    const int i = base + threadIdx.x;
    const int v = i < n ? a[i] : 0;
    int inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      int t = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += t;
    }
    if (lane == 31) warp_sums[warp] = inc;
    __syncthreads();
    if (warp == 0) {
      int w = lane < nw ? warp_sums[lane] : 0;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        int t = __shfl_up_sync(0xffffffffu, w, o);
        if (lane >= o) w += t;
      }
      if (lane < nw) warp_sums[lane] = w;   // inclusive warp prefix
    }
    __syncthreads();
    const int before = carry + (warp > 0 ? warp_sums[warp - 1] : 0) + inc - v;
    if (i < n) a[i] = before;
    __syncthreads();
    if (threadIdx.x == blockDim.x - 1) carry = before + v;
    __syncthreads();
  }
  if (threadIdx.x == 0 && total) *total = carry;
}

void launch_scan_counts(int *counts, int n, int *total, cudaStream_t s) {
  k_scan<<<1, 1024, 0, s>>>(counts, n, total);
}

// Records of a block are contiguous in the output (its offset from the scan,
// then rank order), so they are built in shared memory and written out with
// coalesced stores.
//
// kRecords: whole records (get_boxes itself).  Otherwise what the pipeline's NMS looks at (the root box and the score) and
// the position, from which the records of the few kept ones are formed at the end (nms_batch.cu): 24 bytes a
// detection instead of 156.  Score stage: 640x480 car+person 41 -> 25 us, 1920x1080 139 -> 45 us
template <bool kRecords>
__global__ void __launch_bounds__(kScoreThreads) k_boxes(const ScoreJob *__restrict__ jobs,
                                                         const int2 *__restrict__ blocks, float thresh,
                                                         const float *__restrict__ arena,
                                                         const int *__restrict__ arena_i,
                                                         const int *__restrict__ block_offsets, int GL,
                                                         float *__restrict__ boxes, NmsCandidates cand) {
  extern __shared__ float rec_s[];   // [count][GL]
  __shared__ int warp_cnt[kScoreThreads / 32];
  const int2 blk = blocks[blockIdx.x];
  const ScoreJob &J = jobs[blk.x];
  const int n = J.r0 * J.r1;
  const int i = blk.y * kScoreThreads + threadIdx.x;
  float s = 0.f;
  int flag = 0;
  if (i < n) {
    s = arena[J.score_off + i];
    flag = s > thresh;
  }
  const unsigned bal = __ballot_sync(0xffffffffu, flag);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) warp_cnt[warp] = __popc(bal);
  __syncthreads();
  int rank = __popc(bal & ((1u << lane) - 1)), count = 0;
  for (int w = 0; w < kScoreThreads / 32; w++) {
    if (w < warp) rank += warp_cnt[w];
    count += warp_cnt[w];
  }
  if (count == 0) return;
  if (!kRecords) {
    if (flag) {
      const int o = block_offsets[blockIdx.x] + rank;
      float P[4];
      root_box(i / J.r0, i % J.r0, J.scale, J.rsize0, J.rsize1, P);
      cand.box[o] = make_float4(P[0], P[1], P[2], P[3]);
      cand.score[o] = s;
      cand.ref[o] = blockIdx.x * kScoreThreads + threadIdx.x;
    }
    return;
  }
  if (flag) {
    const int y = i % J.r0, x = i / J.r0;
    float *P = rec_s + rank * GL;
    root_box(x, y, J.scale, J.rsize0, J.rsize1, P);
    for (int k = 0; k < J.np; k++) part_box(J, k, x, y, arena_i, P + 4 * (k + 1));
    float *Q = P + 4 * (J.np + 1);
    Q[0] = (float)J.comp;
    Q[1] = s;
    Q[2] = J.scale;
  }
  __syncthreads();
  float *out = boxes + (size_t)block_offsets[blockIdx.x] * GL;
  for (int t = threadIdx.x; t < count * GL; t += kScoreThreads) out[t] = rec_s[t];
}

void launch_boxes(const ScoreJob *d_jobs, const int2 *d_blocks, int n_blocks, float thresh, const float *arena,
                  const int *arena_i, const int *block_offsets, int GL, float *boxes, cudaStream_t s) {
  if (n_blocks <= 0) return;
  const size_t smem = sizeof(float) * kScoreThreads * GL;
  static SmemAttr attr;
  raise_smem(attr, k_boxes<true>, smem);
  k_boxes<true><<<n_blocks, kScoreThreads, smem, s>>>(d_jobs, d_blocks, thresh, arena, arena_i, block_offsets, GL, boxes,
                                                     NmsCandidates{});
}

void launch_candidates(const ScoreJob *d_jobs, const int2 *d_blocks, int n_blocks, float thresh, const float *arena,
                       const int *block_offsets, const NmsCandidates &out, cudaStream_t s) {
  if (n_blocks <= 0) return;
  k_boxes<false><<<n_blocks, kScoreThreads, 0, s>>>(d_jobs, d_blocks, thresh, arena, nullptr, block_offsets, 0, nullptr, out);
}

// A_SCORE in gather form: target pixel (X, Y) takes the max over every
// (level, component) of the score at the cell that the reference's scatter
// loop maps from source pixel (X - RX, Y - RY) -- looked up in the plan's
// per-map column and row tables -- then the threshold/offset of
// get_boxes.cpp:1765-1776 and a running maximum for the normalisation.
// A block owns a tile of kAsX columns of kAsY pixels and stages the tile's table entries of
// every map (kAsJobs at a time) in shared memory, so only the score gathers touch global memory.  The maximum is exact
// in any order.  A thread takes four pixels of a column: a cell is four pixels or more in every map but those of models with
// small cells, so the four lie in two cells at most and two gathers serve them; where a quad of the tile has a third
// cell between (found while staging), the block looks every pixel up.
// What bounds it alone is latency (12 us a model at 640x480, with a thread per pixel too), but it runs beside NMS and, in a
// server or batch, beside other frames, where the instructions and warps it takes count: with a thread per pixel (a gather
// and nine instructions each) 16 served frames of 640x480 took 3434 us, 3351 so; eight mixed frames 2265 and 2205;
// 1920x1080 1771 and 1744.
constexpr int kAsX = 16, kAsY = 32, kAsThreads = kAsX * kAsY / 4, kAsJobs = 128;

__global__ void __launch_bounds__(kAsThreads) k_ascore(const int *__restrict__ col, const int *__restrict__ row,
                                                       int n_jobs, const float *__restrict__ arena,
                                                       float *__restrict__ a_score, int im_w, int im_h,
                                                       float thresh, unsigned *max_bits) {
  __shared__ int4 row_s[kAsJobs * (kAsY / 4)];
  __shared__ int col_s[kAsJobs * kAsX];
  const int X0 = blockIdx.y * kAsX, Y0 = blockIdx.x * kAsY;
  const int tx = threadIdx.x / (kAsY / 4), ty = threadIdx.x % (kAsY / 4);
  const int X = X0 + tx, Y = Y0 + 4 * ty;
  const size_t idx = (size_t)X * im_h + Y;
  const int n = X < im_w ? min(4, im_h - Y) : 0;   // pixels of this thread
  float a[4];
#pragma unroll
  for (int k = 0; k < 4; k++) a[k] = k < n ? a_score[idx + k] : 0.f;
  const float none = -INFINITY;   // never above a score
  for (int j0 = 0; j0 < n_jobs; j0 += kAsJobs) {
    const int nj = min(kAsJobs, n_jobs - j0);
    if (j0) __syncthreads();
    for (int i = threadIdx.x; i < nj * kAsY; i += kAsThreads) {
      const int j = j0 + i / kAsY, k = i % kAsY;
      reinterpret_cast<int *>(row_s)[i] = Y0 + k < im_h ? row[(size_t)j * im_h + Y0 + k] : -1;
    }
    for (int i = threadIdx.x; i < nj * kAsX; i += kAsThreads) {
      const int j = j0 + i / kAsX, k = i % kAsX;
      col_s[i] = X0 + k < im_w ? col[(size_t)j * im_w + X0 + k] : -1;
    }
    __syncthreads();
    bool third = false;
    for (int i = threadIdx.x; i < nj * (kAsY / 4); i += kAsThreads) {
      const int4 r = row_s[i];
      third |= (r.y != r.x && r.y != r.w) || (r.z != r.x && r.z != r.w);
    }
    third = __syncthreads_or(third);
    if (n <= 0) continue;
    const int *tc = col_s + tx;
    const int4 *tr = row_s + ty;
    if (!third) {
#pragma unroll 8   // sixteen gathers in flight per thread
      for (int j = 0; j < nj; j++) {
        const int c = tc[j * kAsX];
        const int4 r = tr[j * (kAsY / 4)];
        const float u = (c | r.x) >= 0 ? arena[c + r.x] : none, v = (c | r.w) >= 0 ? arena[c + r.w] : none;
        const float s1 = r.y == r.x ? u : v, s2 = r.z == r.x ? u : v;
        if (u > a[0]) a[0] = u;
        if (s1 > a[1]) a[1] = s1;
        if (s2 > a[2]) a[2] = s2;
        if (v > a[3]) a[3] = v;
      }
    } else {
#pragma unroll 2
      for (int j = 0; j < nj; j++) {
        const int c = tc[j * kAsX];
        const int4 r = tr[j * (kAsY / 4)];
        const int e[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
        for (int k = 0; k < 4; k++) {
          const float sc = (c | e[k]) >= 0 ? arena[c + e[k]] : none;
          if (sc > a[k]) a[k] = sc;
        }
      }
    }
  }
  unsigned local_max = 0;
  if (n > 0) {
    const float AS_OFF = fabsf(thresh);
#pragma unroll
    for (int k = 0; k < 4; k++) {
      if (k >= n) break;
      if (a[k] < thresh) a[k] = 0.0;
      else a[k] += AS_OFF;
      a_score[idx + k] = a[k];
      if (a[k] > 0.0f) local_max = max(local_max, __float_as_uint(a[k]));
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) local_max = max(local_max, __shfl_xor_sync(0xffffffffu, local_max, o));
  if ((threadIdx.x & 31) == 0 && local_max) atomicMax(max_bits, local_max);
}

__global__ void k_ascore_norm(float *__restrict__ a_score, int n, const unsigned *__restrict__ max_bits) {
  const float max_ac = __uint_as_float(*max_bits);
  if (!(max_ac > 0.0f)) return;
  // the reference's double reciprocal, once per warp (the FP64 pipe is narrow)
  float ac_ratio = 0.f;
  if ((threadIdx.x & 31) == 0) ac_ratio = 1.0 / max_ac;
  ac_ratio = __shfl_sync(0xffffffffu, ac_ratio, 0);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) a_score[i] *= ac_ratio;
}

void launch_ascore(const int *col, const int *row, int n_jobs, const float *arena, float *a_score, int im_w,
                  int im_h, float thresh, unsigned *max_bits, cudaStream_t s) {
  dim3 grid((im_h + kAsY - 1) / kAsY, (im_w + kAsX - 1) / kAsX);
  k_ascore<<<grid, kAsThreads, 0, s>>>(col, row, n_jobs, arena, a_score, im_w, im_h, thresh, max_bits);
}

void launch_ascore_normalize(float *a_score, int n, const unsigned *max_bits, cudaStream_t s) {
  int blocks = (n + 255) / 256;
  if (blocks > 4096) blocks = 4096;
  k_ascore_norm<<<blocks, 256, 0, s>>>(a_score, n, max_bits);
}

// get_new_rects on kept records
__global__ void k_new_rects(const float *__restrict__ kept, const int *__restrict__ d_kept, int GL, int np,
                            const float *__restrict__ coef, int img_w, int img_h, float ratio, int *point,
                            int *or_point, int *type, float *scale, float *score) {
  const int K = *d_kept;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < 4 * K; e += gridDim.x * blockDim.x) {
    const int k = e >> 2, c = e & 3;
    const float *P = kept + (size_t)k * GL;
    const int v = new_rect_side(P, GL, np, coef, img_w, img_h, c);
    point[e] = v;
    or_point[e] = (int)((float)v / ratio);
    if (c == 0) type[k] = (int)P[GL - 3];
    if (c == 1) scale[k] = P[GL - 1];
    if (c == 2) score[k] = P[GL - 2];
  }
}

void launch_new_rects(const float *kept, const int *d_kept, int GL, int np, const float *coef, int img_w,
                      int img_h, float ratio, int *point, int *or_point, int *type, float *scale, float *score,
                      cudaStream_t s) {
  k_new_rects<<<16, 256, 0, s>>>(kept, d_kept, GL, np, coef, img_w, img_h, ratio, point, or_point, type, scale,
                                 score);
}

}  // namespace geye
