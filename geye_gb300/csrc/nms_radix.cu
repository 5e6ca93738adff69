// nms_radix.cu -- the detections in score order for the pipeline NMS, every
// model of a frame at once: a stable least-significant-digit radix sort of the
// scores (descending) with the input index as the order among equal scores.
//
// The greedy suppression of CAR_TRACKING/nms.cpp:86-217 walks the boxes in the
// order of the reference's quicksort (nms.cpp:70-84).  That order and this one
// differ only inside runs of equal scores, and the kept set can depend on the
// order inside a run only when
//   (a) two boxes of one run are both alive when the run's turn comes and one
//       suppresses the other, or
//   (b) the last pick's run holds another pick (which of them is last decides
//       the reference's rule for a box that is alone at its turn),
// or when a score is NaN (the quicksort places it by its comparisons).  The
// greedy rounds (nms_batch.cu) check (a) and (b) as they go and take the
// quicksort's order there (nms_quick.h), and from the start for a model whose
// flag is raised here (NaN).  The kept set is the reference's either way.
//
//   k_rs_load     keys (order-preserving transform of the float score, -0 as
//                 +0, complemented for descending order), indices, the
//                 greedy state, and the digit counts of the first
//                 pass per tile of nms_rs_tile(cap) keys; NaN raises the flag.
//   k_rs_pass     four passes of eight bits, one kernel each: a block per tile
//                 adds up the tiles' digit counts before it (at most a few
//                 hundred coalesced rows, so no scan kernel between the
//                 passes), ranks its keys (warp match, warp prefix: stable),
//                 writes them out and counts the next pass's digits at the
//                 tile each key lands in.  The last pass also brings the boxes
//                 into sorted order.
// What bounds it is latency: a kernel boundary per pass.  With a count, a scan
// (one block per model) and a scatter kernel per pass and a gather behind them,
// 14 launches instead of 5, the 640x480 pair's NMS took 285 us; see nms_batch.cu.
// Keys ping-pong between (key, ord) and (Lpos, Rpos); after the fourth pass
// they are back in (key, ord): key holds the transformed keys (equal keys <=>
// equal scores), ord the input index of each sorted position.
#include "nms_common.h"

namespace geye {

constexpr int kRsNT = 512;
constexpr int kRsWarps = kRsNT / 32;

__device__ __forceinline__ unsigned rs_key(float v, bool &nan) {
  unsigned u = __float_as_uint(v);
  if (u == 0x80000000u) u = 0u;   // -0 sorts with +0 (the quicksort's comparisons see them equal)
  nan = v != v;
  const unsigned asc = (u & 0x80000000u) ? ~u : (u | 0x80000000u);
  return ~asc;   // ascending keys = descending scores
}

__global__ void __launch_bounds__(kRsNT) k_rs_load(const int *__restrict__ d_num, int cap, int *si, float *sf, int *need, int *host) {
  __shared__ int h[256];
  const int m = blockIdx.y, t = blockIdx.x;
  Slots S = slots(si, sf, m, cap);
  const int D = max(0, min(d_num[m], cap)), T = nms_rs_tile(cap);
  if (t == 0 && threadIdx.x == 0) {
    BatchState &st = *S.st;
    st.D = D;
    st.stage = D > 0 ? kNmsStart : kNmsDone;
    st.quick = st.next = st.npicks = st.batches = st.n_mid = st.n_small = st.n_left = 0;
    host[m] = D;
    host[32 + m] = 0;
  }
  const int e0 = t * T;
  if (e0 >= D) return;
  if (threadIdx.x < 256) h[threadIdx.x] = 0;
  __syncthreads();
  bool nan = false;
  for (int i = e0 + threadIdx.x; i < min(e0 + T, D); i += kRsNT) {
    const unsigned k = rs_key(S.score[i], nan);
    if (nan) need[m] = 1;
    S.key[i] = k;
    S.ord[i] = i;
    atomicAdd(&h[k & 255u], 1);
  }
  __syncthreads();
  const size_t pass_words = (size_t)256 * nms_rs_tiles(cap);
  if (threadIdx.x < 256) {
    int *H = S.hist + (size_t)256 * t + threadIdx.x;
    H[0] = h[threadIdx.x];
    for (int p = 1; p < 4; p++) H[p * pass_words] = 0;
  }
}

// pass p reads (key, ord) for even p and (Lpos, Rpos) for odd p
__device__ __forceinline__ void rs_bufs(const Slots &S, int pass, const unsigned *&sk, const int *&si_, unsigned *&dk,
                                        int *&di) {
  unsigned *a_k = S.key, *b_k = reinterpret_cast<unsigned *>(S.Lpos);
  int *a_i = S.ord, *b_i = S.Rpos;
  if (pass & 1) {
    sk = b_k; si_ = b_i; dk = a_k; di = a_i;
  } else {
    sk = a_k; si_ = a_i; dk = b_k; di = b_i;
  }
}

// IT keys per thread (a tile of kRsNT * IT); pass 3 gathers the boxes
template <int IT>
__global__ void __launch_bounds__(kRsNT) k_rs_pass(int pass, int cap,
                                                   int *si, float *sf) {
  constexpr int T = kRsNT * IT;
  __shared__ int before_s[2][256], total_s[2][256];
  __shared__ int cnt[kRsWarps][256];
  __shared__ int wsum[8];
  const int m = blockIdx.y, t = blockIdx.x;
  Slots S = slots(si, sf, m, cap);
  const int D = S.st->D, nt = (D + T - 1) / T;
  if (t >= nt) return;
  const unsigned *sk;
  const int *sidx;
  unsigned *dk;
  int *di;
  rs_bufs(S, pass, sk, sidx, dk, di);
  const int shift = 8 * pass;
  const size_t pass_words = (size_t)256 * nms_rs_tiles(cap);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // the thread's keys: a warp's 32 * IT are consecutive
  unsigned key[IT];
  int idx[IT], rank[IT];
#pragma unroll
  for (int k = 0; k < IT; k++) {
    const int e = t * T + warp * (32 * IT) + 32 * k + lane;
    key[k] = e < D ? sk[e] : 0u;
    idx[k] = e < D ? sidx[e] : -1;
  }
  {   // digit counts of the tiles before this one, and of all: two threads per digit, half of the tiles each
    const int d = threadIdx.x & 255, half = threadIdx.x >> 8, mid = (nt + 1) / 2;
    const int *H = S.hist + pass * pass_words + d;
    int before = 0, total = 0;
#pragma unroll 8
    for (int u = half ? mid : 0; u < (half ? nt : mid); u++) {
      const int c = H[(size_t)256 * u];
      total += c;
      if (u < t) before += c;
    }
    before_s[half][d] = before;
    total_s[half][d] = total;
    for (int k = threadIdx.x; k < kRsWarps * 256; k += kRsNT) (&cnt[0][0])[k] = 0;
  }
  __syncthreads();
  int tot = 0, inc = 0;
  if (threadIdx.x < 256) {   // exclusive scan of the totals
    tot = total_s[0][threadIdx.x] + total_s[1][threadIdx.x];
    inc = tot;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += v;
    }
    if (lane == 31) wsum[warp] = inc;
  }
  const unsigned lt = (1u << lane) - 1u;
#pragma unroll
  for (int k = 0; k < IT; k++) {
    const int digit = (int)((key[k] >> shift) & 255u);
    // lanes past the end match nobody (a value no digit takes)
    const unsigned peers = __match_any_sync(0xffffffffu, idx[k] >= 0 ? digit : 256 + lane);
    const int prev = cnt[warp][digit];
    __syncwarp();
    if (idx[k] >= 0 && (peers & lt) == 0u) cnt[warp][digit] = prev + __popc(peers);
    __syncwarp();
    rank[k] = prev + __popc(peers & lt);
  }
  __syncthreads();
  if (threadIdx.x < 256) {
    int acc = inc - tot + before_s[0][threadIdx.x] + before_s[1][threadIdx.x];
    for (int w = 0; w < warp; w++) acc += wsum[w];
#pragma unroll
    for (int w = 0; w < kRsWarps; w++) {
      const int c = cnt[w][threadIdx.x];
      cnt[w][threadIdx.x] = acc;
      acc += c;
    }
  }
  __syncthreads();
  int *Hn = S.hist + (pass + 1) * pass_words;
#pragma unroll
  for (int k = 0; k < IT; k++) {
    const bool valid = idx[k] >= 0;
    const int p = cnt[warp][(key[k] >> shift) & 255u] + rank[k];
    if (valid) {
      dk[p] = key[k];
      di[p] = idx[k];
    }
    if (pass < 3) {   // one addition per (tile, digit) of the warp
      const int q = valid ? (p / T) * 256 + (int)((key[k] >> (shift + 8)) & 255u) : -1 - lane;
      const unsigned peers = __match_any_sync(0xffffffffu, q);
      if (valid && (peers & lt) == 0u) atomicAdd(&Hn[q], __popc(peers));
    } else if (valid) {
      const float4 b = S.box[idx[k]];
      const float y1 = b.x, x1 = b.y, y2 = b.z, x2 = b.w;
      S.y1[p] = y1; S.x1[p] = x1; S.y2[p] = y2; S.x2[p] = x2;
      S.ar[p] = (x2 - x1 + 1.0) * (y2 - y1 + 1.0);   // nms.cpp's area expression
    }
  }
}

void launch_nms_radix(const int *d_num, int n_models, int cap, int *si, float *sf,
                      int *need, int *host, cudaStream_t s) {
  const dim3 grid(nms_rs_tiles(cap), n_models);
  k_rs_load<<<grid, kRsNT, 0, s>>>(d_num, cap, si, sf, need, host);
  for (int p = 0; p < 4; p++) {
    if (nms_rs_tile(cap) == 2 * kRsNT) k_rs_pass<2><<<grid, kRsNT, 0, s>>>(p, cap, si, sf);
    else k_rs_pass<8><<<grid, kRsNT, 0, s>>>(p, cap, si, sf);
  }
}

}  // namespace geye
