// nms_quick.h -- the reference's quicksort of the detection scores
// (CAR_TRACKING/nms.cpp:70-84) by one cluster, with its exact order for equal
// scores, as far as the greedy rounds (nms_batch.cu) ask for it.
//
// Each partition reproduces one pass of the reference's loop (key = the middle
// element, i stops at a[i] <= key, j at a[j] >= key, swap, recurse on [lo, i-1]
// and [j+1, hi]): with L the positions holding a value <= key in ascending
// order and R those holding a value >= key in descending order, the sequential
// loop swaps L[k] with R[k] for every k < K, K = #{k : L[k] < R[k]} (a prefix,
// since L rises and R falls), and stops at i = min(L[K], R[K-1]),
// j = max(R[K], L[K-1]) (i = L[0], j = R[0] when K = 0).
//
// What the greedy rounds need to know is the order inside a few runs of equal
// scores.  A run takes the same places in every order of the scores, so only
// the segments that hold one of those places are partitioned further: after
// the first few passes next to nothing of the array.  quick_sort does that
// inside the greedy kernel: the cluster partitions segments above kQuickSmall one at a
// time, the others are finished by a block each in shared memory: partitions by
// the block, by warps below kQuickWarp and by threads below kTiny.
//
// Where the order of all boxes is needed, the cluster only splits the array into segments of
// kQuickMid; k_quick_mid (a block per segment, in global memory) and k_quick_small (shared memory)
// finish them over the whole chip.
//
// What bounds it is latency: three cluster barriers and five dependent L2 round
// trips a pass, 14 000 cycles for a segment of 30 000 or less, 85 000 for 600 000.  The places of a run of
// 30 among 600 000 boxes: 250 us (20 passes and one block's segment of 3500, 100 000 cycles); all boxes over the grid: 1050 us.
// All boxes here: 370 us for the split, 200 for the rest.
#pragma once
#include <cooperative_groups.h>

#include "nms_common.h"

namespace geye {

namespace cg = cooperative_groups;

constexpr int kCluster = 16;         // blocks per model (8 where a device cannot place 16)
constexpr int kResNT = 512, kResWarps = kResNT / 32;
constexpr int kRuns = 16;            // runs asked for at once
constexpr int kQuickMid = 32768, kQuickSmall = 4096, kQuickWarp = 512, kTiny = 32;
constexpr int kQuickList = 256, kQuickWarpList = 64;
constexpr int kQuickLeft = 512;      // segments kept between two calls (in S.hist: 4 * 256 ints at least)

struct SortRuns {   // places of the sorted order, ascending
  int n;
  int2 r[kRuns];
};

struct QuickSmem {
  float a[kQuickSmall];
  int o[kQuickSmall];
  uint16_t Lp[kQuickSmall], Rp[kQuickSmall];
  int2 list[kQuickList];            // segments for one block each
  int2 left[kQuickLeft];            // segments that no run has asked for, or whose order is in S.place only
  int2 stk[40], sstk[16];           // segments for the cluster (for the block in k_quick_mid), of a block's shared memory
  int2 wl[kQuickWarpList];          // segments for one warp
  int2 tiny[kResWarps][32];         // per warp: segments for one thread
  int tiny_n[kResWarps];
  int2 wc[kResWarps], tot[kCluster];
  int wk[kResWarps], ktot[kCluster];
  int nst, nl, nleft, ns, wl_n, wl_next;
};

// whether a segment holds a place of the runs
__device__ __forceinline__ bool quick_wanted(const SortRuns &runs, int lo, int hi) {
  bool w = false;
  for (int k = 0; k < runs.n; k++) w |= lo <= runs.r[k].y && hi >= runs.r[k].x;
  return w;
}

// a segment's wanted children, the larger one first (a stack's depth is then log2 of the segment at most): fn(child);
// the others to left(child)
template <class F, class G>
__device__ __forceinline__ void quick_children(const SortRuns &runs, int base, int lo, int hi, int i, int j, F fn, G left) {
  int2 ch[2] = {make_int2(lo, i - 1), make_int2(j + 1, hi)};
  if (ch[0].y - ch[0].x < ch[1].y - ch[1].x) { const int2 t = ch[0]; ch[0] = ch[1]; ch[1] = t; }
#pragma unroll
  for (int u = 0; u < 2; u++)
    if (ch[u].x < ch[u].y) {
      if (quick_wanted(runs, base + ch[u].x, base + ch[u].y)) fn(ch[u]);
      else left(ch[u]);
    }
}

// One pass over val[lo..hi]: by the whole cluster (kCl) or by one block.  Positions of lists Lp, Rp in type P; shared
// memory (a block's small segments) or global memory, read past L1 there: other blocks have written it.  Returns (i, j).
template <bool kCl, class P>
__device__ __forceinline__ int2 quick_partition(cg::cluster_group &cluster, QuickSmem &Q, float *val, int *ord, P *Lpos,
                                                P *Rpos, int lo, int hi) {
  (void)cluster;
  constexpr bool kGlobal = sizeof(P) == 4;
  constexpr int kU = kGlobal ? 8 : 1;   // loads in flight per thread
  auto ld = [](const auto *p) {
    if constexpr (kGlobal) return __ldcg(p);
    else return *p;
  };
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int rank = kCl ? (int)cluster.block_rank() : 0, blocks = kCl ? (int)cluster.num_blocks() : 1;
  const int gw = rank * kResWarps + warp, nw = blocks * kResWarps;
  const int per = ((hi - lo + nw) / nw + 31) & ~31;   // a stretch of positions per warp
  const int p0 = min(lo + gw * per, hi + 1), p1 = min(p0 + per, hi + 1);
  const unsigned lt = (1u << lane) - 1u;
  const float key = ld(val + (lo + hi) / 2);
  int bl = 0, br = 0;
  for (int p = p0 + lane; p < p1; p += 32 * kU) {
    float v[kU];
#pragma unroll
    for (int u = 0; u < kU; u++) v[u] = p + 32 * u < p1 ? ld(val + p + 32 * u) : key;
#pragma unroll
    for (int u = 0; u < kU; u++) {
      bl += p + 32 * u < p1 && !(v[u] > key);
      br += p + 32 * u < p1 && !(v[u] < key);
    }
  }
  bl = __reduce_add_sync(0xffffffffu, bl);
  br = __reduce_add_sync(0xffffffffu, br);
  if (lane == 0) Q.wc[warp] = make_int2(bl, br);
  __syncthreads();
  bl = br = 0;
  int nL = 0, nR = 0;
  for (int w = 0; w < kResWarps; w++) {
    const int2 c = Q.wc[w];
    if (w < warp) { bl += c.x; br += c.y; }
    nL += c.x;
    nR += c.y;
  }
  if (kCl) {
    if (threadIdx.x < blocks) cluster.map_shared_rank(&Q, threadIdx.x)->tot[rank] = make_int2(nL, nR);
    cluster.sync();
    nL = nR = 0;
    for (int b = 0; b < blocks; b++) {
      const int2 c = Q.tot[b];
      if (b < rank) { bl += c.x; br += c.y; }
      nL += c.x;
      nR += c.y;
    }
  }
  P *Lp = Lpos + lo, *Rp = Rpos + lo;
  for (int p = p0; p < p1; p += 32 * kU) {
    float v[kU];
#pragma unroll
    for (int u = 0; u < kU; u++) v[u] = p + 32 * u + lane < p1 ? ld(val + p + 32 * u + lane) : key;
#pragma unroll
    for (int u = 0; u < kU; u++) {
      const int q = p + 32 * u + lane;
      const bool l = q < p1 && !(v[u] > key), r = q < p1 && !(v[u] < key);
      const unsigned ml = __ballot_sync(0xffffffffu, l), mr = __ballot_sync(0xffffffffu, r);
      if (l) Lp[bl + __popc(ml & lt)] = (P)q;
      if (r) Rp[nR - 1 - (br + __popc(mr & lt))] = (P)q;
      bl += __popc(ml);
      br += __popc(mr);
    }
  }
  if (kCl) cluster.sync();
  else __syncthreads();
  const int lim = min(nL, nR), step = 32 * nw;
  int c = 0;
  for (int k0 = 32 * gw + lane; k0 < lim; k0 += kU * step) {
    int a[kU], b[kU], oa[kU], ob[kU];
    float va[kU], vb[kU];
#pragma unroll
    for (int u = 0; u < kU; u++) {
      const int k = k0 + u * step;
      a[u] = k < lim ? (int)ld(Lp + k) : 1;
      b[u] = k < lim ? (int)ld(Rp + k) : 0;
    }
#pragma unroll
    for (int u = 0; u < kU; u++)
      if (a[u] < b[u]) {
        va[u] = ld(val + a[u]); vb[u] = ld(val + b[u]);
        oa[u] = ld(ord + a[u]); ob[u] = ld(ord + b[u]);
      }
#pragma unroll
    for (int u = 0; u < kU; u++)
      if (a[u] < b[u]) {
        val[a[u]] = vb[u]; val[b[u]] = va[u];
        ord[a[u]] = ob[u]; ord[b[u]] = oa[u];
        c++;
      }
  }
  c = __reduce_add_sync(0xffffffffu, c);
  if (lane == 0) Q.wk[warp] = c;
  __syncthreads();
  int K = 0;
  for (int w = 0; w < kResWarps; w++) K += Q.wk[w];
  if (kCl) {
    if (threadIdx.x < blocks) cluster.map_shared_rank(&Q, threadIdx.x)->ktot[rank] = K;
    cluster.sync();
    K = 0;
    for (int b = 0; b < blocks; b++) K += Q.ktot[b];
  }
  if (K == 0) return make_int2((int)ld(Lp), (int)ld(Rp));
  const int lk = (int)ld(Lp + K - 1), rk = (int)ld(Rp + K - 1);
  return make_int2(K < nL ? min((int)ld(Lp + K), rk) : rk, K < nR ? max((int)ld(Rp + K), lk) : lk);
}

// the same of shared memory by one warp
__device__ __forceinline__ int2 quick_warp_partition(QuickSmem &Q, int lo, int hi) {
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  const float key = Q.a[(lo + hi) / 2];
  uint16_t *Lp = Q.Lp + lo, *Rp = Q.Rp + lo;
  int nL = 0, nR = 0;
  for (int base = lo; base <= hi; base += 32) {
    const int p = base + lane;
    const bool f = p <= hi && !(Q.a[min(p, hi)] > key);
    const unsigned bal = __ballot_sync(0xffffffffu, f);
    if (f) Lp[nL + __popc(bal & lt)] = (uint16_t)p;
    nL += __popc(bal);
  }
  for (int top = hi; top >= lo; top -= 32) {
    const int p = top - lane;
    const bool f = p >= lo && !(Q.a[max(p, lo)] < key);
    const unsigned bal = __ballot_sync(0xffffffffu, f);
    if (f) Rp[nR + __popc(bal & lt)] = (uint16_t)p;
    nR += __popc(bal);
  }
  __syncwarp();
  const int lim = min(nL, nR);
  int K = 0;
  for (int k0 = 0; k0 < lim; k0 += 32) {
    const int k = k0 + lane;
    const unsigned bal = __ballot_sync(0xffffffffu, k < lim && Lp[k] < Rp[k]);
    K += __popc(bal);
    if (bal != 0xffffffffu) break;
  }
  for (int k = lane; k < K; k += 32) {
    const int a = Lp[k], b = Rp[k];
    const float tv = Q.a[a]; Q.a[a] = Q.a[b]; Q.a[b] = tv;
    const int to = Q.o[a]; Q.o[a] = Q.o[b]; Q.o[b] = to;
  }
  __syncwarp();
  int2 ij;
  if (K == 0) ij = make_int2(Lp[0], Rp[0]);
  else
    ij = make_int2(K < nL ? min((int)Lp[K], (int)Rp[K - 1]) : (int)Rp[K - 1],
                   K < nR ? max((int)Rp[K], (int)Lp[K - 1]) : (int)Lp[K - 1]);
  __syncwarp();
  return ij;
}

// the reference's recursive quicksort, one thread, segment of <= kTiny elements
__device__ __forceinline__ void thread_qsort(float *a, int *ord, int lo0, int hi0) {
  int st[2 * 16];
  int sp = 0;
  st[sp++] = lo0; st[sp++] = hi0;
  while (sp > 0) {
    const int last = st[--sp], first = st[--sp];
    int i = first, j = last;
    const float key = a[(first + last) / 2];
    for (;;) {
      while (a[i] > key) i++;
      while (a[j] < key) j--;
      if (i >= j) break;
      const float tv = a[i]; a[i] = a[j]; a[j] = tv;
      const int to = ord[i]; ord[i] = ord[j]; ord[j] = to;
      i++; j--;
    }
    const bool l = first < i - 1, r = last > j + 1;
    // larger half first so the smaller is popped next: depth <= log2(kTiny) + 1
    if (l && r) {
      if (i - 1 - first > last - j - 1) { st[sp++] = first; st[sp++] = i - 1; st[sp++] = j + 1; st[sp++] = last; }
      else { st[sp++] = j + 1; st[sp++] = last; st[sp++] = first; st[sp++] = i - 1; }
    } else if (l) { st[sp++] = first; st[sp++] = i - 1; }
    else if (r) { st[sp++] = j + 1; st[sp++] = last; }
    if (sp > 2 * 16 - 4) break;   // unreachable for kTiny = 32
  }
}

// per warp: queue a tiny segment; 32 queued ones are sorted at once, a lane each.
// Every lane reads the count before lane 0 changes it (the __syncwarp after the read).
__device__ __forceinline__ void quick_tiny(QuickSmem &Q, int2 seg) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int cnt = Q.tiny_n[warp];
  __syncwarp();
  if (cnt == 32) {
    const int2 t = Q.tiny[warp][lane];
    thread_qsort(Q.a, Q.o, t.x, t.y);
    __syncwarp();
    cnt = 0;
  }
  if (lane == 0) {
    Q.tiny[warp][cnt] = seg;
    Q.tiny_n[warp] = cnt + 1;
  }
  __syncwarp();
}

// A segment of <= kQuickSmall elements, by one block in shared memory.  places: only the places of the runs' boxes are
// written (S.place), not their order (what of it no run asked for is not complete)
__device__ __forceinline__ void quick_small(cg::cluster_group &cluster, QuickSmem &Q, const SortRuns &runs, const Slots &S,
                                            int base, int hi, bool places, int *err) {
  auto none = [](int2) {};
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, len = hi - base + 1;
  for (int i = threadIdx.x; i < len; i += kResNT) {
    Q.a[i] = __ldcg(S.qv + base + i);
    Q.o[i] = __ldcg(S.qo + base + i);
  }
  if (lane == 0) Q.tiny_n[warp] = 0;
  if (threadIdx.x == 0) {
    Q.ns = Q.wl_n = Q.wl_next = 0;
    if (len > kQuickWarp) Q.sstk[Q.ns++] = make_int2(0, len - 1);
    else Q.wl[Q.wl_n++] = make_int2(0, len - 1);
  }
  __syncthreads();
  for (;;) {
    while (Q.ns > 0 && Q.wl_n <= kQuickWarpList - 2) {
      const int2 seg = Q.sstk[Q.ns - 1];
      __syncthreads();   // everyone has read the top entry
      const int2 ij = quick_partition<false>(cluster, Q, Q.a, Q.o, Q.Lp, Q.Rp, seg.x, seg.y);
      if (threadIdx.x == 0) {
        Q.ns--;
        quick_children(runs, base, seg.x, seg.y, ij.x, ij.y, [&](int2 c) {
          if (c.y - c.x >= kQuickWarp) {
            if (Q.ns < 16) Q.sstk[Q.ns++] = c;
            else atomicOr(err, 2048);   // impossible: depth <= log2(kQuickSmall / kQuickWarp) + 1
          } else {
            Q.wl[Q.wl_n++] = c;
          }
        }, none);
      }
      __syncthreads();
    }
    // the queued segments by a warp each, depth first
    for (;;) {
      int k = 0;
      if (lane == 0) k = atomicAdd(&Q.wl_next, 1);
      k = __shfl_sync(0xffffffffu, k, 0);
      if (k >= Q.wl_n) break;
      int2 stk[16];
      int sp = 0;
      stk[sp++] = Q.wl[k];
      while (sp > 0) {
        const int2 seg = stk[--sp];
        if (seg.y - seg.x < kTiny) {
          quick_tiny(Q, seg);
          continue;
        }
        const int2 ij = quick_warp_partition(Q, seg.x, seg.y);
        quick_children(runs, base, seg.x, seg.y, ij.x, ij.y, [&](int2 c) {
          if (c.y - c.x < kTiny) quick_tiny(Q, c);
          else if (sp < 16) stk[sp++] = c;
          else if (lane == 0) atomicOr(err, 4096);   // impossible: depth <= log2(kQuickWarp / kTiny) + 1
        }, none);
      }
    }
    __syncthreads();
    if (threadIdx.x == 0) Q.wl_n = Q.wl_next = 0;
    __syncthreads();
    if (Q.ns == 0) break;
  }
  if (lane < Q.tiny_n[warp]) {
    const int2 t = Q.tiny[warp][lane];
    thread_qsort(Q.a, Q.o, t.x, t.y);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < len; i += kResNT) {
    if (places) {
      if (quick_wanted(runs, base + i, base + i)) S.place[Q.o[i]] = base + i;
    } else {
      S.qv[base + i] = Q.a[i];
      S.qo[base + i] = Q.o[i];
    }
  }
  __syncthreads();
}

// The places of the runs' boxes (`runs` the same in every block) in the order that the reference's quicksort leaves them
// in, into S.place by box.  split: all boxes; only the segments above kQuickMid are partitioned, the others are left in
// S.Lpos (S.st->n_mid).  What has been partitioned stays so for the next call.
// Collective over the cluster; the blocks' writes are visible to one another on return.
__device__ __noinline__ void quick_sort(QuickSmem &Q, const SortRuns &runs, const Slots &S, bool split, int *err) {
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank(), blocks = (int)cluster.num_blocks(), D = S.st->D, had = __ldcg(&S.st->n_left);
  __syncthreads();   // Q may have been in other use
  if (had == 0) {
    for (int i0 = rank * kResNT + threadIdx.x, step = blocks * kResNT; i0 < D; i0 += 8 * step) {
      float v[8];
#pragma unroll
      for (int u = 0; u < 8; u++) v[u] = i0 + u * step < D ? S.score[i0 + u * step] : 0.0f;
#pragma unroll
      for (int u = 0; u < 8; u++)
        if (i0 + u * step < D) {
          S.qv[i0 + u * step] = v[u];
          S.qo[i0 + u * step] = i0 + u * step;
        }
    }
    if (threadIdx.x == 0) Q.left[0] = make_int2(0, D - 1);
  }
  if (had > 0 && !split)   // elements that an earlier call has put in their places (the others' are written below)
    for (int k = 0; k < runs.n; k++)
      for (int p = runs.r[k].x + rank * kResNT + threadIdx.x; p <= runs.r[k].y; p += blocks * kResNT)
        S.place[__ldcg(S.qo + p)] = p;
  for (int k = threadIdx.x; k < had; k += kResNT) Q.left[k] = __ldcg(reinterpret_cast<const int2 *>(S.hist) + k);
  const int limit = split ? kQuickMid : kQuickSmall, nleft = max(had, 1);
  // by thread 0:
  auto push = [&](int2 c) {
    if (c.y - c.x >= limit) {
      if (Q.nst < 40) Q.stk[Q.nst++] = c;
      else atomicOr(err, 256);   // impossible: depth <= log2(D) + 1
    } else if (!split) {
      Q.list[Q.nl++] = c;
    } else if (rank == 0) {
      reinterpret_cast<int2 *>(S.Lpos)[Q.nl++] = c;   // (disjoint segments of two elements or more: they fit)
    }
  };
  auto keep = [&](int2 c) {
    if (Q.nleft < kQuickLeft) Q.left[Q.nleft] = c;
    Q.nleft++;
  };
  auto alone = [&](int p) {   // an element in its place
    if (!split && quick_wanted(runs, p, p)) S.place[__ldcg(S.qo + p)] = p;
  };
  if (threadIdx.x == 0) {
    Q.nst = Q.nl = 0;
    Q.nleft = nleft;
  }
  cluster.sync();
  // every block alike: the segments kept so far, one after the other; at the end the small ones that wait
  for (int e = 0; e <= nleft; e++) {
    if (e < nleft) {
      const int2 kept = Q.left[e];
      if (kept.x >= kept.y || !quick_wanted(runs, kept.x, kept.y)) continue;
      __syncthreads();
      if (threadIdx.x == 0) {
        Q.left[e] = make_int2(0, 0);
        push(kept);
      }
      __syncthreads();
    }
    while (Q.nst > 0 || (!split && Q.nl > (e == nleft ? 0 : kQuickList - 2))) {
      if (Q.nst > 0 && (split || Q.nl <= kQuickList - 2)) {
        const int2 seg = Q.stk[Q.nst - 1];
        __syncthreads();   // everyone has read the top entry
        const int2 ij = quick_partition<true>(cluster, Q, S.qv, S.qo, S.qL, S.qR, seg.x, seg.y);
        if (threadIdx.x == 0) {
          Q.nst--;
          quick_children(runs, 0, seg.x, seg.y, ij.x, ij.y, push, keep);
          if (rank == 0) {
            if (seg.x == ij.x - 1) alone(seg.x);
            if (seg.y == ij.y + 1) alone(seg.y);
            if (ij.x == ij.y) alone(ij.x);
          }
        }
        __syncthreads();
      } else {
        for (int k = rank; k < Q.nl; k += blocks) quick_small(cluster, Q, runs, S, Q.list[k].x, Q.list[k].y, true, err);
        __syncthreads();
        if (threadIdx.x == 0) {
          for (int k = 0; k < Q.nl; k++) keep(Q.list[k]);
          Q.nl = 0;
        }
        __syncthreads();
      }
    }
  }
  if (rank == 0 && threadIdx.x == 0) {
    if (split) {
      S.st->n_mid = Q.nl;
    } else {   // (more than fit: the next call begins anew)
      int n = 0;
      for (int k = 0; k < min(Q.nleft, kQuickLeft); k++)
        if (Q.left[k].x < Q.left[k].y) reinterpret_cast<int2 *>(S.hist)[n++] = Q.left[k];
      S.st->n_left = Q.nleft <= kQuickLeft ? n : 0;
    }
  }
  cluster.sync();
}

}  // namespace geye
