// dt.cu -- generalized distance transform with argmax displacements.
//
// Reference: CAR_TRACKING/dt.cpp:61-136.  dt_helper is a divide-and-conquer
// monotone argmin: for the middle d of [d1, d2] it scans s in [s1, s2]
// keeping the leftmost minimum of
//     f_d(s) = (v[s] + (a*t)*t) + b*t,  t = d - s   (float, no FMA)
// and recurses on [d1, d-1] x [s1, s*] and [d+1, d2] x [s*, s2].
//
// GPU form.  Let g(d) be the leftmost global argmin of f_d over the whole
// line.  If g is non-decreasing in d, the recursion returns g(d) for every d
// (each node's range [s1, s2] then contains g(d), and no smaller index in it
// reaches the minimum).  So every output of a line is computed in parallel.
// Where dt_monotone proves from the line's value range and (a, b) that the
// computed g cannot decrease (the usual case: a >= 8 times the rounding bound),
// nothing else is needed, and pass 2 computes only the entries it stores;
// otherwise g is checked to be non-decreasing, and only if it is not does one
// thread replay the recursion exactly (counted in *fallback_count).
//
// g(d) is searched in a window |d - s| < K.  K is chosen so that every s
// outside the window has f_d(s) > max(v) >= f_d(d): with u = 2^-24,
// f_d(s) >= v_min + (1-8u) a t^2 - (1+8u)|b t| - 8u max|v| for a > 0, and K
// is the first integer past the positive root of that bound minus v_max.
// For a <= 0 the window is the whole line.
//
// Strips (k_dt_strip), where the order is proven and K <= kDtEdge in both directions:
//   k_dt_range finds a map's value range; a block takes a strip of 8 to 64 of its rows through both passes.
//   Pass 1 stages columns of the strip with K - 1 rows above and below (+inf outside the map: such a candidate
//   never wins a strict comparison) and leaves the strip's values and displacements in shared memory; its
//   windows come from the whole map's range, so every strip of a map takes them alike.  Pass 2 walks
//   along x there, windows from the strip's own range, a lane per row: consecutive rows are consecutive
//   words, and a row computes only the entries that are stored of it.  The per-offset terms
//   (a*t)*t and b*t are in registers, with the same roundings as dt_f.
// General form (dt_tile), for the others: tiles of L lines (about kDtTile outputs) of one pass; windows per tile in
//   pass 1 and per line in pass 2.  The strips share out the columns, k_dt_rest takes the rows.
//
// What bounds the strips is issue (69 % of it, 120 instructions an element of which 45 are the candidates of
// pass 1, 2K - 1 = 5 to 11 of them at five instructions).  Both passes as kernels of tiles, with the values and indices
// between them through memory: 270 instructions an element in pass 1 and 2 each.  DT stage, car+person: 640x480 98 -> 59 us,
// 1280x720 254 -> 131, 1920x1080 555 -> 272; trained-like 1280x720 160 -> 102.  dt() of 151x111: 76 -> 72 us.
#include <math.h>

#include <algorithm>

#include "internal.h"

namespace geye {

constexpr int kDtThreads = 256;
// kDtElems (outputs per block, about) is in internal.h: plans tune it
constexpr int kDtPad = 64;          // largest window half-width served by the general form's unchecked loop
constexpr int kDtTile = 512;       // outputs per tile of the general form, about
constexpr int kDtEdge = 16;         // largest window half-width of the strips
constexpr int kDtStage = 2048;      // values of a strip staged at a time
constexpr int kDtChunk = 8192;      // values per block of k_dt_range
constexpr int kDtParts = 152;       // blocks in the general form, at least
constexpr int kDtOwnRange = 32768;  // a lone map's strips read the range of up to so many values themselves (a launch less)

// e / n by mg = dt_magic(n), for e < 2^32 / n
__device__ __forceinline__ unsigned dt_magic(int n) { return 0xFFFFFFFFu / (unsigned)n + 1u; }
__device__ __forceinline__ int dt_div(int e, unsigned mg) { return mg ? (int)__umulhi((unsigned)e, mg) : e; }   // (0: n = 1)

__device__ __forceinline__ float dt_f(float v, float a, float b, int t) {
  return v + a * t * t + b * t;      // ((v + (a*t)*t) + b*t), each op rounded (no FMA)
}

// window half-width bound K for one line (a > 0); returns n when unbounded.
// Float arithmetic (the FP64 pipe is narrow on this GPU): A and B are pushed
// down and up by 2^-18 and the root up by 2^-16, far more than the few
// 2^-24 roundings of the expression, so K never falls below the exact bound.
__device__ __forceinline__ int dt_window(float vmin, float vmax, float vabs, float a, float b, int n) {
  if (!(a > 0.f)) return n;
  const float u = 8.0f * 5.9604644775390625e-08f;   // 8 * 2^-24
  const float lo = 1.0f - 3.814697265625e-06f;      // 1 - 2^-18
  const float hi = 1.0f + 3.814697265625e-06f;      // 1 + 2^-18
  const float A = (1.0f - u) * a * lo;
  const float B = (1.0f + u) * fabsf(b) * hi;
  const float R = ((vmax - vmin) * hi + u * vabs * hi) * hi + 1e-30f;
  const float root = (B + sqrtf(B * B * hi + 4.0f * A * R * hi)) / (2.0f * A) * (1.0f + 1.52587890625e-05f);
  if (!(root < (float)n)) return n;
  return (int)floorf(root) + 2;
}

// Exact replay of dt_helper for one line (one thread).
__device__ void dt_replay(const float *v, int n, float a, float b, float *out, int *arg) {
  int st[4 * 64];
  int sp = 0;
  st[sp++] = 0; st[sp++] = n - 1; st[sp++] = 0; st[sp++] = n - 1;
  while (sp > 0) {
    const int d2 = st[--sp], d1 = st[--sp], s2 = st[--sp], s1 = st[--sp];
    if (d2 < d1) continue;
    const int d = (d1 + d2) >> 1;
    int s = s1;
    float src_ss = v[s];
    for (int p = s1 + 1; p <= s2; p++) {
      int t1 = d - s, t2 = d - p;
      if (src_ss + a * t1 * t1 + b * t1 > v[p] + a * t2 * t2 + b * t2) {
        s = p;
        src_ss = v[s];
      }
    }
    const int D = d - s;
    out[d] = v[s] + a * D * D + b * D;
    arg[d] = s;
    if (sp + 8 <= 4 * 64) {
      st[sp++] = s; st[sp++] = s2; st[sp++] = d + 1; st[sp++] = d2;
      st[sp++] = s1; st[sp++] = s; st[sp++] = d1; st[sp++] = d - 1;
    }
  }
}

// lines per block: pass 1 (columns, contiguous) any count up to 64; pass 2
// (rows, strided in memory) a power of two up to 16 so that staging is coalesced
__host__ __device__ __forceinline__ int dt_lines1(int n, int elems) { return max(1, min(64, elems / max(n, 1))); }
__host__ __device__ __forceinline__ int dt_lg_lines2(int n, int elems) {
  int lg = 0;
  while (lg < 4 && (2 << lg) * n <= elems) lg++;
  return lg;
}
__host__ __device__ __forceinline__ size_t dt_smem_bytes(int L, int n) {
  return sizeof(float) * ((size_t)kDtPad + (size_t)L * (n + kDtPad) + 2 * (size_t)L * n + 2 * (2 * kDtPad - 1)) +
         sizeof(int) * (2 * (size_t)L + 1) + sizeof(float) * 3 * (kDtThreads / 32) + sizeof(int);
}

// Leftmost minimum of output d over the window |t| < KM of a padded line,
// unrolled; At/Bt: (a*t)*t and b*t tabulated in shared memory (broadcast
// reads).  KM may exceed the line's own K: candidates past K lose to f_d(d)
// anyway, so a wider window returns the same leftmost minimum.
template <int KM>
__device__ __forceinline__ int dt_scan_fixed(const float *__restrict__ line, int d, const float *__restrict__ At,
                                             const float *__restrict__ Bt, float &best) {
  const float *v = line + d - (KM - 1);   // v[i] = line[d - t], t = KM-1-i: p ascending
  best = INFINITY;
  int s = -1;
#pragma unroll
  for (int i = 0; i < 2 * KM - 1; i++) {
    const float f = (v[i] + At[KM - 1 - i]) + Bt[KM - 1 - i];
    if (f < best) { best = f; s = i; }
  }
  return s < 0 ? -1 : d - (KM - 1) + s;
}

// Leftmost minimum of output d over its line's window (K rounded up to an
// unrolled size, a loop beyond 16, a bounds-checked loop past the padding).
__device__ __forceinline__ int dt_full(const float *__restrict__ line, int d, int K, int n, float a, float b,
                                       const float *__restrict__ At, const float *__restrict__ Bt, float &best) {
  int p;
  if (K <= 3) p = dt_scan_fixed<3>(line, d, At, Bt, best);
  else if (K <= 4) p = dt_scan_fixed<4>(line, d, At, Bt, best);
  else if (K <= 5) p = dt_scan_fixed<5>(line, d, At, Bt, best);
  else if (K <= 6) p = dt_scan_fixed<6>(line, d, At, Bt, best);
  else if (K <= 8) p = dt_scan_fixed<8>(line, d, At, Bt, best);
  else if (K <= 12) p = dt_scan_fixed<12>(line, d, At, Bt, best);
  else if (K <= 16) p = dt_scan_fixed<16>(line, d, At, Bt, best);
  else if (K <= kDtPad) {
    best = INFINITY;
    p = -1;
    for (int t = K - 1; t > -K; t--) {   // p = d - t ascending
      const float f = (line[d - t] + At[t]) + Bt[t];
      if (f < best) { best = f; p = d - t; }
    }
  } else {
    const int lo = max(0, d - K + 1), hi = min(n - 1, d + K - 1);
    p = lo;
    best = dt_f(line[lo], a, b, d - lo);
    for (int q = lo + 1; q <= hi; q++) {
      const float fq = dt_f(line[q], a, b, d - q);
      if (best > fq) { best = fq; p = q; }
    }
  }
  if (p < 0) {   // every candidate was NaN: the reference keeps the window's first index
    p = max(0, d - K + 1);
    best = dt_f(line[p], a, b, d - p);
  }
  return p;
}

// Every output of the tile, spread over all threads (e -> line e / n, the division by a precomputed reciprocal), each
// with its own line's window.
__device__ __forceinline__ void dt_scan_tile(const float *__restrict__ v_s, int stride, int n, int nl, float a,
                                             float b, const int *__restrict__ K_s, const float *__restrict__ At,
                                             const float *__restrict__ Bt, float *__restrict__ o_s,
                                             int *__restrict__ g_s) {
  const unsigned mg = dt_magic(n);
  for (int e = threadIdx.x; e < nl * n; e += blockDim.x) {
    const int l = dt_div(e, mg), d = e - l * n;
    float best;
    const int p = dt_full(v_s + l * stride, d, K_s[l], n, a, b, At, Bt, best);
    o_s[e] = best;
    g_s[e] = p;
  }
}

// True when the computed leftmost argmin g(d) of a line is certainly
// non-decreasing in d.  For s < p, the exact terms give
//   [f_d(s) - f_d(p)] - [f_{d-1}(s) - f_{d-1}(p)] = 2a(p - s) >= 2a,
// and each computed f (four roundings, no FMA) is within
// E = 4u(|v| + a t^2 + |b t|) of the exact one (u = 2^-24, |t| <= K for the
// argmins of d and d - 1, which lie in their windows).  g(d) < g(d-1) needs
// the computed bracket below zero, so 2a > 4E; a >= 8E rules it out with a
// factor 4 to spare (the 1e-37 covers subnormal roundings).  NaN or infinite
// values, a <= 0 and windows past the padding fail the test.
__device__ __forceinline__ bool dt_monotone(float vabs, float a, float b, int K) {
  if (!(a > 0.f) || K > kDtPad - 2 || !(vabs <= 3.0e38f)) return false;
  const float T = (float)(K + 1);
  const float E = 4.0f * 5.9604644775390625e-08f * (vabs + a * T * T + fabsf(b) * T) + 1e-37f;
  return a >= 8.0f * E;
}

// The general form: lines [line0, line_end) at most of a map, a tile of them, by one block.
// PASS 1: along y (dim 0) of each column x of the negated part map -> tmpM, tmpI.
// PASS 2: along x (dim 1) of each row y of tmpM -> M, Ix, Iy = tmpIy[Ix*d0 + y]
// (dt.cpp:123-133).
template <int PASS>
__device__ __noinline__ void dt_tile(const DtJob &J, int line0, int line_end, float *__restrict__ arena,
                                    int *__restrict__ arena_i, int *fallback_count, float *dsm) {
  const int d0 = J.d0;
  const int n = PASS == 1 ? J.d0 : J.d1;           // line length
  const int lgL = PASS == 1 ? 0 : dt_lg_lines2(n, kDtTile);
  const int L = PASS == 1 ? dt_lines1(n, kDtTile) : (1 << lgL);
  const int nl = min(L, line_end - line0);
  const int stride = n + kDtPad;
  __syncthreads();   // the last tile's shared memory is free
  float *v_s = dsm + kDtPad;                       // line l at v_s[l * stride], +inf pads between
  float *o_s = dsm + kDtPad + (size_t)L * stride;  // [L][n]
  int *g_s = reinterpret_cast<int *>(o_s + (size_t)L * n);
  float *At = reinterpret_cast<float *>(g_s + (size_t)L * n) + (kDtPad - 1);   // At[t], |t| < kDtPad
  float *Bt = At + (2 * kDtPad - 1);
  int *K_s = reinterpret_cast<int *>(Bt + kDtPad);
  int *bad_s = K_s + L;
  int *mono_s = bad_s + L;   // every line's argmin certainly non-decreasing
  const float a = PASS == 1 ? J.ay : J.ax, b = PASS == 1 ? J.by : J.bx;
  const int tid = threadIdx.x, nth = blockDim.x;
  const int cnt = nl * n;
  const unsigned magic = dt_magic(n);

  // stage the tile (pass 1: with each thread's value range), the pads and the per-offset terms
  float vmin = INFINITY, vmax = -INFINITY, vabs = 0.f;
  bool nan = false;   // fminf/fmaxf skip NaN
  if (PASS == 1) {
    const float *src = arena + J.in_off + (size_t)line0 * n;
    for (int e = tid; e < cnt; e += nth) {
      const int l = dt_div(e, magic), d = e - l * n;
      const float x = J.negate ? -src[e] : src[e];   // inverse_Q (GPU_function.cu:695-794)
      v_s[l * stride + d] = x;
      vmin = fminf(vmin, x); vmax = fmaxf(vmax, x); vabs = fmaxf(vabs, fabsf(x)); nan |= x != x;
    }
  } else {
    const float *tm = arena + J.tmpM_off;
    for (int e = tid; e < (n << lgL); e += nth) {
      const int l = e & (L - 1), x = e >> lgL;
      if (l < nl) {
        v_s[l * stride + x] = tm[(size_t)x * d0 + line0 + l];
      }
    }
  }
  for (int i = tid; i < (nl + 1) * kDtPad; i += nth) {
    const int l = i / kDtPad, k = i - l * kDtPad;
    v_s[l * stride - kDtPad + k] = INFINITY;   // pad before line l (l = nl: after the last line)
  }
  if (tid == 0) *mono_s = 1;
  for (int t = tid - (kDtPad - 1); t < kDtPad; t += nth) {
    const float ft = (float)t;
    At[t] = a * ft * ft;
    Bt[t] = b * ft;
  }
  __syncthreads();

  // window bounds.  Pass 1 (many short lines per tile): one bound for the
  // whole tile, from the tile's value range (a wider window than a line's own
  // returns the same leftmost minimum, and the order proof only gets more
  // conservative).  Pass 2 (a few long lines): a bound per line, each line's
  // range reduced by a warp.
  const int lane = tid & 31, warp = tid >> 5;
  int K = 0;
  if (PASS == 1) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      vmin = fminf(vmin, __shfl_xor_sync(0xffffffffu, vmin, o));
      vmax = fmaxf(vmax, __shfl_xor_sync(0xffffffffu, vmax, o));
      vabs = fmaxf(vabs, __shfl_xor_sync(0xffffffffu, vabs, o));
    }
    nan = __any_sync(0xffffffffu, nan);
    float *red = reinterpret_cast<float *>(mono_s + 1);   // [3][warps]: the warps' min, max, max |x| (-1: NaN)
    if (lane == 0) {
      red[warp] = vmin;
      red[kDtThreads / 32 + warp] = vmax;
      red[2 * (kDtThreads / 32) + warp] = nan ? -1.0f : vabs;
    }
    __syncthreads();
    float mn = INFINITY, mx = -INFINITY, ab = 0.f;
    bool tile_nan = false;
    for (int w = 0; w < (nth >> 5); w++) {
      mn = fminf(mn, red[w]);
      mx = fmaxf(mx, red[kDtThreads / 32 + w]);
      const float aw = red[2 * (kDtThreads / 32) + w];
      tile_nan |= aw < 0.f;
      ab = fmaxf(ab, aw);
    }
    K = dt_window(mn, mx, ab, a, b, n);
    if (tid == 0 && (tile_nan || !dt_monotone(ab, a, b, K))) *mono_s = 0;
    for (int l = tid; l < nl; l += nth) {
      K_s[l] = K;
      bad_s[l] = 0;
    }
  } else {
    for (int l = warp; l < nl; l += nth >> 5) {
      const float *v = v_s + l * stride;
      float lmin = INFINITY, lmax = -INFINITY, labs = 0.f;
      bool lnan = false;
      for (int i = lane; i < n; i += 32) {
        const float x = v[i];
        lmin = fminf(lmin, x);
        lmax = fmaxf(lmax, x);
        labs = fmaxf(labs, fabsf(x));
        lnan |= x != x;
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        lmin = fminf(lmin, __shfl_xor_sync(0xffffffffu, lmin, o));
        lmax = fmaxf(lmax, __shfl_xor_sync(0xffffffffu, lmax, o));
        labs = fmaxf(labs, __shfl_xor_sync(0xffffffffu, labs, o));
      }
      lnan = __any_sync(0xffffffffu, lnan);
      if (lane == 0) {
        const int Kl = dt_window(lmin, lmax, labs, a, b, n);
        K_s[l] = Kl;
        bad_s[l] = 0;
        if (lnan || !dt_monotone(labs, a, b, Kl)) *mono_s = 0;
      }
    }
  }
  __syncthreads();

  if (*mono_s) {   // the order holds: no check, no replay
    dt_scan_tile(v_s, stride, n, nl, a, b, K_s, At, Bt, o_s, g_s);
    __syncthreads();   // every output of the tile written before the stores read them
  } else {
    // every output's window, then the order check and the exact replay
    dt_scan_tile(v_s, stride, n, nl, a, b, K_s, At, Bt, o_s, g_s);
    __syncthreads();
    for (int e = tid; e < cnt; e += nth) {
      const int l = dt_div(e, magic), d = e - l * n;
      if (d + 1 < n && g_s[e] > g_s[e + 1]) bad_s[l] = 1;
    }
    __syncthreads();
    for (int l = tid; l < nl; l += nth)
      if (bad_s[l]) {
        dt_replay(v_s + l * stride, n, a, b, o_s + (size_t)l * n, g_s + (size_t)l * n);
        atomicAdd(fallback_count, 1);
      }
    __syncthreads();
  }

  if (PASS == 1) {
    float *tm = arena + J.tmpM_off + (size_t)line0 * n;
    int *ti = arena_i + J.tmpI_off + (size_t)line0 * n;
    for (int e = tid; e < cnt; e += nth) {
      tm[e] = o_s[e];
      ti[e] = g_s[e];
    }
  } else {
    float *M = arena + J.M_off;
    int *Ix = arena_i + J.Ix_off;
    int *Iy = arena_i + J.Iy_off;
    const int *tIy = arena_i + J.tmpI_off;
    for (int e = tid; e < (n << lgL); e += nth) {
      const int l = e & (L - 1), x = e >> lgL;
      if (l >= nl) continue;
      const int y = line0 + l;
      const bool mpos = (y & 1) == J.par_y && (x & 1) == J.par_x;
      const bool ipos = (y & 1) != J.par_y && (x & 1) != J.par_x;
      const bool wm = !J.samp_m || mpos, wi = !J.samp_i || ipos;
      const size_t o = (size_t)x * d0 + y;
      const int ix = g_s[l * n + x];
      if (wm) M[J.cm0 ? (size_t)((x - J.par_x) >> 1) * J.cm0 + ((y - J.par_y) >> 1) : o] = o_s[l * n + x];
      if (wi) {
        const size_t oi = J.ci0 ? (size_t)((x - 1 + J.par_x) >> 1) * J.ci0 + ((y - 1 + J.par_y) >> 1) : o;
        Ix[oi] = ix;
        Iy[oi] = tIy[(size_t)ix * d0 + y];
      }
    }
  }
}

// ---------------------------------------------------------------------------
// strips
// ---------------------------------------------------------------------------
struct DtRange {
  float lo, hi;
  bool nan;   // (fminf and fmaxf skip it)
  __device__ __forceinline__ void take(float x) {
    lo = fminf(lo, x);
    hi = fmaxf(hi, x);
    nan |= x != x;
  }
};

// The range of the block's threads' values, in every thread; red: three floats a warp
__device__ __forceinline__ DtRange dt_block_range(DtRange r, float (*red)[kDtThreads / 32]) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    r.lo = fminf(r.lo, __shfl_xor_sync(0xffffffffu, r.lo, o));
    r.hi = fmaxf(r.hi, __shfl_xor_sync(0xffffffffu, r.hi, o));
  }
  r.nan = __any_sync(0xffffffffu, r.nan);
  __syncthreads();   // red is free
  if ((threadIdx.x & 31) == 0) {
    red[0][threadIdx.x >> 5] = r.lo;
    red[1][threadIdx.x >> 5] = r.hi;
    red[2][threadIdx.x >> 5] = r.nan ? 1.0f : 0.0f;
  }
  __syncthreads();
#pragma unroll
  for (int w = 0; w < kDtThreads / 32; w++) {
    r.lo = fminf(r.lo, red[0][w]);
    r.hi = fmaxf(r.hi, red[1][w]);
    r.nan |= red[2][w] != 0.0f;
  }
  return r;
}

// The range of values [first, first + n) of a map, this thread's part
__device__ __forceinline__ DtRange dt_values_range(const float *src, int n) {
  DtRange r{INFINITY, -INFINITY, false};
  const int head = min(n, (int)((0u - (unsigned)(reinterpret_cast<uintptr_t>(src) >> 2)) & 3u)), quads = (n - head) >> 2;
  const float4 *q = reinterpret_cast<const float4 *>(src + head);   // (16-byte loads)
#pragma unroll 4
  for (int e = threadIdx.x; e < quads; e += kDtThreads) {
    const float4 v = q[e];
    r.take(v.x); r.take(v.y); r.take(v.z); r.take(v.w);
  }
  const int left = n - 4 * quads;   // the values before and behind them
  if ((int)threadIdx.x < left) r.take(src[(int)threadIdx.x < head ? threadIdx.x : 4 * quads + threadIdx.x]);
  return r;
}

__global__ void __launch_bounds__(kDtThreads) k_dt_range(const DtJob *__restrict__ jobs, const int2 *__restrict__ chunks,
                                                         const float *__restrict__ arena, float4 *__restrict__ ranges,
                                                         int *n_rest) {
  __shared__ float red[3][kDtThreads / 32];
  const int2 blk = chunks[blockIdx.x];
  const DtJob &J = jobs[blk.x];
  if (blockIdx.x == 0 && threadIdx.x == 0) *n_rest = 0;
  const DtRange r = dt_block_range(dt_values_range(arena + J.in_off + blk.y, min(kDtChunk, J.d0 * J.d1 - blk.y)), red);
  if (threadIdx.x == 0) ranges[blockIdx.x] = make_float4(r.lo, r.hi, r.nan ? 1.0f : 0.0f, 0.0f);
}

// Rows of a strip (about 2 * elems outputs, evenly over the map)
static int dt_strip_rows(int d0, int d1, int elems) {
  const int most = std::max(8, std::min(64, 2 * elems / d1)), strips = (d0 + most - 1) / most;
  return (d0 + strips - 1) / strips;
}

// The leftmost minimum over the window |t| < KM, v[j] the value at t = KM - 1 - j (candidates in ascending order): t of it.
// A[t], B[t] = (a * t) * t and b * t for t >= 0, the roundings of dt_f; at -t they are A[t] and -B[t] exactly.
// (The least value first, three a step, then its first place: as many instructions, and slower.)
template <int KM>
__device__ __forceinline__ int dt_window_min(const float *v, const float (&A)[KM], const float (&B)[KM], float &best) {
  best = INFINITY;
  int t = 0;
#pragma unroll
  for (int j = 0; j < 2 * KM - 1; j++) {
    const int k = KM - 1 - j;
    const float f = k >= 0 ? (v[j] + A[k]) + B[k] : (v[j] + A[-k]) - B[-k];
    if (f < best) { best = f; t = k; }
  }
  return t;
}

template <int KM>
__device__ __forceinline__ void dt_terms(float a, float b, float (&A)[KM], float (&B)[KM]) {
#pragma unroll
  for (int t = 0; t < KM; t++) {
    const float ft = (float)t;
    A[t] = a * ft * ft;
    B[t] = b * ft;
  }
}

struct DtStrip {
  int y0, nr;      // its rows
  float *S;        // kDtStage values: columns with KM - 1 rows above and below the strip
  float *T;        // pass 1's values: column x at T + x * nr, kDtEdge columns of +inf before and kDtEdge + 8 behind
  int8_t *t1;      // pass 1's displacements y - Iy
};

// Pass 1 of a strip (windows of KM); the range of its values into lo, hi (this thread's)
template <int KM>
__device__ __forceinline__ void dt_strip1(const DtJob &J, const DtStrip &Z, const float *__restrict__ arena, float &lo,
                                          float &hi) {
  constexpr int H = KM - 1;
  const int d0 = J.d0, d1 = J.d1, nr = Z.nr, tid = threadIdx.x;
  const int pairs = (nr + 1) >> 1, rs = 2 * pairs + 2 * H, cols = kDtStage / rs;   // (an even number of rows staged)
  float A[KM], B[KM];
  dt_terms<KM>(J.ay, J.by, A, B);
  const float *src = arena + J.in_off;
  const bool neg = J.negate != 0;
  const unsigned mg_s = dt_magic(rs), mg_p = dt_magic(pairs);
  for (int x0 = 0; x0 < d1; x0 += cols) {
    const int nc = min(cols, d1 - x0);
    for (int e0 = tid; e0 < nc * rs; e0 += 4 * kDtThreads) {
      float v[4];
#pragma unroll
      for (int u = 0; u < 4; u++) {
        const int e = e0 + u * kDtThreads, c = dt_div(e, mg_s), y = Z.y0 - H + e - c * rs;
        v[u] = INFINITY;
        if (e < nc * rs && (unsigned)y < (unsigned)d0) {
          const float x = src[(x0 + c) * d0 + y];
          v[u] = neg ? -x : x;   // inverse_Q (GPU_function.cu:695-794)
        }
      }
#pragma unroll
      for (int u = 0; u < 4; u++)
        if (e0 + u * kDtThreads < nc * rs) Z.S[e0 + u * kDtThreads] = v[u];
    }
    __syncthreads();
    for (int e = tid; e < nc * pairs; e += kDtThreads) {   // two rows of a column
      const int c = dt_div(e, mg_p), y = 2 * (e - c * pairs);
      float v[2 * KM];
      const float2 *p = reinterpret_cast<const float2 *>(Z.S + c * rs + y);
#pragma unroll
      for (int k = 0; k < KM; k++) {
        const float2 w = p[k];
        v[2 * k] = w.x;
        v[2 * k + 1] = w.y;
      }
      float best;
      int t = dt_window_min<KM>(v, A, B, best);
      float *o = Z.T + (x0 + c) * nr + y;
      int8_t *o1 = Z.t1 + (x0 + c) * nr + y;
      o[0] = best;
      o1[0] = (int8_t)t;
      lo = fminf(lo, best);
      hi = fmaxf(hi, best);
      if (y + 1 < nr) {
        t = dt_window_min<KM>(v + 1, A, B, best);
        o[1] = best;
        o1[1] = (int8_t)t;
        lo = fminf(lo, best);
        hi = fmaxf(hi, best);
      }
    }
    __syncthreads();
  }
}

// Pass 2 of a strip: a thread walks along x on a row, kG outputs at a time.  kQ = 2: both the score sum's and the part
// boxes' reads are sampled, a row holds outputs of one of the two only, one parity class of x
template <int KM, int kQ>
__device__ __forceinline__ void dt_strip2(const DtJob &J, const DtStrip &Z, float *__restrict__ arena,
                                          int *__restrict__ arena_i) {
  constexpr int kG = KM <= 6 ? 4 : 2, W = 2 * KM - 1 + (kG - 1) * kQ;
  const int d1 = J.d1, nr = Z.nr, yl = threadIdx.x % nr, y = Z.y0 + yl;
  const int step = kDtThreads / nr, i0 = threadIdx.x / nr;
  if (i0 >= step) return;
  float A[KM], B[KM];
  dt_terms<KM>(J.ax, J.bx, A, B);
  const bool my = (y & 1) == J.par_y;
  const int c = kQ == 1 ? 0 : my ? J.par_x : 1 - J.par_x, m = (d1 - c + kQ - 1) / kQ;
  float *M = arena + J.M_off;
  int *Ix = arena_i + J.Ix_off, *Iy = arena_i + J.Iy_off;
  // kQ = 2: output i of the row's class is at place + i * pitch of its array, in either layout
  const int compact = my ? J.cm0 : J.ci0, pitch = compact ? compact : 2 * J.d0;
  const int place = compact ? (y - (my ? J.par_y : 1 - J.par_y)) >> 1 : c * J.d0 + y;
  for (int i = i0 * kG; i < m; i += step * kG) {
    float v[W];
    const float *p = Z.T + (c + kQ * i - (KM - 1)) * nr + yl;
#pragma unroll
    for (int k = 0; k < W; k++) v[k] = p[k * nr];
#pragma unroll
    for (int g = 0; g < kG; g++) {
      float best;
      const int t = dt_window_min<KM>(v + g * kQ, A, B, best);
      const int x = c + kQ * (i + g), ix = x - t;
      if (x >= d1) break;
      if (kQ == 2) {
        const int o = place + (i + g) * pitch;
        if (my) {
          M[o] = best;
        } else {
          Ix[o] = ix;
          Iy[o] = y - Z.t1[ix * nr + yl];
        }
      } else {
        const int o = x * J.d0 + y;
        const bool mx = (x & 1) == J.par_x;
        if (!J.samp_m || (my && mx)) M[J.cm0 ? ((x - J.par_x) >> 1) * J.cm0 + ((y - J.par_y) >> 1) : o] = best;
        if (!J.samp_i || (!my && !mx)) {
          const int oi = J.ci0 ? ((x - 1 + J.par_x) >> 1) * J.ci0 + ((y - 1 + J.par_y) >> 1) : o;
          Ix[oi] = ix;
          Iy[oi] = y - Z.t1[ix * nr + yl];
        }
      }
    }
  }
}

// One strip of rows of a map, both passes; see the top of the file.
__global__ void __launch_bounds__(kDtThreads, 4) k_dt_strip(const DtJob *__restrict__ jobs, const int2 *__restrict__ blocks,
                                                            const float4 *__restrict__ ranges, int *n_rest, int4 *rest,
                                                            float *__restrict__ arena, int *__restrict__ arena_i,
                                                            int *fallback_count, int n_strips) {
  extern __shared__ float dsm[];
  __shared__ float red[3][kDtThreads / 32];
  // (the blocks behind the strips are a lone map's)
  const int2 blk = (int)blockIdx.x < n_strips ? blocks[blockIdx.x] : make_int2(0, blockIdx.x * jobs[0].rows);
  const DtJob &J = jobs[blk.x];
  const int d0 = J.d0, d1 = J.d1, tid = threadIdx.x;
  DtStrip Z;
  Z.y0 = blk.y;
  const int nr = Z.nr = min(J.rows, d0 - blk.y);
  Z.S = dsm;
  Z.T = dsm + kDtStage + kDtEdge * nr;
  Z.t1 = reinterpret_cast<int8_t *>(Z.T + (d1 + kDtEdge + 8) * nr);
  DtRange r{INFINITY, -INFINITY, false};
  if (J.n_rng == 0) r = dt_block_range(dt_values_range(arena + J.in_off, d0 * d1), red);
  for (int k = 0; k < J.n_rng; k++) {
    const float4 c = ranges[J.rng + k];
    r.lo = fminf(r.lo, c.x);
    r.hi = fmaxf(r.hi, c.y);
    r.nan |= c.z != 0.0f;
  }
  if (J.negate) r = DtRange{-r.hi, -r.lo, r.nan};
  float ab = fmaxf(fabsf(r.lo), fabsf(r.hi));
  int K = dt_window(r.lo, r.hi, ab, J.ay, J.by, d0);
  if (r.nan || K > kDtEdge || !dt_monotone(ab, J.ay, J.by, K)) {
    // the map's columns in the general form, shared out over its blocks; its rows by k_dt_rest
    const int L = dt_lines1(d0, kDtTile);
    for (int x = blk.y / J.rows * L; x < d1; x += J.parts * L) dt_tile<1>(J, x, d1, arena, arena_i, fallback_count, dsm);
    if (tid == 0 && nr > 0) rest[atomicAdd(n_rest, 1)] = make_int4(blk.x, blk.y, blk.y + nr, 0);
    return;
  }
  if (nr <= 0) return;
  for (int e = tid; e < (2 * kDtEdge + 8) * nr; e += kDtThreads)
    Z.T[e < kDtEdge * nr ? e - kDtEdge * nr : e - kDtEdge * nr + d1 * nr] = INFINITY;
  float lo = INFINITY, hi = -INFINITY;
  if (K <= 3) dt_strip1<3>(J, Z, arena, lo, hi);
  else if (K <= 4) dt_strip1<4>(J, Z, arena, lo, hi);
  else if (K <= 5) dt_strip1<5>(J, Z, arena, lo, hi);
  else if (K <= 6) dt_strip1<6>(J, Z, arena, lo, hi);
  else if (K <= 8) dt_strip1<8>(J, Z, arena, lo, hi);
  else if (K <= 12) dt_strip1<12>(J, Z, arena, lo, hi);
  else dt_strip1<kDtEdge>(J, Z, arena, lo, hi);
  // pass 2's windows from the strip's own range
  r = dt_block_range(DtRange{lo, hi, false}, red);
  ab = fmaxf(fabsf(r.lo), fabsf(r.hi));
  K = dt_window(r.lo, r.hi, ab, J.ax, J.bx, d1);
  if (K > kDtEdge || !dt_monotone(ab, J.ax, J.bx, K)) {   // the strip's rows in the general form, by k_dt_rest
    float *tm = arena + J.tmpM_off;
    int *ti = arena_i + J.tmpI_off;
    for (int e = tid; e < d1 * nr; e += kDtThreads) {
      const int x = e / nr, y = Z.y0 + e - x * nr;
      tm[x * d0 + y] = Z.T[e];
      ti[x * d0 + y] = y - Z.t1[e];
    }
    if (tid == 0) rest[atomicAdd(n_rest, 1)] = make_int4(blk.x, blk.y, blk.y + nr, 0);
    return;
  }
  const bool half = J.samp_m && J.samp_i;
#define DT_ROWS(KM)                                            \
  do {                                                         \
    if (half) dt_strip2<KM, 2>(J, Z, arena, arena_i);          \
    else dt_strip2<KM, 1>(J, Z, arena, arena_i);               \
  } while (0)
  if (K <= 3) DT_ROWS(3);
  else if (K <= 4) DT_ROWS(4);
  else if (K <= 5) DT_ROWS(5);
  else if (K <= 6) DT_ROWS(6);
  else if (K <= 8) DT_ROWS(8);
  else if (K <= 12) DT_ROWS(12);
  else DT_ROWS(kDtEdge);
#undef DT_ROWS
}

// Pass 2 of the strips that k_dt_strip has left, in the general form
__global__ void __launch_bounds__(kDtThreads) k_dt_rest(const DtJob *__restrict__ jobs, const int *n_rest, const int4 *rest,
                                                        float *__restrict__ arena, int *__restrict__ arena_i,
                                                        int *fallback_count) {
  extern __shared__ float dsm[];
  const int n = *n_rest;
  const int share = max(1, (int)gridDim.x / max(n, 1));   // blocks to a strip, where there are few of them
  for (int e = blockIdx.x / share; e < n; e += gridDim.x / share) {
    const int4 r = rest[e];
    const int L = 1 << dt_lg_lines2(jobs[r.x].d1, kDtTile);
    for (int y = r.y + blockIdx.x % share * L; y < r.z; y += share * L)
      dt_tile<2>(jobs[r.x], y, r.z, arena, arena_i, fallback_count, dsm);
  }
}

void dt_strip_sizes(std::vector<DtJob> &jobs, int elems) {
  for (DtJob &J : jobs) J.rows = dt_strip_rows(J.d0, J.d1, elems);
}

void dt_block_lists(std::vector<DtJob> &jobs, DtBlocks &B) {
  B = DtBlocks{};
  B.rest_blocks = kDtParts;
  for (size_t j = 0; j < jobs.size(); j++) {
    DtJob &J = jobs[j];
    J.rng = (int)B.chunks.size();
    if (jobs.size() > 1 || J.d0 * J.d1 > kDtOwnRange)
      for (int e = 0; e < J.d0 * J.d1; e += kDtChunk) B.chunks.push_back(make_int2((int)j, e));
    J.n_rng = (int)B.chunks.size() - J.rng;
    J.parts = (J.d0 + J.rows - 1) / J.rows;
    for (int k = 0; k < J.parts; k++) B.strips.push_back(make_int2((int)j, k * J.rows));
    if (jobs.size() == 1) {   // (beyond its strips they only help in the general form)
      B.rest_blocks = std::max(kDtParts, std::min(4 * kDtParts, J.d0 * J.d1 / kDtTile));
      J.parts = std::max(J.parts, B.rest_blocks);
    }
    B.blocks += J.parts;
    const size_t nr = std::min(J.rows, J.d0);
    B.smem = std::max(B.smem, sizeof(float) * (kDtStage + (J.d1 + 2 * kDtEdge + 8) * nr) + J.d1 * nr);
    // tiles of the general form
    B.smem_rest = std::max({B.smem_rest, dt_smem_bytes(dt_lines1(J.d0, kDtTile), J.d0),
                            dt_smem_bytes(1 << dt_lg_lines2(J.d1, kDtTile), J.d1)});
  }
  B.smem = std::max(B.smem, B.smem_rest);
  // the largest maps' strips first, so the long blocks start in the first wave
  std::stable_sort(B.strips.begin(), B.strips.end(), [&](const int2 &x, const int2 &y) {
    return (long long)jobs[x.x].rows * jobs[x.x].d1 > (long long)jobs[y.x].rows * jobs[y.x].d1;
  });
}

size_t dt_work_words(const DtBlocks &B) { return 4 + 4 * B.strips.size() + 4 * B.chunks.size(); }

cudaError_t launch_dt(const DtJob *d_jobs, const int2 *d_chunks, const int2 *d_strips, const DtBlocks &B, float *arena,
                      int *arena_i, int *work, int *fallback_count, cudaStream_t s) {
  const int n_chunks = (int)B.chunks.size(), n_strips = (int)B.strips.size();
  if (n_strips <= 0) return cudaSuccess;
  static SmemAttr a1, a2;
  cudaError_t e = raise_smem(a1, k_dt_strip, B.smem);
  if (e == cudaSuccess) e = raise_smem(a2, k_dt_rest, B.smem_rest);
  if (e != cudaSuccess) return e;
  int4 *rest = reinterpret_cast<int4 *>(work + 4);
  float4 *ranges = reinterpret_cast<float4 *>(rest + n_strips);
  if (n_chunks) k_dt_range<<<n_chunks, kDtThreads, 0, s>>>(d_jobs, d_chunks, arena, ranges, work);
  k_dt_strip<<<B.blocks, kDtThreads, B.smem, s>>>(d_jobs, d_strips, ranges, work, rest, arena, arena_i, fallback_count,
                                                  n_strips);
  k_dt_rest<<<B.rest_blocks, kDtThreads, B.smem_rest, s>>>(d_jobs, work, rest, arena, arena_i, fallback_count);
  return cudaGetLastError();
}

}  // namespace geye
