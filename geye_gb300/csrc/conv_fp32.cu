// conv_fp32.cu -- root/part filter convolution in FP32 on the CUDA cores.
//
// Arithmetic of CAR_TRACKING/GPU_function.cu:302-358 (process_root) and
// :630-685 (process_part), whose loop is the only statement of the
// reference's fconvsMT arithmetic: for each of the 31 features f,
//   val = sum_{xp} sum_{yp} A[f][x+xp][y+yp] * B[f][xp][yp]   (xp outer)
//   add_val += val
// and the output is 0 + add_val.  This kernel repeats that order exactly (a
// multiplication and an addition per tap, never fused), so its maps are
// bit-identical to the oracle's.
//
// What bounds it: the issue of FP32 instructions.  A tap costs two roundings, so
// two instructions per lane: 2 * MACs / (SMs * 128 * clock) at best, and a loop of
// nothing but dependent-free mul and add reaches 111 of the 128 lanes a clock.
// The packed forms (mul/add.rn.f32x2) are no way around it: they run at the
// same rate per lane (103 measured), and the assembler contracts a packed
// product and sum into one fused operation, -fmad=false or not.
//
// A thread owns CR rows of two columns for G filters of one size: a column's
// features are read once into registers (16-byte reads) and serve every tap
// and filter, the taps come as 16-byte broadcasts.  Features arrive as planes
// with 16-byte columns and filters as a bank laid out at plan time (a chunk of
// four channels contiguous), so staging is 16-byte asynchronous copies, the
// next chunk's in flight during this one's taps.
//
// Two splits of the work over a block's four warps, the same bits:
//   whole   a warp takes a tile of its own and every channel: least staging and
//           no exchange, for plans with enough tiles (kConvWhole) and groups
//           of three or four filters;
//   split   the sums of the channels are independent until they are added in
//           channel order, so the warps take a channel each of the same tile
//           and then share the additions of the chunk's sums in order.  Tiles
//           are a quarter the size and a block's serial chain a quarter as long,
//           which fills the chip on small frames and in the last wave.
// Measured (conv stage of a frame, both models; before: a thread per output
// column with a launch per model and kind): 320x240 car 266 -> 69 us, 641x479
// trained-like models 1210 -> 406 us, 1280x720 car+person 2229 -> 1499 us
// (24.7 TFLOP/s of the 35.0 that 111 lanes a clock would give; 14% of the
// lanes work on the padding of tiles).  split / whole: 1280x720 car+person 1690 /
// 1499 us, 641x479 car+person 554 / 510, trained-like 406 / 430.
#include <algorithm>

#include "internal.h"

namespace geye {

constexpr int kCThreads = 128, kCWarps = 4;
constexpr int kChunk = 4;                 // channels per chunk: one per warp
constexpr int kChunks = (kFeat + kChunk - 1) / kChunk;
constexpr size_t kConvSmem = 55 * 1024;        // four blocks an SM
constexpr size_t kConvSmemMax = 200 * 1024;    // for filters whose columns need more
// split tiles of a launch from which on whole tiles (four times the size) are taken: about eight waves of
// four blocks an SM.  641x479: car+person (5607 tiles) 554 split, 510 us whole; 480x360 (2981) 305 and 342
constexpr long long kConvWhole = 5000;

typedef unsigned long long f32x2;   // two floats in one 64-bit register

__device__ __forceinline__ f32x2 pack2(float x, float y) {
  f32x2 d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(x), "f"(y));
  return d;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ void copy16(uint32_t dst, const void *src, bool valid) {   // zeros where not valid
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid ? 16 : 0) : "memory");
}

// rows and columns per thread for a group of g filters
__host__ __device__ constexpr int conv_cr(int g) { return g <= 2 ? 8 : 4; }
constexpr int kCX = 2;

template <int G, int CR>
__device__ __forceinline__ void conv_zero(float (&v)[G][kCX][CR]) {
#pragma unroll
  for (int g = 0; g < G; g++)
#pragma unroll
    for (int j = 0; j < kCX; j++)
#pragma unroll
      for (int r = 0; r < CR; r++) v[g][j][r] = 0.f;
}

// N taps of a filter column: val[g][j][h] holds rows 2h, 2h + 1 of column j.  Ax: the
// features under the first tap at the thread's first row and column (jx floats between
// its columns); Bx: the taps (b0p between filters).
template <int G, int CR, int N>
__device__ __forceinline__ void conv_column(float (&val)[G][kCX][CR], const float *__restrict__ Ax, int jx,
                                            const float *__restrict__ Bx, int b0p) {
  constexpr int W = (CR + N - 1 + 3) & ~3;
  float w[kCX][W];
#pragma unroll
  for (int j = 0; j < kCX; j++)
#pragma unroll
    for (int r = 0; r < W; r += 4) {
      const float4 v = *reinterpret_cast<const float4 *>(Ax + j * jx + r);
      w[j][r] = v.x; w[j][r + 1] = v.y; w[j][r + 2] = v.z; w[j][r + 3] = v.w;
    }
#pragma unroll
  for (int k = 0; k < N; k += 4) {
    float b[G][4];
#pragma unroll
    for (int g = 0; g < G; g++) {
      const float4 p = *reinterpret_cast<const float4 *>(Bx + g * b0p + k);
      b[g][0] = p.x; b[g][1] = p.y; b[g][2] = p.z; b[g][3] = p.w;
    }
#pragma unroll
    for (int i = 0; i < 4 && k + i < N; i++)
#pragma unroll
      for (int j = 0; j < kCX; j++)
#pragma unroll
        for (int r = 0; r < CR; r++)
#pragma unroll
          for (int g = 0; g < G; g++) val[g][j][r] += w[j][k + i + r] * b[g][i];
  }
}

// N taps of xb filter columns
template <int G, int CR, int N>
__device__ __forceinline__ void conv_columns(float (&val)[G][kCX][CR], const float *__restrict__ Ax, int RP,
                                             int jx, const float *__restrict__ Bx, int b0p, int xb) {
  for (int xp = 0; xp < xb; xp++)
    conv_column<G, CR, N>(val, Ax + xp * RP, jx, Bx + xp * G * b0p, b0p);
}

// One warp's channel of a chunk over xb filter columns, tap by tap (Ac: [x][RP] floats, Bc: [xp][g][b0p] floats);
// columns of 4 to 10 taps are unrolled, others take four at a time
template <int G, int CR>
__device__ __forceinline__ void conv_taps(float (&val)[G][kCX][CR], const float *__restrict__ Ac, int RP, int jx,
                                          const float *__restrict__ Bc, int b0, int b0p, int xb) {
  switch (b0) {
    case 1: case 2: case 3: break;
    case 4: return conv_columns<G, CR, 4>(val, Ac, RP, jx, Bc, b0p, xb);
    case 5: return conv_columns<G, CR, 5>(val, Ac, RP, jx, Bc, b0p, xb);
    case 6: return conv_columns<G, CR, 6>(val, Ac, RP, jx, Bc, b0p, xb);
    case 7: return conv_columns<G, CR, 7>(val, Ac, RP, jx, Bc, b0p, xb);
    case 8: return conv_columns<G, CR, 8>(val, Ac, RP, jx, Bc, b0p, xb);
    case 9: return conv_columns<G, CR, 9>(val, Ac, RP, jx, Bc, b0p, xb);
    case 10: return conv_columns<G, CR, 10>(val, Ac, RP, jx, Bc, b0p, xb);
    default: break;
  }
  for (int xp = 0; xp < xb; xp++) {
    const float *Ax = Ac + xp * RP;
    const float *Bx = Bc + xp * G * b0p;
    int y = 0;
    for (; y + 4 <= b0; y += 4) conv_column<G, CR, 4>(val, Ax + y, jx, Bx + y, b0p);
    if (b0 & 2) {
      if (b0 & 1) conv_column<G, CR, 3>(val, Ax + y, jx, Bx + y, b0p);
      else conv_column<G, CR, 2>(val, Ax + y, jx, Bx + y, b0p);
    } else if (b0 & 1) {
      conv_column<G, CR, 1>(val, Ax + y, jx, Bx + y, b0p);
    }
  }
}

template <int G, bool SPLIT>
__device__ __forceinline__ void conv_tile(const ConvJob &J, int tile, const float *__restrict__ bank_all,
                                          const float *__restrict__ arena_in, float *__restrict__ arena_out,
                                          float *sm) {
  constexpr int CR = conv_cr(G), NP = G * kCX * CR / 2, NQ = NP / kCWarps;   // packed sums of a position, a warp's share
  const int TY = J.ty, TX = J.tx, b0 = J.b0, b0p = J.b0p, RP = J.RP;
  const int WY = J.wy, WX = SPLIT ? 1 : kCWarps / WY;       // warps' tiles along y and x
  const int ty0 = (tile % J.tiles_y) * (WY * TY * CR), tx0 = (tile / J.tiles_y) * (WX * kCX * TX);
  const int cols = WX * kCX * TX + J.xb - 1, chan = cols * RP;   // staged columns; floats of a channel
  const int bcol = G * b0p;                                 // taps of a filter column
  const size_t bchan = (size_t)J.b1 * bcol;                 // of a channel in the bank
  float *A_s = sm;                                          // [2][kChunk][cols][RP]
  float *B_s = A_s + 2 * kChunk * chan;                     // [2][kChunk][xb][G][b0p]
  f32x2 *V_s = reinterpret_cast<f32x2 *>(B_s + 2 * kChunk * J.xb * bcol);              // [kChunk][NP][32]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // the thread's first row and column in the block's tile
  const int row = ((SPLIT ? 0 : warp % WY) * TY + lane % TY) * CR;
  const int col = (SPLIT ? 0 : warp / WY) * (kCX * TX) + lane / TY;
  const bool active = lane / TY < TX;
  const int S0 = feat_stride(J.a0);
  const size_t plane = (size_t)S0 * J.a1;
  const float *feat = arena_in + J.feat_off + (size_t)tx0 * S0 + ty0;
  const float *bank = bank_all + J.bank_off;

  // stage s: chunk s / nx, filter columns from (s % nx) * xb on
  const int nx = (J.b1 + J.xb - 1) / J.xb, nst = kChunks * nx;
  auto stage = [&](int s) {
    const int ck = s / nx, xp0 = (s - ck * nx) * J.xb, xb = min(J.xb, J.b1 - xp0);
    const int c0 = ck * kChunk, nc = min(kChunk, kFeat - c0);
    const int q = RP >> 2, colq = cols * q;   // 16-byte pieces of a column, of a channel
    const uint32_t a_dst = (uint32_t)__cvta_generic_to_shared(A_s + (s & 1) * kChunk * chan);
    const float *src = feat + c0 * plane + (size_t)xp0 * S0;
    // piece i = (channel, column, quarter): walked with increments of kCThreads
    int k = tid % q, t = tid / q, cx = t % cols, c = t / cols;
    const int dk = kCThreads % q, dt = kCThreads / q, dx = dt % cols, dc = dt / cols;
    for (int i = tid; i < nc * colq; i += kCThreads) {
      const bool ok = ty0 + 4 * k < S0 && tx0 + xp0 + cx < J.a1;
      copy16(a_dst + 16 * i, ok ? src + c * plane + (size_t)cx * S0 + 4 * k : src, ok);
      k += dk;
      cx += dx;
      c += dc;
      if (k >= q) { k -= q; cx++; }
      if (cx >= cols) { cx -= cols; c++; }
    }
    const int run = xb * bcol / 4;   // 16-byte pieces of a channel's columns
    const uint32_t b_dst = (uint32_t)__cvta_generic_to_shared(B_s + (s & 1) * kChunk * J.xb * bcol);
    const float *bsrc = bank + (size_t)c0 * bchan + (size_t)xp0 * bcol;
    for (int ch = 0; ch < nc; ch++)
      for (int i = tid; i < run; i += kCThreads)
        copy16(b_dst + 16 * (ch * (J.xb * bcol / 4) + i), bsrc + ch * bchan + 4 * i, true);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  stage(0);
  int s = 0;
  if constexpr (SPLIT) {   // a warp takes a channel of the chunk; the sums are added in channel order through V_s
    f32x2 add[NQ];
#pragma unroll
    for (int p = 0; p < NQ; p++) add[p] = 0ull;
    for (int c0 = 0; c0 < kFeat; c0 += kChunk) {
      const int nc = min(kChunk, kFeat - c0);
      float val[G][kCX][CR];
      conv_zero<G, CR>(val);
      for (int xp0 = 0; xp0 < J.b1; xp0 += J.xb, s++) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();   // stage s has landed; everyone is done with stage s - 1 and the last chunk's sums
        if (s + 1 < nst) stage(s + 1);
        if (active && warp < nc)
          conv_taps<G, CR>(val, A_s + ((s & 1) * kChunk + warp) * chan + col * RP + row, RP, TX * RP,
                           B_s + ((s & 1) * kChunk + warp) * J.xb * bcol, b0, b0p, min(J.xb, J.b1 - xp0));
      }
#pragma unroll
      for (int g = 0; g < G; g++)
#pragma unroll
        for (int j = 0; j < kCX; j++)
#pragma unroll
          for (int h = 0; h < CR / 2; h++)
            V_s[(warp * NP + (g * kCX + j) * (CR / 2) + h) * 32 + lane] = pack2(val[g][j][2 * h], val[g][j][2 * h + 1]);
      __syncthreads();
#pragma unroll
      for (int p = 0; p < NQ; p++)
        for (int c = 0; c < nc; c++) add[p] = add2(add[p], V_s[(c * NP + warp * NQ + p) * 32 + lane]);
    }
    if (!active) return;
#pragma unroll
    for (int p = 0; p < NQ; p++) {
      const int e = warp * NQ + p, g = e / (kCX * CR / 2), j = e / (CR / 2) % kCX, h = e % (CR / 2);
      const int x = tx0 + col + j * TX, y = ty0 + row + 2 * h;
      if (x >= J.c1) continue;
      float *out = arena_out + J.out_off[g] + (size_t)x * J.c0 + y;
      const float2 v = *reinterpret_cast<const float2 *>(&add[p]);
      if (y < J.c0) out[0] = 0.0f + v.x;
      if (y + 1 < J.c0) out[1] = 0.0f + v.y;
    }
  } else {   // a warp takes a tile of its own and every channel
    float add[G][kCX][CR];
    conv_zero<G, CR>(add);
    const bool some = active && ty0 + row < J.c0 && tx0 + col < J.c1;
    for (int c0 = 0; c0 < kFeat; c0 += kChunk) {
      const int nc = min(kChunk, kFeat - c0);
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      __syncthreads();   // stage s has landed; everyone is done with stage s - 1
      if (s + 1 < nst) stage(s + 1);
      if (some)
        for (int c = 0; c < nc; c++) {
          float val[G][kCX][CR];
          conv_zero<G, CR>(val);
          conv_taps<G, CR>(val, A_s + ((s & 1) * kChunk + c) * chan + col * RP + row, RP, TX * RP,
                           B_s + ((s & 1) * kChunk + c) * J.xb * bcol, b0, b0p, J.b1);
#pragma unroll
          for (int g = 0; g < G; g++)
#pragma unroll
            for (int j = 0; j < kCX; j++)
#pragma unroll
              for (int r = 0; r < CR; r++) add[g][j][r] += val[g][j][r];
        }
      s++;
    }
    if (!some) return;
#pragma unroll
    for (int g = 0; g < G; g++)
#pragma unroll
      for (int j = 0; j < kCX; j++) {
        const int x = tx0 + col + j * TX, y = ty0 + row;
        if (x >= J.c1) continue;
        float *out = arena_out + J.out_off[g] + (size_t)x * J.c0 + y;
#pragma unroll
        for (int r = 0; r < CR; r++)
          if (y + r < J.c0) out[r] = 0.0f + add[g][j][r];
      }
  }
}

__global__ void __launch_bounds__(kCThreads, 4) k_conv_fp32(const ConvJob *__restrict__ jobs,
                                                         const int2 *__restrict__ blocks,
                                                         const float *__restrict__ bank,
                                                         const float *__restrict__ arena_in,
                                                         float *__restrict__ arena_out) {
  extern __shared__ __align__(16) float sm[];
  const int2 blk = blocks[blockIdx.x];
  const ConvJob &J = jobs[blk.x];
  if (J.split) {
    switch (J.n_filt) {
      case 1: conv_tile<1, true>(J, blk.y, bank, arena_in, arena_out, sm); break;
      case 2: conv_tile<2, true>(J, blk.y, bank, arena_in, arena_out, sm); break;
      case 3: conv_tile<3, true>(J, blk.y, bank, arena_in, arena_out, sm); break;
      default: conv_tile<4, true>(J, blk.y, bank, arena_in, arena_out, sm); break;
    }
  } else {
    switch (J.n_filt) {
      case 1: conv_tile<1, false>(J, blk.y, bank, arena_in, arena_out, sm); break;
      case 2: conv_tile<2, false>(J, blk.y, bank, arena_in, arena_out, sm); break;
      case 3: conv_tile<3, false>(J, blk.y, bank, arena_in, arena_out, sm); break;
      default: conv_tile<4, false>(J, blk.y, bank, arena_in, arena_out, sm); break;
    }
  }
}

static size_t conv_smem(const ConvJob &J) {
  const int g = J.n_filt, cols = (J.split ? 1 : kCWarps / J.wy) * kCX * J.tx + J.xb - 1;
  return 4 * (size_t)(2 * kChunk * cols * J.RP) + 4 * (size_t)(2 * kChunk * J.xb * g * J.b0p) +
         (J.split ? 8 * (size_t)(kChunk * g * kCX * conv_cr(g) / 2 * 32) : 0);
}

// The launch shape of a job from its sizes and filter count; false when none fits.
static bool conv_shape(ConvJob &J, bool split, size_t limit = kConvSmem) {
  const int cr = conv_cr(J.n_filt);
  J.b0p = (J.b0 + 3) & ~3;
  J.split = split;
  double best = -1;
  const ConvJob in = J;
  for (int ty = 1; ty <= 32; ty++)
    for (int wy = 1; wy <= (split ? 1 : kCWarps); wy *= 2) {
      ConvJob C = in;
      const int wx = split ? 1 : kCWarps / wy;
      C.ty = ty;
      C.tx = 32 / ty;
      C.wy = wy;
      C.tiles_y = (C.c0 + wy * ty * cr - 1) / (wy * ty * cr);
      C.tiles_x = (C.c1 + wx * kCX * C.tx - 1) / (wx * kCX * C.tx);
      C.RP = wy * ty * cr + C.b0p;   // a thread's last window ends there
      C.xb = C.b1;
      if (split)
        for (C.xb = std::min(C.b1, 16); C.xb > 1 && conv_smem(C) > kConvSmem; C.xb--) {}
      if (conv_smem(C) > limit) continue;
      // a block's cost per chunk, in operations of a warp: the taps of the warps' channels, and what
      // the copies of features and taps and the exchange of the sums come to (about 12 per 16 bytes and thread)
      const double warps = split ? 1 : (double)((C.c0 + ty * cr - 1) / (ty * cr)) *
                                           ((C.c1 + kCX * C.tx - 1) / (kCX * C.tx)) / (C.tiles_y * C.tiles_x);
      const double taps = 2.0 * C.n_filt * kCX * cr * C.b0 * C.b1 * warps;
      const double pieces = (double)C.RP * (wx * kCX * C.tx + C.b1 - 1) + 1.0 * C.n_filt * C.b0p * C.b1;
      const double cost = (taps + 12.0 * pieces / kCThreads + 200) * C.tiles_y * C.tiles_x;
      if (best < 0 || cost < best) {
        best = cost;
        J = C;
      }
    }
  J.cost = std::min(J.b0 * J.b1, 1 << 18) * J.n_filt * cr * (split ? 1 : kCWarps);
  return best >= 0;
}

// The bank of a group: [channel, padded to whole chunks][filter column][filter][b0p] taps.
static void conv_bank(const ConvJob &J, const std::vector<const float *> &w, std::vector<float> &bank) {
  const size_t at = bank.size();
  bank.resize(at + (size_t)kChunks * kChunk * J.b1 * J.n_filt * J.b0p, 0.f);
  for (int c = 0; c < kFeat; c++)
    for (int x = 0; x < J.b1; x++)
      for (int g = 0; g < J.n_filt; g++) {
        float *d = bank.data() + at + ((((size_t)c * J.b1 + x) * J.n_filt + g) * J.b0p);
        for (int y = 0; y < J.b0; y++) d[y] = w[g][((size_t)c * J.b1 + x) * J.b0 + y];
      }
}

bool conv_fp32_jobs(ConvJob J, const std::vector<const float *> &filters, const std::vector<int> &out_off,
                    ConvBank &bank, std::vector<ConvJob> &jobs) {
  const int n = (int)filters.size();
  J.c0 = J.a0 - J.b0 + 1;
  J.c1 = J.a1 - J.b1 + 1;
  // groups of equal length; where the taps of a group do not fit, one filter at a time
  for (int groups : {(n + kConvGroup - 1) / kConvGroup, n}) {
    std::vector<ConvJob> out;
    bool fits = true;
    for (int g = 0, i = 0; g < groups && fits; g++) {
      ConvJob C = J;
      std::vector<const float *> w;
      for (const int end = (int)((long long)n * (g + 1) / groups); i < end; i++) {
        w.push_back(filters[i]);
        C.out_off[C.n_filt++] = out_off[i];
      }
      fits = conv_shape(C, true) || conv_shape(C, true, kConvSmemMax);
      if (fits) {   // every level's group of these filters shares one bank
        const auto key = std::make_pair(std::make_pair(C.b0, C.b1), w);
        auto it = bank.at.find(key);
        if (it == bank.at.end()) {
          it = bank.at.emplace(key, (int)bank.taps.size()).first;
          conv_bank(C, w, bank.taps);
        }
        C.bank_off = it->second;
      }
      out.push_back(C);
    }
    if (fits) {
      jobs.insert(jobs.end(), out.begin(), out.end());
      return true;
    }
  }
  return n == 0;
}

size_t conv_fp32_blocks(std::vector<ConvJob> &jobs, std::vector<int2> &blocks) {
  blocks.clear();
  size_t smem = 0;
  long long tiles = 0;
  for (auto &J : jobs) tiles += (long long)J.tiles_y * J.tiles_x;
  if (tiles >= kConvWhole)
    for (auto &J : jobs) {   // (groups of one or two filters stage more per tap: 1280x720 trained-like 1104 us, 1264 with them)
      ConvJob C = J;
      if (C.n_filt >= 3 && conv_shape(C, false)) J = C;
    }
  for (size_t j = 0; j < jobs.size(); j++) {
    smem = std::max(smem, conv_smem(jobs[j]));
    for (int t = 0; t < jobs[j].tiles_y * jobs[j].tiles_x; t++) blocks.push_back(make_int2((int)j, t));
  }
  std::stable_sort(blocks.begin(), blocks.end(),
                   [&](const int2 &x, const int2 &y) { return jobs[x.x].cost > jobs[y.x].cost; });
  return smem;
}

void launch_conv_fp32(const ConvJob *d_jobs, const int2 *d_blocks, int n_blocks, size_t smem, const float *d_bank,
                      const float *arena_in, float *arena_out, cudaStream_t s) {
  if (n_blocks <= 0) return;
  static SmemAttr attr;
  raise_smem(attr, k_conv_fp32, smem);
  k_conv_fp32<<<n_blocks, kCThreads, smem, s>>>(d_jobs, d_blocks, d_bank, arena_in, arena_out);
}

}  // namespace geye
