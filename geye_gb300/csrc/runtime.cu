// runtime.cu -- host runtime of libgeye_dpm: models, plans and the pipeline.
//
// Host-side arithmetic that sizes the pyramid (scale schedule, resize output
// sizes, tap tables, feature sizes, level skipping) repeats the reference's C
// expressions with the same float/double types; this file is compiled with
// -ffp-contract=off so the host compiler fuses nothing either.
//   ini_scales           CAR_TRACKING/featurepyramid.cpp:174-239
//   pyramid schedule     CAR_TRACKING/featurepyramid.cpp.org:547-661
//   resize sizes / taps  CAR_TRACKING/resize.cc:68-160
//   feature sizes        CAR_TRACKING/featurepyramid.cpp:277-281
//   level skip, conv and part-map sizes  CAR_TRACKING/fconvsMT.cpp:420-470
//   score assembly inputs                CAR_TRACKING/get_boxes.cpp:1000-1360
#include <math.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <map>
#include <mutex>
#include <sstream>

#include "runtime.h"

namespace geye {

static thread_local std::string g_err;
void set_error(const std::string &msg) { g_err = msg; }



bool injected(geye_ctx *ctx, const char *op) {
  if (!ctx || ctx->inject_countdown <= 0 || ctx->inject_op != op) return false;
  if (--ctx->inject_countdown == 0) {
    ctx->inject_op.clear();
    return true;
  }
  return false;
}

geye_status park_pending(geye_ctx *ctx, Plan &P) {
  if (ctx->pending != &P || P.parked) return GEYE_OK;
  const size_t bytes = P.models.size() * (size_t)P.max_cap * 11 * sizeof(int);
  GEYE_TRY(P.d_parked.alloc(ctx, bytes));
  if (!P.h_parked) CUDA_TRY(cudaMallocHost(&P.h_parked, 64 * sizeof(int)));
  CUDA_TRY(cudaMemcpyAsync(P.h_parked, P.d_small.p, 64 * sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
  CUDA_TRY(cudaMemcpyAsync(P.d_parked.p, P.d_result.p, bytes, cudaMemcpyDeviceToDevice, ctx->stream));
  CUDA_TRY(cudaEventRecord(P.ev_done, ctx->stream));   // the submitted frame is done when they are there
  P.parked = true;
  return GEYE_OK;
}

geye_status read_result(Plan &P, int mi, geye_result *out, bool parked) {
  const int *h = static_cast<const int *>(parked ? P.h_parked : P.h_res);
  const int K = h[32 + mi];
  P.last_D[mi] = h[mi];
  P.last_K[mi] = K;
  if (!out) return GEYE_OK;
  memset(out, 0, sizeof(*out));
  out->num = K;
  const size_t k = std::max(K, 1);
  out->point = (int *)malloc(sizeof(int) * 4 * k);
  out->or_point = (int *)malloc(sizeof(int) * 4 * k);
  out->type = (int *)malloc(sizeof(int) * k);
  out->scale = (float *)malloc(sizeof(float) * k);
  out->score = (float *)malloc(sizeof(float) * k);
  if (!out->point || !out->or_point || !out->type || !out->scale || !out->score) {
    geye_result_free(out);
    set_error("host allocation failed");
    return GEYE_ERR_NOMEM;
  }
  // field f of `per` ints a record: its place in the pinned block, and (for records past it) on the device
  const int *src = h + 64 + (size_t)mi * 11 * kHostRes;
  const int *res = (parked ? P.d_parked : P.d_result).as<int>() + (size_t)mi * P.max_cap * 11;
  const int n = parked ? 0 : std::min(K, kHostRes);
  struct { void *to; int at, per; } f[5] = {{out->point, 0, 4}, {out->or_point, 4, 4}, {out->type, 8, 1},
                                            {out->scale, 9, 1}, {out->score, 10, 1}};
  for (auto &x : f) {
    if (n) memcpy(x.to, src + (size_t)x.at * kHostRes, sizeof(int) * x.per * n);
    if (K > n)
      CUDA_TRY(cudaMemcpy(static_cast<int *>(x.to) + x.per * n, res + (size_t)x.at * P.max_cap + x.per * n,
                          sizeof(int) * x.per * (size_t)(K - n), cudaMemcpyDeviceToHost));
  }
  return GEYE_OK;
}

geye_status upload_bytes(geye_ctx *ctx, DevBuf &buf, const void *src, size_t n) {
  GEYE_TRY(buf.alloc(ctx, std::max<size_t>(n, 16)));
  if (n) CUDA_TRY(cudaMemcpyAsync(buf.p, src, n, cudaMemcpyHostToDevice, ctx->stream));
  return GEYE_OK;
}

template <class T>
static geye_status upload(geye_ctx *ctx, DevBuf &buf, const std::vector<T> &v) {
  GEYE_TRY(buf.alloc(ctx, sizeof(T) * std::max<size_t>(v.size(), 1)));
  if (!v.empty()) {
    if (injected(ctx, "h2d")) {
      set_error("injected host-to-device copy failure");
      return GEYE_ERR_INJECTED;
    }
    CUDA_TRY(cudaMemcpyAsync(buf.p, v.data(), sizeof(T) * v.size(), cudaMemcpyHostToDevice, ctx->stream));
  }
  return GEYE_OK;
}

// ----------------------------------------------------------------------------
// model CSV (load_model.cpp:57-558); values are read with fscanf("%f,") like
// the reference so every weight is the same float
// ----------------------------------------------------------------------------
static int scan_f(FILE *f, float *v) { return fscanf(f, "%f,", v) == 1 ? 0 : -1; }

static geye_status parse_model(const char *comp, const char *root, const char *part, HostModel &m) {
  FILE *f = fopen(comp, "r");
  if (!f) { set_error(std::string("model component file not found: ") + comp); return GEYE_ERR_MODEL; }
  float t1, t2, t3, t4;
  int bad = 0;
  bad |= scan_f(f, &t1); m.numcomponent = (int)t1;
  bad |= scan_f(f, &t1); m.sbin = (int)t1;
  bad |= scan_f(f, &t1); m.interval = (int)t1;
  bad |= scan_f(f, &t1); m.max_Y = (int)t1;
  bad |= scan_f(f, &t1); m.max_X = (int)t1;
  const int nc = m.numcomponent;
  if (bad || nc <= 0 || nc > 64 || m.sbin <= 0 || m.interval <= 0) { fclose(f); set_error("bad component header"); return GEYE_ERR_MODEL; }
  m.ridx.resize(nc); m.oidx.resize(nc); m.offw.resize(nc); m.rsize.resize(2 * nc); m.numpart.resize(nc);
  m.pidx.resize(nc); m.didx.resize(nc); m.psize.resize(nc);
  for (int c = 0; c < nc; c++) {
    bad |= scan_f(f, &t1); m.ridx[c] = (int)t1 - 1;
    bad |= scan_f(f, &t1); m.oidx[c] = (int)t1 - 1;
    bad |= scan_f(f, &t1); m.offw[c] = t1;
    bad |= scan_f(f, &t1); bad |= scan_f(f, &t2);
    m.rsize[2 * c] = (int)t1; m.rsize[2 * c + 1] = (int)t2;
    bad |= scan_f(f, &t1); m.numpart[c] = (int)t1;
    const int np = m.numpart[c];
    if (bad || np < 0 || np > kMaxParts) { fclose(f); set_error("bad component record"); return GEYE_ERR_MODEL; }
    m.pidx[c].resize(np); m.didx[c].resize(np); m.psize[c].resize(2 * np);
    for (int k = 0; k < np; k++) {
      bad |= scan_f(f, &t1); m.pidx[c][k] = (int)t1 - 1;
      bad |= scan_f(f, &t1); m.didx[c][k] = (int)t1 - 1;
      bad |= scan_f(f, &t1); bad |= scan_f(f, &t2);
      m.psize[c][2 * k] = (int)t1; m.psize[c][2 * k + 1] = (int)t2;
    }
  }
  bad |= scan_f(f, &t1);
  m.DefL = (int)t1;
  if (bad || m.DefL < 0 || m.DefL > 4096) { fclose(f); set_error("bad deformation count"); return GEYE_ERR_MODEL; }
  m.def.resize(4 * m.DefL); m.anchor.resize(2 * m.DefL);
  for (int k = 0; k < m.DefL; k++) {
    bad |= scan_f(f, &t1); bad |= scan_f(f, &t2); bad |= scan_f(f, &t3); bad |= scan_f(f, &t4);
    m.def[4 * k] = t1; m.def[4 * k + 1] = t2; m.def[4 * k + 2] = t3; m.def[4 * k + 3] = t4;
    bad |= scan_f(f, &t1); bad |= scan_f(f, &t2);
    m.anchor[2 * k] = (int)t1; m.anchor[2 * k + 1] = (int)t2;
  }
  m.x1.resize(nc); m.y1.resize(nc); m.x2.resize(nc); m.y2.resize(nc);
  for (int c = 0; c < nc; c++) {
    const int GL = 1 + 2 * (1 + m.numpart[c]);
    for (auto *v : {&m.x1[c], &m.y1[c], &m.x2[c], &m.y2[c]}) {
      v->resize(GL);
      for (int j = 0; j < GL; j++) { bad |= scan_f(f, &t1); (*v)[j] = t1; }
    }
  }
  fclose(f);
  if (bad) { set_error("truncated component file"); return GEYE_ERR_MODEL; }
  // load_model.cpp:552-553: the pad is forced to zero
  m.padx = 0;
  m.pady = 0;

  auto read_filters = [&](const char *path, bool parts, int &n, std::vector<int> &sz,
                          std::vector<std::vector<float>> &w) -> geye_status {
    FILE *g = fopen(path, "r");
    if (!g) { set_error(std::string("filter file not found: ") + path); return GEYE_ERR_MODEL; }
    float a, b, c;
    int bd = scan_f(g, &a);
    n = (int)a;
    if (bd || n < 0 || n > 4096) { fclose(g); set_error("bad filter count"); return GEYE_ERR_MODEL; }
    sz.resize(3 * n); w.resize(n);
    if (parts) m.part_partner.resize(n);
    for (int i = 0; i < n; i++) {
      bd |= scan_f(g, &a); bd |= scan_f(g, &b); bd |= scan_f(g, &c);
      sz[3 * i] = (int)a; sz[3 * i + 1] = (int)b; sz[3 * i + 2] = (int)c;
      const int num = (int)a * (int)b * (int)c;
      if (bd || num <= 0 || (int)c != kFeat) { fclose(g); set_error("bad filter size"); return GEYE_ERR_MODEL; }
      w[i].resize(num);
      for (int j = 0; j < num; j++) { bd |= scan_f(g, &a); w[i][j] = a; }
      if (parts) { bd |= scan_f(g, &a); m.part_partner[i] = (int)a; }
    }
    fclose(g);
    if (bd) { set_error("truncated filter file"); return GEYE_ERR_MODEL; }
    return GEYE_OK;
  };
  GEYE_TRY(read_filters(root, false, m.NoR, m.root_size, m.rootfilter));
  GEYE_TRY(read_filters(part, true, m.NoP, m.part_size, m.partfilter));
  // shapes the kernels assume
  if (m.NoR < nc) { set_error("fewer root filters than components"); return GEYE_ERR_UNSUPPORTED; }
  for (int c = 1; c < nc; c++)
    if (m.numpart[c] != m.numpart[0]) {
      // get_boxes.cpp:1746 sizes every record with numpart[0]
      set_error("components with different part counts");
      return GEYE_ERR_UNSUPPORTED;
    }
  for (int c = 0; c < nc; c++)
    for (int k = 0; k < m.numpart[c]; k++)
      if (m.pidx[c][k] < 0 || m.pidx[c][k] >= m.NoP || m.didx[c][k] < 0 || m.didx[c][k] >= m.DefL) {
        set_error("part or deformation index out of range");
        return GEYE_ERR_MODEL;
      }
  if (m.sbin > 8) { set_error("sbin above 8 is not supported by the HOG kernel"); return GEYE_ERR_UNSUPPORTED; }
  return GEYE_OK;
}

// ----------------------------------------------------------------------------
// scale schedule and sizes
// ----------------------------------------------------------------------------
static int max_scale_for(const HostModel &m, int width, int height) {
  const int sbin = m.sbin, interval = m.interval;
  const float sc = pow(2.0, (1 / (double)interval));
  int max_scale = 36;
  const int L_NUM = interval + max_scale;
  float MRY = (float)m.rsize[0];
  float MRX = (float)m.rsize[1];
  for (int kk = 1; kk < m.numcomponent; kk++) {
    if (m.rsize[kk * 2] < MRY) MRY = m.rsize[kk * 2];
    if (m.rsize[kk * 2 + 1] < MRX) MRX = m.rsize[kk * 2 + 1];
  }
  MRY /= 2;
  MRX /= 2;
  float h = (float)height / (float)sbin;
  float w = (float)width / (float)sbin;
  float sc_step = 1 / sc;
  for (int kk = 0; kk < L_NUM; kk++) {
    h *= sc_step;
    w *= sc_step;
    if (h < MRY || w < MRX) { max_scale = kk - interval - 1; break; }
  }
  if (max_scale < interval) max_scale = interval;
  return max_scale;
}

static void resize_dims(int h, int w, float scale, int &oh, int &ow) {
  if (scale == 1.0f) { oh = h; ow = w; return; }
  oh = (int)((float)h * scale + 0.5);
  ow = (int)((float)w * scale + 0.5);
}

// taps of one 1-D pass (resize.cc:68-105), grouped by destination index
static void build_taps(int sheight, int dheight, std::vector<int> &start, std::vector<int> &si,
                       std::vector<float> &alpha) {
  float scale = (float)dheight / (float)sheight;
  float invscale = (float)sheight / (float)dheight;
  for (int dy = 0; dy < dheight; dy++) {
    start.push_back((int)si.size());
    float fsy1 = dy * invscale;
    float fsy2 = fsy1 + invscale;
    int sy1 = (int)(fsy1 + 0.99);
    int sy2 = (int)fsy2;
    if (sy1 - fsy1 > 1e-3) { si.push_back(sy1 - 1); alpha.push_back((sy1 - fsy1) * scale); }
    for (int sy = sy1; sy < sy2; sy++) { si.push_back(sy); alpha.push_back(scale); }
    if (fsy2 - sy2 > 1e-3) { si.push_back(sy2); alpha.push_back((fsy2 - sy2) * scale); }
  }
  start.push_back((int)si.size());
  // float rounding could name a source row one past the end (the reference
  // would read past its buffer); keep every read inside the image
  for (auto &v : si) v = std::min(std::max(v, 0), sheight - 1);
}

static void feature_dims(int h, int w, int sbin, int &b0, int &b1, int &fs0, int &fs1) {
  b0 = (int)floor((double)h / (double)sbin + 0.5);
  b1 = (int)floor((double)w / (double)sbin + 0.5);
  fs0 = std::max(b0 - 2, 0);
  fs1 = std::max(b1 - 2, 0);
}

// ----------------------------------------------------------------------------
// plan construction
// ----------------------------------------------------------------------------
// The maps of a list of filters (sizes sz) over one feature level: their places in the
// arena, and in FP32 mode the jobs that fill them.
static geye_status conv_level(geye_ctx *ctx, Plan &P, ModelPlan &mp, ArenaAlloc &A, const LevelInfo &L,
                              const std::vector<int> &sz, const std::vector<std::vector<float>> &filters, int n,
                              const char *too_large, std::vector<int> &out_off) {
  out_off.assign(n, -1);
  std::map<std::pair<int, int>, std::vector<int>> by_size;
  for (int i = 0; i < n; i++) {
    const int b0 = sz[3 * i], b1 = sz[3 * i + 1], c0 = L.fs0 - b0 + 1, c1 = L.fs1 - b1 + 1;
    if (c0 < 1 || c1 < 1) { set_error(too_large); return GEYE_ERR_UNSUPPORTED; }
    out_off[i] = A.take((size_t)c0 * c1);
    by_size[{b0, b1}].push_back(i);
    mp.conv_flops += 2.0 * c0 * c1 * b0 * b1 * kFeat;
    mp.conv_bytes += 4.0 * c0 * c1;
  }
  if (n) mp.conv_bytes += 128.0 * L.fs0 * L.fs1;
  if (ctx->conv_mode != GEYE_CONV_FP32 && !P.from_features) return GEYE_OK;
  for (auto &g : by_size) {
    ConvJob J{};
    J.feat_off = L.feat_off; J.a0 = L.fs0; J.a1 = L.fs1;
    J.b0 = g.first.first; J.b1 = g.first.second;
    std::vector<const float *> w;
    std::vector<int> o;
    for (int i : g.second) {
      w.push_back(filters[i].data());
      o.push_back(out_off[i]);
    }
    if (!conv_fp32_jobs(J, w, o, P.conv_bank, P.conv_jobs)) {
      set_error("filter too large for the FP32 convolution");
      return GEYE_ERR_UNSUPPORTED;
    }
  }
  return GEYE_OK;
}

static geye_status plan_dt(geye_ctx *ctx, const ModelPlan &mp, int elems, std::unique_ptr<DtPlan> &out) {
  auto D = std::make_unique<DtPlan>();
  D->elems = elems;
  D->jobs = mp.dt_jobs;
  dt_strip_sizes(D->jobs, elems);
  dt_block_lists(D->jobs, D->blocks);
  GEYE_TRY(upload(ctx, D->d_jobs, D->jobs));
  GEYE_TRY(upload(ctx, D->d_chunks, D->blocks.chunks));
  GEYE_TRY(upload(ctx, D->d_strips, D->blocks.strips));
  GEYE_TRY(D->d_work.alloc(ctx, sizeof(int) * dt_work_words(D->blocks)));
  out = std::move(D);
  return GEYE_OK;
}

static cudaError_t launch_plan_dt(geye_ctx *ctx, Plan &P, const DtPlan &D) {
  if (D.blocks.chunks.empty()) {   // a lone map's strips have no k_dt_range before them to clear the count of those left
    const cudaError_t e = cudaMemsetAsync(D.d_work.p, 0, sizeof(int), ctx->stream);
    if (e != cudaSuccess) return e;
  }
  return launch_dt(D.d_jobs.as<DtJob>(), D.d_chunks.as<int2>(), D.d_strips.as<int2>(), D.blocks, P.arena.as<float>(),
                   P.arena.as<int>(), D.d_work.as<int>(), ctx->d_diag.as<int>(), ctx->stream);
}

static geye_status build_model_plan(geye_ctx *ctx, Plan &P, geye_model *mdl, int LEN_m, ArenaAlloc &A) {
  const HostModel &m = mdl->h;
  auto mp = std::make_unique<ModelPlan>();
  mp->model = mdl;
  mp->LEN = LEN_m;
  const int interval = m.interval, NoC = m.numcomponent, NoP = m.NoP;
  mp->root_map_off.assign((size_t)LEN_m * NoC, -1);
  mp->root_r0.assign((size_t)LEN_m * NoC, 0);
  mp->root_r1.assign((size_t)LEN_m * NoC, 0);
  mp->part_map_off.assign((size_t)LEN_m * std::max(NoP, 1), -1);
  mp->part_d0.assign((size_t)LEN_m * std::max(NoP, 1), 0);
  mp->part_d1.assign((size_t)LEN_m * std::max(NoP, 1), 0);
  mp->skipped.assign(LEN_m, 1);
  for (int level = interval; level < LEN_m; level++) {
    const LevelInfo &L = P.lv[level];
    if (L.fs0 + 2 * m.pady < m.max_Y || L.fs1 + 2 * m.padx < m.max_X) continue;   // fconvsMT.cpp:425
    mp->skipped[level] = 0;
    // roots (filter c for component c) at this level, parts at level - interval
    const int Lv = level - interval;
    std::vector<int> out_off;
    GEYE_TRY(conv_level(ctx, P, *mp, A, L, m.root_size, m.rootfilter, NoC, "root filter larger than a kept feature level", out_off));
    for (int c = 0; c < NoC; c++) {
      mp->root_map_off[level * NoC + c] = out_off[c];
      mp->root_r0[level * NoC + c] = L.fs0 - m.root_size[3 * c] + 1;
      mp->root_r1[level * NoC + c] = L.fs1 - m.root_size[3 * c + 1] + 1;
    }
    const LevelInfo &PL = P.lv[Lv];
    GEYE_TRY(conv_level(ctx, P, *mp, A, PL, m.part_size, m.partfilter, NoP, "part filter larger than its feature level", out_off));
    for (int p = 0; p < NoP; p++) {
      mp->part_map_off[Lv * NoP + p] = out_off[p];
      mp->part_d0[Lv * NoP + p] = PL.fs0 - m.part_size[3 * p] + 1;
      mp->part_d1[Lv * NoP + p] = PL.fs1 - m.part_size[3 * p + 1] + 1;
    }
    // DT per (component, part) and score jobs per component
    for (int c = 0; c < NoC; c++) {
      ScoreJob S{};
      const int r0 = mp->root_r0[level * NoC + c], r1 = mp->root_r1[level * NoC + c];
      S.root_off = mp->root_map_off[level * NoC + c];
      S.r0 = r0; S.r1 = r1;
      S.off = m.offw[m.ridx[c]];
      S.score_off = A.take((size_t)r0 * r1);
      S.np = m.numpart[c];
      S.comp = c;
      S.level = level;
      S.scale = (float)m.sbin / P.lv[level].scale;
      S.rsize0 = m.rsize[2 * c];
      S.rsize1 = m.rsize[2 * c + 1];
      int block_pad = (int)(S.scale / 2.0);
      S.RY = (int)((float)S.rsize0 * S.scale / 2.0 - 1.0 + block_pad);
      S.RX = (int)((float)S.rsize1 * S.scale / 2.0 - 1.0 + block_pad);
      mp->cap += r0 * r1;
      mp->score_max_r = std::max(mp->score_max_r, r0 * r1);
      for (int k = 0; k < S.np; k++) {
        const int p = m.pidx[c][k], di = m.didx[c][k];
        const int d0 = mp->part_d0[Lv * NoP + p], d1 = mp->part_d1[Lv * NoP + p];
        DtJob D{};
        D.in_off = mp->part_map_off[Lv * NoP + p];
        D.d0 = d0; D.d1 = d1;
        D.tmpM_off = A.take((size_t)d0 * d1);
        D.tmpI_off = A.take((size_t)d0 * d1);
        D.ax = m.def[4 * di]; D.bx = m.def[4 * di + 1]; D.ay = m.def[4 * di + 2]; D.by = m.def[4 * di + 3];
        D.negate = 1;
        // the score sum reads M at (anchor_y + 2y, anchor_x + 2x) (dt.cpp:38-55); the
        // part boxes read Ix/Iy one row and column before (get_boxes.cpp:243-258)
        D.samp_m = 1;
        D.par_y = m.anchor[di * 2 + 1] & 1;
        D.par_x = m.anchor[di * 2] & 1;
        {   // the box probes (anchor - 1 + 2k) all inside the map: no linear wrap, no entry-0 reads
          const int ay0 = m.anchor[di * 2 + 1] - 1, ax0 = m.anchor[di * 2] - 1;
          D.samp_i = ay0 >= 0 && ax0 >= 0 && ay0 + 2 * (r0 - 1) < d0 && ax0 + 2 * (r1 - 1) < d1;
        }
        // the sampled entries, stored compactly (a quarter of the map each)
        const int qy = 1 - D.par_y, qx = 1 - D.par_x;
        D.cm0 = (d0 - D.par_y + 1) >> 1;
        D.ci0 = D.samp_i ? (d0 - qy + 1) >> 1 : 0;
        D.M_off = A.take((size_t)D.cm0 * ((d1 - D.par_x + 1) >> 1));
        const size_t ni = D.samp_i ? (size_t)D.ci0 * ((d1 - qx + 1) >> 1) : (size_t)d0 * d1;
        D.Ix_off = A.take(ni);
        D.Iy_off = A.take(ni);
        mp->dt_jobs.push_back(D);
        mp->dt_max_d0 = std::max(mp->dt_max_d0, d0);
        mp->dt_max_d1 = std::max(mp->dt_max_d1, d1);
        mp->dt_bytes += 16.0 * d0 * d1;
        S.part_M[k] = D.M_off; S.part_Ix[k] = D.Ix_off; S.part_Iy[k] = D.Iy_off;
        S.part_d0[k] = d0; S.part_d1[k] = d1;
        S.part_cm0[k] = D.cm0; S.part_ci0[k] = D.ci0;
        S.ax[k] = m.anchor[di * 2] + 1;
        S.ay[k] = m.anchor[di * 2 + 1] + 1;
        S.psize0[k] = m.psize[c][2 * k];
        S.psize1[k] = m.psize[c][2 * k + 1];
        // add_part_calculation reads M up to (ax-1+2(r1-1), ay-1+2(r0-1)); the kernels trust it
        const int xmax = S.ax[k] - 1 + 2 * (r1 - 1), ymax = S.ay[k] - 1 + 2 * (r0 - 1);
        if (S.ax[k] - 1 < 0 || S.ay[k] - 1 < 0 || xmax >= d1 || ymax >= d0) {
          set_error("part anchor places a part outside its score map");
          return GEYE_ERR_UNSUPPORTED;
        }
      }
      mp->score_bytes += 8.0 * r0 * r1 + 4.0 * S.np * r0 * r1;
      mp->score_jobs.push_back(S);
    }
  }
  if (mp->dt_max_d0 > 1100 || mp->dt_max_d1 > 1100) { set_error("frame too large for the DT kernels"); return GEYE_ERR_UNSUPPORTED; }
  GEYE_TRY(plan_dt(ctx, *mp, kDtElems, mp->dt));
  GEYE_TRY(upload(ctx, mp->d_score_jobs, mp->score_jobs));
  {
    std::vector<int2> sb;
    score_block_list(mp->score_jobs, sb);
    mp->score_nblocks = (int)sb.size();
    GEYE_TRY(upload(ctx, mp->d_score_blocks, sb));
  }
  GEYE_TRY(mp->d_counts.alloc(ctx, sizeof(int) * ((size_t)std::max(mp->score_nblocks, 1) + 8)));
  P.models.push_back(std::move(mp));
  return GEYE_OK;
}

// Pyramid levels of a frame: sizes (featurepyramid.cpp.org:578-628) and jobs.
static geye_status build_pyramid_plan(geye_ctx *ctx, Plan &P, int width, int height, int LEN, int interval, int sbin,
                                      ArenaAlloc &A, int tc_planes) {
  P.width = width; P.height = height; P.LEN = LEN; P.interval = interval; P.sbin = sbin;
  P.lv.assign(LEN, LevelInfo{});
  const int sbin2 = (int)floor((double)sbin / 2.0);
  const float sc = pow(2, (1.0 / (double)interval));
  // image sizes and scales
  std::vector<int> own(LEN, 0);
  for (int ii = 0; ii < interval && ii < LEN; ii++) {
    float st = 1.0 / pow(sc, ii);
    int oh, ow;
    resize_dims(height, width, st, oh, ow);
    P.lv[ii].img_h = oh; P.lv[ii].img_w = ow; P.lv[ii].img_level = ii; own[ii] = 1;
    P.lv[ii].scale = st * 2;
    if (ii + interval < LEN) {
      P.lv[ii + interval].img_h = oh; P.lv[ii + interval].img_w = ow; P.lv[ii + interval].img_level = ii;
      P.lv[ii + interval].scale = st;
    }
    int rh = oh, rw = ow;
    for (int jj = ii + interval; jj < LEN - interval; jj += interval) {
      int nh, nw;
      resize_dims(rh, rw, 0.5f, nh, nw);
      P.lv[jj + interval].img_h = nh; P.lv[jj + interval].img_w = nw; P.lv[jj + interval].img_level = jj + interval;
      own[jj + interval] = 1;
      P.lv[jj + interval].scale = 0.5 * (P.lv[jj].scale);
      rh = nh; rw = nw;
    }
  }
  for (int l = 0; l < LEN; l++) {
    LevelInfo &L = P.lv[l];
    if (L.img_h < 3 || L.img_w < 3) { set_error("frame too small for the pyramid"); return GEYE_ERR_ARG; }
    if (own[l]) L.img_off = A.take((size_t)3 * L.img_h * L.img_w);
  }
  for (int l = 0; l < LEN; l++) {
    LevelInfo &L = P.lv[l];
    if (!own[l]) L.img_off = P.lv[L.img_level].img_off;
  }
  // resize phases: phase 0 = base levels 1..interval-1 from level 0; phase k>=1 = octave k+1
  std::vector<int> tstart, tsi;
  std::vector<float> talpha;
  auto add_taps = [&](int src, int dst, int &start_off, int &tap_off) {
    start_off = (int)tstart.size();
    tap_off = (int)tsi.size();
    std::vector<int> st, si;
    std::vector<float> al;
    build_taps(src, dst, st, si, al);
    tstart.insert(tstart.end(), st.begin(), st.end());
    tsi.insert(tsi.end(), si.begin(), si.end());
    talpha.insert(talpha.end(), al.begin(), al.end());
  };
  auto add_job = [&](std::vector<ResizeJob> &jobs, int src_level, int dst_level) {
    const LevelInfo &S = P.lv[src_level], &D = P.lv[dst_level];
    ResizeJob J{};
    J.src_off = S.img_off; J.dst_off = D.img_off; J.src_h = S.img_h; J.src_w = S.img_w; J.dst_h = D.img_h; J.dst_w = D.img_w;
    add_taps(S.img_h, D.img_h, J.v_start_off, J.v_tap_off);
    add_taps(S.img_w, D.img_w, J.h_start_off, J.h_tap_off);
    jobs.push_back(J);
    P.bytes_resize += 4.0 * 3 * (S.img_h * S.img_w + D.img_h * D.img_w);
  };
  auto add_phase = [&](const std::vector<ResizeJob> &jobs) {
    int most = 0;
    for (const ResizeJob &J : jobs) most = std::max(most, resize_blocks(J));
    P.rjobs.push_back(jobs);
    P.r_max_blocks.push_back(most);
  };
  {
    std::vector<ResizeJob> jobs;
    for (int ii = 1; ii < interval && ii < LEN; ii++) {
      if (P.lv[ii].img_h == P.lv[0].img_h && P.lv[ii].img_w == P.lv[0].img_w && 1.0 / pow(sc, ii) == 1.0) continue;
      add_job(jobs, 0, ii);
    }
    add_phase(jobs);
  }
  for (int base = 2 * interval; base < LEN; base += interval) {
    std::vector<ResizeJob> jobs;
    for (int l = base; l < std::min(base + interval, LEN); l++) add_job(jobs, P.lv[l - interval].img_level, l);
    add_phase(jobs);
  }
  P.bytes_resize += (double)3 * width * height + 12.0 * width * height;   // ingest
  // HOG
  size_t ref_words = 0;
  for (int l = 0; l < LEN; l++) {
    LevelInfo &L = P.lv[l];
    L.sbin = l < interval ? sbin2 : sbin;
    int b0, b1;
    feature_dims(L.img_h, L.img_w, L.sbin, b0, b1, L.fs0, L.fs1);
    L.feat_off = A.take(std::max<size_t>(feat_words(L.fs0, L.fs1), 1));
    if (tc_planes) {   // tc_planes planes [fs0*fs1 + kTcPlanePad][16 B]
      size_t o = (P.arena16_elems + 63) & ~size_t(63);
      L.feat16_off = (int)o;
      P.arena16_elems = o + (size_t)tc_planes * ((size_t)L.fs0 * L.fs1 + kTcPlanePad) * 8;
      // root levels in BF16 mode: the BF16 remainder planes right after (root filters
      // run on split operands, conv_tc.cu)
      if (tc_planes == 4 && l >= interval) {
        L.feat16lo_off = (int)P.arena16_elems;
        P.arena16_elems += (size_t)4 * ((size_t)L.fs0 * L.fs1 + kTcPlanePad) * 8;
      }
    }
    L.hist_off = A.take((size_t)19 * std::max(b0 * b1, 1));
    if (b0 > 0 && b1 > 0) {
      HogJob J{};
      J.img_off = L.img_off; J.h = L.img_h; J.w = L.img_w; J.sbin = L.sbin; J.b0 = b0; J.b1 = b1;
      J.hist_off = L.hist_off; J.fs0 = L.fs0; J.fs1 = L.fs1; J.feat_off = L.feat_off; J.feat16_off = L.feat16_off;
      J.feat16lo_off = L.feat16lo_off;
      J.ref_off = (int)ref_words;
      J.tc_planes = tc_planes;
      J.fast = tc_planes ? 1 : 0;
      J.corner_off = A.take((size_t)(L.fs0 + 1) * (L.fs1 + 1));
      J.mag_off = L.img_level;   // resolved below, once the image's pixel buffer is placed
      P.hog_jobs.push_back(J);
      P.hog_max_b0 = std::max(P.hog_max_b0, b0);
      P.hog_max_b1 = std::max(P.hog_max_b1, b1);
      P.bytes_hog += 12.0 * L.img_h * L.img_w + 124.0 * L.fs0 * L.fs1;
    }
    ref_words += (size_t)kFeat * L.fs0 * L.fs1;
  }
  // one (bin, magnitude) buffer per image, covering the widest visible area of its levels
  {
    std::map<int, int> pix_of;   // image level -> pix job
    for (auto &J : P.hog_jobs) {
      const int il = J.mag_off;
      auto it = pix_of.find(il);
      if (it == pix_of.end()) {
        HogPixJob X{};
        X.img_off = J.img_off; X.h = J.h; X.w = J.w;
        it = pix_of.emplace(il, (int)P.pix_jobs.size()).first;
        P.pix_jobs.push_back(X);
      }
      HogPixJob &X = P.pix_jobs[it->second];
      X.xe = std::max(X.xe, J.b1 * J.sbin - 1);
      X.ye = std::max(X.ye, J.b0 * J.sbin - 1);
    }
    for (auto &X : P.pix_jobs) {
      X.Y = (X.ye + 4) & ~3;
      const size_t n = (size_t)(X.xe + 1) * X.Y;
      X.mag_off = A.take(n);
      X.bin_off = A.take((n + 3) / 4);
      P.pix_max_xe = std::max(P.pix_max_xe, X.xe);
      P.bytes_hog += 5.0 * n;
    }
    for (auto &J : P.hog_jobs) {
      const HogPixJob &X = P.pix_jobs[pix_of[J.mag_off]];
      J.mag_off = X.mag_off; J.bin_off = X.bin_off; J.pix_Y = X.Y;
    }
  }
  GEYE_TRY(upload(ctx, P.d_tap_start, tstart));
  GEYE_TRY(upload(ctx, P.d_tap_si, tsi));
  GEYE_TRY(upload(ctx, P.d_tap_alpha, talpha));
  P.d_rjobs.resize(P.rjobs.size());
  for (size_t i = 0; i < P.rjobs.size(); i++) GEYE_TRY(upload(ctx, P.d_rjobs[i], P.rjobs[i]));
  GEYE_TRY(upload(ctx, P.d_hog_jobs, P.hog_jobs));
  {
    std::vector<int2> vb;
    hog_vote_blocks(P.hog_jobs, vb);
    P.hog_vote_nblocks = (int)vb.size();
    GEYE_TRY(upload(ctx, P.d_hog_vote_blocks, vb));
  }
  GEYE_TRY(upload(ctx, P.d_pix_jobs, P.pix_jobs));
  return GEYE_OK;
}

static geye_status finish_plan(geye_ctx *ctx, Plan &P, ArenaAlloc &A) {
  if (!P.conv_jobs.empty()) {
    std::vector<int2> blocks;
    P.conv_smem = conv_fp32_blocks(P.conv_jobs, blocks);
    P.conv_nblocks = (int)blocks.size();
    GEYE_TRY(upload(ctx, P.d_conv_jobs, P.conv_jobs));
    GEYE_TRY(upload(ctx, P.d_conv_blocks, blocks));
    GEYE_TRY(upload(ctx, P.d_conv_bank, P.conv_bank.taps));
    P.conv_bank = ConvBank();
  }
  P.arena_words = A.words + 64;
  GEYE_TRY(P.arena.alloc(ctx, P.arena_words * 4));
  if (P.arena16_elems) {
    // after the last plane, a tail that slabs of filters smaller than their group's
    // tap grid may read (the widest filter's columns of the largest level)
    int fb0 = 1, fb1 = 1, fs0 = 1;
    for (auto &mp : P.models) {
      const HostModel &h = mp->model->h;
      for (int r = 0; r < h.NoR; r++) { fb0 = std::max(fb0, h.root_size[3 * r]); fb1 = std::max(fb1, h.root_size[3 * r + 1]); }
      for (int q = 0; q < h.NoP; q++) { fb0 = std::max(fb0, h.part_size[3 * q]); fb1 = std::max(fb1, h.part_size[3 * q + 1]); }
    }
    for (auto &L : P.lv) fs0 = std::max(fs0, L.fs0);
    P.arena16_elems += ((size_t)fb1 * fs0 + fb0 + 16 * 128) * 8;
    GEYE_TRY(P.arena16.alloc(ctx, P.arena16_elems * 2));
    // plane tails are read (and their outputs discarded) but never written: keep them zero
    CUDA_TRY(cudaMemsetAsync(P.arena16.p, 0, P.arena16_elems * 2, ctx->stream));
  }
  int cap = 0;
  for (auto &mp : P.models) cap = std::max(cap, mp->cap);
  // multiple of 32: per-model NMS scratch (int2 queues) stays 8-byte aligned
  P.max_cap = (std::max(cap, 1) + 31) & ~31;
  const size_t nm = std::max<size_t>(P.models.size(), 1);
  GEYE_TRY(P.d_nms_f.alloc(ctx, sizeof(float) * nm * P.max_cap * 16));
  GEYE_TRY(P.d_nms_i.alloc(ctx, sizeof(int) * nm * nms_model_words(P.max_cap)));
  GEYE_TRY(P.d_small.alloc(ctx, 4096));
  if (P.width > 0) {
    GEYE_TRY(P.d_ascore.alloc(ctx, sizeof(float) * nm * P.width * P.height));
    // A_SCORE lookups (get_boxes.cpp:265-300): per score map, the score column of every
    // image column X and the score row of every image row Y, or -1 where the
    // reference's loop maps nothing there; the division is the reference's float one.
    for (auto &mp : P.models) {
      const int nj = (int)mp->score_jobs.size();
      std::vector<int> col((size_t)nj * P.width), row((size_t)nj * P.height);
      for (int j = 0; j < nj; j++) {
        const ScoreJob &S = mp->score_jobs[j];
        for (int X = 0; X < P.width; X++) {
          const int ii = X - S.RX;
          const int Xn = ii < 0 ? -1 : (int)((float)ii / S.scale + 0);
          col[(size_t)j * P.width + X] = (Xn >= 0 && Xn < S.r1) ? S.score_off + Xn * S.r0 : -1;
        }
        for (int Y = 0; Y < P.height; Y++) {
          const int jj = Y - S.RY;
          const int Yn = jj < 0 ? -1 : (int)((float)jj / S.scale + 0);
          row[(size_t)j * P.height + Y] = (Yn >= 0 && Yn < S.r0) ? Yn : -1;
        }
      }
      GEYE_TRY(upload(ctx, mp->d_as_col, col));
      GEYE_TRY(upload(ctx, mp->d_as_row, row));
    }
  }
  // result arrays: point, or_point (4 ints each), type, scale, score per kept box
  GEYE_TRY(P.d_result.alloc(ctx, nm * (size_t)P.max_cap * 11 * 4));
  P.last_D.assign(nm, 0);
  P.last_K.assign(nm, 0);
  return GEYE_OK;
}

static std::string plan_key(int width, int height, geye_model *const *models, int n, const int *LENs, int mode) {
  std::ostringstream os;
  os << width << "x" << height << "m" << mode;
  for (int i = 0; i < n; i++) os << ":" << models[i]->id << "/" << LENs[i];
  return os.str();
}

static geye_status get_frame_plan(geye_ctx *ctx, geye_model *const *models, int n_models, int width, int height,
                                  Plan **out) {
  if (n_models <= 0 || n_models > 16) { set_error("n_models out of range"); return GEYE_ERR_ARG; }
  const int interval = models[0]->h.interval, sbin = models[0]->h.sbin;
  std::vector<int> LENs(n_models);
  int LEN = 0;
  for (int i = 0; i < n_models; i++) {
    geye_model *m = models[i];
    if (m->h.interval != interval || m->h.sbin != sbin) {
      set_error("models in one call must share sbin and interval");
      return GEYE_ERR_UNSUPPORTED;
    }
    // ini_scales latch (featurepyramid.cpp:178-236)
    if (m->ini) {
      m->max_scale = max_scale_for(m->h, width, height);
      m->ini = false;
    }
    LENs[i] = m->max_scale + interval;
    LEN = std::max(LEN, LENs[i]);
  }
  const int tc_planes = ctx->conv_mode == GEYE_CONV_BF16 ? 4 : ctx->conv_mode == GEYE_CONV_FP8 ? 2 : 0;
  std::string key = plan_key(width, height, models, n_models, LENs.data(), (int)ctx->conv_mode);
  auto it = ctx->plans.find(key);
  if (it != ctx->plans.end()) { *out = it->second.get(); return GEYE_OK; }
  auto P = std::make_unique<Plan>();
  ArenaAlloc A;
  GEYE_TRY(build_pyramid_plan(ctx, *P, width, height, LEN, interval, sbin, A, tc_planes));
  for (int i = 0; i < n_models; i++) GEYE_TRY(build_model_plan(ctx, *P, models[i], LENs[i], A));
  if (ctx->conv_mode != GEYE_CONV_FP32) GEYE_TRY(plan_tc(ctx, *P, A));
  GEYE_TRY(finish_plan(ctx, *P, A));
  // after the arena exists: the tile shapes are tuned on it
  if (ctx->conv_mode != GEYE_CONV_FP32) GEYE_TRY(build_tc_plan(ctx, *P));
  GEYE_TRY(P->d_bgr.alloc(ctx, (size_t)width * height * 3 + 64));
  CUDA_TRY(cudaMallocHost(&P->h_res, sizeof(int) * res_block_ints(n_models)));
  if (ctx->plans.size() > 32) ctx->plans.clear();
  *out = P.get();
  ctx->plans[key] = std::move(P);
  return GEYE_OK;
}

// ----------------------------------------------------------------------------
// pipeline
// ----------------------------------------------------------------------------
enum { ST_PYR = 0, ST_HOG, ST_CONV, ST_DT, ST_SCORE, ST_NMS, ST_TOTAL };

struct StageTimer {
  geye_ctx *ctx;
  explicit StageTimer(geye_ctx *c) : ctx(c) {}
  void mark(int i) {
    if (!ctx->timing) return;
    // inside a capture the record becomes an event-record node of the graph
    if (ctx->capturing) cudaEventRecordWithFlags(ctx->ev[i], ctx->stream, cudaEventRecordExternal);
    else cudaEventRecord(ctx->ev[i], ctx->stream);
  }
};

static geye_status check_launch(geye_ctx *ctx, const char *what) {
  ctx->launches++;
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_error(std::string(what) + ": " + cudaGetErrorString(e));
    return GEYE_ERR_CUDA;
  }
  return GEYE_OK;
}

geye_status run_ingest(geye_ctx *ctx, Plan &P, const uint8_t *d_bgr, int width_step) {
  if (injected(ctx, "launch")) { set_error("injected launch failure"); return GEYE_ERR_INJECTED; }
  launch_ingest(d_bgr, P.width, P.height, width_step, P.arena.as<float>() + P.lv[0].img_off, ctx->stream);
  return check_launch(ctx, "ingest");
}

geye_status run_resize(geye_ctx *ctx, Plan &P) {
  cudaStream_t s = ctx->stream;
  float *arena = P.arena.as<float>();
  for (size_t ph = 0; ph < P.rjobs.size(); ph++) {
    if (P.rjobs[ph].empty()) continue;
    launch_resize(P.d_rjobs[ph].as<ResizeJob>(), (int)P.rjobs[ph].size(), P.r_max_blocks[ph], P.d_tap_start.as<int>(),
                  P.d_tap_si.as<int>(), P.d_tap_alpha.as<float>(), arena, s);
    GEYE_TRY(check_launch(ctx, "resize"));
  }
  return GEYE_OK;
}

geye_status run_pyramid(geye_ctx *ctx, Plan &P, const uint8_t *d_bgr, int width_step) {
  GEYE_TRY(run_ingest(ctx, P, d_bgr, width_step));
  return run_resize(ctx, P);
}

// floats: also write the float feature planes (for the FP32 convolution), or (ref) the levels in the reference layout there
geye_status run_hog(geye_ctx *ctx, Plan &P, bool floats, float *ref) {
  const bool fast = !P.hog_jobs.empty() && P.hog_jobs[0].fast;
  launch_hog(P.d_hog_jobs.as<HogJob>(), (int)P.hog_jobs.size(), P.d_hog_vote_blocks.as<int2>(), P.hog_vote_nblocks,
             P.hog_max_b0, P.hog_max_b1, P.d_pix_jobs.as<HogPixJob>(), (int)P.pix_jobs.size(), P.pix_max_xe,
             P.arena.as<float>(), P.arena16.p, !fast, floats, ref, ctx->stream);
  ctx->launches += 3;   // pixels, votes, corner norms, features
  return check_launch(ctx, "hog");
}

// FP32 convolution of every model, roots and parts (the tensor-core modes: run_conv_tc)
geye_status run_conv(geye_ctx *ctx, Plan &P) {
  if (!P.conv_nblocks) return GEYE_OK;
  launch_conv_fp32(P.d_conv_jobs.as<ConvJob>(), P.d_conv_blocks.as<int2>(), P.conv_nblocks, P.conv_smem,
                   P.d_conv_bank.as<float>(), P.arena.as<float>(), P.arena.as<float>(), ctx->stream);
  return check_launch(ctx, "conv");
}

geye_status run_dt(geye_ctx *ctx, Plan &P, ModelPlan &mp) {
  if (mp.dt_jobs.empty()) return GEYE_OK;
  if (launch_plan_dt(ctx, P, *mp.dt) != cudaSuccess) {
    set_error("dt launch");
    return GEYE_ERR_CUDA;
  }
  ctx->launches++;
  return check_launch(ctx, "dt");
}

// DT tile size of each model of a plan, timed on the maps its last frame left
// in the arena (the DT's cost depends on the values: they set the window
// bounds and whether the argmin order is proven): each of kDtElemsChoices
// runs once untimed and three times timed with CUDA events on the context's
// stream, and the fastest is kept.  A DT run rewrites its outputs from its
// inputs, so the frame's results are unchanged.  Returns true when a plan's
// block lists changed (its frame graphs must be captured again).
static bool tune_dt(geye_ctx *ctx, Plan &P) {
  bool changed = false;
  for (auto &mpp : P.models) {
    ModelPlan &mp = *mpp;
    if (mp.dt_tuned || mp.dt_jobs.empty()) continue;
    mp.dt_tuned = true;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    if (cudaEventCreate(&e0) != cudaSuccess || cudaEventCreate(&e1) != cudaSuccess) {
      if (e0) cudaEventDestroy(e0);
      return changed;
    }
    int best = -1;
    std::unique_ptr<DtPlan> trial[3];
    for (int c = 0; c < 3; c++) {
      const bool own = kDtElemsChoices[c] == mp.dt->elems;
      if (!own && plan_dt(ctx, mp, kDtElemsChoices[c], trial[c]) != GEYE_OK) break;
      float ms = 0.f;
      cudaError_t e = cudaSuccess;
      for (int rep = 0; rep < 4 && e == cudaSuccess; rep++) {
        if (rep == 1) cudaEventRecord(e0, ctx->stream);
        e = launch_plan_dt(ctx, P, own ? *mp.dt : *trial[c]);
      }
      cudaEventRecord(e1, ctx->stream);
      if (cudaEventSynchronize(e1) != cudaSuccess || e != cudaSuccess || cudaEventElapsedTime(&ms, e0, e1) != cudaSuccess) break;
      mp.dt_ms[c] = ms / 3.0f;
      if (best < 0 || mp.dt_ms[c] < mp.dt_ms[best]) best = c;
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaGetLastError();
    if (best >= 0 && trial[best]) {
      mp.dt = std::move(trial[best]);
      changed = true;
    }
  }
  return changed;
}

// score maps and detections: the count at d_small[mi], the NMS candidates, or (records) the whole records there
geye_status run_score(geye_ctx *ctx, Plan &P, ModelPlan &mp, int mi, float thresh, float *records) {
  int *counts = mp.d_counts.as<int>();
  int *d_num = P.d_small.as<int>() + mi;
  const int nj = (int)mp.score_jobs.size();
  if (nj == 0) {
    CUDA_TRY(cudaMemsetAsync(d_num, 0, sizeof(int), ctx->stream));
    return GEYE_OK;
  }
  launch_score(mp.d_score_jobs.as<ScoreJob>(), mp.d_score_blocks.as<int2>(), mp.score_nblocks, thresh,
               P.arena.as<float>(), counts, ctx->stream);
  GEYE_TRY(check_launch(ctx, "score"));
  launch_scan_counts(counts, mp.score_nblocks, d_num, ctx->stream);
  GEYE_TRY(check_launch(ctx, "scan"));
  if (records)
    launch_boxes(mp.d_score_jobs.as<ScoreJob>(), mp.d_score_blocks.as<int2>(), mp.score_nblocks, thresh,
                 P.arena.as<float>(), P.arena.as<int>(), counts, mp.model->gl(), records, ctx->stream);
  else
    launch_candidates(mp.d_score_jobs.as<ScoreJob>(), mp.d_score_blocks.as<int2>(), mp.score_nblocks, thresh,
                      P.arena.as<float>(), counts, nms_candidates(P.d_nms_f.as<float>(), mi, P.max_cap), ctx->stream);
  return check_launch(ctx, "boxes");
}

// A_SCORE starts from the caller's map or from ini_ac_score's -100 (detect.cpp:136-145)
static geye_status ascore_init(geye_ctx *ctx, Plan &P, int mi, const float *h_init) {
  float *a = P.d_ascore.as<float>() + (size_t)mi * P.width * P.height;
  const size_t n = (size_t)P.width * P.height;
  if (h_init) {
    if (injected(ctx, "h2d")) { set_error("injected host-to-device copy failure"); return GEYE_ERR_INJECTED; }
    CUDA_TRY(cudaMemcpyAsync(a, h_init, n * sizeof(float), cudaMemcpyHostToDevice, ctx->stream));
    return GEYE_OK;
  }
  launch_fill(a, n, -100.0f, ctx->stream);
  return check_launch(ctx, "fill");
}

static geye_status ascore_compute(geye_ctx *ctx, Plan &P, ModelPlan &mp, int mi, float thresh, cudaStream_t s) {
  float *a = P.d_ascore.as<float>() + (size_t)mi * P.width * P.height;
  const size_t n = (size_t)P.width * P.height;
  unsigned *maxb = reinterpret_cast<unsigned *>(P.d_small.as<int>() + 64 + mi);
  CUDA_TRY(cudaMemsetAsync(maxb, 0, sizeof(unsigned), s));
  launch_ascore(mp.d_as_col.as<int>(), mp.d_as_row.as<int>(), (int)mp.score_jobs.size(), P.arena.as<float>(), a,
                P.width, P.height, thresh, maxb, s);
  GEYE_TRY(check_launch(ctx, "a_score"));
  launch_ascore_normalize(a, (int)n, maxb, s);
  return check_launch(ctx, "a_score normalise");
}

geye_status run_ascore(geye_ctx *ctx, Plan &P, ModelPlan &mp, int mi, float thresh, const float *h_init) {
  GEYE_TRY(ascore_init(ctx, P, mi, h_init));
  return ascore_compute(ctx, P, mp, mi, thresh, ctx->stream);
}

// After a plan's first frame has completed: its DT tile sizes are tuned, once, on that frame's maps
// (tune_dt).  A change drops the plan's frame graphs after its stream has
// drained; the next frame captures them again.
void tune_plan(geye_ctx *ctx, Plan &P) {
  if (P.from_features || !tune_dt(ctx, P)) return;   // (behind the frame on its stream)
  cudaStreamSynchronize(ctx->stream);
  for (auto &g : P.graphs)
    if (g.second.exec) cudaGraphExecDestroy(g.second.exec);
  P.graphs.clear();
}

geye_status run_nms(geye_ctx *ctx, Plan &P, int n_models, float overlap) {
  int *d_num = P.d_small.as<int>();
  int *d_kept = d_num + 32;
  int *err = d_num + 128;
  NmsResults res{};
  for (int mi = 0; mi < n_models; mi++) {
    geye_model *m = P.models[mi]->model;
    res.m[mi] = {m->d_coef, m->h.numpart[0], m->h.ratio, P.models[mi]->d_score_jobs.as<ScoreJob>(),
                 P.models[mi]->d_score_blocks.as<int2>()};
  }
  res.arena_i = P.arena.as<int>();
  res.out = P.d_result.as<int>();
  res.host = static_cast<int *>(P.h_res);
  res.host_cap = kHostRes;
  res.img_w = P.width;
  res.img_h = P.height;
  const cudaError_t ge =
      launch_nms_batch(d_num, n_models, overlap,
                       P.max_cap, P.d_nms_i.as<int>(),
                       P.d_nms_f.as<float>(), res, d_kept, err, reinterpret_cast<long long *>(d_num + 512),
                       d_num + kNmsNeed, ctx->nms_order, ctx->stream,
                       (ctx->capturing && ctx->nms_if_node) ? ctx->aux : nullptr);
  if (ge != cudaSuccess) {
    set_error(std::string("nms graph nodes: ") + cudaGetErrorString(ge));
    return GEYE_ERR_CUDA;
  }
  return check_launch(ctx, "nms");
}

// Everything after the ingest and the A_SCORE initialisation: plan-static, so
// it is captured once per (plan, threshold, overlap, timing) as a CUDA graph.
static geye_status run_body(geye_ctx *ctx, Plan &P, float thresh, float overlap) {
  StageTimer T(ctx);
  if (!ctx->front_external) GEYE_TRY(run_resize(ctx, P));
  T.mark(1);
  if (!ctx->front_external) GEYE_TRY(run_hog(ctx, P, ctx->conv_mode == GEYE_CONV_FP32, nullptr));
  T.mark(2);
  const bool tc = ctx->conv_mode != GEYE_CONV_FP32;
  GEYE_TRY(tc ? run_conv_tc(ctx, P) : run_conv(ctx, P));   // every model's filters in one launch
  if (ctx->timing || P.models.size() < 2) {   // stage by stage (per-stage times)
    T.mark(3);
    for (auto &mp : P.models) GEYE_TRY(run_dt(ctx, P, *mp));
    T.mark(4);
    for (size_t mi = 0; mi < P.models.size(); mi++) GEYE_TRY(run_score(ctx, P, *P.models[mi], (int)mi, thresh, nullptr));
  } else {
    // each model's DT -> score chain reads only the conv maps and writes only its
    // own maps and records: models 1.. run on the side stream beside model 0
    // (their kernels take the context's stream, swapped while they are issued),
    // joined before NMS
    auto chain = [&](size_t mi) -> geye_status {
      GEYE_TRY(run_dt(ctx, P, *P.models[mi]));
      return run_score(ctx, P, *P.models[mi], (int)mi, thresh, nullptr);
    };
    CUDA_TRY(cudaEventRecord(ctx->ev_fork, ctx->stream));
    CUDA_TRY(cudaStreamWaitEvent(ctx->side, ctx->ev_fork, 0));
    std::swap(ctx->stream, ctx->side);
    geye_status st1 = GEYE_OK;
    for (size_t mi = 1; mi < P.models.size() && st1 == GEYE_OK; mi++) st1 = chain(mi);
    std::swap(ctx->stream, ctx->side);
    CUDA_TRY(cudaEventRecord(ctx->ev_join, ctx->side));
    const geye_status st0 = chain(0);
    CUDA_TRY(cudaStreamWaitEvent(ctx->stream, ctx->ev_join, 0));   // joined on every path
    GEYE_TRY(st0);
    GEYE_TRY(st1);
  }
  T.mark(5);
  // A_SCORE feeds nothing in the frame: it runs on the side stream beside NMS
  CUDA_TRY(cudaEventRecord(ctx->ev_fork, ctx->stream));
  CUDA_TRY(cudaStreamWaitEvent(ctx->side, ctx->ev_fork, 0));
  geye_status st = GEYE_OK;
  for (size_t mi = 0; mi < P.models.size() && st == GEYE_OK; mi++)
    st = ascore_compute(ctx, P, *P.models[mi], (int)mi, thresh, ctx->side);
  CUDA_TRY(cudaEventRecord(ctx->ev_join, ctx->side));
  if (st == GEYE_OK) st = run_nms(ctx, P, (int)P.models.size(), overlap);
  CUDA_TRY(cudaStreamWaitEvent(ctx->stream, ctx->ev_join, 0));   // joined on every path
  GEYE_TRY(st);
  T.mark(6);
  return GEYE_OK;
}

static geye_status run_body_graph(geye_ctx *ctx, Plan &P, float thresh, float overlap) {
  char key[64];
  unsigned tb, ob;
  memcpy(&tb, &thresh, 4);
  memcpy(&ob, &overlap, 4);
  snprintf(key, sizeof key, "%08x:%08x:%d:%d", tb, ob, ctx->timing ? 1 : 0, ctx->nms_order);
  Plan::FrameGraph &g = P.graphs[key];
  if (!g.exec) {
    const int before = ctx->launches;
    cudaGraph_t graph = nullptr;
    ctx->capturing = true;
    CUDA_TRY(cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeRelaxed));
    const geye_status st = run_body(ctx, P, thresh, overlap);
    const cudaError_t e = cudaStreamEndCapture(ctx->stream, &graph);
    ctx->capturing = false;
    ctx->launches = before;
    if (st != GEYE_OK) {
      if (graph) cudaGraphDestroy(graph);
      P.graphs.erase(key);
      return st;
    }
    if (e != cudaSuccess) {
      P.graphs.erase(key);
      set_error(std::string("frame graph capture: ") + cudaGetErrorString(e));
      return GEYE_ERR_CUDA;
    }
    size_t n = 0;
    cudaGraphGetNodes(graph, nullptr, &n);
    std::vector<cudaGraphNode_t> nodes(n);
    if (n) cudaGraphGetNodes(graph, nodes.data(), &n);
    int kernels = 0;
    for (auto nd : nodes) {
      cudaGraphNodeType t;
      if (cudaGraphNodeGetType(nd, &t) == cudaSuccess && t == cudaGraphNodeTypeKernel) kernels++;
    }
    const cudaError_t ie = cudaGraphInstantiate(&g.exec, graph, 0);
    cudaGraphDestroy(graph);
    if (ie != cudaSuccess) {
      g.exec = nullptr;
      P.graphs.erase(key);
      set_error(std::string("frame graph instantiate: ") + cudaGetErrorString(ie));
      return GEYE_ERR_CUDA;
    }
    g.kernels = kernels;
  }
  CUDA_TRY(cudaGraphLaunch(g.exec, ctx->stream));
  ctx->launches += g.kernels;
  return GEYE_OK;
}

// Whole path for n models on a frame already on the device.
geye_status run_frame(geye_ctx *ctx, Plan &P, const uint8_t *d_bgr, int width_step, float thresh, float overlap,
                      const float *const *h_ascore_init) {
  GEYE_TRY(park_pending(ctx, P));
  StageTimer T(ctx);
  ctx->launches = 0;
  CUDA_TRY(cudaMemsetAsync(P.d_small.p, 0, 4096, ctx->stream));
  T.mark(0);
  if (!ctx->front_external) GEYE_TRY(run_ingest(ctx, P, d_bgr, width_step));
  for (size_t mi = 0; mi < P.models.size(); mi++)
    GEYE_TRY(ascore_init(ctx, P, (int)mi, h_ascore_init ? h_ascore_init[mi] : nullptr));
  if (ctx->use_graphs) GEYE_TRY(run_body_graph(ctx, P, thresh, overlap));
  else GEYE_TRY(run_body(ctx, P, thresh, overlap));
  if (ctx->timing) {
    // stage bytes / flops for the roofline report
    double conv_b = 0, conv_f = 0, dt_b = 0, sc_b = 0;
    for (auto &mp : P.models) { conv_b += mp->conv_bytes; conv_f += mp->conv_flops; dt_b += mp->dt_bytes; sc_b += mp->score_bytes; }
    ctx->stage_bytes[ST_PYR] = P.bytes_resize;
    ctx->stage_bytes[ST_HOG] = P.bytes_hog;
    ctx->stage_bytes[ST_CONV] = conv_b;
    ctx->stage_bytes[ST_DT] = dt_b;
    ctx->stage_bytes[ST_SCORE] = sc_b;
    ctx->stage_bytes[ST_NMS] = 0;
    ctx->stage_bytes[ST_TOTAL] = P.bytes_resize + P.bytes_hog + conv_b + dt_b + sc_b;
    ctx->conv_flops = conv_f;
  }
  ctx->last_plan = &P;
  return GEYE_OK;
}

geye_status collect_stage_times(geye_ctx *ctx) {
  if (!ctx->timing) return GEYE_OK;
  CUDA_TRY(cudaEventSynchronize(ctx->ev[6]));
  for (int i = 0; i < 6; i++) CUDA_TRY(cudaEventElapsedTime(&ctx->stage_ms[i], ctx->ev[i], ctx->ev[i + 1]));
  CUDA_TRY(cudaEventElapsedTime(&ctx->stage_ms[6], ctx->ev[0], ctx->ev[6]));
  return GEYE_OK;
}

geye_status frame_plan(geye_ctx *ctx, geye_model *const *models, int n, int w, int h, Plan **out) {
  return get_frame_plan(ctx, models, n, w, h, out);
}

void drop_frame_plans(geye_ctx *ctx, int w, int h) {
  for (auto it = ctx->plans.begin(); it != ctx->plans.end();) {
    Plan *P = it->second.get();
    if (!P->from_features && P->width == w && P->height == h) {
      if (ctx->last_plan == P) ctx->last_plan = nullptr;
      if (ctx->pending == P) ctx->pending = nullptr;
      it = ctx->plans.erase(it);
    } else {
      ++it;
    }
  }
}

geye_status parse_model_files(const char *c, const char *r, const char *p, HostModel &m) { return parse_model(c, r, p, m); }

int model_max_scale(const HostModel &m, int w, int h) { return max_scale_for(m, w, h); }

}  // namespace geye

namespace geye {

const char *last_error_cstr() { return g_err.c_str(); }

// Plan over caller-supplied features (get_boxes stage entry point): no images,
// levels take their sizes and scales from the caller.
geye_status features_plan(geye_ctx *ctx, geye_model *model, const int *ftsize, const float *scales, int n_levels,
                          int img_w, int img_h, Plan **out) {
  const HostModel &m = model->h;
  auto P = std::make_unique<Plan>();
  P->from_features = true;
  P->width = img_w;
  P->height = img_h;
  P->interval = m.interval;
  P->sbin = m.sbin;
  P->LEN = n_levels;
  P->lv.assign(n_levels, LevelInfo{});
  ArenaAlloc A;
  for (int l = 0; l < n_levels; l++) {
    LevelInfo &L = P->lv[l];
    L.fs0 = ftsize[2 * l];
    L.fs1 = ftsize[2 * l + 1];
    L.scale = scales[l];
    L.sbin = l < m.interval ? m.sbin / 2 : m.sbin;
    L.feat_off = A.take(std::max<size_t>(feat_words(L.fs0, L.fs1), 1));
  }
  GEYE_TRY(build_model_plan(ctx, *P, model, n_levels, A));
  GEYE_TRY(finish_plan(ctx, *P, A));
  std::string key = "features:" + std::to_string((uintptr_t)P.get());
  *out = P.get();
  ctx->plans[key] = std::move(P);
  return GEYE_OK;
}

void drop_plan(geye_ctx *ctx, Plan *P) {
  for (auto it = ctx->plans.begin(); it != ctx->plans.end(); ++it)
    if (it->second.get() == P) {
      if (ctx->last_plan == P) ctx->last_plan = nullptr;
      ctx->plans.erase(it);
      return;
    }
}

}  // namespace geye
