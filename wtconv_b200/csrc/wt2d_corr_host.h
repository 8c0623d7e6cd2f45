// Planner of the parameter-gradient launches (see wt2d_corr.cuh).
#pragma once

#include <vector>

#include "wt2d_host.h"

namespace wt {

struct CorrStage {
  PlanarStage p;
  int deep = 0;                 // 1: wt2d_corr_deep_kernel
  int nsplit = 1, gvec = 1;
  int level = 1;                // first layer level of the stage (1-based)
  long long in_off = -1;        // floats into the scratch: low-pass planes of the input read (the gradient's follow), -1: the tensors
  long long out_off = -1;       // low-pass planes written, -1: none
};
struct CorrChain {
  std::vector<CorrStage> stages;
  long long scratch_floats = 0;
  int status = 0;
};

// One level (nlev 1) or the base path alone (nlev 0) of a plane set: the channel group and tile that keep most
// warps busy for the work they add (halo cells are loaded and transformed again by every tile).
inline bool plan_corr_level(PlanarStage& p, int B, int C, int K, int H, int W, int nlev, bool base, const long long* xs, int elem, int align) {
  PlanarStage best = PlanarStage();
  double best_score = 0.0;
  const bool cl = xs[1] == 1 && C > 1;
  const int h1 = cdiv(H, 2), w1 = cdiv(W, 2), HS = K / 2;
  for (int G = 8; G >= 1; G /= 2) {
    if (G > 1 && G / 2 >= C) continue;
    for (int pick = 0; pick < 8; ++pick) {
      static const int rows[8] = {0, 32, 24, 16, 12, 8, 32, 16};          // 0: whole planes; the last two: tiles of 16 columns
      p = PlanarStage();
      p.B = B; p.C = C; p.K = K; p.nlev = nlev; p.lvl0 = 0; p.has_base = base ? 1 : 0;
      p.ctas = K <= 5 ? 2 : 1; p.frames_only = 1;
      p.h[0] = H; p.w[0] = W; p.h[1] = h1; p.w[1] = w1;
      p.Hsrc = H; p.Wsrc = W;
      for (int i = 0; i < 4; ++i) p.xs[i] = xs[i];
      p.xvec = row_vec(xs, elem, align);
      if (cl)
        for (int bytes = 16; bytes >= 4 && !p.xchunk; bytes /= 2) {
          const int v = bytes / elem;
          if (v <= G && align >= bytes && xs[0] % v == 0 && xs[2] % v == 0 && xs[3] % v == 0) p.xchunk = v;
        }
      p.G = G;
      p.tiled = pick > 0 ? 1 : 0;
      double work = 1.0;
      if (!p.tiled) {
        if (h1 > 64 || w1 > 64) continue;
        p.TH = round_up(h1, 4); p.TW = round_up(w1, 4);
      } else {
        const int th = rows[pick], tw = pick >= 6 ? 16 : 32;
        if (th >= round_up(h1, 4) && tw >= round_up(w1, 4)) continue;     // the whole plane
        p.TH = round_up(cdiv(h1, cdiv(h1, th)), 4); p.TW = round_up(cdiv(w1, cdiv(w1, tw)), 4);
        work = (58.0 + 25.0 * (p.TH + 2 * HS) * (p.TW + 2 * HS) / ((double)p.TH * p.TW)) / 83.0;
      }
      planar_layout(p);
      const int red = p.nthreads / 32 * 5 * (K * K + 1) * G;              // the final sums share the frames' space
      p.smem_bytes = 4 * (p.zero_floats > red ? p.zero_floats : red);
      if (p.smem_bytes > (K <= 5 ? kSmemTwoPerSm : kSmemLimitBytes)) continue;
      double score = p.score / work;
      if (cl) score *= p.xchunk * elem >= 16 ? 1.0 : p.xchunk * elem == 8 ? 0.8 : p.xchunk ? 0.5 : 0.3;
      if (score > best_score * 1.03) { best_score = score; best = p; }
    }
  }
  if (best_score == 0.0) return false;
  p = best;
  return true;
}

inline CorrChain plan_corr(const Layer2d& ly) {          // ly.ys / y_align: the output gradient at full resolution
  CorrChain ch;
  std::vector<int> Hl(ly.L + 1), Wl(ly.L + 1);
  Hl[0] = ly.H; Wl[0] = ly.W;
  for (int j = 1; j <= ly.L; ++j) { Hl[j] = (Hl[j - 1] + 1) / 2; Wl[j] = (Wl[j - 1] + 1) / 2; }
  auto tiles = [&](int j) { return cdiv(Hl[j], 4) * cdiv(Wl[j], 4); };
  int deep = ly.L + 1, sum = 0;                          // first level of the deep kernel
  while (deep > 2 && ly.L - deep + 2 <= kPlanarMaxLev && sum + tiles(deep - 1) <= 8) sum += tiles(--deep);
  long long off = 0, in = -1;
  auto resident = [](const PlanarStage& p) { return planar_resident(p); };
  for (int j = 1; j < deep || j == 1; ++j) {
    CorrStage st;
    const int nlev = ly.L == 0 ? 0 : 1;
    const long long hw = (long long)Hl[j - 1] * Wl[j - 1];
    const long long dense[4] = {ly.C * hw, hw, Wl[j - 1], 1};
    if (!plan_corr_level(st.p, ly.B, ly.C, ly.K, Hl[j - 1], Wl[j - 1], nlev, j == 1, j == 1 ? ly.xs : dense, j == 1 ? ly.elem_size : 4,
                         j == 1 ? ly.x_align : 16)) { ch.status = -6; return ch; }
    st.gvec = j == 1 ? row_vec(ly.ys, ly.elem_size, ly.y_align) : row_vec(dense, 4, 16);
    st.level = j;
    st.in_off = in;
    if (j < ly.L) {                                      // both tensors' low-pass planes for the next stage
      st.out_off = off;
      off += 2 * (((long long)ly.B * ly.C * Hl[j] * Wl[j] + 3) / 4 * 4);
    }
    in = st.out_off;
    const long long items = (long long)st.p.B * st.p.nty * st.p.ntx;
    long long split = 148LL * resident(st.p) / st.p.ngroups;
    // one-warp CTAs (planes of one tile: nothing waits at a barrier; 256x768x7x7 step 304 -> 248 us): at least four items
    // each, because 5 (K*K + 1) sums per channel end as atomics
    if (split > (items + 3) / 4 && st.p.nthreads == 32) split = (items + 3) / 4;
    if (split > items) split = items;
    st.nsplit = (int)(split < 1 ? 1 : split);
    if ((long long)st.nsplit * st.p.ngroups >= (1LL << 31) || items >= (1LL << 31)) { ch.status = -6; return ch; }
    ch.stages.push_back(st);
  }
  if (deep <= ly.L) {
    CorrStage st;
    PlanarStage& p = st.p;
    p = PlanarStage();
    p.B = ly.B; p.C = ly.C; p.K = ly.K; p.nlev = ly.L - deep + 1;
    p.ctas = ly.K <= 5 ? 2 : 1; p.frames_only = 1;
    p.G = 8;                                             // channels per warp: its eight tile slots shared evenly
    while (p.G > 1 && (sum > 8 / p.G || p.G / 2 >= ly.C)) p.G /= 2;
    for (int j = 0; j <= p.nlev; ++j) { p.h[j] = Hl[deep - 1 + j]; p.w[j] = Wl[deep - 1 + j]; }
    p.TH = round_up(p.h[1], 4); p.TW = round_up(p.w[1], 4);
    p.Hsrc = p.h[0]; p.Wsrc = p.w[0];
    p.xs[0] = (long long)ly.C * p.h[0] * p.w[0]; p.xs[1] = (long long)p.h[0] * p.w[0]; p.xs[2] = p.w[0]; p.xs[3] = 1;
    p.xvec = row_vec(p.xs, 4, 16);
    planar_layout(p);
    p.nthreads = kPlanarMaxThreads;
    while (p.nthreads > 64 && 2LL * p.zero_floats * 4 * (p.nthreads / 32) > kSmemTwoPerSm) p.nthreads -= 32;
    const int nw = p.nthreads / 32, red = nw * 32 * ly.K * ly.K, frames = nw * 2 * p.zero_floats;
    p.smem_bytes = 4 * (frames > red ? frames : red);
    int split = cdiv(148 * resident(p), p.ngroups);      // a CTA per channel group and share of the batch
    if (split > cdiv(ly.B, nw)) split = cdiv(ly.B, nw);
    st.nsplit = imax(split, 1);
    st.deep = 1; st.level = deep; st.in_off = in;
    ch.stages.push_back(st);
  }
  ch.scratch_floats = off;
  return ch;
}

// x, gy: the tensors (dtype 0 fp32, 1 bf16, 2 fp16) or fp32 planes in scratch (dtype 0)
struct CorrArgs;
cudaError_t launch_corr(const CorrStage& st, const CorrArgs& a, int dtype, const void* x, const void* gy, cudaStream_t stream);

}  // namespace wt
