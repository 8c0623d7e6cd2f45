// Parameter gradients of WTConv2d: correlation sums between the sub-band pyramids of the input and of the
// output gradient (see wt2d_wgrad.cuh for the sums and what follows from them), kernel sizes 3, 5, 7.
//
// The kernels of wt2d_wgrad.cuh wrote both pyramids to memory in fp32 (one launch per level and tensor) and
// read every window from there, lanes over channels (stage-1 layer at batch 64: 130 us of pyramids and 187 us of
// sums for 1.1 G multiply-adds, 32 us at the FP32 rate; now 160 + 38 + 30 us, bound by the latency of the fill and by the
// issue slots, half busy).  Here
//
//   * wt2d_corr_kernel takes one level (and the base path with the first): the input's frames are filled as
//     in wt2d_planar.cuh, and a lane again owns one sub-band of a 4 x 4 tile.  The gradient never enters
//     shared memory: the four lanes of a tile load its pixel quadrants and swap them into the four
//     sub-bands by two exchange steps (the transpose of planar_synthesis).  The K*K sums of a lane's
//     sub-band and of the base path stay in registers over all samples and tiles of its CTA, which is fixed
//     to one channel group;
//   * the low-pass planes of both tensors leave as fp32 planes for the next level, a quarter of the elements
//     each time;
//   * wt2d_corr_deep_kernel takes all levels whose tiles together fit the eight tile slots of a warp: a warp
//     owns a (sample, channel) plane, every lane one tile of one sub-band of one level.
#pragma once

#include "wt2d_corr_args.h"
#include "wt2d_planar.cuh"

namespace wt {

#ifdef __CUDA_ARCH__
// acc[dy][dx] += sum over the tile of g[i][q] * window[i + dy][q + dx]
template <int K>
__device__ __forceinline__ void planar_corr(const float* __restrict__ p, int pitch, const float (&g)[4][4], float (&acc)[K * K]) {
  constexpr int NV = (4 + K - 1 + 3) / 4;
#pragma unroll
  for (int iy = 0; iy < 4 + K - 1; ++iy) {
    float row[4 * NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      const float4 t = *reinterpret_cast<const float4*>(p + iy * pitch + 4 * v);
      row[4 * v] = t.x; row[4 * v + 1] = t.y; row[4 * v + 2] = t.z; row[4 * v + 3] = t.w;
    }
#pragma unroll
    for (int dy = 0; dy < K; ++dy) {
      const int i = iy - dy;
      if (i < 0 || i >= 4) continue;
#pragma unroll
      for (int q = 0; q < 4; ++q)                      // neighbouring sums are independent: dx innermost
#pragma unroll
        for (int dx = 0; dx < K; ++dx) acc[dy * K + dx] = fmaf(g[i][q], row[q + dx], acc[dy * K + dx]);
    }
  }
}

// 4 x 4 pixels in their own type, 16-bit ones two to a register; rows at and beyond `nrow` and columns outside
// [0, W) are zero
template <typename T>
struct GradQuad {
  static constexpr int EPW = 4 / (int)sizeof(T);
  unsigned w[16 / EPW];
  __device__ __forceinline__ void load(const T* __restrict__ p, int x, int W, int s2, int s3, bool wide, int nrow) {
#pragma unroll
    for (int i = 0; i < 16 / EPW; ++i) w[i] = 0u;
    if (wide) {
      typedef typename RawChunk<4 * (int)sizeof(T)>::type raw_t;
      union { raw_t raw[4]; unsigned u[16 / EPW]; } v;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        v.raw[i] = raw_t();
        if (i < nrow && x < W) v.raw[i] = __ldg(reinterpret_cast<const raw_t*>(p + i * s2 + x));
      }
#pragma unroll
      for (int i = 0; i < 16 / EPW; ++i) w[i] = v.u[i];
      return;
    }
    const T* q = p + x * s3;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (!(i < nrow && x + k < W)) continue;
        Chunk<T, 4> c;
        c.raw = w[(4 * i + k) / EPW];
        c.set(k % EPW, q[i * s2 + k * s3]);
        w[(4 * i + k) / EPW] = c.raw;
      }
  }
  __device__ __forceinline__ void widen(float (&v)[4][4]) const {
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      Chunk<T, 4> c;
      c.raw = w[i / EPW];
      v[i / 4][i % 4] = Elem<T>::to_f(c.get(i % EPW));
    }
  }
};

// Transpose of planar_synthesis: lane t = 2 ty + tx of a tile holds its 4 x 4 pixel quadrant; afterwards lane s
// holds the un-normalised sub-band s at the tile's 4 x 4 positions.
__device__ __forceinline__ void planar_split(const float (&o)[4][4], float (&v)[4][4], int lane) {
  constexpr unsigned kFull = 0xffffffffu;
  const bool b0 = lane & 1, b1 = lane & 2;
  float m[2][4][2];
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const float e = o[2 * i + a][2 * q] + o[2 * i + a][2 * q + 1], d = o[2 * i + a][2 * q] - o[2 * i + a][2 * q + 1];
        const float keep = b1 ? d : e, r = __shfl_xor_sync(kFull, b1 ? e : d, 2);
        m[a][i][q] = b1 ? r : keep;
        m[a][2 + i][q] = b1 ? keep : r;
      }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const float e = m[0][i][q] + m[1][i][q], d = m[0][i][q] - m[1][i][q];
      const float keep = b0 ? d : e, r = __shfl_xor_sync(kFull, b0 ? e : d, 1);
      v[i][q] = b0 ? r : keep;
      v[i][2 + q] = b0 ? keep : r;
    }
}
#endif

// grid: nsplit CTAs per channel group (group fastest); a CTA walks over the (sample, tile) items of its group
template <typename T, int K, bool BASE>
__global__ void __launch_bounds__(kPlanarMaxThreads, K <= 5 ? 2 : 1)
wt2d_corr_kernel(const __grid_constant__ PlanarStage p, const __grid_constant__ CorrArgs a, const T* __restrict__ x, const T* __restrict__ gy) {
#ifdef __CUDA_ARCH__
  extern __shared__ __align__(128) float planar_smem[];
  float* const sm = planar_smem;
  constexpr int HS = K / 2, KK = K * K;
  const int tid = threadIdx.x, nthr = blockDim.x, lane = tid & 31, warp = tid >> 5, nwarp = nthr >> 5;
  const int s = lane & 3, u = lane >> 2;
  const int cg = (int)(blockIdx.x % (unsigned)p.ngroups), split = (int)(blockIdx.x / (unsigned)p.ngroups);
  const int c0 = cg << p.gshift, gc = imin(p.G, p.C - c0);
  const int gpl = p.gshift, tpw = 8 >> gpl;            // at most eight channels: a lane keeps its channel
  const int g = u & (p.G - 1);
  for (int i = tid; i < p.zero_floats / 4; i += nthr) reinterpret_cast<float4*>(sm)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  __syncthreads();
  float accb[BASE ? KK : 1], accs[KK], sum = 0.f;
#pragma unroll
  for (int k = 0; k < KK; ++k) { accs[k] = 0.f; if (BASE) accb[BASE ? k : 0] = 0.f; }
  const int per = p.nty * p.ntx, items = p.B * per;
  const bool wide = a.gvec >= 4 && p.w[0] % 4 == 0;
  for (int item = split; item < items; item += a.nsplit) {
    const int n = item / per, t2 = item - n * per;
    const int tile_y = t2 / p.ntx, tile_x = t2 - tile_y * p.ntx;
    const int Y0 = tile_y * p.TH, X0 = tile_x * p.TW;
    // tiles of the item that lie on the plane
    const int tyn = imin(p.tyn[1], (p.h[1] - Y0 + 3) >> 2), txn = imin(p.txn[1], (p.w[1] - X0 + 3) >> 2);
    const int ntile = tyn * txn, slots = (ntile + tpw - 1) >> (3 - gpl);
    const float inv = 1.f / (float)txn;
    // K = 7 (one CTA per SM, registers to spare): the gradient pixels of a slot are requested one slot ahead, those
    // of the first before the frames are filled.  (32x96x40x40 step 312 -> 287 us; with two CTAs per SM
    // at K = 5 the registers cost more than the wait, 477 -> 488 us.)
    constexpr bool AHEAD = K == 7;
    GradQuad<T> gq;
    auto request = [&](int slot) {
      const int tq = (slot << (3 - gpl)) + (u >> gpl), t = imin(tq, ntile - 1);
      const int ty = planar_div(t, inv), tx = t - ty * txn;
      const int yy = 2 * Y0 + 8 * ty + 4 * (s >> 1), xx = 2 * X0 + 8 * tx + 4 * (s & 1);
      const T* gp = gy + (long long)n * a.gs[0] + (long long)(c0 + g) * a.gs[1] + (long long)yy * a.gs[2];
      gq.load(gp, xx, p.w[0], (int)a.gs[2], (int)a.gs[3], wide, slot < slots && tq < ntile && g < gc ? p.h[0] - yy : 0);
    };
    if (AHEAD) request(warp);
    {
      PlanarFill<T, K, BASE, 0> f{p, sm, x + (long long)n * p.xs[0] + (long long)c0 * p.xs[1], gc, Y0 - HS, X0 - HS, 0, 0, 0, 0, 0.f};
      if (p.tiled) { f.rb = 4 * p.tyn[1] + 2 * HS; f.cb = 4 * p.txn[1] + 2 * HS; }
      else { f.ra = HS; f.rb = HS + p.h[1]; f.ca = HS; f.cb = HS + p.w[1]; }
      f.inv_nr = p.inv_rows;
      f.run(tid, nthr);
    }
    __syncthreads();
#pragma unroll 1
    for (int slot = warp; slot < slots; slot += nwarp) {
      const int tq = (slot << (3 - gpl)) + (u >> gpl), t = imin(tq, ntile - 1);
      const bool live = tq < ntile && g < gc;
      const int ty = planar_div(t, inv), tx = t - ty * txn;
      const int qy = 8 * ty + 4 * (s >> 1), qx = 8 * tx + 4 * (s & 1);      // this lane's pixel quadrant in the frame
      float q4[4][4];
      if (!AHEAD) request(slot);
      gq.widen(q4);
      if (AHEAD) request(slot + nwarp);
      if constexpr (BASE) {
#pragma unroll
        for (int i = 0; i < 4; ++i) sum += (q4[i][0] + q4[i][1]) + (q4[i][2] + q4[i][3]);
        planar_corr<K>(sm + p.xoff + g * p.xplane + qy * p.xpitch + qx, p.xpitch, q4, accb);
      }
      if (p.nlev == 0) continue;
      float v[4][4];
      planar_split(q4, v, lane);
      planar_corr<K>(sm + p.soff[1] + (4 * g + s) * p.splane[1] + 4 * ty * p.spitch[1] + 4 * tx, p.spitch[1], v, accs);
      if (a.llx && live && s < 2) {                    // lane 0: the gradient's low-pass tile, lane 1: the input's
        if (s) {
          const float* e = sm + p.soff[1] + 4 * g * p.splane[1] + (4 * ty + HS) * p.spitch[1] + 4 * tx + HS;
#pragma unroll
          for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int q = 0; q < 4; ++q) v[i][q] = e[i * p.spitch[1] + q];
        }
        const int hy = Y0 + 4 * ty, hx = X0 + 4 * tx, w1 = p.w[1];
        float* d = (s ? a.llx : a.llg) + (((long long)n * p.C + c0 + g) * p.h[1] + hy) * w1 + hx;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if (hy + i >= p.h[1]) break;
          if ((w1 & 3) == 0) *reinterpret_cast<float4*>(d) = make_float4(v[i][0], v[i][1], v[i][2], v[i][3]);
          else {
#pragma unroll
            for (int q = 0; q < 4; ++q)
              if (hx + q < w1) d[q] = v[i][q];
          }
          d += w1;
        }
      }
    }
    __syncthreads();                                   // the frames are rewritten by the next item
  }

  // ---- sums of the CTA -> stats: the lanes of a warp that share a channel and sub-band meet by shuffles, the
  // warps in shared memory ([warp][set 0..4][K*K + 1][channel]), then one atomic per sum
  float* const red = sm;
  constexpr int SETS = 5, ROW = KK + 1;
  const int each = SETS * ROW * p.G;
#pragma unroll
  for (int k = 0; k <= KK; ++k) {
    float* d = red + warp * each + k * p.G + g;
    if (BASE) {
      float b = k < KK ? accb[BASE ? (k < KK ? k : 0) : 0] : sum;
      b += __shfl_xor_sync(0xffffffffu, b, 1);
      b += __shfl_xor_sync(0xffffffffu, b, 2);
      for (int m = 4 << gpl; m < 32; m <<= 1) b += __shfl_xor_sync(0xffffffffu, b, m);
      if (s == 0 && u < p.G) d[0] = b;
    }
    if (k < KK) {
      float b = accs[k < KK ? k : 0];
      for (int m = 4 << gpl; m < 32; m <<= 1) b += __shfl_xor_sync(0xffffffffu, b, m);
      if (u < p.G) d[(1 + s) * ROW * p.G] = b;
    }
  }
  __syncthreads();
  for (int i = tid; i < SETS * ROW * p.G; i += nthr) {
    const int ch = i & (p.G - 1), k = (i >> gpl) % ROW, set = (i >> gpl) / ROW;
    if (ch >= gc || (set == 0 && !BASE) || (set > 0 && (p.nlev == 0 || k == KK))) continue;
    const int out_set = set == 0 ? 0 : a.set0 + set - 1;
    float v = 0.f;
    for (int w = 0; w < nwarp; ++w) v += red[w * each + i];
    atomicAdd(a.stats + ((size_t)out_set * ROW + k) * p.C + c0 + ch, v);
  }
#endif
}

// A warp takes the planes of p.G channels of a sample, 8 / p.G tile slots each; grid: nsplit CTAs per channel
// group.  xin, gin: (B, C, h[0], w[0]) fp32 planes.
template <int K>
__global__ void __launch_bounds__(kPlanarMaxThreads, K <= 5 ? 2 : 1)
wt2d_corr_deep_kernel(const __grid_constant__ PlanarStage p, const __grid_constant__ CorrArgs a, const float* __restrict__ xin, const float* __restrict__ gin) {
#ifdef __CUDA_ARCH__
  extern __shared__ __align__(128) float planar_smem[];
  constexpr int HS = K / 2, KK = K * K, ROW = KK + 1;
  const int tid = threadIdx.x, nthr = blockDim.x, lane = tid & 31, warp = tid >> 5, nwarp = nthr >> 5;
  const int s = lane & 3, u = lane >> 2, per = 8 >> p.gshift;
  float* const fx = planar_smem + warp * 2 * p.zero_floats;      // frames of the input, then of the gradient
  float* const fg = fx + p.zero_floats;
  const int cg = (int)(blockIdx.x / (unsigned)a.nsplit), split = (int)(blockIdx.x - (unsigned)cg * (unsigned)a.nsplit);
  const int c0 = cg << p.gshift, gc = imin(p.G, p.C - c0);
  for (int i = tid; i < nwarp * 2 * p.zero_floats / 4; i += nthr) reinterpret_cast<float4*>(planar_smem)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  __syncthreads();
  // channel, level and tile of this lane
  const int g = u / per;
  int lev = 1, t = u - g * per;
  while (lev <= p.nlev && t >= p.tyn[lev] * p.txn[lev]) { t -= p.tyn[lev] * p.txn[lev]; ++lev; }
  const bool used = lev <= p.nlev;
  if (!used) { lev = 1; t = 0; }
  const int ty = t / p.txn[lev], tx = t - ty * p.txn[lev], pitch = p.spitch[lev];
  const int win = p.soff[lev] + (4 * g + s) * p.splane[lev] + 4 * ty * pitch + 4 * tx;
  float acc[KK];
#pragma unroll
  for (int k = 0; k < KK; ++k) acc[k] = 0.f;
  for (int n = split * nwarp + warp; n < p.B; n += a.nsplit * nwarp) {
    const long long at = ((long long)n * p.C + c0) * p.h[0] * p.w[0];
    PlanarFill<float, K, false, 0> f{p, fx, xin + at, gc, -HS, -HS, HS, HS + p.h[1], HS, HS + p.w[1], p.inv_rows};
    f.run(lane, 32);
    PlanarFill<float, K, false, 0> f2{p, fg, gin + at, gc, -HS, -HS, HS, HS + p.h[1], HS, HS + p.w[1], p.inv_rows};
    f2.run(lane, 32);
    __syncwarp();
    for (int j = 2; j <= p.nlev; ++j) {
      planar_analysis<K>(p, fx, j, 0, gc, lane, 32);
      planar_analysis<K>(p, fg, j, 0, gc, lane, 32);
      __syncwarp();
    }
    float v[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int q = 0; q < 4; ++q) v[i][q] = fg[win + (HS + i) * pitch + HS + q];
    planar_corr<K>(fx + win, pitch, v, acc);
    __syncwarp();                                      // the frames are rewritten by the next planes
  }
  // warps and tiles of a (channel, level, sub-band) -> stats: [warp][slot][K*K] in shared memory
  __syncthreads();
  float* const red = planar_smem;
#pragma unroll
  for (int k = 0; k < KK; ++k) red[(warp * 32 + lane) * KK + k] = used ? acc[k] : 0.f;
  __syncthreads();
  for (int i = tid; i < gc * p.nlev * 4 * KK; i += nthr) {
    const int k = i % KK, set = (i / KK) % (4 * p.nlev), ch = i / (KK * 4 * p.nlev), l = set / 4 + 1, sb = set & 3;
    int first = ch * per;                              // tile slots of the level
    for (int j = 1; j < l; ++j) first += p.tyn[j] * p.txn[j];
    const int nt = p.tyn[l] * p.txn[l];
    float v = 0.f;
    for (int w = 0; w < nwarp; ++w)
      for (int q = 0; q < nt; ++q) v += red[(w * 32 + 4 * (first + q) + sb) * KK + k];
    atomicAdd(a.stats + ((size_t)(a.set0 + set) * ROW + k) * p.C + c0 + ch, v);
  }
#endif
}

}  // namespace wt
