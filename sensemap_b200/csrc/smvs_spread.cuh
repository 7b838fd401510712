// smvs_spread.cuh — checkerboard kernels for launches with few pixels (internal).
//
// The thread-per-pixel kernels (smvs_sweep.cuh) need some 75,000 pixels to fill
// the GPU; a 160x120 map has 9,600 a launch, 38 blocks on 148 SMs, and its launch
// takes as long as one thread's 14 x N window costs. Here a block is kSpreadWarps
// warps over 32 pixels, one pixel a lane, and the warps share the pixels: each
// scores one of the 10 propagated hypotheses, then half of the views of one of
// the four refinement hypotheses. The cost of one (hypothesis, view) pair stays
// one thread's work with the thread-per-pixel kernels' arithmetic in the same
// order, and every selection is made from the same values in the same order, so
// maps do not depend on the form. The pixels' state is in shared memory; so are
// their windows' bilateral weights, which all pairs of a pixel share.
// All lanes of a warp sample the same view: a texture object that differs within
// a warp is served once per object, and a handle that the compiler cannot prove
// uniform doubles the launch, so views are loop counters, never functions of
// the warp's index.
//
// Measured per sweep launch, thread per pixel -> spread (window radius 5):
//   160x120,  4 views, step 2, u8:  0.149 -> 0.062 ms (local optimisation 0.052 -> 0.027)
//   160x120, 10 views, step 1, f16: 0.711 -> 0.234 ms (0.286 -> 0.097)
//   320x240, 10 views, step 2, f16: 0.391 -> 0.304 ms (0.133 -> 0.113)
// Larger launches stay with the thread-per-pixel form (UseSpread): their time is
// the texture unit's, and the barriers between the phases cost them up to 30 %.
#pragma once

namespace smvs {
namespace detail {
namespace {

// A pixel's window in shared memory, [tap][lane]: the bilateral weight and the
// reference value of every tap, the same for all pairs of the pixel.
template <int R, int S>
struct Window {
  static constexpr int kRows = 2 * R / S + 1;
  static constexpr int kTaps = kRows * kRows;
};

// The bilateral weight of a tap, its exponent rounded as NccCost's expression is
// compiled. Taps that share their spatial product with another (kUnrolled: all
// but the centre tap; else those left and right of the centre column) fuse the
// colour product, the others the spatial one.
template <bool kUnrolled>
__device__ __forceinline__ float TapWeight(int dr, int dc, float cd, float sn, float cn) {
  const float a = (float)(dr * dr) + (float)(dc * dc);
  const float cc = __fmul_rn(cd, cd);
  const bool spatial = dc == 0 && (!kUnrolled || dr == 0);
  const float e = spatial ? __fmaf_rn(-a, sn, -__fmul_rn(cc, cn)) : __fmaf_rn(-cc, cn, -__fmul_rn(a, sn));
  return __expf(e);
}

// Fills the taps w, w + warps, ... of the block's pixels. `win` is the pixel's
// top-left tap in the reference tile (row stride ws).
template <int R, int S, bool kUnrolled>
__device__ __forceinline__ void FillWindow(float2* taps, const float* win, int ws, float center, float sn, float cn,
                                           int w, int warps, int lane) {
  for (int t = w; t < Window<R, S>::kTaps; t += warps) {
    const int i = t / Window<R, S>::kRows, j = t - i * Window<R, S>::kRows;
    const int dr = -R + i * S, dc = -R + j * S;
    const float rc = win[(dr + R) * ws + R + dc];
    const float wgt = TapWeight<kUnrolled>(dr, dc, center - rc, sn, cn);
    taps[t * 32 + lane] = make_float2(wgt, rc);
  }
}

// 1 / (sum of the window's weights), summed in NccCost's order.
template <int R, int S>
__device__ __forceinline__ float WindowInvSum(const float2* taps, int lane) {
  constexpr int kRows = Window<R, S>::kRows;
  float sw[4] = {0.f, 0.f, 0.f, 0.f};
  for (int q = 0; q < kRows; q += 4)
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (q + k < kRows)
#pragma unroll
        for (int j = 0; j < kRows; ++j) sw[k] += taps[((q + k) * kRows + j) * 32 + lane].x;
  return 1.0f / ((sw[0] + sw[1]) + (sw[2] + sw[3]));
}

// NccCost over a filled window: the same source positions, products and sums, the
// moments' last steps rounded as NccCost's are compiled.
template <int R, int S>
__device__ __forceinline__ float WindowCost(cudaTextureObject_t tex, const float* pose, int row, int col, float depth,
                                            const float n[3], const float iK[4], int W, int H, float rsum, float rvar,
                                            float isw, const float2* taps) {
  constexpr float kMaxCost = 2.0f;
  constexpr int kRows = Window<R, S>::kRows;
  float Hm[9];
  ComposeHomography(pose, row, col, depth, n, iK, Hm);
  const float inv_z0 = 1.0f / (Hm[6] * col + Hm[7] * row + Hm[8]);
  const int u = (int)((Hm[0] * col + Hm[1] * row + Hm[2]) * inv_z0);
  const int v = (int)((Hm[3] * col + Hm[4] * row + Hm[5]) * inv_z0);
  // [quirk] bounds are the reference image's width/height (:1265-1270).
  if (u < 0 || u >= W || v < 0 || v >= H) return kMaxCost;
  const int row_start = row - R, col_start = col - R;
  float bcol = Hm[0] * col_start + Hm[1] * row_start + Hm[2];
  float brow = Hm[3] * col_start + Hm[4] * row_start + Hm[5];
  float bz = Hm[6] * col_start + Hm[7] * row_start + Hm[8];
  const float h0 = S * Hm[0], h1 = S * Hm[1], h3 = S * Hm[3], h4 = S * Hm[4], h6 = S * Hm[6], h7 = S * Hm[7];
  float ss[4] = {0.f, 0.f, 0.f, 0.f}, sss[4] = {0.f, 0.f, 0.f, 0.f}, srs[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
  for (int q = 0; q < kRows; q += 4) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (q + k < kRows) {
        const float2* trow = taps + (q + k) * kRows * 32;
        float col_src = bcol, row_src = brow, z = bz;
#pragma unroll
        for (int j = 0; j < kRows; ++j) {
          const float iz = 1.0f / z;
          const float fu = iz * col_src + 0.5f;
          const float fv = iz * row_src + 0.5f;
          const float sc = tex2D<float>(tex, fu, fv);
          const float2 tap = trow[j * 32];
          const float wsc = tap.x * sc;
          ss[k] += wsc;
          sss[k] += wsc * sc;
          srs[k] += wsc * tap.y;
          col_src += h0;
          row_src += h3;
          z += h6;
        }
      }
      bcol += h1; brow += h4; bz += h7;
    }
  }
  float tss = (ss[0] + ss[1]) + (ss[2] + ss[3]);
  float tsss = (sss[0] + sss[1]) + (sss[2] + sss[3]);
  float tsrs = (srs[0] + srs[1]) + (srs[2] + srs[3]);
  tss = __fmul_rn(tss, isw);
  const float svar = __fmaf_rn(tsss, isw, -__fmul_rn(tss, tss));
  if (rvar < 1e-5f || svar < 1e-5f) return kMaxCost;
  const float cov = __fmaf_rn(-rsum, tss, __fmul_rn(tsrs, isw));
  const float val = 1.0f - cov * rsqrtf(rvar * svar);
  return fmaxf(0.0f, fminf(kMaxCost, val));
}

// The pixel of this lane and what its costs need.
struct PixWin {
  int row, col;
  float rsum, rvar, isw;
  const float2* taps;  // + lane
  float vd[3];
};

// ViewCost over a filled window.
template <int R, int S>
__device__ __forceinline__ float PairCost(const JobParams& p, const float* poses, int v, float depth, const float n[3],
                                          const PixWin& px, const float* Kgeom) {
  const float* pose = poses + v * SMVS_POSE_FLOATS;
  float cost = WindowCost<R, S>(p.src_tex[v], pose, px.row, px.col, depth, n, p.refiK, p.W, p.H, px.rsum, px.rvar,
                                px.isw, px.taps);
  if (p.geom)
    cost += p.geom_reg *
            GeomCost(pose, p.dep_tex[v], (float)px.row, (float)px.col, depth, px.vd, Kgeom, p.geom_max);
  return cost;
}


// The block's shared memory after the tile: poses | taps | M | HY | VW | PV | CS.
struct SpreadSmem {
  float* poses;
  float2* taps;  // [taps][32] window
  float* M;      // [kMaxHyp][nb][32] cost of a slot's hypothesis on a view
  float* HY;     // [kMaxHyp][4][32] hypotheses: normal xyz, depth
  float* VW;     // [nb][32] view weights
  float* PV;     // [nb][32] view probabilities (-1: not a good view), then their CDF
  float* CS;     // [kMaxHyp][32] costs
};

template <int R, int S>
__device__ __forceinline__ SpreadSmem CarveSpread(float* tile, int tw, int th, int nb, int hyps) {
  SpreadSmem m;
  m.poses = tile + tw * th;
  m.taps = reinterpret_cast<float2*>(m.poses + nb * SMVS_POSE_FLOATS);  // nb is a multiple of 4
  m.M = reinterpret_cast<float*>(m.taps + Window<R, S>::kTaps * 32);
  m.HY = m.M + hyps * nb * 32;
  m.VW = m.HY + hyps * 4 * 32;
  m.PV = m.VW + nb * 32;
  m.CS = m.PV + nb * 32;
  return m;
}

#define M_(s, v) sm.M[((s) * nb + (v)) * 32 + lane]
#define HY_(s, c) sm.HY[((s) * 4 + (c)) * 32 + lane]
#define VW_(v) sm.VW[(v) * 32 + lane]
#define PV_(v) sm.PV[(v) * 32 + lane]
#define CS_(s) sm.CS[(s) * 32 + lane]

// SweepFromCheckerBoardOpt (kernel_functions.cu:2136-2560) without the prior and
// propagate-depth paths (jobs with a prior run the thread-per-pixel kernels).
template <int R, int S>
__global__ void __launch_bounds__(32 * kSpreadWarps, 2) SweepKernelSpread(const Batch b, int colour) {
  constexpr int L = kSpreadWarps;
  extern __shared__ float smem[];
  __shared__ JobParams sp;
  __shared__ uint64_t mbar;
  __shared__ uint32_t valid[kMaxHyp];  // per slot: the lanes that hold a hypothesis
  __shared__ uint32_t alive;
  int job, blk, iter;
  DecodeBlock(b, b.block_start, blockIdx.x, sp, job, blk, iter);
  const JobParams& p = sp;
  if (iter >= p.num_iterations) return;  // finished job of the batch (block-uniform)
  const float th_mc = p.th_tab[iter];
  const uint64_t skey = StageKey(p.seed, StageSweep(iter, colour));
  const int nb = b.NB, tiles_x = SpreadTilesX(p.W);
  const int tw = RefTileW(kSpreadX, R), th = kSpreadRows + 2 * R;
  float* tile = Align128(smem);  // a TMA destination starts on a 128-byte boundary
  const SpreadSmem sm = CarveSpread<R, S>(tile, tw, th, nb, kMaxHyp);
  const int col0 = (blk % tiles_x) * 2 * kSpreadX, row0 = (blk / tiles_x) * kSpreadRows;
  uint32_t tma_uses = 0;
  if (!StageRefTile<R>(b, job, p, kSpreadX, tile, row0, col0, kSpreadRows, sm.poses, &mbar, tma_uses))
    return;  // block-uniform
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  __syncthreads();
  const int W = p.W, H = p.H, N = p.N;
  const int ly = lane / kSpreadX, row = row0 + ly;
  const int col = col0 + 2 * (lane % kSpreadX) + ((row + colour) & 1);
  const bool inside = col < W && row < H;
  const size_t WH = (size_t)W * H;
  const size_t pix = inside ? (size_t)row * W + col : 0;
  const float* iK = p.refiK;
  PixWin px;
  px.row = row;
  px.col = col;
  px.vd[0] = iK[0] * col + iK[1]; px.vd[1] = iK[2] * row + iK[3]; px.vd[2] = 1.0f;
  px.taps = sm.taps + lane;
  const float* vd = px.vd;
  const float ivl = rsqrtf(vd[0] * vd[0] + vd[1] * vd[1] + vd[2] * vd[2]);
  px.rsum = inside ? p.ref_sum[pix] : 0.f;
  px.rvar = inside ? p.ref_sqsum[pix] - px.rsum * px.rsum : 0.f;
  FillWindow<R, S, false>(sm.taps, tile + ly * tw + (col - col0) + RefTileShift(R), tw,
                          inside ? p.ref[pix] : 0.f, p.sn, p.cn, w, L, lane);

  // Hypothesis slots: 0 the pixel's own, 1 and 2 its best direct neighbours',
  // 3..10 the best of each direction. Each warp fills some.
  auto propose = [&](int s, bool ok, int r, int c) {
    if (ok) {
      const size_t q = (size_t)r * W + c;
      float nn[3] = {p.normal[q], p.normal[WH + q], p.normal[2 * WH + q]};
      CorrectNormal(nn, vd, ivl);
      const float pd = PropagateDepth(p.depth[q], nn, iK, r, c, vd);
      HY_(s, 0) = nn[0]; HY_(s, 1) = nn[1]; HY_(s, 2) = nn[2]; HY_(s, 3) = pd;
    }
    const uint32_t who = __ballot_sync(0xffffffffu, ok);
    if (lane == 0) valid[s] = who;
  };
  for (int task = w; task < 9; task += L) {
    if (task < 8) {  // :2278-2327
      int br = 0, bc = 0;
      float best = FLT_MAX;
      if (inside) {
#pragma unroll
        for (int s = 0; s < 10; ++s) {
          const int nr = row + kDirSamples[task][2 * s], nc = col + kDirSamples[task][2 * s + 1];
          if (nr < 0 || nr >= H || nc < 0 || nc >= W) continue;
          const float nconf = p.conf[(size_t)nr * W + nc];
          if (best > nconf) { br = nr; bc = nc; best = nconf; }
        }
      }
      propose(3 + task, best < FLT_MAX, br, bc);
    } else {  // :2237-2276
      float nconf[4], O[4];
      int nvalid = 0;
      const bool edge = inside && p.grad[pix] >= 1.0f;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        O[i] = (float)i;
        nconf[i] = FLT_MAX;
        const int u = kNeighborOffs[i][1] + col, v = kNeighborOffs[i][0] + row;
        if (!edge || u < 0 || u >= W || v < 0 || v >= H) continue;
        nvalid++;
        nconf[i] = p.conf[(size_t)v * W + u];
      }
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3 - i; ++j)
          if (nconf[j] > nconf[j + 1]) {
            float t = nconf[j]; nconf[j] = nconf[j + 1]; nconf[j + 1] = t;
            t = O[j]; O[j] = O[j + 1]; O[j + 1] = t;
          }
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int idx = (int)O[i];
        propose(1 + i, edge && i < nvalid, kNeighborOffs[idx][0] + row, kNeighborOffs[idx][1] + col);
      }
      if (inside) {
        HY_(0, 0) = p.normal[pix]; HY_(0, 1) = p.normal[WH + pix]; HY_(0, 2) = p.normal[2 * WH + pix];
        HY_(0, 3) = p.depth[pix];
      }
      const uint32_t who = __ballot_sync(0xffffffffu, inside);
      if (lane == 0) valid[0] = who;
    }
  }
  if (inside)
    for (int v = w; v < N; v += L) M_(0, v) = p.cost[(size_t)v * WH + pix];
  __syncthreads();
  px.isw = WindowInvSum<R, S>(sm.taps, lane);

  uint32_t have = 0;  // this pixel's slots
#pragma unroll
  for (int s = 0; s < kMaxHyp; ++s) have |= ((valid[s] >> lane) & 1u) << s;
  const int half = (N + 1) / 2;
  Rng r(skey, (uint32_t)pix);
  float best = FLT_MAX, normal[3] = {0.f, 0.f, 0.f}, depth = 0.f;
  bool live = false;
  // The propagated hypotheses, one a warp.
  {
    const int s = 1 + w;
    const bool mine = (have >> s) & 1u;
    const float hn[3] = {HY_(s, 0), HY_(s, 1), HY_(s, 2)};
    const float hd = HY_(s, 3);
    if (mine)
      for (int v = 0; v < N; ++v) M_(s, v) = PairCost<R, S>(p, sm.poses, v, hd, hn, px, p.refK);
  }
  __syncthreads();

  // ACMM view selection, :2364-2427: a view's probability, -1 where it is not good.
  for (int v = w; v < N; v += L) {
    unsigned n1 = 0, n2 = 0;
    float pv = 0.f;
    for (int s = 0; s < kMaxHyp; ++s) {
      if (!((have >> s) & 1u)) continue;
      const float cst = M_(s, v);
      pv += __expf(-cst * cst * p.inv_beta2);
      n1 += (cst < th_mc);
      n2 += (cst > p.max_mc);
    }
    PV_(v) = ((int)n1 >= p.num_good && (int)n2 <= p.num_bad) ? pv : -1.0f;
  }
  __syncthreads();
  if (w == 0) {
    bool ok = false;
    if (inside) {
      uint32_t flags = 0;
      float sum = 0.f;
      for (int v = 0; v < N; ++v) {
        float pv = PV_(v);
        if (pv != -1.0f) flags |= 1u << v; else pv = 0.f;
        sum += pv;
      }
      if (flags != 0) {
        const float inv = 1.0f / sum;
        float cum = 0.f;
        for (int v = 0; v < N; ++v) {
          const float pv = PV_(v);
          cum += (pv != -1.0f ? pv : 0.f) * inv;
          PV_(v) = cum;
          VW_(v) = 0.f;
        }
        for (int s = 0; s < p.num_samples; ++s) {
          const float rp = r.Uniform() - FLT_EPSILON;
          for (int v = 0; v < N; ++v)
            if (PV_(v) > rp) {
              if (p.random_opt) VW_(v) = 1.0f; else VW_(v) += 1.0f;
              break;
            }
        }
        float wn = 0.f;
        for (int v = 0; v < N; ++v) wn += VW_(v);
        if (!(wn <= 1e-5f)) {
          ok = true;
          const float iwn = 1.0f / wn;
          uint32_t sel = 0;
          for (int v = 0; v < N; ++v) {
            const float x = VW_(v) * iwn;
            VW_(v) = x;
            if (x > 0) sel |= (1u << v);
          }
          p.view_sel[pix] = sel;
        }
      }
    }
    const uint32_t who = __ballot_sync(0xffffffffu, ok);
    if (lane == 0) alive = who;
  }
  __syncthreads();
  live = (alive >> lane) & 1u;
  if (live)
    for (int s = w; s < kMaxHyp; s += L) {
      if (!((have >> s) & 1u)) continue;
      float cs = 0.f;
      for (int v = 0; v < N; ++v) cs += VW_(v) * M_(s, v);
      CS_(s) = cs;
    }
  __syncthreads();
  int mi = -1;
  if (live) {
    for (int s = 0; s < kMaxHyp; ++s)
      if (((have >> s) & 1u) && CS_(s) <= best) { best = CS_(s); mi = s; }  // FindMinCost :648-659 ('<=')
  }
  live = mi >= 0;
  if (live) {
    normal[0] = HY_(mi, 0); normal[1] = HY_(mi, 1); normal[2] = HY_(mi, 2);
    depth = HY_(mi, 3);
    if (mi != 0)
      for (int v = w; v < N; v += L) M_(0, v) = M_(mi, v);
  }
  __syncthreads();  // slots 1..4 are free from here

  // Refinement hypotheses, :2449-2486, one a warp. The draws follow the view
  // samples in a fixed order: depth, normal (2), random depth, random normal.
  if (w < 4 && live) {
    float hn[3] = {normal[0], normal[1], normal[2]};
    float hd = depth;
    if (w == 0) {
      const float a1 = fminf(p.rand_a1, (float)(180.0 * 0.0174532925199432));
      const float a2 = fminf(p.rand_a2, (float)(90.0 * 0.0174532925199432));
      r.draw = p.num_samples + 1;
      PerturbNormalACMH(normal, hn, a1, a2, r);
      CorrectNormal(hn, vd, ivl);
    } else if (w == 1) {
      const float pd_min = (1.0f - p.rand_depth_ratio) * depth, pd_max = (1.0f + p.rand_depth_ratio) * depth;
      r.draw = p.num_samples;
      hd = r.Uniform() * (pd_max - pd_min) + pd_min;  // PerturbDepth :141-147
    } else if (w == 2) {
      r.draw = p.num_samples + 4;
      RandomNormal(r, vd, hn);
      CorrectNormal(hn, vd, ivl);
    } else {
      const float depth_min = p.depth_min;
      const float depth_max = (float)(1.2 * (double)p.depth_max);  // [quirk] :2213
      r.draw = p.num_samples + 3;
      hd = r.Uniform() * (depth_max - depth_min) + depth_min;
    }
    HY_(w + 1, 0) = hn[0]; HY_(w + 1, 1) = hn[1]; HY_(w + 1, 2) = hn[2]; HY_(w + 1, 3) = hd;
  }
  __syncthreads();
  // Half of the views of a refinement hypothesis a warp; once the views scored
  // so far prove it worse than the pixel's best, the others are not sampled
  // (FLT_MAX in their place keeps it from winning).
  if (w < 8 && live) {
    const int s = 1 + (w & 3);
    const float hn[3] = {HY_(s, 0), HY_(s, 1), HY_(s, 2)};
    const float hd = HY_(s, 3);
    float sum = 0.f;
    bool out = false;
    for (int v = 0; v < N; ++v) {
      if ((v < half) != (w < 4)) continue;
      float cost = FLT_MAX;
      if (!out) {
        cost = PairCost<R, S>(p, sm.poses, v, hd, hn, px, p.refK);
        sum += VW_(v) * cost;
        out = WorseThan(sum, best);
      }
      M_(s, v) = cost;
    }
  }
  __syncthreads();
  // :2488-2559: weighted refinement costs, argmin, write back.
  if (w < 4 && live) {
    float cs = 0.f;
    for (int v = 0; v < N; ++v) cs += VW_(v) * M_(w + 1, v);
    CS_(w + 1) = cs;
  }
  __syncthreads();
  if (live) {
    int mj = 0;
    for (int s = 1; s < 5; ++s)
      if (CS_(s) <= best) { best = CS_(s); mj = s; }
    if (w == 0) {
      p.conf[pix] = best;
      p.depth[pix] = mj ? HY_(mj, 3) : depth;
      p.normal[pix] = mj ? HY_(mj, 0) : normal[0];
      p.normal[WH + pix] = mj ? HY_(mj, 1) : normal[1];
      p.normal[2 * WH + pix] = mj ? HY_(mj, 2) : normal[2];
    }
    for (int v = w; v < N; v += L) p.cost[(size_t)v * WH + pix] = M_(mj, v);
  }
}

// LocalOptimization (kernel_functions.cu:2736-2931): two warps per random
// hypothesis, half of the views each.
template <int R, int S>
__global__ void __launch_bounds__(32 * kSpreadWarps, 2) LocalOptKernelSpread(const Batch b, int colour) {
  constexpr int L = kSpreadWarps;
  extern __shared__ float smem[];
  __shared__ JobParams sp;
  __shared__ uint64_t mbar;
  int job, blk, iter;
  DecodeBlock(b, b.block_start, blockIdx.x, sp, job, blk, iter);
  const JobParams& p = sp;
  // Iterations > 2 only (patch_match_cuda.cu:861-880); block-uniform.
  if (iter >= p.num_iterations || !p.local_opt || iter <= 2) return;
  const uint64_t skey = StageKey(p.seed, StageLocal(iter, colour));
  const int nb = b.NB, tiles_x = SpreadTilesX(p.W);
  const int tw = RefTileW(kSpreadX, R), th = kSpreadRows + 2 * R;
  float* tile = Align128(smem);  // a TMA destination starts on a 128-byte boundary
  const SpreadSmem sm = CarveSpread<R, S>(tile, tw, th, nb, 5);
  const int col0 = (blk % tiles_x) * 2 * kSpreadX, row0 = (blk / tiles_x) * kSpreadRows;
  uint32_t tma_uses = 0;
  if (!StageRefTile<R>(b, job, p, kSpreadX, tile, row0, col0, kSpreadRows, sm.poses, &mbar, tma_uses))
    return;  // block-uniform
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int h = w < 5 ? w : w - 5;  // this warp's hypothesis
  __syncthreads();
  const int W = p.W, H = p.H, N = p.N;
  const int ly = lane / kSpreadX, row = row0 + ly;
  const int col = col0 + 2 * (lane % kSpreadX) + ((row + colour) & 1);
  const bool inside = col < W && row < H;
  const size_t WH = (size_t)W * H;
  const size_t pix = inside ? (size_t)row * W + col : 0;
  const float* iK = p.refiK;
  PixWin px;
  px.row = row;
  px.col = col;
  px.vd[0] = iK[0] * col + iK[1]; px.vd[1] = iK[2] * row + iK[3]; px.vd[2] = 1.0f;
  px.taps = sm.taps + lane;
  px.rsum = inside ? p.ref_sum[pix] : 0.f;
  px.rvar = inside ? p.ref_sqsum[pix] - px.rsum * px.rsum : 0.f;
  FillWindow<R, S, (Window<R, S>::kRows <= 8)>(sm.taps, tile + ly * tw + (col - col0) + RefTileShift(R), tw,
                                               inside ? p.ref[pix] : 0.f, p.sn, p.cn, w, L, lane);
  const uint32_t every = N < 32 ? (1u << N) - 1u : 0xffffffffu;
  const uint32_t sel = inside ? p.view_sel[pix] & every : 0u;
  float conf = inside ? p.conf[pix] : 0.f;
  float hcur[4] = {0.f, 0.f, 0.f, 0.f};
  if (inside) {
    const float a1 = (float)(4.0 * 0.0174532925199432), a2 = (float)(2.0 * 0.0174532925199432);
    float m[3] = {p.normal[pix], p.normal[WH + pix], p.normal[2 * WH + pix]};
    float lo = p.depth[pix], hi = lo;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int u = kNeighborOffs[i][1] + col, v = kNeighborOffs[i][0] + row;
      if (u < 0 || u >= W || v < 0 || v >= H) continue;
      const size_t q = (size_t)v * W + u;
      const float nd = p.depth[q];
      m[0] += p.normal[q]; m[1] += p.normal[WH + q]; m[2] += p.normal[2 * WH + q];
      if (nd <= lo) lo = nd;
      if (nd > hi) hi = nd;
    }
    const float inv_norm = rsqrtf(m[0] * m[0] + m[1] * m[1] + m[2] * m[2]);
    m[0] *= inv_norm; m[1] *= inv_norm; m[2] *= inv_norm;
    Rng r(skey, (uint32_t)pix);
    r.draw = 3 * h;  // three draws a hypothesis
    hcur[3] = r.Uniform() * (hi - lo) + lo;
    PerturbNormalACMH(m, hcur, a1, a2, r);
    if (w < 5) { HY_(h, 0) = hcur[0]; HY_(h, 1) = hcur[1]; HY_(h, 2) = hcur[2]; HY_(h, 3) = hcur[3]; }
  }
  __syncthreads();
  px.isw = WindowInvSum<R, S>(sm.taps, lane);
  // Its selected views; once the views scored so far prove the mean above the
  // pixel's cost, the others are not sampled (FLT_MAX in their place).
  const float mw = (float)__popc(sel);
  const int half = (N + 1) / 2;
  {
    float sum = 0.f;
    bool out = false;
    for (int v = 0; v < N; ++v) {
      if ((v < half) != (w < 5) || !((sel >> v) & 1u)) continue;
      float cost = FLT_MAX;
      if (!out) {
        cost = PairCost<R, S>(p, sm.poses, v, hcur[3], hcur, px, p.refK);
        sum += cost;
        out = WorseThan(sum, conf * mw);
      }
      M_(h, v) = cost;
    }
  }
  __syncthreads();
  if (w < 5 && sel != 0u) {
    float mconf = 0.f;
    for (int v = 0; v < N; ++v)
      if ((sel >> v) & 1u) mconf += M_(h, v);
    CS_(h) = mconf / mw;
  }
  __syncthreads();
  int mi = -1;
  if (sel != 0u)
#pragma unroll
    for (int k = 0; k < 5; ++k)
      if (CS_(k) < conf) { conf = CS_(k); mi = k; }
  if (mi < 0) return;
  // The winner is scored again on the unselected views, a share per warp.
  // [quirk] :2916-2919 passes the inverse intrinsics where K is expected.
  hcur[0] = HY_(mi, 0); hcur[1] = HY_(mi, 1); hcur[2] = HY_(mi, 2); hcur[3] = HY_(mi, 3);
  if (w == 0) {
    p.conf[pix] = conf;
    p.depth[pix] = hcur[3];
    p.normal[pix] = hcur[0]; p.normal[WH + pix] = hcur[1]; p.normal[2 * WH + pix] = hcur[2];
  }
  for (int v = 0; v < N; ++v) {
    if (v % L != w) continue;
    p.cost[(size_t)v * WH + pix] = ((sel >> v) & 1u)
                                       ? M_(mi, v)
                                       : PairCost<R, S>(p, sm.poses, v, hcur[3], hcur, px, p.refiK);
  }
}

#undef M_
#undef HY_
#undef VW_
#undef PV_
#undef CS_

template <int R, int S>
cudaError_t LaunchSpread(const Batch& b, int colour, bool local, cudaStream_t stream) {
  if (b.total_blocks <= 0) return cudaSuccess;
  const size_t smem = SpreadSmemBytes(R, S, b.NB);
  if (local)
    LocalOptKernelSpread<R, S><<<b.total_blocks, 32 * kSpreadWarps, smem, stream>>>(b, colour);
  else
    SweepKernelSpread<R, S><<<b.total_blocks, 32 * kSpreadWarps, smem, stream>>>(b, colour);
  return cudaGetLastError();
}

}  // namespace
}  // namespace detail
}  // namespace smvs
