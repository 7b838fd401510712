// smvs_fusion.cu — fusion of depth maps into a point cloud (StereoFusion).
//
// StereoFusion's image loop (SenseMap src/mvs/fusion.cc:1160-1215), FuseImage
// (:1730-1792) and Fuse (:1794-2182) on the GPU, with the results of the
// reference run seed after seed (its fusion threads' row slices taken one
// after another). Compiled with -fmad=false -prec-div=true -prec-sqrt=true
// -ftz=false: the same IEEE single-precision operations, in the same order, as
// the reference's Eigen expressions (see the float helpers below).
//
// Each image is fused in five steps, all in stream order:
//   1. closure: every seed pixel (one warp each, its state in shared memory)
//      collects the pixels its traversal could ever accept — those that pass
//      its reprojection, depth and normal tests, are not fused yet and are
//      reachable from it through such pixels — with the push lists between
//      them in the reference's push order (the seed's record); records over
//      the shared capacity take a thread-per-seed overflow pass;
//   2. claims: for every pixel the seeds whose records hold it; each seed's
//      predecessors are the earlier claimants of its pixels;
//   3. order: a ticket order in which every predecessor comes first (the seed
//      grid sheared so that key = column + K x row grows along every
//      predecessor pair);
//   4. replay: warps take tickets, wait until their predecessors are settled
//      (have run, or had their pixel fused and never will), read the masks of
//      their record's pixels and find the pixels the reference's traversal
//      fuses — in parallel (a frontier search) where no limit can bind, else
//      by replaying its depth-first traversal (explicit stack, limits) — and
//      mark them, their own last; then they compute the fused point (medians);
//   5. compaction of the points in seed order.
// A traversal only reads or writes the masks of pixels that pass its tests
// (a pixel that fails them is skipped whether or not it is fused), so two
// seeds whose records share no pixel commute, and waiting for every earlier
// claimant of each pixel reproduces the sequential order exactly.
#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <vector>

#include <cuda_runtime.h>

#include "../../include/smvs.h"
#include "../../include/smvs_testing.h"

extern "C" void smvs_internal_set_error(const char* msg);
cudaMemPool_t smvs_internal_device_pool(int device);
cudaError_t smvs_internal_alloc(void** p, size_t bytes, cudaMemPool_t pool, cudaStream_t stream);

namespace {

constexpr int kBlank = 3;              // blank_size (fusion.cc:1757, :1831)
constexpr int kCap = 256;              // record capacity of the closure pass (pixels)
constexpr int kBigCap = 65535;         // record capacity of the overflow pass (u16 indices)
constexpr int kBigBatch = 256;         // overflow seeds per launch
// Scratch bytes of one overflow thread: gid (u32) | derr (f32) | vid (u16) |
// hash slots (u16, from the next 16-byte boundary) | eoff (u32); a multiple of
// 16 so every thread's arrays stay aligned.
constexpr size_t kBigSlotsOff = ((size_t)kBigCap * 10u + 15u) & ~(size_t)15u;
constexpr size_t kBigEoffOff = kBigSlotsOff + 2u * 2u * 65536u;  // eoff (u32, kBigCap + 1)
constexpr size_t kBigStride = (kBigEoffOff + 4u * ((size_t)kBigCap + 1u) + 15u) & ~(size_t)15u;
constexpr uint32_t kEmpty = 0xffffffffu;
constexpr uint32_t kOver = 0xfffffffeu;
constexpr uint32_t kRetry = 0xfffffffdu;  // the record did not fit the pool; built again after it grows
constexpr int kReplayWarps = 4;        // warps per replay block
constexpr int kStackSh = 512;          // replay stack entries kept in shared memory per warp
constexpr int kScanItems = 4096;       // items per scan block (256 threads x 16)
constexpr unsigned long long kWaitLimitNs = 20ull * 1000 * 1000 * 1000;  // bounded waits: 20 s
// Test hooks (smvs_test_fusion_waits): a shorter wait bound and a seed whose
// successors are never released, for this thread's next runs.
thread_local unsigned long long t_wait_limit_ns = 0;  // 0: kWaitLimitNs
thread_local long long t_withhold = -1;
// Test hook (smvs_test_fusion_paths) for fusions created on this thread: no
// projection table; no predecessor lists.
thread_local bool t_in_place = false, t_walk = false;

// Status bits written by the kernels.
constexpr uint32_t kStTimeout = 1u, kStPool = 2u, kStBad = 4u, kStBig = 8u;

int Fail(int code, const char* fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof(buf), fmt, ap);
  va_end(ap);
  smvs_internal_set_error(buf);
  return code;
}

#define FU_CUDA(call)                                                                                      \
  do {                                                                                                     \
    cudaError_t e_ = (call);                                                                               \
    if (e_ != cudaSuccess) return Fail(SMVS_ECUDA, "%s: %s (%s:%d)", #call, cudaGetErrorString(e_), __FILE__, __LINE__); \
  } while (0)

// One image as the kernels see it.
struct FView {
  float P[12];   // K [R | T], ComposeProjectionMatrix (src/mvs/utils.cc:35-42)
  float iP[12];  // top rows of [P; 0 0 0 1]^-1 (double inverse rounded once)
  int W, H;
  uint32_t base;  // first pixel of the image in the concatenated arrays
  int ov_begin, ov_end;
  int pad;
};

// Per-pixel arrays of all images, concatenated.
struct FMaps {
  const FView* views;
  const int* ov;          // overlapping_images_, concatenated
  const uint8_t* trav;    // per image: used and not yet fused
  // Two float4 per pixel, one 32-byte sector: a candidate's test reads both.
  //   [2 g]     inv_P * (col d, row d, d, 1) (fusion.cc:1953-1955), depth d
  //   [2 g + 1] inv_R * normal (:1939-1941), red-channel gradient (:2007-2021)
  const float4* pix;
  const uint32_t* proj;   // [pixel][deg]: the pixel's place in its overlapping images (pixel index, kNoKey: outside)
  int deg;                // overlapping images of the image that has most
  int num_views;
  const uint8_t* rgb;     // W*H*3 per image
  uint8_t* mask;          // fused_pixel_masks_
};
constexpr uint32_t kNoKey = 0xffffffffu;

struct FConsts {
  float max_sq_reproj;  // max_squared_reproj_error_ (float)
  float min_cos;        // min_cos_normal_error_ (float)
  float derr_thr;       // largest float <= max_depth_error: x > derr_thr <=> (double)x > max_depth_error
  double max_depth_error;
  int with_normal, min_pix, max_pix, max_depth, min_vis;
};

struct FImage {
  int view;
  int cap;  // closure capacity of the fast pass (<= kCap)
  int Rs, Cs, step;
  uint32_t nseeds;
  const int* rows;  // Rs image rows of the seed grid
};

// Record pool of one image. A record (u32 words): cnt, nE, gid[cnt], derr[cnt],
// eoff[cnt + 1], vid[cnt] (u16), edges[nE bound] (u8 in records of at most kCap
// pixels, else u16).
struct FRecs {
  uint32_t* pool;
  unsigned long long pool_words;
  unsigned long long* used;   // bump cursor (words)
  uint32_t* rec_off;          // per seed: word offset, or kEmpty, kOver, kRetry (no record)
  uint32_t* over_list;        // seeds over kCap
  uint32_t* n_over;
  uint32_t* stats;            // [0] max cnt, [1] max nE, [2] status
};

__host__ __device__ inline uint32_t RecWords(uint32_t cnt, uint32_t ebound) {
  return 2u + 2u * cnt + (cnt + 1u) + (cnt + 1u) / 2u + (cnt <= (uint32_t)kCap ? (ebound + 3u) / 4u : (ebound + 1u) / 2u);
}

// Bytes of one replay warp's scratch region: stack (u32) | vals (f32) | ids (u32)
// | acc (u16) | flags (u8), rounded to 16.
__host__ __device__ inline size_t ScratchPer(uint32_t cnt, uint32_t stack) {
  return ((size_t)stack * 4u + (size_t)cnt * 11u + 31u) & ~(size_t)15u;
}

// ---- float helpers: the reference's Eigen evaluation order ----------------
// A 3x4 row-major matrix times a Vector4f: one SSE packet product reduced as
// (p0 + p2) + (p1 + p3) (Eigen's predux).
__device__ __forceinline__ float Dot4p(const float* a, float x, float y, float z, float w) {
  return __fadd_rn(__fadd_rn(__fmul_rn(a[0], x), __fmul_rn(a[2], z)), __fadd_rn(__fmul_rn(a[1], y), __fmul_rn(a[3], w)));
}
// P * xyz.homogeneous(): the 3x3 block product plus the last column.
__device__ __forceinline__ float Dot3h(const float* a, float x, float y, float z) {
  return __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(a[0], x), __fmul_rn(a[1], y)), __fmul_rn(a[2], z)), a[3]);
}
// Vector3f dot product / 3x3 times Vector3f row.
__device__ __forceinline__ float Dot3(float a0, float a1, float a2, float x, float y, float z) {
  return __fadd_rn(__fadd_rn(__fmul_rn(a0, x), __fmul_rn(a1, y)), __fmul_rn(a2, z));
}
__device__ __forceinline__ bool ValidDepth(float d) { return d > 0.0f && isfinite(d); }
// Total order of floats (sign first): the order the medians use.
__device__ __forceinline__ uint32_t FKey(float f) {
  const uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

// Rounded projection of a point into image u (fusion.cc:2080-2091); false if
// it falls outside the blank border.
__device__ __forceinline__ bool ProjectPixel(const FView& fu, float x, float y, float z, int* row, int* col) {
  const float q0 = Dot3h(fu.P, x, y, z), q1 = Dot3h(fu.P + 4, x, y, z), q2 = Dot3h(fu.P + 8, x, y, z);
  const float uc = roundf(__fdiv_rn(q0, q2)), ur = roundf(__fdiv_rn(q1, q2));
  if (!(uc >= (float)kBlank && ur >= (float)kBlank && uc < (float)(fu.W - kBlank) && ur < (float)(fu.H - kBlank)))
    return false;
  *col = (int)uc;
  *row = (int)ur;
  return true;
}

// ---- point maps -------------------------------------------------------------
__global__ void PointMapKernel(FView v, float R0, float R1, float R2, float R3, float R4, float R5, float R6,
                               float R7, float R8, const float* __restrict__ depth_in,
                               const float* __restrict__ normal_in, int with_normal, int has_color,
                               float4* __restrict__ pix, const uint8_t* __restrict__ rgb) {
  const uint32_t plane = (uint32_t)v.W * (uint32_t)v.H;
  for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < plane; p += gridDim.x * blockDim.x) {
    const int row = (int)(p / (uint32_t)v.W), col = (int)(p - (uint32_t)row * (uint32_t)v.W);
    const size_t g = (size_t)v.base + p;
    const float d = depth_in[p];
    const float cd = __fmul_rn((float)col, d), rd = __fmul_rn((float)row, d);
    pix[2 * g] = make_float4(Dot4p(v.iP, cd, rd, d, 1.0f), Dot4p(v.iP + 4, cd, rd, d, 1.0f),
                             Dot4p(v.iP + 8, cd, rd, d, 1.0f), d);
    float4 n = make_float4(0.f, 0.f, 0.f, 0.f);
    if (with_normal) {
      const float n0 = normal_in[p], n1 = normal_in[plane + p], n2 = normal_in[2 * (size_t)plane + p];
      // inv_R = R^T: row i of inv_R is column i of R.
      n.x = Dot3(R0, R3, R6, n0, n1, n2);
      n.y = Dot3(R1, R4, R7, n0, n1, n2);
      n.z = Dot3(R2, R5, R8, n0, n1, n2);
    }
    if (has_color && col > 1 && col < v.W - 1 && row > 1 && row < v.H - 1) {
      const uint8_t* px = rgb + 3ull * g;
      const float gx = __fdiv_rn((float)((int)px[-3] - (int)px[3]), 255.0f);
      const float gy = __fdiv_rn((float)((int)px[-3 * v.W] - (int)px[3 * v.W]), 255.0f);
      n.w = __fsqrt_rn(__fadd_rn(__fmul_rn(gx, gx), __fmul_rn(gy, gy)));
    }
    pix[2 * g + 1] = n;
  }
}

// Row and column of pixel px of an image W wide. The product is at most one row off
// below some four million rows and a few hundred at 2^31 pixels of one column.
__host__ __device__ __forceinline__ void RowAndColumn(uint32_t px, int W, int* row, int* col) {
#ifdef __CUDA_ARCH__
  int r = (int)__fmul_rn((float)px, __frcp_rn((float)W));
#else
  int r = (int)((float)px * (1.0f / (float)W));
#endif
  int c = (int)(px - (uint32_t)r * (uint32_t)W);
  while (c < 0) { c += W; --r; }
  while (c >= W) { c -= W; ++r; }
  *row = r;
  *col = c;
}

// Where the pixels of image `view` fall in its overlapping images. A closure
// asks for these places again in every seed that reaches the pixel (some 100
// seeds in the first image of 11 views): the table replaces two divisions, nine
// products and the point's read by one word, of ten that lie together.
__global__ void ProjectTableKernel(FMaps m, int view, uint32_t* __restrict__ proj) {
  const FView& v = m.views[view];
  const uint32_t plane = (uint32_t)v.W * (uint32_t)v.H;
  const int deg = v.ov_end - v.ov_begin;
  for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < plane; p += gridDim.x * blockDim.x) {
    const size_t g = (size_t)v.base + p;
    const float4 x = m.pix[2 * g];
    const bool ok = ValidDepth(x.w);
    for (int k = 0; k < m.deg; ++k) {
      uint32_t e = kNoKey;
      int row, col;
      if (ok && k < deg) {
        const int u = m.ov[v.ov_begin + k];
        const FView& fu = m.views[u];
        if (m.trav[u] && ProjectPixel(fu, x.x, x.y, x.z, &row, &col))
          e = fu.base + (uint32_t)row * (uint32_t)fu.W + (uint32_t)col;
      }
      proj[g * (size_t)m.deg + k] = e;
    }
  }
}

// ---- closure ---------------------------------------------------------------
// Membership of a closure under construction: open addressing over the pixel
// index, slots hold node index + 1 (0 = empty).
struct NodeSet {
  uint16_t* slot;
  uint32_t mask;  // table size - 1 (a power of two, at least twice the capacity)
  __device__ __forceinline__ uint32_t Home(uint32_t g) const { return (g * 0x9E3779B1u) >> 7 & mask; }
  __device__ __forceinline__ void Clear() const {
    for (uint32_t i = 0; i <= mask; ++i) slot[i] = 0;
  }
  __device__ __forceinline__ int Find(const uint32_t* gid, uint32_t g) const {
    for (uint32_t h = Home(g);; h = (h + 1) & mask) {
      const uint32_t e = slot[h];
      if (e == 0) return -1;
      if (gid[e - 1] == g) return (int)e - 1;
    }
  }
  __device__ __forceinline__ void Insert(uint32_t g, int idx) const {
    uint32_t h = Home(g);
    while (slot[h] != 0) h = (h + 1) & mask;
    slot[h] = (uint16_t)(idx + 1);
  }
};

// The seed point's projection into image u (column, row, depth), computed once
// per image: a small direct-mapped cache keyed by the image index.
struct SeedProj {
  int u[16];
  float col[16], row[16], z[16];
  __device__ __forceinline__ void Clear() {
    for (int i = 0; i < 16; ++i) u[i] = -1;
  }
  __device__ __forceinline__ void Get(const FView& fu, int ui, float sx, float sy, float sz, float* pc, float* pr,
                                      float* pz) {
    const int h = ui & 15;
    if (u[h] != ui) {
      const float p0 = Dot4p(fu.P, sx, sy, sz, 1.0f), p1 = Dot4p(fu.P + 4, sx, sy, sz, 1.0f),
                  p2 = Dot4p(fu.P + 8, sx, sy, sz, 1.0f);
      u[h] = ui;
      col[h] = __fdiv_rn(p0, p2);
      row[h] = __fdiv_rn(p1, p2);
      z[h] = p2;
    }
    *pc = col[h];
    *pr = row[h];
    *pz = z[h];
  }
};

// The pixels the seed's traversal can accept (see the file comment) into
// gid/vid/derr, and the push lists between them (eoff/edges, in the reference's
// push order: overlapping_images_ of the pixel's image, :2073-2092) while they
// fit `ecap` (*ne > ecap otherwise). Returns the pixel count, 0 when the seed
// itself is fused or has no valid depth, -1 when there are more than `cap`.
__device__ __forceinline__ int BuildClosure(const FMaps& m, const FConsts& c, uint32_t sg, int sv, uint32_t* gid,
                                            uint16_t* vid, float* derr, const NodeSet& set, int cap,
                                            uint32_t* eoff, uint16_t* edges, uint32_t ecap, uint32_t* ne) {
  *ne = 0;
  if (m.mask[sg]) return 0;
  const float4 sp = m.pix[2 * (size_t)sg], sn = m.pix[2 * (size_t)sg + 1];
  if (!ValidDepth(sp.w)) return 0;
  const float sx = sp.x, sy = sp.y, sz = sp.z, s0 = sn.x, s1 = sn.y, s2 = sn.z;
  SeedProj proj;
  proj.Clear();
  set.Clear();
  gid[0] = sg;
  vid[0] = (uint16_t)sv;
  derr[0] = 0.0f;
  set.Insert(sg, 0);
  int cnt = 1;
  uint32_t e = 0;
  for (int i = 0; i < cnt; ++i) {
    eoff[i] = e;
    const uint32_t g = gid[i];
    const FView& fv = m.views[vid[i]];
    const float4 gp = m.pix[2 * (size_t)g];
    for (int k = fv.ov_begin; k < fv.ov_end; ++k) {
      const int u = m.ov[k];
      if (!m.trav[u]) continue;
      const FView& fu = m.views[u];
      int row, col;
      if (!ProjectPixel(fu, gp.x, gp.y, gp.z, &row, &col)) continue;
      const uint32_t q = fu.base + (uint32_t)row * (uint32_t)fu.W + (uint32_t)col;
      if (m.mask[q]) continue;
      int j = set.Find(gid, q);
      if (j < 0) {
        const float dq = m.pix[2 * (size_t)q].w;
        if (!ValidDepth(dq)) continue;
        // Reprojection and depth error of the seed point in image u (:1893-1912).
        float pc, pr, pz;
        proj.Get(fu, u, sx, sy, sz, &pc, &pr, &pz);
        const float cdiff = __fsub_rn(pc, (float)col), rdiff = __fsub_rn(pr, (float)row);
        const float sq = __fadd_rn(__fmul_rn(cdiff, cdiff), __fmul_rn(rdiff, rdiff));
        if (sq > c.max_sq_reproj) continue;
        const float de = __fdiv_rn(fabsf(__fsub_rn(pz, dq)), dq);
        if (de > c.derr_thr) continue;
        const float4 nq = m.pix[2 * (size_t)q + 1];
        if (c.with_normal && Dot3(s0, s1, s2, nq.x, nq.y, nq.z) < c.min_cos) continue;  // :1944-1948
        if (cnt == cap) return -1;
        j = cnt;
        gid[cnt] = q;
        vid[cnt] = (uint16_t)u;
        derr[cnt] = de;
        set.Insert(q, cnt);
        ++cnt;
      }
      if (e < ecap) edges[e] = (uint16_t)j;
      ++e;
    }
  }
  eoff[cnt] = e;
  *ne = e;
  return cnt;
}

// Writes the record of a closure; false when the pool is full. The push lists
// are copied from BuildClosure's, or computed again when they did not fit.
__device__ bool WriteRecord(const FMaps& m, const FRecs& r, uint32_t seed, const uint32_t* gid, const uint16_t* vid,
                            const float* derr, const NodeSet& set, int cnt, const uint32_t* leoff,
                            const uint16_t* ledges, uint32_t lne, bool have_edges) {
  uint32_t ebound = lne;
  if (!have_edges) {
    ebound = 0;
    for (int i = 0; i < cnt; ++i) {
      const FView& fv = m.views[vid[i]];
      ebound += (uint32_t)(fv.ov_end - fv.ov_begin);
    }
  }
  const uint32_t words = RecWords((uint32_t)cnt, ebound);
  const unsigned long long off = atomicAdd(r.used, (unsigned long long)words);
  if (off + words > r.pool_words || off + words > 0xfffffff0ull) {
    atomicOr(&r.stats[2], kStPool);
    r.rec_off[seed] = kRetry;
    return false;
  }
  uint32_t* rec = r.pool + off;
  uint32_t* rg = rec + 2;
  float* rd = reinterpret_cast<float*>(rg + cnt);
  uint32_t* eoff = reinterpret_cast<uint32_t*>(rd + cnt);
  uint16_t* rv = reinterpret_cast<uint16_t*>(eoff + cnt + 1);
  uint16_t* edges = rv + 2 * ((cnt + 1) / 2);
  uint8_t* edges8 = cnt <= kCap ? reinterpret_cast<uint8_t*>(edges) : nullptr;
  for (int i = 0; i < cnt; ++i) {
    rg[i] = gid[i];
    rd[i] = derr[i];
    rv[i] = vid[i];
  }
  uint32_t e = 0;
  if (have_edges) {
    for (int i = 0; i <= cnt; ++i) eoff[i] = leoff[i];
    for (uint32_t q = 0; q < lne; ++q)
      if (edges8) edges8[q] = (uint8_t)ledges[q]; else edges[q] = ledges[q];
    e = lne;
  } else {
    for (int i = 0; i < cnt; ++i) {
      eoff[i] = e;
      const uint32_t g = gid[i];
      const FView& fv = m.views[vid[i]];
      const float4 gp = m.pix[2 * (size_t)g];
      for (int k = fv.ov_begin; k < fv.ov_end; ++k) {
        const int u = m.ov[k];
        if (!m.trav[u]) continue;
        const FView& fu = m.views[u];
        int row, col;
        if (!ProjectPixel(fu, gp.x, gp.y, gp.z, &row, &col)) continue;
        const int j = set.Find(gid, fu.base + (uint32_t)row * (uint32_t)fu.W + (uint32_t)col);
        if (j < 0) continue;
        if (e < ebound) {
          if (edges8) edges8[e] = (uint8_t)j; else edges[e] = (uint16_t)j;
        }
        ++e;
      }
    }
    eoff[cnt] = e;
    if (e > ebound) atomicOr(&r.stats[2], kStBad);
  }
  rec[0] = (uint32_t)cnt;
  rec[1] = e;
  r.rec_off[seed] = (uint32_t)off;
  atomicMax(&r.stats[0], (uint32_t)cnt);
  atomicMax(&r.stats[1], e);
  return true;
}

__device__ __forceinline__ uint32_t SeedPixel(const FMaps& m, const FImage& im, uint32_t s) {
  const uint32_t i = s / (uint32_t)im.Cs, j = s - i * (uint32_t)im.Cs;
  const FView& fv = m.views[im.view];
  const uint32_t row = (uint32_t)im.rows[i], col = (uint32_t)(kBlank + (int)j * im.step);
  return fv.base + row * (uint32_t)fv.W + col;
}

constexpr int kSetSlots = 2 * kCap;          // hash slots of the closure pass
constexpr int kBigSetSlots = 2 * 65536;      // hash slots of the overflow pass
constexpr int kEdgeLocal = 2048;             // push-list entries kept by the closure pass
// Rejected pixels kept in a closure's hash set: with the round that reaches a
// bound (32 lanes each) and kCap accepted ones the set is never full.
constexpr int kMaxRejected = kSetSlots - kCap - 96;
constexpr uint16_t kReject = 0xffff;

// One warp per seed. The closure under construction lives in shared memory:
// a hash set of its pixels (key = pixel index, value = node index), the
// nodes (pixel, image, depth error, point) and their push lists.
constexpr int kClosureWarps = 4;  // warps (seeds in flight) per closure block
struct ClosureShared {
  uint32_t keys[kSetSlots];
  uint32_t gid[kCap];
  float seed[3][32];                   // the seed's column, row and depth in images 0..31
  uint16_t kidx[kSetSlots];
  uint16_t vid[kCap];
};

// A closure warp's global staging (L2-resident for the whole grid): the push
// lists, their offsets and the depth errors, each written once and read when
// the record is written.
constexpr size_t kStageEoff = (size_t)kEdgeLocal;                       // u32[kCap + 1]
constexpr size_t kStageDerr = kStageEoff + 4u * ((size_t)kCap + 1u);   // f32[kCap]
constexpr size_t kStageBytes = (kStageDerr + 4u * (size_t)kCap + 15u) & ~(size_t)15u;

constexpr size_t kClosureSmem = sizeof(ClosureShared) * kClosureWarps;

// `stage`: kStageBytes per warp of the grid (global memory; tens of MB for the
// whole grid, so they stay in L2). kTable: the projections come from m.proj.
// The kernel is bound by the latency of its gathers (a frontier pixel's places, a
// candidate's sector and mask), so these are few and independent, the next
// round's places are read ahead, and the seed's own projections, which every
// candidate's test needs, are computed once per image. Measured on the first
// image of 11 views 1600x1200: 26.1 ms (60.9 with eight separate maps, every
// projection in place and each candidate read whatever its distance). Now its
// instructions bound it: 67 % of the issue slots, 17 of 32 lanes.
template <bool kTable>
__global__ void __launch_bounds__(32 * kClosureWarps) ClosureKernel(FMaps m, FConsts c, FImage im, FRecs r,
                                                                    int only_retry, uint8_t* stage) {
  extern __shared__ __align__(16) unsigned char closure_smem[];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  ClosureShared& sh = reinterpret_cast<ClosureShared*>(closure_smem)[w];
  uint8_t* const wstage = stage + ((size_t)blockIdx.x * kClosureWarps + w) * kStageBytes;
  uint8_t* const edges = wstage;
  uint32_t* const eoff = reinterpret_cast<uint32_t*>(wstage + kStageEoff);
  float* const derr = reinterpret_cast<float*>(wstage + kStageDerr);
  const unsigned lt = (1u << lane) - 1u;
  const int D = m.deg > 0 ? m.deg : 1;
  const int q32 = 32 / D, r32 = 32 - q32 * D;
  for (uint32_t s = blockIdx.x * kClosureWarps + w; s < im.nseeds; s += gridDim.x * kClosureWarps) {
    if (only_retry && r.rec_off[s] != kRetry) continue;
    const uint32_t sg = SeedPixel(m, im, s);
    const float4 sp = m.pix[2 * (size_t)sg];
    if (m.mask[sg] || !ValidDepth(sp.w)) {
      if (lane == 0) r.rec_off[s] = kEmpty;
      continue;
    }
    const float4 sn = m.pix[2 * (size_t)sg + 1];
    for (int h = lane; h < kSetSlots; h += 32) sh.keys[h] = kNoKey;
    if (lane < m.num_views && m.trav[lane]) {
      const FView& fu = m.views[lane];
      const float p0 = Dot4p(fu.P, sp.x, sp.y, sp.z, 1.0f), p1 = Dot4p(fu.P + 4, sp.x, sp.y, sp.z, 1.0f),
                  p2 = Dot4p(fu.P + 8, sp.x, sp.y, sp.z, 1.0f);
      sh.seed[0][lane] = __fdiv_rn(p0, p2);
      sh.seed[1][lane] = __fdiv_rn(p1, p2);
      sh.seed[2][lane] = p2;
    }
    __syncwarp();
    if (lane == 0) {
      const uint32_t h = ((sg * 0x9E3779B1u) >> 7) & (uint32_t)(kSetSlots - 1);
      sh.keys[h] = sg;
      sh.kidx[h] = 0;
      sh.gid[0] = sg;
      sh.vid[0] = (uint16_t)im.view;
      derr[0] = 0.0f;
      eoff[0] = 0;
    }
    __syncwarp();
    int cnt = 1, head = 0, rejected = 0;
    uint32_t ecur = 0;
    bool over = false;
    // Breadth-first waves: every (frontier pixel, overlapping image) pair is
    // one lane's candidate; pairs run in pixel-major, image order, so the push
    // lists come out in the reference's order. Every pixel counts D pairs; those
    // beyond its image's list are empty.
    while (m.deg > 0 && head < cnt && !over) {
      const int tail = cnt;
      int i = head + lane / D, k = lane - (lane / D) * D;
      uint32_t place = kNoKey;
      if (kTable && i < tail) place = m.proj[(size_t)sh.gid[i] * m.deg + k];
      while (__any_sync(0xffffffffu, i < tail)) {
        // The next round's pair and place.
        int ni = i + q32, nk = k + r32;
        if (nk >= D) { nk -= D; ++ni; }
        uint32_t nplace = kNoKey;
        if (kTable && ni < tail) nplace = m.proj[(size_t)sh.gid[ni] * m.deg + nk];
        // 0 none, 1 found/duplicate (read kidx[h] later), 2 owner of a new node, 3
        // of a pixel that was read and rejected (kept too, so that it is read once)
        int kind = 0, u = 0;
        uint32_t h = 0, q = kNoKey;
        float de = 0.f;
        int row = 0, col = 0;
        if (kTable) {
          q = place;
        } else if (i < tail) {
          const FView& fv = m.views[sh.vid[i]];
          if (fv.ov_begin + k < fv.ov_end) {
            u = m.ov[fv.ov_begin + k];
            const FView& fu = m.views[u];
            const float4 gp = m.pix[2 * (size_t)sh.gid[i]];
            if (m.trav[u] && ProjectPixel(fu, gp.x, gp.y, gp.z, &row, &col))
              q = fu.base + (uint32_t)row * (uint32_t)fu.W + (uint32_t)col;
          }
        }
        if (q != kNoKey) {
          h = ((q * 0x9E3779B1u) >> 7) & (uint32_t)(kSetSlots - 1);
          const volatile uint32_t* vkeys = sh.keys;  // other lanes insert concurrently
          uint32_t key;
          while ((key = vkeys[h]) != kNoKey && key != q) h = (h + 1) & (uint32_t)(kSetSlots - 1);
          if (key == q) {
            kind = 1;
          } else {
            // The reprojection test first: it needs no read, and most of the
            // pixels that fail fail it.
            if (kTable) u = m.ov[m.views[sh.vid[i]].ov_begin + k];
            const FView& fu = m.views[u];
            if (kTable) RowAndColumn(q - fu.base, fu.W, &row, &col);
            float pc, pr, pz;
            if (u < 32) {
              pc = sh.seed[0][u];
              pr = sh.seed[1][u];
              pz = sh.seed[2][u];
            } else {
              const float p0 = Dot4p(fu.P, sp.x, sp.y, sp.z, 1.0f), p1 = Dot4p(fu.P + 4, sp.x, sp.y, sp.z, 1.0f);
              pz = Dot4p(fu.P + 8, sp.x, sp.y, sp.z, 1.0f);
              pc = __fdiv_rn(p0, pz);
              pr = __fdiv_rn(p1, pz);
            }
            const float cdiff = __fsub_rn(pc, (float)col), rdiff = __fsub_rn(pr, (float)row);
            const float sq = __fadd_rn(__fmul_rn(cdiff, cdiff), __fmul_rn(rdiff, rdiff));
            const bool close = m.trav[u] && !(sq > c.max_sq_reproj);
            bool ok = close;
            if (close) {
              const uint8_t fused = m.mask[q];
              const float4 xq = m.pix[2 * (size_t)q], nq = m.pix[2 * (size_t)q + 1];
              ok = !fused && ValidDepth(xq.w);
              if (ok) {
                de = __fdiv_rn(fabsf(__fsub_rn(pz, xq.w)), xq.w);
                ok = !(de > c.derr_thr);
              }
              if (ok && c.with_normal) ok = !(Dot3(sn.x, sn.y, sn.z, nq.x, nq.y, nq.z) < c.min_cos);
            }
            if (ok || (close && rejected < kMaxRejected)) {  // claim a slot; a lane of this round may hold the same pixel
              for (;;) {
                const uint32_t old = atomicCAS(&sh.keys[h], kNoKey, q);
                if (old == kNoKey) { kind = ok ? 2 : 3; break; }
                if (old == q) { kind = 1; break; }
                h = (h + 1) & (uint32_t)(kSetSlots - 1);
              }
              if (kind == 3) sh.kidx[h] = kReject;
            }
          }
        }
        __syncwarp();
        const unsigned fresh = __ballot_sync(0xffffffffu, kind == 2);
        int j = -1;
        if (kind == 2) {
          j = cnt + __popc(fresh & lt);
          if (j < im.cap) {
            sh.kidx[h] = (uint16_t)j;
            sh.gid[j] = q;
            sh.vid[j] = (uint16_t)u;
            derr[j] = de;
          }
        }
        cnt += __popc(fresh);
        rejected += __popc(__ballot_sync(0xffffffffu, kind == 3));
        if (cnt > im.cap) over = true;
        __syncwarp();
        if (kind == 1) {
          const uint32_t e = sh.kidx[h];
          j = e == kReject ? -1 : (int)e;
        }
        const unsigned val = __ballot_sync(0xffffffffu, j >= 0);
        const uint32_t at = ecur + (uint32_t)__popc(val & lt);
        if (!over) {
          if (i < tail && k == 0) eoff[i] = at;
          if (j >= 0 && at < (uint32_t)kEdgeLocal) edges[at] = (uint8_t)j;
        }
        ecur += (uint32_t)__popc(val);
        if (ecur > (uint32_t)kEdgeLocal) over = true;
        __syncwarp();
        if (over) break;
        i = ni;
        k = nk;
        place = nplace;
      }
      head = tail;
    }
    if (!over && lane == 0) eoff[cnt] = ecur;
    __syncwarp();
    if (over) {
      if (lane == 0) {
        r.rec_off[s] = kOver;
        const uint32_t k = atomicAdd(r.n_over, 1u);
        r.over_list[k] = s;
      }
      continue;
    }
    // The record, written by the warp.
    const uint32_t ne = ecur;
    const uint32_t words = RecWords((uint32_t)cnt, ne);
    unsigned long long off = 0;
    if (lane == 0) off = atomicAdd(r.used, (unsigned long long)words);
    off = __shfl_sync(0xffffffffu, off, 0);
    if (off + words > r.pool_words || off + words > 0xfffffff0ull) {
      if (lane == 0) {
        atomicOr(&r.stats[2], kStPool);
        r.rec_off[s] = kRetry;
      }
      continue;
    }
    uint32_t* rec = r.pool + off;
    uint32_t* rg = rec + 2;
    float* rd = reinterpret_cast<float*>(rg + cnt);
    uint32_t* reo = reinterpret_cast<uint32_t*>(rd + cnt);
    uint16_t* rv = reinterpret_cast<uint16_t*>(reo + cnt + 1);
    uint8_t* redg = reinterpret_cast<uint8_t*>(rv + 2 * ((cnt + 1) / 2));
    for (int k = lane; k < cnt; k += 32) {
      rg[k] = sh.gid[k];
      rd[k] = derr[k];
      rv[k] = sh.vid[k];
    }
    for (int k = lane; k <= cnt; k += 32) reo[k] = eoff[k];
    for (uint32_t k = lane; k < (ne + 3u) / 4u; k += 32)
      reinterpret_cast<uint32_t*>(redg)[k] = reinterpret_cast<const uint32_t*>(edges)[k];
    if (lane == 0) {
      rec[0] = (uint32_t)cnt;
      rec[1] = ne;
      r.rec_off[s] = (uint32_t)off;
      atomicMax(&r.stats[0], (uint32_t)cnt);
      atomicMax(&r.stats[1], ne);
    }
    __syncwarp();
  }
}

// Seeds over the closure pass's capacity, with their scratch in global memory.
__global__ void __launch_bounds__(64) ClosureBigKernel(FMaps m, FConsts c, FImage im, FRecs r, uint32_t first,
                                                       uint32_t count, uint8_t* scratch) {
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= count) return;
  const uint32_t s = r.over_list[first + t];
  uint8_t* base = scratch + (size_t)t * kBigStride;
  uint32_t* gid = reinterpret_cast<uint32_t*>(base);
  float* derr = reinterpret_cast<float*>(base + (size_t)kBigCap * 4u);
  uint16_t* vid = reinterpret_cast<uint16_t*>(base + (size_t)kBigCap * 8u);
  uint16_t* slots = reinterpret_cast<uint16_t*>(base + kBigSlotsOff);
  uint32_t* eoff = reinterpret_cast<uint32_t*>(base + kBigEoffOff);
  const NodeSet set{slots, (uint32_t)kBigSetSlots - 1u};
  uint32_t ne = 0;
  const int cnt = BuildClosure(m, c, SeedPixel(m, im, s), im.view, gid, vid, derr, set, kBigCap, eoff, nullptr, 0,
                               &ne);
  if (cnt <= 0) {  // cannot be empty here; over kBigCap is reported
    if (cnt < 0) atomicOr(&r.stats[2], kStBig);
    r.rec_off[s] = kEmpty;
    return;
  }
  WriteRecord(m, r, s, gid, vid, derr, set, cnt, eoff, nullptr, 0, false);
}

// ---- claims and predecessors ------------------------------------------------
struct RecView {
  uint32_t cnt, ne;
  const uint32_t* gid;
  const float* derr;
  const uint32_t* eoff;
  const uint16_t* vid;
  const uint16_t* edges;  // of a record over kCap pixels, else edges8
  const uint8_t* edges8;
};

__device__ __forceinline__ RecView OpenRecord(uint32_t* pool, uint32_t off) {
  RecView v;
  uint32_t* rec = pool + off;
  v.cnt = rec[0];
  v.ne = rec[1];
  v.gid = rec + 2;
  v.derr = reinterpret_cast<const float*>(v.gid + v.cnt);
  v.eoff = rec + 2 + 2 * v.cnt;
  v.vid = reinterpret_cast<const uint16_t*>(v.eoff + v.cnt + 1);
  v.edges = v.vid + 2 * ((v.cnt + 1) / 2);
  v.edges8 = reinterpret_cast<const uint8_t*>(v.edges);
  return v;
}

// One warp per seed in the claim and predecessor kernels: lanes take the
// record's pixels, so the record is read coalesced and the atomics of a seed
// are in flight together.
__global__ void __launch_bounds__(256) ClaimCountKernel(FRecs r, uint32_t nseeds, uint32_t* claim_cnt) {
  const uint32_t s = (uint32_t)(((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  const uint32_t lane = threadIdx.x & 31;
  if (s >= nseeds) return;
  const uint32_t off = r.rec_off[s];
  if (off >= kRetry) return;
  const RecView v = OpenRecord(r.pool, off);
  for (uint32_t k = lane; k < v.cnt; k += 32) atomicAdd(&claim_cnt[v.gid[k]], 1u);
}

__global__ void __launch_bounds__(256) ClaimFillKernel(FRecs r, uint32_t nseeds, uint32_t* claim_cnt,
                                                       const uint32_t* claim_off, uint32_t* claim_list) {
  const uint32_t s = (uint32_t)(((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  const uint32_t lane = threadIdx.x & 31;
  if (s >= nseeds) return;
  const uint32_t off = r.rec_off[s];
  if (off >= kRetry) return;
  const RecView v = OpenRecord(r.pool, off);
  for (uint32_t k = lane; k < v.cnt; k += 32) {
    const uint32_t g = v.gid[k];
    const uint32_t slot = atomicSub(&claim_cnt[g], 1u) - 1u;  // leaves claim_cnt at zero
    claim_list[claim_off[g] + slot] = s;
  }
}

// The predecessors of a seed are the earlier seeds that claim one of its pixels,
// each once (the replay waits for all of them). They are listed as the pixels of
// those seeds, whose masks the replay polls: a seed is settled once its own
// pixel is fused. Also the shear K of the ticket order: key(p) < key(s) for every
// predecessor p of s needs K (i_s - i_p) > j_p - j_s.
struct FPreds {
  uint32_t* off;   // per seed: first entry in list
  uint32_t* cnt;   // per seed: entries, or kWalk: walk the claims of the record's pixels
  uint32_t* list;  // seed pixels
  unsigned long long* used;
  unsigned long long cap;
  const uint32_t* claim_off;
  const uint32_t* claim_list;
};
constexpr uint32_t kWalk = 0xffffffffu;
constexpr int kFarSlots = 128;   // hash slots of the distinct predecessors outside the window
constexpr int kFarMost = 64;     // with more of them the replay walks the claims

// One warp per seed. Nearly all predecessors lie in the seed grid's 8 rows x 32
// columns up to the seed (a record's pixels are within the reprojection radius of
// its seed's point), so they are collected as bits of 8 words, each set once: a
// claim whose bit is set costs a read and a test. The others go through a small
// hash set. Measured with the claim kernels on the first image of 11 views
// 1600x1200 (some 640 claims a seed): 9.2 ms; 22 with one hash set for all.
__global__ void __launch_bounds__(256) PredKernel(FMaps m, FImage im, FRecs r, FPreds pr, int* shear) {
  __shared__ uint32_t far_all[8][kFarSlots];
  __shared__ uint32_t near_all[8][8];
  __shared__ uint32_t count_all[8];
  const uint32_t s = (uint32_t)(((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  uint32_t* keys = far_all[w];
  uint32_t* near = near_all[w];
  volatile uint32_t* count = count_all + w;
  if (s >= im.nseeds) return;
  const uint32_t off = r.rec_off[s];
  if (off >= kRetry) return;
  const RecView v = OpenRecord(r.pool, off);
  for (int i = lane; i < kFarSlots; i += 32) keys[i] = kNoKey;
  if (lane < 8) near[lane] = 0u;
  if (lane == 0) *count = 0;
  __syncwarp();
  const uint32_t Cs = (uint32_t)im.Cs;
  const float inv_cs = 1.0f / (float)im.Cs;
  const volatile uint32_t* vnear = near;
  const volatile uint32_t* vk = keys;
  auto add = [&](uint32_t cl) {
    if (cl >= s) return;
    // s - cl = rows * Cs + columns with columns in [-16, 15].
    const uint32_t d = s - cl + 16u;
    const uint32_t row = (uint32_t)((float)d * inv_cs);
    const uint32_t bit = d - row * Cs;  // wraps to a large value where row was rounded up
    if (Cs >= 32u && row < 8u && bit < 32u) {
      if (!((vnear[row] >> bit) & 1u)) atomicOr(near + row, 1u << bit);
      return;
    }
    if (*count > (uint32_t)kFarMost) return;  // the table never fills up
    uint32_t h = (cl * 0x9E3779B1u) >> 25;  // 128 slots
    for (;;) {
      uint32_t key = vk[h];
      if (key == kNoKey) key = atomicCAS(keys + h, kNoKey, cl);
      if (key == kNoKey) { atomicAdd(count_all + w, 1u); return; }
      if (key == cl) return;
      h = (h + 1) & (uint32_t)(kFarSlots - 1);
    }
  };
  for (uint32_t k = lane; k < v.cnt; k += 32) {
    const uint32_t g = v.gid[k];
    const uint32_t end = pr.claim_off[g + 1];
    for (uint32_t q = pr.claim_off[g]; q < end; q += 4) {  // four claims in flight
      const uint32_t c0 = pr.claim_list[q];
      const uint32_t c1 = q + 1 < end ? pr.claim_list[q + 1] : s;
      const uint32_t c2 = q + 2 < end ? pr.claim_list[q + 2] : s;
      const uint32_t c3 = q + 3 < end ? pr.claim_list[q + 3] : s;
      add(c0);
      add(c1);
      add(c2);
      add(c3);
    }
  }
  __syncwarp();
  const uint32_t nfar = *count;
  uint32_t n = nfar;
  for (int i = 0; i < 8; ++i) n += (uint32_t)__popc(near[i]);
  unsigned long long at = 0;
  const bool many = nfar > (uint32_t)kFarMost;
  if (lane == 0 && n > 0 && !many) at = atomicAdd(pr.used, (unsigned long long)n);
  at = __shfl_sync(0xffffffffu, at, 0);
  const bool walk = many || at + n > pr.cap;
  if (lane == 0) {
    pr.off[s] = (uint32_t)at;
    pr.cnt[s] = walk ? kWalk : n;
  }
  // The list, and what the predecessors need of the shear (with too many far
  // ones, of every claim).
  const int is = (int)(s / Cs), js = (int)(s - (uint32_t)is * Cs);
  int need = 1;
  auto shear_of = [&](uint32_t p) {
    const int ip = (int)(p / Cs), jp = (int)(p - (uint32_t)ip * Cs);
    if (ip < is) {
      const int num = jp - js, den = is - ip;
      const int fl = num >= 0 ? num / den : -((-num + den - 1) / den);
      need = max(need, fl + 1);
    }
  };
  if (many) {
    for (uint32_t k = lane; k < v.cnt; k += 32) {
      const uint32_t g = v.gid[k];
      for (uint32_t q = pr.claim_off[g], end = pr.claim_off[g + 1]; q < end; ++q)
        if (pr.claim_list[q] < s) shear_of(pr.claim_list[q]);
    }
  } else {
    uint32_t pos = 0;
    auto put = [&](bool has, uint32_t p) {
      const unsigned who = __ballot_sync(0xffffffffu, has);
      if (has) {
        shear_of(p);
        if (!walk) pr.list[at + pos + (uint32_t)__popc(who & ((1u << lane) - 1u))] = SeedPixel(m, im, p);
      }
      pos += (uint32_t)__popc(who);
    };
    for (uint32_t row = 0; row < 8; ++row) put((near[row] >> lane) & 1u, s + 16u - row * Cs - lane);
    if (nfar > 0)
      for (int i0 = 0; i0 < kFarSlots; i0 += 32) put(keys[i0 + lane] != kNoKey, keys[i0 + lane]);
  }
  for (int o = 16; o > 0; o >>= 1) need = max(need, __shfl_xor_sync(0xffffffffu, need, o));
  if (lane == 0 && need > 1) atomicMax(shear, min(need, im.Cs));
}

// ---- ticket order ------------------------------------------------------------
__device__ __forceinline__ int KeyRowMin(long long k, int Cs, int K) {
  const long long num = k - Cs + 1;
  return num <= 0 ? 0 : (int)((num + K - 1) / K);
}

__global__ void KeyCountKernel(uint32_t nkeys_cap, int Rs, int Cs, const int* shear, uint32_t* keycnt) {
  const int K = *shear;
  for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < nkeys_cap; k += gridDim.x * blockDim.x) {
    const int imin = KeyRowMin(k, Cs, K);
    const int imax = min(Rs - 1, (int)(k / (uint32_t)K));
    keycnt[k] = imax >= imin ? (uint32_t)(imax - imin + 1) : 0u;
  }
}

__global__ void SeqKernel(uint32_t nseeds, int Cs, const int* shear, const uint32_t* keyoff, uint32_t* seq) {
  const int K = *shear;
  const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= nseeds) return;
  const int i = (int)(s / (uint32_t)Cs), j = (int)(s - (uint32_t)i * (uint32_t)Cs);
  const long long k = (long long)j + (long long)K * i;
  seq[keyoff[k] + (uint32_t)(i - KeyRowMin(k, Cs, K))] = s;
}

// ---- replay -----------------------------------------------------------------
struct FReplay {
  const uint32_t* seq;
  uint32_t nseeds;
  FImage im;
  FPreds preds;
  unsigned int* ticket;
  smvs_fused_point* slot_pts;
  uint32_t* slot_has;
  uint32_t* slot_nvis;
  uint32_t* slot_visoff;
  uint32_t* vis_pool;
  unsigned long long* vis_cursor;
  uint8_t* scratch;           // per-warp scratch for records over the shared budget
  uint32_t scratch_cnt;       // node capacity of a scratch region
  uint32_t scratch_stack;     // stack capacity of a scratch region
  int shared_cnt;             // records up to this many pixels ...
  int shared_stack;           // ... and stack entries replay in shared memory
  uint32_t* level;            // with profiling: dependency depth by seed pixel of the image (else null)
  uint32_t* chain;            // with profiling: the image's longest dependency chain
  unsigned long long* times;  // with profiling: summed ns [waiting, after the wait until release], seeds
  unsigned long long wait_limit_ns;  // bound of a predecessor wait
  long long withhold;         // test hook: this seed's successors are never released (-1: none, -2: all)
};

struct alignas(16) WarpShared {
  alignas(16) float vals[kCap];  // read as uint4 by WarpMedian64
  uint32_t stack[kStackSh];
  uint32_t gid[kCap];        // the record's pixels, staged before the wait
  uint32_t ids[kCap];
  uint16_t acc[kCap];
  uint8_t flags[kCap];
  uint8_t node[kCap];        // the open pixels (not fused before the wait) in the record
  uint8_t place[kCap];       // and a record pixel's place among them
  uint32_t images[32];       // images of the cluster (the first 1024)
  float med[2];
  int nacc;
};
constexpr int kOpenMost = 128;  // open pixels searched in registers

__device__ __forceinline__ uint32_t LoadMask(const uint8_t* p) {
  uint32_t v;
  asm volatile("ld.relaxed.gpu.global.u8 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void StoreMask(uint8_t* p) {
  asm volatile("st.relaxed.gpu.global.u8 [%0], %1;" ::"l"(p), "r"(1u) : "memory");
}
__device__ __forceinline__ unsigned long long GlobalTimer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Median over vals[0..n) (internal::Median, fusion.cc:47-60) in the total
// order of FKey; ties between equal keys are broken by position.
__device__ float WarpMedian(const float* vals, int n, float* med, int lane) {
  const int mid = n / 2;
  for (int i = lane; i < n; i += 32) {
    const uint32_t ki = FKey(vals[i]);
    int rank = 0;
    for (int j = 0; j < n; ++j) {
      const uint32_t kj = FKey(vals[j]);
      rank += (kj < ki || (kj == ki && j < i)) ? 1 : 0;
    }
    if (rank == mid) med[0] = vals[i];
    if ((n & 1) == 0 && rank == mid - 1) med[1] = vals[i];
  }
  __syncwarp();
  const float r = (n & 1) ? med[0] : __fdiv_rn(__fadd_rn(med[0], med[1]), 2.0f);
  __syncwarp();
  return r;
}

// The same for n <= 64 values, lane l holding values l and l + 32 (anything
// beyond n; `vals`: 64 words on a 16-byte boundary): each lane ranks its two against all keys, read four at a time.
__device__ __forceinline__ float WarpMedian64(float a, float b, int n, float* vals, float* med, int lane) {
  uint32_t* keys = reinterpret_cast<uint32_t*>(vals);
  const uint32_t ka = lane < n ? FKey(a) : 0xffffffffu, kb = lane + 32 < n ? FKey(b) : 0xffffffffu;
  keys[lane] = ka;
  keys[lane + 32] = kb;
  __syncwarp();
  // Keys below, and keys equal and before (ties are broken by position). The
  // padding is the largest key and comes last.
  int ra = 0, rb = 0;
  for (int j = 0; j < n; j += 4) {
    const uint4 k = *reinterpret_cast<const uint4*>(keys + j);
    ra += (k.x < ka || (k.x == ka && j < lane)) + (k.y < ka || (k.y == ka && j + 1 < lane)) +
          (k.z < ka || (k.z == ka && j + 2 < lane)) + (k.w < ka || (k.w == ka && j + 3 < lane));
    if (n > 32)
      rb += (k.x < kb || (k.x == kb && j < lane + 32)) + (k.y < kb || (k.y == kb && j + 1 < lane + 32)) +
            (k.z < kb || (k.z == kb && j + 2 < lane + 32)) + (k.w < kb || (k.w == kb && j + 3 < lane + 32));
  }
  const int mid = n / 2;
  if (lane < n) {
    if (ra == mid) med[0] = a;
    if ((n & 1) == 0 && ra == mid - 1) med[1] = a;
  }
  if (lane + 32 < n) {
    if (rb == mid) med[0] = b;
    if ((n & 1) == 0 && rb == mid - 1) med[1] = b;
  }
  __syncwarp();
  const float r = (n & 1) ? med[0] : __fdiv_rn(__fadd_rn(med[0], med[1]), 2.0f);
  __syncwarp();
  return r;
}

// Waits until the masks of the seed pixels that the lanes hold (bit i of `pending`:
// pixel[i]) are set, or the seed's own pixel is (true: another seed fused it,
// nothing is left to do). A short spin, then a back-off; bounded in time (status
// bit on timeout). Called by the whole warp.
__device__ __forceinline__ bool WaitSettled(const uint8_t* mask, uint32_t own, const uint32_t pixel[4],
                                            uint32_t pending, uint32_t* stats, unsigned long long limit_ns) {
  const int lane = threadIdx.x & 31;
  unsigned long long t0 = 0;
  for (uint32_t it = 0;; ++it) {
    uint32_t set[4] = {0u, 0u, 0u, 0u};
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if ((pending >> i) & 1u) set[i] = LoadMask(mask + pixel[i]);
    bool fused = false;
    if (lane == 31) fused = LoadMask(mask + own) != 0u;
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (set[i]) pending &= ~(1u << i);
    const unsigned open = __ballot_sync(0xffffffffu, pending != 0u);
    if (__any_sync(0xffffffffu, fused)) return true;
    if (!open) return false;
    if (it < 16) continue;
    __nanosleep(it < 64 ? 32 : 128);
    if ((it & 63u) != 16u) continue;
    const unsigned long long t = __shfl_sync(0xffffffffu, GlobalTimer(), 0);
    if (t0 == 0) t0 = t;
    // One wait that gave up ends the others too.
    const uint32_t status = *(volatile const uint32_t*)(stats + 2);
    if (t - t0 > limit_ns || __any_sync(0xffffffffu, (status & kStTimeout) != 0u)) {
      if (lane == 0) atomicOr(&stats[2], kStTimeout);
      return false;
    }
  }
}

// The reference's traversal (:1836-2094) on a record, by one lane: LIFO stack
// of (pixel, traversal depth). flags: nonzero = already fused; accepted pixels
// are flagged and listed in acc in the order the reference fuses them. A
// pushed pixel that is already fused would be skipped when popped, so it is
// not pushed. Returns the number accepted.
template <typename Edge>
__device__ int SeqTraversal(uint8_t* __restrict__ flags, uint32_t* __restrict__ stack, uint16_t* __restrict__ acc,
                            const uint32_t* __restrict__ reoff, const Edge* __restrict__ redges, int max_pix,
                            int max_depth) {
  int nacc = 0, top = 0;
  if (!flags[0]) stack[top++] = 0u;
  while (top > 0) {
    const uint32_t e = stack[--top];
    const uint32_t k = e & 0xffffu, d = e >> 16;
    if (flags[k]) continue;
    flags[k] = 1;
    acc[nacc++] = (uint16_t)k;
    if (nacc >= max_pix) break;
    if ((int)d + 1 >= max_depth) continue;
    const uint32_t nd = (d + 1 < 0xffffu ? d + 1 : 0xffffu) << 16;
    uint32_t q = reoff[k];
    const uint32_t qe = reoff[k + 1];
    // Four pushes at a time: the loads of a batch overlap (pushes only write
    // the stack, so the flags they read do not change within the batch).
    for (; q + 4 <= qe; q += 4) {
      const uint32_t j0 = redges[q], j1 = redges[q + 1], j2 = redges[q + 2], j3 = redges[q + 3];
      const uint8_t f0 = flags[j0], f1 = flags[j1], f2 = flags[j2], f3 = flags[j3];
      if (!f0) stack[top++] = j0 | nd;
      if (!f1) stack[top++] = j1 | nd;
      if (!f2) stack[top++] = j2 | nd;
      if (!f3) stack[top++] = j3 | nd;
    }
    for (; q < qe; ++q) {
      const uint32_t j = redges[q];
      if (!flags[j]) stack[top++] = j | nd;
    }
  }
  return nacc;
}

// Bound by its chain of dependent seeds (the first image of 11 views 1600x1200: 2,759
// run one after another, each fusing some 36 pixels): what counts is the time
// from a predecessor's mark to this seed's, so everything that does not depend on
// the masks is done before the wait. 16 to 20 warps an SM are enough, more only
// share the issue slots with the seeds on the chain. Measured for that image:
// 65.6 ms when every earlier claimant's ticket was waited for and the search read
// its push lists after the wait, now 27.6.
__global__ void __launch_bounds__(32 * kReplayWarps, 4) ReplayKernel(FMaps m, FConsts c, FRecs r, FReplay rp) {
  __shared__ WarpShared shm[kReplayWarps];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  WarpShared& sh = shm[w];
  const size_t gw = (size_t)blockIdx.x * kReplayWarps + w;
  for (;;) {
    uint32_t t = 0;
    if (lane == 0) t = atomicAdd(rp.ticket, 1u);
    t = __shfl_sync(0xffffffffu, t, 0);
    if (t >= rp.nseeds) break;
    const uint32_t s = rp.seq[t];
    const uint32_t off = r.rec_off[s];
    if (off >= kRetry) continue;  // no record: nothing to fuse, nobody waits for it
    const uint32_t own = SeedPixel(m, rp.im, s);
    if (__any_sync(0xffffffffu, LoadMask(m.mask + own) != 0u)) continue;  // fused by an earlier seed
    const RecView v = OpenRecord(r.pool, off);
    const int cnt = (int)v.cnt;
    // Storage: the per-pixel arrays in shared memory when the record has at
    // most shared_cnt pixels, the stack when it fits shared_stack entries, and
    // the record itself staged there when it fits; anything larger lives in
    // this warp's global scratch (or is read from the record in place).
    const bool node_sh = cnt <= rp.shared_cnt;
    const bool stack_sh = v.ne + 1 <= (uint32_t)rp.shared_stack;
    if ((!node_sh && (uint32_t)cnt > rp.scratch_cnt) || (!stack_sh && v.ne + 1 > rp.scratch_stack) ||
        ((!node_sh || !stack_sh) && !rp.scratch)) {
      if (lane == 0) {
        atomicOr(&r.stats[2], kStBad);
        StoreMask(m.mask + own);
      }
      continue;
    }
    uint8_t* base = rp.scratch ? rp.scratch + gw * ScratchPer(rp.scratch_cnt, rp.scratch_stack) : nullptr;
    uint32_t* stack = stack_sh ? sh.stack : reinterpret_cast<uint32_t*>(base);
    float* vals;
    uint32_t* ids;
    uint16_t* acc;
    uint8_t* flags;
    if (node_sh) {
      vals = sh.vals;
      ids = sh.ids;
      acc = sh.acc;
      flags = sh.flags;
    } else {
      vals = reinterpret_cast<float*>(base + (size_t)rp.scratch_stack * 4u);
      ids = reinterpret_cast<uint32_t*>(base + (size_t)rp.scratch_stack * 4u + (size_t)rp.scratch_cnt * 4u);
      acc = reinterpret_cast<uint16_t*>(base + (size_t)rp.scratch_stack * 4u + (size_t)rp.scratch_cnt * 8u);
      flags = base + (size_t)rp.scratch_stack * 4u + (size_t)rp.scratch_cnt * 10u;
    }
    const uint32_t* rgid = v.gid;
    const uint32_t* reoff = v.eoff;
    // A record over kCap pixels has 16-bit push lists.
    const bool wide = cnt > kCap;
    const uint8_t* redges = v.edges8;
    // Before the wait: the pixels that earlier seeds have not fused yet (marks
    // are never taken back), and their push lists as bits. Lane l holds the rows
    // of open pixels l, l + 32, l + 64 and l + 96, so that a step of the search
    // after the wait, which every successor waits for, is four tests and four
    // warp-wide ORs.
    int nopen = kOpenMost + 1;
    uint32_t rows[4][4], open_gid[4];
    if (node_sh) {
      nopen = 0;
      for (int k0 = 0; k0 < cnt; k0 += 32) {
        const int k = k0 + lane;
        bool is_open = false;
        if (k < cnt) {
          const uint32_t g = v.gid[k];
          sh.gid[k] = g;
          const uint8_t f = __ldcg(m.mask + g);
          flags[k] = f;
          is_open = f == 0;
        }
        const unsigned who = __ballot_sync(0xffffffffu, is_open);
        if (is_open) {
          const int at = nopen + __popc(who & ((1u << lane) - 1u));
          sh.node[at] = (uint8_t)k;
          sh.place[k] = (uint8_t)at;
        }
        nopen += __popc(who);
      }
      __syncwarp();
      if (flags[0]) continue;  // fused by an earlier seed
      rgid = sh.gid;
      if (nopen <= kOpenMost) {
#pragma unroll
        for (int a = 0; a < 4; ++a) {
          rows[a][0] = rows[a][1] = rows[a][2] = rows[a][3] = 0u;
          open_gid[a] = own;
          const int i = lane + 32 * a;
          if (i >= nopen) continue;
          const int k = sh.node[i];
          open_gid[a] = sh.gid[k];
          for (uint32_t q = reoff[k], qe = reoff[k + 1]; q < qe; ++q) {
            const uint32_t j = redges[q];
            if (flags[j]) continue;
            const uint32_t at = sh.place[j], bit = 1u << (at & 31u), word = at >> 5;
#pragma unroll
            for (uint32_t t = 0; t < 4; ++t) rows[a][t] |= word == t ? bit : 0u;
          }
        }
      }
    }
    const bool in_regs = nopen <= kOpenMost;
    auto traverse = [&]() -> int {
      return wide ? SeqTraversal(flags, stack, acc, reoff, v.edges, c.max_pix, c.max_depth)
                  : SeqTraversal(flags, stack, acc, reoff, redges, c.max_pix, c.max_depth);
    };
    unsigned long long tw0 = 0;
    if (rp.times) tw0 = GlobalTimer();
    // Wait for the predecessors (every earlier seed that may touch these
    // pixels) until each is settled: it has run, or an earlier seed fused its
    // pixel and it never will. A seed marks its own pixel last, so all its marks
    // are visible then; a seed fused by another leaves none. The wait ends at
    // once when another seed has fused this one's pixel.
    bool fused = false;
    const uint32_t npred = rp.preds.cnt[s];
    if (npred != kWalk) {
      const uint32_t* list = rp.preds.list + rp.preds.off[s];
      for (uint32_t k0 = 0; k0 < npred && !fused; k0 += 128) {
        uint32_t pixel[4], some = 0u;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const uint32_t k = k0 + 32u * i + lane;
          pixel[i] = k < npred ? list[k] : own;
          some |= k < npred ? 1u << i : 0u;
        }
        fused = WaitSettled(m.mask, own, pixel, some, r.stats, rp.wait_limit_ns);
      }
    } else {
      for (int k = 0; k < cnt && !fused; ++k) {
        const uint32_t g = v.gid[k];
        const uint32_t c1 = rp.preds.claim_off[g + 1];
        for (uint32_t q0 = rp.preds.claim_off[g]; q0 < c1 && !fused; q0 += 32) {
          const uint32_t cl = q0 + lane < c1 ? rp.preds.claim_list[q0 + lane] : s;
          const uint32_t pixel[4] = {cl < s ? SeedPixel(m, rp.im, cl) : own, own, own, own};
          fused = WaitSettled(m.mask, own, pixel, cl < s ? 1u : 0u, r.stats, rp.wait_limit_ns);
        }
      }
    }
    if (fused) continue;
    // Orders the predecessors' marks, seen above, before these reads for the
    // whole warp (the barrier orders the lanes).
    __threadfence();
    __syncwarp();
    unsigned long long tw1 = 0;
    if (rp.times) tw1 = GlobalTimer();
    // Masks are read from L2 (ld.global.cg): other SMs wrote them; a batch of
    // loads is in flight at once.
    uint32_t open[4] = {0u, 0u, 0u, 0u};  // the same in every lane
    if (in_regs) {
      uint8_t f[4];
#pragma unroll
      for (int a = 0; a < 4; ++a) f[a] = lane + 32 * a < nopen ? __ldcg(m.mask + open_gid[a]) : 1;
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        open[a] = __ballot_sync(0xffffffffu, f[a] == 0);
        if (lane + 32 * a < nopen) flags[sh.node[lane + 32 * a]] = f[a];
      }
    } else {
      for (int k = lane; k < cnt; k += 128) {
        const uint8_t a0 = __ldcg(m.mask + rgid[k]);
        const uint8_t a1 = k + 32 < cnt ? __ldcg(m.mask + rgid[k + 32]) : 0;
        const uint8_t a2 = k + 64 < cnt ? __ldcg(m.mask + rgid[k + 64]) : 0;
        const uint8_t a3 = k + 96 < cnt ? __ldcg(m.mask + rgid[k + 96]) : 0;
        flags[k] = a0;
        if (k + 32 < cnt) flags[k + 32] = a1;
        if (k + 64 < cnt) flags[k + 64] = a2;
        if (k + 96 < cnt) flags[k + 96] = a3;
      }
    }
    if (rp.level) {  // profiling: the longest chain of waits ending at this seed
      uint32_t lv = 0;
      const uint32_t base_px = m.views[rp.im.view].base;
      for (uint32_t k = lane; npred != kWalk && k < npred; k += 32)
        lv = max(lv, *(volatile const uint32_t*)(rp.level + (rp.preds.list[rp.preds.off[s] + k] - base_px)));
      for (int o = 16; o > 0; o >>= 1) lv = max(lv, __shfl_xor_sync(0xffffffffu, lv, o));
      if (lane == 0) {
        rp.level[own - base_px] = lv + 1;
        atomicMax(rp.chain, lv + 1);
      }
    }
    __syncwarp();
    unsigned long long tw_m = 0;
    if (rp.times) tw_m = GlobalTimer();
    // Which record pixels the traversal fuses. Without a binding limit it fuses
    // exactly the pixels reachable from the seed through pixels not fused yet:
    // the warp finds them in parallel (state 0 free, 1 fused before, 2 reached,
    // 3 expanded). The limits cannot bind when at most min(max_num_pixels,
    // max_traversal_depth) pixels are reachable (a pixel's traversal depth is
    // below the number fused); otherwise lane 0 replays the traversal itself.
    bool in_order = false;
    if (in_regs) {
      uint32_t seen[4] = {0u, 0u, 0u, 0u}, front[4] = {open[0] & 1u, 0u, 0u, 0u};
      while (front[0] | front[1] | front[2] | front[3]) {
        uint32_t next[4] = {0u, 0u, 0u, 0u};
#pragma unroll
        for (int a = 0; a < 4; ++a) {
          seen[a] |= front[a];
          if ((front[a] >> lane) & 1u) {
#pragma unroll
            for (int t = 0; t < 4; ++t) next[t] |= rows[a][t];
          }
        }
#pragma unroll
        for (int t = 0; t < 4; ++t) front[t] = __reduce_or_sync(0xffffffffu, next[t]) & open[t] & ~seen[t];
      }
      int reach = 0;
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        if ((seen[a] >> lane) & 1u) acc[reach + __popc(seen[a] & ((1u << lane) - 1u))] = sh.node[lane + 32 * a];
        reach += __popc(seen[a]);
      }
      __syncwarp();
      if (rp.times && lane == 0) {
        atomicAdd(rp.times + 3, (unsigned long long)cnt);
        atomicAdd(rp.times + 4, (unsigned long long)reach);
        if (reach > c.max_pix || reach > c.max_depth) atomicAdd(rp.times + 5, 1ull);
      }
      if (reach > c.max_pix || reach > c.max_depth) {  // flags still hold 1 = fused before
        if (lane == 0) reach = traverse();
        reach = __shfl_sync(0xffffffffu, reach, 0);
        in_order = true;
      }
      if (lane == 0) sh.nacc = reach;
    } else {
      volatile uint8_t* vf = flags;
      if (lane == 0 && vf[0] == 0) vf[0] = 2;
      __syncwarp();
      for (;;) {
        bool any = false;
        for (int k = lane; k < cnt; k += 32) {
          if (vf[k] != 2) continue;
          vf[k] = 3;
          any = true;
          for (uint32_t q = reoff[k], qe = reoff[k + 1]; q < qe; ++q) {
            const uint32_t j = wide ? v.edges[q] : redges[q];
            if (vf[j] == 0) vf[j] = 2;
          }
        }
        __syncwarp();
        if (!__any_sync(0xffffffffu, any)) break;
      }
      int reach = 0;
      for (int k0 = 0; k0 < cnt; k0 += 32) {
        const int k = k0 + lane;
        const bool a = k < cnt && vf[k] == 3;
        const unsigned bal = __ballot_sync(0xffffffffu, a);
        if (a) acc[reach + __popc(bal & ((1u << lane) - 1u))] = (uint16_t)k;
        reach += __popc(bal);
      }
      if (rp.times && lane == 0) {
        atomicAdd(rp.times + 3, (unsigned long long)cnt);
        atomicAdd(rp.times + 4, (unsigned long long)reach);
        if (reach > c.max_pix || reach > c.max_depth) atomicAdd(rp.times + 5, 1ull);
      }
      if (reach > c.max_pix || reach > c.max_depth) {
        for (int k = lane; k < cnt; k += 32) vf[k] = vf[k] == 1 ? 1 : 0;
        __syncwarp();
        if (lane == 0) reach = traverse();
        reach = __shfl_sync(0xffffffffu, reach, 0);
        in_order = true;
      }
      if (lane == 0) sh.nacc = reach;
    }
    __syncwarp();
    const int n = sh.nacc;
    unsigned long long tw_b = 0;
    if (rp.times) tw_b = GlobalTimer();
    for (int i = lane; i < n; i += 32)
      if (acc[i] != 0) *(volatile uint8_t*)(m.mask + rgid[acc[i]]) = 1;
    // The seed's own pixel last, which releases the successors: the barrier and
    // the fence order every lane's marks before it.
    __syncwarp();
    if (lane == 0 && rp.withhold != -2 && (long long)s != rp.withhold) {
      __threadfence();
      StoreMask(m.mask + own);
    }
    if (rp.times && lane == 0) {
      const unsigned long long tw2 = GlobalTimer();
      atomicAdd(rp.times, tw1 - tw0);
      atomicAdd(rp.times + 1, tw2 - tw1);
      atomicAdd(rp.times + 2, 1ull);
      atomicAdd(rp.times + 6, tw_m - tw1);
      atomicAdd(rp.times + 7, tw_b - tw_m);
      atomicAdd(rp.times + 8, tw2 - tw_b);
    }
    // The fused point (:2098-2180).
    if (n < c.min_pix) continue;
    // Images of the cluster, ascending: as bits when there are at most 1024.
    const bool few_views = m.num_views <= 1024;
    int nvis = 0;
    if (few_views) {
      sh.images[lane] = 0u;
      __syncwarp();
      for (int i = lane; i < n; i += 32) {
        const uint32_t id = v.vid[acc[i]];
        atomicOr(&sh.images[id >> 5], 1u << (id & 31u));
      }
      __syncwarp();
      nvis = __reduce_add_sync(0xffffffffu, __popc(sh.images[lane]));
    } else {
      for (int i = lane; i < n; i += 32) ids[i] = v.vid[acc[i]];
      __syncwarp();
      for (int i0 = 0; i0 < n; i0 += 32) {
        const int i = i0 + lane;
        bool first = false;
        if (i < n) {
          first = true;
          for (int j = 0; j < i; ++j)
            if (ids[j] == ids[i]) {
              first = false;
              break;
            }
        }
        nvis += __popc(__ballot_sync(0xffffffffu, first));
      }
    }
    if (nvis < c.min_vis) continue;
    smvs_fused_point pt;
    memset(&pt, 0, sizeof(pt));
    const float* values = reinterpret_cast<const float*>(m.pix);  // 8 a pixel
    // Up to 64 pixels: lane l keeps the values of pixels l and l + 32 of the
    // cluster, all read at once, and the medians take them from there.
    const bool small = n <= 64;
    float4 e0a, e0b, e1a, e1b;
    uint32_t c0 = 0, c1 = 0;
    if (small) {
      const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
      e0a = e0b = e1a = e1b = zero;
      if (lane < n) {
        const size_t g = rgid[acc[lane]];
        e0a = m.pix[2 * g];
        e0b = m.pix[2 * g + 1];
        c0 = (uint32_t)m.rgb[3 * g] | (uint32_t)m.rgb[3 * g + 1] << 8 | (uint32_t)m.rgb[3 * g + 2] << 16;
      }
      if (lane + 32 < n) {
        const size_t g = rgid[acc[lane + 32]];
        e1a = m.pix[2 * g];
        e1b = m.pix[2 * g + 1];
        c1 = (uint32_t)m.rgb[3 * g] | (uint32_t)m.rgb[3 * g + 1] << 8 | (uint32_t)m.rgb[3 * g + 2] << 16;
      }
    }
    float xyz[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      if (small) {
        xyz[a] = WarpMedian64(a == 0 ? e0a.x : a == 1 ? e0a.y : e0a.z, a == 0 ? e1a.x : a == 1 ? e1a.y : e1a.z, n,
                              sh.vals, sh.med, lane);
      } else {
        for (int i = lane; i < n; i += 32) vals[i] = values[8 * (size_t)rgid[acc[i]] + a];
        __syncwarp();
        xyz[a] = WarpMedian(vals, n, sh.med, lane);
      }
    }
    if (!isfinite(xyz[0]) || !isfinite(xyz[1]) || !isfinite(xyz[2])) continue;
    pt.x = xyz[0];
    pt.y = xyz[1];
    pt.z = xyz[2];
    if (c.with_normal) {
      float fn[3];
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        if (small) {
          fn[a] = WarpMedian64(a == 0 ? e0b.x : a == 1 ? e0b.y : e0b.z, a == 0 ? e1b.x : a == 1 ? e1b.y : e1b.z, n,
                               sh.vals, sh.med, lane);
        } else {
          for (int i = lane; i < n; i += 32) vals[i] = values[8 * (size_t)rgid[acc[i]] + 4 + a];
          __syncwarp();
          fn[a] = WarpMedian(vals, n, sh.med, lane);
        }
      }
      const float norm =
          __fsqrt_rn(__fadd_rn(__fadd_rn(__fmul_rn(fn[0], fn[0]), __fmul_rn(fn[1], fn[1])), __fmul_rn(fn[2], fn[2])));
      if (norm < 1.1920928955078125e-07f) continue;  // FLT_EPSILON
      pt.nx = __fdiv_rn(fn[0], norm);
      pt.ny = __fdiv_rn(fn[1], norm);
      pt.nz = __fdiv_rn(fn[2], norm);
    }
    uint8_t rgb[3];
#pragma unroll
    for (int ch = 0; ch < 3; ++ch) {
      float med;
      if (small) {
        med = WarpMedian64((float)((c0 >> (8 * ch)) & 0xffu), (float)((c1 >> (8 * ch)) & 0xffu), n, sh.vals, sh.med,
                           lane);
      } else {
        for (int i = lane; i < n; i += 32) vals[i] = (float)m.rgb[3ull * rgid[acc[i]] + ch];
        __syncwarp();
        med = WarpMedian(vals, n, sh.med, lane);
      }
      med = roundf(med);
      med = med < 255.0f ? med : 255.0f;  // TruncateCast<float, uint8_t>
      med = med > 0.0f ? med : 0.0f;
      rgb[ch] = (uint8_t)med;
    }
    pt.r = rgb[0];
    pt.g = rgb[1];
    pt.b = rgb[2];
    // Mean gradient in traversal order, then the score (:2157-2166). The mean
    // only counts below three images; it needs the pixels in the order the
    // reference fused them, which the parallel search does not give.
    float m_conf = 1.0f;
    if (nvis < 3) {
      if (!in_order) {
        for (int k = lane; k < cnt; k += 32) flags[k] = flags[k] == 1 ? 1 : 0;
        __syncwarp();
        if (lane == 0) traverse();
        __syncwarp();
      }
      for (int i = lane; i < n; i += 32) vals[i] = values[8 * (size_t)rgid[acc[i]] + 7];
      __syncwarp();
      if (lane == 0) {
        m_conf = 0.0f;
        for (int i = 0; i < n; ++i) m_conf = __fadd_rn(m_conf, vals[i]);
        m_conf = __fdiv_rn(m_conf, (float)n);
      }
      m_conf = __shfl_sync(0xffffffffu, m_conf, 0);
    }
    m_conf = __fsub_rn(1.0f, m_conf);
    __syncwarp();
    float med_err;
    if (n - 1 <= 64) {
      med_err = WarpMedian64(lane + 1 < n ? v.derr[acc[lane + 1]] : 0.f, lane + 33 < n ? v.derr[acc[lane + 33]] : 0.f,
                             n - 1, sh.vals, sh.med, lane);
    } else {
      for (int i = lane + 1; i < n; i += 32) vals[i - 1] = v.derr[acc[i]];
      __syncwarp();
      med_err = WarpMedian(vals, n - 1, sh.med, lane);
    }
    float score = (float)((double)med_err / c.max_depth_error);
    const float mixed = __fadd_rn(__fmul_rn(0.6f, score), __fmul_rn(0.4f, m_conf));
    score = (1.0f < mixed) ? 1.0f : mixed;
    if (!isfinite(score)) continue;
    pt.score = score;
    // Output slot of this seed: the point and its images, ascending.
    uint32_t vbase = 0;
    if (lane == 0) vbase = (uint32_t)atomicAdd(rp.vis_cursor, (unsigned long long)nvis);
    vbase = __shfl_sync(0xffffffffu, vbase, 0);
    if (few_views) {
      const uint32_t mine = sh.images[lane];
      uint32_t before = (uint32_t)__popc(mine);
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, before, o);
        if (lane >= o) before += y;
      }
      before -= (uint32_t)__popc(mine);
      for (uint32_t left = mine; left; left &= left - 1u)
        rp.vis_pool[vbase + before++] = (uint32_t)(32 * lane + __ffs((int)left) - 1);
    } else {
      for (int i = lane; i < n; i += 32) {
        bool first = true;
        for (int j = 0; j < i; ++j)
          if (ids[j] == ids[i]) {
            first = false;
            break;
          }
        if (!first) continue;
        int rank = 0;  // distinct images below this one
        for (int j = 0; j < n; ++j) {
          if (ids[j] >= ids[i]) continue;
          bool fj = true;
          for (int q = 0; q < j; ++q)
            if (ids[q] == ids[j]) {
              fj = false;
              break;
            }
          rank += fj ? 1 : 0;
        }
        rp.vis_pool[vbase + rank] = ids[i];
      }
    }
    if (lane == 0) {
      rp.slot_pts[s] = pt;
      rp.slot_nvis[s] = (uint32_t)nvis;
      rp.slot_visoff[s] = vbase;
      rp.slot_has[s] = 1u;
    }
    __syncwarp();
  }
}

// ---- scan (exclusive, out[n] = total) ---------------------------------------
// A block takes kScanItems items, a thread four uint4 of them; bound by memory
// (with the four scans of an image in shared memory item by item: 0.13 ms more).
__device__ __forceinline__ uint4 ScanLoad(const uint32_t* in, uint32_t i, uint32_t n) {
  if (i + 4u <= n) return *reinterpret_cast<const uint4*>(in + i);  // i and the arrays are multiples of 4 words
  uint4 x = make_uint4(0u, 0u, 0u, 0u);
  if (i < n) x.x = in[i];
  if (i + 1u < n) x.y = in[i + 1u];
  if (i + 2u < n) x.z = in[i + 2u];
  return x;
}

__global__ void __launch_bounds__(256) ScanReduceKernel(const uint32_t* in, uint32_t n, uint32_t* sums) {
  __shared__ uint32_t red[8];
  const uint32_t b0 = blockIdx.x * (uint32_t)kScanItems;
  uint32_t acc = 0;
#pragma unroll
  for (int k = 0; k < kScanItems / 1024; ++k) {
    const uint4 x = ScanLoad(in, b0 + (uint32_t)k * 1024u + 4u * threadIdx.x, n);
    acc += x.x + x.y + x.z + x.w;
  }
  acc = __reduce_add_sync(0xffffffffu, acc);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; ++w) acc += red[w];
    sums[blockIdx.x] = acc;
  }
}

// Inclusive scan over the warp.
__device__ __forceinline__ uint32_t WarpScan(uint32_t x, int lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  return x;
}

__global__ void __launch_bounds__(1024) ScanSumsKernel(uint32_t* sums, uint32_t nb) {
  __shared__ uint32_t part[32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  uint32_t carry = 0;
  for (uint32_t b0 = 0; b0 < nb; b0 += 1024) {
    const uint32_t i = b0 + threadIdx.x;
    const uint32_t x = i < nb ? sums[i] : 0u;
    const uint32_t incl = WarpScan(x, lane);
    if (lane == 31) part[w] = incl;
    __syncthreads();
    const uint32_t p = WarpScan(part[lane], lane);  // every warp: the warps' totals
    const uint32_t before = w > 0 ? __shfl_sync(0xffffffffu, p, w - 1) : 0u;
    const uint32_t total = __shfl_sync(0xffffffffu, p, 31);
    if (i < nb) sums[i] = carry + before + incl - x;
    carry += total;
    __syncthreads();
  }
  if (threadIdx.x == 0) sums[nb] = carry;
}

__global__ void __launch_bounds__(256) ScanBlockKernel(const uint32_t* in, uint32_t n, const uint32_t* sums,
                                                       uint32_t nb, uint32_t* out) {
  constexpr int kRounds = kScanItems / 1024;
  __shared__ uint32_t part[kRounds][8];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const uint32_t b0 = blockIdx.x * (uint32_t)kScanItems;
  uint4 x[kRounds];
  uint32_t before[kRounds];  // items of the round before this thread's
#pragma unroll
  for (int k = 0; k < kRounds; ++k) {
    x[k] = ScanLoad(in, b0 + (uint32_t)k * 1024u + 4u * threadIdx.x, n);
    const uint32_t s = x[k].x + x[k].y + x[k].z + x[k].w;
    const uint32_t incl = WarpScan(s, lane);
    before[k] = incl - s;
    if (lane == 31) part[k][w] = incl;
  }
  __syncthreads();
  uint32_t carry = sums[blockIdx.x];
#pragma unroll
  for (int k = 0; k < kRounds; ++k) {
    uint32_t at = carry + before[k];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const uint32_t t = part[k][j];
      if (j < w) at += t;
      carry += t;
    }
    const uint32_t i = b0 + (uint32_t)k * 1024u + 4u * threadIdx.x;
    const uint4 o = make_uint4(at, at + x[k].x, at + x[k].x + x[k].y, at + x[k].x + x[k].y + x[k].z);
    if (i + 4u <= n) {
      *reinterpret_cast<uint4*>(out + i) = o;
    } else {
      if (i < n) out[i] = o.x;
      if (i + 1u < n) out[i + 1u] = o.y;
      if (i + 2u < n) out[i + 2u] = o.z;
    }
  }
  if (blockIdx.x == nb - 1 && threadIdx.x == 0) out[n] = sums[nb];
}

// ---- per-image bookkeeping and compaction ------------------------------------
__global__ void ImageStartKernel(int* shear, unsigned int* ticket, unsigned long long* rec_used,
                                 unsigned long long* vis_cursor, uint32_t* n_over, uint32_t* stats) {
  *shear = 1;
  *ticket = 0u;
  *rec_used = 0ull;
  *vis_cursor = 0ull;
  *n_over = 0u;
  stats[0] = 0u;
  stats[1] = 0u;
}

__global__ void CompactKernel(uint32_t nseeds, const uint32_t* slot_has, const uint32_t* pt_idx,
                              const uint32_t* vis_idx, const smvs_fused_point* slot_pts, const uint32_t* slot_nvis,
                              const uint32_t* slot_visoff, const uint32_t* vis_pool,
                              const unsigned long long* totals, smvs_fused_point* out_pts, uint64_t* out_visoff,
                              uint32_t* out_vis) {
  const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= nseeds || !slot_has[s]) return;
  const unsigned long long bp = totals[0], bv = totals[1];
  const unsigned long long dst = bp + pt_idx[s], vdst = bv + vis_idx[s];
  out_pts[dst] = slot_pts[s];
  out_visoff[dst] = vdst;
  const uint32_t nv = slot_nvis[s], src = slot_visoff[s];
  for (uint32_t i = 0; i < nv; ++i) out_vis[vdst + i] = vis_pool[src + i];
}

__global__ void AdvanceKernel(unsigned long long* totals, const uint32_t* pt_idx, const uint32_t* vis_idx,
                              uint32_t nseeds, uint64_t* out_visoff) {
  totals[0] += pt_idx[nseeds];
  totals[1] += vis_idx[nseeds];
  out_visoff[totals[0]] = totals[1];
}

}  // namespace

// ---- host object ---------------------------------------------------------------
struct smvs_fusion {
  smvs_fusion_options opt;
  int device = 0;
  cudaStream_t stream = nullptr;
  bool own_stream = false;
  cudaMemPool_t pool = nullptr;
  int num_views = 0;
  std::vector<smvs_fusion_view> views;  // sizes and poses (map pointers are not kept)
  std::vector<FView> h_views;
  std::vector<uint8_t> used, fused;
  std::vector<int32_t> ov_off, ov_img;
  std::vector<int> order;
  uint64_t total = 0;  // pixels of all images
  FConsts consts{};
  // Device arrays.
  FView* d_views = nullptr;
  int* d_ov = nullptr;
  uint8_t* d_trav = nullptr;
  float4* d_pix = nullptr;    // 2 per pixel (FMaps::pix)
  uint32_t* d_proj = nullptr; // FMaps::proj, when it fits
  float* d_depth_in = nullptr;  // the depth map that is being taken in (during create)
  int deg = 0;                // overlapping images of the image that has most
  bool walk = false;          // test hook: the replay walks the claims
  uint8_t* d_rgb = nullptr;
  uint8_t* d_mask = nullptr;
  uint32_t *d_claim_cnt = nullptr, *d_claim_off = nullptr, *d_claim_list = nullptr;
  size_t claim_list_cap = 0;
  uint32_t* d_pool = nullptr;
  size_t pool_words = 0;
  uint32_t *d_rec_off = nullptr, *d_over_list = nullptr, *d_seq = nullptr;
  uint32_t *d_pred_off = nullptr, *d_pred_cnt = nullptr, *d_pred_list = nullptr;
  unsigned long long* d_pred_used = nullptr;
  uint32_t *d_keycnt = nullptr, *d_keyoff = nullptr;
  size_t key_cap = 0;
  smvs_fused_point* d_slot_pts = nullptr;
  uint32_t *d_slot_has = nullptr, *d_slot_nvis = nullptr, *d_slot_visoff = nullptr;
  uint32_t *d_pt_idx = nullptr, *d_vis_idx = nullptr, *d_vis_pool = nullptr;
  size_t seed_cap = 0;
  uint32_t* d_scan_sums = nullptr;
  size_t scan_sums_cap = 0;
  int* d_rows = nullptr;
  size_t rows_cap = 0;
  uint8_t* d_big_scratch = nullptr;
  uint8_t* d_replay_scratch = nullptr;
  size_t replay_scratch_bytes = 0;
  uint32_t replay_scratch_cnt = 0, replay_scratch_stack = 0;
  // Small device scalars: shear, ticket, n_over, stats[3], counters.
  int* d_shear = nullptr;
  unsigned int* d_ticket = nullptr;
  uint32_t* d_n_over = nullptr;
  uint32_t* d_stats = nullptr;
  unsigned long long* d_used = nullptr;
  unsigned long long* d_vis_cursor = nullptr;
  unsigned long long* d_totals = nullptr;  // [0] points, [1] visibility entries
  // Outputs.
  smvs_fused_point* d_out_pts = nullptr;
  uint64_t* d_out_visoff = nullptr;
  uint32_t* d_out_vis = nullptr;
  uint64_t num_points = 0, num_vis = 0;
  bool ran = false;
  int replay_blocks = 0;
  int closure_blocks = 0;
  uint8_t* d_stage = nullptr;  // the closure warps' global staging
  int cap_closure = kCap, cap_replay = kCap, cap_stack = kStackSh;
  uint32_t* d_level = nullptr;  // profiling: per-seed dependency depth, per-image longest chain
  uint32_t* d_chain = nullptr;
  unsigned long long* d_times = nullptr;  // profiling: per image [wait ns, post-wait ns, seeds]
  size_t level_cap = 0;
  int64_t launches = 0;
  std::vector<int> h_rows;
  bool profiling = false;
  struct Timed { int kind, image; cudaEvent_t a, b; };
  std::vector<double> prof_image_ms;  // 4 per image in fusion order
  std::vector<Timed> timed;
  int prof_count[4] = {0, 0, 0, 0};
  double prof_ms[4] = {0, 0, 0, 0};
};

namespace {

struct ProfScope {
  smvs_fusion* f;
  int kind;
  cudaEvent_t a = nullptr, b = nullptr;
  ProfScope(smvs_fusion* f_, int kind_) : f(f_), kind(kind_) {
    if (!f->profiling) return;
    if (cudaEventCreate(&a) != cudaSuccess || cudaEventCreate(&b) != cudaSuccess) { a = b = nullptr; return; }
    cudaEventRecord(a, f->stream);
  }
  ~ProfScope() {
    if (!a) return;
    cudaEventRecord(b, f->stream);
    f->timed.push_back({kind, (int)f->order.size(), a, b});
  }
};

void Harvest(smvs_fusion* f) {
  for (auto& t : f->timed) {
    float ms = 0.f;
    if (cudaEventSynchronize(t.b) == cudaSuccess && cudaEventElapsedTime(&ms, t.a, t.b) == cudaSuccess) {
      f->prof_count[t.kind] += 1;
      f->prof_ms[t.kind] += ms;
      if ((size_t)(4 * t.image + 4) > f->prof_image_ms.size()) f->prof_image_ms.resize(4 * t.image + 4, 0.0);
      f->prof_image_ms[4 * t.image + t.kind] += ms;
    }
    cudaEventDestroy(t.a);
    cudaEventDestroy(t.b);
  }
  f->timed.clear();
}

template <typename T>
int Alloc(smvs_fusion* f, T** p, size_t count) {
  const size_t bytes = std::max<size_t>(count * sizeof(T), 16);
  cudaError_t err = smvs_internal_alloc(reinterpret_cast<void**>(p), bytes, f->pool, f->stream);
  if (err == cudaErrorMemoryAllocation && f->d_proj) {
    // The closures can do without the projection table (and launch by whether it is
    // there): it makes room first.
    (void)cudaGetLastError();
    cudaFreeAsync(f->d_proj, f->stream);
    f->d_proj = nullptr;
    if (cudaStreamSynchronize(f->stream) == cudaSuccess && cudaMemPoolTrimTo(f->pool, 0) == cudaSuccess)
      err = smvs_internal_alloc(reinterpret_cast<void**>(p), bytes, f->pool, f->stream);
  }
  if (err != cudaSuccess) {
    *p = nullptr;
    return Fail(SMVS_ENOMEM, "fusion: device allocation of %zu bytes: %s", bytes, cudaGetErrorString(err));
  }
  return SMVS_OK;
}

template <typename T>
void Free(smvs_fusion* f, T*& p) {
  if (p) cudaFreeAsync(p, f->stream);
  p = nullptr;
}

void FreeAll(smvs_fusion* f) {
  Harvest(f);
  if (f->pool) {
    Free(f, f->d_views); Free(f, f->d_ov); Free(f, f->d_trav);
    Free(f, f->d_pix); Free(f, f->d_proj); Free(f, f->d_depth_in);
    Free(f, f->d_rgb); Free(f, f->d_mask);
    Free(f, f->d_claim_cnt); Free(f, f->d_claim_off); Free(f, f->d_claim_list);
    Free(f, f->d_pool); Free(f, f->d_rec_off); Free(f, f->d_over_list); Free(f, f->d_seq);
    Free(f, f->d_pred_off); Free(f, f->d_pred_cnt); Free(f, f->d_pred_list); Free(f, f->d_pred_used);
    Free(f, f->d_keycnt); Free(f, f->d_keyoff);
    Free(f, f->d_slot_pts); Free(f, f->d_slot_has); Free(f, f->d_slot_nvis); Free(f, f->d_slot_visoff);
    Free(f, f->d_pt_idx); Free(f, f->d_vis_idx); Free(f, f->d_vis_pool);
    Free(f, f->d_scan_sums); Free(f, f->d_rows); Free(f, f->d_big_scratch); Free(f, f->d_replay_scratch);
    Free(f, f->d_shear); Free(f, f->d_ticket); Free(f, f->d_n_over); Free(f, f->d_stats);
    Free(f, f->d_used); Free(f, f->d_vis_cursor); Free(f, f->d_totals);
    Free(f, f->d_out_pts); Free(f, f->d_out_visoff); Free(f, f->d_out_vis);
    Free(f, f->d_level); Free(f, f->d_chain); Free(f, f->d_stage); Free(f, f->d_times);
  }
  if (f->stream) cudaStreamSynchronize(f->stream);
  if (f->own_stream && f->stream) cudaStreamDestroy(f->stream);
}

// P = K [R | T] in float, Eigen's packet product of a 3x3 and a 3x4 matrix.
void ComposeP(const float K[9], const float R[9], const float T[3], float P[12]) {
  float M[12];
  for (int r = 0; r < 3; ++r) {
    M[4 * r] = R[3 * r];
    M[4 * r + 1] = R[3 * r + 1];
    M[4 * r + 2] = R[3 * r + 2];
    M[4 * r + 3] = T[r];
  }
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 4; ++j) {
      volatile float a = K[3 * i] * M[j];
      volatile float b = K[3 * i + 1] * M[4 + j];
      volatile float ab = a + b;
      volatile float c = K[3 * i + 2] * M[8 + j];
      P[4 * i + j] = ab + c;
    }
}

// [P; 0 0 0 1]^-1 in double (adjugate), rounded once.
void ComposeInvP(const float P[12], float iP[12]) {
  const double m0 = P[0], m1 = P[1], m2 = P[2], m3 = P[4], m4 = P[5], m5 = P[6], m6 = P[8], m7 = P[9], m8 = P[10];
  const double c00 = m4 * m8 - m5 * m7, c01 = m2 * m7 - m1 * m8, c02 = m1 * m5 - m2 * m4;
  const double c10 = m5 * m6 - m3 * m8, c11 = m0 * m8 - m2 * m6, c12 = m2 * m3 - m0 * m5;
  const double c20 = m3 * m7 - m4 * m6, c21 = m1 * m6 - m0 * m7, c22 = m0 * m4 - m1 * m3;
  const double det = m0 * c00 + m1 * c10 + m2 * c20;
  const double inv[9] = {c00 / det, c01 / det, c02 / det, c10 / det, c11 / det,
                         c12 / det, c20 / det, c21 / det, c22 / det};
  const double p[3] = {P[3], P[7], P[11]};
  for (int i = 0; i < 3; ++i) {
    iP[4 * i] = (float)inv[3 * i];
    iP[4 * i + 1] = (float)inv[3 * i + 1];
    iP[4 * i + 2] = (float)inv[3 * i + 2];
    iP[4 * i + 3] = (float)(-(inv[3 * i] * p[0] + inv[3 * i + 1] * p[1] + inv[3 * i + 2] * p[2]));
  }
}

// FindNextImage (fusion.cc:697-727).
int FindNextImage(const smvs_fusion* f, int prev) {
  for (int pass = 0; pass < 2; ++pass)
    for (int32_t k = f->ov_off[prev]; k < f->ov_off[prev + 1]; ++k) {
      const int i = f->ov_img[k];
      if (f->used[i] && !f->fused[i] && (pass == 1 || !f->views[i].is_rig)) return i;
    }
  for (int pass = 0; pass < 2; ++pass)
    for (int i = 0; i < f->num_views; ++i)
      if (f->used[i] && !f->fused[i] && (pass == 1 || !f->views[i].is_rig)) return i;
  return -1;
}

uint32_t Blocks(uint64_t n, int threads) { return (uint32_t)std::max<uint64_t>(1, (n + threads - 1) / threads); }

int EnsureScanSums(smvs_fusion* f, uint64_t n) {
  const size_t nb = (size_t)((n + kScanItems - 1) / kScanItems);
  if (nb + 1 <= f->scan_sums_cap) return SMVS_OK;
  Free(f, f->d_scan_sums);
  f->scan_sums_cap = 0;
  const int st = Alloc(f, &f->d_scan_sums, nb + 1);
  if (!st) f->scan_sums_cap = nb + 1;
  return st;
}

// Exclusive scan of n values into out[0..n], out[n] = total.
int Scan(smvs_fusion* f, const uint32_t* in, uint64_t n, uint32_t* out) {
  if (n == 0) return Fail(SMVS_EINVAL, "fusion: empty scan");
  int st = EnsureScanSums(f, n);
  if (st) return st;
  const uint32_t nb = (uint32_t)((n + kScanItems - 1) / kScanItems);
  ScanReduceKernel<<<nb, 256, 0, f->stream>>>(in, (uint32_t)n, f->d_scan_sums);
  ScanSumsKernel<<<1, 1024, 0, f->stream>>>(f->d_scan_sums, nb);
  ScanBlockKernel<<<nb, 256, 0, f->stream>>>(in, (uint32_t)n, f->d_scan_sums, nb, out);
  f->launches += 3;
  FU_CUDA(cudaGetLastError());
  return SMVS_OK;
}

FMaps Maps(const smvs_fusion* f) {
  FMaps m;
  m.views = f->d_views;
  m.ov = f->d_ov;
  m.trav = f->d_trav;
  m.pix = f->d_pix;
  m.proj = f->d_proj;
  m.deg = f->deg;
  m.num_views = f->num_views;
  m.rgb = f->d_rgb;
  m.mask = f->d_mask;
  return m;
}

FRecs Recs(const smvs_fusion* f) {
  FRecs r;
  r.pool = f->d_pool;
  r.pool_words = f->pool_words;
  r.used = f->d_used;
  r.rec_off = f->d_rec_off;
  r.over_list = f->d_over_list;
  r.n_over = f->d_n_over;
  r.stats = f->d_stats;
  return r;
}

FPreds Preds(const smvs_fusion* f) {
  FPreds p;
  p.off = f->d_pred_off;
  p.cnt = f->d_pred_cnt;
  p.list = f->d_pred_list;
  p.used = f->d_pred_used;
  p.cap = f->walk || !f->d_pred_list ? 0ull : std::min<unsigned long long>(f->claim_list_cap, 0xffffffffull);
  p.claim_off = f->d_claim_off;
  p.claim_list = f->d_claim_list;
  return p;
}

// Per-seed arrays for an image of n seeds.
int EnsureSeeds(smvs_fusion* f, uint64_t n, uint64_t nkeys) {
  int st = SMVS_OK;
  if (n > f->seed_cap) {
    Free(f, f->d_rec_off); Free(f, f->d_over_list); Free(f, f->d_seq);
    Free(f, f->d_pred_off); Free(f, f->d_pred_cnt);
    Free(f, f->d_slot_pts); Free(f, f->d_slot_has); Free(f, f->d_slot_nvis); Free(f, f->d_slot_visoff);
    Free(f, f->d_pt_idx); Free(f, f->d_vis_idx);
    f->seed_cap = n;
    if ((st = Alloc(f, &f->d_rec_off, n)) || (st = Alloc(f, &f->d_over_list, n)) || (st = Alloc(f, &f->d_seq, n)) ||
        (st = Alloc(f, &f->d_pred_off, n)) || (st = Alloc(f, &f->d_pred_cnt, n)) || (st = Alloc(f, &f->d_slot_pts, n)) || (st = Alloc(f, &f->d_slot_has, n)) ||
        (st = Alloc(f, &f->d_slot_nvis, n)) || (st = Alloc(f, &f->d_slot_visoff, n)) ||
        (st = Alloc(f, &f->d_pt_idx, n + 1)) || (st = Alloc(f, &f->d_vis_idx, n + 1))) {
      f->seed_cap = 0;
      return st;
    }
  }
  if (nkeys > f->key_cap) {
    Free(f, f->d_keycnt); Free(f, f->d_keyoff);
    f->key_cap = nkeys;
    if ((st = Alloc(f, &f->d_keycnt, nkeys)) || (st = Alloc(f, &f->d_keyoff, nkeys + 1))) {
      f->key_cap = 0;
      return st;
    }
  }
  return SMVS_OK;
}

int ReadStats(smvs_fusion* f, uint32_t stats[3], uint32_t* n_over, unsigned long long* used) {
  FU_CUDA(cudaMemcpyAsync(stats, f->d_stats, 3 * sizeof(uint32_t), cudaMemcpyDeviceToHost, f->stream));
  FU_CUDA(cudaMemcpyAsync(n_over, f->d_n_over, sizeof(uint32_t), cudaMemcpyDeviceToHost, f->stream));
  FU_CUDA(cudaMemcpyAsync(used, f->d_used, sizeof(unsigned long long), cudaMemcpyDeviceToHost, f->stream));
  FU_CUDA(cudaStreamSynchronize(f->stream));
  return SMVS_OK;
}

int FuseImage(smvs_fusion* f, int image) {
  const smvs_fusion_view& v = f->views[image];
  const int W = v.width, H = v.height, T = f->opt.num_slices, step = f->opt.step_size;
  // The seed rows of FuseImage's slices (fusion.cc:1733-1764), in order.
  f->h_rows.clear();
  const int hs = (H + T - 1) / T;
  for (int t = 0; t < T; ++t) {
    const int limit = std::min(hs * (t + 1), H);
    const int row_end = std::min(limit, H - kBlank);
    for (int row = std::max(hs * t, kBlank); row < row_end; row += step) f->h_rows.push_back(row);
  }
  const int Rs = (int)f->h_rows.size();
  const int Cs = W - 2 * kBlank > 0 ? (W - 2 * kBlank + step - 1) / step : 0;
  if (Rs == 0 || Cs == 0) {  // no seed pixel: the image is fused all the same
    FU_CUDA(cudaMemsetAsync(f->d_trav + image, 0, 1, f->stream));
    return SMVS_OK;
  }
  const uint64_t nseeds = (uint64_t)Rs * (uint64_t)Cs;
  const uint64_t nkeys = (uint64_t)Cs * (uint64_t)Rs + (uint64_t)Cs;
  int st = EnsureSeeds(f, nseeds, nkeys);
  if (st) return st;
  if ((size_t)Rs > f->rows_cap) {
    Free(f, f->d_rows);
    f->rows_cap = (size_t)Rs;
    if ((st = Alloc(f, &f->d_rows, (size_t)Rs))) { f->rows_cap = 0; return st; }
  }
  FU_CUDA(cudaMemcpyAsync(f->d_rows, f->h_rows.data(), (size_t)Rs * sizeof(int), cudaMemcpyHostToDevice, f->stream));
  FImage im;
  im.view = image;
  im.cap = f->cap_closure;
  im.Rs = Rs;
  im.Cs = Cs;
  im.step = step;
  im.nseeds = (uint32_t)nseeds;
  im.rows = f->d_rows;
  const FMaps m = Maps(f);
  // 1. Closure records (the pool grows until every record fits).
  uint32_t stats[3] = {0, 0, 0}, n_over = 0;
  unsigned long long used = 0;
  ImageStartKernel<<<1, 1, 0, f->stream>>>(f->d_shear, f->d_ticket, f->d_used, f->d_vis_cursor, f->d_n_over,
                                           f->d_stats);
  ++f->launches;
  {
    ProfScope ps(f, SMVS_FUSION_KERNEL_CLOSURE);
    (f->d_proj ? ClosureKernel<true> : ClosureKernel<false>)<<<f->closure_blocks, 32 * kClosureWarps, kClosureSmem,
                                                              f->stream>>>(m, f->consts, im, Recs(f), 0, f->d_stage);
    ++f->launches;
  }
  FU_CUDA(cudaGetLastError());
  uint32_t big_done = 0;
  for (int attempt = 0;; ++attempt) {
    if ((st = ReadStats(f, stats, &n_over, &used))) return st;
    if (n_over > big_done) {  // seeds over the closure pass's capacity
      if (!f->d_big_scratch && (st = Alloc(f, &f->d_big_scratch, (size_t)kBigBatch * kBigStride))) return st;
      for (uint32_t first = big_done; first < n_over; first += kBigBatch) {
        const uint32_t count = std::min<uint32_t>(kBigBatch, n_over - first);
        ProfScope ps(f, SMVS_FUSION_KERNEL_CLOSURE);
        ClosureBigKernel<<<Blocks(count, 64), 64, 0, f->stream>>>(m, f->consts, im, Recs(f), first, count,
                                                                  f->d_big_scratch);
        ++f->launches;
      }
      FU_CUDA(cudaGetLastError());
      big_done = n_over;
      if ((st = ReadStats(f, stats, &n_over, &used))) return st;
    }
    if (stats[2] & kStBig)
      return Fail(SMVS_EINVAL, "fusion: a seed of image %d reaches more than %d candidate pixels", image, kBigCap);
    if (stats[2] & kStBad) return Fail(SMVS_ECUDA, "fusion: inconsistent cluster record (image %d)", image);
    if (!(stats[2] & kStPool)) break;
    if (attempt >= 8) return Fail(SMVS_ENOMEM, "fusion: record pool cannot grow further");
    // Grow the pool to what this image asked for, plus a margin, keeping the
    // records that fit; only the seeds whose records did not fit run again.
    const size_t old_words = f->pool_words;
    const size_t want = (size_t)std::min<unsigned long long>(used + used / 4 + (1ull << 20), 0xfffffff0ull);
    if (want <= old_words) return Fail(SMVS_ENOMEM, "fusion: record pool limit (16 GB) reached");
    uint32_t* grown = nullptr;
    if ((st = Alloc(f, &grown, want))) return st;
    FU_CUDA(cudaMemcpyAsync(grown, f->d_pool, old_words * sizeof(uint32_t), cudaMemcpyDeviceToDevice, f->stream));
    Free(f, f->d_pool);
    f->d_pool = grown;
    f->pool_words = want;
    const unsigned long long resume = old_words;
    const uint32_t status = stats[2] & ~kStPool;
    FU_CUDA(cudaMemcpyAsync(f->d_used, &resume, sizeof(resume), cudaMemcpyHostToDevice, f->stream));
    FU_CUDA(cudaMemcpyAsync(f->d_stats + 2, &status, sizeof(status), cudaMemcpyHostToDevice, f->stream));
    {
      ProfScope ps(f, SMVS_FUSION_KERNEL_CLOSURE);
      (f->d_proj ? ClosureKernel<true> : ClosureKernel<false>)<<<f->closure_blocks, 32 * kClosureWarps, kClosureSmem,
                                                              f->stream>>>(m, f->consts, im, Recs(f), 1, f->d_stage);
      ++f->launches;
    }
    FU_CUDA(cudaGetLastError());
  }
  const uint32_t max_cnt = stats[0], max_ne = stats[1];
  // 2. Claims and predecessors.
  {
    ProfScope ps(f, SMVS_FUSION_KERNEL_ORDER);
    const uint64_t claims = used / 3 + 1;  // a record of cnt pixels takes more than 3 cnt words
    if (claims > f->claim_list_cap) {
      Free(f, f->d_claim_list);
      Free(f, f->d_pred_list);
      f->claim_list_cap = (size_t)claims + 1024;
      if ((st = Alloc(f, &f->d_claim_list, f->claim_list_cap))) { f->claim_list_cap = 0; return st; }
      // Without room for the predecessor lists the replay walks the claims.
      if (Alloc(f, &f->d_pred_list, f->claim_list_cap)) (void)cudaGetLastError();
    }
    ClaimCountKernel<<<Blocks(32 * nseeds, 256), 256, 0, f->stream>>>(Recs(f), (uint32_t)nseeds, f->d_claim_cnt);
    ++f->launches;
    if ((st = Scan(f, f->d_claim_cnt, f->total, f->d_claim_off))) return st;
    ClaimFillKernel<<<Blocks(32 * nseeds, 256), 256, 0, f->stream>>>(Recs(f), (uint32_t)nseeds, f->d_claim_cnt,
                                                                 f->d_claim_off, f->d_claim_list);
    FU_CUDA(cudaMemsetAsync(f->d_pred_used, 0, sizeof(unsigned long long), f->stream));
    PredKernel<<<Blocks(32 * nseeds, 256), 256, 0, f->stream>>>(m, im, Recs(f), Preds(f), f->d_shear);
    // 3. Ticket order.
    KeyCountKernel<<<Blocks(nkeys, 256), 256, 0, f->stream>>>((uint32_t)nkeys, Rs, Cs, f->d_shear, f->d_keycnt);
    f->launches += 3;
    if ((st = Scan(f, f->d_keycnt, nkeys, f->d_keyoff))) return st;
    SeqKernel<<<Blocks(nseeds, 256), 256, 0, f->stream>>>((uint32_t)nseeds, Cs, f->d_shear, f->d_keyoff, f->d_seq);
    ++f->launches;
    FU_CUDA(cudaGetLastError());
  }
  // 4. Replay.
  if (max_cnt > (uint32_t)f->cap_replay || max_ne + 1 > (uint32_t)f->cap_stack) {
    const uint32_t cap_cnt = std::max<uint32_t>(max_cnt, 1), cap_stack = max_ne + 1;
    const size_t per = ScratchPer(cap_cnt, cap_stack);
    const size_t need = per * (size_t)f->replay_blocks * kReplayWarps;
    if (need > f->replay_scratch_bytes || cap_cnt > f->replay_scratch_cnt || cap_stack > f->replay_scratch_stack) {
      Free(f, f->d_replay_scratch);
      f->replay_scratch_bytes = need;
      if ((st = Alloc(f, &f->d_replay_scratch, need))) { f->replay_scratch_bytes = 0; return st; }
    }
    f->replay_scratch_cnt = cap_cnt;
    f->replay_scratch_stack = cap_stack;
  }
  FU_CUDA(cudaMemsetAsync(f->d_slot_has, 0, nseeds * sizeof(uint32_t), f->stream));
  FU_CUDA(cudaMemsetAsync(f->d_slot_nvis, 0, nseeds * sizeof(uint32_t), f->stream));
  {
    FReplay rp;
    rp.seq = f->d_seq;
    rp.nseeds = (uint32_t)nseeds;
    rp.im = im;
    rp.preds = Preds(f);
    rp.ticket = f->d_ticket;
    rp.slot_pts = f->d_slot_pts;
    rp.slot_has = f->d_slot_has;
    rp.slot_nvis = f->d_slot_nvis;
    rp.slot_visoff = f->d_slot_visoff;
    rp.vis_pool = f->d_vis_pool;
    rp.vis_cursor = f->d_vis_cursor;
    rp.scratch = f->d_replay_scratch;
    rp.scratch_cnt = f->d_replay_scratch ? f->replay_scratch_cnt : 0;
    rp.scratch_stack = f->d_replay_scratch ? f->replay_scratch_stack : 0;
    rp.shared_cnt = f->cap_replay;
    rp.shared_stack = f->cap_stack;
    rp.level = nullptr;
    rp.chain = nullptr;
    rp.times = nullptr;
    rp.wait_limit_ns = t_wait_limit_ns ? t_wait_limit_ns : kWaitLimitNs;
    rp.withhold = t_withhold;
    if (f->profiling) {
      const size_t plane = (size_t)W * (size_t)H;
      if (plane > f->level_cap) {
        Free(f, f->d_level);
        f->level_cap = plane;
        if ((st = Alloc(f, &f->d_level, plane))) { f->level_cap = 0; return st; }
      }
      FU_CUDA(cudaMemsetAsync(f->d_level, 0, plane * sizeof(uint32_t), f->stream));
      if (!f->d_chain && (st = Alloc(f, &f->d_chain, 2 * (size_t)f->num_views))) return st;
      const int k = (int)f->order.size();
      FU_CUDA(cudaMemsetAsync(f->d_chain + k, 0, sizeof(uint32_t), f->stream));
      FU_CUDA(cudaMemcpyAsync(f->d_chain + f->num_views + k, f->d_shear, sizeof(uint32_t),
                              cudaMemcpyDeviceToDevice, f->stream));
      rp.level = f->d_level;
      rp.chain = f->d_chain + k;
      if (!f->d_times && (st = Alloc(f, &f->d_times, 9 * (size_t)f->num_views))) return st;
      FU_CUDA(cudaMemsetAsync(f->d_times + 9 * k, 0, 9 * sizeof(unsigned long long), f->stream));
      rp.times = f->d_times + 9 * k;
    }
    ProfScope ps(f, SMVS_FUSION_KERNEL_REPLAY);
    ReplayKernel<<<f->replay_blocks, 32 * kReplayWarps, 0, f->stream>>>(m, f->consts, Recs(f), rp);
    ++f->launches;
    FU_CUDA(cudaGetLastError());
  }
  // 5. Compaction in seed order.
  {
    ProfScope ps(f, SMVS_FUSION_KERNEL_OTHER);
    if ((st = Scan(f, f->d_slot_has, nseeds, f->d_pt_idx))) return st;
    if ((st = Scan(f, f->d_slot_nvis, nseeds, f->d_vis_idx))) return st;
    CompactKernel<<<Blocks(nseeds, 256), 256, 0, f->stream>>>(
        (uint32_t)nseeds, f->d_slot_has, f->d_pt_idx, f->d_vis_idx, f->d_slot_pts, f->d_slot_nvis,
        f->d_slot_visoff, f->d_vis_pool, f->d_totals, f->d_out_pts, f->d_out_visoff, f->d_out_vis);
    AdvanceKernel<<<1, 1, 0, f->stream>>>(f->d_totals, f->d_pt_idx, f->d_vis_idx, (uint32_t)nseeds,
                                          f->d_out_visoff);
    f->launches += 2;
    FU_CUDA(cudaGetLastError());
  }
  // The image is fused: no later traversal enters it.
  FU_CUDA(cudaMemsetAsync(f->d_trav + image, 0, 1, f->stream));
  return SMVS_OK;
}

thread_local int t_cap_closure = 0, t_cap_replay = 0, t_cap_stack = 0;

int CheckStatus(smvs_fusion* f) {
  uint32_t stats[3];
  FU_CUDA(cudaMemcpyAsync(stats, f->d_stats, sizeof(stats), cudaMemcpyDeviceToHost, f->stream));
  FU_CUDA(cudaStreamSynchronize(f->stream));
  if (stats[2] & kStTimeout) return Fail(SMVS_ETIMEDOUT, "fusion: a replay wait gave up (predecessor never released)");
  if (stats[2] & kStBad) return Fail(SMVS_ECUDA, "fusion: inconsistent replay state");
  return SMVS_OK;
}

// ---- clean-up passes after the image loop ----------------------------------
// The passes work on the cloud where it lies. Their scratch is what the image loop
// has left: the pixel records (32 bytes a pixel), the claims and the visibility
// pool are not read after it, and Run may be called once.
struct Carve {
  smvs_fusion* f;
  char* at;
  size_t left;
  void* own[16] = {};
  int nown = 0;
  explicit Carve(smvs_fusion* fusion)
      : f(fusion), at(reinterpret_cast<char*>(fusion->d_pix)), left(32 * (size_t)fusion->total) {}
  ~Carve() {
    for (int k = 0; k < nown; ++k) cudaFreeAsync(own[k], f->stream);
  }
  template <typename T>
  int Take(T** p, size_t count) {
    const size_t bytes = (std::max<size_t>(count * sizeof(T), 1) + 255) / 256 * 256;
    if (bytes <= left) {
      *p = reinterpret_cast<T*>(at);
      at += bytes;
      left -= bytes;
      return SMVS_OK;
    }
    if (nown == (int)(sizeof(own) / sizeof(own[0]))) return Fail(SMVS_ENOMEM, "fusion: too many scratch arrays");
    const int st = Alloc(f, p, count);
    if (!st) own[nown++] = *p;
    return st;
  }
};

// Per point: its number of images where it is kept, else 0.
__global__ void KeptCountKernel(uint32_t n, const uint64_t* __restrict__ off, const uint32_t* __restrict__ keep,
                                uint32_t* __restrict__ nvis) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) nvis[i] = keep[i] ? (uint32_t)(off[i + 1] - off[i]) : 0u;
}

__global__ void KeepKernel(uint32_t n, const uint32_t* __restrict__ keep, const uint32_t* __restrict__ pt_idx,
                           const uint32_t* __restrict__ vis_idx, const smvs_fused_point* __restrict__ pts,
                           const uint64_t* __restrict__ off, const uint32_t* __restrict__ vis,
                           smvs_fused_point* __restrict__ new_pts, uint64_t* __restrict__ new_off,
                           uint32_t* __restrict__ new_vis) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i > n) return;
  const uint32_t j = pt_idx[i], v = vis_idx[i];
  if (i == n) {
    new_off[j] = v;
    return;
  }
  if (!keep[i]) return;
  new_pts[j] = pts[i];
  new_off[j] = v;
  const uint64_t b = off[i];
  const uint32_t cnt = (uint32_t)(off[i + 1] - b);
  for (uint32_t k = 0; k < cnt; ++k) new_vis[v + k] = vis[b + k];
}

// What Compact needs. Taken before a pass changes the cloud: a pass that runs out
// of memory leaves it as it was.
struct CompactScratch {
  uint32_t *nvis, *pt_idx, *vis_idx;
  smvs_fused_point* new_pts;
  uint64_t* new_off;
  int Take(smvs_fusion* f, Carve& scratch) {
    const size_t n = f->num_points;
    int st;
    if ((st = scratch.Take(&nvis, n)) || (st = scratch.Take(&pt_idx, n + 1)) || (st = scratch.Take(&vis_idx, n + 1)) ||
        (st = scratch.Take(&new_pts, n)) || (st = scratch.Take(&new_off, n + 1)))
      return st;
    return EnsureScanSums(f, n);
  }
};

// Keeps the points with keep[i] (1 or 0; order preserved, as the reference's
// in-place compaction loops do). The device arrays stay where they are and only shrink.
int Compact(smvs_fusion* f, const CompactScratch& c, const uint32_t* keep, size_t* removed) {
  const uint32_t n = (uint32_t)f->num_points;
  uint32_t *nvis = c.nvis, *pt_idx = c.pt_idx, *vis_idx = c.vis_idx, *new_vis = f->d_claim_cnt;
  smvs_fused_point* new_pts = c.new_pts;
  uint64_t* new_off = c.new_off;
  int st;
  const int blocks = Blocks((size_t)n + 1, 256);
  KeptCountKernel<<<blocks, 256, 0, f->stream>>>(n, f->d_out_visoff, keep, nvis);
  if ((st = Scan(f, keep, n, pt_idx)) || (st = Scan(f, nvis, n, vis_idx))) return st;
  KeepKernel<<<blocks, 256, 0, f->stream>>>(n, keep, pt_idx, vis_idx, f->d_out_pts, f->d_out_visoff, f->d_out_vis,
                                            new_pts, new_off, new_vis);
  f->launches += 2;
  FU_CUDA(cudaGetLastError());
  uint32_t j = 0, v = 0;
  FU_CUDA(cudaMemcpyAsync(&j, pt_idx + n, 4, cudaMemcpyDeviceToHost, f->stream));
  FU_CUDA(cudaMemcpyAsync(&v, vis_idx + n, 4, cudaMemcpyDeviceToHost, f->stream));
  FU_CUDA(cudaStreamSynchronize(f->stream));
  if (j) FU_CUDA(cudaMemcpyAsync(f->d_out_pts, new_pts, j * sizeof(smvs_fused_point), cudaMemcpyDeviceToDevice,
                                 f->stream));
  FU_CUDA(cudaMemcpyAsync(f->d_out_visoff, new_off, ((size_t)j + 1) * 8, cudaMemcpyDeviceToDevice, f->stream));
  if (v) FU_CUDA(cudaMemcpyAsync(f->d_out_vis, new_vis, (size_t)v * 4, cudaMemcpyDeviceToDevice, f->stream));
  FU_CUDA(cudaStreamSynchronize(f->stream));
  if (removed) *removed = n - j;
  f->num_points = j;
  f->num_vis = v;
  return SMVS_OK;
}

// RemoveDuplicatePoints (fusion.cc:2184-2266): points in fusion order claim the
// pixel they project to in each of their images; a point meeting an occupant seen
// by more images is dropped (and looks no further), otherwise it takes the pixel
// and the occupant is dropped. The occupants of a pixel are seen by ever more (or as
// many) images, so point i is stopped at a pixel exactly if an earlier point seen by
// more images took it, and is dropped there exactly if a later point took it too.
// Points of one number of images do not stop one another: from the largest number
// down, each level is two launches over its points (where is each stopped; the
// pixels before that are taken), then one over all points finds the dropped ones. A
// walk on the host took 7 ms for 66,000 points of 6 views 640x480 (and the cloud's
// way there and back), now 0.2 ms; 470,000 of 11 views 1600x1200 110 ms, now 0.5 ms.
struct DupView {
  float K[9], R[9], T[3];
  int W, H;
  uint32_t base;
};
constexpr uint32_t kNoCell = 0xffffffffu;
constexpr int kDupBins = 1024;  // numbers of images counted in shared memory

__global__ void __launch_bounds__(256) DupLevelsKernel(uint32_t n, const uint64_t* __restrict__ off, int max_level,
                                                       uint32_t* __restrict__ counts) {
  __shared__ uint32_t bins[kDupBins];
  for (int k = threadIdx.x; k < kDupBins; k += 256) bins[k] = 0;
  __syncthreads();
  for (uint32_t i = blockIdx.x * 256 + threadIdx.x; i < n; i += gridDim.x * 256) {
    const int level = (int)min(off[i + 1] - off[i], (uint64_t)max_level);
    atomicAdd(level < kDupBins ? bins + level : counts + level, 1u);
  }
  __syncthreads();
  for (int k = threadIdx.x; k < min(kDupBins, max_level + 1); k += 256)
    if (bins[k]) atomicAdd(counts + k, bins[k]);
}

// Lists the points by level: cursor[level] starts at the level's first place. All
// lanes of a warp match; those past the end share a level that no point has.
__global__ void DupOrderKernel(uint32_t n, const uint64_t* __restrict__ off, int max_level,
                               uint32_t* __restrict__ cursor, uint32_t* __restrict__ list) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  const int level = i < n ? (int)min(off[i + 1] - off[i], (uint64_t)max_level) : -1;
  const unsigned same = __match_any_sync(0xffffffffu, level);
  const int lane = threadIdx.x % 32, leader = __ffs(same) - 1;
  uint32_t first = 0;
  if (i < n && lane == leader) first = atomicAdd(cursor + level, (uint32_t)__popc(same));
  first = __shfl_sync(0xffffffffu, first, leader);
  if (i < n) list[first + __popc(same & ((1u << lane) - 1))] = i;
}

// Eigen 3.3's float evaluation of K * (R * X + T) (coefficient-based 3x3 products
// reduce as (p0 + p1) + p2), then proj / z rounded half away from zero (std::round),
// as RemoveDuplicatePoints projects (fusion.cc:2216-2219); kNoCell outside the image
// and where an int cannot hold the result.
__device__ __forceinline__ uint32_t DupCell(const DupView& v, const smvs_fused_point& p) {
  float c[3], q[3];
  for (int r = 0; r < 3; ++r) c[r] = ((v.R[3 * r] * p.x + v.R[3 * r + 1] * p.y) + v.R[3 * r + 2] * p.z) + v.T[r];
  for (int r = 0; r < 3; ++r) q[r] = (v.K[3 * r] * c[0] + v.K[3 * r + 1] * c[1]) + v.K[3 * r + 2] * c[2];
  const float u = roundf(q[0] / q[2]), w = roundf(q[1] / q[2]);
  if (!(u >= 0.0f && u < (float)v.W && w >= 0.0f && w < (float)v.H)) return kNoCell;
  const int iu = (int)u, iw = (int)w;
  if (iu >= v.W || iw >= v.H) return kNoCell;  // sizes that a float rounds up
  return v.base + (uint32_t)iw * (uint32_t)v.W + (uint32_t)iu;
}

// earliest[cell]: the first point of a higher level that took the cell.
__global__ void DupStopKernel(const uint32_t* __restrict__ list, uint32_t count,
                              const smvs_fused_point* __restrict__ pts, const uint64_t* __restrict__ off,
                              const uint32_t* __restrict__ vis, const DupView* __restrict__ views,
                              const uint32_t* __restrict__ earliest, uint32_t* __restrict__ cells,
                              uint32_t* __restrict__ keep) {
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= count) return;
  const uint32_t i = list[t];
  const smvs_fused_point p = pts[i];
  bool stopped = false;
  for (uint64_t k = off[i]; k < off[i + 1]; ++k) {
    uint32_t cell = stopped ? kNoCell : DupCell(views[vis[k]], p);
    if (cell != kNoCell && earliest[cell] < i) {
      stopped = true;
      cell = kNoCell;
    }
    cells[k] = cell;
  }
  keep[i] = !stopped;
}

__global__ void DupTakeKernel(const uint32_t* __restrict__ list, uint32_t count, const uint64_t* __restrict__ off,
                              const uint32_t* __restrict__ cells, uint32_t* __restrict__ earliest,
                              uint32_t* __restrict__ latest) {
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= count) return;
  const uint32_t i = list[t];
  for (uint64_t k = off[i]; k < off[i + 1]; ++k) {
    const uint32_t cell = cells[k];
    if (cell == kNoCell) continue;
    atomicMin(earliest + cell, i);
    atomicMax(latest + cell, i);
  }
}

__global__ void DupDropKernel(uint32_t n, const uint64_t* __restrict__ off, const uint32_t* __restrict__ cells,
                              const uint32_t* __restrict__ latest, uint32_t* __restrict__ keep) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  bool dropped = false;
  for (uint64_t k = off[i]; k < off[i + 1] && !dropped; ++k) dropped = cells[k] != kNoCell && latest[cells[k]] > i;
  if (dropped) keep[i] = 0;
}

// ---- outliers ---------------------------------------------------------------
// Order-preserving map float -> uint32, for minima and maxima.
__host__ __device__ __forceinline__ uint32_t FloatKey(float f) {
  uint32_t b;
  memcpy(&b, &f, 4);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__host__ __device__ __forceinline__ float KeyFloat(uint32_t k) {
  const uint32_t b = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
  float f;
  memcpy(&f, &b, 4);
  return f;
}

// The numbers that the outlier pass gathers over the cloud: keys of the smallest
// (even) and largest (odd) x, y, z and score, and the score histogram. A NaN takes
// no part in a minimum or maximum (std::min and std::max with it second).
struct CloudStats {
  uint32_t range[8];
  uint32_t bins[256];
};

__global__ void StatsResetKernel(CloudStats* __restrict__ s) {
  const int t = threadIdx.x;
  if (t < 8) s->range[t] = t & 1 ? 0u : 0xffffffffu;
  s->bins[t] = 0;
}

__device__ __forceinline__ void FoldKeys(const uint32_t (&key)[8], int first, int last, CloudStats* s) {
  for (int k = first; k < last; ++k) {
    const uint32_t v = k & 1 ? __reduce_max_sync(0xffffffffu, key[k]) : __reduce_min_sync(0xffffffffu, key[k]);
    if (threadIdx.x % 32 != 0) continue;
    if (k & 1) atomicMax(s->range + k, v);
    else atomicMin(s->range + k, v);
  }
}

__global__ void __launch_bounds__(256) CloudBoxKernel(const smvs_fused_point* __restrict__ pts, uint32_t n,
                                                      CloudStats* __restrict__ s) {
  uint32_t key[8] = {0xffffffffu, 0u, 0xffffffffu, 0u, 0xffffffffu, 0u, 0xffffffffu, 0u};
  for (uint32_t i = blockIdx.x * 256 + threadIdx.x; i < n; i += gridDim.x * 256) {
    const float x[3] = {pts[i].x, pts[i].y, pts[i].z};
    for (int a = 0; a < 3; ++a)
      if (!isnan(x[a])) {
        key[2 * a] = min(key[2 * a], FloatKey(x[a]));
        key[2 * a + 1] = max(key[2 * a + 1], FloatKey(x[a]));
      }
  }
  FoldKeys(key, 0, 6, s);
}

// Blends each score with its spacing ratio (fusion.cc:2542-2611) and finds the range.
__global__ void __launch_bounds__(256) ScoreKernel(smvs_fused_point* __restrict__ pts, uint32_t n,
                                                   const float* __restrict__ spacing, int blend, double unit,
                                                   CloudStats* __restrict__ s) {
  uint32_t key[8] = {0xffffffffu, 0u, 0xffffffffu, 0u, 0xffffffffu, 0u, 0xffffffffu, 0u};
  for (uint32_t i = blockIdx.x * 256 + threadIdx.x; i < n; i += gridDim.x * 256) {
    float score = pts[i].score;
    if (blend) {
      const float factor = (float)((double)spacing[i] / unit);
      score = (float)((double)score * 0.6 + (double)factor * 0.4);
      pts[i].score = score;
    }
    if (!isnan(score)) {
      key[6] = min(key[6], FloatKey(score));
      key[7] = max(key[7], FloatKey(score));
    }
  }
  FoldKeys(key, 6, 8, s);
}

// One score for every point (range 0) puts all points in bin 0: none is dropped
// (the reference divides 0 by 0 there).
__device__ __forceinline__ int ScoreBin(float score, float smin, float range) {
  if (!(range > 0)) return 0;
  const float gray = (score - smin) / range;
  return min(max((int)(gray * 255), 0), 255);
}

__global__ void __launch_bounds__(256) HistKernel(const smvs_fused_point* __restrict__ pts, uint32_t n,
                                                  CloudStats* __restrict__ s) {
  __shared__ uint32_t bins[256];
  bins[threadIdx.x] = 0;
  __syncthreads();
  const float smin = KeyFloat(s->range[6]), range = KeyFloat(s->range[7]) - smin;
  for (uint32_t i = blockIdx.x * 256 + threadIdx.x; i < n; i += gridDim.x * 256)
    atomicAdd(bins + ScoreBin(pts[i].score, smin, range), 1u);
  __syncthreads();
  if (bins[threadIdx.x]) atomicAdd(s->bins + threadIdx.x, bins[threadIdx.x]);
}

struct BinMask {
  uint32_t drop[8];  // a bit per bin
};

__global__ void BinKeepKernel(const smvs_fused_point* __restrict__ pts, uint32_t n, const CloudStats* __restrict__ s,
                              BinMask mask, uint32_t* __restrict__ keep) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float smin = KeyFloat(s->range[6]), range = KeyFloat(s->range[7]) - smin;
  const int b = ScoreBin(pts[i].score, smin, range);
  keep[i] = !((mask.drop[b / 32] >> (b % 32)) & 1u);
}

// Exact k-nearest-neighbour spacing on a uniform grid. Points are bucketed by cell
// (counting sort, positions copied into cell order); a query scans the cube of
// half-width r cells around its own cell, keeping the K smallest squared distances
// (double, the coordinate differences squared and summed x, y, z as CGAL's Euclidean
// distance does), and doubles r until the K-th lies within r cell widths (every
// point nearer than that is inside the cube) or the cube covers the grid. A margin
// of 1e-7 covers the rounding of the cell assignment.
constexpr int kMaxKnn = 64;
constexpr double kKnnMargin = 1.0 - 1e-7;

struct KnnGrid {
  double minx, miny, minz, h, inv_h;
  int gx, gy, gz;
};

__device__ __forceinline__ int CellCoord(double v, double lo, double inv_h, int g) {
  int c = (int)floor((v - lo) * inv_h);
  return c < 0 ? 0 : (c >= g ? g - 1 : c);
}

__global__ void KnnCountKernel(const smvs_fused_point* __restrict__ pts, uint32_t n, KnnGrid g,
                               uint32_t* __restrict__ cell_of, uint32_t* __restrict__ counts) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int cx = CellCoord((double)pts[i].x, g.minx, g.inv_h, g.gx);
  const int cy = CellCoord((double)pts[i].y, g.miny, g.inv_h, g.gy);
  const int cz = CellCoord((double)pts[i].z, g.minz, g.inv_h, g.gz);
  const uint32_t cell = ((uint32_t)cz * g.gy + (uint32_t)cy) * g.gx + (uint32_t)cx;
  cell_of[i] = cell;
  atomicAdd(counts + cell, 1u);
}

// sorted: position and (in w) index of the points, by cell; uses the counts up.
__global__ void KnnScatterKernel(const smvs_fused_point* __restrict__ pts, uint32_t n,
                                 const uint32_t* __restrict__ cell_of, const uint32_t* __restrict__ start,
                                 uint32_t* __restrict__ counts, float4* __restrict__ sorted) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t c = cell_of[i];
  sorted[start[c] + atomicSub(counts + c, 1u) - 1u] = make_float4(pts[i].x, pts[i].y, pts[i].z, __uint_as_float(i));
}

// The kReg smallest distances met, in order.
template <int kReg>
struct Nearest {
  double best[kReg];
  __device__ __forceinline__ void Reset() {
#pragma unroll
    for (int k = 0; k < kReg; ++k) best[k] = INFINITY;
  }
  __device__ __forceinline__ void Add(double d, int K) {
    if constexpr (kReg <= 16) {  // in registers
      if (!(d < best[kReg - 1])) return;
#pragma unroll
      for (int k = kReg - 1; k > 0; --k) best[k] = d < best[k - 1] ? best[k - 1] : (d < best[k] ? d : best[k]);
      best[0] = d < best[0] ? d : best[0];
    } else {
      if (!(d < best[K - 1])) return;
      int m = K - 1;
      while (m > 0 && best[m - 1] > d) { best[m] = best[m - 1]; --m; }
      best[m] = d;
    }
  }
  __device__ __forceinline__ double At(int j) const {
    if constexpr (kReg <= 16) {
      double v = best[0];
#pragma unroll
      for (int k = 1; k < kReg; ++k) v = k == j ? best[k] : v;
      return v;
    } else {
      return best[j];
    }
  }
};

// ComputeAverageDistance's per-point spacing (patch_match_controller.cc:160-181):
// the mean distance of the query's K = nb_neighbors + 1 nearest points (itself
// included, at distance 0) over K - 1, accumulated nearest first in float with
// each distance added in double. Queries go in cell order, so a warp reads the same
// cells; a cube's cells of one row (along x) are one range of `sorted`; rows that
// lie further than the K-th distance are passed over. Up to 16 distances stay in
// registers. 65,000 points, K = 7: the whole pass takes 0.48 ms (0.69 ms
// with a cell per point), with queries in point order, cells read one by one and the
// points through an index 1.65 ms; 470,000 points 1.34 ms (1 cell a point 2.19, 27
// 1.12). On the host's side of it the cloud went both ways: 3.95 and 24.2 ms.
template <int kReg>
__global__ void __launch_bounds__(128) KnnSpacingKernel(const float4* __restrict__ sorted, uint32_t n, KnnGrid g,
                                                        const uint32_t* __restrict__ start, int K,
                                                        float* __restrict__ spacing) {
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const float4 q = __ldg(sorted + t);
  const uint32_t i = __float_as_uint(q.w);
  const double qx = q.x, qy = q.y, qz = q.z;
  if (isnan(q.x) || isnan(q.y) || isnan(q.z)) {
    spacing[i] = NAN;
    return;
  }
  const int cx = CellCoord(qx, g.minx, g.inv_h, g.gx);
  const int cy = CellCoord(qy, g.miny, g.inv_h, g.gy);
  const int cz = CellCoord(qz, g.minz, g.inv_h, g.gz);
  Nearest<kReg> near;
  for (int r = 1;; r = r < (1 << 28) ? 2 * r : r) {
    near.Reset();
    const int x0 = max(cx - r, 0), x1 = min(cx + r, g.gx - 1), y0 = max(cy - r, 0), y1 = min(cy + r, g.gy - 1),
              z0 = max(cz - r, 0), z1 = min(cz + r, g.gz - 1);
    double kth = INFINITY;
    for (int z = z0; z <= z1; ++z) {
      const double dz = (double)max(abs(z - cz) - 1, 0) * (g.h * kKnnMargin);
      if (dz * dz > kth) continue;
      for (int y = y0; y <= y1; ++y) {
        const double dy = (double)max(abs(y - cy) - 1, 0) * (g.h * kKnnMargin);
        if (dz * dz + dy * dy > kth) continue;
        const uint32_t row = ((uint32_t)z * g.gy + (uint32_t)y) * g.gx;
        const uint32_t end = __ldg(start + row + x1 + 1);
        for (uint32_t k = __ldg(start + row + x0); k < end; ++k) {
          const float4 p = __ldg(sorted + k);
          const double dx = qx - (double)p.x, ey = qy - (double)p.y, ez = qz - (double)p.z;
          double d = dx * dx;
          d += ey * ey;
          d += ez * ez;
          near.Add(d, K);
        }
        kth = near.At(K - 1);
      }
    }
    const double reach = (double)r * (g.h * kKnnMargin);
    if (kth <= reach * reach || (x1 - x0 + 1 == g.gx && y1 - y0 + 1 == g.gy && z1 - z0 + 1 == g.gz)) break;
  }
  float s = 0.0f;
  int cnt = 0;
  for (int k = 0; k < K; ++k) {
    const double d = near.At(k);
    if (d == INFINITY) break;
    s = (float)((double)s + sqrt(d));
    ++cnt;
  }
  if (cnt > 1) s /= (float)(cnt - 1);
  spacing[i] = s;
}

}  // namespace

extern "C" {

int smvs_fusion_options_default(smvs_fusion_options* o) {
  if (!o) return Fail(SMVS_EINVAL, "null options");
  o->step_size = 1;
  o->min_num_pixels = 5;
  o->max_num_pixels = 10000;
  o->min_num_visible_images = 3;
  o->max_traversal_depth = 100;
  o->max_reproj_error = 2.0;
  o->max_depth_error = (double)0.01f;
  o->max_normal_error = 10.0;
  o->with_normal = 1;
  o->num_slices = 1;
  o->gpu_index = 0;
  return SMVS_OK;
}

int smvs_fusion_create(const smvs_fusion_options* opt, const smvs_fusion_view* views, int num_views,
                       const int32_t* overlap_offsets, const int32_t* overlap_images, int memory, void* stream,
                       smvs_fusion** out) {
  if (!opt || !views || num_views < 1 || !overlap_offsets || !out)
    return Fail(SMVS_EINVAL, "fusion: null argument or no images");
  *out = nullptr;
  if (memory != SMVS_MEM_HOST && memory != SMVS_MEM_DEVICE) return Fail(SMVS_EINVAL, "fusion: bad memory kind");
  if (opt->step_size < 1 || opt->min_num_pixels < 2 || opt->max_num_pixels < opt->min_num_pixels ||
      opt->max_traversal_depth < 1 || opt->min_num_visible_images < 0 || opt->num_slices < 1 ||
      !(opt->max_reproj_error >= 0) || !(opt->max_depth_error >= 0) || !(opt->max_normal_error >= 0))
    return Fail(SMVS_EINVAL, "fusion: bad options (min_num_pixels >= 2, max_num_pixels >= min_num_pixels, "
                             "max_traversal_depth > 0, step_size > 0, num_slices > 0, errors >= 0)");
  if (num_views > 65535) return Fail(SMVS_EINVAL, "fusion: more than 65535 images");
  if (overlap_offsets[0] != 0) return Fail(SMVS_EINVAL, "fusion: overlap_offsets[0] must be 0");
  for (int v = 0; v < num_views; ++v) {
    if (overlap_offsets[v + 1] < overlap_offsets[v]) return Fail(SMVS_EINVAL, "fusion: decreasing overlap offsets");
    for (int32_t k = overlap_offsets[v]; k < overlap_offsets[v + 1]; ++k)
      if (!overlap_images || overlap_images[k] < 0 || overlap_images[k] >= num_views)
        return Fail(SMVS_EINVAL, "fusion: overlapping image index out of range");
  }
  uint64_t total = 0;
  for (int v = 0; v < num_views; ++v) {
    const smvs_fusion_view& fv = views[v];
    if (!fv.depth) continue;
    if (fv.width < 1 || fv.height < 1) return Fail(SMVS_EINVAL, "fusion: image %d has no size", v);
    if (opt->with_normal && !fv.normal) return Fail(SMVS_EINVAL, "fusion: image %d has no normal map", v);
    total += (uint64_t)fv.width * (uint64_t)fv.height;
  }
  if (total >= (1ull << 31)) return Fail(SMVS_EINVAL, "fusion: 2^31 pixels or more");
  smvs_fusion* f = new (std::nothrow) smvs_fusion();
  if (!f) return Fail(SMVS_ENOMEM, "fusion: out of host memory");
  f->opt = *opt;
  f->num_views = num_views;
  f->views.assign(views, views + num_views);
  f->ov_off.assign(overlap_offsets, overlap_offsets + num_views + 1);
  f->ov_img.assign(overlap_images ? overlap_images : overlap_offsets,
                   (overlap_images ? overlap_images : overlap_offsets) + overlap_offsets[num_views]);
  f->used.assign(num_views, 0);
  f->fused.assign(num_views, 0);
  f->total = std::max<uint64_t>(total, 1);
  f->device = opt->gpu_index;
  if (t_cap_closure > 0) f->cap_closure = std::min(t_cap_closure, kCap);
  if (t_cap_replay > 0) f->cap_replay = std::min(t_cap_replay, kCap);
  if (t_cap_stack > 0) f->cap_stack = std::min(t_cap_stack, kStackSh);
  auto fail = [&](int st) {
    FreeAll(f);
    delete f;
    return st;
  };
  if (cudaSetDevice(f->device) != cudaSuccess) return fail(Fail(SMVS_ECUDA, "fusion: cannot use GPU %d", f->device));
  if (stream) {
    f->stream = (cudaStream_t)stream;
  } else {
    if (cudaStreamCreateWithFlags(&f->stream, cudaStreamNonBlocking) != cudaSuccess)
      return fail(Fail(SMVS_ECUDA, "fusion: cannot create a stream"));
    f->own_stream = true;
  }
  f->pool = smvs_internal_device_pool(f->device);
  if (!f->pool) return fail(Fail(SMVS_ECUDA, "fusion: no device memory pool"));
  // Constants (StereoFusion's constructor, fusion.cc:648-663).
  FConsts& c = f->consts;
  c.max_sq_reproj = (float)(opt->max_reproj_error * opt->max_reproj_error);
  c.min_cos = (float)std::cos(opt->max_normal_error * 0.0174532925199432954743716805978692718781530857086181640625);
  float thr = (float)opt->max_depth_error;
  if ((double)thr > opt->max_depth_error) thr = std::nextafter(thr, -INFINITY);
  c.derr_thr = thr;
  c.max_depth_error = opt->max_depth_error;
  c.with_normal = opt->with_normal ? 1 : 0;
  c.min_pix = opt->min_num_pixels;
  c.max_pix = opt->max_num_pixels;
  c.max_depth = opt->max_traversal_depth;
  c.min_vis = opt->min_num_visible_images;
  // Image table.
  f->h_views.resize(num_views);
  uint64_t base = 0;
  for (int v = 0; v < num_views; ++v) {
    FView& hv = f->h_views[v];
    memset(&hv, 0, sizeof(hv));
    ComposeP(views[v].K, views[v].R, views[v].T, hv.P);
    ComposeInvP(hv.P, hv.iP);
    hv.W = views[v].width;
    hv.H = views[v].height;
    hv.base = (uint32_t)base;
    hv.ov_begin = overlap_offsets[v];
    hv.ov_end = overlap_offsets[v + 1];
    f->used[v] = views[v].depth != nullptr;
    if (f->used[v]) base += (uint64_t)hv.W * (uint64_t)hv.H;
    else hv.W = hv.H = 0;
  }
  int st;
  const size_t T = (size_t)f->total;
  const size_t nov = std::max<size_t>((size_t)overlap_offsets[num_views], 1);
  if ((st = Alloc(f, &f->d_views, (size_t)num_views)) || (st = Alloc(f, &f->d_ov, nov)) ||
      (st = Alloc(f, &f->d_trav, (size_t)num_views)) || (st = Alloc(f, &f->d_pix, 2 * T)) ||
      (st = Alloc(f, &f->d_rgb, 3 * T)) || (st = Alloc(f, &f->d_mask, T)) || (st = Alloc(f, &f->d_claim_cnt, T)) ||
      (st = Alloc(f, &f->d_claim_off, T + 1)) || (st = Alloc(f, &f->d_vis_pool, T)) ||
      (st = Alloc(f, &f->d_out_pts, T / 2 + 1)) || (st = Alloc(f, &f->d_out_visoff, T / 2 + 2)) ||
      (st = Alloc(f, &f->d_out_vis, T)) || (st = Alloc(f, &f->d_shear, 1)) || (st = Alloc(f, &f->d_ticket, 1)) ||
      (st = Alloc(f, &f->d_n_over, 1)) || (st = Alloc(f, &f->d_stats, 3)) || (st = Alloc(f, &f->d_used, 1)) ||
      (st = Alloc(f, &f->d_pred_used, 1)) ||
      (st = Alloc(f, &f->d_vis_cursor, 1)) || (st = Alloc(f, &f->d_totals, 2)))
    return fail(st);
  // Record pool: 64 words per pixel of the largest image to start with; grows on demand.
  uint64_t max_px = 1;
  for (int v = 0; v < num_views; ++v)
    if (f->used[v]) max_px = std::max<uint64_t>(max_px, (uint64_t)views[v].width * views[v].height);
  // A seed's record holds at most the pixels within the reprojection radius of
  // its point in the image and in each overlapping image (about 16 each for
  // the default 2 pixels), each with one push per overlapping image. Start the
  // pool at that bound for the largest image (within a quarter of the free
  // device memory, but at least 64 words a pixel); it grows if an image needs more.
  int max_deg = 0;
  for (int v = 0; v < num_views; ++v) {
    max_deg = std::max(max_deg, overlap_offsets[v + 1] - overlap_offsets[v]);
    if (f->used[v]) f->deg = std::max(f->deg, overlap_offsets[v + 1] - overlap_offsets[v]);
  }
  const double radius = std::max(opt->max_reproj_error, 0.5);
  const uint64_t disk = (uint64_t)std::ceil((2.0 * radius + 1.0) * (2.0 * radius + 1.0));
  const uint32_t cnt_est = (uint32_t)std::min<uint64_t>(kCap, disk * (uint64_t)(1 + max_deg));
  size_t free_b = 0, total_b = 0;
  if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess) free_b = 0;
  uint64_t est = max_px * (uint64_t)RecWords(cnt_est, cnt_est * (uint32_t)max_deg);
  est = std::min<uint64_t>(est, std::max<uint64_t>(free_b / 16, max_px * 64ull));
  f->pool_words = (size_t)std::min<uint64_t>(std::max<uint64_t>(est, max_px * 64ull), 0xfffffff0ull);
  if ((st = Alloc(f, &f->d_pool, f->pool_words))) return fail(st);
  // The projection table: a word per pixel and overlapping image (845 MB for 11
  // views 1600x1200), when that is at most an eighth of the memory still free and
  // can be had; else the closures project in place.
  f->walk = t_walk;
  if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess) free_b = 0;
  const size_t table = T * (size_t)f->deg;
  if (!t_in_place && table > 0 && table * sizeof(uint32_t) <= free_b / 8 && Alloc(f, &f->d_proj, table))
    (void)cudaGetLastError();
  auto up = [&](void* dst, const void* src, size_t bytes) -> cudaError_t {
    return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDefault, f->stream);
  };
  std::vector<uint8_t> trav(f->used.begin(), f->used.end());
  if (up(f->d_views, f->h_views.data(), sizeof(FView) * num_views) != cudaSuccess ||
      (overlap_offsets[num_views] > 0 &&
       up(f->d_ov, overlap_images, sizeof(int32_t) * overlap_offsets[num_views]) != cudaSuccess) ||
      up(f->d_trav, trav.data(), (size_t)num_views) != cudaSuccess ||
      cudaMemsetAsync(f->d_mask, 0, T, f->stream) != cudaSuccess ||
      cudaMemsetAsync(f->d_claim_cnt, 0, T * 4, f->stream) != cudaSuccess ||
      cudaMemsetAsync(f->d_rgb, 0, 3 * T, f->stream) != cudaSuccess ||
      cudaMemsetAsync(f->d_totals, 0, 2 * sizeof(unsigned long long), f->stream) != cudaSuccess ||
      cudaMemsetAsync(f->d_out_visoff, 0, sizeof(uint64_t), f->stream) != cudaSuccess ||
      cudaMemsetAsync(f->d_stats, 0, 3 * sizeof(uint32_t), f->stream) != cudaSuccess)
    return fail(Fail(SMVS_ECUDA, "fusion: upload failed"));
  // Maps and point maps.
  if ((st = Alloc(f, &f->d_depth_in, (size_t)max_px))) return fail(st);
  const cudaMemcpyKind kind = memory == SMVS_MEM_HOST ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToDevice;
  for (int v = 0; v < num_views; ++v) {
    if (!f->used[v]) continue;
    const FView& hv = f->h_views[v];
    const size_t plane = (size_t)hv.W * hv.H;
    // A copy of a device map too: it takes an address of any alignment and a map on
    // another device, which the kernel could not read.
    if (cudaMemcpyAsync(f->d_depth_in, views[v].depth, plane * 4, kind, f->stream) != cudaSuccess)
      return fail(Fail(SMVS_ECUDA, "fusion: depth map copy failed"));
    if (views[v].color &&
        cudaMemcpyAsync(f->d_rgb + 3ull * hv.base, views[v].color, plane * 3, kind, f->stream) != cudaSuccess)
      return fail(Fail(SMVS_ECUDA, "fusion: color copy failed"));
    float* d_normal = nullptr;
    if (opt->with_normal) {
      if (memory == SMVS_MEM_HOST) {
        if ((st = Alloc(f, &d_normal, 3 * plane))) return fail(st);
        if (cudaMemcpyAsync(d_normal, views[v].normal, plane * 12, kind, f->stream) != cudaSuccess)
          return fail(Fail(SMVS_ECUDA, "fusion: normal map copy failed"));
      } else {
        d_normal = const_cast<float*>(views[v].normal);
      }
    }
    const float* R = views[v].R;
    PointMapKernel<<<Blocks(plane, 256), 256, 0, f->stream>>>(
        hv, R[0], R[1], R[2], R[3], R[4], R[5], R[6], R[7], R[8], f->d_depth_in, d_normal, c.with_normal,
        views[v].color != nullptr, f->d_pix, f->d_rgb);
    ++f->launches;
    if (f->d_proj) {
      ProjectTableKernel<<<Blocks(plane, 256), 256, 0, f->stream>>>(Maps(f), v, f->d_proj);
      ++f->launches;
    }
    if (memory == SMVS_MEM_HOST) Free(f, d_normal);
    if (cudaGetLastError() != cudaSuccess) return fail(Fail(SMVS_ECUDA, "fusion: point map launch failed"));
  }
  Free(f, f->d_depth_in);
  // The caller's maps are not referenced after this point.
  if (cudaStreamSynchronize(f->stream) != cudaSuccess) return fail(Fail(SMVS_ECUDA, "fusion: upload failed"));
  // Replay grid: every block resident.
  int per_sm = 0, sms = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, ReplayKernel, 32 * kReplayWarps, 0) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, f->device) != cudaSuccess || per_sm < 1)
    return fail(Fail(SMVS_ECUDA, "fusion: cannot size the replay grid"));
  f->replay_blocks = per_sm * sms;
  const auto closure = f->d_proj ? ClosureKernel<true> : ClosureKernel<false>;
  for (const auto kernel : {ClosureKernel<true>, ClosureKernel<false>})  // the table may have to go during the run
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kClosureSmem) != cudaSuccess)
      return fail(Fail(SMVS_ECUDA, "fusion: cannot size the closure grid"));
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, closure, 32 * kClosureWarps, kClosureSmem) !=
          cudaSuccess ||
      per_sm < 1)
    return fail(Fail(SMVS_ECUDA, "fusion: cannot size the closure grid"));
  f->closure_blocks = per_sm * sms;
  if ((st = Alloc(f, &f->d_stage, (size_t)f->closure_blocks * kClosureWarps * kStageBytes))) return fail(st);
  *out = f;
  return SMVS_OK;
}

int smvs_fusion_run(smvs_fusion* f) {
  if (!f) return Fail(SMVS_EINVAL, "null fusion");
  if (f->ran) return Fail(SMVS_ESTATE, "fusion: run may be called once");
  if (cudaSetDevice(f->device) != cudaSuccess) return Fail(SMVS_ECUDA, "fusion: cannot use GPU %d", f->device);
  f->ran = true;
  int start = 0;
  for (int i = 0; i < f->num_views; ++i)
    if (!f->views[i].is_rig) {
      start = i;
      break;
    }
  for (int image = start; image >= 0; image = FindNextImage(f, image)) {
    if (!f->used[image]) continue;
    int st = FuseImage(f, image);
    if (st) return st;
    f->fused[image] = 255;
    f->order.push_back(image);
  }
  int st = CheckStatus(f);
  if (st) return st;
  unsigned long long totals[2];
  FU_CUDA(cudaMemcpyAsync(totals, f->d_totals, sizeof(totals), cudaMemcpyDeviceToHost, f->stream));
  FU_CUDA(cudaStreamSynchronize(f->stream));
  f->num_points = totals[0];
  f->num_vis = totals[1];
  Harvest(f);
  return SMVS_OK;
}

int smvs_fusion_get_sizes(smvs_fusion* f, size_t* num_points, size_t* num_visibility) {
  if (!f) return Fail(SMVS_EINVAL, "null fusion");
  if (!f->ran) return Fail(SMVS_ESTATE, "fusion: run first");
  if (num_points) *num_points = (size_t)f->num_points;
  if (num_visibility) *num_visibility = (size_t)f->num_vis;
  return SMVS_OK;
}

int smvs_fusion_get_points(smvs_fusion* f, smvs_fused_point* points, uint64_t* vis_offsets, uint32_t* vis_images) {
  if (!f) return Fail(SMVS_EINVAL, "null fusion");
  if (!f->ran) return Fail(SMVS_ESTATE, "fusion: run first");
  if (points && f->num_points)
    FU_CUDA(cudaMemcpyAsync(points, f->d_out_pts, f->num_points * sizeof(smvs_fused_point), cudaMemcpyDefault,
                            f->stream));
  if (vis_offsets)
    FU_CUDA(cudaMemcpyAsync(vis_offsets, f->d_out_visoff, (f->num_points + 1) * sizeof(uint64_t), cudaMemcpyDefault,
                            f->stream));
  if (vis_images && f->num_vis)
    FU_CUDA(cudaMemcpyAsync(vis_images, f->d_out_vis, f->num_vis * sizeof(uint32_t), cudaMemcpyDefault, f->stream));
  FU_CUDA(cudaStreamSynchronize(f->stream));
  return SMVS_OK;
}

int smvs_fusion_get_device_points(smvs_fusion* f, const smvs_fused_point** points, const uint64_t** vis_offsets,
                                  const uint32_t** vis_images) {
  if (!f) return Fail(SMVS_EINVAL, "null fusion");
  if (!f->ran) return Fail(SMVS_ESTATE, "fusion: run first");
  if (points) *points = f->d_out_pts;
  if (vis_offsets) *vis_offsets = f->d_out_visoff;
  if (vis_images) *vis_images = f->d_out_vis;
  return SMVS_OK;
}

int smvs_fusion_get_image_order(smvs_fusion* f, int* order, int* count) {
  if (!f || !count) return Fail(SMVS_EINVAL, "null argument");
  *count = (int)f->order.size();
  if (order && !f->order.empty()) memcpy(order, f->order.data(), f->order.size() * sizeof(int));
  return SMVS_OK;
}

int smvs_fusion_get_mask(smvs_fusion* f, int view, uint8_t* out) {
  if (!f || !out) return Fail(SMVS_EINVAL, "null argument");
  if (view < 0 || view >= f->num_views) return Fail(SMVS_EINVAL, "fusion: image %d out of range", view);
  const FView& hv = f->h_views[view];
  const size_t plane = (size_t)f->views[view].width * (size_t)f->views[view].height;
  if (!f->used[view]) {
    memset(out, 0, plane);
    return SMVS_OK;
  }
  FU_CUDA(cudaMemcpyAsync(out, f->d_mask + hv.base, plane, cudaMemcpyDefault, f->stream));
  FU_CUDA(cudaStreamSynchronize(f->stream));
  return SMVS_OK;
}

int smvs_fusion_set_profiling(smvs_fusion* f, int enable) {
  if (!f) return Fail(SMVS_EINVAL, "null fusion");
  f->profiling = enable != 0;
  return SMVS_OK;
}

int smvs_fusion_get_profile(smvs_fusion* f, int kind, int* count, double* total_ms) {
  if (!f || !count || !total_ms || kind < 0 || kind > 3) return Fail(SMVS_EINVAL, "bad profile query");
  Harvest(f);
  *count = f->prof_count[kind];
  *total_ms = f->prof_ms[kind];
  return SMVS_OK;
}

int64_t smvs_fusion_launch_count(smvs_fusion* f) { return f ? f->launches : 0; }

int smvs_test_fusion_chains(smvs_fusion* f, uint32_t* chains, uint32_t* shears, int capacity, int* count) {
  if (!f || !count || capacity < 0 || (capacity > 0 && !chains)) return Fail(SMVS_EINVAL, "null argument");
  if (!f->ran || !f->d_chain) return Fail(SMVS_ESTATE, "fusion chains: run with profiling first");
  const int n = std::min<int>((int)f->order.size(), capacity);
  *count = (int)f->order.size();
  if (n > 0) {
    FU_CUDA(cudaMemcpyAsync(chains, f->d_chain, (size_t)n * sizeof(uint32_t), cudaMemcpyDeviceToHost, f->stream));
    if (shears)
      FU_CUDA(cudaMemcpyAsync(shears, f->d_chain + f->num_views, (size_t)n * sizeof(uint32_t), cudaMemcpyDeviceToHost,
                              f->stream));
    FU_CUDA(cudaStreamSynchronize(f->stream));
  }
  return SMVS_OK;
}

int smvs_test_fusion_image_ms(smvs_fusion* f, double* ms, int capacity, int* count) {
  if (!f || !count || capacity < 0 || (capacity > 0 && !ms)) return Fail(SMVS_EINVAL, "null argument");
  Harvest(f);
  const int n = (int)(f->prof_image_ms.size() / 4);
  *count = n;
  for (int i = 0; i < std::min(n, capacity) * 4; ++i) ms[i] = f->prof_image_ms[i];
  return SMVS_OK;
}

int smvs_test_fusion_replay_times(smvs_fusion* f, double* out, int capacity, int* count) {
  if (!f || !count || capacity < 0 || (capacity > 0 && !out)) return Fail(SMVS_EINVAL, "null argument");
  if (!f->ran || !f->d_times) return Fail(SMVS_ESTATE, "fusion replay times: run with profiling first");
  const int n = (int)f->order.size();
  *count = n;
  std::vector<unsigned long long> t(9 * (size_t)n);
  if (n > 0) {
    FU_CUDA(cudaMemcpyAsync(t.data(), f->d_times, t.size() * sizeof(unsigned long long), cudaMemcpyDeviceToHost,
                            f->stream));
    FU_CUDA(cudaStreamSynchronize(f->stream));
  }
  for (int i = 0; i < std::min(n, capacity); ++i) {
    const unsigned long long* ti = t.data() + 9 * i;
    const double seeds = (double)std::max<unsigned long long>(ti[2], 1);
    double* o = out + 9 * i;
    o[0] = (double)ti[0] / seeds / 1000.0;
    o[1] = (double)ti[1] / seeds / 1000.0;
    o[2] = (double)ti[2];
    o[3] = (double)ti[3] / seeds;
    o[4] = (double)ti[4] / seeds;
    o[5] = (double)ti[5];
    o[6] = (double)ti[6] / seeds / 1000.0;
    o[7] = (double)ti[7] / seeds / 1000.0;
    o[8] = (double)ti[8] / seeds / 1000.0;
  }
  return SMVS_OK;
}

int smvs_test_row_and_column(const uint32_t* px, int n, int width, int32_t* rows, int32_t* cols) {
  if (n < 0 || width < 1 || (n > 0 && (!px || !rows || !cols))) return Fail(SMVS_EINVAL, "row and column: bad arguments");
  for (int i = 0; i < n; ++i) RowAndColumn(px[i], width, rows + i, cols + i);
  return SMVS_OK;
}

int smvs_test_fusion_paths(int in_place, int walk) {
  t_in_place = in_place != 0;
  t_walk = walk != 0;
  return SMVS_OK;
}

int smvs_test_fusion_caps(int closure_cap, int replay_cap, int replay_stack) {
  if (closure_cap < 0 || replay_cap < 0 || replay_stack < 0 || (replay_stack > 0 && replay_stack < 2))
    return Fail(SMVS_EINVAL, "fusion caps: bad values");
  t_cap_closure = closure_cap;
  t_cap_replay = replay_cap;
  t_cap_stack = replay_stack;
  return SMVS_OK;
}

int smvs_test_fusion_waits(double limit_seconds, long long withhold_seed) {
  if (limit_seconds < 0 || withhold_seed < -2) return Fail(SMVS_EINVAL, "fusion waits: bad values");
  t_wait_limit_ns = (unsigned long long)(limit_seconds * 1e9);
  t_withhold = withhold_seed;
  return SMVS_OK;
}

int smvs_fusion_remove_duplicate_points(smvs_fusion* f, size_t* num_removed) {
  if (!f) return Fail(SMVS_EINVAL, "null fusion");
  if (!f->ran) return Fail(SMVS_ESTATE, "fusion: run first");
  if (cudaSetDevice(f->device) != cudaSuccess) return Fail(SMVS_ECUDA, "fusion: cannot use GPU %d", f->device);
  if (num_removed) *num_removed = 0;
  const uint32_t n = (uint32_t)f->num_points;  // at most half the pixels, fewer than 2^30
  if (n == 0) return SMVS_OK;
  const int max_level = f->num_views;  // a point lists an image once
  uint32_t *cells = f->d_vis_pool, *earliest = f->d_claim_cnt, *latest = f->d_claim_off;
  uint32_t *keep, *list, *counts;
  DupView* d_views;
  Carve scratch(f);
  CompactScratch compact;
  int st;
  if ((st = scratch.Take(&keep, n)) || (st = scratch.Take(&list, n)) ||
      (st = scratch.Take(&counts, (size_t)max_level + 1)) || (st = scratch.Take(&d_views, (size_t)f->num_views)) ||
      (st = compact.Take(f, scratch)))
    return st;
  std::vector<DupView> views(f->num_views);
  for (int v = 0; v < f->num_views; ++v) {
    const smvs_fusion_view& fv = f->views[v];
    memcpy(views[v].K, fv.K, sizeof(fv.K));
    memcpy(views[v].R, fv.R, sizeof(fv.R));
    memcpy(views[v].T, fv.T, sizeof(fv.T));
    views[v].W = f->h_views[v].W;
    views[v].H = f->h_views[v].H;
    views[v].base = f->h_views[v].base;
  }
  FU_CUDA(cudaMemcpyAsync(d_views, views.data(), views.size() * sizeof(DupView), cudaMemcpyHostToDevice, f->stream));
  FU_CUDA(cudaMemsetAsync(counts, 0, ((size_t)max_level + 1) * 4, f->stream));
  FU_CUDA(cudaMemsetAsync(earliest, 0xff, (size_t)f->total * 4, f->stream));
  FU_CUDA(cudaMemsetAsync(latest, 0, (size_t)f->total * 4, f->stream));
  DupLevelsKernel<<<std::min<uint32_t>(Blocks(n, 256), 296), 256, 0, f->stream>>>(n, f->d_out_visoff, max_level, counts);
  FU_CUDA(cudaGetLastError());
  std::vector<uint32_t> count((size_t)max_level + 1), start((size_t)max_level + 1);
  FU_CUDA(cudaMemcpyAsync(count.data(), counts, count.size() * 4, cudaMemcpyDeviceToHost, f->stream));
  FU_CUDA(cudaStreamSynchronize(f->stream));
  uint32_t at = 0;
  for (int level = max_level; level >= 0; --level) {
    start[level] = at;
    at += count[level];
  }
  FU_CUDA(cudaMemcpyAsync(counts, start.data(), start.size() * 4, cudaMemcpyHostToDevice, f->stream));
  DupOrderKernel<<<Blocks(n, 256), 256, 0, f->stream>>>(n, f->d_out_visoff, max_level, counts, list);
  f->launches += 2;
  for (int level = max_level; level >= 0; --level) {
    if (!count[level]) continue;
    DupStopKernel<<<Blocks(count[level], 128), 128, 0, f->stream>>>(list + start[level], count[level], f->d_out_pts,
                                                                    f->d_out_visoff, f->d_out_vis, d_views, earliest,
                                                                    cells, keep);
    DupTakeKernel<<<Blocks(count[level], 128), 128, 0, f->stream>>>(list + start[level], count[level], f->d_out_visoff,
                                                                    cells, earliest, latest);
    f->launches += 2;
  }
  DupDropKernel<<<Blocks(n, 256), 256, 0, f->stream>>>(n, f->d_out_visoff, cells, latest, keep);
  ++f->launches;
  FU_CUDA(cudaGetLastError());
  return Compact(f, compact, keep, num_removed);
}

int smvs_fusion_remove_outliers(smvs_fusion* f, int nb_neighbors, double max_spacing_factor, size_t* num_removed) {
  if (!f) return Fail(SMVS_EINVAL, "null fusion");
  if (!f->ran) return Fail(SMVS_ESTATE, "fusion: run first");
  if (nb_neighbors < 1 || nb_neighbors + 1 > kMaxKnn)
    return Fail(SMVS_EINVAL, "fusion: nb_neighbors must be in 1..%d", kMaxKnn - 1);
  if (!(max_spacing_factor > 0)) return Fail(SMVS_EINVAL, "fusion: max_spacing_factor must be > 0");
  if (cudaSetDevice(f->device) != cudaSuccess) return Fail(SMVS_ECUDA, "fusion: cannot use GPU %d", f->device);
  if (num_removed) *num_removed = 0;
  const size_t n = f->num_points;
  if (n == 0) return SMVS_OK;
  if (n >= (1ull << 32) - 1) return Fail(SMVS_EINVAL, "fusion: too many points for the neighbour grid");
  const uint32_t nn = (uint32_t)n;
  Carve scratch(f);
  CompactScratch compact;
  CloudStats* stats;
  uint32_t* keep;
  int st;
  if ((st = scratch.Take(&stats, 1)) || (st = scratch.Take(&keep, n))) return st;
  const int sweep = std::min<uint32_t>(Blocks(n, 256), 296);
  StatsResetKernel<<<1, 256, 0, f->stream>>>(stats);
  CloudBoxKernel<<<sweep, 256, 0, f->stream>>>(f->d_out_pts, nn, stats);
  f->launches += 2;
  FU_CUDA(cudaGetLastError());
  CloudStats h_stats;
  FU_CUDA(cudaMemcpyAsync(h_stats.range, stats->range, sizeof(h_stats.range), cudaMemcpyDeviceToHost, f->stream));
  FU_CUDA(cudaStreamSynchronize(f->stream));
  // Grid over the bounding box: cells of equal side, at least one per axis, at most
  // 2^24 per axis, about kCells per point. The points lie on surfaces, so an
  // occupied cell holds about (n / kCells^2)^(1/3) of them (10 of 65,000) and a
  // cube of 27 cells is near the smallest that holds the neighbours.
  constexpr int kCells = 8;
  double lo[3], hi[3];
  for (int a = 0; a < 3; ++a) {
    const bool any = h_stats.range[2 * a] <= h_stats.range[2 * a + 1];
    lo[a] = any ? KeyFloat(h_stats.range[2 * a]) : INFINITY;
    hi[a] = any ? KeyFloat(h_stats.range[2 * a + 1]) : -INFINITY;
  }
  if (!(std::isfinite(lo[0]) && std::isfinite(lo[1]) && std::isfinite(lo[2]) && std::isfinite(hi[0]) &&
        std::isfinite(hi[1]) && std::isfinite(hi[2])))
    return Fail(SMVS_EINVAL, "fusion: non-finite point coordinates");
  const double ext[3] = {hi[0] - lo[0], hi[1] - lo[1], hi[2] - lo[2]};
  const double emax = std::max(ext[0], std::max(ext[1], ext[2]));
  double vol = 1.0;
  int flat = 0;
  for (int a = 0; a < 3; ++a) {
    if (ext[a] > emax * 1e-6) vol *= ext[a];
    else ++flat;
  }
  double h = emax > 0 ? std::pow(vol / ((double)kCells * (double)n), 1.0 / (3 - std::min(flat, 2))) : 1.0;
  if (!(h > 0)) h = 1.0;
  KnnGrid g;
  g.minx = lo[0]; g.miny = lo[1]; g.minz = lo[2];
  int dims[3];
  for (;;) {
    for (int a = 0; a < 3; ++a) dims[a] = (int)std::min(16777216.0, std::floor(ext[a] / h) + 1.0);
    if ((double)dims[0] * dims[1] * dims[2] <= std::min(2.0 * kCells * (double)n + 64.0, 2147483648.0)) break;
    h *= 1.26;
  }
  g.h = h; g.inv_h = 1.0 / h;
  g.gx = dims[0]; g.gy = dims[1]; g.gz = dims[2];
  const size_t cells = (size_t)g.gx * g.gy * g.gz;
  uint32_t *cell_of, *counts, *startv;
  float4* sorted;
  float* spacing;
  if ((st = scratch.Take(&cell_of, n)) || (st = scratch.Take(&counts, cells)) ||
      (st = scratch.Take(&startv, cells + 1)) || (st = scratch.Take(&sorted, n)) || (st = scratch.Take(&spacing, n)) ||
      (st = compact.Take(f, scratch)))
    return st;
  const int K = nb_neighbors + 1;
  FU_CUDA(cudaMemsetAsync(counts, 0, cells * sizeof(uint32_t), f->stream));
  KnnCountKernel<<<Blocks(n, 256), 256, 0, f->stream>>>(f->d_out_pts, nn, g, cell_of, counts);
  if ((st = Scan(f, counts, cells, startv))) return st;
  KnnScatterKernel<<<Blocks(n, 256), 256, 0, f->stream>>>(f->d_out_pts, nn, cell_of, startv, counts, sorted);
  auto knn = K <= 8 ? KnnSpacingKernel<8> : K <= 16 ? KnnSpacingKernel<16> : KnnSpacingKernel<kMaxKnn>;
  knn<<<Blocks(n, 128), 128, 0, f->stream>>>(sorted, nn, g, startv, K, spacing);
  f->launches += 3;
  FU_CUDA(cudaGetLastError());
  std::vector<float> dists(n);
  FU_CUDA(cudaMemcpyAsync(dists.data(), spacing, n * sizeof(float), cudaMemcpyDeviceToHost, f->stream));
  FU_CUDA(cudaStreamSynchronize(f->stream));
  // ComputeAverageDistance's mean (patch_match_controller.cc:184-227): a float
  // sum in point order, whose roundings no other order gives.
  float average = 0.0f;
  for (size_t i = 0; i < n; ++i) average += dists[i];
  average /= (float)n;
  // RemoveOutliers (fusion.cc:2542-2611): blend each score with its spacing
  // ratio, histogram the scores over 256 bins of [min, max], and drop points
  // in a bin holding under 1 % of the points at or above the 90th cumulative
  // percent.
  ScoreKernel<<<sweep, 256, 0, f->stream>>>(f->d_out_pts, nn, spacing, average > 1e-6,
                                            max_spacing_factor * (double)average, stats);
  HistKernel<<<sweep, 256, 0, f->stream>>>(f->d_out_pts, nn, stats);
  f->launches += 2;
  FU_CUDA(cudaGetLastError());
  FU_CUDA(cudaMemcpyAsync(h_stats.bins, stats->bins, sizeof(h_stats.bins), cudaMemcpyDeviceToHost, f->stream));
  FU_CUDA(cudaStreamSynchronize(f->stream));
  BinMask mask{};
  float sum = 0.0f;
  for (int k = 0; k < 256; ++k) {
    // The reference counts in floats, which stop at 2^24.
    const float ratio = (float)std::min<uint32_t>(h_stats.bins[k], 1u << 24) / (float)n;
    sum += ratio;
    if ((double)ratio < 0.01 && (double)sum >= 0.9) mask.drop[k / 32] |= 1u << (k % 32);
  }
  BinKeepKernel<<<Blocks(n, 256), 256, 0, f->stream>>>(f->d_out_pts, nn, stats, mask, keep);
  ++f->launches;
  FU_CUDA(cudaGetLastError());
  return Compact(f, compact, keep, num_removed);
}

void smvs_fusion_destroy(smvs_fusion* f) {
  if (!f) return;
  cudaSetDevice(f->device);
  FreeAll(f);
  delete f;
}

}  // extern "C"
