// Depth ingest, bilateral filter, depth pyramid and input vertex/normal maps.
//
// HBM-bound streaming stages: one pass over the uint16 frame, shared-memory
// tiles with halos, coalesced 2D blocks.  Every kernel is persistent over the
// tiles of all sessions of a batch table (one session = a table of one).
// Each kernel restates one reference routine (paths relative to
// VCL_Volume_Scanner/):
//   k_bilateral_*    d_bilateral_filter  STAC/Engine/GPU/z_yooji_cuda_img_proc.cu:103-141
//   k_pyramid_batch  sdg5 + ddh          STAC/Engine/CPU/z_yooji_image_processor.cpp:567-596,857-937
//   k_inmap_*        cpm + enm           STAC/Engine/CPU/z_yooji_image_processor.cpp:119-227
#include <cuda_runtime.h>
#include <stdint.h>

#include <cstring>

#include "vs_internal.cuh"

namespace vs {
namespace {

constexpr int BX = 32, BY = 8;  // threads of a filter block (BY: default rows; 4 and 16 also built)
constexpr int kPerThread = 2;   // outputs per thread, consecutive rows (1 also built, for small float maps)
constexpr int kScanSmem = 64 * 1024;  // staged normal-rejection bitmasks of one level

// The reference reads a linear-filtered texture at integer coordinates, so
// every tap is the mean of the 2x2 texels (X-1..X, Y-1..Y); out-of-range texel
// coordinates clamp to the edge.  A tile of BX x 2R outputs needs taps
// X in [x0-2, x0+BX+1] and texels in [x0-3, x0+BX+1].
//
// Bound by the 24 exponentials of a pixel on the special-function unit (an
// eighth of a warp per cycle and scheduler: 192 cycles per warp and row) and
// as much by its other instructions (eight per tap).  A thread filters
// consecutive rows of a column, so taps are read from shared memory 15 times
// per pixel instead of 25 and the tile's borders shrink, and holes need no
// test per tap.  With one output per thread in 32 x 8 tiles 1920x1080 took
// 33.5 us, and takes 25.2; four rows per thread 26 us, and 2 us more for one
// 640x480 frame, whose tiles are few.
template <int R, int P>
struct BilateralSmem {
  float tex[P * R + 5][BX + 6];
  float tap[P * R + 4][BX + 5];
};

// exp2 by the special-function unit (ex2.approx.ftz.f32)
__device__ __forceinline__ float exp2_approx(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// The filter of P pixels, rows ty0 .. of column tx.  Every sum runs in
// the reference's order with its roundings.  A tap that is not above 0 is stored as
// -infinity: as the centre it makes the sum infinite, elsewhere its weight is
// 0 and their product not a number.
template <bool FROM_MM, int R, int P>
__device__ inline void bilateral_px(const BilateralSmem<R, P>& m, int tx, int ty0, bool finite, float out[P]) {
  // The Gaussian of delta 4 (:275-286), exp(-x^2 / (2 * 4^2)).  The range
  // weight's exponent is -mod / (2 sigma_r^2), 2 sigma_r^2 = 2.0f * 0.1f *
  // 0.1f with sigma_r = 0.1 m (z_yooji_cuda_img_proc.cu:44,91), here the
  // product with the folded constant -1 / (2 sigma_r^2): one rounding more
  // than the quotient (a relative 1.2e-7 of an exponent that matters only
  // below ~20), far inside the 1e-5 m tolerance of the filtered depth, and no
  // division per tap.  Its exponential is that of the product with log2(e) to
  // the base 2; below 2^-126 it gives 0, which no sum of weights that holds
  // the centre's 1 tells from the subnormal.
  constexpr float g1 = 0.96923321f, g2 = 0.88249689f;  // exp(-1 / 32), exp(-4 / 32) rounded to float
  constexpr float g[5] = {g2, g1, 1.0f, g1, g2};
  constexpr float kNegInvDenom = -1.0f / (2.0f * 0.1f * 0.1f), kLog2e = 1.44269504f;
  float c[P], t[P], sum[P];
#pragma unroll
  for (int r = 0; r < P; r++) {
    c[r] = m.tap[ty0 + r + 2][tx + 2];
    t[r] = sum[r] = 0.0f;
  }
#pragma unroll
  for (int k = 0; k < P + 4; k++) {
    float a[5];
#pragma unroll
    for (int j = 0; j < 5; j++) a[j] = m.tap[ty0 + k][tx + j];
#pragma unroll
    for (int r = 0; r < P; r++) {
      const int i = k - r;
      if (i < 0 || i > 4) continue;
#pragma unroll
      for (int j = 0; j < 5; j++) {
        if (i == 2 && j == 2) {  // the centre: weight 1
          t[r] += c[r];
          sum[r] += 1.0f;
          continue;
        }
        const float d = c[r] - a[j];
        const float w = (g[i] * g[j]) * exp2_approx(d * d * kNegInvDenom * kLog2e);
        t[r] += w * a[j];
        sum[r] += w;
      }
    }
  }
#pragma unroll
  for (int r = 0; r < P; r++) {
    out[r] = t[r] / sum[r];
    if (!(t[r] >= 0.0f)) {
      bool hole = finite;  // finite inputs: only a hole gives this
      // (a frame of units comes here with an unusual scale only: unrolled, the
      // search would take 72 registers instead of 40 for every frame)
      if (!finite)
#pragma unroll FROM_MM ? 1 : 25
        for (int i = 0; i < 25; i++) hole |= m.tap[ty0 + r + i / 5][tx + i % 5] == __int_as_float(0xff800000);
      if (hole) out[r] = 0.0f;
    }
  }
}

// one BX x P R output tile; the block's BX x R threads all take part (two barriers)
template <bool FROM_MM, int R, int P>
__device__ inline void bilateral_tile(BilateralSmem<R, P>& m, const uint16_t* __restrict__ mm,
                                      const float* __restrict__ fin, float scale, float* __restrict__ raw_out,
                                      float* __restrict__ out, int W, int H, int x0, int y0,
                                      float2* __restrict__ dl_out = nullptr, const float* __restrict__ lam = nullptr) {
  constexpr int TR = P * R;
  const int tx = threadIdx.x, ty = threadIdx.y;
  // a warp per texel row: BX columns, then the five beyond
#pragma unroll
  for (int q = 0; q < (TR + 5 + R - 1) / R; q++) {
    const int r = ty + q * R;
    if (r < TR + 5) {
      const int gy = min(max(y0 - 3 + r, 0), H - 1);
      const int gx = min(max(x0 - 3 + tx, 0), W - 1), gx2 = min(max(x0 - 3 + BX + tx, 0), W - 1);
      if (FROM_MM) {
        m.tex[r][tx] = (float)mm[(size_t)gy * W + gx] * scale;
        if (tx < 5) m.tex[r][BX + tx] = (float)mm[(size_t)gy * W + gx2] * scale;
      } else {
        m.tex[r][tx] = fin[(size_t)gy * W + gx];
        if (tx < 5) m.tex[r][BX + tx] = fin[(size_t)gy * W + gx2];
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < (TR + 4 + R - 1) / R; q++) {
    const int r = ty + q * R;
    if (r < TR + 4) {
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const int x = tx + e * BX;
        if (e == 0 || tx < 4) {
          const float v = 0.25f * ((m.tex[r][x] + m.tex[r][x + 1]) + (m.tex[r + 1][x] + m.tex[r + 1][x + 1]));
          m.tap[r][x] = v <= 0.0f ? __int_as_float(0xff800000) : v;
        }
      }
    }
  }
  __syncthreads();
  const int x = x0 + tx, yb = y0 + ty * P;
  if (x < W && yb < H) {
    float f[P];
    // scaled units are finite, and so are the sums of their taps, unless the
    // session's scale itself is out of range (65535 units of 1e30 are 6.6e34)
    bilateral_px<FROM_MM>(m, tx, ty * P, FROM_MM && fabsf(scale) <= 1.0e30f, f);
#pragma unroll
    for (int r = 0; r < P; r++) {
      if (yb + r >= H) break;
      const size_t i = (size_t)(yb + r) * W + x;
      if (FROM_MM) {
        const float raw = m.tex[ty * P + r + 3][tx + 3];
        raw_out[i] = raw;
        if (dl_out) dl_out[i] = make_float2(raw, __ldg(lam + i));
      }
      out[i] = f[r];
    }
  }
}

// Frames read in place (device memory, or pinned host memory over the host
// link) into the sessions' frame buffers: each pixel crosses the link once, in
// 8-byte reads.  (The filter reading such a frame itself read every pixel 2.9
// times with its tiles' borders: the filter stage of the 64-session step from
// pinned frames took 0.98 ms, and takes 0.70.)  A slot's filter tiles count its
// chunks of 2 BX BY pixels: they cover the image, so the chunks do.
__global__ void __launch_bounds__(BX* BY) k_ingest(const BatchTable* __restrict__ bt) {
  const int n = bt->n;
  const int total = bt->fil[n];
  for (int item = blockIdx.x; item < total; item += gridDim.x) {
    int t;
    const int slot = find_slot(bt->fil, n, item, t);
    const SessionDev* __restrict__ s = bt->s[slot];
    const uint16_t* __restrict__ src = bt->frame[slot];
    if (!src || src == s->depth_mm) continue;
    uint16_t* __restrict__ dst = s->depth_mm;
    const int px = s->lv[0].W * s->lv[0].H, chunk = kPerThread * BX * bt->bil_rows;
    const bool wide = (reinterpret_cast<uintptr_t>(src) & 7) == 0;
    for (int i = t * chunk + threadIdx.x * 4; i < min(px, (t + 1) * chunk); i += BX * BY * 4) {
      if (wide && i + 4 <= px) {
        *reinterpret_cast<uint2*>(dst + i) = *reinterpret_cast<const uint2*>(src + i);
      } else {
        for (int k = i; k < min(px, i + 4); k++) dst[k] = src[k];
      }
    }
  }
}

template <int R>
__global__ void __launch_bounds__(BX* R) k_bilateral_batch(const BatchTable* __restrict__ bt) {
  __shared__ BilateralSmem<R, kPerThread> m;
  const int n = bt->n;
  const int total = bt->fil[n];
  for (int item = blockIdx.x; item < total; item += gridDim.x) {
    int t;
    const int slot = find_slot(bt->fil, n, item, t);
    const SessionDev* __restrict__ s = bt->s[slot];
    const int W = s->lv[0].W, H = s->lv[0].H;
    const int tw = (W + BX - 1) / BX, tyy = t / tw;
    const int x0 = (t - tyy * tw) * BX, y0 = tyy * R * kPerThread;
    bilateral_tile<true, R, kPerThread>(m, s->depth_mm, nullptr, s->depth_scale, s->depth_raw, s->depth[0], W, H, x0,
                                        y0, s->lam_map ? s->dl_map : nullptr, s->lam_map);
    if (s->rgb_packed) {
      // the colour frame as one word per pixel, for the integration's gathers
      const int x = x0 + threadIdx.x;
      for (int y = y0 + threadIdx.y; x < W && y < min(H, y0 + R * kPerThread); y += R) {
        const size_t i = (size_t)y * W + x, plane = (size_t)W * H;
        s->rgb_packed[i] = pack_rgb(s->rgb_in[i], s->rgb_in[plane + i], s->rgb_in[2 * plane + i]);
      }
    }
    __syncthreads();  // the next tile overwrites the shared tiles
  }
}

template <int P>
__global__ void __launch_bounds__(BX* BY, 6)
    k_bilateral_float(const float* __restrict__ in, float* __restrict__ out, int W, int H) {
  __shared__ BilateralSmem<BY, P> m;
  bilateral_tile<false, BY, P>(m, nullptr, in, 1.0f, nullptr, out, W, H, blockIdx.x * BX, blockIdx.y * BY * P);
}

// level l -> l+1: separable [1 4 6 4 1] smoothing (borders 0, no validity
// mask) evaluated only at the kept pixel (2 i2 + 1, 2 j2 + 1)
__global__ void __launch_bounds__(256) k_pyramid_batch(const BatchTable* __restrict__ bt, int l2) {
  const int n = bt->n;
  const int* pre = bt->pyr[l2 - 1];
  const int total = pre[n];
  for (int item = blockIdx.x; item < total; item += gridDim.x) {
    int t;
    const int slot = find_slot(pre, n, item, t);
    const SessionDev* __restrict__ s = bt->s[slot];
    const int w = s->lv[l2 - 1].W, h = s->lv[l2 - 1].H, w2 = s->lv[l2].W, h2 = s->lv[l2].H;
    const int tw = (w2 + 31) / 32;
    const int i2 = (t % tw) * 32 + threadIdx.x, j2 = (t / tw) * 8 + threadIdx.y;
    if (i2 >= w2 || j2 >= h2) continue;
    const float* __restrict__ in = s->depth[l2 - 1];
    int i = 2 * i2 + 1, j = 2 * j2 + 1;
    float v = 0.0f;
    if (i >= 2 && i < w - 2 && j >= 2 && j < h - 2) {
      float pad[5];
#pragma unroll
      for (int r = 0; r < 5; r++) {
        const float* p = in + (size_t)(j - 2 + r) * w;
        pad[r] = p[i - 2] + p[i + 2] + 4.0f * p[i - 1] + 4.0f * p[i + 1] + 6.0f * p[i];
      }
      v = (pad[0] + pad[4] + 4.0f * pad[1] + 4.0f * pad[3] + 6.0f * pad[2]) / (16.0f * 16.0f);
    }
    s->depth[l2][(size_t)j2 * w2 + i2] = v;
  }
}

// ---------------------------------------------------------------------------
// input vertex / normal maps (enm_Estimate_Normal_Map semantics)
//
// pass 1 (parallel): per interior pixel, code 0 = no normal (an invalid
//   point among the 5, or |dx|,|dy| < 1e-7), 1 = normal accepted,
//   2 = normal rejected by the 60 degree test; accepted normals are stored,
//   and codes 1 and 2 as bitmasks of 32 pixels per word.
// pass 2 (one block per level, rows in order): the reference rewrites the
//   point map in place on a rejection, which blocks the right and lower
//   neighbours.  With C = code2 & ~R(row above), a row solves
//   R_j = C_j & ~R_{j-1}: inside each run of C the rejected pixels alternate
//   starting at the run's first pixel.  Runs are smeared with one addition
//   per 32-bit word; the words of a row and the rows themselves are swept as
//   a wavefront across the lanes of one warp.  The block then counts the
//   valid normals before each word.
// pass 3 (parallel): vertex valid = depth > 0 and not rejected; normal valid =
//   code 1 and neither the left nor the upper neighbour rejected: the normals
//   that are not are overwritten, and the valid ones' pixels are listed in
//   raster order for the tracker.
// A session's items cover its levels in order; the per-level tile counts
// follow from the level sizes.
//
// Passes 1 and 3 are bound by instruction issue and by their writes (16 B
// normal and 16 B vertex per pixel, each written once but for the normals
// that pass 3 takes back; 32-row tiles spread the table search of a tile over
// four rows per thread), pass 2 by the wavefront's chain (about 80 cycles per
// row; 24 us for 640x480 with the counting, 37 before).  Before, pass 1 wrote
// candidate normals and a code byte that pass 3 read and wrote again: the
// filter stage of one 640x480 frame went from 72 to 60 us, of the 64-session
// step (frames read from pinned memory) from 1.12 to 0.98 ms.
// ---------------------------------------------------------------------------
__device__ inline int level_of_tile(const SessionDev& s, int tile_w, int tile_h, int& t) {
  int l = 0;
  for (; l < s.levels - 1; l++) {
    const int nt = ((s.lv[l].W + tile_w - 1) / tile_w) * ((s.lv[l].H + tile_h - 1) / tile_h);
    if (t < nt) break;
    t -= nt;
  }
  return l;
}

constexpr int kMapRows = 32;  // a tile of the map passes is 32 x kMapRows pixels, 8 rows at a time

// Normals and their codes.  Bound by latency, then issue: with the five depths
// of a pixel behind one another's tests a 640x480 frame's levels took 7.4 us and
// 32 sessions' 94, read together 6.1 and 74.
__global__ void __launch_bounds__(256) k_inmap_pre(const BatchTable* __restrict__ bt) {
  const int n = bt->n;
  const int total = bt->imap[n];
  for (int item = blockIdx.x; item < total; item += gridDim.x) {
    int t;
    const int slot = find_slot(bt->imap, n, item, t);
    const SessionDev& s = *bt->s[slot];
    const int l = level_of_tile(s, 32, kMapRows, t);
    const int w = s.lv[l].W, h = s.lv[l].H;
    const float K[4] = {s.lv[l].K[0], s.lv[l].K[1], s.lv[l].K[2], s.lv[l].K[3]};
    const float* __restrict__ depth = s.depth[l];
    const int tw = (w + 31) / 32, ty = t / tw, tx = t - ty * tw;
    const int x = tx * 32 + threadIdx.x;
#pragma unroll 1
    for (int y = ty * kMapRows + threadIdx.y; y < min(h, (ty + 1) * kMapRows); y += 8) {
      // a warp is one 32-pixel word of a row
      int code = 0;
      float4 nv = make_float4(-100.0f, -100.0f, -100.0f, 0.0f);
      if (x >= 1 && x < w - 1 && y >= 1 && y < h - 1) {
        // the five reads go out before any test
        const float* __restrict__ at = depth + (size_t)y * w + x;
        const float dc = at[0], dl = at[-1], dr = at[1], du = at[-w], dd = at[w];
        if (!(dc <= 0.0f) && !(dl <= 0.0f) && !(dr <= 0.0f) && !(du <= 0.0f) && !(dd <= 0.0f)) {
          const F3 x1 = back_project((float)(x - 1), (float)y, K, dl);
          const F3 x2 = back_project((float)(x + 1), (float)y, K, dr);
          const F3 y1 = back_project((float)x, (float)(y - 1), K, du);
          const F3 y2 = back_project((float)x, (float)(y + 1), K, dd);
          float dx = x2.x - x1.x;
          float dy = y2.y - y1.y;
          if (!(fabsf(dx) < 1.0e-7f) && !(fabsf(dy) < 1.0e-7f)) {
            float dzdx = (x2.z - x1.z) / dx;
            float dzdy = (y2.z - y1.z) / dy;
            float len = sqrtf(dzdx * dzdx + dzdy * dzdy + 1.0f);
            float nz = -1.0f / len;
            // -n_z < cos(60 deg), the threshold taken in double as the reference's cos():
            // a float is below it iff it is at most 0.5
            if (-nz <= 0.5f) {
              code = 2;
            } else {
              code = 1;
              nv = make_float4(dzdx / len, dzdy / len, nz, 1.0f);
            }
          }
        }
      }
      const unsigned m2 = __ballot_sync(0xffffffffu, code == 2), m1 = __ballot_sync(0xffffffffu, code == 1);
      if (threadIdx.x == 0) {
        s.in_amask[l][y * tw + tx] = m2;
        s.in_cmask[l][y * tw + tx] = m1;
      }
      if (x < w) s.in_nrm[l][(size_t)y * w + x] = nv;
    }
  }
}

// Row sweep of one level: warp 0 sweeps the rows as a wavefront: at step t
// lane l solves row t - l for its words, taking the carry of the row's earlier
// words from lane l - 1 (computed at step t - 1) and the rejections of the row
// above from its own registers, so one step costs one shuffle.  am: the
// level's code-2 bitmasks; rm receives the rejections (the same array where
// they are in shared memory: a word is read one step before it is written).
__device__ __forceinline__ void scan_level(const uint32_t* am, uint32_t* rm, int w, int h) {
  const int nw = (w + 31) >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t M0 = 0x55555555u, M1 = 0xaaaaaaaau;
  const int wpl = (nw + 31) >> 5;  // words per lane (1 up to 1024 pixels, 2 up to 2048)
  const int steps = h + 31;
  if (wpl == 1) {
    // Both outcomes of a word are formed before its carry arrives (a carry
    // travels as a mask of 32 equal bits, so that choosing is one logic
    // operation), the next word is read a step ahead, and rows outside the
    // image hold no code, so they need no test: a step's critical path is a
    // chain of eight operations from the row above, beside one of a shuffle
    // and four.  Row 0 is never processed (interior rows only).
    const bool act = lane < nw;
    const uint32_t not_first = lane ? ~0u : 0u;
    const unsigned rows = act ? (unsigned)h : 0u, ahead = act ? (unsigned)h - 1u : 0u;  // none for an idle lane
    uint32_t rup = 0u, cout = 0u, next = 0u, next1 = 0u;
    int i = lane - lane * nw;  // word of row t - lane
#pragma unroll 4
    for (int t = 0; t < steps; t++, i += nw) {
      const unsigned row = (unsigned)(t - lane);
      const uint32_t C = next & ~rup, C1 = next1 & ~(rup << 1);  // C1 = C << 1
      next = 0u;
      if (row < ahead) next = am[i + nw];
      next1 = next << 1;
      // run starts at even and odd bits (C & ~C1; one at bit 0 apart), and the
      // runs they smear over
      const uint32_t e = C + (C & ~C1 & (M0 & ~1u)), o = C + (C & ~C1 & M1), z = C + (C & 1u);
      const uint32_t both = C & (((e ^ C) & M0) | ((o ^ C) & M1)), zero = C & (z ^ C);
      // a run at bit 0 continues the previous word's alternation: even
      // parity after a clear carry, odd after a set one
      const uint32_t cin = __shfl_up_sync(0xffffffffu, cout, 1) & not_first;
      const uint32_t R = both | (zero & (M0 ^ cin));
      if (row < rows) rm[i] = R;
      rup = R;
      cout = (uint32_t)((int)R >> 31);
    }
    return;
  }
  uint32_t rup[2] = {0u, 0u};  // this lane's words of the row above
  uint32_t cout_prev = 0u;
  for (int t = 0; t < steps; t++) {
    uint32_t cin = __shfl_up_sync(0xffffffffu, cout_prev, 1);
    if (lane == 0) cin = 0u;
    const int row = t - lane;
    uint32_t cout = 0u;
    if (row >= 0 && row < h) {
#pragma unroll
      for (int q = 0; q < 2; q++) {
        const int wi = lane * wpl + q;
        if (q < wpl && wi < nw) {
          uint32_t R = 0u;
          if (row > 0) {
            const uint32_t C = am[row * nw + wi] & ~rup[q];
            const uint32_t st = C & ~(C << 1);
            const uint32_t rest = st & ~1u;
            const uint32_t se = (rest & M0) | (cin ? 0u : (st & 1u));
            const uint32_t so = (rest & M1) | (cin ? (st & 1u) : 0u);
            R = ((C & ((C + se) ^ C)) & M0) | ((C & ((C + so) ^ C)) & M1);
          }
          rm[row * nw + wi] = R;
          rup[q] = R;
          cin = R >> 31;
        }
      }
      cout = cin;
    }
    cout_prev = cout;
  }
}

// i / n for 0 <= i < 2^14 and 1 <= n <= 64 without an integer division: (i +
// 0.5) / n lies at least 0.5 / n from every integer, far more than the float
// rounding of (i + 0.5) * (1 / n)
__device__ __forceinline__ int small_div(int i, float inv_n) { return (int)(((float)i + 0.5f) * inv_n); }

// the valid normals of word i (row y, word k of nw) from the code-1 mask and
// the rejections
__device__ __forceinline__ uint32_t valid_word(uint32_t code1, const uint32_t* rm, int i, int y, int k, int nw) {
  const uint32_t left = (rm[i] << 1) | (k > 0 ? rm[i - 1] >> 31 : 0u), up = y > 0 ? rm[i - nw] : 0u;
  return code1 & ~left & ~up;
}

// one block per (session, level) item
__global__ void __launch_bounds__(1024) k_inmap_scan(const BatchTable* __restrict__ bt) {
  extern __shared__ uint32_t mask[];  // [h][nw] of the current item: code 2, then rejections
  __shared__ int wsum[33];
  const int n = bt->n;
  const int total = bt->scan[n];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int item = blockIdx.x; item < total; item += gridDim.x) {
    int l;
    const int slot = find_slot(bt->scan, n, item, l);
    const SessionDev& s = *bt->s[slot];
    const int w = s.lv[l].W, h = s.lv[l].H;
    const int nw = (w + 31) >> 5, nwords = h * nw;
    const uint32_t* __restrict__ src = s.in_amask[l];
    const uint32_t* __restrict__ cm = s.in_cmask[l];
    uint32_t* rm = s.in_rmask[l];
    // the valid normals before each word are counted by all warps: each takes
    // `strips` runs of 32 words, and reads its code-1 words before the sweep
    constexpr int kStrips = kScanSmem / 4 / 1024;
    const int strips = (nwords + 1023) / 1024;
    const int first = warp * strips * 32 + lane;
    const bool staged = nwords * 4 <= kScanSmem;
    uint32_t c1[kStrips];
    if (staged) {
      for (int i = threadIdx.x; i < nwords; i += blockDim.x) mask[i] = src[i];
#pragma unroll
      for (int q = 0; q < kStrips; q++) c1[q] = (q < strips && first + q * 32 < nwords) ? cm[first + q * 32] : 0u;
    }
    __syncthreads();
    if (warp == 0) {
      if (staged)
        scan_level(mask, mask, w, h);
      else
        scan_level(src, rm, w, h);
    }
    __syncthreads();
    const float inv = 1.0f / (float)nw;
    int sum = 0;  // the lane's words
    if (staged) {
#pragma unroll
      for (int q = 0; q < kStrips; q++) {
        const int i = first + q * 32;
        if (q < strips && i < nwords) {
          const int y = small_div(i, inv);
          c1[q] = (uint32_t)__popc(valid_word(c1[q], mask, i, y, i - y * nw, nw));
          sum += (int)c1[q];
          rm[i] = mask[i];
        }
      }
    } else {
      for (int q = 0; q < strips; q++) {
        const int i = first + q * 32;
        if (i < nwords) {
          const int y = i / nw;
          sum += __popc(valid_word(cm[i], rm, i, y, i - y * nw, nw));
        }
      }
    }
    sum = __reduce_add_sync(0xffffffffu, sum);
    if (lane == 0) wsum[warp] = sum;
    __syncthreads();
    int base = 0;  // before the warp's words
    {
      const int v = wsum[lane];
      base = __reduce_add_sync(0xffffffffu, lane < warp ? v : 0);
      const int all = __reduce_add_sync(0xffffffffu, v);
      if (threadIdx.x == 0) s.in_count[l] = (uint32_t)all;
    }
    auto prefix = [&](int i, int c) {
      int v = c;
#pragma unroll
      for (int m = 1; m < 32; m <<= 1) {
        const int o = __shfl_up_sync(0xffffffffu, v, m);
        if (lane >= m) v += o;
      }
      if (i < nwords) s.in_base[l][i] = (uint32_t)(base + v - c);
      base += __shfl_sync(0xffffffffu, v, 31);
    };
    if (staged) {
#pragma unroll
      for (int q = 0; q < kStrips; q++)
        if (q < strips) prefix(first + q * 32, (int)c1[q]);
    } else {
      for (int q = 0; q < strips; q++) {
        const int i = first + q * 32;
        int c = 0;
        if (i < nwords) {
          const int y = i / nw;
          c = __popc(valid_word(cm[i], rm, i, y, i - y * nw, nw));
        }
        prefix(i, c);
      }
    }
    __syncthreads();  // the next item restages the shared masks
  }
}

__global__ void __launch_bounds__(256) k_inmap_post(const BatchTable* __restrict__ bt) {
  const int n = bt->n;
  const int total = bt->imap[n];
  for (int item = blockIdx.x; item < total; item += gridDim.x) {
    int t;
    const int slot = find_slot(bt->imap, n, item, t);
    const SessionDev& s = *bt->s[slot];
    const int l = level_of_tile(s, 32, kMapRows, t);
    const int w = s.lv[l].W, h = s.lv[l].H;
    const int nw = (w + 31) >> 5, ty = t / nw, k = t - ty * nw;
    const int x = k * 32 + threadIdx.x;
    if (x >= w) continue;
    const float K[4] = {s.lv[l].K[0], s.lv[l].K[1], s.lv[l].K[2], s.lv[l].K[3]};
    const uint32_t* __restrict__ rm = s.in_rmask[l];
    const uint32_t* __restrict__ cm = s.in_cmask[l];
    const uint32_t* __restrict__ base = s.in_base[l];
    const float* __restrict__ depth = s.depth[l];
    float4* __restrict__ vtx = s.in_vtx[l];
    float4* __restrict__ nrm = s.in_nrm[l];
    uint32_t* __restrict__ list = s.in_list[l];
    const uint32_t bit = 1u << threadIdx.x;
#pragma unroll 2
    for (int y = ty * kMapRows + threadIdx.y; y < min(h, (ty + 1) * kMapRows); y += 8) {
      // a warp is one 32-pixel word of a row
      const int i = y * nw + k;
      const uint32_t code1 = cm[i];
      const uint32_t valid = valid_word(code1, rm, i, y, k, nw);
      const size_t idx = (size_t)y * w + x;
      const float d = depth[idx];
      float4 v = make_float4(-100.0f, -100.0f, -100.0f, 0.0f);
      if (d > 0.0f && !(rm[i] & bit)) {
        F3 p = back_project((float)x, (float)y, K, d);
        v = make_float4(p.x, p.y, p.z, 1.0f);
      }
      vtx[idx] = v;
      if (code1 & ~valid & bit) nrm[idx] = make_float4(-100.0f, -100.0f, -100.0f, 0.0f);
      if (valid & bit) list[base[i] + __popc(valid & (bit - 1u))] = (uint32_t)((y << 16) | x);
    }
  }
}

}  // namespace

void launch_filter(const BatchTable* bt, cudaStream_t st, int rows, bool ingest) {
  const int grid = sm_count() * 8;
  if (ingest) k_ingest<<<grid, BX * BY, 0, st>>>(bt);
  switch (rows) {
    case 4:
      k_bilateral_batch<4><<<grid * 2, dim3(BX, 4), 0, st>>>(bt);
      break;
    case 16:
      k_bilateral_batch<16><<<grid / 2, dim3(BX, 16), 0, st>>>(bt);
      break;
    default:
      k_bilateral_batch<BY><<<grid, dim3(BX, BY), 0, st>>>(bt);
      break;
  }
  for (int l = 1; l < kMaxLevels; l++) k_pyramid_batch<<<grid, dim3(32, 8), 0, st>>>(bt, l);
}

void launch_input_maps(const BatchTable* bt, cudaStream_t st) {
  const int grid = sm_count() * 8;
  k_inmap_pre<<<grid, dim3(32, 8), 0, st>>>(bt);
  k_inmap_scan<<<kMaxSlots * kMaxLevels, 1024, kScanSmem, st>>>(bt);
  k_inmap_post<<<grid, dim3(32, 8), 0, st>>>(bt);
}

void launch_bilateral_float(const SessionDev& h, const float* in, float* out, cudaStream_t st) {
  const int W = h.lv[0].W, H = h.lv[0].H;
  const int cols = (W + BX - 1) / BX, rows = (H + BY - 1) / BY;
  // One row per thread while its tiles are all resident (six blocks per SM):
  // a thread's chain is half as long, 2.4 instead of 3.3 us for 160x120, 4.4
  // and 4.6 for 512x424 (848 tiles); beyond, two rows: 640x480 5.9 and 5.6 us,
  // 1920x1080 26.9 and 24.3.
  if (cols * rows <= sm_count() * 6)
    k_bilateral_float<1><<<dim3(cols, rows), dim3(BX, BY), 0, st>>>(in, out, W, H);
  else
    k_bilateral_float<kPerThread>
        <<<dim3(cols, (rows + kPerThread - 1) / kPerThread), dim3(BX, BY), 0, st>>>(in, out, W, H);
}

cudaError_t configure_filter_kernels() {
  return cudaFuncSetAttribute(k_inmap_scan, cudaFuncAttributeMaxDynamicSharedMemorySize, kScanSmem);
}

// work-item prefixes of a batch; host_recs are the host copies of the
// session records, dev_recs their device addresses
void fill_batch_table(BatchTable& hb, const SessionDev* const* host_recs, const SessionDev* const* dev_recs, int n,
                      int ray_lx, int bil_rows) {
  std::memset(&hb, 0, sizeof(hb));
  hb.n = n;
  hb.ray_lx = ray_lx;
  hb.bil_rows = (bil_rows == 4 || bil_rows == 16) ? bil_rows : BY;
  const int rx = 1 << ray_lx, ry = 32 >> ray_lx;
  for (int i = 0; i < n; i++) {
    const SessionDev& h = *host_recs[i];
    hb.s[i] = dev_recs[i];
    const bool nm = h.cos_normal > -2.0f;
    int imap = 0, ray = 0;
    for (int l = 0; l < h.levels; l++) {
      const int w = h.lv[l].W, hh = h.lv[l].H;
      imap += ((w + 31) / 32) * ((hh + kMapRows - 1) / kMapRows);
      ray += ((w + rx - 1) / rx) * ((hh + ry - 1) / ry);
    }
    hb.bil[i + 1] = hb.bil[i] + ((h.lv[0].W + BX - 1) / BX) * ((h.lv[0].H + hb.bil_rows - 1) / hb.bil_rows);
    const int fr = hb.bil_rows * kPerThread;
    hb.fil[i + 1] = hb.fil[i] + ((h.lv[0].W + BX - 1) / BX) * ((h.lv[0].H + fr - 1) / fr);
    for (int l = 1; l < kMaxLevels; l++)
      hb.pyr[l - 1][i + 1] =
          hb.pyr[l - 1][i] + (l < h.levels ? ((h.lv[l].W + 31) / 32) * ((h.lv[l].H + 7) / 8) : 0);
    hb.imap[i + 1] = hb.imap[i] + (nm ? imap : 0);
    hb.scan[i + 1] = hb.scan[i] + (nm ? h.levels : 0);
    for (int l = 0; l < kMaxLevels; l++)
      hb.icp[l][i + 1] = hb.icp[l][i] + (l < h.levels ? icp_blocks(h.lv[l].W * h.lv[l].H, l) : 0);
    hb.ray[i + 1] = hb.ray[i] + ray;
    hb.slab[i + 1] = hb.slab[i] + (h.bdist ? h.nb[2] : 0);
  }
}

}  // namespace vs
