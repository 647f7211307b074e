// TSDF ray casting into model depth / vertex / normal maps.
//
// Reference: g_rmi_Render_Maps_for_ICP, d_crtc_Cast_Ray_on_TSDF_Cube_NEW,
// d_gtvu / d_gtvi and d_csnt (STAC/Engine/GPU/z_yooji_cuda_tsdf_renderer.cu:
// 1069-1209, 466-635, 68-153, 288-464; host set-up :1642-1700).  The
// reference launches one 16x16-block grid per pyramid level; here one
// persistent launch (k_ray_fused) covers every level of every session of a
// batch table, marching each ray to its surface point and computing the
// surface normal and the maps there.  Colour ray-casts, whose shading needs
// more registers, run as two launches: k_ray_march writes the surface points
// to a hit buffer and k_ray_shade shades them.  Each warp takes 8x4-ray tiles
// from an atomic work counter, so a slow tile near a surface holds up neither
// a grid row nor the other warps of its block.  A ray keeps its whole march
// state in registers, and every voxel read is one 32-bit word that carries
// both the TSDF value and the weight (one gather instead of the reference's
// separate float and uchar arrays).  Before the march, the distance field of
// the band sub-cubes is rebuilt (k_band), which lets the march
// jump through free space.
//
// The reference's march loop has no iteration bound: a fine-search ray whose
// signed steps keep changing direction never leaves it.  The loop here ends
// after 4 * (2 r_cube / voxel) + 64 steps and reports no hit; the CPU oracle
// applies the same bound.
#include <cuda_runtime.h>
#include <stdint.h>

#include "vs_internal.cuh"

namespace vs {
namespace {

constexpr int kRayThreads = 128;  // a warp's 32 rays form a (1 << lx) x (32 >> lx) tile

struct RayArgs {
  const BatchTable* bt;
  unsigned* work;       // [0] next tile, [1] finished warps; zero between launches
  int level;            // < 0: every level of every slot into the model maps
  // explicit poses and outputs of a one-level, one-slot call (reference layout)
  const float* Tgc;
  const float* Tcg;
  float center[3];
  float light[3];
  int gate;
  float* out_depth;
  float* out_vtx3;
  float* out_nrm3;
  uint8_t* out_img;
  uint8_t* out_rgb;     // planar colour image (NULL: none)
  int mode;             // kRay* bits of the external render variants (0: the ICP maps)
};

// Volume reads.  Every voxel read is one word (TSDF value and weight); a
// voxel never written holds weight 0 and reads "no value".  Free space is
// skipped through the band distance field, so the samples the march does take
// lie near band bricks, where a separate occupancy test would only add
// instructions.
template <class S>
struct Vol {
  const typename S::word* v;
  const uint8_t* bdist;  // distance in bricks to the nearest band brick
  float dim[3];
  uint32_t nbx, nbxy;  // bricks per row / per slab
  uint32_t sy, sz;  // word strides of one brick row / one brick slab: 512 nb[0], 512 nb[0] nb[1]
  // The word index of voxel (x, y, z) >= 0 is the sum of one term per axis
  // (brick part + offset inside the brick), in 32 bits (volumes of at most
  // 1024^3 voxels have fewer than 2^30 words).  Stencils compute each axis
  // term once and add them.
  __device__ inline uint32_t wx(int x) const { return (((uint32_t)x >> 3) << 9) + ((uint32_t)x & 7u); }
  __device__ inline uint32_t wy(int y) const { return ((uint32_t)y >> 3) * sy + (((uint32_t)y & 7u) << 3); }
  __device__ inline uint32_t wz(int z) const { return ((uint32_t)z >> 3) * sz + (((uint32_t)z & 7u) << 6); }
  // the value of word i, and whether its weight is > 0
  __device__ inline bool word_ok(uint32_t i, float& t) const {
    const typename S::word u = __ldg(v + i);
    t = S::value(u);
    return S::weighted(u);
  }
  // The nearest voxel of p (ROUNDF), and whether it is in range.  ROUNDF(p) is
  // negative for every p <= -0.5 and equals (int)(p + 0.5) for every p > -0.5
  // (both branches give 0 on (-0.5, 0)), so one comparison per coordinate
  // decides the lower bound, and a NaN coordinate fails it too; the integer
  // part of p + 0.5 is below dim iff p + 0.5 is.
  struct Near {
    int x, y, z;
    bool in;
  };
  __device__ inline Near nearest(F3 p) const {
    const float x = p.x + 0.5f, y = p.y + 0.5f, z = p.z + 0.5f;
    Near v;
    v.in = p.x > -0.5f && p.y > -0.5f && p.z > -0.5f && x < dim[0] && y < dim[1] && z < dim[2];
    v.x = (int)x, v.y = (int)y, v.z = (int)z;
    return v;
  }
  // d_gtvu_Get_TSDF_Value_Uninterpolated: nearest voxel, weight > 0
  __device__ inline bool gtvu(const Near& v, float& out) const {
    out = 1.0f;
    float t;
    if (!v.in || !word_ok(wx(v.x) + wy(v.y) + wz(v.z), t)) return false;
    out = t;
    return true;
  }
  // Free-space run: how many of the next steps p + k inc (k = 1..m) are
  // certain to read TSDF 1 ("no value", or a voxel whose value is 1) -
  // outside the volume, or inside the box of bricks that holds no band brick
  // (the bricks within Chebyshev distance bdist - 1 of a position's brick) -
  // so that the march only has to advance the position for them.  Boxes are
  // chained: the step after a box joins the run when it certainly reads 1
  // too, and the next box starts there.  The bounds are pulled in by 0.05
  // voxel, far more than the rounding of a position p + k inc (one product
  // and one sum: under 1e-3 voxel wherever both p and the position lie within
  // 2048 voxels of the volume) or of the approximate reciprocals of the
  // increment, so a step counted here reads 1 however its position rounds.  A negative result -k
  // says p lies in a band brick that the ray leaves after about k steps; the
  // caller need not ask again before then (asking late only delays a run, it
  // never changes a sample).  A NaN coordinate fails every comparison below
  // and gives 0.
  static constexpr int kMaxRun = 4096;
  static constexpr int kMaxBoxes = 2;
  __device__ inline int free_run(F3 p, F3 inc, const Near& near) const {
    const float d = 0.05f;
    const float pa[3] = {p.x, p.y, p.z}, ia[3] = {inc.x, inc.y, inc.z};
    const float ra[3] = {rcp_approx(inc.x), rcp_approx(inc.y), rcp_approx(inc.z)};
    int run = 0;
#pragma unroll
    for (int j = 0; j < kMaxBoxes; j++) {
      // q: step `run` (j = 0: the current sample, which read 1; after that
      // the step following the last box, a candidate for the run)
      float q[3];
#pragma unroll
      for (int a = 0; a < 3; a++) q[a] = j == 0 ? pa[a] : (float)run * ia[a] + pa[a];
      const Near v = j == 0 ? near : nearest(f3(q[0], q[1], q[2]));
      float t;
      bool band = false, sure = false;  // sure: q reads 1 however it rounds
      if (!v.in) {
        // outside until every coordinate that is out of range has come in
        t = 0.0f;
#pragma unroll
        for (int a = 0; a < 3; a++) {
          const float hi = dim[a] - 0.5f;
          if (q[a] <= -0.5f) {
            t = fmaxf(t, ia[a] > 0.0f ? (-0.5f - d - q[a]) * ra[a] : 1e30f);
            sure |= q[a] < -0.5f - d;
          } else if (q[a] >= hi) {
            t = fmaxf(t, ia[a] < 0.0f ? (hi + d - q[a]) * ra[a] : 1e30f);
            sure |= q[a] > hi + d;
          }
        }
      } else {
        // brick b holds the nearest voxel, and the box of bricks b - h .. b + h
        // (h = bdist - 1) holds no band brick; in a band brick (bdist
        // 0) the box is the brick itself.  (The box bounds are halves, exact.)
        const int b[3] = {v.x >> 3, v.y >> 3, v.z >> 3};
        const int dist = __ldg(bdist + (uint32_t)b[2] * nbxy + (uint32_t)b[1] * nbx + (uint32_t)b[0]);
        band = dist == 0;
        sure = !band;
        const float h = band ? 0.0f : (float)(dist - 1), h1 = h + 1.0f;
        t = 1e30f;
#pragma unroll
        for (int a = 0; a < 3; a++) {
          const float bf = (float)b[a];
          const float lo = fmaf(bf - h, 8.0f, -0.5f) + d, hi = fmaf(bf + h1, 8.0f, -0.5f) - d;
          sure &= q[a] > lo && q[a] < hi;
          const float u = ((ia[a] > 0.0f ? hi : lo) - q[a]) * ra[a];
          if (ia[a] != 0.0f) t = fminf(t, u);
        }
      }
      if (j > 0 && !sure) return run - 1;
      // steps k >= 1 from q with k < t: ceil(t) - 1
      t = fminf(t, (float)(kMaxRun + 1));
      const int m = max(__float2int_ru(t), 1) - 1;
      if (j == 0 && band) return -m;
      run += m;
      if (run >= kMaxRun) return run;
      run++;  // the next candidate
    }
    return run - 1;
  }

  // d_gtvi_Get_TSDF_Value_Interpolated (offset = floor, see the oracle); the
  // eight reads have no side effects, so reading all of them before the
  // validity test gives the short-circuit form's result
  __device__ inline bool gtvi(F3 p, float& out) const {
    out = 1.0f;
    // the eight corners floor(p), floor(p) + 1 are in range iff 0 <= p < dim - 1
    // (false for a NaN)
    if (!(p.x >= 0.0f && p.x < dim[0] - 1.0f && p.y >= 0.0f && p.y < dim[1] - 1.0f && p.z >= 0.0f &&
          p.z < dim[2] - 1.0f))
      return false;
    const int cx = (int)p.x, cy = (int)p.y, cz = (int)p.z;
    const float rx = p.x - (float)cx, ry = p.y - (float)cy, rz = p.z - (float)cz;
    bool ok = true;
    const uint32_t x0 = wx(cx), x1 = wx(cx + 1), y0 = wy(cy), y1 = wy(cy + 1), z0 = wz(cz), z1 = wz(cz + 1);
    float f0, f1, f2, f3_, b0, b1, b2, b3;
    ok &= word_ok(z0 + y0 + x0, f0);
    ok &= word_ok(z0 + y0 + x1, f1);
    ok &= word_ok(z0 + y1 + x0, f2);
    ok &= word_ok(z0 + y1 + x1, f3_);
    ok &= word_ok(z1 + y0 + x0, b0);
    ok &= word_ok(z1 + y0 + x1, b1);
    ok &= word_ok(z1 + y1 + x0, b2);
    ok &= word_ok(z1 + y1 + x1, b3);
    if (!ok) return false;
    float inf = (1.0f - ry) * ((1.0f - rx) * f0 + rx * f1) + ry * ((1.0f - rx) * f2 + rx * f3_);
    float inb = (1.0f - ry) * ((1.0f - rx) * b0 + rx * b1) + ry * ((1.0f - rx) * b2 + rx * b3);
    out = (1.0f - rz) * inf + rz * inb;
    return true;
  }
};

// d_csnt_Compute_Surface_Normal_from_TSDF: gradient of the trilinear field from
// a 4 + 12 + 12 + 4 voxel stencil
template <class S>
__device__ bool surface_normal(const Vol<S>& V, const SessionDev& s, F3 p3d, F3& nout) {
  F3 vox;
  if (!pos_in_voxel(p3d, s, vox)) return false;
  // the stencil spans floor(v) - 1 .. floor(v) + 2 on every axis and uses each
  // of those values, so it is in range iff 1 <= v < dim - 2 (false for a NaN)
  if (!(vox.x >= 1.0f && vox.x < V.dim[0] - 2.0f && vox.y >= 1.0f && vox.y < V.dim[1] - 2.0f && vox.z >= 1.0f &&
        vox.z < V.dim[2] - 2.0f))
    return false;
  const int cx = (int)vox.x, cy = (int)vox.y, cz = (int)vox.z;
  const float rx = vox.x - (float)cx, ry = vox.y - (float)cy, rz = vox.z - (float)cz;
  const int dx1[4] = {0, 1, 0, 1}, dy1[4] = {0, 0, 1, 1};
  const int dx2[12] = {0, 1, -1, 0, 1, 2, -1, 0, 1, 2, 0, 1};
  const int dy2[12] = {-1, -1, 0, 0, 0, 0, 1, 1, 1, 1, 2, 2};
  // all 32 reads are issued before any validity test (no side effects, so
  // the result equals the reference's read-and-return-early order)
  bool ok = true;
  uint32_t X[4], Y[4], Z[4];
#pragma unroll
  for (int k = 0; k < 4; k++) X[k] = V.wx(cx - 1 + k), Y[k] = V.wy(cy - 1 + k), Z[k] = V.wz(cz - 1 + k);
  float fm[4], fr[12], bk[12], bm[4];
#pragma unroll
  for (int i = 0; i < 4; i++) ok &= V.word_ok(Z[0] + Y[1 + dy1[i]] + X[1 + dx1[i]], fm[i]);
#pragma unroll
  for (int i = 0; i < 12; i++) ok &= V.word_ok(Z[1] + Y[1 + dy2[i]] + X[1 + dx2[i]], fr[i]);
#pragma unroll
  for (int i = 0; i < 12; i++) ok &= V.word_ok(Z[2] + Y[1 + dy2[i]] + X[1 + dx2[i]], bk[i]);
#pragma unroll
  for (int i = 0; i < 4; i++) ok &= V.word_ok(Z[3] + Y[1 + dy1[i]] + X[1 + dx1[i]], bm[i]);
  if (!ok) return false;
  float a4[4], b4[4], a2[2], b2[2], gx, gy, gz;
  a4[0] = (1.0f - rz) * fr[2] + rz * bk[2];
  a4[1] = (1.0f - rz) * fr[3] + rz * bk[3];
  a4[2] = (1.0f - rz) * fr[4] + rz * bk[4];
  a4[3] = (1.0f - rz) * fr[5] + rz * bk[5];
  b4[0] = (1.0f - rz) * fr[6] + rz * bk[6];
  b4[1] = (1.0f - rz) * fr[7] + rz * bk[7];
  b4[2] = (1.0f - rz) * fr[8] + rz * bk[8];
  b4[3] = (1.0f - rz) * fr[9] + rz * bk[9];
  a2[0] = (1.0f - rx) * a4[0] + rx * a4[1];
  a2[1] = (1.0f - rx) * b4[0] + rx * b4[1];
  b2[0] = (1.0f - rx) * a4[2] + rx * a4[3];
  b2[1] = (1.0f - rx) * b4[2] + rx * b4[3];
  gx = (1.0f - ry) * b2[0] + ry * b2[1];
  gx -= (1.0f - ry) * a2[0] + ry * a2[1];
  a4[0] = (1.0f - rz) * fr[0] + rz * bk[0];
  a4[1] = (1.0f - rz) * fr[3] + rz * bk[3];
  a4[2] = (1.0f - rz) * fr[7] + rz * bk[7];
  a4[3] = (1.0f - rz) * fr[10] + rz * bk[10];
  b4[0] = (1.0f - rz) * fr[1] + rz * bk[1];
  b4[1] = (1.0f - rz) * fr[4] + rz * bk[4];
  b4[2] = (1.0f - rz) * fr[8] + rz * bk[8];
  b4[3] = (1.0f - rz) * fr[11] + rz * bk[11];
  a2[0] = (1.0f - ry) * a4[0] + ry * a4[1];
  a2[1] = (1.0f - ry) * b4[0] + ry * b4[1];
  b2[0] = (1.0f - ry) * a4[2] + ry * a4[3];
  b2[1] = (1.0f - ry) * b4[2] + ry * b4[3];
  gy = (1.0f - rx) * b2[0] + rx * b2[1];
  gy -= (1.0f - rx) * a2[0] + rx * a2[1];
  a4[0] = (1.0f - ry) * fm[0] + ry * fm[2];
  a4[1] = (1.0f - ry) * fr[3] + ry * fr[7];
  a4[2] = (1.0f - ry) * bk[3] + ry * bk[7];
  a4[3] = (1.0f - ry) * bm[0] + ry * bm[2];
  b4[0] = (1.0f - ry) * fm[1] + ry * fm[3];
  b4[1] = (1.0f - ry) * fr[4] + ry * fr[8];
  b4[2] = (1.0f - ry) * bk[4] + ry * bk[8];
  b4[3] = (1.0f - ry) * bm[1] + ry * bm[3];
  a2[0] = (1.0f - rz) * a4[0] + rz * a4[1];
  a2[1] = (1.0f - rz) * b4[0] + rz * b4[1];
  b2[0] = (1.0f - rz) * a4[2] + rz * a4[3];
  b2[1] = (1.0f - rz) * b4[2] + rz * b4[3];
  gz = (1.0f - rx) * b2[0] + rx * b2[1];
  gz -= (1.0f - rx) * a2[0] + rx * a2[1];
  if (gx == 0.0f && gy == 0.0f && gz == 0.0f) return false;
  nout = normalised(f3(gx, gy, gz));
  return true;
}

// What every ray of one level of one session has in common, in shared memory
// per warp: formed when the warp's tiles come to another level or session
// instead of by each lane for its ray (a tenth of a ray's instructions).
struct TileCam {
  float Tcg[12], Tgc[12];
  F3 cam;             // camera centre
  float theta_max;    // half angle of the cube's view cone
  F3 ncc;             // direction of the cube's centre
  float dmin, dmax;   // the marched segment
  float K[4];
  float step_scale, total_max;  // full step and length of the march, in voxels
};

// The state of a march
struct March {
  F3 vs;          // position in voxels
  float total;    // distance marched
  float tsdf;     // the sample there
  int state;
  int recheck;    // full steps before the next free-space test
};
enum { COARSE, FINE, BEHIND };
enum { kMarchMiss, kMarchZero, kMarchBehind, kMarchLong };

__device__ __forceinline__ bool same_bits(float a, float b) { return __float_as_uint(a) == __float_as_uint(b); }
// Whether two states take the same samples from here on: the next position,
// sample and search state follow from these alone (a recheck of 0 or less is
// due).  The distance and the iteration count differ, but all they can do is
// end the march without a hit.
__device__ __forceinline__ bool same_course(const March& a, const March& b) {
  return same_bits(a.vs.x, b.vs.x) && same_bits(a.vs.y, b.vs.y) && same_bits(a.vs.z, b.vs.z) &&
         same_bits(a.tsdf, b.tsdf) && a.state == b.state && max(a.recheck, 0) == max(b.recheck, 0);
}

// The march loop: kMarchMiss, kMarchZero (the sample is 0 at m.vs) or
// kMarchBehind (the sample is behind the surface).  left: the steps left
// before the iteration cap (those of free-space runs included).
//
// A fine-search ray whose signed steps return it to where it was repeats
// itself until the iteration cap ends it without a hit: some 2700 turns in a
// 384^3 volume, a millisecond that the whole launch waits for, on one ray in
// ten million.  A ray still marching after kLongTurns turns (the usual one
// takes 8, the longest regular ones about 60) goes on in the LONG form, which
// keeps an earlier state (the one at the last power of two of its turns, R.
// Brent, BIT 20, 1980) and ends the ray when it comes back to it.  An
// integration and ray-cast of a 512x424 view into 384^3 that had such rays in
// some frames took 290 to 680 us on average, and 160 us now as without them.
//
// Bound by instruction issue: about 65 instructions a turn and 160 a
// free-space run, which six of eight turns compute.  The two boxes of a run
// unrolled, the sample's nearest voxel shared with the run, reciprocal
// approximations and the view's constants per tile took the ray-cast stage of
// the 64-session step from 2.06 to 1.88 ms (of sixteen sessions 0.522 to
// 0.475).  (Additions that round instead of conversions between float and
// integer were slower, 2.21 ms: a conversion is one issue slot.)
constexpr int kLongTurns = 64;
template <class S, bool LONG>
__device__ __forceinline__ int march_loop(const Vol<S>& V, F3 rd, float step_scale, float total_max, March& m, int& left) {
  March kept = m;
  for (int turns = 0; LONG || turns < kLongTurns; turns++) {
    if (LONG) {
      if (turns && same_course(m, kept)) return kMarchMiss;
      if ((turns & (turns - 1)) == 0) kept = m;
    }
    if (--left < 0) return kMarchMiss;
    float step;
    if (m.state == COARSE)
      step = step_scale;
    else
      step = (m.tsdf > 0.0f) ? fmaxf(step_scale * m.tsdf, 1.0f) : fminf(step_scale * m.tsdf, -1.0f);
    m.vs = add(m.vs, scale(step, rd));
    m.total += step;
    if (m.total > total_max) return kMarchMiss;
    const typename Vol<S>::Near near = V.nearest(m.vs);
    V.gtvu(near, m.tsdf);
    if (m.tsdf > -1.0f && m.tsdf < 1.0f) {
      V.gtvi(m.vs, m.tsdf);
      if (m.tsdf < 0.0f) return m.state == COARSE ? kMarchMiss : kMarchBehind;
      if (m.tsdf == 0.0f) return kMarchZero;
      if (m.state == COARSE) m.state = FINE;
    }
    if (m.tsdf == 1.0f && --m.recheck < 0) {
      // While samples read TSDF 1 (no value, or a voxel whose value is 1) the
      // state and the step stay as they are, so the `run` steps of a
      // free-space run are taken at once: p + run * inc and total + run * sn.
      // The step-by-step sums of the reference round after every step; the
      // jump rounds once, so the position after a run of m steps differs
      // from theirs by at most about m / 2 ulps of the voxel coordinate
      // (under 1e-2 voxel for runs of a few hundred steps and coordinates
      // below 1024), which moves the later samples and the surface point by
      // far less than the 1 mm ray-cast tolerance.
      const float sn = (m.state == COARSE) ? step_scale : fmaxf(step_scale * m.tsdf, 1.0f);
      const F3 inc = scale(sn, rd);
      int k = V.free_run(m.vs, inc, near);
      if (k < 0) {
        m.recheck = -k;
        k = 0;
      }
      // the loop above would stop one step past the cap: run at most `left`
      // steps here, then stop as it would.  total only grows (sn > 0), so it
      // passed total_max inside the run iff it is past it at the end, and the
      // ray then ends without a hit whichever step it was.
      const bool capped = k > left;
      const int run = capped ? left : k;
      if (run > 0) {
        const float fr = (float)run;
        m.vs = add(m.vs, scale(fr, inc));
        m.total += fr * sn;
      }
      if (m.total > total_max) return kMarchMiss;
      if (capped) return kMarchMiss;
      left -= run;
    }
  }
  return kMarchLong;
}

// out of line: its registers are not the usual ray's
template <class S>
__device__ __noinline__ int march_long(const Vol<S>& V, F3 rd, float step_scale, float total_max, March& m, int left) {
  return march_loop<S, true>(V, rd, step_scale, total_max, m, left);
}

template <class S, bool SCENE>
__device__ bool cast_ray(const Vol<S>& V, const SessionDev& s, const TileCam& c, float px, float py, F3& p3d) {
  const F3 pe = transform(back_project(px, py, c.K, c.dmax), c.Tcg);
  const F3 rd = normalised(sub(pe, c.cam));
  if (!SCENE) {
    const float theta = acosf(dot(rd, c.ncc));
    if (theta > c.theta_max) return false;
  }
  const F3 ps = add(c.cam, scale(c.dmin, rd));
  const float step_scale = c.step_scale, total_max = c.total_max;
  March m;
  m.total = 0.0f;
  m.recheck = 0;
  pos_in_voxel(ps, s, m.vs);
  if (!V.gtvu(V.nearest(m.vs), m.tsdf))
    m.state = COARSE;
  else if (m.tsdf >= 0.0f)
    m.state = FINE;
  else
    return false;
  int left = 4 * (int)total_max + 64;
  int end = march_loop<S, false>(V, rd, step_scale, total_max, m, left);
  if (end == kMarchLong) {
    March far = m;
    end = march_long<S>(V, rd, step_scale, total_max, far, left);
    m.vs = far.vs, m.tsdf = far.tsdf;
  }
  if (end == kMarchZero) {
    p3d = pos_in_world(m.vs, s);
    return true;
  }
  if (end == kMarchBehind) {
    float step = step_scale * m.tsdf;
    F3 vs = add(m.vs, scale(step, rd));
    float tsdf;
    V.gtvi(vs, tsdf);
    step = step_scale * tsdf;
    vs = add(vs, scale(step, rd));
    p3d = pos_in_world(vs, s);
    return true;
  }
  return false;
}

// tiles of (1 << lx) x (32 >> lx) rays of level l
__device__ inline int ray_tiles(const SessionDev& s, int l, int lx) {
  return ((s.lv[l].W + (1 << lx) - 1) >> lx) * ((s.lv[l].H + (32 >> lx) - 1) >> (5 - lx));
}

template <bool SCENE>
__device__ inline void load_tile_cam(const RayArgs& a, const SessionDev& s, int l, TileCam& c) {
  const int lane = threadIdx.x & 31;
  const bool ext = a.level >= 0;
  const float* Tcg = ext ? a.Tcg : s.pose->Tcg;
  const float* Tgc = ext ? a.Tgc : s.pose->Tgc;
  const F3 cam = ext ? f3(a.center[0], a.center[1], a.center[2])
                     : f3(s.pose->center[0], s.pose->center[1], s.pose->center[2]);
  // host-side set-up of rmi_Render_Maps_for_ICP (:1667-1675)
  const F3 cc = f3(s.cube_center[0], s.cube_center[1], s.cube_center[2]);
  const F3 vcc = sub(cc, cam);
  const F3 ncc = normalised(vcc);
  const float dist_cc = length(vcc);
  const float theta_max = asinf(s.r_cube / dist_cc);
  __syncwarp();  // the previous tile's rays have read theirs
  if (lane < 12) c.Tcg[lane] = Tcg[lane], c.Tgc[lane] = Tgc[lane];
  if (lane < 4) c.K[lane] = s.lv[l].K[lane];
  if (lane == 0) {
    c.cam = cam;
    c.theta_max = theta_max;
    c.ncc = ncc;
    // object mode (d_crtc_NEW, :466-635): the segment of the ray through the
    // cube's bounding sphere inside its view cone; scene mode (d_crtcs,
    // :908-1066): from the camera centre to 2 r_cube, no cone
    c.dmin = SCENE ? 0.0f : dist_cc - s.r_cube;
    c.dmax = SCENE ? 2.0f * s.r_cube : dist_cc + s.r_cube;
    c.step_scale = 0.9f * s.mu * s.vox_inv;
    c.total_max = 2.0f * s.r_cube * s.vox_inv;
  }
  __syncwarp();
}

// Hands the calling warp ray tiles until none are left and calls
// f(session, level, x, y, camera) for each lane's pixel inside its level.  The
// last warp to finish clears the counters for the next launch.
template <bool SCENE, class F>
__device__ inline void for_each_ray_tile(const RayArgs& a, F&& f) {
  __shared__ TileCam cams[kRayThreads / 32];
  TileCam& cam = cams[threadIdx.x >> 5];
  const BatchTable* __restrict__ bt = a.bt;
  const int lane = threadIdx.x & 31;
  const int n = bt->n;
  const int lx = bt->ray_lx, rx = 1 << lx;
  const int total = (a.level >= 0) ? ray_tiles(*bt->s[0], a.level, lx) : bt->ray[n];
  int loaded = -1;  // slot and level of cam
  for (;;) {
    int item = 0;
    if (lane == 0) item = (int)atomicAdd(a.work, 1u);
    item = __shfl_sync(0xffffffffu, item, 0);
    if (item >= total) break;
    int t, l, slot;
    if (a.level >= 0) {
      slot = 0;
      l = a.level;
      t = item;
    } else {
      slot = find_slot(bt->ray, n, item, t);
      const SessionDev& s = *bt->s[slot];
      l = 0;
      for (; l < s.levels - 1; l++) {
        const int nt = ray_tiles(s, l, lx);
        if (t < nt) break;
        t -= nt;
      }
    }
    const SessionDev& s = *bt->s[slot];
    if (a.gate && s.pose->failed) continue;
    if (loaded != slot * kMaxLevels + l) {
      loaded = slot * kMaxLevels + l;
      load_tile_cam<SCENE>(a, s, l, cam);
    }
    const int tw = (s.lv[l].W + rx - 1) >> lx, ty = t / tw;
    const int x = ((t - ty * tw) << lx) + (lane & (rx - 1)), y = (ty << (5 - lx)) + (lane >> lx);
    if (x < s.lv[l].W && y < s.lv[l].H) f(s, l, x, y, cam);
  }
  if (lane == 0) {
    __threadfence();
    const unsigned warps = gridDim.x * (blockDim.x >> 5);
    if (atomicAdd(a.work + 1, 1u) == warps - 1) {
      a.work[0] = 0u;
      a.work[1] = 0u;
      __threadfence();
    }
  }
}

// offset of level l's pixels in the per-session hit buffer
__device__ inline size_t hit_offset(const SessionDev& s, int l) {
  size_t o = 0;
  for (int k = 0; k < l; k++) o += (size_t)s.lv[k].W * s.lv[k].H;
  return o;
}

template <class S>
__device__ inline Vol<S> volume_of(const SessionDev& s) {
  Vol<S> V;
  V.v = reinterpret_cast<const typename S::word*>(s.vol);
  V.bdist = s.bdist;
  for (int k = 0; k < 3; k++) V.dim[k] = (float)s.dim[k];
  V.nbx = (uint32_t)s.nb[0];
  V.nbxy = (uint32_t)s.nb[0] * (uint32_t)s.nb[1];
  V.sy = (uint32_t)s.nb[0] << 9;
  V.sz = ((uint32_t)s.nb[0] * (uint32_t)s.nb[1]) << 9;
  return V;
}

// Band distance field: the Chebyshev distance in bricks to the nearest band
// brick, saturating at kBandReach + 1.  The bricks within distance k of a band
// brick are the band dilated by a cube of half-width k, so the distance of a
// brick is the number of k in 0..kBandReach whose dilation leaves it out.  One
// block per z slab: the band flags of the slabs within reach as bits, a word
// per 32 bricks of a row; for every k the OR over the slabs, then the rows,
// then the shifts within k; and the distances back as bytes.  Bound by the
// latency of its six steps: 64 x 64 x 64 bricks take 5.5 us (4.8 in blocks of
// 1024 threads, which halve the slabs in flight: 32 sessions 55 us instead of
// 38), 40 and 41 bricks a side 4.8 and 6.0.  Two passes over bytes (the x and
// y windows of a slab, then the z windows of a row, 15 compares a brick each)
// took 7.9 + 5.4 and 59 + 24 (the two sizes 7.8 and 8.0).
constexpr int kBandThreads = 512;
constexpr int kBandSlabs = 2 * kBandReach + 1;
constexpr int kBandWords = kMaxBricksAxis / 32 * kMaxBricksAxis;  // most words of a slab

// i / n for 0 <= i < 2^14 and 1 <= n <= 2^9 without an integer division:
// (i + 0.5) / n lies at least 0.5 / n from every integer, far more than the
// float rounding of (i + 0.5) * (1 / n)
__device__ inline int small_div(int i, float inv_n) { return (int)(((float)i + 0.5f) * inv_n); }

// four bytes of 0 or 1 -> four bits, first byte lowest
__device__ __forceinline__ uint32_t pack4(uint32_t v) { return (v * 0x10204080u) >> 28; }
__device__ __forceinline__ uint32_t unpack4(uint32_t bits) { return (bits * 0x00204081u) & 0x01010101u; }

__global__ void __launch_bounds__(kBandThreads) k_band(const BatchTable* __restrict__ bt) {
  // the slabs' bits, then (k - 1) the OR over the rows; the OR over the slabs, then the dilation
  __shared__ uint32_t B[kBandSlabs][kBandWords], D[kBandReach][kBandWords];
  const int n = bt->n;
  const int total = bt->slab[n];
  for (int item = blockIdx.x; item < total; item += gridDim.x) {
    int z;
    const SessionDev* __restrict__ s = bt->s[find_slot(bt->slab, n, item, z)];
    const int nb0 = s->nb[0], nb1 = s->nb[1], nb2 = s->nb[2], np = nb0 * nb1;
    const int nw = (nb0 + 31) >> 5, words = nb1 * nw;
    const float inv_words = 1.0f / (float)words, inv_nw = 1.0f / (float)nw;
    const uint8_t* __restrict__ band = s->band;
    __syncthreads();  // the previous slab's reads are done
    // a thread per word; its flags in the widest reads that the rows' length
    // aligns, all in flight together
    for (int i = threadIdx.x; i < kBandSlabs * words; i += kBandThreads) {
      const int dz = small_div(i, inv_words), w = i - dz * words, zz = z + dz - kBandReach;
      uint32_t bits = 0u;
      if (zz >= 0 && zz < nb2) {
        const int y = small_div(w, inv_nw), x = (w - y * nw) * 32, left = nb0 - x;
        const uint8_t* __restrict__ src = band + (size_t)zz * np + y * nb0 + x;
        if (nb0 % 16 == 0) {
          const uint4 a = reinterpret_cast<const uint4*>(src)[0];
          bits = pack4(a.x) | pack4(a.y) << 4 | pack4(a.z) << 8 | pack4(a.w) << 12;
          if (left > 16) {
            const uint4 b = reinterpret_cast<const uint4*>(src)[1];
            bits |= (pack4(b.x) | pack4(b.y) << 4 | pack4(b.z) << 8 | pack4(b.w) << 12) << 16;
          }
        } else if (nb0 % 4 == 0) {
#pragma unroll
          for (int k = 0; k < 8; k++)
            if (4 * k < left) bits |= pack4(reinterpret_cast<const uint32_t*>(src)[k]) << (4 * k);
        } else {
#pragma unroll
          for (int k = 0; k < 32; k++)
            if (k < left) bits |= (uint32_t)src[k] << k;
        }
      }
      B[dz][w] = bits;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kBandReach * words; i += kBandThreads) {
      const int k = small_div(i, inv_words) + 1, w = i - (k - 1) * words;
      uint32_t v = B[kBandReach][w];
      for (int d = 1; d <= k; d++) v |= B[kBandReach - d][w] | B[kBandReach + d][w];
      D[k - 1][w] = v;
    }
    __syncthreads();
    uint32_t own = 0u;  // the slab's own bits: B is overwritten
    if (threadIdx.x < words) own = B[kBandReach][threadIdx.x];
    __syncthreads();
    for (int i = threadIdx.x; i < kBandReach * words; i += kBandThreads) {
      const int k = small_div(i, inv_words) + 1, w = i - (k - 1) * words, y = small_div(w, inv_nw);
      const uint32_t* src = D[k - 1] + (w - y * nw);
      uint32_t v = 0u;
      for (int q = max(y - k, 0); q <= min(y + k, nb1 - 1); q++) v |= src[q * nw];
      B[k][w] = v;
    }
    if (threadIdx.x < words) B[0][threadIdx.x] = own;
    __syncthreads();
    for (int i = threadIdx.x; i < kBandReach * words; i += kBandThreads) {
      const int k = small_div(i, inv_words) + 1, w = i - (k - 1) * words, x = w - small_div(w, inv_nw) * nw;
      const uint32_t v = B[k][w], lo = x > 0 ? B[k][w - 1] : 0u, hi = x + 1 < nw ? B[k][w + 1] : 0u;
      uint32_t o = v;
      for (int d = 1; d <= k; d++) o |= __funnelshift_l(lo, v, d) | __funnelshift_r(v, hi, d);
      D[k - 1][w] = o;
    }
    __syncthreads();
    uint8_t* __restrict__ out = s->bdist + (size_t)z * np;
    if (nb0 % 4 == 0) {
      const float inv = 4.0f / (float)nb0;
      for (int i = threadIdx.x; i < np / 4; i += kBandThreads) {
        const int y = small_div(i, inv), x = i * 4 - y * nb0, w = y * nw + (x >> 5), sh = x & 31;
        uint32_t left = 0x08080808u - unpack4((B[0][w] >> sh) & 15u);
#pragma unroll
        for (int k = 0; k < kBandReach; k++) left -= unpack4((D[k][w] >> sh) & 15u);
        reinterpret_cast<uint32_t*>(out)[i] = left;
      }
    } else {
      const float inv = 1.0f / (float)nb0;
      for (int i = threadIdx.x; i < np; i += kBandThreads) {
        const int y = small_div(i, inv), x = i - y * nb0, w = y * nw + (x >> 5), sh = x & 31;
        uint32_t left = 8u - ((B[0][w] >> sh) & 1u);
#pragma unroll
        for (int k = 0; k < kBandReach; k++) left -= (D[k][w] >> sh) & 1u;
        out[i] = (uint8_t)left;
      }
    }
  }
}
static_assert(kBandReach == 7, "a brick's distance counts eight dilations");
static_assert(kBandWords <= kBandThreads && kBandSlabs * kBandWords < (1 << 14), "one word per thread; small_div");

#ifndef VS_RAY_MIN_BLOCKS
#define VS_RAY_MIN_BLOCKS 8  // resident 128-thread blocks per SM the register allocation must allow
#endif
#ifndef VS_SHADE_MIN_BLOCKS
#define VS_SHADE_MIN_BLOCKS 8
#endif

// phase 1: march every ray to its surface point (global coordinates; w = 1
// hit, 0 none) in the session's hit buffer
template <class S, bool SCENE>
__global__ void __launch_bounds__(kRayThreads, VS_RAY_MIN_BLOCKS) k_ray_march(RayArgs a) {
  for_each_ray_tile<SCENE>(a, [&](const SessionDev& s, int l, int x, int y, const TileCam& c) {
    F3 pg;
    const bool hit = cast_ray<S, SCENE>(volume_of<S>(s), s, c, (float)x, (float)y, pg);
    s.ray_hit[hit_offset(s, l) + (size_t)y * s.lv[l].W + x] =
        hit ? make_float4(pg.x, pg.y, pg.z, 1.0f) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  });
}

// d_grvi_Get_RGB_Value_Interpolated (z_yooji_cuda_tsdf_renderer.cu:232-284):
// trilinear colour of the eight voxels around the hit, every one in range with
// weight > 0 (d_grvu, :194-229), rounded to 8 bits as InfiniTAM's toUChar
// (round half away from zero, clamp to 0..255); 0 when a neighbour fails.
// The 16 reads (weights and colours) are issued before any test.
template <class S>
__device__ uint32_t trilinear_color(const Vol<S>& V, const SessionDev& s, F3 pg) {
  F3 v;
  pos_in_voxel(pg, s, v);
  if (isnan(v.x) || isnan(v.y) || isnan(v.z)) return 0u;
  const float fx = floorf(v.x), fy = floorf(v.y), fz = floorf(v.z);
  const int ox = (int)fx, oy = (int)fy, oz = (int)fz;
  const float rx = v.x - fx, ry = v.y - fy, rz = v.z - fz;
  float tdummy;
  bool ok = ox >= 0 && ox + 1 < s.dim[0] && oy >= 0 && oy + 1 < s.dim[1] && oz >= 0 && oz + 1 < s.dim[2];
  const int cx = min(max(ox, 0), s.dim[0] - 2), cy = min(max(oy, 0), s.dim[1] - 2), cz = min(max(oz, 0), s.dim[2] - 2);
  const uint32_t X[2] = {V.wx(cx), V.wx(cx + 1)}, Y[2] = {V.wy(cy), V.wy(cy + 1)}, Z[2] = {V.wz(cz), V.wz(cz + 1)};
  uint32_t c[8];
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const uint32_t w = Z[i >> 2] + Y[(i >> 1) & 1] + X[i & 1];
    ok &= V.word_ok(w, tdummy);
    c[i] = __ldg(s.col + w);
  }
  if (!ok) return 0u;
  uint32_t out[3];
#pragma unroll
  for (int k = 0; k < 3; k++) {
    float f[4], b[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
      f[i] = (float)rgb_channel(c[i], k);
      b[i] = (float)rgb_channel(c[4 + i], k);
    }
    const float inf = (1.0f - ry) * ((1.0f - rx) * f[0] + rx * f[1]) + ry * ((1.0f - rx) * f[2] + rx * f[3]);
    const float inb = (1.0f - ry) * ((1.0f - rx) * b[0] + rx * b[1]) + ry * ((1.0f - rx) * b[2] + rx * b[3]);
    const float val = (1.0f - rz) * inf + rz * inb;
    const float rounded = (val < 0.0f) ? (val - 0.5f) : (val + 0.5f);
    out[k] = (uint32_t)(uint8_t)fmaxf(0.0f, fminf(255.0f, rounded));
  }
  return pack_rgb(out[0], out[1], out[2]);
}

// d_grvu_Get_RGB_Value_Uninterpolated (z_yooji_cuda_tsdf_renderer.cu:155-229)
// for the scene maps: the colour of the nearest voxel (ROUNDF) if it is in
// range with weight > 0, else 0.  (The reference's scene image writes the green
// channel into the red plane, marked there as temporary; the true colour is
// written here.)
template <class S>
__device__ uint32_t nearest_color(const Vol<S>& V, const SessionDev& s, F3 pg) {
  F3 v;
  pos_in_voxel(pg, s, v);
  if (isnan(v.x) || isnan(v.y) || isnan(v.z)) return 0u;
  const int x = roundf_ref(v.x), y = roundf_ref(v.y), z = roundf_ref(v.z);
  if (x < 0 || x >= s.dim[0] || y < 0 || y >= s.dim[1] || z < 0 || z >= s.dim[2]) return 0u;
  const uint32_t w = V.wx(x) + V.wy(y) + V.wz(z);
  float t;
  if (!V.word_ok(w, t)) return 0u;
  return __ldg(s.col + w);
}

// surface normal of a hit (d_csnt), camera-frame vertex and normal, shading,
// colour, into the model maps or the external outputs
template <class S, bool COLOR>
__device__ inline void shade_ray(const RayArgs& a, const Vol<S>& V, const SessionDev& s, const TileCam& c, int l,
                                 int x, int y, bool hit, F3 pg) {
  const bool ext = a.level >= 0;
  const size_t idx = (size_t)y * s.lv[l].W + x;
  F3 sn;
  bool valid = hit;
  if (valid) valid = surface_normal(V, s, pg, sn);
  float dep = 0.0f, img = 0.0f;
  uint32_t rgb = 0u;
  F3 pc = f3(-100.0f, -100.0f, -100.0f), sc = f3(-100.0f, -100.0f, -100.0f);
  if (valid) {
    if (COLOR && s.col) rgb = (a.mode & kRayNearestColor) ? nearest_color(V, s, pg) : trilinear_color(V, s, pg);
    pc = transform(pg, c.Tgc);
    dep = pc.z;
    sc = (a.mode & kRayGlobalNormals) ? sn : rotate(sn, c.Tgc);
    float ang = sc.x * a.light[0] + sc.y * a.light[1] + sc.z * a.light[2];
    img = fmaxf(0.0f, fminf(255.0f, (0.8f * ang + 0.2f) * 255.0f));
  }
  if (ext) {
    if (!valid && (a.mode & kRayWhiteBackground)) rgb = 0x00ffffffu;
    a.out_depth[idx] = dep;
    if (a.out_vtx3) {
      a.out_vtx3[3 * idx] = pc.x;
      a.out_vtx3[3 * idx + 1] = pc.y;
      a.out_vtx3[3 * idx + 2] = pc.z;
    }
    a.out_nrm3[3 * idx] = sc.x;
    a.out_nrm3[3 * idx + 1] = sc.y;
    a.out_nrm3[3 * idx + 2] = sc.z;
    if (a.out_img) a.out_img[idx] = (uint8_t)img;
    if (COLOR && a.out_rgb) {
      const size_t plane = (size_t)s.lv[l].W * s.lv[l].H;
      a.out_rgb[idx] = (uint8_t)rgb_channel(rgb, 0);
      a.out_rgb[plane + idx] = (uint8_t)rgb_channel(rgb, 1);
      a.out_rgb[2 * plane + idx] = (uint8_t)rgb_channel(rgb, 2);
    }
  } else {
    const float vw = valid ? 1.0f : 0.0f;
    s.m_depth[l][idx] = dep;
    s.m_vtx[l][idx] = make_float4(pc.x, pc.y, pc.z, vw);
    s.m_nrm[l][idx] = make_float4(sc.x, sc.y, sc.z, vw);
    s.m_img[l][idx] = (uint8_t)img;
    if (COLOR && s.col) s.m_rgb[l][idx] = rgb;
  }
}

// phase 2: the maps of every ray from its surface point in the hit buffer
template <class S>
__global__ void __launch_bounds__(kRayThreads, VS_SHADE_MIN_BLOCKS) k_ray_shade(RayArgs a) {
  for_each_ray_tile<false>(a, [&](const SessionDev& s, int l, int x, int y, const TileCam& c) {
    const float4 h = s.ray_hit[hit_offset(s, l) + (size_t)y * s.lv[l].W + x];
    shade_ray<S, true>(a, volume_of<S>(s), s, c, l, x, y, h.w != 0.0f, f3(h.x, h.y, h.z));
  });
}

#ifndef VS_FUSED_MIN_BLOCKS
#define VS_FUSED_MIN_BLOCKS 8
#endif

// both phases in one pass, without the hit buffer (every ray-cast without
// colour)
template <class S, bool SCENE>
__global__ void __launch_bounds__(kRayThreads, VS_FUSED_MIN_BLOCKS) k_ray_fused(RayArgs a) {
  for_each_ray_tile<SCENE>(a, [&](const SessionDev& s, int l, int x, int y, const TileCam& c) {
    const Vol<S> V = volume_of<S>(s);
    F3 pg;
    const bool hit = cast_ray<S, SCENE>(V, s, c, (float)x, (float)y, pg);
    shade_ray<S, false>(a, V, s, c, l, x, y, hit, pg);
  });
}

__global__ void k_maps_export(const float4* __restrict__ mv, const float4* __restrict__ mn,
                              const float4* __restrict__ iv, const float4* __restrict__ in, size_t n,
                              float* v3, float* n3, float* iv3, float* in3) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    if (v3) {
      float4 a = mv[i];
      v3[3 * i] = a.x, v3[3 * i + 1] = a.y, v3[3 * i + 2] = a.z;
    }
    if (n3) {
      float4 a = mn[i];
      n3[3 * i] = a.x, n3[3 * i + 1] = a.y, n3[3 * i + 2] = a.z;
    }
    if (iv3) {
      float4 a = iv[i];
      iv3[3 * i] = a.x, iv3[3 * i + 1] = a.y, iv3[3 * i + 2] = a.z;
    }
    if (in3) {
      float4 a = in[i];
      in3[3 * i] = a.x, in3[3 * i + 1] = a.y, in3[3 * i + 2] = a.z;
    }
  }
}

}  // namespace

template <class K>
int max_per_sm(K kernel) {
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kRayThreads, 0) != cudaSuccess || per_sm < 1)
    per_sm = 4;
  return per_sm;
}

// of the march grid (with the shading in it, unless a session keeps colour)
// and the shading grid
template <class S>
int ray_max_per_sm(bool shade, bool color) {
  static const int f = max_per_sm(k_ray_fused<S, false>);
  static const int m = max_per_sm(k_ray_march<S, false>);
  static const int h = max_per_sm(k_ray_shade<S>);
  return shade ? h : color ? m : f;
}

int grid_of(int want, int most) { return sm_count() * ((want > 0 && want < most) ? want : most); }

template <class S>
void launch_ray_phases(const RayArgs& a0, const LaunchShape& shape, bool color, cudaStream_t st) {
  RayArgs a = a0;
  k_band<<<sm_count() * 4, kBandThreads, 0, st>>>(a.bt);
  const int march = grid_of(shape.march_blocks_per_sm, ray_max_per_sm<S>(false, color));
  if (!color) {
    if (a.mode & kRayScene)
      k_ray_fused<S, true><<<march, kRayThreads, 0, st>>>(a);
    else
      k_ray_fused<S, false><<<march, kRayThreads, 0, st>>>(a);
    return;
  }
  if (a.mode & kRayScene)
    k_ray_march<S, true><<<march, kRayThreads, 0, st>>>(a);
  else
    k_ray_march<S, false><<<march, kRayThreads, 0, st>>>(a);
  a.work = a0.work + 2;
  k_ray_shade<S><<<grid_of(shape.shade_blocks_per_sm, ray_max_per_sm<S>(true, color)), kRayThreads, 0, st>>>(a);
}

void launch_raycast(const BatchTable* bt, int tsdf_type, int level, const float* Tgc, const float* Tcg,
                    const float* center, float lx, float ly, float lz, bool gate, float* out_depth, float* out_vtx3,
                    float* out_nrm3, uint8_t* out_img, cudaStream_t st, const LaunchShape& shape, uint8_t* out_rgb,
                    bool color, int mode) {
  RayArgs a;
  a.bt = bt;
  a.work = const_cast<unsigned*>(bt->work);  // [0..1] march, [2..3] shade
  a.level = level;
  a.Tgc = Tgc;
  a.Tcg = Tcg;
  for (int k = 0; k < 3; k++) a.center[k] = center ? center[k] : 0.0f;  // by value: no copy goes before the launch
  a.light[0] = lx;
  a.light[1] = ly;
  a.light[2] = lz;
  a.gate = gate ? 1 : 0;
  a.out_depth = out_depth;
  a.out_vtx3 = out_vtx3;
  a.out_nrm3 = out_nrm3;
  a.out_img = out_img;
  a.out_rgb = out_rgb;
  a.mode = mode;
  switch (tsdf_type) {
    case VS_TSDF_FP16:
      launch_ray_phases<StoreF16>(a, shape, color, st);
      break;
    case VS_TSDF_FP32:
      launch_ray_phases<StoreF32>(a, shape, color, st);
      break;
    default:
      launch_ray_phases<StoreI16>(a, shape, color, st);
      break;
  }
}

int ray_max_blocks_per_sm(int tsdf_type, bool shade, bool color) {
  switch (tsdf_type) {
    case VS_TSDF_FP16:
      return ray_max_per_sm<StoreF16>(shade, color);
    case VS_TSDF_FP32:
      return ray_max_per_sm<StoreF32>(shade, color);
    default:
      return ray_max_per_sm<StoreI16>(shade, color);
  }
}

void launch_maps_export(const SessionDev& h, int level, float* vtx3, float* nrm3, float* ivtx3, float* inrm3,
                        cudaStream_t st) {
  size_t n = (size_t)h.lv[level].W * h.lv[level].H;
  k_maps_export<<<(int)((n + 255) / 256), 256, 0, st>>>(h.m_vtx[level], h.m_nrm[level], h.in_vtx[level],
                                                         h.in_nrm[level], n, vtx3, nrm3, ivtx3, inrm3);
}

}  // namespace vs
