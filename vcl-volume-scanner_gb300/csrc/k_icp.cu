// Projective point-to-plane ICP, entirely on the device.
//
// The reference (STAC/Engine/GPU/z_yooji_cuda_pose_tracker.cu:548-697 and
// :790-1042) launches one kernel per iteration, copies 1200 x 42 block
// partial sums to the host, adds them serially in FP32, solves the 6x6 system
// with an FP32 Cholesky on the host and copies the new increment back: three
// blocking transfers per iteration.  Here one launch does every iteration:
//   per pixel   FP32 Jacobian row A (6) and residual b (d_cssfp, :279-395)
//   per thread  accumulation of the 27 unique sums (21 of ATA, 6 of ATb)
//               plus count and sum b^2, in the configured precision
//   per block   warp-shuffle butterfly, then shared memory across warps
//   per grid    the last block to finish an iteration (atomic ticket) sums
//               the block partials in a fixed order, solves the 6x6 system in
//               FP64 (elimination without divisions; the reference's failure
//               rules, _yooji_cuda_math.h:489-592, from a float LDL^T beside
//               it), tests convergence
//               (|x|_inf < 5e-7, :971-972) and applies the SE(3) update in
//               FP64 (T_12 <- exp(x) T_12, :976-978)
//
// Batches: the launch serves every session of a batch table.  A session at
// level l owns icp_blocks(W_l H_l) block ranges ("virtual blocks"), laid out
// as they would be in a grid of that size; the persistent grid's blocks claim
// ranges of any session, each session has its own partial buffer and arrival
// counter, and the range that arrives last for a session reduces and solves
// that session's system.  Sums therefore run in the same order whatever else
// shares the launch.
#include <cuda_runtime.h>
#include <stdint.h>

#include "vs_internal.cuh"

namespace vs {
namespace {

constexpr int kThreads = 256;

// Bilinear taps of a float4 map at (xf, yf) (d_gii-style interpolation of the
// reference, _yooji_cuda_math.h:365-481): taps with zero weight are neither
// tested nor used (they count as 0), a used tap holding the -100 sentinel
// rejects the sample, and NaN coordinates are rejected (see the oracle).
// The four reads are issued together; a zero-weight tap reads its row/column
// neighbour inside the map and is replaced by 0 before use, which gives the
// read-and-test-in-turn form's result exactly.
struct Taps {
  int i00, i01, i10, i11;
  float rx, ry;
};

__device__ inline bool tap_setup(float xf, float yf, int w, int h, Taps& t) {
  if (!(xf >= 0.0f && xf <= (float)(w - 1) && yf >= 0.0f && yf <= (float)(h - 1))) return false;
  const int x = (int)xf, y = (int)yf;
  t.rx = xf - (float)x;
  t.ry = yf - (float)y;
  const int xb = t.rx > 0.0f ? x + 1 : x, yb = t.ry > 0.0f ? y + 1 : y;
  t.i00 = y * w + x;
  t.i01 = y * w + xb;
  t.i10 = yb * w + x;
  t.i11 = yb * w + xb;
  return true;
}

__device__ inline bool interp(const Taps& t, float4 a, float4 b, float4 c, float4 d, F3& out) {
  const bool ub = t.rx > 0.0f, uc = t.ry > 0.0f, ud = ub && uc;
  if (a.x == -100.0f || (ub && b.x == -100.0f) || (uc && c.x == -100.0f) || (ud && d.x == -100.0f)) return false;
  const F3 A = f3(a.x, a.y, a.z);
  const F3 B = ub ? f3(b.x, b.y, b.z) : f3(0, 0, 0);
  const F3 C = uc ? f3(c.x, c.y, c.z) : f3(0, 0, 0);
  const F3 D = ud ? f3(d.x, d.y, d.z) : f3(0, 0, 0);
  const float rx = t.rx, ry = t.ry, ix = 1.0f - rx, iy = 1.0f - ry;
  out.x = iy * (ix * A.x + rx * B.x) + ry * (ix * C.x + rx * D.x);
  out.y = iy * (ix * A.y + rx * B.y) + ry * (ix * C.y + rx * D.y);
  out.z = iy * (ix * A.z + rx * B.z) + ry * (ix * C.z + rx * D.z);
  return true;
}

// d_cssfp_Compute_Single_Summand_with_Forward_Params.  Two rounds of reads:
// the pixel's depth (and input normal), then the eight model-map taps.
// The per-pixel arithmetic is the reference's, operation for operation
// (IEEE divisions and square root): every pixel's term, and therefore every
// correspondence decision at the distance threshold, equals the float
// oracle's.  (Products with inverse focal lengths, one reciprocal of z and a
// reciprocal square root were 4 % faster, but moved the correspondence set
// of frames whose pixels sit on the threshold, up to 3.5e-4 rad per frame.)
__device__ inline bool icp_term(int x, int y, int w, int h, const float* K, float d1, float4 q,
                                const float4* __restrict__ mvtx, const float4* __restrict__ mnrm, const float* T21,
                                float th_icp, float cos_normal, float A[6], float& b) {
  const bool ntest = cos_normal > -2.0f;
  if (d1 < 1.0e-6f) return false;
  F3 tp = back_project((float)x, (float)y, K, d1);
  F3 p1 = transform(tp, T21);
  float u, v;
  project(p1, K, u, v);
  Taps t;
  if (!tap_setup(u, v, w, h, t)) return false;
  const float4 va = __ldg(mvtx + t.i00), vb = __ldg(mvtx + t.i01), vc = __ldg(mvtx + t.i10), vd = __ldg(mvtx + t.i11);
  F3 p0;
  if (!interp(t, va, vb, vc, vd, p0)) return false;
  float dd = (p0.x - p1.x) * (p0.x - p1.x) + (p0.y - p1.y) * (p0.y - p1.y) + (p0.z - p1.z) * (p0.z - p1.z);
  if (dd > th_icp) return false;
  const float4 na = __ldg(mnrm + t.i00), nb = __ldg(mnrm + t.i01), nc = __ldg(mnrm + t.i10), nd = __ldg(mnrm + t.i11);
  F3 n;
  if (!interp(t, na, nb, nc, nd, n)) return false;
  n = normalised(n);
  if (ntest) {
    if (q.w == 0.0f) return false;
    F3 nin = rotate(f3(q.x, q.y, q.z), T21);
    if (dot(nin, n) < cos_normal) return false;
  }
  A[0] = p1.z * n.y + (-p1.y) * n.z;
  A[1] = (-p1.z) * n.x + p1.x * n.z;
  A[2] = p1.y * n.x + (-p1.x) * n.y;
  A[3] = -n.x;
  A[4] = -n.y;
  A[5] = -n.z;
  b = dot(n, sub(p0, p1));
  return true;
}

// Two pixels with the normal test at once: the same operations without a
// branch, so that the taps of both are in flight together
__device__ __forceinline__ void icp_pair(const int (&x)[2], const int (&y)[2], int w, int h, const float* K,
                                         const float (&d1)[2], const float4 (&q)[2], const float4* __restrict__ mvtx,
                                         const float4* __restrict__ mnrm, const float* T21, float th_icp,
                                         float cos_normal, float (&A)[2][6], float (&b)[2], bool (&ok)[2]) {
  F3 p0[2], p1[2];
  Taps t[2];
  float4 v[2][4];
#pragma unroll
  for (int k = 0; k < 2; k++) {
    p1[k] = transform(back_project((float)x[k], (float)y[k], K, d1[k]), T21);
    float u, vv;
    project(p1[k], K, u, vv);
    ok[k] = tap_setup(u, vv, w, h, t[k]) && !(d1[k] < 1.0e-6f);
    if (!ok[k]) t[k].i00 = t[k].i01 = t[k].i10 = t[k].i11 = 0, t[k].rx = t[k].ry = 0.0f;  // (the map's first value)
  }
#pragma unroll
  for (int k = 0; k < 2; k++)
    v[k][0] = __ldg(mvtx + t[k].i00), v[k][1] = __ldg(mvtx + t[k].i01), v[k][2] = __ldg(mvtx + t[k].i10),
    v[k][3] = __ldg(mvtx + t[k].i11);
#pragma unroll
  for (int k = 0; k < 2; k++) {
    ok[k] &= interp(t[k], v[k][0], v[k][1], v[k][2], v[k][3], p0[k]);
    const float dd = (p0[k].x - p1[k].x) * (p0[k].x - p1[k].x) + (p0[k].y - p1[k].y) * (p0[k].y - p1[k].y) +
                     (p0[k].z - p1[k].z) * (p0[k].z - p1[k].z);
    ok[k] &= !(dd > th_icp);
  }
#pragma unroll
  for (int k = 0; k < 2; k++)
    v[k][0] = __ldg(mnrm + t[k].i00), v[k][1] = __ldg(mnrm + t[k].i01), v[k][2] = __ldg(mnrm + t[k].i10),
    v[k][3] = __ldg(mnrm + t[k].i11);
#pragma unroll
  for (int k = 0; k < 2; k++) {
    F3 n;
    ok[k] &= interp(t[k], v[k][0], v[k][1], v[k][2], v[k][3], n);
    n = normalised(n);
    const F3 nin = rotate(f3(q[k].x, q[k].y, q[k].z), T21);
    ok[k] &= q[k].w != 0.0f && !(dot(nin, n) < cos_normal);
    A[k][0] = p1[k].z * n.y + (-p1[k].y) * n.z;
    A[k][1] = (-p1[k].z) * n.x + p1[k].x * n.z;
    A[k][2] = p1[k].y * n.x + (-p1[k].x) * n.y;
    A[k][3] = -n.x;
    A[k][4] = -n.y;
    A[k][5] = -n.z;
    b[k] = dot(n, sub(p0[k], p1[k]));
  }
}

// error-free addition (Knuth two-sum): s + e == a + b exactly
__device__ inline void two_sum(float a, float b, float& s, float& e) {
  s = a + b;
  float bb = s - a;
  e = (a - (s - bb)) + (b - bb);
}

// Per-thread sums of the (few) pixels a thread owns are plain float (FP32
// and compensated modes) or double (FP64 mode); the compensated mode carries
// (sum, error) pairs only from the warp reduction on, where thousands of
// values meet, so the pixel loop keeps 29 accumulators in registers.
//
// Warp reduction: a butterfly reduce-scatter over the 29 sums (padded to
// 32).  At the level of lane bit m every lane keeps one half of its current
// values, sends the other half to lane ^ m and adds what it receives, so the
// five levels cost 16 + 8 + 4 + 2 + 1 exchanges instead of 29 per level, and
// lane q ends with the warp's sum of quantity q, in a fixed order.
template <int HALF, int M, class T>
__device__ __forceinline__ void rs_level(T* a, int lane) {
  const bool hi = (lane & M) != 0;
#pragma unroll
  for (int i = 0; i < HALF; i++) {
    const T keep = hi ? a[HALF + i] : a[i];
    const T send = hi ? a[i] : a[HALF + i];
    a[i] = keep + __shfl_xor_sync(0xffffffffu, send, M);
  }
}
template <int HALF, int M>
__device__ __forceinline__ void rs_level_pair(float* s, float* c, int lane) {
  const bool hi = (lane & M) != 0;
#pragma unroll
  for (int i = 0; i < HALF; i++) {
    const float ks = hi ? s[HALF + i] : s[i], kc = hi ? c[HALF + i] : c[i];
    const float ss = hi ? s[i] : s[HALF + i], sc = hi ? c[i] : c[HALF + i];
    const float rs = __shfl_xor_sync(0xffffffffu, ss, M), rc = __shfl_xor_sync(0xffffffffu, sc, M);
    float t, e;
    two_sum(ks, rs, t, e);
    s[i] = t;
    c[i] = kc + rc + e;
  }
}

template <int MODE>
struct Acc;
template <>
struct Acc<VS_REDUCE_FP32> {
  float s[32];
  __device__ void zero() {
#pragma unroll
    for (int k = 0; k < 32; k++) s[k] = 0.0f;
  }
  __device__ void add(int k, float v) { s[k] += v; }
  // lane q < 29 returns the warp's sum of quantity q
  __device__ float2 reduce_scatter(int lane) {
    rs_level<16, 16>(s, lane);
    rs_level<8, 8>(s, lane);
    rs_level<4, 4>(s, lane);
    rs_level<2, 2>(s, lane);
    rs_level<1, 1>(s, lane);
    return make_float2(s[0], 0.0f);
  }
};
template <>
struct Acc<VS_REDUCE_KAHAN> {
  float s[32];
  __device__ void zero() {
#pragma unroll
    for (int k = 0; k < 32; k++) s[k] = 0.0f;
  }
  __device__ void add(int k, float v) { s[k] += v; }
  __device__ float2 reduce_scatter(int lane) {
    float c[16];
    // first level: plain values in, (sum, error) pairs out
    {
      const bool hi = (lane & 16) != 0;
#pragma unroll
      for (int i = 0; i < 16; i++) {
        const float keep = hi ? s[16 + i] : s[i];
        const float send = hi ? s[i] : s[16 + i];
        float t, e;
        two_sum(keep, __shfl_xor_sync(0xffffffffu, send, 16), t, e);
        s[i] = t;
        c[i] = e;
      }
    }
    rs_level_pair<8, 8>(s, c, lane);
    rs_level_pair<4, 4>(s, c, lane);
    rs_level_pair<2, 2>(s, c, lane);
    rs_level_pair<1, 1>(s, c, lane);
    return make_float2(s[0], c[0]);
  }
};
template <>
struct Acc<VS_REDUCE_FP64> {
  double s[32];
  __device__ void zero() {
#pragma unroll
    for (int k = 0; k < 32; k++) s[k] = 0.0;
  }
  __device__ void add(int k, float v) { s[k] += (double)v; }
  __device__ double2 reduce_scatter(int lane) {
    rs_level<16, 16>(s, lane);
    rs_level<8, 8>(s, lane);
    rs_level<4, 4>(s, lane);
    rs_level<2, 2>(s, lane);
    rs_level<1, 1>(s, lane);
    return make_double2(s[0], 0.0);
  }
};

// Partial sums travel as (sum, error) pairs in the mode's own type: float2
// for the FP32 and compensated modes (no conversions to double, which run on
// the narrow FP64 pipe), double2 for the FP64 mode.
template <int MODE>
struct PartT {
  typedef float2 type;
};
template <>
struct PartT<VS_REDUCE_FP64> {
  typedef double2 type;
};
__device__ inline float2 combine(float2 a, float2 b, int mode) {
  if (mode == VS_REDUCE_FP32) return make_float2(a.x + b.x, 0.0f);
  float t, e;
  two_sum(a.x, b.x, t, e);
  return make_float2(t, a.y + b.y + e);
}
__device__ inline double2 combine(double2 a, double2 b, int) { return make_double2(a.x + b.x, 0.0); }
__device__ inline float2 shfl_xor2(float2 v, int m) {
  return make_float2(__shfl_xor_sync(0xffffffffu, v.x, m), __shfl_xor_sync(0xffffffffu, v.y, m));
}
__device__ inline double2 shfl_xor2(double2 v, int m) {
  return make_double2(__shfl_xor_sync(0xffffffffu, v.x, m), __shfl_xor_sync(0xffffffffu, v.y, m));
}

__device__ inline int tri_index(int i, int j) { return i * 6 - i * (i - 1) / 2 + (j - i); }

// one pixel's products
template <class ACC>
__device__ __forceinline__ void add_term(ACC& acc, const float (&A)[6], float b) {
#pragma unroll
  for (int i = 0; i < 6; i++)
#pragma unroll
    for (int j = i; j < 6; j++) acc.add(tri_index(i, j), A[i] * A[j]);
#pragma unroll
  for (int i = 0; i < 6; i++) acc.add(21 + i, A[i] * b);
  acc.add(27, 1.0f);
  acc.add(28, b * b);
}

// ---- FP64 pose algebra ------------------------------------------------------
// FP64 runs on a narrow pipe on this part: an operation of a warp takes 64
// cycles whatever the number of active lanes, and the next one does not start
// before (measured, dependent or not; a conversion or a reciprocal
// approximation takes about 10 and 23, passing a double to another lane 34).
// So what counts between an iteration's sums and its new pose is the number
// of FP64 operations that one warp issues:
//   * the 6x6 system is eliminated without divisions, one element per lane,
//     with the right-hand side as a seventh row: two operations per column;
//   * the float factorisation that only decides failure runs beside it in
//     another warp;
//   * the three series of the exponential are one series with lane-dependent
//     coefficients, every element of the 4x4 results a lane's few fused
//     multiply-adds.
// One column per step with a reciprocal and separate products and sums, and one
// series per lane, took 10.0 us from an iteration's sums to its published
// pose (6.4 us where the step ended the level); this takes about 4 (3).  A
// 640x480 frame went from 545 to 486 us, a 320x240 frame from 427 to 367.

// lane -> (row, col) of the lower triangle, row-major: lane = row*(row+1)/2 + col
__device__ __forceinline__ int low_lane(int r, int c) { return r * (r + 1) / 2 + c; }
__device__ __forceinline__ void low_rc(int lane, int& r, int& c) {
  r = 0;
  while (low_lane(r + 1, 0) <= lane) r++;
  c = lane - low_lane(r, 0);
}

// The 6x6 solve: d_lld_LL_Decomposition + d_sls_Solve_Linear_System_using_LLD
// (_yooji_cuda_math.h:489-592), restated as an L D L^T factorisation
// (D_j = L_jj^2).  The factorisation is done twice.  In float - the
// reference's own precision - it decides failure by the reference's pivot
// rules unchanged: a pivot with sqrt(D_j) < 1e-8 fails the solve (1); a
// negative or NaN pivot makes the reference's square root NaN, its column
// zero and the solution NaN, which the convergence test reads as converged
// (2).  In FP64, from the FP64 sums, it gives the solution.

// float factorisation, one matrix element per lane: returns 0, 1 or 2; lane
// i < 6 receives the float solution in v (used only where the FP64 factors
// have no positive pivot, or to record a solution that is not applied)
__device__ int warp_decide6(const double* fin, int lane, float& v) {
  const unsigned M = 0xffffffffu;
  int r = 0, c = 0;
  if (lane < 21) low_rc(lane, r, c);
  float a = (lane < 21) ? (float)fin[tri_index(c, r)] : 0.0f;
  bool nanp = false, fail = false;
#pragma unroll
  for (int j = 0; j < 6; j++) {
    const float d = __shfl_sync(M, a, low_lane(j, j));
    const bool neg = !(d >= 0.0f);
    const bool tiny = !neg && !(sqrtf(d) >= 1e-8f);
    nanp |= neg;
    fail |= tiny;
    const bool ok = !neg && !tiny;
    if (lane < 21 && c == j && r > j) a = ok ? a / d : 0.0f;
    const bool upd = lane < 21 && c > j;
    const int sr = upd ? low_lane(r, j) : lane, sc = upd ? low_lane(c, j) : lane;
    const float lr = __shfl_sync(M, a, sr), lc = __shfl_sync(M, a, sc);
    if (upd && ok) a -= lr * d * lc;
  }
  v = (lane < 6) ? (float)fin[21 + lane] : 0.0f;
#pragma unroll
  for (int j = 0; j < 6; j++) {
    const float vj = __shfl_sync(M, v, j);
    const bool upd = lane < 6 && lane > j;
    const float lij = __shfl_sync(M, a, upd ? low_lane(lane, j) : lane);
    if (upd) v -= lij * vj;
  }
  const float dd = __shfl_sync(M, a, lane < 6 ? low_lane(lane, lane) : lane);
  if (lane < 6) v = v / dd;
#pragma unroll
  for (int j = 5; j >= 0; j--) {
    const float xj = __shfl_sync(M, v, j);
    const bool upd = lane < j;
    const float lji = __shfl_sync(M, a, upd ? low_lane(j, lane) : lane);
    if (upd) v -= lji * xj;
  }
  return fail ? 1 : (nanp ? 2 : 0);
}

// rcp.approx.ftz.f64: a first approximation of 1 / d, good to about 2^-20
// (PTX ISA); subnormals flush, so it is used well inside the normal range
__device__ __forceinline__ double rcp_start(double d) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
  return r;
}

// the exponent of a normal number (0 .. 2046 as stored)
__device__ __forceinline__ int exponent_bits(double d) { return (__double2hiint(d) >> 20) & 0x7ff; }

// x 2^(1023 - eb) in integer operations; a zero (or subnormal) x gives 0
__device__ __forceinline__ double scaled_down(double x, int eb) {
  const int hi = __double2hiint(x);
  if ((hi & 0x7ff00000) == 0) return 0.0;
  return __hiloint2double(hi - ((eb - 1023) << 20), __double2loint(x));
}

// positive, not NaN, and well inside the normal range (integer operations)
__device__ __forceinline__ bool good_pivot(double d) {
  const int hi = __double2hiint(d);
  return hi > (32 << 20) && hi < (2014 << 20);
}

// FP64 solve of the 6x6 system, one warp: lane low_lane(r, c), c <= r < 6,
// holds element (r, c) of the lower triangle and lane 21 + c element c of the
// right-hand side (row 6).  Column j is eliminated without a division: every
// later element becomes a d - u_r u_c with the pivot d and column j's
// elements u, where d and u_c are scaled by the power of two that brings d
// into [1, 2), so the rows (scaled alike with their right-hand side) stay in
// range; then each row is divided by its pivot, all at once, and substituted
// back.  1 / d = r0 (1 + e + e^2) with r0 ~ 1 / d and e = 1 - d r0
// (|e| < 2^-20), up to e^3, below the double rounding.  (Against exact
// arithmetic, random systems of condition 1e1 to 1e10: relative errors 0.6 to
// 1.0 times those of an L D L^T factorisation with reciprocal pivots and
// separate products.)  Lane 21 + j receives x_j; false: a pivot is not
// positive.
__device__ __forceinline__ bool warp_solve6(const double* fin, int lane, double& x) {
  const unsigned M = 0xffffffffu;
  int r = 6, c = lane - 21;
  if (lane < 21) low_rc(lane, r, c);
  const bool held = lane < 27;
  if (!held) c = 0;
  double a = held ? (r < 6 ? fin[tri_index(c, r)] : fin[21 + c]) : 0.0;
  bool pos = true;
#pragma unroll
  for (int j = 0; j < 5; j++) {
    const bool upd = held && c > j;
    const double d = __shfl_sync(M, a, low_lane(j, j));
    const double ur = __shfl_sync(M, a, upd ? low_lane(r, j) : lane);
    const double uc = __shfl_sync(M, a, upd ? low_lane(c, j) : lane);
    pos &= good_pivot(d);
    const int eb = exponent_bits(d);
    const double m = a * scaled_down(d, eb);
    const double n = fma(-ur, scaled_down(uc, eb), m);
    if (upd) a = n;
  }
  const double d = __shfl_sync(M, a, low_lane(c, c));
  pos = __all_sync(M, pos && good_pivot(d));
  const double r0 = rcp_start(d);
  const double e = fma(-d, r0, 1.0);
  const double w = a * r0;
  const double l = fma(w, fma(e, e, e), w);
  double lc[6];  // lane 21 + j: element (k, j) of the unit triangle
#pragma unroll
  for (int k = 1; k < 6; k++) lc[k] = __shfl_sync(M, l, r == 6 && c < k ? low_lane(k, c) : lane);
  x = l;
#pragma unroll
  for (int k = 5; k > 0; k--) {
    const double xk = __shfl_sync(M, x, 21 + k);
    if (r == 6 && c < k) x = fma(-lc[k], xk, x);
  }
  return pos;
}

// SE(3) exponential of the twist q = [w; v] in the reference's parameterisation
// (z_uitme_Update_Incremental_Tracking_with_Matrix_Exponential,
// z_yooji_cuda_pose_tracker.cu:50-149: R = I + sin(th)[u]x +
// (1 - cos(th))[u]x^2 with u = w / th, t = (I - R)[u]x v / th + u u^T v),
// written with W = [w]x as R = I + A W + B W^2, t = v + B (w x v) +
// C (w (w.v) - th^2 v), A = sin(th)/th, B = (1 - cos(th))/th^2,
// C = (th - sin(th))/th^3 - the same function, with no division by th.  For
// th < 0.1 the three coefficients come from their Taylor series in th^2
// (truncation below 1e-17 relative), lane l < 3 the l-th (the constants are selected, not read: a read would
// miss in the closing SM's constant cache);
// otherwise from sin/cos.  Lane l < 16 returns element l of the 4x4 result.
__device__ __noinline__ void se3_far(double th2, double* k) {
  const double th = sqrt(th2);
  const double sn = sin(th), cs = cos(th);
  k[0] = sn / th;
  k[1] = (1.0 - cs) / th2;
  k[2] = (th - sn) / (th2 * th);
}
__device__ __forceinline__ double se3_exp(const double q[6], int lane) {
  const unsigned M = 0xffffffffu;
  auto pick = [](int i, double u, double v, double w) { return i == 0 ? u : (i == 1 ? v : w); };
  // lanes 0..15: th^2 = w.w; lanes 16..31: w.v
  const bool lo = lane < 16;
  double dt = q[0] * (lo ? q[0] : q[3]);
  dt = fma(q[1], lo ? q[1] : q[4], dt);
  dt = fma(q[2], lo ? q[2] : q[5], dt);
  const double th2 = __shfl_sync(M, dt, 0), wv = __shfl_sync(M, dt, 16);
  // element (r, c) of [R t] is base + Y W + X (q_r m - th^2 base)
  const int r = (lane >> 2) & 3, c = lane & 3;
  const double qr = pick(r, q[0], q[1], q[2]), qc = pick(c, q[0], q[1], q[2]);
  const double vr = pick(r, q[3], q[4], q[5]);
  // (w x v)_r = w_(r+1) v_(r+2) - w_(r+2) v_(r+1)
  double f = pick(r, q[2], q[0], q[1]) * pick(r, q[4], q[5], q[3]);
  f = fma(pick(r, q[1], q[2], q[0]), pick(r, q[5], q[3], q[4]), -f);
  const bool rot = c < 3;
  double off = r == c ? 0.0 : pick(3 - r - c, q[0], q[1], q[2]);  // [w]x, with its signs
  if (c == (r + 1) % 3) off = -off;
  const double base = rot ? (r == c ? 1.0 : 0.0) : vr, W = rot ? off : f;
  const double p = fma(-th2, base, qr * (rot ? qc : wv));
  double A, B, C;
  if (th2 < 0.01) {
    const int g = lane & 3;
    double k = pick(g, -1.0 / 39916800, -1.0 / 479001600, -1.0 / 6227020800);
    k = fma(k, th2, pick(g, 1.0 / 362880, 1.0 / 3628800, 1.0 / 39916800));
    k = fma(k, th2, pick(g, -1.0 / 5040, -1.0 / 40320, -1.0 / 362880));
    k = fma(k, th2, pick(g, 1.0 / 120, 1.0 / 720, 1.0 / 5040));
    k = fma(k, th2, pick(g, -1.0 / 6, -1.0 / 24, -1.0 / 120));
    k = fma(k, th2, pick(g, 1.0, 1.0 / 2, 1.0 / 6));
    A = __shfl_sync(M, k, 0), B = __shfl_sync(M, k, 1), C = __shfl_sync(M, k, 2);
  } else {
    double k[3];
    se3_far(th2, k);
    A = k[0], B = k[1], C = k[2];
  }
  const double el = fma(rot ? B : C, p, fma(rot ? A : B, W, base));
  return lane >= 16 || r == 3 ? (lane == 15 ? 1.0 : 0.0) : el;
}

// fabs(x) >= y for a positive y, in integer operations; false for a NaN
__device__ __forceinline__ bool abs_at_least(double x, double y) {
  const unsigned long long u = (unsigned long long)__double_as_longlong(x) & 0x7fffffffffffffffull;
  return u >= (unsigned long long)__double_as_longlong(y) && u <= 0x7ff0000000000000ull;
}

// out = A * B (4x4, lane l < 16 computes element l); A in shared memory, B in
// global memory, read from L2 (another block of the launch may have written it)
__device__ void warp_compose(const double* A, const double* B, double* out, int lane) {
  if (lane < 16) {
    const int r = lane >> 2, c = lane & 3;
    double s = 0.0;
#pragma unroll
    for (int k = 0; k < 4; k++) s += A[r * 4 + k] * __ldcg(B + k * 4 + c);
    out[lane] = s;
  }
  __syncwarp();
}
// inverse of a rigid transform [R t; 0 1] held in shared memory; lane l < 16
// receives element l
__device__ void warp_rigid_inverse(const double* T, int lane, double& out) {
  out = 0.0;
  if (lane < 16) {
    const int r = lane >> 2, c = lane & 3;
    if (r == 3)
      out = (c == 3) ? 1.0 : 0.0;
    else if (c < 3)
      out = T[c * 4 + r];
    else
      out = -(T[0 * 4 + r] * T[3] + T[1 * 4 + r] * T[7] + T[2 * 4 + r] * T[11]);
  }
}
// ---- scheduling: one persistent launch for every iteration of every session
//
// words[slot] is a session's work word: [31:30] the pyramid level its current
// iteration runs at (kWordDone: no iteration left), [29:16] the iterations
// finished at that level, [15:0] the next range of the current iteration.  A
// block claims a range with one atomicAdd on the word; the block whose range
// arrives last closes the iteration (sums, solve, pose update) and publishes
// the next one by storing a new word.  Sessions therefore move through their
// iterations independently: while one is being closed, the blocks work on
// another's ranges, and an iteration that a session does not need (it
// converged) costs nothing.  With one launch per iteration every iteration
// paid the launch, the reads of the tables and the slowest session's closing
// block: tracking of one 640x480 frame took 307 us in 19 launches and 242 when
// this launch replaced them, with FP64 sums 603 and 440 (148 and 255 now, with
// the closing and the lists below; the kernel alone in each case).
//
// Progress needs no block but the running ones: a range is claimed only by a
// block that then runs it, a closer goes on claiming ranges itself, and a
// block that finds nothing to claim holds nothing, so it may leave at any
// time.  It leaves when every session is done, or when the unfinished
// sessions could not give it a range (blocks are numbered, and the block's
// number is not below the sum of their largest range counts), which frees its
// SM for other streams' kernels, or when it has looked kIdleLimit times.  A
// session's outcome is written by the block that ends its tracking alone: until
// then its frame counts as lost, and stays so if nobody ends it.
constexpr unsigned kWordDone = 3u;
constexpr int kIdleLimit = 1 << 22;  // looks without a range before a block leaves (seconds; none in a sound run)

__device__ __forceinline__ unsigned work_word(int level, int iter) {
  return ((unsigned)level << 30) | ((unsigned)iter << 16);
}
__device__ __forceinline__ unsigned load_word(const unsigned* p) { return *(const volatile unsigned*)p; }

// the session's next level with iterations, from l down; -1: none
__device__ inline int next_level(const SessionDev* s, int l) {
  while (l >= 0 && s->iters[l] <= 0) l--;
  return l;
}

// end of a session's tracking, one warp: T_gc <- T12 T_gc unless it failed
// or was skipped, and the outcome
__device__ void icp_finish(Pose* P, bool skip, bool failed, int ln, double* Tn, double* A) {
  if (!skip && !failed) {
    if (ln < 16) A[ln] = __ldcg(&P->T12[ln]);
    __syncwarp();
    double Ti;
    warp_compose(A, P->T_gc, Tn, ln);
    if (ln < 16) P->T_gc[ln] = Tn[ln];
    warp_rigid_inverse(Tn, ln, Ti);
    if (ln < 16) {
      P->Tgc[ln] = (float)Tn[ln];
      P->Tcg[ln] = (float)Ti;
    }
    if (ln == 3 || ln == 7 || ln == 11) P->center[ln >> 2] = (float)Ti;
  }
  if (ln == 0) {
    P->tracked = failed ? 0 : 1;
    P->failed = failed ? 1 : 0;
  }
}

// one warp per slot: the increment of this frame starts at identity (or at
// `init`, and then only level 0 runs), its frame is counted, as lost until its
// tracking ends, and the session's first iteration is published
__global__ void k_icp_begin(const BatchTable* __restrict__ bt, unsigned* words, int frame_mode, int with_init,
                            const float* init) {
  if ((int)blockIdx.x >= bt->n) return;
  const SessionDev* s = bt->s[blockIdx.x];
  Pose* P = s->pose;
  const int ln = threadIdx.x;
  __shared__ double T[16], Tn[16], A[16];
  const bool skip = frame_mode && P->frame == 0;
  if (ln < 16) T[ln] = (with_init && init) ? (double)init[ln] : ((ln % 5 == 0) ? 1.0 : 0.0);
  __syncwarp();
  double Ti;
  warp_rigid_inverse(T, ln, Ti);
  if (ln < 16) {
    P->T12[ln] = T[ln];
    P->T21[ln] = (float)Ti;
  }
  const int l = skip ? -1 : next_level(s, with_init ? 0 : s->levels - 1);
  __syncwarp();
  if (ln == 0) {
    P->skip = skip ? 1 : 0;
    P->tracked = 0;
    P->failed = 1;
    if (frame_mode) P->frame += 1;
    P->iters_run = 0;
    P->valid_count = 0;
  }
  if (l < 0) icp_finish(P, skip, false, ln, Tn, A);
  if (ln == 0) {
    *s->icp_counter = 0u;
    words[blockIdx.x] = l < 0 ? kWordDone << 30 : work_word(l, 0);
  }
}

// Closes a session's iteration from its sums; called by warps 0 and 1 of the
// closing block together.  Warp 1 decides failure and records the
// sums; warp 0 solves, updates the pose and returns the session's next work
// word (to be published once its lanes' writes are out).
__device__ __forceinline__ unsigned icp_close(const SessionDev* s, const double* fin, int level, int iter) {
  __shared__ double A[16], Tn[16];
  __shared__ float xf[6];
  __shared__ int status;
  Pose* P = s->pose;
  const int ln = threadIdx.x & 31;
  if (threadIdx.x >= 32) {
    if (ln < 29) P->last_sums[ln] = fin[ln];
    if (ln == 0) {
      atomicAdd(&P->iters_run, 1);
      P->valid_count = (int)fin[27];
    }
    float v;
    const int st = warp_decide6(fin, ln, v);
    if (ln < 6) xf[ln] = v;
    if (ln == 0) status = st;
    __syncwarp();
    asm volatile("bar.sync 1, 64;" ::: "memory");
    return 0u;
  }
  // column ln & 3 of T12, read while the system is solved
  double t12[4];
#pragma unroll
  for (int k = 0; k < 4; k++) t12[k] = __ldcg(&P->T12[k * 4 + (ln & 3)]);
  double xl;
  const bool pos = warp_solve6(fin, ln, xl);
  double x[6];
#pragma unroll
  for (int k = 0; k < 6; k++) x[k] = __shfl_sync(0xffffffffu, xl, 21 + k);
  asm volatile("bar.sync 1, 64;" ::: "memory");
  const int st = status;
  const bool failed = st == 1;
  if (!failed) {
    // st 2: the reference's solution is NaN here and reads as converged; the
    // pose is not updated and the float factors' (finite) solution is only
    // recorded.  !pos: a pivot that float rounding left positive and FP64 does
    // not (a system singular to FP64 precision): the float solution.
    if (st == 2 || !pos) {
#pragma unroll
      for (int k = 0; k < 6; k++) x[k] = (double)xf[k];
    }
    // |x|_inf < 5e-7 ends the level (d_niv_Norm_Infinity_Vector: NaN entries never
    // raise the maximum, so an all-NaN solution also ends it)
    bool big = false;
#pragma unroll
    for (int k = 0; k < 6; k++) {
      big |= abs_at_least(x[k], 5.0e-7);
      if (ln == k) P->last_x[k] = (float)x[k];
    }
    const bool ends = st == 2 || !big;
    if (!ends) {
      // T12 <- E T12 and T21 = its inverse in float; lane l < 16 holds element l
      const unsigned M = 0xffffffffu;
      const double e = se3_exp(x, ln);
      const int row = ln & 12, r = (ln >> 2) & 3, c = ln & 3;
      const double e0 = __shfl_sync(M, e, row), e1 = __shfl_sync(M, e, row + 1), e2 = __shfl_sync(M, e, row + 2),
                   e3 = __shfl_sync(M, e, row + 3);
      const double n = fma(e0, t12[0], fma(e1, t12[1], fma(e2, t12[2], e3 * t12[3])));
      // transposed element, and for the last column -(R^T t)_r
      const double nt = __shfl_sync(M, n, (c < 3 ? c * 4 : 0) + r);
      double u[3], t[3];
#pragma unroll
      for (int k = 0; k < 3; k++) u[k] = __shfl_sync(M, n, k * 4 + r), t[k] = __shfl_sync(M, n, k * 4 + 3);
      const double tr = -fma(u[2], t[2], fma(u[1], t[1], u[0] * t[0]));
      if (ln < 16) {
        P->T12[ln] = n;
        P->T21[ln] = r == 3 ? (c == 3 ? 1.0f : 0.0f) : (float)(c < 3 ? nt : tr);
      }
    }
    if (!ends && iter + 1 < s->iters[level]) return work_word(level, iter + 1);
    const int l = next_level(s, level - 1);
    if (l >= 0) return work_word(l, 0);
    __syncwarp();
  }
  icp_finish(P, false, failed, ln, Tn, A);
  return kWordDone << 30;
}

// The closing of an iteration by the block whose range arrived last (every
// thread; out of line, so that the pixel loop's register allocation does not
// carry it): the ranges' partials in a fixed order,
// then the solve.  Warp 0 receives the next work word, with every write of
// the block visible to whoever reads that word after a fence.
template <int MODE>
__device__ __noinline__ unsigned close_iteration(const SessionDev* s, int nvb, int level, int iter) {
  typedef typename PartT<MODE>::type PT;
  __shared__ double fin[29];
  // 8 threads per quantity, each a fixed stride over the ranges, then a fixed
  // shuffle tree
  const int k = threadIdx.x >> 3, j = threadIdx.x & 7;
  PT v;
  v.x = 0;
  v.y = 0;
  if (k < 29) {
    // the partials of up to 160 ranges in flight at once (64 in double),
    // combined in the same order as one at a time
    constexpr int kFly = MODE == VS_REDUCE_FP64 ? 8 : 20;
    const PT* base = reinterpret_cast<const PT*>(s->partials) + k;
    for (int bb = j; bb < nvb; bb += 8 * kFly) {
      PT t[kFly];
#pragma unroll
      for (int u = 0; u < kFly; u++) {
        t[u].x = 0, t[u].y = 0;  // (left undefined, it would hold a register over the pixel loop)
        if (bb + 8 * u < nvb) t[u] = __ldcg(base + (size_t)(bb + 8 * u) * kPartials);
      }
#pragma unroll
      for (int u = 0; u < kFly; u++)
        if (bb + 8 * u < nvb) v = combine(v, t[u], MODE);
    }
  }
#pragma unroll
  for (int m = 4; m >= 1; m >>= 1) v = combine(v, shfl_xor2(v, m), MODE);
  if (k < 29 && j == 0) fin[k] = (double)v.x + (double)v.y;
  __syncthreads();
  unsigned next = 0u;
  if (threadIdx.x < 64) next = icp_close(s, fin, level, iter);
  if (threadIdx.x < 32) {
    __syncwarp();
    __threadfence();
  }
  return next;
}

#ifndef VS_ICP_MIN_BLOCKS
#define VS_ICP_MIN_BLOCKS 3  // resident 256-thread blocks per SM the register allocation must allow
#endif

// One warp claims a range: *out_slot its session (-1: leave), *out_word the
// session's word with the range.  The block stays with the session it worked
// on (prefer) while that has ranges; otherwise it takes the first session that
// does, so that few sessions are under way at a time and their maps stay in
// L2 over their iterations.
__device__ __noinline__ void claim_range(unsigned* __restrict__ words, int n, const int (*sNvb)[kMaxSlots],
                                         int prefer, int* out_slot, unsigned* out_word) {
  const int lane = threadIdx.x & 31;
  int slot = -1;
  unsigned w = 0u;
  auto available = [&](int q, unsigned v) { return (int)(v & 0xffffu) < sNvb[v >> 30][q]; };
  for (int look = 0;; look++) {
    int first = prefer;
    if (first < 0) {
      int need = 0;
#pragma unroll
      for (int h = 0; h < kMaxSlots; h += 32) {
        const int q = h + lane;
        const unsigned v = q < n ? load_word(words + q) : kWordDone << 30;
        const unsigned m = __ballot_sync(0xffffffffu, available(q, v));
        if (m && first < 0) first = h + __ffs(m) - 1;
        if ((v >> 30) != kWordDone) need += max(sNvb[0][q], max(sNvb[1][q], sNvb[2][q]));
      }
      need = __reduce_add_sync(0xffffffffu, need);
      if (first < 0) {
        if ((int)blockIdx.x >= need || look >= kIdleLimit) break;
        __nanosleep(40);
        continue;
      }
    }
    if (lane == 0) w = atomicAdd(words + first, 1u);
    w = __shfl_sync(0xffffffffu, w, 0);
    if (available(first, w)) {
      slot = first;
      break;
    }
    prefer = -1;  // no range left there, or another block was faster
  }
  if (lane == 0) {
    *out_slot = slot;
    *out_word = w;
    __threadfence();  // the block reads the session's pose after its word (and the barrier that follows)
  }
}

// Ranges of a level whose pixels are listed: a session that tests normals has
// no term where the input normal is invalid, so its ranges run over the list
// of the pixels with a valid one (in raster order).  Those are 5 to 15 % of
// the pixels of the serving mix (the 60 degree test of the normal estimation
// on noisy depth), in 15 to 30 % of the 32-pixel words.  Reading depth and model
// taps of every pixel, tracking took 2.01 ms of the 64-session step and 0.606
// of sixteen sessions'; over the list 0.52 and 0.26 (a 640x480 frame 490 ->
// 434 us).  A range of 256 pixels is one per thread, and its blocks are done
// sooner; 512 pay the reduction of a range half as often.  Up to 8192 listed
// pixels (by the session's own count alone, so that its sums do not depend on
// what shares the launch) a level does not fill the launch's blocks: 256 there
// made a 640x480 frame 385 -> 377 us, a 320x240 frame 313 -> 299, FP64 tracking
// of 640x480 316 -> 285, sixteen sessions 1344 -> 1331, and 64 sessions 3872 ->
// 3897 (two runs of one side: 35 apart).  256 at every count took 64 sessions
// 4.5 % longer.  Every session has at least one range, which closes its
// iterations.
__device__ __forceinline__ int listed_ranges(int count) {
  const int per = count <= 8192 ? kThreads : 2 * kThreads;
  const int r = (count + per - 1) / per;
  return min(max(r, 1), kIcpMaxBlocks);
}

// a load that the compiler does not merge with an earlier one
template <class T>
__device__ __forceinline__ T reload(const T* p) {
  return *const_cast<const volatile T*>(p);
}

template <int MODE>
__global__ void __launch_bounds__(kThreads, VS_ICP_MIN_BLOCKS)
    k_icp_run(const BatchTable* __restrict__ bt, unsigned* __restrict__ words) {
  typedef typename PartT<MODE>::type PT;
  __shared__ PT wsum[kThreads / 32][29];
  __shared__ float sT21[12], sK[4];
  __shared__ const SessionDev* sS[kMaxSlots];
  __shared__ int sNvb[4][kMaxSlots];  // ranges of an iteration at level 0..2 (0: no such level); [3]: none (done)
  __shared__ int s_slot, s_close;
  __shared__ unsigned s_word;
  const int n = bt->n;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x < kMaxSlots) {
    const int i = threadIdx.x;
    sS[i] = i < n ? bt->s[i] : nullptr;
    const bool listed = i < n && sS[i]->cos_normal > -2.0f;
#pragma unroll
    for (int l = 0; l < kMaxLevels; l++) {
      int r = i < n ? bt->icp[l][i + 1] - bt->icp[l][i] : 0;
      if (r && listed) r = listed_ranges((int)sS[i]->in_count[l]);
      sNvb[l][i] = r;
    }
    sNvb[kMaxLevels][i] = 0;
  }
  __syncthreads();

  auto claim = [&](int prefer) { claim_range(words, n, sNvb, prefer, &s_slot, &s_word); };
  if (warp == 0) claim(-1);
  __syncthreads();
  while (s_slot >= 0) {
    const int level = (int)(s_word >> 30), vb = (int)(s_word & 0xffffu);
    const int nvb = sNvb[level][s_slot];
    const SessionDev* __restrict__ s = sS[s_slot];
    const int w = s->lv[level].W, h = s->lv[level].H;
    // the pose and intrinsics are read from shared memory in the pixel loop,
    // which leaves the registers to the 29 running sums; the pose comes from
    // L2 (this SM's L1 may hold an earlier iteration's)
    if (threadIdx.x < 12) sT21[threadIdx.x] = __ldcg(&s->pose->T21[threadIdx.x]);
    if (threadIdx.x >= 32 && threadIdx.x < 36) sK[threadIdx.x - 32] = s->lv[level].K[threadIdx.x - 32];
    const float* K = sK;
    const float* T21 = sT21;
    const float th = s->th_icp, cosn = s->cos_normal;
    const float* depth = s->depth[level];
    const float4* mvtx = s->m_vtx[level];
    const float4* mnrm = s->m_nrm[level];
    const float4* innrm = s->in_nrm[level];

    Acc<MODE> acc;
    acc.zero();
    const bool ntest = cosn > -2.0f;
    const uint32_t* list = ntest ? s->in_list[level] : nullptr;
    const int count = ntest ? (int)s->in_count[level] : w * h;
    const int stride = nvb * kThreads;
    // the first-round reads (depth, input normal) of a thread's next pixel are
    // in flight while its current pixel's taps are read, and the list entry
    // of the one after that
    int p = vb * kThreads + threadIdx.x;
    if (MODE == VS_REDUCE_FP64 && ntest && count <= 2 * stride) {
      // A listed range, one or two pixels per thread.  With FP64 sums, whose
      // 58 registers leave the loop below no room to read ahead, the two are
      // taken together before any sum is held (tracking of a 640x480 frame 332
      // -> 315 us, sixteen sessions 1655 -> 1619); the float sums gain nothing
      // (640x480 frames 385 and 385 us, a served mix 1050 and 1058).
      int xs[2], ys[2];
      float ds[2];
      float4 qs[2];
#pragma unroll
      for (int k = 0; k < 2; k++) {
        const uint32_t e = p + k * stride < count ? __ldg(list + p + k * stride) : 0u;
        xs[k] = (int)(e & 0xffffu), ys[k] = (int)(e >> 16);
      }
#pragma unroll
      for (int k = 0; k < 2; k++) {
        const bool in = p + k * stride < count;
        ds[k] = in ? __ldg(depth + ys[k] * w + xs[k]) : 0.0f;
        qs[k] = in ? __ldg(innrm + ys[k] * w + xs[k]) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      }
      __syncthreads();  // the pose
      float A[2][6], b[2];
      bool ok[2];
      icp_pair(xs, ys, w, h, K, ds, qs, mvtx, mnrm, T21, th, cosn, A, b, ok);
#pragma unroll
      for (int k = 0; k < 2; k++)
        if (ok[k]) add_term(acc, A[k], b[k]);
    } else {
      int x = 0, y = 0, dx = 0, dy = 0;
      uint32_t xy = 0u;
      float d_next = 0.0f;
      float4 q_next = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      if (ntest) {
        if (p < count) {
          xy = __ldg(list + p);
          x = (int)(xy & 0xffffu), y = (int)(xy >> 16);
          d_next = __ldg(depth + y * w + x);
          q_next = __ldg(innrm + y * w + x);
          if (p + stride < count) xy = __ldg(list + p + stride);
        }
      } else {
        y = p / w, x = p - y * w;
        dy = stride / w, dx = stride - dy * w;
        if (p < count) d_next = __ldg(depth + p);
      }
      __syncthreads();
      while (p < count) {
        const float d1 = d_next;
        const float4 qn = q_next;
        const int xc = x, yc = y;
        p += stride;
        if (ntest) {
          if (p < count) {
            x = (int)(xy & 0xffffu), y = (int)(xy >> 16);
            d_next = __ldg(depth + y * w + x);
            q_next = __ldg(innrm + y * w + x);
            if (p + stride < count) xy = __ldg(list + p + stride);
          }
        } else {
          x += dx;
          y += dy;
          if (x >= w) x -= w, y++;
          if (p < count) d_next = __ldg(depth + p);
        }
        float A[6], b;
        if (!icp_term(xc, yc, w, h, K, d1, qn, mvtx, mnrm, T21, th, cosn, A, b)) continue;
        add_term(acc, A, b);
      }
    }
    const PT mine = acc.reduce_scatter(lane);
    if (lane < 29) wsum[warp][lane] = mine;
    __syncthreads();
    if (warp == 0) {
      // the range again, read back from shared memory: over the pixel loop it
      // would hold registers.  Only this warp reads it here, because its claim
      // below writes the next one before the other warps pass a barrier.
      const int slot = reload(&s_slot);
      const unsigned word = reload(&s_word);
      const SessionDev* sr = reload(&sS[slot]);
      const int ranges = reload(&sNvb[word >> 30][slot]);
      if (lane < 29) {
        PT v = wsum[0][lane];
        for (int q = 1; q < kThreads / 32; q++) v = combine(v, wsum[q][lane], MODE);
        reinterpret_cast<PT*>(sr->partials)[(size_t)(word & 0xffffu) * kPartials + lane] = v;
        __threadfence();
      }
      __syncwarp();
      unsigned t = 0u;
      if (lane == 0) t = atomicAdd(sr->icp_counter, 1u);
      t = __shfl_sync(0xffffffffu, t, 0);
      const bool last = t == (unsigned)ranges - 1u;
      if (lane == 0) {
        s_close = last;
        if (last) {
          __threadfence();  // the block reads the other ranges' partials after the arrivals
          *sr->icp_counter = 0u;
        }
      }
      if (!last) claim(slot);
    }
    __syncthreads();
    if (s_close) {
      // ---- last range of this iteration: no claim was made, so the range
      // stands until the one after the closing (and its barrier) ----
      const int slot = reload(&s_slot);
      const unsigned word = reload(&s_word);
      const SessionDev* sr = reload(&sS[slot]);
      const int ranges = reload(&sNvb[word >> 30][slot]);
      const unsigned next = close_iteration<MODE>(sr, ranges, (int)(word >> 30), (int)((word >> 16) & 0x3fffu));
      if (warp == 0) {
        if (lane == 0) atomicExch(words + slot, next);
        claim((next >> 30) == kWordDone ? -1 : slot);
      }
      __syncthreads();
    }
  }
}

__global__ void k_pose_set(SessionDev* s, const double* T) {
  Pose* P = s->pose;
  const int ln = threadIdx.x;
  __shared__ double Tn[16];
  if (ln < 16) Tn[ln] = T[ln];
  __syncwarp();
  double Ti;
  warp_rigid_inverse(Tn, ln, Ti);
  if (ln < 16) {
    P->T_gc[ln] = Tn[ln];
    P->Tgc[ln] = (float)Tn[ln];
    P->Tcg[ln] = (float)Ti;
  }
  if (ln == 3 || ln == 7 || ln == 11) P->center[ln >> 2] = (float)Ti;
}

// the 80-byte pose heads (float pose, tracked, iterations, count, frame) of
// every slot, packed slot after slot for one device-to-host copy
__global__ void k_gather_heads(const BatchTable* __restrict__ bt, uint32_t* __restrict__ out) {
  const int slot = blockIdx.x;
  if (slot >= bt->n) return;
  constexpr int kWords = (int)(kPoseHeadBytes / 4);
  const uint32_t* src = reinterpret_cast<const uint32_t*>(bt->s[slot]->pose);
  if (threadIdx.x < kWords) out[slot * kWords + threadIdx.x] = src[threadIdx.x];
}

}  // namespace

void launch_gather_heads(const BatchTable* bt, void* out, cudaStream_t st) {
  k_gather_heads<<<kMaxSlots, 32, 0, st>>>(bt, reinterpret_cast<uint32_t*>(out));
}

// pixels per ICP range at level 0 and at the coarser levels.  A range is
// the unit between two block barriers and one partial write: long ranges
// spend less of the launch in barriers and reductions, short ranges keep
// more blocks busy on the small coarse levels (and on a lone session).
#ifndef VS_ICP_PIXELS_PER_RANGE
#define VS_ICP_PIXELS_PER_RANGE 2048
#endif
#ifndef VS_ICP_PIXELS_PER_RANGE_COARSE
#define VS_ICP_PIXELS_PER_RANGE_COARSE 512
#endif

int icp_blocks(int npix, int level) {
  const int ppr = level == 0 ? VS_ICP_PIXELS_PER_RANGE : VS_ICP_PIXELS_PER_RANGE_COARSE;
  int b = (npix + ppr - 1) / ppr;
  if (b < 1) b = 1;
  if (b > kIcpMaxBlocks) b = kIcpMaxBlocks;
  return b;
}

// An SM divides its storage between L1 and shared memory when its first block
// arrives and keeps the division while a block runs.  By default it suits the
// 4 to 6 KB of this launch's blocks, which then hold their SMs for the whole of
// the tracking: kernels of a batch's other branch that need more (the scan of
// the input maps, the update's partial sums, the filter) found no SM and the
// branches ran one after the other.  With 40 % of the storage as shared memory
// they fit beside: steps of 8, 12, 16 and 24 sessions 850 -> 725, 1172 -> 1018,
// 1302 -> 1172 and 1766 -> 1655 us; of 1 and 64 the same.  (15 and 25 % the same
// within 1 %; 60 and 100 % leave L1 too little, 1.5 and 3 % more with one
// session or 64 of them.)
cudaError_t configure_icp_kernels() {
  constexpr int kShared = 40;
  for (auto k : {k_icp_run<VS_REDUCE_FP32>, k_icp_run<VS_REDUCE_KAHAN>, k_icp_run<VS_REDUCE_FP64>}) {
    const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, kShared);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

void launch_icp(const BatchTable* bt, int reduce_mode, cudaStream_t st, bool frame_mode, const float* init_T12) {
  // frame-level calls skip tracking on the first frame as so_Scan_Object does
  // (zz_flag_track, z_yooji_object_scanner.cpp:534,572-576); explicit
  // tp_Track_Pose calls always track
  unsigned* words = const_cast<unsigned*>(bt->icp_word);
  k_icp_begin<<<kMaxSlots, 32, 0, st>>>(bt, words, frame_mode ? 1 : 0, init_T12 ? 1 : 0, init_T12);
  // Two of the three blocks that fit an SM: the rest of each SM takes the
  // other branch's kernels while this launch waits for a closer.  (Sixteen
  // sessions, two branches: 1955 us per step with three blocks, 1894 with
  // two, 1922 with one and a half; 64 sessions 5990, 5970, 5925; one session
  // the same.)
  const int grid = sm_count() * 2;
  switch (reduce_mode) {
    case VS_REDUCE_FP32:
      k_icp_run<VS_REDUCE_FP32><<<grid, kThreads, 0, st>>>(bt, words);
      break;
    case VS_REDUCE_FP64:
      k_icp_run<VS_REDUCE_FP64><<<grid, kThreads, 0, st>>>(bt, words);
      break;
    default:
      k_icp_run<VS_REDUCE_KAHAN><<<grid, kThreads, 0, st>>>(bt, words);
      break;
  }
}

void launch_pose_set(const SessionDev* d, const double* T_gc, cudaStream_t st) {
  k_pose_set<<<1, 32, 0, st>>>(const_cast<SessionDev*>(d), T_gc);
}

}  // namespace vs
