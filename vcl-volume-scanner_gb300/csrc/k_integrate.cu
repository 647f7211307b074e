// TSDF integration: sub-cube activation + gated update of the active bricks.
//
// Reference: g_fvsc_Find_Visible_Sub_Cubes and g_ctvc_Compute_TSDF_of_Voxels
// _with_Color (STAC/Engine/GPU/z_yooji_cuda_volume_integrator.cu:84-152,
// 265-402, host :976-1031).  The reference resets a byte flag per 8^3
// sub-cube, marks the sub-cubes that lie on every depth ray between 4 mu in
// front of and 1 mu behind the measured point, then runs one thread per
// sub-cube over its 512 voxels in the x-fastest global layout: uncoalesced,
// and most threads of its 512x512x1-voxel launch grid idle.
//
// GB300 layout: the volume is stored as bricks (one brick = one sub-cube =
// 512 consecutive 32-bit words, 2 KB), so an active sub-cube is one
// contiguous, perfectly coalesced 2 KB read and write.  Activation appends a
// brick to a compact list the first time its flag flips (atomicExch), and the
// update kernel is persistent: one warp per listed brick (or 2, 4 warps where
// the bricks are few), 16-byte vector loads, 16 voxels per lane.  Flags hold a
// stamp per integration, so no full-volume pass touches HBM.  Voxel centres and the per-pixel
// ray scale K^-1 [x y 1] come from per-session tables built once with the
// same IEEE operations as the per-voxel reference formula, so the result
// stays bit-identical while the divisions leave the inner loop.
//
// Batches: activation is persistent over the level-0 tiles of every session
// of a batch table, each session filling its own brick list; the update
// kernel walks the concatenation of the lists (a brick touches only its own
// session's voxels, so the order across sessions changes no result).
#include <cuda_runtime.h>
#include <stdint.h>

#include "vs_internal.cuh"

namespace vs {
namespace {

constexpr int kIntThreads = 256;
constexpr int kActBlocks = 5;      // resident activation blocks per SM (48 registers a thread, no spills)
constexpr int kMaxDimLut = 1024;   // voxels per axis (bricks fit 21 index bits)
constexpr int kMaxImgLut = 2048;   // pixels per image axis

// 1 / w for every weight an update can produce (w = 1..65535), IEEE-rounded
// exactly as the division it replaces
__device__ float g_inv_weight[65536];

// per-session tables: voxel centre coordinate per axis
// (d_gpw_Get_Position_in_World), the level-0 ray components K^-1 [x y 1] and,
// when kept, the per-pixel ray scale lambda^-1 = 1 / |K^-1 [x y 1]| of
// g_ctvc (z_yooji_cuda_volume_integrator.cu:357-372), each with the
// reference's own operations
__device__ __forceinline__ void session_tables(const SessionDev& s, int i) {
  const int d0 = s.dim[0], d1 = s.dim[1], d2 = s.dim[2];
  if (i < d0) s.lut_vox[i] = ((float)i + 0.5f) / s.vox_inv + s.origin[0];
  if (i < d1) s.lut_vox[d0 + i] = ((float)i + 0.5f) / s.vox_inv + s.origin[1];
  if (i < d2) s.lut_vox[d0 + d1 + i] = ((float)i + 0.5f) / s.vox_inv + s.origin[2];
  const float* K = s.lv[0].K;
  const int W = s.lv[0].W, H = s.lv[0].H;
  if (i < W) s.lut_ray[i] = 1.0f * ((float)i - K[2]) / K[0];
  if (i < H) s.lut_ray[W + i] = 1.0f * ((float)i - K[3]) / K[1];
  if (i < 65536) g_inv_weight[i] = 1.0f / (float)i;
  if (s.lam_map && i < W * H) {
    const int x = i % W, y = i / W;
    const float rx = 1.0f * ((float)x - K[2]) / K[0], ry = 1.0f * ((float)y - K[3]) / K[1];
    s.lam_map[i] = 1.0f / sqrtf(rx * rx + ry * ry + 1.0f);
  }
}
__global__ void k_session_tables(const SessionDev* __restrict__ s) {
  session_tables(*s, blockIdx.x * blockDim.x + threadIdx.x);
}

// The set-up of a call that brings its own volume: the descriptor and the
// one-slot work table (kernel arguments) into their scratch, its tables, and
// its counters and activation flags cleared
__global__ void k_call_setup(const __grid_constant__ SessionDev h, const __grid_constant__ BatchTable t, SessionDev* d,
                             BatchTable* dt, uint32_t nbr) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  constexpr uint32_t kHw = sizeof(SessionDev) / 4, kTw = sizeof(BatchTable) / 4;
  static_assert(sizeof(SessionDev) % 4 == 0 && sizeof(BatchTable) % 4 == 0, "word copies");
  static_assert(sizeof(SessionDev) + sizeof(BatchTable) + 64 <= 32764, "arguments exceed the parameter space");
  if (i < kHw) reinterpret_cast<uint32_t*>(d)[i] = reinterpret_cast<const uint32_t*>(&h)[i];
  if (i < kTw) reinterpret_cast<uint32_t*>(dt)[i] = reinterpret_cast<const uint32_t*>(&t)[i];
  if (i < kBrickCounters) h.brick_count[i] = 0u;
  for (uint32_t k = i; k < nbr; k += gridDim.x * blockDim.x) h.brick_flag[k] = 0u;
  session_tables(h, (int)i);
}

// The counters of a session (brick_count), handed from one integration's two
// kernels to the next integration's, so that no launch stands between them to
// clear them:
//   [0] active bricks, [1] voxels updated, of the last integration
//   [2] activation stamp of the last integration (0: none yet)
//   [3] which of the two list counters, [4] or [5], the next one counts in
//   [6] what activation found: that choice, or kNoUpdate; [7] its new stamp
// Activation reads [2] and [3], counts in [4] or [5], and writes [1], [6] and
// [7]; the update reads [4] to [7], and writes [0], [2], [3] and, for the next
// time, the other list counter.  A session whose tracking failed (gate) does
// not integrate and keeps its stamp and flags.
//
// A brick's flag holds the stamp of the last integration that activated it, so
// no pass clears flags: the flagged set of the last integration is {b :
// flag[b] == stamp != 0}, the reference's per-sub-cube bytes (cube_valid)
// after its reset and marking (z_yooji_cuda_volume_integrator.cu:1006-1016),
// which g_uvv_Update_Valid_Volume visits later.
constexpr uint32_t kNoUpdate = 2u;

// What activation needs of a session, in shared memory: a block's rows nearly
// all belong to one session.
struct __align__(16) ActSession {
  float4 T[3];                 // T_cg
  float4 K;
  float4 grid;                 // volume origin, 1 / voxel size
  float4 edge;                 // dim - 0.5 per axis, mu
  int nb[3];
  uint32_t stamp;
  int W, H, tw, skip;
  const float* depth;
  uint32_t* flags;
  uint32_t* list;
  uint32_t* count;
  uint8_t* band;
};

__device__ inline void load_session(ActSession& a, const SessionDev* __restrict__ s, const float* depth_ext,
                                    const float* Tcg_ext, bool gate, bool dry, bool first) {
  const float* __restrict__ T = Tcg_ext ? Tcg_ext : s->pose->Tcg;
#pragma unroll
  for (int k = 0; k < 3; k++) a.T[k] = make_float4(T[4 * k], T[4 * k + 1], T[4 * k + 2], T[4 * k + 3]);
  const float* K = s->lv[0].K;
  a.K = make_float4(K[0], K[1], K[2], K[3]);
  a.grid = make_float4(s->origin[0], s->origin[1], s->origin[2], s->vox_inv);
  a.edge = make_float4((float)s->dim[0] - 0.5f, (float)s->dim[1] - 0.5f, (float)s->dim[2] - 0.5f, s->mu);
  for (int k = 0; k < 3; k++) a.nb[k] = s->nb[k];
  a.stamp = s->brick_count[2] + 1u;
  if (a.stamp == 0u) a.stamp = 1u;
  const uint32_t turn = s->brick_count[3];
  a.W = s->lv[0].W;
  a.H = s->lv[0].H;
  a.tw = (a.W + 31) / 32;
  a.skip = gate && s->pose->failed;
  a.depth = depth_ext ? depth_ext : s->depth_raw;
  a.flags = s->brick_flag;
  a.list = s->brick_list;
  a.count = s->brick_count + 4 + turn;
  a.band = dry ? nullptr : s->band;
  if (first) {
    s->brick_count[1] = 0u;
    s->brick_count[6] = a.skip ? kNoUpdate : turn;
    s->brick_count[7] = a.stamp;
  }
}

__device__ __forceinline__ F3 transform(F3 p, const float4 (&T)[3]) {
  return f3(T[0].x * p.x + T[0].y * p.y + T[0].z * p.z + T[0].w, T[1].x * p.x + T[1].y * p.y + T[1].z * p.z + T[1].w,
            T[2].x * p.x + T[2].y * p.y + T[2].z * p.z + T[2].w);
}

// A block takes a contiguous run of tiles, so the session's values are read
// once; a lane takes one pixel of each of its rows.  A pixel's six sub-cubes
// are computed first and their flags read together: read one after the other,
// each paid the L2's latency, and so did the exchanges and the claims of list
// places.  Lanes of a run that meet the same unlisted sub-cube leave the
// exchange to the first.  A 640x480 frame: 11.7 us (15.4 one after the other,
// one tile per block); 431x333: 8.3 (11.1).
__global__ void __launch_bounds__(256, kActBlocks) k_activate(const BatchTable* __restrict__ bt,
                                                                 const float* __restrict__ depth_ext,
                                                                 const float* __restrict__ Tcg_ext, int gate,
                                                                 int dry) {
  __shared__ ActSession a;
  const int n = bt->n;
  const int total = bt->bil[n];
  const int rows = bt->bil_rows;
  const int lane = threadIdx.x;
  const int first = (int)((long long)blockIdx.x * total / gridDim.x);
  const int end = (int)((long long)(blockIdx.x + 1) * total / gridDim.x);
  if (first >= end) return;
  int t0;
  int slot = find_slot(bt->bil, n, first, t0);
  int next = first - t0;  // first tile of the next session to load
  int base = next;
  slot--;
  for (int item = first; item < end; item++) {
    if (item >= next) {
      do next = bt->bil[++slot + 1];
      while (item >= next);
      base = bt->bil[slot];
      __syncthreads();
      // the block of the session's first tile passes on what the update needs
      if (threadIdx.x == 0 && threadIdx.y == 0)
        load_session(a, bt->s[slot], depth_ext, Tcg_ext, gate != 0, dry != 0, item == base);
      __syncthreads();
    }
    if (a.skip) {
      item = next - 1;
      continue;
    }
    const int t = item - base;
    const int x = (t % a.tw) * 32 + lane, yt = (t / a.tw) * rows;
    for (int ty = threadIdx.y; ty < rows; ty += blockDim.y) {
      const int y = yt + ty;
      if (y >= a.H) break;
      const float td = x < a.W ? a.depth[(size_t)y * a.W + x] : 0.0f;
      int b[6];
#pragma unroll
      for (int k = 0; k < 6; k++) b[k] = -1;
      if (td > 0.0f) {
        const float K[4] = {a.K.x, a.K.y, a.K.z, a.K.w};
        const F3 p = transform(back_project((float)x, (float)y, K, td), a.T);
        const F3 pe = transform(back_project((float)x, (float)y, K, 100.0f), a.T);
        const F3 dv = normalised(sub(pe, p));
        int prev = -1;
        bool on = true;  // false once a sub-cube index left the grid
#pragma unroll
        for (int k = 0; k < 6; k++) {
          // pos_in_voxel
          const F3 q = add(p, scale((float)(k - 4) * a.edge.w, dv));
          const float vx = (q.x - a.grid.x) * a.grid.w - 0.5f, vy = (q.y - a.grid.y) * a.grid.w - 0.5f,
                      vz = (q.z - a.grid.z) * a.grid.w - 0.5f;
          const float low = fminf(fminf(vx, vy), vz);
          const bool in = !(low < -0.5f || vx >= a.edge.x || vy >= a.edge.y || vz >= a.edge.z);
          // ROUNDF(v)/8 as the unparenthesised reference macro evaluates it
          // (z_yooji_cuda_volume_integrator.cu:133-135), (int)(v - 0.5) for
          // v < 0 and (int)(v + 0.5) / 8 above: with v >= -0.5 the first is -1
          // (off the grid) where v - 0.5 reaches -1, else 0 like the second
          const int xs = (int)(vx + 0.5f) >> 3, ys = (int)(vy + 0.5f) >> 3, zs = (int)(vz + 0.5f) >> 3;
          on = on && !(in && (low - 0.5f <= -1.0f || xs >= a.nb[0] || ys >= a.nb[1] || zs >= a.nb[2]));
          const int c = (zs * a.nb[1] + ys) * a.nb[0] + xs;
          if (on && in && c != prev) b[k] = prev = c;
        }
      }
      // an L1-cached read of the flag may be stale, but only ever with an
      // older stamp, and the exchange then decides: it returns the current
      // stamp to every thread but the first
      uint32_t was[6];
      bool any = false;
#pragma unroll
      for (int k = 0; k < 6; k++) {
        was[k] = b[k] >= 0 ? a.flags[b[k]] : a.stamp;
        any |= was[k] != a.stamp;
      }
      if (!__any_sync(0xffffffffu, any)) continue;
#pragma unroll
      for (int k = 0; k < 6; k++) {
        const int mine = was[k] != a.stamp ? b[k] : -1;
        const int left = __shfl_up_sync(0xffffffffu, mine, 1);
        was[k] = (mine >= 0 && (lane == 0 || left != mine)) ? atomicExch(a.flags + mine, a.stamp) : a.stamp;
      }
      // one claim of list places for the warp
      unsigned won = 0u;
#pragma unroll
      for (int k = 0; k < 6; k++) won += __popc(__ballot_sync(0xffffffffu, was[k] != a.stamp));
      if (won == 0u) continue;
      uint32_t pos = 0u;
      if (lane == 0) pos = atomicAdd(a.count, won);
      pos = __shfl_sync(0xffffffffu, pos, 0);
#pragma unroll
      for (int k = 0; k < 6; k++) {
        const bool mine = was[k] != a.stamp;
        const unsigned m = __ballot_sync(0xffffffffu, mine);
        if (mine) {
          a.list[pos + __popc(m & ((1u << lane) - 1u))] = (uint32_t)b[k];
          // the update sets the flag of a brick that holds a band voxel
          if (a.band) a.band[b[k]] = 0;
        }
        pos += __popc(m);
      }
    }
  }
}

// What the update needs of a session, one copy per warp in shared memory: a
// warp's bricks nearly always belong to one session, the reads are broadcasts
// of some 30 cycles, and no register holds a value between its uses.
struct __align__(16) IntSession {
  float T[12];              // T_gc
  float C[3], mu;           // camera centre
  float K[4];
  float inv_mu, max_w;
  int W, H;
  uint32_t nb0, nb1, by_nb0, by_nb1;  // brick grid; ceil(2^31 / nb0), ceil(2^31 / nb1)
  const float* lut[3];      // voxel centres of the three axes
  const float* ray;         // level-0 ray components, columns then rows
  // depth source: the session's packed {depth, lambda^-1} map (packed), or a
  // depth map with the lambda^-1 map beside it (lam) or without (NULL:
  // computed per voxel from the ray table)
  const void* src;
  const float* lam;
  const uint32_t* list;
  uint32_t* counters;
  void* vol;
  uint8_t* band;
  uint32_t* occ;
  uint32_t* col;            // colour bricks (NULL: no colour)
  const uint32_t* rgb;      // packed colour frame
  int packed;
  int fast;                 // principal point within the bound of nearest_pixel's fast path
};

__device__ inline void load_session(IntSession& q, const SessionDev* __restrict__ s, const float* depth_ext,
                                    const float* Tgc_ext, const float* Tcg_ext, bool color) {
  const float* __restrict__ Tgc = Tgc_ext ? Tgc_ext : s->pose->Tgc;
  const float* __restrict__ Tcg = Tcg_ext ? Tcg_ext : s->pose->Tcg;
#pragma unroll
  for (int k = 0; k < 12; k++) q.T[k] = Tgc[k];
#pragma unroll
  for (int k = 0; k < 3; k++) q.C[k] = Tcg[4 * k + 3];
#pragma unroll
  for (int k = 0; k < 4; k++) q.K[k] = s->lv[0].K[k];
  q.mu = s->mu;
  q.inv_mu = 1.0f / s->mu;
  q.max_w = s->max_w;
  q.W = s->lv[0].W;
  q.H = s->lv[0].H;
  q.nb0 = (uint32_t)s->nb[0];
  q.nb1 = (uint32_t)s->nb[1];
  q.by_nb0 = (0x80000000u + q.nb0 - 1u) / q.nb0;
  q.by_nb1 = (0x80000000u + q.nb1 - 1u) / q.nb1;
  q.lut[0] = s->lut_vox;
  q.lut[1] = s->lut_vox + s->dim[0];
  q.lut[2] = s->lut_vox + s->dim[0] + s->dim[1];
  q.ray = s->lut_ray;
  q.packed = !depth_ext && s->dl_map;
  const float* depth = depth_ext ? depth_ext : s->depth_raw;
  q.src = q.packed ? static_cast<const void*>(s->dl_map) : static_cast<const void*>(depth);
  q.lam = q.packed ? nullptr : s->lam_map;
  q.list = s->brick_list;
  q.counters = s->brick_count;
  q.vol = s->vol;
  q.band = s->band;
  q.occ = s->occ;
  q.col = color ? s->col : nullptr;
  q.rgb = s->rgb_packed;
  q.fast = fabsf(q.K[2]) < 4096.0f && fabsf(q.K[3]) < 4096.0f;
}

// a / nb for a < 2^21 and nb <= 128, m = ceil(2^31 / nb): a m / 2^31 exceeds
// a / nb by less than a / 2^31 < 2^-10, less than the 1 / nb that separates
// it from the next integer
__device__ __forceinline__ uint32_t div_small(uint32_t a, uint32_t m) {
  return (uint32_t)(((unsigned long long)a * m) >> 31);
}

// The colour part of g_ctvc (z_yooji_cuda_volume_integrator.cu:404-455, the
// registered-colour path): for every voxel of the round whose depth was just
// updated, the colour at its projection, interpolated as
// d_gii_Get_Interpolated_Intensity (_yooji_cuda_math.h:305-332) per channel,
// is blended as (w * old + sample) / (w + 1) and truncated to 8 bits.  When a
// channel cannot be interpolated (outside the image, or a used texel <= 0) the
// voxel keeps its colour (the reference would blend an uninitialised value).
// The four taps and the old colour of four voxels are read in one round.
__device__ inline bool interp_channel(uint32_t a, uint32_t b, uint32_t c, uint32_t d, int k, float rx, float ry,
                                      float& out) {
  const float d1 = (float)rgb_channel(a, k);
  if (d1 <= 0.0f) return false;
  float d2 = 0.0f, d3 = 0.0f, d4 = 0.0f;
  if (rx > 0.0f) {
    d2 = (float)rgb_channel(b, k);
    if (d2 <= 0.0f) return false;
  }
  if (ry > 0.0f) {
    d3 = (float)rgb_channel(c, k);
    if (d3 <= 0.0f) return false;
  }
  if (rx > 0.0f && ry > 0.0f) {
    d4 = (float)rgb_channel(d, k);
    if (d4 <= 0.0f) return false;
  }
  out = (1.0f - ry) * ((1.0f - rx) * d1 + rx * d2) + ry * ((1.0f - rx) * d3 + rx * d4);
  return true;
}

// wv: the round's words, [vector][voxel in vector]; v0: the lane's index of
// the round's first voxel.  A vector's colour words are 16 (or 8) consecutive
// bytes of the brick's colour and are read and written together; the words of
// its other voxels are stored back as they were read (a brick's round has one
// writer).
template <class S, int kPerVec, int kRound, class WV>
__device__ __forceinline__ void color_round(const IntSession& q, unsigned upd, int v0, int lane, int bx, int by, int bz,
                                            uint32_t b, const WV& wv) {
  constexpr int kV = kRound / kPerVec;
  uint32_t t00[kRound], t01[kRound], t10[kRound], t11[kRound], oc[kRound];
  float rxs[kRound], rys[kRound];
  bool ok[kRound];
#pragma unroll
  for (int v = 0; v < kV; v++) {
    const uint32_t* src = q.col + (size_t)b * kBrickVox + ((v0 / kPerVec + v) * 32 + lane) * kPerVec;
    if (kPerVec == 4) {
      const uint4 w = *reinterpret_cast<const uint4*>(src);
      oc[v * kPerVec] = w.x;
      oc[v * kPerVec + 1] = w.y;
      oc[v * kPerVec + 2 % kPerVec] = w.z;
      oc[v * kPerVec + 3 % kPerVec] = w.w;
    } else {
      const uint2 w = *reinterpret_cast<const uint2*>(src);
      oc[v * kPerVec] = w.x;
      oc[v * kPerVec + 1] = w.y;
    }
  }
#pragma unroll
  for (int j = 0; j < kRound; j++) {
    ok[j] = false;
    if (!((upd >> j) & 1u)) continue;
    const int li = ((v0 / kPerVec + j / kPerVec) * 32 + lane) * kPerVec + j % kPerVec;
    const int xc = bx * 8 + (li & 7), yc = by * 8 + ((li >> 3) & 7), zc = bz * 8 + (li >> 6);
    const F3 pg = f3(__ldg(q.lut[0] + xc), __ldg(q.lut[1] + yc), __ldg(q.lut[2] + zc));
    float u, vv;
    project(transform(pg, q.T), q.K, u, vv);
    if (!(u >= 0.0f && u <= (float)(q.W - 1) && vv >= 0.0f && vv <= (float)(q.H - 1))) continue;
    const int x = (int)u, y = (int)vv;
    rxs[j] = u - (float)x;
    rys[j] = vv - (float)y;
    const int xb = rxs[j] > 0.0f ? x + 1 : x, yb = rys[j] > 0.0f ? y + 1 : y;
    t00[j] = __ldg(q.rgb + y * q.W + x);
    t01[j] = __ldg(q.rgb + y * q.W + xb);
    t10[j] = __ldg(q.rgb + yb * q.W + x);
    t11[j] = __ldg(q.rgb + yb * q.W + xb);
    ok[j] = true;
  }
#pragma unroll
  for (int v = 0; v < kV; v++) {
    bool put = false;
#pragma unroll
    for (int e = 0; e < kPerVec; e++) {
      const int j = v * kPerVec + e;
      if (!ok[j]) continue;
      float tn;
      uint32_t wn;
      S::decode(wv[v][e], tn, wn);  // the updated word: weight w + 1
      const float oldW = (float)(wn - 1u), inewW = __ldg(g_inv_weight + wn);
      float smp[3];
      bool good = true;
#pragma unroll
      for (int c = 0; c < 3; c++) good &= interp_channel(t00[j], t01[j], t10[j], t11[j], c, rxs[j], rys[j], smp[c]);
      if (!good) continue;
      uint32_t ch[3];
#pragma unroll
      for (int c = 0; c < 3; c++)
        ch[c] = (uint32_t)(uint8_t)(fmaxf(0.0f, fminf(255.0f, (oldW * (float)rgb_channel(oc[j], c) + smp[c]) * inewW)));
      oc[j] = pack_rgb(ch[0], ch[1], ch[2]);
      put = true;
    }
    if (!put) continue;
    uint32_t* dst = q.col + (size_t)b * kBrickVox + ((v0 / kPerVec + v) * 32 + lane) * kPerVec;
    if (kPerVec == 4)
      *reinterpret_cast<uint4*>(dst) = make_uint4(oc[v * kPerVec], oc[v * kPerVec + 1], oc[v * kPerVec + 2 % kPerVec],
                                                  oc[v * kPerVec + 3 % kPerVec]);
    else
      *reinterpret_cast<uint2*>(dst) = make_uint2(oc[v * kPerVec], oc[v * kPerVec + 1]);
  }
}

// Resident 256-thread blocks per SM: 64 registers without spills at 4 (5
// spills, 38.7 instead of 29.6 us for the 640x480 frame below; 3 leaves too few
// warps, 33.9), 80 registers at 3 for the colour variant (a 384^3 colour frame
// 51.9 us; 57.8 at 2, 58.5 at 4).
constexpr int kIntBlocks = 4, kIntColorBlocks = 3;

// log2 of the parts (1, 2 or 4 warps) that a brick's update is split in: the
// shift with the least waves x cost, where an item costs 1 (brick set-up) + 3
// per round of four voxels a lane.  The costs are from the update of a 640x480
// frame, 8,867 bricks on 4,864 warps: 30.2 us whole, 32.0 in halves, 35.8 in
// quarters; with about 3,000 bricks 16.6 whole and 14.2 in quarters.
__device__ __forceinline__ int part_shift(uint32_t total, uint32_t nwarps) {
  int best = 0;
  uint32_t least = 0xffffffffu;
#pragma unroll
  for (int ps = 0; ps < 3; ps++) {
    const uint32_t cost = (((total << ps) + nwarps - 1) / nwarps) * (1u + (12u >> ps));
    if (cost < least) {
      least = cost;
      best = ps;
    }
  }
  return best;
}

// Nearest pixel of a camera-frame point: (__float2int_rn(u), __float2int_rn(v))
// of d_p_Project's u = K0 x / z + K2, v = K1 y / z + K3 with IEEE division
// (_yooji_cuda_math.h:205-210, z_yooji_cuda_volume_integrator.cu:344-347),
// bit for bit, at the price of a reciprocal instead of two divisions for all
// but a few voxels.
//
// u' = RN(RN(K0 x * rcp(z)) + K2) differs from u = RN(RN(K0 x / z) + K2) by
// at most 2^-22 |K0 x / z| + ulp(u): rcp has at most 1 ulp of error and each
// product / sum one rounding.  A pixel inside an image of at most 2048
// columns needs |u| < 2048, so |K0 x / z| < 2048 + |K2| < 6144 when
// |K2| < 4096, and |u' - u| < 1.5e-3 + 2.5e-4 < 2^-8 =: m.  If u' is farther
// than m from every half-integer, no rounding boundary lies between u and
// u', so rint(u') = rint(u).  Otherwise, and for z <= 1e-4 (or NaN), the
// IEEE divisions run.  (Outside the image both forms give columns out of
// range, where the exact value does not matter.)  `fast` is false when the
// principal point is out of the bound.
__device__ __forceinline__ void nearest_pixel(float x, float y, float z, const float* K, bool fast, int& px,
                                              int& py) {
  constexpr float kEdge = 0.5f - 1.0f / 256.0f;
  const float a = K[0] * x, b = K[1] * y;
  float u = 0.0f, v = 0.0f;
  bool exact = !(fast && z > 1e-4f);
  if (!exact) {
    const float r = rcp_approx(z);
    u = a * r + K[2];
    v = b * r + K[3];
    exact = fabsf(u - rintf(u)) > kEdge || fabsf(v - rintf(v)) > kEdge;
  }
  if (exact) {
    u = a / z + K[2];
    v = b / z + K[3];
  }
  px = __float2int_rn(u);
  py = __float2int_rn(v);
}

// g_ctvc's depth update, per voxel in the reference's operation order
// (z_yooji_cuda_volume_integrator.cu:340-402): world centre p_g, camera point
// T_gc p_g, nearest pixel, depth d; lambda^-1 |p_g - C|; sdf = d - that;
// skip if sdf < -mu; tsdf = min(1, sdf / mu); weighted mean with the old
// value; weight + 1.  The weights and the skip decisions are bit-identical
// to that order.  Two rewrites that keep every rounding:
//  * a lane's voxels share their y coordinate, take kPerVec x and kLaneVec
//    z values, so the partial sums M0 x + M1 y (and M4, M8 rows) and
//    (x - Cx)^2 + (y - Cy)^2 are formed once per x value, and the rest of
//    each sum is added in the same order as the full expression;
//  * the pixel rounding uses nearest_pixel above.
// The one change of a rounding: sdf / mu is the product with 1 / mu and one
// Markstein correction step (q = s r; e = fma(-q, mu, s); q + e r, P.
// Markstein, IBM J. Res. Dev. 34(1), 1990), which returns the IEEE quotient in
// all but rare cases and otherwise differs by one ulp (6e-8 of a TSDF value,
// below 0.002 of an int16 step), inside the one-step tolerance.
//
// Bound by latency, then by issue (some 130 instructions a voxel): every load
// of a round is issued before the round's square roots, session values come
// from shared memory, and the rounds share one copy of the code.  A 640x480
// frame into 512^3 (8,867 bricks): 29.6 us, of which 16 are issue slots; 59.8
// with per-voxel loads in branches, session values re-read from L2 at each
// brick and unrolled rounds.  A 384^3 colour frame: 51.9 us (80.6).
template <class S, bool COLOR>
__global__ void __launch_bounds__(kIntThreads, COLOR ? kIntColorBlocks : kIntBlocks)
    k_integrate(const BatchTable* __restrict__ bt, const float* __restrict__ depth_ext,
                const float* __restrict__ Tgc_ext, const float* __restrict__ Tcg_ext, int color, int dry) {
  __shared__ uint32_t pre[kMaxSlots + 1];  // prefix of the slots' active-brick counts
  __shared__ IntSession ses[kIntThreads / 32];
  // per thread, per x value of its voxels: the transform rows' partial sums
  // M0 x + M1 y, M4 x + M5 y, M8 x + M9 y and (x - Cx)^2 + (y - Cy)^2
  // ([x value][thread]: a warp's 16-byte reads are consecutive, no bank conflicts)
  __shared__ float4 xpart[16 / sizeof(typename S::word)][kIntThreads];
  const int n = bt->n;
  if (threadIdx.x < 32) {
    const int ln = threadIdx.x;
    auto listed = [&](int i) -> uint32_t {
      if (i >= n) return 0u;
      uint32_t* bc = bt->s[i]->brick_count;
      const uint4 c = __ldcg(reinterpret_cast<const uint4*>(bc) + 1);  // [4] to [7]
      const uint32_t count = c.z == kNoUpdate ? 0u : c.z ? c.y : c.x;
      if (blockIdx.x == 0) {  // nothing in this launch reads these
        bc[0] = count;
        if (c.z != kNoUpdate) {
          bc[2] = c.w;
          bc[3] = c.z ^ 1u;
          bc[4 + (c.z ^ 1u)] = 0u;
        }
      }
      return count;
    };
    const uint32_t c0 = listed(2 * ln), c1 = listed(2 * ln + 1);
    uint32_t v = c0 + c1;
#pragma unroll
    for (int m = 1; m < 32; m <<= 1) {
      const uint32_t o = __shfl_up_sync(0xffffffffu, v, m);
      if (ln >= m) v += o;
    }
    pre[2 * ln + 2] = v;
    pre[2 * ln + 1] = v - c1;
    if (ln == 0) pre[0] = 0u;
  }
  __syncthreads();
  const uint32_t total = pre[n];

  typedef typename S::word word;
  constexpr int kPerVec = 16 / sizeof(word);    // voxels per 16-byte vector, consecutive in x
  constexpr int kVecs = kBrickVox / kPerVec;    // 16-byte vectors per brick
  constexpr int kLaneVec = kVecs / 32;          // vectors per lane, one z value each
  constexpr int kRV = 4 / kPerVec > 0 ? 4 / kPerVec : 1;  // 16-byte vectors per round
  constexpr int kRound = kRV * kPerVec;                    // 4 voxels per round, gathers in flight together
  constexpr int kRounds = kLaneVec / kRV;
  static_assert(kRounds == 4, "a brick is split in 1, 2 or 4 parts");
  const int lane = threadIdx.x & 31;
  const uint32_t gwarp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
  const int ps = part_shift(total, nwarps);
  const uint32_t items = total << ps;
  const int rounds = kRounds >> ps;
  // the lane's voxel coordinates inside a brick: word (k * 32 + lane) * kPerVec + e
  // is x = x0 + e, y = y0, z = z0 + k * kPerVec / 2
  const int x0 = (lane * kPerVec) & 7, y0 = ((lane * kPerVec) >> 3) & 7, z0 = (lane * kPerVec) >> 6;
  constexpr int kZStep = kPerVec / 2;
  IntSession& q = ses[threadIdx.x >> 5];
  int slot = -1;

  for (uint32_t i = gwarp; i < items; i += nwarps) {
    const uint32_t at = i >> ps;
    int lo = 0, hi = n - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (pre[mid] <= at)
        lo = mid;
      else
        hi = mid - 1;
    }
    __syncwarp();
    if (lo != slot) {
      slot = lo;
      if (lane == 0) load_session(q, bt->s[lo], depth_ext, Tgc_ext, Tcg_ext, COLOR && color);
      __syncwarp();
    }
    const uint32_t b = __ldcg(q.list + (at - pre[lo]));
    int nupd = 0;
    bool band = false;  // some voxel of the part, after the update, is a band voxel
    const uint32_t byz = div_small(b, q.by_nb0);
    const int bx = (int)(b - byz * q.nb0);
    const int bz = (int)div_small(byz, q.by_nb1);
    const int by = (int)(byz - (uint32_t)bz * q.nb1);
    uint4* bv = reinterpret_cast<uint4*>(reinterpret_cast<word*>(q.vol) + (size_t)b * kBrickVox) + lane;
    const int r0 = (int)(i & ((1u << ps) - 1u)) * rounds, r1 = r0 + rounds;
    // Rounds of kRV vectors (4 voxels): the next round's vectors are read
    // while this round's voxels run, and a round's vectors are written back
    // as soon as it ends, so at most two rounds of voxel words are live.
    uint4 cur[kRV];
#pragma unroll
    for (int v = 0; v < kRV; v++) cur[v] = bv[(r0 * kRV + v) * 32];
    {
      // per-x partial sums of the transform rows and of |p_g - C|^2, kept in
      // shared memory (one 16-byte read per voxel) rather than in 16
      // registers per thread
      const float py = __ldg(q.lut[1] + by * 8 + y0);
      const float dy = py - q.C[1];
#pragma unroll
      for (int e = 0; e < kPerVec; e++) {
        const float px = __ldg(q.lut[0] + bx * 8 + x0 + e);
        const float dx = px - q.C[0];
        xpart[e][threadIdx.x] = make_float4(q.T[0] * px + q.T[1] * py, q.T[4] * px + q.T[5] * py,
                                            q.T[8] * px + q.T[9] * py, dx * dx + dy * dy);
      }
    }
    // one copy of the round's code: unrolled, the four rounds (and the
    // colour's four more) run the instruction cache over
#pragma unroll 1
    for (int r = r0; r < r1; r++) {
      uint4 nxt[kRV];
#pragma unroll
      for (int v = 0; v < kRV; v++) nxt[v] = (r + 1 < r1) ? bv[((r + 1) * kRV + v) * 32] : make_uint4(0u, 0u, 0u, 0u);
      word wv[kRV][kPerVec];
#pragma unroll
      for (int v = 0; v < kRV; v++) memcpy(wv[v], &cur[v], 16);
      // this round's z values, one per vector
      float tz0[kRV], tz1[kRV], tz2[kRV], dz2[kRV];
#pragma unroll
      for (int v = 0; v < kRV; v++) {
        const float pz = __ldg(q.lut[2] + bz * 8 + z0 + (r * kRV + v) * kZStep);
        tz0[v] = q.T[2] * pz;
        tz1[v] = q.T[6] * pz;
        tz2[v] = q.T[10] * pz;
        const float dz = pz - q.C[2];
        dz2[v] = dz * dz;
      }
      // nearest pixel of every voxel, then everything the four voxels read,
      // all in flight together, while the distances are computed
      float2 g[kRound];
      float nrm[kRound], iw[kRound], rx[kRound], ry[kRound];
      int px[kRound], py[kRound];
#pragma unroll
      for (int j = 0; j < kRound; j++) {
        const int v = j / kPerVec, e = j % kPerVec;
        // T_gc p_g, each row summed as M0 x + M1 y + M2 z + M3
        const float4 xp = xpart[e][threadIdx.x];
        const float cx = (xp.x + tz0[v]) + q.T[3];
        const float cy = (xp.y + tz1[v]) + q.T[7];
        const float cz = (xp.z + tz2[v]) + q.T[11];
        nrm[j] = xp.w + dz2[v];
        nearest_pixel(cx, cy, cz, q.K, q.fast != 0, px[j], py[j]);
      }
#pragma unroll
      for (int j = 0; j < kRound; j++) {
        float told;
        uint32_t wold;
        S::decode(wv[j / kPerVec][j % kPerVec], told, wold);
        g[j] = make_float2(0.0f, 0.0f);
        iw[j] = rx[j] = ry[j] = 0.0f;
        if ((float)wold < q.max_w && (unsigned)px[j] <= (unsigned)(q.W - 1) && (unsigned)py[j] <= (unsigned)(q.H - 1)) {
          const int pix = py[j] * q.W + px[j];
          if (q.packed) {
            g[j] = __ldg(reinterpret_cast<const float2*>(q.src) + pix);
          } else {
            g[j].x = __ldg(reinterpret_cast<const float*>(q.src) + pix);
            if (q.lam) {
              g[j].y = __ldg(q.lam + pix);
            } else {
              rx[j] = __ldg(q.ray + px[j]);
              ry[j] = __ldg(q.ray + q.W + py[j]);
            }
          }
          iw[j] = __ldg(g_inv_weight + (int)((float)wold + 1.0f));
        }
      }
#pragma unroll
      for (int j = 0; j < kRound; j++) nrm[j] = sqrtf(nrm[j]);
      if (!q.packed && !q.lam) {
#pragma unroll
        for (int j = 0; j < kRound; j++) g[j].y = 1.0f / sqrtf(rx[j] * rx[j] + ry[j] * ry[j] + 1.0f);
      }
      bool changed[kRV];
#pragma unroll
      for (int v = 0; v < kRV; v++) changed[v] = false;
      unsigned upd = 0u;  // voxels of this round whose depth was updated
#pragma unroll
      for (int j = 0; j < kRound; j++) {
        const int v = j / kPerVec, e = j % kPerVec;
        const float sdf = g[j].x - g[j].y * nrm[j];
        if (!(g[j].x > 0.0f) || sdf < -q.mu) continue;
        float told;
        uint32_t wold;
        S::decode(wv[v][e], told, wold);
        const float oldW = (float)wold;
        const float q0 = sdf * q.inv_mu;
        const float ts = fminf(1.0f, fmaf(fmaf(-q0, q.mu, sdf), q.inv_mu, q0));
        const float tnew = (oldW * told + ts) * iw[j];
        wv[v][e] = S::encode(tnew, (uint32_t)(oldW + 1.0f));
        changed[v] = true;
        upd |= 1u << j;
        nupd++;
      }
      if (COLOR && q.col && upd && !dry) color_round<S, kPerVec, kRound>(q, upd, r * kRound, lane, bx, by, bz, b, wv);
#pragma unroll
      for (int v = 0; v < kRV; v++)
#pragma unroll
        for (int e = 0; e < kPerVec; e++) band |= S::band(wv[v][e]);
#pragma unroll
      for (int v = 0; v < kRV; v++) {
        if (changed[v] && !dry) {
          memcpy(&cur[v], wv[v], 16);
          bv[(r * kRV + v) * 32] = cur[v];
        }
        cur[v] = nxt[v];
      }
    }
    nupd = (int)__reduce_add_sync(0xffffffffu, (unsigned)nupd);
    band = __any_sync(0xffffffffu, band);
    if (lane == 0 && !dry) {
      // activation cleared the brick's band flag; its parts set it
      if (band && q.band) q.band[b] = 1;
      if (nupd) {
        atomicAdd(q.counters + 1, (uint32_t)nupd);
        // weights never decrease, so a brick that got an update stays occupied
        if (q.occ) set_bit_once(q.occ, b);
      }
    }
  }
}

template <class S>
__global__ void k_volume_fill(typename S::word* vol, size_t n) {
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const typename S::word v = S::initial();
  for (; i < n; i += (size_t)gridDim.x * blockDim.x) vol[i] = v;
}

// bricked <-> x-fastest linear layout, for a slab of z in [z0, z0 + nz)
template <class S>
__global__ void k_volume_export(const typename S::word* vol, int X, int Y, int z0, int nz, const int* nb3,
                                int nb0, int nb1, float* tsdf, uint16_t* w) {
  size_t n = (size_t)X * Y * nz;
  int nb[3] = {nb0, nb1, 0};
  (void)nb3;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    int x = (int)(i % X), y = (int)((i / X) % Y), z = z0 + (int)(i / ((size_t)X * Y));
    float t;
    uint32_t ww;
    S::decode(vol[brick_word_index(x, y, z, nb)], t, ww);
    if (tsdf) tsdf[i] = t;
    if (w) w[i] = (uint16_t)(ww > 65535u ? 65535u : ww);
  }
}
template <class S>
__global__ void k_volume_import(typename S::word* vol, int X, int Y, int z0, int nz, int nb0, int nb1,
                                const float* tsdf, const uint16_t* w) {
  size_t n = (size_t)X * Y * nz;
  int nb[3] = {nb0, nb1, 0};
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    int x = (int)(i % X), y = (int)((i / X) % Y), z = z0 + (int)(i / ((size_t)X * Y));
    size_t idx = brick_word_index(x, y, z, nb);
    float t;
    uint32_t ww;
    S::decode(vol[idx], t, ww);
    if (tsdf) t = tsdf[i];
    if (w) ww = w[i];
    vol[idx] = S::encode(t, ww);
  }
}

// recomputes the occupancy bits and band flags from the volume (after an import);
// one warp per brick
template <class S>
__global__ void k_occupancy(const SessionDev* __restrict__ s) {
  const typename S::word* vol = reinterpret_cast<const typename S::word*>(s->vol);
  const int nb0 = s->nb[0], nb1 = s->nb[1];
  const size_t nbr = (size_t)nb0 * nb1 * s->nb[2];
  const int lane = threadIdx.x & 31;
  const size_t gw = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const size_t nwarp = ((size_t)gridDim.x * blockDim.x) >> 5;
  for (size_t b = gw; b < nbr; b += nwarp) {
    bool any = false, band = false;
    for (int k = lane; k < kBrickVox; k += 32) {
      const typename S::word v = vol[b * kBrickVox + k];
      float t;
      uint32_t w;
      S::decode(v, t, w);
      any |= w != 0u;
      band |= S::band(v);
    }
    const unsigned m = __ballot_sync(0xffffffffu, any);
    band = __any_sync(0xffffffffu, band);
    if (lane == 0) {
      if (m) set_bit_once(s->occ, (uint32_t)b);
      if (s->band) s->band[b] = band ? 1 : 0;
    }
  }
}

__global__ void k_pack_color(const uint8_t* __restrict__ rgb, uint32_t* __restrict__ out, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = pack_rgb(rgb[i], rgb[n + i], rgb[2 * n + i]);
}

// bricked colour words <-> three planes of x-fastest bytes (cube_color)
__global__ void k_color_volume(uint32_t* col, int X, int Y, int Z, int nb0, int nb1, uint8_t* planes, int do_export) {
  const size_t n = (size_t)X * Y * Z;
  int nb[3] = {nb0, nb1, 0};
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const int x = (int)(i % X), y = (int)((i / X) % Y), z = (int)(i / ((size_t)X * Y));
    const size_t w = brick_word_index(x, y, z, nb);
    if (do_export) {
      const uint32_t c = col[w];
      planes[i] = (uint8_t)rgb_channel(c, 0);
      planes[n + i] = (uint8_t)rgb_channel(c, 1);
      planes[2 * n + i] = (uint8_t)rgb_channel(c, 2);
    } else {
      col[w] = pack_rgb(planes[i], planes[n + i], planes[2 * n + i]);
    }
  }
}

__global__ void k_color_map_export(const uint32_t* __restrict__ m, int n, uint8_t* __restrict__ planes) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) {
    const uint32_t c = m[i];
    planes[i] = (uint8_t)rgb_channel(c, 0);
    planes[n + i] = (uint8_t)rgb_channel(c, 1);
    planes[2 * n + i] = (uint8_t)rgb_channel(c, 2);
  }
}

}  // namespace

void launch_pack_color(const SessionDev& h, const uint8_t* rgb, cudaStream_t st) {
  const int n = h.lv[0].W * h.lv[0].H;
  k_pack_color<<<(n + 255) / 256, 256, 0, st>>>(rgb ? rgb : h.rgb_in, h.rgb_packed, n);
}

void launch_color_volume(const SessionDev& h, bool do_export, uint8_t* planes, cudaStream_t st) {
  k_color_volume<<<sm_count() * 8, 256, 0, st>>>(h.col, h.dim[0], h.dim[1], h.dim[2], h.nb[0], h.nb[1], planes,
                                                 do_export ? 1 : 0);
}

void launch_color_map_export(const SessionDev& h, int level, uint8_t* planes, cudaStream_t st) {
  const int n = h.lv[level].W * h.lv[level].H;
  k_color_map_export<<<(n + 255) / 256, 256, 0, st>>>(h.m_rgb[level], n, planes);
}

int sm_count() {
  static int n = 0;
  if (!n) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (n <= 0) n = 152;
  }
  return n;
}

template <class S, bool COLOR>
int resident_blocks() {
  // one query per kernel variant (the answer depends only on the compiled kernel)
  static int per_sm = -1;
  if (per_sm < 0) {
    int v = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, k_integrate<S, COLOR>, kIntThreads, 0) != cudaSuccess ||
        v < 1)
      v = 1;
    per_sm = v;
  }
  return sm_count() * per_sm;
}

template <class S>
void launch_update(const BatchTable* bt, const float* depth, const float* Tgc, const float* Tcg, bool color,
                   cudaStream_t st, int blocks_per_sm, bool dry) {
  const int most = color ? resident_blocks<S, true>() : resident_blocks<S, false>();
  const int grid = (blocks_per_sm > 0 && blocks_per_sm * sm_count() < most) ? blocks_per_sm * sm_count() : most;
  if (color)
    k_integrate<S, true><<<grid, kIntThreads, 0, st>>>(bt, depth, Tgc, Tcg, 1, dry ? 1 : 0);
  else
    k_integrate<S, false><<<grid, kIntThreads, 0, st>>>(bt, depth, Tgc, Tcg, 0, dry ? 1 : 0);
}

void launch_session_tables(const SessionDev& h, SessionDev* d, cudaStream_t st) {
  int m = 65536;
  for (int v : {h.dim[0], h.dim[1], h.dim[2], h.lv[0].W * h.lv[0].H}) m = v > m ? v : m;
  k_session_tables<<<(m + 255) / 256, 256, 0, st>>>(d);
}

void launch_call_setup(const SessionDev& h, const BatchTable& t, SessionDev* d, BatchTable* dt, cudaStream_t st) {
  const int nbr = h.nb[0] * h.nb[1] * h.nb[2];
  k_call_setup<<<256, 256, 0, st>>>(h, t, d, dt, (uint32_t)nbr);  // 65,536 threads: the weight table's entries
}

void launch_integrate(const BatchTable* bt, int tsdf_type, const float* depth, const float* Tgc, const float* Tcg,
                      bool gate, cudaStream_t st, bool color, int blocks_per_sm, bool dry) {
  const int c = color ? 1 : 0;
  k_activate<<<sm_count() * kActBlocks, dim3(32, 8), 0, st>>>(bt, depth, Tcg, gate ? 1 : 0, dry ? 1 : 0);
  // persistent grid: every block resident at once
  switch (tsdf_type) {
    case VS_TSDF_FP16:
      launch_update<StoreF16>(bt, depth, Tgc, Tcg, c != 0, st, blocks_per_sm, dry);
      break;
    case VS_TSDF_FP32:
      launch_update<StoreF32>(bt, depth, Tgc, Tcg, c != 0, st, blocks_per_sm, dry);
      break;
    default:
      launch_update<StoreI16>(bt, depth, Tgc, Tcg, c != 0, st, blocks_per_sm, dry);
      break;
  }
}

void launch_volume_init(const SessionDev& h, cudaStream_t st) {
  size_t n = (size_t)h.nb[0] * h.nb[1] * h.nb[2] * kBrickVox;
  int blocks = sm_count() * 8;
  switch (h.tsdf_type) {
    case VS_TSDF_FP16:
      k_volume_fill<StoreF16><<<blocks, 256, 0, st>>>((uint32_t*)h.vol, n);
      break;
    case VS_TSDF_FP32:
      k_volume_fill<StoreF32><<<blocks, 256, 0, st>>>((uint2*)h.vol, n);
      break;
    default:
      k_volume_fill<StoreI16><<<blocks, 256, 0, st>>>((uint32_t*)h.vol, n);
      break;
  }
}

// exports / imports one z-slab [z0, z0+nz) through device staging buffers
void launch_volume_slab(const SessionDev& h, bool do_export, int z0, int nz, float* tsdf, uint16_t* w,
                        cudaStream_t st) {
  int blocks = sm_count() * 8;
  const int X = h.dim[0], Y = h.dim[1];
  switch (h.tsdf_type) {
    case VS_TSDF_FP16:
      if (do_export)
        k_volume_export<StoreF16><<<blocks, 256, 0, st>>>((const uint32_t*)h.vol, X, Y, z0, nz, nullptr, h.nb[0],
                                                          h.nb[1], tsdf, w);
      else
        k_volume_import<StoreF16><<<blocks, 256, 0, st>>>((uint32_t*)h.vol, X, Y, z0, nz, h.nb[0], h.nb[1], tsdf, w);
      break;
    case VS_TSDF_FP32:
      if (do_export)
        k_volume_export<StoreF32><<<blocks, 256, 0, st>>>((const uint2*)h.vol, X, Y, z0, nz, nullptr, h.nb[0],
                                                          h.nb[1], tsdf, w);
      else
        k_volume_import<StoreF32><<<blocks, 256, 0, st>>>((uint2*)h.vol, X, Y, z0, nz, h.nb[0], h.nb[1], tsdf, w);
      break;
    default:
      if (do_export)
        k_volume_export<StoreI16><<<blocks, 256, 0, st>>>((const uint32_t*)h.vol, X, Y, z0, nz, nullptr, h.nb[0],
                                                          h.nb[1], tsdf, w);
      else
        k_volume_import<StoreI16><<<blocks, 256, 0, st>>>((uint32_t*)h.vol, X, Y, z0, nz, h.nb[0], h.nb[1], tsdf, w);
      break;
  }
}
// g_uvv_Update_Valid_Volume (z_yooji_cuda_volume_integrator.cu:718-799, host
// :1035-1060): every sub-cube flagged by the last integration whose voxels
// are all invalid in `valid` (one byte per voxel, x fastest, 0 = invalid) is
// reset to the empty state (TSDF 1, weight 0, colour 0) and unflagged;
// sub-cubes with a valid voxel, and unflagged ones, are left as they are.
// One warp per brick: a lane tests rows 2 lane and 2 lane + 1 (8 bytes
// each, aligned: dim[0] is a multiple of 8 and `valid` 8-byte aligned).  The
// brick's occupancy bit is cleared (it holds no weight any more); the coarse
// cells around it stay set, which only costs the ray-caster a skip.
template <class S>
__global__ void k_carve(const SessionDev* __restrict__ s, const uint8_t* __restrict__ valid, unsigned* carved) {
  typename S::word* vol = reinterpret_cast<typename S::word*>(s->vol);
  const int nb0 = s->nb[0], nb1 = s->nb[1];
  const size_t nbr = (size_t)nb0 * nb1 * s->nb[2];
  const size_t X = (size_t)s->dim[0], XY = X * (size_t)s->dim[1];
  const uint32_t stamp = s->brick_count[2];
  const int lane = threadIdx.x & 31;
  const size_t gw = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const size_t nwarp = ((size_t)gridDim.x * blockDim.x) >> 5;
  for (size_t b = gw; b < nbr; b += nwarp) {
    const uint32_t f = s->brick_flag[b];
    if (f == 0u || f != stamp) continue;  // the same for the whole warp
    const int bx = (int)(b % nb0), by = (int)((b / nb0) % nb1), bz = (int)(b / ((size_t)nb0 * nb1));
    bool any = false;
#pragma unroll
    for (int k = 0; k < 2; k++) {
      const int r = 2 * lane + k;
      const size_t o = (size_t)(bz * 8 + (r >> 3)) * XY + (size_t)(by * 8 + (r & 7)) * X + (size_t)bx * 8;
      const uint2 v = __ldg(reinterpret_cast<const uint2*>(valid + o));
      any |= (v.x | v.y) != 0u;
    }
    if (__any_sync(0xffffffffu, any)) continue;
    const typename S::word e = S::initial();
    for (int k = lane; k < kBrickVox; k += 32) vol[b * kBrickVox + k] = e;
    if (s->col)
      for (int k = lane; k < kBrickVox; k += 32) s->col[b * kBrickVox + k] = 0u;
    if (lane == 0) {
      s->brick_flag[b] = 0u;
      if (s->band) s->band[b] = 0;
      atomicAnd(s->occ + (b >> 5), ~(1u << (b & 31)));
      atomicAdd(carved, 1u);
    }
  }
}

size_t occupancy_words(const SessionDev& h) { return (((size_t)h.nb[0] * h.nb[1] * h.nb[2]) + 31) / 32; }

void launch_occupancy_clear(const SessionDev& h, cudaStream_t st) {
  cudaMemsetAsync(h.occ, 0, occupancy_words(h) * 4, st);
  if (h.band) cudaMemsetAsync(h.band, 0, (size_t)h.nb[0] * h.nb[1] * h.nb[2], st);
}

void launch_occupancy_rebuild(const SessionDev& h, const SessionDev* d, cudaStream_t st) {
  launch_occupancy_clear(h, st);
  const int blocks = sm_count() * 8;
  switch (h.tsdf_type) {
    case VS_TSDF_FP16:
      k_occupancy<StoreF16><<<blocks, 256, 0, st>>>(d);
      break;
    case VS_TSDF_FP32:
      k_occupancy<StoreF32><<<blocks, 256, 0, st>>>(d);
      break;
    default:
      k_occupancy<StoreI16><<<blocks, 256, 0, st>>>(d);
      break;
  }
}

void launch_carve(const SessionDev& h, const SessionDev* d, const uint8_t* valid, unsigned* carved, cudaStream_t st) {
  const int blocks = sm_count() * 8;
  switch (h.tsdf_type) {
    case VS_TSDF_FP16:
      k_carve<StoreF16><<<blocks, 256, 0, st>>>(d, valid, carved);
      break;
    case VS_TSDF_FP32:
      k_carve<StoreF32><<<blocks, 256, 0, st>>>(d, valid, carved);
      break;
    default:
      k_carve<StoreI16><<<blocks, 256, 0, st>>>(d, valid, carved);
      break;
  }
}

int integrate_max_dim() { return kMaxDimLut; }
int integrate_max_image() { return kMaxImgLut; }

}  // namespace vs
