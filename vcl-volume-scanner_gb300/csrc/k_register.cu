// Depth -> colour camera registration (vs_warp_depth_to_color,
// vs_warp_depth_mm_to_color in include/vs.h).
//
// Reference: z_tdrcc_Transform_Depth_to_Rgb_Camera_Coordinates
// (STAC/Engine/CPU/z_yooji_object_scanner.cpp:2429-2476) with
// CKvYooji_MatrixRgbD::convert_pixel_coord (STAC/Object/CPU/
// z_yooji_matrix_rgbd.cpp:101-118) and the KAISION-style camera helpers of
// STAC/Object/CPU/z_yooji_camera_parameters.cpp:89-108,678-685: every depth
// pixel with depth d > 0 is back-projected with the depth intrinsics,
// transformed by the depth-to-colour extrinsics, projected with the colour
// intrinsics and rounded with ROUNDF; a colour pixel keeps the smallest depth
// that lands on it (the depth value of the depth camera, as the reference
// stores it), 0 where none lands.  The reference runs this per frame on the
// host ("always start from the depth seen by the RGB camera",
// z_yooji_object_scanner.cpp:806-820).  Here one thread per depth pixel
// lands its depth by compare-and-swap on the value's bits, which order
// positive floats (and uint16) as their values, so the result does not
// depend on the order the threads arrive in.
//
// The minimum runs in the caller's output itself, where 0 is both "empty" and
// the answer for a pixel where nothing lands: two small launches, and the
// host's part of them, bound it (512x424 into 1280x960: 20 us a call).  With a
// scratch image from the stream's pool, a minimum beside "all ones" and a pass
// to the output, 24 to 27 us, and 300 us when the pool had given its memory
// back to the system between two calls.  Only an output that overlaps the
// input needs the scratch.
#include <cuda_runtime.h>
#include <stdint.h>

#include "vs_internal.cuh"

namespace vs {
namespace {

struct WarpArgs {
  int wd, hd, wr, hr;
  float Kd[4], Kr[4], T[12];
  float scale;  // depth units -> metres (1 for metres)
};

// T is float (metres) or uint16 (units); the bits that order a depth
__device__ __forceinline__ unsigned order_bits(float, float td) { return __float_as_uint(td); }
__device__ __forceinline__ unsigned short order_bits(uint16_t raw, float) { return raw; }

// the smallest of the values that land on *p, 0: none yet
template <class W>
__device__ __forceinline__ void land(W* p, W v) {
  W old = *(volatile W*)p;
  while (old == 0 || v < old) {  // after the first value, the stored one falls at each turn
    const W seen = atomicCAS(p, old, v);
    if (seen == old) break;
    old = seen;
  }
}
template <class T>
struct Bits {
  typedef unsigned word;
};
template <>
struct Bits<uint16_t> {
  typedef unsigned short word;
};

template <class T>
__global__ void k_warp_depth(const T* __restrict__ in, WarpArgs a, typename Bits<T>::word* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= a.wd || j >= a.hd) return;
  const T raw = in[(size_t)j * a.wd + i];
  const float td = (float)raw * a.scale;
  if (!(td > 0.0f)) return;
  const F3 p = transform(back_project((float)i, (float)j, a.Kd, td), a.T);
  float u, v;
  project(p, a.Kr, u, v);
  if (isnan(u) || isnan(v)) return;
  const int tx = roundf_ref(u), ty = roundf_ref(v);
  if (tx < 0 || tx > a.wr - 1 || ty < 0 || ty > a.hr - 1) return;
  land(out + (size_t)ty * a.wr + tx, order_bits(raw, td));
}

// zeroes n values: the 16-byte words among them, and the values before and
// after those
template <class W>
__global__ void k_warp_clear(W* p, int n) {
  constexpr int E = 16 / sizeof(W);
  const int head = min(n, (int)((16 - (reinterpret_cast<uintptr_t>(p) & 15)) & 15) / (int)sizeof(W));
  const int body = (n - head) / E, tail = n - head - body * E;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < body) reinterpret_cast<uint4*>(p + head)[i] = make_uint4(0u, 0u, 0u, 0u);
  if (i < head) p[i] = 0;
  if (i < tail) p[n - 1 - i] = 0;
}

}  // namespace

template <class T>
void launch_warp_depth(const T* in, int wd, int hd, const float* Kd, const float* T_rgb_d, const float* Kr, int wr,
                       int hr, float scale, T* out, cudaStream_t st) {
  WarpArgs a;
  a.wd = wd;
  a.hd = hd;
  a.wr = wr;
  a.hr = hr;
  for (int k = 0; k < 4; k++) a.Kd[k] = Kd[k], a.Kr[k] = Kr[k];
  for (int k = 0; k < 12; k++) a.T[k] = T_rgb_d[k];
  a.scale = scale;
  const int n = wr * hr;
  typedef typename Bits<T>::word W;
  W* bits = reinterpret_cast<W*>(out);
  const int blocks = (n / (16 / (int)sizeof(W)) + 16 + 255) / 256;
  k_warp_clear<W><<<blocks, 256, 0, st>>>(bits, n);
  k_warp_depth<T><<<dim3((wd + 31) / 32, (hd + 7) / 8), dim3(32, 8), 0, st>>>(in, a, bits);
}

template void launch_warp_depth<float>(const float*, int, int, const float*, const float*, const float*, int, int,
                                       float, float*, cudaStream_t);
template void launch_warp_depth<uint16_t>(const uint16_t*, int, int, const float*, const float*, const float*, int,
                                          int, float, uint16_t*, cudaStream_t);

}  // namespace vs
