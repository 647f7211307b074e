// Runs blocks of the tracking kernels on the host: icp_main SCENARIO MODE
// LISTED prints the outcome of two frames as one JSON line (alone: one block;
// idle: a second block that runs out of looks while the first holds a range;
// stuck: a frame whose iteration nobody ends, then a clean one).
#include <stdio.h>
#include <stdlib.h>

#include <condition_variable>
#include <mutex>

#include "cuda_emu.h"
#include "vs_internal.cuh"

using namespace vs;
void emu_begin_a(const BatchTable*, unsigned*, int);
void emu_track_a(const BatchTable*, unsigned*, int, int);
void emu_track_b(const BatchTable*, unsigned*, int, int);
std::function<void(const void*)> emu_before_atomic;

namespace {

constexpr int kW = 40, kH = 32, kRanges = 3;

// a curved surface seen by the camera, and the same seen 2 mm beside
struct Scene {
  SessionDev s;
  BatchTable t;
  Pose pose;
  std::vector<float> depth;
  std::vector<float4> mvtx, mnrm, innrm;
  std::vector<uint32_t> list;
  std::vector<double> partials;
  uint32_t count[4];
  unsigned counter;

  explicit Scene(bool listed) {
    memset(&s, 0, sizeof(s));
    memset(&t, 0, sizeof(t));
    memset(&pose, 0, sizeof(pose));
    s.levels = 1;
    s.lv[0].W = kW, s.lv[0].H = kH;
    const float K[4] = {40.0f, 40.0f, 0.5f * kW - 0.5f, 0.5f * kH - 0.5f};
    memcpy(s.lv[0].K, K, sizeof(K));
    s.iters[0] = 2;
    s.th_icp = 0.01f;
    s.cos_normal = listed ? 0.5f : -3.0f;
    auto surface = [](float x, float y) { return 1.0f + 0.05f * sinf(5.0f * x + 1.0f) + 0.04f * cosf(6.0f * y); };
    for (int y = 0; y < kH; y++)
      for (int x = 0; x < kW; x++) {
        const float rx = ((float)x - K[2]) / K[0], ry = ((float)y - K[3]) / K[1];
        for (int shifted = 0; shifted < 2; shifted++) {
          const float dx = shifted ? 0.002f : 0.0f;
          float z = 1.0f;
          for (int k = 0; k < 30; k++) z = surface(rx * z + dx, ry * z);
          if (shifted) {
            depth.push_back(z);
            continue;
          }
          const float gx = 0.25f * cosf(5.0f * rx * z + 1.0f), gy = -0.24f * sinf(6.0f * ry * z);
          const float len = sqrtf(gx * gx + gy * gy + 1.0f);
          mvtx.push_back(make_float4(rx * z, ry * z, z, 1.0f));
          mnrm.push_back(make_float4(gx / len, gy / len, -1.0f / len, 1.0f));
        }
        list.push_back((uint32_t)(y << 16 | x));
      }
    innrm = mnrm;
    partials.resize((size_t)kIcpMaxBlocks * kPartials * 2);
    s.depth[0] = depth.data();
    s.in_nrm[0] = innrm.data();
    s.m_vtx[0] = mvtx.data();
    s.m_nrm[0] = mnrm.data();
    s.in_list[0] = list.data();
    count[0] = listed ? (uint32_t)list.size() : 0u;
    s.in_count = count;
    s.partials = partials.data();
    s.icp_counter = &counter;
    s.pose = &pose;
    t.n = 1;
    t.s[0] = &s;
    t.icp[0][1] = kRanges;  // dense: 1280 pixels in 3 ranges; listed: 5 of 256
    for (int k = 0; k < 16; k += 5) pose.T_gc[k] = 1.0;
    pose.frame = 1;
    pose.tracked = 1;
  }
  unsigned* words() { return t.icp_word; }
  void print(const char* key) const {
    printf("\"%s\": {\"tracked\": %d, \"failed\": %d, \"frame\": %d, \"iters\": %d, \"count\": %d, \"T_gc\": [", key,
           pose.tracked, pose.failed, pose.frame, pose.iters_run, pose.valid_count);
    for (int k = 0; k < 16; k++) printf("%s%.17g", k ? ", " : "", pose.T_gc[k]);
    printf("]}");
  }
};

}  // namespace

int main(int argc, char** argv) {
  if (argc != 4) return 2;
  const std::string what = argv[1];
  const int mode = atoi(argv[2]);
  const bool listed = atoi(argv[3]) != 0;
  Scene c(listed);
  const int ranges = listed ? (kW * kH + 255) / 256 : kRanges;
  printf("{");
  emu_begin_a(&c.t, c.words(), 1);
  if (what == "alone") {
    emu_track_a(&c.t, c.words(), 0, mode);
  } else if (what == "idle") {
    // the first block is held before the arrival of its first iteration's
    // last range; the second finds no range, and must leave
    std::mutex m;
    std::condition_variable cv;
    int arrivals = 0;
    bool held = false, left = false;
    emu_before_atomic = [&](const void* p) {
      if (p != &c.counter) return;
      std::unique_lock<std::mutex> l(m);
      if (++arrivals != ranges) return;
      held = true;
      cv.notify_all();
      cv.wait(l, [&] { return left; });
    };
    std::thread first([&] { emu_track_a(&c.t, c.words(), 0, mode); });
    {
      std::unique_lock<std::mutex> l(m);
      cv.wait(l, [&] { return held; });
    }
    emu_track_b(&c.t, c.words(), 1, mode);
    {
      std::unique_lock<std::mutex> l(m);
      left = true;
      cv.notify_all();
    }
    first.join();
    emu_before_atomic = nullptr;
  } else {
    c.t.icp_word[0] += (unsigned)ranges;  // every range taken, by blocks that never arrive
    emu_track_b(&c.t, c.words(), 1, mode);
  }
  c.print("frame");
  printf(", ");
  emu_begin_a(&c.t, c.words(), 1);
  emu_track_a(&c.t, c.words(), 0, mode);
  c.print("next");
  printf("}\n");
  return 0;
}
