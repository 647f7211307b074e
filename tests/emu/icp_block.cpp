// One block of the tracking kernels (EMU_BLOCK: a name of its own; EMU_ICP:
// the kernels' source, prepared by the test)
#include "cuda_emu.h"
#include EMU_ICP

#define EMU_CAT2(a, b) a##b
#define EMU_CAT(a, b) EMU_CAT2(a, b)

void EMU_CAT(emu_begin_, EMU_BLOCK)(const vs::BatchTable* t, unsigned* words, int frame_mode) {
  emu_run(0, 32, [=] { vs::k_icp_begin(t, words, frame_mode, 0, nullptr); });
}
void EMU_CAT(emu_track_, EMU_BLOCK)(const vs::BatchTable* t, unsigned* words, int block, int mode) {
  emu_run(block, kEmuThreads, [=] {
    if (mode == VS_REDUCE_FP64)
      vs::k_icp_run<VS_REDUCE_FP64>(t, words);
    else
      vs::k_icp_run<VS_REDUCE_KAHAN>(t, words);
  });
}
