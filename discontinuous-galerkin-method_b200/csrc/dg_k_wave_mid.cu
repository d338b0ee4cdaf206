// dg_k_wave_mid.cu — instances of the wavefront step on resident blocks for the shot counts
// between the powers of two from 16 on: multiples of 4 up to 40 and of 8 up to 120 (other counts
// are padded up to the next).  FP32 in the form with staged old values, FP32-Kahan in the plain
// one, the faster for each.  Compiled in parts (DG_WAVE_PART 0..3).
#include "dg_kernels.cuh"

#ifndef DG_WAVE_PART
#define DG_WAVE_PART 0
#endif

namespace dg {

#define DG_WM(SS)                                                                                  \
  if (S == SS)                                                                                     \
    return kahan ? (WaveFn)k_step_wave_p<WaveTwoShots<SS>, true> : (WaveFn)k_step_wave_p<WaveTwoShotsAsync<SS>, false>;
WaveFn kernel_wave_mid1(int S, bool kahan);
WaveFn kernel_wave_mid2(int S, bool kahan);
WaveFn kernel_wave_mid3(int S, bool kahan);
#if DG_WAVE_PART == 0
WaveFn kernel_wave_mid(int S, bool kahan) {
  DG_WM(20) DG_WM(24) DG_WM(28) DG_WM(36)
  WaveFn k = kernel_wave_mid1(S, kahan);
  if (!k) k = kernel_wave_mid2(S, kahan);
  if (!k) k = kernel_wave_mid3(S, kahan);
  return k;
}
#elif DG_WAVE_PART == 1
WaveFn kernel_wave_mid1(int S, bool kahan) {
  DG_WM(40) DG_WM(48) DG_WM(56) DG_WM(72)
  return nullptr;
}
#elif DG_WAVE_PART == 2
WaveFn kernel_wave_mid2(int S, bool kahan) {
  DG_WM(80) DG_WM(88) DG_WM(96)
  return nullptr;
}
#elif DG_WAVE_PART == 3
WaveFn kernel_wave_mid3(int S, bool kahan) {
  DG_WM(104) DG_WM(112) DG_WM(120)
  return nullptr;
}
#endif

}  // namespace dg
