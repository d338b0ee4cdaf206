// dg_k_resident.cu — instances of the resident step (k_step_resident): FP32 one shot and two shots
// per lane, plain and Kahan, FP64 and the reference operators.  FP64 and plain FP32 on two shots
// have a second instance for blocks of up to 256 threads, which keeps all its values in registers
// (255 and 228 a thread, no spills; 168 and up to 76 bytes of spills at 384 threads).
#include "dg_kernels.cuh"

namespace dg {

// both instances of a kernel: the step counted by the host, and by the device (ResKernel)
#define DG_RES(A, KAHAN, MAXT) {{k_step_resident<A, KAHAN, MAXT, false>, k_step_resident<A, KAHAN, MAXT, true>}, MAXT}

ResKernel<ArithP2<float>> kernel_resident_f1(bool kahan) {
  if (kahan) return DG_RES(ArithP2<float>, true, 384);
  return DG_RES(ArithP2<float>, false, 512);
}
ResKernel<ArithP2<float2>> kernel_resident_f2(bool kahan, bool small) {
  if (kahan) return DG_RES(ArithP2<float2>, true, 256);
  if (small) return DG_RES(ArithP2<float2>, false, 256);
  return DG_RES(ArithP2<float2>, false, 384);
}
ResKernel<ArithOps<double>> kernel_resident_d(bool small) {
  if (small) return DG_RES(ArithOps<double>, false, 256);
  return DG_RES(ArithOps<double>, false, 384);
}
ResKernel<ArithRef> kernel_resident_ref() { return DG_RES(ArithRef, false, 256); }

}  // namespace dg
