// dg_k_resident.cu — instances of the resident step (k_step_resident): FP32 one shot and two shots
// per lane, plain and Kahan, FP64 and the reference operators.  FP64 and plain FP32 on two shots
// have a second instance for blocks of up to 256 threads, which keeps all its values in registers
// (255 and 224 a thread, no spills; 168 and up to 76 bytes of spills at 384 threads).
#include "dg_kernels.cuh"

namespace dg {

ResKernel<ArithP2<float>> kernel_resident_f1(bool kahan) {
  if (kahan) return {k_step_resident<ArithP2<float>, true, 384>, 384};
  return {k_step_resident<ArithP2<float>, false, 512>, 512};
}
ResKernel<ArithP2<float2>> kernel_resident_f2(bool kahan, bool small) {
  if (kahan) return {k_step_resident<ArithP2<float2>, true, 256>, 256};
  if (small) return {k_step_resident<ArithP2<float2>, false, 256>, 256};
  return {k_step_resident<ArithP2<float2>, false, 384>, 384};
}
ResKernel<ArithOps<double>> kernel_resident_d(bool small) {
  if (small) return {k_step_resident<ArithOps<double>, false, 256>, 256};
  return {k_step_resident<ArithOps<double>, false, 384>, 384};
}
ResKernel<ArithRef> kernel_resident_ref() { return {k_step_resident<ArithRef, false, 256>, 256}; }

}  // namespace dg
