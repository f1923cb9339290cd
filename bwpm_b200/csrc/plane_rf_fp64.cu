// Register-resident 3D slab-step kernels, fields of FP64 (see plane_rf.cuh).
#include "plane_rf.cuh"

namespace bwpm {

template <>
RfKernels rf_kernels<double>(int n) {
  using T = double;
  switch (n) {
    case 256: return rf_fixed<T, 256, 32, 2, 8, 4, 8>();
    case 384: return rf_fixed<T, 384, 48, 2, 8, 6, 8>();
    case 512: return rf_fixed<T, 512, 64, 2, 8, 8, 8>();
    case 768: return rf_fixed<T, 768, 96, 2, 8, 12, 8>();
    case 1024: return rf_fixed<T, 1024, 128, 2, 8, 4, 4, 8>();
    default: break;
  }
  static const std::vector<RfRuntime<T>> all = {
      rf_runtime<T, 2>(), rf_runtime<T, 3>(), rf_runtime<T, 4>(), rf_runtime<T, 5>(),
      rf_runtime<T, 6>(), rf_runtime<T, 7>(), rf_runtime<T, 8>(), rf_runtime<T, 9>(),
      rf_runtime<T, 10>()};
  return rf_pick_runtime(all, n);
}

}  // namespace bwpm
