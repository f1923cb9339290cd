// 2D Born slab kernels, fields of complex64 (see born2d.cuh).
//
// Only the 8·8·8 core on one, two and eight CTAs. Error against FP64, this kernel ÷ the
// multi-kernel form, mean over seeded δn volumes (transmitted, reflected): 512 points 0.98, 1.02 and
// 1024 points 1.00, 0.90 (16 seeds, within their spread), 4096 points 1.00, 1.01 (96 seeds, ± 0.02).
// On four CTAs (2048 points) it was 1.06, 1.00 and with run-time lengths (3000 points) 1.04, 1.08
// (96 seeds, ± 0.02-0.03): those lengths, and the ones not measured, keep the multi-kernel form. (At 2048
// points both forms have the radices 8·8·8·4; a split line runs the inverse transform's C-point stage
// first, the multi-kernel form last.)
#include "born2d.cuh"

namespace bwpm {

namespace {
template <int C>
BornKernel born_core() {
  BornKernel k;
  born_fill<float, ch::FixedLine<float, 512, 64, rf::Radices<8, 8, 8>>, C>(k, 512 * C, 64, {8, 8, 8});
  return k;
}
}  // namespace

template <>
BornKernel born_kernel<float>(int n) {
  switch (n) {
    case 512: return born_core<1>();
    case 1024: return born_core<2>();
    case 4096: return born_core<8>();
    default: return BornKernel{};
  }
}

}  // namespace bwpm
