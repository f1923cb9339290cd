// 2D Born slab kernels, fields of complex64 (see born2d.cuh).
#include "born2d.cuh"

namespace bwpm {

template <>
BornKernel born_kernel<float>(int n) {
  return born_pick<float>(n);
}

}  // namespace bwpm
