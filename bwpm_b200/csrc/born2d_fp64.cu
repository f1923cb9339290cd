// 2D Born slab kernels, fields of FP64 (see born2d.cuh).
#include "born2d.cuh"

namespace bwpm {

template <>
BornKernel born_kernel<double>(int n) {
  return born_pick<double>(n);
}

}  // namespace bwpm
