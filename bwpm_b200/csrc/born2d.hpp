// Registry of the 2D Born slab kernels (born2d.cuh).
#pragma once

#include <cstddef>
#include <vector>

#include "common.cuh"

namespace bwpm {

struct BornKernel {
  const void* fn = nullptr;   // null: no kernel for the length
  int ctas = 1;               // cluster size: the line is split over this many CTAs
  int threads = 0;
  std::size_t smem = 0;
  int basis_smem = 0;         // Krylov vectors kept in shared memory
  std::vector<int> radices;   // of the per-CTA transform (n / ctas points)
};

template <typename T>
BornKernel born_kernel(int n);

}  // namespace bwpm
