// Registry of the 2D chain kernels (chain2d.cuh): per field type and line length one kernel that
// runs all sweeps of a 2D solve in one launch.
#pragma once

#include <cstddef>
#include <vector>

#include "common.cuh"

namespace bwpm {

struct ChainKernel {
  const void* fn = nullptr;   // null: no chain kernel for the length (or its shared memory)
  int ctas = 1;               // CTAs per line (a cluster when more than one)
  int threads = 0;
  std::size_t smem = 0;       // dynamic shared memory per CTA
  std::vector<int> radices;   // of the n / ctas points of a part
  int tw_smem = 0;            // the stage twiddles sit in shared memory
  int mask_smem = 0;          // the mask does
  int spec_smem = 0;          // the spectrum line of a multi-pass step does
};

// The chain kernel of lines of n points with fields of type T (double or float).
template <typename T>
ChainKernel chain_kernel(int n, bool masked);

}  // namespace bwpm
