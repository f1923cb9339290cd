// Registry of the register-resident 3D slab-step kernels (plane_rf.cuh).
#pragma once

#include <cstddef>
#include <vector>

namespace bwpm {

struct RfKernels {
  const void* cols = nullptr;  // null: no kernels for the length
  const void* rows = nullptr;
  int lines = 0;               // lines per CTA
  int threads = 0;             // threads per CTA
  std::size_t cols_smem = 0;   // dynamic shared memory per CTA
  std::size_t rows_smem = 0;
  std::vector<int> radices;    // the transform's stages
};

// The kernels of lateral length n with fields of type T (double or float).
template <typename T>
RfKernels rf_kernels(int n);

}  // namespace bwpm
