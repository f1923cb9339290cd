// 2D chain kernels, fields of FP64 (see chain2d.cuh).
#include "chain2d.cuh"

namespace bwpm {

template <>
ChainKernel chain_kernel<double>(int n, bool masked) {
  using T = double;
  ChainKernel k;
  switch (n) {
    case 256: k = chain_fixed<T, 1, 256, 64, 4, 4, 4, 4>(); break;
    case 384: k = chain_fixed<T, 1, 384, 96, 4, 6, 4, 4>(); break;
    case 512: k = chain_fixed<T, 1, 512, 128, 4, 8, 4, 4>(); break;
    case 768: k = chain_fixed<T, 1, 768, 96, 8, 12, 8>(); break;
    case 1024: k = chain_fixed<T, 4, 256, 64, 4, 4, 4, 4>(); break;
    case 1536: k = chain_fixed<T, 4, 384, 96, 4, 6, 4, 4>(); break;
    case 2048: k = chain_fixed<T, 8, 256, 64, 4, 4, 4, 4>(); break;
    case 3072: k = chain_fixed<T, 8, 384, 96, 4, 6, 4, 4>(); break;
    case 4096: k = chain_fixed<T, 8, 512, 64, 8, 8, 8>(); break;
    case 6144: k = chain_fixed<T, 8, 768, 96, 8, 12, 8>(); break;
    case 8192: k = chain_fixed<T, 8, 1024, 128, 8, 4, 4, 8>(); break;
    default: {
      static const std::vector<ChainRuntime> all = [] {
        std::vector<ChainRuntime> v;
        chain_runtime<T, 2>(v);
        chain_runtime<T, 3>(v);
        chain_runtime<T, 4>(v);
        chain_runtime<T, 5>(v);
        chain_runtime<T, 6>(v);
        chain_runtime<T, 7>(v);
        chain_runtime<T, 8>(v);
        chain_runtime<T, 9>(v);
        chain_runtime<T, 10>(v);
        chain_runtime<T, 12>(v);
        chain_runtime<T, 15>(v);
        chain_runtime_split<T, 3, 4>(v);
        chain_runtime_split<T, 4, 4>(v);
        chain_runtime_split<T, 5, 4>(v);
        chain_runtime_split<T, 6, 4>(v);
        chain_runtime_split<T, 9, 4>(v);
        chain_runtime_split<T, 3, 5>(v);
        chain_runtime_split<T, 4, 5>(v);
        chain_runtime_split<T, 5, 5>(v);
        chain_runtime_split<T, 6, 5>(v);
        chain_runtime_split<T, 9, 5>(v);
        chain_runtime_split<T, 3, 6>(v);
        chain_runtime_split<T, 5, 6>(v);
        chain_runtime_split<T, 9, 6>(v);
        chain_runtime_split<T, 4, 8>(v);
        chain_runtime_split<T, 5, 8>(v);
        chain_runtime_split<T, 6, 8>(v);
        return v;
      }();
      return chain_runtime_kernel<T>(all, n, masked, {8, 6, 5, 4});
    }
  }
  if (k.fn) chain_smem<T>(n, masked, k);
  return k;
}

}  // namespace bwpm
