// 2D chain kernels, fields of FP64 (see chain2d.cuh).
#include "chain2d.cuh"

namespace bwpm {

template <>
ChainKernel chain_kernel<double>(int n, bool masked) {
  using T = double;
  ChainKernel k;
  switch (n) {
    case 256: k = chain_fixed<T, 256, 32, 8, 4, 8>(); break;
    case 384: k = chain_fixed<T, 384, 48, 8, 6, 8>(); break;
    case 512: k = chain_fixed<T, 512, 64, 8, 8, 8>(); break;
    case 768: k = chain_fixed<T, 768, 96, 8, 12, 8>(); break;
    case 1024: k = chain_fixed<T, 1024, 128, 8, 4, 4, 8>(); break;
    case 1536: k = chain_fixed<T, 1536, 192, 8, 4, 6, 8>(); break;
    case 2048: k = chain_fixed<T, 2048, 256, 8, 8, 4, 8>(); break;
    case 3072: k = chain_fixed<T, 3072, 384, 8, 8, 6, 8>(); break;
    case 4096: k = chain_fixed<T, 4096, 512, 8, 8, 8, 8>(); break;
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
        return v;
      }();
      k = chain_pick_runtime(all, n);
    }
  }
  if (k.fn) chain_smem<T>(n, masked, k);
  return k;
}

}  // namespace bwpm
