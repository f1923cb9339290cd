// 2D chain kernels, fields of complex64 (see chain2d.cuh).
#include "chain2d.cuh"

namespace bwpm {

namespace {
// Parts of a run-time length, in the order they are tried: five and four before eight and six. Of the
// noise of the cross stage of C parts what falls on propagating waves stays: its comb has the teeth
// N/C, and a line sampled at λ/8 carries waves up to 0.19 N, so of 8 and 6 parts two neighbouring teeth
// stay, of 5 and 4 none. Error against the launch-per-step kernels, mean over facet and lens volumes
// (transmitted, reflected; 15-30 plans each): 8 parts 1.02, 1.03, 6 parts 1.03, 0.99, 5 parts 0.98,
// 0.97, 4 parts 0.99, 0.97. Longer parts take more time than that is worth (µs per step: 2000 points on
// 8 6.5, on 5 5.6; 3600 6.8, 6.9; 3024 points on 4 are 9 % behind 6, 5000 on 5 14 % behind 8).
std::vector<int> chain_parts(int n) {
  std::vector<int> parts;
  for (int c : {5, 4})
    if (n % c == 0 && n / c <= 720) parts.push_back(c);
  for (int c : {8, 6, 5, 4})
    if (std::find(parts.begin(), parts.end(), c) == parts.end()) parts.push_back(c);
  return parts;
}
}  // namespace

template <>
ChainKernel chain_kernel<float>(int n, bool masked) {
  using T = float;
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
      return chain_runtime_kernel<T>(all, n, masked, chain_parts(n));
    }
  }
  if (k.fn) chain_smem<T>(n, masked, k);
  return k;
}

}  // namespace bwpm
