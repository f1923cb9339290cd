// Kernel variants of the resident 2D engine for lengths 256-1536 (see variants.hpp).
#include "resident2d.cuh"
#include "variants.hpp"

namespace bwpm {

namespace {
using rf::Radices;

template <int N, int NT, int... R>
FixedVariant fixed() {
  return {N, NT, 1, {R...}, (const void*)k_resident2d_fixed<N, NT, Radices<R...>>, fixed_smem_bytes<N>()};
}

}  // namespace

void add_variants_small(std::vector<FixedVariant>& v) {
  // per length, only variants that no other variant beats in both per-step latency and SM time
  // (measured on a B200: 1 item, tilted slab, 400 slabs; µs per step, the variant replaced in
  // brackets). Four values a thread on twice the warps win up to 512 points, inner stages of any
  // radix (rf::gfft) at the lengths with a factor 3.
  v.push_back(fixed<256, 64, 4, 4, 4, 4>());    // 0.74 (8·8·4 on 32 threads: 0.92)
  v.push_back(fixed<384, 96, 4, 6, 4, 4>());    // 0.89 (4·4·4·3·2 on 32 threads: 2.0)
  v.push_back(fixed<512, 128, 4, 8, 4, 4>());   // 1.02 (8·8·8 on 64 threads: 1.11)
  v.push_back(fixed<768, 96, 8, 12, 8>());      // 1.47 (4·4·4·4·3 on 64 threads: 2.4)
  v.push_back(fixed<1024, 128, 8, 8, 8, 2>());  // 1.74 (4·8·8·4 on 256 threads: 2.1)
  // 3.0 (8·8·8·3 3.6; 8·4·6·8 3 % slower and 5 % less exact on the reflected field)
  v.push_back(fixed<1536, 192, 8, 8, 3, 8>());
  v.push_back(fixed<1536, 128, 4, 4, 4, 4, 2, 3>());  // 3.9 on fewer threads
}

const std::vector<FixedVariant>& fixed_variants() {
  static const std::vector<FixedVariant> all = [] {
    std::vector<FixedVariant> v;
    add_variants_small(v);
    add_variants_large(v);
    return v;
  }();
  return all;
}

}  // namespace bwpm
