// Run-time-length register-resident kernels of the resident 2D engine (see rgen.cuh).
#include "rgen.cuh"
#include "variants.hpp"

namespace bwpm {

const std::vector<RtVariant>& rt_variants() {
  using rg::rt_max_threads;
  static const std::vector<RtVariant> v = {
      // equal outer radices: one exchange per stage boundary (2430 points 27 → 12 µs per step)
      {4, (const void*)k_resident2d_rt<4, 512, true>, 512, true},
      {5, (const void*)k_resident2d_rt<5, 512, true>, 512, true},
      {6, (const void*)k_resident2d_rt<6, 512, true>, 512, true},
      {8, (const void*)k_resident2d_rt<8, 512, true>, 512, true},
      {9, (const void*)k_resident2d_rt<9, 512, true>, 512, true},
      {10, (const void*)k_resident2d_rt<10, 512, true>, 512, true},
      {12, (const void*)k_resident2d_rt<12, 512, true>, 512, true},
      {15, (const void*)k_resident2d_rt<15, 512, true>, 512, true},
      // any E that divides the length
      {8, (const void*)k_resident2d_rt<8>, rt_max_threads(8), false},
      {9, (const void*)k_resident2d_rt<9>, rt_max_threads(9), false},
      {10, (const void*)k_resident2d_rt<10>, rt_max_threads(10), false},
      {12, (const void*)k_resident2d_rt<12>, rt_max_threads(12), false},
      {15, (const void*)k_resident2d_rt<15>, rt_max_threads(15), false},
      {16, (const void*)k_resident2d_rt<16>, rt_max_threads(16), false},
      {20, (const void*)k_resident2d_rt<20>, rt_max_threads(20), false},
      {24, (const void*)k_resident2d_rt<24>, rt_max_threads(24), false},
      {30, (const void*)k_resident2d_rt<30>, rt_max_threads(30), false},
      // wide forms (512 threads, 128 registers) for lines beyond the default thread limit
      {9, (const void*)k_resident2d_rt<9, 512>, 512, false},
      {10, (const void*)k_resident2d_rt<10, 512>, 512, false},
      {12, (const void*)k_resident2d_rt<12, 512>, 512, false}};
  return v;
}

}  // namespace bwpm
