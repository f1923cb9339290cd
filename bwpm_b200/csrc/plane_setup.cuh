// Set-up of the plane engine on the device: per slab step, the label pairs present, the pair-id
// plane (which pair each pixel selects) and the sorted list of interface pixels, from a uint8
// label volume in device memory.
//
// This is the per-step analysis of cpp/src/solver.cpp:384-417 and :419-459 (pairs of a step in
// std::set order, the I_r,s selection, reflection sources where ñ(plane p) ≠ ñ(plane p + 1)),
// done once per solve for all steps at once instead of per slab on the host: codes
// (r + 1)·m + s sort like the pairs, a presence bitmask per step gives the pairs in order, and
// the interface pixels are compacted in pixel order by segment (count, scan, ballots).
#pragma once

#include <cstdint>

#include "common.cuh"

namespace bwpm {

constexpr int kSetupThreads = 1024;

struct SetupVolume {
  const std::uint8_t* labels;  // (nz, ny, nx) labels, device
  long long nn;                // ny·nx
  int nz, ny, nx, m;           // m materials; codes (r + 1)·m + s, r = −1: before the volume
  int words;                   // presence words per step: ⌈(m + 1)·m / 32⌉
};

__device__ __forceinline__ int setup_code(const SetupVolume& v, int p, long long q) {
  const int r = p == 0 ? -1 : static_cast<int>(v.labels[(p - 1) * v.nn + q]);
  const int s = v.labels[p * v.nn + q];
  return (r + 1) * v.m + s;
}

// grid (blocks per step, nz): presence bits of the codes and the number of interface pixels
// (code_iface[code] ≠ 0) per step; bits/count zeroed by the caller.
__global__ void __launch_bounds__(256)
    k_setup_presence(SetupVolume v, const std::uint8_t* code_iface, unsigned* bits,
                     unsigned long long* iface_count) {
  extern __shared__ unsigned s_bits[];
  __shared__ unsigned s_count;
  const int p = blockIdx.y;
  for (int w = threadIdx.x; w < v.words; w += blockDim.x) s_bits[w] = 0u;
  if (threadIdx.x == 0) s_count = 0u;
  __syncthreads();
  unsigned local = 0;
  for (long long q = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; q < v.nn;
       q += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int code = setup_code(v, p, q);
    atomicOr(&s_bits[code >> 5], 1u << (code & 31));
    local += code_iface[code];
  }
  for (int o = 16; o > 0; o >>= 1) local += __shfl_down_sync(0xffffffffu, local, o);
  if ((threadIdx.x & 31) == 0 && local) atomicAdd(&s_count, local);
  __syncthreads();
  for (int w = threadIdx.x; w < v.words; w += blockDim.x)
    if (s_bits[w]) atomicOr(&bits[static_cast<long long>(p) * v.words + w], s_bits[w]);
  if (threadIdx.x == 0 && s_count) atomicAdd(&iface_count[p], static_cast<unsigned long long>(s_count));
}

// grid (blocks per step, steps listed in `steps`): pid[q] = code_id[table row][code] for the
// steps with more than one pair.
__global__ void k_setup_pid(SetupVolume v, const int* steps, const long long* pid_off,
                            const std::uint8_t* code_id, int ncode, std::uint8_t* pid_pool) {
  const int k = blockIdx.y;
  const int p = steps[k];
  std::uint8_t* out = pid_pool + pid_off[k];
  const std::uint8_t* table = code_id + static_cast<long long>(k) * ncode;
  for (long long q = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; q < v.nn;
       q += static_cast<long long>(gridDim.x) * blockDim.x)
    out[q] = table[setup_code(v, p, q)];
}

// The interface pixels of the listed steps in increasing pixel order, in three kernels over segments
// of `seg` pixels (3D: rows): count, scan, write. (One CTA per step, scanning row by row, took
// 0.6 ms for 12 slabs of 512² and 1.1 ms for 1024²: a dozen SMs, three barriers per row.)
// grid (⌈nseg/8⌉, steps), one warp per segment: its number of interface pixels.
__global__ void __launch_bounds__(256)
    k_setup_iface_count(SetupVolume v, const int* steps, const std::uint8_t* code_iface, int seg, int nseg,
                        int* segoff) {
  const int s = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (s >= nseg) return;
  const int p = steps[blockIdx.y];
  const long long q0 = static_cast<long long>(s) * seg, q1 = min(q0 + seg, v.nn);
  int n = 0;
  for (long long q = q0 + lane; q < q1; q += 32) n += code_iface[setup_code(v, p, q)] != 0;
  for (int o = 16; o > 0; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
  if (lane == 0) segoff[static_cast<long long>(blockIdx.y) * (nseg + 1) + s] = n;
}

// One CTA per step: counts → offsets (nseg + 1 values), copied to the row offsets in 3D
// (rowoff_off[k] ≥ 0).
__global__ void __launch_bounds__(kSetupThreads)
    k_setup_iface_scan(int nseg, int* segoff, const long long* rowoff_off, int* rowoff_pool) {
  __shared__ int s_warp[kSetupThreads / 32];
  const int k = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int* off = segoff + static_cast<long long>(k) * (nseg + 1);
  int* rowoff = rowoff_off[k] >= 0 ? rowoff_pool + rowoff_off[k] : nullptr;
  int running = 0;  // uniform across the CTA
  for (int base = 0; base < nseg; base += kSetupThreads) {
    const int i = base + threadIdx.x;
    const int c = i < nseg ? off[i] : 0;
    int sum = c;  // inclusive scan of the warp
    for (int o = 1; o < 32; o <<= 1) {
      const int up = __shfl_up_sync(0xffffffffu, sum, o);
      if (lane >= o) sum += up;
    }
    if (lane == 31) s_warp[warp] = sum;
    __syncthreads();
    int before = running, total = 0;
    for (int w = 0; w < kSetupThreads / 32; ++w) {
      if (w < warp) before += s_warp[w];
      total += s_warp[w];
    }
    if (i < nseg) {
      off[i] = before + sum - c;
      if (rowoff) rowoff[i] = before + sum - c;
    }
    running += total;
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    off[nseg] = running;
    if (rowoff) rowoff[nseg] = running;
  }
}

// grid as k_setup_iface_count: the pixels of each segment at its offset.
__global__ void __launch_bounds__(256)
    k_setup_iface_write(SetupVolume v, const int* steps, const long long* iface_off,
                        const std::uint8_t* code_iface, int seg, int nseg, const int* segoff,
                        int* iface_pool) {
  const int s = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (s >= nseg) return;
  const int k = blockIdx.y, p = steps[k];
  const int* off = segoff + static_cast<long long>(k) * (nseg + 1) + s;
  if (off[0] == off[1]) return;
  int* out = iface_pool + iface_off[k] + off[0];
  const long long q0 = static_cast<long long>(s) * seg, q1 = min(q0 + seg, v.nn);
  for (long long b = q0; b < q1; b += 32) {
    const long long q = b + lane;
    const bool flag = q < q1 && code_iface[setup_code(v, p, q)];
    const unsigned ballot = __ballot_sync(0xffffffffu, flag);
    if (flag) out[__popc(ballot & ((1u << lane) - 1u))] = static_cast<int>(q);
    out += __popc(ballot);
  }
}

// One warp per row of the pair-id planes: bit i of row_pairs[row] when pair i occurs in it (a step
// has at most kMaxPasses/2 = 64 pairs).
__global__ void k_setup_row_pairs(const std::uint8_t* pid, long long rows, int nx,
                                  unsigned long long* row_pairs) {
  const long long row = (blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x) >> 5;
  if (row >= rows) return;
  const int lane = threadIdx.x & 31;
  unsigned long long m = 0;
  for (int x = lane; x < nx; x += 32) m |= 1ull << pid[row * nx + x];
  for (int o = 16; o > 0; o >>= 1) m |= __shfl_xor_sync(0xffffffffu, m, o);
  if (lane == 0) row_pairs[row] = m;
}

// int32 labels → uint8 (device); sets *bad when a label is outside [0, m).
__global__ void k_labels_to_u8(const std::int32_t* in, std::uint8_t* out, long long count, int m,
                               int* bad) {
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < count;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const std::int32_t v = in[i];
    if (v < 0 || v >= m) {
      *bad = 1;
      out[i] = 0;
    } else {
      out[i] = static_cast<std::uint8_t>(v);
    }
  }
}

}  // namespace bwpm
