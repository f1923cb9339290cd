// 2D chain kernels of the plane engine: every sweep of a 2D solve (nx = 1) in one launch.
//
// In 2D E_x and E_y are independent (k_x = 0 exactly), so a launch has two CTAs, one per
// component, each running the whole run (forward and backward sweeps, all iterations,
// cpp/src/solver.cpp:444-528) with its line in registers. The launch-per-step form they replace
// (k_step2d) is bound by latency: a launch gap, a global round trip of the line and a shared-memory
// transform with two barriers per stage for every step, on two SMs. Here a step is a register-
// resident forward transform (rfft.cuh, rgen.cuh: one exchange and one barrier per stage), per
// pass the operator product, the inverse transform and the epilogue (selection by pair id, mask,
// reflection gather), then the sparse sources; records of the next step load while the current
// one computes, operator values are brought into L1 during the forward transform. Per step (200
// slabs, tilted facet and mask, launch per step → chain): FP64 256 points 10.5 → 1.8 µs, 1024
// 17.3 → 3.1, 2430 44.4 → 13.7, 4096 41.1 → 15.9; complex64 1024 14.3 → 2.7, 4096 31.0 → 13.4.
//
// A step that nothing acts on in real space (one pair, no mask, no sources to add, plane not
// kept, not the last of its sweep) leaves its result in the spectrum: the inverse transform and
// the next step's forward one are inverse to each other and are both left out (1024 points, planar
// slab without a mask: 14.6 → 0.75 µs per step in FP64).
#pragma once

#include <algorithm>
#include <cstdlib>

#include "chain2d.hpp"
#include "plan.hpp"
#include "plane_kernels.cuh"
#include "resident2d.cuh"
#include "rgen.cuh"

namespace bwpm {

// One run. Component c of pixel q sits at [2·q + c] in all planes and sources.
template <typename T>
struct ChainArgs {
  const cx<T>* input;        // (N, 2)
  cx<T>* t_out;              // (iterations, N, 2); iterations = 0: one plane
  cx<T>* r_out;              // (iterations, N, 2)
  cx<T>* kept_f;             // kept planes, by slot
  cx<T>* kept_b;
  const int* keep;           // (nz + 1) slot of each plane or −1, or null: no plane is kept
  const R2Step* steps;       // nz records; offsets into the pools below
  const PassRec* passes;
  const std::uint8_t* pids;
  const int* iface;
  cx<T>* src_fwd;            // sources of the forward sweep (gathered by the backward one)
  cx<T>* src_bwd;
  const T* mask;             // (N) (FP32: N hi, then N lo values), or null
  cx<T>* spec;               // (2, N) scratch for the spectrum where shared memory has no room
  const Tw<T>* tw;
  int n, nz, iterations;
  int ntw;                   // stage twiddles
  int tw_smem, mask_smem, spec_smem;
  T inv_n;                   // FP64: 1/N after an inverse transform (FP32 tables carry it)
};

namespace ch {

// Lines of a compile-time length: NT threads, N/NT values each.
template <typename T_, int N, int NT_, class RADS>
struct FixedLine {
  using T = T_;
  static constexpr int E = N / NT_, kMaxThreads = NT_;
  static constexpr bool kRuntime = false;
  cx<T>*b0, *b1;
  const Tw<T>* tw;
  int t, phase;
  __device__ __forceinline__ FixedLine(const FftPlan&, const unsigned*, int, const Tw<T>* w, cx<T>* base,
                                       int thread, int)
      : b0(base), b1(base + rf::padded<T>(N)), tw(w), t(thread), phase(0) {}
  __device__ __forceinline__ int n() const { return N; }
  __device__ __forceinline__ int threads() const { return NT_; }
  __device__ __forceinline__ int pos(int m) const { return t + m * NT_; }
  __device__ __forceinline__ bool own() const { return true; }
  template <int DIR>
  __device__ __forceinline__ void fft(cx<T> (&v)[E]) {
    rf::gfft<DIR, N, NT_>(v, b0, b1, phase, tw, t, RADS{});
  }
};

// Lines of any length n = E·nt with a plan (E, inner radices, E) in shared memory; threads t ≥ nt
// own nothing, take their share of the inner stages and join the barriers.
template <typename T_, int E_, int NTMAX>
struct RuntimeLine {
  using T = T_;
  static constexpr int E = E_, kMaxThreads = NTMAX;
  static constexpr bool kRuntime = true;
  const FftPlan& plan;
  const unsigned* magic;
  cx<T>*b0, *b1;
  const Tw<T>* tw;
  int t, gn, nt, n_, phase;
  // thread `thread` of the line's `group` threads
  __device__ __forceinline__ RuntimeLine(const FftPlan& p, const unsigned* mg, int len, const Tw<T>* w,
                                         cx<T>* base, int thread, int group)
      : plan(p), magic(mg), b0(base), b1(base + rf::padded<T>(len)), tw(w), t(thread), gn(group),
        nt(len / E_), n_(len), phase(0) {}
  __device__ __forceinline__ int n() const { return n_; }
  __device__ __forceinline__ int threads() const { return nt; }
  __device__ __forceinline__ int pos(int m) const { return t + m * nt; }
  __device__ __forceinline__ bool own() const { return t < nt; }
  template <int DIR>
  __device__ __forceinline__ void fft(cx<T> (&v)[E]) {
    rg::gfft<DIR, E>(v, b0, b1, phase, plan, magic, tw, t, nt, gn);
  }
};

// Operator value q of a pass: FP64 one value; FP32 hi, and lo three blocks of n further on.
template <typename T>
__device__ __forceinline__ cx<T> op(cx<T> u, const cx<T>* m, int q, int n) {
  return tmul(u, m, q, 3LL * n);
}

template <typename T>
__device__ __forceinline__ void op_prefetch(const cx<T>* m, int q, int n) {
  prefetch_l1(m + q);
  if constexpr (sizeof(T) != sizeof(double)) prefetch_l1(m + 3LL * n + q);
}

// Value times the mask m (FP32: hi values, then lo values n further on).
template <typename T>
__device__ __forceinline__ cx<T> masked(cx<T> v, const T* m, int q, int n) {
  return mmul(v, m, q, n);
}

}  // namespace ch

// Records of the coming step, loaded one step ahead.
struct ChainNext {
  R2Step st;
  PassRec p0;
};

template <class Line>
__global__ void __launch_bounds__(Line::kMaxThreads, 1)
    k_chain2d(const __grid_constant__ ChainArgs<typename Line::T> a,
              const __grid_constant__ FftPlan plan) {
  using T = typename Line::T;
  using C = cx<T>;
  constexpr int E = Line::E, EW = (E + 3) / 4;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ FftPlan s_plan;
  __shared__ unsigned s_magic[kMaxStages];
  const int c = blockIdx.x, t = threadIdx.x, nthr = blockDim.x;
  if constexpr (Line::kRuntime) {
    if (t == 0) {
      s_plan = plan;
      for (int s = 0; s < plan.nstages; ++s)
        s_magic[s] = 0xffffffffu / static_cast<unsigned>(plan.len[s]) + 1u;
    }
    __syncthreads();
  }
  C* lines = reinterpret_cast<C*>(smem_raw);
  Line ln(s_plan, s_magic, a.n, a.tw, lines, t, nthr);
  const int n = ln.n(), pn = rf::padded<T>(n);
  const bool own = ln.own();
  // beside the two exchange lines, where they fit: the stage twiddles, the mask (8 bytes a point
  // in both types), the spectrum of a multi-pass step
  unsigned char* more = smem_raw + 2 * pn * sizeof(C);
  if (a.tw_smem) {
    Tw<T>* tws = reinterpret_cast<Tw<T>*>(more);
    for (int i = t; i < a.ntw; i += nthr) tws[i] = a.tw[i];
    ln.tw = tws;
    more += a.ntw * sizeof(Tw<T>);
  }
  const T* mk = a.mask;
  if (a.mask && a.mask_smem) {
    T* mask_s = reinterpret_cast<T*>(more);
    constexpr int MV = sizeof(T) == sizeof(double) ? 1 : 2;  // mask values per point
    for (int i = t; i < MV * n; i += nthr) mask_s[i] = a.mask[i];
    mk = mask_s;
    more += (8 * n + 15) / 16 * 16;
  }
  C* S = a.spec_smem ? reinterpret_cast<C*>(more) : a.spec + static_cast<long long>(c) * n;
  __syncthreads();
  C v[E], out[E];
  const int sweeps = a.iterations > 0 ? 2 * a.iterations : 1;
  const int iters = a.iterations > 0 ? a.iterations : 1;
  const int eoff = c == 0 ? 0 : 2 * n;  // m00 for E_x, m11 for E_y
  ChainNext nx;
  nx.st = a.steps[0];
  nx.p0 = a.passes[nx.st.fwd_off];
  for (int sw = 0; sw < sweeps; ++sw) {
    const bool backward = sw & 1;
    const int iter = sw >> 1;
    const bool keeps = a.keep && iter == iters - 1;
    C* kept = backward ? a.kept_b : a.kept_f;
    const int first = backward ? a.nz : 0;
    const int slot0 = keeps ? a.keep[first] : -1;
    if (own) {
#pragma unroll
      for (int m = 0; m < E; ++m) {
        const int q = ln.pos(m);
        v[m] = backward ? C{0, 0} : a.input[2 * q + c];
        if (slot0 >= 0) kept[static_cast<long long>(slot0) * 2 * n + 2 * q + c] = v[m];
      }
    }
    bool spectral = false;  // v holds the spectrum (uniform)
    for (int s = 0; s < a.nz; ++s) {
      const int p = backward ? a.nz - 1 - s : s;  // step p: planes p and p + 1
      const R2Step st = nx.st;
      PassRec cur = nx.p0;
      bool next_backward;
      const int next_p = next_step(s, p, a.nz, sw, sweeps, backward, next_backward);
      const bool reflect = r2_reflects(st, backward, a.iterations);
      const int off = backward ? st.bwd_off : st.fwd_off;
      const int npass = r2_passes(st, backward, reflect);
      const bool has_add = st.niface > 0 && (backward || iter > 0);
      C* store = (backward ? a.src_fwd : a.src_bwd) + 2 * st.iface + c;
      const C* add = (backward ? a.src_bwd : a.src_fwd) + 2 * st.iface + c;
      const std::uint8_t* pid = st.pid >= 0 ? a.pids + st.pid : nullptr;
      const int* iface = a.iface + st.iface;
      if (next_p >= 0) nx.st = a.steps[next_p];
      const int slot = keeps ? a.keep[backward ? p : p + 1] : -1;
      // first round of the interface loops
      const bool own_if = t < st.niface;
      const int q0 = own_if ? iface[t] : 0;
      const C a0 = (has_add && own_if) ? add[2 * t] : C{0, 0};
      std::uint32_t pw[EW];
      if (pid && own) {
#pragma unroll
        for (int w = 0; w < EW; ++w) pw[w] = 0;
#pragma unroll
        for (int m = 0; m < E; ++m)
          pw[m >> 2] |= static_cast<std::uint32_t>(pid[ln.pos(m)]) << (8 * (m & 3));
      }
      if (own) {
        const C* m0 = static_cast<const C*>(cur.tab) + eoff;
#pragma unroll
        for (int m = 0; m < E; ++m) ch::op_prefetch(m0, ln.pos(m), n);
      }
      if (!spectral) ln.template fft<-1>(v);
      if (next_p >= 0) nx.p0 = a.passes[next_backward ? nx.st.bwd_off : nx.st.fwd_off];
      const int pid0 = (pid && own_if) ? pid[q0] : 0;
      if (npass > 1 && own) {
#pragma unroll
        for (int m = 0; m < E; ++m) S[ln.pos(m)] = v[m];
      }
      spectral = npass == 1 && !mk && !has_add && slot < 0 && s + 1 < a.nz;
      for (int j = 0; j < npass; ++j) {
        PassRec nxt = cur;
        if (j + 1 < npass) {
          nxt = a.passes[off + j + 1];
          if (own) {
            const C* mn = static_cast<const C*>(nxt.tab) + eoff;
#pragma unroll
            for (int m = 0; m < E; ++m) ch::op_prefetch(mn, ln.pos(m), n);
          }
        }
        const C* tab = static_cast<const C*>(cur.tab) + eoff;
        if (own) {
#pragma unroll
          for (int m = 0; m < E; ++m) {
            const int q = ln.pos(m);
            v[m] = ch::op(npass > 1 ? S[q] : v[m], tab, q, n);
            if ((m & 3) == 3) asm volatile("" ::: "memory");
          }
        }
        if (spectral) {  // FP32 tables carry 1/N for the inverse transform left out here
          if (sizeof(T) != sizeof(double) && own) {
#pragma unroll
            for (int m = 0; m < E; ++m) v[m] = v[m] * static_cast<T>(n);
          }
          break;
        }
        ln.template fft<+1>(v);
        if (own) {
#pragma unroll
          for (int m = 0; m < E; ++m) v[m] = v[m] * a.inv_n;
        }
        if (!cur.refl) {
          if (own) {
#pragma unroll
            for (int m = 0; m < E; ++m) {
              const int q = ln.pos(m);
              if (mk) v[m] = ch::masked(v[m], mk, q, n);
              if (!pid || unpack_pid<E>(pw, m) == cur.pair) out[m] = v[m];
            }
          }
        } else {  // gather at the interface pixels through the free exchange line
          C* buf = ln.phase ? ln.b1 : ln.b0;
          if (own) {
#pragma unroll
            for (int m = 0; m < E; ++m) buf[rf::pad<T>(ln.pos(m))] = v[m];
          }
          __syncthreads();
          if (own_if && (!pid || pid0 == cur.pair)) store[2 * t] = buf[rf::pad<T>(q0)];
          for (int k = t + nthr; k < st.niface; k += nthr) {
            const int q = iface[k];
            if (!pid || pid[q] == cur.pair) store[2 * k] = buf[rf::pad<T>(q)];
          }
          ln.phase ^= 1;
        }
        cur = nxt;
      }
      if (spectral) continue;
      if (own) {
#pragma unroll
        for (int m = 0; m < E; ++m) v[m] = out[m];
      }
      if (has_add) {  // sparse sources at this step's interface pixels
        C* buf = ln.phase ? ln.b1 : ln.b0;
        if (own) {
#pragma unroll
          for (int m = 0; m < E; ++m) buf[rf::pad<T>(ln.pos(m))] = v[m];
        }
        __syncthreads();
        if (own_if) {
          const int q = rf::pad<T>(q0);
          buf[q] = buf[q] + a0;
        }
        for (int k = t + nthr; k < st.niface; k += nthr) {
          const int q = rf::pad<T>(iface[k]);
          buf[q] = buf[q] + add[2 * k];
        }
        __syncthreads();
        if (own) {
#pragma unroll
          for (int m = 0; m < E; ++m) v[m] = buf[rf::pad<T>(ln.pos(m))];
        }
        ln.phase ^= 1;
      }
      if (slot >= 0 && own) {
#pragma unroll
        for (int m = 0; m < E; ++m)
          kept[static_cast<long long>(slot) * 2 * n + 2 * ln.pos(m) + c] = v[m];
      }
    }
    C* dst = (backward ? a.r_out : a.t_out) + static_cast<long long>(iter) * 2 * n + c;
    if (own) {
#pragma unroll
      for (int m = 0; m < E; ++m) dst[2 * ln.pos(m)] = v[m];
    }
  }
}

// ---- host side ---------------------------------------------------------------------------------

// Shared memory of a chain kernel: two exchange lines, then what fits of the stage twiddles (read
// in every stage), the mask (in every step) and the spectrum line (in multi-pass steps). With the
// twiddles left to L1, which the tables and shared memory's share leave small, a 2430-point FP64
// line ran at an L1 hit rate of 38 % and waited on L2 (long scoreboard).
template <typename T>
inline void chain_smem(int n, bool masked, ChainKernel& k) {
  const std::size_t cap = 220 * 1024;
  const std::size_t line = static_cast<std::size_t>(rf::padded<T>(n)) * sizeof(cx<T>);
  const std::size_t mask = (8 * static_cast<std::size_t>(n) + 15) / 16 * 16;
  const std::size_t tw = static_cast<std::size_t>(n - 1) * sizeof(Tw<T>);
  k.smem = 2 * line;
  if (k.smem > cap) {
    k.fn = nullptr;
    return;
  }
  k.tw_smem = k.smem + tw <= cap;
  if (k.tw_smem) k.smem += tw;
  k.mask_smem = masked && k.smem + mask <= cap;
  if (k.mask_smem) k.smem += mask;
  k.spec_smem = k.smem + n * sizeof(cx<T>) <= cap;
  if (k.spec_smem) k.smem += n * sizeof(cx<T>);
}

template <typename T, int N, int NT, int... R>
inline ChainKernel chain_fixed() {
  ChainKernel k;
  k.fn = (const void*)k_chain2d<ch::FixedLine<T, N, NT, rf::Radices<R...>>>;
  k.threads = NT;
  k.radices = {R...};
  return k;
}

// Run-time lengths: the kernel of E values per thread and its thread limit.
struct ChainRuntime {
  int e, max_threads;
  const void* fn;
};
template <typename T, int E>
inline void chain_runtime(std::vector<ChainRuntime>& v) {
  v.push_back({E, 256, (const void*)k_chain2d<ch::RuntimeLine<T, E, 256>>});
  v.push_back({E, 384, (const void*)k_chain2d<ch::RuntimeLine<T, E, 384>>});
  v.push_back({E, 512, (const void*)k_chain2d<ch::RuntimeLine<T, E, 512>>});
}

// The run-time kernel of length n: the E (E² divides n, n/E within the thread limit) with the
// smallest estimate, in the form with the most registers that takes n/E threads (at 128 registers
// FP64 lines spill: 2430 points 17.0 µs per step, 13.7 at 168). 900 FP64 points: E = 5 5.6 µs,
// 3 5.8, 2 6.5, 6 6.9, 10 10.6. Lengths without such an E keep the launch-per-step kernels.
inline ChainKernel chain_pick_runtime(const std::vector<ChainRuntime>& all, int n) {
  ChainKernel best;
  double best_score = 1e30;
  int best_e = 0;
  const char* force = std::getenv("BWPM_CHAIN_E");  // tuning measurements
  for (const ChainRuntime& c : all) {
    if (force && std::atoi(force) != c.e) continue;
    // ordered by thread limit: the first that takes n has the most registers
    if (c.e == best_e || n % (c.e * c.e) || n / c.e > c.max_threads || n >= 1 << 15) continue;
    const int threads = (n / c.e + 31) / 32 * 32;
    std::vector<int> inner;
    const double score = 2 * (14.0 + c.e) + chain_inner(n / (c.e * c.e), n, threads, 10, inner);
    if (score < best_score - 1e-9) {
      best_score = score;
      best_e = c.e;
      best.fn = c.fn;
      best.threads = threads;
      best.radices = {c.e};
      best.radices.insert(best.radices.end(), inner.begin(), inner.end());
      best.radices.push_back(c.e);
    }
  }
  return best;
}

}  // namespace bwpm
