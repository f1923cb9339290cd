// 2D chain kernels of the plane engine: every sweep of a 2D solve (nx = 1) in one launch.
//
// In 2D E_x and E_y are independent (k_x = 0 exactly), so a launch has one CTA, or for long lines
// one cluster, per component, which runs the whole run (forward and backward sweeps, all
// iterations, cpp/src/solver.cpp:444-528) with its line in registers. The launch-per-step form it
// replaces (k_step2d) is bound by latency: a launch gap, a global round trip of the line and a
// shared-memory transform with two barriers per stage for every step, on two SMs. Here a step is a
// register-resident forward transform (rfft.cuh, rgen.cuh: one exchange and one barrier per stage),
// per pass the operator product, the inverse transform and the epilogue (selection by pair id, mask,
// reflection gather), then the sparse sources; records of the next step load while the current
// one computes, operator values are brought into L1 during the forward transform. A line on one SM
// is bound by that SM's FP64 rate and issue from ≈ 1000 points on, so longer lines are split over
// up to eight CTAs (cline.cuh), at an exchange of ≈ 0.7 µs per transform. On split lines the
// cluster-scope acquire of each exchange empties L1, so there the prefetch reaches L2 only: without it
// steps with a mask are 2-4 % faster, steps that stay in the spectrum (below) 3-4 % slower (1024 and 1536
// points, FP64). Per step (200 slabs, tilted facet and mask; launch per step → one CTA → split): FP64 256
// points 10.5 → 1.4 µs, 1024 17.3 → 3.1 → 2.7, 2430 44.4 → 13.7 → 6.9, 4096 41.1 → 15.9 → 5.3, 8192
// 129 → 9.9 (split); complex64 1024 14.3 → 2.7, 2430 26.0 → 11.9 → 7.3, 4096 31.0 → 13.4 → 5.9.
//
// A step that nothing acts on in real space (one pair, no mask, no sources to add, plane not
// kept, not the last of its sweep) leaves its result in the spectrum: the inverse transform and
// the next step's forward one are inverse to each other and are both left out (1024 points, planar
// slab without a mask: 14.6 → 0.75 µs per step in FP64).
#pragma once

#include <algorithm>
#include <cstdlib>

#include "chain2d.hpp"
#include "cline.cuh"
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
  cx<T>* spec;               // scratch for the spectrum where shared memory has no room
  const Tw<T>* tw;           // stage twiddles (of the part), split lines: then w_N^{c·k}
  int n, nz, iterations;
  int* status;               // set to 1 when an exchange of a split line gave up
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

// A whole line on one CTA, or split over a cluster (cline.cuh): real-space values pos(m) (lpos: their
// number within the CTA), spectral values spos(s) (sidx: their place in a CTA-local array).
template <class Inner>
struct Whole {
  using T = typename Inner::T;
  using In = Inner;
  static constexpr int C = 1, E = Inner::E, S = E, ES = E;
  Inner in;
  __device__ __forceinline__ Whole(Inner i) : in(i) {}
  __device__ __forceinline__ Inner& line() { return in; }
  __device__ __forceinline__ bool own() const { return in.own(); }
  __device__ __forceinline__ bool sown(int) const { return in.own(); }
  __device__ __forceinline__ int pos(int m) const { return in.pos(m); }
  __device__ __forceinline__ int lpos(int m) const { return in.pos(m); }
  __device__ __forceinline__ int spos(int s) const { return in.pos(s); }
  __device__ __forceinline__ int sidx(int s) const { return in.pos(s); }
  __device__ __forceinline__ bool mine(int) const { return true; }
  __device__ __forceinline__ int local(int q) const { return q; }
  __device__ __forceinline__ void forward(cx<T> (&v)[ES]) { in.template fft<-1>(v); }
  __device__ __forceinline__ void inverse(cx<T> (&v)[ES]) { in.template fft<+1>(v); }
};

template <class Inner, int C_>
struct Split {
  using T = typename Inner::T;
  using In = Inner;
  using L = cl::Line<Inner, C_>;
  static constexpr int C = C_, E = L::E, S = L::S, ES = L::ES;
  L ln;
  cl::Xch x;
  __device__ __forceinline__ Split(L l, cl::Xch xch) : ln(l), x(xch) {}
  __device__ __forceinline__ Inner& line() { return ln.in; }
  __device__ __forceinline__ bool own() const { return ln.own(); }
  __device__ __forceinline__ bool sown(int s) const { return ln.sown(s); }
  __device__ __forceinline__ int pos(int m) const { return ln.pos(m); }
  __device__ __forceinline__ int lpos(int m) const { return ln.in.pos(m); }
  __device__ __forceinline__ int spos(int s) const { return ln.spos(s); }
  __device__ __forceinline__ int sidx(int s) const { return ln.slot(s); }
  __device__ __forceinline__ bool mine(int q) const { return q % C == ln.rank; }
  __device__ __forceinline__ int local(int q) const { return q / C; }
  __device__ __forceinline__ void forward(cx<T> (&v)[ES]) {
    ln.forward(v, x, static_cast<unsigned>(C * ln.mb * sizeof(cx<T>)));
  }
  __device__ __forceinline__ void inverse(cx<T> (&v)[ES]) {
    ln.inverse(v, x, static_cast<unsigned>(ln.M * sizeof(cx<T>)));
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

// Step `s` of sweep `sw` in execution order, and its record's number; past the last step of the run
// it stays where it is.
struct ChainAt {
  int s, sw;
  __device__ __forceinline__ bool backward() const { return sw & 1; }
  __device__ __forceinline__ int record(int nz) const { return backward() ? nz - 1 - s : s; }
  __device__ __forceinline__ ChainAt next(int nz, int sweeps) const {
    if (s + 1 < nz) return {s + 1, sw};
    if (sw + 1 < sweeps) return {0, sw + 1};
    return *this;
  }
  __device__ __forceinline__ int first_pass(const R2Step& st) const {
    return backward() ? st.bwd_off : st.fwd_off;
  }
};

template <class W>
__global__ void __launch_bounds__(W::In::kMaxThreads, 1)
    k_chain2d(const __grid_constant__ ChainArgs<typename W::T> a,
              const __grid_constant__ FftPlan plan) {
  using T = typename W::T;
  using C = cx<T>;
  constexpr int E = W::E, S = W::S, ES = W::ES, EW = (E + 3) / 4, K = W::C;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ FftPlan s_plan;
  __shared__ unsigned s_magic[kMaxStages];
  __shared__ alignas(8) unsigned long long s_mbar[2];
  // K CTAs (a cluster) per component; M points per CTA, MB of them in its spectral block
  const int c = blockIdx.x / K, rank = blockIdx.x - c * K, t = threadIdx.x, nthr = blockDim.x;
  const int n = a.n, M = n / K, MB = (M + K - 1) / K, pn = rf::padded<T>(M);
  if (t == 0) {
    if constexpr (W::In::kRuntime) {
      s_plan = plan;
      for (int s = 0; s < plan.nstages; ++s)
        s_magic[s] = 0xffffffffu / static_cast<unsigned>(plan.len[s]) + 1u;
    }
    if constexpr (K > 1) {
      r2c::mbar_init(r2c::smem_u32(&s_mbar[0]), 1);
      r2c::mbar_init(r2c::smem_u32(&s_mbar[1]), 1);
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
  }
  // two exchange lines; split lines: two receive buffers and the cross twiddles; then, where they
  // fit, the stage twiddles, the mask (8 bytes a point in both types) and the spectrum of a
  // multi-pass step
  C* lines = reinterpret_cast<C*>(smem_raw);
  unsigned char* more = smem_raw + 2 * pn * sizeof(C);
  const Tw<T>* tws = a.tw;
  Tw<T>*xfs = nullptr, *xis = nullptr;
  cl::Xch x{};
  if constexpr (K > 1) {
    x.base = more;
    x.len = static_cast<unsigned>(K * MB * sizeof(C));
    x.mbar0 = r2c::smem_u32(&s_mbar[0]);
    x.status = a.status;
    more += 2 * x.len;
    xfs = reinterpret_cast<Tw<T>*>(more);
    xis = xfs + M;
    more += (M + K * MB) * sizeof(Tw<T>);
    const Tw<T>* xg = a.tw + (M - 1);
    for (int i = t; i < M; i += nthr) xfs[i] = xg[static_cast<long long>(rank) * M + i];
    for (int i = t; i < K * MB; i += nthr) {
      const int d = i / MB, k1 = rank * MB + i - d * MB;
      if (k1 < M) xis[i] = xg[static_cast<long long>(d) * M + k1];
    }
  }
  if (a.tw_smem) {
    Tw<T>* s = reinterpret_cast<Tw<T>*>(more);
    for (int i = t; i < M - 1; i += nthr) s[i] = a.tw[i];
    tws = s;
    more += (M - 1) * sizeof(Tw<T>);
  }
  const T* mk = a.mask;  // staged: indexed by the CTA's own numbering, lo parts M further on
  if (a.mask && a.mask_smem) {
    T* mask_s = reinterpret_cast<T*>(more);
    for (int i = t; i < M; i += nthr) {
      mask_s[i] = a.mask[K * i + rank];
      if constexpr (sizeof(T) != sizeof(double)) mask_s[M + i] = a.mask[n + K * i + rank];
    }
    mk = mask_s;
    more += (8 * M + 15) / 16 * 16;
  }
  C* spec_line = a.spec_smem ? reinterpret_cast<C*>(more)
                             : a.spec + static_cast<long long>(c * K + rank) * K * MB;
  auto make = [&]() {
    typename W::In in(s_plan, s_magic, M, tws, lines, t, nthr);
    if constexpr (K > 1)
      return W(typename W::L{in, rank, 0, M, MB, max(0, min(MB, M - rank * MB)), xfs, xis}, x);
    else
      return W(in);
  };
  __syncthreads();
  W ln = make();
  auto& in = ln.line();
  const bool own = ln.own();
  const int mo = a.mask_smem ? M : n;  // distance of a mask's lo parts
  if constexpr (K > 1)
    cl::cg::this_cluster().sync();
  else
    __syncthreads();
  C v[ES], out[E];
  const int sweeps = a.iterations > 0 ? 2 * a.iterations : 1;
  const int iters = a.iterations > 0 ? a.iterations : 1;
  const int eoff = c == 0 ? 0 : 2 * n;  // m00 for E_x, m11 for E_y
  // records ahead: the step's own, the next step's, and one pass record each
  ChainAt at1 = ChainAt{0, 0}.next(a.nz, sweeps);
  R2Step st0 = a.steps[0], st1 = a.steps[at1.record(a.nz)];
  PassRec p0 = a.passes[st0.fwd_off];
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
      const R2Step st = st0;
      PassRec cur = p0;
      // the next step's first pass (its record is here) and the record after it: a step that stays
      // in the spectrum is otherwise three dependent loads long
      p0 = a.passes[at1.first_pass(st1)];
      const ChainAt at2 = at1.next(a.nz, sweeps);
      const R2Step st2 = a.steps[at2.record(a.nz)];
      const bool reflect = r2_reflects(st, backward, a.iterations);
      const int off = backward ? st.bwd_off : st.fwd_off;
      const int npass = r2_passes(st, backward, reflect);
      const bool has_add = st.niface > 0 && (backward || iter > 0);
      C* store = (backward ? a.src_fwd : a.src_bwd) + 2 * st.iface + c;
      const C* add = (backward ? a.src_bwd : a.src_fwd) + 2 * st.iface + c;
      const std::uint8_t* pid = st.pid >= 0 ? a.pids + st.pid : nullptr;
      const int* iface = a.iface + st.iface;
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
      {
        const C* m0 = static_cast<const C*>(cur.tab) + eoff;
#pragma unroll
        for (int s2 = 0; s2 < S; ++s2)
          if (ln.sown(s2)) ch::op_prefetch(m0, ln.spos(s2), n);
      }
      if (!spectral) ln.forward(v);
      const int pid0 = (pid && own_if) ? pid[q0] : 0;
      if (npass > 1) {
#pragma unroll
        for (int s2 = 0; s2 < S; ++s2)
          if (ln.sown(s2)) spec_line[ln.sidx(s2)] = v[s2];
      }
      spectral = npass == 1 && !mk && !has_add && slot < 0 && s + 1 < a.nz;
      for (int j = 0; j < npass; ++j) {
        PassRec nxt = cur;
        if (j + 1 < npass) {
          nxt = a.passes[off + j + 1];
          const C* mn = static_cast<const C*>(nxt.tab) + eoff;
#pragma unroll
          for (int s2 = 0; s2 < S; ++s2)
            if (ln.sown(s2)) ch::op_prefetch(mn, ln.spos(s2), n);
        }
        const C* tab = static_cast<const C*>(cur.tab) + eoff;
#pragma unroll
        for (int s2 = 0; s2 < S; ++s2) {
          if (ln.sown(s2)) v[s2] = ch::op(npass > 1 ? spec_line[ln.sidx(s2)] : v[s2], tab, ln.spos(s2), n);
          if ((s2 & 3) == 3) asm volatile("" ::: "memory");
        }
        if (spectral) {  // FP32 tables carry 1/N for the inverse transform left out here
          if constexpr (sizeof(T) != sizeof(double)) {
#pragma unroll
            for (int s2 = 0; s2 < S; ++s2) v[s2] = v[s2] * static_cast<T>(n);
          }
          break;
        }
        ln.inverse(v);
        if (own) {
#pragma unroll
          for (int m = 0; m < E; ++m) v[m] = v[m] * a.inv_n;
        }
        if (!cur.refl) {
          if (own) {
#pragma unroll
            for (int m = 0; m < E; ++m) {
              if (mk) v[m] = ch::masked(v[m], mk, a.mask_smem ? ln.lpos(m) : ln.pos(m), mo);
              if (!pid || unpack_pid<E>(pw, m) == cur.pair) out[m] = v[m];
            }
          }
        } else {  // gather at the interface pixels through the free exchange line
          C* buf = in.phase ? in.b1 : in.b0;
          if (own) {
#pragma unroll
            for (int m = 0; m < E; ++m) buf[rf::pad<T>(ln.lpos(m))] = v[m];
          }
          __syncthreads();
          if (own_if && ln.mine(q0) && (!pid || pid0 == cur.pair))
            store[2 * t] = buf[rf::pad<T>(ln.local(q0))];
          for (int k = t + nthr; k < st.niface; k += nthr) {
            const int q = iface[k];
            if (ln.mine(q) && (!pid || pid[q] == cur.pair)) store[2 * k] = buf[rf::pad<T>(ln.local(q))];
          }
          in.phase ^= 1;
        }
        cur = nxt;
      }
      st0 = st1;
      st1 = st2;
      at1 = at2;
      if (spectral) continue;
      if (own) {
#pragma unroll
        for (int m = 0; m < E; ++m) v[m] = out[m];
      }
      if (has_add) {  // sparse sources at this step's interface pixels
        C* buf = in.phase ? in.b1 : in.b0;
        if (own) {
#pragma unroll
          for (int m = 0; m < E; ++m) buf[rf::pad<T>(ln.lpos(m))] = v[m];
        }
        __syncthreads();
        if (own_if && ln.mine(q0)) {
          const int q = rf::pad<T>(ln.local(q0));
          buf[q] = buf[q] + a0;
        }
        for (int k = t + nthr; k < st.niface; k += nthr) {
          const int g = iface[k];
          if (!ln.mine(g)) continue;
          const int q = rf::pad<T>(ln.local(g));
          buf[q] = buf[q] + add[2 * k];
        }
        __syncthreads();
        if (own) {
#pragma unroll
          for (int m = 0; m < E; ++m) v[m] = buf[rf::pad<T>(ln.lpos(m))];
        }
        in.phase ^= 1;
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
  if constexpr (K > 1) cl::cg::this_cluster().sync();  // no CTA leaves while a peer may still send
}

// ---- host side ---------------------------------------------------------------------------------

// Shared memory of a chain kernel: two exchange lines, then what fits of the stage twiddles (read
// in every stage), the mask (in every step) and the spectrum line (in multi-pass steps). With the
// twiddles left to L1, which the tables and shared memory's share leave small, a 2430-point FP64
// line ran at an L1 hit rate of 38 % and waited on L2 (long scoreboard).
template <typename T>
inline void chain_smem(int n, bool masked, ChainKernel& k) {
  const std::size_t cap = 220 * 1024;
  const int m = n / k.ctas, mb = (m + k.ctas - 1) / k.ctas;
  const std::size_t line = static_cast<std::size_t>(rf::padded<T>(m)) * sizeof(cx<T>);
  const std::size_t mask = (8 * static_cast<std::size_t>(m) + 15) / 16 * 16;
  const std::size_t tw = static_cast<std::size_t>(m - 1) * sizeof(Tw<T>);
  const std::size_t spec = static_cast<std::size_t>(k.ctas) * mb * sizeof(cx<T>);
  k.smem = 2 * line;
  if (k.ctas > 1) k.smem += 2 * spec + (m + static_cast<std::size_t>(k.ctas) * mb) * sizeof(Tw<T>);
  if (k.smem > cap) {
    k.fn = nullptr;
    return;
  }
  k.tw_smem = k.smem + tw <= cap;
  if (k.tw_smem) k.smem += tw;
  k.mask_smem = masked && k.smem + mask <= cap;
  if (k.mask_smem) k.smem += mask;
  k.spec_smem = k.smem + spec <= cap;
  if (k.spec_smem) k.smem += spec;
}

// Compiled lengths: K parts of N points on NT threads each.
template <typename T, int K, int N, int NT, int... R>
inline ChainKernel chain_fixed() {
  using In = ch::FixedLine<T, N, NT, rf::Radices<R...>>;
  ChainKernel k;
  if constexpr (K == 1)
    k.fn = (const void*)k_chain2d<ch::Whole<In>>;
  else
    k.fn = (const void*)k_chain2d<ch::Split<In, K>>;
  k.ctas = K;
  k.threads = NT;
  k.radices = {R...};
  return k;
}

// Run-time lengths from here on are split over a cluster where they divide (FP64, µs per step, whole →
// split: 1000 points 4.9 → 4.7, 1080 6.1 → 4.6, 1500 7.1 → 5.3; complex64 5.2 → 5.4, 6.1 → 4.8,
// 7.3 → 5.8; 900 points and below gain nothing).
constexpr int kChainSplitMin = 1024;

// Run-time lengths: the kernel of E values per thread, its thread limit and parts per line.
struct ChainRuntime {
  int e, max_threads, ctas;
  const void* fn;
};
template <typename T, int E>
inline void chain_runtime(std::vector<ChainRuntime>& v) {
  v.push_back({E, 256, 1, (const void*)k_chain2d<ch::Whole<ch::RuntimeLine<T, E, 256>>>});
  v.push_back({E, 384, 1, (const void*)k_chain2d<ch::Whole<ch::RuntimeLine<T, E, 384>>>});
  v.push_back({E, 512, 1, (const void*)k_chain2d<ch::Whole<ch::RuntimeLine<T, E, 512>>>});
}
template <typename T, int E, int K>
inline void chain_runtime_split(std::vector<ChainRuntime>& v) {
  v.push_back({E, 256, K, (const void*)k_chain2d<ch::Split<ch::RuntimeLine<T, E, 256>, K>>});
}

// Whether E values per thread suit a line of `ctas` parts. Whole lines: 4 to 8; outer radices 2 and 3
// cost rounding error (against the launch-per-step kernels, mean over 25 plans of E = 3: complex64 1.03,
// FP64 1.02; E = 4 to 8 0.98, 0.90) and stages (972 points FP64 6.7 → 5.9 µs per step), above 8 a line
// has a warp or two (225 points, E = 5 3.6 µs, 15 4.8). Parts: at most one block of the cross stage per
// thread, E ≤ ctas (4374 points on 6 CTAs, E = 3 7.9 µs per step, E = 9 14.2).
inline bool chain_suits(int e, int ctas) { return ctas == 1 ? e >= 4 && e <= 8 : e <= ctas; }

// The run-time kernel of length n among those of `ctas` parts: the E (E² divides n/ctas, within the
// thread limit) with the smallest cost, in the form with the most registers that takes its threads
// (at 128 registers FP64 lines spill: 2430 points 17.0 µs per step, 13.7 at 168). `suits`: only E that
// suit the parts. Lengths without an E keep the launch-per-step kernels.
inline ChainKernel chain_pick_runtime(const std::vector<ChainRuntime>& all, int n, int ctas, bool suits) {
  ChainKernel best;
  double best_score = 1e29;
  int best_e = 0;
  if (n % ctas || n >= 1 << 15) return best;
  const int m = n / ctas;
  for (const ChainRuntime& c : all) {
    // ordered by thread limit: the first that takes n has the most registers
    if (c.ctas != ctas || c.e == best_e || m % c.e || m / c.e > c.max_threads) continue;
    if (suits && !chain_suits(c.e, ctas)) continue;
    const int threads = (m / c.e + 31) / 32 * 32;
    std::vector<int> radices;
    const double score = equal_outer_plan(m, c.e, threads, radices);
    if (score < best_score - 1e-9) {
      best_score = score;
      best_e = c.e;
      best.fn = c.fn;
      best.ctas = ctas;
      best.threads = threads;
      best.radices = radices;
    }
  }
  return best;
}

// The run-time chain kernel of length n, of the first part count that has a plan and its shared memory:
// from kChainSplitMin points on those of `parts`, with an E that suits them, then with any; then the
// whole line.
template <typename T>
inline ChainKernel chain_runtime_kernel(const std::vector<ChainRuntime>& all, int n, bool masked,
                                        std::vector<int> parts) {
  if (n < kChainSplitMin) parts.clear();
  for (const std::vector<int>& counts : {parts, std::vector<int>{1}})
    for (bool suits : {true, false})
      for (int ctas : counts) {
        ChainKernel k = chain_pick_runtime(all, n, ctas, suits);
        if (k.fn) chain_smem<T>(n, masked, k);
        if (k.fn) return k;
      }
  return ChainKernel{};
}

}  // namespace bwpm
