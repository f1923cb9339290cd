// A line of N = C·M points over a thread-block cluster of C CTAs, FP64 or complex64.
//
// The two-factor split of cluster2d.cuh for any per-CTA line (compiled or run-time lengths): CTA c
// holds the real-space points C·m + c; a transform is a local register-resident M-point
// transform, the cross twiddles w_N^{c·k1} and one all-to-all of st.async stores through
// distributed shared memory that completes the C-point stage. The spectrum is owned by blocks of
// MB = ⌈M/C⌉ values k1.
#pragma once

#include <cooperative_groups.h>

#include "cluster2d.cuh"
#include "rgen.cuh"

namespace bwpm {

namespace cl {

namespace cg = cooperative_groups;

__device__ __forceinline__ void st_async16(unsigned raddr, cd v, unsigned rmbar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.b64 [%0], {%1, %2}, [%3];"
               :: "r"(raddr), "l"(__double_as_longlong(v.re)), "l"(__double_as_longlong(v.im)), "r"(rmbar)
               : "memory");
}
__device__ __forceinline__ void send(unsigned raddr, cd v, unsigned rmbar) { st_async16(raddr, v, rmbar); }
__device__ __forceinline__ void send(unsigned raddr, cf v, unsigned rmbar) { r2c::st_async(raddr, v, rmbar); }

// The CTA's exchange state: two receive buffers used in turn, one mbarrier each (see "exchanges
// through distributed shared memory" in cluster2d.cuh: a buffer is written again only after every
// peer has received the exchange between). Fields and inner products take turns on it alike.
struct Xch {
  unsigned char* base;   // the buffers, `len` bytes each
  unsigned len, mbar0;   // and their mbarriers, 8 bytes apart (shared-window address)
  unsigned parity;
  int cur;
  int* status;
  __device__ __forceinline__ unsigned char* buf() const { return base + cur * len; }
  __device__ __forceinline__ unsigned mbar() const { return mbar0 + 8 * cur; }
  __device__ __forceinline__ void open(unsigned bytes) {
    if (threadIdx.x == 0) r2c::mbar_expect(mbar(), bytes);
  }
  __device__ __forceinline__ void wait() {
    r2c::Exchange e;  // one exchange on the current buffer (r2c::xwait: bounded)
    e.mbar[0] = mbar();
    e.parity = (parity >> cur) & 1u;
    e.cur = 0;
    e.status = status;
    r2c::xwait(e);
    parity ^= 1u << cur;
    cur ^= 1;
  }
};

// A component's line over the cluster. Thread t of the group owns the real-space points
// C·(t + m·nt) + c (m < E) and the spectral points c·MB + t + b·nt + M·k2 (b < SB, k2 < C).
template <class Inner, int C>
struct Line {
  using T = typename Inner::T;
  static constexpr int E = Inner::E, SB = (E + C - 1) / C, S = SB * C, ES = S > E ? S : E;
  Inner in;
  int rank, group, M, MB, mb;  // mb: spectral block of this CTA
  const Tw<T>*xf, *xi;         // cross twiddles: w_N^{rank·k1}; block entries [d·MB + k1l] of w_N^{d·k1}
  __device__ __forceinline__ int pos(int m) const { return C * in.pos(m) + rank; }
  __device__ __forceinline__ bool own() const { return in.own(); }
  __device__ __forceinline__ int k1l(int b) const { return in.t + b * in.threads(); }
  __device__ __forceinline__ bool sown(int s) const { return in.own() && k1l(s % SB) < mb; }
  __device__ __forceinline__ int spos(int s) const { return rank * MB + k1l(s % SB) + M * (s / SB); }
  // own slot in a CTA-local array of M spectral values
  __device__ __forceinline__ int slot(int s) const { return k1l(s % SB) + MB * (s / SB); }
  __device__ __forceinline__ cx<T>* recv(const Xch& x) const {
    return reinterpret_cast<cx<T>*>(x.buf()) + group * C * MB;
  }

  // real → spectrum; bytes: what this CTA receives over all groups
  __device__ __forceinline__ void forward(cx<T> (&v)[ES], Xch& x, unsigned bytes) {
    cx<T> u[E];
#pragma unroll
    for (int m = 0; m < E; ++m) u[m] = v[m];
    in.template fft<-1>(u);
    if constexpr (C == 1) {
#pragma unroll
      for (int m = 0; m < E; ++m) v[m] = u[m];
    } else {
      cx<T>* buf = recv(x);
      const unsigned base = r2c::smem_u32(buf), mb0 = x.mbar();
      x.open(bytes);
      if (own()) {
#pragma unroll
        for (int m = 0; m < E; ++m) {
          const int k1 = in.pos(m), dst = k1 / MB;
          const unsigned off = static_cast<unsigned>(rank * MB + k1 - dst * MB) * sizeof(cx<T>);
          send(r2c::mapa(base, dst) + off, rank == 0 ? u[m] : twmul<-1>(u[m], xf[k1]), r2c::mapa(mb0, dst));
        }
      }
      x.wait();
#pragma unroll
      for (int b = 0; b < SB; ++b) {
        cx<T> d[C];
        if (in.own() && k1l(b) < mb) {
#pragma unroll
          for (int r = 0; r < C; ++r) d[r] = buf[r * MB + k1l(b)];
          rf::dft<-1, C>(d);
#pragma unroll
          for (int r = 0; r < C; ++r) v[r * SB + b] = d[r];
        }
      }
    }
  }

  // spectrum → real (unnormalised)
  __device__ __forceinline__ void inverse(cx<T> (&v)[ES], Xch& x, unsigned bytes) {
    cx<T> u[E];
    if constexpr (C == 1) {
#pragma unroll
      for (int m = 0; m < E; ++m) u[m] = v[m];
    } else {
      cx<T>* buf = recv(x);
      const unsigned base = r2c::smem_u32(buf), mb0 = x.mbar();
      x.open(bytes);
#pragma unroll
      for (int b = 0; b < SB; ++b) {
        if (in.own() && k1l(b) < mb) {
          cx<T> d[C];
#pragma unroll
          for (int r = 0; r < C; ++r) d[r] = v[r * SB + b];
          rf::dft<+1, C>(d);
          const unsigned off = static_cast<unsigned>(rank * MB + k1l(b)) * sizeof(cx<T>);
#pragma unroll
          for (int r = 0; r < C; ++r)
            send(r2c::mapa(base, r) + off, r == 0 ? d[r] : twmul<+1>(d[r], xi[r * MB + k1l(b)]),
                 r2c::mapa(mb0, r));
        }
      }
      x.wait();
      if (own()) {
#pragma unroll
        for (int m = 0; m < E; ++m) u[m] = buf[in.pos(m)];
      }
    }
    in.template fft<+1>(u);
#pragma unroll
    for (int m = 0; m < E; ++m) v[m] = u[m];
  }
};

}  // namespace cl
}  // namespace bwpm
