// Register-resident 3D slab-step kernels, FP64 and complex64: compiled lengths (256, 384, 512, 768,
// 1024) and run-time lengths n = E²·m.
//
// Same step as k_cols_step + k_rows_select (plane_kernels.cuh), the path of
// cpp/src/solver_cuda.cu:140-330 (FFT → operator × propagator → inverse FFT → selection by pair
// id → mask), with the transforms held in registers: a thread owns the positions t + m·NT
// (m < E) of one field component of its line, and a stage exchanges through shared memory once
// (two buffers per line, one barrier). Neighbouring lanes hold the two components of the same
// positions, so memory accesses cover whole pixels and the 2×2 operator takes the other
// component by a shuffle. (With both components in a thread a 512² plane gave each SM seven warps,
// issuing on a quarter of the cycles.) The general kernels stage every radix-2..8 pass through
// shared memory twice with two barriers and hold up to 16 values per thread in flight, which left
// them latency-bound with spills.
//
// What a step moves (the planes sit in L2, so this is L2 traffic, and HBM traffic for the tables
// of large planes) bounds it next, and is kept low:
// - Operator tables hold the quarter plane kx ≤ nx/2, ky ≤ ny/2: m00 and m11 are even and m01 is
//   odd in kx and in ky, exactly so in floating point (the entries are products of kx and ky with
//   even terms), so every mode reads the mirrored entry. A CTA's columns are x and nx − x, which
//   read the same entries, once from L2; the row of a pass's table comes into shared memory by bulk
//   copies while the pass before is transformed. At 1024² in complex64 the tables of a two-material
//   volume shrink from 264 to 66 MB (L2: 126 MB).
// - A transmission between equal indices is the propagator alone: one value per mode.
// - A pass serves the rows in which its label pair occurs (row_pairs): the column kernel stores
//   only those, and a CTA of the row kernel transforms only the passes of its rows.
//
// Kernel times of a step (column + row kernel, mean over a lens or facet volume of 12 slabs, warm
// caches), the kernels before → these: FP64 512² 37 + 32 → 12 + 13 µs, 375 × 250 32 + 49 → 15 + 11;
// complex64 512² 9.8 + 12.5 → 9.4 + 10.4, 1024² 73 + 86 → 58 + 32. They issue on a third of the
// cycles; the rest waits on shared memory, barriers and the planes' loads. The prologue of each
// kernel overlaps the end of the one before (programmatic dependent launch).
//
// Data layouts of xbuf and the work planes: x-major (pixel (x, y) at (x·ny + y)·2 + c); `out`,
// pair ids and masks row-major. The twiddles are the per-stage tables of plan.hpp.
#pragma once

#include <algorithm>
#include <utility>
#include <vector>

#include "bulk.cuh"
#include "chain2d.cuh"
#include "plane_kernels.cuh"
#include "plane_rf.hpp"
#include "rfft.cuh"
#include "rgen.cuh"

namespace bwpm {

constexpr int kRfThreads = 512;  // threads per CTA of the run-time lengths, at most

template <typename T>
struct RfCols {
  const cx<T>* in;       // x-transformed field, x-major
  cx<T>* work;           // npass planes, x-major
  cx<T>* spec_out;       // full spectrum F{e} (N, 2) row-major, or null
  const unsigned long long* row_pairs;  // (ny) pairs present in each row, or null: one pair
  const Tw<T>* tw;
  int ny, nx;
  int* status;           // set to 1 when a table copy does not complete in time
};

template <typename T>
struct RfRows {
  const cx<T>* work;        // npass planes after the inverse y transform, x-major
  cx<T>* out;               // (N, 2)
  const uint8_t* pid;       // or null
  const unsigned long long* row_pairs;  // as above
  const T* mask;            // or null
  const int* iface;         // interface pixels of the step (sorted), or null
  const int* rowoff;        // (ny + 1) offsets into iface per row
  cx<T>* refl_out;          // (niface, 2) or null
  const cx<T>* add;         // (niface, 2) or null
  cx<T>* xnext;             // or null: also the x transform of the output rows, x-major
  const Tw<T>* tw;
  int ny, nx;
  int store_out;            // with xnext: 0 when nothing reads `out` later
  T inv_n;
};

namespace rfp {

// A line's exchange buffer holds both components side by side, position pos of component c at
// 2·pos + c, padded by two elements per 16: lanes are (position, component) pairs, so contiguous
// reads and the scattered writes of power-of-two strides are free of bank conflicts in both types.
__device__ __forceinline__ int at(int pos, int c) {
  const int a = 2 * pos + c;
  return a + 2 * (a >> 4);
}
__host__ __device__ constexpr int buffer_len(int n) { return 2 * n + 2 * ((2 * n) >> 4) + 2; }
// Two buffers of a line, and the step to the next line: half a bank row off, so that the lanes of
// a row kernel's two lines do not collide.
template <typename T>
__host__ __device__ constexpr int line_len(int n) {
  constexpr int row = 128 / sizeof(cx<T>);
  return (2 * buffer_len(n) + row - 1) / row * row + row / 2;
}

// Index of position pos + r·STRIDE given b = at(pos, c): a constant step where the padding allows.
template <int STRIDE>
__device__ __forceinline__ int step_at(int b, int pos, int r, int c) {
  if constexpr ((2 * STRIDE) % 16 == 0)
    return b + r * (2 * STRIDE + STRIDE / 4);
  else
    return at(pos + r * STRIDE, c);
}

// One stage of the component's line (cf. rf::gstage).
template <int DIR, int N, int NT, int R, int L, int OFF, bool FIRST, bool LAST, typename T>
__device__ __forceinline__ void stage1(cx<T> (&v)[N / NT], const cx<T>* in, cx<T>* out,
                                       const Tw<T>* __restrict__ tw, int t, int c) {
  constexpr int E = N / NT, NB = N / R, KG = (NB + NT - 1) / NT, K = FIRST || LAST ? E / R : 1;
  static_assert(!(FIRST || LAST) || E % R == 0, "the outer radices must divide the values per thread");
#pragma unroll
  for (int j = 0; j < KG; ++j) {
    const int i = t + j * NT;
    if (NB % NT == 0 || i < NB) {
      const int k = i % L;
      cx<T> u[R];
      const int bi = at(i, c);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        if constexpr (FIRST)
          u[r] = v[j + r * K];
        else
          u[r] = in[step_at<NB>(bi, i, r, c)];
      }
      if constexpr (L > 1) {
#pragma unroll
        for (int r = 1; r < R; ++r) u[r] = twmul<DIR>(u[r], tw[OFF + (r - 1) * L + k]);
      }
      rf::dft<DIR, R>(u);
      if constexpr (LAST) {
#pragma unroll
        for (int r = 0; r < R; ++r) v[j + r * K] = u[r];
      } else {
        const int base = (i - k) * R + k;
        const int bo = at(base, c);
#pragma unroll
        for (int r = 0; r < R; ++r) {
          if constexpr (L == 1 && 16 % (2 * R) == 0)  // one butterfly's outputs share a padding block
            out[bo + 2 * r] = u[r];
          else
            out[step_at<L>(bo, base, r, c)] = u[r];
        }
      }
    }
    asm volatile("" ::: "memory");
  }
  if constexpr (!LAST) __syncthreads();
}

template <int DIR, int N, int NT, int L, int OFF, bool FIRST, int R, int... Rest, typename T>
__device__ __forceinline__ void stages1(cx<T> (&v)[N / NT], cx<T>* base, int& phase,
                                        const Tw<T>* __restrict__ tw, int t, int c) {
  constexpr bool last = sizeof...(Rest) == 0;
  constexpr int B = buffer_len(N);
  stage1<DIR, N, NT, R, L, OFF, FIRST, last>(v, base + (phase ^ 1) * B, base + phase * B, tw, t, c);
  if constexpr (!last) {
    phase ^= 1;
    stages1<DIR, N, NT, L * R, OFF + L * (R - 1), false, Rest...>(v, base, phase, tw, t, c);
  }
}

// An inner stage of radix R of a run-time line over its nt threads.
template <int DIR, int R, typename T>
__device__ __forceinline__ void mid1(const cx<T>* in, cx<T>* out, const Tw<T>* __restrict__ tw, int n,
                                     int L, unsigned magic, int t, int nt, int c) {
  const int nb = n / R;
  for (int i = t; i < nb; i += nt) {
    const int k = rg::mod_magic(i, L, magic);
    cx<T> u[R];
#pragma unroll
    for (int r = 0; r < R; ++r) u[r] = in[at(i + r * nb, c)];
#pragma unroll
    for (int r = 1; r < R; ++r) u[r] = twmul<DIR>(u[r], tw[(r - 1) * L + k]);
    rf::dft<DIR, R>(u);
    const int base = (i - k) * R + k;
#pragma unroll
    for (int r = 0; r < R; ++r) out[at(base + r * L, c)] = u[r];
  }
}

// ---- line policies: geometry of a CTA's lines and the transform of a component's line ----------
// Thread bits from the lowest: the component; rows: the line (an x-major access then covers whole
// sectors), then the position; columns: the position, then the line.

template <typename T_, int N_, int NT_, int LN_, class RADS>
struct Fixed;
template <typename T_, int N_, int NT_, int LN_, int... Rs>
struct Fixed<T_, N_, NT_, LN_, rf::Radices<Rs...>> {
  using T = T_;
  static constexpr int E = N_ / NT_, kThreads = 2 * NT_ * LN_;
  int c, line, t, phase;
  cx<T>* base;
  const Tw<T>* tw;
  __device__ __forceinline__ Fixed(const FftPlan&, int, const Tw<T>* w, unsigned char* smem, bool rows)
      : c(threadIdx.x & 1), phase(0), tw(w) {
    const int h = threadIdx.x >> 1;
    line = rows ? h % LN_ : h / NT_;
    t = rows ? h / LN_ : h % NT_;
    base = line_base(smem, line);
  }
  static __device__ __forceinline__ cx<T>* line_base(unsigned char* smem, int line) {
    return reinterpret_cast<cx<T>*>(smem) + line * line_len<T>(N_);
  }
  // the free buffer of another line of the CTA
  __device__ __forceinline__ cx<T>* free_of(unsigned char* smem, int other) const {
    return line_base(smem, other) + phase * buffer_len(N_);
  }
  __device__ __forceinline__ int lines() const { return LN_; }
  __device__ __forceinline__ bool own() const { return true; }
  __device__ __forceinline__ int pos(int m) const { return t + m * NT_; }
  template <int DIR>
  __device__ __forceinline__ void fft(cx<T> (&v)[E]) {
    stages1<DIR, N_, NT_, 1, 0, true, Rs...>(v, base, phase, tw, t, c);
  }
};

// Run-time length n = E·nt, radices (E, inner …, E); the CTA's first 2·lines·nt threads own values.
template <typename T_, int E_>
struct Runtime {
  using T = T_;
  static constexpr int E = E_, kThreads = kRfThreads;
  int c, line, t, phase, n_, nt, ln;
  cx<T>* base;
  const Tw<T>* tw;
  const FftPlan& plan;
  __device__ __forceinline__ Runtime(const FftPlan& p, int lines, const Tw<T>* w, unsigned char* smem,
                                     bool rows)
      : c(threadIdx.x & 1), phase(0), n_(p.n), nt(p.n / E_), ln(lines), tw(w), plan(p) {
    const int h = threadIdx.x >> 1;
    line = rows ? h % ln : h / nt;
    t = rows ? h / ln : h % nt;
    if (!own()) line = 0;
    base = line_base(smem, line);
  }
  __device__ __forceinline__ cx<T>* line_base(unsigned char* smem, int other) const {
    return reinterpret_cast<cx<T>*>(smem) + other * line_len<T>(n_);
  }
  __device__ __forceinline__ cx<T>* free_of(unsigned char* smem, int other) const {
    return line_base(smem, other) + phase * buffer_len(n_);
  }
  __device__ __forceinline__ int lines() const { return ln; }
  __device__ __forceinline__ bool own() const { return static_cast<int>(threadIdx.x) < 2 * ln * nt; }
  __device__ __forceinline__ int pos(int m) const { return t + m * nt; }
  template <int DIR>
  __device__ __forceinline__ void fft(cx<T> (&v)[E]) {
    const int B = buffer_len(n_);
    if (own()) {
      cx<T>* out = base + phase * B;
      rf::dft<DIR, E>(v);
#pragma unroll
      for (int r = 0; r < E; ++r) out[at(t * E + r, c)] = v[r];
    }
    __syncthreads();
    phase ^= 1;
    for (int s = 1; s + 1 < plan.nstages; ++s) {
      const int L = plan.len[s];
      const Tw<T>* w = tw + plan.twoff[s];
      const unsigned mg = 0xffffffffu / static_cast<unsigned>(L) + 1u;
      if (own()) {
        const cx<T>* in = base + (phase ^ 1) * B;
        cx<T>* out = base + phase * B;
        switch (plan.radix[s]) {
          case 2: mid1<DIR, 2>(in, out, w, n_, L, mg, t, nt, c); break;
          case 3: mid1<DIR, 3>(in, out, w, n_, L, mg, t, nt, c); break;
          case 4: mid1<DIR, 4>(in, out, w, n_, L, mg, t, nt, c); break;
          case 5: mid1<DIR, 5>(in, out, w, n_, L, mg, t, nt, c); break;
          case 6: mid1<DIR, 6>(in, out, w, n_, L, mg, t, nt, c); break;
          case 7: mid1<DIR, 7>(in, out, w, n_, L, mg, t, nt, c); break;
          case 8: mid1<DIR, 8>(in, out, w, n_, L, mg, t, nt, c); break;
          case 9: mid1<DIR, 9>(in, out, w, n_, L, mg, t, nt, c); break;
          case 10: mid1<DIR, 10>(in, out, w, n_, L, mg, t, nt, c); break;
          default: break;  // the host plans inner radices 2 to 10 only
        }
      }
      __syncthreads();
      phase ^= 1;
    }
    if (own()) {  // last stage: sub-length nt, butterfly t
      const cx<T>* in = base + (phase ^ 1) * B;
      const Tw<T>* w = tw + plan.twoff[plan.nstages - 1];
#pragma unroll
      for (int r = 0; r < E; ++r) v[r] = in[at(t + r * nt, c)];
#pragma unroll
      for (int r = 1; r < E; ++r) v[r] = twmul<DIR>(v[r], w[(r - 1) * nt + t]);
      rf::dft<DIR, E>(v);
    }
  }
};

// The other component's value at the same position: lane pairs (2i, 2i + 1) hold them.
template <typename T>
__device__ __forceinline__ cx<T> other_component(cx<T> v) {
  return {__shfl_xor_sync(0xffffffffu, v.re, 1), __shfl_xor_sync(0xffffffffu, v.im, 1)};
}

// CTAs per SM the kernels' registers are sized for: 512 threads per SM, 128 registers (complex64 at
// 768 threads and 80 registers spills: 512² columns 10.4 → 11.2 µs).
constexpr int blocks(int threads) { return 512 / threads > 1 ? 512 / threads : 1; }

// Field value times a table entry: FP64 one value, FP32 hi and lo (16 bytes in both, one load).
__device__ __forceinline__ cd entry(cd u, const Tw<double>& m) { return u * m.hi; }
__device__ __forceinline__ cf entry(cf u, const Tw<float>& m) { return pmul(u, m.hi, m.lo); }
__device__ __forceinline__ Tw<double> signed_entry(Tw<double> m, bool neg) {
  if (neg) m.hi = -m.hi;
  return m;
}
__device__ __forceinline__ Tw<float> signed_entry(Tw<float> m, bool neg) {
  if (neg) {
    m.hi = -m.hi;
    m.lo = -m.lo;
  }
  return m;
}

// Copies the n − 1 stage twiddles of a line's plan to shared memory (room for n). Read through
// L1 they shared it with the planes and tables streaming through (hit rate 50-70 %), and waiting
// for them was two thirds of the stalls.
template <typename T>
__device__ __forceinline__ void stage_twiddles(Tw<T>* dst, const Tw<T>* src, int n) {
  for (int i = threadIdx.x; i < n - 1; i += blockDim.x) dst[i] = src[i];
}

// Programmatic dependent launch: the next kernel of the stream may start its prologue; all reads
// of what the kernel before wrote come after wait_previous (which waits for its completion).
__device__ __forceinline__ void allow_next() { asm volatile("griddepcontrol.launch_dependents;"); }
__device__ __forceinline__ void wait_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

}  // namespace rfp

// y transform of each column, per pass the operator product and the inverse y transform into
// the pass's work plane. A thread holds one component's E values and their spectrum; the other
// component's spectrum comes from the neighbouring lane.
template <class Line>
__global__ void __launch_bounds__(Line::kThreads, rfp::blocks(Line::kThreads))
    k_cols_rf(const __grid_constant__ RfCols<typename Line::T> a, const PassRec* __restrict__ ps,
              int npass, const __grid_constant__ FftPlan plan, int lines) {
  using T = typename Line::T;
  using C = cx<T>;
  constexpr int E = Line::E;
  extern __shared__ __align__(16) unsigned char smem_tw[];
  __shared__ alignas(8) std::uint64_t s_mbar[2];
  const int ny = plan.n, nx = a.nx, hy = ny / 2 + 1;
  // twiddles, the rows' pairs, two buffers of a pass's table row (3 blocks of hy entries), lines
  Tw<T>* tabs = reinterpret_cast<Tw<T>*>(smem_tw + ny * sizeof(Tw<T>) + (ny + 1) / 2 * 16);
  unsigned char* smem_raw = reinterpret_cast<unsigned char*>(tabs + 6 * hy);
  Line ln(plan, lines, reinterpret_cast<const Tw<T>*>(smem_tw), smem_raw, false);
  const long long n = static_cast<long long>(ny) * nx;
  // two lines: columns b and nx − b (0 and, for even nx, nx/2 alone), which read one table row
  const int bx = blockIdx.x, c = ln.c;
  const int x = ln.line == 0 ? bx : nx - bx;
  const bool own = ln.own() && (ln.line == 0 || (bx > 0 && 2 * bx < nx));
  const bool xm = x > nx / 2;
  // quarter-plane tables (blocks m00, m01, m11): row xi of hy entries
  const long long blk = static_cast<long long>(hy) * (nx / 2 + 1);
  const long long trow = static_cast<long long>(2 * bx > nx ? nx - bx : bx) * hy;
  auto fetch = [&](const PassRec& pr, int b) {  // pass table row → buffer b (one thread)
    const Tw<T>* tab = static_cast<const Tw<T>*>(pr.tab) + trow;
    const unsigned bytes = hy * sizeof(Tw<T>);
    bulk_expect(&s_mbar[b], (pr.scalar ? 1u : 3u) * bytes);
    for (int e = 0; e < (pr.scalar ? 1 : 3); ++e)
      bulk_load(tabs + (3 * b + e) * hy, tab + e * blk, bytes, &s_mbar[b]);
  };
  if (threadIdx.x == 0) {
    bulk_mbar_init(&s_mbar[0], 1);
    bulk_mbar_init(&s_mbar[1], 1);
    bulk_fence_init();
  }
  rfp::allow_next();
  // what no kernel of the run writes comes before the wait: twiddles, the rows' pairs, tables
  rfp::stage_twiddles(reinterpret_cast<Tw<T>*>(smem_tw), a.tw, ny);
  unsigned long long* pairs = nullptr;  // the pairs of each row, read by every column and pass
  if (a.row_pairs) {
    pairs = reinterpret_cast<unsigned long long*>(smem_tw + ny * sizeof(Tw<T>));
    for (int y = threadIdx.x; y < ny; y += blockDim.x) pairs[y] = a.row_pairs[y];
  }
  __syncthreads();
  if (threadIdx.x == 0) fetch(ps[0], 0);
  rfp::wait_previous();
  C s[E], w[E];
  if (own) {
#pragma unroll
    for (int m = 0; m < E; ++m) s[m] = a.in[(static_cast<long long>(x) * ny + ln.pos(m)) * 2 + c];
  }
  ln.template fft<-1>(s);
  if (a.spec_out && own)
#pragma unroll
    for (int m = 0; m < E; ++m)
      a.spec_out[2 * (static_cast<long long>(ln.pos(m)) * nx + x) + c] = s[m];
  PassRec pr = ps[0], next = pr;
  unsigned parity = 0;  // bit b: the phase awaited on buffer b
  for (int j = 0; j < npass; ++j, pr = next) {
    const int b = j & 1;
    if (j + 1 < npass) {
      next = ps[j + 1];
      // the other buffer was last read before the previous pass's transform and its barriers
      if (threadIdx.x == 0) fetch(next, b ^ 1);
    }
    bulk_wait(&s_mbar[b], (parity >> b) & 1u, a.status);
    parity ^= 1u << b;
    const Tw<T>* tab = tabs + 3 * b * hy;
    if (pr.scalar) {
      if (own)
#pragma unroll
        for (int m = 0; m < E; ++m) {
          const int y = ln.pos(m);
          w[m] = rfp::entry(s[m], tab[y > ny / 2 ? ny - y : y]);
        }
    } else {
#pragma unroll
      for (int m = 0; m < E; ++m) {
        const C o = rfp::other_component(s[m]);
        const int y = ln.pos(m);
        const bool ym = y > ny / 2;
        const int yi = ym ? ny - y : y;
        if (own) {
          const Tw<T> diag = tab[(c ? 2 * hy : 0) + yi];
          const Tw<T> off = rfp::signed_entry(tab[hy + yi], xm != ym);  // m01 is odd
          w[m] = rfp::entry(s[m], diag) + rfp::entry(o, off);
        }
      }
    }
    ln.template fft<+1>(w);
    C* dst = a.work + static_cast<long long>(j) * 2 * n;
    if (own) {
#pragma unroll
      for (int m = 0; m < E; ++m) {
        const int y = ln.pos(m);
        if (!pairs || (pairs[y] >> pr.pair) & 1)
          dst[(static_cast<long long>(x) * ny + y) * 2 + c] = w[m];
      }
    }
  }
}

// Per CTA its rows: per pass of a pair that occurs in them the inverse x transform of the work
// planes' rows, the selection by pair id, mask and reflection gather; then the sparse sources, the
// output rows and (with xnext) their forward x transform, stored x-major (k_rows_select's
// contract). Every pixel belongs to exactly one transmission pass (its pair's).
template <class Line>
__global__ void __launch_bounds__(Line::kThreads, rfp::blocks(Line::kThreads))
    k_rows_rf(const __grid_constant__ RfRows<typename Line::T> a, const PassRec* __restrict__ ps,
              int npass, const __grid_constant__ FftPlan plan, int lines) {
  using T = typename Line::T;
  using C = cx<T>;
  constexpr int E = Line::E, EW = (E + 3) / 4;
  __shared__ int s_pass[kMaxPasses];
  extern __shared__ __align__(16) unsigned char smem_tw[];
  const int ny = a.ny, nx = plan.n;
  unsigned char* smem_raw = smem_tw + nx * sizeof(Tw<T>);
  Line ln(plan, lines, reinterpret_cast<const Tw<T>*>(smem_tw), smem_raw, true);
  const int LN = ln.lines(), c = ln.c;
  const long long n = static_cast<long long>(ny) * nx;
  const int y0 = blockIdx.x * LN, y1 = min(y0 + LN, ny);
  const bool own = ln.own() && y0 + ln.line < ny;
  const int y = own ? y0 + ln.line : y0;
  const long long row = static_cast<long long>(y) * nx;
  const int k0 = a.iface ? a.rowoff[y0] : 0, k1 = a.iface ? a.rowoff[y1] : 0;
  unsigned long long here = ~0ull;  // pairs in this CTA's rows
  if (a.row_pairs) {
    here = 0;
    for (int r = y0; r < y1; ++r) here |= a.row_pairs[r];
  }
  rfp::allow_next();
  // what no kernel of the run writes comes before the wait: twiddles, pair ids (four to a
  // register), the mask's lines
  rfp::stage_twiddles(reinterpret_cast<Tw<T>*>(smem_tw), a.tw, nx);
  std::uint32_t pw[EW];
#pragma unroll
  for (int i = 0; i < EW; ++i) pw[i] = 0;
  if (a.pid && own) {
#pragma unroll
    for (int m = 0; m < E; ++m)
      pw[m >> 2] |= static_cast<std::uint32_t>(a.pid[row + ln.pos(m)]) << (8 * (m & 3));
  }
  if (a.mask && own)
#pragma unroll
    for (int m = 0; m < E; ++m) {
      prefetch_l1(a.mask + row + ln.pos(m));
      if constexpr (sizeof(T) != sizeof(double)) prefetch_l1(a.mask + n + row + ln.pos(m));
    }
  // the passes of this CTA's rows: pair, and bit 16 for a reflection; −1: left out
  for (int j = threadIdx.x; j < npass; j += blockDim.x) {
    const PassRec r = ps[j];
    s_pass[j] = (here >> r.pair) & 1 ? r.pair | r.refl << 16 : -1;
  }
  __syncthreads();
  rfp::wait_previous();
  auto next_pass = [&](int j) {
    while (j < npass && s_pass[j] < 0) ++j;
    return j;
  };
  C o[E], w[E];
#pragma unroll
  for (int m = 0; m < E; ++m) o[m] = C{0, 0};
  auto load = [&](C(&v)[E], int j) {
    const C* src = a.work + static_cast<long long>(j) * 2 * n;
    if (own) {
#pragma unroll
      for (int m = 0; m < E; ++m) v[m] = src[(static_cast<long long>(ln.pos(m)) * ny + y) * 2 + c];
    }
  };
  // the next pass's values load during the transform where the registers allow
  constexpr bool kAhead = E * sizeof(C) <= 64;
  int j = next_pass(0), jn = j;
  if (j < npass) load(w, j);
  for (; j < npass; j = jn) {
    const int pair = s_pass[j] & 0xffff, refl = s_pass[j] >> 16;
    jn = next_pass(j + 1);
    C wn[kAhead ? E : 1];
    if constexpr (kAhead) {
      if (jn < npass) load(wn, jn);
    }
    ln.template fft<+1>(w);
    if (!refl) {
      if (own) {
#pragma unroll
        for (int m = 0; m < E; ++m)
          if (!a.pid || unpack_pid<E>(pw, m) == pair) o[m] = w[m] * a.inv_n;
      }
    } else {
      // the gather reads other threads' values: through the free buffers, natural order
      if (own) {
        C* f = ln.free_of(smem_raw, ln.line);
#pragma unroll
        for (int m = 0; m < E; ++m) f[rfp::at(ln.pos(m), c)] = w[m];
      }
      __syncthreads();
      for (int k = k0 + threadIdx.x; k < k1; k += blockDim.x) {
        const int q = a.iface[k];
        if (a.pid && a.pid[q] != pair) continue;
        const int qy = q / nx, qx = q - qy * nx;
        const C* f = ln.free_of(smem_raw, qy - y0);
        st_px(a.refl_out + 2 * k, f[rfp::at(qx, 0)] * a.inv_n, f[rfp::at(qx, 1)] * a.inv_n);
      }
      __syncthreads();  // the next transform writes these buffers first
    }
    if constexpr (kAhead) {
#pragma unroll
      for (int m = 0; m < E; ++m) w[m] = wn[m];
    } else {
      if (jn < npass) load(w, jn);
    }
  }
  if (a.mask && own)
#pragma unroll
    for (int m = 0; m < E; ++m) o[m] = mmul(o[m], a.mask, row + ln.pos(m), n);
  if (a.add && k1 > k0) {  // sparse sources (distinct pixels) through the free buffers
    C* f = ln.free_of(smem_raw, ln.line);
    if (own) {
#pragma unroll
      for (int m = 0; m < E; ++m) f[rfp::at(ln.pos(m), c)] = o[m];
    }
    __syncthreads();
    for (int k = k0 + threadIdx.x; k < k1; k += blockDim.x) {
      const int q = a.iface[k];
      const int qy = q / nx, qx = q - qy * nx;
      C* g = ln.free_of(smem_raw, qy - y0);
      C s0, s1;
      ld_px(a.add + 2 * k, s0, s1);
      g[rfp::at(qx, 0)] = g[rfp::at(qx, 0)] + s0;
      g[rfp::at(qx, 1)] = g[rfp::at(qx, 1)] + s1;
    }
    __syncthreads();
    if (own) {
#pragma unroll
      for (int m = 0; m < E; ++m) o[m] = f[rfp::at(ln.pos(m), c)];
    }
    __syncthreads();  // the next transform writes these buffers first
  }
  if ((a.store_out || !a.xnext) && own)
#pragma unroll
    for (int m = 0; m < E; ++m) a.out[2 * (row + ln.pos(m)) + c] = o[m];
  if (a.xnext) {
    ln.template fft<-1>(o);
    if (own) {
#pragma unroll
      for (int m = 0; m < E; ++m) a.xnext[(static_cast<long long>(ln.pos(m)) * ny + y) * 2 + c] = o[m];
    }
  }
}

// CTAs of the column kernel: mirrored pairs of columns, or single ones.
inline unsigned rf_column_ctas(int nx, int lines) {
  return static_cast<unsigned>(lines == 2 ? nx / 2 + 1 : nx);
}

// ---- host side: kernels, shared memory and radix order per run-time length --------------------

// stage twiddles, exchange buffers and, for the column kernel, the rows' pairs and table rows
template <typename T>
constexpr std::size_t rf_smem(int n, int lines, bool cols) {
  return n * sizeof(Tw<T>) + (cols ? (n + 1) / 2 * 16 + 6 * (n / 2 + 1) * sizeof(Tw<T>) : 0) +
         static_cast<std::size_t>(lines) * rfp::line_len<T>(n) * sizeof(cx<T>);
}

template <typename T, int N, int NT, int LN, int... R>
inline RfKernels rf_fixed() {
  using Line = rfp::Fixed<T, N, NT, LN, rf::Radices<R...>>;
  return {(const void*)k_cols_rf<Line>, (const void*)k_rows_rf<Line>, LN, 2 * NT * LN, rf_smem<T>(N, LN, true),
          rf_smem<T>(N, LN, false), {R...}};
}

template <typename T>
struct RfRuntime {
  int e;
  const void *cols, *rows;
};
template <typename T, int E>
inline RfRuntime<T> rf_runtime() {
  using Line = rfp::Runtime<T, E>;
  return {E, (const void*)k_cols_rf<Line>, (const void*)k_rows_rf<Line>};
}

// The run-time kernels of length n: of the E (E² divides n, n/E threads per component and line) from 4
// on with 24 threads or more the one with the fewest stages, each an exchange of both lines and a
// barrier, then the smallest cost (equal_outer_plan); else the other E with the smallest cost. Two lines
// per CTA where they fit. Outer radices 2 and 3 cost rounding error (complex64 against the general
// kernels, mean over facet and lens volumes, transmitted and reflected: E = 3 1.01, 1.02, E = 4 0.96,
// 0.98, E = 6 0.95, 1.04, E = 8 and 10 0.97, 0.98; E = 2 up to 1.12) and threads (24 steps, ms: 500² FP64
// 10·5·10 1.83, 2·5·5·5·2 2.43; 432² FP64 4·3·9·4 1.60, 3·8·6·3 1.72; 405² complex64 9·5·9 1.22, 3·9·5·3
// 1.68); fewer threads leave latency (162² on 18 threads 10 % behind 54). Lengths without an E keep
// the general kernels.
template <typename T>
inline RfKernels rf_pick_runtime(const std::vector<RfRuntime<T>>& all, int n) {
  RfKernels best;
  for (bool suits : {true, false}) {
    std::pair<std::size_t, double> best_score{100, 1e29};
    for (const RfRuntime<T>& c : all) {
      if (2 * (n / c.e) > kRfThreads || n >= 1 << 15 || rf_smem<T>(n, 1, true) > 200 * 1024) continue;
      const int nt = n / c.e;
      if (suits != (c.e >= 4 && nt >= 24)) continue;
      std::vector<int> radices;
      const double cost = equal_outer_plan(n, c.e, nt, radices);
      if (radices.empty()) continue;
      const std::pair<std::size_t, double> score{suits ? radices.size() : 0, cost};
      if (!(score < best_score)) continue;
      best_score = score;
      best.cols = c.cols;
      best.rows = c.rows;
      best.lines = 1;
      if (4 * nt <= kRfThreads && rf_smem<T>(n, 2, true) <= 200 * 1024) best.lines = 2;
      best.threads = (2 * best.lines * nt + 31) / 32 * 32;
      best.cols_smem = rf_smem<T>(n, best.lines, true);
      best.rows_smem = rf_smem<T>(n, best.lines, false);
      best.radices = radices;
    }
    if (best.cols) return best;
  }
  return best;
}

}  // namespace bwpm
