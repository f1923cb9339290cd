// A whole Born slab of a 2D solve in one launch of one thread-block cluster.
//
// Per Born slab and direction (cpp/src/solver.cpp:215-382): the Cayley step by GMRES(30), its
// field increment, the sources of the back-scatter and the plane they radiate. As one CUDA graph
// per Born step (build_born_graph in plane_solver.cu, which 3D volumes and other lengths keep)
// that is ≈ 100 small dependent kernels of 2-5 µs on a line of a few thousand points: 730 µs per
// slab and direction at 4096 points in FP64, 106 µs here. The three components' lines are split over a
// cluster of C CTAs and stay on chip: N = C·M, CTA c holds the real-space points C·m + c and a
// block of the spectrum, a transform is a local register-resident M-point transform and one
// all-to-all through distributed shared memory (the scheme of cluster2d.cuh). A thread group per
// component; all pointwise work is on a thread's own values, inner products are all-reduced
// through the same st.async exchange, every CTA applies the Givens rotations itself on the same
// values, so all of them take the same decisions. Where the slab's step is one transmission over
// all pixels, the launch does it too: F⁻¹ is linear, so step and increment share one inverse
// transform and the slab needs no other launch. What is left is latency: per slab and direction of
// a 4096-point chain 10 scatter rounds (two of the sources, the right-hand side, seven operator
// applications) of two transforms and two exchanges each, and 23 all-reduces.
//
// The arithmetic of the pointwise factors and of the inner products is FP64 for both field
// types. Every wait is bounded (status word).
#pragma once

#include <algorithm>

#include "born2d.hpp"
#include "born_kernels.cuh"
#include "chain2d.cuh"
#include "cline.cuh"
#include "gmres_kernels.cuh"

namespace bwpm {

// Mode factors of a host medium (FP64, built once per distinct host): SoA blocks of N values.
// Zero on non-propagating and grazing waves.
enum BornTab : int {
  kBtGreen = 0,  // i dz/(2 k_z)
  kBtG11,        // green·k_z²/k²: the transverse part of the y source
  kBtG12,        // −green·k_y k_z/k²: times the direction, of the z source
  kBtKr,         // k_y/k_z
  kBtHalf,       // e^{i k_z dz/2}
  kBtHalfInv,    // e^{−i k_z dz/2}
  kBtPh0,        // e^{i k_z ζ_0 dz}, then ζ_1
  kBtPh1,
  kBtPh0Inv,
  kBtPh1Inv,
  kBtCount
};

static __global__ void k_born_modes(cd* out, BornGrid g) {
  const long long n = g.ny;
  const long long q = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
  if (q >= n) return;
  const BornPoint p = born_point(g, q);
  if (!p.prop) {
    for (int i = 0; i < kBtCount; ++i) out[i * n + q] = cd{0.0, 0.0};
    return;
  }
  const cd k = g.host * g.k0, k2 = k * k, i{0.0, 1.0};
  const double r3 = 0.57735026918962576451;  // 1/√3
  const double z0 = (1.0 - r3) / 2.0 * g.dz, z1 = (1.0 + r3) / 2.0 * g.dz;
  const cd green = cdiv(cd{0.0, g.dz}, 2.0 * p.kz);
  out[kBtGreen * n + q] = green;
  out[kBtG11 * n + q] = green * cdiv(p.kz * p.kz, k2);
  out[kBtG12 * n + q] = -(green * cdiv(p.ky * p.kz, k2));
  out[kBtKr * n + q] = cdiv(cd{p.ky, 0.0}, p.kz);
  out[kBtHalf * n + q] = cexp(i * p.kz * (g.dz / 2.0));
  out[kBtHalfInv * n + q] = cexp(-i * p.kz * (g.dz / 2.0));
  out[kBtPh0 * n + q] = cexp(i * p.kz * z0);
  out[kBtPh1 * n + q] = cexp(i * p.kz * z1);
  out[kBtPh0Inv * n + q] = cexp(-i * p.kz * z0);
  out[kBtPh1Inv * n + q] = cexp(-i * p.kz * z1);
}

template <typename T>
struct BornSlab {
  const cx<T>* in;       // (N, 2) the plane the slab acts on, or null: its spectrum is given
  const cx<T>* spec;     // F{in} (N, 2) where `in` is null
  const cx<T>* step_tab; // the slab step's transmission table (one pair over all pixels), or null
  cx<T>* out;            // with step_tab: the step's output, set; else a plane the increment is added to
  const cx<T>* incoming; // a radiated plane (times N) added to the output, or null
  cx<T>* radiated;       // the plane radiated against the direction (times N), or null
  const T* mask;         // of the step and its increment, or null
  const cx<T>* pot;      // V per pixel
  const cd* modes;       // kBtCount blocks of N
  const Tw<T>* tw;       // stage twiddles of the M-point plan, then w_N^{c·k1} (C blocks of M)
  cx<T>* basis;          // Krylov vectors beyond those in shared memory, per CTA
  GmresState* state;     // err and applies are written
  int* status;
  int n, dir, basis_smem;
  double tol;
};

// Vectors of a CTA's global scratch: the Krylov basis, the right-hand side, the solution, the spectrum.
constexpr int kBornVectors = kGmresRestart + 4;

namespace born {

// GMRES scalars of a CTA (each CTA computes the same values).
struct Scalars {
  cd h[(kGmresRestart + 1) * kGmresRestart];
  cd cs[kGmresRestart], sn[kGmresRestart], g[kGmresRestart + 1], y[kGmresRestart];
  int flag;
};

}  // namespace born

// threads per CTA, at most: three groups
template <class Inner>
constexpr int born_threads() {
  return Inner::kRuntime ? Inner::kMaxThreads : 3 * Inner::kMaxThreads;
}

template <class Inner, int C>
__global__ void __launch_bounds__(born_threads<Inner>(), 1)
    k_born2d(const __grid_constant__ BornSlab<typename Inner::T> a, const __grid_constant__ FftPlan plan) {
  using T = typename Inner::T;
  using V = cx<T>;
  using L = cl::Line<Inner, C>;
  constexpr int E = L::E, S = L::S, ES = L::ES;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ FftPlan s_plan;
  __shared__ unsigned s_magic[kMaxStages];
  __shared__ alignas(8) unsigned long long s_mbar[2];
  __shared__ cd s_red[16];
  __shared__ born::Scalars sc;
  const int tid = threadIdx.x, group_threads = blockDim.x / 3;
  const int comp = tid / group_threads, t = tid - comp * group_threads;
  int rank = 0;
  if constexpr (C > 1) rank = static_cast<int>(cl::cg::this_cluster().block_rank());
  const int n = a.n, M = n / C, MB = (M + C - 1) / C, pm = rf::padded<T>(M);
  const int mb = max(0, min(MB, M - rank * MB));
  if (tid == 0) {
    s_plan = plan;
    for (int s = 0; s < plan.nstages; ++s)
      s_magic[s] = 0xffffffffu / static_cast<unsigned>(plan.len[s]) + 1u;
    if constexpr (C > 1) {
      r2c::mbar_init(r2c::smem_u32(&s_mbar[0]), 1);
      r2c::mbar_init(r2c::smem_u32(&s_mbar[1]), 1);
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
  }
  // shared memory: exchange lines, receive buffers, twiddles, mode factors of the own block (green,
  // g11, g12, kr), potential, the y/z hand-over, then Krylov vectors
  unsigned char* at = smem;
  auto take = [&](std::size_t bytes) {
    unsigned char* q = at;
    at += (bytes + 15) / 16 * 16;
    return q;
  };
  V* lines = reinterpret_cast<V*>(take(3 * 2 * pm * sizeof(V)));
  const std::size_t recv = C > 1 ? 3 * C * MB * sizeof(V) : 0;
  cl::Xch x;
  x.len = static_cast<unsigned>((recv > 256 ? recv : 256) + 15) / 16 * 16;
  x.base = take(2 * x.len);
  x.mbar0 = r2c::smem_u32(&s_mbar[0]);
  x.parity = 0;
  x.cur = 0;
  x.status = a.status;
  Tw<T>* tws = reinterpret_cast<Tw<T>*>(take(M * sizeof(Tw<T>)));
  Tw<T>* xfs = reinterpret_cast<Tw<T>*>(take((C > 1 ? M : 0) * sizeof(Tw<T>)));
  Tw<T>* xis = reinterpret_cast<Tw<T>*>(take((C > 1 ? C * MB : 0) * sizeof(Tw<T>)));
  cd* modes = reinterpret_cast<cd*>(take(4 * C * MB * sizeof(cd)));
  V* pot = reinterpret_cast<V*>(take(M * sizeof(V)));
  V* hand = reinterpret_cast<V*>(take(C * MB * sizeof(V)));
  V* basis_s = reinterpret_cast<V*>(at);
  for (int i = tid; i < M - 1; i += blockDim.x) tws[i] = a.tw[i];
  if constexpr (C > 1) {
    const Tw<T>* xg = a.tw + (M - 1);
    for (int i = tid; i < M; i += blockDim.x) xfs[i] = xg[static_cast<long long>(rank) * M + i];
    for (int i = tid; i < C * MB; i += blockDim.x) {
      const int d = i / MB, k1 = rank * MB + i - d * MB;
      if (k1 < M) xis[i] = xg[static_cast<long long>(d) * M + k1];
    }
  }
  for (int i = tid; i < C * MB; i += blockDim.x) {
    const int k2 = i / MB, k1 = rank * MB + i - k2 * MB;
    if (k1 < M)
      for (int f = 0; f < 4; ++f) modes[f * C * MB + i] = a.modes[static_cast<long long>(f) * n + k1 + M * k2];
  }
  const double inv_n = 1.0 / static_cast<double>(n);
  for (int i = tid; i < M; i += blockDim.x) pot[i] = a.pot[C * i + rank] * static_cast<T>(inv_n);
  // constants so far; what other kernels of the run write is read after the wait (programmatic
  // dependent launch: this prologue overlaps the slab before)
  asm volatile("griddepcontrol.launch_dependents;");
  L ln{Inner(s_plan, s_magic, M, tws, lines + 2 * comp * pm, t, group_threads), rank, comp, M, MB, mb, xfs, xis};
  const unsigned field_bytes = static_cast<unsigned>(3 * C * mb * sizeof(V));      // forward
  const unsigned inv_bytes = static_cast<unsigned>(3 * M * sizeof(V));             // inverse
  if constexpr (C > 1)
    cl::cg::this_cluster().sync();
  else
    __syncthreads();
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const bool own = ln.own();
  const double dir = static_cast<double>(a.dir);
  auto mode = [&](int f, int s) { return modes[f * C * MB + ln.slot(s)]; };
  // Krylov vector j of this thread's component (x and y): its slots, in shared or global memory
  auto basis_at = [&](int j, int s) -> V* {
    const long long vec = 2LL * C * MB;
    V* b = j < a.basis_smem ? basis_s + j * vec
                            : a.basis + (static_cast<long long>(rank) * kBornVectors + j) * vec;
    return b + comp * C * MB + ln.slot(s);
  };
  constexpr int kRhs = kGmresRestart + 1, kY = kRhs + 1, kSpec = kRhs + 2;  // further vectors
  auto vec_at = [&](int j, int s) -> V* {  // rhs, solution, spectrum: always in global memory
    const long long vec = 2LL * C * MB;
    return a.basis + (static_cast<long long>(rank) * kBornVectors + j) * vec + comp * C * MB + ln.slot(s);
  };
  const bool xy = comp < 2;  // the groups that hold the field's components (the third: E_z)
  auto mine = [&](int s) { return xy && ln.sown(s); };

  // Σ conj(u)·v over the x and y components of the whole line, the same bits in every thread
  auto all_dot = [&](const V (&u)[ES], const V (&v)[ES]) -> cd {
    cd acc{0.0, 0.0};
#pragma unroll
    for (int s = 0; s < S; ++s)
      if (mine(s)) acc = acc + conj(cast<double>(u[s])) * cast<double>(v[s]);
    for (int o = 16; o > 0; o >>= 1) {
      acc.re += __shfl_xor_sync(0xffffffffu, acc.re, o);
      acc.im += __shfl_xor_sync(0xffffffffu, acc.im, o);
    }
    if ((tid & 31) == 0) s_red[tid >> 5] = acc;
    __syncthreads();
    cd sum{0.0, 0.0};
    const int warps = blockDim.x >> 5;
    if constexpr (C == 1) {
      for (int w = 0; w < warps; ++w) sum = sum + s_red[w];
      __syncthreads();
    } else {
      const cd* part = reinterpret_cast<const cd*>(x.buf());
      x.open(C * sizeof(cd));
      if (tid < C) {  // thread d sends this CTA's sum to CTA d
        cd p{0.0, 0.0};
        for (int w = 0; w < warps; ++w) p = p + s_red[w];
        cl::st_async16(r2c::mapa(r2c::smem_u32(part), tid) + rank * sizeof(cd), p,
                         r2c::mapa(x.mbar(), tid));
      }
      x.wait();
      for (int r = 0; r < C; ++r) sum = sum + part[r];
      __syncthreads();  // s_red is written again by the next sum
    }
    return sum;
  };
  // G·w from the scattered sources in direction d: x: green·s_x, y: g11·s_y + d·g12·s_z
  auto radiate = [&](const V (&w)[ES], int s, double d) -> cd {
    if (comp == 0) return mode(kBtGreen, s) * cast<double>(w[s]);
    return mode(kBtG11, s) * cast<double>(w[s]) + d * (mode(kBtG12, s) * cast<double>(hand[ln.slot(s)]));
  };
  auto factor = [&](int f, int s) { return a.modes[static_cast<long long>(f) * n + ln.spos(s)]; };

  // The slab as a loop over transforms, so that the code holds one forward and one inverse
  // transform: each round brings a vector w to real space (all but kInit), acts there, and (scatter
  // rounds: w → F{V·F⁻¹{w}} of three components, kInit) back to the spectrum. `cur` is the vector in
  // hand: the spectrum, then the solution, then the Krylov vector v_j.
  enum { kInit, kSource, kEmit, kRhsOp, kResidual, kArnoldi, kFinal, kIncrement };
  int st = a.in ? kInit : a.radiated ? kSource : kRhsOp;
  V cur[ES], w[ES];
#pragma unroll
  for (int s = 0; s < ES; ++s) cur[s] = V{0, 0};
  if (!a.in)
#pragma unroll
    for (int s = 0; s < S; ++s)
      if (mine(s)) cur[s] = a.spec[2 * ln.spos(s) + comp];
  cd acc[S];
#pragma unroll
  for (int s = 0; s < S; ++s) acc[s] = cd{0.0, 0.0};
  int g = 0, j = 0, outer = 0;
  double tolb = 0.0;
  long long applies = 0;
  bool err = false;
  for (;;) {
    const bool scatter = st != kInit && st != kEmit && st != kIncrement;
#pragma unroll
    for (int s = 0; s < ES; ++s) w[s] = V{0, 0};
    if (st == kInit) {
      if (xy && own)
#pragma unroll
        for (int m = 0; m < E; ++m) w[m] = a.in[2 * ln.pos(m) + comp];
    } else if (st == kResidual || st == kArnoldi || st == kFinal) {  // restricted to propagating waves
#pragma unroll
      for (int s = 0; s < S; ++s)
        if (mine(s)) {
          const cd gr = mode(kBtGreen, s);
          if (gr.re != 0.0 || gr.im != 0.0) w[s] = cur[s];
        }
    } else if (st == kEmit) {
#pragma unroll
      for (int s = 0; s < S; ++s)
        if (mine(s)) w[s] = cast<T>(acc[s]);
    } else {
      // sources: phase to the Gauss point, ζ_g or 1 − ζ_g = ζ_{1−g}; P_½; P_½^{±}
      const int f = st == kSource   ? (a.dir > 0 ? kBtPh0 + g : kBtPh1 - g)
                    : st == kRhsOp  ? static_cast<int>(kBtHalf)
                    : a.dir > 0     ? static_cast<int>(kBtHalf)
                                    : static_cast<int>(kBtHalfInv);
#pragma unroll
      for (int s = 0; s < S; ++s)
        if (mine(s)) w[s] = cast<T>(cast<double>(cur[s]) * factor(f, s));
      if (st == kIncrement && a.step_tab) {
        // the step's transmission and the increment in one inverse transform: forward
        // M·Ê + P_½ y, backward M·(Ê + P_½⁻¹ y); complex64 tables carry 1/N
#pragma unroll
        for (int s = 0; s < S; ++s)
          if (mine(s)) {
            const V e = *vec_at(kSpec, s);
            const cx<T>* tab = a.step_tab + (comp == 0 ? 0 : 2 * n);
            const V u = a.dir > 0 ? e : e + w[s];
            V v = tmul(u, tab, ln.spos(s), 3LL * n);
            if (a.dir > 0) v = v + w[s] * (sizeof(T) == sizeof(double) ? T(1) : static_cast<T>(inv_n));
            w[s] = v;
          }
      }
    }
    if (scatter) {  // E_z = −d·k_y E_y/k_z on the third group
      if (comp == 1)
#pragma unroll
        for (int s = 0; s < S; ++s)
          if (ln.sown(s)) hand[ln.slot(s)] = w[s];
      __syncthreads();
      if (comp == 2)
#pragma unroll
        for (int s = 0; s < S; ++s)
          if (ln.sown(s)) w[s] = cast<T>(-dir * (mode(kBtKr, s) * cast<double>(hand[ln.slot(s)])));
    }
    if (st != kInit) ln.inverse(w, x, inv_bytes);
    if (scatter) {
      if (own)
#pragma unroll
        for (int m = 0; m < E; ++m) w[m] = w[m] * pot[ln.in.pos(m)];
    } else if (st == kEmit) {
      if (xy && own)
#pragma unroll
        for (int m = 0; m < E; ++m) a.radiated[2 * ln.pos(m) + comp] = w[m];
      st = kRhsOp;
      continue;
    } else if (st == kIncrement) {
      if (xy && own)
#pragma unroll
        for (int m = 0; m < E; ++m) {
          const int q = ln.pos(m);
          V v = w[m];
          if (!a.step_tab || sizeof(T) == sizeof(double)) v = v * static_cast<T>(inv_n);
          if (a.mask) v = mmul(v, a.mask, q, static_cast<long long>(n));
          if (!a.step_tab) v = a.out[2 * q + comp] + v;
          if (a.incoming) v = v + a.incoming[2 * q + comp] * static_cast<T>(inv_n);
          a.out[2 * q + comp] = v;
        }
      break;
    }
    ln.forward(w, x, field_bytes);
    if (st == kInit) {
#pragma unroll
      for (int s = 0; s < S; ++s) cur[s] = w[s];
      st = a.radiated ? kSource : kRhsOp;
      continue;
    }
    __syncthreads();
    if (comp == 2)
#pragma unroll
      for (int s = 0; s < S; ++s)
        if (ln.sown(s)) hand[ln.slot(s)] = w[s];
    __syncthreads();
    if (st == kSource) {  // ½·e^{i d′ k_z (1 − ζ_g) dz}·G_{d′} of the source, d′ = −d
      const int f = a.dir > 0 ? kBtPh1Inv - g : kBtPh1 - g;
#pragma unroll
      for (int s = 0; s < S; ++s)
        if (mine(s)) acc[s] = acc[s] + (0.5 * factor(f, s)) * radiate(w, s, -dir);
      if (++g == 2) st = kEmit;
      continue;
    }
    if (st == kRhsOp) {  // rhs = G·P_½Ê, the start y = rhs
#pragma unroll
      for (int s = 0; s < S; ++s) {
        if (mine(s) && a.step_tab) *vec_at(kSpec, s) = cur[s];
        cur[s] = V{0, 0};
        if (mine(s)) {
          cur[s] = cast<T>(radiate(w, s, dir));
          *vec_at(kRhs, s) = cur[s];
          *vec_at(kY, s) = cur[s];
        }
      }
      const double bnorm = sqrt(all_dot(cur, cur).re);
      tolb = a.tol * bnorm;
      st = bnorm == 0.0 ? kIncrement : kResidual;
      continue;
    }
    // w = cur − G·cur/2
    ++applies;
#pragma unroll
    for (int s = 0; s < S; ++s)
      if (mine(s)) {
        const V gv = cast<T>(radiate(w, s, dir));
        w[s] = cast<T>(cast<double>(cur[s]) + -0.5 * cast<double>(gv));
      }
    if (st != kArnoldi) {  // residual of the solution in hand
#pragma unroll
      for (int s = 0; s < S; ++s)
        if (mine(s)) w[s] = cast<T>(cast<double>(*vec_at(kRhs, s)) - cast<double>(w[s]));
      const double beta = sqrt(all_dot(w, w).re);
      if (st == kFinal) {
        st = beta <= tolb * 10.0 ? kIncrement : kResidual;
        continue;
      }
      if (beta <= tolb || outer >= 100) {
        err = !(beta <= tolb);
        st = kIncrement;
        continue;
      }
      ++outer;
#pragma unroll
      for (int s = 0; s < S; ++s)
        if (mine(s)) {
          cur[s] = cast<T>(cast<double>(w[s]) * (1.0 / beta));
          *basis_at(0, s) = cur[s];
        }
      if (tid <= kGmresRestart) sc.g[tid] = cd{tid == 0 ? beta : 0.0, 0.0};
      __syncthreads();
      j = 0;
      st = kArnoldi;
      continue;
    }
    // Arnoldi step j (modified Gram-Schmidt)
    V vi[ES], vn[ES];
#pragma unroll
    for (int s = 0; s < S; ++s)
      if (mine(s)) vn[s] = *basis_at(0, s);
    for (int i = 0; i <= j; ++i) {
#pragma unroll
      for (int s = 0; s < S; ++s) vi[s] = vn[s];
      if (i < j)  // the next vector's loads are in flight during the all-reduce
#pragma unroll
        for (int s = 0; s < S; ++s)
          if (mine(s)) vn[s] = *basis_at(i + 1, s);
      const cd h = all_dot(vi, w);
      if (tid == 0) sc.h[i * kGmresRestart + j] = h;
#pragma unroll
      for (int s = 0; s < S; ++s)
        if (mine(s)) w[s] = cast<T>(cast<double>(w[s]) - h * cast<double>(vi[s]));
    }
    const double hnext = sqrt(all_dot(w, w).re);
    if (hnext > 0.0)
#pragma unroll
      for (int s = 0; s < S; ++s)
        if (mine(s)) {
          cur[s] = cast<T>(cast<double>(w[s]) * (1.0 / hnext));
          *basis_at(j + 1, s) = cur[s];
        }
    if (tid == 0) {  // earlier rotations, the new one (gmres_givens)
      constexpr int m = kGmresRestart;
      for (int i = 0; i < j; ++i) {
        const cd p = sc.h[i * m + j], q = sc.h[(i + 1) * m + j];
        sc.h[i * m + j] = sc.cs[i] * p + sc.sn[i] * q;
        sc.h[(i + 1) * m + j] = -(conj(sc.sn[i]) * p) + sc.cs[i] * q;
      }
      const cd p = sc.h[j * m + j];
      const double aa = hypot(p.re, p.im), rr = sqrt(aa * aa + hnext * hnext);
      if (aa == 0.0) {
        sc.cs[j] = cd{0.0, 0.0};
        sc.sn[j] = cd{1.0, 0.0};
      } else {
        sc.cs[j] = cd{aa / rr, 0.0};
        sc.sn[j] = (p / aa) * (hnext / rr);
      }
      sc.h[j * m + j] = sc.cs[j] * p + sc.sn[j] * hnext;
      sc.g[j + 1] = -(conj(sc.sn[j]) * sc.g[j]);
      sc.g[j] = sc.cs[j] * sc.g[j];
      sc.flag = hypot(sc.g[j + 1].re, sc.g[j + 1].im) <= tolb || hnext == 0.0;
    }
    __syncthreads();
    const bool done = sc.flag;
    if (!done && j + 1 < kGmresRestart) {
      ++j;
      __syncthreads();  // sc.flag is written again
      continue;
    }
    const int used = j + 1;
    if (tid == 0)
      for (int i = used - 1; i >= 0; --i) {
        cd sum = sc.g[i];
        for (int k = i + 1; k < used; ++k) sum = sum - sc.h[i * kGmresRestart + k] * sc.y[k];
        sc.y[i] = cdiv(sum, sc.h[i * kGmresRestart + i]);
      }
    __syncthreads();
#pragma unroll
    for (int s = 0; s < S; ++s)
      if (mine(s)) {
        V v = *vec_at(kY, s);
        for (int k = 0; k < used; ++k)
          v = cast<T>(sc.y[k] * cast<double>(*basis_at(k, s)) + cast<double>(v));
        cur[s] = v;
        *vec_at(kY, s) = v;
      }
    __syncthreads();  // sc is written again by the next cycle
    st = done ? kFinal : kResidual;
  }
  if (rank == 0 && tid == 0) {
    a.state->applies += applies;
    if (err) a.state->err = 1;
  }
  if constexpr (C > 1) cl::cg::this_cluster().sync();  // no CTA leaves while a peer may still send
}

// ---- host side ---------------------------------------------------------------------------------

template <typename T>
inline std::size_t born_smem(int n, int ctas, int basis) {
  const std::size_t M = n / ctas, MB = (M + ctas - 1) / ctas, V = sizeof(cx<T>), blk = ctas * MB;
  auto r16 = [](std::size_t b) { return (b + 15) / 16 * 16; };
  const std::size_t recv = ctas > 1 ? 3 * blk * V : 0;
  return r16(3 * 2 * rf::padded<T>(static_cast<int>(M)) * V) + 2 * r16(std::max<std::size_t>(recv, 256)) +
         r16(M * sizeof(Tw<T>)) + (ctas > 1 ? r16(M * sizeof(Tw<T>)) + r16(blk * sizeof(Tw<T>)) : 0) +
         r16(4 * blk * sizeof(cd)) + r16(M * V) + r16(blk * V) + basis * 2 * blk * V;
}

template <typename T, class Inner, int C>
inline bool born_fill(BornKernel& k, int n, int nt, std::vector<int> radices) {
  const int group = (nt + 31) / 32 * 32;  // whole warps per component
  if (3 * group > born_threads<Inner>()) return false;
  const std::size_t cap = 208 * 1024;  // beside 17 KB of static shared memory
  if (born_smem<T>(n, C, 0) > cap) return false;
  k.fn = (const void*)k_born2d<Inner, C>;
  k.ctas = C;
  k.threads = 3 * group;
  k.radices = std::move(radices);
  while (k.basis_smem < kGmresRestart + 1 && born_smem<T>(n, C, k.basis_smem + 1) <= cap) ++k.basis_smem;
  k.smem = born_smem<T>(n, C, k.basis_smem);
  return true;
}

// The kernel of per-CTA length m = n / C with E values per thread.
template <typename T, int E, int C>
inline bool born_runtime(BornKernel& k, int n) {
  const int m = n / C;
  std::vector<int> radices;
  if (equal_outer_plan(m, E, std::max(1, m / E), radices) >= 1e29) return false;
  return born_fill<T, ch::RuntimeLine<T, E, 384>, C>(k, n, m / E, radices);
}

template <typename T, int C>
inline bool born_cluster(BornKernel& k, int n) {
  if (n % C) return false;
  if (n / C == 512) return born_fill<T, ch::FixedLine<T, 512, 64, rf::Radices<8, 8, 8>>, C>(k, n, 64, {8, 8, 8});
  return born_runtime<T, 8, C>(k, n) || born_runtime<T, 7, C>(k, n) || born_runtime<T, 6, C>(k, n) ||
         born_runtime<T, 5, C>(k, n) || born_runtime<T, 4, C>(k, n) || born_runtime<T, 3, C>(k, n);
}

// Up to 8 CTAs of about 512 points: fewer points leave the exchanges' latency, more the local
// transforms'. FP64, µs per slab and direction: 512 points on one CTA 72 (two 158), 1024 on two 103 (four
// 167), 2048 on four 109 (eight 165), 4096 on eight 109, all on the 8·8·8 core; run-time lengths 640 points
// on two 181, 1280 on four 185, 2560 on eight 185. The largest E is not the fastest of those: E = 4
// takes 106 µs at 640 points, 107 at 1280, 111 at 1536 (E = 8 190), 182 at 2560.
template <typename T>
inline BornKernel born_pick(int n) {
  BornKernel k;
  if ((n >= 2560 && born_cluster<T, 8>(k, n)) || (n >= 1280 && born_cluster<T, 4>(k, n)) ||
      (n >= 640 && born_cluster<T, 2>(k, n)) || born_cluster<T, 1>(k, n) || born_cluster<T, 2>(k, n) ||
      born_cluster<T, 4>(k, n) || born_cluster<T, 8>(k, n))
    return k;
  return BornKernel{};
}

}  // namespace bwpm
