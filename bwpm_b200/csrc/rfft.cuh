// Register-resident FFT for lines of a compile-time length N (complex64 with split constants, or
// FP64).
//
// NT threads, E = N/NT values per thread. Thread t owns positions t + m·NT (m < E): the
// "owned pattern". In the Stockham stage of radix R (sub-length L) the thread's butterflies are
// i = t + j·NT (j < E/R); their inputs x[i + r·N/R] = x[t + (j + r·E/R)·NT] are exactly owned
// positions, and in the last stage (L = N/R) the outputs x'[i + r·L] are owned positions too.
// So a transform takes its input from registers and leaves its output in registers (natural
// order, owned pattern); between stages the values go through shared memory once
// (write scattered, barrier, read owned), alternating two buffers so one barrier suffices.
// Buffers are padded by one element per 16 (pad()), which makes the scattered writes of every
// power-of-two stride and the owned reads free of bank conflicts.
//
// Twiddles: the per-stage r-major tables of plan.hpp (entry (r − 1)·L + k of stage s at offset
// Σ_{s'<s} L_s'·(R_s' − 1)), stored as FP32 (hi, lo) pairs or FP64 values; see fft.cuh for why every
// FP32 constant is carried as a pair.
#pragma once

#include "fft.cuh"

namespace bwpm {
namespace rf {

template <int... Rs>
struct Radices {};

// Padding by the element's size: FP32 complex values (8 bytes) one element per 16, FP64 ones
// (16 bytes: a quarter warp covers the banks) one per 8.
template <typename T = float>
__device__ __forceinline__ int pad(int a) { return a + (a >> (sizeof(T) == sizeof(double) ? 3 : 4)); }
template <typename T = float>
__host__ __device__ constexpr int padded(int n) { return n + n / (sizeof(T) == sizeof(double) ? 8 : 16) + 1; }

// pad(pos + r·STRIDE) given b = pad(pos): a constant step where STRIDE is whole padding blocks.
template <int STRIDE, typename T>
__device__ __forceinline__ int pad_step(int b, int pos, int r) {
  constexpr int blk = sizeof(T) == sizeof(double) ? 8 : 16;
  if constexpr (STRIDE % blk == 0)
    return b + r * (STRIDE + STRIDE / blk);
  else
    return pad<T>(pos + r * STRIDE);
}

// x·exp(DIR·2πi·e/16) with exact (±1, ±i) cases and split constants otherwise.
template <int DIR, int EXP>
__device__ __forceinline__ cf w16mul(cf x) {
  constexpr int e = EXP % 16;
  if constexpr (e == 0) {
    return x;
  } else if constexpr (e == 4) {
    return mul_i<DIR>(x);
  } else if constexpr (e == 8) {
    return -x;
  } else if constexpr (e == 12) {
    return mul_i<-DIR>(x);
  } else {
    constexpr double pi = 3.141592653589793238462643383279502884;
    // cos and sin of 2πe/16 for e = 1, 2, 3, 5, 6, 7, 9, … from the octant values
    constexpr double c1 = 0.92387953251128675613, s1 = 0.38268343236508977173;
    constexpr double r2 = 0.70710678118654752440;
    constexpr double cs[16][2] = {{1, 0},   {c1, s1},   {r2, r2},   {s1, c1},
                                  {0, 1},   {-s1, c1},  {-r2, r2},  {-c1, s1},
                                  {-1, 0},  {-c1, -s1}, {-r2, -r2}, {-s1, -c1},
                                  {0, -1},  {s1, -c1},  {r2, -r2},  {c1, -s1}};
    (void)pi;
    constexpr double c = cs[e][0], s = DIR * cs[e][1];
    const cf hi{static_cast<float>(c), static_cast<float>(s)};
    const cf lo{static_cast<float>(c - static_cast<double>(static_cast<float>(c))),
                static_cast<float>(s - static_cast<double>(static_cast<float>(s)))};
    return pmul(x, hi, lo);
  }
}

template <int DIR>
__device__ __forceinline__ void dft16(cf* u) {
  // n = 4·n1 + n2, m = m1 + 4·m2: DFT4 over n1, twiddle w16^(n2·m1), DFT4 over n2
  cf a[4][4];
#pragma unroll
  for (int n2 = 0; n2 < 4; ++n2) {
    cf x0 = u[n2], x1 = u[n2 + 4], x2 = u[n2 + 8], x3 = u[n2 + 12];
    fftdetail::dft4<DIR>(x0, x1, x2, x3);
    a[n2][0] = x0;
    a[n2][1] = x1;
    a[n2][2] = x2;
    a[n2][3] = x3;
  }
  a[1][1] = w16mul<DIR, 1>(a[1][1]);
  a[1][2] = w16mul<DIR, 2>(a[1][2]);
  a[1][3] = w16mul<DIR, 3>(a[1][3]);
  a[2][1] = w16mul<DIR, 2>(a[2][1]);
  a[2][2] = w16mul<DIR, 4>(a[2][2]);
  a[2][3] = w16mul<DIR, 6>(a[2][3]);
  a[3][1] = w16mul<DIR, 3>(a[3][1]);
  a[3][2] = w16mul<DIR, 6>(a[3][2]);
  a[3][3] = w16mul<DIR, 9>(a[3][3]);
#pragma unroll
  for (int m1 = 0; m1 < 4; ++m1) {
    cf x0 = a[0][m1], x1 = a[1][m1], x2 = a[2][m1], x3 = a[3][m1];
    fftdetail::dft4<DIR>(x0, x1, x2, x3);
    u[m1] = x0;
    u[m1 + 4] = x1;
    u[m1 + 8] = x2;
    u[m1 + 12] = x3;
  }
}

// x·(c ± i·s) for a constant c + i·s (FP32: split).
template <int DIR, typename T>
__device__ __forceinline__ cx<T> cmulk(cx<T> x, double c, double s) {
  const double si = DIR * s;
  if constexpr (sizeof(T) == sizeof(double)) {
    return {fma(x.re, c, -x.im * si), fma(x.re, si, x.im * c)};
  } else {
    const cf hi{static_cast<float>(c), static_cast<float>(si)};
    const cf lo{static_cast<float>(c - static_cast<double>(hi.re)),
                static_cast<float>(si - static_cast<double>(hi.im))};
    return pmul(x, hi, lo);
  }
}

// Radix 9 as 3 × 3: n = 3·n1 + n2, m = m1 + 3·m2, twiddles w9^(n2·m1) (cosines and sines of
// 40°, 80° and 160°).
template <int DIR, typename T>
__device__ __forceinline__ void dft9(cx<T>* u) {
  constexpr double c1 = 0.76604444311897803520, s1 = 0.64278760968653932632;
  constexpr double c2 = 0.17364817766693034885, s2 = 0.98480775301220805937;
  constexpr double c4 = -0.93969262078590838405, s4 = 0.34202014332566873304;
  cx<T> a[3][3];
#pragma unroll
  for (int n2 = 0; n2 < 3; ++n2) {
#pragma unroll
    for (int n1 = 0; n1 < 3; ++n1) a[n2][n1] = u[3 * n1 + n2];
    fftdetail::dft3<DIR>(a[n2]);
  }
  a[1][1] = cmulk<DIR>(a[1][1], c1, s1);
  a[1][2] = cmulk<DIR>(a[1][2], c2, s2);
  a[2][1] = cmulk<DIR>(a[2][1], c2, s2);
  a[2][2] = cmulk<DIR>(a[2][2], c4, s4);
#pragma unroll
  for (int m1 = 0; m1 < 3; ++m1) {
    cx<T> b[3] = {a[0][m1], a[1][m1], a[2][m1]};
    fftdetail::dft3<DIR>(b);
#pragma unroll
    for (int m2 = 0; m2 < 3; ++m2) u[m1 + 3 * m2] = b[m2];
  }
}

// Radix A·B of coprime A, B without twiddles (prime-factor map, I. J. Good 1958): inputs
// n = B·n1 + A·n2, outputs k ≡ k1 (mod A), k2 (mod B).
__host__ __device__ constexpr int pfa_out(int k1, int k2, int A, int B) {
  for (int k = 0; k < A * B; ++k)
    if (k % A == k1 && k % B == k2) return k;
  return 0;
}
template <int DIR, int A, int B, typename T>
__device__ __forceinline__ void dft_pfa(cx<T>* u) {
  cx<T> a[B][A];
#pragma unroll
  for (int n2 = 0; n2 < B; ++n2) {
#pragma unroll
    for (int n1 = 0; n1 < A; ++n1) a[n2][n1] = u[(B * n1 + A * n2) % (A * B)];
    fftdetail::dft<DIR, A>(a[n2]);
  }
#pragma unroll
  for (int k1 = 0; k1 < A; ++k1) {
    cx<T> b[B];
#pragma unroll
    for (int n2 = 0; n2 < B; ++n2) b[n2] = a[n2][k1];
    fftdetail::dft<DIR, B>(b);
#pragma unroll
    for (int k2 = 0; k2 < B; ++k2) u[pfa_out(k1, k2, A, B)] = b[k2];
  }
}

template <int DIR, int R, typename T>
__device__ __forceinline__ void dft(cx<T>* u) {
  static_assert(R != 16 || sizeof(T) == sizeof(float), "radix 16 is FP32 only");
  if constexpr (R == 16)
    dft16<DIR>(u);
  else if constexpr (R == 6)
    dft_pfa<DIR, 2, 3>(u);
  else if constexpr (R == 9)
    dft9<DIR>(u);
  else if constexpr (R == 10)
    dft_pfa<DIR, 2, 5>(u);
  else if constexpr (R == 12)
    dft_pfa<DIR, 3, 4>(u);
  else if constexpr (R == 15)
    dft_pfa<DIR, 3, 5>(u);
  else
    fftdetail::dft<DIR, R>(u);
}

// One stage; v holds the owned values on entry (stage input) and on exit (next stage's input,
// or the transform's output after the last stage).
template <int DIR, int N, int NT, int R, int L, int OFF, bool LAST, typename T>
__device__ __forceinline__ void stage(cx<T> (&v)[N / NT], cx<T>* buf, const Tw<T>* __restrict__ tw,
                                      int t) {
  constexpr int E = N / NT, K = E / R;
  static_assert(E % R == 0, "radix must divide the values per thread");
#pragma unroll
  for (int j = 0; j < K; ++j) {
    const int i = t + j * NT;
    const int k = i % L;
    cx<T> u[R];
#pragma unroll
    for (int r = 0; r < R; ++r) u[r] = v[j + r * K];
    if constexpr (L > 1) {
#pragma unroll
      for (int r = 1; r < R; ++r) u[r] = twmul<DIR>(u[r], tw[OFF + (r - 1) * L + k]);
    }
    dft<DIR, R>(u);
    if constexpr (LAST) {
#pragma unroll
      for (int r = 0; r < R; ++r) v[j + r * K] = u[r];
    } else {
      const int base = (i - k) * R + k;
      const int pb = pad<T>(base);
#pragma unroll
      for (int r = 0; r < R; ++r) buf[pad_step<L, T>(pb, base, r)] = u[r];
    }
    // compiler-only fence: one butterfly's twiddles and temporaries are dead before the next
    // butterfly's loads are issued (keeps the live registers of a stage at one butterfly)
    asm volatile("" ::: "memory");
  }
  if constexpr (!LAST) {
    __syncthreads();
    const int pt = pad<T>(t);
#pragma unroll
    for (int m = 0; m < E; ++m) v[m] = buf[pad_step<NT, T>(pt, t, m)];
  }
}

// A stage whose radix does not divide the values per thread E: the owned values go to in_buf,
// each thread gathers whole butterflies i = t + j·NT < N/R (the last round partly idle), writes
// their outputs to out_buf and reads back its owned values. Two barriers instead of one; the
// caller leaves `phase` as it was (both buffers were used, the last reads were from out_buf).
template <int DIR, int N, int NT, int R, int L, int OFF, typename T>
__device__ __forceinline__ void stage_gather(cx<T> (&v)[N / NT], cx<T>* in_buf, cx<T>* out_buf,
                                             const Tw<T>* __restrict__ tw, int t) {
  constexpr int E = N / NT, NB = N / R, KG = (NB + NT - 1) / NT;
#pragma unroll
  for (int m = 0; m < E; ++m) in_buf[pad<T>(t + m * NT)] = v[m];
  __syncthreads();
#pragma unroll
  for (int j = 0; j < KG; ++j) {
    const int i = t + j * NT;
    if (NB % NT == 0 || i < NB) {
      const int k = i % L;
      cx<T> u[R];
#pragma unroll
      for (int r = 0; r < R; ++r) u[r] = in_buf[pad<T>(i + r * NB)];
      if constexpr (L > 1) {
#pragma unroll
        for (int r = 1; r < R; ++r) u[r] = twmul<DIR>(u[r], tw[OFF + (r - 1) * L + k]);
      }
      dft<DIR, R>(u);
      const int base = (i - k) * R + k;
#pragma unroll
      for (int r = 0; r < R; ++r) out_buf[pad<T>(base + r * L)] = u[r];
    }
    asm volatile("" ::: "memory");
  }
  __syncthreads();
#pragma unroll
  for (int m = 0; m < E; ++m) v[m] = out_buf[pad<T>(t + m * NT)];
}

template <int DIR, int N, int NT, int L, int OFF, int R, int... Rest, typename T>
__device__ __forceinline__ void stages(cx<T> (&v)[N / NT], cx<T>* b0, cx<T>* b1, int& phase,
                                       const Tw<T>* __restrict__ tw, int t) {
  constexpr bool last = sizeof...(Rest) == 0;
  if constexpr ((N / NT) % R == 0) {
    stage<DIR, N, NT, R, L, OFF, last>(v, phase ? b1 : b0, tw, t);
    if constexpr (!last) phase ^= 1;
  } else {
    stage_gather<DIR, N, NT, R, L, OFF>(v, phase ? b1 : b0, phase ? b0 : b1, tw, t);
  }
  if constexpr (!last) stages<DIR, N, NT, L * R, OFF + L * (R - 1), Rest...>(v, b0, b1, phase, tw, t);
}

// ---- transforms whose inner stages take any radix -----------------------------------------------
//
// The first and the last stage's radix divides E, so the transform still goes registers to
// registers in the owned pattern; every stage between reads whole butterflies i = t + j·NT < N/R
// from the exchange buffer that the stage before wrote and writes the other one: one exchange and
// one barrier per stage boundary for any inner radix (stage_gather takes two exchanges). With the
// composite radices 6, 9, 10, 12 and 15 a 3·2^k or 5-smooth line needs as few stages as a power
// of two (384 = 8·6·8, 3072 = 8·8·6·8, 2430 = 9·5·6·9).

template <int DIR, int N, int NT, int R, int L, int OFF, bool FIRST, bool LAST, typename T>
__device__ __forceinline__ void gstage(cx<T> (&v)[N / NT], const cx<T>* in_buf, cx<T>* out_buf,
                                       const Tw<T>* __restrict__ tw, int t) {
  constexpr int E = N / NT, NB = N / R, KG = (NB + NT - 1) / NT, K = FIRST || LAST ? E / R : 1;
  static_assert(!(FIRST || LAST) || E % R == 0, "the outer radices must divide the values per thread");
#pragma unroll
  for (int j = 0; j < KG; ++j) {
    const int i = t + j * NT;
    if (NB % NT == 0 || i < NB) {
      const int k = i % L;
      cx<T> u[R];
      const int pi = pad<T>(i);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        if constexpr (FIRST)
          u[r] = v[j + r * K];
        else
          u[r] = in_buf[pad_step<NB, T>(pi, i, r)];
      }
      if constexpr (L > 1) {
#pragma unroll
        for (int r = 1; r < R; ++r) u[r] = twmul<DIR>(u[r], tw[OFF + (r - 1) * L + k]);
      }
      dft<DIR, R>(u);
      if constexpr (LAST) {
#pragma unroll
        for (int r = 0; r < R; ++r) v[j + r * K] = u[r];
      } else {
        const int base = (i - k) * R + k;
        const int pb = pad<T>(base);
#pragma unroll
        for (int r = 0; r < R; ++r) out_buf[pad_step<L, T>(pb, base, r)] = u[r];
      }
    }
    asm volatile("" ::: "memory");
  }
  if constexpr (!LAST) __syncthreads();
}

template <int DIR, int N, int NT, int L, int OFF, bool FIRST, int R, int... Rest, typename T>
__device__ __forceinline__ void gstages(cx<T> (&v)[N / NT], cx<T>* b0, cx<T>* b1, int& phase,
                                        const Tw<T>* __restrict__ tw, int t) {
  constexpr bool last = sizeof...(Rest) == 0;
  // reads the buffer written by the stage before (phase ^ 1), writes buffer `phase`
  gstage<DIR, N, NT, R, L, OFF, FIRST, last>(v, phase ? b0 : b1, phase ? b1 : b0, tw, t);
  if constexpr (!last) {
    phase ^= 1;
    gstages<DIR, N, NT, L * R, OFF + L * (R - 1), false, Rest...>(v, b0, b1, phase, tw, t);
  }
}

// As fft(), with any inner radices.
template <int DIR, int N, int NT, int... Rs, typename T>
__device__ __forceinline__ void gfft(cx<T> (&v)[N / NT], cx<T>* b0, cx<T>* b1, int& phase,
                                     const Tw<T>* __restrict__ tw, int t, Radices<Rs...>) {
  static_assert((1 * ... * Rs) == N, "radices must multiply to N");
  gstages<DIR, N, NT, 1, 0, true, Rs...>(v, b0, b1, phase, tw, t);
}

// In-register transform of the owned values (DIR −1 forward, +1 inverse unnormalised).
// `phase` selects the exchange buffer and must be uniform across the block; the buffer it
// points to after the transform is free for the caller (no thread still reads it).
template <int DIR, int N, int NT, int... Rs, typename T>
__device__ __forceinline__ void fft(cx<T> (&v)[N / NT], cx<T>* b0, cx<T>* b1, int& phase,
                                   const Tw<T>* __restrict__ tw, int t, Radices<Rs...>) {
  static_assert((1 * ... * Rs) == N, "radices must multiply to N");
  constexpr int E = N / NT;
  constexpr int r[] = {Rs...};
  constexpr bool all = ((E % Rs == 0) && ...);
  if constexpr (!all && E % r[0] == 0 && E % r[sizeof...(Rs) - 1] == 0)
    gfft<DIR, N, NT>(v, b0, b1, phase, tw, t, Radices<Rs...>{});  // inner radices that E does not hold
  else
    stages<DIR, N, NT, 1, 0, Rs...>(v, b0, b1, phase, tw, t);
}

}  // namespace rf
}  // namespace bwpm
