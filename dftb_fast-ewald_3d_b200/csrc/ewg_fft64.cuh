// ewg_fft64.cuh -- the five FP64 transform passes at the lengths of kLengths64,
// each a product of two radices of at most 24.
//
// What bounds a pass is the traffic of its grids through L2 and HBM and, before
// that, how many loads an SM has in flight: with three radices of at most 8 a
// line went three times through registers and twice through shared memory, each
// thread with 5 to 8 loads outstanding between barriers.  Here a line goes
// through registers twice (32,769 atoms, 192 points per axis, in us: x R2C 23, y
// forward 16, z 41, y inverse 41, x C2R 81; 216,000 sites, 336 points: 146, 88, 265,
// 262, 560, the last two at 4.0 and 3.4 TB/s; a batch of 128 cells: forward 425, inverse
// 598): a thread loads R0 elements of its line at once, does
// an R0-point transform in registers, leaves them in one shared buffer, and after
// one barrier takes R1 of them through the second transform and out.  A CTA
// holds 8 lines (128-byte rows: global and shared accesses are coalesced and
// free of conflicts) and 8 max(R0, R1) threads.
//
// A single cell runs one kernel per pass and length.  The cells of a batch have
// many lengths: launches per length would each end in a part-filled wave, and one
// launch for all would give every block the registers, threads and shared memory
// of the longest, so a batch runs one kernel per pass and class of lengths
// (kClass64), its blocks ordered from the longest line to the shortest.
#pragma once

#include <atomic>
#include <initializer_list>
#include <type_traits>
#include <utility>

#include "ewg_dft.cuh"
#include "ewg_kernels.h"

namespace ewg {

// The lengths that have these passes, each with its two radices, its class and the
// source file (a single cell's kernels; they build in parallel) that instantiates it:
// whole tiles of 8 points, the products of two radices of at most 24 that the grids
// of either window reach most often.  504 = 24 x 21 and the lengths above 576 are left
// to the runtime schedule.  The class bounds the registers, threads (64, 96, 128, 192) and shared
// memory that a batch's launch gives every block.
struct Length64 {
  int n, r0, r1, klass, unit;
};
constexpr int kUnits64 = 7;
constexpr Length64 kLengths64[] = {
    {16, 4, 4, 0, 0},
    {24, 6, 4, 0, 1},
    {32, 8, 4, 0, 2},
    {40, 8, 5, 0, 4},
    {48, 8, 6, 0, 0},
    {56, 8, 7, 0, 5},
    {64, 8, 8, 0, 4},
    {72, 9, 8, 1, 2},
    {80, 10, 8, 1, 1},
    {96, 12, 8, 1, 6},
    {112, 14, 8, 2, 0},
    {120, 12, 10, 2, 3},
    {128, 16, 8, 2, 3},
    {144, 12, 12, 2, 1},
    {160, 16, 10, 2, 6},
    {168, 14, 12, 2, 2},
    {192, 16, 12, 2, 4},
    {200, 20, 10, 3, 1},
    {216, 18, 12, 3, 0},
    {224, 16, 14, 2, 5},
    {240, 16, 15, 2, 2},
    {256, 16, 16, 2, 4},
    {280, 20, 14, 3, 5},
    {288, 18, 16, 3, 3},
    {320, 20, 16, 3, 6},
    {336, 21, 16, 3, 6},
    {360, 20, 18, 3, 5},
    {384, 24, 16, 3, 3},
    {400, 20, 20, 3, 4},
    {432, 24, 18, 3, 2},
    {480, 24, 20, 3, 1},
    {576, 24, 24, 3, 0},
};
constexpr int kCount64 = sizeof(kLengths64) / sizeof(kLengths64[0]);

// LF: lines that are neighbours in the thread index (and in shared memory), 8 for
// the strided axes, whose memory holds neighbouring lines side by side, 4 or 1 for
// the x axis, whose memory holds a line's elements side by side.  The CTA's 8 / LF
// groups of lines follow one another.
template <int N, int R0, int R1>
struct TwoPass {
  static_assert(R0 * R1 == N, "radices");
  static constexpr int L = 8;
  static constexpr int length = N;
  static constexpr int radix0 = R0, radix1 = R1;
  static constexpr int per_line = R0 > R1 ? R0 : R1;  // threads per line
  static constexpr int threads = L * per_line;
  // Element e of a line between the radices sits at (e + e / R0) LF (+ the line): the
  // padding keeps the strided writes of the first radix free of bank conflicts
  // when fewer than 8 lines lie side by side.
  static constexpr int padded(int lf) { return lf < 8 ? N + R1 : N; }
  // Shared elements of one transform.
  static constexpr int elems(int lf) { return padded(lf) * L; }

  // This thread's place: line within its group, butterfly, group.
  template <int LF>
  struct At {
    int line, i, group;
    // A batch's CTA can have more threads than this length uses: they get an i or a
    // group past the last.
    __device__ __forceinline__ At()
        : line(threadIdx.x % LF),
          i(LF == 8 ? threadIdx.x / 8 : threadIdx.x / LF % per_line),
          group(LF == 8 ? 0 : threadIdx.x / (LF * per_line)) {}
  };

  // First radix: u holds elements i + j R1 of the thread's line.
  template <int SIGN, int LF>
  __device__ __forceinline__ static void first(const At<LF>& t, cx<double> (&u)[R0],
                                               cx<double>* __restrict__ a) {
    constexpr int kStep = LF < 8 ? R0 + 1 : R0;
    dft_reg<double, SIGN, R0>(u);
    cx<double>* dst = a + (t.group * padded(LF) + t.i * kStep) * LF + t.line;
#pragma unroll
    for (int j = 0; j < R0; ++j) dst[j * LF] = u[j];
  }
  // Second radix: v becomes elements i + j R0 of the result.
  template <int SIGN, int LF>
  __device__ __forceinline__ static void second(const At<LF>& t, const cx<double>* __restrict__ a,
                                                const cx<double>* __restrict__ tw,
                                                cx<double> (&v)[R1]) {
    constexpr int kStep = LF < 8 ? R0 + 1 : R0;
    const cx<double>* src = a + (t.group * padded(LF) + t.i) * LF + t.line;
#pragma unroll
    for (int j = 0; j < R1; ++j) v[j] = src[j * kStep * LF];
    // Twiddles w^(i j), w = exp(SIGN 2 pi i / N): every fourth power from the table,
    // the others one or two products away (a few ulp).
    cx<double> w1 = twiddle(tw, t.i, SIGN), w2, w3;
    if (R1 > 2) w2 = mul(w1, w1);
    if (R1 > 3) w3 = mul(w2, w1);
    cx<double> base = w1;
#pragma unroll
    for (int j = 1; j < R1; ++j) {
      if (j % 4 == 0) base = twiddle(tw, t.i * j, SIGN);
      cx<double> w;
      if (j < 4)
        w = j == 1 ? w1 : (j == 2 ? w2 : w3);
      else
        w = j % 4 == 0 ? base : mul(base, j % 4 == 1 ? w1 : (j % 4 == 2 ? w2 : w3));
      v[j] = mul(v[j], w);
    }
    dft_reg<double, SIGN, R1>(v);
  }
};

__device__ __forceinline__ cx<double> times_i(cx<double> v, double f) { return mk(-f * v.y, f * v.x); }

// x, real to complex: row pairs (2p, 2p+1) form one complex line; k1 = 0..K1-1
// of each row is kept.  Neighbouring threads take neighbouring x of one line.
template <class SH>
__device__ __forceinline__ void x_r2c_body(const PassCell& pc, int bx) {
  constexpr int L = SH::L, n1 = SH::length, R0 = SH::radix0, R1 = SH::radix1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cx<double>* a = reinterpret_cast<cx<double>*>(smem_raw);
  const cx<double>* tw = plan_twiddles<double>(pc.fft[0]);
  const int K1 = pc.g.K1, npairs = pc.g.n[1] * pc.g.n[2] / 2;
  const typename SH::template At<1> t;
  const int pair0 = bx * L, mine = min(pair0 + t.group, npairs - 1);
  if (t.i < R1 && t.group < L) {
    const double* ra = static_cast<const double*>(pc.grid) + static_cast<size_t>(2 * mine) * n1 + t.i;
    cx<double> u[R0];
#pragma unroll
    for (int j = 0; j < R0; ++j) u[j] = mk(ra[j * R1], ra[n1 + j * R1]);
    SH::template first<-1, 1>(t, u, a);
  }
  __syncthreads();
  cx<double> v[R1];
  const bool on = t.i < R0 && t.group < L;
  if (on) SH::template second<-1, 1>(t, a, tw, v);
  __syncthreads();
  if (on) {
#pragma unroll
    for (int j = 0; j < R1; ++j) a[t.group * n1 + t.i + j * R0] = v[j];
  }
  __syncthreads();
  // The two rows' spectra from the line's, k1 fastest: whole rows of output.
  cx<double>* A1 = static_cast<cx<double>*>(pc.A1);
  for (int l = threadIdx.x / 32; l < L && pair0 + l < npairs; l += (blockDim.x + 31) / 32) {
    const cx<double>* z0 = a + l * n1;
    cx<double>* o = A1 + static_cast<size_t>(2 * (pair0 + l)) * K1;
    for (int k = threadIdx.x & 31; k < K1; k += min(32, blockDim.x - (threadIdx.x & ~31))) {
      const cx<double> z = z0[k], zc = z0[k == 0 ? 0 : n1 - k];
      o[k] = mk(0.5 * (z.x + zc.x), 0.5 * (z.y - zc.y));
      o[K1 + k] = mk(0.5 * (z.y + zc.y), -0.5 * (z.x - zc.x));
    }
  }
}

// y forward: lines over i2 for (i3, 8 values of k1); keeps k2 in [-H2, H2].
template <class SH>
__device__ __forceinline__ void y_fwd_body(const PassCell& pc, int local) {
  constexpr int L = SH::L, n2 = SH::length, R0 = SH::radix0, R1 = SH::radix1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cx<double>* a = reinterpret_cast<cx<double>*>(smem_raw);
  const cx<double>* tw = plan_twiddles<double>(pc.fft[1]);
  const int K1 = pc.g.K1, K2 = pc.g.K2, H2 = (K2 - 1) / 2, kb = (K1 + L - 1) / L;
  const int i3 = local / kb, kl = (local - i3 * kb) * L + (threadIdx.x & (L - 1));
  const bool kin = kl < K1;
  const cx<double>* src =
      static_cast<const cx<double>*>(pc.A1) + static_cast<size_t>(i3) * n2 * K1 + (kin ? kl : 0);
  cx<double>* dst = static_cast<cx<double>*>(pc.A2) + static_cast<size_t>(i3) * K2 * K1 + kl;
  const typename SH::template At<8> t;
  if (t.i < R1) {
    cx<double> u[R0];
#pragma unroll
    for (int j = 0; j < R0; ++j) u[j] = src[(t.i + j * R1) * K1];
    SH::template first<-1, 8>(t, u, a);
  }
  __syncthreads();
  if (t.i >= R0) return;
  cx<double> v[R1];
  SH::template second<-1, 8>(t, a, tw, v);
#pragma unroll
  for (int j = 0; j < R1; ++j) {
    const int e = t.i + j * R0, k2i = e <= H2 ? e + H2 : e - n2 + H2;
    if (kin && (e <= H2 || e >= n2 - H2)) dst[k2i * K1] = v[j];
  }
}

// z forward, influence weights, z inverse of P and (forces) T3 = 2 pi i k3 P, for
// (k2, 8 values of k1); STRESS as in fft_z_influence_body.
template <class SH, bool STRESS>
__device__ __forceinline__ void z_body(const PassCell& pc, int local, int nz,
                                       double* __restrict__ stress) {
  constexpr int L = SH::L, n3 = SH::length, R0 = SH::radix0, R1 = SH::radix1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cx<double>* a = reinterpret_cast<cx<double>*>(smem_raw);
  cx<double>* q = a + SH::elems(8);  // K3 weighted modes per line
  const cx<double>* tw = plan_twiddles<double>(pc.fft[2]);
  const int K1 = pc.g.K1, K2 = pc.g.K2, K3 = pc.g.K3, kb = (K1 + L - 1) / L;
  const int h1 = K1 - 1, h2 = (K2 - 1) / 2, h3 = (K3 - 1) / 2;
  const int k2i = local / kb, line = threadIdx.x & (L - 1), k1 = (local - k2i * kb) * L + line;
  const int k2 = k2i - h2;
  const bool kin = k1 < K1;
  const size_t zstride = static_cast<size_t>(K2) * K1;
  const size_t at = static_cast<size_t>(k2i) * K1 + (kin ? k1 : 0);
  const typename SH::template At<8> t;
  if (t.i < R1) {
    // Addresses one from the other: as offsets of one pointer they would hold two
    // registers each.
    const cx<double>* src = static_cast<const cx<double>*>(pc.A2) + at + t.i * zstride;
    const size_t step = R1 * zstride;
    cx<double> u[R0];
#pragma unroll
    for (int j = 0; j < R0; ++j, src += step) u[j] = *src;
    SH::template first<-1, 8>(t, u, a);
  }
  __syncthreads();
  if (t.i < R0) {
    cx<double> v[R1];
    SH::template second<-1, 8>(t, a, tw, v);
#pragma unroll
    for (int j = 0; j < R1; ++j) {
      const int e = t.i + j * R0;
      if (e <= h3)
        q[(e + h3) * L + line] = v[j];
      else if (e >= n3 - h3)
        q[(e - n3 + h3) * L + line] = v[j];
    }
  }
  // Influence weights.  Each thread weights the modes that it has put into q itself
  // (no barrier), two at a time: inlined into the transform, one exponential and one
  // division per output cost it 100 registers, and one at a time they are a chain
  // of latencies.
  constexpr double twoPi = 2.0 * 3.14159265358979323846;
  double sv[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  if (t.i < R0) {
    // The mode's share of the weight that does not depend on k3.
    const double inv4a2 = 1.0 / (4.0 * (pc.g.alpha * pc.g.alpha));
    // c(k) = ([k in S] + [-k in S]) / 2, S_d = [M/2 - M, M/2 - 1]: per axis the
    // flags of k_d and -k_d (k_d = -M/2 of an even M lies in S, +M/2 does not).
    const int lo1 = pc.g.M[0] / 2 - pc.g.M[0], hi1 = pc.g.M[0] / 2 - 1;
    const int lo2 = pc.g.M[1] / 2 - pc.g.M[1], hi2 = pc.g.M[1] / 2 - 1;
    const int lo3 = pc.g.M[2] / 2 - pc.g.M[2], hi3 = pc.g.M[2] / 2 - 1;
    const bool in12 = k1 >= lo1 && k1 <= hi1 && k2 >= lo2 && k2 <= hi2;
    const bool im12 = -k1 >= lo1 && -k1 <= hi1 && -k2 >= lo2 && -k2 <= hi2;
    const double w12 = kin ? 2.0 * 3.14159265358979323846 / pc.g.volume * pc.corr2[0][k1 + h1] *
                                 pc.corr2[1][k2i]
                           : 0.0;
    const double* corr3 = pc.corr2[2] + h3;
    double b12[3], b3[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      b12[c] = twoPi * (k1 * pc.g.rec[0][c] + k2 * pc.g.rec[1][c]);
      b3[c] = twoPi * pc.g.rec[2][c];
    }
#pragma unroll 2
    for (int e = t.i; e < n3; e += R0) {
      if (e > h3 && e < n3 - h3) continue;
      const int k3 = e <= h3 ? e : e - n3;
      const double kx = fma(static_cast<double>(k3), b3[0], b12[0]);
      const double ky = fma(static_cast<double>(k3), b3[1], b12[1]);
      const double kz = fma(static_cast<double>(k3), b3[2], b12[2]);
      const double kk2 = kx * kx + ky * ky + kz * kz;
      const double ik2 = 1.0 / kk2;
      const int in3 = (in12 && k3 >= lo3 && k3 <= hi3) + (im12 && -k3 >= lo3 && -k3 <= hi3);
      const bool on = kk2 >= 1.0e-24 && (k1 != 0 || k2 != 0 || k3 != 0) && in3 > 0;
      const double wt = on ? in3 * w12 * exp(-kk2 * inv4a2) * ik2 * corr3[k3] : 0.0;
      cx<double>* m = q + (k3 + h3) * L + line;
      const cx<double> v = *m;
      if constexpr (STRESS) {
        if (on) {
          const double en = (k1 > 0 ? 1.0 : 0.5) * wt * (v.x * v.x + v.y * v.y);
          const double f = 2.0 * (inv4a2 + ik2);
          sv[0] += en * (f * kx * kx - 1.0);
          sv[1] += en * (f * ky * ky - 1.0);
          sv[2] += en * (f * kz * kz - 1.0);
          sv[3] += en * f * kx * ky;
          sv[4] += en * f * kx * kz;
          sv[5] += en * f * ky * kz;
        }
      }
      *m = mk(wt * v.x, wt * v.y);
    }
  }
  __syncthreads();
  if constexpr (STRESS) {  // fixed-order CTA sum: shuffle tree per warp, then warps in order
    __shared__ double sred[32][6];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int lanes = min(32, SH::threads - 32 * warp);  // the last warp may be part of one
    const unsigned live = 0xffffffffu >> (32 - lanes);
#pragma unroll
    for (int j = 0; j < 6; ++j) {
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) {
        const double o = __shfl_xor_sync(live, sv[j], off);
        if ((lane ^ off) < lanes) sv[j] += o;
      }
      if (lane == 0) sred[warp][j] = sv[j];
    }
    __syncthreads();
    if (threadIdx.x < 6) {
      double t = 0.0;
      for (int w = 0; w < (SH::threads + 31) / 32; ++w) t += sred[w][threadIdx.x];
      stress[static_cast<size_t>(local) * 6 + threadIdx.x] = t;
    }
  }
#pragma unroll 1
  for (int c = 0; c < nz; ++c) {
    // An index that the compiler takes for a new one in each round: it would keep
    // the rounds' common factors and twiddles, 50 registers of them, across both.
    typename SH::template At<8> r = t;
    asm volatile("" : "+r"(r.i));
    if (r.i < R1) {
      cx<double> u[R0];
#pragma unroll
      for (int j = 0; j < R0; ++j) {
        const int e = r.i + j * R1, k3 = e <= h3 ? e : e - n3;
        u[j] = mk(0.0, 0.0);
        if (e <= h3 || e >= n3 - h3) {
          u[j] = q[(k3 + h3) * L + line];
          if (c > 0) u[j] = times_i(u[j], twoPi * k3);  // 2 pi i k3 v
        }
      }
      SH::template first<1, 8>(r, u, a);
    }
    __syncthreads();
    if (r.i < R0) {
      cx<double> v[R1];
      SH::template second<1, 8>(r, a, tw, v);
      cx<double>* dst = static_cast<cx<double>*>(pc.B2) + at +
                        (static_cast<size_t>(c) * n3 + r.i) * zstride;
      const size_t step = R0 * zstride;
#pragma unroll
      for (int j = 0; j < R1; ++j, dst += step)
        if (kin) *dst = v[j];
    }
    __syncthreads();
  }
}

// y inverse: the zero-padded k2 box to i2 for (component, i3, 8 values of k1);
// components IFFT_y(P) and, for forces, IFFT_y(2 pi i k2 P), IFFT_y(T3).
template <class SH>
__device__ __forceinline__ void y_inv_body(const PassCell& pc, int local) {
  constexpr int L = SH::L, n2 = SH::length, R0 = SH::radix0, R1 = SH::radix1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cx<double>* a = reinterpret_cast<cx<double>*>(smem_raw);
  const cx<double>* tw = plan_twiddles<double>(pc.fft[1]);
  const int K1 = pc.g.K1, K2 = pc.g.K2, H2 = (K2 - 1) / 2, n3 = pc.g.n[2], kb = (K1 + L - 1) / L;
  const int ci = local / kb, kl = (local - ci * kb) * L + (threadIdx.x & (L - 1));
  const int c = ci / n3, i3 = ci - c * n3;
  const int cs = c == 2 ? 1 : 0;
  const bool dk2 = c == 1, kin = kl < K1;
  const cx<double>* src = static_cast<const cx<double>*>(pc.B2) +
                          ((static_cast<size_t>(cs) * n3 + i3) * K2 + H2) * K1 + (kin ? kl : 0);
  cx<double>* dst =
      static_cast<cx<double>*>(pc.B1) + (static_cast<size_t>(c) * n3 + i3) * n2 * K1 + kl;
  const typename SH::template At<8> t;
  if (t.i < R1) {
    cx<double> u[R0];
#pragma unroll
    for (int j = 0; j < R0; ++j) {
      const int i2 = t.i + j * R1, k2 = i2 <= H2 ? i2 : i2 - n2;
      u[j] = load_if(src + k2 * K1, i2 <= H2 || i2 >= n2 - H2);
    }
    if (dk2) {
#pragma unroll
      for (int j = 0; j < R0; ++j) {
        const int i2 = t.i + j * R1;
        u[j] = times_i(u[j], 2.0 * 3.14159265358979323846 * (i2 <= H2 ? i2 : i2 - n2));
      }
    }
    SH::template first<1, 8>(t, u, a);
  }
  __syncthreads();
  if (t.i >= R0 || !kin) return;
  cx<double> v[R1];
  SH::template second<1, 8>(t, a, tw, v);
#pragma unroll
  for (int j = 0; j < R1; ++j) dst[(t.i + j * R0) * K1] = v[j];
}

// x, complex to real: a line is a row pair's component, the NC components of one
// pair neighbours, so that neighbouring threads write one point's components and
// neighbouring points; outputs phi = C2R(Y0) and, with NC = 4, D1 = C2R(2 pi i k1 Y0),
// C2R(Y2), C2R(Y3), interleaved.
template <class SH, int NC>
__device__ __forceinline__ void x_c2r_body(const PassCell& pc, int bx) {
  constexpr int L = SH::L, n1 = SH::length, NP = L / NC, R0 = SH::radix0, R1 = SH::radix1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cx<double>* a = reinterpret_cast<cx<double>*>(smem_raw);
  const cx<double>* tw = plan_twiddles<double>(pc.fft[0]);
  const int K1 = pc.g.K1, nrows = pc.g.n[1] * pc.g.n[2];
  const typename SH::template At<NC> t;
  const int pr = bx * NP + t.group;
  const bool valid = 2 * pr < nrows && t.group < NP;
  if (t.i < R1 && t.group < NP) {
    const int cs = t.line <= 1 ? 0 : t.line - 1;
    const cx<double>* sa = static_cast<const cx<double>*>(pc.B1) +
                           (static_cast<size_t>(cs) * nrows + (valid ? 2 * pr : 0)) * K1;
    cx<double> u[R0];
    // The rows' two halves of the loads in turn: R0 of them in flight at a time.
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      cx<double> fa[(R0 + 1) / 2], fb[(R0 + 1) / 2];
#pragma unroll
      for (int j = h; j < R0; j += 2) {
        const int x = t.i + j * R1, kx = x < K1 ? x : n1 - x;
        const bool in = x < K1 || x > n1 - K1;
        fa[j / 2] = load_if(sa + kx, in);
        fb[j / 2] = load_if(sa + K1 + kx, in);
      }
#pragma unroll
      for (int j = h; j < R0; j += 2) {
        const int x = t.i + j * R1;
        cx<double> p = fa[j / 2], q = fb[j / 2];
        if (t.line == 1) {
          const double f = 2.0 * 3.14159265358979323846 * (x < K1 ? x : n1 - x);
          p = times_i(p, f);
          q = times_i(q, f);
        }
        // Hermitian continuation; the k1 = 0 modes' imaginary parts drop out.
        const double s = x == 0 ? 0.0 : (x < K1 ? 1.0 : -1.0);
        u[j] = mk(p.x - s * q.y, s * p.y + q.x);
      }
    }
    SH::template first<1, NC>(t, u, a);
  }
  __syncthreads();
  if (t.i >= R0 || !valid) return;
  cx<double> v[R1];
  SH::template second<1, NC>(t, a, tw, v);
  double* oa = static_cast<double*>(pc.out) + (2 * static_cast<size_t>(pr) * n1 + t.i) * NC + t.line;
#pragma unroll
  for (int j = 0; j < R1; ++j) {
    oa[j * R0 * NC] = v[j].x;
    oa[(n1 + j * R0) * NC] = v[j].y;
  }
}

// ---- kernels ----------------------------------------------------------------
// VAR: z, 1 with the stress sums; x C2R, the components.
template <class SH, int PASS, int VAR>
__device__ __forceinline__ void pass64_body(const PassCell& pc, int local, int nz,
                                            double* __restrict__ stress) {
  if constexpr (PASS == P64_R2C) x_r2c_body<SH>(pc, local);
  if constexpr (PASS == P64_YFWD) y_fwd_body<SH>(pc, local);
  if constexpr (PASS == P64_Z) z_body<SH, VAR != 0>(pc, local, nz, stress);
  if constexpr (PASS == P64_YINV) y_inv_body<SH>(pc, local);
  if constexpr (PASS == P64_C2R) x_c2r_body<SH, VAR>(pc, local);
}

// CTAs per SM that the z pass's registers are bounded for (without spills: 92 at radices
// up to 16, 168 above); unbounded it took 144 and 255, 12 and 6 warps an SM.
constexpr int min_blocks64(int pass, int threads) {
  return pass == P64_Z ? (threads <= 128 ? 5 : 2) : 0;
}

template <class SH, int PASS, int VAR>
__global__ void __launch_bounds__(SH::threads, min_blocks64(PASS, SH::threads))
    k64_pass(const __grid_constant__ PassCell pc, int nz, double* __restrict__ stress) {
  chain_enter();
  pass64_body<SH, PASS, VAR>(pc, blockIdx.x, nz, stress);
}

constexpr int pass64_axis(int pass) {
  return pass == P64_R2C || pass == P64_C2R ? 0 : pass == P64_Z ? 2 : 1;
}

// The largest dynamic shared memory of a pass at length n: one transform's buffer and,
// in the z pass, the modes, of which a line has fewer than points (K3 < n).
constexpr int most_smem64(int pass, int n, int elems) {
  return static_cast<int>(sizeof(cx<double>)) * (elems + (pass == P64_Z ? 8 * n : 0));
}

// Launches KERNEL with sm <= MOST bytes of dynamic shared memory.  The limit of a kernel
// is shared by the host threads that use the device, each with its own context: it is
// set once per device, to the most that any launch takes, and never to one launch's
// size, which could fall short of another thread's launch.
template <auto KERNEL, int MOST, class... A>
void go64(const Launch64& l, int threads, size_t sm, const A&... args) {
  if constexpr (MOST > 48 * 1024) {
    static std::atomic<unsigned long long> done{0};  // a bit per device
    int dev = 0;
    cudaGetDevice(&dev);
    const unsigned long long bit = 1ull << (dev & 63);
    if (dev > 63 || !(done.load(std::memory_order_acquire) & bit)) {
      cudaFuncSetAttribute(KERNEL, cudaFuncAttributeMaxDynamicSharedMemorySize, MOST);
      done.fetch_or(bit, std::memory_order_release);
    }
  }
  launch_chained(KERNEL, l.blocks, threads, sm, l.st, args...);
  ++g_launches;
}

// A single cell's pass at the length of SH.
template <class SH, int PASS, int VAR, class... A>
void go64_one(const Launch64& l, const A&... args) {
  constexpr int elems = SH::elems(PASS == P64_R2C || PASS == P64_C2R ? 1 : 8);
  const size_t sm = sizeof(cx<double>) *
                    (elems + (PASS == P64_Z ? SH::L * static_cast<size_t>(l.K3) : 0));
  go64<k64_pass<SH, PASS, VAR>, most_smem64(PASS, SH::length, elems)>(l, SH::threads, sm, args...);
}

template <class SH>
void launch64(const Launch64& l) {
  switch (l.pass) {
    case P64_R2C: go64_one<SH, P64_R2C, 0>(l, *l.one, 1, l.stress); break;
    case P64_YFWD: go64_one<SH, P64_YFWD, 0>(l, *l.one, 1, l.stress); break;
    case P64_Z:
      if (l.stress)
        go64_one<SH, P64_Z, 1>(l, *l.one, l.nz, l.stress);
      else
        go64_one<SH, P64_Z, 0>(l, *l.one, l.nz, l.stress);
      break;
    case P64_YINV: go64_one<SH, P64_YINV, 0>(l, *l.one, 1, l.stress); break;
    default:
      if (l.nc == 4)
        go64_one<SH, P64_C2R, 4>(l, *l.one, 1, l.stress);
      else
        go64_one<SH, P64_C2R, 1>(l, *l.one, 1, l.stress);
  }
}

// The bound of a batch's kernel, which holds the lengths of a class.
constexpr int min_blocks_seg(int pass, int threads) {
  return pass != P64_Z ? 0 : threads <= 64 ? 14 : threads <= 96 ? 8 : threads <= 128 ? 4 : 2;
}

// A batch's pass over the cells whose length lies in SHS (all of one class).
template <int THREADS, int PASS, int VAR, class... SHS>
__global__ void __launch_bounds__(THREADS, min_blocks_seg(PASS, THREADS))
    k64_pass_seg(const BatchCell* __restrict__ cells, PassGroup g, int nz) {
  chain_enter();
  const int m = seg_cell(g.prefix, g.n, blockIdx.x);
  const PassCell& pc = cells[g.cell[m]];
  const int local = static_cast<int>(blockIdx.x) - g.prefix[m];
  const int n = pc.g.n[pass64_axis(PASS)];
  ((n == SHS::length ? pass64_body<SHS, PASS, VAR>(pc, local, nz, nullptr) : void()), ...);
}

// Launches a single cell's pass if length n belongs to source file U.
template <int U, int I>
bool launch64_entry(int n, const Launch64& l) {
  if constexpr (kLengths64[I].unit == U) {
    if (n != kLengths64[I].n) return false;
    launch64<TwoPass<kLengths64[I].n, kLengths64[I].r0, kLengths64[I].r1>>(l);
    return true;
  }
  return false;
}
template <int U, int... I>
bool launch64_unit(int n, const Launch64& l, std::integer_sequence<int, I...>) {
  return (launch64_entry<U, I>(n, l) || ...);
}
template <int U>
bool launch64_unit(int n, const Launch64& l) {
  return launch64_unit<U>(n, l, std::make_integer_sequence<int, kCount64>{});
}

template <class... SHS>
struct Seg64 {
  static constexpr int most(std::initializer_list<int> v) {
    int t = 0;
    for (int x : v) t = x > t ? x : t;
    return t;
  }
  static constexpr int threads = most({SHS::threads...});
  template <int PASS, int VAR>
  static void go(const Launch64& l) {
    constexpr int x = PASS == P64_R2C || PASS == P64_C2R ? 1 : 8;
    constexpr int bound = most({most_smem64(PASS, SHS::length, SHS::elems(x))...});
    size_t sm = sizeof(cx<double>) * most({(SHS::length <= l.nmax ? SHS::elems(x) : 0)...});
    if (PASS == P64_Z) sm += sizeof(cx<double>) * 8 * static_cast<size_t>(l.K3);
    go64<k64_pass_seg<threads, PASS, VAR, SHS...>, bound>(l, threads, sm, l.cells, l.group, l.nz);
  }
  static void launch(const Launch64& l) {
    switch (l.pass) {
      case P64_R2C: go<P64_R2C, 0>(l); break;
      case P64_YFWD: go<P64_YFWD, 0>(l); break;
      case P64_Z: go<P64_Z, 0>(l); break;
      case P64_YINV: go<P64_YINV, 0>(l); break;
      default:
        if (l.nc == 4)
          go<P64_C2R, 4>(l);
        else
          go<P64_C2R, 1>(l);
    }
  }
};

// The lengths of class K as a Seg64.
template <class... SHS>
struct List64 {
  using Seg = Seg64<SHS...>;
};
template <class... A, class... B>
constexpr List64<A..., B...> operator+(List64<A...>, List64<B...>) {
  return {};
}
template <int K, int I>
using Entry64 = std::conditional_t<
    kLengths64[I].klass == K,
    List64<TwoPass<kLengths64[I].n, kLengths64[I].r0, kLengths64[I].r1>>, List64<>>;
template <int K, int... I>
constexpr auto class64(std::integer_sequence<int, I...>) {
  return (List64<>{} + ... + Entry64<K, I>{});
}
template <int K>
using Class64 =
    typename decltype(class64<K>(std::make_integer_sequence<int, kCount64>{}))::Seg;

}  // namespace ewg
