// ewg_fft64.cuh -- the five FP64 transform passes at the lengths of fft64_lengths,
// each a product of two radices of at most 24.
//
// What bounds a pass is the traffic of its grids through L2 and HBM and, before
// that, how many loads an SM has in flight: with three radices of at most 8 a
// line went three times through registers and twice through shared memory, each
// thread with 5 to 8 loads outstanding between barriers.  Here a line goes
// through registers twice: a thread loads R0 elements of its line at once, does
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

#include <initializer_list>

#include "ewg_dft.cuh"
#include "ewg_kernels.h"

namespace ewg {

template <int N, int R0, int R1>
struct TwoPass {
  static_assert(R0 * R1 == N, "radices");
  static constexpr int L = 8;
  static constexpr int length = N;
  static constexpr int radix0 = R0;
  static constexpr int threads = L * (R0 > R1 ? R0 : R1);
  // Shared elements of one transform.
  static constexpr int elems = N * L;

  // ld(e) gives element e of this thread's line, st(e, v) takes element e of the
  // result.  OWN: st writes to `a`, so every thread has read its elements first.
  template <int SIGN, bool OWN, class Ld, class St>
  __device__ __forceinline__ static void run(cx<double>* __restrict__ a,
                                             const cx<double>* __restrict__ tw, Ld ld, St st) {
    const int line = threadIdx.x & (L - 1), i = threadIdx.x / L;
    if (i < R1) {
      cx<double> u[R0];
#pragma unroll
      for (int j = 0; j < R0; ++j) u[j] = ld(i + j * R1);
      dft_reg<double, SIGN, R0>(u);
      cx<double>* dst = a + i * R0 * L + line;
#pragma unroll
      for (int j = 0; j < R0; ++j) dst[j * L] = u[j];
    }
    __syncthreads();
    cx<double> v[R1];
    if (i < R0) {
      const cx<double>* src = a + i * L + line;
#pragma unroll
      for (int j = 0; j < R1; ++j) v[j] = src[j * R0 * L];
      // Twiddles w^(i j), w = exp(SIGN 2 pi i / N): every fourth power from the
      // table, the others one or two products away (a few ulp).
      cx<double> w1 = twiddle(tw, i, SIGN), w2, w3;
      if (R1 > 2) w2 = mul(w1, w1);
      if (R1 > 3) w3 = mul(w2, w1);
      cx<double> base = w1;
#pragma unroll
      for (int j = 1; j < R1; ++j) {
        if (j % 4 == 0) base = twiddle(tw, i * j, SIGN);
        cx<double> w;
        if (j < 4)
          w = j == 1 ? w1 : (j == 2 ? w2 : w3);
        else
          w = j % 4 == 0 ? base : mul(base, j % 4 == 1 ? w1 : (j % 4 == 2 ? w2 : w3));
        v[j] = mul(v[j], w);
      }
      dft_reg<double, SIGN, R1>(v);
    }
    if (OWN) __syncthreads();
    if (i < R0) {
#pragma unroll
      for (int j = 0; j < R1; ++j) st(i + j * R0, v[j]);
    }
  }
};

// x, real to complex: row pairs (2p, 2p+1) form one complex line; k1 = 0..K1-1
// of each row is kept.
template <class SH>
__device__ __forceinline__ void x_r2c_body(const PassCell& pc, int bx) {
  constexpr int L = SH::L, n1 = SH::length;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cx<double>* a = reinterpret_cast<cx<double>*>(smem_raw);
  const cx<double>* tw = plan_twiddles<double>(pc.fft[0]);
  const int K1 = pc.g.K1, npairs = pc.g.n[1] * pc.g.n[2] / 2;
  const int pair0 = bx * L, mine = pair0 + (threadIdx.x & (L - 1));
  const bool valid = mine < npairs;
  const double* ra = static_cast<const double*>(pc.grid) + static_cast<size_t>(2 * (valid ? mine : 0)) * n1;
  auto load = [&](int x) { return mk(ra[x], ra[n1 + x]); };
  auto store = [&](int k, cx<double> v) { a[k * L + (threadIdx.x & (L - 1))] = v; };
  SH::template run<-1, true>(a, tw, load, store);
  __syncthreads();
  // Output k1 fastest: consecutive threads write consecutive k1 of one row pair.
  cx<double>* A1 = static_cast<cx<double>*>(pc.A1);
  for (int t = threadIdx.x; t < L * K1; t += blockDim.x) {
    const int l = t & (L - 1), k = t / L;
    if (pair0 + l >= npairs) continue;
    const cx<double> z = a[k * L + l];
    cx<double> zc = a[(k == 0 ? 0 : n1 - k) * L + l];
    zc.y = -zc.y;
    cx<double>* o = A1 + static_cast<size_t>(2 * (pair0 + l)) * K1 + k;
    o[0] = mk(0.5 * (z.x + zc.x), 0.5 * (z.y + zc.y));
    o[K1] = mk(0.5 * (z.y - zc.y), -0.5 * (z.x - zc.x));
  }
}

// y forward: lines over i2 for (i3, 8 values of k1); keeps k2 in [-H2, H2].
template <class SH>
__device__ __forceinline__ void y_fwd_body(const PassCell& pc, int local) {
  constexpr int L = SH::L, n2 = SH::length;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cx<double>* a = reinterpret_cast<cx<double>*>(smem_raw);
  const cx<double>* tw = plan_twiddles<double>(pc.fft[1]);
  const int K1 = pc.g.K1, K2 = pc.g.K2, H2 = (K2 - 1) / 2, kb = (K1 + L - 1) / L;
  const int i3 = local / kb, kl = (local - i3 * kb) * L + (threadIdx.x & (L - 1));
  const bool kin = kl < K1;
  const cx<double>* src =
      static_cast<const cx<double>*>(pc.A1) + static_cast<size_t>(i3) * n2 * K1 + (kin ? kl : 0);
  cx<double>* dst = static_cast<cx<double>*>(pc.A2) + static_cast<size_t>(i3) * K2 * K1 + kl;
  auto load = [&](int i2) { return src[i2 * K1]; };
  auto store = [&](int e, cx<double> v) {
    const int k2i = e <= H2 ? e + H2 : e - n2 + H2;
    if (kin && (e <= H2 || e >= n2 - H2)) dst[k2i * K1] = v;
  };
  SH::template run<-1, false>(a, tw, load, store);
}

// z forward, influence weights, z inverse of P and (forces) T3 = 2 pi i k3 P, for
// (k2, 8 values of k1); STRESS as in fft_z_influence_body.
template <class SH, bool STRESS>
__device__ __forceinline__ void z_body(const PassCell& pc, int local, int nz,
                                       double* __restrict__ stress) {
  constexpr int L = SH::L, n3 = SH::length;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cx<double>* a = reinterpret_cast<cx<double>*>(smem_raw);
  cx<double>* q = a + SH::elems;  // K3 weighted modes per line
  const cx<double>* tw = plan_twiddles<double>(pc.fft[2]);
  const int K1 = pc.g.K1, K2 = pc.g.K2, K3 = pc.g.K3, kb = (K1 + L - 1) / L;
  const int h1 = K1 - 1, h2 = (K2 - 1) / 2, h3 = (K3 - 1) / 2;
  const int k2i = local / kb, line = threadIdx.x & (L - 1), k1 = (local - k2i * kb) * L + line;
  const int k2 = k2i - h2;
  const bool kin = k1 < K1;
  const size_t zstride = static_cast<size_t>(K2) * K1;
  const size_t at = static_cast<size_t>(k2i) * K1 + (kin ? k1 : 0);
  const cx<double>* src = static_cast<const cx<double>*>(pc.A2) + at;
  auto load_fwd = [&](int i3) { return src[i3 * zstride]; };
  // The mode's share of the weight that does not depend on k3.
  constexpr double twoPi = 2.0 * 3.14159265358979323846;
  const double inv4a2 = 1.0 / (4.0 * (pc.g.alpha * pc.g.alpha));
  // c(k) = ([k in S] + [-k in S]) / 2, S_d = [M/2 - M, M/2 - 1]: per axis the
  // flags of k_d and -k_d (k_d = -M/2 of an even M lies in S, +M/2 does not).
  const int lo1 = pc.g.M[0] / 2 - pc.g.M[0], hi1 = pc.g.M[0] / 2 - 1;
  const int lo2 = pc.g.M[1] / 2 - pc.g.M[1], hi2 = pc.g.M[1] / 2 - 1;
  const int lo3 = pc.g.M[2] / 2 - pc.g.M[2], hi3 = pc.g.M[2] / 2 - 1;
  const int in12 = (k1 >= lo1 && k1 <= hi1 && k2 >= lo2 && k2 <= hi2) ? 1 : 0;
  const int im12 = (-k1 >= lo1 && -k1 <= hi1 && -k2 >= lo2 && -k2 <= hi2) ? 1 : 0;
  const double w12 = kin ? 4.0 * 3.14159265358979323846 / pc.g.volume * pc.corr2[0][k1 + h1] *
                               pc.corr2[1][k2i]
                         : 0.0;
  double b12[3], b3[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    b12[c] = twoPi * (k1 * pc.g.rec[0][c] + k2 * pc.g.rec[1][c]);
    b3[c] = twoPi * pc.g.rec[2][c];
  }
  const double* corr3 = pc.corr2[2];
  double sv[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  auto keep = [&](int e, cx<double> v) {
    if (e <= h3)
      q[(e + h3) * L + line] = v;
    else if (e >= n3 - h3)
      q[(e - n3 + h3) * L + line] = v;
  };
  SH::template run<-1, false>(a, tw, load_fwd, keep);
  // Each thread weights the modes that it has put into q itself (no barrier), in
  // a loop that is not unrolled: inlined into the transform, one exponential and
  // one division per output cost it 100 registers.
  const int i = threadIdx.x / L;
#pragma unroll 1
  for (int e = i; i < SH::radix0 && e < n3; e += SH::radix0) {
    if (e > h3 && e < n3 - h3) continue;
    const int k3 = e <= h3 ? e : e - n3;
    const double kx = fma(static_cast<double>(k3), b3[0], b12[0]);
    const double ky = fma(static_cast<double>(k3), b3[1], b12[1]);
    const double kz = fma(static_cast<double>(k3), b3[2], b12[2]);
    const double kk2 = kx * kx + ky * ky + kz * kz;
    const int in3 = (k3 >= lo3 && k3 <= hi3) ? in12 : 0, im3 = (-k3 >= lo3 && -k3 <= hi3) ? im12 : 0;
    const cx<double> v = q[(k3 + h3) * L + line];
    double wt = 0.0;
    if (kk2 >= 1.0e-24 && in3 + im3 > 0 && !(k1 == 0 && k2 == 0 && k3 == 0)) {
      const double ik2 = 1.0 / kk2;
      wt = 0.5 * (in3 + im3) * w12 * exp(-kk2 * inv4a2) * ik2 * corr3[k3 + h3];
      if constexpr (STRESS) {
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
    q[(k3 + h3) * L + line] = mk(wt * v.x, wt * v.y);
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
  cx<double>* dst = static_cast<cx<double>*>(pc.B2) + at;
  for (int c = 0; c < nz; ++c) {
    auto load_inv = [&](int e) {
      if (e > h3 && e < n3 - h3) return mk(0.0, 0.0);
      const int k3 = e <= h3 ? e : e - n3;
      const cx<double> v = q[(k3 + h3) * L + line];
      if (c == 0) return v;
      const double t = twoPi * k3;
      return mk(-t * v.y, t * v.x);  // 2 pi i k3 v
    };
    auto store = [&](int i3, cx<double> v) {
      if (kin) dst[i3 * zstride] = v;
    };
    SH::template run<1, false>(a, tw, load_inv, store);
    dst += n3 * zstride;
    __syncthreads();
  }
}

// y inverse: the zero-padded k2 box to i2 for (component, i3, 8 values of k1);
// components IFFT_y(P) and, for forces, IFFT_y(2 pi i k2 P), IFFT_y(T3).
template <class SH>
__device__ __forceinline__ void y_inv_body(const PassCell& pc, int local) {
  constexpr int L = SH::L, n2 = SH::length;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cx<double>* a = reinterpret_cast<cx<double>*>(smem_raw);
  const cx<double>* tw = plan_twiddles<double>(pc.fft[1]);
  const int K1 = pc.g.K1, K2 = pc.g.K2, H2 = (K2 - 1) / 2, n3 = pc.g.n[2], kb = (K1 + L - 1) / L;
  const int t = local / kb, kl = (local - t * kb) * L + (threadIdx.x & (L - 1));
  const int c = t / n3, i3 = t - c * n3;
  const int cs = c == 2 ? 1 : 0;
  const bool dk2 = c == 1, kin = kl < K1;
  const cx<double>* src = static_cast<const cx<double>*>(pc.B2) +
                          ((static_cast<size_t>(cs) * n3 + i3) * K2 + H2) * K1 + (kin ? kl : 0);
  cx<double>* dst =
      static_cast<cx<double>*>(pc.B1) + (static_cast<size_t>(c) * n3 + i3) * n2 * K1 + kl;
  auto load = [&](int i2) {
    if (i2 > H2 && i2 < n2 - H2) return mk(0.0, 0.0);
    const int k2 = i2 <= H2 ? i2 : i2 - n2;
    const cx<double> v = src[k2 * K1];
    if (!dk2) return v;
    const double f = 2.0 * 3.14159265358979323846 * k2;
    return mk(-f * v.y, f * v.x);
  };
  auto store = [&](int i2, cx<double> v) {
    if (kin) dst[i2 * K1] = v;
  };
  SH::template run<1, false>(a, tw, load, store);
}

// x, complex to real: the lines of a CTA are (row pair, component), the component
// fastest, so neighbouring threads write one point's components; outputs phi =
// C2R(Y0) and, with NC = 4, D1 = C2R(2 pi i k1 Y0), C2R(Y2), C2R(Y3), interleaved.
template <class SH, int NC>
__device__ __forceinline__ void x_c2r_body(const PassCell& pc, int bx) {
  constexpr int L = SH::L, n1 = SH::length, NP = L / NC;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cx<double>* a = reinterpret_cast<cx<double>*>(smem_raw);
  const cx<double>* tw = plan_twiddles<double>(pc.fft[0]);
  const int K1 = pc.g.K1, nrows = pc.g.n[1] * pc.g.n[2];
  const int line = threadIdx.x & (L - 1), cc = line % NC, pr = bx * NP + line / NC;
  const bool valid = 2 * pr < nrows;
  const int cs = cc <= 1 ? 0 : cc - 1;
  const bool dk1 = cc == 1;
  const cx<double>* sa = static_cast<const cx<double>*>(pc.B1) +
                         (static_cast<size_t>(cs) * nrows + (valid ? 2 * pr : 0)) * K1;
  double* oa = static_cast<double*>(pc.out) + 2 * static_cast<size_t>(pr) * n1 * NC + cc;
  auto load = [&](int x) {
    if (x >= K1 && x <= n1 - K1) return mk(0.0, 0.0);
    const bool lo = x < K1;
    const int kx = lo ? x : n1 - x;
    cx<double> fa = sa[kx], fb = sa[K1 + kx];
    if (dk1) {
      const double t = 2.0 * 3.14159265358979323846 * kx;
      fa = mk(-t * fa.y, t * fa.x);
      fb = mk(-t * fb.y, t * fb.x);
    }
    // Hermitian continuation; the k1 = 0 modes' imaginary parts drop out.
    const double s = x == 0 ? 0.0 : (lo ? 1.0 : -1.0);
    return mk(fa.x - s * fb.y, s * fa.y + fb.x);
  };
  auto store = [&](int x, cx<double> v) {
    if (!valid) return;
    oa[x * NC] = v.x;
    oa[(n1 + x) * NC] = v.y;
  };
  SH::template run<1, false>(a, tw, load, store);
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

template <class SH, int PASS, int VAR>
__global__ void __launch_bounds__(SH::threads) k64_pass(const __grid_constant__ PassCell pc, int nz,
                                                        double* __restrict__ stress) {
  chain_enter();
  pass64_body<SH, PASS, VAR>(pc, blockIdx.x, nz, stress);
}

constexpr int pass64_axis(int pass) {
  return pass == P64_R2C || pass == P64_C2R ? 0 : pass == P64_Z ? 2 : 1;
}

template <class SH, class K, class... A>
void go64(K kernel, const Launch64& l, size_t sm, A... args) {
  if (sm > 48 * 1024)
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(sm));
  launch_chained(kernel, l.blocks, SH::threads, sm, l.st, args...);
  ++g_launches;
}

// A single cell's pass at the length of SH.
template <class SH>
void launch64(const Launch64& l) {
  const size_t sm = sizeof(cx<double>) * SH::elems;
  const size_t smz = sm + sizeof(cx<double>) * SH::L * static_cast<size_t>(l.K3);
  switch (l.pass) {
    case P64_R2C: go64<SH>(k64_pass<SH, P64_R2C, 0>, l, sm, *l.one, 1, l.stress); break;
    case P64_YFWD: go64<SH>(k64_pass<SH, P64_YFWD, 0>, l, sm, *l.one, 1, l.stress); break;
    case P64_Z:
      if (l.stress)
        go64<SH>(k64_pass<SH, P64_Z, 1>, l, smz, *l.one, l.nz, l.stress);
      else
        go64<SH>(k64_pass<SH, P64_Z, 0>, l, smz, *l.one, l.nz, l.stress);
      break;
    case P64_YINV: go64<SH>(k64_pass<SH, P64_YINV, 0>, l, sm, *l.one, 1, l.stress); break;
    default:
      if (l.nc == 4)
        go64<SH>(k64_pass<SH, P64_C2R, 4>, l, sm, *l.one, 1, l.stress);
      else
        go64<SH>(k64_pass<SH, P64_C2R, 1>, l, sm, *l.one, 1, l.stress);
  }
}

// A batch's pass over the cells whose length lies in SHS (all of one class).
template <int THREADS, int PASS, int VAR, class... SHS>
__global__ void __launch_bounds__(THREADS) k64_pass_seg(const BatchCell* __restrict__ cells,
                                                        PassGroup g, int nz) {
  chain_enter();
  const int m = seg_cell(g.prefix, g.n, blockIdx.x);
  const PassCell& pc = cells[g.cell[m]];
  const int local = static_cast<int>(blockIdx.x) - g.prefix[m];
  const int n = pc.g.n[pass64_axis(PASS)];
  ((n == SHS::length ? pass64_body<SHS, PASS, VAR>(pc, local, nz, nullptr) : void()), ...);
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
    size_t sm = sizeof(cx<double>) * 8 * static_cast<size_t>(l.nmax);
    if (PASS == P64_Z) sm += sizeof(cx<double>) * 8 * static_cast<size_t>(l.K3);
    go64<Seg64>(k64_pass_seg<threads, PASS, VAR, SHS...>, l, sm, l.cells, l.group, l.nz);
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

}  // namespace ewg
