// ewg_stencil.cu -- the particle side of the NFFT: window weights, spread and
// gather (nfft/nfft.f90:122-159, :253-278, :380-402).
//
// Tiling.  The fine grid is cut into tiles of 8 x 8 x 8 points.  Along each
// axis an atom's stencil (2m + 1 points with the Gaussian window, 14 with the
// Kaiser-Bessel window; mod n) runs through at most S_d consecutive tiles
// starting at tile f_d; the atom meets every tile of that S_x x S_y x S_z block
// once ("slots").
//
// Weights.  Per atom and axis the window weights are stored already laid out
// per touched tile (S_d * 8 values; zero outside the stencil and beyond the
// grid end; points a wrapping stencil reaches twice carry the sum).  A kernel
// then reads an atom's weights for a tile with no index arithmetic.
//
// Pairs.  Once per geometry, every (atom, tile) pair is binned by tile, and the
// spread puts its tile's bucket in atom order (for the FP32 CUDA-core spread a kernel
// of its own does so), so each tile owns an exact,
// deterministic list of the atoms that reach it.  Where the geometry stays for later
// calls every bucket is also written out in order, whichever spread comes first: a
// later call takes it as it is, with its own choice of spread.
//
// Spread: a CTA owns a tile and writes it once (no atomics, no zeroing, fixed
// order).  Both precision forms contract on the FP64 tensor cores (DMMA); the
// mixed form's FP32 weight rows are widened to FP64 as they are staged and its
// grid is written in FP32.  The FP32 CUDA-core spread (a kernel shape of the
// mixed form) keeps two x-pencils of 8 points per lane in registers and adds
// q w1 w2 w3 atom by atom in list order (groups of 16 atoms in FP32, the group
// sums in FP64).
// Gather: a CTA stages its tile in shared memory and contracts it with the
// weight rows of its atoms on the tensor cores (FP32 tiles widened as they are
// staged), or, on the FP32 CUDA cores, walks the tile's points in lockstep so
// every grid value is a shared-memory broadcast.  Each atom's partial goes to
// its slot for this tile; a final kernel sums each atom's slots in a fixed
// order.  Results are bitwise reproducible.

#include <cuda_runtime.h>

#include <climits>
#include <mutex>
#include <type_traits>
#include <vector>

#include "ewg_kernels.h"

namespace ewg {

namespace {

constexpr int TX = kTileX, TY = kTileY, TZ = kTileZ;
constexpr int kSpreadLanes = TY * TZ / 2;  // FP32 spread: one warp, two x-pencils per lane
constexpr int kSpreadChunk = 64;   // atoms whose weights are staged at once
constexpr int kSpreadGroup = 16;   // FP32 spread: atoms summed in FP32 before the FP64 add
// Gather: atoms per lane and warps sharing one staged tile, per precision.
template <typename R>
struct GatherShape {
  static constexpr int atoms = 2;
  static constexpr int warps = sizeof(R) == 8 ? 1 : 2;
};

__device__ __forceinline__ int pmod(int a, int n) {
  int r = a % n;
  return r < 0 ? r + n : r;
}

// One tile row of eight weights, 16-byte aligned.
__device__ __forceinline__ void store_row(float* out, const float (&v)[8]) {
  reinterpret_cast<float4*>(out)[0] = make_float4(v[0], v[1], v[2], v[3]);
  reinterpret_cast<float4*>(out)[1] = make_float4(v[4], v[5], v[6], v[7]);
}
__device__ __forceinline__ void store_row(double* out, const double (&v)[8]) {
#pragma unroll
  for (int p = 0; p < 8; p += 2)
    reinterpret_cast<double2*>(out)[p / 2] = make_double2(v[p], v[p + 1]);
}

__device__ __forceinline__ int slot_first(int packed) { return packed & 0xffff; }
__device__ __forceinline__ int slot_count(int packed) { return packed >> 16; }

// Mesh stencil origin of a wrapped fractional coordinate: lowest grid point
// floor(s n) (mod n) and the fraction s n - lowest (nfft/nfft.f90:148-152).  A coordinate
// that is not a number, which converts to the lowest int, goes to point 0.
__device__ __forceinline__ int lowest_point(double s, int n, double* frac) {
  const double scaled = s * n;
  const int lowest = static_cast<int>(floor(scaled));
  *frac = scaled - static_cast<double>(lowest);
  return lowest > 0 && lowest < n ? lowest : 0;
}

// Tiles the stencil [c + lo, c + lo + W - 1] (mod n) runs through, starting at
// `first`; a stencil that comes back into its first tile, or covers the whole
// axis, touches every tile once (repeated points are folded into the weights).
__device__ __forceinline__ void stencil_tiles(int c, const StencilDims& sd, int d, int* first,
                                              int* count) {
  const int nd = sd.n[d], nt = sd.ntiles[d];
  if (sd.W >= nd) {
    *first = 0;
    *count = nt;
    return;
  }
  const int p0 = pmod(c + sd.lo, nd);
  int t = p0 / kTileX;
  *first = t;
  int covered = min((t + 1) * kTileX, nd) - p0, m = 1;
  while (covered < sd.W) {
    t = t + 1 == nt ? 0 : t + 1;
    ++m;
    covered += min((t + 1) * kTileX, nd) - t * kTileX;
  }
  *count = min(m, nt);
}

// The Kaiser-Bessel weights of the stencil points as polynomials in t = 2 frac - 1.
constexpr int kKbCoefs = kKbDegree + 1;
__constant__ double c_kb[kKbKinds * kKbWidth * kKbCoefs];

// Point j's weight under the window of kind kb and, with ad, its derivative with
// respect to t.
__device__ __forceinline__ void kb_weight(int kb, int j, double t, int ad, double* v, double* dv) {
  const double* cf = c_kb + ((kb - 1) * kKbWidth + j) * kKbCoefs;
  double w = cf[kKbDegree], dw = 0.0;
#pragma unroll
  for (int e = kKbDegree - 1; e >= 0; --e) {
    if (ad) dw = fma(dw, t, w);
    w = fma(w, t, cf[e]);
  }
  *v = w;
  *dv = dw;
}

// ---------------------------------------------------------------------------
// Tiled window weights of wide windows (rows beyond kAxisRow values per atom),
// one thread per (atom, axis, tile slot), eight points each.  A batch comes here
// when one of its cells is that wide; the others may have the Kaiser-Bessel window.
// ---------------------------------------------------------------------------
// Row r (axis and slot) of sorted atom k.
template <typename R>
__device__ __forceinline__ void weights_row(const double4* __restrict__ s4s, int k, int r,
                                            const StencilDims& sd, R* __restrict__ wtab,
                                            R* __restrict__ qk, int4* __restrict__ slot) {
  const int d = r < sd.S[0] ? 0 : (r < sd.S[0] + sd.S[1] ? 1 : 2);
  const int s = r - (d == 0 ? 0 : (d == 1 ? sd.S[0] : sd.S[0] + sd.S[1]));
  const double4 s4 = s4s[k];
  const int nd = sd.n[d], T = sd.T[d], nt = sd.ntiles[d];
  double frac;
  const int c = lowest_point(d == 0 ? s4.x : (d == 1 ? s4.y : s4.z), nd, &frac);
  const int lo = sd.lo, hi = sd.lo + sd.W - 1, W = sd.W;
  int first, count;
  stencil_tiles(c, sd, d, &first, &count);
  R* out = wtab + static_cast<size_t>(k) * sd.wstride + sd.woff[d] + s * T;
  // Window derivative with respect to the atom's fractional coordinate s_d:
  // the point sits at u = o - frac grid units from the atom, and
  // d/ds_d [pref exp(-u^2 / b)] = n_d (2 u / b) pref exp(-u^2 / b).
  const double dscale = -2.0 * static_cast<double>(nd) / sd.b;
  const int origin = ((first + s) % nt) * T;
  R wv[TX], dv[TX];
  static_assert(TX == TY && TY == TZ, "one row length for all axes");
  if (sd.kb) {  // more points than the window is wide, in whole tiles
    const int o0 = pmod(origin - c, nd);
    for (int p = 0; p < TX; ++p) {
      int o = o0 + p;
      if (o >= nd) o -= nd;
      if (o > hi) o -= nd;  // largest offset <= hi congruent to P - c
      double e = 0.0, de = 0.0;
      if (s < count && o >= lo) kb_weight(sd.kb, o - lo, 2.0 * frac - 1.0, sd.ad, &e, &de);
      wv[p] = static_cast<R>(e);
      dv[p] = static_cast<R>(2.0 * static_cast<double>(nd) * de);  // dt/ds_d = 2 n
    }
  } else if (W < nd) {
    // Every point has at most one image in [lo, hi]: the offsets of the row are
    // consecutive (one wrap at most) and the eight terms are independent.
    const int o0 = pmod(origin - c, nd);
#pragma unroll
    for (int p = 0; p < TX; ++p) {
      int o = o0 + p;
      if (o >= nd) o -= nd;
      if (o > hi) o -= nd;  // largest offset <= hi congruent to P - c
      const bool live = s < count && origin + p < nd && o >= lo;
      const double dd = frac - static_cast<double>(o);
      const double e = sd.pref * exp(-(dd * dd) / sd.b);
      wv[p] = static_cast<R>(live ? e : 0.0);
      dv[p] = static_cast<R>(live ? dscale * dd * e : 0.0);
    }
  } else {
#pragma unroll
    for (int p = 0; p < TX; ++p) {
      const int P = origin + p;
      double w = 0.0, dw = 0.0;
      if (s < count && P < nd) {
        int o = pmod(P - c, nd);  // largest offset <= hi congruent to P - c
        while (o > hi) o -= nd;
        while (o + nd <= hi) o += nd;
        for (; o >= lo; o -= nd) {
          const double dd = frac - static_cast<double>(o);
          const double e = sd.pref * exp(-(dd * dd) / sd.b);
          w += e;
          dw += dscale * dd * e;
        }
      }
      wv[p] = static_cast<R>(w);
      dv[p] = static_cast<R>(dw);
    }
  }
  // Rows start on multiples of eight values: whole 16-byte stores.
  store_row(out, wv);
  if (sd.ad) store_row(out + sd.dwoff, dv);
  if (s != 0) return;  // the axis' first slot thread writes the slot record
  int* sp = reinterpret_cast<int*>(&slot[k]);
  sp[d] = first | (count << 16);
  if (d == 0) {
    sp[3] = 0;
    qk[k] = static_cast<R>(s4.w);
  }
}

template <typename R>
__global__ void k_weights_tiled(const double4* __restrict__ s4s, int n, StencilDims sd,
                                R* __restrict__ wtab, R* __restrict__ qk,
                                int4* __restrict__ slot) {
  chain_enter();
  const int SS = sd.S[0] + sd.S[1] + sd.S[2];
  const long idx = static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (idx >= static_cast<long>(SS) * n) return;
  const int k = static_cast<int>(idx / SS);
  weights_row<R>(s4s, k, static_cast<int>(idx - static_cast<long>(k) * SS), sd, wtab, qk, slot);
}

// Every cell of a batch: item idx is (atom, row) of its cell (prefix over the
// cells' natoms (S_x + S_y + S_z)); the weight rows keep the batch's common
// per-atom stride.
template <typename R>
__global__ void k_weights_seg(const BatchCell* __restrict__ cells, const int* __restrict__ prefix,
                              int ncells, long nitems, const double4* __restrict__ s4s,
                              R* __restrict__ wtab, R* __restrict__ qk, int4* __restrict__ slot) {
  chain_enter();
  const long idx = static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (idx >= nitems) return;
  const int c = seg_cell(prefix, ncells, idx);
  const BatchCell& bc = cells[c];
  const StencilDims sd = bc.sd;
  const int SS = sd.S[0] + sd.S[1] + sd.S[2];
  const int local = static_cast<int>(idx - prefix[c]);
  const int kl = local / SS;
  weights_row<R>(s4s, bc.atom0 + kl, local - kl * SS, sd, wtab, qk, slot);
}

// Slot s of the S_x x S_y x S_z block of an atom with slot record si: its tile
// (the cell's own numbering) and packed slot; false for slots past the atom's own
// tile counts.
__device__ __forceinline__ bool pair_of(const int4& si, int s, const StencilDims& sd, int* tile,
                                        int* packed) {
  const int sx = s % sd.S[0], sy = (s / sd.S[0]) % sd.S[1], sz = s / (sd.S[0] * sd.S[1]);
  if (sx >= slot_count(si.x) || sy >= slot_count(si.y) || sz >= slot_count(si.z)) return false;
  const int tx = (slot_first(si.x) + sx) % sd.ntiles[0];
  const int ty = (slot_first(si.y) + sy) % sd.ntiles[1];
  const int tz = (slot_first(si.z) + sz) % sd.ntiles[2];
  *tile = (tz * sd.ntiles[1] + ty) * sd.ntiles[0] + tx;
  *packed = sx | (sy << 8) | (sz << 16);
  return true;
}

// ---------------------------------------------------------------------------
// Tiled window weights, a warp per axis of 32 atoms, a lane per atom (or of 8 atoms, four
// lanes to each), and the counts of the (atom, tile) pairs.
//
// The lanes evaluate exactly the W points of their stencils: the Kaiser-Bessel
// weights as polynomials in the atom's fraction with the same coefficients for
// every lane, constant operands without a memory access; the Gaussian by its
// exponential.  (One thread per row of 8 points evaluated 24 or 32 points for 13 to
// 25, and neighbouring lanes would gather different polynomials.)  The values go
// to the tiled rows through shared memory, from where the CTA writes the rows of
// its atoms, a contiguous piece of the table, with 16-byte stores; those bound it
// (576 B per atom and 14 points in FP64).  Then the CTA counts its atoms' tiles
// and keeps each pair's arrival number in its tile, which saves a launch and the
// scatter its own round of atomics.
// ---------------------------------------------------------------------------
// Atoms per CTA: 32, or 8 where 32 would leave SMs without a CTA.  Under the Gaussian four
// lanes then share an atom's points: up to 32 atoms per SM the call is shorter (tolerance
// 1e-8, half-width 9, us with 8 for 32: 300 atoms 103 for 119, 1,500 132 for 143, 4,500 196
// for 206; from 9,000 atoms equal, and mixed precision at 32,769 348 for 337).  The
// Kaiser-Bessel window has a lane per atom in both, and gains where each CTA of 8 has its
// own SM (300 atoms 97 for 107, 1,500 122 for 121, 4,096 162 for 157).
constexpr int kAxisMany = 32, kAxisFew = 8;
constexpr int kAxisFewGaussian = 148 * kAxisMany, kAxisFewBessel = 148 * kAxisFew;
constexpr int kAxisRow = 200;     // most values per atom: 52 KB of rows (half-width 12 with
                                  // derivatives and a part tile on an axis has up to 240)

// Shared values per atom: the rows (and, for ad, derivative rows) plus padding
// that spreads the lanes over the banks and keeps rows 16-byte aligned.
__host__ __device__ constexpr int axis_pitch(int row) { return row + 2; }

// The Kaiser-Bessel weights of an axis into the shared row `out` (row0: the first
// point's place in it).  The kind is fixed at compile time for constant operands.
template <int KB>
__device__ __forceinline__ void axis_kaiser_bessel(double frac, int row0, const StencilDims& sd,
                                                   int nd, double* __restrict__ out) {
  const double t = 2.0 * frac - 1.0;
  const double dscale = 2.0 * static_cast<double>(nd);  // dt/ds_d
#pragma unroll
  for (int j = 0; j < kKbWidth; ++j) {
    double v, dv;
    kb_weight(KB, j, t, sd.ad, &v, &dv);
    int r = row0 + j;
    if (r >= nd) r -= nd;  // back in the first tile (nt = 2)
    out[r] = v;
    if (sd.ad) out[sd.dwoff + r] = dscale * dv;
  }
}

// The weights of an atom with fractional coordinate s along axis d into its shared
// row w, zeroed before (with sd.ad the derivatives dwoff further on); returns the
// slot record.  SUB lanes (sub: 0 .. SUB - 1) take the atom's points in turn, with the
// Kaiser-Bessel window and where points are reached twice the first lane all of them.
template <int SUB>
__device__ __forceinline__ int axis_weights(double s, int d, int sub, const StencilDims& sd,
                                            double* __restrict__ w) {
  const int nd = sd.n[d], nt = sd.ntiles[d];
  double frac;
  const int c = lowest_point(s, nd, &frac);
  int first, count;
  stencil_tiles(c, sd, d, &first, &count);
  double* out = w + sd.woff[d];
  if (sd.kb) {  // more points than the window is wide, in whole tiles
    int p0 = c + kKbLow;
    if (p0 < 0) p0 += nd;
    const int row0 = p0 - first * kTileX;
    static_assert(kKbKinds == 2, "a call per kind");
    if (sub > 0) return first | (count << 16);
    if (sd.kb == 1)
      axis_kaiser_bessel<1>(frac, row0, sd, nd, out);
    else
      axis_kaiser_bessel<2>(frac, row0, sd, nd, out);
  } else {
    // d/ds_d [pref exp(-u^2 / b)] = n_d (2 u / b) pref exp(-u^2 / b) at u = o - frac.
    const double dscale = -2.0 * static_cast<double>(nd) / sd.b;
    const bool alone = SUB == 1 || sd.W > nd;  // a lane for all points
    if (alone && sub > 0) return first | (count << 16);
    const int step = alone ? 1 : SUB;
    int o = sd.lo + sd.W - 1 - sub;
    int p = pmod(c + o, nd);
    for (; o >= sd.lo; o -= step) {
      const double dd = frac - static_cast<double>(o);
      const double e = sd.pref * exp(-(dd * dd) / sd.b);
      const int t = p / kTileX;
      int sl = t - first;
      if (sl < 0) sl += nt;
      const int r = sl * kTileX + (p - t * kTileX);
      out[r] += e;  // a point that the stencil reaches again carries the sum
      if (sd.ad) out[sd.dwoff + r] += dscale * dd * e;
      p = p < step ? p - step + nd : p - step;  // a next point has step < W <= nd, or step 1
    }
  }
  return first | (count << 16);
}

// Row values as the table's type, 16 bytes at a time (rows are multiples of 8 values).
__device__ __forceinline__ void copy_row(double* __restrict__ dst, const double* __restrict__ src,
                                         int v) {
  *reinterpret_cast<double2*>(dst + v) = *reinterpret_cast<const double2*>(src + v);
}
__device__ __forceinline__ void copy_row(float* __restrict__ dst, const double* __restrict__ src,
                                         int v) {
  *reinterpret_cast<float4*>(dst + v) =
      make_float4(static_cast<float>(src[v]), static_cast<float>(src[v + 1]),
                  static_cast<float>(src[v + 2]), static_cast<float>(src[v + 3]));
}

// dims(k): the stencil geometry of atom k; pairs0(k): the atom's first place in
// arrival; tile0(k): its cell's first tile.
template <typename R, int ATOMS, class Dims, class Pairs0, class Tile0>
__device__ __forceinline__ void weights_axis_body(double* __restrict__ sm, int row, int wstride,
                                                  int pstride, const double4* __restrict__ s4s,
                                                  int n, R* __restrict__ wtab,
                                                  R* __restrict__ qk, int4* __restrict__ slot,
                                                  int* __restrict__ tile_counts,
                                                  int* __restrict__ arrival, Dims dims,
                                                  Pairs0 pairs0, Tile0 tile0) {
  __shared__ int sslot[3][ATOMS];
  constexpr int SUB = 32 / ATOMS;
  const int atom = threadIdx.x % ATOMS, sub = threadIdx.x % 32 / ATOMS, d = threadIdx.x >> 5;
  const int k0 = blockIdx.x * ATOMS, na = min(ATOMS, n - k0);
  const int pitch = axis_pitch(row);
  for (int e = threadIdx.x; e < ATOMS * pitch; e += 96) sm[e] = 0.0;
  __syncthreads();
  if (atom < na) {
    const double4 s4 = s4s[k0 + atom];
    const int record = axis_weights<SUB>(d == 0 ? s4.x : (d == 1 ? s4.y : s4.z), d, sub,
                                         dims(k0 + atom), sm + atom * pitch);
    if (sub == 0) {
      sslot[d][atom] = record;
      if (d == 0) qk[k0 + atom] = static_cast<R>(s4.w);
    }
  }
  __syncthreads();
  constexpr int kVec = 16 / sizeof(R);
  const int chunks = row / kVec;
  for (int e = threadIdx.x; e < na * chunks; e += 96) {
    const int a = e / chunks, v = kVec * (e - a * chunks);
    copy_row(wtab + static_cast<size_t>(k0 + a) * wstride, sm + a * pitch, v);
  }
  if (threadIdx.x < na)
    slot[k0 + threadIdx.x] =
        make_int4(sslot[0][threadIdx.x], sslot[1][threadIdx.x], sslot[2][threadIdx.x], 0);
  for (int e = threadIdx.x; e < na * pstride; e += 96) {
    const int a = e / pstride, k = k0 + a, s = e - a * pstride;
    const StencilDims& sd = dims(k);
    if (s >= sd.S[0] * sd.S[1] * sd.S[2]) continue;
    int tile, packed;
    if (pair_of(make_int4(sslot[0][a], sslot[1][a], sslot[2][a], 0), s, sd, &tile, &packed))
      arrival[pairs0(k) + s] = atomicAdd(&tile_counts[tile0(k) + tile], 1);
  }
}

template <typename R, int ATOMS>
__global__ void __launch_bounds__(96) k_weights_axis(const double4* __restrict__ s4s, int n,
                                                     const __grid_constant__ StencilDims sd,
                                                     R* __restrict__ wtab,
                                                     R* __restrict__ qk, int4* __restrict__ slot,
                                                     int* __restrict__ tile_counts,
                                                     int* __restrict__ arrival) {
  chain_enter();
  extern __shared__ __align__(16) double sm_rows[];
  const int S = sd.S[0] * sd.S[1] * sd.S[2];
  const StencilDims* dims = &sd;  // the parameter itself, no copy per thread
  weights_axis_body<R, ATOMS>(
      sm_rows, sd.wstride, sd.wstride, S, s4s, n, wtab, qk, slot, tile_counts, arrival,
      [dims](int) -> const StencilDims& { return *dims; },
      [S](int k) { return static_cast<size_t>(k) * S; }, [](int) { return 0; });
}

// Every cell of a batch (atom_prefix: first atom of each cell, slot_prefix: first
// (atom, slot) item).
template <typename R, int ATOMS>
__global__ void __launch_bounds__(96) k_weights_axis_seg(
    const BatchCell* __restrict__ cells, const int* __restrict__ atom_prefix,
    const int* __restrict__ slot_prefix, int ncells, int n, int wstride, int pstride,
    const double4* __restrict__ s4s, R* __restrict__ wtab, R* __restrict__ qk,
    int4* __restrict__ slot, int* __restrict__ tile_counts, int* __restrict__ arrival) {
  chain_enter();
  extern __shared__ __align__(16) double sm_rows[];
  __shared__ int cid[ATOMS];
  const int k0 = blockIdx.x * ATOMS;
  if (threadIdx.x < ATOMS)
    cid[threadIdx.x] = seg_cell(atom_prefix, ncells, min(k0 + static_cast<int>(threadIdx.x), n - 1));
  __syncthreads();
  weights_axis_body<R, ATOMS>(
      sm_rows, wstride, wstride, pstride, s4s, n, wtab, qk, slot, tile_counts, arrival,
      [&](int k) -> const StencilDims& { return cells[cid[k - k0]].sd; },
      [&](int k) {
        const int c = cid[k - k0];
        const StencilDims& sd = cells[c].sd;
        return slot_prefix[c] + static_cast<size_t>(k - cells[c].atom0) * sd.S[0] * sd.S[1] * sd.S[2];
      },
      [&](int k) { return cells[cid[k - k0]].tile0; });
}

// ---------------------------------------------------------------------------
// (atom, tile) pair binning: counts (with arrival numbers), scan, scatter, and the
// order of each tile's list by atom, which the tensor-core spread makes itself (the
// gathers do not depend on it).
// ---------------------------------------------------------------------------
// Item idx of a batch's (atom, slot) launch: its cell, sorted atom, tile
// (global numbering: the cell's tile0 added) and packed slot.
__device__ __forceinline__ bool pair_of_seg(const BatchCell* __restrict__ cells,
                                            const int* __restrict__ prefix, int ncells, long idx,
                                            const int4* __restrict__ slot, int* tile, int* k,
                                            int* packed) {
  const int c = seg_cell(prefix, ncells, idx);
  const BatchCell& bc = cells[c];
  const int S = bc.sd.S[0] * bc.sd.S[1] * bc.sd.S[2];
  const int local = static_cast<int>(idx - prefix[c]);
  const int kl = local / S;
  *k = bc.atom0 + kl;
  const StencilDims sd = bc.sd;
  if (!pair_of(slot[*k], local - kl * S, sd, tile, packed)) return false;
  *tile += bc.tile0;
  return true;
}

__global__ void k_pair_count_seg(const BatchCell* __restrict__ cells,
                                 const int* __restrict__ prefix, int ncells, long nitems,
                                 const int4* __restrict__ slot, int* __restrict__ counts,
                                 int* __restrict__ arrival) {
  const long idx = static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x;
  int tile, k, packed;
  if (idx < nitems && pair_of_seg(cells, prefix, ncells, idx, slot, &tile, &k, &packed))
    arrival[idx] = atomicAdd(&counts[tile], 1);
}

__global__ void k_pair_scatter_seg(const BatchCell* __restrict__ cells,
                                   const int* __restrict__ prefix, int ncells, long nitems,
                                   const int4* __restrict__ slot, const int* __restrict__ starts,
                                   const int* __restrict__ arrival, int2* __restrict__ tmp) {
  chain_enter();
  const long idx = static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x;
  int tile, k, packed;
  if (idx < nitems && pair_of_seg(cells, prefix, ncells, idx, slot, &tile, &k, &packed))
    tmp[starts[tile] + arrival[idx]] = make_int2(k, packed);
}

__device__ __forceinline__ bool pair_of_thread(const int4* __restrict__ slot, int n,
                                               const StencilDims& sd, int* tile, int* k,
                                               int* packed) {
  const int S = sd.S[0] * sd.S[1] * sd.S[2];
  const long t = static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (t >= static_cast<long>(n) * S) return false;
  *k = static_cast<int>(t / S);
  const int s = static_cast<int>(t - static_cast<long>(*k) * S);
  return pair_of(slot[*k], s, sd, tile, packed);
}

__global__ void k_pair_count(const int4* __restrict__ slot, int n, StencilDims sd,
                             int* __restrict__ counts, int* __restrict__ arrival) {
  int tile, k, packed;
  if (pair_of_thread(slot, n, sd, &tile, &k, &packed))
    arrival[static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x] = atomicAdd(&counts[tile], 1);
}

__global__ void k_pair_scatter(const int4* __restrict__ slot, int n, StencilDims sd,
                               const int* __restrict__ starts, const int* __restrict__ arrival,
                               int2* __restrict__ tmp) {
  chain_enter();
  int tile, k, packed;
  if (pair_of_thread(slot, n, sd, &tile, &k, &packed))
    tmp[starts[tile] + arrival[static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x]] =
        make_int2(k, packed);
}

// For the FP32 CUDA-core spread, one thread per entry: orders each tile's bucket by
// atom index (atoms are unique within a bucket) by counting the bucket's entries with
// a smaller atom.  The entry's tile follows from its atom's slot record and its packed slot.
__global__ void k_pair_rank(const int2* __restrict__ tmp, const int* __restrict__ starts,
                            int ntiles, const int4* __restrict__ slot, StencilDims sd,
                            int2* __restrict__ pairs) {
  chain_enter();
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= starts[ntiles]) return;
  const int2 v = tmp[e];
  const int4 si = slot[v.x];
  const int tx = (slot_first(si.x) + (v.y & 0xff)) % sd.ntiles[0];
  const int ty = (slot_first(si.y) + ((v.y >> 8) & 0xff)) % sd.ntiles[1];
  const int tz = (slot_first(si.z) + (v.y >> 16)) % sd.ntiles[2];
  const int tile = (tz * sd.ntiles[1] + ty) * sd.ntiles[0] + tx;
  const int b = starts[tile], end = starts[tile + 1];
  int r = 0;
  for (int j = b; j < end; ++j) r += tmp[j].x < v.x;
  pairs[b + r] = v;
}

// Eight consecutive FP32 weights (32 B; every per-tile weight row starts on
// such a boundary) with vector loads.
__device__ __forceinline__ void load8(const float* __restrict__ p, float* out) {
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const float4 v = reinterpret_cast<const float4*>(p)[i];
    out[4 * i] = v.x;
    out[4 * i + 1] = v.y;
    out[4 * i + 2] = v.z;
    out[4 * i + 3] = v.w;
  }
}

// ---------------------------------------------------------------------------
// Spread
// ---------------------------------------------------------------------------
// FP32 form: one warp per tile; each lane owns two x-pencils, (py, pz) and
// (py + 4, pz), so every pair of shared-memory reads of an atom's x weights
// feeds 16 multiply-adds.
template <typename R>
__device__ __forceinline__ void spread_tiles_body(int tx, int ty, int tz,
                                                  const int* __restrict__ tile_start,
                                                               const int2* __restrict__ pairs,
                                                               const R* __restrict__ wtab,
                                                               const R* __restrict__ qk,
                                                               StencilDims sd, R* __restrict__ grid) {
  chain_enter();
  __shared__ R sW1[kSpreadChunk][TX];
  __shared__ R sW2[kSpreadChunk][TY];
  __shared__ R sW3[kSpreadChunk][TZ];
  const int tile = (tz * sd.ntiles[1] + ty) * sd.ntiles[0] + tx;
  const int x0 = tx * TX, y0 = ty * TY, z0 = tz * TZ;
  const int py = threadIdx.x % (TY / 2), pz = threadIdx.x / (TY / 2);
  double acc[2][TX];
#pragma unroll
  for (int x = 0; x < TX; ++x) acc[0][x] = acc[1][x] = 0.0;
  const int p0 = tile_start[tile], p1 = tile_start[tile + 1];
  for (int b0 = p0; b0 < p1; b0 += kSpreadChunk) {
    const int nb = min(kSpreadChunk, p1 - b0);
    __syncthreads();  // the previous chunk's weights are no longer read
    // Each lane stages whole atoms of the chunk: its pair, charge and the
    // 3 x 8 weights for this tile, in independent vector loads.
    for (int a = threadIdx.x; a < nb; a += kSpreadLanes) {
      const int2 pr = pairs[b0 + a];
      const R* wk = wtab + static_cast<size_t>(pr.x) * sd.wstride;
      R t1[TX], t2[TY], t3[TZ];
      load8(wk + sd.woff[0] + (pr.y & 0xff) * TX, t1);
      load8(wk + sd.woff[1] + ((pr.y >> 8) & 0xff) * TY, t2);
      load8(wk + sd.woff[2] + (pr.y >> 16) * TZ, t3);
      const R qa = qk[pr.x];
#pragma unroll
      for (int x = 0; x < TX; ++x) sW1[a][x] = t1[x];
#pragma unroll
      for (int y = 0; y < TY; ++y) sW2[a][y] = t2[y];
#pragma unroll
      for (int z = 0; z < TZ; ++z) sW3[a][z] = t3[z] * qa;
    }
    __syncthreads();
    // Groups of kSpreadGroup atoms are summed in R, each group sum then
    // added to the FP64 pencil: one FP32 -> FP64 conversion per point and
    // group instead of per point and atom (the conversions, not the
    // multiply-adds, bounded the FP32 form).
    for (int g0 = 0; g0 < nb; g0 += kSpreadGroup) {
      const int g1 = min(g0 + kSpreadGroup, nb);
      R part[2][TX];
#pragma unroll
      for (int x = 0; x < TX; ++x) part[0][x] = part[1][x] = R(0);
      for (int a = g0; a < g1; ++a) {
        const R w3 = sW3[a][pz];
        const R s0 = sW2[a][py] * w3, s1 = sW2[a][py + TY / 2] * w3;
#pragma unroll
        for (int x = 0; x < TX; ++x) {
          const R w1 = sW1[a][x];
          part[0][x] = fma(s0, w1, part[0][x]);
          part[1][x] = fma(s1, w1, part[1][x]);
        }
      }
#pragma unroll
      for (int x = 0; x < TX; ++x) {
        acc[0][x] += static_cast<double>(part[0][x]);
        acc[1][x] += static_cast<double>(part[1][x]);
      }
    }
  }
  const int ex = min(TX, sd.n[0] - x0), ey = min(TY, sd.n[1] - y0), ez = min(TZ, sd.n[2] - z0);
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int y = py + h * (TY / 2);
    if (y < ey && pz < ez) {
      R* row = grid + (static_cast<size_t>(z0 + pz) * sd.n[1] + y0 + y) * sd.n[0] + x0;
#pragma unroll
      for (int x = 0; x < TX; ++x)
        if (x < ex) row[x] = static_cast<R>(acc[h][x]);
    }
  }
}

// ---------------------------------------------------------------------------
// FP64 spread on the tensor cores.  For each z-plane of the tile the spread is
// a sum of rank-one products, G_z[y][x] = sum_a (q_a w3_a(z) w2_a(y)) w1_a(x),
// i.e. the 8 x 8 matrix product U_z W1 with U_z[y][a] = q_a w3_a(z) w2_a(y) and
// W1[a][x] = w1_a(x).  A CTA owns a tile and accumulates its eight planes
// with DMMA (mma.sync m8n8k4, FP64 in and out, IEEE fused multiply-adds), four
// atoms per step, in list order: deterministic, no atomics.
// Fragment layouts (m8n8k4, .row.col): A[y][k] at lane 4y + k, B[k][x] at lane
// 4x + k, C[y][x] at lane 4y + x/2 (element x mod 2).
// ---------------------------------------------------------------------------
__device__ __forceinline__ void dmma_m8n8k4(double& c0, double& c1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
               : "+d"(c0), "+d"(c1)
               : "d"(a), "d"(b));
}

constexpr int kGatherWarps = 4;   // tensor-core i k gather: warps per tile (batch, short lists)
constexpr int kGatherMB = 2;      // tensor-core i k gather: M blocks of 8 atoms per warp and round
constexpr int kGatherAdWarps = 2;  // tensor-core gather with window derivatives: warps per tile
// FP32 CUDA-core gather with window derivatives: one atom per lane (74 registers, so
// about 13 CTAs per SM) and two warps per tile.
constexpr int kGatherAdF32Atoms = 1, kGatherAdF32Warps = 2;
// Tensor-core spread: atoms staged per round.  With 16 the rows take half the shared
// memory and 28 instead of 20 warps fit an SM (216,000 sites 237 -> 217 us, a batch
// of 128 cells 129 -> 112); where the tiles do not fill the SMs anyway, 32 take fewer
// rounds (729 tiles 15.1 -> 13.8 us).
constexpr int kSpreadFew = 16, kSpreadMany = 32, kSpreadFull = 148 * 20;
constexpr int kSpreadList = 128;  // longest tile list that the spread orders in shared memory
constexpr int kWRow = 12;         // doubles per staged weight row: 8 used; the
                                  // padding makes the fragment reads conflict-free

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
}

// Two consecutive elements from global into shared memory as doubles: a
// 16-byte cp.async for FP64 data; for the mixed form's FP32 tiles and weight
// rows an 8-byte load widened to FP64, so the same DMMA code contracts them.
__device__ __forceinline__ void stage2(double* dst, const double* src) { cp_async16(dst, src); }
__device__ __forceinline__ void stage2(double* dst, const float* src) {
  const float2 v = __ldg(reinterpret_cast<const float2*>(src));
  dst[0] = v.x;
  dst[1] = v.y;
}

// Puts the list [p0, p1) into pairs in order of its atoms (unique within a tile), a warp
// to a list: the atoms of a window of kOrderWindow consecutive indices are marked in a
// bitmap, an entry's place is the number of marks below its own, and the next window
// starts at the smallest atom left, so a list takes two passes for each window that
// holds some of it, whatever its length.  (Counting the smaller entries of every entry
// costs the square of the length: with 5,000 charges in a ball of 0.02 of their cell,
// lists of some thousand, the spread took 2.2 ms that way and 0.16 so, in the mixed
// form 14.8 and 0.41.  A launch of its own with a thread per entry took 147 us with the
// spread at 32,769 atoms of the mixed form and lists of 500, this 93.)
constexpr int kOrderWords = 512, kOrderWindow = 32 * kOrderWords;
constexpr int kOrderInts = 2 * (kOrderWords + kOrderWords / 16);  // scratch
__device__ __forceinline__ void order_list(const int2* __restrict__ unordered, int2* pairs, int p0,
                                           int p1, int* scratch) {
  const int lane = threadIdx.x & 31;
  // Word w of the bitmap and the place of its first mark, at w + w / 16: a lane sums 16
  // consecutive words without bank conflicts.
  unsigned* bits = reinterpret_cast<unsigned*>(scratch);
  int* first = scratch + kOrderInts / 2;
  int lo = INT_MAX;
#pragma unroll 4
  for (int e = p0 + lane; e < p1; e += 32) lo = min(lo, unordered[e].x);
  lo = __reduce_min_sync(0xffffffffu, lo);
  int placed = p0;
  while (lo != INT_MAX) {  // each window starts at an atom past the last one's end
    for (int w = lane; w < kOrderInts / 2; w += 32) bits[w] = 0;
    __syncwarp();
    int next = INT_MAX;
#pragma unroll 4
    for (int e = p0 + lane; e < p1; e += 32) {
      const int id = unordered[e].x, r = id - lo;
      if (r >= 0 && r < kOrderWindow)
        atomicOr(&bits[(r >> 5) + (r >> 9)], 1u << (r & 31));
      else if (r > 0)
        next = min(next, id);
    }
    __syncwarp();
    int sum = 0;
#pragma unroll
    for (int j = 0; j < 16; ++j) sum += __popc(bits[17 * lane + j]);
    int x = sum;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, off);
      if (lane >= off) x += y;
    }
    int run = placed + x - sum;
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      first[17 * lane + j] = run;
      run += __popc(bits[17 * lane + j]);
    }
    __syncwarp();
#pragma unroll 4
    for (int e = p0 + lane; e < p1; e += 32) {
      const int2 v = unordered[e];
      const int r = v.x - lo;
      if (r >= 0 && r < kOrderWindow) {
        const int w = (r >> 5) + (r >> 9);
        pairs[first[w] + __popc(bits[w] & ((1u << (r & 31)) - 1u))] = v;
      }
    }
    placed += __shfl_sync(0xffffffffu, x, 31);
    lo = __reduce_min_sync(0xffffffffu, next);
    __syncwarp();
  }
}

// One warp per tile owning all eight z-planes, so each step's x and y weights
// are read from shared memory once for the eight planes.  Bound by the latency of
// staging the weight rows, so the warps that fit an SM and the sectors per access
// count: a row of 64 bytes is copied by four lanes (whole sectors; one lane a row
// took 55.6 us at 32,769 atoms and 281 at 216,000 sites, this 43.7 and 203), and
// the entries of a round are read before its first copy, which the compiler moves
// no load across.
//
// unordered: the tile lists in no fixed order, or null when pairs holds them in order;
// keep: the ordered lists go to pairs, all of them (else only the long ones do).
template <typename R, int ATOMS>
__device__ __forceinline__ void spread_tiles_dmma_body(int tx, int ty, int tz,
                                                       const int* __restrict__ tile_start,
                                                       const int2* __restrict__ unordered,
                                                       int2* pairs, bool keep,
                                                       const R* __restrict__ wtab,
                                                       const R* __restrict__ qk,
                                                       const StencilDims& sd,
                                                       R* __restrict__ grid) {
  chain_enter();
  __shared__ __align__(16) double sW[3][ATOMS][kWRow];
  __shared__ double sQ[ATOMS];
  const int tile = (tz * sd.ntiles[1] + ty) * sd.ntiles[0] + tx;
  const int x0 = tx * TX, y0 = ty * TY, z0 = tz * TZ;
  const int lane = threadIdx.x;
  const int fr = lane >> 2, fk = lane & 3;  // fragment row (y, or x for B) and k
  double acc[TZ][2];
#pragma unroll
  for (int z = 0; z < TZ; ++z) acc[z][0] = acc[z][1] = 0.0;
  const int p0 = tile_start[tile], p1 = tile_start[tile + 1];
  // The list in order of its atoms (unique within a tile): an entry's place is the
  // number of entries with a smaller atom.  The lists hold some 40 entries, counted
  // by a lane each in shared memory, four atoms to a load: less work than a launch
  // of its own and than the list's way through global memory.
  __shared__ int2 sList[kSpreadList];
  const bool in_shared = unordered && p1 - p0 <= kSpreadList;
  if (in_shared) {
    const int m = p1 - p0;
    int* ids = reinterpret_cast<int*>(&sW[0][0][0]);
    int2 v[kSpreadList / 32];
#pragma unroll
    for (int h = 0; h < kSpreadList / 32; ++h) {
      const int e = h * 32 + lane;
      v[h] = e < m ? unordered[p0 + e] : make_int2(INT_MAX, 0);
      ids[e] = v[h].x;
    }
    __syncwarp();
    int place[kSpreadList / 32] = {0};
    for (int j = 0; j < m; j += 4) {
      const int4 x = *reinterpret_cast<const int4*>(ids + j);
#pragma unroll
      for (int h = 0; h < kSpreadList / 32; ++h)
        place[h] += (x.x < v[h].x) + (x.y < v[h].x) + (x.z < v[h].x) + (x.w < v[h].x);
    }
#pragma unroll
    for (int h = 0; h < kSpreadList / 32; ++h)
      if (h * 32 + lane < m) {
        sList[place[h]] = v[h];
        if (keep) pairs[p0 + place[h]] = v[h];
      }
    __syncwarp();
  } else if (unordered) {  // a long list goes through its ordered copy
    static_assert(sizeof(sW) >= kOrderInts * sizeof(int), "scratch");
    order_list(unordered, pairs, p0, p1, reinterpret_cast<int*>(&sW[0][0][0]));
  }
  for (int b0 = p0; b0 < p1; b0 += ATOMS) {
    const int nb = min(ATOMS, p1 - b0);
    __syncwarp();  // the previous round's weights are no longer read
    // Four lanes per weight row of 64 bytes, whole sectors to an access; all entries
    // before the first copy, which the compiler does not move loads across.
    int2 pr[ATOMS / 8];
    R q[ATOMS / 8];
#pragma unroll
    for (int h = 0; h < ATOMS / 8; ++h) {
      const int a = h * 8 + fr;
      pr[h] = a >= nb ? make_int2(0, 0) : (in_shared ? sList[b0 - p0 + a] : pairs[b0 + a]);
    }
#pragma unroll
    for (int h = 0; h < ATOMS / 8; ++h) q[h] = fk == 0 && h * 8 + fr < nb ? qk[pr[h].x] : R(0);
#pragma unroll
    for (int h = 0; h < ATOMS / 8; ++h) {
      const int a = h * 8 + fr;
      if (a < nb) {
        const R* wk = wtab + static_cast<size_t>(pr[h].x) * sd.wstride + 2 * fk;
        stage2(&sW[0][a][2 * fk], wk + sd.woff[0] + (pr[h].y & 0xff) * TX);
        stage2(&sW[1][a][2 * fk], wk + sd.woff[1] + ((pr[h].y >> 8) & 0xff) * TY);
        stage2(&sW[2][a][2 * fk], wk + sd.woff[2] + (pr[h].y >> 16) * TZ);
      } else if (a < ((nb + 3) & ~3)) {  // padding atoms of the last group of four
#pragma unroll
        for (int d = 0; d < 3; ++d) sW[d][a][2 * fk] = sW[d][a][2 * fk + 1] = 0.0;
      }
      if (fk == 0) sQ[a] = q[h];
    }
    cp_async_wait_all();
    __syncwarp();
    for (int k0 = 0; k0 < nb; k0 += 4) {
      const int aa = k0 + fk;
      const double bw = sW[0][aa][fr];            // B[k][x = fr]
      const double w2q = sW[1][aa][fr] * sQ[aa];  // A[y = fr][k] = q w2(y) w3(z)
#pragma unroll
      for (int z = 0; z < TZ; ++z) dmma_m8n8k4(acc[z][0], acc[z][1], w2q * sW[2][aa][z], bw);
    }
  }
  const int ex = min(TX, sd.n[0] - x0), ey = min(TY, sd.n[1] - y0), ez = min(TZ, sd.n[2] - z0);
  const int y = fr, x = 2 * fk;
  if (y < ey) {
#pragma unroll
    for (int z = 0; z < TZ; ++z) {
      if (z >= ez) break;
      R* row = grid + (static_cast<size_t>(z0 + z) * sd.n[1] + y0 + y) * sd.n[0] + x0 + x;
      if (x + 1 < ex) {
        row[0] = static_cast<R>(acc[z][0]);
        row[1] = static_cast<R>(acc[z][1]);
      } else if (x < ex) {
        row[0] = static_cast<R>(acc[z][0]);
      }
    }
  }
}

// ---------------------------------------------------------------------------
// Gather.  One warp per CTA; each lane carries A atoms of the tile's list, so
// every grid value read from shared memory (a broadcast: all lanes read the
// same point) feeds A atoms.
// ---------------------------------------------------------------------------
template <typename R, int NC, int A, int WARPS>
__device__ __forceinline__ void gather_tiles_body(int tx, int ty, int tz,
                                                  const int* __restrict__ tile_start,
                                                             const int2* __restrict__ pairs,
                                                             const R* __restrict__ wtab,
                                                             StencilDims sd,
                                                             const R* __restrict__ grid,
                                                             double* __restrict__ part) {
  chain_enter();
  using V = typename std::conditional<
      NC == 4, typename std::conditional<sizeof(R) == 8, double4, float4>::type, R>::type;
  __shared__ V sG[TZ * TY * TX];
  __shared__ R sW3[WARPS][TZ][32 * A];  // z weights, lane fastest
  const int tile = (tz * sd.ntiles[1] + ty) * sd.ntiles[0] + tx;
  const int x0 = tx * TX, y0 = ty * TY, z0 = tz * TZ;
  const int ex = min(TX, sd.n[0] - x0), ey = min(TY, sd.n[1] - y0), ez = min(TZ, sd.n[2] - z0);
  const int p0 = tile_start[tile], p1 = tile_start[tile + 1];
  if (p0 == p1) return;  // no atom reaches this tile
#pragma unroll 4
  for (int t = threadIdx.x; t < TX * TY * TZ; t += 32 * WARPS) {
    const int x = t % TX, y = (t / TX) % TY, z = t / (TX * TY);
    V v;
    if (x < ex && y < ey && z < ez) {
      v = reinterpret_cast<const V*>(grid)[(static_cast<size_t>(z0 + z) * sd.n[1] + y0 + y) * sd.n[0] +
                                           x0 + x];
    } else {
      if constexpr (NC == 4)
        v = V{R(0), R(0), R(0), R(0)};
      else
        v = R(0);
    }
    sG[t] = v;
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nslots = sd.pstride;
  for (int a0 = p0 + warp * 32 * A; a0 < p1; a0 += WARPS * 32 * A) {
    R w1[A][TX], w2[A][TY];
    int2 pr[A];
    bool act[A];
#pragma unroll
    for (int a = 0; a < A; ++a) {
      const int e = a0 + a * 32 + lane;
      act[a] = e < p1;
      pr[a] = act[a] ? pairs[e] : make_int2(0, 0);
      const R* wk = wtab + static_cast<size_t>(pr[a].x) * sd.wstride;
#pragma unroll
      for (int x = 0; x < TX; ++x) w1[a][x] = act[a] ? wk[sd.woff[0] + (pr[a].y & 0xff) * TX + x] : R(0);
#pragma unroll
      for (int y = 0; y < TY; ++y)
        w2[a][y] = act[a] ? wk[sd.woff[1] + ((pr[a].y >> 8) & 0xff) * TY + y] : R(0);
      const R* wz = wk + sd.woff[2] + (pr[a].y >> 16) * TZ;
#pragma unroll
      for (int z = 0; z < TZ; ++z) sW3[warp][z][a * 32 + lane] = act[a] ? wz[z] : R(0);
    }
    __syncwarp();
    double acc[A][NC];
#pragma unroll
    for (int a = 0; a < A; ++a)
#pragma unroll
      for (int c = 0; c < NC; ++c) acc[a][c] = 0.0;
#pragma unroll 1
    for (int z = 0; z < TZ; ++z) {
      R w3[A];
#pragma unroll
      for (int a = 0; a < A; ++a) w3[a] = sW3[warp][z][a * 32 + lane];
      // The plane's rows are summed in R, the plane sum then added in FP64.
      R pl[A][NC];
#pragma unroll
      for (int a = 0; a < A; ++a)
#pragma unroll
        for (int c = 0; c < NC; ++c) pl[a][c] = R(0);
#pragma unroll
      for (int y = 0; y < TY; ++y) {
        R w23[A];
        bool any = false;
#pragma unroll
        for (int a = 0; a < A; ++a) {
          w23[a] = w2[a][y] * w3[a];
          any = any || (w23[a] != R(0));
        }
        if (!__any_sync(0xffffffffu, any)) continue;
        R rs[A][NC];
#pragma unroll
        for (int a = 0; a < A; ++a)
#pragma unroll
          for (int c = 0; c < NC; ++c) rs[a][c] = R(0);
        const V* row = sG + (z * TY + y) * TX;
#pragma unroll
        for (int x = 0; x < TX; ++x) {
          const V g = row[x];
#pragma unroll
          for (int a = 0; a < A; ++a) {
            if constexpr (NC == 4) {
              rs[a][0] = fma(w1[a][x], g.x, rs[a][0]);
              rs[a][1] = fma(w1[a][x], g.y, rs[a][1]);
              rs[a][2] = fma(w1[a][x], g.z, rs[a][2]);
              rs[a][3] = fma(w1[a][x], g.w, rs[a][3]);
            } else {
              rs[a][0] = fma(w1[a][x], g, rs[a][0]);
            }
          }
        }
#pragma unroll
        for (int a = 0; a < A; ++a)
#pragma unroll
          for (int c = 0; c < NC; ++c) pl[a][c] = fma(w23[a], rs[a][c], pl[a][c]);
      }
#pragma unroll
      for (int a = 0; a < A; ++a)
#pragma unroll
        for (int c = 0; c < NC; ++c) acc[a][c] += static_cast<double>(pl[a][c]);
    }
#pragma unroll
    for (int a = 0; a < A; ++a) {
      if (!act[a]) continue;
      const int ps = pr[a].y;
      const int sidx = ((ps >> 16) * sd.S[1] + ((ps >> 8) & 0xff)) * sd.S[0] + (ps & 0xff);
      double* dst = part + (static_cast<size_t>(pr[a].x) * nslots + sidx) * NC;
#pragma unroll
      for (int c = 0; c < NC; ++c) dst[c] = acc[a][c];
    }
    __syncwarp();  // sW3 is rewritten by the next iteration
  }
}

// ---------------------------------------------------------------------------
// FP32 gather with window derivatives (force scheme ad).  The tile holds the
// potential grid g alone.  With W = w1 w2 w3 and D_d the same product with
// axis d's weights replaced by their derivatives with respect to s_d, an atom
// needs phi = sum W g and D_d = sum D_d g.  The derivative weights change sign
// across the stencil while g carries a large smooth part, so in FP32 the sums
// would cancel; they run instead on g' = g - c, with c the grid value at the
// tile's first point (subtracted once, when the tile is staged), and the
// tile's c terms are added back in FP64 from the tile's weight sums:
//   phi_t = sum_t W g' + c Sx Sy Sz,  D_1,t = sum_t dW_1 g' + c dSx Sy Sz, ...
// (S, dS: sums over the tile's points of the weights and their derivatives).
// Per (z, y) row two x sums, r0 = sum_x w1 g' and r1 = sum_x dw1 g', feed all
// four:  phi += w2 w3 r0, D_1 += w2 w3 r1, D_2 += dw2 w3 r0, D_3 += w2 dw3 r0.
// Lanes carry A atoms of the tile's list as in k_gather_tiles (x weights in
// registers, y and z rows staged in shared memory); products and plane sums in
// FP32, the sum over planes in FP64; the four partials go to the atom's slot.
// ---------------------------------------------------------------------------
template <int A, int WARPS>
__device__ __forceinline__ void gather_tiles_ad_body(int tx, int ty, int tz,
                                                     const int* __restrict__ tile_start,
                                                                const int2* __restrict__ pairs,
                                                                const float* __restrict__ wtab,
                                                                StencilDims sd,
                                                                const float* __restrict__ grid,
                                                                double* __restrict__ part) {
  chain_enter();
  __shared__ float sG[TZ * TY * TX];
  // y and z weights and their derivatives, lane fastest: [kind][row][lane]
  // with kind 0 = w2, 1 = dw2, 2 = w3, 3 = dw3.
  __shared__ float sYZ[WARPS][4][TY][32 * A];
  static_assert(TY == TZ, "y and z rows share one staging layout");
  const int tile = (tz * sd.ntiles[1] + ty) * sd.ntiles[0] + tx;
  const int x0 = tx * TX, y0 = ty * TY, z0 = tz * TZ;
  const int ex = min(TX, sd.n[0] - x0), ey = min(TY, sd.n[1] - y0), ez = min(TZ, sd.n[2] - z0);
  const int p0 = tile_start[tile], p1 = tile_start[tile + 1];
  if (p0 == p1) return;  // no atom reaches this tile
  const float cg = grid[(static_cast<size_t>(z0) * sd.n[1] + y0) * sd.n[0] + x0];
#pragma unroll 4
  for (int t = threadIdx.x; t < TX * TY * TZ; t += 32 * WARPS) {
    const int x = t % TX, y = (t / TX) % TY, z = t / (TX * TY);
    // points past the grid's end carry zero weight for every atom
    sG[t] = (x < ex && y < ey && z < ez)
                ? grid[(static_cast<size_t>(z0 + z) * sd.n[1] + y0 + y) * sd.n[0] + x0 + x] - cg
                : 0.0f;
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nslots = sd.pstride;
  float(*YZ)[TY][32 * A] = sYZ[warp];
  for (int a0 = p0 + warp * 32 * A; a0 < p1; a0 += WARPS * 32 * A) {
    float w1[A][TX], d1[A][TX];
    int2 pr[A];
    bool act[A];
#pragma unroll
    for (int a = 0; a < A; ++a) {
      const int e = a0 + a * 32 + lane;
      act[a] = e < p1;
      pr[a] = act[a] ? pairs[e] : make_int2(0, 0);
      const float* wk = wtab + static_cast<size_t>(pr[a].x) * sd.wstride;
      const int ox = sd.woff[0] + (pr[a].y & 0xff) * TX;
      const int oy = sd.woff[1] + ((pr[a].y >> 8) & 0xff) * TY;
      const int oz = sd.woff[2] + (pr[a].y >> 16) * TZ;
      float t[4][8];
      if (act[a]) {
        load8(wk + ox, w1[a]);
        load8(wk + sd.dwoff + ox, d1[a]);
        load8(wk + oy, t[0]);
        load8(wk + sd.dwoff + oy, t[1]);
        load8(wk + oz, t[2]);
        load8(wk + sd.dwoff + oz, t[3]);
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) w1[a][j] = d1[a][j] = t[0][j] = t[1][j] = t[2][j] = t[3][j] = 0.0f;
      }
#pragma unroll
      for (int kd = 0; kd < 4; ++kd)
#pragma unroll
        for (int j = 0; j < 8; ++j) YZ[kd][j][a * 32 + lane] = t[kd][j];
    }
    __syncwarp();
    double acc[A][4];
    float sz[A], dsz[A];
#pragma unroll
    for (int a = 0; a < A; ++a) {
      sz[a] = dsz[a] = 0.0f;
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[a][c] = 0.0;
    }
#pragma unroll 1
    for (int z = 0; z < TZ; ++z) {
      float w3[A], d3[A], pl[A][4];
#pragma unroll
      for (int a = 0; a < A; ++a) {
        w3[a] = YZ[2][z][a * 32 + lane];
        d3[a] = YZ[3][z][a * 32 + lane];
        sz[a] += w3[a];
        dsz[a] += d3[a];
        pl[a][0] = pl[a][1] = pl[a][2] = pl[a][3] = 0.0f;  // plane sums, FP32
      }
#pragma unroll
      for (int y = 0; y < TY; ++y) {
        // A zero window product means the row lies outside the atom's stencil
        // along y or z, where the derivatives vanish as well.
        float w2[A], d2[A], w23[A];
        bool any = false;
#pragma unroll
        for (int a = 0; a < A; ++a) {
          w2[a] = YZ[0][y][a * 32 + lane];
          d2[a] = YZ[1][y][a * 32 + lane];
          w23[a] = w2[a] * w3[a];
          any = any || (w23[a] != 0.0f);
        }
        if (!__any_sync(0xffffffffu, any)) continue;
        float r0[A], r1[A];
#pragma unroll
        for (int a = 0; a < A; ++a) r0[a] = r1[a] = 0.0f;
        const float* row = sG + (z * TY + y) * TX;
#pragma unroll
        for (int x = 0; x < TX; ++x) {
          const float g = row[x];
#pragma unroll
          for (int a = 0; a < A; ++a) {
            r0[a] = fmaf(w1[a][x], g, r0[a]);
            r1[a] = fmaf(d1[a][x], g, r1[a]);
          }
        }
#pragma unroll
        for (int a = 0; a < A; ++a) {
          pl[a][0] = fmaf(w23[a], r0[a], pl[a][0]);
          pl[a][1] = fmaf(w23[a], r1[a], pl[a][1]);
          pl[a][2] = fmaf(d2[a] * w3[a], r0[a], pl[a][2]);
          pl[a][3] = fmaf(w2[a] * d3[a], r0[a], pl[a][3]);
        }
      }
#pragma unroll
      for (int a = 0; a < A; ++a)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[a][c] += static_cast<double>(pl[a][c]);
    }
#pragma unroll
    for (int a = 0; a < A; ++a) {
      if (!act[a]) continue;
      // the c terms of this tile: c (S or dS along each axis)
      double sx = 0.0, dsx = 0.0, sy = 0.0, dsy = 0.0;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        sx += w1[a][j];
        dsx += d1[a][j];
        sy += YZ[0][j][a * 32 + lane];
        dsy += YZ[1][j][a * 32 + lane];
      }
      const double c = cg;
      acc[a][0] += c * sx * sy * sz[a];
      acc[a][1] += c * dsx * sy * sz[a];
      acc[a][2] += c * sx * dsy * sz[a];
      acc[a][3] += c * sx * sy * dsz[a];
      const int ps = pr[a].y;
      const int sidx = ((ps >> 16) * sd.S[1] + ((ps >> 8) & 0xff)) * sd.S[0] + (ps & 0xff);
      double* dst = part + (static_cast<size_t>(pr[a].x) * nslots + sidx) * 4;
#pragma unroll
      for (int c4 = 0; c4 < 4; ++c4) dst[c4] = acc[a][c4];
    }
    __syncwarp();  // the staged rows are rewritten by the next iteration
  }
}

// ---------------------------------------------------------------------------
// FP64 gather on the tensor cores.  With the tile's values G[z][y][x][c] in
// shared memory, an atom's result is
//   phi_a,c = sum_z w3_a(z) sum_y w2_a(y) T_a[z][y][c],
//   T_a[z][y][c] = sum_x w1_a(x) G[z][y][x][c],
// and T is a matrix product: rows are atoms (M blocks of 8), the contraction
// runs over x (two k-steps of 4), columns over (c, y) (N blocks of the 8 y
// values of one component).  Scaling the A fragment by w3_a(z) lets the DMMA
// accumulators sum over the planes too.  Each warp takes up to MB M blocks of
// a round of 8 MB WARPS atoms; per plane and component it issues two DMMAs per M block.
// The weight rows are staged as in the spread, four threads to a row of 64 bytes (one
// value, 12,000 sites, 8 calls: 286 -> 238 us; a batch of 128 cells 511 -> 471).
// At the end the lane holding C for (atom, y pair) folds in w2, and the four
// lanes of an atom are summed with shuffles in a fixed order.  Partials go to the (atom, slot) array as in the CUDA-core
// gather; results are deterministic.
// Tile layout in shared memory: row (z, y) holds 8 points x NC values, padded
// to kGRow doubles so the B-fragment reads are nearly conflict-free.
// ---------------------------------------------------------------------------
template <int NC>
struct GatherRow {
  static constexpr int value = NC == 4 ? 34 : 12;  // 16-byte multiples
};
// WARPS warps per CTA, MB M blocks of 8 atoms per warp and round.
template <typename R, int NC, int WARPS, int MB>
__device__ __forceinline__ void gather_tiles_dmma_body(int tx, int ty, int tz,
                                                       const int* __restrict__ tile_start,
                                                       const int2* __restrict__ pairs,
                                                       const R* __restrict__ wtab, StencilDims sd,
                                                       const R* __restrict__ grid,
                                                       double* __restrict__ part) {
  chain_enter();
  constexpr int RS = GatherRow<NC>::value;
  constexpr int kGatherAtoms = WARPS * MB * 8;  // atoms staged per round
  __shared__ __align__(16) double sG[TZ * TY * RS];
  __shared__ __align__(16) double sW[3][kGatherAtoms][kWRow];
  __shared__ int2 sPair[kGatherAtoms];
  const int tile = (tz * sd.ntiles[1] + ty) * sd.ntiles[0] + tx;
  const int p0 = tile_start[tile], p1 = tile_start[tile + 1];
  if (p0 == p1) return;  // no atom reaches this tile
  const int x0 = tx * TX, y0 = ty * TY, z0 = tz * TZ;
  const int ex = min(TX, sd.n[0] - x0), ey = min(TY, sd.n[1] - y0), ez = min(TZ, sd.n[2] - z0);
  // Stage the tile: 16-byte chunks (NC = 4: half a point; NC = 1: two points).
  constexpr int kChunksPerRow = TX * NC / 2;
  for (int t = threadIdx.x; t < TZ * TY * kChunksPerRow; t += blockDim.x) {
    const int row = t / kChunksPerRow, h = t - row * kChunksPerRow;
    const int z = row / TY, y = row - z * TY;
    const int x = NC == 4 ? h / 2 : 2 * h;  // first point of the chunk
    double* dst = sG + row * RS + 2 * h;
    if (z < ez && y < ey && x < ex) {
      const R* src = grid + ((static_cast<size_t>(z0 + z) * sd.n[1] + y0 + y) * sd.n[0] + x0) * NC + 2 * h;
      stage2(dst, src);
    } else {
      dst[0] = 0.0;
      dst[1] = 0.0;
    }
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int fr = lane >> 2, fk = lane & 3;
  const int nslots = sd.pstride;
  for (int b0 = p0; b0 < p1; b0 += kGatherAtoms) {
    const int nb = min(kGatherAtoms, p1 - b0);
    __syncthreads();  // the previous round's weights are no longer read
    // Four threads per weight row of 64 bytes, whole sectors to an access; the entries
    // before the first copy, which the compiler does not move loads across.
    int2 pr[MB];
#pragma unroll
    for (int h = 0; h < MB; ++h) {
      const int a = h * (8 * WARPS) + (threadIdx.x >> 2);
      pr[h] = a < nb ? pairs[b0 + a] : make_int2(0, 0);
    }
#pragma unroll
    for (int h = 0; h < MB; ++h) {
      const int a = h * (8 * WARPS) + (threadIdx.x >> 2), c = 2 * (threadIdx.x & 3);
      if (a < nb) {
        if (c == 0) sPair[a] = pr[h];
        const R* wk = wtab + static_cast<size_t>(pr[h].x) * sd.wstride + c;
        stage2(&sW[0][a][c], wk + sd.woff[0] + (pr[h].y & 0xff) * TX);
        stage2(&sW[1][a][c], wk + sd.woff[1] + ((pr[h].y >> 8) & 0xff) * TY);
        stage2(&sW[2][a][c], wk + sd.woff[2] + (pr[h].y >> 16) * TZ);
      } else {  // rows past the list: zero weights, results discarded
#pragma unroll
        for (int d = 0; d < 3; ++d) sW[d][a][c] = sW[d][a][c + 1] = 0.0;
      }
    }
    cp_async_wait_all();  // also completes the tile copies on the first round
    __syncthreads();
    // This warp's M blocks: atoms warp * 32 + mb * 8 + (0..7) of the round.
    const int abase = warp * (MB * 8);
    if (abase >= nb) continue;
    const int nmb = min(MB, (nb - abase + 7) / 8);
    double fa[MB][2], cacc[MB][NC][2];
#pragma unroll
    for (int mb = 0; mb < MB; ++mb) {
      const int am = abase + mb * 8 + fr;  // this lane's atom row
      fa[mb][0] = sW[0][am][fk];           // A[m][k], k-step 0: x = k
      fa[mb][1] = sW[0][am][4 + fk];       // k-step 1: x = 4 + k
#pragma unroll
      for (int c = 0; c < NC; ++c) cacc[mb][c][0] = cacc[mb][c][1] = 0.0;
    }
    // w3 is folded into the A fragment, so C sums over z as well:
    // C[m][y] = sum_z sum_x w3_m(z) w1_m(x) G[z][y][x][c].
#pragma unroll 1
    for (int z = 0; z < TZ; ++z) {
      double a0[MB], a1[MB];
#pragma unroll
      for (int mb = 0; mb < MB; ++mb) {
        const double w3 = sW[2][abase + mb * 8 + fr][z];
        a0[mb] = fa[mb][0] * w3;
        a1[mb] = fa[mb][1] * w3;
      }
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        // B[k][n] = G[z][y = n][x = 4 ks + k][c] at lane 4n + k.
        const double* gz = sG + (z * TY + fr) * RS + c;
        const double b0v = gz[fk * NC];
        const double b1v = gz[(4 + fk) * NC];
#pragma unroll
        for (int mb = 0; mb < MB; ++mb) {
          if (mb < nmb) {
            dmma_m8n8k4(cacc[mb][c][0], cacc[mb][c][1], a0[mb], b0v);
            dmma_m8n8k4(cacc[mb][c][0], cacc[mb][c][1], a1[mb], b1v);
          }
        }
      }
    }
#pragma unroll
    for (int mb = 0; mb < MB; ++mb) {
      if (mb >= nmb) break;
      // This lane holds C for y = 2 fk and 2 fk + 1: weight them by w2 and sum
      // the four lanes of the atom.
      const int am = abase + mb * 8 + fr;
      const double w20 = sW[1][am][2 * fk], w21 = sW[1][am][2 * fk + 1];
      double acc[NC];
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        acc[c] = fma(w20, cacc[mb][c][0], w21 * cacc[mb][c][1]);
        acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], 1);
        acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], 2);
      }
      const int a = abase + mb * 8 + fr;
      if (fk == 0 && a < nb) {
        const int2 pr = sPair[a];
        const int ps = pr.y;
        const int sidx = ((ps >> 16) * sd.S[1] + ((ps >> 8) & 0xff)) * sd.S[0] + (ps & 0xff);
        double* dst = part + (static_cast<size_t>(pr.x) * nslots + sidx) * NC;
        if constexpr (NC == 4) {
          reinterpret_cast<double2*>(dst)[0] = make_double2(acc[0], acc[1]);
          reinterpret_cast<double2*>(dst)[1] = make_double2(acc[2], acc[3]);
        } else {
          dst[0] = acc[0];
        }
      }
    }
  }
}

// ---------------------------------------------------------------------------
// FP64 gather with window derivatives (force scheme ad) on the tensor cores.
// The tile holds the potential grid alone.  Per plane z the x contraction
// takes two A operands that do not change from plane to plane, w1 and dw1:
//   C_w[z][m][y] = sum_x w1_m(x) G[z][y][x],  C_d[z][m][y] = sum_x dw1_m(x) G[z][y][x]
// (four DMMAs per plane for 8 atoms, each plane its own accumulators, so the
// 32 DMMAs of a tile are independent), and the y and z weights are applied
// afterwards:
//   phi = sum_z w3 sum_y w2 C_w,  D_1 = sum_z w3 sum_y w2 C_d,
//   D_2 = sum_z w3 sum_y dw2 C_w,  D_3 = sum_z dw3 sum_y w2 C_w.
// WARPS warps per tile, each taking blocks of 8 atoms (one M block) on its own.
// Shared layout and fragment mapping as in k_gather_tiles_dmma with NC = 1; six
// weight rows per atom (w1 w2 w3 dw1 dw2 dw3).
// ---------------------------------------------------------------------------
template <typename R, int WARPS>
__device__ __forceinline__ void gather_tiles_dmma_ad_body(
    int tx, int ty, int tz, const int* __restrict__ tile_start, const int2* __restrict__ pairs,
    const R* __restrict__ wtab, StencilDims sd, const R* __restrict__ grid,
    double* __restrict__ part) {
  chain_enter();
  constexpr int RS = GatherRow<1>::value;
  __shared__ __align__(16) double sG[TZ * TY * RS];
  __shared__ __align__(16) double sW[WARPS][6][8][kWRow];  // per warp: its 8 atoms' rows
  const int tile = (tz * sd.ntiles[1] + ty) * sd.ntiles[0] + tx;
  const int p0 = tile_start[tile], p1 = tile_start[tile + 1];
  if (p0 == p1) return;  // no atom reaches this tile
  const int x0 = tx * TX, y0 = ty * TY, z0 = tz * TZ;
  const int ex = min(TX, sd.n[0] - x0), ey = min(TY, sd.n[1] - y0), ez = min(TZ, sd.n[2] - z0);
  // Stage the tile: 16-byte chunks of two points.
  constexpr int kChunksPerRow = TX / 2;
  for (int t = threadIdx.x; t < TZ * TY * kChunksPerRow; t += blockDim.x) {
    const int row = t / kChunksPerRow, h = t - row * kChunksPerRow;
    const int z = row / TY, y = row - z * TY;
    const int x = 2 * h;
    double* dst = sG + row * RS + 2 * h;
    if (z < ez && y < ey && x < ex) {
      stage2(dst, grid + (static_cast<size_t>(z0 + z) * sd.n[1] + y0 + y) * sd.n[0] + x0 + x);
    } else {
      dst[0] = 0.0;
      dst[1] = 0.0;
    }
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int fr = lane >> 2, fk = lane & 3;
  const int nslots = sd.pstride;
  double(*W)[8][kWRow] = sW[warp];
  cp_async_wait_all();
  __syncthreads();  // the tile, staged by all warps; the only CTA barrier
  // Each warp takes blocks of 8 atoms of the tile's list on its own.  Lane
  // (fr, fk) stages 16-byte chunk fk of atom fr's six rows and later holds
  // that atom's fragments.
  for (int b0 = p0 + warp * 8; b0 < p1; b0 += WARPS * 8) {
    const int nb = min(8, p1 - b0);
    __syncwarp();  // the previous block's rows are no longer read
    int2 pr = make_int2(0, 0);
    if (fr < nb) {
      pr = pairs[b0 + fr];
      const R* wk = wtab + static_cast<size_t>(pr.x) * sd.wstride;
      const int off[3] = {sd.woff[0] + (pr.y & 0xff) * TX, sd.woff[1] + ((pr.y >> 8) & 0xff) * TY,
                          sd.woff[2] + (pr.y >> 16) * TZ};
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        stage2(&W[d][fr][2 * fk], wk + off[d] + 2 * fk);
        stage2(&W[3 + d][fr][2 * fk], wk + sd.dwoff + off[d] + 2 * fk);
      }
    } else {  // rows past the list: zero weights, results discarded
#pragma unroll
      for (int d = 0; d < 6; ++d) W[d][fr][2 * fk] = W[d][fr][2 * fk + 1] = 0.0;
    }
    cp_async_wait_all();
    __syncwarp();
    const double fw0 = W[0][fr][fk], fw1 = W[0][fr][4 + fk];
    const double fd0 = W[3][fr][fk], fd1 = W[3][fr][4 + fk];
    double cw[TZ][2], cd[TZ][2];
#pragma unroll
    for (int z = 0; z < TZ; ++z) {
      // B[k][n] = G[z][y = n][x = 4 ks + k] at lane 4n + k.
      const double* gz = sG + (z * TY + fr) * RS;
      const double b0v = gz[fk], b1v = gz[4 + fk];
      cw[z][0] = cw[z][1] = cd[z][0] = cd[z][1] = 0.0;
      dmma_m8n8k4(cw[z][0], cw[z][1], fw0, b0v);
      dmma_m8n8k4(cw[z][0], cw[z][1], fw1, b1v);
      dmma_m8n8k4(cd[z][0], cd[z][1], fd0, b0v);
      dmma_m8n8k4(cd[z][0], cd[z][1], fd1, b1v);
    }
    // This lane holds C for y = 2 fk and 2 fk + 1 of every plane.
    const double w20 = W[1][fr][2 * fk], w21 = W[1][fr][2 * fk + 1];
    const double d20 = W[4][fr][2 * fk], d21 = W[4][fr][2 * fk + 1];
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (int z = 0; z < TZ; ++z) {
      const double w3 = W[2][fr][z], d3 = W[5][fr][z];
      const double pw = fma(w20, cw[z][0], w21 * cw[z][1]);
      const double pd = fma(w20, cd[z][0], w21 * cd[z][1]);
      const double qw = fma(d20, cw[z][0], d21 * cw[z][1]);
      acc[0] = fma(w3, pw, acc[0]);
      acc[1] = fma(w3, pd, acc[1]);
      acc[2] = fma(w3, qw, acc[2]);
      acc[3] = fma(d3, pw, acc[3]);
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], 1);
      acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], 2);
    }
    if (fk == 0 && fr < nb) {
      const int ps = pr.y;
      const int sidx = ((ps >> 16) * sd.S[1] + ((ps >> 8) & 0xff)) * sd.S[0] + (ps & 0xff);
      double* dst = part + (static_cast<size_t>(pr.x) * nslots + sidx) * 4;
      reinterpret_cast<double2*>(dst)[0] = make_double2(acc[0], acc[1]);
      reinterpret_cast<double2*>(dst)[1] = make_double2(acc[2], acc[3]);
    }
  }
}

// Final per-atom sum of the slot partials in a fixed order, with the assembly
// of fft/ewald_fft_3d.f90:121-132: pot = (sr + lr) + self, force = sr + q lr.
// A group of lanes per atom (a warp, or 8 lanes when the atom has at most 32
// slots) reads the atom's slots (contiguous, coalesced), then a shuffle tree
// sums them (a fixed order: results are reproducible).
// Dual basis rows for the ad partials (on = 0: ik partials, Cartesian already).
struct RecRows {
  double b[3][3];
  int on;
};

// LPA lanes per atom (32, or 8 when an atom has at most 32 slots: four atoms
// per warp).
template <int NC, int LPA>
__device__ __forceinline__ void gather_final_body(const int4* __restrict__ slot,
                                                  const int* __restrict__ perm,
                                                  const double* __restrict__ part, int k,
                                                  int lane, bool live, const StencilDims& sd,
                                                  const double* __restrict__ q, double self_coef,
                                                  double pot_shift,
                                                  const double* __restrict__ pot_sr,
                                                  const double* __restrict__ f_sr,
                                                  double* __restrict__ pot,
                                                  double* __restrict__ force, const RecRows& rr) {
  const int4 si = live ? slot[k] : make_int4(0, 0, 0, 0);
  const int cx = slot_count(si.x), cy = slot_count(si.y), cz = slot_count(si.z);
  const int nslots = sd.S[0] * sd.S[1] * sd.S[2];
  const double* pk = part + static_cast<size_t>(live ? k : 0) * sd.pstride * NC;
  double acc[NC];
#pragma unroll
  for (int c = 0; c < NC; ++c) acc[c] = 0.0;
  for (int s = lane; s < (live ? nslots : 0); s += LPA) {
    const int sx = s % sd.S[0], sy = (s / sd.S[0]) % sd.S[1], sz = s / (sd.S[0] * sd.S[1]);
    if (sx < cx && sy < cy && sz < cz) {  // slots past the atom's tiles hold no partial
      if constexpr (NC == 4) {  // a slot's four values, 32 bytes, in two loads
        const double2 p0 = reinterpret_cast<const double2*>(pk)[2 * s];
        const double2 p1 = reinterpret_cast<const double2*>(pk)[2 * s + 1];
        acc[0] += p0.x;
        acc[1] += p0.y;
        acc[2] += p1.x;
        acc[3] += p1.y;
      } else {
        acc[0] += pk[s];
      }
    }
  }
  // A fixed shuffle tree within the atom's LPA lanes.
#pragma unroll
  for (int c = 0; c < NC; ++c)
#pragma unroll
    for (int off = LPA / 2; off > 0; off >>= 1) acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], off);
  if (lane != 0 || !live) return;
  const int i = perm[k];
  const double qi = q[i];
  pot[i] = (pot_sr[i] + acc[0]) + self_coef * qi + pot_shift;
  if (NC == 4 && force) {
    if (rr.on) {  // ad: F = -q sum_e D_e b_e, D_e the derivative along s_e
#pragma unroll
      for (int d = 0; d < 3; ++d)
        force[3 * i + d] =
            f_sr[3 * i + d] - qi * (acc[1] * rr.b[0][d] + acc[2] * rr.b[1][d] + acc[3] * rr.b[2][d]);
    } else {
#pragma unroll
      for (int d = 0; d < 3; ++d) force[3 * i + d] = f_sr[3 * i + d] + qi * acc[1 + d];
    }
  }
}

template <int NC, int LPA>
__global__ void k_gather_final(const int4* __restrict__ slot, const int* __restrict__ perm,
                               const double* __restrict__ part, int n, StencilDims sd,
                               const double* __restrict__ q, double self_coef, double pot_shift,
                               const double* __restrict__ pot_sr, const double* __restrict__ f_sr,
                               double* __restrict__ pot, double* __restrict__ force, RecRows rr) {
  const long t = static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x;
  const int k = static_cast<int>(t / LPA);
  // Lanes past the last atom stay to the end: the shuffles below take the whole warp.
  gather_final_body<NC, LPA>(slot, perm, part, k, static_cast<int>(t % LPA), k < n, sd, q,
                             self_coef, pot_shift, pot_sr, f_sr, pot, force, rr);
}

// Every cell of a batch: the atom's cell gives its slot layout, self term and
// dual basis (window-derivative partials are fractional derivatives).
template <int NC, int LPA>
__global__ void k_gather_final_seg(const BatchCell* __restrict__ cells,
                                   const int* __restrict__ prefix, int ncells,
                                   const int4* __restrict__ slot, const int* __restrict__ perm,
                                   const double* __restrict__ part, int n,
                                   const double* __restrict__ q, const double* __restrict__ pot_sr,
                                   const double* __restrict__ f_sr, double* __restrict__ pot,
                                   double* __restrict__ force) {
  const long t = static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x;
  const int k = static_cast<int>(t / LPA);
  const bool live = k < n;
  const BatchCell& bc = cells[seg_cell(prefix, ncells, live ? k : n - 1)];
  RecRows rr;
  rr.on = 1;
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int d = 0; d < 3; ++d) rr.b[a][d] = bc.rec[a][d];
  const StencilDims sd = bc.sd;
  gather_final_body<NC, LPA>(slot, perm, part, k, static_cast<int>(t % LPA), live, sd, q,
                             bc.self_coef, 0.0, pot_sr, f_sr, pot, force, rr);
}

// FP64 tensor-core throughput probe: every warp issues independent DMMAs on
// register operands (eight accumulator pairs, no memory traffic), so the
// measured rate is the m8n8k4 FP64 pipe's own.
__global__ void __launch_bounds__(128) k_dmma_peak(int iters, double seed, double* sink) {
  double acc[8][2];
#pragma unroll
  for (int i = 0; i < 8; ++i) acc[i][0] = acc[i][1] = 0.0;
  const double a = seed + 1.0e-9 * threadIdx.x, b = 1.0 - seed;
  for (int it = 0; it < iters; ++it) {
#pragma unroll
    for (int i = 0; i < 8; ++i) dmma_m8n8k4(acc[i][0], acc[i][1], a, b);
  }
  double t = 0.0;
#pragma unroll
  for (int i = 0; i < 8; ++i) t += acc[i][0] + acc[i][1];
  if (t == -1.0) sink[threadIdx.x] = t;  // never true; keeps the work live
}

// ---- the tile kernels: one tile per CTA (blockIdx = tile), or, for a batch,
// the tiles of every cell (blockIdx.x over the cells' tiles end to end; the
// cell's tile list, weights layout and grid from the batch table).
__device__ __forceinline__ const BatchCell& tile_of_block(const BatchCell* __restrict__ cells,
                                                          const int* __restrict__ prefix,
                                                          int ncells, int* tx, int* ty, int* tz) {
  const int c = seg_cell(prefix, ncells, blockIdx.x);
  const BatchCell& bc = cells[c];
  const int local = static_cast<int>(blockIdx.x) - prefix[c];
  *tx = local % bc.sd.ntiles[0];
  *ty = (local / bc.sd.ntiles[0]) % bc.sd.ntiles[1];
  *tz = local / (bc.sd.ntiles[0] * bc.sd.ntiles[1]);
  return bc;
}

template <typename R>
__global__ void __launch_bounds__(kSpreadLanes) k_spread_tiles(const int* __restrict__ tile_start,
                                                               const int2* __restrict__ pairs,
                                                               const R* __restrict__ wtab,
                                                               const R* __restrict__ qk,
                                                               StencilDims sd, R* __restrict__ grid) {
  spread_tiles_body<R>(blockIdx.x, blockIdx.y, blockIdx.z, tile_start, pairs, wtab, qk, sd, grid);
}
template <typename R, int ATOMS>
__global__ void __launch_bounds__(32) k_spread_tiles_dmma(const int* __restrict__ tile_start,
                                                          const int2* __restrict__ unordered,
                                                          int2* pairs, bool keep,
                                                          const R* __restrict__ wtab,
                                                          const R* __restrict__ qk,
                                                          StencilDims sd, R* __restrict__ grid) {
  spread_tiles_dmma_body<R, ATOMS>(blockIdx.x, blockIdx.y, blockIdx.z, tile_start, unordered, pairs,
                                   keep, wtab, qk, sd, grid);
}
template <typename R, int ATOMS>
__global__ void __launch_bounds__(32) k_spread_tiles_dmma_seg(
    const BatchCell* __restrict__ cells, const int* __restrict__ prefix, int ncells,
    const int* __restrict__ tile_start, const int2* __restrict__ unordered, int2* pairs,
    const R* __restrict__ wtab, const R* __restrict__ qk) {
  int tx, ty, tz;
  const BatchCell& bc = tile_of_block(cells, prefix, ncells, &tx, &ty, &tz);
  spread_tiles_dmma_body<R, ATOMS>(tx, ty, tz, tile_start + bc.tile0, unordered, pairs, false, wtab, qk,
                                   bc.sd, static_cast<R*>(bc.grid));
}

template <typename R, int NC, int A, int WARPS>
__global__ void __launch_bounds__(32 * WARPS) k_gather_tiles(const int* __restrict__ tile_start,
                                                             const int2* __restrict__ pairs,
                                                             const R* __restrict__ wtab,
                                                             StencilDims sd,
                                                             const R* __restrict__ grid,
                                                             double* __restrict__ part) {
  gather_tiles_body<R, NC, A, WARPS>(blockIdx.x, blockIdx.y, blockIdx.z, tile_start, pairs, wtab,
                                     sd, grid, part);
}
template <int A, int WARPS>
__global__ void __launch_bounds__(32 * WARPS) k_gather_tiles_ad(const int* __restrict__ tile_start,
                                                                const int2* __restrict__ pairs,
                                                                const float* __restrict__ wtab,
                                                                StencilDims sd,
                                                                const float* __restrict__ grid,
                                                                double* __restrict__ part) {
  gather_tiles_ad_body<A, WARPS>(blockIdx.x, blockIdx.y, blockIdx.z, tile_start, pairs, wtab, sd,
                                 grid, part);
}
template <typename R, int NC, int WARPS, int MB>
__global__ void __launch_bounds__(32 * WARPS) k_gather_tiles_dmma(const int* __restrict__ tile_start,
                                                                  const int2* __restrict__ pairs,
                                                                  const R* __restrict__ wtab,
                                                                  StencilDims sd,
                                                                  const R* __restrict__ grid,
                                                                  double* __restrict__ part) {
  gather_tiles_dmma_body<R, NC, WARPS, MB>(blockIdx.x, blockIdx.y, blockIdx.z, tile_start, pairs,
                                           wtab, sd, grid, part);
}
template <typename R, int NC, int WARPS, int MB>
__global__ void __launch_bounds__(32 * WARPS) k_gather_tiles_dmma_seg(
    const BatchCell* __restrict__ cells, const int* __restrict__ prefix, int ncells,
    const int* __restrict__ tile_start, const int2* __restrict__ pairs,
    const R* __restrict__ wtab, double* __restrict__ part) {
  int tx, ty, tz;
  const BatchCell& bc = tile_of_block(cells, prefix, ncells, &tx, &ty, &tz);
  gather_tiles_dmma_body<R, NC, WARPS, MB>(tx, ty, tz, tile_start + bc.tile0, pairs, wtab, bc.sd,
                                           static_cast<const R*>(bc.out), part);
}

template <typename R, int WARPS>
__global__ void __launch_bounds__(32 * WARPS) k_gather_tiles_dmma_ad(
    const int* __restrict__ tile_start, const int2* __restrict__ pairs,
    const R* __restrict__ wtab, StencilDims sd, const R* __restrict__ grid,
    double* __restrict__ part) {
  gather_tiles_dmma_ad_body<R, WARPS>(blockIdx.x, blockIdx.y, blockIdx.z, tile_start, pairs, wtab,
                                      sd, grid, part);
}
template <typename R, int WARPS>
__global__ void __launch_bounds__(32 * WARPS) k_gather_tiles_dmma_ad_seg(
    const BatchCell* __restrict__ cells, const int* __restrict__ prefix, int ncells,
    const int* __restrict__ tile_start, const int2* __restrict__ pairs,
    const R* __restrict__ wtab, double* __restrict__ part) {
  int tx, ty, tz;
  const BatchCell& bc = tile_of_block(cells, prefix, ncells, &tx, &ty, &tz);
  gather_tiles_dmma_ad_body<R, WARPS>(tx, ty, tz, tile_start + bc.tile0, pairs, wtab, bc.sd,
                                      static_cast<const R*>(bc.out), part);
}

inline int blocks_for(long n, int threads) { return static_cast<int>((n + threads - 1) / threads); }

}  // namespace

namespace {
size_t axis_smem(int row, int atoms) { return sizeof(double) * atoms * axis_pitch(row); }

template <typename R>
void weights_bins(const MeshPlan& mp, const double4* s4s, int n, R* wtab, R* qk, int4* slot,
                  const PairBins& b, cudaStream_t st) {
  const StencilDims& sd = mp.sd;
  const int ntiles = sd.ntiles[0] * sd.ntiles[1] * sd.ntiles[2];
  const long items = static_cast<long>(n) * sd.S[0] * sd.S[1] * sd.S[2];
  if (sd.wstride <= kAxisRow) {
    const bool few = n <= (sd.kb ? kAxisFewBessel : kAxisFewGaussian);
    const int atoms = few ? kAxisFew : kAxisMany;
    launch_chained(few ? k_weights_axis<R, kAxisFew> : k_weights_axis<R, kAxisMany>,
                   blocks_for(n, atoms), 96, axis_smem(sd.wstride, atoms), st, s4s, n, sd, wtab, qk,
                   slot, b.counts, b.arrival);
    ++g_launches;
  } else {
    const long threads = static_cast<long>(sd.S[0] + sd.S[1] + sd.S[2]) * n;
    launch_chained(k_weights_tiled<R>, blocks_for(threads, 128), 128, 0, st, s4s, n, sd, wtab, qk,
                   slot);
    k_pair_count<<<blocks_for(items, 256), 256, 0, st>>>(slot, n, sd, b.counts, b.arrival);
    g_launches += 2;
  }
  launch_scan(b.counts, ntiles, b.starts, st);
  launch_chained(k_pair_scatter, blocks_for(items, 256), 256, 0, st, slot, n, sd, b.starts,
                 b.arrival, b.unordered);
  ++g_launches;
}
}  // namespace

void launch_weights_bins(const MeshPlan& mp, const double4* s4s, int n, void* wtab, void* qk,
                         int4* slot, const PairBins& b, cudaStream_t st) {
  if (n == 0) {
    const int ntiles = mp.sd.ntiles[0] * mp.sd.ntiles[1] * mp.sd.ntiles[2];
    cudaMemsetAsync(b.starts, 0, sizeof(int) * (ntiles + 1), st);
    return;
  }
  if (mp.mixed)
    weights_bins(mp, s4s, n, static_cast<float*>(wtab), static_cast<float*>(qk), slot, b, st);
  else
    weights_bins(mp, s4s, n, static_cast<double*>(wtab), static_cast<double*>(qk), slot, b, st);
}

void launch_spread(const MeshPlan& mp, const PairBins& b, const int4* slot, int n, bool ordered,
                   bool keep, const void* wtab, const void* qk, void* grid, cudaStream_t st) {
  const int ntiles = mp.sd.ntiles[0] * mp.sd.ntiles[1] * mp.sd.ntiles[2];
  const size_t items = static_cast<size_t>(n) * mp.sd.S[0] * mp.sd.S[1] * mp.sd.S[2];
  const bool cores = mp.mixed && mp.stencil == 2;
  const int* tile_start = b.starts;
  int2* pairs = b.pairs;
  const int2* unordered = ordered ? nullptr : b.unordered;
  if (n > 0 && !ordered && cores) {
    launch_chained(k_pair_rank, blocks_for(items, 256), 256, 0, st, unordered, tile_start, ntiles,
                   slot, mp.sd, pairs);
    ++g_launches;
    unordered = nullptr;
  }
  dim3 grd(mp.sd.ntiles[0], mp.sd.ntiles[1], mp.sd.ntiles[2]);
  if (cores)  // FP32 CUDA-core spread
    launch_chained(k_spread_tiles<float>, grd, kSpreadLanes, 0, st, tile_start, pairs,
                   static_cast<const float*>(wtab), static_cast<const float*>(qk), mp.sd,
                   static_cast<float*>(grid));
  else if (mp.mixed)  // FP32 weights and grid, FP64 products on the tensor cores
    launch_chained(ntiles > kSpreadFull ? k_spread_tiles_dmma<float, kSpreadFew>
                                        : k_spread_tiles_dmma<float, kSpreadMany>,
                   grd, 32, 0, st, tile_start, unordered, pairs, keep,
                   static_cast<const float*>(wtab), static_cast<const float*>(qk), mp.sd,
                   static_cast<float*>(grid));
  else
    launch_chained(ntiles > kSpreadFull ? k_spread_tiles_dmma<double, kSpreadFew>
                                        : k_spread_tiles_dmma<double, kSpreadMany>,
                   grd, 32, 0, st, tile_start, unordered, pairs, keep,
                   static_cast<const double*>(wtab), static_cast<const double*>(qk), mp.sd,
                   static_cast<double*>(grid));
  ++g_launches;
}

void launch_gather(const MeshPlan& mp, const int* tile_start, const int2* pairs, const void* wtab,
                   const void* grid, int nc, double* part, cudaStream_t st) {
  dim3 grd(mp.sd.ntiles[0], mp.sd.ntiles[1], mp.sd.ntiles[2]);
#define EWG_GATHER(R, NC)                                                                \
  launch_chained(k_gather_tiles<R, NC, GatherShape<R>::atoms, GatherShape<R>::warps>, grd,  \
                 32 * GatherShape<R>::warps, 0, st, tile_start, pairs,                       \
                 static_cast<const R*>(wtab), mp.sd, static_cast<const R*>(grid), part)
  const bool cores = mp.mixed && mp.stencil == 2;  // FP32 CUDA-core stencils
  if (mp.sd.ad && nc == 1) {  // force wanted, ad scheme: potential grid, four partials
    if (cores)
      launch_chained(k_gather_tiles_ad<kGatherAdF32Atoms, kGatherAdF32Warps>, grd,
                     32 * kGatherAdF32Warps, 0, st, tile_start, pairs,
                     static_cast<const float*>(wtab), mp.sd, static_cast<const float*>(grid), part);
    else if (mp.mixed)
      launch_chained(k_gather_tiles_dmma_ad<float, kGatherAdWarps>, grd, 32 * kGatherAdWarps, 0,
                     st, tile_start, pairs, static_cast<const float*>(wtab), mp.sd,
                     static_cast<const float*>(grid), part);
    else
      launch_chained(k_gather_tiles_dmma_ad<double, kGatherAdWarps>, grd, 32 * kGatherAdWarps, 0,
                     st, tile_start, pairs, static_cast<const double*>(wtab), mp.sd,
                     static_cast<const double*>(grid), part);
  } else if (cores) {
    if (nc == 4)
      EWG_GATHER(float, 4);
    else
      EWG_GATHER(float, 1);
  } else {
    // The kernel shape's warps per tile; every shape stages 64 atoms per round
    // (warps x blocks of 8 atoms per warp) and gives bitwise the same partials.
#define EWG_GATHER64(R, NC, WARPS, MB)                                                          \
  launch_chained(k_gather_tiles_dmma<R, NC, WARPS, MB>, grd, 32 * WARPS, 0, st, tile_start, pairs, \
                 static_cast<const R*>(wtab), mp.sd, static_cast<const R*>(grid), part)
#define EWG_GATHER64_SHAPES(R, NC)          \
  do {                                      \
    if (mp.gather_warps == 2)               \
      EWG_GATHER64(R, NC, 2, 4);            \
    else if (mp.gather_warps == 8)          \
      EWG_GATHER64(R, NC, 8, 1);            \
    else                                    \
      EWG_GATHER64(R, NC, kGatherWarps, kGatherMB); \
  } while (0)
    static_assert(kGatherWarps * kGatherMB == 8, "64 atoms per round");
    if (mp.mixed) {  // FP32 tiles and weights, FP64 products on the tensor cores
      if (nc == 4)
        EWG_GATHER64_SHAPES(float, 4);
      else
        EWG_GATHER64_SHAPES(float, 1);
    } else {
      if (nc == 4)
        EWG_GATHER64_SHAPES(double, 4);
      else
        EWG_GATHER64_SHAPES(double, 1);
    }
#undef EWG_GATHER64_SHAPES
#undef EWG_GATHER64
  }
#undef EWG_GATHER
  ++g_launches;
}

void launch_gather_final(const MeshPlan& mp, const int4* slot, const int* perm, const double* part,
                         int nparts, int n, const double* q, double self_coef, double pot_shift,
                         const double* pot_sr, const double* f_sr, double* pot, double* force,
                         const double (*rec)[3], cudaStream_t st) {
  if (n == 0) return;
  RecRows rr{};
  if (rec) {
    rr.on = 1;
    for (int i = 0; i < 3; ++i)
      for (int d = 0; d < 3; ++d) rr.b[i][d] = rec[i][d];
  }
  const bool narrow = mp.sd.S[0] * mp.sd.S[1] * mp.sd.S[2] <= 32;
  if (nparts == 4) {
    if (narrow)
      k_gather_final<4, 8><<<blocks_for(8L * n, 256), 256, 0, st>>>(
          slot, perm, part, n, mp.sd, q, self_coef, pot_shift, pot_sr, f_sr, pot, force, rr);
    else
      k_gather_final<4, 32><<<blocks_for(32L * n, 256), 256, 0, st>>>(
          slot, perm, part, n, mp.sd, q, self_coef, pot_shift, pot_sr, f_sr, pot, force, rr);
  } else {
    if (narrow)
      k_gather_final<1, 8><<<blocks_for(8L * n, 256), 256, 0, st>>>(
          slot, perm, part, n, mp.sd, q, self_coef, pot_shift, pot_sr, f_sr, pot, nullptr, rr);
    else
      k_gather_final<1, 32><<<blocks_for(32L * n, 256), 256, 0, st>>>(
          slot, perm, part, n, mp.sd, q, self_coef, pot_shift, pot_sr, f_sr, pot, nullptr, rr);
  }
  ++g_launches;
}

namespace {
template <typename R>
void weights_bins_seg(const BatchLaunch& b, const double4* s4s, R* wtab, R* qk, int4* slot,
                      const PairBins& pb, cudaStream_t st) {
  if (b.wstride <= kAxisRow) {
    const bool few = b.n_atoms <= (b.mixed ? kAxisFewGaussian : kAxisFewBessel);
    const int atoms = few ? kAxisFew : kAxisMany;
    launch_chained(few ? k_weights_axis_seg<R, kAxisFew> : k_weights_axis_seg<R, kAxisMany>,
                   blocks_for(b.n_atoms, atoms), 96, axis_smem(b.wstride, atoms), st, b.cells,
                   b.p_atoms, b.p_slots, b.ncells, b.n_atoms, b.wstride, b.pstride, s4s, wtab, qk,
                   slot, pb.counts, pb.arrival);
    ++g_launches;
  } else {
    launch_chained(k_weights_seg<R>, blocks_for(b.n_weights, 128), 128, 0, st, b.cells,
                   b.p_weights, b.ncells, b.n_weights, s4s, wtab, qk, slot);
    k_pair_count_seg<<<blocks_for(b.n_slots, 256), 256, 0, st>>>(
        b.cells, b.p_slots, b.ncells, b.n_slots, slot, pb.counts, pb.arrival);
    g_launches += 2;
  }
  launch_scan(pb.counts, b.n_tiles, pb.starts, st);
  launch_chained(k_pair_scatter_seg, blocks_for(b.n_slots, 256), 256, 0, st, b.cells, b.p_slots,
                 b.ncells, b.n_slots, slot, pb.starts, pb.arrival, pb.unordered);
  ++g_launches;
}
}  // namespace

void launch_weights_bins_seg(const BatchLaunch& b, const double4* s4s, void* wtab, void* qk,
                             int4* slot, const PairBins& pb, cudaStream_t st) {
  if (b.n_slots == 0) {
    cudaMemsetAsync(pb.starts, 0, sizeof(int) * (b.n_tiles + 1), st);
    return;
  }
  if (b.mixed)
    weights_bins_seg(b, s4s, static_cast<float*>(wtab), static_cast<float*>(qk), slot, pb, st);
  else
    weights_bins_seg(b, s4s, static_cast<double*>(wtab), static_cast<double*>(qk), slot, pb, st);
}

void launch_spread_seg(const BatchLaunch& b, const PairBins& pb, const void* wtab, const void* qk,
                       cudaStream_t st) {
  if (b.n_tiles == 0) return;
  const int* tile_start = pb.starts;
  int2* pairs = pb.pairs;
  const int2* unordered = pb.unordered;
  if (b.mixed)
    launch_chained(k_spread_tiles_dmma_seg<float, kSpreadFew>, b.n_tiles, 32, 0, st, b.cells,
                   b.p_tiles, b.ncells, tile_start, unordered, pairs, static_cast<const float*>(wtab),
                   static_cast<const float*>(qk));
  else
    launch_chained(k_spread_tiles_dmma_seg<double, kSpreadFew>, b.n_tiles, 32, 0, st, b.cells,
                   b.p_tiles, b.ncells, tile_start, unordered, pairs, static_cast<const double*>(wtab),
                   static_cast<const double*>(qk));
  ++g_launches;
}

void launch_gather_seg(const BatchLaunch& b, const int* tile_start, const int2* pairs,
                       const void* wtab, double* part, cudaStream_t st) {
  if (b.n_tiles == 0) return;
  const int nb = b.n_tiles;
  if (b.ad && b.nc == 1 && b.nparts == 4) {  // window-differentiated forces
    if (b.mixed)
      launch_chained(k_gather_tiles_dmma_ad_seg<float, kGatherAdWarps>, nb, 32 * kGatherAdWarps, 0,
                     st, b.cells, b.p_tiles, b.ncells, tile_start, pairs,
                     static_cast<const float*>(wtab), part);
    else
      launch_chained(k_gather_tiles_dmma_ad_seg<double, kGatherAdWarps>, nb, 32 * kGatherAdWarps,
                     0, st, b.cells, b.p_tiles, b.ncells, tile_start, pairs,
                     static_cast<const double*>(wtab), part);
  } else if (b.mixed) {
    const float* w = static_cast<const float*>(wtab);
    if (b.nc == 4)
      launch_chained(k_gather_tiles_dmma_seg<float, 4, kGatherWarps, kGatherMB>, nb,
                     32 * kGatherWarps, 0, st, b.cells, b.p_tiles, b.ncells, tile_start, pairs, w,
                     part);
    else
      launch_chained(k_gather_tiles_dmma_seg<float, 1, kGatherWarps, kGatherMB>, nb,
                     32 * kGatherWarps, 0, st, b.cells, b.p_tiles, b.ncells, tile_start, pairs, w,
                     part);
  } else {
    const double* w = static_cast<const double*>(wtab);
    if (b.nc == 4)
      launch_chained(k_gather_tiles_dmma_seg<double, 4, kGatherWarps, kGatherMB>, nb,
                     32 * kGatherWarps, 0, st, b.cells, b.p_tiles, b.ncells, tile_start, pairs, w,
                     part);
    else
      launch_chained(k_gather_tiles_dmma_seg<double, 1, kGatherWarps, kGatherMB>, nb,
                     32 * kGatherWarps, 0, st, b.cells, b.p_tiles, b.ncells, tile_start, pairs, w,
                     part);
  }
  ++g_launches;
}

void launch_gather_final_seg(const BatchLaunch& b, const int4* slot, const int* perm,
                             const double* part, const double* q, const double* pot_sr,
                             const double* f_sr, double* pot, double* force, cudaStream_t st) {
  if (b.n_atoms == 0) return;
  const int n = b.n_atoms;
  const int blocks = blocks_for(static_cast<long>(b.lpa) * n, 256);
#define EWG_FINAL(NC, LPA)                                                                   \
  k_gather_final_seg<NC, LPA><<<blocks, 256, 0, st>>>(b.cells, b.p_atoms, b.ncells, slot, perm, \
                                                      part, n, q, pot_sr, f_sr, pot,         \
                                                      NC == 4 ? force : nullptr)
  if (b.nparts == 4) {
    if (b.lpa == 8)
      EWG_FINAL(4, 8);
    else
      EWG_FINAL(4, 32);
  } else {
    if (b.lpa == 8)
      EWG_FINAL(1, 8);
    else
      EWG_FINAL(1, 32);
  }
#undef EWG_FINAL
  ++g_launches;
}

int stencil_configure_kernels() {
  const int rows = static_cast<int>(axis_smem(kAxisRow, kAxisMany));
  static_assert(8 * kAxisFew * axis_pitch(kAxisRow) <= 48 * 1024, "needs no larger limit");
  for (const void* k : {reinterpret_cast<const void*>(k_weights_axis<double, kAxisMany>),
                        reinterpret_cast<const void*>(k_weights_axis<float, kAxisMany>),
                        reinterpret_cast<const void*>(k_weights_axis_seg<double, kAxisMany>),
                        reinterpret_cast<const void*>(k_weights_axis_seg<float, kAxisMany>)})
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, rows);
  // The windows' polynomials, once per device: other contexts' kernels may be reading
  // them later.
  static std::mutex lock;
  static std::vector<bool> done;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return EWG_ERR_CUDA;
  const std::lock_guard<std::mutex> hold(lock);
  if (dev < static_cast<int>(done.size()) && done[dev]) return EWG_OK;
  double coef[kKbKinds * kKbWidth * kKbCoefs];
  for (int kb = 1; kb <= kKbKinds; ++kb)
    kb_polynomials(kb, coef + (kb - 1) * kKbWidth * kKbCoefs);
  if (cudaMemcpyToSymbol(c_kb, coef, sizeof(coef)) != cudaSuccess) return EWG_ERR_CUDA;
  if (dev >= static_cast<int>(done.size())) done.resize(dev + 1, false);
  done[dev] = true;
  return EWG_OK;
}

int measure_dmma_peak(cudaStream_t st, double* tflops) {
  int dev = 0, nsm = 0;
  cudaGetDevice(&dev);
  if (cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return EWG_ERR_CUDA;
  const int blocks = 4 * nsm, threads = 128, iters = 4096;
  cudaEvent_t e0, e1;
  if (cudaEventCreate(&e0) != cudaSuccess || cudaEventCreate(&e1) != cudaSuccess) return EWG_ERR_CUDA;
  k_dmma_peak<<<blocks, threads, 0, st>>>(iters / 8, 0.25, nullptr);  // warm-up
  cudaEventRecord(e0, st);
  k_dmma_peak<<<blocks, threads, 0, st>>>(iters, 0.25, nullptr);
  cudaEventRecord(e1, st);
  g_launches += 2;
  float ms = 0.0f;
  const bool ok = cudaEventSynchronize(e1) == cudaSuccess &&
                  cudaEventElapsedTime(&ms, e0, e1) == cudaSuccess && ms > 0.0f;
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (!ok) return EWG_ERR_CUDA;
  const double mmas = static_cast<double>(blocks) * (threads / 32) * iters * 8;
  *tflops = mmas * 2.0 * 8 * 8 * 4 / (ms * 1e-3) / 1e12;
  return EWG_OK;
}

}  // namespace ewg
