// Tile spreading, interpolation and ES-derivative gradient kernels.
//
// Work unit: a subproblem = up to `maxsub` consecutive sorted points of one bin.
// All of a bin's footprints lie in its padded tile (tile + ns - 1 cells per
// axis, periodic wrap applied only when the tile is read from / flushed to the
// fine grid), so each CTA works entirely in shared memory:
//
//  * spread (nufftax/core/spread.py:285-339, 435-494, 596-658; Pallas twin
//    nufftax/core/pallas_spread.py:337-613): 2D, and 3D widths up to 8, sum the
//    window of a block of neighbouring points in a warp's registers and send it
//    to the grid (nfx_spread_window.cuh).  The rest goes through a shared-memory
//    tile: cell by cell with shared-memory atomics on distinct addresses
//    (spread_subproblem_cells: 1D, and 3D of width 10 and more with points
//    denser than cells), or plane by plane without atomics
//    (spread_subproblem_owner: sparse 3D).  A finished tile is flushed with one
//    vectorised `red.global.add.v2.f32` per non-zero cell, coalesced along x.
//  * interp (nufftax/core/spread.py:342-381, 497-540, 661-709): the padded tile
//    is staged into shared memory with coalesced loads, then each thread
//    evaluates one point as a separable sum (x innermost); no atomics.
//  * grad (nufftax/core/spread.py:820-1305): the same staged tile, with the ES
//    derivative weights (dphi/dx = -phi'(z) nf / 2pi) for each axis, giving the
//    interpolated value and all coordinate gradients in one pass.
#pragma once


#include <algorithm>
#include <type_traits>

#include "nfx_internal.h"

namespace nfx {

template <int NS, int DIM>
struct Pow {
  static constexpr int value = NS * Pow<NS, DIM - 1>::value;
};
template <int NS>
struct Pow<NS, 0> {
  static constexpr int value = 1;
};

template <typename T>
struct PointArgs {
  const T* sc[3];  // folded coordinates in sorted order (SortView::coord); unused axes nullptr
  int64_t M;
  int n_trans;
  int64_t grid_stride;  // complex elements per transform of the fine grid
  int win_part;         // window spread: points of one work item; 0: an item is a subproblem
  int win_group;        // window spread: items that one takes together when their points share a block; 0: none
  int tma;              // 1: the interpolation stages interior tiles with the kernel's tensor map
  int* status;          // device status word (nonzero after a bounded wait gave up); set when tma = 1
  Geom g;
  T beta, kc;
  SortView s;
  EsPoly poly;
  std::conditional_t<sizeof(T) == 8, EsPolyD, char> polyd;  // double only
};

// The NS weights of one axis: w[q] = phi(i0 + q - xs).  float with a fitted
// polynomial: Horner in v = 2 (xs - i0) - (NS - 1) (exact in float: xs - i0 is
// exact because xs and i0 are within NS of each other and i0 is an integer),
// degree kPolyEvalDeg, each coefficient a fixed offset in the argument block
// (an operand of its FMA, no load).  double likewise, but the two edge weights
// by exp/sqrt: 10 DFMA a weight instead of about 55 double operations, which
// bound the complex128 kernels (2D, 200 k points, ns 14: spread 97 us, of them
// about two thirds the 28 weights of a point).  Otherwise exp/sqrt
// (nufftax/core/kernel.py:79-111).
template <typename T, int NS>
__device__ __forceinline__ void axis_weights(const PointArgs<T>& a, int i0, T xs, T* w) {
  if (std::is_same<T, float>::value && a.poly.deg > 0) {
    // weights q and NS - 1 - q from one even / odd split of polynomial q:
    // P(+-v) = E(v^2) +- v O(v^2)  (phi is even)
    static_assert(kPolyEvalDeg % 2 == 1, "odd evaluation degree: E and O of equal length");
    const float v = 2.0f * (float)(xs - (T)i0) - (float)(NS - 1);
    const float u = v * v;
    float e[NS / 2], o[NS / 2];
#pragma unroll
    for (int q = 0; q < NS / 2; ++q) {
      e[q] = a.poly.a[q][kPolyEvalDeg - 1];
      o[q] = a.poly.a[q][kPolyEvalDeg];
    }
#pragma unroll
    for (int d = kPolyEvalDeg - 3; d >= 0; d -= 2) {
#pragma unroll
      for (int q = 0; q < NS / 2; ++q) {
        e[q] = fmaf(e[q], u, a.poly.a[q][d]);
        o[q] = fmaf(o[q], u, a.poly.a[q][d + 1]);
      }
    }
#pragma unroll
    for (int q = 0; q < NS / 2; ++q) {
      w[q] = (T)fmaf(v, o[q], e[q]);
      w[NS - 1 - q] = (T)fmaf(-v, o[q], e[q]);
    }
    return;
  }
  if constexpr (sizeof(T) == 8 && NS >= 4) {
    if (a.polyd.deg > 0) {
      static_assert(kPolyEvalDegD % 2 == 1, "odd evaluation degree: E and O of equal length");
      const double v = 2.0 * (xs - (T)i0) - (double)(NS - 1);
      const double u = v * v;
#pragma unroll
      for (int q = 1; q < NS / 2; ++q) {
        double e = a.polyd.a[q - 1][kPolyEvalDegD - 1], o = a.polyd.a[q - 1][kPolyEvalDegD];
#pragma unroll
        for (int d = kPolyEvalDegD - 3; d >= 0; d -= 2) {
          e = fma(e, u, a.polyd.a[q - 1][d]);
          o = fma(o, u, a.polyd.a[q - 1][d + 1]);
        }
        w[q] = fma(v, o, e);
        w[NS - 1 - q] = fma(-v, o, e);
      }
      w[0] = es_weight(rn_sub((T)i0, xs), a.beta, a.kc);
      w[NS - 1] = es_weight(rn_sub((T)(i0 + NS - 1), xs), a.beta, a.kc);
      return;
    }
  }
#pragma unroll
  for (int q = 0; q < NS; ++q) w[q] = es_weight(rn_sub((T)(i0 + q), xs), a.beta, a.kc);
}

// End of the subproblem of bin b that starts at sorted position k0.
__device__ __forceinline__ int sub_end(const SortView& s, int b, int k0) {
  return k0 + min(s.maxsub, s.bin_start[b + 1] - k0);
}

__device__ __forceinline__ void bin_origin(const Geom& g, int b, int& o0, int& o1, int& o2) {
  int bx = b % g.nb[0];
  int r = b / g.nb[0];
  int by = r % g.nb[1];
  int bz = r / g.nb[1];
  o0 = bx * g.tile[0];
  o1 = by * g.tile[1];
  o2 = bz * g.tile[2];
}

__device__ __forceinline__ int wrap_up(int i, int n) {
  while (i >= n) i -= n;
  return i;
}

// Folded coordinate of axis d of the k-th sorted point (a coalesced read).
template <typename T>
__device__ __forceinline__ T sorted_coord(const PointArgs<T>& a, int d, int k) {
  return a.sc[d][k];
}

template <typename T>
__device__ __forceinline__ cplx_t<T> cmul(cplx_t<T> u, cplx_t<T> v) {
  cplx_t<T> r;
  r.x = u.x * v.x - u.y * v.y;
  r.y = u.x * v.y + u.y * v.x;
  return r;
}

// Type-3 sorts carry a complex factor per sorted point (SortView::extra): the
// spread multiplies it into the strength, the interpolation into its result.
template <typename T>
__device__ __forceinline__ cplx_t<T> with_extra(const PointArgs<T>& a, int k, cplx_t<T> v) {
  return a.s.extra != nullptr ? cmul<T>(v, reinterpret_cast<const cplx_t<T>*>(a.s.extra)[k]) : v;
}

// ---------------------------------------------------------------------------
// Spread
// ---------------------------------------------------------------------------

// Adds a finished padded tile (planar) into the fine grid, one vectorised red
// per non-zero cell: one warp per tile row, lanes along x (coalesced); periodic
// wrap applied here.
template <typename T>
__device__ __forceinline__ void flush_tile(const Geom& g, const int o[3], const T* s_re, const T* s_im,
                                           cplx_t<T>* __restrict__ out) {
  const int row = g.pitch;
  const int plane = g.pitch * g.pad[1];
  const int nrows = g.pad[1] * g.pad[2];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  for (int r = warp; r < nrows; r += nw) {
    const int ly = r % g.pad[1];
    const int lz = r / g.pad[1];
    const int gy = wrap_up(o[1] + ly, g.nf[1]);
    const int gz = wrap_up(o[2] + lz, g.nf[2]);
    cplx_t<T>* dst = out + ((int64_t)gz * g.nf[1] + gy) * g.nf[0];
    const T* sr = s_re + lz * plane + ly * row;
    const T* si = s_im + lz * plane + ly * row;
    for (int lx = lane; lx < g.pad[0]; lx += 32) {
      const T vr = sr[lx], vi = si[lx];
      if (vr != (T)0 || vi != (T)0) {
        cplx_t<T> v;
        v.x = vr;
        v.y = vi;
        red_add(dst + wrap_up(o[0] + lx, g.nf[0]), v);
      }
    }
  }
}

// From a point's folded coordinates xf (in [0, nf]), computes its tile offset
// and per-axis weights.  Returns false for a point outside its bin's tile (the
// folded coordinates come from the same sort as the bins, so this does not
// happen; the check keeps a corrupted workspace from indexing out of the tile).
template <typename T, int DIM, int NS>
__device__ __forceinline__ bool footprint(const PointArgs<T>& a, const T (&xf)[DIM], const int o[3], int row,
                                          int plane, int& off, T (&w)[DIM][NS]) {
  const Geom& g = a.g;
  bool inside = true;
  off = 0;
#pragma unroll
  for (int d = 0; d < DIM; ++d) {
    const T xs = xf[d];
    const int i0 = left_cell<T, NS>(xs);
    const int l = wrap_index(i0, g.nf[d]) - o[d];
    inside = inside && (unsigned)l < (unsigned)g.tile[d];
    off += l * (d == 0 ? 1 : (d == 1 ? row : plane));
    axis_weights<T, NS>(a, i0, xs, w[d]);
  }
  return inside;
}

template <typename T, int DIM>
__device__ __forceinline__ void load_sorted(const PointArgs<T>& a, int k, T (&xf)[DIM]) {
#pragma unroll
  for (int d = 0; d < DIM; ++d) xf[d] = sorted_coord(a, d, k);
}

template <typename T, int DIM, int NS>
__device__ __forceinline__ bool point_footprint(const PointArgs<T>& a, int k, const int o[3], int row, int plane,
                                                int& off, T (&w)[DIM][NS]) {
  T xf[DIM];
  load_sorted<T, DIM>(a, k, xf);
  return footprint<T, DIM, NS>(a, xf, o, row, plane, off, w);
}

// A 16-byte vector of T.
template <typename T>
struct Vec16;
template <>
struct Vec16<float> {
  using type = float4;
};
template <>
struct Vec16<double> {
  using type = double2;
};

}  // namespace nfx

#include "nfx_spread_window.cuh"

namespace nfx {

// Spread of one subproblem where no window exists (1D; 3D widths from 10).  Points
// are staged 32 at a time per warp (weights axis-major), then walked footprint cell
// by footprint cell with shared-memory atomics on distinct addresses within each
// instruction.
template <typename T, int DIM, int NS, int NW>
__device__ __forceinline__ void spread_subproblem_cells(const PointArgs<T>& a, const cplx_t<T>* __restrict__ c,
                                                        cplx_t<T>* __restrict__ fw, int sidx, unsigned char* smem_raw) {
  using CT = cplx_t<T>;
  static_assert(DIM == 1 || DIM == 3, "2D spreads by windows");
  constexpr int CELLS = Pow<NS, DIM>::value;
  constexpr int SW = NW * 32 + 1;  // staging stride: odd, so both the per-lane writes and
                                   // the per-point reads across q hit distinct banks
  const Geom& g = a.g;
  const int tile_cells = g.pad[2] * g.pad[1] * g.pitch;
  T* s_re = reinterpret_cast<T*>(smem_raw);
  T* s_im = s_re + tile_cells;
  T* s_w = s_im + tile_cells;          // [DIM*NS][SW]
  T* s_cr = s_w + DIM * NS * SW;       // [NW*32]
  T* s_ci = s_cr + NW * 32;            // [NW*32]
  int* s_off = reinterpret_cast<int*>(s_ci + NW * 32);  // [NW*32]
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int row = g.pitch;
  const int plane = g.pitch * g.pad[1];
  const int b = a.s.sub_bin[sidx];
  const int k0 = a.s.sub_start[sidx];
  const int k1 = sub_end(a.s, b, k0);
  int o[3];
  bin_origin(g, b, o[0], o[1], o[2]);
  for (int t = 0; t < a.n_trans; ++t) {
    for (int i = threadIdx.x; i < 2 * tile_cells; i += blockDim.x) s_re[i] = (T)0;
    __syncthreads();
    const int per = ((k1 - k0 + NW - 1) / NW + 31) / 32 * 32;
    const int w0 = k0 + min(warp * per, k1 - k0);
    const int w1 = w0 + min(per, k1 - w0);
    for (int kb = w0; (unsigned)kb < (unsigned)w1; kb += 32) {
      const int k = kb + lane;
      const int slot = warp * 32 + lane;
      if ((unsigned)k < (unsigned)w1) {
        const int p = a.s.perm[k];
        int off;
        T w[DIM][NS];
        const bool inside = point_footprint<T, DIM, NS>(a, k, o, row, plane, off, w);
#pragma unroll
        for (int d = 0; d < DIM; ++d)
#pragma unroll
          for (int q = 0; q < NS; ++q) s_w[(d * NS + q) * SW + slot] = w[d][q];
        const CT cv = with_extra(a, k, c[(int64_t)t * a.M + p]);
        s_off[slot] = inside ? off : 0;
        s_cr[slot] = inside ? cv.x : (T)0;
        s_ci[slot] = inside ? cv.y : (T)0;
      }
      __syncwarp();
      const int cnt = min(32, w1 - kb);
      if constexpr (DIM == 3) {
        // large footprints: one point at a time, straight to shared memory
        constexpr int R = (CELLS + 31) / 32;
        for (int j = 0; j < cnt; ++j) {
          const int sj = warp * 32 + j;
          const T cr = s_cr[sj], ci = s_ci[sj];
          const int off = s_off[sj];
#pragma unroll 4
          for (int r = 0; r < R; ++r) {
            const int q = lane + 32 * r;
            if (CELLS % 32 == 0 || q < CELLS) {
              const int kx = q % NS;
              const int ky = (q / NS) % NS;
              const int kz = q / (NS * NS);
              const T w = (s_w[(2 * NS + kz) * SW + sj] * s_w[(NS + ky) * SW + sj]) * s_w[kx * SW + sj];
              const int addr = off + kz * plane + ky * row + kx;
              atomicAdd(&s_re[addr], cr * w);
              atomicAdd(&s_im[addr], ci * w);
            }
          }
        }
      } else {
        // small footprints: several points per instruction
        const int items = cnt * CELLS;
        for (int it = lane; it < items; it += 32) {
          const int j = it / CELLS;
          const int kx = it - j * CELLS;
          const int sj = warp * 32 + j;
          const T w = s_w[kx * SW + sj];
          const int addr = s_off[sj] + kx;
          atomicAdd(&s_re[addr], s_cr[sj] * w);
          atomicAdd(&s_im[addr], s_ci[sj] * w);
        }
      }
      __syncwarp();
    }
    __syncthreads();
    flush_tile<T>(g, o, s_re, s_im, fw + (int64_t)t * a.grid_stride);
    __syncthreads();
  }
}

// Work items of a spread: slices of the sorted points (window spread) or
// subproblems.
template <typename T>
__device__ __forceinline__ int spread_items(const PointArgs<T>& a) {
  return a.win_part > 0 ? (int)((a.M + a.win_part - 1) / a.win_part) : *a.s.nsub;
}
// What spread_item needs of an item ahead of it (the ungrouped window spread).
template <typename T, int DIM, int NS>
__device__ __forceinline__ int item_keys(const PointArgs<T>& a, int item) {
  if constexpr (DIM == 2 && sizeof(T) == 4)
    return win_group_keys(a, item);
  else
    return 0;
}
template <typename T, int DIM, int NS, int NW>
__device__ __forceinline__ void spread_item(const PointArgs<T>& a, const cplx_t<T>* __restrict__ c,
                                            cplx_t<T>* __restrict__ fw, int item, int ahead,
                                            unsigned char* smem_raw) {
  if constexpr (WinShape<T, DIM, NS>::on) {
    spread_window<T, DIM, NS, NW>(a, c, fw, item, ahead, smem_raw);
  } else {
    spread_subproblem_cells<T, DIM, NS, NW>(a, c, fw, item, smem_raw);
  }
}

// CTAs per SM the spread's registers must allow for (0: the compiler's choice): the
// window's accumulators take them, a tile spread runs on its residency (1D, 2M points,
// ns 8: 177 us unbounded, 187 with the window's bounds, which let it have 56 registers
// instead of 40).
template <typename T, int DIM, int NS>
constexpr int spread_min_ctas() {
  if (!WinShape<T, DIM, NS>::on) return 0;
  return DIM == 3 || sizeof(T) == 8 ? 2 : (NS <= 8 ? 4 : 3);
}

template <typename T, int DIM, int NS, int NW>
__global__ void __launch_bounds__(NW * 32, spread_min_ctas<T, DIM, NS>()) k_spread(const __grid_constant__ PointArgs<T> a, const cplx_t<T>* __restrict__ c,
                                                    cplx_t<T>* __restrict__ fw) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const int nitems = spread_items(a);
  int ahead = (int)blockIdx.x < nitems ? item_keys<T, DIM, NS>(a, blockIdx.x) : 0;
  for (int item = blockIdx.x; item < nitems; item += gridDim.x) {
    const int keys = ahead;
    const int next = item + gridDim.x;
    if (next < nitems) ahead = item_keys<T, DIM, NS>(a, next);  // arrives while this item is spread
    spread_item<T, DIM, NS, NW>(a, c, fw, item, keys, smem_raw);
  }
}

// Plane-owner spread (3D, points sparser than cells).  The CTA stages up to
// NW*32 points at a time (every thread folds one point: c * w_x, y and z
// weights, its tile origin); then warp w adds every staged point into the
// tile planes z with z % NW == w, each plane's ns x ns cells spread over the
// lanes, with plain shared-memory read-add-write: a plane belongs to one warp,
// whose lanes touch distinct cells in each instruction, so no atomics are
// needed and every cell sums its points in sorted order.  With NW = ns every
// footprint (ns consecutive planes) gives each warp exactly one plane.  Slots
// are 16-byte aligned (owner_slot_reals): staged with 16-byte stores, read with
// 8-byte loads of (c w_x re, im), (offset, z) and pairs of y weights.
// The tile of the plane-owner spread holds interleaved complex cells (one
// 8- or 16-byte load and store per cell update).  Flushed like flush_tile.
template <typename T>
__device__ __forceinline__ void flush_tile_c(const Geom& g, const int o[3], const cplx_t<T>* s_tile,
                                             cplx_t<T>* __restrict__ out) {
  const int row = g.pitch;
  const int plane = g.pitch * g.pad[1];
  const int nrows = g.pad[1] * g.pad[2];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  for (int r = warp; r < nrows; r += nw) {
    const int ly = r % g.pad[1];
    const int lz = r / g.pad[1];
    const int gy = wrap_up(o[1] + ly, g.nf[1]);
    const int gz = wrap_up(o[2] + lz, g.nf[2]);
    cplx_t<T>* dst = out + ((int64_t)gz * g.nf[1] + gy) * g.nf[0];
    const cplx_t<T>* src = s_tile + lz * plane + ly * row;
    for (int lx = lane; lx < g.pad[0]; lx += 32) {
      const cplx_t<T> v = src[lx];
      if (v.x != (T)0 || v.y != (T)0) red_add(dst + wrap_up(o[0] + lx, g.nf[0]), v);
    }
  }
}

// A non-negative int carried in a real's bits (read back as the low int of the
// real's bytes).
template <typename T>
__device__ __forceinline__ T int_bits(int v) {
  if constexpr (sizeof(T) == 4)
    return __int_as_float(v);
  else
    return __longlong_as_double((long long)v);
}

// Row pitch (cells) of the plane-owner tile: at ns = 8 (complex64) lanes
// 0-15 of an update touch two rows 1 apart, so a pitch of 8 mod 16 cells puts
// their 64-byte segments in opposite halves of the banks; at ns = 4 the four
// rows of a half-warp need a pitch of 4 mod 8.  Other widths and complex128
// keep the tile's own pitch.
__host__ __device__ inline int owner_pitch(int pitch, int pad0, int ns, int real_bytes) {
  if (real_bytes != 4) return pitch;
  if (ns == 8) return pad0 + ((8 - pad0 % 16) + 16) % 16;
  if (ns == 4) return pad0 + ((4 - pad0 % 8) + 8) % 8;
  return pitch;
}

template <typename T, int NS, int NW>
__device__ __forceinline__ void spread_subproblem_owner(const PointArgs<T>& a, const cplx_t<T>* __restrict__ c,
                                                        cplx_t<T>* __restrict__ fw, int sidx,
                                                        unsigned char* smem_raw) {
  using CT = cplx_t<T>;
  using V16 = typename Vec16<T>::type;
  constexpr int R = 16 / (int)sizeof(T);  // reals per 16-byte vector
  static_assert((2 * NS) % R == 0, "c * w_x pairs fill whole vectors");
  constexpr int SLOT = owner_slot_reals((int)sizeof(T), NS);
  constexpr int YO = 2 * NS;                 // y weights
  constexpr int ZO = YO + owner_pad(NS, R);  // z weights
  constexpr int OO = ZO + owner_pad(NS, R);  // origin (offset, z) as raw int bits
  constexpr int NT = NW * 32;
  // cells of one footprint plane handled by this lane: column kx = lane % NS
  // and rows ky0 + i * LPR (i < IT): at NS = 8 one update touches rows
  // 0-3 (lanes 0-31), the next rows 4-7
  constexpr int LPR = 32 / NS;             // row blocks (lanes per column)
  constexpr int IT = (NS + LPR - 1) / LPR;  // rows per lane per plane
  // y weights in pair order (w_y[ky0], w_y[ky0 + LPR]) when a lane's two rows
  // are LPR apart and cover the NS rows exactly (NS = 8): one 8-byte load
  constexpr bool PAIRS = IT == 2 && 2 * LPR == NS;
  const Geom& g = a.g;
  const int tile_cells = g.pad[2] * g.pad[1] * g.pitch;
  CT* s_tile = reinterpret_cast<CT*>(smem_raw);
  T* s_st = reinterpret_cast<T*>(smem_raw) + owner_pad(2 * tile_cells, R);  // [NT][SLOT], 16-byte aligned
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int row = g.pitch;
  const int plane = g.pitch * g.pad[1];
  const int b = a.s.sub_bin[sidx];
  const int k0 = a.s.sub_start[sidx];
  const int k1 = sub_end(a.s, b, k0);
  int o[3];
  bin_origin(g, b, o[0], o[1], o[2]);
  const int kx = lane % NS;
  const int ky0 = lane / NS;
  const bool lane_on = ky0 < LPR;
  for (int t = 0; t < a.n_trans; ++t) {
    for (int i = threadIdx.x; i < tile_cells; i += blockDim.x) s_tile[i] = CT{(T)0, (T)0};
    for (unsigned kb = k0; kb < (unsigned)k1; kb += NT) {
      const unsigned k = kb + threadIdx.x;
      if (k < (unsigned)k1) {
        const int p = a.s.perm[k];
        T xv[3];
        load_sorted<T, 3>(a, k, xv);
        int off;
        T w[3][NS];
        const bool inside = footprint<T, 3, NS>(a, xv, o, row, plane, off, w);
        CT cv = with_extra(a, k, c[(int64_t)t * a.M + p]);
        if (!inside) {
          cv.x = cv.y = (T)0;
          off = 0;
        }
        T v[SLOT];
#pragma unroll
        for (int i = 0; i < SLOT; ++i) v[i] = (T)0;
#pragma unroll
        for (int q = 0; q < NS; ++q) {
          v[2 * q] = cv.x * w[0][q];
          v[2 * q + 1] = cv.y * w[0][q];
          v[ZO + q] = w[2][q];
        }
#pragma unroll
        for (int q = 0; q < NS; ++q) {
          if constexpr (PAIRS)
            v[YO + 2 * (q % LPR) + q / LPR] = w[1][q];
          else
            v[YO + q] = w[1][q];
        }
        v[OO] = int_bits<T>(off);
        v[OO + 1] = int_bits<T>(off / plane);  // z of the footprint origin in the tile
        V16* sp = reinterpret_cast<V16*>(s_st + threadIdx.x * SLOT);
#pragma unroll
        for (int i = 0; i < SLOT / R; ++i) {
          V16 u;
          if constexpr (R == 4) {
            u.x = v[4 * i];
            u.y = v[4 * i + 1];
            u.z = v[4 * i + 2];
            u.w = v[4 * i + 3];
          } else {
            u.x = v[2 * i];
            u.y = v[2 * i + 1];
          }
          sp[i] = u;
        }
      }
      __syncthreads();  // also orders the tile zeroing before the first adds
      const int cnt = min(NT, k1 - (int)kb);
      static_assert((NW & (NW - 1)) == 0, "warps per CTA a power of two");
      // planes of each footprint this warp owns: dz0 + pl * NW < NS, at most
      // ceil(NS / NW) (exactly NS / NW when NW divides NS)
      constexpr int PLANES = (NS + NW - 1) / NW;
      for (int j = 0; j < cnt; ++j) {
        const T* sp = s_st + j * SLOT;
        int off, oz;
        if constexpr (sizeof(T) == 4) {
          const int2 so = *reinterpret_cast<const int2*>(sp + OO);  // 8-byte aligned: OO is a multiple of 4
          off = so.x;
          oz = so.y;
        } else {
          const int* so = reinterpret_cast<const int*>(sp + OO);
          off = so[0];
          oz = so[2];
        }
        const int dz0 = (warp - oz) & (NW - 1);
#pragma unroll
        for (int pl = 0; pl < PLANES; ++pl) {
          const int dz = dz0 + pl * NW;
          if (NS % NW != 0 && dz >= NS) break;
          const T wz = sp[ZO + dz];
          const int base = off + dz * plane + kx;
          const CT cx = *reinterpret_cast<const CT*>(sp + 2 * kx);  // c * w_x[kx]
          if (lane_on) {
            T wyr[IT];
            if constexpr (PAIRS) {
              const CT pr = *reinterpret_cast<const CT*>(sp + YO + 2 * ky0);
              wyr[0] = pr.x;
              wyr[1] = pr.y;
            } else {
#pragma unroll
              for (int i = 0; i < IT; ++i) wyr[i] = ky0 + i * LPR < NS ? sp[YO + ky0 + i * LPR] : (T)0;
            }
#pragma unroll
            for (int i = 0; i < IT; ++i) {
              const int ky = ky0 + i * LPR;
              if (ky < NS) {
                const T wy = wz * wyr[i];
                CT* cell = s_tile + base + ky * row;
                CT u = *cell;
                u.x += wy * cx.x;
                u.y += wy * cx.y;
                *cell = u;
              }
            }
          }
        }
      }
      __syncthreads();
    }
    flush_tile_c<T>(g, o, s_tile, fw + (int64_t)t * a.grid_stride);
    __syncthreads();
  }
}

template <typename T, int NS, int NW>
__global__ void __launch_bounds__(NW * 32) k_spread_owner(PointArgs<T> a, const cplx_t<T>* __restrict__ c,
                                                          cplx_t<T>* __restrict__ fw) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const int nsub = *a.s.nsub;
  for (int sidx = blockIdx.x; sidx < nsub; sidx += gridDim.x)
    spread_subproblem_owner<T, NS, NW>(a, c, fw, sidx, smem_raw);
}

// ---------------------------------------------------------------------------
// Stage a padded tile of one transform's grid into shared memory (interleaved).
// ---------------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ void stage_tile(const Geom& g, const int o[3], const cplx_t<T>* __restrict__ grid,
                                           cplx_t<T>* s_tile) {
  const int row = g.pitch;
  const int plane = g.pitch * g.pad[1];
  const int nrows = g.pad[1] * g.pad[2];
  // one warp per row, lanes along x: coalesced
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  for (int r = warp; r < nrows; r += nw) {
    const int ly = r % g.pad[1];
    const int lz = r / g.pad[1];
    const int gy = wrap_up(o[1] + ly, g.nf[1]);
    const int gz = wrap_up(o[2] + lz, g.nf[2]);
    const cplx_t<T>* src = grid + ((int64_t)gz * g.nf[1] + gy) * g.nf[0];
    cplx_t<T>* dst = s_tile + lz * plane + ly * row;
    for (int lx = lane; lx < g.pad[0]; lx += 32) dst[lx] = src[wrap_up(o[0] + lx, g.nf[0])];
  }
}

// ---------------------------------------------------------------------------
// Tile staging by TMA.  The interpolation's padded tile of a bin whose padded
// extent lies inside the grid on every axis (no periodic wrap) is one box of
// the fine grid: one thread issues a cp.async.bulk.tensor load of it from the
// kernel's tensor map (this GPU's own grid, no multicast) into the tile
// buffer, completing on an mbarrier; the others wait on the barrier.  Tiles
// that wrap keep the plain loads (stage_tile).  Box (pitch, pad_y[, pad_z], 1)
// of elements of 8 bytes (complex64; complex128 as two), coordinates
// (x, y[, z], transform), so the box lands with the tile's own row pitch.
// The barrier wait is bounded (kTmaWaitPolls polls and kTmaWaitNs of the
// global timer, whichever ends first): a wait that gives up records
// NFX_STATUS_TMA_TIMEOUT in the status word (nfx_device_status) and the CTA
// stops, so a copy that never lands cannot hang the GPU.
// ---------------------------------------------------------------------------
constexpr int kTmaWaitPolls = 1 << 24;
constexpr unsigned long long kTmaWaitNs = 500000000ull;  // 0.5 s

struct TmaStage {
  const CUtensorMap* map;
  unsigned mbar;   // shared-memory address of the barrier
  unsigned phase;  // parity of the next completion
};

__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void tma_init(uint64_t* mbar) {
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(mbar)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
}

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ bool tma_wait(unsigned mbar, unsigned phase) {
  const unsigned long long t0 = global_ns();
  for (int it = 0; it < kTmaWaitPolls; ++it) {
    unsigned done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(done)
        : "r"(mbar), "r"(phase)
        : "memory");
    if (done) return true;
    if ((it & 255) == 255 && global_ns() - t0 > kTmaWaitNs) break;
  }
  return false;
}

// Stages transform t's padded tile at origin o into s_tile: by TMA when
// allowed, the tile does not wrap and the buffer is 128-byte aligned, else with
// plain loads.  Must be called by every thread of the CTA between barriers;
// false (for every thread) when a TMA wait gave up, and the caller then stops.
template <typename T>
__device__ __forceinline__ bool stage_interp_tile(const PointArgs<T>& a, const int o[3], const cplx_t<T>* grid, int t,
                                                  cplx_t<T>* s_tile, TmaStage& ts) {
  const Geom& g = a.g;
  const bool interior = a.tma && o[0] + g.pitch <= g.nf[0] && o[1] + g.pad[1] <= g.nf[1] &&
                        (g.dim < 3 || o[2] + g.pad[2] <= g.nf[2]) && (smem_addr(s_tile) & 127u) == 0;
  if (!interior) {
    stage_tile<T>(g, o, grid + (int64_t)t * a.grid_stride, s_tile);
    return true;
  }
  if (threadIdx.x == 0) {
    const unsigned bytes = (unsigned)(sizeof(cplx_t<T>) * g.pitch * g.pad[1] * g.pad[2]);
    const int x = o[0] * (int)(sizeof(cplx_t<T>) / 8);  // in 8-byte elements
    const uint64_t map = reinterpret_cast<uint64_t>(ts.map);
    const unsigned dst = smem_addr(s_tile);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // earlier reads of the buffer before the async write
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(ts.mbar), "r"(bytes) : "memory");
    if (g.dim == 2)
      asm volatile(
          "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
          "[%5];" ::"r"(dst),
          "l"(map), "r"(x), "r"(o[1]), "r"(t), "r"(ts.mbar)
          : "memory");
    else
      asm volatile(
          "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, "
          "%5}], [%6];" ::"r"(dst),
          "l"(map), "r"(x), "r"(o[1]), "r"(o[2]), "r"(t), "r"(ts.mbar)
          : "memory");
  }
  const bool landed = tma_wait(ts.mbar, ts.phase);
  ts.phase ^= 1u;
  if (__syncthreads_and(landed)) return true;
  if (threadIdx.x == 0) atomicOr(a.status, NFX_STATUS_TMA_TIMEOUT);
  return false;
}

// ---------------------------------------------------------------------------
// Interpolation with one lane group per point (2D and 3D).  GL lanes (the power
// of two >= NS) share a point: lane kx = lane % GL reads footprint column kx of
// every row (ky, or (ky, kz) in 3D).  The 32 / GL points of one warp
// instruction are consecutive in cell order, so their rows overlap in shared
// memory (few wavefronts; thread-per-point reads of 32 scattered footprints
// conflict on many of theirs).  Each lane computes only its own column's weight
// per axis; the other axes' weights reach the group's lanes by shuffles, and the
// group sums its columns with a butterfly of shuffles.
// ---------------------------------------------------------------------------
template <int NS>
__host__ __device__ constexpr int group_lanes() {
  return NS <= 4 ? 4 : (NS <= 8 ? 8 : 16);
}

// Weight q of one axis: float as axis_weights for that q (cq = the polynomial
// coefficients of q when the polynomial is in use), double by exp/sqrt.
template <typename T, int NS>
__device__ __forceinline__ T axis_weight_q(const PointArgs<T>& a, const float (&cq)[kPolyEvalDeg + 1], int i0, T xs,
                                           int q) {
  if (std::is_same<T, float>::value && a.poly.deg > 0) {
    const float v = 2.0f * (float)(xs - (T)i0) - (float)(NS - 1);
    float h = cq[kPolyEvalDeg];
#pragma unroll
    for (int d = kPolyEvalDeg - 1; d >= 0; --d) h = fmaf(h, v, cq[d]);
    return (T)h;
  }
  return es_weight(rn_sub((T)(i0 + q), xs), a.beta, a.kc);
}

// Left cells and tile offset of a point with folded coordinates xv (false:
// outside its bin's tile, see footprint).
template <typename T, int DIM, int NS>
__device__ __forceinline__ bool group_point(const PointArgs<T>& a, const T (&xv)[3], const int o[3], int row,
                                            int plane, int& off, T (&xs)[3], int (&i0)[3]) {
  const Geom& g = a.g;
  bool inside = true;
  off = 0;
#pragma unroll
  for (int d = 0; d < DIM; ++d) {
    xs[d] = xv[d];
    i0[d] = left_cell<T, NS>(xs[d]);
    const int l = wrap_index(i0[d], g.nf[d]) - o[d];
    inside = inside && (unsigned)l < (unsigned)g.tile[d];
    off += l * (d == 0 ? 1 : (d == 1 ? row : plane));
  }
  return inside;
}

// One round of 32 points for a warp: lane L takes point kb + L (left cells,
// tile offset; off = -1 outside the tile); the lane groups then take the
// points PPW at a time by shuffles (group_take).  The loads are pipelined
// across rounds: the next round's permutation entries and folded coordinates
// (both read in sorted order) are in flight while a round is processed.
template <typename T>
struct WarpPoints {
  int p, off;
  T xs[3];
  int i0[3];
};

__device__ __forceinline__ int round_perm(const SortView& s, int kb, int k1) {
  const int k = kb + (threadIdx.x & 31);
  return (unsigned)k < (unsigned)k1 ? s.perm[k] : -1;  // kb may be past the last position (and int)
}

template <typename T, int DIM>
__device__ __forceinline__ void round_coords(const PointArgs<T>& a, int kb, int k1, T (&xv)[3]) {
  const int k = kb + (threadIdx.x & 31);
#pragma unroll
  for (int d = 0; d < 3; ++d) xv[d] = (d < DIM && (unsigned)k < (unsigned)k1) ? sorted_coord(a, d, k) : (T)0;
}

template <typename T, int DIM, int NS>
__device__ __forceinline__ WarpPoints<T> warp_points(const PointArgs<T>& a, int p, const T (&xv)[3], const int o[3],
                                                     int row, int plane) {
  WarpPoints<T> w;
  w.p = p >= 0 ? p : 0;
  w.off = -1;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    w.xs[d] = (T)0;
    w.i0[d] = 0;
  }
  if (p >= 0) {
    int off;
    const bool inside = group_point<T, DIM, NS>(a, xv, o, row, plane, off, w.xs, w.i0);
    w.off = inside ? off : -1;
  }
  return w;
}

template <typename T, int DIM>
__device__ __forceinline__ WarpPoints<T> group_take(const WarpPoints<T>& w, int src) {
  constexpr unsigned kAll = 0xffffffffu;
  WarpPoints<T> r;
  r.p = __shfl_sync(kAll, w.p, src);
  r.off = __shfl_sync(kAll, w.off, src);
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    r.xs[d] = d < DIM ? __shfl_sync(kAll, w.xs[d], src) : (T)0;
    r.i0[d] = d < DIM ? __shfl_sync(kAll, w.i0[d], src) : 0;
  }
  return r;
}

template <typename T, int DIM, int NS, int NW>
__device__ __forceinline__ void interp_group(const PointArgs<T>& a, const cplx_t<T>* __restrict__ fw,
                                             cplx_t<T>* __restrict__ cout, int sidx, unsigned char* smem_raw,
                                             TmaStage& ts) {
  using CT = cplx_t<T>;
  constexpr int GL = group_lanes<NS>();
  constexpr int PPW = 32 / GL;
  constexpr unsigned kAll = 0xffffffffu;
  CT* s_tile = reinterpret_cast<CT*>(smem_raw);
  const Geom& g = a.g;
  const int row = g.pitch;
  const int plane = g.pitch * g.pad[1];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int kx = lane % GL;
  const int leader = lane - kx;
  const bool col_on = kx < NS;
  float cq[kPolyEvalDeg + 1];  // this lane's coefficients (constant-indexed parameter reads)
#pragma unroll
  for (int d = 0; d <= kPolyEvalDeg; ++d) cq[d] = a.poly.a[0][d];
#pragma unroll
  for (int q = 1; q < NS; ++q) {
    if (kx == q) {
#pragma unroll
      for (int d = 0; d <= kPolyEvalDeg; ++d) cq[d] = a.poly.a[q][d];
    }
  }
  const int b = a.s.sub_bin[sidx];
  const int k0 = a.s.sub_start[sidx];
  const int k1 = sub_end(a.s, b, k0);
  int o[3];
  bin_origin(g, b, o[0], o[1], o[2]);
  for (int t = 0; t < a.n_trans; ++t) {
    __syncthreads();
    if (!stage_interp_tile<T>(a, o, fw, t, s_tile, ts)) return;
    __syncthreads();
    constexpr int kStep = NW * 32;
    int p_cur = round_perm(a.s, k0 + warp * 32, k1);
    T x_cur[3];
    round_coords<T, DIM>(a, k0 + warp * 32, k1, x_cur);
    for (unsigned kb = k0 + warp * 32; kb < (unsigned)k1; kb += kStep) {  // warp-uniform
      const int p_next = round_perm(a.s, kb + kStep, k1);
      T x_next[3];
      round_coords<T, DIM>(a, kb + kStep, k1, x_next);
      const WarpPoints<T> wp = warp_points<T, DIM, NS>(a, p_cur, x_cur, o, row, plane);
      p_cur = p_next;
#pragma unroll
      for (int d = 0; d < 3; ++d) x_cur[d] = x_next[d];
      const int npts = min(32, k1 - (int)kb);
      for (int j0 = 0; j0 < npts; j0 += PPW) {
        const int j = j0 + lane / GL;
        const bool valid = j < npts;
        const WarpPoints<T> pt = group_take<T, DIM>(wp, valid ? j : 0);
        const bool on = col_on && pt.off >= 0;
        const T wx = axis_weight_q<T, NS>(a, cq, pt.i0[0], pt.xs[0], kx);
        const T wyq = axis_weight_q<T, NS>(a, cq, pt.i0[1], pt.xs[1], kx);
        T wy[NS];
#pragma unroll
        for (int q = 0; q < NS; ++q) wy[q] = __shfl_sync(kAll, wyq, leader + q);
        CT s;
        s.x = s.y = (T)0;
        if constexpr (DIM == 3) {
          const T wzq = axis_weight_q<T, NS>(a, cq, pt.i0[2], pt.xs[2], kx);
          T wz[NS];
#pragma unroll
          for (int q = 0; q < NS; ++q) wz[q] = __shfl_sync(kAll, wzq, leader + q);
          if (on) {
            const CT* base = s_tile + pt.off + kx;
            // one independent accumulator per z plane: NS chains in flight
            CT acc[NS];
#pragma unroll
            for (int kz = 0; kz < NS; ++kz) acc[kz].x = acc[kz].y = (T)0;
#pragma unroll
            for (int ky = 0; ky < NS; ++ky) {
#pragma unroll
              for (int kz = 0; kz < NS; ++kz) acc[kz] = fma2(splat2(wy[ky]), base[kz * plane + ky * row], acc[kz]);
            }
#pragma unroll
            for (int kz = 0; kz < NS; ++kz) s = fma2(splat2(wz[kz]), acc[kz], s);
          }
        } else {
          if (on) {
            const CT* base = s_tile + pt.off + kx;
            CT s1;
            s1.x = s1.y = (T)0;  // two chains
#pragma unroll
            for (int ky = 0; ky < NS; ky += 2) {
              s = fma2(splat2(wy[ky]), base[ky * row], s);
              s1 = fma2(splat2(wy[ky + 1]), base[(ky + 1) * row], s1);
            }
            s.x += s1.x;
            s.y += s1.y;
          }
        }
        T sr = on ? s.x * wx : (T)0, si = on ? s.y * wx : (T)0;
#pragma unroll
        for (int m = GL / 2; m >= 1; m >>= 1) {
          sr += __shfl_xor_sync(kAll, sr, m);
          si += __shfl_xor_sync(kAll, si, m);
        }
        if (valid && kx == 0) {
          CT r;
          r.x = sr;
          r.y = si;
          cout[(int64_t)t * a.M + pt.p] = with_extra(a, kb + j, r);
        }
      }
    }
  }
}

// ---------------------------------------------------------------------------
// Interp
// ---------------------------------------------------------------------------
// Threads per point of the interpolation: one lane group (the 3D default) or
// one thread.  MODE is the variant compiled into a kernel (NFX_PER_POINT_GROUP
// or _THREAD), or NFX_PER_POINT_AUTO to choose per problem at run time from
// Geom::interp_mode (the batched kernel).
template <int DIM>
__host__ __device__ __forceinline__ bool interp_by_group(int mode) {
  return DIM >= 2 && (mode == NFX_PER_POINT_GROUP || (mode == NFX_PER_POINT_AUTO && DIM == 3));
}

template <typename T, int DIM, int NS, int NW, int MODE = NFX_PER_POINT_AUTO>
__device__ __forceinline__ void interp_subproblem(const PointArgs<T>& a, const cplx_t<T>* __restrict__ fw,
                                                  cplx_t<T>* __restrict__ cout, int sidx, unsigned char* smem_raw,
                                                  TmaStage& ts) {
  using CT = cplx_t<T>;
  if constexpr (DIM >= 2 && MODE != NFX_PER_POINT_THREAD) {
    if (MODE == NFX_PER_POINT_GROUP || interp_by_group<DIM>(a.g.interp_mode)) {
      interp_group<T, DIM, NS, NW>(a, fw, cout, sidx, smem_raw, ts);
      return;
    }
  }
  CT* s_tile = reinterpret_cast<CT*>(smem_raw);
  const Geom& g = a.g;
  const int row = g.pitch;
  const int plane = g.pitch * g.pad[1];
  {
    const int b = a.s.sub_bin[sidx];
    const int k0 = a.s.sub_start[sidx];
    const int k1 = sub_end(a.s, b, k0);
    int o[3];
    bin_origin(g, b, o[0], o[1], o[2]);
    for (int t = 0; t < a.n_trans; ++t) {
      __syncthreads();
      if (!stage_interp_tile<T>(a, o, fw, t, s_tile, ts)) return;
      __syncthreads();
      // loads pipelined across iterations: the next iteration's permutation
      // entry and folded coordinates (both in sorted order)
      const int kStep = blockDim.x;
      int k = k0 + threadIdx.x;
      int p_cur = (unsigned)k < (unsigned)k1 ? a.s.perm[k] : 0;
      T x_cur[DIM];
#pragma unroll
      for (int d = 0; d < DIM; ++d) x_cur[d] = (unsigned)k < (unsigned)k1 ? sorted_coord(a, d, k) : (T)0;
      for (; (unsigned)k < (unsigned)k1; k += kStep) {
        const int p = p_cur;
        T xv[DIM];
#pragma unroll
        for (int d = 0; d < DIM; ++d) xv[d] = x_cur[d];
        {
          const bool more = position_before(k, kStep, k1);
          p_cur = more ? a.s.perm[k + kStep] : 0;
#pragma unroll
          for (int d = 0; d < DIM; ++d) x_cur[d] = more ? sorted_coord(a, d, k + kStep) : (T)0;
        }
        T w[DIM][NS];
        int off = 0;
        bool inside = true;
#pragma unroll
        for (int d = 0; d < DIM; ++d) {
          const T xs = xv[d];
          const int i0 = left_cell<T, NS>(xs);
          const int l = wrap_index(i0, g.nf[d]) - o[d];
          inside = inside && (unsigned)l < (unsigned)g.tile[d];
          off += l * (d == 0 ? 1 : (d == 1 ? row : plane));
          axis_weights<T, NS>(a, i0, xs, w[d]);
        }
        if (!inside) {  // stale sort: see k_spread
          CT zero;
          zero.x = zero.y = (T)0;
          cout[(int64_t)t * a.M + p] = zero;
          continue;
        }
        T ar = 0, ai = 0;
        const CT* base = s_tile + off;
        CT wxp[NS];  // (w_x, w_x) pairs, built once per point
#pragma unroll
        for (int kx = 0; kx < NS; ++kx) wxp[kx] = splat2(w[0][kx]);
#pragma unroll 1
        for (int kz = 0; kz < (DIM == 3 ? NS : 1); ++kz) {
          T zr = 0, zi = 0;
#pragma unroll
          for (int ky = 0; ky < (DIM >= 2 ? NS : 1); ++ky) {
            const CT* rp = base + kz * plane + ky * row;
            CT xa;
            xa.x = xa.y = (T)0;
#pragma unroll
            for (int kx = 0; kx < NS; ++kx) xa = fma2(wxp[kx], rp[kx], xa);
            const T xr = xa.x, xi = xa.y;
            if (DIM >= 2) {
              zr += xr * w[DIM >= 2 ? 1 : 0][ky];
              zi += xi * w[DIM >= 2 ? 1 : 0][ky];
            } else {
              zr += xr;
              zi += xi;
            }
          }
          if (DIM == 3) {
            ar += zr * w[DIM - 1][kz];
            ai += zi * w[DIM - 1][kz];
          } else {
            ar += zr;
            ai += zi;
          }
        }
        CT r;
        r.x = ar;
        r.y = ai;
        cout[(int64_t)t * a.M + p] = with_extra(a, k, r);
      }
    }
  }
}

// CTAs per SM the interpolation's registers must allow for (0: the compiler's
// choice).  The polynomial weights gave complex128 in 2D 148 registers and more from
// ns 12, one CTA an SM, which shows where few points a bin wait for their tiles: ns
// 14 on 512^2, us by exp/sqrt, one CTA, two: 5 k points 19.5, 25.6, 17.4; 500 k 107,
// 100, 82; 3M 506, 444, 363 (the spills it costs are small beside that).
template <typename T, int DIM, int NS, int MODE>
constexpr int interp_min_ctas() {
  return sizeof(T) == 8 && DIM == 2 && NS >= 12 && MODE == NFX_PER_POINT_THREAD ? 2 : 0;
}

template <typename T, int DIM, int NS, int NW, int MODE>
__global__ void __launch_bounds__(NW * 32, interp_min_ctas<T, DIM, NS, MODE>()) k_interp(PointArgs<T> a, const cplx_t<T>* __restrict__ fw,
                                                    cplx_t<T>* __restrict__ cout, const __grid_constant__ CUtensorMap tmap) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t mbar;
  TmaStage ts{&tmap, smem_addr(&mbar), 0u};
  if (a.tma) tma_init(&mbar);
  const int nsub = *a.s.nsub;
  for (int sidx = blockIdx.x; sidx < nsub; sidx += gridDim.x)
    interp_subproblem<T, DIM, NS, NW, MODE>(a, fw, cout, sidx, smem_raw, ts);
}

// ---------------------------------------------------------------------------
// Batched launches: many problems (own points, grid, tiling and sort) in one
// persistent launch.  `items` is a device table; `sub_prefix[p]` is the number
// of work items of problems < p (k_batch_prefix; slices of the sorted points or
// subproblems), so the CTAs walk one global work queue of (problem, item) pairs.
// ---------------------------------------------------------------------------
template <typename T>
struct BatchItem {
  PointArgs<T> a;
  const void* src;  // spread: strengths; interp: fine grid
  void* dst;        // spread: fine grid (zeroed by the caller); interp: values
};

__device__ __forceinline__ int batch_find(const int* __restrict__ prefix, int n, int g) {
  int lo = 0, hi = n;  // largest p with prefix[p] <= g
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (prefix[mid] <= g)
      lo = mid;
    else
      hi = mid;
  }
  return lo;
}

// CTAs per SM the batched spread's registers must allow for (0: the compiler's
// choice): as the plain spread's where a window exists.
template <typename T, int DIM, int NS>
constexpr int batch_min_ctas() {
  return WinShape<T, DIM, NS>::on ? spread_min_ctas<T, DIM, NS>() : 0;
}

template <typename T, int DIM, int NS, int NW>
__global__ void __launch_bounds__(NW * 32, batch_min_ctas<T, DIM, NS>())
    k_spread_batch(const BatchItem<T>* __restrict__ items, int nitems, const int* __restrict__ sub_prefix) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const int total = sub_prefix[nitems];
  for (int gi = blockIdx.x; gi < total; gi += gridDim.x) {
    const int p = batch_find(sub_prefix, nitems, gi);
    const BatchItem<T>& it = items[p];
    const int item = gi - sub_prefix[p];
    spread_item<T, DIM, NS, NW>(it.a, (const cplx_t<T>*)it.src, (cplx_t<T>*)it.dst, item,
                                item_keys<T, DIM, NS>(it.a, item), smem_raw);
    __syncthreads();
  }
}

template <typename T, int DIM, int NS, int NW>
__global__ void __launch_bounds__(NW * 32) k_interp_batch(const BatchItem<T>* __restrict__ items, int nitems,
                                                          const int* __restrict__ sub_prefix) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const int total = sub_prefix[nitems];
  TmaStage ts{nullptr, 0u, 0u};  // batched items stage with plain loads (their PointArgs have tma = 0)
  for (int gi = blockIdx.x; gi < total; gi += gridDim.x) {
    const int p = batch_find(sub_prefix, nitems, gi);
    const BatchItem<T>& it = items[p];
    interp_subproblem<T, DIM, NS, NW>(it.a, (const cplx_t<T>*)it.src, (cplx_t<T>*)it.dst, gi - sub_prefix[p],
                                      smem_raw, ts);
  }
}

// ---------------------------------------------------------------------------
// Gradient pass with one lane group per point (3D; layout as interp_group): lane
// kx reads footprint column kx of every (ky, kz) once and uses it for the value
// and all three derivative sums.  A thread per point reads 32 scattered
// footprints at a time, and the bank conflicts of those were 54 % of its
// shared-memory wavefronts, which bound it (88 % of that roof).
// ---------------------------------------------------------------------------
template <typename T, int NS, int NW>
__device__ __forceinline__ bool grad_group(const PointArgs<T>& a, const cplx_t<T>* __restrict__ G,
                                           const cplx_t<T>* __restrict__ V, cplx_t<T>* __restrict__ out_interp,
                                           T* __restrict__ dx, T* __restrict__ dy, T* __restrict__ dz, int sidx,
                                           unsigned char* smem_raw, TmaStage& ts) {
  using CT = cplx_t<T>;
  constexpr int GL = group_lanes<NS>();
  constexpr int PPW = 32 / GL;
  constexpr unsigned kAll = 0xffffffffu;
  CT* s_tile = reinterpret_cast<CT*>(smem_raw);
  const Geom& g = a.g;
  const int row = g.pitch;
  const int plane = g.pitch * g.pad[1];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int kx = lane % GL;
  const int leader = lane - kx;
  const bool col_on = kx < NS;
  T scale[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) scale[d] = -(T)((double)g.nf[d] / (2.0 * kPi));
  // the group's first lanes store one output each: the value, then dx, dy, dz
  T* dout = kx == 1 ? dx : (kx == 2 ? dy : (kx == 3 ? dz : nullptr));
  const int b = a.s.sub_bin[sidx];
  const int k0 = a.s.sub_start[sidx];
  const int k1 = sub_end(a.s, b, k0);
  int o[3];
  bin_origin(g, b, o[0], o[1], o[2]);
  for (int t = 0; t < a.n_trans; ++t) {
    __syncthreads();
    if (!stage_interp_tile<T>(a, o, G, t, s_tile, ts)) return false;
    __syncthreads();
    constexpr int kStep = NW * 32;
    const int kw = k0 + warp * 32;
    // permutation two rounds ahead, coordinates and V one round ahead
    int p_cur = round_perm(a.s, kw, k1), p_next = round_perm(a.s, kw + kStep, k1);
    T x_cur[3];
    round_coords<T, 3>(a, kw, k1, x_cur);
    CT v_cur;
    v_cur.x = v_cur.y = (T)0;
    if (p_cur >= 0) v_cur = V[(int64_t)t * a.M + p_cur];
    for (unsigned kb = kw; kb < (unsigned)k1; kb += kStep) {  // warp-uniform
      const WarpPoints<T> wp = warp_points<T, 3, NS>(a, p_cur, x_cur, o, row, plane);
      const CT vv = v_cur;
      p_cur = p_next;
      p_next = round_perm(a.s, kb + 2 * kStep, k1);
      round_coords<T, 3>(a, kb + kStep, k1, x_cur);
      if (p_cur >= 0) v_cur = V[(int64_t)t * a.M + p_cur];
      const int npts = min(32, k1 - (int)kb);
#pragma unroll 1
      for (int j0 = 0; j0 < npts; j0 += PPW) {
        const int j = j0 + lane / GL;
        const bool valid = j < npts;
        const int src = valid ? j : 0;
        const WarpPoints<T> pt = group_take<T, 3>(wp, src);
        CT v;
        v.x = __shfl_sync(kAll, vv.x, src);
        v.y = __shfl_sync(kAll, vv.y, src);
        const bool on = col_on && pt.off >= 0;
        T w[3], dw[3];  // this lane's weight q = kx of each axis, and its derivative
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          es_weight_deriv(rn_sub((T)(pt.i0[d] + kx), pt.xs[d]), a.beta, a.kc, w[d], dw[d]);
          dw[d] *= scale[d];
        }
        // one accumulator pair per z plane: plain and y-differentiated
        CT acc[NS], accd[NS];
#pragma unroll
        for (int kz = 0; kz < NS; ++kz) acc[kz].x = acc[kz].y = accd[kz].x = accd[kz].y = (T)0;
        const CT* base = s_tile + (on ? pt.off + kx : 0);
#pragma unroll
        for (int ky = 0; ky < NS; ++ky) {
          const T wy = __shfl_sync(kAll, w[1], leader + ky), dwy = __shfl_sync(kAll, dw[1], leader + ky);
#pragma unroll
          for (int kz = 0; kz < NS; ++kz) {
            const CT u = base[kz * plane + ky * row];
            acc[kz] = fma2(splat2(wy), u, acc[kz]);
            accd[kz] = fma2(splat2(dwy), u, accd[kz]);
          }
        }
        CT s0, sy, sz;
        s0.x = s0.y = sy.x = sy.y = sz.x = sz.y = (T)0;
#pragma unroll
        for (int kz = 0; kz < NS; ++kz) {
          const T wz = __shfl_sync(kAll, w[2], leader + kz), dwz = __shfl_sync(kAll, dw[2], leader + kz);
          s0 = fma2(splat2(wz), acc[kz], s0);
          sy = fma2(splat2(wz), accd[kz], sy);
          sz = fma2(splat2(dwz), acc[kz], sz);
        }
        // Re(conj(v) * s) = v.x s.x + v.y s.y per column, then summed over the columns
        T r[5];
        r[0] = on ? s0.x * w[0] : (T)0;
        r[1] = on ? s0.y * w[0] : (T)0;
        r[2] = on ? (v.x * s0.x + v.y * s0.y) * dw[0] : (T)0;
        r[3] = on ? (v.x * sy.x + v.y * sy.y) * w[0] : (T)0;
        r[4] = on ? (v.x * sz.x + v.y * sz.y) * w[0] : (T)0;
#pragma unroll
        for (int m = GL / 2; m >= 1; m >>= 1) {
#pragma unroll
          for (int i = 0; i < 5; ++i) r[i] += __shfl_xor_sync(kAll, r[i], m);
        }
        if (valid) {
          if (kx == 0 && out_interp != nullptr) {
            CT u;
            u.x = r[0];
            u.y = r[1];
            out_interp[(int64_t)t * a.M + pt.p] = u;
          }
          if (dout != nullptr) {
            const T val = kx == 1 ? r[2] : (kx == 2 ? r[3] : r[4]);
            dout[pt.p] = t == 0 ? val : dout[pt.p] + val;
          }
        }
      }
    }
  }
  return true;
}

// ---------------------------------------------------------------------------
// Gradient pass (see launch_grad in nfx_internal.h)
// ---------------------------------------------------------------------------
// CTAs per SM the gradient pass's registers must allow for (0: the compiler's
// choice).  1D complex128 at small widths runs on its residency: ns 6, 2M points,
// 107 us with four CTAs, 116 with three; 3D complex64 at widths 4 and 6 too (ns 6, 4M
// points on 256^3: 718 us with three, 937 with two).
template <typename T, int DIM, int NS>
constexpr int grad_min_ctas() {
  if (sizeof(T) == 4 && DIM == 3 && (NS == 4 || NS == 6)) return 3;
  return sizeof(T) == 8 && DIM == 1 && NS <= 6 ? (NS == 2 ? 5 : 4) : 0;
}

template <typename T, int DIM, int NS, int NW>
__global__ void __launch_bounds__(NW * 32, grad_min_ctas<T, DIM, NS>()) k_grad(const __grid_constant__ PointArgs<T> a, const cplx_t<T>* __restrict__ G,
                                                  const cplx_t<T>* __restrict__ V, cplx_t<T>* __restrict__ out_interp,
                                                  T* __restrict__ dx, T* __restrict__ dy, T* __restrict__ dz,
                                                  const __grid_constant__ CUtensorMap tmap) {
  using CT = cplx_t<T>;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t mbar;
  TmaStage ts{&tmap, smem_addr(&mbar), 0u};
  if (a.tma) tma_init(&mbar);
  CT* s_tile = reinterpret_cast<CT*>(smem_raw);
  const Geom& g = a.g;
  const int row = g.pitch;
  const int plane = g.pitch * g.pad[1];
  const int nsub = *a.s.nsub;
  T* douts[3] = {dx, dy, dz};
  for (int sidx = blockIdx.x; sidx < nsub; sidx += gridDim.x) {
    const int b = a.s.sub_bin[sidx];
    // 3D width 8, a lane group per point where the bin holds fewer points than cells
    // (and enough for four warps): a warp's 32 points are then many cells apart and
    // their footprint reads conflict.  In denser bins neighbouring threads read nearly
    // the same cells, and a thread per point is the faster one.  Thread -> group, us,
    // complex64: 8M on 256^3 (0.5 a cell) 2592 -> 2176, 1M on 192x225x256 583 -> 539;
    // but 4M on 128^3 (1.9 a cell) 881 -> 946, 1M clustered 254 -> 311, 100 k on 128^3
    // (98 a bin) 138 -> 142.  Other widths lose: ns 4, 4M on 256^3 520 -> 674 (the group
    // form also takes its registers from 80 to 99), ns 6 398 -> 445, complex128 ns 10
    // 315 -> 381.
    if constexpr (DIM == 3 && NS == 8) {
      const int in_bin = a.s.bin_start[b + 1] - a.s.bin_start[b];
      if (in_bin >= 128 && in_bin < g.tile[0] * g.tile[1] * g.tile[2]) {
        if (!grad_group<T, NS, NW>(a, G, V, out_interp, dx, dy, dz, sidx, smem_raw, ts)) return;
        continue;
      }
    }
    const int k0 = a.s.sub_start[sidx];
    const int k1 = sub_end(a.s, b, k0);
    int o[3];
    bin_origin(g, b, o[0], o[1], o[2]);
    for (int t = 0; t < a.n_trans; ++t) {
      __syncthreads();
      if (!stage_interp_tile<T>(a, o, G, t, s_tile, ts)) return;
      __syncthreads();
      // loads pipelined across iterations: the permutation two iterations
      // ahead, folded coordinates (sorted order) and V one iteration ahead
      const int kStep = blockDim.x;
      int k = k0 + threadIdx.x;
      int p_cur = (unsigned)k < (unsigned)k1 ? a.s.perm[k] : 0;
      int p_next = position_before(k, kStep, k1) ? a.s.perm[k + kStep] : 0;
      T x_cur[DIM];
      CT v_cur;
      v_cur.x = v_cur.y = (T)0;
#pragma unroll
      for (int d = 0; d < DIM; ++d) x_cur[d] = (unsigned)k < (unsigned)k1 ? sorted_coord(a, d, k) : (T)0;
      if ((unsigned)k < (unsigned)k1) v_cur = V[(int64_t)t * a.M + p_cur];
      for (; (unsigned)k < (unsigned)k1; k += kStep) {
        const int p = p_cur;
        T xv[DIM];
#pragma unroll
        for (int d = 0; d < DIM; ++d) xv[d] = x_cur[d];
        const CT vv = v_cur;
        {
          const bool more = position_before(k, kStep, k1);
          const int p_after = position_before(k, 2 * kStep, k1) ? a.s.perm[k + 2 * kStep] : 0;
#pragma unroll
          for (int d = 0; d < DIM; ++d) x_cur[d] = more ? sorted_coord(a, d, k + kStep) : (T)0;
          if (more) v_cur = V[(int64_t)t * a.M + p_next];
          p_cur = p_next;
          p_next = p_after;
        }
        T w[DIM][NS], dw[DIM][NS];
        int off = 0;
        bool inside = true;
#pragma unroll
        for (int d = 0; d < DIM; ++d) {
          const T xs = xv[d];
          const int i0 = left_cell<T, NS>(xs);
          const int l = wrap_index(i0, g.nf[d]) - o[d];
          inside = inside && (unsigned)l < (unsigned)g.tile[d];
          off += l * (d == 0 ? 1 : (d == 1 ? row : plane));
          const T scale = -(T)((double)g.nf[d] / (2.0 * kPi));
#pragma unroll
          for (int q = 0; q < NS; ++q) {
            T ph, dph;
            es_weight_deriv(rn_sub((T)(i0 + q), xs), a.beta, a.kc, ph, dph);
            w[d][q] = ph;
            dw[d][q] = dph * scale;
          }
        }
        // S[0] = sum G w ; S[1+d] = sum G (w with axis d differentiated)
        T sr[1 + DIM], si[1 + DIM];
#pragma unroll
        for (int i = 0; i <= DIM; ++i) sr[i] = si[i] = (T)0;
        const CT* base = s_tile + (inside ? off : 0);
        CT wxp[NS], dwxp[NS];  // (w_x, w_x) and (w_x', w_x') pairs, built once per point
#pragma unroll
        for (int kx = 0; kx < NS; ++kx) {
          wxp[kx] = splat2(w[0][kx]);
          dwxp[kx] = splat2(dw[0][kx]);
        }
#pragma unroll 1
        for (int kz = 0; kz < (inside && DIM == 3 ? NS : (inside ? 1 : 0)); ++kz) {
          // per-z accumulators: [0] plain, [1] d/dx, [2] d/dy
          T zr0 = 0, zi0 = 0, zr1 = 0, zi1 = 0, zr2 = 0, zi2 = 0;
#pragma unroll
          for (int ky = 0; ky < (DIM >= 2 ? NS : 1); ++ky) {
            const CT* rp = base + kz * plane + ky * row;
            CT xa, xa1;
            xa.x = xa.y = xa1.x = xa1.y = (T)0;
#pragma unroll
            for (int kx = 0; kx < NS; ++kx) {
              const CT v = rp[kx];
              xa = fma2(wxp[kx], v, xa);
              xa1 = fma2(dwxp[kx], v, xa1);
            }
            const T xr = xa.x, xi = xa.y, xr1 = xa1.x, xi1 = xa1.y;
            if (DIM >= 2) {
              const T wy = w[DIM >= 2 ? 1 : 0][ky], dwy = dw[DIM >= 2 ? 1 : 0][ky];
              zr0 += xr * wy;
              zi0 += xi * wy;
              zr1 += xr1 * wy;
              zi1 += xi1 * wy;
              zr2 += xr * dwy;
              zi2 += xi * dwy;
            } else {
              zr0 += xr;
              zi0 += xi;
              zr1 += xr1;
              zi1 += xi1;
            }
          }
          if (DIM == 3) {
            // z weights by an unrolled select: a dynamic index would put w / dw in local memory
            T wz = (T)0, dwz = (T)0;
#pragma unroll
            for (int q = 0; q < NS; ++q) {
              if (q == kz) {
                wz = w[DIM - 1][q];
                dwz = dw[DIM - 1][q];
              }
            }
            sr[0] += zr0 * wz;
            si[0] += zi0 * wz;
            sr[1] += zr1 * wz;
            si[1] += zi1 * wz;
            sr[2] += zr2 * wz;
            si[2] += zi2 * wz;
            sr[DIM] += zr0 * dwz;
            si[DIM] += zi0 * dwz;
          } else {
            sr[0] += zr0;
            si[0] += zi0;
            sr[1] += zr1;
            si[1] += zi1;
            if (DIM == 2) {
              sr[DIM] += zr2;
              si[DIM] += zi2;
            }
          }
        }
        if (out_interp != nullptr) {
          CT r;
          r.x = sr[0];
          r.y = si[0];
          out_interp[(int64_t)t * a.M + p] = r;
        }
#pragma unroll
        for (int d = 0; d < DIM; ++d) {
          if (douts[d] != nullptr) {
            // Re(conj(v) * s) = v.x s.x + v.y s.y ; accumulate over transforms
            const T val = vv.x * sr[1 + d] + vv.y * si[1 + d];
            if (t == 0)
              douts[d][p] = val;
            else
              douts[d][p] += val;
          }
        }
      }
    }
  }
}

// ---------------------------------------------------------------------------
// Host-side launch helpers (per instantiation)
// ---------------------------------------------------------------------------
template <typename T, int DIM, int NS>
struct Launch {
  static constexpr int NW = warps_per_cta(sizeof(T), DIM, NS);
  static constexpr int SW = win_warps<T, DIM, NS>();  // of the spread
  static size_t tile_smem(const Geom& g) { return (size_t)g.pad[2] * g.pad[1] * g.pitch * sizeof(cplx_t<T>); }

  // Chooses the work items of a spread of M_total points (over all problems of
  // the launch, which has room for `ctas` CTAs at a time); returns a bound on
  // this problem's items.
  static int64_t split_items(int64_t M_total, int ctas, PointArgs<T>& a) {
    if constexpr (WinShape<T, DIM, NS>::on) {
      const WinSplit w = win_split(DIM, WinShape<T, DIM, NS>::GROUP, SW, M_total, ctas, a.s.maxsub);
      a.win_part = w.part;
      a.win_group = w.group;
      return (a.M + a.win_part - 1) / a.win_part;
    } else {
      return a.s.max_subs;
    }
  }
  // Shared memory of the spread kernels (plain and batched) on a grid geometry.
  static size_t smem_spread(const Geom& g) {
    if constexpr (WinShape<T, DIM, NS>::on)
      return win_smem_bytes<T, DIM, NS>();
    else
      return spread_smem_bytes(sizeof(T), DIM, NS, g);
  }

  template <typename K>
  static cudaError_t prep(K kernel, size_t smem, int& grid, int64_t max_subs) {
    return kernel_grid(reinterpret_cast<const void*>(kernel), NW * 32, smem, max_subs, grid);
  }

  static cudaError_t spread(const PointArgs<T>& a, const cplx_t<T>* c, cplx_t<T>* fw, cudaStream_t st) {
    int grid = 0;
    if constexpr (DIM == 3 && NS >= 4) {
      // The plane-owner spread where no register window exists (widths from 10)
      // and points are sparser than grid cells, and for complex128 of width 8 on
      // such sets: its 9^3-cell windows hold about one point there, and their
      // reds cost more than the tile (100 k points on 96^3: window 355 us, owner
      // 265; 300 k: 592 against 556; widths 4 and 6: 83 against 103, 181 against
      // 265).  complex64 windows win at every density (1e4 points on 128^3: 52
      // against 99 us, 8M on 256^3: 1725 against 3645).
      const bool sparse = a.M < (int64_t)a.g.nf[0] * a.g.nf[1] * a.g.nf[2];
      const bool window = WinShape<T, DIM, NS>::on && (sizeof(T) == 4 || NS <= 6 || !sparse);
      if (a.g.spread_mode == NFX_PER_POINT_CTA || (a.g.spread_mode == NFX_PER_POINT_AUTO && sparse && !window)) {
        // the tile's row pitch is this kernel's own (footprint offsets follow it)
        PointArgs<T> ao = a;
        ao.g.pitch = owner_pitch(a.g.pitch, a.g.pad[0], NS, (int)sizeof(T));
        const size_t smem = owner_smem_bytes(sizeof(T), NS, NW, ao.g);
        cudaError_t e = prep(k_spread_owner<T, NS, NW>, smem, grid, ao.s.max_subs);
        if (e != cudaSuccess) return e;
        k_spread_owner<T, NS, NW><<<grid, NW * 32, smem, st>>>(ao, c, fw);
        return cudaGetLastError();
      }
    }
    const size_t smem = smem_spread(a.g);
    PointArgs<T> as = a;
    cudaError_t e = kernel_grid(reinterpret_cast<const void*>(k_spread<T, DIM, NS, SW>), SW * 32, smem, INT32_MAX, grid);
    if (e != cudaSuccess) return e;
    grid = (int)std::max<int64_t>(1, std::min<int64_t>(grid, split_items(as.M, grid, as)));
    k_spread<T, DIM, NS, SW><<<grid, SW * 32, smem, st>>>(as, c, fw);
    return cudaGetLastError();
  }
  template <int MODE>
  static cudaError_t interp_as(const PointArgs<T>& a0, const cplx_t<T>* fw, cplx_t<T>* out, cudaStream_t st) {
    // the interpolation only reads the tile, so its row pitch is free
    PointArgs<T> a = a0;
    CUtensorMap tmap{};
    tma_args(a, fw, &tmap);
    size_t smem = tile_smem(a.g);
    int grid = 0;
    cudaError_t e = prep(k_interp<T, DIM, NS, NW, MODE>, smem, grid, a.s.max_subs);
    if (e != cudaSuccess) return e;
    k_interp<T, DIM, NS, NW, MODE><<<grid, NW * 32, smem, st>>>(a, fw, out, tmap);
    return cudaGetLastError();
  }
  static cudaError_t interp(const PointArgs<T>& a, const cplx_t<T>* fw, cplx_t<T>* out, cudaStream_t st) {
    if constexpr (DIM >= 2) {
      if (interp_by_group<DIM>(a.g.interp_mode)) return interp_as<NFX_PER_POINT_GROUP>(a, fw, out, st);
    }
    return interp_as<NFX_PER_POINT_THREAD>(a, fw, out, st);
  }
  // The tile staging of the interpolation and gradient passes: a tensor map of
  // the grid for TMA box loads of interior tiles when the rules allow (else
  // a.tma = 0 and plain loads); a complex64 tile gets an even row pitch.
  static void tma_args(PointArgs<T>& a, const cplx_t<T>* grid, CUtensorMap* tmap) {
    a.tma = 0;
    if constexpr (DIM >= 2) {
      Geom gt = a.g;
      if (sizeof(T) == 4 && (gt.pitch & 1)) ++gt.pitch;
      if (interp_tile_map(tmap, sizeof(T), DIM, gt, a.n_trans, grid)) {
        a.status = device_status_word();
        if (a.status != nullptr) {
          a.g = gt;
          a.tma = 1;
        }
      }
    }
  }
  static cudaError_t grad(const PointArgs<T>& a0, const cplx_t<T>* G, const cplx_t<T>* V, cplx_t<T>* oi, T* dx,
                          T* dy, T* dz, cudaStream_t st) {
    PointArgs<T> a = a0;
    CUtensorMap tmap{};
    tma_args(a, G, &tmap);
    size_t smem = tile_smem(a.g);
    int grid = 0;
    cudaError_t e = prep(k_grad<T, DIM, NS, NW>, smem, grid, a.s.max_subs);
    if (e != cudaSuccess) return e;
    k_grad<T, DIM, NS, NW><<<grid, NW * 32, smem, st>>>(a, G, V, oi, dx, dy, dz, tmap);
    return cudaGetLastError();
  }
};

template <typename T, int DIM, int NS>
struct BatchLaunch {
  static constexpr int NW = warps_per_cta(sizeof(T), DIM, NS);
  static constexpr int SW = win_warps<T, DIM, NS>();
  // CTAs of the batched window spread that the GPU holds at a time (its shared
  // memory does not depend on the problem).
  static int window_ctas() {
    int grid = 0;
    if constexpr (WinShape<T, DIM, NS>::on) {
      if (kernel_grid(reinterpret_cast<const void*>(k_spread_batch<T, DIM, NS, SW>), SW * 32,
                      win_smem_bytes<T, DIM, NS>(), INT32_MAX, grid) != cudaSuccess)
        grid = 0;  // the launch reports it
    }
    return std::max(grid, 1);
  }
  static cudaError_t spread(const void* items, int n, const int* prefix, int64_t max_subs, size_t smem,
                            cudaStream_t st) {
    int grid = 0;
    cudaError_t e = kernel_grid(reinterpret_cast<const void*>(k_spread_batch<T, DIM, NS, SW>), SW * 32, smem, max_subs,
                                grid);
    if (e != cudaSuccess) return e;
    k_spread_batch<T, DIM, NS, SW><<<grid, SW * 32, smem, st>>>((const BatchItem<T>*)items, n, prefix);
    return cudaGetLastError();
  }
  static cudaError_t interp(const void* items, int n, const int* prefix, int64_t max_subs, size_t smem,
                            cudaStream_t st) {
    int grid = 0;
    cudaError_t e = kernel_grid(reinterpret_cast<const void*>(k_interp_batch<T, DIM, NS, NW>), NW * 32, smem, max_subs,
                                grid);
    if (e != cudaSuccess) return e;
    k_interp_batch<T, DIM, NS, NW><<<grid, NW * 32, smem, st>>>((const BatchItem<T>*)items, n, prefix);
    return cudaGetLastError();
  }
};

template <typename T, int DIM>
cudaError_t dispatch_batch(int ns, bool spread, const void* items, int n, const int* prefix, int64_t max_subs,
                           size_t smem, cudaStream_t st) {
  switch (ns) {
#define NFX_CASE(N)                                                                    \
  case N:                                                                              \
    return spread ? BatchLaunch<T, DIM, N>::spread(items, n, prefix, max_subs, smem, st) \
                  : BatchLaunch<T, DIM, N>::interp(items, n, prefix, max_subs, smem, st);
    NFX_CASE(2) NFX_CASE(4) NFX_CASE(6) NFX_CASE(8) NFX_CASE(10) NFX_CASE(12) NFX_CASE(14) NFX_CASE(16)
#undef NFX_CASE
    default:
      return cudaErrorInvalidValue;
  }
}

// Shared memory of the spread of one problem (the batched launches take the
// largest of theirs).
template <typename T, int DIM>
size_t spread_smem_dim(int ns, const Geom& g) {
  switch (ns) {
#define NFX_CASE(N) \
  case N:           \
    return Launch<T, DIM, N>::smem_spread(g);
    NFX_CASE(2) NFX_CASE(4) NFX_CASE(6) NFX_CASE(8) NFX_CASE(10) NFX_CASE(12) NFX_CASE(14) NFX_CASE(16)
#undef NFX_CASE
    default:
      return 0;
  }
}

// Work items of one problem of a batched spread (Launch::split_items).
template <typename T, int DIM>
int64_t split_spread_items(int ns, int64_t M_total, PointArgs<T>& a) {
  switch (ns) {
#define NFX_CASE(N) \
  case N:           \
    return Launch<T, DIM, N>::split_items(M_total, BatchLaunch<T, DIM, N>::window_ctas(), a);
    NFX_CASE(2) NFX_CASE(4) NFX_CASE(6) NFX_CASE(8) NFX_CASE(10) NFX_CASE(12) NFX_CASE(14) NFX_CASE(16)
#undef NFX_CASE
    default:
      return 0;
  }
}

template <typename T, int DIM>
cudaError_t dispatch_spread(int ns, const PointArgs<T>& a, const void* c, void* fw, cudaStream_t st) {
  using CT = cplx_t<T>;
  switch (ns) {
#define NFX_CASE(N) \
  case N:           \
    return Launch<T, DIM, N>::spread(a, (const CT*)c, (CT*)fw, st);
    NFX_CASE(2) NFX_CASE(4) NFX_CASE(6) NFX_CASE(8) NFX_CASE(10) NFX_CASE(12) NFX_CASE(14) NFX_CASE(16)
#undef NFX_CASE
    default:
      return cudaErrorInvalidValue;
  }
}

template <typename T, int DIM>
cudaError_t dispatch_interp(int ns, const PointArgs<T>& a, const void* fw, void* out, cudaStream_t st) {
  using CT = cplx_t<T>;
  switch (ns) {
#define NFX_CASE(N) \
  case N:           \
    return Launch<T, DIM, N>::interp(a, (const CT*)fw, (CT*)out, st);
    NFX_CASE(2) NFX_CASE(4) NFX_CASE(6) NFX_CASE(8) NFX_CASE(10) NFX_CASE(12) NFX_CASE(14) NFX_CASE(16)
#undef NFX_CASE
    default:
      return cudaErrorInvalidValue;
  }
}

template <typename T, int DIM>
cudaError_t dispatch_grad(int ns, const PointArgs<T>& a, const void* G, const void* V, void* oi, void* dx, void* dy,
                          void* dz, cudaStream_t st) {
  using CT = cplx_t<T>;
  switch (ns) {
#define NFX_CASE(N)                                                                                             \
  case N:                                                                                                       \
    return Launch<T, DIM, N>::grad(a, (const CT*)G, (const CT*)V, (CT*)oi, (T*)dx, (T*)dy, (T*)dz, st);
    NFX_CASE(2) NFX_CASE(4) NFX_CASE(6) NFX_CASE(8) NFX_CASE(10) NFX_CASE(12) NFX_CASE(14) NFX_CASE(16)
#undef NFX_CASE
    default:
      return cudaErrorInvalidValue;
  }
}

template <typename T>
PointArgs<T> make_args(const Geom& g, double beta, double kc, int64_t M, int n_trans, const SortView& s) {
  PointArgs<T> a;
  for (int d = 0; d < 3; ++d) a.sc[d] = (const T*)s.coord[d];
  a.M = M;
  a.n_trans = n_trans;
  a.grid_stride = (int64_t)g.nf[0] * g.nf[1] * g.nf[2];
  a.win_part = 0;
  a.win_group = 1;
  a.tma = 0;
  a.status = nullptr;
  a.g = g;
  a.beta = (T)beta;
  a.kc = (T)kc;
  a.s = s;
  a.poly.deg = 0;
  if constexpr (sizeof(T) == 8) a.polyd.deg = 0;
  return a;
}

}  // namespace nfx
