// Register-window spreading (2D, and 3D for the widths whose windows fit in
// registers).
//
// A warp takes the points whose left cells lie in one small block (BX x BY [x BZ]
// cells) and keeps the whole window those footprints cover (NS + B - 1 cells per
// axis) in its registers: every point adds (c w_x) w_y [w_z] to all of the
// window's cells, with zero weights outside its own footprint, so the inner loop
// has no address, no branch and no shared-memory update per cell.  When the
// block changes the window goes straight to the fine grid with vectorised reds,
// lanes along x.
//
// Why: a spread that adds every footprint cell to a shared-memory tile is bound
// by that update (a float add on shared memory is a compare-and-swap loop here,
// a plain read-add-write 64 of the 107 shared wavefronts a 3D point cost at
// ns = 8) while the FMA pipe idles.  Reds of windows to L2 run at 590 G complex64
// cells/s when the blocks follow the bin order (4x4x4 windows of a 256^3 grid,
// 348 M cells in 594 us; a CTA tile flushed by compare-and-swap takes as long)
// and are fire-and-forget, and the window sums the block's points first: at 0.5
// points per cell a 3D point costs 43 reds instead of 512 updates.
//
// Block shapes.  3D: 4x4x4 cells for complex64 (window 11^3 at ns = 8: 44 paired
// FMAs a lane and point, 17 ns per point and SM alone; 4x4x2 needs 36 but 1.6
// times the reds), 2x2x2 for complex128 (accumulators of twice the registers).
// A 3D block's points are not contiguous in the sorted order (cells x-fastest),
// so each CTA first groups its item's points by block with a counting sort of
// 16-bit indices in shared memory (two passes over the sorted keys).  2D
// complex64: segments of 8x1 cells, which are contiguous, so nothing is grouped
// (8x4 blocks measured 227 us on 4M clustered points, segments 157: grouping
// and the wider window cost more than the reds they save).  2D complex128:
// blocks, since a wide kernel's window is all reds.
//
// What bounds it now (sorted points, L2 flushed before each call; before = the
// shared-memory tile spreads it replaces): 3D 8M points on 256^3, ns 8: 3645 ->
// 1700 us (FMA pipe 52 %, issue 51 %); 1M on 192x225x256: 781 -> 509 us (reds);
// 2D 524 k radial on 1024^2, ns 8: 91 -> 54 us; complex128 ns 14, 200 k points: 412
// -> 79 us (reds).  Dense 2D complex64 sets are bound by their staging (issue 65 %,
// shared memory) and gain little or lose: 4M clustered points 163 -> 157 us, 8M 242
// -> 261.
#pragma once

#include <type_traits>

#include "nfx_internal.h"

namespace nfx {

constexpr int kWinRound = 2048;   // most points of a work item (16-bit list entries)
// Most blocks (of all its bins) an item is grouped by.  3D: what 2048 points span at
// half a point a block, below which grouping saves few reds.  With 1024, sparse sets
// on large grids went ungrouped: ns 8, 600 k points on 288^3 1770 us (grouped 1011,
// the plane-owner spread 1052), on 320^3 2008 (1271, 1353), 4M on 512^3 11740 (6153,
// 8400), 1M 4611 (3893, 6726); 300 points to 1M on 64^3 to 256^3 are unchanged.
constexpr int win_blocks(int dim) { return dim == 3 ? 4096 : 1024; }

// Block and lane layout per dimension and width.  2D: lane = (x, row group),
// LW x positions times H row groups of RL rows each.  3D: a lane owns NCOL
// (x, y) columns of WZ cells.
template <typename T, int DIM, int NS>
struct WinShape;

template <typename T, int NS>
struct WinShape<T, 2, NS> {
  static constexpr bool on = true;
  // complex64: row segments of BX cells, contiguous in the sorted order, so no
  // grouping; complex128: BX x BY blocks (wide kernels, costly window reds)
  static constexpr bool GROUP = sizeof(T) == 8;
  static constexpr int LW = 16;
  static constexpr int H = 32 / LW;
  static constexpr int BX = NS <= 8 ? 8 : (NS <= 12 ? 4 : (NS == 14 ? 2 : 1));
  static constexpr int BY = GROUP ? 4 : 1;
  static constexpr int BZ = 1;
  static constexpr int WX = NS + BX - 1, WY = NS + BY - 1;
  static constexpr int RL = (WY + H - 1) / H;
  static_assert(WX <= LW, "the window's x extent fits the lanes");
  // slot: c * w_x per x position, then the row weights, both zero outside the
  // footprint; an odd number of 16-byte units, so that slots of consecutive
  // points start in different banks
  static constexpr int YO = 2 * LW;
  static constexpr int R16 = 16 / (int)sizeof(T);
  static constexpr int RS = (RL + R16 - 1) / R16 * R16;  // a row group's weights, whole 16-byte units
  static constexpr int YN = H * RS;
  static constexpr int RAW = (YO + YN) / R16;
  static constexpr int SLOT = (RAW % 2 == 0 ? RAW + 1 : RAW) * R16;
};

// Whether a (type, width) has a 3D window: NCOL * WZ complex accumulators a lane.
template <typename T, int NS>
struct WinShape<T, 3, NS> {
  static constexpr bool on = NS <= 8;
  static constexpr bool GROUP = true;
  static constexpr int B = sizeof(T) == 4 ? 4 : 2;
  static constexpr int BX = B, BY = B, BZ = B;
  static constexpr int WX = NS + BX - 1, WY = NS + BY - 1, WZ = NS + BZ - 1;
  static constexpr int NC = WX * WY;
  static constexpr int NCOL = (NC + 31) / 32;
  // slot: w_z, c * w_x (complex), w_y
  static constexpr int R16 = 16 / (int)sizeof(T);
  static constexpr int ZN = (WZ + R16 - 1) / R16 * R16;
  static constexpr int XO = ZN;
  static constexpr int XN = (2 * WX + R16 - 1) / R16 * R16;
  static constexpr int YO = XO + XN;
  static constexpr int YN = (WY + R16 - 1) / R16 * R16;
  static constexpr int RAW = (YO + YN) / R16;
  static constexpr int SLOT = (RAW % 2 == 0 ? RAW + 1 : RAW) * R16;
};

template <typename T, int NS>
struct WinShape<T, 1, NS> {
  static constexpr bool on = false;
};

// Warps per CTA of the spread (the window of 44 complex64 cells a lane needs
// 168 registers, 68 bytes of them spilled).
template <typename T, int DIM, int NS>
constexpr int win_warps() {
  return sizeof(T) == 4 && DIM == 3 && NS == 8 ? 6 : warps_per_cta(sizeof(T), DIM, NS);
}

// Shared memory of a window spread: the warps' slots, a count per block and
// the block-ordered list.
template <typename T, int DIM, int NS>
size_t win_smem_bytes() {
  return (size_t)win_warps<T, DIM, NS>() * 32 * WinShape<T, DIM, NS>::SLOT * sizeof(T) +
         (WinShape<T, DIM, NS>::GROUP ? win_blocks(DIM) * sizeof(int) + kWinRound * sizeof(unsigned short) : 0);
}

// Work items of a spread of M points on `ctas` resident CTAs: points of one item,
// and the items of a group that one CTA takes when their points share a block.
// The items are equal, so as many as the CTAs take in whole rounds, of at most
// kWinRound points (2D: 1024; 2048 gives 4M clustered points on 1024^2 167 us for
// 161, on 4096^2 255 for 202, uniform 4M 148 for 153).  They go down to 32 points (a
// warp then stages a few): with at least 64, 1 k points on 1024^2 15.4 us, 13.3 with
// 32, 3D on 64^3 35.7 and 25.5; with at least 512 in 2D above 37,888 points (74 items
// for 148 SMs) 38 k points 31.8 us, 21.5 now, 100 k clustered 35.8 and 23.6.
// Groups (2D complex64) reach the size of a subproblem, so that a crowded cell gets no more
// partial sums than one tile per subproblem would send.  Float error of 2D points in
// one cell, over the root of the sum of squares: 100 k 2.0e-7, 1M 4.2e-7, 4M 5.6e-7
// (by shared-memory tiles 2.9e-7, 5.9e-7, 7.4e-7; every slice by itself 5.9e-7,
// 1.2e-6, 2.2e-6); 1M 3D points 5.9e-7 (4.7e-7, 9.7e-7).
// Spreads of at most 512 slices send every slice by itself (group 0).  8M points in
// few blocks, ns 6: 341 us, 286 without groups, 314 by shared-memory tiles.
struct WinSplit {
  int part, group;
};
inline WinSplit win_split(int dim, bool grouped, int warps, int64_t M, int ctas, int maxsub) {
  const int64_t most = dim == 2 ? 1024 : kWinRound;
  const int64_t rounds = (M + ctas * most - 1) / (ctas * most);
  int group = grouped ? 1 : (int)(maxsub < most ? 1 : (maxsub > 4 * most ? 4 : maxsub / most));
  int64_t n = rounds > 0 ? (M + ctas * rounds - 1) / (ctas * rounds) : 1;
  n = (n + 31) / 32 * 32;
  if (!grouped && rounds <= 1 && maxsub > n) group = (int)(maxsub / n < 16 ? maxsub / n : 16);
  if (M * warps <= 512 * n) group = 0;
  return WinSplit{(int)n, group};
}

// Adds one point whose strength or coordinates are not finite cell by cell
// (its window would turn zero weights of other cells into NaN): rare, so one
// lane loops over the footprint.
template <typename T, int DIM, int NS>
__device__ __forceinline__ void win_add_direct(const PointArgs<T>& a, cplx_t<T> cv, T x, T y, T z,
                                               cplx_t<T>* __restrict__ out) {
  const Geom& g = a.g;
  const int ix = left_cell<T, NS>(x), iy = left_cell<T, NS>(y), iz = DIM == 3 ? left_cell<T, NS>(z) : 0;
#pragma unroll 1
  for (int q = 0; q < (DIM == 3 ? NS * NS * NS : NS * NS); ++q) {
    const int kx = q % NS, ky = (q / NS) % NS, kz = q / (NS * NS);
    T w = es_weight(rn_sub((T)(ix + kx), x), a.beta, a.kc) * es_weight(rn_sub((T)(iy + ky), y), a.beta, a.kc);
    if (DIM == 3) w *= es_weight(rn_sub((T)(iz + kz), z), a.beta, a.kc);
    cplx_t<T> v;
    v.x = w * cv.x;
    v.y = w * cv.y;
    const int gx = wrap_index(ix + kx, g.nf[0]), gy = wrap_index(iy + ky, g.nf[1]);
    const int gz = DIM == 3 ? wrap_index(iz + kz, g.nf[2]) : 0;
    red_add(out + ((int64_t)gz * g.nf[1] + gy) * g.nf[0] + gx, v);
  }
}

// i >= 0 wrapped into axis d of the grid (no branch; windows may be wider than a tiny grid).
__device__ __forceinline__ int wrap_mod(int i, int d, const Geom& g) {
  return i - fast_div(i, g.ndiv[d]) * g.nf[d];
}

template <typename T>
__device__ __forceinline__ bool is_finite(T v) {
  return v - v == (T)0;
}

template <typename T>
__device__ __forceinline__ void zero_pair(cplx_t<T>& v) {
  v.x = v.y = (T)0;
}

// A slot section of N reals (a multiple of 16 bytes, 16-byte aligned): zeros,
// then NS weights from dl on (times the strength for the complex section).
template <int N, typename T>
__device__ __forceinline__ void stage_zero(T* s) {
  constexpr int R = 16 / (int)sizeof(T);
  static_assert(N % R == 0, "whole 16-byte units");
#pragma unroll
  for (int i = 0; i < N / R; ++i) reinterpret_cast<float4*>(s)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
}
template <int NS, int N, typename T>
__device__ __forceinline__ void stage_cw(T* s, cplx_t<T> cv, const T (&w)[NS], int dl) {
  stage_zero<N>(s);
#pragma unroll
  for (int q = 0; q < NS; ++q) reinterpret_cast<cplx_t<T>*>(s)[dl + q] = mul2(splat2(w[q]), cv);
}
template <int NS, int N, typename T>
__device__ __forceinline__ void stage_w(T* s, const T (&w)[NS], int dl) {
  stage_zero<N>(s);
#pragma unroll
  for (int q = 0; q < NS; ++q) s[dl + q] = w[q];
}

// The window accumulators of one lane: add(slot) takes a staged point,
// flush() sends the window to the grid and clears it.
template <typename T, int DIM, int NS>
struct Window;

// acc[k] += z[k] * v[k] for the first N of the reals at zs (16-byte loads; a
// real times a complex is one paired FMA, the real used for both halves).
template <int N, typename T, typename F>
__device__ __forceinline__ void for_weights(const T* zs, F f) {
  using V16 = typename Vec16<T>::type;
  constexpr int R = 16 / (int)sizeof(T);
#pragma unroll
  for (int k = 0; k < N; k += R) {
    const V16 z = *reinterpret_cast<const V16*>(zs + k);
    f(k, z.x);
    if (k + 1 < N) f(k + 1, z.y);
    if constexpr (R == 4) {
      if (k + 2 < N) f(k + 2, z.z);
      if (k + 3 < N) f(k + 3, z.w);
    }
  }
}

template <typename T, int NS>
struct Window<T, 2, NS> {
  using CT = cplx_t<T>;
  using PT = typename PairOf<T>::type;
  using W = WinShape<T, 2, NS>;
  static constexpr int CELLS = W::RL;
  // Grid index of a lane's cell i of the window that starts at `first`; -1: none.
  static __device__ __forceinline__ int cell_at(const Geom& g, int i, int lane, const int (&first)[3]) {
    const int x = lane % W::LW, row = (lane / W::LW) * W::RL + i;
    if (first[0] < 0 || x >= W::WX || row >= W::WY) return -1;
    return wrap_mod(first[1] + row, 1, g) * g.nf[0] + wrap_mod(first[0] + x, 0, g);
  }
  PT acc[W::RL];  // complex cells of this lane's rows
  int xo, yo;     // this lane's entries of a slot
  int zeros_at;   // x offset around which this lane's own slot holds zeros; -1: none

  __device__ __forceinline__ explicit Window(int lane) {
    xo = 2 * (lane % W::LW);
    yo = W::YO + (lane / W::LW) * W::RS;
    zeros_at = -1;
    clear();
  }
  __device__ __forceinline__ PT& cell(int i) { return acc[i]; }
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int i = 0; i < W::RL; ++i) acc[i] = pair_of((T)0, (T)0);
  }
  // Axis D's weights (times the strength on x) at offset dl of its section, zeros
  // in the rest of it: on x they are still there from the lane's last point while
  // the offset stays (8M clustered points 269 -> 261 us, sparse sets as before), a row block's
  // offset is always 0.
  template <int D>
  __device__ __forceinline__ void stage(T* sp, CT cv, const T (&w)[NS], int dl) {
    if constexpr (D == 0) {
      if (dl != zeros_at) stage_zero<W::YO>(sp);
      zeros_at = dl;
#pragma unroll
      for (int q = 0; q < NS; ++q) reinterpret_cast<CT*>(sp)[dl + q] = mul2(splat2(w[q]), cv);
    } else if constexpr (W::BY == 1) {
      auto at = [&](int p) { return p % W::RS < W::RL && p / W::RS * W::RL + p % W::RS < NS; };
      using V16 = typename Vec16<T>::type;
#pragma unroll
      for (int p = 0; p < W::YN; p += W::R16) {
        T v[W::R16];
#pragma unroll
        for (int i = 0; i < W::R16; ++i) v[i] = at(p + i) ? w[at(p + i) ? (p + i) / W::RS * W::RL + (p + i) % W::RS : 0] : (T)0;
        *reinterpret_cast<V16*>(sp + W::YO + p) = *reinterpret_cast<const V16*>(v);
      }
    } else {
      stage_zero<W::YN>(sp + W::YO);
#pragma unroll
      for (int q = 0; q < NS; ++q) {
        const int row = dl + q;  // row group row / RL starts at a multiple of RS
        sp[W::YO + row + (W::RS != W::RL && row >= W::RL ? W::RS - W::RL : 0)] = w[q];
      }
    }
  }
  // The slots' memory was used for something else.
  __device__ __forceinline__ void forget_slot() { zeros_at = -1; }
  __device__ __forceinline__ void add(const T* sp) { add_to(acc, sp); }
  __device__ __forceinline__ void add_to(PT (&sum)[W::RL], const T* sp) {
    const PT cw = *reinterpret_cast<const PT*>(sp + xo);
    for_weights<W::RL>(sp + yo, [&](int r, T w) { sum[r] = fma2(pair_of(w, w), cw, sum[r]); });
  }
  // Points j .. je - 1 of one block, four at a time.  A crowded block's alternate
  // between two sums, which halves the length (and float rounding) of each.
  __device__ __forceinline__ void add_run(const T*& sp, int& j, int je, bool crowded) {
    if (sizeof(T) == 4 && crowded) {
      PT other[W::RL];
#pragma unroll
      for (int r = 0; r < W::RL; ++r) other[r] = pair_of((T)0, (T)0);
      for (; j + 4 <= je; j += 4, sp += 4 * W::SLOT) {
#pragma unroll
        for (int q = 0; q < 4; q += 2) {
          add(sp + q * W::SLOT);
          add_to(other, sp + (q + 1) * W::SLOT);
        }
      }
#pragma unroll
      for (int r = 0; r < W::RL; ++r) acc[r] = add2(acc[r], other[r]);
    } else {
      for (; j + 4 <= je; j += 4, sp += 4 * W::SLOT) {
#pragma unroll
        for (int q = 0; q < 4; ++q) add(sp + q * W::SLOT);
      }
    }
#pragma unroll 1
    for (; j < je; ++j, sp += W::SLOT) add(sp);
  }
  // (ox, oy, oz): the window's first cell per axis (inside the grid)
  __device__ __forceinline__ void flush(const Geom& g, int ox, int oy, int, int lane, CT* __restrict__ out) {
    const int x = lane % W::LW;
    const int row0 = (lane / W::LW) * W::RL;
    if (x < W::WX) {
      int gy = wrap_mod(oy + row0, 1, g);
      int at = gy * g.nf[0] + wrap_mod(ox + x, 0, g);  // grids have fewer than 2^31 cells
#pragma unroll
      for (int r = 0; r < W::RL; ++r) {
        // no test for zero: skipping a red costs more than most zeros' reds
        if ((W::H - 1) * W::RL + r < W::WY || row0 + r < W::WY) red_add(out + at, unpair(acc[r]));
        at += g.nf[0];
        if (++gy == g.nf[1]) {
          gy = 0;
          at -= g.nf[0] * g.nf[1];
        }
      }
    }
    clear();
  }
};

template <typename T, int NS>
struct Window<T, 3, NS> {
  using CT = cplx_t<T>;
  using PT = typename PairOf<T>::type;
  using W = WinShape<T, 3, NS>;
  static constexpr int CELLS = W::NCOL * W::WZ;
  // As in 2D.
  static __device__ __forceinline__ int cell_at(const Geom& g, int i, int lane, const int (&first)[3]) {
    const int c = lane + 32 * (i / W::WZ);
    if (first[0] < 0 || c >= W::NC) return -1;
    return (wrap_mod(first[2] + i % W::WZ, 2, g) * g.nf[1] + wrap_mod(first[1] + c / W::WX, 1, g)) * g.nf[0] +
           wrap_mod(first[0] + c % W::WX, 0, g);
  }
  PT acc[W::NCOL][W::WZ];      // complex cells
  int xo[W::NCOL], yo[W::NCOL];  // this lane's columns' entries of a slot

  __device__ __forceinline__ explicit Window(int lane) {
#pragma unroll
    for (int i = 0; i < W::NCOL; ++i) {
      const int c = lane + 32 * i < W::NC ? lane + 32 * i : 0;
      xo[i] = W::XO + 2 * (c % W::WX);
      yo[i] = W::YO + c / W::WX;
    }
    clear();
  }
  __device__ __forceinline__ PT& cell(int i) { return acc[i / W::WZ][i % W::WZ]; }
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int i = 0; i < W::NCOL; ++i)
#pragma unroll
      for (int k = 0; k < W::WZ; ++k) acc[i][k] = pair_of((T)0, (T)0);
  }
  __device__ __forceinline__ void forget_slot() {}
  template <int D>
  static __device__ __forceinline__ void stage(T* sp, CT cv, const T (&w)[NS], int dl) {
    if constexpr (D == 0) {
      stage_cw<NS, W::XN>(sp + W::XO, cv, w, dl);
    } else if constexpr (D == 1) {
      stage_w<NS, W::YN>(sp + W::YO, w, dl);
    } else {
      stage_w<NS, W::ZN>(sp, w, dl);
    }
  }
  __device__ __forceinline__ void add(const T* sp) {
    PT v[W::NCOL];
#pragma unroll
    for (int i = 0; i < W::NCOL; ++i) {
      const CT cw = *reinterpret_cast<const CT*>(sp + xo[i]);
      const T wy = sp[yo[i]];
      v[i] = pair_of(cw.x * wy, cw.y * wy);
    }
    for_weights<W::WZ>(sp, [&](int k, T z) {
      const PT zd = pair_of(z, z);
#pragma unroll
      for (int i = 0; i < W::NCOL; ++i) acc[i][k] = fma2(zd, v[i], acc[i][k]);
    });
  }
  __device__ __forceinline__ void add_run(const T*& sp, int& j, int je, bool) {
    for (; j + 2 <= je; j += 2, sp += 2 * W::SLOT) {
      add(sp);
      add(sp + W::SLOT);
    }
#pragma unroll 1
    for (; j < je; ++j, sp += W::SLOT) add(sp);
  }
  __device__ __forceinline__ void flush(const Geom& g, int ox, int oy, int oz, int lane, CT* __restrict__ out) {
    const int plane = g.nf[0] * g.nf[1];  // grids have fewer than 2^31 cells
    int at[W::NCOL];
#pragma unroll
    for (int i = 0; i < W::NCOL; ++i) {
      const int c = lane + 32 * i;
      at[i] = (oz * g.nf[1] + wrap_mod(oy + c / W::WX, 1, g)) * g.nf[0] + wrap_mod(ox + c % W::WX, 0, g);
    }
    const bool last_on = W::NC % 32 == 0 || lane + 32 * (W::NCOL - 1) < W::NC;  // this lane has a last column
    int gz = oz;  // a block starts inside the grid
#pragma unroll
    for (int k = 0; k < W::WZ; ++k) {
      // no test for zero: skipping a red costs more than most zeros' reds
#pragma unroll
      for (int i = 0; i < W::NCOL - 1; ++i) red_add(out + at[i], unpair(acc[i][k]));
      if (last_on) red_add(out + at[W::NCOL - 1], unpair(acc[W::NCOL - 1][k]));
      int step = plane;
      if (++gz == g.nf[2]) {
        gz = 0;
        step = plane - plane * g.nf[2];
      }
#pragma unroll
      for (int i = 0; i < W::NCOL; ++i) at[i] += step;
    }
    clear();
  }
};

// Block of a point's cell within its tile, from its composite key.
template <typename T, int DIM, int NS>
__device__ __forceinline__ int key_block(const Geom& g, int cell) {
  using W = WinShape<T, DIM, NS>;
  const int nbx = (g.tile[0] + W::BX - 1) / W::BX, nby = (g.tile[1] + W::BY - 1) / W::BY;
  const int r = fast_div(cell, g.tdiv[0]);
  const int cx = cell - r * g.tile[0];
  if (DIM == 2) return r / W::BY * nbx + cx / W::BX;
  const int cz = fast_div(r, g.tdiv[1]);
  const int cy = r - cz * g.tile[1];
  return (cz / W::BZ * nby + cy / W::BY) * nbx + cx / W::BX;
}
template <typename T, int DIM, int NS>
__device__ __forceinline__ bool same_block(const PointArgs<T>& a, int key, int other) {
  const int cmask = (1 << a.s.cbits) - 1;
  return key >> a.s.cbits == other >> a.s.cbits &&
         key_block<T, DIM, NS>(a.g, key & cmask) == key_block<T, DIM, NS>(a.g, other & cmask);
}

// Sends the open windows of a crowded item's warps (whose points share a block) to
// the grid as their sum, formed in the slots' shared memory by all warps.  Every
// addition to a grid cell rounds at the size of the whole sum: what a crowded block
// sends should be few large partial sums.  Returns whether this warp still holds a
// window: one of another block than the first warp's (tiles that are no multiple of
// the block) stays with its warp.
template <typename T, int DIM, int NS, int NW>
__device__ __forceinline__ bool send_sum(Window<T, DIM, NS>& win, const int (&cur)[3], const Geom& g, T* s_slots,
                                         int warp, int lane, cplx_t<T>* __restrict__ out) {
  using PT = typename PairOf<T>::type;
  using W = WinShape<T, DIM, NS>;
  constexpr int CELLS = Window<T, DIM, NS>::CELLS;
  constexpr int PER = W::SLOT / 2;  // cells a lane that a warp's slots hold
  __shared__ int s_cur[NW][3];
  PT* const buf = reinterpret_cast<PT*>(s_slots) + lane;  // warp w's cells start at w * 32 * PER
  if (lane < 3) s_cur[warp][lane] = lane == 0 ? cur[0] : (lane == 1 ? cur[1] : cur[2]);
  auto same = [&](int w) {
    return s_cur[w][0] == s_cur[0][0] && s_cur[w][1] == s_cur[0][1] && s_cur[w][2] == s_cur[0][2];
  };
#pragma unroll
  for (int h = 0; h < CELLS; h += PER) {
    __syncthreads();  // the slots' points, or the cells of the part before, are done with
#pragma unroll
    for (int i = h; i < CELLS && i < h + PER; ++i) buf[(warp * PER + i - h) * 32] = win.cell(i);
    __syncthreads();
#pragma unroll 1
    for (int i = h + warp; i < CELLS && i < h + PER; i += NW) {
      const int at = Window<T, DIM, NS>::cell_at(g, i, lane, s_cur[0]);
      if (at < 0) continue;
      PT sum = buf[(i - h) * 32];
#pragma unroll 1
      for (int w = 1; w < NW; ++w)
        if (same(w)) sum = add2(sum, buf[(w * PER + i - h) * 32]);
      red_add(out + at, unpair(sum));
    }
  }
  const bool sent = same(warp);
  __syncthreads();
  if (sent) win.clear();
  win.forget_slot();
  return !sent && cur[0] >= 0;
}

// First point and points of the group of items that `item` belongs to.
template <typename T>
__device__ __forceinline__ int win_group_points(const PointArgs<T>& a, int item, int& n) {
  const int k = (item - item % a.win_group) * a.win_part;
  n = (int)min((int64_t)a.win_part * a.win_group, a.M - k);
  return k;
}
// The keys of that group's first and last point, in lanes 0 and 1, which an item of
// an ungrouped kernel needs ahead.
template <typename T>
__device__ __forceinline__ int win_group_keys(const PointArgs<T>& a, int item) {
  if (a.win_group == 0) return 0;
  int n;
  const int k = win_group_points(a, item, n), lane = threadIdx.x & 31;
  return lane < 2 ? a.s.keys[lane == 0 ? k : k + n - 1] : 0;
}

// The points k0 .. k0 + n - 1 of an item, in the order of `list` (nullptr: as they
// are), each warp a slice; one_block: the item is crowded.
template <typename T, int DIM, int NS, int NW>
__device__ __forceinline__ void spread_slices(const PointArgs<T>& a, const cplx_t<T>* __restrict__ c,
                                              cplx_t<T>* __restrict__ fw, int k0, int n, const unsigned short* list,
                                              bool one_block, T* s_slots) {
  using CT = cplx_t<T>;
  using W = WinShape<T, DIM, NS>;
  const Geom& g = a.g;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  T* my_slot = s_slots + (warp * 32 + lane) * W::SLOT;
  const T* warp_slots = s_slots + warp * 32 * W::SLOT;
  auto list_at = [&](int i) { return W::GROUP && list != nullptr ? (int)list[i] : i; };
  const int p0 = (int)((int64_t)n * warp / NW);  // slices differ by at most one point
  const int p1 = (int)((int64_t)n * (warp + 1) / NW);
  Window<T, DIM, NS> win(lane);
  for (int t = 0; t < a.n_trans; ++t) {
    const CT* ct = c + (int64_t)t * a.M;
    CT* const out = fw + (int64_t)t * a.grid_stride;
    // this lane's point of the next 32 (kn < 0: none), two list entries ahead
    T xn[DIM];
    CT cn;
    zero_pair<T>(cn);
#pragma unroll
    for (int d = 0; d < DIM; ++d) xn[d] = (T)0;
    int kn = p0 + lane < p1 ? k0 + list_at(p0 + lane) : -1;
    if (kn >= 0) {
      load_sorted<T, DIM>(a, kn, xn);
      cn = ct[a.s.perm[kn]];
    }
    int k2 = p0 + 32 + lane < p1 ? k0 + list_at(p0 + 32 + lane) : -1;
    int pn = k2 >= 0 ? a.s.perm[k2] : 0;
    int cur[3] = {-1, -1, -1};  // the open window's first cell per axis, -1: none
    for (int p = p0; p < p1; p += 32) {
      const int cnt = min(32, p1 - p);
      const int k = kn;
      T xv[DIM];
#pragma unroll
      for (int d = 0; d < DIM; ++d) xv[d] = xn[d];
      CT cv = cn;
      kn = k2;
      if (kn >= 0) {
        load_sorted<T, DIM>(a, kn, xn);
        cn = ct[pn];
      }
      k2 = p + 64 + lane < p1 ? k0 + list_at(p + 64 + lane) : -1;
      pn = k2 >= 0 ? a.s.perm[k2] : 0;
      // stage this lane's point, axis by axis (points added directly stage zeros)
      int base[3] = {0, 0, 0};
      int i0[DIM], dl[DIM];
      bool fin = true;
#pragma unroll
      for (int d = 0; d < DIM; ++d) {
        constexpr int kB[3] = {W::BX, W::BY, W::BZ};
        i0[d] = left_cell<T, NS>(xv[d]);
        const int l = wrap_index(i0[d], g.nf[d]);
        base[d] = (int)((unsigned)l / kB[d]) * kB[d];
        dl[d] = l - base[d];
        fin = fin && is_finite(xv[d]);
      }
      if (k >= 0) cv = with_extra(a, k, cv);
      fin = fin && is_finite(cv.x) && is_finite(cv.y);
      if (k >= 0 && !fin) win_add_direct<T, DIM, NS>(a, cv, xv[0], xv[1], xv[DIM - 1], out);
      if (k < 0 || !fin) {
        zero_pair<T>(cv);
#pragma unroll
        for (int d = 0; d < DIM; ++d) {
          dl[d] = i0[d] = 0;
          xv[d] = (T)(NS / 2);
        }
      }
      T w[NS];
      axis_weights<T, NS>(a, i0[0], xv[0], w);
      win.template stage<0>(my_slot, cv, w, dl[0]);
      axis_weights<T, NS>(a, i0[1], xv[1], w);
      win.template stage<1>(my_slot, cv, w, dl[1]);
      if constexpr (DIM == 3) {
        axis_weights<T, NS>(a, i0[2], xv[2], w);
        win.template stage<2>(my_slot, cv, w, dl[2]);
      }
      // lane j starts a block when its block differs from point j - 1's
      bool differs = false;
#pragma unroll
      for (int d = 0; d < DIM; ++d) {
        int prev = __shfl_up_sync(0xffffffffu, base[d], 1);
        if (lane == 0) prev = cur[d];
        differs = differs || prev != base[d];
      }
      const unsigned starts = __ballot_sync(0xffffffffu, differs && lane < cnt);
      __syncwarp();
      int j = 0;
      do {  // one block (or the rest of one) per trip
        if ((starts >> j) & 1u) {
          if (cur[0] >= 0) win.flush(g, cur[0], cur[1], cur[2], lane, out);
#pragma unroll
          for (int d = 0; d < DIM; ++d) cur[d] = __shfl_sync(0xffffffffu, base[d], j);
          if (DIM == 2) cur[2] = 0;
        }
        const unsigned later = j < 31 ? starts >> (j + 1) : 0u;
        const int je = later != 0u ? min(j + __ffs(later), cnt) : cnt;
        const T* sp = warp_slots + j * W::SLOT;
        win.add_run(sp, j, je, one_block);
      } while (j < cnt);
      __syncwarp();
    }
    bool open = cur[0] >= 0;
    if (one_block) open = send_sum<T, DIM, NS, NW>(win, cur, g, s_slots, warp, lane, out);
    if (open) win.flush(g, cur[0], cur[1], cur[2], lane, out);
  }
}

// A crowded 3D item, by itself: inlined beside the ordinary one, its sum over the
// warps cost that one's loop 200 bytes of spills (8M points on 256^3 1721 -> 1818 us).
template <typename T, int DIM, int NS, int NW>
__device__ __noinline__ void spread_crowded(const PointArgs<T>& a, const cplx_t<T>* __restrict__ c,
                                            cplx_t<T>* __restrict__ fw, int k0, int n) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  spread_slices<T, DIM, NS, NW>(a, c, fw, k0, n, nullptr, true, reinterpret_cast<T*>(smem_raw));
}

// One work item: `a.win_part` consecutive points of the sorted order (of one or
// several bins); ahead: its win_group_keys (ungrouped).  The CTA groups them by block,
// then every warp takes a contiguous slice of the grouped list 32 points at a time:
// each lane stages one point, and the warp adds the 32 one after another, flushing
// the window whenever the block changes.  The next 32 points are fetched while the
// current ones are added.
// A crowded item's points all lie in one block; its warps send one window.  Where a
// block's points are contiguous, one item of a group of `a.win_group` whose points
// share a block takes the whole group and the others nothing; which one rotates
// with the group's place in the grid-stride order, so that each CTA gets its share.
template <typename T, int DIM, int NS, int NW>
__device__ __forceinline__ void spread_window(const PointArgs<T>& a, const cplx_t<T>* __restrict__ c,
                                              cplx_t<T>* __restrict__ fw, int item, int ahead,
                                              unsigned char* smem_raw) {
  using W = WinShape<T, DIM, NS>;
  constexpr int NT = NW * 32;
  constexpr int PER = (kWinRound + NT - 1) / NT;  // most points of an item per thread
  __shared__ int s_warp[32];
  const Geom& g = a.g;
  int k0 = item * a.win_part;
  int n = (int)min((int64_t)a.win_part, a.M - k0);
  bool one_block = false;
  if constexpr (!W::GROUP) {  // a block's points are contiguous: the ends decide
    one_block = a.win_group > 0 && same_block<T, DIM, NS>(a, __shfl_sync(0xffffffffu, ahead, 0),
                                                          __shfl_sync(0xffffffffu, ahead, 1));
    if (one_block) {
      k0 = win_group_points(a, item, n);
      const unsigned members = (unsigned)((n + a.win_part - 1) / a.win_part);
      if (item % a.win_group != (int)((unsigned)item / gridDim.x % members)) return;
    }
  }
  T* s_slots = reinterpret_cast<T*>(smem_raw);
  int* s_cnt = reinterpret_cast<int*>(s_slots + NT * W::SLOT);  // per block: points, then its list start
  unsigned short* s_list = reinterpret_cast<unsigned short*>(s_cnt + win_blocks(DIM));
  // ---- group the points by block: bins in order, blocks within a bin ----
  bool listed = false;
  if constexpr (W::GROUP) {
    const int per_bin = key_block<T, DIM, NS>(g, g.tile[0] * g.tile[1] * g.tile[2] - 1) + 1;  // blocks
    const int bin0 = a.s.keys[k0] >> a.s.cbits;
    const int64_t span = (int64_t)((a.s.keys[k0 + n - 1] >> a.s.cbits) - bin0 + 1) * per_bin;
    // more: sparse points, few of them share a block
    listed = span <= win_blocks(DIM) && span >= 1;
    if (listed) {
      const int nblk = (int)span;
      const int cmask = (1 << a.s.cbits) - 1;
      for (int i = threadIdx.x; i < nblk; i += NT) s_cnt[i] = 0;
      int key[PER], rank[PER];
#pragma unroll
      for (int i = 0; i < PER; ++i) {
        const int j = i * NT + threadIdx.x;
        key[i] = j < n ? a.s.keys[k0 + j] : -1;
      }
      __syncthreads();
#pragma unroll
      for (int i = 0; i < PER; ++i) {
        if (key[i] >= 0) {
          const int blk = ((key[i] >> a.s.cbits) - bin0) * per_bin + key_block<T, DIM, NS>(g, key[i] & cmask);
          key[i] = min(max(blk, 0), nblk - 1);  // keys of a sound sort are in range
          rank[i] = atomicAdd(&s_cnt[key[i]], 1);
        }
      }
      __syncthreads();
      const int per = (nblk + NT - 1) / NT;
      const int i0 = min((int)threadIdx.x * per, nblk), i1 = min(i0 + per, nblk);
      int sum = 0, total;
      for (int i = i0; i < i1; ++i) sum += s_cnt[i];
      int run = block_exclusive_scan(sum, s_warp, total);
      for (int i = i0; i < i1; ++i) {
        const int v = s_cnt[i];
        s_cnt[i] = run;
        run += v;
      }
      __syncthreads();
      bool first = true;  // whether the thread's points lie in the first block that has any
#pragma unroll
      for (int i = 0; i < PER; ++i) {
        if (key[i] >= 0) {
          const int at = s_cnt[key[i]];
          first = first && at == 0;
          s_list[at + rank[i]] = (unsigned short)(i * NT + threadIdx.x);
        }
      }
      one_block = __syncthreads_and(first) && a.win_group > 0;
    }
  }
  if constexpr (DIM == 3) {
    if (one_block)
      spread_crowded<T, DIM, NS, NW>(a, c, fw, k0, n);
    else
      spread_slices<T, DIM, NS, NW>(a, c, fw, k0, n, listed ? s_list : nullptr, false, s_slots);
  } else {
    spread_slices<T, DIM, NS, NW>(a, c, fw, k0, n, listed ? s_list : nullptr, one_block, s_slots);
  }
  if constexpr (W::GROUP) __syncthreads();  // the list and counts are free for the next item
}

}  // namespace nfx
