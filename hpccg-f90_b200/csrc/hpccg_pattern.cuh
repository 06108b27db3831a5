// hpccg_pattern.cuh -- row patterns: a lossless compressed form of a stored matrix.
//
// A row's pattern is its sequence of (column - row, value) over the 27 ELL slots,
// values compared bit for bit.  A matrix made by a stencil has few distinct ones
// (generate_matrix: one per combination of faces a grid point lies on, at most
// 27), so a row is a 2-byte code into a table, and an SpMV that streams 12 bytes
// per slot of the ELL reads 2 bytes per row instead.  The row sum adds the same
// terms in the same order as the ELL kernel's, so it is bit for bit the same.
// The format is found from the stored entries alone (row_patterns below), holds
// for any matrix with few enough patterns, and every row is compared with its
// table entry before it is used.
#pragma once
#include "hpccg_internal.cuh"
#include "hpccg_stencil.cuh"

namespace hpccg {

constexpr int kPatW = 27;    // slots of a pattern (the ELL width)
constexpr int kPatLocal = 32;  // patterns of a table that an SpMV block copies to shared memory

__device__ __forceinline__ PatEntry64 pat_entry(const PatEntry64 *p) {
  const int4 q = __ldg(reinterpret_cast<const int4 *>(p));
  return PatEntry64{__hiloint2double(q.y, q.x), q.z, 0};
}
__device__ __forceinline__ PatEntry32 pat_entry(const PatEntry32 *p) {
  const int2 q = __ldg(reinterpret_cast<const int2 *>(p));
  return PatEntry32{q.x, __int_as_float(q.y)};
}

// Looks for at most max_count patterns in the rows [0, n) of a 27-slot ELL;
// out->count = 0 when there are more, or no memory for the tables.  Synchronises the stream.
int row_patterns(const int32_t *ell_col, const double *ell_val, int npad, int n, int max_count, int num_sms,
                 cudaStream_t s, RowPatterns *out);
void free_patterns(RowPatterns *p);
// For a matrix on a known grid: the patterns as values at the 3x3x3 neighbours
// (p->box64 and its roundings); p->boxes tells whether every one's entries lie
// there in order (no where memory is short).  Synchronises the stream.
int pattern_boxes(RowPatterns *p, int nx, int ny, cudaStream_t s);
// The same for patterns of several grids: place[c] = (nx, ny, box number) of pattern c, on
// the device; nx = 0: no box.
int pattern_boxes_placed(RowPatterns *p, const int4 *place, cudaStream_t s);

__device__ __forceinline__ double pat_term(double s, const PatEntry64 &e, const double *__restrict__ x) {
  return __dadd_rn(s, __dmul_rn(e.v, __ldg(x + e.off)));  // the ELL kernels' operations
}
__device__ __forceinline__ float pat_term(float s, const PatEntry32 &e, const float *__restrict__ x) {
  return fmaf(e.v, __ldg(x + e.off), s);
}

// The block's copy of the table.
template <typename Entry>
__device__ __forceinline__ const Entry *pattern_table(const Entry *__restrict__ table, int count) {
  __shared__ Entry local[kPatLocal * kPatW];
  for (int i = threadIdx.x; i < count * kPatW; i += blockDim.x) local[i] = table[i];
  __syncthreads();
  return local;
}

// Grid-stride rows, one at a time; a row's terms are added in slot order, as in the
// ELL kernels.  A warp whose lanes share a pattern reads one address of the table.
template <typename Real, typename Entry, class Done>
__device__ __forceinline__ void pattern_stride(int n, const uint16_t *__restrict__ code,
                                               const Entry *__restrict__ table, int count,
                                               const Real *__restrict__ x, Done &&done) {
  const Entry *local = pattern_table(table, count);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const Entry *t = local + (int)__ldg(code + i) * kPatW;
    Real s = Real(0);
#pragma unroll 9
    for (int k = 0; k < kPatW; ++k) s = pat_term(s, t[k], x + i);
    done(i, s);
  }
}

// ---- walks of a known grid with the patterns' values as 3x3x3 boxes -----------------
// A walk along z loads each plane's neighbourhood once (9 values for a column, 12
// for a column pair) for the three rows that need it, instead of 27 gathers a
// row; the sums are split at the planes as in stencil_column2 and take each row's
// own values (its pattern's box, in shared memory).  A neighbour that a row does
// not have adds 0 * 0 (outside the grid) to a sum that is never -0.0, so the sums
// are the ELL kernels', bit for bit.
__device__ __forceinline__ double box_term(double s, double v, double x) { return __dadd_rn(s, __dmul_rn(v, x)); }
__device__ __forceinline__ float box_term(float s, float v, float x) { return fmaf(v, x, s); }

// The sums in flight of RY rows side by side in y: lead = plane z-1's nine terms of
// the next plane's rows, mid = the current plane's rows through their own plane.
template <typename Real, int RY>
struct BoxSums {
  Real lead[RY], mid[RY], xc[RY];
  // plane p's values (lines y-1 .. y+RY, three each) and the boxes of the rows of
  // planes p-1 (te), p (tm) and p+1 (tl): END the rows of p-1 (into s), MID those of
  // p, and start the leads of p+1.  Rows of a pair that share a box read it once.
  template <bool END, bool MID>
  __device__ __forceinline__ void plane(const Real *v, const Real *const *te, const Real *const *tm,
                                        const Real *const *tl, Real *s) {
    bool same = true;
    if (RY == 2) same = te[0] == te[RY - 1] && tm[0] == tm[RY - 1] && tl[0] == tl[RY - 1];
    if (RY == 1 || __all_sync(__activemask(), same)) step<END, MID, true>(v, te, tm, tl, s);
    else step<END, MID, false>(v, te, tm, tl, s);
  }
  template <bool END, bool MID, bool SAME>
  __device__ __forceinline__ void step(const Real *v, const Real *const *te, const Real *const *tm,
                                       const Real *const *tl, Real *s) {
    if (END) {
#pragma unroll
      for (int r = 0; r < RY; ++r) s[r] = mid[r];
#pragma unroll
      for (int j = 0; j < 9; ++j) {
        const Real t = te[0][18 + j];
#pragma unroll
        for (int r = 0; r < RY; ++r) s[r] = box_term(s[r], SAME ? t : te[r][18 + j], v[3 * r + j]);
      }
    }
    if (MID) {
#pragma unroll
      for (int r = 0; r < RY; ++r) {
        mid[r] = lead[r];
        xc[r] = v[3 * r + 4];
      }
#pragma unroll
      for (int j = 0; j < 9; ++j) {
        const Real t = tm[0][9 + j];
#pragma unroll
        for (int r = 0; r < RY; ++r) mid[r] = box_term(mid[r], SAME ? t : tm[r][9 + j], v[3 * r + j]);
      }
    }
#pragma unroll
    for (int r = 0; r < RY; ++r) lead[r] = Real(0);
#pragma unroll
    for (int j = 0; j < 9; ++j) {
      const Real t = tl[0][j];
#pragma unroll
      for (int r = 0; r < RY; ++r) lead[r] = box_term(lead[r], SAME ? t : tl[r][j], v[3 * r + j]);
    }
  }
};

// Walks rows [z0, z1) of the column c (and c + nx): load(p, v) gives plane p's values
// and returns false to stop; done(row, sum, x) in the order of thread_rows.
template <typename Real, int RY, class Load, class Done>
__device__ __forceinline__ void box_walk(int c, int z0, int z1, int nx, int plane, int nz,
                                         const uint16_t *__restrict__ code, const Real *table, Load &&load,
                                         Done &&done) {
  const Real *te[RY], *tm[RY], *tl[RY];
  auto box = [&](int z, int r) {  // the row's box (any, beyond the last plane)
    return table + (int)__ldg(code + c + r * nx + min(z, nz - 1) * plane) * kPatW;
  };
  Real v[3 * (RY + 2)], s[RY];
  BoxSums<Real, RY> w;
#pragma unroll
  for (int r = 0; r < RY; ++r) te[r] = tm[r] = tl[r] = box(z0, r);
  if (!load(z0 - 1, v)) return;
  w.template plane<false, false>(v, te, tm, tl, s);
#pragma unroll
  for (int r = 0; r < RY; ++r) tl[r] = box(z0 + 1, r);
  if (!load(z0, v)) return;
  w.template plane<false, true>(v, te, tm, tl, s);
  for (int z = z0; z < z1; ++z) {
#pragma unroll
    for (int r = 0; r < RY; ++r) {
      te[r] = tm[r];
      tm[r] = tl[r];
      tl[r] = box(z + 2, r);
    }
    if (!load(z + 1, v)) return;
    Real x[RY];
#pragma unroll
    for (int r = 0; r < RY; ++r) x[r] = w.xc[r];
    w.template plane<true, true>(v, te, tm, tl, s);
#pragma unroll
    for (int r = 0; r < RY; ++r) done(c + r * nx + z * plane, s[r], x[r]);
  }
}

// The block's copy of the boxes.
template <typename Real>
__device__ __forceinline__ const Real *box_table(const Real *__restrict__ table, int count) {
  __shared__ Real local[kPatLocal * kPatW];
  for (int i = threadIdx.x; i < count * kPatW; i += blockDim.x) local[i] = table[i];
  __syncthreads();
  return local;
}

// The calling thread's rows under a map of the grid, from plain loads.
template <typename Real, class Done>
__device__ __forceinline__ void box_rows(const StencilGeom &g, const PlaneMap &m, const uint16_t *__restrict__ code,
                                         const Real *__restrict__ table, int count, const Real *__restrict__ x,
                                         Done &&done) {
  const Real *local = box_table(table, count);
  int c, z0, z1;
  if (m.tiles_x > 0) {
    const TileSpan sp = tile_span(m, g.nz);
    if (!sp.rows) return;
    c = sp.c, z0 = sp.z0, z1 = sp.z1;
  } else {
    const PlaneSpan sp = plane_span(m, g.nz);
    c = sp.c, z0 = sp.z0, z1 = sp.z1;
  }
  if (z0 >= z1) return;
  const int iy = c / g.nx, ix = c - iy * g.nx;
  const Real *xc = x + c;
  if (m.ry == 2) {
    const unsigned mask = stencil_mask4(g, ix, iy);
    box_walk<Real, 2>(c, z0, z1, g.nx, m.plane, g.nz, code, local,
                      [&](int p, Real *v) {
                        stencil_plane4<Real, false>(xc + (int64_t)p * m.plane, g.nx, mask, (unsigned)p < (unsigned)g.nz, v);
                        return true;
                      },
                      done);
  } else {
    const unsigned mask = stencil_mask(g, ix, iy);
    box_walk<Real, 1>(c, z0, z1, g.nx, m.plane, g.nz, code, local,
                      [&](int p, Real *v) {
                        stencil_plane<Real>(xc + (int64_t)p * m.plane, g.nx, mask, (unsigned)p < (unsigned)g.nz, v);
                        return true;
                      },
                      done);
  }
}

}  // namespace hpccg
