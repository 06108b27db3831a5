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
// out->count = 0 when there are more.  Synchronises the stream.
int row_patterns(const int32_t *ell_col, const double *ell_val, int npad, int n, int max_count, int num_sms,
                 cudaStream_t s, RowPatterns *out);
void free_patterns(RowPatterns *p);

__device__ __forceinline__ double pat_term(double s, const PatEntry64 &e, const double *__restrict__ x) {
  return __dadd_rn(s, __dmul_rn(e.v, __ldg(x + e.off)));  // the ELL kernels' operations
}
__device__ __forceinline__ float pat_term(float s, const PatEntry32 &e, const float *__restrict__ x) {
  return fmaf(e.v, __ldg(x + e.off), s);
}

// Sums of G rows (row(r), r < count), handed to done(row, sum) in order; a row's
// terms are added in slot order, as in the ELL kernels.  `table` is the block's
// copy in shared memory: a warp whose lanes share a pattern reads one address.
// SHARE: the rows lie along a walk of the grid and mostly have one pattern, so
// when all G agree each entry is read once for them.
template <int G, bool SHARE, typename Real, typename Entry, class Row, class Done>
__device__ __forceinline__ void pattern_group(Row &&row, int count, const uint16_t *__restrict__ code,
                                              const Entry *table, const Real *__restrict__ x, Done &&done) {
  int t[G];
  bool same = count == G;
#pragma unroll
  for (int r = 0; r < G; ++r) {
    t[r] = (r < count ? (int)__ldg(code + row(r)) : 0) * kPatW;
    same = same && t[r] == t[0];
  }
  Real s[G];
#pragma unroll
  for (int r = 0; r < G; ++r) s[r] = Real(0);
  if (SHARE && same) {
#pragma unroll 9
    for (int k = 0; k < kPatW; ++k) {
      const Entry e = table[t[0] + k];
#pragma unroll
      for (int r = 0; r < G; ++r) s[r] = pat_term(s[r], e, x + row(r));
    }
  } else if (!SHARE) {
#pragma unroll 9
    for (int k = 0; k < kPatW; ++k)
#pragma unroll
      for (int r = 0; r < G; ++r)
        if (r < count) s[r] = pat_term(s[r], table[t[r] + k], x + row(r));
  } else {
#pragma unroll
    for (int r = 0; r < G; ++r)
      if (r < count)
#pragma unroll 9
        for (int k = 0; k < kPatW; ++k) s[r] = pat_term(s[r], table[t[r] + k], x + row(r));
  }
#pragma unroll
  for (int r = 0; r < G; ++r)
    if (r < count) done(row(r), s[r]);
}

// The block's copy of the table.
template <typename Entry>
__device__ __forceinline__ const Entry *pattern_table(const Entry *__restrict__ table, int count) {
  __shared__ Entry local[kPatLocal * kPatW];
  for (int i = threadIdx.x; i < count * kPatW; i += blockDim.x) local[i] = table[i];
  __syncthreads();
  return local;
}

// The calling thread's rows under a map of the grid, in the order of thread_rows
// (hpccg_rows.cuh): the column pair of a tile or two-line map two planes at a
// time, or a column two planes at a time.
template <typename Real, typename Entry, class Done>
__device__ __forceinline__ void pattern_walk(int n, const PlaneMap &m, const uint16_t *__restrict__ code,
                                             const Entry *__restrict__ table, int count, const Real *__restrict__ x,
                                             Done &&done) {
  const Entry *local = pattern_table(table, count);
  if (m.ry == 2) {
    int c, z0, z1;
    if (m.tiles_x > 0) {
      const TileSpan sp = tile_span(m, n / m.plane);
      if (!sp.rows) return;
      c = sp.c, z0 = sp.z0, z1 = sp.z1;
    } else {
      const PlaneSpan sp = plane_span(m, n / m.plane);
      c = sp.c, z0 = sp.z0, z1 = sp.z1;
    }
    for (int z = z0; z < z1; z += 2) {
      const int i = c + z * m.plane;
      pattern_group<4, true>([&](int r) { return i + (r & 1) * m.nx + (r >> 1) * m.plane; }, min(4, 2 * (z1 - z)), code,
                             local, x, done);
    }
  } else {
    const PlaneSpan sp = plane_span(m, n / m.plane);
    for (int z = sp.z0; z < sp.z1; z += 2) {
      const int i = sp.c + z * m.plane;
      pattern_group<2, true>([&](int r) { return i + r * m.plane; }, min(2, sp.z1 - z), code, local, x, done);
    }
  }
}
// Grid-stride rows, one at a time.
template <typename Real, typename Entry, class Done>
__device__ __forceinline__ void pattern_stride(int n, const uint16_t *__restrict__ code,
                                               const Entry *__restrict__ table, int count,
                                               const Real *__restrict__ x, Done &&done) {
  const Entry *local = pattern_table(table, count);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    pattern_group<1, false>([&](int) { return i; }, 1, code, local, x, done);
}

}  // namespace hpccg
