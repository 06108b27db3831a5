// hpccg_pattern.cu -- finds the row patterns of a stored matrix (hpccg_pattern.cuh).
#include <algorithm>
#include <vector>

#include "hpccg_pattern.cuh"

namespace hpccg {

constexpr int kPatSlots = 1 << 14;  // hash table; a quarter full at most
constexpr int kPatMax = kPatSlots / 4;

struct PatTable {
  unsigned long long key[kPatSlots];  // 0 = free
  int rep[kPatSlots];                 // smallest row with the key
  int id[kPatSlots];                  // pattern number
  int rows[kPatMax];                  // representative row of each pattern
  int count;                          // keys inserted
  int bad;                            // a row that differs from its pattern (equal keys)
};

// 64-bit key of row i (never 0): each slot's offset and value bits mixed in order.
__device__ __forceinline__ unsigned long long row_key(const int32_t *col, const double *val, int npad, int i) {
  unsigned long long h = 0x9E3779B97F4A7C15ull;
#pragma unroll
  for (int k = 0; k < kPatW; ++k) {
    const size_t o = (size_t)k * npad + i;
    const unsigned long long a = (unsigned long long)(unsigned)(__ldcs(col + o) - i);
    const unsigned long long b = (unsigned long long)__double_as_longlong(__ldcs(val + o));
    h = (h ^ a) * 0xBF58476D1CE4E5B9ull;
    h = ((h ^ (h >> 29)) ^ b) * 0x94D049BB133111EBull;
    h ^= h >> 32;
  }
  return h | 1ull;
}

// The table slot of a key; with `row` >= 0 the key is inserted if it is new
// (-1 when the table is full enough to give up).
__device__ __forceinline__ int key_slot(PatTable *t, unsigned long long key, int row, int max_count) {
  int s = (int)(key >> 40) & (kPatSlots - 1);
  for (int probe = 0; probe < kPatSlots; ++probe, s = (s + 1) & (kPatSlots - 1)) {
    unsigned long long k = *(volatile unsigned long long *)&t->key[s];
    if (row >= 0 && *(volatile int *)&t->count > max_count) return -1;
    if (k == 0 && row >= 0) {
      k = atomicCAS(&t->key[s], 0ull, key);
      if (k == 0) {
        atomicAdd(&t->count, 1);
        k = key;
      }
    }
    if (k == key) return s;
    if (k == 0) return -1;
  }
  return -1;
}

__global__ void k_pat_insert(const int32_t *col, const double *val, int npad, int n, int max_count, PatTable *t) {
  unsigned long long last = 0;
  int s = -1;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    if (*(volatile int *)&t->count > max_count) return;
    const unsigned long long key = row_key(col, val, npad, i);
    if (key != last) {
      last = key;
      s = key_slot(t, key, i, max_count);
      // a thread's rows ascend: only the first of a run can lower the minimum
      if (s >= 0 && *(volatile int *)&t->rep[s] > i) atomicMin(&t->rep[s], i);
    }
  }
}

__global__ void k_pat_fill(const int32_t *col, const double *val, int npad, const PatTable *t, int count,
                           PatEntry64 *t64, PatEntry32 *t32, PatEntry32 *t16) {
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < count * kPatW; e += gridDim.x * blockDim.x) {
    const int row = t->rows[e / kPatW];
    const size_t o = (size_t)(e % kPatW) * npad + row;
    const int32_t off = col[o] - row;
    const double v = val[o];
    t64[e] = PatEntry64{v, off, 0};
    t32[e] = PatEntry32{off, (float)v};
    t16[e] = PatEntry32{off, __bfloat162float(__double2bfloat16(v))};
  }
}

// Each row's code, and the row compared with its table entry slot by slot.
__global__ void k_pat_assign(const int32_t *col, const double *val, int npad, int n, PatTable *t,
                             const PatEntry64 *t64, uint16_t *code) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int s = key_slot(t, row_key(col, val, npad, i), -1, 0);
    const int id = s >= 0 ? t->id[s] : -1;
    bool same = id >= 0;
    for (int k = 0; k < kPatW && same; ++k) {
      const size_t o = (size_t)k * npad + i;
      const PatEntry64 p = t64[(size_t)id * kPatW + k];
      same = col[o] - i == p.off && __double_as_longlong(val[o]) == __double_as_longlong(p.v);
    }
    if (!same) t->bad = 1;
    code[i] = (uint16_t)(same ? id : 0);
  }
}

void free_patterns(RowPatterns *p) {
  if (p->memory) cudaFree(p->memory);
  *p = RowPatterns{};
}

int row_patterns(const int32_t *ell_col, const double *ell_val, int npad, int n, int max_count, int num_sms,
                 cudaStream_t s, RowPatterns *out) {
  free_patterns(out);
  if (n < 1 || max_count < 1) return HPCCG_OK;
  max_count = std::min(max_count, kPatMax);
  // one allocation (each costs a synchronisation when it is freed): the search's
  // table, the tables, the codes
  const size_t most = (size_t)max_count * kPatW;
  size_t bytes = 0;
  auto part = [&](size_t n) {
    const size_t at = bytes;
    bytes += (n + 255) / 256 * 256;
    return at;
  };
  const size_t at_t = part(sizeof(PatTable)), at64 = part(sizeof(PatEntry64) * most), at32 = part(sizeof(PatEntry32) * most),
               at16 = part(sizeof(PatEntry32) * most), b64 = part(sizeof(double) * most),
               b32 = part(sizeof(float) * most), b16 = part(sizeof(float) * most), atf = part(sizeof(int)),
               atc = part(sizeof(uint16_t) * (size_t)npad);
  if (cudaError_t e = cudaMalloc(&out->memory, bytes); e != cudaSuccess) {
    out->memory = nullptr;
    return optional_table(e);
  }
  unsigned char *mem = static_cast<unsigned char *>(out->memory);
  PatTable *t = reinterpret_cast<PatTable *>(mem + at_t);
  out->t64 = reinterpret_cast<PatEntry64 *>(mem + at64);
  out->t32 = reinterpret_cast<PatEntry32 *>(mem + at32);
  out->t16 = reinterpret_cast<PatEntry32 *>(mem + at16);
  out->box64 = reinterpret_cast<double *>(mem + b64);
  out->box32 = reinterpret_cast<float *>(mem + b32);
  out->box16 = reinterpret_cast<float *>(mem + b16);
  out->flag = reinterpret_cast<int *>(mem + atf);
  out->code = reinterpret_cast<uint16_t *>(mem + atc);
  const int grid = (int)std::max<int64_t>(1, std::min<int64_t>(((int64_t)n + kBlock - 1) / kBlock, (int64_t)num_sms * 8));
  std::vector<int> rep(kPatSlots), id(kPatSlots, -1), rows;
  int flags[2] = {0, 0};
  cudaError_t e = cudaMemsetAsync(t, 0, sizeof(PatTable), s);
  if (e == cudaSuccess) e = cudaMemsetAsync(t->rep, 0x7f, sizeof(t->rep), s);
  if (e == cudaSuccess) {
    k_pat_insert<<<grid, kBlock, 0, s>>>(ell_col, ell_val, npad, n, max_count, t);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpyAsync(rep.data(), t->rep, sizeof(t->rep), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(flags, &t->count, sizeof(flags), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e == cudaSuccess && flags[0] <= max_count) {
    // patterns in the order of their first rows
    std::vector<std::pair<int, int>> found;
    for (int k = 0; k < kPatSlots; ++k)
      if (rep[k] < n) found.push_back({rep[k], k});
    std::sort(found.begin(), found.end());
    for (size_t k = 0; k < found.size(); ++k) {
      id[found[k].second] = (int)k;
      rows.push_back(found[k].first);
    }
    const size_t ne = found.size() * kPatW;
    if (e == cudaSuccess) e = cudaMemsetAsync(out->code, 0, sizeof(uint16_t) * (size_t)npad, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(t->id, id.data(), sizeof(t->id), cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(t->rows, rows.data(), sizeof(int) * rows.size(), cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) {
      k_pat_fill<<<(int)((ne + 255) / 256), 256, 0, s>>>(ell_col, ell_val, npad, t, (int)rows.size(), out->t64,
                                                         out->t32, out->t16);
      k_pat_assign<<<grid, kBlock, 0, s>>>(ell_col, ell_val, npad, n, t, out->t64, out->code);
      e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(&flags[1], &t->bad, sizeof(int), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e == cudaSuccess && !flags[1]) out->count = (int)rows.size();
  }
  if (e != cudaSuccess || !out->count) free_patterns(out);
  return optional_table(e);
}

// One thread per pattern: its entries (without the padding slots, offset 0 and value
// +0.0, at the end) at their places of the 3x3x3 box, in order; *bad where one has none
// or the grid is narrower than a box (its neighbours' offsets coincide, so that a place
// would be found, but not always the right one).  place (may be null): each pattern's
// own (nx, ny, box number), nx = 0 for none.
__global__ void k_pat_boxes(const PatEntry64 *t64, int count, int nx, int ny, const int4 *place, double *box64,
                            float *box32, float *box16, int *bad) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= count) return;
  int at = c;
  if (place) {
    nx = place[c].x;
    ny = place[c].y;
    at = place[c].z;
    if (nx == 0) return;
  }
  if (nx < 3 || ny < 3) {
    *bad = 1;
    return;
  }
  const PatEntry64 *row = t64 + (size_t)c * kPatW;
  int len = kPatW;
  while (len > 0 && row[len - 1].off == 0 && __double_as_longlong(row[len - 1].v) == 0) --len;
  int k = 0;
  for (int j = 0; j < kPatW; ++j) {
    const int off = ((j / 9 - 1) * ny + (j / 3 % 3 - 1)) * nx + (j % 3 - 1);
    const bool have = k < len && row[k].off == off;
    const double v = have ? row[k].v : 0.0;
    k += have;
    box64[(size_t)at * kPatW + j] = v;
    box32[(size_t)at * kPatW + j] = (float)v;
    box16[(size_t)at * kPatW + j] = __bfloat162float(__double2bfloat16(v));
  }
  if (k != len) *bad = 1;
}

static int fill_boxes(RowPatterns *p, int nx, int ny, const int4 *place, cudaStream_t s);

int pattern_boxes(RowPatterns *p, int nx, int ny, cudaStream_t s) {
  p->boxes = false;
  p->box_nx = nx;
  p->box_ny = ny;
  if (!p->count || nx < 3 || ny < 3) return HPCCG_OK;  // k_pat_boxes would refuse it
  return fill_boxes(p, nx, ny, nullptr, s);
}

int pattern_boxes_placed(RowPatterns *p, const int4 *place, cudaStream_t s) {
  p->boxes = false;
  return p->count ? fill_boxes(p, 0, 0, place, s) : HPCCG_OK;
}

static int fill_boxes(RowPatterns *p, int nx, int ny, const int4 *place, cudaStream_t s) {
  int bad = 1;
  cudaError_t e = cudaMemsetAsync(p->flag, 0, sizeof(int), s);
  if (e == cudaSuccess) {
    k_pat_boxes<<<(p->count + 31) / 32, 32, 0, s>>>(p->t64, p->count, nx, ny, place, p->box64, p->box32, p->box16,
                                                    p->flag);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpyAsync(&bad, p->flag, sizeof(int), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  p->boxes = e == cudaSuccess && !bad;
  return optional_table(e);
}

}  // namespace hpccg
