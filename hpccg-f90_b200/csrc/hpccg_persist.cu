// hpccg_persist.cu -- the whole FP64 CG of a small stored system in one kernel.
//
// The graph of hpccg_cg.cu launches three kernels an iteration; below a few
// hundred thousand rows they are shorter than the gaps between them (32^3: 22 us
// an iteration, 15 in kernels of 2 to 8 us).  Here one cooperative launch keeps a
// block per SM resident and an iteration has two grid-wide steps:
//   rows:   p_j = r_j + beta p_j formed where it is gathered (so p needs no step
//           of its own; two p buffers), Ap, the deferred x update, p.Ap
//   rows:   r -= alpha Ap, r.r
// Each ends in grid_sum, which is the barrier too.  The rows are the pattern form
// (hpccg_pattern.cuh) with the reference's operations and order per row; scalars
// follow hpccg_cg.cu step by step (MPI/src/numerics.F90:91-147), every block
// computing them from the same sums.  Dot products are associated per thread,
// warp, block and over the blocks in index order: reproducible, but not the
// graph's order.
// An iteration in us, graph of the same pattern rows | this:
//   gathers  32^3 20.0 | 8.4, 64^3 26.5 | 17.7, 97 x 75 x 61 28.6 | 21.0,
//            100^3 40.7 | 37.4, 128^3 65 | 73, hence kPersistRows
//   boxes    72^3 24.1 | 22.2, 100 x 90 x 51 24.5 | 24.1, 80^3 24.9 | 26.2,
//            96^3 26.6 | 34.8, hence kPersistBoxRows
// At 32^3 it is bound by the two steps' round trips (two hops through L2 of about
// 1 us each and the sums on the way), above by the gathers.
// Where its buffers find no memory or its blocks cannot all be resident, the graph runs.
#include <algorithm>

#include "hpccg_pattern.cuh"
#include "hpccg_persist.cuh"
#include "hpccg_rows.cuh"

namespace hpccg {

constexpr int kPersistThreads = 1024;        // at most, per block
constexpr int kPersistBlocks = 160;          // at most: ten groups of 16
constexpr int kPersistSlots = kPersistBlocks + 16;  // words of one step: the blocks', the groups'
constexpr unsigned kPersistSpin = 1u << 20;  // polls before a barrier gives up (about a second)

struct __align__(16) PersistSlot {
  double v;
  unsigned long long epoch;
};

struct PersistArgs {
  int n;
  const uint16_t *code;
  const PatEntry64 *table;
  int patterns;
  const double *b;
  double *x, *r, *p0, *p1, *Ap;
  CgState *st;
  double *hist;
  int hist_cap;
  PersistSlot *slots;  // [2][kPersistSlots], zero at launch
};

__device__ __forceinline__ void slot_store(PersistSlot *s, double v, unsigned long long epoch) {
  asm volatile(
      "{\n\t.reg .b128 q;\n\tmov.b128 q, {%1, %2};\n\tst.release.gpu.global.b128 [%0], q;\n\t}" ::"l"(s),
      "l"(__double_as_longlong(v)), "l"(epoch)
      : "memory");
}
__device__ __forceinline__ double slot_load(const PersistSlot *s, unsigned long long *epoch) {
  unsigned long long v;
  asm volatile("{\n\t.reg .b128 q;\n\tld.relaxed.gpu.global.b128 q, [%2];\n\tmov.b128 {%0, %1}, q;\n\t}"
               : "=l"(v), "=l"(*epoch)
               : "l"(s)
               : "memory");
  return __longlong_as_double((long long)v);
}

// Polls `slots` (one a lane, lanes < count) for step `epoch`; 0 and *ok = false in a
// lane whose slot did not come within the spin limit.
__device__ __forceinline__ double slot_wait(const PersistSlot *slots, int lane, int count, unsigned long long epoch,
                                            bool *ok) {
  double w = 0.0;
  if (lane < count) {
    unsigned long long e = 0;
    for (unsigned spin = 0; spin < kPersistSpin; ++spin) {
      w = slot_load(slots + lane, &e);
      if (e == epoch) break;
    }
    if (e != epoch) {
      *ok = false;
      w = 0.0;
    }
  }
  return w;
}
// Butterfly over the first W lanes (W a power of two).
template <int W>
__device__ __forceinline__ double lanes_sum(double v) {
#pragma unroll
  for (int o = W / 2; o > 0; o >>= 1) v = __dadd_rn(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// Sum of v over the grid, the same in every thread, and a grid-wide barrier: what
// any thread wrote before it is seen by every thread after it.  A block publishes
// its sum and the step's number as one 16-byte word; the first block of each group
// of 16 polls its group's words and publishes the group's sum the same way, and
// every block polls the (at most ten) group words.  Relaxed polls and one acquire
// fence at the end: an acquire per poll empties L1 every time, and all blocks
// polling all words cost 3.3 us a step more at 128 blocks.  Two arrays of words in
// turn: a block reaches step e + 2 only after all have read step e.  false: a word
// did not come within the spin limit.
__device__ __forceinline__ bool grid_sum(const PersistArgs &g, double v, unsigned long long epoch, double *total) {
  __shared__ double warp_part[kPersistThreads / 32];
  __shared__ double s_total;
  __shared__ int s_ok;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  v = warp_sum(v);
  if (lane == 0) warp_part[wid] = v;
  __syncthreads();  // also: every thread of the block has done its writes
  if (wid == 0) {
    double t = lane < nw ? warp_part[lane] : 0.0;
    t = nw <= 8 ? lanes_sum<8>(t) : lanes_sum<32>(t);
    PersistSlot *slots = g.slots + (epoch & 1) * kPersistSlots, *groups = slots + kPersistBlocks;
    if (lane == 0) slot_store(slots + blockIdx.x, t, epoch);
    const int ngroup = ((int)gridDim.x + 15) / 16;
    bool ok = true;
    if (blockIdx.x % 16 == 0) {
      double q = slot_wait(slots + blockIdx.x, lane, min(16, (int)gridDim.x - (int)blockIdx.x), epoch, &ok);
      asm volatile("fence.acq_rel.gpu;" ::: "memory");
      ok = __all_sync(0xffffffffu, ok);
      q = lanes_sum<16>(q);
      if (ok && lane == 0) slot_store(groups + blockIdx.x / 16, q, epoch);
    }
    double sum = ok ? slot_wait(groups, lane, ngroup, epoch, &ok) : 0.0;
    asm volatile("fence.acq_rel.gpu;" ::: "memory");
    ok = __all_sync(0xffffffffu, ok);
    sum = lanes_sum<16>(sum);
    if (lane == 0) {
      s_total = sum;
      s_ok = ok;
    }
  }
  __syncthreads();
  *total = s_total;
  return s_ok != 0;
}

struct StatusWord {
  int *w;
  __device__ void set(int v) const { atomicExch(w, v); }
  __device__ void set_if_ok(int v) const { atomicCAS(w, HPCCG_OK, v); }
};

// THREADS: of a block, at most (its registers).  ONE: every thread has at most one
// row, whose r, p, x and Ap stay in registers; only the neighbours' r and p are
// loaded.
template <int THREADS, bool ONE>
__global__ void __launch_bounds__(THREADS, 1) k_cg_persist(const __grid_constant__ PersistArgs g) {
  __shared__ PatEntry64 table[kPatLocal * kPatW];
  for (int i = threadIdx.x; i < g.patterns * kPatW; i += blockDim.x) table[i] = g.table[i];
  __syncthreads();
  constexpr int kUnroll = THREADS <= 512 ? 27 : 9;
  const int n = g.n, tid = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
  const bool lead = tid == 0;
  const int max_iter = g.st->max_iter;
  const double tolerance = g.st->tolerance;
  unsigned long long epoch = 1;
  double part = 0.0, rtrans = 0.0;
  double r1 = 0.0, p1 = 0.0, x1 = 0.0, a1 = 0.0;  // ONE: the thread's row
  const PatEntry64 *t1 = table + (ONE && tid < n ? g.code[tid] : 0) * kPatW;
  bool ok;
  // prepare (:91-104): r = b - A x
  for (int i = tid; i < n; i += stride) {
    const PatEntry64 *t = ONE ? t1 : table + g.code[i] * kPatW;
    double s = 0.0;
#pragma unroll kUnroll
    for (int k = 0; k < kPatW; ++k) s = __dadd_rn(s, __dmul_rn(t[k].v, g.x[i + t[k].off]));
    const double ri = __dsub_rn(g.b[i], s);
    g.r[i] = ri;
    if (ONE) {
      r1 = ri;
      x1 = g.x[i];
    }
    part = __dadd_rn(part, __dmul_rn(ri, ri));
    if (ONE) break;
  }
  ok = grid_sum(g, part, epoch++, &rtrans);
  double normr = sqrt(rtrans), alpha = 0.0, beta = 0.0;
  int k = 1, niters = 0, status = HPCCG_OK;
  bool pending = false;  // x += alpha p of the last iteration is due
  if (lead && g.hist_cap > 0) g.hist[0] = normr;
  bool cont = ok && max_iter >= 1 && !(normr < tolerance);
  if (lead && cont && g.hist_cap > 1) g.hist[1] = normr;
  const double *po = g.p0;  // p of the iteration before
  double *pn = g.p1;
  while (cont) {
    part = 0.0;
    for (int i = tid; i < n; i += stride) {
      const PatEntry64 *t = ONE ? t1 : table + g.code[i] * kPatW;
      double s = 0.0, pi = ONE ? r1 : g.r[i];
      if (k == 1) {  // p = r
#pragma unroll kUnroll
        for (int j = 0; j < kPatW; ++j) s = __dadd_rn(s, __dmul_rn(t[j].v, g.r[i + t[j].off]));
      } else {
#pragma unroll kUnroll
        for (int j = 0; j < kPatW; ++j) {
          const int c = i + t[j].off;
          s = __dadd_rn(s, __dmul_rn(t[j].v, __dadd_rn(g.r[c], __dmul_rn(beta, po[c]))));
        }
        const double pold = ONE ? p1 : po[i];
        const double xi = __dadd_rn(ONE ? x1 : g.x[i], __dmul_rn(alpha, pold));
        if (ONE) x1 = xi;
        else g.x[i] = xi;
        pi = __dadd_rn(pi, __dmul_rn(beta, pold));
      }
      pn[i] = pi;
      if (ONE) {
        p1 = pi;
        a1 = s;
      } else {
        g.Ap[i] = s;
      }
      part = __dadd_rn(part, __dmul_rn(pi, s));
      if (ONE) break;
    }
    pending = false;
    double pAp;
    if (!(ok = grid_sum(g, part, epoch++, &pAp))) break;
    const double a = rtrans / pAp;
    if (!isfinite(a)) {
      status = HPCCG_ERR_BREAKDOWN;
      break;
    }
    alpha = a;
    part = 0.0;
    for (int i = tid; i < n; i += stride) {
      const double ri = __dadd_rn(ONE ? r1 : g.r[i], __dmul_rn(-alpha, ONE ? a1 : g.Ap[i]));
      g.r[i] = ri;
      if (ONE) r1 = ri;
      part = __dadd_rn(part, __dmul_rn(ri, ri));
      if (ONE) break;
    }
    double rr;
    if (!(ok = grid_sum(g, part, epoch++, &rr))) break;
    niters = k;
    pending = true;
    cont = k + 1 <= max_iter && !(normr < tolerance);
    if (cont) {
      ++k;
      beta = rr / rtrans;
      rtrans = rr;
      normr = sqrt(rr);
      if (lead && k < g.hist_cap) g.hist[k] = normr;
      double *q = pn;
      pn = const_cast<double *>(po);
      po = q;
    }
  }
  for (int i = tid; i < n; i += stride) {
    if (ONE || pending) {
      const double xi = ONE ? x1 : g.x[i];
      g.x[i] = pending && ok ? __dadd_rn(xi, __dmul_rn(alpha, ONE ? p1 : pn[i])) : xi;
    }
  }
  persist_report(StatusWord{&g.st->status}, lead, ok, status);
  if (lead) {
    g.st->rtrans = rtrans;
    g.st->normr = normr;
    g.st->niters = niters;
  }
}

bool cg_persist_fits(const hpccg_ctx *c) {
  if (c->persist_off || c->spmv_kind != kSpmvPattern || !c->pat.count) return false;
  return c->nrow <= (spmv_args(c).pat_box ? kPersistBoxRows : kPersistRows);
}

int cg_persist(hpccg_ctx *c, bool *launched) {
  *launched = false;
  cudaError_t e = cudaSuccess;
  if (!c->d_slots && (e = cudaMalloc(&c->d_slots, sizeof(PersistSlot) * 2 * kPersistSlots)) != cudaSuccess)
    c->d_slots = nullptr;
  if (e == cudaSuccess && !c->d_p2 && (e = cudaMalloc(&c->d_p2, sizeof(double) * (size_t)c->npad)) != cudaSuccess)
    c->d_p2 = nullptr;
  if (e != cudaSuccess) return optional_table(e);
  // one row a thread while that fills no more than a block per SM (its rows in
  // registers), in blocks of 256 or 512 threads; else blocks of 1024
  const int sms = std::min(c->num_sms, kPersistBlocks);
  const int threads = (int64_t)256 * sms >= c->nrow ? 256 : ((int64_t)512 * sms >= c->nrow ? 512 : kPersistThreads);
  const int blocks = std::min(sms, (c->nrow + threads - 1) / threads);
  HPCCG_CUDA(cudaMemsetAsync(c->d_slots, 0, sizeof(PersistSlot) * 2 * kPersistSlots, c->stream));
  PersistArgs g;
  g.n = c->nrow;
  g.code = c->pat.code;
  g.table = c->pat.t64;
  g.patterns = c->pat.count;
  g.b = c->d_b;
  g.x = c->d_x;
  g.r = c->d_r;
  g.p0 = c->d_p;
  g.p1 = c->d_p2;
  g.Ap = c->d_Ap;
  g.st = c->d_state;
  g.hist = c->d_hist;
  g.hist_cap = c->hist_cap;
  g.slots = static_cast<PersistSlot *>(c->d_slots);
  void *args[] = {&g};
  const void *kern = threads == 256   ? (const void *)k_cg_persist<256, true>
                     : threads == 512 ? (const void *)k_cg_persist<512, true>
                                      : (const void *)k_cg_persist<kPersistThreads, false>;
  e = cudaLaunchCooperativeKernel(kern, dim3(blocks), dim3(threads), args, 0, c->stream);
  if (e == cudaErrorCooperativeLaunchTooLarge) {  // the process has fewer SMs than the device
    cudaGetLastError();
    c->persist_off = true;
    return HPCCG_OK;
  }
  *launched = e == cudaSuccess;
  return optional_table(e);
}

}  // namespace hpccg
