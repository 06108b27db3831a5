// unet_conv_win.cu -- 3x3x3 convolutions with 16 output channels on tcgen05, the
// weights as the MMA's A operand.
//
// A tcgen05.mma with M = 128 takes ~45 cycles for any N up to 64, 64 cycles for
// N = 128 and 128 for N = 256 (measured): with the voxels as M and the 16 output
// channels as N the tensor pipe runs at 0.18 of its rate.  Here the voxels are N
// and M = 128 holds the 16 output channels of EIGHT output rows (y .. y+7) of
// the same x and z.  An input row contributes to the output rows y-1, y, y+1
// only, so for each (dz, dx) the A operand of input row j of a tile is a window
// of eight 16x16 blocks, block g = W[dy = j - 1 - g] or zero: the weights are laid
// out once per CTA as runs [7 zero blocks][W(+1) W(0) W(-1)][7 zero blocks] per
// (dz, dx, input group), neighbouring runs sharing their zeros, and a window is
// a start address into its run.  A tile of eight rows takes ten input rows x 9
// (dz, dx) MMAs per input group, 0.30 of the multiplications useful, at the full
// MMA rate: 5.8 cycles per voxel and group where the voxels-as-M form takes 13.
// At 256^3 a 16 -> 16 layer went 0.78 -> 0.47 ms and 32 -> 16 (+ projection)
// 1.24 -> 0.81 ms, at 32^3 33 -> 8 us and 46 -> 11 us; the forward pass 3.20 ->
// 2.26 ms (2.48 under the power cap of a long run).  The 32 -> 16 layer is bound
// by the MMAs (0.86 of its time), the 16 -> 16 one by the MMAs and the warp that
// issues them (0.77), small grids by one tile's chain of set-up, first slab, ten
// slabs and drain.  The zero blocks add exact zeros and a voxel's terms keep
// their order (dy, dz, dx, input group), so the outputs are bit for bit those of
// the voxels-as-M form.  Only an infinite or NaN input breaks this: its zero blocks
// make NaNs in rows that it does not touch.  So every output that is not finite is
// formed again from its own taps (win_again), found by 0 * v as it is stored: one
// instruction a pair of channels, the ReLU being part of the conversion to BF16 (the
// forward pass at 256^3 2288 us before and 2277 with it, 64^3 batch 4 gradient 1061
// and 1024; the rows formed again in line instead of in a function: 2306 and 1055).  A
// forward pass at 128^3 with two infinite inputs takes 4.4 ms instead of 0.44.
//
// Columns: a tile spans tc z-planes of one x block (at most 126 voxels); its
// input rows ("slabs": one y, tc+2 z-planes, x block with a one-voxel halo, both
// halves) are one TMA box per input group with pitch txb+2 units, zeros outside
// the grid, so N can run over several z-planes in one MMA (the two halo columns
// between planes are computed and not stored) and taps in x and z are start
// addresses too.  (One bulk copy per row and half cost ~170 cycles of issue each,
// more than the slab's MMAs.)  A unit is a run of tiles in y; its slabs stream
// through a ring once, slabs 8 and 9 of a tile being 0 and 1 of the next.
// conv_win_plan picks tc and the run length.
//
// Roles: warp 0 fetches, warp 1 issues the MMAs, warps 2-9 drain the
// accumulators (two of 256 TMEM columns).  TMEM lanes are (row g, channel),
// columns are voxels; 16x256b loads give each thread two neighbouring voxels of
// one channel, which pack to BF16 pairs, and movmatrix transposes 8 channels x 8
// voxels to the row-planar layout in registers: each store of a warp is one full
// 128-byte line.
#include <algorithm>

#include "unet_conv.cuh"

namespace hpccg {

using namespace tc;

constexpr int kWinRows = 8;    // output rows per tile (M = 128)
constexpr int kWinMaxX = 126;  // x block: with its halo a box of 128 units
constexpr int kWinMaxSlots = 8;
constexpr int kWinBytesPerClk = 20;  // what an SM draws from L2 when all of them do
constexpr int kWinPad = 256;   // MMAs read up to 15 columns past the last slab
constexpr int kWinProjBytes = 8 * 2 * 16 * 17 * 4;  // the projection's transposes, one per epilogue warp
constexpr int kWinSmem = 226 * 1024;  // of the 227 KB a CTA may use; the barriers are static

__host__ __device__ constexpr int win_blocks(int nin) { return 10 * 9 * nin + 7; }
__host__ __device__ constexpr int win_weight_bytes(int nin) { return win_blocks(nin) * kWTapBytes; }

// Axes: r ("rows", the M direction) and c (the columns' planes) are y and z, or
// z and y with zrows.
struct WinPlan {
  int zrows;
  int nr, nc;           // grid extents along r and c
  int sr, sc;           // grid row (b*nz + z)*ny + y per step of r and c
  int txb, nxb;         // x block and count
  int r1, nsub, nn;     // c-planes per MMA, MMAs per tap, columns per MMA (a multiple of 16)
  int inv;              // 65536 / pitch, rounded up: column / pitch = column * inv >> 16 (columns < 256)
  int tc, ntc;          // c-planes per tile (r1 * nsub) and count
  int rows, nru;        // rows per unit (a multiple of kWinRows) and count
  int nunits;
  int plane_bytes, input_bytes, slots;  // one half; one input group of a slab (a multiple of 128); slabs in the ring
};

struct WinArgs {
  ConvArgs a;
  WinPlan p;
  CUtensorMap in[2];  // box: pitch units x (tc + 2) c-planes x 2 halves
};

struct WinUnit {
  int b, c0, x0, ra, rb;
};
__device__ __forceinline__ WinUnit win_unit(const WinPlan &p, int u) {
  WinUnit w;
  const int c = u % p.nru;
  u /= p.nru;
  w.x0 = (u % p.nxb) * p.txb;
  u /= p.nxb;
  w.c0 = (u % p.ntc) * p.tc;
  w.b = u / p.ntc;
  w.ra = c * p.rows;
  w.rb = min(p.nr, w.ra + p.rows);
  return w;
}

// 16 lanes x 32 columns: r[4i], r[4i+1] = lane t/4, columns 8i + 2(t%4) + {0, 1};
// r[4i+2], r[4i+3] = lane t/4 + 8, the same columns.
__device__ __forceinline__ void tmem_ld_16x256_x4(uint32_t taddr, uint32_t *r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
      "%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ uint32_t transpose8x8(uint32_t a) {
  uint32_t d;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(d) : "r"(a));
  return d;
}
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  const __nv_bfloat162 p = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t *>(&p);
}

// The pair, negative numbers as zeros, NaNs as NaNs.
__device__ __forceinline__ uint32_t pack2_relu(float lo, float hi) {
  uint32_t d;
  asm("cvt.rn.relu.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
  return d;
}
__device__ __forceinline__ float max_nan(float a, float b) {  // NaN where either is
  float d;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(d) : "f"(a), "f"(b));
  return d;
}
// Whether a BF16 pair holds an infinity or a NaN; chk collects 0 * v of several.
__device__ __forceinline__ uint32_t zero_times(uint32_t v, uint32_t chk) {
  const __nv_bfloat162 r = __hfma2(*reinterpret_cast<const __nv_bfloat162 *>(&v), __float2bfloat162_rn(0.f),
                                   *reinterpret_cast<const __nv_bfloat162 *>(&chk));
  return *reinterpret_cast<const uint32_t *>(&r);
}
__device__ __forceinline__ bool not_finite(uint32_t v) { return zero_times(v, 0u) & 0x7fff7fffu; }
__device__ __forceinline__ bool not_finite(float v) { return !(0.f * v == 0.f); }

// The sums of one voxel for the output channels co and co + 1 (co even) from its own 27
// taps, outside ones as zeros; the loads of three taps at a time.
template <int NIN>
__device__ __forceinline__ float2 win_direct(const ConvArgs &a, int b, int z, int y, int x, int co) {
  const ConvGeom &g = a.g;
  float s0 = 0.f, s1 = 0.f;
  for (int t = 0; t < 9; ++t) {
    const int zz = z + t / 3 - 1, yy = y + t % 3 - 1;
    const bool line = (unsigned)zz < (unsigned)g.nz && (unsigned)yy < (unsigned)g.ny;
    const int64_t row = ((int64_t)b * g.nz + zz) * g.ny + yy;
#pragma unroll
    for (int k = 0; k < 2 * NIN; ++k) {  // input group, half
      const uint4 *src = reinterpret_cast<const uint4 *>(k >= 2 ? a.in1 : a.in0);
      const uint4 *wp = reinterpret_cast<const uint4 *>(a.wpack) + (((k >> 1) * 27 + 3 * t) * 2 + (k & 1)) * 16 + co;
      uint4 q[3], w[3][2];
#pragma unroll
      for (int dx = 0; dx < 3; ++dx) {
        const int xx = x + dx - 1;
        q[dx] = line && (unsigned)xx < (unsigned)g.nx ? __ldg(src + act_unit(row, k & 1, xx, g.nx)) : make_uint4(0, 0, 0, 0);
        w[dx][0] = __ldg(wp + 32 * dx);
        w[dx][1] = __ldg(wp + 32 * dx + 1);
      }
#pragma unroll
      for (int dx = 0; dx < 3; ++dx) {
        const uint32_t qv[4] = {q[dx].x, q[dx].y, q[dx].z, q[dx].w};
        const uint32_t w0[4] = {w[dx][0].x, w[dx][0].y, w[dx][0].z, w[dx][0].w};
        const uint32_t w1[4] = {w[dx][1].x, w[dx][1].y, w[dx][1].z, w[dx][1].w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float lo = __uint_as_float(qv[j] << 16), hi = __uint_as_float(qv[j] & 0xffff0000u);
          s0 = fmaf(hi, __uint_as_float(w0[j] & 0xffff0000u), fmaf(lo, __uint_as_float(w0[j] << 16), s0));
          s1 = fmaf(hi, __uint_as_float(w1[j] & 0xffff0000u), fmaf(lo, __uint_as_float(w1[j] << 16), s1));
        }
      }
    }
    if (s0 != s0 && s1 != s1) break;
  }
  return make_float2(s0, s1);
}

// Forms again the outputs that this lane has just stored and that are not finite:
// rows r and r + 1, the columns from c0 on of MMA `sub` of unit u, mapped as in the epilogue.
template <int NIN, int EPI>
__device__ __noinline__ void win_again(const WinArgs &w, int u, int r, int sub, int c0, int lane) {
  const ConvArgs &a = w.a;
  const WinPlan &p = w.p;
  const ConvGeom &g = a.g;
  const WinUnit w0 = win_unit(p, u);
  const int pitch = p.txb + 2, tr = lane >> 2, tc2 = (lane & 3) * 2;
  constexpr int kCols = EPI == kEpiProject ? 1 : (EPI == kEpiRawF32 ? 8 : 4);
  for (int i = 0; i < kCols; ++i) {
    const int c = c0 + (EPI == kEpiProject ? lane & 15 : (EPI == kEpiRawF32 ? 8 * (i >> 1) + tc2 + (i & 1) : 8 * i + tr));
    const int zi = p.r1 > 1 ? c * p.inv >> 16 : 0, x = w0.x0 + c - zi * pitch, cc = w0.c0 + sub * p.r1 + zi;
    if (c >= p.nn || zi >= p.r1 || c - zi * pitch >= p.txb || x >= g.nx || cc >= min(p.nc, w0.c0 + p.tc)) continue;
    for (int k = 0; k < (EPI == kEpiProject ? 1 : 4); ++k) {
      const int rr = r + (EPI == kEpiProject ? lane >> 4 : k >> 1), h = k & 1;
      if (rr >= w0.rb) continue;
      const int64_t row = (int64_t)w0.b * g.nz * g.ny + (int64_t)rr * p.sr + (int64_t)cc * p.sc;
      auto sum = [&](int co) { return win_direct<NIN>(a, w0.b, p.zrows ? rr : cc, p.zrows ? cc : rr, x, co); };
      if constexpr (EPI == kEpiProject) {
        float acc = a.proj[16];
        for (int co = 0; co < 16; co += 2) {
          const float2 f = sum(co);
          acc = fmaf(a.proj[co], fmaxf(f.x + a.bias[co], 0.f), acc);
          acc = fmaf(a.proj[co + 1], fmaxf(f.y + a.bias[co + 1], 0.f), acc);
        }
        static_cast<float *>(a.out)[row * g.nx + x] = acc;
      } else if constexpr (EPI == kEpiRawF32) {
        float *o = static_cast<float *>(a.out) + act_unit(row, h, x, g.nx) * 8 + tr;
        if (!not_finite(*o)) continue;
        const float2 f = sum(8 * h + (tr & ~1));
        *o = tr & 1 ? f.y : f.x;
      } else {
        const int64_t at = act_unit(row, h, x, g.nx) * 4 + (lane & 3);
        uint32_t *o = static_cast<uint32_t *>(a.out) + at;
        if (!not_finite(*o)) continue;
        const int co = 8 * h + tc2;
        float2 f = sum(co);
        if (EPI != kEpiMask && a.bias) {
          f.x += a.bias[co];
          f.y += a.bias[co + 1];
        }
        if (EPI == kEpiBiasRelu) f = make_float2(fmaxf(f.x, 0.f), fmaxf(f.y, 0.f));
        uint32_t v = pack2(f.x, f.y);
        if constexpr (EPI == kEpiMask) v = relu_mask2(v, __ldg(reinterpret_cast<const uint32_t *>(a.act) + at));
        *o = v;
      }
    }
  }
}

constexpr int kWinEpiWarps = 8;  // two per TMEM lane quarter
constexpr int kWinThreads = 64 + 32 * kWinEpiWarps;

template <int NIN, int EPI>
__global__ void __launch_bounds__(kWinThreads, 1) k_conv3_win(const __grid_constant__ WinArgs w) {
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ uint64_t full[kWinMaxSlots], empty[kWinMaxSlots], acc_full[2], acc_empty[2], drain;
  __shared__ uint32_t slot;
  const ConvArgs &a = w.a;
  const WinPlan &p = w.p;
  const ConvGeom &g = a.g;
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  constexpr int kWPlane = win_blocks(NIN) * 256;  // one K half (8 input channels) of every block
  uint8_t *sW = smem, *sA = smem + win_weight_bytes(NIN);
  const int pitch = p.txb + 2, slab = NIN * p.input_bytes;
  // the slabs of this CTA's units in order: fetch the next into ring slot sl
  int fu = blockIdx.x, frs = 0;
  WinUnit fq = win_unit(p, fu);
  frs = fq.ra - 1;
  auto fetch = [&](int sl) {
    mbar_expect_tx(&full[sl], NIN * 2 * p.plane_bytes);
#pragma unroll
    for (int in = 0; in < NIN; ++in)
      tma_g2s_5d(sA + sl * slab + in * p.input_bytes, &w.in[in], 2 * (fq.x0 - 1), fq.c0 - 1, 0, frs, fq.b, &full[sl]);
    if (++frs > fq.rb) {
      fu += gridDim.x;
      if (fu < p.nunits) {
        fq = win_unit(p, fu);
        frs = fq.ra - 1;
      }
    }
  };
  int fetched = 0;
  if (threadIdx.x == 0) {
    for (int s = 0; s < p.slots; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&acc_full[s], 1);
      mbar_init(&acc_empty[s], kWinEpiWarps);
    }
    mbar_init(&drain, 1);
    fence_mbar_init();
    chain_wait();
    for (; fetched < p.slots && fu < p.nunits; ++fetched) fetch(fetched);  // under the weights' set-up
  }
  if (warp == 1) {
    tmem_alloc(&slot, 512);
    tmem_relinquish();
  }
  // weights: run (dc * 3 + dx) * NIN + in, its blocks 7, 8, 9 = W(dr = +1, 0, -1); 16-byte units [in][tap][half][co]
  constexpr int kWUnits = NIN * 27 * 32, kWLoads = (kWUnits + kWinThreads - 1) / kWinThreads;
  uint4 wv[kWLoads];
#pragma unroll
  for (int k = 0; k < kWLoads; ++k) {
    const int i = threadIdx.x + k * kWinThreads;
    if (i < kWUnits) wv[k] = __ldg(reinterpret_cast<const uint4 *>(a.wpack) + i);
  }
  for (int i = threadIdx.x; i < win_weight_bytes(NIN) / 16; i += kWinThreads)
    reinterpret_cast<uint4 *>(sW)[i] = make_uint4(0, 0, 0, 0);
  __syncthreads();
#pragma unroll
  for (int k = 0; k < kWLoads; ++k) {
    const int i = threadIdx.x + k * kWinThreads;
    if (i >= kWUnits) break;
    const int co = i & 15, kc = (i >> 4) & 1, tap = (i >> 5) % 27, in = (i >> 5) / 27;
    const int dz = tap / 9, dy = tap / 3 % 3, dx = tap % 3, dr = p.zrows ? dz : dy, dc = p.zrows ? dy : dz;
    const int blk = 10 * ((dc * 3 + dx) * NIN + in) + 9 - dr;
    *reinterpret_cast<uint4 *>(sW + kc * kWPlane + blk * 256 + co * 16) = wv[k];
  }
  fence_proxy_async_smem();  // weights -> tensor-core proxy
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = slot;
  chain_wait();
  chain_release();  // the TMEM is allocated

  if (warp == 0) {
    if (lane == 0) {
      int sl = 0, par = 0;
      bool ok = true;
      while (fu < p.nunits) {
        if (!(ok = mbar_wait(&empty[sl], par, a.err, 51))) break;
        fetch(sl);
        ++fetched;
        if (++sl == p.slots) {
          sl = 0;
          par ^= 1;
        }
      }
      // every issued copy has landed before the CTA may exit
      for (int j = max(0, fetched - p.slots); j < fetched; ++j)
        mbar_wait(&full[j % p.slots], (j / p.slots) & 1, a.err, 52);
    }
  } else if (warp == 1) {
    // the whole warp walks the slabs; one lane issues
    const uint32_t leader = elect_one();
    const uint32_t idesc = idesc_bf16(128, p.nn);
    const uint64_t wd = smem_desc(sW, kWPlane, 128), bd_ring = smem_desc(sA, p.plane_bytes, 128);
    const uint32_t slab16 = slab >> 4, in16 = p.input_bytes >> 4;
    int sl = 0;
    uint32_t par = 0, t0 = 0;  // ring phase; tiles before this unit
    bool ok = true;
    for (int u = blockIdx.x; u < p.nunits && ok; u += gridDim.x) {
      const WinUnit q = win_unit(p, u);
      const int rows = q.rb - q.ra, ntile = (rows + kWinRows - 1) / kWinRows;
      for (int s = 0; s < rows + 2; ++s) {
        if (!(ok = mbar_wait(&full[sl], par, a.err, 53))) break;
        tc_fence_after();
        const uint64_t bds = bd_ring + (uint64_t)(sl * slab16);
        // slab s is row j = s - 8k of tile k, and row 8 or 9 of the tile before
        const int kt = s / kWinRows;
        for (int k = kt - (s % kWinRows <= 1 ? 1 : 0); k <= kt; ++k) {
          if (k < 0 || k >= ntile) continue;
          const int j = s - kWinRows * k;
          const uint32_t t = t0 + k, buf = t & 1;
          if (j == 0 && t >= 2) {
            if (!(ok = mbar_wait(&acc_empty[buf], ((t >> 1) - 1) & 1, a.err, 54))) break;
            tc_fence_after();
          }
          const uint64_t wj = wd + (uint64_t)((9 - j) * 16);
          const uint32_t acc = j > 0;
          for (int sub = 0; sub < p.nsub; ++sub) {
            const uint32_t d = tmem + buf * 256 + sub * p.nn;
            uint64_t bd = bds + (uint64_t)(sub * p.r1 * pitch);
#pragma unroll
            for (int dc = 0; dc < 3; ++dc, bd += (uint64_t)pitch)
#pragma unroll
              for (int dx = 0; dx < 3; ++dx)
#pragma unroll
                for (int in = 0; in < NIN; ++in)
                  mma_bf16_warp(d, wj + (uint64_t)(160 * ((dc * 3 + dx) * NIN + in)),
                                bd + (uint64_t)dx + (uint64_t)(in * in16), idesc,
                                dc > 0 || dx > 0 || in > 0 ? 1u : acc, leader);
          }
          if (j == min(kWinRows, rows - kWinRows * k) + 1) mma_commit_warp(&acc_full[buf], leader);
        }
        if (!ok) break;
        mma_commit_warp(&empty[sl], leader);
        if (++sl == p.slots) {
          sl = 0;
          par ^= 1;
        }
      }
      t0 += ntile;
    }
    mma_commit_warp(&drain, leader);
    mbar_wait(&drain, 0, a.err, 55);
  } else {
    // the TMEM lane quarter of this warp (rows 2q and 2q+1 of a tile) and its share of the columns
    const int q = warp & 3, part = (warp - 2) >> 2;
    float *stage = reinterpret_cast<float *>(sA + p.slots * NIN * p.input_bytes + kWinPad) + (warp - 2) * (2 * 16 * 17);
    const int tr = lane >> 2, tc2 = (lane & 3) * 2;
    float b0 = 0.f, b1 = 0.f, proj[17];
    if (EPI == kEpiProject) {
      b0 = a.bias[lane & 15];
#pragma unroll
      for (int c = 0; c < 17; ++c) proj[c] = a.proj[c];
    } else if (EPI != kEpiRawF32 && EPI != kEpiMask && a.bias) {
      b0 = a.bias[tr];
      b1 = a.bias[tr + 8];
    }
    uint32_t t = 0;
    bool ok = true;
    for (int u = blockIdx.x; u < p.nunits && ok; u += gridDim.x) {
      const WinUnit w0 = win_unit(p, u);
      const int xe = min(p.txb, g.nx - w0.x0), ce = min(p.tc, p.nc - w0.c0);
      for (int r0 = w0.ra; r0 < w0.rb; r0 += kWinRows, ++t) {
        if (!(ok = mbar_wait(&acc_full[t & 1], (t >> 1) & 1, a.err, 56))) break;
        tc_fence_after();
        const int r = r0 + 2 * q;  // this warp's rows r and r + 1
        const bool rok[2] = {r < w0.rb, r + 1 < w0.rb};
        const uint32_t base = tmem + ((uint32_t)(q * 32) << 16) + (t & 1) * 256;
        const int64_t row0 = (int64_t)w0.b * g.nz * g.ny + (int64_t)r * p.sr + (int64_t)w0.c0 * p.sc;
        for (int sub = 0; sub < p.nsub && sub * p.r1 < ce; ++sub) {
          // column c is c-plane ci of the tile and voxel x of the block, if it is one
          auto column = [&](int c, int *ci) -> int {
            const int zi = p.r1 > 1 ? c * p.inv >> 16 : 0, x = c - zi * pitch;
            *ci = sub * p.r1 + zi;
            return zi < p.r1 && x < xe && *ci < ce ? x : -1;
          };
          // (the loads of the accumulators and the transposes take the whole warp)
          if constexpr (EPI == kEpiProject) {
            for (int c0 = 16 * part; c0 < p.nn; c0 += 32, __syncwarp()) {
              float v[16];
              tmem_ld16(base + sub * p.nn + c0, v);
              __syncwarp();  // the previous columns' sums have been read
#pragma unroll
              for (int k = 0; k < 16; ++k)
                stage[((lane >> 4) * 16 + k) * 17 + (lane & 15)] = max_nan(v[k] + b0, 0.f);
              __syncwarp();
              float acc = proj[16];
#pragma unroll
              for (int c = 0; c < 16; ++c) acc = fmaf(proj[c], stage[lane * 17 + c], acc);
              int ci;
              const int x = column(c0 + (lane & 15), &ci), gs = lane >> 4;
              if (x >= 0 && rok[gs]) {
                static_cast<float *>(a.out)[(row0 + gs * p.sr + (int64_t)ci * p.sc) * g.nx + w0.x0 + x] = acc;
                if (not_finite(acc)) win_again<NIN, EPI>(w, u, r, sub, c0, lane);
              }
            }
          } else {
            for (int c0 = 32 * part; c0 < p.nn; c0 += 64, __syncwarp()) {
              uint32_t act[EPI == kEpiMask ? 4 : 1][2][2];  // all loads of the mask ahead of the sums
              if constexpr (EPI == kEpiMask) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                  int ci = 0;
                  const int x = c0 + 8 * i < p.nn ? column(c0 + 8 * i + tr, &ci) : -1;
                  const uint32_t *m = reinterpret_cast<const uint32_t *>(a.act) +
                                      act_unit(row0 + (int64_t)ci * p.sc, 0, w0.x0 + x, g.nx) * 4 + (lane & 3);
#pragma unroll
                  for (int gs = 0; gs < 2; ++gs)
#pragma unroll
                    for (int h = 0; h < 2; ++h)
                      act[i][gs][h] = x >= 0 && rok[gs] ? __ldg(m + ((int64_t)gs * p.sr * 2 + h) * g.nx * 4) : 0;
                }
              }
              uint32_t d[2][16], chk = 0;  // 0 * what is stored
              float zero = 0.f;
              tmem_ld_16x256_x4(base + sub * p.nn + c0, d[0]);
              tmem_ld_16x256_x4(base + (16u << 16) + sub * p.nn + c0, d[1]);
              tmem_wait_ld();
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                if (c0 + 8 * i >= p.nn) break;
                if constexpr (EPI == kEpiRawF32) {
                  // eight channels of one voxel are a full 32-byte sector
#pragma unroll
                  for (int e = 0; e < 2; ++e) {
                    int ci;
                    const int x = column(c0 + 8 * i + tc2 + e, &ci);
                    if (x < 0) continue;
                    float *o = static_cast<float *>(a.out) +
                               act_unit(row0 + (int64_t)ci * p.sc, 0, w0.x0 + x, g.nx) * 8 + tr;
#pragma unroll
                    for (int gs = 0; gs < 2; ++gs)
                      if (rok[gs])
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                          const float v = __uint_as_float(d[gs][4 * i + 2 * h + e]);
                          o[((int64_t)gs * p.sr * 2 + h) * g.nx * 8] = v;
                          zero = fmaf(0.f, v, zero);
                        }
                  }
                } else {
                  int ci;
                  const int x = column(c0 + 8 * i + tr, &ci);
                  uint32_t *o = static_cast<uint32_t *>(a.out) +
                                act_unit(row0 + (int64_t)ci * p.sc, 0, w0.x0 + x, g.nx) * 4 + (lane & 3);
#pragma unroll
                  for (int gs = 0; gs < 2; ++gs)
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                      const float bias = h ? b1 : b0;
                      float lo = __uint_as_float(d[gs][4 * i + 2 * h]);
                      float hi = __uint_as_float(d[gs][4 * i + 2 * h + 1]);
                      if (EPI != kEpiMask) {
                        lo += bias;
                        hi += bias;
                      }
                      // channels tc2, tc2+1 of half h, voxel tr
                      uint32_t v = transpose8x8(EPI == kEpiBiasRelu ? pack2_relu(lo, hi) : pack2(lo, hi));
                      if constexpr (EPI == kEpiMask) v = relu_mask2(v, act[i][gs][h]);
                      if (x >= 0 && rok[gs]) {
                        o[((int64_t)gs * p.sr * 2 + h) * g.nx * 4] = v;
                        chk = zero_times(v, chk);
                      }
                    }
                }
              }
              if (EPI == kEpiRawF32 ? !(zero == 0.f) : (chk & 0x7fff7fffu) != 0) win_again<NIN, EPI>(w, u, r, sub, c0, lane);
            }
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&acc_empty[t & 1]);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

// Axes, tile and run lengths of a volume.  Rows run along y where nx >= 64, along
// z on narrower grids: a voxel's terms are then added in the order (dy, dz, dx)
// or (dz, dy, dx), the order of brick tiles on those grids, whose bits the
// outputs keep (either way costs the same).  The lengths are the candidate with
// the fewest cycles in the longest CTA's share: a slab costs its MMAs (max(46, N/2)
// cycles each) or, where that is more, its bytes at kWinBytesPerClk; about 1500
// cycles to fill and drain a unit.
static bool conv_win_plan(const ConvGeom &g, int nin, bool project, int num_sms, WinPlan *best) {
  const int nxb = (g.nx + kWinMaxX - 1) / kWinMaxX, txb = (g.nx + nxb - 1) / nxb, pitch = txb + 2;
  const int avail = kWinSmem - win_weight_bytes(nin) - kWinPad - (project ? kWinProjBytes : 0);
  WinPlan p{};
  p.zrows = g.nx < 64;
  p.nr = p.zrows ? g.nz : g.ny;
  p.nc = p.zrows ? g.ny : g.nz;
  p.sr = p.zrows ? g.ny : 1;
  p.sc = p.zrows ? 1 : g.ny;
  p.txb = txb;
  p.nxb = nxb;
  p.inv = (65536 + pitch - 1) / pitch;
  int64_t best_cost = -1;
  for (int tc = 1; tc <= std::min(p.nc, 14); ++tc) {
    p.nn = ((tc - 1) * pitch + txb + 15) / 16 * 16;
    p.r1 = tc;
    p.nsub = 1;
    if (p.nn > 256) {  // one MMA per c-plane, two planes at most (256 TMEM columns per accumulator)
      p.nn = (txb + 15) / 16 * 16;
      p.r1 = 1;
      p.nsub = tc;
      if (p.nn * p.nsub > 256) break;
    }
    p.tc = tc;
    p.ntc = (p.nc + tc - 1) / tc;
    p.plane_bytes = (tc + 2) * pitch * 16;
    p.input_bytes = (2 * p.plane_bytes + 127) / 128 * 128;
    p.slots = std::min(kWinMaxSlots, avail / (nin * p.input_bytes));
    if (p.slots < 3) break;
    for (int tiles = 1; tiles <= 8; tiles *= 2) {
      p.rows = tiles * kWinRows;
      p.nru = (p.nr + p.rows - 1) / p.rows;
      const int64_t units = (int64_t)p.nru * p.nxb * p.ntc * g.nb;
      if (units >= ((int64_t)1 << 31)) continue;
      p.nunits = (int)units;
      const int64_t waves = (units + num_sms - 1) / num_sms;
      const int rows = std::min(p.rows, p.nr), steps = rows + 2 * ((rows + kWinRows - 1) / kWinRows);
      const int64_t mma = (int64_t)steps * 9 * nin * p.nsub * std::max(46, p.nn / 2);
      const int64_t load = (int64_t)(rows + 2) * nin * p.input_bytes / kWinBytesPerClk;
      const int64_t cost = waves * (std::max(mma, load) + 1500);
      if (best_cost < 0 || cost < best_cost) {
        best_cost = cost;
        *best = p;
      }
    }
  }
  return best_cost >= 0;
}

template <int NIN, int EPI>
static int launch_win(const WinArgs &w, int num_sms, cudaStream_t s) {
  const int smem = win_weight_bytes(NIN) + w.p.slots * NIN * w.p.input_bytes + kWinPad + (EPI == kEpiProject ? kWinProjBytes : 0);
  // the attribute is per device: set every time
  HPCCG_CUDA(cudaFuncSetAttribute(k_conv3_win<NIN, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, kWinSmem));
  HPCCG_CUDA(launch_chained(k_conv3_win<NIN, EPI>, std::min(w.p.nunits, num_sms), kWinThreads, smem, s, w.a.chained, w));
  return HPCCG_OK;
}

int launch_conv3_win(int nin, int epi, const ConvArgs &a, int num_sms, cudaStream_t s) {
  WinArgs w;
  w.a = a;
  if (!conv_win_plan(a.g, nin, epi == kEpiProject, num_sms, &w.p)) return HPCCG_ERR_UNSUPPORTED;
  const ActDim c = w.p.zrows ? kDimY : kDimZ, r = w.p.zrows ? kDimZ : kDimY;
  for (int i = 0; i < nin; ++i)
    if (const int rc = act_tmap(&w.in[i], i ? a.in1 : a.in0, a.g, w.p.txb + 2, c, w.p.tc + 2, kDimH, 2, r, 1)) return rc;
  if (nin == 1) {
    switch (epi) {
      case kEpiBiasRelu: return launch_win<1, kEpiBiasRelu>(w, num_sms, s);
      case kEpiBias: return launch_win<1, kEpiBias>(w, num_sms, s);
      case kEpiProject: return launch_win<1, kEpiProject>(w, num_sms, s);
      case kEpiMask: return launch_win<1, kEpiMask>(w, num_sms, s);
      default: return launch_win<1, kEpiRawF32>(w, num_sms, s);
    }
  }
  switch (epi) {
    case kEpiBiasRelu: return launch_win<2, kEpiBiasRelu>(w, num_sms, s);
    case kEpiBias: return launch_win<2, kEpiBias>(w, num_sms, s);
    case kEpiProject: return launch_win<2, kEpiProject>(w, num_sms, s);
    default: return launch_win<2, kEpiRawF32>(w, num_sms, s);
  }
}

}  // namespace hpccg
