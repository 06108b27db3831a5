// unet_dw.cu -- weight and bias gradients of the U-Net's convolutions.
//
// dW[tap][ci][co] = sum_v X[v + off(tap)][ci] dY[v][co], dbias[co] = sum_v dY[v][co].
// Layers with BF16 inputs run as a GEMM on tcgen05 (k_dW_tc); the 1-channel
// input layer keeps its FP32 input and runs on the CUDA cores (k_dW_in1).
// Both leave one partial per CTA, [block][27*cin + 1][16], which
// k_reduce_partials sums in block order, so gradients are reproducible.
#include <algorithm>

#include "unet_ops.cuh"

namespace hpccg {

using namespace tc;

// ---- BF16 inputs: tcgen05 ------------------------------------------------------------
// The contraction runs over voxels.  Both operands are "MN-major": the
// row-planar layout holds, for 8 channels, 8 consecutive voxels as 128
// contiguous bytes, which is a no-swizzle core matrix of 8 channels x 8 voxels.
// For one x row j of X (three z planes, all input groups) the A operand's M
// index is (input group, half, dz, channel) -- planes of one slab at a uniform
// stride -- and B's N index is (dY row j-1, j, j+1; co): one MMA of M = 128,
// N = 48, K = 16 voxels forms the nine (dz, dy) taps of all channels, and the
// three dx taps are the same A shifted by one voxel (16 bytes) into three
// accumulators of 48 TMEM columns.  So 16 voxels cost 3 MMAs (an N = 48 MMA
// takes the ~46 cycles of an N = 16 one) where a tap-by-tap GEMM needs 27.
// A plane of ones behind each slab's planes gives the bias gradient in the same
// MMAs.  BF16 products are exact in FP32, but the tensor core's accumulation
// truncates: left in TMEM over a CTA's ~450 steps the sums were 5e-6 off at
// 64^3, batch 4, ten times what the FP32 FMA chain of the CUDA cores is
// (4.4e-7).  So the accumulators are drained after at most kDwChain steps and
// added up in registers with rounded FP32 additions (1.6e-7); two accumulator
// sets let the drain run under the next steps' MMAs.
//
// Zeros stand for what lies outside the grid, so an infinity or NaN at a face makes NaNs
// in the sums of taps that leave the grid there.  A sum that is a NaN at the end is formed
// again from the terms inside the grid (dw_again), until it is a NaN for good.
//
// A unit is (batch, z, 8 rows of y, up to 112 voxels of x): its ten dY rows
// (double-buffered) and the X slabs (a ring) arrive by TMA, one box per tensor.
// Rows outside the grid, the x halo and the padding of dY to whole 16-voxel
// steps are zeros.  A's rows past the ones plane read whatever follows in
// shared memory; they only reach accumulator rows that nobody stores.
//
// Against the CUDA-core kernel it replaces (one thread per (tap, ci), each
// re-reading its input voxel from global memory): the 13 layers of a 64^3,
// batch 4 training step 25.7 -> 0.29 ms (the 1-channel layer's 0.05 included).
// Issued by a branch for one lane the MMAs took 0.09 ms more: the gradient of
// that step 1.15 -> 1.05 ms, of 64^3 641 -> 610 us, of 32^3 493 -> 465.  Bound by
// the MMAs, then by start-up, drain and the first copies of each unit.
constexpr int kDwThreads = 192;  // producer warp, MMA warp, four draining warps
constexpr int kDwRows = 8;   // y rows per unit
constexpr int kDwSlots = 4;  // X slabs in flight
constexpr int kDwMaxX = 112;  // with the pitch's 8 more units a box of at most 128
constexpr int kDwChain = 8;  // MMA steps between two drains

struct DwTcArgs {
  ConvGeom g;  // volume and batch only
  const __nv_bfloat16 *x[2], *dy;
  CUtensorMap xmap[2], ymap;  // of them; boxes: pitch units x 3 z x 2 halves; kx units x 2 halves x 10 y
  float *partial;
  int *err;
  int kx;                    // voxels per unit row, a multiple of 16
  int nxb, nyb, nunits;      // x and y blocks, units
};

// a plane's pitch: one-voxel halos, rounded so that every box starts on 128 bytes
__host__ __device__ constexpr int dw_plane_bytes(int kx) { return (kx + 8) * 16; }
__host__ __device__ constexpr int dw_planes(int nin) { return 6 * nin + 1; }
__host__ __device__ constexpr int dw_dy_bytes(int kx) { return (kDwRows + 2) * 2 * kx * 16; }
// dY buffers, slabs, and the planes that the last slab's M = 128 rows read beyond it
__host__ __device__ constexpr int dw_smem_bytes(int nin, int kx) {
  return 2 * dw_dy_bytes(kx) + (kDwSlots * dw_planes(nin) + 16 - dw_planes(nin)) * dw_plane_bytes(kx);
}

// Instruction descriptor: as idesc_bf16, with A and B MN-major (bits 15, 16).
__host__ __device__ constexpr uint32_t idesc_bf16_mn(int M, int N) {
  return idesc_bf16(M, N) | (1u << 15) | (1u << 16);
}

__device__ __forceinline__ void dw_unit(const DwTcArgs &a, int u, int &b, int &z, int &ya, int &yb, int &x0) {
  x0 = (u % a.nxb) * a.kx;
  u /= a.nxb;
  ya = (u % a.nyb) * kDwRows;
  yb = min(a.g.ny, ya + kDwRows);
  u /= a.nyb;
  z = u % a.g.nz;
  b = u / a.g.nz;
}

// The 16 sums at `out` that are NaN, again: this CTA's terms of one tap and input channel
// ci (ci < 0: of the bias), one after the other.
__device__ __noinline__ void dw_again(const DwTcArgs &a, int tap, int ci, float *out) {
  const ConvGeom &g = a.g;
  const int oz = ci < 0 ? 0 : tap / 9 - 1, oy = ci < 0 ? 0 : tap / 3 % 3 - 1, ox = ci < 0 ? 0 : tap % 3 - 1;
  float s[16];
#pragma unroll
  for (int c = 0; c < 16; ++c) s[c] = 0.f;
  for (int u = blockIdx.x; u < a.nunits; u += gridDim.x) {
    int b, z, ya, yb, x0;
    dw_unit(a, u, b, z, ya, yb, x0);
    if ((unsigned)(z + oz) >= (unsigned)g.nz) continue;
    for (int y = ya; y < yb; ++y) {  // the row of X
      if ((unsigned)(y - oy) >= (unsigned)g.ny) continue;
      const int64_t xrow = ((int64_t)b * g.nz + z + oz) * g.ny + y, drow = ((int64_t)b * g.nz + z) * g.ny + y - oy;
#pragma unroll 2
      for (int x = max(x0, -ox); x < min(min(x0 + a.kx, g.nx), g.nx - ox); ++x) {
        const float v = ci < 0 ? 1.f : __bfloat162float(a.x[ci >> 4][act_elem(xrow, x + ox, ci & 15, g.nx)]);
        float d[16];
        load_voxel(a.dy, act_unit(drow, 0, x, g.nx), g.nx, d);
#pragma unroll
        for (int c = 0; c < 16; ++c) s[c] = fmaf(v, d[c], s[c]);
      }
      bool left = false;  // a sum that may still be a number
#pragma unroll
      for (int c = 0; c < 16; ++c) left |= out[c] != out[c] && s[c] == s[c];
      if (!left) return;
    }
  }
#pragma unroll
  for (int c = 0; c < 16; ++c)
    if (out[c] != out[c]) out[c] = s[c];
}

template <int NIN>
__global__ void __launch_bounds__(kDwThreads, 1) k_dW_tc(const __grid_constant__ DwTcArgs a) {
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ uint64_t fullx[kDwSlots], emptyx[kDwSlots], fully[2], emptyy[2], acc_full[2], acc_empty[2], drain;
  __shared__ uint32_t slot;
  constexpr int P = dw_planes(NIN);
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int ps = dw_plane_bytes(a.kx), slab = P * ps, dyb = dw_dy_bytes(a.kx);
  uint8_t *sY = smem, *sX = smem + 2 * dyb;
  for (int s = 0; s < kDwSlots; ++s) {  // the ones planes: written once, no copy touches them
    uint32_t *o = reinterpret_cast<uint32_t *>(sX + s * slab + (P - 1) * ps);
    for (int i = threadIdx.x; i < ps / 4; i += kDwThreads) o[i] = 0x3f803f80u;
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < kDwSlots; ++s) {
      mbar_init(&fullx[s], 1);
      mbar_init(&emptyx[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&fully[s], 1);
      mbar_init(&emptyy[s], 1);
      mbar_init(&acc_full[s], 1);
      mbar_init(&acc_empty[s], 4);
    }
    mbar_init(&drain, 1);
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc(&slot, 512);
    tmem_relinquish();
  }
  fence_proxy_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = slot;
  chain_wait();
  chain_release();  // the TMEM is allocated
  const int ksteps = a.kx / 16, chunk = max(1, kDwChain / ksteps);  // rows between two drains
  auto unit = [&](int u, int &b, int &z, int &ya, int &yb, int &x0) { dw_unit(a, u, b, z, ya, yb, x0); };
  if (warp == 0) {
    if (lane == 0) {
      uint32_t sc = 0, uc = 0;
      bool ok = true;
      for (int u = blockIdx.x; u < a.nunits && ok; u += gridDim.x, ++uc) {
        int b, z, ya, yb, x0;
        unit(u, b, z, ya, yb, x0);
        const int yp = uc & 1;
        if (uc >= 2 && !(ok = mbar_wait(&emptyy[yp], ((uc >> 1) - 1) & 1, a.err, 41))) break;
        mbar_expect_tx(&fully[yp], dyb);
        tma_g2s_5d(sY + yp * dyb, &a.ymap, 2 * x0, 0, ya - 1, z, b, &fully[yp]);
        for (int y = ya; y < yb; ++y, ++sc) {
          const int s = sc % kDwSlots;
          const uint32_t n = sc / kDwSlots;
          if (n > 0 && !(ok = mbar_wait(&emptyx[s], (n - 1) & 1, a.err, 42))) break;
          mbar_expect_tx(&fullx[s], 6 * NIN * ps);
#pragma unroll
          for (int in = 0; in < NIN; ++in)
            tma_g2s_5d(sX + s * slab + in * 6 * ps, &a.xmap[in], 2 * (x0 - 1), z - 1, 0, y, b, &fullx[s]);
        }
      }
      // every issued copy has landed before the CTA may exit
      for (uint32_t j = sc > (uint32_t)kDwSlots ? sc - kDwSlots : 0; j < sc; ++j)
        mbar_wait(&fullx[j % kDwSlots], (j / kDwSlots) & 1, a.err, 43);
      for (uint32_t j = uc > 2u ? uc - 2 : 0; j < uc; ++j) mbar_wait(&fully[j & 1], (j >> 1) & 1, a.err, 44);
    }
  } else if (warp == 1) {
    // the whole warp walks the rows; one lane issues (a branch for one lane takes ~70 cycles an
    // MMA to issue, more than the 46 that it runs)
    const uint32_t leader = elect_one();
    constexpr uint32_t idesc = idesc_bf16_mn(128, 48);
    // MN-major: lbo = distance of 8-voxel groups (K), sbo = of 8-channel groups
    const uint64_t ad0 = smem_desc(sX, 128, ps), bd0 = smem_desc(sY, 128, a.kx * 16);
    const uint32_t slab16 = slab >> 4, dyb16 = dyb >> 4, dyrow16 = 2 * a.kx;
    uint32_t uc = 0, cc = 0, sl = 0, par = 0;  // units, chunks of rows; X ring
    int in_chunk = 0;
    bool ok = true;
    for (int u = blockIdx.x; u < a.nunits && ok; u += gridDim.x, ++uc) {
      int b, z, ya, yb, x0;
      unit(u, b, z, ya, yb, x0);
      if (!(ok = mbar_wait(&fully[uc & 1], (uc >> 1) & 1, a.err, 45))) break;
      uint64_t brow = bd0 + (uint64_t)((uc & 1) * dyb16);
      for (int y = ya; y < yb; ++y, brow += dyrow16) {
        if (in_chunk == 0 && cc >= 2 && !(ok = mbar_wait(&acc_empty[cc & 1], ((cc >> 1) - 1) & 1, a.err, 48))) break;
        if (!(ok = mbar_wait(&fullx[sl], par, a.err, 46))) break;
        tc_fence_after();
        const uint32_t d = tmem + 256 * (cc & 1);
        uint64_t ad = ad0 + (uint64_t)(sl * slab16), bd = brow;
        uint32_t more = in_chunk > 0;
        for (int k = 0; k < ksteps; ++k, ad += 16, bd += 16, more = 1)
#pragma unroll
          for (int dx = 0; dx < 3; ++dx) mma_bf16_warp(d + 48 * dx, ad + dx, bd, idesc, more, leader);
        mma_commit_warp(&emptyx[sl], leader);
        if (++sl == kDwSlots) {
          sl = 0;
          par ^= 1;
        }
        if (++in_chunk == chunk) {
          mma_commit_warp(&acc_full[cc & 1], leader);
          in_chunk = 0;
          ++cc;
        }
      }
      if (!ok) break;
      mma_commit_warp(&emptyy[uc & 1], leader);
    }
    if (ok && in_chunk) mma_commit_warp(&acc_full[cc & 1], leader);
    mma_commit_warp(&drain, leader);
    mbar_wait(&drain, 0, a.err, 47);
  } else {
    int rows = 0;
    for (int u = blockIdx.x; u < a.nunits; u += gridDim.x) {
      int b, z, ya, yb, x0;
      unit(u, b, z, ya, yb, x0);
      rows += yb - ya;
    }
    const int q = warp & 3;  // the TMEM lane quarter this warp may read
    const uint32_t base = tmem + ((uint32_t)(q * 32) << 16);
    float acc[144];
#pragma unroll
    for (int i = 0; i < 144; ++i) acc[i] = 0.f;
    const uint32_t chunks = (uint32_t)((rows + chunk - 1) / chunk);
    for (uint32_t cc = 0; cc < chunks; ++cc) {
      if (!mbar_wait(&acc_full[cc & 1], (cc >> 1) & 1, a.err, 49)) break;
      tc_fence_after();
#pragma unroll
      for (int j = 0; j < 9; ++j) {
        float v[16];
        tmem_ld16(base + 256 * (cc & 1) + 16 * j, v);
#pragma unroll
        for (int i = 0; i < 16; ++i) acc[16 * j + i] += v[i];
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[cc & 1]);
    }
    // accumulator row m = 8 * plane + channel; columns dx * 48 + ii * 16 + co, dY row j - 1 + ii
    constexpr int cin = 16 * NIN;
    const int m = q * 32 + lane, plane = m >> 3, c = m & 7;
    const int dz = plane % 3, ci = plane / 3 * 8 + c;  // plane = (input group * 2 + half) * 3 + dz
    float *out = a.partial + (size_t)blockIdx.x * (27 * cin + 1) * 16;
#pragma unroll
    for (int dx = 0; dx < 3; ++dx)
#pragma unroll
      for (int ii = 0; ii < 3; ++ii) {
        const float *v = acc + dx * 48 + ii * 16;
        int row = -1;
        if (plane < 6 * NIN) row = (dz * 9 + (2 - ii) * 3 + dx) * cin + ci;
        else if (m == 48 * NIN && dx == 1 && ii == 1) row = 27 * cin;  // ones: the bias
        if (row >= 0) {
          float4 *o = reinterpret_cast<float4 *>(out + (size_t)row * 16);
#pragma unroll
          for (int k = 0; k < 4; ++k) o[k] = make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
          float nan = 0.f;
#pragma unroll
          for (int k = 0; k < 16; ++k) nan = fmaf(0.f, v[k], nan);
          if (!(nan == 0.f)) dw_again(a, dz * 9 + (2 - ii) * 3 + dx, plane < 6 * NIN ? ci : -1, out + (size_t)row * 16);
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

// ---- the 1-channel FP32 input ----------------------------------------------------------
// A unit is 16 rows of y by up to 32 voxels of x at one z: its dY as FP32 and the
// inputs around it (three z planes of 18 rows) are staged in shared memory.  A lane
// owns a row and eight output channels, a warp the inputs of one dz and one half
// of the voxels: a thread slides a 3 x 3 window along its row, so that three
// inputs and two 16-byte dY quads feed 72 multiply-adds (paired, two channels an
// instruction).  The rows of a warp and then the two halves of x are added up at
// the end.  (Pieces of one row, each staging nine lines, four channels and three taps
// a thread: 127 us at 64^3, batch 4; this 53 us, bound by the multiply-adds (14 us)
// and by the staging between them, 12 warps an SM.)
constexpr int kDwInThreads = 192;  // x half (2), dz (3), lane = row (16) x channel half (2)
constexpr int kDwInX = 32, kDwInRows = 16, kDwInPerSm = 2;
constexpr int kDwInLine = kDwInX + 3;                     // odd: the 16 rows of a warp in 16 banks
constexpr int kDwInRow = kDwInX * 8 + 8;                  // dY: 8 channels a voxel; rows 8 banks apart,
constexpr int kDwInHalf = kDwInRows * kDwInRow + 4;       // halves 4
constexpr int kDwInSmem = (2 * kDwInHalf + 3 * (kDwInRows + 2) * kDwInLine) * (int)sizeof(float);

// Channel co of tap `tap` (27: the bias) over this block's units, terms inside the grid only.
__device__ __noinline__ float dw_in1_again(const DwArgs &a, int xb, int tap, int co) {
  const int nx = a.nx, ny = a.ny, nz = a.nz;
  const int nxb = (nx + xb - 1) / xb, nyb = (ny + kDwInRows - 1) / kDwInRows;
  const int64_t nunit = (int64_t)nxb * nyb * nz * a.nb;
  float s = 0.f;
  for (int64_t u = blockIdx.x; u < nunit; u += gridDim.x) {
    const int64_t p = u / nxb, plane = p / nyb;
    const int x0 = (int)(u - p * nxb) * xb, y0 = (int)(p - plane * nyb) * kDwInRows, z = (int)(plane % nz);
    for (int y = y0; y < min(ny, y0 + kDwInRows); ++y)
      for (int x = x0; x < min(nx, x0 + xb); ++x) {
        const float d = __bfloat162float(a.dy[act_elem(plane * ny + y, x, co, nx)]);
        const int xx = x + tap % 3 - 1, yy = y + tap / 3 % 3 - 1, dz = tap / 9 - 1;
        if (tap == 27)
          s += d;
        else if ((unsigned)xx < (unsigned)nx && (unsigned)yy < (unsigned)ny && (unsigned)(z + dz) < (unsigned)nz)
          s = fmaf(a.x_f32[((plane + dz) * ny + yy) * nx + xx], d, s);
        if (s != s) return s;
      }
  }
  return s;
}

__global__ void __launch_bounds__(kDwInThreads, kDwInPerSm) k_dW_in1(const __grid_constant__ DwArgs a,
                                                                   int xb) {
  __shared__ __align__(16) float sm[kDwInSmem / sizeof(float)];
  float *sdy = sm, *sin = sm + 2 * kDwInHalf;
  const int nx = a.nx, ny = a.ny, nz = a.nz;
  const int nxb = (nx + xb - 1) / xb, nyb = (ny + kDwInRows - 1) / kDwInRows;
  const int64_t nunit = (int64_t)nxb * nyb * nz * a.nb;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5, xh = warp / 3, dzi = warp % 3;
  const int h = lane & 1, r = lane >> 1;
  chain_wait();
  chain_release();
  unsigned long long acc[9][4], bs[4];
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    bs[c] = 0ull;
#pragma unroll
    for (int k = 0; k < 9; ++k) acc[k][c] = 0ull;
  }
  for (int64_t u = blockIdx.x; u < nunit; u += gridDim.x) {
    const int64_t p = u / nxb, plane = p / nyb;  // (b, z)
    const int x0 = (int)(u - p * nxb) * xb, y0 = (int)(p - plane * nyb) * kDwInRows, z = (int)(plane % nz);
    const int w = min(xb, nx - x0), rows = min(kDwInRows, ny - y0);
    // all loads of the unit in flight before the first store
    constexpr int kIn = 3 * (kDwInRows + 2) * (kDwInX + 2), kInN = (kIn + kDwInThreads - 1) / kDwInThreads;
    constexpr int kDy = 2 * kDwInRows * kDwInX, kDyN = (kDy + kDwInThreads - 1) / kDwInThreads;
    float iv[kInN];
    uint4 dv[kDyN];
#pragma unroll
    for (int k = 0; k < kInN; ++k) {
      const int e = t + k * kDwInThreads, l = e / (kDwInX + 2), i = e % (kDwInX + 2);
      const int dz = l / (kDwInRows + 2) - 1, y = y0 + l % (kDwInRows + 2) - 1, x = x0 + i - 1;
      iv[k] = e < kIn && i < w + 2 && (unsigned)x < (unsigned)nx && (unsigned)y < (unsigned)ny && (unsigned)(z + dz) < (unsigned)nz
                  ? __ldg(a.x_f32 + ((plane + dz) * ny + y) * nx + x) : 0.f;
    }
#pragma unroll
    for (int k = 0; k < kDyN; ++k) {
      const int e = t + k * kDwInThreads, x = e % kDwInX, l = e / kDwInX;
      if (x < w && l < 2 * rows)
        dv[k] = __ldg(reinterpret_cast<const uint4 *>(a.dy) + act_unit(plane * ny + y0 + (l >> 1), l & 1, x0 + x, nx));
    }
    __syncthreads();  // the previous unit has been read
#pragma unroll
    for (int k = 0; k < kInN; ++k) {
      const int e = t + k * kDwInThreads;
      if (e < kIn) sin[e / (kDwInX + 2) * kDwInLine + e % (kDwInX + 2)] = iv[k];
    }
#pragma unroll
    for (int k = 0; k < kDyN; ++k) {
      const int e = t + k * kDwInThreads, x = e % kDwInX, l = e / kDwInX;
      if (x < w && l < 2 * rows) {
        const __nv_bfloat162 *p2 = reinterpret_cast<const __nv_bfloat162 *>(&dv[k]);
        const float2 f0 = __bfloat1622float2(p2[0]), f1 = __bfloat1622float2(p2[1]);
        const float2 f2 = __bfloat1622float2(p2[2]), f3 = __bfloat1622float2(p2[3]);
        float4 *d = reinterpret_cast<float4 *>(sdy + (l & 1) * kDwInHalf + (l >> 1) * kDwInRow + x * 8);
        d[0] = make_float4(f0.x, f0.y, f1.x, f1.y);
        d[1] = make_float4(f2.x, f2.y, f3.x, f3.y);
      }
    }
    __syncthreads();
    const int xm = (w + 1) / 2, xa = xh ? xm : 0, xe = xh ? w : xm;
    if (r < rows && xa < xe) {
      const float *s = sin + (dzi * (kDwInRows + 2) + r) * kDwInLine;  // voxel x's taps: s[x], s[x + 1], s[x + 2]
      const float *dy = sdy + h * kDwInHalf + r * kDwInRow;
      unsigned long long v[3][3];
#pragma unroll
      for (int j = 0; j < 3; ++j)
#pragma unroll
        for (int k = 0; k < 2; ++k) v[j][k] = pack_f32x2(s[j * kDwInLine + xa + k], s[j * kDwInLine + xa + k]);
      for (int x = xa; x < xe; ++x) {
        const ulonglong2 d0 = *reinterpret_cast<const ulonglong2 *>(dy + x * 8);
        const ulonglong2 d1 = *reinterpret_cast<const ulonglong2 *>(dy + x * 8 + 4);
        const unsigned long long d[4] = {d0.x, d0.y, d1.x, d1.y};
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          const float n = s[j * kDwInLine + x + 2];
          v[j][2] = pack_f32x2(n, n);
#pragma unroll
          for (int k = 0; k < 3; ++k)
#pragma unroll
            for (int c = 0; c < 4; ++c) fma_f32x2(acc[j * 3 + k][c], v[j][k], d[c]);
          v[j][0] = v[j][1];
          v[j][1] = v[j][2];
        }
        if (dzi == 1) {
          const unsigned long long one = pack_f32x2(1.f, 1.f);
#pragma unroll
          for (int c = 0; c < 4; ++c) fma_f32x2(bs[c], one, d[c]);
        }
      }
    }
  }
  // rows of the warp by shuffles, then the two x halves in order: red[tap][co], the bias as tap 27
  float *red = sm;
  auto finish = [&](int tap, const unsigned long long *v) {
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      float lo, hi;
      unpack_f32x2(v[c], lo, hi);
#pragma unroll
      for (int o = 2; o < 32; o <<= 1) {
        lo += __shfl_xor_sync(0xffffffffu, lo, o);
        hi += __shfl_xor_sync(0xffffffffu, hi, o);
      }
      if (lane < 2) {
        float *d = red + tap * 16 + 8 * h + 2 * c;
        d[0] = xh ? d[0] + lo : lo;
        d[1] = xh ? d[1] + hi : hi;
      }
    }
  };
  for (int k = 0; k < 2; ++k) {
    __syncthreads();
    if (xh == k) {
#pragma unroll
      for (int j = 0; j < 9; ++j) finish(dzi * 9 + j, acc[j]);
      if (dzi == 1) finish(27, bs);
    }
  }
  __syncthreads();
  for (int e = t; e < 28 * 16; e += kDwInThreads) {
    float v = red[e];
    if (v != v) v = dw_in1_again(a, xb, e >> 4, e & 15);  // a NaN may be a zero outside the grid times an infinity
    a.partial[(size_t)blockIdx.x * 28 * 16 + e] = v;
  }
}

// Partials of one layer's gradient (a.partial holds max_blocks of them); *blocks: how many.
int launch_dW(const DwArgs &a, int max_blocks, int *err, int num_sms, cudaStream_t s, int *blocks) {
  if (a.x_f32) {
    const int nxb = (a.nx + kDwInX - 1) / kDwInX, xb = (a.nx + nxb - 1) / nxb;
    const int64_t units = (int64_t)((a.ny + kDwInRows - 1) / kDwInRows) * a.nz * a.nb * nxb;
    // its partials are 1/30 of a 32-channel layer's, which max_blocks counts
    *blocks = (int)std::min<int64_t>(std::min(30 * max_blocks, kDwInPerSm * num_sms), units);
    HPCCG_CUDA(launch_chained(k_dW_in1, *blocks, kDwInThreads, 0, s, true, a, xb));
    return HPCCG_OK;
  }
  DwTcArgs t{};
  t.g.nx = a.nx;
  t.g.ny = a.ny;
  t.g.nz = a.nz;
  t.g.nb = a.nb;
  t.x[0] = a.x0;
  t.x[1] = a.x1;
  t.dy = a.dy;
  t.partial = a.partial;
  t.err = err;
  t.nxb = (a.nx + kDwMaxX - 1) / kDwMaxX;
  t.kx = ((a.nx + t.nxb - 1) / t.nxb + 15) / 16 * 16;
  t.nxb = (a.nx + t.kx - 1) / t.kx;
  t.nyb = (a.ny + kDwRows - 1) / kDwRows;
  const int64_t units = (int64_t)t.nxb * t.nyb * a.nz * a.nb;
  if (units >= ((int64_t)1 << 31)) return HPCCG_ERR_TOO_LARGE;
  t.nunits = (int)units;
  *blocks = (int)std::min<int64_t>(std::min(max_blocks, num_sms), units);
  static_assert(dw_smem_bytes(2, kDwMaxX) <= 226 * 1024, "shared memory of a CTA");
  int rc = act_tmap(&t.ymap, a.dy, t.g, t.kx, kDimH, 2, kDimY, kDwRows + 2, kDimZ, 1);
  if (!rc) rc = act_tmap(&t.xmap[0], a.x0, t.g, t.kx + 8, kDimZ, 3, kDimH, 2, kDimY, 1);
  if (!rc && a.cin == 32) rc = act_tmap(&t.xmap[1], a.x1, t.g, t.kx + 8, kDimZ, 3, kDimH, 2, kDimY, 1);
  if (rc) return rc;
  const int nin = a.cin / 16, smem = dw_smem_bytes(nin, t.kx);
  auto kern = nin == 2 ? k_dW_tc<2> : k_dW_tc<1>;
  // the attribute is per device: set every time, to the most any width needs
  HPCCG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, dw_smem_bytes(nin, kDwMaxX)));
  HPCCG_CUDA(launch_chained(kern, *blocks, kDwThreads, smem, s, true, t));
  return HPCCG_OK;
}

}  // namespace hpccg
