// unet_conv.cu -- the brick form of the tcgen05 3x3x3 convolutions and the
// 1-channel input layer (layout in unet_conv.cuh; the network's 16- and
// 32-channel layers run the kernels of unet_conv_win.cu).  Operand tiles arrive
// by 1D bulk copies of row-planar spans; grid faces are zero-filled with ordinary
// stores, fenced into the async proxy before the tensor cores read them.
#include <stdlib.h>

#include <algorithm>
#include <type_traits>

#include "unet_conv.cuh"

namespace hpccg {

using namespace tc;

struct TileOrigin {
  int b, x0, y0, z0;
};

__device__ __forceinline__ TileOrigin tile_origin(const ConvGeom &g, int t) {
  TileOrigin o;
  int r = t;
  o.x0 = (r % g.tx) * g.bx;
  r /= g.tx;
  o.y0 = (r % g.ty) * g.by;
  r /= g.ty;
  o.z0 = (r % g.tz) * g.bz;
  o.b = r / g.tz;
  return o;
}

// Epilogue of one voxel: row m of tile t holds its 16 accumulated channels in v.
template <int EPI>
__device__ __forceinline__ void conv_store(const ConvArgs &a, int t, int m, const float *v, const float *bias,
                                           const float *proj) {
  const ConvGeom &g = a.g;
  const TileOrigin o = tile_origin(g, t);
  const int x = o.x0 + m % g.bx, y = o.y0 + (m / g.bx) % g.by, z = o.z0 + m / (g.bx * g.by);
  const int64_t row = ((int64_t)o.b * g.nz + z) * g.ny + y;
  if (EPI == kEpiRawF32) {
    float *out = static_cast<float *>(a.out);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float4 *o4 = reinterpret_cast<float4 *>(out + act_unit(row, h, x, g.nx) * 8);
      o4[0] = make_float4(v[8 * h], v[8 * h + 1], v[8 * h + 2], v[8 * h + 3]);
      o4[1] = make_float4(v[8 * h + 4], v[8 * h + 5], v[8 * h + 6], v[8 * h + 7]);
    }
  } else if (EPI == kEpiProject) {
    float acc = proj[16];
#pragma unroll
    for (int c = 0; c < 16; ++c) acc = fmaf(proj[c], fmaxf(v[c] + bias[c], 0.f), acc);
    static_cast<float *>(a.out)[row * g.nx + x] = acc;
  } else {
    __nv_bfloat16 *out = static_cast<__nv_bfloat16 *>(a.out);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      uint32_t w[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        float lo = v[8 * h + 2 * c] + bias[8 * h + 2 * c], hi = v[8 * h + 2 * c + 1] + bias[8 * h + 2 * c + 1];
        if (EPI == kEpiBiasRelu) {
          lo = fmaxf(lo, 0.f);
          hi = fmaxf(hi, 0.f);
        }
        const __nv_bfloat162 p = __floats2bfloat162_rn(lo, hi);
        w[c] = *reinterpret_cast<const uint32_t *>(&p);
      }
      *reinterpret_cast<uint4 *>(out + act_unit(row, h, x, g.nx) * 8) = make_uint4(w[0], w[1], w[2], w[3]);
    }
  }
}

// Shared set-up of both kernels: weights to smem, barriers, TMEM (32 columns).
// bars: full[STAGES], empty[STAGES], acc_full[2], acc_empty[2], drain.
template <int NIN, int STAGES>
__device__ __forceinline__ uint32_t conv_setup(const ConvArgs &a, uint8_t *sW, uint64_t *bars, uint32_t *slot,
                                               int warp) {
  constexpr int kWBytes = NIN * 27 * kWTapBytes;
  for (int i = threadIdx.x; i < kWBytes / 16; i += kConvThreads)
    reinterpret_cast<uint4 *>(sW)[i] = reinterpret_cast<const uint4 *>(a.wpack)[i];
  if (threadIdx.x == 0) {
    for (int s = 0; s < 2 * STAGES; ++s) mbar_init(&bars[s], 1);
    mbar_init(&bars[2 * STAGES + 0], 1);
    mbar_init(&bars[2 * STAGES + 1], 1);
    mbar_init(&bars[2 * STAGES + 2], 4);
    mbar_init(&bars[2 * STAGES + 3], 4);
    mbar_init(&bars[2 * STAGES + 4], 1);
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc(slot, 32);
    tmem_relinquish();
  }
  fence_proxy_async_smem();  // weights -> tensor-core proxy
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  return *slot;
}

// Epilogue role (warps 2-5): drain each tile's accumulator and store it.
template <int EPI>
__device__ __forceinline__ void conv_epilogue(const ConvArgs &a, uint64_t *acc_full, uint64_t *acc_empty,
                                              uint32_t tmem, int warp, int lane, int where) {
  const int q = warp & 3;
  uint32_t tcount = 0;
  float bias[16], proj[17];
#pragma unroll
  for (int c = 0; c < 16; ++c) bias[c] = (EPI == kEpiRawF32 || !a.bias) ? 0.f : a.bias[c];
  if (EPI == kEpiProject)
#pragma unroll
    for (int c = 0; c < 17; ++c) proj[c] = a.proj[c];
  for (int t = blockIdx.x; t < a.g.ntiles; t += gridDim.x, ++tcount) {
    const int buf = tcount & 1;
    if (!mbar_wait(&acc_full[buf], (tcount >> 1) & 1, a.err, where)) break;
    tc_fence_after();
    float v[16];
    tmem_ld16(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * 16), v);
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(&acc_empty[buf]);
    conv_store<EPI>(a, t, q * 32 + lane, v, bias, proj);
  }
}

// ---- brick tiles: one fetch per (tap, input) ---------------------------------------------
template <int NIN, int EPI>
__global__ void __launch_bounds__(kConvThreads, 1) k_conv3_brick(ConvArgs a) {
  extern __shared__ __align__(1024) uint8_t smem[];
  constexpr int kWBytes = NIN * 27 * kWTapBytes;
  constexpr int S = kBrickStages;
  uint8_t *sW = smem;
  uint8_t *sA = smem + kWBytes;
  uint64_t *full = reinterpret_cast<uint64_t *>(sA + S * kBrickStageBytes);
  uint64_t *empty = full + S;
  uint64_t *acc_full = empty + S;
  uint64_t *acc_empty = acc_full + 2;
  uint64_t *drain = acc_empty + 2;
  uint32_t *slot = reinterpret_cast<uint32_t *>(drain + 1);
  static_assert((2 * S + 5) * 8 + 4 <= bar_bytes(S), "barrier area");
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t tmem = conv_setup<NIN, S>(a, sW, full, slot, warp);
  const ConvGeom &g = a.g;
  constexpr int ksteps = 27 * NIN;

  if (warp == 0) {
    // fetch: 2 halves x by*bz rows per k-step, one span per lane (at most 32)
    const int nrows = g.by * g.bz;
    uint32_t it = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < g.ntiles && ok; t += gridDim.x) {
      const TileOrigin o = tile_origin(g, t);
      for (int ks = 0; ks < ksteps; ++ks, ++it) {
        const int s = it % S;
        const uint32_t n = it / S;
        if (n > 0 && !(ok = warp_wait(&empty[s], (n - 1) & 1, a.err, 1, lane))) break;
        const int tap = ks / NIN, in = ks % NIN;
        const int dz = tap / 9 - 1, dy = (tap / 3) % 3 - 1, dx = tap % 3 - 1;
        const __nv_bfloat16 *base = (NIN > 1 && in) ? a.in1 : a.in0;
        uint8_t *stage = sA + s * kBrickStageBytes;
        Span sp[1];
        int nsp = 0;
        if (lane < 2 * nrows) {
          const int h = lane / nrows, rr = lane % nrows;
          const int my = rr % g.by, mz = rr / g.by;
          sp[0] = plan_span(g, base, o.b, o.z0 + mz + dz, o.y0 + my + dy, h, o.x0 + dx, g.bx,
                            stage + h * (kBrickStageBytes / 2) + rr * g.bx * 16);
          nsp = 1;
        }
        post_spans(sp, nsp, &full[s], lane);
      }
    }
    if (lane == 0) {  // every issued copy has landed before the CTA may exit
      const uint32_t first = it > (uint32_t)S ? it - S : 0;
      for (uint32_t j = first; j < it; ++j) mbar_wait(&full[j % S], (j / S) & 1, a.err, 5);
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc = idesc_bf16(128, 16);
      const uint64_t ad0 = smem_desc(sA, kBrickStageBytes / 2, 128), wd = smem_desc(sW, 256, 128);
      uint32_t it = 0, tcount = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < g.ntiles && ok; t += gridDim.x, ++tcount) {
        const int buf = tcount & 1;
        const uint32_t use = tcount >> 1;
        if (use > 0 && !(ok = mbar_wait(&acc_empty[buf], (use - 1) & 1, a.err, 2))) break;
        tc_fence_after();
        const uint32_t d = tmem + (uint32_t)(buf * 16);
        for (int ks = 0; ks < ksteps; ++ks, ++it) {
          const int s = it % S;
          if (!(ok = mbar_wait(&full[s], (it / S) & 1, a.err, 3))) break;
          tc_fence_after();
          const uint64_t ad = ad0 + (uint64_t)((s * kBrickStageBytes) >> 4);
          const uint64_t bd = wd + (uint64_t)((ks % NIN * 27 + ks / NIN) * (kWTapBytes >> 4));
          mma_bf16(d, ad, bd, idesc, ks > 0 ? 1u : 0u);
          mma_commit(&empty[s]);
        }
        if (!ok) break;
        mma_commit(&acc_full[buf]);
      }
      mma_commit(drain);
      mbar_wait(drain, 0, a.err, 6);
    }
  } else {
    conv_epilogue<EPI>(a, acc_full, acc_empty, tmem, warp, lane, 4);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 32);
  }
}

// ---- the 1-channel input layer on tcgen05 (nx a multiple of 128) -------------------------
// An im2col GEMM per tile of 128 voxels of one x row: A[m][k] = in(x0+m+dx, y+dy, z+dz)
// in BF16 for tap k = (dz+1)*9 + (dy+1)*3 + (dx+1) (k = 27..31 zero), B[c][k] = W[k][c];
// two MMAs (M = 128, N = 16, K = 16) into a 16-column FP32 accumulator.  A CTA walks a
// contiguous range of tiles, y innermost: thread m keeps its voxel's 27 taps in
// registers, and from one tile to the next takes over two of the three rows of each
// z plane and forms the third from one load per plane, a tile ahead, and its
// neighbours' lanes (the lanes at a warp's ends load their outer neighbour).  It
// writes the taps to its A row; thread 0 issues the tile's MMAs; every warp drains
// its TMEM lane quarter of the PREVIOUS tile (bias, ReLU, BF16 stores), so a tile's
// MMAs run while the next tile is built.  A and the accumulator are double-buffered:
// one barrier per tile.  Against nine lines per tile staged in shared memory and 27
// reads of them a thread: 282 -> 202 us at 256^3 (2.7 TB/s of stores), 46 -> 34 at
// 128^3.  Bound by instruction issue, 250 a warp and tile; with 5, 7 or 8 CTAs an SM 205,
// 234 and 278 us.
constexpr int kIn1Threads = 128;
constexpr int kIn1ABytes = 4 * 128 * 16;  // [4 K chunks of 8 taps][128 rows][8 BF16]
constexpr int kIn1BBytes = 4 * 16 * 16;   // [4 K chunks][16 output channels][8 BF16]
constexpr int kIn1PerSm = 6;

__global__ void __launch_bounds__(kIn1Threads, kIn1PerSm) k_conv3_in1_tc(const float *in, const float *W,
                                                                         const float *bias, __nv_bfloat16 *out,
                                                                         int nx, int ny, int nz, int nb, int relu,
                                                                         int *err) {
  __shared__ __align__(1024) uint8_t sA[2][kIn1ABytes];
  __shared__ __align__(128) uint8_t sB[kIn1BBytes];
  __shared__ __align__(16) float sBias[16];
  __shared__ uint64_t done[2], fin;
  __shared__ uint32_t slot;
  __shared__ int s_fail;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  for (int e = tid; e < 32 * 16; e += kIn1Threads) {  // B element (k, c): chunk k/8, row c, position k%8
    const int k = e / 16, c = e % 16;
    reinterpret_cast<__nv_bfloat16 *>(sB)[((k >> 3) * 16 + c) * 8 + (k & 7)] =
        __float2bfloat16(k < 27 ? W[k * 16 + c] : 0.f);
  }
  if (tid < 16) sBias[tid] = bias[tid];
  if (tid == 0) {
    mbar_init(&done[0], 1);
    mbar_init(&done[1], 1);
    mbar_init(&fin, 1);
    fence_mbar_init();
    s_fail = 0;
  }
  if (warp == 0) {
    tmem_alloc(&slot, 32);
    tmem_relinquish();
  }
  fence_proxy_async_smem();
  tc_fence_before();
  __syncthreads();  // B, the bias, the barriers and the TMEM slot
  tc_fence_after();
  const uint32_t tmem = slot;
  chain_release();  // the TMEM is allocated
  constexpr uint32_t idesc = idesc_bf16(128, 16);
  const uint64_t bd = smem_desc(sB, 256, 128);

  // tile t = ((b*nz + z)*tx + xb)*ny + y; 32-bit indices (a grid has fewer than 2^31 tiles)
  const int tx = nx / 128, ntiles = tx * ny * nz * nb;
  int t = (int)((int64_t)blockIdx.x * ntiles / gridDim.x);
  const int t_hi = (int)((int64_t)(blockIdx.x + 1) * ntiles / gridDim.x);
  const int64_t plane_step = (int64_t)nx * ny;
  int y = t % ny;
  const float *src;  // row y, this thread's voxel
  uint4 *dst;        // its first unit of the output
  bool ok[3], edge[3];
  auto column = [&]() {  // what a column of tiles shares
    const int col = t / ny, plane = col / tx, xb = col - plane * tx, z = plane % nz, x = xb * 128 + tid;
    src = in + (int64_t)plane * plane_step + (int64_t)y * nx + x;
    dst = reinterpret_cast<uint4 *>(out) + act_unit((int64_t)plane * ny + y, 0, x, nx);
    const bool has = lane == 0 ? x > 0 : lane == 31 && x + 1 < nx;
#pragma unroll
    for (int p = 0; p < 3; ++p) {
      ok[p] = (unsigned)(z + p - 1) < (unsigned)nz;
      edge[p] = ok[p] && has;
    }
  };
  const int xe = lane ? 1 : -1;
  // row y + dy of the three planes: this thread's element and, at a warp's ends, its outer neighbour's
  float c[3], e[3];
  auto load = [&](int dy) {
    const bool row = (unsigned)(y + dy) < (unsigned)ny;
    const float *q = src + (int64_t)dy * nx - plane_step;
#pragma unroll
    for (int p = 0; p < 3; ++p, q += plane_step) {
      c[p] = row && ok[p] ? __ldg(q) : 0.f;
      e[p] = row && edge[p] ? __ldg(q + xe) : 0.f;
    }
  };
  // the taps (x-1, x, x+1) of the loaded rows: BF16 in the low half of v[plane][slot][dx]
  uint32_t v[3][3][3];
  const uint32_t left = lane == 0 ? 0x0076u : 0x0010u, right = lane == 31 ? 0x0076u : 0x0010u;  // neighbour's | own outer
  auto taps = [&](int slot_) {
#pragma unroll
    for (int p = 0; p < 3; ++p) {
      const __nv_bfloat162 h = __floats2bfloat162_rn(c[p], e[p]);
      const uint32_t m = *reinterpret_cast<const uint32_t *>(&h);
      v[p][slot_][0] = __byte_perm(__shfl_up_sync(0xffffffffu, m, 1), m, left);
      v[p][slot_][1] = m;
      v[p][slot_][2] = __byte_perm(__shfl_down_sync(0xffffffffu, m, 1), m, right);
    }
  };
  // bias, ReLU and stores of a tile: accumulator buf in its use-th use
  auto drain = [&](uint4 *o, int buf, uint32_t use) {
    if (!mbar_wait(&done[buf], use & 1u, err, 31)) s_fail = 1;
    tc_fence_after();
    float a[16];
    tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(buf * 16), a);
    tc_fence_before();
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      uint32_t w[4];
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const float4 b = reinterpret_cast<const float4 *>(sBias)[2 * h + k];
        __nv_bfloat162 p0 = __floats2bfloat162_rn(a[8 * h + 4 * k] + b.x, a[8 * h + 4 * k + 1] + b.y);
        __nv_bfloat162 p1 = __floats2bfloat162_rn(a[8 * h + 4 * k + 2] + b.z, a[8 * h + 4 * k + 3] + b.w);
        if (relu) {
          p0 = __hmax2(p0, __float2bfloat162_rn(0.f));
          p1 = __hmax2(p1, __float2bfloat162_rn(0.f));
        }
        w[2 * k] = *reinterpret_cast<const uint32_t *>(&p0);
        w[2 * k + 1] = *reinterpret_cast<const uint32_t *>(&p1);
      }
      o[(int64_t)h * nx] = make_uint4(w[0], w[1], w[2], w[3]);
    }
  };
  int it = 0;
  uint4 *prev = nullptr;  // the tile whose MMAs run
  uint8_t *const arow = sA[0] + (tid >> 3) * 128 + (tid & 7) * 16;
  // One tile; rows y-1, y, y+1 are in slots R, R+1, R+2 (mod 3).  False: the range's last, or a wait ran out.
  auto step = [&](auto rot) -> bool {
    constexpr int R = decltype(rot)::value;
    const int buf = it & 1;
    load(2);  // the next tile's new row, in flight until the end of this one
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      uint32_t w[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int i = 8 * k + 2 * j;
        if (i > 26)
          w[j] = 0;
        else if (i == 26)
          w[j] = v[2][(R + 2) % 3][2] & 0xffffu;
        else
          w[j] = __byte_perm(v[i / 9][(R + i / 3) % 3][i % 3], v[(i + 1) / 9][(R + (i + 1) / 3) % 3][(i + 1) % 3], 0x5410);
      }
      *reinterpret_cast<uint4 *>(arow + buf * kIn1ABytes + k * 2048) = make_uint4(w[0], w[1], w[2], w[3]);
    }
    fence_proxy_async_smem();  // the A rows -> tensor-core proxy
    tc_fence_before();
    __syncthreads();  // A written; the drain of this buffer's last tile is done
    tc_fence_after();
    if (s_fail) return false;  // read by every thread after the same barrier
    if (tid == 0) {
      const uint64_t ad = smem_desc(sA[buf], 2048, 128);
      const uint32_t d = tmem + (uint32_t)(buf * 16);
      mma_bf16(d, ad, bd, idesc, 0u);
      mma_bf16(d, ad + (uint64_t)(4096 >> 4), bd + (uint64_t)(512 >> 4), idesc, 1u);
      mma_commit(&done[buf]);
    }
    if (it > 0) drain(prev, buf ^ 1, (uint32_t)((it - 1) >> 1));
    prev = dst;
    ++it;
    if (++t >= t_hi) return false;
    src += nx;
    dst += 2 * nx;
    if (++y < ny) {
      taps(R);  // the oldest row's slot
    } else {
      y = 0;
      column();
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        load(r - 1);
        taps((R + 1 + r) % 3);
      }
    }
    return true;
  };
  if (t < t_hi) {
    column();
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      load(r - 1);
      taps(r);
    }
    while (step(std::integral_constant<int, 0>()) && step(std::integral_constant<int, 1>()) &&
           step(std::integral_constant<int, 2>())) {
    }
  }
  if (it > 0 && !s_fail) drain(prev, (it - 1) & 1, (uint32_t)((it - 1) >> 1));
  if (tid == 0) {  // every MMA this thread issued has completed before TMEM is freed
    mma_commit(&fin);
    mbar_wait(&fin, 0, err, 32);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem, 32);
  }
}

int launch_conv3_in1_tc(const float *in, const float *W, const float *bias, __nv_bfloat16 *out, int nx, int ny,
                        int nz, int nb, int relu, int *err, int num_sms, cudaStream_t s) {
  if (nx % 128 || ny < 1 || nz < 1 || nb < 1) return HPCCG_ERR_UNSUPPORTED;
  const int64_t ntiles = (int64_t)(nx / 128) * ny * nz * nb;
  if (ntiles >= ((int64_t)1 << 31)) return HPCCG_ERR_TOO_LARGE;
  const int grid = (int)std::min<int64_t>(ntiles, (int64_t)num_sms * kIn1PerSm);
  k_conv3_in1_tc<<<grid, kIn1Threads, 0, s>>>(in, W, bias, out, nx, ny, nz, nb, relu, err);
  HPCCG_CUDA(cudaGetLastError());
  return HPCCG_OK;
}

template <int NIN, int EPI>
static int launch_brick(const ConvArgs &a, int num_sms, cudaStream_t s) {
  constexpr int smem = brick_smem_bytes(NIN);
  static_assert(smem <= 227 * 1024, "conv CTA exceeds the shared-memory limit");
  auto kern = k_conv3_brick<NIN, EPI>;
  // the attribute is per device: set every time
  HPCCG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  // resident CTAs per SM by shared memory (each CTA also reserves 1 KB)
  constexpr int per_sm = (227 * 1024) / (smem + 1024);
  kern<<<std::min(a.g.ntiles, num_sms * (per_sm > 1 ? per_sm : 1)), kConvThreads, smem, s>>>(a);
  HPCCG_CUDA(cudaGetLastError());
  return HPCCG_OK;
}

int launch_conv3_brick(int nin, int epi, const ConvArgs &a, int num_sms, cudaStream_t s) {
  if (nin == 1) {
    switch (epi) {
      case kEpiBiasRelu: return launch_brick<1, kEpiBiasRelu>(a, num_sms, s);
      case kEpiBias: return launch_brick<1, kEpiBias>(a, num_sms, s);
      case kEpiProject: return launch_brick<1, kEpiProject>(a, num_sms, s);
      default: return launch_brick<1, kEpiRawF32>(a, num_sms, s);
    }
  }
  switch (epi) {
    case kEpiBiasRelu: return launch_brick<2, kEpiBiasRelu>(a, num_sms, s);
    case kEpiBias: return launch_brick<2, kEpiBias>(a, num_sms, s);
    case kEpiProject: return launch_brick<2, kEpiProject>(a, num_sms, s);
    default: return launch_brick<2, kEpiRawF32>(a, num_sms, s);
  }
}

}  // namespace hpccg
