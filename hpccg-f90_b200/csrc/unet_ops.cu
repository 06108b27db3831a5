// unet_ops.cu -- CUDA-core kernels of the U-Net: the 1-channel input conv and
// small-volume convs, weight packing for the tcgen05 convs, pooling,
// upsampling, ReLU masks, weight/bias gradients, the output projection, the
// loss and the Adam update.  All are memory-bound or tiny.  16-channel
// tensors use the row-planar layout of unet_conv.cuh (act_unit / act_elem).
#include <algorithm>

#include "unet_ops.cuh"

namespace hpccg {

// ---- weight packing ------------------------------------------------------------------
// Forward B operand of input group `in`: packed[in][tap][kc][co][j] =
// W[tap][in*16 + kc*8 + j][co] (W is FP32 [27][cin][16]).
__global__ void k_pack_fwd(const float *W, int cin, int nin, __nv_bfloat16 *packed) {
  const int total = nin * 27 * 256;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < total; e += gridDim.x * blockDim.x) {
    const int j = e & 7, co = (e >> 3) & 15, kc = (e >> 7) & 1, tap = (e >> 8) % 27, in = (e >> 8) / 27;
    packed[e] = __float2bfloat16(W[((size_t)tap * cin + in * 16 + kc * 8 + j) * 16 + co]);
  }
}
// Backward-data operand for the gradient w.r.t. input group g: a conv over dY
// (16 channels) with taps flipped and in/out transposed:
// packed[tap][kc][ci][j] = W[26 - tap][g*16 + ci][kc*8 + j].
__global__ void k_pack_bwd(const float *W, int cin, int g, __nv_bfloat16 *packed) {
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < 27 * 256; e += gridDim.x * blockDim.x) {
    const int j = e & 7, ci = (e >> 3) & 15, kc = (e >> 7) & 1, tap = e >> 8;
    packed[e] = __float2bfloat16(W[((size_t)(26 - tap) * cin + g * 16 + ci) * 16 + kc * 8 + j]);
  }
}
// The same flipped/transposed weights in FP32 [27][16][16] for the CUDA-core conv.
__global__ void k_flip_fp32(const float *W, int cin, int g, float *Wf) {
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < 27 * 256; e += gridDim.x * blockDim.x) {
    const int ci = e & 15, co = (e >> 4) & 15, tap = e >> 8;  // Wf[tap][co as input][ci as output]
    Wf[e] = W[((size_t)(26 - tap) * cin + g * 16 + ci) * 16 + co];
  }
}

// ---- direct conv on CUDA cores --------------------------------------------------------
// out[v][co] = sum_tap sum_ci in[v + off(tap)][ci] * W[tap][ci][co] (+ bias, ReLU), for
// volumes without 128-voxel bricks; FP32 weights.  Inputs: in0/in1 row-planar BF16
// 16-channel tensors (in1 nullable).  A thread forms CO of the 16 channels of V
// voxels (x, y .. y+V-1), lanes along x: per tap and input group it loads its voxels'
// channels as 16-byte units, and every weight, read from the block's copy in shared
// memory (one address for the warp, or one per channel group), feeds V fused
// multiply-adds, two channels at a time.  A voxel's terms are added in the order
// tap, group, channel; taps outside the grid are left out.  V and CO fall with the
// volume so that it fills the SMs (launch_conv3_cc).
// One voxel a thread with scalar loads, against this: forward pass at 192^3 27.7 ->
// 8.4 ms, 96^3 4.30 -> 1.36, 24^3 1.41 -> 0.27.  Bound by the FP32 pipe on large volumes
// (6912 multiply-adds a voxel and group: 226 G of them at 192^3, 7.8 ms, 80% of its
// rate), by the latency of the 27 taps on small ones.
// One tap and input group of N voxels: q = their 16 channels, w = the weights [16 ci][16 co]
// from the thread's first channel on.
template <int N, int CO>
__device__ __forceinline__ void cc_tap(const uint4 (*q)[2], const float *w, unsigned long long (*acc)[CO / 2]) {
#pragma unroll
  for (int ci = 0; ci < 16; ++ci) {
    unsigned long long wv[CO / 2];
#pragma unroll
    for (int c = 0; c < CO / 4; ++c) {
      const ulonglong2 t = *reinterpret_cast<const ulonglong2 *>(w + ci * 16 + 4 * c);
      wv[2 * c] = t.x;
      wv[2 * c + 1] = t.y;
    }
#pragma unroll
    for (int v = 0; v < N; ++v) {
      const uint4 &u = q[v][ci >> 3];
      const uint32_t p = (ci & 7) < 2 ? u.x : (ci & 7) < 4 ? u.y : (ci & 7) < 6 ? u.z : u.w;
      const float f = __uint_as_float(ci & 1 ? p & 0xffff0000u : p << 16);
      const unsigned long long ff = pack_f32x2(f, f);
#pragma unroll
      for (int c = 0; c < CO / 2; ++c) fma_f32x2(acc[v][c], ff, wv[c]);
    }
  }
}

constexpr int kCcThreads = 128;
// resident blocks an SM (the registers of V * CO sums)
template <int V, int CO>
constexpr int cc_blocks() { return V == 4 ? 3 : 8; }

template <int V, int CO>
__global__ void __launch_bounds__(kCcThreads, cc_blocks<V, CO>()) k_conv3_cc(CcConvArgs a) {
  extern __shared__ __align__(16) float cc_w[];  // [27][cin][16]
  const int nx = a.nx, ny = a.ny, nz = a.nz, cin = 16 * a.nin;
  for (int e = threadIdx.x; e < 27 * cin * 4; e += blockDim.x)
    reinterpret_cast<float4 *>(cc_w)[e] = __ldg(reinterpret_cast<const float4 *>(a.W) + e);
  chain_wait();
  chain_release();
  __syncthreads();
  constexpr int NG = 16 / CO;
  const int nyg = (ny + V - 1) / V;
  const int64_t total = (int64_t)nx * nyg * nz * a.nb * NG;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    const int c0 = (int)(e % NG) * CO;
    int64_t t = e / NG;
    const int x = (int)(t % nx);
    t /= nx;
    const int y = (int)(t % nyg) * V;
    t /= nyg;
    const int z = (int)(t % nz);
    const int64_t row = t * ny + y;  // (b * nz + z) * ny + y
    const int nv = min(V, ny - y);
    unsigned long long acc[V][CO / 2];
#pragma unroll
    for (int v = 0; v < V; ++v)
#pragma unroll
      for (int c = 0; c < CO / 2; ++c) acc[v][c] = 0ull;
    for (int tap = 0; tap < 27; ++tap) {
      const int dx = tap % 3 - 1, dy = tap / 3 % 3 - 1, dz = tap / 9 - 1;
      if ((unsigned)(x + dx) >= (unsigned)nx || (unsigned)(z + dz) >= (unsigned)nz) continue;
      const int64_t r0 = row + dz * ny + dy;
      const int lo = max(0, -(y + dy)), hi = min(nv, ny - (y + dy));  // voxels whose row y+v+dy is inside
      for (int g = 0; g < a.nin; ++g) {
        const uint4 *src = reinterpret_cast<const uint4 *>(g ? a.in1 : a.in0);
        const float *w = cc_w + (tap * cin + g * 16) * 16 + c0;
        uint4 q[V][2];
        if (lo == 0 && hi == V) {
#pragma unroll
          for (int v = 0; v < V; ++v)
#pragma unroll
            for (int h = 0; h < 2; ++h) q[v][h] = __ldg(src + act_unit(r0 + v, h, x + dx, nx));
          cc_tap<V, CO>(q, w, acc);
        } else {
#pragma unroll
          for (int v = 0; v < V; ++v)
            if (v >= lo && v < hi) {
#pragma unroll
              for (int h = 0; h < 2; ++h) q[v][h] = __ldg(src + act_unit(r0 + v, h, x + dx, nx));
              cc_tap<1, CO>(q + v, w, acc + v);
            }
        }
      }
    }
#pragma unroll
    for (int v = 0; v < V; ++v) {
      if (v >= nv) break;
      float o[CO];
#pragma unroll
      for (int c = 0; c < CO / 2; ++c) unpack_f32x2(acc[v][c], o[2 * c], o[2 * c + 1]);
      if (a.epi == kEpiRawF32) {
        float *dst = static_cast<float *>(a.out);
#pragma unroll
        for (int c = 0; c < CO; c += 4)
          *reinterpret_cast<float4 *>(dst + act_elem(row + v, x, c0 + c, nx)) =
              make_float4(o[c], o[c + 1], o[c + 2], o[c + 3]);
      } else if (CO == 16 && a.epi == kEpiProject) {
        float r = a.proj[16];
#pragma unroll
        for (int c = 0; c < CO; ++c) r = fmaf(a.proj[c], fmaxf(o[c] + a.bias[c], 0.f), r);
        static_cast<float *>(a.out)[(row + v) * nx + x] = r;
      } else {
        __nv_bfloat16 *dst = static_cast<__nv_bfloat16 *>(a.out);
#pragma unroll
        for (int c = 0; c < CO; c += 4) {
          const int64_t at = act_elem(row + v, x, c0 + c, nx);
          uint32_t p[2];
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            float f[2];
#pragma unroll
            for (int j = 0; j < 2; ++j) {
              f[j] = o[c + 2 * k + j];
              if (a.bias) f[j] += a.bias[c0 + c + 2 * k + j];
              if (a.epi == kEpiBiasRelu) f[j] = fmaxf(f[j], 0.f);
            }
            const __nv_bfloat162 b = __floats2bfloat162_rn(f[0], f[1]);
            p[k] = *reinterpret_cast<const uint32_t *>(&b);
          }
          if (a.epi == kEpiMask) {
            const uint2 m = __ldg(reinterpret_cast<const uint2 *>(a.act + at));
            p[0] = relu_mask2(p[0], m.x);
            p[1] = relu_mask2(p[1], m.y);
          }
          *reinterpret_cast<uint2 *>(dst + at) = make_uint2(p[0], p[1]);
        }
      }
    }
  }
}

template <int V, int CO>
static int launch_cc(const CcConvArgs &a, int num_sms, cudaStream_t s) {
  const int64_t threads = (int64_t)a.nx * ((a.ny + V - 1) / V) * a.nz * a.nb * (16 / CO);
  constexpr int kBlocks = cc_blocks<V, CO>();
  const int grid = (int)std::max<int64_t>(1, std::min<int64_t>((threads + kCcThreads - 1) / kCcThreads,
                                                               (int64_t)num_sms * kBlocks));
  // The blocks of a chained launch start where the predecessor's end first and would
  // pile up there: shared memory is padded so that no SM takes more than its share
  // (72^3 forward: plain launches 779 us, unpadded 886, padded 753; 88^3 1237, 1243, 1155).
  const int per_sm = (grid + num_sms - 1) / num_sms;
  int smem = 27 * 16 * a.nin * 16 * (int)sizeof(float);
  if (per_sm < kBlocks) smem = std::max(smem, 228 * 1024 / (per_sm + 1) - 1024 + 128);
  // the attribute is per device: set every time, to the most any launch needs
  HPCCG_CUDA(cudaFuncSetAttribute(k_conv3_cc<V, CO>, cudaFuncAttributeMaxDynamicSharedMemorySize, 114 * 1024));
  HPCCG_CUDA(launch_chained(k_conv3_cc<V, CO>, grid, kCcThreads, smem, s, a.chained, a));
  return HPCCG_OK;
}

// Four voxels a thread where that leaves every SM 256 threads, one where one does, else
// several threads a voxel (the projection needs all channels in one).  Forward pass
// with the lines at half | this | eight times the size: 56^3 0.54 | 0.52 | 0.59 ms,
// 72^3 0.75 | 0.75 | 0.95, 88^3 1.29 | 1.20 | 1.58, 40x72x24 0.34 | 0.34 | 0.37.
int launch_conv3_cc(const CcConvArgs &a, int num_sms, cudaStream_t s) {
  const int64_t n = (int64_t)a.nx * a.ny * a.nz * a.nb, fill = (int64_t)num_sms * 256;
  if (n >= 4 * fill) return launch_cc<4, 16>(a, num_sms, s);
  if (n >= fill || a.epi == kEpiProject) return launch_cc<1, 16>(a, num_sms, s);
  if (2 * n >= fill) return launch_cc<1, 8>(a, num_sms, s);
  return launch_cc<1, 4>(a, num_sms, s);
}

// The 1-channel input layer: out[v][co] = act(sum_tap in[v+off] W[tap][co] + b[co]).
// A thread forms V voxels consecutive in x (nx a multiple of V): per (dz, dy)
// line it loads the V+2 inputs once, and each tap's 16 weights (shared memory)
// once for all V voxels; two 16-byte BF16 stores per voxel.
template <int V>
__device__ __forceinline__ void conv3_in1_body(const float *in, const float *W, const float *bias,
                                               __nv_bfloat16 *out, int nx, int ny, int nz, int nb, int relu) {
  __shared__ __align__(16) float sw[27 * 16 + 16];
  for (int e = threadIdx.x; e < 27 * 16 + 16; e += blockDim.x) sw[e] = e < 27 * 16 ? W[e] : bias[e - 27 * 16];
  chain_wait();
  chain_release();
  __syncthreads();
  const int64_t ngroups = (int64_t)nx * ny * nz * nb / V;
  for (int64_t gi = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; gi < ngroups;
       gi += (int64_t)gridDim.x * blockDim.x) {
    const int64_t v0 = gi * V;
    const int64_t row = v0 / nx;  // (b, z, y)
    const int x0 = (int)(v0 - row * nx), y = (int)(row % ny), z = (int)((row / ny) % nz);
    float acc[V][16];
#pragma unroll
    for (int j = 0; j < V; ++j)
#pragma unroll
      for (int c = 0; c < 16; ++c) acc[j][c] = sw[27 * 16 + c];
    // the nine (dz, dy) lines in turn; line li+1 is loaded while line li is used
    float s[2][V + 2];
    auto load_line = [&](int li, float *dst) {
      const int dz = li / 3 - 1, dy = li % 3 - 1;
      const bool line = (unsigned)(y + dy) < (unsigned)ny && (unsigned)(z + dz) < (unsigned)nz;
      const float *p = in + v0 + (int64_t)dy * nx + (int64_t)dz * nx * ny;
#pragma unroll
      for (int k = 0; k < V + 2; ++k) {
        const int xx = x0 + k - 1;
        dst[k] = (line && (unsigned)xx < (unsigned)nx) ? __ldg(p + k - 1) : 0.f;
      }
    };
    load_line(0, s[0]);
#pragma unroll
    for (int li = 0; li < 9; ++li) {
      if (li + 1 < 9) load_line(li + 1, s[(li + 1) & 1]);
      const float *sl = s[li & 1];
#pragma unroll
      for (int dx = -1; dx <= 1; ++dx) {
        const float4 *w4 = reinterpret_cast<const float4 *>(sw + (li * 3 + (dx + 1)) * 16);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float4 w = w4[q];
#pragma unroll
          for (int j = 0; j < V; ++j) {
            const float a = sl[j + dx + 1];
            acc[j][4 * q] = fmaf(a, w.x, acc[j][4 * q]);
            acc[j][4 * q + 1] = fmaf(a, w.y, acc[j][4 * q + 1]);
            acc[j][4 * q + 2] = fmaf(a, w.z, acc[j][4 * q + 2]);
            acc[j][4 * q + 3] = fmaf(a, w.w, acc[j][4 * q + 3]);
          }
        }
      }
    }
#pragma unroll
    for (int j = 0; j < V; ++j) {
      uint32_t w[8];
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        float lo = acc[j][2 * c], hi = acc[j][2 * c + 1];
        if (relu) {
          lo = fmaxf(lo, 0.f);
          hi = fmaxf(hi, 0.f);
        }
        const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
        w[c] = *reinterpret_cast<const uint32_t *>(&h);
      }
      *reinterpret_cast<uint4 *>(out + act_unit(row, 0, x0 + j, nx) * 8) = make_uint4(w[0], w[1], w[2], w[3]);
      *reinterpret_cast<uint4 *>(out + act_unit(row, 1, x0 + j, nx) * 8) = make_uint4(w[4], w[5], w[6], w[7]);
    }
  }
}
__global__ void __launch_bounds__(256) k_conv3_in1(const float *in, const float *W, const float *bias,
                                                   __nv_bfloat16 *out, int nx, int ny, int nz, int nb, int relu) {
  conv3_in1_body<1>(in, W, bias, out, nx, ny, nz, nb, relu);
}
__global__ void __launch_bounds__(256, 2) k_conv3_in1x4(const float *in, const float *W, const float *bias,
                                                     __nv_bfloat16 *out, int nx, int ny, int nz, int nb, int relu) {
  conv3_in1_body<4>(in, W, bias, out, nx, ny, nz, nb, relu);
}

// ---- resampling (row-planar 16-channel tensors; fine dims nx, ny, nz even) -------------------
// Decomposes a unit index of a row-planar tensor into (row, half, x).  Indices
// below 2^32 (every grid of fewer than 2^31 voxels) divide in 32 bits, several
// times cheaper than the 64-bit division.
__device__ __forceinline__ void unit_coords(int64_t u, int nx, int64_t *row, int *h, int *x) {
  if ((uint64_t)u <= 0xFFFFFFFFull) {
    const uint32_t uu = (uint32_t)u, t = uu / (uint32_t)nx;
    *x = (int)(uu - t * (uint32_t)nx);
    *h = (int)(t & 1u);
    *row = (int64_t)(t >> 1);
    return;
  }
  *x = (int)(u % nx);
  const int64_t t = u / nx;
  *h = (int)(t & 1);
  *row = t >> 1;
}
// Row index of (b, z, y) and its inverse.
__device__ __forceinline__ void row_coords(int64_t row, int ny, int nz, int64_t *b, int *z, int *y) {
  if ((uint64_t)row <= 0xFFFFFFFFull) {
    const uint32_t r = (uint32_t)row, t = r / (uint32_t)ny, bb = t / (uint32_t)nz;
    *y = (int)(r - t * (uint32_t)ny);
    *z = (int)(t - bb * (uint32_t)nz);
    *b = (int64_t)bb;
    return;
  }
  *y = (int)(row % ny);
  const int64_t t = row / ny;
  *z = (int)(t % nz);
  *b = t / nz;
}

// 2x2x2 average pooling, one thread per coarse 16-byte unit (8 channels).
__global__ void k_pool(const __nv_bfloat16 *in, __nv_bfloat16 *out, int nx, int ny, int nz, int nb) {
  chain_wait();
  chain_release();
  const int cx = nx / 2, cy = ny / 2, cz = nz / 2;
  const int64_t n = (int64_t)cx * cy * cz * nb * 2;
  const uint4 *src = reinterpret_cast<const uint4 *>(in);
  uint4 *dst = reinterpret_cast<uint4 *>(out);
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
    int64_t row, b;
    int h, xc, zc, yc;
    unit_coords(e, cx, &row, &h, &xc);
    row_coords(row, cy, cz, &b, &zc, &yc);
    float s[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    for (int k = 0; k < 8; ++k) {
      const int64_t rf = (b * nz + 2 * zc + (k >> 2)) * ny + 2 * yc + ((k >> 1) & 1);
      const uint4 q = src[act_unit(rf, h, 2 * xc + (k & 1), nx)];
      const __nv_bfloat162 *p2 = reinterpret_cast<const __nv_bfloat162 *>(&q);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const float2 f = __bfloat1622float2(p2[c]);
        s[2 * c] += f.x;
        s[2 * c + 1] += f.y;
      }
    }
    uint4 o;
    __nv_bfloat162 *o2 = reinterpret_cast<__nv_bfloat162 *>(&o);
#pragma unroll
    for (int c = 0; c < 4; ++c) o2[c] = __floats2bfloat162_rn(0.125f * s[2 * c], 0.125f * s[2 * c + 1]);
    dst[e] = o;
  }
}
// v to p[0] and p[1], one 32-byte store (p on a 32-byte boundary).
__device__ __forceinline__ void store_twice(uint4 *p, uint4 v) {
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %1, %2, %3, %4};" ::"l"(p), "r"(v.x), "r"(v.y), "r"(v.z),
               "r"(v.w)
               : "memory");
}
// Nearest-neighbour 2x upsampling: fine (nx,ny,nz) from coarse (nx/2,...).  One
// thread per coarse 16-byte unit: one load, and its eight fine copies as one
// 32-byte store in each of the four fine rows (nx is even, so two fine units start on
// 32 bytes).  Two 16-byte stores, each filling half of its sectors: 174 us for the
// three levels of a 256^3 pass; 100 here, bound by the bytes.
__global__ void k_upsample(const __nv_bfloat16 *in, __nv_bfloat16 *out, int nx, int ny, int nz, int nb) {
  chain_wait();
  chain_release();
  const int cx = nx / 2, cy = ny / 2, cz = nz / 2;
  const int64_t n = (int64_t)cx * cy * cz * nb * 2;
  const uint4 *src = reinterpret_cast<const uint4 *>(in);
  uint4 *dst = reinterpret_cast<uint4 *>(out);
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
    int64_t row, b;
    int h, xc, zc, yc;
    unit_coords(e, cx, &row, &h, &xc);
    row_coords(row, cy, cz, &b, &zc, &yc);
    const uint4 v = src[e];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int64_t rf = (b * nz + 2 * zc + (k >> 1)) * ny + 2 * yc + (k & 1);
      store_twice(dst + act_unit(rf, h, 2 * xc, nx), v);
    }
  }
}
// Backward of pooling, of the skip connection beside it and of the ReLU before
// both: out = act > 0 ? skip + d_coarse / 8 : 0 in BF16 (skip and d_coarse FP32
// row-planar).  One thread per 16-byte unit of out.  One pass over the three
// tensors where a pass each for the sum and the mask, a float a thread, took
// 144 us at 64^3, batch 4; 22 us here.
__global__ void k_pool_bwd(const float *dc, const float *skip, const __nv_bfloat16 *act, __nv_bfloat16 *out, int nx,
                           int ny, int nz, int nb) {
  chain_wait();
  chain_release();
  const int cx = nx / 2, cy = ny / 2, cz = nz / 2;
  const int64_t n = (int64_t)nx * ny * nz * nb * 2;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
    int64_t row, b;
    int h, x, z, y;
    unit_coords(e, nx, &row, &h, &x);
    row_coords(row, ny, nz, &b, &z, &y);
    const float4 *c4 = reinterpret_cast<const float4 *>(dc) + 2 * act_unit((b * cz + z / 2) * cy + y / 2, h, x / 2, cx);
    const float4 *s4 = reinterpret_cast<const float4 *>(skip) + 2 * e;
    const uint4 m = __ldg(reinterpret_cast<const uint4 *>(act) + e);
    const uint32_t mw[4] = {m.x, m.y, m.z, m.w};
    uint32_t o[4];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const float4 c = __ldg(c4 + k), f = __ldg(s4 + k);
      const __nv_bfloat162 lo = __floats2bfloat162_rn(fmaf(0.125f, c.x, f.x), fmaf(0.125f, c.y, f.y));
      const __nv_bfloat162 hi = __floats2bfloat162_rn(fmaf(0.125f, c.z, f.z), fmaf(0.125f, c.w, f.w));
      o[2 * k] = relu_mask2(*reinterpret_cast<const uint32_t *>(&lo), mw[2 * k]);
      o[2 * k + 1] = relu_mask2(*reinterpret_cast<const uint32_t *>(&hi), mw[2 * k + 1]);
    }
    reinterpret_cast<uint4 *>(out)[e] = make_uint4(o[0], o[1], o[2], o[3]);
  }
}
// Backward of nearest upsampling and of the ReLU before it: out = act > 0 ? the
// sum of the 8 fine children : 0 in BF16.  One thread per 16-byte unit of out.
__global__ void k_up_bwd(const float *df, const __nv_bfloat16 *act, __nv_bfloat16 *out, int nx, int ny, int nz,
                         int nb) {
  chain_wait();
  chain_release();
  const int cx = nx / 2, cy = ny / 2, cz = nz / 2;
  const int64_t n = (int64_t)cx * cy * cz * nb * 2;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
    int64_t row, b;
    int h, xc, zc, yc;
    unit_coords(e, cx, &row, &h, &xc);
    row_coords(row, cy, cz, &b, &zc, &yc);
    const uint4 m = __ldg(reinterpret_cast<const uint4 *>(act) + e);
    float4 s[2] = {};
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int64_t rf = (b * nz + 2 * zc + (k >> 2)) * ny + 2 * yc + ((k >> 1) & 1);
      const float4 *f4 = reinterpret_cast<const float4 *>(df) + 2 * act_unit(rf, h, 2 * xc + (k & 1), nx);
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const float4 f = __ldg(f4 + j);
        s[j].x += f.x;
        s[j].y += f.y;
        s[j].z += f.z;
        s[j].w += f.w;
      }
    }
    const uint32_t mw[4] = {m.x, m.y, m.z, m.w};
    uint32_t o[4];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const __nv_bfloat162 lo = __floats2bfloat162_rn(s[j].x, s[j].y), hi = __floats2bfloat162_rn(s[j].z, s[j].w);
      o[2 * j] = relu_mask2(*reinterpret_cast<const uint32_t *>(&lo), mw[2 * j]);
      o[2 * j + 1] = relu_mask2(*reinterpret_cast<const uint32_t *>(&hi), mw[2 * j + 1]);
    }
    reinterpret_cast<uint4 *>(out)[e] = make_uint4(o[0], o[1], o[2], o[3]);
  }
}

// ---- gradients --------------------------------------------------------------------------------
// grad[k] (+)= sum over blocks of partial[block][k], k < n.  Thread (k, r) of a
// block's 32 x 8 sums the partials r, r + 8, ... in order, then the eight sums
// are added in order, all in FP64: the result does not depend on the grid.
// (One thread per k summing every partial: 14.8 against 4 us a layer.)
__global__ void __launch_bounds__(256) k_reduce_partials(const float *partial, int nblocks, int n, float *grad,
                                                         int accumulate) {
  chain_wait();
  chain_release();
  __shared__ double s[8][32];
  const int c = threadIdx.x & 31, r = threadIdx.x >> 5, k = blockIdx.x * 32 + c;
  double v = 0.0;
  if (k < n)
    for (int b = r; b < nblocks; b += 8) v += (double)partial[(size_t)b * n + k];
  s[r][c] = v;
  __syncthreads();
  if (r == 0 && k < n) {
    for (int j = 1; j < 8; ++j) v += s[j][c];
    grad[k] = accumulate ? grad[k] + (float)v : (float)v;
  }
}

// Voxel index -> unit of its first half.
__device__ __forceinline__ int64_t voxel_unit(int64_t v, int nx) {
  const int64_t row = (uint64_t)v <= 0xFFFFFFFFull ? (int64_t)((uint32_t)v / (uint32_t)nx) : v / nx;
  return act_unit(row, 0, (int)(v - row * nx), nx);
}

// Output projection (training path): out[v] = proj . act[v] + proj_b.
__global__ void k_proj_fwd(const __nv_bfloat16 *act, const float *proj, float *out, int64_t nvox, int nx) {
  chain_wait();
  chain_release();
  for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < nvox; v += (int64_t)gridDim.x * blockDim.x) {
    float f[16], r = proj[16];
    load_voxel(act, voxel_unit(v, nx), nx, f);
#pragma unroll
    for (int c = 0; c < 16; ++c) r = fmaf(proj[c], f[c], r);
    out[v] = r;
  }
}
// d act = proj * dOut (masked by act > 0, to BF16); per-block partials of
// dproj[c] = sum act[v][c] dOut[v] and dproj_b = sum dOut[v] ([block][17]).
// 16-byte units in and out (one element at a time: 56 us at 64^3, batch 4; 16 us here).
__global__ void __launch_bounds__(256) k_proj_bwd(const __nv_bfloat16 *act, const float *proj, const float *dout,
                                                  __nv_bfloat16 *dact, float *partial, int64_t nvox, int nx) {
  chain_wait();
  chain_release();
  __shared__ float red[17][256];
  float acc[17];
#pragma unroll
  for (int c = 0; c < 17; ++c) acc[c] = 0.f;
  for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < nvox; v += (int64_t)gridDim.x * blockDim.x) {
    const float d = dout[v];
    const int64_t u = voxel_unit(v, nx);
    float f[16];
    load_voxel(act, u, nx, f);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      uint32_t w[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        float o[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int c = 8 * h + 2 * k + j;
          acc[c] = fmaf(f[c], d, acc[c]);
          o[j] = f[c] > 0.f ? proj[c] * d : 0.f;
        }
        const __nv_bfloat162 b = __floats2bfloat162_rn(o[0], o[1]);
        w[k] = *reinterpret_cast<const uint32_t *>(&b);
      }
      reinterpret_cast<uint4 *>(dact)[u + (int64_t)h * nx] = make_uint4(w[0], w[1], w[2], w[3]);
    }
    acc[16] += d;
  }
#pragma unroll
  for (int c = 0; c < 17; ++c) red[c][threadIdx.x] = acc[c];
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if (threadIdx.x < w)
      for (int c = 0; c < 17; ++c) red[c][threadIdx.x] += red[c][threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x < 17) partial[(size_t)blockIdx.x * 17 + threadIdx.x] = red[threadIdx.x][0];
}

// Mean squared error over n values and dL/dout; per-block loss partials.
__global__ void __launch_bounds__(256) k_mse(const float *out, const float *tgt, float *dout, float *partial,
                                             int64_t n) {
  chain_wait();
  chain_release();
  __shared__ float red[256];
  float s = 0.f;
  const float scale = 2.f / (float)n;
  for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x) {
    const float e = out[v] - tgt[v];
    s += e * e;
    dout[v] = scale * e;
  }
  red[threadIdx.x] = s;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) partial[blockIdx.x] = red[0];
}

// Four floats at p, which need not be 16-byte aligned.
__device__ __forceinline__ float4 load4(const float *p) {
  if (((uintptr_t)p & 15) == 0) return __ldg(reinterpret_cast<const float4 *>(p));
  return make_float4(__ldg(p), __ldg(p + 1), __ldg(p + 2), __ldg(p + 3));
}

// Energy-norm loss of the HPCCG operator A (the 27-point generate_matrix
// stencil: 27 on the diagonal, -1 for each neighbour inside the grid):
// L = (1/n) d.(A d), d = target - out, per grid of the batch; dL/dout = -(2/n) A d.
// A thread forms four voxels of a row (nx a multiple of 4): per (dz, dy) line it
// loads the six differences around them once, out-of-grid ones as zeros.  99 -> 18 us
// at 64^3, batch 4, against a voxel a thread and 54 loads one by one.
__global__ void __launch_bounds__(256) k_energy(const float *out, const float *tgt, float *dout, float *partial,
                                                int nx, int ny, int nz, int nb) {
  chain_wait();
  chain_release();
  __shared__ float red[256];
  const int64_t n = (int64_t)nx * ny * nz * nb;
  const float scale = 2.f / (float)n;
  float s = 0.f;
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n / 4; q += (int64_t)gridDim.x * blockDim.x) {
    const int64_t v = 4 * q, row = (uint64_t)v <= 0xFFFFFFFFull ? (int64_t)((uint32_t)v / (uint32_t)nx) : v / nx;
    int64_t b;
    int y, z;
    const int x = (int)(v - row * nx);
    row_coords(row, ny, nz, &b, &z, &y);
    float ad[4] = {0.f, 0.f, 0.f, 0.f}, dc[4];
#pragma unroll
    for (int li = 0; li < 9; ++li) {
      const int dy = li % 3 - 1, dz = li / 3 - 1;
      const bool line = (unsigned)(y + dy) < (unsigned)ny && (unsigned)(z + dz) < (unsigned)nz;
      const int64_t u = v + ((int64_t)dz * ny + dy) * nx;
      float d[6];
      d[0] = line && x > 0 ? __ldg(tgt + u - 1) - __ldg(out + u - 1) : 0.f;
      d[5] = line && x + 4 < nx ? __ldg(tgt + u + 4) - __ldg(out + u + 4) : 0.f;
      const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
      const float4 t4 = line ? load4(tgt + u) : zero, o4 = line ? load4(out + u) : zero;
      d[1] = t4.x - o4.x;
      d[2] = t4.y - o4.y;
      d[3] = t4.z - o4.z;
      d[4] = t4.w - o4.w;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (li == 4) dc[j] = d[j + 1];
#pragma unroll
        for (int k = 0; k < 3; ++k) ad[j] = fmaf(li == 4 && k == 1 ? 27.f : -1.f, d[j + k], ad[j]);
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      s = fmaf(dc[j], ad[j], s);
      dout[v + j] = -scale * ad[j];
    }
  }
  red[threadIdx.x] = s;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) partial[blockIdx.x] = red[0];
}

__global__ void k_adam(float *p, const float *g, float *m, float *v, int n, float lr, float b1, float b2, float eps,
                       float c1, float c2) {
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
    const float gk = g[k];
    const float mk = b1 * m[k] + (1.f - b1) * gk;
    const float vk = b2 * v[k] + (1.f - b2) * gk * gk;
    m[k] = mk;
    v[k] = vk;
    p[k] -= lr * (mk / c1) / (sqrtf(vk / c2) + eps);
  }
}

}  // namespace hpccg
