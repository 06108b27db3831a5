// unet_ops.cuh -- declarations of the CUDA-core U-Net kernels (unet_ops.cu).
#pragma once
#include "unet_conv.cuh"

namespace hpccg {

struct CcConvArgs {
  int nx, ny, nz, nb;
  int nin;                           // 16-channel input groups
  const __nv_bfloat16 *in0, *in1;    // row-planar BF16 inputs
  const float *W;                    // FP32 [27][16 nin][16]
  const float *bias;                 // [16] or null
  const float *proj;                 // [17] for kEpiProject
  const __nv_bfloat16 *act;          // for kEpiMask
  int epi;
  void *out;
  bool chained;                      // launch_chained
};

struct DwArgs {
  int nx, ny, nz, nb, cin;
  const __nv_bfloat16 *x0, *x1;      // forward inputs (channels 0-15, 16-31)
  const float *x_f32;                // or the 1-channel FP32 input
  const __nv_bfloat16 *dy;           // gradient w.r.t. the pre-activation output
  float *partial;                    // [gridDim.x][27*cin + 1][16]
};

// The 16 channels of a voxel as floats.
__device__ __forceinline__ void load_voxel(const __nv_bfloat16 *act, int64_t unit0, int nx, float *f) {
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const uint4 q = __ldg(reinterpret_cast<const uint4 *>(act) + unit0 + (int64_t)h * nx);
    const __nv_bfloat162 *p2 = reinterpret_cast<const __nv_bfloat162 *>(&q);
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const float2 t = __bfloat1622float2(p2[c]);
      f[8 * h + 2 * c] = t.x;
      f[8 * h + 2 * c + 1] = t.y;
    }
  }
}
// Two FP32 numbers in a register pair, and their fused multiply-add.
__device__ __forceinline__ unsigned long long pack_f32x2(float lo, float hi) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack_f32x2(unsigned long long v, float &lo, float &hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ void fma_f32x2(unsigned long long &d, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}

__global__ void k_pack_fwd(const float *W, int cin, int nin, __nv_bfloat16 *packed);
__global__ void k_pack_bwd(const float *W, int cin, int g, __nv_bfloat16 *packed);
__global__ void k_flip_fp32(const float *W, int cin, int g, float *Wf);
int launch_conv3_cc(const CcConvArgs &a, int num_sms, cudaStream_t s);
__global__ void k_conv3_in1(const float *in, const float *W, const float *bias, __nv_bfloat16 *out, int nx, int ny,
                            int nz, int nb, int relu);
__global__ void k_conv3_in1x4(const float *in, const float *W, const float *bias, __nv_bfloat16 *out, int nx, int ny,
                              int nz, int nb, int relu);  // nx a multiple of 4
__global__ void k_pool(const __nv_bfloat16 *in, __nv_bfloat16 *out, int nx, int ny, int nz, int nb);
__global__ void k_upsample(const __nv_bfloat16 *in, __nv_bfloat16 *out, int nx, int ny, int nz, int nb);
__global__ void k_pool_bwd(const float *dc, const float *skip, const __nv_bfloat16 *act, __nv_bfloat16 *out, int nx,
                           int ny, int nz, int nb);
__global__ void k_up_bwd(const float *df, const __nv_bfloat16 *act, __nv_bfloat16 *out, int nx, int ny, int nz, int nb);
__global__ void k_reduce_partials(const float *partial, int nblocks, int n, float *grad, int accumulate);
__global__ void k_proj_fwd(const __nv_bfloat16 *act, const float *proj, float *out, int64_t nvox, int nx);
__global__ void k_proj_bwd(const __nv_bfloat16 *act, const float *proj, const float *dout, __nv_bfloat16 *dact,
                           float *partial, int64_t nvox, int nx);
__global__ void k_mse(const float *out, const float *tgt, float *dout, float *partial, int64_t n);
__global__ void k_energy(const float *out, const float *tgt, float *dout, float *partial, int nx, int ny, int nz,
                         int nb);
__global__ void k_adam(float *p, const float *g, float *m, float *v, int n, float lr, float b1, float b2, float eps,
                       float c1, float c2);

// Weight and bias gradient partials of one layer (unet_dw.cu): at most max_blocks
// of [27*cin + 1][16] in a.partial; *blocks receives their number.
int launch_dW(const DwArgs &a, int max_blocks, int *err, int num_sms, cudaStream_t s, int *blocks);

}  // namespace hpccg
