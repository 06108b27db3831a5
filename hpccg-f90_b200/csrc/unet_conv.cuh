// unet_conv.cuh -- 3x3x3 convolutions with 16 output channels on tcgen05.
//
// Activation layout ("row-planar"): a 16-channel tensor of nb grids of
// nx*ny*nz voxels is stored as [b][z][y][h][x][8] -- for every grid row
// (b,z,y), first the 8-channel half h=0 of all nx voxels, then h=1.  A voxel
// half is one 16-byte unit, and a run of consecutive voxels of one row and
// half is one contiguous span, which is exactly the layout the tensor cores
// read (no-swizzle K-major core matrices: 8 rows x 16 bytes; the two halves
// are the two K chunks).  So operand tiles are fetched as they lie: boxes of a
// 5D tensor map (act_tmap) or whole row spans, with zero fill at the grid faces.
//
// A conv is an implicit GEMM on tcgen05 over the 27 taps and each 16-channel
// input group, accumulated in FP32 in TMEM:
//  * window tiles (unet_conv_win.cu, with its roles and copies): the network's
//    form; voxels are the MMA's N, eight output rows x 16 channels its M;
//  * brick tiles (unet_conv.cu): 128 voxels of a bx*by*bz brick are M, the 16
//    channels N, each tap's shifted brick fetched on its own.  Kept as the
//    independent form that hpccg_unet_conv3_layer offers beside the other two.
//    192 threads: warp 0 fetches (its lanes issue 1D bulk copies of the row spans in
//    parallel), warp 1 allocates TMEM and lane 0 issues the MMAs, warps 2-5 (one
//    per TMEM lane quarter) run the epilogue.
#pragma once
#include "hpccg_internal.cuh"
#include "unet_tc.cuh"

namespace hpccg {

// Offsets in the row-planar layout; row = (b*nz + z)*ny + y.
__host__ __device__ __forceinline__ int64_t act_unit(int64_t row, int h, int x, int nx) {
  return (row * 2 + h) * (int64_t)nx + x;
}
__host__ __device__ __forceinline__ int64_t act_elem(int64_t row, int x, int c, int nx) {
  return act_unit(row, c >> 3, x, nx) * 8 + (c & 7);
}

constexpr int kConvThreads = 192;
constexpr int kWTapBytes = 16 * 16 * 2;  // one tap of B: 16 x 16 BF16

// Brick tiles: one stage per k-step (tap, input): 2 halves x 128 units.
constexpr int kBrickStages = 24;
constexpr int kBrickStageBytes = 2 * 128 * 16;
// mbarriers: full[S], empty[S], acc_full[2], acc_empty[2], drain, + TMEM slot.
__host__ __device__ constexpr int bar_bytes(int stages) { return (2 * stages + 5) * 8 + 16; }
__host__ __device__ constexpr int brick_smem_bytes(int nin) {
  return nin * 27 * kWTapBytes + kBrickStages * kBrickStageBytes + bar_bytes(kBrickStages);
}

// ---- chained launches -----------------------------------------------------------------
// The network's kernels run one after the other in a stream, many of them for less
// than 10 us.  launch_chained lets a kernel's blocks start while its predecessor
// drains, so that their set-up (barriers, TMEM, weights in shared memory) and the launch
// itself are off the path.  Two rules keep that sound:
//  - Every thread calls chain_wait() before it touches memory that a kernel of the
//    chain writes: it returns when the predecessor has finished and its results
//    are visible.  chain_release(), which lets the successor start, comes after it,
//    so a kernel starts after all but its direct predecessor have finished.  Weights
//    may be read before the wait: the kernels that pack them are no part of a
//    chain, whose first kernel is launched the plain way.
//  - chain_release() comes after the block has its TMEM.  A successor's block on
//    the same SM may hold TMEM while it waits for this kernel; were this block
//    still to allocate, neither would go on.
// Forward pass / gradient, plain against chained launches: 32^3 195 -> 147 / 658 ->
// 494 us, 64^3 batch 4 332 -> 293 / 1265 -> 1155, 128^3 467 -> 425, 256^3 2251 ->
// 2238, 24^3 298 -> 242 / 832 -> 650.
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void chain_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename... P, typename... A>
inline cudaError_t launch_chained(void (*kern)(P...), int grid, int block, int smem, cudaStream_t s, bool chained,
                                  A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at = {};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = chained ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...);
}

enum ConvEpi : int {
  kEpiBiasRelu = 0,   // out_bf16 = relu(acc + bias)
  kEpiBias = 1,       // out_bf16 = acc + bias
  kEpiProject = 2,    // out_f32[voxel] = proj . relu(acc + bias) + proj_bias
  kEpiRawF32 = 3,     // out_f32 = acc (16 channels, row-planar)
  kEpiMask = 4,       // out_bf16 = act > 0 ? acc : 0, act as wide as out (backward of a ReLU; one input group)
};

struct ConvGeom {
  int nx, ny, nz, nb;  // volume and batch
  int bx, by, bz;      // tile brick (bx*by*bz = 128)
  int tx, ty, tz;      // tiles per dimension
  int ntiles;
};

struct ConvArgs {
  ConvGeom g;
  const __nv_bfloat16 *in0, *in1;  // row-planar inputs
  const __nv_bfloat16 *wpack;      // [nin][27][2][16][8] BF16
  const float *bias;               // [16] (null for kEpiRawF32)
  const float *proj;               // [17] for kEpiProject
  const __nv_bfloat16 *act;        // for kEpiMask
  void *out;
  int *err;
  bool chained;                    // launch_chained
};

// Two BF16 gradients where the activations' pair is positive, zeros elsewhere.
__device__ __forceinline__ uint32_t relu_mask2(uint32_t grad, uint32_t act) {
  return grad & __hgt2_mask(*reinterpret_cast<const __nv_bfloat162 *>(&act), __float2bfloat162_rn(0.f));
}

// Host: brick and tile counts for a volume (dims must be divisible by the brick).
inline bool conv_geom(int nx, int ny, int nz, int nb, ConvGeom *g) {
  if ((int64_t)nx * ny * nz < 128) return false;
  int bx = nx < 128 ? nx : 128;
  int by = 128 / bx;
  if (by > ny) by = ny;
  int bz = 128 / (bx * by);
  if (bx < 8 || bx * by * bz != 128 || nx % bx || ny % by || nz % bz) return false;
  g->nx = nx;
  g->ny = ny;
  g->nz = nz;
  g->nb = nb;
  g->bx = bx;
  g->by = by;
  g->bz = bz;
  g->tx = nx / bx;
  g->ty = ny / by;
  g->tz = nz / bz;
  g->ntiles = g->tx * g->ty * g->tz * nb;
  return true;
}

// One lane's share of a fetch: the span of `len` units of half h of grid row
// (b, z, y) starting at voxel xs goes to dst.  Units outside the grid are
// zeroed here (generic stores); the in-grid part is described for a later
// bulk copy.
struct Span {
  const __nv_bfloat16 *src;
  uint8_t *dst;
  uint32_t bytes;
  bool zeroed;  // this lane wrote zero fill with ordinary stores
};

__device__ __forceinline__ Span plan_span(const ConvGeom &g, const __nv_bfloat16 *base, int b, int z, int y, int h,
                                          int xs, int len, uint8_t *dst) {
  Span sp{nullptr, nullptr, 0, false};
  const uint4 zero = make_uint4(0, 0, 0, 0);
  if (z < 0 || z >= g.nz || y < 0 || y >= g.ny) {
    for (int u = 0; u < len; ++u) reinterpret_cast<uint4 *>(dst)[u] = zero;
    sp.zeroed = true;
    return sp;
  }
  const int lo = max(xs, 0), hi = min(xs + len, g.nx);
  for (int u = 0; u < lo - xs; ++u) reinterpret_cast<uint4 *>(dst)[u] = zero;
  for (int u = hi - xs; u < len; ++u) reinterpret_cast<uint4 *>(dst)[u] = zero;
  sp.zeroed = lo > xs || hi < xs + len;
  if (hi <= lo) return sp;
  const int64_t row = ((int64_t)b * g.nz + z) * g.ny + y;
  sp.src = base + act_unit(row, h, lo, g.nx) * 8;
  sp.dst = dst + (lo - xs) * 16;
  sp.bytes = (uint32_t)(hi - lo) * 16;
  return sp;
}

// Posts the stage: lanes that zero-filled fence their stores into the async
// proxy, lane 0 arms the barrier with the warp's total bulk bytes, then every
// lane issues its copies.
__device__ __forceinline__ void post_spans(const Span *sp, int nsp, uint64_t *bar, int lane) {
  uint32_t bytes = 0;
  bool zeroed = false;
  for (int i = 0; i < nsp; ++i) {
    bytes += sp[i].bytes;
    zeroed |= sp[i].zeroed;
  }
  if (zeroed) tc::fence_proxy_async_smem();  // only lanes that stored zeros
  const uint32_t total = __reduce_add_sync(0xffffffffu, bytes);
  __syncwarp();
  if (lane == 0) tc::mbar_expect_tx(bar, total);
  __syncwarp();
  for (int i = 0; i < nsp; ++i)
    if (sp[i].bytes) tc::bulk_g2s(sp[i].dst, sp[i].src, sp[i].bytes, bar);
}

// Lane 0 waits, the result is shared with the warp.
__device__ __forceinline__ bool warp_wait(uint64_t *bar, uint32_t parity, int *err, int where, int lane) {
  bool ok = true;
  if (lane == 0) ok = tc::mbar_wait(bar, parity, err, where);
  ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
  __syncwarp();
  return ok;
}

// Tensor maps of an activation tensor.  Elements are 8 bytes (half of a 16-byte
// unit), so a box may be 128 units long in x; zeros outside the grid.  The box's
// dimensions come in the given order, each with its extent in the box.
enum ActDim : int { kDimH, kDimY, kDimZ };
inline int act_tmap(CUtensorMap *map, const __nv_bfloat16 *base, const ConvGeom &g, int box_units, ActDim d1, int n1,
                    ActDim d2, int n2, ActDim d3, int n3) {
  const ActDim d[3] = {d1, d2, d3};
  const int n[3] = {n1, n2, n3};
  cuuint64_t dims[5] = {(cuuint64_t)2 * g.nx, 0, 0, 0, (cuuint64_t)g.nb}, strides[4];
  cuuint32_t box[5] = {(cuuint32_t)(2 * box_units), 0, 0, 0, 1};
  const cuuint64_t row = (cuuint64_t)g.nx * 32;  // bytes of a grid row, both halves
  for (int i = 0; i < 3; ++i) {
    dims[i + 1] = d[i] == kDimH ? 2 : (d[i] == kDimY ? g.ny : g.nz);
    strides[i] = d[i] == kDimH ? row / 2 : (d[i] == kDimY ? row : row * g.ny);
    box[i + 1] = (cuuint32_t)n[i];
  }
  strides[3] = row * g.ny * g.nz;
  return encode_tmap(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 5, base, dims, strides, box,
                     CU_TENSOR_MAP_L2_PROMOTION_L2_256B);
}

// Launch the tensor-core conv: window tiles (any volume; reads nx, ny, nz, nb of
// a.g only) and brick tiles (a.g from conv_geom).
int launch_conv3_win(int nin, int epi, const ConvArgs &a, int num_sms, cudaStream_t s);
int launch_conv3_brick(int nin, int epi, const ConvArgs &a, int num_sms, cudaStream_t s);
// The 1-channel input layer (FP32 input [nb][nz][ny][nx], W [27][16], bias [16])
// on the tensor cores, BF16 operands, FP32 accumulation; nx a multiple of 128,
// else HPCCG_ERR_UNSUPPORTED.
int launch_conv3_in1_tc(const float *in, const float *W, const float *bias, __nv_bfloat16 *out, int nx, int ny,
                        int nz, int nb, int relu, int *err, int num_sms, cudaStream_t s);

}  // namespace hpccg
