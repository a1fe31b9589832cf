// fcb_conv.cu -- 3x3x3 convolutions (16 -> 16 channels, stride 1, zero padding 1) for the
// learned reconstruction's CNN, on the 5th-generation tensor cores (sm_100a tcgen05).
//
// Activations are BF16 in a channel-half-major layout, [z][y][2][x][8]: for every (z, y) row
// the 8 channels of half 0 of all x, then those of half 1, so that a TMA box of one half of
// one row is contiguous (no 32-byte sector is fetched for 16 useful bytes).  Weights BF16
// [27 taps][16 out][16 in]; accumulation FP32 in tensor memory.  Implicit GEMM: a CTA owns
// 128 consecutive x-voxels of one (y, z) row -> D[128 x 16] = sum over 27 taps of
// A_tap[128 x 16 in] * B_tap[16 in x 16 out].  The A operands of the three x-shifts of a tap
// row are the same TMA-loaded row of 130 voxels addressed 16 bytes apart, so 9 row loads
// (x 2 channel halves) feed all 27 MMAs.  Out-of-volume rows/voxels arrive as zeros from the
// TMA unit, which is the zero padding.  One elected thread issues the 27
// tcgen05.mma.cta_group::1.kind::f16 (M=128, N=16, K=16) and commits to an mbarrier; four
// warps read their TMEM lane quadrant back (tcgen05.ld 32x32b.x16), add the bias, apply
// ReLU and store.
//
// The same kernels compute the input gradient (transposed, tap-flipped weights, prepared by
// the caller); conv3d16n_kernel is the default form.  The weight gradient, a
// 6912-entry reduction over all voxels, runs on the tensor cores too
// (conv3d16_wgrad_tc_kernel, BF16 dY) with a CUDA-core kernel for FP32 dY and comparison.
#include <stdlib.h>
#include <string.h>

#include <algorithm>

#include "fcb_internal.h"

namespace fcb {
namespace tc {

__device__ __forceinline__ void tmem_alloc(uint32_t* dst, uint32_t ncols)
{
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dev::smem_u32(dst)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish()
{
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols)
{
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// D(tmem) (+)= A(smem desc) * B(smem desc), BF16 inputs, FP32 accumulator.
__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                         uint32_t accumulate)
{
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.u32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void mma_commit(uint64_t* bar)
{
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                   dev::smem_u32(bar))
               : "memory");
}
// 32 lanes x 16 consecutive 32-bit columns: thread i of the warp gets row (lane base + i).
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16])
{
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// zeros into 32 lanes x 16 consecutive 32-bit columns
__device__ __forceinline__ void tmem_zero16(uint32_t taddr)
{
  asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1};" ::"r"(
                   taddr),
               "r"(0u)
               : "memory");
}

// Shared-memory matrix descriptor, K-major, no swizzle ("interleaved" core matrices of 8
// rows x 16 bytes): start address, leading byte offset (between the two 8-element K
// halves), stride byte offset (between 8-row groups), descriptor version 1 (sm_100).
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo)
{
  return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

// Instruction descriptor, kind::f16: FP32 accumulator, BF16 A and B, both K-major, N, M.
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N)
{
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void tma_load_5d(void* dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1,
                                            int c2, int c3, int c4)
{
  asm volatile(
      "cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3, %4, %5, %6}], [%7];" ::"r"(dev::smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4),
      "r"(dev::smem_u32(bar))
      : "memory");
}

// Offset (elements) of channel c of voxel (x, y, z) in the [z][y][2][x][8] layout.
__host__ __device__ __forceinline__ size_t act_index(int x, int y, int z, int c, int nx, int ny)
{
  return ((((size_t)z * ny + y) * 2 + (c >> 3)) * nx + x) * 8 + (c & 7);
}

}  // namespace tc

constexpr int CV_TILE = 128;                  // voxels per CTA tile (MMA M)
constexpr int CV_ROW = CV_TILE + 2;           // staged voxels per tap row (x halo)
constexpr int CV_BOX_BYTES = CV_ROW * 16;     // one channel half of one tap row
constexpr int CV_RB = 2176;                   // CV_BOX_BYTES rounded up to 128 B
static_assert((CV_ROW + 2) / 2 * 32 <= CV_RB && CV_BOX_BYTES <= CV_RB, "a staged box fits its slot");
constexpr int CV_A_BYTES = 9 * 2 * CV_RB;     // 39168
constexpr int CV_W_BYTES = 27 * 512;          // 13824
constexpr int CV_SMEM = CV_A_BYTES + CV_W_BYTES + 64 + 32 + 16;

struct ConvParams {
  int gs;                  // log2 of the voxels per box row
  int yl, zl;              // rows and planes of a walk (conv3d16n_kernel)
  uint32_t box_bytes;      // bytes of one TMA box
  const __nv_bfloat16* w;  // [27][16 out][16 in]
  const float* bias;       // [16] or null
  void* out;               // [z][y][x][16], bf16 or f32
  int out_f32;
  int relu;
  int nx, ny, nz;
  int tiles_x;
  int* status;
};

__global__ void __launch_bounds__(128) conv3d16_kernel(const __grid_constant__ CUtensorMap xmap,
                                                       const __grid_constant__ ConvParams P)
{
  extern __shared__ __align__(1024) unsigned char smem[];
  unsigned char* A = smem;
  unsigned char* Wsm = smem + CV_A_BYTES;
  float* bias = reinterpret_cast<float*>(Wsm + CV_W_BYTES);
  uint64_t* bars = reinterpret_cast<uint64_t*>(Wsm + CV_W_BYTES + 64);  // [0] tma, [1] mma
  uint32_t* tslot = reinterpret_cast<uint32_t*>(Wsm + CV_W_BYTES + 64 + 16);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tile = blockIdx.x;
  const int x0 = (tile % P.tiles_x) * CV_TILE;
  const int yz = tile / P.tiles_x;
  const int y = yz % P.ny, z = yz / P.ny;

  if (threadIdx.x == 0) {
    dev::mbar_init(&bars[0], 1);
    dev::mbar_init(&bars[1], 1);
    dev::fence_mbar_init();
  }
  if (warp == 0) {
    tc::tmem_alloc(tslot, 32);
    tc::tmem_relinquish();
  }
  tc::fence_before();
  __syncthreads();

  if (threadIdx.x == 0) {
    dev::tma_prefetch(&xmap);
    dev::mbar_arrive_expect_tx(&bars[0], 18u * P.box_bytes);
    for (int r = 0; r < 9; r++) {
      const int dz = r / 3, dy = r % 3;
      for (int kh = 0; kh < 2; kh++)
        tc::tma_load_5d(A + (r * 2 + kh) * CV_RB, &xmap, &bars[0], 0, (x0 >> P.gs) - 1, kh,
                        y + dy - 1, z + dz - 1);
    }
  }
  // weights -> core-matrix layout: tap t, K half kh, row n (out channel): 16 bytes of 8 in-channels
  const uint4* wg = reinterpret_cast<const uint4*>(P.w);
  for (int i = threadIdx.x; i < 27 * 16 * 2; i += blockDim.x) {
    const int t = i / 32, n = (i / 2) % 16, kh = i % 2;
    reinterpret_cast<uint4*>(Wsm + t * 512 + kh * 256 + n * 16)[0] = wg[(t * 16 + n) * 2 + kh];
  }
  if (threadIdx.x < 16) bias[threadIdx.x] = P.bias ? P.bias[threadIdx.x] : 0.0f;
  // generic-proxy shared stores -> visible to the tensor core's async-proxy reads
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  __syncthreads();
  tc::fence_after();
  const uint32_t taddr = *tslot;

  bool ok = true;
  if (threadIdx.x == 0) {
    ok = dev::mbar_wait(&bars[0], 0);
    if (ok) {
      tc::fence_after();
      const uint32_t abase = dev::smem_u32(A), wbase = dev::smem_u32(Wsm);
      constexpr uint32_t IDESC = tc::idesc_bf16(CV_TILE, 16);
      for (int t = 0; t < 27; t++) {
        const int r = t / 3, dx = t % 3;
        const uint64_t ad = tc::smem_desc(abase + r * 2 * CV_RB + (dx + (1 << P.gs) - 1) * 16, CV_RB, 128);
        const uint64_t bd = tc::smem_desc(wbase + t * 512, 256, 128);
        tc::mma_bf16(taddr, ad, bd, IDESC, t > 0 ? 1u : 0u);
      }
      tc::mma_commit(&bars[1]);
    } else {
      dev::record_status(P.status, DEV_TIMEOUT);
      dev::mbar_wait(&bars[0], 0, 100000000ull);  // let in-flight copies land before exit
    }
  }
  // every thread waits (bounded) for the MMA commit; the result must be warp-uniform
  // because tcgen05.ld is a warp-collective instruction
  const bool done = __all_sync(0xffffffffu, dev::mbar_wait(&bars[1], 0) ? 1 : 0) != 0;
  tc::fence_after();
  if (done) {
    uint32_t r[16];
    tc::tmem_ld16(taddr + ((uint32_t)(warp * 32) << 16), r);
    const int row = warp * 32 + lane;
    const int xv = x0 + row;
    if (xv < P.nx) {
      float v[16];
#pragma unroll
      for (int c = 0; c < 16; c++) {
        v[c] = __uint_as_float(r[c]) + bias[c];
        if (P.relu) v[c] = fmaxf(v[c], 0.0f);
      }
      const size_t i0 = tc::act_index(xv, y, z, 0, P.nx, P.ny), i1 = tc::act_index(xv, y, z, 8, P.nx, P.ny);
      if (P.out_f32) {
        float4* o0 = reinterpret_cast<float4*>(reinterpret_cast<float*>(P.out) + i0);
        float4* o1 = reinterpret_cast<float4*>(reinterpret_cast<float*>(P.out) + i1);
        o0[0] = make_float4(v[0], v[1], v[2], v[3]);
        o0[1] = make_float4(v[4], v[5], v[6], v[7]);
        o1[0] = make_float4(v[8], v[9], v[10], v[11]);
        o1[1] = make_float4(v[12], v[13], v[14], v[15]);
      } else {
        uint32_t pk[8];
#pragma unroll
        for (int q = 0; q < 8; q++) {
          __nv_bfloat162 b = __floats2bfloat162_rn(v[2 * q], v[2 * q + 1]);
          pk[q] = *reinterpret_cast<uint32_t*>(&b);
        }
        __nv_bfloat16* ob = reinterpret_cast<__nv_bfloat16*>(P.out);
        *reinterpret_cast<uint4*>(ob + i0) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
        *reinterpret_cast<uint4*>(ob + i1) = make_uint4(pk[4], pk[5], pk[6], pk[7]);
      }
    }
  } else if (threadIdx.x == 32) {
    dev::record_status(P.status, DEV_TIMEOUT);
  }
  // MMAs must have finished before the accumulator columns are released
  if (!done && threadIdx.x == 0 && ok) dev::mbar_wait(&bars[1], 0, 100000000ull);
  tc::fence_before();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(taddr, 32);
}

// Persistent, pipelined form of the same convolution: one CTA per SM walks the row tiles
// (tile = blockIdx.x + i * gridDim.x) with warp-specialised roles --
//   warp 4 (one lane): TMA producer, 18 row boxes per tile into a ring of CVP_STAGES buffers;
//   warp 5 (one lane): MMA issuer, 27 tcgen05.mma per tile into one of two TMEM
//                       accumulators (16 columns each), commits to the ring's empty barrier
//                       and to the accumulator's full barrier;
//   warps 0-3:         epilogue, each reads its 32-lane TMEM quadrant of the finished
//                       accumulator, releases it, adds bias / ReLU and stores.
// The weights are staged once per CTA, TMEM is allocated once, and the loads of the next
// tiles, the MMAs of this one and the stores of the previous one overlap.  Every wait is
// bounded; a role that times out records the status and stops, and the others stop at their
// next (bounded) wait.
constexpr int CVP_STAGES = 4;
constexpr int CVP_THREADS = 192;
constexpr int CVP_SMEM = CVP_STAGES * CV_A_BYTES + CV_W_BYTES + 64 + 8 * (2 * CVP_STAGES + 4) + 16;

__global__ void __launch_bounds__(CVP_THREADS, 1) conv3d16p_kernel(const __grid_constant__ CUtensorMap xmap,
                                                                  const __grid_constant__ ConvParams P,
                                                                  int ntiles)
{
  extern __shared__ __align__(1024) unsigned char smem[];
  unsigned char* A = smem;
  unsigned char* Wsm = smem + CVP_STAGES * CV_A_BYTES;
  float* bias = reinterpret_cast<float*>(Wsm + CV_W_BYTES);
  uint64_t* full = reinterpret_cast<uint64_t*>(Wsm + CV_W_BYTES + 64);
  uint64_t* empty = full + CVP_STAGES;
  uint64_t* accf = empty + CVP_STAGES;  // [2] accumulator written (MMA commit)
  uint64_t* acce = accf + 2;            // [2] accumulator read (4 epilogue warps)
  uint32_t* tslot = reinterpret_cast<uint32_t*>(acce + 2);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nmine = blockIdx.x < ntiles ? (ntiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < CVP_STAGES; s++) {
      dev::mbar_init(&full[s], 1);
      dev::mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; b++) {
      dev::mbar_init(&accf[b], 1);
      dev::mbar_init(&acce[b], 4);
    }
    dev::fence_mbar_init();
  }
  if (warp == 5) {
    tc::tmem_alloc(tslot, 32);
    tc::tmem_relinquish();
  }
  const uint4* wg = reinterpret_cast<const uint4*>(P.w);
  for (int i = threadIdx.x; i < 27 * 16 * 2; i += blockDim.x) {
    const int t = i / 32, n = (i / 2) % 16, kh = i % 2;
    reinterpret_cast<uint4*>(Wsm + t * 512 + kh * 256 + n * 16)[0] = wg[(t * 16 + n) * 2 + kh];
  }
  if (threadIdx.x < 16) bias[threadIdx.x] = P.bias ? P.bias[threadIdx.x] : 0.0f;
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t taddr = *tslot;

  if (warp == 4) {
    // ---------------------------------------------------------------- TMA producer
    if (lane == 0) {
      dev::tma_prefetch(&xmap);
      int issued = 0;
      for (int i = 0; i < nmine; i++) {
        const int s = i % CVP_STAGES;
        if (i >= CVP_STAGES && !dev::mbar_wait(&empty[s], ((i / CVP_STAGES) - 1) & 1)) {
          dev::record_status(P.status, DEV_TIMEOUT);
          break;
        }
        issued = i + 1;
        const int tile = blockIdx.x + i * gridDim.x;
        const int x0 = (tile % P.tiles_x) * CV_TILE;
        const int yz = tile / P.tiles_x;
        const int y = yz % P.ny, z = yz / P.ny;
        unsigned char* As = A + s * CV_A_BYTES;
        dev::mbar_arrive_expect_tx(&full[s], 18u * P.box_bytes);
        for (int r = 0; r < 9; r++) {
          const int dz = r / 3, dy = r % 3;
          for (int kh = 0; kh < 2; kh++)
            tc::tma_load_5d(As + (r * 2 + kh) * CV_RB, &xmap, &full[s], 0, (x0 >> P.gs) - 1,
                            kh, y + dy - 1, z + dz - 1);
        }
      }
      // no copy may still be landing in shared memory when the CTA leaves (bounded waits;
      // immediate unless another role stopped early)
      for (int j = max(0, issued - CVP_STAGES); j < issued; j++)
        dev::mbar_wait(&full[j % CVP_STAGES], (j / CVP_STAGES) & 1, 100000000ull);
    }
  } else if (warp == 5) {
    // ---------------------------------------------------------------- MMA issuer
    if (lane == 0) {
      const uint32_t wbase = dev::smem_u32(Wsm);
      constexpr uint32_t IDESC = tc::idesc_bf16(CV_TILE, 16);
      for (int i = 0; i < nmine; i++) {
        const int s = i % CVP_STAGES, b = i & 1;
        if (!dev::mbar_wait(&full[s], (i / CVP_STAGES) & 1) ||
            (i >= 2 && !dev::mbar_wait(&acce[b], ((i >> 1) - 1) & 1))) {
          dev::record_status(P.status, DEV_TIMEOUT);
          break;
        }
        tc::fence_after();
        const uint32_t abase = dev::smem_u32(A + s * CV_A_BYTES);
        for (int t = 0; t < 27; t++) {
          const int r = t / 3, dx = t % 3;
          const uint64_t ad = tc::smem_desc(abase + r * 2 * CV_RB + (dx + (1 << P.gs) - 1) * 16, CV_RB, 128);
          const uint64_t bd = tc::smem_desc(wbase + t * 512, 256, 128);
          tc::mma_bf16(taddr + (uint32_t)(b * 16), ad, bd, IDESC, t > 0 ? 1u : 0u);
        }
        tc::mma_commit(&empty[s]);
        tc::mma_commit(&accf[b]);
      }
    }
  } else {
    // ---------------------------------------------------------------- epilogue (warps 0-3)
    for (int i = 0; i < nmine; i++) {
      const int b = i & 1;
      // warp-uniform: tcgen05.ld below is a warp-collective instruction
      if (!__all_sync(0xffffffffu, dev::mbar_wait(&accf[b], (i >> 1) & 1))) {
        if (lane == 0) dev::record_status(P.status, DEV_TIMEOUT);
        break;
      }
      tc::fence_after();
      uint32_t r[16];
      tc::tmem_ld16(taddr + (uint32_t)(b * 16) + ((uint32_t)(warp * 32) << 16), r);
      tc::fence_before();
      __syncwarp();
      if (lane == 0) dev::mbar_arrive(&acce[b]);
      const int tile = blockIdx.x + i * gridDim.x;
      const int x0 = (tile % P.tiles_x) * CV_TILE;
      const int yz = tile / P.tiles_x;
      const int y = yz % P.ny, z = yz / P.ny;
      const int xv = x0 + warp * 32 + lane;
      if (xv < P.nx) {
        float v[16];
#pragma unroll
        for (int c = 0; c < 16; c++) {
          v[c] = __uint_as_float(r[c]) + bias[c];
          if (P.relu) v[c] = fmaxf(v[c], 0.0f);
        }
        const size_t i0 = tc::act_index(xv, y, z, 0, P.nx, P.ny), i1 = tc::act_index(xv, y, z, 8, P.nx, P.ny);
        if (P.out_f32) {
          float4* o0 = reinterpret_cast<float4*>(reinterpret_cast<float*>(P.out) + i0);
          float4* o1 = reinterpret_cast<float4*>(reinterpret_cast<float*>(P.out) + i1);
          o0[0] = make_float4(v[0], v[1], v[2], v[3]);
          o0[1] = make_float4(v[4], v[5], v[6], v[7]);
          o1[0] = make_float4(v[8], v[9], v[10], v[11]);
          o1[1] = make_float4(v[12], v[13], v[14], v[15]);
        } else {
          uint32_t pk[8];
#pragma unroll
          for (int q = 0; q < 8; q++) {
            __nv_bfloat162 bb = __floats2bfloat162_rn(v[2 * q], v[2 * q + 1]);
            pk[q] = *reinterpret_cast<uint32_t*>(&bb);
          }
          __nv_bfloat16* ob = reinterpret_cast<__nv_bfloat16*>(P.out);
          *reinterpret_cast<uint4*>(ob + i0) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
          *reinterpret_cast<uint4*>(ob + i1) = make_uint4(pk[4], pk[5], pk[6], pk[7]);
        }
      }
    }
  }
  // all MMAs this CTA issued must be complete before the columns are released: the
  // epilogue waited for every accumulator commit, and the issuer waits (bounded) for its last
  // one in case the epilogue stopped early
  if (warp == 5 && lane == 0 && nmine > 0) {
    const int last = nmine - 1;
    dev::mbar_wait(&accf[last & 1], (last >> 1) & 1, 100000000ull);
  }
  tc::fence_before();
  __syncthreads();
  if (warp == 5) {
    tc::fence_after();
    tc::tmem_dealloc(taddr, 32);
  }
}

// The default form.  An MMA of N = 16 reads its 4 KB of A from shared memory for 8 cycles' worth of
// arithmetic, so the kernels above are bound by operand reads and a fixed cost per MMA (27 per tile
// at about 53 cycles).  Here one MMA covers the three dz taps: an input plane contributes to the
// output planes below, at and above it, whose accumulators lie side by side in tensor memory, so one
// A row (per dy and dx) times the three taps' weights (N = 48) updates all three.
// A CTA walks up to P.zl output planes of CVN_Y rows of one x tile.  Output plane q of the walk has
// the columns of block q mod 3 of its row, so the order of the taps along N turns with the plane:
// the weights lie as dz = 2, 1, 0, 2, 1, of which each order is a window.  Input plane k updates
// planes k - 1, k, k + 1 of those the walk has and completes plane k - 1; the planes of a row are
// updated by nine MMAs in a row, and every output gathers its taps in the order dz, dy, dx of the
// kernels above: the same bits (and the same signs around zero, which a ReLU's gradient passes on).
//   warp 4 (one lane): TMA producer, the CVN_Y + 2 rows of an input plane per stage, one box;
//   warp 5 (one lane): MMA issuer; commits free the stage and hand finished rows over;
//   warps 0-3:         epilogue: read their TMEM lane quadrant of a finished row, clear it for the
//                      plane that takes its block next (accumulators start from zero), release it,
//                      then bias / ReLU / store.
// 256^3 on one B200: 0.328 ms per layer (HBM floor 0.165; the operand reads of an MMA take 44 cycles
// of shared memory, here one takes about 65).  0.646 with N = 16 and row reuse; 0.440 with N = 48
// over the dy taps of one plane, where three MMAs on one accumulator were followed by three on one
// that overlapped it (97 cycles each) and a plane was staged three times.
constexpr int CVN_Y = 5;                   // output rows of a walk
constexpr int CVN_STAGES = 3;
constexpr int CVN_THREADS = 192;
constexpr int CVN_STAGE = (CVN_Y + 2) * 2 * (CV_ROW + 2) * 16;  // [row][channel half][voxel] x 16 B
constexpr int CVN_WB = 80 * 32;            // weights of one (dy, dx): [K half][dz = 2, 1, 0, 2, 1][16 out] x 16 B
constexpr int CVN_COLS = 256;              // TMEM columns (48 a row): two CTAs per SM
constexpr int CVN_ACC = 3 * CVN_Y;         // accumulator blocks
constexpr int CVN_SMEM = CVN_STAGES * CVN_STAGE + 9 * CVN_WB + 64 + 8 * (2 * CVN_STAGES + 2 * CVN_ACC + 1) + 16;
static_assert(CVN_STAGE % 128 == 0 && 3 * CVN_SMEM > 227 * 1024 && 2 * (CVN_SMEM + 1024) <= 228 * 1024 &&
                  16 * CVN_ACC <= CVN_COLS && 2 * CVN_COLS <= 512,
              "two CTAs per SM");

// The walks of a volume: c -> x tile, rows [y0, y1), planes [z0, z1)
struct ConvChunks {
  int tiles_x, ny, nz, yl, zl, ych;
  __device__ __forceinline__ void at(int c, int& x0, int& y0, int& y1, int& z0, int& z1) const
  {
    const int yc = c % ych, col = c / ych;
    x0 = (col % tiles_x) * CV_TILE;
    y0 = yc * yl;
    y1 = min(ny, y0 + yl);
    z0 = col / tiles_x * zl;
    z1 = min(nz, z0 + zl);
  }
};

__global__ void __launch_bounds__(CVN_THREADS, 2) conv3d16n_kernel(const __grid_constant__ CUtensorMap xmap,
                                                                  const __grid_constant__ ConvParams P,
                                                                  int nchunks)
{
  extern __shared__ __align__(1024) unsigned char smem[];
  unsigned char* A = smem;
  unsigned char* Wsm = smem + CVN_STAGES * CVN_STAGE;
  float* bias = reinterpret_cast<float*>(Wsm + 9 * CVN_WB);
  uint64_t* full = reinterpret_cast<uint64_t*>(Wsm + 9 * CVN_WB + 64);
  uint64_t* empty = full + CVN_STAGES;
  uint64_t* accf = empty + CVN_STAGES;  // [CVN_ACC] row of a plane complete (MMA commit)
  uint64_t* acce = accf + CVN_ACC;      // [CVN_ACC] row read and cleared (4 epilogue warps)
  uint64_t* fin = acce + CVN_ACC;       // every MMA issued is complete, after a wait that ran out
  uint32_t* tslot = reinterpret_cast<uint32_t*>(fin + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const ConvChunks CH{P.tiles_x, P.ny, P.nz, P.yl, P.zl, (P.ny + P.yl - 1) / P.yl};

  if (threadIdx.x == 0) {
    for (int q = 0; q < CVN_STAGES; q++) {
      dev::mbar_init(&full[q], 1);
      dev::mbar_init(&empty[q], 1);
    }
    for (int q = 0; q < CVN_ACC; q++) {
      dev::mbar_init(&accf[q], 1);
      dev::mbar_init(&acce[q], 4);
    }
    dev::mbar_init(fin, 1);
    dev::fence_mbar_init();
  }
  if (warp == 5) {
    tc::tmem_alloc(tslot, CVN_COLS);
    tc::tmem_relinquish();
  }
  // weights: (dy, dx), K half kh, dz block, out channel n: 16 bytes of 8 in-channels
  const uint4* wg = reinterpret_cast<const uint4*>(P.w);
  for (int i = threadIdx.x; i < 45 * 16 * 2; i += blockDim.x) {
    const int t = i / 160, blk = i / 32 % 5, n = i / 2 % 16, kh = i % 2;
    const int dz = (5 - blk) % 3;  // 2, 1, 0, 2, 1
    reinterpret_cast<uint4*>(Wsm + t * CVN_WB + kh * (CVN_WB / 2) + (blk * 16 + n) * 16)[0] =
        wg[((dz * 9 + t) * 16 + n) * 2 + kh];
  }
  if (threadIdx.x < 16) bias[threadIdx.x] = P.bias ? P.bias[threadIdx.x] : 0.0f;
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t taddr = *tslot;
  const uint32_t lanes = (uint32_t)(warp * 32) << 16;
  if (warp < 4) {
    for (int q = 0; q < CVN_ACC; q++) tc::tmem_zero16(taddr + lanes + (uint32_t)(16 * q));
    tc::tmem_wait_st();
  }
  tc::fence_before();
  __syncthreads();
  tc::fence_after();

  if (warp == 4) {
    // ---------------------------------------------------------------- TMA producer
    if (lane == 0) {
      dev::tma_prefetch(&xmap);
      int issued = 0, s = 0;
      uint32_t ph = 0;
      bool failed = false;
      for (int c = blockIdx.x; c < nchunks && !failed; c += gridDim.x) {
        int x0, y0, y1, z0, z1;
        CH.at(c, x0, y0, y1, z0, z1);
        for (int z = z0 - 1; z <= z1; z++) {  // rows past the walk's are read, not used
          if (issued >= CVN_STAGES && !dev::mbar_wait(&empty[s], ph ^ 1u)) {
            dev::record_status(P.status, DEV_TIMEOUT);
            failed = true;
            break;
          }
          dev::mbar_arrive_expect_tx(&full[s], P.box_bytes);
          tc::tma_load_5d(A + s * CVN_STAGE, &xmap, &full[s], 0, (x0 >> P.gs) - 1, 0, y0 - 1, z);
          issued++;
          if (++s == CVN_STAGES) { s = 0; ph ^= 1u; }
        }
      }
      // no copy may still be landing in shared memory when the CTA leaves (bounded waits)
      for (int j = max(0, issued - CVN_STAGES); j < issued; j++)
        dev::mbar_wait(&full[j % CVN_STAGES], (j / CVN_STAGES) & 1, 100000000ull);
    }
  } else if (warp == 5) {
    // ---------------------------------------------------------------- MMA issuer
    if (lane == 0) {
      const uint32_t wbase = dev::smem_u32(Wsm), abase = dev::smem_u32(A);
      int s = 0;
      uint32_t ph = 0;
      uint32_t used = 0;  // bit q: parity of the uses of accumulator block q so far
      int stages = 0;     // stages issued
      const uint32_t half = P.box_bytes / (2 * (CVN_Y + 2));  // one channel half of one staged row
      bool failed = false;
      for (int c = blockIdx.x; c < nchunks && !failed; c += gridDim.x) {
        int x0, y0, y1, z0, z1;
        CH.at(c, x0, y0, y1, z0, z1);
        const int n = y1 - y0, len = z1 - z0;
        int b1 = 0;  // block of plane k + 1
        for (int k = -1; k <= len; k++) {
          bool ok = dev::mbar_wait(&full[s], ph);
          const int b0 = b1 == 0 ? 2 : b1 - 1, bm = b1 == 2 ? 0 : b1 + 1;  // of planes k, k - 1
          tc::fence_after();
          for (int p = 0; ok && p < n; p++) {
            if (k + 1 < len) {  // plane k + 1 joins: the block's previous plane must have been read and cleared
              const int q = 3 * p + b1;
              ok = dev::mbar_wait(&acce[q], ((used >> q) & 1u) ^ 1u);
              if (!ok) break;
              used ^= 1u << q;
              tc::fence_after();
            }
            const uint32_t d = taddr + (uint32_t)(48 * p);
            const uint32_t a0 = abase + s * CVN_STAGE + p * 2 * half + ((1 << P.gs) - 1) * 16;
            // blocks [col, col + count), weights from block `win` of 2, 1, 0, 2, 1
            auto mmas = [&](int col, int count, int win) {
              const uint32_t idesc = tc::idesc_bf16(CV_TILE, 16 * count);
              const uint32_t w0 = wbase + win * 256;
#pragma unroll
              for (int t = 0; t < 9; t++)
                tc::mma_bf16(d + 16 * col, tc::smem_desc(a0 + (t / 3) * 2 * half + (t % 3) * 16, half, 128),
                             tc::smem_desc(w0 + t * CVN_WB, CVN_WB / 2, 128), idesc, 1u);
            };
            const bool vm = k >= 1, v0 = k >= 0 && k < len, v1 = k + 1 < len;  // planes k - 1, k, k + 1 of the walk
            if (vm && v0 && v1) mmas(0, 3, bm == 0 ? 0 : bm == 1 ? 2 : 1);
            else if (v0 && v1 && b0 < b1) mmas(b0, 2, 1);
            else if (vm && v0 && bm < b0) mmas(bm, 2, 0);
            else {
              if (vm) mmas(bm, 1, 0);
              if (v0) mmas(b0, 1, 1);
              if (v1) mmas(b1, 1, 2);
            }
            if (vm) tc::mma_commit(&accf[3 * p + bm]);
          }
          if (!ok) {
            dev::record_status(P.status, DEV_TIMEOUT);
            failed = true;
            break;
          }
          b1 = b1 == 2 ? 0 : b1 + 1;
          tc::mma_commit(&empty[s]);
          stages++;
          if (++s == CVN_STAGES) { s = 0; ph ^= 1u; }
        }
      }
      // every MMA issued must be complete before the columns are released: the last stage's commit, or,
      // where a plane was given up halfway, one behind them all
      if (failed) {
        tc::mma_commit(fin);
        dev::mbar_wait(fin, 0, 100000000ull);
      } else if (stages > 0) {
        dev::mbar_wait(&empty[(stages - 1) % CVN_STAGES], ((stages - 1) / CVN_STAGES) & 1, 100000000ull);
      }
    }
  } else {
    // ---------------------------------------------------------------- epilogue (warps 0-3)
    uint32_t used = 0;
    bool failed = false;
    for (int c = blockIdx.x; c < nchunks && !failed; c += gridDim.x) {
      int x0, y0, y1, z0, z1;
      CH.at(c, x0, y0, y1, z0, z1);
      const int n = y1 - y0;
      const int xv = x0 + warp * 32 + lane;
      for (int i = 0; i < n * (z1 - z0); i++) {
        const int k = i / n, p = i - k * n, z = z0 + k, q = 3 * p + k % 3;
        // warp-uniform: the tcgen05 instructions below are warp-collective
        if (!__all_sync(0xffffffffu, dev::mbar_wait(&accf[q], (used >> q) & 1u))) {
          if (lane == 0) dev::record_status(P.status, DEV_TIMEOUT);
          failed = true;
          break;
        }
        used ^= 1u << q;
        tc::fence_after();
        uint32_t r[16];
        tc::tmem_ld16(taddr + lanes + (uint32_t)(16 * q), r);
        tc::tmem_zero16(taddr + lanes + (uint32_t)(16 * q));
        tc::tmem_wait_st();
        tc::fence_before();
        __syncwarp();
        if (lane == 0) dev::mbar_arrive(&acce[q]);
        if (xv < P.nx) {
          const int y = y0 + p;
          float v[16];
#pragma unroll
          for (int q = 0; q < 16; q++) {
            v[q] = __uint_as_float(r[q]) + bias[q];
            if (P.relu) v[q] = fmaxf(v[q], 0.0f);
          }
          const size_t i0 = tc::act_index(xv, y, z, 0, P.nx, P.ny), i1 = tc::act_index(xv, y, z, 8, P.nx, P.ny);
          if (P.out_f32) {
            float4* o0 = reinterpret_cast<float4*>(reinterpret_cast<float*>(P.out) + i0);
            float4* o1 = reinterpret_cast<float4*>(reinterpret_cast<float*>(P.out) + i1);
            o0[0] = make_float4(v[0], v[1], v[2], v[3]);
            o0[1] = make_float4(v[4], v[5], v[6], v[7]);
            o1[0] = make_float4(v[8], v[9], v[10], v[11]);
            o1[1] = make_float4(v[12], v[13], v[14], v[15]);
          } else {
            uint32_t pk[8];
#pragma unroll
            for (int q = 0; q < 8; q++) {
              __nv_bfloat162 bb = __floats2bfloat162_rn(v[2 * q], v[2 * q + 1]);
              pk[q] = *reinterpret_cast<uint32_t*>(&bb);
            }
            __nv_bfloat16* ob = reinterpret_cast<__nv_bfloat16*>(P.out);
            *reinterpret_cast<uint4*>(ob + i0) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
            *reinterpret_cast<uint4*>(ob + i1) = make_uint4(pk[4], pk[5], pk[6], pk[7]);
          }
        }
      }
    }
  }
  tc::fence_before();
  __syncthreads();
  if (warp == 5) {
    tc::fence_after();
    tc::tmem_dealloc(taddr, CVN_COLS);
  }
}

// Weight gradient on the CUDA cores: dW[t][co][ci] += sum_v dY[v][co] * X[v + off(t)][ci].
// Thread (co, ci) slides along a row of 128 voxels keeping the three x-neighbours of each of
// the 9 tap rows in registers; CTAs loop over tiles and add their 27 partial sums once.
struct WgradParams {
  const __nv_bfloat16* x;
  const void* dy;
  int dy_f32;
  float* dw;
  int nx, ny, nz, tiles_x, ntiles;
};

__device__ __forceinline__ float ld_act(const __nv_bfloat16* p) { return __bfloat162float(*p); }

constexpr int WG_TILE = 64;
__global__ void __launch_bounds__(256) conv3d16_wgrad_kernel(const WgradParams P)
{
  __shared__ float xs[9][WG_TILE + 2][17];
  __shared__ float ds[WG_TILE][17];
  const int co = threadIdx.x >> 4, ci = threadIdx.x & 15;
  float acc[27];
#pragma unroll
  for (int t = 0; t < 27; t++) acc[t] = 0.0f;
  for (int tile = blockIdx.x; tile < P.ntiles; tile += gridDim.x) {
    const int x0 = (tile % P.tiles_x) * WG_TILE;
    const int yz = tile / P.tiles_x;
    const int y = yz % P.ny, z = yz / P.ny;
    __syncthreads();
    for (int i = threadIdx.x; i < 9 * (WG_TILE + 2) * 16; i += blockDim.x) {
      const int c = i & 15, xr = (i >> 4) % (WG_TILE + 2), r = i / (16 * (WG_TILE + 2));
      const int zz = z + r / 3 - 1, yy = y + r % 3 - 1, xx = x0 + xr - 1;
      float v = 0.0f;
      if (zz >= 0 && zz < P.nz && yy >= 0 && yy < P.ny && xx >= 0 && xx < P.nx)
        v = ld_act(P.x + tc::act_index(xx, yy, zz, c, P.nx, P.ny));
      xs[r][xr][c] = v;
    }
    for (int i = threadIdx.x; i < WG_TILE * 16; i += blockDim.x) {
      const int c = i & 15, xr = i >> 4, xx = x0 + xr;
      float v = 0.0f;
      if (xx < P.nx) {
        const size_t o = tc::act_index(xx, y, z, c, P.nx, P.ny);
        v = P.dy_f32 ? reinterpret_cast<const float*>(P.dy)[o]
                     : ld_act(reinterpret_cast<const __nv_bfloat16*>(P.dy) + o);
      }
      ds[xr][c] = v;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < 9; r++) {
      float a = xs[r][0][ci], b = xs[r][1][ci];
      for (int v = 0; v < WG_TILE; v++) {
        const float c = xs[r][v + 2][ci];
        const float g = ds[v][co];
        acc[r * 3 + 0] = fmaf(g, a, acc[r * 3 + 0]);
        acc[r * 3 + 1] = fmaf(g, b, acc[r * 3 + 1]);
        acc[r * 3 + 2] = fmaf(g, c, acc[r * 3 + 2]);
        a = b;
        b = c;
      }
    }
  }
#pragma unroll
  for (int t = 0; t < 27; t++) atomicAdd(P.dw + (t * 16 + co) * 16 + ci, acc[t]);
}

// Weight gradient on the tensor cores (BF16 dY).  dW[t][co][ci] = sum over voxels v of
// dY[v][co] X[v + off(t)][ci] is a GEMM whose reduction dimension K is the voxels, 16 per
// MMA.  For one input row r = (dz, dy) and u = the X voxels x0-1 .. x0+142 of a 128-voxel
// tile (9 K-steps of 16):
//   D_r[s*16 + co][ci] = sum_u A[s*16 + co][u] * X_r[u][ci],   A[s*16 + co][u] = dY[u + 1 - s][co]
// with dY taken as zero outside the tile: rows s = 0, 1, 2 of D_r are the taps dx = s of row
// r (v = u + 1 - s runs over the tile).  The nine rows (dy, dz) lie one after the other in
// shared memory, so one MMA per K-step covers them: M = 128 (rows 0-47 used), N = 144
// (dy, dz, ci), K = 16 -- 9 MMAs per tile give all 27 taps.  A lives in tensor memory: writer
// warps put the three shifted copies of the tile's dY there, transposed on the way by ldmatrix
// (dy_step); B is the staged X rows, MN-major straight from the activation layout (8 channels
// of one voxel = one 16-byte core-matrix row).  TMEM: the accumulators' 144 columns + WGT_ABUF
// A buffers of 72.
// A CTA walks chunks of WGT_YCH consecutive y rows of one (x tile, z) column; each tile loads
// its new X row (three planes, two halves: one box) into a ring of WGT_RING positions that runs
// on from chunk to chunk, positions 0 and 1 also into WGT_RING and WGT_RING + 1, so that rows
// y-1, y, y+1 always occupy three consecutive slots (a uniform N stride for B); dY rows are
// staged WGT_LEAD deep;
//   warp 2 (one lane):  TMA producer, up to WGT_LEAD tiles ahead of the MMAs;
//   warps 0-1 and 4-5:  A writers, tiles in turn; then warps 0-1 the epilogue: TMEM lanes 0-47
//                       of the accumulators -> dW (FP32 atomics, once per CTA);
//   warp 3 (one lane):  MMA issuer, commits to the tile's done barrier.
// Dynamic shared memory above half an SM's keeps one CTA per SM (512-column allocation).
//
// 256^3 on one B200: 0.468 ms, the tensor pipe 70 % active (an MMA of N = 144 takes its 72 cycles;
// 80 of the 128 rows are idle).  Before, 1.08 ms: an MMA per dz took 84 cycles at N = 48 (one per
// K-step: 0.83), one pair of writer warps gathered dY by 16-bit loads (three pairs: 0.56;
// ldmatrix: 0.47; ldmatrix and one pair 0.63), and every chunk began with an empty ring (0.56 to
// 0.535).
constexpr int WGT_GROUPS = 2;                        // pairs of A writer warps: 0-1, 4-5
constexpr int WGT_THREADS = 192;
constexpr int WGT_YCH = 32;                          // rows per chunk
constexpr int WGT_KSTEPS = 9;                        // 144 voxels u per tile
constexpr int WGT_XROW = 152;                        // staged X voxels per row (from x0 - group)
constexpr int WGT_RB = WGT_XROW * 16;                // one channel half of a staged X row
constexpr int WGT_XSLOT = 6 * WGT_RB;                // the row's three planes and two halves: one TMA box
static_assert((WGT_KSTEPS * 16 + 7) * 16 <= WGT_RB && WGT_XROW % 8 == 0 && WGT_XSLOT % 128 == 0, "X row slot");
constexpr int WGT_DY_BYTES = 2048;                   // one channel half of 128 dY voxels (TMA box)
constexpr int WGT_DYH = 2432;                        // its slot: 8 zero voxels, the box, 16 zero voxels
// Pipeline depth: X rows in a ring of WGT_RING positions, so the producer runs up to
// WGT_LEAD = WGT_RING - 2 tiles ahead of the MMAs; as many dY stages; WGT_ABUF A buffers.
constexpr int WGT_RING = 8;
constexpr int WGT_LEAD = WGT_RING - 2;
constexpr int WGT_ABUF = 5;
constexpr int WGT_DY = WGT_LEAD * 2 * WGT_DYH;       // dY stages x 2 halves
constexpr int WGT_XPOS = WGT_RING + 2;               // ring positions + the two duplicates
constexpr int WGT_X = WGT_XPOS * WGT_XSLOT;          // X row ring
constexpr int WGT_BAR = WGT_DY + WGT_X;
constexpr int WGT_NBAR = 2 * WGT_RING + WGT_ABUF + 1;
constexpr int WGT_SMEM_USED = WGT_BAR + 8 * WGT_NBAR + 16;
static_assert(WGT_DYH >= (8 + CV_TILE + 16) * 16 && WGT_DYH % 128 == 0 && WGT_DY % 128 == 0, "dY slots");
constexpr int WGT_SMEM = 200 * 1024;                 // > half an SM: one CTA per SM
static_assert(WGT_SMEM_USED <= WGT_SMEM, "wgrad shared memory");
constexpr uint32_t WGT_ACOL = 144;                   // first A column (after the accumulators)
constexpr uint32_t WGT_ACOLS = WGT_KSTEPS * 8;       // 72 columns per A buffer
static_assert(WGT_ACOL + WGT_ABUF * WGT_ACOLS <= 512, "TMEM columns");

struct WgradTcParams {
  float* dw;
  int nx, ny, nz, tiles_x;
  int gs;  // log2 of the voxels per box row
  int* status;
};

namespace tc {
// D(tmem) (+)= A(tmem) * B(smem desc), BF16 inputs, FP32 accumulator.
__device__ __forceinline__ void mma_bf16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc,
                                            uint32_t accumulate)
{
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.u32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(tmem_d),
      "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// One K-step of one shift: 16 voxels x 16 channels of staged dY (16 bytes per voxel and channel
// half) into 16 TMEM lanes (channels) x 8 columns (voxel pairs).  ldmatrix transposes: thread t
// gets channel t / 4 and voxel pair t % 4 of each 8 x 8 matrix, as the 16x128b store wants them
// (registers: lanes 0-7 and 8-15 of columns 0-3, then of 4-7).
__device__ __forceinline__ void dy_step(uint32_t taddr, uint32_t row)
{
  uint32_t r0, r1, r2, r3;
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(row) : "memory");
  asm volatile("tcgen05.st.sync.aligned.16x128b.x2.b32 [%0], {%1,%2,%3,%4};" ::"r"(taddr), "r"(r0), "r"(r1), "r"(r2),
               "r"(r3)
               : "memory");
}
}  // namespace tc

__global__ void __launch_bounds__(WGT_THREADS, 1) conv3d16_wgrad_tc_kernel(const __grid_constant__ CUtensorMap xmap,
                                                                         const __grid_constant__ CUtensorMap dymap,
                                                                         const __grid_constant__ WgradTcParams P,
                                                                         int nchunks)
{
  extern __shared__ __align__(1024) unsigned char smem[];
  unsigned char* DY = smem;
  unsigned char* X = smem + WGT_DY;
  uint64_t* rows_full = reinterpret_cast<uint64_t*>(smem + WGT_BAR);  // [WGT_RING] per tile
  uint64_t* tile_done = rows_full + WGT_RING;                           // [WGT_RING] per tile
  uint64_t* a_full = tile_done + WGT_RING;                              // [WGT_ABUF] A buffer written
  uint64_t* fin = a_full + WGT_ABUF;                                    // every MMA of the CTA done
  uint32_t* tslot = reinterpret_cast<uint32_t*>(fin + 1);
  volatile int* failed_flag = reinterpret_cast<volatile int*>(tslot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ych = (P.ny + WGT_YCH - 1) / WGT_YCH;

  if (threadIdx.x == 0) {
    for (int q = 0; q < WGT_RING; q++) {
      dev::mbar_init(&rows_full[q], 1);
      dev::mbar_init(&tile_done[q], 1);
    }
    for (int b = 0; b < WGT_ABUF; b++) dev::mbar_init(&a_full[b], 2);
    dev::mbar_init(fin, 1);
    *failed_flag = 0;
    dev::fence_mbar_init();
  }
  // the dY slots' margins (voxels x0-8 .. x0-1 and x0+128 .. x0+143) stay zero: dY outside
  // the tile, which the shifted copies must not see
  for (int q = threadIdx.x; q < 2 * WGT_LEAD * 24; q += blockDim.x) {
    const int slot = q / 24, v = q % 24;
    reinterpret_cast<uint4*>(DY + slot * WGT_DYH)[v < 8 ? v : 128 + v] = make_uint4(0, 0, 0, 0);
  }
  if (warp == 3) {
    tc::tmem_alloc(tslot, 512);
    tc::tmem_relinquish();
  }
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t taddr = *tslot;

  auto chunk_of = [&](int c, int& x0, int& z, int& y0, int& y1) {
    const int yc = c % ych, col = c / ych;
    x0 = (col % P.tiles_x) * CV_TILE;
    z = col / P.tiles_x;
    y0 = yc * WGT_YCH;
    y1 = min(P.ny, y0 + WGT_YCH);
  };
  int last = -1;  // tiles this CTA handles, minus one
  for (int c = blockIdx.x; c < nchunks; c += gridDim.x) {
    int x0, z, y0, y1;
    chunk_of(c, x0, z, y0, y1);
    last += y1 - y0;
  }

  if (warp == 2) {
    // ---------------------------------------------------------------- TMA producer
    if (lane == 0) {
      dev::tma_prefetch(&xmap);
      dev::tma_prefetch(&dymap);
      int i = 0, issued = 0, n = 0;    // tiles; rows staged
      int pn = -WGT_RING, pi = 0;      // the previous chunk's first row and tile
      bool failed = false;
      for (int c = blockIdx.x; c < nchunks && !failed; c += gridDim.x) {
        int x0, z, y0, y1;
        chunk_of(c, x0, z, y0, y1);
        const int cn = n, ci = i;  // this chunk's
        for (int y = y0; y < y1; y++, i++) {
          const int r0 = y == y0 ? -1 : 1;  // new rows y + r0 .. y + 1
          // The row that the last new one replaces was read last by the tile it is the first row
          // of, or by its chunk's last tile; the dY stage by the A writers of tile i - WGT_LEAD,
          // which finished before its MMAs.
          const int old = n + (1 - r0) - WGT_RING;
          const int reader = old >= cn ? ci + old - cn : old >= pn ? min(pi + old - pn, ci - 1) : pi - 1;
          const int wt = max(reader, i - WGT_LEAD);
          if (wt >= 0 && !dev::mbar_wait(&tile_done[wt % WGT_RING], (wt / WGT_RING) & 1)) {
            dev::record_status(P.status, DEV_TIMEOUT);
            *failed_flag = 1;
            failed = true;
            break;
          }
          int ncopies = 0;
          for (int dy = r0; dy <= 1; dy++) ncopies += ((n + dy - r0) & (WGT_RING - 1)) < 2 ? 2 : 1;
          uint64_t* full = &rows_full[i % WGT_RING];
          dev::mbar_arrive_expect_tx(full, (uint32_t)ncopies * WGT_XSLOT + 2u * WGT_DY_BYTES);
          for (int dy = r0; dy <= 1; dy++, n++) {
            const int pos = n & (WGT_RING - 1);
            for (int dup = 0; dup < (pos < 2 ? 2 : 1); dup++)
              tc::tma_load_5d(X + (pos + dup * WGT_RING) * WGT_XSLOT, &xmap, full, 0, (x0 >> P.gs) - 1,
                              0, y + dy, z - 1);
          }
          unsigned char* dst = DY + (i % WGT_LEAD) * 2 * WGT_DYH + 128;  // after the 8 zero voxels
          for (int kh = 0; kh < 2; kh++)
            tc::tma_load_5d(dst + kh * WGT_DYH, &dymap, full, 0, x0 >> P.gs, kh, y, z);
          issued = i + 1;
        }
        pn = cn;
        pi = ci;
      }
      for (int j = max(0, issued - WGT_RING); j < issued; j++)
        dev::mbar_wait(&rows_full[j % WGT_RING], (j / WGT_RING) & 1, 100000000ull);
    }
  } else if (warp == 3) {
    // ---------------------------------------------------------------- MMA issuer
    if (lane == 0) {
      const uint32_t xbase = dev::smem_u32(X);
      // M = 128 (rows 0-47 used), N = 144, A K-major in TMEM, B MN-major in shared memory
      constexpr uint32_t IDESC = tc::idesc_bf16(CV_TILE, 144) | (1u << 16);
      int i = 0, n = 0;
      bool failed = false;
      for (int c = blockIdx.x; c < nchunks && !failed; c += gridDim.x) {
        int x0, z, y0, y1;
        chunk_of(c, x0, z, y0, y1);
        for (int y = y0; y < y1; y++, i++, n++) {
          if (!dev::mbar_wait(&rows_full[i % WGT_RING], (i / WGT_RING) & 1) ||
              !dev::mbar_wait(&a_full[i % WGT_ABUF], (i / WGT_ABUF) & 1)) {
            dev::record_status(P.status, DEV_TIMEOUT);
            *failed_flag = 1;
            failed = true;
            break;
          }
          tc::fence_after();
          // MN-major B over the slots of rows y-1, y, y+1, three planes each: N core matrices (dy, dz, ci
          // half) every WGT_RB bytes (SBO), K core matrices of 8 voxels every 128 bytes (LBO);
          // a K-step of 16 voxels moves the start address by 256 B (16 in the descriptor's
          // address field, which stays below 2^14 inside shared memory)
          const uint64_t bd = tc::smem_desc(xbase + (n & (WGT_RING - 1)) * WGT_XSLOT + ((1 << P.gs) - 1) * 16, 128, WGT_RB);
          const uint32_t aaddr = taddr + WGT_ACOL + (uint32_t)(i % WGT_ABUF) * WGT_ACOLS;
          for (int ks = 0; ks < WGT_KSTEPS; ks++)
            tc::mma_bf16_ts(taddr, aaddr + (uint32_t)(ks * 8), bd + (uint64_t)(ks * 16), IDESC, i > 0 || ks > 0);
          tc::mma_commit(&tile_done[i % WGT_RING]);
        }
        n += 2;  // the chunk's last two rows
      }
      // one phase that completes when every MMA issued here has (or at once if none was)
      if (i > 0) tc::mma_commit(fin);
      else dev::mbar_arrive(fin);
    }
  } else if ((warp & 3) < 2) {
    // ---------------------------------------------------------------- A writers (warps 0-1 and 4-5)
    const int group = warp >> 2;
    const int s0 = 2 * (warp & 1);  // first of the shifts s = 0, 1 or s = 2 (TMEM lanes 16 s + co)
    const uint32_t lane_base = (uint32_t)(16 * s0) << 16;
    // this lane's row of the four 8 x 8 matrices (voxel half, channel half) of a K-step
    const uint32_t row = dev::smem_u32(DY) + (lane >> 3 & 1) * WGT_DYH + (8 + (lane >> 4) * 8 + (lane & 7)) * 16;
    int i = 0;
    bool failed = false;
    for (int c = blockIdx.x; c < nchunks && !failed; c += gridDim.x) {
      int x0, z, y0, y1;
      chunk_of(c, x0, z, y0, y1);
      for (int y = y0; y < y1; y++, i++) {
        if (i % WGT_GROUPS != group) continue;
        // the dY row of tile i is staged, and the A buffer's previous readers (the MMAs of
        // tile i - WGT_ABUF) are done
        bool ok = dev::mbar_wait(&rows_full[i % WGT_RING], (i / WGT_RING) & 1);
        const int pt = i - WGT_ABUF;
        if (ok && pt >= 0) ok = dev::mbar_wait(&tile_done[pt % WGT_RING], (pt / WGT_RING) & 1);
        if (!__all_sync(0xffffffffu, ok)) {
          if (lane == 0) {
            dev::record_status(P.status, DEV_TIMEOUT);
            *failed_flag = 1;
          }
          failed = true;
          break;
        }
        tc::fence_after();
        // A[u] = dY[x0 + rel], rel = 16 ks + k - s: slot voxel rel + 8 (zero outside the tile)
        const uint32_t src = row + (uint32_t)(i % WGT_LEAD) * 2 * WGT_DYH;
        const uint32_t dst = taddr + lane_base + WGT_ACOL + (uint32_t)(i % WGT_ABUF) * WGT_ACOLS;
#pragma unroll
        for (int ks = 0; ks < WGT_KSTEPS; ks++) {
          tc::dy_step(dst + (uint32_t)(ks * 8), src + (uint32_t)(ks * 256 - s0 * 16));
          if (s0 == 0) tc::dy_step(dst + (16u << 16) + (uint32_t)(ks * 8), src + (uint32_t)(ks * 256 - 16));
        }
        tc::tmem_wait_st();
        tc::fence_before();
        __syncwarp();
        if (lane == 0) dev::mbar_arrive(&a_full[i % WGT_ABUF]);
      }
    }
    // ---------------------------------------------------------------- epilogue
    if (last >= 0 && group == 0) {
      const int s = 2 * warp + (lane >> 4), co = lane & 15;
      const bool done = __all_sync(0xffffffffu, dev::mbar_wait(fin, 0)) != 0;
      tc::fence_after();
      if (done && !*failed_flag) {
        for (int r = 0; r < 9; r++) {
          uint32_t v[16];
          tc::tmem_ld16(taddr + ((uint32_t)(warp * 32) << 16) + (uint32_t)(r * 16), v);
          if (s < 3) {
            float* d = P.dw + (((r % 3 * 3 + r / 3) * 3 + s) * 16 + co) * 16;  // columns (dy, dz), taps (dz, dy, dx)
#pragma unroll
            for (int q = 0; q < 16; q++) atomicAdd(d + q, __uint_as_float(v[q]));
          }
        }
      } else if (!done && lane == 0) {
        dev::record_status(P.status, DEV_TIMEOUT);
      }
    }
  }
  // every MMA issued must be complete before the columns are released
  if (warp == 3 && lane == 0 && last >= 0) dev::mbar_wait(fin, 0, 100000000ull);
  tc::fence_before();
  __syncthreads();
  if (warp == 3) {
    tc::fence_after();
    tc::tmem_dealloc(taddr, 512);
  }
}

// =====================================================================================
// The incoming gradient of a layer
// =====================================================================================
// gb = BF16(gy * (y > 0)) (gy itself without `y`) and the per-channel sums of those products in
// FP32, in one pass: what the input and weight gradients read, and the bias gradient.  Separate
// element-wise passes in FP32 moved six times the bytes (and took 2.2 ms more of a 256^3 layer's
// forward and backward); the bound is HBM.  Block b sums the channels of half b mod 2; the blocks' sums are added in block
// order in FP64, so the result does not depend on timing.
constexpr int CGP_BLOCKS = 148 * 8, CGP_THREADS = 256;
template <bool F32, bool MASK>
__global__ void __launch_bounds__(CGP_THREADS) conv_grad_prep_kernel(const void* __restrict__ gy,
                                                                     const uint4* __restrict__ y,
                                                                     uint4* __restrict__ gb,
                                                                     float* __restrict__ part, int nx,
                                                                     unsigned groups)
{
  const int half = blockIdx.x & 1;
  float acc[8];
#pragma unroll
  for (int c = 0; c < 8; c++) acc[c] = 0.0f;
  // groups of 8 channels of one half: voxel j -> row j / nx (rows of the halves alternate)
  for (unsigned j = (blockIdx.x >> 1) * CGP_THREADS + threadIdx.x; j < groups; j += (CGP_BLOCKS / 2) * CGP_THREADS) {
    const unsigned row = j / (unsigned)nx;
    const size_t o = ((size_t)row * 2 + half) * nx + (j - row * nx);
    float g[8];
    if constexpr (F32) {
      const float4 a = reinterpret_cast<const float4*>(gy)[2 * o], b = reinterpret_cast<const float4*>(gy)[2 * o + 1];
      g[0] = a.x; g[1] = a.y; g[2] = a.z; g[3] = a.w;
      g[4] = b.x; g[5] = b.y; g[6] = b.z; g[7] = b.w;
    } else {
      const uint4 a = reinterpret_cast<const uint4*>(gy)[o];
      const uint32_t w[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
      for (int q = 0; q < 4; q++) {
        g[2 * q] = __uint_as_float(w[q] << 16);
        g[2 * q + 1] = __uint_as_float(w[q] & 0xffff0000u);
      }
    }
    if constexpr (MASK) {
      const uint4 a = y[o];
      const uint32_t w[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
      for (int q = 0; q < 4; q++) {  // a product, not a select: what is not finite stays so
        g[2 * q] *= __uint_as_float(w[q] << 16) > 0.0f ? 1.0f : 0.0f;
        g[2 * q + 1] *= __uint_as_float(w[q] & 0xffff0000u) > 0.0f ? 1.0f : 0.0f;
      }
    }
    uint32_t pk[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const __nv_bfloat162 b = __floats2bfloat162_rn(g[2 * q], g[2 * q + 1]);
      pk[q] = *reinterpret_cast<const uint32_t*>(&b);
    }
    gb[o] = make_uint4(pk[0], pk[1], pk[2], pk[3]);
#pragma unroll
    for (int c = 0; c < 8; c++) acc[c] += g[c];
  }
  __shared__ float sums[CGP_THREADS / 32][8];
#pragma unroll
  for (int c = 0; c < 8; c++) {
    for (int o = 16; o > 0; o >>= 1) acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], o);
    if ((threadIdx.x & 31) == 0) sums[threadIdx.x >> 5][c] = acc[c];
  }
  __syncthreads();
  if (threadIdx.x < 8) {
    float v = 0.0f;
    for (int w = 0; w < CGP_THREADS / 32; w++) v += sums[w][threadIdx.x];
    part[blockIdx.x * 8 + threadIdx.x] = v;
  }
}

// db[c] = the blocks' sums of channel c; warp c of one block
__global__ void conv_bias_sum_kernel(const float* __restrict__ part, float* __restrict__ db)
{
  const int c = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double v = 0.0;
  for (int b = (c >> 3) + 2 * lane; b < CGP_BLOCKS; b += 64) v += (double)part[b * 8 + (c & 7)];
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if (lane == 0) db[c] = (float)v;
}

}  // namespace fcb

using namespace fcb;

extern "C" int fcb_conv3d16_grad_prep_device(const void* gy, int gyType, const void* y, void* gb, float* db,
                                             float* scratch, int nx, int ny, int nz, void* stream)
try {
  if (!gy || !gb || !db || !scratch || nx <= 0 || ny <= 0 || nz <= 0 || (gyType != FCB_F32 && gyType != FCB_BF16))
    return set_error(FCB_ERR_INVALID, "bad conv3d gradient arguments");
  if (((uintptr_t)gy & 15) || ((uintptr_t)y & 15) || ((uintptr_t)gb & 15))
    return set_error(FCB_ERR_INVALID, "conv3d buffers must be 16-byte aligned");
  const long long groups = (long long)nx * ny * nz;
  if (groups > 0x7fffffffll) return set_error(FCB_ERR_RANGE, "conv3d volume too large");
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  auto kern = gyType == FCB_F32 ? (y ? conv_grad_prep_kernel<true, true> : conv_grad_prep_kernel<true, false>)
                                : (y ? conv_grad_prep_kernel<false, true> : conv_grad_prep_kernel<false, false>);
  kern<<<CGP_BLOCKS, CGP_THREADS, 0, st>>>(gy, reinterpret_cast<const uint4*>(y), reinterpret_cast<uint4*>(gb), scratch,
                                           nx, (unsigned)groups);
  conv_bias_sum_kernel<<<1, 512, 0, st>>>(scratch, db);
  FCB_CUDA_TRY(cudaGetLastError());
  return ok();
}
FCB_CATCH_STATUS

static_assert(CGP_BLOCKS * 8 == FCB_CONV_GRAD_SCRATCH, "gradient scratch");

// log2 of the voxels per TMA box row.  Activations are [z][y][2][x][8], a row of one channel half
// contiguous, read as dims (channels of 2^gs voxels, x >> gs, half, y, z): the copy engine takes a
// box row at a time, and rows of 16 bytes fetch every sector twice.  A tile's box starts one group
// before its first voxel, its operands 2^gs - 1 voxels into the box, so gs <= `most` must divide nx.
// The weight gradient takes groups of up to 8 (256^3: 0.468 ms, with pairs 0.49); the forward
// kernel, not bound by its copies, pairs, whose margins fit its stages (groups of 8 made no difference
// to the kernel before it, which staged three rows of one plane: 0.444 ms against 0.440).
static int box_group(int nx, int most)
{
  int gs = most;
  while (nx & ((1 << gs) - 1)) gs--;
  return gs;
}

extern "C" int fcb_conv3d16_device(const void* x, const void* w, const float* bias, void* y, int yType,
                                   int nx, int ny, int nz, int relu, void* stream)
try {
  if (!x || !w || !y || nx <= 0 || ny <= 0 || nz <= 0 || (yType != FCB_F32 && yType != FCB_BF16))
    return set_error(FCB_ERR_INVALID, "bad conv3d arguments");
  if (((uintptr_t)x & 15) || ((uintptr_t)w & 15) || ((uintptr_t)y & 15))
    return set_error(FCB_ERR_INVALID, "conv3d buffers must be 16-byte aligned");
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  CUtensorMap map;
  // FCB_CONV_SIMPLE=1: one CTA per tile; FCB_CONV_SIMPLE=2: persistent without row reuse (both for
  // comparison, one channel half of one row per box); default: three dz taps per MMA
  const char* env = getenv("FCB_CONV_SIMPLE");
  const int variant = env ? atoi(env) : 0;
  const bool simple = variant == 1 || variant == 2;
  const int gs = box_group(nx, 1), group = 1 << gs;
  const uint64_t dims[5] = {8ull * group, (uint64_t)(nx / group), 2, (uint64_t)ny, (uint64_t)nz};
  const uint64_t strides[4] = {16ull * group, 16ull * nx, 32ull * nx, 32ull * nx * ny};
  const uint32_t box[5] = {8u * group, (uint32_t)((CV_ROW + 2 * group - 2) / group), simple ? 1u : 2u,
                           simple ? 1u : (uint32_t)(CVN_Y + 2), 1};
  FCB_TRY(encode_tmap(&map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<void*>(x), dims, strides, box));
  int* status = nullptr;
  FCB_TRY(device_status_ptr(&status));
  ConvParams P;
  P.gs = gs;
  P.box_bytes = box[0] * box[1] * box[2] * box[3] * 2;
  P.w = reinterpret_cast<const __nv_bfloat16*>(w);
  P.bias = bias;
  P.out = y;
  P.out_f32 = yType == FCB_F32;
  P.relu = relu;
  P.nx = nx; P.ny = ny; P.nz = nz;
  P.tiles_x = (nx + CV_TILE - 1) / CV_TILE;
  P.status = status;
  const long long tiles = (long long)P.tiles_x * ny * nz;
  if (tiles > 0x7fffffffll) return set_error(FCB_ERR_RANGE, "conv3d volume too large");
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (variant == 1) {
    FCB_CUDA_TRY(cudaFuncSetAttribute(conv3d16_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, CV_SMEM));
    conv3d16_kernel<<<(unsigned)tiles, 128, CV_SMEM, st>>>(map, P);
  } else if (variant == 2) {
    FCB_CUDA_TRY(cudaFuncSetAttribute(conv3d16p_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, CVP_SMEM));
    const int grid = (int)std::min<long long>(tiles, sms);
    conv3d16p_kernel<<<grid, CVP_THREADS, CVP_SMEM, st>>>(map, P, (int)tiles);
  } else {
    // Rows and planes per walk: those with the least work on the busiest CTA, (planes + 2) passes over
    // the rows per walk and about one row's worth to start each pass; three rows at least (fewer
    // would wait for the epilogue).  64^3: 3 x 5, 22.3 us (5 x 3: 24.6); 256^3: 5 x 32.
    long long nchunks = 0, best = 0;
    for (int yl = std::min(3, ny); yl <= std::min(CVN_Y, ny); yl++)
      for (int z = std::min(64, nz); z >= 1; z--) {
        const int walks = (nz + z - 1) / z, zl = (nz + walks - 1) / walks;
        const long long units = (long long)P.tiles_x * ((ny + yl - 1) / yl) * walks;
        const long long cost = (units + 2 * sms - 1) / (2 * sms) * (zl + 2) * (yl + 1);
        if (best == 0 || cost < best) {
          best = cost;
          nchunks = units;
          P.yl = yl;
          P.zl = zl;
        }
      }
    FCB_CUDA_TRY(cudaFuncSetAttribute(conv3d16n_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, CVN_SMEM));
    const int grid = (int)std::min<long long>(nchunks, 2ll * sms);
    conv3d16n_kernel<<<grid, CVN_THREADS, CVN_SMEM, st>>>(map, P, (int)nchunks);
  }
  FCB_CUDA_TRY(cudaGetLastError());
  return ok();
}
FCB_CATCH_STATUS

extern "C" int fcb_conv3d16_wgrad_device(const void* x, const void* dy, int dyType, float* dw, int nx, int ny,
                                         int nz, void* stream)
try {
  if (!x || !dy || !dw || nx <= 0 || ny <= 0 || nz <= 0 || (dyType != FCB_F32 && dyType != FCB_BF16))
    return set_error(FCB_ERR_INVALID, "bad conv3d wgrad arguments");
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  // BF16 dY: tensor cores (FCB_WGRAD_SIMT=1 selects the CUDA-core kernel for comparison)
  const char* simt = getenv("FCB_WGRAD_SIMT");
  if (dyType == FCB_BF16 && !(simt && simt[0] == '1')) {
    if (((uintptr_t)x & 15) || ((uintptr_t)dy & 15))
      return set_error(FCB_ERR_INVALID, "conv3d wgrad buffers must be 16-byte aligned");
    const int gs = box_group(nx, 3), group = 1 << gs;
    const uint64_t dims[5] = {8ull * group, (uint64_t)(nx / group), 2, (uint64_t)ny, (uint64_t)nz};
    const uint64_t strides[4] = {16ull * group, 16ull * nx, 32ull * nx, 32ull * nx * ny};
    const uint32_t xbox[5] = {8u * group, (uint32_t)(WGT_XROW / group), 2, 1, 3};
    const uint32_t dybox[5] = {8u * group, (uint32_t)(CV_TILE / group), 1, 1, 1};
    CUtensorMap xmap, dymap;
    FCB_TRY(encode_tmap(&xmap, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<void*>(x), dims, strides, xbox));
    FCB_TRY(encode_tmap(&dymap, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<void*>(dy), dims, strides, dybox));
    int* status = nullptr;
    FCB_TRY(device_status_ptr(&status));
    WgradTcParams T;
    T.dw = dw;
    T.nx = nx; T.ny = ny; T.nz = nz;
    T.tiles_x = (nx + CV_TILE - 1) / CV_TILE;
    T.gs = gs;
    T.status = status;
    const long long nchunks = (long long)T.tiles_x * nz * ((ny + WGT_YCH - 1) / WGT_YCH);
    if (nchunks > 0x7fffffffll) return set_error(FCB_ERR_RANGE, "conv3d volume too large");
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    FCB_CUDA_TRY(cudaFuncSetAttribute(conv3d16_wgrad_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, WGT_SMEM));
    const int grid = (int)std::min<long long>(nchunks, sms);
    conv3d16_wgrad_tc_kernel<<<grid, WGT_THREADS, WGT_SMEM, st>>>(xmap, dymap, T, (int)nchunks);
    FCB_CUDA_TRY(cudaGetLastError());
    return ok();
  }
  WgradParams P;
  P.x = reinterpret_cast<const __nv_bfloat16*>(x);
  P.dy = dy;
  P.dy_f32 = dyType == FCB_F32;
  P.dw = dw;
  P.nx = nx; P.ny = ny; P.nz = nz;
  P.tiles_x = (nx + WG_TILE - 1) / WG_TILE;
  P.ntiles = P.tiles_x * ny * nz;
  const int grid = std::min(P.ntiles, 148 * 4);
  conv3d16_wgrad_kernel<<<grid, 256, 0, st>>>(P);
  FCB_CUDA_TRY(cudaGetLastError());
  return ok();
}
FCB_CATCH_STATUS
