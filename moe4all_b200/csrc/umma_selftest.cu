// Self-test of the tcgen05 helpers: C[128, N] = A[128, 64] * B[N, 64]^T with f16 operands the way the grouped GEMM has them - a pair of
// CTAs, A in the tensor memory of each (here the same 128 rows in both), half of B's rows in the shared memory of each, four MMAs of
// K = 16 issued by the first for both.  Each CTA writes the columns of its half of B from its own accumulators, so the product is right
// only if both tensor cores read both halves.  This entry point lets the test-suite check the helpers against a plain matrix product.
#include "kernels.cuh"
#include "umma.cuh"

namespace infr {
namespace {

constexpr uint32_t ST_A_COL = 256;  // accumulators: columns 0 .. 255

__global__ void __launch_bounds__(128) k_umma_selftest(const __half* __restrict__ A, const __half* __restrict__ B,
                                                       float* __restrict__ C, int N, DeviceStatus* status) {
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t s_bar;
  __shared__ uint32_t s_tmem;
  unsigned char* tB = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, rank = (int)umma::pair_rank();
  const int n = (N + 31) & ~31, half = n / 2;

  for (int i = tid; i < half * 8; i += 128) {
    const int r = i >> 3, c = i & 7, row = rank * half + r;
    *reinterpret_cast<uint4*>(tB + r * 128 + ((c ^ (r & 7)) << 4)) =
        row < N ? *reinterpret_cast<const uint4*>(B + (size_t)row * 64 + c * 8) : make_uint4(0, 0, 0, 0);
  }
  if (tid == 0) {
    mbar_init(&s_bar, 1);
    mbar_fence_init();
  }
  if (warp == 0) umma::tmem_alloc_pair(&s_tmem);
  umma::fence_before_sync();
  umma::pair_sync();
  umma::fence_after_sync();
  const uint32_t tmem = s_tmem, lanes = tmem + ((uint32_t)(warp * 32) << 16);
  uint32_t a[32];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const uint4 v = *reinterpret_cast<const uint4*>(A + (size_t)tid * 64 + i * 8);
    a[4 * i] = v.x, a[4 * i + 1] = v.y, a[4 * i + 2] = v.z, a[4 * i + 3] = v.w;
  }
  umma::tmem_st_32x32(lanes + ST_A_COL, a);
  umma::fence_proxy_async();
  umma::fence_before_sync();
  umma::pair_sync();
  umma::fence_after_sync();

  if (rank == 0 && warp == 0) {
    if (umma::elect_one()) {
      const uint32_t idesc = umma::idesc_f16_f32(256, n);
#pragma unroll
      for (int k = 0; k < 4; ++k)
        umma::mma_f16_ta(tmem, tmem + ST_A_COL + 8 * k, umma::smem_desc_k_major_swz128(tB, k), idesc, k > 0 ? 1u : 0u);
      umma::commit_pair(&s_bar);
    }
    __syncwarp();
  }
  const bool ok = __all_sync(0xFFFFFFFFu, mbar_wait_bounded(&s_bar, 0));
  umma::fence_after_sync();
  if (ok) {
    for (int c0 = rank * half; c0 < (rank + 1) * half; c0 += 16) {
      float v[2][8], again[2][8];
      const uint32_t at = lanes + (uint32_t)c0;
      umma::tmem_ld_16x16_quad(at, at + (16u << 16), at, at + (16u << 16), v[0], v[1], again[0], again[1]);
      for (int h = 0; h < 2; ++h)
        for (int i = 0; i < 8; ++i) {
          const int row = warp * 32 + 16 * h + (lane >> 2) + 8 * ((i >> 1) & 1), col = c0 + 8 * (i >> 2) + 2 * (lane & 3) + (i & 1);
          if (col < N) C[(size_t)row * N + col] = v[h][i];
        }
    }
  } else if (lane == 0) {
    atomicExch(&status->timeout, 9);
  }
  umma::fence_before_sync();
  __syncwarp();
  umma::pair_sync();
  __syncwarp();
  if (warp == 0) umma::tmem_dealloc_pair(tmem);
}

}  // namespace

int32_t launch_umma_selftest(infr_cuda_ctx* ctx, const __half* a, const __half* b, float* c, int n) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2);
  cfg.blockDim = dim3(128);
  cfg.dynamicSmemBytes = 1024 + 128 * 128;  // up to 128 rows of B in each CTA
  cfg.stream = ctx->stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim = {2, 1, 1};
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, k_umma_selftest, a, b, c, n, ctx->status);
  if (e != cudaSuccess) return check_cuda(ctx, e, "umma selftest launch");
  ctx->launches += 1;
  return check_cuda(ctx, cudaGetLastError(), "umma selftest launch");
}

}  // namespace infr
