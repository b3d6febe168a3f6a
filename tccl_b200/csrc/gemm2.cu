// Stand-alone bf16 GEMM on the CTA-pair mainloop (gemm_tcgen05_2cta.cuh):
// C = A * Bt^T with 256 x 256 tiles per pair of SMs, persistent over the tiles.
// The reference has no GEMM (presentation.pdf, slide 4, names the fusion with one as a goal).
#include "gemm_host.cuh"
#include "gemm_tcgen05_2cta.cuh"

namespace tccl {
namespace gemm2 {

struct PlainPolicy2 {
  static constexpr bool kEpiBarrier = false;
  const CUtensorMap *map_a, *map_b128, *map_b64;
  __nv_bfloat16* C;
  int M, N, ldc;  // N: rows of Bt
  int swiglu;
  Raster raster;
  TailSplitSchedule sched;
  __device__ __forceinline__ bool tile(int i, int& mt, int& nt, int& half) const {
    int t;
    if (!sched.unit(blockIdx.x >> 1, i, t, half)) return false;
    raster.at(t, mt, nt);
    mt *= 2;
    return true;
  }
  __device__ __forceinline__ void b_tile(int nt, int half, int cta, const CUtensorMap*& map, int& y) const {
    map = half ? map_b64 : map_b128;
    // gate | up packing: a half tile is 64 gate columns (CTA 0) and the 64 matching up columns (CTA 1)
    y = (swiglu && half) ? nt * BN2 + cta * 128 + (half == 2 ? 64 : 0) : b_rows_default(nt, half, cta);
  }
  __device__ __forceinline__ bool before_load(int, int, const Abort&) const { return true; }
  __device__ __forceinline__ void a_tile(int mt, const CUtensorMap*& map, int& y) const {
    map = map_a;
    y = mt * 128;
  }
  __device__ __forceinline__ void epilogue_finish(int, int, const Abort&) const {}
  __device__ __forceinline__ void between_tiles(int, int, const Abort&) const {}
  __device__ __forceinline__ void epilogue_begin(int, int, const Abort&) const {}
  __device__ __forceinline__ bool epilogue(int mt, int nt, int col0, int ncols, uint32_t taddr, int quad, int lane,
                                           const Abort&, const Smem2& sm) const {
    if (swiglu) {
      store_rows_swiglu(sm.epi[0] + quad * 4096, C, ldc, mt * 128 + quad * 32, M, nt * (BN2 / 2) + col0 / 2, N / 2,
                        ncols / 2, taddr, lane);
      return true;
    }
    store_rows(sm.epi[0] + quad * 4096, C, ldc, mt * 128 + quad * 32, M, nt * BN2 + col0, N, ncols, taddr, lane);
    return true;
  }
};

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b128,
                 const __grid_constant__ CUtensorMap map_b64, const Shape shp, PlainPolicy2 pol, uint32_t* status,
                 uint64_t timeout_ns, uint64_t* trace) {
  tccl_comm fake;
  fake.local = status ? status - TCCL_LOCAL_STATUS : nullptr;
  pol.map_a = &map_a;
  pol.map_b128 = &map_b128;
  pol.map_b64 = &map_b64;
  run_mainloop2(shp, pol, status ? &fake : nullptr, timeout_ns, trace ? trace + (size_t)blockIdx.x * 64 : nullptr);
}

int check_gemm_args(const tccl_gemm_args* g) {
  if (!g || g->m <= 0 || g->n <= 0 || g->k <= 0) return -TCCL_EINVAL;
  if ((g->lda % 8) || (g->ldb % 8) || (g->ldc % 8) || (g->n % 8) || (g->k % 8)) return -TCCL_EALIGN;
  if (((uintptr_t)g->a | (uintptr_t)g->bt | (uintptr_t)g->c) & 15) return -TCCL_EALIGN;
  if (g->swiglu && (g->n % BN2)) return -TCCL_ESIZE;  // whole gate|up tiles only
  return 0;
}

int launch_gemm_pair(const tccl_gemm_args* g, int grid, cudaStream_t stream, uint64_t timeout_ns, uint64_t* trace) {
  int rc = check_gemm_args(g);
  if (rc) return rc;
  if (grid <= 0 && !trace && launch_gemm_skinny(g, stream, timeout_ns, &rc)) return rc;
  CUtensorMap ma, mb128, mb64;
  rc = make_tmap_bf16_kmajor(&ma, g->a, g->m, g->k, g->lda, 128);  // each CTA loads 128 rows of A ...
  if (rc) return rc;
  rc = make_tmap_bf16_kmajor(&mb128, g->bt, g->n, g->k, g->ldb, 128);  // ... and 128 rows of Bt (64 for a half tile)
  if (rc) return rc;
  rc = make_tmap_bf16_kmajor(&mb64, g->bt, g->n, g->k, g->ldb, 64);
  if (rc) return rc;
  PlainPolicy2 pol{};
  pol.C = reinterpret_cast<__nv_bfloat16*>(g->c);
  pol.M = g->m;
  pol.N = g->n;
  pol.ldc = g->ldc;
  pol.swiglu = g->swiglu;
  const int tm = (g->m + 255) / 256, tn = (g->n + BN2 - 1) / BN2, total = tm * tn;
  pol.raster = Raster{tn, raster_group(tm, g->k), tm};
  if (grid <= 0) grid = tccl_num_sms();
  grid &= ~1;
  // fewer tiles than pairs: half tiles if every half then has a pair of its own, else one whole tile each
  if (grid > 2 * total) grid = grid >= 4 * total ? 4 * total : 2 * total;
  if (grid < 2) return -TCCL_EINVAL;
  pol.sched.init(total, grid / 2);
  static bool attr_set = false;
  if (!attr_set) {
    cudaError_t e = cudaFuncSetAttribute(gemm_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem2);
    if (e != cudaSuccess) return (int)e;
    attr_set = true;
  }
  Shape shp{g->m, g->n, g->k};
  return launch_dependent(gemm_pair_kernel, dim3(grid), kThreads, kSmem2, stream, 0, ma, mb128, mb64, shp, pol,
                          reinterpret_cast<uint32_t*>(g->status), timeout_ns, trace);
}

}  // namespace gemm2
}  // namespace tccl

extern "C" int tccl_gemm_bf16_pair(const tccl_gemm_args* g, int grid, void* stream) {
  return tccl::gemm2::launch_gemm_pair(g, grid, reinterpret_cast<cudaStream_t>(stream), 2000000000ull, nullptr);
}
