// bf16 GEMM of few rows (a decode step: 1 .. 128 tokens): C[m, n] = A[m, k] * Bt[n, k]^T, optionally with the SwiGLU
// epilogue over a packed gate | up Bt.
//
// What bounds it: reading Bt once from DRAM (235 MB for a [28672, 4096] gate/up projection: 37 us).  A 256 x 256
// pair tile is the wrong shape for that: 16 rows use 1/16 of its A half, two thirds of a 256-wide wave are idle, and
// N = 4096 leaves 16 of 74 pairs with work (59 us for 117 MB).  So here
//  * the operands change places: 128 rows of Bt are the M side of tcgen05.mma, the tokens (padded to 16, 32, 64 or
//    128) its N side, so a stage is 16 KB of weights plus only as many bytes of A as there are tokens;
//  * K is split over the S CTAs of a cluster.  Each keeps its fp32 partial [tokens][128] in its own shared memory (the
//    pipeline's, which is idle by then), and after one cluster barrier every CTA sums the partials of its share of the
//    tokens over distributed shared memory, in rank order: no workspace, no atomics, the same bits every time;
//  * two CTAs share an SM (about 100 KB of stages each), so one's fill and drain hide behind the other's stream.
// S is the largest power of two that keeps all CTAs resident at once: then they all stream at an equal share of the
// DRAM bandwidth and end together, and there is no partial last wave.
//
// The reference has no GEMM (presentation.pdf, slide 4, names the fusion with one as a goal).
#include "gemm_host.cuh"
#include "gemm_tcgen05_2cta.cuh"

namespace tccl {
namespace gemm2 {

constexpr int kSkinnyRows = 128;  // rows of Bt per tile
constexpr uint32_t kSkinnyW = kSkinnyRows * 64 * 2;

template <int TN> struct SkinnyCfg {
  static constexpr uint32_t kStageBytes = kSkinnyW + TN * 128;
  static constexpr int kStages = TN <= 16 ? 6 : (TN <= 32 ? 5 : (TN <= 64 ? 4 : 3));
  static constexpr uint32_t kPartBytes = TN * kSkinnyRows * 4;  // aliases the stages
  static constexpr uint32_t kTmem = TN < 32 ? 32 : TN;
  static constexpr size_t kSmem = 1024 + (size_t)kStages * kStageBytes + 256;
  static_assert(kPartBytes <= kStages * kStageBytes, "partials alias the stages");
};

struct SkinnyArgs {
  __nv_bfloat16* C;
  int M, N, K, ldc;   // N: columns of C
  int swiglu;         // rows of Bt: 256-row blocks of 128 gate rows and the 128 matching up rows; C has half as many columns
  uint32_t* status;
};

__device__ __forceinline__ float4 ld_dsmem_f4(uint32_t cluster_addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(cluster_addr) : "memory");
  return v;
}

template <int TN>
__global__ void __launch_bounds__(kThreads, 2)
gemm_skinny_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a,
                   const SkinnyArgs p, const int splits) {
  using Cfg = SkinnyCfg<TN>;
  constexpr int NS = Cfg::kStages;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint64_t* full = reinterpret_cast<uint64_t*>(base + NS * Cfg::kStageBytes);
  uint64_t *empty = full + NS, *done = empty + NS;
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(done + 1);
  int* abort_flag = reinterpret_cast<int*>(tmem_ptr + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tile = blockIdx.x / splits, s = blockIdx.x - tile * splits;
  const int num_kb = (p.K + 63) / 64;
  const int kb0 = (int)((long long)num_kb * s / splits), kb1 = (int)((long long)num_kb * (s + 1) / splits);

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&map_w);
    tma_prefetch_desc(&map_a);
    *abort_flag = 0;
    for (int i = 0; i < NS; ++i) {
      mbar_init(full + i, 1);
      mbar_init(empty + i, 1);
    }
    mbar_init(done, 1);
    fence_barrier_init();
  }
  if (warp == 2) {
    tmem_alloc(tmem_ptr, Cfg::kTmem);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_ptr;
  Abort ab{abort_flag, nullptr, p.status, globaltimer() + 2000000000ull};

  if (warp == 0) {
    if (elect_one()) {
      // first row of Bt of this tile; with SwiGLU 64 gate rows and, 128 further on, the 64 matching up rows
      const int y0 = p.swiglu ? (tile >> 1) * 256 + (tile & 1) * 64 : tile * kSkinnyRows;
      const int y1 = y0 + (p.swiglu ? 128 : 64);
      bool ok = true;
      int it = 0;
      for (int kb = kb0; ok && kb < kb1; ++kb, ++it) {
        const int st = it % NS;
        ok = mbar_wait(empty + st, ((it / NS) & 1) ^ 1, ab);
        if (!ok) break;
        uint8_t* w = base + (size_t)st * Cfg::kStageBytes;
        mbar_arrive_expect_tx(full + st, Cfg::kStageBytes);
        tma_load_2d(w, &map_w, full + st, kb * 64, y0);
        tma_load_2d(w + kSkinnyW / 2, &map_w, full + st, kb * 64, y1);
        tma_load_2d(w + kSkinnyW, &map_a, full + st, kb * 64, 0);
      }
      // copies in flight land before the CTA goes on to reuse or leave the shared memory
      const int pending = it < NS ? it : NS;
      int dummy = 0;
      Abort drain{&dummy, nullptr, nullptr, globaltimer() + 2000000000ull};
      for (int j = it - pending; j < it; ++j) mbar_wait(full + j % NS, (j / NS) & 1, drain);
    }
  } else if (warp == 1) {
    if (elect_one()) {
      constexpr uint32_t idesc = make_idesc_bf16(kSkinnyRows, TN);
      bool ok = true;
      int it = 0;
      for (int kb = kb0; ok && kb < kb1; ++kb, ++it) {
        const int st = it % NS;
        ok = mbar_wait(full + st, (it / NS) & 1, ab);
        if (!ok) break;
        tc_fence_after();
        const uint32_t w = smem_u32(base + (size_t)st * Cfg::kStageBytes);
        const uint64_t ad = make_desc_sw128(w), bd = make_desc_sw128(w + kSkinnyW);
#pragma unroll
        for (int k = 0; k < 4; ++k)
          tc_mma_bf16(tmem, ad + (uint64_t)(k * 2), bd + (uint64_t)(k * 2), idesc, (it | k) ? 1u : 0u);
        tc_commit(empty + st);
      }
      tc_commit(done);
    }
  }
  __syncwarp();
  if (warp >= kEpiWarp0) {
    // the partial, token by token: lane = row of Bt, so consecutive lanes store consecutive words
    const int row = (warp - kEpiWarp0) * 32 + lane;
    float* part = reinterpret_cast<float*>(base);
    if (mbar_wait(done, 0, ab)) {
      tc_fence_after();
      const uint32_t taddr = tmem + ((uint32_t)((warp - kEpiWarp0) * 32) << 16);
#pragma unroll 1
      for (int c = 0; c < TN; c += 32) {
        uint32_t r[32];
        tmem_ld_32x32(taddr + c, r);  // (16 tokens: the other 16 columns are allocated and ignored)
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; ++i)
          if (c + i < TN) part[(c + i) * kSkinnyRows + row] = __uint_as_float(r[i]);
      }
    }
    tc_fence_before();
  }
  // every CTA of the cluster has its partial in shared memory
  if (splits > 1) cluster_sync();
  else __syncthreads();
  const int ncta = p.swiglu ? kSkinnyRows / 2 : kSkinnyRows;  // columns of C per tile
  const int vpt = ncta / 8;                                   // 16-byte vectors per token
  const uint32_t part0 = smem_u32(base);
  for (int i = threadIdx.x; i < TN / splits * vpt; i += kThreads) {
    const int tok = (i / vpt) * splits + s, v = i % vpt;  // tokens are dealt to the CTAs in turn
    const int col = tile * ncta + v * 8;
    if (tok >= p.M || col >= p.N) continue;
    float acc[8], up[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[e] = up[e] = 0.f;
    const uint32_t off = part0 + (uint32_t)(tok * kSkinnyRows + v * 8) * 4;
    for (int q = 0; q < splits; ++q) {
      const uint32_t a = mapa(off, q);
      const float4 x = ld_dsmem_f4(a), y = ld_dsmem_f4(a + 16);
      acc[0] += x.x; acc[1] += x.y; acc[2] += x.z; acc[3] += x.w;
      acc[4] += y.x; acc[5] += y.y; acc[6] += y.z; acc[7] += y.w;
      if (p.swiglu) {
        const float4 z = ld_dsmem_f4(a + 256), w = ld_dsmem_f4(a + 272);  // 64 rows further on
        up[0] += z.x; up[1] += z.y; up[2] += z.z; up[3] += z.w;
        up[4] += w.x; up[5] += w.y; up[6] += w.z; up[7] += w.w;
      }
    }
    if (p.swiglu) {
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[e] = swiglu(acc[e], up[e]);
    }
    uint32_t o[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) o[e] = __float_as_uint(acc[e]);
    st_local(p.C + (size_t)tok * p.ldc + col, pack8_bf16(o));
  }
  // nobody leaves while another CTA of the cluster may still read its partial
  __syncthreads();
  if (splits > 1) cluster_sync_relaxed();
  if (warp == 2) {
    tc_fence_after();
    tmem_dealloc(tmem, Cfg::kTmem);
  }
}

template <int TN>
static int launch_tn(const tccl_gemm_args* g, int splits, int tiles, cudaStream_t stream) {
  CUtensorMap mw, ma;
  int rc = make_tmap_bf16_kmajor(&mw, g->bt, g->n, g->k, g->ldb, 64);
  if (rc) return rc;
  rc = make_tmap_bf16_kmajor(&ma, g->a, g->m, g->k, g->lda, TN);
  if (rc) return rc;
  static bool attr_set = false;
  if (!attr_set) {
    cudaError_t e = cudaFuncSetAttribute(gemm_skinny_kernel<TN>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)SkinnyCfg<TN>::kSmem);
    if (e != cudaSuccess) return (int)e;
    attr_set = true;
  }
  const SkinnyArgs p{reinterpret_cast<__nv_bfloat16*>(g->c), g->m, g->swiglu ? g->n / 2 : g->n, g->k, g->ldc, g->swiglu,
                     reinterpret_cast<uint32_t*>(g->status)};
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(tiles * splits);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = SkinnyCfg<TN>::kSmem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = splits;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return (int)cudaLaunchKernelEx(&cfg, gemm_skinny_kernel<TN>, mw, ma, p, splits);
}

int launch_gemm_skinny(const tccl_gemm_args* g, cudaStream_t stream) {
  const int tiles = (g->n + kSkinnyRows - 1) / kSkinnyRows, num_kb = (g->k + 63) / 64;
  const int slots = 2 * tccl_num_sms();
  int splits = 1;
  while (splits < 8 && tiles * splits * 2 <= slots && num_kb >= splits * 2 * 2) splits *= 2;
  if (g->m <= 16) return launch_tn<16>(g, splits, tiles, stream);
  if (g->m <= 32) return launch_tn<32>(g, splits, tiles, stream);
  if (g->m <= 64) return launch_tn<64>(g, splits, tiles, stream);
  return launch_tn<128>(g, splits, tiles, stream);
}

}  // namespace gemm2
}  // namespace tccl
