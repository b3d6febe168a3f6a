// bf16 GEMM with one tile per CTA (or per pair of CTAs): C[m, n] = A[m, k] * Bt[n, k]^T, optionally with the SwiGLU
// epilogue over a packed gate | up Bt.  For products that leave the persistent 256 x 256 pair kernel (gemm2.cu) short of
// tiles: decode steps of 1 .. 128 tokens, and anything with fewer tiles than the GPU has pairs of SMs.
//
// What bounds a decode step: reading Bt once from DRAM (235 MB for a [28672, 4096] gate/up projection: 37 us).  A 256 x
// 256 pair tile is the wrong shape for that: 16 rows use 1/16 of its A half, two thirds of a 256-wide wave are idle, and
// N = 4096 leaves 16 of 74 pairs with work.  So here
//  * the operands change places: 128 rows of Bt (256 on a pair) are the M side of tcgen05.mma, TN = 16 .. 256 tokens its
//    N side, so a stage is 16 KB of weights plus only as many bytes of A as there are tokens;
//  * K is split over the CTAs (or pairs) of a cluster.  Each keeps its fp32 partial [tokens][128] in its own shared memory
//    (the pipeline's, which is idle by then), and after one cluster barrier every CTA sums the partials of its share of
//    the tokens over distributed shared memory, in rank order: no workspace, no atomics, the same bits every time;
//  * with few tokens two CTAs share an SM (about 100 KB of stages each), so one's fill and drain hide behind the other's
//    stream, and the launch is a dependent one: it overlaps the previous kernel's drain.
// Measured (start: pair kernel only), inputs from DRAM: 16 x 28672 x 4096 63.2 -> 38.8 us (6.05 TB/s of weights);
// 16 x 4096 x 14336 69.0 -> 21.0; 16 x 2048 x 2048 15.8 -> 5.3; 300 x 1000 x 1000 13.6 -> 7.1; 1000 x 1792 x 4096
// 29.5 -> 15.6.  Which configuration, and from where on the pair kernel: `choose` below.
//
// The reference has no GEMM (presentation.pdf, slide 4, names the fusion with one as a goal).
#include <math.h>

#include "gemm_host.cuh"
#include "gemm_tcgen05_2cta.cuh"

namespace tccl {
namespace gemm2 {

constexpr int kSkinnyRows = 128;  // rows of Bt per tile
constexpr uint32_t kSkinnyW = kSkinnyRows * 64 * 2;

// TN tokens per tile on CG CTAs (1, or a pair with tcgen05.mma.cta_group::2: 256 rows of Bt, each CTA loads its own 128
// and half of the tokens)
template <int TN, int CG> struct SkinnyCfg {
  static constexpr uint32_t kStageBytes = kSkinnyW + TN / CG * 128;
  static constexpr uint32_t kPartBytes = TN * kSkinnyRows * 4;  // aliases the stages
  static constexpr uint32_t kTmem = TN < 32 ? 32 : TN;
  // stages for `per_sm` CTAs on an SM (the partial of 256 tokens needs an SM to itself)
  static constexpr int stages(int per_sm) { return (int)((per_sm == 2 ? 110u << 10 : 222u << 10) / kStageBytes); }
  static constexpr size_t smem(int per_sm) { return 1024 + (size_t)stages(per_sm) * kStageBytes + 512; }
  static_assert(kPartBytes <= stages(TN <= 128 ? 2 : 1) * kStageBytes, "partials alias the stages");
};

struct SkinnyArgs {
  __nv_bfloat16* C;
  int M, N, K, ldc;   // N: columns of C
  int swiglu;         // rows of Bt: 256-row blocks of 128 gate rows and the 128 matching up rows; C has half as many columns
  uint32_t* status;
  uint64_t timeout_ns;  // bound of the kernel's waits together
};

__device__ __forceinline__ float4 ld_dsmem_f4(uint32_t cluster_addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(cluster_addr) : "memory");
  return v;
}

// Sum of the S partials of this CTA's tokens (dealt to the splits in turn) and the stores to C.  A thread takes four
// columns of C at a time, several such pieces together: neighbouring lanes read neighbouring 16 bytes, and all loads
// are in flight before the first sum (one piece of 8 columns at a time took 4.5 us for 256 tokens over two splits).
template <int TN, int CG, int S, bool kSwiglu>
__device__ __forceinline__ void skinny_reduce(const SkinnyArgs& p, uint32_t part0, int rt, int tok0, int s, int c) {
  constexpr int kCols = kSwiglu ? kSkinnyRows / 2 : kSkinnyRows, kVpt = kCols / 4;  // columns, pieces per token
  constexpr int kTotal = TN / S * kVpt, kLd = kSwiglu ? 2 : 1;
  constexpr int U = S * kLd >= 16 ? 1 : 16 / (S * kLd);
  for (int i0 = threadIdx.x; i0 < kTotal; i0 += U * kThreads) {
    float4 v[U][S][kLd];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = i0 + u * kThreads, tok = i / kVpt * S + s;
      // from another CTA only what is stored below is loaded: a load that nothing waits for could outlive that CTA
      if (i < kTotal && tok0 + tok < p.M && (S == 1 || rt * kCols + i % kVpt * 4 < p.N)) {
        const uint32_t off = part0 + (uint32_t)(tok * kSkinnyRows + i % kVpt * 4) * 4;
#pragma unroll
        for (int q = 0; q < S; ++q) {
          const uint32_t a = mapa(off, q * CG + c);
          v[u][q][0] = ld_dsmem_f4(a);
          if (kSwiglu) v[u][q][kLd - 1] = ld_dsmem_f4(a + 256);  // the matching up rows, 64 further on
        }
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = i0 + u * kThreads, tok = i / kVpt * S + s, col = rt * kCols + i % kVpt * 4;
      if (i >= kTotal || tok0 + tok >= p.M || col >= p.N) continue;
      float4 t[kLd];
#pragma unroll
      for (int e = 0; e < kLd; ++e) {
        t[e] = v[u][0][e];
#pragma unroll
        for (int q = 1; q < S; ++q) {
          t[e].x += v[u][q][e].x; t[e].y += v[u][q][e].y; t[e].z += v[u][q][e].z; t[e].w += v[u][q][e].w;
        }
      }
      if (kSwiglu) {
        const float4 w = t[kLd - 1];
        t[0] = float4{swiglu(t[0].x, w.x), swiglu(t[0].y, w.y), swiglu(t[0].z, w.z), swiglu(t[0].w, w.w)};
      }
      const uint2 o{Acc<__nv_bfloat16>::pk(t[0].x, t[0].y), Acc<__nv_bfloat16>::pk(t[0].z, t[0].w)};
      *reinterpret_cast<uint2*>(p.C + (size_t)(tok0 + tok) * p.ldc + col) = o;
    }
  }
}

template <int TN, int CG>
__global__ void __launch_bounds__(kThreads, TN <= 128 ? 2 : 1)
gemm_skinny_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a,
                   const SkinnyArgs p, const int splits, const int NS) {
  using Cfg = SkinnyCfg<TN, CG>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint64_t* full = reinterpret_cast<uint64_t*>(base + NS * Cfg::kStageBytes);
  uint64_t *empty = full + NS, *done = empty + NS;
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(done + 1);
  int* abort_flag = reinterpret_cast<int*>(tmem_ptr + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // cluster = CG * splits CTAs: CTA c of pair s is rank s * CG + c; rt = this CTA's 128-row tile of Bt
  const int cl = CG * splits, rank = (int)blockIdx.x % cl, s = rank / CG, c = rank % CG;
  const int rt = (int)blockIdx.x / cl * CG + c, tok0 = blockIdx.y * TN;
  const bool leader = c == 0;
  const int num_kb = (p.K + 63) / 64;
  const int kb0 = (int)((long long)num_kb * s / splits), kb1 = (int)((long long)num_kb * (s + 1) / splits);

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&map_w);
    tma_prefetch_desc(&map_a);
    *abort_flag = 0;
    for (int i = 0; i < NS; ++i) {
      mbar_init(full + i, 2);  // both producers' arrive.expect_tx
      mbar_init(empty + i, 1);
    }
    mbar_init(done, 1);
    fence_barrier_init();
  }
  if (warp == 2) {
    if (CG == 2) {
      tmem_alloc2(tmem_ptr, Cfg::kTmem);
      tmem_relinquish2();
    } else {
      tmem_alloc(tmem_ptr, Cfg::kTmem);
      tmem_relinquish();
    }
  }
  tc_fence_before();
  __syncthreads();
  if (CG == 2) cluster_sync();  // the pair's barriers are initialised before anyone signals across
  tc_fence_after();
  const uint32_t tmem = *tmem_ptr;
  grid_dependency_wait();
  Abort ab{abort_flag, nullptr, p.status, globaltimer() + p.timeout_ns};

  if (warp == 0 || warp == 3) {
    // ------------------------------------------------------ TMA producers: warp 0 loads rows of Bt, warp 3 tokens.  Two
    // threads, because what a k-block costs here is issuing it (~0.15 us for a wait, an expect and three copies
    // whatever their size), not its bytes.
    if (elect_one()) {
      const bool weights = warp == 0;
      // the CTA's rows of Bt: 128, or with SwiGLU 64 gate rows and, 128 further on, the 64 matching up rows
      const int y = !weights ? tok0 + c * (TN / CG) : (p.swiglu ? (rt >> 1) * 256 + (rt & 1) * 64 : rt * kSkinnyRows);
      const CUtensorMap* map = weights ? &map_w : &map_a;
      const uint32_t bytes = CG * (weights ? kSkinnyW : Cfg::kStageBytes - kSkinnyW);
      const uint32_t off = weights ? 0 : kSkinnyW;
      const uint32_t leader_full = mapa(smem_u32(full), rank & ~(CG - 1));
      bool ok = true;
      int it = 0, st = 0;
      uint32_t ph = 0;
      for (int kb = kb0; ok && kb < kb1; ++kb, ++it) {
        ok = mbar_wait(empty + st, ph ^ 1, ab);
        if (!ok) break;
        uint8_t* dst = base + (size_t)st * Cfg::kStageBytes + off;
        if (leader) mbar_arrive_expect_tx(full + st, bytes);
        if (CG == 2) {
          const uint32_t bar = leader_full + st * 8;
          tma_load_2d_pair(dst, map, bar, kb * 64, y);
          if (weights && p.swiglu) tma_load_2d_pair(dst + kSkinnyW / 2, map, bar, kb * 64, y + 128);
        } else {
          tma_load_2d(dst, map, full + st, kb * 64, y);
          if (weights && p.swiglu) tma_load_2d(dst + kSkinnyW / 2, map, full + st, kb * 64, y + 128);
        }
        if (++st == NS) st = 0, ph ^= 1;
      }
      if (leader && !ok) {  // after a failed wait: copies in flight land before the CTAs leave
        const int pending = it < NS ? it : NS;
        int dummy = 0;
        Abort drain{&dummy, nullptr, nullptr, globaltimer() + 2000000000ull};
        for (int j = it - pending; j < it; ++j) mbar_wait(full + j % NS, (j / NS) & 1, drain);
      }
    }
  } else if (warp == 1 && leader) {
    if (elect_one()) {
      constexpr uint32_t idesc = make_idesc_bf16(CG * kSkinnyRows, TN);
      bool ok = true;
      int it = 0, st = 0;
      uint32_t ph = 0;
      const uint32_t peer_empty = CG == 2 ? mapa(smem_u32(empty), rank | 1) : 0;
      for (int kb = kb0; ok && kb < kb1; ++kb, ++it) {
        ok = mbar_wait(full + st, ph, ab);
        if (!ok) break;
        tc_fence_after();
        const uint32_t w = smem_u32(base + (size_t)st * Cfg::kStageBytes);
        const uint64_t ad = make_desc_sw128(w), bd = make_desc_sw128(w + kSkinnyW);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          if (CG == 2) tc_mma2_bf16(tmem, ad + (uint64_t)(k * 2), bd + (uint64_t)(k * 2), idesc, (it | k) ? 1u : 0u);
          else tc_mma_bf16(tmem, ad + (uint64_t)(k * 2), bd + (uint64_t)(k * 2), idesc, (it | k) ? 1u : 0u);
        }
        if (CG == 2) {
          tc_commit2(smem_u32(empty + st));
          tc_commit2(peer_empty + (uint32_t)st * 8);
        } else {
          tc_commit(empty + st);
        }
        if (++st == NS) st = 0, ph ^= 1;
      }
      if (CG == 2) {
        tc_commit2(smem_u32(done));
        tc_commit2(mapa(smem_u32(done), rank | 1));
      } else {
        tc_commit(done);
      }
    }
  }
  __syncwarp();
  {
    // the partial, token by token: lane = row of Bt, so consecutive lanes store consecutive words.  Warps w and w + 4
    // read the same quarter of the tensor memory's lanes; they share its columns.
    const int quad = warp & 3, row = quad * 32 + lane;
    float* part = reinterpret_cast<float*>(base);
    if (agree<false>(mbar_wait(done, 0, ab))) {
      tc_fence_after();
      const uint32_t taddr = tmem + ((uint32_t)(quad * 32) << 16);
#pragma unroll 1
      for (int t = (warp >> 2) * 32; t < TN && tok0 + t < p.M; t += 64) {
        uint32_t r[32];
        tmem_ld_32x32(taddr + t, r);  // (16 tokens: the other 16 columns are allocated and ignored)
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; ++i)
          if (t + i < TN) part[(t + i) * kSkinnyRows + row] = __uint_as_float(r[i]);
      }
    }
    tc_fence_before();
  }
  // every CTA of the cluster has its partial in shared memory
  if (splits > 1) cluster_sync();
  else __syncthreads();
  const uint32_t part0 = smem_u32(base);
#define TCCL_SKINNY_REDUCE(S)                                                             \
  case S:                                                                                 \
    if (p.swiglu) skinny_reduce<TN, CG, S, true>(p, part0, rt, tok0, s, c);               \
    else skinny_reduce<TN, CG, S, false>(p, part0, rt, tok0, s, c);                       \
    break;
  switch (splits) {
    TCCL_SKINNY_REDUCE(1)
    TCCL_SKINNY_REDUCE(2)
    TCCL_SKINNY_REDUCE(4)
    TCCL_SKINNY_REDUCE(8)
  }
#undef TCCL_SKINNY_REDUCE
  // Nobody leaves while another CTA of the cluster may still read its partial, or while the leader's commits are still on
  // their way to this CTA's barriers: each lane looks at the last phase of one stage's (all landed long ago, unless a wait
  // failed; a thread that waited for one stage after the other where the loads end cost 1.5 us).
  __syncthreads();
  if (cl > 1) cluster_arrive_relaxed();
  if (CG == 2 && !leader && warp == 0 && lane < NS && lane < kb1 - kb0)
    drain_ring(empty + lane, 1, (uint32_t)((kb1 - kb0 - 1 - lane) / NS + 1), !*ab.flag, p.timeout_ns);
  __syncwarp();
  if (cl > 1) cluster_wait();
  if (warp == 2) {
    tc_fence_after();
    if (CG == 2) tmem_dealloc2(tmem, Cfg::kTmem);
    else tmem_dealloc(tmem, Cfg::kTmem);
  }
}

template <int TN, int CG>
static int launch_tn(const tccl_gemm_args* g, int splits, int per_sm, uint64_t timeout_ns, cudaStream_t stream) {
  using Cfg = SkinnyCfg<TN, CG>;
  CUtensorMap mw, ma;
  int rc = make_tmap_bf16_kmajor(&mw, g->bt, g->n, g->k, g->ldb, g->swiglu ? 64 : 128);
  if (rc) return rc;
  rc = make_tmap_bf16_kmajor(&ma, g->a, g->m, g->k, g->lda, TN / CG);
  if (rc) return rc;
  static bool attr_set = false;
  if (!attr_set) {
    cudaError_t e = cudaFuncSetAttribute(gemm_skinny_kernel<TN, CG>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)Cfg::smem(1));
    if (e != cudaSuccess) return (int)e;
    attr_set = true;
  }
  const SkinnyArgs p{reinterpret_cast<__nv_bfloat16*>(g->c), g->m, g->swiglu ? g->n / 2 : g->n, g->k, g->ldc, g->swiglu,
                     reinterpret_cast<uint32_t*>(g->status), timeout_ns};
  const int tiles = (g->n + CG * kSkinnyRows - 1) / (CG * kSkinnyRows);
  return launch_dependent(gemm_skinny_kernel<TN, CG>, dim3(tiles * splits * CG, (g->m + TN - 1) / TN), kThreads,
                          Cfg::smem(per_sm), stream, splits * CG, mw, ma, p, splits, Cfg::stages(per_sm));
}

// The tiles there are: `tn` tokens by `cg` * 128 rows of Bt
static const struct { int tn, cg; } kTiles[] = {{16, 1}, {32, 1}, {64, 1}, {128, 1}, {32, 2}, {64, 2}, {128, 2}, {256, 2}};
static int max_per_sm(int tn) { return tn <= 128 ? 2 : 1; }

// K split `splits` ways, `per_sm` CTAs on an SM; every split has at least one k-block
static int launch_as(const tccl_gemm_args* g, int tn, int cg, int splits, int per_sm, uint64_t timeout_ns,
                     cudaStream_t stream) {
  if (splits < 1 || (splits & (splits - 1)) || cg * splits > 8 || splits > (g->k + 63) / 64) return -TCCL_ESIZE;
  if (per_sm < 1 || per_sm > max_per_sm(tn)) return -TCCL_ESIZE;
  switch (tn * 4 + cg) {
    case 16 * 4 + 1: return launch_tn<16, 1>(g, splits, per_sm, timeout_ns, stream);
    case 32 * 4 + 1: return launch_tn<32, 1>(g, splits, per_sm, timeout_ns, stream);
    case 64 * 4 + 1: return launch_tn<64, 1>(g, splits, per_sm, timeout_ns, stream);
    case 128 * 4 + 1: return launch_tn<128, 1>(g, splits, per_sm, timeout_ns, stream);
    case 32 * 4 + 2: return launch_tn<32, 2>(g, splits, per_sm, timeout_ns, stream);
    case 64 * 4 + 2: return launch_tn<64, 2>(g, splits, per_sm, timeout_ns, stream);
    case 128 * 4 + 2: return launch_tn<128, 2>(g, splits, per_sm, timeout_ns, stream);
    case 256 * 4 + 2: return launch_tn<256, 2>(g, splits, per_sm, timeout_ns, stream);
    default: return -TCCL_ESIZE;
  }
}

// ------------------------------------------------------------------ which kernel, which shape
// A cost model in microseconds, fitted to 142 products (71 shapes from 1 to 1454 rows, inputs in L2 and not) timed with
// every configuration: the configuration it picks costs 2.3 % more than the best one on average.  Its terms are the limits
// that the profiles show: the latency of recycling a stage, L2 -> SM bandwidth of all CTAs together (about 13 TB/s), the
// tensor pipe, DRAM, and what the partials cost.
struct SkinnyChoice {
  int tn, cg, splits, per_sm;
  float us;
};
static float skinny_cost(int m, int n, int k, int tn, int cg, int splits, int per_sm) {
  const int num_kb = (k + 63) / 64, kb = (num_kb + splits - 1) / splits, cl = cg * splits;
  const float ctas = (float)((n + 128 * cg - 1) / (128 * cg)) * cg * ((m + tn - 1) / tn) * splits;
  // clusters of 8 and 4 do not fill every GPC
  const float slots = (cl == 8 ? 127.9f : (cl == 4 ? 136.f : 148.f)) * per_sm, act = ctas < slots ? ctas : slots;
  const float per = act > 148.f ? act / 148.f : 1.f, sb = 16384.f + tn / cg * 128;
  const float ns = floorf((per_sm == 2 ? 110.f : 222.f) * 1024.f / sb);
  const float flow = fmaxf(per * tn * 1.14e-3f, act * sb * (per_sm == 2 ? 7.4e-8f : 7.9e-8f));  // one k-block of all CTAs
  const float fill = fmaxf(0.f, kb - ns) * fmaxf(flow, 1.75f / ns) + fminf((float)kb, ns) * fmaxf(flow, 0.137f);
  const float rounds = ctas <= slots ? 1.f : (per_sm == 1 ? ceilf(ctas / slots) : ctas / slots + 0.13f);
  const float sms = rounds * (fill + 0.89f), dram = ((float)m * k + (float)n * k) * 2.f * 1.87e-7f;
  const float used = fminf(1.f, (float)((m + 31) / 32 * 32) / tn) * tn / 128.f;
  const float gather = tn == 16 ? 0.060f : (tn == 32 ? 0.166f : (tn == 64 ? 0.463f : (tn == 128 ? 1.287f : 3.578f)));
  const float part = 1.1f * used + (splits == 1 ? 0.f : 0.47f + gather);
  return 1.54f + sqrtf(sqrtf(sms * sms * sms * sms + dram * dram * dram * dram)) + part * rounds;
}
static float pair_cost(int m, int n, int k) {
  const int kb = (k + 63) / 64, tiles = ((m + 255) / 256) * ((n + 255) / 256);
  if (tiles <= 37) return 5.04f + kb * fmaxf(0.183f, 2 * tiles * 49152.f * 7.9e-8f);
  if (tiles <= 74) return 5.04f + kb * fmaxf(0.365f, tiles * 65536.f * 7.9e-8f);
  const float units = tiles / 74 + (tiles % 74 ? 0.5f * ((2 * (tiles % 74) + 73) / 74) : 0.f);
  return 5.04f + units * (kb * 0.383f + 0.26f);
}
// tn == 0: the pair kernel
static SkinnyChoice choose(int m, int n, int k) {
  SkinnyChoice best{0, 0, 0, 0, pair_cost(m, n, k)};
  for (const auto& t : kTiles) {
    if (t.tn >= 32 && t.tn >= 4 * m) continue;
    for (int splits = 1; splits * t.cg <= 8 && splits <= (k + 63) / 64; splits *= 2)
      for (int per_sm = 1; per_sm <= max_per_sm(t.tn); ++per_sm) {
        const float us = skinny_cost(m, n, k, t.tn, t.cg, splits, per_sm);
        if (us < best.us) best = SkinnyChoice{t.tn, t.cg, splits, per_sm, us};
      }
  }
  return best;
}

static bool too_many_tiles(int m, int n) {  // far beyond where a tile per CTA can win
  return (long long)m * n > 6144ll * 6144;
}

bool launch_gemm_skinny(const tccl_gemm_args* g, cudaStream_t stream, uint64_t timeout_ns, int* rc) {
  if (too_many_tiles(g->m, g->n)) return false;
  // a program multiplies a few shapes over and over: remember their choices (per thread, so without a lock)
  struct Entry { int m, n, k; SkinnyChoice c; };
  static thread_local Entry memo[64] = {};
  Entry& e = memo[((unsigned)g->m * 31u + (unsigned)g->n * 17u + (unsigned)g->k) % 64u];
  if (e.m != g->m || e.n != g->n || e.k != g->k) e = Entry{g->m, g->n, g->k, choose(g->m, g->n, g->k)};
  if (!e.c.tn) return false;
  *rc = launch_as(g, e.c.tn, e.c.cg, e.c.splits, e.c.per_sm, timeout_ns, stream);
  return true;
}

}  // namespace gemm2
}  // namespace tccl

extern "C" int tccl_gemm_choice(int m, int n, int k, tccl_few_rows* out) {
  using namespace tccl::gemm2;
  if (m <= 0 || n <= 0 || k <= 0) return -TCCL_EINVAL;
  const SkinnyChoice c = too_many_tiles(m, n) ? SkinnyChoice{} : choose(m, n, k);
  *out = tccl_few_rows{c.tn, c.cg, c.splits, c.per_sm};
  return 0;
}

extern "C" int tccl_gemm_few_rows(const tccl_gemm_args* g, const tccl_few_rows* f, void* stream) {
  using namespace tccl::gemm2;
  const int rc = check_gemm_args(g);
  if (rc) return rc;
  return launch_as(g, f->tokens, f->ctas, f->splits, f->per_sm, 2000000000ull, reinterpret_cast<cudaStream_t>(stream));
}
