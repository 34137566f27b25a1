// Dense bf16 GEMM on pairs of SMs: C[M,N] = A[M,K] * W[N,K]^T (+ epilogue), 256 x 256 tiles per cluster of two CTAs.
//
// Bound: the tensor cores, and what keeps them from their rate is operand traffic in shared memory.  With one CTA per 128 x 256 tile an SM reads 128 + 256
// operand rows for each 128 x 256 products; tcgen05.mma.cta_group::2 (M = 256) lets the two CTAs of a cluster each hold 128 rows of A and 128 rows of W, and
// both tensor cores take the whole 256 of W from the two halves: a third less to load and to store per product, and room for six stages.
//
//   warp 0     of each CTA: TMA loads of its own halves; all bytes of a stage are counted on the leader's barrier
//   warp 1     of the leader: tcgen05.mma from one thread; commits arrive on both CTAs' barriers
//   warps 2-5  of each CTA: its 128 rows from TMEM (two accumulators of 256 columns), epilogue as in gemm_tcgen05.cu
// No load is multicast.  Every mbarrier wait is bounded.
//
// Measured (B200, single calls, one-SM kernel -> this one): 4096 x 28672 x 4096 742 -> 675 us (1426 TFLOP/s, 0.88 of the measured cuBLAS burst), 5600 x 4096 x 14336
// 501 -> 439 (1498), 4096 x 5120 x 2880 138 -> 92; back to back under the power cap 4096 x 28672 x 4096 900 -> 839.
#include "act.cuh"
#include "common.cuh"
#include "host_util.h"

namespace mx {

constexpr int GP_BM = 128, GP_BN = 256, GP_BK = 64, GP_ST = 6;
constexpr int GP_A = GP_BM * GP_BK * 2, GP_B = (GP_BN / 2) * GP_BK * 2, GP_STAGE = GP_A + GP_B;
constexpr int GP_SMEM = GP_ST * GP_STAGE + 1024;

struct GemmPairParams {
  int M, N, K, m_tiles, n_tiles;       // tiles of 256 x 256
  void* C;
  int ldc, out_f32;
  const float* bias;
  const float* row_scale;
  int act;
  float act_alpha, act_limit;
  int* status;
};

__device__ __forceinline__ uint32_t cluster_rank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ uint32_t map_to_rank(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void pair_load_2d(uint32_t dst, const void* tmap, uint32_t bar, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
               ::"r"(dst), "l"(tmap), "r"(bar), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void pair_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}\n"
               ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void pair_commit(uint32_t bar) {              // the barrier at this offset in both CTAs
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"((uint16_t)3) : "memory");
}

// 32 columns of a row: bias, activation, scale, store
__device__ __forceinline__ void pair_store(const GemmPairParams& p, const uint32_t (&r)[32], int row, int col0, float rs) {
  float v[32];
#pragma unroll
  for (int j = 0; j < 32; ++j) {
    v[j] = __uint_as_float(r[j]);
    if (p.bias && col0 + j < p.N) v[j] += p.bias[col0 + j];
  }
  const bool gated = act_gated(p.act);
  int oc = col0, on = p.N, n = 32;
  if (gated) {                                                           // 16 gate columns, then their 16 up columns
    oc >>= 1; on >>= 1; n = 16;
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = glu_apply(p.act, v[j], v[16 + j], p.act_alpha, p.act_limit);
  } else if (p.act) {
    act_unary_run<false>(p.act, v, p.act_alpha, p.act_limit);
  }
#pragma unroll
  for (int j = 0; j < 32; ++j) v[j] *= rs;
  const size_t at = (size_t)row * p.ldc + oc;
  const bool whole = oc + n <= on && (p.ldc & 7) == 0 && (((uintptr_t)p.C) & 15) == 0;
  if (p.out_f32 == 1) {
    float* o = (float*)p.C + at;
    if (whole) {
#pragma unroll
      for (int j = 0; j < 32; j += 4)
        if (j < n) *reinterpret_cast<float4*>(o + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
    } else {
#pragma unroll
      for (int j = 0; j < 32; ++j)
        if (j < n && oc + j < on) o[j] = v[j];
    }
  } else {
    const bool h = p.out_f32 == 2;
    __nv_bfloat16* o = (__nv_bfloat16*)p.C + at;
    if (whole) {
#pragma unroll
      for (int j = 0; j < 32; j += 8)
        if (j < n)
          *reinterpret_cast<uint4*>(o + j) = h ? make_uint4(pack_f16(v[j], v[j + 1]), pack_f16(v[j + 2], v[j + 3]), pack_f16(v[j + 4], v[j + 5]), pack_f16(v[j + 6], v[j + 7]))
                                               : make_uint4(pack_bf16(v[j], v[j + 1]), pack_bf16(v[j + 2], v[j + 3]), pack_bf16(v[j + 4], v[j + 5]), pack_bf16(v[j + 6], v[j + 7]));
    } else {
#pragma unroll
      for (int j = 0; j < 32; ++j)
        if (j < n && oc + j < on) {
          if (h) ((__half*)o)[j] = __float2half(v[j]); else o[j] = __float2bfloat16(v[j]);
        }
    }
  }
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(192, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b, const GemmPairParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t s_bar[2 * GP_ST + 4];
  __shared__ uint32_t s_tmem;
  __shared__ int s_abort;
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;           // (the same offset in both CTAs)
  const uint32_t bar_full = smem_u32(s_bar), bar_empty = bar_full + 8 * GP_ST, bar_tfull = bar_empty + 8 * GP_ST, bar_tempty = bar_tfull + 16;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  volatile int* abort_flag = &s_abort;
  if (threadIdx.x == 0) {
    for (int s = 0; s < GP_ST; ++s) { mbar_init(bar_full + 8 * s, 1); mbar_init(bar_empty + 8 * s, 1); }
    for (int a = 0; a < 2; ++a) { mbar_init(bar_tfull + 8 * a, 1); mbar_init(bar_tempty + 8 * a, 8); }      // four warps of either CTA
    s_abort = 0;
    fence_mbar_init();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&s_tmem)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  cluster_sync_all();
  tc_fence_after();
  const uint32_t tmem = s_tmem;
  const int tiles = p.m_tiles * p.n_tiles, k_iters = (p.K + GP_BK - 1) / GP_BK;
  const int first = blockIdx.x >> 1, step = gridDim.x >> 1;
  // groups of four m-tiles: a wave of clusters shares a band of A and a band of W in L2
  auto coords = [&](int t, int& mt, int& nt) {
    const int per = 4 * p.n_tiles, g = t / per, r = t - g * per, gm = min(4, p.m_tiles - g * 4);
    mt = g * 4 + r % gm;
    nt = r / gm;
  };

  if (warp == 0) {
    if (lane == 0) {
      prefetch_tmap(&tmap_a); prefetch_tmap(&tmap_b);
      uint32_t s = 0, ph = 1;
      bool ok = true;
      for (int t = first; t < tiles && ok; t += step) {
        int mt, nt;
        coords(t, mt, nt);
        const int row = mt * 256 + (int)rank * GP_BM, col = nt * GP_BN + (int)rank * (GP_BN / 2);
        for (int k = 0; k < k_iters; ++k) {
          if (!(ok = mbar_wait(bar_empty + 8 * s, ph, p.status, ERR_MBAR_TIMEOUT_PRODUCER, abort_flag))) break;
          if (rank == 0) mbar_expect_tx(bar_full + 8 * s, 2 * GP_STAGE);
          const uint32_t full = map_to_rank(bar_full + 8 * s, 0), dst = base + s * GP_STAGE;
          pair_load_2d(dst, &tmap_a, full, k * GP_BK, row);
          pair_load_2d(dst + GP_A, &tmap_b, full, k * GP_BK, col);
          if (++s == GP_ST) { s = 0; ph ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0 && rank == 0) {
      constexpr uint32_t idesc = umma_idesc_bf16(256, GP_BN, 0, 0);
      uint32_t s = 0, ph = 0, n = 0;
      bool ok = true;
      for (int t = first; t < tiles && ok; t += step, ++n) {
        const uint32_t acc = n & 1;
        if (!(ok = mbar_wait(bar_tempty + 8 * acc, ((n >> 1) & 1) ^ 1, p.status, ERR_MBAR_TIMEOUT_MMA, abort_flag))) break;
        tc_fence_after();
        for (int k = 0; k < k_iters; ++k) {
          if (!(ok = mbar_wait(bar_full + 8 * s, ph, p.status, ERR_MBAR_TIMEOUT_MMA, abort_flag))) break;
          tc_fence_after();
          const uint64_t a = umma_desc_k_sw128(base + s * GP_STAGE), b = umma_desc_k_sw128(base + s * GP_STAGE + GP_A);
#pragma unroll
          for (int kk = 0; kk < GP_BK / 16; ++kk) pair_mma(tmem + acc * GP_BN, a + 2 * kk, b + 2 * kk, idesc, (k | kk) != 0);
          pair_commit(bar_empty + 8 * s);
          if (++s == GP_ST) { s = 0; ph ^= 1; }
        }
        if (ok) pair_commit(bar_tfull + 8 * acc);
      }
    }
  } else {
    const int q = warp & 3;
    uint32_t n = 0;
    bool ok = true;
    for (int t = first; t < tiles && ok; t += step, ++n) {
      int mt, nt;
      coords(t, mt, nt);
      const uint32_t acc = n & 1;
      if (!(ok = mbar_wait(bar_tfull + 8 * acc, (n >> 1) & 1, p.status, ERR_MBAR_TIMEOUT_EPILOGUE, abort_flag, 64))) break;
      tc_fence_after();
      const int row = mt * 256 + (int)rank * GP_BM + q * 32 + lane;
      const float rs = p.row_scale && row < p.M ? p.row_scale[row] : 1.f;
#pragma unroll 1
      for (int c0 = 0; c0 < GP_BN; c0 += 32) {
        uint32_t r[32];
        tmem_ld_32x32(tmem + ((uint32_t)(q * 32) << 16) + acc * GP_BN + c0, r);
        tmem_ld_wait();
        if (row < p.M && nt * GP_BN + c0 < p.N) pair_store(p, r, row, nt * GP_BN + c0, rs);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(map_to_rank(bar_tempty + 8 * acc, 0)) : "memory");
    }
  }
  if (*abort_flag)                               // a wait ran out: copies still in flight land before shared memory is released
    for (int i = 0; i < 200; ++i) __nanosleep(1000);
  tc_fence_before();
  __syncwarp();
  cluster_sync_all();                            // the pair's loads, products and arrivals use both CTAs' memory
  if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
}

}  // namespace mx

using namespace mx;

// C[M, N (/2 when gated)] = A[M,K] W[N,K]^T; K a multiple of 8, A and W dense with 16-byte aligned bases.  out_kind 0 bf16, 1 fp32, 2 fp16.
MX_HOST_API int mx_gemm_pair(const void* a, const void* w, void* c, int ldc, int out_kind, const float* bias, const float* row_scale, int act, float act_alpha,
                             float act_limit, int M, int N, int K, cudaStream_t st) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if (K % 8 || (((uintptr_t)a | (uintptr_t)w) & 15)) return -101;
  if (act_gated(act) && N % 32) return -104;
  GemmPairParams p{M, N, K, (M + 255) / 256, (N + GP_BN - 1) / GP_BN, c, ldc, out_kind, bias, row_scale, act, act_alpha, act_limit, status_word()};
  CUtensorMap ta, tb;
  uint64_t da[2] = {(uint64_t)K, (uint64_t)M}, db[2] = {(uint64_t)K, (uint64_t)N}, strides[1] = {(uint64_t)K * 2};
  uint32_t box[2] = {GP_BK, 128};
  int r = make_tmap_bf16(&ta, a, 2, da, strides, box, 1);
  if (!r) r = make_tmap_bf16(&tb, w, 2, db, strides, box, 1);
  if (r) return r;
  static std::atomic<int> clusters[64];
  const int dev = DeviceOnce::ordinal();
  int most = clusters[dev].load(std::memory_order_acquire);
  if (!most) {                                   // clusters that are resident at once (a GPC's odd SM has no partner)
    cudaError_t e = cudaFuncSetAttribute(gemm_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, GP_SMEM);
    if (e != cudaSuccess) return (int)e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(sm_count() / 2 * 2); cfg.blockDim = dim3(192); cfg.dynamicSmemBytes = GP_SMEM;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 2; at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at; cfg.numAttrs = 1;
    e = cudaOccupancyMaxActiveClusters(&most, gemm_pair_kernel, &cfg);
    if (e != cudaSuccess) return (int)e;
    if (most < 1) return -116;
    clusters[dev].store(most, std::memory_order_release);
  }
  const int tiles = p.m_tiles * p.n_tiles;
  gemm_pair_kernel<<<2 * (tiles < most ? tiles : most), 192, GP_SMEM, st>>>(ta, tb, p);
  return (int)cudaGetLastError();
}

