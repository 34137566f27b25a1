// Products of a few activation rows with a large weight matrix, bound by reading the weights: C[M][N] = A[M][K] W[N][K]^T for the rows of a
// decode batch (up to 64), and expert banks whose experts see a few dozen rows each.  Weights bf16 or Q8 (int8 codes, fp16 scale per 32).
//
// Why not tcgen05: at these sizes the tensor time is a small part of the memory time either way, and what counts is that every SM streams an
// equal share of the weights without a pause.  The tcgen05 kernel walks whole tiles (192 tiles of 32 columns on 148 SMs are two
// waves, the second nearly empty) with 128-row activation boxes of mostly padding, and int8 codes have to be widened into a second
// shared-memory tile by producer warps first, which bounded it at 1.5 TB/s.  Here
//   * the weights are the M side of mma.m16n8k16 and the activation rows its N side: 8 rows per column group, no padding to 128;
//   * one warp issues TMA boxes of 128 weight rows x 128 bytes (and the activation rows' matching columns) into a ring of NST
//     stages; four warps own 32 weight rows each and never wait for each other;
//   * int8 codes go from the swizzled tile through ldmatrix to registers and are widened to bf16 exactly (four instructions per pair); each
//     32-element block is summed on its own and scaled in fp32, so the weights are not rounded to bf16;
//   * up to 8 rows of bf16, where the GEMVs of fp32 additions are the alternative: the tensor cores cut a running sum off where an addition rounds (4096
//     x 4096, error against 64 bits 4.0e-7 that way, 0.87e-7 in the GEMV), so every instruction's 16 products are summed on their own, and the
//     sums are added in fp32 with the rounding errors carried along (0.72e-7, in the same time);
//   * the work is the list of (group of rows, 128 weight rows, K step) laid end to end, of which every CTA takes an equal run.  A
//     tile that is cut leaves fp32 partials (at most two per CTA); the warp that arrives last adds them in the order of the CTAs.
// A gated pair (16 gate rows, then 16 up rows) lies in one lane's accumulators.
//
// Measured (B200, cold caches, before -> now): bf16 40 x 6144 x 4096 33.6 -> 20.8 us, 16 x 28672 x 4096 71 -> 58 (a bare stream of those weights through
// the same ring takes 53: what is left is the launch, the partials of cut tiles and the epilogue); Q8 16 x 28672 x 4096 100 -> 47, 512 experts of
// Q8 1024 x 2048 and 2048 x 512 with 19.5 rows each 1181 -> 823 (there the widening of the codes bounds it; looking up every tile of a run, instead of
// stepping from one to the next, took 56 us of it).
//
// Bank conflicts: weight and activation tiles have the 128-byte TMA swizzle, ldmatrix rows differ in their low three bits.  With int8 codes a lane
// holds four consecutive k, so its activations are 8-byte loads; column g of a group is row 2 (g & 3) + g / 4 of it, which spreads the
// half-warp's rows over all banks.
#include "act.cuh"
#include "common.cuh"
#include "host_util.h"

#include <type_traits>

namespace mx {

constexpr int GR_ROWS = 128;             // weight rows per tile
constexpr int GR_WARPS = 4;
constexpr int GR_MAX_ENTRIES = 1024;     // groups of activation rows of a launch
constexpr int GR_MAX_GRID = 512;
static_assert(GR_MAX_GRID * GR_WARPS <= CUT_TICKETS, "a counter per warp");

struct GemmRowsParams {
  int M, N, K, n_tiles, k_steps, chunk;  // chunk: activation rows per group (at most 8 NT)
  void* C;
  int ldc, out_f32;
  const float* bias;                     // [N] or [E][N]
  const float* row_scale;                // [M]
  int act;
  float act_alpha, act_limit;
  const int* tile_expert;                // grouped: expert and live rows of every 128-row tile of A, number of tiles
  const int* tile_valid;
  const int* num_tiles;
  int max_tiles, max_valid;              // tiles of more live rows than max_valid are left out
  float* part;                           // [grid][2][warp][2 NT][32] float4
  int* tickets;                          // [grid][warp]
  int* status;
};

__device__ __forceinline__ void gr_ldsm4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void gr_ldsm2(uint32_t& r0, uint32_t& r1, uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0, %1}, [%2];" : "=r"(r0), "=r"(r1) : "r"(addr) : "memory");
}
__device__ __forceinline__ void gr_mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void gr_mma_zero(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
               : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}
// signed bytes 0, 1 (SEL 0x4140) or 2, 3 (0x4342) of w as bf16, exactly: the low seven bits above 128, minus 128 or 256
template <int SEL> __device__ __forceinline__ uint32_t gr_s8_pair(uint32_t w) {
  const uint32_t t = __byte_perm(w, 0, SEL);
  const uint32_t x = (t & 0x007f007fu) | 0x43004300u, y = (t & 0x00800080u) | 0x43004300u;
  const __nv_bfloat162 d = __hsub2(*reinterpret_cast<const __nv_bfloat162*>(&x), *reinterpret_cast<const __nv_bfloat162*>(&y));
  return *reinterpret_cast<const uint32_t*>(&d);
}
// sum += v, with what the rounded sums before it have lost
__device__ __forceinline__ void add_exact(float& sum, float& lost, float v) {
  const float y = v - lost, r = sum + y, e = (r - sum) - y;
  lost = fabsf(e) < INFINITY ? e : 0.f;                      // (an infinite sum stays one)
  sum = r;
}
__device__ __forceinline__ uint32_t gr_lds32(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ uint2 gr_lds64(uint32_t addr) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr) : "memory");
  return v;
}

template <bool Q8, int NT> struct GemmRowsShape {
  static constexpr int KS = Q8 ? 128 : 64;                   // K per stage: 128 bytes of a weight row
  static constexpr int W_BYTES = GR_ROWS * 128;
  static constexpr int X_BOX = NT * 8 * 128;                 // 64 columns of the activation rows
  static constexpr int X_BYTES = X_BOX * (Q8 ? 2 : 1);
  static constexpr int D_BYTES = Q8 ? GR_ROWS * 16 : 0;      // eight scales of a row: two steps' worth, since a box row is 16 bytes at least
  static constexpr int STAGE = W_BYTES + X_BYTES + D_BYTES;
  // int8 codes: widening them takes most of the issue slots, and two warps per scheduler leave many of them empty.  Up to two column groups, two
  // warps share 32 rows, each the half of every step (64 k): 2 rows x 32768 x 4096 50 -> 46 us; more accumulators do not fit 96 registers (40 rows: 71 -> 84)
  static constexpr int SPLIT = Q8 && NT <= 2 ? 2 : 1;
  static constexpr int WARPS = GR_WARPS * SPLIT;
  static constexpr int XCH = SPLIT == 2 ? GR_WARPS * 2 * NT * 512 : 0;                        // accumulators handed from the second warp of a pair to the first
  static constexpr int NST = (106 * 1024 - XCH) / STAGE < 8 ? (106 * 1024 - XCH) / STAGE : 8;     // two CTAs per SM
  static constexpr int SMEM = NST * STAGE + XCH + 1024;
};

// Units of work per CTA.  An equal share each, but cutting a tile into ever shorter runs costs the last warp the partials' read: about NT / 15 of a step's
// time per part, so runs are at least sqrt(steps NT / 15) long; and no CTA lies without a step between two others.
__host__ __device__ inline int rows_run(int total, int grid, int steps_nt, int cost) {
  int per = (total - 1) / grid + 1;
  if (per < cost) per = cost;
  while ((long long)per * per * 15 < steps_nt) ++per;
  return per;
}
__host__ __device__ inline int rows_cost(bool weighted, int rows) { return weighted ? 5 + 2 * ((rows + 7) / 8) : 1; }

template <bool Q8, int NT>
__global__ void __launch_bounds__(GemmRowsShape<Q8, NT>::WARPS * 32 + 32, 2) gemm_rows_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_x,
                                                                          const __grid_constant__ CUtensorMap tm_d, const GemmRowsParams p) {
  using S = GemmRowsShape<Q8, NT>;
  constexpr int NST = S::NST;
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t s_bar[2 * NST + 2 * GR_WARPS];
  __shared__ int s_abort;
  __shared__ int s_pre[GR_MAX_ENTRIES + 1];                  // grouped: groups of rows before tile i
  __shared__ uint8_t s_valid[GR_MAX_ENTRIES];                // and its live rows
  __shared__ int s_sum[S::WARPS + 1];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t bar_full = smem_u32(s_bar), bar_empty = bar_full + 8 * NST, bar_xch = bar_empty + 8 * NST;
  pdl_launch_dependents();
  if (tid == 0) {
    for (int s = 0; s < NST; ++s) {
      mbar_init(bar_full + 8 * s, 1);
      mbar_init(bar_empty + 8 * s, S::WARPS);
    }
    for (int s = 0; s < 2 * GR_WARPS; ++s) mbar_init(bar_xch + 8 * s, 1);
    s_abort = 0;
    fence_mbar_init();
  }
  __syncthreads();
  volatile int* abort_flag = &s_abort;
  const bool grouped = p.tile_expert != nullptr;

  // ---- the list of work: groups of activation rows x weight tiles x K steps.  A step of a group costs `cost` units: with int8 codes the
  // instructions grow with the live column groups (about 5 + 2 per group), bf16 steps are bound by their bytes.
  auto cost = [&](int rows) { return rows_cost(Q8 && grouped, rows); };
  int units = 1, live_tiles = 0;
  if (grouped) {
    pdl_wait();
    live_tiles = min(min(*p.num_tiles, p.max_tiles), GR_MAX_ENTRIES);
    int run = 0;
    for (int i0 = 0; i0 < live_tiles; i0 += S::WARPS * 32 + 32) {
      const int i = i0 + tid;
      int valid = i < live_tiles ? p.tile_valid[i] : 0;
      if (valid > p.max_valid) valid = 0;
      if (i < live_tiles) s_valid[i] = (uint8_t)valid;
      int incl = valid / p.chunk * cost(p.chunk) + (valid % p.chunk ? cost(valid % p.chunk) : 0);
      const int own = incl;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += u;
      }
      if (lane == 31) s_sum[warp] = incl;
      __syncthreads();
      int before = run;
#pragma unroll
      for (int w = 0; w <= S::WARPS; ++w) {
        if (w < warp) before += s_sum[w];
        run += s_sum[w];
      }
      if (i < live_tiles) s_pre[i] = before + incl - own;
      __syncthreads();
    }
    units = run;
    if (tid == 0) s_pre[live_tiles] = run;
    __syncthreads();
  }
  const int steps_of = p.n_tiles * p.k_steps, total = units * steps_of;       // (of one unit of cost)
  const int per = rows_run(total, (int)gridDim.x, p.k_steps * NT, cost(p.chunk));
  const int my0 = min(total, (int)blockIdx.x * per), my1 = min(total, my0 + per);

  // A run is walked step by step: position `at` (in units of cost) of the step's start.  A step belongs to the CTA in whose run it starts.
  struct Place { int e, row0, rows, nt, cost, start, k; };   // start: position of the tile's first step; k: step
  auto advance = [&](Place& r) {                             // the next tile's first step (past the list: its start is `total`)
    r.start += p.k_steps * r.cost;
    r.k = 0;
    if (++r.nt < p.n_tiles || !grouped) return;
    r.nt = 0;
    int i = r.row0 >> 7;
    if ((r.row0 & 127) + p.chunk < s_valid[i]) {
      r.row0 += p.chunk;
    } else {
      do ++i; while (i < live_tiles && !s_valid[i]);
      r.row0 = i * 128;
      r.e = i < live_tiles ? p.tile_expert[i] : 0;
    }
    r.rows = i < live_tiles ? min(p.chunk, s_valid[i] - (r.row0 & 127)) : 1;
    r.cost = cost(r.rows);
  };
  auto place = [&](int pos) {                                // the first step that starts at or after pos (< total)
    Place r;
    r.e = 0; r.row0 = 0; r.rows = p.M; r.cost = 1;
    int base_pos = 0;
    if (grouped) {
      const int g = pos / steps_of;                          // cost units before: the tile of A with s_pre <= g
      int lo = 0, hi = live_tiles - 1;                       // (the last one: tiles left out start where the next tile does)
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (s_pre[mid] <= g) lo = mid; else hi = mid - 1;
      }
      const int full = cost(p.chunk), c = (pos - s_pre[lo] * steps_of) / (full * steps_of);
      r.rows = min(p.chunk, s_valid[lo] - c * p.chunk);
      r.cost = cost(r.rows);
      r.e = p.tile_expert[lo];
      r.row0 = lo * 128 + c * p.chunk;
      base_pos = s_pre[lo] * steps_of + c * full * steps_of;
    }
    const int i = (pos - base_pos + r.cost - 1) / r.cost;
    r.nt = i / p.k_steps;
    r.k = i - r.nt * p.k_steps;
    if (r.nt == p.n_tiles) { --r.nt; r.k = p.k_steps; }      // between the last step of a group and the next group
    r.start = base_pos + r.nt * p.k_steps * r.cost;
    if (r.k == p.k_steps) advance(r);
    return r;
  };

  if (warp == S::WARPS) {
    // ------------------------------------------------ TMA producer
    if (lane == 0 && my0 < my1) {
      prefetch_tmap(&tm_w); prefetch_tmap(&tm_x);
      if (Q8) prefetch_tmap(&tm_d);
      auto load_w = [&](int s, const Place& at) {
        const uint32_t st = base + s * S::STAGE;
        mbar_expect_tx(bar_full + 8 * s, S::STAGE);
        tma_load_3d(st, &tm_w, bar_full + 8 * s, at.k * 64, at.nt * GR_ROWS, at.e);    // (64 two-byte elements: 128 bytes)
        if (Q8) tma_load_3d(st + S::W_BYTES + S::X_BYTES, &tm_d, bar_full + 8 * s, (at.k >> 1) * 8, at.nt * GR_ROWS, at.e);
      };
      auto load_x = [&](int s, const Place& at) {
        const uint32_t st = base + s * S::STAGE + S::W_BYTES;
        tma_load_2d(st, &tm_x, bar_full + 8 * s, at.k * S::KS, at.row0);
        if (Q8) tma_load_2d(st + S::X_BOX, &tm_x, bar_full + 8 * s, at.k * S::KS + 64, at.row0);
      };
      auto next = [&](Place& at) {                           // (false: past the run)
        if (at.start + (at.k + 1) * at.cost >= my1) return false;
        if (++at.k == p.k_steps) advance(at);
        return true;
      };
      Place at = place(my0);
      bool more = at.start + at.k * at.cost < my1;
      int ahead = 0;
      if (!grouped) {
        // dense: the weights of the first stages are on their way before the previous kernel has finished
        for (Place w = at; more && ahead < NST; ++ahead) {
          load_w(ahead, w);
          if (!next(w)) { ++ahead; break; }
        }
        pdl_wait();
      }
      uint32_t s = 0, ph = 1;
      for (int i = 0; more; ++i) {
        if (i >= ahead) {
          if (!mbar_wait(bar_empty + 8 * s, ph, p.status, ERR_MBAR_TIMEOUT_PRODUCER, abort_flag)) break;
          load_w(s, at);
        }
        load_x(s, at);
        if (++s == NST) { s = 0; ph ^= 1; }
        more = next(at);
      }
    }
  } else {
    // ------------------------------------------------ four warps (or pairs) of 32 weight rows
    if (!grouped) pdl_wait();
    const int g = lane >> 2, t4 = lane & 3, wr = warp % GR_WARPS, kh = warp / GR_WARPS;      // kh: which half of a step's k
    uint32_t xch_ph = 0;
    const uint32_t lrow = (lane & 7) + ((lane >> 3) & 1) * 8, lchunk = lane >> 4;
    const int xg = ((g & 3) << 1) | (g >> 2);                // Q8: the row of a column group that is column g
    uint32_t wo[4], xo[4];                                   // swizzled offsets of a lane's reads in a tile: the same in every step
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      wo[i] = (wr * 32 + lrow) * 128 + (((2 * i + lchunk) ^ (lrow & 7)) << 4);
      xo[i] = S::W_BYTES + kh * S::X_BOX + (Q8 ? xg * 128 + (((2 * i + (t4 >> 1)) ^ xg) << 4) + (t4 & 1) * 8
                               : (lane & 7) * 128 + (((2 * i + ((lane >> 3) & 1)) ^ (lane & 7)) << 4));
    }
    uint32_t s = 0, ph = 0;
    bool ok = true;
    Place at;
    at.start = total; at.k = at.cost = 0;
    if (my0 < my1) at = place(my0);
    for (; ok && at.start + at.k * at.cost < my1; advance(at)) {
      const int first = at.k, n = min((my1 - at.start + at.cost - 1) / at.cost, p.k_steps) - first;      // steps that start before the run's end
      const int nt_live = (at.rows + 7) / 8;
      float acc[2][NT][4];
#pragma unroll
      for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
          for (int i = 0; i < 4; ++i) acc[m][j][i] = 0.f;
      float lost[2][4] = {};                                 // (bf16, NT = 1)
      // the K steps, over NL live column groups: a count the compiler knows, so that a step is one straight run of instructions
      auto steps = [&](auto live) {
        constexpr int NL = decltype(live)::value;
        for (int k = 0; k < n; ++k) {
          if (!(ok = mbar_wait(bar_full + 8 * s, ph, p.status, ERR_MBAR_TIMEOUT_MMA, abort_flag))) break;
          const uint32_t st = base + s * S::STAGE;
          if constexpr (!Q8) {
            float sum[2][2][4];                              // (NT = 1)
  #pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
              uint32_t a[2][4], b[NL][2];
  #pragma unroll
              for (int m = 0; m < 2; ++m) gr_ldsm4(a[m], st + wo[kk] + m * 2048);
  #pragma unroll
              for (int j = 0; j + 1 < NL; j += 2) {
                uint32_t r[4];
                gr_ldsm4(r, st + xo[kk] + (lane >> 4) * 1024 + j * 1024);
                b[j][0] = r[0]; b[j][1] = r[1]; b[j + 1][0] = r[2]; b[j + 1][1] = r[3];
              }
              if constexpr (NL & 1) gr_ldsm2(b[NL - 1][0], b[NL - 1][1], st + xo[kk] + (NL - 1) * 1024);
  #pragma unroll
              for (int m = 0; m < 2; ++m)
  #pragma unroll
                for (int j = 0; j < NL; ++j) {
                  if constexpr (NT > 1) {
                    gr_mma(acc[m][j], a[m], b[j][0], b[j][1]);
                  } else {                                   // 16 products on their own; the four of a step meet in pairs
                    float t[4];
                    gr_mma_zero(t, a[m], b[j][0], b[j][1]);
  #pragma unroll
                    for (int i = 0; i < 4; ++i) sum[m][kk >> 1][i] = kk & 1 ? sum[m][kk >> 1][i] + t[i] : t[i];
                  }
                }
            }
            if constexpr (NT == 1) {                         // and join the running sum, whose rounding errors are carried along
  #pragma unroll
              for (int m = 0; m < 2; ++m)
  #pragma unroll
                for (int i = 0; i < 4; ++i) add_exact(acc[m][0][i], lost[m][i], sum[m][0][i] + sum[m][1][i]);
            }
          } else {
            uint32_t sd = st + S::W_BYTES + S::X_BYTES + (wr * 32 + g) * 16 + ((first + k) & 1) * 8 + kh * 4, sx = st;
#pragma unroll 1
            for (int half = kh; half < (S::SPLIT == 2 ? kh + 1 : 2); ++half, sd += 4, sx += S::X_BOX) {       // of 64: a run of code short enough for the instruction cache
              float2 d[2][2];                                // scales of the lane's rows, two blocks each
#pragma unroll
              for (int m = 0; m < 2; ++m)
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                  const uint32_t v = gr_lds32(sd + (m * 16 + i * 8) * 16);
                  d[m][i] = __half22float2(*reinterpret_cast<const __half2*>(&v));
                }
#pragma unroll
              for (int q = 0; q < 2; ++q) {                    // blocks of 32
                uint2 b[NL][2];
  #pragma unroll
                for (int j = 0; j < NL; ++j)
  #pragma unroll
                  for (int h = 0; h < 2; ++h) b[j][h] = gr_lds64(sx + xo[2 * q + h] + j * 1024);
  #pragma unroll
                for (int m = 0; m < 2; ++m) {
                  uint32_t w[4];
                  gr_ldsm4(w, st + (half ? wo[2 + q] : wo[q]) + m * 2048);
                  const uint32_t a0[4] = {gr_s8_pair<0x4140>(w[0]), gr_s8_pair<0x4140>(w[1]), gr_s8_pair<0x4342>(w[0]), gr_s8_pair<0x4342>(w[1])};
                  const uint32_t a1[4] = {gr_s8_pair<0x4140>(w[2]), gr_s8_pair<0x4140>(w[3]), gr_s8_pair<0x4342>(w[2]), gr_s8_pair<0x4342>(w[3])};
                  const float d0 = q ? d[m][0].y : d[m][0].x, d1 = q ? d[m][1].y : d[m][1].x;
  #pragma unroll
                  for (int j = 0; j < NL; ++j) {
                    float t[4];
                    gr_mma_zero(t, a0, b[j][0].x, b[j][0].y);
                    gr_mma(t, a1, b[j][1].x, b[j][1].y);
                    acc[m][j][0] = fmaf(t[0], d0, acc[m][j][0]); acc[m][j][1] = fmaf(t[1], d0, acc[m][j][1]);
                    acc[m][j][2] = fmaf(t[2], d1, acc[m][j][2]); acc[m][j][3] = fmaf(t[3], d1, acc[m][j][3]);
                  }
                }
              }
            }
          }
          __syncwarp();
          if (lane == 0) mbar_arrive(bar_empty + 8 * s);
          if (++s == NST) { s = 0; ph ^= 1; }
        }
      };
      if constexpr (NT <= 4) {                               // groups of a bank's rows are often short
        if (NT > 3 && nt_live == 3) steps(std::integral_constant<int, NT < 3 ? NT : 3>());
        else if (NT > 2 && nt_live == 2) steps(std::integral_constant<int, NT < 2 ? NT : 2>());
        else if (NT > 1 && nt_live == 1) steps(std::integral_constant<int, 1>());
        else steps(std::integral_constant<int, NT>());
      } else {
        steps(std::integral_constant<int, NT>());
      }
      if (!ok) break;

      if constexpr (S::SPLIT == 2) {                         // the second warp's half of the sums
        const uint32_t full = bar_xch + 8 * wr, empty = full + 8 * GR_WARPS;
        float4* box = reinterpret_cast<float4*>(smem_raw + (base - smem_u32(smem_raw)) + NST * S::STAGE) + wr * (2 * NT * 32) + lane;
        if (kh) {
          if (!(ok = mbar_wait(empty, xch_ph ^ 1, p.status, ERR_MBAR_TIMEOUT_MMA, abort_flag))) break;
#pragma unroll
          for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int j = 0; j < NT; ++j)
              if (j < nt_live) box[(m * NT + j) * 32] = make_float4(acc[m][j][0], acc[m][j][1], acc[m][j][2], acc[m][j][3]);
          __syncwarp();
          if (lane == 0) mbar_arrive(full);
          xch_ph ^= 1;
          continue;
        }
        if (!(ok = mbar_wait(full, xch_ph, p.status, ERR_MBAR_TIMEOUT_MMA, abort_flag))) break;
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
          for (int j = 0; j < NT; ++j)
            if (j < nt_live) {
              const float4 v = box[(m * NT + j) * 32];
              acc[m][j][0] += v.x; acc[m][j][1] += v.y; acc[m][j][2] += v.z; acc[m][j][3] += v.w;
            }
        __syncwarp();
        if (lane == 0) mbar_arrive(empty);
        xch_ph ^= 1;
      }

      // ---- a cut tile: partials, and the last warp to arrive adds them up
      if (n < p.k_steps) {
        const int c0 = at.start / per, c1 = (at.start + (p.k_steps - 1) * at.cost) / per;
        float4* part = reinterpret_cast<float4*>(p.part);
        auto slab = [&](int c) { return part + (((size_t)c * 2 + (c == c0 ? 1 : 0)) * GR_WARPS + wr) * (2 * NT * 32) + lane; };
        float4* mine = slab(blockIdx.x);
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
          for (int j = 0; j < NT; ++j)
            if (j < nt_live) mine[(m * NT + j) * 32] = make_float4(acc[m][j][0], acc[m][j][1], acc[m][j][2], acc[m][j][3]);
        __threadfence();
        __syncwarp();
        int prev = 0;
        if (lane == 0) {
          prev = atomicAdd(p.tickets + c0 * GR_WARPS + wr, 1);
          if (prev == c1 - c0) p.tickets[c0 * GR_WARPS + wr] = 0;
        }
        prev = __shfl_sync(0xffffffffu, prev, 0);
        if (prev != c1 - c0) continue;
        __threadfence();
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
          for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[m][j][i] = lost[m][i] = 0.f;
        if constexpr (!Q8 && NT == 1) {                        // four parts at a time, in pairs
          for (int c = c0; c <= c1; c += 4) {
            float4 v[4][2];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
              for (int m = 0; m < 2; ++m) v[i][m] = c + i <= c1 ? __ldcg(slab(c + i) + m * 32) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int m = 0; m < 2; ++m) {
              add_exact(acc[m][0][0], lost[m][0], (v[0][m].x + v[1][m].x) + (v[2][m].x + v[3][m].x));
              add_exact(acc[m][0][1], lost[m][1], (v[0][m].y + v[1][m].y) + (v[2][m].y + v[3][m].y));
              add_exact(acc[m][0][2], lost[m][2], (v[0][m].z + v[1][m].z) + (v[2][m].z + v[3][m].z));
              add_exact(acc[m][0][3], lost[m][3], (v[0][m].w + v[1][m].w) + (v[2][m].w + v[3][m].w));
            }
          }
        } else {
          for (int c = c0; c <= c1; ++c) {
            const float4* src = slab(c);
#pragma unroll
            for (int m = 0; m < 2; ++m)
#pragma unroll
              for (int j = 0; j < NT; ++j)
                if (j < nt_live) {
                  const float4 v = __ldcg(src + (m * NT + j) * 32);
                  acc[m][j][0] += v.x; acc[m][j][1] += v.y; acc[m][j][2] += v.z; acc[m][j][3] += v.w;
                }
          }
        }
      }

      // ---- epilogue: a lane holds weight rows g, g + 8 (and 16 further: the up rows of a gated pair) of columns 2 t4, 2 t4 + 1
      const int n0 = at.nt * GR_ROWS + wr * 32;
      const bool gated = act_gated(p.act);
      const float* bias = p.bias ? p.bias + (size_t)at.e * p.N : nullptr;
      const int on = gated ? p.N >> 1 : p.N;
      float bv[2][2];
#pragma unroll
      for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int r = n0 + m * 16 + i * 8 + g;
          bv[m][i] = bias && r < p.N ? bias[r] : 0.f;
        }
#pragma unroll
      for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int cj = 0; cj < 2; ++cj) {
          const int col = 2 * t4 + cj, t = j * 8 + (Q8 ? ((col & 3) << 1 | col >> 2) : col);
          if (t >= at.rows) continue;
          const int row = at.row0 + t;
          const float rs = p.row_scale ? p.row_scale[row] : 1.f;
#pragma unroll
          for (int m = 0; m < 2; ++m) {
            if (gated && m) continue;
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              float v = acc[m][j][2 * i + cj] + bv[m][i];
              int oc;
              if (gated) {
                v = glu_apply(p.act, v, acc[1][j][2 * i + cj] + bv[1][i], p.act_alpha, p.act_limit);
                oc = (n0 >> 1) + i * 8 + g;
              } else {
                if (p.act) v = act_unary<false>(p.act, v, p.act_alpha, p.act_limit);
                oc = n0 + m * 16 + i * 8 + g;
              }
              if (oc >= on) continue;
              v *= rs;
              const size_t o = (size_t)row * p.ldc + oc;
              if (p.out_f32 == 1) ((float*)p.C)[o] = v;
              else if (p.out_f32 == 2) ((__half*)p.C)[o] = __float2half(v);
              else ((__nv_bfloat16*)p.C)[o] = __float2bfloat16(v);
            }
          }
        }
    }
  }
  if (s_abort)                                               // a wait ran out: copies still in flight land before shared memory is released
    for (int i = 0; i < 200; ++i) __nanosleep(1000);
  __syncthreads();
}

template <bool Q8, int NT> static int launch_rows(const CUtensorMap& tw, const CUtensorMap& tx, const CUtensorMap& td, const GemmRowsParams& p, cudaStream_t st) {
  using S = GemmRowsShape<Q8, NT>;
  auto kern = gemm_rows_kernel<Q8, NT>;
  static DeviceOnce configured;
  if (configured.pending()) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, S::SMEM);
    if (e != cudaSuccess) return (int)e;
    configured.mark();
  }
  const int grid = 2 * sm_count() < GR_MAX_GRID ? 2 * sm_count() : GR_MAX_GRID;
  launch_pdl(kern, dim3(grid), dim3(S::WARPS * 32 + 32), S::SMEM, st, tw, tx, td, p);
  return (int)cudaGetLastError();
}

}  // namespace mx

using namespace mx;

// Column groups of 8 activation rows of an instance that holds `rows`.
static int rows_nt(int rows) { return rows <= 48 ? (rows + 7) / 8 : 8; }

// Floats of scratch (16-byte aligned) for mx_gemm_rows with groups of up to `rows` activation rows; 0: not taken.
MX_HOST_API int mx_gemm_rows_scratch(int rows) {
  if (rows < 1 || rows > 64) return 0;
  return GR_MAX_GRID * 2 * GR_ROWS * 8 * rows_nt(rows);
}

// Whether mx_gemm_rows takes a bank of experts: its kernel counts the tiles in shared memory and the work in 32 bits.
MX_HOST_API int mx_gemm_rows_takes(int wfmt, int max_tiles, int chunk, int N, int K) {
  if (chunk < 1 || chunk > 64 || max_tiles > GR_MAX_ENTRIES) return 0;
  const long long units = (128 + chunk - 1) / chunk * rows_cost(wfmt == WF_Q8, chunk);
  const int ks = wfmt == WF_Q8 ? 128 : 64;
  return units * max_tiles * ((N + GR_ROWS - 1) / GR_ROWS) * ((K + ks - 1) / ks) < 1ll << 30;
}
MX_HOST_API int mx_gemm_rows_run(int total, int grid, int steps_nt, int cost) { return rows_run(total, grid, steps_nt, cost); }

// C[M, N (/2 when gated)] = A[M,K] W[(E,) N, K]^T (+ bias, activation, row scale).  wfmt bf16 or Q8 (w1: scales, rows padded to 16 bytes).  Dense: M <= 64 and
// tile_expert null.  Grouped: A is packed in 128-row tiles (tile_expert, tile_valid, num_tiles on the device, at most max_tiles of them: mx_gemm_rows_takes), taken in
// groups of `chunk` rows; rows past a tile's live ones, and tiles of more than max_valid of them, are not written.  tickets: see host_util.h.  out_kind 0 bf16, 1 fp32, 2 fp16.
MX_HOST_API int mx_gemm_rows(const void* a, int wfmt, const void* w0, const void* w1, int n_experts, void* c, int ldc, int out_kind, const float* bias,
                             const float* row_scale, int act, float act_alpha, float act_limit, int M, int N, int K, const int* tile_expert,
                             const int* tile_valid, const int* num_tiles, int max_tiles, int max_valid, int chunk, float* scratch,
                             int* tickets, cudaStream_t st) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  const bool q8 = wfmt == WF_Q8;
  if ((!q8 && wfmt != WF_BF16) || K % 8 || (q8 && K % 32)) return -101;
  if (act_gated(act) && N % 32) return -104;
  if (chunk < 1 || chunk > 64 || (tile_expert ? (!mx_gemm_rows_takes(wfmt, max_tiles, chunk, N, K) || !tile_valid || !num_tiles || row_scale) : M > chunk)) return -106;
  if (((uintptr_t)a | (uintptr_t)w0 | (uintptr_t)w1 | (uintptr_t)scratch) & 15) return -114;
  const int nt = rows_nt(chunk), ks = q8 ? 128 : 64;
  GemmRowsParams p;
  p.M = M; p.N = N; p.K = K; p.n_tiles = (N + GR_ROWS - 1) / GR_ROWS; p.k_steps = (K + ks - 1) / ks; p.chunk = chunk;
  p.C = c; p.ldc = ldc; p.out_f32 = out_kind; p.bias = bias; p.row_scale = row_scale; p.act = act; p.act_alpha = act_alpha; p.act_limit = act_limit;
  p.tile_expert = tile_expert; p.tile_valid = tile_valid; p.num_tiles = num_tiles; p.max_tiles = max_tiles; p.max_valid = max_valid; p.part = scratch; p.status = status_word();
  p.tickets = tickets;
  CUtensorMap tw, tx, td;
  {
    // int8 codes travel as two-byte elements: the tile is bytes either way
    const uint64_t row = q8 ? (uint64_t)K : (uint64_t)K * 2;
    uint64_t dims[3] = {row / 2, (uint64_t)N, (uint64_t)n_experts}, strides[2] = {row, row * (uint64_t)N};
    uint32_t box[3] = {64, GR_ROWS, 1};
    int r = make_tmap_bf16(&tw, w0, 3, dims, strides, box, 1);
    if (r) return r;
  }
  {
    uint64_t dims[2] = {(uint64_t)K, (uint64_t)M}, strides[1] = {(uint64_t)K * 2};
    uint32_t box[2] = {64, (uint32_t)(8 * nt)};
    int r = make_tmap_bf16(&tx, a, 2, dims, strides, box, 1);
    if (r) return r;
  }
  td = tx;
  if (q8) {
    const uint64_t row = ((uint64_t)(K / 32) * 2 + 15) / 16 * 16;
    uint64_t dims[3] = {row / 2, (uint64_t)N, (uint64_t)n_experts}, strides[2] = {row, row * (uint64_t)N};
    uint32_t box[3] = {8, GR_ROWS, 1};
    int r = make_tmap_bf16(&td, w1, 3, dims, strides, box, 0);
    if (r) return r;
  }
#define MX_GR(NT_) case NT_: return q8 ? launch_rows<true, NT_>(tw, tx, td, p, st) : launch_rows<false, NT_>(tw, tx, td, p, st)
  switch (nt) {
    MX_GR(1); MX_GR(2); MX_GR(3); MX_GR(4); MX_GR(5); MX_GR(6); MX_GR(8);
    default: return -106;
  }
#undef MX_GR
}
