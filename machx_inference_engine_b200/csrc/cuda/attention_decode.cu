// Paged decode attention on the tensor cores: few query tokens per sequence (decode steps, speculative verification, short tails of prompts)
// against a bf16 or int8 cache, head dimensions 64 / 128 / 256.
//
// Bound: the cache is read once, so the target is the memory rate, and what keeps a kernel from it is (a) loads that wait for arithmetic and
// (b) ragged batches, where the longest sequence is walked by one CTA while the rest of the chip is idle.
//   (a) The query heads of a KV head are the 8-wide N side of mma.m16n8k16 and the keys (or, for P V, the value columns) its M side, so a
//       group of 4 or 8 heads needs no padded rows.  A warp owns steps of 16 or 32 keys and its own ring of cp.async stages: three steps
//       (24 to 48 KB per warp) are in flight and no CTA barrier lies in the key loop.
//   (b) Work is the list of 64-key tiles of all (sequence, query tile, KV head) groups laid end to end, and every CTA takes an equal run of
//       it, so a group may be cut anywhere.  A CTA has at most two cut groups, its first and its last: the scratch is two partials per CTA,
//       whatever the batch.  The CTA that arrives last at a cut group's ticket merges its partials.
//
// Precision: products of bf16 (or int8, exact in bf16) operands with fp32 sums, scores scaled in fp32.  The probabilities stay fp32: they
// enter P V as the sum of three bf16 terms (8 + 8 + 8 mantissa bits), which costs three instructions where the memory rate leaves room for ten.
// An int8 cache is read as it is: its key scales multiply the scores, its value scales the probabilities, in fp32.
//
// Measured (B200, with the CUDA-core kernel of attention.cu before it): 64 sequences of 256 to 4096 keys, 64 / 8 heads of 64: 460 -> 70 us (4.1 TB/s,
// 0.62 of the measured copy rate); 4 sequences of 16000 to 32000 keys, 32 / 8 heads of 128: 410 -> 74 us (5.3 TB/s, 0.82).
#include "act.cuh"
#include "common.cuh"
#include "host_util.h"

namespace mx {

constexpr int DA_WARPS = 4;
constexpr int DA_TILE = 64;               // unit of work and of the window's arithmetic
constexpr int DA_MAX_ENTRIES = 512;       // (sequence, query tile) pairs of a launch

struct DecodeAttnParams {
  const __nv_bfloat16* q;      // [Tq] rows of [n_q][HD], q_ld elements apart (4-byte aligned rows)
  const uint8_t* k_cache;      // [block][kv_head][block_size][HD] bf16 or int8
  const uint8_t* v_cache;
  const float* k_scale;        // int8: [block][kv_head][block_size]
  const float* v_scale;
  const int* block_table;      // [B][max_blocks]
  const int* seq_lens;
  const int* cu_q;
  const float* sinks;
  const float* q_scale;
  const __nv_bfloat16* gate;
  __nv_bfloat16* out;          // [Tq][n_q][HD]
  float* o_part;               // [grid][2][pairs][HD]
  float* ml_part;              // [grid][2][pairs][2]
  int* tickets;                // one counter per CTA: that of the cut group which is the CTA's last
  int q_scale_n, q_ld, gate_ld, gate_heads, keep_first;
  int B, n_q, n_kv, max_blocks, block_size, q_tile, max_q_tiles, window;
  float scale, softcap;
};

// one (sequence, query tile) of the batch
struct DecodeEntry {
  int b, q_row, nt, pos0, kv_hi, tile_lo, n_keep, n_tiles;
};
__device__ __forceinline__ DecodeEntry decode_entry(const DecodeAttnParams& p, int e) {
  DecodeEntry r;
  r.b = e / p.max_q_tiles;
  const int t0 = (e % p.max_q_tiles) * p.q_tile;
  const int q_begin = __ldg(p.cu_q + r.b), q_len = __ldg(p.cu_q + r.b + 1) - q_begin, seq_len = __ldg(p.seq_lens + r.b);
  r.q_row = q_begin + t0;
  r.nt = min(p.q_tile, q_len - t0);
  r.pos0 = seq_len - q_len + t0;
  r.kv_hi = min(seq_len, r.pos0 + r.nt);
  const int kv_lo = p.window > 0 ? max(0, r.pos0 - p.window + 1) : 0;
  r.tile_lo = kv_lo / DA_TILE;
  r.n_keep = min((p.keep_first + DA_TILE - 1) / DA_TILE, r.tile_lo);
  r.n_tiles = r.nt > 0 && r.kv_hi > 0 ? r.n_keep + (r.kv_hi + DA_TILE - 1) / DA_TILE - r.tile_lo : 0;
  return r;
}

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool live) {      // (not live: zeros)
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(live ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async4(uint32_t dst, const void* src, bool live) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(live ? 4 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm4_t(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ uint32_t mat_trans(uint32_t v) {
  uint32_t d;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(d) : "r"(v));
  return d;
}
__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], const uint32_t b0, const uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// two signed bytes of w (selected by sel into the low bytes of the halves) as bf16, exactly: the low seven bits above 128, minus 128 or 256
template <int SEL> __device__ __forceinline__ uint32_t s8_pair_bf16(uint32_t w) {
  const uint32_t t = __byte_perm(w, 0, SEL);
  const uint32_t x = (t & 0x007f007fu) | 0x43004300u, y = (t & 0x00800080u) | 0x43004300u;
  const __nv_bfloat162 d = __hsub2(*reinterpret_cast<const __nv_bfloat162*>(&x), *reinterpret_cast<const __nv_bfloat162*>(&y));
  return *reinterpret_cast<const uint32_t*>(&d);
}

// Tiles per CTA.  An equal share, but not so little that merging costs more than it saves: a partial is read back at about an eighth of a tile's time,
// so n / per partials and per tiles balance at per = sqrt(n / 8).
__host__ __device__ inline int decode_run(int total, int grid, int most) {
  int per = total > grid ? (total - 1) / grid + 1 : 1;
  while ((long long)per * per * 8 < most) ++per;
  return per;
}

template <int HD, int NT, bool KV8> struct DecodeShape {
  static constexpr int RB = HD * (KV8 ? 1 : 2);                         // bytes of a cache row
  static constexpr int SK = RB <= 128 ? 32 : 16;                        // keys per warp step
  static constexpr int KVB = 2 * SK * RB;                               // K rows, V rows
  static constexpr int SLOT = KVB + (KV8 ? 256 : 0);                    // and their scales
  static constexpr int NST = 3;
  static constexpr int PAIRS = NT * 8;
  static constexpr int SMEM = DA_WARPS * NST * SLOT;
  static constexpr int NTP = NT < KVB / (8 * HD * 4) ? NT : KVB / (8 * HD * 4);   // column groups merged over the warps at a time, in freed slots
  // byte offset of 16-byte chunk c of row r: eight consecutive rows at one chunk lie in eight bank groups
  static __device__ __forceinline__ uint32_t at(int r, int c) {
    if constexpr (RB >= 128) return r * RB + ((c ^ (r & 7)) << 4);
    else return r * RB + ((c ^ ((r >> 1) & 3)) << 4);
  }
};

template <int HD, int NT, bool KV8>
__global__ void __launch_bounds__(DA_WARPS * 32, HD == 256 ? 1 : 2) attn_decode_kernel(const DecodeAttnParams p) {
  using S = DecodeShape<HD, NT, KV8>;
  constexpr int SK = S::SK, KT = SK / 16, RB = S::RB, CH = RB / 16, PAIRS = S::PAIRS, NST = S::NST, MT = HD / 16;
  constexpr int SPT = DA_TILE / SK;                                      // steps per tile
  pdl_prologue();
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ int s_pre[DA_MAX_ENTRIES + 1];
  __shared__ int s_red[2][DA_WARPS];
  __shared__ float s_m[DA_WARPS][PAIRS], s_l[DA_WARPS][PAIRS];
  __shared__ float s_w[PAIRS][33];
  __shared__ float s_inv[PAIRS];
  __shared__ int s_last;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t4 = lane & 3;
  const int entries = p.B * p.max_q_tiles, gqa = p.n_q / p.n_kv;

  // ---- tiles of every entry, their running sum, and this CTA's run of the list
  int most = 0;
  {
    int base = 0;
    for (int e0 = 0; e0 < entries; e0 += DA_WARPS * 32) {
      const int e = e0 + tid;
      int n = e < entries ? decode_entry(p, e).n_tiles : 0, incl = n;
      most = max(most, n);
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += u;
      }
      if (lane == 31) s_red[0][warp] = incl;
      __syncthreads();
      int before = base;
#pragma unroll
      for (int w = 0; w < DA_WARPS; ++w) {
        if (w < warp) before += s_red[0][w];
        base += s_red[0][w];
      }
      if (e < entries) s_pre[e + 1] = before + incl;
      __syncthreads();
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) most = max(most, __shfl_xor_sync(0xffffffffu, most, o));
    if (lane == 0) s_red[1][warp] = most;
    if (tid == 0) s_pre[0] = 0;
    __syncthreads();
#pragma unroll
    for (int w = 0; w < DA_WARPS; ++w) most = max(most, s_red[1][w]);
  }
  const int total = s_pre[entries] * p.n_kv;
  const int per = decode_run(total, (int)gridDim.x, most);
  const int my0 = blockIdx.x * per, my1 = min(total, my0 + per);
  if (my0 >= total) return;
  int e_first = 0;
  {
    int lo = 0, hi = entries - 1;                                        // the last entry that starts at or before my0 (empty ones start where the next does)
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (s_pre[mid] * p.n_kv <= my0) lo = mid; else hi = mid - 1;
    }
    e_first = lo;
  }

  // ---- the warp's loads: they run ahead of the arithmetic, across groups
  const uint32_t ring = smem_u32(smem) + warp * (NST * S::SLOT);
  struct {
    int u, e, s, n_steps, kvh, t0, kv_hi, b, tile_lo, n_keep;
  } ld = {my0, e_first, 0, 0, 0, 0, 0, 0, 0, 0};
  auto ld_group = [&]() {                                                // the group at ld.u (< my1)
    while (s_pre[ld.e + 1] * p.n_kv <= ld.u) ++ld.e;
    const DecodeEntry en = decode_entry(p, ld.e);
    const int off = ld.u - s_pre[ld.e] * p.n_kv;
    ld.kvh = off / en.n_tiles;
    ld.t0 = off % en.n_tiles;
    const int n = min(my1 - ld.u, en.n_tiles - ld.t0);
    ld.u += n;
    ld.n_steps = n * SPT;
    ld.s = warp;
    ld.kv_hi = en.kv_hi; ld.b = en.b; ld.tile_lo = en.tile_lo; ld.n_keep = en.n_keep;
  };
  auto ld_key = [&]() {
    const int tl = ld.t0 + ld.s / SPT;
    return (tl < ld.n_keep ? tl : ld.tile_lo + tl - ld.n_keep) * DA_TILE + (ld.s % SPT) * SK;
  };
  int ld_blk = 0;
  bool ld_live = true;
  auto ld_seek = [&]() {                                                 // the next step this warp owns, and its page
    while (ld.s >= ld.n_steps) {
      if (ld.u >= my1) { ld_live = false; return; }
      ld_group();
    }
    ld_blk = __ldg(p.block_table + (size_t)ld.b * p.max_blocks + ld_key() / p.block_size);
  };
  int ld_slot = 0;
  auto ld_issue = [&]() {
    if (ld_live) {
      const int key = ld_key();
      const size_t row0 = ((size_t)ld_blk * p.n_kv + ld.kvh) * p.block_size + key % p.block_size;
      const uint32_t dst = ring + ld_slot * S::SLOT;
      const uint8_t* kp = p.k_cache + row0 * RB;
      const uint8_t* vp = p.v_cache + row0 * RB;
      const int live = ld.kv_hi - key;                                   // rows past the sequence's end are not read: zeros
#pragma unroll
      for (int i = 0; i < SK * CH / 32; ++i) {
        const int at = i * 32 + lane, r = at / CH, c = at % CH;
        cp_async16(dst + S::at(r, c), kp + r * RB + c * 16, r < live);
        cp_async16(dst + SK * RB + S::at(r, c), vp + r * RB + c * 16, r < live);
      }
      if constexpr (KV8) {
        if (lane < SK) {
          cp_async4(dst + S::KVB + lane * 4, p.k_scale + row0 + lane, lane < live);
          cp_async4(dst + S::KVB + 128 + lane * 4, p.v_scale + row0 + lane, lane < live);
        }
      }
      ld.s += DA_WARPS;
      ld_seek();
    }
    cp_async_commit();
    ld_slot = ld_slot + 1 == NST ? 0 : ld_slot + 1;
  };
  ld_seek();
#pragma unroll
  for (int i = 0; i < NST - 1; ++i) ld_issue();

  // ---- the groups of this CTA
  int slot = 0;
  for (int u = my0, e = e_first; u < my1;) {
    while (s_pre[e + 1] * p.n_kv <= u) ++e;
    const DecodeEntry en = decode_entry(p, e);
    const int g0 = s_pre[e] * p.n_kv, kvh = (u - g0) / en.n_tiles, t0 = (u - g0) % en.n_tiles;
    const int n = min(my1 - u, en.n_tiles - t0), total_pairs = en.nt * gqa;
    const int gs = u - t0, ge = gs + en.n_tiles;                         // the whole group in the list
    // queries as B operands; a lane's two columns per column group: pair 8 nt + 2 t4 (+ 1)
    uint32_t qf[MT][NT][2];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      const int pr = nt * 8 + g;
      const __nv_bfloat16* qr = p.q + (size_t)(en.q_row + pr / gqa) * p.q_ld + (size_t)(kvh * gqa + pr % gqa) * HD;
#pragma unroll
      for (int kk = 0; kk < MT; ++kk)
#pragma unroll
        for (int j = 0; j < 2; ++j)
          qf[kk][nt][j] = pr < total_pairs ? *reinterpret_cast<const uint32_t*>(qr + kk * 16 + (KV8 ? 4 * t4 + 2 * j : 2 * t4 + 8 * j)) : 0u;
    }
    int qpos[NT][2];
    float fac[NT][2], m[NT][2], l[NT][2], acc[MT][NT][4];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int pr = nt * 8 + 2 * t4 + j;
        qpos[nt][j] = pr < total_pairs ? en.pos0 + pr / gqa : -1;        // (-1: sees no key)
        fac[nt][j] = p.scale;
        if (p.q_scale && pr < total_pairs) fac[nt][j] *= p.q_scale[min(qpos[nt][j], p.q_scale_n - 1)];
        m[nt][j] = -1e30f; l[nt][j] = 0.f;
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) acc[mt][nt][j] = acc[mt][nt][2 + j] = 0.f;
      }
    for (int s = warp; s < n * SPT; s += DA_WARPS) {
      ld_issue();
      cp_async_wait<NST - 1>();
      __syncwarp();
      const int tl = t0 + s / SPT;
      const int key0 = (tl < en.n_keep ? tl : en.tile_lo + tl - en.n_keep) * DA_TILE + (s % SPT) * SK;
      const uint32_t sk = ring + slot * S::SLOT, sv = sk + SK * RB;
      const float* scl = reinterpret_cast<const float*>(smem + warp * (NST * S::SLOT) + slot * S::SLOT + S::KVB);
      // S^T [keys][pairs]
      float sc[KT][NT][4];
#pragma unroll
      for (int kt = 0; kt < KT; ++kt) {
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
          for (int i = 0; i < 4; ++i) sc[kt][nt][i] = 0.f;
        const int r = kt * 16 + (lane & 7) + ((lane >> 3) & 1) * 8, c = lane >> 4;
        if constexpr (!KV8) {
#pragma unroll
          for (int kk = 0; kk < MT; ++kk) {
            uint32_t a[4];
            ldsm4(a, sk + S::at(r, 2 * kk + c));
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) mma_bf16(sc[kt][nt], a, qf[kk][nt][0], qf[kk][nt][1]);
          }
        } else {
#pragma unroll
          for (int kk = 0; kk < MT; kk += 2) {
            uint32_t w[4];
            ldsm4(w, sk + S::at(r, kk + c));
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const uint32_t a[4] = {s8_pair_bf16<0x4140>(w[2 * h]), s8_pair_bf16<0x4140>(w[2 * h + 1]), s8_pair_bf16<0x4342>(w[2 * h]),
                                     s8_pair_bf16<0x4342>(w[2 * h + 1])};
#pragma unroll
              for (int nt = 0; nt < NT; ++nt) mma_bf16(sc[kt][nt], a, qf[kk + h][nt][0], qf[kk + h][nt][1]);
            }
          }
        }
      }
      // scale, mask, running maximum
      float mx[NT][2];
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) mx[nt][0] = mx[nt][1] = -INFINITY;
#pragma unroll
      for (int kt = 0; kt < KT; ++kt)
#pragma unroll
        for (int i2 = 0; i2 < 2; ++i2) {
          const int r = kt * 16 + g + 8 * i2, kpos = key0 + r;
          const float ks = KV8 ? scl[r] : 1.f;
#pragma unroll
          for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int j = 0; j < 2; ++j) {
              float v = sc[kt][nt][2 * i2 + j] * fac[nt][j];
              if constexpr (KV8) v *= ks;
              if (p.softcap > 0.f) v = p.softcap * tanhf(v / p.softcap);
              const int qp = qpos[nt][j];
              const bool ok = kpos <= qp && (p.window <= 0 || kpos > qp - p.window || kpos < p.keep_first);
              v = ok ? v : -INFINITY;
              sc[kt][nt][2 * i2 + j] = v;
              mx[nt][j] = fmaxf(mx[nt][j], v);
            }
        }
      bool grew = false;
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
#pragma unroll
          for (int o = 4; o < 32; o <<= 1) mx[nt][j] = fmaxf(mx[nt][j], __shfl_xor_sync(0xffffffffu, mx[nt][j], o));
          grew |= mx[nt][j] > m[nt][j];
        }
      if (__any_sync(0xffffffffu, grew)) {
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            const float mn = fmaxf(m[nt][j], mx[nt][j]), corr = __expf(m[nt][j] - mn);
            m[nt][j] = mn;
            l[nt][j] *= corr;
#pragma unroll
            for (int mt = 0; mt < MT; ++mt) {
              acc[mt][nt][j] *= corr;
              acc[mt][nt][2 + j] *= corr;
            }
          }
      }
      // P^T as B operands, in three bf16 terms; O^T [d][pairs] += V^T P^T
#pragma unroll
      for (int kt = 0; kt < KT; ++kt) {
        uint32_t pf[NT][3][2];
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
          for (int i2 = 0; i2 < 2; ++i2) {
            float a = __expf(sc[kt][nt][2 * i2] - m[nt][0]), b = __expf(sc[kt][nt][2 * i2 + 1] - m[nt][1]);
            l[nt][0] += a;
            l[nt][1] += b;
            if constexpr (KV8) {
              const float vs = scl[32 + kt * 16 + g + 8 * i2];
              a *= vs;
              b *= vs;
            }
#pragma unroll
            for (int k = 0; k < 3; ++k) {
              const uint32_t h = pack_bf16(a, b);
              pf[nt][k][i2] = mat_trans(h);
              a -= bf16_lo(h);
              b -= bf16_hi(h);
            }
          }
        if constexpr (!KV8) {
          const int r = kt * 16 + (lane & 7) + (lane >> 4) * 8, c = (lane >> 3) & 1;
#pragma unroll
          for (int mt = 0; mt < MT; ++mt) {
            uint32_t a[4];
            ldsm4_t(a, sv + S::at(r, 2 * mt + c));
#pragma unroll
            for (int k = 0; k < 3; ++k)
#pragma unroll
              for (int nt = 0; nt < NT; ++nt) mma_bf16(acc[mt][nt], a, pf[nt][k][0], pf[nt][k][1]);
          }
        } else {
          const int r = kt * 16 + (lane & 7) + ((lane >> 3) & 1) * 8, c = lane >> 4;
#pragma unroll
          for (int mt = 0; mt < MT; mt += 2) {
            uint32_t w[4];
            ldsm4_t(w, sv + S::at(r, mt + c));
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const uint32_t a[4] = {s8_pair_bf16<0x4240>(w[2 * h]), s8_pair_bf16<0x4341>(w[2 * h]), s8_pair_bf16<0x4240>(w[2 * h + 1]),
                                     s8_pair_bf16<0x4341>(w[2 * h + 1])};
#pragma unroll
              for (int k = 0; k < 3; ++k)
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) mma_bf16(acc[mt + h][nt], a, pf[nt][k][0], pf[nt][k][1]);
            }
          }
        }
      }
      __syncwarp();                                                      // the slot is read: the next issue may overwrite it
      slot = slot + 1 == NST ? 0 : slot + 1;
    }

    // ---- the warps' parts of this group: their slots that no load is under way to take the sums, NTP column groups at a time
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int j = 0; j < 2; ++j) {
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) l[nt][j] += __shfl_xor_sync(0xffffffffu, l[nt][j], o);
        if (g == 0) {
          s_m[warp][nt * 8 + 2 * t4 + j] = m[nt][j];
          s_l[warp][nt * 8 + 2 * t4 + j] = l[nt][j];
        }
      }
    // the slot after the last one issued: NST - 1 steps are under way behind the warp's current slot
    uint8_t* const freed = smem + warp * (NST * S::SLOT) + ld_slot * S::SLOT;
    const int free_at = (int)(freed - smem);
    __shared__ int s_free[DA_WARPS];
    if (lane == 0) s_free[warp] = free_at;
    __syncthreads();
    const bool cut = t0 > 0 || n < en.n_tiles;
    const int c0 = gs / per, c1 = (ge - 1) / per;
    const size_t part = ((size_t)blockIdx.x * 2 + (cut && (int)blockIdx.x == c0 ? 1 : 0)) * PAIRS;
#pragma unroll
    for (int n0 = 0; n0 < NT; n0 += S::NTP) {
#pragma unroll
      for (int nn = 0; nn < S::NTP; ++nn) {
        const int nt = n0 + nn;
        if (nt >= NT) continue;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int pr = nt * 8 + 2 * t4 + j;
          float M = m[nt][j];
#pragma unroll
          for (int w = 0; w < DA_WARPS; ++w) M = fmaxf(M, s_m[w][pr]);
          const float f = __expf(m[nt][j] - M);
          float* row = reinterpret_cast<float*>(freed) + (nn * 8 + 2 * t4 + j) * HD;
#pragma unroll
          for (int mt = 0; mt < MT; ++mt) {                              // (words 8 t4 apart in a row: conflict-free stores)
            row[(mt * 16 + (KV8 ? 2 * g : g)) ^ (8 * t4)] = acc[mt][nt][j] * f;
            row[(mt * 16 + (KV8 ? 2 * g + 1 : 8 + g)) ^ (8 * t4)] = acc[mt][nt][2 + j] * f;
          }
        }
      }
      __syncthreads();
      for (int i = tid; i < S::NTP * 8 * HD / 4; i += DA_WARPS * 32) {
        const int lp = i / (HD / 4), d = (i % (HD / 4)) * 4, pr = n0 * 8 + lp;
        if (pr >= total_pairs) continue;
        float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
        float M = -1e30f, L = 0.f;
#pragma unroll
        for (int w = 0; w < DA_WARPS; ++w) {
          const float4 v = *reinterpret_cast<const float4*>(smem + s_free[w] + (lp * HD + (d ^ (8 * ((lp >> 1) & 3)))) * 4);
          o.x += v.x; o.y += v.y; o.z += v.z; o.w += v.w;
          M = fmaxf(M, s_m[w][pr]);
        }
#pragma unroll
        for (int w = 0; w < DA_WARPS; ++w) L += s_l[w][pr] * __expf(s_m[w][pr] - M);
        if (cut) {
          *reinterpret_cast<float4*>(p.o_part + (part + pr) * HD + d) = o;
          if (d == 0) *reinterpret_cast<float2*>(p.ml_part + (part + pr) * 2) = make_float2(M, L);
        } else {
          const int hq = kvh * gqa + pr % gqa;
          const size_t row = en.q_row + pr / gqa;
          float f = 1.f;
          if (p.sinks) {
            const float M2 = fmaxf(M, p.sinks[hq]);
            f = __expf(M - M2);
            L = L * f + __expf(p.sinks[hq] - M2);
          }
          f = L > 0.f ? f / L : 0.f;
          float v[4] = {o.x * f, o.y * f, o.z * f, o.w * f};
          if (p.gate) {
            const __nv_bfloat16* gr = p.gate + row * p.gate_ld + (p.gate_heads ? hq : (size_t)hq * HD + d);
#pragma unroll
            for (int k = 0; k < 4; ++k) v[k] *= sigmoid_f<false>(__bfloat162float(gr[p.gate_heads ? 0 : k]));
          }
          *reinterpret_cast<uint2*>(p.out + (row * p.n_q + hq) * HD + d) = make_uint2(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]));
        }
      }
      __syncthreads();
    }

    // ---- a cut group: the CTA that arrives last merges the partials, in the order of the CTAs
    if (cut) {
      const int parts = c1 - c0 + 1;
      __threadfence();
      __syncthreads();
      if (tid == 0) {
        const int prev = atomicAdd(p.tickets + c0, 1);
        s_last = prev == parts - 1;
        if (s_last) p.tickets[c0] = 0;
      }
      __syncthreads();
      if (s_last) {
        __threadfence();
        auto row_of = [&](int i) { return ((size_t)(c0 + i) * 2 + (i == 0 ? 1 : 0)) * PAIRS; };
        for (int pr = warp; pr < PAIRS; pr += DA_WARPS) {                // maximum and denominator over all parts
          if (pr >= total_pairs) continue;
          const int hq = kvh * gqa + pr % gqa;
          float M = p.sinks ? p.sinks[hq] : -1e30f, L = 0.f;
          for (int i = lane; i < parts; i += 32) M = fmaxf(M, __ldcg(p.ml_part + (row_of(i) + pr) * 2));
          M = warp_max(M);
          for (int i = lane; i < parts; i += 32) {
            const float2 ml = __ldcg(reinterpret_cast<const float2*>(p.ml_part + (row_of(i) + pr) * 2));
            L += ml.y * __expf(ml.x - M);
          }
          L = warp_sum(L) + (p.sinks ? __expf(p.sinks[hq] - M) : 0.f);
          if (lane == 0) { s_m[0][pr] = M; s_inv[pr] = L > 0.f ? 1.f / L : 0.f; }
        }
        constexpr int V4 = PAIRS * HD / 4 / (DA_WARPS * 32);             // float4 of the output per thread
        float4 o[V4];
#pragma unroll
        for (int k = 0; k < V4; ++k) o[k] = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int i0 = 0; i0 < parts; i0 += 32) {
          __syncthreads();
          for (int i = tid; i < PAIRS * 32; i += DA_WARPS * 32) {
            const int pr = i >> 5, at = i0 + (i & 31);
            s_w[pr][i & 31] = pr < total_pairs && at < parts ? __expf(__ldcg(p.ml_part + (row_of(at) + pr) * 2) - s_m[0][pr]) : 0.f;
          }
          __syncthreads();
          const int cnt = min(32, parts - i0);
#pragma unroll 4
          for (int i = 0; i < cnt; ++i) {
            const float* src = p.o_part + row_of(i0 + i) * HD;
#pragma unroll
            for (int k = 0; k < V4; ++k) {
              const int at = (k * DA_WARPS * 32 + tid) * 4, pr = at / HD;
              if (pr >= total_pairs) continue;
              const float4 v = __ldcg(reinterpret_cast<const float4*>(src + at));
              const float w = s_w[pr][i];
              o[k].x = fmaf(v.x, w, o[k].x); o[k].y = fmaf(v.y, w, o[k].y); o[k].z = fmaf(v.z, w, o[k].z); o[k].w = fmaf(v.w, w, o[k].w);
            }
          }
        }
#pragma unroll
        for (int k = 0; k < V4; ++k) {
          const int at = (k * DA_WARPS * 32 + tid) * 4, pr = at / HD, d = at % HD;
          if (pr >= total_pairs) continue;
          const int hq = kvh * gqa + pr % gqa;
          const size_t row = en.q_row + pr / gqa;
          const float f = s_inv[pr];
          float v[4] = {o[k].x * f, o[k].y * f, o[k].z * f, o[k].w * f};
          if (p.gate) {
            const __nv_bfloat16* gr = p.gate + row * p.gate_ld + (p.gate_heads ? hq : (size_t)hq * HD + d);
#pragma unroll
            for (int j = 0; j < 4; ++j) v[j] *= sigmoid_f<false>(__bfloat162float(gr[p.gate_heads ? 0 : j]));
          }
          *reinterpret_cast<uint2*>(p.out + (row * p.n_q + hq) * HD + d) = make_uint2(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]));
        }
        __syncthreads();                                                 // s_m is written again by the next group
      }
    }
    u += n;
  }
  cp_async_wait<0>();
}

constexpr int DA_MAX_GRID = 512;
static_assert(DA_MAX_GRID <= CUT_TICKETS, "a counter per CTA");

struct DecodePlan { int nt = 0, q_tile = 0, max_q_tiles = 0; };

// Column groups of 8 (query, head) pairs per CTA: as few as hold the queries of a sequence, at most 32 pairs (16 with 256-wide heads: the
// accumulators are 16 registers per 64 columns and group).
static bool decode_plan(int hd, int B, int n_q, int n_kv, int max_q_len, DecodePlan& pl) {
  if ((hd != 64 && hd != 128 && hd != 256) || n_kv < 1 || n_q % n_kv || B < 1 || max_q_len < 1) return false;
  const int gqa = n_q / n_kv, cap = hd == 256 ? 2 : 4;
  if (gqa > 8 * cap) return false;
  const long long pairs = (long long)max_q_len * gqa;
  pl.nt = pairs <= 8 ? 1 : (pairs <= 16 || cap == 2) ? 2 : 4;
  pl.q_tile = 8 * pl.nt / gqa;
  if (pl.q_tile > max_q_len) pl.q_tile = max_q_len;
  pl.max_q_tiles = (max_q_len + pl.q_tile - 1) / pl.q_tile;
  return (long long)B * pl.max_q_tiles <= DA_MAX_ENTRIES;
}

template <int HD, int NT, bool KV8> static int decode_grid() {          // resident CTAs of the device
  static int grid[64] = {0};
  const int dev = DeviceOnce::ordinal();
  if (!grid[dev]) {
    auto kern = attn_decode_kernel<HD, NT, KV8>;
    using S = DecodeShape<HD, NT, KV8>;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, S::SMEM) != cudaSuccess) return -1;
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, DA_WARPS * 32, S::SMEM) != cudaSuccess || per_sm < 1) return -1;
    const int n = sm_count() * per_sm;
    grid[dev] = n < DA_MAX_GRID ? n : DA_MAX_GRID;
  }
  return grid[dev];
}

template <int HD, int NT, bool KV8> static int launch_decode(DecodeAttnParams& p, float* scratch, cudaStream_t st) {
  using S = DecodeShape<HD, NT, KV8>;
  const int grid = decode_grid<HD, NT, KV8>();
  if (grid < 1) return -116;
  p.o_part = scratch;
  p.ml_part = scratch + (size_t)DA_MAX_GRID * 2 * S::PAIRS * HD;
  launch_pdl(attn_decode_kernel<HD, NT, KV8>, dim3(grid), dim3(DA_WARPS * 32), S::SMEM, st, p);
  return (int)cudaGetLastError();
}

}  // namespace mx

using namespace mx;

// Floats of scratch (16-byte aligned) that mx_attention_decode needs, or 0 when it does not take such a call.
MX_HOST_API int mx_attention_decode_scratch(int hd, int B, int n_q, int n_kv, int max_q_len) {
  DecodePlan pl;
  if (!decode_plan(hd, B, n_q, n_kv, max_q_len, pl)) return 0;
  return DA_MAX_GRID * 2 * 8 * pl.nt * (hd + 2);
}

MX_HOST_API int mx_attention_decode_run(int total, int grid, int most) { return decode_run(total, grid, most); }

// Arguments as in mx_attention_ext / mx_attention_kv8 (k_scale non-null: an int8 cache).  q 4-byte aligned with an even q_ld, cache pages 16-byte
// aligned, out 8-byte aligned.  tickets: see host_util.h.
MX_HOST_API int mx_attention_decode(const void* q, int q_ld, const void* k_cache, const void* v_cache, const float* k_scale, const float* v_scale,
                                    const int* block_table, const int* seq_lens, const int* cu_q, const float* sinks, const void* gate, int gate_ld,
                                    const float* q_scale, int q_scale_n, void* out, float* scratch, int* tickets, int B, int Tq, int max_q_len, int n_q, int n_kv, int hd,
                                    int max_blocks, int block_size, int window, int keep_first, int gate_heads, float scale, float softcap,
                                    cudaStream_t st) {
  if (B <= 0 || Tq <= 0) return 0;
  if (block_size % DA_TILE) return -110;
  DecodePlan pl;
  if (!decode_plan(hd, B, n_q, n_kv, max_q_len, pl)) return -112;
  if ((q_ld & 1) || ((uintptr_t)q & 3) || ((uintptr_t)out & 7) || (((uintptr_t)k_cache | (uintptr_t)v_cache | (uintptr_t)scratch) & 15)) return -114;
  if ((k_scale != nullptr) != (v_scale != nullptr)) return -113;
  DecodeAttnParams p;
  p.q = (const __nv_bfloat16*)q; p.k_cache = (const uint8_t*)k_cache; p.v_cache = (const uint8_t*)v_cache; p.k_scale = k_scale; p.v_scale = v_scale;
  p.block_table = block_table; p.seq_lens = seq_lens; p.cu_q = cu_q; p.sinks = sinks; p.q_scale = q_scale; p.gate = (const __nv_bfloat16*)gate;
  p.out = (__nv_bfloat16*)out; p.q_scale_n = q_scale_n; p.q_ld = q_ld; p.gate_ld = gate_ld; p.gate_heads = gate_heads;
  p.keep_first = window > 0 ? keep_first : 0;
  p.B = B; p.n_q = n_q; p.n_kv = n_kv; p.max_blocks = max_blocks; p.block_size = block_size; p.q_tile = pl.q_tile; p.max_q_tiles = pl.max_q_tiles;
  p.window = window; p.scale = scale; p.softcap = softcap;
  p.tickets = tickets;
#define MX_DA(HD_, NT_) (k_scale ? launch_decode<HD_, NT_, true>(p, scratch, st) : launch_decode<HD_, NT_, false>(p, scratch, st))
  if (hd == 64) return pl.nt == 1 ? MX_DA(64, 1) : pl.nt == 2 ? MX_DA(64, 2) : MX_DA(64, 4);
  if (hd == 128) return pl.nt == 1 ? MX_DA(128, 1) : pl.nt == 2 ? MX_DA(128, 2) : MX_DA(128, 4);
  return pl.nt == 1 ? MX_DA(256, 1) : MX_DA(256, 2);
#undef MX_DA
}
