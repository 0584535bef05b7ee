// attn_premix_tc.cu -- prompt attention whose scaled and capped scores are mixed over the heads BEFORE the softmax (s'_a = sum_b mix[a][b] s_b), 8, 16 or 32 heads of 128 + 128,
// two per key/value head, bf16 cache.
//
// A mixed score needs every head's score of its (query, key) pair, and no SM holds the running outputs of 32 heads beside the operands of a useful tile.  So the pass is cut at the
// mixed scores, which go through a scratch buffer that stays in L2 for the most part:
//   premix_scores  a unit is QB query tokens x 128 keys x ALL heads.  Keys are the M of the products, so a thread owns a key (its TMEM lane) and QB / 4 tokens, and the mix of its
//                  pairs needs nothing from other threads: per key/value head, S^T[128 keys][QB x 2 heads x 2] = K . Q^T on tcgen05.mma (queries as bf16 value + remainder, the two
//                  halves in columns of their own), TMEM -> registers, scale and cap, and heads x QB / 4 running sums take two packed multiply-adds per pair of heads.  K and Q come
//                  in through TMA, a ring of stages that runs on across units; S through a ring of TMEM slots.
//   premix_values  64 query tokens of one key/value head's two heads per CTA: the scratch rows as they are (fp32), causal mask, online softmax, P . V on warp-level MMAs with the
//                  weights as bf16 value + remainder, the turn back by the query's position, one rounding.
// Units of whole tiles are cut into launches that fit the scratch.
// Measured, 4 x 1024 tokens of 32 heads: the cluster kernel of attn_heads.cu 1860 us, here 212 + 180 (16 heads: 495 -> 86 + 126).  premix_scores takes 187 us without the mix and the
// cap (K and Q on their way, 640 bytes a pair from L2, in 2 KB copies 226) and the mix's multiply-adds 70 at the FMA pipe's rate; sixteen warps with the matrix in shared memory took 314,
// eight 330, the matrix in constant memory with running places 299.  premix_values is bound by the warp-level MMAs (40 % busy) and the latencies between them.
#include "kernels.h"

#include <algorithm>
#include <type_traits>

namespace b2 {

namespace {

constexpr int PT_KEYS = 128, PT_MIX_WARPS = 16, PT_THREADS = 32 * (PT_MIX_WARPS + 2), PT_MAX_TILES = 1024, PT_DIM = 128;
constexpr int PT_K_BYTES = PT_KEYS * PT_DIM * 2;

template <int H>
struct PtCfg {
  static constexpr int QB = H == 32 ? 8 : 16;          // query tokens of a unit: heads x QB / 4 running sums a thread
  static constexpr int G = H / 2, NCOL = QB * 4;       // columns of one key/value head: token, head of two, value or remainder
  static constexpr int STAGE_BYTES = PT_K_BYTES + NCOL * PT_DIM * 2;
  static constexpr int STAGES = H == 32 ? 5 : 4;
  static constexpr int SLOTS = 256 / NCOL;             // of two key/value heads each
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024;
  static constexpr size_t UNIT_FLOATS = (size_t)H * QB * PT_KEYS;
};

// [b][a]: head b's weight in the mix of head a.  A kernel parameter: the multiply-adds then take it from constant memory, while 128 bytes of shared memory for every head and warp
// would take as long as the sums themselves.
template <int H>
struct alignas(16) PtMix {
  float m[H * H];
};

struct PtArgs {
  HeadsGeom g;
  const int32_t* block_table;
  int bt_stride, block_size;
  const PrefillTile* tiles;   // of this launch
  int ntiles, T;
  float* scores;              // [unit][head][token][key]
};

__host__ __device__ inline int pt_key_blocks(const PrefillTile& t) { return (t.q_pos0 + t.nrows - 1) / PT_KEYS + 1; }
__host__ __device__ inline int pt_units(const PrefillTile& t, int qb) { return t.nrows <= 0 ? 0 : (t.nrows + qb - 1) / qb * pt_key_blocks(t); }

__device__ __forceinline__ void fma2(unsigned long long& d, unsigned long long a, unsigned long long b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b)); }

__device__ __forceinline__ void pt_tmem_ld8(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}

// One unit: its query tokens' first position and count, its key block.  Units of a tile: query blocks, each with all key blocks of the tile.
struct PtUnit {
  PrefillTile t;
  int q0, ntok, pos0, last, key0;   // q0: token row of the batch
  bool seen;                        // some token sees a key of the block
};
template <int QB>
__device__ __forceinline__ PtUnit pt_unit(const PtArgs& a, const int* base, int u) {
  int lo = 0, hi = a.ntiles - 1;
  while (lo < hi) {   // the last tile whose first unit is not behind u
    const int mid = (lo + hi + 1) >> 1;
    if (base[mid] <= u) lo = mid;
    else hi = mid - 1;
  }
  PtUnit x;
  x.t = a.tiles[lo];
  const int nkb = pt_key_blocks(x.t), i = u - base[lo], qb = i / nkb;
  x.key0 = (i - qb * nkb) * PT_KEYS;
  x.q0 = x.t.q_row0 + qb * QB;
  x.pos0 = x.t.q_pos0 + qb * QB;
  x.ntok = min(QB, x.t.nrows - qb * QB);
  x.last = x.pos0 + x.ntok - 1;
  x.seen = x.key0 <= x.last;
  return x;
}

template <int H>
__global__ void __launch_bounds__(PT_THREADS, 1)
premix_scores_kernel(const __grid_constant__ CUtensorMap tmap_k, const __grid_constant__ CUtensorMap tmap_q, const PtArgs a, const __grid_constant__ PtMix<H> mix_of, const B2WaitLimit limit) {
  using C = PtCfg<H>;
  constexpr int QB = C::QB, G = C::G, QT = QB / (PT_MIX_WARPS / 4), CT = 4 * QT;   // a mix thread's tokens and its columns of one key/value head
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t full_bar[C::STAGES];
  __shared__ __align__(8) uint64_t empty_bar[C::STAGES];
  __shared__ __align__(8) uint64_t slot_full[C::SLOTS];
  __shared__ __align__(8) uint64_t slot_empty[C::SLOTS];
  __shared__ __align__(8) uint64_t drained;
  __shared__ uint32_t tmem_slot;
  __shared__ volatile uint32_t gave_up;
  __shared__ int base[PT_MAX_TILES + 1];         // first unit of every tile
  __shared__ int part[PT_THREADS / 32];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  if (tid == 0) {
    for (int s = 0; s < C::STAGES; ++s) {
      mbar_init(smem_u32(&full_bar[s]), 1);
      mbar_init(smem_u32(&empty_bar[s]), 1);
    }
    for (int s = 0; s < C::SLOTS; ++s) {
      mbar_init(smem_u32(&slot_full[s]), 1);
      mbar_init(smem_u32(&slot_empty[s]), PT_MIX_WARPS);
    }
    mbar_init(smem_u32(&drained), 1);
    gave_up = 0;
    mbar_fence_init();
  }
  if (warp == PT_MIX_WARPS + 1) {
    tmem_alloc(smem_u32(&tmem_slot), 512);
    tmem_relinquish();
  }
  {   // (the tile list is an upload: read in front of the wait)
    constexpr int PER = (PT_MAX_TILES + PT_THREADS - 1) / PT_THREADS;   // neighbouring tiles a thread
    int n[PER], sum = 0;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int t = tid * PER + i;
      n[i] = t < a.ntiles ? pt_units(a.tiles[t], QB) : 0;
      sum += n[i];
    }
    int up = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, up, o);
      if (lane >= o) up += v;
    }
    if (lane == 31) part[warp] = up;
    __syncthreads();
    int at = up - sum;
    for (int w = 0; w < warp; ++w) at += part[w];
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int t = tid * PER + i;
      if (t <= a.ntiles && t <= PT_MAX_TILES) base[t] = at;
      at += n[i];
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_slot;
  const B2Waits wait{&gave_up, limit};
  const int units = base[a.ntiles];
  pdl_wait();   // queries and cache rows are the kernel's in front; the scratch may still be read by an older one
  pdl_launch_dependents();
  int sent = 0;   // (producer: stages filled)

  auto produce = [&]() {   // (a warp: lanes 0-7 sixteen rows of K each, lanes 8 and 9 a half of the queries' dims)
    if (lane == 0) {
      tma_prefetch_desc(&tmap_k);
      tma_prefetch_desc(&tmap_q);
    }
    for (int u = blockIdx.x; u < units; u += gridDim.x) {
      const PtUnit x = pt_unit<QB>(a, base, u);
      if (!x.seen) continue;
      int row = 0;   // (keys behind the last token's position are not seen by anyone: any rows of the cache will do)
      const int kp = x.key0 + lane * 16;
      if (lane < 8 && kp <= x.last) row = a.block_table[(size_t)x.t.bt_row * a.bt_stride + kp / a.block_size] * a.block_size + kp % a.block_size;
      for (int g = 0; g < G; ++g, ++sent) {
        const int s = sent % C::STAGES;
        if (!wait.warp(empty_bar[s], ((sent / C::STAGES) & 1) ^ 1)) return;
        const uint32_t fb = smem_u32(&full_bar[s]), at = smem_base + s * C::STAGE_BYTES;
        if (lane == 0) mbar_arrive_expect_tx(fb, C::STAGE_BYTES);
        __syncwarp();
        // (K: a kilobyte is eight rows of half the dims, the halves alternate, so that one copy brings whole rows)
        if (lane < 8) tma_load_4d(at + lane * 4096, &tmap_k, 0, 0, 2 * g, row >> 3, fb);
        else if (lane < 10) tma_load_2d(at + PT_K_BYTES + (lane - 8) * (C::NCOL * 128), &tmap_q, (lane - 8) * 64, (g * a.T + x.q0) * 4, fb);
      }
    }
  };
  auto multiply = [&]() {   // (one thread)
    constexpr uint32_t idesc = umma_idesc_bf16(PT_KEYS, C::NCOL);
    int it = 0;
    for (int u = blockIdx.x; u < units; u += gridDim.x) {
      if (!pt_unit<QB>(a, base, u).seen) continue;
      for (int g = 0; g < G; ++g, ++it) {
        const int s = it % C::STAGES, pair = it >> 1, sl = pair % C::SLOTS;
        if ((it & 1) == 0 && !wait(slot_empty[sl], ((pair / C::SLOTS) & 1) ^ 1)) return;
        if (!wait(full_bar[s], (it / C::STAGES) & 1)) return;
        tc_fence_after();
        const uint32_t at = smem_base + s * C::STAGE_BYTES, d = tmem_base + (uint32_t)(sl * 2 * C::NCOL + (it & 1) * C::NCOL);
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          const uint64_t dk = umma_desc_sw128(at + half * 1024, 2048), dq = umma_desc_sw128(at + PT_K_BYTES + half * (C::NCOL * 128));
#pragma unroll
          for (int k = 0; k < 4; ++k) tc_mma_bf16(d, dk + (uint64_t)(2 * k), dq + (uint64_t)(2 * k), idesc, (half > 0 || k > 0) ? 1u : 0u);
        }
        tc_commit(smem_u32(&empty_bar[s]));
        if (it & 1) tc_commit(smem_u32(&slot_full[sl]));
      }
    }
  };
  auto mix = [&]() {   // sixteen warps: lane = key, four warps per lane quarter with a quarter of the tokens each
    const int quarter = warp & 3, th = warp >> 2;
    const float per_cap = a.g.softcap > 0.f ? a.g.scale / a.g.softcap : 0.f;
    const uint32_t from = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(th * CT);
    int it = 0;
    for (int u = blockIdx.x; u < units; u += gridDim.x) {
      const PtUnit x = pt_unit<QB>(a, base, u);
      if (!x.seen) continue;
      unsigned long long acc[H / 2][QT];   // heads 2 i, 2 i + 1
#pragma unroll
      for (int i = 0; i < H / 2; ++i)
#pragma unroll
        for (int t = 0; t < QT; ++t) acc[i][t] = 0ull;
#pragma unroll
      for (int g2 = 0; g2 < G / 2; ++g2, ++it) {   // (unrolled: the matrix's entries have fixed places in constant memory then, and are operands of the sums; loads of them 299 -> 212 us.  Two key/value heads at a time: a warp's way from the barrier to its scores is longer than its sums for one)
        const int sl = it % C::SLOTS;
        if (!wait.warp(slot_full[sl], (it / C::SLOTS) & 1)) return;
        tc_fence_after();
        float s[4][QT];   // heads 4 g2 ..
        {
          uint32_t r[2][CT];
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            if constexpr (CT == 8) pt_tmem_ld8(from + (uint32_t)(sl * 2 * C::NCOL + i * C::NCOL), r[i]);
            else tmem_ld16(from + (uint32_t)(sl * 2 * C::NCOL + i * C::NCOL), r[i]);
          }
          tmem_ld_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&slot_empty[sl]));
#pragma unroll
          for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 2 * QT; ++j) s[2 * i + (j & 1)][j / 2] = __uint_as_float(r[i][2 * j]) + __uint_as_float(r[i][2 * j + 1]);
        }
        if (a.g.softcap > 0.f) {   // (cap - 2 cap / (e^(2 s / cap) + 1) would lose the small scores of a high cap)
#pragma unroll
          for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int t = 0; t < QT; ++t) s[j][t] = a.g.softcap * tanhf(s[j][t] * per_cap);
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int t = 0; t < QT; ++t) s[j][t] *= a.g.scale;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const ulonglong2* row = reinterpret_cast<const ulonglong2*>(mix_of.m + (4 * g2 + j) * H);
          unsigned long long v[QT];
#pragma unroll
          for (int t = 0; t < QT; ++t) asm("mov.b64 %0, {%1, %1};" : "=l"(v[t]) : "f"(s[j][t]));
#pragma unroll
          for (int i = 0; i < H / 4; ++i) {
            const ulonglong2 w = row[i];
#pragma unroll
            for (int t = 0; t < QT; ++t) {
              fma2(acc[2 * i][t], w.x, v[t]);
              fma2(acc[2 * i + 1][t], w.y, v[t]);
            }
          }
        }
      }
      float* out = a.scores + (size_t)u * C::UNIT_FLOATS + (size_t)(th * QT) * PT_KEYS + quarter * 32 + lane;
#pragma unroll
      for (int t = 0; t < QT; ++t) {
        if (th * QT + t >= x.ntok) break;
#pragma unroll
        for (int i = 0; i < H / 2; ++i) {
          float lo, hi;
          asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(acc[i][t]));
          out[(size_t)(2 * i * QB + t) * PT_KEYS] = lo;
          out[(size_t)((2 * i + 1) * QB + t) * PT_KEYS] = hi;
        }
      }
    }
  };
  if (warp < PT_MIX_WARPS) {
    mix();
  } else if (warp == PT_MIX_WARPS) {
    produce();
  } else if (lane == 0) {
    multiply();
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (gave_up != 0 && lane == 0) {   // copies and MMAs under way end before shared memory and TMEM are given back
    if (warp == PT_MIX_WARPS) {
      for (int k = max(0, sent - C::STAGES); k < sent; ++k) b2_drain(full_bar[k % C::STAGES], (k / C::STAGES) & 1);
    } else if (warp == PT_MIX_WARPS + 1) {
      tc_commit(smem_u32(&drained));
      b2_drain(drained, 0);
    }
  }
  __syncthreads();
  if (warp == PT_MIX_WARPS + 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// A CTA: the 64 query tokens of a tile, the two heads of key/value head blockIdx.x, a warp per (head, 16 tokens).  Steps of 64 keys: V rows and every warp's own scratch rows come in a
// step ahead (cp.async).  The k index of a product stands for another key than its own -- 2 f, 2 f + 1, 2 f + 8, 2 f + 9 for keys 4 f .. 4 f + 3 -- so that a thread reads the
// four weights of a row that it owns in 16 bytes; the rows of V are picked to match.
constexpr int PV_KEYS = 64, PV_V_BYTES = PV_KEYS * PT_DIM * 2, PV_S_BYTES = 16 * PV_KEYS * 4;
constexpr int PV_SMEM = 2 * PV_V_BYTES + 8 * 2 * PV_S_BYTES;
__device__ __forceinline__ uint32_t pv_swizzle(int key) { return (uint32_t)((key & 1) | ((key >> 2) & 3) << 1); }   // the rows of one ldmatrix fall on eight chunks

__device__ __forceinline__ float pv_exp2(float v) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
  return r;
}
__device__ __forceinline__ void pv_ldmatrix_trans(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void pv_mma(float (&d)[4], const uint32_t (&x)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(x[0]), "r"(x[1]), "r"(x[2]), "r"(x[3]), "r"(b0), "r"(b1));
}

template <int H>
__global__ void __launch_bounds__(256, 2) premix_values_kernel(const PtArgs a, const bf16* v_rows, const float* turn, bf16* out) {
  using C = PtCfg<H>;
  constexpr int QB = C::QB, G = C::G;
  extern __shared__ __align__(128) uint8_t smem_raw[];
  __shared__ int part[8];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, fg = lane >> 2, ft = lane & 3;
  const int g = blockIdx.x, ti = gridDim.y - 1 - blockIdx.y;   // (the late tiles of a prompt see the most keys: they start first)
  const PrefillTile tl = a.tiles[ti];
  int first = 0;   // the tile's first unit
  for (int t = tid; t < ti; t += 256) first += pt_units(a.tiles[t], QB);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) first += __shfl_xor_sync(0xffffffffu, first, o);
  if (lane == 0) part[warp] = first;
  __syncthreads();
  first = 0;
#pragma unroll
  for (int w = 0; w < 8; ++w) first += part[w];
  pdl_wait();
  pdl_launch_dependents();
  if (tl.nrows <= 0) return;
  const int nkb = pt_key_blocks(tl), pos_hi = tl.q_pos0 + tl.nrows - 1;
  const int hd = warp >> 2, row0 = (warp & 3) * 16;   // this warp's head of the two, its first token of the tile
  const uint32_t vs = smem_u32(smem_raw), ss = vs + 2 * PV_V_BYTES + warp * (2 * PV_S_BYTES);
  const int32_t* bt = a.block_table + (size_t)tl.bt_row * a.bt_stride;
  const int last_key = tl.q_pos0 + min(row0 + 15, tl.nrows - 1);   // of this warp's queries
  const int steps = pos_hi / PV_KEYS + 1, mine = row0 < tl.nrows ? last_key / PV_KEYS + 1 : 0;   // steps with keys that this warp sees

  // scratch rows of this lane: 2 i + (lane >> 4) of the warp's sixteen; eight (QB 8) or all of them lie in one unit, the others nkb units on
  const int r1 = lane >> 4, c16 = lane & 15;
  const float* s0 = a.scores + (size_t)(first + (row0 / QB) * nkb) * C::UNIT_FLOATS + ((size_t)(2 * g + hd) * QB + row0 % QB + r1) * PT_KEYS + c16 * 4;
  const size_t s_next = row0 + 8 < tl.nrows ? (size_t)nkb * C::UNIT_FLOATS : 0;   // (no rows there: nothing is read)
  const uint32_t s_at = r1 * 256 + ((c16 ^ (r1 << 2)) << 4);
  const bf16* v0 = v_rows + (size_t)g * PT_DIM + c16 * 8;
  auto load = [&](int j) {
    const int k0 = j * PV_KEYS;
    const uint32_t vd = vs + (j & 1) * PV_V_BYTES, sd = ss + (j & 1) * PV_S_BYTES + s_at;
    if (j < mine) {
      const float* src = s0 + (size_t)(k0 / PT_KEYS) * C::UNIT_FLOATS + k0 % PT_KEYS;
#pragma unroll
      for (int i = 0; i < 8; ++i)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(sd + i * 512), "l"(src + (QB == 8 && i >= 4 ? s_next : 0) + (QB == 8 ? i & 3 : i) * 2 * PT_KEYS),
                     "r"(row0 + 2 * i + r1 < tl.nrows ? 16 : 0)
                     : "memory");
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int key = (tid >> 4) + 16 * i, kp = k0 + key;
      const bool in = kp <= pos_hi;
      const size_t row = in ? (size_t)bt[kp / a.block_size] * a.block_size + kp % a.block_size : 0;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(vd + key * 256 + ((c16 ^ pv_swizzle(key)) << 4)), "l"(v0 + row * (G * PT_DIM)), "r"(in ? 16 : 0) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  float o[16][4];
#pragma unroll
  for (int n = 0; n < 16; ++n)
#pragma unroll
    for (int e = 0; e < 4; ++e) o[n][e] = 0.f;
  float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};   // rows fg, fg + 8
  load(0);
  for (int j = 0; j < steps; ++j) {
    if (j + 1 < steps) load(j + 1);
    else asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();
    if (j < mine) {
      const int k0 = j * PV_KEYS;
      const uint32_t sd = ss + (j & 1) * PV_S_BYTES, vd = vs + (j & 1) * PV_V_BYTES;
      float s[2][16];
#pragma unroll
      for (int rr = 0; rr < 2; ++rr)
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
          asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];"
                       : "=f"(s[rr][4 * kk]), "=f"(s[rr][4 * kk + 1]), "=f"(s[rr][4 * kk + 2]), "=f"(s[rr][4 * kk + 3])
                       : "r"(sd + (fg + 8 * rr) * 256 + (((4 * kk + ft) ^ ((fg & 1) << 2)) << 4)));
      if (k0 + PV_KEYS - 1 > tl.q_pos0 + row0 || row0 + 16 > tl.nrows) {
#pragma unroll
        for (int rr = 0; rr < 2; ++rr) {
          const int tok = row0 + fg + 8 * rr, seen = tok < tl.nrows ? tl.q_pos0 + tok - k0 : -1;   // last key of the step that the row sees
#pragma unroll
          for (int e = 0; e < 16; ++e)
            if (16 * (e >> 2) + 4 * ft + (e & 3) > seen) s[rr][e] = -INFINITY;
        }
      }
      float corr[2];
#pragma unroll
      for (int rr = 0; rr < 2; ++rr) {
        float mx = s[rr][0];
#pragma unroll
        for (int e = 1; e < 16; ++e) mx = fmaxf(mx, s[rr][e]);
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
        const float mn = fmaxf(m[rr], mx), ref = mn == -INFINITY ? 0.f : mn;
        corr[rr] = m[rr] == -INFINITY ? 0.f : pv_exp2((m[rr] - ref) * 1.4426950408889634f);
        m[rr] = mn;
        float sum = 0.f;
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          s[rr][e] = pv_exp2((s[rr][e] - ref) * 1.4426950408889634f);
          sum += s[rr][e];
        }
        l[rr] = l[rr] * corr[rr] + sum;
      }
      if (__any_sync(0xffffffffu, corr[0] != 1.f || corr[1] != 1.f)) {
#pragma unroll
        for (int n = 0; n < 16; ++n) {
          o[n][0] *= corr[0]; o[n][1] *= corr[0];
          o[n][2] *= corr[1]; o[n][3] *= corr[1];
        }
      }
      const int k = lane & 15, key = k < 8 ? 4 * (k >> 1) + (k & 1) : 4 * ((k - 8) >> 1) + 2 + (k & 1);
      // A weight of 0 times an infinity is a NaN: what lies behind the last key that the warp's sixteen queries see stays out of their products.
      const int last_seen = last_key - k0;   // (>= 0)
      auto product = [&](int kk, auto at_end) {   // keys 16 kk .. of the step; at_end: those behind `last_seen` count as zeros
        uint32_t hi[4], lo[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {   // rows fg, fg + 8 of keys 4 ft, 4 ft + 1, then of 4 ft + 2, 4 ft + 3
          const float x = s[i & 1][4 * kk + 2 * (i >> 1)], y = s[i & 1][4 * kk + 2 * (i >> 1) + 1];
          hi[i] = pack_bf16x2(x, y);
          lo[i] = pack_bf16x2(x - bf16lo(hi[i]), y - bf16hi(hi[i]));
        }
        uint32_t keep[2];   // of the pairs of keys 4 ft, 4 ft + 1 and 4 ft + 2, 4 ft + 3
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int left = last_seen - (16 * kk + 4 * ft + 2 * i);
          keep[i] = left >= 1 ? 0xffffffffu : left == 0 ? 0xffffu : 0u;
        }
        const uint32_t vrow = vd + (16 * kk + key) * 256, sw = pv_swizzle(key);   // (16 kk does not move the swizzle)
#pragma unroll
        for (int nb = 0; nb < 8; nb += 2) {   // (four sums at a time: a product waits for the one before it on the same sum)
          uint32_t vb[2][4];
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            pv_ldmatrix_trans(vb[i], vrow + (((uint32_t)(2 * (nb + i) + (lane >> 4)) ^ sw) << 4));
            if constexpr (decltype(at_end)::value) {
#pragma unroll
              for (int r = 0; r < 4; ++r) vb[i][r] &= keep[r & 1];
            }
          }
#pragma unroll
          for (int i = 0; i < 4; ++i) pv_mma(o[2 * nb + i], lo, vb[i >> 1][2 * (i & 1)], vb[i >> 1][2 * (i & 1) + 1]);
#pragma unroll
          for (int i = 0; i < 4; ++i) pv_mma(o[2 * nb + i], hi, vb[i >> 1][2 * (i & 1)], vb[i >> 1][2 * (i & 1) + 1]);
        }
      };
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) {
        if (16 * kk + 15 <= last_seen) product(kk, std::false_type{});
        else if (16 * kk <= last_seen) product(kk, std::true_type{});
      }
    }
    __syncthreads();   // this step's buffers are read: the load of the step after the next may write them
  }
#pragma unroll
  for (int rr = 0; rr < 2; ++rr) {
    l[rr] += __shfl_xor_sync(0xffffffffu, l[rr], 1);
    l[rr] += __shfl_xor_sync(0xffffffffu, l[rr], 2);
    const int tok = row0 + fg + 8 * rr;
    if (tok >= tl.nrows) continue;
    const float inv = 1.0f / l[rr];
    bf16* dst = out + ((size_t)(tl.q_row0 + tok) * H + 2 * g + hd) * PT_DIM + 2 * ft;
    const float* cs = turn != nullptr ? turn + (size_t)(tl.q_row0 + tok) * PT_DIM + 2 * ft : nullptr;
#pragma unroll
    for (int n = 0; n < 8; ++n) {
      float u[2], w[2];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        u[e] = o[n][2 * rr + e];
        w[e] = o[n + 8][2 * rr + e];
      }
      if (cs != nullptr) {   // turned back by the query's position: the pair (d, d + 64) by minus the angle
        const float2 c = *reinterpret_cast<const float2*>(cs + 8 * n), sn = *reinterpret_cast<const float2*>(cs + 64 + 8 * n);
        const float u0 = u[0], u1 = u[1];
        u[0] = u0 * c.x + w[0] * sn.x;
        u[1] = u1 * c.y + w[1] * sn.y;
        w[0] = w[0] * c.x - u0 * sn.x;
        w[1] = w[1] * c.y - u1 * sn.y;
      }
      *reinterpret_cast<uint32_t*>(dst + 8 * n) = pack_bf16x2(u[0] * inv, u[1] * inv);
      *reinterpret_cast<uint32_t*>(dst + 64 + 8 * n) = pack_bf16x2(w[0] * inv, w[1] * inv);
    }
  }
}

template <int H>
int launch_premix_tc(const bf16* q_planes, const bf16* k_cache, const bf16* v_cache, int64_t cache_rows, const HeadsGeom& g, const float* talk_host, const float* turn,
                     const int32_t* block_table, int bt_stride, int block_size, const PrefillTile* tiles, const PrefillTile* tiles_host, int ntiles, bf16* out, int T,
                     float* scratch, size_t scratch_floats, const B2WaitLimit& wait, cudaStream_t s) {
  using C = PtCfg<H>;
  CUtensorMap tk, tq;
  const uint64_t ld = (uint64_t)C::G * PT_DIM * 2, k_dims[4] = {64, 8, 2 * C::G, (uint64_t)cache_rows / 8}, k_strides[3] = {ld, 128, 8 * ld};
  const uint32_t k_box[4] = {64, 8, 2, 2};
  int rc = b2_make_tmap_bf16_swizzled(&tk, k_cache, 4, k_dims, k_strides, k_box);
  if (rc != 0) return rc;
  rc = b2_make_tmap_bf16(&tq, q_planes, (uint64_t)C::G * T * 4, PT_DIM, PT_DIM, C::NCOL);
  if (rc != 0) return rc;
  static B2PerDeviceOnce once;
  if (once.need()) {
    B2_CUDA_OK(cudaFuncSetAttribute(premix_scores_kernel<H>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES));
    B2_CUDA_OK(cudaFuncSetAttribute(premix_values_kernel<H>, cudaFuncAttributeMaxDynamicSharedMemorySize, PV_SMEM));
  }
  PtMix<H> mix;
  for (int i = 0; i < H * H; ++i) mix.m[(i % H) * H + i / H] = talk_host[i];
  int sms = 0, dev = 0;
  B2_CUDA_OK(cudaGetDevice(&dev));
  B2_CUDA_OK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const size_t cap = scratch_floats / C::UNIT_FLOATS;
  for (int t0 = 0; t0 < ntiles;) {   // whole tiles that fit the scratch
    size_t units = 0;
    int n = 0;
    while (t0 + n < ntiles && n < PT_MAX_TILES && units + pt_units(tiles_host[t0 + n], C::QB) <= cap) units += pt_units(tiles_host[t0 + n++], C::QB);
    B2_REQUIRE(n > 0, "heads_premix_tc: a tile of %d keys does not fit %zu numbers of scratch", tiles_host[t0].q_pos0 + tiles_host[t0].nrows, scratch_floats);
    if (units > 0) {
      const PtArgs a{g, block_table, bt_stride, block_size, tiles + t0, n, T, scratch};
      B2_CUDA_OK(b2_launch(premix_scores_kernel<H>, dim3((unsigned)std::min<size_t>(units, sms)), dim3(PT_THREADS), C::SMEM_BYTES, s, tk, tq, a, mix, wait));
      B2_CUDA_OK(b2_launch(premix_values_kernel<H>, dim3(C::G, n), dim3(256), PV_SMEM, s, a, v_cache, turn, out));
    }
    t0 += n;
  }
  return 0;
}

}  // namespace

// Sizes: a mix thread holds heads x QB / 4 running sums (64 registers' worth at 16 and 32 heads, beside the scores of two key/value heads) and the matrix's entries as operands at fixed
// places, so a head count is a kernel of its own; heads are swept in fours; a score's columns are laid out for two heads of a key/value head, its operand rows for 128 dims, and the values'
// turn back pairs d with d + 64.  Others keep attn_heads.cu.  Sixteen rows of a page are one copy of K: pages in multiples of that.
bool heads_premix_tc_ok(const HeadsGeom& g, int block_size) {
  return (g.heads == 8 || g.heads == 16 || g.heads == 32) && g.kv_heads * 2 == g.heads && g.dim == 128 && g.vdim == 128 && g.window <= 0 && g.rot_dims % 8 == 0 && block_size > 0 && block_size % 16 == 0;
}

// Room for the units of a whole call, at most 512 MB (4 096 units of 32 heads).  4 x 1024 tokens of 32 heads, 2 304 units: in 192 MB 68 us more than with room for all (two launches of each
// kernel, and their last waves).
size_t heads_premix_tc_scratch_floats(const HeadsGeom& g, int max_tokens, int max_context) {
  const int qb = g.heads == 32 ? 8 : 16;
  const size_t unit = (size_t)g.heads * qb * PT_KEYS, blocks = ((size_t)max_context + PT_KEYS - 1) / PT_KEYS + 1;
  const size_t most = (size_t)128 * 1024 * 1024 / unit, tile = 64 / qb * blocks;
  return std::min(most, std::max(tile, ((size_t)max_tokens / qb + 64) * blocks)) * unit;
}

// A call takes this form where all of its tiles fit the scratch and where it is the faster one.  Behind long contexts the scratch holds few tiles' scores: a launch of premix_values then is a
// CTA per tile and key/value head, 68 ns a key of its longest context whatever else the chip could do, and the next launch waits for it.  The kernels of attn_heads.cu walk a context with
// a CTA (a cluster) per sixteen queries, slower but all of them at the same time.  ms a call of one layer, theirs / this: 32 heads, 64 tokens behind 60 000: 16.8 / 5.1, 384: 26.7 / 27.1,
// 3000: 158 / 215; 3000 behind 16 000: 45.0 / 24.7; 16 heads, 512 behind 60 000: 18.4 / 17.2, 3000: 37.2 / 105, 3000 behind 16 000: 10.8 / 10.5; 8 heads, 768 behind 32 000: 5.4 / 4.8, 1024:
// 5.5 / 7.1.  The estimates pick the faster form, to 3 %, at all of 270 points (64 - 4096 tokens behind 1000 - 60 000).
bool heads_premix_tc_pays(const HeadsGeom& g, const PrefillTile* tiles_host, int ntiles, size_t scratch_floats) {
  const int qb = g.heads == 32 ? 8 : 16;
  const long cap = (long)(scratch_floats / ((size_t)g.heads * qb * PT_KEYS));
  const double unit_ns = g.heads == 32 ? 92 : g.heads == 16 ? 75 : 30;        // of premix_scores, the chip full
  const double chain_ns = g.heads == 32 ? 420 : g.heads == 16 ? 306 : 162;   // a key, of a walk over a context there
  const long walks = g.heads == 32 ? 32 : 148;                                // at the same time
  double here = 0, keys_sum = 0;
  long units = 0, longest = 0, launch_longest = 0, groups = 0;
  int n = 0;
  for (int t = 0; t < ntiles; ++t) {
    const PrefillTile& tl = tiles_host[t];
    const long u = pt_units(tl, qb), keys = (long)tl.q_pos0 + tl.nrows, k16 = (tl.nrows + 15) / 16;
    if (u > cap) return false;
    if (tl.nrows <= 0) continue;
    if (units + u > cap || n == PT_MAX_TILES) {   // (the launches of launch_premix_tc)
      here += 68.0 * launch_longest + unit_ns * units;
      units = launch_longest = n = 0;
    }
    units += u;
    ++n;
    launch_longest = std::max(launch_longest, keys);
    longest = std::max(longest, keys);
    groups += k16;
    keys_sum += (double)k16 * keys;
  }
  if (groups == 0) return true;
  here += 68.0 * launch_longest + unit_ns * units;
  const double there = chain_ns * std::max((double)longest, keys_sum / groups * ((groups + walks - 1) / walks));
  return here <= there;
}

int launch_heads_premix_tc(const bf16* q_planes, const bf16* k_cache, const bf16* v_cache, int64_t cache_rows, const HeadsGeom& g, const float* talk_host, const float* turn,
                           const int32_t* block_table, int bt_stride, int block_size, const PrefillTile* tiles, const PrefillTile* tiles_host, int ntiles, bf16* out, int T,
                           float* scratch, size_t scratch_floats, const B2WaitLimit& wait, cudaStream_t s) {
  if (T <= 0 || ntiles <= 0) return 0;
  B2_REQUIRE(heads_premix_tc_ok(g, block_size) && talk_host != nullptr && scratch != nullptr, "heads_premix_tc: %d heads of %d + %d on %d have no such form", g.heads, g.dim, g.vdim, g.kv_heads);
  auto f = g.heads == 8 ? launch_premix_tc<8> : g.heads == 16 ? launch_premix_tc<16> : launch_premix_tc<32>;
  return f(q_planes, k_cache, v_cache, cache_rows, g, talk_host, turn, block_table, bt_stride, block_size, tiles, tiles_host, ntiles, out, T, scratch, scratch_floats, wait, s);
}

}  // namespace b2
