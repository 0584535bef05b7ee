// attn_prefill_tc.cu -- causal prefill attention over the paged KV cache on the 5th-generation tensor cores
// (HF:integrations/sdpa_attention.py:40-104 at T > 1; eager form HF:models/qwen3/modeling_qwen3.py:196-218).
// Same contract and the same tile list as attn_prefill.cu (the mma.sync kernel, kept as the cross-check and for
// callers without a tensor map): fp32 scores, fp32 online-softmax statistics, probabilities rounded to bf16 for P.V,
// the row sum from the unrounded fp32 probabilities, fp32 accumulation, one multiply by 1/l, one rounding.
//
// A UNIT is 128 MMA rows of one kv head: one 64-query tile x both query heads of the GQA group (row r = head (r >> 6), query
// token (r & 63)), or, for models with one query head per kv head (pair_mode), two consecutive 64-query tiles of that head.
// A CTA takes one unit, and two CTAs share an SM; beside a rotated key piece (below) two consecutive units of a sequence, for which the keys come in once:
//   S[128 x 128 keys]  = Q[128 x 128 dims] . K^T      tcgen05.mma, A and B K-major from shared memory, S in TMEM
//   softmax            : 128 threads per unit, one per row, 64 keys at a time: tcgen05.ld, scale / mask, row maximum, probabilities; P
//                        (bf16) goes back into TMEM over S columns that have been read
//   O[128 x 128 dims] += P[128 x 128 keys] . V        A from TMEM; V is the B operand in MN-major form: the page layout
//                        [key][128 dims] with its 16-byte chunks XOR-swizzled by (key & 7) IS the canonical MN-major
//                        128-byte-swizzle layout once the two 64-dim halves of every row are stored apart; O stays in TMEM
// K and V pages come in through TMA (a 2-D map over the page pool, box 64 dims x 16 keys, no TMA swizzle: the pool is
// stored swizzled): half h of key row k lands at [h][k][128 bytes], which serves as K-major B for Q.K^T and as
// MN-major B for P.V without any re-layout.
//
// What bounds it: per unit and key tile the MMAs take about 1 050 cycles and the exponentials 1 024 (16 a cycle and SM), and within a unit everything
// waits for something: S for K and for the P.V that reads the columns it is written to (only MMAs on one accumulator are ordered by themselves), the
// probabilities for S, P.V for a half tile of probabilities.  What fills the gaps is another unit on the same SM.  As a CTA of its own (96 KB of shared memory
// and 256 TMEM columns each, K and V in single buffers) it does so at least as well as in turn within one CTA (192 KB, K and V in two stages, one softmax thread
// per row in both), needs no neighbour of the same sequence, and a launch that fills the chip less than twice keeps all SMs.  us per launch, 8 kv heads of 2,
// with one unit per CTA, with two, and with one unit whose P went through shared memory over K (two threads per row, two passes over S):
//   12 prompts of 133 to 4096 tokens    271   284   384        40 prompts of 64 tokens              16.2   22.9   16.8
//   one prompt of 4096                  110   113   163        40 x 64 behind 1000 cached tokens    56.8   85.4   77.5
//   one prompt of 2048                 40.8  40.5  60.6        20 x 192 behind 1000                 61.5   76.5   86.6
//   one prompt of 1600                 32.9  31.2  47.6        24 x 64 behind 4000                  87.6   130    130
//   one prompt of 1216                 24.4  24.8  33.0        4 x 448 behind 2048                  53.9   77.0   76.9
//
// rot (layers whose heads share a rotated key piece): S gets a third block of 64 dims, Q from fp32 queries, K from a pool of
// [page][16][64] rows that all heads read; a per-head sink joins the row sum.
#include "kernels.h"

namespace b2 {

namespace {

constexpr int PT_TQ = 64;                    // query tokens per tile
constexpr int PT_M = 128;                    // MMA rows of a unit
constexpr int PT_BN = 128;                   // keys per key tile
constexpr int PT_SN = 64;                    // keys of half a tile: what a softmax thread holds at a time
constexpr int PT_HD = 128;
constexpr int PT_BLOCK = PT_BN * 128;        // 128 rows x 64 dims (128 bytes): 16 KB
constexpr int PT_MAX_PAGES = 1024;           // longest block-table row (16 K tokens of context)
// NK: 64-dim blocks of Q . K^T (3 with a rotated piece).  NU: units of a CTA.  One unit: single stages, 96 or 128 KB.  Two units (beside three blocks):
// K is two stages deep, 224 KB.
template <int NK, int NU>
struct PtCfg {
  static constexpr int KS = NU, VS = 1;
  static constexpr int Q_BYTES = NK * PT_BLOCK, K_BYTES = NK * PT_BLOCK, V_BYTES = 2 * PT_BLOCK;
  static constexpr int K_OFF = NU * Q_BYTES, V_OFF = K_OFF + KS * K_BYTES;
  static constexpr int BAR_OFF = V_OFF + VS * V_BYTES;
  static constexpr int SMEM = BAR_OFF + 256 + 1024;
  static constexpr int TMEM_COLS = 256 * NU;               // S of every unit (P over its first half), then O of every unit
  static constexpr uint32_t O_COL = 128 * NU;
  static constexpr int MMA_WARP = 4 * NU, LOAD_WARPS = 3, THREADS = 32 * (MMA_WARP + 1 + LOAD_WARPS);
};

// K-major, 128-byte swizzle (rows of 128 bytes, 8-row groups 1024 bytes apart): Q and K tiles
__device__ __forceinline__ uint64_t pt_desc_k(uint32_t smem_addr) { return umma_desc_sw128(smem_addr); }
// MN-major, 128-byte swizzle: the V tile.  64 contiguous dims (128 bytes) per key, 8-key groups 1024 bytes apart
// (stride byte offset), the other 64 dims 16 KB further on (leading byte offset).
__device__ __forceinline__ uint64_t pt_desc_mn(uint32_t smem_addr) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr & 0x3FFFFu) >> 4);
  d |= (uint64_t)(PT_BLOCK >> 4) << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}
// D[tmem] (+)= A[tmem] * B[smem]: A is bf16, two neighbouring k in a 32-bit column
__device__ __forceinline__ void pt_mma_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n"
      "}\n" ::"r"(tmem_d),
      "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
// waits for the loads under way and ties their registers to the wait: nothing that uses them moves in front of it
__device__ __forceinline__ void pt_ld_wait(uint32_t (&r)[32]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]), "+r"(r[10]),
                 "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]), "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]),
                 "+r"(r[21]), "+r"(r[22]), "+r"(r[23]), "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]), "+r"(r[29]), "+r"(r[30]), "+r"(r[31])
               :
               : "memory");
}
__device__ __forceinline__ float pt_ex2(float x) {  // 2^x, one MUFU (results below 2^-126 flush to zero: they are probabilities)
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
typedef unsigned long long pt_x2;   // two fp32 numbers in a register pair
__device__ __forceinline__ pt_x2 pt_pair(float x, float y) {
  pt_x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ float2 pt_split(pt_x2 v) {
  float2 f;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
  return f;
}
__device__ __forceinline__ pt_x2 pt_fma2(pt_x2 x, pt_x2 y, pt_x2 z) {
  pt_x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(x), "l"(y), "l"(z));
  return r;
}
__device__ __forceinline__ pt_x2 pt_add2(pt_x2 x, pt_x2 y) {
  pt_x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(x), "l"(y));
  return r;
}
__device__ __forceinline__ float pt_max3(float x, float y, float z) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(x), "f"(y), "f"(z));
  return r;
}
__device__ __forceinline__ void pt_ld16(uint32_t taddr, uint32_t (&r)[16]) {   // loads and waits
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n\ttcgen05.wait::ld.sync.aligned;"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]),
                 "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
               : "r"(taddr)
               : "memory");
}
constexpr uint32_t PT_IDESC_QK = umma_idesc_bf16(PT_M, PT_BN);                // both operands K-major
constexpr uint32_t PT_IDESC_PV = umma_idesc_bf16(PT_M, PT_HD) | (1u << 16);  // B (V) MN-major

// Threads: four softmax warps per unit (a thread per row), then the MMA issuer (and TMEM allocator), then three warps for the TMA loads (a
// cp.async.bulk.tensor costs about 100 cycles to issue, and a key tile needs 32).
constexpr float PT_RESCALE = 8.0f;  // log2 units: the reference maximum is raised only when the row maximum grew by 2^8

struct PtArgs {
  const bf16* q;
  const int32_t* block_table;
  int bt_stride;
  const PrefillTile* tiles;
  bf16* out;
  int nq, nkv, units;
  float scale_log2;
  int window, pair_mode, head_step, chunk;
  const float* q_rot;      // [tokens][heads][rot_dim]
  int rot_dim;
  const float* sink;       // [heads] or null
  B2WaitLimit wait;
};

template <int NK, int NU>
__global__ void __launch_bounds__(PtCfg<NK, NU>::THREADS, NU == 1 && NK == 2 ? 2 : 1)
attn_prefill_tc_kernel(const __grid_constant__ CUtensorMap tmap_k, const __grid_constant__ CUtensorMap tmap_v, const __grid_constant__ CUtensorMap tmap_r, PtArgs a) {
  using C = PtCfg<NK, NU>;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t k_s = base + C::K_OFF, v_s = base + C::V_OFF;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem_raw + (base - smem_u32(smem_raw)) + C::BAR_OFF);
  // per unit: q_full, s_full, o_half (P.V of a tile's first half has landed), o_full; per unit and half: p_full; per stage: k / v full and free
  uint64_t *q_full = bars, *s_full = bars + 2, *o_half = bars + 4, *o_full = bars + 6, *p_full = bars + 8, *k_full = bars + 12, *k_free = bars + 14, *v_full = bars + 16, *v_free = bars + 18;
  uint64_t& drained = bars[20];
  uint32_t& tmem_slot = *reinterpret_cast<uint32_t*>(bars + 21);
  volatile uint32_t& gave_up = *reinterpret_cast<volatile uint32_t*>(bars + 22);
  const B2Waits wait{&gave_up, a.wait};
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int kvh = blockIdx.y;
  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&q_full[i]), PT_M);
      mbar_init(smem_u32(&s_full[i]), 1);
      mbar_init(smem_u32(&o_half[i]), 1);
      mbar_init(smem_u32(&o_full[i]), 1);
      mbar_init(smem_u32(&k_full[i]), 1);
      mbar_init(smem_u32(&k_free[i]), 1);
      mbar_init(smem_u32(&v_full[i]), 1);
      mbar_init(smem_u32(&v_free[i]), 1);
    }
    for (int i = 0; i < 4; ++i) mbar_init(smem_u32(&p_full[i]), PT_M);
    mbar_init(smem_u32(&drained), 1);
    gave_up = 0;
    mbar_fence_init();
  }
  // All 512 columns (two units) are taken only when every CTA of the kernel in front has ended, and before the kernel behind may start its CTAs
  if (NU == 2) pdl_wait();
  if (warp == C::MMA_WARP) {
    tmem_alloc(smem_u32(&tmem_slot), C::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  if (NU == 1) pdl_wait();  // q and the newest K/V rows come from the kernel before this one
  if (threadIdx.x == 0) pdl_launch_dependents();

  // Blocks are dispatched in index order and a unit late in its sequence has the most key tiles: walking the list backwards starts the long
  // CTAs first and leaves the short ones for the kernel's last wave.  In pair_mode the host pads every sequence to an even number of tiles (a tile with
  // nrows == 0), so tiles 2u and 2u + 1 of a unit belong together.  head_step 1 (pair_mode only): queries and outputs hold the real heads side by side; 2:
  // an all-zero partner head stands behind every head (its rows are not written: the output projection's columns for them are zeros).
  const int blk = gridDim.x - 1 - blockIdx.x;
  auto tile_of = [&](int u, int half) { return a.tiles[a.pair_mode ? 2 * u + half : u]; };
  const int u_first = NU * blk, u_last = min(NU * blk + NU - 1, a.units - 1);
  bool together = false;   // two units that continue one another share the key tiles; else they go one after the other
  if (u_last > u_first) {
    const PrefillTile x = tile_of(u_first, a.pair_mode ? 1 : 0), y = tile_of(u_last, 0);
    together = x.bt_row == y.bt_row && x.nrows == PT_TQ && y.q_pos0 == x.q_pos0 + PT_TQ && y.nrows > 0;
  }
  const int n_items = together ? 1 : u_last - u_first + 1;
  struct Item {
    int u[2];            // second -1: none
    int lo[2], hi[2];    // key tiles [lo, hi) of each unit: its rows meet no others (a value that is not finite would reach them through a weight of 0).  The
                         // second starts and ends no earlier than the first, and starts no later than that ends: keys from lo[0] to n_kt come in
    int n_kt;
    const int32_t* bt;
    __device__ __forceinline__ bool has(int k, int kt) const { return u[k] >= 0 && kt >= lo[k] && kt < hi[k]; }
  };
  auto item_of = [&](int i) {
    Item it;
    it.u[0] = u_first + i;
    it.u[1] = together ? u_last : -1;
    for (int k = 0; k < 2; ++k) {
      it.lo[k] = it.hi[k] = 0;
      if (it.u[k] < 0) continue;
      const PrefillTile f = tile_of(it.u[k], 0), l = tile_of(it.u[k], 1);
      it.lo[k] = first_seen_key(f.q_pos0, a.window, a.chunk) / PT_BN;
      it.hi[k] = (max(f.q_pos0 + f.nrows, l.nrows > 0 ? l.q_pos0 + l.nrows : 0) + PT_BN - 1) / PT_BN;
      if (k == 0) it.bt = a.block_table + (size_t)f.bt_row * a.bt_stride;
    }
    it.n_kt = max(it.hi[0], it.hi[1]);
    return it;
  };

  int k_sent = 0, v_sent = 0;   // (loaders: key tiles whose pages this warp has asked for)
  auto load_tiles = [&]() {
    // ---- loaders: each takes three (the last: two) of a key tile's eight pages; a tile's K goes out one tile ahead of its V ----
    const int j = warp - C::MMA_WARP - 1, p0 = 3 * j, np = min(3, 8 - p0);
    int n = 0;   // key tiles so far
    for (int i = 0; i < n_items; ++i) {
      const Item it = item_of(i);
      auto page_ids = [&](int kt) {   // lane p: page p of this warp's; past the sequence the null page 0
        const int at = kt * (PT_BN / 16) + p0 + min(lane, 2);
        return kt < it.n_kt && at < a.bt_stride && p0 + lane < 8 ? it.bt[at] : 0;
      };
      auto load = [&](bool is_v, int kn, int ids) {
        const int stages = is_v ? C::VS : C::KS, st = kn % stages;
        if (kn >= stages && !wait.warp(is_v ? v_free[st] : k_free[st], (kn / stages - 1) & 1)) return false;
        const uint32_t fb = smem_u32(is_v ? &v_full[st] : &k_full[st]);
        const uint32_t dst = (is_v ? v_s + st * C::V_BYTES : k_s + st * C::K_BYTES) + (uint32_t)(p0 * 16 * 128);
        if (lane == 0 && j == 0) mbar_arrive_expect_tx(fb, is_v ? C::V_BYTES : C::K_BYTES);  // the other warps only add bytes
#pragma unroll
        for (int pg = 0; pg < 3; ++pg) {
          const int page = __shfl_sync(0xffffffffu, ids, pg);
          if (lane == 0 && pg < np) {
            const int row0 = (page * a.nkv + kvh) * 16;
            const CUtensorMap* tm = is_v ? &tmap_v : &tmap_k;
            tma_load_2d(dst + pg * 16 * 128, tm, 0, row0, fb);
            tma_load_2d(dst + PT_BLOCK + pg * 16 * 128, tm, 64, row0, fb);
            if (NK == 3 && !is_v) tma_load_2d(dst + 2 * PT_BLOCK + pg * 16 * 128, &tmap_r, 0, page * 16, fb);
          }
        }
        __syncwarp();
        (is_v ? v_sent : k_sent) = kn + 1;
        return true;
      };
      int ids = page_ids(it.lo[0]);
      if (!load(false, n, ids)) return;
      for (int kt = it.lo[0]; kt < it.n_kt; ++kt, ++n) {
        const int next = page_ids(kt + 1);
        if (NU == 2 && kt + 1 < it.n_kt && !load(false, n + 1, next)) return;
        if (!load(true, n, ids)) return;
        if (NU == 1 && kt + 1 < it.n_kt && !load(false, n + 1, next)) return;
        ids = next;
      }
    }
  };
  auto multiply = [&]() {   // (one thread)
    int n = 0;                 // key tiles that came in so far
    int done[2] = {0, 0};      // key tiles of each unit so far
    auto scores = [&](int u, int kn) {   // S(u) = Q(u) . K^T
      const uint32_t ks = k_s + (uint32_t)(kn % C::KS) * C::K_BYTES, qs = base + (uint32_t)u * C::Q_BYTES;
#pragma unroll
      for (int kb = 0; kb < NK; ++kb) {
        const uint64_t da = pt_desc_k(qs + kb * PT_BLOCK), db = pt_desc_k(ks + kb * PT_BLOCK);
#pragma unroll
        for (int k = 0; k < 4; ++k) tc_mma_bf16(tmem + 128u * u, da + (uint64_t)(2 * k), db + (uint64_t)(2 * k), PT_IDESC_QK, (kb | k) ? 1u : 0u);
      }
      tc_commit(smem_u32(&s_full[u]));
    };
    for (int i = 0; i < n_items; ++i) {
      const Item it = item_of(i);
#pragma unroll
      for (int u = 0; u < NU; ++u)
        if (it.u[u] >= 0 && !wait(q_full[u], i & 1)) return;
      if (!wait(k_full[n % C::KS], (n / C::KS) & 1)) return;
      tc_fence_after();
#pragma unroll
      for (int u = 0; u < NU; ++u)
        if (it.has(u, it.lo[0])) scores(u, n);
      tc_commit(smem_u32(&k_free[n % C::KS]));
      for (int kt = it.lo[0]; kt < it.n_kt; ++kt, ++n) {
        const uint32_t vs = v_s + (uint32_t)(n % C::VS) * C::V_BYTES;
        bool v_in = false, k_in = false;
#pragma unroll
        for (int u = 0; u < NU; ++u) {
          const bool now = it.has(u, kt), next = it.has(u, kt + 1);
          // O (+)= P . V : 8 MMAs of 16 keys, the first half of the keys as soon as their P stands.  O stays in TMEM across key tiles; the softmax
          // threads rescale it in place when a row's reference maximum moves.
          if (now) {
            for (int half = 0; half < 2; ++half) {
              if (!wait(p_full[2 * u + half], done[u] & 1)) return;
              if (!v_in && !wait(v_full[n % C::VS], (n / C::VS) & 1)) return;
              v_in = true;
              tc_fence_after();
#pragma unroll
              for (int k = 4 * half; k < 4 * half + 4; ++k)
                pt_mma_ts(tmem + C::O_COL + 128u * u, tmem + 128u * u + 8u * k, pt_desc_mn(vs + (uint32_t)(k * 16 * 128)), PT_IDESC_PV, (kt > it.lo[u] || k) ? 1u : 0u);
              if (half == 0) tc_commit(smem_u32(&o_half[u]));
            }
            if (u == NU - 1 || !it.has(1, kt)) tc_commit(smem_u32(&v_free[n % C::VS]));
            tc_commit(smem_u32(&o_full[u]));
          }
          if (next) {   // the next S takes this P's place, which P.V still reads: MMAs on different accumulators have no order by themselves
            if (!k_in && !wait(k_full[(n + 1) % C::KS], ((n + 1) / C::KS) & 1)) return;
            k_in = true;
            if (now && !wait(o_full[u], done[u] & 1)) return;
            tc_fence_after();
            scores(u, n + 1);
            if (u == NU - 1 || !it.has(1, kt + 1)) tc_commit(smem_u32(&k_free[(n + 1) % C::KS]));
          }
          if (now) ++done[u];
        }
      }
    }
  };
  auto weigh = [&]() {
    // ---- softmax: unit u = warp / 4; thread r owns MMA row r = (head r >> 6, query token r & 63), in pair_mode (tile r >> 6, token r & 63) ----
    const int u = warp >> 2, r = threadIdx.x & 127, t = r & 63;
    const int h = a.pair_mode ? 0 : r >> 6;
    const uint32_t srow = tmem + ((uint32_t)((warp & 3) * 32) << 16) + 128u * u, orow = tmem + ((uint32_t)((warp & 3) * 32) << 16) + C::O_COL + 128u * u;
    int n = 0;   // key tiles of this unit so far
    for (int i = 0; i < n_items; ++i) {
      const Item it = item_of(i);
      const int unit = u == 0 ? it.u[0] : it.u[1], lo = u == 0 ? it.lo[0] : it.lo[1], hi = u == 0 ? it.hi[0] : it.hi[1];
      if (unit < 0) continue;
      const PrefillTile tile_a = tile_of(unit, 0), tile_b = tile_of(unit, 1);
      const PrefillTile mt = (r >> 6) ? tile_b : tile_a;  // the tile this row belongs to
      const bool row_ok = t < mt.nrows;
      const int qpos = mt.q_pos0 + t, row_kv_len = mt.q_pos0 + mt.nrows;
      // stage Q: rows in the K-major swizzled layout, 16 bytes per thread and step (rows past the tile are zeros)
      const uint32_t qs = base + (uint32_t)u * C::Q_BYTES;
#pragma unroll
      for (int k = 0; k < 16; ++k) {  // 16 cp.async per thread, all in flight together
        const int idx = r + k * 128, row = idx >> 4, c = idx & 15, rh = row >> 6, rt = row & 63;
        const bool in = rt < (rh ? tile_b : tile_a).nrows;
        const bf16* src = a.q + ((size_t)((rh ? tile_b : tile_a).q_row0 + (in ? rt : 0)) * a.nq + kvh * a.head_step + (a.pair_mode ? 0 : rh)) * PT_HD + c * 8;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(qs + (c >> 3) * PT_BLOCK + row * 128 + (((c & 7) ^ (row & 7)) << 4)), "l"(src), "r"(in ? 16 : 0)
                     : "memory");
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
      if constexpr (NK == 3) {   // the rotated piece: fp32 rows of rot_dim numbers, rounded here; zeros behind them
        for (int k = 0; k < 8; ++k) {
          const int idx = r + k * 128, row = idx >> 3, c = idx & 7, rh = row >> 6, rt = row & 63;
          const bool in = rt < (rh ? tile_b : tile_a).nrows;
          const float* src = a.q_rot + ((size_t)((rh ? tile_b : tile_a).q_row0 + (in ? rt : 0)) * a.nq + kvh * a.head_step + (a.pair_mode ? 0 : rh)) * a.rot_dim;
          float v[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) v[e] = in && c * 8 + e < a.rot_dim ? src[c * 8 + e] : 0.f;
          const uint4 pk = pack8(v);
          asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(qs + 2 * PT_BLOCK + row * 128 + ((c ^ (row & 7)) << 4)), "r"(pk.x), "r"(pk.y), "r"(pk.z), "r"(pk.w) : "memory");
        }
      }
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      fence_proxy_async();
      mbar_arrive(smem_u32(&q_full[u]));

      // m_ref: the value the probabilities of this row are scaled by, 2^(s - m_ref).  It follows the running row maximum
      // lazily -- only when the maximum has grown by more than PT_RESCALE -- so that most key tiles leave O (in TMEM)
      // untouched; probabilities then reach 2^8 at most, and l and O carry the same factor, which cancels in O / l.
      float m_ref = -INFINITY;
      pt_x2 l2[2] = {0ull, 0ull};   // running sums
      // Valid keys of this row are a contiguous range [lo_col, hi_col] (causal bound, sequence end, window).  Half a tile that lies wholly
      // inside the range of EVERY row of the unit takes no per-element masks.
      const int hi_col = row_ok ? min(qpos, row_kv_len - 1) : -1;
      const int lo_col = first_seen_key(qpos, a.window, a.chunk);
      const bool all_rows = tile_a.nrows == PT_TQ && tile_b.nrows == PT_TQ;
      const int lo_all = first_seen_key(tile_b.q_pos0 + PT_TQ - 1, a.window, a.chunk);
      const pt_x2 sc2 = pt_pair(a.scale_log2, a.scale_log2);
      for (int kt = lo; kt < hi; ++kt, ++n) {
        if (!wait.warp(s_full[u], n & 1)) return;   // (S comes behind the tile before's P.V: O is complete up to there)
        tc_fence_after();
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          const int key0 = kt * PT_BN + half * PT_SN;
          uint32_t sa[32], sb[32];
          tmem_ld32(srow + 64u * half, sa);
          tmem_ld32(srow + 64u * half + 32u, sb);
          pt_ld_wait(sa);
          pt_ld_wait(sb);
          if (!(all_rows && key0 + PT_SN - 1 <= tile_a.q_pos0 && lo_all <= key0)) {
            const int jlo = lo_col - key0;
            const unsigned span = (unsigned)(hi_col - lo_col);  // hi < lo (nothing valid) wraps to a huge span: guard below
            const bool any = hi_col >= lo_col;
#pragma unroll
            for (int e = 0; e < 32; ++e) {
              if (!any || (unsigned)(e - jlo) > span) sa[e] = 0xff800000u;
              if (!any || (unsigned)(e + 32 - jlo) > span) sb[e] = 0xff800000u;
            }
          }
          // the row maximum (the scale is positive: max(s * c) = c * max(s)); four chains of three-input maxima
          float m4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
          for (int e = 0; e < 32; ++e) m4[e & 3] = pt_max3(m4[e & 3], __uint_as_float(sa[e]), __uint_as_float(sb[e]));
          const float mx = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3])) * a.scale_log2;
          // raise the reference?  (the very first half: O does not exist yet, the first P.V overwrites it)
          const bool raise = mx > m_ref + PT_RESCALE || (m_ref == -INFINITY && mx > -INFINITY);
          if ((half == 1 || kt > lo) && __any_sync(0xffffffffu, raise)) {
            const float corr = raise ? exp2f(m_ref - mx) : 1.0f;  // m_ref == -inf: 0 (O and l of such a row are zeros so far)
            if (half == 1) {
              if (!wait.warp(o_half[u], n & 1)) return;   // the first half has landed in O
              tc_fence_after();
            }
#pragma unroll 1
            for (int c0 = 0; c0 < PT_HD; c0 += 16) {
              uint32_t ov[16];
              pt_ld16(orow + (uint32_t)c0, ov);
#pragma unroll
              for (int e = 0; e < 16; ++e) ov[e] = __float_as_uint(__uint_as_float(ov[e]) * corr);
              tmem_st16(orow + (uint32_t)c0, ov);
            }
            l2[0] = pt_fma2(l2[0], pt_pair(corr, corr), 0ull);
            l2[1] = pt_fma2(l2[1], pt_pair(corr, corr), 0ull);
          }
          if (raise) m_ref = mx;
          const float msub = (m_ref == -INFINITY) ? 0.f : m_ref;
          // probabilities, their fp32 sum, and P as bf16 (masked scores: 2^-inf = 0) over S columns that this thread has read
          const pt_x2 sub2 = pt_pair(-msub, -msub);
          auto probs = [&](const uint32_t (&sv)[32], uint32_t col) {
            uint32_t pk[16];
#pragma unroll
            for (int e = 0; e < 32; e += 2) {
              const float2 x = pt_split(pt_fma2(pt_pair(__uint_as_float(sv[e]), __uint_as_float(sv[e + 1])), sc2, sub2));
              const float p0 = pt_ex2(x.x), p1 = pt_ex2(x.y);
              l2[(e >> 1) & 1] = pt_add2(l2[(e >> 1) & 1], pt_pair(p0, p1));
              pk[e >> 1] = pack_bf16x2(p0, p1);
            }
            tmem_st16(srow + col, pk);
          };
          probs(sa, 32u * half);
          probs(sb, 32u * half + 16u);
          tmem_st_wait();
          tc_fence_before();
          mbar_arrive(smem_u32(&p_full[2 * u + half]));
        }
      }
      // ---- O / l, once ----
      const float2 l_0 = pt_split(l2[0]), l_1 = pt_split(l2[1]);
      float l_row = (l_0.x + l_0.y) + (l_1.x + l_1.y);
      if (a.sink != nullptr && m_ref > -INFINITY) l_row += exp2f(a.sink[kvh * a.head_step + h] * 1.4426950408889634f - m_ref);
      const float inv = l_row > 0.f ? __fdiv_rn(1.0f, l_row) : 0.f;
      if (!wait.warp(o_full[u], (n - 1) & 1)) return;   // the last tile's P.V
      tc_fence_after();
      bf16* dst = a.out + ((size_t)(mt.q_row0 + t) * a.nq + kvh * a.head_step + h) * PT_HD;
#pragma unroll 1
      for (int c0 = 0; c0 < PT_HD; c0 += 32) {
        uint32_t ov[32];
        tmem_ld32(orow + (uint32_t)c0, ov);
        pt_ld_wait(ov);
        if (row_ok) {
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            float v[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) v[e] = __uint_as_float(ov[c * 8 + e]) * inv;
            reinterpret_cast<uint4*>(dst + c0)[c] = pack8(v);
          }
        }
      }
      tc_fence_before();   // (the next item's P arrival releases P.V over this O)
    }
  };
  if (warp > C::MMA_WARP) {
    load_tiles();
  } else if (warp == C::MMA_WARP) {
    if (lane == 0) multiply();
  } else {
    weigh();
  }
  tc_fence_before();
  __syncthreads();
  if (gave_up != 0) {   // (the same for the whole CTA: nobody waits any more) copies and MMAs under way end before shared memory and TMEM are given back
    if (warp > C::MMA_WARP) {
      for (int k = max(0, k_sent - C::KS); k < k_sent; ++k) b2_drain(k_full[k % C::KS], (k / C::KS) & 1);
      for (int k = max(0, v_sent - C::VS); k < v_sent; ++k) b2_drain(v_full[k % C::VS], (k / C::VS) & 1);
    } else if (warp == C::MMA_WARP && lane == 0) {
      tc_commit(smem_u32(&drained));
      b2_drain(drained, 0);
    }
    __syncthreads();
  }
  if (warp == C::MMA_WARP) {
    tc_fence_after();
    tmem_dealloc(tmem, C::TMEM_COLS);
  }
}

template <int NK, int NU>
int launch_pt(const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& tr, const PtArgs& a, cudaStream_t s) {
  using C = PtCfg<NK, NU>;
  static B2PerDeviceOnce attr_once;
  if (attr_once.need()) B2_CUDA_OK(cudaFuncSetAttribute(attn_prefill_tc_kernel<NK, NU>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM));
  B2_CUDA_OK(b2_launch(attn_prefill_tc_kernel<NK, NU>, dim3((a.units + NU - 1) / NU, a.nkv), dim3(C::THREADS), (size_t)C::SMEM, s, tk, tv, tr, a));
  return 0;
}

}  // namespace

// num_pages: pages in the pool k_pages / v_pages point to (the TMA maps cover exactly the pool).
int launch_attn_prefill_tc(const bf16* q, const bf16* k_pages, const bf16* v_pages, int64_t num_pages, const int32_t* block_table,
                           int bt_stride, const PrefillTile* tiles_dev, int ntiles, bf16* out, int nq, int nkv, int hd, int block_size,
                           cudaStream_t s, const B2WaitLimit& wait, float softmax_scale, int window, int pair_mode, int chunk, const PrefillRot* rot) {
  if (ntiles <= 0) return 0;
  const int head_step = pair_mode && nq == nkv ? 1 : 2;
  B2_REQUIRE(hd == PT_HD && block_size == 16 && nq == head_step * nkv, "attn_prefill_tc: built for 128-wide heads in GQA groups of two, 16-token pages");
  B2_REQUIRE(num_pages >= 1, "attn_prefill_tc: the page pool's size is needed for the tensor maps");
  B2_REQUIRE(bt_stride <= PT_MAX_PAGES, "attn_prefill_tc: contexts beyond %d tokens not built (block table row of %d pages)", PT_MAX_PAGES * 16, bt_stride);
  B2_REQUIRE(!pair_mode || ntiles % 2 == 0, "attn_prefill_tc: pair mode needs an even tile list (each sequence padded to an even number of tiles)");
  B2_REQUIRE(rot == nullptr || rot->rot_dim <= 64, "attn_prefill_tc: rotated pieces wider than 64 not built");
  CUtensorMap tk, tv, tr;
  const uint64_t rows = (uint64_t)num_pages * nkv * 16;
  int rc = b2_make_tmap_bf16_ex(&tk, k_pages, rows, PT_HD, PT_HD, 64, 16, /*swizzle128=*/0);
  if (rc != 0) return rc;
  rc = b2_make_tmap_bf16_ex(&tv, v_pages, rows, PT_HD, PT_HD, 64, 16, 0);
  if (rc != 0) return rc;
  tr = tk;
  if (rot != nullptr && rot->rot_dim > 0) {
    rc = b2_make_tmap_bf16_ex(&tr, rot->k_pages, (uint64_t)num_pages * 16, 64, 64, 64, 16, 0);
    if (rc != 0) return rc;
  }
  const double scale = softmax_scale > 0.f ? (double)softmax_scale : 1.0 / sqrt((double)hd);
  PtArgs a{};
  a.q = q; a.block_table = block_table; a.bt_stride = bt_stride; a.tiles = tiles_dev; a.out = out;
  a.nq = nq; a.nkv = nkv; a.units = pair_mode ? ntiles / 2 : ntiles;
  a.scale_log2 = (float)(scale * 1.4426950408889634);
  a.window = window; a.pair_mode = pair_mode; a.head_step = head_step; a.chunk = chunk;
  a.wait = wait;
  if (rot != nullptr) {
    a.q_rot = rot->q_rot;
    a.rot_dim = rot->rot_dim;
    a.sink = rot->sink;
  }
  if (rot == nullptr || rot->rot_dim == 0) return launch_pt<2, 1>(tk, tv, tr, a, s);
  // Beside a rotated piece one unit takes 128 KB and an SM to itself: a second one in turn fills its gaps once every SM has a unit.  One unit / two, us at
  // 16 heads: 1 x 1024 tokens (128 units) 25.6 / 31.5; 1 x 1280 (160) 39.1 / 39.6; 4 x 512 (256) 35.6 / 29.2; 8 x 1024 (1024) 124.8 / 103.6; units that do not
  // continue one another 25.0 / 27.2 (10 x 128) to 30.4 / 29.4 (16 x 128), three to a sequence 35.8 / 38.3 (8 x 384).
  static const int sms = device_num_sms();
  return (long)a.units * nkv > sms ? launch_pt<3, 2>(tk, tv, tr, a, s) : launch_pt<3, 1>(tk, tv, tr, a, s);
}

}  // namespace b2
