// gemm_few.cu -- the decode step of a Qwen3-geometry layer for at most eight sequences (HF:models/qwen3/modeling_qwen3.py:236-263, 81-83, 339-351):
//   few_qkv     q | k | v = bf16(RMSNorm(h) . Wqkv^T)
//   few_attn    QK-norm, RoPE, page write of the new token, attention over the pages
//   few_resid   h += bf16(x . W^T)                      (O and down projections)
//   few_gateup  act = bf16(bf16(silu(g)) * u), g | u = bf16(RMSNorm(h) . Wgu^T)
//
// Five launches a layer, each a link of a chain whose time is hand-offs and latencies, not bytes (31 MB of weights a layer are 4.7 us at the copy rate; with the
// 64-token kernels of gemm_pair.cu, gemm_resid.cu and attn_decode.cu a layer of one sequence of 140 tokens took 28 us, with these 15.5: 2.8 + 3.8 + 2.6 + 3.6 + 2.7,
// of which about 2 are the hand-off).  So:
//   * a CTA's share of the weights sits in its REGISTERS before the kernel in front has ended: it is requested before the dependency wait, and every kernel lets
//     the next one start at its own start, so the weight streams of two or three kernels run beside the one that computes.  (Constants and page tables only:
//     everything that a kernel in front writes is read behind the wait, through pointers that are not __restrict__: read-only loads may be moved across it. A
//     kernel that is through its wait has all kernels before it complete.)
//   * 128 CTAs of 8 warps; a CTA owns whole weight rows (no sums between CTAs), its warps split K.  Inside a 32-wide k chunk lane (n, c) = (lane / 4, lane % 4)
//     takes elements [8c, 8c + 8) of weight row n and of token n; elements 0..3 feed one m16n8k16 (tokens on M, weight rows on N; an MMA does not care which
//     physical k sits behind its logical k as long as both operands agree), elements 4..7 the next: operands go from global memory into the fragments as they are.
//   * the norm is applied to the rows of h as they arrive (every CTA forms the statistic itself: two shuffles and one exchange through shared memory), the
//     per-head norm and RoPE by the attention kernel's CTAs, each for its own head: no launches of their own.
//   * attention: a cluster of eight CTAs per (sequence, kv head), warp w of the 32 takes pages w, w + 32, ...; the shares are folded through distributed
//     shared memory.
// Rounding points are those of the kernels that larger batches take; sums are fp32 in a fixed order that does not depend on the number of sequences.
#include "kernels.h"

namespace b2 {

namespace {

constexpr int FEW_WARPS = 8, FEW_THREADS = 32 * FEW_WARPS, FEW_T = 8;   // tokens at most

__device__ __forceinline__ uint4 few_ldw(const bf16* p) {   // streamed past L1; not .nc: such a load may be moved behind the dependency wait
  uint4 v;
  asm volatile("ld.global.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
  return v;
}
// d[token g: weight rows 2c, 2c + 1] += the first eight tokens' rows (the other eight of the instruction are zero)
__device__ __forceinline__ void few_mma(float (&d)[2], uint32_t a0, uint32_t a2, uint32_t b0, uint32_t b1) {
  float z0 = 0.f, z1 = 0.f;
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%5}, {%7,%8}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(z0), "+f"(z1)
               : "r"(a0), "r"(0u), "r"(a2), "r"(b0), "r"(b1));
}

enum { FEW_QKV = 0, FEW_RESID = 1, FEW_GATEUP = 2 };

// TILES tiles of eight weight rows per CTA.  GATEUP: tile 2p is gate rows, tile 2p + 1 the up rows of the same features.  CH chunks of 32 k per warp and round
// (a warp's chunks are warp, warp + 8, ...); the first round's weights are in registers before the wait.
template <int CH, int TILES, int MODE>
__global__ void __launch_bounds__(FEW_THREADS) few_kernel(const bf16* __restrict__ w, const bf16* x, const bf16* __restrict__ gain, float eps, bf16* out, int T,
                                                          int N, int K, int up_row0) {
  constexpr bool NORM = MODE != FEW_RESID;
  constexpr int OUT_TILES = MODE == FEW_GATEUP ? TILES / 2 : TILES;
  __shared__ float red[FEW_WARPS][TILES][FEW_T][8 + 1];
  __shared__ float ssq[FEW_WARPS][FEW_T];
  pdl_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, c = lane & 3;
  const int chunks = K / 32, row0 = blockIdx.x * OUT_TILES * 8;
  auto weight_row = [&](int t) {
    const int r = MODE == FEW_GATEUP ? row0 + (t >> 1) * 8 + g : row0 + t * 8 + g;
    return min(r, N - 1) + (MODE == FEW_GATEUP && (t & 1) ? up_row0 : 0);   // (rows past N: computed and dropped)
  };
  uint4 wr[TILES][CH], gr[NORM ? CH : 1];
  auto load_weights = [&](int base) {
#pragma unroll
    for (int t = 0; t < TILES; ++t) {
      const bf16* p = w + (size_t)weight_row(t) * K + c * 8;
#pragma unroll
      for (int i = 0; i < CH; ++i) {
        const int k = base + warp + i * FEW_WARPS;
        wr[t][i] = k < chunks ? few_ldw(p + k * 32) : make_uint4(0u, 0u, 0u, 0u);
      }
    }
    if constexpr (NORM) {
#pragma unroll
      for (int i = 0; i < CH; ++i) {
        const int k = base + warp + i * FEW_WARPS;
        gr[i] = k < chunks ? *reinterpret_cast<const uint4*>(gain + k * 32 + c * 8) : make_uint4(0u, 0u, 0u, 0u);
      }
    }
  };
  load_weights(0);
  pdl_wait();
  auto load_x = [&](int base, uint4 (&xr)[CH]) {
#pragma unroll
    for (int i = 0; i < CH; ++i) {
      const int k = base + warp + i * FEW_WARPS;
      xr[i] = k < chunks && g < T ? *reinterpret_cast<const uint4*>(x + (size_t)g * K + k * 32 + c * 8) : make_uint4(0u, 0u, 0u, 0u);
    }
  };
  uint4 xr[CH];
  load_x(0, xr);
  uint32_t hv = 0;   // RESID: the residual stream's number that this thread adds to
  const int o_row = threadIdx.x & 7, o_tok = (threadIdx.x >> 3) & 7;
  if (MODE == FEW_RESID && threadIdx.x < OUT_TILES * 64 && o_tok < T && row0 + (threadIdx.x >> 6) * 8 + o_row < N)
    hv = reinterpret_cast<const unsigned short*>(out)[(size_t)o_tok * N + row0 + (threadIdx.x >> 6) * 8 + o_row];
  float rstd = 0.f;
  if constexpr (NORM) {   // the statistic of all rows of h
    float ss = 0.f;
    for (int base = 0;; ) {
#pragma unroll
      for (int i = 0; i < CH; ++i) {
        float f[8];
        unpack8(xr[i], f);
#pragma unroll
        for (int e = 0; e < 8; ++e) ss = fmaf(f[e], f[e], ss);
      }
      base += CH * FEW_WARPS;
      if (base >= chunks) break;
      load_x(base, xr);
    }
    ss += __shfl_xor_sync(0xffffffffu, ss, 1);
    ss += __shfl_xor_sync(0xffffffffu, ss, 2);
    if (c == 0) ssq[warp][g] = ss;
    __syncthreads();
    float tot = 0.f;
#pragma unroll
    for (int v = 0; v < FEW_WARPS; ++v) tot += ssq[v][g];
    rstd = __fdiv_rn(1.0f, __fsqrt_rn(tot / (float)K + eps));
    if (chunks > CH * FEW_WARPS) load_x(0, xr);
  }
  float acc[TILES][2];
#pragma unroll
  for (int t = 0; t < TILES; ++t) acc[t][0] = acc[t][1] = 0.f;
  for (int base = 0;; ) {
#pragma unroll
    for (int i = 0; i < CH; ++i) {
      uint32_t a[4] = {xr[i].x, xr[i].y, xr[i].z, xr[i].w};
      if constexpr (NORM) {   // bf16(gain * bf16(h * rstd))
        float f[8];
        unpack8(xr[i], f);
        const uint32_t* g2 = &gr[i].x;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const uint32_t nx = pack_bf16x2(f[2 * e] * rstd, f[2 * e + 1] * rstd);
          const __nv_bfloat162 n = __hmul2(*reinterpret_cast<const __nv_bfloat162*>(&g2[e]), *reinterpret_cast<const __nv_bfloat162*>(&nx));
          a[e] = *reinterpret_cast<const uint32_t*>(&n);
        }
      }
#pragma unroll
      for (int t = 0; t < TILES; ++t) {
        few_mma(acc[t], a[0], a[1], wr[t][i].x, wr[t][i].y);
        few_mma(acc[t], a[2], a[3], wr[t][i].z, wr[t][i].w);
      }
    }
    base += CH * FEW_WARPS;
    if (base >= chunks) break;
    load_weights(base);
    load_x(base, xr);
  }
#pragma unroll
  for (int t = 0; t < TILES; ++t) {
    red[warp][t][g][2 * c] = acc[t][0];
    red[warp][t][g][2 * c + 1] = acc[t][1];
  }
  __syncthreads();
  auto sum = [&](int t, int tok, int row) {
    float v = 0.f;
#pragma unroll
    for (int k = 0; k < FEW_WARPS; ++k) v += red[k][t][tok][row];
    return v;
  };
  for (int i = threadIdx.x; i < OUT_TILES * 64; i += FEW_THREADS) {
    const int row = i & 7, tok = (i >> 3) & 7, t = i >> 6, col = row0 + t * 8 + row;
    if (tok >= T || col >= N) continue;
    bf16* d = out + (size_t)tok * N + col;
    if constexpr (MODE == FEW_QKV) {
      *d = __float2bfloat16_rn(sum(t, tok, row));
    } else if constexpr (MODE == FEW_RESID) {   // (one round: OUT_TILES * 64 <= FEW_THREADS)
      *d = __float2bfloat16_rn(__uint_as_float(hv << 16) + bf16_round(sum(t, tok, row)));
    } else {
      const float gf = bf16_round(sum(2 * t, tok, row)), uf = bf16_round(sum(2 * t + 1, tok, row));
      const float s = bf16_round(gf / (1.0f + expf(-gf)));
      *d = __float2bfloat16_rn(s * uf);
    }
  }
}

// ---- heads: at most sixteen rows against many weight rows ----
// out [T][N] fp32 = alpha * x [T][K] . w [N][K]^T, or (ARGMAX) bf16 logits, written where out is given, and the largest with the lowest index per row.  A CTA per SM walks the tiles of eight weight rows with stride gridDim.x; its warps split K as above, the rows of x stay
// in fragments (HALVES: one or two times eight of them), and while a tile is multiplied the next DEPTH - 1 are under way into registers, the first ones before the
// dependency wait.  Bound: HBM.  What a launch adds to a step, us, the tcgen05 kernel with its 16-row tiles before and this one: 32000 x 2048, 4 rows 27.7 -> 21.8 (6.0 TB/s),
// 16 rows 29.5 -> 25.3; 151936 x 1024, 1 row 60 -> 47.5 (6.5 TB/s).
template <int CH, int HALVES, int DEPTH, bool ARGMAX>
__global__ void __launch_bounds__(FEW_THREADS, CH <= 4 ? 2 : 1) few_head_kernel(const bf16* __restrict__ w, const bf16* x, void* out, int T, int N,
                                                                                  int K, float alpha, unsigned long long* best_packed) {
  __shared__ float red[2][FEW_WARPS][HALVES * FEW_T][8 + 1];
  pdl_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, c = lane & 3;
  const int chunks = K / 32, tiles = (N + 7) / 8;
  uint4 wr[DEPTH][CH];
  auto load = [&](int tile, uint4 (&r)[CH]) {
    const bf16* p = w + (size_t)min(tile * 8 + g, N - 1) * K + c * 8;   // (rows past N: computed and dropped)
#pragma unroll
    for (int i = 0; i < CH; ++i) {
      const int k = warp + i * FEW_WARPS;
      r[i] = tile < tiles && k < chunks ? few_ldw(p + k * 32) : make_uint4(0u, 0u, 0u, 0u);
    }
  };
#pragma unroll
  for (int d = 0; d < DEPTH - 1; ++d) load(blockIdx.x + d * gridDim.x, wr[d]);
  pdl_wait();
  uint4 xr[HALVES][CH];
#pragma unroll
  for (int h = 0; h < HALVES; ++h)
#pragma unroll
    for (int i = 0; i < CH; ++i) {
      const int k = warp + i * FEW_WARPS, t = h * 8 + g;
      xr[h][i] = k < chunks && t < T ? *reinterpret_cast<const uint4*>(x + (size_t)t * K + k * 32 + c * 8) : make_uint4(0u, 0u, 0u, 0u);
    }
  int parity = 0;
  unsigned long long best = 0ull;   // ARGMAX: (value, -index) of this thread's row, as gemm_tc.cu packs it
  for (int t0 = blockIdx.x; t0 < tiles; t0 += DEPTH * gridDim.x) {
#pragma unroll
    for (int d = 0; d < DEPTH; ++d) {
      const int tile = t0 + d * gridDim.x;
      if (tile >= tiles) break;
      load(tile + (DEPTH - 1) * gridDim.x, wr[(d + DEPTH - 1) % DEPTH]);
      float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int i = 0; i < CH; ++i) {
        const uint4 b = wr[d][i], a0 = xr[0][i], a1 = HALVES == 2 ? xr[HALVES - 1][i] : make_uint4(0u, 0u, 0u, 0u);
        asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                     : "+f"(acc[0]), "+f"(acc[1]), "+f"(acc[2]), "+f"(acc[3])
                     : "r"(a0.x), "r"(a1.x), "r"(a0.y), "r"(a1.y), "r"(b.x), "r"(b.y));
        asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                     : "+f"(acc[0]), "+f"(acc[1]), "+f"(acc[2]), "+f"(acc[3])
                     : "r"(a0.z), "r"(a1.z), "r"(a0.w), "r"(a1.w), "r"(b.z), "r"(b.w));
      }
#pragma unroll
      for (int h = 0; h < HALVES; ++h) {
        red[parity][warp][h * 8 + g][2 * c] = acc[2 * h];
        red[parity][warp][h * 8 + g][2 * c + 1] = acc[2 * h + 1];
      }
      __syncthreads();   // (the other parity's sums were read before this tile's were written by every warp: one barrier a tile)
      if (threadIdx.x < HALVES * 64) {
        const int row = threadIdx.x & 7, t = threadIdx.x >> 3, col = tile * 8 + row;
        float v = 0.f;
#pragma unroll
        for (int k = 0; k < FEW_WARPS; ++k) v += red[parity][k][t][row];
        if (t < T && col < N) {
          if constexpr (ARGMAX) {
            const bf16 b = __float2bfloat16_rn(v);
            if (out != nullptr) reinterpret_cast<bf16*>(out)[(size_t)t * N + col] = b;
            const float lv = __bfloat162float(b);
            const uint32_t u = __float_as_uint(lv), key = (u & 0x80000000u) ? ~u : (u | 0x80000000u);
            const unsigned long long p = lv == lv ? ((unsigned long long)key << 32) | (unsigned long long)(0xffffffffu - (uint32_t)col) : 0ull;
            best = p > best ? p : best;
          } else {
            reinterpret_cast<float*>(out)[(size_t)t * N + col] = v * alpha;
          }
        }
      }
      parity ^= 1;
    }
  }
  if (ARGMAX && threadIdx.x < HALVES * 64) {   // (whole warps; eight lanes hold a row)
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) {
      const unsigned long long other = __shfl_xor_sync(0xffffffffu, best, o);
      best = other > best ? other : best;
    }
    if ((threadIdx.x & 7) == 0 && best != 0ull) atomicMax(best_packed + (threadIdx.x >> 3), best);
  }
}

// ---- attention ----
constexpr int FA_CTAS = 8, FA_WARPS = 4, FA_SHARES = FA_CTAS * FA_WARPS, FA_HD = 128, FA_BS = 16;
struct FaRecord { float o[2][FA_HD], m[2], l[2]; };   // one share: unnormalised output, maximum and sum of the two query heads

// grid (8, kv heads, sequences), clusters of eight along x; qkv: bf16 rows of (nq + 2 nkv) * 128
__global__ void __launch_bounds__(32 * FA_WARPS) __cluster_dims__(FA_CTAS, 1, 1)
few_attn_kernel(const bf16* qkv, const bf16* __restrict__ qw, const bf16* __restrict__ kw, const bf16* __restrict__ cos_sin,
                const int32_t* positions, const int32_t* slots, bf16* k_pages, bf16* v_pages,
                const int32_t* __restrict__ block_table, int bt_stride, const int32_t* seq_lens, bf16* out, int nq, int nkv, float eps,
                float scale) {
  __shared__ __align__(16) float qs[2][FA_HD];            // the two query heads, scaled
  __shared__ __align__(16) bf16 kv_new[2][FA_HD];         // the new token's key and value
  __shared__ FaRecord rec[FA_WARPS], all[FA_CTAS];
  pdl_launch_dependents();
  asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");   // this CTA runs: see the first remote store
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint32_t rank;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  const int kvh = blockIdx.y, b = blockIdx.z;
  // page table, lengths, norm gains and rotary rows are older than the kernel in front
  const int S = seq_lens[b], pos = max(positions[b], 0), pages = S > 0 ? (S + FA_BS - 1) / FA_BS : 0;
  const uint2 gain = *reinterpret_cast<const uint2*>((warp == 2 ? kw : qw) + lane * 4);
  const uint2 cosr = *reinterpret_cast<const uint2*>(cos_sin + (size_t)pos * FA_HD + (lane * 4 & 63)), sinr = *reinterpret_cast<const uint2*>(cos_sin + (size_t)pos * FA_HD + 64 + (lane * 4 & 63));
  const int share = (int)rank * FA_WARPS + warp;
  const int first_page = share < pages ? block_table[(size_t)b * bt_stride + share] : 0;
  const int t = lane >> 1, half = lane & 1;   // scores: two lanes per key, 64 dimensions each
  auto page_at = [&](int page) { return ((size_t)page * nkv + kvh) * (FA_BS * FA_HD); };
  uint4 kr[8];
  uint2 vr[FA_BS];
  // the rows of a page that hold earlier tokens (row r of the page is token p * 16 + r; the new token's row is written by the owner of the last page)
  auto load_keys = [&](int page, int p) {
    const int old = min(FA_BS, S - 1 - p * FA_BS);
    const bf16* kp = k_pages + page_at(page) + t * FA_HD;
#pragma unroll
    for (int i = 0; i < 8; ++i)
      kr[i] = t < old ? *reinterpret_cast<const uint4*>(kp + kv_swizzled_chunk(t, half * 8 + i) * 8) : make_uint4(0u, 0u, 0u, 0u);
  };
  auto load_values = [&](int page, int p) {
    const int old = min(FA_BS, S - 1 - p * FA_BS);
    const bf16* vp = v_pages + page_at(page);
#pragma unroll
    for (int r = 0; r < FA_BS; ++r)
      vr[r] = r < old ? *reinterpret_cast<const uint2*>(vp + r * FA_HD + kv_swizzled_chunk(r, lane >> 1) * 8 + (lane & 1) * 4) : make_uint2(0u, 0u);
  };
  if (share < pages) {   // (rows a step old and older)
    load_keys(first_page, share);
    load_values(first_page, share);
  }
  pdl_wait();
  // ---- warps 0, 1: the query heads; 2: the key; 3: the value ----
  {
    const int head = warp < 2 ? kvh * 2 + warp : warp == 2 ? nq + kvh : nq + nkv + kvh;
    const uint2 raw = *reinterpret_cast<const uint2*>(qkv + (size_t)b * (nq + 2 * nkv) * FA_HD + (size_t)head * FA_HD + lane * 4);
    if (warp == 3) {
      *reinterpret_cast<uint2*>(&kv_new[1][lane * 4]) = raw;
    } else {
      const float v[4] = {bf16lo(raw.x), bf16hi(raw.x), bf16lo(raw.y), bf16hi(raw.y)};
      float ss = v[0] * v[0] + v[1] * v[1] + v[2] * v[2] + v[3] * v[3];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
      const float rstd = __fdiv_rn(1.0f, __fsqrt_rn(ss / (float)FA_HD + eps));
      uint32_t res[2];
      const uint32_t gw[2] = {gain.x, gain.y}, co[2] = {cosr.x, cosr.y}, si[2] = {sinr.x, sinr.y};
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const uint32_t nx = pack_bf16x2(v[2 * e] * rstd, v[2 * e + 1] * rstd);   // bf16(x * rstd)
        const __nv_bfloat162 n = __hmul2(*reinterpret_cast<const __nv_bfloat162*>(&gw[e]), *reinterpret_cast<const __nv_bfloat162*>(&nx));
        const uint32_t nu = *reinterpret_cast<const uint32_t*>(&n);
        const uint32_t partner = __shfl_xor_sync(0xffffffffu, nu, 16) ^ (lane < 16 ? 0x80008000u : 0u);   // dimensions 0..63 take minus the other half
        const __nv_bfloat162 a = __hmul2(n, *reinterpret_cast<const __nv_bfloat162*>(&co[e]));
        const __nv_bfloat162 r = __hmul2(*reinterpret_cast<const __nv_bfloat162*>(&partner), *reinterpret_cast<const __nv_bfloat162*>(&si[e]));
        const uint32_t au = *reinterpret_cast<const uint32_t*>(&a), ru = *reinterpret_cast<const uint32_t*>(&r);
        res[e] = pack_bf16x2(bf16lo(au) + bf16lo(ru), bf16hi(au) + bf16hi(ru));
      }
      if (warp == 2)
        *reinterpret_cast<uint2*>(&kv_new[0][lane * 4]) = make_uint2(res[0], res[1]);
      else
        *reinterpret_cast<float4*>(&qs[warp][lane * 4]) =
            make_float4(bf16lo(res[0]) * scale, bf16hi(res[0]) * scale, bf16lo(res[1]) * scale, bf16hi(res[1]) * scale);
    }
  }
  __syncthreads();
  // the new token's row goes to its page (one CTA of the cluster), for the steps to come
  const int slot = slots[b];
  if (rank == 0 && warp >= 2 && slot >= 0) {
    bf16* base = (warp == 2 ? k_pages : v_pages) + page_at(slot / FA_BS) + (slot % FA_BS) * FA_HD;
    if (lane < 16) *reinterpret_cast<uint4*>(base + kv_swizzled_chunk(slot % FA_BS, lane) * 8) = *reinterpret_cast<const uint4*>(&kv_new[warp - 2][lane * 8]);
  }
  float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f}, o[2][4] = {};
  for (int p = share; p < pages; p += FA_SHARES) {
    const int next = p + FA_SHARES, next_page = next < pages ? block_table[(size_t)b * bt_stride + next] : 0;
    const int at_new = S - 1 - p * FA_BS;   // the new token's row in this page, if it is in it
    if (t == at_new) {
#pragma unroll
      for (int i = 0; i < 8; ++i) kr[i] = *reinterpret_cast<const uint4*>(&kv_new[0][half * 64 + i * 8]);
    }
    if (at_new < FA_BS) {
      const uint2 nv = *reinterpret_cast<const uint2*>(&kv_new[1][lane * 4]);
#pragma unroll
      for (int r = 0; r < FA_BS; ++r) vr[r] = r == at_new ? nv : vr[r];
    }
    float s[2] = {0.f, 0.f};
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      float f[8];
      unpack8(kr[i], f);
#pragma unroll
      for (int hq = 0; hq < 2; ++hq) {
        const float4 q0 = *reinterpret_cast<const float4*>(&qs[hq][half * 64 + i * 8]), q1 = *reinterpret_cast<const float4*>(&qs[hq][half * 64 + i * 8 + 4]);
        s[hq] = fmaf(f[0], q0.x, s[hq]); s[hq] = fmaf(f[1], q0.y, s[hq]); s[hq] = fmaf(f[2], q0.z, s[hq]); s[hq] = fmaf(f[3], q0.w, s[hq]);
        s[hq] = fmaf(f[4], q1.x, s[hq]); s[hq] = fmaf(f[5], q1.y, s[hq]); s[hq] = fmaf(f[6], q1.z, s[hq]); s[hq] = fmaf(f[7], q1.w, s[hq]);
      }
    }
    if (next < pages) load_keys(next_page, next);   // (the keys' registers are free: the next page's arrive under the rest)
#pragma unroll
    for (int hq = 0; hq < 2; ++hq) {
      s[hq] += __shfl_xor_sync(0xffffffffu, s[hq], 1);
      if (t > at_new) s[hq] = -INFINITY;   // (rows behind the end)
      float top = s[hq];
#pragma unroll
      for (int x = 2; x < 32; x <<= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, x));
      const float mn = fmaxf(m[hq], top), keep = m[hq] == mn ? 1.0f : __expf(m[hq] - mn);   // (a page holds at least one key)
      const float e = s[hq] == -INFINITY ? 0.f : __expf(s[hq] - mn);
      float sum = e;
#pragma unroll
      for (int x = 2; x < 32; x <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, x);
      l[hq] = l[hq] * keep + sum;
      m[hq] = mn;
#pragma unroll
      for (int d = 0; d < 4; ++d) o[hq][d] *= keep;
#pragma unroll
      for (int r = 0; r < FA_BS; ++r) {
        const float pr = __shfl_sync(0xffffffffu, e, 2 * r);
        o[hq][0] = fmaf(pr, bf16lo(vr[r].x), o[hq][0]);
        o[hq][1] = fmaf(pr, bf16hi(vr[r].x), o[hq][1]);
        o[hq][2] = fmaf(pr, bf16lo(vr[r].y), o[hq][2]);
        o[hq][3] = fmaf(pr, bf16hi(vr[r].y), o[hq][3]);
      }
    }
    if (next < pages) load_values(next_page, next);
  }
  // ---- fold: the CTA's warps, then the cluster's CTAs on its first one ----
#pragma unroll
  for (int hq = 0; hq < 2; ++hq) {
    *reinterpret_cast<float4*>(&rec[warp].o[hq][lane * 4]) = make_float4(o[hq][0], o[hq][1], o[hq][2], o[hq][3]);
    if (lane == 0) {
      rec[warp].m[hq] = m[hq];
      rec[warp].l[hq] = l[hq];
    }
  }
  __syncthreads();
  auto fold = [&](const FaRecord* r, int n, int hq, int d, float& mo, float& lo) {
    mo = -INFINITY;
    for (int k = 0; k < n; ++k) mo = fmaxf(mo, r[k].m[hq]);
    float v = 0.f;
    lo = 0.f;
    for (int k = 0; k < n; ++k) {
      const float f = r[k].l[hq] > 0.f ? __expf(r[k].m[hq] - mo) : r[k].l[hq];   // (a share without keys; a sum that is no number stays one)
      v = fmaf(r[k].o[hq][d], f, v);
      lo = fmaf(r[k].l[hq], f, lo);
    }
    return v;
  };
  // every CTA of the cluster has started (its shared memory is live) before anyone stores into the first one's: a CTA without pages is here almost at once,
  // and the dependency wait says nothing about the other CTAs
  asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
  const uint32_t mine = (uint32_t)__cvta_generic_to_shared(&all[rank]);
  uint32_t dst;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(dst) : "r"(mine));
  for (int i = threadIdx.x; i < 2 * FA_HD; i += 32 * FA_WARPS) {
    const int hq = i >> 7, d = i & 127;
    float mo, lo;
    const float v = fold(rec, FA_WARPS, hq, d, mo, lo);
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(dst + (uint32_t)((hq * FA_HD + d) * 4)), "f"(v) : "memory");
    if (d == 0) {
      asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(dst + (uint32_t)((2 * FA_HD + hq) * 4)), "f"(mo) : "memory");
      asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(dst + (uint32_t)((2 * FA_HD + 2 + hq) * 4)), "f"(lo) : "memory");
    }
  }
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  if (rank != 0) return;
  for (int i = threadIdx.x; i < 2 * FA_HD; i += 32 * FA_WARPS) {
    const int hq = i >> 7, d = i & 127;
    float mo, lo;
    const float v = fold(all, FA_CTAS, hq, d, mo, lo);
    out[((size_t)b * nq + kvh * 2 + hq) * FA_HD + d] = __float2bfloat16_rn(pages > 0 ? v / lo : 0.f);
  }
}

template <int CH, int TILES, int MODE>
int launch_few(const bf16* w, const bf16* x, const bf16* gain, float eps, bf16* out, int T, int N, int K, int up_row0, cudaStream_t s) {
  constexpr int OUT_TILES = MODE == FEW_GATEUP ? TILES / 2 : TILES;
  B2_CUDA_OK(b2_launch(few_kernel<CH, TILES, MODE>, dim3((N + OUT_TILES * 8 - 1) / (OUT_TILES * 8)), dim3(FEW_THREADS), 0, s, w, x, gain, eps, out, T, N, K, up_row0));
  return 0;
}

}  // namespace

bool few_shapes_ok(int T, int H, int q_size, int I) { return T >= 1 && T <= FEW_T && H % 32 == 0 && q_size % 32 == 0 && I % 32 == 0 && H >= 32 && I >= 32; }

int launch_few_qkv(const bf16* w, const bf16* h, const bf16* gain, float eps, bf16* qkv, int T, int N, int K, cudaStream_t s) {
  return launch_few<4, 4, FEW_QKV>(w, h, gain, eps, qkv, T, N, K, 0, s);
}
int launch_few_gateup(const bf16* wgu, const bf16* h, const bf16* gain, float eps, bf16* act, int T, int I, int K, cudaStream_t s) {
  return launch_few<4, 6, FEW_GATEUP>(wgu, h, gain, eps, act, T, I, K, I, s);
}
// (a warp's 12 chunks of a K of 3072 are 48 registers of weights; a K of 2048 takes eight)
int launch_few_resid(const bf16* w, const bf16* x, bf16* h, int T, int N, int K, cudaStream_t s) {
  if (K > 2048) return launch_few<12, 1, FEW_RESID>(w, x, nullptr, 0.f, h, T, N, K, 0, s);
  return launch_few<8, 1, FEW_RESID>(w, x, nullptr, 0.f, h, T, N, K, 0, s);
}
// K up to 2048 for sixteen rows, up to 4096 for eight (the fragments of x and of the tiles under way are registers)
bool few_head_ok(int T, int N, int K) { return T >= 1 && N >= 1 && K % 32 == 0 && K >= 32 && (T <= 8 ? K <= 4096 : T <= 16 && K <= 2048); }
template <bool ARGMAX>
static int launch_head(const bf16* w, const bf16* x, void* out, int T, int N, int K, float alpha, unsigned long long* best, cudaStream_t s) {
  const dim3 grid(std::min((N + 7) / 8, device_num_sms() * (K <= 1024 ? 2 : 1)));   // (a tile of 16 KB is done before its barrier: two CTAs per SM)
#define B2_FEW_HEAD(C, H, D)                                                                                                   \
  do {                                                                                                                         \
    B2_CUDA_OK(b2_launch(few_head_kernel<C, H, D, ARGMAX>, grid, dim3(FEW_THREADS), 0, s, w, x, out, T, N, K, alpha, best));   \
    return 0;                                                                                                                  \
  } while (0)
  if (T <= 8) {
    if (K <= 1024) B2_FEW_HEAD(4, 1, 4);
    if (K <= 2048) B2_FEW_HEAD(8, 1, 4);
    B2_FEW_HEAD(16, 1, 2);
  }
  if (K <= 1024) B2_FEW_HEAD(4, 2, 4);
  B2_FEW_HEAD(8, 2, 3);
#undef B2_FEW_HEAD
}
int launch_few_head(const bf16* w, const bf16* x, float* out, int T, int N, int K, float alpha, cudaStream_t s) { return launch_head<false>(w, x, out, T, N, K, alpha, nullptr, s); }
int launch_few_head_argmax(const bf16* w, const bf16* x, bf16* logits, unsigned long long* best, int T, int N, int K, cudaStream_t s) {
  return launch_head<true>(w, x, logits, T, N, K, 1.f, best, s);
}
int launch_few_attn(const bf16* qkv, const bf16* qw, const bf16* kw, const bf16* cos_sin, const int32_t* positions, const int32_t* slots, bf16* k_pages, bf16* v_pages,
                    const int32_t* block_table, int bt_stride, const int32_t* seq_lens, bf16* out, int B, int nq, int nkv, float eps, float scale, cudaStream_t s) {
  B2_REQUIRE(nq == 2 * nkv && B >= 1 && B <= FEW_T, "few_attn: %d query heads on %d, %d sequences not built", nq, nkv, B);
  B2_CUDA_OK(b2_launch(few_attn_kernel, dim3(FA_CTAS, nkv, B), dim3(32 * FA_WARPS), 0, s, qkv, qw, kw, cos_sin, positions, slots, k_pages, v_pages, block_table, bt_stride,
                       seq_lens, out, nq, nkv, eps, scale));
  return 0;
}

}  // namespace b2
