// gemm_sum.cu -- prompt-sized products of the layer-list families, fp32 sums out, on pairs of CTAs (tcgen05 cta_group::2):
// y[row][N] = x[row][K] . W_g[N][K]^T, where the rows are one block (G = 1) or the ragged blocks of G experts in one launch.
//
// The pair's tile is gemm_mc.cu's: 256 weight rows (128 in each CTA) x BN rows of x (half of them loaded by each CTA, read by the MMA of both where they are),
// 64-wide k-blocks through a ring of stages, a double-buffered accumulator in TMEM, every wait with a limit.  What differs:
//   * groups: the experts' first rows are read from the device's own table when the kernel starts, so the host neither waits for it nor launches per expert.  A
//     cluster walks the list of all experts' tiles with stride `clusters`, weight-row pair fastest; the rows that a group's last tile reads past its end belong to
//     the next group (or to nobody: zero-filled) and are not stored.
//   * epilogue: fp32 sums straight from registers (a warp's 32 weight rows are 128 contiguous bytes of an output row), or, for squared-ReLU experts and Tinevik's dense
//     feed-forward (4096 x 16384 at K 4096: 268 MB of sums written and read again otherwise, 2364 -> 2228 us of a whole call), the activation rounded to the bf16
//     operand of the second product.
//   * SPLIT 3: x is fp32, given as three bf16 planes whose sum it is (split3_kernel: 8 + 8 + 8 bits of the 24), and the weights are bf16 numbers, so the three
//     products are exact.  The tensor pipe's accumulator rounds every addition towards zero, so it holds only 128 of the K at a time, smallest plane first: the
//     epilogue's warps keep the running sums of a tile in registers and add a chunk, rounded to nearest, while the next one is multiplied.  SPLIT 1: the same
//     sums for bf16 x.
// Bound: tensor pipe under the power cap, and the last wave.
#include "cta_pair.cuh"
#include "kernels.h"

namespace b2 {

namespace {

constexpr int GS_BM = 128, GS_BK = 64, GS_MAX_GROUPS = 512;
constexpr int GS_W_BYTES = GS_BM * GS_BK * 2;   // 16 KB
template <int BN>
struct GsCfg {
  static constexpr int XH_BYTES = BN / 2 * GS_BK * 2;   // one CTA's half of the rows of x
  static constexpr int STAGE_BYTES = GS_W_BYTES + XH_BYTES;
  static constexpr int STAGES = BN == 256 ? 6 : 8;
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024;
  static constexpr int TMEM_COLS = 2 * BN;
};
constexpr int GS_CHUNK_KB = 2;   // SPLIT: k-blocks per chunk
constexpr int GS_EPI_WARPS = 8, GS_THREADS = 64 + 32 * GS_EPI_WARPS;

// The tiles of all groups, in order: group by group, tile of rows by tile of rows, weight-row pair fastest.  A walker moves forward only.
template <int BN>
struct GsWalk {
  const int* off;   // [groups + 1] first rows (shared memory)
  int groups, m_pairs;
  int g = 0, base = 0;   // the group the walker is in, and the number of its first tile
  int row0, rows, pair;  // the tile: first row, rows that are its own, weight-row pair
  __device__ __forceinline__ GsWalk(const int* o, int n, int m) : off(o), groups(n), m_pairs(m) {}
  __device__ __forceinline__ bool at(int p) {
    while (g < groups) {
      const int n = off[g + 1] - off[g], tiles = (n + BN - 1) / BN * m_pairs;
      if (p < base + tiles) {
        const int t = p - base, nt = t / m_pairs;
        pair = t - nt * m_pairs;
        row0 = off[g] + nt * BN;
        rows = min(BN, n - nt * BN);
        return true;
      }
      base += tiles;
      ++g;
    }
    return false;
  }
};

// offsets: [groups + 1] first rows of the groups in device memory, or null: groups of rows_total / groups rows
template <int BN, int EPI, int SPLIT>   // SPLIT: planes of x (0: x as it is, its whole K in the accumulator)
__global__ void __launch_bounds__(GS_THREADS, 1)
linear_sum_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x, const int32_t* offsets, int groups,
                  int rows_total, void* out, int N, int K, int ldo, const B2WaitLimit limit, const float* pq) {
  using C = GsCfg<BN>;
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t full_bar[C::STAGES];
  __shared__ __align__(8) uint64_t empty_bar[C::STAGES];
  __shared__ __align__(8) uint64_t tmem_full_bar[2];
  __shared__ __align__(8) uint64_t tmem_empty_bar[2];
  __shared__ __align__(8) uint64_t drained;
  __shared__ uint32_t tmem_slot;
  __shared__ volatile uint32_t gave_up;
  __shared__ int s_off[GS_MAX_GROUPS + 1];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = pair_rank();
  const int cluster = blockIdx.x >> 1, clusters = gridDim.x >> 1;
  constexpr int PLANES = SPLIT > 0 ? SPLIT : 1;
  const int kb_total = K / GS_BK, chunk_kb = SPLIT > 0 ? GS_CHUNK_KB : kb_total, m_pairs = (N + 2 * GS_BM - 1) / (2 * GS_BM);

  if (threadIdx.x == 0) {
    for (int s = 0; s < C::STAGES; ++s) {
      mbar_init(smem_u32(&full_bar[s]), 1);
      mbar_init(smem_u32(&empty_bar[s]), 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(smem_u32(&tmem_full_bar[a]), 1);
      mbar_init(smem_u32(&tmem_empty_bar[a]), 2 * GS_EPI_WARPS);
    }
    mbar_init(smem_u32(&drained), 1);
    gave_up = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(C::TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  pdl_wait();   // (rows of x and the groups' table are the kernels' in front)
  if (threadIdx.x == 0) pdl_launch_dependents();
  if (offsets != nullptr) {
    for (int i = threadIdx.x; i <= groups; i += GS_THREADS) s_off[i] = min(max(offsets[i], 0), rows_total);
  } else {   // groups of the same size
    for (int i = threadIdx.x; i <= groups; i += GS_THREADS) s_off[i] = rows_total / groups * i;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_slot;
  const B2Waits wait{&gave_up, limit};
  pair_cluster_sync();  // the peer's barriers exist before anything of mine can arrive on them, and its TMEM is taken
  int sent = 0;       // (producer: stages filled)

  auto produce = [&]() {   // (one thread)
    tma_prefetch_desc(&tmap_w);
    tma_prefetch_desc(&tmap_x);
    GsWalk<BN> w(s_off, groups, m_pairs);
    for (int p = cluster; w.at(p); p += clusters) {
      const int wrow = w.g * N + (2 * w.pair + (int)rank) * GS_BM;   // (rows past the group's N: the next group's or zeros, not stored)
      const int xrow = w.row0 + (int)rank * (BN / 2);
      for (int c0 = 0; c0 < kb_total; c0 += chunk_kb)
        for (int plane = PLANES - 1; plane >= 0; --plane)
          for (int kb = c0; kb < min(kb_total, c0 + chunk_kb); ++kb) {
            const int s = sent % C::STAGES;
            if (!wait(empty_bar[s], ((sent / C::STAGES) & 1) ^ 1)) return;  // the pair's MMAs are done with this stage
            const uint32_t fb = pair_first_cta(smem_u32(&full_bar[s]));
            if (rank == 0) mbar_arrive_expect_tx(smem_u32(&full_bar[s]), 2 * C::STAGE_BYTES);
            const uint32_t ws = smem_base + s * C::STAGE_BYTES;
            pair_tma_load_2d(ws, &tmap_w, kb * GS_BK, wrow, fb);
            pair_tma_load_2d(ws + GS_W_BYTES, &tmap_x, kb * GS_BK, plane * rows_total + xrow, fb);   // (rows behind a plane's end: the next plane's, not stored)
            ++sent;
          }
    }
    // the releases of the last stages have landed on this CTA's barriers before it goes to the final cluster barrier and exits
    for (int j = max(0, sent - C::STAGES); j < sent; ++j)
      if (!wait(empty_bar[j % C::STAGES], (j / C::STAGES) & 1)) return;
  };
  auto multiply = [&]() {   // (one thread of the first CTA)
    constexpr uint32_t idesc = umma_idesc_bf16(2 * GS_BM, BN);
    int it = 0, lt = 0;
    GsWalk<BN> w(s_off, groups, m_pairs);
    for (int p = cluster; w.at(p); p += clusters)
      for (int c0 = 0; c0 < kb_total; c0 += chunk_kb, ++lt) {
        const int as = lt & 1, steps = PLANES * min(chunk_kb, kb_total - c0);
        if (!wait(tmem_empty_bar[as], ((lt >> 1) & 1) ^ 1)) return;
        tc_fence_after();
        const uint32_t tmem_d = tmem_base + (uint32_t)(as * BN);
        for (int i = 0; i < steps; ++i, ++it) {
          const int s = it % C::STAGES;
          if (!wait(full_bar[s], (it / C::STAGES) & 1)) return;
          tc_fence_after();
          const uint32_t ws = smem_base + s * C::STAGE_BYTES;
          const uint64_t da = umma_desc_sw128(ws), db = umma_desc_sw128(ws + GS_W_BYTES);
#pragma unroll
          for (int k = 0; k < GS_BK / 16; ++k)
            pair_mma_bf16(tmem_d, da + (uint64_t)(2 * k), db + (uint64_t)(2 * k), idesc, (i > 0 || k > 0) ? 1u : 0u);
          pair_commit(smem_u32(&empty_bar[s]));
        }
        pair_commit(smem_u32(&tmem_full_bar[as]));
      }
  };
  auto finish = [&]() {
    // thread = weight row (TMEM lane), two warps per lane quarter that take every other 32 rows of x
    const int q = warp & 3, half = (warp - 2) >> 2;
    int lt = 0;
    GsWalk<BN> w(s_off, groups, m_pairs);
    auto hand_back = [&](int as) {   // this warp's share of the accumulator is in registers: back to the MMA thread, which waits for both CTAs' warps
      tc_fence_before();
      __syncwarp();
      if (lane == 0)
        pair_arrive(pair_first_cta(smem_u32(&tmem_empty_bar[as])));
    };
    XieluCoef xc{};
    if constexpr (EPI == SUM_EPI_XIELU) xc = xielu_coef(pq);
    auto store = [&](int c0, int col, const uint32_t (&r)[32]) {   // 32 rows of x from c0 of the tile on, this thread's weight row
      if (col >= N) return;
      const size_t at = (size_t)(w.row0 + c0) * ldo + col;
      const int have = w.rows - c0;   // rows of this block that are the group's
      if constexpr (EPI == SUM_EPI_F32) {
        float* d = reinterpret_cast<float*>(out) + at;
        if (have >= 32) {
#pragma unroll
          for (int j = 0; j < 32; ++j) d[(size_t)j * ldo] = __uint_as_float(r[j]);
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j)
            if (j < have) d[(size_t)j * ldo] = __uint_as_float(r[j]);
        }
      } else {
        bf16* d = reinterpret_cast<bf16*>(out) + at;
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          const float z = __uint_as_float(r[j]), a = fmaxf(z, 0.f);
          if (j < have) d[(size_t)j * ldo] = __float2bfloat16_rn(EPI == SUM_EPI_XIELU ? xielu(xc, z) : a * a);
        }
      }
    };
    for (int p = cluster; w.at(p); p += clusters) {
      const int col = (2 * w.pair + (int)rank) * GS_BM + q * 32 + lane;
      const uint32_t tq = tmem_base + ((uint32_t)(q * 32) << 16);
      if constexpr (SPLIT > 0) {
        uint32_t sum[BN / 64][32];
#pragma unroll
        for (int b = 0; b < BN / 64; ++b)
#pragma unroll
          for (int j = 0; j < 32; ++j) sum[b][j] = 0u;
        for (int c0 = 0; c0 < kb_total; c0 += chunk_kb, ++lt) {
          const int as = lt & 1;
          if (!wait.warp(tmem_full_bar[as], (lt >> 1) & 1)) return;
          tc_fence_after();
#pragma unroll
          for (int b = 0; b < BN / 64; ++b) {
            uint32_t r[32];
            tmem_ld32(tq + (uint32_t)(as * BN + half * 32 + b * 64), r);
            tmem_ld_wait();
            if (b == BN / 64 - 1) hand_back(as);
#pragma unroll
            for (int j = 0; j < 32; ++j) sum[b][j] = __float_as_uint(__uint_as_float(sum[b][j]) + __uint_as_float(r[j]));
          }
        }
#pragma unroll
        for (int b = 0; b < BN / 64; ++b) store(half * 32 + b * 64, col, sum[b]);
      } else {
        const int as = lt & 1;
        if (!wait.warp(tmem_full_bar[as], (lt >> 1) & 1)) return;
        tc_fence_after();
#pragma unroll 1
        for (int c0 = half * 32; c0 < BN; c0 += 64) {
          uint32_t r[32];
          tmem_ld32(tq + (uint32_t)(as * BN + c0), r);
          tmem_ld_wait();
          if (c0 + 64 >= BN) hand_back(as);
          store(c0, col, r);
        }
        ++lt;
      }
    }
  };
  if (warp == 0) {
    if (lane == 0) produce();
  } else if (warp == 1) {
    if (lane == 0 && rank == 0) multiply();
  } else {
    finish();
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (gave_up != 0 && rank == 0 && lane == 0) {   // copies and MMAs of the pair that are under way end before shared memory and TMEM are given back
    if (warp == 0) {
      for (int k = max(0, sent - C::STAGES); k < sent; ++k) b2_drain(full_bar[k % C::STAGES], (k / C::STAGES) & 1);
    } else if (warp == 1) {
      asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(&drained)) : "memory");
      b2_drain(drained, 0);
    }
  }
  // no CTA leaves while its peer's loads may still be counted on its barriers, or the pair's MMAs read its shared memory
  __syncwarp();
  pair_cluster_sync();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(C::TMEM_COLS) : "memory");
  }
}

// planes [3][n] bf16 whose sum is x: every plane the nearest bf16 to what is left (a value that rounds to infinity is cut instead; infinities and NaN stay in the first).
// w given: fp32 numbers that are bf16 numbers, written to narrow as such
__global__ void __launch_bounds__(256) split3_kernel(const float4* x, uint2* planes, size_t n4, const uint4* __restrict__ w, uint2* narrow, size_t w4) {
  pdl_wait();
  pdl_launch_dependents();
  for (size_t i = (size_t)blockIdx.x * 256 + threadIdx.x; i < n4; i += (size_t)gridDim.x * 256) {
    const float4 v = x[i];
    const float in[4] = {v.x, v.y, v.z, v.w};
    uint32_t h[3][4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      float left = in[c];
      const bool finite = fabsf(left) < INFINITY;
#pragma unroll
      for (int p = 0; p < 3; ++p) {
        uint32_t b = (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(left));
        if (finite && (b & 0x7fffu) == 0x7f80u) b = __float_as_uint(left) >> 16;
        h[p][c] = b;
        left = finite ? left - __uint_as_float(b << 16) : 0.f;
      }
    }
#pragma unroll
    for (int p = 0; p < 3; ++p) planes[(size_t)p * n4 + i] = make_uint2(h[p][0] | h[p][1] << 16, h[p][2] | h[p][3] << 16);
  }
#pragma unroll 4
  for (size_t i = (size_t)blockIdx.x * 256 + threadIdx.x; i < w4; i += (size_t)gridDim.x * 256) {
    const uint4 v = w[i];
    narrow[i] = make_uint2(__byte_perm(v.x, v.y, 0x7632), __byte_perm(v.z, v.w, 0x7632));   // (the upper halves)
  }
}

template <int BN, int EPI, int SPLIT = 0>
int launch_sum(const void* x, const void* w, const int32_t* offsets, int groups, int rows, void* out, int N, int K, const B2WaitLimit& wait, cudaStream_t s, int ldo = 0, const float* pq = nullptr) {
  using C = GsCfg<BN>;
  static B2PerDeviceOnce attr_once;
  if (attr_once.need()) B2_CUDA_OK(cudaFuncSetAttribute(linear_sum_kernel<BN, EPI, SPLIT>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES));
  CUtensorMap tw, tx;
  int rc = b2_make_tmap_bf16(&tw, w, (uint64_t)groups * N, (uint64_t)K, (uint64_t)K, GS_BM);
  if (rc == 0) rc = b2_make_tmap_bf16(&tx, x, (uint64_t)rows * (SPLIT > 0 ? SPLIT : 1), (uint64_t)K, (uint64_t)K, BN / 2);
  if (rc != 0) return rc;
  const int m_pairs = (N + 2 * GS_BM - 1) / (2 * GS_BM);
  const long most = ((long)rows / BN + groups) * m_pairs;   // tiles at most
  const int sms = device_num_sms(), clusters = (int)std::min<long>(most, sms / 2);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * clusters);
  cfg.blockDim = dim3(GS_THREADS);
  cfg.dynamicSmemBytes = C::SMEM_BYTES;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = b2_pdl_enabled() ? 2 : 1;
  B2_CUDA_OK(cudaLaunchKernelEx(&cfg, linear_sum_kernel<BN, EPI, SPLIT>, tw, tx, offsets, groups, rows, out, N, K, ldo > 0 ? ldo : N, wait, pq));
  return 0;
}

// The rows of x that a tile takes: 256, or 128 where the busiest cluster then has no more tiles to do.  A 128-row tile takes 0.84 - 0.93 of the time of a
// 256-row one (24 KB per k-block and SM instead of 32, and the same waits, for half the MMAs): 8192 x 12288 x 2048 510 us against 304, 1011 x 2048 x 2048 (one wave
// of either) 17.1 against 18.0, 512 x 1024 x 1024 10.3 against 11.7.
int sum_pick_bn(int rows, int groups, int N) {
  const long m_pairs = (N + 2 * GS_BM - 1) / (2 * GS_BM), clusters = device_num_sms() / 2;
  auto waves = [&](int bn) {
    const long tiles = (((long)rows + bn - 1) / bn + (groups - 1) / 2) * m_pairs;   // (half a tile more per group on average)
    return (tiles + clusters - 1) / clusters;
  };
  return waves(128) <= waves(256) ? 128 : 256;
}

}  // namespace

// One block of rows: from two tiles per cluster on the pairs are faster than gemm_tc.cu's single CTAs (us, pairs / single: 1011 x 12288 x 2048 46 / 50, 3000 x 6144 x 2048
// 59 / 63, 8192 x 2048 x 2048 61 / 66, 8192 x 12288 x 2048 305 / 350); below they start later and reduce nothing (2000 x 2048 x 2048 20.6 / 18.0, 8192 x 1024 x 1024 28 / 26).
bool linear_sum_pays(int rows, int N) { return ((long)rows + 255) / 256 * ((N + 255) / 256) > 2L * (device_num_sms() / 2); }

bool linear_sum_shapes_ok(int rows, int groups, int N, int K) { return rows >= 1 && groups >= 1 && groups <= GS_MAX_GROUPS && N >= 64 && K >= 64 && K % GS_BK == 0; }

int launch_linear_sum(const void* x, const void* w, const int32_t* offsets, int groups, int rows, void* out, int N, int K, int epilogue, const B2WaitLimit& wait,
                      cudaStream_t s, int bn, const float* pq) {
  if (rows <= 0) return 0;
  B2_REQUIRE(epilogue != SUM_EPI_XIELU || pq != nullptr, "linear_sum: the activation needs its numbers");
  B2_REQUIRE(linear_sum_shapes_ok(rows, groups, N, K) && (offsets != nullptr || rows % groups == 0), "linear_sum: %d rows in %d groups, N=%d K=%d not built", rows, groups, N, K);
  if (bn == 0) bn = sum_pick_bn(rows, groups, N);
#define B2_SUM_CASE(B, E) if (bn == B && epilogue == E) return launch_sum<B, E>(x, w, offsets, groups, rows, out, N, K, wait, s, 0, pq)
  B2_SUM_CASE(256, SUM_EPI_F32);
  B2_SUM_CASE(128, SUM_EPI_F32);
  B2_SUM_CASE(256, SUM_EPI_RELU2);
  B2_SUM_CASE(128, SUM_EPI_RELU2);
  B2_SUM_CASE(256, SUM_EPI_XIELU);
  B2_SUM_CASE(128, SUM_EPI_XIELU);
#undef B2_SUM_CASE
  b2_set_error("linear_sum: tile %d, epilogue %d not built", bn, epilogue);
  return -22;
}

static int launch_split3(const float* x, bf16* planes, size_t nx, const float* w, bf16* narrow, size_t nw, cudaStream_t s) {
  const size_t n4 = nx / 4, w4 = nw / 4;
  B2_CUDA_OK(b2_launch(split3_kernel, dim3((unsigned)std::min<size_t>((std::max(n4, w4) + 255) / 256, (size_t)device_num_sms() * 16)), dim3(256), 0, s, (const float4*)x,
                       (uint2*)planes, n4, (const uint4*)w, (uint2*)narrow, w4));
  return 0;
}
static int launch_planes(const bf16* planes, const bf16* w, float* out, int rows, int N, int K, int ldo, const B2WaitLimit& wait, cudaStream_t s, int bn) {
  if (bn == 0) bn = sum_pick_bn(rows, 1, N);
  return bn == 128 ? launch_sum<128, SUM_EPI_F32, 3>(planes, w, nullptr, 1, rows, out, N, K, wait, s, ldo)
                   : launch_sum<256, SUM_EPI_F32, 3>(planes, w, nullptr, 1, rows, out, N, K, wait, s, ldo);
}
int launch_linear_split3(const float* x, bf16* planes, const bf16* w, float* out, int rows, int N, int K, const B2WaitLimit& wait, cudaStream_t s, int bn) {
  if (rows <= 0) return 0;
  B2_REQUIRE(linear_sum_shapes_ok(rows, 1, N, K) && (reinterpret_cast<uintptr_t>(x) & 15) == 0, "linear_split3: %d rows, N=%d K=%d not built", rows, N, K);
  int rc = launch_split3(x, planes, (size_t)rows * K, nullptr, nullptr, 0, s);
  return rc != 0 ? rc : launch_planes(planes, w, out, rows, N, K, 0, wait, s, bn);
}

// Rows of x and of w that the scratch takes at a time, in whole tiles where they are not all of them (0: none)
static int split3_piece(int rows, int K, size_t numbers) {
  const size_t most = numbers / (size_t)K;
  return (size_t)rows <= most ? rows : (int)(most / 256 * 256);
}
bool linear_split3_wide_ok(const Split3Scratch& t, const void* x, const void* w, int rows, int N, int K) {
  return t.planes != nullptr && t.narrow != nullptr && linear_sum_shapes_ok(rows, 1, N, K) && ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w)) & 15) == 0 &&
         split3_piece(rows, K, t.plane_numbers) > 0 && split3_piece(N, K, t.narrow_numbers) >= std::min(N, 256);
}
int launch_linear_split3_wide(const float* x, const float* w, float* out, int rows, int N, int K, const Split3Scratch& t, const B2WaitLimit& wait, cudaStream_t s) {
  if (rows <= 0) return 0;
  B2_REQUIRE(linear_split3_wide_ok(t, x, w, rows, N, K), "linear_split3_wide: %d rows, N=%d K=%d not built", rows, N, K);
  const int pr = split3_piece(rows, K, t.plane_numbers), pn = split3_piece(N, K, t.narrow_numbers);
  for (int n0 = 0; n0 < N; n0 += pn) {
    const int nn = std::min(pn, N - n0);
    for (int r0 = 0; r0 < rows; r0 += pr) {
      const int rr = std::min(pr, rows - r0);
      int rc = launch_split3(x + (size_t)r0 * K, t.planes, (size_t)rr * K, r0 == 0 ? w + (size_t)n0 * K : nullptr, t.narrow, r0 == 0 ? (size_t)nn * K : 0, s);
      if (rc == 0) rc = launch_planes(t.planes, t.narrow, out + (size_t)r0 * N + n0, rr, nn, K, N, wait, s, 0);
      if (rc != 0) return rc;
    }
  }
  return 0;
}

int launch_linear_sum_fine(const void* x, const void* w, float* out, int rows, int N, int K, const B2WaitLimit& wait, cudaStream_t s) {
  if (rows <= 0) return 0;
  B2_REQUIRE(linear_sum_shapes_ok(rows, 1, N, K), "linear_sum_fine: %d rows, N=%d K=%d not built", rows, N, K);
  return launch_sum<128, SUM_EPI_F32, 1>(x, w, nullptr, 1, rows, out, N, K, wait, s);
}

}  // namespace b2
