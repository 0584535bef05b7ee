// attn_postmix.cu -- prompt attention whose softmax weights are mixed over the heads before they meet the values (Kedasun's gated mixer, up to sixteen heads, bf16 cache):
//   out[t][a] = sigmoid(gate[t][a]) * sum_j (sum_b talk[a][b] P_b[t][j]) v_{kv(a)}[j]
//
// The sum over the heads is linear, so either the outputs are mixed -- then every head's weights meet the values of every key/value head (heads_attention_mma_kernel with
// `cross`, 16 heads on 8 key/value heads: 8 times the products, an fp32 [T][heads][kv heads][vdim] between the two kernels) -- or the weights are, which needs
// them normalised: two passes over the keys, the first for the rows' maxima and sums alone, the second for scores again, weights, mix and one product with the values.
// Per (query, key) pair that is 6 400 multiply-adds instead of 33 000 (16 heads of 128 + 128).
//
// A CTA takes sixteen queries of ALL heads, a warp per head (m16n8k16 MMAs); key tiles of sixteen, keys and values of all key/value heads in shared memory, two
// tiles under way.  Second pass, per tile: warp b writes its weights [16 queries][16 keys] as bf16 pairs high + low; after a barrier warp w mixes query w: the mix is the
// MMA  talk [16 x 16 heads] . P [16 heads x 8 keys], three products of the high and low parts, fp32 sums; the mixed weights, high + low again, replace the weights;
// after another barrier warp a multiplies head a's with the values.  The weights therefore carry sixteen bits into the product where the other form's carried eight.
// Bound: instruction issue (half of the slots) and latencies between the barriers; the tensor pipe is a quarter busy.  4 100 queries of eight prompts, window 512 + 16
// kept, 16 heads on 8 of 128: 600 + 98 us for the cross products and the mix of the outputs, 200 here (16 x 1.7 queries per SM: the last wave is three
// quarters full; 188 without the low parts in the product with the values).
#include "kernels.h"

#include <type_traits>

namespace b2 {

namespace {

constexpr int PX_ROWS = 16, PX_KEYS = 16, PX_HEADS = 16;
constexpr int PX_QLD = PX_KEYS + 8;                         // weights of a query: 16 keys and padding (48 bytes: eight rows of an ldmatrix fall on different banks)
constexpr int PX_HLD = PX_ROWS * PX_QLD + 8;                // ... of a head
constexpr float PX_LOG2E = 1.4426950408889634f;

__device__ __forceinline__ void px_mma(float* c, const uint32_t* a, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void px_ldsm(uint32_t* r, uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void px_ldsm_t(uint32_t* r, uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
// a pair of numbers as two bf16 pairs, high and what it leaves
__device__ __forceinline__ void px_split(float a, float b, uint32_t& hi, uint32_t& lo) {
  hi = pack_bf16x2(a, b);
  lo = pack_bf16x2(a - bf16lo(hi), b - bf16hi(hi));
}

// grid (query tiles * 4 of sixteen rows); block 32 * heads
template <int D, int DV>
__global__ void __launch_bounds__(32 * PX_HEADS, 1)
heads_postmix_kernel(const float* q, const bf16* k_cache, const bf16* v_cache, HeadsGeom g, const int32_t* __restrict__ block_table,
                     int bt_stride, int block_size, const PrefillTile* __restrict__ tiles, const float* __restrict__ talk, const float* gate, int gate_ld,
                     bf16* out) {
  extern __shared__ __align__(128) unsigned char px_smem[];
  constexpr int KC = D / 8, VC = DV / 8;                                         // 16-byte chunks of a row; chunk c of row r lies at c ^ (r & 7)
  bf16* Qs = reinterpret_cast<bf16*>(px_smem);                                   // [heads][16][D]
  bf16* Ks = Qs + g.heads * PX_ROWS * D;                                         // [2][kv heads][16][D]
  bf16* Vs = Ks + 2 * g.kv_heads * PX_KEYS * D;                                  // [2][kv heads][16][DV]
  bf16* Ph = Vs + 2 * g.kv_heads * PX_KEYS * DV;                                 // [2: high, low][16 heads][PX_HLD]
  pdl_wait();
  pdl_launch_dependents();
  const int item = gridDim.x - 1 - blockIdx.x;                                   // the tiles late in a sequence see the most keys: they start first
  PrefillTile tl = tiles[item >> 2];
  const int sub = (item & 3) * PX_ROWS;
  if (sub >= tl.nrows) return;
  tl.q_row0 += sub;
  tl.q_pos0 += sub;
  tl.nrows = min(PX_ROWS, tl.nrows - sub);
  const int nt = blockDim.x, warps = nt >> 5, a = threadIdx.x >> 5, lane = threadIdx.x & 31, gq = lane >> 2, tq = lane & 3;
  const int kvh = a / (g.heads / g.kv_heads), krow = g.kv_heads * D, vrow = g.kv_heads * DV;
  for (int i = threadIdx.x; i < g.heads * PX_ROWS * (D / 4); i += nt) {          // queries: fp32 -> bf16, rows past the tile's end are zero
    const int c4 = i % (D / 4), hr = i / (D / 4), r = hr % PX_ROWS, h = hr / PX_ROWS;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (r < tl.nrows) v = *reinterpret_cast<const float4*>(q + ((size_t)(tl.q_row0 + r) * g.heads + h) * D + c4 * 4);
    *reinterpret_cast<uint2*>(Qs + hr * D + (((c4 >> 1) ^ (r & 7)) * 8) + (c4 & 1) * 4) = make_uint2(pack_bf16x2(v.x, v.y), pack_bf16x2(v.z, v.w));
  }
  for (int i = threadIdx.x; i < 2 * PX_HEADS * PX_HLD / 2; i += nt) reinterpret_cast<uint32_t*>(Ph)[i] = 0u;   // (heads that are not there mix as zeros)
  // the mix as the MMA's 16 x 16 operand, high and low
  uint32_t th[4], tlo[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = gq + (i & 1) * 8, c = 2 * tq + (i >> 1) * 8;
    const float x = r < g.heads && c < g.heads ? talk[r * g.heads + c] : 0.f, y = r < g.heads && c + 1 < g.heads ? talk[r * g.heads + c + 1] : 0.f;
    px_split(x, y, th[i], tlo[i]);
  }
  const float slope = g.slopes ? (float)exp2(-(double)g.slope_exp * (double)(a + 1) / (double)g.heads) : 0.f;
  const int p0 = tl.q_pos0 + gq, p1 = p0 + 8;                                    // this thread's two query rows
  const bool live0 = gq < tl.nrows, live1 = gq + 8 < tl.nrows;
  const int last_key = tl.q_pos0 + tl.nrows - 1, last_tile = last_key / PX_KEYS;
  const int lo_min = first_seen_key(tl.q_pos0, g.window, g.chunk), lo_max = first_seen_key(last_key, g.window, g.chunk);
  const int lo0 = first_seen_key(p0, g.window, g.chunk), lo1 = first_seen_key(p1, g.window, g.chunk);
  const int nA = (min(g.keep_first, lo_min) + PX_KEYS - 1) / PX_KEYS, tB = max(lo_min / PX_KEYS, nA);
  const int total = nA + (last_tile - tB + 1);
  const int psh = (block_size & (block_size - 1)) == 0 ? 31 - __clz(block_size) : -1;
  const int32_t* bt = block_table + (size_t)tl.bt_row * bt_stride;
  auto key_of = [&](int vi) { return (vi < nA ? vi : tB + (vi - nA)) * PX_KEYS; };
  // step i of 2 * total: the first pass takes keys, the second keys and values; a tile's rows are one run of its page; rows past the end are filled with zeros
  auto stage = [&](int i) {
    const int key0 = key_of(i < total ? i : i - total), buf = i & 1;
    const size_t row0 = psh >= 0 ? ((size_t)bt[key0 >> psh] << psh) + (key0 & (block_size - 1)) : (size_t)bt[key0 / block_size] * block_size + key0 % block_size;
    auto rows = [&](const bf16* src, bf16* dst, auto chunks_c, int ld) {         // a warp per row; ld numbers per cache row
      constexpr int chunks = decltype(chunks_c)::value;                          // 16-byte chunks of a head's row
      for (int r = a; r < PX_KEYS; r += warps) {
        const bool in = key0 + r <= last_key;
        const bf16* from = src + (in ? (row0 + r) * ld : 0);
#pragma unroll 4
        for (int hc = lane; hc < ld / 8; hc += 32) {
          const int h = hc / chunks, c = hc % chunks;
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst + ((h * PX_KEYS + r) * chunks + (c ^ (r & 7))) * 8)), "l"(from + hc * 8),
                       "r"(in ? 16 : 0));   // (ordered by the commit and wait below, which do clobber memory)
        }
      }
    };
    rows(k_cache, Ks + buf * g.kv_heads * PX_KEYS * D, std::integral_constant<int, KC>(), krow);
    if (i >= total) rows(v_cache, Vs + buf * g.kv_heads * PX_KEYS * DV, std::integral_constant<int, VC>(), vrow);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  const int fr = (lane & 7) + ((lane >> 3) & 1) * 8, fc = lane >> 4;             // ldmatrix: row and chunk of this lane's address (16 x 16 operand)
  // scores of tile vi in buffer buf: scaled, penalised, masked
  auto scores = [&](int vi, int buf, float (&sc)[2][4]) {
    const int key0 = key_of(vi);
    const bf16* Kt = Ks + (buf * g.kv_heads + kvh) * PX_KEYS * D;
#pragma unroll
    for (int n = 0; n < 2; ++n) sc[n][0] = sc[n][1] = sc[n][2] = sc[n][3] = 0.f;
#pragma unroll
    for (int kk = 0; kk < D / 16; kk += 2) {
      uint32_t q0[4], q1[4];
      px_ldsm(q0, smem_u32(Qs + (a * PX_ROWS + fr) * D + ((kk * 2 + fc) ^ (fr & 7)) * 8));
      px_ldsm(q1, smem_u32(Qs + (a * PX_ROWS + fr) * D + ((kk * 2 + 2 + fc) ^ (fr & 7)) * 8));
#pragma unroll
      for (int n = 0; n < 2; ++n) {
        uint32_t kf[4];   // four 8 x 8 blocks: two k-steps of eight keys
        const int r = n * 8 + (lane & 7);
        px_ldsm(kf, smem_u32(Kt + r * D + ((kk * 2 + (lane >> 3)) ^ (r & 7)) * 8));
        px_mma(sc[n], q0, kf[0], kf[1]);
        px_mma(sc[n], q1, kf[2], kf[3]);
      }
    }
    if (tl.nrows == PX_ROWS && key0 + PX_KEYS - 1 <= tl.q_pos0 && (lo_max <= key0 || key0 + PX_KEYS <= g.keep_first)) {   // a tile that every row sees whole
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) sc[n][e] = sc[n][e] * g.scale - slope * (float)(((e & 2) ? p1 : p0) - (key0 + n * 8 + 2 * tq + (e & 1)));
      return;
    }
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int j = key0 + n * 8 + 2 * tq + (e & 1), p = (e & 2) ? p1 : p0;
        const bool ok = ((e & 2) ? live1 : live0) && j <= p && (j >= ((e & 2) ? lo1 : lo0) || j < g.keep_first);
        sc[n][e] = ok ? sc[n][e] * g.scale - slope * (float)(p - j) : -INFINITY;
      }
  };
  float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f}, o[DV / 8][4];
#pragma unroll
  for (int n = 0; n < DV / 8; ++n) o[n][0] = o[n][1] = o[n][2] = o[n][3] = 0.f;
  stage(0);
  for (int i = 0; i < 2 * total; ++i) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();   // this tile is there for every warp, and every warp has left the other buffer and the weights
    if (i + 1 < 2 * total) stage(i + 1);
    float sc[2][4];
    scores(i < total ? i : i - total, i & 1, sc);
    if (i < total) {   // a thread's own columns; the quads are joined behind the last tile
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const float top = fmaxf(fmaxf(sc[0][2 * r], sc[0][2 * r + 1]), fmaxf(sc[1][2 * r], sc[1][2 * r + 1]));
        const float mn = fmaxf(m[r], top), base = mn == -INFINITY ? 0.f : mn;
        l[r] = l[r] * exp2f((m[r] - base) * PX_LOG2E) + ((exp2f((sc[0][2 * r] - base) * PX_LOG2E) + exp2f((sc[0][2 * r + 1] - base) * PX_LOG2E)) +
                                                         (exp2f((sc[1][2 * r] - base) * PX_LOG2E) + exp2f((sc[1][2 * r + 1] - base) * PX_LOG2E)));
        m[r] = mn;
      }
      if (i + 1 == total) {
#pragma unroll
        for (int r = 0; r < 2; ++r) {
#pragma unroll
          for (int x = 1; x < 4; x <<= 1) {
            const float mo = __shfl_xor_sync(0xffffffffu, m[r], x), lo = __shfl_xor_sync(0xffffffffu, l[r], x);
            const float mn = fmaxf(m[r], mo), base = mn == -INFINITY ? 0.f : mn;
            l[r] = l[r] * exp2f((m[r] - base) * PX_LOG2E) + lo * exp2f((mo - base) * PX_LOG2E);
            m[r] = mn;
          }
          m[r] = m[r] == -INFINITY ? 0.f : m[r];
          l[r] = l[r] == 0.f ? 0.f : 1.0f / l[r];   // from here on: one over the sum (rows past the end: zero)
        }
      }
      continue;
    }
    // ---- weights ----
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        uint32_t hi, lo;
        px_split(exp2f((sc[n][2 * r] - m[r]) * PX_LOG2E) * l[r], exp2f((sc[n][2 * r + 1] - m[r]) * PX_LOG2E) * l[r], hi, lo);
        bf16* dst = Ph + a * PX_HLD + (gq + 8 * r) * PX_QLD + n * 8 + 2 * tq;
        *reinterpret_cast<uint32_t*>(dst) = hi;
        *reinterpret_cast<uint32_t*>(dst + PX_HEADS * PX_HLD) = lo;
      }
    __syncthreads();
    // ---- mix: one query of all heads, in place ----
    for (int qr = a; qr < PX_ROWS; qr += warps) {
      bf16* base = Ph + qr * PX_QLD;
      uint32_t ph[4], pl[4];   // heads 0..7 and 8..15 of keys 0..7, then of keys 8..15
      px_ldsm_t(ph, smem_u32(base + fr * PX_HLD + fc * 8));
      px_ldsm_t(pl, smem_u32(base + PX_HEADS * PX_HLD + fr * PX_HLD + fc * 8));
      __syncwarp();
#pragma unroll
      for (int n = 0; n < 2; ++n) {
        float mx[4] = {0.f, 0.f, 0.f, 0.f};
        px_mma(mx, th, pl[2 * n], pl[2 * n + 1]);
        px_mma(mx, tlo, ph[2 * n], ph[2 * n + 1]);
        px_mma(mx, th, ph[2 * n], ph[2 * n + 1]);
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          uint32_t hi, lo;
          px_split(mx[2 * r], mx[2 * r + 1], hi, lo);
          bf16* dst = base + (gq + 8 * r) * PX_HLD + n * 8 + 2 * tq;
          *reinterpret_cast<uint32_t*>(dst) = hi;
          *reinterpret_cast<uint32_t*>(dst + PX_HEADS * PX_HLD) = lo;
        }
      }
    }
    __syncthreads();
    // ---- head a's mixed weights times the values ----
    uint32_t wh[4], wl[4];
    px_ldsm(wh, smem_u32(Ph + a * PX_HLD + fr * PX_QLD + fc * 8));
    px_ldsm(wl, smem_u32(Ph + PX_HEADS * PX_HLD + a * PX_HLD + fr * PX_QLD + fc * 8));
    const bf16* Vt = Vs + ((i & 1) * g.kv_heads + kvh) * PX_KEYS * DV;
#pragma unroll
    for (int n = 0; n < DV / 8; n += 2) {
      uint32_t vb[4];
      px_ldsm_t(vb, smem_u32(Vt + fr * DV + ((n + fc) ^ (fr & 7)) * 8));
      px_mma(o[n], wl, vb[0], vb[1]);
      px_mma(o[n + 1], wl, vb[2], vb[3]);
      px_mma(o[n], wh, vb[0], vb[1]);
      px_mma(o[n + 1], wh, vb[2], vb[3]);
    }
  }
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    if (!(r ? live1 : live0)) continue;
    const size_t row = (size_t)(tl.q_row0 + gq + 8 * r);
    const float gv = gate ? 1.0f / (1.0f + expf(-gate[row * gate_ld + a])) : 1.0f;
    bf16* orow = out + (row * g.heads + a) * DV + 2 * tq;
#pragma unroll
    for (int n = 0; n < DV / 8; ++n) *reinterpret_cast<uint32_t*>(orow + n * 8) = pack_bf16x2(o[n][2 * r] * gv, o[n][2 * r + 1] * gv);
  }
}

size_t postmix_smem(const HeadsGeom& g) {
  return ((size_t)g.heads * PX_ROWS * g.dim + (size_t)2 * g.kv_heads * PX_KEYS * (g.dim + g.vdim) + (size_t)2 * PX_HEADS * PX_HLD) * sizeof(bf16);
}

template <int D, int DV>
int launch_postmix(const float* q, const bf16* k, const bf16* v, const HeadsGeom& g, const int32_t* bt, int bt_stride, int block_size, const PrefillTile* tiles, int ntiles,
                   const float* talk, const float* gate, int gate_ld, bf16* out, cudaStream_t s) {
  static B2PerDeviceOnce once;
  if (once.need()) B2_CUDA_OK(cudaFuncSetAttribute(heads_postmix_kernel<D, DV>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
  B2_CUDA_OK(b2_launch(heads_postmix_kernel<D, DV>, dim3(ntiles * 4), dim3(32 * g.heads), postmix_smem(g), s, q, k, v, g, bt, bt_stride, block_size, tiles, talk, gate, gate_ld, out));
  return 0;
}

}  // namespace

// Sixteen heads at most (the mix is one 16 x 16 MMA operand), heads of 64 or 128 (a row's chunks are permuted within eight), pages of whole key tiles, tiles of all
// key/value heads twice in shared memory.
bool heads_postmix_ok(const HeadsGeom& g, int block_size) {
  return g.heads >= 1 && g.heads <= PX_HEADS && g.kv_heads >= 1 && g.heads % g.kv_heads == 0 && (g.dim == 64 || g.dim == 128) && (g.vdim == 64 || g.vdim == 128) &&
         block_size > 0 && block_size % PX_KEYS == 0 && postmix_smem(g) <= 227 * 1024;
}

int launch_heads_postmix(const float* q, const bf16* k_cache, const bf16* v_cache, const HeadsGeom& g, const int32_t* block_table, int bt_stride, int block_size,
                         const PrefillTile* tiles, int ntiles, const float* talk, const float* gate, int gate_ld, bf16* out, cudaStream_t s) {
  if (ntiles <= 0) return 0;
  B2_REQUIRE(heads_postmix_ok(g, block_size), "heads_postmix: %d heads of %d and %d, pages of %d not built", g.heads, g.dim, g.vdim, block_size);
#define B2_PX_CASE(A, B) \
  if (g.dim == A && g.vdim == B) return launch_postmix<A, B>(q, k_cache, v_cache, g, block_table, bt_stride, block_size, tiles, ntiles, talk, gate, gate_ld, out, s)
  B2_PX_CASE(128, 128);
  B2_PX_CASE(128, 64);
  B2_PX_CASE(64, 128);
  B2_PX_CASE(64, 64);
#undef B2_PX_CASE
  return -22;
}

}  // namespace b2
