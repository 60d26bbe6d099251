// GEMMs with few rows (decode steps, short sequences): Y[T,N] = X[T,K] W^T, bound by streaming W once.
//
// The tiled kernel of gemm_sm100.cu gives a CTA 128 rows of X and 256 outputs: with 77 rows the
// output projection of a 4096-wide layer is 16 CTAs, each pulling 2 MB of weights through one SM
// (about 80 GB/s), while HBM would feed all 148.  Here the roles are swapped and the contraction is split:
//   * W is the A operand: 128 output features are the 128 lanes of the accumulator, and the tokens
//     are the N dimension of the MMA (a multiple of 16 up to 128), so no MMA or shared-memory bandwidth goes into rows
//     that do not exist beyond the next multiple of 16 (but for the last half chunk of the accumulator's read at 48, 80 or 112);
//   * a cluster of S <= 8 CTAs shares one 128-feature tile, each CTA contracting over 1/S of K.
//     The fp32 partial tiles meet in distributed shared memory, where every CTA adds the S partials of
//     1/S of the tokens in rank order (no workspace, no atomics, the same result every run).
// Two CTAs fit an SM, so one's pipeline fill overlaps the other's epilogue.
// 77 rows of a 4096-wide layer with 14336-wide MLP, us per call before / now: q|k|v 36 / 18, o 34 / 15, gate|up
// 56 / 49, down 98 / 29 (4.0 TB/s); one row of a 102,400 x 2048 head 133 / 66 (6.3 TB/s).
//
//   warp 0      TMA producer: ring of {W 128x64, X NTx64} stages
//   warp 1      MMA issuer: tcgen05.mma 128 x NT x 16
//   warps 2..5  accumulator (TMEM) -> shared memory; then all warps reduce and write
//
// W may be stored [N][K] (forward) or [K][N] (input gradients, expert weights); with the latter X may be
// [K][T] too (weight gradients with few tiles: C = dY^T X contracts over the tokens).  With the SwiGLU
// epilogue a tile is 64 gate and the same 64 up features.  Grouped mode: rows are grouped by expert in
// segments padded to the token-tile width, so a token tile belongs to one expert.
//
// F32 instantiations are for results that are kept in fp32 (router and inference logits).  The tensor core cuts an
// accumulator to 24 bits after every MMA, towards zero: over K = 2048 such a sum is 2e-6 off, an fp32 one 1e-7.  Here
// every MMA (16 products) starts from zero in columns of its own, and warps 2..5 add up the results k-block by k-block
// as pairs of floats (sum and what the sum's rounding lost).  Distance from 64 bits 3e-8 to 5e-8 for K from 512 to 7168,
// where the library's fp32 product of fp32 copies is 6e-8 to 1.2e-6 off.  Bound by memory for a vocabulary head and by those
// additions for a router; us, this / sums left in the accumulator / library: 4 x 102,400 x 2048 71 / 68 / 790,
// 1500 x 64 x 2048 15 / 7 / 46, 3000 x 256 x 7168 119 / 20 / 353.

#include "common.cuh"
#include "tpb.h"

namespace tpb {

int make_tmap_2d(CUtensorMap* map, const void* ptr, uint64_t inner, uint64_t outer, uint64_t pitch_elems,
                 uint32_t box_inner, uint32_t box_outer, int elem_bytes);  // tma.cu
int make_tmap_3d(CUtensorMap* map, const void* ptr, uint64_t d0, uint64_t d1, uint64_t d2, uint64_t stride1_elems,
                 uint64_t stride2_elems, uint32_t box0, uint32_t box1);
int sm_count();  // runtime.cu

constexpr int SK_THREADS = 192;
constexpr int SK_TN = 128;                       // output features per tile
constexpr int SK_BK = 64;
constexpr int SK_W_BYTES = SK_TN * SK_BK * 2;    // 16 KB
constexpr int SK_MAX_SPLIT = 8;                  // portable cluster size
constexpr int SK_PREFETCH = 8;                   // k-blocks asked for ahead of the kernel before: 128 KB a CTA, 38 MB in all

// A tile holds `nt` rows of X, a multiple of 16 up to the instantiation's NT: no MMA, no shared memory and no exchange for
// more.  The smaller tile leaves room for more stages.  (A decoder layer of 77 tokens, 4096 wide with a 14336-wide MLP,
// as tiles of 80 rows instead of 128: 122 -> 116 us.)
constexpr int SK_MAX_STAGES = 6;
constexpr int SK_RING = 108 * 1024;              // two CTAs per SM
constexpr int SK_SMEM = SK_RING + 1024 + 256;
static_assert(2 * (SK_SMEM + 1024) <= 227 * 1024 + 1024, "two CTAs per SM");
static int skinny_stage(int nt) { return SK_W_BYTES + nt * SK_BK * 2; }
static int skinny_stages(int nt) { return SK_RING / skinny_stage(nt) < SK_MAX_STAGES ? SK_RING / skinny_stage(nt) : SK_MAX_STAGES; }

struct SkinnyParams {
  int T, N, K;          // N: output columns (for SwiGLU: of the activation, i.e. half the features of W)
  void* C;
  long long ldc;
  const __nv_bfloat16* aux;
  long long ldaux;
  __nv_bfloat16* c2;    // SwiGLU: [gate | up] before the activation, or null
  long long ldc2;
  int up_off;           // SwiGLU: feature offset of the "up" half inside the second W map
  float alpha;
  const float* alpha_dev;   // one more factor, in device memory, or null
  int epi;
  int t_tiles, splits, num_kb, kb_per;
  int nt, stages, stage_bytes;
  const int* tile_expert;   // grouped: expert of every token tile (-1: unused); null: dense
  int* status;
  // Two products of one X: feature tiles from n1_tiles on are those of the second W (the second map), with results of their
  // own.  INT_MAX: one product.
  int n1_tiles, N2;
  void* C2;
  long long ldC2;
};

// (hi, lo) += c, with lo the sum of hi's rounding errors.
__device__ __forceinline__ void add_two(float& hi, float& lo, float c) {
  const float s = __fadd_rn(hi, c), t = __fsub_rn(s, hi);
  lo = __fadd_rn(lo, __fadd_rn(__fsub_rn(hi, __fsub_rn(s, t)), __fsub_rn(c, t)));
  hi = s;
}

__device__ __forceinline__ float4 ld_dsmem4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(addr)
               : "memory");
  return v;
}

// Sum of the S partials of 4 consecutive features, in rank order; all loads are in flight together.
__device__ __forceinline__ float4 sum_partials(uint32_t local_addr, int splits) {
  float4 v[SK_MAX_SPLIT];
#pragma unroll
  for (int s = 0; s < SK_MAX_SPLIT; ++s)
    if (s < splits) v[s] = ld_dsmem4(map_to_cta(local_addr, s));
  float4 a = v[0];
#pragma unroll
  for (int s = 1; s < SK_MAX_SPLIT; ++s)
    if (s < splits) { a.x += v[s].x; a.y += v[s].y; a.z += v[s].z; a.w += v[s].w; }
  return a;
}

// The same for partials kept as pairs (`lo_off` bytes apart), added in 64 bits and rounded once.
__device__ __forceinline__ float4 sum_pairs(uint32_t local_addr, uint32_t lo_off, int splits) {
  double a[4] = {};
  for (int s = 0; s < splits; ++s) {
    const float4 h = ld_dsmem4(map_to_cta(local_addr, s)), l = ld_dsmem4(map_to_cta(local_addr + lo_off, s));
    a[0] += (double)h.x + l.x; a[1] += (double)h.y + l.y; a[2] += (double)h.z + l.z; a[3] += (double)h.w + l.w;
  }
  return make_float4((float)a[0], (float)a[1], (float)a[2], (float)a[3]);
}

// `n` (1..4) consecutive bf16 results; 8-byte store when all four exist.
__device__ __forceinline__ void store4(__nv_bfloat16* dst, const float4& v, int n) {
  if (n >= 4) {
    *reinterpret_cast<uint2*>(dst) = make_uint2(pack_bf16(v.x, v.y), pack_bf16(v.z, v.w));
  } else {
    const float f[4] = {v.x, v.y, v.z, v.w};
    for (int j = 0; j < n; ++j) dst[j] = __float2bfloat16(f[j]);
  }
}

template <int NT, bool W_MN, bool X_MN, bool F32>
__global__ void __launch_bounds__(SK_THREADS, 2)
gemm_skinny_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmW2,
                   const __grid_constant__ CUtensorMap tmX, const SkinnyParams p) {
  constexpr int KSTEPS = SK_BK / 16;
  constexpr uint32_t TMEM_COLS = F32 ? 2 * KSTEPS * NT : NT < 32 ? 32 : NT;   // F32: two buffers of a k-block's results
  static_assert(!F32 || TMEM_COLS <= 256, "two CTAs per SM");
  static_assert((F32 ? 2 : 1) * NT * SK_TN * 4 <= 4 * (SK_W_BYTES + 16 * SK_BK * 2), "the fp32 partial tiles reuse the ring");
  const int nt = F32 || X_MN ? NT : p.nt;               // rows of X in a tile
  const int stages = p.stages, stage_bytes = p.stage_bytes;
  const bool swiglu = p.epi == TPB_EPI_SWIGLU;
  const int rank = (int)blockIdx.x % p.splits;          // == %cluster_ctarank of the 1-D cluster
  const int unit = (int)blockIdx.x / p.splits;
  const int bt = unit % p.t_tiles;                      // token tiles of one W tile run together (L2)
  const int t0 = bt * nt;
  const bool second = unit / p.t_tiles >= p.n1_tiles;
  const int n0 = (unit / p.t_tiles - (second ? p.n1_tiles : 0)) * (swiglu ? SK_TN / 2 : SK_TN);
  const CUtensorMap* mw = second ? &tmW2 : &tmW;        // the tile's first 64 features
  const CUtensorMap* mw_hi = swiglu ? &tmW2 : mw;       // and the others
  const int N = second ? p.N2 : p.N;
  int ez = 0;
  if (p.tile_expert) {
    if (!chain_wait()) return;
    ez = p.tile_expert[bt];
    if (ez < 0) return;      // the whole cluster leaves together
  }

  extern __shared__ uint8_t sk_smem_raw[];
  uint8_t* smem = sk_smem_raw + ((1024u - (smem_u32(sk_smem_raw) & 1023u)) & 1023u);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + SK_RING);
  uint64_t* empty = full + SK_MAX_STAGES;
  uint64_t* acc_full = empty + SK_MAX_STAGES;
  uint64_t* blk_full = acc_full + 1;      // F32: [2] a k-block's results are in their buffer
  uint64_t* blk_empty = blk_full + 2;     // F32: [2] and have been read (one arrival per warp)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(blk_empty + 2);
  float* part = reinterpret_cast<float*>(smem);         // [NT][128] after the main loop

  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int kb0 = rank * p.kb_per, kb1 = min(p.num_kb, kb0 + p.kb_per);

  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(acc_full, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&blk_full[i], 1);
      mbar_init(&blk_empty[i], 4);
    }
    fence_barrier_init();
    if (!p.tile_expert) {
      // The weights do not come from the kernel before: their first tiles move to L2 while it still runs.
      const int nb = swiglu ? p.up_off + n0 : n0 + 64;
      for (int kb = kb0; kb < min(kb1, kb0 + SK_PREFETCH); ++kb) {
        const int k0 = kb * SK_BK;
        tma_prefetch_3d(mw, W_MN ? n0 : k0, W_MN ? k0 : n0, 0);
        tma_prefetch_3d(mw_hi, W_MN ? nb : k0, W_MN ? k0 : nb, 0);
      }
    }
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  chain_launch();
  if (!chain_wait()) return;

  if (warp == 0) {
    if (elect_one()) {
      tma_prefetch_desc(mw);
      tma_prefetch_desc(&tmX);
      int stage = 0;
      uint32_t phase = 0;
      const int nb = swiglu ? p.up_off + n0 : n0 + 64;   // second half of the 128 features
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!mbar_wait(&empty[stage], phase ^ 1, p.status, kTimeoutStageFree, 81)) break;
        uint8_t* sW = smem + stage * stage_bytes;
        const int k0 = kb * SK_BK;
        mbar_expect_tx(&full[stage], stage_bytes);
        if (!W_MN) {          // boxes {64 k, 64 features}
          tma_load_3d(sW, mw, &full[stage], k0, n0, ez);
          tma_load_3d(sW + SK_W_BYTES / 2, mw_hi, &full[stage], k0, nb, ez);
        } else {              // boxes {64 features, 64 k}
          tma_load_3d(sW, mw, &full[stage], n0, k0, ez);
          tma_load_3d(sW + SK_W_BYTES / 2, mw_hi, &full[stage], nb, k0, ez);
        }
        if (!X_MN) {
          tma_load_2d(sW + SK_W_BYTES, &tmX, &full[stage], k0, t0);
        } else {              // boxes {64 rows of X, 64 k}
#pragma unroll
          for (int c = 0; c < NT / 64; ++c) tma_load_2d(sW + SK_W_BYTES + c * 8192, &tmX, &full[stage], t0 + c * 64, k0);
        }
        if (++stage == stages) {
          stage = 0;
          phase ^= 1;
        }
      }
    }
  } else if (warp == 1) {
    if (kb1 > kb0) {
      const uint32_t idesc = make_idesc_bf16(SK_TN, nt, W_MN, X_MN);
      constexpr uint32_t desc_hi = smem_desc_hi(1024);
      const uint32_t base = smem_u32(smem);
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!mbar_wait_warp(&full[stage], phase, p.status, kTimeoutTmaFull, 82)) { ok = false; break; }
        const int blk = kb - kb0;
        if (F32 && !mbar_wait_warp(&blk_empty[blk & 1], ((blk >> 1) & 1) ^ 1, p.status, kTimeoutAccFree, 84)) { ok = false; break; }
        tc_fence_after();
        const uint32_t sW = base + stage * stage_bytes;
        const uint32_t a_lo = smem_desc_lo(sW, W_MN ? 8192 : 16);
        const uint32_t b_lo = smem_desc_lo(sW + SK_W_BYTES, X_MN ? 8192 : 16);
        one_lane([&] {
#pragma unroll
          for (int k = 0; k < KSTEPS; ++k)
            mma_ss_w(F32 ? tmem_base + ((blk & 1) * KSTEPS + k) * NT : tmem_base, a_lo + (W_MN ? k * 128 : k * 2), desc_hi,
                     b_lo + (X_MN ? k * 128 : k * 2), desc_hi, idesc, !F32 && (blk | k) != 0);
          tc_commit(&empty[stage]);
          if (F32) tc_commit(&blk_full[blk & 1]);
        });
        if (++stage == stages) {
          stage = 0;
          phase ^= 1;
        }
      }
      if (ok && !F32) one_lane([&] { tc_commit(acc_full); });
    }
  } else if (F32) {
    const int q = warp & 3;
    const uint32_t t_addr = tmem_base + ((uint32_t)(q * 32) << 16);
    const int live = min(NT, p.T - t0);          // tokens of this tile
    float hi[NT], lo[NT];
#pragma unroll
    for (int j = 0; j < NT; ++j) hi[j] = lo[j] = 0.f;
    bool have = true;
    for (int kb = kb0; kb < kb1; ++kb) {
      const int blk = kb - kb0;
      have = __all_sync(0xffffffffu, mbar_wait(&blk_full[blk & 1], (blk >> 1) & 1, p.status, kTimeoutAccFull, 85));
      if (!have) break;
      tc_fence_after();
      constexpr int PER = 64 / NT;               // MMAs whose results are read together
#pragma unroll
      for (int k0 = 0; k0 < KSTEPS; k0 += PER) {
        uint32_t v[64];
#pragma unroll
        for (int k = 0; k < PER; ++k) {
          const uint32_t col = t_addr + ((blk & 1) * KSTEPS + k0 + k) * NT;
          if (NT == 16) tmem_ld16(col, v + k * NT); else tmem_ld32(col, v + k * NT);
        }
        tmem_wait_ld();
        if (k0 + PER == KSTEPS) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&blk_empty[blk & 1]);
        }
#pragma unroll
        for (int j0 = 0; j0 < NT; j0 += 4)
          if (j0 < live) {
#pragma unroll
            for (int j = j0; j < j0 + 4; ++j) {
              float c = __fadd_rn(__uint_as_float(v[j]), __uint_as_float(v[NT + j]));
              if (PER == 4) c = __fadd_rn(c, __fadd_rn(__uint_as_float(v[2 * NT + j]), __uint_as_float(v[3 * NT + j])));
              add_two(hi[j], lo[j], c);
            }
          }
      }
    }
    if (have) {                                  // (every MMA has read its operands: the ring is free)
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        part[j * SK_TN + q * 32 + lane] = hi[j];
        part[(NT + j) * SK_TN + q * 32 + lane] = fabsf(hi[j]) <= 3.402823466e38f ? lo[j] : 0.f;   // inf and NaN stay as they are
      }
    }
    tc_fence_before();
  } else {
    // accumulator lane = feature, column = token: part[token][feature], conflict-free
    const int q = warp & 3;
    const int f = q * 32 + lane;
    const uint32_t t_addr = tmem_base + ((uint32_t)(q * 32) << 16);
    bool have = kb1 > kb0;
    if (have) have = mbar_wait(acc_full, 0, p.status, kTimeoutAccFull, 83);
    tc_fence_after();
    if (kb1 <= kb0 || have) {   // (after a wait that ran out copies may still be landing in the ring)
      constexpr int CH = NT < 32 ? 16 : 32;
#pragma unroll 1
      for (int c = 0; c < nt; c += CH) {      // (of a last half chunk the rest is written and not read)
        uint32_t v[CH];
        if (have) {
          if (CH == 16) tmem_ld16(t_addr + c, v); else tmem_ld32(t_addr + c, v);
          tmem_wait_ld();
        } else {
#pragma unroll
          for (int j = 0; j < CH; ++j) v[j] = 0;
        }
#pragma unroll
        for (int j = 0; j < CH; ++j) part[(c + j) * SK_TN + f] = __uint_as_float(v[j]);
      }
    }
    tc_fence_before();
  }
  __syncwarp();
  cluster_sync_all();           // every CTA's partial tile is in its shared memory

  {
    const float alpha = p.alpha_dev ? p.alpha * *p.alpha_dev : p.alpha;
    const int per = nt / p.splits;                    // tokens this CTA finishes (splits divides 16)
    const int gpt = swiglu ? SK_TN / 8 : SK_TN / 4;   // groups of four features per token
    for (int i = threadIdx.x; i < per * gpt; i += SK_THREADS) {
      const int t = rank * per + i / gpt, c = (i % gpt) * 4;
      const int row = t0 + t, col = n0 + c;
      if (row >= p.T || col >= N) continue;
      const int n = min(4, N - col);
      // (the residual is asked for ahead of the neighbours' sums)
      const __nv_bfloat16* res = p.epi == TPB_EPI_BF16_RES ? p.aux + (long long)row * p.ldaux + col : nullptr;
      uint2 old = make_uint2(0, 0);
      if (res && n >= 4) old = *reinterpret_cast<const uint2*>(res);
      float4 a = F32 ? sum_pairs(smem_u32(part + t * SK_TN + c), NT * SK_TN * 4, p.splits)
                     : sum_partials(smem_u32(part + t * SK_TN + c), p.splits);
      a.x *= alpha; a.y *= alpha; a.z *= alpha; a.w *= alpha;
      if (swiglu) {
        float4 u = sum_partials(smem_u32(part + t * SK_TN + SK_TN / 2 + c), p.splits);
        u.x *= alpha; u.y *= alpha; u.z *= alpha; u.w *= alpha;
        if (p.c2) {
          store4(p.c2 + (long long)row * p.ldc2 + col, a, n);
          store4(p.c2 + (long long)row * p.ldc2 + p.N + col, u, n);
        }
        a.x = a.x / (1.0f + __expf(-a.x)) * u.x; a.y = a.y / (1.0f + __expf(-a.y)) * u.y;
        a.z = a.z / (1.0f + __expf(-a.z)) * u.z; a.w = a.w / (1.0f + __expf(-a.w)) * u.w;
      }
      if (p.epi == TPB_EPI_F32) {
        float* dst = reinterpret_cast<float*>(p.C) + (long long)row * p.ldc + col;
        if (n >= 4) {
          *reinterpret_cast<float4*>(dst) = a;
        } else {
          const float f[4] = {a.x, a.y, a.z, a.w};
          for (int j = 0; j < n; ++j) dst[j] = f[j];
        }
        continue;
      }
      if (res) {
        if (n >= 4) {
          const float2 r0 = unpack_bf16(old.x), r1 = unpack_bf16(old.y);
          a.x += r0.x; a.y += r0.y; a.z += r1.x; a.w += r1.y;
        } else {
          a.x += __bfloat162float(res[0]);
          if (n > 1) a.y += __bfloat162float(res[1]);
          if (n > 2) a.z += __bfloat162float(res[2]);
        }
      }
      store4(reinterpret_cast<__nv_bfloat16*>(second ? p.C2 : p.C) + (long long)row * (second ? p.ldC2 : p.ldc) + col, a, n);
    }
  }
  __syncwarp();
  cluster_leave();           // nobody's shared memory goes away while a neighbour reads it
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

template <int NT, bool W_MN, bool X_MN = false, bool F32 = false>
static cudaError_t launch_skinny(const CUtensorMap& tw, const CUtensorMap& tw2, const CUtensorMap& tx,
                                 const SkinnyParams& p, int grid, cudaStream_t stream) {
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(gemm_skinny_kernel<NT, W_MN, X_MN, F32>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         SK_SMEM);
    if (e != cudaSuccess) return e;
    configured = true;
  }
  return chain_clusters(gemm_skinny_kernel<NT, W_MN, X_MN, F32>, p.splits, grid, SK_THREADS, SK_SMEM, stream, tw, tw2,
                        tx, p);
}

// Rows of a token tile: equal tiles of 128 rows at most, to the next multiple of 16.
static int skinny_nt(int rows) {
  const int tiles = (rows + 127) / 128;
  return ((rows + tiles - 1) / tiles + 15) / 16 * 16;
}

// K splits: double while the grid still fits the machine at two CTAs per SM and every CTA keeps four
// k-blocks (256 of K) to amortise its pipeline fill.
static int skinny_splits(long long tiles, int num_kb) {
  int s = 1;
  while (s < SK_MAX_SPLIT && tiles * s * 2 <= 2LL * sm_count() && num_kb / (2 * s) >= 4) s *= 2;
  return s;
}

// Whether this kernel is the faster one for a dense product of M rows.  Up to 128 rows (one token tile) the tiled kernel
// has few CTAs, each with the whole contraction; what this one adds is an epilogue whose length goes with the rows, so a
// short contraction does not pay for many of them (us, weights from HBM, tiled kernel / this one, 4096 outputs):
//   K = 256:  32 rows 6.5 / 5.8, 64 rows 6.6 / 7.1     K = 512: 64 rows 8.5 / 7.4, 96 rows 8.7 / 9.1
//   K = 1024: 128 rows 12.2 / 9.2                      K = 4096: 32 / 15    (28672 outputs, K = 1024: 20.3 / 21.0)
// Beyond that while the tiled kernel's 128 x 256 tiles leave half of the SMs idle (three quarters for a contraction that is
// hardly worth splitting); by the number of its tiles (N x K):
//   1024 x 1024: 32 tiles 10.8 / 10.5, 48 tiles 10.6 / 12.0      576 x 1536: 36 tiles 12.8 / 10.7, 72 tiles 13.0 / 13.8
//   4096 x 2048: 32 tiles 18.7 / 13.0, 64 tiles 18.6 / 16.3      3072 x 2048: 36 tiles 18.4 / 19.2, 72 tiles 18.5 / 16.3
//   4096 x 4096: 64 tiles 32 / 24, 96 tiles 32 / 36              2048 x 10944: 64 tiles 74 / 47, 96 tiles 75 / 77
bool skinny_wins(int M, int N, int K, bool swiglu) {
  if (M <= 128) return M <= 32 || 8 * M <= K;
  if (K < 1024) return false;
  const long long tiles = (long long)((M + 127) / 128) * (((swiglu ? N / 2 : N) + (swiglu ? 127 : 255)) / (swiglu ? 128 : 256));
  return tiles <= sm_count() / (K < 2048 ? 4 : 2);
}

// The same for a weight gradient (both operands contracted over their rows, K of them): bound by the tensor cores,
// so only where the tiled kernel leaves half of the SMs idle, and with a contraction that pays for the split.
// us per call, tiled / this kernel, for 256, 1024, 4096 rows:
//   576 x 2048, 40 tiles: 7 / 10, 13 / 12, 31 / 22      4096 x 512, 64 tiles: 8 / 11, 13 / 13, 31 / 23
//   64 x 2048, 8 tiles: 7 / 7, 11 / 7, 31 / 10          2048 x 2048, 128 tiles: 8 / 13, 13 / 18, 34 / 37
// Against the CTA pairs that take 256 x 256 tiles otherwise, 1500, 2048, 3000 rows, pairs / this kernel (with the launch):
//   4096 x 512: 12.7 / 14.2, 15.4 / 16.0, 19.6 / 19.2      576 x 2048: 12.1 / 13.0, 14.7 / 14.6, 19.0 / 17.7
//   2048 x 1024: 12.6 / 13.4, 15.2 / 15.1, 19.6 / 18.5
bool skinny_wins_wgrad(int M, int N, int K) {
  const long long tiles = (long long)((M + 127) / 128) * ((N + 255) / 256);
  return K >= (tiles <= 16 ? 1024 : 2048) && tiles <= sm_count() / 2;
}

// x [T,K], or [K,T] with x_mn (for grouped mode: all padded rows), w dense [N,K] (w_mn = 0) or [K,N] (w_mn = 1), with
// `experts` of them `w_stride` elements apart.  N counts both halves for SwiGLU.  nt / splits 0: by
// the rules above.  f32: sums as exact as fp32 ones (the F32 kernels; w [N,K], x [T,K]).  Returns -2 when the shape or
// alignment is not supported.
int skinny_gemm(const void* x, const void* w, const void* w2, void* c, int T, int N, int K, int experts,
                long long ldx, long long ldw, long long w_stride, long long ldc, int x_mn, int w_mn, int epi, float alpha,
                const void* aux, long long ldaux, void* c2, long long ldc2, const int* tile_expert, int experts_hit,
                int nt, int splits, cudaStream_t stream, bool f32, const float* alpha_dev) {
  if (T <= 0 || N <= 0 || K <= 0) return 0;
  const bool swiglu = epi == TPB_EPI_SWIGLU;
  if (!swiglu && epi != TPB_EPI_BF16 && epi != TPB_EPI_BF16_RES && epi != TPB_EPI_F32) return -2;
  auto misaligned = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) % 16) != 0; };
  if ((ldx % 8) || (ldw % 8) || (w_stride % 8) || (ldc % (epi == TPB_EPI_F32 ? 4 : 8)) || misaligned(x) ||
      misaligned(w) || (w2 && misaligned(w2)) || misaligned(c))
    return -2;
  if (swiglu && ((N % 2) || ((N / 2) % 8) || (c2 && ((ldc2 % 4) || (reinterpret_cast<uintptr_t>(c2) % 8))))) return -2;
  if (epi == TPB_EPI_BF16_RES && (!aux || (ldaux % 4) || (reinterpret_cast<uintptr_t>(aux) % 8))) return -2;
  if (tile_expert && (nt == 0 || T % nt)) return -2;
  const bool two_w = swiglu && w2 != nullptr && w2 != w;
  const int extent = two_w ? N / 2 : N;
  const int tile_n = swiglu ? SK_TN / 2 : SK_TN;
  const int n_out = swiglu ? N / 2 : N;
  if (nt == 0) nt = f32 ? (T > 16 ? 32 : 16) : x_mn ? (T > 64 ? 128 : 64) : skinny_nt(T);
  if (f32 && (epi != TPB_EPI_F32 || x_mn || w_mn || tile_expert || nt > 32)) return -2;
  if (x_mn) {
    if (!w_mn || swiglu || tile_expert) return -2;
    if (nt < 64) nt = 64;       // X arrives in blocks of 64 rows
  }
  if (nt < 16 || nt > 128 || nt % 16 || (x_mn && nt % 64)) return -2;
  SkinnyParams p = {};
  p.n1_tiles = 0x7fffffff;
  p.nt = nt; p.stages = skinny_stages(nt); p.stage_bytes = skinny_stage(nt);
  p.T = T; p.N = n_out; p.K = K;
  p.C = c; p.ldc = ldc;
  p.aux = reinterpret_cast<const __nv_bfloat16*>(aux); p.ldaux = ldaux;
  p.c2 = reinterpret_cast<__nv_bfloat16*>(c2); p.ldc2 = ldc2;
  p.up_off = two_w ? 0 : N / 2;
  p.alpha = alpha; p.alpha_dev = alpha_dev; p.epi = epi;
  p.t_tiles = (T + nt - 1) / nt;
  p.num_kb = (K + SK_BK - 1) / SK_BK;
  p.tile_expert = tile_expert;
  p.status = status_block();
  const long long n_tiles = (n_out + tile_n - 1) / tile_n;
  const long long tiles = n_tiles * p.t_tiles;
  // grouped: about one token tile runs per expert that is hit
  if (splits == 0) splits = skinny_splits(tile_expert ? n_tiles * experts_hit : tiles, p.num_kb);
  if (splits != 1 && splits != 2 && splits != 4 && splits != 8) return -2;
  p.splits = splits;
  p.kb_per = (p.num_kb + splits - 1) / splits;
  if (tiles * splits > 0x7fffffffLL) return -2;
  CUtensorMap tw, tw2, tx;
  const uint64_t stride = experts > 1 ? (uint64_t)w_stride : (uint64_t)ldw * (w_mn ? K : extent);
  auto make_w = [&](CUtensorMap* m, const void* ptr) {
    return !w_mn ? make_tmap_3d(m, ptr, K, extent, experts, ldw, stride, 64, 64)
                 : make_tmap_3d(m, ptr, extent, K, experts, ldw, stride, 64, 64);
  };
  if (!x_mn ? make_tmap_2d(&tx, x, K, T, ldx, 64, nt, 2) : make_tmap_2d(&tx, x, T, K, ldx, 64, 64, 2)) return -3;
  if (make_w(&tw, w)) return -4;
  if (two_w) {
    if (make_w(&tw2, w2)) return -5;
  } else {
    tw2 = tw;
  }
  const int grid = (int)(tiles * splits);
  cudaError_t e;
#define TPB_SK(NT_) (w_mn ? launch_skinny<NT_, true>(tw, tw2, tx, p, grid, stream) \
                          : launch_skinny<NT_, false>(tw, tw2, tx, p, grid, stream))
  if (f32)
    e = nt == 16 ? launch_skinny<16, false, false, true>(tw, tw2, tx, p, grid, stream)
                 : launch_skinny<32, false, false, true>(tw, tw2, tx, p, grid, stream);
  else if (x_mn)
    e = nt == 64 ? launch_skinny<64, true, true>(tw, tw2, tx, p, grid, stream)
                 : launch_skinny<128, true, true>(tw, tw2, tx, p, grid, stream);
  else
    e = nt <= 16 ? TPB_SK(16) : nt <= 32 ? TPB_SK(32) : nt <= 64 ? TPB_SK(64) : TPB_SK(128);
#undef TPB_SK
  return e == cudaSuccess ? 0 : 1000 + (int)e;
}

}  // namespace tpb

using namespace tpb;

// y1 = x w1^T and y2 = x w2^T, x [T,K], all rows back to back, in one launch (a decode step's query and latent projections: six of
// its microseconds are a second launch).  -2 where one of the two is not this kernel's by the rules above.
extern "C" int tpb_linear_pair_pays(int T, int N1, int N2, int K) {
  return T > 0 && N1 > 0 && N2 > 0 && K > 0 && K % 8 == 0 && N1 % 8 == 0 && N2 % 8 == 0 && skinny_wins(T, N1, K, false) &&
         skinny_wins(T, N2, K, false);
}
extern "C" int tpb_linear_pair_bf16(const void* x, const void* w1, const void* w2, void* y1, void* y2, int T, int N1, int N2, int K,
                                    void* stream) {
  if (!tpb_linear_pair_pays(T, N1, N2, K)) return -2;
  for (const void* q : {x, w1, w2, (const void*)y1, (const void*)y2})
    if (reinterpret_cast<uintptr_t>(q) % 16) return -2;
  SkinnyParams p = {};
  p.T = T; p.N = N1; p.K = K; p.C = y1; p.ldc = N1;
  p.n1_tiles = (N1 + SK_TN - 1) / SK_TN; p.N2 = N2; p.C2 = y2; p.ldC2 = N2;
  p.alpha = 1.f; p.epi = TPB_EPI_BF16;
  const int nt = skinny_nt(T);
  p.nt = nt; p.stages = skinny_stages(nt); p.stage_bytes = skinny_stage(nt);
  p.t_tiles = (T + nt - 1) / nt;
  p.num_kb = (K + SK_BK - 1) / SK_BK;
  p.status = status_block();
  const long long tiles = ((long long)p.n1_tiles + (N2 + SK_TN - 1) / SK_TN) * p.t_tiles;
  p.splits = skinny_splits(tiles, p.num_kb);
  p.kb_per = (p.num_kb + p.splits - 1) / p.splits;
  if (tiles * p.splits > 0x7fffffffLL) return -2;
  CUtensorMap t1, t2, tx;
  if (make_tmap_2d(&tx, x, K, T, K, 64, nt, 2)) return -3;
  if (make_tmap_3d(&t1, w1, K, N1, 1, K, (uint64_t)K * N1, 64, 64)) return -4;
  if (make_tmap_3d(&t2, w2, K, N2, 1, K, (uint64_t)K * N2, 64, 64)) return -5;
  const int grid = (int)(tiles * p.splits);
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const cudaError_t e = nt <= 16   ? launch_skinny<16, false>(t1, t2, tx, p, grid, st)
                        : nt <= 32 ? launch_skinny<32, false>(t1, t2, tx, p, grid, st)
                        : nt <= 64 ? launch_skinny<64, false>(t1, t2, tx, p, grid, st)
                                   : launch_skinny<128, false>(t1, t2, tx, p, grid, st);
  return e == cudaSuccess ? 0 : 1000 + (int)e;
}

// y = x w^T of bf16 operands in fp32: x [T,K], w [N,K], y [T,N].
extern "C" int tpb_linear_f32(const void* x, const void* w, float* y, int T, int N, int K, long long ldx, long long ldw,
                              long long ldy, void* stream) {
  return skinny_gemm(x, w, nullptr, y, T, N, K, 1, ldx, ldw, 0, ldy, 0, 0, TPB_EPI_F32, 1.0f, nullptr, 0, nullptr, 0, nullptr,
                     0, 0, 0, reinterpret_cast<cudaStream_t>(stream), true, nullptr);
}

// The kernel with an explicit token-tile width and K split (0: by rule); see tpb_gemm_bf16 for the rest.
extern "C" int tpb_gemm_skinny_bf16(const void* x, const void* w, const void* w2, void* c, int T, int N, int K,
                                    long long ldx, long long ldw, long long ldc, int x_mn, int w_mn, int epi, float alpha,
                                    const void* aux, long long ldaux, void* c2, long long ldc2, int nt, int splits,
                                    void* stream) {
  return skinny_gemm(x, w, w2, c, T, N, K, 1, ldx, ldw, 0, ldc, x_mn, w_mn, epi, alpha, aux, ldaux, c2, ldc2, nullptr, 0, nt,
                     splits, reinterpret_cast<cudaStream_t>(stream), false, nullptr);
}

// Rows grouped by expert in segments padded to `nt` rows (16 or 32); tile_expert[rows / nt].  Token tiles of expert -1
// are not written.  experts_hit: how many experts have rows, at most.
extern "C" int tpb_grouped_gemm_skinny_bf16(const void* x, const void* w, const void* w2, void* c, int rows, int N,
                                            int K, int E, long long ldx, long long ldw, long long w_stride,
                                            long long ldc, int w_mn, int epi, const int* tile_expert, int experts_hit,
                                            int nt, void* stream) {
  if (!tile_expert || E < 1 || experts_hit < 1 || (nt != 16 && nt != 32)) return -2;
  return skinny_gemm(x, w, w2, c, rows, N, K, E, ldx, ldw, w_stride, ldc, 0, w_mn, epi, 1.0f, nullptr, 0, nullptr, 0,
                     tile_expert, experts_hit, nt, 0, reinterpret_cast<cudaStream_t>(stream), false, nullptr);
}
