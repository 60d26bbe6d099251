// Flash-attention backward for sm_100a (tcgen05 + TMEM + TMA), GQA-native, head dim 128.
//
// Two tensor-core kernels working on 128 x 128 score tiles; neither needs atomics or a
// cross-CTA reduction.  Every MMA is 128 x 128 x 16, the smallest shape that runs at the full
// tensor rate with operands in shared memory (a 128 x 64 MMA is bound by operand fetch).
//
//  attn_bwd_dkv_kernel   one CTA per (128-key block, kv head, batch).  K and V of the block
//      stay in shared memory; dK and dV accumulate in TMEM over every 128-row query tile and
//      every query head of the GQA group that can see the block.  Transposed frame (TMEM lane
//      = key row); TMEM: dK [0,128), dV [128,256), S^T [256,384), dP^T [384,512).
//        S^T  = K Q^T  (SS)              dP^T = V dO^T  (SS)
//        P^T  = exp2(S^T*c - lse)        bf16, written over S^T      (compute phase 1)
//        dS^T = P^T o (dP^T - delta)     bf16, written over dP^T     (compute phase 2)
//        dV  += P^T dO (TS)              dK  += dS^T Q (TS; scale applied in the epilogue)
//      Tensor stream per step i:  dV(i), S^T(i+1), dK(i), dP^T(i+1): phase 1 of step i+1
//      overlaps dK(i) and dP^T(i+1), phase 2 overlaps dV(i+1) and S^T(i+2).
//
//  attn_bwd_dq_kernel    one CTA per (128-row query tile, query head, batch); TMEM lane =
//      query row; TMEM: dQ [0,128), S double buffered [128,384), dP [384,512).
//        S  = Q K^T (SS)    dP = dO V^T (SS)    dS = exp2(S*c - lse) o (dP - delta)  over dP
//        dQ += dS K (TS, B = K tile MN-major; scale applied in the epilogue)
//      Tensor stream per step j:  S(j+1), dQ(j), dP(j+1).
//
// Both kernels: warp 0 TMA producer, warp 1 MMA issuer, warps 2-9 compute.  Warps w and w+4
// share a TMEM lane quarter and take every other 32 of the 128 score columns of a step; each writes its bf16
// result over the first half of its OWN 32 input columns, so the two never touch each other's
// columns and the A operand of the following MMA is addressed per 16-column k-step.  That result is handed over in two
// halves, columns 0..63 first, so that its product starts while the second one is being made and sums in their order.
//
// Bound by the products themselves and the cap on power: a 128 x 128 step's MMAs are 2048 clocks in the dK/dV kernel and 1536 in
// the dQ kernel, at 1.4 GHz under the cap.  What the dK/dV kernel waits for is its first phase (1250 clocks
// between S^T and P^T).  us through autograd, before the issuing warps stayed together, the halves, the exchange of Q's and dO's
// places and the list of visible tiles / now: one row of 8192 tokens, 32/8 heads, 1710 to 1800 / 1430 to 1510, of 4096 505 / 473; two
// rows of 1999 tokens 296 / 284, in segments 204 / 165 to 190.

#include "common.cuh"
#include "tpb.h"

namespace tpb {

int make_tmap_3d(CUtensorMap* map, const void* ptr, uint64_t d0, uint64_t d1, uint64_t d2, uint64_t stride1_elems,
                 uint64_t stride2_elems, uint32_t box0, uint32_t box1);
int sm_count();

constexpr int BWD_D = 128;
constexpr int BWD_T = 128;         // score tile edge (rows and columns) in both kernels
constexpr int BWD_THREADS = 320;   // TMA warp, MMA warp, 8 compute warps
constexpr int TILE_BYTES = BWD_T * BWD_D * 2;   // one 128 x 128 bf16 operand tile: 32 KB
constexpr int KV_AUX = 4;          // dK/dV kernel: steps whose lse2 and delta rows are in shared memory
constexpr int KV_MAX_TILES = 512;  // query tiles whose list fits in shared memory
constexpr int DQ_KSTAGES = 3;      // dQ kernel: K tile ring (a K tile is held from S(j) to dQ(j))
constexpr int DQ_VSTAGES = 2;      // dQ kernel: V tile ring
constexpr float kLog2e = 1.4426950408889634f;
constexpr int SEG_BLK = 64;        // tokens per entry of the segment-range tables

// Segment-id range of the 128-token tile `t` of batch row `b` from the table of 64-token ranges.
__device__ __forceinline__ int2 seg_range128(const int2* rng, int b, int t, int S) {
  const int2* r = rng + (long long)b * ((S + SEG_BLK - 1) / SEG_BLK) + t * (BWD_T / SEG_BLK);
  int2 a = r[0];
  if (t * BWD_T + SEG_BLK < S) {
    const int2 c = r[1];
    a.x = min(a.x, c.x); a.y = max(a.y, c.y);
  }
  return a;
}

struct AttnBwdParams {
  int B, Sq, Sk, Hq, Hkv;
  float scale, scale_log2;
  float softcap_in;     // logit soft cap: scores become cap * tanh(q.k * scale / cap); this is scale / cap (0: off),
                        // and scale_log2 is then cap * log2(e)
  int causal, window;
  const int* q_pos;
  const int* q_seg;
  const int* kv_seg;
  const int2* q_rng;    // smallest and largest segment id of every 64 queries / keys, or null
  const int2* kv_rng;   // (attn_seg_ranges_kernel of the forward)
  const float* lse2;    // [B,Hq,Sq_pad] log-sum-exp in log2 units, +inf in the padding rows
  const float* delta;   // [B,Hq,Sq_pad] rowsum(dO o O), 0 in the padding rows
  float* delta_out;     // the same, for the kernel that replaces it (attn_bwd_dq192_kernel<true>)
  int Sq_pad;           // Sq rounded up to 128
  int aux_bulk;         // q_pos / q_seg rows can be bulk-copied (16-byte aligned for every tile)
  __nv_bfloat16* dQ; long long lddq;
  __nv_bfloat16* dK; long long lddk;
  __nv_bfloat16* dV; long long lddv;
  int* status;
};

namespace dkv {
constexpr int OFF_K = 0;
constexpr int OFF_V = OFF_K + TILE_BYTES;
constexpr int OFF_QDO = OFF_V + TILE_BYTES;                  // four tiles, see q_slot()
constexpr int OFF_AUX = OFF_QDO + 4 * TILE_BYTES;            // per step: lse2[128], delta[128], qpos[128], qseg[128]
constexpr int AUX_STAGE = 4 * BWD_T * 4;
constexpr int OFF_LIST = OFF_AUX + KV_AUX * AUX_STAGE;       // ushort: the visible tiles in order, kMasked set where scores need a mask
constexpr int OFF_FLAGS = OFF_LIST + 2 * KV_MAX_TILES;       // uchar per tile: 0 not visible, 1 visible, 2 with a mask
constexpr int OFF_BAR = OFF_FLAGS + KV_MAX_TILES;
// Of a step's two tiles dO is done with first (after dV) and Q last (after dK), and the next step but one needs Q first.  So that
// step's Q goes where this one's dO was and its dO where this one's Q was: both are asked for two products earlier than they
// are needed at least.  (A ring of two each asked for Q one product before: 400 of a step's 2970 clocks were spent on its arrival.)
__device__ __forceinline__ uint32_t q_slot(int i) { return OFF_QDO + (2 * (i & 1) + ((i >> 1) & 1)) * TILE_BYTES; }
__device__ __forceinline__ uint32_t do_slot(int i) { return OFF_QDO + (2 * (i & 1) + (((i >> 1) & 1) ^ 1)) * TILE_BYTES; }
constexpr int TOTAL = OFF_BAR + 256 + 1024;
static_assert(TOTAL <= 227 * 1024, "shared memory of one CTA");
constexpr int T_DK = 0, T_DV = 128, T_S = 256, T_DP = 384;
}  // namespace dkv

namespace dqk {
constexpr int OFF_Q = 0;
constexpr int OFF_DO = OFF_Q + TILE_BYTES;
constexpr int OFF_K = OFF_DO + TILE_BYTES;
constexpr int OFF_V = OFF_K + DQ_KSTAGES * TILE_BYTES;
constexpr int OFF_BAR = OFF_V + DQ_VSTAGES * TILE_BYTES;
constexpr int TOTAL = OFF_BAR + 256 + 1024;
constexpr int T_DQ = 0, T_S = 128, T_DP = 384;
}  // namespace dqk

// delta[b,h,q] = sum_d dO * O and lse2[b,h,q] = lse * log2(e), both with row pitch Sq_pad; the
// padding rows get delta = 0 and lse2 = +inf so that they produce P = 0 without a branch.
// (dO, O: [B*Sq, Hq, 128] contiguous; lse: [B,Hq,Sq])
// Bound by reading dO and O.  A block takes 32 tokens x 4 heads: sixteen lanes per (token, head) row of 128
// values, eight rows per lane group in flight, results through shared memory so that every head's 32 values leave
// as one line.  (A grid-stride loop over rows spent its time on 64-bit divisions and on 4-byte stores to a line each.
// 8192 tokens x 32 heads: 42 -> 33 us; 2 x 1999 tokens: 20.5 -> 13.)
constexpr int DELTA_T = 32, DELTA_H = 4, DELTA_THREADS = 256;
__global__ void __launch_bounds__(DELTA_THREADS)
attn_bwd_delta_kernel(const __nv_bfloat16* __restrict__ dO, const __nv_bfloat16* __restrict__ O,
                      const float* __restrict__ lse, float* __restrict__ lse2, float* __restrict__ delta, int Sq,
                      int Sq_pad, int Hq) {
  if (!chain_begin()) return;
  constexpr int ROWS = DELTA_T * DELTA_H / (DELTA_THREADS / 16);   // rows per group of sixteen lanes
  __shared__ float sums[DELTA_H][DELTA_T];
  const int q_tiles = Sq_pad / DELTA_T, h_tiles = (Hq + DELTA_H - 1) / DELTA_H;
  const int bh = blockIdx.x / q_tiles;
  const int q0 = (blockIdx.x - bh * q_tiles) * DELTA_T;
  const int b = bh / h_tiles, h0 = (bh - b * h_tiles) * DELTA_H;
  const int grp = threadIdx.x >> 4, sub = threadIdx.x & 15;
  uint4 a[ROWS], c[ROWS];
#pragma unroll
  for (int i = 0; i < ROWS; ++i) {
    const int r = grp + i * (DELTA_THREADS / 16), q = q0 + r / DELTA_H, h = h0 + r % DELTA_H;
    const bool in = q < Sq && h < Hq;
    const long long at = (((long long)b * Sq + q) * Hq + h) * BWD_D;
    a[i] = in ? __ldg(reinterpret_cast<const uint4*>(dO + at) + sub) : make_uint4(0, 0, 0, 0);
    c[i] = in ? __ldg(reinterpret_cast<const uint4*>(O + at) + sub) : make_uint4(0, 0, 0, 0);
  }
#pragma unroll
  for (int i = 0; i < ROWS; ++i) {
    const float2 a0 = unpack_bf16(a[i].x), a1 = unpack_bf16(a[i].y), a2 = unpack_bf16(a[i].z), a3 = unpack_bf16(a[i].w);
    const float2 c0 = unpack_bf16(c[i].x), c1 = unpack_bf16(c[i].y), c2 = unpack_bf16(c[i].z), c3 = unpack_bf16(c[i].w);
    float s = (a0.x * c0.x + a0.y * c0.y + a1.x * c1.x + a1.y * c1.y) +
              (a2.x * c2.x + a2.y * c2.y + a3.x * c3.x + a3.y * c3.y);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    const int r = grp + i * (DELTA_THREADS / 16);
    if (sub == 0) sums[r % DELTA_H][r / DELTA_H] = s;
  }
  __syncthreads();
  const int idx = threadIdx.x & (DELTA_T * DELTA_H - 1), q = q0 + idx % DELTA_T, h = h0 + idx / DELTA_T;
  if (h < Hq) {
    const long long row = (long long)b * Hq + h;
    if (threadIdx.x < DELTA_T * DELTA_H) delta[row * Sq_pad + q] = sums[idx / DELTA_T][idx % DELTA_T];
    else lse2[row * Sq_pad + q] = q < Sq ? lse[row * Sq + q] * kLog2e : INFINITY;
  }
}
static_assert(DELTA_THREADS == 2 * DELTA_T * DELTA_H, "half of the threads write delta, half lse2");

__device__ __forceinline__ void bulk_load(void* smem_dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(smem_dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

// Writes one fp32 TMEM accumulator row slice (64 columns starting at `col0`) times `mul` as bf16.
__device__ __forceinline__ void store_acc_row(uint32_t tsrc, int col0, __nv_bfloat16* dst, bool have, bool write,
                                              float mul) {
#pragma unroll 1
  for (int c = 0; c < 2; ++c) {
    uint32_t o[32];
    if (have) {
      tmem_ld32(tsrc + col0 + c * 32, o);
      tmem_wait_ld();
    } else {
#pragma unroll
      for (int e = 0; e < 32; ++e) o[e] = 0;
    }
    if (write) {
#pragma unroll
      for (int v = 0; v < 4; ++v)
        *reinterpret_cast<uint4*>(dst + col0 + c * 32 + v * 8) = make_uint4(
            pack_bf16(__uint_as_float(o[8 * v]) * mul, __uint_as_float(o[8 * v + 1]) * mul),
            pack_bf16(__uint_as_float(o[8 * v + 2]) * mul, __uint_as_float(o[8 * v + 3]) * mul),
            pack_bf16(__uint_as_float(o[8 * v + 4]) * mul, __uint_as_float(o[8 * v + 5]) * mul),
            pack_bf16(__uint_as_float(o[8 * v + 6]) * mul, __uint_as_float(o[8 * v + 7]) * mul));
    }
  }
}

// Elementwise product of two packed bf16 pairs (one HMUL2.BF16).
__device__ __forceinline__ uint32_t mul_bf16x2(uint32_t a, uint32_t b) {
  const __nv_bfloat162 r = __hmul2(*reinterpret_cast<const __nv_bfloat162*>(&a), *reinterpret_cast<const __nv_bfloat162*>(&b));
  return *reinterpret_cast<const uint32_t*>(&r);
}

__device__ __forceinline__ uint32_t pack_pair(f32x2 v) {
  float a, b;
  f2_unpack(v, a, b);
  return pack_bf16(a, b);
}
// 2^v as packed bf16.  A step's 128 x 128 exponentials take the MUFU 1024 clocks, half of what the step's MMAs take the tensor core,
// and stand in the chain between them.  (A fourth of them as a polynomial on the FMA pipe gives 3 % of the backward of 8192 tokens,
// but has 2^-126 where this has 0, makes infinity of a NaN and is ten times as far off.)
__device__ __forceinline__ uint32_t exp2_pair(f32x2 v) {
  float a, b;
  f2_unpack(v, a, b);
  return pack_bf16(ex2_approx(a), ex2_approx(b));
}

// Operand tiles are [128 rows][128 d] in two 64-wide d blocks.  Descriptor low words (the high
// word kDescHi is common): K-major use, k-step k covers 16 d; MN-major use (N = d contiguous,
// K = rows), k-step k covers 16 rows.  The k-dependent part is a compile-time constant.
constexpr uint32_t kDescHi = smem_desc_hi(1024);
__device__ __forceinline__ uint32_t kmajor_lo(uint32_t tile) { return smem_desc_lo(tile, 16); }
__device__ __forceinline__ uint32_t mnmajor_lo(uint32_t tile) { return smem_desc_lo(tile, BWD_T * 128); }
__device__ __forceinline__ constexpr uint32_t kmajor_k(int k) { return (uint32_t)(((k >> 2) * (BWD_T * 128) + (k & 3) * 32) >> 4); }
__device__ __forceinline__ constexpr uint32_t mnmajor_k(int k) { return (uint32_t)((k * 2048) >> 4); }
// TMEM column (relative to the tile) where the bf16 A operand of k-step k lives: compute half
// k >> 2 packed its 64 results into the first 32 columns of its own 64-column range; or, a_col32, the one of every other
// 32 columns its 32 results into the first 16 of them.
__device__ __forceinline__ uint32_t a_col(int k) { return (uint32_t)((k >> 2) * 64 + (k & 3) * 8); }
__device__ __forceinline__ uint32_t a_col32(int k) { return (uint32_t)((k >> 1) * 32 + (k & 1) * 8); }

// The query tiles of QT rows that key block kb of batch row b can see, in order, kMasked set where scores need a mask; from
// the positions (and segments) of each one's rows.  All threads of the block call; the caller synchronises behind it.
constexpr uint32_t kMasked = 0x8000;
template <int QT>
__device__ __forceinline__ void list_visible_tiles(const AttnBwdParams& p, bool seg, int b, int kb, int n_tiles, uint8_t* flags,
                                                   uint16_t* list, int* n_list) {
  const int kv0 = kb * BWD_T, pos_off = p.Sk - p.Sq, lane = threadIdx.x & 31;
  const int2 kseg_rng = seg ? seg_range128(p.kv_rng, b, kb, p.Sk) : make_int2(0, 0);
  for (int t = threadIdx.x; t < n_tiles; t += BWD_THREADS) {
    const int r0 = t * QT, r1 = min(p.Sq, r0 + QT);
    int mn = 0x7fffffff, mx = -0x7fffffff;
    if (p.q_pos) {
      for (int r = r0; r < r1; ++r) {
        const int v = p.q_pos[(long long)b * p.Sq + r];
        mn = min(mn, v); mx = max(mx, v);
      }
    } else {
      mn = r0 + pos_off; mx = r1 - 1 + pos_off;
    }
    bool vis = !(p.causal && mx < kv0) && !(p.window > 0 && mn - (kv0 + BWD_T - 1) >= p.window), one_seg = false;
    if (seg) {
      const int2 qr = QT == SEG_BLK ? p.q_rng[(long long)b * n_tiles + t] : seg_range128(p.q_rng, b, t, p.Sq);
      one_seg = qr.x == qr.y && kseg_rng.x == kseg_rng.y && qr.x == kseg_rng.x;
      if (qr.y < kseg_rng.x || qr.x > kseg_rng.y) vis = false;   // no segment in common
    }
    const bool mask = (kv0 + BWD_T > p.Sk) || (p.causal && mn < kv0 + BWD_T - 1) || (p.window > 0 && mx - kv0 >= p.window) ||
                      (p.q_seg != nullptr && !one_seg);
    flags[t] = vis ? (mask ? 2 : 1) : 0;
  }
  __syncthreads();
  if (threadIdx.x >= 32) return;
  int n = 0;
  for (int t0 = 0; t0 < n_tiles; t0 += 32) {
    const int f = t0 + lane < n_tiles ? flags[t0 + lane] : 0;
    const uint32_t seen = __ballot_sync(0xffffffffu, f != 0);
    if (f) list[n + __popc(seen & ((1u << lane) - 1))] = (uint16_t)((t0 + lane) | (f == 2 ? kMasked : 0u));
    n += __popc(seen);
  }
  if (lane == 0) *n_list = n;
}

// ------------------------------------------------------------------------------------------
// dK / dV
// ------------------------------------------------------------------------------------------
// SEG: segment ids come with their range tables.
template <bool SOFTCAP, bool SEG>
__global__ void __launch_bounds__(BWD_THREADS, 1)
attn_bwd_dkv_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                    const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmdO,
                    const AttnBwdParams p) {
  using namespace dkv;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + OFF_BAR);
  uint64_t* k_full = bars;
  uint64_t* q_full = bars + 1;                    // [2] by step parity
  uint64_t* q_empty = q_full + 2;
  uint64_t* do_full = q_empty + 2;
  uint64_t* do_empty = do_full + 2;
  uint64_t* s_full = do_empty + 2;                // S^T of a step is in TMEM
  uint64_t* p_full = s_full + 1;                  // [2] one arrival per compute warp: each half of its share of P^T written
  uint64_t* dp_full = s_full + 3;
  uint64_t* ds_full = s_full + 4;                 // dS^T written
  uint64_t* acc_done = s_full + 5;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(s_full + 6);
  int* n_list = reinterpret_cast<int*>(s_full + 7);
  uint16_t* list = reinterpret_cast<uint16_t*>(smem + OFF_LIST);
  uint8_t* flags = smem + OFF_FLAGS;

  const int warp = warp_index(), lane = threadIdx.x & 31;
  // linear block id is key-block major so that under a causal mask the blocks with the most
  // visible query tiles (lowest key index) are scheduled first on every head
  const int kb = blockIdx.x / (p.Hkv * p.B);
  const int hkv = (blockIdx.x / p.B) % p.Hkv, b = blockIdx.x % p.B;
  const int G = p.Hq / p.Hkv;
  const int kv0 = kb * BWD_T;
  const int pos_off = p.Sk - p.Sq;
  const int n_tiles = (p.Sq + BWD_T - 1) / BWD_T;   // host guarantees <= KV_MAX_TILES

  if (threadIdx.x == 0) {
    mbar_init(k_full, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&q_full[i], 1); mbar_init(&q_empty[i], 1);
      mbar_init(&do_full[i], 1); mbar_init(&do_empty[i], 1);
    }
    mbar_init(s_full, 1); mbar_init(dp_full, 1); mbar_init(ds_full, 8);
    for (int i = 0; i < 2; ++i) mbar_init(&p_full[i], 8);
    mbar_init(acc_done, 1);
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  if (!chain_wait()) return;
  // K is on its way while the query tiles that can see it are found
  if (warp == 0) {
    __syncwarp();   // thread 0's barriers, for whichever lane issues the copy (the others see them behind the list)
    one_lane([&] {
      tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmK); tma_prefetch_desc(&tmV); tma_prefetch_desc(&tmdO);
      mbar_expect_tx(k_full, TILE_BYTES);
      for (int c = 0; c < BWD_D / 64; ++c)
        tma_load_3d(smem + OFF_K + c * (BWD_T * 128), &tmK, k_full, c * 64, b * p.Sk + kv0, hkv);
    });
  }
  list_visible_tiles<BWD_T>(p, SEG, b, kb, n_tiles, flags, list, n_list);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  chain_launch();
  const int n_vis = *n_list;
  const int n_steps = n_vis * G;

  if (warp == 0) {
    // ------------------------------------------------------------------ producer
    if (n_steps == 0) {
      mbar_wait_warp(k_full, 0, p.status, kTimeoutTmaFull, 22);   // (nothing reads it, but it has to have landed)
    } else {
      const bool aux_rows = p.q_pos != nullptr || p.q_seg != nullptr;
      int step = 0;
      bool ok = true;
      for (int g = 0; g < G && ok; ++g) {
        const int hq = hkv * G + g;
        for (int v = 0; v < n_vis; ++v) {
          const int st = step & 1;
          const uint32_t ph = ((step >> 1) & 1) ^ 1;
          const int q0 = (int)(list[v] & (kMasked - 1)) * BWD_T;
          // Q takes the place of the dO of two steps ago
          if (!mbar_wait_warp(&do_empty[st], ph, p.status, kTimeoutStageFree, 21)) { ok = false; break; }
          float* aux = reinterpret_cast<float*>(smem + OFF_AUX + (step % KV_AUX) * AUX_STAGE);
          int* auxi = reinterpret_cast<int*>(aux);
          if (aux_rows && !p.aux_bulk) {
            // rows that cannot be bulk-copied (unaligned sequence length): plain loads, made
            // visible to the consumers by the release of the arrive below
            for (int c = lane; c < BWD_T; c += 32) {
              const int r = min(q0 + c, p.Sq - 1);
              auxi[2 * BWD_T + c] = p.q_pos ? p.q_pos[(long long)b * p.Sq + r] : 0;
              auxi[3 * BWD_T + c] = p.q_seg ? p.q_seg[(long long)b * p.Sq + r] : 0;
            }
            __syncwarp();
          }
          if (lane == 0) {
            const uint32_t rows_bytes = (uint32_t)min(BWD_T, p.Sq - q0) * 4u;
            uint32_t tx = TILE_BYTES + 2 * BWD_T * 4;
            if (aux_rows && p.aux_bulk) tx += (p.q_pos ? rows_bytes : 0u) + (p.q_seg ? rows_bytes : 0u);
            mbar_expect_tx(&q_full[st], tx);
            for (int c = 0; c < BWD_D / 64; ++c)
              tma_load_3d(smem + q_slot(step) + c * (BWD_T * 128), &tmQ, &q_full[st], c * 64, b * p.Sq + q0, hq);
            const long long li = ((long long)b * p.Hq + hq) * p.Sq_pad + q0;
            bulk_load(aux, p.lse2 + li, BWD_T * 4, &q_full[st]);
            bulk_load(aux + BWD_T, p.delta + li, BWD_T * 4, &q_full[st]);
            if (aux_rows && p.aux_bulk) {
              if (p.q_pos) bulk_load(auxi + 2 * BWD_T, p.q_pos + (long long)b * p.Sq + q0, rows_bytes, &q_full[st]);
              if (p.q_seg) bulk_load(auxi + 3 * BWD_T, p.q_seg + (long long)b * p.Sq + q0, rows_bytes, &q_full[st]);
            }
          }
          __syncwarp();
          // and dO that of its Q
          if (!mbar_wait_warp(&q_empty[st], ph, p.status, kTimeoutStageFree, 29)) { ok = false; break; }
          if (lane == 0) {
            mbar_expect_tx(&do_full[st], step == 0 ? 2 * TILE_BYTES : TILE_BYTES);   // V comes with the first dO
            if (step == 0)
              for (int c = 0; c < BWD_D / 64; ++c)
                tma_load_3d(smem + OFF_V + c * (BWD_T * 128), &tmV, &do_full[0], c * 64, b * p.Sk + kv0, hkv);
            for (int c = 0; c < BWD_D / 64; ++c)
              tma_load_3d(smem + do_slot(step) + c * (BWD_T * 128), &tmdO, &do_full[st], c * 64, b * p.Sq + q0, hq);
          }
          __syncwarp();
          ++step;
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (n_steps > 0) {
      constexpr uint32_t id_s = make_idesc_bf16(BWD_T, BWD_T, false, false);    // S^T, dP^T
      constexpr uint32_t id_acc = make_idesc_bf16(BWD_T, BWD_D, false, true);   // dV, dK (A in TMEM, B MN-major)
      const uint32_t dK = kmajor_lo(smem_u32(smem + OFF_K)), dVd = kmajor_lo(smem_u32(smem + OFF_V));
      const uint32_t base = smem_u32(smem);
      const uint32_t tS = tmem_base + T_S, tDP = tmem_base + T_DP;
      // The MMA queue is shallow, so whatever this thread does between two MMAs is tensor idle
      // time: every wait is therefore placed before the LAST MMA of the preceding group, where
      // its latency hides behind the seven MMAs still in flight.
      auto wait_q = [&](int i) { return mbar_wait_warp(&q_full[i & 1], (i >> 1) & 1, p.status, kTimeoutTmaFull, 23); };
      auto wait_do = [&](int i) { return mbar_wait_warp(&do_full[i & 1], (i >> 1) & 1, p.status, kTimeoutTmaFull, 24); };
      auto wait_p = [&](int i, int part) { return mbar_wait_warp(&p_full[part], i & 1, p.status, kTimeoutSoftmax, 25); };
      auto wait_ds = [&](int i) { return mbar_wait_warp(ds_full, i & 1, p.status, kTimeoutSoftmax, 26); };
      auto group = [&](auto&& mma, auto&& hook, auto&& done) -> bool {
        one_lane([&] {
#pragma unroll
          for (int k = 0; k < 7; ++k) mma(k);
        });
        if (!hook()) return false;
        tc_fence_after();
        one_lane([&] { mma(7); done(); });
        return true;
      };
      bool ok = mbar_wait_warp(k_full, 0, p.status, kTimeoutTmaFull, 22) && wait_q(0);
      tc_fence_after();
      auto issue_s = [&](int i, auto&& hook) -> bool {      // S^T(i) = K Q(i)^T
        const uint32_t dQ = kmajor_lo(base + q_slot(i));
        return group([&](int k) { mma_ss_w(tS, dK + kmajor_k(k), kDescHi, dQ + kmajor_k(k), kDescHi, id_s, k != 0); }, hook,
                     [&] { tc_commit(s_full); });
      };
      auto issue_dp = [&](int i, auto&& hook) -> bool {     // dP^T(i) = V dO(i)^T
        const uint32_t dDO = kmajor_lo(base + do_slot(i));
        return group([&](int k) { mma_ss_w(tDP, dVd + kmajor_k(k), kDescHi, dDO + kmajor_k(k), kDescHi, id_s, k != 0); }, hook,
                     [&] { tc_commit(dp_full); });
      };
      auto none = [] { return true; };
      if (ok) ok = issue_s(0, [&] { return wait_do(0); });
      if (ok) ok = issue_dp(0, none);
      for (int i = 0; i < n_steps && ok; ++i) {
        const uint32_t mQ = mnmajor_lo(base + q_slot(i));
        const uint32_t mDO = mnmajor_lo(base + do_slot(i));
        const bool more = i + 1 < n_steps;
        // Waits on the compute warps stay where the data is needed: hooking them into the previous
        // group would hold back that group's commit, which the compute warps are waiting for.
        // dV += P^T dO, first the k-steps whose P^T is there when the exponentials are half done
        auto dv = [&](int k) { mma_ts_w(tmem_base + T_DV, tS + a_col32(k), mDO + mnmajor_k(k), kDescHi, id_acc, (i | k) != 0); };
        if (!wait_p(i, 0)) break;
        tc_fence_after();
        one_lane([&] { dv(0); dv(1); dv(2); dv(3); });
        if (!wait_p(i, 1)) break;
        tc_fence_after();
        ok = group([&](int k) { if (k >= 4) dv(k); },
                   [&] { return more ? wait_q(i + 1) : true; }, [&] { tc_commit(&do_empty[i & 1]); });
        if (!ok) break;
        if (more && !issue_s(i + 1, none)) break;
        if (!wait_ds(i)) break;
        tc_fence_after();
        // dK += dS^T Q
        ok = group([&](int k) { mma_ts_w(tmem_base + T_DK, tDP + a_col32(k), mQ + mnmajor_k(k), kDescHi, id_acc, (i | k) != 0); },
                   [&] { return more ? wait_do(i + 1) : true; }, [&] { tc_commit(&q_empty[i & 1]); });
        if (!ok) break;
        if (more && !issue_dp(i + 1, none)) break;
      }
      one_lane([&] { tc_commit(acc_done); });
    }
  } else {
    // ------------------------------------------------------------------ compute warps
    // Warp w may touch TMEM lanes 32*(w%4)..+31, so warps w and w+4 share a lane quarter (the
    // same 32 key rows) and split the 128 query columns of a step between them: half * 32 + (0..31) and 64 further on.
    const int qd = warp & 3;
    const int half = (warp - 2) >> 2;
    const int r_local = qd * 32 + lane;           // key row == TMEM lane
    const int kp = kv0 + r_local;                 // key position (keys are in natural order)
    const bool key_ok = kp < p.Sk;
    const int kseg = (p.kv_seg && key_ok) ? p.kv_seg[(long long)b * p.Sk + kp] : 0;
    const uint32_t tb = tmem_base + ((uint32_t)(qd * 32) << 16);
    const uint32_t tS = tb + T_S + half * 32, tDP = tb + T_DP + half * 32;
    const int win = p.window > 0 ? p.window : 0x7fffffff;   // keep needs qp - kp < win
    const int cmax = p.causal ? kp : -0x7fffffff;           // and qp >= cmax
    bool ok = true;

    int step = 0;
    for (int g = 0; g < G && ok; ++g) {
      for (int v = 0; v < n_vis && ok; ++v) {
        const uint32_t entry = list[v];
        const int t = (int)(entry & (kMasked - 1));
        const bool need_mask = (entry & kMasked) != 0;
        const float* aux = reinterpret_cast<const float*>(smem + OFF_AUX + (step % KV_AUX) * AUX_STAGE);
        const int* auxi = reinterpret_cast<const int*>(aux);
        // ---- phase 1: P^T = exp2(S^T * c - lse), kept packed for phase 2 and written over S^T
        if (!mbar_wait(s_full, step & 1, p.status, kTimeoutAccFull, 27)) { ok = false; break; }
        tc_fence_after();
        uint32_t keep0 = 0xffffffffu, keep1 = 0xffffffffu;   // of this half's queries those that may see the key
        if (need_mask) {
          if (p.q_pos) {
            const int4* qp4 = reinterpret_cast<const int4*>(auxi + 2 * BWD_T + half * 32);
            keep0 = keep1 = 0;
#pragma unroll 1
            for (int c4 = 0; c4 < 8; ++c4) {
              const int4 a = qp4[c4], c = qp4[c4 + 16];
              const int qa[4] = {a.x, a.y, a.z, a.w}, qc[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                keep0 |= (uint32_t)((qa[e] >= cmax) & (qa[e] - kp < win)) << (4 * c4 + e);
                keep1 |= (uint32_t)((qc[e] >= cmax) & (qc[e] - kp < win)) << (4 * c4 + e);
              }
            }
          } else {
            const int at = t * BWD_T + pos_off + half * 32;   // position of the first one
            const int hi = kp - at + min(win, 0x40000000) - 1, lo = p.causal ? kp - at - 1 : -1;   // (kp - at < 2^30)
            keep0 = bits_upto(hi) & ~bits_upto(lo);
            keep1 = bits_upto(hi - 64) & ~bits_upto(lo - 64);
          }
          if (p.q_seg || p.kv_seg) {
            const int* qs = auxi + 3 * BWD_T + half * 32;
            same_segment_bits(p.q_seg ? qs[lane] : 0, p.q_seg ? qs[64 + lane] : 0, kseg, keep0, keep1);
          }
          if (!key_ok) keep0 = keep1 = 0;
        }
        uint32_t pk_p[32];
        uint32_t pk_f[SOFTCAP ? 32 : 1];   // 1 - tanh^2 of the capped scores (the derivative of the cap)
        uint32_t sreg[64];
        tmem_ld32(tS, sreg);
        tmem_ld32(tS + 64, sreg + 32);
        tmem_wait_ld();
#pragma unroll
        for (int ch = 0; ch < 2; ++ch) {
          const uint32_t* s = sreg + ch * 32;
          const float4* lse4 = reinterpret_cast<const float4*>(aux + half * 32 + ch * 64);
          if (!need_mask && !SOFTCAP) {
            const f32x2 c2 = f2_pack(p.scale_log2, p.scale_log2);
#pragma unroll
            for (int c4 = 0; c4 < 8; ++c4) {
              const float4 L = lse4[c4];
              pk_p[ch * 16 + 2 * c4] = exp2_pair(f2_fma(f2_pack_bits(s[4 * c4], s[4 * c4 + 1]), c2, f2_pack(-L.x, -L.y)));
              pk_p[ch * 16 + 2 * c4 + 1] = exp2_pair(f2_fma(f2_pack_bits(s[4 * c4 + 2], s[4 * c4 + 3]), c2, f2_pack(-L.z, -L.w)));
            }
          } else if (!need_mask) {
#pragma unroll
            for (int c4 = 0; c4 < 8; ++c4) {
              const float4 L = lse4[c4];
              float sv[4] = {__uint_as_float(s[4 * c4]), __uint_as_float(s[4 * c4 + 1]), __uint_as_float(s[4 * c4 + 2]),
                             __uint_as_float(s[4 * c4 + 3])};
              if (SOFTCAP) {
#pragma unroll
                for (int e = 0; e < 4; ++e) sv[e] = tanh_approx(sv[e] * p.softcap_in);
                pk_f[ch * 16 + 2 * c4] = pack_bf16(1.f - sv[0] * sv[0], 1.f - sv[1] * sv[1]);
                pk_f[ch * 16 + 2 * c4 + 1] = pack_bf16(1.f - sv[2] * sv[2], 1.f - sv[3] * sv[3]);
              }
              const float p0 = exp2f(fmaf(sv[0], p.scale_log2, -L.x));
              const float p1 = exp2f(fmaf(sv[1], p.scale_log2, -L.y));
              const float p2 = exp2f(fmaf(sv[2], p.scale_log2, -L.z));
              const float p3 = exp2f(fmaf(sv[3], p.scale_log2, -L.w));
              pk_p[ch * 16 + 2 * c4] = pack_bf16(p0, p1);
              pk_p[ch * 16 + 2 * c4 + 1] = pack_bf16(p2, p3);
            }
          } else {
            const uint32_t keep = ch ? keep1 : keep0;
#pragma unroll
            for (int c4 = 0; c4 < 8; ++c4) {
              const float4 L = lse4[c4];
              const float l[4] = {L.x, L.y, L.z, L.w};
              float pv[4], fv[4];
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                float sv = __uint_as_float(s[4 * c4 + e]);
                if (SOFTCAP) {
                  sv = tanh_approx(sv * p.softcap_in);
                  fv[e] = 1.f - sv * sv;
                }
                const float pe = exp2f(fmaf(sv, p.scale_log2, -l[e]));
                pv[e] = (keep & (1u << (4 * c4 + e))) ? pe : 0.f;
              }
              if (SOFTCAP) {
                pk_f[ch * 16 + 2 * c4] = pack_bf16(fv[0], fv[1]);
                pk_f[ch * 16 + 2 * c4 + 1] = pack_bf16(fv[2], fv[3]);
              }
              pk_p[ch * 16 + 2 * c4] = pack_bf16(pv[0], pv[1]);
              pk_p[ch * 16 + 2 * c4 + 1] = pack_bf16(pv[2], pv[3]);
            }
          }
          tmem_st16(tS + ch * 64, pk_p + ch * 16);
          tmem_wait_st();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&p_full[ch]);
        }
        if (SOFTCAP) {   // dV takes P^T as it is; dS^T takes P^T times the derivative of the cap
#pragma unroll
          for (int c = 0; c < 32; ++c) pk_p[c] = mul_bf16x2(pk_p[c], pk_f[c]);
        }
        // ---- phase 2: dS^T = P^T o (dP^T - delta), written over dP^T
        if (!mbar_wait(dp_full, step & 1, p.status, kTimeoutAccFull, 28)) { ok = false; break; }
        tc_fence_after();
        {
          uint32_t dreg[64], pk_ds[32];
          tmem_ld32(tDP, dreg);
          tmem_ld32(tDP + 64, dreg + 32);
          tmem_wait_ld();
          const float4* dlt4 = reinterpret_cast<const float4*>(aux + BWD_T + half * 32);
#pragma unroll
          for (int c4 = 0; c4 < 16; ++c4) {
            const float4 Dl = dlt4[c4 + (c4 >> 3) * 8];
            pk_ds[2 * c4] = mul_bf16x2(pk_p[2 * c4], pack_pair(f2_sub(f2_pack_bits(dreg[4 * c4], dreg[4 * c4 + 1]), f2_pack(Dl.x, Dl.y))));
            pk_ds[2 * c4 + 1] =
                mul_bf16x2(pk_p[2 * c4 + 1], pack_pair(f2_sub(f2_pack_bits(dreg[4 * c4 + 2], dreg[4 * c4 + 3]), f2_pack(Dl.z, Dl.w))));
          }
          // all 64 inputs of this warp are in registers, so the first halves of its columns can be overwritten
          tmem_st16(tDP, pk_ds);
          tmem_st16(tDP + 64, pk_ds + 16);
        }
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(ds_full);
        ++step;
      }
    }
    // ---- dK / dV
    if (ok && n_steps > 0) ok = mbar_wait(acc_done, 0, p.status, kTimeoutAccFull, 28);
    tc_fence_after();
    const bool have = ok && n_steps > 0;
    store_acc_row(tb + T_DK, half * 64, p.dK + ((long long)b * p.Sk + kp) * p.lddk + (long long)hkv * BWD_D, have,
                  key_ok, p.scale);
    store_acc_row(tb + T_DV, half * 64, p.dV + ((long long)b * p.Sk + kp) * p.lddv + (long long)hkv * BWD_D, have,
                  key_ok, 1.f);
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// ------------------------------------------------------------------------------------------
// dQ
// ------------------------------------------------------------------------------------------
template <bool SOFTCAP, bool SEG>
__global__ void __launch_bounds__(BWD_THREADS, 1)
attn_bwd_dq_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                   const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmdO,
                   const AttnBwdParams p) {
  using namespace dqk;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + OFF_BAR);
  uint64_t* q_full = bars;
  uint64_t* k_full = bars + 1;                    // [DQ_KSTAGES]
  uint64_t* k_empty = k_full + DQ_KSTAGES;
  uint64_t* v_full = k_empty + DQ_KSTAGES;        // [DQ_VSTAGES]
  uint64_t* v_empty = v_full + DQ_VSTAGES;
  uint64_t* s_full = v_empty + DQ_VSTAGES;        // [2]
  uint64_t* dp_full = s_full + 2;
  uint64_t* ds_full = s_full + 3;                 // [2] one arrival per compute warp: each half of its share of dS written
  uint64_t* acc_done = s_full + 5;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(s_full + 6);
  int* tile_minmax = reinterpret_cast<int*>(s_full + 7);  // [2]
  int* seg_lohi = reinterpret_cast<int*>(s_full + 8);     // [2] first and last key block with a segment of this tile

  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int n_qtiles = (p.Sq + BWD_T - 1) / BWD_T;
  // heaviest (latest) query tiles first under a causal mask
  const int qt = n_qtiles - 1 - (int)(blockIdx.x / (p.Hq * p.B));
  const int hq = (blockIdx.x / p.B) % p.Hq, b = blockIdx.x % p.B;
  const int hkv = hq / (p.Hq / p.Hkv);
  const int q0 = qt * BWD_T;
  const int pos_off = p.Sk - p.Sq;

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int i = 0; i < DQ_KSTAGES; ++i) { mbar_init(&k_full[i], 1); mbar_init(&k_empty[i], 1); }
    for (int i = 0; i < DQ_VSTAGES; ++i) { mbar_init(&v_full[i], 1); mbar_init(&v_empty[i], 1); }
    mbar_init(&s_full[0], 1); mbar_init(&s_full[1], 1);
    mbar_init(dp_full, 1); mbar_init(&ds_full[0], 8); mbar_init(&ds_full[1], 8);
    mbar_init(acc_done, 1);
    tile_minmax[0] = 0x7fffffff;
    tile_minmax[1] = -0x7fffffff;
    if (SEG) { seg_lohi[0] = 0x7fffffff; seg_lohi[1] = -1; }
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  chain_launch();
  if (!chain_wait()) return;

  // Q is on its way while the key blocks that it can see are found
  if (warp == 0) {
    one_lane([&] {
      tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmK); tma_prefetch_desc(&tmV); tma_prefetch_desc(&tmdO);
      mbar_expect_tx(q_full, TILE_BYTES);
#pragma unroll
      for (int c = 0; c < BWD_D / 64; ++c)
        tma_load_3d(smem + OFF_Q + c * (BWD_T * 128), &tmQ, q_full, c * 64, b * p.Sq + q0, hq);
    });
  }
  int qpos_min = q0 + pos_off, qpos_max = min(q0 + BWD_T, p.Sq) - 1 + pos_off;
  if (p.q_pos) {
    if (threadIdx.x < BWD_T && q0 + (int)threadIdx.x < p.Sq) {
      const int qp = p.q_pos[(long long)b * p.Sq + q0 + threadIdx.x];
      atomicMin(&tile_minmax[0], qp);
      atomicMax(&tile_minmax[1], qp);
    }
    __syncthreads();
    qpos_min = tile_minmax[0];
    qpos_max = tile_minmax[1];
  }
  const int nblk_total = (p.Sk + BWD_T - 1) / BWD_T;
  int blk_hi = p.causal ? min(nblk_total, qpos_max / BWD_T + 1) : nblk_total;
  int blk_lo = (p.window > 0 && qpos_min >= p.window) ? (qpos_min - p.window + 1) / BWD_T : 0;
  if (p.causal && qpos_max < 0) blk_hi = 0;
  int2 qr = make_int2(0, 0);
  if (SEG) {   // as in the forward: only the key blocks between the first and last with a common segment
    qr = seg_range128(p.q_rng, b, qt, p.Sq);
    for (int i = blk_lo + (int)threadIdx.x; i < blk_hi; i += BWD_THREADS) {
      const int2 kr = seg_range128(p.kv_rng, b, i, p.Sk);
      if (kr.x <= qr.y && kr.y >= qr.x) {
        atomicMin(&seg_lohi[0], i);
        atomicMax(&seg_lohi[1], i);
      }
    }
    __syncthreads();
    blk_lo = max(blk_lo, seg_lohi[0]);
    blk_hi = min(blk_hi, seg_lohi[1] + 1);
  }
  const int nblk = max(0, blk_hi - blk_lo);

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (nblk == 0) {
      mbar_wait_warp(q_full, 0, p.status, kTimeoutTmaFull, 32);   // (nothing reads it, but it has to have landed)
    } else if (elect_one()) {
      for (int j = 0; j < nblk; ++j) {
        const int sk = j % DQ_KSTAGES, sv = j % DQ_VSTAGES;
        const int row = b * p.Sk + (blk_lo + j) * BWD_T;
        if (!mbar_wait(&k_empty[sk], ((j / DQ_KSTAGES) & 1) ^ 1, p.status, kTimeoutStageFree, 31)) break;
        mbar_expect_tx(&k_full[sk], TILE_BYTES);
#pragma unroll
        for (int c = 0; c < BWD_D / 64; ++c)
          tma_load_3d(smem + OFF_K + sk * TILE_BYTES + c * (BWD_T * 128), &tmK, &k_full[sk], c * 64, row, hkv);
        if (!mbar_wait(&v_empty[sv], ((j / DQ_VSTAGES) & 1) ^ 1, p.status, kTimeoutStageFree, 35)) break;
        mbar_expect_tx(&v_full[sv], j == 0 ? 2 * TILE_BYTES : TILE_BYTES);   // dO comes with the first V
        if (j == 0) {
#pragma unroll
          for (int c = 0; c < BWD_D / 64; ++c)
            tma_load_3d(smem + OFF_DO + c * (BWD_T * 128), &tmdO, &v_full[0], c * 64, b * p.Sq + q0, hq);
        }
#pragma unroll
        for (int c = 0; c < BWD_D / 64; ++c)
          tma_load_3d(smem + OFF_V + sv * TILE_BYTES + c * (BWD_T * 128), &tmV, &v_full[sv], c * 64, row, hkv);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (nblk > 0) {
      constexpr uint32_t id_s = make_idesc_bf16(BWD_T, BWD_T, false, false);    // S, dP
      constexpr uint32_t id_dq = make_idesc_bf16(BWD_T, BWD_D, false, true);    // dQ (A in TMEM, B MN-major)
      const uint32_t dQ = kmajor_lo(smem_u32(smem + OFF_Q)), dDO = kmajor_lo(smem_u32(smem + OFF_DO));
      const uint32_t aK0 = smem_u32(smem + OFF_K), aV0 = smem_u32(smem + OFF_V);
      const uint32_t tDP = tmem_base + T_DP;
      // Waits sit before the last MMA of the preceding group (see the dK/dV kernel).
      auto wait_k = [&](int j) { return mbar_wait_warp(&k_full[j % DQ_KSTAGES], (j / DQ_KSTAGES) & 1, p.status, kTimeoutTmaFull, 33); };
      auto wait_v = [&](int j) { return mbar_wait_warp(&v_full[j % DQ_VSTAGES], (j / DQ_VSTAGES) & 1, p.status, kTimeoutTmaFull, 37); };
      auto wait_ds = [&](int j, int part) { return mbar_wait_warp(&ds_full[part], j & 1, p.status, kTimeoutSoftmax, 34); };
      auto group = [&](auto&& mma, auto&& hook, auto&& done) -> bool {
        one_lane([&] {
#pragma unroll
          for (int k = 0; k < 7; ++k) mma(k);
        });
        if (!hook()) return false;
        tc_fence_after();
        one_lane([&] { mma(7); done(); });
        return true;
      };
      bool ok = mbar_wait_warp(q_full, 0, p.status, kTimeoutTmaFull, 32) && wait_k(0);
      tc_fence_after();
      auto issue_s = [&](int j, auto&& hook) -> bool {      // S(j) = Q K_j^T
        const uint32_t dK = kmajor_lo(aK0 + (j % DQ_KSTAGES) * TILE_BYTES);
        const uint32_t tS = tmem_base + T_S + (j & 1) * BWD_T;
        return group([&](int k) { mma_ss_w(tS, dQ + kmajor_k(k), kDescHi, dK + kmajor_k(k), kDescHi, id_s, k != 0); }, hook,
                     [&] { tc_commit(&s_full[j & 1]); });
      };
      auto issue_dp = [&](int j, auto&& hook) -> bool {     // dP(j) = dO V_j^T
        const uint32_t dV = kmajor_lo(aV0 + (j % DQ_VSTAGES) * TILE_BYTES);
        return group([&](int k) { mma_ss_w(tDP, dDO + kmajor_k(k), kDescHi, dV + kmajor_k(k), kDescHi, id_s, k != 0); }, hook,
                     [&] { tc_commit(&v_empty[j % DQ_VSTAGES]); tc_commit(dp_full); });
      };
      auto none = [] { return true; };
      if (ok) ok = issue_s(0, [&] { return wait_v(0); });
      if (ok) ok = issue_dp(0, [&] { return nblk > 1 ? wait_k(1) : true; });
      for (int j = 0; j < nblk && ok; ++j) {
        const bool more = j + 1 < nblk;
        if (more && !issue_s(j + 1, none)) break;
        const uint32_t mK = mnmajor_lo(aK0 + (j % DQ_KSTAGES) * TILE_BYTES);
        // dQ += dS K   (K tile [128 keys][128 d]: N = d contiguous)
        auto dq = [&](int k) { mma_ts_w(tmem_base + T_DQ, tDP + a_col32(k), mK + mnmajor_k(k), kDescHi, id_dq, (j | k) != 0); };
        if (!wait_ds(j, 0)) break;   // not hooked into S(j+1): that would hold back its commit
        tc_fence_after();
        one_lane([&] { dq(0); dq(1); dq(2); dq(3); });
        if (!wait_ds(j, 1)) break;
        tc_fence_after();
        ok = group([&](int k) { if (k >= 4) dq(k); },
                   [&] { return more ? wait_v(j + 1) : true; }, [&] { tc_commit(&k_empty[j % DQ_KSTAGES]); });
        if (!ok) break;
        if (more && !issue_dp(j + 1, [&] { return j + 2 < nblk ? wait_k(j + 2) : true; })) break;
      }
      one_lane([&] { tc_commit(acc_done); });
    }
  } else {
    // ------------------------------------------------------------------ compute warps
    const int qd = warp & 3;
    const int half = (warp - 2) >> 2;             // which key columns: half * 32 + (0..31) and 64 further on
    const int r_local = qd * 32 + lane;           // query row == TMEM lane
    const int row = q0 + r_local;
    const bool row_ok = row < p.Sq;
    const long long grow = (long long)b * p.Sq + row;
    const int qpos = row_ok ? (p.q_pos ? p.q_pos[grow] : row + pos_off) : -1;
    const int qseg = (p.q_seg && row_ok) ? p.q_seg[grow] : 0;
    const long long li = ((long long)b * p.Hq + hq) * p.Sq_pad + row;   // row < Sq_pad: padded to 128
    const float lse2 = p.lse2[li];
    const float delta = p.delta[li];
    const uint32_t tb = tmem_base + ((uint32_t)(qd * 32) << 16);
    const uint32_t tDP = tb + T_DP + half * 32;
    const int* ks = p.kv_seg ? p.kv_seg + (long long)b * p.Sk : nullptr;
    const int kmin = p.window > 0 && qpos >= p.window ? qpos - p.window : -1;   // keep needs kmin < kp <= kmax
    const int kmax = p.causal ? min(max(qpos, -1), p.Sk - 1) : p.Sk - 1;
    bool ok = true;

    for (int j = 0; j < nblk && ok; ++j) {
      const int kv0 = (blk_lo + j) * BWD_T;
      bool seg_mask = p.q_seg != nullptr;
      if (SEG) {
        const int2 kr = seg_range128(p.kv_rng, b, blk_lo + j, p.Sk);
        seg_mask = !(qr.x == qr.y && kr.x == kr.y && qr.x == kr.x);
      }
      const bool need_mask = (p.causal && kv0 + BWD_T - 1 > qpos_min) || (kv0 + BWD_T > p.Sk) ||
                             (p.window > 0 && qpos_max - kv0 >= p.window) || seg_mask;
      const uint32_t tS = tb + T_S + (j & 1) * BWD_T + half * 32;
      uint32_t keep0 = 0xffffffffu, keep1 = 0xffffffffu;   // of this half's keys those that the row may see
      if (need_mask) {
        const int k0 = kv0 + half * 32, hi = kmax - k0, lo = kmin - k0;
        keep0 = bits_upto(hi) & ~bits_upto(lo);
        keep1 = bits_upto(hi - 64) & ~bits_upto(lo - 64);
        if (ks && (!SEG || seg_mask))
          same_segment_bits(__ldg(ks + min(k0 + lane, p.Sk - 1)), __ldg(ks + min(k0 + 64 + lane, p.Sk - 1)), qseg, keep0, keep1);
      }
      // ---- phase 1: P = exp2(S * c - lse), packed bf16 in registers
      if (!mbar_wait(&s_full[j & 1], (j >> 1) & 1, p.status, kTimeoutAccFull, 36)) { ok = false; break; }
      tc_fence_after();
      uint32_t pk_p[32];
      uint32_t sreg[64];
      tmem_ld32(tS, sreg);
      tmem_ld32(tS + 64, sreg + 32);
      tmem_wait_ld();
#pragma unroll
      for (int ch = 0; ch < 2; ++ch) {
        const uint32_t* s = sreg + ch * 32;
        if (!need_mask && !SOFTCAP) {
          const f32x2 c2 = f2_pack(p.scale_log2, p.scale_log2), nl2 = f2_pack(-lse2, -lse2);
#pragma unroll
          for (int c = 0; c < 16; ++c)
            pk_p[ch * 16 + c] = exp2_pair(f2_fma(f2_pack_bits(s[2 * c], s[2 * c + 1]), c2, nl2));
        } else if (!need_mask) {
#pragma unroll
          for (int c = 0; c < 32; c += 2) {
            float s0 = __uint_as_float(s[c]), s1 = __uint_as_float(s[c + 1]), f0 = 1.f, f1 = 1.f;
            if (SOFTCAP) {   // P only feeds dS here, so the derivative of the cap is folded into it
              s0 = tanh_approx(s0 * p.softcap_in);
              s1 = tanh_approx(s1 * p.softcap_in);
              f0 = 1.f - s0 * s0;
              f1 = 1.f - s1 * s1;
            }
            pk_p[ch * 16 + c / 2] = pack_bf16(f0 * exp2f(fmaf(s0, p.scale_log2, -lse2)),
                                              f1 * exp2f(fmaf(s1, p.scale_log2, -lse2)));
          }
        } else {
          const uint32_t keep = ch ? keep1 : keep0;
#pragma unroll
          for (int c = 0; c < 32; c += 2) {
            float pv[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              float sv = __uint_as_float(s[c + e]), fv = 1.f;
              if (SOFTCAP) {
                sv = tanh_approx(sv * p.softcap_in);
                fv = 1.f - sv * sv;
              }
              const float pe = fv * exp2f(fmaf(sv, p.scale_log2, -lse2));
              pv[e] = (keep & (1u << (c + e))) ? pe : 0.f;
            }
            pk_p[ch * 16 + c / 2] = pack_bf16(pv[0], pv[1]);
          }
        }
      }
      // ---- phase 2: dS = P o (dP - delta), written over dP
      if (!mbar_wait(dp_full, j & 1, p.status, kTimeoutAccFull, 39)) { ok = false; break; }
      tc_fence_after();
      {
        uint32_t dreg[64], pk[16];
        tmem_ld32(tDP, dreg);
        tmem_ld32(tDP + 64, dreg + 32);
        tmem_wait_ld();
        const f32x2 d2 = f2_pack(delta, delta);
#pragma unroll
        for (int ch = 0; ch < 2; ++ch) {
#pragma unroll
          for (int c = 0; c < 16; ++c)
            pk[c] = mul_bf16x2(pk_p[ch * 16 + c], pack_pair(f2_sub(f2_pack_bits(dreg[32 * ch + 2 * c], dreg[32 * ch + 2 * c + 1]), d2)));
          tmem_st16(tDP + ch * 64, pk);
          tmem_wait_st();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&ds_full[ch]);
        }
      }
    }
    if (ok && nblk > 0) ok = mbar_wait(acc_done, 0, p.status, kTimeoutAccFull, 38);
    tc_fence_after();
    store_acc_row(tb + T_DQ, half * 64, p.dQ + grow * p.lddq + (long long)hq * BWD_D, ok && nblk > 0, row_ok,
                  p.scale);
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// ------------------------------------------------------------------------------------------
// Query / key head dim 192 with value dim 128 (latent attention).
//
// The same two kernels with the tiles that 512 TMEM columns and 227 KB of shared memory leave room for:
//   dK/dV: dK takes 192 columns and dV 128, so score tiles are 128 keys x 64 queries; S^T is double
//          buffered and the score product of step i + 1 runs beside both compute phases of step i.
//          TMEM: dK [0,192), dV [192,320), S^T [320,448), dP^T [448,512).
//          (A 128 x 64 MMA is bound by operand fetch at 2/3 of the tensor rate; with 128 x 128 tiles the
//          accumulators and two score tiles would need 576 columns.)
//   dQ:    128 x 128 tiles, one S buffer: S(j + 1) is issued as soon as the compute warps hold S(j) in
//          registers.  TMEM: dQ [0,192), S [192,320), dP [320,448).
// P stays in fp32 until dS = P o (dP - delta) is formed, which is rounded once.
// FINE: masked calls, whose gradients are those of fp32 probabilities.  P and dS enter the products as two bf16 terms
// (x = hi + lo to 2^-17; the second term lies in the columns the first leaves free), and the dQ kernel, run first, makes a
// pass of its own over the keys for delta = rowsum(P o dP), which from the bf16 result would carry its rounding.  Error of
// dq / dk / dv against 64 bits, 1024 tokens in segments: 1.66e-3, the rounding of the gradients themselves (single bf16 terms:
// 3.5e-3, 3.5e-3, 2.3e-3).
// One row of 2048 tokens, 16 heads, causal: dK/dV, dQ and delta 124 us, 108 with issuers whose warps stay together and the list
// of visible tiles; with all tokens in one segment, so that FINE does it, 1.4
// times that.  (torch's scaled_dot_product_attention, used
// here before: backward 90 us after running its own forward again, 41 us, and three copies.)
// ------------------------------------------------------------------------------------------
constexpr int W_D = 192;                       // query / key head dim
constexpr int W_QT = 64;                       // query rows per step of the dK/dV kernel
constexpr int W_STAGES = 3;                    // its Q and dO rings
constexpr int W_MAX_TILES = 2048;              // its query-tile table: 131,072 queries
constexpr int W_K_BYTES = BWD_T * W_D * 2;     // 48 KB: 128 rows of Q or K
constexpr int W_Q_BYTES = W_QT * W_D * 2;      // 24 KB
constexpr int W_DO_BYTES = W_QT * BWD_D * 2;   // 16 KB

namespace wkv {
constexpr int OFF_K = 0;
constexpr int OFF_V = OFF_K + W_K_BYTES;
constexpr int OFF_Q = OFF_V + TILE_BYTES;
constexpr int OFF_DO = OFF_Q + W_STAGES * W_Q_BYTES;
constexpr int OFF_AUX = OFF_DO + W_STAGES * W_DO_BYTES;      // per Q stage: lse2[64], delta[64], qpos[64], qseg[64]
constexpr int AUX_STAGE = 4 * W_QT * 4;
constexpr int OFF_LIST = OFF_AUX + W_STAGES * AUX_STAGE;     // as in the kernel above
constexpr int OFF_FLAGS = OFF_LIST + 2 * W_MAX_TILES;
constexpr int OFF_BAR = OFF_FLAGS + W_MAX_TILES;
constexpr int TOTAL = OFF_BAR + 256 + 1024;
static_assert(TOTAL <= 227 * 1024, "shared memory of one CTA");
constexpr int T_DK = 0, T_DV = 192, T_S = 320, T_DP = 448;
}  // namespace wkv

namespace wdq {
constexpr int OFF_Q = 0;
constexpr int OFF_DO = OFF_Q + W_K_BYTES;
constexpr int OFF_K = OFF_DO + TILE_BYTES;
constexpr int OFF_V = OFF_K + 2 * W_K_BYTES;
constexpr int OFF_RED = OFF_V + TILE_BYTES;    // FINE: [2][128] partial deltas of the two column halves
constexpr int OFF_BAR = OFF_RED + 2 * BWD_T * 4;
constexpr int TOTAL = OFF_BAR + 256 + 1024;
static_assert(TOTAL <= 227 * 1024, "shared memory of one CTA");
constexpr int T_DQ = 0, T_S = 192, T_DP = 320;
}  // namespace wdq

// Columns [c0, c0 + 32 * n) of one fp32 TMEM accumulator row times `mul` as bf16.
__device__ __forceinline__ void store_acc_cols(uint32_t tsrc, int c0, int n, __nv_bfloat16* dst, bool have, bool write,
                                               float mul) {
#pragma unroll 1
  for (int c = c0; c < c0 + 32 * n; c += 32) {
    uint32_t o[32];
    if (have) {
      tmem_ld32(tsrc + c, o);
      tmem_wait_ld();
    } else {
#pragma unroll
      for (int e = 0; e < 32; ++e) o[e] = 0;
    }
    if (write) {
#pragma unroll
      for (int v = 0; v < 4; ++v)
        *reinterpret_cast<uint4*>(dst + c + v * 8) = make_uint4(
            pack_bf16(__uint_as_float(o[8 * v]) * mul, __uint_as_float(o[8 * v + 1]) * mul),
            pack_bf16(__uint_as_float(o[8 * v + 2]) * mul, __uint_as_float(o[8 * v + 3]) * mul),
            pack_bf16(__uint_as_float(o[8 * v + 4]) * mul, __uint_as_float(o[8 * v + 5]) * mul),
            pack_bf16(__uint_as_float(o[8 * v + 6]) * mul, __uint_as_float(o[8 * v + 7]) * mul));
    }
  }
}

// 32 values of a row as a bf16 A operand in 16 TMEM columns; FINE: what the rounding lost in 16 more, `lo_cols` further on.
template <bool FINE>
__device__ __forceinline__ void store_operand(uint32_t dst, int lo_cols, const float* v) {
  uint32_t hi[16], lo[16];
#pragma unroll
  for (int c = 0; c < 16; ++c) {
    hi[c] = pack_bf16(v[2 * c], v[2 * c + 1]);
    if (FINE) {
      const float2 h = unpack_bf16(hi[c]);     // (no second term for what is not finite)
      lo[c] = pack_bf16(fabsf(h.x) < INFINITY ? v[2 * c] - h.x : 0.f, fabsf(h.y) < INFINITY ? v[2 * c + 1] - h.y : 0.f);
    }
  }
  tmem_st16(dst, hi);
  if (FINE) tmem_st16(dst + lo_cols, lo);
}

template <bool FINE>
__global__ void __launch_bounds__(BWD_THREADS, 1)
attn_bwd_dkv192_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                       const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmdO,
                       const AttnBwdParams p) {
  using namespace wkv;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + OFF_BAR);
  uint64_t* kv_full = bars;
  uint64_t* q_full = bars + 1;                    // [W_STAGES]
  uint64_t* q_empty = q_full + W_STAGES;
  uint64_t* do_full = q_empty + W_STAGES;
  uint64_t* do_empty = do_full + W_STAGES;
  uint64_t* s_full = do_empty + W_STAGES;         // [2] S^T of a step is in its buffer
  uint64_t* p_full = s_full + 2;                  // [2] one arrival per compute warp: P^T written over it
  uint64_t* dp_full = p_full + 2;
  uint64_t* ds_full = dp_full + 1;                // the same: dS^T written
  uint64_t* acc_done = ds_full + 1;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_done + 1);
  int* n_list = reinterpret_cast<int*>(acc_done + 2);
  uint16_t* list = reinterpret_cast<uint16_t*>(smem + OFF_LIST);
  uint8_t* flags = smem + OFF_FLAGS;

  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int kb = blockIdx.x / (p.Hkv * p.B);      // key-block major: the heaviest blocks first under a causal mask
  const int hkv = (blockIdx.x / p.B) % p.Hkv, b = blockIdx.x % p.B;
  const int G = p.Hq / p.Hkv;
  const int kv0 = kb * BWD_T;
  const int pos_off = p.Sk - p.Sq;
  const int n_tiles = (p.Sq + W_QT - 1) / W_QT;   // host guarantees <= W_MAX_TILES

  if (threadIdx.x == 0) {
    mbar_init(kv_full, 1);
    for (int i = 0; i < W_STAGES; ++i) {
      mbar_init(&q_full[i], 1); mbar_init(&q_empty[i], 1);
      mbar_init(&do_full[i], 1); mbar_init(&do_empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) { mbar_init(&s_full[i], 1); mbar_init(&p_full[i], 8); }
    mbar_init(dp_full, 1); mbar_init(ds_full, 8);
    mbar_init(acc_done, 1);
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  if (!chain_wait()) return;
  list_visible_tiles<W_QT>(p, p.kv_rng != nullptr, b, kb, n_tiles, flags, list, n_list);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  chain_launch();
  const int n_vis = *n_list;
  const int n_steps = n_vis * G;

  if (warp == 0) {
    // ------------------------------------------------------------------ producer
    if (n_steps > 0) {
      if (lane == 0) {
        tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmK); tma_prefetch_desc(&tmV); tma_prefetch_desc(&tmdO);
        mbar_expect_tx(kv_full, W_K_BYTES + TILE_BYTES);
        for (int c = 0; c < W_D / 64; ++c)
          tma_load_3d(smem + OFF_K + c * (BWD_T * 128), &tmK, kv_full, c * 64, b * p.Sk + kv0, hkv);
        for (int c = 0; c < BWD_D / 64; ++c)
          tma_load_3d(smem + OFF_V + c * (BWD_T * 128), &tmV, kv_full, c * 64, b * p.Sk + kv0, hkv);
      }
      const bool aux_rows = p.q_pos != nullptr || p.q_seg != nullptr;
      int step = 0;
      bool ok = true;
      for (int g = 0; g < G && ok; ++g) {
        const int hq = hkv * G + g;
        for (int v = 0; v < n_vis; ++v) {
          const int st = step % W_STAGES;
          const uint32_t ph = ((step / W_STAGES) & 1) ^ 1;
          const int q0 = (int)(list[v] & (kMasked - 1)) * W_QT;
          int okw = 1;
          if (lane == 0) okw = mbar_wait(&q_empty[st], ph, p.status, kTimeoutStageFree, 121) ? 1 : 0;
          okw = __shfl_sync(0xffffffffu, okw, 0);
          if (!okw) { ok = false; break; }
          float* aux = reinterpret_cast<float*>(smem + OFF_AUX + st * AUX_STAGE);
          int* auxi = reinterpret_cast<int*>(aux);
          if (aux_rows && !p.aux_bulk) {
            for (int c = lane; c < W_QT; c += 32) {
              const int r = min(q0 + c, p.Sq - 1);
              auxi[2 * W_QT + c] = p.q_pos ? p.q_pos[(long long)b * p.Sq + r] : 0;
              auxi[3 * W_QT + c] = p.q_seg ? p.q_seg[(long long)b * p.Sq + r] : 0;
            }
            __syncwarp();
          }
          if (lane == 0) {
            const uint32_t rows_bytes = (uint32_t)min(W_QT, p.Sq - q0) * 4u;
            uint32_t tx = W_Q_BYTES + 2 * W_QT * 4;
            if (aux_rows && p.aux_bulk) tx += (p.q_pos ? rows_bytes : 0u) + (p.q_seg ? rows_bytes : 0u);
            mbar_expect_tx(&q_full[st], tx);
            for (int c = 0; c < W_D / 64; ++c)
              tma_load_3d(smem + OFF_Q + st * W_Q_BYTES + c * (W_QT * 128), &tmQ, &q_full[st], c * 64, b * p.Sq + q0, hq);
            const long long li = ((long long)b * p.Hq + hq) * p.Sq_pad + q0;
            bulk_load(aux, p.lse2 + li, W_QT * 4, &q_full[st]);
            bulk_load(aux + W_QT, p.delta + li, W_QT * 4, &q_full[st]);
            if (aux_rows && p.aux_bulk) {
              if (p.q_pos) bulk_load(auxi + 2 * W_QT, p.q_pos + (long long)b * p.Sq + q0, rows_bytes, &q_full[st]);
              if (p.q_seg) bulk_load(auxi + 3 * W_QT, p.q_seg + (long long)b * p.Sq + q0, rows_bytes, &q_full[st]);
            }
            if (mbar_wait(&do_empty[st], ph, p.status, kTimeoutStageFree, 129)) {
              mbar_expect_tx(&do_full[st], W_DO_BYTES);
              for (int c = 0; c < BWD_D / 64; ++c)
                tma_load_3d(smem + OFF_DO + st * W_DO_BYTES + c * (W_QT * 128), &tmdO, &do_full[st], c * 64,
                            b * p.Sq + q0, hq);
            } else {
              okw = 0;
            }
          }
          okw = __shfl_sync(0xffffffffu, okw, 0);
          if (!okw) { ok = false; break; }
          ++step;
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (n_steps > 0) {
      constexpr uint32_t id_s = make_idesc_bf16(BWD_T, W_QT, false, false);     // S^T, dP^T
      constexpr uint32_t id_dv = make_idesc_bf16(BWD_T, BWD_D, false, true);    // dV (A in TMEM, B MN-major)
      constexpr uint32_t id_dk = make_idesc_bf16(BWD_T, W_D, false, true);      // dK
      const uint32_t dK = kmajor_lo(smem_u32(smem + OFF_K)), dVd = kmajor_lo(smem_u32(smem + OFF_V));
      const uint32_t aQ0 = smem_u32(smem + OFF_Q), aDO0 = smem_u32(smem + OFF_DO);
      const uint32_t tDP = tmem_base + T_DP;
      // k-step k of a K-major tile of `rows` rows in 64-wide blocks, and the TMEM column of a bf16 A operand
      // whose halves of 32 values lie packed at the start of their own 32 columns (FINE: second terms behind them)
      auto kstep = [](int rows, int k) { return (uint32_t)(((k >> 2) * (rows * 128) + (k & 3) * 32) >> 4); };
      auto acol = [](int k) { return (uint32_t)((k >> 1) * 32 + (k & 1) * 8); };
      auto wait_q = [&](int i) { return mbar_wait_warp(&q_full[i % W_STAGES], (i / W_STAGES) & 1, p.status, kTimeoutTmaFull, 123); };
      auto wait_do = [&](int i) { return mbar_wait_warp(&do_full[i % W_STAGES], (i / W_STAGES) & 1, p.status, kTimeoutTmaFull, 124); };
      auto issue_s = [&](int i) -> bool {      // S^T(i) = K Q(i)^T
        if (!wait_q(i)) return false;
        tc_fence_after();
        const uint32_t dQ = kmajor_lo(aQ0 + (i % W_STAGES) * W_Q_BYTES);
        one_lane([&] {
#pragma unroll
          for (int k = 0; k < W_D / 16; ++k)
            mma_ss_w(tmem_base + T_S + (i & 1) * W_QT, dK + kstep(BWD_T, k), kDescHi, dQ + kstep(W_QT, k), kDescHi, id_s, k != 0);
          tc_commit(&s_full[i & 1]);
        });
        return true;
      };
      auto issue_dp = [&](int i) -> bool {     // dP^T(i) = V dO(i)^T
        if (!wait_do(i)) return false;
        tc_fence_after();
        const uint32_t dDO = kmajor_lo(aDO0 + (i % W_STAGES) * W_DO_BYTES);
        one_lane([&] {
#pragma unroll
          for (int k = 0; k < BWD_D / 16; ++k)
            mma_ss_w(tDP, dVd + kstep(BWD_T, k), kDescHi, dDO + kstep(W_QT, k), kDescHi, id_s, k != 0);
          tc_commit(dp_full);
        });
        return true;
      };
      bool ok = mbar_wait_warp(kv_full, 0, p.status, kTimeoutTmaFull, 122);
      if (ok) ok = issue_s(0) && issue_dp(0);
      for (int i = 0; i < n_steps && ok; ++i) {
        const int st = i % W_STAGES;
        const bool more = i + 1 < n_steps;
        // its buffer held P^T(i - 1), which dV(i - 1), issued before, has read by then
        if (more && !issue_s(i + 1)) break;
        if (!mbar_wait_warp(&p_full[i & 1], (i >> 1) & 1, p.status, kTimeoutSoftmax, 125)) break;
        tc_fence_after();
        const uint32_t mDO = smem_desc_lo(aDO0 + st * W_DO_BYTES, W_QT * 128);
        one_lane([&] {
#pragma unroll
          for (int k = 0; k < W_QT / 16; ++k) {  // dV += P^T dO
            const uint32_t a = tmem_base + T_S + (i & 1) * W_QT + acol(k);
            mma_ts_w(tmem_base + T_DV, a, mDO + mnmajor_k(k), kDescHi, id_dv, (i | k) != 0);
            if (FINE) mma_ts_w(tmem_base + T_DV, a + 16, mDO + mnmajor_k(k), kDescHi, id_dv, 1);
          }
          tc_commit(&do_empty[st]);
        });
        if (!mbar_wait_warp(ds_full, i & 1, p.status, kTimeoutSoftmax, 126)) break;
        tc_fence_after();
        const uint32_t mQ = smem_desc_lo(aQ0 + st * W_Q_BYTES, W_QT * 128);
        one_lane([&] {
#pragma unroll
          for (int k = 0; k < W_QT / 16; ++k) {  // dK += dS^T Q
            mma_ts_w(tmem_base + T_DK, tDP + acol(k), mQ + mnmajor_k(k), kDescHi, id_dk, (i | k) != 0);
            if (FINE) mma_ts_w(tmem_base + T_DK, tDP + acol(k) + 16, mQ + mnmajor_k(k), kDescHi, id_dk, 1);
          }
          tc_commit(&q_empty[st]);
        });
        if (more && !issue_dp(i + 1)) break;
      }
      one_lane([&] { tc_commit(acc_done); });
    }
  } else {
    // ------------------------------------------------------------------ compute warps
    const int qd = warp & 3;
    const int half = (warp - 2) >> 2;             // which 32 of the 64 query columns
    const int r_local = qd * 32 + lane;           // key row == TMEM lane
    const int kp = kv0 + r_local;
    const bool key_ok = kp < p.Sk;
    const int kseg = (p.kv_seg && key_ok) ? p.kv_seg[(long long)b * p.Sk + kp] : 0;
    const uint32_t tb = tmem_base + ((uint32_t)(qd * 32) << 16);
    const uint32_t tDP = tb + T_DP + half * 32;
    const int win = p.window > 0 ? p.window : 0x7fffffff;
    const int cmax = p.causal ? kp : -0x7fffffff;
    bool ok = true;
    int step = 0;
    for (int g = 0; g < G && ok; ++g) {
      for (int v = 0; v < n_vis && ok; ++v) {
        const uint32_t entry = list[v];
        const int t = (int)(entry & (kMasked - 1));
        const float* aux = reinterpret_cast<const float*>(smem + OFF_AUX + (step % W_STAGES) * AUX_STAGE);
        const int* auxi = reinterpret_cast<const int*>(aux);
        const uint32_t tS = tb + T_S + (step & 1) * W_QT + half * 32;
        const bool need_mask = (entry & kMasked) != 0;
        // ---- phase 1: P^T = exp2(S^T * c - lse)
        if (!mbar_wait(&s_full[step & 1], (step >> 1) & 1, p.status, kTimeoutAccFull, 127)) { ok = false; break; }
        tc_fence_after();
        float pf[32];
        {
          uint32_t s[32];
          tmem_ld32(tS, s);
          tmem_wait_ld();
          const float4* lse4 = reinterpret_cast<const float4*>(aux + half * 32);
          const int4* qp4 = reinterpret_cast<const int4*>(auxi + 2 * W_QT + half * 32);
          const int4* qs4 = reinterpret_cast<const int4*>(auxi + 3 * W_QT + half * 32);
          if (!need_mask) {
#pragma unroll
            for (int c4 = 0; c4 < 8; ++c4) {
              const float4 L = lse4[c4];
              pf[4 * c4] = exp2f(fmaf(__uint_as_float(s[4 * c4]), p.scale_log2, -L.x));
              pf[4 * c4 + 1] = exp2f(fmaf(__uint_as_float(s[4 * c4 + 1]), p.scale_log2, -L.y));
              pf[4 * c4 + 2] = exp2f(fmaf(__uint_as_float(s[4 * c4 + 2]), p.scale_log2, -L.z));
              pf[4 * c4 + 3] = exp2f(fmaf(__uint_as_float(s[4 * c4 + 3]), p.scale_log2, -L.w));
            }
          } else {
#pragma unroll
            for (int c4 = 0; c4 < 8; ++c4) {
              const float4 L = lse4[c4];
              const int qn = t * W_QT + pos_off + half * 32 + 4 * c4;   // natural positions
              const int4 QP = p.q_pos ? qp4[c4] : make_int4(qn, qn + 1, qn + 2, qn + 3);
              const int4 QS = p.q_seg ? qs4[c4] : make_int4(0, 0, 0, 0);
              const float l[4] = {L.x, L.y, L.z, L.w};
              const int qp[4] = {QP.x, QP.y, QP.z, QP.w}, qs[4] = {QS.x, QS.y, QS.z, QS.w};
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const bool keep = key_ok & (qp[e] >= cmax) & (qp[e] - kp < win) & (qs[e] == kseg);
                const float pe = exp2f(fmaf(__uint_as_float(s[4 * c4 + e]), p.scale_log2, -l[e]));
                pf[4 * c4 + e] = keep ? pe : 0.f;
              }
            }
          }
          store_operand<FINE>(tS, 16, pf);
        }
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_full[step & 1]);
        // ---- phase 2: dS^T = P^T o (dP^T - delta), written over dP^T
        if (!mbar_wait(dp_full, step & 1, p.status, kTimeoutAccFull, 128)) { ok = false; break; }
        tc_fence_after();
        {
          uint32_t d[32];
          tmem_ld32(tDP, d);
          tmem_wait_ld();
          const float4* dlt4 = reinterpret_cast<const float4*>(aux + W_QT + half * 32);
#pragma unroll
          for (int c4 = 0; c4 < 8; ++c4) {
            const float4 Dl = dlt4[c4];
            pf[4 * c4] *= __uint_as_float(d[4 * c4]) - Dl.x;
            pf[4 * c4 + 1] *= __uint_as_float(d[4 * c4 + 1]) - Dl.y;
            pf[4 * c4 + 2] *= __uint_as_float(d[4 * c4 + 2]) - Dl.z;
            pf[4 * c4 + 3] *= __uint_as_float(d[4 * c4 + 3]) - Dl.w;
          }
          store_operand<FINE>(tDP, 16, pf);
        }
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(ds_full);
        ++step;
      }
    }
    if (ok && n_steps > 0) ok = mbar_wait(acc_done, 0, p.status, kTimeoutAccFull, 130);
    tc_fence_after();
    const bool have = ok && n_steps > 0;
    store_acc_cols(tb + T_DK, half * 96, 3, p.dK + ((long long)b * p.Sk + kp) * p.lddk + (long long)hkv * W_D, have, key_ok,
                   p.scale);
    store_acc_cols(tb + T_DV, half * 64, 2, p.dV + ((long long)b * p.Sk + kp) * p.lddv + (long long)hkv * BWD_D, have,
                   key_ok, 1.f);
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// FINE: the key blocks are run through twice, first for delta (S and dP only), then for dQ.
template <bool FINE>
__global__ void __launch_bounds__(BWD_THREADS, 1)
attn_bwd_dq192_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                      const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmdO,
                      const AttnBwdParams p) {
  using namespace wdq;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + OFF_BAR);
  uint64_t* qdo_full = bars;
  uint64_t* k_full = bars + 1;                    // [2]
  uint64_t* k_empty = bars + 3;                   // [2]
  uint64_t* v_full = bars + 5;
  uint64_t* v_empty = bars + 6;
  uint64_t* s_full = bars + 7;
  uint64_t* s_read = bars + 8;                    // count 256: S is in registers
  uint64_t* dp_full = bars + 9;
  uint64_t* ds_full = bars + 10;                  // count 256
  uint64_t* acc_done = bars + 11;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 12);
  int* tile_minmax = reinterpret_cast<int*>(bars + 13);   // [2]
  int* seg_lohi = reinterpret_cast<int*>(bars + 14);      // [2]
  float* red = reinterpret_cast<float*>(smem + OFF_RED);

  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int n_qtiles = (p.Sq + BWD_T - 1) / BWD_T;
  const int qt = n_qtiles - 1 - (int)(blockIdx.x / (p.Hq * p.B));   // heaviest query tiles first
  const int hq = (blockIdx.x / p.B) % p.Hq, b = blockIdx.x % p.B;
  const int hkv = hq / (p.Hq / p.Hkv);
  const int q0 = qt * BWD_T;
  const int pos_off = p.Sk - p.Sq;

  if (threadIdx.x == 0) {
    mbar_init(qdo_full, 1);
    for (int i = 0; i < 2; ++i) { mbar_init(&k_full[i], 1); mbar_init(&k_empty[i], 1); }
    mbar_init(v_full, 1); mbar_init(v_empty, 1);
    mbar_init(s_full, 1); mbar_init(s_read, 256);
    mbar_init(dp_full, 1); mbar_init(ds_full, 256);
    mbar_init(acc_done, 1);
    tile_minmax[0] = 0x7fffffff;
    tile_minmax[1] = -0x7fffffff;
    seg_lohi[0] = 0x7fffffff;
    seg_lohi[1] = -1;
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  chain_launch();
  if (!chain_wait()) return;

  int qpos_min = q0 + pos_off, qpos_max = min(q0 + BWD_T, p.Sq) - 1 + pos_off;
  if (p.q_pos) {
    if (threadIdx.x < BWD_T && q0 + (int)threadIdx.x < p.Sq) {
      const int qp = p.q_pos[(long long)b * p.Sq + q0 + threadIdx.x];
      atomicMin(&tile_minmax[0], qp);
      atomicMax(&tile_minmax[1], qp);
    }
    __syncthreads();
    qpos_min = tile_minmax[0];
    qpos_max = tile_minmax[1];
  }
  const int nblk_total = (p.Sk + BWD_T - 1) / BWD_T;
  int blk_hi = p.causal ? min(nblk_total, qpos_max / BWD_T + 1) : nblk_total;
  int blk_lo = (p.window > 0 && qpos_min >= p.window) ? (qpos_min - p.window + 1) / BWD_T : 0;
  if (p.causal && qpos_max < 0) blk_hi = 0;
  int2 qr = make_int2(0, 0);
  if (p.kv_rng) {
    qr = seg_range128(p.q_rng, b, qt, p.Sq);
    for (int i = blk_lo + (int)threadIdx.x; i < blk_hi; i += BWD_THREADS) {
      const int2 kr = seg_range128(p.kv_rng, b, i, p.Sk);
      if (kr.x <= qr.y && kr.y >= qr.x) {
        atomicMin(&seg_lohi[0], i);
        atomicMax(&seg_lohi[1], i);
      }
    }
    __syncthreads();
    blk_lo = max(blk_lo, seg_lohi[0]);
    blk_hi = min(blk_hi, seg_lohi[1] + 1);
  }
  const int nblk = max(0, blk_hi - blk_lo);
  const int n_steps = FINE ? 2 * nblk : nblk;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (nblk > 0 && elect_one()) {
      tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmK); tma_prefetch_desc(&tmV); tma_prefetch_desc(&tmdO);
      mbar_expect_tx(qdo_full, W_K_BYTES + TILE_BYTES);
      for (int c = 0; c < W_D / 64; ++c)
        tma_load_3d(smem + OFF_Q + c * (BWD_T * 128), &tmQ, qdo_full, c * 64, b * p.Sq + q0, hq);
      for (int c = 0; c < BWD_D / 64; ++c)
        tma_load_3d(smem + OFF_DO + c * (BWD_T * 128), &tmdO, qdo_full, c * 64, b * p.Sq + q0, hq);
      for (int j = 0; j < n_steps; ++j) {
        const int st = j & 1;
        const int row = b * p.Sk + (blk_lo + (j < nblk ? j : j - nblk)) * BWD_T;
        if (!mbar_wait(&k_empty[st], ((j >> 1) & 1) ^ 1, p.status, kTimeoutStageFree, 131)) break;
        mbar_expect_tx(&k_full[st], W_K_BYTES);
        for (int c = 0; c < W_D / 64; ++c)
          tma_load_3d(smem + OFF_K + st * W_K_BYTES + c * (BWD_T * 128), &tmK, &k_full[st], c * 64, row, hkv);
        if (!mbar_wait(v_empty, (j & 1) ^ 1, p.status, kTimeoutStageFree, 135)) break;
        mbar_expect_tx(v_full, TILE_BYTES);
        for (int c = 0; c < BWD_D / 64; ++c)
          tma_load_3d(smem + OFF_V + c * (BWD_T * 128), &tmV, v_full, c * 64, row, hkv);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (nblk > 0) {
      constexpr uint32_t id_s = make_idesc_bf16(BWD_T, BWD_T, false, false);    // S, dP
      constexpr uint32_t id_dq = make_idesc_bf16(BWD_T, W_D, false, true);      // dQ (A in TMEM, B MN-major)
      const uint32_t dQ = kmajor_lo(smem_u32(smem + OFF_Q)), dDO = kmajor_lo(smem_u32(smem + OFF_DO));
      const uint32_t dV = kmajor_lo(smem_u32(smem + OFF_V));
      const uint32_t aK0 = smem_u32(smem + OFF_K);
      const uint32_t tS = tmem_base + T_S, tDP = tmem_base + T_DP;
      auto kstep = [](int k) { return (uint32_t)(((k >> 2) * (BWD_T * 128) + (k & 3) * 32) >> 4); };
      auto issue_s = [&](int j) -> bool {      // S(j) = Q K_j^T
        if (!mbar_wait_warp(&k_full[j & 1], (j >> 1) & 1, p.status, kTimeoutTmaFull, 133)) return false;
        tc_fence_after();
        const uint32_t dK = kmajor_lo(aK0 + (j & 1) * W_K_BYTES);
        one_lane([&] {
#pragma unroll
          for (int k = 0; k < W_D / 16; ++k) mma_ss_w(tS, dQ + kstep(k), kDescHi, dK + kstep(k), kDescHi, id_s, k != 0);
          tc_commit(s_full);
        });
        return true;
      };
      auto issue_dp = [&](int j) -> bool {     // dP(j) = dO V_j^T
        if (!mbar_wait_warp(v_full, j & 1, p.status, kTimeoutTmaFull, 137)) return false;
        tc_fence_after();
        one_lane([&] {
#pragma unroll
          for (int k = 0; k < BWD_D / 16; ++k) mma_ss_w(tDP, dDO + kstep(k), kDescHi, dV + kstep(k), kDescHi, id_s, k != 0);
          tc_commit(v_empty);
          tc_commit(dp_full);
        });
        return true;
      };
      bool ok = mbar_wait_warp(qdo_full, 0, p.status, kTimeoutTmaFull, 132);
      if (ok) ok = issue_s(0) && issue_dp(0);
      for (int j = 0; j < n_steps && ok; ++j) {
        const bool more = j + 1 < n_steps;
        const int jq = FINE ? j - nblk : j;      // step of the dQ pass
        if (more) {
          if (!mbar_wait_warp(s_read, j & 1, p.status, kTimeoutSoftmax, 140)) break;   // S(j) is in registers
          tc_fence_after();
          if (!issue_s(j + 1)) break;
        }
        if (!mbar_wait_warp(ds_full, j & 1, p.status, kTimeoutSoftmax, 134)) break;
        tc_fence_after();
        const uint32_t mK = mnmajor_lo(aK0 + (j & 1) * W_K_BYTES);
        one_lane([&] {
          if (jq >= 0) {
#pragma unroll
            for (int k = 0; k < BWD_T / 16; ++k) {   // dQ += dS K
              mma_ts_w(tmem_base + T_DQ, tDP + a_col(k), mK + mnmajor_k(k), kDescHi, id_dq, (jq | k) != 0);
              if (FINE) mma_ts_w(tmem_base + T_DQ, tDP + a_col(k) + 32, mK + mnmajor_k(k), kDescHi, id_dq, 1);
            }
          }
          tc_commit(&k_empty[j & 1]);
        });
        if (more && !issue_dp(j + 1)) break;
      }
      one_lane([&] { tc_commit(acc_done); });
    }
  } else {
    // ------------------------------------------------------------------ compute warps
    const int qd = warp & 3;
    const int half = (warp - 2) >> 2;             // which 64 of the 128 key columns
    const int r_local = qd * 32 + lane;           // query row == TMEM lane
    const int row = q0 + r_local;
    const bool row_ok = row < p.Sq;
    const long long grow = (long long)b * p.Sq + row;
    const int qpos = row_ok ? (p.q_pos ? p.q_pos[grow] : row + pos_off) : -1;
    const int qseg = (p.q_seg && row_ok) ? p.q_seg[grow] : 0;
    const long long li = ((long long)b * p.Hq + hq) * p.Sq_pad + row;   // row < Sq_pad: padded to 128
    const float lse2 = p.lse2[li];
    float delta = FINE ? 0.f : p.delta[li];
    const uint32_t tb = tmem_base + ((uint32_t)(qd * 32) << 16);
    const uint32_t tS = tb + T_S + half * 64, tDP = tb + T_DP + half * 64;
    const int* ks = p.kv_seg ? p.kv_seg + (long long)b * p.Sk : nullptr;
    const int win = p.window > 0 ? p.window : 0x7fffffff;
    const int kmax = p.causal ? min(qpos, p.Sk - 1) : p.Sk - 1;   // keep needs kp <= kmax
    bool ok = true;

    for (int pass = FINE ? 0 : 1; pass < 2; ++pass) {
      float own = 0.f;              // this thread's part of delta
      for (int jb = 0; jb < nblk && ok; ++jb) {
        const int j = FINE && pass ? nblk + jb : jb;
        const int kv0 = (blk_lo + jb) * BWD_T;
        bool seg_mask = p.q_seg != nullptr;
        if (p.kv_rng) {
          const int2 kr = seg_range128(p.kv_rng, b, blk_lo + jb, p.Sk);
          seg_mask = !(qr.x == qr.y && kr.x == kr.y && qr.x == kr.x);
        }
        const bool need_mask = (p.causal && kv0 + BWD_T - 1 > qpos_min) || (kv0 + BWD_T > p.Sk) ||
                               (p.window > 0 && qpos_max - kv0 >= p.window) || seg_mask;
        // ---- phase 1: P = exp2(S * c - lse), in registers
        if (!mbar_wait(s_full, j & 1, p.status, kTimeoutAccFull, 136)) { ok = false; break; }
        tc_fence_after();
        float pf[64];
        uint32_t sreg[64];
        tmem_ld32(tS, sreg);
        tmem_ld32(tS + 32, sreg + 32);
        tmem_wait_ld();
        tc_fence_before();
        mbar_arrive(s_read);
#pragma unroll
        for (int ch = 0; ch < 2; ++ch) {
          const uint32_t* s = sreg + ch * 32;
          if (!need_mask) {
#pragma unroll
            for (int c = 0; c < 32; ++c) pf[ch * 32 + c] = exp2f(fmaf(__uint_as_float(s[c]), p.scale_log2, -lse2));
          } else {
            const int kbase = kv0 + half * 64 + ch * 32;
#pragma unroll
            for (int c = 0; c < 32; ++c) {
              const int kp = kbase + c;
              bool keep = (kp <= kmax) & (qpos - kp < win);
              if (ks && seg_mask) keep = keep & (__ldg(ks + min(kp, p.Sk - 1)) == qseg);
              const float pe = exp2f(fmaf(__uint_as_float(s[c]), p.scale_log2, -lse2));
              pf[ch * 32 + c] = keep ? pe : 0.f;
            }
          }
        }
        // ---- phase 2: dS = P o (dP - delta), written over dP; or this block's share of delta
        if (!mbar_wait(dp_full, j & 1, p.status, kTimeoutAccFull, 139)) { ok = false; break; }
        tc_fence_after();
        {
          uint32_t dreg[64];
          tmem_ld32(tDP, dreg);
          tmem_ld32(tDP + 32, dreg + 32);
          tmem_wait_ld();
          if (pass == 0) {
#pragma unroll
            for (int c = 0; c < 64; ++c) own = fmaf(pf[c], __uint_as_float(dreg[c]), own);
          } else {
#pragma unroll
            for (int c = 0; c < 64; ++c) pf[c] *= __uint_as_float(dreg[c]) - delta;
            store_operand<FINE>(tDP, 32, pf);
            store_operand<FINE>(tDP + 16, 32, pf + 32);
          }
        }
        tmem_wait_st();
        tc_fence_before();
        mbar_arrive(ds_full);
      }
      if (pass == 0) {              // (reached by every compute thread, whatever became of its waits)
        red[half * BWD_T + r_local] = own;
        named_bar_sync(1, 256);
        delta = row_ok ? red[r_local] + red[BWD_T + r_local] : 0.f;
        if (half == 0) p.delta_out[li] = delta;
      }
    }
    if (ok && nblk > 0) ok = mbar_wait(acc_done, 0, p.status, kTimeoutAccFull, 138);
    tc_fence_after();
    store_acc_cols(tb + T_DQ, half * 96, 3, p.dQ + grow * p.lddq + (long long)hq * W_D, ok && nblk > 0, row_ok, p.scale);
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

}  // namespace tpb

using namespace tpb;


// Floats of scratch `tpb_attn_bwd` needs (scaled log-sum-exp and delta rows, padded to 128).
extern "C" long long tpb_attn_bwd_scratch_floats(int B, int Sq, int Hq) {
  const long long sq_pad = (Sq + BWD_T - 1) / BWD_T * BWD_T;
  return 2LL * B * Hq * sq_pad;
}

// `softcap` > 0: the scores were capped as softcap * tanh(q.k * scale / softcap) in the forward pass.
extern "C" int tpb_attn_bwd_softcap(const void* dO, const void* q, const void* k, const void* v, const void* o,
                                    const float* lse, float* scratch, void* dq, void* dk, void* dv, int B, int Sq,
                                    int Sk, int Hq, int Hkv, int dqk, int dvd, long long ldq, long long ldk,
                                    long long ldv, long long lddo, long long lddq, long long lddk, long long lddv,
                                    float scale, int causal, int window, const int* q_pos, const int* q_seg,
                                    const int* kv_seg, const int* q_rng, const int* kv_rng, float softcap,
                                    void* stream_) {
  const bool wide = dqk == W_D;
  if ((dqk != 128 && !wide) || dvd != 128 || Hq % Hkv || (wide && softcap > 0.f)) return -2;
  if ((ldq % 8) || (ldk % 8) || (ldv % 8) || (lddo % 8) || (lddq % 8) || (lddk % 8) || (lddv % 8)) return -2;
  if (lddo != (long long)Hq * dvd) return -2;   // dO and O are contiguous [B*Sq, Hq, 128]
  if (B <= 0 || Sq <= 0 || Sk <= 0) return 0;
  if (wide ? (Sq + W_QT - 1) / W_QT > W_MAX_TILES : (Sq + BWD_T - 1) / BWD_T > KV_MAX_TILES) return -6;
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  const int sq_pad = (Sq + BWD_T - 1) / BWD_T * BWD_T;
  float* lse2 = scratch;
  float* delta = scratch + (long long)B * Hq * sq_pad;
  {
    const long long blocks = (long long)B * ((Hq + DELTA_H - 1) / DELTA_H) * (sq_pad / DELTA_T);
    if (blocks > 0x7fffffff) return -2;
    chain(attn_bwd_delta_kernel, (int)blocks, DELTA_THREADS, 0, stream,
          reinterpret_cast<const __nv_bfloat16*>(dO), reinterpret_cast<const __nv_bfloat16*>(o), lse, lse2, delta, Sq, sq_pad, Hq);
  }
  AttnBwdParams p;
  p.B = B; p.Sq = Sq; p.Sk = Sk; p.Hq = Hq; p.Hkv = Hkv;
  p.scale = scale;
  p.softcap_in = softcap > 0.f ? scale / softcap : 0.f;
  p.scale_log2 = (softcap > 0.f ? softcap : scale) * kLog2e;
  p.causal = causal; p.window = window;
  p.q_pos = q_pos; p.q_seg = q_seg; p.kv_seg = kv_seg;
  const bool ranges = q_seg && kv_seg && q_rng && kv_rng;
  p.q_rng = ranges ? reinterpret_cast<const int2*>(q_rng) : nullptr;
  p.kv_rng = ranges ? reinterpret_cast<const int2*>(kv_rng) : nullptr;
  p.lse2 = lse2; p.delta = delta; p.delta_out = delta; p.Sq_pad = sq_pad;
  p.aux_bulk = (Sq % 4 == 0) && (reinterpret_cast<uintptr_t>(q_pos) % 16 == 0) &&
               (reinterpret_cast<uintptr_t>(q_seg) % 16 == 0);
  p.dQ = reinterpret_cast<__nv_bfloat16*>(dq); p.lddq = lddq;
  p.dK = reinterpret_cast<__nv_bfloat16*>(dk); p.lddk = lddk;
  p.dV = reinterpret_cast<__nv_bfloat16*>(dv); p.lddv = lddv;
  p.status = status_block();
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaSuccess;
    auto allow = [&](const void* kernel, int bytes) {
      if (e == cudaSuccess) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    };
    allow((const void*)attn_bwd_dkv_kernel<false, false>, dkv::TOTAL); allow((const void*)attn_bwd_dq_kernel<false, false>, dqk::TOTAL);
    allow((const void*)attn_bwd_dkv_kernel<false, true>, dkv::TOTAL); allow((const void*)attn_bwd_dq_kernel<false, true>, dqk::TOTAL);
    allow((const void*)attn_bwd_dkv_kernel<true, false>, dkv::TOTAL); allow((const void*)attn_bwd_dq_kernel<true, false>, dqk::TOTAL);
    allow((const void*)attn_bwd_dkv_kernel<true, true>, dkv::TOTAL); allow((const void*)attn_bwd_dq_kernel<true, true>, dqk::TOTAL);
    allow((const void*)attn_bwd_dkv192_kernel<false>, wkv::TOTAL); allow((const void*)attn_bwd_dq192_kernel<false>, wdq::TOTAL);
    allow((const void*)attn_bwd_dkv192_kernel<true>, wkv::TOTAL); allow((const void*)attn_bwd_dq192_kernel<true>, wdq::TOTAL);
    if (e != cudaSuccess) return 1000 + (int)e;
    configured = true;
  }
  // every operand is streamed as 128-row tiles in two 64-wide d blocks
  CUtensorMap tq, tk, tv, tdo;
  if (make_tmap_3d(&tq, q, dqk, (uint64_t)B * Sq, Hq, ldq, dqk, 64, BWD_T)) return -3;
  if (make_tmap_3d(&tk, k, dqk, (uint64_t)B * Sk, Hkv, ldk, dqk, 64, BWD_T)) return -4;
  if (make_tmap_3d(&tv, v, dvd, (uint64_t)B * Sk, Hkv, ldv, dvd, 64, BWD_T)) return -5;
  if (make_tmap_3d(&tdo, dO, dvd, (uint64_t)B * Sq, Hq, lddo, dvd, 64, BWD_T)) return -5;
  dim3 grid_kv(((Sk + BWD_T - 1) / BWD_T) * Hkv * B, 1, 1);
  if (wide) {
    CUtensorMap tq64, tdo64;      // the dK/dV kernel takes its queries 64 rows at a time
    if (make_tmap_3d(&tq64, q, dqk, (uint64_t)B * Sq, Hq, ldq, dqk, 64, W_QT)) return -3;
    if (make_tmap_3d(&tdo64, dO, dvd, (uint64_t)B * Sq, Hq, lddo, dvd, 64, W_QT)) return -5;
    const bool fine = q_pos || q_seg || kv_seg || window > 0 || (causal && Sq != Sk);
    const int grid_wq = ((Sq + BWD_T - 1) / BWD_T) * Hq * B;
    // (FINE: dK/dV takes the deltas that the dQ kernel leaves)
    chain(fine ? attn_bwd_dq192_kernel<true> : attn_bwd_dq192_kernel<false>, grid_wq, BWD_THREADS, wdq::TOTAL, stream,
          tq, tk, tv, tdo, p);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return 1000 + (int)e;
    chain(fine ? attn_bwd_dkv192_kernel<true> : attn_bwd_dkv192_kernel<false>, grid_kv, BWD_THREADS, wkv::TOTAL, stream,
          tq64, tk, tv, tdo64, p);
    e = cudaGetLastError();
    return e == cudaSuccess ? 0 : 1000 + (int)e;
  }
  chain(softcap > 0.f ? (ranges ? attn_bwd_dkv_kernel<true, true> : attn_bwd_dkv_kernel<true, false>)
                      : (ranges ? attn_bwd_dkv_kernel<false, true> : attn_bwd_dkv_kernel<false, false>),
        grid_kv, BWD_THREADS, dkv::TOTAL, stream, tq, tk, tv, tdo, p);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return 1000 + (int)e;
  dim3 grid_q(((Sq + BWD_T - 1) / BWD_T) * Hq * B, 1, 1);
  chain(softcap > 0.f ? (ranges ? attn_bwd_dq_kernel<true, true> : attn_bwd_dq_kernel<true, false>)
                      : (ranges ? attn_bwd_dq_kernel<false, true> : attn_bwd_dq_kernel<false, false>),
        grid_q, BWD_THREADS, dqk::TOTAL, stream, tq, tk, tv, tdo, p);
  e = cudaGetLastError();
  return e == cudaSuccess ? 0 : 1000 + (int)e;
}

extern "C" int tpb_attn_bwd(const void* dO, const void* q, const void* k, const void* v, const void* o,
                            const float* lse, float* scratch, void* dq, void* dk, void* dv, int B, int Sq,
                            int Sk, int Hq, int Hkv, int dqk, int dvd, long long ldq, long long ldk, long long ldv,
                            long long lddo, long long lddq, long long lddk, long long lddv, float scale, int causal,
                            int window, const int* q_pos, const int* q_seg, const int* kv_seg, void* stream_) {
  return tpb_attn_bwd_softcap(dO, q, k, v, o, lse, scratch, dq, dk, dv, B, Sq, Sk, Hq, Hkv, dqk, dvd, ldq, ldk, ldv, lddo,
                              lddq, lddk, lddv, scale, causal, window, q_pos, q_seg, kv_seg, nullptr, nullptr, 0.f, stream_);
}
