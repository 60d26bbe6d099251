// Mixture-of-experts support kernels: fused router top-k (softmax / sigmoid with
// group-limited selection), row gather into the expert-grouped layout, weighted combine
// back to token order and the routing-weight gradient.  The grouped GEMMs themselves are
// the grouped modes of gemm_sm100.cu.

#include "common.cuh"
#include "tpb.h"

namespace tpb {

int sm_count();

constexpr int ROUTER_MAX_PER_LANE = 8;  // experts per lane -> up to 256 experts

struct ArgMax {
  float v;
  int i;
};
__device__ __forceinline__ ArgMax warp_argmax(float v, int i) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, v, o);
    const int oi = __shfl_xor_sync(0xffffffffu, i, o);
    if (ov > v || (ov == v && oi < i)) { v = ov; i = oi; }
  }
  return {v, i};
}
__device__ __forceinline__ float warp_sum_f(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// One warp per token.  Expert e lives in register e / 32 of lane e % 32.
//   mode 0: p = softmax(logits); top-k of p; weights renormalised to sum 1 (if norm_topk).
//   mode 1: s = sigmoid(logits); selection score = s + bias, restricted to the topk_group
//           groups with the largest (sum of top-2 selection scores); weights = s at the
//           selected experts, normalised (if norm_topk) and multiplied by `scale`.
// (The bias may be bf16, as a model keeps it: a conversion was a launch of its own, and one that breaks the chain of launches.)
template <typename T>
__global__ void router_topk_kernel(const T* __restrict__ logits, const void* __restrict__ bias, int bias_bf16,
                                   float* __restrict__ w_out, int* __restrict__ idx_out,
                                   float* __restrict__ scores_out, int tokens, int E, int K, int mode, int n_group,
                                   int topk_group, int norm_topk, float scale) {
  if (!chain_begin()) return;
  const int lane = threadIdx.x & 31;
  const int per_lane = (E + 31) / 32;
  for (int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < tokens; t += (gridDim.x * blockDim.x) >> 5) {
    float s[ROUTER_MAX_PER_LANE], sel[ROUTER_MAX_PER_LANE];
    float mx = -INFINITY;
#pragma unroll
    for (int j = 0; j < ROUTER_MAX_PER_LANE; ++j) {
      const int e = j * 32 + lane;
      float x = -INFINITY;
      if (j < per_lane && e < E) x = (float)logits[(long long)t * E + e];
      s[j] = x;
      mx = fmaxf(mx, x);
    }
    if (mode == 0) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      float sum = 0.f;
#pragma unroll
      for (int j = 0; j < ROUTER_MAX_PER_LANE; ++j) {
        s[j] = (s[j] == -INFINITY) ? 0.f : __expf(s[j] - mx);
        sum += s[j];
      }
      sum = warp_sum_f(sum);
      const float inv = 1.f / sum;
#pragma unroll
      for (int j = 0; j < ROUTER_MAX_PER_LANE; ++j) {
        s[j] *= inv;
        const int e = j * 32 + lane;
        sel[j] = (j < per_lane && e < E) ? s[j] : -INFINITY;
      }
    } else {
#pragma unroll
      for (int j = 0; j < ROUTER_MAX_PER_LANE; ++j) {
        const int e = j * 32 + lane;
        const bool ok = j < per_lane && e < E;
        s[j] = ok ? 1.f / (1.f + __expf(-s[j])) : 0.f;
        sel[j] = -INFINITY;
        if (ok)
          sel[j] = s[j] + (!bias ? 0.f
                           : bias_bf16 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(bias)[e])
                                       : reinterpret_cast<const float*>(bias)[e]);
      }
      if (n_group > 1) {
        const int gs = E / n_group;
        float gscore = -INFINITY;  // lane g keeps the score of group g
        for (int g = 0; g < n_group; ++g) {
          float best = -INFINITY;
          int besti = 0x7fffffff;
#pragma unroll
          for (int j = 0; j < ROUTER_MAX_PER_LANE; ++j) {
            const int e = j * 32 + lane;
            if (j < per_lane && e < E && e / gs == g && sel[j] > best) { best = sel[j]; besti = e; }
          }
          const ArgMax a1 = warp_argmax(best, besti);
          float second = -INFINITY;
          int secondi = 0x7fffffff;
#pragma unroll
          for (int j = 0; j < ROUTER_MAX_PER_LANE; ++j) {
            const int e = j * 32 + lane;
            if (j < per_lane && e < E && e / gs == g && e != a1.i && sel[j] > second) { second = sel[j]; secondi = e; }
          }
          const ArgMax a2 = warp_argmax(second, secondi);
          const float sc = a1.v + (gs > 1 ? a2.v : 0.f);
          if (lane == g) gscore = sc;
        }
        unsigned keep_groups = 0;
        for (int r = 0; r < topk_group; ++r) {
          const ArgMax a = warp_argmax(gscore, lane);
          keep_groups |= 1u << a.i;
          if (lane == a.i) gscore = -INFINITY;
        }
#pragma unroll
        for (int j = 0; j < ROUTER_MAX_PER_LANE; ++j) {
          const int e = j * 32 + lane;
          if (j < per_lane && e < E && !((keep_groups >> (e / gs)) & 1u)) sel[j] = 0.f;
        }
      }
    }
    if (scores_out) {
#pragma unroll
      for (int j = 0; j < ROUTER_MAX_PER_LANE; ++j) {
        const int e = j * 32 + lane;
        if (j < per_lane && e < E) scores_out[(long long)t * E + e] = s[j];
      }
    }
    // top-k by repeated warp arg-max (ties go to the lower expert index)
    float wsum = 0.f;
    float my_w = 0.f;   // lane r keeps the r-th weight
    int my_i = 0;
    for (int r = 0; r < K; ++r) {
      float best = -INFINITY;
      int besti = 0x7fffffff;
#pragma unroll
      for (int j = 0; j < ROUTER_MAX_PER_LANE; ++j) {
        const int e = j * 32 + lane;
        if (j < per_lane && e < E && (sel[j] > best || (sel[j] == best && e < besti))) { best = sel[j]; besti = e; }
      }
      const ArgMax a = warp_argmax(best, besti);
      float val = 0.f;
#pragma unroll
      for (int j = 0; j < ROUTER_MAX_PER_LANE; ++j) {
        const int e = j * 32 + lane;
        if (e == a.i) { val = s[j]; sel[j] = -INFINITY; }
      }
      val = warp_sum_f(val);   // only the owning lane contributed
      wsum += val;
      if (lane == r) { my_w = val; my_i = a.i; }
    }
    float norm = 1.f;
    if (norm_topk) norm = (mode == 0) ? 1.f / wsum : 1.f / (wsum + 1e-20f);
    if (lane < K) {
      w_out[(long long)t * K + lane] = my_w * norm * scale;
      idx_out[(long long)t * K + lane] = my_i;
    }
  }
}

// Gradient of the routing weights (and of the scores, when dscores is given) with respect to the logits.
// One warp per token, experts laid out over the lanes as above; the K selected experts' terms are found by
// comparing indices, so there is no gather or scatter.  As a dozen torch operators over [T, E] this was
// launch-bound (about 35 us for 1500 x 64 logits, 3.5 us here).  The scores are rederived to the last fp32 bit or
// two: this file is compiled with fast exponentials and divisions, whose error grows with the logit (35 ulp at -30), so the
// exponential is the 64-bit one and divisions are rounded ones.
template <typename T>
__global__ void router_bwd_kernel(const T* __restrict__ logits, const int* __restrict__ idx,
                                  const float* __restrict__ dw, const float* __restrict__ dscores,
                                  T* __restrict__ dlogits, int tokens, int E, int K, int mode, int norm_topk,
                                  float scale) {
  if (!chain_begin()) return;
  const int lane = threadIdx.x & 31;
  for (int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < tokens; t += (gridDim.x * blockDim.x) >> 5) {
    float s[ROUTER_MAX_PER_LANE], ds[ROUTER_MAX_PER_LANE];
    float mx = -INFINITY;
#pragma unroll
    for (int j = 0; j < ROUTER_MAX_PER_LANE; ++j) {
      const int e = j * 32 + lane;
      s[j] = e < E ? (float)logits[(long long)t * E + e] : -INFINITY;
      mx = fmaxf(mx, s[j]);
    }
    if (mode == 0) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      float sum = 0.f;
#pragma unroll
      for (int j = 0; j < ROUTER_MAX_PER_LANE; ++j) {
        s[j] = s[j] == -INFINITY ? 0.f : (float)exp((double)s[j] - mx);
        sum += s[j];
      }
      sum = warp_sum_f(sum);
#pragma unroll
      for (int j = 0; j < ROUTER_MAX_PER_LANE; ++j) s[j] = __fdiv_rn(s[j], sum);
    } else {
#pragma unroll
      for (int j = 0; j < ROUTER_MAX_PER_LANE; ++j) 
        s[j] = s[j] == -INFINITY ? 0.f : __frcp_rn(1.f + (float)exp(-(double)s[j]));
    }
#pragma unroll
    for (int j = 0; j < ROUTER_MAX_PER_LANE; ++j) {
      const int e = j * 32 + lane;
      ds[j] = (dscores && e < E) ? dscores[(long long)t * E + e] : 0.f;
    }
    if (dw) {
      // w_r = scale * s_r / W with W = sum of the selected scores (or 1); dL/ds_r = scale * (dw_r - c) / W
      const int my_i = lane < K ? idx[(long long)t * K + lane] : -1;
      const float my_d = lane < K ? dw[(long long)t * K + lane] : 0.f;
      float sel = 0.f, dot = 0.f;      // this lane's share of W and of sum dw_r s_r
      for (int r = 0; r < K; ++r) {
        const int e = __shfl_sync(0xffffffffu, my_i, r);
        const float d = __shfl_sync(0xffffffffu, my_d, r);
#pragma unroll
        for (int j = 0; j < ROUTER_MAX_PER_LANE; ++j)
          if (j * 32 + lane == e) { sel += s[j]; dot += d * s[j]; }
      }
      float inv_w = 1.f, c = 0.f;
      if (norm_topk) {
        inv_w = __frcp_rn(warp_sum_f(sel) + (mode == 0 ? 0.f : 1e-20f));
        c = warp_sum_f(dot) * inv_w;
      }
      for (int r = 0; r < K; ++r) {
        const int e = __shfl_sync(0xffffffffu, my_i, r);
        const float d = __shfl_sync(0xffffffffu, my_d, r);
#pragma unroll
        for (int j = 0; j < ROUTER_MAX_PER_LANE; ++j)
          if (j * 32 + lane == e) ds[j] += scale * (d - c) * inv_w;
      }
    }
    float mean = 0.f;
    if (mode == 0) {
#pragma unroll
      for (int j = 0; j < ROUTER_MAX_PER_LANE; ++j) mean += s[j] * ds[j];
      mean = warp_sum_f(mean);
    }
#pragma unroll
    for (int j = 0; j < ROUTER_MAX_PER_LANE; ++j) {
      const int e = j * 32 + lane;
      if (e < E) dlogits[(long long)t * E + e] = (T)(mode == 0 ? s[j] * (ds[j] - mean) : ds[j] * s[j] * (1.f - s[j]));
    }
  }
}

// out[r, :] = (src_row[r] >= 0) ? scale[r] * x[src_row[r], :] : 0       (rows of 16-byte vectors)
// PAD false: padding rows are left unwritten (for readers that ignore them).
template <bool PAD>
__global__ void moe_gather_kernel(const uint4* __restrict__ x, const int* __restrict__ src_row,
                                  const float* __restrict__ row_scale, uint4* __restrict__ out, long long rows,
                                  int nvec) {
  if (!chain_begin()) return;
  const long long total = rows * nvec;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const long long r = i / nvec;
    const int c = (int)(i % nvec);
    const int src = src_row[r];
    if (!PAD && src < 0) continue;
    uint4 v = make_uint4(0, 0, 0, 0);
    if (src >= 0) {
      v = x[(long long)src * nvec + c];
      if (row_scale) {
        const float sc = row_scale[r];
        float2 a = unpack_bf16(v.x), b = unpack_bf16(v.y), cc = unpack_bf16(v.z), d = unpack_bf16(v.w);
        v = make_uint4(pack_bf16(a.x * sc, a.y * sc), pack_bf16(b.x * sc, b.y * sc), pack_bf16(cc.x * sc, cc.y * sc),
                       pack_bf16(d.x * sc, d.y * sc));
      }
    }
    out[i] = v;
  }
}

// out[t, :] = sum_k w[t,k] * rows[dest[t,k], :]   (dest < 0: dropped pair; w null: weight 1)
// The rows of KA pairs of a thread are on their way together: eight where there are fewer threads than the machine holds (a decode
// step's four tokens of six experts 9.3 -> 7.3 us with its launch, 300 tokens 11.3 -> 9.3), one where the others hide
// the wait and registers count (4096 tokens, two experts 26.7 us; 31.8 with eight), and for one pair (16 tokens of 5120 2.7 -> 2.2).
template <int KA>
__global__ void moe_combine_kernel(const uint4* __restrict__ rows, const int* __restrict__ dest,
                                   const float* __restrict__ w, uint4* __restrict__ out, long long tokens, int K,
                                   int nvec) {
  if (!chain_begin()) return;
  const long long total = tokens * nvec;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const long long t = i / nvec;
    const int c = (int)(i % nvec);
    float acc[8] = {};
    auto add = [&](int k, const uint4& v) {
      const float wk = w ? w[t * K + k] : 1.f;
      const float2 a = unpack_bf16(v.x), b = unpack_bf16(v.y), cc = unpack_bf16(v.z), d = unpack_bf16(v.w);
      acc[0] += wk * a.x; acc[1] += wk * a.y; acc[2] += wk * b.x; acc[3] += wk * b.y;
      acc[4] += wk * cc.x; acc[5] += wk * cc.y; acc[6] += wk * d.x; acc[7] += wk * d.y;
    };
    if (KA == 1) {
      for (int k = 0; k < K; ++k) {
        const int r = dest[t * K + k];
        if (r < 0) continue;
        add(k, rows[(long long)r * nvec + c]);
      }
    } else {
      for (int k0 = 0; k0 < K; k0 += KA) {
        int r[KA];
        uint4 v[KA];
#pragma unroll
        for (int k = 0; k < KA; ++k) r[k] = k0 + k < K ? dest[t * K + k0 + k] : -1;
#pragma unroll
        for (int k = 0; k < KA; ++k)
          if (r[k] >= 0) v[k] = rows[(long long)r[k] * nvec + c];
#pragma unroll
        for (int k = 0; k < KA; ++k)
          if (r[k] >= 0) add(k0 + k, v[k]);
      }
    }
    out[i] = make_uint4(pack_bf16(acc[0], acc[1]), pack_bf16(acc[2], acc[3]), pack_bf16(acc[4], acc[5]),
                        pack_bf16(acc[6], acc[7]));
  }
}

// dw[t,k] = <rows[dest[t,k], :], dout[t, :]>     (one warp per (t,k) pair)
__global__ void moe_combine_dw_kernel(const uint4* __restrict__ rows, const int* __restrict__ dest,
                                      const uint4* __restrict__ dout, float* __restrict__ dw, long long pairs, int K,
                                      int nvec) {
  if (!chain_begin()) return;
  const int lane = threadIdx.x & 31;
  for (long long pr = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5; pr < pairs;
       pr += ((long long)gridDim.x * blockDim.x) >> 5) {
    const int r = dest[pr];
    float acc = 0.f;
    if (r >= 0) {
      const long long t = pr / K;
#pragma unroll 4
      for (int c = lane; c < nvec; c += 32) {
        const uint4 a = rows[(long long)r * nvec + c], b = dout[t * nvec + c];
        float2 a0 = unpack_bf16(a.x), a1 = unpack_bf16(a.y), a2 = unpack_bf16(a.z), a3 = unpack_bf16(a.w);
        float2 b0 = unpack_bf16(b.x), b1 = unpack_bf16(b.y), b2 = unpack_bf16(b.z), b3 = unpack_bf16(b.w);
        acc += a0.x * b0.x + a0.y * b0.y + a1.x * b1.x + a1.y * b1.y + a2.x * b2.x + a2.y * b2.y + a3.x * b3.x +
               a3.y * b3.y;
      }
    }
    acc = warp_sum_f(acc);
    if (lane == 0) dw[pr] = acc;
  }
}

static inline int grid_for_items(long long items, int threads, int waves = 8) {
  long long blocks = (items + threads - 1) / threads;
  const long long cap = (long long)sm_count() * waves;
  if (blocks > cap) blocks = cap;
  return blocks < 1 ? 1 : (int)blocks;
}


// ----------------------------------------------------------------------------
// Variable-size all-to-all of rows over NVLink, done by this GPU's own stores (expert-parallel
// dispatch and return).  Rows [src_start[r], src_start[r+1]) of `src` go to rank r's receive buffer,
// starting at row dst_row0[r] there; plain 16-byte stores to peer memory (posted writes).  When the
// last CTA has finished, the flag "rank `me` has delivered" is raised in every rank's flag array.
// ----------------------------------------------------------------------------
struct A2APushParams {
  const uint4* src;
  int vec_per_row;
  int n_rows;
  int world, me;
  int src_start[9];
  long long dst_row0[8];
  uint4* dst[8];
  unsigned* flags[8];
  unsigned epoch;
  unsigned* done_counter;   // one zero-initialised word of local memory
};

__global__ void a2a_push_kernel(const A2APushParams p) {
  for (int row = blockIdx.x; row < p.n_rows; row += gridDim.x) {
    int r = 0;
    while (r + 1 < p.world && row >= p.src_start[r + 1]) ++r;
    const uint4* s = p.src + (long long)row * p.vec_per_row;
    uint4* d = p.dst[r] + (p.dst_row0[r] + (row - p.src_start[r])) * p.vec_per_row;
    for (int i = threadIdx.x; i < p.vec_per_row; i += blockDim.x) d[i] = s[i];
  }
  __threadfence_system();
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned prev = atomicAdd(p.done_counter, 1u);
    if (prev == gridDim.x - 1) {          // every CTA's stores are fenced: publish
      __threadfence_system();
      for (int r = 0; r < p.world; ++r)
        asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(p.flags[r] + p.me), "r"(p.epoch) : "memory");
      *p.done_counter = 0;
    }
  }
}

// ----------------------------------------------------------------------------
// Dispatch plan: a stable counting sort of the (token, slot) pairs by expert into 128-row padded
// segments, in one CTA or, for many pairs, in a cluster of them.  Every warp owns a contiguous range of pairs; sweep 1 counts
// per (warp, expert), a prefix over CTAs and warps gives each warp its first row in every expert's segment, sweep 2
// walks the range again and hands out rows in order (match_any groups equal experts inside a
// warp, the lane order breaks ties), so the result does not depend on scheduling.
// Bound by latency: a sweep's steps follow one another, and one CTA took nine of them for 9000 pairs (64 experts: 25 us; a cluster
// of eight 10 us).
// Outputs: counts[E], k_offsets[E+1] (multiples of `align`), dest[n] (row of each pair), src_row[M]
// (token feeding a row), src_pair[M] (pair feeding a row; both -1 in padding rows) and
// tile_expert[M / tile] (-1 past the last segment), tile = min(align, 128) rows.
// ----------------------------------------------------------------------------
constexpr int PLAN_THREADS = 1024;
constexpr int PLAN_MAX_E = 256;
constexpr int PLAN_CLUSTER = 8;

__global__ void __launch_bounds__(PLAN_THREADS, 1)
moe_plan_kernel(const int* __restrict__ idx, int n, int K, int E, int M, int align, int* __restrict__ counts,
                int* __restrict__ k_offsets, int* __restrict__ dest, int* __restrict__ src_row,
                long long* __restrict__ src_pair, int* __restrict__ tile_expert) {
  if (!chain_begin()) return;
  __shared__ int wcount[32][PLAN_MAX_E];     // sweep 1: pairs of (warp, expert); sweep 2: next row
  __shared__ int off_pad[PLAN_MAX_E + 1];
  __shared__ int own_s[PLAN_MAX_E];          // pairs of this CTA per expert, read by the others of the cluster
  __shared__ int total_s[PLAN_MAX_E];
  __shared__ int scan[PLAN_MAX_E / 32];
  const int ctas = gridDim.x, rank = blockIdx.x;               // one cluster
  const int tile_log = 31 - __clz(min(align, 128));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int gtid = rank * PLAN_THREADS + threadIdx.x, gthreads = ctas * PLAN_THREADS;
  for (int e = lane; e < E; e += 32) wcount[warp][e] = 0;
  __syncwarp();
  const int warps = 32 * ctas, gwarp = rank * 32 + warp;
  const int per_warp = ((n + warps - 1) / warps + 31) / 32 * 32;      // multiple of 32 so that lanes stay aligned
  const int lo = (int)min((long long)n, (long long)gwarp * per_warp), hi = (int)min((long long)n, (long long)lo + per_warp);
  for (int base = lo; base < hi; base += 32) {
    const int i = base + lane;
    const int e = i < hi ? idx[i] : -1;
    const bool ok = e >= 0 && e < E;
    const unsigned m = __match_any_sync(0xffffffffu, ok ? e : -1);
    if (ok && (m & ((1u << lane) - 1)) == 0) wcount[warp][e] += __popc(m);
    __syncwarp();
  }
  __syncthreads();
  int own = 0, before = 0, total = 0;        // of expert threadIdx.x: this CTA's pairs, those of the CTAs in front, all
  if (threadIdx.x < E) {
#pragma unroll 8
    for (int w = 0; w < 32; ++w) own += wcount[w][threadIdx.x];
    own_s[threadIdx.x] = own;
  }
  if (ctas > 1) {
    cluster_sync_all();
    if (threadIdx.x < E) {
      const uint32_t at = smem_u32(own_s + threadIdx.x);
#pragma unroll
      for (int r = 0; r < PLAN_CLUSTER; ++r) {
        int v;
        asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(map_to_cta(at, r)) : "memory");
        if (r < rank) before += v;
        total += v;
      }
    }
  } else {
    total = own;
  }
  // padded segments: a scan over the experts, 32 to a warp (align and tile are powers of two)
  int pad = 0, start = 0;
  if (threadIdx.x < PLAN_MAX_E) {
    pad = threadIdx.x < E ? (total + align - 1) & ~(align - 1) : 0;
    int sum = pad;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, sum, o);
      if (lane >= o) sum += v;
    }
    if (lane == 31) scan[warp] = sum;
    start = sum - pad;
  }
  __syncthreads();
  if (threadIdx.x < E) {
    for (int w = 0; w < warp; ++w) start += scan[w];
    const int end = start + pad;
    off_pad[threadIdx.x] = start;
    total_s[threadIdx.x] = total;
    if (threadIdx.x == E - 1) off_pad[E] = end;
    if (rank == 0) {
      counts[threadIdx.x] = total;
      k_offsets[threadIdx.x] = start;
      if (threadIdx.x == E - 1) k_offsets[E] = end;
      for (int t = start >> tile_log; t < end >> tile_log; ++t) tile_expert[t] = threadIdx.x;
    }
    int run = start + before;
#pragma unroll 8
    for (int w = 0; w < 32; ++w) {
      const int c = wcount[w][threadIdx.x];
      wcount[w][threadIdx.x] = run;
      run += c;
    }
  }
  __syncthreads();
  for (int t = (off_pad[E] >> tile_log) + gtid; t < M >> tile_log; t += gthreads) tile_expert[t] = -1;
  // padding rows: the end of every expert's segment (one warp per expert) and everything past the last
  // one (filled here and not by memsets of the whole arrays: three launches fewer)
  for (int e = gwarp; e < E; e += warps) {
    for (int r = off_pad[e] + total_s[e] + lane; r < off_pad[e + 1]; r += 32) {
      src_row[r] = -1;
      src_pair[r] = -1;
    }
  }
  for (int r = off_pad[E] + gtid; r < M; r += gthreads) {
    src_row[r] = -1;
    src_pair[r] = -1;
  }
  for (int base = lo; base < hi; base += 32) {
    const int i = base + lane;
    const int e = i < hi ? idx[i] : -1;
    const bool ok = e >= 0 && e < E;
    const unsigned m = __match_any_sync(0xffffffffu, ok ? e : -1);
    int pos = -1;
    if (ok) pos = wcount[warp][e] + __popc(m & ((1u << lane) - 1));
    __syncwarp();
    if (ok && (m & ((1u << lane) - 1)) == 0) wcount[warp][e] += __popc(m);
    __syncwarp();
    if (i < hi) dest[i] = pos;
    if (ok) {
      src_row[pos] = i / K;
      src_pair[pos] = i;
    }
  }
  __syncwarp();
  if (ctas > 1) cluster_leave();             // own_s is read by the others until here
}

// Block form of the push: the source rows are a sequence of `n_blocks` contiguous blocks, block b =
// rows [start[b], start[b+1]) going to rank dst_rank[b] at row dst_row0[b] of its receive buffer.
// The descriptors live in device memory as 64-bit words: start[n_blocks + 1], dst_rank[n_blocks],
// dst_row0[n_blocks].  One block per (destination rank, expert) lets rows land at the receiver
// already grouped by expert, whatever rank they came from.
struct A2ABlocksParams {
  const uint4* src;
  int vec_per_row;
  int n_rows;
  int n_blocks;
  int world, me;
  const long long* desc;
  uint4* dst[8];
  unsigned* flags[8];
  unsigned epoch;
  unsigned* done_counter;
};

__global__ void a2a_push_blocks_kernel(const A2ABlocksParams p) {
  extern __shared__ long long a2a_desc[];
  const int nd = 3 * p.n_blocks + 1;
  for (int i = threadIdx.x; i < nd; i += blockDim.x) a2a_desc[i] = p.desc[i];
  __syncthreads();
  const long long* start = a2a_desc;
  const long long* dst_rank = a2a_desc + p.n_blocks + 1;
  const long long* dst_row0 = dst_rank + p.n_blocks;
  for (int row = blockIdx.x; row < p.n_rows; row += gridDim.x) {
    int lo = 0, hi = p.n_blocks - 1;                    // last block whose first row is <= row
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (start[mid] <= row) lo = mid; else hi = mid - 1;
    }
    const int r = (int)dst_rank[lo];
    if (r < 0 || r >= p.world) continue;
    const uint4* s = p.src + (long long)row * p.vec_per_row;
    uint4* d = p.dst[r] + (dst_row0[lo] + (row - start[lo])) * p.vec_per_row;
    for (int i = threadIdx.x; i < p.vec_per_row; i += blockDim.x) d[i] = s[i];
  }
  __threadfence_system();
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned prev = atomicAdd(p.done_counter, 1u);
    if (prev == gridDim.x - 1) {
      __threadfence_system();
      for (int r = 0; r < p.world; ++r)
        asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(p.flags[r] + p.me), "r"(p.epoch) : "memory");
      *p.done_counter = 0;
    }
  }
}

// Stream-ordered wait (bounded) until every rank has delivered its rows for `epoch`.
__global__ void a2a_wait_kernel(const unsigned* flags, int world, unsigned epoch, int* status) {
  if (threadIdx.x != 0) return;
  for (int r = 0; r < world; ++r) {
    long long t0 = 0;
    int spins = 0;
    while (true) {
      unsigned v;
      asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(flags + r) : "memory");
      if (v == epoch) break;
      if (++spins == 64) {
        spins = 0;
        if (t0 == 0) t0 = clock64();
        else if (clock64() - t0 > kSpinBudgetCycles) { report(status, kTimeoutPeerFlag, 61); return; }
        __nanosleep(200);
      }
    }
  }
}

// ----------------------------------------------------------------------------
// Gradients of fp32 logits y = x w^T (x [T,K], w [N,K] bf16, dy [T,N] fp32), N of a router's size: products and sums in fp32
// on the FMA pipe, one rounding to bf16.  As library products each operand was first copied to fp32 and each result from it: 72 us
// for 1500 tokens, 64 experts, K = 2048, of which these take 33.  Bound by FMA issue: 0.2 G of them each.
// ----------------------------------------------------------------------------
// dx = dy w.  A CTA makes 64 rows x 128 columns, a warp eight rows, a thread 8 x 4; dy is read as broadcasts.
constexpr int RG_THREADS = 256, RG_ROWS = 64, RG_COLS = 128, RG_STEP = 64;
__global__ void __launch_bounds__(RG_THREADS)
logit_dx_kernel(const float* __restrict__ dy, const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ dx, int T, int N,
                int K, long long ldw) {
  if (!chain_begin()) return;
  __shared__ __align__(16) float sdy[RG_ROWS][RG_STEP + 4];
  __shared__ __align__(16) __nv_bfloat16 sw[RG_STEP][RG_COLS];
  const int t0 = blockIdx.x * RG_ROWS, c0 = blockIdx.y * RG_COLS;   // (only a grid's first dimension holds any number of rows)
  const int lane = threadIdx.x & 31, r0 = (threadIdx.x >> 5) * 8;
  float acc[8][4] = {};
  for (int n0 = 0; n0 < N; n0 += RG_STEP) {
    if (n0) __syncthreads();
    for (int i = threadIdx.x; i < RG_ROWS * RG_STEP; i += RG_THREADS) {
      const int r = i / RG_STEP, n = i % RG_STEP;
      sdy[r][n] = t0 + r < T && n0 + n < N ? dy[(size_t)(t0 + r) * N + n0 + n] : 0.f;
    }
    for (int i = threadIdx.x; i < RG_STEP * RG_COLS / 8; i += RG_THREADS) {
      const int n = i / (RG_COLS / 8), c = i % (RG_COLS / 8) * 8;
      uint4 v = make_uint4(0, 0, 0, 0);       // (K is a multiple of 8)
      if (n0 + n < N && c0 + c < K) v = *reinterpret_cast<const uint4*>(w + (size_t)(n0 + n) * ldw + c0 + c);
      *reinterpret_cast<uint4*>(&sw[n][c]) = v;
    }
    __syncthreads();
#pragma unroll 4
    for (int n = 0; n < RG_STEP; n += 4) {
      float4 d[8];
#pragma unroll
      for (int r = 0; r < 8; ++r) d[r] = *reinterpret_cast<const float4*>(&sdy[r0 + r][n]);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const uint2 u = *reinterpret_cast<const uint2*>(&sw[n + e][lane * 4]);
        const float2 a = unpack_bf16(u.x), b = unpack_bf16(u.y);
#pragma unroll
        for (int r = 0; r < 8; ++r) {
          const float x = e == 0 ? d[r].x : e == 1 ? d[r].y : e == 2 ? d[r].z : d[r].w;
          acc[r][0] = fmaf(x, a.x, acc[r][0]);
          acc[r][1] = fmaf(x, a.y, acc[r][1]);
          acc[r][2] = fmaf(x, b.x, acc[r][2]);
          acc[r][3] = fmaf(x, b.y, acc[r][3]);
        }
      }
    }
  }
  const int c = c0 + lane * 4;
  if (c >= K) return;
#pragma unroll
  for (int r = 0; r < 8; ++r)
    if (t0 + r0 + r < T)
      *reinterpret_cast<uint2*>(dx + (size_t)(t0 + r0 + r) * K + c) =
          make_uint2(pack_bf16(acc[r][0], acc[r][1]), pack_bf16(acc[r][2], acc[r][3]));
}

// dw = dy^T x.  64 x 64 results to a cluster of eight CTAs, each adding up an eighth of the tokens (a thread 4 x 4); the eight sums of a
// result meet in distributed shared memory and are added in rank order.
constexpr int RG_SPLIT = 8, RG_TOK = 32, RG_TILE = 64;
__global__ void __launch_bounds__(RG_THREADS)
logit_dw_kernel(const float* __restrict__ dy, const __nv_bfloat16* __restrict__ x, __nv_bfloat16* __restrict__ dw, int T, int N,
                int K, long long ldx) {
  if (!chain_begin()) return;
  __shared__ __align__(16) float sdy[RG_TOK][RG_TILE];
  __shared__ __align__(16) float sx[RG_TOK][RG_TILE];
  __shared__ __align__(16) float part[RG_TILE][RG_TILE];
  const int rank = (int)cluster_ctarank();
  const int c0 = (int)(blockIdx.x / RG_SPLIT) * RG_TILE, n0 = blockIdx.y * RG_TILE;
  const int per = (T + RG_SPLIT - 1) / RG_SPLIT, t_begin = rank * per, t_end = min(T, t_begin + per);
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  float acc[4][4] = {};
  float dreg[RG_TOK * RG_TILE / RG_THREADS];
  uint4 xreg = make_uint4(0, 0, 0, 0);
  const int xt = threadIdx.x / (RG_TILE / 8), xc = threadIdx.x % (RG_TILE / 8) * 8;
  auto fetch = [&](int t0) {
#pragma unroll
    for (int i = 0; i < RG_TOK * RG_TILE / RG_THREADS; ++i) {
      const int at = i * RG_THREADS + (int)threadIdx.x, t = t0 + at / RG_TILE, n = n0 + at % RG_TILE;
      dreg[i] = t < t_end && n < N ? dy[(size_t)t * N + n] : 0.f;
    }
    xreg = make_uint4(0, 0, 0, 0);
    if (t0 + xt < t_end && c0 + xc < K) xreg = *reinterpret_cast<const uint4*>(x + (size_t)(t0 + xt) * ldx + c0 + xc);
  };
  fetch(t_begin);
  for (int t0 = t_begin; t0 < t_end; t0 += RG_TOK) {
    __syncthreads();
#pragma unroll
    for (int i = 0; i < RG_TOK * RG_TILE / RG_THREADS; ++i) (&sdy[0][0])[i * RG_THREADS + threadIdx.x] = dreg[i];
    const float2 a = unpack_bf16(xreg.x), b = unpack_bf16(xreg.y), c = unpack_bf16(xreg.z), d = unpack_bf16(xreg.w);
    *reinterpret_cast<float4*>(&sx[xt][xc]) = make_float4(a.x, a.y, b.x, b.y);
    *reinterpret_cast<float4*>(&sx[xt][xc + 4]) = make_float4(c.x, c.y, d.x, d.y);
    __syncthreads();
    fetch(t0 + RG_TOK);
#pragma unroll 8
    for (int t = 0; t < RG_TOK; ++t) {
      const float4 g = *reinterpret_cast<const float4*>(&sdy[t][ty * 4]), v = *reinterpret_cast<const float4*>(&sx[t][tx * 4]);
      const float gg[4] = {g.x, g.y, g.z, g.w}, vv[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(gg[i], vv[j], acc[i][j]);
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
    *reinterpret_cast<float4*>(&part[ty * 4 + i][tx * 4]) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
  cluster_sync_all();
  // this CTA's eight of the 64 rows, two columns to a thread
  const int n = rank * (RG_TILE / RG_SPLIT) + (int)threadIdx.x / (RG_TILE / 2), c = (int)threadIdx.x % (RG_TILE / 2) * 2;
  if (n0 + n < N && c0 + c < K) {   // (around the loads too: one whose result is not stored could still be under way at the end)
    float s0 = 0.f, s1 = 0.f;
#pragma unroll
    for (int r = 0; r < RG_SPLIT; ++r) {
      float a, b;
      asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(a), "=f"(b) : "r"(map_to_cta(smem_u32(&part[n][c]), r)) : "memory");
      s0 += a; s1 += b;
    }
    *reinterpret_cast<uint32_t*>(dw + (size_t)(n0 + n) * K + c0 + c) = pack_bf16(s0, s1);
  }
  __syncwarp();
  cluster_leave();           // nobody's shared memory goes away while a neighbour reads it
}

}  // namespace tpb

using namespace tpb;

// Gradients of y = x w^T with fp32 y (tpb_linear_f32): dx [T,K], dw [N,K] bf16, contiguous (either may be null); dy contiguous.
extern "C" int tpb_linear_f32_bwd(const float* dy, const void* x, const void* w, void* dx, void* dw, int T, int N, int K,
                                  long long ldx, long long ldw, void* stream) {
  if (T <= 0 || N <= 0 || K <= 0) return -2;
  if (K % 8 || ldx % 8 || ldw % 8 || (K + RG_COLS - 1) / RG_COLS > 65535 || (N + RG_TILE - 1) / RG_TILE > 65535) return -2;
  for (const void* p : {x, w, (const void*)dx, (const void*)dw})
    if (reinterpret_cast<uintptr_t>(p) % 16) return -2;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (dx)
    chain(logit_dx_kernel, dim3((T + RG_ROWS - 1) / RG_ROWS, (K + RG_COLS - 1) / RG_COLS), RG_THREADS, 0, s, dy,
          (const __nv_bfloat16*)w, (__nv_bfloat16*)dx, T, N, K, ldw);
  if (dw)
    chain_clusters(logit_dw_kernel, RG_SPLIT, dim3(RG_SPLIT * ((K + RG_TILE - 1) / RG_TILE), (N + RG_TILE - 1) / RG_TILE), RG_THREADS, 0,
                   s, dy, (const __nv_bfloat16*)x, (__nv_bfloat16*)dw, T, N, K, ldx);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : 1000 + (int)e;
}
#define STREAM(s) reinterpret_cast<cudaStream_t>(s)
static inline int rc_of(cudaError_t e) { return e == cudaSuccess ? 0 : 1000 + (int)e; }

extern "C" int tpb_router_topk(const void* logits, int bf16, const void* bias, float* w_out, int* idx_out,
                               float* scores_out, int tokens, int E, int K, int mode, int n_group, int topk_group,
                               int norm_topk, float scale, void* stream) {
  if (E > 32 * ROUTER_MAX_PER_LANE || K > 32 || K > E || E <= 0) return -2;
  if (mode == 1 && n_group > 1 && (E % n_group || n_group > 32 || topk_group > n_group)) return -2;
  if (tokens <= 0) return 0;
  const int grid = grid_for_items((long long)tokens * 32, 256);
  const int bias_bf16 = (bf16 >> 1) & 1;
  if (bf16 & 1)
    chain(router_topk_kernel<__nv_bfloat16>, grid, 256, 0, STREAM(stream),
          (const __nv_bfloat16*)logits, bias, bias_bf16, w_out, idx_out, scores_out, tokens, E, K, mode, n_group, topk_group,
        norm_topk, scale);
  else
    chain(router_topk_kernel<float>, grid, 256, 0, STREAM(stream), (const float*)logits, bias, bias_bf16, w_out, idx_out, scores_out,
                                                                tokens, E, K, mode, n_group, topk_group, norm_topk,
                                                                scale);
  return rc_of(cudaGetLastError());
}

// dw [tokens, K] or null, dscores [tokens, E] or null; dlogits has the type of logits.
extern "C" int tpb_router_bwd(const void* logits, int logits_is_bf16, const int* idx, const float* dw,
                              const float* dscores, void* dlogits, int tokens, int E, int K, int mode, int norm_topk,
                              float scale, void* stream) {
  if (E > 32 * ROUTER_MAX_PER_LANE || K > 32 || K > E || E <= 0) return -2;
  if (tokens <= 0) return 0;
  const int grid = grid_for_items((long long)tokens * 32, 256);
  if (logits_is_bf16)
    chain(router_bwd_kernel<__nv_bfloat16>, grid, 256, 0, STREAM(stream),
          (const __nv_bfloat16*)logits, idx, dw, dscores, (__nv_bfloat16*)dlogits, tokens, E, K, mode, norm_topk, scale);
  else
    chain(router_bwd_kernel<float>, grid, 256, 0, STREAM(stream), (const float*)logits, idx, dw, dscores, (float*)dlogits,
                                                               tokens, E, K, mode, norm_topk, scale);
  return rc_of(cudaGetLastError());
}

extern "C" int tpb_moe_gather(const void* x, const int* src_row, const float* row_scale, void* out, long long rows,
                              int dim, void* stream) {
  if (dim % 8) return -2;
  if (rows <= 0) return 0;
  chain(moe_gather_kernel<true>, grid_for_items(rows * (dim / 8), 256), 256, 0, STREAM(stream),
        (const uint4*)x, src_row, row_scale, (uint4*)out, rows, dim / 8);
  return rc_of(cudaGetLastError());
}

// The same without a scale and without writing the padding rows.
extern "C" int tpb_moe_gather_real(const void* x, const int* src_row, void* out, long long rows, int dim,
                                   void* stream) {
  if (dim % 8) return -2;
  if (rows <= 0) return 0;
  chain(moe_gather_kernel<false>, grid_for_items(rows * (dim / 8), 256), 256, 0, STREAM(stream),
        (const uint4*)x, src_row, nullptr, (uint4*)out, rows, dim / 8);
  return rc_of(cudaGetLastError());
}

extern "C" int tpb_moe_combine(const void* rows, const int* dest, const float* w, void* out, long long tokens, int K,
                               int dim, void* stream) {
  if (dim % 8) return -2;
  if (tokens <= 0) return 0;
  const long long items = tokens * (dim / 8);
  if (K > 1 && items <= 512LL * sm_count())
    chain(moe_combine_kernel<8>, grid_for_items(items, 256), 256, 0, STREAM(stream), (const uint4*)rows, dest, w, (uint4*)out, tokens,
          K, dim / 8);
  else
    chain(moe_combine_kernel<1>, grid_for_items(items, 256), 256, 0, STREAM(stream), (const uint4*)rows, dest, w, (uint4*)out, tokens,
          K, dim / 8);
  return rc_of(cudaGetLastError());
}

extern "C" int tpb_moe_combine_dw(const void* rows, const int* dest, const void* dout, float* dw, long long tokens,
                                  int K, int dim, void* stream) {
  if (dim % 8) return -2;
  if (tokens <= 0) return 0;
  chain(moe_combine_dw_kernel, grid_for_items(tokens * K * 32, 256), 256, 0, STREAM(stream),
        (const uint4*)rows, dest, (const uint4*)dout, dw, tokens * K, K, dim / 8);
  return rc_of(cudaGetLastError());
}

// src: [n_rows, dim] bf16 rows sorted by destination rank; src_start[world + 1] row offsets of the
// blocks; dst_row0[r]: first row of this rank's block in rank r's receive buffer dst[r]; flags[r]:
// rank r's flag array (one word per source rank); done_counter: a zero-initialised local word.
extern "C" int tpb_a2a_push_rows(const void* src, int n_rows, int dim, int world, int me, const int* src_start,
                                 const long long* dst_row0, void* const* dst, unsigned* const* flags, unsigned epoch,
                                 unsigned* done_counter, void* stream) {
  if (dim % 8 || world < 1 || world > 8 || me < 0 || me >= world) return -2;
  A2APushParams p{};
  p.src = (const uint4*)src; p.vec_per_row = dim / 8; p.n_rows = n_rows; p.world = world; p.me = me;
  for (int r = 0; r <= world; ++r) p.src_start[r] = src_start[r];
  for (int r = 0; r < world; ++r) {
    p.dst_row0[r] = dst_row0[r];
    p.dst[r] = (uint4*)dst[r];
    p.flags[r] = flags[r];
  }
  p.epoch = epoch; p.done_counter = done_counter;
  int grid = n_rows < 1 ? 1 : (n_rows < 4 * sm_count() ? n_rows : 4 * sm_count());
  a2a_push_kernel<<<grid, 256, 0, STREAM(stream)>>>(p);
  return rc_of(cudaGetLastError());
}

// idx [tokens, K] int32 (entries outside [0, E) are dropped: dest = -1).  align: 16, 32, 128 or 256 rows per
// segment step.  rows = static row count of the padded layout, a multiple of align that holds n pairs and
// align - 1 padding rows for every expert that can be hit.  Everything is on the device; no host read.
extern "C" int tpb_moe_plan(const int* idx, int tokens, int K, int E, int rows, int align, int* counts, int* k_offsets,
                            int* dest, int* src_row, long long* src_pair, int* tile_expert, void* stream) {
  if (E < 1 || E > PLAN_MAX_E || K < 1 || tokens < 0 || rows < 0) return -2;
  if ((align != 16 && align != 32 && align != 128 && align != 256) || rows % align) return -2;
  const long long n = (long long)tokens * K;
  if (n > (1LL << 30) || rows < n + (long long)(align - 1) * (n < E ? n : E)) return -2;
  // (a cluster's launch and exchange cost what two or three sweep steps do)
  const int ctas = n > 1536 ? PLAN_CLUSTER : 1;
  chain_clusters(moe_plan_kernel, ctas, ctas, PLAN_THREADS, 0, STREAM(stream), idx, (int)n, K, E, rows, align, counts, k_offsets, dest,
                 src_row, src_pair, tile_expert);
  return rc_of(cudaGetLastError());
}

extern "C" int tpb_a2a_push_blocks(const void* src, int n_rows, int dim, int n_blocks, int world, int me,
                                   const long long* desc_dev, void* const* dst, unsigned* const* flags,
                                   unsigned epoch, unsigned* done_counter, void* stream) {
  if (dim % 8 || world < 1 || world > 8 || me < 0 || me >= world || n_blocks < 1 || n_blocks > 1024 || !desc_dev)
    return -2;
  A2ABlocksParams p{};
  p.src = (const uint4*)src; p.vec_per_row = dim / 8; p.n_rows = n_rows; p.n_blocks = n_blocks;
  p.world = world; p.me = me; p.desc = desc_dev;
  for (int r = 0; r < world; ++r) {
    p.dst[r] = (uint4*)dst[r];
    p.flags[r] = flags[r];
  }
  p.epoch = epoch; p.done_counter = done_counter;
  int grid = n_rows < 1 ? 1 : (n_rows < 4 * sm_count() ? n_rows : 4 * sm_count());
  a2a_push_blocks_kernel<<<grid, 256, (3 * n_blocks + 1) * sizeof(long long), STREAM(stream)>>>(p);
  return rc_of(cudaGetLastError());
}

extern "C" int tpb_a2a_wait(const unsigned* flags, int world, unsigned epoch, void* stream) {
  a2a_wait_kernel<<<1, 32, 0, STREAM(stream)>>>(flags, world, epoch, status_block());
  return rc_of(cudaGetLastError());
}
