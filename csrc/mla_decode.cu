// One decode step of latent attention over a compressed cache (one new token per sequence).
//
// The cache holds, per token, the normalised latent (C values) and the shared rotary key (R values), both
// bf16.  The key up-projection is folded into the query and the value up-projection is applied to the
// weighted sum, so a step has to read C + R numbers per cached token and the up-projection weights once.
// All arithmetic is that of fp32 on bf16 inputs (queries folded through the up-projection and the weights of the sum stay
// fp32, as three bf16 terms where the tensor cores take them): what bounds the step is latency and launches.
// Written as torch operators the same step converts the whole cache and the up-projection to fp32 and
// runs about thirty kernels per layer, 150 us and the host's time for them.  A decode step of four sequences of 1500 cached
// tokens through three layers (16 heads, C = 512, the whole model's step): 372 us with fp32 multiply-adds in the split kernel
// and every CTA of the merge kernel merging all latent columns, 315 this way.
//
//   mla_prep_kernel     per sequence: rotate the queries' rotary part, normalise the new latent and rotate
//                       the new rotary key straight into the cache
//   mla_fold_kernel     qa[b,h,:] = sum_d q[b,h,d] Wk[h,d,:]               (reads Wk once)
//   mla_split_kernel    per (sequence, 16 heads, range of keys): scores, running softmax, weighted latent sum
//   mla_merge_kernel    per (sequence, head): merge the ranges, out[j] = sum_c olat[c] Wv[h,j,c]

#include "common.cuh"
#include "tpb.h"

namespace tpb {

int sm_count();

constexpr int MLA_MAX_C = 512;      // latent width: two columns per thread of 256
constexpr int MLA_R = 64;           // rotary width
constexpr int MLA_HG = 16;          // heads per CTA of the split kernel
constexpr int MLA_KEYS = 32;        // keys per step of the split kernel: one per lane
constexpr int MLA_THREADS = 256;
constexpr int MLA_MAX_B = 8;        // sequences per CTA of the fold kernel

__device__ __forceinline__ float mla_rbf(float v) { return __bfloat162float(__float2bfloat16(v)); }

// Rotation of pair i of a rotary slice; interleaved pairs (2i, 2i+1) stay where they are.
__device__ __forceinline__ void mla_rotate(const __nv_bfloat16* x, __nv_bfloat16* y, int i, int interleaved, float cs,
                                           float sn) {
  const int ia = interleaved ? 2 * i : i, ib = interleaved ? 2 * i + 1 : i + MLA_R / 2;
  const float a = __bfloat162float(x[ia]), b = __bfloat162float(x[ib]);
  y[ia] = __float2bfloat16(a * cs - b * sn);
  y[ib] = __float2bfloat16(b * cs + a * sn);
}

// One CTA per sequence.  q [B, H * (dn + R)] is rotated in place; ckv [B, C + R] goes to row `pos` of
// the caches [B, S, C] and [B, S, R].
__global__ void __launch_bounds__(MLA_THREADS)
mla_prep_kernel(__nv_bfloat16* __restrict__ q, const __nv_bfloat16* __restrict__ ckv,
                const __nv_bfloat16* __restrict__ norm_w, const float* __restrict__ cosT,
                const float* __restrict__ sinT, __nv_bfloat16* __restrict__ kv_cache,
                __nv_bfloat16* __restrict__ pe_cache, long long kv_bs, long long pe_bs, int pos, int H, int dn, int C,
                float eps, int interleaved) {
  if (!chain_begin()) return;
  __shared__ float red[8];
  const int b = blockIdx.x;
  const float* cs = cosT + (size_t)pos * (MLA_R / 2);
  const float* sn = sinT + (size_t)pos * (MLA_R / 2);
  const __nv_bfloat16* row = ckv + (size_t)b * (C + MLA_R);
  // the latent and its weight are asked for first: their sum is the longest way through this kernel
  constexpr int PER = MLA_MAX_C / MLA_THREADS;
  float v[PER], nw[PER], ss = 0.f;
#pragma unroll
  for (int k = 0; k < PER; ++k) {
    const int i = threadIdx.x + k * MLA_THREADS;
    v[k] = i < C ? __bfloat162float(row[i]) : 0.f;
    nw[k] = i < C ? __bfloat162float(norm_w[i]) : 0.f;
  }
  for (int i = threadIdx.x; i < H * (MLA_R / 2); i += MLA_THREADS) {
    const int h = i / (MLA_R / 2), j = i % (MLA_R / 2);
    __nv_bfloat16* x = q + ((size_t)b * H + h) * (dn + MLA_R) + dn;
    mla_rotate(x, x, j, interleaved, cs[j], sn[j]);
  }
  if (threadIdx.x < MLA_R / 2)
    mla_rotate(row + C, pe_cache + b * pe_bs + (size_t)pos * MLA_R, threadIdx.x, interleaved, cs[threadIdx.x],
               sn[threadIdx.x]);
#pragma unroll
  for (int k = 0; k < PER; ++k) ss += v[k] * v[k];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
  __syncthreads();
  ss = 0.f;
#pragma unroll
  for (int w = 0; w < 8; ++w) ss += red[w];
  const float rstd = rsqrtf(ss / (float)C + eps);
  // the same two roundings as the norm kernel of the other paths
#pragma unroll
  for (int k = 0; k < PER; ++k) {
    const int i = threadIdx.x + k * MLA_THREADS;
    if (i < C) kv_cache[b * kv_bs + (size_t)pos * C + i] = __float2bfloat16(nw[k] * mla_rbf(v[k] * rstd));
  }
}

// Grid (H, C / 64, ceil(B / 8)).  A thread holds 8 columns of every 32nd d: its 16-byte loads of the weight
// (four for dn = 128) are all in flight at once; the 32 slices meet by shuffles and in shared memory.  (With
// 4-byte loads, sixteen per thread one after the other, 10 us instead of 5 at B = 4, H = 16.)
__global__ void __launch_bounds__(MLA_THREADS)
mla_fold_kernel(const __nv_bfloat16* __restrict__ q, const __nv_bfloat16* __restrict__ w, float* __restrict__ qa, int B,
                int H, int dn, int dv, int C) {
  if (!chain_begin()) return;
  __shared__ float acc_s[8][MLA_MAX_B][64];
  extern __shared__ float fold_q[];                  // [MLA_MAX_B][dn]
  const int h = blockIdx.x, c0 = blockIdx.y * 64, b0 = blockIdx.z * MLA_MAX_B;
  const int nb = min(MLA_MAX_B, B - b0);
  const int vec = threadIdx.x & 7, slice = threadIdx.x >> 3;
  const uint4* wr = reinterpret_cast<const uint4*>(w + (size_t)h * (dn + dv) * C + c0) + vec;
  uint4 wv[4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
    if (slice + 32 * i < dn) wv[i] = wr[(size_t)(slice + 32 * i) * (C / 8)];
  for (int i = threadIdx.x; i < MLA_MAX_B * dn; i += MLA_THREADS) {
    const int b = i / dn, d = i % dn;
    fold_q[i] = b < nb ? __bfloat162float(q[((size_t)(b0 + b) * H + h) * (dn + MLA_R) + d]) : 0.f;
  }
  __syncthreads();
  float a[MLA_MAX_B][8] = {};
  auto add = [&](const uint4& u, int d) {
    const float2 p0 = unpack_bf16(u.x), p1 = unpack_bf16(u.y), p2 = unpack_bf16(u.z), p3 = unpack_bf16(u.w);
#pragma unroll
    for (int b = 0; b < MLA_MAX_B; ++b) {
      if (b >= nb) break;
      const float x = fold_q[b * dn + d];
      a[b][0] += x * p0.x; a[b][1] += x * p0.y; a[b][2] += x * p1.x; a[b][3] += x * p1.y;
      a[b][4] += x * p2.x; a[b][5] += x * p2.y; a[b][6] += x * p3.x; a[b][7] += x * p3.y;
    }
  };
#pragma unroll
  for (int i = 0; i < 4; ++i)
    if (slice + 32 * i < dn) add(wv[i], slice + 32 * i);
  for (int d = slice + 128; d < dn; d += 32) add(wr[(size_t)d * (C / 8)], d);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int b = 0; b < MLA_MAX_B; ++b) {
    if (b >= nb) break;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      float v = a[b][e];
      v += __shfl_xor_sync(0xffffffffu, v, 8);
      v += __shfl_xor_sync(0xffffffffu, v, 16);
      if (lane < 8) acc_s[warp][b][vec * 8 + e] = v;
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < nb * 64; i += MLA_THREADS) {
    const int b = i / 64, c = i % 64;
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) s += acc_s[k][b][c];
    qa[((size_t)(b0 + b) * H + h) * C + c0 + c] = s;
  }
}

struct MlaSplitSmem {
  // rows of queries and keys are padded by 16 bytes: 8 rows of 16 bytes at one column touch every bank once
  static __host__ __device__ int pitch(int C) { return (C + MLA_R) * 2 + 16; }
  static constexpr int SROW = MLA_KEYS + 8;       // floats per head in the score and weight arrays
  static __host__ __device__ int bytes(int C) {
    return (3 * MLA_HG + MLA_KEYS) * pitch(C) + 3 * MLA_HG * SROW * 4 + MLA_HG * 4;
  }
};

// x as three bf16 terms, x = hi + mid + lo to 2^-24; two values to a register.
__device__ __forceinline__ void split3(float a, float b, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  hi = pack_bf16(a, b);
  const float2 h = unpack_bf16(hi);
  const float ra = a - h.x, rb = b - h.y;
  mid = pack_bf16(ra, rb);
  const float2 m = unpack_bf16(mid);
  lo = pack_bf16(ra - m.x, rb - m.y);
}
__device__ __forceinline__ void ldsm4(uint32_t addr, uint32_t* r) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm4_t(uint32_t addr, uint32_t* r) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
// d += A (16 x 16) B (16 x 8), bf16 operands
__device__ __forceinline__ void mma16816(float* d, const uint32_t* a, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Grid (ranges, head groups, B).  Keys [range * per, min(n_keys, (range + 1) * per)), per a multiple of 32.
// part_o [B, H, ranges, C], part_ml [B, H, ranges, 2] = (running maximum in log2 units, sum).
//
// Sixteen heads are one row block of mma.sync m16n8k16 (a tcgen05 tile would be seven eighths empty): scores from the
// queries as three bf16 terms, the weighted sum from the weights as three, so that nothing of the fp32 values is lost, and
// every 16-deep product starts from zero and is added to its sum in fp32 (the tensor core's own sums are cut, not rounded).
// Bound by latency: the first keys are brought to L2 before the kernel in front has ended.
__global__ void __launch_bounds__(MLA_THREADS, 2)
mla_split_kernel(const float* __restrict__ qa, const __nv_bfloat16* __restrict__ q,
                 const __nv_bfloat16* __restrict__ kv_cache, const __nv_bfloat16* __restrict__ pe_cache,
                 long long kv_bs, long long pe_bs, float* __restrict__ part_o, float* __restrict__ part_ml, int n_keys,
                 int per, int H, int dn, int C, float scale_log2) {
  extern __shared__ __align__(16) uint8_t split_smem[];
  constexpr int SROW = MlaSplitSmem::SROW;
  const int D = C + MLA_R, pitch = MlaSplitSmem::pitch(C), plane = MLA_HG * pitch;
  uint8_t* sq = split_smem;                                         // [3 terms][16 heads][pitch]
  uint8_t* sk = sq + 3 * plane;                                     // [32 keys][pitch]
  float* ss = reinterpret_cast<float*>(sk + MLA_KEYS * pitch);      // [2 halves of D][16][SROW] scores
  float* sp = ss + 2 * MLA_HG * SROW;                               // [16][SROW] weights
  float* s_alpha = sp + MLA_HG * SROW;                              // [16]
  const int range = blockIdx.x, h0 = blockIdx.y * MLA_HG, b = blockIdx.z, ranges = gridDim.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int k_begin = range * per, k_end = min(n_keys, k_begin + per);
  const int cv = C / 8, dvec = D / 8;
  const uint32_t sk_at = smem_u32(sk), sq_at = smem_u32(sq);
  chain_launch();
  // The first keys move to L2 while the fold kernel runs (a line each; they are read after the wait).
  for (int i = threadIdx.x; i < MLA_KEYS * (C / 64 + 1); i += MLA_THREADS) {
    const int r = i / (C / 64 + 1), c = i - r * (C / 64 + 1), key = min(k_begin + r, k_end - 1);
    const __nv_bfloat16* at = c < C / 64 ? kv_cache + b * kv_bs + (size_t)key * C + c * 64 : pe_cache + b * pe_bs + (size_t)key * MLA_R;
    asm volatile("prefetch.global.L2 [%0];" ::"l"(at));
  }
  if (!chain_wait()) return;
  auto fetch_keys = [&](int k0) {                // asynchronous; keys past the range are zeros
    for (int i = threadIdx.x; i < MLA_KEYS * dvec; i += MLA_THREADS) {
      const int r = i / dvec, c = i - r * dvec, key = min(k0 + r, k_end - 1);
      const void* src = c < cv ? (const void*)(kv_cache + b * kv_bs + (size_t)key * C + c * 8)
                               : (const void*)(pe_cache + b * pe_bs + (size_t)key * MLA_R + (c - cv) * 8);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(sk_at + r * pitch + c * 16), "l"(src),
                   "r"(k0 + r < k_end ? 16 : 0)
                   : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  fetch_keys(k_begin);
  for (int i = threadIdx.x; i < MLA_HG * (MLA_R / 4); i += MLA_THREADS) {     // the rotary parts: bf16 as they are
    const int h = i / (MLA_R / 4), d = (i % (MLA_R / 4)) * 4;
    uint2 u = make_uint2(0, 0);
    if (h0 + h < H) u = *reinterpret_cast<const uint2*>(q + ((size_t)b * H + h0 + h) * (dn + MLA_R) + dn + d);
    *reinterpret_cast<uint2*>(sq + h * pitch + (C + d) * 2) = u;
  }
#pragma unroll 8
  for (int i = threadIdx.x; i < MLA_HG * (C / 4); i += MLA_THREADS) {
    const int h = i / (C / 4), d = (i % (C / 4)) * 4;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (h0 + h < H) v = *reinterpret_cast<const float4*>(qa + ((size_t)b * H + h0 + h) * C + d);
    uint2 hi, mid, lo;
    split3(v.x, v.y, hi.x, mid.x, lo.x);
    split3(v.z, v.w, hi.y, mid.y, lo.y);
    uint8_t* at = sq + h * pitch + d * 2;
    *reinterpret_cast<uint2*>(at) = hi;
    *reinterpret_cast<uint2*>(at + plane) = mid;
    *reinterpret_cast<uint2*>(at + 2 * plane) = lo;
  }
  const int hw = warp * 2;                       // this warp's two heads in the softmax
  float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.f, l1 = 0.f;
  const int g = lane >> 2, t = lane & 3;         // mma fragment row and column pair
  const int nt = warp & 3, half = warp >> 2;     // score phase: eight keys, half of the contraction
  const int ksteps = D / 32;                     // 16-deep steps per half (D is a multiple of 64: an even number)
  const bool owner = warp * 64 < C;              // sum phase: latent columns [64 warp, 64 warp + 64)
  float acc[8][4] = {};
  for (int k0 = k_begin; k0 < k_end; k0 += MLA_KEYS) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    {
      float s[4] = {};
      const uint32_t a_at = sq_at + ((lane & 7) + ((lane >> 3) & 1) * 8) * pitch + (lane >> 4) * 16;
      const uint32_t b_at = sk_at + (nt * 8 + (lane & 7)) * pitch + (lane >> 3) * 16;
#pragma unroll 2
      for (int k = half * ksteps; k < (half + 1) * ksteps; k += 2) {
        uint32_t bb[4];
        ldsm4(b_at + k * 32, bb);                // two steps' keys
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          float d[4] = {};
          const bool rot = (k + e) * 16 >= C;    // the rotary part has one term
#pragma unroll
          for (int term = 2; term >= 0; --term) {
            if (rot && term > 0) continue;
            uint32_t a[4];
            ldsm4(a_at + term * plane + (k + e) * 32, a);
            mma16816(d, a, bb[2 * e], bb[2 * e + 1]);
          }
#pragma unroll
          for (int x = 0; x < 4; ++x) s[x] += d[x];
        }
      }
      float* dst = ss + (half * MLA_HG + g) * SROW + nt * 8 + 2 * t;
      *reinterpret_cast<float2*>(dst) = make_float2(s[0], s[1]);
      *reinterpret_cast<float2*>(dst + 8 * SROW) = make_float2(s[2], s[3]);
    }
    __syncthreads();
    const bool live = k0 + lane < k_end;
    const float s0 = live ? (ss[hw * SROW + lane] + ss[(MLA_HG + hw) * SROW + lane]) * scale_log2 : -INFINITY;
    const float s1 = live ? (ss[(hw + 1) * SROW + lane] + ss[(MLA_HG + hw + 1) * SROW + lane]) * scale_log2 : -INFINITY;
    float n0 = s0, n1 = s1;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      n0 = fmaxf(n0, __shfl_xor_sync(0xffffffffu, n0, o));
      n1 = fmaxf(n1, __shfl_xor_sync(0xffffffffu, n1, o));
    }
    n0 = fmaxf(m0, n0);                          // finite: the step has at least one key
    n1 = fmaxf(m1, n1);
    const float p0 = exp2f(s0 - n0), p1 = exp2f(s1 - n1);
    const float al0 = exp2f(m0 - n0), al1 = exp2f(m1 - n1);
    float t0 = p0, t1 = p1;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      t0 += __shfl_xor_sync(0xffffffffu, t0, o);
      t1 += __shfl_xor_sync(0xffffffffu, t1, o);
    }
    l0 = l0 * al0 + t0; l1 = l1 * al1 + t1;
    m0 = n0; m1 = n1;
    sp[hw * SROW + lane] = p0;
    sp[(hw + 1) * SROW + lane] = p1;
    if (lane == 0) { s_alpha[hw] = al0; s_alpha[hw + 1] = al1; }
    __syncthreads();
    if (owner) {
      uint32_t a[2][3][4];                       // [16 keys][term]
#pragma unroll
      for (int ks = 0; ks < 2; ++ks)
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          const float2 w = *reinterpret_cast<const float2*>(sp + (g + (x & 1) * 8) * SROW + ks * 16 + (x >> 1) * 8 + 2 * t);
          split3(w.x, w.y, a[ks][0][x], a[ks][1][x], a[ks][2][x]);
        }
      const float alg = s_alpha[g], alh = s_alpha[g + 8];
      const uint32_t v_at = sk_at + ((lane & 7) + ((lane >> 3) & 1) * 8) * pitch + (warp * 64 + (lane >> 4) * 8) * 2;
#pragma unroll
      for (int n = 0; n < 8; n += 2) {
        uint32_t v0[4], v1[4];                   // keys 0-15 and 16-31 of two column groups
        ldsm4_t(v_at + n * 16, v0);
        ldsm4_t(v_at + 16 * pitch + n * 16, v1);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          float d[4] = {}, d2[4] = {};
#pragma unroll
          for (int term = 2; term >= 0; --term) {
            mma16816(d, a[0][term], v0[2 * e], v0[2 * e + 1]);
            mma16816(d2, a[1][term], v1[2 * e], v1[2 * e + 1]);
          }
          acc[n + e][0] = acc[n + e][0] * alg + (d[0] + d2[0]);
          acc[n + e][1] = acc[n + e][1] * alg + (d[1] + d2[1]);
          acc[n + e][2] = acc[n + e][2] * alh + (d[2] + d2[2]);
          acc[n + e][3] = acc[n + e][3] * alh + (d[3] + d2[3]);
        }
      }
    }
    if (k0 + MLA_KEYS < k_end) {
      __syncthreads();                           // this step's keys and weights are used up
      fetch_keys(k0 + MLA_KEYS);
    }
  }
  if (owner) {
#pragma unroll
    for (int hh = 0; hh < 2; ++hh) {
      const int h = h0 + g + 8 * hh;
      if (h < H) {
        float* dst = part_o + (((size_t)b * H + h) * ranges + range) * C + warp * 64 + 2 * t;
#pragma unroll
        for (int n = 0; n < 8; ++n)
          *reinterpret_cast<float2*>(dst + n * 8) = make_float2(acc[n][2 * hh], acc[n][2 * hh + 1]);
      }
    }
  }
  if (lane == 0) {
    if (h0 + hw < H) {
      float* ml = part_ml + (((size_t)b * H + h0 + hw) * ranges + range) * 2;
      ml[0] = m0; ml[1] = l0;
    }
    if (h0 + hw + 1 < H) {
      float* ml = part_ml + (((size_t)b * H + h0 + hw + 1) * ranges + range) * 2;
      ml[0] = m1; ml[1] = l1;
    }
  }
}

// Grid (H, B, slices of `rows` outputs), in clusters of `share` slices.  Every range holds at least one key, so its sum is
// positive and its maximum finite.  The CTAs of a cluster merge C / share latent columns each and read the others' from
// their shared memory (each merging all of them, the ranges' partial sums were read four times over.)
// EARLY: everything that comes from memory is asked for at once: the weight rows of a warp, the first partial sums and the
// ranges' maxima.  (One after the other, each waiting for the one before, a decode step of three layers took 294 us;
// this way, with the norms' weights and the residuals asked for early too, 281.)  It takes 128 registers for 39, which pays while the
// CTAs all run at once; with more of them, three times as many an SM matter more: us a step, early / late, 16 sequences of 128
// heads over 30 keys 174 / 119, 64 of 16 heads 93 / 69.
template <bool EARLY>
__global__ void __launch_bounds__(MLA_THREADS)
mla_merge_kernel(const float* __restrict__ part_o, const float* __restrict__ part_ml, const __nv_bfloat16* __restrict__ w,
                 __nv_bfloat16* __restrict__ out, int ranges, int H, int dn, int dv, int C, int rows, int share) {
  if (!chain_begin()) return;
  __shared__ __align__(16) float olat[MLA_MAX_C];
  __shared__ float2 sums[MLA_THREADS];
  extern __shared__ float merge_w[];             // [ranges]
  const int h = blockIdx.x, b = blockIdx.y;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const float* ml = part_ml + ((size_t)b * H + h) * ranges * 2;
  const int rank = share > 1 ? (int)cluster_ctarank() : 0;
  const int cols = C / share, pairs = cols / 2;      // this CTA's columns, two to a thread
  const int groups = MLA_THREADS / pairs;            // threads with the same columns take every groups-th range
  const int pr = threadIdx.x % pairs, grp = threadIdx.x / pairs;
  const uint4* wv = reinterpret_cast<const uint4*>(w + ((size_t)h * (dn + dv) + dn) * C);
  const int cv = C / 8;
  const int j0 = blockIdx.z * rows, j1 = min(dv, j0 + rows);
  constexpr int WK = MLA_MAX_C / 8 / 32, AHEAD = EARLY ? 12 : 0;
  uint4 wr[EARLY ? WK : 1][4];
  auto load_part = [&](int j, int k, uint4 (&to)[4]) {
#pragma unroll
    for (int r = 0; r < 4; ++r)
      to[r] = (lane + 32 * k < cv && j + r < j1) ? wv[(size_t)(j + r) * cv + lane + 32 * k] : make_uint4(0, 0, 0, 0);
  };
  auto load_rows = [&](int j) {
#pragma unroll
    for (int k = 0; k < WK; ++k) load_part(j, k, wr[EARLY ? k : 0]);
  };
  if (EARLY) load_rows(j0 + 4 * warp);
  const float* po = part_o + ((size_t)b * H + h) * ranges * C + rank * cols + 2 * pr;
  float2 ahead[AHEAD > 0 ? AHEAD : 1];
#pragma unroll
  for (int i = 0; i < AHEAD; ++i) {
    const int r = grp + i * groups;
    if (grp < groups && r < ranges) ahead[i] = *reinterpret_cast<const float2*>(po + (size_t)r * C);
  }
  if (warp == 0) {
    float m = -INFINITY;
    for (int r = lane; r < ranges; r += 32) m = fmaxf(m, ml[2 * r]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    float l = 0.f;
    for (int r = lane; r < ranges; r += 32) {
      const float e = exp2f(ml[2 * r] - m);
      merge_w[r] = e;
      l += e * ml[2 * r + 1];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
    const float inv = 1.f / l;
    for (int r = lane; r < ranges; r += 32) merge_w[r] *= inv;
  }
  __syncthreads();
  {
    float x = 0.f, y = 0.f;
    if (grp < groups) {
#pragma unroll
      for (int i = 0; i < AHEAD; ++i) {
        const int r = grp + i * groups;
        if (r < ranges) {
          x += merge_w[r] * ahead[i].x;
          y += merge_w[r] * ahead[i].y;
        }
      }
#pragma unroll 8
      for (int r = grp + AHEAD * groups; r < ranges; r += groups) {
        const float2 v = *reinterpret_cast<const float2*>(po + (size_t)r * C);
        x += merge_w[r] * v.x;
        y += merge_w[r] * v.y;
      }
    }
    sums[threadIdx.x] = make_float2(x, y);
    __syncthreads();
    if ((int)threadIdx.x < pairs) {
      for (int k = 1; k < groups; ++k) { x += sums[k * pairs + pr].x; y += sums[k * pairs + pr].y; }
      olat[rank * cols + 2 * pr] = x;
      olat[rank * cols + 2 * pr + 1] = y;
    }
  }
  if (share > 1) {
    cluster_sync_all();
    for (int c = threadIdx.x; c < C; c += MLA_THREADS)
      if (c / cols != rank) {
        float v;
        asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(map_to_cta(smem_u32(olat + c), c / cols)) : "memory");
        olat[c] = v;
      }
    cluster_sync_all();                              // (nobody leaves or reads on while a neighbour still reads here)
  } else {
    __syncthreads();
  }
  // a warp takes four rows at a time: their loads are in flight together
  for (int j = j0 + 4 * warp; j < j1; j += 4 * (MLA_THREADS / 32)) {
    if (EARLY && j != j0 + 4 * warp) load_rows(j);
    float s[4] = {};
#pragma unroll
    for (int k = 0; k < WK; ++k) {
      const int c = lane + 32 * k;
      if (!EARLY) load_part(j, k, wr[0]);
      const uint4* v = wr[EARLY ? k : 0];
      if (c < cv) {
        const float4 x0 = *reinterpret_cast<const float4*>(olat + c * 8), x1 = *reinterpret_cast<const float4*>(olat + c * 8 + 4);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const float2 a = unpack_bf16(v[r].x), bb = unpack_bf16(v[r].y), cc = unpack_bf16(v[r].z), d = unpack_bf16(v[r].w);
          s[r] += x0.x * a.x + x0.y * a.y + x0.z * bb.x + x0.w * bb.y + x1.x * cc.x + x1.y * cc.y + x1.z * d.x + x1.w * d.y;
        }
      }
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s[r] += __shfl_xor_sync(0xffffffffu, s[r], o);
      if (lane == 0 && j + r < j1) out[((size_t)b * H + h) * dv + j + r] = __float2bfloat16(s[r]);
    }
  }
}

}  // namespace tpb

using namespace tpb;

// Ranges of keys the split kernel uses for `n_keys` cached tokens: one step of 32 keys each until the
// machine holds two CTAs per SM, then longer ranges.
extern "C" int tpb_mla_decode_ranges(int B, int H, int n_keys) {
  if (B < 1 || H < 1 || n_keys < 1) return 0;
  const long long groups = (long long)B * ((H + MLA_HG - 1) / MLA_HG);
  const int steps = (n_keys + MLA_KEYS - 1) / MLA_KEYS;
  long long want = 2LL * sm_count() / groups;
  if (want < 1) want = 1;
  const int per = (int)((steps + want - 1) / want);
  return (steps + per - 1) / per;
}

// q [B, H * (dn + 64)] (rotated in place), ckv [B, C + 64], w = kv_b_proj [H * (dn + dv), C], out [B, H * dv], all
// contiguous bf16; the new token goes to row `pos` of the caches (rows C and 64 wide, kv_bs / pe_bs
// elements between sequences) and attends to rows 0 .. pos.  qa: B*H*C floats; part_o: B*H*ranges*C;
// part_ml: B*H*ranges*2, with ranges = tpb_mla_decode_ranges(B, H, pos + 1).
extern "C" int tpb_mla_decode(void* q, const void* ckv, const void* norm_w, const float* cosT, const float* sinT,
                              void* kv_cache, void* pe_cache, long long kv_bs, long long pe_bs, const void* w, void* out,
                              float* qa, float* part_o, float* part_ml, int B, int H, int dn, int dv, int C, int R,
                              int pos, float scale, float eps, int interleaved, int ranges, void* stream_) {
  if (R != MLA_R || C % 64 || C > MLA_MAX_C || C < 64 || dn < 8 || dn % 8 || dn > 512 || dv < 1 || dv > 4096 || H < 1 || pos < 0) return -2;
  if (kv_bs % 8 || pe_bs % 8 || B > 65535) return -2;
  for (const void* a : {(const void*)q, ckv, norm_w, (const void*)kv_cache, (const void*)pe_cache, w, (const void*)out})
    if (reinterpret_cast<uintptr_t>(a) % 16) return -2;
  if (B <= 0) return 0;
  const int n_keys = pos + 1;
  if (ranges != tpb_mla_decode_ranges(B, H, n_keys)) return -2;
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  auto* qb = reinterpret_cast<__nv_bfloat16*>(q);
  auto* kc = reinterpret_cast<__nv_bfloat16*>(kv_cache);
  auto* pc = reinterpret_cast<__nv_bfloat16*>(pe_cache);
  const auto* wb = reinterpret_cast<const __nv_bfloat16*>(w);
  chain(mla_prep_kernel, B, MLA_THREADS, 0, stream, qb, reinterpret_cast<const __nv_bfloat16*>(ckv),
                                                 reinterpret_cast<const __nv_bfloat16*>(norm_w), cosT, sinT, kc, pc,
                                                 kv_bs, pe_bs, pos, H, dn, C, eps, interleaved);
  chain(mla_fold_kernel, dim3(H, C / 64, (B + MLA_MAX_B - 1) / MLA_MAX_B), MLA_THREADS, MLA_MAX_B * dn * 4, stream,
        qb, wb, qa, B, H, dn, dv, C);
  const int steps = (n_keys + MLA_KEYS - 1) / MLA_KEYS;
  const int per = (steps + ranges - 1) / ranges * MLA_KEYS;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(mla_split_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         MlaSplitSmem::bytes(MLA_MAX_C));
    if (e != cudaSuccess) return 1000 + (int)e;
    configured = true;
  }
  chain(mla_split_kernel, dim3(ranges, (H + MLA_HG - 1) / MLA_HG, B), MLA_THREADS, MlaSplitSmem::bytes(C), stream,
        qa, qb, kc, pc, kv_bs, pe_bs, part_o, part_ml, n_keys, per, H, dn, C, scale * 1.4426950408889634f);
  const int rows = 32;     // one pass of the eight warps
  const int slices = (dv + rows - 1) / rows, share = slices % 4 == 0 ? 4 : slices % 2 == 0 ? 2 : 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(H, B, slices);
  cfg.blockDim = dim3(MLA_THREADS, 1, 1);
  cfg.dynamicSmemBytes = ranges * 4;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = 1;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = share;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  const bool early = (long long)H * B * slices <= 2 * sm_count();     // (128 registers: two CTAs per SM)
  cudaLaunchKernelEx(&cfg, early ? mla_merge_kernel<true> : mla_merge_kernel<false>, (const float*)part_o, (const float*)part_ml, wb,
                     reinterpret_cast<__nv_bfloat16*>(out), ranges, H, dn, dv, C, rows, share);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : 1000 + (int)e;
}
