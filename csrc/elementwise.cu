// Bandwidth-bound kernels of the training step: RMSNorm (+residual) fwd/bwd, RoPE,
// SwiGLU, softmax cross-entropy (fused forward + gradient), embedding gather /
// scatter-add, fused AdamW and the gradient-norm reduction.  All of them move
// 16-byte vectors, keep a row in registers between its passes and run on grids
// sized from the SM count.

#include "common.cuh"
#include "tpb.h"

namespace tpb {

int sm_count();

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
// Block-wide sum; `red` is 32 floats of shared memory.  All threads get the result.
__device__ __forceinline__ float block_sum(float v, float* red) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) red[w] = v;
  __syncthreads();
  float t = lane < nw ? red[lane] : 0.f;
  return warp_sum(t);
}
__device__ __forceinline__ float block_max(float v, float* red) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_max(v);
  __syncthreads();
  if (lane == 0) red[w] = v;
  __syncthreads();
  float t = lane < nw ? red[lane] : -INFINITY;
  return warp_max(t);
}

__device__ __forceinline__ void unpack8(const uint4& u, float* f) {
  float2 a = unpack_bf16(u.x), b = unpack_bf16(u.y), c = unpack_bf16(u.z), d = unpack_bf16(u.w);
  f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y; f[4] = c.x; f[5] = c.y; f[6] = d.x; f[7] = d.y;
}
__device__ __forceinline__ uint4 pack8(const float* f) {
  return make_uint4(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]), pack_bf16(f[4], f[5]), pack_bf16(f[6], f[7]));
}
// bf16 rounding of a float (keeps fp32 type) so results match torch's bf16 ops
__device__ __forceinline__ float rbf(float x) { return __bfloat162float(__float2bfloat16(x)); }

// ----------------------------------------------------------------------------
// RMSNorm
// ----------------------------------------------------------------------------
constexpr int NORM_THREADS = 256;
constexpr int NORM_VPT = 4;  // most 16-byte vectors kept in registers per thread (dim <= 8192)
// The kernels are instantiated for 1, 2 and 4 vectors per thread: a 4096-wide row needs two, and
// the instantiation that holds exactly that many leaves registers for more resident CTAs, which
// is what a latency-bound row-per-CTA kernel needs to fill the memory pipe.
// EARLY: the weight is asked for with the row and not behind its sum.  That is for few rows, where the chain of loads is all there is
// (16 rows of 4096: 2.6 -> 2.4 us); its registers cost resident CTAs (8192 rows of 4096 with a residual 49 -> 60 us, 2048 wide 25 ->
// 32.5), but for rows of more than 4096, which have fewer than that anyway (8192 rows of 8192 with a residual 113 both ways).
template <int VPT, bool EARLY>
__global__ void __launch_bounds__(NORM_THREADS)
rmsnorm_fwd_kernel(const uint4* __restrict__ x, const uint4* __restrict__ res, const uint4* __restrict__ w,
                   uint4* __restrict__ y, uint4* __restrict__ h_out, float* __restrict__ rstd_out, int rows,
                   int nvec, float eps) {
  if (!chain_begin()) return;
  __shared__ float red[32];
  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    const uint4* xr = x + (size_t)row * nvec;
    float vals[VPT][8];
    uint4 wu[VPT];
    float ss = 0.f;
#pragma unroll
    for (int j = 0; j < VPT; ++j) {
      int i = threadIdx.x + j * NORM_THREADS;
      if (i < nvec) {
        if (EARLY) wu[j] = w[i];
        unpack8(xr[i], vals[j]);
        if (res) {
          float r[8];
          unpack8(res[(size_t)row * nvec + i], r);
#pragma unroll
          for (int e = 0; e < 8; ++e) vals[j][e] = rbf(vals[j][e] + r[e]);
          if (h_out) h_out[(size_t)row * nvec + i] = pack8(vals[j]);
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) ss += vals[j][e] * vals[j][e];
      }
    }
    ss = block_sum(ss, red);
    const float rstd = rsqrtf(ss / (float)(nvec * 8) + eps);
    if (threadIdx.x == 0 && rstd_out) rstd_out[row] = rstd;
#pragma unroll
    for (int j = 0; j < VPT; ++j) {
      int i = threadIdx.x + j * NORM_THREADS;
      if (i < nvec) {
        float wv[8], o[8];
        unpack8(EARLY ? wu[j] : w[i], wv);
#pragma unroll
        for (int e = 0; e < 8; ++e) o[e] = wv[e] * rbf(vals[j][e] * rstd);
        y[(size_t)row * nvec + i] = pack8(o);
      }
    }
  }
}

// dx of a vector from o = g - xh * dot, with every rounding said: g = dy * w and xh = x * rstd are products rounded by themselves,
// and the residual's gradient is added to the rounded value or (fused) inside the last multiplication.  Which of the two is what the
// compiler once chose, kept so that a size's gradients stay the same bits: fused in rows above 2048 where a CTA takes a row, and
// in streamed rows for all but the last of the 1, 2 or 4 vectors that a thread of 256 would have.
__device__ __forceinline__ void norm_dx(float (&o)[8], float rs, const uint4* res, bool fused) {
  if (res) {
    float r[8];
    unpack8(*res, r);
#pragma unroll
    for (int e = 0; e < 8; ++e) o[e] = fused ? fmaf(rs, o[e], r[e]) : __fadd_rn(__fmul_rn(rs, o[e]), r[e]);
  } else {
#pragma unroll
    for (int e = 0; e < 8; ++e) o[e] = __fmul_rn(rs, o[e]);
  }
}

template <int VPT>
__global__ void __launch_bounds__(NORM_THREADS)
rmsnorm_bwd_kernel(const uint4* __restrict__ dy, const uint4* __restrict__ x, const uint4* __restrict__ w,
                   const float* __restrict__ rstd, const uint4* __restrict__ dres, uint4* __restrict__ dx,
                   float* __restrict__ dw, int rows, int nvec) {
  if (!chain_begin()) return;
  __shared__ float red[32];
  float dw_acc[VPT][8];
  float wv[VPT][8];
#pragma unroll
  for (int j = 0; j < VPT; ++j) {
    int i = threadIdx.x + j * NORM_THREADS;
#pragma unroll
    for (int e = 0; e < 8; ++e) dw_acc[j][e] = 0.f;
    if (i < nvec) unpack8(w[i], wv[j]);
  }
  const float inv_d = 1.0f / (float)(nvec * 8);
  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    const float rs = rstd[row];
    float g[VPT][8], xh[VPT][8];
    float dot = 0.f;
#pragma unroll
    for (int j = 0; j < VPT; ++j) {
      int i = threadIdx.x + j * NORM_THREADS;
      if (i < nvec) {
        float dyv[8], xv[8];
        unpack8(dy[(size_t)row * nvec + i], dyv);
        unpack8(x[(size_t)row * nvec + i], xv);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          xh[j][e] = __fmul_rn(xv[e], rs);
          dw_acc[j][e] = fmaf(dyv[e], xh[j][e], dw_acc[j][e]);
          g[j][e] = __fmul_rn(dyv[e], wv[j][e]);
          dot = fmaf(g[j][e], xh[j][e], dot);
        }
      }
    }
    dot = block_sum(dot, red) * inv_d;
#pragma unroll
    for (int j = 0; j < VPT; ++j) {
      int i = threadIdx.x + j * NORM_THREADS;
      if (i < nvec) {
        float o[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) o[e] = fmaf(-xh[j][e], dot, g[j][e]);
        norm_dx(o, rs, dres ? dres + (size_t)row * nvec + i : nullptr, VPT > 1);
        dx[(size_t)row * nvec + i] = pack8(o);
      }
    }
  }
  if (dw) {
#pragma unroll
    for (int j = 0; j < VPT; ++j) {
      int i = threadIdx.x + j * NORM_THREADS;
      if (i < nvec) {
        // two 16-byte vector reductions instead of eight scalar atomics
        float* dst = dw + i * 8;
        asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst), "f"(dw_acc[j][0]), "f"(dw_acc[j][1]),
                     "f"(dw_acc[j][2]), "f"(dw_acc[j][3])
                     : "memory");
        asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst + 4), "f"(dw_acc[j][4]),
                     "f"(dw_acc[j][5]), "f"(dw_acc[j][6]), "f"(dw_acc[j][7])
                     : "memory");
      }
    }
  }
}

// ---- Many rows: streamed forms.
// Both directions are bound by memory, and a CTA per row (above) by latency: it loads, reduces over the block, stores and only
// then asks for the next row.  Here rows arrive in shared memory by bulk copies that run ahead, and what works on a row is no
// larger than the row needs, so that no barrier of a whole block stands in its way and several rows of an SM are at
// different points of theirs.
constexpr int NS_MAX_STAGES = 4;
constexpr int NS_SMEM = 200 * 1024;            // rings of one CTA; one CTA per SM
__device__ __forceinline__ void bulk_row_load(void* smem_dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(smem_dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

// The sum of a row in the order of 256 threads: p[w] is what the lanes of their warp w hold, added up over the lanes as warp_sum does
// and over the warps as block_sum does, in twelve shuffles (each halves the number of sums a lane has under way).
__device__ __forceinline__ float sum_of_warps(const float (&p)[8]) {
  const int lane = threadIdx.x & 31;
  float q[4], r[2];
#pragma unroll
  for (int i = 0; i < 4; ++i) q[i] = (lane & 16 ? p[i + 4] : p[i]) + __shfl_xor_sync(0xffffffffu, lane & 16 ? p[i] : p[i + 4], 16);
#pragma unroll
  for (int i = 0; i < 2; ++i) r[i] = (lane & 8 ? q[i + 2] : q[i]) + __shfl_xor_sync(0xffffffffu, lane & 8 ? q[i] : q[i + 2], 8);
  float s = (lane & 4 ? r[1] : r[0]) + __shfl_xor_sync(0xffffffffu, lane & 4 ? r[0] : r[1], 4);
  s += __shfl_xor_sync(0xffffffffu, s, 2);
  s += __shfl_xor_sync(0xffffffffu, s, 1);         // the sum of warp lane / 4 (bits 4, 3, 2)
  s += __shfl_xor_sync(0xffffffffu, s, 16);
  s += __shfl_xor_sync(0xffffffffu, s, 8);
  s += __shfl_xor_sync(0xffffffffu, s, 4);
  return s;
}

// Forward: a warp to a row, the row in its registers (VPL 16-byte vectors a lane), its next rows on their way.  The sum over
// the row is twelve shuffles, in the order of the other forms, so that all give the same bits.  8192 x 4096: 26.7 us (5.0 TB/s), 27.8
// with 256 threads to a row and three barriers; x 3072 20 and 29.
template <int VPL>
__global__ void __launch_bounds__(512)
rmsnorm_fwd_rows_kernel(const uint4* __restrict__ x, const uint4* __restrict__ w, uint4* __restrict__ y,
                        float* __restrict__ rstd_out, int rows, int nvec, float eps, int stages, int* status) {
  if (!chain_begin()) return;
  extern __shared__ uint8_t nf_smem_raw[];
  uint8_t* smem = nf_smem_raw + ((128u - (smem_u32(nf_smem_raw) & 127u)) & 127u);
  const int warp = warp_index(), lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  const uint32_t row_bytes = (uint32_t)nvec * 16u;
  uint64_t* full = reinterpret_cast<uint64_t*>(smem) + warp * NS_MAX_STAGES;
  uint4* sw = reinterpret_cast<uint4*>(smem + 16 * NS_MAX_STAGES * 8);
  uint4* ring = sw + nvec + (size_t)warp * stages * nvec;
  const int first = warp * gridDim.x + blockIdx.x, step = warps * gridDim.x;
  const int mine = first < rows ? (rows - 1 - first) / step + 1 : 0;
  auto issue = [&](int k) {   // one lane
    mbar_expect_tx(&full[k % stages], row_bytes);
    bulk_row_load(ring + (k % stages) * nvec, x + ((size_t)first + (size_t)k * step) * nvec, row_bytes, &full[k % stages]);
  };
  const int ahead = min(stages, mine);
  if (lane == 0) {
    for (int s = 0; s < stages; ++s) mbar_init(&full[s], 1);
    fence_barrier_init();
    for (int i = 0; i < ahead; ++i) issue(i);
  }
  int issued = ahead;
  for (int i = threadIdx.x; i < nvec; i += blockDim.x) sw[i] = w[i];
  __syncthreads();
  int k = 0;
  for (; k < mine; ++k) {
    if (!mbar_wait_warp(&full[k % stages], (uint32_t)(k / stages) & 1u, status, kTimeoutTmaFull, 73)) break;
    const uint4* sx = ring + (k % stages) * nvec;
    uint4 v[VPL];
    float ss[8] = {};           // by warps of 256 threads: vector i is thread i % 256's
#pragma unroll
    for (int j = 0; j < VPL; ++j) {
      const int i = lane + 32 * j;
      if (i < nvec) {
        v[j] = sx[i];
        float f[8];
        unpack8(v[j], f);
#pragma unroll
        for (int e = 0; e < 8; ++e) ss[j & 7] += f[e] * f[e];
      }
    }
    __syncwarp();
    if (lane == 0 && issued < mine) {
      fence_proxy_async();
      issue(issued);
    }
    issued += issued < mine;
    const float rstd = rsqrtf(sum_of_warps(ss) / (float)(nvec * 8) + eps);
    const size_t row = (size_t)first + (size_t)k * step;
    if (lane == 0 && rstd_out) rstd_out[row] = rstd;
#pragma unroll
    for (int j = 0; j < VPL; ++j) {
      const int i = lane + 32 * j;
      if (i < nvec) {
        float f[8], wv[8];
        unpack8(v[j], f);
        unpack8(sw[i], wv);
#pragma unroll
        for (int e = 0; e < 8; ++e) f[e] = wv[e] * rbf(f[e] * rstd);
        y[row * nvec + i] = pack8(f);
      }
    }
  }
  for (; k < issued; ++k)   // a wait ran out: what was asked for still lands here (bounded again)
    mbar_wait_warp(&full[k % stages], (uint32_t)(k / stages) & 1u, status, kTimeoutTmaFull, 74);
}

// Forward of wide rows: 256 threads to a row, three CTAs per SM, each with two rows of shared memory.  (A warp's share of a row of
// 8192 is 1 KB in its registers, and six warps are all that the rings leave room for.)  The weight stays in registers.  The next row
// is asked for when this one has arrived: bound by memory, where more rows under way are slower (8192 x 8192, us: 44, asked
// for a row earlier 45, two 50; 3000 x 8192 18, 18, 18.4).  A stage is handed back by the barrier that opens every iteration, which
// also carries the give-up decision of a wait that ran out.
template <int VPT>
__global__ void __launch_bounds__(NORM_THREADS)
rmsnorm_fwd_wide_kernel(const uint4* __restrict__ x, const uint4* __restrict__ w, uint4* __restrict__ y,
                        float* __restrict__ rstd_out, int rows, int nvec, float eps, int* status) {
  if (!chain_begin()) return;
  extern __shared__ uint8_t nw_smem_raw[];
  uint8_t* smem = nw_smem_raw + ((128u - (smem_u32(nw_smem_raw) & 127u)) & 127u);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem);   // [2]
  uint4* stage = reinterpret_cast<uint4*>(smem + 128);
  __shared__ float red[32];
  const uint32_t row_bytes = (uint32_t)nvec * 16u;
  const int mine = (rows - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;   // grid <= rows
  auto issue = [&](int k) {   // thread 0
    mbar_expect_tx(&full[k & 1], row_bytes);
    bulk_row_load(stage + (k & 1) * nvec, x + ((size_t)blockIdx.x + (size_t)k * gridDim.x) * nvec, row_bytes, &full[k & 1]);
  };
  int issued = 0;
  if (threadIdx.x == 0) {
    mbar_init(&full[0], 1);
    mbar_init(&full[1], 1);
    fence_barrier_init();
    issue(issued++);
  }
  float wv[VPT][8];
#pragma unroll
  for (int j = 0; j < VPT; ++j) {
    const int i = threadIdx.x + j * NORM_THREADS;
    if (i < nvec) unpack8(w[i], wv[j]);
  }
  bool ok = true;
  int k = 0, drain_from = -1;
  for (; k < mine; ++k) {
    ok = __syncthreads_and(ok);     // every thread is done with the stage the next request goes into (and sees the barriers)
    if (!ok) break;
    ok = mbar_wait(&full[k & 1], (uint32_t)(k >> 1) & 1u, status, kTimeoutTmaFull, 75);
    if (!ok && drain_from < 0) drain_from = k;
    if (threadIdx.x == 0 && ok && issued < mine) {
      fence_proxy_async();
      issue(issued++);
    }
    const uint4* sx = stage + (k & 1) * nvec;
    const size_t row = (size_t)blockIdx.x + (size_t)k * gridDim.x;
    float v[VPT][8];
    float ss = 0.f;
#pragma unroll
    for (int j = 0; j < VPT; ++j) {
      const int i = threadIdx.x + j * NORM_THREADS;
      if (i < nvec) {
        unpack8(sx[i], v[j]);
#pragma unroll
        for (int e = 0; e < 8; ++e) ss += v[j][e] * v[j][e];
      }
    }
    const float rstd = rsqrtf(block_sum(ss, red) / (float)(nvec * 8) + eps);
    if (threadIdx.x == 0 && rstd_out) rstd_out[row] = rstd;
#pragma unroll
    for (int j = 0; j < VPT; ++j) {
      const int i = threadIdx.x + j * NORM_THREADS;
      if (i < nvec) {
        float o[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) o[e] = wv[j][e] * rbf(v[j][e] * rstd);
        y[row * nvec + i] = pack8(o);
      }
    }
  }
  if (drain_from < 0 && k < mine) drain_from = k;
  if (drain_from >= 0 && threadIdx.x == 0)   // a wait ran out: what was asked for still lands here (bounded again)
    for (int kk = drain_from; kk < issued; ++kk)
      mbar_wait(&full[kk & 1], (uint32_t)(kk >> 1) & 1u, status, kTimeoutTmaFull, 76);
}

// Backward: 128 threads to a row, GROUPS of them in a CTA, each with a ring of rows (dy | x | dres) of its own.  A thread
// holds its share of the row and of the column sums for the weight's gradient (VPT vectors); one barrier of its
// group adds up the row and frees the stage.  The column sums of a CTA's groups meet in shared memory and leave as one row of
// `parts`, which norm_dw_kernel adds up: no atomics, no clearing, the same bits every time.
// 8192 x 4096 with a residual: 50 us (5.4 TB/s of four tensors), 55 with 256 threads to a row and three barriers; x 5120 60 and 93.
constexpr int NB_GROUP = 128;
template <int VPT, int GROUPS>
__global__ void __launch_bounds__(NB_GROUP * GROUPS, 1)
rmsnorm_bwd_rows_kernel(const uint4* __restrict__ dy, const uint4* __restrict__ x, const uint4* __restrict__ w,
                        const float* __restrict__ rstd, const uint4* __restrict__ dres, uint4* __restrict__ dx,
                        float* __restrict__ parts, int rows, int nvec, int stages, int* status) {
  if (!chain_begin()) return;
  extern __shared__ uint8_t nb_smem_raw[];
  uint8_t* smem = nb_smem_raw + ((128u - (smem_u32(nb_smem_raw) & 127u)) & 127u);
  __shared__ __align__(16) float red[GROUPS][2][8];
  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int grp = warp / 4, tid = threadIdx.x % NB_GROUP;
  const uint32_t row_bytes = (uint32_t)nvec * 16u;
  uint64_t* full = reinterpret_cast<uint64_t*>(smem) + grp * NS_MAX_STAGES;
  uint4* sw = reinterpret_cast<uint4*>(smem + GROUPS * NS_MAX_STAGES * 8);
  uint4* rings = sw + nvec;
  uint4* ring = rings + (size_t)grp * stages * 3 * nvec;
  const int first = grp * gridDim.x + blockIdx.x, step = GROUPS * gridDim.x;
  const int mine = first < rows ? (rows - 1 - first) / step + 1 : 0;
  const int ntens = dres ? 3 : 2;
  auto issue = [&](int k) {   // one thread
    const int s = k % stages;
    const size_t off = ((size_t)first + (size_t)k * step) * nvec;
    uint4* dst = ring + (size_t)s * 3 * nvec;
    mbar_expect_tx(&full[s], (uint32_t)ntens * row_bytes);
    bulk_row_load(dst, dy + off, row_bytes, &full[s]);
    bulk_row_load(dst + nvec, x + off, row_bytes, &full[s]);
    if (dres) bulk_row_load(dst + 2 * nvec, dres + off, row_bytes, &full[s]);
  };
  const int ahead = min(stages, mine);
  if (tid == 0) {
    for (int s = 0; s < stages; ++s) mbar_init(&full[s], 1);
    fence_barrier_init();
    for (int i = 0; i < ahead; ++i) issue(i);
  }
  int issued = ahead;
  for (int i = threadIdx.x; i < nvec; i += blockDim.x) sw[i] = w[i];
  __syncthreads();
  float acc[VPT][8];
#pragma unroll
  for (int j = 0; j < VPT; ++j)
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[j][e] = 0.f;
  const float inv_d = 1.0f / (float)(nvec * 8);
  float rs = mine > 0 ? rstd[first] : 0.f;
  int k = 0;
  for (; k < mine; ++k) {
    const bool ok = mbar_wait_warp(&full[k % stages], (uint32_t)(k / stages) & 1u, status, kTimeoutTmaFull, 71);
    const uint4* sdy = ring + (size_t)(k % stages) * 3 * nvec;
    const size_t row = (size_t)first + (size_t)k * step;
    const float rs_next = k + 1 < mine ? rstd[row + step] : 0.f;
    uint4 dv[VPT], xv[VPT], rv[VPT];
    float dots[2] = {};         // this thread's of 256, and thread + 128's
#pragma unroll
    for (int j = 0; j < VPT; ++j) {
      const int i = tid + j * NB_GROUP;
      if (i < nvec) {
        dv[j] = sdy[i];
        xv[j] = sdy[nvec + i];
        if (dres) rv[j] = sdy[2 * nvec + i];
        float d[8], xf[8], wv[8];
        unpack8(dv[j], d);
        unpack8(xv[j], xf);
        unpack8(sw[i], wv);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const float xh = __fmul_rn(xf[e], rs);
          acc[j][e] = fmaf(d[e], xh, acc[j][e]);
          dots[j & 1] = fmaf(__fmul_rn(d[e], wv[e]), xh, dots[j & 1]);
        }
      }
    }
    dots[0] = warp_sum(dots[0]);
    dots[1] = warp_sum(dots[1]);
    if (lane == 0) {
      red[grp][k & 1][warp & 3] = dots[0];
      red[grp][k & 1][4 + (warp & 3)] = dots[1];
    }
    // the row's sum is complete, its stage has been read, and all of the group know whether one of them gave up waiting
    int all;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %1, 0;\n\tbarrier.cta.red.and.pred q, %2, %3, p;\n\tselp.b32 %0, 1, 0, q;\n\t}"
                 : "=r"(all)
                 : "r"((int)ok), "r"(1 + grp), "n"(NB_GROUP)
                 : "memory");
    if (!all) break;
    if (tid == 0 && issued < mine) {
      fence_proxy_async();
      issue(issued);
    }
    issued += issued < mine;
    const float4 a4 = *reinterpret_cast<const float4*>(red[grp][k & 1]), b4 = *reinterpret_cast<const float4*>(red[grp][k & 1] + 4);
    const float dot = (((a4.x + b4.x) + (a4.z + b4.z)) + ((a4.y + b4.y) + (a4.w + b4.w))) * inv_d;   // as block_sum adds eight warps
#pragma unroll
    for (int j = 0; j < VPT; ++j) {
      const int i = tid + j * NB_GROUP;
      if (i < nvec) {
        float d[8], xf[8], wv[8], o[8];
        unpack8(dv[j], d);
        unpack8(xv[j], xf);
        unpack8(sw[i], wv);
#pragma unroll
        for (int e = 0; e < 8; ++e) o[e] = fmaf(-__fmul_rn(xf[e], rs), dot, __fmul_rn(d[e], wv[e]));
        norm_dx(o, rs, dres ? &rv[j] : nullptr, (j >> 1) < (VPT <= 2 ? 0 : VPT <= 4 ? 1 : 3));
        dx[row * nvec + i] = pack8(o);
      }
    }
    rs = rs_next;
  }
  for (; k < issued; ++k)   // a wait ran out: what was asked for still lands here (bounded again)
    mbar_wait_warp(&full[k % stages], (uint32_t)(k / stages) & 1u, status, kTimeoutTmaFull, 72);
  __syncthreads();
  float4* sums = reinterpret_cast<float4*>(rings);     // [GROUPS][2 * nvec]; the rings are free
#pragma unroll
  for (int j = 0; j < VPT; ++j) {
    const int i = tid + j * NB_GROUP;
    if (i < nvec) {
      sums[(size_t)grp * 2 * nvec + 2 * i] = make_float4(acc[j][0], acc[j][1], acc[j][2], acc[j][3]);
      sums[(size_t)grp * 2 * nvec + 2 * i + 1] = make_float4(acc[j][4], acc[j][5], acc[j][6], acc[j][7]);
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 2 * nvec; i += blockDim.x) {
    float4 a = sums[i];
#pragma unroll
    for (int g = 1; g < GROUPS; ++g) {
      const float4 c = sums[(size_t)g * 2 * nvec + i];
      a.x += c.x; a.y += c.y; a.z += c.z; a.w += c.w;
    }
    reinterpret_cast<float4*>(parts)[(size_t)blockIdx.x * 2 * nvec + i] = a;
  }
}

// dw[c] = (`add`: dw[c] +) sum over the n rows of parts, in fp32 and, with dw_bf16, rounded.  A block takes 64 columns: sixteen threads of four
// columns each side by side, sixteen rows at a time.
__global__ void __launch_bounds__(256)
norm_dw_kernel(const float4* __restrict__ parts, float4* __restrict__ dw, uint2* __restrict__ dw_bf16, int n, int dim4, int add) {
  if (!chain_begin()) return;
  __shared__ float4 sums[16][16];
  const int c = threadIdx.x & 15, r0 = threadIdx.x >> 4, col = blockIdx.x * 16 + c;
  float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
  if (col < dim4) {
#pragma unroll 4
    for (int r = r0; r < n; r += 16) {
      const float4 v = parts[(size_t)r * dim4 + col];
      a.x += v.x; a.y += v.y; a.z += v.z; a.w += v.w;
    }
  }
  sums[r0][c] = a;
  __syncthreads();
  if (r0 != 0 || col >= dim4) return;
#pragma unroll
  for (int r = 1; r < 16; ++r) {
    const float4 v = sums[r][c];
    a.x += v.x; a.y += v.y; a.z += v.z; a.w += v.w;
  }
  if (add) {
    const float4 v = dw[col];
    a.x += v.x; a.y += v.y; a.z += v.z; a.w += v.w;
  }
  dw[col] = a;
  if (dw_bf16) dw_bf16[col] = make_uint2(pack_bf16(a.x, a.y), pack_bf16(a.z, a.w));
}

// ----------------------------------------------------------------------------
// RoPE (rotate-half; optional interleaved-pair input layout), in place.
// One thread handles 8 consecutive elements of the first half and their partners.
// ----------------------------------------------------------------------------
__global__ void rope_kernel(__nv_bfloat16* __restrict__ x, long long ld, int col0, int heads, int dim, int head_stride,
                            const float* __restrict__ cosT, const float* __restrict__ sinT,
                            const int* __restrict__ pos, long long tokens, int seq_len, float sign,
                            int interleaved) {
  if (!chain_begin()) return;
  const int half = dim / 2;
  const int vec_per_head = half / 8;
  const long long total = tokens * heads * vec_per_head;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const int v = (int)(idx % vec_per_head);
    const long long th = idx / vec_per_head;
    const int h = (int)(th % heads);
    const long long t = th / heads;
    const int p = pos ? pos[t] : (int)(t % seq_len);
    __nv_bfloat16* base = x + t * ld + col0 + h * head_stride;
    const float* c = cosT + (size_t)p * half + v * 8;
    const float* s = sinT + (size_t)p * half + v * 8;
    float a[8], b[8];
    if (!interleaved) {
      unpack8(*reinterpret_cast<const uint4*>(base + v * 8), a);
      unpack8(*reinterpret_cast<const uint4*>(base + half + v * 8), b);
    } else {
      // pairs (2i, 2i+1): element i of the first half is x[2i], of the second half x[2i+1]
      float lo[8], hi[8];
      unpack8(*reinterpret_cast<const uint4*>(base + v * 16), lo);
      unpack8(*reinterpret_cast<const uint4*>(base + v * 16 + 8), hi);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        a[e] = lo[2 * e]; b[e] = lo[2 * e + 1];
        a[4 + e] = hi[2 * e]; b[4 + e] = hi[2 * e + 1];
      }
    }
    float oa[8], ob[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const float cs = c[e], sn = s[e] * sign;
      oa[e] = a[e] * cs - b[e] * sn;
      ob[e] = b[e] * cs + a[e] * sn;
    }
    if (!interleaved) {
      *reinterpret_cast<uint4*>(base + v * 8) = pack8(oa);
      *reinterpret_cast<uint4*>(base + half + v * 8) = pack8(ob);
    }
    if (interleaved) {
      // The permuted (half-layout) result cannot be written in place by independent
      // threads without a race, so the interleaved variant keeps the pair layout:
      // attention scores are invariant to a fixed permutation applied to both q and k.
      float lo[8], hi[8];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        lo[2 * e] = oa[e]; lo[2 * e + 1] = ob[e];
        hi[2 * e] = oa[4 + e]; hi[2 * e + 1] = ob[4 + e];
      }
      *reinterpret_cast<uint4*>(base + v * 16) = pack8(lo);
      *reinterpret_cast<uint4*>(base + v * 16 + 8) = pack8(hi);
    }
  }
}

// ----------------------------------------------------------------------------
// SwiGLU
// ----------------------------------------------------------------------------
__global__ void swiglu_fwd_kernel(const uint4* __restrict__ gu, uint4* __restrict__ act, long long rows, int fvec) {
  if (!chain_begin()) return;
  const long long total = rows * fvec;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const long long r = idx / fvec;
    const int c = (int)(idx % fvec);
    float g[8], u[8], o[8];
    unpack8(gu[r * 2 * fvec + c], g);
    unpack8(gu[r * 2 * fvec + fvec + c], u);
#pragma unroll
    for (int e = 0; e < 8; ++e) o[e] = g[e] / (1.f + __expf(-g[e])) * u[e];
    act[idx] = pack8(o);
  }
}
__global__ void swiglu_bwd_kernel(const uint4* __restrict__ dact, const uint4* __restrict__ gu,
                                  uint4* __restrict__ dgu, long long rows, int fvec) {
  if (!chain_begin()) return;
  const long long total = rows * fvec;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const long long r = idx / fvec;
    const int c = (int)(idx % fvec);
    float g[8], u[8], d[8], dg[8], du[8];
    unpack8(gu[r * 2 * fvec + c], g);
    unpack8(gu[r * 2 * fvec + fvec + c], u);
    unpack8(dact[idx], d);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const float sg = 1.f / (1.f + __expf(-g[e]));
      const float silu = g[e] * sg;
      du[e] = d[e] * silu;
      dg[e] = d[e] * u[e] * (sg + silu * (1.f - sg));
    }
    dgu[r * 2 * fvec + c] = pack8(dg);
    dgu[r * 2 * fvec + fvec + c] = pack8(du);
  }
}

// ----------------------------------------------------------------------------
// Cross entropy: one CTA per row, online (max, sum) pass then gradient pass.
// Two resident CTAs per SM, so that the rows being worked on (296 x 256 KB at a 128k vocabulary) stay in L2 between the
// passes, and four vectors in flight per thread.  Bound by reading the rows from HBM once and writing them once, with two
// exponentials per element close behind (16 per clock and SM).  (Four CTAs per SM, one vector at a time and a 64-bit
// compare per element: 414 us for 3001 rows of 128,256 logits; this way 323.)
// ----------------------------------------------------------------------------
constexpr int CE_THREADS = 512;
constexpr int CE_UNROLL = 4;
__global__ void __launch_bounds__(CE_THREADS, 2)
ce_kernel(__nv_bfloat16* __restrict__ logits, long long ld, const long long* __restrict__ targets,
          float* __restrict__ loss_sum, const float* __restrict__ grad_scale, int rows, int vocab) {
  if (!chain_begin()) return;
  __shared__ float red[32];
  const int nvec = vocab / 8;  // host guarantees vocab % 8 == 0
  const float log2e = 1.4426950408889634f;
  const f32x2 log2e2 = f2_pack(log2e, log2e);
  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    uint4* lr = reinterpret_cast<uint4*>(logits + (size_t)row * ld);
    const long long tgt = targets[row];
    if (tgt < 0) {
      for (int i = threadIdx.x; i < nvec; i += CE_THREADS) lr[i] = make_uint4(0, 0, 0, 0);
      continue;
    }
    float m = -INFINITY, s = 0.f;
    for (int i0 = threadIdx.x; i0 < nvec; i0 += CE_THREADS * CE_UNROLL) {
      uint4 v[CE_UNROLL];
#pragma unroll
      for (int u = 0; u < CE_UNROLL; ++u) {
        const int i = i0 + u * CE_THREADS;
        v[u] = i < nvec ? lr[i] : make_uint4(0xff80ff80u, 0xff80ff80u, 0xff80ff80u, 0xff80ff80u);   // -inf
      }
      float f[CE_UNROLL][8], mx[CE_UNROLL];
#pragma unroll
      for (int u = 0; u < CE_UNROLL; ++u) {
        unpack8(v[u], f[u]);
        mx[u] = fmaxf(fmax3(fmaxf(f[u][0], f[u][1]), f[u][2], f[u][3]), fmax3(fmaxf(f[u][4], f[u][5]), f[u][6], f[u][7]));
      }
      float lm = mx[0];
#pragma unroll
      for (int u = 1; u < CE_UNROLL; ++u) lm = fmaxf(lm, mx[u]);
      if (lm > m) {
        s *= __expf(m - lm);
        m = lm;
      }
      const float m_fin = m == -INFINITY ? 0.f : m;      // (nothing but -inf so far: their exponentials are 0)
      const f32x2 nm = f2_pack(-m_fin, -m_fin);
      f32x2 acc = 0ull;
#pragma unroll
      for (int u = 0; u < CE_UNROLL; ++u)
#pragma unroll
        for (int e = 0; e < 8; e += 2) {
          float a, b;
          f2_unpack(f2_mul(f2_add(f2_pack(f[u][e], f[u][e + 1]), nm), log2e2), a, b);
          acc = f2_add(acc, f2_pack(ex2_approx(a), ex2_approx(b)));
        }
      float a, b;
      f2_unpack(acc, a, b);
      s += a + b;
    }
    const float gm = block_max(m, red);
    s *= (m == -INFINITY) ? 0.f : __expf(m - gm);
    const float gs = block_sum(s, red);
    const float lse = gm + __logf(gs);
    const float scale = grad_scale ? *grad_scale : 1.f;
    if (threadIdx.x == 0) {
      const float lt = __bfloat162float(logits[(size_t)row * ld + tgt]);
      atomicAdd(loss_sum, lse - lt);
    }
    __syncthreads();  // the target logit is read before it is overwritten below
    const float inv = 1.f / gs;
    const f32x2 ngm = f2_pack(-gm, -gm), inv2 = f2_pack(inv, inv), scale2 = f2_pack(scale, scale);
    const int tgt_vec = (int)(tgt / 8), tgt_e = (int)(tgt % 8);
    for (int i0 = threadIdx.x; i0 < nvec; i0 += CE_THREADS * CE_UNROLL) {
      uint4 v[CE_UNROLL];
#pragma unroll
      for (int u = 0; u < CE_UNROLL; ++u)
        if (i0 + u * CE_THREADS < nvec) v[u] = lr[i0 + u * CE_THREADS];
#pragma unroll
      for (int u = 0; u < CE_UNROLL; ++u) {
        const int i = i0 + u * CE_THREADS;
        if (i >= nvec) break;
        float f[8], p[8];
        unpack8(v[u], f);
#pragma unroll
        for (int e = 0; e < 8; e += 2) {
          float a, b;
          f2_unpack(f2_mul(f2_add(f2_pack(f[e], f[e + 1]), ngm), log2e2), a, b);
          f2_unpack(f2_mul(f2_pack(ex2_approx(a), ex2_approx(b)), inv2), p[e], p[e + 1]);
        }
        if (i == tgt_vec) {
#pragma unroll
          for (int e = 0; e < 8; ++e) p[e] -= e == tgt_e ? 1.f : 0.f;
        }
#pragma unroll
        for (int e = 0; e < 8; e += 2) f2_unpack(f2_mul(f2_pack(p[e], p[e + 1]), scale2), p[e], p[e + 1]);
        lr[i] = pack8(p);
      }
    }
  }
}

// ----------------------------------------------------------------------------
// Embedding
// ----------------------------------------------------------------------------
__global__ void embedding_fwd_kernel(const uint4* __restrict__ table, const long long* __restrict__ ids,
                                     uint4* __restrict__ out, long long tokens, int nvec, long long vocab,
                                     long long row0) {
  if (!chain_begin()) return;
  const long long total = tokens * nvec;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const long long t = idx / nvec;
    const int c = (int)(idx % nvec);
    const long long id = ids[t] - row0;
    out[idx] = (id >= 0 && id < vocab) ? table[id * nvec + c] : make_uint4(0, 0, 0, 0);
  }
}
template <bool F32>
__global__ void embedding_bwd_kernel(const __nv_bfloat162* __restrict__ dout, const long long* __restrict__ ids,
                                     void* __restrict__ dtable, long long tokens, int dim2, long long rows_local,
                                     long long row0) {
  const long long total = tokens * dim2;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const long long t = idx / dim2;
    const int c = (int)(idx % dim2);
    const long long id = ids[t] - row0;
    if (id < 0 || id >= rows_local) continue;
    const __nv_bfloat162 g = dout[idx];
    if (F32) {
      float* d = reinterpret_cast<float*>(dtable) + (id * dim2 + c) * 2;
      atomicAdd(d, __low2float(g));
      atomicAdd(d + 1, __high2float(g));
    } else {
      atomicAdd(reinterpret_cast<__nv_bfloat162*>(dtable) + id * dim2 + c, g);
    }
  }
}

// ----------------------------------------------------------------------------
// Optimizer
// ----------------------------------------------------------------------------
template <bool GBF16>
__global__ void adamw_kernel(float4* __restrict__ p32, float4* __restrict__ m, float4* __restrict__ v,
                             const void* __restrict__ grad, uint2* __restrict__ p16, long long n4, float lr,
                             float b1, float b2, float eps, float wd, float inv_bc1, float inv_sqrt_bc2,
                             const float* __restrict__ clip) {
  const float gs = clip ? *clip : 1.f;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n4;
       i += (long long)gridDim.x * blockDim.x) {
    float g[4];
    if (GBF16) {
      uint2 u = reinterpret_cast<const uint2*>(grad)[i];
      float2 a = unpack_bf16(u.x), b = unpack_bf16(u.y);
      g[0] = a.x; g[1] = a.y; g[2] = b.x; g[3] = b.y;
    } else {
      float4 u = reinterpret_cast<const float4*>(grad)[i];
      g[0] = u.x; g[1] = u.y; g[2] = u.z; g[3] = u.w;
    }
    float4 P = p32[i], M = m[i], V = v[i];
    float* pp = &P.x; float* mm = &M.x; float* vv = &V.x;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float ge = g[e] * gs;
      mm[e] = b1 * mm[e] + (1.f - b1) * ge;
      vv[e] = b2 * vv[e] + (1.f - b2) * ge * ge;
      const float denom = sqrtf(vv[e]) * inv_sqrt_bc2 + eps;
      pp[e] = pp[e] * (1.f - lr * wd) - lr * inv_bc1 * mm[e] / denom;
    }
    p32[i] = P; m[i] = M; v[i] = V;
    if (p16) p16[i] = make_uint2(pack_bf16(P.x, P.y), pack_bf16(P.z, P.w));
  }
}

template <bool BF16>
__global__ void sumsq_kernel(const void* __restrict__ g, long long n, float* __restrict__ out) {
  __shared__ float red[32];
  float acc = 0.f;
  if (BF16) {
    const long long nv = n / 8;
    const uint4* gv = reinterpret_cast<const uint4*>(g);
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nv;
         i += (long long)gridDim.x * blockDim.x) {
      float f[8];
      unpack8(gv[i], f);
#pragma unroll
      for (int e = 0; e < 8; ++e) acc += f[e] * f[e];
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      const __nv_bfloat16* gs = reinterpret_cast<const __nv_bfloat16*>(g);
      for (long long i = nv * 8; i < n; ++i) {
        float f = __bfloat162float(gs[i]);
        acc += f * f;
      }
    }
  } else {
    const long long nv = n / 4;
    const float4* gv = reinterpret_cast<const float4*>(g);
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nv;
         i += (long long)gridDim.x * blockDim.x) {
      float4 f = gv[i];
      acc += f.x * f.x + f.y * f.y + f.z * f.z + f.w * f.w;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      const float* gs = reinterpret_cast<const float*>(g);
      for (long long i = nv * 4; i < n; ++i) acc += gs[i] * gs[i];
    }
  }
  acc = block_sum(acc, red);
  if (threadIdx.x == 0) atomicAdd(out, acc);
}

__global__ void clip_coef_kernel(const float* sumsq, float max_norm, float* coef, float* norm_out) {
  const float n = sqrtf(*sumsq);
  if (norm_out) *norm_out = n;
  if (coef) *coef = (max_norm > 0.f) ? fminf(1.f, max_norm / (n + 1e-6f)) : 1.f;
}

__global__ void cast_kernel(const float4* __restrict__ src, uint2* __restrict__ dst, long long n4, float scale,
                            int accumulate) {
  if (!chain_begin()) return;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n4;
       i += (long long)gridDim.x * blockDim.x) {
    float4 s = src[i];
    s.x *= scale; s.y *= scale; s.z *= scale; s.w *= scale;
    if (accumulate) {
      uint2 o = dst[i];
      float2 a = unpack_bf16(o.x), b = unpack_bf16(o.y);
      s.x += a.x; s.y += a.y; s.z += b.x; s.w += b.y;
    }
    dst[i] = make_uint2(pack_bf16(s.x, s.y), pack_bf16(s.z, s.w));
  }
}

// dst = bf16(src * *scale): a weight gradient kept in fp32 through its accumulation, delivered in one pass.
// Bound by memory (6 bytes per value); two float4 loads in flight per thread, read once and not kept in L2.
// 128,256 x 4096 values: 0.51 ms (6.1 TB/s) where a multiplication and a cast took 1.86 ms.
__global__ void scale_cast_kernel(const float4* __restrict__ src, uint4* __restrict__ dst, long long n8,
                                  const float* __restrict__ scale) {
  if (!chain_begin()) return;
  const float sc = *scale;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n8;
       i += (long long)gridDim.x * blockDim.x) {
    const float4 a = __ldcs(src + 2 * i), b = __ldcs(src + 2 * i + 1);
    dst[i] = make_uint4(pack_bf16(a.x * sc, a.y * sc), pack_bf16(a.z * sc, a.w * sc), pack_bf16(b.x * sc, b.y * sc),
                        pack_bf16(b.z * sc, b.w * sc));
  }
}

inline int grid_for(long long work_items, int threads, int waves = 8) {
  long long blocks = (work_items + threads - 1) / threads;
  long long cap = (long long)sm_count() * waves;
  if (blocks > cap) blocks = cap;
  if (blocks < 1) blocks = 1;
  return (int)blocks;
}
inline int rc(cudaError_t e) { return e == cudaSuccess ? 0 : 1000 + (int)e; }

static void launch_rmsnorm_bwd(const void* dy, const void* x, const void* w, const float* rstd, const void* dres,
                               void* dx, float* dw_f32, int rows, int dim, cudaStream_t stream) {
  const int nvec = dim / 8;
  const int vpt = (nvec + NORM_THREADS - 1) / NORM_THREADS;
  const int per_sm = vpt <= 2 ? 4 : 2;
  const int grid = rows < sm_count() * per_sm ? rows : sm_count() * per_sm;
#define TPB_LAUNCH_NORM_BWD(V) chain(rmsnorm_bwd_kernel<V>, grid, NORM_THREADS, 0, stream, \
      (const uint4*)dy, (const uint4*)x, (const uint4*)w, rstd, (const uint4*)dres, (uint4*)dx, dw_f32, rows, nvec)
  if (vpt <= 1) TPB_LAUNCH_NORM_BWD(1); else if (vpt == 2) TPB_LAUNCH_NORM_BWD(2); else TPB_LAUNCH_NORM_BWD(4);
#undef TPB_LAUNCH_NORM_BWD
}

}  // namespace tpb

using namespace tpb;
#define STREAM(s) reinterpret_cast<cudaStream_t>(s)

static bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// Streamed forms: rows that can be bulk-copied (16-byte aligned bases; the pitch is a multiple of 16 bytes), no residual
// added in the forward, and enough of them: fewer rows than warps of the streamed forward leave it with nothing to run ahead
// of, and the CTAs of one row each start sooner.  us, CTAs per row / streamed, inputs larger than L2 in all:
//   forward, a warp to a row: 512 wide: 2600 rows 4.3 / 4.5, 4000 5.2 / 4.7, 32768 30.8 / 23.8;   1024: 2600 rows 4.5 / 5.3, 10000 12.4 /
//     12.4, 32768 38 / 31;   2048: 2600 rows 5.9 / 7.6, 12000 20.4 / 20.1, 32768 52.5 / 47.5 (one vector to a thread of the CTA: quick);
//     2304: 2300 rows 8.7 / 6.3, 8192 25 / 16;   3072: 2200 9.2 / 7.4, 8192 29 / 20;   4096: 3200 rows 11.6 / 12.9, 4500 17.1 / 16.8, 8192 34 / 27
//   forward, 256 threads to a row / a warp to a row: 5120: 900 rows 6.9 / 6.1 / 7.1, 8192 44 / 32.5 / 35.5;   6144: 2200 13.0 / 11.2 / 16.4,
//     8192 48 / 36 / 47;   8192: 1200 11.2 / 8.9 / 17, 3200 26.7 / 18.5 / 31.5, 8192 61 / 43.7 / 75.5
//   backward with a residual, 4096 wide: 1000 rows 23 / 19, 4000 33 / 31, 8192 55 / 50;   5120 wide: 2000 29 / 22, 8192 93 / 60;
//     8192 wide: 600 rows 23.4 / 16.0, 1000 33.5 / 19.3
static int norm_bwd_rows_from(int dim) { return dim > 4096 ? 592 : 1024; }
static int norm_fwd_rows_from(int nvec) { return nvec <= 96 ? 3000 : nvec <= 256 ? 12000 : nvec <= 384 ? 2048 : 4500; }
static bool launch_rmsnorm_fwd_rows(const void* x, const void* w, void* y, float* rstd, int rows, int dim, float eps,
                                    cudaStream_t stream) {
  static const bool disabled = []() { const char* v = getenv("TPB_RMSNORM_FWD_BULK"); return v && v[0] == '0'; }();
  if (disabled) return false;
  const int nvec = dim / 8, row_bytes = dim * 2;
  if (nvec > 512 || !aligned16(x) || !aligned16(y) || !aligned16(w) || rows < norm_fwd_rows_from(nvec)) return false;
  constexpr int most = 16;
  int stages = NS_SMEM / (most * row_bytes);
  stages = stages > NS_MAX_STAGES ? NS_MAX_STAGES : stages < 2 ? 2 : stages;
  int warps = NS_SMEM / (stages * row_bytes);
  if (warps > most) warps = most;
  const size_t smem = 128 + 16 * NS_MAX_STAGES * 8 + (size_t)row_bytes * (1 + warps * stages);
#define TPB_NORM_FWD(V)                                                                                                      \
  do {                                                                                                                       \
    static const cudaError_t set =                                                                                           \
        cudaFuncSetAttribute(rmsnorm_fwd_rows_kernel<V>, cudaFuncAttributeMaxDynamicSharedMemorySize, 226 * 1024);           \
    if (set != cudaSuccess) return false;                                                                                    \
    chain(rmsnorm_fwd_rows_kernel<V>, sm_count(), 32 * warps, smem, stream, (const uint4*)x, (const uint4*)w, (uint4*)y, rstd, \
          rows, nvec, eps, stages, status_block());                                                                          \
  } while (0)
  if (nvec <= 256) TPB_NORM_FWD(8); else TPB_NORM_FWD(16);
#undef TPB_NORM_FWD
  return true;
}

constexpr int NS_WIDE_CTAS = 3, NS_WIDE_SMEM = 66 * 1024;   // (as much as lets three on an SM and no fourth beside an idle one)
static bool launch_rmsnorm_fwd_wide(const void* x, const void* w, void* y, float* rstd, int rows, int dim, float eps,
                                    cudaStream_t stream) {
  static const bool disabled = []() { const char* v = getenv("TPB_RMSNORM_FWD_BULK"); return v && v[0] == '0'; }();
  const int nvec = dim / 8, grid = NS_WIDE_CTAS * sm_count();
  if (disabled || nvec <= 512 || !aligned16(x) || !aligned16(y) || !aligned16(w) || rows < 2 * grid) return false;
  static const cudaError_t set =
      cudaFuncSetAttribute(rmsnorm_fwd_wide_kernel<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, NS_WIDE_SMEM);
  if (set != cudaSuccess) return false;
  chain(rmsnorm_fwd_wide_kernel<4>, grid, NORM_THREADS, NS_WIDE_SMEM, stream, (const uint4*)x, (const uint4*)w, (uint4*)y, rstd,
        rows, nvec, eps, status_block());
  return true;
}

extern "C" int tpb_rmsnorm_fwd(const void* x, const void* res, const void* w, void* y, void* h_out, float* rstd,
                               int rows, int dim, float eps, void* stream) {
  if (dim % 8 || dim > 8 * NORM_THREADS * NORM_VPT) return -2;
  if (rows <= 0) return 0;
  if (!res && (launch_rmsnorm_fwd_rows(x, w, y, rstd, rows, dim, eps, STREAM(stream)) ||
               launch_rmsnorm_fwd_wide(x, w, y, rstd, rows, dim, eps, STREAM(stream))))
    return rc(cudaGetLastError());
  const int nvec = dim / 8;
  const int vpt = (nvec + NORM_THREADS - 1) / NORM_THREADS;
  const int per_sm = vpt <= 2 ? 8 : 4;
  const int grid = rows < sm_count() * per_sm ? rows : sm_count() * per_sm;
  const bool early = rows <= 2 * sm_count();
#define TPB_LAUNCH_NORM_FWD(V, EARLY) chain(rmsnorm_fwd_kernel<V, EARLY>, grid, NORM_THREADS, 0, STREAM(stream), \
      (const uint4*)x, (const uint4*)res, (const uint4*)w, (uint4*)y, (uint4*)h_out, rstd, rows, nvec, eps)
  if (vpt > 2) TPB_LAUNCH_NORM_FWD(4, true);
  else if (vpt == 2) { if (early) TPB_LAUNCH_NORM_FWD(2, true); else TPB_LAUNCH_NORM_FWD(2, false); }
  else if (early) TPB_LAUNCH_NORM_FWD(1, true); else TPB_LAUNCH_NORM_FWD(1, false);
#undef TPB_LAUNCH_NORM_FWD
  return rc(cudaGetLastError());
}

static int norm_bwd_groups(int nvec) { return nvec <= 512 ? 4 : nvec <= 640 ? 3 : 2; }
static bool launch_rmsnorm_bwd_rows(const void* dy, const void* x, const void* w, const float* rstd, const void* dres, void* dx,
                                    float* parts, int rows, int dim, cudaStream_t stream) {
  const int nvec = dim / 8, stage_bytes = 3 * dim * 2, groups = norm_bwd_groups(nvec);
  int stages = NS_SMEM / (groups * stage_bytes);
  if (stages > NS_MAX_STAGES) stages = NS_MAX_STAGES;
  const size_t smem = 128 + groups * NS_MAX_STAGES * 8 + (size_t)dim * 2 + (size_t)groups * stages * stage_bytes;
#define TPB_NORM_BWD(V, G)                                                                                              \
  do {                                                                                                                  \
    static const cudaError_t set =                                                                                      \
        cudaFuncSetAttribute(rmsnorm_bwd_rows_kernel<V, G>, cudaFuncAttributeMaxDynamicSharedMemorySize, 226 * 1024);   \
    if (set != cudaSuccess) return false;                                                                               \
    chain(rmsnorm_bwd_rows_kernel<V, G>, sm_count(), NB_GROUP * G, smem, stream, (const uint4*)dy, (const uint4*)x,     \
          (const uint4*)w, rstd, (const uint4*)dres, (uint4*)dx, parts, rows, nvec, stages, status_block());            \
  } while (0)
  if (nvec <= 128) TPB_NORM_BWD(1, 4); else if (nvec <= 256) TPB_NORM_BWD(2, 4); else if (nvec <= 512) TPB_NORM_BWD(4, 4);
  else if (nvec <= 640) TPB_NORM_BWD(5, 3); else TPB_NORM_BWD(8, 2);
#undef TPB_NORM_BWD
  return true;
}

// Rows of scratch that tpb_rmsnorm_bwd_dw takes.
extern "C" int tpb_rmsnorm_bwd_parts(int rows, int dim) {
  static const bool disabled = []() { const char* v = getenv("TPB_RMSNORM_BWD_BULK"); return v && v[0] == '0'; }();
  return disabled || dim % 8 || dim > 8 * NORM_THREADS * NORM_VPT || rows < norm_bwd_rows_from(dim) ? 0 : sm_count();
}

extern "C" int tpb_rmsnorm_bwd(const void* dy, const void* x, const void* w, const float* rstd, const void* dres,
                               void* dx, float* dw_f32, int rows, int dim, void* stream) {
  if (dim % 8 || dim > 8 * NORM_THREADS * NORM_VPT) return -2;
  if (rows <= 0) return 0;
  launch_rmsnorm_bwd(dy, x, w, rstd, dres, dx, dw_f32, rows, dim, STREAM(stream));
  return rc(cudaGetLastError());
}

extern "C" int tpb_rope_strided(void* x, long long ld, int col0, int heads, int dim, int head_stride,
                                const float* cos, const float* sin, const int* pos, int tokens, int seq_len,
                                int inverse, int interleaved, void* stream) {
  if (dim % 16 || ld % 8 || col0 % 8 || head_stride % 8 || head_stride < dim) return -2;
  if (tokens <= 0 || heads <= 0) return 0;
  long long total = (long long)tokens * heads * (dim / 16);
  chain(rope_kernel, grid_for(total, 256), 256, 0, STREAM(stream), (__nv_bfloat16*)x, ld, col0, heads, dim, head_stride,
                                                                cos, sin, pos, tokens, seq_len,
                                                                inverse ? -1.f : 1.f, interleaved);
  return rc(cudaGetLastError());
}

extern "C" int tpb_rope(void* x, long long ld, int col0, int heads, int dim, const float* cos, const float* sin,
                        const int* pos, int tokens, int seq_len, int inverse, int interleaved, void* stream) {
  return tpb_rope_strided(x, ld, col0, heads, dim, dim, cos, sin, pos, tokens, seq_len, inverse, interleaved, stream);
}

extern "C" int tpb_swiglu_fwd(const void* gu, void* act, int rows, int f, void* stream) {
  if (f % 8) return -2;
  if (rows <= 0) return 0;
  chain(swiglu_fwd_kernel, grid_for((long long)rows * (f / 8), 256), 256, 0, STREAM(stream), (const uint4*)gu,
                                                                                         (uint4*)act, rows, f / 8);
  return rc(cudaGetLastError());
}
extern "C" int tpb_swiglu_bwd(const void* dact, const void* gu, void* dgu, int rows, int f, void* stream) {
  if (f % 8) return -2;
  if (rows <= 0) return 0;
  chain(swiglu_bwd_kernel, grid_for((long long)rows * (f / 8), 256), 256, 0, STREAM(stream),
        (const uint4*)dact, (const uint4*)gu, (uint4*)dgu, rows, f / 8);
  return rc(cudaGetLastError());
}

extern "C" int tpb_ce_fwd_bwd(void* logits, long long ld, const long long* targets, float* loss_sum,
                              const float* grad_scale, int rows, int vocab, void* stream) {
  if (vocab % 8 || ld % 8) return -2;
  if (rows <= 0) return 0;
  const int grid = rows < sm_count() * 2 ? rows : sm_count() * 2;
  chain(ce_kernel, grid, CE_THREADS, 0, STREAM(stream), (__nv_bfloat16*)logits, ld, targets, loss_sum, grad_scale, rows,
                                                     vocab);
  return rc(cudaGetLastError());
}

extern "C" int tpb_adamw(float* p32, float* m, float* v, const void* grad, void* p16, long long n, float lr,
                         float beta1, float beta2, float eps, float wd, float bc1, float bc2, const float* clip_coef,
                         int grad_is_bf16, void* stream) {
  if (n % 4) return -2;
  if (n <= 0) return 0;
  const int grid = grid_for(n / 4, 256, 16);
  const float inv_bc1 = 1.f / bc1, inv_sqrt_bc2 = 1.f / sqrtf(bc2);
  if (grad_is_bf16)
    adamw_kernel<true><<<grid, 256, 0, STREAM(stream)>>>((float4*)p32, (float4*)m, (float4*)v, grad, (uint2*)p16,
                                                         n / 4, lr, beta1, beta2, eps, wd, inv_bc1, inv_sqrt_bc2,
                                                         clip_coef);
  else
    adamw_kernel<false><<<grid, 256, 0, STREAM(stream)>>>((float4*)p32, (float4*)m, (float4*)v, grad, (uint2*)p16,
                                                          n / 4, lr, beta1, beta2, eps, wd, inv_bc1, inv_sqrt_bc2,
                                                          clip_coef);
  return rc(cudaGetLastError());
}

extern "C" int tpb_sumsq(const void* g, long long n, int is_bf16, float* out, void* stream) {
  if (n <= 0) return 0;
  const int grid = grid_for(n / 8 + 1, 512, 4);
  if (is_bf16) sumsq_kernel<true><<<grid, 512, 0, STREAM(stream)>>>(g, n, out);
  else sumsq_kernel<false><<<grid, 512, 0, STREAM(stream)>>>(g, n, out);
  return rc(cudaGetLastError());
}

extern "C" int tpb_clip_coef(const float* sumsq, float max_norm, float* coef, float* norm_out, void* stream) {
  clip_coef_kernel<<<1, 1, 0, STREAM(stream)>>>(sumsq, max_norm, coef, norm_out);
  return rc(cudaGetLastError());
}

extern "C" int tpb_embedding_fwd(const void* table, const long long* ids, void* out, int tokens, int dim,
                                 long long vocab, long long row0, void* stream) {
  if (dim % 8) return -2;
  if (tokens <= 0) return 0;
  chain(embedding_fwd_kernel, grid_for((long long)tokens * (dim / 8), 256), 256, 0, STREAM(stream),
        (const uint4*)table, ids, (uint4*)out, tokens, dim / 8, vocab, row0);
  return rc(cudaGetLastError());
}
extern "C" int tpb_embedding_bwd(const void* dout, const long long* ids, void* dtable, int tokens, int dim,
                                 long long rows_local, long long row0, int dtable_is_f32, void* stream) {
  if (dim % 2) return -2;
  if (tokens <= 0) return 0;
  const int grid = grid_for((long long)tokens * (dim / 2), 256);
  if (dtable_is_f32)
    embedding_bwd_kernel<true><<<grid, 256, 0, STREAM(stream)>>>((const __nv_bfloat162*)dout, ids, dtable, tokens,
                                                                 dim / 2, rows_local, row0);
  else
    embedding_bwd_kernel<false><<<grid, 256, 0, STREAM(stream)>>>((const __nv_bfloat162*)dout, ids, dtable, tokens,
                                                                  dim / 2, rows_local, row0);
  return rc(cudaGetLastError());
}

extern "C" int tpb_cast_f32_to_bf16(const float* src, void* dst, long long n, float scale, int accumulate,
                                    void* stream) {
  if (n % 4) return -2;
  if (n <= 0) return 0;
  chain(cast_kernel, grid_for(n / 4, 256), 256, 0, STREAM(stream), (const float4*)src, (uint2*)dst, n / 4, scale,
                                                                accumulate);
  return rc(cudaGetLastError());
}

// n % 8 == 0, 16-byte aligned pointers; `scale` is one float in device memory.
extern "C" int tpb_scale_cast_bf16(const float* src, void* dst, long long n, const float* scale, void* stream) {
  if ((n % 8) || (reinterpret_cast<uintptr_t>(src) % 16) || (reinterpret_cast<uintptr_t>(dst) % 16)) return -2;
  if (n <= 0) return 0;
  chain(scale_cast_kernel, grid_for(n / 8, 256, 16), 256, 0, STREAM(stream), (const float4*)src, (uint4*)dst, n / 8, scale);
  return rc(cudaGetLastError());
}

// tpb_rmsnorm_bwd with the weight gradient written to dw_f32 or, with `add`, added to what is there; with dw_bf16 the result is
// also delivered in bf16.
extern "C" int tpb_rmsnorm_bwd_dw(const void* dy, const void* x, const void* w, const float* rstd, const void* dres, void* dx,
                                  float* dw_f32, void* dw_bf16, float* parts, int add, int rows, int dim, void* stream) {
  const int n = parts ? tpb_rmsnorm_bwd_parts(rows, dim) : 0;
  if (n > 0 && aligned16(dy) && aligned16(x) && aligned16(w) && aligned16(dx) && aligned16(dres) && aligned16(dw_f32) &&
      aligned16(parts) && reinterpret_cast<uintptr_t>(dw_bf16) % 8 == 0 &&
      launch_rmsnorm_bwd_rows(dy, x, w, rstd, dres, dx, parts, rows, dim, STREAM(stream))) {
    chain(norm_dw_kernel, (dim / 4 + 15) / 16, 256, 0, STREAM(stream), (const float4*)parts, (float4*)dw_f32, (uint2*)dw_bf16, n,
          dim / 4, add);
    return rc(cudaGetLastError());
  }
  const cudaError_t e = add ? cudaSuccess : cudaMemsetAsync(dw_f32, 0, sizeof(float) * dim, STREAM(stream));
  if (e != cudaSuccess) return rc(e);
  const int r = tpb_rmsnorm_bwd(dy, x, w, rstd, dres, dx, dw_f32, rows, dim, stream);
  return r || !dw_bf16 ? r : tpb_cast_f32_to_bf16(dw_f32, dw_bf16, dim, 1.f, 0, stream);
}

// ----------------------------------------------------------------------------
// Allocation-free variant of the RMSNorm backward (see tpb_noalloc.h).
// ----------------------------------------------------------------------------
#include "tpb_noalloc.h"

namespace tpb {
// fp32 weight-gradient accumulator shared by every call on this device.  In host code this
// name is only a handle; the device address comes from cudaGetSymbolAddress below.
static __device__ __align__(256) float g_noalloc_dw_scratch[TPB_NOALLOC_MAX_DIM];

constexpr int kMaxDevices = 64;
static float* g_noalloc_dw_ptr[kMaxDevices] = {nullptr};

// Device address of the scratch array for the current device (looked up once per device).
static float* noalloc_scratch_for_current_device() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return nullptr;
  if (g_noalloc_dw_ptr[dev] == nullptr) {
    float* ptr = nullptr;
    if (cudaGetSymbolAddress(reinterpret_cast<void**>(&ptr), g_noalloc_dw_scratch) != cudaSuccess) return nullptr;
    g_noalloc_dw_ptr[dev] = ptr;
  }
  return g_noalloc_dw_ptr[dev];
}

__global__ void noalloc_store_dw_kernel(const float* __restrict__ acc, __nv_bfloat16* __restrict__ out, int dim) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < dim; i += gridDim.x * blockDim.x)
    out[i] = __float2bfloat16(acc[i]);
}
}  // namespace tpb

extern "C" int tpb_rmsnorm_bwd_noalloc(const void* dy, const void* x, const void* w, const float* rstd,
                                       const void* dres, void* dx, void* dw_bf16, int rows, int dim, void* stream) {
  if (dim <= 0 || dim % 8) return -2;
  if (dim > TPB_NOALLOC_MAX_DIM) return -6;
  float* scratch = noalloc_scratch_for_current_device();
  if (!scratch) return -7;
  cudaStream_t s = STREAM(stream);
  // the accumulator keeps the previous call's sums: clear what this call will add into
  cudaError_t e = cudaMemsetAsync(scratch, 0, sizeof(float) * dim, s);
  if (e != cudaSuccess) return 1000 + (int)e;
  if (rows > 0) {
    launch_rmsnorm_bwd(dy, x, w, rstd, dres, dx, scratch, rows, dim, s);
    e = cudaGetLastError();
    if (e != cudaSuccess) return 1000 + (int)e;
  }
  noalloc_store_dw_kernel<<<(dim + 255) / 256, 256, 0, s>>>(scratch, (__nv_bfloat16*)dw_bf16, dim);
  return rc(cudaGetLastError());
}

extern "C" const char* tpb_noalloc_strerror(int code) {
  switch (code) {
    case 0: return "ok";
    case -2: return "dim must be a positive multiple of 8";
    case -6: return "dim exceeds TPB_NOALLOC_MAX_DIM (8192): the built-in scratch accumulator is too small";
    case -7: return "could not resolve the device address of the built-in scratch (cudaGetSymbolAddress failed)";
    default: return code >= 1000 ? "CUDA launch failed (code - 1000 is the cudaError_t)" : "unknown error";
  }
}
