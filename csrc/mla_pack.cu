// Keys and values of latent attention in the layout the attention kernels take, and back.
//
// The up-projection yields [token][head][dn key values | dv values]; every head's key is completed by the
// token's one rotary key.  Forward: k[t,h] = [kv[t,h,:dn] | rot[t]], v[t,h] = kv[t,h,dn:].  Backward: dkv from
// dk and dv, drot[t] = sum_h dk[t,h,dn:] (fp32, in a fixed order: heads modulo sixteen
// first, then those sums).  One pass each, 16-byte vectors, bound by
// memory; as torch operators the same is a concatenation and a copy forward and seven launches backward
// (zero-filled slice gradients and their sum), each over the whole tensors: about 110 us together at 2048 tokens and
// 16 heads of 128 + 64 / 128, against 5 + 5 us (from L2).

#include <initializer_list>

#include "common.cuh"
#include "tpb.h"

namespace tpb {

int sm_count();

constexpr int PACK_WARPS = 8, PACK_HEADS = 4;

// One warp per token and four of its heads, a lane per 16-byte vector: what a kernel of this length spends is latency, so a
// lane has five independent loads under way (four heads and the rotary key, which is read once for the four) and finds its
// place without a division.  A thread per vector of the grid, two 64-bit divisions each: 300 / 900 / 2048 tokens of 16 heads
// 2.9 / 5.7 / 9.2 us, 2048 tokens of 128 heads 85.7; this way 2.7 / 3.2 / 4.8 and 45.3.
__global__ void __launch_bounds__(PACK_WARPS * 32)
mla_pack_kernel(const uint4* __restrict__ kv, const uint4* __restrict__ rot, long long rot_ld, uint4* __restrict__ k,
                uint4* __restrict__ v, long long tokens, int H, int dn8, int dr8, int dv8, long long k_batch,
                long long v_batch) {
  if (!chain_begin()) return;
  const long long row = blockIdx.z;              // of the batch: its keys and values are k_batch and v_batch vectors apart
  kv += row * tokens * H * (dn8 + dv8);
  rot += row * tokens * rot_ld;
  k += row * k_batch;
  v += row * v_batch;
  const int lane = threadIdx.x & 31, h0 = blockIdx.x * PACK_HEADS, heads = min(PACK_HEADS, H - h0);
  const int per = dn8 + dv8, dk8 = dn8 + dr8;
  for (long long t = blockIdx.y * (long long)PACK_WARPS + (threadIdx.x >> 5); t < tokens;
       t += (long long)gridDim.y * PACK_WARPS) {
    const long long th = t * H + h0;
    for (int j = lane; j < max(per, dr8); j += 32) {
      uint4 r, x[PACK_HEADS];
      if (j < dr8) r = rot[t * rot_ld + j];
#pragma unroll
      for (int h = 0; h < PACK_HEADS; ++h)
        if (h < heads && j < per) x[h] = kv[(th + h) * per + j];
#pragma unroll
      for (int h = 0; h < PACK_HEADS; ++h) {
        if (h >= heads) break;
        if (j < dn8) k[(th + h) * dk8 + j] = x[h];
        else if (j < per) v[(th + h) * dv8 + j - dn8] = x[h];
        if (j < dr8) k[(th + h) * dk8 + dn8 + j] = r;
      }
    }
  }
}

constexpr int UNPACK_SUMS = 16;

// The same split: a warp per token and four heads copies, and a warp per token (the blocks with blockIdx.x = 0) sums the
// rotary slices of all heads, a lane per pair of columns with sixteen heads under way, without shared memory or a barrier.
// A block per token whose threads met in shared memory: 3.5 / 5.0 / 7.9 us and, at 512 tokens of 128 heads, 16.3; this way
// 2.1 / 3.0 / 4.9 and 15.5.
__global__ void __launch_bounds__(PACK_WARPS * 32)
mla_unpack_kernel(const uint4* __restrict__ dk, const uint4* __restrict__ dv, uint4* __restrict__ dkv,
                  uint32_t* __restrict__ drot, long long tokens, int H, int dn8, int dr8, int dv8) {
  if (!chain_begin()) return;
  const int lane = threadIdx.x & 31, per = dn8 + dv8, dk8 = dn8 + dr8;
  const long long t0 = blockIdx.y * (long long)PACK_WARPS + (threadIdx.x >> 5), step = (long long)gridDim.y * PACK_WARPS;
  if (blockIdx.x == 0) {
    for (long long t = t0; t < tokens; t += step)
      for (int j = lane; j < dr8 * 4; j += 32) {
        const uint32_t* src = reinterpret_cast<const uint32_t*>(dk + t * H * dk8 + dn8) + j;
        float2 s[UNPACK_SUMS] = {};
        for (int h0 = 0; h0 < H; h0 += UNPACK_SUMS) {
          uint32_t u[UNPACK_SUMS];
#pragma unroll
          for (int i = 0; i < UNPACK_SUMS; ++i) u[i] = h0 + i < H ? src[(long long)(h0 + i) * dk8 * 4] : 0u;
#pragma unroll
          for (int i = 0; i < UNPACK_SUMS; ++i) {
            const float2 x = unpack_bf16(u[i]);
            s[i].x += x.x;
            s[i].y += x.y;
          }
        }
#pragma unroll
        for (int i = 1; i < UNPACK_SUMS; ++i) {
          s[0].x += s[i].x;
          s[0].y += s[i].y;
        }
        drot[t * dr8 * 4 + j] = pack_bf16(s[0].x, s[0].y);
      }
    return;
  }
  const int h0 = (blockIdx.x - 1) * PACK_HEADS, heads = min(PACK_HEADS, H - h0);
  for (long long t = t0; t < tokens; t += step) {
    const long long th = t * H + h0;
    for (int j = lane; j < per; j += 32) {
      uint4 x[PACK_HEADS];
#pragma unroll
      for (int h = 0; h < PACK_HEADS; ++h)
        if (h < heads) x[h] = j < dn8 ? dk[(th + h) * dk8 + j] : dv[(th + h) * dv8 + j - dn8];
#pragma unroll
      for (int h = 0; h < PACK_HEADS; ++h)
        if (h < heads) dkv[(th + h) * per + j] = x[h];
    }
  }
}

// Rotation of eight pairs; interleaved: 16 consecutive values (2i, 2i + 1), else x[0..7] and x[half..half + 7].
__device__ __forceinline__ void rotate8(const uint4& u, const uint4& v, uint4& ou, uint4& ov, const float* cs, const float* sn,
                                        float sign, bool interleaved) {
  float x[16];
  const uint32_t w[8] = {u.x, u.y, u.z, u.w, v.x, v.y, v.z, v.w};
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float2 p = unpack_bf16(w[i]);
    x[2 * i] = p.x; x[2 * i + 1] = p.y;
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int ia = interleaved ? 2 * i : i, ib = interleaved ? 2 * i + 1 : i + 8;
    const float a = x[ia], b = x[ib], c = cs[i], s = sn[i] * sign;
    x[ia] = a * c - b * s;
    x[ib] = b * c + a * s;
  }
  ou = make_uint4(pack_bf16(x[0], x[1]), pack_bf16(x[2], x[3]), pack_bf16(x[4], x[5]), pack_bf16(x[6], x[7]));
  ov = make_uint4(pack_bf16(x[8], x[9]), pack_bf16(x[10], x[11]), pack_bf16(x[12], x[13]), pack_bf16(x[14], x[15]));
}

// SPLIT: rows of [latent | rotary key] into two dense matrices, the key rotated on the way; else back, the key's gradient
// rotated the other way.  One pass, bound by memory and its launch: as a rotation in place and two copies, and a
// concatenation and a rotation back, five launches: prefill of 300 / 900 tokens 586 / 771 us, this way 559 / 748; the attention
// block of 600 tokens, forward and backward, 390 / 345.
template <bool SPLIT>
__global__ void latent_kernel(const uint4* wide_in, uint4* wide_out, const uint4* lat_in, uint4* lat_out, const uint4* rot_in,
                              uint4* rot_out, const float* cosT, const float* sinT, const int* pos, long long tokens,
                              int seq_len, int c8, int dr8, int interleaved) {
  if (!chain_begin()) return;
  const int pairs = dr8 / 2, per = c8 + pairs;       // 16-byte vectors of the latent, then groups of eight pairs
  const long long total = tokens * per;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const long long t = i / per;
    const int j = (int)(i - t * per);
    if (j < c8) {
      if (SPLIT) lat_out[t * c8 + j] = wide_in[t * (c8 + dr8) + j];
      else wide_out[t * (c8 + dr8) + j] = lat_in[t * c8 + j];
      continue;
    }
    const int g = j - c8, at = pos ? pos[t] : (int)(t % seq_len);
    const int v0 = interleaved ? 2 * g : g, v1 = interleaved ? 2 * g + 1 : g + pairs;
    const float* cs = cosT + (size_t)at * (dr8 * 4) + g * 8;
    const float* sn = sinT + (size_t)at * (dr8 * 4) + g * 8;
    const uint4* src = SPLIT ? wide_in + t * (c8 + dr8) + c8 : rot_in + t * dr8;
    uint4* dst = SPLIT ? rot_out + t * dr8 : wide_out + t * (c8 + dr8) + c8;
    uint4 a, b;
    rotate8(src[v0], src[v1], a, b, cs, sn, SPLIT ? 1.f : -1.f, interleaved != 0);
    dst[v0] = a;
    dst[v1] = b;
  }
}

static bool latent_args_ok(std::initializer_list<const void*> ptrs, int c, int dr, int seq_len) {
  for (const void* a : ptrs)
    if (reinterpret_cast<uintptr_t>(a) % 16) return false;
  return c >= 8 && c % 8 == 0 && dr >= 16 && dr % 16 == 0 && seq_len > 0;
}

static bool mla_pack_args_ok(int H, int dn, int dr, int dv) {
  return H > 0 && dn >= 8 && dr >= 8 && dv >= 8 && dn % 8 == 0 && dr % 8 == 0 && dv % 8 == 0 && dr <= 512;
}

}  // namespace tpb

using namespace tpb;

// kv [batch, tokens, H * (dn + dv)], rot: [batch, tokens] rows of dr values rot_ld elements apart; k [tokens, H, dn + dr] and
// v [tokens, H, dv] of a row of the batch are dense, k_batch and v_batch elements from the next row's; 16-byte aligned.
// (Into the caches of three layers without six copies: 2.5 % of a prefill of 900 tokens, 710 -> 686 us with the split above.)
extern "C" int tpb_mla_pack_rows(const void* kv, const void* rot, long long rot_ld, void* k, long long k_batch, void* v,
                                 long long v_batch, int batch, long long tokens, int H, int dn, int dr, int dv, void* stream) {
  if (!mla_pack_args_ok(H, dn, dr, dv) || rot_ld % 8 || k_batch % 8 || v_batch % 8 || batch > 65535) return -2;
  for (const void* a : {kv, rot, (const void*)k, (const void*)v})
    if (reinterpret_cast<uintptr_t>(a) % 16) return -2;
  if (tokens <= 0 || batch <= 0) return 0;
  const long long rows = (tokens + PACK_WARPS - 1) / PACK_WARPS;
  const dim3 grid((H + PACK_HEADS - 1) / PACK_HEADS, (unsigned)(rows < 65535 ? rows : 65535), batch);
  chain(mla_pack_kernel, grid, PACK_WARPS * 32, 0, reinterpret_cast<cudaStream_t>(stream), (const uint4*)kv, (const uint4*)rot,
        rot_ld / 8, (uint4*)k, (uint4*)v, tokens, H, dn / 8, dr / 8, dv / 8, k_batch / 8, v_batch / 8);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : 1000 + (int)e;
}

// The same of one dense row.
extern "C" int tpb_mla_pack(const void* kv, const void* rot, long long rot_ld, void* k, void* v, long long tokens, int H,
                            int dn, int dr, int dv, void* stream) {
  return tpb_mla_pack_rows(kv, rot, rot_ld, k, 0, v, 0, 1, tokens, H, dn, dr, dv, stream);
}

// dk [tokens, H, dn + dr], dv [tokens, H, dv] -> dkv [tokens, H * (dn + dv)], drot [tokens, dr].
extern "C" int tpb_mla_unpack(const void* dk, const void* dv_, void* dkv, void* drot, long long tokens, int H, int dn,
                              int dr, int dv, void* stream) {
  if (!mla_pack_args_ok(H, dn, dr, dv)) return -2;
  for (const void* a : {dk, dv_, (const void*)dkv, (const void*)drot})
    if (reinterpret_cast<uintptr_t>(a) % 16) return -2;
  if (tokens <= 0) return 0;
  const long long rows = (tokens + PACK_WARPS - 1) / PACK_WARPS;
  const dim3 grid(1 + (H + PACK_HEADS - 1) / PACK_HEADS, (unsigned)(rows < 65535 ? rows : 65535));
  chain(mla_unpack_kernel, grid, PACK_WARPS * 32, 0, reinterpret_cast<cudaStream_t>(stream),
        (const uint4*)dk, (const uint4*)dv_, (uint4*)dkv, (uint32_t*)drot, tokens, H, dn / 8, dr / 8, dv / 8);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : 1000 + (int)e;
}

// ckv [tokens, c + dr] -> lat [tokens, c], rot [tokens, dr] rotated (cos / sin [positions, dr / 2]; pos or token % seq_len).
extern "C" int tpb_latent_split(const void* ckv, void* lat, void* rot, const float* cosT, const float* sinT, const int* pos,
                                long long tokens, int seq_len, int c, int dr, int interleaved, void* stream) {
  if (!latent_args_ok({ckv, lat, rot}, c, dr, seq_len)) return -2;
  if (tokens <= 0) return 0;
  const long long blocks = (tokens * (c / 8 + dr / 16) + 255) / 256, cap = (long long)sm_count() * 16;
  cudaError_t e = chain(latent_kernel<true>, (int)(blocks < cap ? blocks : cap), 256, 0, reinterpret_cast<cudaStream_t>(stream),
                        (const uint4*)ckv, (uint4*)nullptr, (const uint4*)nullptr, (uint4*)lat, (const uint4*)nullptr, (uint4*)rot,
                        cosT, sinT, pos, tokens, seq_len, c / 8, dr / 8, interleaved);
  return e == cudaSuccess ? 0 : 1000 + (int)e;
}

// The gradient of that: dckv from dlat and drot.
extern "C" int tpb_latent_join(const void* dlat, const void* drot, void* dckv, const float* cosT, const float* sinT,
                               const int* pos, long long tokens, int seq_len, int c, int dr, int interleaved, void* stream) {
  if (!latent_args_ok({dlat, drot, dckv}, c, dr, seq_len)) return -2;
  if (tokens <= 0) return 0;
  const long long blocks = (tokens * (c / 8 + dr / 16) + 255) / 256, cap = (long long)sm_count() * 16;
  cudaError_t e = chain(latent_kernel<false>, (int)(blocks < cap ? blocks : cap), 256, 0, reinterpret_cast<cudaStream_t>(stream),
                        (const uint4*)nullptr, (uint4*)dckv, (const uint4*)dlat, (uint4*)nullptr, (const uint4*)drot,
                        (uint4*)nullptr, cosT, sinT, pos, tokens, seq_len, c / 8, dr / 8, interleaved);
  return e == cudaSuccess ? 0 : 1000 + (int)e;
}
