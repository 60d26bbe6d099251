// Keys and values of latent attention in the layout the attention kernels take, and back.
//
// The up-projection yields [token][head][dn key values | dv values]; every head's key is completed by the
// token's one rotary key.  Forward: k[t,h] = [kv[t,h,:dn] | rot[t]], v[t,h] = kv[t,h,dn:].  Backward: dkv from
// dk and dv, drot[t] = sum_h dk[t,h,dn:] (fp32, in a fixed order: heads modulo 256 / (dr / 8)
// first, then those groups).  One pass each, 16-byte vectors, bound by
// memory; as torch operators the same is a concatenation and a copy forward and seven launches backward
// (zero-filled slice gradients and their sum), each over the whole tensors: about 110 us together at 2048 tokens and
// 16 heads of 128 + 64 / 128, against 11 + 10 us.

#include <initializer_list>

#include "common.cuh"
#include "tpb.h"

namespace tpb {

int sm_count();

__global__ void mla_pack_kernel(const uint4* __restrict__ kv, const uint4* __restrict__ rot, long long rot_ld,
                                uint4* __restrict__ k, uint4* __restrict__ v, long long heads_total, int H, int dn8,
                                int dr8, int dv8) {
  if (!chain_begin()) return;
  const int per = dn8 + dr8 + dv8;
  const long long total = heads_total * per;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const long long th = i / per;
    const int j = (int)(i - th * per);
    if (j < dn8) k[th * (dn8 + dr8) + j] = kv[th * (dn8 + dv8) + j];
    else if (j < dn8 + dr8) k[th * (dn8 + dr8) + j] = rot[(th / H) * rot_ld + j - dn8];
    else v[th * dv8 + j - dn8 - dr8] = kv[th * (dn8 + dv8) + j - dr8];
  }
}

constexpr int UNPACK_THREADS = 256;

// One CTA per token (grid-stride).  drot: the rotary slice of every head, split over the threads as
// (vector of 8, head modulo G), met in shared memory in head-group order.
__global__ void __launch_bounds__(UNPACK_THREADS)
mla_unpack_kernel(const uint4* __restrict__ dk, const uint4* __restrict__ dv, uint4* __restrict__ dkv,
                  uint4* __restrict__ drot, long long tokens, int H, int dn8, int dr8, int dv8) {
  if (!chain_begin()) return;
  extern __shared__ float unpack_s[];            // [G][dr]
  const int G = UNPACK_THREADS / dr8, dr = dr8 * 8;
  for (long long t = blockIdx.x; t < tokens; t += gridDim.x) {
    const long long th0 = t * H;
    const int per = dn8 + dv8;
    for (int i = threadIdx.x; i < H * per; i += UNPACK_THREADS) {
      const int h = i / per, j = i - h * per;
      dkv[(th0 + h) * per + j] = j < dn8 ? dk[(th0 + h) * (dn8 + dr8) + j] : dv[(th0 + h) * dv8 + j - dn8];
    }
    const int vec = threadIdx.x % dr8, grp = threadIdx.x / dr8;
    if (grp < G) {
      float a[8] = {};
      for (int h = grp; h < H; h += G) {
        const uint4 u = dk[(th0 + h) * (dn8 + dr8) + dn8 + vec];
        const float2 x = unpack_bf16(u.x), y = unpack_bf16(u.y), z = unpack_bf16(u.z), w = unpack_bf16(u.w);
        a[0] += x.x; a[1] += x.y; a[2] += y.x; a[3] += y.y; a[4] += z.x; a[5] += z.y; a[6] += w.x; a[7] += w.y;
      }
#pragma unroll
      for (int e = 0; e < 8; ++e) unpack_s[grp * dr + vec * 8 + e] = a[e];
    }
    __syncthreads();
    const int used = min(G, H);
    if ((int)threadIdx.x < dr8) {
      float a[8] = {};
      for (int g = 0; g < used; ++g)
#pragma unroll
        for (int e = 0; e < 8; ++e) a[e] += unpack_s[g * dr + threadIdx.x * 8 + e];
      drot[t * dr8 + threadIdx.x] = make_uint4(pack_bf16(a[0], a[1]), pack_bf16(a[2], a[3]), pack_bf16(a[4], a[5]),
                                               pack_bf16(a[6], a[7]));
    }
    __syncthreads();
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

// kv [tokens, H * (dn + dv)], rot: [tokens] rows of dr values rot_ld elements apart; k [tokens, H, dn + dr],
// v [tokens, H, dv]; 16-byte aligned.
extern "C" int tpb_mla_pack(const void* kv, const void* rot, long long rot_ld, void* k, void* v, long long tokens, int H,
                            int dn, int dr, int dv, void* stream) {
  if (!mla_pack_args_ok(H, dn, dr, dv) || rot_ld % 8) return -2;
  for (const void* a : {kv, rot, (const void*)k, (const void*)v})
    if (reinterpret_cast<uintptr_t>(a) % 16) return -2;
  if (tokens <= 0) return 0;
  const long long items = tokens * H * ((dn + dr + dv) / 8);
  long long blocks = (items + 255) / 256, cap = (long long)sm_count() * 16;
  chain(mla_pack_kernel, (int)(blocks < cap ? blocks : cap), 256, 0, reinterpret_cast<cudaStream_t>(stream),
        (const uint4*)kv, (const uint4*)rot, rot_ld / 8, (uint4*)k, (uint4*)v, tokens * H, H, dn / 8, dr / 8, dv / 8);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : 1000 + (int)e;
}

// dk [tokens, H, dn + dr], dv [tokens, H, dv] -> dkv [tokens, H * (dn + dv)], drot [tokens, dr].
extern "C" int tpb_mla_unpack(const void* dk, const void* dv_, void* dkv, void* drot, long long tokens, int H, int dn,
                              int dr, int dv, void* stream) {
  if (!mla_pack_args_ok(H, dn, dr, dv)) return -2;
  for (const void* a : {dk, dv_, (const void*)dkv, (const void*)drot})
    if (reinterpret_cast<uintptr_t>(a) % 16) return -2;
  if (tokens <= 0) return 0;
  const long long cap = (long long)sm_count() * 8;
  const int smem = UNPACK_THREADS / (dr / 8) * dr * 4;
  chain(mla_unpack_kernel, (int)(tokens < cap ? tokens : cap), UNPACK_THREADS, smem, reinterpret_cast<cudaStream_t>(stream),
        (const uint4*)dk, (const uint4*)dv_, (uint4*)dkv, (uint4*)drot, tokens, H, dn / 8, dr / 8, dv / 8);
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
