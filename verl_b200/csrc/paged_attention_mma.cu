// Paged-KV decode attention on tensor cores, fragments straight from the paged cache ([num_blocks, Hk, block_size, D] bf16, block_size
// a power of two of 8 or more, D 64 or 128, up to 16 query heads per KV head).
//
// Bound by reading K and V once; with few sequences by the chain from the block table to the result. A CTA of four warps serves one
// (sequence, KV head, split); its warps take 16 keys in turn and share nothing before the end: no ring of tiles, no barriers, no
// block-wide maximum per 128 keys. Calls in a chain, us, in brackets the tcgen05 kernel it replaced, which staged 128-key tiles by TMA
// (D 64: the CUDA-core kernel), and the time of the bytes:
//   128 sequences of 430, 28 / 4 heads of 128: 31.8 (47.3; 17.0)     48 of 500: 17.0 (35.1; 7.7)     1 of 8000: 16.4 (19.8; 2.3)
//   256 of 1000: 99.5 (147.8; 81.5)     128 of 1000, 32 / 8 heads: 95.8 (123.1; 80.5)     16 of 4000: 33.0 (54.0; 20.5)
//   14 / 2 heads of 64: 1 of 85 2.8 (15.8)     16 of 500 5.6 (21.1; 0.6)     128 of 500 9.2 (40.5; 5.1)
//
//   S[heads, keys]  = Q[16, D] . K^T   mma.m16n8k16; the order of dims inside a product is free as long as Q and K share it, so a
//                                      lane's 16 bytes of a key are two steps' operands as they come
//   O^T[dims, heads] += V^T . P^T      P: the scores' own registers, as bf16; V's operand holds two keys of a dim per register: a lane
//                                      loads 16 bytes of four keys and pairs them
//
// Heads of 64, and pages above 128 rows, keep their weights in fp32: three bf16 terms hold all 24 bits, their products of 16 keys are
// summed on their own and added to the rest with rounding to nearest. Against 64 bits (relative 2-norm before the result is rounded) 1.7e-7
// to 2.5e-7, on CUDA cores 1.9e-7 to 4.5e-7, with one term 1.2e-3 (which moves a bf16 result from 1.6e-3 to 2.0e-3); one term would be 0.1 to
// 0.2 us faster. Heads of 128 in smaller pages take one term, as the tcgen05 kernel did (1.2e-3, that one 1.4e-3): three would take 10 to 20 %
// longer there (128 of 430: 36.8 us, 30.9 with one).
//
// Next keys' K loads are in flight while V and the softmax of these are worked on. fp32 softmax, base 2, online per warp.
#include "common.cuh"
#include "host_utils.h"

namespace vb {

constexpr int DM_WARPS = 4, DM_CHUNK = 128;  // the keys of a split: whole chunks (vb_decode_num_splits)

__device__ __forceinline__ uint32_t word(const uint4& v, int i) { return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w; }

// HI: more than eight query heads per KV head (rows 8 .. 15 of the products hold some). TERMS: bf16 terms that a weight is cut into.
template <int D, bool HI, int TERMS>
__global__ void __launch_bounds__(DM_WARPS * 32, HI ? 2 : 3)
paged_decode_mma_kernel(const __nv_bfloat16* q, long long q_stride, const __nv_bfloat16* kc, const __nv_bfloat16* vc,
                        const int* block_table, int max_blocks, const int* seq_lens, int Hq, int Hk, int shift, float scale_log2,
                        int num_splits, __nv_bfloat16* __restrict__ out, long long out_stride, float* __restrict__ o_part,
                        float* __restrict__ ml_part) {
  constexpr int KI = D / 32, VC = D / 64, ROWS = HI ? 16 : 8, R = HI ? 2 : 1;
  __shared__ float o_s[DM_WARPS][ROWS][D + 4];
  __shared__ float2 ml_s[DM_WARPS][ROWS];
  const int b = blockIdx.x, h = blockIdx.y, split = blockIdx.z;
  const int G = Hq / Hk, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int page_mask = (1 << shift) - 1;
  pdl_trigger();
  pdl_wait();
  const int seq_len = seq_lens[b];
  const int chunks = (seq_len + DM_CHUNK - 1) / DM_CHUNK, per_split = (chunks + num_splits - 1) / num_splits;
  const int k_begin = split * per_split * DM_CHUNK, k_end = min(seq_len, k_begin + per_split * DM_CHUNK);
  const int* table = block_table + (long long)b * max_blocks;
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);

  uint4 qf[KI][R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int head = g + 8 * r;
    const __nv_bfloat16* row = q + (long long)b * q_stride + (long long)(h * G + head) * D + t * 8;
    const bool vec = (reinterpret_cast<uintptr_t>(row) & 15) == 0;
#pragma unroll
    for (int i = 0; i < KI; ++i) {
      qf[i][r] = zero;
      if (head < G) {
        if (vec) {
          qf[i][r] = *reinterpret_cast<const uint4*>(row + i * 32);
        } else {
          const unsigned short* s = reinterpret_cast<const unsigned short*>(row + i * 32);
          qf[i][r] = make_uint4(s[0] | (uint32_t)s[1] << 16, s[2] | (uint32_t)s[3] << 16, s[4] | (uint32_t)s[5] << 16,
                                s[6] | (uint32_t)s[7] << 16);
        }
      }
    }
  }
  // row of the cache of the first of the eight keys at `key`; past the end: of the last eight (nothing is read there)
  auto cache_row = [&](int key) {
    key = min(key, (seq_len - 1) & ~7);
    return (((long long)table[key >> shift] * Hk + h) << shift) + (key & page_mask);
  };

  float m[R], l[R], acc[R][VC][4][4];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    m[r] = -INFINITY;
    l[r] = 0.f;
  }
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int c = 0; c < VC; ++c)
#pragma unroll
      for (int e = 0; e < 4; ++e)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[r][c][e][i] = 0.f;

  int key0 = k_begin + warp * 16;
  uint4 kf[2][KI];
  long long row[2];
  auto load_k = [&]() {
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int i = 0; i < KI; ++i) {
        kf[j][i] = zero;
        if (key0 + j * 8 + g < k_end) kf[j][i] = *reinterpret_cast<const uint4*>(kc + (row[j] + g) * D + i * 32 + t * 8);
      }
  };
  if (key0 < k_end) {
    row[0] = cache_row(key0);
    row[1] = cache_row(key0 + 8);
    load_k();
  }
  while (key0 < k_end) {
    uint4 vf[VC][4];
#pragma unroll
    for (int c = 0; c < VC; ++c)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int in8 = 2 * t + (j & 1);
        vf[c][j] = zero;
        if (key0 + (j >> 1) * 8 + in8 < k_end)
          vf[c][j] = *reinterpret_cast<const uint4*>(vc + (row[j >> 1] + in8) * D + c * 64 + g * 8);
      }
    float s[2][4] = {};
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int i = 0; i < KI; ++i) {
        const uint4 a = qf[i][0], a8 = HI ? qf[i][R - 1] : zero;
        mma_bf16(s[j], a.x, a8.x, a.y, a8.y, kf[j][i].x, kf[j][i].y);
        mma_bf16(s[j], a.z, a8.z, a.w, a8.w, kf[j][i].z, kf[j][i].w);
      }
    const int now = key0;
    key0 += DM_WARPS * 16;
    if (key0 < k_end) {
      row[0] = cache_row(key0);
      row[1] = cache_row(key0 + 8);
      load_k();
    }
    uint32_t p[TERMS][2][R];  // [term][eight keys][row]: bf16 pairs
#pragma unroll
    for (int r = 0; r < R; ++r) {
      float x[4], nm = m[r];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        x[i] = now + (i >> 1) * 8 + 2 * t + (i & 1) < k_end ? s[i >> 1][2 * r + (i & 1)] * scale_log2 : -INFINITY;
        nm = fmaxf(nm, x[i]);
      }
      nm = fmaxf(nm, __shfl_xor_sync(0xffffffffu, nm, 1));
      nm = fmaxf(nm, __shfl_xor_sync(0xffffffffu, nm, 2));
      const float to = nm == -INFINITY ? 0.f : nm, alpha = exp2f(m[r] - to);
      m[r] = nm;
      l[r] *= alpha;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        x[i] = exp2f(x[i] - to);
        l[r] += x[i];
      }
#pragma unroll
      for (int n = 0; n < TERMS; ++n)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          p[n][j][r] = pack_bf16x2(x[2 * j], x[2 * j + 1]);
          x[2 * j] -= __uint_as_float(p[n][j][r] << 16);
          x[2 * j + 1] -= __uint_as_float(p[n][j][r] & 0xffff0000u);
        }
      if (__any_sync(0xffffffffu, alpha != 1.f)) {
        const float a0 = __shfl_sync(0xffffffffu, alpha, 8 * t), a1 = __shfl_sync(0xffffffffu, alpha, 8 * t + 4);  // heads 2t, 2t + 1
#pragma unroll
        for (int c = 0; c < VC; ++c)
#pragma unroll
          for (int e = 0; e < 4; ++e)
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[r][c][e][i] *= (i & 1) ? a1 : a0;
      }
    }
#pragma unroll
    for (int c = 0; c < VC; ++c)
#pragma unroll
      for (int e = 0; e < 4; ++e) {  // rows of the product: dims 2e and 2e + 1 of the lane's eight
        const uint32_t k0 = word(vf[c][0], e), k1 = word(vf[c][1], e), k2 = word(vf[c][2], e), k3 = word(vf[c][3], e);
        const uint32_t a0 = __byte_perm(k0, k1, 0x5410), a1 = __byte_perm(k0, k1, 0x7632);
        const uint32_t a2 = __byte_perm(k2, k3, 0x5410), a3 = __byte_perm(k2, k3, 0x7632);
#pragma unroll
        for (int r = 0; r < R; ++r) {
          if (TERMS == 1) {
            mma_bf16(acc[r][c][e], a0, a1, a2, a3, p[0][0][r], p[0][1][r]);
          } else {  // 16 keys on their own, then a sum that is rounded to nearest
            float part[4] = {};
#pragma unroll
            for (int n = TERMS - 1; n >= 0; --n) mma_bf16(part, a0, a1, a2, a3, p[n][0][r], p[n][1][r]);
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[r][c][e][i] += part[i];
          }
        }
      }
  }

  // the warps' results: rows g and g + 8 of product (c, e) are dims 64 c + 8 g + 2 e and the next one, its columns heads
#pragma unroll
  for (int r = 0; r < R; ++r) {
    l[r] += __shfl_xor_sync(0xffffffffu, l[r], 1);
    l[r] += __shfl_xor_sync(0xffffffffu, l[r], 2);
    if (t == 0) ml_s[warp][g + 8 * r] = make_float2(m[r], l[r]);
#pragma unroll
    for (int c = 0; c < VC; ++c)
#pragma unroll
      for (int e = 0; e < 4; ++e)
#pragma unroll
        for (int i = 0; i < 2; ++i)
          *reinterpret_cast<float2*>(&o_s[warp][2 * t + i + 8 * r][c * 64 + g * 8 + e * 2]) = make_float2(acc[r][c][e][i], acc[r][c][e][2 + i]);
  }
  __syncthreads();
  for (int i = tid; i < G * D; i += DM_WARPS * 32) {
    const int head = i / D, d = i % D;
    float mx = -INFINITY, ls = 0.f, o = 0.f;
#pragma unroll
    for (int w = 0; w < DM_WARPS; ++w) mx = fmaxf(mx, ml_s[w][head].x);
    const float to = mx == -INFINITY ? 0.f : mx;
#pragma unroll
    for (int w = 0; w < DM_WARPS; ++w) {
      const float f = exp2f(ml_s[w][head].x - to);
      ls += ml_s[w][head].y * f;
      o += o_s[w][head][d] * f;
    }
    const int hq = h * G + head;
    if (num_splits == 1) {
      out[(long long)b * out_stride + (long long)hq * D + d] = __float2bfloat16(ls > 0.f ? o / ls : 0.f);
    } else {
      const long long at = ((long long)b * Hq + hq) * num_splits + split;
      o_part[at * D + d] = o;
      if (d == 0) {
        ml_part[at * 2] = mx * 0.6931471805599453f;  // the merge takes natural exponents
        ml_part[at * 2 + 1] = ls;
      }
    }
  }
}

}  // namespace vb

using namespace vb;

int vb_decode_merge_parts(const float* o_part, const float* ml_part, int B, int Hq, int D, int num_splits, void* out, long long out_stride,
                          cudaStream_t stream);  // paged_attention.cu

extern "C" int vb_paged_decode_mma_supported(int Hq, int Hk, int D, int block_size) {
  return (D == 64 || D == 128) && Hk > 0 && Hq % Hk == 0 && Hq / Hk >= 1 && Hq / Hk <= 16 && block_size >= 8 &&
         (block_size & (block_size - 1)) == 0;
}

// Arguments as vb_paged_decode; kc and vc on 16-byte boundaries.
extern "C" int vb_paged_decode_mma(const void* q, long long q_stride, const void* kc, const void* vc, const int* block_table,
                                   int max_blocks, const int* seq_lens, int B, int Hq, int Hk, int D, int block_size, float scale,
                                   int num_splits, void* out, long long out_stride, float* work, cudaStream_t stream) {
  if (B <= 0) return 0;
  if (!vb_paged_decode_mma_supported(Hq, Hk, D, block_size) || num_splits < 1 || (num_splits > 1 && work == nullptr) ||
      ((reinterpret_cast<uintptr_t>(kc) | reinterpret_cast<uintptr_t>(vc)) & 15) != 0)
    return -3;
  float* ml_part = work ? work + (long long)B * Hq * num_splits * D : nullptr;
  int shift = 0;
  while ((1 << shift) < block_size) ++shift;
  const float scale_log2 = scale * 1.4426950408889634f;
  cudaError_t e;
#define VB_DM(DD, HI, TERMS)                                                                                                     \
  e = vb_launch_pdl(paged_decode_mma_kernel<DD, HI, TERMS>, dim3(B, Hk, num_splits), dim3(DM_WARPS * 32), 0, stream, 1,           \
                    (const __nv_bfloat16*)q, q_stride, (const __nv_bfloat16*)kc, (const __nv_bfloat16*)vc, block_table, max_blocks, \
                    seq_lens, Hq, Hk, shift, scale_log2, num_splits, (__nv_bfloat16*)out, out_stride, work, ml_part)
  const bool hi = Hq / Hk > 8;
  if (D == 64 && hi) VB_DM(64, true, 3);
  else if (D == 64) VB_DM(64, false, 3);
  else if (block_size > 128 && hi) VB_DM(128, true, 3);
  else if (block_size > 128) VB_DM(128, false, 3);
  else if (hi) VB_DM(128, true, 1);
  else VB_DM(128, false, 1);
#undef VB_DM
  vb_count_launch(num_splits > 1 ? 2 : 1);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess || num_splits == 1) return (int)e;
  return vb_decode_merge_parts(work, ml_part, B, Hq, D, num_splits, out, out_stride, stream);
}
