// Block-scaled fp8 (e4m3) GEMM and the quantisation kernels that feed it.
//
// Scaling scheme of the reference's fp8 rollout path (verl/utils/kernel/fp8_kernel.py:53-106, 312;
// verl/utils/vllm/vllm_fp8_utils.py:182-431): weights carry one fp32 scale per 128 x 128 block, activations one per
// (row, 128 columns); scale = absmax / 448, optionally rounded up to a power of two (UE8M0-representable).
//
//   vb_fp8_quant_weight   W [N, K] bf16 -> Wq [N, K] e4m3 + sw [ceil(N/128), ceil(K/128)] fp32
//   vb_fp8_quant_act      X [M, K] bf16 -> Xq [M, K] e4m3 + sx [M, ceil(K/128)] fp32
//   vb_fp8_gemm_blockscale  C[M, N] (bf16) = sum over 128-wide k blocks of (Xq_kb . Wq_kb^T) * sx[m, kb] * sw[nb, kb]
//
// GEMM: one CTA per 128 x 128 output tile (persistent over tiles). Per k block the tensor core computes the
// unscaled partial product with tcgen05.mma kind::f8f6f4 (4 MMAs of K = 32) into one of two TMEM buffers; the four
// epilogue warps read the partial, multiply by the two scales and accumulate in registers while the MMA of the
// next k block runs into the other buffer ("promotion" of every 128-deep partial sum to fp32 outside the tensor
// core, which is what block scaling with plain fp32 scales requires).
//
// Up to 128 rows of X (decode steps) take fp8_gemm_skinny_kernel: W's rows are the MMA's 128 rows and X's rows its columns, so that the
// promotion costs a column per row of X instead of 128, and the CTAs of a cluster share a tile's K.
#include "common.cuh"
#include "host_utils.h"

#include <cuda_fp8.h>

namespace vb {

constexpr float FP8_MAX = 448.f;

__device__ __forceinline__ float scale_of(float amax, int pow2) {
  float s = fmaxf(amax, 1e-10f) / FP8_MAX;
  if (pow2) {
    // smallest power of two >= s, from the exponent bits (log2f under fast-math is not exact at powers of two)
    int e;
    const float m = frexpf(s, &e);  // s = m * 2^e, m in [0.5, 1)
    s = ldexpf(1.f, m == 0.5f ? e - 1 : e);
  }
  return s;
}

// one block (256 threads) per 128 x 128 tile of W
__global__ void fp8_quant_weight_kernel(const __nv_bfloat16* __restrict__ w, long long ldw, int N, int K,
                                        __nv_fp8_storage_t* __restrict__ q, long long ldq, float* __restrict__ scales,
                                        int pow2) {
  const int nb = blockIdx.y, kb = blockIdx.x;
  const int n0 = nb * 128, k0 = kb * 128;
  __shared__ float red[8];
  __shared__ float s_scale;
  float amax = 0.f;
  for (int i = threadIdx.x; i < 128 * 128; i += blockDim.x) {
    const int r = n0 + i / 128, c = k0 + i % 128;
    if (r < N && c < K) amax = fmaxf(amax, fabsf(__bfloat162float(w[(long long)r * ldw + c])));
  }
  amax = warp_reduce_max(amax);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = amax;
  __syncthreads();
  if (threadIdx.x == 0) {
    float m = 0.f;
    for (int i = 0; i < (int)(blockDim.x >> 5); ++i) m = fmaxf(m, red[i]);
    s_scale = scale_of(m, pow2);
    scales[(long long)nb * gridDim.x + kb] = s_scale;
  }
  __syncthreads();
  const float inv = 1.f / s_scale;
  for (int i = threadIdx.x; i < 128 * 128; i += blockDim.x) {
    const int r = n0 + i / 128, c = k0 + i % 128;
    if (r < N && c < K)
      q[(long long)r * ldq + c] = __nv_cvt_float_to_fp8(__bfloat162float(w[(long long)r * ldw + c]) * inv, __NV_SATFINITE, __NV_E4M3);
  }
}

// one warp per (row, 128-column block)
__global__ void fp8_quant_act_kernel(const __nv_bfloat16* x, long long ldx, long long M, int K,
                                     __nv_fp8_storage_t* __restrict__ q, long long ldq, float* __restrict__ scales, int pow2) {
  pdl_trigger();
  pdl_wait();
  const int nkb = (K + 127) / 128;
  const long long unit = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (unit >= M * nkb) return;
  const long long row = unit / nkb;
  const int kb = (int)(unit % nkb), lane = threadIdx.x & 31;
  const int c0 = kb * 128 + lane * 4;
  float v[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] = (c0 + i < K) ? __bfloat162float(x[row * ldx + c0 + i]) : 0.f;
  float amax = fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3])));
  amax = warp_reduce_max(amax);
  const float s = scale_of(amax, pow2), inv = 1.f / s;
  if (lane == 0) scales[row * nkb + kb] = s;
#pragma unroll
  for (int i = 0; i < 4; ++i)
    if (c0 + i < K) q[row * ldq + c0 + i] = __nv_cvt_float_to_fp8(v[i] * inv, __NV_SATFINITE, __NV_E4M3);
}

// ------------------------------------------------------------------------------------------------ GEMM
constexpr int F8_BM = 128, F8_BN = 128, F8_BK = 128;       // BK in elements = 128 bytes = one swizzle span
constexpr int F8_STAGES = 6;
constexpr int F8_TILE = 128 * 128;                          // 16 KB per operand tile
constexpr int F8_STAGE = 2 * F8_TILE;
constexpr int F8_BAR_OFF = F8_STAGES * F8_STAGE;
constexpr int F8_SMEM = F8_BAR_OFF + (2 * F8_STAGES + 4) * 8 + 16 + 1024;
constexpr int F8_THREADS = 192;

struct F8Params {
  int M, N, K;
  __nv_bfloat16* C;
  long long ldc;
  const float* sx;  // [M, nkb]
  const float* sw;  // [ceil(N/128), nkb]
  const __nv_bfloat16* bias;
  int* status;
};

__global__ void __launch_bounds__(F8_THREADS, 1)
fp8_gemm_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const F8Params p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + F8_BAR_OFF);
  uint64_t* empty = full + F8_STAGES;
  uint64_t* pfull = empty + F8_STAGES;   // [2] partial of a k block is in TMEM buffer i
  uint64_t* pempty = pfull + 2;          // [2] the epilogue warps have read buffer i
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(pempty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int num_m = (p.M + F8_BM - 1) / F8_BM, num_n = (p.N + F8_BN - 1) / F8_BN;
  const int num_kb = (p.K + F8_BK - 1) / F8_BK;
  const int num_tiles = num_m * num_n;

  if (threadIdx.x == 0) {
    for (int s = 0; s < F8_STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&pfull[i], 1);
      mbar_init(&pempty[i], 4);
    }
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 256);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    if (lane == 0) {
      tma_prefetch_desc(&tmA);
      tma_prefetch_desc(&tmB);
      int s = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int t = blockIdx.x; ok && t < num_tiles; t += gridDim.x) {
        const int mb = t % num_m, nb = t / num_m;
        for (int kb = 0; kb < num_kb; ++kb) {
          if (*abort_flag || !mbar_wait(&empty[s], phase ^ 1)) {
            report_error(p.status, ERR_WAIT_EMPTY, kb);
            *abort_flag = 1;
            ok = false;
            break;
          }
          mbar_arrive_expect_tx(&full[s], F8_STAGE);
          tma_load_2d(smem + s * F8_STAGE, &tmA, &full[s], kb * F8_BK, mb * F8_BM);
          tma_load_2d(smem + s * F8_STAGE + F8_TILE, &tmB, &full[s], kb * F8_BK, nb * F8_BN);
          if (++s == F8_STAGES) {
            s = 0;
            phase ^= 1;
          }
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      // kind::f8f6f4: formats 0 = e4m3 for both operands, K-major, fp32 accumulate, M = N = 128, K = 32 per MMA
      constexpr uint32_t idesc = umma_idesc(0, 0, 0, 0, F8_BM, F8_BN);
      int s = 0;
      uint32_t phase = 0;
      long long it = 0;  // running k-block counter: TMEM buffer = it & 1
      bool ok = true;
      for (int t = blockIdx.x; ok && t < num_tiles; t += gridDim.x) {
        for (int kb = 0; kb < num_kb; ++kb, ++it) {
          const int buf = (int)(it & 1);
          if (*abort_flag || !mbar_wait(&pempty[buf], (uint32_t)((it >> 1) & 1) ^ 1) || !mbar_wait(&full[s], phase)) {
            report_error(p.status, ERR_WAIT_FULL, kb);
            *abort_flag = 1;
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t a_addr = smem_u32(smem + s * F8_STAGE), b_addr = a_addr + F8_TILE;
#pragma unroll
          for (int k = 0; k < F8_BK / 32; ++k)
            tc_mma_f8(tmem_base + buf * F8_BN, umma_smem_desc(a_addr + k * 32, 16, 1024), umma_smem_desc(b_addr + k * 32, 16, 1024),
                      idesc, k != 0);
          tc_commit(&empty[s]);
          tc_commit(&pfull[buf]);
          if (++s == F8_STAGES) {
            s = 0;
            phase ^= 1;
          }
        }
      }
    }
  } else {
    const int quad = warp & 3;
    const int row_in_tile = quad * 32 + lane;
    const uint32_t lane_base = ((uint32_t)(quad * 32)) << 16;
    long long it = 0;
    bool ok = true;
    for (int t = blockIdx.x; ok && t < num_tiles; t += gridDim.x) {
      const int mb = t % num_m, nb = t / num_m;
      const int row = mb * F8_BM + row_in_tile;
      const bool row_ok = row < p.M;
      float acc[F8_BN];
#pragma unroll
      for (int i = 0; i < F8_BN; ++i) acc[i] = 0.f;
      for (int kb = 0; kb < num_kb; ++kb, ++it) {
        const int buf = (int)(it & 1);
        if (*abort_flag || !mbar_wait(&pfull[buf], (uint32_t)((it >> 1) & 1))) {
          report_error(p.status, ERR_WAIT_TMEM_FULL, kb);
          *abort_flag = 1;
          ok = false;
          break;
        }
        tc_fence_after();
        const float sc = (row_ok ? p.sx[(long long)row * num_kb + kb] : 0.f) * p.sw[(long long)nb * num_kb + kb];
#pragma unroll
        for (int c = 0; c < F8_BN / 32; ++c) {
          uint32_t v[32];
          tmem_ld_32x32(tmem_base + lane_base + buf * F8_BN + c * 32, v);
          tmem_ld_wait();
#pragma unroll
          for (int e = 0; e < 32; ++e) acc[c * 32 + e] = fmaf(__uint_as_float(v[e]), sc, acc[c * 32 + e]);
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&pempty[buf]);
      }
      if (ok && row_ok) {
        __nv_bfloat16* dst = p.C + (long long)row * p.ldc + nb * F8_BN;
        const int ncol = min(F8_BN, p.N - nb * F8_BN);
        if (p.bias != nullptr) {
#pragma unroll
          for (int i = 0; i < F8_BN; ++i)
            if (i < ncol) acc[i] += __bfloat162float(p.bias[nb * F8_BN + i]);
        }
        if (ncol == F8_BN && (p.ldc & 7) == 0) {
#pragma unroll
          for (int i = 0; i < F8_BN / 8; ++i) {
            uint4 w;
            w.x = pack_bf16x2(acc[8 * i], acc[8 * i + 1]);
            w.y = pack_bf16x2(acc[8 * i + 2], acc[8 * i + 3]);
            w.z = pack_bf16x2(acc[8 * i + 4], acc[8 * i + 5]);
            w.w = pack_bf16x2(acc[8 * i + 6], acc[8 * i + 7]);
            reinterpret_cast<uint4*>(dst)[i] = w;
          }
        } else {
#pragma unroll
          for (int i = 0; i < F8_BN; ++i)
            if (i < ncol) dst[i] = __float2bfloat16(acc[i]);
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 256);
  }
}

// ------------------------------------------------------------------------------------------------ decode
// C^T tile [128 rows of W, NT rows of X] per cluster of `splits` CTAs, each with its part of the k blocks. What bounds it is reading W
// once; the kernel above read 68 MB on 28 SMs with a promotion of 128 columns per k block (48 rows of X; 18 944 -> 3584: 69 us, now
// 18, floor 11). Partial products wait in F8S_BUFS tensor-memory buffers; the fp32 sums of a cluster meet in shared memory, in slice
// order. The first rows of W are asked for in L2 while the kernel before still runs (a hint, it may come before the wait).
constexpr int F8S_BUFS = 4;
template <int NT>
struct F8Skinny {
  static_assert(NT <= 64 && NT % 16 == 0, "two CTAs per SM");
  static constexpr int COLS = NT <= 32 ? 32 : 64;  // tensor-memory columns of a buffer
  static constexpr int BUFS = F8S_BUFS;
  static constexpr int STAGE = F8_TILE + NT * 128;
  static constexpr int STAGES = NT <= 32 ? 5 : 4;
  static constexpr int SCALE_OFF = STAGES * STAGE;                  // [4 warps][2][NT] fp32
  static constexpr int BAR_OFF = SCALE_OFF + 4 * 2 * NT * 4;
  static constexpr int SMEM = BAR_OFF + (2 * STAGES + 2 * BUFS) * 8 + 16 + 1024;
  static_assert(NT * 128 * 4 <= STAGES * STAGE, "the partial tile takes the stages' place");
};

template <int NT>
__global__ void __launch_bounds__(F8_THREADS, 2)
fp8_gemm_skinny_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const F8Params p,
                       const uint8_t* w, long long ldw, int m_tiles, int splits, int kb_per) {
  using L = F8Skinny<NT>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  float* scale_s = reinterpret_cast<float*>(smem + L::SCALE_OFF);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + L::BAR_OFF);
  uint64_t* empty = full + L::STAGES;
  uint64_t* pfull = empty + L::STAGES;  // the product of a k block is in TMEM buffer i
  uint64_t* pempty = pfull + L::BUFS;   // the epilogue warps have read buffer i
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(pempty + L::BUFS);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int num_kb = (p.K + F8_BK - 1) / F8_BK;
  const int rank = blockIdx.x % splits, nb = blockIdx.x / splits / m_tiles, m0 = blockIdx.x / splits % m_tiles * NT;
  const int kb0 = rank * kb_per, kb1 = min(num_kb, kb0 + kb_per);

  if (threadIdx.x == 0) {
    for (int s = 0; s < L::STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int i = 0; i < L::BUFS; ++i) {
      mbar_init(&pfull[i], 1);
      mbar_init(&pempty[i], 4);
    }
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, L::BUFS * L::COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_trigger();  // TMEM is held
  if (warp >= 2) {
    const int n = nb * F8_BN + (int)threadIdx.x - 64;  // a row of W per thread
    if (n < p.N)
      for (int kb = kb0; kb < min(kb1, kb0 + L::STAGES); ++kb)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(w + (long long)n * ldw + kb * F8_BK));
  }
  pdl_wait();

  bool ok = true;
  if (warp == 0) {
    if (lane == 0) {
      tma_prefetch_desc(&tmW);
      tma_prefetch_desc(&tmX);
      int s = 0, issued = 0;
      uint32_t phase = 0;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (*abort_flag || !mbar_wait(&empty[s], phase ^ 1)) {
          report_error(p.status, ERR_WAIT_EMPTY, kb);
          *abort_flag = 1;
          break;
        }
        mbar_arrive_expect_tx(&full[s], L::STAGE);
        tma_load_2d(smem + s * L::STAGE, &tmW, &full[s], kb * F8_BK, nb * F8_BN);
        tma_load_2d(smem + s * L::STAGE + F8_TILE, &tmX, &full[s], kb * F8_BK, m0);
        ++issued;
        if (++s == L::STAGES) {
          s = 0;
          phase ^= 1;
        }
      }
      // no copy outlives the CTA (after an error; else they have all been waited for)
      for (int i = max(0, issued - L::STAGES); i < issued; ++i) mbar_wait(&full[i % L::STAGES], (uint32_t)((i / L::STAGES) & 1));
    }
    __syncwarp();
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc = umma_idesc(0, 0, 0, 0, 128, NT);
      int s = 0;
      uint32_t phase = 0;
      for (int kb = kb0; kb < kb1; ++kb) {
        const int it = kb - kb0, buf = it % L::BUFS;
        if (*abort_flag || !mbar_wait(&pempty[buf], (uint32_t)((it / L::BUFS) & 1) ^ 1) || !mbar_wait(&full[s], phase)) {
          report_error(p.status, ERR_WAIT_FULL, kb);
          *abort_flag = 1;
          break;
        }
        tc_fence_after();
        const uint32_t w_addr = smem_u32(smem + s * L::STAGE), x_addr = w_addr + F8_TILE;
#pragma unroll
        for (int k = 0; k < F8_BK / 32; ++k)
          tc_mma_f8(tmem_base + buf * L::COLS, umma_smem_desc(w_addr + k * 32, 16, 1024), umma_smem_desc(x_addr + k * 32, 16, 1024),
                    idesc, k != 0);
        tc_commit(&empty[s]);
        tc_commit(&pfull[buf]);
        if (++s == L::STAGES) {
          s = 0;
          phase ^= 1;
        }
      }
    }
    __syncwarp();
  }
  float acc[NT];
  const int quad = warp & 3, row = quad * 32 + lane;  // row of the tile of W
  if (warp >= 2) {
    const uint32_t t_row = tmem_base + (((uint32_t)(quad * 32)) << 16);
    float* sc = scale_s + quad * 2 * NT;
#pragma unroll
    for (int i = 0; i < NT; ++i) acc[i] = 0.f;
    float next[(NT + 31) / 32];
    auto fetch = [&](int kb) {  // the scales of k block kb: of X's rows, a row per lane, times that of the tile of W
      if (kb >= kb1) return;
      const float sw = p.sw[(long long)nb * num_kb + kb];
#pragma unroll
      for (int j = 0; j < (NT + 31) / 32; ++j) {
        const int m = m0 + j * 32 + lane;
        next[j] = j * 32 + lane < NT && m < p.M ? p.sx[(long long)m * num_kb + kb] * sw : 0.f;
      }
    };
    fetch(kb0);
    for (int kb = kb0; kb < kb1; ++kb) {
      const int it = kb - kb0, buf = it % L::BUFS;
      float* mine = sc + (it & 1) * NT;  // read by this warp in the turn before the last: every lane has passed a barrier since
#pragma unroll
      for (int j = 0; j < (NT + 31) / 32; ++j)
        if (j * 32 + lane < NT) mine[j * 32 + lane] = next[j];
      __syncwarp();
      fetch(kb + 1);
      if (*abort_flag || !mbar_wait(&pfull[buf], (uint32_t)((it / L::BUFS) & 1))) {
        report_error(p.status, ERR_WAIT_TMEM_FULL, kb);
        *abort_flag = 1;
        ok = false;
        break;
      }
      __syncwarp();
      tc_fence_after();
      uint32_t v[NT / 16][16];
#pragma unroll
      for (int c = 0; c < NT / 16; ++c) tmem_ld_32x16(t_row + buf * L::COLS + c * 16, v[c]);
      tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < NT; i += 4) {
        const float4 f = *reinterpret_cast<const float4*>(mine + i);
        acc[i] = fmaf(__uint_as_float(v[i / 16][i % 16]), f.x, acc[i]);
        acc[i + 1] = fmaf(__uint_as_float(v[i / 16][i % 16 + 1]), f.y, acc[i + 1]);
        acc[i + 2] = fmaf(__uint_as_float(v[i / 16][i % 16 + 2]), f.z, acc[i + 2]);
        acc[i + 3] = fmaf(__uint_as_float(v[i / 16][i % 16 + 3]), f.w, acc[i + 3]);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&pempty[buf]);
    }
  }
  const int rows = min(NT, p.M - m0);
  if (splits == 1) {
    const int n = nb * F8_BN + row;
    if (warp >= 2 && ok && n < p.N) {
      const float b = p.bias ? __bfloat162float(p.bias[n]) : 0.f;
#pragma unroll
      for (int m = 0; m < NT; ++m)
        if (m < rows) p.C[(long long)(m0 + m) * p.ldc + n] = __float2bfloat16(acc[m] + b);
    }
  } else {
    // all products of this CTA have been read, so its stages are idle: [NT][128] fp32
    float* part = reinterpret_cast<float*>(smem);
    __syncthreads();
    if (warp >= 2) {
#pragma unroll
      for (int m = 0; m < NT; ++m) part[m * 128 + row] = acc[m];
    }
    cluster_sync_all();
    // a warp per row of X, four columns per lane, the loads of all slices in flight together
    const int n = nb * F8_BN + lane * 4;
    float b[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) b[i] = p.bias && n + i < p.N ? __bfloat162float(p.bias[n + i]) : 0.f;
    const bool whole = n + 4 <= p.N && (p.ldc & 3) == 0 && (reinterpret_cast<uintptr_t>(p.C) & 7) == 0;
    for (int m = rank + splits * warp; m < rows; m += splits * (F8_THREADS / 32)) {
      const uint32_t at = smem_u32(part + m * 128 + lane * 4);
      float4 v[8];
#pragma unroll
      for (int r = 0; r < 8; ++r)
        if (r < splits)
          asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                       : "=f"(v[r].x), "=f"(v[r].y), "=f"(v[r].z), "=f"(v[r].w)
                       : "r"(map_to_cta(at, r)));
      float sum[4] = {};
#pragma unroll
      for (int r = 0; r < 8; ++r)
        if (r < splits) {
          sum[0] += v[r].x;
          sum[1] += v[r].y;
          sum[2] += v[r].z;
          sum[3] += v[r].w;
        }
      __nv_bfloat16* c = p.C + (long long)(m0 + m) * p.ldc + n;
      if (whole) {
        *reinterpret_cast<uint2*>(c) = make_uint2(pack_bf16x2(sum[0] + b[0], sum[1] + b[1]), pack_bf16x2(sum[2] + b[2], sum[3] + b[3]));
      } else {
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (n + i < p.N) c[i] = __float2bfloat16(sum[i] + b[i]);
      }
    }
    cluster_sync_all();  // the others have read this CTA's part
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, L::BUFS * L::COLS);
  }
}

template <int NT>
static int launch_fp8_skinny(const void* xq, const void* wq, long long ldx, long long ldw, const F8Params& p, cudaStream_t stream) {
  using L = F8Skinny<NT>;
  CUtensorMap tmW, tmX;
  int rc = vb_make_tmap_2d(&tmW, wq, 1, (uint64_t)p.K, (uint64_t)p.N, (uint64_t)ldw, F8_BK, 128);
  if (rc) return rc;
  rc = vb_make_tmap_2d(&tmX, xq, 1, (uint64_t)p.K, (uint64_t)p.M, (uint64_t)ldx, F8_BK, NT);
  if (rc) return rc;
  auto kern = fp8_gemm_skinny_kernel<NT>;
  static bool attr_set[64] = {};
  int dev = 0;
  VB_CUDA_CHECK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64 || !attr_set[dev]) {
    VB_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::SMEM));
    if (dev >= 0 && dev < 64) attr_set[dev] = true;
  }
  // The most CTAs of about one wave (two per SM, less what clusters leave idle in a part of the chip: 288 of 296 took longer than 216),
  // six k blocks or more per CTA: below, the cluster's exchange costs more than it gives. Waves are not asked from the occupancy
  // calculator: it allowed 28 clusters of four where 28 of eight run (18 944 -> 3584, 48 rows: 25.5 against 17.8 us).
  const int m_tiles = (p.M + NT - 1) / NT, tiles = (p.N + 127) / 128 * m_tiles, nkb = (p.K + F8_BK - 1) / F8_BK;
  int splits = 1, per = nkb;
  for (int s = 2; s <= 8 && s * 6 <= nkb && tiles * s * 4 <= 7 * vb_num_sms(); ++s) {
    const int each = (nkb + s - 1) / s;
    if ((nkb + each - 1) / each != s) continue;
    splits = s;
    per = each;
  }
  cudaError_t e = vb_launch_ex(kern, dim3(tiles * splits), dim3(F8_THREADS), L::SMEM, stream, (unsigned)splits, true, tmW, tmX, p,
                               (const uint8_t*)wq, ldw, m_tiles, splits, per);
  vb_count_launch();
  return e != cudaSuccess ? (int)e : (int)cudaGetLastError();
}

}  // namespace vb

using namespace vb;

// W [N, K] bf16 (row stride ldw) -> q [N, K] e4m3 (row stride ldq, a multiple of 16) + scales [ceil(N/128), ceil(K/128)].
extern "C" int vb_fp8_quant_weight(const void* w, long long ldw, int N, int K, void* q, long long ldq, float* scales, int pow2,
                                   cudaStream_t stream) {
  if (N <= 0 || K <= 0) return 0;
  dim3 grid((K + 127) / 128, (N + 127) / 128);
  fp8_quant_weight_kernel<<<grid, 256, 0, stream>>>(reinterpret_cast<const __nv_bfloat16*>(w), ldw, N, K,
                                                    reinterpret_cast<__nv_fp8_storage_t*>(q), ldq, scales, pow2);
  vb_count_launch();
  return (int)cudaGetLastError();
}

// X [M, K] bf16 -> q [M, K] e4m3 + scales [M, ceil(K/128)].
extern "C" int vb_fp8_quant_act(const void* x, long long ldx, long long M, int K, void* q, long long ldq, float* scales,
                                int pow2, cudaStream_t stream) {
  if (M <= 0 || K <= 0) return 0;
  const long long units = M * ((K + 127) / 128);
  cudaError_t e = vb_launch_pdl(fp8_quant_act_kernel, dim3((unsigned)((units + 7) / 8)), dim3(256), 0, stream, 1,
                                reinterpret_cast<const __nv_bfloat16*>(x), ldx, M, K, reinterpret_cast<__nv_fp8_storage_t*>(q), ldq,
                                scales, pow2);
  vb_count_launch();
  return e != cudaSuccess ? (int)e : (int)cudaGetLastError();
}

// C [M, N] bf16 = dequantised Xq . Wq^T (+ bias). Xq [M, K], Wq [N, K] e4m3 with row strides (bytes = elements)
// that are multiples of 16; sx [M, ceil(K/128)], sw [ceil(N/128), ceil(K/128)] fp32.
extern "C" int vb_fp8_gemm_blockscale(const void* xq, const void* wq, const float* sx, const float* sw, void* C,
                                      const void* bias, int M, int N, int K, long long ldx, long long ldw, long long ldc,
                                      int* status, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if ((ldx & 15) || (ldw & 15)) return -3;
  F8Params p{};
  p.M = M; p.N = N; p.K = K;
  p.C = reinterpret_cast<__nv_bfloat16*>(C); p.ldc = ldc;
  p.sx = sx; p.sw = sw; p.bias = reinterpret_cast<const __nv_bfloat16*>(bias); p.status = status;
  // us, the kernel below -> the decode kernel (M = 1 / 48 / 64 / 96 / 128):
  //   3584 -> 4608   16 -> 7.0 / 8.9 / 10 / 12 / 14   18944 -> 3584  68 -> 14 / 18 / 22 / 26 / 33   4096 -> 6144  18 -> 8.1 / 11 / 13 / 19 / 20
  //   3584 -> 37888  36 -> 24 / 26 / 28 / 34 / 34     4096 -> 28672  40 -> 21 / 27 / 32 / 36 / 37    4864 -> 896   20 -> 6.2 / 7.6 / 8.5 / 8.3 / 9.5
  // More than 64 rows of X are two tiles, which read W twice (from L2): worth it while all tiles together leave half of the SMs
  // without one, so that the kernel below would, too.
  if (M <= 16) return launch_fp8_skinny<16>(xq, wq, ldx, ldw, p, stream);
  if (M <= 32) return launch_fp8_skinny<32>(xq, wq, ldx, ldw, p, stream);
  if (M <= 48) return launch_fp8_skinny<48>(xq, wq, ldx, ldw, p, stream);
  if (M <= 64) return launch_fp8_skinny<64>(xq, wq, ldx, ldw, p, stream);
  if (M <= 128 && (N + 127) / 128 * 4 <= vb_num_sms())
    return M <= 96 ? launch_fp8_skinny<48>(xq, wq, ldx, ldw, p, stream) : launch_fp8_skinny<64>(xq, wq, ldx, ldw, p, stream);
  CUtensorMap tmA, tmB;
  int rc = vb_make_tmap_2d(&tmA, xq, 1, (uint64_t)K, (uint64_t)M, (uint64_t)ldx, F8_BK, F8_BM);
  if (rc) return rc;
  rc = vb_make_tmap_2d(&tmB, wq, 1, (uint64_t)K, (uint64_t)N, (uint64_t)ldw, F8_BK, F8_BN);
  if (rc) return rc;
  static bool attr_set = false;
  if (!attr_set) {
    VB_CUDA_CHECK(cudaFuncSetAttribute(fp8_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, F8_SMEM));
    attr_set = true;
  }
  const int tiles = ((M + F8_BM - 1) / F8_BM) * ((N + F8_BN - 1) / F8_BN);
  const int grid = tiles < vb_num_sms() ? tiles : vb_num_sms();
  fp8_gemm_kernel<<<grid, F8_THREADS, F8_SMEM, stream>>>(tmA, tmB, p);
  vb_count_launch();
  return (int)cudaGetLastError();
}
