// C [M, N] = A [M, K] . B [N, K]^T (+ bias) for up to 32 rows of A: the projections of a decode step with few sequences.
//
// Bound by reading B once. The tcgen05 kernel has 128 rows per tile whatever M is, and its chain (barriers, tensor memory, TMA,
// reduction of the K slices over a cluster) takes 7 us before a byte of B counts; here a block owns 16 * RT rows of B, its warps take
// turns along K, and their sums meet in shared memory. Products run on mma.m16n8k16 with the rows of B as its 16 and the rows of A as
// its 8: a lane's 16-byte loads are fragments as they come, since the order of k inside a product is free as long as both operands
// share it. fp32 sums, as in the tcgen05 kernel. While the kernel before it runs, a block asks for its first rows of B in L2 (a hint,
// so that it may come before the wait).
#include "common.cuh"
#include "host_utils.h"

namespace vb {

// Not the read-only path: the kernel before this one may write B (a product of two activations) while this one has begun already.
__device__ __forceinline__ uint4 ld_stream(const __nv_bfloat16* p) {
  uint4 v;
  asm volatile("ld.global.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
  return v;
}

constexpr int SK_WARPS = 8;

// NT: groups of 8 rows of A; RT: groups of 16 rows of B per warp; UB: 64-wide steps of k whose loads are in flight together.
// GLU (RT 2): B = [gate; up], 2 N rows; a block takes the same 16 rows of both and stores silu(gate) * up of their sums, rounded to bf16
// first as a product of its own would store them.
template <int NT, int RT, int UB, bool GLU = false>
__global__ void __launch_bounds__(SK_WARPS * 32, 2)
gemm_skinny_kernel(const __nv_bfloat16* A, const __nv_bfloat16* B, void* __restrict__ C, const __nv_bfloat16* bias, int M, int N, int K,
                   long long lda, long long ldb, long long ldc, int out_fp32) {
  constexpr int ROWS = 16 * RT, COLS = 8 * NT;
  __shared__ float red[SK_WARPS][ROWS][COLS + 1];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int n0 = blockIdx.x * (GLU ? 16 : ROWS);
  static_assert(!GLU || RT == 2, "16 rows of gate and of up");
  // row `i` of the block in B; rows past the ends repeat the last one: their sums are not stored
  auto row_of = [&](int i) { return GLU ? min(n0 + (i & 15), N - 1) + (i >> 4) * N : min(n0 + i, N - 1); };
  pdl_trigger();
  {
    const int lines = (K + 63) >> 6;  // of 128 bytes per row
    for (int i = threadIdx.x; i < ROWS * lines && i < 4 * SK_WARPS * 32; i += SK_WARPS * 32) {
      const __nv_bfloat16* p = B + (long long)row_of(i % ROWS) * ldb + (i / ROWS) * 64;
      asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
    }
  }
  pdl_wait();
  const __nv_bfloat16* b[RT * 2];
  const __nv_bfloat16* a[NT];
#pragma unroll
  for (int r = 0; r < RT * 2; ++r) b[r] = B + (long long)row_of(r * 8 + g) * ldb + t * 8;
#pragma unroll
  for (int j = 0; j < NT; ++j) a[j] = A + (long long)min(j * 8 + g, M - 1) * lda + t * 8;
  float acc[RT][NT][4] = {};
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  for (int k0 = warp * 64; k0 < K; k0 += SK_WARPS * 64 * UB) {
    uint4 w[UB][2][RT * 2], x[UB][2][NT];
#pragma unroll
    for (int u = 0; u < UB; ++u)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int k = k0 + u * (SK_WARPS * 64) + h * 32;
        const bool in = k + t * 8 < K;  // K is a multiple of 8
#pragma unroll
        for (int r = 0; r < RT * 2; ++r) w[u][h][r] = in ? ld_stream(b[r] + k) : zero;
#pragma unroll
        for (int j = 0; j < NT; ++j) x[u][h][j] = in ? *reinterpret_cast<const uint4*>(a[j] + k) : zero;
      }
#pragma unroll
    for (int u = 0; u < UB; ++u)
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int r = 0; r < RT; ++r)
#pragma unroll
          for (int j = 0; j < NT; ++j) {
            const uint4 lo = w[u][h][2 * r], hi = w[u][h][2 * r + 1], v = x[u][h][j];
            mma_bf16(acc[r][j], lo.x, hi.x, lo.y, hi.y, v.x, v.y);
            mma_bf16(acc[r][j], lo.z, hi.z, lo.w, hi.w, v.z, v.w);
          }
  }
#pragma unroll
  for (int r = 0; r < RT; ++r)
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int i = 0; i < 4; ++i) red[warp][r * 16 + (i >> 1) * 8 + g][j * 8 + 2 * t + (i & 1)] = acc[r][j][i];
  __syncthreads();
  if (GLU) {
    for (int i = threadIdx.x; i < 16 * COLS; i += SK_WARPS * 32) {
      const int n = n0 + i % 16, m = i / 16;
      if (n >= N || m >= M) continue;
      float gt = 0.f, up = 0.f;
#pragma unroll
      for (int v = 0; v < SK_WARPS; ++v) {
        gt += red[v][i % 16][m];
        up += red[v][ROWS - 16 + i % 16][m];
      }
      gt = __bfloat162float(__float2bfloat16(gt));
      up = __bfloat162float(__float2bfloat16(up));
      reinterpret_cast<__nv_bfloat16*>(C)[m * ldc + n] = __float2bfloat16(gt / (1.f + __expf(-gt)) * up);
    }
    return;
  }
  for (int i = threadIdx.x; i < ROWS * COLS; i += SK_WARPS * 32) {
    const int n = n0 + i % ROWS, m = i / ROWS;
    if (n >= N || m >= M) continue;
    float s = 0.f;
#pragma unroll
    for (int v = 0; v < SK_WARPS; ++v) s += red[v][i % ROWS][m];
    if (bias) s += __bfloat162float(bias[n]);
    if (out_fp32) reinterpret_cast<float*>(C)[m * ldc + n] = s;
    else reinterpret_cast<__nv_bfloat16*>(C)[m * ldc + n] = __float2bfloat16(s);
  }
}

}  // namespace vb

using namespace vb;

// Measured against the tcgen05 kernel, chains of launches on alternating matrices (us, M = 1 / 16 / 24 / 32; its own in brackets):
//   896 -> 1152    2.3 / 2.6 / 3.1 / 3.3 (6.8)           3584 -> 4608   6.5 / 7.9 / 8.9 / 10.3 (17.4, at 24 and 32: 15.3)
//   896 -> 9728    5.6 / 6.2 / 8.0 / 9.1 (14.6, 12.7)    2048 -> 5120   5.2 / 7.2 / 8.1 / 9.3 (13.5)
//   3584 -> 37888  45 / 59 / 67 / 81 (66 / 52 / 46 / 46)  18944 -> 3584  23 / 27 / 32 / 40 (30 to 38)
// Beyond 8 rows the loads of A (from L2, by every block) grow to those of B: where tiles of the tcgen05 kernel fill all SMs it is as
// fast at 16 rows and faster beyond, and with long rows (K) its staged operands win, the earlier the fewer SMs the blocks of 16 columns
// occupy. `most`: the longest K by rows (8, 16, 24, 32) and by N: fewer blocks than SMs, at most two blocks per SM, a second turn of the
// SMs that is nearly empty, more. us here (tcgen05), inside | outside, matrices from memory:
//    8 rows  768: 18944 16.8 (16.1) | 1792: 28672 25.9 (24.0)     5120: 14336 29.7 (32.1) | 18944 43.1 (39.8)    8192: 28672 72 (83)
//   16 rows  768: 7168 9.2 (9.6) | 10240 12.4 (11.4)    2304: 14336 19.3 (19.5) | 18944 25.2 (23.1)    3584: 18944 27.0 (29.5)
//            5120: 10240 25.0 (25.4) | 14336 34.1 (32.1)    6144: 28672 66 (78)
//   24 rows  768: 5120 8.5 (8.4) | 6144 10.0 (9.0)    2304: 8192 15.2 (15.2)    5120: 6144 17.6 (18.4) | 4864: 8192 23.1 (21.4)
//   32 rows  768: 3072 7.2 (7.2) | 4096 8.9 (7.8)     2304: 4096 10.5 (11.8)
bool vb_gemm_skinny_rows(int M, int N, int K) {
  constexpr int ANY = 0x7fffffff;
  static const int most[4][4] = {{20480, ANY, 16384, ANY}, {8192, 16384, 10240, ANY}, {5120, 8192, 6144, 8192}, {3072, 4096, 4096, 4096}};
  const int sms = vb_num_sms();
  if (M > 32 || (M > 8 && N >= 256 * sms)) return false;
  const int by_n = N < 16 * sms ? 0 : N <= 32 * sms ? 1 : N <= 40 * sms ? 2 : 3;
  return K <= most[(M - 1) / 8][by_n] || (M <= 16 && by_n == 1 && N >= 20 * sms && K <= 20480);
}
bool vb_gemm_skinny_ok(const void* A, const void* B, int M, int N, int K, long long lda, long long ldb) {
  const uintptr_t at = reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B);
  return !((K & 7) || (lda & 7) || (ldb & 7) || (at & 15)) && vb_gemm_skinny_rows(M, N, K);
}

extern "C" int vb_gemm_skinny(const void* A, const void* B, void* C, const void* bias, int M, int N, int K, long long lda,
                              long long ldb, long long ldc, int out_fp32, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if (!vb_gemm_skinny_ok(A, B, M, N, K, lda, ldb)) return -3;
  cudaError_t e;
#define VB_SKINNY(NT, RT, UB)                                                                                              \
  e = vb_launch_pdl(gemm_skinny_kernel<NT, RT, UB>, dim3((N + 16 * RT - 1) / (16 * RT)), dim3(SK_WARPS * 32), 0, stream, 1, \
                    (const __nv_bfloat16*)A, (const __nv_bfloat16*)B, C, (const __nv_bfloat16*)bias, M, N, K, lda, ldb, ldc, \
                    out_fp32)
  // 32 rows of B per block halve the loads of A; taken when the blocks still fill the SMs and their rows are long enough
  // (2048 -> 5120 at 32 rows: 9.3 us against 12.3; 3584 -> 4608, 144 blocks: 13.1 against 10.3)
  const bool two = N >= 32 * vb_num_sms() && K >= 2048;
  if (M <= 8) VB_SKINNY(1, 1, 4);
  else if (M <= 16 && two) VB_SKINNY(2, 2, 2);
  else if (M <= 16) VB_SKINNY(2, 1, 2);
  else if (M <= 24 && two) VB_SKINNY(3, 2, 1);
  else if (M <= 24) VB_SKINNY(3, 1, 1);
  else if (two) VB_SKINNY(4, 2, 1);
  else VB_SKINNY(4, 1, 1);
#undef VB_SKINNY
  vb_count_launch();
  return e != cudaSuccess ? (int)e : (int)cudaGetLastError();
}

// C [M, I] = silu(A . W[:I]^T) * (A . W[I:]^T) for up to 16 rows, rows and pointers as vb_gemm_skinny takes them.
int vb_gemm_skinny_swiglu(const void* A, const void* W, void* C, int M, int I, int K, long long lda, long long ldw, long long ldc,
                          cudaStream_t stream) {
  cudaError_t e;
#define VB_SKINNY(NT, UB)                                                                                                        \
  e = vb_launch_pdl(gemm_skinny_kernel<NT, 2, UB, true>, dim3((I + 15) / 16), dim3(SK_WARPS * 32), 0, stream, 1,                    \
                    (const __nv_bfloat16*)A, (const __nv_bfloat16*)W, C, (const __nv_bfloat16*)nullptr, M, I, K, lda, ldw, ldc, 0)
  if (M <= 8) VB_SKINNY(1, 2);
  else VB_SKINNY(2, 2);
#undef VB_SKINNY
  vb_count_launch();
  return e != cudaSuccess ? (int)e : (int)cudaGetLastError();
}
