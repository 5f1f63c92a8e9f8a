// Memory-bound model kernels: RMSNorm (with fused residual add), rotary embedding,
// SwiGLU, embedding gather/scatter, fused AdamW on flat shards, squared-norm reduction.
// All use 16-byte vector accesses; bf16 storage, fp32 math.
//
// These replace what the reference gets from HF eager / liger / apex
// (verl/models/llama/megatron/layers/parallel_rmsnorm.py:40-49, parallel_mlp.py) and
// torch.optim.AdamW + clip_grad_norm_ (verl/workers/actor/dp_actor.py:391-415).
#include "common.cuh"
#include "host_utils.h"

namespace vb {

struct alignas(16) bf16x8 {
  __nv_bfloat162 v[4];
};

__device__ __forceinline__ void load8(const __nv_bfloat16* p, float (&f)[8]) {
  bf16x8 t = *reinterpret_cast<const bf16x8*>(p);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 x = __bfloat1622float2(t.v[i]);
    f[2 * i] = x.x;
    f[2 * i + 1] = x.y;
  }
}
__device__ __forceinline__ void store8(__nv_bfloat16* p, const float (&f)[8]) {
  bf16x8 t;
#pragma unroll
  for (int i = 0; i < 4; ++i) t.v[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  *reinterpret_cast<bf16x8*>(p) = t;
}

__device__ __forceinline__ float block_reduce_sum(float v, float* sh) {
  v = warp_reduce_sum(v);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nw = (blockDim.x + 31) >> 5;
  __syncthreads();
  if (lane == 0) sh[warp] = v;
  __syncthreads();
  float t = (lane < nw) ? sh[lane] : 0.f;
  t = warp_reduce_sum(t);
  return t;
}

// ------------------------------- RMSNorm ------------------------------------
// y = (x [+ res]) * rstd * w ; optionally writes the pre-norm sum to res_out.
__global__ void rmsnorm_fwd_kernel(const __nv_bfloat16* x, const __nv_bfloat16* res,
                                   const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ y,
                                   __nv_bfloat16* __restrict__ res_out, float* __restrict__ rstd_out, int H,
                                   float eps) {
  __shared__ float sh[32];
  pdl_trigger();
  pdl_wait();
  const long long row = blockIdx.x;
  const __nv_bfloat16* xr = x + row * H;
  const int nvec = H >> 3;
  float ss = 0.f;
  for (int v = threadIdx.x; v < nvec; v += blockDim.x) {
    float f[8];
    load8(xr + v * 8, f);
    if (res) {
      float g[8];
      load8(res + row * H + v * 8, g);
#pragma unroll
      for (int i = 0; i < 8; ++i) f[i] += g[i];
      if (res_out) {
        store8(res_out + row * H + v * 8, f);
        // re-round so the norm sees exactly what later layers will read
        load8(res_out + row * H + v * 8, f);
      }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) ss += f[i] * f[i];
  }
  ss = block_reduce_sum(ss, sh);
  const float rstd = rsqrtf(ss / H + eps);
  if (threadIdx.x == 0 && rstd_out) rstd_out[row] = rstd;
  const __nv_bfloat16* src = (res && res_out) ? (res_out + row * H) : xr;
  for (int v = threadIdx.x; v < nvec; v += blockDim.x) {
    float f[8], wv[8];
    load8(src + v * 8, f);
    if (res && !res_out) {
      float g[8];
      load8(res + row * H + v * 8, g);
#pragma unroll
      for (int i = 0; i < 8; ++i) f[i] += g[i];
    }
    load8(w + v * 8, wv);
#pragma unroll
    for (int i = 0; i < 8; ++i) f[i] = f[i] * rstd * wv[i];
    store8(y + row * H + v * 8, f);
  }
}

// dx = rstd * (g - xhat * mean(g * xhat)), g = dy * w ; optionally dx += dres (gradient
// arriving through the residual path). dw partial sums go to dw_partial[gridDim.x, H].
__global__ void rmsnorm_bwd_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x,
                                   const __nv_bfloat16* __restrict__ w, const float* __restrict__ rstd,
                                   const __nv_bfloat16* __restrict__ dres, __nv_bfloat16* __restrict__ dx,
                                   float* __restrict__ dw_partial, int rows, int H) {
  extern __shared__ float dw_acc[];  // [H]
  __shared__ float sh[32];
  const int nvec = H >> 3;
  for (int i = threadIdx.x; i < H; i += blockDim.x) dw_acc[i] = 0.f;
  __syncthreads();
  for (long long row = blockIdx.x; row < rows; row += gridDim.x) {
    const float rs = rstd[row];
    float dot = 0.f;
    for (int v = threadIdx.x; v < nvec; v += blockDim.x) {
      float fx[8], fdy[8], fw[8];
      load8(x + row * H + v * 8, fx);
      load8(dy + row * H + v * 8, fdy);
      load8(w + v * 8, fw);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float xh = fx[i] * rs;
        dot += fdy[i] * fw[i] * xh;
        dw_acc[v * 8 + i] += fdy[i] * xh;
      }
    }
    dot = block_reduce_sum(dot, sh) / H;
    for (int v = threadIdx.x; v < nvec; v += blockDim.x) {
      float fx[8], fdy[8], fw[8], o[8];
      load8(x + row * H + v * 8, fx);
      load8(dy + row * H + v * 8, fdy);
      load8(w + v * 8, fw);
#pragma unroll
      for (int i = 0; i < 8; ++i) o[i] = rs * (fdy[i] * fw[i] - fx[i] * rs * dot);
      if (dres) {
        float fr[8];
        load8(dres + row * H + v * 8, fr);
#pragma unroll
        for (int i = 0; i < 8; ++i) o[i] += fr[i];
      }
      store8(dx + row * H + v * 8, o);
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < H; i += blockDim.x) dw_partial[(long long)blockIdx.x * H + i] = dw_acc[i];
}

// out[c] (+)= sum over the rows of partial [nparts, H]. A block takes 32 columns with 32 warps in turns along the rows: with a thread
// per column and 256 of them per block, four SMs walked 888 rows of 896 one load at a time, 29 us; now 4.
template <typename T>
__global__ void __launch_bounds__(1024) colsum_kernel(const float* __restrict__ partial, int nparts, int H, T* __restrict__ out,
                                                      int accumulate) {
  __shared__ float part[32][33];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, c = blockIdx.x * 32 + lane;
  float s = 0.f;
  if (c < H) {
#pragma unroll 4
    for (int i = warp; i < nparts; i += 32) s += partial[(long long)i * H + c];
  }
  part[warp][lane] = s;
  __syncthreads();
  s = warp_reduce_sum(part[lane][warp]);  // column `warp` of the block
  const int col = blockIdx.x * 32 + warp;
  if (lane == 0 && col < H) out[col] = (T)(accumulate ? (float)out[col] + s : s);
}

// Column sums of bf16 rows (the gradient of a bias), first half: a block sums every gridDim.y-th row of 512 columns. Bound by reading
// the rows once; a conversion to fp32 and a library reduction moved them five times.
__global__ void __launch_bounds__(256) colsum_rows_kernel(const __nv_bfloat16* __restrict__ x, long long stride, int rows, int H,
                                                          float* __restrict__ partial) {
  const int c = (blockIdx.x * 256 + threadIdx.x) * 2;
  if (c >= H) return;
  float a = 0.f, b = 0.f;
#pragma unroll 8
  for (int r = blockIdx.y; r < rows; r += gridDim.y) {
    const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(x + (long long)r * stride + c));
    a += f.x;
    b += f.y;
  }
  *reinterpret_cast<float2*>(partial + (long long)blockIdx.y * H + c) = make_float2(a, b);
}

// ------------------------------- RoPE ----------------------------------------
// In-place rotate-half rotary embedding on packed q [T, Hq, D] and k [T, Hk, D]
// (row strides given in elements). cos/sin tables are [max_pos, D/2] fp32.
// sign = +1 forward, -1 backward (transpose of the rotation).
__global__ void rope_kernel(__nv_bfloat16* __restrict__ q, __nv_bfloat16* __restrict__ k, long long q_stride,
                            long long k_stride, const long long* pos, const float* __restrict__ cos_t,
                            const float* __restrict__ sin_t, int T, int Hq, int Hk, int D, float sign, int mrope_s0,
                            int mrope_s1) {
  // multimodal rotary embedding (mrope_s0 > 0): pos is [3, T] (temporal, height, width); rotary frequency j takes the
  // position of axis 0 for j < s0, of axis 1 for j < s0 + s1, of axis 2 above (sections are multiples of 8, so the 8
  // frequencies of one thread share an axis)
  pdl_trigger();
  pdl_wait();
  const int half = D >> 1;
  const int vec_per_head = half >> 3;
  const long long total = (long long)T * (Hq + Hk) * vec_per_head;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const int v = idx % vec_per_head;
    const long long th = idx / vec_per_head;
    const int h = th % (Hq + Hk);
    const long long t = th / (Hq + Hk);
    __nv_bfloat16* base = (h < Hq) ? (q + t * q_stride + (long long)h * D) : (k + t * k_stride + (long long)(h - Hq) * D);
    long long p;
    if (mrope_s0 > 0) {
      const int j = v * 8;
      const int axis = j < mrope_s0 ? 0 : (j < mrope_s0 + mrope_s1 ? 1 : 2);
      p = pos[(long long)axis * T + t];
    } else {
      p = pos[t];
    }
    const float* c = cos_t + p * half + v * 8;
    const float* s = sin_t + p * half + v * 8;
    float a[8], b[8];
    load8(base + v * 8, a);
    load8(base + half + v * 8, b);
    float oa[8], ob[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float cs = c[i], sn = s[i] * sign;
      oa[i] = a[i] * cs - b[i] * sn;
      ob[i] = b[i] * cs + a[i] * sn;
    }
    store8(base + v * 8, oa);
    store8(base + half + v * 8, ob);
  }
}

// What lies between a layer's projection and its attention, in one pass over packed rows qkv [T, (Hq + 2 Hk) D]: RMS norm of every q
// and k head (weights [D] shared by the heads; null: none; rounded to bf16, as a norm of its own is), rotate-half positions, to `out`
// (may be qkv); k and v also to their places in the paged caches [num_blocks, Hk, block_size, D] (slots null: no cache; slot < 0: no
// write). D / 8 lanes per head, each with four elements of both halves. Bound by latency in a decode step, by its bytes in a prefill or
// in training. It took the place of a rotation and a cache write, with norms also of two copies, two norms and a concatenation: a decode
// step of 24 sequences, 32 / 4 heads with norms: 16 us a layer in seven launches, 3 in one; a forward on 6400
// such tokens 490 us a layer, 122 in one.
template <int D>
struct HeadPart {  // a lane's share of a head
  float a[4], b[4];
  __device__ __forceinline__ void load(const __nv_bfloat16* x) {
    const uint2 ra = *reinterpret_cast<const uint2*>(x), rb = *reinterpret_cast<const uint2*>(x + D / 2);
    const __nv_bfloat162 *pa = reinterpret_cast<const __nv_bfloat162*>(&ra), *pb = reinterpret_cast<const __nv_bfloat162*>(&rb);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const float2 fa = __bfloat1622float2(pa[i]), fb = __bfloat1622float2(pb[i]);
      a[2 * i] = fa.x, a[2 * i + 1] = fa.y, b[2 * i] = fb.x, b[2 * i + 1] = fb.y;
    }
  }
  __device__ __forceinline__ void store(__nv_bfloat16* x) const {
    *reinterpret_cast<uint2*>(x) = make_uint2(pack_bf16x2(a[0], a[1]), pack_bf16x2(a[2], a[3]));
    *reinterpret_cast<uint2*>(x + D / 2) = make_uint2(pack_bf16x2(b[0], b[1]), pack_bf16x2(b[2], b[3]));
  }
  __device__ __forceinline__ void round() {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      a[i] = __bfloat162float(__float2bfloat16(a[i]));
      b[i] = __bfloat162float(__float2bfloat16(b[i]));
    }
  }
  // by the angles at the token's position; sign -1: back
  __device__ __forceinline__ void rotate(const float* cos_t, const float* sin_t, float sign) {
    const float4 c = *reinterpret_cast<const float4*>(cos_t), s = *reinterpret_cast<const float4*>(sin_t);
    const float cs[4] = {c.x, c.y, c.z, c.w}, sn[4] = {s.x * sign, s.y * sign, s.z * sign, s.w * sign};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float x = a[i], y = b[i];
      a[i] = __fmaf_rn(x, cs[i], -__fmul_rn(y, sn[i]));  // as rope_kernel comes out, bit for bit
      b[i] = __fmaf_rn(y, cs[i], __fmul_rn(x, sn[i]));
    }
  }
  // sum over the head of a * p.a + b * p.b; the D / 8 lanes of a head call it together
  __device__ __forceinline__ float dot(const HeadPart& p) const {
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) s += a[i] * p.a[i] + b[i] * p.b[i];
#pragma unroll
    for (int o = 1; o < D / 8; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
  }
};

template <int D>
__global__ void __launch_bounds__(256) head_norm_rope_kernel(
    const __nv_bfloat16* qkv, long long stride, __nv_bfloat16* out, long long out_stride, const long long* pos,
    const float* __restrict__ cos_t, const float* __restrict__ sin_t, const __nv_bfloat16* __restrict__ qw,
    const __nv_bfloat16* __restrict__ kw, float eps, long long T, int Hq, int Hk, const long long* slots, __nv_bfloat16* kc,
    __nv_bfloat16* vc, int block_size) {
  constexpr int LPH = D / 8, HALF = D / 2;
  pdl_trigger();
  pdl_wait();
  const int heads = Hq + Hk + (slots || out != qkv ? Hk : 0);
  const long long unit = ((long long)blockIdx.x * 256 + threadIdx.x) / LPH;
  const int sub = threadIdx.x % LPH;
  if (unit - threadIdx.x % 32 / LPH >= T * heads) return;  // whole warps: the lanes of a norm stay together
  const bool in = unit < T * heads;
  const long long t = in ? unit / heads : 0;
  const int h = in ? (int)(unit % heads) : 0;
  HeadPart<D> x;
  x.load(qkv + t * stride + (long long)h * D + sub * 4);
  if (qw != nullptr) {
    const float rs = rsqrtf(x.dot(x) / D + eps);
    if (h < Hq + Hk) {
      HeadPart<D> w;
      w.load((h < Hq ? qw : kw) + sub * 4);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        x.a[i] = x.a[i] * rs * w.a[i];
        x.b[i] = x.b[i] * rs * w.b[i];
      }
      x.round();
    }
  }
  if (!in) return;
  if (h < Hq + Hk) x.rotate(cos_t + pos[t] * HALF + sub * 4, sin_t + pos[t] * HALF + sub * 4, 1.f);
  if (h < Hq + Hk || out != qkv) x.store(out + t * out_stride + (long long)h * D + sub * 4);
  if (slots != nullptr && h >= Hq) {
    const long long slot = slots[t];
    if (slot < 0) return;
    const bool key = h < Hq + Hk;
    const long long row = (slot / block_size * Hk + (h - Hq - (key ? 0 : Hk))) * block_size + slot % block_size;
    x.store((key ? kc : vc) + row * D + sub * 4);
  }
}

// Gradient of the projection from those of q [T, Hq D], k and v [T, Hk D]: rotation back (rounded, as a rotation of its own is), norm,
// and the sums of the norms' weights per block, part [2][gridDim.x][D] (with norms). x: the projection (with norms). One pass in place
// of three zero-filled buffers, their sum, a copy, a rotation and two norms.
template <int D>
__global__ void __launch_bounds__(256) head_norm_rope_bwd_kernel(
    const __nv_bfloat16* __restrict__ dq, const __nv_bfloat16* __restrict__ dk, const __nv_bfloat16* __restrict__ dv,
    const __nv_bfloat16* __restrict__ x, long long x_stride, const long long* __restrict__ pos, const float* __restrict__ cos_t,
    const float* __restrict__ sin_t, const __nv_bfloat16* __restrict__ qw, const __nv_bfloat16* __restrict__ kw, float eps, long long T,
    int Hq, int Hk, __nv_bfloat16* __restrict__ dqkv, float* __restrict__ part) {
  constexpr int LPH = D / 8, HALF = D / 2, GROUPS = 256 / LPH;
  __shared__ float sums[2][GROUPS][D];
  const int heads = Hq + 2 * Hk, sub = threadIdx.x % LPH, group = threadIdx.x / LPH;
  const long long total = T * heads;
  HeadPart<D> sq{}, sk{};
  for (long long u0 = (long long)blockIdx.x * GROUPS; u0 < total; u0 += (long long)gridDim.x * GROUPS) {
    const bool in = u0 + group < total;
    const long long unit = in ? u0 + group : 0, t = unit / heads;
    const int h = (int)(unit % heads);
    const __nv_bfloat16* from = h < Hq ? dq + (t * Hq + h) * D : h < Hq + Hk ? dk + (t * Hk + h - Hq) * D : dv + (t * Hk + h - Hq - Hk) * D;
    HeadPart<D> d;
    d.load(from + sub * 4);
    if (h < Hq + Hk) {
      d.rotate(cos_t + pos[t] * HALF + sub * 4, sin_t + pos[t] * HALF + sub * 4, -1.f);
      d.round();
    }
    if (qw != nullptr) {
      HeadPart<D> y, w;
      y.load(x + t * x_stride + (long long)h * D + sub * 4);
      w.load((h < Hq ? qw : kw) + sub * 4);
      const float rs = rsqrtf(y.dot(y) / D + eps);
      HeadPart<D> g;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        y.a[i] *= rs;
        y.b[i] *= rs;
        g.a[i] = d.a[i] * w.a[i];
        g.b[i] = d.b[i] * w.b[i];
      }
      const float mean = g.dot(y) / D;
      if (in && h < Hq + Hk) {
        const float to_q = h < Hq ? 1.f : 0.f, to_k = 1.f - to_q;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float pa = d.a[i] * y.a[i], pb = d.b[i] * y.b[i];
          sq.a[i] = fmaf(to_q, pa, sq.a[i]);
          sq.b[i] = fmaf(to_q, pb, sq.b[i]);
          sk.a[i] = fmaf(to_k, pa, sk.a[i]);
          sk.b[i] = fmaf(to_k, pb, sk.b[i]);
          d.a[i] = rs * (g.a[i] - y.a[i] * mean);
          d.b[i] = rs * (g.b[i] - y.b[i] * mean);
        }
      }
    }
    if (in) d.store(dqkv + unit * D + sub * 4);
  }
  if (qw == nullptr) return;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    sums[0][group][sub * 4 + i] = sq.a[i];
    sums[0][group][HALF + sub * 4 + i] = sq.b[i];
    sums[1][group][sub * 4 + i] = sk.a[i];
    sums[1][group][HALF + sub * 4 + i] = sk.b[i];
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 2 * D; i += 256) {
    float s = 0.f;
#pragma unroll
    for (int g = 0; g < GROUPS; ++g) s += sums[i / D][g][i % D];
    part[((long long)(i / D) * gridDim.x + blockIdx.x) * D + i % D] = s;
  }
}

// ------------------------------- SwiGLU --------------------------------------
// gu: [T, 2I] (gate | up), out: [T, I]
// blk_expert (null: none): rows of a buffer sorted by expert, blocks of 128 rows without one are left out.
__global__ void swiglu_fwd_kernel(const __nv_bfloat16* gu, __nv_bfloat16* __restrict__ out, long long T, int I,
                                  const int* blk_expert) {
  pdl_trigger();
  pdl_wait();
  const int nvec = I >> 3;
  const long long total = T * nvec;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const long long t = idx / nvec;
    const int v = idx % nvec;
    if (blk_expert != nullptr && blk_expert[t >> 7] < 0) continue;
    float g[8], u[8], o[8];
    load8(gu + t * 2 * I + v * 8, g);
    load8(gu + t * 2 * I + I + v * 8, u);
#pragma unroll
    for (int i = 0; i < 8; ++i) o[i] = g[i] / (1.f + __expf(-g[i])) * u[i];
    store8(out + t * I + v * 8, o);
  }
}

__global__ void swiglu_bwd_kernel(const __nv_bfloat16* __restrict__ gu, const __nv_bfloat16* __restrict__ dout,
                                  __nv_bfloat16* __restrict__ dgu, long long T, int I,
                                  const int* __restrict__ blk_expert) {
  const int nvec = I >> 3;
  const long long total = T * nvec;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const long long t = idx / nvec;
    const int v = idx % nvec;
    if (blk_expert != nullptr && blk_expert[t >> 7] < 0) continue;
    float g[8], u[8], d[8], dg[8], du[8];
    load8(gu + t * 2 * I + v * 8, g);
    load8(gu + t * 2 * I + I + v * 8, u);
    load8(dout + t * I + v * 8, d);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float sg = 1.f / (1.f + __expf(-g[i]));
      const float silu = g[i] * sg;
      dg[i] = d[i] * u[i] * (sg + silu * (1.f - sg));
      du[i] = d[i] * silu;
    }
    store8(dgu + t * 2 * I + v * 8, dg);
    store8(dgu + t * 2 * I + I + v * 8, du);
  }
}

// ------------------------------- Embedding -----------------------------------
__global__ void embedding_fwd_kernel(const long long* __restrict__ ids, const __nv_bfloat16* __restrict__ w,
                                     __nv_bfloat16* __restrict__ out, long long T, int H) {
  const int nvec = H >> 3;
  const long long total = T * nvec;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const long long t = idx / nvec;
    const int v = idx % nvec;
    *reinterpret_cast<uint4*>(out + t * H + v * 8) = *reinterpret_cast<const uint4*>(w + ids[t] * H + v * 8);
  }
}

// dW[ids[t], :] += dy[t, :] into an fp32 gradient buffer.
__global__ void embedding_bwd_kernel(const long long* __restrict__ ids, const __nv_bfloat16* __restrict__ dy,
                                     float* __restrict__ dw, long long T, int H) {
  const int nvec = H >> 3;
  const long long total = T * nvec;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const long long t = idx / nvec;
    const int v = idx % nvec;
    float f[8];
    load8(dy + t * H + v * 8, f);
    float* dst = dw + ids[t] * H + v * 8;
#pragma unroll
    for (int i = 0; i < 8; ++i) atomicAdd(dst + i, f[i]);
  }
}

// ------------------------------- AdamW ---------------------------------------
// Flat-shard AdamW with fp32 master weights; writes the bf16 working copy in the same pass.
//   grad is fp32 (grad_bf16 == 0) or bf16. scale_ptr (device) multiplies the gradient
//   (clip coefficient and/or 1/world); skip_ptr (device) != 0 leaves everything unchanged
//   (non-finite gradient norm: verl/workers/actor/dp_actor.py:410-412).
__global__ void adamw_kernel(float* __restrict__ p32, const void* __restrict__ grad, int grad_bf16,
                             float* __restrict__ m, float* __restrict__ v, __nv_bfloat16* __restrict__ p16,
                             long long n, float lr, float b1, float b2, float eps, float wd, float bc1, float bc2,
                             const float* __restrict__ scale_ptr, const int* __restrict__ skip_ptr) {
  if (skip_ptr && *skip_ptr) return;
  const float gs = scale_ptr ? *scale_ptr : 1.f;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    float g = grad_bf16 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(grad)[i])
                        : reinterpret_cast<const float*>(grad)[i];
    g *= gs;
    float p = p32[i];
    float mi = m[i] * b1 + (1.f - b1) * g;
    float vi = v[i] * b2 + (1.f - b2) * g * g;
    m[i] = mi;
    v[i] = vi;
    p = p * (1.f - lr * wd);
    p -= lr * (mi / bc1) / (sqrtf(vi / bc2) + eps);
    p32[i] = p;
    if (p16) p16[i] = __float2bfloat16(p);
  }
}

// out[0] += sum(x^2)  (fp32 or bf16 input)
__global__ void sumsq_kernel(const void* __restrict__ x, int is_bf16, long long n, float* __restrict__ out) {
  __shared__ float sh[32];
  float s = 0.f;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const float f = is_bf16 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(x)[i])
                            : reinterpret_cast<const float*>(x)[i];
    s += f * f;
  }
  s = block_reduce_sum(s, sh);
  if (threadIdx.x == 0) atomicAdd(out, s);
}

// scale_out = min(1, max_norm / (sqrt(sumsq) + 1e-6)); skip_out = !isfinite(norm); norm_out = norm
__global__ void clip_coef_kernel(const float* __restrict__ sumsq, float max_norm, float* __restrict__ scale_out,
                                 int* __restrict__ skip_out, float* __restrict__ norm_out, float extra_scale) {
  const float norm = sqrtf(*sumsq) * extra_scale;
  const bool finite = isfinite(norm);
  float c = 1.f;
  if (max_norm > 0.f && finite) c = fminf(1.f, max_norm / (norm + 1e-6f));
  *scale_out = c * extra_scale;
  *skip_out = finite ? 0 : 1;
  *norm_out = norm;
}

// bf16 <- fp32 cast (flat), and fp32 <- bf16
__global__ void cast_f32_to_bf16_kernel(const float* __restrict__ src, __nv_bfloat16* __restrict__ dst, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    dst[i] = __float2bfloat16(src[i]);
}

static inline int grid_for(long long work, int block, int max_blocks) {
  long long g = (work + block - 1) / block;
  if (g > max_blocks) g = max_blocks;
  if (g < 1) g = 1;
  return (int)g;
}

}  // namespace vb

using namespace vb;

extern "C" int vb_rmsnorm_fwd(const void* x, const void* res, const void* w, void* y, void* res_out, float* rstd,
                              long long rows, int H, float eps, cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (H & 7) return -3;
  const int threads = H >= 4096 ? 512 : 256;
  cudaError_t e = vb_launch_pdl(rmsnorm_fwd_kernel, dim3((unsigned)rows), dim3(threads), 0, stream, 1,
                                (const __nv_bfloat16*)x, (const __nv_bfloat16*)res, (const __nv_bfloat16*)w,
                                (__nv_bfloat16*)y, (__nv_bfloat16*)res_out, rstd, H, eps);
  vb_count_launch();
  return e != cudaSuccess ? (int)e : (int)cudaGetLastError();
}

// Number of partial rows the backward uses; dw_partial must hold that many rows of H floats.
extern "C" int vb_rmsnorm_bwd_parts(long long rows) {
  const int g = 6 * vb_num_sms();  // six resident blocks per SM: 75 % of the warp slots (two left the loads starved)
  return rows < g ? (int)rows : g;
}

extern "C" int vb_rmsnorm_bwd(const void* dy, const void* x, const void* w, const float* rstd, const void* dres,
                              void* dx, float* dw_partial, float* dw, int dw_accumulate, long long rows, int H,
                              cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (H & 7) return -3;
  const int parts = vb_rmsnorm_bwd_parts(rows);
  const size_t smem = (size_t)H * sizeof(float);
  if (smem > 48 * 1024) {
    VB_CUDA_CHECK(cudaFuncSetAttribute(rmsnorm_bwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  }
  rmsnorm_bwd_kernel<<<parts, 256, smem, stream>>>((const __nv_bfloat16*)dy, (const __nv_bfloat16*)x,
                                                  (const __nv_bfloat16*)w, rstd, (const __nv_bfloat16*)dres,
                                                  (__nv_bfloat16*)dx, dw_partial, (int)rows, H);
  colsum_kernel<float><<<(H + 31) / 32, 1024, 0, stream>>>(dw_partial, parts, H, dw, dw_accumulate);
  vb_count_launch(2);
  return (int)cudaGetLastError();
}

// out [H] bf16 = sum over the rows of x [rows, H] bf16 (H and the stride even, x on a 4-byte boundary); work: fp32 [parts, H].
extern "C" int vb_colsum_parts(int rows) { return rows < 1 ? 1 : rows < 512 ? (rows + 7) / 8 : 64; }
extern "C" int vb_colsum_bf16(const void* x, long long stride, int rows, int H, float* work, void* out, cudaStream_t stream) {
  if (rows < 0 || H <= 0) return -3;
  if ((H & 1) || (stride & 1) || (reinterpret_cast<uintptr_t>(x) & 3)) return -3;
  const int parts = vb_colsum_parts(rows);
  colsum_rows_kernel<<<dim3((H + 511) / 512, parts), 256, 0, stream>>>((const __nv_bfloat16*)x, stride, rows, H, work);
  colsum_kernel<__nv_bfloat16><<<(H + 31) / 32, 1024, 0, stream>>>(work, parts, H, (__nv_bfloat16*)out, 0);
  vb_count_launch(2);
  return (int)cudaGetLastError();
}

static int rope_launch(void* q, void* k, long long q_stride, long long k_stride, const long long* pos, const float* cos_t,
                       const float* sin_t, int T, int Hq, int Hk, int D, int backward, int s0, int s1, cudaStream_t stream);

extern "C" int vb_rope(void* q, void* k, long long q_stride, long long k_stride, const long long* pos,
                       const float* cos_t, const float* sin_t, int T, int Hq, int Hk, int D, int backward,
                       cudaStream_t stream) {
  return rope_launch(q, k, q_stride, k_stride, pos, cos_t, sin_t, T, Hq, Hk, D, backward, 0, 0, stream);
}

// D 64, 128 or 256; rows, results, caches and norms on 8-byte boundaries, tables on 16-byte ones. qw and kw both or neither.
extern "C" int vb_head_norm_rope(const void* qkv, long long stride, void* out, long long out_stride, const long long* pos,
                                 const float* cos_t, const float* sin_t, const void* qw, const void* kw, float eps, long long T, int Hq,
                                 int Hk, int D, const long long* slots, void* kc, void* vc, int block_size, cudaStream_t stream) {
  if (T <= 0) return 0;
  if (((stride | out_stride) & 3) || ((reinterpret_cast<uintptr_t>(qkv) | reinterpret_cast<uintptr_t>(out)) & 7) ||
      (qw == nullptr) != (kw == nullptr) ||
      ((reinterpret_cast<uintptr_t>(qw) | reinterpret_cast<uintptr_t>(kw)) & 7) ||
      ((reinterpret_cast<uintptr_t>(cos_t) | reinterpret_cast<uintptr_t>(sin_t)) & 15) ||
      (slots && (((reinterpret_cast<uintptr_t>(kc) | reinterpret_cast<uintptr_t>(vc)) & 7) || block_size <= 0)))
    return -3;
  const long long threads = T * (Hq + Hk + (slots || out != qkv ? Hk : 0)) * (D / 8), blocks = (threads + 255) / 256;
  if (blocks > 0x7fffffffLL) return -3;
  cudaError_t e;
#define VB_HNR(DD)                                                                                                                  \
  e = vb_launch_pdl(head_norm_rope_kernel<DD>, dim3((unsigned)blocks), dim3(256), 0, stream, 1, (const __nv_bfloat16*)qkv, stride,    \
                    (__nv_bfloat16*)out, out_stride, pos, cos_t, sin_t, (const __nv_bfloat16*)qw, (const __nv_bfloat16*)kw, eps, T, Hq, \
                    Hk, slots, (__nv_bfloat16*)kc, (__nv_bfloat16*)vc, block_size)
  if (D == 64) VB_HNR(64);
  else if (D == 128) VB_HNR(128);
  else if (D == 256) VB_HNR(256);
  else return -3;
#undef VB_HNR
  vb_count_launch();
  return e != cudaSuccess ? (int)e : (int)cudaGetLastError();
}

// dq, dk, dv, dqkv contiguous and on 8-byte boundaries, norms and tables as above. With norms: x the projection, part fp32 [2, parts, D], dqw and dkw fp32 [D]
// (accumulate: added to).
extern "C" int vb_head_norm_rope_bwd_parts() { return 4 * vb_num_sms(); }
extern "C" int vb_head_norm_rope_bwd(const void* dq, const void* dk, const void* dv, const void* x, long long x_stride,
                                     const long long* pos, const float* cos_t, const float* sin_t, const void* qw, const void* kw,
                                     float eps, long long T, int Hq, int Hk, int D, void* dqkv, float* part, float* dqw, float* dkw,
                                     int accumulate_q, int accumulate_k, cudaStream_t stream) {
  if (T <= 0) return 0;
  const uintptr_t at = reinterpret_cast<uintptr_t>(dq) | reinterpret_cast<uintptr_t>(dk) | reinterpret_cast<uintptr_t>(dv) |
                       reinterpret_cast<uintptr_t>(dqkv) | (qw ? reinterpret_cast<uintptr_t>(x) : 0);
  if ((at & 7) || (qw && ((x_stride & 3) || !kw || !part || !dqw || !dkw)) ||
      ((reinterpret_cast<uintptr_t>(qw) | reinterpret_cast<uintptr_t>(kw)) & 7) ||
      ((reinterpret_cast<uintptr_t>(cos_t) | reinterpret_cast<uintptr_t>(sin_t)) & 15))
    return -3;
  const int parts = vb_head_norm_rope_bwd_parts();
#define VB_HNRB(DD)                                                                                                                \
  head_norm_rope_bwd_kernel<DD><<<parts, 256, 0, stream>>>((const __nv_bfloat16*)dq, (const __nv_bfloat16*)dk, (const __nv_bfloat16*)dv, \
                                                           (const __nv_bfloat16*)x, x_stride, pos, cos_t, sin_t,                    \
                                                           (const __nv_bfloat16*)qw, (const __nv_bfloat16*)kw, eps, T, Hq, Hk,      \
                                                           (__nv_bfloat16*)dqkv, part)
  if (D == 64) VB_HNRB(64);
  else if (D == 128) VB_HNRB(128);
  else if (D == 256) VB_HNRB(256);
  else return -3;
#undef VB_HNRB
  if (qw) {
    colsum_kernel<float><<<(D + 31) / 32, 1024, 0, stream>>>(part, parts, D, dqw, accumulate_q);
    colsum_kernel<float><<<(D + 31) / 32, 1024, 0, stream>>>(part + (long long)parts * D, parts, D, dkw, accumulate_k);
  }
  vb_count_launch(qw ? 3 : 1);
  return (int)cudaGetLastError();
}

// Multimodal RoPE: pos is [3, T]; s0 / s1 = number of rotary frequencies (of D / 2) that follow the temporal / height
// positions (the rest follow the width positions); both multiples of 8.
extern "C" int vb_mrope(void* q, void* k, long long q_stride, long long k_stride, const long long* pos3,
                        const float* cos_t, const float* sin_t, int T, int Hq, int Hk, int D, int s0, int s1, int backward,
                        cudaStream_t stream) {
  if (s0 <= 0 || s1 < 0 || (s0 & 7) || (s1 & 7) || s0 + s1 > D / 2) return -3;
  return rope_launch(q, k, q_stride, k_stride, pos3, cos_t, sin_t, T, Hq, Hk, D, backward, s0, s1, stream);
}

static int rope_launch(void* q, void* k, long long q_stride, long long k_stride, const long long* pos, const float* cos_t,
                       const float* sin_t, int T, int Hq, int Hk, int D, int backward, int s0, int s1, cudaStream_t stream) {
  if (T <= 0) return 0;
  if (D & 15) return -3;
  const long long total = (long long)T * (Hq + Hk) * (D / 16);
  cudaError_t e = vb_launch_pdl(rope_kernel, dim3(grid_for(total, 256, 148 * 16)), dim3(256), 0, stream, 1,
                                (__nv_bfloat16*)q, (__nv_bfloat16*)k, q_stride, k_stride, pos, cos_t, sin_t, T, Hq, Hk,
                                D, backward ? -1.f : 1.f, s0, s1);
  vb_count_launch();
  return e != cudaSuccess ? (int)e : (int)cudaGetLastError();
}

extern "C" int vb_swiglu_fwd(const void* gu, void* out, long long T, int I, const int* blk_expert, cudaStream_t stream) {
  if (T <= 0) return 0;
  if (I & 7) return -3;
  cudaError_t e = vb_launch_pdl(swiglu_fwd_kernel, dim3(grid_for(T * (I / 8), 256, 148 * 16)), dim3(256), 0, stream, 1,
                                (const __nv_bfloat16*)gu, (__nv_bfloat16*)out, T, I, blk_expert);
  vb_count_launch();
  return e != cudaSuccess ? (int)e : (int)cudaGetLastError();
}

extern "C" int vb_swiglu_bwd(const void* gu, const void* dout, void* dgu, long long T, int I, const int* blk_expert,
                             cudaStream_t stream) {
  if (T <= 0) return 0;
  if (I & 7) return -3;
  swiglu_bwd_kernel<<<grid_for(T * (I / 8), 256, 148 * 16), 256, 0, stream>>>(
      (const __nv_bfloat16*)gu, (const __nv_bfloat16*)dout, (__nv_bfloat16*)dgu, T, I, blk_expert);
  vb_count_launch();
  return (int)cudaGetLastError();
}

extern "C" int vb_embedding_fwd(const long long* ids, const void* w, void* out, long long T, int H,
                                cudaStream_t stream) {
  if (T <= 0) return 0;
  if (H & 7) return -3;
  embedding_fwd_kernel<<<grid_for(T * (H / 8), 256, 148 * 16), 256, 0, stream>>>(ids, (const __nv_bfloat16*)w,
                                                                                 (__nv_bfloat16*)out, T, H);
  vb_count_launch();
  return (int)cudaGetLastError();
}

extern "C" int vb_embedding_bwd(const long long* ids, const void* dy, float* dw, long long T, int H,
                                cudaStream_t stream) {
  if (T <= 0) return 0;
  if (H & 7) return -3;
  embedding_bwd_kernel<<<grid_for(T * (H / 8), 256, 148 * 16), 256, 0, stream>>>(ids, (const __nv_bfloat16*)dy, dw,
                                                                                 T, H);
  vb_count_launch();
  return (int)cudaGetLastError();
}

extern "C" int vb_adamw(float* p32, const void* grad, int grad_bf16, float* m, float* v, void* p16, long long n,
                        float lr, float b1, float b2, float eps, float wd, int step, const float* scale_ptr,
                        const int* skip_ptr, cudaStream_t stream) {
  if (n <= 0) return 0;
  const float bc1 = 1.f - powf(b1, (float)step);
  const float bc2 = 1.f - powf(b2, (float)step);
  adamw_kernel<<<grid_for(n, 256, 148 * 16), 256, 0, stream>>>(p32, grad, grad_bf16, m, v, (__nv_bfloat16*)p16, n, lr,
                                                               b1, b2, eps, wd, bc1, bc2, scale_ptr, skip_ptr);
  vb_count_launch();
  return (int)cudaGetLastError();
}

extern "C" int vb_sumsq(const void* x, int is_bf16, long long n, float* out, cudaStream_t stream) {
  if (n <= 0) return 0;
  sumsq_kernel<<<grid_for(n, 256, 148 * 8), 256, 0, stream>>>(x, is_bf16, n, out);
  vb_count_launch();
  return (int)cudaGetLastError();
}

extern "C" int vb_clip_coef(const float* sumsq, float max_norm, float extra_scale, float* scale_out, int* skip_out,
                            float* norm_out, cudaStream_t stream) {
  clip_coef_kernel<<<1, 1, 0, stream>>>(sumsq, max_norm, scale_out, skip_out, norm_out, extra_scale);
  vb_count_launch();
  return (int)cudaGetLastError();
}

extern "C" int vb_cast_f32_bf16(const float* src, void* dst, long long n, cudaStream_t stream) {
  if (n <= 0) return 0;
  cast_f32_to_bf16_kernel<<<grid_for(n, 256, 148 * 16), 256, 0, stream>>>(src, (__nv_bfloat16*)dst, n);
  vb_count_launch();
  return (int)cudaGetLastError();
}
