// RL math kernels: fused PPO token loss (forward + gradient + metrics in one pass),
// GAE reverse scan, group-normalised (GRPO) advantages, and the rollout sampler.
//
// Formulas follow verl/trainer/ppo/core_algos.py: GAE :214-262, GRPO :266-330,
// vanilla/dual-clip policy loss :1159-1250, kl_penalty :1841-1902. The reference
// runs these as many small torch launches (GAE is a Python loop over T).
#include "common.cuh"
#include "host_utils.h"

namespace vb {

__device__ __forceinline__ float block_sum(float v, float* sh) {
  v = warp_reduce_sum(v);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nw = (blockDim.x + 31) >> 5;
  __syncthreads();
  if (lane == 0) sh[warp] = v;
  __syncthreads();
  float t = (lane < nw) ? sh[lane] : 0.f;
  return warp_reduce_sum(t);
}

// metrics layout (sums over masked tokens):
// 0 pg_loss, 1 clipfrac, 2 ppo_kl, 3 clipfrac_lower, 4 kl_loss, 5 entropy, 6 mask count
struct PpoArgs {
  const float* logp;
  const float* old_logp;  // null => on-policy (old = logp detached)
  const float* adv;
  const float* mask;
  const float* ref_logp;  // null => no KL loss
  const float* entropy;   // null => no entropy bonus
  const float* is_weight; // null => no rollout importance weights
  float* d_logp;
  float* d_entropy;
  float* metrics;
  long long n;
  float clip_low, clip_high, clip_c, kl_coef, entropy_coeff, inv_denom;
  int kl_type;  // 0 kl(k1), 1 abs, 2 mse(k2), 3 low_var_kl(k3)
};

__global__ void ppo_loss_kernel(PpoArgs a) {
  __shared__ float sh[32];
  float acc[7] = {0, 0, 0, 0, 0, 0, 0};
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < a.n;
       i += (long long)gridDim.x * blockDim.x) {
    const float mk = a.mask[i];
    const float lp = a.logp[i];
    const float olp = a.old_logp ? a.old_logp[i] : lp;
    const float A = a.adv[i];
    const float w = a.is_weight ? a.is_weight[i] : 1.f;
    const float raw = lp - olp;
    const float nkl = fminf(fmaxf(raw, -20.f), 20.f);
    const bool in_range = (raw > -20.f) && (raw < 20.f);
    const float ratio = __expf(nkl);
    const float l1 = -A * ratio;
    const float rc = fminf(fmaxf(ratio, 1.f - a.clip_low), 1.f + a.clip_high);
    const float l2 = -A * rc;
    const float clip1 = fmaxf(l1, l2);
    const float l3 = -A * a.clip_c;
    const float clip2 = fminf(l3, clip1);
    const bool neg = A < 0.f;
    const float pg = neg ? clip2 : clip1;
    // gradient of pg wrt logp
    const float dl1 = in_range ? -A * ratio : 0.f;
    const bool ratio_clipped = (ratio < 1.f - a.clip_low) || (ratio > 1.f + a.clip_high);
    const float dl2 = ratio_clipped ? 0.f : dl1;
    float dclip1 = (l1 > l2) ? dl1 : ((l2 > l1) ? dl2 : 0.5f * (dl1 + dl2));
    float dpg = dclip1;
    if (neg) dpg = (l3 < clip1) ? 0.f : ((l3 > clip1) ? dclip1 : 0.5f * dclip1);
    float loss_grad = dpg * w;
    float kl = 0.f;
    if (a.ref_logp) {
      const float rlp = a.ref_logp[i];
      float dkl = 0.f;
      if (a.kl_type == 0) {
        kl = lp - rlp;
        dkl = 1.f;
      } else if (a.kl_type == 1) {
        kl = fabsf(lp - rlp);
        dkl = (lp > rlp) ? 1.f : ((lp < rlp) ? -1.f : 0.f);
      } else if (a.kl_type == 2) {
        kl = 0.5f * (lp - rlp) * (lp - rlp);
        dkl = lp - rlp;
      } else {
        const float draw = rlp - lp;
        const float d = fminf(fmaxf(draw, -20.f), 20.f);
        const float e = __expf(d);
        const float k3 = e - d - 1.f;
        kl = fminf(fmaxf(k3, -10.f), 10.f);
        const bool pass = (draw > -20.f) && (draw < 20.f) && (k3 > -10.f) && (k3 < 10.f);
        dkl = pass ? (1.f - e) : 0.f;
      }
      loss_grad += a.kl_coef * dkl;
    }
    a.d_logp[i] = loss_grad * mk * a.inv_denom;
    float ent = 0.f;
    if (a.entropy) {
      ent = a.entropy[i];
      if (a.d_entropy) a.d_entropy[i] = -a.entropy_coeff * mk * a.inv_denom;
    }
    acc[0] += pg * w * mk;
    acc[1] += (l2 > l1 ? 1.f : 0.f) * mk;
    acc[2] += -nkl * mk;
    acc[3] += ((clip1 > l3) && neg ? 1.f : 0.f) * mk;
    acc[4] += kl * mk;
    acc[5] += ent * mk;
    acc[6] += mk;
  }
#pragma unroll
  for (int j = 0; j < 7; ++j) {
    const float s = block_sum(acc[j], sh);
    if (threadIdx.x == 0) atomicAdd(a.metrics + j, s);
  }
}

// GAE: one thread per sequence, reverse scan with mask-aware carry
// (observation tokens keep nextvalues/lastgaelam: core_algos.py:214-262).
__global__ void gae_kernel(const float* __restrict__ rewards, const float* __restrict__ values,
                           const float* __restrict__ mask, float* __restrict__ adv, float* __restrict__ ret, int B,
                           int T, float gamma, float lam) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= B) return;
  const long long off = (long long)b * T;
  float nextv = 0.f, last = 0.f;
  for (int t = T - 1; t >= 0; --t) {
    const float mk = mask[off + t];
    const float v = values[off + t];
    const float delta = rewards[off + t] + gamma * nextv - v;
    const float l_ = delta + gamma * lam * last;
    nextv = v * mk + (1.f - mk) * nextv;
    last = l_ * mk + (1.f - mk) * last;
    adv[off + t] = last;
    ret[off + t] = last + v;
  }
}

// GRPO: per-group mean / unbiased std of sequence scores; singleton groups use mean 0, std 1.
__global__ void group_stats_kernel(const float* __restrict__ scores, const int* __restrict__ gid, int B,
                                   float* __restrict__ gsum, float* __restrict__ gsq, float* __restrict__ gcnt) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= B) return;
  const float s = scores[b];
  atomicAdd(gsum + gid[b], s);
  atomicAdd(gsq + gid[b], s * s);
  atomicAdd(gcnt + gid[b], 1.f);
}

__global__ void group_adv_kernel(const float* __restrict__ scores, const int* __restrict__ gid,
                                 const float* __restrict__ gsum, const float* __restrict__ gsq,
                                 const float* __restrict__ gcnt, const float* __restrict__ mask,
                                 float* __restrict__ adv, int B, int T, float eps, int norm_by_std) {
  const int b = blockIdx.x;
  const int g = gid[b];
  const float n = gcnt[g];
  float mean = 0.f, sd = 1.f;
  if (n > 1.5f) {
    mean = gsum[g] / n;
    const float var = fmaxf((gsq[g] - n * mean * mean) / (n - 1.f), 0.f);
    sd = sqrtf(var);
  }
  float a = scores[b] - mean;
  if (norm_by_std) a = a / (sd + eps);
  for (int t = threadIdx.x; t < T; t += blockDim.x) adv[(long long)b * T + t] = a * mask[(long long)b * T + t];
}

// ------------------------------- sampler -------------------------------------
__device__ __forceinline__ uint32_t mulhilo(uint32_t a, uint32_t b, uint32_t* hi) {
  const uint64_t p = (uint64_t)a * b;
  *hi = (uint32_t)(p >> 32);
  return (uint32_t)p;
}
// Philox-4x32-10, returns 4 x 32 random bits for (counter, key).
__device__ __forceinline__ uint4 philox(uint4 c, uint2 k) {
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    uint32_t hi0, hi1;
    const uint32_t lo0 = mulhilo(0xD2511F53u, c.x, &hi0);
    const uint32_t lo1 = mulhilo(0xCD9E8D57u, c.z, &hi1);
    c = make_uint4(hi1 ^ c.y ^ k.x, lo1, hi0 ^ c.w ^ k.y, lo0);
    k.x += 0x9E3779B9u;
    k.y += 0xBB67AE85u;
  }
  return c;
}
__device__ __forceinline__ float u01(uint32_t x) { return ((float)(x >> 8) + 0.5f) * (1.f / 16777216.f); }
// Gumbel noise of a uniform draw. The largest draws round up to one (16777215.5 has no fp32 form) and the fast logarithm is off by
// up to 2^-22 there: without the floor -log(u) could be zero, the noise infinite, and one token in 2^24 a draw no matter its logit.
__device__ __forceinline__ float gumbel(uint32_t x) { return -__logf(fmaxf(-__logf(u01(x)), 2.98e-8f)); }

// Four consecutive logits starting at v0 (a multiple of 4) as floats; elements past V read as -inf. `vec` says that the
// row base is aligned for one 16-byte (fp32) / 8-byte (bf16) load.
__device__ __forceinline__ void load4_logits(const float* lg, bool vec, int v0, int V, float (&x)[4]) {
  if (vec && v0 + 3 < V) {
    const float4 t = *reinterpret_cast<const float4*>(lg + v0);
    x[0] = t.x; x[1] = t.y; x[2] = t.z; x[3] = t.w;
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j) x[j] = v0 + j < V ? lg[v0 + j] : -INFINITY;
  }
}
__device__ __forceinline__ void load4_logits(const __nv_bfloat16* lg, bool vec, int v0, int V, float (&x)[4]) {
  if (vec && v0 + 3 < V) {
    const uint2 t = *reinterpret_cast<const uint2*>(lg + v0);
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&t.x));
    const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&t.y));
    x[0] = a.x; x[1] = a.y; x[2] = b.x; x[3] = b.y;
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j) x[j] = v0 + j < V ? __bfloat162float(lg[v0 + j]) : -INFINITY;
  }
}

// One row per cluster of C blocks (C = 1, 2, 4, 8), a contiguous part of the vocabulary per block. Gumbel-max sampling from
// softmax(logits / T) restricted by top-k / top-p, greedy when temperature == 0. Outputs the token and the log-prob of the sampled
// token under the *processed* distribution (temperature applied, restricted support renormalised), which is what the rollout
// reports as rollout_log_probs (vllm logprobs_mode=processed_logprobs in the reference config).
//
// Unrestricted rows take ONE pass: each thread keeps an online (max, sum of exp) pair and the Gumbel-max candidate of its elements;
// the argmax of logit / T + noise needs no normaliser, and the log-prob of the winner is x - max - log(sum). That pass is bound by
// the arithmetic of the noise (128 rows of 152 064: 47 us, greedy 27 us; one row on eight SMs 19 us, on one it was 43).
//
// The support of a restricted row is {p >= thr}, thr found by 30 steps of bisection on the probability. Instead of 30 passes over the
// row, a pass counts the tokens above four guesses (2^-4 .. 2^-16 of the largest probability, then closer ones): once a guess leaves
// at most SMP_CAND tokens and satisfies the restriction, the threshold lies above it, these tokens go to the first block of the
// cluster, and one warp takes all steps on them. Rows where no guess does (very many equal probabilities) are counted step by step.
// Groups of four tokens that are clearly below what a pass looks for cost a load and a comparison; the row comes from L2 after the
// first pass. 152 064 fp32 logits, top-k 50, top-p 0.95: 128 rows 85 us, one row 37 us; when a block per row counted all 30 steps
// on the row it was 1000 us for one row and for 128. Equal logits (counted step by step): 602 us, before 1008.
constexpr int SMP_THREADS = 1024;
constexpr int SMP_CAND = 1024;
constexpr int SMP_MAX_C = 8;
constexpr int SMP_LEVELS = 4;

struct SampleShared {
  float red_a[32], red_b[32];
  int red_i[32];
  float red_l[2 * SMP_LEVELS][32];
  float xch[2][2 * SMP_LEVELS][SMP_MAX_C];
  float cand[SMP_CAND];
  float thr;
  float fin_m[SMP_MAX_C], fin_best[SMP_MAX_C], fin_z[SMP_MAX_C];
  int fin_i[SMP_MAX_C];
};

__device__ __forceinline__ void st_cluster_f32(const void* local, uint32_t rank, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(map_to_cta(smem_u32(local), rank)), "f"(v) : "memory");
}
__device__ __forceinline__ void st_cluster_s32(const void* local, uint32_t rank, int v) {
  asm volatile("st.shared::cluster.s32 [%0], %1;" ::"r"(map_to_cta(smem_u32(local), rank)), "r"(v) : "memory");
}

// Every block of the cluster gets every block's N numbers in sh.xch[turn][.][block]. Two turns alternate: a block writes a turn's
// slots again only after the barrier of the other turn, which every block reaches after it has read them.
template <int N>
__device__ __forceinline__ void cluster_exchange(SampleShared& sh, int turn, uint32_t rank, int C, const float (&v)[N]) {
  if ((int)threadIdx.x < C) {
#pragma unroll
    for (int i = 0; i < N; ++i) st_cluster_f32(&sh.xch[turn][i][rank], threadIdx.x, v[i]);
  }
  cluster_sync_all();
}

// (m, z) and (om, oz): maxima and sums of exp(x - maximum) of two sets -> of both
__device__ __forceinline__ void merge_max_sum(float& m, float& z, float om, float oz) {
  const float nm = fmaxf(m, om);
  z = nm > -INFINITY ? z * __expf(m - nm) + oz * __expf(om - nm) : 0.f;
  m = nm;
}
__device__ __forceinline__ void merge_best(float& best, int& best_i, float ob, int oi) {  // ties: the lowest index
  if (ob > best || (ob == best && oi < best_i)) {
    best = ob;
    best_i = oi;
  }
}

template <typename T>
__global__ void __launch_bounds__(SMP_THREADS, 1)
sample_kernel(const T* __restrict__ logits, long long row_stride, int V, int C, int per_block,
              const float* __restrict__ temperature, const int* __restrict__ top_k, const float* __restrict__ top_p,
              unsigned long long seed, const long long* __restrict__ step, long long* __restrict__ token_out,
              float* __restrict__ logprob_out) {
  __shared__ SampleShared sh;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t rank = C > 1 ? cluster_ctarank() : 0;
  const int row = blockIdx.x / C;
  const int begin = min(V, (int)rank * per_block), end = min(V, begin + per_block);
  const int quads = (end - begin + 3) / 4;
  const T* lg = logits + (long long)row * row_stride;
  const bool vec = (reinterpret_cast<uintptr_t>(lg) & (4 * sizeof(T) - 1)) == 0;
  const float temp = temperature ? temperature[row] : 1.f;
  const bool greedy = temp <= 1e-6f;
  const float inv_t = greedy ? 1.f : 1.f / temp;
  const int k = top_k ? top_k[row] : -1;
  const float tp = top_p ? top_p[row] : 1.f;
  const bool need_k = !greedy && k > 0 && k < V, need_p = !greedy && tp < 1.f;
  const bool restricted = need_k || need_p;  // the same for every thread of the cluster
  const unsigned long long st = step ? (unsigned long long)(*step) : 0ull;
  auto noise = [&](int v0, uint32_t (&rr)[4]) {
    const uint4 rnd = philox(make_uint4((uint32_t)v0, (uint32_t)row, (uint32_t)st, (uint32_t)(st >> 32)),
                             make_uint2((uint32_t)seed, (uint32_t)(seed >> 32)));
    rr[0] = rnd.x; rr[1] = rnd.y; rr[2] = rnd.z; rr[3] = rnd.w;
  };

  float mx = -INFINITY, best = -INFINITY, sum = 0.f;
  int best_i = restricted ? 0 : 0x7fffffff;
  float thr = 0.f;
  if (!restricted) {
    float next[4];
    load4_logits(lg, vec, begin + tid * 4, end, next);  // -inf past the end
    for (int i = tid; i < quads; i += SMP_THREADS) {
      const int v0 = begin + i * 4;
      float x[4] = {next[0], next[1], next[2], next[3]};
      load4_logits(lg, vec, v0 + SMP_THREADS * 4, end, next);
#pragma unroll
      for (int j = 0; j < 4; ++j) x[j] *= inv_t;
      const float gm = fmaxf(fmaxf(x[0], x[1]), fmaxf(x[2], x[3]));
      if (gm > mx) {
        sum *= __expf(mx - gm);  // mx = -inf: the sum is still 0
        mx = gm;
      }
      if (mx > -INFINITY) sum += __expf(x[0] - mx) + __expf(x[1] - mx) + __expf(x[2] - mx) + __expf(x[3] - mx);
      // no noise is larger than 17.34: what lies further below a score that is there already cannot win
      if (gm >= best - (greedy ? 0.f : 17.4f)) {
        uint32_t rr[4] = {0u, 0u, 0u, 0u};
        if (!greedy) noise(v0, rr);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (v0 + j < end) {
            const float s = greedy ? x[j] : x[j] + gumbel(rr[j]);
            if (s > best) {  // indices only grow inside a thread: ties keep the lowest
              best = s;
              best_i = v0 + j;
            }
          }
        }
      }
    }
    cluster_sync_all();  // every block of the cluster runs: its shared memory may be written
  } else {
#pragma unroll 4
    for (int i = tid; i < quads; i += SMP_THREADS) {
      float x[4];
      load4_logits(lg, vec, begin + i * 4, end, x);
      mx = fmaxf(mx, fmaxf(fmaxf(x[0], x[1]), fmaxf(x[2], x[3])) * inv_t);
    }
    mx = warp_reduce_max(mx);
    if (lane == 0) sh.red_a[warp] = mx;
    cluster_sync_all();  // every block of the cluster runs: its shared memory may be written
    mx = warp_reduce_max(sh.red_a[lane]);
    int turn = 0;
    if (C > 1) {
      const float m1[1] = {mx};
      cluster_exchange(sh, turn, rank, C, m1);
      for (int r = 0; r < C; ++r) mx = fmaxf(mx, sh.xch[turn][0][r]);
      turn ^= 1;
    }
    // Every pass takes a token's probability exp(below) / z by this one form: it comes out the same, bit by bit, where the threshold
    // is searched and where it is applied (the threshold can be the probability of the last token inside).
    auto below = [&](float y) { return __fmaf_rn(y, inv_t, -mx); };
    float z = 0.f;
#pragma unroll 4
    for (int i = tid; i < quads; i += SMP_THREADS) {
      float x[4];
      load4_logits(lg, vec, begin + i * 4, end, x);
#pragma unroll
      for (int j = 0; j < 4; ++j) z += __expf(below(x[j]));
    }
    z = block_sum(z, sh.red_a);
    if (C > 1) {
      const float z1[1] = {z};
      cluster_exchange(sh, turn, rank, C, z1);
      z = 0.f;
      for (int r = 0; r < C; ++r) z += sh.xch[turn][0][r];
      turn ^= 1;
    }
    // f(logits, probabilities, index of the first) for the groups of four that may hold a probability of `least` or more
    auto visit = [&](float least, auto f) {
      const float far = least > 0.f ? __logf(least * z) - 0.01f : -INFINITY;
#pragma unroll 4
      for (int i = tid; i < quads; i += SMP_THREADS) {
        float y[4], q[4];
        load4_logits(lg, vec, begin + i * 4, end, y);
        if (below(fmaxf(fmaxf(y[0], y[1]), fmaxf(y[2], y[3]))) < far) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) q[j] = __expf(below(y[j])) / z;
        f(y, q, begin + i * 4);
      }
    };
    // keep tokens with p >= thr. Bisection on thr in [0, p_max]: count(p >= thr) and mass(p >= thr) never grow with thr.
    // (top-k set) intersected with (top-p nucleus): thr = max(thr_k, thr_p), and thr <= max(thr_k, thr_p) iff either
    // constraint alone is still feasible at thr.
    auto feasible = [&](int n, float mass) { return (need_k && n >= k) || (need_p && mass >= tp); };
    float lo = 0.f, hi = 1.f / z;  // p_max = exp(0) / z
    // adds the block's and the cluster's numbers up; even ones are counts
    auto total = [&](auto& v) {
      constexpr int N = sizeof(v) / sizeof(float);
#pragma unroll
      for (int i = 0; i < N; ++i)
        v[i] = (i & 1) ? warp_reduce_sum(v[i]) : __int_as_float(__reduce_add_sync(0xffffffffu, (int)v[i]));
      __syncthreads();
      if (lane == 0) {
#pragma unroll
        for (int i = 0; i < N; ++i) sh.red_l[i][warp] = v[i];
      }
      __syncthreads();
#pragma unroll
      for (int i = 0; i < N; ++i)
        v[i] = (i & 1) ? warp_reduce_sum(sh.red_l[i][lane])
                       : __int_as_float(__reduce_add_sync(0xffffffffu, __float_as_int(sh.red_l[i][lane])));
      if (C > 1) {
        cluster_exchange(sh, turn, rank, C, v);
#pragma unroll
        for (int i = 0; i < N; ++i) {
          float a = 0.f;
          int n = 0;
          for (int r = 0; r < C; ++r) {
            a += sh.xch[turn][i][r];
            n += __float_as_int(sh.xch[turn][i][r]);
          }
          v[i] = (i & 1) ? a : __int_as_float(n);
        }
        turn ^= 1;
      }
    };
    // guesses: `cut` > 0 once one is feasible with few tokens above it
    float cut = 0.f;
    if (V > SMP_CAND) {
      float few = hi, many = 0.f;  // above the one too few tokens, above the other too many
      for (int pass = 0; pass < 6 && cut == 0.f; ++pass) {
        float level[SMP_LEVELS], sums[2 * SMP_LEVELS];
        const float ratio = pass == 0 || many == 0.f ? 0.0625f : exp2f(__log2f(many / few) * (1.f / (SMP_LEVELS + 1)));
#pragma unroll
        for (int l = 0; l < SMP_LEVELS; ++l) {
          level[l] = (l == 0 ? few : level[l - 1]) * ratio;
          sums[2 * l] = sums[2 * l + 1] = 0.f;  // a thread's counts are small whole numbers
        }
        visit(level[SMP_LEVELS - 1], [&](float (&)[4], float (&q)[4], int) {
#pragma unroll
          for (int l = 0; l < SMP_LEVELS; ++l)
#pragma unroll
            for (int j = 0; j < 4; ++j)
              if (q[j] >= level[l]) {
                sums[2 * l] += 1.f;
                sums[2 * l + 1] += q[j];
              }
        });
        total(sums);
        bool done = false;
#pragma unroll
        for (int l = 0; l < SMP_LEVELS; ++l) {
          const int n = __float_as_int(sums[2 * l]);
          if (!done) {
            if (!feasible(n, sums[2 * l + 1])) {
              few = level[l];
            } else {
              done = true;
              if (n <= SMP_CAND) cut = level[l];
              else many = level[l];
            }
          }
        }
        if (!(few > many && level[SMP_LEVELS - 1] > 0.f)) break;  // no number, or nothing left to divide
      }
    }

    int cnt_lo = V, cnt_hi = 0, it = 0;  // tokens at or above the bounds (hi: once it has moved, `hi_mass` is their mass)
    float hi_mass = 0.f;
    bool hi_moved = false;
    if (cut == 0.f) {
      for (; it < 30 && cnt_lo - cnt_hi > SMP_CAND; ++it) {
        const float mid = 0.5f * (lo + hi);
        float one[2] = {0.f, 0.f};
        visit(mid, [&](float (&)[4], float (&q)[4], int) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            one[0] += q[j] >= mid ? 1.f : 0.f;
            one[1] += q[j] >= mid ? q[j] : 0.f;
          }
        });
        total(one);
        const int n = __float_as_int(one[0]);
        if (feasible(n, one[1])) {
          lo = mid;
          cnt_lo = n;
        } else {
          hi = mid;
          cnt_hi = n;
          hi_mass = one[1];
          hi_moved = true;
        }
      }
    }
    if (it < 30) {
      // the few tokens that still decide, in a fixed order, to the first block of the cluster
      const float least = fmaxf(lo, cut);
      auto decides = [&](float q, int v) { return v < end && q >= least && !(hi_moved && q >= hi); };
      int mine = 0;
      visit(least, [&](float (&)[4], float (&q)[4], int v0) {
#pragma unroll
        for (int j = 0; j < 4; ++j) mine += decides(q[j], v0 + j) ? 1 : 0;
      });
      int incl = mine;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
      }
      __syncthreads();
      if (lane == 31) sh.red_i[warp] = incl;
      __syncthreads();
      const int before = __reduce_add_sync(0xffffffffu, lane < warp ? sh.red_i[lane] : 0);
      const float all_mine[1] = {__int_as_float(__reduce_add_sync(0xffffffffu, sh.red_i[lane]))};
      cluster_exchange(sh, turn, rank, C, all_mine);
      int at = before + incl - mine, all = 0;
      for (int r = 0; r < C; ++r) {
        const int t = __float_as_int(sh.xch[turn][0][r]);
        if (r < (int)rank) at += t;
        all += t;
      }
      if (mine > 0) {
        visit(least, [&](float (&)[4], float (&q)[4], int v0) {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (decides(q[j], v0 + j)) {
              if (at < SMP_CAND) st_cluster_f32(&sh.cand[at], 0, q[j]);
              ++at;
            }
        });
      }
      cluster_sync_all();
      if (rank == 0 && warp == 0) {
        all = min(all, SMP_CAND);
        for (; it < 30; ++it) {
          const float mid = 0.5f * (lo + hi);
          int n = 0;
          float mass = 0.f;
          if (mid >= cut) {
            for (int i = lane; i < all; i += 32) {
              const float q = sh.cand[i];
              n += q >= mid ? 1 : 0;
              mass += q >= mid ? q : 0.f;
            }
            n = cnt_hi + __reduce_add_sync(0xffffffffu, n);
            mass = hi_mass + warp_reduce_sum(mass);
          }
          if (mid < cut || feasible(n, mass)) lo = mid; else hi = mid;
        }
        if (lane < C) st_cluster_f32(&sh.thr, lane, lo);
      }
      cluster_sync_all();
      lo = sh.thr;
    }
    thr = lo;
    // Gumbel-max over the support, and its normaliser
    visit(thr, [&](float (&y)[4], float (&q)[4], int v0) {
      if (!(fmaxf(fmaxf(q[0], q[1]), fmaxf(q[2], q[3])) >= thr)) return;
      uint32_t rr[4];
      noise(v0, rr);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (v0 + j < end && q[j] >= thr) {
          const float d = below(y[j]);
          sum += __expf(d);
          const float s = d + gumbel(rr[j]);
          if (s > best) {
            best = s;
            best_i = v0 + j;
          }
        }
      }
    });
  }

  // winner and normaliser over the block, then over the cluster. Restricted rows: sums over the support, to the row's maximum.
  auto reduce = [&]() {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      merge_best(best, best_i, __shfl_xor_sync(0xffffffffu, best, o), __shfl_xor_sync(0xffffffffu, best_i, o));
      const float om = __shfl_xor_sync(0xffffffffu, mx, o), os = __shfl_xor_sync(0xffffffffu, sum, o);
      if (restricted) sum += os;
      else merge_max_sum(mx, sum, om, os);
    }
  };
  reduce();
  __syncthreads();
  if (lane == 0) {
    sh.red_a[warp] = best;
    sh.red_b[warp] = sum;
    sh.red_i[warp] = best_i;
    sh.red_l[0][warp] = mx;
  }
  __syncthreads();
  if (warp == 0) {
    best = sh.red_a[lane];
    sum = sh.red_b[lane];
    best_i = sh.red_i[lane];
    mx = sh.red_l[0][lane];
    reduce();
    if (lane == 0) {
      st_cluster_f32(&sh.fin_best[rank], 0, best);
      st_cluster_f32(&sh.fin_z[rank], 0, sum);
      st_cluster_f32(&sh.fin_m[rank], 0, mx);
      st_cluster_s32(&sh.fin_i[rank], 0, best_i);
    }
  }
  cluster_sync_all();
  if (rank == 0 && tid == 0) {
    for (int r = 1; r < C; ++r) {
      merge_best(best, best_i, sh.fin_best[r], sh.fin_i[r]);
      if (restricted) sum += sh.fin_z[r];
      else merge_max_sum(mx, sum, sh.fin_m[r], sh.fin_z[r]);
    }
    const int tok = best_i < V ? best_i : 0;
    token_out[row] = tok;
    if (logprob_out) logprob_out[row] = ((float)lg[tok] * inv_t - mx) - __logf(sum);
  }
}

}  // namespace vb

using namespace vb;

extern "C" int vb_ppo_loss(const float* logp, const float* old_logp, const float* adv, const float* mask,
                           const float* ref_logp, const float* entropy, const float* is_weight, float* d_logp,
                           float* d_entropy, float* metrics, long long n, float clip_low, float clip_high,
                           float clip_c, float kl_coef, int kl_type, float entropy_coeff, float inv_denom,
                           cudaStream_t stream) {
  if (n <= 0) return 0;
  PpoArgs a{logp, old_logp, adv, mask, ref_logp, entropy, is_weight, d_logp, d_entropy, metrics, n,
            clip_low, clip_high, clip_c, kl_coef, entropy_coeff, inv_denom, kl_type};
  long long g = (n + 255) / 256;
  if (g > 148 * 4) g = 148 * 4;
  ppo_loss_kernel<<<(int)g, 256, 0, stream>>>(a);
  vb_count_launch();
  return (int)cudaGetLastError();
}

extern "C" int vb_gae(const float* rewards, const float* values, const float* mask, float* adv, float* ret, int B,
                      int T, float gamma, float lam, cudaStream_t stream) {
  if (B <= 0 || T <= 0) return 0;
  gae_kernel<<<(B + 63) / 64, 64, 0, stream>>>(rewards, values, mask, adv, ret, B, T, gamma, lam);
  vb_count_launch();
  return (int)cudaGetLastError();
}

// work: 3 * num_groups floats, zeroed by this call.
extern "C" int vb_grpo_adv(const float* scores, const int* gid, const float* mask, float* adv, float* work, int B,
                           int T, int num_groups, float eps, int norm_by_std, cudaStream_t stream) {
  if (B <= 0) return 0;
  VB_CUDA_CHECK(cudaMemsetAsync(work, 0, sizeof(float) * 3 * num_groups, stream));
  group_stats_kernel<<<(B + 127) / 128, 128, 0, stream>>>(scores, gid, B, work, work + num_groups,
                                                         work + 2 * num_groups);
  group_adv_kernel<<<B, 128, 0, stream>>>(scores, gid, work, work + num_groups, work + 2 * num_groups, mask, adv, B,
                                          T, eps, norm_by_std);
  vb_count_launch(2);
  return (int)cudaGetLastError();
}

// logits: [B, V] (dtype 0 = fp32, 1 = bf16), row_stride in elements. temperature/top_k/top_p are
// per-row device arrays (null = 1.0 / off / off). step is a device counter mixed into the RNG so a
// CUDA-graph replay draws fresh numbers when the caller increments it.
extern "C" int vb_sample(const void* logits, int dtype, long long row_stride, int B, int V, const float* temperature,
                         const int* top_k, const float* top_p, unsigned long long seed, const long long* step,
                         long long* token_out, float* logprob_out, cudaStream_t stream) {
  if (B <= 0 || V <= 0) return 0;
  // one block per row and SM; several blocks per row while there are SMs without one (each with 4096 tokens or more)
  int C = 1;
  auto part = [&](int c) { return ((V + c - 1) / c + 3) / 4 * 4; };
  while (C < SMP_MAX_C && (long long)B * C * 2 <= vb_num_sms() && part(2 * C) >= 4096) C *= 2;
  const int per = part(C);
  if ((long long)B * C > 0x7fffffffLL) return -3;
  cudaError_t e;
#define VB_SAMPLE(T)                                                                                                          \
  vb_launch_ex(sample_kernel<T>, dim3(B * C), dim3(SMP_THREADS), 0, stream, (unsigned)C, false, (const T*)logits, row_stride,  \
               V, C, per, temperature, top_k, top_p, seed, step, token_out, logprob_out)
  e = dtype == 0 ? VB_SAMPLE(float) : VB_SAMPLE(__nv_bfloat16);
#undef VB_SAMPLE
  vb_count_launch();
  return e != cudaSuccess ? (int)e : (int)cudaGetLastError();
}

// ---------------------------------------------------------------------------------------------------------------
// Decode-step chaining: the last kernel of a decode step turns the sampled tokens into the inputs of the next step,
// so that several steps (replays of one CUDA graph) run back to back without the host in between.
//   ring:   out_tok / out_lp [kmax, B] row *bpos receives this step's tokens / log-probs (-1 / 0 for rows that ended)
//   rows that are alive: a row ends when it samples `eos` (unless flags bit 0 = ignore eos) or reaches its length limit
//           (position + 2 >= limit: the sequence then holds `limit` tokens); it stops advancing and its cache slot
//           becomes -1, which the KV write skips
//   others: ids <- token, pos += 1, lens += 1, slot <- block_table[pos / block_size] * block_size + pos % block_size
//           (the host has reserved the pages of the whole burst before it started)
// One block; also advances the sampler's step counter and *bpos.
namespace vb {
__global__ void decode_advance_kernel(const long long* __restrict__ tok, const float* __restrict__ lp,
                                      long long* __restrict__ ids, long long* __restrict__ pos,
                                      long long* __restrict__ slots, int* __restrict__ lens,
                                      const int* __restrict__ bt, int mb, int block_size, const int* __restrict__ limit,
                                      int* __restrict__ alive, const int* __restrict__ flags, long long eos,
                                      long long* __restrict__ out_tok, float* __restrict__ out_lp, int* bpos,
                                      long long* sampler_step, int B, int kmax) {
  const int s = *bpos;
  __syncthreads();
  for (int b = threadIdx.x; b < B; b += blockDim.x) {
    const int a = alive[b];
    const long long t = tok[b];
    if (s >= 0 && s < kmax) {
      out_tok[(long long)s * B + b] = a ? t : -1;
      out_lp[(long long)s * B + b] = a ? lp[b] : 0.f;
    }
    if (a) {
      // lens[b] counts the tokens in the cache after this step: the token just processed has index lens - 1. The
      // RoPE position may differ from the token index (multimodal RoPE offsets text after images), so slots and the
      // length limit follow the index and the position just advances by one.
      const long long ti = (long long)lens[b] - 1;
      const bool done = (((flags[b] & 1) == 0) && t == eos) || (ti + 2 >= (long long)limit[b]);
      if (done) {
        alive[b] = 0;
        slots[b] = -1;
      } else {
        const long long ni = ti + 1;
        const int blk = (int)(ni / block_size);
        ids[b] = t;
        pos[b] += 1;
        lens[b] += 1;
        slots[b] = blk < mb ? (long long)bt[(long long)b * mb + blk] * block_size + (ni % block_size) : -1;
        if (blk >= mb) alive[b] = 0;
      }
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    *bpos = s + 1;
    if (sampler_step != nullptr) *sampler_step += 1;
  }
}
}  // namespace vb

extern "C" int vb_decode_advance(const long long* tok, const float* lp, long long* ids, long long* pos, long long* slots,
                                 int* lens, const int* bt, int mb, int block_size, const int* limit, int* alive,
                                 const int* flags, long long eos, long long* out_tok, float* out_lp, int* bpos,
                                 long long* sampler_step, int B, int kmax, cudaStream_t stream) {
  if (B <= 0 || kmax <= 0 || block_size <= 0) return -3;
  vb::decode_advance_kernel<<<1, 256, 0, stream>>>(tok, lp, ids, pos, slots, lens, bt, mb, block_size, limit, alive, flags,
                                                   eos, out_tok, out_lp, bpos, sampler_step, B, kmax);
  vb_count_launch();
  return (int)cudaGetLastError();
}
