// The non-GEMM layers of the GPT-2 training step (embedding, layernorm, attention, GELU backward,
// residual, softmax + cross-entropy, AdamW), written for the model driver in model.cu. They keep the
// reference's tensor layouts (src/layers/*.cu of vnnm404/gpt2.cu: activations [B*T][C], qkv
// [B*T][3C] with q | k | v side by side, wte stored [C][V]) but not its kernels: attention is
// flash-style (no [B,NH,T,T] tensors; only the log-sum-exp per row is kept for the backward pass),
// softmax and cross-entropy are one pass that leaves dlogits in place of the logits, and layernorm
// works a row per warp. All fp32 CUDA-core code; the GEMMs around them are the tcgen05 path.
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdlib.h>
#include <string.h>
#include <math.h>

#include "layers.h"
#include "linear_internal.h"
#include "ptx_sm100.cuh"

namespace g2l {

static inline int cdiv(long long a, int b) { return (int)((a + b - 1) / b); }

// ------------------------------------------------------------------------------------
// embedding: out[m][c] = wte[c][tok[m]] + wpe[t][c]     (reference: embedding.cu:11-27; wte is [C][V])
// ------------------------------------------------------------------------------------
__global__ void embedding_forward_kernel(float *out, const int *tokens, const float *wte, const float *wpe, int M,
                                         int T, int C, int Vp) {
  ptx::pdl_trigger();
  ptx::pdl_wait();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (long long)M * C) return;
  const int m = (int)(i / C), c = (int)(i % C);
  const int tok = tokens[m], t = m % T;
  out[i] = wte[(long long)c * Vp + tok] + wpe[(long long)t * C + c];
}

// g_wte[c][tok] += g[m][c]; g_wpe[t][c] += g[m][c]. (The reference indexes g_wte as [V][C] here,
// embedding.cu:93, which does not match its own forward; the PyTorch model is the semantics kept.)
__global__ void embedding_backward_kernel(float *g_wte, float *g_wpe, const float *g, const int *tokens, int M, int T,
                                          int C, int Vp) {
  ptx::pdl_trigger();
  ptx::pdl_wait();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (long long)M * C) return;
  const int m = (int)(i / C), c = (int)(i % C);
  const int tok = tokens[m], t = m % T;
  const float v = g[i];
  atomicAdd(g_wte + (long long)c * Vp + tok, v);
  atomicAdd(g_wpe + (long long)t * C + c, v);
}

// ------------------------------------------------------------------------------------
// layernorm, one warp per row (eps 1e-5 as layernorm.cu:54-116)
// ------------------------------------------------------------------------------------
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__global__ void __launch_bounds__(256)
layernorm_forward_kernel(float *out, float *mean, float *rstd, const float *in, const float *w, const float *b,
                         int M, int C) {
  ptx::pdl_trigger();
  ptx::pdl_wait();
  const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (row >= M) return;
  const float *x = in + (long long)row * C;
  float s = 0.f;
  for (int c = lane; c < C; c += 32) s += x[c];
  const float mu = warp_sum(s) / C;
  float v = 0.f;
  for (int c = lane; c < C; c += 32) { const float d = x[c] - mu; v += d * d; }
  const float rs = rsqrtf(warp_sum(v) / C + 1e-5f);
  float *o = out + (long long)row * C;
  for (int c = lane; c < C; c += 32) o[c] = (x[c] - mu) * rs * w[c] + b[c];
  if (lane == 0) { mean[row] = mu; rstd[row] = rs; }
}

// the same with the row held in registers (K4 float4 per lane): one read of x, one write of out
template <int K4>  // C <= 128 * K4, C a multiple of 4
__global__ void __launch_bounds__(256)
layernorm_forward_vec_kernel(float *out, float *mean, float *rstd, const float *in, const float *w, const float *b,
                             int M, int C) {
  ptx::pdl_trigger();
  ptx::pdl_wait();
  const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (row >= M) return;
  const float *x = in + (long long)row * C;
  float4 v[K4];
  float s = 0.f;
#pragma unroll
  for (int k = 0; k < K4; ++k) {
    const int c = 4 * (lane + 32 * k);
    v[k] = c < C ? *reinterpret_cast<const float4 *>(x + c) : make_float4(0.f, 0.f, 0.f, 0.f);
    s += v[k].x + v[k].y + v[k].z + v[k].w;
  }
  const float mu = warp_sum(s) / C;
  float q = 0.f;
#pragma unroll
  for (int k = 0; k < K4; ++k) {
    const int c = 4 * (lane + 32 * k);
    if (c < C) {
      const float dx = v[k].x - mu, dy = v[k].y - mu, dz = v[k].z - mu, dw = v[k].w - mu;
      q += dx * dx + dy * dy + dz * dz + dw * dw;
    }
  }
  const float rs = rsqrtf(warp_sum(q) / C + 1e-5f);
  float *o = out + (long long)row * C;
#pragma unroll
  for (int k = 0; k < K4; ++k) {
    const int c = 4 * (lane + 32 * k);
    if (c < C) {
      const float4 wv = __ldg(reinterpret_cast<const float4 *>(w + c));
      const float4 bv = __ldg(reinterpret_cast<const float4 *>(b + c));
      *reinterpret_cast<float4 *>(o + c) =
          make_float4((v[k].x - mu) * rs * wv.x + bv.x, (v[k].y - mu) * rs * wv.y + bv.y,
                      (v[k].z - mu) * rs * wv.z + bv.z, (v[k].w - mu) * rs * wv.w + bv.w);
    }
  }
  if (lane == 0) { mean[row] = mu; rstd[row] = rs; }
}

// g_in[row] += layernorm backward of g_out[row]; g_w / g_b accumulate over rows. A warp owns a row at a
// time and lane l always owns columns l, l+32, ...: the column sums for g_w / g_b stay in registers
// across the rows of the block and are combined once (the warps' sums halve twice through shared memory, then one
// atomicAdd per column per block). A warp's rows are a chain of dependent reductions, so a short batch gets a
// row per warp: 256 rows x 768 in blocks of 32 rows took 15.7 us (8 blocks), 5.0 us in blocks of 8.
template <int K4>  // float4 columns per lane: C <= 128 * K4 (C is a multiple of 4)
__global__ void __launch_bounds__(256, (K4 <= 6 ? 2 : 1))
layernorm_backward_kernel(float *g_in, float *g_w, float *g_b, const float *g_out, const float *in, const float *w,
                          const float *mean, const float *rstd, int M, int C, int rows_per_block) {
  ptx::pdl_trigger();
  ptx::pdl_wait();
  extern __shared__ __align__(16) float sm[];  // [4][C]: column sums of four warps
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
  float4 aw[K4], ab[K4];
#pragma unroll
  for (int k = 0; k < K4; ++k) {
    aw[k] = make_float4(0.f, 0.f, 0.f, 0.f);
    ab[k] = aw[k];
  }
  const int r0 = blockIdx.x * rows_per_block;
  const int r1 = min(M, r0 + rows_per_block);
  for (int row = r0 + warp; row < r1; row += nwarps) {
    const float *x = in + (long long)row * C;
    const float *go = g_out + (long long)row * C;
    const float mu = mean[row], rs = rstd[row];
    float *gi = g_in + (long long)row * C;
    float4 nh[K4], g[K4], o[K4];
    float s1 = 0.f, s2 = 0.f;
#pragma unroll
    for (int k = 0; k < K4; ++k) {  // needed last, fetched first: its latency hides behind the two reductions
      const int c = 4 * (lane + 32 * k);
      if (c < C) o[k] = *reinterpret_cast<const float4 *>(gi + c);
    }
#pragma unroll
    for (int k = 0; k < K4; ++k) {
      const int c = 4 * (lane + 32 * k);
      const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
      const float4 xv = c < C ? *reinterpret_cast<const float4 *>(x + c) : make_float4(mu, mu, mu, mu);
      g[k] = c < C ? *reinterpret_cast<const float4 *>(go + c) : zero;
      nh[k] = make_float4((xv.x - mu) * rs, (xv.y - mu) * rs, (xv.z - mu) * rs, (xv.w - mu) * rs);
      const float4 wv = c < C ? __ldg(reinterpret_cast<const float4 *>(w + c)) : zero;
      const float4 dn = make_float4(g[k].x * wv.x, g[k].y * wv.y, g[k].z * wv.z, g[k].w * wv.w);
      s1 += dn.x + dn.y + dn.z + dn.w;
      s2 += dn.x * nh[k].x + dn.y * nh[k].y + dn.z * nh[k].z + dn.w * nh[k].w;
    }
    s1 = warp_sum(s1) / C;
    s2 = warp_sum(s2) / C;
#pragma unroll
    for (int k = 0; k < K4; ++k) {
      const int c = 4 * (lane + 32 * k);
      if (c < C) {
        const float4 wv = __ldg(reinterpret_cast<const float4 *>(w + c));
        o[k].x += (g[k].x * wv.x - s1 - nh[k].x * s2) * rs;
        o[k].y += (g[k].y * wv.y - s1 - nh[k].y * s2) * rs;
        o[k].z += (g[k].z * wv.z - s1 - nh[k].z * s2) * rs;
        o[k].w += (g[k].w * wv.w - s1 - nh[k].w * s2) * rs;
        *reinterpret_cast<float4 *>(gi + c) = o[k];
      }
      aw[k].x += g[k].x * nh[k].x; aw[k].y += g[k].y * nh[k].y; aw[k].z += g[k].z * nh[k].z; aw[k].w += g[k].w * nh[k].w;
      ab[k].x += g[k].x; ab[k].y += g[k].y; ab[k].z += g[k].z; ab[k].w += g[k].w;
    }
  }
  // (eight warps) 4..7 hand their sums to 0..3, then the four are added column by column
  auto combine = [&](float4 (&v)[K4], float *dst) {
    float4 *buf = reinterpret_cast<float4 *>(sm + (warp & 3) * C);
    if (warp >= 4) {
#pragma unroll
      for (int k = 0; k < K4; ++k)
        if (4 * (lane + 32 * k) < C) buf[lane + 32 * k] = v[k];
    }
    __syncthreads();
    if (warp < 4) {
#pragma unroll
      for (int k = 0; k < K4; ++k)
        if (4 * (lane + 32 * k) < C) {
          const float4 t = buf[lane + 32 * k];
          buf[lane + 32 * k] = make_float4(v[k].x + t.x, v[k].y + t.y, v[k].z + t.z, v[k].w + t.w);
        }
    }
    __syncthreads();
    for (int c = threadIdx.x; c < C; c += blockDim.x) atomicAdd(dst + c, (sm[c] + sm[C + c]) + (sm[2 * C + c] + sm[3 * C + c]));
    __syncthreads();
  };
  combine(aw, g_w);
  combine(ab, g_b);
}

// ------------------------------------------------------------------------------------
// elementwise
// ------------------------------------------------------------------------------------
__global__ void add_kernel(float *out, const float *a, const float *b, long long n) {
  const long long i = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * 4;
  if (i + 3 < n) {
    const float4 x = *reinterpret_cast<const float4 *>(a + i), y = *reinterpret_cast<const float4 *>(b + i);
    *reinterpret_cast<float4 *>(out + i) = make_float4(x.x + y.x, x.y + y.y, x.z + y.z, x.w + y.w);
  } else {
    for (long long j = i; j < n; ++j) out[j] = a[j] + b[j];
  }
}

__device__ __forceinline__ float gelu_grad(float x) {
  const float k = 0.7978845608028654f;
  const float cube = 0.044715f * x * x * x;
  const float th = tanhf(k * (x + cube));
  const float sech2 = 1.f - th * th;
  return 0.5f * (1.f + th) + x * 0.5f * sech2 * k * (1.f + 3.f * 0.044715f * x * x);
}
// g[i] = g[i] * gelu'(pre[i])     (gelu.cu:49-63 computes the same derivative, accumulating)
__global__ void gelu_backward_kernel(float *g, const float *pre, long long n) {
  const long long i = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * 4;
  if (i + 3 < n) {
    float4 gv = *reinterpret_cast<float4 *>(g + i);
    const float4 p = *reinterpret_cast<const float4 *>(pre + i);
    gv.x *= gelu_grad(p.x); gv.y *= gelu_grad(p.y); gv.z *= gelu_grad(p.z); gv.w *= gelu_grad(p.w);
    *reinterpret_cast<float4 *>(g + i) = gv;
  } else {
    for (long long j = i; j < n; ++j) g[j] *= gelu_grad(pre[j]);
  }
}

// ------------------------------------------------------------------------------------
// softmax + cross-entropy, one block per row: loss[row] = -log softmax(logits[row])[target], and the
// logits row is overwritten with dlogits = (p - onehot) * scale (pad columns V..Vp-1 get 0).
// (reference: softmax.cu, cross_entropy.cu:24-93; scale = 1 / (B*T).)
// ------------------------------------------------------------------------------------
__global__ void __launch_bounds__(1024)
softmax_xent_kernel(float *logits, float *losses, const int *targets, int V, int Vp, float scale) {
  // the row (V floats, 196 KiB for GPT-2) is read from HBM once and kept in shared memory
  extern __shared__ float srow[];
  __shared__ float red[32];
  float *row = logits + (long long)blockIdx.x * Vp;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
  float mx = -INFINITY;
  const int V4 = V & ~3;
  for (int c = tid * 4; c < V4; c += blockDim.x * 4) {
    const float4 v = *reinterpret_cast<const float4 *>(row + c);
    *reinterpret_cast<float4 *>(srow + c) = v;
    mx = fmaxf(fmaxf(mx, fmaxf(v.x, v.y)), fmaxf(v.z, v.w));
  }
  for (int c = V4 + tid; c < V; c += blockDim.x) { const float v = row[c]; srow[c] = v; mx = fmaxf(mx, v); }
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if (lane == 0) red[warp] = mx;
  __syncthreads();
  mx = red[0];
  for (int i = 1; i < nw; ++i) mx = fmaxf(mx, red[i]);
  __syncthreads();
  float s = 0.f;
  for (int c = tid; c < V; c += blockDim.x) { const float e = __expf(srow[c] - mx); srow[c] = e; s += e; }
  s = warp_sum(s);
  if (lane == 0) red[warp] = s;
  __syncthreads();
  s = 0.f;
  for (int i = 0; i < nw; ++i) s += red[i];
  const int tgt = targets[blockIdx.x];
  const float inv = 1.f / s;
  if (tid == 0) losses[blockIdx.x] = -logf(srow[tgt] * inv);
  const float k = inv * scale;
  for (int c = tid * 4; c < Vp; c += blockDim.x * 4) {  // Vp is a multiple of 4
    float4 g;
    g.x = c + 0 < V ? srow[c + 0] * k - (c + 0 == tgt ? scale : 0.f) : 0.f;
    g.y = c + 1 < V ? srow[c + 1] * k - (c + 1 == tgt ? scale : 0.f) : 0.f;
    g.z = c + 2 < V ? srow[c + 2] * k - (c + 2 == tgt ? scale : 0.f) : 0.f;
    g.w = c + 3 < V ? srow[c + 3] * k - (c + 3 == tgt ? scale : 0.f) : 0.f;
    *reinterpret_cast<float4 *>(row + c) = g;
  }
}

// The same without shared-memory staging: pass 1 streams the row from HBM once and keeps a running
// (max, sum) pair per thread; pass 2 reads the row again (from L2: the rows in flight on all SMs are a few
// tens of MB) and writes dlogits. No large shared-memory footprint, so several blocks share an SM and
// the loads of one row overlap the stores of another.
__global__ void __launch_bounds__(512, 3)
softmax_xent_online_kernel(float *logits, float *losses, const int *targets, int V, int Vp, float scale) {
  __shared__ float red_m[16], red_s[16];
  float *row = logits + (long long)blockIdx.x * Vp;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const float L2E = 1.4426950408889634f;
  float m = -INFINITY, s = 0.f;  // base-2 domain: m = max(x * log2e), s = sum 2^(x*log2e - m)
  const int V4 = V & ~3;
  for (int c = tid * 4; c < V4; c += 512 * 4) {
    float4 v = *reinterpret_cast<const float4 *>(row + c);
    v.x *= L2E; v.y *= L2E; v.z *= L2E; v.w *= L2E;
    const float mn = fmaxf(fmaxf(m, fmaxf(v.x, v.y)), fmaxf(v.z, v.w));
    s = s * exp2f(m - mn) + exp2f(v.x - mn) + exp2f(v.y - mn) + exp2f(v.z - mn) + exp2f(v.w - mn);
    m = mn;
  }
  for (int c = V4 + tid; c < V; c += 512) {
    const float v = row[c] * L2E;
    const float mn = fmaxf(m, v);
    s = s * exp2f(m - mn) + exp2f(v - mn);
    m = mn;
  }
  // combine (m, s) pairs: warp, then block. A thread that saw no element holds (-inf, 0); guard the
  // -inf - -inf case.
  for (int o = 16; o > 0; o >>= 1) {
    const float m2 = __shfl_xor_sync(0xffffffffu, m, o), s2 = __shfl_xor_sync(0xffffffffu, s, o);
    const float mn = fmaxf(m, m2);
    s = (m == -INFINITY ? 0.f : s * exp2f(m - mn)) + (m2 == -INFINITY ? 0.f : s2 * exp2f(m2 - mn));
    m = mn;
  }
  if (lane == 0) { red_m[warp] = m; red_s[warp] = s; }
  __syncthreads();
  m = red_m[0]; s = red_s[0];
  for (int i = 1; i < 16; ++i) {
    const float m2 = red_m[i], s2 = red_s[i];
    const float mn = fmaxf(m, m2);
    s = (m == -INFINITY ? 0.f : s * exp2f(m - mn)) + (m2 == -INFINITY ? 0.f : s2 * exp2f(m2 - mn));
    m = mn;
  }
  const int tgt = targets[blockIdx.x];
  // loss = -(x_t - max - ln(sum)) in natural units
  if (tid == 0) losses[blockIdx.x] = -((row[tgt] * L2E - m) - log2f(s)) * 0.6931471805599453f;
  __syncthreads();  // the target logit is read before anyone overwrites it
  const float k = scale / s;
  for (int c = tid * 4; c < Vp; c += 512 * 4) {  // Vp is a multiple of 4
    float4 g = *reinterpret_cast<const float4 *>(row + c);
    g.x = c + 0 < V ? exp2f(g.x * L2E - m) * k - (c + 0 == tgt ? scale : 0.f) : 0.f;
    g.y = c + 1 < V ? exp2f(g.y * L2E - m) * k - (c + 1 == tgt ? scale : 0.f) : 0.f;
    g.z = c + 2 < V ? exp2f(g.z * L2E - m) * k - (c + 2 == tgt ? scale : 0.f) : 0.f;
    g.w = c + 3 < V ? exp2f(g.w * L2E - m) * k - (c + 3 == tgt ? scale : 0.f) : 0.f;
    *reinterpret_cast<float4 *>(row + c) = g;
  }
}

// the same in three passes over global memory, for vocabularies that do not fit in shared memory
__global__ void __launch_bounds__(512)
softmax_xent_large_kernel(float *logits, float *losses, const int *targets, int V, int Vp, float scale) {
  __shared__ float red[32];
  float *row = logits + (long long)blockIdx.x * Vp;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
  float mx = -INFINITY;
  for (int c = tid; c < V; c += blockDim.x) mx = fmaxf(mx, row[c]);
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if (lane == 0) red[warp] = mx;
  __syncthreads();
  mx = red[0];
  for (int i = 1; i < nw; ++i) mx = fmaxf(mx, red[i]);
  __syncthreads();
  float s = 0.f;
  for (int c = tid; c < V; c += blockDim.x) s += expf(row[c] - mx);
  s = warp_sum(s);
  if (lane == 0) red[warp] = s;
  __syncthreads();
  s = 0.f;
  for (int i = 0; i < nw; ++i) s += red[i];
  const int tgt = targets[blockIdx.x];
  const float inv = 1.f / s;
  if (tid == 0) losses[blockIdx.x] = -(row[tgt] - mx - logf(s));
  __syncthreads();
  for (int c = tid; c < Vp; c += blockDim.x) {
    float g = 0.f;
    if (c < V) g = (expf(row[c] - mx) * inv - (c == tgt ? 1.f : 0.f)) * scale;
    row[c] = g;
  }
}

// ------------------------------------------------------------------------------------
// second half of the fused lm_head + softmax + cross-entropy: the GEMM epilogue left, per row and per
// column tile, (max, sum of 2^(x - max)) in the base-2 domain; a warp per row folds the `stride` pairs into
// lse[m] = max + log2(sum) and losses[m] = (lse[m] - logit[m][target] * log2 e) * ln 2.
// ------------------------------------------------------------------------------------
__global__ void xent_combine_kernel(float *lse, float *losses, const float2 *stats, int stride, const float *logits,
                                    long long ld, const int *targets, int M) {
  ptx::pdl_trigger();
  ptx::pdl_wait();
  const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (row >= M) return;
  const float2 *s = stats + (size_t)row * stride;
  float m = -INFINITY, sum = 0.f;
  for (int i = lane; i < stride; i += 32) {
    const float2 v = s[i];
    const float mn = fmaxf(m, v.x);
    if (mn > -INFINITY) sum = (m == -INFINITY ? 0.f : sum * exp2f(m - mn)) + (v.x == -INFINITY ? 0.f : v.y * exp2f(v.x - mn));
    m = mn;
  }
  for (int o = 16; o > 0; o >>= 1) {
    const float m2 = __shfl_xor_sync(0xffffffffu, m, o), s2 = __shfl_xor_sync(0xffffffffu, sum, o);
    const float mn = fmaxf(m, m2);
    sum = (m == -INFINITY ? 0.f : sum * exp2f(m - mn)) + (m2 == -INFINITY ? 0.f : s2 * exp2f(m2 - mn));
    m = mn;
  }
  if (lane == 0) {
    const float l2 = m + log2f(sum);
    lse[row] = l2;
    losses[row] = (l2 - logits[(long long)row * ld + targets[row]] * 1.4426950408889634f) * 0.6931471805599453f;
  }
}

// logits[m][c] <- (2^(logits[m][c] log2 e - lse[m]) - [c == target[m]]) * scale for c < V, 0 for the pad columns:
// the gradient of the mean cross-entropy, in place, one read and one write of the tensor (the row maxima and
// sums are known already, so nothing is reduced here). A block per row.
__global__ void __launch_bounds__(512)
xent_grad_inplace_kernel(float *logits, const float *lse, const int *targets, int V, int Vp, float scale) {
  ptx::pdl_trigger();
  ptx::pdl_wait();
  float *row = logits + (long long)blockIdx.x * Vp;
  const float l2 = lse[blockIdx.x];
  const int tgt = targets[blockIdx.x];
  const float L2E = 1.4426950408889634f;
  for (int c = threadIdx.x * 4; c < Vp; c += 512 * 4) {  // Vp is a multiple of 4
    float4 g = *reinterpret_cast<const float4 *>(row + c);
    g.x = c + 0 < V ? (exp2f(g.x * L2E - l2) - (c + 0 == tgt ? 1.f : 0.f)) * scale : 0.f;
    g.y = c + 1 < V ? (exp2f(g.y * L2E - l2) - (c + 1 == tgt ? 1.f : 0.f)) * scale : 0.f;
    g.z = c + 2 < V ? (exp2f(g.z * L2E - l2) - (c + 2 == tgt ? 1.f : 0.f)) * scale : 0.f;
    g.w = c + 3 < V ? (exp2f(g.w * L2E - l2) - (c + 3 == tgt ? 1.f : 0.f)) * scale : 0.f;
    *reinterpret_cast<float4 *>(row + c) = g;
  }
}

// ------------------------------------------------------------------------------------
// causal self-attention in fp32, flash style, head size 64, any sequence length. qkv[m][3C] = q | k | v, head h at
// columns h*64. forward: out[m][h*64 + d], lse[b][h][t] = log sum_j exp(q_t.k_j / 8).
//
// Everything is 64 x 64 tiles of a block of 256 threads: thread (ty, tx) holds rows ty + 16 i and columns tx + 16 j of a
// score tile (i, j < 4), rows ty + 16 i and columns 4 tx .. 4 tx + 3 of an output tile. All tiles sit in shared memory as
// they do in memory, rows of 64 with a pitch of 68 floats: a score takes both operands four d at a time and keeps two
// partial sums (even and odd d) in a packed FMA, an output takes a row of the second operand, and neither read has a
// bank conflict. A score tile is written and read back by the same 16 lanes, so it needs no barrier of the block.
// Bound by the FMA pipe: 4 x 777 tokens, 12 heads, forward 403 -> 135 us, dq 448 -> 181, dk and dv 660 -> 245 against a
// thread per row with single FMAs (which waited for a chain of 64 FMAs per key).
// Masked scores take no part in a product, so a NaN or infinity in a later token does not reach an earlier one.
// ------------------------------------------------------------------------------------
constexpr int HS = 64;
constexpr int AT = ATT_TILE;  // tile edge
constexpr int ALD = AT + 4;   // tile pitch in floats
constexpr int ATILE = AT * ALD;
constexpr int ATT_THREADS = 256;

// rows row0 .. row0 + 63 of a [T][ld] matrix (64 columns), zeros past the end
__device__ __forceinline__ void att_load(float *tile, const float *src, long long ld, int row0, int T) {
#pragma unroll
  for (int i = 0; i < AT * HS / 4 / ATT_THREADS; ++i) {
    const int e = threadIdx.x + i * ATT_THREADS, r = e >> 4, c = (e & 15) * 4;
    const bool live = row0 + r < T;
    const float *from = live ? src + (long long)(row0 + r) * ld + c : src;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(tile + r * ALD + c)),
                 "l"(from), "r"(live ? 16 : 0)
                 : "memory");
  }
}
__device__ __forceinline__ void att_loads_done() {
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
}

__device__ __forceinline__ float pair_sum(unsigned long long v) {
  return __uint_as_float((uint32_t)v) + __uint_as_float((uint32_t)(v >> 32));
}

// s[i][j] = sum_d A[ty + 16 i][d] * B[tx + 16 j][d]
__device__ __forceinline__ void att_dot(float (&s)[4][4], const float *A, const float *B, int ty, int tx) {
  unsigned long long acc[4][4] = {};
#pragma unroll 4
  for (int d = 0; d < HS; d += 4) {
    ulonglong2 a[4], b[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) a[i] = *reinterpret_cast<const ulonglong2 *>(A + (ty + 16 * i) * ALD + d);
#pragma unroll
    for (int j = 0; j < 4; ++j) b[j] = *reinterpret_cast<const ulonglong2 *>(B + (tx + 16 * j) * ALD + d);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = ptx::fma2(a[i].y, b[j].y, ptx::fma2(a[i].x, b[j].x, acc[i][j]));
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) s[i][j] = pair_sum(acc[i][j]);
}

// acc[i] (columns 4 tx ..) += sum_k P[ty + 16 i][k] * V[k][4 tx ..]. DIAG: only the k a row may see, k <= row (+1) or
// k >= row (-1), row and k counted from the same token.
template <int DIAG>
__device__ __forceinline__ void att_axpy(unsigned long long (&acc)[4][2], const float *P, const float *V, int ty, int tx) {
#pragma unroll 2
  for (int k = 0; k < AT; k += 4) {
    float p[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float4 v = *reinterpret_cast<const float4 *>(P + (ty + 16 * i) * ALD + k);
      p[i][0] = v.x; p[i][1] = v.y; p[i][2] = v.z; p[i][3] = v.w;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const ulonglong2 v = *reinterpret_cast<const ulonglong2 *>(V + (k + u) * ALD + 4 * tx);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (DIAG > 0 && k + u > ty + 16 * i) continue;
        if (DIAG < 0 && k + u < ty + 16 * i) continue;
        const unsigned long long w = ptx::both(p[i][u]);
        acc[i][0] = ptx::fma2(w, v.x, acc[i][0]);
        acc[i][1] = ptx::fma2(w, v.y, acc[i][1]);
      }
    }
  }
}

__device__ __forceinline__ float4 att_quad(const unsigned long long (&a)[2], float scale) {
  return make_float4(__uint_as_float((uint32_t)a[0]) * scale, __uint_as_float((uint32_t)(a[0] >> 32)) * scale,
                     __uint_as_float((uint32_t)a[1]) * scale, __uint_as_float((uint32_t)(a[1] >> 32)) * scale);
}

template <bool LONG>  // one of several launches (att_launch_tiles)
__global__ void __launch_bounds__(ATT_THREADS, 2)
attention_forward_kernel(float *out, float *lse, const float *qkv, int T, int C, int NH, int last) {
  extern __shared__ __align__(16) float sm[];
  float *sq = sm, *sk = sm + ATILE, *sv = sm + 2 * ATILE, *sp = sm + 3 * ATILE;
  const int h = blockIdx.x, b = blockIdx.y, q0 = ((LONG ? last + 1 : gridDim.z) - 1 - blockIdx.z) * AT;  // the longest rows first
  const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
  const float scale = 0.125f;  // 1 / sqrt(64)
  const long long ld = 3LL * C;
  const float *base = qkv + (long long)b * T * ld + h * HS;
  att_load(sq, base, ld, q0, T);
  unsigned long long acc[4][2] = {};
  float m[4], l[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) { m[i] = -INFINITY; l[i] = 0.f; }
  for (int k0 = 0; k0 <= q0; k0 += AT) {
    if (k0) __syncthreads();  // everyone is done with the previous keys
    att_load(sk, base + C, ld, k0, T);
    att_load(sv, base + 2 * C, ld, k0, T);
    att_loads_done();
    float s[4][4];
    att_dot(s, sq, sk, ty, tx);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float mx = -INFINITY;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        s[i][j] = (k0 == q0 && tx + 16 * j > ty + 16 * i) ? -INFINITY : s[i][j] * scale;
        mx = fmaxf(mx, s[i][j]);
      }
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      const float mn = fmaxf(m[i], mx);  // finite from the first tile on: key 0 is seen by every row
      const float corr = __expf(m[i] - mn);
      float sum = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float p = __expf(s[i][j] - mn);
        sp[(ty + 16 * i) * ALD + tx + 16 * j] = p;
        sum += p;
      }
      l[i] = l[i] * corr + sum;  // (this lane's keys; the lanes meet at the end)
      m[i] = mn;
      const unsigned long long c2 = ptx::both(corr);
      acc[i][0] = ptx::fma2(acc[i][0], c2, 0ull);
      acc[i][1] = ptx::fma2(acc[i][1], c2, 0ull);
    }
    __syncwarp();
    if (k0 == q0) att_axpy<1>(acc, sp, sv, ty, tx);
    else att_axpy<0>(acc, sp, sv, ty, tx);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int t = q0 + ty + 16 * i;
    float li = l[i];
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) li += __shfl_xor_sync(0xffffffffu, li, o);
    if (t >= T) continue;
    *reinterpret_cast<float4 *>(out + ((long long)b * T + t) * C + h * HS + 4 * tx) = att_quad(acc[i], 1.f / li);
    if (tx == 0) lse[((long long)b * NH + h) * T + t] = m[i] + logf(li);
  }
}

// dS_ij = p_ij (dO_i.V_j - delta_i), dQ_i = sum_j dS_ij K_j / 8
template <bool LONG>  // one of several launches (att_launch_tiles)
__global__ void __launch_bounds__(ATT_THREADS, 2)
attention_backward_dq_kernel(float *dqkv, const float *dout, const float *qkv, const float *lse, const float *delta,
                             int T, int C, int NH, int last) {
  extern __shared__ __align__(16) float sm[];
  float *sq = sm, *sg = sm + ATILE, *sk = sm + 2 * ATILE, *sv = sm + 3 * ATILE, *ss = sm + 4 * ATILE;
  const int h = blockIdx.x, b = blockIdx.y, q0 = ((LONG ? last + 1 : gridDim.z) - 1 - blockIdx.z) * AT;
  const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
  const float scale = 0.125f;
  const long long ld = 3LL * C, vbase = ((long long)b * NH + h) * T;
  const float *base = qkv + (long long)b * T * ld + h * HS;
  att_load(sq, base, ld, q0, T);
  att_load(sg, dout + (long long)b * T * C + h * HS, C, q0, T);
  float L[4], D[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int t = q0 + ty + 16 * i;
    L[i] = t < T ? lse[vbase + t] : 0.f;
    D[i] = t < T ? delta[vbase + t] : 0.f;
  }
  unsigned long long acc[4][2] = {};
  for (int k0 = 0; k0 <= q0; k0 += AT) {
    if (k0) __syncthreads();
    att_load(sk, base + C, ld, k0, T);
    att_load(sv, base + 2 * C, ld, k0, T);
    att_loads_done();
    float s[4][4], dp[4][4];
    att_dot(s, sq, sk, ty, tx);
    att_dot(dp, sg, sv, ty, tx);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j)
        ss[(ty + 16 * i) * ALD + tx + 16 * j] = __expf(s[i][j] * scale - L[i]) * (dp[i][j] - D[i]) * scale;
    __syncwarp();
    if (k0 == q0) att_axpy<1>(acc, ss, sk, ty, tx);
    else att_axpy<0>(acc, ss, sk, ty, tx);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int t = q0 + ty + 16 * i;
    if (t < T) *reinterpret_cast<float4 *>(dqkv + ((long long)b * T + t) * ld + h * HS + 4 * tx) = att_quad(acc[i], 1.f);
  }
}

// dV_j = sum_i p_ij dO_i;  dK_j = sum_i dS_ij Q_i / 8: rows of a tile are keys, its columns the queries at or after them
template <bool LONG>  // one of several launches (att_launch_tiles)
__global__ void __launch_bounds__(ATT_THREADS, 2)
attention_backward_dkv_kernel(float *dqkv, const float *dout, const float *qkv, const float *lse, const float *delta,
                              int T, int C, int NH, int first) {
  extern __shared__ __align__(16) float sm[];
  float *sk = sm, *sv = sm + ATILE, *sq = sm + 2 * ATILE, *sg = sm + 3 * ATILE, *sp = sm + 4 * ATILE, *ss = sm + 5 * ATILE;
  const int h = blockIdx.x, b = blockIdx.y, k0 = (blockIdx.z + (LONG ? first : 0)) * AT;  // the keys most queries see first
  const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
  const float scale = 0.125f;
  const long long ld = 3LL * C, vbase = ((long long)b * NH + h) * T;
  const float *base = qkv + (long long)b * T * ld + h * HS;
  att_load(sk, base + C, ld, k0, T);
  att_load(sv, base + 2 * C, ld, k0, T);
  unsigned long long dk[4][2] = {}, dv[4][2] = {};
  for (int q0 = k0; q0 < T; q0 += AT) {
    if (q0 != k0) __syncthreads();
    att_load(sq, base, ld, q0, T);
    att_load(sg, dout + (long long)b * T * C + h * HS, C, q0, T);
    float L[4], D[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int t = q0 + tx + 16 * j;
      L[j] = t < T ? lse[vbase + t] : 0.f;
      D[j] = t < T ? delta[vbase + t] : 0.f;
    }
    att_loads_done();
    float s[4][4], dp[4][4];
    att_dot(s, sk, sq, ty, tx);
    att_dot(dp, sv, sg, ty, tx);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const bool live = q0 + tx + 16 * j < T;  // (a zero score of a row past the end would count as e^0)
        const float p = __expf(s[i][j] * scale - L[j]);
        sp[(ty + 16 * i) * ALD + tx + 16 * j] = live ? p : 0.f;
        ss[(ty + 16 * i) * ALD + tx + 16 * j] = live ? p * (dp[i][j] - D[j]) * scale : 0.f;
      }
    __syncwarp();
    if (q0 == k0) {
      att_axpy<-1>(dv, sp, sg, ty, tx);
      att_axpy<-1>(dk, ss, sq, ty, tx);
    } else {
      att_axpy<0>(dv, sp, sg, ty, tx);
      att_axpy<0>(dk, ss, sq, ty, tx);
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int t = k0 + ty + 16 * i;
    if (t >= T) continue;
    float *row = dqkv + ((long long)b * T + t) * ld + h * HS + 4 * tx;
    *reinterpret_cast<float4 *>(row + C) = att_quad(dk[i], 1.f);
    *reinterpret_cast<float4 *>(row + 2 * C) = att_quad(dv[i], 1.f);
  }
}

// ------------------------------------------------------------------------------------
// AdamW over the flat parameter buffer; decay on every element, bias-corrected (adamw.cu:11-48)
// ------------------------------------------------------------------------------------
__device__ __forceinline__ void adamw_one(float &p, float &m, float &v, float gi, float lr, float b1, float b2, float eps,
                                          float wd, float bc1, float bc2) {
  const float mi = b1 * m + (1.f - b1) * gi;
  const float vi = b2 * v + (1.f - b2) * gi * gi;
  m = mi;
  v = vi;
  const float mh = mi / bc1, vh = vi / bc2;
  p -= lr * (mh / (sqrtf(vh) + eps) + wd * p);
}

// `head` scalar elements bring the pointers to a 16-byte boundary, then float4 elements, then a scalar
// tail (a range of the flat buffer may start anywhere); every element sees the same arithmetic.
__global__ void adamw_kernel(float *p, float *m, float *v, const float *g, long long n, long long head, long long n4,
                             float lr, float b1, float b2, float eps, float wd, float bc1, float bc2) {
  ptx::pdl_trigger();
  ptx::pdl_wait();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n4) {
    const long long o = head + 4 * i;
    float4 pp = *reinterpret_cast<float4 *>(p + o), mm = *reinterpret_cast<float4 *>(m + o),
           vv = *reinterpret_cast<float4 *>(v + o);
    const float4 gg = *reinterpret_cast<const float4 *>(g + o);
    adamw_one(pp.x, mm.x, vv.x, gg.x, lr, b1, b2, eps, wd, bc1, bc2);
    adamw_one(pp.y, mm.y, vv.y, gg.y, lr, b1, b2, eps, wd, bc1, bc2);
    adamw_one(pp.z, mm.z, vv.z, gg.z, lr, b1, b2, eps, wd, bc1, bc2);
    adamw_one(pp.w, mm.w, vv.w, gg.w, lr, b1, b2, eps, wd, bc1, bc2);
    *reinterpret_cast<float4 *>(p + o) = pp;
    *reinterpret_cast<float4 *>(m + o) = mm;
    *reinterpret_cast<float4 *>(v + o) = vv;
  } else {
    // the few elements before and after the aligned body
    const long long j = i - n4;
    const long long tail0 = head + 4 * n4;
    const long long o = j < head ? j : tail0 + (j - head);
    if (o < n) adamw_one(p[o], m[o], v[o], g[o], lr, b1, b2, eps, wd, bc1, bc2);
  }
}

// The gradients that a backward pass adds into, rather than writes: `head` floats (wpe) at g, then `pairs` layernorms of
// 2C floats each, two a layer (at first and first + second, layers `layer` floats apart), the last one behind all layers.
__global__ void __launch_bounds__(256)
zero_accumulated_kernel(float *g, long long head, float *first, long long second, long long layer, long long last, int pairs,
                        int two_c) {
  ptx::pdl_trigger();
  ptx::pdl_wait();
  const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
  if (i < head) {
    g[i] = 0.f;
    return;
  }
  const long long j = i - head;
  const int k = (int)(j / two_c), c = (int)(j % two_c);
  if (k >= pairs) return;
  const long long at = k == pairs - 1 ? last : (k >> 1) * layer + (k & 1) * second;
  first[at + c] = 0.f;
}

// ------------------------------------------------------------------------------------
// launchers
// ------------------------------------------------------------------------------------
#define LAUNCH_OK() (count_launch(), cudaGetLastError() == cudaSuccess ? GPT2L_OK : GPT2L_ERR_CUDA)
// (for launch_pdl, which returns the launch's own error)
static int launched(cudaError_t e) {
  count_launch();
  return e == cudaSuccess ? GPT2L_OK : GPT2L_ERR_CUDA;
}

int embedding_forward(float *out, const int *tokens, const float *wte, const float *wpe, int B, int T, int C, int Vp,
                      cudaStream_t s) {
  const long long n = (long long)B * T * C;
  return launched(launch_pdl(embedding_forward_kernel, cdiv(n, 256), 256, 0, s, out, tokens, wte, wpe, B * T, T, C, Vp));
}
int zero_accumulated(float *g, long long head, float *first, long long second, long long layer, long long last, int pairs,
                     int two_c, cudaStream_t s) {
  return launched(launch_pdl(zero_accumulated_kernel, cdiv(head + (long long)pairs * two_c, 256), 256, 0, s, g, head, first,
                             second, layer, last, pairs, two_c));
}
int embedding_backward(float *g_wte, float *g_wpe, const float *g, const int *tokens, int B, int T, int C, int Vp,
                       cudaStream_t s) {
  const long long n = (long long)B * T * C;
  return launched(launch_pdl(embedding_backward_kernel, cdiv(n, 256), 256, 0, s, g_wte, g_wpe, g, tokens, B * T, T, C, Vp));
}
int layernorm_forward(float *out, float *mean, float *rstd, const float *in, const float *w, const float *b, int M,
                      int C, cudaStream_t s) {
  auto launch = [&](auto kernel) {
    return launched(launch_pdl(kernel, cdiv(M, 8), 256, 0, s, out, mean, rstd, in, w, b, M, C));
  };
  if ((C & 3) || C > 2048) return launch(layernorm_forward_kernel);
  if (C <= 128) return launch(layernorm_forward_vec_kernel<1>);
  if (C <= 256) return launch(layernorm_forward_vec_kernel<2>);
  if (C <= 512) return launch(layernorm_forward_vec_kernel<4>);
  if (C <= 768) return launch(layernorm_forward_vec_kernel<6>);
  if (C <= 1024) return launch(layernorm_forward_vec_kernel<8>);
  if (C <= 1280) return launch(layernorm_forward_vec_kernel<10>);
  return launch(layernorm_forward_vec_kernel<16>);
}
int layernorm_backward(float *g_in, float *g_w, float *g_b, const float *g_out, const float *in, const float *w,
                       const float *mean, const float *rstd, int M, int C, cudaStream_t s) {
  // At most one block per resident slot (two per SM), so that all end at about the same time and the column sums meet in global
  // memory only ~300 times, and whole rounds of a row per warp: from 8 rows a slot on the rows of a block are rounded up to
  // 16, 24, ..., which leaves up to half of the slots idle just past each line (2376 rows: 149 blocks of 16).
  static const int slots = [] {
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0)
      sms = 148;
    return 2 * sms;
  }();
  const int rows_per_block = cdiv(cdiv(M, slots), 8) * 8;
  const int blocks = cdiv(M, rows_per_block);
  const size_t smem = 4 * (size_t)C * sizeof(float);
  if (C & 3) return GPT2L_ERR_BAD_ARG;
  auto launch = [&](auto kernel) {
    return launched(launch_pdl(kernel, blocks, 256, smem, s, g_in, g_w, g_b, g_out, in, w, mean, rstd, M, C, rows_per_block));
  };
  if (C <= 128) return launch(layernorm_backward_kernel<1>);
  if (C <= 256) return launch(layernorm_backward_kernel<2>);
  if (C <= 512) return launch(layernorm_backward_kernel<4>);
  if (C <= 768) return launch(layernorm_backward_kernel<6>);
  if (C <= 1024) return launch(layernorm_backward_kernel<8>);
  if (C <= 1280) return launch(layernorm_backward_kernel<10>);
  if (C <= 2048) return launch(layernorm_backward_kernel<16>);
  return GPT2L_ERR_TOO_LARGE;
}
int add_forward(float *out, const float *a, const float *b, long long n, cudaStream_t s) {
  add_kernel<<<cdiv((n + 3) / 4, 256), 256, 0, s>>>(out, a, b, n);
  return LAUNCH_OK();
}
int gelu_backward(float *g, const float *pre, long long n, cudaStream_t s) {
  gelu_backward_kernel<<<cdiv((n + 3) / 4, 256), 256, 0, s>>>(g, pre, n);
  return LAUNCH_OK();
}
int softmax_xent(float *logits, float *losses, const int *targets, int M, int V, int Vp, cudaStream_t s) {
  const size_t row_bytes = (size_t)V * sizeof(float);
  static const bool staged = [] { const char *e = getenv("GPT2_SOFTMAX_XENT"); return e && !strcmp(e, "staged"); }();
  if (!staged && (Vp & 3) == 0) {
    softmax_xent_online_kernel<<<M, 512, 0, s>>>(logits, losses, targets, V, Vp, 1.f / (float)M);
  } else if (row_bytes <= 220 * 1024) {
    // per device and cheap: set every time rather than tracking which devices have seen it
    if (cudaFuncSetAttribute(softmax_xent_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024) !=
        cudaSuccess)
      return GPT2L_ERR_CUDA;
    softmax_xent_kernel<<<M, 1024, row_bytes, s>>>(logits, losses, targets, V, Vp, 1.f / (float)M);
  } else {
    softmax_xent_large_kernel<<<M, 512, 0, s>>>(logits, losses, targets, V, Vp, 1.f / (float)M);
  }
  return LAUNCH_OK();
}
int launch_xent_combine(float *lse, float *losses, const float *stats, int stride, const float *logits, long long ld,
                        const int *targets, int M, cudaStream_t s) {
  return launched(launch_pdl(xent_combine_kernel, cdiv(M, 8), 256, 0, s, lse, losses, reinterpret_cast<const float2 *>(stats),
                             stride, logits, ld, targets, M));
}
int xent_grad_inplace(float *logits, const float *lse, const int *targets, int M, int V, int Vp, cudaStream_t s) {
  if (Vp & 3) return GPT2L_ERR_BAD_ARG;
  return launched(launch_pdl(xent_grad_inplace_kernel, M, 512, 0, s, logits, lse, targets, V, Vp, 1.f / (float)M));
}
template <bool LONG>
static int attention_forward_launches(float *out, float *lse, const float *qkv, int B, int T, int C, int NH, cudaStream_t s) {
  constexpr int smem = 4 * ATILE * (int)sizeof(float);
  // (per device and cheap: set every time rather than tracking which devices have seen it)
  if (cudaFuncSetAttribute(attention_forward_kernel<LONG>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)
    return GPT2L_ERR_CUDA;
  int err = GPT2L_OK;
  for (int first = 0, n; err == GPT2L_OK && (n = att_launch_tiles(T, first)) > 0; first += n) {
    attention_forward_kernel<LONG><<<dim3(NH, B, n), ATT_THREADS, smem, s>>>(out, lse, qkv, T, C, NH, (T - 1) / AT - first);
    err = LAUNCH_OK();
  }
  return err;
}
template <bool LONG>
static int attention_backward_launches(float *dqkv, const float *delta, const float *dout, const float *qkv, const float *lse,
                                       int B, int T, int C, int NH, cudaStream_t s) {
  constexpr int smem_q = 5 * ATILE * (int)sizeof(float), smem_kv = 6 * ATILE * (int)sizeof(float);
  auto dq = attention_backward_dq_kernel<LONG>;
  auto dkv = attention_backward_dkv_kernel<LONG>;
  if (cudaFuncSetAttribute(dq, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_q) != cudaSuccess ||
      cudaFuncSetAttribute(dkv, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_kv) != cudaSuccess)
    return GPT2L_ERR_CUDA;
  int err = GPT2L_OK;
  for (int first = 0, n; err == GPT2L_OK && (n = att_launch_tiles(T, first)) > 0; first += n) {
    const dim3 grid(NH, B, n);
    dq<<<grid, ATT_THREADS, smem_q, s>>>(dqkv, dout, qkv, lse, delta, T, C, NH, (T - 1) / AT - first);
    count_launch();
    dkv<<<grid, ATT_THREADS, smem_kv, s>>>(dqkv, dout, qkv, lse, delta, T, C, NH, first);
    err = LAUNCH_OK();
  }
  return err;
}
static bool att_long(int T) { return att_launch_tiles(T, 65535) > 0; }

int attention_forward(float *out, float *lse, const float *qkv, int B, int T, int C, int NH, cudaStream_t s) {
  if (C != NH * HS) return GPT2L_ERR_BAD_ARG;
  return att_long(T) ? attention_forward_launches<true>(out, lse, qkv, B, T, C, NH, s)
                     : attention_forward_launches<false>(out, lse, qkv, B, T, C, NH, s);
}
int attention_backward(float *dqkv, float *delta, const float *dout, const float *out, const float *qkv,
                       const float *lse, int B, int T, int C, int NH, cudaStream_t s) {
  if (C != NH * HS) return GPT2L_ERR_BAD_ARG;
  const int e = attention_row_dot(delta, dout, out, B, T, C, NH, s);
  if (e) return e;
  return att_long(T) ? attention_backward_launches<true>(dqkv, delta, dout, qkv, lse, B, T, C, NH, s)
                     : attention_backward_launches<false>(dqkv, delta, dout, qkv, lse, B, T, C, NH, s);
}
int adamw_update(float *p, float *m, float *v, const float *g, long long n, float lr, float b1, float b2, float eps,
                 float wd, int t, cudaStream_t s) {
  const float bc1 = 1.f - powf(b1, (float)t), bc2 = 1.f - powf(b2, (float)t);
  // all four buffers are offset alike from 256-byte aligned allocations, so p decides the alignment
  long long head = (long long)((16 - (reinterpret_cast<uintptr_t>(p) & 15)) & 15) / 4;
  if (head > n) head = n;
  const long long n4 = (n - head) / 4;
  const long long extra = n - 4 * n4;  // head + tail, at most 6
  return launched(launch_pdl(adamw_kernel, cdiv(n4 + extra, 256), 256, 0, s, p, m, v, g, n, head, n4, lr, b1, b2, eps, wd, bc1,
                             bc2));
}

}  // namespace g2l
