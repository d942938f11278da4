// CUDA-core kernels that sit beside the tcgen05 path:
//   * a strided fp32 GEMM for shapes TMA cannot address (row strides or pointers that are not
//     16-byte multiples, e.g. the unpadded vocabulary 50257) — still GPU code, never a CPU path;
//   * a deterministic column sum (the bias gradient when a fixed summation order is asked for).
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <atomic>

#include "linear_internal.h"
#include "ptx_sm100.cuh"

namespace g2l {

// ------------------------------------------------------------------------------------
// C[i][j] = sum_k A(i,k) * B(k,j) (+ bias[j]) in fp32 FMAs. Rows may start at any 4-byte boundary, so operands come in
// by 4-byte asynchronous copies (out-of-range elements zero-filled) into a ring of SIMT_STAGES slabs of 16 k, both
// stored k-major; 256 threads hold a BM x BN tile, (BM/16) x (BN/16) values each, and read the slabs with 16-byte
// shared-memory loads. A tile leaves through shared memory, so that its stores are whole lines although a
// thread's columns are four apart in the matrix.
//
// A cluster of S CTAs along z shares one output tile when there are too few tiles for the SMs: each takes a
// contiguous part of the reduction, and the partial tiles are added in the order of the parts through distributed
// shared memory. No workspace, no atomics, the same result on every run. Without a split an element is one
// chain of FMAs in ascending k.
//
// Bound by the FMA pipe's issue slots: two columns go into one packed FMA (fma.rn.f32x2, 64 multiply-adds per
// instruction, the same rounding), 50 TFLOP/s where single FMAs reached 44 (4096 x 768 x 8001). Against the
// 64 x 64 tiles of 4 x 4 single FMAs without a split that were here before, 256 x 768 x 50257: forward 917 -> 439 us,
// input gradient (12 tiles, 50257 deep) 8792 -> 717 us, weight gradient 980 -> 392 us.
// ------------------------------------------------------------------------------------
constexpr int SK = 16;  // k per slab
constexpr int SIMT_STAGES = 3;
constexpr int SIMT_THREADS = 256;
constexpr int SIMT_MAX_PARTS = 16;  // (clusters of more than 8 need the kernel's consent and a device that can place them)

template <int BMT, int BNT>
struct SimtCfg {
  static constexpr int LDA = BMT + 4, LDB = BNT + 4;  // slab rows: 16-byte aligned, four banks apart
  static constexpr int SLAB = SK * (LDA + LDB);       // floats of one stage
  static constexpr int RING_FLOATS = SIMT_STAGES * SLAB;
  static constexpr int TILE_FLOATS = BMT * LDB;  // the finished tile, over the ring
  static constexpr int SMEM = (RING_FLOATS > TILE_FLOATS ? RING_FLOATS : TILE_FLOATS) * 4;
};

__device__ __forceinline__ void cp_async4(uint32_t dst, const float *src, bool live) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(live ? 4 : 0) : "memory");
}

// One operand's slab: EXT rows (i or j) by SK k. KC: contiguous in k (a warp copies 8 k of 4 rows, which the row
// pitch of 4 mod 32 banks stores without conflict); else contiguous in the row index.
template <int EXT, bool KC>
struct SlabLoader {
  const float *base;  // any readable address, for copies that are out of range
  const float *src;   // this thread's first element of the next slab
  long long row_step, k_step;
  uint32_t dst0;
  int e0, n_ext, k, n_k;  // row index of the first element, its bound; k of the next slab, its bound
  static constexpr int N = EXT * SK / SIMT_THREADS;

  __device__ __forceinline__ void init(const float *p, long long e_stride, long long k_stride, int first, int ext, int k0,
                                       int k1, int tid) {
    const int lane = tid & 31, warp = tid >> 5;
    base = p;
    if (KC) {
      e0 = first + 4 * (warp >> 1) + (lane >> 3);
      k = k0 + (warp & 1) * 8 + (lane & 7);
      row_step = 16 * e_stride;
      dst0 = (uint32_t)((k - k0) * (EXT + 4) + (e0 - first)) * 4u;
    } else {
      e0 = first + tid % EXT;
      k = k0 + tid / EXT;
      row_step = (SIMT_THREADS / EXT) * k_stride;
      dst0 = (uint32_t)((tid / EXT) * (EXT + 4) + tid % EXT) * 4u;
    }
    k_step = SK * k_stride;
    n_ext = ext;
    n_k = k1;
    src = p + (long long)e0 * e_stride + (long long)k * k_stride;
  }
  __device__ __forceinline__ void load(uint32_t slab) {
#pragma unroll
    for (int i = 0; i < N; ++i) {
      bool live;
      uint32_t d;
      if (KC) {
        live = k < n_k && e0 + 16 * i < n_ext;
        d = slab + dst0 + 64u * i;
      } else {
        live = k + (SIMT_THREADS / EXT) * i < n_k && e0 < n_ext;
        d = slab + dst0 + (uint32_t)((SIMT_THREADS / EXT) * (EXT + 4) * 4) * i;
      }
      cp_async4(d, live ? src + i * row_step : base, live);
    }
    src += k_step;
    k += SK;
  }
};

template <int BMT, int BNT, bool A_KC, bool B_KC>
__global__ void __launch_bounds__(SIMT_THREADS, BNT == 128 ? 2 : 3)
gpt2_linear_simt_kernel(float *__restrict__ c, const float *__restrict__ a, const float *__restrict__ b,
                        const float *__restrict__ bias, int Mc, int Nc, int Kc, long long ai, long long ak,
                        long long bk, long long bj, long long ldc, int k_per_part, int tiles_n) {
  using G = SimtCfg<BMT, BNT>;
  extern __shared__ __align__(16) float sm[];
  constexpr int TM = BMT / 16, TN = BNT / 16;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int i0 = (int)(blockIdx.x / tiles_n) * BMT, j0 = (int)(blockIdx.x % tiles_n) * BNT;
  const int part = blockIdx.z, parts = gridDim.z;
  const int k0 = part * k_per_part, k1 = min(Kc, k0 + k_per_part);

  SlabLoader<BMT, A_KC> la;
  SlabLoader<BNT, B_KC> lb;
  la.init(a, ai, ak, i0, Mc, k0, k1, tid);
  lb.init(b, bj, bk, j0, Nc, k0, k1, tid);
  const uint32_t ring = (uint32_t)__cvta_generic_to_shared(sm);
  const int n_slab = (k1 - k0 + SK - 1) / SK;
  constexpr uint32_t SLAB_BYTES = G::SLAB * 4u, B_OFF = SK * G::LDA * 4u;
#pragma unroll
  for (int s = 0; s < SIMT_STAGES - 1; ++s) {
    if (s < n_slab) {
      la.load(ring + s * SLAB_BYTES);
      lb.load(ring + s * SLAB_BYTES + B_OFF);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }

  // warps 4 x 2 over the tile, lanes 4 x 8 over a warp's part; a thread's rows and columns come in groups of four
  const int r_lane = (warp >> 1) * (BMT / 4) + (lane >> 3) * 4;
  const int c_lane = (warp & 1) * (BNT / 2) + (lane & 7) * 4;
  unsigned long long acc[TM][TN / 2] = {};  // two neighbouring columns per register pair
  int stage = 0;
  for (int s = 0; s < n_slab; ++s) {
    asm volatile("cp.async.wait_group %0;" ::"n"(SIMT_STAGES - 2) : "memory");
    __syncthreads();  // slab s has landed for everyone, and everyone is done with slab s - 1
    const int next = stage == 0 ? SIMT_STAGES - 1 : stage - 1;
    if (s + SIMT_STAGES - 1 < n_slab) {
      la.load(ring + next * SLAB_BYTES);
      lb.load(ring + next * SLAB_BYTES + B_OFF);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    const float *sa = sm + stage * G::SLAB + r_lane;
    const float *sb = sm + stage * G::SLAB + SK * G::LDA + c_lane;
#pragma unroll
    for (int k = 0; k < SK; ++k) {
      unsigned long long av[TM], bv[TN / 2];
#pragma unroll
      for (int h = 0; h < TM / 4; ++h) {
        const float4 v = *reinterpret_cast<const float4 *>(sa + k * G::LDA + 16 * h);
        av[4 * h] = ptx::both(v.x); av[4 * h + 1] = ptx::both(v.y); av[4 * h + 2] = ptx::both(v.z); av[4 * h + 3] = ptx::both(v.w);
      }
#pragma unroll
      for (int h = 0; h < TN / 4; ++h) {
        const ulonglong2 v = *reinterpret_cast<const ulonglong2 *>(sb + k * G::LDB + 32 * h);
        bv[2 * h] = v.x; bv[2 * h + 1] = v.y;
      }
#pragma unroll
      for (int u = 0; u < TM; ++u)
#pragma unroll
        for (int v = 0; v < TN / 2; ++v) acc[u][v] = ptx::fma2(av[u], bv[v], acc[u][v]);
    }
    stage = stage + 1 == SIMT_STAGES ? 0 : stage + 1;
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
#pragma unroll
  for (int u = 0; u < TM; ++u)
#pragma unroll
    for (int h = 0; h < TN / 4; ++h)
      *reinterpret_cast<ulonglong2 *>(sm + (r_lane + 16 * (u >> 2) + (u & 3)) * G::LDB + c_lane + 32 * h) =
          make_ulonglong2(acc[u][2 * h], acc[u][2 * h + 1]);
  if (parts > 1) ptx::cluster_sync_all();
  else __syncthreads();
  // rows of the tile this CTA stores; a warp takes a row at a time
  const int rows = BMT / parts;
  for (int rr = warp; rr < rows; rr += SIMT_THREADS / 32) {
    const int rl = part * rows + rr, gi = i0 + rl;
    if (gi >= Mc) continue;
#pragma unroll
    for (int cc = 0; cc < BNT; cc += 32) {
      const int gj = j0 + cc + lane;
      float v = 0.f;
      if (parts == 1) {
        v = sm[rl * G::LDB + cc + lane];
      } else {
        const uint32_t at = ring + (uint32_t)(rl * G::LDB + cc + lane) * 4u;
        for (int p = 0; p < parts; ++p) {
          float w;
          asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(w) : "r"(ptx::mapa_cluster(at, (uint32_t)p)));
          v = p == 0 ? w : v + w;
        }
      }
      if (gj < Nc) c[gi * ldc + gj] = v + (bias ? bias[gj] : 0.f);
    }
  }
  if (parts > 1) ptx::cluster_sync_all();  // nobody's shared memory goes away while it is read
}

// out[j] = sum_i x[i][j], fixed order: a block owns 32 columns of one part of the rows, 8 row lanes add every eighth row,
// then a fixed tree combines them; the parts (a cluster along z) are added in order through distributed shared
// memory. Bound by the latency of the row loads, hence eight in flight per thread and the split: without either a
// thread of a 768-wide sum over 8192 rows made 1024 dependent trips to memory.
__global__ void __launch_bounds__(256)
gpt2_linear_colsum_kernel(float *__restrict__ out, const float *__restrict__ x, int rows, int cols, int rows_per_part) {
  __shared__ float part[8][33];
  __shared__ float total[32];
  const int cx = threadIdx.x % 32, ry = threadIdx.x / 32;
  const int j = blockIdx.x * 32 + cx;
  const int r0 = blockIdx.z * rows_per_part, r1 = min(rows, r0 + rows_per_part);
  float s = 0.f;
  if (j < cols) {
    int i = r0 + ry;
    for (; i + 56 < r1; i += 64) {
      float v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = x[(long long)(i + 8 * u) * cols + j];
#pragma unroll
      for (int u = 0; u < 8; ++u) s += v[u];
    }
    for (; i < r1; i += 8) s += x[(long long)i * cols + j];
  }
  part[ry][cx] = s;
  __syncthreads();
  if (ry == 0) {
    float t = 0.f;
    for (int r = 0; r < 8; ++r) t += part[r][cx];
    total[cx] = t;
  }
  if (gridDim.z > 1) ptx::cluster_sync_all();
  else __syncthreads();
  if (blockIdx.z == 0 && ry == 0 && j < cols) {
    float t = total[cx];
    const uint32_t at = (uint32_t)__cvta_generic_to_shared(&total[cx]);
    for (unsigned p = 1; p < gridDim.z; ++p) {
      float w;
      asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(w) : "r"(ptx::mapa_cluster(at, p)));
      t += w;
    }
    out[j] = t;
  }
  if (gridDim.z > 1) ptx::cluster_sync_all();
}

// dst[c][r] = src[r][c] for src[rows][cols]; 32 x 32 tiles through shared memory, both sides coalesced.
__global__ void __launch_bounds__(256)
gpt2_linear_transpose_kernel(float *__restrict__ dst, const float *__restrict__ src, int rows, int cols) {
  ptx::pdl_trigger();
  ptx::pdl_wait();
  __shared__ float tile[32][33];
  const int tx = threadIdx.x % 32, ty = threadIdx.x / 32;
  const int c0 = blockIdx.x * 32, r0 = blockIdx.y * 32;
  for (int i = ty; i < 32; i += 8) {
    const int r = r0 + i, c = c0 + tx;
    tile[i][tx] = (r < rows && c < cols) ? src[(long long)r * cols + c] : 0.f;
  }
  __syncthreads();
  for (int i = ty; i < 32; i += 8) {
    const int c = c0 + i, r = r0 + tx;
    if (c < cols && r < rows) dst[(long long)c * rows + r] = tile[tx][i];
  }
}

// What a split or a bias gradient adds into: a[0 .. 4 n4) and b[0 .. nb). One launch that may overlap the kernel before it
// (a memset may not, and stood between the launches of a chain twice per call).
__global__ void __launch_bounds__(256)
gpt2_linear_zero_kernel(float4 *a, long long n4, float *b, int nb) {
  ptx::pdl_trigger();
  ptx::pdl_wait();
  const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
  if (i < n4) a[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  else if (i - n4 < nb) b[i - n4] = 0.f;
}

int launch_zero(float *a, long long n, float *b, int nb, cudaStream_t stream) {
  const cudaError_t e = launch_pdl(gpt2_linear_zero_kernel, dim3((unsigned)((n / 4 + nb + 255) / 256)), 256, 0, stream,
                                   reinterpret_cast<float4 *>(a), n / 4, b, nb);
  count_launch();
  return e == cudaSuccess ? GPT2L_OK : GPT2L_ERR_CUDA;
}

int launch_transpose(float *dst, const float *src, int rows, int cols, cudaStream_t stream) {
  dim3 grid((cols + 31) / 32, (rows + 31) / 32);
  const cudaError_t e = launch_pdl(gpt2_linear_transpose_kernel, grid, 256, 0, stream, dst, src, rows, cols);
  count_launch();
  return e == cudaSuccess ? GPT2L_OK : GPT2L_ERR_CUDA;
}

// The tile and the split whose busiest SM has the least to do. Smaller tiles cost more per product (shared-memory
// reads per FMA), a CTA that has its SM to itself reaches 73 % of what two reach together (23.7 against 50 TFLOP/s x
// 96 / 148 SMs), and a part pays for filling its ring and for the exchange of the partial tiles, counted as
// SIMT_FIXED_K more k. `max_parts`: the largest cluster the device can place.
SimtPlan simt_plan(int Mc, int Nc, int Kc, int sms, int max_parts) {
  constexpr double SIMT_FIXED_K = 48.0;
  static const struct { int bm, bn; double per_product; } tile[3] = {{128, 128, 1.0}, {128, 64, 1.2}, {64, 64, 1.6}};
  SimtPlan best = {128, 128, 1, 0};
  double best_cost = 1e300;
  for (const auto &t : tile) {
    const double tiles = (double)((Mc + t.bm - 1) / t.bm) * ((Nc + t.bn - 1) / t.bn);
    for (int parts = 1; parts <= max_parts; parts *= 2) {
      const int per = ((Kc + parts - 1) / parts + SK - 1) / SK * SK;
      if (parts > 1 && (long long)per * (parts - 1) >= Kc) break;  // an empty part
      const double ctas_per_sm = ceil(tiles * parts / sms);
      const double fill = ctas_per_sm < 2.0 ? 1.37 : 1.0;
      const double cost = ctas_per_sm * fill * (per + SIMT_FIXED_K * (parts > 1 ? 2.0 : 1.0)) * t.bm * t.bn * t.per_product;
      if (cost < best_cost) {
        best_cost = cost;
        best = {t.bm, t.bn, parts, per};
      }
    }
  }
  return best;
}

namespace {

using SimtKernel = void (*)(float *, const float *, const float *, const float *, int, int, int, long long, long long, long long,
                            long long, long long, int, int);

cudaLaunchConfig_t simt_config(cudaLaunchAttribute *attr, long long tiles, int parts, size_t smem, cudaStream_t stream) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)tiles, 1, (unsigned)parts);
  cfg.blockDim = dim3(SIMT_THREADS, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = (unsigned)parts;
  cfg.attrs = attr;
  cfg.numAttrs = parts > 1 ? 1 : 0;
  return cfg;
}

int simt_attributes(SimtKernel kernel, int smem) {
  // (per device and cheap: set every time rather than tracking which devices have seen it)
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) == cudaSuccess &&
                 cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess
             ? GPT2L_OK
             : GPT2L_ERR_CUDA;
}

// The largest cluster of the 128 x 128 kernel, the one with the most shared memory, that the current device can place (a
// partition of a GPU may not hold 16 CTAs side by side); asked once per device.
int simt_max_parts(int dev) {
  constexpr int DEVICES = 16;
  static std::atomic<int> known[DEVICES];
  const bool keep = dev >= 0 && dev < DEVICES;
  if (keep && known[dev].load(std::memory_order_relaxed) > 0) return known[dev].load(std::memory_order_relaxed);
  constexpr int smem = SimtCfg<128, 128>::SMEM;
  SimtKernel kernel = gpt2_linear_simt_kernel<128, 128, true, true>;
  int parts = simt_attributes(kernel, smem) == GPT2L_OK ? SIMT_MAX_PARTS : 1;
  for (; parts > 1; parts /= 2) {
    cudaLaunchAttribute attr[1];
    const cudaLaunchConfig_t cfg = simt_config(attr, 1, parts, smem, nullptr);
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) == cudaSuccess && clusters > 0) break;
    (void)cudaGetLastError();
  }
  if (keep) known[dev].store(parts, std::memory_order_relaxed);
  return parts;
}

template <int BMT, int BNT>
int simt_launch(const SimtPlan &pl, float *c, const float *a, const float *b, const float *bias, int Mc, int Nc, int Kc,
                long long ai, long long ak, long long bk, long long bj, cudaStream_t stream) {
  using G = SimtCfg<BMT, BNT>;
  const long long tiles_n = (Nc + BNT - 1) / BNT, tiles = tiles_n * ((Mc + BMT - 1) / BMT);
  if (tiles > 0x7fffffffll) return GPT2L_ERR_TOO_LARGE;
  const SimtKernel kernel = ak == 1 ? (bj == 1 ? gpt2_linear_simt_kernel<BMT, BNT, true, false> : gpt2_linear_simt_kernel<BMT, BNT, true, true>)
                        : gpt2_linear_simt_kernel<BMT, BNT, false, false>;
  if (simt_attributes(kernel, G::SMEM)) return GPT2L_ERR_CUDA;
  cudaLaunchAttribute attr[1];
  const cudaLaunchConfig_t cfg = simt_config(attr, tiles, pl.parts, G::SMEM, stream);
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, c, a, b, bias, Mc, Nc, Kc, ai, ak, bk, bj, (long long)Nc,
                                           pl.k_per_part, (int)tiles_n);
  count_launch();
  if (e != cudaSuccess) {
    (void)cudaGetLastError();
    return GPT2L_ERR_CUDA;
  }
  return GPT2L_OK;
}

}  // namespace

int launch_simt(const GemmDesc &d, cudaStream_t stream) {
  int Mc, Nc, Kc;
  long long ai, ak, bk, bj;
  const float *bias = nullptr;
  switch (d.kind) {
    case GPT2L_OP_FORWARD:
      Mc = d.M; Nc = d.N; Kc = d.K; ai = d.K; ak = 1; bk = d.N; bj = 1; bias = d.bias; break;
    case GPT2L_OP_BACKWARD_INPUT:
      Mc = d.M; Nc = d.K; Kc = d.N; ai = d.N; ak = 1; bk = 1; bj = d.N; break;
    case GPT2L_OP_BACKWARD_WEIGHT:
      Mc = d.K; Nc = d.N; Kc = d.M; ai = 1; ak = d.K; bk = d.N; bj = 1; break;
    default:
      return GPT2L_ERR_BAD_ARG;
  }
  int dev = -1, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0)
    sms = 148;
  const SimtPlan pl = simt_plan(Mc, Nc, Kc, sms, simt_max_parts(dev));
  int e;
  if (pl.bn == 128) e = simt_launch<128, 128>(pl, d.out, d.a, d.b, bias, Mc, Nc, Kc, ai, ak, bk, bj, stream);
  else if (pl.bm == 128) e = simt_launch<128, 64>(pl, d.out, d.a, d.b, bias, Mc, Nc, Kc, ai, ak, bk, bj, stream);
  else e = simt_launch<64, 64>(pl, d.out, d.a, d.b, bias, Mc, Nc, Kc, ai, ak, bk, bj, stream);
  if (e) return e;
  if (d.kind == GPT2L_OP_BACKWARD_WEIGHT && d.out_bias) return launch_colsum(d.out_bias, d.b, d.M, d.N, stream);
  return GPT2L_OK;
}

int launch_colsum(float *out, const float *x, int rows, int cols, cudaStream_t stream) {
  int parts = 1;
  while (parts < 8 && rows > 128 * parts) parts *= 2;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  cfg.gridDim = dim3((unsigned)((cols + 31) / 32), 1, (unsigned)parts);
  cfg.blockDim = dim3(256, 1, 1);
  cfg.stream = stream;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = (unsigned)parts;
  cfg.attrs = attr;
  cfg.numAttrs = parts > 1 ? 1 : 0;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, gpt2_linear_colsum_kernel, out, x, rows, cols, (rows + parts - 1) / parts);
  count_launch();
  if (e != cudaSuccess) {
    (void)cudaGetLastError();
    return GPT2L_ERR_CUDA;
  }
  return GPT2L_OK;
}

}  // namespace g2l
