// C ABI of libgpt2_linear.so: device context, the three linear-layer calls (device and
// host-buffer flavours). Declarations and the reference interfaces they replace are in
// include/gpt2_linear.h.
#include <cuda_runtime.h>
#include <stdio.h>
#include <string.h>

#include <mutex>
#include <unordered_map>
#include <vector>

#include "linear_internal.h"

namespace g2l {

constexpr int MAX_DEVICES = 16;
static DeviceCtx g_ctx[MAX_DEVICES];
static std::mutex g_mu;        // context table and the shared split-K workspace
static std::mutex g_stage_mu;  // host-call staging buffers (held for a whole *_host call)

// ---------------------------------------------------------------------------------------
// Pipelined host-buffer calls: three streams (copy in, compute, copy out) and two sets of staging
// buffers, so that the host->device copies of call n+1 run while call n computes and copies its
// results out (PCIe is full duplex). A set is reused by every second call, behind the event that
// marks its previous results as copied out.
// ---------------------------------------------------------------------------------------
struct HostPipe {
  cudaStream_t s_in = nullptr, s_run = nullptr, s_out = nullptr;
  struct Set {
    float *buf[4] = {nullptr, nullptr, nullptr, nullptr};
    size_t bytes[4] = {0, 0, 0, 0};
    cudaEvent_t ev_in = nullptr, ev_run = nullptr, ev_free = nullptr;
    bool used = false;
  } set[2];
  unsigned long long calls = 0;
  // Inputs uploaded since the last synchronise, by host address and size. The contract of the pipelined
  // calls forbids changing an input before the synchronise, so a buffer passed to several calls (the
  // weight to forward and backward_input, the activations to forward and backward_weight, ...) crosses
  // PCIe once. The device copies go back to `pool` at the synchronise and are reused by later windows.
  struct Input {
    const void *host;
    size_t bytes;
    float *dev;
    size_t cap;
  };
  std::vector<Input> inputs;
  std::vector<Input> pool;  // host / bytes unused
  unsigned long long uploaded_bytes = 0, reused_bytes = 0;
};

static void destroy_pipe(HostPipe *p) {
  if (!p) return;
  for (auto &i : p->inputs) cudaFree(i.dev);
  for (auto &i : p->pool) cudaFree(i.dev);
  for (auto &s : p->set) {
    for (float *b : s.buf)
      if (b) cudaFree(b);
    if (s.ev_in) cudaEventDestroy(s.ev_in);
    if (s.ev_run) cudaEventDestroy(s.ev_run);
    if (s.ev_free) cudaEventDestroy(s.ev_free);
  }
  if (p->s_in) cudaStreamDestroy(p->s_in);
  if (p->s_run) cudaStreamDestroy(p->s_run);
  if (p->s_out) cudaStreamDestroy(p->s_out);
  delete p;
}

static HostPipe *get_pipe(DeviceCtx *ctx) {
  if (ctx->pipe) return ctx->pipe;
  HostPipe *p = new HostPipe();
  bool ok = cudaStreamCreateWithFlags(&p->s_in, cudaStreamNonBlocking) == cudaSuccess &&
            cudaStreamCreateWithFlags(&p->s_run, cudaStreamNonBlocking) == cudaSuccess &&
            cudaStreamCreateWithFlags(&p->s_out, cudaStreamNonBlocking) == cudaSuccess;
  for (auto &s : p->set)
    ok = ok && cudaEventCreateWithFlags(&s.ev_in, cudaEventDisableTiming) == cudaSuccess &&
         cudaEventCreateWithFlags(&s.ev_run, cudaEventDisableTiming) == cudaSuccess &&
         cudaEventCreateWithFlags(&s.ev_free, cudaEventDisableTiming) == cudaSuccess;
  if (!ok) {
    destroy_pipe(p);
    return nullptr;
  }
  ctx->pipe = p;
  return p;
}
constexpr size_t SEM_COUNT = 1u << 20;  // split-K arrival counters (one per output tile and lane quarter)

DeviceCtx *ctx_current(int *err) {
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= MAX_DEVICES) {
    (void)cudaGetLastError();
    *err = GPT2L_ERR_NO_DEVICE;
    return nullptr;
  }
  if (!g_ctx[dev].ready) {
    *err = GPT2L_ERR_NOT_INIT;
    return nullptr;
  }
  *err = GPT2L_OK;
  return &g_ctx[dev];
}

static int ensure_bytes(float **buf, size_t *have, size_t need) {
  if (need <= *have) return GPT2L_OK;
  if (*buf) cudaFree(*buf);
  *buf = nullptr;
  *have = 0;
  // grow in 64 MiB steps so that repeated slightly larger requests do not reallocate
  size_t want = (need + (64u << 20) - 1) / (64u << 20) * (64u << 20);
  if (cudaMalloc(reinterpret_cast<void **>(buf), want) != cudaSuccess) {
    (void)cudaGetLastError();
    return GPT2L_ERR_CUDA;
  }
  *have = want;
  return GPT2L_OK;
}

// Built ops (tiling, instruction descriptor and the three or four tensor maps) keyed by everything that
// went into them: a training loop makes the same calls on the same buffers every step, so the tensor maps
// are encoded once per (pointers, shape, options) instead of once per call.
struct OpKey {
  alignas(16) unsigned char bytes[sizeof(GemmDesc)];
  bool operator==(const OpKey &o) const { return memcmp(bytes, o.bytes, sizeof(bytes)) == 0; }
};
struct OpKeyHash {
  size_t operator()(const OpKey &k) const {
    size_t h = 1469598103934665603ull;  // FNV-1a
    for (unsigned char b : k.bytes) h = (h ^ b) * 1099511628211ull;
    return h;
  }
};
static std::unordered_map<OpKey, GemmOp, OpKeyHash> g_op_cache[MAX_DEVICES];
static std::mutex g_cache_mu;
constexpr size_t OP_CACHE_MAX = 4096;

static OpKey key_of(const GemmDesc &d) {
  OpKey k;
  memset(k.bytes, 0, sizeof(k.bytes));
  GemmDesc *dst = reinterpret_cast<GemmDesc *>(k.bytes);  // field by field: padding bytes stay zero
  dst->kind = d.kind; dst->M = d.M; dst->K = d.K; dst->N = d.N;
  dst->xent_stats = d.xent_stats; dst->xent_vocab = d.xent_vocab;
  dst->out = d.out; dst->out_bias = d.out_bias; dst->a = d.a; dst->b = d.b; dst->bias = d.bias;
  dst->opts.mode = d.opts.mode; dst->opts.flags = d.opts.flags; dst->opts.split_k = d.opts.split_k;
  dst->opts.deterministic = d.opts.deterministic; dst->opts.out2 = d.opts.out2; dst->opts.force_simt = d.opts.force_simt;
  dst->opts.cta_pair = d.opts.cta_pair; dst->opts.aux = d.opts.aux; dst->opts.aux_op = d.opts.aux_op;
  dst->opts.xent_lse = d.opts.xent_lse; dst->opts.xent_targets = d.opts.xent_targets;
  dst->opts.xent_vocab = d.opts.xent_vocab; dst->opts.xent_scale = d.opts.xent_scale;
  return k;
}

static int build_op_cached(DeviceCtx *ctx, const GemmDesc &d, GemmOp *op) {
  const OpKey k = key_of(d);
  {
    std::lock_guard<std::mutex> lk(g_cache_mu);
    auto &cache = g_op_cache[ctx->device];
    auto it = cache.find(k);
    if (it != cache.end()) {
      *op = it->second;
      return GPT2L_OK;
    }
  }
  int e = build_op(d, ctx->num_sms, op);
  if (e) return e;
  std::lock_guard<std::mutex> lk(g_cache_mu);
  auto &cache = g_op_cache[ctx->device];
  if (cache.size() >= OP_CACHE_MAX) cache.clear();
  cache.emplace(k, *op);
  return GPT2L_OK;
}

static int run_gemm(GemmDesc &d, cudaStream_t st) {
  int err;
  DeviceCtx *ctx = ctx_current(&err);
  if (!ctx) return err;
  // a kernel of an earlier call gave up on a wait: nothing more is launched (it would unwind at its
  // first wait anyway) until gpt2_linear_last_status() has read and cleared the record
  if (*reinterpret_cast<volatile int *>(ctx->h_flag) != 0) return GPT2L_DEV_TIMEOUT;
  if (d.M <= 0 || d.K <= 0 || d.N <= 0 || !d.out || !d.a || !d.b) return GPT2L_ERR_BAD_ARG;
  if (d.opts.mode != GPT2L_MODE_TF32 && d.opts.mode != GPT2L_MODE_TF32X3) return GPT2L_ERR_BAD_ARG;
  if ((long long)d.M * d.N >= (1ll << 40) || (long long)d.M * d.K >= (1ll << 40)) return GPT2L_ERR_TOO_LARGE;
  if (d.opts.force_simt || !tma_eligible(d)) {
    if ((d.opts.flags & GPT2L_EPI_GELU_DUAL) || d.opts.aux_op || d.opts.xent_lse || d.xent_stats) return GPT2L_ERR_BAD_ARG;
    return launch_simt(d, st);
  }
  if (d.opts.xent_lse && (d.kind == GPT2L_OP_FORWARD || d.opts.deterministic)) return GPT2L_ERR_BAD_ARG;
  // bias gradient: fused into the kernel (column sums of the staged g_out blocks) unless a
  // fixed summation order is requested, which the stand-alone column-sum kernel provides.
  float *fused_bias = d.out_bias;
  if (d.kind == GPT2L_OP_BACKWARD_WEIGHT && d.out_bias && d.opts.deterministic) {
    fused_bias = nullptr;
  }
  GemmDesc dd = d;
  dd.out_bias = fused_bias;
  dd.opts.cta_pair = choose_cta_pair(d, ctx->num_sms, ctx->max_pairs);
  GemmOp op;
  // Wide weight gradients (lm_head: N = 50304 against K = 768): the tensor core reads an MN-major A
  // operand about 20 % slower than a K-major one, and here A = in^T is tiny next to the GEMM. So
  // `in` is transposed once into scratch (2 * M * K * 4 bytes of traffic, ~1 % of the GEMM's time) and
  // the product runs in the forward form g_w[K][N] = inT[K][M] . g_out[M][N] with a K-major A.
  bool transposed_a = false;
  if (d.kind == GPT2L_OP_BACKWARD_WEIGHT && d.N >= 8192 && d.N >= 8 * d.K && (d.M & 3) == 0 && d.M > 1) {
    {
      std::lock_guard<std::mutex> lk(g_mu);
      err = ensure_bytes(&ctx->xt, &ctx->xt_bytes, (size_t)d.M * d.K * sizeof(float));
    }
    if (err) return err;
    err = launch_transpose(ctx->xt, d.a, d.M, d.K, st);
    if (err) return err;
    dd.kind = GPT2L_OP_FORWARD;
    dd.M = d.K;  // output rows
    dd.K = d.M;  // reduction
    dd.a = ctx->xt;
    dd.b = d.b;
    dd.bias = nullptr;
    dd.opts.flags = 0;
    transposed_a = true;
  }
  err = build_op_cached(ctx, dd, &op);
  if (err) return err;
  if (transposed_a) {  // the B operand is still g_out: its column sums are g_b
    op.colsum = fused_bias;
    op.colsum_spread = fused_bias ? 1 : 0;
    op.cs_src = d.b;
  }
  if (op.splits > 1 && !op.atomic_out) {
    std::lock_guard<std::mutex> lk(g_mu);
    if ((size_t)op.tiles_m * op.tiles_n * 4 > ctx->ws_sem_count) return GPT2L_ERR_TOO_LARGE;
    err = ensure_bytes(&ctx->ws, &ctx->ws_bytes, op_workspace_bytes(op));
    if (err) return err;
    op.ws = ctx->ws;
    op.ws_sem = ctx->ws_sem;
  }
  // (Nc is a multiple of four and C 16-byte aligned: tma_eligible)
  const bool zero_c = op.splits > 1 && op.atomic_out, zero_cs = op.colsum && (op.splits > 1 || op.colsum_spread);
  if (zero_c || zero_cs) {
    err = launch_zero(op.C, zero_c ? (long long)op.Mc * op.Nc : 0, op.colsum, zero_cs ? op.Nc : 0, st);
    if (err) return err;
  }
  err = launch_single(ctx, op, st);
  if (err) return err;
  if (d.kind == GPT2L_OP_BACKWARD_WEIGHT && d.out_bias && !fused_bias)
    return launch_colsum(d.out_bias, d.b, d.M, d.N, st);
  return GPT2L_OK;
}

static gpt2_linear_opts opts_or_default(const gpt2_linear_opts *o) {
  gpt2_linear_opts r;
  memset(&r, 0, sizeof(r));
  if (o) r = *o;
  return r;
}

static int read_status(DeviceCtx *ctx, Status *out, bool clear) {
  if (cudaMemcpy(ctx->h_status, ctx->d_status, sizeof(Status), cudaMemcpyDeviceToHost) != cudaSuccess)
    return GPT2L_ERR_CUDA;
  *out = *ctx->h_status;
  // the flag alone is set when the launch that gave up kept its record elsewhere (a schedule's own status)
  const int flag = *reinterpret_cast<volatile int *>(ctx->h_flag);
  if (out->status == 0 && flag != 0) out->status = flag;
  if (clear && out->status != 0) {
    cudaMemset(ctx->d_status, 0, sizeof(Status));
    *reinterpret_cast<volatile int *>(ctx->h_flag) = 0;
  }
  return GPT2L_OK;
}

}  // namespace g2l

using namespace g2l;

extern "C" {

int gpt2_linear_version(void) { return 100; }

long long gpt2_linear_launch_count(void) { return launch_count_value(); }

int gpt2_linear_init(int device) {
  int n = 0;
  if (cudaGetDeviceCount(&n) != cudaSuccess || n <= 0) {
    (void)cudaGetLastError();
    return GPT2L_ERR_NO_DEVICE;
  }
  if (device < 0 || device >= n || device >= MAX_DEVICES) return GPT2L_ERR_BAD_ARG;
  if (cudaSetDevice(device) != cudaSuccess) return GPT2L_ERR_CUDA;
  std::lock_guard<std::mutex> lk(g_mu);
  DeviceCtx &c = g_ctx[device];
  if (c.ready) return GPT2L_OK;
  cudaDeviceProp prop;
  if (cudaGetDeviceProperties(&prop, device) != cudaSuccess) return GPT2L_ERR_CUDA;
  if (prop.major != 10) return GPT2L_ERR_NO_DEVICE;  // tcgen05 / TMEM exist on sm_100 only
  if (!get_encode_fn()) return GPT2L_ERR_CUDA;
  int e = set_kernel_attributes();
  if (e) return e;
  e = pair_set_kernel_attributes();
  if (e) return e;
  c.device = device;
  c.num_sms = prop.multiProcessorCount;
  c.max_pairs = pair_max_pairs(c.num_sms);
  if (cudaMalloc(reinterpret_cast<void **>(&c.d_status), sizeof(Status)) != cudaSuccess) return GPT2L_ERR_CUDA;
  cudaMemset(c.d_status, 0, sizeof(Status));
  if (cudaMallocHost(reinterpret_cast<void **>(&c.h_status), sizeof(Status)) != cudaSuccess) return GPT2L_ERR_CUDA;
  if (cudaHostAlloc(reinterpret_cast<void **>(&c.h_flag), sizeof(int), cudaHostAllocMapped) != cudaSuccess ||
      cudaHostGetDevicePointer(reinterpret_cast<void **>(&c.d_flag), c.h_flag, 0) != cudaSuccess)
    return GPT2L_ERR_CUDA;
  *c.h_flag = 0;
  if (cudaMalloc(reinterpret_cast<void **>(&c.ws_sem), SEM_COUNT * sizeof(unsigned)) != cudaSuccess)
    return GPT2L_ERR_CUDA;
  cudaMemset(c.ws_sem, 0, SEM_COUNT * sizeof(unsigned));
  c.ws_sem_count = SEM_COUNT;
  c.ready = true;
  return GPT2L_OK;
}

void gpt2_linear_shutdown(void) {
  std::lock_guard<std::mutex> lk(g_mu);
  int cur = -1;
  cudaGetDevice(&cur);
  for (int d = 0; d < MAX_DEVICES; ++d) {
    DeviceCtx &c = g_ctx[d];
    if (!c.ready) continue;
    cudaSetDevice(d);
    cudaDeviceSynchronize();
    cudaFree(c.d_status);
    cudaFreeHost(c.h_status);
    cudaFreeHost(c.h_flag);
    cudaFree(c.ws_sem);
    if (c.ws) cudaFree(c.ws);
    if (c.xt) cudaFree(c.xt);
    if (c.xstats) cudaFree(c.xstats);
    for (int i = 0; i < 4; ++i)
      if (c.stage[i]) cudaFree(c.stage[i]);
    destroy_pipe(c.pipe);
    {
      std::lock_guard<std::mutex> lk2(g_cache_mu);
      g_op_cache[d].clear();
    }
    c = DeviceCtx();
  }
  if (cur >= 0) cudaSetDevice(cur);
  (void)cudaGetLastError();
}

int gpt2_linear_last_status(int out[6]) {
  int err;
  DeviceCtx *ctx = ctx_current(&err);
  if (!ctx) return err;
  Status s;
  err = read_status(ctx, &s, true);
  if (err) return err;
  if (out) {
    out[0] = s.status; out[1] = s.op; out[2] = s.counter; out[3] = s.seen; out[4] = s.expected; out[5] = s.where;
  }
  return s.status;
}

int gpt2_linear_forward(float *out, const float *in, const float *w, const float *b, int B, int S, int K, int N,
                        const gpt2_linear_opts *opts, gpt2l_stream_t stream) {
  if (B <= 0 || S <= 0) return GPT2L_ERR_BAD_ARG;
  if ((long long)B * S > 0x7fffffffll) return GPT2L_ERR_TOO_LARGE;
  GemmDesc d;
  d.kind = GPT2L_OP_FORWARD;
  d.M = B * S; d.K = K; d.N = N;
  d.out = out; d.out_bias = nullptr; d.a = in; d.b = w; d.bias = b;
  d.opts = opts_or_default(opts);
  if (d.opts.xent_lse) return GPT2L_ERR_BAD_ARG;  // the fused cross-entropy has its own forward entry point
  return run_gemm(d, static_cast<cudaStream_t>(stream));
}

int gpt2_linear_forward_xent(float *logits, float *losses, float *lse, const float *in, const float *w,
                             const int *targets, int B, int S, int K, int N, int V, const gpt2_linear_opts *opts,
                             gpt2l_stream_t stream) {
  if (B <= 0 || S <= 0 || !losses || !lse || !targets || V <= 0 || V > N) return GPT2L_ERR_BAD_ARG;
  if ((long long)B * S > 0x7fffffffll) return GPT2L_ERR_TOO_LARGE;
  int err;
  DeviceCtx *ctx = ctx_current(&err);
  if (!ctx) return err;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  GemmDesc d;
  d.kind = GPT2L_OP_FORWARD;
  d.M = B * S; d.K = K; d.N = N;
  d.out = logits; d.out_bias = nullptr; d.a = in; d.b = w; d.bias = nullptr;
  d.opts = opts_or_default(opts);
  if (d.opts.flags || d.opts.aux_op || d.opts.xent_lse || d.opts.force_simt || !logits || !in || !w || K <= 0 || N <= 0 ||
      !tma_eligible(d))
    return GPT2L_ERR_BAD_ARG;
  // the statistics buffer's size and row stride follow the tiling, so the op that will be launched is planned first,
  // with everything that decides its tiling settled
  GemmOp probe;
  d.xent_stats = reinterpret_cast<float *>(16);  // any non-null value: plan_op only looks at shapes
  d.xent_vocab = V;
  d.opts.cta_pair = choose_cta_pair(d, ctx->num_sms, ctx->max_pairs);
  err = plan_op(d, ctx->num_sms, &probe);
  if (err) return err;
  {
    std::lock_guard<std::mutex> lk(g_mu);
    err = ensure_bytes(&ctx->xstats, &ctx->xstats_bytes, xent_stats_floats(probe) * sizeof(float));
  }
  if (err) return err;
  d.xent_stats = ctx->xstats;
  err = run_gemm(d, st);
  if (err) return err;
  return launch_xent_combine(lse, losses, ctx->xstats, probe.xent_stride, logits, N, targets, d.M, st);
}

int gpt2_linear_backward_input(float *g_in, const float *g_out, const float *w, int B, int S, int K, int N,
                               const gpt2_linear_opts *opts, gpt2l_stream_t stream) {
  if (B <= 0 || S <= 0) return GPT2L_ERR_BAD_ARG;
  if ((long long)B * S > 0x7fffffffll) return GPT2L_ERR_TOO_LARGE;
  GemmDesc d;
  d.kind = GPT2L_OP_BACKWARD_INPUT;
  d.M = B * S; d.K = K; d.N = N;
  d.out = g_in; d.out_bias = nullptr; d.a = g_out; d.b = w; d.bias = nullptr;
  d.opts = opts_or_default(opts);
  return run_gemm(d, static_cast<cudaStream_t>(stream));
}

int gpt2_linear_backward_weight(float *g_w, float *g_b, const float *g_out, const float *in, int B, int S, int K,
                                int N, const gpt2_linear_opts *opts, gpt2l_stream_t stream) {
  if (B <= 0 || S <= 0) return GPT2L_ERR_BAD_ARG;
  if ((long long)B * S > 0x7fffffffll) return GPT2L_ERR_TOO_LARGE;
  GemmDesc d;
  d.kind = GPT2L_OP_BACKWARD_WEIGHT;
  d.M = B * S; d.K = K; d.N = N;
  d.out = g_w; d.out_bias = g_b; d.a = in; d.b = g_out; d.bias = nullptr;
  d.opts = opts_or_default(opts);
  return run_gemm(d, static_cast<cudaStream_t>(stream));
}

// ---------------------------------------------------------------------------------------
// host-buffer flavours
// ---------------------------------------------------------------------------------------
static int stage_in(DeviceCtx *ctx, int slot, const float *host, size_t count, cudaStream_t st) {
  int e = ensure_bytes(&ctx->stage[slot], &ctx->stage_bytes[slot], count * sizeof(float));
  if (e) return e;
  if (host &&
      cudaMemcpyAsync(ctx->stage[slot], host, count * sizeof(float), cudaMemcpyHostToDevice, st) != cudaSuccess)
    return GPT2L_ERR_CUDA;
  return GPT2L_OK;
}

static int finish_host(DeviceCtx *ctx, cudaStream_t st) {
  if (cudaStreamSynchronize(st) != cudaSuccess) return GPT2L_ERR_CUDA;
  Status s;
  int e = read_status(ctx, &s, true);
  if (e) return e;
  return s.status;
}

int gpt2_linear_forward_host(float *out, const float *in, const float *w, const float *b, int B, int S, int K,
                             int N, const gpt2_linear_opts *opts, gpt2l_stream_t stream) {
  int err;
  DeviceCtx *ctx = ctx_current(&err);
  if (!ctx) return err;
  if (!out || !in || !w || B <= 0 || S <= 0 || K <= 0 || N <= 0) return GPT2L_ERR_BAD_ARG;
  if (opts && (opts->flags & GPT2L_EPI_GELU_DUAL)) return GPT2L_ERR_BAD_ARG;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const size_t M = (size_t)B * S;
  std::lock_guard<std::mutex> lk(g_stage_mu);
  if ((err = stage_in(ctx, 0, in, M * K, st))) return err;
  if ((err = stage_in(ctx, 1, w, (size_t)K * N, st))) return err;
  if ((err = stage_in(ctx, 2, nullptr, M * N, st))) return err;
  if (b && (err = stage_in(ctx, 3, b, (size_t)N, st))) return err;
  err = gpt2_linear_forward(ctx->stage[2], ctx->stage[0], ctx->stage[1], b ? ctx->stage[3] : nullptr, B, S, K, N,
                            opts, stream);
  if (err) return err;
  if (cudaMemcpyAsync(out, ctx->stage[2], M * N * sizeof(float), cudaMemcpyDeviceToHost, st) != cudaSuccess)
    return GPT2L_ERR_CUDA;
  return finish_host(ctx, st);
}

int gpt2_linear_backward_input_host(float *g_in, const float *g_out, const float *w, int B, int S, int K, int N,
                                    const gpt2_linear_opts *opts, gpt2l_stream_t stream) {
  int err;
  DeviceCtx *ctx = ctx_current(&err);
  if (!ctx) return err;
  if (!g_in || !g_out || !w || B <= 0 || S <= 0 || K <= 0 || N <= 0) return GPT2L_ERR_BAD_ARG;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const size_t M = (size_t)B * S;
  std::lock_guard<std::mutex> lk(g_stage_mu);
  if ((err = stage_in(ctx, 0, g_out, M * N, st))) return err;
  if ((err = stage_in(ctx, 1, w, (size_t)K * N, st))) return err;
  if ((err = stage_in(ctx, 2, nullptr, M * K, st))) return err;
  err = gpt2_linear_backward_input(ctx->stage[2], ctx->stage[0], ctx->stage[1], B, S, K, N, opts, stream);
  if (err) return err;
  if (cudaMemcpyAsync(g_in, ctx->stage[2], M * K * sizeof(float), cudaMemcpyDeviceToHost, st) != cudaSuccess)
    return GPT2L_ERR_CUDA;
  return finish_host(ctx, st);
}

int gpt2_linear_backward_weight_host(float *g_w, float *g_b, const float *g_out, const float *in, int B, int S,
                                     int K, int N, const gpt2_linear_opts *opts, gpt2l_stream_t stream) {
  int err;
  DeviceCtx *ctx = ctx_current(&err);
  if (!ctx) return err;
  if (!g_w || !g_out || !in || B <= 0 || S <= 0 || K <= 0 || N <= 0) return GPT2L_ERR_BAD_ARG;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const size_t M = (size_t)B * S;
  std::lock_guard<std::mutex> lk(g_stage_mu);
  if ((err = stage_in(ctx, 0, in, M * K, st))) return err;
  if ((err = stage_in(ctx, 1, g_out, M * N, st))) return err;
  if ((err = stage_in(ctx, 2, nullptr, (size_t)K * N, st))) return err;
  if (g_b && (err = stage_in(ctx, 3, nullptr, (size_t)N, st))) return err;
  err = gpt2_linear_backward_weight(ctx->stage[2], g_b ? ctx->stage[3] : nullptr, ctx->stage[1], ctx->stage[0], B,
                                    S, K, N, opts, stream);
  if (err) return err;
  if (cudaMemcpyAsync(g_w, ctx->stage[2], (size_t)K * N * sizeof(float), cudaMemcpyDeviceToHost, st) !=
      cudaSuccess)
    return GPT2L_ERR_CUDA;
  if (g_b && cudaMemcpyAsync(g_b, ctx->stage[3], (size_t)N * sizeof(float), cudaMemcpyDeviceToHost, st) !=
                 cudaSuccess)
    return GPT2L_ERR_CUDA;
  return finish_host(ctx, st);
}


// ---- pipelined flavours: return once everything is enqueued; results are in the host buffers after
// gpt2_linear_host_synchronize()
namespace {
struct AsyncCall {
  HostPipe *p;
  HostPipe::Set *s;
};

// takes the next staging set and makes the copy-in stream wait until its previous user is done
int async_begin(DeviceCtx *ctx, AsyncCall *c) {
  HostPipe *p = get_pipe(ctx);
  if (!p) return GPT2L_ERR_CUDA;
  HostPipe::Set *s = &p->set[p->calls++ & 1];
  if (s->used && cudaStreamWaitEvent(p->s_in, s->ev_free, 0) != cudaSuccess) return GPT2L_ERR_CUDA;
  c->p = p;
  c->s = s;
  return GPT2L_OK;
}

// room for `count` floats in slot `slot`; copies `host` in when given
int async_stage(AsyncCall &c, int slot, const float *host, size_t count) {
  HostPipe::Set *s = c.s;
  if (count * sizeof(float) > s->bytes[slot]) {
    // growing frees the old buffer: its last user must be done
    if (s->used && cudaEventSynchronize(s->ev_free) != cudaSuccess) return GPT2L_ERR_CUDA;
    int e = ensure_bytes(&s->buf[slot], &s->bytes[slot], count * sizeof(float));
    if (e) return e;
  }
  if (host && cudaMemcpyAsync(s->buf[slot], host, count * sizeof(float), cudaMemcpyHostToDevice, c.p->s_in) !=
                  cudaSuccess)
    return GPT2L_ERR_CUDA;
  return GPT2L_OK;
}

// device copy of a host input: the one uploaded earlier in this window, or a fresh upload
int async_input(AsyncCall &c, const float *host, size_t count, float **dev) {
  HostPipe *p = c.p;
  const size_t bytes = count * sizeof(float);
  for (const auto &i : p->inputs)
    if (i.host == host && i.bytes == bytes) {
      *dev = i.dev;
      p->reused_bytes += bytes;
      return GPT2L_OK;
    }
  HostPipe::Input in = {host, bytes, nullptr, 0};
  int best = -1;
  for (int k = 0; k < (int)p->pool.size(); ++k)
    if (p->pool[k].cap >= bytes && (best < 0 || p->pool[k].cap < p->pool[best].cap)) best = k;
  if (best >= 0) {
    in.dev = p->pool[best].dev;
    in.cap = p->pool[best].cap;
    p->pool.erase(p->pool.begin() + best);
  } else {
    const size_t want = (bytes + ((1u << 20) - 1)) & ~(size_t)((1u << 20) - 1);  // 1 MiB granules
    if (cudaMalloc(reinterpret_cast<void **>(&in.dev), want) != cudaSuccess) {
      (void)cudaGetLastError();
      return GPT2L_ERR_CUDA;
    }
    in.cap = want;
  }
  if (cudaMemcpyAsync(in.dev, host, bytes, cudaMemcpyHostToDevice, p->s_in) != cudaSuccess) {
    p->pool.push_back(in);
    return GPT2L_ERR_CUDA;
  }
  p->uploaded_bytes += bytes;
  p->inputs.push_back(in);
  *dev = in.dev;
  return GPT2L_OK;
}

int async_inputs_done(AsyncCall &c) {
  if (cudaEventRecord(c.s->ev_in, c.p->s_in) != cudaSuccess) return GPT2L_ERR_CUDA;
  return cudaStreamWaitEvent(c.p->s_run, c.s->ev_in, 0) == cudaSuccess ? GPT2L_OK : GPT2L_ERR_CUDA;
}

int async_compute_done(AsyncCall &c) {
  if (cudaEventRecord(c.s->ev_run, c.p->s_run) != cudaSuccess) return GPT2L_ERR_CUDA;
  return cudaStreamWaitEvent(c.p->s_out, c.s->ev_run, 0) == cudaSuccess ? GPT2L_OK : GPT2L_ERR_CUDA;
}

int async_out(AsyncCall &c, float *host, int slot, size_t count) {
  return cudaMemcpyAsync(host, c.s->buf[slot], count * sizeof(float), cudaMemcpyDeviceToHost, c.p->s_out) ==
                 cudaSuccess ? GPT2L_OK : GPT2L_ERR_CUDA;
}

int async_end(AsyncCall &c) {
  c.s->used = true;
  return cudaEventRecord(c.s->ev_free, c.p->s_out) == cudaSuccess ? GPT2L_OK : GPT2L_ERR_CUDA;
}
}  // namespace

#define AK(call)                   \
  do {                             \
    int _e = (call);               \
    if (_e != GPT2L_OK) return _e; \
  } while (0)

int gpt2_linear_forward_host_async(float *out, const float *in, const float *w, const float *b, int B, int S, int K,
                                   int N, const gpt2_linear_opts *opts) {
  int err;
  DeviceCtx *ctx = ctx_current(&err);
  if (!ctx) return err;
  if (!out || !in || !w || B <= 0 || S <= 0 || K <= 0 || N <= 0) return GPT2L_ERR_BAD_ARG;
  if (opts && ((opts->flags & GPT2L_EPI_GELU_DUAL) || opts->aux_op)) return GPT2L_ERR_BAD_ARG;
  const size_t M = (size_t)B * S;
  std::lock_guard<std::mutex> lk(g_stage_mu);
  AsyncCall c;
  AK(async_begin(ctx, &c));
  float *d_in = nullptr, *d_w = nullptr, *d_b = nullptr;
  AK(async_input(c, in, M * K, &d_in));
  AK(async_input(c, w, (size_t)K * N, &d_w));
  if (b) AK(async_input(c, b, (size_t)N, &d_b));
  AK(async_stage(c, 2, nullptr, M * N));
  AK(async_inputs_done(c));
  AK(gpt2_linear_forward(c.s->buf[2], d_in, d_w, d_b, B, S, K, N, opts, c.p->s_run));
  AK(async_compute_done(c));
  AK(async_out(c, out, 2, M * N));
  return async_end(c);
}

int gpt2_linear_backward_input_host_async(float *g_in, const float *g_out, const float *w, int B, int S, int K, int N,
                                          const gpt2_linear_opts *opts) {
  int err;
  DeviceCtx *ctx = ctx_current(&err);
  if (!ctx) return err;
  if (!g_in || !g_out || !w || B <= 0 || S <= 0 || K <= 0 || N <= 0) return GPT2L_ERR_BAD_ARG;
  if (opts && opts->aux_op) return GPT2L_ERR_BAD_ARG;
  const size_t M = (size_t)B * S;
  std::lock_guard<std::mutex> lk(g_stage_mu);
  AsyncCall c;
  AK(async_begin(ctx, &c));
  float *d_go = nullptr, *d_w = nullptr;
  AK(async_input(c, g_out, M * N, &d_go));
  AK(async_input(c, w, (size_t)K * N, &d_w));
  AK(async_stage(c, 2, nullptr, M * K));
  AK(async_inputs_done(c));
  AK(gpt2_linear_backward_input(c.s->buf[2], d_go, d_w, B, S, K, N, opts, c.p->s_run));
  AK(async_compute_done(c));
  AK(async_out(c, g_in, 2, M * K));
  return async_end(c);
}

int gpt2_linear_backward_weight_host_async(float *g_w, float *g_b, const float *g_out, const float *in, int B, int S,
                                           int K, int N, const gpt2_linear_opts *opts) {
  int err;
  DeviceCtx *ctx = ctx_current(&err);
  if (!ctx) return err;
  if (!g_w || !g_out || !in || B <= 0 || S <= 0 || K <= 0 || N <= 0) return GPT2L_ERR_BAD_ARG;
  const size_t M = (size_t)B * S;
  std::lock_guard<std::mutex> lk(g_stage_mu);
  AsyncCall c;
  AK(async_begin(ctx, &c));
  float *d_in = nullptr, *d_go = nullptr;
  AK(async_input(c, in, M * K, &d_in));
  AK(async_input(c, g_out, M * N, &d_go));
  AK(async_stage(c, 2, nullptr, (size_t)K * N));
  if (g_b) AK(async_stage(c, 3, nullptr, (size_t)N));
  AK(async_inputs_done(c));
  AK(gpt2_linear_backward_weight(c.s->buf[2], g_b ? c.s->buf[3] : nullptr, d_go, d_in, B, S, K, N, opts,
                                 c.p->s_run));
  AK(async_compute_done(c));
  AK(async_out(c, g_w, 2, (size_t)K * N));
  if (g_b) AK(async_out(c, g_b, 3, (size_t)N));
  return async_end(c);
}

int gpt2_linear_host_synchronize(void) {
  int err;
  DeviceCtx *ctx = ctx_current(&err);
  if (!ctx) return err;
  std::lock_guard<std::mutex> lk(g_stage_mu);
  HostPipe *p = ctx->pipe;
  if (p) {
    if (cudaStreamSynchronize(p->s_in) != cudaSuccess || cudaStreamSynchronize(p->s_run) != cudaSuccess ||
        cudaStreamSynchronize(p->s_out) != cudaSuccess)
      return GPT2L_ERR_CUDA;
    // the window is over: inputs may change now, so their device copies are only storage from here on
    for (auto &i : p->inputs) p->pool.push_back(i);
    p->inputs.clear();
  }
  Status s;
  int e = read_status(ctx, &s, true);
  if (e) return e;
  return s.status;
}

}  // extern "C"
