// Prints the tiling that the library plans for calls read from standard input, on a machine with or without a GPU:
//   mode kind M K N split_k cta_pair deterministic aux gelu stats  ->  error pair bn splits kb_per_split tiles_n
// With the argument "simt", the CUDA-core GEMM's plan instead:
//   Mc Nc Kc max_parts  ->  tile rows, tile columns, parts, k per part
// With "attention", the launches of the fp32 attention kernels:
//   T  ->  64-row tiles of each launch
#include <cstdio>
#include <cstring>

#include "layers.h"
#include "linear_internal.h"

static int simt() {
  int Mc, Nc, Kc, max_parts;
  while (scanf("%d %d %d %d", &Mc, &Nc, &Kc, &max_parts) == 4) {
    const g2l::SimtPlan p = g2l::simt_plan(Mc, Nc, Kc, 148, max_parts);
    printf("%d %d %d %d\n", p.bm, p.bn, p.parts, p.k_per_part);
  }
  return 0;
}

static int attention() {
  int T;
  while (scanf("%d", &T) == 1) {
    for (int first = 0, n; (n = g2l::att_launch_tiles(T, first)) > 0; first += n) printf("%d ", n);
    printf("\n");
  }
  return 0;
}

int main(int argc, char **argv) {
  if (argc > 1 && !strcmp(argv[1], "attention")) return attention();
  if (argc > 1 && !strcmp(argv[1], "simt")) return simt();
  constexpr int SMS = 148, PAIRS = 74;
  int mode, kind, M, K, N, split, pair, det, aux, gelu, stats;
  while (scanf("%d %d %d %d %d %d %d %d %d %d %d", &mode, &kind, &M, &K, &N, &split, &pair, &det, &aux, &gelu, &stats) == 11) {
    float *any = reinterpret_cast<float *>(16);  // plans look at shapes and options, not at memory
    g2l::GemmDesc d = {};
    d.kind = kind; d.M = M; d.K = K; d.N = N;
    d.out = any; d.a = any; d.b = any;
    d.opts.mode = mode; d.opts.split_k = split; d.opts.cta_pair = pair; d.opts.deterministic = det;
    if (aux) { d.opts.aux_op = aux; d.opts.aux = any; }
    if (gelu) { d.opts.flags = GPT2L_EPI_GELU_DUAL; d.opts.out2 = any; }
    if (stats) { d.xent_stats = any; d.xent_vocab = N; }
    d.opts.cta_pair = g2l::choose_cta_pair(d, SMS, PAIRS);
    g2l::GemmOp op;
    const int e = g2l::plan_op(d, SMS, &op);
    printf("%d %d %d %d %d %d\n", e, op.pair, op.bn, op.splits, op.kb_per_split, op.tiles_n);
  }
}
