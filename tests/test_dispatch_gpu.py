"""Calls that the automatic choices (CTA pairs, tile width, splits) send different ways, and the gradients a whole backward
pass has to start from zero."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


# mode, M, K, N: 3xTF32 just under and over the line for pairs (16 k-blocks a pair) with ragged edges; TF32 over the line
# for plain calls (96); short batches, with and without a split of the reduction
@pytest.mark.parametrize("mode,M,K,N", [(1, 1030, 768, 1028), (1, 2052, 1028, 1540), (0, 4100, 3072, 772), (0, 4096, 772, 3072),
                                        (0, 256, 768, 2304), (0, 200, 2304, 772), (0, 60, 64, 68)])
def test_every_direction_against_float64(gpu, mode, M, K, N):
    gen = torch.Generator(device="cuda").manual_seed(M + N)
    x, w, b, dy = (torch.randn(s, device="cuda", generator=gen) for s in ((M, K), (K, N), (N,), (M, N)))
    y, dx, dw, db = (torch.full(s, float("nan"), device="cuda") for s in ((M, N), (M, K), (K, N), (N,)))
    o = gpu.make_opts(mode=mode)
    gpu.check("forward", gpu.forward(y, x, w, b, 1, M, K, N, o))
    gpu.check("backward_input", gpu.backward_input(dx, dy, w, 1, M, K, N, o))
    gpu.check("backward_weight", gpu.backward_weight(dw, db, dy, x, 1, M, K, N, o))
    torch.cuda.synchronize()
    X, W, D = x.double(), w.double(), dy.double()

    def rel(got, want):
        return float((got.double() - want).norm() / want.norm())

    # operands truncated to 10 mantissa bits: up to 2^-10 each, 7.7e-4 on average over both; 3xTF32 keeps 21 bits and is
    # bounded by the tensor core's fp32 accumulation, 3e-5 for 8192 terms
    tol = 1.5e-3 if mode == 0 else 6e-5
    assert rel(y, X @ W + b.double()) <= tol
    assert rel(dx, D @ W.t()) <= tol
    assert rel(dw, X.t() @ D) <= tol
    assert rel(db, D.sum(0)) <= 1e-5


def test_3xtf32_keeps_its_split(gpu):
    """30 k-blocks a part leave 6.6e-6, one part of 148 leaves 3.3e-5 (the tensor core's own sums lose about 2e-8 a term)"""
    M, K, N = 3620, 4724, 860
    gen = torch.Generator(device="cuda").manual_seed(1)
    x, w = (torch.randn(s, device="cuda", generator=gen) for s in ((M, K), (K, N)))
    y = torch.empty((M, N), device="cuda")
    gpu.check("forward", gpu.forward(y, x, w, None, 1, M, K, N, gpu.make_opts(mode=1)))
    want = x.double() @ w.double()
    assert float((y.double() - want).norm() / want.norm()) <= 1e-5


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("pair", [0, 1, 2])
@pytest.mark.parametrize("split,det", [(0, 0), (0, 1), (5, 0), (5, 1)])
@pytest.mark.parametrize("M,K,N", [(1000, 132, 64), (516, 260, 36), (2048, 64, 4)])
def test_narrow_outputs_against_float64(gpu, mode, pair, split, det, M, K, N):
    """outputs narrower than a pair's narrowest tile, in one part or several, added by the copy engine or in fixed order"""
    gen = torch.Generator(device="cuda").manual_seed(M + N)
    x, w, dy = (torch.randn(s, device="cuda", generator=gen) for s in ((M, K), (K, N), (M, N)))
    y, dx, dw, db = (torch.full(s, float("nan"), device="cuda") for s in ((M, N), (M, K), (K, N), (N,)))
    o = gpu.make_opts(mode=mode, cta_pair=pair, split_k=split, deterministic=det)
    gpu.check("forward", gpu.forward(y, x, w, None, 1, M, K, N, o))
    gpu.check("backward_input", gpu.backward_input(dx, dy, w, 1, M, K, N, o))
    gpu.check("backward_weight", gpu.backward_weight(dw, db, dy, x, 1, M, K, N, o))
    torch.cuda.synchronize()
    X, W, D = x.double(), w.double(), dy.double()
    # operands keep 10 mantissa bits (3xTF32: 21), sums are fp32: within c times the sum of the products' magnitudes
    c = 2.0 ** -9 if mode == 0 else 2.0 ** -19
    for got, a, b, terms in ((y, X, W, K), (dx, D, W.t(), N), (dw, X.t(), D, M)):
        assert bool(((got.double() - a @ b).abs() <= (c + 2 * (terms + 1) * 2.0 ** -24) * (a.abs() @ b.abs())).all())
    assert bool(((db.double() - D.sum(0)).abs() <= 2 * M * 2.0 ** -24 * D.abs().sum(0)).all())


class _View:
    def __init__(self, ptr, count):
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": "<f4", "data": (ptr, False), "version": 3}


@pytest.mark.parametrize("layers", [1, 3])
def test_backward_does_not_depend_on_old_gradients(gpu, layers):
    """every gradient is overwritten or starts from zero, whatever the buffer held; the parts called one by one agree"""
    B, T, C, V, Vp = 2, 32, 128, 250, 256
    m = gpu.Model(V, Vp, layers, C // 64, C, 48, B, T, mode=1)
    rng = np.random.default_rng(1)
    m.set_params((rng.standard_normal(m.num_params) * 0.05).astype(np.float32))
    tok, tgt = (torch.from_numpy(rng.integers(0, V, B * T).astype(np.int32)).cuda() for _ in range(2))
    grads = torch.as_tensor(_View(m.grads_ptr(), m.num_params), device="cuda")

    def parts():
        gpu.check("head", m.backward_head())
        for l in reversed(range(layers)):
            gpu.check("layer", m.backward_layer(l))
        gpu.check("embedding", m.backward_embedding())

    got = []
    for backward, fill in ((lambda: gpu.check("backward", m.backward()), 0.0),
                           (lambda: gpu.check("backward", m.backward()), float("nan")), (parts, float("nan"))):
        gpu.check("forward", m.forward(tok, tgt))
        grads.fill_(fill)
        backward()
        torch.cuda.synchronize()
        got.append(grads.clone())
    assert bool(torch.isfinite(got[1]).all())
    for g in got[1:]:  # sums by atomics: the same terms in another order
        assert float((g - got[0]).abs().max()) <= 1e-5 * float(got[0].abs().max())
    m.close()
