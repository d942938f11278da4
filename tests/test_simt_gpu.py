"""The fp32 CUDA-core GEMM (rows TMA cannot address, or force_simt) at the edges of its tiles and splits."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# one element; smaller than a tile; an edge on either side of 64 and 128; three k (less than a slab of 16);
# few tiles with a deep reduction (16 parts, the last one short); many tiles without a split
SIZES = [(1, 1, 1), (3, 5, 7), (63, 64, 65), (65, 129, 63), (128, 127, 129), (129, 3, 1001), (31, 4099, 33),
         (2, 769, 5001), (257, 771, 643), (2100, 770, 1001)]


@pytest.mark.parametrize("M,K,N", SIZES)
def test_every_direction_against_float64(gpu, M, K, N):
    gen = torch.Generator(device="cuda").manual_seed(M + K + N)
    x, w, b, dy = (torch.randn(s, device="cuda", generator=gen) for s in ((M, K), (K, N), (N,), (M, N)))
    y, dx, dw, db = (torch.full(s, float("nan"), device="cuda") for s in ((M, N), (M, K), (K, N), (N,)))
    o = gpu.make_opts(force_simt=1)
    gpu.check("forward", gpu.forward(y, x, w, b, 1, M, K, N, o))
    gpu.check("backward_input", gpu.backward_input(dx, dy, w, 1, M, K, N, o))
    gpu.check("backward_weight", gpu.backward_weight(dw, db, dy, x, 1, M, K, N, o))
    torch.cuda.synchronize()
    X, W, b64, D = (t.double() for t in (x, w, b, dy))

    def close(got, want, terms, magnitude):
        # a sum of n products in fp32, in any order and with one rounding each, is within n * 2^-24 of the sum of
        # the magnitudes (first order; twice that covers the rest for every n here)
        assert bool(((got.double() - want).abs() <= 2 * (terms + 1) * 2.0 ** -24 * magnitude).all())

    close(y, X @ W + b64, K, X.abs() @ W.abs() + b64.abs())
    close(dx, D @ W.t(), N, D.abs() @ W.abs().t())
    close(dw, X.t() @ D, M, X.abs().t() @ D.abs())
    close(db, D.sum(0), M, D.abs().sum(0))
    again = torch.empty_like(dx)
    gpu.check("backward_input", gpu.backward_input(again, dy, w, 1, M, K, N, o))
    assert torch.equal(again, dx)  # parts are added in a fixed order
