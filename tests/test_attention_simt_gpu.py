"""The fp32 attention kernels at the edges of their 64-row tiles."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _truth(qkv, dout, B, T, NH):
    C = NH * 64
    x = qkv.double().requires_grad_()
    q, k, v = (z.view(B, T, NH, 64).transpose(1, 2) for z in x.split(C, 1))
    s = (q @ k.transpose(-1, -2)) / 8
    s = s.masked_fill(~torch.ones(T, T, dtype=torch.bool, device=s.device).tril(), float("-inf"))
    o = (torch.softmax(s, -1) @ v).transpose(1, 2).reshape(B * T, C)
    (g,) = torch.autograd.grad(o, x, dout.double())
    return o.detach(), torch.logsumexp(s, -1).detach(), g


def _run(gpu, qkv, dout, B, T, NH):
    C = NH * 64
    out, g = torch.full((B * T, C), float("nan"), device="cuda"), torch.full((B * T, 3 * C), float("nan"), device="cuda")
    lse, row = torch.empty(B, NH, T, device="cuda"), torch.empty(B, NH, T, device="cuda")
    gpu.check("forward", gpu.attention_forward(out, lse, None, qkv, B, T, NH, C, gpu.ATT_SIMT, 0))
    gpu.check("backward", gpu.attention_backward(g, dout, qkv, out, lse, None, row, None, B, T, C, NH, gpu.ATT_SIMT, 0))
    torch.cuda.synchronize()
    return out, lse, g


def _inputs(B, T, NH):
    gen = torch.Generator(device="cuda").manual_seed(T)
    qkv = torch.randn(B * T, 3 * NH * 64, device="cuda", generator=gen)
    return qkv, torch.randn(B * T, NH * 64, device="cuda", generator=gen) * 0.1


@pytest.mark.parametrize("T", [1, 2, 63, 64, 65, 127, 129, 333, 1000])
def test_against_float64(gpu, T):
    B, NH = 2, 3
    qkv, dout = _inputs(B, T, NH)
    got = _run(gpu, qkv, dout, B, T, NH)
    for a, e in zip(got, _truth(qkv, dout, B, T, NH)):
        # scores of 64 products (|s| < 40): 64 * 2^-24 * 40 = 1.5e-4 at worst in the exponent, random signs an eighth
        # of it; gradients sum up to T such terms of both signs: 2e-5 of the largest entry covers T = 1000
        assert float((a.double() - e).abs().max()) <= 2e-5 * max(1.0, float(e.abs().max()))


def test_a_later_token_does_not_reach_an_earlier_one(gpu):
    B, T, NH = 1, 150, 2
    qkv, dout = _inputs(B, T, NH)
    clean = _run(gpu, qkv, dout, B, T, NH)
    qkv[100] = float("nan")  # inside the second tile, seen by rows 100 ..
    dirty = _run(gpu, qkv, dout, B, T, NH)
    assert torch.equal(clean[0][:100], dirty[0][:100])
    assert torch.equal(clean[2][:100, :128], dirty[2][:100, :128])  # dq of the rows before it
    assert bool(dirty[0][100:].isnan().all())
