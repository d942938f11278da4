"""The work whose speed is kept track of: calls of the library's public entry points with the shapes,
options and value distributions that training GPT-2 with it meets.

Five kinds of case:
  linear     one linear layer: forward, gradient of the input, gradient of weight and bias
  mlp        the two linear layers of a block with their epilogues: fc with the GELU dual store, fc-proj with
             the residual add, and backward with the GELU gradient in the epilogue
  head       the tied lm_head: logits with loss and log-sum-exp, then both gradients
  attention  causal self-attention, forward and backward
  train      one training step of a whole model: forward, backward, AdamW
"""
import importlib.util
import math
import os
import sys

import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_VOCAB, _PADDED_VOCAB = 50257, 50304


def _package():
    """the package directory has a dot in its name, so it is imported by path (once per process)"""
    name = "gpt2cu_b200"
    if name not in sys.modules:
        where = os.path.join(_ROOT, "gpt2.cu_b200")
        spec = importlib.util.spec_from_file_location(name, os.path.join(where, "__init__.py"),
                                                      submodule_search_locations=[where])
        mod = importlib.util.module_from_spec(spec)
        sys.modules[name] = mod
        spec.loader.exec_module(mod)
    return sys.modules[name]


def listed():
    return [
        # the smallest calls: one QKV layer at the batch shape the trainer ships with (4 sequences of 64 tokens)
        {"name": "linear_qkv_b4_t64", "kind": "linear", "B": 4, "S": 64, "K": 768, "N": 2304, "mode": 0, "bias": True},
        # an ordinary layer with sizes that are no multiples of a tile: short batch of odd-length sequences
        {"name": "linear_ragged_b3_t777", "kind": "linear", "B": 3, "S": 777, "K": 1028, "N": 772, "mode": 0, "bias": True},
        # fc-proj at the benchmark's 8 x 1024 tokens in the fp32-faithful mode that loss parity runs use
        {"name": "linear_fcproj_3xtf32_b8_t1024", "kind": "linear", "B": 8, "S": 1024, "K": 3072, "N": 768, "mode": 1,
         "bias": True},
        # the lm_head with the vocabulary as it is, 50257, unpadded: rows that are not 16-byte multiples
        {"name": "linear_head_vocab50257_b4_t64", "kind": "linear", "B": 4, "S": 64, "K": 768, "N": _VOCAB, "mode": 0,
         "bias": False},
        # a block's MLP at the benchmark's 8 x 1024 tokens, epilogues as the training step uses them
        {"name": "mlp_b8_t1024", "kind": "mlp", "B": 8, "S": 1024, "C": 768, "mode": 0},
        # the lm_head with cross-entropy at 8 x 1024 tokens: the largest GEMMs there are
        {"name": "head_b8_t1024", "kind": "head", "B": 8, "S": 1024, "C": 768, "mode": 0},
        # attention of a GPT-2 small layer at the trained sequence length, 16 sequences
        {"name": "attention_b16_t1024", "kind": "attention", "B": 16, "T": 1024, "NH": 12, "impl": 0, "mode": 0},
        # attention at the shipped batch shape, where the model takes the batched GEMMs (T is no multiple of 128)
        {"name": "attention_gemm_b4_t64", "kind": "attention", "B": 4, "T": 64, "NH": 12, "impl": 1, "mode": 0},
        # attention in the fp32-faithful mode
        {"name": "attention_3xtf32_b4_t1024", "kind": "attention", "B": 4, "T": 1024, "NH": 12, "impl": 1, "mode": 1},
        # attention over sequences of an odd length
        {"name": "attention_b4_t777", "kind": "attention", "B": 4, "T": 777, "NH": 12, "impl": 2, "mode": 0},
        # the training step of GPT-2 small at the shipped shape, forward and backward replayed from a graph
        {"name": "train_small_b4_t64", "kind": "train", "B": 4, "T": 64, "L": 12, "NH": 12, "V": _VOCAB,
         "Vp": _PADDED_VOCAB, "mode": 0, "graph": True},
        # the training step of GPT-2 small at 8 x 1024 tokens, separate launches as every rank of a job makes them
        {"name": "train_small_b8_t1024", "kind": "train", "B": 8, "T": 1024, "L": 12, "NH": 12, "V": _VOCAB,
         "Vp": _PADDED_VOCAB, "mode": 0, "graph": False},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _draw_mode(rng):
    return 1 if rng.random() < 0.35 else 0


def draw(rng):
    kind = rng.choice(["linear", "linear", "linear", "mlp", "head", "attention", "attention", "attention", "train"])
    if kind == "linear":
        rows = _log_int(rng, 64, 16384)
        batch = rng.randint(1, 8)
        case = {"kind": "linear", "B": batch, "S": max(1, rows // batch), "mode": _draw_mode(rng),
                "bias": rng.random() < 0.7}
        if rng.random() < 0.25:  # sizes that are no multiples of four
            case["K"], case["N"] = 768 + rng.choice([0, 0, 1, 3]), _log_int(rng, 100, 4000) * 2 + 1
            case["S"] = max(1, min(case["S"], 4096 // batch))
        else:
            case["K"], case["N"] = 4 * _log_int(rng, 16, 1280), 4 * _log_int(rng, 16, 1280)
        return case
    if kind == "mlp":
        return {"kind": "mlp", "B": rng.randint(1, 8), "S": _log_int(rng, 32, 1024), "C": 64 * rng.randint(6, 20),
                "mode": _draw_mode(rng)}
    if kind == "head":
        return {"kind": "head", "B": rng.randint(1, 8), "S": _log_int(rng, 32, 1024), "C": 64 * rng.randint(6, 16),
                "mode": 0}
    if kind == "attention":
        impl = rng.choice([0, 1, 2])
        step = {0: 128, 1: 32, 2: 1}[impl]
        length = max(step, _log_int(rng, 32, 1024) // step * step)
        return {"kind": "attention", "B": rng.randint(1, 12 if impl == 0 else 4), "T": length, "NH": rng.randint(6, 16),
                "impl": impl, "mode": _draw_mode(rng) if impl == 1 else 0}
    return {"kind": "train", "B": rng.randint(1, 4), "T": 32 * rng.randint(2, 16), "L": rng.randint(2, 6),
            "NH": rng.choice([6, 8, 12]), "V": 2000 + rng.randint(0, 40), "Vp": 2048, "mode": _draw_mode(rng),
            "graph": rng.random() < 0.5}


# ------------------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------------------
_HYPER = (0.9, 0.95, 1e-8, 0.1)  # AdamW betas, eps, weight decay
_WARMUP_STEPS, _PEAK_LR = 2000, 3e-4  # linear warm-up: the first steps of a run


def _inputs(case, seed):
    """every input tensor of a case, fp32 on the GPU, from the seed alone"""
    gen = torch.Generator(device="cuda").manual_seed(1000003 * (seed + 1) % (1 << 62))

    def normal(*shape, std=1.0):
        t = torch.randn(shape, device="cuda", generator=gen)
        return t if std == 1.0 else t.mul_(std)

    k = case["kind"]
    if k == "linear":
        M, K, N = case["B"] * case["S"], case["K"], case["N"]
        return {"x": normal(M, K), "w": normal(K, N, std=0.02), "b": normal(N, std=0.02) if case["bias"] else None,
                "dy": normal(M, N, std=0.01)}
    if k == "mlp":
        M, C = case["B"] * case["S"], case["C"]
        return {"x": normal(M, C), "w1": normal(C, 4 * C, std=0.02), "b1": normal(4 * C, std=0.02),
                "w2": normal(4 * C, C, std=0.02), "b2": normal(C, std=0.02), "res": normal(M, C),
                "dy": normal(M, C, std=0.01)}
    if k == "head":
        M, C = case["B"] * case["S"], case["C"]
        w = normal(C, _PADDED_VOCAB, std=0.02)
        w[:, _VOCAB:] = 0.0
        tgt = torch.randint(0, _VOCAB, (M,), dtype=torch.int32, device="cuda", generator=gen)
        return {"x": normal(M, C), "w": w, "tgt": tgt, "dy": normal(M, _PADDED_VOCAB, std=1e-4)}
    if k == "attention":
        M, C = case["B"] * case["T"], case["NH"] * 64
        return {"qkv": normal(M, 3 * C), "dout": normal(M, C, std=0.1)}
    M = case["B"] * case["T"]
    tok = torch.randint(0, case["V"], (M,), dtype=torch.int32, device="cuda", generator=gen)
    tgt = torch.randint(0, case["V"], (M,), dtype=torch.int32, device="cuda", generator=gen)
    C, L, Vp = case["NH"] * 64, case["L"], case["Vp"]
    params = normal(C * Vp + max(1024, case["T"]) * C + L * (12 * C * C + 13 * C) + 2 * C, std=0.02)
    params[: C * Vp].view(C, Vp)[:, case["V"]:] = 0.0
    for name, first, shape in _param_layout(case):
        if name.endswith(("ln1_w", "ln2_w", "lnf_w")):
            params[first: first + shape[0]] = 1.0
    return {"tok": tok, "tgt": tgt, "params": params}


def _param_layout(case):
    """(name, offset, shape) of every tensor of the flat parameter buffer, in its order"""
    C, L, Vp, P = case["NH"] * 64, case["L"], case["Vp"], max(1024, case["T"])
    names = [("wte", (C, Vp)), ("wpe", (P, C))]
    for i in range(L):
        names += [(f"{i}.ln1_w", (C,)), (f"{i}.ln1_b", (C,)), (f"{i}.qkv_w", (C, 3 * C)), (f"{i}.qkv_b", (3 * C,)),
                  (f"{i}.proj_w", (C, C)), (f"{i}.proj_b", (C,)), (f"{i}.ln2_w", (C,)), (f"{i}.ln2_b", (C,)),
                  (f"{i}.fc_w", (C, 4 * C)), (f"{i}.fc_b", (4 * C,)), (f"{i}.fcproj_w", (4 * C, C)),
                  (f"{i}.fcproj_b", (C,))]
    names += [("lnf_w", (C,)), ("lnf_b", (C,))]
    out, at = [], 0
    for name, shape in names:
        out.append((name, at, shape))
        at += math.prod(shape)
    return out


class _DeviceView:
    """a model's own buffer; holds the model, so that a tensor over the buffer keeps it alive"""

    def __init__(self, owner, ptr, count):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": "<f4", "data": (ptr, False), "version": 3}


def prepare(case, seed):
    g = _package()
    device = torch.cuda.current_device()
    g.init(device)
    t = _inputs(case, seed)
    k = case["kind"]

    def empty(*shape):
        return torch.empty(shape, device="cuda")

    if k == "linear":
        M, K, N = case["B"] * case["S"], case["K"], case["N"]
        t.update(y=empty(M, N), dx=empty(M, K), dw=empty(K, N), db=empty(N) if case["bias"] else None)
    elif k == "mlp":
        M, C = case["B"] * case["S"], case["C"]
        t.update(h=empty(M, 4 * C), act=empty(M, 4 * C), y=empty(M, C), dh=empty(M, 4 * C), dx=empty(M, C),
                 dw1=empty(C, 4 * C), db1=empty(4 * C), dw2=empty(4 * C, C), db2=empty(C))
    elif k == "head":
        M, C = case["B"] * case["S"], case["C"]
        t.update(logits=empty(M, _PADDED_VOCAB), loss=empty(M), lse=empty(M), dx=empty(M, C),
                 dw=empty(C, _PADDED_VOCAB))
    elif k == "attention":
        B, T, NH = case["B"], case["T"], case["NH"]
        M, C = B * T, NH * 64
        square = case["impl"] == g.ATT_GEMM
        t.update(out=empty(M, C), lse=empty(B, NH, T), row=empty(B, NH, T), dqkv=empty(M, 3 * C),
                 probs=empty(B, NH, T, T) if square else None, tt=empty(B, NH, T, T) if square else None)
    else:
        C = case["NH"] * 64
        model = g.Model(case["V"], case["Vp"], case["L"], case["NH"], C, max(1024, case["T"]), case["B"], case["T"],
                        mode=case["mode"])
        params = torch.as_tensor(_DeviceView(model, model.params_ptr(), model.num_params), device="cuda")
        grads = torch.as_tensor(_DeviceView(model, model.grads_ptr(), model.num_params), device="cuda")
        params.copy_(t.pop("params"))
        t.update(model=model, p=params, grad=grads, step=0)
        if case["graph"]:  # a training program replays its graph from the third step on
            stream = torch.cuda.current_stream().cuda_stream
            for _ in range(2):
                g.check("graph", model.forward_backward_graph(t["tok"], t["tgt"], stream))
    t.update(g=g, case=case)
    return t


# ------------------------------------------------------------------------------------------------------
# one pass
# ------------------------------------------------------------------------------------------------------
def run(state):
    s, case, g = state, state["case"], state["g"]
    stream = torch.cuda.current_stream().cuda_stream
    k = case["kind"]
    if k == "linear":
        B, S, K, N = case["B"], case["S"], case["K"], case["N"]
        o = g.make_opts(mode=case["mode"])
        g.check("forward", g.forward(s["y"], s["x"], s["w"], s["b"], B, S, K, N, o, stream))
        g.check("dgrad", g.backward_input(s["dx"], s["dy"], s["w"], B, S, K, N, o, stream))
        g.check("wgrad", g.backward_weight(s["dw"], s["db"], s["dy"], s["x"], B, S, K, N, o, stream))
        return {n: s[n] for n in ("y", "dx", "dw", "db") if s[n] is not None}
    if k == "mlp":
        B, S, C, mode = case["B"], case["S"], case["C"], case["mode"]
        plain = g.make_opts(mode=mode)
        gelu = g.make_opts(mode=mode, flags=g.EPI_GELU_DUAL, out2=s["act"].data_ptr())
        residual = g.make_opts(mode=mode, aux=s["res"], aux_op=g.AUX_ADD)
        gelu_back = g.make_opts(mode=mode, aux=s["h"], aux_op=g.AUX_GELU_GRAD)
        g.check("fc", g.forward(s["h"], s["x"], s["w1"], s["b1"], B, S, C, 4 * C, gelu, stream))
        g.check("fcproj", g.forward(s["y"], s["act"], s["w2"], s["b2"], B, S, 4 * C, C, residual, stream))
        g.check("fcproj dgrad", g.backward_input(s["dh"], s["dy"], s["w2"], B, S, 4 * C, C, gelu_back, stream))
        g.check("fcproj wgrad", g.backward_weight(s["dw2"], s["db2"], s["dy"], s["act"], B, S, 4 * C, C, plain, stream))
        g.check("fc dgrad", g.backward_input(s["dx"], s["dh"], s["w1"], B, S, C, 4 * C, plain, stream))
        g.check("fc wgrad", g.backward_weight(s["dw1"], s["db1"], s["dh"], s["x"], B, S, C, 4 * C, plain, stream))
        return {n: s[n] for n in ("h", "act", "y", "dh", "dw2", "db2", "dx", "dw1", "db1")}
    if k == "head":
        B, S, C = case["B"], case["S"], case["C"]
        o = g.make_opts(mode=case["mode"])
        g.check("head", g.forward_xent(s["logits"], s["loss"], s["lse"], s["x"], s["w"], s["tgt"], B, S, C,
                                       _PADDED_VOCAB, _VOCAB, o, stream))
        g.check("head dgrad", g.backward_input(s["dx"], s["dy"], s["w"], B, S, C, _PADDED_VOCAB, o, stream))
        g.check("head wgrad", g.backward_weight(s["dw"], None, s["dy"], s["x"], B, S, C, _PADDED_VOCAB, o, stream))
        return {n: s[n] for n in ("logits", "loss", "lse", "dx", "dw")}
    if k == "attention":
        B, T, NH, impl, mode = case["B"], case["T"], case["NH"], case["impl"], case["mode"]
        C = NH * 64
        g.check("attention", g.attention_forward(s["out"], s["lse"], s["probs"], s["qkv"], B, T, NH, C, impl, mode,
                                                 stream))
        g.check("attention backward", g.attention_backward(s["dqkv"], s["dout"], s["qkv"], s["out"], s["lse"],
                                                           s["probs"], s["row"], s["tt"], B, T, C, NH, impl, mode,
                                                           stream))
        return {"out": s["out"], "dqkv": s["dqkv"]}
    m = s["model"]
    s["step"] += 1
    if case["graph"]:
        g.check("graph", m.forward_backward_graph(s["tok"], s["tgt"], stream))
    else:
        g.check("forward", m.forward(s["tok"], s["tgt"], stream))
        g.check("backward", m.backward(stream))
    g.check("update", m.update(_PEAK_LR * s["step"] / _WARMUP_STEPS, *_HYPER, s["step"], stream))
    return {"grad": s["grad"], "p": s["p"]}


# ------------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ------------------------------------------------------------------------------------------------------
def work(case):
    k = case["kind"]
    if k == "linear":
        M, K, N = case["B"] * case["S"], case["K"], case["N"]
        nb = N if case["bias"] else 0
        return {"bytes": 4 * (2 * M * K + 2 * M * N + 2 * K * N + 2 * nb), "flops": 6 * M * K * N}
    if k == "mlp":
        M, C = case["B"] * case["S"], case["C"]
        # x, residual, dy in; y, dx out; h, act, dh (4C wide) out; weights in, their gradients out
        return {"bytes": 4 * (M * C * 5 + 3 * M * 4 * C + 16 * C * C + 10 * C), "flops": 6 * 2 * M * C * 4 * C}
    if k == "head":
        M, C, N = case["B"] * case["S"], case["C"], _PADDED_VOCAB
        return {"bytes": 4 * (2 * M * C + 2 * M * N + 2 * C * N + 3 * M), "flops": 6 * M * C * N}
    if k == "attention":
        B, T, NH = case["B"], case["T"], case["NH"]
        M, C = B * T, NH * 64
        # causal: half of each T x T product; two products forward, five backward
        return {"bytes": 4 * (3 * M * C + 2 * M * C + 3 * M * C), "flops": 7 * B * NH * T * T * 64}
    C, L, Vp = case["NH"] * 64, case["L"], case["Vp"]
    M = case["B"] * case["T"]
    n = sum(math.prod(shape) for _, _, shape in _param_layout(case))
    gemm = 6 * M * (L * 12 * C * C + C * Vp)
    att = 7 * L * case["B"] * case["NH"] * case["T"] ** 2 * 64
    # parameters, both moments and the gradient: read and written once
    return {"bytes": 4 * (3 * n * 2 + n), "flops": gemm + att}


def tolerance(case):
    """about four times the distance to 64 bits that was measured over these ranges"""
    k = case["kind"]
    if k == "attention" and case["impl"] == 2:
        return {"rel": 1e-5}  # fp32 arithmetic throughout: 6e-7
    if k == "linear" and (case["K"] % 4 or case["N"] % 4):
        return {"rel": 2e-5}  # fp32 arithmetic throughout: 4e-6 for a reduction over 50257
    if case["mode"] == 1:  # fp32 accumulation in the tensor core: 3e-5 for a reduction over 8192
        return {"rel": 1.2e-4}
    # operands truncated to TF32: 8e-4 per product, 1.6e-3 behind another one, 2e-3 through a whole model
    return {"rel": 8e-3 if k == "train" else 4e-3}


# ------------------------------------------------------------------------------------------------------
# the same in 64 bits
# ------------------------------------------------------------------------------------------------------
def _gelu(x):
    return 0.5 * x * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (x + 0.044715 * x ** 3)))


def _exact_attention(q, k, v):
    """q, k, v [B, NH, T, 64] -> [B, NH, T, 64]"""
    T = q.shape[2]
    s = (q @ k.transpose(-1, -2)) * 0.125
    keep = torch.ones(T, T, dtype=torch.bool, device=q.device).tril()
    return torch.softmax(s.masked_fill(~keep, float("-inf")), -1) @ v


def _heads(x, B, T, NH):
    return x.view(B, T, NH, 64).transpose(1, 2)


def _exact_train(case, t):
    B, T, L, NH = case["B"], case["T"], case["L"], case["NH"]
    C = NH * 64
    layout = _param_layout(case)
    flat = t["params"].double()
    p = {n: flat[o: o + math.prod(sh)].view(sh).requires_grad_() for n, o, sh in layout}
    tok, tgt = t["tok"].long(), t["tgt"].long()
    x = p["wte"].t()[tok] + p["wpe"][:T].repeat(B, 1)
    ln = torch.nn.functional.layer_norm
    for i in range(L):
        def q(n):
            return p[f"{i}.{n}"]
        h = ln(x, (C,), q("ln1_w"), q("ln1_b")) @ q("qkv_w") + q("qkv_b")
        a = _exact_attention(*(_heads(z, B, T, NH) for z in h.split(C, 1)))
        x = x + a.transpose(1, 2).reshape(B * T, C) @ q("proj_w") + q("proj_b")
        h = _gelu(ln(x, (C,), q("ln2_w"), q("ln2_b")) @ q("fc_w") + q("fc_b"))
        x = x + h @ q("fcproj_w") + q("fcproj_b")
    logits = (ln(x, (C,), p["lnf_w"], p["lnf_b"]) @ p["wte"])[:, : case["V"]]
    loss = torch.nn.functional.cross_entropy(logits, tgt)
    grads = torch.autograd.grad(loss, [p[n] for n, _, _ in layout])
    grad = torch.cat([z.reshape(-1) for z in grads])
    b1, b2, eps, wd = _HYPER
    lr = _PEAK_LR / _WARMUP_STEPS
    flat = flat.detach()
    step = grad / ((grad * grad).sqrt() + eps) + wd * flat  # first step: the bias corrections cancel the decay rates
    return {"grad": grad, "p": flat - lr * step}


def exact(case, seed):
    k = case["kind"]
    if k == "train" and case["B"] * case["T"] > 2048:
        return None
    t = _inputs(case, seed)
    if k == "train":
        return _exact_train(case, t)
    d = {n: (v.double() if v is not None and v.is_floating_point() else v) for n, v in t.items()}
    if k == "linear":
        out = {"y": d["x"] @ d["w"] + (d["b"] if case["bias"] else 0.0), "dx": d["dy"] @ d["w"].t(),
               "dw": d["x"].t() @ d["dy"]}
        if case["bias"]:
            out["db"] = d["dy"].sum(0)
        return out
    if k == "mlp":
        h = (d["x"] @ d["w1"] + d["b1"]).requires_grad_()
        act = _gelu(h)
        dact = d["dy"] @ d["w2"].t()
        (dh,) = torch.autograd.grad(act, h, dact)
        h, act = h.detach(), act.detach()
        return {"h": h, "act": act, "y": act @ d["w2"] + d["b2"] + d["res"], "dh": dh, "dw2": act.t() @ d["dy"],
                "db2": d["dy"].sum(0), "dx": dh @ d["w1"].t(), "dw1": d["x"].t() @ dh, "db1": dh.sum(0)}
    if k == "head":
        logits = d["x"] @ d["w"]
        lse = torch.logsumexp(logits[:, :_VOCAB], 1)
        loss = lse - logits.gather(1, t["tgt"].long()[:, None])[:, 0]
        return {"logits": logits, "loss": loss, "lse": lse * math.log2(math.e), "dx": d["dy"] @ d["w"].t(),
                "dw": d["x"].t() @ d["dy"]}
    B, T, NH = case["B"], case["T"], case["NH"]
    C = NH * 64
    outs, grads = [], []
    for b in range(B):  # a sequence at a time: T x T tensors in 64 bits are large
        rows = slice(b * T, (b + 1) * T)
        qkv = d["qkv"][rows].clone().requires_grad_()
        o = _exact_attention(*(_heads(z, 1, T, NH) for z in qkv.split(C, 1))).transpose(1, 2).reshape(T, C)
        (gq,) = torch.autograd.grad(o, qkv, d["dout"][rows])
        outs.append(o.detach())
        grads.append(gq)
    return {"out": torch.cat(outs), "dqkv": torch.cat(grads)}
