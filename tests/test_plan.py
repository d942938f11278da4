"""The automatic choices of a linear-layer call (CTA pairs, tile width, splits), planned for 148 SMs without a GPU."""
import os
import random
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
LIBDIR = os.path.join(ROOT, "gpt2.cu_b200", "lib")


@pytest.fixture(scope="module")
def plan_dump(built, tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("plan") / "plan_dump")
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    r = subprocess.run([nvcc, "-std=c++17", "-I", os.path.join(ROOT, "include"), "-I", os.path.join(ROOT, "gpt2.cu_b200", "csrc"),
                        os.path.join(ROOT, "tests", "plan_dump.cpp"), "-o", exe, "-L", LIBDIR, "-lgpt2_linear",
                        f"-Xlinker=-rpath={LIBDIR}"], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    return exe


def _lines(command, rows):
    text = "\n".join(" ".join(map(str, r)) for r in rows) + "\n"
    out = subprocess.run(command, input=text, capture_output=True, text=True, check=True).stdout
    return [tuple(map(int, line.split())) for line in out.splitlines()]


@pytest.fixture(scope="module")
def plans(plan_dump):
    def run(calls):
        """calls: dicts of mode, kind, M, K, N and options -> one dict per call"""
        fields = ("mode", "kind", "M", "K", "N", "split", "pair", "det", "aux", "gelu", "stats")
        rows = _lines([plan_dump], [[c.get(f, 0) for f in fields] for c in calls])
        return [dict(zip(("err", "pair", "bn", "splits", "per", "tiles_n"), r)) for r in rows]

    return run


FORWARD, BACKWARD_INPUT, BACKWARD_WEIGHT = 0, 1, 2


@pytest.mark.parametrize("mode", [0, 1])
def test_narrow_outputs_keep_their_reduction_split(plans, mode):
    deep = dict(mode=mode, kind=BACKWARD_WEIGHT, M=16384, K=5120, N=64)
    deeper = dict(deep, K=768)
    asked = dict(deep, split=7)
    for p, at_least in zip(plans([deep, deeper, asked]), (7, 24, 7)):
        assert p["err"] == 0 and p["pair"] == 0 and p["bn"] == 64 and p["splits"] >= at_least
    # a caller who asks for pairs gets their narrowest tile, split as asked or as the rows need it
    (p, q) = plans([dict(asked, pair=2), dict(deeper, pair=2)])
    assert p["pair"] == q["pair"] == 1 and p["bn"] == q["bn"] == 128
    assert p["splits"] == 7 and q["splits"] > 8


def test_pairs_where_they_stage_less(plans):
    rows = 8192
    calls = [dict(mode=1, kind=k, M=rows, K=a, N=b) for k in range(3) for a, b in ((768, 3072), (3072, 768), (768, 2304))]
    calls += [dict(mode=0, kind=k, M=rows, K=768, N=n) for k in range(3) for n in (3072, 50304)]
    assert all(p["pair"] == 1 and p["bn"] == 256 for p in plans(calls))
    # 128 rows leave half of a pair's tile empty; 100 columns more than half of one; two k-blocks are all hand-shake
    calls = [dict(mode=1, kind=BACKWARD_INPUT, M=128, K=3212, N=11824), dict(mode=1, kind=BACKWARD_INPUT, M=1936, K=100, N=14408),
             dict(mode=1, kind=FORWARD, M=12668, K=64, N=5772)]
    assert all(p["pair"] == 0 for p in plans(calls))


def test_pairs_sum_no_longer_chains_in_3xtf32(plans):
    """the accumulation bounds this mode's error, so the choice that is left open never lengthens it"""
    rng = random.Random(3)
    calls = [dict(mode=1, kind=FORWARD, M=3620, K=4724, N=860), dict(mode=1, kind=BACKWARD_WEIGHT, M=4320, K=1096, N=3200)]
    calls += [dict(mode=1, kind=rng.randrange(3), **{k: 4 * round(2 ** rng.uniform(4, 12)) for k in "MKN"}) for _ in range(3000)]
    chosen, single = plans(calls), plans([dict(c, pair=1) for c in calls])
    assert sum(p["pair"] for p in chosen) > 500
    assert all(p["per"] <= q["per"] for p, q in zip(chosen, single))


@pytest.mark.parametrize("max_parts", [1, 2, 4, 8, 16])
def test_cuda_core_splits_fit_the_device(plan_dump, max_parts):
    """no more parts than the largest cluster the device can place, none of them empty, nothing left out"""
    rng = random.Random(5)
    shapes = [(768, 256, 50257), (1, 1, 1)] + [tuple(round(2 ** rng.uniform(0, 15)) for _ in range(3)) for _ in range(500)]
    plans = _lines([plan_dump, "simt"], [s + (max_parts,) for s in shapes])
    for (_, _, depth), (bm, bn, parts, per) in zip(shapes, plans):
        assert 1 <= parts <= max_parts and per % 16 == 0 and (bm, bn) in ((128, 128), (128, 64), (64, 64))
        assert per * (parts - 1) < depth <= per * parts
    assert plans[0][2] == max_parts  # 12 or 24 tiles, 50257 deep: as many parts as there may be


def test_fp32_attention_covers_every_sequence_length(plan_dump):
    """every 64-row tile in one launch or, past the 65535 of a grid's third dimension, in several"""
    lengths = [1, 64, 65, 65535 * 64, 65535 * 64 + 1, (1 << 31) - 1]
    for T, launches in zip(lengths, _lines([plan_dump, "attention"], [(T,) for T in lengths])):
        assert sum(launches) == -(-T // 64) and max(launches) <= 65535 and all(n == 65535 for n in launches[:-1])
