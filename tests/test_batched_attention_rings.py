"""The batched decode attention where a warp's two-stage ring turns over, from the 16-bit and from the 8-bit cache: sequences that end just
before, at and behind a multiple of 16 positions x warps, so that the new position's tile is a warp's first, its second or a later one, stages
are asked for again, and tiles, warps or whole parts are empty.  Six warps a CTA from 19 sequences on (148 SMs), twelve below; the keys of
an item in three parts (6 sequences), none (16, 19, 64) or four for the last ones (41).  Every sequence against the restatement."""
import pytest
import torch

from helpers import logit_report
from megaqwen_b200.spec import QWEN3_TINY
from megaqwen_b200.synthetic import random_prompt, random_weights
from test_kv_fp8 import FP8_MAX_TOL, FP8_MEAN_TOL

pytestmark = pytest.mark.gpu
MAX_SEQ, STEPS = 1344, [11, 407, 3021]
# from three tokens on: the 8-bit scale of a one-token prompt is that of a single row, whose last bit moves the whole grid of the next ones
LENS = [3, 14, 15, 16, 95, 96, 97, 190, 191, 192, 193, 382, 383, 384, 385, 577, 700, 1150, 1250]


@pytest.fixture(scope="module")
def model():
    w = random_weights(QWEN3_TINY, MAX_SEQ)
    e = w["embed_weight"].cuda()
    return w, (e, [t.cuda() for t in w["layer_weights"]], w["final_norm_weight"].cuda(), e, w["cos_table"].cuda(), w["sin_table"].cuda(), QWEN3_TINY.num_layers)


@pytest.fixture(scope="module")
def expected(model):
    """Logits of the forced steps behind a prompt of n tokens, made once per length and kind of cache."""
    from oracle.qwen3_restatement import RestatedQwen3
    seen = {}

    def get(n, fp8):
        if (n, fp8) not in seen:
            ref = RestatedQwen3(QWEN3_TINY, model[0], MAX_SEQ, kv_fp8=fp8)
            ref.forward(random_prompt(QWEN3_TINY, n, 51, n))
            seen[n, fp8] = [ref.forward([t]) for t in STEPS]
        return seen[n, fp8]

    return get


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("batch,split", [(6, True), (6, False), (16, True), (19, True), (41, True), (41, False), (64, True)])
def test_rings(model, expected, batch, split, fp8):
    from megaqwen_b200.batch import MegakernelBatchDecoder
    bd = MegakernelBatchDecoder(*model[1], MAX_SEQ, batch, 1250, kv_fp8=fp8)
    bd.use_split_kv = split
    lens = [LENS[(len(LENS) - 1 - i) % len(LENS)] for i in range(batch)]          # the longest are in every batch
    bd.prefill_batch([random_prompt(QWEN3_TINY, n, 51, n) for n in lens])
    most = {"max": FP8_MAX_TOL, "mean": FP8_MEAN_TOL} if fp8 else {"max": 6e-2, "mean": 8e-3}
    for step, t in enumerate(STEPS):
        _, lg = bd.decode_batch(torch.full((batch,), t, dtype=torch.int32), return_logits=True)
        lg = lg.cpu()
        for b, n in enumerate(lens):
            rep = logit_report(lg[b], expected(n, fp8)[step])
            assert rep["max"] <= most["max"] and rep["mean"] <= most["mean"], (n, step, rep)
    bd.check_status()
