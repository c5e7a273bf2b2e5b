"""Few rows against the restatement: prompts of up to 128 tokens, and the cluster chain of a batch's steps at the edges of its
operand widths (16, 32, 64 rows) and of the shares that the CTAs of a cluster finish."""
import pytest
import torch

from helpers import assert_logits_close
from megaqwen_b200.spec import QWEN3_TINY
from megaqwen_b200.synthetic import random_prompt, random_weights

pytestmark = pytest.mark.gpu
MAX_SEQ = 384


@pytest.fixture(scope="module")
def tiny():
    from megaqwen_b200.decoder import MegakernelDecoder
    from oracle.qwen3_restatement import RestatedQwen3
    w = random_weights(QWEN3_TINY, MAX_SEQ)
    g = torch.Generator().manual_seed(3)
    for i, t in enumerate(w["layer_weights"]):
        if t.dim() == 1:                                     # norm weights that differ from column to column
            w["layer_weights"][i] = (1.0 + 0.2 * torch.randn(t.shape, generator=g)).to(torch.bfloat16)
    e = w["embed_weight"].cuda()
    args = (e, [t.cuda() for t in w["layer_weights"]], w["final_norm_weight"].cuda(), e, w["cos_table"].cuda(), w["sin_table"].cuda(), QWEN3_TINY.num_layers)
    return MegakernelDecoder(*args, MAX_SEQ, MAX_SEQ), args, RestatedQwen3(QWEN3_TINY, w, MAX_SEQ), w


def check_cache(got, want, rows, tol=2 ** -4):
    """bf16 values of the size of one: two spacings at [4, 8)."""
    assert float((got[:, :, :rows].float().cpu() - want[:, :, :rows].float()).abs().max()) <= tol


@pytest.mark.parametrize("rows", [1, 2, 3, 15, 16, 17, 31, 32, 33, 63, 64, 65, 96, 127, 128])
def test_prompts_of_few_rows(tiny, rows):
    """A prompt, then a second one of as many rows appended to it."""
    dec, _, ref, _ = tiny
    dec.reset()
    ref.reset()
    a, b = random_prompt(QWEN3_TINY, rows, 21, rows), random_prompt(QWEN3_TINY, rows, 22, rows)
    _, lg = dec.prefill_step_logits(a)
    assert_logits_close(lg.cpu(), ref.forward(a), rows)
    _, lg = dec.prefill_step_logits(b, append=True)
    assert_logits_close(lg.cpu(), ref.forward(b), rows)
    check_cache(dec.get_k_cache(), ref.k_cache, 2 * rows)
    check_cache(dec.get_v_cache(), ref.v_cache, 2 * rows)
    assert float(dec.get_k_cache()[:, :, 2 * rows:].abs().max()) == 0.0 if 2 * rows < MAX_SEQ else True


@pytest.mark.parametrize("batch", [1, 2, 15, 17, 32, 33, 64])
def test_batches_of_few_rows(tiny, batch):
    """One step of a batch whose sequences stand at different positions; a few of them against the restatement."""
    from megaqwen_b200.batch import MegakernelBatchDecoder
    _, args, ref, _ = tiny
    bd = MegakernelBatchDecoder(*args, MAX_SEQ, batch, 40)
    prompts = [random_prompt(QWEN3_TINY, 1 + (7 * i) % 40, 23, i) for i in range(batch)]
    bd.prefill_batch(prompts)
    cur = [int(p[0]) for p in prompts]
    _, lg = bd.decode_batch(torch.tensor(cur, dtype=torch.int32), return_logits=True)
    for b in sorted({0, 1 % batch, batch // 2, batch - 1}):
        ref.reset()
        ref.forward(prompts[b])
        assert_logits_close(lg[b].cpu(), ref.forward([cur[b]]), (batch, b))
        n = int(prompts[b].numel()) + 1
        check_cache(bd.get_k_cache()[b], ref.k_cache, n)
        check_cache(bd.get_v_cache()[b], ref.v_cache, n)
    bd.check_status()
