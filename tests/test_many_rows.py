"""Prompts of many rows: the linears on pairs of SMs at the row counts where they take over and at the edges of their 256-row
tiles, and the tcgen05 attention over several packed prompts at the edges of its 128-row tiles."""
import pytest
import torch

from megaqwen_b200.spec import QWEN3_TINY
from megaqwen_b200.synthetic import random_prompt, random_weights

pytestmark = pytest.mark.gpu
MAX_SEQ = 2600


@pytest.fixture(scope="module")
def args():
    w = random_weights(QWEN3_TINY, MAX_SEQ)
    e = w["embed_weight"].cuda()
    return (e, [t.cuda() for t in w["layer_weights"]], w["final_norm_weight"].cuda(), e, w["cos_table"].cuda(), w["sin_table"].cuda(), QWEN3_TINY.num_layers)


@pytest.mark.parametrize("rows", [1025, 1152, 1153, 1280, 1281, 2048, 2304, 2305, 2560, 2561])
def test_whole_prompt_against_portions(args, rows):
    """The same prompt in two or three portions of 513 to 900 rows, which take the tiles of one SM.  The first layer's keys and values come from the
    same sums in the same order; behind it the attention walks its key tiles from other query tiles and two bf16
    computations differ by their roundings: values of the size of one, two spacings at [4, 8) at most."""
    from megaqwen_b200.decoder import MegakernelDecoder
    dec = MegakernelDecoder(*args, MAX_SEQ, MAX_SEQ)
    p = random_prompt(QWEN3_TINY, rows, 31, rows)
    tok, lg = dec.prefill_step_logits(p)
    k, v = dec.get_k_cache().clone(), dec.get_v_cache().clone()
    dec.reset()
    parts = torch.tensor_split(p, (rows + 899) // 900)
    dec.prefill_step(parts[0])
    for part in parts[1:]:
        other = dec.prefill_append(part)
    for x, y in ((k, dec.get_k_cache()), (v, dec.get_v_cache())):
        assert torch.equal(x[0], y[0])
        assert float((x.float() - y.float()).abs().max()) <= 2 ** -4
    assert bool(torch.isfinite(lg).all())
    assert tok == other or float(lg[tok] - lg[other]) <= 6e-2


@pytest.mark.parametrize("rows", [129, 256, 257, 384, 385, 511, 512, 513, 768, 769, 1000, 1024])
def test_prompt_against_portions_of_few_rows(args, rows):
    """Every choice of tiles up to 1024 rows against portions of at most 128 rows, whose attention walks its keys in other tiles: two
    bf16 computations that differ by their roundings, two spacings at [4, 8) at most."""
    from megaqwen_b200.decoder import MegakernelDecoder
    dec = MegakernelDecoder(*args, MAX_SEQ, MAX_SEQ)
    p = random_prompt(QWEN3_TINY, rows, 33, rows)
    tok, lg = dec.prefill_step_logits(p)
    k, v = dec.get_k_cache().clone(), dec.get_v_cache().clone()
    dec.reset()
    parts = torch.tensor_split(p, (rows + 127) // 128)
    other = dec.prefill_step(parts[0])
    for part in parts[1:]:
        other = dec.prefill_append(part)
    for x, y in ((k, dec.get_k_cache()), (v, dec.get_v_cache())):
        assert float((x.float() - y.float()).abs().max()) <= 2 ** -4
        assert float((x.float() - y.float()).abs().mean()) <= 4e-3
    assert bool(torch.isfinite(lg).all())
    assert tok == other or float(lg[tok] - lg[other]) <= 6e-2


def test_packed_prompts_against_one_by_one(args):
    """Every prompt's bits are those of a pass of its own, whatever the cache holds behind it and however many rows the pass has."""
    from megaqwen_b200.batch import MegakernelBatchDecoder
    lens = [1, 63, 64, 65, 127, 128, 129, 255, 256, 257, 400, 511, 190]
    bd = MegakernelBatchDecoder(*args, 600, len(lens), 600)
    prompts = [random_prompt(QWEN3_TINY, n, 32, i) for i, n in enumerate(lens)]

    def run(packed, cap=None):
        bd.reset()
        for c in (bd.get_k_cache(), bd.get_v_cache()):
            c.fill_(float("nan"))
        bd.use_packed_prefill = packed
        keep = bd._pf.max_tokens
        bd._pf.max_tokens = cap or keep
        out = bd.prefill_batch(prompts).tolist()
        bd._pf.max_tokens = keep
        bd.check_status()
        return out, [(bd.get_k_cache()[i, :, :, :n].clone(), bd.get_v_cache()[i, :, :, :n].clone()) for i, n in enumerate(lens)]

    assert sum(lens) > 18 * 128 and bd._pf.max_tokens >= sum(lens)
    want, rows = run(False)
    for cap in (None, 1200, 700):
        got, caches = run(True, cap)
        assert got == want
        for (k, v), (k1, v1) in zip(rows, caches):
            assert bool(torch.isfinite(k).all()) and torch.equal(k, k1) and torch.equal(v, v1)


def test_layer_listed_prompt_against_portions():
    """A layer-listed model whose input projections take pairs of SMs at 1300 rows and not at 325: the same prompt whole and in portions.
    Both sides differ from 64 bits by at most 0.04 in any position's logits (the parity tests' bound), so by 0.08 from each other."""
    import hybrid_models as hm
    from megaqwen_b200.hybrid import HybridDecoder
    cfg = hm.config([hm.lightning(16, 128, 128), hm.latent(16, 128, 64, 128, 512)], width=1024, ff=3072, mult=0.2)
    dec = HybridDecoder(hm.weights(cfg, 3), 1400, 1400, dtype="bfloat16")
    ids = hm.tokens(cfg, 1300, 4)
    places = [0, 255, 256, 700, 1299]
    whole = dec.step_logits(ids, places)
    dec.reset()
    rows = []
    for i in range(0, 1300, 325):
        rows.append(dec.step_logits(ids[i:i + 325], [p - i for p in places if i <= p < i + 325]))
    e = hm.errors(whole, torch.cat([r.cpu() for r in rows if r.numel()]))
    assert float(e.max()) <= 0.08, e
