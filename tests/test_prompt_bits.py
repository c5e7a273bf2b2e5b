"""A row's keys and values do not depend on how many rows are read with it, nor on the caller's scratch: below 512 rows every
sum over K is taken whole, in the order that prompts of more than 2048 rows have, whatever the tile.  (Between, O and down add two halves.)"""
import pytest
import torch

from megaqwen_b200.spec import QWEN3_TINY
from megaqwen_b200.synthetic import random_prompt, random_weights

pytestmark = pytest.mark.gpu
MAX_SEQ = 2100
FEW = [1, 2, 23, 63, 64, 65, 127]              # attention on mma.sync
MORE = [128, 129, 256, 257, 384, 385, 511]     # on tcgen05


@pytest.fixture(scope="module")
def args():
    w = random_weights(QWEN3_TINY, MAX_SEQ)
    e = w["embed_weight"].cuda()
    return (e, [t.cuda() for t in w["layer_weights"]], w["final_norm_weight"].cuda(), e, w["cos_table"].cuda(), w["sin_table"].cuda(), QWEN3_TINY.num_layers)


@pytest.fixture(scope="module")
def rows(args):
    """The rows that the first n tokens of one prompt leave in both caches, per n."""
    from megaqwen_b200.decoder import MegakernelDecoder
    dec = MegakernelDecoder(*args, MAX_SEQ, MAX_SEQ)
    p = random_prompt(QWEN3_TINY, MAX_SEQ, 41, 0)
    out = {}
    for n in FEW + MORE + [MAX_SEQ]:
        dec.reset()
        dec.prefill_step(p[:n])
        out[n] = torch.stack([dec.get_k_cache()[:, :, :n], dec.get_v_cache()[:, :, :n]]).clone()
    return p, out


@pytest.mark.parametrize("n", FEW + MORE)
def test_first_token(rows, n):
    """All layers: the first token's attention is its own value row, exactly, in either kernel, so only the linears count."""
    _, got = rows
    assert torch.equal(got[n][:, :, :, 0], got[MAX_SEQ][:, :, :, 0])


@pytest.mark.parametrize("n", FEW + MORE)
def test_first_layer(rows, n):
    _, got = rows
    assert torch.equal(got[n][:, 0], got[MAX_SEQ][:, 0, :, :n])


@pytest.mark.parametrize("n,of", [(n, FEW[-1]) for n in FEW[:-1]] + [(n, MORE[-1]) for n in MORE[:-1]])
def test_all_layers(rows, n, of):
    _, got = rows
    assert torch.equal(got[n], got[of][:, :, :, :n])


@pytest.mark.parametrize("n", FEW + MORE)
def test_without_scratch(args, rows, n):
    """The batch decoder reads a prompt alone without the decode path's scratch."""
    from megaqwen_b200.batch import MegakernelBatchDecoder
    p, got = rows
    bd = MegakernelBatchDecoder(*args, 600, 1, 600)
    bd.prefill_batch([p[:n]])
    assert torch.equal(bd.get_k_cache()[0, :, :, :n], got[n][0]) and torch.equal(bd.get_v_cache()[0, :, :, :n], got[n][1])
