"""A bounded wait that runs out (a load that is never requested): the kernel returns, sets the status bit, stores nothing of what it
could not compute, and the next call is right."""
import pytest
import torch

from megaqwen_b200 import _lib
from megaqwen_b200.spec import QWEN3_TINY
from megaqwen_b200.synthetic import random_weights

pytestmark = pytest.mark.gpu
QKV, O, GATE_UP, DOWN = range(4)
CTAS = {QKV: 4, O: 8, GATE_UP: 4, DOWN: 8}           # of a cluster, and blocks of 64 columns each of them has
BLOCKS = {QKV: 4, O: 4, GATE_UP: 4, DOWN: 6}


@pytest.mark.parametrize("which", [QKV, O, GATE_UP, DOWN])
@pytest.mark.parametrize("batch", [3, 17, 64])
def test_chain_of_a_batch(which, batch):
    from megaqwen_b200.batch import MegakernelBatchDecoder
    w = random_weights(QWEN3_TINY, 64)
    e = w["embed_weight"].cuda()
    bd = MegakernelBatchDecoder(e, [t.cuda() for t in w["layer_weights"]], w["final_norm_weight"].cuda(), e, w["cos_table"].cuda(),
                                w["sin_table"].cuda(), QWEN3_TINY.num_layers, 64, batch, 16)
    g = torch.Generator(device="cuda").manual_seed(batch)
    for t in bd._act:
        t.copy_(torch.randn(t.shape, generator=g, device="cuda"))
    bd._partials[:8 * batch] = bd._act[0][:batch].float().pow(2).reshape(batch, 8, 128).sum(-1).reshape(-1)
    bd._positions.copy_(torch.arange(batch) % 60)
    state = [*bd._act, bd.k_cache_, bd.v_cache_, bd._partials]
    start = [t.clone() for t in state]

    def run(drop):
        for t, s in zip(state, start):
            t.copy_(s)
        bd._scalars.zero_()
        rc = bd._lib.mq_debug_chain_drop_load(_lib.C.byref(bd._model), _lib.C.byref(bd._bb(batch)), which, drop, bd._stream())
        _lib.check(rc, "mq_debug_chain_drop_load")
        torch.cuda.synchronize()
        return int(bd._scalars[1])

    assert run(-1) == 0
    right = [t.clone() for t in state]
    assert not all(torch.equal(t, s) for t, s in zip(right, start))
    for drop in (0, 16 * (CTAS[which] - 1) + BLOCKS[which] - 1):
        assert run(drop) == _lib.MQ_STATUS_WAIT_TIMEOUT
        assert all(torch.equal(t, s) for t, s in zip(state, start)), drop
        assert run(-1) == 0
        assert all(torch.equal(t, s) for t, s in zip(state, right)), drop
