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


@pytest.mark.parametrize("m,k,drop,whole", [(300, 1024, 0, 0), (300, 1024, 9, 0), (300, 128, 1, 0), (256 * 80, 128, 3, 74), (256 * 80, 1024, 31, 74)])
def test_gemm_on_pairs(m, k, drop, whole):
    """``whole``: 256-row tiles ahead of the first one that lacks a block, on 74 pairs of SMs (the last two cases drop a block of a pair's second tile)."""
    lib = _lib.lib()
    g = torch.Generator(device="cuda").manual_seed(m + k)
    a, b, r = (torch.randn(s, generator=g, device="cuda", dtype=torch.bfloat16) for s in ((m, k), (256, k), (m, 256)))
    status = torch.zeros(1, dtype=torch.int32, device="cuda")

    def run(drop_kb, before=0):
        c = torch.full((m, 256), 7.0, dtype=torch.bfloat16, device="cuda")
        status.fill_(before)
        rc = lib.mq_debug_gemm_pair_drop_load(a.data_ptr(), k, b.data_ptr(), c.data_ptr(), r.data_ptr(), m, 256, k, 256, status.data_ptr(),
                                              torch.cuda.current_stream().cuda_stream, drop_kb)
        _lib.check(rc, "mq_debug_gemm_pair_drop_load")
        torch.cuda.synchronize()
        return c, int(status)

    right, st = run(-1)
    ref = (a.float() @ b.float().T).bfloat16().float() + r.float()
    assert st == 0 and float((right.float() - ref).abs().max()) <= 2 ** -7 * float(ref.abs().max())
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        whole = 0 if whole == 0 else None
    c, st = run(drop)
    assert st == _lib.MQ_STATUS_WAIT_TIMEOUT
    if whole is not None:
        assert torch.equal(c[:256 * whole], right[:256 * whole]) and bool((c[256 * whole:] == 7.0).all())
    again, st = run(-1)
    assert st == 0 and torch.equal(again, right)
    for _ in range(20):                                # behind an expired wait every wait gives up after a few polls: whatever is in flight ends first
        run(-1, _lib.MQ_STATUS_WAIT_TIMEOUT)
        again, st = run(-1)
        assert st == 0 and torch.equal(again, right)
