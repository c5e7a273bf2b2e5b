"""The launches that a call says it makes are the kernels that a capture of it holds."""
import ctypes as C

import pytest
import torch

from megaqwen_b200 import _lib
from megaqwen_b200.spec import QWEN3_TINY
from megaqwen_b200.synthetic import random_prompt, random_weights

pytestmark = pytest.mark.gpu
MAX_SEQ = 2400


def nodes(call):
    """Kernels that ``call`` puts on the current stream."""
    torch.cuda.synchronize()
    g, s = torch.cuda.CUDAGraph(keep_graph=True), torch.cuda.Stream()
    with torch.cuda.stream(s):
        with torch.cuda.graph(g, stream=s):
            call()
    n = C.c_size_t(0)
    assert C.CDLL("libcudart.so.12").cudaGraphGetNodes(C.c_void_p(g.raw_cuda_graph()), None, C.byref(n)) == 0
    return n.value


@pytest.fixture(scope="module")
def args():
    w = random_weights(QWEN3_TINY, MAX_SEQ)
    e = w["embed_weight"].cuda()
    return (e, [t.cuda() for t in w["layer_weights"]], w["final_norm_weight"].cuda(), e, w["cos_table"].cuda(), w["sin_table"].cuda(), QWEN3_TINY.num_layers, MAX_SEQ)


@pytest.mark.parametrize("rows", [1, 127, 128, 511, 512, 513, 1024, 1025, 1152, 1153, 2048, 2049])
def test_prompts(args, rows):
    from megaqwen_b200.decoder import MegakernelDecoder
    dec = MegakernelDecoder(*args, MAX_SEQ)
    ids = random_prompt(QWEN3_TINY, rows, 61, rows)
    before = dec.launches
    dec.prefill_step(ids)
    dev = ids.cuda()
    got = nodes(lambda: _lib.check(dec._lib.mq_launch_prefill(C.byref(dec._model), C.byref(dec._buf), C.byref(dec._pf), dev.data_ptr(), rows, 0,
                                                              dec._scalars.data_ptr(), None, dec._stream()), "prefill"))
    assert got == dec.launches - before


@pytest.mark.parametrize("batch,splitk", [(1, True), (64, True), (64, False), (65, True)])
def test_steps_of_a_batch(args, batch, splitk):
    from megaqwen_b200.batch import MegakernelBatchDecoder
    bd = MegakernelBatchDecoder(*args[:7], 128, batch, 16)
    bd.use_splitk = splitk
    cur = bd.prefill_batch([random_prompt(QWEN3_TINY, 3 + i % 9, 62, i) for i in range(batch)])
    before = bd.launches
    bd.decode_batch(cur)
    step = bd.launches - before
    tin, out = cur.cuda(), torch.empty(batch, dtype=torch.int32, device="cuda")
    assert nodes(lambda: bd._step(tin.data_ptr(), out.data_ptr())) == step


@pytest.mark.parametrize("lens", [[3, 5], [400, 200], [900, 300]])
def test_packed_prompts(args, lens):
    from megaqwen_b200.batch import MegakernelBatchDecoder
    bd = MegakernelBatchDecoder(*args[:7], 1024, len(lens), 1000)
    prompts = [random_prompt(QWEN3_TINY, n, 63, n) for n in lens]
    before = bd.launches
    bd.prefill_batch(prompts)
    said = bd.launches - before
    lib, calls = bd._lib, []

    class Recorder:                                    # the arguments of the packed call
        def __getattr__(self, name):
            return getattr(lib, name)

        def mq_launch_prefill_packed(self, *a):
            calls.append(a)
            return lib.mq_launch_prefill_packed(*a)

    bd._lib = Recorder()
    bd.prefill_batch(prompts)
    assert len(calls) == 1
    assert nodes(lambda: _lib.check(lib.mq_launch_prefill_packed(*calls[0][:-1], bd._stream()), "packed")) == said
