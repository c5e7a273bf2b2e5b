"""The 32-bit products of several tokens add their terms one after the other, first k to last, whatever the tile: bit for bit what plain
32-bit additions on the host give.  The model's layers add nothing to a constant embedding, so the head multiplies one constant by
weights that are powers of two: every product is exact and only the order of the additions shows."""
import numpy as np
import pytest
import torch

import hybrid_models as hm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,vocab", [(16, 33), (48, 331), (64, 64), (80, 500), (112, 130), (1040, 331)])
def test_order_of_the_sums(width, vocab):
    from megaqwen_b200.hybrid import HybridDecoder
    cfg = hm.config([(hm.lightning(2, 16, 16), 32)], width=width, vocab=vocab, embed_scale=1.0)
    w = hm.weights(cfg)
    g = torch.Generator().manual_seed(width)
    for name, t in w["tensors"].items():
        if name.endswith(("mix.o", "mlp.down", "final.norm")):
            t.zero_()
        elif name == "embed":
            t.fill_(3.0)
        elif name == "head":
            t.copy_(torch.exp2(torch.randint(-12, 13, t.shape, generator=g).float()) * (torch.randint(0, 2, t.shape, generator=g) * 2 - 1))
            t[0] = 0.0
            t[0, 0] = 1.0                                            # its logit is the constant itself
    head = w["tensors"]["head"].float().numpy()
    dec = HybridDecoder(w, 160, 160, dtype="float32")
    want = None
    for n in (2, 8, 9, 16, 17, 96, 97, 128, 129, 150):               # one row alone is a step's; the edges of the tiles and of their rules
        dec.reset()
        got = dec.step_logits(hm.tokens(cfg, n), list(range(n))).cpu().numpy()
        if want is None:
            v, want = got[0, 0], np.zeros(vocab, np.float32)
            for k in range(width):
                want = want + v * head[:, k]
            assert abs(v - 1) < 1e-5 and want.dtype == np.float32
            assert not np.array_equal(want, (v * head).sum(1, dtype=np.float64).astype(np.float32))      # the order shows
        assert np.array_equal(got, np.broadcast_to(want, got.shape)), n
