"""The 32-bit products of several tokens add their terms one after the other, first k to last, whatever the tile, those of one token
along the lanes of a warp: bit for bit what plain 32-bit additions on the host give.  The model's layers add nothing to a constant embedding, so
the head multiplies one constant by weights that are powers of two: every product is exact and only the order of the additions shows."""
import numpy as np
import pytest
import torch

import hybrid_models as hm

pytestmark = pytest.mark.gpu


def powers_of_two(width, vocab):
    """(weights, head [vocab, width]): final hidden states of one value, head rows of powers of two with either sign; row 0 gives the value."""
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
            t[0, 0] = 1.0
    return cfg, w, w["tensors"]["head"].float().numpy()


@pytest.mark.parametrize("width,vocab", [(16, 33), (48, 331), (64, 64), (80, 500), (112, 130), (1040, 331)])
def test_order_of_the_sums(width, vocab):
    from megaqwen_b200.hybrid import HybridDecoder
    cfg, w, head = powers_of_two(width, vocab)
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


@pytest.mark.parametrize("width,vocab", [(16, 33), (112, 331), (512, 2001), (528, 130), (1040, 5003), (2064, 2501)])
def test_order_of_a_steps_sums(width, vocab):
    """One token: columns below, at and above a ring slot's 512, an odd number of rows, one CTA per SM and (the last two) two."""
    from megaqwen_b200.hybrid import HybridDecoder
    cfg, w, head = powers_of_two(width, vocab)
    dec = HybridDecoder(w, 8, 8, dtype="float32")
    got = dec.step_logits([1], [0])[0].cpu().numpy()
    v = got[0]
    wide = np.zeros((vocab, (width + 127) // 128 * 128), np.float32)
    wide[:, :width] = head
    lanes = np.zeros((vocab, 32), np.float32)
    for k in range(0, wide.shape[1], 128):                           # a lane has four columns of every 128, the last of them first
        for c in (3, 2, 1, 0):
            lanes = lanes + v * wide[:, k + c:k + 128:4]
    for o in (16, 8, 4, 2, 1):
        lanes = lanes + lanes[:, np.arange(32) ^ o]
    assert abs(v - 1) < 1e-5 and np.array_equal(got, lanes[:, 0])
