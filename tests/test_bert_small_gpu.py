"""The encoder's one-launch kernel (up to 64 tokens per cluster of blocks) against the oracle, at the edges of its row tiles and clusters."""
import numpy as np
import pytest

from oracle import bert as obert
from oracle import synth

import test_bert_gpu as B

pytestmark = pytest.mark.gpu


# one token; a row tile and a row on both sides of it; the most tokens of a cluster, one cluster and six (148 SMs hold at least as many); several sentences per
# cluster with a last one that holds fewer; more sentences than clusters; one token or one sentence too many (the launch chain)
@pytest.mark.parametrize("b,t", [(1, 1), (1, 16), (1, 17), (1, 33), (1, 64), (6, 64), (3, 21), (8, 64), (9, 30), (20, 5), (37, 7), (256, 2), (1, 65), (40, 40)])
def test_short_sentences(b, t):
    cfg = obert.MINILM_L6
    w = obert.synth_weights(cfg, 0, 0.02)
    m = B._product(cfg, w)
    ids = synth.token_ids(500 + t, cfg.vocab_size, (b, t))
    mask = np.ones((b, t), dtype=np.uint32)
    mask[1:, -(t // 3):] = 0 if t >= 3 else 1
    for k in (None, mask):
        want, got = obert.MiniLM(cfg, w).embed_ids(ids, k), m.embed_ids(ids, k)
        assert B._cos(got, want).min() >= B.COS_TOL and np.abs(got - want).max() <= 2e-2
    # a sentence's embedding is that of the sentence alone, beyond the order of sums
    alone = m.embed_ids(ids[-1:])
    assert B._cos(alone, m.embed_ids(ids)[-1:]).min() >= B.COS_TOL


@pytest.mark.parametrize("t", [1, 2, 5, 15, 16, 17, 19, 32, 33, 48, 49, 64])
def test_same_bits_as_the_launch_chain(t):
    """a sentence comes out the same whether it is embedded with few others (one launch) or in a batch that takes the chain: every sum of the
    one-launch kernel runs in the chain's order"""
    cfg = obert.MINILM_L6
    w = obert.synth_weights(cfg, 0, 0.02)
    m = B._product(cfg, w)
    b = 16 * (64 // t + 1)              # more than 64 tokens for each of up to 16 clusters (148 SMs hold seven to nine)
    ids = synth.token_ids(700 + t, cfg.vocab_size, (b, t))
    mask = np.ones((b, t), dtype=np.uint32)
    mask[1::3, -(t // 3):] = 0 if t >= 3 else 1
    for k in (None, mask):
        whole = m.embed_ids(ids, k)
        for few in (1, 2, 6, 9, min(b, 6 * (64 // t)), min(b, 9 * (64 // t))):
            assert np.array_equal(m.embed_ids(ids[:few], None if k is None else k[:few]), whole[:few])
            assert np.array_equal(m.embed_ids(ids[-few:], None if k is None else k[-few:]), whole[-few:])
