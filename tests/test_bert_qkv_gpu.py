"""The kernel of q|k|v and attention (bert_qkv.cuh), which sentences of up to 128 tokens take, at the edges of its groups of sentences, of its 16-row and
16-key tiles and of its pairs of SMs, against the oracle."""
from pathlib import Path

import numpy as np
import pytest

from oracle import bert as obert
from oracle import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def encoder():
    from fastllm_b200 import models
    cfg = obert.BertConfig(384, 12, 2, 1536, 128, 1e-12, 512)
    w = obert.synth_weights(cfg, 11, 0.06)
    return cfg, obert.MiniLM(cfg, w), models.MiniLMModel(models.BertConfig(384, 12, 2, 1536, 128, 1e-12, 512), w, 0)


# a whole tile, one row less; two sentences a group and one; rows of a tile left over (43: 42 of 128; 25: three); sentences within a 16-row tile; an odd
# number of groups; runs of one to four heads, four as three and one (76 x 43: a pair of groups ends behind every third run; 41 x 128) or as two and two (38 x 85);
# longer runs that begin and end inside a pair's; the two kernels' route (38 x 70)
@pytest.mark.parametrize("b,t", [(1, 128), (2, 127), (37, 128), (19, 64), (21, 63), (10, 65), (36, 65), (31, 43), (33, 25), (70, 17), (75, 16), (150, 8), (223, 5), (700, 1), (300, 113),
                                 (152, 64), (41, 128), (76, 43), (38, 85), (38, 70)])
def test_against_the_oracle(encoder, b, t):
    """bf16 operands: 2^-9 of a value per rounding, four roundings between sums of hundreds per layer; a misplaced row, head or key is a cosine below 0.9"""
    cfg, oracle, model = encoder
    ids = synth.token_ids(1000 + b * 131 + t, cfg.vocab_size, (b, t))
    picked = sorted({0, 1 % b, b // 2, b - 2 if b > 1 else 0, b - 1})
    got, want = model.embed_ids(ids)[picked], oracle.embed_ids(ids[picked])
    cos = (got * want).sum(1) / (np.linalg.norm(got, axis=1) * np.linalg.norm(want, axis=1))
    assert cos.min() >= 0.999 and np.abs(got - want).max() <= 2e-2


@pytest.mark.parametrize("b,t", [(60, 20), (200, 7), (41, 50), (10, 127)])
def test_sentences_do_not_see_each_other(encoder, b, t):
    """another sentence in its place leaves the neighbours in its tile as they are, to the bit"""
    cfg, _, model = encoder
    ids = synth.token_ids(7, cfg.vocab_size, (b, t))
    before = model.embed_ids(ids)
    ids[b // 2] = synth.token_ids(8, cfg.vocab_size, (t,))
    after = model.embed_ids(ids)
    others = np.arange(b) != b // 2
    assert np.array_equal(after[others], before[others]) and not np.array_equal(after[b // 2], before[b // 2])


@pytest.mark.parametrize("b,t", [(1, 64), (2, 127), (31, 43), (75, 16), (223, 5), (300, 113), (50, 70), (38, 70), (256, 128)])
def test_same_bits_as_gemm_and_attention_kernel(encoder, b, t):
    """golden/bert_attention_bits.npz holds what these sentences gave (first, middle, last) when the q|k|v GEMM and bert_attn_kernel took them: the kernels
    that attend on the chip (one sentence of 64 tokens: the one-launch kernel) run every sum and every rounding in that order"""
    cfg, _, model = encoder
    ids = synth.token_ids(1000 + b * 131 + t, cfg.vocab_size, (b, t))
    want = np.load(Path(__file__).parent / "golden" / "bert_attention_bits.npz")[f"{b}x{t}"]
    assert np.array_equal(model.embed_ids(ids)[sorted({0, b // 2, b - 1})], want)


def test_only_the_buffers_of_a_route():
    """256 x 128 tokens: x and ctx are 25 MB each; q|k|v, which stay on the chip, would be 75 MB more.  A repeat finds every buffer of its route, whatever calls came before"""
    import torch
    from fastllm_b200 import models
    model = models.MiniLMModel(models.BertConfig(), None, 0, random_seed=3)
    ids = np.random.default_rng(1).integers(3, 30000, (256, 128)).astype(np.uint32)
    free = torch.cuda.mem_get_info()[0]
    model.embed_ids(ids)
    assert free - torch.cuda.mem_get_info()[0] < 70 << 20
    for b, t in ((38, 70), (256, 128), (1, 19), (30, 400)):        # GEMM and attention kernel; the front; one launch; long sentences
        assert np.array_equal(model.embed_ids_timed(ids.reshape(-1)[:b * t].reshape(b, t), 2)[0], model.embed_ids(ids.reshape(-1)[:b * t].reshape(b, t)))
