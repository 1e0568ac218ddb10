"""The one-kernel rest of an encoder layer (bert_block.cuh), which large batches reach, against the same sentences in batches that take the
launch chain, and against the oracle."""
import numpy as np
import pytest

from oracle import bert as obert

pytestmark = pytest.mark.gpu


def launches(model, ids):
    """-> embeddings, kernels launched: three per layer with the block kernel, seven in the chain"""
    from fastllm_b200 import models
    before = models.launch_count()
    out = model.embed_ids(ids)
    return out, models.launch_count() - before


# tiles of 256 tokens (pairs of SMs: 74): 45, the last with rows in its first half and 5 in its second; 44 full ones; 46, the last with 64 rows, none in
# its second half; 90, two per pair for some; 47 of sentences of several key tiles; 37, half a wave
@pytest.mark.parametrize("b,t", [(87, 131), (176, 64), (181, 64), (180, 127), (30, 400), (73, 128)])
def test_block_equals_chain(b, t):
    from fastllm_b200 import models
    model = models.MiniLMModel(models.BertConfig(), None, 0, random_seed=5)
    ids = np.random.default_rng(b).integers(3, 30000, (b, t)).astype(np.uint32)
    got, block_launches = launches(model, ids)
    parts = [launches(model, ids[i:i + 15]) for i in range(0, b, 15)]
    assert block_launches < parts[0][1]
    want = np.concatenate([p[0] for p in parts])
    # the two differ in the order of the norms' f32 sums, which moves activations across bf16 roundings: within what either is from 64 bits (5e-3)
    assert np.linalg.norm(got - want, axis=1).max() <= 5e-3


@pytest.mark.parametrize("b,t", [(56, 128), (106, 67)])
def test_fewest_tiles_of_the_block_kernel(b, t):
    """28 tiles of 256 tokens, the last one full or of 190 rows"""
    test_block_equals_chain(b, t)


def test_block_against_the_oracle():
    """norm weights between 1/2 and 3/2 and biases everywhere, so that no column may stand in another's place; sentences at the borders of the tiles"""
    cfg = obert.BertConfig(384, 12, 2, 1536, 96, 1e-12, 512)
    rng = np.random.default_rng(3)
    w = {}
    for name, shape, kind in obert.tensor_names(cfg):
        w[name] = (rng.uniform(0.5, 1.5, shape) if kind == "norm" else rng.normal(0, 0.05 if len(shape) == 2 else 0.3, shape)).astype(np.float32)
        if len(shape) == 2:         # (matrices that bf16 holds, as the device stores them)
            w[name] = ((w[name].view(np.uint32) + 0x8000) & 0xFFFF0000).view(np.float32)
    from fastllm_b200 import models
    model = models.MiniLMModel(models.BertConfig(384, 12, 2, 1536, 96, 1e-12, 512), w, 0)
    b, t = 141, 70                  # 9870 tokens: 39 tiles, the last with 142 rows
    ids = rng.integers(3, 512, (b, t)).astype(np.uint32)
    got, block_launches = launches(model, ids)
    assert block_launches < launches(model, ids[:15])[1]
    picked = [0, 1, 3, 69, 70, 137, 138, 139, 140]
    want = obert.MiniLM(cfg, w).embed_ids(ids[picked])
    # about ten activations of a token are rounded to bf16 (relative 2^-9, each its own way): 2^-9 sqrt(10); pooling over 70 tokens only lessens it
    err = np.linalg.norm(got[picked] - want, axis=1)
    print("block against the oracle: largest distance of a unit vector", err.max())
    assert err.max() <= 2.0 ** -9 * 10 ** 0.5
