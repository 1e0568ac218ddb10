"""The one-kernel rest of an encoder layer (bert_block.cuh), which large batches reach, against the same sentences in batches that take the
launch chain."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# 45 tiles of 256 tokens, the last with a row in its second half and with none; 90 tiles: two per pair of SMs; sentences of several key tiles
@pytest.mark.parametrize("b,t", [(87, 131), (176, 64), (180, 127), (30, 400)])
def test_block_equals_chain(b, t):
    from fastllm_b200 import models
    model = models.MiniLMModel(models.BertConfig(), None, 0, random_seed=5)
    ids = np.random.default_rng(b).integers(3, 30000, (b, t)).astype(np.uint32)
    got = model.embed_ids(ids)
    want = np.concatenate([model.embed_ids(ids[i:i + 15]) for i in range(0, b, 15)])
    # the two differ in the order of the norms' f32 sums, which moves activations across bf16 roundings: within what either is from 64 bits (5e-3)
    assert np.linalg.norm(got - want, axis=1).max() <= 5e-3
