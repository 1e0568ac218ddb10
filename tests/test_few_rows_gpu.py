"""Calls of up to 128 rows: GEMMs cut evenly over the chip (gemm_dec.cuh), whose blocks take stages of a matrix across tile borders."""
import numpy as np
import pytest

from oracle import causal_lm as ocl
from oracle import synth

from helpers import product_model

pytestmark = pytest.mark.gpu
KERNEL_TOL = 3e-3           # as in test_parity_gpu.py


# widths: K ends inside a stage (320, 1000: k blocks 5 and 15.6), rows end inside a tile (1000), more stages than blocks with borders inside
# tiles (2048 x 5640, 12000 x 2048), fewer stages than blocks (320 x 320)
@pytest.mark.parametrize("hidden,inter,vocab,heads,kv", [(320, 1000, 1000, 10, 5), (2048, 5640, 12000, 16, 4)])
@pytest.mark.parametrize("rows", [3, 16, 17, 32, 33, 64, 65, 128])
def test_rows_against_the_oracle(hidden, inter, vocab, heads, kv, rows):
    from fastllm_b200 import models
    cfg = ocl.CausalLMConfig("llama", hidden, inter, vocab, 1, heads, kv, 1e-5, 1e4, 256)
    w = ocl.synth_weights(cfg, 0, 0.5 * hidden ** -0.5)
    model = product_model(cfg, w)[0]
    ids = synth.token_ids(7, vocab, (rows, 2))
    ref, cache = ocl.CausalLM(cfg, w, kv_dtype="bf16"), models.DeviceCache(model.dev, rows, 64)
    for t in range(2):      # one row per sequence: eager first, then the captured step
        want = ref.forward(ids[:, t:t + 1], t)
        assert np.abs(cache.forward(ids[:, t:t + 1], t) - want).max() <= KERNEL_TOL
    with_prompt = models.DeviceCache(model.dev, 1, 256).forward(synth.token_ids(8, vocab, (1, rows)), 0)       # all rows of one sequence
    want = ocl.CausalLM(cfg, w, kv_dtype="bf16").forward(synth.token_ids(8, vocab, (1, rows)), 0)
    assert np.abs(with_prompt - want).max() <= KERNEL_TOL
