"""Logits and arg-max of the causal models' calls: maxima that tie, and results of several megabytes, which leave the device in parts."""
import dataclasses

import numpy as np
import pytest

from oracle import causal_lm as ocl
from oracle import synth

from helpers import TINY, product_model

pytestmark = pytest.mark.gpu
KERNEL_TOL = 3e-3           # as in test_parity_gpu.py


def _setup(vocab, repeats=1):
    cfg = dataclasses.replace(TINY["llama"], vocab_size=vocab)
    w = ocl.synth_weights(cfg, 0, 0.05)
    if repeats > 1:         # equal rows of the vocabulary projection: equal logits
        w["lm_head.weight"] = np.tile(w["lm_head.weight"][:vocab // repeats], (repeats, 1))
    return cfg, w, product_model(cfg, w)[0]


@pytest.mark.parametrize("vocab,repeats", [(2048, 2), (2048, 16), (600, 2), (1536, 3)])
@pytest.mark.parametrize("b", [1, 3, 40])
def test_last_of_equal_maxima(vocab, repeats, b):
    """equal maxima in one part of a row and in several: the last one is taken, as the host's arg-max takes it"""
    from fastllm_b200 import models
    cfg, w, model = _setup(vocab, repeats)
    prompt = synth.token_ids(5, cfg.vocab_size, (b, 4))
    logits = models.DeviceCache(model.dev, b, 64).forward(prompt, 0)
    assert np.array_equal(logits[:, :vocab // repeats], logits[:, -(vocab // repeats):])
    want = vocab - 1 - np.argmax(logits[:, ::-1], axis=1)
    assert (want >= vocab - vocab // repeats).all()
    assert [models.sample_argmax(r) for r in logits] == want.tolist()
    assert np.array_equal(np.asarray(models.DeviceCache(model.dev, b, 64).forward_greedy(prompt, 0)).ravel(), want)


@pytest.mark.parametrize("vocab,b", [(32000, 32), (32768, 32), (32008, 40), (32008, 81)])
def test_large_logits(vocab, b):
    """just below two parts, at two, at two of odd lengths, at four: every logit against the oracle, through both calls"""
    from fastllm_b200 import models
    cfg, w, model = _setup(vocab)
    prompt = synth.token_ids(6, cfg.vocab_size, (b, 3))
    want = ocl.CausalLM(cfg, w, kv_dtype="bf16").forward(prompt, 0)
    got = models.DeviceCache(model.dev, b, 64).forward(prompt, 0)
    assert np.abs(got - want).max() <= KERNEL_TOL
    slots = models.DeviceCache(model.dev, b, 64)
    assert np.abs(slots.forward_slots(list(range(b)), prompt, [0] * b) - want).max() <= KERNEL_TOL
