"""Result arrays over page-locked memory: what a program may do with any array of its own."""
import os
import signal
import time

import numpy as np
import pytest

from oracle import causal_lm as ocl
from oracle import synth

from helpers import product_model

pytestmark = pytest.mark.gpu


def _cache(vocab):
    from fastllm_b200 import models
    cfg = ocl.CausalLMConfig("llama", 64, 96, vocab, 1, 4, 2, 1e-5, 1e4, 64)
    model = product_model(cfg, ocl.synth_weights(cfg, 0, 0.05))[0]
    return models.DeviceCache(model.dev, 8, 32)


# eight rows: 128 KB, enough for a page-locked array, and 1.25 MB, which lies in huge pages
@pytest.mark.parametrize("vocab", [4096, 40000])
def test_a_forked_child_keeps_the_result_it_holds(vocab):
    from fastllm_b200 import models
    cache = _cache(vocab)
    out = cache.forward(synth.token_ids(1, vocab, (8, 1)), 0)
    assert isinstance(out.base, models._Block)                  # page-locked
    before, where = out.copy(), out.__array_interface__["data"][0]
    go, told = os.pipe()
    pid = os.fork()
    if pid == 0:            # no call of the library here: the context belongs to the parent
        os.read(go, 1)
        same = bool((out == before).all())
        out[:] = -1.0       # and its writes are its own
        os._exit(0 if same else 3)
    del out
    again = cache.forward(synth.token_ids(2, vocab, (8, 1)), 1)
    others = cache.forward(synth.token_ids(3, vocab, (8, 1)), 2)
    reused = [a for a in (again, others) if a.__array_interface__["data"][0] == where]
    kept = [a.copy() for a in (again, others)]
    os.write(told, b"x")
    for _ in range(200):
        done, status = os.waitpid(pid, os.WNOHANG)
        if done:
            break
        time.sleep(0.1)
    else:
        os.kill(pid, signal.SIGKILL)
        os.waitpid(pid, 0)
        pytest.fail("the child did not end")
    assert reused and not (reused[0] == before).all()           # the device has written over the block the child looked at
    assert status == 0
    assert (again == kept[0]).all() and (others == kept[1]).all()


def test_a_refused_allocation_fails_one_call():
    """memory that cannot be had is reported by the call that asked for it, not once more by the next one of the thread"""
    from fastllm_b200 import _lib, models
    encoder = models.MiniLMModel(models.BertConfig(), None, 0, random_seed=5)
    ids = np.full((2, 7), 100, dtype=np.uint32)
    want = encoder.embed_ids(ids)
    cf = models.ConfigFile(8192, 8192, 1 << 30, 1, 64, 64, 1e-5, 1e4, 64, None)      # an embedding table of 16 TB
    with pytest.raises(_lib.FastllmError, match="out of memory"):
        models.LlamaWithConfig.initialize_model(cf, None, random_seed=0)
    assert (encoder.embed_ids(ids) == want).all()
