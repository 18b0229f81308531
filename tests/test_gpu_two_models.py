"""Two loaded models in one process: what the second load sets leaves the first one's launches as they are."""
import dataclasses
import json

import numpy as np
import pytest

from ai00_server_b200 import capi, runtime, synth

pytestmark = pytest.mark.gpu


def _prompt(m, n):
    m.state.reset(0)
    return m.infer_raw([0], [n], [1 + i % 90 for i in range(n)], [capi.OPTION_LAST])[0].copy()


def test_a_narrower_rwkv_model_loaded_later():
    """Shared memory of the norm stage of prompt steps grows with the width (12 KB at 1024, above the default 48 KB from 4096 on)."""
    wide = runtime.Model(synth.make_st(dataclasses.replace(synth.PRESETS["tiny6"], L=1, C=4352, F=512), 1), max_batch=1, token_chunk_size=128)
    want = _prompt(wide, 40)
    narrow = runtime.Model(synth.make_st("tiny6", 1), max_batch=1, token_chunk_size=128)
    try:
        _prompt(narrow, 40)
        assert np.array_equal(_prompt(wide, 40), want)
        assert np.isfinite(_prompt(wide, 70)).all()           # a step shape that is captured only now
    finally:
        narrow.close()
        wide.close()


@pytest.mark.parametrize("precision", [0, 1])
def test_a_latent_attention_of_smaller_ranks_loaded_later(precision):
    def load(rank):
        cfg, st, _ = synth.make_kemirax([synth.kemirax_layer("latent_attention", kv_rank=rank, mlp=False)], seed=4)
        assert json.loads(cfg)
        return runtime.Model(st, max_batch=1, token_chunk_size=128, config=cfg, kv_tokens=256, kv_page=16, precision=precision)
    wide = load(256)
    want = _prompt(wide, 20)
    narrow = load(16)
    try:
        _prompt(narrow, 20)
        assert np.array_equal(_prompt(wide, 20), want)
        assert np.isfinite(_prompt(wide, 70)).all()
    finally:
        narrow.close()
        wide.close()
