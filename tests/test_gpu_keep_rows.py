"""The logits row a slot keeps for sampling, at vocabularies whose rows do not begin on 16-byte boundaries."""
import dataclasses

import numpy as np
import pytest

from ai00_server_b200 import capi, runtime, synth
from oracle import sampling_numpy as S

pytestmark = pytest.mark.gpu


def _check(m, n_tok):
    V = m.info["num_vocab"]
    rng = np.random.default_rng(V)
    slots = [0, 1, 2]
    for s in slots:
        m.state.reset(s)
    toks = rng.integers(1, 90, (3, n_tok)).tolist()
    rows = m.infer_raw(slots, [n_tok] * 3, sum(toks, []), [capi.OPTION_LAST] * 3)
    for top_k in (1, 40):
        ids, probs = m.sample_topk(slots, top_k=top_k)
        for i in slots:
            want_ids, want_p = S.sorted_candidates(rows[i][0], top_k=top_k)
            assert np.array_equal(ids[i], want_ids)
            np.testing.assert_allclose(probs[i], want_p, rtol=2e-5, atol=1e-12)
    snap = m.state.read(1)                       # the row travels with the state
    assert np.array_equal(m.state.snapshot_back(snap, with_logits=True)[1], rows[1][0])
    snap.free()


@pytest.mark.parametrize("n_tok", [1, 20])
@pytest.mark.parametrize("vocab", [509, 511, 514])
def test_rwkv(vocab, n_tok):
    m = runtime.Model(synth.make_st(dataclasses.replace(synth.PRESETS["tiny6"], V=vocab), 3), max_batch=3, token_chunk_size=128)
    try:
        _check(m, n_tok)
    finally:
        m.close()


@pytest.mark.parametrize("n_tok", [1, 20])
def test_config_json_family(n_tok):
    cfg, st, _ = synth.make_panupel([synth.panupel_layer("delta", heads=3, dim=24, ff=48)], width=136, vocab=97, seed=4, loop=None)
    m = runtime.Model(st, max_batch=3, token_chunk_size=128, config=cfg, kv_tokens=128, kv_page=16)
    try:
        _check(m, n_tok)
    finally:
        m.close()
