"""Every path of the sampling front half (csrc/sample.cuh) against a full sort: whole and odd vocabularies, those smaller than top_k, rows
beyond the inline slots, ties, masks that leave next to nothing, and slices with more candidates than a CTA may share."""
import dataclasses
import json

import numpy as np
import pytest

from ai00_server_b200 import capi, runtime, synth
from oracle import sampling_numpy as S

pytestmark = pytest.mark.gpu


def _model(vocab, slots, zero_head=False):
    st = synth.make_st(dataclasses.replace(synth.PRESETS["tiny6"], L=1, V=vocab), 5)
    if zero_head:
        st = st.copy()
        n = int(st[:8].view("<u8")[0])
        a, b = json.loads(bytes(st[8:8 + n]))["head.weight"]["data_offsets"]
        st[8 + n + a:8 + n + b] = 0
    m = runtime.Model(st, max_batch=slots, token_chunk_size=128)
    rows = m.infer_raw(list(range(slots)), [1] * slots, [1 + i % 90 for i in range(slots)], [capi.OPTION_LAST] * slots)
    return m, [r[0].copy() for r in rows]


def _check(m, rows, top_k, pen=None, allow=None, bias=None):
    n = len(rows)
    ids, probs = m.sample_topk(list(range(n)), penalties=pen, allow=allow, bias=bias, top_k=top_k)
    for i in range(n):
        want, p = S.sorted_candidates(rows[i], pen[i] if pen else None, allow[i] if allow is not None else None, bias[i] if bias else None, top_k=top_k)
        k = len(want)
        assert np.array_equal(ids[i][:k], want), (i, top_k)
        # one f32 exponential and one division either side, a sum of up to 65536 terms in another order
        np.testing.assert_allclose(probs[i][:k], p, rtol=2e-5, atol=1e-12)
        assert (ids[i][k:] == 0xFFFFFFFF).all() and not probs[i][k:].any()


@pytest.mark.parametrize("vocab", [100, 509, 2048, 8188, 8191, 8192, 20001, 50304, 65535, 65536])
def test_plain_masked_and_adjusted_rows(vocab):
    m, rows = _model(vocab, 3)
    try:
        rng = np.random.default_rng(vocab)
        few = np.zeros((3, vocab), bool)
        for i in range(3):
            few[i, rng.integers(0, vocab, 9)] = True
        pen = [{int(t): float(v) for t, v in zip(rng.integers(0, vocab, 60), rng.random(60))} for _ in rows]
        for top_k in (1, 9, 127, 128):
            _check(m, rows, top_k)
            _check(m, rows, top_k, pen=pen)
            _check(m, rows, top_k, allow=few)
            _check(m, rows, top_k, pen=pen, allow=~few)
        _check(m, rows, 128, allow=np.zeros((3, vocab), bool))
    finally:
        m.close()


@pytest.mark.parametrize("vocab", [2048, 65536])
def test_more_rows_than_inline_slots(vocab):
    m, rows = _model(vocab, 70)
    try:
        _check(m, rows, 128)
        _check(m, rows[:64], 128)
        _check(m, rows, 40, pen=[{i: 1.0} for i in range(70)])
    finally:
        m.close()


@pytest.mark.parametrize("vocab", [300, 2048, 65536])
def test_a_row_of_equal_logits(vocab):
    m, rows = _model(vocab, 1, zero_head=True)
    try:
        assert not rows[0].any()
        for top_k in (1, 17, 128):
            _check(m, rows, top_k)
            _check(m, rows, top_k, bias=[{vocab - 1: 1.0, 5: -1.0}])
    finally:
        m.close()


@pytest.mark.parametrize("cta", [0, 3, 7])
@pytest.mark.parametrize("threads", [1, 16, 17, 127, 128, 256])
def test_the_best_elements_in_the_hands_of_few_threads(threads, cta):
    """All 32 elements of some threads of one CTA far above the rest of the row: up to 127 x 32 candidates, of which a CTA may share 512."""
    m, rows = _model(65536, 1)
    try:
        place = [cta * 8192 + (q * 256 + t) * 4 + e for t in range(threads) for q in range(8) for e in range(4)]
        lift = np.random.default_rng(threads).permutation(len(place))
        bias = [{p: 50.0 + 0.01 * int(v) for p, v in zip(place, lift)}]
        for top_k in (1, 100, 128):
            _check(m, rows, top_k, bias=bias)
    finally:
        m.close()


@pytest.mark.parametrize("vocab, cta", [(2048, 5), (8000, 2)])
def test_the_best_elements_in_a_small_slice(vocab, cta):
    m, rows = _model(vocab, 1)
    try:
        size = (-(-vocab // 8) + 3) & ~3
        place = range(cta * size, (cta + 1) * size)
        lift = np.random.default_rng(vocab).permutation(size)
        for top_k in (1, 100, 128):
            _check(m, rows, top_k, bias=[{p: 50.0 + 0.01 * int(v) for p, v in zip(place, lift)}])
    finally:
        m.close()


@pytest.mark.parametrize("count, top_k", [(512, 128), (513, 128), (4097, 128), (8192, 9), (100, 128)])
def test_equal_logits_of_one_slice(count, top_k):
    """Logits that differ in their ids alone, as many as a CTA may share, one more, more than its list holds and a whole slice: the bound they set lets all of them through."""
    m, rows = _model(65536, 2, zero_head=True)
    try:
        bias = [{int(t): 1.0 for t in range(8192, 8192 + count)}, {int(t): 1.0 + (t % 3) for t in range(0, 3 * count, 3)}]
        _check(m, rows, top_k, bias=bias)
    finally:
        m.close()
