"""Prompt steps of the RWKV path at the edges of their shapes: token counts around every tile size of the projection kernel,
row counts of the head, sequences of unequal length, against the CPU oracle in the same operand precision."""
import numpy as np
import pytest

from ai00_server_b200 import capi, runtime, synth
from oracle import rwkv_numpy as O

pytestmark = pytest.mark.gpu

# f16 operands, f32 sums: a projection over k inputs is off by about sqrt(k) * 2^-24 of its terms in either order of summation; what
# remains between engine and oracle are operands that such a difference moves to the neighbouring f16 value (2^-11 of one input)
TOL = 1e-3


def _check(preset, lens, full, chunk=512):
    st = synth.make_st(preset, 3)
    orc = O.Oracle(O.parse_st(st), "f16")
    V = orc.info.num_vocab
    rng = np.random.default_rng(sum(lens))
    toks = [rng.integers(1, V, n).tolist() for n in lens]
    m = runtime.Model(st, max_batch=len(lens), token_chunk_size=chunk)
    try:
        for s in range(len(lens)):
            m.state.reset(s)
        opt = capi.OPTION_FULL if full else capi.OPTION_LAST
        rows = m.infer_raw(list(range(len(lens))), lens, [t for x in toks for t in x], [opt] * len(lens))
        for s, x in enumerate(toks):
            want, state = orc.run(x, orc.state_init(), full=full)
            err = np.abs(rows[s] - want).max() / np.abs(want).max()
            assert err <= TOL, (preset, lens, s, err)
            got = m.state.back(s)
            assert np.abs(got - state).max() <= TOL * np.abs(state).max()
    finally:
        m.close()


@pytest.mark.parametrize("n", [17, 31, 33, 64, 65, 100, 127, 128, 129, 200, 255, 256, 257])
@pytest.mark.parametrize("preset", ["tiny6", "tiny7"])
def test_step_sizes(preset, n):
    _check(preset, [n], full=False)


@pytest.mark.parametrize("lens", [[1, 130, 3], [40, 41, 42, 43, 44, 45, 46], [5] * 29])
@pytest.mark.parametrize("preset", ["tiny5", "tiny6", "tiny7"])
def test_full_rows_of_ragged_batches(preset, lens):
    _check(preset, lens, full=True)


@pytest.mark.parametrize("lens, rows", [([200], [(0, 128, 200)]), ([130, 140, 5], [(1, 121, 140)])])
def test_last_hidden_answers_the_last_portion(lens, rows):
    """Without keep_hidden the hidden rows are those of the call's last portion of at most 128 tokens, whatever a step holds."""
    st = synth.make_st("tiny6", 3)
    orc = O.Oracle(O.parse_st(st), "f16")
    rng = np.random.default_rng(9)
    toks = [rng.integers(1, 500, n).tolist() for n in lens]
    m = runtime.Model(st, max_batch=len(lens), token_chunk_size=128)
    try:
        for s in range(len(lens)):
            m.state.reset(s)
        m.infer_raw(list(range(len(lens))), lens, sum(toks, []), [capi.OPTION_NONE] * len(lens))
        got = m.last_hidden(max_rows=128)
        want = np.concatenate([orc.hidden(toks[s], orc.state_init())[0][a:b] for s, a, b in rows])
        assert got.shape == want.shape
        assert np.abs(got - want).max() <= TOL * np.abs(want).max()
    finally:
        m.close()
