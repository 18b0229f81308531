"""Snapshot records given back while a copy out of them may still be in flight, and runs of a record that are cut into several."""
import numpy as np
import pytest

from ai00_server_b200 import capi, runtime, synth

pytestmark = pytest.mark.gpu


def test_a_record_freed_right_behind_its_write():
    m = runtime.Model(synth.make_st("small6", 2), max_batch=3, token_chunk_size=128)
    try:
        rng = np.random.default_rng(0)
        for s in range(3):
            m.state.reset(s)
        m.infer_raw([0, 1], [30, 40], rng.integers(1, 2000, 70).tolist(), [capi.OPTION_LAST] * 2)
        want = m.state.back(0)
        for _ in range(20):
            a = m.state.read(0)
            m.state.write(a, 2)
            a.free()
            b = m.state.read(1)                  # may get the memory of the freed record
            assert np.array_equal(m.state.back(2), want)
            b.free()
    finally:
        m.close()


@pytest.mark.parametrize("rank", [512, 510])
def test_a_long_sequence_of_cache_rows(rank):
    """A run of cache rows longer than one run of the transfer kernel (2^22 floats), of whole float4 and of single floats."""
    cfg, st, _ = synth.make_kemirax([synth.kemirax_layer("latent_attention", heads=1, kv_rank=rank, mlp=False)], seed=4)
    n = 8120
    m = runtime.Model(st, max_batch=2, token_chunk_size=512, config=cfg, kv_tokens=2 * n + 64, kv_page=32)
    try:
        toks = np.random.default_rng(1).integers(1, 90, n).tolist()
        m.state.reset(0)
        m.state.reset(1)
        m.infer_raw([0], [n], toks, [capi.OPTION_LAST])
        assert n * (rank + 8) > 1 << 22
        snap = m.state.read(0)
        m.state.write(snap, 1)
        assert np.array_equal(m.state.back(1), m.state.back(0))
        a, b = m.infer_raw([0, 1], [1, 1], [5, 5], [capi.OPTION_LAST] * 2)
        assert np.array_equal(a, b)
        snap.free()
    finally:
        m.close()
