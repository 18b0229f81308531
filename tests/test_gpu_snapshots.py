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
