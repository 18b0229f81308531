"""Stamp rows of the profiling replay: a launch of more CTAs than a row has places stays inside its own row."""
import ctypes as C
import dataclasses

import numpy as np
import pytest

from ai00_server_b200 import capi, runtime, synth

pytestmark = pytest.mark.gpu

ROW = 512


def test_rows_of_launches_with_many_ctas():
    """The second low-rank launch of a step of more than 64 tokens has a CTA per 128 outputs of five matrices: 170 at width 4352."""
    shape = dataclasses.replace(synth.PRESETS["tiny6"], L=2, C=4352, F=512)
    m = runtime.Model(synth.make_st(shape, 1), max_batch=72, token_chunk_size=128)
    try:
        slots = list(range(72))
        m.profile_insitu(slots, np.arange(1, 73, dtype=np.uint32), reps=1)
        buf, types, n = np.zeros(1024 * ROW, np.uint64), np.zeros(1024, np.int32), C.c_int32(0)
        capi.check(capi.lib().b200rwkv_debug_trace(m._h, capi.ptr(buf), buf.size, capi.ptr(types), C.byref(n)), m._h)
        rows, types = buf[:n.value * ROW].reshape(-1, ROW), types[:n.value]
        proj = types >= 1000000
        assert proj.sum() >= 2 * 5
        # this kernel leaves the stamps 1, 3 and 4 alone, and its places hold an SM number first
        assert not rows[proj][:, [1, 3, 4]].any()
        assert (rows[proj][:, 8:8 + 3 * 168:3] < 1024).all()
        # launches of other kernels have no places
        assert not rows[~proj][:, 8:].any()
        times = rows[proj][:, [0, 7]].astype(np.float64)
        assert (times[:, 1] >= times[:, 0]).all() and np.ptp(times) < 1e9
    finally:
        m.close()


@pytest.mark.parametrize("slots", [1, 16, 17, 40, 72, 130])
def test_windows_of_every_projection(slots):
    """The profiling replay answers a window for every projection launch, whatever kernel the step's size takes."""
    m = runtime.Model(synth.make_st("tiny6", 1), max_batch=slots, token_chunk_size=128)
    try:
        win, step_us = m.profile_insitu(list(range(slots)), np.arange(1, slots + 1, dtype=np.uint32), reps=2)
        proj = [w for w in win if w["type"] >= 1000000]
        # per layer at least R/K/V/G, output and two channel-mix launches, and the head
        assert len(proj) >= 2 * 4 + 1
        assert all(0 <= w["start_us"] < w["end_us"] <= step_us + 1e-3 for w in proj) and sum(w["bytes"] for w in proj) > 0
    finally:
        m.close()


def test_stamps_of_one_launch_class():
    """Every layer's launch has a whole row on the device, of which the first 16 words come back."""
    shape = dataclasses.replace(synth.PRESETS["tiny6"], L=5)
    m = runtime.Model(synth.make_st(shape, 1), max_batch=4, token_chunk_size=32)
    try:
        ms, nb, tr = C.c_float(0), C.c_int64(0), np.zeros((5, 16), np.uint64)
        capi.check(capi.lib().b200rwkv_debug_gemm_time(m._h, 10, 2, C.byref(ms), C.byref(nb), capi.ptr(tr)), m._h)
        entry, leave = tr[:, 0].astype(np.int64), tr[:, 7].astype(np.int64)
        assert ms.value > 0 and nb.value > 0
        assert (entry > 0).all() and (leave >= entry).all() and (np.diff(entry) > 0).all()
    finally:
        m.close()
