"""CPU tests of the oracle itself: pinned against the independent fla fixtures and the
committed regression goldens (tests/golden/, generated by oracle/make_golden.py)."""
import os

import numpy as np
import pytest

from ai00_server_b200 import synth
from oracle import rwkv_numpy as O


def test_wkv6_matches_fla_fixture(golden_dir):
    g = np.load(os.path.join(golden_dir, "wkv6_fla.npz"))
    out, S = O.wkv6_seq(g["r"], g["k"], g["v"], np.exp(-np.exp(g["wraw"])), g["u"], g["S0"])
    assert np.abs(out - g["out"]).max() <= 1e-4 * np.abs(g["out"]).max()
    assert np.abs(S - g["S"]).max() <= 1e-5 * max(1.0, np.abs(g["S"]).max())


def test_wkv7_matches_fla_fixture(golden_dir):
    g = np.load(os.path.join(golden_dir, "wkv7_fla.npz"))
    out, S = O.wkv7_seq(g["r"], g["k"], g["v"], g["w"], g["kk"], g["a"], g["S0"])
    assert np.abs(out - g["out"]).max() <= 1e-4 * np.abs(g["out"]).max()
    assert np.abs(S - g["S"]).max() <= 1e-5 * max(1.0, np.abs(g["S"]).max())


@pytest.mark.parametrize("preset", ["tiny5", "tiny6", "tiny7"])
def test_model_goldens(golden_dir, preset):
    g = np.load(os.path.join(golden_dir, f"model_{preset}.npz"))
    w = O.parse_st(synth.make_st(preset, 0))
    for act in ("f16", "f32"):
        orc = O.Oracle(w, act)
        logits, st = orc.run(list(g["tokens"]), orc.state_init(), full=True)
        np.testing.assert_allclose(logits, g[f"logits_{act}"], rtol=0, atol=2e-5)
        if act == "f16":
            np.testing.assert_allclose(st, g["state_f16"], rtol=0, atol=2e-5)


def test_oracle_wkv_inside_model_equals_standalone():
    """The per-head loop in the layer code and the stand-alone recurrence are the same math."""
    w = O.parse_st(synth.make_st("tiny6", 3))
    orc = O.Oracle(w, "f32")
    orc.trace = {}
    st0 = orc.state_init()
    st0[:, 1:65, :] = np.random.default_rng(0).standard_normal(st0[:, 1:65, :].shape).astype(np.float32)
    _, st1 = orc.run([7], st0)
    i = orc.info
    H, N = i.num_head, i.head_size
    r, k, v, dec = (orc.trace[f"0.{n}"].reshape(1, H, N) for n in ("r", "k", "v", "w"))
    u = np.asarray(w["blocks.0.att.time_first"], np.float32)
    S0 = st0[0, 1:1 + N].reshape(N, H, N).transpose(1, 0, 2)
    _, S = O.wkv6_seq(r, k, v, dec, u, S0)
    got = st1[0, 1:1 + N].reshape(N, H, N).transpose(1, 0, 2)
    np.testing.assert_allclose(got, S, atol=1e-6)


def test_full_vs_last_and_split_runs():
    w = O.parse_st(synth.make_st("tiny6", 1))
    orc = O.Oracle(w)
    toks = [3, 9, 100, 4, 77]
    full, s_full = orc.run(toks, orc.state_init(), full=True)
    last, s_last = orc.run(toks, orc.state_init(), full=False)
    np.testing.assert_array_equal(full[-1:], last)
    np.testing.assert_array_equal(s_full, s_last)
    _, s1 = orc.run(toks[:2], orc.state_init())
    l2, s2 = orc.run(toks[2:], s1)
    np.testing.assert_array_equal(l2, last)
    np.testing.assert_array_equal(s2, s_last)


def test_state_init_time_state():
    import dataclasses
    shp = dataclasses.replace(synth.PRESETS["tiny6"], time_state=True)
    w = O.parse_st(synth.make_st(shp, 0))
    orc = O.Oracle(w)
    st = orc.state_init()
    ts = np.asarray(w["blocks.1.att.time_state"], np.float32)     # [H, i, j]
    assert st[1, 1 + 5, 2 * 64 + 9] == ts[2, 5, 9]
    assert np.all(st[:, 0] == 0) and np.all(st[:, 65] == 0)


def test_synth_c_fill_matches_numpy():
    a = synth.make_st("tiny7", 5)
    b = synth.make_st("tiny7", 5, force_numpy=True)
    assert np.array_equal(a, b)


def test_st_image_readable_by_safetensors():
    st = pytest.importorskip("safetensors.numpy")
    img = synth.make_st("tiny6", 0)
    ref = st.load(img.tobytes())
    mine = O.parse_st(img)
    assert set(ref) == set(mine)
    for k in ref:
        assert ref[k].dtype == np.float16
        assert np.array_equal(ref[k], mine[k])


def test_info_and_algorithmic_bytes_match_baseline_table():
    # the published shapes
    assert abs(synth.num_params("v6-7b") / 1e9 - 7.636) < 1e-3
    assert abs(synth.algorithmic_bytes_per_step("v6-7b", 16) / 1e9 - 15.846) < 1e-3
    assert abs(synth.algorithmic_bytes_per_step("v6-1b6", 1) / 1e9 - 2.958) < 1e-3
    assert abs(synth.algorithmic_bytes_per_step("v6-3b", 1) / 1e9 - 5.908) < 1e-3
    assert abs(synth.algorithmic_bytes_per_step("v7-2b9", 8) / 1e9 - 5.909) < 1e-3


def test_softmax_rows():
    x = np.random.default_rng(0).standard_normal((3, 512)).astype(np.float32) * 5
    p = O.softmax_rows(x)
    np.testing.assert_allclose(p.sum(1), 1.0, atol=1e-5)
    assert (p.argmax(1) == x.argmax(1)).all()


@pytest.mark.parametrize("preset,fixture", [("tiny6", "layer6_fla.npz"), ("tiny7", "layer7_fla.npz")])
def test_layers_match_fla_layer_fixtures(golden_dir, preset, fixture):
    """Time-mix and channel-mix sub-layers against flash-linear-attention's own `RWKV6Attention / RWKV6FeedForward /
    RWKV7Attention / RWKV7FeedForward` forward passes on the same weights (oracle/make_golden_fla_layers.py): independent
    pins of the ddlerp / LoRA / decay / bonus / GroupNorm-gate / value-residual composition around the recurrences."""
    g = np.load(os.path.join(golden_dir, fixture))
    w = O.parse_st(synth.make_st(preset, seed=0, force_numpy=True))
    orc = O.Oracle(w, "f32")
    orc.trace = {}
    state = orc.state_init()
    L = int(g["layers"])
    got = [{k: [] for k in ("xx1", "part_att", "xx2", "ffn")} for _ in range(L)]
    for tok in g["tokens"]:
        orc._token(int(tok), state)
        for l in range(L):
            t = orc.trace
            got[l]["xx1"].append(t[f"{l}.xx1"].copy()); got[l]["part_att"].append(t[f"{l}.part_att"].copy())
            got[l]["xx2"].append(t[f"{l}.xx2"].copy())
            got[l]["ffn"].append((t[f"{l}.rr"] * t[f"{l}.part_ffn"]) if preset == "tiny6" else t[f"{l}.part_ffn"].copy())
    rel = lambda a, b: float(np.abs(a - b).max() / np.abs(b).max())
    for l in range(L):
        # the fixture's inputs are the LayerNorm'ed rows the oracle produced when it was generated: still the same
        assert rel(np.stack(got[l]["xx1"]), g[f"att_in_{l}"]) <= 1e-6
        assert rel(np.stack(got[l]["xx2"]), g[f"ffn_in_{l}"]) <= 1e-6
        assert rel(np.stack(got[l]["part_att"]), g[f"att_out_{l}"]) <= 2e-5, l
        assert rel(np.stack(got[l]["ffn"]), g[f"ffn_out_{l}"]) <= 2e-5, l


@pytest.mark.parametrize("preset,fixture", [("tiny6", "model6_fla.npz"), ("tiny7", "model7_fla.npz")])
def test_whole_model_matches_fla_causal_lm_fixture(golden_dir, preset, fixture):
    """Logits of flash-linear-attention's `RWKV6ForCausalLM` / `RWKV7ForCausalLM` on the same weights (oracle/
    make_golden_fla_layers.py `gen_models`): embedding, ln0, every block, ln_out and head of an independent implementation."""
    g = np.load(os.path.join(golden_dir, fixture))
    w = O.parse_st(synth.make_st(preset, seed=0, force_numpy=True))
    orc = O.Oracle(w, "f32")
    got, state = orc.run(g["tokens"].tolist(), orc.state_init(), full=True)
    assert float(np.abs(got - g["logits"]).max() / np.abs(g["logits"]).max()) <= 1e-5
    assert (got.argmax(1) == g["logits"].argmax(1)).all()
    # what fla's cache holds after the run: both token-shift rows and the WKV state S[head][key][value] of every layer
    i = orc.info
    N, H = i.head_size, i.num_head
    for l in range(i.num_layer):
        rows = state[l, 1:1 + N].reshape(N, H, N).transpose(1, 0, 2)          # state rows of head h: [h][row][col]
        kv = rows if i.version == 6 else rows.transpose(0, 2, 1)               # v6 rows = key index, v7 rows = value index
        assert float(np.abs(kv - g[f"wkv_kv_{l}"]).max() / np.abs(kv).max()) <= 1e-5
        assert np.abs(state[l, 0] - g[f"att_shift_{l}"]).max() <= 1e-5
        assert np.abs(state[l, N + 1] - g[f"ffn_shift_{l}"]).max() <= 1e-5
    # the f16 activation contract stays within the documented distance of it
    got16, _ = O.Oracle(w, "f16").run(g["tokens"].tolist(), orc.state_init(), full=True)
    assert float(np.abs(got16 - g["logits"]).max() / np.abs(g["logits"]).max()) <= 2e-3
