"""Prompt steps of many sequences: the kernels that take over once a step fills the chip (attention of 128 rows on the tensor cores, recurrences sixteen tokens at a time or with two
state columns a thread, convolutions in registers), at the edges of their tiles, against the families' restatements."""
import json

import numpy as np
import pytest

from ai00_server_b200 import capi, runtime, synth
from oracle import degavik_numpy, fufipel_numpy, kemirax_numpy, panupel_numpy
from oracle import rwkv_numpy as O

pytestmark = pytest.mark.gpu

# f32 engine against float64: the bound the families' own tests hold (2e-4 of the logits' spread in any row); bf16 operands (2^-9 each): a few percent in the
# median row, a wrong row is off by its own size
TIGHT, BF16_TOL, ROW_TOL = 2e-4, 5e-2, 0.5
N_SEQ = 48


def _errs(got, want):
    return np.sqrt(((got - want) ** 2).mean(1)) / np.sqrt((want ** 2).mean())


def _check(make, module, layers, precision, kv=16, **kw):
    """48 sequences of 1 to 97 tokens in one call (steps of several hundred tokens); four of them against the restatement, row by row, then five tokens more
    of those four (the states and caches the step left)."""
    cfg, st, w = make(layers, seed=4, **kw)
    rng = np.random.default_rng(7)
    lens = [97, 1, 64, 33] + rng.integers(1, 90, N_SEQ - 4).tolist()
    toks = [rng.integers(1, 90, n + 5).tolist() for n in lens]
    m = runtime.Model(st, max_batch=N_SEQ, token_chunk_size=512, precision=precision, config=cfg, kv_tokens=sum(lens) + 8 * N_SEQ, kv_page=kv)
    try:
        for s in range(N_SEQ):
            m.state.reset(s)
        opt = [capi.OPTION_FULL] * 4 + [capi.OPTION_LAST] * (N_SEQ - 4)
        got = m.infer_raw(list(range(N_SEQ)), lens, sum((t[:n] for t, n in zip(toks, lens)), []), opt)
        more = m.infer_raw([0, 1, 2, 3], [5] * 4, sum((toks[s][lens[s]:] for s in range(4)), []), [capi.OPTION_FULL] * 4)
        for s in range(4):
            want = module.run(json.loads(cfg), w, toks[s])
            err = _errs(np.concatenate([got[s], more[s]]), want)
            if precision == 1:
                assert err.max() <= TIGHT, (s, int(err.argmax()), float(err.max()))
            else:
                assert np.median(err) <= BF16_TOL and err.max() <= ROW_TOL, (s, float(np.median(err)), int(err.argmax()), float(err.max()))
    finally:
        m.close()


P, F, K, D = synth.panupel_layer, synth.fufipel_layer, synth.kemirax_layer, synth.degavik_layer


@pytest.mark.parametrize("heads, kv_heads, dim, vdim", [(4, 4, 24, 24), (4, 1, 40, 72), (6, 2, 128, 128), (3, 1, 16, 112)])
def test_attention_over_the_whole_context(heads, kv_heads, dim, vdim):
    """128 rows are 128, 32, 42 and 42 tokens of one key head; sizes below, at and between the 64-entry halves of a value row."""
    _check(synth.make_panupel, panupel_numpy, [P("parallel", heads=heads, kv_heads=kv_heads, dim=dim, vdim=vdim, mm_heads=2, mm_dim=72)], 1, width=96, loop=None)


@pytest.mark.parametrize("window, keep", [(8, 2), (33, 0), (40, 5), (63, 0), (64, 3), (65, 0), (65, 2)])
def test_attention_in_a_window(window, keep):
    """Kept first tokens in front of windows that end inside, at and behind a tile of 64 keys, sequences longer than the window, a bias per distance, a gate per entry; a chunked layer
    beside it."""
    _check(synth.make_fufipel, fufipel_numpy, [F("attention", heads=4, kv_heads=2, dim=20, window=window, keep_first=keep), F("parallel", heads=2, dim=24, chunk=11)], 1, width=80)


@pytest.mark.parametrize("heads, kv_heads, dim, vdim", [(4, 1, 128, 128), (2, 2, 128, 128), (5, 1, 32, 104), (3, 1, 20, 36)])
def test_attention_at_the_edges_of_key_tiles(heads, kv_heads, dim, vdim):
    """Contexts below, at and behind the borders of 64-key tiles, 128 rows of 32, 128, 25 and 42 tokens; heads of 128 channels, of multiples of eight and of four."""
    cfg, st, w = synth.make_panupel([P("parallel", heads=heads, kv_heads=kv_heads, dim=dim, vdim=vdim, mm_heads=1, mm_dim=16)], seed=5, width=96, loop=None)
    lens = [63, 64, 65, 129, 200]
    toks = [np.random.default_rng(n).integers(1, 90, n).tolist() for n in lens]
    m = runtime.Model(st, max_batch=len(lens), token_chunk_size=512, precision=1, config=cfg, kv_tokens=sum(lens) + 16 * len(lens), kv_page=16)
    try:
        for s in range(len(lens)):
            m.state.reset(s)
        got = m.infer_raw(list(range(len(lens))), lens, sum(toks, []), [capi.OPTION_FULL] * len(lens))
        for s in range(len(lens)):
            err = _errs(got[s], panupel_numpy.run(json.loads(cfg), w, toks[s]))
            assert err.max() <= TIGHT, (s, int(err.argmax()), float(err.max()))
    finally:
        m.close()


@pytest.mark.parametrize("make, module, layers", [
    (synth.make_kemirax, kemirax_numpy, [K("gla", heads=2, dim=40, vdim=24, mlp=False), K("latent_attention", heads=3, kv_rank=24, rot_dim=8, mlp=False)]),
    (synth.make_panupel, panupel_numpy, [P("delta", heads=2, dim=24), P("parallel", heads=4, kv_heads=2, dim=24, mm_heads=2, mm_dim=24)]),
    (synth.make_fufipel, fufipel_numpy, [F("attention", heads=4, kv_heads=2, dim=20, window=8, keep_first=2), F("parallel", heads=2, dim=24, chunk=11)])])
def test_steps_of_one_row_count_and_several_numbers_of_sequences(make, module, layers):
    """Steps of 24 tokens in one sequence, eight, nine, twelve and eighteen (captured ones hold CTAs for the next power of two, eight at least), and longer ones of 3 and 20 (as many as
    there are)."""
    cfg, st, w = make(layers, seed=4, width=96, **({"loop": None} if make is synth.make_panupel else {}))
    m = runtime.Model(st, max_batch=24, token_chunk_size=512, precision=1, config=cfg, kv_tokens=2048, kv_page=16)
    try:
        for lens in ([24], [3] * 8, [3, 3, 3, 3, 3, 3, 2, 2, 2], [2] * 12, [24], [2] * 6 + [1] * 12, [200, 3, 330], [30] * 20, [2] * 12):
            toks = [np.random.default_rng([n, i]).integers(1, 90, n).tolist() for i, n in enumerate(lens)]
            for s in range(len(lens)):
                m.state.reset(s)
            got = m.infer_raw(list(range(len(lens))), lens, sum(toks, []), [capi.OPTION_FULL] * len(lens))
            for s in (0, len(lens) // 2, len(lens) - 1):
                err = _errs(got[s], module.run(json.loads(cfg), w, toks[s]))
                assert err.max() <= TIGHT, (lens, s, int(err.argmax()), float(err.max()))
    finally:
        m.close()


@pytest.mark.parametrize("heads, kv_heads, dim, vdim, longest", [(4, 4, 24, 24, 32), (3, 3, 128, 128, 32), (12, 3, 32, 36, 14), (9, 3, 72, 104, 8), (3, 3, 64, 4, 33), (4, 2, 40, 40, 33)])
def test_attention_of_many_short_sequences(heads, kv_heads, dim, vdim, longest):
    """64 sequences of 1 to `longest` tokens, then five more of each: the form for few (token, head) rows a key head, below and behind one of its tiles of 32 keys, rows of one, three
    and four query heads (whose 64 leave one over); and the other side of its rule.  A token that is not a number reaches no row before it and no other sequence."""
    cfg, st, w = synth.make_panupel([P("parallel", heads=heads, kv_heads=kv_heads, dim=dim, vdim=vdim, mm_heads=1, mm_dim=16)], seed=5, width=96, loop=None)
    st = st.copy()
    head = int(st[:8].view("<u8")[0])
    e = json.loads(bytes(st[8:8 + head]))["embed"]
    st[8 + head + e["data_offsets"][0]:8 + head + e["data_offsets"][1]].view("<u2").reshape(e["shape"])[7] = 0x7fc0
    rng = np.random.default_rng(longest)
    B = 64
    lens = [longest, 1, 2, longest - 1] + rng.integers(1, longest, B - 4).tolist()
    toks = [rng.integers(10, 90, n + 5).tolist() for n in lens]
    toks[3][longest // 2] = 7
    m = runtime.Model(st, max_batch=B, token_chunk_size=512, precision=1, config=cfg, kv_tokens=sum(lens) + 24 * B, kv_page=16)
    try:
        for s in range(B):
            m.state.reset(s)
        opt = [capi.OPTION_FULL] * B
        got = m.infer_raw(list(range(B)), lens, sum((t[:n] for t, n in zip(toks, lens)), []), opt)
        more = m.infer_raw(list(range(B)), [5] * B, sum((t[n:] for t, n in zip(toks, lens)), []), opt)
        for s in (0, 1, 2, 3, 4, B - 1):
            rows, n = np.concatenate([got[s], more[s]]), longest // 2 if s == 3 else lens[s] + 5
            assert np.isfinite(rows[:n]).all() and np.isnan(rows[n:]).all(), (s, np.isfinite(rows).all(1).tolist())
            err = _errs(rows[:n], panupel_numpy.run(json.loads(cfg), w, toks[s][:n]))
            assert err.max() <= TIGHT, (s, int(err.argmax()), float(err.max()))
        assert all(np.isfinite(got[s]).all() and np.isfinite(more[s]).all() for s in range(B) if s != 3)
    finally:
        m.close()


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("dim, vdim, conv", [(72, 72, 4), (128, 40, 4), (24, 24, 4), (40, 72, 3)])
def test_delta_rule(dim, vdim, conv, precision):
    """One and two columns a thread (vdim above and below the columns a CTA holds), convolutions of four taps in registers and of three as before."""
    _check(synth.make_panupel, panupel_numpy, [P("delta", heads=2, dim=dim, vdim=vdim, conv=conv)], precision, width=96, loop=None)


def test_delta_rule_with_a_decay_per_channel():
    _check(synth.make_degavik, degavik_numpy, [D("channel_delta", heads=2, dim=72, vdim=72, conv=4)], 1, width=96)


@pytest.mark.parametrize("dim, vdim", [(72, 72), (16, 24)])
def test_gated_linear_attention(dim, vdim):
    _check(synth.make_kemirax, kemirax_numpy, [K("gla", heads=2, dim=dim, vdim=vdim, mlp=False)], 1, width=96)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("dim, vdim, tau", [(128, 128, 8.0), (72, 40, 8.0), (34, 33, 8.0), (128, 128, 0.5), (40, 128, 0.02)])
def test_gated_linear_attention_in_runs(dim, vdim, tau, precision):
    """Sequences of about a run of sixteen tokens, several and parts of them, continued in a second call; sizes that are no multiples of eight or four; decays that cut runs short,
    and such that tokens go one by one."""
    cfg, st, w = synth.make_kemirax([K("gla", heads=3, dim=dim, vdim=vdim, tau=tau, mlp=False)], seed=8, width=96)
    lens = [15, 16, 17, 33, 120]
    toks = [np.random.default_rng(n).integers(1, 90, n + 37).tolist() for n in lens]
    m = runtime.Model(st, max_batch=len(lens), token_chunk_size=512, precision=precision, config=cfg, kv_tokens=512)
    try:
        for s in range(len(lens)):
            m.state.reset(s)
        opt = [capi.OPTION_FULL] * len(lens)
        got = m.infer_raw(list(range(len(lens))), lens, sum((t[:n] for t, n in zip(toks, lens)), []), opt)
        more = m.infer_raw(list(range(len(lens))), [37] * len(lens), sum((t[n:] for t, n in zip(toks, lens)), []), opt)
        for s in range(len(lens)):
            err = _errs(np.concatenate([got[s], more[s]]), kemirax_numpy.run(json.loads(cfg), w, toks[s]))
            if precision == 1:
                assert err.max() <= TIGHT, (s, int(err.argmax()), float(err.max()))
            else:
                assert np.median(err) <= BF16_TOL and err.max() <= ROW_TOL, (s, float(np.median(err)), int(err.argmax()), float(err.max()))
    finally:
        m.close()


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("layer", [P("delta", heads=2, dim=128, vdim=128, conv=4), P("delta", heads=3, dim=72, vdim=40, conv=4), P("delta", heads=4, kv_heads=2, dim=34, vdim=33, conv=4),
                                   P("parallel", mm_heads=2, mm_dim=128), P("parallel", mm_heads=3, mm_dim=72, mm_vdim=40), P("parallel", mm_heads=2, mm_dim=33, mm_vdim=66)])
def test_recurrences_with_one_decay_a_head_in_runs(layer, precision):
    """Sequences of about a run of sixteen tokens, several and parts of them, continued in a second call; sizes that are no multiples of eight or four; keys of two heads in common."""
    cfg, st, w = synth.make_panupel([layer], seed=8, width=96, loop=None)
    lens, then = [15, 16, 17, 33, 280], 70
    toks = [np.random.default_rng(n).integers(1, 90, n + then).tolist() for n in lens]
    m = runtime.Model(st, max_batch=len(lens), token_chunk_size=512, precision=precision, config=cfg, kv_tokens=1024)
    try:
        for s in range(len(lens)):
            m.state.reset(s)
        opt = [capi.OPTION_FULL] * len(lens)
        got = m.infer_raw(list(range(len(lens))), lens, sum((t[:n] for t, n in zip(toks, lens)), []), opt)
        more = m.infer_raw(list(range(len(lens))), [then] * len(lens), sum((t[n:] for t, n in zip(toks, lens)), []), opt)
        for s in range(len(lens)):
            err = _errs(np.concatenate([got[s], more[s]]), panupel_numpy.run(json.loads(cfg), w, toks[s]))
            if precision == 1:
                assert err.max() <= TIGHT, (s, int(err.argmax()), float(err.max()))
            else:
                assert np.median(err) <= BF16_TOL and err.max() <= ROW_TOL, (s, float(np.median(err)), int(err.argmax()), float(err.max()))
    finally:
        m.close()


@pytest.mark.parametrize("heads, kv_rank, rot_dim", [(4, 24, 8), (16, 40, 16), (5, 72, 4), (20, 64, 8)])
def test_latent_attention(heads, kv_rank, rot_dim):
    """64 rows of 4, 16, 5 and 20 (two CTAs) heads; latent rows with and without pad columns; channels that do not fill eight warps."""
    _check(synth.make_kemirax, kemirax_numpy, [K("latent_attention", heads=heads, kv_rank=kv_rank, rot_dim=rot_dim, experts=6, top=3)], 0, width=96)


@pytest.mark.parametrize("heads, kv_rank, rot_dim", [(16, 128, 64), (3, 20, 4), (8, 200, 24)])
def test_latent_attention_at_the_edges_of_key_tiles(heads, kv_rank, rot_dim):
    """Contexts below, at and behind the borders of 32-key tiles, latent rows of one, part of one and several pieces of 128 entries, of multiples of eight and of four."""
    cfg, st, w = synth.make_kemirax([K("latent_attention", heads=heads, kv_rank=kv_rank, rot_dim=rot_dim, mlp=False)], seed=6, width=96)
    lens = [31, 32, 33, 65, 150]
    toks = [np.random.default_rng(n).integers(1, 90, n).tolist() for n in lens]
    m = runtime.Model(st, max_batch=len(lens), token_chunk_size=512, config=cfg, kv_tokens=sum(lens) + 16 * len(lens), kv_page=16)
    try:
        for s in range(len(lens)):
            m.state.reset(s)
        got = m.infer_raw(list(range(len(lens))), lens, sum(toks, []), [capi.OPTION_FULL] * len(lens))
        for s in range(len(lens)):
            err = _errs(got[s], kemirax_numpy.run(json.loads(cfg), w, toks[s]))
            assert np.median(err) <= BF16_TOL and err.max() <= ROW_TOL, (s, float(np.median(err)), int(err.argmax()), float(err.max()))
    finally:
        m.close()


@pytest.mark.parametrize("heads, kv_rank, rot_dim", [(16, 42, 8), (20, 512, 64), (5, 30, 4)])
def test_latent_attention_of_single_tokens(heads, kv_rank, rot_dim):
    """One token of every sequence behind contexts of one key, parts of a 32-key tile, and several tiles in parts of their own; latent rows that are no whole runs of sixteen bytes, of
    as many channels as the kernel holds, and of fewer than its warps take."""
    cfg, st, w = synth.make_kemirax([K("latent_attention", heads=heads, kv_rank=kv_rank, rot_dim=rot_dim, mlp=False)], seed=6, width=96)
    lens, more = [1, 31, 64, 150, 500], 3
    toks = [np.random.default_rng(n).integers(1, 90, n + more).tolist() for n in lens]
    m = runtime.Model(st, max_batch=len(lens), token_chunk_size=512, config=cfg, kv_tokens=sum(lens) + 32 * len(lens), kv_page=16)
    try:
        for s in range(len(lens)):
            m.state.reset(s)
        opt = [capi.OPTION_FULL] * len(lens)
        m.infer_raw(list(range(len(lens))), lens, sum((t[:n] for t, n in zip(toks, lens)), []), opt)
        rows = [m.infer_raw(list(range(len(lens))), [1] * len(lens), [t[n + i] for t, n in zip(toks, lens)], opt) for i in range(more)]
        for s, n in enumerate(lens):
            err = _errs(np.concatenate([r[s] for r in rows]), kemirax_numpy.run(json.loads(cfg), w, toks[s])[n:])
            assert np.median(err) <= BF16_TOL and err.max() <= ROW_TOL, (s, float(np.median(err)), int(err.argmax()), float(err.max()))
    finally:
        m.close()


@pytest.mark.parametrize("width", [98, 260, 4096, 4104])
def test_rows_in_pieces_of_sixteen_bytes(width):
    """Norms, token shift, router and the experts' sum at widths that are no whole pieces, of a part of a CTA's pieces, of all of them, and of more."""
    cfg, st, w = synth.make_kemirax([K("gla", heads=2, dim=16, vdim=16, experts=11, top=3)], seed=3, width=width)
    lens = [1, 5, 40]
    toks = [np.random.default_rng(n).integers(1, 90, n + 1).tolist() for n in lens]
    m = runtime.Model(st, max_batch=len(lens), token_chunk_size=512, precision=1, config=cfg, kv_tokens=256)
    try:
        for s in range(len(lens)):
            m.state.reset(s)
        opt = [capi.OPTION_FULL] * len(lens)
        got = m.infer_raw(list(range(len(lens))), lens, sum((t[:n] for t, n in zip(toks, lens)), []), opt)
        more = m.infer_raw(list(range(len(lens))), [1] * len(lens), [t[n] for t, n in zip(toks, lens)], opt)
        for s in range(len(lens)):
            err = _errs(np.concatenate([got[s], more[s]]), kemirax_numpy.run(json.loads(cfg), w, toks[s]))
            assert err.max() <= TIGHT, (s, int(err.argmax()), float(err.max()))
    finally:
        m.close()


@pytest.mark.parametrize("n", [17, 100, 300])
@pytest.mark.parametrize("ranks", [(64, 128), (32, 32), (64, 64)])
def test_low_rank_second_stages(ranks, n):
    """Both kernels of lora2.cuh at every rank they are built for, one tile of tokens and several."""
    _check_low_ranks(ranks, n)


@pytest.mark.parametrize("n", [17, 70, 128, 300])
@pytest.mark.parametrize("ranks", [(96, 160), (160, 64), (264, 128)])
def test_low_ranks_of_other_sizes(ranks, n):
    """Ranks lora2.cuh is not built for, of one k block (128) and of several: the projections' own epilogue mixes the rows, in every form that can meet it."""
    _check_low_ranks(ranks, n)


def _check_low_ranks(ranks, n):
    st = synth.make_st(synth.Shape(6, 2, 256, 896, V=512, Dm=ranks[0], Dd=ranks[1]), 3)
    orc = O.Oracle(O.parse_st(st), "f16")
    toks = np.random.default_rng(n).integers(1, 500, n).tolist()
    m = runtime.Model(st, max_batch=1, token_chunk_size=128)
    try:
        m.state.reset(0)
        got = m.infer_raw([0], [n], toks, [capi.OPTION_LAST])[0]
        want, state = orc.run(toks, orc.state_init())
        assert np.abs(got - want).max() <= 1e-3 * np.abs(want).max()
        assert np.abs(m.state.back(0) - state).max() <= 1e-3 * np.abs(state).max()
    finally:
        m.close()
