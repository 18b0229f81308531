"""Prompt steps of the RWKV path at the edges of their shapes: token counts around every tile size of the projection kernel,
row counts of the head, sequences of unequal length, against the CPU oracle in the same operand precision."""
import json

import numpy as np
import pytest

from ai00_server_b200 import capi, runtime, synth
from oracle import kemirax_numpy, panupel_numpy, sampling_numpy
from oracle import rwkv_numpy as O

pytestmark = pytest.mark.gpu

# f16 operands, f32 sums: a projection over k inputs is off by about sqrt(k) * 2^-24 of its terms in either order of summation; what
# remains between engine and oracle are operands that such a difference moves to the neighbouring f16 value (2^-11 of one input)
TOL = 1e-3


def _check(preset, lens, full, chunk=512, state_norm=np.inf):
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
            assert np.linalg.norm((got - state).ravel(), state_norm) <= TOL * np.linalg.norm(state.ravel(), state_norm)
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


# steps of more than 128 tokens: 128- and 256-token tiles of the two-SM projections and their remainders, more tokens than a step holds (2048),
# a model whose row-parallel projections keep one part (384 / 3 k blocks) and one with odd numbers of 128-row weight tiles
@pytest.mark.parametrize("n", [383, 385, 513, 1100, 2300])
@pytest.mark.parametrize("shape", ["tiny6", "tiny7", "odd6"])
def test_steps_of_many_tiles(shape, n):
    st = synth.Shape(6, 2, 320, 1160, V=512, Dm=32, Dd=64) if shape == "odd6" else shape
    _check(st, [n], full=False)


@pytest.mark.parametrize("lens", [[1017], [1023], [1031], [7, 1, 8, 6, 1012], [14, 1002, 7, 7, 3], [7, 8, 6, 13, 15, 1] * 21])
@pytest.mark.parametrize("shape", ["tiny5", "tiny7", "odd6"])
def test_rows_of_steps_in_groups_of_seven(shape, lens):
    """Norm and token shift of long steps take seven rows and the one before them a CTA: sequences that begin and end inside, at and between the groups; rows of 320 columns."""
    _check(synth.Shape(6, 2, 320, 1160, V=512, Dm=32, Dd=64) if shape == "odd6" else shape, lens, full=False)


@pytest.mark.parametrize("shape, count", [("tiny5", 240), ("odd6", 96)])
def test_scans_of_many_heads_and_sequences(shape, count):
    """More (head, sequence) pairs than three an SM: groups of eight tokens, parts of one, one and several."""
    _check(synth.Shape(6, 2, 320, 1160, V=512, Dm=32, Dd=64) if shape == "odd6" else shape, ([6, 17, 8] * count)[:count], full=False)


@pytest.mark.parametrize("lens", [[300, 250, 1, 700], [90] * 9])
@pytest.mark.parametrize("preset", ["tiny5", "tiny6", "tiny7"])
def test_rows_of_long_steps(preset, lens):
    """More logits rows than a step keeps (512), more than the bucketed head holds (128), sequences of unequal length."""
    _check(preset, lens, full=True)


@pytest.mark.parametrize("preset", ["tiny5", "tiny6", "tiny7"])
@pytest.mark.parametrize("each", [1, 3])
def test_many_sequences_of_few_tokens(preset, each):
    """Long steps whose sequences hold a few tokens each: the decode recurrence reads and writes tiled operands.

    States by their 2-norm: among 150 x 50 000 entries the largest single one is an entry whose key and value both moved to the neighbouring
    f16 operand, 2 x 2^-11 of it; all entries of a state at once do not, and a wrong row is off by its own size."""
    _check(preset, [each] * 150, full=False, state_norm=2)


@pytest.mark.parametrize("chunk", [1, 9, 33, 100])
def test_long_steps_of_small_chunks(chunk):
    """A step holds sixteen portions of the caller's chunk size, whatever they divide."""
    _check("tiny6", [700, 31], full=False, chunk=chunk)


def test_debug_reads_of_steps_of_every_form():
    """The residual behind a layer's mixer is the one in front of it plus the partial sums of the output projection, and the f16 operands hold the same rows, whatever form
    the last step had and whether it was captured or replayed."""
    st = synth.make_st(synth.Shape(6, 2, 512, 1792, V=512), 3)
    m = runtime.Model(st, max_batch=1, token_chunk_size=128)
    try:
        m.state.reset(0)
        for n in (100, 5, 300, 100, 40, 5, 200):
            m.infer_raw([0], [n], list(range(1, n + 1)), [capi.OPTION_NONE])
            x_a, x_b, parts = (m.debug_read(k, n) for k in ("x_a", "x_b", "part_att"))
            assert np.abs(x_b - x_a - parts).max() <= 1e-5 * np.abs(x_b).max(), n          # f32 sums of a few parts, in another order
            d = m.debug_read("a_x1", n).astype(np.float64)                                # the key operand of the last layer: RWKV-6's mix between xx and sx
            assert np.isfinite(d).all() and (np.abs(d).sum(1) > 0).all(), n
    finally:
        m.close()


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


@pytest.mark.parametrize("lens", [[1100], [700, 500, 3]])
@pytest.mark.parametrize("preset", ["tiny6", "tiny7"])
def test_hidden_rows_of_steps_of_many_rows(preset, lens):
    """keep_hidden over steps of more than a thousand rows, eight of them to a CTA; the logits of the last tokens beside them."""
    st = synth.make_st(preset, 3)
    orc = O.Oracle(O.parse_st(st), "f16")
    toks = [np.random.default_rng(n).integers(1, 500, n).tolist() for n in lens]
    m = runtime.Model(st, max_batch=len(lens), token_chunk_size=128)
    try:
        for s in range(len(lens)):
            m.state.reset(s)
        m.keep_hidden(True)
        rows = m.infer_raw(list(range(len(lens))), lens, sum(toks, []), [capi.OPTION_LAST] * len(lens))
        got = m.last_hidden(max_rows=sum(lens))
        assert got.shape[0] == sum(lens)
        at = 0
        for s, n in enumerate(lens):
            want, _ = orc.hidden(toks[s], orc.state_init())
            assert np.abs(got[at:at + n] - want).max() <= TOL * np.abs(want).max(), s
            last, _ = orc.run(toks[s], orc.state_init())
            assert np.abs(rows[s] - last).max() <= TOL * np.abs(last).max(), s
            at += n
    finally:
        m.close()


# serving precision of the config.json families: bf16 operands (2^-9 each), f32 sums.  A row of a few layers is off by a few of those
# roundings, a few percent where a norm divides by a small read-out; a wrong tile, edge or row list is off by its own size
BF16_TOL = 5e-2
# every single row, the last of a tile among them: a row that was not computed (zeros) is off by its own size, 1, one that holds another row's
# or stale sums by about 1.4
ROW_TOL = 0.5


def _check_family(make, layers, module, n, chunk=512, **kw):
    _check_image(*make(layers, seed=4, **kw), module, n, 0, chunk)


def _check_image(cfg, st, w, module, n, precision, chunk=512):
    toks = np.random.default_rng(n).integers(1, 90, n).tolist()
    m = runtime.Model(st, max_batch=1, token_chunk_size=chunk, config=cfg, kv_tokens=n + 64, kv_page=16, precision=precision)
    try:
        m.state.reset(0)
        got = m.infer_raw([0], [n], toks, [capi.OPTION_FULL])[0]
        want = module.run(json.loads(cfg), w, toks)
        err = np.sqrt(((got - want) ** 2).mean(1)) / np.sqrt((want ** 2).mean())
        assert np.median(err) <= (BF16_TOL if precision == 0 else 2e-4) and err.max() <= (ROW_TOL if precision == 0 else 2e-4), (n, float(np.median(err)), int(err.argmax()), float(err.max()))
    finally:
        m.close()


@pytest.mark.parametrize("family", ["rwkv", "panupel", "kemirax"])
def test_kept_rows_of_long_steps(family):
    """The row a slot keeps for sampling, found through the metadata of a step of more than 128 and of more than 512 tokens."""
    lens = [130, 700, 5]
    rng = np.random.default_rng(5)
    toks = [rng.integers(1, 90, n).tolist() for n in lens]
    kw = {"max_batch": 3, "token_chunk_size": 512}
    if family == "rwkv":
        st = synth.make_st("tiny6", 3)
    else:
        layer = synth.panupel_layer("delta", heads=3, dim=24, ff=200) if family == "panupel" else synth.kemirax_layer("latent_attention", mlp=False)
        cfg, st, _ = (synth.make_panupel if family == "panupel" else synth.make_kemirax)([layer], seed=4)
        kw.update(config=cfg, kv_tokens=1024, kv_page=16)
    m = runtime.Model(st, **kw)
    try:
        for s in range(3):
            m.state.reset(s)
        for call in ([0, 2], [1, 2]):                # 135 tokens in the first step; 705 in the second call's
            rows = m.infer_raw(call, [lens[s] for s in call], sum((toks[s] for s in call), []), [capi.OPTION_LAST] * 2)
            ids, _ = m.sample_topk(call, top_k=20)
            for i in range(2):
                assert np.array_equal(ids[i], sampling_numpy.sorted_candidates(rows[i][0], top_k=20)[0])
    finally:
        m.close()


@pytest.mark.parametrize("n", [17, 32, 33, 64, 65, 127, 128, 129, 300, 513, 1100, 2100])
def test_projections_of_a_step_of_n_rows(n):
    """Row tiles of 32 / 64 / 128, of 128 / 256 on pairs of SMs, and their remainders, outputs and k ranges that are no multiple of a tile; more rows
    than a step holds (2048)."""
    L = synth.panupel_layer
    _check_family(synth.make_panupel, [L("delta", heads=3, dim=24, ff=200), L("parallel", heads=2, dim=40, mm_heads=1, mm_dim=24, ff=72)], panupel_numpy, n,
                  width=136)


@pytest.mark.parametrize("n", [20, 70, 130, 700])
@pytest.mark.parametrize("experts, top", [(3, 1), (8, 4)])
def test_routed_projections_of_a_step_of_n_rows(n, experts, top):
    """Row lists of experts: groups of very unequal size, empty ones among them."""
    layer = synth.kemirax_layer("gla", heads=2, dim=16, vdim=24, experts=experts, identity=1, top=top, ff=88, shared_ff=40)
    _check_family(synth.make_kemirax, [layer], kemirax_numpy, n, width=72)


@pytest.mark.parametrize("n", [130, 300])
@pytest.mark.parametrize("experts, top", [(40, 3), (256, 8), (300, 2)])
def test_row_lists_of_many_experts(n, experts, top):
    """Lists built by matching lanes for more experts than a warp has lanes, for the most that form takes, and one by one for more."""
    layer = synth.kemirax_layer("gla", heads=2, dim=16, vdim=24, experts=experts, identity=1, top=top, ff=24, shared_ff=40)
    _check_family(synth.make_kemirax, [layer], kemirax_numpy, n, width=72)


@pytest.mark.parametrize("chunk", [20, 33, 40, 100])
def test_full_steps_of_chunks_between_the_row_counts_of_launches(chunk):
    """Sixteen chunks that are no row count of a launch (powers of two, multiples of 256): a full step and a little more, grouped projections (a group a head, a group an
    expert) and their operands' buffers at their last rows."""
    layer = synth.kemirax_layer("latent_attention", heads=16, kv_rank=40, rot_dim=16, experts=6, top=3)
    _check_family(synth.make_kemirax, [layer], kemirax_numpy, 16 * chunk + 21, chunk=chunk, width=96)


@pytest.mark.parametrize("n", [1, 9, 16])
@pytest.mark.parametrize("ff", [4740, 4744, 600])
def test_projections_of_a_step_of_few_rows(n, ff):
    """Steps of up to 16 rows: 32 outputs a CTA (2 ff from 9472 on) and 16, ragged last CTAs, k ranges that are no multiple of a lane's 8."""
    _check_family(synth.make_panupel, [synth.panupel_layer("delta", heads=3, dim=24, ff=ff)], panupel_numpy, n, width=136)


@pytest.mark.parametrize("n", [5, 40])
@pytest.mark.parametrize("width", [138, 1020, 1028, 2056, 4104])
def test_boundaries_of_a_row_of_n_columns(width, n):
    """Rows of 1 .. 8 float4 a thread, of whole float4 without whole bf16 operands (1020), and of neither (138)."""
    _check_family(synth.make_panupel, [synth.panupel_layer("delta", heads=2, dim=24, ff=48)], panupel_numpy, n, width=width)


@pytest.mark.parametrize("family, precision", [("kemirax", 0), ("panupel", 0), ("panupel", 1)])
def test_a_token_that_is_not_a_number_reaches_no_row_before_it(family, precision):
    """Attention works on 64 and 128 rows of neighbouring tokens at a time: a later token's value has weight zero in the earlier ones, and zero times NaN must not count."""
    if family == "kemirax":
        layers, make, module = [synth.kemirax_layer("latent_attention", heads=4, mlp=False)], synth.make_kemirax, kemirax_numpy
        cfg, st, w = make(layers, seed=4)
    else:
        layers, make, module = [synth.panupel_layer("parallel", heads=4, kv_heads=2, dim=24, mm_heads=2, mm_dim=24)], synth.make_panupel, panupel_numpy
        cfg, st, w = make(layers, seed=4, width=96, loop=None)
    toks = np.random.default_rng(3).integers(10, 90, 31).tolist()
    toks[20] = 7
    st = st.copy()
    head = int(st[:8].view("<u8")[0])
    e = json.loads(bytes(st[8:8 + head]))["embed"]
    rows = st[8 + head + e["data_offsets"][0]:8 + head + e["data_offsets"][1]].reshape(e["shape"][0], -1)
    rows[7] = np.full(rows.shape[1] // 2, 0x7fc0, "<u2").view(np.uint8)
    m = runtime.Model(st, max_batch=1, token_chunk_size=64, config=cfg, kv_tokens=64, kv_page=16, precision=precision)
    try:
        m.state.reset(0)
        got = m.infer_raw([0], [31], toks, [capi.OPTION_FULL])[0]
        assert np.isnan(got[20:]).all() and np.isfinite(got[:20]).all(), np.isfinite(got).all(1).tolist()
        want = module.run(json.loads(cfg), w, toks[:20])
        err = np.sqrt(((got[:20] - want) ** 2).mean(1)) / np.sqrt((want ** 2).mean())
        assert np.median(err) <= (BF16_TOL if precision == 0 else 2e-4) and err.max() <= (ROW_TOL if precision == 0 else 2e-4), err.tolist()
    finally:
        m.close()


def _tensor(st, name):
    """View of a bf16 tensor's bytes in a file image."""
    head = int(st[:8].view("<u8")[0])
    e = json.loads(bytes(st[8:8 + head]))[name]
    return st[8 + head + e["data_offsets"][0]:8 + head + e["data_offsets"][1]].view("<u2").reshape(e["shape"])


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("dim, vdim", [(72, 40), (128, 128)])
def test_a_decay_that_is_not_a_number_reaches_no_row_before_it(dim, vdim, precision):
    """Gated linear attention sums the logarithms of sixteen tokens' decays: one channel's decay (its bias inf, so 1, or not a number where the low rank overflows to -inf) against the
    same tokens one a step."""
    cfg, st, w = synth.make_kemirax([synth.kemirax_layer("gla", heads=2, dim=dim, vdim=vdim, mlp=False)], seed=9, width=96)
    st = st.copy()
    c = dim + 5                                                    # a channel of the second head
    _tensor(st, "l0.mix.a2.b")[c] = 0x7f80
    _tensor(st, "l0.mix.a2")[c, 0] = 0x7f00                        # 2^127: overflows at -2, about one token in forty
    w = dict(w)
    w["l0.mix.a2.b"] = np.array(w["l0.mix.a2.b"])
    w["l0.mix.a2.b"][c] = 700.0                                    # (decays of one)
    B, n = 8, 60
    toks = np.random.default_rng(3).integers(1, 90, (B, n)).tolist()
    m = runtime.Model(st, max_batch=2 * B, token_chunk_size=512, config=cfg, kv_tokens=64, precision=precision)
    try:
        for s in range(2 * B):
            m.state.reset(s)
        opt = [capi.OPTION_FULL] * B
        got = m.infer_raw(list(range(B)), [n] * B, sum(toks, []), opt)
        one = np.stack([np.concatenate(m.infer_raw(list(range(B, 2 * B)), [1] * B, [t[i] for t in toks], opt)) for i in range(n)], 1)
        first = [int(np.isnan(one[s]).any(1).argmax()) if np.isnan(one[s]).any() else n for s in range(B)]
        assert sum(4 <= f < n and f % 16 >= 4 for f in first) >= 2, first
        for s, f in enumerate(first):
            assert np.isnan(got[s][f:]).all() and np.isfinite(got[s][:f]).all(), (s, f, np.isfinite(got[s]).all(1).tolist())
            want = kemirax_numpy.run(json.loads(cfg), w, toks[s][:f])
            err = np.sqrt(((got[s][:f] - want) ** 2).mean(1)) / np.sqrt((want ** 2).mean())
            assert np.median(err) <= (BF16_TOL if precision == 0 else 2e-4) and err.max() <= (ROW_TOL if precision == 0 else 2e-4), (s, f, err.tolist())
    finally:
        m.close()


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("dim, vdim, n", [(72, 40, 60), (128, 128, 200), (24, 24, 60)])
def test_a_decay_rate_beyond_f32(dim, vdim, n, precision):
    """A head of the delta rule that keeps nothing from token to token (e^100 a token: its logarithms are -inf in f32) beside one that does."""
    cfg, st, w = synth.make_panupel([synth.panupel_layer("delta", heads=2, dim=dim, vdim=vdim)], seed=4, width=96, loop=None)
    st, w = st.copy(), dict(w)
    _tensor(st, "l0.mix.A_log")[1] = 0x42c8
    w["l0.mix.A_log"] = np.array([w["l0.mix.A_log"][0], 100.0])
    _check_image(cfg, st, w, panupel_numpy, n, precision)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("family, layer", [("kemirax", dict(kind="gla", heads=2, dim=72, vdim=40, mlp=False)), ("kemirax", dict(kind="gla", heads=2, dim=128, vdim=128, mlp=False)),
                                           ("panupel", dict(kind="delta", heads=2, dim=72, vdim=40)), ("panupel", dict(kind="delta", heads=2, dim=128, vdim=128)),
                                           ("panupel", dict(kind="parallel", heads=2, dim=24, mm_heads=2, mm_dim=128, mm_vdim=72))])
def test_a_token_that_is_not_a_number_in_a_run_of_sixteen(family, layer, precision):
    """The recurrences that take a prompt's tokens sixteen at a time: a token in the middle of a run leaves the rows before it, in the same run too, as they are."""
    if family == "kemirax":
        make, module, kw, at = synth.make_kemirax, kemirax_numpy, {}, synth.kemirax_layer
    else:
        make, module, kw, at = synth.make_panupel, panupel_numpy, {"loop": None}, synth.panupel_layer
    cfg, st, w = make([at(**layer)], seed=4, width=96, **kw)
    toks = np.random.default_rng(3).integers(10, 90, 80).tolist()
    toks[40] = 7
    st = st.copy()
    _tensor(st, "embed")[7] = 0x7fc0
    m = runtime.Model(st, max_batch=1, token_chunk_size=128, config=cfg, kv_tokens=128, kv_page=16, precision=precision)
    try:
        m.state.reset(0)
        got = m.infer_raw([0], [80], toks, [capi.OPTION_FULL])[0]
        assert np.isnan(got[40:]).all() and np.isfinite(got[:40]).all(), np.isfinite(got).all(1).tolist()
        want = module.run(json.loads(cfg), w, toks[:40])
        err = np.sqrt(((got[:40] - want) ** 2).mean(1)) / np.sqrt((want ** 2).mean())
        assert np.median(err) <= (BF16_TOL if precision == 0 else 2e-4) and err.max() <= (ROW_TOL if precision == 0 else 2e-4), err.tolist()
    finally:
        m.close()


def test_a_nan_stays_one_in_latent_attention():
    """A key that is not a number makes every later row so (rounding to TF32 by integer arithmetic must not turn it into a number)."""
    cfg, st, _ = synth.make_kemirax([synth.kemirax_layer("latent_attention", mlp=False)], seed=4)
    st = st.copy()
    head = int(st[:8].view("<u8")[0])
    e = json.loads(bytes(st[8:8 + head]))["embed"]
    rows = st[8 + head + e["data_offsets"][0]:8 + head + e["data_offsets"][1]].reshape(e["shape"][0], -1)
    rows[7] = np.full(rows.shape[1] // 2, 0x7fc0, "<u2").view(np.uint8)
    m = runtime.Model(st, max_batch=1, token_chunk_size=32, config=cfg, kv_tokens=64, kv_page=16)
    try:
        m.state.reset(0)
        got = m.infer_raw([0], [24], [1, 2, 7] + list(range(10, 31)), [capi.OPTION_FULL])[0]
        assert np.isnan(got[2:]).all()
    finally:
        m.close()
