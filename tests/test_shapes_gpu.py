"""Kernels at the sizes where their tiles, chunks and lists begin, end and change over."""

import numpy as np
import pytest

from distributed_kge_poplar_b200 import capi
from helpers import assert_close, engine_settings, make_oracle, random_state, write_state
from oracle import step_oracle as so
from oracle.step_oracle import StepConfig
from test_predict_gpu import RW, _clear, _predict

pytestmark = pytest.mark.gpu
RTOL = 1e-5


@pytest.mark.parametrize("fn", [capi.L1, capi.L2, capi.DOT], ids=["l1", "l2", "dot"])
@pytest.mark.parametrize("shape", [(64, 37889, 4), (65, 18950, 36), (1, 37890, 32)])
def test_scores_in_whole_tiles(fn, shape):
    """Enough 64 x 128 tiles to fill the GPU: full and ragged tiles, one chunk of k and a remainder."""
    m, n, k = shape
    rng = np.random.RandomState(n)
    a, b = rng.normal(size=(m, k)).astype(np.float32), rng.normal(size=(n, k)).astype(np.float32)
    b[7] = a[0]
    a64, b64 = a.astype(np.float64), b.astype(np.float64)
    want = {capi.L1: so.l1_distance, capi.L2: so.l2_distance, capi.DOT: lambda x, y: x @ y.T}[fn](a64, b64)
    assert_close(capi.op_pairwise(fn, a, b), want, RTOL, f"scores {shape}")


@pytest.mark.parametrize("shape", [(1, 64, 64), (8, 65, 63), (9, 63, 65), (17, 129, 2), (600, 590, 250)])
def test_l1_gradients_add_up_in_order(shape):
    """Chunks of 64 and column tiles of 64 with and without a remainder; one and two rows per warp.  The terms are added
    in index order, so the result has the bits of a plain fp32 loop."""
    m, n, k = shape
    rng = np.random.RandomState(m + n + k)
    a, b = rng.normal(size=(m, k)).astype(np.float32), rng.normal(size=(n, k)).astype(np.float32)
    b[-1] = a[0]
    g = rng.normal(size=(m, n)).astype(np.float32)
    want_a, want_b = np.zeros_like(a), np.zeros_like(b)
    for j in range(n):
        want_a += g[:, j : j + 1] * np.sign(a - b[j])
    for i in range(m):
        want_b += g[i, :, None] * np.sign(b - a[i])
    got_a, got_b = capi.op_pairwise_grad(capi.L1, a, b, g)
    np.testing.assert_array_equal(got_a, want_a)
    np.testing.assert_array_equal(got_b, want_b)


@pytest.mark.parametrize("n,rows", [(1, 1), (31, 2), (32, 63), (33, 64), (511, 65), (512, 4095), (513, 4096), (4095, 3), (4096, 4097)])
def test_lookups_are_sorted_stably(n, rows):
    """Radix passes of six bits (1, 63, 64, 65, 4095 ... rows), warps with no, some and all of their positions."""
    rng = np.random.RandomState(n)
    idx = (rows * rng.random_sample(n) ** 3).astype(np.uint32)
    grad = rng.normal(size=(n, 5)).astype(np.float32)
    want = np.zeros((rows, 5), np.float32)
    np.add.at(want, idx, grad)
    np.testing.assert_array_equal(capi.op_scatter_add_rows(grad, idx, rows), want)


@pytest.mark.parametrize("score_fn,distance_fn", [("TransE", "L1"), ("TransE", "L2"), ("DistMult", "MatMul")])
@pytest.mark.parametrize("n_best", [1, 32, 33, 128])
@pytest.mark.parametrize("pass_rows", [256, 640])
def test_ranking_lists(monkeypatch, score_fn, distance_fn, n_best, pass_rows):
    """First scans, appended merges and full lists: the shortest and longest lists, and the change from one to four
    largest keys per lane."""
    monkeypatch.setenv("KGE_PREDICT_PASS_ROWS", str(pass_rows))
    cfg = StepConfig(n_shard=2, n_entity=1500, n_relation_type=4, embedding_size=16, entity_feature_size=0, batch_size=8, a2a_size=6,
                     score_fn=score_fn, distance_fn=distance_fn, gamma=8.0)
    state = random_state(cfg, 3, warm=True)
    engine = capi.CEngine(engine_settings(cfg, rw_batch=RW, **{"execution.predict_hr_batch_size": 9, "execution.predict_n_best": n_best}))
    write_state(engine, cfg, state, RW)
    rng = np.random.RandomState(1)
    queries = np.stack([np.arange(18) % 2, 1 + rng.randint(1499, size=18), rng.randint(4, size=18)], axis=1)
    counts = np.array([1499, 700])
    got_idx, got_score = _predict(engine, cfg, queries, counts, 9, n_best)
    engine.close()
    want_idx, want_score = make_oracle(cfg, state).predict(queries, counts, n_best)
    assert_close(got_score, want_score, RTOL, "ranking: scores")
    clear = _clear(want_score) if n_best > 1 else np.ones_like(want_score, bool)
    np.testing.assert_array_equal(got_idx[clear], want_idx[clear])


def _rank_whole_tiles(cfg, state, queries, counts):
    engine = capi.CEngine(engine_settings(cfg, rw_batch=RW, feature_dtype="float16", **{"execution.predict_hr_batch_size": len(queries), "execution.predict_n_best": 10}))
    write_state(engine, cfg, state, RW)
    engine.set_kernel_timing(True)
    got = _predict(engine, cfg, queries, counts, len(queries), 10)
    assert "predict_planes" in engine.kernel_times(), "the tensor cores have not ranked"
    engine.close()
    return got


@pytest.mark.parametrize("score_fn,distance_fn", [("TransE", "L2"), ("DistMult", "MatMul")])
@pytest.mark.parametrize("queries,rows,size,features", [(129, 9473, 20, 0), (130, 9500, 132, 70), (5, 18945, 12, 9)])
def test_ranking_in_whole_tiles(monkeypatch, score_fn, distance_fn, queries, rows, size, features):
    """Passes with 148 and more tiles (float16 planes): ragged rows, columns and depths, rows of very different size, and
    a last pass below 148."""
    monkeypatch.setenv("KGE_PREDICT_PASS_ROWS", str(rows // 4 * 4))
    n_entity = rows + 300
    cfg = StepConfig(n_shard=1, n_entity=n_entity, n_relation_type=4, embedding_size=size, entity_feature_size=features, batch_size=8, a2a_size=8,
                     score_fn=score_fn, distance_fn=distance_fn, gamma=8.0)
    state = random_state(cfg, 3, fp16_features=True, warm=True)
    state["entity_data"][0, 1::3, :size] *= 1e-3
    rng = np.random.RandomState(1)
    hr = np.stack([np.zeros(queries, int), 1 + rng.randint(n_entity - 1, size=queries), rng.randint(4, size=queries)], axis=1)
    got_idx, got_score = _rank_whole_tiles(cfg, state, hr, np.array([n_entity - 1]))
    want_idx, want_score = make_oracle(cfg, state).predict(hr, np.array([n_entity - 1]), 10)
    assert_close(got_score, want_score, RTOL, "ranking: scores")
    clear = _clear(want_score)
    np.testing.assert_array_equal(got_idx[clear], want_idx[clear])


@pytest.mark.parametrize("score_fn,distance_fn", [("TransE", "L2"), ("DistMult", "MatMul")])
@pytest.mark.parametrize("filter_in_scores", ["1", "0"])
def test_ranking_in_several_passes_of_whole_tiles(monkeypatch, score_fn, distance_fn, filter_in_scores):
    """From the second pass on every query has a cut-off, and scores reach the lists through the filter inside the
    whole-tile kernel or the kernel of its own; rows that equal the best candidate tie with it in every pass."""
    monkeypatch.setenv("KGE_PREDICT_PASS_ROWS", "9472")
    monkeypatch.setenv("KGE_PREDICT_FILTER_IN_SCORES", filter_in_scores)
    rows, size, n_query = 3 * 9472 + 1, 20, 130
    cfg = StepConfig(n_shard=1, n_entity=rows, n_relation_type=4, embedding_size=size, entity_feature_size=0, batch_size=8, a2a_size=8,
                     score_fn=score_fn, distance_fn=distance_fn, gamma=8.0)
    state = random_state(cfg, 9)
    for first in (50, 9000, 15000, 28000):  # pairs of equal rows, the second a pass or a few rows later
        state["entity_data"][0, first + 400] = state["entity_data"][0, first]
    rng = np.random.RandomState(1)
    queries = np.stack([np.zeros(n_query, int), 1 + rng.randint(rows - 1, size=n_query), rng.randint(4, size=n_query)], axis=1)
    queries[:4, 1] = [50, 9000, 15000, 28000]
    state["relation_embedding"][0] = 0 if distance_fn == "L2" else 1  # the queries' own rows are the best candidates
    queries[:4, 2] = 0
    got_idx, got_score = _rank_whole_tiles(cfg, state, queries, np.array([rows - 1]))
    want_idx, want_score = make_oracle(cfg, state).predict(queries, np.array([rows - 1]), 10)
    assert_close(got_score, want_score, RTOL, "ranking: scores")
    clear = _clear(want_score)
    np.testing.assert_array_equal(got_idx[clear], want_idx[clear])
    if distance_fn == "L2":
        np.testing.assert_array_equal(got_idx[:4, :2, 1], [[r, r + 400] for r in (50, 9000, 15000, 28000)])


def test_transh_ranking_in_one_pass_of_more_than_2_32_values(monkeypatch):
    """A pass of 1 060 000 rows of 4096 columns: offsets into its hidden rows need more than 32 bits.  Passes of the usual
    length give the same lists."""
    rows, size, queries, n_best = 1_060_000, 4096, 8, 128
    cfg = StepConfig(n_shard=1, n_entity=rows, n_relation_type=2, embedding_size=size, entity_feature_size=0, batch_size=4, a2a_size=4,
                     score_fn="TransH", distance_fn="L1", gamma=8.0)
    rng = np.random.RandomState(2)
    variables = {name: rng.normal(size=(2, size)).astype(np.float32) for name in ("relation_embedding", "relation_normal")}
    got = []
    for pass_rows in (None, rows):
        if pass_rows:
            monkeypatch.setenv("KGE_PREDICT_PASS_ROWS", str(pass_rows))
        engine = capi.CEngine(engine_settings(cfg, dtype="float16", rw_batch=RW, **{"execution.predict_hr_batch_size": queries, "execution.predict_n_best": n_best}))
        engine.run("initialise_entities", {})
        for name, value in variables.items():
            engine.run("write", {"value": value}, name=name)
        hr = np.stack([np.zeros(queries, int), 1 + np.arange(queries) * 1000, np.arange(queries) % 2], axis=1)
        got.append(_predict(engine, cfg, hr, np.array([rows - 1]), queries, n_best))
        engine.close()
    (idx, score), (idx_whole, score_whole) = got
    assert np.sum(idx[..., 1] >= 2**32 // size) > 0, "no candidate behind the first 2^32 values: the case shows nothing"
    np.testing.assert_array_equal(score_whole, score)
    np.testing.assert_array_equal(idx_whole, idx)


@pytest.mark.parametrize("score_fn,distance_fn", [("TransE", "L2"), ("DistMult", "MatMul")])
@pytest.mark.parametrize("spread", [6, 12, 20])
def test_ranking_rows_with_columns_of_very_different_size(monkeypatch, score_fn, distance_fn, spread):
    """Passes on float16 planes whose rows range over 2^(2 * spread).  For products the queries range the other way round,
    so that every column counts alike: 2^12 fits the planes, 2^24 needs all of them, and at 2^40 the values that matter lie
    below their last bit and the pair is recomputed.  1e-5, as two TF32 planes keep it."""
    rows, size, n_query = 9473, 132, 129
    monkeypatch.setenv("KGE_PREDICT_PASS_ROWS", str(rows // 4 * 4))
    cfg = StepConfig(n_shard=1, n_entity=rows, n_relation_type=4, embedding_size=size, entity_feature_size=0, batch_size=8, a2a_size=8,
                     score_fn=score_fn, distance_fn=distance_fn, gamma=8.0)
    state = random_state(cfg, 5)
    scale = np.exp2(np.random.RandomState(6).permutation(np.linspace(-spread, spread, size).round())).astype(np.float32)
    state["entity_data"][..., :size] *= scale
    state["relation_embedding"] *= scale if distance_fn == "L2" else 1 / scale**2
    rng = np.random.RandomState(1)
    queries = np.stack([np.zeros(n_query, int), 1 + rng.randint(rows - 1, size=n_query), rng.randint(4, size=n_query)], axis=1)
    got_idx, got_score = _rank_whole_tiles(cfg, state, queries, np.array([rows - 1]))
    want_idx, want_score = make_oracle(cfg, state).predict(queries, np.array([rows - 1]), 10)
    assert_close(got_score, want_score, RTOL, "ranking: scores")
    clear = _clear(want_score)
    np.testing.assert_array_equal(got_idx[clear], want_idx[clear])


@pytest.mark.parametrize("spread,masked", [(6, False), (12, False), (12, True), (25, True)])
def test_ranking_with_a_projection_of_very_different_rows(monkeypatch, spread, masked):
    """The hidden rows' contraction: projection rows that range over 2^(2 * spread) against features that range the other
    way round (float16, so over 2^24 at most), or whose features are zero where the projection is large: what is left lies
    2^spread below the largest value of its column.  At 2^25 the planes are too short and the pass takes the TF32 ones."""
    rows, size, features, n_query = 9500, 132, 70, 130
    monkeypatch.setenv("KGE_PREDICT_PASS_ROWS", str(rows // 4 * 4))
    cfg = StepConfig(n_shard=1, n_entity=rows, n_relation_type=4, embedding_size=size, entity_feature_size=features, batch_size=8, a2a_size=8,
                     score_fn="DistMult", distance_fn="MatMul", gamma=8.0)
    state = random_state(cfg, 7, fp16_features=True)
    state["entity_data"][..., :size] *= 1e-3  # the scores show the projection
    feat = state["entity_data"][..., 3 * size :]
    if masked:
        large = np.arange(features) % 2 == 0
        feat[..., large] = 0
        state["feature_projection"][large] *= np.float32(2.0 ** (2 * spread - 6))
        state["feature_projection"][~large] *= np.float32(2.0**-6)
        feat *= np.float32(2.0**6)
    else:
        scale = np.exp2(np.random.RandomState(8).permutation(np.linspace(-spread, spread, features).round())).astype(np.float32)
        feat[...] = (feat * scale).astype(np.float16).astype(np.float32)
        state["feature_projection"] /= scale[:, None]
    rng = np.random.RandomState(1)
    queries = np.stack([np.zeros(n_query, int), 1 + rng.randint(rows - 1, size=n_query), rng.randint(4, size=n_query)], axis=1)
    got_idx, got_score = _rank_whole_tiles(cfg, state, queries, np.array([rows - 1]))
    want_idx, want_score = make_oracle(cfg, state).predict(queries, np.array([rows - 1]), 10)
    assert_close(got_score, want_score, RTOL, "ranking: scores")
    clear = _clear(want_score)
    np.testing.assert_array_equal(got_idx[clear], want_idx[clear])
